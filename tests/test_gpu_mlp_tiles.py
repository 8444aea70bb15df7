"""The fused training kernel at the sizes where a tile can go wrong: one row,
a tile less and more one row, more tiles than SMs (a CTA takes several), and a
permutation of the rows, against FP64 autograd of the same network."""
import numpy as np
import pytest
import torch

from noa_gb300.surrogate import NPARAM, Surrogate, init_params
from tests.test_gpu_mlp import BLOCKS, torch_reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000, 128 * 152 + 1])
def test_gradient_sizes(cuda_device, n):
    rng = np.random.default_rng(n)
    params = init_params(seed=7)
    params[33664:33792] *= 10
    X = rng.uniform(-1, 1, (n, 4)).astype(np.float32)
    T = rng.normal(0, 1, n).astype(np.float32)
    s = Surrogate(1, batch=128 * 160)
    s.set_params(params, np.zeros(10, np.float32))
    g, loss = s.gradient(torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda())
    ref_loss, ref_g = torch_reference(params, X, T)
    g = g.cpu().numpy().astype(np.float64)
    # bars of the gradient test: BF16 gradient operands, 2^-8 per element, averaged
    # over the rows; a single row has no averaging
    bar = 2e-2 if n > 100 else 4e-2
    assert abs(loss - ref_loss) <= 1e-4 * abs(ref_loss)
    for name, (a, b) in BLOCKS.items():
        rel = np.linalg.norm(g[a:b] - ref_g[a:b]) / max(np.linalg.norm(ref_g[a:b]), 1e-30)
        assert rel < bar, (name, rel)


@pytest.mark.parametrize("n", [1, 127, 129, 128 * 153])
def test_prediction_sizes(cuda_device, n):
    rng = np.random.default_rng(n)
    s = Surrogate(2, batch=128)
    s.set_params(init_params(seed=8), np.zeros(10, np.float32))
    X = torch.from_numpy(rng.uniform(-1, 1, (n, 4)).astype(np.float32)).cuda()
    whole = s.predict(X)
    # a row's prediction depends on the row only
    order = torch.randperm(n, generator=torch.Generator().manual_seed(1)).cuda()
    assert torch.equal(s.predict(X[order]), whole[order])


def test_training_step_is_adam_on_the_permuted_batch(cuda_device):
    rng = np.random.default_rng(2)
    n, batch = 700, 256
    X = torch.from_numpy(rng.uniform(-1, 1, (n, 4)).astype(np.float32)).cuda()
    T = torch.from_numpy(rng.normal(0, 1, n).astype(np.float32)).cuda()
    s = Surrogate(1, batch=batch)
    p0 = init_params(seed=9)
    s.set_params(p0, np.zeros(10, np.float32))
    perm = torch.randperm(n, generator=torch.Generator(device="cuda").manual_seed(0), device="cuda")[:batch]
    g, loss = s.gradient(X[perm], T[perm])
    losses = s.fit(X, T, steps=1, lr=1e-3, lr_final=1e-3, seed=0)
    p1, m, v, step = s.get_params()
    g = g.cpu().numpy()
    assert step == 1 and abs(float(losses[0]) - loss) <= 1e-5 * loss
    # float32 atomics in another order move a gradient entry by about 1e-6 of its block
    np.testing.assert_allclose(m, 0.1 * g, rtol=1e-3, atol=1e-7 + 1e-5 * np.abs(g).max())
    big = np.abs(g) > 1e-3 * np.abs(g).max()
    np.testing.assert_allclose((p0 - p1)[big], 1e-3 * np.sign(g[big]), rtol=1e-2)
    assert p1.size == NPARAM
