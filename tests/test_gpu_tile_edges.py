"""The sizes at which a launch's tile or its number of steps changes, from the SM
count and the constants in the kernels' sources: from the smallest tile to the next
and from one step to two and three.  A pair's bits must not depend on them, and
nothing outside the call's range may be written."""
import os
import re

import pytest
import torch

from noa_gb300 import build, dcs
from noa_gb300.elements import ELEMENTS
from noa_gb300.workload import kinetic_recoil
from tests.parity import PROCESSES

pytestmark = pytest.mark.gpu


def find(source, pattern):
    with open(os.path.join(build.CSRC, source)) as f:
        return [int(x) for x in re.search(pattern, f.read()).groups()]


def shape(process, precision):
    """Resident CTAs an SM, largest tile and smallest tile."""
    if precision == "fp64":
        if process in (0, 3):  # one pair a thread, no tile
            return 1, find("dcs_fp64.cu", r"MAP_THREADS = (\d+);")[0], 1
        ctas = find("dcs_fp64.cu", r"define NOA_DCS_%s_MIN_CTAS (\d+)" % ("PPROD", "PHOTO")[process - 1])[0]
        threads, items = (find("dcs_fp64.cu", r"%s = (\d+);" % n)[0] for n in ("CMP_THREADS", "CMP_ITEMS"))
        return ctas, threads * items, find("dcs_fp64.cu", r"tile = tile < (\d+) \? \1 : tile;")[0]
    by_process = find("dcs_fp32c.cu", r"NOA_DCS_PROC_PPROD \? (\d+) : \(PROC == NOA_DCS_PROC_PHOTO \? (\d+) : (\d+)\)")
    ctas = by_process[{1: 0, 2: 1}.get(process, 2)]
    threads, items = (find("dcs_fp32c.cu", r"%s = (\d+);" % n)[0] for n in ("F_THREADS", "F_ITEMS"))
    return ctas, threads * items, find("dcs_fp32c.cu", r"tile = tile < (\d+) \? \1 : tile;")[0]


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("process", range(4), ids=PROCESSES)
def test_tile_and_step_edges(cuda_device, process, precision):
    ctas, most, least = shape(process, precision)
    cap = torch.cuda.get_device_properties(0).multi_processor_count * ctas
    sizes = [edge + d for edge in (least * cap, (least + 1) * cap, most * cap, 2 * most * cap) for d in (-1, 0, 1)]
    K, q = (torch.from_numpy(a).cuda() for a in kinetic_recoil(max(sizes) + 7, offset=6 << 20))
    whole = dcs.map(process, K, q, ELEMENTS[26], precision=precision)
    for n in sizes:
        for start in (0, 7):
            got = torch.full((n + 2,), -7.0, dtype=torch.float64, device="cuda")
            dcs.vmap(process, got[1:n + 1], K[start:start + n], q[start:start + n], ELEMENTS[26], precision=precision)
            assert torch.equal(got[1:n + 1].view(torch.int64), whole[start:start + n].view(torch.int64)), n
            assert float(got[0]) == -7.0 and float(got[n + 1]) == -7.0
