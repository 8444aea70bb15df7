// Host check of the batched engine's tile layout (the plan's own source): for
// every tile shape, the tile that a sampled layout (the autotuner's) is timed at is
// the one that the plan runs, and the layout covers each segment's sample.  Prints
// "shapes <n> wrong <m>".  Built and run by tests/test_batch_tiles_host.py.
#include "../noa_gb300/csrc/dcs_batch_plan.cu"

#include <cstdlib>

cudaError_t noa_dcs_batched_launch64(int, int, const void *, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t noa_dcs_batched_launch32(int, int, const void *, int, size_t, cudaStream_t) { return cudaSuccess; }
int noa_dcs_batched_occupancy64(int, int, size_t) { return 2; }
int noa_dcs_batched_occupancy32(int, int, size_t) { return 2; }

int main() {
    const int64_t sample = 1 << 17;
    const int64_t sizes[] = {100, 1000, 20001, 131072, 300000, 2400000, 30000000};
    int shapes = 0, wrong = 0;
    for (int precision : {NOA_DCS_FP64, NOA_DCS_FP32C})
        for (int64_t size : sizes)
            for (int n_seg : {1, 3, 10})
                for (int threads : {128, 256})
                    for (int items : {1, 2, 4, 8})
                        for (int ctas : {1, 2, 4}) {
                            noa_dcs_batch_plan p;
                            std::memset(&p.params, 0, sizeof p.params);
                            p.precision = precision;
                            p.sms = 152;
                            p.threads = threads;
                            p.items = items;
                            p.ctas_per_sm = ctas;
                            p.params.n_seg = n_seg;
                            for (int s = 0; s < n_seg; s++)
                                p.params.seg_begin[s + 1] = p.params.seg_begin[s] + (s % 2 ? size / 7 : size);
                            noa_dcs_batch_plan t = p;
                            set_tiles(&p);
                            set_tiles(&t, sample);
                            bool ok = t.params.tile == p.params.tile && t.params.items == p.params.items;
                            for (int s = 0; s < n_seg; s++) {
                                int64_t count = p.params.seg_begin[s + 1] - p.params.seg_begin[s];
                                count = count < sample ? count : sample;
                                const int64_t tiles = t.params.tile_begin[s + 1] - t.params.tile_begin[s];
                                ok = ok && tiles * t.params.tile >= count && (tiles - 1) * t.params.tile < count;
                            }
                            shapes++;
                            wrong += ok ? 0 : 1;
                        }
    std::printf("shapes %d wrong %d\n", shapes, wrong);
    return 0;
}
