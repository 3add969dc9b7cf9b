// decode_layers.cuh for Q6_K weights (a file per format: they compile side by side).
#include "decode_layers.cuh"

int decode_layers_launch_q6k(slai_ctx* ctx, const declayers::LayersParams& P, int arch, bool f16, int grid, size_t smem) {
    return declayers::launch_fmt<gemvfmt::Q6K>(ctx, P, arch, f16, grid, smem);
}
