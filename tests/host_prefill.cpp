// The prompt GEMM's operand staging (slai_b200/csrc/prefill_dequant.cuh) on the host: one 16-row tile, every thread of the warp
// that serves it in turn.  Usage: host_prefill <fmt> <K> <blocks.bin (16 rows, GGUF order)>  -> 16 x K doubles (binary, stdout):
// the weights as the kernel's products see them (the words that go to tensor memory, both planes added, times the row scale, minus
// the minimum term).
#include <cstdio>
#include <cstdlib>
#include <vector>
#include <cuda_fp16.h>

#include "../slai_b200/csrc/gemv_formats.cuh"
#include "../slai_b200/csrc/prefill_dequant.cuh"

namespace hostemu {
thread_local int lane;
thread_local Warp* warp;
}  // namespace hostemu

static double at(const unsigned char* plane, int row_bytes, int swz, int r, int k) {
    const int c = (k >> 3) ^ swz;
    return (double)__half2float(*reinterpret_cast<const __half*>(plane + r * row_bytes + 16 * c + 2 * (k & 7)));
}
static double half_bits(uint32_t b) {
    __half_raw h;
    h.x = (unsigned short)b;
    return (double)__half2float(__half(h));
}

template <int FMT>
static void run(const std::vector<uint8_t>& tile, int K, std::vector<double>& out) {
    using F = pfq::Fmt<FMT>;
    const int elems = layout::step_elems(FMT), steps = (int)layout::num_steps(FMT, K);
    for (int tile_row = 0; tile_row < 128; tile_row += 112)  // first and last 16 rows of a CTA's 128
        for (int c = 0; c < steps; c++) {
            alignas(16) unsigned char mn[128 * 32];
            const unsigned char* blk = tile.data() + (size_t)c * F::STEP;
            for (int lane = 0; lane < 32 && F::MIN; lane++) pfq::min_row(blk, lane & 15, tile_row + (lane & 15), lane >> 4, mn);
            for (int st = 0; st < F::STAGES; st++) {
                double sum[16][64];  // 16 rows, the stage's 64 columns
                for (int lane = 0; lane < 32; lane++) {
                    const int r16 = lane & 15, part = lane >> 4;
                    pfq::Packed p = {};
                    pfq::fetch<FMT>(blk, r16, part, st, p);
                    uint32_t hi[16], lo[16] = {};
                    pfq::make<FMT>(p, st, hi, lo);
                    for (int i = 0; i < 32; i++) {  // the words' halves
                        const int col = FMT == 8 ? 32 * part + i : 32 * (i >> 4) + 16 * part + (i & 15), sh = 16 * (i & 1);
                        sum[r16][col] = half_bits((hi[i >> 1] >> sh) & 0xFFFF) + (F::PLANES == 2 ? half_bits((lo[i >> 1] >> sh) & 0xFFFF) : 0.0);
                    }
                }
                for (int r16 = 0; r16 < 16; r16++) {
                    const int r = tile_row + r16;
                    const uint32_t dd = F::SCALED ? pfq::row_scale<FMT>(blk, r16) : 0u;
                    for (int k = 0; k < 64; k++) {
                        const int col = c * elems + 64 * st + k;
                        if (col >= K) continue;
                        double w = sum[r16][k];
                        if (F::SCALED) w *= half_bits(dd & 0xFFFF);
                        if (F::MIN) {
                            const int j = 2 * st + (k >> 5), sw = (r >> 2) & 1;
                            const double m = at(mn, 32, sw, r, j);
                            if (at(mn, 32, sw, r, 8 + j) * 2048.0 != m) exit(3);
                            w -= half_bits(dd >> 16) * m;
                        }
                        double& o = out[(size_t)r16 * K + col];
                        if (tile_row > 0 && o != w) exit(4);  // the same whatever the tile's place in the CTA
                        o = w;
                    }
                }
            }
        }
}

int main(int argc, char** argv) {
    if (argc < 4) return 2;
    const int fmt = atoi(argv[1]), K = atoi(argv[2]);
    const int be = fmt == 8 ? 32 : 256, bb = fmt == 8 ? 34 : fmt == 12 ? 144 : fmt == 13 ? 176 : 210, nbk = K / be;
    std::vector<uint8_t> raw((size_t)16 * nbk * bb);
    FILE* f = fopen(argv[3], "rb");
    if (!f || fread(raw.data(), 1, raw.size(), f) != raw.size()) return 2;
    fclose(f);
    std::vector<uint8_t> tile((size_t)layout::tile_bytes(fmt, K) + 16, 0);
    for (int r = 0; r < 16; r++)
        for (int b = 0; b < nbk; b++) layout::place_block(fmt, raw.data() + ((size_t)r * nbk + b) * bb, tile.data(), r, b, K);
    std::vector<double> out((size_t)16 * K, 0.0);
    switch (fmt) {
        case 8: run<8>(tile, K, out); break;
        case 12: run<12>(tile, K, out); break;
        case 13: run<13>(tile, K, out); break;
        case 14: run<14>(tile, K, out); break;
    }
    fwrite(out.data(), 8, out.size(), stdout);
    return 0;
}
