// Host side of the layers of a decode step in one launch (decode_layers.cuh): which models take it, and its parameters.
#include <limits.h>
#include <math.h>

#include <algorithm>

#include "attention.cuh"
#include "decode_layers.cuh"

using namespace declayers;

namespace {
// Floats of the splits' partial outputs every block reads back when it stages the attention output (one more split of 4096 rows costs
// about 0.3 us a layer).
constexpr int MAX_PART = 32768;

// Layers of few bytes go to one cluster of 16 blocks instead of the whole chip: the cluster's hardware barrier takes 0.25 us, the grid's 1.0 to 1.2, five times a
// layer, which is more than 16 SMs lose on few bytes.  us a token, whole chip / one cluster: tiny story model (1.1 MB a layer, Q8_0) 125.7 / 111.1,
// 256 wide Q4_K (0.5 MB) 171 / 149, 512 wide Q4_K (1.8 MB) 171 / 161, 512 wide Q6_K (2.2 MB) 202 / 195; but 768 wide Q5_K (5.1 MB) 182 / 200 and
// 1024 wide Q6_K (9.4 MB) 226 / 277.  Keys and values count half, since their loads are ahead of the barrier: 16 SMs read them in all (at most 16 / items splits).
// us a token at positions 500, 2000, 8000 of 8 layers 512 wide, f32 cache, whole chip 176, 198, 264, one cluster 174, 241, 558 (kernel by kernel 221, 246, 317);
// f16 173, 182, 228 and 171, 200, 390; 256 wide, f16 170, 178, 202 and 147, 161, 237.
constexpr int CLUSTER = 16;
constexpr long long CLUSTER_BYTES = 3000000;
long long weight_bytes(const DecodeLayers& D) {  // of a layer
    const long long rows_dim = (long long)D.q_dim + 2 * D.kv_dim + (D.arch == ARCH_LLAMA ? 2 : 1) * (long long)D.hidden;  // matrices of width `dim`
    auto bytes = [&](long long rows, int K) { return rows * layout::num_steps(D.fmt, K) * layout::step_bytes(D.fmt) / 16; };
    return bytes(rows_dim, D.dim) + bytes(D.dim, D.q_dim) + bytes(D.dim, D.hidden);
}
bool one_cluster(const DecodeLayers& D) { return !D.whole_chip && weight_bytes(D) < CLUSTER_BYTES; }

struct Plan {
    int grid = 0;
    size_t smem = 0;
};

bool plan(slai_ctx* ctx, const DecodeLayers& D, bool cluster, LayersParams& P, Plan& pl) {
    const int esz = D.kv_f16 ? 2 : 4, hs = D.head_size;
    if (ctx->sm_count <= 0 || D.n_layers < 1 || D.n_layers > MAX_LAYERS) return false;
    if (hs % 8 || hs * esz < 64 || hs * esz > 512) return false;  // a cached row is 4 to 32 lanes, 16 bytes each; eight elements share a lane's work
    if (D.arch == ARCH_GPT2 && (D.dim > 256 * WARPS || D.kv_mul != 1)) return false;  // (stage_steps: a LayerNorm in one round)
    if (D.q_dim >= 1 << 16 || (long long)D.kv_dim * D.seq_len >= 1ll << 31) return false;  // (hs_magic; a cache layer's elements)
    const int be = fmt_block_elems(D.fmt);
    if (D.fmt == SLAI_FMT_F32 || be == 0 || D.dim % be || D.q_dim % be || D.hidden % be) return false;
    int step_b = layout::step_bytes(D.fmt);
    if (step_b == 0) return false;

    auto tiles = [](int rows) { return (rows + 15) / 16; };
    P.tile_k = tiles(D.q_dim);
    P.tile_v = P.tile_k + tiles(D.kv_dim);
    P.q_rows = D.q_dim;
    P.kv_rows = D.kv_dim;
    const int K[PH_COUNT] = {D.dim, D.q_dim, D.dim, D.hidden};
    const int items[PH_COUNT] = {P.tile_v + tiles(D.kv_dim), tiles(D.dim), tiles(D.hidden), tiles(D.dim)};
    const int rows[PH_COUNT] = {0, D.dim, D.hidden, D.dim};
    const int share = attn::attn_kv_share(D.kv_mul);
    P.kv_share = share;
    P.kvq = D.kv_mul / share;
    P.n_heads = D.n_heads;
    P.n_items = D.n_heads / P.kvq;
    // What the kernels one by one refuse (attention.cu, gemv.cu) is theirs to refuse: they are what the statistics run too.
    if (D.kv_mul > 8 || P.kvq > 2 || D.n_heads / D.kv_mul * share > 1024) return false;
    for (int k : K)
        if (!gemv_width_fits(D.fmt, k)) return false;
    // No more blocks than some phase has tiles: a barrier of fewer blocks is quicker.
    pl.grid = std::min(ctx->sm_count, *std::max_element(items, items + PH_COUNT));
    P.cluster = cluster && one_cluster(D) ? 1 : 0;
    if (P.cluster) pl.grid = CLUSTER;

    size_t dig = 0;
    int red = 0, inv = 0;
    for (int p = 0; p < PH_COUNT; p++) {
        PhaseGeom& g = P.ph[p];
        g.K = K[p];
        g.nsteps = (int)layout::num_steps(D.fmt, K[p]);
        g.nmat = p == PH_FF1 && D.arch == ARCH_LLAMA ? 2 : 1;
        g.rows = rows[p];
        g.base = items[p] / pl.grid;
        g.rem = items[p] % pl.grid;
        dig = std::max(dig, gemv_dig_region(D.fmt, K[p]));
        if (g.base + (g.rem ? 1 : 0) > MAX_TILES) return false;
        red = std::max(red, ((g.base + (g.rem ? 1 : 0)) * g.nmat + WARPS) * 16);
        inv = std::max(inv, (K[p] + 1023) / 1024 * 4);
    }
    dig = std::max(dig, (ZERO_BYTES + (size_t)WARPS * 2 * (hs + 2) * 4 + 127) & ~(size_t)127);  // attention_phase's sums of the warps
    const int qkv_rows = 16 * (P.ph[PH_QKV].base + (P.ph[PH_QKV].rem ? 1 : 0));
    const size_t fixed = dig + 4 * (size_t)(red + inv) + 256 + 16 * WARPS * PH_COUNT + 4 * MAX_TILES + 16 * (size_t)qkv_rows + 128;
    const size_t stride = ((size_t)chunk_of(D.fmt) * step_b + 8 + 127) & ~(size_t)127;
    P.nstage = fixed >= SMEM_LIMIT ? 0 : (int)std::min((SMEM_LIMIT - fixed) / (WARPS * stride), (size_t)MAX_STAGES);
    if (P.nstage < 2) return false;
    P.dig_region = (int)dig;
    P.red_floats = red;
    P.inv_floats = inv;
    P.qkv_rows = qkv_rows;
    pl.smem = fixed + (size_t)P.nstage * WARPS * stride;

    P.hs = hs;
    P.hs_magic = (unsigned int)(((1ull << 32) + hs - 1) / hs);
    P.lanes_log = 0;
    while ((16 << P.lanes_log) < hs * esz) P.lanes_log++;
    P.head_elems = (long long)D.seq_len * hs;
    P.sqrt_hs = sqrtf((float)hs);
    P.max_splits = std::max(1, std::min({MAX_SPLITS, pl.grid / P.n_items, MAX_PART / D.q_dim}));
    return true;
}
}  // namespace

bool decode_layers_supported(slai_ctx* ctx, const DecodeLayers& D) {
    static thread_local LayersParams P;  // (some 20 KB: not on the caller's stack)
    Plan pl;
    return plan(ctx, D, false, P, pl);  // (one cluster is only ever taken instead)
}

int decode_layers_cluster_positions(const DecodeLayers& D) {
    const long long left = CLUSTER_BYTES - weight_bytes(D), row = 2ll * D.kv_dim * (D.kv_f16 ? 2 : 4);  // keys and values of a position
    return left <= 0 || 2 * left / row >= D.seq_len ? INT_MAX : (int)(2 * left / row);
}

size_t decode_layers_scratch_bytes(const DecodeLayers& D) {
    return 256 + (size_t)std::max(MAX_PART, D.q_dim) * 4 + (size_t)MAX_SPLITS * D.n_heads * 8;
}

unsigned int* decode_layers_counter(void* scratch) { return reinterpret_cast<unsigned int*>(scratch); }

static int launch(slai_ctx* ctx, const DecodeLayers& D, const DecodeLayerPtrs* layers, void* scratch, bool cluster) {
    static thread_local LayersParams P;
    P = LayersParams{};
    Plan pl;
    if (!plan(ctx, D, cluster, P, pl)) {
        if (cluster) return DECODE_LAYERS_NO_FIT;  // (a few tall matrices: more rows than 16 blocks' epilogues take)
        return slai_set_error(ctx, SLAI_ERR_SHAPE, "decode: these layers do not fit one launch");
    }
    P.n_layers = D.n_layers;
    P.eps = D.eps;
    P.x = D.x; P.q = D.q; P.xb = D.xb; P.hb = D.hb;
    P.rope_cs = D.rope_cs;
    P.d_pos = D.d_pos;
    P.kcache = reinterpret_cast<unsigned char*>(D.kcache);
    P.vcache = reinterpret_cast<unsigned char*>(D.vcache);
    P.layer_bytes = (long long)D.layer_bytes;
    unsigned char* s = reinterpret_cast<unsigned char*>(scratch);
    P.bar = decode_layers_counter(scratch);
    P.part_ml = reinterpret_cast<float*>(s + 256);
    P.part_o = reinterpret_cast<float*>(s + 256 + (size_t)MAX_SPLITS * D.n_heads * 8);
    P.err_flag = ctx->d_counters + CNT_ERR_FLAG;
    P.wait_limit = ctx->wait_limit;
#ifdef SLAI_TRACE
    P.tl = ctx->tl;
#endif
    for (int l = 0; l < D.n_layers; l++) {
        for (int i = 0; i < 7; i++) {
            P.layer[l].w[i] = layers[l].w[i];
            SLAI_REQUIRE(ctx, ((uintptr_t)layers[l].w[i] & 15) == 0, SLAI_ERR_INVALID_ARG, "decode: matrix data must be 16-byte aligned");
        }
        for (int i = 0; i < 2; i++) {
            P.layer[l].norm_w[i] = layers[l].norm_w[i];
            P.layer[l].norm_b[i] = layers[l].norm_b[i];
        }
        for (int i = 0; i < 6; i++) P.layer[l].bias[i] = layers[l].bias[i];
    }
    switch (D.fmt) {
        case SLAI_FMT_Q4_K: return decode_layers_launch_q4k(ctx, P, D.arch, D.kv_f16, pl.grid, pl.smem);
        case SLAI_FMT_Q5_K: return decode_layers_launch_q5k(ctx, P, D.arch, D.kv_f16, pl.grid, pl.smem);
        case SLAI_FMT_Q6_K: return decode_layers_launch_q6k(ctx, P, D.arch, D.kv_f16, pl.grid, pl.smem);
        case SLAI_FMT_Q8_0: return decode_layers_launch_q80(ctx, P, D.arch, D.kv_f16, pl.grid, pl.smem);
    }
    return slai_set_error(ctx, SLAI_ERR_UNSUPPORTED_FORMAT, "decode: format %d has no kernel", D.fmt);
}

int decode_layers_launch(slai_ctx* ctx, const DecodeLayers& D, const DecodeLayerPtrs* layers, void* scratch) {
    const int rc = launch(ctx, D, layers, scratch, true);
    return rc == DECODE_LAYERS_NO_FIT ? launch(ctx, D, layers, scratch, false) : rc;
}
