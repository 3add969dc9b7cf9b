// One pass over a quantised matrix for a batch of 2..8 input vectors (GemvQuant::launch with a matrix-shaped `v`,
// crates/slai/src/ops/gemv_quant.rs:206-312: the reference's shader loops over the columns inside one dispatch).
//
// The single-vector kernel (gemv.cu) spends the eight columns of the integer MMA on one vector (four digit planes x two
// sub-blocks); looping it over a batch streams the matrix once per vector.  Here the packed weights of a tile-step block
// are loaded and unpacked into MMA operands once and every pair of vectors adds its own MMAs (`compute_pairs`,
// gemv_formats.cuh; Q6_K, whose sub-blocks of 16 fill half an MMA's depth, one vector at a time): the same integer sums as
// the single-vector code.
//
// Shape, three launches (dependent launches: each one's start overlaps its predecessor's end):
//   digits   every vector's 256-element (Q8_0: 128) steps are turned once into digit planes, digit sums and a power-of-two
//            scale of their own, records of `BatchGeom::REC` bytes per (step, vector); with an RmsNorm in front when asked.
//            (Staged by every block of the product instead, this was half of its time: 16 row groups redid the same chunk.)
//   product  the digit planes of 8 vectors over the whole of K do not fit in shared memory, so K is cut into chunks of `ch`
//            steps and a unit of work is (chunk, group of 16 row tiles).  A block keeps the records of its current and its next
//            unit (one bulk copy each); each of its 16 warps walks its own tile's blocks through a ring of three stages
//            that runs on across units and starts before the predecessor has finished (weights do not depend on it).
//   reduce   adds the chunks' partial sums in order (deterministic; no atomics) and stores.
#include <stdlib.h>

#include "common.cuh"
#include "gemv_formats.cuh"
#include "layout.cuh"

namespace {

using namespace gemvfmt;
using namespace frag;

constexpr int BWARPS = 16;
constexpr int BTHREADS = 32 * BWARPS;
constexpr int MAX_CH = 8;
constexpr int BSTAGES = 3;  // weight blocks a warp has in flight
constexpr int BSMEM_LIMIT = 227 * 1024 - 256;  // the barriers are static

struct BatchParams {
    const uint8_t* w[3];   // up to three matrices of the same format and K that share the input (q / k / v, gate / up): their
    int t0[3];             // 16-row tiles form one tile space, matrix i starts at tile t0[i]
    int nw;
    long long tile_bytes;
    int ntiles, nsteps, K;
    int ch, nch, ngroups;  // steps per chunk, chunks, groups of 16 tiles
    int n_batch;           // vectors that exist (the others of the instantiation's NV are zero)
    const float* v;        // [n_batch][K]
    const float* norm_w;   // optional RmsNorm of the vectors
    float eps;
    unsigned char* rec;    // [nsteps][NV][REC] digit records
    float* part;           // [nch][NV][mp] partial sums
    int mp;                // ntiles * 16
    unsigned int* err_flag;
    unsigned int wait_limit;
};

template <class F>
struct BatchGeom {
    static constexpr uint32_t STEP = F::STEP_BYTES;
    static constexpr uint32_t STRIDE = (STEP + 127) & ~127u;
    static constexpr uint32_t PLANE = F::STEP + 32;  // planes 32 bytes apart modulo 128: the four digit columns hit different banks
    static constexpr uint32_t SUMS = 4 * PLANE;      // byte table of the digit sums (Q4_K / Q5_K)
    static constexpr uint32_t REC = SUMS + (F::PAIRED && F::SV_GRAN == 32 ? 128 : 0);
    static constexpr uint32_t INV = F::STEP;         // 1 / scale, in the gap after the first plane
};

__device__ __forceinline__ float bmax4(const float4& x) { return fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(x.z), fabsf(x.w))); }

// One warp per (vector, step); block (x, y): vector y, steps x * 16 + warp, onwards by the grid's width.  With a norm one
// block serves the whole vector.
template <class F>
__global__ void __launch_bounds__(BTHREADS) batch_digits_kernel(const __grid_constant__ BatchParams P, int nv) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    using G = BatchGeom<F>;
    constexpr int PER = F::STEP / 128;  // float4 per lane
    const int v = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool have = v < P.n_batch;
    const float* x = P.v + (size_t)(have ? v : 0) * P.K;
    float mul = 1.f;
    if (P.norm_w && have) {  // ops/rms_norm.rs:68-77
        __shared__ float sh[BWARPS];
        float s = 0.f;
        for (int i = threadIdx.x; i < P.K / 4; i += BTHREADS) {
            const float4 q = __ldcg(reinterpret_cast<const float4*>(x) + i);
            s += q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) sh[warp] = s;
        __syncthreads();
        s = 0.f;
        for (int w = 0; w < BWARPS; w++) s += sh[w];
        mul = 1.0f / sqrtf(s / (float)P.K + P.eps);
    }
    for (int step = blockIdx.x * BWARPS + warp; step < P.nsteps; step += gridDim.x * BWARPS) {
        float4 q[PER];
        float mx = 0.f;
#pragma unroll
        for (int e = 0; e < PER; e++) {
            const int k = step * F::STEP + (PER * lane + e) * 4;
            q[e] = have && k < P.K ? __ldcg(reinterpret_cast<const float4*>(x + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
            if (P.norm_w && have && k < P.K) {
                const float4 w = __ldg(reinterpret_cast<const float4*>(P.norm_w + k));
                q[e].x = (q[e].x * mul) * w.x; q[e].y = (q[e].y * mul) * w.y; q[e].z = (q[e].z * mul) * w.z; q[e].w = (q[e].w * mul) * w.w;
            }
            mx = fmaxf(mx, bmax4(q[e]));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        float scale = 1.f;
        if (mx > 0.f && mx < 3.0e38f) {
            int e = (int)((__float_as_uint(mx) >> 23) & 0xffu) - 126;  // mx = f * 2^e with f in [0.5, 1) (normal numbers)
            if ((__float_as_uint(mx) >> 23) == 0u) e = -126;
            e = e < -90 ? -90 : e;
            scale = __uint_as_float((uint32_t)(127 + 26 - e) << 23);  // 2^(26 - e), exact
        }
        unsigned char* rec = P.rec + ((size_t)step * nv + v) * G::REC;
        uint32_t pw[PER][4];
#pragma unroll
        for (int e = 0; e < PER; e++)
            digit_planes(digits_word(__float2int_rn(q[e].x * scale)), digits_word(__float2int_rn(q[e].y * scale)), digits_word(__float2int_rn(q[e].z * scale)),
                         digits_word(__float2int_rn(q[e].w * scale)), pw[e]);
#pragma unroll
        for (int p = 0; p < 4; p++)
#pragma unroll
            for (int e = 0; e < PER; e++) *reinterpret_cast<uint32_t*>(rec + p * G::PLANE + (PER * lane + e) * 4) = pw[e][p];
        if (lane == 0) *reinterpret_cast<float*>(rec + G::INV) = 1.0f / scale;
        if (F::PAIRED && F::SV_GRAN == 32) {
            // Q4_K / Q5_K: sum of a sub-block's digits (four lanes of eight elements) per plane, as two base-128 digits in the byte
            // table of the step: row 2p the high, row 2p + 1 the low digit of plane p, byte j of a row = sub-block j, bytes 8..15 zero
            const int j = lane >> 2;
#pragma unroll
            for (int p = 0; p < 4; p++) {
                int sd = 0;
#pragma unroll
                for (int e = 0; e < PER; e++) sd = __dp4a((int)pw[e][p], 0x01010101, sd);
                sd += __shfl_xor_sync(0xffffffffu, sd, 1);
                sd += __shfl_xor_sync(0xffffffffu, sd, 2);
                const int hi = (sd + 64) >> 7, lo = sd - (hi << 7);
                if ((lane & 3) == 0) {
                    rec[G::SUMS + (2 * p) * 16 + j] = (unsigned char)hi;
                    rec[G::SUMS + (2 * p + 1) * 16 + j] = (unsigned char)lo;
                }
            }
            if (lane < 8) *reinterpret_cast<uint2*>(rec + G::SUMS + lane * 16 + 8) = make_uint2(0u, 0u);
        }
    }
}

// One tile-step block, global -> this warp's stage: 16 bytes per lane and round.
template <class F>
__device__ __forceinline__ void stage_request(const uint8_t* src, uint32_t dst, int lane) {
    const size_t gsrc = __cvta_generic_to_global(src);
#pragma unroll
    for (uint32_t r = 0; r < BatchGeom<F>::STEP; r += 512u) {
        const uint32_t off = r + 16u * lane;
        if (off < BatchGeom<F>::STEP) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + off), "l"(gsrc + off) : "memory");
    }
}
__device__ __forceinline__ void stage_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// A warp's walk over its blocks: unit by unit, `nst` steps of one tile each.
struct BatchWalk {
    int unit, step, nst;
    const uint8_t* src;  // the unit's first block of this warp's tile (null: the group has no tile for this warp)
};
template <class F>
__device__ __forceinline__ void walk_open(BatchWalk& W, const BatchParams& P, int warp) {
    W.step = 0;
    W.nst = 0;
    if (W.unit >= P.ngroups * P.nch) return;
    const int c = W.unit / P.ngroups, tile = (W.unit - c * P.ngroups) * BWARPS + warp;
    W.nst = min(P.ch, P.nsteps - c * P.ch);
    const uint8_t* base = P.w[0];
    int t0 = 0;
    if (P.nw > 1 && tile >= P.t0[1]) { base = P.w[1]; t0 = P.t0[1]; }
    if (P.nw > 2 && tile >= P.t0[2]) { base = P.w[2]; t0 = P.t0[2]; }
    W.src = tile < P.ntiles ? base + (size_t)(tile - t0) * P.tile_bytes + (size_t)c * P.ch * BatchGeom<F>::STEP : nullptr;
}

template <class F, int NV>
__global__ void __launch_bounds__(BTHREADS, 1) gemv_batch_kernel(const __grid_constant__ BatchParams P) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) unsigned long long bars[2];
    using G = BatchGeom<F>;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem), bar = (uint32_t)__cvta_generic_to_shared(bars);
    const uint32_t slot_bytes = (uint32_t)P.ch * NV * G::REC;
    const uint32_t wb = sbase + ZERO_BYTES + 2 * slot_bytes + (uint32_t)warp * BSTAGES * G::STRIDE;
    const int units = P.ngroups * P.nch, stride = (int)gridDim.x;

    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (tid < ZERO_BYTES / 4) reinterpret_cast<uint32_t*>(smem)[tid] = 0u;
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar + 8) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    BatchWalk W;  // the request cursor, BSTAGES - 1 blocks ahead
    W.unit = (int)blockIdx.x;
    walk_open<F>(W, P, warp);
    auto request = [&](int stage) {
        if (W.nst > 0) {
            if (W.src) stage_request<F>(W.src + (size_t)W.step * G::STEP, wb + (uint32_t)stage * G::STRIDE, lane);
            if (++W.step == W.nst) {
                W.unit += stride;
                walk_open<F>(W, P, warp);
            }
        }
        stage_commit();
    };
#pragma unroll
    for (int s = 0; s < BSTAGES - 1; s++) request(s);

    asm volatile("griddepcontrol.wait;" ::: "memory");
    __syncthreads();
    auto fetch_records = [&](int unit, int slot) {  // one thread; the slot has been read by everyone
        const int c = unit / P.ngroups;
        const uint32_t bytes = (uint32_t)min(P.ch, P.nsteps - c * P.ch) * NV * G::REC, b = bar + 8 * slot;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(bytes) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(sbase + ZERO_BYTES + slot * slot_bytes),
                     "l"(__cvta_generic_to_global(P.rec + (size_t)c * P.ch * NV * G::REC)), "r"(bytes), "r"(b)
                     : "memory");
    };
    if (tid == 0) {
        fetch_records((int)blockIdx.x, 0);
        if ((int)blockIdx.x + stride < units) fetch_records((int)blockIdx.x + stride, 1);
    }

    Smem S;
    S.zero = sbase;
    S.plane = G::PLANE;
    LaneCtx L;
    unsigned int limit = P.wait_limit;
    int stage = 0, it = 0;
    for (int unit = (int)blockIdx.x; unit < units; unit += stride, it++) {
        const int c = unit / P.ngroups, grp = unit - c * P.ngroups, slot = it & 1;
        const int nst = min(P.ch, P.nsteps - c * P.ch), tile = grp * BWARPS + warp;
        bounded_wait<false, false, 6>(bar + 8 * slot, (uint32_t)(it >> 1) & 1u, limit, P.err_flag);  // the unit's records
        S.dig = sbase + ZERO_BYTES + slot * slot_bytes;
        // ---- this warp's tile: `nst` blocks against all vectors ----
        constexpr int NA = F::PAIRED ? NV / 2 : NV;
        float accA[NA], accB[NA];
#pragma unroll
        for (int v = 0; v < NA; v++) accA[v] = accB[v] = 0.f;
#pragma unroll 1
        for (int s = 0; s < nst; s++) {
            request(stage == 0 ? BSTAGES - 1 : stage - 1);  // into the stage consumed one block ago
            asm volatile("cp.async.wait_group %0;" ::"n"(BSTAGES - 1) : "memory");  // all but the newest requests have landed: this block is here
            __syncwarp();
            S.sv = S.dig + G::SUMS;
            lane_init<F>(L, lane, S);
            const uint32_t blk = wb + (uint32_t)stage * G::STRIDE;
            float a[NA], b[NA];
#pragma unroll
            for (int v = 0; v < NA; v++) a[v] = b[v] = 0.f;
            if constexpr (F::PAIRED) F::template compute_pairs<NV>(blk, 0, L, S, G::REC, a, b);
            else F::template compute_batch<NV>(blk, 0, L, S, L.bmul ? G::REC : 0u, G::REC, a, b);
#pragma unroll
            for (int v = 0; v < NA; v++) {  // every step has its own scale
                const float inv = __uint_as_float(prim::lds32(S.dig + (F::PAIRED ? 2 * v + (L.t >> 1) : v) * G::REC + G::INV));
                accA[v] = fmaf(inv, a[v], accA[v]);
                accB[v] = fmaf(inv, b[v], accB[v]);
            }
            S.dig += NV * G::REC;
            __syncwarp();
            if (++stage == BSTAGES) stage = 0;
        }
#pragma unroll
        for (int v = 0; v < NA; v++) {
            accA[v] += __shfl_xor_sync(0xffffffffu, accA[v], 1);
            accB[v] += __shfl_xor_sync(0xffffffffu, accB[v], 1);
            if (!F::PAIRED) {
                accA[v] += __shfl_xor_sync(0xffffffffu, accA[v], 2);
                accB[v] += __shfl_xor_sync(0xffffffffu, accB[v], 2);
            }
        }
        if (tile < P.ntiles) {
            float* dst = P.part + (size_t)c * NV * P.mp + (size_t)tile * 16;
#pragma unroll
            for (int v = 0; v < NA; v++) {
                if (F::PAIRED) {  // lanes t and t ^ 1 hold vector 2v + (t >> 1): the even one stores row g, the odd one row g + 8
                    dst[(size_t)(2 * v + (L.t >> 1)) * P.mp + L.g + 8 * (L.t & 1)] = (L.t & 1) ? accB[v] : accA[v];
                } else if ((v & 3) == L.t) {  // the four lanes of a row hold the same sums: lane t stores vectors t and t + 4
                    dst[(size_t)v * P.mp + L.g] = accA[v];
                    dst[(size_t)v * P.mp + L.g + 8] = accB[v];
                }
            }
        }
        __syncthreads();  // the unit's records have been read
        if (tid == 0 && limit && unit + 2 * stride < units) fetch_records(unit + 2 * stride, slot);  // (given up: what was requested has had its time to land)
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Sum of n values `stride` apart, in order; U loads in flight.
template <int U>
__device__ __forceinline__ float batch_sum(const float* p, int n, size_t stride) {
    float s = 0.f;
    for (int c0 = 0; c0 < n; c0 += U) {
        float x[U];
#pragma unroll
        for (int i = 0; i < U; i++) x[i] = c0 + i < n ? __ldcg(p + (size_t)(c0 + i) * stride) : 0.f;
#pragma unroll
        for (int i = 0; i < U; i++) s += x[i];
    }
    return s;
}

// out[v][m] = sum over the chunks, in order, of the partial sums.
// epi: BATCH_STORE, BATCH_ADD (out += sum: the residual streams of the batch), BATCH_SILU (out = sum * silu(gate), gate laid
// out like out: ops/silu.rs:50-58 with the sum as h2 and gate as h1), BATCH_PAIR_SILU (two matrices of M rows each in one
// launch, gate then up: out = up sum * silu(gate sum)).
template <int U>
__global__ void gemv_batch_reduce_kernel(float* out, long long ldo, const float* part, int nch, int nv, int mp, int M, int n_batch, int epi,
                                         const float* gate) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)n_batch * M) return;
    const int v = (int)(idx / M), m = (int)(idx - (long long)v * M);
    float s = batch_sum<U>(part + (size_t)v * mp + m, nch, (size_t)nv * mp);
    const long long o = (long long)v * ldo + m;
    if (epi == BATCH_ADD) {
        s = out[o] + s;
    } else if (epi == BATCH_SILU) {
        const float g = gate[o];
        s = s * (g / (1.0f + expf(-g)));
    } else if (epi == BATCH_PAIR_SILU) {
        const float u = batch_sum<U>(part + (size_t)v * mp + M + m, nch, (size_t)nv * mp);
        s = u * (s / (1.0f + expf(-s)));
    }
    out[o] = s;
}

template <class F>
size_t batch_smem(int nv, int ch) {
    return ZERO_BYTES + 2 * (size_t)ch * nv * BatchGeom<F>::REC + (size_t)BWARPS * BSTAGES * BatchGeom<F>::STRIDE;
}

template <class F, int NV>
int launch_batch_inst(slai_ctx* ctx, BatchParams& P, float* d_out, long long ldo, int M, int epi, const float* gate, bool pdl) {
    // Steps per chunk: the fewest rounds of (start of a unit + ch steps) over the SMs; a unit's start costs about one step.
    const int G = ctx->sm_count > 0 ? ctx->sm_count : 148;
    int best_ch = 1;
    long long best_cost = -1;
    for (int ch = 1; ch <= MAX_CH && batch_smem<F>(NV, ch) <= (size_t)BSMEM_LIMIT; ch++) {
        const long long nch = (P.nsteps + ch - 1) / ch;
        const long long rounds = (nch * P.ngroups + G - 1) / G;
        const long long cost = rounds * (1 + ch);
        if (best_cost < 0 || cost <= best_cost) {
            best_cost = cost;
            best_ch = ch;
        }
    }
    P.ch = best_ch;
    P.nch = (P.nsteps + P.ch - 1) / P.ch;
    const size_t smem = batch_smem<F>(NV, P.ch);
    SLAI_REQUIRE(ctx, smem <= (size_t)BSMEM_LIMIT, SLAI_ERR_SHAPE, "gemv: the batched kernel needs %zu bytes of shared memory", smem);
    const size_t rec_bytes = ((size_t)P.nsteps * NV * BatchGeom<F>::REC + 255) & ~(size_t)255;
    int rc = ensure_scratch(ctx, rec_bytes + (size_t)P.nch * NV * P.mp * sizeof(float));
    if (rc) return rc;
    P.rec = reinterpret_cast<unsigned char*>(ctx->d_scratch);
    P.part = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(ctx->d_scratch) + rec_bytes);
    auto kern = gemv_batch_kernel<F, NV>;
    static PerDeviceOnce attr;  // per instantiation
    if (attr.need(ctx->device)) {
        SLAI_CHECK_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, BSMEM_LIMIT));
        attr.set(ctx->device);
    }
    const int dblocks = P.norm_w ? 1 : (P.nsteps + BWARPS - 1) / BWARPS;
    if ((rc = launch_dependent(ctx, batch_digits_kernel<F>, dim3((unsigned)dblocks, NV), BTHREADS, 0, pdl, P, NV))) return rc;
    const long long units = (long long)P.ngroups * P.nch;
    if ((rc = launch_dependent(ctx, kern, dim3((unsigned)(units < G ? units : G)), BTHREADS, smem, ctx->use_pdl, P))) return rc;
    const long long total = (long long)P.n_batch * M;
    // More than eight chunks: 32 loads in flight.  Eight at a time, the 32 chunks of a short wide matrix were four trips to memory one
    // after the other: Q8_0 1000 x 4096, 2 vectors 12.0 -> 8.3 us, 8 vectors 13.5 -> 8.4; Q5_K 4096 x 11008, 8 vectors 21.9 -> 20.3.
    // (Summed by the last block of a row group inside the product instead, one launch less, 32000 x 4096 Q4_K with 8 vectors took
    // 43.8 us for 35.6, and 2048 x 2048 10.6 for 8.6: every unit pays the fence and the ticket.)
    auto reduce = P.nch <= 8 ? gemv_batch_reduce_kernel<8> : gemv_batch_reduce_kernel<32>;
    return launch_dependent(ctx, reduce, dim3((unsigned)((total + 255) / 256)), 256, 0, ctx->use_pdl, d_out, ldo, P.part, P.nch, NV, P.mp, M,
                            P.n_batch, epi, gate);
}

template <class F>
int launch_batch_fmt(slai_ctx* ctx, BatchParams& P, float* d_out, long long ldo, int M, int epi, const float* gate, bool pdl) {
    if (P.n_batch <= 2) return launch_batch_inst<F, 2>(ctx, P, d_out, ldo, M, epi, gate, pdl);
    if (P.n_batch <= 4) return launch_batch_inst<F, 4>(ctx, P, d_out, ldo, M, epi, gate, pdl);
    if (P.n_batch <= 6) return launch_batch_inst<F, 6>(ctx, P, d_out, ldo, M, epi, gate, pdl);
    return launch_batch_inst<F, 8>(ctx, P, d_out, ldo, M, epi, gate, pdl);
}

}  // namespace

bool gemv_batch_supported(const slai_qmatrix* w) {
    return w->fmt == SLAI_FMT_Q8_0 || w->fmt == SLAI_FMT_Q4_K || w->fmt == SLAI_FMT_Q5_K || w->fmt == SLAI_FMT_Q6_K;
}

// out[b * ldo + m] = sum_k W[m][k] v[b][k] for b < n_batch (2..8), one pass over W (ldo 0: the rows of `out` are M apart);
// `d_norm_w` puts an RmsNorm of the vectors in front; `pdl`: the first launch may begin before its predecessor in the stream has
// ended (it waits for it itself); `epi` folds a residual add or the SiLU gate into the store.  W is the concatenation by rows of `nw` (1..3) matrices of the
// same format and width (all but the last with a multiple of 16 rows); with BATCH_PAIR_SILU the two matrices are gate and up
// of equal height M and out[b * ldo + m], m < M, receives up * silu(gate).
int gemv_batch_launch_multi(slai_ctx* ctx, float* d_out, const slai_qmatrix* const* ws, int nw, const float* d_v, int n_batch, long long ldo,
                            int epi, const float* d_gate, const float* d_norm_w, float eps, bool pdl) {
    SLAI_REQUIRE(ctx, nw >= 1 && nw <= 3 && ws && ws[0], SLAI_ERR_INVALID_ARG, "gemv: %d matrices in one batched launch", nw);
    const slai_qmatrix* w = ws[0];
    SLAI_REQUIRE(ctx, gemv_batch_supported(w), SLAI_ERR_UNSUPPORTED_FORMAT, "gemv: format %d has no batched kernel", w->fmt);
    SLAI_REQUIRE(ctx, n_batch >= 2 && n_batch <= 8, SLAI_ERR_INVALID_ARG, "gemv: batch of %d", n_batch);
    SLAI_REQUIRE(ctx, (reinterpret_cast<uintptr_t>(d_v) & 15) == 0, SLAI_ERR_INVALID_ARG, "gemv: the input vectors must be 16-byte aligned");
    BatchParams P = {};
    int rows_total = 0, tiles = 0;
    for (int i = 0; i < nw; i++) {
        SLAI_REQUIRE(ctx, ws[i] && ws[i]->fmt == w->fmt && ws[i]->ncols == w->ncols && ws[i]->tile_bytes == w->tile_bytes, SLAI_ERR_SHAPE,
                     "gemv: matrices of one batched launch must share format and width");
        SLAI_REQUIRE(ctx, i == nw - 1 || ws[i]->nrows % 16 == 0, SLAI_ERR_SHAPE, "gemv: %lld rows before another matrix of the launch",
                     (long long)ws[i]->nrows);
        SLAI_REQUIRE(ctx, (reinterpret_cast<uintptr_t>(ws[i]->data) & 15) == 0 && ws[i]->tile_bytes % 16 == 0, SLAI_ERR_INVALID_ARG,
                     "gemv: matrix data must be 16-byte aligned");
        P.w[i] = ws[i]->data;
        P.t0[i] = tiles;
        tiles += (int)layout::num_tiles(ws[i]->nrows);
        rows_total += (int)ws[i]->nrows;
    }
    P.nw = nw;
    P.tile_bytes = w->tile_bytes;
    P.ntiles = tiles;
    P.nsteps = (int)layout::num_steps(w->fmt, w->ncols);
    P.K = (int)w->ncols;
    P.ngroups = (P.ntiles + BWARPS - 1) / BWARPS;
    P.n_batch = n_batch;
    P.v = d_v;
    P.norm_w = d_norm_w;
    P.eps = eps;
    P.err_flag = ctx->d_counters + CNT_ERR_FLAG;
    P.wait_limit = ctx->wait_limit;
    P.mp = P.ntiles * 16;
    int M = rows_total;
    if (epi == BATCH_PAIR_SILU) {
        SLAI_REQUIRE(ctx, nw == 2 && ws[0]->nrows == ws[1]->nrows, SLAI_ERR_SHAPE, "gemv: the gate / up epilogue takes two matrices of equal height");
        M = (int)ws[0]->nrows;
    }
    if (ldo <= 0) ldo = M;
    SLAI_REQUIRE(ctx, ldo >= M, SLAI_ERR_SHAPE, "gemv: output rows %lld apart hold fewer than %d values", ldo, M);
    SLAI_REQUIRE(ctx, epi == BATCH_STORE || epi == BATCH_ADD || epi == BATCH_PAIR_SILU || (epi == BATCH_SILU && d_gate), SLAI_ERR_INVALID_ARG,
                 "gemv: batch epilogue %d", epi);
    switch (w->fmt) {
        case SLAI_FMT_Q8_0: return launch_batch_fmt<Q80>(ctx, P, d_out, ldo, M, epi, d_gate, pdl);
        case SLAI_FMT_Q4_K: return launch_batch_fmt<Q4K>(ctx, P, d_out, ldo, M, epi, d_gate, pdl);
        case SLAI_FMT_Q5_K: return launch_batch_fmt<Q5K>(ctx, P, d_out, ldo, M, epi, d_gate, pdl);
        case SLAI_FMT_Q6_K: return launch_batch_fmt<Q6K>(ctx, P, d_out, ldo, M, epi, d_gate, pdl);
    }
    return SLAI_ERR_UNSUPPORTED_FORMAT;
}

int gemv_batch_launch(slai_ctx* ctx, float* d_out, const slai_qmatrix* w, const float* d_v, int n_batch, long long ldo, int epi,
                      const float* d_gate, const float* d_norm_w, float eps, bool pdl) {
    return gemv_batch_launch_multi(ctx, d_out, &w, 1, d_v, n_batch, ldo, epi, d_gate, d_norm_w, eps, pdl);
}
