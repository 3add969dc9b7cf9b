// All layers of a decode step in one cooperative launch (one block of 16 warps per SM), device side.
//
// What bounds it.  The step's weights are read once, 117 MB a layer for the 7B shape: 17.7 us of HBM time.  Launched kernel by kernel
// (gemv.cu, attention.cu) a layer takes 48 us: between two products nothing is read, and from the end of one launch to the first digit of the next product's
// input it is 3.1 us, five times a layer.  Here the launches are phases of one kernel with a grid-wide barrier between them (1.2 us and 0.5
// for the load of the input behind it), and the rings of weight blocks run on across the barriers.  What is left of the 43 us a layer now takes are chains of latencies: four
// warps a scheduler issue one of their instructions every 8 cycles, so what counts is the number of instructions between two barriers, and
// the size of the code (all of it is run once a layer; 137 KB of it took 24 % longer than 60 KB).
// us a token, kernel by kernel (whose vectors are staged the same way by now) / here: Llama-2 7B Q4_K at position 515 1484 / 1458, with an f32 cache 1471 / 1500; 8
// layers of the 70B shape at 3500 1239 / 1136; GPT-2 XL 1476 / 1353; the tiny story model 107.5 / 110.8: what is left is the gain of LayerNorm models and of
// grouped queries.  All SMs are taken at once: two contexts that decode at the same time take turns (8 layers 1024 wide: 5381 tokens/s together, kernel by kernel
// 8032; 512 wide 6790 and 10582; 4096 wide 2989 and 3590), and a step waits for other streams' kernels (SLAI_SEPARATE_LAYERS).
//
// A layer is five phases, as many as the separate path has launches:
//   q/k/v    norm of x, product, RoPE, q to its buffer, k and v to the cache (PH_QKV)
//   attention  (head, split of the positions) items, one block each; rows that are already in the cache are loaded before the
//            barrier, the newest one and the queries after it
//   o        x += W (merge of the splits), the merge done by every block while it stages the vector (PH_O)
//   ff1      norm of x, gate and up with SiLU, or one matrix with GELU (PH_FF1)
//   ff2      x += W h (PH_FF2)
// The products are those of gemv_kernel.cuh: the same tiles, digit planes, per-warp rings, and integer sums.  A warp's piece of a phase is a
// contiguous run of the block's (tile, matrix, step) units; the partial sums of run (tile-matrix j, warp w) go to slot j + w, which no other
// run of the phase has (the runs are ordered, each next one is a tile or a warp further).
//
// Every wait on memory is bounded (bounded_wait, grid_barrier; the hardware's barrier of a cluster has no limit to give, and every block arrives on it as often
// as the others): the error flag is raised and the step goes on.  A warp that has given up on its ring requests nothing more, and waits for its copies in
// flight before the block ends.
#pragma once
#include "decode_layers.h"
#include "gemv_kernel.cuh"

namespace declayers {

using namespace gemvk;

enum Phase { PH_QKV = 0, PH_O = 1, PH_FF1 = 2, PH_FF2 = 3, PH_COUNT = 4 };
enum Arch { ARCH_LLAMA = 0, ARCH_GPT2 = 1 };
constexpr int MAX_LAYERS = 128;
constexpr int MAX_SPLITS = 16;
constexpr int MAX_TILES = THREADS / 16;  // row tiles of a block in a phase: its rows are the epilogue's threads

struct LayerPtrs {
    const uint8_t* w[7];     // q, k, v, o, gate (or the only matrix), up, down
    const float* norm_w[2];  // in front of q/k/v, of the feed-forward part
    const float* norm_b[2];
    const float* bias[6];    // q, k, v, o, feed-forward in, feed-forward out (null: none)
};
struct PhaseGeom {
    int K, nsteps, nmat;
    int base, rem;  // 16-row tiles per block: base each, one more for the first `rem`
    int rows;       // rows of a matrix of the phase (PH_QKV: unused)
};
struct LayersParams {
    PhaseGeom ph[PH_COUNT];
    int tile_k, tile_v;      // first tile of k and of v in the q/k/v tile space
    int q_rows, kv_rows;
    int n_layers, nstage, dig_region, red_floats, inv_floats, qkv_rows;
    float eps;
    float *x, *q, *xb, *hb;
    const float* rope_cs;    // (cos, sin) pairs of the position (null: no rotation)
    const int* d_pos;
    unsigned char *kcache, *vcache;
    long long layer_bytes;   // cache bytes of a layer
    long long head_elems;    // elements between cache heads (positions are hs apart)
    float sqrt_hs;
    unsigned int hs_magic;   // ceil(2^32 / hs): row / hs of rows below 2^16
    int hs, lanes_log;       // head size; log2 of the lanes that hold a cached row, 16 bytes each
    int n_heads, kvq, kv_share, n_items;  // query heads; query heads an item serves; items per cache head; items per split
    int max_splits;
    float* part_o;           // [split][n_heads * hs]
    float* part_ml;          // [split][n_heads][2]
    unsigned int* bar;       // zero at launch
    int cluster;             // the blocks are one cluster
    unsigned int* err_flag;
    unsigned int wait_limit;
#ifdef SLAI_TRACE
    unsigned long long* tl;
#endif
    LayerPtrs layer[MAX_LAYERS];
};
__device__ __forceinline__ int splits_of(int n, int rows_round, int max_splits) {
    const int want = (n + rows_round - 1) / rows_round;
    return want > max_splits ? max_splits : want;
}
constexpr int ROWS_PER_LANE = 4;  // cached rows a lane group has in flight

// (gemv_kernel.cuh's warp_max starts at magnitudes)
__device__ __forceinline__ float warp_max_signed(float x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
    return x;
}

// A stage of the ring: up to CH blocks of one run and the barrier they complete on.  Two blocks where a block is small (Q8_0: a stage's request,
// wait and turn-over cost as much as half a block's product; GPT-2 XL 1329 -> 1282 us a token); one otherwise (Q4_K, 7B: 1402 against 1427).
constexpr int chunk_of(int fmt) { return fmt == SLAI_FMT_Q8_0 ? 2 : 1; }
template <class F>
struct Stage {
    static constexpr int CH = chunk_of(F::FMT);
    static constexpr uint32_t MBAR = CH * F::STEP_BYTES, STRIDE = (MBAR + 8 + 127) & ~127u;
};

// ---- weight ring across phases ------------------------------------------------------------------------------------------
struct Feed {
    uint32_t base, end, c_addr, c_phase, lane0;
    unsigned int limit;
    unsigned int issued;      // copies requested
    // producer
    int layer, ph, li, mat, left, run;
    const uint8_t* ptr;
    uint32_t table;           // shared address of this warp's pieces: int4 {tile, matrix, step, units} per phase
};
__device__ __forceinline__ int4 piece_of(uint32_t table, int ph) {
    int4 r;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(table + 16 * ph) : "memory");
    return r;
}
// The next run of this warp: the next tile-matrix of its piece, or its piece of the next phase (of this or a later layer) that has one.
template <class F>
__device__ __forceinline__ void feed_advance(Feed& R, const LayersParams& P) {
    int step = 0;
    if (R.left > 0) {
        R.mat ^= P.ph[R.ph].nmat - 1;
        R.li += R.mat ^ 1;
    } else {
        int4 t;
        do {
            if (++R.ph == PH_COUNT) {
                R.ph = 0;
                if (++R.layer >= P.n_layers) return;  // (run stays 0)
            }
            t = piece_of(R.table, R.ph);
        } while (t.w == 0);
        R.li = t.x;
        R.mat = t.y;
        step = t.z;
        R.left = t.w;
    }
    const PhaseGeom& g = P.ph[R.ph];
    const int b = (int)blockIdx.x;
    int tile = b * g.base + min(b, g.rem) + R.li, w = R.ph == PH_FF1 ? 4 + R.mat : R.ph == PH_O ? 3 : 6;
    if (R.ph == PH_QKV) {
        w = tile >= P.tile_v ? 2 : tile >= P.tile_k ? 1 : 0;
        tile -= w == 2 ? P.tile_v : w == 1 ? P.tile_k : 0;
    }
    R.run = min(R.left, g.nsteps - step);
    R.left -= R.run;
    R.ptr = P.layer[R.layer].w[w] + (size_t)(unsigned int)(tile * g.nsteps + step) * F::STEP_BYTES;
}
// Request the next blocks of the warp's sequence (up to Stage<F>::CH of one run) into the stage at `stage`, which this warp has finished reading.
template <class F>
__device__ __forceinline__ void feed_step(Feed& R, const LayersParams& P, uint32_t stage) {
    const int k = min(R.run, Stage<F>::CH);
    const uint32_t bytes = (uint32_t)k * F::STEP_BYTES;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t"
        "@p fence.proxy.async.shared::cta;\n\t"
        "@p mbarrier.arrive.expect_tx.shared::cta.b64 _, [%4], %3;\n\t"
        "@p cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%1], [%2], %3, [%4];\n\t}"
        :
        : "r"(k > 0 ? R.lane0 : 0u), "r"(stage), "l"(R.ptr), "r"(bytes), "r"(stage + Stage<F>::MBAR)
        : "memory");
    if (k > 0) {
        R.ptr += bytes;
        R.issued++;
        R.run -= k;
        if (R.run == 0) feed_advance<F>(R, P);
    }
}

// Elements 4i .. 4i+7 of the attention output (one head's): the splits' sums, weighted; four splits' loads in flight.
__device__ __forceinline__ void merged(const LayersParams& P, int S, int i, float4 (&q)[2]) {
    const int head = (int)__umulhi((unsigned int)(4 * i), P.hs_magic), dim = P.n_heads * P.hs;
    float M = -INFINITY, den = 0.f;
    q[0] = q[1] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int s0 = 0; s0 < S; s0 += 4) {
        float2 ml[4];
        float4 o[4][2];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            ml[u] = make_float2(-INFINITY, 0.f);
            o[u][0] = o[u][1] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (s0 + u < S) {
                ml[u] = __ldcg(reinterpret_cast<const float2*>(P.part_ml) + (s0 + u) * P.n_heads + head);
                const float4* src = reinterpret_cast<const float4*>(P.part_o + (s0 + u) * dim) + i;
                o[u][0] = __ldcg(src);
                o[u][1] = __ldcg(src + 1);
            }
        }
        const float Mn = fmaxf(fmaxf(fmaxf(ml[0].x, ml[1].x), fmaxf(ml[2].x, ml[3].x)), M), base = Mn == -INFINITY ? 0.f : Mn;
        const float a = expf(M - base);
        M = Mn;
        den *= a;
#pragma unroll
        for (int e = 0; e < 2; e++) { q[e].x *= a; q[e].y *= a; q[e].z *= a; q[e].w *= a; }
#pragma unroll
        for (int u = 0; u < 4; u++) {  // (a split without positions: weight 0, sums 0)
            const float b = expf(ml[u].x - base);
            den = fmaf(b, ml[u].y, den);
#pragma unroll
            for (int e = 0; e < 2; e++) {
                q[e].x = fmaf(b, o[u][e].x, q[e].x); q[e].y = fmaf(b, o[u][e].y, q[e].y); q[e].z = fmaf(b, o[u][e].z, q[e].z); q[e].w = fmaf(b, o[u][e].w, q[e].w);
            }
        }
    }
    const float r = 1.0f / den;
#pragma unroll
    for (int e = 0; e < 2; e++) { q[e].x *= r; q[e].y *= r; q[e].z *= r; q[e].w *= r; }
}

// The input of a phase's product for stage_steps: a vector, or the splits' partial outputs of the attention.
struct PhaseInput {
    const LayersParams& P;
    const float4* x4;
    int merge;  // splits to be merged (0, 1: none)
    __device__ __forceinline__ float4 load(int j) const { return merge <= 1 ? __ldcg(x4 + j) : make_float4(0.f, 0.f, 0.f, 0.f); }
    __device__ __forceinline__ void finish(int i, int n4, float4 (&q)[2]) const {
        if (merge > 1 && i < n4) {
            merged(P, merge, i, q);
            if (blockIdx.x == 0) {  // (for slai_llama_read_state: nobody reads it inside the step)
                reinterpret_cast<float4*>(P.xb)[i] = q[0];
                reinterpret_cast<float4*>(P.xb)[i + 1] = q[1];
            }
        }
    }
};

// The oldest stage's blocks are here.  A wait that gives up: nothing more is requested (Feed::run stays 0).
template <class F>
__device__ __forceinline__ void feed_wait(Feed& R, const LayersParams& P) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(R.c_addr + Stage<F>::MBAR), "r"(R.c_phase)
                 : "memory");
    if (!ok && !bounded_wait<false, false, 1>(R.c_addr + Stage<F>::MBAR, R.c_phase, R.limit, P.err_flag)) R.run = 0;
}

// ---- grid barrier ------------------------------------------------------------------------------------------------------------
// Counter in L2, one arrival and one polling thread per block (measured against arrivals per cluster, flags per block, several counters,
// separate lines for arrivals and polls, values tagged with a sequence number: 2350 cycles with 148 blocks, none of them is below 1950).  The release covers
// the block's writes (ordered before it by the block barrier), the acquire what its threads read after theirs.
struct GridBar {
    unsigned int target, limit;
};
constexpr unsigned int BARRIER_POLLS = 1u << 14;  // fewest polls (some 10 ms): the wait is for the other blocks' phase, not for a copy (position 3900, 7B shape: more than 64)
__device__ __forceinline__ void grid_barrier(const LayersParams& P, GridBar& B) {
    if (P.cluster) {  // the grid is one cluster: the hardware's barrier, 0.25 us
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        return;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        B.target += gridDim.x;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(P.bar) : "memory");
        unsigned int seen, n = 0;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(P.bar) : "memory");
        } while (seen < B.target && ++n < B.limit);
        if (seen < B.target) {
            atomicExch(P.err_flag, 2u);
            B.limit = 1;
        }
    }
    __syncthreads();
}

// ---- attention ----------------------------------------------------------------------------------------------------------------
// Two f32 values a register pair, one instruction for both (fma.rn.f32x2).
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
template <typename T> struct Row;
template <> struct Row<__half> {  // 16 bytes of a cached row as pairs
    __device__ static __forceinline__ void unpack(const uint4& v, unsigned long long (&f)[4]) {
        const __half2* h = reinterpret_cast<const __half2*>(&v);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float2 x = __half22float2(h[i]);
            f[i] = pack2(x.x, x.y);
        }
    }
};
template <> struct Row<float> {
    __device__ static __forceinline__ void unpack(const uint4& v, unsigned long long (&f)[2]) {
        f[0] = pack2(__uint_as_float(v.x), __uint_as_float(v.y));
        f[1] = pack2(__uint_as_float(v.z), __uint_as_float(v.w));
    }
};

// Items (vh, split): MAXQ query heads against the positions of the split.  A group of 2^lanes_log lanes holds one cached row (16 bytes a lane),
// takes every 512 / 2^lanes_log-th position, four at a time, with a running softmax of its own; the groups of a warp meet through shuffles,
// the warps in shared memory.  A phase is a chain of latencies (four warps a scheduler issue one of their instructions every 8 cycles), so
// the rows of the first round are requested before `barrier` (all but the newest, which is written in front of it), a round's four scores
// are summed over the lanes together (each lane ends with one of them, of which it takes the exponential), and products go two to an instruction.
template <typename T, int MAXQ, class Barrier>
__device__ __forceinline__ void attention_phase(const LayersParams& P, int layer, int n, int S, unsigned char* smb, Barrier&& barrier) {
    constexpr int ESZ = (int)sizeof(T), EPL = 16 / ESZ, E2 = EPL / 2, U = ROWS_PER_LANE;
    static_assert(U == 4, "the scores of a round are summed by two halvings");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int hs = P.hs, ll = P.lanes_log, LPR = 1 << ll;
    const int gl = lane & (LPR - 1), gi = (warp << (5 - ll)) + (lane >> ll), GB = WARPS << (5 - ll);
    const bool live = gl * EPL < hs, up1 = gl & (LPR >> 1), up0 = gl & (LPR >> 2);
    const int own = (up1 ? 2 : 0) + (up0 ? 1 : 0), lead = lane & ~(LPR - 1);  // the round's row whose score this lane ends with
    const int chunk = (n + S - 1) / S, items = P.n_items * S;
    const int pitch = hs * ESZ;
    float* wo = reinterpret_cast<float*>(smb);              // [WARPS][MAXQ * hs]
    float* wml = wo + WARPS * MAXQ * hs;                    // [WARPS][MAXQ][2]
    bool first = true;
#pragma unroll 1
    for (int item = (int)blockIdx.x; first || item < items; item += (int)gridDim.x) {
        const int sp = item / P.n_items, vh = item - sp * P.n_items;
        const int t0 = sp * chunk, t1 = item < items ? min(n, t0 + chunk) : 0;
        const size_t at = (size_t)layer * P.layer_bytes + (size_t)(vh / P.kv_share) * P.head_elems * ESZ + 16 * gl;
        const unsigned char *kb = P.kcache + at, *vb = P.vcache + at;
        uint4 kr[U], vr[U];
        auto rows = [&](uint4 (&r)[U], const unsigned char* base, int tb, int lo, int hi) {  // positions lo .. hi - 1 of the round at tb
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int t = tb + gi + u * GB;
                if (t >= lo && t < hi && live) r[u] = __ldcg(reinterpret_cast<const uint4*>(base + (size_t)(unsigned int)(t * pitch)));
            }
        };
#pragma unroll
        for (int u = 0; u < U; u++) kr[u] = vr[u] = make_uint4(0u, 0u, 0u, 0u);
        const int told = first ? min(t1, n - 1) : t1;
        rows(kr, kb, t0, t0, told);
        rows(vr, vb, t0, t0, told);
        if (first) barrier();
        first = false;
        if (item >= items) break;
        if (told < t1) {
            rows(kr, kb, t0, told, t1);
            rows(vr, vb, t0, told, t1);
        }
        unsigned long long qf[MAXQ][E2], o[MAXQ][E2];
        float m[MAXQ], l[MAXQ];
#pragma unroll
        for (int h = 0; h < MAXQ; h++) {
            m[h] = -INFINITY;
            l[h] = 0.f;
#pragma unroll
            for (int e = 0; e < E2; e += 2) {
                const float4 x = live ? __ldcg(reinterpret_cast<const float4*>(P.q + (size_t)(vh * MAXQ + h) * hs + gl * EPL + 2 * e)) : make_float4(0.f, 0.f, 0.f, 0.f);
                qf[h][e] = pack2(x.x, x.y);
                qf[h][e + 1] = pack2(x.z, x.w);
                o[h][e] = o[h][e + 1] = 0ull;
            }
        }
#pragma unroll 1
        for (int tb = t0; tb < t1; tb += U * GB) {
            float sc[MAXQ][U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                unsigned long long kf[E2];
                Row<T>::unpack(kr[u], kf);
#pragma unroll
                for (int h = 0; h < MAXQ; h++) {
                    unsigned long long p = 0ull;
#pragma unroll
                    for (int e = 0; e < E2; e++) p = fma2(kf[e], qf[h][e], p);
                    const float2 p2 = unpack2(p);
                    sc[h][u] = p2.x + p2.y;
                }
            }
            const bool more = tb + U * GB < t1;
            if (more) rows(kr, kb, tb + U * GB, t0, t1);
            float pr[MAXQ];
#pragma unroll
            for (int h = 0; h < MAXQ; h++) {
                const float a0 = (up1 ? sc[h][2] : sc[h][0]) + __shfl_xor_sync(0xffffffffu, up1 ? sc[h][0] : sc[h][2], LPR >> 1);
                const float a1 = (up1 ? sc[h][3] : sc[h][1]) + __shfl_xor_sync(0xffffffffu, up1 ? sc[h][1] : sc[h][3], LPR >> 1);
                pr[h] = (up0 ? a1 : a0) + __shfl_xor_sync(0xffffffffu, up0 ? a0 : a1, LPR >> 2);
            }
#pragma unroll 1
            for (int w = LPR >> 3; w > 0; w >>= 1)
#pragma unroll
                for (int h = 0; h < MAXQ; h++) pr[h] += __shfl_xor_sync(0xffffffffu, pr[h], w);
#pragma unroll
            for (int h = 0; h < MAXQ; h++) {
                const float s = tb + gi + own * GB < t1 ? pr[h] / P.sqrt_hs : -INFINITY;
                float mn = fmaxf(s, __shfl_xor_sync(0xffffffffu, s, LPR >> 1));
                mn = fmaxf(m[h], fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, LPR >> 2)));
                const float base = mn == -INFINITY ? 0.f : mn;  // (nothing yet: the factors are exp(-inf) = 0)
                const float resc = expf(m[h] - base);
                m[h] = mn;
                pr[h] = expf(s - base);
                l[h] = l[h] * resc + pr[h];
                const unsigned long long r2 = pack2(resc, resc);
#pragma unroll
                for (int e = 0; e < E2; e++) o[h][e] = fma2(o[h][e], r2, 0ull);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                unsigned long long vf[E2];
                Row<T>::unpack(vr[u], vf);
#pragma unroll
                for (int h = 0; h < MAXQ; h++) {
                    const float p = __shfl_sync(0xffffffffu, pr[h], lead + (u >> 1) * (LPR >> 1) + (u & 1) * (LPR >> 2));
                    const unsigned long long p2 = pack2(p, p);
#pragma unroll
                    for (int e = 0; e < E2; e++) o[h][e] = fma2(p2, vf[e], o[h][e]);
                }
            }
            if (more) {
#pragma unroll
                for (int u = 0; u < U; u++) vr[u] = make_uint4(0u, 0u, 0u, 0u);  // (a weight may be 0 without its value being finite)
                rows(vr, vb, tb + U * GB, t0, t1);
            }
        }
        // the groups of a warp
        float of[MAXQ][EPL];
#pragma unroll
        for (int h = 0; h < MAXQ; h++) {
            l[h] += __shfl_xor_sync(0xffffffffu, l[h], LPR >> 1);
            l[h] += __shfl_xor_sync(0xffffffffu, l[h], LPR >> 2);
#pragma unroll
            for (int e = 0; e < E2; e++) {
                const float2 x = unpack2(o[h][e]);
                of[h][2 * e] = x.x;
                of[h][2 * e + 1] = x.y;
            }
        }
#pragma unroll 1
        for (int w = LPR; w < 32; w <<= 1)
#pragma unroll
            for (int h = 0; h < MAXQ; h++) {
                const float mo = __shfl_xor_sync(0xffffffffu, m[h], w), lo = __shfl_xor_sync(0xffffffffu, l[h], w);
                const float M = fmaxf(m[h], mo), base = M == -INFINITY ? 0.f : M;
                const float a = expf(m[h] - base), b = expf(mo - base);
                l[h] = l[h] * a + lo * b;
                m[h] = M;
#pragma unroll
                for (int e = 0; e < EPL; e++) of[h][e] = of[h][e] * a + __shfl_xor_sync(0xffffffffu, of[h][e], w) * b;
            }
#pragma unroll
        for (int h = 0; h < MAXQ; h++) {
            if (lane < LPR && live)
#pragma unroll
                for (int e = 0; e < EPL; e += 4)
                    *reinterpret_cast<float4*>(wo + (warp * MAXQ + h) * hs + gl * EPL + e) = make_float4(of[h][e], of[h][e + 1], of[h][e + 2], of[h][e + 3]);
            if (lane == 0) *reinterpret_cast<float2*>(wml + 2 * (warp * MAXQ + h)) = make_float2(m[h], l[h]);
        }
        __syncthreads();
        // Eight elements a warp and round, four lanes each; lane w computes the weight of warp w's sums.
#pragma unroll 1
        for (int d0 = 8 * warp; d0 < MAXQ * hs; d0 += 8 * WARPS) {
            const int h = MAXQ > 1 && d0 >= hs ? 1 : 0, i = d0 + (lane & 7), w0 = 4 * (lane >> 3);
            const float2 ml = *reinterpret_cast<const float2*>(wml + 2 * ((lane & (WARPS - 1)) * MAXQ + h));
            const float M = warp_max_signed(ml.x), s = expf(ml.x - (M == -INFINITY ? 0.f : M)), L = 0.5f * warp_sum(s * ml.y);  // (every warp's pair is there twice)
            float a = 0.f;
#pragma unroll
            for (int w = 0; w < 4; w++) a = fmaf(__shfl_sync(0xffffffffu, s, w0 + w), wo[(w0 + w) * MAXQ * hs + i], a);
            a += __shfl_xor_sync(0xffffffffu, a, 8);
            a += __shfl_xor_sync(0xffffffffu, a, 16);
            if (lane < 8) {
                const int at = vh * MAXQ * hs + i, hd = vh * MAXQ + h;
                if (S == 1) {
                    P.xb[at] = a / L;
                } else {
                    P.part_o[sp * P.n_heads * hs + at] = a;
                    if (i == h * hs) *reinterpret_cast<float2*>(P.part_ml + 2 * (sp * P.n_heads + hd)) = make_float2(M, L);
                }
            }
        }
        __syncthreads();
    }
}
#ifdef SLAI_TRACE
#define DL_STAMP(k) if (blockIdx.x == 0 && tid == 0) st[k] = slai_globaltimer();
#else
#define DL_STAMP(k)
#endif

// 16 warps leave 128 registers a thread.  Two query heads an item with an f16 cache (most grouped-query models) is the one instance that does not fit: it spills
// 60 bytes (120 bytes of loads) in every format, in the attention phase.
template <class F, int ARCH, int MAXQ, typename T>
__global__ void __launch_bounds__(THREADS, 1) decode_layers_kernel(const __grid_constant__ LayersParams P) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // [zero page, digit planes, digit sums: dig_region][partial sums: red_floats][statistics][pieces][1 / scale of every 256 elements]
    // [first and last warp of every tile-matrix][q/k/v rows][ring]
    float* red = reinterpret_cast<float*>(smem_raw + P.dig_region);
    float* stat = red + P.red_floats;
    int4* table = reinterpret_cast<int4*>(stat + 64);  // [WARPS][PH_COUNT]
    float* inv = reinterpret_cast<float*>(table + WARPS * PH_COUNT);
    unsigned char* first_warp = reinterpret_cast<unsigned char*>(inv + P.inv_floats);
    unsigned char* last_warp = first_warp + MAX_TILES * 2;
    int4* rows_qkv = reinterpret_cast<int4*>(last_warp + MAX_TILES * 2);  // of this block, the same in every layer: {cos, +-sin, where to, matrix | rotated << 2 | row << 3}
    const uint32_t smem = (uint32_t)__cvta_generic_to_shared(smem_raw);

    Feed R;
    {
        const uint32_t ring = (smem + (uint32_t)P.dig_region + 4u * (uint32_t)(P.red_floats + P.inv_floats) + 256u + 16u * WARPS * PH_COUNT + 4u * MAX_TILES + 16u * (uint32_t)P.qkv_rows + 127u) & ~127u;
        R.base = ring + warp * P.nstage * Stage<F>::STRIDE;
        R.end = R.base + P.nstage * Stage<F>::STRIDE;
        R.c_addr = R.base;
        R.c_phase = 0;
        R.lane0 = lane == 0 ? 1u : 0u;
        R.limit = P.wait_limit;
        R.issued = 0;
        R.layer = 0;
        R.ph = -1;
        R.left = R.run = 0;
        R.table = (uint32_t)__cvta_generic_to_shared(table + warp * PH_COUNT);
        int mine = 0;
        if (lane < PH_COUNT) {  // this warp's pieces, the same in every layer
            const PhaseGeom& g = P.ph[lane];
            const int U = (g.base + ((int)blockIdx.x < g.rem ? 1 : 0)) * g.nsteps * g.nmat;
            // 16 equal parts; with fewer units than warps one each for the first warps (no warp without units between two of a tile's)
            const int u0 = U < WARPS ? min(warp, U) : U * warp / WARPS, left = (U < WARPS ? min(warp + 1, U) : U * (warp + 1) / WARPS) - u0;
            const int jm = u0 / g.nsteps;
            table[warp * PH_COUNT + lane] = make_int4(jm / g.nmat, jm % g.nmat, u0 - jm * g.nsteps, left);
            mine = left;
        }
        const bool has_units = __any_sync(0xffffffffu, mine > 0);
        if (lane == 0) {
            for (uint32_t a = R.base; a < R.end; a += Stage<F>::STRIDE) mbar_init(a + Stage<F>::MBAR, 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        if (tid < ZERO_BYTES / 4) reinterpret_cast<uint32_t*>(smem_raw)[tid] = 0u;
        __syncwarp();
        if (has_units) feed_advance<F>(R, P);
#pragma unroll 1
        for (uint32_t a = R.base; a < R.end; a += Stage<F>::STRIDE) feed_step<F>(R, P, a);
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // (all blocks are resident; the next kernel waits for this one's end)
    const int pos = __ldcg(P.d_pos), n = pos + 1;
    const int rows_round = ROWS_PER_LANE * (WARPS << (5 - P.lanes_log));
    const int S_att = splits_of(n, rows_round, P.max_splits);
    {
        const PhaseGeom& g = P.ph[PH_QKV];
        const int b = (int)blockIdx.x;
        if (tid < (g.base + (b < g.rem ? 1 : 0)) * 16) {
            const int item = b * g.base + min(b, g.rem) + (tid >> 4), seg = item >= P.tile_v ? 2 : item >= P.tile_k ? 1 : 0;
            const int row = (item - (seg == 2 ? P.tile_v : seg == 1 ? P.tile_k : 0)) * 16 + (tid & 15);
            const int head = row / P.hs, hd = row - head * P.hs;
            const bool valid = row < (seg ? P.kv_rows : P.q_rows);
            float2 r = make_float2(1.f, 0.f);
            if (P.rope_cs && seg < 2 && valid) r = __ldcg(reinterpret_cast<const float2*>(P.rope_cs) + (hd >> 1));
            rows_qkv[tid] = make_int4(__float_as_int(r.x), __float_as_int((tid & 1) ? r.y : -r.y),
                                      !valid ? -1 : seg == 0 ? row : (int)(head * P.head_elems + (long long)pos * P.hs + hd), seg | (P.rope_cs && seg < 2 ? 4 : 0) | (valid ? row << 3 : 0));
        }
    }
    // The rows of x this thread updates, the same ones in both phases that do (PH_O, PH_FF2): kept here.
    const int x_row = ((int)blockIdx.x * P.ph[PH_O].base + min((int)blockIdx.x, P.ph[PH_O].rem)) * 16 + tid;
    float x_own = tid < (P.ph[PH_O].base + ((int)blockIdx.x < P.ph[PH_O].rem ? 1 : 0)) * 16 && x_row < P.ph[PH_O].rows ? __ldcg(P.x + x_row) : 0.f;
    GridBar B{0u, max(P.wait_limit, BARRIER_POLLS)};
    auto barrier = [&] { grid_barrier(P, B); };

#pragma unroll 1
    for (int layer = 0; layer < P.n_layers; layer++) {
        const LayerPtrs& W = P.layer[layer];
#pragma unroll 1
        for (int ph = 0; ph < PH_COUNT; ph++) {
#ifdef SLAI_TRACE
            unsigned long long st[TL_SLOTS] = {};
#endif
            DL_STAMP(0)
            if (ph == PH_O) {
                attention_phase<T, MAXQ>(P, layer, n, S_att, smem_raw + ZERO_BYTES, barrier);  // (the zero page stays)
                DL_STAMP(1)
                barrier();
            } else if (layer > 0 || ph > 0) {
                barrier();
            }
            DL_STAMP(2)
            const PhaseGeom& G = P.ph[ph];
            const int b = (int)blockIdx.x;
            const int i0 = b * G.base + min(b, G.rem), n_local = G.base + (b < G.rem ? 1 : 0);
            // what the phase after this one reads first: its norm's weights, into L2
            if (b == (int)gridDim.x - 1 && (ph & 1)) {
                const float *nw = nullptr, *nb = nullptr;
                if (ph == PH_O) {
                    nw = W.norm_w[1];
                    nb = W.norm_b[1];
                } else if (layer + 1 < P.n_layers) {
                    nw = P.layer[layer + 1].norm_w[0];
                    nb = P.layer[layer + 1].norm_b[0];
                }
                for (int i = tid * 32; i < P.ph[PH_QKV].K; i += THREADS * 32) {
                    if (nw) asm volatile("prefetch.global.L2 [%0];" ::"l"(nw + i));
                    if (nb) asm volatile("prefetch.global.L2 [%0];" ::"l"(nb + i));
                }
            }
            if (n_local > 0) {  // (block-uniform)
                const int K = G.K;
                Smem S;
                S.zero = smem;
                S.dig = S.zero + ZERO_BYTES;
                S.plane = ((K + 255) & ~255) + 32;
                S.sv = S.dig + 4 * S.plane;
                const bool norm = ph == PH_QKV || ph == PH_FF1;
                const float* src = norm ? P.x : ph == PH_O ? P.xb : P.hb;
                float sq = stage_steps<F, ARCH == ARCH_GPT2>(PhaseInput{P, reinterpret_cast<const float4*>(src), ph == PH_O ? S_att : 0},
                                                             norm ? W.norm_w[ph >> 1] : nullptr, W.norm_b[ph >> 1], K, P.eps, S, inv, stat);
                if (ARCH == ARCH_LLAMA && norm) {
                    sq = warp_sum(sq);
                    if (lane == 0) stat[warp] = sq;
                }
                __syncthreads();
                DL_STAMP(3)
                LaneCtx L;
                lane_init<F>(L, lane, S);
                // The bias of the thread's row is on its way during the loop.
                const int row = ph == PH_QKV ? rows_qkv[tid < n_local * 16 ? tid : 0].w >> 3 : i0 * 16 + tid;
                float e_bias = 0.f;
                if (tid < n_local * 16 && (ph == PH_QKV || row < G.rows)) {
                    const float* bias = W.bias[ph == PH_QKV ? rows_qkv[tid].w & 3 : 2 + ph];
                    if (bias) e_bias = bias[row];
                }

                int4 c = piece_of(R.table, ph);  // tile, matrix, step, units left
#pragma unroll 1
                while (c.w > 0) {
                    const int run = min(c.w, G.nsteps - c.z), jm = c.x * G.nmat + c.y;
                    float accA = 0.f, accB = 0.f;
                    int step = c.z;
#pragma unroll 1
                    while (step < c.z + run) {
                        const int end = min(step + Stage<F>::CH, c.z + run);
                        feed_wait<F>(R, P);
                        uint32_t at = R.c_addr;
#pragma unroll 1
                        do {
                            float a = 0.f, bb = 0.f;
                            F::compute(at, step, L, S, a, bb);
                            const float sc = inv[F::STEP == 256 ? step : step >> 1];
                            accA = fmaf(sc, a, accA);
                            accB = fmaf(sc, bb, accB);
                            at += F::STEP_BYTES;
                        } while (++step < end && Stage<F>::CH > 1);
                        __syncwarp();
                        feed_step<F>(R, P, R.c_addr);
                        R.c_addr += Stage<F>::STRIDE;
                        if (R.c_addr == R.end) {
                            R.c_addr = R.base;
                            R.c_phase ^= 1;
                        }
                    }
                    accA += __shfl_xor_sync(0xffffffffu, accA, 1);
                    accA += __shfl_xor_sync(0xffffffffu, accA, 2);
                    accB += __shfl_xor_sync(0xffffffffu, accB, 1);
                    accB += __shfl_xor_sync(0xffffffffu, accB, 2);
                    if (L.t == 0) {
                        float* dst = red + (jm + warp) * 16;
                        dst[L.g] = accA;
                        dst[L.g + 8] = accB;
                    }
                    if (lane == 0) {  // the warps that share a tile-matrix: the one with its first step, the one with its last
                        if (c.z == 0) first_warp[jm] = (unsigned char)warp;
                        if (c.z + run == G.nsteps) last_warp[jm] = (unsigned char)warp;
                    }
                    c.w -= run;
                    c.z = 0;
                    if (G.nmat == 2 && c.y == 0) {
                        c.y = 1;
                    } else {
                        c.y = 0;
                        c.x++;
                    }
                }
                DL_STAMP(4)
                __syncthreads();
                DL_STAMP(5)
                // Epilogue: the partial sums of a row in warp order, then what the phase does with it.
                if (tid < n_local * 16) {
                    float mul = 1.f;
                    if (ARCH == ARCH_LLAMA && norm) {
                        float ts = 0.f;
#pragma unroll
                        for (int w = 0; w < WARPS; w += 4) {
                            const float4 t = *reinterpret_cast<const float4*>(stat + w);
                            ts += (t.x + t.y) + (t.z + t.w);
                        }
                        mul = 1.0f / sqrtf(ts / (float)K + P.eps);
                    }
                    float val[2] = {0.f, 0.f};
#pragma unroll
                    for (int mat = 0; mat < 2; mat++)
                        if (mat < G.nmat) {
                            const int jm = (tid >> 4) * G.nmat + mat, w1 = last_warp[jm];
                            const float* part = red + jm * 16 + (tid & 15);
                            float s = 0.f;
#pragma unroll 1
                            for (int w = first_warp[jm]; w <= w1; w += 4) {
                                float x[4];
#pragma unroll
                                for (int u = 0; u < 4; u++) x[u] = w + u <= w1 ? part[(w + u) * 16] : 0.f;
#pragma unroll
                                for (int u = 0; u < 4; u++) s += x[u];
                            }
                            val[mat] = s * mul;
                        }
                    float y = val[0] + e_bias;
                    if (ph == PH_QKV) {
                        const int4 r = rows_qkv[tid];
                        const float other = __shfl_xor_sync(__activemask(), y, 1);  // rows 2i, 2i + 1 sit in neighbouring lanes
                        if (r.w & 4) y = __int_as_float(r.y) * other + __int_as_float(r.x) * y;
                        if (r.z >= 0) {
                            const int seg = r.w & 3;
                            if (seg == 0) {
                                P.q[r.z] = y;
                            } else {
                                unsigned char* cache = (seg == 1 ? P.kcache : P.vcache) + (size_t)layer * P.layer_bytes;
                                if constexpr (sizeof(T) == 2) reinterpret_cast<__half*>(cache)[r.z] = __float2half_rn(y);
                                else reinterpret_cast<float*>(cache)[r.z] = y;
                            }
                        }
                    } else if (row < G.rows) {
                        if (ph != PH_FF1) P.x[row] = x_own = x_own + y;
                        else if (ARCH == ARCH_GPT2) P.hb[row] = gelu_ref(y);
                        else P.hb[row] = val[1] * (val[0] / (1.0f + expf(-val[0])));
                    }
                }
            }
            DL_STAMP(6)
#ifdef SLAI_TRACE
            if (blockIdx.x == 0 && tid == 0 && P.tl) slai_tl_append(P.tl, 2000 + ph, st);
#endif
        }
    }
    if (R.limit == 0) {  // a wait gave up: this warp's copies land before the block ends
        const int nst = P.nstage;
        unsigned int limit = LAST_POLLS;
        for (int s = 0; s < nst; s++) {
            const int arms = ((int)R.issued - s + nst - 1) / nst;  // copies that went into stage s
            if ((int)R.issued > s) bounded_wait<false, false, 1>(R.base + s * Stage<F>::STRIDE + Stage<F>::MBAR, (uint32_t)(arms - 1) & 1u, limit, P.err_flag);
        }
    }
}

template <class F, int ARCH, int MAXQ, typename T>
int launch_inst(slai_ctx* ctx, const LayersParams& P, int grid, size_t smem) {
    auto kern = decode_layers_kernel<F, ARCH, MAXQ, T>;
    static PerDeviceOnce attr;
    if (attr.need(ctx->device)) {
        SLAI_CHECK_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT));
        SLAI_CHECK_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        SLAI_CHECK_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        attr.set(ctx->device);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[1];  // the blocks wait on one another: all of them resident, or none
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (P.cluster) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned int)grid;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        int clusters = 0;  // (none on a part of a chip without that many neighbouring SMs)
        if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess || clusters < 1) {
            cudaGetLastError();
            return DECODE_LAYERS_NO_FIT;
        }
    } else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    }
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, P);
    if (e == cudaErrorCooperativeLaunchTooLarge) {  // the process has a part of the chip that its properties do not tell of
        cudaGetLastError();
        return DECODE_LAYERS_NO_FIT;
    }
    SLAI_CHECK_CUDA(ctx, e);
    return SLAI_OK;
}
template <class F, typename T>
int launch_t(slai_ctx* ctx, const LayersParams& P, int arch, int grid, size_t smem) {
    if (arch == ARCH_GPT2) return launch_inst<F, ARCH_GPT2, 1, T>(ctx, P, grid, smem);
    return P.kvq == 1 ? launch_inst<F, ARCH_LLAMA, 1, T>(ctx, P, grid, smem) : launch_inst<F, ARCH_LLAMA, 2, T>(ctx, P, grid, smem);
}
template <class F>
int launch_fmt(slai_ctx* ctx, const LayersParams& P, int arch, bool f16, int grid, size_t smem) {
    return f16 ? launch_t<F, __half>(ctx, P, arch, grid, smem) : launch_t<F, float>(ctx, P, arch, grid, smem);
}

}  // namespace declayers

int decode_layers_launch_q4k(slai_ctx* ctx, const declayers::LayersParams& P, int arch, bool f16, int grid, size_t smem);
int decode_layers_launch_q5k(slai_ctx* ctx, const declayers::LayersParams& P, int arch, bool f16, int grid, size_t smem);
int decode_layers_launch_q6k(slai_ctx* ctx, const declayers::LayersParams& P, int arch, bool f16, int grid, size_t smem);
int decode_layers_launch_q80(slai_ctx* ctx, const declayers::LayersParams& P, int arch, bool f16, int grid, size_t smem);
