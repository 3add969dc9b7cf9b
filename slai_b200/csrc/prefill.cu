// Prompt processing: the kernels around the GEMMs (prefill_gemm.cu) of a pass over T prompt tokens at once.
//
// The reference feeds a prompt one token at a time through its decode step (crates/slai-chat/src/chat_llama2.rs:109-115
// loops forward_logits over the prompt; the operator sequence is Llama2::launch, crates/slai/src/models/llama2/
// transformer.rs:316-381).  For a prompt of T tokens that streams every weight T times.  Here the T activation rows go
// through each matrix together: Y[T x M] = X[T x K] W^T, the only place on this path where the work is a GEMM.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "dequant.cuh"

// All of these launch behind their predecessor's start.  What a kernel in front of them wrote (activations, q / k / v, caches) is
// read with __ldcg and without __restrict__: the read-only path asks for memory that is constant as long as the kernel runs, and
// a load marked so may move in front of griddepcontrol.wait.  Weights and tables may use both.
namespace {

// ---- causal attention of a block of prompt tokens ---------------------------------------------------------------------
// The decode step's attention serves one query token and streams that token's whole key / value history; run once per
// prompt token it reads the caches T / 2 times over.  Here one CTA takes 16 consecutive query tokens of one head and walks
// the positions they may attend to in tiles of 32: a tile of keys and values is brought into shared memory once (as f32)
// and serves all 16 queries.  Warp w owns queries 4w .. 4w + 3; for the scores lane = position of the tile (a 128-bit read
// of its own key row per four dimensions, the queries broadcast), then a streaming softmax per query (running maximum
// and sum, ops/batched_multiquery_attention.rs:102-156 computes the same softmax over all positions at once), then for the
// weighted sum of values lane = four output dimensions.  Plain f32 arithmetic, like the decode step's kernel.
constexpr int PA_QT = 16, PA_KT = 32, PA_THREADS = 128, PA_MAXC = 2;  // head_size <= 128 * PA_MAXC

template <typename T>
__device__ __forceinline__ void pa_load_rows(const T* g, long long row_stride, int rows, int hs, float* s, int s_stride, int tid) {
    constexpr int VEC = 16 / (int)sizeof(T);  // elements per 16-byte piece
    const int ppr = hs / VEC;
    for (int idx = tid; idx < PA_KT * ppr; idx += PA_THREADS) {
        const int r = idx / ppr, c = idx - r * ppr;
        float v[VEC];
        if (r < rows) {
            const uint4 raw = __ldcg(reinterpret_cast<const uint4*>(g + (long long)r * row_stride) + c);
            if (sizeof(T) == 2) {
                const __half2* h2 = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
                for (int i = 0; i < VEC / 2; i++) {
                    const float2 f = __half22float2(h2[i]);
                    v[2 * i] = f.x;
                    v[2 * i + 1] = f.y;
                }
            } else {
                const float* f = reinterpret_cast<const float*>(&raw);
#pragma unroll
                for (int i = 0; i < VEC; i++) v[i] = f[i];
            }
        } else {
#pragma unroll
            for (int i = 0; i < VEC; i++) v[i] = 0.f;
        }
        float* dst = s + (size_t)r * s_stride + c * VEC;
#pragma unroll
        for (int i = 0; i < VEC; i += 4) *reinterpret_cast<float4*>(dst + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    }
}

template <typename T>
__global__ void __launch_bounds__(PA_THREADS)
prefill_attn_kernel(const float* q, int q_ld, const T* kc, const T* vc, long long head_stride, int hs, int kv_mul, int pos0, int n_tokens, float* out,
                    int out_ld) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    extern __shared__ __align__(16) float pa_sm[];
    const int ks = hs + 4;              // key rows 4 floats apart modulo 32 banks: the lanes' 128-bit reads do not collide
    float* q_s = pa_sm;                 // [PA_QT][hs], already divided by sqrt(hs)
    float* k_s = q_s + PA_QT * hs;      // [PA_KT][hs + 4]
    float* v_s = k_s + PA_KT * ks;      // [PA_KT][hs]
    float* p_s = v_s + PA_KT * hs;      // [PA_QT][PA_KT]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int head = blockIdx.x, t0 = blockIdx.y * PA_QT;
    const int nq = min(PA_QT, n_tokens - t0);
    const int kvh = head / kv_mul;
    const T* kbase = kc + (long long)kvh * head_stride;
    const T* vbase = vc + (long long)kvh * head_stride;
    const float inv = 1.0f / sqrtf((float)hs);
    for (int i = tid; i < PA_QT * hs; i += PA_THREADS) {
        const int tq = i / hs, d = i - tq * hs;
        q_s[i] = tq < nq ? __ldcg(q + (size_t)(t0 + tq) * q_ld + (size_t)head * hs + d) * inv : 0.f;
    }
    float m[4], l[4], acc[4][PA_MAXC][4];
#pragma unroll
    for (int qi = 0; qi < 4; qi++) {
        m[qi] = -INFINITY;
        l[qi] = 0.f;
#pragma unroll
        for (int c = 0; c < PA_MAXC; c++) acc[qi][c][0] = acc[qi][c][1] = acc[qi][c][2] = acc[qi][c][3] = 0.f;
    }
    const int last_pos = pos0 + t0 + nq - 1;           // last position any query of this tile attends to
    const int warp_last = pos0 + t0 + 4 * warp + 3;    // ... any query of this warp
    for (int kt0 = 0; kt0 <= last_pos; kt0 += PA_KT) {
        const int cnt = min(PA_KT, last_pos + 1 - kt0);
        __syncthreads();  // the previous tile has been consumed (and, the first time round, q_s is complete)
        pa_load_rows<T>(kbase + (long long)kt0 * hs, hs, cnt, hs, k_s, ks, tid);
        pa_load_rows<T>(vbase + (long long)kt0 * hs, hs, cnt, hs, v_s, hs, tid);
        __syncthreads();
        if (kt0 > warp_last || 4 * warp >= nq) continue;  // nothing in this tile for this warp's queries (warp-uniform)
        float sc[4] = {0.f, 0.f, 0.f, 0.f};
        const float* kr = k_s + lane * ks;
        const float* qr = q_s + 4 * warp * hs;
        for (int d = 0; d < hs; d += 4) {
            const float4 kv = *reinterpret_cast<const float4*>(kr + d);
#pragma unroll
            for (int qi = 0; qi < 4; qi++) {
                const float4 qv = *reinterpret_cast<const float4*>(qr + qi * hs + d);
                sc[qi] = fmaf(kv.x, qv.x, fmaf(kv.y, qv.y, fmaf(kv.z, qv.z, fmaf(kv.w, qv.w, sc[qi]))));
            }
        }
#pragma unroll
        for (int qi = 0; qi < 4; qi++) {
            const int qpos = pos0 + t0 + 4 * warp + qi;
            const bool valid = lane < cnt && kt0 + lane <= qpos && 4 * warp + qi < nq;
            const float sv = valid ? sc[qi] : -INFINITY;
            float mt = sv;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, o));
            const float m_new = fmaxf(m[qi], mt);
            const float pv = valid ? expf(sv - m_new) : 0.f;
            float ps = pv;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, o);
            const float resc = m[qi] == -INFINITY ? 0.f : expf(m[qi] - m_new);  // nothing accumulated yet: acc and l are zero anyway
            l[qi] = l[qi] * resc + ps;
            m[qi] = m_new;
#pragma unroll
            for (int c = 0; c < PA_MAXC; c++) {
                acc[qi][c][0] *= resc; acc[qi][c][1] *= resc; acc[qi][c][2] *= resc; acc[qi][c][3] *= resc;
            }
            p_s[(4 * warp + qi) * PA_KT + lane] = pv;
        }
        __syncwarp();
        const float* pr = p_s + 4 * warp * PA_KT;
        for (int j = 0; j < cnt; j += 4) {
            float4 pq[4];
#pragma unroll
            for (int qi = 0; qi < 4; qi++) pq[qi] = *reinterpret_cast<const float4*>(pr + qi * PA_KT + j);
#pragma unroll
            for (int jj = 0; jj < 4; jj++) {
#pragma unroll
                for (int c = 0; c < PA_MAXC; c++) {
                    const int d = 128 * c + 4 * lane;
                    if (d < hs) {
                        const float4 vv = *reinterpret_cast<const float4*>(v_s + (size_t)(j + jj) * hs + d);  // rows >= cnt are zero
#pragma unroll
                        for (int qi = 0; qi < 4; qi++) {
                            const float pw = jj == 0 ? pq[qi].x : jj == 1 ? pq[qi].y : jj == 2 ? pq[qi].z : pq[qi].w;
                            acc[qi][c][0] = fmaf(pw, vv.x, acc[qi][c][0]);
                            acc[qi][c][1] = fmaf(pw, vv.y, acc[qi][c][1]);
                            acc[qi][c][2] = fmaf(pw, vv.z, acc[qi][c][2]);
                            acc[qi][c][3] = fmaf(pw, vv.w, acc[qi][c][3]);
                        }
                    }
                }
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int qi = 0; qi < 4; qi++) {
        const int tq = 4 * warp + qi;
        if (tq < nq) {
#pragma unroll
            for (int c = 0; c < PA_MAXC; c++) {
                const int d = 128 * c + 4 * lane;
                if (d < hs) {
                    const float il = 1.0f / l[qi];  // position 0 is always attended to: l > 0
                    *reinterpret_cast<float4*>(out + (size_t)(t0 + tq) * out_ld + (size_t)head * hs + d) =
                        make_float4(acc[qi][c][0] * il, acc[qi][c][1] * il, acc[qi][c][2] * il, acc[qi][c][3] * il);
                }
            }
        }
    }
}

// The same attention on the tensor cores, for f16 caches and heads of 64 or 128 dimensions: 64 query tokens of one head per
// CTA (16 per warp), tiles of 64 positions, keys and values in shared memory as they are cached (two tiles in flight, cp.async,
// 16-byte chunks xor-swizzled so that ldmatrix meets no bank conflict).  The f32 kernel above is bound by its shared-memory reads
// (five 16-byte reads for 16 FMAs per lane): 511 tokens x 32 heads took 217 us of a 7B layer's 820.
//
// Numerics: keys and values are f16 already; queries and probabilities are f32 and go in as pairs of halves (v = hi + lo, 22
// bits; a row's queries scaled by a power of two so that neither end of their range is lost, probabilities times 4096, so that
// lo keeps its bits), two products each.  The tensor core truncates when it adds, so sums are kept short: the small products
// first, the large ones in two halves (scores), and a fresh accumulator per tile that is added to the running output in f32
// arithmetic (values).  Relative error over the whole output against 64 bits, the f32 kernel's / this one's (heads of 128, 511
// tokens): normal queries and keys 3.4e-7 / 2.1e-7, queries 30 times that 2.3e-6 / 0.7e-6, a thousandth 1.7e-7 / 1.0e-7, a mean of
// 3 on both 4.8e-6 / 1.1e-6; no larger at any of 50 settings (heads of 64 and 128, 37 to 3064 positions).
//
// A short turn has one CTA per head, which walks the whole conversation tile by tile (5 us a tile): the tiles of a (head, 64 queries) are dealt to the CTAs
// of a cluster along z, whose outputs and (max, sum) pairs meet through distributed shared memory in rank order.
constexpr int PM_QT = 64, PM_KT = 64, PM_THREADS = 128;

__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void split2(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(x, y);
    const __half2 l = __floats2half2_rn(x - __low2float(h), y - __high2float(h));
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

template <int HS>
__global__ void __launch_bounds__(PM_THREADS, 2)
prefill_attn_mma_kernel(const float* q, int q_ld, const __half* kc, const __half* vc, long long head_stride, int kv_mul, int pos0, int n_tokens, float* out,
                        int out_ld) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr int ROW = HS * 2, CH = HS / 8, TILE = PM_KT * ROW;  // bytes of a cached row, its 16-byte chunks, bytes of a tile
    constexpr int KS = HS / 16, NT8 = HS / 8;                     // 16-deep steps of the scores, 8-wide tiles of the output
    extern __shared__ __align__(128) unsigned char pm_sm[];       // [2][keys, values][64][HS]
    const uint32_t sm = (uint32_t)__cvta_generic_to_shared(pm_sm);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int head = blockIdx.x, t0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * PM_QT;  // the longest histories start first
    const int nq = min(PM_QT, n_tokens - t0);
    const __half* kb = kc + (long long)(head / kv_mul) * head_stride;
    const __half* vb = vc + (long long)(head / kv_mul) * head_stride;
    const int last_pos = pos0 + t0 + nq - 1;  // last position any query of this CTA attends to
    const int all_tiles = last_pos / PM_KT + 1, ranks = (int)gridDim.z, rank = (int)blockIdx.z;  // (the grid is one cluster deep)
    const int tile_lo = all_tiles * rank / ranks, tiles = all_tiles * (rank + 1) / ranks;

    auto load_tile = [&](int tile) {
        const int p0 = tile * PM_KT;
        const uint32_t dst = sm + (tile & 1) * 2 * TILE;
#pragma unroll
        for (int i = 0; i < PM_KT * CH / PM_THREADS; i++) {
            const int idx = tid + i * PM_THREADS, r = idx / CH, c = idx % CH;
            const uint32_t off = r * ROW + ((c ^ (r & 7)) << 4);
            const bool in = p0 + r <= last_pos;  // rows behind the last position: zeros, nothing is read
            const size_t src = (size_t)(in ? p0 + r : 0) * HS + c * 8;
            const uint32_t n = in ? 16u : 0u;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + off), "l"(__cvta_generic_to_global(kb + src)), "r"(n) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + TILE + off), "l"(__cvta_generic_to_global(vb + src)), "r"(n) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (tile_lo < tiles) load_tile(tile_lo);

    // Queries of this warp (rows g and g + 8 of its 16), divided by sqrt(head size), each row times a power of two that puts its largest
    // element below 2^15: whatever their size they fit a pair of halves.  `unit` takes the power out of the row's scores again.
    uint32_t qh[KS][4], ql[KS][4];
    const int row0 = t0 + 16 * warp + g;
    float unit[2];
    {
        float2 v[KS][4];
        float mx[2] = {0.f, 0.f};
#pragma unroll
        for (int k = 0; k < KS; k++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int row = row0 + 8 * (i & 1), d = 16 * k + 2 * t + 8 * (i >> 1);
                v[k][i] = make_float2(0.f, 0.f);
                if (row < n_tokens) v[k][i] = __ldcg(reinterpret_cast<const float2*>(q + (size_t)row * q_ld + (size_t)head * HS + d));
                mx[i & 1] = fmaxf(mx[i & 1], fmaxf(fabsf(v[k][i].x), fabsf(v[k][i].y)));
            }
        float up[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
            mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
            // 2^(14 - e) for a largest element of 2^e .. 2^(e + 1); e is held at -112, where the scores are zero for any key
            const int e = max((int)(__float_as_uint(mx[h]) >> 23), 15);  // biased by 127
            up[h] = __uint_as_float((uint32_t)(127 + 14 + 127 - e) << 23) * (1.0f / sqrtf((float)HS));
            unit[h] = __uint_as_float((uint32_t)(e - 14) << 23);
        }
#pragma unroll
        for (int k = 0; k < KS; k++)
#pragma unroll
            for (int i = 0; i < 4; i++) split2(v[k][i].x * up[i & 1], v[k][i].y * up[i & 1], qh[k][i], ql[k][i]);
    }
    float acc[NT8][4];
#pragma unroll
    for (int n = 0; n < NT8; n++) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
    const int warp_last = pos0 + t0 + 16 * warp + 15;  // last position any query of this warp attends to
    const int qpos[2] = {pos0 + row0, pos0 + row0 + 8};

    for (int tile = tile_lo; tile < tiles; tile++) {
        if (tile + 1 < tiles) load_tile(tile + 1);
        else asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const int p0 = tile * PM_KT;
        if (p0 <= warp_last && 16 * warp < nq) {
            const uint32_t ks = sm + (tile & 1) * 2 * TILE, vs = ks + TILE;
            float sc[8][4];
#pragma unroll
            for (int n = 0; n < 8; n++) {
                // B of 8 positions: matrices of 8 positions x 8 dimensions, four (= 32 dimensions) per load
                float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};
                uint32_t b[KS / 2][4];
                const int r = 8 * n + (lane & 7);
#pragma unroll
                for (int k2 = 0; k2 < KS / 2; k2++) ldsm4(ks + r * ROW + (((4 * k2 + (lane >> 3)) ^ (r & 7)) << 4), b[k2]);
#pragma unroll
                for (int k = 0; k < KS; k++) mma_f16((k & 1) ? c1 : c0, ql[k], b[k >> 1][2 * (k & 1)], b[k >> 1][2 * (k & 1) + 1]);
#pragma unroll
                for (int k = 0; k < KS; k++) mma_f16((k & 1) ? c1 : c0, qh[k], b[k >> 1][2 * (k & 1)], b[k >> 1][2 * (k & 1) + 1]);
#pragma unroll
                for (int i = 0; i < 4; i++) sc[n][i] = (c0[i] + c1[i]) * unit[i >> 1];
            }
            if (p0 + PM_KT - 1 > pos0 + t0 + 16 * warp) {  // the diagonal passes through: positions after a query's own do not count
#pragma unroll
                for (int n = 0; n < 8; n++)
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        if (p0 + 8 * n + 2 * t + (i & 1) > qpos[i >> 1]) sc[n][i] = -INFINITY;
            }
            float resc[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {  // rows g, g + 8: streaming softmax
                float mt = -INFINITY;
#pragma unroll
                for (int n = 0; n < 8; n++) mt = fmaxf(mt, fmaxf(sc[n][2 * h], sc[n][2 * h + 1]));
                mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, 1));
                mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, 2));
                const float m_new = fmaxf(m[h], mt);
                resc[h] = m[h] == -INFINITY ? 0.f : expf(m[h] - m_new);  // nothing accumulated yet: acc and l are zero anyway
                m[h] = m_new;
                float ps = 0.f;
#pragma unroll
                for (int n = 0; n < 8; n++)
#pragma unroll
                    for (int i = 2 * h; i < 2 * h + 2; i++) {
                        const float p = sc[n][i] == -INFINITY ? 0.f : expf(sc[n][i] - m_new);
                        ps += p;
                        sc[n][i] = p * 4096.f;
                    }
                l[h] = l[h] * resc[h] + ps;  // (this lane's positions only: added up at the end)
            }
            uint32_t ph[4][4], pl[4][4];
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int i = 0; i < 4; i++) split2(sc[2 * j + (i >> 1)][2 * (i & 1)], sc[2 * j + (i >> 1)][2 * (i & 1) + 1], ph[j][i], pl[j][i]);
            auto add_values = [&](auto diagonal) {
                // Positions behind the warp's last query have probability zero; their values are not multiplied (an infinite one
                // would reach the queries before it).
                const int wl = warp_last - p0;
#pragma unroll
                for (int n2 = 0; n2 < NT8 / 2; n2++) {  // 16 output dimensions
                    float c[2][4] = {};
                    uint32_t b[4][4];
#pragma unroll
                    for (int j = 0; j < 4; j++) {  // matrices: positions 16j .. + 7, + 8 .. + 15 of 8 dimensions, then of the next 8
                        const int r = 16 * j + (lane & 15);
                        ldsm4t(vs + r * ROW + (((2 * n2 + (lane >> 4)) ^ (r & 7)) << 4), b[j]);
                    }
                    if (decltype(diagonal)::value) {
#pragma unroll
                        for (int j = 0; j < 4; j++)
#pragma unroll
                            for (int i = 0; i < 4; i++) {
                                const int p = 16 * j + 8 * (i & 1) + 2 * t;  // this lane's positions p (low half), p + 1
                                b[j][i] = p > wl ? 0u : p + 1 > wl ? b[j][i] & 0xFFFFu : b[j][i];
                            }
                    }
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        mma_f16(c[0], pl[j], b[j][0], b[j][1]);
                        mma_f16(c[1], pl[j], b[j][2], b[j][3]);
                    }
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        mma_f16(c[0], ph[j], b[j][0], b[j][1]);
                        mma_f16(c[1], ph[j], b[j][2], b[j][3]);
                    }
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        float& a = acc[2 * n2 + (i >> 2)][i & 3];
                        a = fmaf(a, resc[(i & 3) >> 1], c[i >> 2][i & 3]);
                    }
                }
            };
            if (p0 + PM_KT - 1 > warp_last) add_values(std::true_type());
            else add_values(std::false_type());
        }
        __syncthreads();  // the tile's buffer is loaded again next round
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 1);
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 2);
    }
    if (ranks == 1) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int row = row0 + 8 * h;
            if (row < n_tokens) {
                const float il = 1.0f / (l[h] * 4096.f);  // position 0 is always attended to: l > 0
#pragma unroll
                for (int n = 0; n < NT8; n++)
                    *reinterpret_cast<float2*>(out + (size_t)row * out_ld + (size_t)head * HS + 8 * n + 2 * t) = make_float2(acc[n][2 * h] * il, acc[n][2 * h + 1] * il);
            }
        }
        return;
    }
    // [64][HS] outputs, [64][2] (max, sum) where the tiles were (all of them have been read)
    float* so = reinterpret_cast<float*>(pm_sm);
    float* sml = so + PM_QT * HS;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int r = 16 * warp + g + 8 * h;
#pragma unroll
        for (int n = 0; n < NT8; n++) *reinterpret_cast<float2*>(so + r * HS + 8 * n + 2 * t) = make_float2(acc[n][2 * h], acc[n][2 * h + 1]);
        if (t == 0) *reinterpret_cast<float2*>(sml + 2 * r) = make_float2(m[h], l[h]);
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int lo = nq * rank / ranks * (HS / 4), hi = nq * (rank + 1) / ranks * (HS / 4);  // this CTA's share of the rows, four elements a thread
    for (int i = lo + tid; i < hi; i += PM_THREADS) {
        const int r = i / (HS / 4), d = 4 * (i - r * (HS / 4));
        float4 num = make_float4(0.f, 0.f, 0.f, 0.f);
        float M = -INFINITY, den = 0.f;
        for (int z0 = 0; z0 < ranks; z0 += 4) {
            float2 ml[4];
            float4 o[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                ml[u] = make_float2(-INFINITY, 0.f);
                o[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (z0 + u < ranks) {
                    uint32_t a, b;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(sm + 4 * (PM_QT * HS + 2 * r)), "r"(z0 + u));
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(sm + 4 * (r * HS + d)), "r"(z0 + u));
                    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(ml[u].x), "=f"(ml[u].y) : "r"(a) : "memory");
                    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(o[u].x), "=f"(o[u].y), "=f"(o[u].z), "=f"(o[u].w) : "r"(b) : "memory");
                }
            }
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (ml[u].y > 0.f || ml[u].y != ml[u].y) {  // (a rank without positions of this query has no sum; a NaN stays one)
                    const float Mn = fmaxf(M, ml[u].x);
                    const float a = M == -INFINITY ? 0.f : expf(M - Mn), b = expf(ml[u].x - Mn);
                    num.x = num.x * a + b * o[u].x; num.y = num.y * a + b * o[u].y; num.z = num.z * a + b * o[u].z; num.w = num.w * a + b * o[u].w;
                    den = den * a + b * ml[u].y;
                    M = Mn;
                }
        }
        const float il = 1.0f / (den * 4096.f);
        *reinterpret_cast<float4*>(out + (size_t)(t0 + r) * out_ld + (size_t)head * HS + d) = make_float4(num.x * il, num.y * il, num.z * il, num.w * il);
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");  // nobody leaves while another reads
}

// ---- small kernels around the GEMMs ---------------------------------------------------------------------------------
__device__ __forceinline__ float block_sum256(float x, float* sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = x;
    __syncthreads();
    float t = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sh[w];
    return t;
}
// Four neighbouring activations (group `i` of row t) as the GEMM's operands: fp16 pairs, y = hi + lo, into planes of
// [t_pad][K]; and, where `sum` is given (K a multiple of 256), the sum over each 32-element sub-block of hi + lo, divided by 32 (so
// that it stays inside fp16's range whenever the activations do), as 16 columns per super-block of 256: eight fp16 sums,
// then 2048 times their rounding errors (the minimum term of Q4_K / Q5_K, prefill_dequant.cuh).  Eight lanes hold a sub-block;
// whole warps call this (`on`: the group exists).
__device__ __forceinline__ void store_operands(__half* hi, __half* lo, __half* sum, int t, int K, int i, bool on, float4 y) {
    const float v[4] = {y.x, y.y, y.z, y.w};
    __half h[4], l[4];
    float s = 0.f;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        h[e] = __float2half_rn(v[e]);
        l[e] = __float2half_rn(v[e] - __half2float(h[e]));
        s += __half2float(h[e]) + __half2float(l[e]);
    }
    if (on) {
        *reinterpret_cast<uint2*>(hi + (size_t)t * K + 4 * i) = *reinterpret_cast<const uint2*>(h);
        *reinterpret_cast<uint2*>(lo + (size_t)t * K + 4 * i) = *reinterpret_cast<const uint2*>(l);
    }
    if (sum) {
        if (!on) s = 0.f;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (on && (i & 7) == 0) {
            s *= 0.03125f;
            const __half sh = __float2half_rn(s);
            __half* d = sum + (size_t)t * (K >> 4) + (i >> 6) * 16 + ((i >> 3) & 7);
            d[0] = sh;
            d[8] = __float2half_rn((s - __half2float(sh)) * 2048.f);
        }
    }
}

// Row t of X (optionally RmsNorm'd: ops/rms_norm.rs:68-77) as GEMM operands.
__global__ void prefill_split_kernel(const float* x, int ldx, const float* __restrict__ norm_w, float eps, int K, __half* hi, __half* lo, __half* sum) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ float sh[32];
    const int t = blockIdx.x, n4 = K >> 2;
    const float4* xr = reinterpret_cast<const float4*>(x + (size_t)t * ldx);
    const float4* w4 = reinterpret_cast<const float4*>(norm_w);
    float mul = 1.f;
    if (norm_w) {
        float s = 0.f;
        for (int i = threadIdx.x; i < n4; i += blockDim.x) {
            const float4 v = __ldcg(xr + i);
            s += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
        }
        s = block_sum256(s, sh);
        mul = 1.0f / sqrtf(s / (float)K + eps);
    }
    for (int i0 = 0; i0 < n4; i0 += blockDim.x) {
        const int i = i0 + threadIdx.x;
        float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < n4) {
            y = __ldcg(xr + i);
            if (norm_w) {
                const float4 w = w4[i];
                y.x = __fmul_rn(__fmul_rn(y.x, mul), w.x); y.y = __fmul_rn(__fmul_rn(y.y, mul), w.y);
                y.z = __fmul_rn(__fmul_rn(y.z, mul), w.z); y.w = __fmul_rn(__fmul_rn(y.w, mul), w.w);
            }
        }
        store_operands(hi, lo, sum, t, K, i, i < n4, y);
    }
}

// Row t of X after LayerNorm with gamma / beta (ops/layernorm.rs:104-111 and the caller's scale and shift,
// models/gpt2/cpu.rs:239-240) as GEMM operands; same arithmetic as the decode step's fused prologue.
__global__ void prefill_split_ln_kernel(const float* x, int ldx, const float* __restrict__ gamma, const float* __restrict__ beta, float eps, int K, __half* hi,
                                        __half* lo, __half* sum) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ float sh[32];
    const int t = blockIdx.x, n4 = K >> 2;
    const float4* xr = reinterpret_cast<const float4*>(x + (size_t)t * ldx);
    const float4 *g4 = reinterpret_cast<const float4*>(gamma), *b4 = reinterpret_cast<const float4*>(beta);
    float s = 0.f;
    for (int i = threadIdx.x; i < n4; i += blockDim.x) {
        const float4 v = __ldcg(xr + i);
        s += (v.x + v.y) + (v.z + v.w);
    }
    const float mean = block_sum256(s, sh) / (float)K;
    float v = 0.f;
    for (int i = threadIdx.x; i < n4; i += blockDim.x) {
        float4 d = __ldcg(xr + i);
        d.x -= mean; d.y -= mean; d.z -= mean; d.w -= mean;
        v += d.x * d.x + d.y * d.y + d.z * d.z + d.w * d.w;
    }
    v = block_sum256(v, sh);
    const float mul = 1.0f / sqrtf(v / (float)K + eps);
    for (int i0 = 0; i0 < n4; i0 += blockDim.x) {
        const int i = i0 + threadIdx.x;
        float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < n4) {
            y = __ldcg(xr + i);
            const float4 g = g4[i], b = beta ? b4[i] : make_float4(0.f, 0.f, 0.f, 0.f);
            y.x = __fmul_rn(__fmul_rn(y.x - mean, mul), g.x) + b.x; y.y = __fmul_rn(__fmul_rn(y.y - mean, mul), g.y) + b.y;
            y.z = __fmul_rn(__fmul_rn(y.z - mean, mul), g.z) + b.z; y.w = __fmul_rn(__fmul_rn(y.w - mean, mul), g.w) + b.w;
        }
        store_operands(hi, lo, sum, t, K, i, i < n4, y);
    }
}

// gelu (ops/unary.rs:81-85) of [T][H] straight into the operands of the next GEMM.
__device__ __forceinline__ float gelu1(float x) {
    const float A = 0.044715f, Sq = 0.7978846f;
    return 0.5f * x * (1.0f + tanhf(Sq * x * (1.0f + A * x * x)));
}
__global__ void prefill_gelu_split_kernel(const float* g, int H, __half* hi, __half* lo, __half* sum) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int t = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool on = i < (H >> 2);
    float4 y = on ? __ldcg(reinterpret_cast<const float4*>(g + (size_t)t * H) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    y.x = gelu1(y.x); y.y = gelu1(y.y); y.z = gelu1(y.z); y.w = gelu1(y.w);
    store_operands(hi, lo, sum, t, H, i, on, y);
}

// x[t] += row (pos0 + t) of a table of position vectors (models/gpt2/cpu.rs:227-228).
__global__ void prefill_add_rows_kernel(float* x, int dim, const float* __restrict__ table, int pos0) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int t = blockIdx.y;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < dim) x[(size_t)t * dim + i] = __ldcg(x + (size_t)t * dim + i) + table[(size_t)(pos0 + t) * dim + i];
}

// hb = up * gate / (1 + exp(-gate)) (ops/silu.rs:50-58) straight into the operands of the down projection.
__device__ __forceinline__ float silu1(float g, float u) { return u * (g / (1.0f + expf(-g))); }
__global__ void prefill_silu_split_kernel(const float* gate, const float* up, int H, __half* hi, __half* lo, __half* sum) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int t = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool on = i < (H >> 2);
    float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
    if (on) {
        const float4 g = __ldcg(reinterpret_cast<const float4*>(gate + (size_t)t * H) + i), u = __ldcg(reinterpret_cast<const float4*>(up + (size_t)t * H) + i);
        y = make_float4(silu1(g.x, u.x), silu1(g.y, u.y), silu1(g.z, u.z), silu1(g.w, u.w));
    }
    store_operands(hi, lo, sum, t, H, i, on, y);
}

// x[t] = row token[t] of the embedding table (f32 table or quantised matrix).
__global__ void prefill_embed_kernel(float* __restrict__ x, int dim, const int* __restrict__ tokens, const float* __restrict__ table,
                                     int fmt, const uint8_t* __restrict__ qdata) {
    const int t = blockIdx.y;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= dim) return;
    const long long row = tokens[t];
    x[(size_t)t * dim + i] = table ? table[row * dim + i] : dequant_elem(fmt, qdata, dim, row, i);
}

// RoPE (ops/rope.rs:88-125; both variants) on q and k of token t at position pos0 + t (or *d_pos + t), q to `q_out`
// (may be its source), k and, when given, v into the cache ([kv_head][position][head_size], f16 or f32): the q/k/v
// epilogue of the decode step for T tokens at once, and the decode step's own RoPE stage where the fused epilogue
// cannot serve (pairs half a head apart, dense f32 matrices).
__global__ void rope_kv_store_kernel(const float* q_src, const float* k_src, const float* v_src, int ld, int q_dim, int kv_dim, int head_size, int pos0,
                                     const int* d_pos, const float* __restrict__ theta, int neox, float* q_out, int ldq, void* kcache, void* vcache,
                                     int kv_f16, long long kv_head_stride, long long seq_stride) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int t = blockIdx.y;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;  // pair index over q then k; then plain copies of v
    // seq_stride > 0: row t is a sequence of its own, at position d_pos[t] of caches seq_stride bytes after row t - 1's
    const int pos = seq_stride > 0 ? __ldcg(d_pos + t) : (d_pos ? __ldcg(d_pos) : pos0) + t;
    if (pos < 0) return;
    kcache = reinterpret_cast<char*>(kcache) + (size_t)t * seq_stride;
    vcache = reinterpret_cast<char*>(vcache) + (size_t)t * seq_stride;
    const int nq = q_dim / 2, nk = kv_dim / 2;
    if (p < nq + nk) {
        const bool is_k = p >= nq;
        const int i = is_k ? p - nq : p;
        const float* src = (is_k ? k_src : q_src) + (size_t)t * ld;
        const int head = (2 * i) / head_size, fi = ((2 * i) % head_size) >> 1;
        int a, b;
        if (neox) {
            a = head * head_size + fi;
            b = a + head_size / 2;
        } else {
            a = 2 * i;
            b = a + 1;
        }
        float sn, cs;
        sincosf((float)pos * theta[fi], &sn, &cs);
        const float xa = __ldcg(src + a), xb = __ldcg(src + b);
        const float ya = cs * xa - sn * xb, yb = sn * xa + cs * xb;
        if (!is_k) {
            q_out[(size_t)t * ldq + a] = ya;
            q_out[(size_t)t * ldq + b] = yb;
        } else {
            const int ha = a / head_size, da = a % head_size, hb = b / head_size, db = b % head_size;
            const long long oa = (long long)pos * head_size + ha * kv_head_stride + da, ob = (long long)pos * head_size + hb * kv_head_stride + db;
            if (kv_f16) {
                reinterpret_cast<__half*>(kcache)[oa] = __float2half_rn(ya);
                reinterpret_cast<__half*>(kcache)[ob] = __float2half_rn(yb);
            } else {
                reinterpret_cast<float*>(kcache)[oa] = ya;
                reinterpret_cast<float*>(kcache)[ob] = yb;
            }
        }
    } else if (v_src && p < nq + nk + kv_dim) {
        const int e = p - nq - nk;
        const float y = __ldcg(v_src + (size_t)t * ld + e);
        const long long o = (long long)pos * head_size + (e / head_size) * kv_head_stride + e % head_size;
        if (kv_f16) reinterpret_cast<__half*>(vcache)[o] = __float2half_rn(y);
        else reinterpret_cast<float*>(vcache)[o] = y;
    }
}

// The q/k/v epilogue of a prompt: as rope_kv_store_kernel, one block per token, the angles' sines and cosines once per
// token instead of once per head (they were most of that kernel's time: 511 tokens x 32 heads 23.7 us).
__global__ void prefill_rope_kv_kernel(const float* qkv, int ld, int q_dim, int kv_dim, int head_size, int pos0, const float* __restrict__ theta,
                                       int neox, float* q_out, int ldq, void* kcache, void* vcache, int kv_f16, long long kv_head_stride) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    extern __shared__ float2 rope_cs[];  // [head_size / 2] (cos, sin)
    const int t = blockIdx.x, pos = pos0 + t, hh = head_size >> 1;
    for (int i = threadIdx.x; i < hh; i += blockDim.x) {
        float sn, cs;
        sincosf((float)pos * theta[i], &sn, &cs);
        rope_cs[i] = make_float2(cs, sn);
    }
    __syncthreads();
    const float* row = qkv + (size_t)t * ld;
    // Pairs by (head of q, k and v together, pair in it); a thread's next pair is `dh` heads and `df` pairs on, without a division.  Four pairs' loads
    // before the first store.  (One at a time and divided, 511 tokens x 12288 rows took 22.5 us.)
    const int hq = q_dim / head_size, hk = kv_dim / head_size, heads = hq + 2 * hk;
    const int step = gridDim.y * blockDim.x, dh = step / hh, df = step - dh * hh;
    int head = (int)(blockIdx.y * blockDim.x + threadIdx.x) / hh, fi = (int)(blockIdx.y * blockDim.x + threadIdx.x) - head * hh;
    while (head < heads) {
        float2 v[4];
        int hd[4], f[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            hd[u] = head;
            f[u] = fi;
            if (head < heads) {
                const float* src = row + head * head_size;
                if (neox && head < hq + hk) v[u] = make_float2(__ldcg(src + fi), __ldcg(src + fi + hh));  // the pair's elements lie half a head apart
                else v[u] = __ldcg(reinterpret_cast<const float2*>(src) + fi);                            // neighbours travel together
            }
            head += dh;
            fi += df;
            if (fi >= hh) {
                fi -= hh;
                head++;
            }
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (hd[u] >= heads) break;
            const bool halves = neox && hd[u] < hq + hk;
            const int da = halves ? f[u] : 2 * f[u], db = halves ? f[u] + hh : 2 * f[u] + 1;
            float2 y = v[u];
            if (hd[u] < hq + hk) {
                const float2 w = rope_cs[f[u]];
                y = make_float2(w.x * y.x - w.y * y.y, w.y * y.x + w.x * y.y);
            }
            if (hd[u] < hq) {
                float* o = q_out + (size_t)t * ldq + hd[u] * head_size;
                if (halves) {
                    o[da] = y.x;
                    o[db] = y.y;
                } else {
                    *reinterpret_cast<float2*>(o + da) = y;
                }
            } else {
                const int kvh = hd[u] < hq + hk ? hd[u] - hq : hd[u] - hq - hk;
                const long long o = (long long)pos * head_size + kvh * kv_head_stride;
                void* cache = hd[u] < hq + hk ? kcache : vcache;
                if (kv_f16) {
                    __half* c = reinterpret_cast<__half*>(cache) + o;
                    if (halves) {
                        c[da] = __float2half_rn(y.x);
                        c[db] = __float2half_rn(y.y);
                    } else {
                        *reinterpret_cast<__half2*>(c + da) = __floats2half2_rn(y.x, y.y);
                    }
                } else {
                    float* c = reinterpret_cast<float*>(cache) + o;
                    if (halves) {
                        c[da] = y.x;
                        c[db] = y.y;
                    } else {
                        *reinterpret_cast<float2*>(c + da) = y;
                    }
                }
            }
        }
    }
}

}  // namespace

// ---- host side ------------------------------------------------------------------------------------------------------
// (the sums are laid out per super-block of 256 columns: only formats whose width is a multiple of 256 use them)
static __half* sums_for(const PrefillOperands& o, int K) { return K % 256 == 0 ? o.sum : nullptr; }

int prefill_split_launch(slai_ctx* ctx, const float* x, int ldx, const float* norm_w, float eps, int T, int K, const PrefillOperands& o) {
    return launch_dependent(ctx, prefill_split_kernel, dim3((unsigned)T), 256, 0, ctx->use_pdl, x, ldx, norm_w, eps, K, o.hi, o.lo, sums_for(o, K));
}
int prefill_split_ln_launch(slai_ctx* ctx, const float* x, int ldx, const float* gamma, const float* beta, float eps, int T, int K,
                            const PrefillOperands& o) {
    return launch_dependent(ctx, prefill_split_ln_kernel, dim3((unsigned)T), 256, 0, ctx->use_pdl, x, ldx, gamma, beta, eps, K, o.hi, o.lo,
                            sums_for(o, K));
}
int prefill_gelu_split_launch(slai_ctx* ctx, const float* g, int T, int H, const PrefillOperands& o) {
    return launch_dependent(ctx, prefill_gelu_split_kernel, dim3((H / 4 + 255) / 256, T), 256, 0, ctx->use_pdl, g, H, o.hi, o.lo, sums_for(o, H));
}
int prefill_add_rows_launch(slai_ctx* ctx, float* x, int dim, const float* table, int pos0, int T) {
    return launch_dependent(ctx, prefill_add_rows_kernel, dim3((dim + 255) / 256, T), 256, 0, ctx->use_pdl, x, dim, table, pos0);
}
int prefill_silu_split_launch(slai_ctx* ctx, const float* gate, const float* up, int T, int H, const PrefillOperands& o) {
    return launch_dependent(ctx, prefill_silu_split_kernel, dim3((H / 4 + 255) / 256, T), 256, 0, ctx->use_pdl, gate, up, H, o.hi, o.lo,
                            sums_for(o, H));
}
int prefill_embed_launch(slai_ctx* ctx, float* x, int dim, const int* d_tokens, int T, const float* table, const slai_qmatrix* qtable) {
    prefill_embed_kernel<<<dim3((dim + 255) / 256, T), 256, 0, ctx->stream>>>(x, dim, d_tokens, table, qtable ? qtable->fmt : 0,
                                                                             qtable ? qtable->data : nullptr);
    SLAI_CHECK_CUDA(ctx, cudaGetLastError());
    return SLAI_OK;
}
// Causal attention of prompt tokens pos0 .. pos0 + T - 1 over the caches (which already hold their keys and values).
// Returns SLAI_ERR_UNSUPPORTED_FORMAT for head sizes the kernel does not take (the caller then uses the decode kernel).
bool prefill_attention_supported(int head_size, int kv_f16, const void* kc, const void* vc, long long head_stride) {
    const int esz = kv_f16 ? 2 : 4;
    const uintptr_t bits = reinterpret_cast<uintptr_t>(kc) | reinterpret_cast<uintptr_t>(vc) | (uintptr_t)(head_stride * esz) | (uintptr_t)(head_size * esz);
    return head_size % 8 == 0 && head_size <= 128 * PA_MAXC && (bits & 15) == 0;
}
int prefill_attention_launch(slai_ctx* ctx, const float* q, int q_ld, const void* kc, const void* vc, int kv_f16, long long head_stride, int head_size,
                             int n_heads, int kv_mul, int pos0, int T, float* out, int out_ld) {
    SLAI_REQUIRE(ctx, prefill_attention_supported(head_size, kv_f16, kc, vc, head_stride) && q_ld % 4 == 0 && out_ld % 4 == 0, SLAI_ERR_UNSUPPORTED_FORMAT,
                 "prefill attention: head size %d / alignment not supported", head_size);
    if (kv_f16 && (head_size == 64 || head_size == 128) && q_ld % 2 == 0) {
        // (other heads and f32 caches: the f32 kernel below)
        const size_t sm = (size_t)4 * PM_KT * head_size * 2;
        const int q_tiles = (T + PM_QT - 1) / PM_QT, tiles = (pos0 + T - 1) / PM_KT + 1;
        // CTAs that share a (head, 64 queries): while all of them run side by side (two to an SM) and none is left without a tile for long.
        int ranks = 1;
        while (ranks < 8 && ranks < tiles && (long long)n_heads * q_tiles * ranks * 2 <= 2 * (ctx->sm_count > 0 ? ctx->sm_count : 148)) ranks *= 2;
        static PerDeviceOnce once;
        if (once.need(ctx->device)) {
            SLAI_CHECK_CUDA(ctx, cudaFuncSetAttribute(prefill_attn_mma_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * PM_KT * 128 * 2));
            once.set(ctx->device);
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)n_heads, (unsigned)q_tiles, (unsigned)ranks);
        cfg.blockDim = dim3(PM_THREADS);
        cfg.dynamicSmemBytes = sm;
        cfg.stream = ctx->stream;
        cudaLaunchAttribute at[2];
        int n = 0;
        if (ranks > 1) {
            at[n].id = cudaLaunchAttributeClusterDimension;
            at[n].val.clusterDim.x = at[n].val.clusterDim.y = 1;
            at[n++].val.clusterDim.z = (unsigned)ranks;
        }
        if (ctx->use_pdl) {
            at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            at[n++].val.programmaticStreamSerializationAllowed = 1;
        }
        cfg.attrs = at;
        cfg.numAttrs = n;
        SLAI_CHECK_CUDA(ctx, cudaLaunchKernelEx(&cfg, head_size == 64 ? prefill_attn_mma_kernel<64> : prefill_attn_mma_kernel<128>, q, q_ld, (const __half*)kc,
                                                (const __half*)vc, (long long)head_stride, kv_mul, pos0, T, out, out_ld));
        return SLAI_OK;
    }
    const size_t smem = ((size_t)PA_QT * head_size + (size_t)PA_KT * (head_size + 4) + (size_t)PA_KT * head_size + PA_QT * PA_KT) * 4;
    const dim3 grid((unsigned)n_heads, (unsigned)((T + PA_QT - 1) / PA_QT));
    static PerDeviceOnce attr;
    if (attr.need(ctx->device)) {
        SLAI_CHECK_CUDA(ctx, cudaFuncSetAttribute(prefill_attn_kernel<__half>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024));
        SLAI_CHECK_CUDA(ctx, cudaFuncSetAttribute(prefill_attn_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024));
        attr.set(ctx->device);
    }
    if (kv_f16)
        return launch_dependent(ctx, prefill_attn_kernel<__half>, grid, PA_THREADS, smem, ctx->use_pdl, q, q_ld, (const __half*)kc, (const __half*)vc,
                                head_stride, head_size, kv_mul, pos0, T, out, out_ld);
    return launch_dependent(ctx, prefill_attn_kernel<float>, grid, PA_THREADS, smem, ctx->use_pdl, q, q_ld, (const float*)kc, (const float*)vc, head_stride,
                            head_size, kv_mul, pos0, T, out, out_ld);
}
int prefill_rope_kv_launch(slai_ctx* ctx, const float* qkv, int ld, int q_dim, int kv_dim, int head_size, int pos0, int T,
                           const float* theta, int neox, float* q_out, void* kcache, void* vcache, int kv_f16, long long kv_head_stride) {
    // (few tokens: several blocks each)
    const int pairs = q_dim / 2 + kv_dim, parts = T >= 256 ? 2 : std::min((pairs + 255) / 256, (512 + T - 1) / T);
    return launch_dependent(ctx, prefill_rope_kv_kernel, dim3((unsigned)T, (unsigned)parts), 256, (size_t)head_size * 4, ctx->use_pdl, qkv, ld, q_dim, kv_dim,
                            head_size, pos0, theta, neox, q_out, q_dim, kcache, vcache, kv_f16, kv_head_stride);
}
// One token at the device-side position: q rotated in place, k (and v when given) into the cache.
int rope_kv_store_launch(slai_ctx* ctx, float* q, const float* k, const float* v, int q_dim, int kv_dim, int head_size, const int* d_pos,
                         const float* theta, int neox, void* kcache, void* vcache, int kv_f16, long long kv_head_stride, bool pdl) {
    const int work = q_dim / 2 + kv_dim / 2 + (v ? kv_dim : 0);
    (void)pdl;
    rope_kv_store_kernel<<<dim3((work + 255) / 256, 1), 256, 0, ctx->stream>>>(q, k, v, 0, q_dim, kv_dim, head_size, 0, d_pos, theta, neox, q, q_dim,
                                                                              kcache, vcache, kv_f16, kv_head_stride, 0);
    SLAI_CHECK_CUDA(ctx, cudaGetLastError());
    return SLAI_OK;
}
int rope_kv_store_seqs_launch(slai_ctx* ctx, const float* qkv, int ld, int q_dim, int kv_dim, int head_size, const int* d_pos, int B,
                              const float* theta, int neox, float* q_out, void* kcache, void* vcache, int kv_f16, long long kv_head_stride,
                              long long seq_stride, bool pdl) {
    SLAI_REQUIRE(ctx, seq_stride > 0 && d_pos && B >= 1, SLAI_ERR_INVALID_ARG, "rope: a batch of sequences needs positions and a cache stride");
    const int work = q_dim / 2 + kv_dim / 2 + kv_dim;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((work + 255) / 256, B);
    cfg.blockDim = dim3(256);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    SLAI_CHECK_CUDA(ctx, cudaLaunchKernelEx(&cfg, rope_kv_store_kernel, qkv, qkv + q_dim, qkv + q_dim + kv_dim, ld, q_dim, kv_dim, head_size, 0, d_pos, theta,
                                            neox, q_out, q_dim, kcache, vcache, kv_f16, kv_head_stride, seq_stride));
    return SLAI_OK;
}
