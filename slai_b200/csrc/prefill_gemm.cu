// Y[T x M] = X[T x K] W^T for a prompt of T tokens on the 5th-generation tensor cores, W quantised (tile-major, layout.cuh).
//
// Numerics.  Parity with the sequential path is the contract, and a single fp16 rounding of both operands (4e-4 per GEMM)
// would spend its budget.  The activations are fp16 pairs v = hi + lo (22 bits).  The weights of Q4_K / Q5_K go in as the
// exact integers sc * q, so two products per 16 columns suffice (hi, lo); the super-block scale d multiplies the f32 sums
// of each 256 columns, in registers, and the minimum term is one more product per super-block with its own sums and scale
// dmin.  Q6_K (integers beyond fp16's 11 bits) and Q8_0 (a scale every 32 columns) carry the weights as pairs too: three
// products (hi hi, hi lo, lo hi), about 2^-21 each.  The tensor cores truncate a sum at every step, so whatever the format a sum ends with its
// super-block (256 columns, Q8_0: 128) and the next one is added to it in registers: the error depends neither on K nor on how K is shared out.
// (Q8_0 summed a CTA's whole share of K before.  One product against the sequential pass, before / now: 512 columns, 37 tokens 5.7e-7 / 1.9e-7; 4096
// columns, 400 tokens 8.5e-6 / 3.5e-7.  4 layers of the 7B shape: 37 tokens 579 / 602 us, 511 tokens 2080 / 2360; sums of 256 columns: 603, 2210, 6.2e-7.)
//
// One CTA computes 128 weight rows x NT tokens (<= 128) over its share of K:
//   warp 0      TMA: the activations' hi and lo planes, 64 columns per stage; the sums plane, 16 columns per super-block
//   warp 1      issues tcgen05.mma (kind::f16, M = 128, N = NT, K = 16), commits stages and super-blocks to mbarriers
//   warp 2      bulk copies of the packed tile-step blocks (8 row tiles x one super-block), two or three super-blocks ahead: a
//               few tokens read the matrix from HBM, which takes some 40 KB in flight per SM
//   warps 4-11  packed bytes -> operand rows in tensor memory (prefill_dequant.cuh), one row a thread
//   warps 12-19 sums of a super-block out of tensor memory (two buffers) into registers, times d (and dmin), while the tensor
//               cores work on the next one.  (Done by warps 4-11 between two stages, this put a super-block's drain and the
//               next stages' operands one after the other: 1000 cycles per stage whatever the number of tokens.)
// CTAs are persistent: a tile's sums are stored by warps 12-19 while the other warps are in the next tile.  A CTA (pair) takes whole tiles, or an equal share
// of the launch's super-blocks that begins and ends inside tiles: the CTA with a tile's first super-blocks adds the sums that the ones behind it
// left in memory, which was the first thing they did.  (It waits for CTAs of its own launch, all of which start without waiting for any other; the wait is bounded.)
// Few tokens leave most SMs without a tile (4096 rows x 37 tokens: 32 tiles): there K is split over a cluster of up to 8
// CTAs, whose sums meet through distributed shared memory in rank order (deterministic, no second launch).
//
// What bounds it: from some 200 tokens on power (the clock falls to 1.6 GHz with the tensor cores 63 % busy; 511 tokens, gate and up: 1180 TFLOP/s
// executed, where cuBLAS keeps 1375); with few tokens the chain of a stage through operand writer, product and commit (some 620 cycles for products of
// 200), and 8 us of start and end a launch.  us per product of the 7B shape, Q4_K (ncu, serialised: the power limit is not reached): 37 tokens q/k/v 26, o 16, gate and
// up 35, down 25; 511 tokens 91, 40, 151, 80.
// Every wait is bounded (bounded_wait): `wait_limit` polls, after which the error flag is raised, then LAST_POLLS more, because what it waits for is this CTA's
// (pair's) own work and copies, which have to land before the CTA ends.  Only a thread whose last polls ran out too goes on without: it arrives on nothing and
// requests nothing from then on, so that no barrier completes a phase it has not reached.  Whoever requested copies or products waits for
// the last of them at its end.
#include <math.h>

#include <algorithm>

#include <cuda.h>

#include "common.cuh"
#include "prefill_dequant.cuh"

namespace {

constexpr int PG_THREADS = 640;
constexpr int PG_BM = 128, PG_BK = 64;          // weight rows per CTA, columns per stage (one 128-byte swizzle row of fp16)
constexpr int PG_MAX_NT = 128;
constexpr int PG_MAX_CTAS = CNT_PROMPT_FLAG_WORDS;
constexpr int PG_MAX_STAGES = 6, PG_MAX_PACK = 3, PG_MAX_KS = 8;
constexpr int PG_A_COLS = PG_BK / 2;            // tensor-memory columns of one operand plane of a stage
constexpr int PG_SMEM_LIMIT = 227 * 1024 - 512; // the barriers are static
constexpr unsigned int PART_POLLS = 1u << 14;   // fewest polls for another CTA's sums: some 10 ms, its whole work is a few

struct PgSeg {
    const uint8_t* w;
    float* out;
    const float* bias;
    int rows, tile0;  // logical rows; first 128-row tile in the launch's tile space
};
struct PgParams {
    PgSeg seg[3];
    int nseg;
    long long tile_bytes;  // bytes of one 16-row tile (all K steps)
    int nch;               // packed blocks (super-blocks) along K
    int T, NT, NTP;        // tokens, tokens per tile, the same rounded up to a power of two (tensor-memory columns)
    int ldo;
    const float* resid;    // optional [T][ldr]: out = resid + y (may alias out)
    int ldr;
    int n_tiles, tiles;    // token tiles, all tiles (token tiles fastest: neighbours share the weights in L2)
    int ks;                // CTAs of a cluster that share K
    int shared;            // CTAs have equal shares of the super-blocks (else whole tiles)
    float* part;           // [CTA][tokens of a tile][128]: sums of a tile that another CTA finishes
    unsigned int* flags;   // [CTA]: `seq` when they are there
    unsigned int seq;      // of this launch
    int stages, packs;     // operand stages, packed blocks in flight
    unsigned int* err_flag;
    unsigned int wait_limit;
};

// ---- PTX wrappers ---------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t a, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t a) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t a, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(bytes) : "memory");
}
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait(uint32_t a, uint32_t parity, unsigned int& limit, unsigned int* err_flag) {
    return bounded_wait<CLUSTER, true, 5>(a, parity, limit, err_flag);
}
__device__ __forceinline__ uint32_t map_rank(uint32_t a, uint32_t rank) {  // the same shared-memory address in another CTA of the cluster
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
// Arrive on the barrier of the CTA that issues the products (a pair's first).  Default semantics (release at CTA scope): what the
// arrival announces is read by the tensor core out of the writer's own shared memory, and the writer's proxy fence comes first; a
// release at cluster scope held every operand writer for some 600 cycles per arrival.
template <bool PAIR>
__device__ __forceinline__ void arrive_issuer(uint32_t a) {
    if (PAIR) asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(map_rank(a, 0)) : "memory");
    else mbar_arrive(a);
}
// Box at (x, y) into this CTA's shared memory; the bytes count on the issuing CTA's barrier.
template <bool PAIR>
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t mbar) {
    if (PAIR)
        asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
                     "l"(map), "r"(map_rank(mbar, 0)), "r"(x), "r"(y)
                     : "memory");
    else
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
                     "l"(map), "r"(mbar), "r"(x), "r"(y)
                     : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t mbar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(mbar)
                 : "memory");
}
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// Shared-memory matrix descriptor of a K-major operand tile: start address / 16 in bits 0-13, leading offset (unused with a
// swizzle of the row length) 1 in bits 16-29, stride between 8-row groups / 16 in bits 32-45, descriptor version 1 in bits
// 46-47, swizzle mode in bits 61-63 (2: rows of 128 bytes, 6: rows of 32 bytes).
__device__ __forceinline__ uint64_t desc128(uint32_t a) {
    return (uint64_t)((a >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ uint64_t desc32(uint32_t a) {
    return (uint64_t)((a >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(256 >> 4) << 32) | (1ull << 46) | (6ull << 61);
}
// Instruction descriptor, kind::f16: f32 accumulator (bits 4-5 = 1), A and B fp16 (0), both K-major (bits 15, 16 = 0),
// N / 8 in bits 17-22, M / 16 in bits 24-28.
__device__ __forceinline__ uint32_t umma_idesc(int m, int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24); }
template <bool PAIR>
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    if (PAIR)
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
            "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
            "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
            : "memory");
}
// The same with A in tensor memory: row = lane, two columns of the operand to a word.
template <bool PAIR>
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    if (PAIR)
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
            "r"(tmem_a), "l"(b), "r"(idesc), "r"(accumulate)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
            "r"(tmem_a), "l"(b), "r"(idesc), "r"(accumulate)
            : "memory");
}
// Arrives on the barrier (a pair: on both CTAs') when everything issued so far has completed.
template <bool PAIR>
__device__ __forceinline__ void umma_commit(uint32_t mbar) {
    if (PAIR)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(mbar), "h"((unsigned short)3)
                     : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}
// ... on this CTA's barrier alone.
template <bool PAIR>
__device__ __forceinline__ void umma_commit_here(uint32_t mbar) {
    if (PAIR) asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
    else umma_commit<false>(mbar);
}
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
                 "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ float ld_cluster(uint32_t local, uint32_t rank) {
    uint32_t a;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Dynamic shared memory, from a 1024-byte boundary: operand planes of the activations, the operands of the
// minimum term (two super-blocks), row scales (four super-blocks), packed blocks.
struct PgLayout {
    uint32_t b, amin, bmin, scale, pack, total;
};
template <int FMT>
__host__ __device__ inline PgLayout pg_layout(int NB, int stages, int packs) {
    using F = pfq::Fmt<FMT>;
    PgLayout L;
    L.b = 0;
    L.amin = L.b + (uint32_t)stages * 2 * NB * PG_BK * 2;
    L.bmin = L.amin + (F::MIN ? 2 * PG_BM * 32 : 0);
    L.scale = L.bmin + (F::MIN ? 2 * (uint32_t)NB * 32 : 0);
    L.pack = L.scale + 4 * PG_BM * 4;
    L.total = L.pack + (uint32_t)packs * 8 * F::STEP;
    return L;
}

// PG_PLAIN: one CTA, a product with each of the two activation planes.  PG_MERGED (at most 64 tokens): the planes lie one behind the
// other and are one operand of twice the width, with sums of their own.  PG_PAIR: two CTAs of a cluster hold 128 rows each and
// half of the tokens' operands each, one of them issues products of 256 rows (cta_group::2).
enum { PG_PLAIN = 0, PG_MERGED = 1, PG_PAIR = 2 };

template <int FMT, int MODE>
__global__ void __launch_bounds__(PG_THREADS, 1)
prefill_gemm_kernel(const __grid_constant__ PgParams P, const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo,
                    const __grid_constant__ CUtensorMap map_sum) {
    using F = pfq::Fmt<FMT>;
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
    constexpr bool PAIR = MODE == PG_PAIR, MERGED = MODE == PG_MERGED;
    const int NB = PAIR ? P.NT / 2 : P.NT;  // tokens whose operands this CTA holds
    const PgLayout L = pg_layout<FMT>(NB, P.stages, P.packs);
    const int NT = P.NT, S = P.stages, PK = P.packs;
    const uint32_t b_bytes = (uint32_t)NB * PG_BK * 2;  // one activation plane of a stage
    __shared__ __align__(8) unsigned long long bars[2 * PG_MAX_STAGES + 2 * PG_MAX_PACK + 12];
    __shared__ uint32_t tmem_slot;
    const uint32_t sb = smem_u32(smem);
    const uint32_t full = smem_u32(bars), empty = full + 8 * PG_MAX_STAGES,
                   pk_full = empty + 8 * PG_MAX_STAGES, pk_empty = pk_full + 8 * PG_MAX_PACK, dfull = pk_empty + 8 * PG_MAX_PACK,
                   dempty = dfull + 16, bmin_full = dempty + 16, sc_full = bmin_full + 16, mempty = sc_full + 32, all_done = mempty + 8;

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;  // (warp: uniform for the compiler too)
    const int pr = PAIR ? (int)(blockIdx.x & 1) : 0;  // rank in the pair
    // This CTA's (pair's) super-blocks of the launch, in order of tiles: whole tiles, or an equal share of all of them, from
    // somewhere in a tile to somewhere in another.
    const int rank = !PAIR && P.ks > 1 ? (int)(blockIdx.x % P.ks) : 0, me = (int)blockIdx.x / (PAIR ? 2 : P.ks), many = (int)gridDim.x / (PAIR ? 2 : P.ks);
    auto share = [&](int i) { return P.shared ? (int)((long long)P.tiles * P.nch * i / many) : (int)((long long)P.tiles * i / many) * P.nch; };
    const int u_lo = P.ks > 1 ? me * P.nch + (int)((long long)P.nch * rank / P.ks) : share(me);
    const int u_hi = P.ks > 1 ? me * P.nch + (int)((long long)P.nch * (rank + 1) / P.ks) : share(me + 1);
    // ... and the part of them that is of one tile: super-blocks c0 .. c0 + nc - 1 of it
    struct Part {
        int tile, c0, nc;
    };
    auto part_at = [&](int un) {
        Part q;
        q.tile = un / P.nch;
        q.c0 = un - q.tile * P.nch;
        q.nc = min(P.nch - q.c0, u_hi - un);
        return q;
    };
    // a tile's matrix, first row in it and first token
    auto tile_of = [&](int tile, PgSeg& sg, int& m0, int& n0) {
        const int mt = tile / P.n_tiles;
        n0 = (tile - mt * P.n_tiles) * NT;
        sg = P.seg[0];
        if (P.nseg > 1 && mt >= P.seg[1].tile0) sg = P.seg[1];
        if (P.nseg > 2 && mt >= P.seg[2].tile0) sg = P.seg[2];
        m0 = PAIR ? (mt - sg.tile0) * 2 * PG_BM + pr * PG_BM : (mt - sg.tile0) * PG_BM;
    };

    if (tid == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(full + 8 * s, (PAIR ? 16 : 8) + 1);  // the operand-writing warps and the activations' request (and its bytes)
            mbar_init(empty + 8 * s, 1);
        }
        for (int s = 0; s < PK; s++) {
            mbar_init(pk_full + 8 * s, 1);
            mbar_init(pk_empty + 8 * s, 8);
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(dfull + 8 * s, 1);
            mbar_init(dempty + 8 * s, PAIR ? 16 : 8);
            mbar_init(bmin_full + 8 * s, 1);
        }
        for (int s = 0; s < 4; s++) mbar_init(sc_full + 8 * s, 8);
        mbar_init(mempty, PAIR ? 16 : 8);
        mbar_init(all_done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async();
    }
    // tensor memory: two buffers of sums, the minimum term, the weights' operand planes of all stages
    const int DS = MERGED ? 2 * P.NTP : P.NTP;
    const uint32_t TA = 2 * DS + (F::MIN ? P.NTP : 0);
    int ncols = 32;
    while (ncols < (int)TA + S * F::PLANES * PG_A_COLS) ncols <<= 1;
    if (warp == 1) {  // the MMA warp owns the tensor-memory allocation
        if (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(ncols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(ncols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (PAIR) cluster_sync();  // the other CTA's barriers are ready
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    unsigned int limit = P.wait_limit;
    // Dependent launch: the weights' warps fill their rings while the kernel before this one ends, and wait for its end before their first
    // wait on a slot that has been used: its consumers cannot start sooner, and that time is not this kernel's to count (a
    // bounded wait in its place gave up on a healthy predecessor at up to 1024 rounds, where 96 are enough now).  Everything else waits here.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (warp < 2 || warp >= 12) griddep_wait();
    // readers of the sums (warps 12-19): 32 rows each, every other group of 16 tokens
    constexpr int NG = MERGED ? 2 : 4;
    float acc[NG][16];
    const int quad = warp & 3, half = (warp - 12) >> 2;

    if (warp == 0) {
        // ---- activations: the whole warp walks the loop and one elected lane issues, as for the products (issued by lane 0 of a diverged warp, a
        // copy took some 200 cycles: more than half of the tensor cores' waiting was for them) ----
        int slot = 0, issued = 0, gc = 0;  // gc: super-blocks so far
        uint32_t ph = 0;
        bool ok = true;
        for (int un = u_lo; un < u_hi && ok;) {
            const Part q = part_at(un);
            const int c0 = q.c0, nc = q.nc;
            un += nc;
            PgSeg sg;
            int m0, n0;
            tile_of(q.tile, sg, m0, n0);
            for (int c = 0; c < nc && ok; c++, gc++) {
                if (F::MIN) {
                    const int buf = gc & 1;
                    if (gc >= 2 && !(ok = __all_sync(0xffffffffu, mbar_wait(dfull + 8 * buf, ((gc >> 1) - 1) & 1, limit, P.err_flag)))) break;
                    if (elect_one()) {
                        if (pr == 0) mbar_expect_tx(bmin_full + 8 * buf, (uint32_t)NT * 32);
                        tma_load_2d<PAIR>(sb + L.bmin + buf * NB * 32, &map_sum, 16 * (c0 + c), n0 + pr * NB, bmin_full + 8 * buf);
                    }
                    __syncwarp();
                }
                for (int st = 0; st < F::STAGES; st++) {
                    if (!(ok = __all_sync(0xffffffffu, mbar_wait(empty + 8 * slot, ph ^ 1, limit, P.err_flag)))) break;
                    const int x = ((c0 + c) * F::STAGES + st) * PG_BK;
                    if (elect_one()) {
                        if (pr == 0) mbar_expect_tx(full + 8 * slot, (PAIR ? 4 : 2) * b_bytes);
                        tma_load_2d<PAIR>(sb + L.b + slot * 2 * b_bytes, &map_hi, x, n0 + pr * NB, full + 8 * slot);
                        tma_load_2d<PAIR>(sb + L.b + slot * 2 * b_bytes + b_bytes, &map_lo, x, n0 + pr * NB, full + 8 * slot);
                    }
                    __syncwarp();
                    issued++;
                    if (++slot == S) {
                        slot = 0;
                        ph ^= 1;
                    }
                }
            }
        }
        if (pr == 0) {  // the last copies land before the CTA (the pair) ends
            limit = LAST_POLLS;
            for (int i = max(0, issued - S); i < issued; i++) mbar_wait(full + 8 * (i % S), (i / S) & 1, limit, P.err_flag);
            limit = LAST_POLLS;
            for (int i = max(0, gc - 2); F::MIN && i < gc; i++) mbar_wait(bmin_full + 8 * (i & 1), (i >> 1) & 1, limit, P.err_flag);
        }
    } else if (warp == 1) {
        if (pr == 0) {
        // ---- tensor cores: the whole warp walks the loop, so that descriptors live in uniform registers, one lane issues ----
        const uint32_t idesc = umma_idesc(PAIR ? 2 * PG_BM : PG_BM, NT), idesc2 = umma_idesc(PG_BM, 2 * NT);
        const uint64_t db0 = desc128(sb + L.b);
        int slot = 0, u = 0;  // u: super-blocks so far, their sums alternately in two buffers
        uint32_t ph = 0;
        for (int un = u_lo, nc; un < u_hi; un += nc) {
        nc = part_at(un).nc;
        for (int c = 0; c < nc; c++, u++) {
            const int buf = u & 1;
            const uint32_t d = tmem + buf * DS;
            if (u >= 2) mbar_wait<PAIR>(dempty + 8 * buf, ((u >> 1) - 1) & 1, limit, P.err_flag);
            for (int st = 0; st < F::STAGES; st++) {
                mbar_wait<PAIR>(full + 8 * slot, ph, limit, P.err_flag);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                __syncwarp();
                // 16 elements = 32 bytes further along the swizzled row: 2 in the descriptor's units of 16 bytes
                const uint32_t ah = tmem + TA + slot * F::PLANES * PG_A_COLS;
                const uint64_t dbh = db0 + (uint64_t)(slot * 2 * (b_bytes >> 4));
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < PG_BK / 16; kk++) {
                        const bool first = kk == 0 && st == 0;
                        if (MERGED) {
                            umma_f16_ts<PAIR>(d, ah + 8 * kk, dbh + 2 * kk, idesc2, first ? 0u : 1u);
                        } else {
                            umma_f16_ts<PAIR>(d, ah + 8 * kk, dbh + 2 * kk, idesc, first ? 0u : 1u);
                            umma_f16_ts<PAIR>(d, ah + 8 * kk, dbh + (b_bytes >> 4) + 2 * kk, idesc, 1u);
                        }
                        if (F::PLANES == 2) umma_f16_ts<PAIR>(d, ah + PG_A_COLS + 8 * kk, dbh + 2 * kk, idesc, 1u);
                    }
                    if (limit) umma_commit<PAIR>(empty + 8 * slot);  // (behind the products: in front of them the test costs 20 cycles a stage)
                }
                __syncwarp();
                if (++slot == S) {
                    slot = 0;
                    ph ^= 1;
                }
            }
            if (F::MIN) {
                // (one buffer: read out for the super-block before)
                if (PAIR && u >= 1) mbar_wait<PAIR>(mempty, (u - 1) & 1, limit, P.err_flag);
                if (!PAIR && u >= 1) mbar_wait<PAIR>(dempty + 8 * (buf ^ 1), ((u - 1) >> 1) & 1, limit, P.err_flag);
                mbar_wait<PAIR>(bmin_full + 8 * buf, (u >> 1) & 1, limit, P.err_flag);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                __syncwarp();
            }
            if (elect_one()) {
                if (F::MIN)
                    umma_f16<PAIR>(tmem + 2 * DS, desc32(sb + L.amin + buf * PG_BM * 32), desc32(sb + L.bmin + buf * NB * 32), idesc, 0u);
                if (limit) umma_commit<PAIR>(dfull + 8 * buf);
            }
            __syncwarp();
        }
        }
        if (elect_one()) umma_commit_here<PAIR>(all_done);  // no product is under way when the CTA ends
        limit = LAST_POLLS;
        mbar_wait<PAIR>(all_done, 0, limit, P.err_flag);
        __syncwarp();
        }
    } else if (warp == 2) {
        // ---- packed weights ----
        int slot = 0, issued = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int un = u_lo; un < u_hi && ok;) {
            const Part q = part_at(un);
            const int c0 = q.c0, nc = q.nc;
            un += nc;
            PgSeg sg;
            int m0, n0;
            tile_of(q.tile, sg, m0, n0);
            const int nt = max(0, min(8, (sg.rows - m0 + 15) >> 4));  // 16-row tiles that exist
            const uint8_t* src = sg.w + (long long)(m0 >> 4) * P.tile_bytes + (long long)c0 * F::STEP;
            for (int c = 0; c < nc; c++) {
                if (issued == PK) griddep_wait();
                if (!(ok = __all_sync(0xffffffffu, mbar_wait(pk_empty + 8 * slot, ph ^ 1, limit, P.err_flag)))) break;
                if (elect_one()) {
                    fence_async();  // the warps' reads of the block before come before the copy's writes
                    mbar_expect_tx(pk_full + 8 * slot, (uint32_t)nt * F::STEP);
                    for (int i = 0; i < nt; i++)
                        bulk_load(sb + L.pack + (slot * 8 + i) * F::STEP, src + i * P.tile_bytes + (long long)c * F::STEP, F::STEP, pk_full + 8 * slot);
                }
                __syncwarp();
                issued++;
                if (++slot == PK) {
                    slot = 0;
                    ph ^= 1;
                }
            }
        }
        limit = LAST_POLLS;
        for (int i = max(0, issued - PK); i < issued; i++) mbar_wait(pk_full + 8 * (i % PK), (i / PK) & 1, limit, P.err_flag);  // the last copies have landed
    } else if (warp >= 4 && warp < 12) {
        // ---- weights into operand rows in tensor memory ----
        // Thread = row: a warp reaches the 32 lanes of its quarter; the two warps of a quarter share the columns.  (In shared memory the rows cost, per
        // stage and SM, 128 cycles to write and 256 to read for the two products, of 820 the stage took.)
        // (Sixteen of these warps, every other two stages each: no faster at 37 tokens, 35.5 for 34.4 us.)
        const int q4 = warp & 3, w8 = 2 * q4 + (lane >> 4), r16 = lane & 15, r = 32 * q4 + lane;
        const int part = (warp - 4) >> 2;
        const uint32_t mine = tmem + TA + ((uint32_t)(32 * q4) << 16) + (FMT == SLAI_FMT_Q8_0 ? 16 : 8) * part;
        uint32_t* scales = reinterpret_cast<uint32_t*>(smem + L.scale);
        int slot = 0, ps = 0;
        uint32_t ph = 0, pph = 0;
        bool behind = false;
        for (int c = 0; c < u_hi - u_lo; c++) {  // super-blocks
            mbar_wait(pk_full + 8 * ps, pph, limit, P.err_flag);
            const unsigned char* blk = smem + L.pack + (ps * 8 + w8) * F::STEP;
            if (F::MIN) {
                if (c >= 2) mbar_wait(dfull + 8 * (c & 1), ((c >> 1) - 1) & 1, limit, P.err_flag);  // c - 2's product has read its operand
                pfq::min_row(blk, r16, r, part, smem + L.amin + (c & 1) * PG_BM * 32);
            }
            if (F::SCALED) {
                // (four super-blocks of scales: stages run at most one and a half ahead of the products, those at most two ahead of
                // the readers)
                if (part == 0) scales[(c & 3) * PG_BM + r] = pfq::row_scale<FMT>(blk, r16);
                __syncwarp();
                if (lane == 0 && limit) mbar_arrive(sc_full + 8 * (c & 3));
            }
            // two stages at a time: a warp's way through one is a chain of latencies (load, arithmetic, store, arrive)
#pragma unroll
            for (int st = 0; st < F::STAGES; st += 2) {
                const int slot0 = slot, slot1 = slot + 1 == S ? 0 : slot + 1;
                const uint32_t ph0 = ph, ph1 = slot + 1 == S ? ph ^ 1 : ph;
                slot += 2;
                if (slot >= S) {
                    slot -= S;
                    ph ^= 1;
                }
                pfq::Packed pk[2];
                pfq::fetch<FMT>(blk, r16, part, st, pk[0]);
                pfq::fetch<FMT>(blk, r16, part, st + 1, pk[1]);
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const uint32_t p = k ? ph1 : ph0;
                    if (p && !behind) {
                        griddep_wait();
                        behind = true;
                    }
                    mbar_wait(empty + 8 * (k ? slot1 : slot0), p ^ 1, limit, P.err_flag);
                    __syncwarp();
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    uint32_t hi[16], lo[16];
                    pfq::make<FMT>(pk[k], st + k, hi, lo);
                    const uint32_t a = mine + (k ? slot1 : slot0) * F::PLANES * PG_A_COLS;
                    tmem_st8(a, hi);
                    tmem_st8(a + (FMT == SLAI_FMT_Q8_0 ? 8 : 16), hi + 8);
                    if (F::PLANES == 2) {
                        tmem_st8(a + PG_A_COLS, lo);
                        tmem_st8(a + PG_A_COLS + (FMT == SLAI_FMT_Q8_0 ? 8 : 16), lo + 8);
                    }
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                if (F::MIN && st == 0) fence_async();  // the minimum term's operand comes before the tensor core's reads
                __syncwarp();
                if (lane == 0 && limit) {
                    arrive_issuer<PAIR>(full + 8 * slot0);
                    arrive_issuer<PAIR>(full + 8 * slot1);
                    if (st == F::STAGES - 2) mbar_arrive(pk_empty + 8 * ps);
                }
            }
            if (++ps == PK) {
                ps = 0;
                pph ^= 1;
            }
        }
    } else if (warp >= 12) {
        // ---- sums out of tensor memory ----
        const uint32_t* scales = reinterpret_cast<const uint32_t*>(smem + L.scale);
        int u = 0;
        unsigned int part_polls = max(P.wait_limit, PART_POLLS);
        for (int un = u_lo; un < u_hi;) {
            const Part q = part_at(un);
            const int nc = q.nc;
            un += nc;
#pragma unroll
            for (int i = 0; i < NG; i++)
#pragma unroll
                for (int j = 0; j < 16; j++) acc[i][j] = 0.f;
            for (int c = 0; c < nc; c++, u++) {
                const int buf = u & 1;
                float d = 1.f, mn = 0.f;
                if (F::SCALED) {
                    mbar_wait(sc_full + 8 * (u & 3), (u >> 2) & 1, limit, P.err_flag);
                    const uint32_t dd = scales[(u & 3) * PG_BM + 32 * quad + lane];
                    d = __half2float(__ushort_as_half((unsigned short)(dd & 0xFFFFu)));
                    if (F::MIN) mn = -32.f * __half2float(__ushort_as_half((unsigned short)(dd >> 16)));  // the sums plane holds sums / 32
                }
                mbar_wait(dfull + 8 * buf, (u >> 1) & 1, limit, P.err_flag);
                __syncwarp();
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t tq = tmem + ((uint32_t)(32 * quad) << 16), t0 = tq + buf * DS;
                if (PAIR && F::MIN) {  // first, because it has one buffer (511 tokens, gate and up 156 -> 151 us)
#pragma unroll
                    for (int i = 0; i < NG; i++) {
                        const int col = 16 * (2 * i + half);
                        if (col < NT) {
                            uint32_t v[16];
                            tmem_ld16(tq + 2 * DS + col, v);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                            for (int j = 0; j < 16; j++) acc[i][j] = fmaf(mn, __uint_as_float(v[j]), acc[i][j]);
                        }
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0 && limit) arrive_issuer<PAIR>(mempty);
                }
#pragma unroll
                for (int i = 0; i < NG; i++) {
                    const int col = 16 * (2 * i + half);
                    if (col < NT) {
                        uint32_t v[16], w[16], z[16];  // (few tokens: all of a group's loads, then one wait)
                        tmem_ld16(t0 + col, v);
                        if (MERGED) tmem_ld16(t0 + NT + col, w);
                        if (MERGED && F::MIN) tmem_ld16(tq + 2 * DS + col, z);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int j = 0; j < 16; j++) acc[i][j] = F::SCALED ? fmaf(d, __uint_as_float(v[j]), acc[i][j]) : acc[i][j] + __uint_as_float(v[j]);
                        if (MERGED) {
#pragma unroll
                            for (int j = 0; j < 16; j++) acc[i][j] = F::SCALED ? fmaf(d, __uint_as_float(w[j]), acc[i][j]) : acc[i][j] + __uint_as_float(w[j]);
                        }
                        if (!PAIR && F::MIN) {
                            if (!MERGED) {
                                tmem_ld16(tq + 2 * DS + col, z);
                                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                            }
#pragma unroll
                            for (int j = 0; j < 16; j++) acc[i][j] = fmaf(mn, __uint_as_float(z[j]), acc[i][j]);
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0 && limit) arrive_issuer<PAIR>(dempty + 8 * buf);
            }
            if (!PAIR && P.ks > 1) break;  // one tile per cluster, stored below
            const size_t slot_floats = (size_t)NT * PG_BM;
            if (q.c0 > 0) {  // the tile's first super-blocks, and its sums, are another CTA's
                float* dst = P.part + blockIdx.x * slot_floats + 32 * quad + lane;
#pragma unroll
                for (int i = 0; i < NG; i++)
#pragma unroll
                    for (int j = 0; j < 16; j++)
                        if (16 * (2 * i + half) < NT) __stcg(dst + (16 * (2 * i + half) + j) * PG_BM, acc[i][j]);
                __threadfence();
                asm volatile("bar.sync 1, 256;" ::: "memory");  // (warps 12-19)
                if (warp == 12 && lane == 0) asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(P.flags + blockIdx.x), "r"(P.seq) : "memory");
                continue;
            }
            // The rest of the tile is the first work of the CTAs that follow, and done by now (or they end where this one does): added in order.
            for (int p = me + 1; q.c0 + nc < P.nch && p < many && share(p) < (q.tile + 1) * P.nch; p++) {
                const int cta = PAIR ? 2 * p + pr : p;
                bool there = false;
                for (unsigned int i = 0; i < part_polls && !there; i++) {
                    unsigned int f;
                    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(f) : "l"(P.flags + cta) : "memory");
                    there = f == P.seq;
                    if (!there && i > 64) __nanosleep(40);
                }
                if (!there) {  // nothing of this CTA's own depends on it: on without those sums
                    atomicExch(P.err_flag, 5u);
                    part_polls = 1;
                }
                __syncwarp();
                const float* src = P.part + cta * slot_floats + 32 * quad + lane;
#pragma unroll
                for (int i = 0; i < NG; i++)
                    if (16 * (2 * i + half) < NT) {
                        float x[16];
#pragma unroll
                        for (int j = 0; j < 16; j++) x[j] = __ldcg(src + (16 * (2 * i + half) + j) * PG_BM);
#pragma unroll
                        for (int j = 0; j < 16; j++) acc[i][j] += x[j];
                    }
            }
            PgSeg sg;
            int m0, n0;
            tile_of(q.tile, sg, m0, n0);
            const int row = m0 + 32 * quad + lane;
            if (row < sg.rows) {
                const float bias = sg.bias ? sg.bias[row] : 0.f;
#pragma unroll
                for (int i = 0; i < NG; i++) {
                    const int t0 = n0 + 16 * (2 * i + half);
                    if (16 * (2 * i + half) < NT && t0 < P.T) {
                        float res[16];  // all residuals on their way before the first store (the output may be the residual)
#pragma unroll
                        for (int j = 0; j < 16; j++) res[j] = P.resid && t0 + j < P.T ? __ldcg(P.resid + (size_t)(t0 + j) * P.ldr + row) : 0.f;
#pragma unroll
                        for (int j = 0; j < 16; j++)
                            if (t0 + j < P.T) sg.out[(size_t)(t0 + j) * P.ldo + row] = P.resid ? res[j] + (acc[i][j] + bias) : acc[i][j] + bias;
                    }
                }
            }
        }
    }

    // ---- K split over a cluster ----
    __syncwarp();
    if (!PAIR && P.ks > 1) {
        griddep_wait();
        PgSeg sg;
        int m0, n0;
        tile_of(me, sg, m0, n0);
        // every CTA leaves its sums [token][row] in its own shared memory (the operand planes are free: all products are done)
        float* red = reinterpret_cast<float*>(smem);
        if (warp >= 12) {
#pragma unroll
            for (int i = 0; i < NG; i++)
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const int col = 16 * (2 * i + half) + j;
                    if (col < NT) red[col * PG_BM + 32 * quad + lane] = acc[i][j];
                }
        }
        cluster_sync();
        const int lo = NT * rank / P.ks * PG_BM, hi = NT * (rank + 1) / P.ks * PG_BM;  // this CTA adds and stores a share of the tokens
        for (int i = lo + tid; i < hi; i += PG_THREADS) {
            const int t = n0 + i / PG_BM, m = m0 + i % PG_BM;
            float y = 0.f;
            for (int z = 0; z < P.ks; z++) y += ld_cluster(sb + 4 * i, z);
            if (m < sg.rows && t < P.T) {
                if (sg.bias) y += sg.bias[m];
                if (P.resid) y = P.resid[(size_t)t * P.ldr + m] + y;
                sg.out[(size_t)t * P.ldo + m] = y;
            }
        }
        cluster_sync();  // no CTA leaves while another reads its sums
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (PAIR) cluster_sync();  // neither CTA leaves while the other reads its operands or arrives on its barriers
    if (warp == 1) {
        if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
    }
}

// ---- host side ------------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// fp16 plane [rows][cols] row-major -> boxes of `box_cols` x `box_rows`, swizzled over rows of 128 (64 columns) or 32 bytes (16).
int make_plane_map(slai_ctx* ctx, CUtensorMap* map, const __half* base, int rows, int cols, int box_cols, int box_rows) {
    EncodeTiledFn enc = encode_tiled();
    SLAI_REQUIRE(ctx, enc, SLAI_ERR_CUDA, "prefill: the driver does not provide cuTensorMapEncodeTiled");
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half*>(base), dims, strides, box, elem,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, box_cols == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_32B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    SLAI_REQUIRE(ctx, r == CUDA_SUCCESS, SLAI_ERR_CUDA, "prefill: cuTensorMapEncodeTiled failed (%d)", (int)r);
    return SLAI_OK;
}

template <int FMT, int MODE>
int launch_mode(slai_ctx* ctx, PgParams& P, const CUtensorMap& hi, const CUtensorMap& lo, const CUtensorMap& sum) {
    const int NB = MODE == PG_PAIR ? P.NT / 2 : P.NT;
    const int cluster = MODE == PG_PAIR ? 2 : P.ks, rows = MODE == PG_PAIR ? 2 * PG_BM : PG_BM;
    int tiles = 0;
    for (int i = 0; i < P.nseg; i++) {
        P.seg[i].tile0 = tiles;
        tiles += (P.seg[i].rows + rows - 1) / rows;
    }
    P.tiles = tiles * P.n_tiles;
    // Packed blocks in flight first (three if two stages still fit beside them), then as many operand stages as fit.
    P.packs = pg_layout<FMT>(NB, 4, 3).total <= PG_SMEM_LIMIT - 1024 ? 3 : 2;
    P.stages = 2;
    const int sums = (MODE == PG_MERGED ? 4 : 2) * P.NTP + (pfq::Fmt<FMT>::MIN ? P.NTP : 0);  // tensor-memory columns, of 512
    while (P.stages < PG_MAX_STAGES && pg_layout<FMT>(NB, P.stages + 1, P.packs).total <= PG_SMEM_LIMIT - 1024 &&
           sums + (P.stages + 1) * pfq::Fmt<FMT>::PLANES * PG_A_COLS <= 512)
        P.stages++;
    const size_t smem = pg_layout<FMT>(NB, P.stages, P.packs).total + 1024;
    auto kern = prefill_gemm_kernel<FMT, MODE>;
    static PerDeviceOnce attr;  // per instantiation
    if (attr.need(ctx->device)) {
        SLAI_CHECK_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PG_SMEM_LIMIT));
        attr.set(ctx->device);
    }
    const int sms = std::min(ctx->sm_count > 0 ? ctx->sm_count : 148, PG_MAX_CTAS);
    cudaLaunchConfig_t cfg = {};
    const int grid = MODE != PG_PAIR && P.ks > 1 ? P.tiles * P.ks
                                                 : std::min((int)std::min((long long)P.tiles * (P.shared ? P.nch : 1), 1ll << 20), sms / cluster) * cluster;
    cfg.gridDim = dim3((unsigned)grid);
    if (P.shared) {
        const int rc = ensure_scratch(ctx, (size_t)grid * P.NT * PG_BM * sizeof(float));
        if (rc) return rc;
        P.part = reinterpret_cast<float*>(ctx->d_scratch);
        P.flags = ctx->d_counters + CNT_PROMPT_FLAGS;
        P.seq = ++ctx->prompt_seq ? ctx->prompt_seq : ++ctx->prompt_seq;  // (0 is what the flags hold at first)
    }
    cfg.blockDim = dim3(PG_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[2];
    int n = 0;
    if (cluster > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = (unsigned)cluster;
        at[n].val.clusterDim.y = 1;
        at[n++].val.clusterDim.z = 1;
    }
    if (ctx->use_pdl) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = n;
    SLAI_CHECK_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, P, hi, lo, sum));
    return SLAI_OK;
}

template <int FMT>
int launch_fmt(slai_ctx* ctx, PgParams& P, const PrefillGemm& G) {
    // What the longest SM has to do, in units of a plain super-block (some 2400 cycles): whole tiles one after the other; an equal share of all super-blocks,
    // where every CTA that a tile is spread over beyond its first costs the one that adds the sums about two; or a share of K of one tile in a
    // cluster, about three and a half for its start and end in every round.  A pair's super-block takes about two thirds of the time (half the
    // activations' L2 and shared-memory traffic per SM).  us per product, 7B shape, without equal shares / as chosen (ncu, serialised; the same
    // build with the rule off): 37 tokens q/k/v 27.2 / 25.7, gate and up 47.6 / 35.1 (o and down stay clusters of 4: 16.0, 24.9); 200 tokens q/k/v 59.5 / 50.4, gate and
    // up 86.0 / 78.0, down 53.4 / 50.9; 511 tokens (pairs) q/k/v 92.9 / 91.3, gate and up 149.5 / 151.4.
    const int sms = std::min(ctx->sm_count > 0 ? ctx->sm_count : 148, PG_MAX_CTAS);
    auto m_tiles = [&](int rows) {
        int t = 0;
        for (int i = 0; i < P.nseg; i++) t += (P.seg[i].rows + rows - 1) / rows;
        return t;
    };
    const long long tiles = (long long)m_tiles(PG_BM) * P.n_tiles, pairs = (long long)m_tiles(2 * PG_BM) * P.n_tiles;
    auto whole = [&](long long t, int ctas) { return (double)((t + ctas - 1) / ctas) * P.nch; };
    auto equal = [&](long long t, int ctas, double sb, double& cost) {
        const double each = (double)t * P.nch / ctas;
        if (each < 1) return false;
        const double c = sb * each + 2 * ceil(P.nch / each);
        if (c >= cost) return false;
        cost = c;
        return true;
    };
    double best = whole(tiles, sms);
    P.ks = 1;
    for (int ks = 2; ks <= PG_MAX_KS && ks <= P.nch; ks *= 2) {
        const double cost = (double)((tiles * ks + sms - 1) / sms) * ((P.nch + ks - 1) / ks + 3.5);
        if (cost < best) {
            best = cost;
            P.ks = ks;
        }
    }
    P.shared = equal(tiles, sms, 1.0, best);
    if (P.shared) P.ks = 1;
    const bool merged = P.NT <= 64;
    double best_pair = 0.65 * whole(pairs, sms / 2);
    const int shared_pair = equal(pairs, sms / 2, 0.65, best_pair);
    const bool pair = !merged && best_pair < best;
    if (pair) {
        P.ks = 1;
        P.shared = shared_pair;
    }
    const int NB = pair ? P.NT / 2 : P.NT, K = (int)G.w[0]->ncols;
    CUtensorMap hi, lo, sum;
    int rc = make_plane_map(ctx, &hi, G.x_hi, G.t_pad, K, PG_BK, NB);
    if (rc) return rc;
    if ((rc = make_plane_map(ctx, &lo, G.x_lo, G.t_pad, K, PG_BK, NB))) return rc;
    sum = hi;
    if (pfq::Fmt<FMT>::MIN && (rc = make_plane_map(ctx, &sum, G.x_sum, G.t_pad, K / 16, 16, NB))) return rc;
    if (pair) return launch_mode<FMT, PG_PAIR>(ctx, P, hi, lo, sum);
    if (merged) return launch_mode<FMT, PG_MERGED>(ctx, P, hi, lo, sum);
    return launch_mode<FMT, PG_PLAIN>(ctx, P, hi, lo, sum);
}

}  // namespace

// Tokens per CTA tile of a prompt of T tokens: as few tiles as 128 tokens allow, of equal size (a multiple of 16).
int prefill_gemm_nt(int T) {
    const int tiles = (T + PG_MAX_NT - 1) / PG_MAX_NT;
    return ((T + tiles - 1) / tiles + 15) / 16 * 16;
}

// Rows that the buffers of a pass with `t_pad` rows get: in steps of 256 above 256, so that a conversation whose turns grow does not
// allocate anew on each (7B shape, 511 tokens after 300: 8.0 ms, of which 6 are the allocation).
int prefill_buffer_rows(int t_pad) { return t_pad <= 256 ? t_pad : (t_pad + 255) / 256 * 256; }

// out_i[t][m] = (resid[t][m] +) sum_k W_i[m][k] X[t][k] (+ bias_i[m]) for t < T and up to three matrices W_i of one format and
// width that share the activations, given as hi / lo planes (and the sub-blocks' sums, see PrefillGemm) of `t_pad` rows.
// Rows T .. t_pad - 1 of the planes may hold anything: a token's sums depend on its own row alone.
int prefill_gemm_launch(slai_ctx* ctx, const PrefillGemm& G) {
    SLAI_REQUIRE(ctx, G.n >= 1 && G.n <= 3 && G.w[0], SLAI_ERR_INVALID_ARG, "prefill: %d matrices in one launch", G.n);
    const slai_qmatrix* w = G.w[0];
    SLAI_REQUIRE(ctx, w->fmt == SLAI_FMT_Q4_K || w->fmt == SLAI_FMT_Q5_K || w->fmt == SLAI_FMT_Q6_K || w->fmt == SLAI_FMT_Q8_0,
                 SLAI_ERR_UNSUPPORTED_FORMAT, "prefill: format %d has no GEMM path", w->fmt);
    const int NT = prefill_gemm_nt(G.T), K = (int)w->ncols;
    SLAI_REQUIRE(ctx, K % PG_BK == 0 && G.T >= 1 && G.t_pad % NT == 0 && G.T <= G.t_pad && (w->fmt == SLAI_FMT_Q8_0 || K % 256 == 0), SLAI_ERR_SHAPE,
                 "prefill: K=%d / %d tokens not supported", K, G.T);
    SLAI_REQUIRE(ctx, (w->fmt != SLAI_FMT_Q4_K && w->fmt != SLAI_FMT_Q5_K) || G.x_sum, SLAI_ERR_INVALID_ARG, "prefill: the minimum term needs the sub-block sums");
    PgParams P = {};
    for (int i = 0; i < G.n; i++) {
        SLAI_REQUIRE(ctx, G.w[i] && G.w[i]->fmt == w->fmt && G.w[i]->ncols == w->ncols && G.w[i]->tile_bytes == w->tile_bytes && G.rows[i] > 0 &&
                              G.rows[i] <= G.w[i]->nrows,
                     SLAI_ERR_SHAPE, "prefill: matrices of one launch must share format and width");
        SLAI_REQUIRE(ctx, (reinterpret_cast<uintptr_t>(G.w[i]->data) & 15) == 0 && w->tile_bytes % 16 == 0, SLAI_ERR_INVALID_ARG,
                     "prefill: matrix data must be 16-byte aligned");
        P.seg[i].w = G.w[i]->data;
        P.seg[i].out = G.out[i];
        P.seg[i].bias = G.bias[i];
        P.seg[i].rows = G.rows[i];
    }
    P.nseg = G.n;
    P.tile_bytes = w->tile_bytes;
    P.nch = (int)layout::num_steps(w->fmt, K);
    P.T = G.T; P.NT = NT; P.n_tiles = G.t_pad / NT; P.ldo = G.ldo; P.resid = G.resid; P.ldr = G.ldr;
    P.NTP = 16;
    while (P.NTP < NT) P.NTP <<= 1;
    P.err_flag = ctx->d_counters + CNT_ERR_FLAG;
    P.wait_limit = ctx->wait_limit;
    switch (w->fmt) {
        case SLAI_FMT_Q4_K: return launch_fmt<SLAI_FMT_Q4_K>(ctx, P, G);
        case SLAI_FMT_Q5_K: return launch_fmt<SLAI_FMT_Q5_K>(ctx, P, G);
        case SLAI_FMT_Q6_K: return launch_fmt<SLAI_FMT_Q6_K>(ctx, P, G);
        default: return launch_fmt<SLAI_FMT_Q8_0>(ctx, P, G);
    }
}
