// Packed quants -> fp16 operand rows of the prompt GEMM (prefill_gemm.cu), without a single type conversion.
//
// A conversion (int -> float, float -> half) issues at a quarter of the rate of the fp16x2 arithmetic or less, and the
// first version of this path needed four per weight: 8192 weights of a stage took about 2000 cycles per SM whatever the
// tile size, which bounded every prompt (7B, 37 tokens: 27 ms).  Here a quant q is OR'ed into the mantissa of the fp16
// number 1024 (0x6400 | q = 1024 + q, exact) and one HFMA2 removes the offset and applies the integer block scale:
// about 1.3 instructions per weight.
//
// What the operand holds, per format (`r` row, `k` column):
//   Q4_K / Q5_K   sc * q, an integer of at most 63 * 31 < 2048: exact in fp16, ONE plane.  The row's f16 super-block scale d
//                 is applied to the f32 sums of 256 columns, and -dmin * m * (sum of the sub-block's activations) is one more
//                 16-deep product per super-block (`min_row`).  No weight is rounded.
//   Q6_K          sc * (q - 32), an integer of up to 4096: fp16 pair hi + lo (lo is exact: a remainder of one or two units).
//                 d as above.
//   Q8_0          d * q: fp16 pair hi + lo, the same two halves as rounding the f32 product and its remainder.
//
// Thread (row r16 of a 16-row tile, part) serves 32 of the 64 columns of a stage.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

#include "layout.cuh"

namespace pfq {

SLAI_HD uint32_t bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
SLAI_HD __half2 h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }
SLAI_HD __half2 both(uint32_t h16) { return h2((h16 & 0xFFFFu) * 0x10001u); }
SLAI_HD __half2 small_int(uint32_t v) { return __hsub2(both(0x6400u | v), h2(0x64006400u)); }  // v < 1024 in both halves, exact

SLAI_HD __half2 fma2(__half2 a, __half2 b, __half2 c) {
#ifdef __CUDA_ARCH__
    return __hfma2(a, b, c);
#else  // the exact sum of the exact product, rounded once
    return __halves2half2(__double2half((double)__half2float(__low2half(a)) * __half2float(__low2half(b)) + __half2float(__low2half(c))),
                          __double2half((double)__half2float(__high2half(a)) * __half2float(__high2half(b)) + __half2float(__high2half(c))));
#endif
}

template <int FMT>
struct Fmt;
template <>
struct Fmt<12> { static constexpr int STEP = 2368, PLANES = 1, STAGES = 4; static constexpr bool MIN = true, SCALED = true; };
template <>
struct Fmt<13> { static constexpr int STEP = 2880, PLANES = 1, STAGES = 4; static constexpr bool MIN = true, SCALED = true; };
template <>
struct Fmt<14> { static constexpr int STEP = 3360, PLANES = 2, STAGES = 4; static constexpr bool MIN = false, SCALED = true; };
template <>
struct Fmt<8> { static constexpr int STEP = 2176, PLANES = 2, STAGES = 2; static constexpr bool MIN = false, SCALED = false; };

// The packed bytes one thread needs of a stage, read from the tile-step block before its operand slot is free.
struct Packed {
    uint4 q[2];   // Q4_K / Q5_K: 16 bytes (both nibbles used), then Q5_K's 16 high-bit bytes; Q6_K: the two ql pieces; Q8_0: 32 values
    uint4 qh;     // Q6_K: 16 bytes of upper bits
    uint32_t sc;  // two scale bytes; Q8_0: the f16 block scale
};

template <int FMT>
SLAI_HD void fetch(const unsigned char* blk, int r16, int part, int st, Packed& P) {
    const int g = r16 & 7, ab = r16 >> 3;
    if (FMT == 12 || FMT == 13) {
        P.sc = *reinterpret_cast<const unsigned short*>(blk + layout::K45_HDR_ROW * r16 + layout::k45_sc_off(2 * st));  // sub-blocks 2 st, 2 st + 1
        const int q0 = FMT == 12 ? layout::K45_HDR : layout::K45_HDR + 512;
        P.q[0] = *reinterpret_cast<const uint4*>(blk + layout::qbyte_off(q0, r16, 32 * st + 16 * part));
        if (FMT == 13) P.q[1] = *reinterpret_cast<const uint4*>(blk + layout::K45_HDR + 32 * r16 + 16 * part);
    } else if (FMT == 14) {
        const int hf = st >> 1, lane = 32 * g + 16 * part;
        P.q[0] = *reinterpret_cast<const uint4*>(blk + ((hf * 2 + 0) * 2 + ab) * 256 + lane);
        P.q[1] = *reinterpret_cast<const uint4*>(blk + ((hf * 2 + 1) * 2 + ab) * 256 + lane);
        P.qh = *reinterpret_cast<const uint4*>(blk + 2048 + (hf * 2 + ab) * 256 + lane);
        const unsigned char* s = blk + 3072 + 16 * r16 + 8 * hf + part + 4 * (st & 1);
        P.sc = (uint32_t)s[0] | ((uint32_t)s[2] << 8);
    } else {
        const int b = 2 * st + part;
        const uint4* q = reinterpret_cast<const uint4*>(blk + layout::qbyte_off(128, r16, 32 * b));
        P.q[0] = q[0];
        P.q[1] = q[1];
        P.sc = *reinterpret_cast<const unsigned short*>(blk + 8 * r16 + 2 * b);
    }
}

// A row's 32 of the 64 columns of a stage as pairs of halves, hi (and lo) plane: words 0-7 and 8-15 are columns 16 part .. and 32 + 16 part ..
// (Q8_0: all sixteen are columns 32 part ..).
template <int FMT>
SLAI_HD void make(const Packed& P, int st, uint32_t (&hi)[16], uint32_t (&lo)[16]) {
    const uint32_t w0[4] = {P.q[0].x, P.q[0].y, P.q[0].z, P.q[0].w};
    const uint32_t w1[4] = {P.q[1].x, P.q[1].y, P.q[1].z, P.q[1].w};
    if (FMT == 12 || FMT == 13) {
        const __half2 sl = small_int(P.sc & 0xFFu), sh = small_int((P.sc >> 8) & 0xFFu);
        const __half2 ol = __hmul2(sl, h2(0xE400E400u));                                         // -1024 sc
        const __half2 sh16 = FMT == 12 ? __hmul2(sh, h2(0x2C002C00u)) : sh;                       // sc / 16 (the high nibble goes in as 16 q)
        const __half2 oh = __hmul2(sh16, h2(0xE400E400u));
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t p = frag::perm_bytes(w0[i >> 1], 0u, (i & 1) ? 0x4342 : 0x4140);  // two bytes, one per half
            if (FMT == 12) {
                hi[i] = bits(fma2(h2((p & 0x000F000Fu) | 0x64006400u), sl, ol));
                hi[8 + i] = bits(fma2(h2((p & 0x00F000F0u) | 0x64006400u), sh16, oh));
            } else {
                const uint32_t h = frag::perm_bytes(w1[i >> 1], 0u, (i & 1) ? 0x4342 : 0x4140) >> (2 * st);
                hi[i] = bits(fma2(h2((p & 0x000F000Fu) | ((h & 0x00010001u) << 4) | 0x64006400u), sl, ol));
                hi[8 + i] = bits(fma2(h2(((p >> 4) & 0x000F000Fu) | ((h & 0x00020002u) << 3) | 0x64006400u), sh16, oh));
            }
        }
    } else if (FMT == 14) {
        const uint32_t h4[4] = {P.qh.x, P.qh.y, P.qh.z, P.qh.w};
#pragma unroll
        for (int u = 0; u < 2; u++) {  // quarter 2 (st & 1) + u of the half super-block
            const __half2 s = __half2half2(__short2half_rn((short)(signed char)((P.sc >> (8 * u)) & 0xFFu)));
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const uint32_t w = u ? w1[i >> 1] : w0[i >> 1];
                const uint32_t sel = (i & 1) ? 0x4342 : 0x4140;
                const uint32_t p = frag::perm_bytes(w, 0u, sel) >> (4 * (st & 1));
                const uint32_t h = frag::perm_bytes(h4[i >> 1], 0u, sel) >> (4 * (st & 1) + 2 * u);
                const __half2 q = __hsub2(h2((p & 0x000F000Fu) | ((h & 0x00030003u) << 4) | 0x64006400u), h2(0x64206420u));  // q - 32
                const __half2 v = __hmul2(q, s);
                hi[8 * u + i] = bits(v);
                lo[8 * u + i] = bits(fma2(q, s, __hneg2(v)));
            }
        }
    } else {
        const __half2 d = both(P.sc);
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const uint32_t w = (i < 8 ? w0[i >> 1] : w1[(i - 8) >> 1]) ^ 0x80808080u;
            const __half2 q = __hsub2(h2(frag::perm_bytes(w, 0x64646464u, (i & 1) ? 0x4342 : 0x4140)), h2(0x64806480u));  // 1024 + 128 + q
            const __half2 v = __hmul2(q, d);
            hi[i] = bits(v);
            lo[i] = bits(fma2(q, d, __hneg2(v)));
        }
    }
}

// Q4_K / Q5_K: row r of the 16-column operand of the minimum term of one super-block: m_0..m_7 (part 0) against the fp16
// sums of the sub-blocks' activations, m_j / 2048 (part 1, exact) against 2048 times what those sums lost in rounding.  Rows of 32
// bytes; 16-byte chunk c of row r at chunk position c ^ ((r >> 2) & 1) (32-byte swizzle).
SLAI_HD void min_row(const unsigned char* blk, int r16, int r, int part, unsigned char* amin) {
    const uint32_t* h = reinterpret_cast<const uint32_t*>(blk + layout::K45_HDR_ROW * r16 + 12);
    const __half2 f = part ? h2(0x10001000u) : h2(0x3C003C00u);  // 2^-11, 1
    uint32_t v[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t p = frag::perm_bytes(h[i >> 1], 0x64646464u, (i & 1) ? 0x4342 : 0x4140);
        v[i] = bits(__hmul2(__hsub2(h2(p), h2(0x64006400u)), f));
    }
    *reinterpret_cast<uint4*>(amin + r * 32 + ((part ^ ((r >> 2) & 1)) << 4)) = make_uint4(v[0], v[1], v[2], v[3]);
}

// f16 d (low half) and dmin (high half) of row r16; Q6_K has no minimum.
template <int FMT>
SLAI_HD uint32_t row_scale(const unsigned char* blk, int r16) {
    if (FMT == 14) return *reinterpret_cast<const unsigned short*>(blk + 3328 + 2 * r16);
    return *reinterpret_cast<const uint32_t*>(blk + layout::K45_HDR_ROW * r16);
}

}  // namespace pfq
