// The per-stream arithmetic coder: bit window, bit sink, decode loop and encode step.
//
// This header compiles both as CUDA device code (the product) and as plain host C++ (only so that
// the CPU test-suite can drive exactly these loops against the oracle without a GPU; the shared
// library never contains or calls a host build of them).
//
// The steps restate the reference's loops
// (LMCache/third_party/torchac_cuda/torchac_kernel_dec_new.cu:262-302 and
//  torchac_kernel_enc_new.cu:255-306) without the 64-bit division, the binary search on `count`
// and the bit-serial renormalisation:
//   * cdf[m] <= count, count = ((value-low+1)*2^16 - 1) / span, holds exactly when
//     (span*cdf[m]) >> 16 <= value - low, so the search compares scaled table entries with
//     value - low directly;
//   * within one symbol the renormalisation loop does a run of "equal top bit" shifts followed
//     by a run of "underflow" shifts, never the other way round; their sum comes from one
//     leading-bit search (renorm_shift), by which the decoder moves its position in the stream and the
//     encoder appends the shifted-out top bits of `low` at once, carries included.
#pragma once

#include <stdint.h>

#if defined(__CUDACC__)
#define CG_HD __host__ __device__ __forceinline__
#else
#define CG_HD inline
#endif
#if defined(__CUDA_ARCH__)
#define CG_UNROLL _Pragma("unroll")
#define CG_NO_UNROLL _Pragma("unroll 1")
#else
#define CG_UNROLL
#define CG_NO_UNROLL
#endif

namespace cg {

constexpr int kGroupChannels = 128;            // streams (threads) per coder block
constexpr int kTableRowBytes = kGroupChannels * 4;  // bytes between table entries m and m+1 of a stream

// ---- grids of the decoders --------------------------------------------------------------------------------
constexpr int kMultiBlocksPerSM = 12;  // of the kernels with two channels a thread, at 33-entry tables

// Blocks to have on an SM at a time where a grid of `chunks` chunks, the first of `ntokens` tokens, would leave a short second wave;
// 0: as many as fit.  Twelve blocks an SM, and then two to four more on each, whose serial chains take most of a wave's time
// with next to nothing beside them: eight or ten at first, so that the others get company.  256 tokens with twelve and so, 7B
// settings: 32 layers x 32 heads (14 blocks an SM) 159.5 and 152.3 us, x 35 (16) 170.4 and 159.7, nine chunks of 32 x 4 (16) 169.7 and
// 163.5; 70B settings: 80 x 14 (16) 174.5 and 162.3, 40 x 28 (16) 164.6 and 165.2.
// Not where it would hold blocks back for longer than it saves: thirteen an SM (40 x 24 151.6 and 153.0), fourteen of several
// chunks, whose blocks come in no order of their work (4 of 32 x 8, the last of 5 tokens, 124.4 and 141.7), few tokens (16 of
// 32 x 32 at 32 bins 20.7 and 21.4) and delta coding (9 of 32 x 4 192.8 and 200.9).
// Short tables (5 to 17 entries): one chunk's KV only, from thirteen and three quarters an SM on.  Half the 7B bins, 32 x 32 141.3 and
// 136.2, x 34 152.8 and 143.7, x 36 155.7 and 144.4; a quarter of them 126.1 and 120.1, 136.2 and 128.9, 140.0 and 130.1; rows that
// are all alike 150.3 and 143.4, 151.9 and 153.4, 153.5 and 155.0.  Below, a fourteenth block that most SMs have not got costs more
// than it gives (40 x 25 135.1 and 138.2); so do several chunks (nine of level 1 at 64 tokens 46.1 and 47.1) and, with rows alike,
// symbols (32 x 32 85.5 and 94.7 for 150 tokens, where half the bins take 86.7 and 82.0).
CG_HD int evened_blocks(int64_t blocks, int64_t sms, int levels, bool symbols, int chunks, int ntokens) {
    const int64_t more = (blocks + sms - 1) / sms - kMultiBlocksPerSM;
    if (levels < 3 || levels > 5 || ntokens < 64 || more > 4) return 0;
    if (levels < 5 && (symbols || chunks > 1 || 4 * blocks < 55 * sms)) return 0;
    return more > 2 ? 10 : more == 2 && chunks == 1 ? 8 : 0;
}

// ---- intrinsics with host stand-ins -----------------------------------------------------------------
CG_HD int cg_clz(uint32_t x) {
#if defined(__CUDA_ARCH__)
    return __clz(static_cast<int>(x));
#else
    return x ? __builtin_clz(x) : 32;
#endif
}
// upper 32 bits of (hi:lo) << (s & 31)
CG_HD uint32_t cg_fshl(uint32_t lo, uint32_t hi, uint32_t s) {
#if defined(__CUDA_ARCH__)
    return __funnelshift_l(lo, hi, s);
#else
    s &= 31u;
    return s ? ((hi << s) | (lo >> (32u - s))) : hi;
#endif
}
// lower 32 bits of (hi:lo) >> min(s, 32)
CG_HD uint32_t cg_fshr_clamp(uint32_t lo, uint32_t hi, uint32_t s) {
#if defined(__CUDA_ARCH__)
    return __funnelshift_rc(lo, hi, s);
#else
    if (s >= 32u) return hi;
    return s ? ((lo >> s) | (hi << (32u - s))) : lo;
#endif
}
CG_HD uint32_t cg_bswap32(uint32_t v) {
#if defined(__CUDA_ARCH__)
    return __byte_perm(v, 0, 0x0123);
#else
    return __builtin_bswap32(v);
#endif
}
CG_HD uint32_t cg_load_stream_word(const uint32_t *p) {
#if defined(__CUDA_ARCH__)
    return __ldg(p);
#else
    return *p;
#endif
}

// ---- shared-memory access --------------------------------------------------------------------------------
// A stream's table is a column tab[m][tid] of a [rows][128] uint32 array (cdf[m] << 16 for the encoder, search_entry(cdf[m])
// for the decoder), addressed
// by byte address: entry m of the column starting at `col` is at col + m * kTableRowBytes.  On the
// device the addresses are shared-memory addresses (bank = lane for every row); on the host they are
// offsets into a plain array.
struct Smem {
#if defined(__CUDA_ARCH__)
    __device__ __forceinline__ uint32_t ld(uint32_t addr) const {
        uint32_t v;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
        return v;
    }
    __device__ __forceinline__ void st(uint32_t addr, uint32_t v) const {
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
    }
#else
    uint8_t *base;
    uint32_t ld(uint32_t addr) const { return *reinterpret_cast<const uint32_t *>(base + addr); }
    void st(uint32_t addr, uint32_t v) const { *reinterpret_cast<uint32_t *>(base + addr) = v; }
#endif
};

// ---- renormalisation shift ----------------------------------------------------------------------------
// After a range update the reference shifts while low and high agree in their top bit, then while low
// starts 01 and high 10 (enc_new.cu:275-293, dec_new.cu:284-301).  Both kinds double the interval, and
// together they stop at the largest s for which [low, high] lies inside a window of 2^(32-s) values that
// starts at a multiple of half its size (the midpoint windows of the second kind included).  With
// d = high - low and b the position of d's top bit, that is 32-s = b+1 when [low, high] touches only two
// cells of 2^b values and b+2 when it touches three, and it touches three exactly when the low b bits
// of low and of d carry into bit b: when bit b, which d has set, is the same in low and in low + d.  So
// s is the number of leading zeros of d, less one when that bit of low ^ high is clear: one leading-bit
// search, one shift for the bit's mask and one three-input test.  Only the bits of low up to b matter, so low
// may carry anything in its top bit after the shift.  (The carry found by adding the low b bits of both at
// the top of a word instead, two multiplies and two adds with carry: one instruction more and four more
// cycles of the multiply pipe a symbol.)
//
// By the size u = d + 1 instead of d (the coders' loops): the top bit is another one only where u is a power of two, and
// s one or two less than it could be where low is a multiple of u or of u / 2 as well.  Nothing is lost by that: the next
// symbol's bounds are exact at any scale of such a range, and its shift makes up for it; and the full range of 2^32, which
// no word holds, does not come about.  (Only u = 2^31 at a multiple of 2^31 gives -1: see EncoderState::steps_at and
// DecoderState.)
//
// The conditional decrement is written as a predicated add: with `if (...) --s` the counters show two executed
// instructions a symbol more.
// low, high = low + d, d (or u)
CG_HD uint32_t renorm_shift(uint32_t low, uint32_t high, uint32_t d) {
#if defined(__CUDA_ARCH__)
    uint32_t s;
    asm("{ .reg .u32 t, b; .reg .pred p;\n"
        "bfind.shiftamt.u32 %0, %3;\n"
        "shf.r.wrap.b32 b, 0x80000000, 0, %0;\n"
        "lop3.b32 t, %1, %2, b, 0x28;\n"  // (low ^ high) & b
        "setp.eq.u32 p, t, 0;\n"
        "@p add.u32 %0, %0, -1; }"
        : "=&r"(s) : "r"(low), "r"(high), "r"(d));
    return s;
#else
    const uint32_t s = d ? static_cast<uint32_t>(cg_clz(d)) : 0xFFFFFFFFu;
    return ((low ^ high) & (0x80000000u >> (s & 31u))) == 0u ? s - 1u : s;
#endif
}
// The same from the size as a float, rounded towards zero, whose exponent is the place of its top bit.
CG_HD float size_as_float(uint32_t u) {
#if defined(__CUDA_ARCH__)
    return __uint2float_rz(u);
#else
    return static_cast<float>(u & ~(u >= (1u << 24) ? (1u << (8 - cg_clz(u))) - 1u : 0u));
#endif
}
CG_HD uint32_t renorm_shift(uint32_t low, uint32_t high, float size) {
#if defined(__CUDA_ARCH__)
    uint32_t s;
    asm("{ .reg .u32 e, t, b; .reg .pred p;\n"
        "shr.u32 e, %3, 23;\n"
        "shf.l.wrap.b32 b, 2, 2, e;\n"  // 1 << e - 127, since 127 is one less than a multiple of 32
        "sub.u32 %0, 158, e;\n"
        "lop3.b32 t, %1, %2, b, 0x28;\n"
        "setp.eq.u32 p, t, 0;\n"
        "@p add.u32 %0, %0, -1; }"
        : "=&r"(s) : "r"(low), "r"(high), "r"(__float_as_uint(size)));
    return s;
#else
    return renorm_shift(low, high, static_cast<uint32_t>(size));
#endif
}
// ---- warp votes and products -------------------------------------------------------------------------------------
CG_HD bool cg_any_lane(uint32_t lanes, bool pred) {
#if defined(__CUDA_ARCH__)
    return __any_sync(lanes, pred) != 0;
#else
    (void)lanes;
    return pred;
#endif
}

CG_HD uint32_t cg_umulhi(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
    return __umulhi(a, b);
#else
    return static_cast<uint32_t>((static_cast<uint64_t>(a) * b) >> 32);
#endif
}
// The same as the upper half of a wide product: the coders' steps, which add to it, execute one or two instructions fewer so.
CG_HD uint32_t cg_umulhi_wide(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
    uint64_t p;
    asm("mul.wide.u32 %0, %1, %2;" : "=l"(p) : "r"(a), "r"(b));
    return static_cast<uint32_t>(p >> 32);
#else
    return cg_umulhi(a, b);
#endif
}
// a + b - 1: one executed instruction fewer than from the C++ form
CG_HD uint32_t cg_add_less_one(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
    uint32_t d;
    asm("{ .reg .u32 t; add.u32 t, %1, %2; add.u32 %0, t, -1; }" : "=r"(d) : "r"(a), "r"(b));
    return d;
#else
    return a + b - 1u;
#endif
}

// ---- bit window ------------------------------------------------------------------------------------------------------
// The 64 bits of a stream from bit `at` on, in two registers, which a decoder reads at a position of its own and does not
// shift: its 32-bit value at position p is one funnel shift, whatever was taken before.  The byte array is read as aligned
// 32-bit words; bits past the stream's last byte are zero, which is what the reference sees in its zero-padded staging
// row (dec_new.cu:229-232).
struct BitWindow {
    const uint32_t *wp;   // the word that holds the window's first bit
    uint32_t off;         // that bit's place in it
    int32_t rem;          // bits of the stream from two words further on, negative past its end
    uint32_t w0, w1, w2;  // the words from wp on, big-endian, bits past the stream's end cleared
    uint32_t hi, lo;      // the window

    // word j from wp on; r: bits of the stream from there on
    CG_HD uint32_t word(int j, int32_t r) const {
        uint32_t w = 0u;
        if (r > 0) w = cg_bswap32(cg_load_stream_word(wp + j));
        return w & ~cg_fshr_clamp(0xFFFFFFFFu, 0u, static_cast<uint32_t>(r));  // (a negative one counts as more than 32)
    }
    CG_HD void cut() {
        hi = cg_fshl(w1, w0, off);
        lo = cg_fshl(w2, w1, off);
    }
    CG_HD void open(const uint8_t *p, uint32_t len) {
        const uintptr_t a = reinterpret_cast<uintptr_t>(p);
        wp = reinterpret_cast<const uint32_t *>(a & ~static_cast<uintptr_t>(3));
        off = static_cast<uint32_t>(a & 3u) * 8u;
        rem = static_cast<int32_t>(off + len * 8u) - 64;
        w0 = word(0, rem + 64);
        w1 = word(1, rem + 32);
        w2 = word(2, rem);
        cut();
    }
    // Moves the window on to position p < 64, which becomes 0 (a negative one stays: see DecoderState).  Straight-line: every
    // lane of the warp runs the same instructions whatever it needs, but only words that a lane has not got are
    // read: with three words read for every lane each time the loads' wavefronts, not the instructions, bound the decode
    // (69 % of their rate where this takes 50; 2,048 Llama-7B tokens 986 us, this way 972).
    CG_HD void advance(int32_t &p) {
        const uint32_t to = off + static_cast<uint32_t>(p > 0 ? p : 0), k = to >> 5;  // words to move on by: 0, 1 or 2
        p = p < 0 ? p : 0;
        off = to & 31u;
        wp += k;
        rem -= static_cast<int32_t>(k * 32u);
#if defined(__CUDA_ARCH__)
        asm("{ .reg .u32 t, m; .reg .s32 r; .reg .pred p1, p2, q;\n"
            "setp.gt.u32 p1, %5, 0;\n"
            "setp.gt.u32 p2, %5, 1;\n"
            "@p1 mov.u32 %0, %1;\n"
            "@p1 mov.u32 %1, %2;\n"
            "@p2 mov.u32 %0, %1;\n"
            "setp.gt.and.s32 q, %4, 0, p1;\n"
            "mov.u32 t, 0;\n"
            "@q ld.global.nc.u32 t, [%3+8];\n"
            "prmt.b32 t, t, 0, 0x0123;\n"
            "shr.u32 m, 0xFFFFFFFF, %4;\n"       // (a shift by more than 31 gives 0)
            "@p1 lop3.b32 %2, t, m, 0, 0x30;\n"  // t & ~m
            "add.s32 r, %4, 32;\n"
            "setp.gt.and.s32 q, r, 0, p2;\n"
            "mov.u32 t, 0;\n"
            "@q ld.global.nc.u32 t, [%3+4];\n"
            "prmt.b32 t, t, 0, 0x0123;\n"
            "shr.u32 m, 0xFFFFFFFF, r;\n"
            "@p2 lop3.b32 %1, t, m, 0, 0x30; }"
            : "+r"(w0), "+r"(w1), "+r"(w2) : "l"(wp), "r"(rem), "r"(k));
#else
        if (k) {
            w0 = word(0, rem + 64);
            w1 = word(1, rem + 32);
            w2 = word(2, rem);
        }
#endif
        cut();
    }
    // 32 bits from position p on, 0 <= p <= 32
    CG_HD uint32_t bits(int32_t p) const {
#if defined(__CUDA_ARCH__)
        return __funnelshift_lc(lo, hi, static_cast<uint32_t>(p));
#else
        return p >= 32 || p < 0 ? lo : cg_fshl(lo, hi, static_cast<uint32_t>(p));
#endif
    }
};

// ---- decode loop ------------------------------------------------------------------------------------------
// Scaled table entry for the current span: (span * c16) >> 32 with span32 = span mod 2^32, which is 0
// exactly when the range is the full 2^32 (then the product is c16 itself).
CG_HD uint32_t scale_exact(uint32_t span32, uint32_t c16) { return span32 ? cg_umulhi(span32, c16) : c16; }

// The decoder's arithmetic state: low, span32 = (high - low + 1) mod 2^32 and the position p of the current 32 bits of the
// stream in its window; value - low of the reference is the difference of those bits and low.  Both kinds of renormalisation
// shift act alike on it: low is shifted left, and what the underflow shifts drop from it ("value -= 2^30") is dropped from
// the stream's bits by the same subtraction modulo 2^32.  low is tracked because the shift counts depend on it.
//
// The fast step takes the shift by the interval's size (see renorm_shift); where that gives -1 (a size of 2^31 at a multiple of
// 2^31) what is left is a span of 0, a low of 0 and p one less than it was, and one shift would have been right, which leaves the
// same span and low and p two more.  So a span of 0 stands for the full range of 2^32 with p two less than the position
// of its bits: at the stream's start, too.  Its scaled bounds are all 0, which no symbol passes.
struct DecoderState {
    static constexpr int32_t kFullRange = -2;
    uint32_t low, span32;
    int32_t p;
    CG_HD void init() {
        low = 0u;
        span32 = 0u;
        p = kFullRange;
    }
    // The bits' distance from low; the position of a full range put right.
    CG_HD uint32_t exact_offset(const BitWindow &bw) {
        if (span32 == 0u) p -= kFullRange;
        return bw.bits(p) - low;
    }
    // range update for the symbol whose scaled bounds are [flo, fhi), then renormalisation
    // (dec_new.cu:277-301), both kinds of shift applied in one go.  On a table that is not increasing the
    // shift count is anything up to 31; every later read stays inside the table column and the stream.
    CG_HD void exact_update(uint32_t flo, uint32_t fhi) {
        const uint32_t d = fhi - flo - 1u;
        low += flo;
        const uint32_t s = renorm_shift(low, low + d, d) & 31u;
        low = cg_fshl(0u, low, s);
        span32 = cg_fshl(0u, fhi - flo, s);
        p += static_cast<int32_t>(s);
        if (span32 == 0u) p += kFullRange;
    }
};

// ---- decode loop: NS streams per lane, search depth chosen by the caller ---------------------------------
// Table entries as the search takes them: 2^23 + cdf as a float.  Its bits shifted by sixteen are cdf << 16, and
// a comparison with an estimate of floor(2^16 offset / span) + 1, which is as whole a number, is the difference cut to
// [0, 1], which is 0 or 1.  A search step is then a multiply-add with saturation and one on the entry's address
// (taken as a denormal float, which adds like an integer): both on the two floating-point pipes, where a compare and a
// predicated add go to the integer pipes, which have half the rate and bind the loop.  8,192 Llama-7B tokens: 4.18 ms with
// integer entries, 4.00 with floats when that was measured.
CG_HD uint32_t search_entry(uint32_t cdf) { return 0x4B000000u | cdf; }
constexpr uint32_t kSearchPadding = 0x7F800000u;  // +inf: above every estimate
CG_HD uint32_t ld_entry(Smem sm, uint32_t addr) {
#if defined(__CUDA_ARCH__)
    return sm.ld(addr);
#else
    const uint32_t v = sm.ld(addr);  // the host's columns hold cdf << 16, padded with 0xFFFFFFFF
    return v == 0xFFFFFFFFu ? kSearchPadding : search_entry(v >> 16);
#endif
}
CG_HD uint32_t entry_c16(uint32_t entry) { return cg_fshl(0u, entry, 16u); }  // cdf << 16

// Exact search with a run-time depth (the rare path of decode_streams).
CG_HD uint32_t exact_search(Smem sm, uint32_t col, uint32_t a_max, uint32_t span32, uint32_t target, int levels) {
    uint32_t a = col;
    for (int b = levels - 1; b >= 0; --b) {
        const uint32_t ca = a + (static_cast<uint32_t>(kTableRowBytes) << b);
        const bool ok = ca <= a_max;
        const bool take = ok && (scale_exact(span32, entry_c16(ld_entry(sm, ok ? ca : a))) <= target);
        a = take ? ca : a;
    }
    return a;
}

// Smallest search depth whose top entry, 2^depth - 1, lies above every symbol 0 .. nsym-1, kept
// within [2, full_levels].
CG_HD int fast_levels_for(int nsym, int full_levels) {
    int fl = 2;
    while (fl < full_levels && (1 << fl) - 1 < nsym) fl++;
    return fl;
}

// 128 + (floor(2^16 offset / span) + 1) / 2^16, or one 2^16th off where the quotient is within 2^-6 or so of a whole number:
// a float from 128 on has sixteen bits behind the point, so the rounding of the last addition is the floor (see search_entry).
// Anything when the span is the full 2^32 (span32 == 0).
CG_HD float ratio_estimate(uint32_t offset, uint32_t span32) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint2float_rn(span32)));
    return __fmaf_rz(__uint2float_rn(offset), r, 128.0f + 1.0f / 65536.0f);
#else
    return span32 ? 128.0f + static_cast<float>((static_cast<uint64_t>(offset) << 16) / span32 + 1u) * (1.0f / 65536.0f) : 128.0f;
#endif
}
// The same in two parts: the size's reciprocal before its renormalisation shift is known, and the estimate after it.
CG_HD float size_reciprocal(float size) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(size));
    return r;
#else
    return size;
#endif
}
CG_HD float ratio_estimate(uint32_t offset, uint32_t span32, float reciprocal, uint32_t s) {
#if defined(__CUDA_ARCH__)
    uint32_t r;  // divided by 2^s
    asm("mad.lo.u32 %0, %1, 0xFF800000, %2;" : "=r"(r) : "r"(s), "r"(__float_as_uint(reciprocal)));
    return __fmaf_rz(__uint2float_rn(offset), __uint_as_float(r), 128.0f + 1.0f / 65536.0f);
#else
    (void)reciprocal;
    (void)s;
    return ratio_estimate(offset, span32);
#endif
}
// address a, or a + STEP if the entry is not above the ratio
template <uint32_t STEP>
CG_HD uint32_t search_step(uint32_t a, uint32_t entry, float ratio) {
#if defined(__CUDA_ARCH__)
    float take;
    asm("{ .reg .f32 n; neg.f32 n, %2; fma.rn.sat.f32 %0, %1, 0f47800000, n; }" : "=f"(take) : "f"(ratio), "f"(__uint_as_float(entry)));
    return __float_as_uint(__fmaf_rn(take, __uint_as_float(STEP), __uint_as_float(a)));
#else
    float e;
    __builtin_memcpy(&e, &entry, 4);
    return ratio * 65536.0f - e >= 1.0f ? a + STEP : a;
#endif
}
// Search steps: the candidate entry is kTableRowBytes << B bytes above `a`.
template <int B>
struct RatioSearch {
    static CG_HD uint32_t run(Smem sm, uint32_t a, float ratio) {
        constexpr uint32_t kStep = static_cast<uint32_t>(kTableRowBytes) << B;
        return RatioSearch<B - 1>::run(sm, search_step<kStep>(a, ld_entry(sm, a + kStep), ratio), ratio);
    }
};
template <>
struct RatioSearch<-1> {
    static CG_HD uint32_t run(Smem, uint32_t a, float) { return a; }
};

// Address a, or a + 1, 2 or 3 STEP: as many as there are entries not above the ratio.  Two levels of the search in one load's
// latency, for one multiply-add and two loads more.
template <uint32_t STEP>
CG_HD uint32_t search_quarter(uint32_t a, uint32_t e0, uint32_t e1, uint32_t e2, float ratio) {
#if defined(__CUDA_ARCH__)
    float t0, t1, t2;
    asm("{ .reg .f32 n; neg.f32 n, %2; fma.rn.sat.f32 %0, %1, 0f47800000, n; }" : "=f"(t0) : "f"(ratio), "f"(__uint_as_float(e0)));
    asm("{ .reg .f32 n; neg.f32 n, %2; fma.rn.sat.f32 %0, %1, 0f47800000, n; }" : "=f"(t1) : "f"(ratio), "f"(__uint_as_float(e1)));
    asm("{ .reg .f32 n; neg.f32 n, %2; fma.rn.sat.f32 %0, %1, 0f47800000, n; }" : "=f"(t2) : "f"(ratio), "f"(__uint_as_float(e2)));
    const float b = __fmaf_rn(t2, __uint_as_float(STEP), __uint_as_float(a));
    return __float_as_uint(__fmaf_rn(__fadd_rn(t0, t1), __uint_as_float(STEP), b));
#else
    a = search_step<STEP>(a, e0, ratio);
    return search_step<STEP>(search_step<STEP>(a, e1, ratio), e2, ratio);
#endif
}
template <int B>
struct QuarterSearch {
    static CG_HD uint32_t run(Smem sm, uint32_t a, float ratio) {
        if (B == 0) return RatioSearch<0>::run(sm, a, ratio);
        constexpr uint32_t kStep = static_cast<uint32_t>(kTableRowBytes) << (B > 0 ? B - 1 : 0);
        const uint32_t e0 = ld_entry(sm, a + kStep), e1 = ld_entry(sm, a + 2 * kStep), e2 = ld_entry(sm, a + 3 * kStep);
        return QuarterSearch<B - 2>::run(sm, search_quarter<kStep>(a, e0, e1, e2, ratio), ratio);
    }
};
template <>
struct QuarterSearch<-1> {
    static CG_HD uint32_t run(Smem, uint32_t a, float) { return a; }
};
template <>
struct QuarterSearch<-2> {
    static CG_HD uint32_t run(Smem, uint32_t a, float) { return a; }
};

// NS streams of one lane decoded side by side (same token count, same table length), the fast
// search limited to the first 2^FL table entries.
//
// The fast search compares the table entries with an estimate of offset / span, which costs one compare a
// level where the scaled entry costs a multiply-high as well (four cycles of the multiply pipe and two of the
// integer pipe a warp, measured).  The symbol is then checked exactly: the offset must lie inside its scaled
// bounds, which the range update needs anyway.  The caller picks FL from what it knows about the symbols (a
// row quantised to `bins` bins holds symbols 0 .. bins-2, so 2^FL >= bins is enough).  The result depends
// on neither: a symbol that fails the check -- an estimate on the wrong side of an entry, a symbol >= 2^FL - 1, a symbol that
// starts from the full 2^32 range (its scaled bounds are both 0) -- is thrown away and the whole warp repeats that symbol with
// the exact, full-depth search.
//
// QUICK: for few warps, which wait for one another's results more than for issue slots: two levels of the search at once, the first two
// from registers, and the reciprocal of a size taken beside its renormalisation shift and not behind it.  More instructions, and more
// registers, for a shorter chain: a token of one warp a scheduler takes 200 ns where the other form takes 223.
//
// The table's last symbol has no upper entry.  With LAST_REPEATED the rows above its entry hold copies of it,
// so that its bounds are equal and the check fails; otherwise they hold kSearchPadding and
// a symbol at or above the address threshold det is repeated as well.  The column needs 2^FL + 1
// readable rows either way.
//   col[i]    table column of stream i (see decode_stream)
//   det       address threshold of entry min(2^FL - 1, maxsym): column-independent because a column's offset
//             inside a table row is below kTableRowBytes (det = table base + entry * kTableRowBytes)
//   emit(a, t4)  receives the NS table-entry addresses of one token's symbols and the start value of t4
//             plus four times the token's index (ntok >= 1)
template <int FL, int NS, bool LAST_REPEATED = false, bool QUICK = false, class Emit>
CG_HD void decode_streams(Smem sm, const uint32_t (&col)[NS], uint32_t det, int maxsym, int full_levels,
                          const uint8_t *const (&stream)[NS], const uint32_t (&len)[NS], int ntok, uint32_t lanes,
                          Emit emit, uint32_t t4 = 0u) {
    static_assert(FL >= 2, "the first level's entry is held in a register");
    BitWindow bw[NS];
    DecoderState st[NS];
    uint32_t mid[NS], low_quarter[NS], high_quarter[NS];
    constexpr uint32_t kTop = static_cast<uint32_t>(kTableRowBytes) << (FL - 1);
    CG_UNROLL
    for (int i = 0; i < NS; ++i) {
        st[i].init();
        bw[i].open(stream[i], len[i]);
        mid[i] = ld_entry(sm, col[i] + kTop);
        if (QUICK) {
            low_quarter[i] = ld_entry(sm, col[i] + kTop / 2);
            high_quarter[i] = ld_entry(sm, col[i] + kTop / 2 * 3);
        }
    }
    uint32_t a[NS], flo[NS], fhi[NS];
    const uint32_t last4 = t4 + static_cast<uint32_t>(ntok - 1) * 4u;
    bool odd = true;  // the first symbol starts from the full range
    // The inner loop is the common case and nothing else, begins behind the estimate for the symbol that it decodes (0.7 % faster than
    // in front of it: 8,192 Llama-7B tokens 3,684 -> 3,663 us) and is left by one vote for a window that has been read to its end, for a
    // symbol whose fast search failed and at the last token; with that code inside it, every pass executed more
    // instructions, whether it took that code or not.
    for (;;) {
        if (odd) {
            CG_UNROLL
            for (int i = 0; i < NS; ++i) {
                const uint32_t offset = st[i].exact_offset(bw[i]);
                const uint32_t a_max = col[i] + static_cast<uint32_t>(maxsym) * kTableRowBytes;
                a[i] = exact_search(sm, col[i], a_max, st[i].span32, offset, full_levels);
                flo[i] = scale_exact(st[i].span32, entry_c16(ld_entry(sm, a[i])));
                fhi[i] = (a[i] == a_max) ? st[i].span32
                                            : scale_exact(st[i].span32, entry_c16(ld_entry(sm, a[i] + kTableRowBytes)));
            }
            emit(a, t4);
            if (t4 == last4) break;  // no range update for the last symbol (dec_new.cu:273-275)
            t4 += 4u;
            CG_UNROLL
            for (int i = 0; i < NS; ++i) st[i].exact_update(flo[i], fhi[i]);
        }
        CG_UNROLL
        for (int i = 0; i < NS; ++i) bw[i].advance(st[i].p);
        uint32_t low[NS], u[NS], s[NS], bits[NS];
        int32_t p[NS];
        float ratio[NS];
        bool rare;  // a symbol that fails the check
        CG_UNROLL
        for (int i = 0; i < NS; ++i) {
            bits[i] = bw[i].bits(st[i].p);
            ratio[i] = ratio_estimate(bits[i] - st[i].low, st[i].span32);
        }
        CG_NO_UNROLL
        for (;;) {
            int32_t beyond = 0;
            rare = false;
            CG_UNROLL
            for (int i = 0; i < NS; ++i)
                a[i] = QUICK ? search_quarter<kTop / 2>(col[i], low_quarter[i], mid[i], high_quarter[i], ratio[i])
                             : search_step<kTop>(col[i], mid[i], ratio[i]);
            CG_UNROLL
            for (int i = 0; i < NS; ++i) a[i] = QUICK ? QuarterSearch<FL - 3>::run(sm, a[i], ratio[i]) : RatioSearch<FL - 2>::run(sm, a[i], ratio[i]);
            uint32_t e0[NS], e1[NS];
            CG_UNROLL
            for (int i = 0; i < NS; ++i) {
                e0[i] = entry_c16(ld_entry(sm, a[i]));
                e1[i] = entry_c16(ld_entry(sm, a[i] + kTableRowBytes));
            }
            float reciprocal[NS];
            CG_UNROLL
            for (int i = 0; i < NS; ++i) {
                const uint32_t f0 = cg_umulhi_wide(st[i].span32, e0[i]), f1 = cg_umulhi_wide(st[i].span32, e1[i]);
                low[i] = st[i].low + f0;
                u[i] = f1 - f0;
                rare = rare | (bits[i] - low[i] >= u[i]);
                if (!LAST_REPEATED) rare = rare | (a[i] >= det);
                const uint32_t high = cg_add_less_one(low[i], u[i]);
                if (QUICK) {
                    const float size = size_as_float(u[i]);
                    reciprocal[i] = size_reciprocal(size);
                    s[i] = renorm_shift(low[i], high, size);
                } else {
                    s[i] = renorm_shift(low[i], high, u[i]);
                }
                p[i] = st[i].p + static_cast<int32_t>(s[i]);
                beyond |= p[i];
            }
            if (cg_any_lane(lanes, rare | ((beyond & ~31) != 0) | (t4 == last4))) break;
            emit(a, t4);
            t4 += 4u;
            CG_UNROLL
            for (int i = 0; i < NS; ++i) {
                st[i].low = cg_fshl(0u, low[i], s[i]);
                st[i].span32 = cg_fshl(0u, u[i], s[i]);
                st[i].p = p[i];
                bits[i] = bw[i].bits(st[i].p);
                const uint32_t offset = bits[i] - st[i].low;
                ratio[i] = QUICK ? ratio_estimate(offset, st[i].span32, reciprocal[i], s[i]) : ratio_estimate(offset, st[i].span32);
            }
        }
        odd = cg_any_lane(lanes, rare);
        if (!odd) {
            emit(a, t4);
            if (t4 == last4) break;
            t4 += 4u;
            CG_UNROLL
            for (int i = 0; i < NS; ++i) {
                st[i].low = cg_fshl(0u, low[i], s[i]);
                st[i].span32 = cg_fshl(0u, u[i], s[i]);
                st[i].p = p[i];
            }
        }
    }
}

// One stream.  col: address of the stream's table column (see search_entry), rows kTableRowBytes apart,
// 2^LEVELS + 1 of them readable, 2^LEVELS >= maxsym + 1; emit(a) receives, token after token, the address of the
// decoded symbol's table entry (symbol = (a - col) / kTableRowBytes).  lanes: the warp's lanes that
// run this loop together (they must all have the same ntok).
template <int LEVELS, class Emit>
CG_HD void decode_stream(Smem sm, uint32_t col, int maxsym, const uint8_t *stream, uint32_t len, int ntok,
                         uint32_t lanes, Emit emit) {
    const uint32_t cols[1] = {col}, lens[1] = {len};
    const uint8_t *const streams[1] = {stream};
    const int top = (1 << LEVELS) - 1;
    const uint32_t det = col + static_cast<uint32_t>(top < maxsym ? top : maxsym) * kTableRowBytes;
    decode_streams<LEVELS, 1>(sm, cols, det, maxsym, LEVELS, streams, lens, ntok, lanes,
                              [&](const uint32_t(&a)[1], uint32_t) { emit(a[0]); });
}

// ---- MSB-first bit writer into one scratch row (add_bits_to_output, enc_new.cu:21-97) ---------------------
// Output bits collect in a 64-bit accumulator.  Whole 32-bit words leave it, big-endian, into the
// stream's scratch row; the common case does that for the whole warp at once (see EncoderState::steps_at)
// so that the store is not a per-lane branch.
//
// The bits are those of the interval's lower end as one long binary fraction, so a later range update can
// still carry into bits that are already here, and out of them into the word before.  That word is held back in a
// register until the next one leaves: the run of ones that lets a carry through reaches the accumulator's end
// for one word in seven (symbols of 2.5 bits), but past the held word about never.  (With carries added to words
// already stored the per-lane read-modify-write ran on 15 % of the word stores.)  Bits that have left as a word
// stay in the accumulator above the pending ones until they are shifted out, and a carry goes on into
// them; the last bit of the held word is one of them, so it has changed exactly if the word is to be one more.
// STEP: words between consecutive words of the row (32: the rows of a warp's streams interleaved, so that
// they take no more cache lines than they have data for and are read back coalesced).  BOUNDED: the row may be
// too short for the stream; otherwise it holds CG_STREAM_CAPACITY bytes, which a strictly increasing table
// never exceeds, and the word in front of its first may be overwritten.
template <int STEP, bool BOUNDED = true>
struct BitSinkT {
    uint32_t *row;    // 4-byte aligned scratch row of this stream
    uint32_t cap_w;   // words that fit in the row
    uint32_t nwords;  // words produced so far, the held one included (may exceed cap_w: then nothing more is stored)
    uint32_t hold;    // the last of them, not yet in the row
    uint32_t acc_hi, acc_lo;  // pending output bits, right-aligned in (acc_hi:acc_lo), older bits above them
    int nacc;                 // number of bits pending, < 64 in front of a symbol (see store_word_if_full); -1: see EncoderState::half_scale

    // p: where the stream's first word goes; nbytes: room for the stream
    CG_HD void init(uint8_t *p, int64_t nbytes) {
        row = reinterpret_cast<uint32_t *>(p);
        cap_w = static_cast<uint32_t>(nbytes >> 2);
        nwords = 0;
        hold = 0;
        acc_hi = 0;
        acc_lo = 0;
        nacc = 0;
    }
    // adds one to the number that the first n words in the row form
    CG_HD void carry_into_row(uint32_t n) {
        if (BOUNDED && n > cap_w) return;  // they are not in the row: reported as an overflow
        for (; n > 0u; --n) {
            const uint32_t v = cg_bswap32(row[(n - 1u) * STEP]) + 1u;
            row[(n - 1u) * STEP] = cg_bswap32(v);
            if (v) return;
        }
    }
    // Moves the oldest 32 pending bits out where there are 32; needs nacc < 64.  Straight-line code: every lane of the
    // warp runs it whatever it needs.  Returns whether the held word, which went to the row (as number nwords - 2 now), has
    // carried into those in front of it, which is left to the caller.
    // DEEP: up to 63 bits were pending before the last shift, by s <= 31, which moved bits out of the accumulator: `above` is
    // its upper word before that shift.
    template <bool DEEP = false>
    CG_HD bool store_word_if_full(uint32_t above = 0u, uint32_t s = 0u) {
#if defined(__CUDA_ARCH__)
        uint32_t w, held, carry, left;
        if (DEEP)
        asm("{ .reg .pred p, q; .reg .u32 lo, hi, x;\n"
            "add.u32 %3, %6, -32;\n"
            "setp.ge.s32 p, %6, 32;\n"
            "setp.ge.s32 q, %6, 64;\n"
            "shf.l.wrap.b32 x, %8, 0, %9;\n"    // the bits above the accumulator
            "selp.b32 lo, %5, %4, q;\n"
            "selp.b32 hi, x, %5, q;\n"
            "shf.r.wrap.b32 %0, lo, hi, %3;\n"
            "shf.r.wrap.b32 %2, hi, 0, %3;\n"
            "lop3.b32 %2, %2, %7, 1, 0x28;\n"
            "@!p mov.u32 %2, 0;\n"
            "add.u32 %1, %7, %2; }"
            : "=&r"(w), "=&r"(held), "=&r"(carry), "=&r"(left) : "r"(acc_lo), "r"(acc_hi), "r"(nacc), "r"(hold), "r"(above), "r"(s));
        else
        asm("{ .reg .pred p;\n"
            "add.u32 %3, %6, -32;\n"
            "setp.ge.s32 p, %6, 32;\n"
            "shf.r.clamp.b32 %0, %4, %5, %3;\n"  // the low word of (hi:lo) >> left
            "shf.r.clamp.b32 %2, %5, 0, %3;\n"
            "lop3.b32 %2, %2, %7, 1, 0x28;\n"    // (acc_hi >> left ^ hold) & 1
            "@!p mov.u32 %2, 0;\n"
            "add.u32 %1, %7, %2; }"
            : "=&r"(w), "=r"(held), "=&r"(carry), "=&r"(left) : "r"(acc_lo), "r"(acc_hi), "r"(nacc), "r"(hold));
        const bool room = !BOUNDED || nwords - 1u < cap_w;
        asm volatile("{ .reg .pred p, q;\n"
            "setp.ge.s32 p, %2, 32;\n"
            "setp.ne.and.u32 q, %7, 0, p;\n"
            "@q st.global.u32 [%3], %4;\n"
            "@p add.u32 %0, %0, 1;\n"
            "@p mov.u32 %1, %5;\n"
            "@p mov.u32 %2, %6; }"
            : "+r"(nwords), "+r"(hold), "+r"(nacc)
            : "l"(row + static_cast<int>(nwords - 1u) * STEP), "r"(cg_bswap32(held)), "r"(w), "r"(left), "r"(static_cast<uint32_t>(room)) : "memory");
        return held < carry;
#else
        if (nacc < 32) return false;
        nacc -= 32;
        const uint32_t left = static_cast<uint32_t>(nacc) & 31u, x = s & 31u ? above >> (32u - (s & 31u)) : 0u;
        const bool q = DEEP && nacc >= 32;
        const uint32_t carry = (((q ? x : acc_hi) >> left) ^ hold) & 1u;
        hold += carry;
        const bool over = hold < carry;
        if (nwords && (!BOUNDED || nwords - 1u < cap_w)) row[(nwords - 1u) * STEP] = cg_bswap32(hold);
        ++nwords;
        hold = q ? cg_fshr_clamp(acc_hi, x, left) : cg_fshr_clamp(acc_lo, acc_hi, left);
        return over;
#endif
    }
    CG_HD void store_and_carry() {
        if (store_word_if_full()) carry_into_row(nwords - 2u);
    }
    // zero-fills to a byte boundary; returns the stream length in bytes
    CG_HD uint32_t finish() {
        if (nacc > 62) nacc = 62;  // only a table that does not increase gets here, or below
        if (nacc < 0) nacc = 0;
        store_and_carry();
        if (nwords) {
            const uint32_t carry = ((acc_lo >> nacc) ^ hold) & 1u;
            hold += carry;
            if (hold < carry) carry_into_row(nwords - 1u);
            if (!BOUNDED || nwords - 1u < cap_w) row[static_cast<int>(nwords - 1u) * STEP] = cg_bswap32(hold);
        }
        const uint32_t bytes = nwords * 4u + ((static_cast<uint32_t>(nacc) + 7u) >> 3);
        if (nacc) {
            const uint32_t w = acc_lo << (32 - nacc);
            if (!BOUNDED || nwords < cap_w) row[nwords * STEP] = cg_bswap32(w);
        }
        return bytes;
    }
};

using BitSink = BitSinkT<1>;

// ---- encoder state and step -----------------------------------------------------------------------------
// Pending bits from which on a lane makes its warp store a word.  Whatever stays below it, or below 32 after the store, has
// to take `symbols` more symbols' bits below bit 63.  A symbol adds at most 18 (the updated interval of a
// strictly increasing table spans at least 2^14 values).  These are the marks of a store without the upper word; the kernels
// use those below, and of pair_high_water only whether it is 0.
constexpr int kSinkHighWater = 44;
// The same where the table was counted from the `ntokens` symbols that are coded with it: a symbol that occurs has at
// least w = floor((0xFFFF - 63) / ntokens) + 1 of the 2^16 shares (normalize_cdf_value), hence an interval of
// w * 2^14 - 1 values or more, and adds at most 18 - floor(log2 w) bits.  0: two symbols may not fit.
CG_HD int counted_symbol_bits(int ntokens) {
    const uint32_t w = (0xFFFFu - 63u) / static_cast<uint32_t>(ntokens) + 1u;
    return 18 - (31 - cg_clz(w));
}
CG_HD int pair_high_water(int ntokens) {
    const int most = counted_symbol_bits(ntokens);
    if (31 + 2 * most > 63) return 0;
    return 64 - 2 * most < kSinkHighWater ? 64 - 2 * most : kSinkHighWater;
}
// Marks where the last symbol in front of a vote may shift pending bits out of the accumulator, because its upper word from
// before that shift is kept (store_word_if_full<true>): only what the symbols before it add has to stay below bit 64.  For two
// symbols of 256 counted tokens 54 instead of 44, for one of any table 64: a stream that has not got a whole word when another is at
// the mark is soon the next one there, so a word's store every 13 bits of the fastest of a warp's streams becomes one every 22.
// The first only where pair_high_water is not 0: what a store leaves is below it then, too.
CG_HD int deep_pair_high_water(int ntokens) { return 64 - counted_symbol_bits(ntokens); }
constexpr int kDeepHighWater = 64;

// The coder without the reference's count of pending bits.  low is the current 32-bit window of the
// interval's lower end L, and all bits of L above the window are in the sink: a range update adds to
// low and carries into the sink, a shift by s moves low's top s bits there.  The reference's underflow
// shifts (low = 01..., high = 10...: drop the second bit, remember one pending bit) are the same
// shift: the bits they leave open are 01..1 in L here, with the last 1 as low's top bit, and become
// 10..0 by the carry exactly when the reference decides for a 1 followed by zeros.
struct EncoderState {
    uint32_t low, span32;  // span32 = (high - low + 1) mod 2^32, 0 for the full range
    CG_HD void init() {
        low = 0u;
        span32 = 0u;
    }
    // The full range of 2^32 does not fit span32.  It is taken at half scale: a window that takes one bit back from the
    // sink (at a stream's start the integer bit of L, which stays 0).  Bounds are exact there, and the next
    // renormalisation shifts by one more.  What uses steps_at starts so.
    template <class Sink>
    CG_HD void half_scale(Sink &out) {
        low = cg_fshl(low, out.acc_lo, 31u);
        out.acc_lo = cg_fshl(out.acc_lo, out.acc_hi, 31u);
        out.acc_hi >>= 1;
        span32 = 0x80000000u;
        --out.nacc;
    }
    template <class Sink>
    CG_HD void add_to_low(uint32_t v, Sink &out) {
#if defined(__CUDA_ARCH__)
        uint32_t l, a, b;
        asm("add.cc.u32 %0, %3, %6; addc.cc.u32 %1, %4, 0; addc.u32 %2, %5, 0;"
            : "=&r"(l), "=&r"(a), "=r"(b) : "r"(low), "r"(out.acc_lo), "r"(out.acc_hi), "r"(v));
        low = l;
        out.acc_lo = a;
        out.acc_hi = b;
#else
        low += v;
        if (low < v && ++out.acc_lo == 0u) ++out.acc_hi;
#endif
    }
    // Range update for the symbol whose scaled bounds are [flo, fhi), then renormalisation, by the interval's size (see
    // renorm_shift) or, EXACT, by its size less one.
    // Returns the shift; above: the accumulator's upper word before it.
    template <bool EXACT, class Sink>
    CG_HD uint32_t take(uint32_t flo, uint32_t fhi, Sink &out, uint32_t &above) {
        const uint32_t u = fhi - flo;
        add_to_low(flo, out);
        const uint32_t s = renorm_shift(low, cg_add_less_one(low, u), EXACT ? u - 1u : u);
        above = out.acc_hi;
        shift(s, u, out);
        return s;
    }
    template <class Sink>
    CG_HD void shift(uint32_t s, uint32_t u, Sink &out) {
        out.acc_hi = cg_fshl(out.acc_lo, out.acc_hi, s);
        out.acc_lo = cg_fshl(low, out.acc_lo, s);
        low = cg_fshl(0u, low, s);
        span32 = cg_fshl(0u, u, s);
        out.nacc += static_cast<int>(s);
    }
    // One symbol by the address a of its table entry, the next one ROW bytes further (enc_new.cu:257-295): whatever the
    // state, by one lane alone.
    template <int ROW, class Sink>
    CG_HD void step_alone(Smem sm, uint32_t a, bool last, Sink &out) {
        out.store_and_carry();
        if (span32 == 0u) half_scale(out);
        const uint32_t flo = cg_umulhi_wide(span32, sm.ld(a));
        uint32_t above;
        take<true>(flo, last ? span32 : cg_umulhi_wide(span32, sm.ld(a + ROW)), out, above);
    }
    // G symbols (1 or 2) of NS streams a lane, by the addresses of their table entries.  The streams' chains are independent,
    // and ONE warp vote after them covers a full word in an accumulator: every lane that has one stores it as soon as one
    // lane is at the high-water mark: with DEEP, as the kernels run it, kDeepHighWater for one symbol and deep_pair_high_water for
    // two, without it kSinkHighWater and pair_high_water.
    // LAST: a symbol may be its table's last, whose upper bound is the range's end (told by `last`; G is 1 then).
    // What hardly ever happens is not mended here but left to encode_again: a carry through a whole word of ones
    // (`carried`), and a range of 2^31 at a multiple of it, which leaves a span of 0, from where on no symbol has a size, so
    // that the span is still 0 at the stream's end.  Code for the like inside the loop cost five executed instructions a
    // symbol without ever being run.
    template <int ROW, int G, int NS, bool LAST = false, bool DEEP = false, class Sink>
    static CG_HD void steps_at(Smem sm, const uint32_t (&a)[G][NS], EncoderState (&enc)[NS], Sink (&out)[NS], int high_water,
                               uint32_t lanes, bool (&carried)[NS], bool last = false) {
        uint32_t e0[G][NS], e1[G][NS], s[NS], above[NS];
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
            for (int i = 0; i < NS; ++i) {
                e0[g][i] = sm.ld(a[g][i]);
                e1[g][i] = sm.ld(a[g][i] + ROW);
            }
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
            for (int i = 0; i < NS; ++i) {
                const uint32_t fhi = cg_umulhi_wide(enc[i].span32, e1[g][i]);
                s[i] = enc[i].template take<false>(cg_umulhi_wide(enc[i].span32, e0[g][i]), LAST && last ? enc[i].span32 : fhi, out[i], above[i]);
            }
        bool full = false;
#pragma unroll
        for (int i = 0; i < NS; ++i) full |= out[i].nacc >= high_water;
        if (cg_any_lane(lanes, full)) {
#pragma unroll
            for (int i = 0; i < NS; ++i) carried[i] |= out[i].template store_word_if_full<DEEP>(above[i], s[i]);
        }
    }
    // whether a stream has met what steps_at leaves
    CG_HD bool unsettled(bool carried) const { return carried | (span32 == 0u); }
    // final flush (enc_new.cu:298-306): two bits that place the stream's value inside the interval, 01 or
    // 10 above the reference's low with its pending bits, which is L plus a quarter of the window cut
    // to two bits; returns the stream length in bytes
    template <class Sink>
    CG_HD uint32_t flush(Sink &out) {
        out.store_and_carry();
        if (span32) shift(renorm_shift(low, cg_add_less_one(low, span32), span32 - 1u), span32, out);  // see take: two bits at most
        add_to_low(0x40000000u, out);
        out.acc_hi = cg_fshl(out.acc_lo, out.acc_hi, 2u);
        out.acc_lo = cg_fshl(low, out.acc_lo, 2u);
        out.nacc += 2;
        return out.finish();
    }
};

}  // namespace cg
