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
//     leading-bit search (renorm_shift), the decoder takes all its new bits in one funnel shift and the
//     encoder appends the shifted-out top bits of `low` at once, carries included.
#pragma once

#include <stdint.h>

#if defined(__CUDACC__)
#define CG_HD __host__ __device__ __forceinline__
#else
#define CG_HD inline
#endif

namespace cg {

constexpr int kGroupChannels = 128;            // streams (threads) per coder block
constexpr int kTableRowBytes = kGroupChannels * 4;  // bytes between table entries m and m+1 of a stream

// ---- intrinsics with host stand-ins -----------------------------------------------------------------
CG_HD int cg_clz(uint32_t x) {
#if defined(__CUDA_ARCH__)
    return __clz(static_cast<int>(x));
#else
    return x ? __builtin_clz(x) : 32;
#endif
}
// x << n, 0 for n >= 32.  On the device a clamping funnel shift: a plain `<<` by 32 or more is undefined.
CG_HD uint32_t cg_shl(uint32_t x, uint32_t n) {
#if defined(__CUDA_ARCH__)
    return __funnelshift_lc(0u, x, n);
#else
    return n >= 32u ? 0u : x << n;
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
// By the size u = d + 1 instead of d (the encoder's loop): the top bit is another one only where u is a power of two, and
// s one or two less than it could be where low is a multiple of u or of u / 2 as well.  Nothing is lost by that: the next
// symbol's bounds are exact at any scale of such a range, and its shift makes up for it; and the full range of 2^32, which
// no word holds, does not come about.  (Only u = 2^31 at a multiple of 2^31 gives -1: see EncoderState::steps_at.)
//
// Returns s and 2^s: for the words that are only shifted left a multiply does it off the integer pipe (a
// shift, a compare or a select takes that pipe for two cycles a warp, and a multiply-high the multiply pipe for four).
//
// The conditional decrement is written as a predicated add: with `if (...) --s` the counters show two executed
// instructions a symbol more.
struct Renorm {
    uint32_t s, p2;
};
// low, high = low + d, d (or u)
CG_HD Renorm renorm_shift(uint32_t low, uint32_t high, uint32_t d) {
    Renorm r;
#if defined(__CUDA_ARCH__)
    asm("{ .reg .u32 t, b; .reg .pred p;\n"
        "bfind.shiftamt.u32 %0, %4;\n"
        "shf.r.wrap.b32 b, 0x80000000, 0, %0;\n"
        "lop3.b32 t, %2, %3, b, 0x28;\n"  // (low ^ high) & b
        "setp.eq.u32 p, t, 0;\n"
        "@p add.u32 %0, %0, -1;\n"
        "shf.l.wrap.b32 %1, 0, 1, %0; }"
        : "=&r"(r.s), "=r"(r.p2) : "r"(low), "r"(high), "r"(d));
#else
    r.s = d ? static_cast<uint32_t>(cg_clz(d)) : 0xFFFFFFFFu;
    if (((low ^ high) & (0x80000000u >> (r.s & 31u))) == 0u) --r.s;
    r.p2 = 1u << (r.s & 31u);
#endif
    return r;
}

// ---- register bit window + warp-synchronous refill -----------------------------------------------------------
// The next 96 unread bits of the stream live in three registers.  The byte array is read as aligned
// 32-bit words; bits before the stream's first byte are shifted out at start-up and words (or word
// tails) past its last byte read as zero, which is what the reference sees in its zero-padded staging
// row (dec_new.cu:229-232).  A refill is taken by the whole warp as soon as any of its lanes has fewer
// bits than a symbol can take and gives a word to every lane with room for one, so the refill code runs once per warp every
// few symbols instead of once per lane.
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
// The same as the upper half of a wide product: the encoder's step, which adds to it, executes two instructions fewer so.
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

struct BitWindow {
    const uint32_t *wp;    // word holding the stream's first byte
    uint32_t end_bit;      // bit index, counted from wp, one past the stream's last bit
    uint32_t next;         // next word to fetch
    uint32_t hi, mid, lo;  // unread bits, hi's top bit first
    int nbits;             // valid bits in hi:mid:lo

    // word j of the stream, big-endian, bits past the stream's end cleared; no branches
    CG_HD uint32_t fetch(uint32_t j) const {
        const uint32_t b0 = j * 32u;
        uint32_t w = 0u;
        if (b0 < end_bit) w = cg_bswap32(cg_load_stream_word(wp + j));
        const uint32_t rem = end_bit - b0;  // >= 2^31 (clamped to 32 below) when the word lies past the end
        return w & ~cg_fshr_clamp(0xFFFFFFFFu, 0u, rem);
    }
    // returns the stream's first 32 bits (the coder's initial `value`, dec_new.cu:257)
    CG_HD uint32_t open(const uint8_t *p, uint32_t len) {
        const uintptr_t a = reinterpret_cast<uintptr_t>(p);
        wp = reinterpret_cast<const uint32_t *>(a & ~static_cast<uintptr_t>(3));
        const uint32_t off = static_cast<uint32_t>(a & 3u) * 8u;
        end_bit = off + len * 8u;
        const uint32_t w0 = fetch(0), w1 = fetch(1), w2 = fetch(2), w3 = fetch(3);
        hi = cg_fshl(w2, w1, off);
        mid = cg_fshl(w3, w2, off);
        lo = w3 << off;
        nbits = 96 - static_cast<int>(off);
        next = 4;
        return cg_fshl(w1, w0, off);
    }
    // drops the bits just shifted into the coder's value
    CG_HD void consume(Renorm r) {
        hi = cg_fshl(mid, hi, r.s);
        mid = cg_fshl(lo, mid, r.s);
        lo *= r.p2;
        nbits -= static_cast<int>(r.s);
    }
    CG_HD bool low_water() const { return nbits <= 32; }
    // fewer valid bits than one symbol can take: a range update shifts by at most 18 bits when the
    // table is strictly increasing (the updated interval spans at least 2^14 values)
    static constexpr int kShort = 18;
    CG_HD bool short_of_bits() const { return nbits < kShort; }
    // Takes the next word where one fits above 32 bits of room (a stream short of bits has 32 or more afterwards),
    // straight-line: every lane of the warp runs the same instructions whatever it needs.
    // Written in predicated instructions (see renorm_shift): filling up to two words a pass with selects took
    // 4.7 instructions a symbol of the fused decode at 0.055 passes a token; one word, 0.09 passes, takes 1.6.
    CG_HD void refill() {
#if defined(__CUDA_ARCH__)
        asm("{ .reg .u32 w, rem, t, b; .reg .u64 at; .reg .pred p, q, a;\n"
            "setp.lt.s32 p, %3, 64;\n"
            "mad.lo.u32 rem, %4, -32, %6;\n"     // bits of the stream from this word on, negative past its end
            "mad.wide.u32 at, %4, 4, %5;\n"
            "mov.u32 w, 0;\n"
            "setp.gt.and.s32 q, rem, 0, p;\n"
            "@q ld.global.nc.u32 w, [at];\n"
            "prmt.b32 w, w, 0, 0x0123;\n"
            "shr.u32 t, 0xFFFFFFFF, rem;\n"      // (a shift by more than 31 gives 0)
            "lop3.b32 w, w, t, 0, 0x30;\n"       // w & ~t
            "shf.r.wrap.b32 t, w, 0, %3;\n"      // the word's upper part, behind the valid bits of their last word
            "shf.r.wrap.b32 b, 0, w, %3;\n"      // and what goes into the word after that
            "setp.lt.s32 a, %3, 32;\n"
            "@a or.b32 %0, %0, t;\n"
            "@a or.b32 %1, %1, b;\n"
            "@!a or.b32 %1, %1, t;\n"
            "@!a or.b32 %2, %2, b;\n"
            "@p add.s32 %3, %3, 32;\n"
            "@p add.u32 %4, %4, 1; }"
            : "+r"(hi), "+r"(mid), "+r"(lo), "+r"(nbits), "+r"(next) : "l"(wp), "r"(end_bit));
#else
        if (nbits >= 64) return;
        const uint32_t w = fetch(next++), p = static_cast<uint32_t>(nbits) & 31u, t = w >> p, b = p ? w << (32u - p) : 0u;
        if (nbits < 32) {
            hi |= t;
            mid |= b;
        } else {
            mid |= t;
            lo |= b;
        }
        nbits += 32;
#endif
    }
};

// ---- decode loop ------------------------------------------------------------------------------------------
// Scaled table entry for the current span: (span * c16) >> 32 with span32 = span mod 2^32, which is 0
// exactly when the range is the full 2^32 (then the product is c16 itself).
CG_HD uint32_t scale_exact(uint32_t span32, uint32_t c16) { return span32 ? cg_umulhi(span32, c16) : c16; }

// The decoder's arithmetic state: low, span32 = (high - low + 1) mod 2^32 and offset = value - low.
// In this form both kinds of renormalisation shift act alike on the pair (offset, span) --
// offset = 2*offset + next bit, span = 2*span -- so the reference's "value -= 2^30" of the underflow
// case needs no separate step; low is still tracked because the shift counts depend on the bit
// patterns of low and high.
struct DecoderState {
    uint32_t low, span32, offset;

    // range update for the symbol whose scaled bounds are [flo, fhi), then renormalisation
    // (dec_new.cu:277-301), both kinds of shift applied in one go.  On a table that is not increasing the
    // shift count is anything up to 31; every later read stays inside the table column and the stream.
    CG_HD void update(uint32_t flo, uint32_t fhi, BitWindow &bw) {
        offset -= flo;
        low += flo;
        span32 = fhi - flo;
        const uint32_t d = span32 - 1u;
        const Renorm r = renorm_shift(low, low + d, d);
        low = cg_fshl(0u, low, r.s);
        span32 = cg_fshl(0u, span32, r.s);
        offset = cg_fshl(bw.hi, offset, r.s);
        bw.consume(r);
    }
};

// ---- decode loop: NS streams per lane, search depth chosen by the caller ---------------------------------
// Table entries as the search takes them: 2^23 (1 + cdf / 2^16) as a float.  Its bits shifted by nine are cdf << 16, and
// a comparison with an estimate of 2^23 (1 + offset / span) + 1, which is as whole a number, is the difference cut to
// [0, 1], which is 0 or 1.  A search step is then a subtraction with saturation and a multiply-add on the entry's address
// (taken as a denormal float, which adds like an integer): both on the two floating-point pipes, where a compare and a
// predicated add go to the integer pipes, which have half the rate and bind the loop.  8,192 Llama-7B tokens: 4.18 ms with
// integer entries.
CG_HD uint32_t search_entry(uint32_t cdf) { return 0x4B000000u | cdf << 7; }
constexpr uint32_t kSearchPadding = 0x7F800000u;  // +inf: above every estimate
CG_HD uint32_t ld_entry(Smem sm, uint32_t addr) {
#if defined(__CUDA_ARCH__)
    return sm.ld(addr);
#else
    const uint32_t v = sm.ld(addr);  // the host's columns hold cdf << 16, padded with 0xFFFFFFFF
    return v == 0xFFFFFFFFu ? kSearchPadding : search_entry(v >> 16);
#endif
}
CG_HD uint32_t entry_c16(uint32_t entry) { return cg_fshl(0u, entry, 9u); }  // cdf << 16

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

// 2^23 (1 + offset / span) + 1, to about 2 (see search_entry); anything when the span is the full 2^32 (span32 == 0).
CG_HD float ratio_estimate(uint32_t offset, uint32_t span32) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint2float_rn(span32)));
    return __fmaf_rn(__uint2float_rn(offset), r * 8388608.0f, 8388609.0f);
#else
    return span32 ? static_cast<float>(offset) * (8388608.0f / static_cast<float>(span32)) + 8388609.0f : 8388609.0f;
#endif
}
// address a, or a + STEP if the entry is not above the ratio
template <uint32_t STEP>
CG_HD uint32_t search_step(uint32_t a, uint32_t entry, float ratio) {
#if defined(__CUDA_ARCH__)
    float take;
    asm("sub.rn.sat.f32 %0, %1, %2;" : "=f"(take) : "f"(ratio), "f"(__uint_as_float(entry)));
    return __float_as_uint(__fmaf_rn(take, __uint_as_float(STEP), __uint_as_float(a)));
#else
    float e;
    __builtin_memcpy(&e, &entry, 4);
    return ratio - e >= 1.0f ? a + STEP : a;
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

// NS streams of one lane decoded side by side (same token count, same table length), the fast
// search limited to the first 2^FL table entries.
//
// The fast search compares the table entries with an estimate of offset / span, which costs one compare a
// level where the scaled entry costs a multiply-high as well (four cycles of the multiply pipe and two of the
// integer pipe a warp, measured).  The symbol is then checked exactly: the offset must lie inside its scaled
// bounds, which the range update needs anyway.  The caller picks FL from what it knows about the symbols (a
// row quantised to `bins` bins holds symbols 0 .. bins-2, so 2^FL >= bins is enough).  The result depends
// on neither: a symbol that fails the check -- an estimate on the wrong side of an entry, a symbol >= 2^FL - 1, a symbol that starts from the full 2^32 range (its scaled bounds are both 0) -- is thrown away
// and the whole warp repeats that symbol with the exact, full-depth search.
//
// The table's last symbol has no upper entry.  With LAST_REPEATED the rows above its entry hold copies of it,
// so that its bounds are equal and the check fails; otherwise they hold kSearchPadding and
// a symbol at or above the address threshold det is repeated as well.  The column needs 2^FL + 1
// readable rows either way.
//   col[i]    table column of stream i (see decode_stream)
//   det       address threshold of entry min(2^FL - 1, maxsym): column-independent because a column's offset
//             inside a table row is below kTableRowBytes (det = table base + entry * kTableRowBytes)
//   emit(a, t4)  receives the NS table-entry addresses of one token's symbols and four times the
//             token's index (ntok >= 1)
template <int FL, int NS, bool LAST_REPEATED = false, class Emit>
CG_HD void decode_streams(Smem sm, const uint32_t (&col)[NS], uint32_t det, int maxsym, int full_levels,
                          const uint8_t *const (&stream)[NS], const uint32_t (&len)[NS], int ntok, uint32_t lanes,
                          Emit emit) {
    static_assert(FL >= 2, "the first level's entry is held in a register");
    BitWindow bw[NS];
    DecoderState st[NS];
    uint32_t mid[NS], a_max[NS];
    constexpr uint32_t kTop = static_cast<uint32_t>(kTableRowBytes) << (FL - 1);
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int i = 0; i < NS; ++i) {
        st[i].low = 0u;
        st[i].span32 = 0u;
        st[i].offset = bw[i].open(stream[i], len[i]);
        a_max[i] = col[i] + static_cast<uint32_t>(maxsym) * kTableRowBytes;
        mid[i] = ld_entry(sm, col[i] + kTop);
    }
    uint32_t a[NS], flo[NS], fhi[NS];
    const uint32_t last4 = static_cast<uint32_t>(ntok - 1) * 4u;
    uint32_t t4 = 0u;  // four times the token index: the caller's emit indexes 4-byte per-token data with it
    // The inner loop is the common case and nothing else, left by one vote for a refill of the bit windows, for a
    // symbol whose fast search failed and at the last token; with that code inside it, every pass executed more
    // instructions, whether it took that code or not.
    for (;;) {
#if defined(__CUDA_ARCH__)
#pragma unroll 1
#endif
        for (;;) {
            float ratio[NS];
            bool rare = false;  // a symbol that fails the check
            int fewest = bw[0].nbits;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
            for (int i = 0; i < NS; ++i) {
                ratio[i] = ratio_estimate(st[i].offset, st[i].span32);
                a[i] = search_step<kTop>(col[i], mid[i], ratio[i]);
            }
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
            for (int i = 0; i < NS; ++i) a[i] = RatioSearch<FL - 2>::run(sm, a[i], ratio[i]);
            uint32_t e0[NS], e1[NS];
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
            for (int i = 0; i < NS; ++i) {
                e0[i] = entry_c16(ld_entry(sm, a[i]));
                e1[i] = entry_c16(ld_entry(sm, a[i] + kTableRowBytes));
            }
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
            for (int i = 0; i < NS; ++i) {
                flo[i] = cg_umulhi(st[i].span32, e0[i]);
                fhi[i] = cg_umulhi(st[i].span32, e1[i]);
                rare = rare | (st[i].offset - flo[i] >= fhi[i] - flo[i]);
                fewest = fewest < bw[i].nbits ? fewest : bw[i].nbits;
                if (!LAST_REPEATED) rare = rare | (a[i] >= det);
            }
            if (cg_any_lane(lanes, rare | (fewest < BitWindow::kShort) | (t4 == last4))) break;
            emit(a, t4);
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
            for (int i = 0; i < NS; ++i) st[i].update(flo[i], fhi[i], bw[i]);
            t4 += 4u;
        }
        if (t4 == last4) break;
        bool low = false, odd = false;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
        for (int i = 0; i < NS; ++i) {
            low = low || bw[i].short_of_bits();
            odd = odd || st[i].offset - flo[i] >= fhi[i] - flo[i];
            if (!LAST_REPEATED) odd = odd || a[i] >= det;
        }
        if (cg_any_lane(lanes, low)) {
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
            for (int i = 0; i < NS; ++i) bw[i].refill();
        }
        if (cg_any_lane(lanes, odd)) {
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
            for (int i = 0; i < NS; ++i) {
                a[i] = exact_search(sm, col[i], a_max[i], st[i].span32, st[i].offset, full_levels);
                flo[i] = scale_exact(st[i].span32, entry_c16(ld_entry(sm, a[i])));
                fhi[i] = (a[i] == a_max[i]) ? st[i].span32
                                            : scale_exact(st[i].span32, entry_c16(ld_entry(sm, a[i] + kTableRowBytes)));
            }
        }
        emit(a, t4);
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
        for (int i = 0; i < NS; ++i) st[i].update(flo[i], fhi[i], bw[i]);
        t4 += 4u;
    }
    // last symbol: no range update (dec_new.cu:273-275), so no new bits either
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int i = 0; i < NS; ++i) a[i] = exact_search(sm, col[i], a_max[i], st[i].span32, st[i].offset, full_levels);
    emit(a, t4);
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
    int nacc;                 // number of bits pending, < 64; -1: see EncoderState::half_scale

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
    CG_HD bool store_word_if_full() {
#if defined(__CUDA_ARCH__)
        uint32_t w, held, carry, left;
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
        const uint32_t carry = ((acc_hi >> nacc) ^ hold) & 1u;
        hold += carry;
        const bool over = hold < carry;
        if (nwords && (!BOUNDED || nwords - 1u < cap_w)) row[(nwords - 1u) * STEP] = cg_bswap32(hold);
        ++nwords;
        hold = cg_fshr_clamp(acc_lo, acc_hi, static_cast<uint32_t>(nacc));
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
// strictly increasing table spans at least 2^14 values).
constexpr int kSinkHighWater = 44;
// The same where the table was counted from the `ntokens` symbols that are coded with it: a symbol that occurs has at
// least w = floor((0xFFFF - 63) / ntokens) + 1 of the 2^16 shares (normalize_cdf_value), hence an interval of
// w * 2^14 - 1 values or more, and adds at most 18 - floor(log2 w) bits.  0: two symbols may not fit.
CG_HD int pair_high_water(int ntokens) {
    const uint32_t w = (0xFFFFu - 63u) / static_cast<uint32_t>(ntokens) + 1u;
    const int most = 18 - (31 - cg_clz(w));
    if (31 + 2 * most > 63) return 0;
    return 64 - 2 * most < kSinkHighWater ? 64 - 2 * most : kSinkHighWater;
}

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
    template <bool EXACT, class Sink>
    CG_HD void take(uint32_t flo, uint32_t fhi, Sink &out) {
        const uint32_t u = fhi - flo;
        add_to_low(flo, out);
        shift(renorm_shift(low, cg_add_less_one(low, u), EXACT ? u - 1u : u), u, out);
    }
    template <class Sink>
    CG_HD void shift(Renorm r, uint32_t u, Sink &out) {
        out.acc_hi = cg_fshl(out.acc_lo, out.acc_hi, r.s);
        out.acc_lo = cg_fshl(low, out.acc_lo, r.s);
        low *= r.p2;
        span32 = u * r.p2;
        out.nacc += static_cast<int>(r.s);
    }
    // One symbol by the address a of its table entry, the next one ROW bytes further (enc_new.cu:257-295): whatever the
    // state, by one lane alone.
    template <int ROW, class Sink>
    CG_HD void step_alone(Smem sm, uint32_t a, bool last, Sink &out) {
        out.store_and_carry();
        if (span32 == 0u) half_scale(out);
        const uint32_t flo = cg_umulhi_wide(span32, sm.ld(a));
        take<true>(flo, last ? span32 : cg_umulhi_wide(span32, sm.ld(a + ROW)), out);
    }
    // G symbols (1 or 2) of NS streams a lane, by the addresses of their table entries.  The streams' chains are independent,
    // and ONE warp vote after them covers a full word in an accumulator: every lane that has one stores it as soon as one
    // lane is at the high-water mark (kSinkHighWater for one symbol, pair_high_water for two).
    // LAST: a symbol may be its table's last, whose upper bound is the range's end (told by `last`; G is 1 then).
    // What hardly ever happens is not mended here but left to encode_again: a carry through a whole word of ones
    // (`carried`), and a range of 2^31 at a multiple of it, which leaves a span of 0, from where on no symbol has a size, so
    // that the span is still 0 at the stream's end.  Code for the like inside the loop cost five executed instructions a
    // symbol without ever being run.
    template <int ROW, int G, int NS, bool LAST = false, class Sink>
    static CG_HD void steps_at(Smem sm, const uint32_t (&a)[G][NS], EncoderState (&enc)[NS], Sink (&out)[NS], int high_water,
                               uint32_t lanes, bool (&carried)[NS], bool last = false) {
        uint32_t e0[G][NS], e1[G][NS];
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
                enc[i].template take<false>(cg_umulhi_wide(enc[i].span32, e0[g][i]), LAST && last ? enc[i].span32 : fhi, out[i]);
            }
        bool full = false;
#pragma unroll
        for (int i = 0; i < NS; ++i) full |= out[i].nacc >= high_water;
        if (cg_any_lane(lanes, full)) {
#pragma unroll
            for (int i = 0; i < NS; ++i) carried[i] |= out[i].store_word_if_full();
        }
    }
    // whether a stream has met what steps_at leaves
    CG_HD bool unsettled(bool carried) const { return carried | (span32 == 0u); }
    // final flush (enc_new.cu:298-306): two bits that place the stream's value inside the interval, 01 or
    // 10 above the reference's low with its pending bits, which is L plus a quarter of the window cut
    // to two bits; returns the stream length in bytes
    template <class Sink>
    CG_HD uint32_t flush(Sink &out) {
        if (span32) shift(renorm_shift(low, cg_add_less_one(low, span32), span32 - 1u), span32, out);  // see take
        if (out.nacc < 64) out.store_and_carry();
        add_to_low(0x40000000u, out);
        out.acc_hi = cg_fshl(out.acc_lo, out.acc_hi, 2u);
        out.acc_lo = cg_fshl(low, out.acc_lo, 2u);
        out.nacc += 2;
        return out.finish();
    }
};

}  // namespace cg
