// The whole encode of one chunk as three launches: quantise (one pass over the KV), histogram + tables +
// arithmetic coding + offsets, gather.  What the separate calls (cg_quantize_cdf, cg_encode_chunk,
// cg_compact_streams) do in seven launches and with three more passes over memory; same tables, streams and scales.
//
// Between the first two, the symbols of four consecutive tokens of one channel are one 32-bit word,
// sym4[row][token / 4][channel] (first token in the low byte): the coder, whose thread owns a channel, reads
// them coalesced, four symbols a load.
#include <string.h>

#include "cg_common.cuh"

namespace cg {

struct KvView {
    const uint16_t *kv;
    int64_t s_layer, s_kv, s_token, s_head;
    int nlayers, ntokens, nheads, head_size;
    uint32_t head_inv;  // ceil(2^32 / head_size): channel / head_size by a multiply-high, exact below 2^16
};

// ---- pass 1: max|x| and quantise ---------------------------------------------------------------------------
// One block per (row, four tokens), one thread per eight channels: the block holds its tokens' channels in
// registers, so max|x| over the channels (cachegen_encoder.py:55) and the quantisation (:56-57) need one
// read of the KV where a max pass and a quantise pass read it twice (a 256-token Llama-7B chunk, 134 MB,
// does not stay in the L2 in between).  Four tokens a block because their symbols share a word; four
// 128-bit loads a thread in flight.
constexpr int kTokensPerWord = 4;

__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
// (x * f + m) + 2^23 for two values: three separately rounded fp32 operations each (enc.py:56-57), the last of which
// rounds half to even and leaves the symbol in the low byte.  The products stay scalar: with packed products in front of
// the packed sums a symbol in 10^7 differed, as if product and sum had been rounded once.
__device__ __forceinline__ void quantize2(float x0, float x1, float f, uint64_t m, uint32_t *b0, uint32_t *b1) {
    const uint64_t magic = 0x4B0000004B000000ull;
    uint64_t v = pack2(__fmul_rn(x0, f), __fmul_rn(x1, f));
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(m));
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(magic));
    asm("mov.b64 {%0, %1}, %2;" : "=r"(*b0), "=r"(*b1) : "l"(v));
}

// Pass 1.  A block takes four tokens of one row, all channels, eight adjacent ones a thread in one or two runs: the 16-bit values
// stay in registers between the scales (a reduction over the block) and the symbols, so the KV is read once where an
// absmax pass and a quantise pass read it twice, and four tokens' symbols of a channel leave as one word.  Bound
// by memory: a 256-token Llama-7B chunk (134 MB in, 67 MB of symbols out) takes 33 us, 6.1 TB/s, where the two passes took
// 31 + 61 us (the second with the histogram, which the coder does now).  With one run a thread, three blocks of sixteen warps an SM
// all waited for loads or all computed: 39.7 us, and 59.3 where 5,120 channels take 41.5, 41 where 10 layers of 8,192 take 26, 19.6 and 17.6
// for 2,048, 60.5 and 58 for 1,999 tokens of 32 layers x 1,024.  9.3 instructions for 32 symbols; with the layer and the half of the
// pair divided out of one grid dimension, the bins halved by a division and every word zeroed before it is loaded 11.6.
// Sixty-four registers and four blocks of eight warps an SM; five blocks (48 registers) 33.9 us, three 36.2.
// The same KV at several bin settings takes one read and one reduction: only the quantisation is done for each.
struct QuantizeOut {
    const float *bins;
    uint16_t *scales_k, *scales_v;
    uint32_t *sym4, *zeroed;
    int max_bins;
};
struct QuantizeLevels {
    QuantizeOut level[CG_MAX_ENCODE_LEVELS];
    int n, nzeroed;
};
template <int DT, int THREADS, int BLOCKS, bool ONE, int RUNS>
__global__ void __launch_bounds__(THREADS, BLOCKS) quantize_tokens_kernel(const KvView v, const __grid_constant__ QuantizeLevels q) {
    __shared__ uint4 part[32];
    __shared__ float4 factor_s[ONE ? 1 : CG_MAX_ENCODE_LEVELS];
    __shared__ uint32_t keep_s;
    const int nlevels = ONE ? 1 : q.n;
    let_next_launch_start();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int layer = blockIdx.y, kv = blockIdx.z, row = kv * v.nlayers + layer, t0 = blockIdx.x * kTokensPerWord;
    const int C = v.nheads * v.head_size;
    if (row == 0 && blockIdx.x == 0)  // the counters of the launches after this one
        for (int l = 0; l < nlevels; ++l)
            for (int i = tid; i < q.nzeroed; i += blockDim.x) q.level[l].zeroed[i] = 0u;
    // run r of this thread's channels starts at 8 (tid + blockDim.x r)
    uint4 x[RUNS][kTokensPerWord];
    const uint16_t *tokens = v.kv + layer * v.s_layer + kv * v.s_kv + t0 * v.s_token;
#pragma unroll
    for (int r = 0; r < RUNS; ++r) {
        const int c = (tid + r * static_cast<int>(blockDim.x)) * 8;
        const int h = static_cast<int>(__umulhi(static_cast<uint32_t>(c), v.head_inv));
        const uint16_t *p = tokens + h * v.s_head + (c - h * v.head_size);
        if (c < C && t0 + kTokensPerWord <= v.ntokens) {
#pragma unroll
            for (int j = 0; j < kTokensPerWord; ++j) x[r][j] = __ldg(reinterpret_cast<const uint4 *>(p + j * v.s_token));
        } else {
#pragma unroll
            for (int j = 0; j < kTokensPerWord; ++j) {
                x[r][j] = make_uint4(0u, 0u, 0u, 0u);
                if (c < C && t0 + j < v.ntokens) x[r][j] = __ldg(reinterpret_cast<const uint4 *>(p + j * v.s_token));
            }
        }
    }
    // |x| as an ordered integer: 16-bit float magnitudes compare like their bit patterns
    uint32_t m[kTokensPerWord];
#pragma unroll
    for (int j = 0; j < kTokensPerWord; ++j) {
        uint32_t a = 0u;
#pragma unroll
        for (int r = 0; r < RUNS; ++r)
            a = __vmaxu2(a, __vmaxu2(__vmaxu2(x[r][j].x & 0x7FFF7FFFu, x[r][j].y & 0x7FFF7FFFu),
                                     __vmaxu2(x[r][j].z & 0x7FFF7FFFu, x[r][j].w & 0x7FFF7FFFu)));
        m[j] = __reduce_max_sync(0xFFFFFFFFu, max(a & 0xFFFFu, a >> 16));
    }
    if (lane == 0) part[warp] = make_uint4(m[0], m[1], m[2], m[3]);
    const float max_of_first = half_range(__ldg(q.level[0].bins + row));
    __syncthreads();
    if (warp == 0) {
        const uint4 r = lane < (blockDim.x >> 5) ? part[lane] : make_uint4(0u, 0u, 0u, 0u);
        m[0] = __reduce_max_sync(0xFFFFFFFFu, r.x);
        m[1] = __reduce_max_sync(0xFFFFFFFFu, r.y);
        m[2] = __reduce_max_sync(0xFFFFFFFFu, r.z);
        m[3] = __reduce_max_sync(0xFFFFFFFFu, r.w);
        if (lane < kTokensPerWord) {
            const uint32_t mine = lane == 0 ? m[0] : lane == 1 ? m[1] : lane == 2 ? m[2] : m[3];
            for (int l = 0; l < nlevels; ++l) {
                const float MAX = l ? half_range(__ldg(q.level[l].bins + row)) : max_of_first;
                reinterpret_cast<float *>(factor_s + l)[lane] = __fdiv_rn(MAX, Half16<DT>::to_float(static_cast<uint16_t>(mine)));
                if (t0 + lane < v.ntokens) {
                    uint16_t *s = row < v.nlayers ? q.level[l].scales_k + static_cast<int64_t>(row) * v.ntokens
                                                  : q.level[l].scales_v + static_cast<int64_t>(row - v.nlayers) * v.ntokens;
                    s[t0 + lane] = static_cast<uint16_t>(mine);
                }
            }
            // an all-zero token: 0 * inf = NaN, which the reference's cast makes symbol 0
            reinterpret_cast<uint8_t *>(&keep_s)[lane] = mine ? 0xFFu : 0u;
        }
    }
    __syncthreads();
    const uint32_t keep = keep_s;
#pragma unroll 1
    for (int l = 0; l < nlevels; ++l) {
        const float f[kTokensPerWord] = {factor_s[l].x, factor_s[l].y, factor_s[l].z, factor_s[l].w};
        const float MAX = l ? half_range(__ldg(q.level[l].bins + row)) : max_of_first;
        const uint64_t m2 = pack2(MAX, MAX);
#pragma unroll
        for (int r = 0; r < RUNS; ++r) {
            const int c = (tid + r * static_cast<int>(blockDim.x)) * 8;
            if (c >= C) break;
            uint32_t w[8];
#pragma unroll
            for (int k = 0; k < 8; k += 2) {
                uint32_t b0[kTokensPerWord], b1[kTokensPerWord];
#pragma unroll
                for (int j = 0; j < kTokensPerWord; ++j) {
                    const uint32_t pair = k == 0 ? x[r][j].x : k == 2 ? x[r][j].y : k == 4 ? x[r][j].z : x[r][j].w;
                    quantize2(Half16<DT>::to_float(static_cast<uint16_t>(pair)), Half16<DT>::to_float(static_cast<uint16_t>(pair >> 16)),
                              f[j], m2, &b0[j], &b1[j]);
                }
                w[k] = __byte_perm(__byte_perm(b0[0], b0[1], 0x0040), __byte_perm(b0[2], b0[3], 0x0040), 0x5410) & keep;
                w[k + 1] = __byte_perm(__byte_perm(b1[0], b1[1], 0x0040), __byte_perm(b1[2], b1[3], 0x0040), 0x5410) & keep;
            }
            // The coder takes any byte above 127 for a bad symbol.  Inputs that are not finite give 255 as they are;
            // other symbols stay below 2*Cq + 1, which only bin counts above max_bins put outside the table.
            const int max_bins = q.level[l].max_bins;
            if (2.0f * MAX >= static_cast<float>(max_bins - 1)) {
                const uint32_t limit = static_cast<uint32_t>(max_bins - 1) * 0x01010101u;
#pragma unroll
                for (int k = 0; k < 8; ++k) w[k] |= __vcmpgeu4(w[k], limit);
            }
            uint4 *o = reinterpret_cast<uint4 *>(q.level[l].sym4 + (static_cast<int64_t>(row) * gridDim.x + blockIdx.x) * C + c);
            o[0] = make_uint4(w[0], w[1], w[2], w[3]);
            o[1] = make_uint4(w[4], w[5], w[6], w[7]);
        }
    }
}

// ---- tables ------------------------------------------------------------------------------------------------
struct TableOut {
    int16_t *cdf;                 // [nrows, C, lp]
    uint8_t *counts;              // byte counts of the non-centre symbols (CG_TABLES_COUNTS), or nullptr
    const int64_t *table_row_off;
    const float *bins;
    uint32_t *group_nz;           // non-zero byte counts per (row, group), or nullptr
};

// The counts of one channel, hist[m * STRIDE] for symbols m < lp - 1, become its table in place (entries
// cdf << 16, one row more than there are symbols) and, as 16-bit entries, in stage[0 .. lp-1]
// (normalize_cdf_value, cal_cdf.cu:11-15,40-49): entry m is m + scale * #{sym < m} / ntokens.
template <int STRIDE>
__device__ __forceinline__ void counts_to_column(uint32_t *hist, uint16_t *stage, int lp, uint32_t ntokens, int cq) {
    const uint32_t scale = 0xFFFFu - static_cast<uint32_t>(lp - 1);
    const uint32_t total = ntokens & 0xFFFFu;  // the reference accumulates in uint16
    // the division: a shift, or the rounded-down reciprocal, whose product is at most one below the quotient
    const bool pow2 = (total & (total - 1u)) == 0u;
    const int sh = 31 - __clz(static_cast<int>(total | 1u));
    const uint32_t inv = 0xFFFFFFFFu / (total | (total == 0u));
    uint32_t cum = 0;
    const auto entry = [&](int m, uint32_t q) {
        const uint32_t e = q + static_cast<uint32_t>(m);
        hist[m * STRIDE] = e << 16;
        stage[m] = static_cast<uint16_t>(e);
    };
    const auto divided = [&](uint32_t prod) {
        uint32_t q = __umulhi(prod, inv);
        if (prod - q * total >= total) ++q;
        return q;
    };
    const int used = min(2 * cq + 1, lp - 1);  // the row's symbols, all that a quantiser of its bins makes
    int m = 0;
    if (pow2) {
#pragma unroll 4
        for (; m < used; ++m) {
            const uint32_t n = hist[m * STRIDE];
            entry(m, scale * (cum & 0xFFFFu) >> sh);
            cum += n;
        }
    } else {
#pragma unroll 4
        for (; m < used; ++m) {
            const uint32_t n = hist[m * STRIDE];
            entry(m, divided(scale * (cum & 0xFFFFu)));
            cum += n;
        }
    }
    for (; cum != ntokens && m < lp; ++m) {  // symbols above those (never with matching bins)
        const uint32_t n = hist[m * STRIDE];
        const uint32_t prod = scale * (cum & 0xFFFFu);
        entry(m, pow2 ? prod >> sh : divided(prod));
        cum += n;
    }
#pragma unroll 4
    for (; m < lp; ++m) entry(m, scale);  // every symbol is below m
}

// The byte counts of one channel (CG_TABLES_COUNTS), before counts_to_column; returns how many are not zero.
template <int STRIDE>
__device__ __forceinline__ int store_counts(const uint32_t *hist, int lp, int cq, uint8_t *counts, int64_t stride, bool *overflow) {
    int nz = 0;
    for (int m = 0; m < lp - 1; ++m) {
        const uint32_t n = hist[m * STRIDE];
        if (m > 2 * cq) {
            *overflow |= n != 0u;
        } else if (m != cq) {
            *counts = static_cast<uint8_t>(n);
            counts += stride;
            nz += n != 0u;
            *overflow |= n > 255u;
        }
    }
    return nz;
}

// Tables staged as 16-bit entries channel after channel to their place, one contiguous run, by `threads` threads.
__device__ __forceinline__ void copy_tables(const uint16_t *stage, uint16_t *dst, int n, int thread, int threads) {
    if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0 && (n & 7) == 0) {
        const uint4 *s = reinterpret_cast<const uint4 *>(stage);
        uint4 *d = reinterpret_cast<uint4 *>(dst);
        for (int i = thread; i < n / 8; i += threads) d[i] = s[i];
    } else {
        for (int i = thread; i < n; i += threads) dst[i] = stage[i];
    }
}

// Tables of a chunk of more than one sub-chunk (the coder's blocks build those of a single one themselves):
// block (slab, row); a lane counts four adjacent channels, a warp every kTableWarps-th word of them, four words a batch without a
// condition inside.  Channel 4 l + j of the slab has column 32 j + l, so that the lanes of a warp are in 32 banks whichever of
// their channels they count.  Bound by the latency of its loads: 1,999 tokens of 32 layers x 1,024 channels take 32 us under
// counters (3.0 instructions for 32 symbols), 38 and 3.8 with a channel a lane and eight 4-byte loads in flight; 700 tokens of 80
// layers x 1,024 channels 30 and 39.  Two and eight loads in flight: 32 and 33 us; 128 and 512 threads: 35 and 33.  The updates alone, one a
// symbol at 1.1 cycles a warp and SM, would take 16.
constexpr int kTableThreads = 256, kTableWarps = kTableThreads / 32;
struct TableJobs {
    TableOut out[CG_MAX_ENCODE_LEVELS];
    const uint32_t *sym4[CG_MAX_ENCODE_LEVELS];
    int32_t *status[CG_MAX_ENCODE_LEVELS];
    int lp[CG_MAX_ENCODE_LEVELS];
};
__global__ void __launch_bounds__(kTableThreads) packed_tables_kernel(const __grid_constant__ TableJobs jobs, int ntokens, int nchannels) {
    const TableOut &out = jobs.out[blockIdx.z];
    int32_t *const status = jobs.status[blockIdx.z];
    const int lp = jobs.lp[blockIdx.z];
    extern __shared__ uint4 smem4[];
    uint32_t *hist = reinterpret_cast<uint32_t *>(smem4);
    uint16_t *stage = reinterpret_cast<uint16_t *>(hist + lp * kGroup);
    __shared__ uint32_t nz_total;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row = blockIdx.y, slab = blockIdx.x * kGroup, nch = min(kGroup, nchannels - slab);  // a multiple of 8
    for (int i = tid; i < lp * kGroup; i += kTableThreads) hist[i] = 0u;
    if (tid == 0) nz_total = 0u;
    __syncthreads();
    const int words = (ntokens + 3) / 4, whole = ntokens / 4;
    if (4 * lane < nch) {
        uint32_t col[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) col[j] = smem_addr(hist + j * 32 * lp + lane);
        const int64_t step = static_cast<int64_t>(kTableWarps) * nchannels;
        const uint32_t *p = jobs.sym4[blockIdx.z] + (static_cast<int64_t>(row) * words + warp) * nchannels + slab + 4 * lane;
        const auto count = [&](uint4 w) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                count_symbol(entry_of(col[0], w.x, k));
                count_symbol(entry_of(col[1], w.y, k));
                count_symbol(entry_of(col[2], w.z, k));
                count_symbol(entry_of(col[3], w.w, k));
            }
        };
        const auto cleaned = [](uint32_t w) { return w & 0x80808080u ? 0u : w; };  // reported by the coder
        constexpr int kAhead = 4;  // loads in flight
        int i = warp;
        for (; i + kTableWarps * (kAhead - 1) < whole; i += kTableWarps * kAhead) {
            uint4 w[kAhead];
            uint32_t any = 0u;
#pragma unroll
            for (int k = 0; k < kAhead; ++k) {
                w[k] = __ldg(reinterpret_cast<const uint4 *>(p));
                p += step;
            }
#pragma unroll
            for (int k = 0; k < kAhead; ++k) any |= w[k].x | w[k].y | w[k].z | w[k].w;
            if (any & 0x80808080u) {
#pragma unroll
                for (int k = 0; k < kAhead; ++k) w[k] = make_uint4(cleaned(w[k].x), cleaned(w[k].y), cleaned(w[k].z), cleaned(w[k].w));
            }
#pragma unroll
            for (int k = 0; k < kAhead; ++k) count(w[k]);
        }
        for (; i < words; i += kTableWarps) {
            uint4 w = __ldg(reinterpret_cast<const uint4 *>(p));
            p += step;
            w = make_uint4(cleaned(w.x), cleaned(w.y), cleaned(w.z), cleaned(w.w));
            if (i < whole) {
                count(w);
                continue;
            }
            for (int k = 0; k < (ntokens & 3); ++k) {
                count_symbol(col[0] + ((w.x >> (8 * k)) & 0xFFu) * kWarpRow);
                count_symbol(col[1] + ((w.y >> (8 * k)) & 0xFFu) * kWarpRow);
                count_symbol(col[2] + ((w.z >> (8 * k)) & 0xFFu) * kWarpRow);
                count_symbol(col[3] + ((w.w >> (8 * k)) & 0xFFu) * kWarpRow);
            }
        }
    }
    __syncthreads();
    bool overflow = false;
    if (tid < kGroup) {
        const int cl = 4 * lane + warp;  // the channel of column tid
        int nz = 0;
        if (cl < nch) {
            const int cq = static_cast<int>(half_range(__ldg(out.bins + row)));
            uint32_t *column = hist + warp * 32 * lp + lane;
            if (out.counts) nz = store_counts<32>(column, lp, cq, out.counts + __ldg(out.table_row_off + row) + slab + cl, nchannels, &overflow);
            counts_to_column<32>(column, stage + cl * lp, lp, ntokens, cq);
        }
        if (out.group_nz) {
            nz = __reduce_add_sync(0xFFFFFFFFu, nz);
            if (lane == 0 && nz) atomicAdd(&nz_total, static_cast<uint32_t>(nz));
        }
    }
    if (overflow && status) atomicOr(status, CG_S_COUNT_OVERFLOW);
    __syncthreads();
    copy_tables(stage, reinterpret_cast<uint16_t *>(out.cdf) + (static_cast<int64_t>(row) * nchannels + slab) * lp, nch * lp, tid, kTableThreads);
    if (tid == 0 && out.group_nz) out.group_nz[row * gridDim.x + blockIdx.x] = nz_total;
}

// ---- pass 2: (histogram, tables,) arithmetic coding, offsets -------------------------------------------------
struct StoreParams {
    const uint32_t *sym4;
    TableOut out;
    int ntokens, nchannels, lp, nrows, nsub;
    int high_water;       // of two symbols a vote, see deep_pair_high_water; 0: one
    uint8_t *scratch;     // [nsub, nrows, nslab, 4 warps, stride / 4 + 1, 32 lanes] words
    int64_t stride;
    int32_t *lengths;     // [nsub, nrows * C]
    int64_t *group_off;   // [nsub, nrows * nslab]: byte offset of each 128-channel group inside its sub-chunk
    int64_t *sub_bytes;   // [nsub]
    uint32_t *tickets;    // [nsub + 1], zero
    int32_t *status;      // zero before pass 1
    int64_t *tail;        // [nsub + 4], see cg_encode_kv_job
};

// Several bin settings of one chunk in one launch: their blocks fill the GPU together where those of one chunk of few channels
// leave most of it idle (a 256-token chunk of 32 layers x 8 heads is 512 blocks, 3.5 an SM).
struct StoreJobs {
    StoreParams job[CG_MAX_ENCODE_LEVELS];
};

// The scratch rows of the 32 streams of a warp lie interleaved: word k of stream `lane` is word 32 (k + 1) + lane
// of the warp's 32 * (stride + 4) bytes.  A stream takes 45 of its 520 bytes on the usual workload: laid out row by
// row that is a cache line or two for every stream (70 MB of lines a Llama-7B chunk, which the L2 did not
// keep), interleaved it is as many lines as there is data, and the gather reads them whole.  One more row in front
// of the first word's (see BitSinkT).
__device__ __forceinline__ uint32_t *scratch_word(uint8_t *scratch, int64_t stride, int64_t group, int tid) {
    return reinterpret_cast<uint32_t *>(scratch + (group * (kGroup / 32) + (tid >> 5)) * 32 * (stride + 4)) + 32 + (tid & 31);
}

// Exclusive scan of n values in place by one block of THREADS threads; returns the sum.
template <int THREADS, class T>
__device__ __forceinline__ int64_t block_scan_in_place(T *v, int n, int64_t *warp_sums, int tid) {
    constexpr int kPer = 8;
    const int lane = tid & 31, w = tid >> 5;
    int64_t base = 0;
    for (int b = 0; b < n; b += THREADS * kPer) {
        const int at = b + tid * kPer;
        int64_t x[kPer], s = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            x[k] = at + k < n ? static_cast<int64_t>(__ldcg(v + at + k)) : 0;
            s += x[k];
        }
        int64_t incl = s;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int64_t y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d) incl += y;
        }
        __syncthreads();
        if (lane == 31) warp_sums[w] = incl;
        __syncthreads();
        int64_t run = base + incl - s;
#pragma unroll
        for (int k = 0; k < THREADS / 32; ++k) {
            if (k < w) run += warp_sums[k];
            base += warp_sums[k];
        }
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            if (at + k < n) v[at + k] = static_cast<T>(run);
            run += x[k];
        }
    }
    return base;
}

// A word of symbols that the launch in front wrote, read behind the wait for it.  The coder's blocks may be resident while the
// quantiser still writes, so the words do not take the path for data that nothing writes while the kernel runs (__ldg): they come
// from the L2, and the compiler leaves such a load behind the wait.  As fast: a 256-token Llama-7B chunk in 199 us, 201 with
// __ldg; 1,999 tokens of 32 layers x 1,024 channels in 411 and 413.
__device__ __forceinline__ uint32_t written_symbols(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.global.cg.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// A stream that has met what the coder's loop leaves (see EncoderState::steps_at) from its start again, by one lane:
// the stream's words of symbols at sp, C words apart.  Returns its length in bytes.  About never run.
template <class Sink>
static __device__ __noinline__ uint32_t encode_again(uint32_t col, const uint32_t *sp, int64_t C, int n, uint8_t *to, int64_t stride) {
    Sink out;
    EncoderState enc;
    out.init(to, stride);
    enc.init();
    uint32_t w = 0u;
    for (int i = 0; i < n; ++i) {
        if ((i & 3) == 0) {
            w = written_symbols(sp + (i >> 2) * C);
            if (w & 0x80808080u) w = 0u;
        }
        enc.step_alone<kWarpRow>(Smem{}, entry_of(col, w, 0), false, out);
        w >>= 8;
    }
    return enc.flush(out);
}

// NS streams per thread, 128 adjacent channels of one row and sub-chunk per block.  TABLES: the chunk is one
// sub-chunk, so the block's symbols are all there are for its tables: it counts them (each thread in its
// own shared-memory columns, where its tables then stand), writes the tables out and codes; the symbols'
// second read comes from the L2.  Otherwise the tables come from packed_tables_kernel.
// The last block of a sub-chunk turns the group sizes into offsets, the last of all writes the tail.
// Bound by instruction issue (the coder's serial step, half of it on the integer pipe): a 256-token Llama-7B
// chunk takes 104 us with its tables under counters, 0.64 T symbols/s, 32.9 instructions for 32 symbols; 107 us and 34.5 with the
// shifts as multiplies by a power of two made for them and words stored at 44 pending bits, 122 us and 40.4 with
// the code for rare cases inside the loop besides, and a vote a symbol.  33 us of it are there without the coder's loop (the counts,
// the tables and two waves' latencies), 12 are the votes and stores.  Eight blocks an SM leave the compiler 64
// registers.  (Seven, for two even waves of a chunk's 2,048 blocks, take the same.)
// Two streams a thread share the step's vote and hide each other's latencies: 1,999 tokens of 32 layers x 1,024
// channels in 152 us under counters (26.4 instructions for 32 symbols), 164 (28.5) and 172 before the same changes; 180 with one
// stream.  (One stream and 32, 40 and 48 warps an SM in place of 24: 168, 171 and 171 us at the time of the 164.)
// G symbols a vote: two, unless the table may give a symbol more bits than the accumulator has room for twice (pair_high_water:
// more than 21,824 tokens in one call).  The tables' part wants the warps more than the chains (a 256-token chunk
// 129 us with two), so it keeps one; and so does a last group of channels that would leave the second without work.
template <bool TABLES, int NS, int G>
__global__ void __launch_bounds__(kGroup / NS, NS == 1 ? 8 : 12) store_encode_kernel(const __grid_constant__ StoreJobs jobs) {
    const int nsub = jobs.job[0].nsub;
    const StoreParams &p = jobs.job[blockIdx.z / nsub];
    constexpr int kThreads = kGroup / NS, kWarps = kThreads / 32;
    constexpr int kWordsAhead = NS == 1 ? 4 : 2;  // words (of four symbols) fetched one group ahead of the coder
    extern __shared__ uint4 smem4[];
    uint32_t *tab = reinterpret_cast<uint32_t *>(smem4);
    __shared__ int64_t warp_sums[kWarps];
    __shared__ int block_sums[2][kWarps];
    __shared__ int last_block;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row = blockIdx.y, sub = blockIdx.z % nsub, nslab = gridDim.x;
    const int t0 = sub * kSubTokens, n = min(kSubTokens, p.ntokens - t0);
    const int64_t C = p.nchannels;
    // channel s of this thread is number tid + kThreads * s of the group; one past the last channel repeats the last
    // and is written nowhere but to its own scratch row
    bool active[NS];
    int64_t g[NS];
    uint32_t *column[NS];
    uint32_t col[NS];
    const uint32_t *sp[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        const int slot = s * kThreads + tid, c = min(blockIdx.x * kGroup + slot, p.nchannels - 1);
        active[s] = blockIdx.x * kGroup + slot < p.nchannels;
        g[s] = row * C + c;
        column[s] = tab + (slot >> 5) * 32 * p.lp + lane;
        col[s] = smem_addr(column[s]);
        sp[s] = p.sym4 + (static_cast<int64_t>(row) * ((p.ntokens + 3) / 4) + t0 / 4) * C + c;
    }
    // the same for a warp; with two streams every warp has channels
    const bool any_active = NS > 1 || blockIdx.x * kGroup + warp * 32 < p.nchannels;
    uint32_t bad = 0;
    int nbytes = 0, nz = 0;
    const float bins = TABLES ? __ldg(p.out.bins + row) : 0.0f;

    if (TABLES && any_active) {
        static_assert(!TABLES || NS == 1, "the tables' part has one stream a thread");
        uint32_t *const mine = column[0];
        uint16_t *stage = reinterpret_cast<uint16_t *>(tab + p.lp * kGroup);
        bool overflow = false;
        for (int m = 0; m < p.lp; ++m) mine[m * 32] = 0u;
        wait_for_launch_before();
        constexpr int kAhead = 16;  // words in flight
        const uint32_t *q = sp[0];
        int i = 0;
        for (; i + 4 * kAhead <= n; i += 4 * kAhead) {
            uint32_t w[kAhead], any = 0u;
#pragma unroll
            for (int k = 0; k < kAhead; ++k) {
                w[k] = written_symbols(q);
                q += C;
            }
#pragma unroll
            for (int k = 0; k < kAhead; ++k) any |= w[k];
            if (any & 0x80808080u) {  // reported below
#pragma unroll
                for (int k = 0; k < kAhead; ++k)
                    if (w[k] & 0x80808080u) w[k] = 0u;
            }
#pragma unroll
            for (int k = 0; k < kAhead; ++k) {
#pragma unroll
                for (int j = 0; j < 4; ++j) count_symbol(entry_of(col[0], w[k], j));
            }
        }
        for (; i < n; i += 4) {
            uint32_t w = written_symbols(q);
            q += C;
            if (w & 0x80808080u) w = 0u;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (i + j < n) count_symbol(entry_of(col[0], w, j));
        }
        const int cq = static_cast<int>(half_range(bins));
        if (p.out.counts && active[0])
            nz = store_counts<32>(mine, p.lp, cq, p.out.counts + __ldg(p.out.table_row_off + row) - row * C + g[0], C, &overflow);
        counts_to_column<32>(mine, stage + tid * p.lp, p.lp, n, cq);
        if (overflow) atomicOr(p.status, CG_S_COUNT_OVERFLOW);
        __syncwarp();
        const int first = blockIdx.x * kGroup + warp * 32, nch = min(32, p.nchannels - first);
        copy_tables(stage + warp * 32 * p.lp, reinterpret_cast<uint16_t *>(p.out.cdf) + (row * C + first) * p.lp, nch * p.lp, lane, 32);
    } else if (any_active) {
        wait_for_launch_before();
#pragma unroll
        for (int s = 0; s < NS; ++s) stage_encode_column<32>(column[s], p.out.cdf + g[s] * p.lp, p.lp, 0);
    }

    if (any_active) {
        using Sink = BitSinkT<32, false>;  // see scratch_word
        Sink out[NS];
        EncoderState enc[NS];
        bool carried[NS] = {};
        const int64_t group = (static_cast<int64_t>(sub) * p.nrows + row) * nslab + blockIdx.x;
        uint32_t w[NS][kWordsAhead], next[NS][kWordsAhead];
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            out[s].init(reinterpret_cast<uint8_t *>(scratch_word(p.scratch, p.stride, group, s * kThreads + tid)), p.stride);
            enc[s].init();
            enc[s].half_scale(out[s]);
#pragma unroll
            for (int k = 0; k < kWordsAhead; ++k) w[s][k] = 4 * k < n ? written_symbols(sp[s] + k * C) : 0u;
        }
        const int high_water = G == 1 ? kDeepHighWater : p.high_water;
        constexpr int kAhead = 4 * kWordsAhead;
        int i = 0;
        for (;; i += kAhead) {
            uint32_t any = 0u;
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                sp[s] += kWordsAhead * C;
#pragma unroll
                for (int k = 0; k < kWordsAhead; ++k) {
                    next[s][k] = i + kAhead + 4 * k < n ? written_symbols(sp[s] + k * C) : 0u;
                    any |= w[s][k];
                }
            }
            if (any & 0x80808080u) {
                bad = 1u;
#pragma unroll
                for (int k = 0; k < kWordsAhead * NS; ++k) {
                    uint32_t &v = w[k / kWordsAhead][k % kWordsAhead];
                    if (v & 0x80808080u) v = 0u;  // as the tables count it
                }
            }
            if (i + kAhead > n) break;
#pragma unroll
            for (int k = 0; k < kWordsAhead; ++k) {
#pragma unroll
                for (int j = 0; j < 4; j += G) {
                    uint32_t a[G][NS];
#pragma unroll
                    for (int g = 0; g < G; ++g)
#pragma unroll
                        for (int s = 0; s < NS; ++s) a[g][s] = entry_of(col[s], w[s][k], j + g);
                    EncoderState::steps_at<kWarpRow, G, NS, false, true>(Smem{}, a, enc, out, high_water, 0xFFFFFFFFu, carried);
                }
            }
#pragma unroll
            for (int k = 0; k < kWordsAhead * NS; ++k) w[k / kWordsAhead][k % kWordsAhead] = next[k / kWordsAhead][k % kWordsAhead];
        }
        for (; i < n; ++i) {  // fewer than kAhead left, all in w
            uint32_t a[1][NS];
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                a[0][s] = entry_of(col[s], w[s][0], 0);
                w[s][0] >>= 8;
                if ((i & 3) == 3) {
#pragma unroll
                    for (int k = 0; k + 1 < kWordsAhead; ++k) w[s][k] = w[s][k + 1];
                }
            }
            EncoderState::steps_at<kWarpRow, 1, NS, false, true>(Smem{}, a, enc, out, kDeepHighWater, 0xFFFFFFFFu, carried);
        }
        int bits = bad ? CG_S_BAD_SYMBOL : 0;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            int len;
            if (enc[s].unsettled(carried[s]))
                len = static_cast<int>(encode_again<Sink>(col[s], p.sym4 + (static_cast<int64_t>(row) * ((p.ntokens + 3) / 4) + t0 / 4) * C +
                                                                      min(blockIdx.x * kGroup + s * kThreads + tid, p.nchannels - 1),
                                                          C, n, reinterpret_cast<uint8_t *>(scratch_word(p.scratch, p.stride, group, s * kThreads + tid)), p.stride));
            else
                len = static_cast<int>(enc[s].flush(out[s]));
            if (!active[s]) continue;
            p.lengths[static_cast<int64_t>(sub) * p.nrows * C + g[s]] = len;
            if (len > p.stride) {
                bits |= CG_S_STREAM_OVERFLOW;
                len = static_cast<int>(p.stride);
            }
            nbytes += len;
        }
        if (bits) atomicOr(p.status, bits);
    }

    wait_for_launch_before();  // warps without channels
    // group sizes, and whose turn it is to make offsets of them
    const int sum = __reduce_add_sync(0xFFFFFFFFu, nbytes);
    const int nz_sum = TABLES && p.out.group_nz ? __reduce_add_sync(0xFFFFFFFFu, nz) : 0;
    if (lane == 0) {
        block_sums[0][warp] = sum;
        block_sums[1][warp] = nz_sum;
    }
    __syncthreads();
    const int ngroups = p.nrows * nslab;
    int64_t *goff = p.group_off + static_cast<int64_t>(sub) * ngroups;
    if (tid == 0) {
        int s = 0, z = 0;
        for (int k = 0; k < kWarps; ++k) {
            s += block_sums[0][k];
            z += block_sums[1][k];
        }
        goff[row * nslab + blockIdx.x] = s;
        if (TABLES && p.out.group_nz) p.out.group_nz[row * nslab + blockIdx.x] = static_cast<uint32_t>(z);
        __threadfence();
        last_block = atomicAdd(p.tickets + sub, 1u) == static_cast<uint32_t>(ngroups - 1);
    }
    __syncthreads();
    if (!last_block) return;
    __threadfence();
    // every stream's status bits are there with its block's ticket
    const int status = tid == 0 ? __ldcg(p.status) : 0;
    const int64_t bytes = block_scan_in_place<kThreads>(goff, ngroups, warp_sums, tid);
    if (nsub > 1) {
        if (tid == 0) {
            p.sub_bytes[sub] = bytes;
            __threadfence();
            last_block = atomicAdd(p.tickets + nsub, 1u) == static_cast<uint32_t>(nsub - 1);
        }
        __syncthreads();
        if (!last_block) return;
        __threadfence();
    }
    int64_t nz_total = 0;
    if (p.out.group_nz) {
        nz_total = block_scan_in_place<kThreads>(p.out.group_nz, ngroups, warp_sums, tid);
        if (tid == 0) p.out.group_nz[ngroups] = static_cast<uint32_t>(nz_total);
    }
    if (tid == 0) {
        int64_t run = 0;
        for (int k = 0; k < nsub; ++k) {
            p.tail[k] = run;
            run += nsub > 1 ? __ldcg(p.sub_bytes + k) : bytes;
        }
        p.tail[nsub] = run;
        p.tail[nsub + 1] = nsub > 1 ? __ldcg(p.status) : status;
        p.tail[nsub + 2] = nz_total;
        __threadfence_system();
        *reinterpret_cast<volatile int64_t *>(p.tail + nsub + 3) = 1;
    }
}

// the tail of the separate calls' results (shapes that the fused passes do not take)
__global__ void publish_tail_kernel(const int64_t *sub_off, const int32_t *status, int nsub, const uint32_t *nz, int64_t *tail) {
    for (int k = threadIdx.x; k <= nsub; k += blockDim.x) tail[k] = sub_off[k];
    if (threadIdx.x == 0) {
        tail[nsub + 1] = *status;
        tail[nsub + 2] = nz ? *nz : 0;
    }
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) *reinterpret_cast<volatile int64_t *>(tail + nsub + 3) = 1;
}

// ---- pass 3: gather ------------------------------------------------------------------------------------------
// Destinations of up to kGatherSubs sub-chunks (kernel parameters).
constexpr int kGatherSubs = 64;
struct GatherTargets {
    uint8_t *bytes[kGatherSubs];
    int32_t *lengths[kGatherSubs];  // [nrows, C]
};
struct GatherJobs {
    const uint8_t *scratch[CG_MAX_ENCODE_LEVELS];
    const int32_t *lengths[CG_MAX_ENCODE_LEVELS];
    const int64_t *group_off[CG_MAX_ENCODE_LEVELS];
    int nsub;
};

// The gather of one sub-chunk's group (gather_run) into final buffers, its lengths beside it.  15 us under
// counters a 256-token Llama-7B chunk (11.8 MB out of scratch that is read in full lines).  Ten blocks an SM are what the
// shared memory allows (see gather_run).
template <bool INTERLEAVED>
__global__ void __launch_bounds__(kGroup, 10) gather_kernel(const __grid_constant__ GatherJobs jobs, int64_t stride, int nchannels, int first,
                                                        const __grid_constant__ GatherTargets out) {
    const int job = (first + blockIdx.z) / jobs.nsub;  // sub-chunk after sub-chunk, job after job
    const uint8_t *scratch = jobs.scratch[job];
    const int32_t *lengths = jobs.lengths[job];
    const int64_t *group_off = jobs.group_off[job];
    const int tid = threadIdx.x;
    const int row = blockIdx.y, sub = (first + blockIdx.z) % jobs.nsub, nrows = gridDim.y, nslab = gridDim.x;
    const int c = blockIdx.x * kGroup + tid;
    const int64_t group = (static_cast<int64_t>(sub) * nrows + row) * nslab + blockIdx.x;
    const int64_t slot = (static_cast<int64_t>(sub) * nrows + row) * nchannels + c;
    const int len = c < nchannels ? __ldg(lengths + slot) : 0;
    if (c < nchannels) out.lengths[blockIdx.z][static_cast<int64_t>(row) * nchannels + c] = len;
    const uint32_t *src = INTERLEAVED ? scratch_word(const_cast<uint8_t *>(scratch), stride, group, tid)
                                      : reinterpret_cast<const uint32_t *>(scratch + slot * stride);
    gather_run<INTERLEAVED ? 32 : 1>(src, min(len, static_cast<int>(stride)), out.bytes[blockIdx.z] + __ldg(group_off + group));
}

// ---- a container (flat_format.py) in one launch ---------------------------------------------------------------
constexpr int kMaxHeader = 128 + 8 * (65536 / kSubTokens + 1);
struct ContainerParams {
    uint8_t header[kMaxHeader];
    int64_t sub_off[kMaxHeader / 8];  // of the sub-chunks' streams in the payload
    int header_bytes, nsub, nchannels, kind;
    uint8_t *blob;
    int64_t off_scales, off_tables, tables_bytes, off_lengths, off_payload, off_masks, off_counts;
    const uint16_t *scales_k, *scales_v;
    int64_t nscales;               // of each
    const uint8_t *tables;         // byte counts, or int16 tables as they are (CG_TABLES_CDF)
    const int64_t *count_row_off, *mask_row_off;
    const float *bins;
    const uint32_t *group_nz;
    const uint8_t *scratch;
    const int32_t *lengths;
    const int64_t *group_off;
    int64_t stride;
};

// 16-bit stream lengths and streams of one sub-chunk's group, as gather_kernel; and in the blocks behind the sub-chunks' the rest:
// masks and non-zero counts of the group in one pass over its byte counts, or a share of dense tables, a share of the scales and
// group offsets, and in the first block the header and the zero bytes between the sections (the same KV gives the same bytes).
// Bound by latency and, where the call is short, by its one launch: 61 tokens of 10 layers x 1,024 channels to a container and back as bytes
// take 203 us, 218 with a clearing, two kernels and a gather, 15 us of launches, in its place.
template <bool INTERLEAVED>
__global__ void __launch_bounds__(kGroup, 10) container_kernel(const __grid_constant__ ContainerParams p) {
    const int tid = threadIdx.x, row = blockIdx.y, nrows = gridDim.y, nslab = gridDim.x;
    const int c = blockIdx.x * kGroup + tid, sub = blockIdx.z;
    if (sub < p.nsub) {
        const int64_t group = (static_cast<int64_t>(sub) * nrows + row) * nslab + blockIdx.x;
        const int64_t slot = (static_cast<int64_t>(sub) * nrows + row) * p.nchannels + c;
        const int len = c < p.nchannels ? __ldg(p.lengths + slot) : 0;
        if (c < p.nchannels) reinterpret_cast<uint16_t *>(p.blob + p.off_lengths)[slot] = static_cast<uint16_t>(len);
        const uint32_t *src = INTERLEAVED ? scratch_word(const_cast<uint8_t *>(p.scratch), p.stride, group, tid)
                                          : reinterpret_cast<const uint32_t *>(p.scratch + slot * p.stride);
        gather_run<INTERLEAVED ? 32 : 1>(src, min(len, static_cast<int>(p.stride)), p.blob + p.off_payload + p.sub_off[sub] + __ldg(p.group_off + group));
        return;
    }
    const int block = row * nslab + blockIdx.x, blocks = nrows * nslab;
    const int64_t i0 = static_cast<int64_t>(block) * kGroup + tid, step = static_cast<int64_t>(blocks) * kGroup;
    uint8_t *const tables = p.blob + p.off_tables;
    if (p.kind == CG_TABLES_SPARSE) {
        __shared__ int warp_sums[kGroup / 32];
        const int nstored = stored_symbols(p.bins, row);
        const uint8_t *cnt = p.tables + __ldg(p.count_row_off + row) + c;
        const int64_t at_mask = __ldg(p.mask_row_off + row);
        uint32_t m = 0u, n[8] = {};
        if (c < p.nchannels) {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                if (j >= nstored) continue;
                const uint32_t v = __ldg(cnt + static_cast<int64_t>(j) * p.nchannels);
                n[j >> 2] |= v << (8 * (j & 3));
                m |= (v ? 1u : 0u) << j;
            }
            uint8_t *mrow = tables + p.off_masks + at_mask;
            if (nstored <= 16) reinterpret_cast<uint16_t *>(mrow)[c] = static_cast<uint16_t>(m);
            else reinterpret_cast<uint32_t *>(mrow)[c] = m;
            if (c == p.nchannels - 1)  // rows of masks start at multiples of four
                for (int64_t k = at_mask + static_cast<int64_t>(p.nchannels) * (nstored <= 16 ? 2 : 4); k < __ldg(p.mask_row_off + row + 1); ++k)
                    tables[p.off_masks + k] = 0;
        }
        const int excl = block_exclusive_scan_128(__popc(m), warp_sums, tid, nullptr);
        uint8_t *o = tables + p.off_counts + __ldg(p.group_nz + block) + excl;
#pragma unroll
        for (int j = 0; j < 32; ++j)
            if ((m >> j) & 1u) *o++ = static_cast<uint8_t>(n[j >> 2] >> (8 * (j & 3)));
        uint32_t *offsets = reinterpret_cast<uint32_t *>(tables);
        for (int64_t i = i0; i <= blocks; i += step) offsets[i] = __ldg(p.group_nz + i);
    } else {  // off_tables is a multiple of 16
        const int64_t whole = (reinterpret_cast<uintptr_t>(p.tables) & 15) ? 0 : p.tables_bytes / 16;
        for (int64_t i = i0; i < whole; i += step) reinterpret_cast<uint4 *>(tables)[i] = __ldg(reinterpret_cast<const uint4 *>(p.tables) + i);
        for (int64_t i = whole * 16 + i0; i < p.tables_bytes; i += step) tables[i] = __ldg(p.tables + i);
    }
    uint16_t *scales = reinterpret_cast<uint16_t *>(p.blob + p.off_scales);
    for (int64_t i = i0; i < p.nscales; i += step) {
        scales[i] = __ldg(p.scales_k + i);
        scales[p.nscales + i] = __ldg(p.scales_v + i);
    }
    if (block) return;
    for (int i = tid; i < p.header_bytes; i += kGroup) p.blob[i] = p.header[i];
    const auto zero = [&](int64_t from, int64_t to) {
        for (int64_t i = from + tid; i < to; i += kGroup) p.blob[i] = 0;
    };
    zero(p.header_bytes, p.off_scales);
    zero(p.off_scales + 4 * p.nscales, p.off_tables);
    if (p.kind == CG_TABLES_SPARSE) {
        zero(p.off_tables + 4 * (static_cast<int64_t>(blocks) + 1), p.off_tables + p.off_masks);
        zero(p.off_tables + p.off_masks + __ldg(p.mask_row_off + nrows), p.off_tables + p.off_counts);
    }
    zero(p.off_tables + p.tables_bytes, p.off_lengths);
    zero(p.off_lengths + static_cast<int64_t>(p.nsub) * nrows * p.nchannels * 2, p.off_payload);
}

}  // namespace cg

using namespace cg;

namespace {

struct Sizes {
    int nrows, nchannels, nslab, nsub;
    int64_t words, stride;
    int64_t sym, scratch, lengths, group_off, sub_bytes, counters, group_nz, sub_off, scales, total;
};

Sizes sizes_of(int nlayers, int ntokens, int nheads, int head_size) {
    Sizes z;
    z.nrows = 2 * nlayers;
    z.nchannels = nheads * head_size;
    z.nslab = (z.nchannels + kGroup - 1) / kGroup;
    z.nsub = (ntokens + kSubTokens - 1) / kSubTokens;
    z.words = (ntokens + 3) / 4;
    z.stride = (CG_STREAM_CAPACITY(ntokens < kSubTokens ? ntokens : kSubTokens) + 3) / 4 * 4;
    const int64_t streams = static_cast<int64_t>(z.nrows) * z.nchannels, groups = static_cast<int64_t>(z.nrows) * z.nslab;
    int64_t at = 0;
    const auto take = [&](int64_t bytes) {
        const int64_t here = at;
        at += (bytes + 255) / 256 * 256;
        return here;
    };
    z.sym = take(streams * z.words * 4);
    z.scratch = take(z.nsub * groups * kGroup * (z.stride + 4));
    z.lengths = take(z.nsub * streams * 4);
    z.group_off = take(z.nsub * groups * 8);
    z.sub_bytes = take(z.nsub * 8);
    z.counters = take((z.nsub + 2) * 4);  // the status word, then the tickets
    z.group_nz = take((groups + 1) * 4);
    z.sub_off = take((z.nsub + 1) * 8);
    z.scales = take(static_cast<int64_t>(z.nrows) * ntokens * 2);
    z.total = at;
    return z;
}

int check_job(const cg_encode_kv_job *job) {
    if (!job) return CG_E_NULL;
    const cg_encode_kv_job &b = *job;
    if (!b.kv || !b.bins || !b.scales_k || !b.scales_v || !b.cdf || !b.workspace || !b.tail) return CG_E_NULL;
    if (b.counts && !b.table_row_off) return CG_E_NULL;
    if (b.nlayers <= 0 || b.ntokens <= 0 || b.nheads <= 0 || b.head_size <= 0 || 2 * b.nlayers > 65535) return CG_E_SHAPE;
    if (static_cast<int64_t>(b.nheads) * b.head_size > 0x7FFFFFFF - kGroup) return CG_E_SHAPE;
    if (b.ntokens >= 65536) return CG_E_HIST;
    if (b.dtype != CG_F16 && b.dtype != CG_BF16) return CG_E_DTYPE;
    if (b.max_bins < 1 || b.max_bins >= CG_MAX_LP) return CG_E_LP;
    if (b.delta_group && !b.res_bins) return CG_E_NULL;
    if (reinterpret_cast<uintptr_t>(b.workspace) & 255) return CG_E_ALIGN;
    if (b.workspace_bytes < sizes_of(b.nlayers, b.ntokens, b.nheads, b.head_size).total) return CG_E_CAPACITY;
    return CG_OK;
}

// Shapes of the fused passes: eight-channel runs inside one head at 16-byte boundaries, a token's channels in one
// block.  The rest, and delta coding, takes the separate calls.
bool fused_ok(const cg_encode_kv_job &b) {
    return !b.delta_group && b.head_size % 8 == 0 && b.nheads * b.head_size <= 8192 &&
           ((reinterpret_cast<uintptr_t>(b.kv) & 15) | (b.s_layer & 7) | (b.s_kv & 7) | (b.s_token & 7) | (b.s_head & 7)) == 0;
}

// Jobs of one call: the same KV, read in the same way, at different bin settings.
bool same_chunk(const cg_encode_kv_job &a, const cg_encode_kv_job &b) {
    return a.kv == b.kv && a.dtype == b.dtype && a.nlayers == b.nlayers && a.ntokens == b.ntokens && a.nheads == b.nheads &&
           a.head_size == b.head_size && a.s_layer == b.s_layer && a.s_kv == b.s_kv && a.s_token == b.s_token && a.s_head == b.s_head &&
           a.delta_group == b.delta_group;
}

}  // namespace

extern "C" int64_t cg_encode_kv_workspace(int nlayers, int ntokens, int nheads, int head_size) {
    if (nlayers <= 0 || ntokens <= 0 || nheads <= 0 || head_size <= 0) return CG_E_SHAPE;
    return sizes_of(nlayers, ntokens, nheads, head_size).total;
}

// the separate calls, for what the fused passes do not take
static int encode_separately(const cg_encode_kv_job &b, cudaStream_t st) {
    const Sizes z = sizes_of(b.nlayers, b.ntokens, b.nheads, b.head_size);
    uint8_t *ws = static_cast<uint8_t *>(b.workspace);
    int32_t *status = reinterpret_cast<int32_t *>(ws + z.counters);
    uint32_t *group_nz = b.counts ? reinterpret_cast<uint32_t *>(ws + z.group_nz) : nullptr;
    int32_t *lengths = reinterpret_cast<int32_t *>(ws + z.lengths);
    int64_t *group_off = reinterpret_cast<int64_t *>(ws + z.group_off);
    const int lp = b.max_bins + 1;
    void *stream = st;
    const cudaError_t e = cudaMemsetAsync(status, 0, 4, st);
    if (e != cudaSuccess) return set_cuda_error(e);
    uint16_t *scales = reinterpret_cast<uint16_t *>(ws + z.scales);
    int8_t *sym = reinterpret_cast<int8_t *>(ws + z.sym);
    if (int rc = cg_quantize_cdf_delta(b.kv, b.dtype, b.s_layer, b.s_kv, b.s_token, b.s_head, b.nlayers, b.ntokens,
                                       b.nheads, b.head_size, b.bins, b.max_bins, b.delta_group, b.res_bins, sym, scales,
                                       b.cdf, b.counts, b.table_row_off, status, stream))
        return rc;
    const size_t half = static_cast<size_t>(b.nlayers) * b.ntokens;
    const cudaError_t e1 = cudaMemcpyAsync(b.scales_k, scales, half * 2, cudaMemcpyDeviceToDevice, st);
    const cudaError_t e2 = cudaMemcpyAsync(b.scales_v, scales + half, half * 2, cudaMemcpyDeviceToDevice, st);
    if (e1 != cudaSuccess || e2 != cudaSuccess) return set_cuda_error(e1 != cudaSuccess ? e1 : e2);
    int64_t *sub_off = reinterpret_cast<int64_t *>(ws + z.sub_off);
    if (int rc = cg_encode_chunk(b.cdf, sym, z.nrows, b.ntokens, z.nchannels, lp, ws + z.scratch, z.stride, lengths,
                                 group_off, sub_off, status, stream))
        return rc;
    if (b.counts)
        if (int rc = launch_sparse_sizes(b.counts, b.table_row_off, b.bins, z.nrows, z.nchannels, group_nz, st)) return rc;
    publish_tail_kernel<<<1, 128, 0, st>>>(sub_off, status, z.nsub,
                                           group_nz ? group_nz + static_cast<int64_t>(z.nrows) * z.nslab : nullptr, b.tail);
    return check_launch();
}

// Shared memory to ask for so that a grid of less than one wave is spread over all SMs.  Blocks that start under the launch in
// front go where that launch's blocks end, up to the eight that fit on an SM, and leave the SMs that end later without any; with
// room for no more than their share of the grid on each, they cannot.  The quantiser and the coder of 256-token chunks, us a
// chunk, with eight blocks an SM and so:
//     10 layers x 8 heads (160 blocks) 66 -> 32    16 x 8 (256) 69 -> 33    32 x 8 (512) 72 -> 47    40 x 8 (640) 74 -> 56
//     32 x 12 (768) 77 -> 66                       32 x 16 (1,024) 84 -> 78
// (one after the other 34, 36, 49, 56, 67 and 79).  Beside chunks on other streams, whose blocks find less room then, it gives
// and takes: twelve chunks by encode_many, 40 x 8 648 -> 610, 32 x 12 694 -> 702, 32 x 16 883 -> 886.  From one wave on there
// is nothing to spread, and evening the waves out does not pay: 80 x 8 (1,280 blocks) takes 96 us as it is, 95 at five and at six an SM;
// 40 x 32 (2,560) 174, and 180 and 176.
static size_t spread_smem(int64_t blocks, size_t dynamic) {
    constexpr int64_t kSmemPerSM = 228 * 1024, kReserved = 1024, kMostResident = 8;  // bytes of an SM, of each block; launch bounds
    const int64_t fit = kSmemPerSM / (static_cast<int64_t>(dynamic) + kMostStaticSmem + kReserved);
    const int64_t sms = sm_count(), share = (blocks + sms - 1) / sms;
    if (share >= (fit < kMostResident ? fit : kMostResident)) return dynamic;
    // the least that keeps one more out, so that the first of them find room beside the launch in front
    const size_t least = static_cast<size_t>(kSmemPerSM / (share + 1) - kReserved + 256);
    return least > dynamic ? least : dynamic;
}

static int encode_jobs(const cg_encode_kv_job *jobs, int njobs, bool alone, void *stream);

extern "C" int cg_encode_kv(const cg_encode_kv_job *job, void *stream) { return encode_jobs(job, 1, true, stream); }

// A single setting is what is left over in front of groups of four (see _encode_infos in cachegen_encoder.py).
extern "C" int cg_encode_kv_levels(const cg_encode_kv_job *jobs, int njobs, void *stream) { return encode_jobs(jobs, njobs, njobs > 1, stream); }

// alone: no other encode follows at once on the stream, or only behind several settings' coder
static int encode_jobs(const cg_encode_kv_job *jobs, int njobs, bool alone, void *stream) {
    if (njobs < 1) return CG_E_SHAPE;
    if (njobs > CG_MAX_ENCODE_LEVELS) return CG_E_CAPACITY;
    if (!jobs) return CG_E_NULL;
    for (int j = 0; j < njobs; ++j) {
        if (int rc = check_job(jobs + j)) return rc;
        if (!same_chunk(jobs[0], jobs[j])) return CG_E_SHAPE;
    }
    const cg_encode_kv_job &b = jobs[0];
    const Sizes z = sizes_of(b.nlayers, b.ntokens, b.nheads, b.head_size);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    for (int j = 0; j < njobs; ++j) jobs[j].tail[z.nsub + 3] = 0;  // host memory: the flag that cg_encode_kv_wait watches
    bool fused = true;
    for (int j = 0; j < njobs; ++j) fused = fused && fused_ok(jobs[j]);
    if (!fused) {
        for (int j = 0; j < njobs; ++j)
            if (int rc = encode_separately(jobs[j], st)) return rc;
        return CG_OK;
    }
    const KvView v{static_cast<const uint16_t *>(b.kv), b.s_layer, b.s_kv, b.s_token, b.s_head,
                   b.nlayers, b.ntokens, b.nheads, b.head_size,
                   0xFFFFFFFFu / static_cast<uint32_t>(b.head_size) + 1u};
    QuantizeLevels q;
    StoreJobs store_jobs;
    TableJobs table_jobs;
    q.n = njobs;
    q.nzeroed = z.nsub + 2;
    int lp = 0;
    for (int j = 0; j < njobs; ++j) {
        const cg_encode_kv_job &k = jobs[j];
        uint8_t *ws = static_cast<uint8_t *>(k.workspace);
        uint32_t *zeroed = reinterpret_cast<uint32_t *>(ws + z.counters);
        q.level[j] = QuantizeOut{k.bins, static_cast<uint16_t *>(k.scales_k), static_cast<uint16_t *>(k.scales_v),
                                 reinterpret_cast<uint32_t *>(ws + z.sym), zeroed, k.max_bins};
        StoreParams &p = store_jobs.job[j];
        p.sym4 = q.level[j].sym4;
        p.out = TableOut{k.cdf, k.counts, k.table_row_off, k.bins, k.counts ? reinterpret_cast<uint32_t *>(ws + z.group_nz) : nullptr};
        p.ntokens = k.ntokens;
        p.nchannels = z.nchannels;
        p.lp = k.max_bins + 1;
        p.nrows = z.nrows;
        p.nsub = z.nsub;
        p.high_water = pair_high_water(k.ntokens) ? deep_pair_high_water(k.ntokens) : 0;
        p.scratch = ws + z.scratch;
        p.stride = z.stride;
        p.lengths = reinterpret_cast<int32_t *>(ws + z.lengths);
        p.group_off = reinterpret_cast<int64_t *>(ws + z.group_off);
        p.sub_bytes = reinterpret_cast<int64_t *>(ws + z.sub_bytes);
        p.tickets = zeroed + 1;
        p.status = reinterpret_cast<int32_t *>(zeroed);
        p.tail = k.tail;
        table_jobs.out[j] = p.out;
        table_jobs.sym4[j] = p.sym4;
        table_jobs.status[j] = p.status;
        table_jobs.lp[j] = p.lp;
        lp = p.lp > lp ? p.lp : lp;
    }
    const dim3 qgrid(static_cast<unsigned>(z.words), static_cast<unsigned>(jobs->nlayers), 2);
    // Two runs of channels a thread from 1,024 channels on; below, what half as many warps have no channels for would cost more
    // (768 channels 7.6 us, 6.8 with one run).  Several settings want more registers.
    const int runs = z.nchannels >= 1024 ? 2 : 1, qthreads = (z.nchannels / 8 + 32 * runs - 1) / (32 * runs) * 32;
#define CG_LAUNCH_QT(DT, THREADS, BLOCKS, BLOCKS_MORE, RUNS)                                                         \
    njobs == 1 ? quantize_tokens_kernel<DT, THREADS, BLOCKS, true, RUNS><<<qgrid, qthreads, 0, st>>>(v, q)            \
               : quantize_tokens_kernel<DT, THREADS, BLOCKS_MORE, false, RUNS><<<qgrid, qthreads, 0, st>>>(v, q)
#define CG_LAUNCH_QD(DT)                                      \
    if (runs == 1) CG_LAUNCH_QT(DT, 128, 12, 12, 1);          \
    else if (qthreads <= 256) CG_LAUNCH_QT(DT, 256, 4, 3, 2); \
    else CG_LAUNCH_QT(DT, 512, 2, 2, 2)
    if (b.dtype == CG_F16) CG_LAUNCH_QD(CG_F16);
    else CG_LAUNCH_QD(CG_BF16);
#undef CG_LAUNCH_QT
#undef CG_LAUNCH_QD
    if (int rc = check_launch()) return rc;
    const dim3 grid(z.nslab, z.nrows, z.nsub * njobs);
    const size_t columns = static_cast<size_t>(lp) * kRowBytes, staged = static_cast<size_t>(lp) * kGroup * 2;
    // The coder of one sub-chunk starts under the quantiser's last blocks: 206 -> 202 us for a 256-token Llama-7B chunk.  Not
    // where another quantiser follows at once, which then starts late, and not behind or in front of the tables' kernel (1,999
    // tokens in one call 415 -> 420).  Three quality levels in one call 197 -> 193.5 us, five in two 278 -> 272.
    const bool early = alone && z.nsub == 1;
    const auto store = [&](auto kernel, int threads, size_t smem) {
        if (early) smem = spread_smem(static_cast<int64_t>(grid.x) * grid.y * grid.z, smem);
        if (int rc = allow_smem(kernel, smem)) return rc;
        return launch(kernel, grid, threads, smem, early, st, store_jobs);
    };
    if (z.nsub == 1) return store(store_encode_kernel<true, 1, 2>, kGroup, columns + staged);
    if (int rc = allow_smem(packed_tables_kernel, columns + staged)) return rc;
    if (int rc = launch(packed_tables_kernel, dim3(z.nslab, z.nrows, njobs), kTableThreads, columns + staged, false, st, table_jobs,
                        static_cast<int>(b.ntokens), static_cast<int>(z.nchannels)))
        return rc;
    if (!store_jobs.job[0].high_water) return store(store_encode_kernel<false, 1, 1>, kGroup, columns);
    // two streams a thread unless the last group has channels for the first alone
    const int last = z.nchannels % kGroup;
    if (last == 0 || last > kGroup / 2) return store(store_encode_kernel<false, 2, 2>, kGroup / 2, columns);
    return store(store_encode_kernel<false, 1, 2>, kGroup, columns);
}

extern "C" int cg_encode_kv_wait(const cg_encode_kv_job *job, void *stream) {
    if (!job || !job->tail) return CG_E_NULL;
    return cg_wait_word(job->tail + (job->ntokens + kSubTokens - 1) / kSubTokens + 3, stream);
}

extern "C" int cg_wait_word(const int64_t *word, void *stream) {
    if (!word) return CG_E_NULL;
    const volatile int64_t *flag = word;
    for (;;) {
        for (int spin = 0; spin < 2000; ++spin)
            if (*flag) {
                __sync_synchronize();
                return CG_OK;
            }
        const cudaError_t e = cudaStreamQuery(static_cast<cudaStream_t>(stream));
        if (e == cudaErrorNotReady) continue;
        if (e != cudaSuccess) return set_cuda_error(e);
        return *flag ? CG_OK : CG_E_SHAPE;  // everything has run and nothing was published: not a started job
    }
}

namespace {
int launch_gather(const cg_encode_kv_job *jobs, int njobs, const Sizes &z, uint8_t *const *bytes, int32_t *const *lengths, cudaStream_t st) {
    GatherJobs g;
    g.nsub = z.nsub;
    for (int j = 0; j < njobs; ++j) {
        const uint8_t *ws = static_cast<const uint8_t *>(jobs[j].workspace);
        g.scratch[j] = ws + z.scratch;
        g.lengths[j] = reinterpret_cast<const int32_t *>(ws + z.lengths);
        g.group_off[j] = reinterpret_cast<const int64_t *>(ws + z.group_off);
    }
    for (int s0 = 0; s0 < z.nsub * njobs; s0 += kGatherSubs) {
        const int n = z.nsub * njobs - s0 < kGatherSubs ? z.nsub * njobs - s0 : kGatherSubs;
        GatherTargets t;
        for (int k = 0; k < n; ++k) {
            t.bytes[k] = bytes[s0 + k];
            t.lengths[k] = lengths[s0 + k];
        }
        const dim3 grid(z.nslab, z.nrows, n);
        if (fused_ok(jobs[0]))  // which of the two encoders wrote the scratch
            gather_kernel<true><<<grid, kGroup, 0, st>>>(g, z.stride, z.nchannels, s0, t);
        else
            gather_kernel<false><<<grid, kGroup, 0, st>>>(g, z.stride, z.nchannels, s0, t);
        if (int rc = check_launch()) return rc;
    }
    return CG_OK;
}
}  // namespace

extern "C" int cg_encode_kv_gather(const cg_encode_kv_job *job, uint8_t *const *bytes_host, int32_t *const *lengths_host,
                                   void *stream) {
    return cg_encode_kv_levels_gather(job, 1, bytes_host, lengths_host, stream);
}

extern "C" int cg_encode_kv_levels_gather(const cg_encode_kv_job *jobs, int njobs, uint8_t *const *bytes_host,
                                          int32_t *const *lengths_host, void *stream) {
    if (njobs < 1) return CG_E_SHAPE;
    if (njobs > CG_MAX_ENCODE_LEVELS) return CG_E_CAPACITY;
    if (!jobs) return CG_E_NULL;
    for (int j = 0; j < njobs; ++j) {
        if (int rc = check_job(jobs + j)) return rc;
        if (!same_chunk(jobs[0], jobs[j])) return CG_E_SHAPE;
    }
    if (!bytes_host || !lengths_host) return CG_E_NULL;
    const Sizes z = sizes_of(jobs->nlayers, jobs->ntokens, jobs->nheads, jobs->head_size);
    for (int k = 0; k < z.nsub * njobs; ++k)
        if (!bytes_host[k] || !lengths_host[k]) return CG_E_NULL;
    return launch_gather(jobs, njobs, z, bytes_host, lengths_host, static_cast<cudaStream_t>(stream));
}

extern "C" int cg_encode_kv_flat(const cg_encode_kv_job *job, const cg_flat_layout *layout, void *stream) {
    if (int rc = check_job(job)) return rc;
    if (!layout) return CG_E_NULL;
    const cg_encode_kv_job &b = *job;
    const cg_flat_layout &f = *layout;
    const Sizes z = sizes_of(b.nlayers, b.ntokens, b.nheads, b.head_size);
    if (!f.blob || !f.header_host || !f.sub_off_host || !f.mask_row_off) return CG_E_NULL;
    if (f.header_bytes <= 0 || f.header_bytes > kMaxHeader || f.off_scales < f.header_bytes || f.off_tables < f.off_scales ||
        f.off_lengths < f.off_tables || f.off_payload < f.off_lengths)
        return CG_E_SHAPE;
    if ((reinterpret_cast<uintptr_t>(f.blob) | f.off_scales | f.off_tables | f.off_lengths) & 15) return CG_E_ALIGN;
    if ((f.table_kind != CG_TABLES_CDF && !b.counts) || f.table_kind < CG_TABLES_CDF || f.table_kind > CG_TABLES_SPARSE) return CG_E_SHAPE;
    if (z.nsub > kMaxHeader / 8) return CG_E_CAPACITY;
    const uint8_t *ws = static_cast<const uint8_t *>(b.workspace);
    ContainerParams p;
    memcpy(p.header, f.header_host, static_cast<size_t>(f.header_bytes));
    memcpy(p.sub_off, f.sub_off_host, 8 * static_cast<size_t>(z.nsub));
    p.header_bytes = static_cast<int>(f.header_bytes);
    p.nsub = z.nsub;
    p.nchannels = z.nchannels;
    p.kind = f.table_kind;
    p.blob = f.blob;
    p.off_scales = f.off_scales;
    p.off_tables = f.off_tables;
    p.tables_bytes = f.tables_bytes;
    p.off_lengths = f.off_lengths;
    p.off_payload = f.off_payload;
    p.off_masks = f.off_masks;
    p.off_counts = f.off_counts;
    p.scales_k = static_cast<const uint16_t *>(b.scales_k);
    p.scales_v = static_cast<const uint16_t *>(b.scales_v);
    p.nscales = static_cast<int64_t>(b.nlayers) * b.ntokens;
    p.tables = f.table_kind == CG_TABLES_CDF ? reinterpret_cast<const uint8_t *>(b.cdf) : b.counts;
    p.count_row_off = b.table_row_off;
    p.mask_row_off = f.mask_row_off;
    p.bins = b.bins;
    p.group_nz = reinterpret_cast<const uint32_t *>(ws + z.group_nz);
    p.scratch = ws + z.scratch;
    p.lengths = reinterpret_cast<const int32_t *>(ws + z.lengths);
    p.group_off = reinterpret_cast<const int64_t *>(ws + z.group_off);
    p.stride = z.stride;
    const dim3 grid(z.nslab, z.nrows, z.nsub + 1);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (fused_ok(b)) container_kernel<true><<<grid, kGroup, 0, st>>>(p);  // which of the two encoders wrote the scratch
    else container_kernel<false><<<grid, kGroup, 0, st>>>(p);
    return check_launch();
}
