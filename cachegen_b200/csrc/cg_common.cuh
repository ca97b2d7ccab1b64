// Shared device helpers of the sm_100a CacheGen codec kernels.
#pragma once

#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include "../../include/cachegen_b200.h"
#include "cg_coder.cuh"

namespace cg {

constexpr int kGroup = kGroupChannels;           // streams (threads) per coder block
constexpr int kRowBytes = kTableRowBytes;        // bytes of one table row in shared memory
static_assert(kGroup == CG_GROUP_CHANNELS, "header and kernels disagree on the group size");
constexpr int kSubTokens = CG_MAX_TOKENS_PER_STREAM;

// ---- error plumbing -------------------------------------------------------------------------
int set_cuda_error(cudaError_t e);  // records the text, returns CG_E_CUDA
inline int check_launch() {
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? CG_OK : set_cuda_error(e);
}

// Dynamic shared memory beyond what a launch gets by itself, 48 KB with the kernel's own arrays: the columns of 64-entry
// tables and their 16-bit copies are 48 KB alone.  Every launch raises its kernel's limit to the same
// value, the most that any of them asks for: a limit that followed the launch could be lowered by another thread between
// this thread's setting it and its launch.
constexpr int64_t kSmemByItself = 48 * 1024, kSmemPerBlock = 227 * 1024;
constexpr int64_t kMostStaticSmem = 256;  // of the kernels that ask
constexpr int64_t kMostDynamicSmem = kSmemPerBlock - kMostStaticSmem;
template <class K>
int allow_smem(K kernel, size_t bytes) {
    if (static_cast<int64_t>(bytes) <= kSmemByItself - kMostStaticSmem) return CG_OK;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kMostDynamicSmem));
    return e == cudaSuccess ? CG_OK : set_cuda_error(e);
}
// ---- launches that overlap the one in front (programmatic dependent launch) ----------------------------------
__device__ __forceinline__ void wait_for_launch_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_launch_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// early: the blocks may start before the launch in front has ended; they call wait_for_launch_before before they touch what
// it reads or writes
template <class... Args>
int launch(void (*kernel)(Args...), dim3 grid, int threads, size_t smem, bool early, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = early ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
    return e == cudaSuccess ? CG_OK : set_cuda_error(e);
}

// multiprocessors of the current device; 1 if it does not say
inline int sm_count() {
    int dev = 0, sms = 0;
    return cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && sms > 0 ? sms : 1;
}

// cg_tables.cu: group offsets of sparse tables
int launch_sparse_sizes(const uint8_t *counts, const int64_t *count_row_off, const float *bins, int nrows, int nchannels,
                        uint32_t *group_off, cudaStream_t st);

// ---- search depth for a table of lp entries ---------------------------------------------------
// Symbols are 0 .. lp-2.  levels = smallest n with 2^n >= lp-1; pow2 when 2^n == lp-1.
inline int search_levels(int lp) {
    int n = 0;
    while ((1 << n) < lp - 1) n++;
    return n;
}

// ---- small PTX wrappers -----------------------------------------------------------------------
__device__ __forceinline__ float ldsf32(uint32_t addr) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t smem_addr(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---- table staging ----------------------------------------------------------------------------
// Every thread owns one (row, channel) table.  It is kept in shared memory as a column tab[m][tid] so that
// lane i always hits bank i, whatever entry m each lane is at: of cdf[m] << 16 for the encoder, of search_entry(cdf[m])
// for the decoder.  Each thread fills (and later reads) only its own column, so no block barrier is needed.  Only the
// entries of the symbols, 0 .. lp-2, are staged; the decoder's rows above them hold kSearchPadding, which a search step
// takes for "above the target", or with REPEAT_LAST copies of the last entry (see decode_streams in cg_coder.cuh).
template <int STRIDE>
__device__ __forceinline__ void stage_encode_column(uint32_t *tab, const int16_t *cdf_row, int lp, int tid) {
    for (int m = 0; m < lp - 1; ++m) tab[m * STRIDE + tid] = static_cast<uint32_t>(static_cast<uint16_t>(__ldg(cdf_row + m))) << 16;
    tab[(lp - 1) * STRIDE + tid] = 0xFFFFFFFFu;
}
template <bool REPEAT_LAST = false>
__device__ __forceinline__ void stage_table_column(uint32_t *tab, const int16_t *cdf_row, int lp, int rows, int tid) {
    const int n = lp - 1 < rows ? lp - 1 : rows;
    uint32_t pad = kSearchPadding, e = 0u;
    for (int m = 0; m < n; ++m) {
        e = search_entry(static_cast<uint32_t>(static_cast<uint16_t>(__ldg(cdf_row + m))));
        tab[m * kGroup + tid] = e;
    }
    if (REPEAT_LAST) pad = e;
    for (int m = n; m < rows; ++m) tab[m * kGroup + tid] = pad;
}

// The same column from the byte counts of the non-centre symbols (CG_TABLES_COUNTS):
// cdf[i] = (uint16)((0xFFFF - max_bins) * #{sym < i} / ntokens) + i, as calculate_cdf builds it
// (cal_cdf.cu:11-15,40-49 in the reference).  cnt points at this channel's first count; counts of one
// symbol are `stride` bytes apart; cq = bins // 2 - 1 is the centre symbol, whose count is implied.
template <bool REPEAT_LAST = false>
__device__ __forceinline__ void stage_table_column_from_counts(uint32_t *tab, const uint8_t *cnt, int64_t stride,
                                                               int cq, int ntokens, int lp, int rows, int tid) {
    const int max_bins = lp - 1;
    uint32_t others = 0;
    for (int j = 0; j < 2 * cq; ++j) others += __ldg(cnt + j * stride);
    const uint32_t centre = static_cast<uint32_t>(ntokens) - others;
    const uint32_t scale = 0xFFFFu - static_cast<uint32_t>(max_bins);
    const uint32_t total = static_cast<uint32_t>(ntokens) & 0xFFFFu;
    const bool pow2 = (total & (total - 1u)) == 0u;
    const int sh = 31 - __clz(static_cast<int>(total | 1u));
    const int n = lp - 1 < rows ? lp - 1 : rows;
    uint32_t cum = 0, pad = kSearchPadding;
    for (int i = 0; i < n; ++i) {
        const uint32_t prod = scale * (cum & 0xFFFFu);
        const uint32_t nv = total ? (pow2 ? (prod >> sh) : (prod / total)) : 0u;
        const uint32_t e = search_entry((nv + static_cast<uint32_t>(i)) & 0xFFFFu);
        tab[i * kGroup + tid] = e;
        if (REPEAT_LAST) pad = e;
        uint32_t count = 0;
        if (i < cq) count = __ldg(cnt + i * stride);
        else if (i == cq) count = centre;
        else if (i <= 2 * cq) count = __ldg(cnt + (i - 1) * stride);
        cum += count;
    }
    for (int i = n; i < rows; ++i) tab[i * kGroup + tid] = pad;
}

// The same column from the sparse byte counts (CG_TABLES_SPARSE): `mask` has bit j set when stored
// symbol j (centre skipped) has a non-zero count, and `nz` points at those counts in rising symbol
// order (nullptr: read them all as zero).  Bound by latency: with the counts read byte by byte as their symbols came up, and a
// division for every entry, 61 tokens of 10 layers x 8 heads took 28.8 us a call, 20.5 this way; 37 of 32 x 8 25.6 and 18.2, 256 of
// 32 x 32 171 and 157.5, 2,048 1,016 and 1,006.
template <bool REPEAT_LAST = false>
__device__ __forceinline__ void stage_table_column_from_sparse(uint32_t *tab, uint32_t mask, const uint8_t *nz, int cq,
                                                               int ntokens, int lp, int rows, int tid) {
    const int max_bins = lp - 1;
    if (2 * cq < 32) mask &= (1u << (2 * cq)) - 1u;
    if (!nz) mask = 0u;
    // the counts, at most 32 bytes, by the aligned words that they lie in, all loads in flight
    const uint32_t lead = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(nz) & 3);
    const uint32_t *words = reinterpret_cast<const uint32_t *>(reinterpret_cast<uintptr_t>(nz) - lead);
    const int end = static_cast<int>(lead) + __popc(mask);
    uint32_t w[9], others = 0;
#pragma unroll
    for (int k = 0; k < 9; ++k) w[k] = mask && 4 * k < end ? __ldg(words + k) : 0u;
    w[0] &= 0xFFFFFFFFu << (8 * lead);
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        if (end - 4 * k < 4) w[k] &= end > 4 * k ? (1u << (8 * (end - 4 * k))) - 1u : 0u;
        others = __dp4a(w[k], 0x01010101u, others);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) w[k] = __funnelshift_r(w[k], w[k + 1], 8 * lead);
    const uint32_t centre = static_cast<uint32_t>(ntokens) - others;
    const uint32_t total = static_cast<uint32_t>(ntokens) & 0xFFFFu;
    const uint32_t scale = total ? 0xFFFFu - static_cast<uint32_t>(max_bins) : 0u;
    const bool pow2 = (total & (total - 1u)) == 0u;
    const int sh = 31 - __clz(static_cast<int>(total | 1u));
    const uint32_t inv = 0xFFFFFFFFu / (total | (total == 0u));  // see counts_to_column
    const int n = lp - 1 < rows ? lp - 1 : rows;
    uint32_t cum = 0, pad = kSearchPadding;
    // four symbols at a time take up to four bytes from the first two words, which are filled up from the others then
#pragma unroll 1
    for (int i0 = 0; i0 < n; i0 += 4) {
        uint32_t taken = 0;  // bits
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int i = i0 + j;
            if (i >= n) break;
            const uint32_t prod = scale * (cum & 0xFFFFu);
            uint32_t nv = prod >> sh;
            if (!pow2) {
                nv = __umulhi(prod, inv);
                if (prod - nv * total >= total) ++nv;
            }
            const uint32_t e = search_entry((nv + static_cast<uint32_t>(i)) & 0xFFFFu);
            tab[i * kGroup + tid] = e;
            if (REPEAT_LAST) pad = e;
            if (i == cq) {
                cum += centre;
            } else {
                const uint32_t bits = (mask & 1u) * 8u;
                mask >>= 1;
                cum += bits ? w[0] & 0xFFu : 0u;
                w[0] = __funnelshift_r(w[0], w[1], bits);
                w[1] >>= bits;
                taken += bits;
            }
        }
        w[1] |= __funnelshift_lc(0u, w[2], 32u - taken);
#pragma unroll
        for (int k = 2; k < 8; ++k) w[k] = __funnelshift_rc(w[k], k < 7 ? w[k + 1] : 0u, taken);
    }
    for (int i = n; i < rows; ++i) tab[i * kGroup + tid] = pad;
}

// ---- block-wide exclusive scan over 32 * NWARPS ints --------------------------------------------
// warp_sums: shared int[NWARPS].  Returns the exclusive prefix of `v` across the block.
template <int NWARPS>
__device__ __forceinline__ int block_exclusive_scan(int v, int *warp_sums, int tid, int *total) {
    const int lane = tid & 31, w = tid >> 5;
    int incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        int n = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += n;
    }
    if (lane == 31) warp_sums[w] = incl;
    __syncthreads();
    int base = 0, all = 0;
#pragma unroll
    for (int i = 0; i < NWARPS; ++i) {
        const int s = warp_sums[i];
        if (i < w) base += s;
        all += s;
    }
    if (total) *total = all;
    return base + incl - v;
}
__device__ __forceinline__ int block_exclusive_scan_128(int v, int *warp_sums, int tid, int *total) {
    return block_exclusive_scan<kGroup / 32>(v, warp_sums, tid, total);
}

// Shared-memory columns of a warp's 32 channels: entry m of lane l at word 32 m + l.  With rows of 128 bytes the
// address of the entry that byte k of a word of symbols names is one dot product: the byte times 128, plus
// the column.
constexpr int kWarpRow = 128;
__device__ __forceinline__ uint32_t entry_of(uint32_t col, uint32_t w, int k) {
    return __dp4a(w, static_cast<uint32_t>(kWarpRow) << (8 * k), col);
}
__device__ __forceinline__ void count_symbol(uint32_t addr) {
    asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(addr) : "memory");
}

// ---- gather of a group's streams (second half of collect_bytes, cachegen_encoder.py:210-222) -----------------
// Called by a block of kGroup threads, one stream each.  A warp's streams are one run of the output: each
// lane shifts its words to the byte they start at and puts them together in shared memory (a word that two
// streams share by an atomic or), and the warp writes the run with 128-bit stores.  Copying stream after stream
// to its place byte by byte took 20 us a 256-token Llama-7B chunk (11.8 MB in 262,144 streams of 45 bytes),
// with words assembled from two source words 24 us: one short dependent copy after the other.  Twelve loads in flight and
// 5 KB of shared memory a warp 15 us under counters, eight and 6 KB 17; eight and 5 KB the same as twelve.
// src: the stream's first word, its words STEP words apart, read-only for the launch; dst0: where the group's
// streams go; pairs: (STEP 1) the words can be read in pairs, to the end of the last one.  Whatever the row holds behind
// its stream: the last word is cut to the stream's bytes, since what it shares a word with there is the next stream (and
// behind the run's last stream the next warp's stage).
constexpr int kGatherWords = 1280;  // words of shared memory a warp

// The streams of some lanes, `total` bytes that go to dst on, through the warp's shared memory.  at: where the lane's own
// stream starts among them, 0 with a len of 0 for the lanes that have no part in it.
template <int STEP>
__device__ __forceinline__ void gather_lanes(uint4 *stage, const uint32_t *src, int len, int at, uint8_t *dst, int total, int lane, bool pairs) {
    const int mis = static_cast<int>(reinterpret_cast<uintptr_t>(dst) & 15u);
    const int nw = (len + 3) >> 2;
    uint32_t *st = reinterpret_cast<uint32_t *>(stage);
    const int units = (mis + total + 15) >> 4;
    for (int i = lane; i < units; i += 32) stage[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncwarp();
    const int o = mis + at, w = o >> 2;
    const uint32_t sh = static_cast<uint32_t>(o & 3) * 8u;
    const uint32_t last_bytes = 0xFFFFFFFFu >> ((-len & 3) * 8);  // of the last word
    const int most = __reduce_max_sync(0xFFFFFFFFu, nw);
    constexpr int kAhead = 12;  // loads in flight
    uint32_t prev = 0u;
    for (int k0 = 0; k0 < most; k0 += kAhead) {
        uint32_t x[kAhead];
        if (STEP == 1 && pairs) {  // a lane reads a row of its own: half as many loads, each of which touches 32 sectors
#pragma unroll
            for (int j = 0; j < kAhead; j += 2) {
                const uint2 q = k0 + j < nw ? __ldg(reinterpret_cast<const uint2 *>(src + k0 + j)) : make_uint2(0u, 0u);
                x[j] = q.x;
                x[j + 1] = k0 + j + 1 < nw ? q.y : 0u;
            }
        } else {
#pragma unroll
            for (int j = 0; j < kAhead; ++j) x[j] = k0 + j < nw ? __ldg(src + (k0 + j) * STEP) : 0u;
        }
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
            const int k = k0 + j;
            if (k < nw) {
                if (k == nw - 1) x[j] &= last_bytes;
                const uint32_t v = __funnelshift_l(prev, x[j], sh);
                if (k == 0 || k == nw - 1) atomicOr(st + w + k, v);
                else st[w + k] = v;
                prev = x[j];
            }
        }
    }
    // what the shift pushed past the last word: not 0 only if the stream's bytes reach into the word there
    const uint32_t over = __funnelshift_l(prev, 0u, sh);
    if (over) atomicOr(st + w + nw, over);
    __syncwarp();
    uint4 *d16 = reinterpret_cast<uint4 *>(dst - mis);
    for (int i = lane; i < units; i += 32) {
        if (i * 16 >= mis && i * 16 + 16 <= mis + total) {
            d16[i] = stage[i];
        } else {
            const uint8_t *b = reinterpret_cast<const uint8_t *>(stage);
            for (int k = max(i * 16, mis); k < min(i * 16 + 16, mis + total); ++k) (dst - mis)[k] = b[k];
        }
    }
}

// A run that does not fit goes in parts of sixteen or of eight streams (of 319 and of 638 bytes on average), and what does not fit
// then byte by byte.  Uniform values at 36 bins, 161 bytes a stream, 32 layers x 32 heads x 256 tokens: 30 us (19 at 159 bytes, in
// one part), 375 byte by byte; row after row 46 and 406.  6 KB a warp take runs of 192 bytes a stream in one part, 20 us, but leave
// room for nine blocks an SM instead of ten: 2,000 tokens of 80 layers x 8 heads, 57 bytes a stream, take 59.9 us instead of 57.6
// (and so they do at the 56 registers a thread that the compiler takes by itself).
template <int STEP>
__device__ __forceinline__ void gather_run(const uint32_t *src, int len, uint8_t *dst0, bool pairs = false) {
    __shared__ uint4 stage[kGroup / 32][kGatherWords / 4];
    __shared__ int warp_sums[kGroup / 32];
    constexpr int kFits = kGatherWords * 4 - 15;  // whatever byte they start at
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int excl = block_exclusive_scan_128(len, warp_sums, tid, nullptr);
    const int first = __shfl_sync(0xFFFFFFFFu, excl, 0), end = __shfl_sync(0xFFFFFFFFu, excl + len, 31);
    if (end - first <= kFits) {
        gather_lanes<STEP>(stage[warp], src, len, excl - first, dst0 + first, end - first, lane, pairs);
        return;
    }
    const int middle = __shfl_sync(0xFFFFFFFFu, excl, 16), part = middle - first <= kFits && end - middle <= kFits ? 16 : 8;
#pragma unroll 1
    for (int l = 0; l < 32; l += part) {
        const int from = __shfl_sync(0xFFFFFFFFu, excl, l), to = __shfl_sync(0xFFFFFFFFu, excl + len, l + part - 1);
        const bool mine = lane >= l && lane < l + part;
        if (to - from <= kFits) {
            __syncwarp();  // the part before has been read
            gather_lanes<STEP>(stage[warp], src, mine ? len : 0, mine ? excl - from : 0, dst0 + from, to - from, lane, pairs);
        } else if (mine) {
            for (int k = 0; k < len; ++k) dst0[excl + k] = static_cast<uint8_t>(__ldg(src + (k >> 2) * STEP) >> (8 * (k & 3)));
        }
    }
}

template <int DT> struct Half16;
template <> struct Half16<CG_F16> {
    static __device__ __forceinline__ float to_float(uint16_t b) { return __half2float(__ushort_as_half(b)); }
    static __device__ __forceinline__ uint16_t from_float(float f) { return __half_as_ushort(__float2half_rn(f)); }
};
template <> struct Half16<CG_BF16> {
    static __device__ __forceinline__ float to_float(uint16_t b) { return __uint_as_float(static_cast<uint32_t>(b) << 16); }
    static __device__ __forceinline__ uint16_t from_float(float f) { return __bfloat16_as_ushort(__float2bfloat16_rn(f)); }
};

__device__ __forceinline__ float half_bits_to_float(uint16_t b, int dtype) {
    return dtype == CG_BF16 ? Half16<CG_BF16>::to_float(b) : Half16<CG_F16>::to_float(b);
}

// Cq of do_dequantize / MAX of torch_quant_vectorized: bins // 2 - 1 on a float tensor.
__device__ __forceinline__ float half_range(float bins) { return __fsub_rn(floorf(__fmul_rn(bins, 0.5f)), 1.0f); }

// Symbols of a row that sparse tables store: all but the centre.
__device__ __forceinline__ int stored_symbols(const float *bins, int row) {
    const int n = 2 * static_cast<int>(half_range(__ldg(bins + row)));
    return n < 32 ? n : 32;  // wider rows cannot be written in this form: the caller rules them out
}

}  // namespace cg
