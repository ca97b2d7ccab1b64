// Arithmetic decoder kernels: one thread per stream, 128 adjacent channels of one row per block.
//
// The per-stream loop lives in cg_coder.cuh; this file stages tables, offsets and scales around it
// and writes either raw symbols (the torchac_cuda entry points) or dequantised 16-bit KV (fused path).
#include <type_traits>

#include "cg_common.cuh"

namespace cg {

// Rows of a staged table: entries 0 .. lp-2 are searched (the entry after the last symbol stands for
// 2^16 and is never read), padded up to the span of the search.
__host__ __device__ inline int table_rows(int lp, int levels) {
    return (1 << levels) > lp - 1 ? (1 << levels) : lp - 1;
}

// What a decode launch follows, when it is launched so that its blocks may start before the launch in front of it
// has ended (programmatic dependent launch).  kAfterOffsets: the group offsets it needs; everything up to
// reading them runs beside that launch.  kAfterBatch: another batch of the same call, on which it does not depend,
// so that its blocks fill what that one's last wave leaves idle; it only must not end first.
enum DecodeAfter { kAfterOffsets = 0, kAfterBatch = 1 };
// A group offset that the launch in front wrote, behind the wait for it (in a later batch: that launch had ended when the
// first batch's blocks let this one start).  From the L2: __ldg is for data that nothing writes while the kernel runs, and
// these blocks may start while that launch still does.
__device__ __forceinline__ int64_t written_offset(const int64_t *p) { return __ldcg(reinterpret_cast<const long long *>(p)); }

// ---- table staging by the block --------------------------------------------------------------------------
// The int16 tables of a block's 128 channels are one contiguous run.  Read channel by channel they are 2-byte
// loads 66 bytes apart, 66 of them one after the other in a thread; here the run is copied to the upper part
// of the table area with 16-byte asynchronous copies and spread into columns from there: the rows below it at
// once, the rest from registers once every thread has read its part.
__device__ __forceinline__ void copy_run_async(void *smem, const void *global, int bytes, int tid, int nthreads) {
    const uint32_t d = smem_addr(smem);
    for (int i = tid * 16; i < bytes; i += nthreads * 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + i), "l"(static_cast<const char *>(global) + i) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void wait_copies() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
constexpr int kMaxStagedLp = 33;  // longer tables would need more registers than the decode loop has
__device__ __forceinline__ int staged_run_offset(int lp, int rows) { return rows * kRowBytes - lp * kGroup * 2; }
// Thread t's channels are 2t and 2t + 1, in columns t and t + 64: their 2 lp entries are lp whole words of the run, which no
// two lanes of a warp read from one bank when lp is odd.  Every thread holds its words before any of them spreads its own.
// rows: the columns' rows, filled up with the last entry.  Called by all threads.
template <int LP>
__device__ __forceinline__ void spread_words(uint32_t *tab, int rows, int tid) {
    const uint32_t *run = tab + (staged_run_offset(LP, rows) >> 2) + tid * LP;
    uint32_t w[LP];
#pragma unroll
    for (int k = 0; k < LP; ++k) w[k] = run[k];
    __syncthreads();
    uint32_t *c0 = tab + tid, *c1 = c0 + kGroup / 2, e = 0u;
#pragma unroll
    for (int h = 0; h < 2 * LP; ++h) {
        const int m = h < LP ? h : h - LP;
        if (m == LP - 1) continue;
        e = __byte_perm(w[h >> 1], 0x4B000000u, h & 1 ? 0x7632 : 0x7610);  // search_entry of one half
        (h < LP ? c0 : c1)[m * kGroup] = e;
    }
    const uint32_t last0 = c0[(LP - 2) * kGroup];
    for (int m = LP - 1; m < rows; ++m) {
        c0[m * kGroup] = last0;
        c1[m * kGroup] = e;
    }
}
__device__ __forceinline__ void spread_run(uint32_t *tab, int lp, int rows, int tid) {
    if (lp == 33) return spread_words<33>(tab, rows, tid);
    if (lp == 17) return spread_words<17>(tab, rows, tid);
    const uint16_t *run = reinterpret_cast<const uint16_t *>(reinterpret_cast<const char *>(tab) + staged_run_offset(lp, rows)) + 2 * tid * lp;
    uint32_t *c0 = tab + tid, *c1 = tab + tid + kGroup / 2;
    const int n = lp - 1;
    uint32_t hold[kMaxStagedLp - 1];
#pragma unroll
    for (int k = 0; k < kMaxStagedLp - 1; ++k)
        hold[k] = k < n ? static_cast<uint32_t>(run[k]) | static_cast<uint32_t>(run[lp + k]) << 16 : 0u;
    const uint32_t last0 = search_entry(run[n - 1]), last1 = search_entry(run[lp + n - 1]);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kMaxStagedLp - 1; ++k)
        if (k < n) {
            c0[k * kGroup] = search_entry(hold[k] & 0xFFFFu);
            c1[k * kGroup] = search_entry(hold[k] >> 16);
        }
    for (int m = n; m < rows; ++m) {
        c0[m * kGroup] = last0;
        c1[m * kGroup] = last1;
    }
}

// A lane behind the last channels decodes what the last lane before it does, from that one's columns, and stores the same to the
// same place: whole warps run the loop, so that neither their votes nor their stores need a mask.
__device__ __forceinline__ void borrow_stream(int64_t &start, int &len, uint32_t lanes) {
    const int from = min(static_cast<int>(threadIdx.x & 31), 31 - __clz(static_cast<int>(lanes)));
    start = __shfl_sync(0xFFFFFFFFu, start, from);
    len = __shfl_sync(0xFFFFFFFFu, len, from);
}

// ---- symbol-output kernels (decode_fast_prefsum / decode_fast_new) -----------------------------------
struct SymDecodeParams {
    const int16_t *cdf;
    const uint8_t *bytes;
    int64_t nbytes;          // total bytes addressable from `bytes`
    const int64_t *prefsum;  // mode 0
    const int32_t *lengths;  // modes 1 and 2
    const int64_t *group_off;  // mode 2: offset of each 128-channel group
    int64_t stream_stride;   // mode 1
    uint8_t *out;
    int64_t o0, o1, o2;
    int ntokens, nchannels, lp;
    int32_t *status;
};

// MODE 0: streams back to back, placed by an inclusive prefix sum of their lengths; 1: one per padded row; 2: back to
// back, placed by group offsets and a scan of the block's lengths.
template <int LEVELS, int MODE>
__global__ void __launch_bounds__(kGroup) decode_symbols_kernel(const SymDecodeParams p) {
    extern __shared__ uint32_t tab[];
    const int tid = threadIdx.x;
    const int row = blockIdx.y;
    const int c = blockIdx.x * kGroup + tid;
    // the lanes that decode together, taken while the warp is still converged
    const uint32_t lanes = __ballot_sync(0xFFFFFFFFu, c < p.nchannels);
    const int64_t g = static_cast<int64_t>(row) * p.nchannels + c;
    int64_t start, len;
    if (MODE == 2) {
        __shared__ int warp_sums[kGroup / 32];
        const int n = c < p.nchannels ? max(0, min(__ldg(p.lengths + g), 1 << 20)) : 0;
        const int excl = block_exclusive_scan_128(n, warp_sums, tid, nullptr);
        wait_for_launch_before();
        start = written_offset(p.group_off + static_cast<int64_t>(row) * gridDim.x + blockIdx.x) + excl;
        len = n;
    }
    if (c >= p.nchannels) return;  // no block barrier from here on
    if (MODE == 0) {
        start = g ? p.prefsum[g - 1] : 0;
        len = p.prefsum[g] - start;
    } else if (MODE == 1) {
        start = g * p.stream_stride;
        len = p.lengths[g];
        if (len > p.stream_stride) len = p.stream_stride;
    }
    bool bad = false;
    if (len < 0) { len = 0; bad = true; }
    if (start < 0) { start = 0; len = 0; bad = true; }
    if (start > p.nbytes) { start = p.nbytes; bad = true; }
    if (start + len > p.nbytes) { len = p.nbytes - start; bad = true; }
    if (len > (1 << 20)) len = 1 << 20;
    if (bad && p.status) atomicOr(p.status, CG_S_BAD_LENGTHS);

    const int rows = table_rows(p.lp, LEVELS);
    stage_table_column(tab, p.cdf + g * p.lp, p.lp, rows, tid);
    uint8_t *o = p.out + row * p.o0 + c * p.o2;
    const int64_t o1 = p.o1;
    const uint32_t col = smem_addr(tab + tid);
    auto emit = [&](uint32_t a) {
        *o = static_cast<uint8_t>((a - col) / kRowBytes);
        o += o1;
    };
    decode_stream<LEVELS>(Smem{}, col, p.lp - 2, p.bytes + start, static_cast<uint32_t>(len), p.ntokens, lanes, emit);
}

// The same with two adjacent channels per thread, whose symbols are adjacent bytes (see decode_dequant_multi_kernel):
// 64 threads a block, one 16-bit store a token.  One 256-token Llama-7B chunk (2,048 blocks): 153 us under counters, eight blocks
// an SM (see evened_blocks), 158 with twelve; 168 with the window shifted at every symbol.
// Shared memory (the tables) allows 12 blocks per SM at the usual table length of 33; asking for no
// more leaves the compiler 80 registers a thread, which it needs to interleave the NS chains.
template <int LEVELS, int MODE>
__global__ void __launch_bounds__(kGroup / 2, kMultiBlocksPerSM) decode_symbols_pair_kernel(const SymDecodeParams p) {
    extern __shared__ uint32_t tab[];
    __shared__ int warp_sums[kGroup / 64];
    constexpr int kThreads = kGroup / 2;
    const int tid = threadIdx.x;
    const int row = blockIdx.y, c0 = blockIdx.x * kGroup + 2 * tid;
    const bool active = c0 < p.nchannels;  // nchannels is even
    const uint32_t lanes = __ballot_sync(0xFFFFFFFFu, active);
    const int64_t g = static_cast<int64_t>(row) * p.nchannels + c0;
    const int rows = table_rows(p.lp, LEVELS) + 1;
    const bool run_staged = p.lp <= kMaxStagedLp && (p.nchannels & 7) == 0 && (reinterpret_cast<uintptr_t>(p.cdf) & 15) == 0 &&
                            static_cast<int>((blockIdx.x + 1) * kGroup) <= p.nchannels;
    if (run_staged)
        copy_run_async(reinterpret_cast<char *>(tab) + staged_run_offset(p.lp, rows),
                       p.cdf + (static_cast<int64_t>(row) * p.nchannels + blockIdx.x * kGroup) * p.lp, p.lp * kGroup * 2, tid, kThreads);
    int64_t start[2] = {0, 0}, len[2] = {0, 0};
    if (MODE == 0) {
        if (active) {
            const int64_t a = g ? p.prefsum[g - 1] : 0, b = p.prefsum[g], e = p.prefsum[g + 1];
            start[0] = a;
            len[0] = b - a;
            start[1] = b;
            len[1] = e - b;
        }
    } else if (MODE == 1) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            start[i] = (g + i) * p.stream_stride;
            len[i] = active ? min(static_cast<int64_t>(p.lengths[g + i]), p.stream_stride) : 0;
        }
    } else {
        if (active) {
            len[0] = max(0, min(__ldg(p.lengths + g), 1 << 20));
            len[1] = max(0, min(__ldg(p.lengths + g + 1), 1 << 20));
        }
        const int excl = block_exclusive_scan<kGroup / 64>(static_cast<int>(len[0] + len[1]), warp_sums, tid, nullptr);
        wait_for_launch_before();
        start[0] = written_offset(p.group_off + static_cast<int64_t>(row) * gridDim.x + blockIdx.x) + excl;
        start[1] = start[0] + len[0];
    }
    if (run_staged) {
        wait_copies();
        __syncthreads();
        spread_run(tab, p.lp, rows, tid);
    } else if (active) {
        stage_table_column<true>(tab, p.cdf + g * p.lp, p.lp, rows, tid);
        stage_table_column<true>(tab, p.cdf + (g + 1) * p.lp, p.lp, rows, tid + kThreads);
    }
    __syncwarp();  // lanes behind the last channel read the last active lane's columns, and a small table meets no block barrier below
    // One search step less where the upper half of the table holds next to nothing, in every channel of the block: the rows of
    // half the bins in a table made for all rows (52 of 64 of a Llama-7B chunk), whose symbols there have one share of 2^16
    // each.  Such a symbol takes the exact search.  175 -> 168 us under counters.
    constexpr uint32_t kHalf = 1u << (LEVELS - 1);
    bool upper = false;
    if (LEVELS > 3 && active && p.lp - 1 > static_cast<int>(kHalf)) {
#pragma unroll
        for (int i = 0; i < 2; ++i) upper |= entry_c16(tab[kHalf * kGroup + tid + i * kThreads]) < (0x10000u - 2u * kHalf) << 16;
    }
    const bool shallow = LEVELS > 3 && !__syncthreads_or(upper);
    if (lanes == 0u) return;  // no block barrier from here on
    bool bad = false;
    const uint8_t *streams[2];
    uint32_t lens[2], col[2];
    const int c = min(c0, p.nchannels - 2);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        if (len[i] < 0) { len[i] = 0; bad = true; }
        if (start[i] < 0) { start[i] = 0; len[i] = 0; bad = true; }
        if (start[i] > p.nbytes) { start[i] = p.nbytes; bad = true; }
        if (start[i] + len[i] > p.nbytes) { len[i] = p.nbytes - start[i]; bad = true; }
        if (len[i] > (1 << 20)) len[i] = 1 << 20;
        int n = static_cast<int>(len[i]);
        if (lanes != 0xFFFFFFFFu) borrow_stream(start[i], n, lanes);
        col[i] = smem_addr(tab + min(tid, static_cast<int>(p.nchannels - blockIdx.x * kGroup) / 2 - 1) + i * kThreads);
        streams[i] = p.bytes + start[i];
        lens[i] = static_cast<uint32_t>(n);
    }
    if (bad && active && p.status) atomicOr(p.status, CG_S_BAD_LENGTHS);
    uint8_t *o = p.out + row * p.o0 + c;
    // the two symbols as bytes of one word: two multiply-adds on the entries' addresses as denormal floats (see search_entry),
    // the first rounded down, the second exact
    uint32_t less = 0x80000000u | ((col[0] >> 9) + (col[1] >> 1));
    int64_t o1 = p.o1;
    asm volatile("" : "+l"(o1), "+r"(less));
    auto emit = [&](const uint32_t (&a)[2], uint32_t) {
        const float m0 = __fmaf_rd(__uint_as_float(a[0]), 1.0f / kRowBytes, __uint_as_float(less));
        const uint32_t both = __float_as_uint(__fmaf_rn(__uint_as_float(a[1]), 256.0f / kRowBytes, m0));
        *reinterpret_cast<uint16_t *>(o) = static_cast<uint16_t>(both);
        o += o1;
    };
    constexpr int kShallow = LEVELS > 3 ? LEVELS - 1 : LEVELS;
    if (shallow) decode_streams<kShallow, 2, true>(Smem{}, col, 0u, p.lp - 2, LEVELS, streams, lens, p.ntokens, 0xFFFFFFFFu, emit);
    else decode_streams<LEVELS, 2, true>(Smem{}, col, 0u, p.lp - 2, LEVELS, streams, lens, p.ntokens, 0xFFFFFFFFu, emit);
}

// ---- one warp per stream (kept for comparison) -------------------------------------------------------------
// The layout usually drawn for a GPU arithmetic decoder: a warp owns one stream, lane m holds table
// entry m in a register, a ballot over "(span * cdf[m]) >> 16 <= value - low" finds the symbol and two
// shuffles fetch its scaled bounds.  It needs no shared memory and no search loop, but all 32 lanes
// repeat the stream's serial range update, so it spends about 30 warp instructions per symbol where
// the thread-per-stream kernels spend 58 for 32 symbols.  Same results; tables of at most 33
// entries; prefix-sum stream layout only.
__global__ void __launch_bounds__(kGroup) decode_symbols_warp_kernel(const SymDecodeParams p, int nrows) {
    const int lane = threadIdx.x & 31;
    const int64_t g = (static_cast<int64_t>(blockIdx.x) * kGroup + threadIdx.x) >> 5;
    if (g >= static_cast<int64_t>(nrows) * p.nchannels) return;
    const int row = static_cast<int>(g / p.nchannels), c = static_cast<int>(g % p.nchannels);
    int64_t start = g ? p.prefsum[g - 1] : 0;
    int64_t len = p.prefsum[g] - start;
    bool bad = false;
    if (len < 0) { len = 0; bad = true; }
    if (start < 0) { start = 0; len = 0; bad = true; }
    if (start > p.nbytes) { start = p.nbytes; bad = true; }
    if (start + len > p.nbytes) { len = p.nbytes - start; bad = true; }
    if (len > (1 << 20)) len = 1 << 20;
    if (bad && lane == 0 && p.status) atomicOr(p.status, CG_S_BAD_LENGTHS);

    const int maxsym = p.lp - 2;
    const uint32_t c16 = lane <= maxsym
                             ? static_cast<uint32_t>(static_cast<uint16_t>(__ldg(p.cdf + g * p.lp + lane))) << 16
                             : 0u;
    BitWindow bw;
    DecoderState st;
    st.init();
    bw.open(p.bytes + start, static_cast<uint32_t>(len));
    uint8_t *o = p.out + row * p.o0 + c * p.o2;
    for (int i = 0; i < p.ntokens; ++i) {
        const uint32_t offset = st.exact_offset(bw);
        const uint32_t f = scale_exact(st.span32, c16);
        const uint32_t votes = __ballot_sync(0xFFFFFFFFu, lane <= maxsym && f <= offset);
        const int sym = 31 - __clz(static_cast<int>(votes | 1u));  // entry 0 is always taken
        if (lane == 0) o[i * p.o1] = static_cast<uint8_t>(sym);
        if (i == p.ntokens - 1) break;
        const uint32_t flo = __shfl_sync(0xFFFFFFFFu, f, sym);
        const uint32_t fnext = __shfl_sync(0xFFFFFFFFu, f, (sym + 1) & 31);
        st.exact_update(flo, sym == maxsym ? st.span32 : fnext);
        if (st.p >= 32) bw.advance(st.p);
    }
}

// ---- fused decode + dequantise + KV-layout store --------------------------------------------------------
struct FusedDecodeParams {
    int njobs, nlayers, nheads, head_size, nchannels, lp, nslab;
    int delta_group;         // 0: every token is coded on its own (the reference's behaviour)
    const float *res_bins;   // anchor-token delta: residual bin count per row, <= 0 for rows without it
    const float *bins;
    int64_t o_layer, o_kv, o_token, o_head;
    int32_t *status;
    int after;  // see DecodeAfter
    cg_decode_job jobs[CG_MAX_DECODE_JOBS];
};

template <int LEVELS, int SCALE_DT, int OUT_DT>
__global__ void __launch_bounds__(kGroup) decode_dequant_kernel(const __grid_constant__ FusedDecodeParams p) {
    extern __shared__ uint32_t smem[];
    __shared__ float scale_f[kSubTokens];
    __shared__ float lut[CG_MAX_LP];
    __shared__ int warp_sums[kGroup / 32];

    const cg_decode_job &job = p.jobs[blockIdx.z];
    const int tid = threadIdx.x;
    const int row = blockIdx.y;
    const int c = blockIdx.x * kGroup + tid;
    const bool active = c < p.nchannels;
    const uint32_t lanes = __ballot_sync(0xFFFFFFFFu, active);  // taken while the warp is still converged
    const int ntok = job.ntokens;
    const int layer = row % p.nlayers, kv = row / p.nlayers;
    const int64_t g = static_cast<int64_t>(row) * p.nchannels + c;

    // stream offsets: group base + exclusive scan of this block's lengths (cachegen_decoder.py:70)
    int len = 0;
    if (active)
        len = job.length_kind == CG_LENGTHS_U16 ? static_cast<int>(__ldg(static_cast<const uint16_t *>(job.lengths) + g))
                                                : __ldg(static_cast<const int32_t *>(job.lengths) + g);
    bool bad = false;
    if (len < 0) { len = 0; bad = true; }
    if (len > (1 << 20)) { len = 1 << 20; bad = true; }
    const int excl = block_exclusive_scan_128(len, warp_sums, tid, nullptr);
    wait_for_launch_before();
    let_next_launch_start();
    int64_t start = written_offset(job.group_off + static_cast<int64_t>(row) * p.nslab + blockIdx.x) + excl;
    if (start < 0) { start = 0; len = 0; bad = true; }
    if (start > job.nbytes) { start = job.nbytes; bad = true; }
    if (start + len > job.nbytes) { len = static_cast<int>(job.nbytes - start); bad = true; }
    if (bad && active && p.status) atomicOr(p.status, CG_S_BAD_LENGTHS);

    // per-token scales of this row and the row's (s - Cq) / Cq table (cachegen_decoder.py:30-32)
    const uint16_t *sc = static_cast<const uint16_t *>(kv ? job.scales_v : job.scales_k) +
                         static_cast<int64_t>(layer) * job.scale_stride;
    for (int t = tid; t < ntok; t += kGroup) scale_f[t] = Half16<SCALE_DT>::to_float(__ldg(sc + t));
    if (tid < p.lp - 1) {
        const float cq = half_range(__ldg(p.bins + row));
        lut[tid] = __fdiv_rn(__fsub_rn(static_cast<float>(tid), cq), cq);
    }
    const int rows = table_rows(p.lp, LEVELS);
    if (job.table_kind == CG_TABLES_SPARSE) {  // the whole block: the counts are found by a scan of the masks
        const int nrows = 2 * p.nlayers;
        const int cq = static_cast<int>(half_range(__ldg(p.bins + row)));
        const uint8_t *base = static_cast<const uint8_t *>(job.tables);
        const int64_t off_masks = (static_cast<int64_t>(nrows) * p.nslab + 1) * 4 + 15 & ~int64_t{15};
        const int64_t off_counts = off_masks + (__ldg(job.table_row_off + nrows) + 15 & ~int64_t{15});
        uint32_t mask = 0;
        bool inside = true;
        if (active) {
            const int width = 2 * cq <= 16 ? 2 : 4;
            const int64_t at_mask = off_masks + __ldg(job.table_row_off + row) + static_cast<int64_t>(c) * width;
            inside = at_mask >= 0 && at_mask + width <= job.tables_nbytes;
            if (inside)
                mask = width == 2 ? __ldg(reinterpret_cast<const uint16_t *>(base + at_mask))
                                  : __ldg(reinterpret_cast<const uint32_t *>(base + at_mask));
            if (2 * cq < 32) mask &= (1u << (2 * cq)) - 1u;
        }
        __syncthreads();  // warp_sums is free again
        const int before = block_exclusive_scan_128(__popc(mask), warp_sums, tid, nullptr);
        const int64_t at = off_counts +
                           __ldg(reinterpret_cast<const uint32_t *>(base) + static_cast<int64_t>(row) * p.nslab + blockIdx.x) +
                           before;
        const bool fits = inside && off_counts <= job.tables_nbytes && at + __popc(mask) <= job.tables_nbytes;
        if (!fits && active && p.status) atomicOr(p.status, CG_S_BAD_TABLE);
        if (active)
            stage_table_column_from_sparse(smem, mask, fits ? base + at : nullptr, cq, job.scale_stride, p.lp,
                                           rows + 1, tid);
    } else if (active) {
        if (job.table_kind == CG_TABLES_COUNTS) {
            const int cq = static_cast<int>(half_range(__ldg(p.bins + row)));
            const int64_t at = __ldg(job.table_row_off + row) + c;
            const bool fits = cq >= 0 && at >= 0 && at + static_cast<int64_t>(2 * cq - 1) * p.nchannels < job.tables_nbytes;
            if (!fits && p.status) atomicOr(p.status, CG_S_BAD_TABLE);
            stage_table_column_from_counts(smem, static_cast<const uint8_t *>(job.tables) + (fits ? at : 0), p.nchannels,
                                           fits ? cq : 0, job.scale_stride, p.lp, rows + 1, tid);
        } else {
            stage_table_column(smem, static_cast<const int16_t *>(job.tables) + g * p.lp, p.lp, rows + 1, tid);
        }
    }
    __syncthreads();
    if (!active) return;

    const int h = c / p.head_size, d = c - h * p.head_size;
    uint16_t *o = static_cast<uint16_t *>(job.out) + layer * p.o_layer + kv * p.o_kv + h * p.o_head + d;
    int64_t o_token = p.o_token;
    const uint32_t col = smem_addr(smem + tid);
    // entry m of the row's (s - Cq)/Cq table is at lut + 4m = lut + (a - col)/128 = (a >> 7) + lut_k,
    // because a - col is a multiple of 512
    uint32_t lut_k = smem_addr(lut) - (col >> 7), sc_a = smem_addr(scale_f);
    int ntok_r = ntok;
    // keep the loop's invariants in registers instead of re-deriving them from kernel parameters
    asm volatile("" : "+l"(o_token), "+r"(lut_k), "+r"(sc_a), "+r"(ntok_r));
    auto emit = [&](uint32_t a) {
        // ((sym - Cq) / Cq) * max in fp32, then one round-to-nearest cast (cachegen_decoder.py:30-33,171-173)
        const float v = __fmul_rn(ldsf32((a >> 7) + lut_k), ldsf32(sc_a));
        *o = Half16<OUT_DT>::from_float(v);
        o += o_token;
        sc_a += 4u;
    };
    decode_stream<LEVELS>(Smem{}, col, p.lp - 2, job.bytes + start, static_cast<uint32_t>(len), ntok_r, lanes, emit);
}

// ---- the same with NS adjacent channels per thread ----------------------------------------------------------
// A block still covers one 128-channel group of one row, with 128 / NS threads: thread t decodes
// channels NS*t .. NS*t + NS-1 side by side (NS independent dependency chains per thread; loop
// control, the warp vote and the token's scale are paid once per NS symbols) and writes their 16-bit
// values with one 2*NS-byte store.  Channel NS*t + i keeps its table in column t + i * (128 / NS), so a
// warp still reads 32 different banks whatever entries its lanes are at.  The search depth is chosen
// per block from the row's bin count (see decode_streams); the result does not depend on it.
// Bound by instruction issue and by the two half-rate integer pipes (52.4 instructions for 32 symbols, four issue slots of
// five).  8,192 Llama-7B tokens: 3.66 ms; 3.68 with the loop begun in front of its estimate; 4.02 and 58.9 instructions with the
// window shifted at every symbol, the shift by the interval's size less one, votes for the active lanes only, 64-bit steps and the
// tables staged by halves of words besides.
// Needs a head size and output strides that are multiples of NS, output pointers aligned to 2*NS bytes and a block's output
// within 32-bit offsets.
template <int OUT_DT>
__device__ __forceinline__ uint32_t pack_pair(float v0, float v1);
template <>
__device__ __forceinline__ uint32_t pack_pair<CG_F16>(float v0, float v1) {
    const __half2 h = __floats2half2_rn(v0, v1);
    return *reinterpret_cast<const uint32_t *>(&h);
}
template <>
__device__ __forceinline__ uint32_t pack_pair<CG_BF16>(float v0, float v1) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v0, v1);
    return *reinterpret_cast<const uint32_t *>(&h);
}

// DELTA (anchor-token delta, see cg_decode_dequant_delta): in rows with residual bins every token that is
// not the first of its group of delta_group adds its value, ((sym - Cq_a) / Cq_r) * max, to its
// anchor's value as the KV dtype holds it; the sum is cast to the output type.
// QUICK: see decode_streams; for grids of at most kQuickBlocksPerSM blocks an SM, which leaves the compiler the registers for it.
// 256 tokens, us a call without and with it: 160 blocks 60.7 and 54.5, 512 66.6 and 62.2, 640 73.9 and 73.1, 1,280 105 and 126;
// 37 tokens of 512 blocks 14.9 and 14.4.
constexpr int kQuickBlocksPerSM = 4;
template <int NS, int OUT_DT, bool DELTA, bool QUICK>
__global__ void __launch_bounds__(kGroup / NS, QUICK ? kQuickBlocksPerSM + 1 : kMultiBlocksPerSM)
decode_dequant_multi_kernel(const __grid_constant__ FusedDecodeParams p, int scale_dt, int full_levels) {
    constexpr int kThreads = kGroup / NS;
    constexpr int kWarps = kThreads / 32;
    extern __shared__ uint32_t smem[];
    __shared__ float scale_f[kSubTokens];
    __shared__ float lut[(DELTA ? 2 : 1) * CG_MAX_LP];  // DELTA: the residual tokens' table follows the anchors'
    __shared__ int warp_sums[kWarps];

    const cg_decode_job &job = p.jobs[blockIdx.z];
    const int tid = threadIdx.x;
    const int row = blockIdx.y;
    const int c0 = blockIdx.x * kGroup + NS * tid;  // nchannels is a multiple of NS: all NS channels exist or none
    const bool active = c0 < p.nchannels;
    const uint32_t lanes = __ballot_sync(0xFFFFFFFFu, active);
    const int ntok = job.ntokens;
    const int layer = row % p.nlayers, kv = row / p.nlayers;
    const int64_t g = static_cast<int64_t>(row) * p.nchannels + c0;

    const int rows = table_rows(p.lp, full_levels < 2 ? 2 : full_levels);  // the register level reads entries 1..3
    // whole groups of 16-byte aligned tables are staged by the block
    const bool run_staged = NS == 2 && job.table_kind == CG_TABLES_CDF && p.lp <= kMaxStagedLp && (p.nchannels & 7) == 0 &&
                            (reinterpret_cast<uintptr_t>(job.tables) & 15) == 0 && static_cast<int>((blockIdx.x + 1) * kGroup) <= p.nchannels;
    if (run_staged)
        copy_run_async(reinterpret_cast<char *>(smem) + staged_run_offset(p.lp, rows + 1),
                       static_cast<const int16_t *>(job.tables) + (static_cast<int64_t>(row) * p.nchannels + blockIdx.x * kGroup) * p.lp,
                       p.lp * kGroup * 2, tid, kThreads);

    // stream lengths
    int len[NS];
    bool bad = false;
    int len_sum = 0;
#pragma unroll
    for (int i = 0; i < NS; ++i) {
        len[i] = 0;
        if (active)
            len[i] = job.length_kind == CG_LENGTHS_U16
                         ? static_cast<int>(__ldg(static_cast<const uint16_t *>(job.lengths) + g + i))
                         : __ldg(static_cast<const int32_t *>(job.lengths) + g + i);
        if (len[i] < 0) { len[i] = 0; bad = true; }
        if (len[i] > (1 << 20)) { len[i] = 1 << 20; bad = true; }
        len_sum += len[i];
    }

    // per-token scales of this row and the row's (s - Cq) / Cq table (cachegen_decoder.py:30-32)
    const uint16_t *sc = static_cast<const uint16_t *>(kv ? job.scales_v : job.scales_k) +
                         static_cast<int64_t>(layer) * job.scale_stride;
    for (int t = tid; t < ntok; t += kThreads) scale_f[t] = half_bits_to_float(__ldg(sc + t), scale_dt);
    const float cqf = half_range(__ldg(p.bins + row));
    for (int m = tid; m < p.lp - 1; m += kThreads) lut[m] = __fdiv_rn(__fsub_rn(static_cast<float>(m), cqf), cqf);
    uint32_t group_mask = 0xFFFFFFFFu;  // token index & group_mask == 0: an anchor (every token without delta)
    if (DELTA) {
        float cqr = 0.0f;
        bool on = false;
        if (p.res_bins) {
            const float rb = __ldg(p.res_bins + row);
            cqr = half_range(rb);
            on = rb > 0.0f && cqr >= 1.0f && cqr <= cqf;
        }
        if (on) {
            group_mask = static_cast<uint32_t>(p.delta_group) * 4u - 1u;  // on four times the token index
            for (int m = tid; m < p.lp - 1; m += kThreads)
                lut[CG_MAX_LP + m] = __fdiv_rn(__fsub_rn(static_cast<float>(m), cqf), cqr);
        } else {
            group_mask = 0u;
        }
    }
    const int cq = cqf >= 0.0f && cqf < 64.0f ? static_cast<int>(cqf) : 64;
    uint32_t *tabs[NS];
#pragma unroll
    for (int i = 0; i < NS; ++i) tabs[i] = smem + min(tid, static_cast<int>(p.nchannels - blockIdx.x * kGroup) / NS - 1) + i * kThreads;
    if (run_staged) {
        wait_copies();
        __syncthreads();
        spread_run(smem, p.lp, rows + 1, tid);
    } else if (job.table_kind == CG_TABLES_SPARSE) {  // the whole block: the counts are found by a scan of the masks
        const int nrows = 2 * p.nlayers;
        const uint8_t *base = static_cast<const uint8_t *>(job.tables);
        const int64_t off_masks = (static_cast<int64_t>(nrows) * p.nslab + 1) * 4 + 15 & ~int64_t{15};
        const int64_t off_counts = off_masks + (__ldg(job.table_row_off + nrows) + 15 & ~int64_t{15});
        uint32_t mask[NS];
        int nset[NS], nset_sum = 0;
        bool inside = true;
        const int width = 2 * cq <= 16 ? 2 : 4;
        const int64_t at_mask = off_masks + __ldg(job.table_row_off + row) + static_cast<int64_t>(c0) * width;
        if (active) inside = at_mask >= 0 && at_mask + NS * width <= job.tables_nbytes;
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            mask[i] = 0;
            if (active && inside)
                mask[i] = width == 2 ? __ldg(reinterpret_cast<const uint16_t *>(base + at_mask) + i)
                                     : __ldg(reinterpret_cast<const uint32_t *>(base + at_mask) + i);
            if (2 * cq < 32) mask[i] &= (1u << (2 * cq)) - 1u;
            nset[i] = __popc(mask[i]);
            nset_sum += nset[i];
        }
        const int before = block_exclusive_scan<kWarps>(nset_sum, warp_sums, tid, nullptr);
        int64_t at = off_counts +
                     __ldg(reinterpret_cast<const uint32_t *>(base) + static_cast<int64_t>(row) * p.nslab + blockIdx.x) +
                     before;
        const bool fits = inside && off_counts <= job.tables_nbytes && at + nset_sum <= job.tables_nbytes;
        if (!fits && active && p.status) atomicOr(p.status, CG_S_BAD_TABLE);
        if (active) {
#pragma unroll
            for (int i = 0; i < NS; ++i) {
                stage_table_column_from_sparse<true>(tabs[i], mask[i], fits ? base + at : nullptr, cq, job.scale_stride, p.lp,
                                               rows + 1, 0);
                at += nset[i];
            }
        }
    } else if (active) {
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            if (job.table_kind == CG_TABLES_COUNTS) {
                const int64_t at = __ldg(job.table_row_off + row) + c0 + i;
                const bool fits = at >= 0 && at + static_cast<int64_t>(2 * cq - 1) * p.nchannels < job.tables_nbytes;
                if (!fits && p.status) atomicOr(p.status, CG_S_BAD_TABLE);
                stage_table_column_from_counts<true>(tabs[i], static_cast<const uint8_t *>(job.tables) + (fits ? at : 0),
                                               p.nchannels, fits ? cq : 0, job.scale_stride, p.lp, rows + 1, 0);
            } else {
                stage_table_column<true>(tabs[i], static_cast<const int16_t *>(job.tables) + (g + i) * p.lp, p.lp, rows + 1, 0);
            }
        }
    }
    __syncthreads();  // warp_sums is free again
    // stream offsets: group base + exclusive scan of this block's lengths (cachegen_decoder.py:70)
    const int excl = block_exclusive_scan<kWarps>(len_sum, warp_sums, tid, nullptr);
    if (p.after == kAfterOffsets) wait_for_launch_before();
    let_next_launch_start();
    int64_t start[NS];
    start[0] = written_offset(job.group_off + static_cast<int64_t>(row) * p.nslab + blockIdx.x) + excl;
#pragma unroll
    for (int i = 1; i < NS; ++i) start[i] = start[i - 1] + len[i - 1];
#pragma unroll
    for (int i = 0; i < NS; ++i) {
        if (start[i] < 0) { start[i] = 0; len[i] = 0; bad = true; }
        if (start[i] > job.nbytes) { start[i] = job.nbytes; bad = true; }
        if (start[i] + len[i] > job.nbytes) { len[i] = static_cast<int>(job.nbytes - start[i]); bad = true; }
    }
    if (bad && active && p.status) atomicOr(p.status, CG_S_BAD_LENGTHS);
    __syncthreads();
    if (lanes == 0u) {
        if (p.after == kAfterBatch) wait_for_launch_before();
        return;
    }

    const int c = min(c0, p.nchannels - NS);
    uint32_t col[NS];
    const uint8_t *streams[NS];
    uint32_t lens[NS];
#pragma unroll
    for (int i = 0; i < NS; ++i) {
        if (lanes != 0xFFFFFFFFu) borrow_stream(start[i], len[i], lanes);
        col[i] = smem_addr(tabs[i]);
        streams[i] = job.bytes + start[i];
        lens[i] = static_cast<uint32_t>(len[i]);
    }
    // Byte offsets from the block's first head, which is the same for all threads, fit 32 bits (offsets_fit; DELTA takes any).
    using Offset = std::conditional_t<DELTA, int64_t, uint32_t>;
    const int h0 = blockIdx.x * kGroup / p.head_size, h = c / p.head_size, d = c - h * p.head_size;
    char *out = reinterpret_cast<char *>(static_cast<uint16_t *>(job.out) + layer * p.o_layer + kv * p.o_kv + h0 * p.o_head);
    Offset o = (static_cast<Offset>(h - h0) * static_cast<Offset>(p.o_head) + static_cast<Offset>(d)) * 2;
    Offset o_token = static_cast<Offset>(p.o_token) * 2;
    // entry m of the row's (s - Cq)/Cq table is at lut + 4m: a 128th of an entry's address, rounded down, plus a constant, taken
    // as denormal floats (see search_entry), because a - col is a multiple of 512
    uint32_t lut_k[NS];
    const uint32_t sc_a = smem_addr(scale_f);
    int ntok_r = ntok;
    // keep the loop's invariants in registers instead of re-deriving them from kernel parameters
    if constexpr (DELTA) asm volatile("" : "+l"(o_token), "+r"(ntok_r));
    else asm volatile("" : "+r"(o_token), "+r"(ntok_r));
#pragma unroll
    for (int i = 0; i < NS; ++i) {
        lut_k[i] = smem_addr(lut) - (col[i] >> 7);
        asm volatile("" : "+r"(lut_k[i]));
    }
    float anchor[NS];
#pragma unroll
    for (int i = 0; i < NS; ++i) anchor[i] = 0.0f;
    // at: the address of the token's scale
    auto emit = [&](const uint32_t (&a)[NS], uint32_t at) {
        // ((sym - Cq) / Cq) * max in fp32, then one round-to-nearest cast (cachegen_decoder.py:30-33,171-173)
        const float s = ldsf32(at);

        float v[NS];
        uint32_t entry[NS];
#pragma unroll
        for (int i = 0; i < NS; ++i)
            entry[i] = __float_as_uint(__fmaf_rd(__uint_as_float(a[i]), 4.0f / kRowBytes, __uint_as_float(lut_k[i])));
        if (!DELTA || ((at - sc_a) & group_mask) == 0u) {
#pragma unroll
            for (int i = 0; i < NS; ++i) {
                v[i] = __fmul_rn(ldsf32(entry[i]), s);
                if (DELTA)  // what the encoder subtracted from the group's other tokens: the value in the KV dtype
                    anchor[i] = scale_dt == CG_BF16 ? Half16<CG_BF16>::to_float(Half16<CG_BF16>::from_float(v[i]))
                                                    : Half16<CG_F16>::to_float(Half16<CG_F16>::from_float(v[i]));
            }
        } else {
#pragma unroll
            for (int i = 0; i < NS; ++i)
                v[i] = __fadd_rn(anchor[i], __fmul_rn(ldsf32(entry[i] + 4u * CG_MAX_LP), s));
        }
        if (NS == 2) {
            *reinterpret_cast<uint32_t *>(out + o) = pack_pair<OUT_DT>(v[0], v[1]);
        } else {
            *reinterpret_cast<uint2 *>(out + o) = make_uint2(pack_pair<OUT_DT>(v[0], v[1]), pack_pair<OUT_DT>(v[2 % NS], v[3 % NS]));
        }
        o += o_token;
    };
    const int maxsym = p.lp - 2;
    const int fl = fast_levels_for(2 * cq + 1, full_levels);
    const int top = (1 << fl) - 1;
    const uint32_t det = smem_addr(smem) + static_cast<uint32_t>(top < maxsym ? top : maxsym) * kRowBytes;
    switch (fl) {
    case 2: decode_streams<2, NS, true, QUICK>(Smem{}, col, det, maxsym, full_levels, streams, lens, ntok_r, 0xFFFFFFFFu, emit, sc_a); break;
    case 3: decode_streams<3, NS, true, QUICK>(Smem{}, col, det, maxsym, full_levels, streams, lens, ntok_r, 0xFFFFFFFFu, emit, sc_a); break;
    case 4: decode_streams<4, NS, true, QUICK>(Smem{}, col, det, maxsym, full_levels, streams, lens, ntok_r, 0xFFFFFFFFu, emit, sc_a); break;
    case 5: decode_streams<5, NS, true, QUICK>(Smem{}, col, det, maxsym, full_levels, streams, lens, ntok_r, 0xFFFFFFFFu, emit, sc_a); break;
    default: decode_streams<6, NS, true, QUICK>(Smem{}, col, det, maxsym, full_levels, streams, lens, ntok_r, 0xFFFFFFFFu, emit, sc_a); break;
    }
    if (p.after == kAfterBatch) wait_for_launch_before();
}

// ---- launch helpers -------------------------------------------------------------------------------------
// dynamic shared memory of a decoder block: the streams' table columns, at most 33 KB
static size_t table_bytes(int lp, int levels) {
    return static_cast<size_t>(table_rows(lp, levels) + 1) * kRowBytes;  // +1: the row read past the last symbol
}
static_assert((CG_MAX_LP + 1) * kRowBytes + 4 * (kSubTokens + 2 * CG_MAX_LP) + 64 <= kSmemByItself, "a decoder block's shared memory");

// Shared memory to ask for so that a grid has as many blocks an SM as evened_blocks says.
template <class Kernel>
static size_t evened_smem(Kernel kernel, int64_t blocks, int levels, bool symbols, int chunks, int ntokens, size_t dynamic) {
    constexpr int64_t kSmemPerSM = 228 * 1024, kReserved = 1024;  // bytes of an SM, of each block
    const int resident = evened_blocks(blocks, sm_count(), levels, symbols, chunks, ntokens);
    cudaFuncAttributes at;
    if (!resident || cudaFuncGetAttributes(&at, kernel) != cudaSuccess) return dynamic;
    const int64_t fixed = static_cast<int64_t>(at.sharedSizeBytes) + kReserved;
    const size_t least = static_cast<size_t>(kSmemPerSM / (resident + 1) - fixed + 256);  // that keeps one more out
    return least > dynamic ? least : dynamic;
}

// Instantiated search depths: 3..6, whatever the table length.
template <int MODE>
static int launch_symbols(const SymDecodeParams &p, int nrows, cudaStream_t st) {
    const int need = search_levels(p.lp);
    const dim3 grid((p.nchannels + kGroup - 1) / kGroup, nrows);
    const int64_t blocks = static_cast<int64_t>(grid.x) * grid.y;
    const bool pairs = p.o2 == 1 && ((p.o0 | p.o1 | p.nchannels) & 1) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 1) == 0;
#define CG_LAUNCH_SYM(L)                                                                                      \
    return pairs ? launch(decode_symbols_pair_kernel<L, MODE>, grid, kGroup / 2,                               \
                          evened_smem(decode_symbols_pair_kernel<L, MODE>, blocks, L, true, 1, p.ntokens, table_bytes(p.lp, L)), MODE == 2, st, p) \
                 : launch(decode_symbols_kernel<L, MODE>, grid, kGroup, table_bytes(p.lp, L), MODE == 2, st, p)
    if (need <= 3) CG_LAUNCH_SYM(3);
    if (need == 4) CG_LAUNCH_SYM(4);
    if (need == 5) CG_LAUNCH_SYM(5);
    CG_LAUNCH_SYM(6);
#undef CG_LAUNCH_SYM
}

template <int SCALE_DT, int OUT_DT>
static int launch_fused(const FusedDecodeParams &p, bool early, cudaStream_t st) {
    const int need = search_levels(p.lp);
    const dim3 grid(p.nslab, 2 * p.nlayers, p.njobs);
#define CG_LAUNCH_FUSED(L) \
    return launch(decode_dequant_kernel<L, SCALE_DT, OUT_DT>, grid, kGroup, table_bytes(p.lp, L), early, st, p)
    if (need <= 3) CG_LAUNCH_FUSED(3);
    if (need == 4) CG_LAUNCH_FUSED(4);
    if (need == 5) CG_LAUNCH_FUSED(5);
    CG_LAUNCH_FUSED(6);
#undef CG_LAUNCH_FUSED
}

// The NS-channels-per-thread kernel needs the NS channels of a thread in one head and aligned packed stores.
static bool multi_layout_ok(const FusedDecodeParams &p, int ns) {
    if ((p.head_size | p.o_layer | p.o_kv | p.o_token | p.o_head) & (ns - 1)) return false;
    for (int j = 0; j < p.njobs; ++j)
        if (reinterpret_cast<uintptr_t>(p.jobs[j].out) & (2 * ns - 1)) return false;
    return true;
}

// A block's output within 32-bit byte offsets of its first head: 256 tokens of the heads that 128 channels touch.  A head's
// tokens 2 GB apart in all go to the general kernel, which takes 64-bit steps.
static bool offsets_fit(const FusedDecodeParams &p) {
    const int64_t most = (int64_t{1} << 31) - p.head_size, heads = kGroup / p.head_size + 1;
    return p.o_token >= 0 && p.o_head >= 0 && p.o_head <= most / heads && p.o_token <= (most - heads * p.o_head) / kSubTokens;
}

template <int NS, int OUT_DT, bool DELTA>
static int launch_fused_multi(const FusedDecodeParams &p, int scale_dt, bool early, cudaStream_t st) {
    const int full = search_levels(p.lp);
    const dim3 grid(p.nslab, 2 * p.nlayers, p.njobs);
    const int64_t blocks = static_cast<int64_t>(grid.x) * grid.y * grid.z;
    const size_t smem = table_bytes(p.lp, full < 2 ? 2 : full);
    if (!DELTA && blocks <= static_cast<int64_t>(kQuickBlocksPerSM) * sm_count())
        return launch(decode_dequant_multi_kernel<NS, OUT_DT, DELTA, !DELTA>, grid, kGroup / NS, smem, early, st, p, scale_dt, full);
    const auto kernel = decode_dequant_multi_kernel<NS, OUT_DT, DELTA, false>;
    const size_t asked = DELTA ? smem : evened_smem(kernel, blocks, full, false, p.njobs, p.jobs[0].ntokens, smem);
    return launch(kernel, grid, kGroup / NS, asked, early, st, p, scale_dt, full);
}

// ---- group offsets ------------------------------------------------------------------------------------------
// One cluster of BLOCKS blocks per job: every block sums the lengths of its share of the 128-channel groups and
// scans its sums, then adds the totals of the blocks before it, which it reads in their shared memory.  One
// launch where a sum kernel and a scan kernel were two (5 us of 23 for a 37-token chunk), and nothing to zero.  Bound
// by latency: 4.2 us for 20,480 lengths in eight blocks with four groups in flight a warp, 13.9 for 262,144, which take 10 in
// sixteen blocks with eight.  Its blocks are launched early and wait for the launch in front before they read anything, the decode's
// start once all of them have waited: 1 to 4 us less a call.
struct OffsetJobs {
    const void *lengths[CG_MAX_DECODE_JOBS];
    int64_t *group_off[CG_MAX_DECODE_JOBS];
    int64_t expect[CG_MAX_DECODE_JOBS];
    int32_t kind[CG_MAX_DECODE_JOBS];
};
constexpr int64_t kWideOffsets = 1024;
constexpr int kOffsetThreads = 512, kMaxOffsetGroups = CG_MAX_OFFSET_GROUPS;

// For callers that wait for the sum of one job's lengths (tail: host memory that the GPU can write): [0] the sum,
// [1] 1 if a length is negative or above `longest`, [2] the word at `extra`, then [3] becomes 1.
struct StreamSizes {
    int64_t *tail;
    const int32_t *extra;
    int longest;
};

__device__ __forceinline__ int clamped_length(int v, int longest, bool *bad) {
    if (v < 0) { v = 0; *bad = true; }
    if (v > longest) { v = longest; *bad = true; }
    return v;
}

template <int BLOCKS, int AHEAD>  // AHEAD: groups a warp has in flight
__global__ void __cluster_dims__(BLOCKS, 1, 1) __launch_bounds__(kOffsetThreads)
group_offsets_kernel(const __grid_constant__ OffsetJobs jobs, int nrows, int nchannels, int nslab, int32_t *status,
                     const StreamSizes sizes, bool behind_another) {
    extern __shared__ int sums[];  // the groups of this block
    __shared__ int64_t warp_sums[kOffsetThreads / 32];
    __shared__ int64_t block_total;
    __shared__ uint32_t block_bad;
    // Behind another batch of the same call, whose blocks have waited for what is in front of both by the time these start, they run
    // beside those; they only must not end first.
    if (!behind_another) wait_for_launch_before();
    let_next_launch_start();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) block_bad = 0u;
    const int j = blockIdx.x / BLOCKS, rank = blockIdx.x % BLOCKS;
    const int ngroups = nrows * nslab, per = (ngroups + BLOCKS - 1) / BLOCKS;
    const int first = min(ngroups, rank * per), count = min(ngroups, first + per) - first;
    const bool u16 = jobs.kind[j] == CG_LENGTHS_U16;
    const void *lengths = jobs.lengths[j];
    // four lengths a load where the rows allow it
    const bool vec = nchannels % kGroup == 0 && (reinterpret_cast<uintptr_t>(lengths) & (u16 ? 7 : 15)) == 0;
    bool bad = false;
    constexpr int kWarps = kOffsetThreads / 32;
    if (vec) {
        for (int k0 = warp; k0 < count; k0 += kWarps * AHEAD) {
            int s[AHEAD];
#pragma unroll
            for (int i = 0; i < AHEAD; ++i) {
                const int k = k0 + i * kWarps;
                const int64_t at = static_cast<int64_t>(first + k) * 32 + lane;
                int4 q = make_int4(0, 0, 0, 0);
                if (k < count) {
                    if (u16) {
                        const ushort4 h = __ldg(static_cast<const ushort4 *>(lengths) + at);
                        q = make_int4(h.x, h.y, h.z, h.w);
                    } else {
                        q = __ldg(static_cast<const int4 *>(lengths) + at);
                    }
                }
                s[i] = clamped_length(q.x, sizes.longest, &bad) + clamped_length(q.y, sizes.longest, &bad) +
                       clamped_length(q.z, sizes.longest, &bad) + clamped_length(q.w, sizes.longest, &bad);
            }
#pragma unroll
            for (int i = 0; i < AHEAD; ++i) {
                s[i] = __reduce_add_sync(0xFFFFFFFFu, s[i]);
                if (lane == 0 && k0 + i * kWarps < count) sums[k0 + i * kWarps] = s[i];
            }
        }
    } else {
        for (int k = warp; k < count; k += kWarps) {
            const int row = (first + k) / nslab, slab = (first + k) % nslab;
            int s = 0;
            for (int c = slab * kGroup + lane; c < min(nchannels, (slab + 1) * kGroup); c += 32) {
                const int64_t at = static_cast<int64_t>(row) * nchannels + c;
                s += clamped_length(u16 ? static_cast<int>(__ldg(static_cast<const uint16_t *>(lengths) + at))
                                        : __ldg(static_cast<const int32_t *>(lengths) + at), sizes.longest, &bad);
            }
            s = __reduce_add_sync(0xFFFFFFFFu, s);
            if (lane == 0) sums[k] = s;
        }
    }
    __syncthreads();
    if (bad) block_bad = 1u;
    // exclusive scan: a run of groups per thread
    const int run = (count + kOffsetThreads - 1) / kOffsetThreads, b = min(count, tid * run), e = min(count, b + run);
    int64_t local = 0;
    for (int k = b; k < e; ++k) local += sums[k];
    int64_t incl = local;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int64_t v = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += v;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    int64_t at = incl - local, total = 0;
#pragma unroll
    for (int k = 0; k < kOffsetThreads / 32; ++k) {
        if (k < warp) at += warp_sums[k];
        total += warp_sums[k];
    }
    if (tid == 0) block_total = total;
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
    int64_t all = 0;
#pragma unroll
    for (int r = 0; r < BLOCKS; ++r) {
        uint32_t remote;
        int64_t v;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_addr(&block_total)), "r"(r));
        asm volatile("ld.shared::cluster.s64 %0, [%1];" : "=l"(v) : "r"(remote));
        if (r < rank) at += v;
        all += v;
    }
    int64_t *out = jobs.group_off[j] + first;
    for (int k = b; k < e; ++k) {
        out[k] = at;
        at += sums[k];
    }
    if (status && (bad || (rank == 0 && tid == 0 && all != jobs.expect[j]))) atomicOr(status, CG_S_BAD_LENGTHS);
    if (sizes.tail && rank == 0 && tid == 0) {
        uint32_t any = 0;
        for (int r = 0; r < BLOCKS; ++r) {
            uint32_t remote, v;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_addr(&block_bad)), "r"(r));
            asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(remote));
            any |= v;
        }
        sizes.tail[0] = all;
        sizes.tail[1] = any;
        sizes.tail[2] = sizes.extra ? *sizes.extra : 0;
        __threadfence_system();
        *reinterpret_cast<volatile int64_t *>(sizes.tail + 3) = 1;
    }
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");  // the totals have been read
    if (behind_another) wait_for_launch_before();
}

static int launch_offsets(const cg_decode_job *jobs, int njobs, int nrows, int nchannels, int32_t *status, cudaStream_t st,
                          const StreamSizes &sizes = StreamSizes{nullptr, nullptr, 1 << 20}, bool behind_another = false) {
    OffsetJobs o;
    for (int j = 0; j < njobs; ++j) {
        o.lengths[j] = jobs[j].lengths;
        o.group_off[j] = const_cast<int64_t *>(jobs[j].group_off);
        o.expect[j] = jobs[j].nbytes;
        o.kind[j] = jobs[j].length_kind;
    }
    const int nslab = (nchannels + kGroup - 1) / kGroup;
    const int64_t groups = static_cast<int64_t>(nrows) * nslab;
    const auto run = [&](auto kernel, int blocks) {
        const size_t sums = static_cast<size_t>((groups + blocks - 1) / blocks) * sizeof(int);
        return launch(kernel, dim3(static_cast<unsigned>(njobs * blocks)), kOffsetThreads, sums, true, st,
                      o, nrows, nchannels, nslab, status, sizes, behind_another);
    };
    // Sixteen blocks where a warp of eight would take more than eight groups, in more than two rounds of loads.  20 tokens, us a
    // call with eight and with sixteen: 640 groups 12.8 and 13.1, 768 12.9 and 12.9, 1,280 16.9 and 15.8, 2,048 25.4 and 23.4.
    // Such clusters have to be allowed, and where a GPU (a part of one, say) has no room for them eight blocks do as well.
    if (groups > kWideOffsets) {
        const auto wide = group_offsets_kernel<16, 8>;
        if (cudaFuncSetAttribute(wide, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
            if (run(wide, 16) == CG_OK) return CG_OK;
        }
        cudaGetLastError();
    }
    return run(group_offsets_kernel<8, 4>, 8);
}

}  // namespace cg

using namespace cg;

static int check_coder_shape(int nrows, int ntokens, int nchannels, int lp) {
    if (nrows <= 0 || ntokens <= 0 || nchannels <= 0) return CG_E_SHAPE;
    if (ntokens > CG_MAX_TOKENS_PER_STREAM) return CG_E_TOKENS;
    if (lp < 2 || lp > CG_MAX_LP) return CG_E_LP;
    if (nrows > 65535) return CG_E_SHAPE;
    return CG_OK;
}

extern "C" int cg_decode_prefsum(const int16_t *cdf, const uint8_t *bytes, int64_t nbytes,
                                 const int64_t *prefsum, uint8_t *out, const int64_t out_strides[3],
                                 int nrows, int ntokens, int nchannels, int lp, int32_t *status,
                                 void *stream) {
    if (!cdf || !prefsum || !out || !out_strides || (!bytes && nbytes > 0)) return CG_E_NULL;
    if (nbytes < 0) return CG_E_SHAPE;
    if (int rc = check_coder_shape(nrows, ntokens, nchannels, lp)) return rc;
    SymDecodeParams p{cdf, bytes, nbytes, prefsum, nullptr, nullptr, 0, out, out_strides[0], out_strides[1],
                      out_strides[2], ntokens, nchannels, lp, status};
    return launch_symbols<0>(p, nrows, static_cast<cudaStream_t>(stream));
}

extern "C" int cg_decode_prefsum_warp(const int16_t *cdf, const uint8_t *bytes, int64_t nbytes,
                                      const int64_t *prefsum, uint8_t *out, const int64_t out_strides[3],
                                      int nrows, int ntokens, int nchannels, int lp, int32_t *status,
                                      void *stream) {
    if (!cdf || !prefsum || !out || !out_strides || (!bytes && nbytes > 0)) return CG_E_NULL;
    if (nbytes < 0) return CG_E_SHAPE;
    if (int rc = check_coder_shape(nrows, ntokens, nchannels, lp)) return rc;
    if (lp > 33) return CG_E_LP;
    SymDecodeParams p{cdf, bytes, nbytes, prefsum, nullptr, nullptr, 0, out, out_strides[0], out_strides[1],
                      out_strides[2], ntokens, nchannels, lp, status};
    const int64_t nstreams = static_cast<int64_t>(nrows) * nchannels;
    const int64_t blocks = (nstreams * 32 + kGroup - 1) / kGroup;
    if (blocks > 0x7FFFFFFF) return CG_E_SHAPE;
    decode_symbols_warp_kernel<<<static_cast<unsigned>(blocks), kGroup, 0, static_cast<cudaStream_t>(stream)>>>(p, nrows);
    return check_launch();
}

extern "C" int cg_decode_padded(const int16_t *cdf, const uint8_t *streams, int64_t stream_stride,
                                const int32_t *lengths, uint8_t *out, const int64_t out_strides[3],
                                int nrows, int ntokens, int nchannels, int lp, int32_t *status,
                                void *stream) {
    if (!cdf || !streams || !lengths || !out || !out_strides) return CG_E_NULL;
    if (stream_stride <= 0) return CG_E_SHAPE;
    if (int rc = check_coder_shape(nrows, ntokens, nchannels, lp)) return rc;
    SymDecodeParams p{cdf, streams, static_cast<int64_t>(nrows) * nchannels * stream_stride, nullptr,
                      lengths, nullptr, stream_stride, out, out_strides[0], out_strides[1], out_strides[2],
                      ntokens, nchannels, lp, status};
    return launch_symbols<1>(p, nrows, static_cast<cudaStream_t>(stream));
}

// Checks the arguments of the fused decode and fills the kernel parameters; launches nothing.
static int fused_params(const cg_decode_job *jobs_host, int njobs, int nlayers, int nheads, int head_size, int lp,
                        const float *bins, int scale_dtype, int out_dtype, int64_t o_layer, int64_t o_kv,
                        int64_t o_token, int64_t o_head, int32_t *status, FusedDecodeParams &p) {
    if (!jobs_host || !bins) return CG_E_NULL;
    if (njobs <= 0 || nlayers <= 0 || nheads <= 0 || head_size <= 0) return CG_E_SHAPE;
    if (njobs > CG_MAX_DECODE_JOBS) return CG_E_CAPACITY;
    if (lp < 2 || lp > CG_MAX_LP) return CG_E_LP;
    if (nlayers > 32767) return CG_E_SHAPE;  // 2 * nlayers rows are a grid dimension
    if (static_cast<int64_t>(nheads) * head_size > 0x7FFFFFFF - kGroup) return CG_E_SHAPE;
    if ((scale_dtype != CG_F16 && scale_dtype != CG_BF16) || (out_dtype != CG_F16 && out_dtype != CG_BF16))
        return CG_E_DTYPE;
    p.njobs = njobs;
    p.nlayers = nlayers;
    p.nheads = nheads;
    p.head_size = head_size;
    p.nchannels = nheads * head_size;
    p.lp = lp;
    p.nslab = (p.nchannels + kGroup - 1) / kGroup;
    p.delta_group = 0;
    p.res_bins = nullptr;
    p.bins = bins;
    p.o_layer = o_layer;
    p.o_kv = o_kv;
    p.o_token = o_token;
    p.o_head = o_head;
    p.status = status;
    p.after = kAfterOffsets;
    for (int j = 0; j < njobs; ++j) {
        const cg_decode_job &jb = jobs_host[j];
        if (!jb.tables || !jb.lengths || !jb.group_off || !jb.scales_k || !jb.scales_v || !jb.out ||
            (!jb.bytes && jb.nbytes > 0) || (jb.table_kind != CG_TABLES_CDF && !jb.table_row_off))
            return CG_E_NULL;
        if ((jb.table_kind != CG_TABLES_CDF && jb.table_kind != CG_TABLES_COUNTS && jb.table_kind != CG_TABLES_SPARSE) ||
            (jb.length_kind != CG_LENGTHS_I32 && jb.length_kind != CG_LENGTHS_U16))
            return CG_E_SHAPE;
        if (jb.table_kind == CG_TABLES_SPARSE) {
            if (jb.tables_nbytes < (static_cast<int64_t>(2 * nlayers) * p.nslab + 1) * 4) return CG_E_CAPACITY;
            if (reinterpret_cast<uintptr_t>(jb.tables) & 3) return CG_E_ALIGN;
        }
        if (jb.table_kind == CG_TABLES_COUNTS && jb.tables_nbytes <= 0) return CG_E_CAPACITY;
        if (jb.ntokens <= 0 || jb.nbytes < 0) return CG_E_SHAPE;
        if (jb.ntokens > CG_MAX_TOKENS_PER_STREAM) return CG_E_TOKENS;
        p.jobs[j] = jb;
    }
    return CG_OK;
}

static int launch_fused_any(const FusedDecodeParams &p, int scale_dtype, int out_dtype, cudaStream_t st, bool early = false) {
    if (p.delta_group > 0) {  // only the two-channels-per-thread kernel knows about anchors
        if (!multi_layout_ok(p, 2)) return CG_E_ALIGN;
        return out_dtype == CG_F16 ? launch_fused_multi<2, CG_F16, true>(p, scale_dtype, early, st)
                                   : launch_fused_multi<2, CG_BF16, true>(p, scale_dtype, early, st);
    }
    if (multi_layout_ok(p, 2) && offsets_fit(p))
        return out_dtype == CG_F16 ? launch_fused_multi<2, CG_F16, false>(p, scale_dtype, early, st)
                                   : launch_fused_multi<2, CG_BF16, false>(p, scale_dtype, early, st);
    if (scale_dtype == CG_F16 && out_dtype == CG_F16) return launch_fused<CG_F16, CG_F16>(p, early, st);
    if (scale_dtype == CG_F16 && out_dtype == CG_BF16) return launch_fused<CG_F16, CG_BF16>(p, early, st);
    if (scale_dtype == CG_BF16 && out_dtype == CG_F16) return launch_fused<CG_BF16, CG_F16>(p, early, st);
    return launch_fused<CG_BF16, CG_BF16>(p, early, st);
}

extern "C" int cg_decode_dequant(const cg_decode_job *jobs_host, int njobs, int nlayers, int nheads,
                                 int head_size, int lp, const float *bins, int scale_dtype,
                                 int out_dtype, int64_t o_layer, int64_t o_kv, int64_t o_token,
                                 int64_t o_head, int32_t *status, void *stream) {
    FusedDecodeParams p;
    if (int rc = fused_params(jobs_host, njobs, nlayers, nheads, head_size, lp, bins, scale_dtype, out_dtype,
                              o_layer, o_kv, o_token, o_head, status, p))
        return rc;
    return launch_fused_any(p, scale_dtype, out_dtype, static_cast<cudaStream_t>(stream));
}

extern "C" int cg_decode_dequant_delta(const cg_decode_job *jobs_host, int njobs, int nlayers, int nheads,
                                       int head_size, int lp, const float *bins, int delta_group,
                                       const float *res_bins, int scale_dtype, int out_dtype, int64_t o_layer,
                                       int64_t o_kv, int64_t o_token, int64_t o_head, int32_t *status, void *stream) {
    FusedDecodeParams p;
    if (int rc = fused_params(jobs_host, njobs, nlayers, nheads, head_size, lp, bins, scale_dtype, out_dtype,
                              o_layer, o_kv, o_token, o_head, status, p))
        return rc;
    if (delta_group) {
        if (!res_bins) return CG_E_NULL;
        if (delta_group < 2 || delta_group > CG_MAX_TOKENS_PER_STREAM || CG_MAX_TOKENS_PER_STREAM % delta_group)
            return CG_E_SHAPE;
        p.delta_group = delta_group;
        p.res_bins = res_bins;
    }
    return launch_fused_any(p, scale_dtype, out_dtype, static_cast<cudaStream_t>(stream));
}

// ---- streams located by their lengths -------------------------------------------------------------------------
static int one_offsets(const int32_t *lengths, int64_t nbytes, int nrows, int nchannels, int64_t *group_off, int32_t *status,
                       cudaStream_t st, const StreamSizes &sizes) {
    if (nrows <= 0 || nchannels <= 0 || nrows > 65535) return CG_E_SHAPE;
    if (static_cast<int64_t>(nrows) * ((nchannels + kGroup - 1) / kGroup) > kMaxOffsetGroups) return CG_E_CAPACITY;
    cg_decode_job job{};
    job.lengths = lengths;
    job.group_off = group_off;
    job.nbytes = nbytes;
    job.length_kind = CG_LENGTHS_I32;
    return launch_offsets(&job, 1, nrows, nchannels, status, st, sizes);
}

extern "C" int cg_stream_sizes(const int32_t *lengths, int nrows, int nchannels, int longest, const int32_t *extra,
                               int64_t *group_off_out, int64_t *tail, void *stream) {
    if (!lengths || !group_off_out || !tail) return CG_E_NULL;
    if (longest < 0) return CG_E_SHAPE;
    tail[3] = 0;
    return one_offsets(lengths, 0, nrows, nchannels, group_off_out, nullptr, static_cast<cudaStream_t>(stream),
                       StreamSizes{tail, extra, longest});
}

extern "C" int cg_decode_packed(const int16_t *cdf, const uint8_t *bytes, int64_t nbytes, const int32_t *lengths,
                                int64_t *group_off, uint8_t *out, const int64_t out_strides[3], int nrows, int ntokens,
                                int nchannels, int lp, int32_t *status, void *stream) {
    if (!cdf || !lengths || !group_off || !out || !out_strides || (!bytes && nbytes > 0)) return CG_E_NULL;
    if (nbytes < 0) return CG_E_SHAPE;
    if (int rc = check_coder_shape(nrows, ntokens, nchannels, lp)) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (int rc = one_offsets(lengths, nbytes, nrows, nchannels, group_off, status, st, StreamSizes{nullptr, nullptr, 1 << 20}))
        return rc;
    SymDecodeParams p{cdf, bytes, nbytes, nullptr, lengths, group_off, 0, out, out_strides[0], out_strides[1],
                      out_strides[2], ntokens, nchannels, lp, status};
    return launch_symbols<2>(p, nrows, st);
}

// ---- offsets and decode of any number of sub-chunks -----------------------------------------------------------
extern "C" int cg_decode_kv(const cg_decode_job *jobs_host, int njobs, int nlayers, int nheads, int head_size, int lp,
                            const float *bins, int delta_group, const float *res_bins, int scale_dtype, int out_dtype,
                            int64_t o_layer, int64_t o_kv, int64_t o_token, int64_t o_head, int32_t *status,
                            void *stream) {
    if (!jobs_host || !bins) return CG_E_NULL;
    if (njobs <= 0) return CG_E_SHAPE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // all arguments are checked before anything is launched
    FusedDecodeParams p;
    const auto fill = [&](int b) {
        const int n = njobs - b < CG_MAX_DECODE_JOBS ? njobs - b : CG_MAX_DECODE_JOBS;
        if (int rc = fused_params(jobs_host + b, n, nlayers, nheads, head_size, lp, bins, scale_dtype, out_dtype, o_layer, o_kv,
                                  o_token, o_head, status, p))
            return rc;
        if (delta_group) {
            if (!res_bins) return CG_E_NULL;
            if (delta_group < 2 || delta_group > CG_MAX_TOKENS_PER_STREAM || CG_MAX_TOKENS_PER_STREAM % delta_group) return CG_E_SHAPE;
            if (!multi_layout_ok(p, 2)) return CG_E_ALIGN;
            p.delta_group = delta_group;
            p.res_bins = res_bins;
        }
        return CG_OK;
    };
    for (int b = 0; b < njobs; b += CG_MAX_DECODE_JOBS)
        if (int rc = fill(b)) return rc;
    const int nrows = 2 * nlayers, nchannels = nheads * head_size, nslab = (nchannels + kGroup - 1) / kGroup;
    const bool fused_offsets = static_cast<int64_t>(nrows) * nslab <= kMaxOffsetGroups;
    for (int b = 0; b < njobs; b += CG_MAX_DECODE_JOBS) {
        const int n = njobs - b < CG_MAX_DECODE_JOBS ? njobs - b : CG_MAX_DECODE_JOBS;
        int rc;
        if (fused_offsets) {
            rc = launch_offsets(jobs_host + b, n, nrows, nchannels, status, st, StreamSizes{nullptr, nullptr, 1 << 20}, b > 0);
        } else {
            rc = CG_OK;
            for (int j = b; j < b + n && rc == CG_OK; ++j)
                rc = cg_decode_offsets(jobs_host + j, 1, nrows, nchannels, const_cast<int64_t *>(jobs_host[j].group_off), status, stream);
        }
        if (rc) return rc;
    }
    for (int b = 0; b < njobs; b += CG_MAX_DECODE_JOBS) {
        if (int rc = fill(b)) return rc;
        // the one-channel kernel waits for the launch in front either way
        p.after = b ? kAfterBatch : kAfterOffsets;
        if (int rc = launch_fused_any(p, scale_dtype, out_dtype, st, true)) return rc;
    }
    return CG_OK;
}

// ---- decode without a caller-provided workspace --------------------------------------------------------------
// Group offsets for callers that cannot allocate (see the header): a fixed array in the library's
// own device image.  In host code `g_static_group_off` is only a handle for the runtime, not a
// device address; the address each device gave the array is looked up once per device below.
static __device__ __align__(256) int64_t g_static_group_off[CG_STATIC_OFFSET_ENTRIES];

#include <mutex>

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_static_mu;
int64_t *g_static_ptr[kMaxDevices];  // device address of g_static_group_off, per device

// Address of the array on the current device; set up on the first call per device.
int static_group_off(int64_t **out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return set_cuda_error(e);
    if (dev < 0 || dev >= kMaxDevices) return CG_E_CAPACITY;
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (!g_static_ptr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_static_group_off);
        if (e != cudaSuccess) return set_cuda_error(e);
        g_static_ptr[dev] = static_cast<int64_t *>(p);
    }
    *out = g_static_ptr[dev];
    return CG_OK;
}
}  // namespace

extern "C" int cg_decode_dequant_static(const cg_decode_job *jobs_host, int njobs, int nlayers, int nheads,
                                        int head_size, int lp, const float *bins, int scale_dtype,
                                        int out_dtype, int64_t o_layer, int64_t o_kv, int64_t o_token,
                                        int64_t o_head, int32_t *status, void *stream) {
    if (!jobs_host || !bins) return CG_E_NULL;
    if (njobs <= 0 || nlayers <= 0 || nheads <= 0 || head_size <= 0) return CG_E_SHAPE;
    if (njobs > CG_MAX_DECODE_JOBS) return CG_E_CAPACITY;
    if (nlayers > 32767 || static_cast<int64_t>(nheads) * head_size > 0x7FFFFFFF - kGroup) return CG_E_SHAPE;
    const int nchannels = nheads * head_size;
    const int64_t ngroups = static_cast<int64_t>(2 * nlayers) * ((nchannels + kGroup - 1) / kGroup);
    if (ngroups * njobs > CG_STATIC_OFFSET_ENTRIES) return CG_E_CAPACITY;
    int64_t *scratch = nullptr;
    if (int rc = static_group_off(&scratch)) return rc;
    cg_decode_job jobs[CG_MAX_DECODE_JOBS];
    for (int j = 0; j < njobs; ++j) {
        jobs[j] = jobs_host[j];
        jobs[j].group_off = scratch + j * ngroups;
    }
    // every argument check of the fused decode comes before the first launch into the shared array
    FusedDecodeParams p;
    if (int rc = fused_params(jobs, njobs, nlayers, nheads, head_size, lp, bins, scale_dtype, out_dtype, o_layer,
                              o_kv, o_token, o_head, status, p))
        return rc;
    if (int rc = cg_decode_offsets(jobs, njobs, 2 * nlayers, nchannels, scratch, status, stream)) return rc;
    return launch_fused_any(p, scale_dtype, out_dtype, static_cast<cudaStream_t>(stream));
}
