/*
 * CPU restatement of the CacheGen KV-cache codec hot path.
 *
 * TEST INFRASTRUCTURE ONLY: this file is the oracle the CUDA product is
 * compared against (and the host-CPU baseline that is timed beside it).  No
 * product code path may call into it.
 *
 * Parity status: the reference ships no golden vectors for this path
 * (LMCache/tests/test_serde.py checks shapes and lengths only).  The oracle is
 * therefore pinned two other ways: (1) quantise / dequantise against fixtures
 * generated by importing the reference's own Python functions on CPU
 * (tests/golden/make_golden_cpu.py); (2) CDF tables, streams and symbols
 * against the reference's own CUDA extension, built unmodified by
 * oracle/build_ref.py and run on a GPU (tests/golden/make_golden_gpu.py writes
 * the fixtures; tests/test_gpu_ref_ext.py and tests/test_gpu_workload_parity.py compare live
 * when the build exists).
 *
 * Every function cites the reference lines it follows; paths are relative to
 * the reference checkout:
 *   enc.py     = LMCache/lmcache/storage_backend/serde/cachegen_encoder.py
 *   dec.py     = LMCache/lmcache/storage_backend/serde/cachegen_decoder.py
 *   cal_cdf.cu / enc_new.cu / dec_new.cu
 *              = LMCache/third_party/torchac_cuda/{cal_cdf,torchac_kernel_enc_new,
 *                torchac_kernel_dec_new}.cu
 * The arithmetic coder is kept bit-serial with the 64-bit division and the
 * binary search, exactly as the reference kernels (and the torchac CPU coder
 * they derive from) are written.
 */
#include <math.h>
#include <pthread.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

/* ---------------------------------------------------------------- 16-bit floats */

static float f16_to_f32(uint16_t h)
{
    uint32_t sign = (uint32_t)(h & 0x8000u) << 16;
    uint32_t exp = (h >> 10) & 0x1Fu;
    uint32_t man = h & 0x3FFu;
    uint32_t bits;
    if (exp == 0) {
        if (man == 0) {
            bits = sign;
        } else { /* subnormal: renormalise */
            int e = -1;
            do { e++; man <<= 1; } while (!(man & 0x400u));
            bits = sign | ((uint32_t)(127 - 15 - e) << 23) | ((man & 0x3FFu) << 13);
        }
    } else if (exp == 31) {
        bits = sign | 0x7F800000u | (man << 13);
    } else {
        bits = sign | ((exp + 112u) << 23) | (man << 13);
    }
    float f;
    memcpy(&f, &bits, 4);
    return f;
}

/* round-to-nearest-even fp32 -> fp16, as torch's .to(torch.float16) */
static uint16_t f32_to_f16(float f)
{
    uint32_t x;
    memcpy(&x, &f, 4);
    uint32_t sign = (x >> 16) & 0x8000u;
    uint32_t ax = x & 0x7FFFFFFFu;
    if (ax >= 0x7F800000u) /* inf / nan */
        return (uint16_t)(sign | 0x7C00u | ((ax > 0x7F800000u) ? 0x200u : 0u));
    if (ax >= 0x477FF000u) /* rounds to >= 65520 -> inf */
        return (uint16_t)(sign | 0x7C00u);
    if (ax < 0x38800000u) { /* result is subnormal or zero (|f| < 2^-14) */
        if (ax < 0x33000000u) /* < 2^-25 -> 0 */
            return (uint16_t)sign;
        uint32_t e = ax >> 23;
        uint32_t m = (ax & 0x7FFFFFu) | 0x800000u;
        uint32_t shift = 126u - e; /* m / 2^shift = value / 2^-24, shift in 14..24 */
        uint32_t q = m >> shift;
        uint32_t rem = m & ((1u << shift) - 1u);
        uint32_t half = 1u << (shift - 1u);
        if (rem > half || (rem == half && (q & 1u)))
            q++;
        return (uint16_t)(sign | q);
    }
    uint32_t e = (ax >> 23) - 112u;
    uint32_t m = ax & 0x7FFFFFu;
    uint32_t h = (e << 10) | (m >> 13);
    uint32_t rem = m & 0x1FFFu;
    if (rem > 0x1000u || (rem == 0x1000u && (h & 1u)))
        h++; /* a carry into the exponent is the correct result */
    return (uint16_t)(sign | h);
}

static float bf16_to_f32(uint16_t h)
{
    uint32_t bits = (uint32_t)h << 16;
    float f;
    memcpy(&f, &bits, 4);
    return f;
}

static uint16_t f32_to_bf16(float f)
{
    uint32_t x;
    memcpy(&x, &f, 4);
    if ((x & 0x7FFFFFFFu) > 0x7F800000u)
        return (uint16_t)((x >> 16) | 0x40u);
    uint32_t lsb = (x >> 16) & 1u;
    x += 0x7FFFu + lsb;
    return (uint16_t)(x >> 16);
}

/* dtype codes shared with the product's C ABI: 0 = fp16, 1 = bf16 */
static float h_to_f32(uint16_t h, int dtype) { return dtype ? bf16_to_f32(h) : f16_to_f32(h); }
static uint16_t f32_to_h(float f, int dtype) { return dtype ? f32_to_bf16(f) : f32_to_f16(f); }

void cgo_f16_to_f32(const uint16_t *in, float *out, int64_t n, int dtype)
{
    for (int64_t i = 0; i < n; i++) out[i] = h_to_f32(in[i], dtype);
}

void cgo_f32_to_f16(const float *in, uint16_t *out, int64_t n, int dtype)
{
    for (int64_t i = 0; i < n; i++) out[i] = f32_to_h(in[i], dtype);
}

/* ---------------------------------------------------------------- quantise */

/*
 * torch_quant_vectorized, enc.py:42-59.  x is [rows, T, C] in fp16/bf16 bits,
 * bins[rows] are the per-row bin counts as float32 (make_key_bins, enc.py:311-322).
 *   MAX    = bins // 2 - 1                       (fp32)
 *   max1   = amax(|x|, -1)                       (input dtype: exact)
 *   factor = MAX / max1                          (fp32 division)
 *   xq     = round(x * factor + MAX).to(int8)    (fp32 mul, fp32 add, half-to-even)
 * Each fp32 operation is rounded separately (no fused multiply-add): build with
 * -ffp-contract=off.  A NaN (all-zero token row: 0 * inf) converts to 0.
 */
void cgo_quantize(const uint16_t *x, int dtype, int rows, int T, int C, const float *bins,
                  int8_t *sym, uint16_t *maxes)
{
    for (int r = 0; r < rows; r++) {
        volatile float MAXv = floorf(bins[r] / 2.0f) - 1.0f;
        const float MAX = MAXv;
        for (int t = 0; t < T; t++) {
            const uint16_t *row = x + ((int64_t)r * T + t) * C;
            int8_t *out = sym + ((int64_t)r * T + t) * C;
            uint16_t best = 0; /* |x| bit patterns order like magnitudes */
            for (int c = 0; c < C; c++) {
                uint16_t a = row[c] & 0x7FFFu;
                if (a > best) best = a;
            }
            maxes[(int64_t)r * T + t] = best;
            volatile float factor = MAX / h_to_f32(best, dtype);
            for (int c = 0; c < C; c++) {
                volatile float p = h_to_f32(row[c], dtype) * factor;
                volatile float q = p + MAX;
                float rr = nearbyintf(q);
                out[c] = (rr != rr) ? 0 : (int8_t)(int32_t)rr;
            }
        }
    }
}

/* ---------------------------------------------------------------- dequantise */

/*
 * do_dequantize + final cast, dec.py:24-34,110,169-173:
 *   t = float(sym); t = t - Cq; t = t / Cq; t = t * float(max); out = cast(t)
 * with Cq = bins // 2 - 1 (fp32).  sym is [rows, T, C] uint8 with element strides
 * (ss0, ss1, ss2); out is written at out[r*os0 + t*os1 + c*os2] so the caller picks
 * the KV layout (stack / reshape / permute of dec.py:165-173).
 */
void cgo_dequantize(const uint8_t *sym, int64_t ss0, int64_t ss1, int64_t ss2, int rows, int T,
                    int C, const float *bins, const uint16_t *maxes, int max_dtype,
                    uint16_t *out, int64_t os0, int64_t os1, int64_t os2, int out_dtype)
{
    for (int r = 0; r < rows; r++) {
        const float Cq = floorf(bins[r] / 2.0f) - 1.0f;
        for (int t = 0; t < T; t++) {
            const float mx = h_to_f32(maxes[(int64_t)r * T + t], max_dtype);
            for (int c = 0; c < C; c++) {
                volatile float v = (float)sym[r * ss0 + t * ss1 + c * ss2];
                v = v - Cq;
                v = v / Cq;
                v = v * mx;
                out[r * os0 + t * os1 + c * os2] = f32_to_h(v, out_dtype);
            }
        }
    }
}

/* ---------------------------------------------------------------- anchor-token delta */

/*
 * Anchor-token delta coding on top of the reference's quantiser.  The reference snapshot has no such
 * step (its serializer quantises every token on its own, enc.py:42-59), so nothing here is compared
 * with the reference: this function IS the definition the CUDA path is tested against.
 *
 * Rows with res_bins[r] > 0 are delta-coded in groups of `group` tokens (group divides 256): a
 * token t with t % group == 0 is an anchor and is quantised exactly as cgo_quantize does; any other
 * token is replaced by its difference from the DEQUANTISED anchor of its group (what a decoder
 * holds: ((sym - Cq)/Cq) * max in fp32, cast to the KV dtype), the difference itself rounded to
 * the KV dtype, and that residual row goes through the same quantiser with res_bins[r] bins:
 *   x^a   = cast(((sym_a - Cq_a) / Cq_a) * max_a)                    Cq_a = bins // 2 - 1
 *   r     = cast(float(x_t) - float(x^a))
 *   max_t = amax(|r|);  s = round(float(r) * (Cq_r / max_t) + Cq_r)   Cq_r = res_bins // 2 - 1
 *   sym_t = s + (Cq_a - Cq_r)        (both kinds of token centre on Cq_a and share one table)
 * maxes[r, t] is the anchor's or the residual's max accordingly.  Rows with res_bins[r] <= 0 are
 * quantised as cgo_quantize does.  Returns -1 when a delta row has Cq_r < 1 or Cq_r > Cq_a.
 */
int cgo_quantize_delta(const uint16_t *x, int dtype, int rows, int T, int C, const float *bins,
                       const float *res_bins, int group, int8_t *sym, uint16_t *maxes)
{
    if (group < 1) return -1;
    float *anchor = (float *)malloc(sizeof(float) * (size_t)C);
    uint16_t *res = (uint16_t *)malloc(sizeof(uint16_t) * (size_t)C);
    if (!anchor || !res) { free(anchor); free(res); return -2; }
    int rc = 0;
    for (int r = 0; r < rows && rc == 0; r++) {
        volatile float cqa_v = floorf(bins[r] / 2.0f) - 1.0f;
        const float CQA = cqa_v;
        const int delta = res_bins && res_bins[r] > 0.0f;
        volatile float cqr_v = delta ? floorf(res_bins[r] / 2.0f) - 1.0f : CQA;
        const float CQR = cqr_v;
        if (delta && (CQR < 1.0f || CQR > CQA)) { rc = -1; break; }
        const int shift = (int)(CQA - CQR);
        for (int t = 0; t < T; t++) {
            const uint16_t *row = x + ((int64_t)r * T + t) * C;
            int8_t *out = sym + ((int64_t)r * T + t) * C;
            const int is_anchor = !delta || (t % group) == 0;
            const uint16_t *src = row;
            if (!is_anchor) {
                for (int c = 0; c < C; c++) {
                    volatile float d = h_to_f32(row[c], dtype) - anchor[c];
                    res[c] = f32_to_h(d, dtype);
                }
                src = res;
            }
            uint16_t best = 0;
            for (int c = 0; c < C; c++) {
                uint16_t a = src[c] & 0x7FFFu;
                if (a > best) best = a;
            }
            maxes[(int64_t)r * T + t] = best;
            const float MAXQ = is_anchor ? CQA : CQR;
            volatile float factor = MAXQ / h_to_f32(best, dtype);
            for (int c = 0; c < C; c++) {
                volatile float p = h_to_f32(src[c], dtype) * factor;
                volatile float q = p + MAXQ;
                float rr = nearbyintf(q);
                const int s = (rr != rr) ? 0 : (int)(int8_t)(int32_t)rr;
                out[c] = (int8_t)(is_anchor ? s : s + shift);
                if (is_anchor && delta) { /* what the decoder will hold for this anchor */
                    volatile float v = (float)(uint8_t)out[c];
                    v = v - CQA;
                    v = v / CQA;
                    v = v * h_to_f32(best, dtype);
                    anchor[c] = h_to_f32(f32_to_h(v, dtype), dtype);
                }
            }
        }
    }
    free(anchor);
    free(res);
    return rc;
}

/*
 * The decoder's side of cgo_quantize_delta: anchors as cgo_dequantize; a residual token adds
 * ((sym - Cq_a) / Cq_r) * max_t to the anchor's value as the KV dtype holds it (max_dtype is the KV
 * dtype), in fp32, and the sum is cast to the output type.  sym [rows, T, C] contiguous.
 */
void cgo_dequantize_delta(const uint8_t *sym, int rows, int T, int C, const float *bins, const float *res_bins,
                          int group, const uint16_t *maxes, int max_dtype, uint16_t *out, int64_t os0,
                          int64_t os1, int64_t os2, int out_dtype)
{
    float *anchor = (float *)malloc(sizeof(float) * (size_t)C);
    for (int r = 0; r < rows; r++) {
        const float CQA = floorf(bins[r] / 2.0f) - 1.0f;
        const int delta = res_bins && res_bins[r] > 0.0f;
        const float CQR = delta ? floorf(res_bins[r] / 2.0f) - 1.0f : CQA;
        for (int t = 0; t < T; t++) {
            const int is_anchor = !delta || (t % group) == 0;
            const float mx = h_to_f32(maxes[(int64_t)r * T + t], max_dtype);
            for (int c = 0; c < C; c++) {
                volatile float v = (float)sym[((int64_t)r * T + t) * C + c];
                v = v - CQA;
                v = v / (is_anchor ? CQA : CQR);
                v = v * mx;
                if (is_anchor) {
                    if (delta) anchor[c] = h_to_f32(f32_to_h(v, max_dtype), max_dtype);
                } else {
                    v = anchor[c] + v;
                }
                out[r * os0 + t * os1 + c * os2] = f32_to_h(v, out_dtype);
            }
        }
    }
    free(anchor);
}

/* ---------------------------------------------------------------- CDF build */

/*
 * calculate_cdf_kernel + normalize_cdf_value, cal_cdf.cu:11-15,29-49.  One table
 * per (row, channel) over the T tokens of the call:
 *   hist[v+1]++ for every symbol v (uint16 counters, they wrap like the kernel's)
 *   hist[i+1] = #{sym <= i} by a running uint16 sum, total = that sum
 *   cdf[i] = (uint16)((0xFFFF - max_bins) * hist[i] / total) + i,  i = 0..max_bins
 * sym has element strides (s0, s1, s2); cdf is [rows, C, max_bins+1] int16.
 */
int cgo_calculate_cdf(const int8_t *sym, int64_t s0, int64_t s1, int64_t s2, int rows, int T,
                      int C, int max_bins, int16_t *cdf)
{
    if (max_bins >= 64 || max_bins < 1) return -1;
    const int Lp = max_bins + 1;
    for (int r = 0; r < rows; r++) {
        for (int c = 0; c < C; c++) {
            uint16_t hist[64];
            memset(hist, 0, sizeof(hist));
            for (int t = 0; t < T; t++) {
                uint8_t v = (uint8_t)sym[r * s0 + t * s1 + c * s2];
                if (v + 1 < 64) hist[v + 1]++;
            }
            uint16_t local_sum = 0;
            for (int i = 0; i < max_bins; i++) {
                uint16_t v = hist[i + 1];
                hist[i + 1] = (uint16_t)(hist[i + 1] + local_sum);
                local_sum = (uint16_t)(local_sum + v);
            }
            if (local_sum == 0) return -2; /* T == 0 or a multiple of 65536: division by zero */
            const uint32_t scale = 0xFFFFu - (uint32_t)max_bins;
            int16_t *o = cdf + ((int64_t)r * C + c) * Lp;
            for (int i = 0; i <= max_bins; i++) {
                uint16_t nv = (uint16_t)(scale * (uint32_t)hist[i] / local_sum);
                o[i] = (int16_t)(uint16_t)(nv + i);
            }
        }
    }
    return 0;
}

/* ---------------------------------------------------------------- bit I/O */

/* MSB-first bit writer with zero-fill flush: add_bits_to_output / spill_*,
 * enc_new.cu:21-97 (same byte order as torchac's OutCacheString). */
typedef struct {
    uint8_t *buf;
    int64_t cap;
    int64_t len;
    uint32_t acc;
    int nacc;
    int overflow;
} bitw_t;

static void bw_put(bitw_t *w, uint32_t bit)
{
    w->acc = (w->acc << 1) | (bit & 1u);
    if (++w->nacc == 8) {
        if (w->len < w->cap) w->buf[w->len] = (uint8_t)w->acc; else w->overflow = 1;
        w->len++;
        w->acc = 0;
        w->nacc = 0;
    }
}

static void bw_put_with_pending(bitw_t *w, uint32_t bit, uint64_t *pending)
{
    bw_put(w, bit);
    while (*pending) { bw_put(w, 1u - bit); (*pending)--; }
}

static void bw_flush(bitw_t *w)
{
    while (w->nacc) bw_put(w, 0);
}

/* ---------------------------------------------------------------- encoder */

/*
 * One stream = the symbols of one (row, channel) over the <=256 tokens of a
 * sub-chunk: the per-thread body of encode_with_accessor_kernel,
 * enc_new.cu:255-306.  cdf points at Lp uint16 entries; sym is read with an
 * element stride.  Returns the stream's length in bytes (which may exceed cap:
 * then *overflow is set and only cap bytes were stored).
 */
int64_t cgo_encode_stream(const uint16_t *cdf, int Lp, const int8_t *sym, int64_t sym_stride,
                          int n, uint8_t *out, int64_t cap, int *overflow)
{
    bitw_t w = {out, cap, 0, 0, 0, 0};
    uint32_t low = 0, high = 0xFFFFFFFFu;
    uint64_t pending = 0;
    const int max_symbol = Lp - 2;
    for (int i = 0; i < n; i++) {
        const uint8_t s = (uint8_t)sym[i * sym_stride];
        const uint64_t span = (uint64_t)high - (uint64_t)low + 1;
        const uint32_t c_low = cdf[s];
        const uint32_t c_high = (s == max_symbol) ? 0x10000u : cdf[s + 1];
        high = (low - 1u) + (uint32_t)((span * (uint64_t)c_high) >> 16);
        low = low + (uint32_t)((span * (uint64_t)c_low) >> 16);
        for (;;) {
            if (high < 0x80000000u) {
                bw_put_with_pending(&w, 0, &pending);
                low <<= 1; high <<= 1; high |= 1u;
            } else if (low >= 0x80000000u) {
                bw_put_with_pending(&w, 1, &pending);
                low <<= 1; high <<= 1; high |= 1u;
            } else if (low >= 0x40000000u && high < 0xC0000000u) {
                pending++;
                low <<= 1; low &= 0x7FFFFFFFu;
                high <<= 1; high |= 0x80000001u;
            } else {
                break;
            }
        }
    }
    pending += 1;
    bw_put_with_pending(&w, (low < 0x40000000u) ? 0u : 1u, &pending);
    bw_flush(&w);
    if (overflow) *overflow = w.overflow;
    return w.len;
}

/* ---------------------------------------------------------------- decoder */

/* binsearch, dec_new.cu:52-71: largest m in [0, max_sym] with cdf[m] <= target
 * for a strictly increasing table (returns on equality, else narrows). */
static uint16_t oracle_binsearch(const uint16_t *cdf, uint16_t target, uint8_t max_sym)
{
    uint16_t left = 0, right = (uint16_t)(max_sym + 1);
    while (left + 1 < right) {
        const uint16_t m = (uint16_t)((left + right) / 2);
        const uint16_t v = cdf[m];
        if (v < target) left = m;
        else if (v > target) right = m;
        else return m;
    }
    return left;
}

/*
 * The per-thread body of decode_prefix_with_accessor_kernel, dec_new.cu:236-302.
 * The stream is `len` bytes at `bytes`; every read past its end yields 0 (the
 * kernel zero-pads its 256-byte staging row, dec_new.cu:229-232).  The kernel's
 * bit cursor starts at byte 4 with bit_idx = 1 and reloads the byte only after a
 * bit is consumed (check_and_update_byte_buffer, dec_new.cu:43-50); a plain
 * "bit position" cursor reads the same bits.  No range update after the last
 * symbol (dec_new.cu:273-275).
 */
void cgo_decode_stream(const uint16_t *cdf, int Lp, const uint8_t *bytes, int64_t len, int n,
                       uint8_t *sym_out, int64_t out_stride)
{
    uint32_t low = 0, high = 0xFFFFFFFFu, value = 0;
    const int max_symbol = Lp - 2;
    for (int i = 0; i < 4; i++) value = (value << 8) | (uint32_t)(i < len ? bytes[i] : 0);
    int64_t bitpos = 32;
    for (int i = 0; i < n; i++) {
        const uint64_t span = (uint64_t)high - (uint64_t)low + 1;
        const uint16_t count =
            (uint16_t)((((uint64_t)value - (uint64_t)low + 1) * 0x10000ull - 1) / span);
        const uint16_t s = oracle_binsearch(cdf, count, (uint8_t)max_symbol);
        sym_out[i * out_stride] = (uint8_t)s;
        if (i == n - 1) break;
        const uint32_t c_low = cdf[s];
        const uint32_t c_high = (s == max_symbol) ? 0x10000u : cdf[s + 1];
        high = (low - 1u) + (uint32_t)((span * (uint64_t)c_high) >> 16);
        low = low + (uint32_t)((span * (uint64_t)c_low) >> 16);
        for (;;) {
            if (low >= 0x80000000u || high < 0x80000000u) {
                low <<= 1; high <<= 1; high |= 1u;
            } else if (low >= 0x40000000u && high < 0xC0000000u) {
                low <<= 1; low &= 0x7FFFFFFFu;
                high <<= 1; high |= 0x80000001u;
                value -= 0x40000000u;
            } else {
                break;
            }
            const int64_t byte = bitpos >> 3;
            const uint32_t b = (byte < len) ? ((bytes[byte] >> (7 - (bitpos & 7))) & 1u) : 0u;
            value = (value << 1) | b;
            bitpos++;
        }
    }
}

/* ---------------------------------------------------------------- threaded drivers */

typedef struct {
    void (*fn)(void *, int64_t, int64_t);
    void *arg;
    int64_t n, grain;
    int64_t next;
    pthread_mutex_t mu;
} pool_t;

static void *pool_worker(void *p_)
{
    pool_t *p = (pool_t *)p_;
    for (;;) {
        pthread_mutex_lock(&p->mu);
        int64_t b = p->next;
        p->next += p->grain;
        pthread_mutex_unlock(&p->mu);
        if (b >= p->n) break;
        int64_t e = b + p->grain < p->n ? b + p->grain : p->n;
        p->fn(p->arg, b, e);
    }
    return NULL;
}

static void parallel_for(int64_t n, int64_t grain, int threads, void (*fn)(void *, int64_t, int64_t),
                         void *arg)
{
    pool_t p = {fn, arg, n, grain > 0 ? grain : 1, 0, PTHREAD_MUTEX_INITIALIZER};
    if (threads <= 1) { fn(arg, 0, n); return; }
    pthread_t *th = (pthread_t *)malloc(sizeof(pthread_t) * (size_t)threads);
    int started = 0;
    for (int i = 0; i < threads - 1; i++)
        if (pthread_create(&th[started], NULL, pool_worker, &p) == 0) started++;
    pool_worker(&p);
    for (int i = 0; i < started; i++) pthread_join(th[i], NULL);
    free(th);
}

/*
 * encode_fast_new + collect_bytes for one sub-chunk (enc.py:210-242): every
 * (row, channel) stream of sym[:, :, :] (strides in elements) is coded with its
 * CDF row; lengths[row, channel] receives the byte count and `bytes` the streams
 * concatenated in (row-major, channel-minor) order.  The caller provides
 * `scratch` of rows*C*cap bytes; streams longer than cap are reported by a
 * non-zero return (the reference kernel silently overruns its 256-byte row,
 * enc_new.cu:11,236).  Returns total bytes, or -1 on overflow.
 */
typedef struct {
    const int16_t *cdf; int Lp;
    const int8_t *sym; int64_t s0, s1, s2;
    int rows, T, C;
    uint8_t *scratch; int64_t cap;
    int32_t *lengths;
    int overflow;
} enc_job_t;

static void enc_range(void *a_, int64_t b, int64_t e)
{
    enc_job_t *a = (enc_job_t *)a_;
    for (int64_t g = b; g < e; g++) {
        const int r = (int)(g / a->C), c = (int)(g % a->C);
        int ov = 0;
        int64_t len = cgo_encode_stream((const uint16_t *)a->cdf + g * a->Lp, a->Lp,
                                        a->sym + r * a->s0 + c * a->s2, a->s1, a->T,
                                        a->scratch + g * a->cap, a->cap, &ov);
        a->lengths[g] = (int32_t)len;
        if (ov) a->overflow = 1;
    }
}

int64_t cgo_encode_chunk(const int16_t *cdf, int Lp, const int8_t *sym, int64_t s0, int64_t s1,
                         int64_t s2, int rows, int T, int C, uint8_t *scratch, int64_t cap,
                         int32_t *lengths, uint8_t *bytes, int64_t bytes_cap, int threads)
{
    enc_job_t job = {cdf, Lp, sym, s0, s1, s2, rows, T, C, scratch, cap, lengths, 0};
    parallel_for((int64_t)rows * C, 256, threads, enc_range, &job);
    if (job.overflow) return -1;
    int64_t total = 0;
    for (int64_t g = 0; g < (int64_t)rows * C; g++) {
        if (total + lengths[g] > bytes_cap) return -1;
        memcpy(bytes + total, scratch + g * cap, (size_t)lengths[g]);
        total += lengths[g];
    }
    return total;
}

/*
 * decode_chunk (dec.py:53-75) + decode_prefix_with_accessor_kernel for one
 * sub-chunk: stream g of the flat byte array spans [prefsum[g-1], prefsum[g])
 * with an inclusive int64 prefix sum of the lengths (dec.py:70, dec_new.cu:215-218).
 * Symbols go to out[row, token, channel] with element strides (o0, o1, o2).
 */
typedef struct {
    const int16_t *cdf; int Lp;
    const uint8_t *bytes; const int64_t *prefsum;
    int rows, T, C;
    uint8_t *out; int64_t o0, o1, o2;
} dec_job_t;

static void dec_range(void *a_, int64_t b, int64_t e)
{
    dec_job_t *a = (dec_job_t *)a_;
    for (int64_t g = b; g < e; g++) {
        const int r = (int)(g / a->C), c = (int)(g % a->C);
        const int64_t start = g ? a->prefsum[g - 1] : 0;
        cgo_decode_stream((const uint16_t *)a->cdf + g * a->Lp, a->Lp, a->bytes + start,
                          a->prefsum[g] - start, a->T, a->out + r * a->o0 + c * a->o2, a->o1);
    }
}

void cgo_decode_chunk(const int16_t *cdf, int Lp, const uint8_t *bytes, const int64_t *prefsum,
                      int rows, int T, int C, uint8_t *out, int64_t o0, int64_t o1, int64_t o2,
                      int threads)
{
    dec_job_t job = {cdf, Lp, bytes, prefsum, rows, T, C, out, o0, o1, o2};
    parallel_for((int64_t)rows * C, 256, threads, dec_range, &job);
}

/*
 * The whole decode path of CacheGenDeserializer.from_bytes for one sub-chunk,
 * used as the timed host-CPU baseline: decode_chunk, then do_dequantize and the
 * stack / permute / cast of dec.py:159-173, writing 16-bit KV at
 * out[row*os0 + token*os1 + channel*os2].  Work is split in blocks of 64
 * adjacent channels so each task decodes into a private [T, 64] tile and then
 * writes 128-byte runs of the output.
 */
typedef struct {
    const int16_t *cdf; int Lp;
    const uint8_t *bytes; const int64_t *prefsum;
    int rows, T, C;
    const float *bins; const uint16_t *maxes; int max_dtype;
    uint16_t *out; int64_t os0, os1, os2; int out_dtype;
} decdq_job_t;

#define CGO_TILE_C 64

static void decdq_range(void *a_, int64_t b, int64_t e)
{
    decdq_job_t *a = (decdq_job_t *)a_;
    const int blocks_per_row = (a->C + CGO_TILE_C - 1) / CGO_TILE_C;
    uint8_t *tile = (uint8_t *)malloc((size_t)a->T * CGO_TILE_C);
    for (int64_t blk = b; blk < e; blk++) {
        const int r = (int)(blk / blocks_per_row);
        const int c0 = (int)(blk % blocks_per_row) * CGO_TILE_C;
        const int nc = (a->C - c0 < CGO_TILE_C) ? a->C - c0 : CGO_TILE_C;
        for (int j = 0; j < nc; j++) {
            const int64_t g = (int64_t)r * a->C + c0 + j;
            const int64_t start = g ? a->prefsum[g - 1] : 0;
            cgo_decode_stream((const uint16_t *)a->cdf + g * a->Lp, a->Lp, a->bytes + start,
                              a->prefsum[g] - start, a->T, tile + j, CGO_TILE_C);
        }
        const float Cq = floorf(a->bins[r] / 2.0f) - 1.0f;
        for (int t = 0; t < a->T; t++) {
            const float mx = h_to_f32(a->maxes[(int64_t)r * a->T + t], a->max_dtype);
            uint16_t *o = a->out + r * a->os0 + t * a->os1 + (int64_t)c0 * a->os2;
            for (int j = 0; j < nc; j++) {
                volatile float v = (float)tile[t * CGO_TILE_C + j];
                v = v - Cq;
                v = v / Cq;
                v = v * mx;
                o[j * a->os2] = f32_to_h(v, a->out_dtype);
            }
        }
    }
    free(tile);
}

void cgo_decode_dequant_chunk(const int16_t *cdf, int Lp, const uint8_t *bytes,
                              const int64_t *prefsum, int rows, int T, int C, const float *bins,
                              const uint16_t *maxes, int max_dtype, uint16_t *out, int64_t os0,
                              int64_t os1, int64_t os2, int out_dtype, int threads)
{
    decdq_job_t job = {cdf, Lp, bytes, prefsum, rows, T, C, bins, maxes, max_dtype,
                       out, os0, os1, os2, out_dtype};
    const int blocks_per_row = (C + CGO_TILE_C - 1) / CGO_TILE_C;
    parallel_for((int64_t)rows * blocks_per_row, 4, threads, decdq_range, &job);
}
