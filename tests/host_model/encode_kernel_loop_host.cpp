// Host build of the encoder's step in the form that the kernels run (EncoderState::steps_at with DEEP, at its marks, in
// cachegen_b200/csrc/cg_coder.cuh), for the CPU tests: two streams a lane that share a vote, each with symbols and a table of its own.
#include <cstring>
#include <vector>

#include "../../cachegen_b200/csrc/cg_coder.cuh"

using namespace cg;

// Symbol t of stream i is sym[2 t + i], its table cdf[i * lp ...], its row `cap` bytes from out + i * cap on.  counted: the tables are
// counted from that many symbols and two symbols go to a vote; 0: any tables, one symbol.  again[i]: the loop left something
// and the stream was coded again; deepest: the most bits pending behind a step.  Returns -2 if pairs are not for such tables.
extern "C" int ek_encode(const uint16_t *cdf, int lp, const uint8_t *sym, int n, uint8_t *out, int64_t cap, int counted, int32_t *len,
                         uint8_t *again, int *deepest) {
    if (counted && !pair_high_water(counted)) return -2;
    const uint32_t col[2] = {4u, 400u}, top = static_cast<uint32_t>(lp - 2);
    std::vector<uint32_t> tab(static_cast<size_t>(lp) * kGroupChannels);
    Smem sm{reinterpret_cast<uint8_t *>(tab.data())};
    std::vector<uint32_t> row[2];
    BitSink sink[2];
    EncoderState enc[2];
    bool carried[2] = {};
    const auto entry = [&](int t, int i) { return col[i] + static_cast<uint32_t>(sym[2 * t + i]) * kTableRowBytes; };
    for (int i = 0; i < 2; ++i) {
        for (int m = 0; m < lp - 1; ++m) sm.st(col[i] + static_cast<uint32_t>(m) * kTableRowBytes, static_cast<uint32_t>(cdf[i * lp + m]) << 16);
        row[i].assign(static_cast<size_t>(cap) / 4 + 1, 0u);
        sink[i].init(reinterpret_cast<uint8_t *>(row[i].data()), cap);
        enc[i].init();
        enc[i].half_scale(sink[i]);
    }
    *deepest = 0;
    for (int t = 0; t < n;) {
        const uint32_t words[2] = {sink[0].nwords, sink[1].nwords};
        if (counted && t + 2 <= n) {
            const uint32_t a[2][2] = {{entry(t, 0), entry(t, 1)}, {entry(t + 1, 0), entry(t + 1, 1)}};
            EncoderState::steps_at<kTableRowBytes, 2, 2, false, true>(sm, a, enc, sink, deep_pair_high_water(counted), 0u, carried);
            t += 2;
        } else if (counted) {
            const uint32_t a[1][2] = {{entry(t, 0), entry(t, 1)}};
            EncoderState::steps_at<kTableRowBytes, 1, 2, false, true>(sm, a, enc, sink, kDeepHighWater, 0u, carried);
            ++t;
        } else {  // one stream after the other: whether a symbol is the last of its table is told for all streams of a step
            for (int i = 0; i < 2; ++i) {
                const uint32_t a[1][1] = {{entry(t, i)}};
                EncoderState e[1] = {enc[i]};
                BitSink s[1] = {sink[i]};
                bool c[1] = {carried[i]};
                EncoderState::steps_at<kTableRowBytes, 1, 1, true, true>(sm, a, e, s, kDeepHighWater, 0u, c, sym[2 * t + i] == top);
                enc[i] = e[0];
                sink[i] = s[0];
                carried[i] = c[0];
            }
            ++t;
        }
        for (int i = 0; i < 2; ++i) {
            const int pending = sink[i].nacc + static_cast<int>(sink[i].nwords - words[i]) * 32;
            *deepest = pending > *deepest ? pending : *deepest;
        }
    }
    for (int i = 0; i < 2; ++i) {
        again[i] = enc[i].unsettled(carried[i]);
        if (again[i]) {
            sink[i].init(reinterpret_cast<uint8_t *>(row[i].data()), cap);
            enc[i].init();
            for (int k = 0; k < n; ++k) enc[i].step_alone<kTableRowBytes>(sm, entry(k, i), !counted && sym[2 * k + i] == top, sink[i]);
        }
        len[i] = static_cast<int32_t>(enc[i].flush(sink[i]));
        if (len[i] > cap) return -1;
        memcpy(out + static_cast<size_t>(i) * cap, row[i].data(), static_cast<size_t>(len[i]));
    }
    return 0;
}
extern "C" int ek_deep_pair_high_water(int ntokens) { return pair_high_water(ntokens) ? deep_pair_high_water(ntokens) : 0; }
