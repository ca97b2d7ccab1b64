// Host build of the encoder's loop step (EncoderState::steps_at in cachegen_b200/csrc/cg_coder.cuh), for the CPU
// tests: two streams a lane, one or two symbols a vote, and the stream coded again by single steps where the loop has
// left something, as the kernels do.
#include <cstring>
#include <vector>

#include "../../cachegen_b200/csrc/cg_coder.cuh"

using namespace cg;

// Both streams hold the same symbols and table; out, of `cap` bytes, receives the first.  pairs: two symbols a vote with
// the high-water mark for tables counted from `counted` tokens (0: one symbol).  Returns the stream's length, -1 if the
// streams differ, -2 if pairs are not for such tables; *again is set if the loop left something, *most to the most
// pending bits.
extern "C" int64_t el_encode(const uint16_t *cdf, int lp, const uint8_t *sym, int n, uint8_t *out, int64_t cap, int counted,
                             int *again, int *most) {
    std::vector<uint32_t> tab(static_cast<size_t>(lp) * kGroupChannels);
    for (int m = 0; m < lp - 1; ++m)
        for (int t = 0; t < kGroupChannels; ++t) tab[m * kGroupChannels + t] = static_cast<uint32_t>(cdf[m]) << 16;
    Smem sm{reinterpret_cast<uint8_t *>(tab.data())};
    const uint32_t col[2] = {4u, 400u}, top = static_cast<uint32_t>(lp - 2);
    const int high_water = counted ? pair_high_water(counted) : kSinkHighWater;
    if (!high_water) return -2;
    using Sink = BitSinkT<1>;
    std::vector<uint32_t> row[2];
    Sink sink[2];
    EncoderState enc[2];
    bool carried[2] = {};
    for (int i = 0; i < 2; ++i) {
        row[i].assign(static_cast<size_t>(cap) / 4 + 1, 0u);
        sink[i].init(reinterpret_cast<uint8_t *>(row[i].data()), cap);
        enc[i].init();
        enc[i].half_scale(sink[i]);
    }
    *most = 0;
    int t = 0;
    for (; counted && t + 2 <= n; t += 2) {
        uint32_t a[2][2];
        for (int g = 0; g < 2; ++g)
            for (int i = 0; i < 2; ++i) a[g][i] = col[i] + sym[t + g] * kTableRowBytes;
        EncoderState::steps_at<kTableRowBytes, 2>(sm, a, enc, sink, high_water, 0u, carried);
        *most = sink[0].nacc > *most ? sink[0].nacc : *most;
    }
    for (; t < n; ++t) {
        const uint32_t a[1][2] = {{col[0] + sym[t] * kTableRowBytes, col[1] + sym[t] * kTableRowBytes}};
        if (counted) EncoderState::steps_at<kTableRowBytes, 1>(sm, a, enc, sink, kSinkHighWater, 0u, carried);
        else EncoderState::steps_at<kTableRowBytes, 1, 2, true>(sm, a, enc, sink, kSinkHighWater, 0u, carried, sym[t] == top);
        *most = sink[0].nacc > *most ? sink[0].nacc : *most;
    }
    int64_t len[2];
    for (int i = 0; i < 2; ++i) {
        if (enc[i].unsettled(carried[i])) {
            *again = 1;
            sink[i].init(reinterpret_cast<uint8_t *>(row[i].data()), cap);
            enc[i].init();
            for (int k = 0; k < n; ++k) enc[i].step_alone<kTableRowBytes>(sm, col[i] + sym[k] * kTableRowBytes, sym[k] == top, sink[i]);
        }
        len[i] = enc[i].flush(sink[i]);
    }
    if (len[0] != len[1] || memcmp(row[0].data(), row[1].data(), static_cast<size_t>(len[0] < cap ? len[0] : cap))) return -1;
    memcpy(out, row[0].data(), static_cast<size_t>(len[0] < cap ? len[0] : cap));
    return len[0];
}
extern "C" int el_pair_high_water(int ntokens) { return pair_high_water(ntokens); }
