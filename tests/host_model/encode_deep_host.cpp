// Host build of the encoder's loop as the kernels run it (EncoderState and BitSinkT of cachegen_b200/csrc/cg_coder.cuh with the
// accumulator's upper word kept), for the CPU tests.
#include <cstring>
#include <vector>

#include "../../cachegen_b200/csrc/cg_coder.cuh"

using namespace cg;

// `lanes` streams, symbol t of stream i at sym[t * lanes + i], each with its table of lp entries and a row of `cap` bytes; a word
// leaves every stream that has one as soon as one stream is at the mark, as in a warp.  counted: the tables are counted from that
// many symbols and two symbols go to a vote; 0: any tables, one symbol.  again[i]: the loop left something and the stream
// was coded again; most: the most bits pending in front of a last shift; deepest: behind it.
extern "C" int ed_encode(const uint16_t *cdf, int lp, const uint8_t *sym, int n, int lanes, uint8_t *out, int64_t cap, int counted,
                         int32_t *len, uint8_t *again, int *most, int *deepest) {
    if (counted && !pair_high_water(counted)) return -2;
    const int group = counted ? 2 : 1, mark = counted ? deep_pair_high_water(counted) : kDeepHighWater;
    const uint32_t top = static_cast<uint32_t>(lp - 2);
    std::vector<uint32_t> tab(static_cast<size_t>(lp) * kGroupChannels * lanes);
    std::vector<uint32_t> rows(static_cast<size_t>(lanes) * (cap / 4 + 2));
    using Sink = BitSinkT<1, false>;
    std::vector<Sink> sink(lanes);
    std::vector<EncoderState> enc(lanes);
    std::vector<uint32_t> above(lanes), s(lanes);
    const auto column = [&](int i) { return Smem{reinterpret_cast<uint8_t *>(tab.data() + static_cast<size_t>(i) * lp * kGroupChannels)}; };
    const auto row = [&](int i) { return reinterpret_cast<uint8_t *>(rows.data() + static_cast<size_t>(i) * (cap / 4 + 2) + 1); };
    for (int i = 0; i < lanes; ++i) {
        for (int m = 0; m < lp - 1; ++m) column(i).st(m * kTableRowBytes, static_cast<uint32_t>(cdf[i * lp + m]) << 16);
        sink[i].init(row(i), cap);
        enc[i].init();
        enc[i].half_scale(sink[i]);
        again[i] = 0;
    }
    *most = *deepest = 0;
    int t = 0;
    for (; t + group <= n; t += group) {
        bool full = false;
        for (int i = 0; i < lanes; ++i) {
            for (int g = 0; g < group; ++g) {
                const uint32_t m = sym[(t + g) * lanes + i], a = m * kTableRowBytes;
                const bool last = !counted && m == top;
                s[i] = enc[i].take<false>(cg_umulhi(enc[i].span32, column(i).ld(a)),
                                          last ? enc[i].span32 : cg_umulhi(enc[i].span32, column(i).ld(a + kTableRowBytes)), sink[i], above[i]);
            }
            const int before = sink[i].nacc - static_cast<int>(s[i]);
            *most = before > *most ? before : *most;
            *deepest = sink[i].nacc > *deepest ? sink[i].nacc : *deepest;
            full |= sink[i].nacc >= mark;
        }
        for (int i = 0; full && i < lanes; ++i) again[i] |= sink[i].store_word_if_full<true>(above[i], s[i]);
    }
    for (; t < n; ++t)
        for (int i = 0; i < lanes; ++i) {
            const uint32_t a[1][1] = {{static_cast<uint32_t>(sym[t * lanes + i]) * kTableRowBytes}};
            EncoderState e[1] = {enc[i]};
            Sink o[1] = {sink[i]};
            bool carried[1] = {again[i] != 0};
            EncoderState::steps_at<kTableRowBytes, 1, 1, false, true>(column(i), a, e, o, kDeepHighWater, 0u, carried);
            enc[i] = e[0];
            sink[i] = o[0];
            again[i] = carried[0];
        }
    for (int i = 0; i < lanes; ++i) {
        if (enc[i].unsettled(again[i])) {
            again[i] = 1;
            sink[i].init(row(i), cap);
            enc[i].init();
            for (int k = 0; k < n; ++k) enc[i].step_alone<kTableRowBytes>(column(i), sym[k * lanes + i] * kTableRowBytes, !counted && sym[k * lanes + i] == top, sink[i]);
        }
        len[i] = static_cast<int32_t>(enc[i].flush(sink[i]));
        if (len[i] > cap) return -1;
        memcpy(out + static_cast<size_t>(i) * cap, row(i), len[i]);
    }
    return 0;
}
