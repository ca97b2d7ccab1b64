// Host build of the encoder's loop as a warp runs it (the two parts of EncoderState::steps_at in cachegen_b200/csrc/cg_coder.cuh, with a
// vote over several streams between them), for the CPU tests.
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
    const int group = counted ? 2 : 1, mark = counted ? pair_high_water(counted) : kHighWater;
    const uint32_t top = static_cast<uint32_t>(lp - 2);
    std::vector<uint32_t> tab(static_cast<size_t>(lp) * kGroupChannels * lanes);
    std::vector<uint32_t> rows(static_cast<size_t>(lanes) * (cap / 4 + 2));
    using Sink = BitSinkT<1, false>;
    struct Lane {  // as the parts of steps_at take them
        EncoderState enc[1];
        Sink sink[1];
        uint32_t s[1], above[1];
        bool carried[1] = {};
    };
    std::vector<Lane> lane(lanes);
    const auto column = [&](int i) { return Smem{reinterpret_cast<uint8_t *>(tab.data() + static_cast<size_t>(i) * lp * kGroupChannels)}; };
    const auto row = [&](int i) { return reinterpret_cast<uint8_t *>(rows.data() + static_cast<size_t>(i) * (cap / 4 + 2) + 1); };
    for (int i = 0; i < lanes; ++i) {
        for (int m = 0; m < lp - 1; ++m) column(i).st(m * kTableRowBytes, static_cast<uint32_t>(cdf[i * lp + m]) << 16);
        lane[i].sink[0].init(row(i), cap);
        lane[i].enc[0].init();
        lane[i].enc[0].half_scale(lane[i].sink[0]);
    }
    *most = *deepest = 0;
    for (int t = 0; t < n; t += t + group <= n ? group : 1) {
        bool full = false;
        for (int i = 0; i < lanes; ++i) {
            Lane &l = lane[i];
            const auto at = [&](int g) { return static_cast<uint32_t>(sym[(t + g) * lanes + i]) * kTableRowBytes; };
            if (counted && t + group <= n) {
                const uint32_t a[2][1] = {{at(0)}, {at(1)}};
                full |= EncoderState::take_at<kTableRowBytes, 2, 1, false>(column(i), a, l.enc, l.sink, mark, false, l.s, l.above);
            } else if (counted) {
                const uint32_t a[1][1] = {{at(0)}};
                full |= EncoderState::take_at<kTableRowBytes, 1, 1, false>(column(i), a, l.enc, l.sink, kHighWater, false, l.s, l.above);
            } else {
                const uint32_t a[1][1] = {{at(0)}};
                full |= EncoderState::take_at<kTableRowBytes, 1, 1, true>(column(i), a, l.enc, l.sink, mark, sym[t * lanes + i] == top, l.s, l.above);
            }
            const int after = l.sink[0].nacc, before = after - static_cast<int>(l.s[0]);
            *most = before > *most ? before : *most;
            *deepest = after > *deepest ? after : *deepest;
        }
        for (int i = 0; full && i < lanes; ++i) EncoderState::store_at(lane[i].sink, lane[i].s, lane[i].above, lane[i].carried);
    }
    for (int i = 0; i < lanes; ++i) {
        EncoderState &enc = lane[i].enc[0];
        Sink &sink = lane[i].sink[0];
        again[i] = enc.unsettled(lane[i].carried[0]);
        if (again[i]) {
            sink.init(row(i), cap);
            enc.init();
            for (int k = 0; k < n; ++k) enc.step_alone<kTableRowBytes>(column(i), sym[k * lanes + i] * kTableRowBytes, !counted && sym[k * lanes + i] == top, sink);
        }
        len[i] = static_cast<int32_t>(enc.flush(sink));
        if (len[i] > cap) return -1;
        memcpy(out + static_cast<size_t>(i) * cap, row(i), len[i]);
    }
    return 0;
}
