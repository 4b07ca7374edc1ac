// Which launches a recurrence over channels takes: the selective scan and the gated recurrent unit (recurrent.cu) have three forms with the same
// results, to the bit, whose times differ by ten in either direction, depending on how the tokens of a step lie. Plain C++: the entry points choose
// with what they are told, the planner of steps, which knows every length, whether short sequences go in a call of their own.
//   chunks   the tile kernel over the plan's chunks, three passes where a sequence has several
//   tile     the tile kernel over whole sequences, many small CTAs: best throughput, slowest along one sequence. The first of two chunks runs from the
//            slot, so up to two chunks a sequence are one after the other in the passes too
//   stream   one CTA per SM and 32 or 64 channels: time by the longest sequence and by rounds of CTAs, however short the others are
// The figures are fits (ns, B200, calls replayed as a graph) over 1024 to 12288 channels and 1 to 4000 tokens, one to 256 sequences. Measured,
// us: scan of 8192 channels, one sequence of 2048: stream 177, chunks 228, tile 433; 10240 channels: stream 351, chunks 285 (two rounds of CTAs); 4096
// channels, 16 sequences of 100: stream 73, tile 55; 8192 channels, 8 of 1000: stream 617, tile 506; 63 single tokens beside 300: stream 76, tile 73, chunks 63,
// single tokens by the tile kernel and then the stream 33. Unit of 4096 channels, the same step: tile 77, chunks 32, apart 22.
#pragma once

#include <algorithm>

namespace ingot_scan {

enum class Kind { none, selective, gated };
enum class Form { chunks, tile, stream };

constexpr int kShort = 64;  // sequences of at most so many tokens never need a stream: four of its tiles do not fill its ring

struct Load {
    long long tokens;  // of all sequences
    int longest, sequences, most_chunks;
};

inline long long groups(int channels, int per_cta) { return (channels + per_cta - 1) / per_cta; }

// Channels of a CTA of the selective stream: 32 where that is at most a CTA per SM.
inline int stream_channels(const Load& w, int channels, int sms) { return groups(channels, 32) * w.sequences <= sms ? 32 : 64; }

// What a token costs with `states` per channel as stored, of what it costs with 16 (8: 0.68 to 0.75 measured, 24: 1.1 to 1.25, 32: 1.37 to 1.58).
inline double by_states(int states) { return 0.45 + 0.55 * states / 16; }

// states: per channel, as stored (selective scans only).
inline double stream_ns(Kind kind, const Load& w, int channels, int states, int sms) {
    const int per_cta = kind == Kind::gated ? 32 : stream_channels(w, channels, sms);
    const double token = kind == Kind::gated ? 25.5 : (per_cta == 32 ? 52.5 : 85.0) * by_states(states), begin = kind == Kind::gated ? 5000 : 3000;
    const double rounds = double((groups(channels, per_cta) * w.sequences + sms - 1) / sms), mean = double(w.tokens) / w.sequences;
    return std::max(w.longest * token + begin, rounds * (mean * token + (kind == Kind::gated ? 4000 : 2500)));
}

inline double tile_ns(Kind kind, const Load& w, int channels, int states) {
    const double values = double(w.tokens) * channels;
    if (kind == Kind::gated) return 270.0 * w.longest + 3.6e-3 * values + 2.0 * w.sequences * groups(channels, 128) + 4000;
    return (170.0 * w.longest + 5.2e-3 * values) * by_states(states) + 4.0 * w.sequences * groups(channels, 64) + 5000;
}

inline double chunks_ns(Kind kind, const Load& w, int channels, int states) {
    const double values = double(w.tokens) * channels;
    if (kind == Kind::gated) return 9.0e-3 * values + 2.7 * (w.sequences - 1) * groups(channels, 128) + 15000;
    return 12.3e-3 * values * by_states(states) + 7.6 * (w.sequences - 1) * groups(channels, 64) + 15000;
}

// The form of a call, and how long it is expected to take.
struct Choice {
    Form form;
    double ns;
};
inline Choice choose(Kind kind, const Load& w, int channels, int states, int sms) {
    // Up to 64 tokens the tile kernel was never slower than chunks (512 to 8192 channels, 1 to 63 sequences; 45 tokens of 4096 channels: scan 10 and 18 us, unit 13 and 18).
    const bool sequential = w.most_chunks <= 2;
    Choice best = {Form::tile, tile_ns(kind, w, channels, states)};
    if (sequential && w.longest <= kShort) return best;
    if (!sequential || (w.most_chunks == 2 && chunks_ns(kind, w, channels, states) < best.ns)) best = {Form::chunks, chunks_ns(kind, w, channels, states)};
    if (w.longest > kShort) {
        const double ns = stream_ns(kind, w, channels, states, sms);
        if (ns < best.ns) best = {Form::stream, ns};
    }
    return best;
}

// Whether the sequences of a step go in two calls, small: those of at most kShort tokens, large: the others; all: both.
inline bool apart(Kind kind, const Load& all, const Load& small, const Load& large, int channels, int states, int sms) {
    if (small.sequences == 0 || large.sequences == 0) return false;
    return choose(kind, small, channels, states, sms).ns + choose(kind, large, channels, states, sms).ns < choose(kind, all, channels, states, sms).ns;
}

}  // namespace ingot_scan
