// In which order the CTAs of a prompt's attention run. Plain C++.
#pragma once

#include <cstddef>

// Side by side: the heads' row tiles of equal place run together, the longest first, so that the longest CTAs of all heads start first. With head after
// head the last heads' long CTAs began when the SMs were about to run dry (4096 tokens, 32 / 8 heads: SMs busy 0.80 of the launch; inside a prompt's step
// 207-241 -> 180-213 us per layer, 2048 tokens with chunks of their own, 8 KV heads: 69 -> 51; B200). With more than two tiles per SM and head each head's own
// tail is short, and one head after the other keeps the keys in use in L2; so it does where the keys and values that the tiles see are more than about
// three times the L2: 32 / 32 heads, 24000 tokens (393 MB) 4.15 ms either way, 40000 (655 MB) 10.9 side by side and 10.3 head after head, 72000 41 and 37;
// 64 / 64 heads, 32768 tokens 17.0 and 15.2. Below: 16384 tokens of 32 / 32 (268 MB) 1.86 and 1.92, 24000 of 16 / 16 (197 MB) 1.92 and 1.97 (B200).
inline bool heads_side_by_side(unsigned tiles, int num_sms, size_t key_bytes) { return tiles <= 2u * unsigned(num_sms) && key_bytes <= size_t(384) << 20; }
