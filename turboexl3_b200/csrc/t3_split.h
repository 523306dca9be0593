// The cut of K of a dense linear at decode rows (host code; see t3_api.cu's plan_dense).
#pragma once

#include <stdint.h>

namespace t3 {

// The most clusters of `size` CTAs that `sms` multiprocessors hold at once with a multiprocessor a CTA:
// cudaOccupancyMaxActiveClusters's for 148 (other devices take their share), written down because plans must be the same without a device.
inline uint32_t clusters_alone(uint32_t sms, uint32_t size) {
    static const uint16_t kOne[17] = {0, 148, 74, 45, 33, 26, 22, 15, 15, 15, 11, 7, 7, 7, 7, 7, 7};
    return kOne[size] * sms / 148u;
}

// K slices of an ordinary dense linear of nb 128-input and `blocks` 128-output blocks, a cluster of s CTAs a block, and whether its CTAs go
// one to a multiprocessor (`alone`): one count a shape and rate, so that a row's bytes are the same alone and in a batch. Only counts whose
// CTAs hold the prepared rows of 32 rows are asked, and the cheapest by its longest slice's time is taken, three times a row's and once that of
// 32 rows. One row: 0.58 us a 128-input block in a CTA that has its multiprocessor to itself, 1.16 in one of two (whatever the rate), and 3 a
// round; 32 rows: 0.8, 2.6 and 6.4, and two fifths more where the ring has one stage. Placement: alone where all clusters fit one CTA to a
// multiprocessor (16 blocks a slice, alone / as they come: 12.8 / 20.3 us, up to the last cluster that fits); else in rounds of as many as fit
// two to a multiprocessor, a last round that fits singly at the single rate; at 32 rows two fit only where their shared memory does. The
// most clusters of each size are cudaOccupancyMaxActiveClusters's, less what clusters of three and five leave when they start beside others
// (92 and 56 output blocks in them ran two rounds: 7.9 -> 9.3 and 13.1 -> 16.5 us), for 148 multiprocessors (others
// take their share), written down because the count must be the same without a device; two to a multiprocessor past eight slices is known
// for sixteen.
// us at 1 / 8 / 17 / 32 rows, powers of two up to eight -> this: 12288 -> 4608 K3 27.8 / 32.9 / 42.2 / 53.4 -> (six) 23.6 / 25.7 / 41.7 /
// 42.8; 13824 -> 5120 K2 34.3 / 35.8 / 56.5 / 58.0 -> (six) 24.6 / 27.3 / 44.7 / 43.1; 10240 -> 4608 K4 22.9 / 28.6 / 35.7 / 43.8 -> (six) 19.6 /
// 21.6 / 33.9 / 36.4; 2560 -> 9728 K4 15.3 / 18.7 / 22.5 / 29.1 -> (three) 12.3 / 15.0 / 19.1 / 24.6; one row of 2048 -> 2048 5.3 -> (six,
// alone) 4.7, 6144 -> 2048 10.1 -> (six) 7.5, 7168 -> 1536 10.7 -> (eight) 6.8. The other way where no count that suits one row holds 32, which
// is at K1 and K2: 6144 -> 14336 K2 31.0 / 32.6 / 53.3 / 68.3 -> (three) 33.9 / 41.6 / 54.1 / 61.1, 11264 -> 8704 K1 30.8 / 34.5 / 79 / 84 -> (five)
// 40.2 / 48.2 / 61 / 66.
// sms: the device's multiprocessors; stage, cap, half: the bytes of a ring stage (two blocks), of a CTA, and of one of two on a
// multiprocessor; held(s, longest): the bytes a CTA of s slices holds beside its ring at 32 rows. 0: no count holds 32 rows.
template <typename Held>
uint32_t pick_split_dense(uint32_t sms, uint32_t nb, uint32_t blocks, uint32_t stage, uint32_t cap, uint32_t half, uint32_t& alone, Held&& held) {
    static const uint16_t kTwo[17] = {0, 296, 148, 88, 71, 50, 45, 37, 33, 0, 0, 0, 0, 0, 0, 0, 14};
    uint32_t best = 0, best_cost = ~0u;
    alone = 0;
#pragma GCC unroll 16  // with s known the divisions are products: 27 to 54 ns, 63 to 84 without
    for (uint32_t s = 16u; s > 0u; --s) {  // from the short slices down: the long ones fall to the first test
        if (s > nb) continue;
        const uint32_t one = clusters_alone(sms, s), two = kTwo[s] * sms / 148u;
        const bool single = blocks <= one;
        if (one == 0u || (!single && two == 0u)) continue;
        const uint32_t longest = (nb + s - 1u) / s, at_once = single ? one : two;
        auto rounds = [&](uint32_t fit, uint32_t block, uint32_t block_single, uint32_t fixed) {  // in 10 ns
            if (blocks <= fit) return longest * block + fixed;
            const uint32_t full = blocks / fit, rest = blocks - full * fit;
            return full * (longest * block + fixed) + (rest ? longest * (rest <= one ? block_single : block) + fixed : 0u);
        };
        const uint32_t row = rounds(at_once, single ? 58u : 116u, 58u, 300u + 10u * s);
        if (3u * row + longest * 80u + 640u + 10u * s > best_cost) continue;
        const uint32_t stages = (longest + 1u) / 2u, bytes = held(s, longest);
        if (bytes + stage > cap) continue;
        const bool pair = !single && bytes + (stages < 3u ? stages : 3u) * stage <= half;
        uint32_t rows = pair ? rounds(at_once, 260u, 80u, 640u + 10u * s) : rounds(one, 80u, 80u, 640u + 10u * s);
        if (stages > 1u && bytes + 2u * stage > cap) rows = rows * 7u / 5u;
        if (3u * row + rows <= best_cost) best = s, best_cost = 3u * row + rows, alone = single;
    }
    return best;
}

}  // namespace t3
