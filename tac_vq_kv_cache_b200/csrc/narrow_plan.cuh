// How the search of 8- and 4-wide groups is divided among the blocks of the tcgen05 kernel, and which of its two kernels takes a call (host
// code; encode_narrow.cu, encode_tc.cu).
#pragma once

#include <stdint.h>

namespace tacvq {
namespace narrow {

constexpr int kRows = 128, kGroups = 4;  // rows of a tile; tiles that a block works on at a time, all of one (head, group) pair
constexpr int kSpan = 128;               // tiles of every pair that are dealt out together

// Tiles are dealt out in units of 1 << `shift` neighbouring tiles of a pair; the whole spans of a call of more than kSpan tiles in units of four.  In its part
// a block copies the tables of `visits` pairs and works in `rounds` rounds of up to four tiles, at most, which take as long as `cost` full rounds.
struct Deal {
    int blocks, shift, rounds, visits;
    double cost;
};

// A round of four tiles is taken for 1, one of two or fewer for 0.7, a table for 0.25 (16 x 8, two stages: 5.8, 4.0 and 1.4 us).
inline Deal deal(int64_t tiles, int64_t pairs, int sms) {
    const int64_t last = tiles > kSpan ? (tiles - 1) % kSpan + 1 : tiles;
    Deal best = {0, 0, 0, 0, 0.0};
    for (int shift = 2; shift >= 0; --shift) {
        const int unit = 1 << shift;
        if (unit > last || (last == kSpan && unit != kGroups)) continue;
        const int64_t per_pair = (last + unit - 1) / unit, units = per_pair * pairs, turns = (units + sms - 1) / sms;
        const int64_t blocks = tiles > kSpan ? sms : (units + turns - 1) / turns;
        const bool whole = units == blocks * turns && (per_pair % turns == 0 || turns % per_pair == 0);  // no part ends inside a pair that goes on
        const int64_t visits = whole ? (turns + per_pair - 1) / per_pair : 1 + (turns - 1 + per_pair - 1) / per_pair;
        const int64_t rest = kGroups - unit;  // tiles that may be missing in the last round of a visit
        const int64_t rounds = turns == 1 ? 1 : whole ? (turns / visits * unit + 3) / 4 * visits : (turns * unit + rest * visits) / 4;
        const int64_t missing = 4 * rounds - turns * unit + turns / per_pair * (per_pair * unit - last);  // a pair's last unit may be short
        const double cost = (double)rounds - 0.15 * (double)(missing < 2 * rounds ? missing : 2 * rounds) + 0.25 * (double)visits;
        if (best.blocks == 0 || cost < best.cost) best = {(int)blocks, shift, (int)rounds, (int)visits, cost};
    }
    return best;
}

// Whether this kernel takes a call, which the mma.sync kernel of many small blocks takes otherwise.  That one goes by rows, and a full round
// here is worth so many rows of a (head, group): fewer the more stages there are, as it keeps fewer blocks on an SM then.  us of the mma.sync / tcgen05 kernel, rows wanted:
//   one stage     16 x 8: one head x 1500 rows 6.2/7.1, 2250 7.2/7.4; 4 x 520 7.0/7.8; 8 x 256 7.0/7.2, 300 10.0/7.9, 520 12.0/10.0; 32 x 128 11.8/16.6
//                 32 x 4: 2 x 520 7.3/7.4; 4 x 300 10.1/7.4; 16 x 130 16.4/16.8
//   two stages    16 x 8: 1 x 2250 10.3/9.5; 2 x 700 8.7/9.2; 4 x 520 10.1/10.2; 8 x 300 14.1/10.2, 1030 31.9/19.8; 32 x 90 17.6/23.0, 130 24.0/25.8
//   three, four   16 x 8: 4 x 450 13.2/11.5; 8 x 190 11.2/11.5; four 2 x 520 11.8/13.6; 4 x 300 13.9/13.6, 450 23.0/13.5; 16 x 128 22.6/20.3
//   eight         16 x 8: 2 x 512 19.9/22.4; 4 x 300 36.4/22.0
inline bool pays(int64_t rows, int64_t pairs, int stages, int sms) {
    const double round = stages <= 1 ? 34500.0 : stages == 2 ? 30500.0 : stages == 3 ? 28000.0 : 18000.0;
    return (double)rows * (double)pairs >= round * deal((rows + kRows - 1) / kRows, pairs, sms).cost;
}

}  // namespace narrow
}  // namespace tacvq
