// Which work items an attention launch goes as. No CUDA in here, so that the CPU tests compile it too.
#pragma once

#include <algorithm>

namespace efa {

// How a launch is cut into work items: items256 of 256 rows, then items128 of 128 rows (a launch of their own where there are both); or
// tiles of 128 rows, one to a block of the one-tile kernel. And the stages of K and V that the last of them keeps, of which an issuing thread takes
// every stage_step-th.
struct FaPlan { int items256 = 0, items128 = 0, tiles = 0, k_slots = 0, v_slots = 0, stage_step = 1; };

struct PlanShape {
    int q_start, q_rows, S, H_local, nsplit, kv_len, causal, d_h;
    bool free_form;         // neither an order table nor the persistent form, which are made for 256-row items
    bool longest_first;     // else in the order of the rows
    long sms;
};

inline FaPlan plan_items(const PlanShape& a)
{
    constexpr int kStage = 128;                            // keys of a stage
    // 128-row items with their keys split over all the warpgroups where one wave of them is the whole launch (d_h 16 / 32 /
    // 64 / 128, 74 items of 256 rows and 16 key stages: 15 / 16 / 19 / 29 us against 25 / 27 / 28 / 37). Three waves of them against
    // two of 256 rows are worth it only where items are long and the tensor pipe is not what an item waits for. In us, 222
    // items of 256 rows: 42 / 48 / 54 against 48 / 52 / 55 (d_h 16 / 32 / 64, 16 stages), 26 / 28 / 34 against 28 / 30 / 34 (8 stages), even at
    // four, 82 against 76 (128, 16 stages).
    const long heads = (long)a.H_local * a.nsplit;
    const long total = heads * ((a.q_rows + 255) / 256), total128 = heads * ((a.q_rows + 127) / 128);
    const long sms = a.sms;
    const long waves256 = (total + sms - 1) / sms, waves128 = (total128 + sms - 1) / sms, rest = total % sms;
    const double keys = a.causal ? a.q_start + 0.5 * (a.q_rows + 256) : a.S;
    const double stages = keys / ((double)kStage * a.nsplit);                  // of an average item
    // Under a causal mask the longest item can be what a launch takes, and as 128-row items it is half of it. When the last item ends, in stages of
    // 256 rows; an item costs two of them besides, and 128 rows take 0.55 of a stage (0.67 at d_h 128). Longest first: the longest item, everything spread
    // over the SMs, or (d_h 128) the two that meet on an SM between two waves. In the order of the rows SMs take items in turn, and the longest comes last,
    // behind one of each wave. The times measured are 0.95 to 1.06 of that, at d_h 128 1.05 to 1.16, hence the lines. (Splits in the order of the
    // rows fit neither; up to d_h 64 they are taken as the first, at 128 as the second. With more than two waves of 256-row items that order
    // costs less than twice as many items: 41216 rows, three heads of 64 956 us, as 128-row items 1034.)
    // us, 256 against 128 rows, d_h 32 / 64 / 128, longest first: S=4096, 8 heads 47 / 47 / 56 against 27 / 28 / 43; S=8192, 4 heads 89 / 86 / 103
    // against 49 / 46 / 78; S=1024, 32 heads 15.6 / 17.0 / 20.1 against 12.9 / 14.0 / 20.8; S=4096, 12 heads 48 / 48 / 59 against 44 / 45 / 71;
    // S=2048, 24 heads 26.5 / 27.8 / 34.0 against 27.8 / 30.1 / 44.8; S=3072, 20 heads, rows from 1536 on, d_h 128 46 against 50; nothing at four
    // stages (S=512, 64 heads 9.7 against 10.4). In the order of the rows: S=4096, 5 heads 48 / 48 / 56 against 34 / 35 / 51; S=4096, 8 heads
    // 49 / 48 / 57 against 41 / 43 / 64; S=8192, 8 heads, rows from 4096 on 91 / 89 / 111 against 86 / 87 / 142; S=768, 32 heads 13 / 15.1 / 17.2 against 14 / 16.2 / 21.3.
    bool short_ends = false, even = true;                  // even: items of about one length, which come in waves
    if (a.causal) {
        const double longest = std::min<double>(a.kv_len, a.q_start + a.q_rows) / kStage, part = a.d_h < 128 ? 0.55 : 0.67, fixed = 2;
        const double shortest = a.nsplit > 1 ? 0 : (a.q_start + 128.) / kStage;
        const bool in_turn = !a.longest_first && (a.nsplit == 1 || a.d_h == 128) && total <= 2 * sms;
        auto end = [&](long n, double cost) {
            const double most = cost * longest, wave = cost * (longest - shortest) * sms / n;      // by which items differ that are a wave apart
            const long waves = (n + sms - 1) / sms;
            if (in_turn) return waves * (most + fixed) - wave * waves * (waves - 1) / 2;
            return std::max({most + fixed, n * (cost * stages + fixed) / sms, a.d_h == 128 && waves == 2 ? 2 * (most - wave + fixed) : 0});
        };
        // In order, heads that end on 128 rows: their last 256-row item, the longest, is half empty and takes less (S=1536, rows from 384 on, 48 heads of 16
        // 30.2 us against 31.9).
        const bool half_ends = in_turn && total * 2 > total128;
        const double line = (a.d_h == 128 ? 0.88 : in_turn ? 0.985 : 0.92) - (half_ends ? 0.08 : 0);
        even = longest < 1.25 * stages;
        short_ends = !even && longest >= 4 && end(total128, part) < line * end(total, 1);
    }
    const bool halves = a.free_form && (waves128 <= 1 || short_ends || (a.d_h < 128 && stages >= 8 && even && waves128 * 4 <= waves256 * 2 * 3));
    FaPlan plan;
    plan.items256 = (int)total;
    // Small heads with few keys and more than one wave of anything: the one-tile kernel. Two small blocks to an SM are faster up to two
    // stages, and above that where the 256-row items are more than one wave and end less evenly (the figures are in
    // fa_fwd_tile_sm100.cu). Without a mask that is so where the last wave of items is poorly filled (below four stages), or where they take more
    // waves than the tiles do two to an SM: a third more up to three stages, half as many again to five. Under a mask below four stages, and
    // to six and a half by the same half more where items are of about one length or tiles more than one wave. Over 900 shapes of one to six and a half
    // stages the form taken is 1.9 % slower than the better one in the mean (0.8 % without a mask; always the one-tile kernel 13 %, never 4 %).
    const long pairs = (total128 + 2 * sms - 1) / (2 * sms);                   // waves of tiles
    const bool half_more = waves256 * 2 >= pairs * 3;
    const bool uneven = a.causal ? stages < 4 || (stages < 6.5 && half_more && (even || pairs > 1))
                                 : (stages < 4 && total * 10 < waves256 * sms * 7) || (stages <= 3 ? waves256 * 3 >= pairs * 4 : stages <= 5 && half_more);
    if (a.d_h < 64 && a.free_form && total128 > sms && (stages <= 2 || (waves256 > 1 && uneven))) {
        plan.items256 = 0;
        plan.tiles = (int)total128;
    } else if (halves) {
        plan.items256 = 0;
        plan.items128 = (int)total128;
    // Items of equal length end in a wave of their own for the rest that does not fill the GPU. Where that rest
    // is at most half of a wave it goes as 128-row items behind the full waves (two of them at least, one at d_h 128: shorter
    // launches are decided above). 65536 keys, two heads of 64, three full waves and 68 items: 2.75 -> 2.59 ms; 37 heads x 2560 rows x 4096 keys
    // of d_h 64 / 32 141 -> 128 / 123 us. From 4096 keys on, where that is worth ten times a launch: 111 heads x 512 rows of d_h 128 140 -> 133 us.
    } else if (a.free_form && !a.causal && total > sms && rest > 0 && rest * 2 <= sms && a.kv_len >= 4096) {
        plan.items256 = (int)(total - rest);
        plan.items128 = (int)rest * 2;
    }
    return plan;
}

}  // namespace efa
