// How many warps a CTA of the dp4a decode kernels gets, how deep its rings are, and whether weight rows go out in pairs: chosen on the host once per
// call, in front of launches of a few microseconds.  So a choice costs some 50 ns whatever the shape (tests/test_gemv_plan.py): one division for the ring
// depths of all counts, and the weights of a count from a table.
#pragma once

#include <cmath>
#include <cstddef>
#include <cstdint>

namespace tpb_gemv {

struct GemvPlan {
    int warps = 0, stages = 0;   // 0: the activations leave no room
    bool pairs = false;          // weight rows are dealt out in pairs (warp_row_pairs)
};

constexpr int kPlanWarps = 20;   // of any kernel
struct PlanWeights {
    double inv[kPlanWarps + 1];      // 1 / w
    double turns[kPlanWarps + 1];    // what w warps cost for filling the SM's four schedulers unevenly
    double worth[kPlanWarps + 1];    // its inverse, and that more warps hide a little more latency
    PlanWeights() : inv{}, turns{}, worth{} {
        for (int w = 1; w <= kPlanWarps; w++) {
            inv[w] = 1.0 / w;
            turns[w] = (double)(4 * ((w + 3) / 4)) / w;
            worth[w] = pow((double)w / kPlanWarps, 0.1) / turns[w];
        }
    }
};
static const PlanWeights kPlanWeights;

inline double ceil_about(double v) { return (double)(long long)(v + 0.999999); }

// Ring stages (of `stage` bytes and an mbarrier each) that fit beside `act` bytes, over all warps.
inline int64_t plan_slots(size_t limit, size_t act, size_t stage) {
    return act + 64 <= limit ? (int64_t)((limit - act - 64) / (stage + 8)) : 0;
}

// Warps and stages of the Q8_0 dp4a kernels for one rows-per-stage choice (stage = its bytes).  The slowest warp carries
// ceil(rows / warps_total) rows.  Among the counts that fit (with >= 2 stages and the activations in shared memory) take the one with the best
// balance; ties go to more warps.  E.g. 5120 rows on 148 SMs: 16 warps -> 2.16 rows per warp (3 vs 2, 72 %), 12 warps -> 2.88 (96 %).
// Kernels that may have more than sixteen warps deal rows out in pairs, one a step (warp_row_pairs).  What counts then is the share of the
// warps' steps that is work -- a third of it, as the last steps of the slowest warps run on an SM that is half empty and so faster -- how evenly the warps
// fill the SM's four schedulers, and a little how many there are.  us at M = 1, at most sixteen warps with ranges cut at any row / so: 5120 x 5120
// 7.9 / 6.6 (twelve warps with two steps / eighteen with one), 17408 x 5120 17.8 / 17.2, 14336 x 4096 12.3 / 11.9, 5120 x 17408 20.3 / 17.8, 20000 x 2304 18.8 / 13.1,
// 32000 x 4096 23.3 / 23.3 (on 20 warps 24.3); the f32 kernel 5120 x 5120 10.7 / 9.4, 14336 x 4096 16.5 / 14.8, 17408 x 5120 23.6 / 21.3, 5120 x 17408 27.2 / 21.7.
// More than sixteen only where each of them gets more than one row: a CTA is launched for every two rows a warp, so a count that leaves warps with one row
// leaves SMs without a CTA (2500 rows on eighteen warps a CTA: 70 CTAs, on nine 139; us, eighteen / nine: f32 2504 x 8704 11.5 / 9.1, 2746 x 11264 13.4 /
// 10.4, Q8_0 at M = 2 2372 x 9216 9.2 / 7.7).
inline GemvPlan dp4a_plan(int sms, size_t limit, size_t act, int64_t rows, int stage, int max_warps, int max_stages) {
    GemvPlan best;
    const int slots = (int)plan_slots(limit, act, (size_t)stage);
    const bool pairs = max_warps > 16;
    const double per_sm = (double)rows / sms;
    double best_eff = -1.0;
    for (int w = max_warps; w >= (max_warps < 16 ? max_warps / 2 : 8); w--) {
        if (2 * w > slots || (w > 16 && rows <= (int64_t)sms * w)) continue;
        const double per_warp = per_sm * kPlanWeights.inv[w];
        double eff = per_warp, margin = 0.02;
        if (pairs && rows > 2ll * sms * w) {
            const double n = per_warp * 0.5;
            eff = n / (0.65 * n + 0.35 * ceil_about(n)) * kPlanWeights.worth[w];
            margin = 0.0;
        } else if (rows >= (int64_t)sms * w) {
            eff = per_warp / ceil_about(per_warp);
        }
        if (eff > best_eff + margin) {
            best_eff = eff;
            best.warps = w;
        }
    }
    if (best.warps != 0) best.stages = max_stages * best.warps <= slots ? max_stages : slots / best.warps;
    return best;
}

// Warps and stages of the dp4a kernels of the other formats.  Every warp owns a contiguous range of whole rows; among the counts that fit with
// >= 2 stages take the one whose ranges divide most evenly (ties: more warps).
// With one or two activation rows and more than one step a warp, rows may be dealt out in pairs, one a step (may_pair): to the number of warps whose cost is
// lowest, its average number of steps and, as the last ones run on an SM that is half empty, a third of what the slowest warp has above it, over how
// evenly the warps fill the four schedulers.  What decides between ranges and pairs is the steps of the slowest warp: pairs are taken
// where they have fewer of them, and with the same number from five on, or from three where the ranges come out at thirteen or fourteen
// warps, which leave schedulers with three warps beside some with four.  Ranges / pairs over 300 shapes and formats at M = 1 and 2, by the slowest warp's steps: 9 / 3
// 1.5 x, 5 / 4 1.07, 3 / 2 1.08, 5 / 5 1.03, 4 / 4 and 3 / 3 on 13 and 14 warps 1.03, 3 / 3 on others 0.94, 2 / 2 0.96; over 300 others the rule's worst choice
// has 0.96.  us at M = 1: 14336 x 4096 q4_k 9.8 (14 warps of 6.92 rows) / 9.1 (16 of 3.03 pairs), q5_k 11.8 / 10.8, q6_k 13.8 / 12.9, iq4_nl 16.5 / 15.4; 13500 x
// 6144 q4_k 19.9 / 10.8; but 10638 x 5632 q6_k (12 of 5.99, 16 of 2.25 pairs) 14.8 / 17.3, 5907 x 1280 q5_k (10 of 3.99, 16 of 1.25) 4.5 / 5.4.
inline GemvPlan kq_plan(int sms, size_t limit, size_t act, size_t stage, int64_t rows, int max_stages, bool may_pair) {
    GemvPlan best;
    const int slots = (int)plan_slots(limit, act, stage);
    may_pair = may_pair && rows > 2ll * 16 * sms;
    const double per_sm = (double)rows / sms;
    double best_eff = -1.0, pair_cost = 0.0;
    int cut_steps = 0, pair_warps = 0, pair_steps = 0;      // steps: of the slowest warp
    for (int w = 16; w >= 4; w--) {
        if (2 * w > slots) continue;
        const double per_warp = per_sm * kPlanWeights.inv[w], most = ceil_about(per_warp);
        const double eff = rows >= (int64_t)sms * w ? per_warp / most : per_warp;
        if (eff > best_eff + 0.02) {
            best_eff = eff;
            best.warps = w;
            cut_steps = ((int)most + 1) / 2;
        }
        if (!may_pair) continue;
        const double steps = 0.5 * per_warp, top = ceil_about(steps);
        const double cost = (0.65 * steps + 0.35 * top) * kPlanWeights.turns[w];
        if (pair_warps == 0 || cost < pair_cost) {
            pair_cost = cost;
            pair_warps = w;
            pair_steps = (int)top;
        }
    }
    const int same_from = best.warps == 13 || best.warps == 14 ? 3 : 5;
    if (pair_warps != 0 && (pair_steps < cut_steps || (pair_steps == cut_steps && pair_steps >= same_from))) {
        best.warps = pair_warps;
        best.pairs = true;
    }
    if (best.warps != 0) best.stages = max_stages * best.warps <= slots ? max_stages : slots / best.warps;
    return best;
}

}  // namespace tpb_gemv
