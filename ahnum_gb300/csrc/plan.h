// Per-FFT-length plans: four-step shape, mixed-radix stage plans and the twiddle tables, built
// once per (device, L) on the host and kept resident on the device.
#pragma once

#include <cstdint>
#include <memory>
#include <vector>

#include "device.h"

namespace kg {

struct LengthPlan {
    uint32_t L = 0, H = 0, R = 0, C = 0;
    FftPlan rp, cp;                   // row plan (C points), column plan (R points)
    std::vector<int2> pairs;          // row pairs (p, p'), p <= p'
    // device copies
    int device = -1;
    int4 *twr = nullptr, *twc = nullptr, *t4 = nullptr, *sw = nullptr;
    int2 *dpairs = nullptr;
    size_t device_bytes = 0;
    ~LengthPlan();
};

// H = R*C with C a multiple of kGroup; the autotuned shape of this length if one was set, else
// rows about four times as long as columns.  false if no usable shape exists.
bool choose_shape(uint32_t H, uint32_t &R, uint32_t &C);
// Rows and column-group width of a batch slot: choose_shape's rows and groups of 8.  Columns of more than
// 896 rows leave no room for 8: groups of 4, or, where the number's digits ask for 8 (min_bits: the
// narrowest; top_digits: L - top_t), the longest columns that do.  false if no shape takes the number.
bool throughput_group(uint32_t H, unsigned min_bits, unsigned top_digits, uint32_t &R, int &G);
// Use R rows for FFT length L from now on (R = 0: back to the default); false if unusable.
bool set_shape_override(uint32_t L, uint32_t R);
// Usable shapes of H = R*C near balance, at most `max`; returns the count.
int shape_candidates(uint32_t H, uint32_t *R, uint32_t *C, int max);
// The stages of a length-n transform; false if n has a prime factor above 7.  narrow: of numbers whose
// digits have no more than kNarrowBits bits.
bool make_fft_plan(int n, FftPlan &pl, bool narrow = false);
constexpr unsigned kNarrowBits = 10;

// exp(-2 pi i j / m), j = 0..m-1, times 2^62 in limbs {c1, c0, s1, s0} (FftStage)
std::vector<int4> roots_neg(uint32_t m);

// Shape and column-group width for one test run alone: spread every pass over the SMs so the
// squaring's latency, not its total work, is smallest (chain_us in plan.cpp).  Throughput (batched) use takes
// choose_shape and G = kGroup instead.  min_bits: the narrowest digit; top_digits: L - top_t.
// An autotuned shape of the length (set_latency_override) comes first wherever the number's
// digits allow its group width.
bool choose_latency_shape(uint32_t H, int nsm, unsigned min_bits, unsigned top_digits, uint32_t &R,
                          uint32_t &C, int &G);
// Use R rows and column groups of G for one test alone at FFT length L from now on (R = 0: back
// to the model); false if the shape is unusable.
bool set_latency_override(uint32_t L, uint32_t R, int G);

// Cached plan for (current device, L, R) (R = 0: choose_shape); nullptr if L cannot be planned or
// the device upload fails.  Thread-safe.
std::shared_ptr<LengthPlan> get_plan(uint32_t L, uint32_t R = 0);
// Host tables only (no device upload).
struct PlanTables {
    std::vector<int4> twr, twc, t4, sw;
};
std::shared_ptr<LengthPlan> build_plan_host(uint32_t L, uint32_t R, PlanTables *tables);

}  // namespace kg
