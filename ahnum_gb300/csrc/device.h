// Structures shared by the host code and the sm_103a kernels.
//
// One squaring of a number of L real words uses a complex transform of H = L/2 points arranged
// four-step as R rows x C columns, element m = r*C + c (row-major):
//   stored form  S[k_r][c] = (column transform over r of u, times w_H^{c*k_r}), rows in natural
//                frequency order, where u_m = x_{2m} w_{2m} + i x_{2m+1} w_{2m+1} are the
//                weighted digits;
//   row pass     forward row transform (C points), real-split square or product, inverse row
//                transform;
//   column pass  conj twiddle, inverse column transform, unweight/round/carry, reweight,
//                forward column transform, twiddle.
// This is the pass structure of the reference's two-pass backend (src/fast2p.c:1-19); the
// kernels that implement it are written for the GPU.
#pragma once

#include <cstdint>
#include <vector_types.h>

namespace kg {

constexpr int kMaxStages = 8;    // of a transform: at most 2048 points, prime factors 2, 3, 5, 7
constexpr int kGroup = 8;        // widest column group (16 digits per row segment); C is a multiple of it
constexpr int kMaxAddend = 4;    // sparse constant digits folded into the normaliser

// One stage of a transform (fixed_fft.cuh).
struct alignas(16) FftStage {
    int radix, span;
    unsigned magic;    // floor(v / span) = v * magic >> 32 for v < 2^16 (span > 1)
    int off;           // twiddle records: for each j < span, radix - 1 of w^(t j), t = 1..radix-1,
                       // w = exp(-2 pi i / (radix span)), each {c1, c0, s1, s0}: the signed 32-bit
                       // limbs of (c + i s) 2^62
};

// Mixed-radix transform of length n in 64-bit fixed point, natural order in and out.  The stages run
// in order, the first with span 1 (no twiddles).
struct FftPlan {
    int n = 0;
    int ns = 0;        // 2 or more
    int headroom = 0;  // bits the modulus of the input stays below 2^62
    int scale = 0;     // the transform leaves a factor 2^-scale
    int renorm = 0;    // the stage before which the values are scaled up to components below 2^61 (0: none)
    FftStage stage[kMaxStages] = {};
};

// Everything a kernel needs for one test (one modulus).  Lives in device memory; a kernel copies
// the descriptor of the item it works on into shared memory (16-byte chunks, hence alignas).
struct alignas(16) TestDesc {
    // shape
    int L, H, R, C, NG;      // NG = C / G column groups
    int G;                   // columns per column group: 2, 4 or 8 (2G digits per row segment)
    FftPlan rp, cp;          // row plan (length C), column plan (length R)
    // twiddles, {c1, c0, s1, s0} as in FftPlan
    const int4 *twr;         // row stages
    const int4 *twc;         // column stages
    const int4 *t4;          // [k_r][c] four-step twiddle w_H^{c * k_r}
    const int4 *sw;          // [k_r][k_c] real-split twiddle w_H^{k_r + R * k_c}
    const int2 *pairs;       // row pairs (k_r, (R - k_r) mod R), k_r <= its partner
    int npairs;
    // per-modulus tables, 64-bit fixed point
    const uint8_t *bits;     // [L]
    const uint8_t *segbits;  // [g][row][2G] the same, by column group: the widths of a row segment
    const long long *w;      // [column][row][2] weights w_j 2^61
    const long long *osc;    // [L] k / (w_j * 4H) 2^(62 - osc_exp): unweight and scale after a product
    const long long *idig;   // [L] 1 / (R * w_j) 2^(62 - idig_exp): unweight after the column inverse alone
    int osc_exp, idig_exp;
    int pitch;               // columns from one row to the next of t4 and osc: C
    int digit_bits;          // digits entering the column forward pass stay below 2^digit_bits
    // scratch
    long long *dig;          // [L] integer digits: a number's in their order, or between the two column
                             // kernels [column][row][2]
    long long *slot;         // [NG * R] carry into segment (g, r), index g*R + r
    unsigned long long *maxerr;  // bits of the largest round-off (non-negative double)
    int *rexp;               // [R] the row pass leaves row k_r as fixed-point numbers times 2^rexp[k_r]
    int *emax;               // no component of any row of it reaches 2^*emax (INT_MIN between products)
    // top fold
    unsigned long long k, k_inv; // k_inv = floor((2^64 - 1) / k)
    int top_t, top_m, top_shift; // top_shift = s_L - s_t
    // constant digits added before the carry (LLR: -2), (index, value)
    int nadd;
    int addj[kMaxAddend];
    long long addv[kMaxAddend];
    // operands of the current operation
    double2 *x;
    const double2 *y;
    int count;      // steps of the current launch sequence this test takes part in
    int err_every;  // round-off is tracked on steps that are multiples of this
};

// A unit of work: the test and the row pair or column group it covers.
struct WorkItem {
    int test;
    int unit;
};

}  // namespace kg
