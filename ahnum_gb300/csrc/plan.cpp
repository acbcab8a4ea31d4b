// Per-FFT-length plans (see plan.h).
#include "plan.h"

#include <cuda_runtime.h>

#include <climits>
#include <cstdint>
#include <cstdlib>

#include "../../include/kite_cuda.h"
#include "kernels.h"

#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <tuple>
#include <utility>

namespace kg {

LengthPlan::~LengthPlan() {
    if (device < 0) return;
    int prev = -1;
    cudaGetDevice(&prev);
    cudaSetDevice(device);
    cudaFree(twr);
    cudaFree(twc);
    cudaFree(t4);
    cudaFree(sw);
    cudaFree(dpairs);
    if (prev >= 0) cudaSetDevice(prev);
}

static bool factorable(uint32_t n) {
    for (uint32_t p : {2u, 3u, 5u, 7u})
        while (n % p == 0) n /= p;
    return n == 1;
}

static bool shape_usable(uint32_t H, uint32_t r, uint32_t c) {
    return r >= 2 && r <= 1024 && c >= 16 && c <= 2048 && c % kGroup == 0 && (uint64_t)r * c == H &&
           factorable(r) && factorable(c);
}

// a column group's two buffers fit shared memory: up to 896 rows in groups of 8, always in narrower ones
static bool column_fits(uint32_t r, int g) { return 2 * (size_t)r * g * sizeof(int4) <= kMaxColSmem; }

// Shapes chosen by the autotuner (or a tuning file), by FFT length L = 2H: R rows.
static std::mutex g_shape_mu;
static std::map<uint32_t, uint32_t> g_shape;

bool set_shape_override(uint32_t L, uint32_t R) {
    std::lock_guard<std::mutex> lock(g_shape_mu);
    if (!R) {
        g_shape.erase(L);
        return true;
    }
    if (L % 2 || R == 0 || (L / 2) % R || !shape_usable(L / 2, R, L / 2 / R)) return false;
    g_shape[L] = R;
    return true;
}

int shape_candidates(uint32_t H, uint32_t *R, uint32_t *C, int max) {
    int n = 0;
    for (uint32_t c = 16; c <= 2048 && c <= H / 2 && n < max; c += kGroup) {
        if (H % c || !shape_usable(H, H / c, c)) continue;
        const double ratio = (double)c / (H / c);
        if (ratio < 0.5 || ratio > 64) continue;  // far from balanced: never the fastest
        R[n] = H / c;
        C[n] = c;
        n++;
    }
    return n;
}

bool choose_shape(uint32_t H, uint32_t &R, uint32_t &C) {
    static std::once_flag env_once;
    std::call_once(env_once, [] {
        if (const char *p = std::getenv("KITE_GB300_TUNING")) kc_tuning_load(p);
    });
    {
        std::lock_guard<std::mutex> lock(g_shape_mu);
        auto it = g_shape.find(2 * H);
        if (it != g_shape.end()) {
            R = it->second;
            C = H / R;
            return true;
        }
    }
    double best = 1e30;
    R = C = 0;
    // rows up to 2048 points: a product's row pass holds 6 rows of C points in shared memory
    for (uint32_t c = 16; c <= 2048 && c <= H / 2; c += kGroup) {
        if (H % c) continue;
        uint32_t r = H / c;
        if (!shape_usable(H, r, c)) continue;
        // rows about four times as long as columns
        double cost = std::fabs(std::log2((double)r) - std::log2((double)c) + 2.0);
        if (cost < best) {
            best = cost;
            R = r;
            C = c;
        }
    }
    return R != 0;
}

// Rounds of a CTA in the stages of `count` transforms of length n together, in units of a radix-4
// round: a stage whose butterflies do not fill the CTA costs as much as one that does.
static double stage_rounds(uint32_t n, uint32_t count) {
    static const std::pair<uint32_t, double> radix[] = {{4, 1.0}, {2, 0.5}, {3, 0.9}, {5, 1.9}, {7, 3.0}};
    double sum = 0;
    uint32_t m = n;
    for (const auto &[p, weight] : radix)
        for (; m % p == 0; m /= p) sum += weight * ((count * (n / p) + kThreads - 1) / kThreads);
    return sum;
}

// Predicted time in us of one squaring of a chain (chain.cuh) of R x C in column groups of G, from
// what every CTA does in a row: fitted to 420 shapes of 23 lengths from 320 to 1769472 digits, whose
// choices are within 1.6% of the best shape on average.
// In one cluster: the rounds of a row pair's and a column group's stages, there and back, and the digits
// of a segment, whose carries are serial.  Up to 2048 digits only: from 3072 on a cluster's wide groups
// lose to narrow ones on more CTAs (13.6 against 12.6 us).  On the whole GPU:
//  - a fixed part, mostly the two grid barriers, the wait for a neighbour and the loads after them;
//  - the same rounds, and the rounds over the items' points besides (loads, squares, carries; a column
//    group has two such passes);
//  - 1.6 times that in a wave which puts two CTAs on an SM: alone, a CTA waits for its own latencies;
//  - a wave more wherever a pass has more items than CTAs stay: one per SM, or two up to kTwoCtaSmem;
//  - the tables read from L2 when they do not stay in shared memory.
static double chain_us(uint32_t R, uint32_t C, int G, int nsm) {
    constexpr size_t kTwoCtaSmem = 108 * 1024;
    constexpr double kFixed = 6.18, kRound = 0.435, kPoints = 0.547, kWave = 3.14, kFromL2 = 4.8, kPerLog = 0.23;
    const uint32_t pairs = R / 2 + 1, groups = C / G, most = std::max(pairs, groups);
    if (most <= (uint32_t)kClusterItems)
        return 3.17 + 0.684 * 2 * (stage_rounds(C, 2) + stage_rounds(R, G)) + 0.444 * G + (R * C > 1024 ? 1e2 : 0);
    const size_t smem = 16 * std::max((size_t)4 * C, (size_t)2 * R * G);
    const size_t table = 16 * ((size_t)2 * C + R + (size_t)4 * R * G) + (size_t)2 * R * G;
    const bool keeps = most <= (uint32_t)nsm && smem + table <= kMaxChainSmem;
    const uint32_t resident = std::min<uint32_t>(most, nsm * (!keeps && smem <= kTwoCtaSmem ? 2 : 1));
    const auto pass = [&](uint32_t items, uint32_t n, uint32_t count, double passes) {
        double us = -kWave * passes;
        const double once = kRound * 2 * stage_rounds(n, count) + kPoints * passes * ((count * n + kThreads - 1) / kThreads);
        for (uint32_t left = items; left; left -= std::min(left, resident))
            us += kWave * passes + once * (std::min(left, resident) > (uint32_t)nsm ? 1.6 : 1.0);
        return us;
    };
    return kFixed + pass(pairs, C, 2, 1) + pass(groups, R, G, 2) + (keeps ? 0 : kFromL2) + kPerLog * std::log2((double)R);
}

// Latency shapes chosen by the autotuner (or a tuning file), by FFT length L = 2H: (R, G).
static std::map<uint32_t, std::pair<uint32_t, int>> g_latency;

// the carry into a segment must be absorbed by 2g-1 digits of at least min_bits (a product's
// carry stays below 2^(51 - b)), and the top region must fit one segment
static bool group_fits(int g, unsigned min_bits, unsigned top_digits) {
    return (2 * g - 1) * (int)min_bits >= 51 - (int)min_bits && (int)top_digits <= 2 * g;
}

bool throughput_group(uint32_t H, unsigned min_bits, unsigned top_digits, uint32_t &R, int &G) {
    uint32_t C = 0;
    if (!choose_shape(H, R, C)) return false;
    G = kGroup;
    if (column_fits(R, G)) return (int)top_digits <= 2 * G;
    G = kGroup / 2;
    if (group_fits(G, min_bits, top_digits)) return true;
    for (uint32_t c = 16; c <= 2048 && c <= H / 2; c += kGroup)
        if (H % c == 0 && shape_usable(H, H / c, c) && column_fits(H / c, kGroup)) {
            R = H / c;  // the longest columns that fit groups of 8
            G = kGroup;
            break;
        }
    return (int)top_digits <= 2 * G;
}

bool set_latency_override(uint32_t L, uint32_t R, int G) {
    std::lock_guard<std::mutex> lock(g_shape_mu);
    if (!R) {
        g_latency.erase(L);
        return true;
    }
    if (L % 2 || (L / 2) % R || !shape_usable(L / 2, R, L / 2 / R) || (G != 2 && G != 4 && G != 8) ||
        (L / 2 / R) % G)
        return false;
    g_latency[L] = {R, G};
    return true;
}

bool choose_latency_shape(uint32_t H, int nsm, unsigned min_bits, unsigned top_digits, uint32_t &R,
                          uint32_t &C, int &G) {
    {
        // an autotuned shape of this length, where this number's digits allow its groups
        std::lock_guard<std::mutex> lock(g_shape_mu);
        auto it = g_latency.find(2 * H);
        const int g = it == g_latency.end() ? 0 : column_fits(it->second.first, it->second.second) ? it->second.second : kGroup / 2;
        if (g && group_fits(g, min_bits, top_digits)) {
            R = it->second.first;
            C = H / R;
            G = g;
            return true;
        }
    }
    double best = 1e300;
    R = C = 0;
    G = kGroup;
    if (nsm < 1) nsm = 1;
    // The second round: where columns are too long for groups of 8 at every shape (from L = 3670017 on),
    // digits that ask for 8 take groups of 4 all the same; the last digit of a segment keeps what the
    // others leave of a carry (TestDesc::digit_bits).
    const bool fits8 = group_fits(kGroup, min_bits, top_digits);
    for (bool narrow : {false, true}) {
        for (uint32_t c = 16; c <= 2048 && c <= H / 2; c += kGroup) {
            if (H % c || !shape_usable(H, H / c, c)) continue;
            const uint32_t r = H / c;
            for (int g : {2, 4, 8}) {
                if (!column_fits(r, g)) continue;
                if (!group_fits(g, min_bits, top_digits) && !(narrow && fits8 && g == 4 && (int)top_digits <= 2 * g)) continue;
                const double cost = chain_us(r, c, g, nsm) + (r < 4 ? 1e3 : 0);  // two rows: where nothing else fits
                if (cost < best - 1e-9) {
                    best = cost;
                    R = r;
                    C = c;
                    G = g;
                }
            }
        }
        if (R) return true;
    }
    return false;
}

bool make_fft_plan(int n, FftPlan &pl, bool narrow) {
    // The odd radices first (the first stage has span 1 and no twiddles), then a radix 2 if needed,
    // then radix 4; a transform of one stage gets a second one of radix 1.
    if (n < 2) return false;
    std::vector<int> rad;
    int m = n;
    for (int p : {7, 5, 3})
        for (; m % p == 0; m /= p) rad.push_back(p);
    int fours = 0;
    for (; m % 4 == 0; m /= 4) fours++;
    if (m % 2 == 0) {
        rad.push_back(2);
        m /= 2;
    }
    if (m != 1) return false;
    rad.insert(rad.end(), fours, 4);
    if (rad.size() == 1) rad.push_back(1);
    if (rad.size() > (size_t)kMaxStages) return false;
    pl = FftPlan{};
    pl.n = n;
    int s = 1, o = 0;
    double growth = 1, largest = 1;  // of the modulus, stage by stage
    for (int p : rad) {
        FftStage &g = pl.stage[pl.ns];
        g.radix = p;
        g.span = s;
        g.magic = s > 1 ? (unsigned)((1ull << 32) / s + 1) : 0;
        g.off = o;
        const bool divides = pl.ns > 0 && p > 2;  // a twiddled butterfly of radix 3, 4, 5, 7
        growth *= divides ? p / 4.0 : p;
        if (divides) pl.scale += 2;
        largest = std::max(largest, growth);
        o += (p - 1) * s;
        s *= p;
        pl.ns++;
    }
    // half a bit for the modulus of two components: every modulus then stays below 2^62 in every stage
    pl.headroom = (int)std::ceil(std::log2(largest) + 0.5 - 1e-9);
    // Random data lose half a bit a level against the bound.  Up to four bits of that leave the
    // round-off below half of what FP64 had at the same length; longer transforms take the bits
    // back before their last two stages, else the loss would pass FP64's from 2^9 points on.  Data that
    // gather on one element keep the bound itself, components up to 2^62, and are never scaled down.
    // Scaled up to components below 2^61 (moduli below 2^61.5), the stages left have to stay below 2^63.
    // Their growth is at most 1 where they are of radix 4 and 2.5 else, but for 686 = 7 7 7 2 (3.5), which is
    // not scaled up.  The first stage whose output can be looked at is stage 1.
    // A twiddled radix 3 takes more from random data than radix 4 (sqrt(3) / 4 against 1 / 2) and its
    // butterflies round more, so plans of 6 stages with three odd ones scale up before stage 2 instead.
    // Largest round-off at 734832 digits (rows of 1512 = 7 3 3 3 2 4) 0.30 before the last two, 0.14 so, FP64
    // 0.23; at 967680 (1080) 0.18, 0.07 and 0.14.  Scaling up at both costs the pass kernels 2 %.
    // Balanced digits lie half a unit below zero on average.  Of narrow ones that is a spectral line, 30 or 40
    // times the others at 250000 digits of 4 bits, and its square takes their bits until the stages have
    // spread it: their transforms, short ones too, scale up early.  Largest round-off at 373248 digits of
    // 4.2 bits 0.50 without, 0.16 so, FP64 0.35.
    if ((narrow || n > 256) && pl.ns >= 4) {
        const int odd = (int)std::count_if(rad.begin(), rad.end(), [](int p) { return p % 2 && p > 1; });
        const auto peak = [&](int from) {  // growth of the stages from `from` on
            double growth = 1, most = 1;
            for (int i = from; i < pl.ns; i++) {
                growth *= pl.stage[i].radix > 2 ? pl.stage[i].radix / 4.0 : 2;
                most = std::max(most, growth);
            }
            return most;
        };
        constexpr double kMost = 2.6;  // 2^61.5 times that is 0.92 2^63
        if ((narrow || (odd >= 3 && pl.ns >= 6)) && peak(2) <= kMost) pl.renorm = 2;
        else if (peak(pl.ns - 2) <= kMost) pl.renorm = pl.ns - 2;
    }
    return true;
}

// round(v 2^62) in signed limbs; the lower one has a negative
static void limbs62(long double v, int &hi, int &lo) {
    int64_t x = (int64_t)std::floor(v * 4611686018427387904.0L + 0.5L);
    if ((int32_t)(uint32_t)x == INT32_MIN) x++;
    hi = (int)((x + 0x80000000ll) >> 32);
    lo = (int)(uint32_t)x;
}

std::vector<int4> roots_neg(uint32_t m) {
    std::vector<int4> r(m);
    for (uint32_t j = 0; 2 * j <= m; j++) {
        // angle pi*x with x = num/den = 2j/m in [0, 1], reduced to [0, 1/4] by exact reflections
        uint64_t num = 2 * (uint64_t)j, den = m;
        bool neg = false, swap = false;
        if (2 * num > den) {  // x -> 1 - x: cos negates
            num = den - num;
            neg = true;
        }
        if (4 * num > den) {  // x -> 1/2 - x: cos and sin swap
            num = den - 2 * num;
            den *= 2;
            swap = true;
        }
        const long double th = 3.14159265358979323846264338327950288L * (long double)num / (long double)den;
        long double c = cosl(th), s = sinl(th);
        if (swap) std::swap(c, s);
        if (neg) c = -c;
        limbs62(c, r[j].x, r[j].y);
        limbs62(-s, r[j].z, r[j].w);
        if (j) {
            r[m - j] = r[j];
            limbs62(s, r[m - j].z, r[m - j].w);
        }
    }
    return r;
}

// Twiddle records of every stage (see FftStage), from the roots of order h, a multiple of pl.n
static void stage_twiddles(const FftPlan &pl, const std::vector<int4> &roots, std::vector<int4> &tw) {
    const uint64_t h = roots.size();
    tw.clear();
    for (int i = 0; i < pl.ns; i++) {
        const int p = pl.stage[i].radix, s = pl.stage[i].span;
        const uint64_t step = h / ((uint64_t)p * s);
        for (int j = 0; j < s; j++)
            for (int t = 1; t < p; t++) tw.push_back(roots[step * t * j]);
    }
}

std::shared_ptr<LengthPlan> build_plan_host(uint32_t L, uint32_t rows, PlanTables *tables) {
    if (L % (2 * kGroup) || L < 64) return nullptr;
    auto pl = std::make_shared<LengthPlan>();
    pl->L = L;
    pl->H = L / 2;
    if (rows) {
        if (pl->H % rows || !shape_usable(pl->H, rows, pl->H / rows)) return nullptr;
        pl->R = rows;
        pl->C = pl->H / rows;
    } else if (!choose_shape(pl->H, pl->R, pl->C)) {
        return nullptr;
    }
    if (!make_fft_plan((int)pl->C, pl->rp) || !make_fft_plan((int)pl->R, pl->cp)) return nullptr;
    const uint32_t R = pl->R, C = pl->C, H = pl->H;
    for (uint32_t kr = 0; kr < R; kr++) {
        uint32_t k2 = (R - kr) % R;
        if (kr <= k2) pl->pairs.push_back(make_int2((int)kr, (int)k2));
    }
    if (tables) {
        const std::vector<int4> roots = roots_neg(H);
        stage_twiddles(pl->rp, roots, tables->twr);
        stage_twiddles(pl->cp, roots, tables->twc);
        tables->t4.resize((size_t)R * C);
        tables->sw.resize((size_t)R * C);
        for (uint32_t kr = 0; kr < R; kr++)
            for (uint32_t c = 0; c < C; c++) {
                tables->t4[(size_t)kr * C + c] = roots[(uint64_t)c * kr % H];
                tables->sw[(size_t)kr * C + c] = roots[kr + (uint64_t)R * c];
            }
    }
    return pl;
}

template <class T>
static bool upload(const std::vector<T> &h, T **d, size_t &bytes) {
    size_t nb = h.size() * sizeof(T);
    if (cudaMalloc((void **)d, nb ? nb : sizeof(T)) != cudaSuccess) return false;
    bytes += nb;
    return !nb || cudaMemcpy(*d, h.data(), nb, cudaMemcpyHostToDevice) == cudaSuccess;
}

std::shared_ptr<LengthPlan> get_plan(uint32_t L, uint32_t R) {
    static std::mutex mu;
    static std::map<std::tuple<int, uint32_t, uint32_t>, std::shared_ptr<LengthPlan>> cache;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    uint32_t C = 0;
    if (L % 2 || (!R && !choose_shape(L / 2, R, C))) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find({dev, L, R});
    if (it != cache.end()) return it->second;
    PlanTables t;
    auto pl = build_plan_host(L, R, &t);
    if (!pl) return nullptr;
    pl->device = dev;
    bool ok = upload(t.twr, &pl->twr, pl->device_bytes) && upload(t.twc, &pl->twc, pl->device_bytes) &&
              upload(t.t4, &pl->t4, pl->device_bytes) && upload(t.sw, &pl->sw, pl->device_bytes) &&
              upload(pl->pairs, &pl->dpairs, pl->device_bytes);
    if (!ok) return nullptr;
    cache[{dev, L, R}] = pl;
    return pl;
}

}  // namespace kg
