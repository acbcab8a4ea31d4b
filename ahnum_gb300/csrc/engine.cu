// Single-modulus engine behind the kc_* C ABI (include/kite_cuda.h).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <vector>

#include "../../include/kite_cuda.h"
#include "kernels.h"
#include "layout.h"
#include "plan.h"
#include "engine_internal.h"

using namespace kg;

bool kc_ok(kc_engine *e, cudaError_t rc) {
    if (rc != cudaSuccess && !e->err) e->err = -(int)rc;
    return rc == cudaSuccess;
}

int kc_get_limbs(kc_engine *e, const double *x, uint64_t *limbs) {
    if (kc_fetch_digits(e, x)) return e->err ? e->err : -1;
    e->lay.digits_to_limbs(reinterpret_cast<const int64_t *>(e->h_dig), limbs);
    return 0;
}

int kc_set_limbs(kc_engine *e, double *x, const uint64_t *limbs) {
    std::vector<int64_t> d(e->lay.L);
    e->lay.limbs_to_digits(limbs, d.data());
    return kc_from_digits(e, x, d.data());
}

void kc_queue_equal(kc_engine *e, cudaStream_t stream, const double *a, const double *b, int *flag) {
    LaunchSet s = e->ls;
    s.stream = stream;
    launch_col_digits(s, (const double2 *)a, e->d_dig);
    launch_col_digits(s, (const double2 *)b, e->d_dig2);
    launch_equal(stream, e->d_desc, 0, e->d_dig, e->d_dig2, flag);
}

int kc_mul_small_host(kc_engine *e, double *x, int64_t m) {
    std::vector<int64_t> d(e->lay.L);
    if (kc_to_digits(e, x, d.data())) return e->err ? e->err : -1;
    for (auto &v : d) v *= m;
    e->lay.carry(d.data());
    return kc_from_digits(e, x, d.data());
}

namespace {

bool ok(kc_engine *e, cudaError_t rc) {
    if (rc != cudaSuccess && !e->err) e->err = -(int)rc;
    return rc == cudaSuccess;
}

bool check_launch(kc_engine *e) { return ok(e, cudaGetLastError()); }

struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        cudaGetDevice(&prev);
        if (prev != dev) cudaSetDevice(dev);
    }
    ~DeviceGuard() {
        int cur = -1;
        cudaGetDevice(&cur);
        if (prev >= 0 && cur != prev) cudaSetDevice(prev);
    }
};

template <class T>
bool dalloc(kc_engine *e, T **p, size_t count) {
    return ok(e, cudaMalloc((void **)p, (count ? count : 1) * sizeof(T)));
}

void release(kc_engine *e) {
    if (e->graph) cudaGraphExecDestroy(e->graph);
    for (cudaEvent_t m : e->marks)
        if (m) cudaEventDestroy(m);
    cudaFree(e->d_desc);
    cudaFree(e->d_work);
    cudaFree(e->d_bits);
    cudaFree(e->d_w);
    cudaFree(e->d_osc);
    cudaFree(e->d_idig);
    cudaFree(e->d_dig);
    cudaFree(e->d_dig2);
    cudaFree(e->d_eq);
    if (e->h_eq) cudaFreeHost(e->h_eq);
    cudaFree(e->d_slot);
    cudaFree(e->d_maxerr);
    cudaFree(e->d_rexp);
    if (e->h_dig) cudaFreeHost(e->h_dig);
    if (e->h_err) cudaFreeHost(e->h_err);
    if (e->stream) cudaStreamDestroy(e->stream);
}

// 2^62 m / w for m in [1/2, 1), w in [1, 2) and inv = 1 / w: the quotient of doubles and what its
// remainder adds
int64_t fixed_ratio(double m, double w, double inv) {
    const double q = m * inv, r = std::fma(-q, w, m) * inv;
    return (int64_t)(q * 0x1p62) + (int64_t)(r * 0x1p62);
}

// Digits after the deferred carry: balanced, but for the last one of a segment, which takes what is
// left of a carry of at most 2^52 after the segment's other digits; below 2^(return value).
int digit_bits(const Layout &lay, int G) {
    unsigned lo = 64, hi = 0;
    for (uint8_t b : lay.bits) {
        lo = b < lo ? b : lo;
        hi = b > hi ? b : hi;
    }
    const int rest = std::max(0, 52 - 2 * G * (int)lo);
    const int64_t most = ((int64_t)1 << (hi - 1)) + ((int64_t)1 << rest) + 3;
    int bits = 0;
    while (((int64_t)1 << bits) <= most) bits++;
    return bits;
}

bool upload_desc(kc_engine *e) {
    return ok(e, cudaMemcpyAsync(e->d_desc, &e->desc, sizeof(TestDesc), cudaMemcpyHostToDevice, e->stream));
}

bool want_err(kc_engine *e) {
    bool t = e->err_every <= 1 || e->op_count % e->err_every == 0;
    e->op_count++;
    return t;
}

// one product pass: row pass (square or multiply), then the two column kernels
int product(kc_engine *e, double2 *x, const double2 *y) {
    const bool track = want_err(e);
    launch_rows(e->ls, y != nullptr, x, y);
    launch_col_inverse(e->ls, x, track ? 0 : 1);  // err_every > 1 when this one is not tracked
    launch_col_forward(e->ls, x, true);
    return check_launch(e) ? 0 : e->err;
}

// Calls between a caller's kernels that a capture in another thread must not forbid or be ended by
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

bool capturing(const kc_engine *e) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(e->stream, &st) == cudaSuccess && st != cudaStreamCaptureStatusNone;
}

// The engines of a device that squared alone and may still have work in their queues
struct Device {
    std::mutex mu;
    std::vector<kc_engine *> busy;
};
Device g_devices[kMaxDevices];

// Whether e's next squarings, which it launches under dev.mu, can be a chain.
//
// A chain's CTAs wait on one another, so all of them have to become resident, and they stay for
// milliseconds.  Chains whose CTAs together have an SM each run side by side; where the engines with
// work queued leave no room for that, the squarings run as launches of the pass kernels, which wait on
// nothing and share the SMs.  us per squaring of all contexts together on GB300, one thread each, with
// chains behind one another -> by this rule, for 1, 2, 4 and 8 contexts of the same length:
//   3584 digits    13.9 13.9 13.7 13.6 -> 14.2  7.1  3.5  2.6   49152   17.6 17.5 17.5 17.5 -> 17.5 11.9  6.4  4.2
//   28672          17.0 16.9 16.9 16.9 -> 16.0  8.2  5.6  3.5   442368  34.2 34.2 34.3 34.4 -> 34.5 33.1 22.8 17.7
bool chain_has_room(Device &dev, const kc_engine *e) {
    const RelaxedCapture relaxed;
    int others = 0;
    for (size_t i = 0; i < dev.busy.size();) {
        const kc_engine *o = dev.busy[i];
        if (o != e && !capturing(o) && cudaStreamQuery(o->stream) != cudaErrorNotReady) {
            dev.busy[i] = dev.busy.back();
            dev.busy.pop_back();
            continue;
        }
        if (o != e) others += o->chain_grid;
        i++;
    }
    if (others) (void)cudaGetLastError();  // not ready is no error
    return !others || others + e->chain_grid <= e->nsm;
}

// A graph of kGraphSteps squarings by the pass kernels, of the number in the second descriptor
bool make_graph(kc_engine *e) {
    if (e->graph) return true;
    const RelaxedCapture relaxed;
    LaunchSet s = e->ls;
    s.tests = e->d_desc + 1;
    cudaGraph_t graph = nullptr;
    if (!ok(e, cudaStreamBeginCapture(e->stream, cudaStreamCaptureModeRelaxed))) return false;
    for (int j = 0; j < (int)kGraphSteps; j++) {
        launch_rows(s, false, nullptr, nullptr, j);
        launch_col_inverse(s, nullptr, j);
        launch_col_forward(s, nullptr, true, j);
    }
    if (!ok(e, cudaStreamEndCapture(e->stream, &graph))) return false;
    const bool made = ok(e, cudaGraphInstantiate(&e->graph, graph, 0));
    cudaGraphDestroy(graph);
    return made;
}

// n squarings of x as launches of the pass kernels: graphs, and the rest one by one
int square_passes(kc_engine *e, double2 *x, uint64_t n) {
    for (; n >= kGraphSteps; n -= kGraphSteps) {
        if (!make_graph(e)) return e->err ? e->err : -1;
        TestDesc d = e->desc;
        d.x = x;
        if (std::memcmp(&d, &e->graph_desc, sizeof d)) {
            std::memcpy(&e->graph_desc, &d, sizeof d);
            if (!ok(e, cudaMemcpyAsync(e->d_desc + 1, &e->graph_desc, sizeof d, cudaMemcpyHostToDevice, e->stream))) return e->err;
        }
        if (!ok(e, cudaGraphLaunch(e->graph, e->stream))) return e->err;
        e->op_count += kGraphSteps;
    }
    for (; n; n--)
        if (product(e, x, nullptr)) return e->err;
    return 0;
}

// The form of the squarings follows what other engines do, so the queue does not run far ahead of the
// GPU: waits until fewer than 3 kAhead squarings of this engine are queued, n of them new.
bool limit_ahead(kc_engine *e, uint64_t n) {
    e->ahead += n;
    if (e->ahead < kAhead) return true;
    const RelaxedCapture relaxed;
    e->ahead = 0;
    cudaEvent_t &mark = e->marks[e->turn ^= 1];
    if (mark ? !ok(e, cudaEventSynchronize(mark)) : !ok(e, cudaEventCreateWithFlags(&mark, cudaEventBlockingSync | cudaEventDisableTiming)))
        return false;
    return ok(e, cudaEventRecord(mark, e->stream));
}

// count squarings of x.  A batch slot's few go by the pass kernels, and so do those that a caller
// captures: a chain counts its meetings from launch to launch and cannot be replayed.
int square_many(kc_engine *e, double2 *x, uint64_t count) {
    if (e->throughput || capturing(e)) {
        for (; count; count--)
            if (product(e, x, nullptr)) return e->err;
        return 0;
    }
    Device &dev = g_devices[e->device];
    while (count) {
        const int n = (int)std::min(count, e->chain_steps);
        if (!limit_ahead(e, (uint64_t)n)) return e->err;
        std::unique_lock<std::mutex> lock(dev.mu);
        const bool chain = e->chain_cluster || chain_has_room(dev, e);
        if (std::find(dev.busy.begin(), dev.busy.end(), e) == dev.busy.end()) dev.busy.push_back(e);
        if (e->chain_cluster || !chain) lock.unlock();  // nothing that has to fit beside another chain
        if (!chain) {
            if (square_passes(e, x, (uint64_t)n)) return e->err;
        } else {
            if (!ok(e, launch_chain(e->ls, e->nsm, e->chain_grid, e->chain_cluster, x, (int)(e->op_count % e->err_every), n, e->d_chain,
                                    e->arrived, e->d_flags, e->chained)))
                return e->err;
            if (!e->chain_cluster) {
                e->arrived += 2u * (unsigned)n * (unsigned)e->chain_grid;
                e->chained += (unsigned)n;
            }
            e->op_count += (uint64_t)n;
        }
        count -= (uint64_t)n;
    }
    return 0;
}

// waits for the engine's queue; false (and sticky) if it failed or a chain's wait gave up
bool wait_queue(kc_engine *e) {
    if (!ok(e, cudaStreamSynchronize(e->stream))) return false;
    if (*(volatile unsigned *)e->h_timeout) ok(e, cudaErrorLaunchTimeout);
    return !e->err;
}

int set_addend(kc_engine *e, int64_t c) {
    if (e->add_cached == (c != 0) && e->add_c == c) return 0;
    uint32_t idx[kMaxAddend];
    int64_t val[kMaxAddend];
    int cnt = 0;
    if (c) {
        cnt = e->lay.constant_digits(c, idx, val, kMaxAddend);
        if (cnt < 0) return -1;
    }
    e->desc.nadd = cnt;
    for (int i = 0; i < cnt; i++) {
        e->desc.addj[i] = (int)idx[i];
        e->desc.addv[i] = val[i];
    }
    e->add_cached = c != 0;
    e->add_c = c;
    return upload_desc(e) ? 0 : e->err;
}

}  // namespace

extern "C" {

kc_engine *kc_engine_new(uint64_t k, uint64_t n, uint32_t L, const uint8_t *bits, const double *w,
                         const double *oscale, uint32_t top_t, uint64_t top_st, uint32_t top_m,
                         uint64_t sL, int device) {
    return kc_engine_create(k, n, L, bits, w, oscale, top_t, top_st, top_m, sL, device, false);
}

}  // extern "C"

kc_engine *kc_engine_create(uint64_t k, uint64_t n, uint32_t L, const uint8_t *bits, const double *w,
                            const double *oscale, uint32_t top_t, uint64_t top_st, uint32_t top_m,
                            uint64_t sL, int device, bool throughput) {
    kc_engine *e = new (std::nothrow) kc_engine();
    if (!e) return nullptr;
    if (device < 0 && cudaGetDevice(&device) != cudaSuccess) {
        delete e;
        return nullptr;
    }
    e->device = device;
    e->throughput = throughput;
    DeviceGuard dg(device);
    if (!e->lay.build(k, n, L)) {
        delete e;
        return nullptr;
    }
    // a caller-provided layout must be the one this (k, n, L) defines
    if ((bits && std::memcmp(bits, e->lay.bits.data(), L)) || (top_t && top_t != e->lay.top_t) ||
        (top_st && top_st != e->lay.top_st) || (top_m && top_m != e->lay.top_m) || (sL && sL != e->lay.sL)) {
        delete e;
        return nullptr;
    }
    const double *wv = w ? w : e->lay.w.data();
    // a test run alone spreads each pass over the SMs (shape and column-group width chosen for
    // latency); a batch slot takes the throughput shape and the widest groups
    const unsigned top_digits = e->lay.L - e->lay.top_t;
    unsigned min_bits = 64;
    for (uint8_t b : e->lay.bits) min_bits = b < min_bits ? b : min_bits;
    if (throughput) {
        uint32_t R = 0;
        if (throughput_group(L / 2, min_bits, top_digits, R, e->G)) e->plan = get_plan(L, R);
    } else {
        int nsm = 1;
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
        uint32_t R = 0, C = 0;
        int G = kGroup;
        if (choose_latency_shape(L / 2, nsm, min_bits, top_digits, R, C, G)) {
            e->G = G;
            e->plan = get_plan(L, R);
        }
    }
    if (!e->plan || top_digits > 2 * (uint32_t)e->G) {
        delete e;
        return nullptr;
    }
    const LengthPlan &P = *e->plan;
    const uint32_t H = P.H;
    e->NG = P.C / e->G;
    // the chain's words after the exponents and emax, aligned; its flags after those
    const size_t chain_at = ((size_t)P.R + 3) & ~(size_t)1, flags_at = (chain_at + sizeof(ChainCtl) / sizeof(int) + 7) & ~(size_t)7;
    bool good = ok(e, cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking)) &&
                dalloc(e, &e->d_desc, 2) && dalloc(e, &e->d_work, P.pairs.size() + e->NG) &&
                dalloc(e, &e->d_bits, 2 * (size_t)L) && dalloc(e, &e->d_w, L) && dalloc(e, &e->d_osc, L) &&
                dalloc(e, &e->d_idig, L) && dalloc(e, &e->d_dig, L) && dalloc(e, &e->d_dig2, L) &&
                dalloc(e, &e->d_eq, 1) && ok(e, cudaMallocHost((void **)&e->h_eq, sizeof(int))) &&
                dalloc(e, &e->d_slot, (size_t)e->NG * P.R) &&
                dalloc(e, &e->d_maxerr, 1) && dalloc(e, &e->d_rexp, flags_at + (size_t)e->NG * kFlagWords) &&
                ok(e, cudaMallocHost((void **)&e->h_dig, (size_t)L * sizeof(long long))) &&
                ok(e, cudaMallocHost((void **)&e->h_err, 2 * sizeof(unsigned long long)));
    if (good) {
        std::vector<int64_t> wfix(L), osc(L), idig(L);
        std::vector<uint8_t> widths(e->lay.bits);  // then TestDesc::segbits
        widths.resize(2 * (size_t)L);
        const uint32_t G = (uint32_t)e->G;
        // k / 4H and 1 / R as m 2^e with m in [1/2, 1)
        const double ms = std::frexp((double)k / (4.0 * H), &e->desc.osc_exp);
        const double mi = std::frexp(1.0 / P.R, &e->desc.idig_exp);
        for (uint32_t j = 0, r = 0, c = 0; j < L; j++) {
            wfix[2 * (c * P.R + r) + j % 2] = (int64_t)(wv[j] * 0x1p61);
            widths[L + 2 * (c / G * G * P.R + r * G + c % G) + j % 2] = e->lay.bits[j];
            if (j % 2 && ++c == P.C) {
                c = 0;
                r++;
            }
            const double inv = 1.0 / wv[j];
            osc[j] = fixed_ratio(ms, wv[j], inv);
            idig[j] = fixed_ratio(mi, wv[j], inv);
        }
        e->h_timeout = reinterpret_cast<unsigned *>(e->h_err + 1);
        *e->h_timeout = 0;
        e->d_chain = reinterpret_cast<ChainCtl *>(e->d_rexp + chain_at);
        e->d_flags = reinterpret_cast<unsigned *>(e->d_rexp + flags_at);
        std::vector<int> words(flags_at + (size_t)e->NG * kFlagWords - P.R, 0);  // from emax on
        words[0] = words[1] = INT_MIN;
        const ChainCtl chain0{0, 0, e->h_timeout};
        std::memcpy(words.data() + chain_at - P.R, &chain0, sizeof chain0);
        std::vector<WorkItem> work;
        for (size_t i = 0; i < P.pairs.size(); i++) work.push_back({0, (int)i});
        for (uint32_t g = 0; g < e->NG; g++) work.push_back({0, (int)g});
        good = ok(e, cudaMemcpy(e->d_bits, widths.data(), 2 * (size_t)L, cudaMemcpyHostToDevice)) &&
               ok(e, cudaMemcpy(e->d_w, wfix.data(), L * sizeof(int64_t), cudaMemcpyHostToDevice)) &&
               ok(e, cudaMemcpy(e->d_osc, osc.data(), L * sizeof(int64_t), cudaMemcpyHostToDevice)) &&
               ok(e, cudaMemcpy(e->d_idig, idig.data(), L * sizeof(int64_t), cudaMemcpyHostToDevice)) &&
               ok(e, cudaMemcpy(e->d_work, work.data(), work.size() * sizeof(WorkItem), cudaMemcpyHostToDevice)) &&
               ok(e, cudaMemset(e->d_maxerr, 0, sizeof(unsigned long long))) &&
               ok(e, cudaMemcpy(e->d_rexp + P.R, words.data(), words.size() * sizeof(int), cudaMemcpyHostToDevice)) &&
               ok(e, cudaMemset(e->d_slot, 0, (size_t)e->NG * P.R * sizeof(long long)));
    }
    if (good) {
        TestDesc &d = e->desc;
        d.L = (int)L;
        d.H = (int)H;
        d.R = (int)P.R;
        d.C = (int)P.C;
        d.NG = (int)e->NG;
        d.G = e->G;
        d.rp = P.rp;
        d.cp = P.cp;
        // narrow digits: the same stages and tables, scaled elsewhere on the way
        if (*std::max_element(e->lay.bits.begin(), e->lay.bits.end()) <= kNarrowBits) {
            make_fft_plan((int)P.C, d.rp, true);
            make_fft_plan((int)P.R, d.cp, true);
        }
        d.twr = P.twr;
        d.twc = P.twc;
        d.t4 = P.t4;
        d.sw = P.sw;
        d.pairs = P.dpairs;
        d.npairs = (int)P.pairs.size();
        d.bits = e->d_bits;
        d.segbits = e->d_bits + L;
        d.w = e->d_w;
        d.osc = e->d_osc;
        d.idig = e->d_idig;
        d.dig = e->d_dig;
        d.slot = e->d_slot;
        d.maxerr = e->d_maxerr;
        d.rexp = e->d_rexp;
        d.emax = e->d_rexp + P.R;
        d.pitch = (int)P.C;
        d.digit_bits = digit_bits(e->lay, e->G);
        d.k = k;
        d.k_inv = ~0ull / k;
        d.top_t = (int)e->lay.top_t;
        d.top_m = (int)e->lay.top_m;
        d.top_shift = (int)(e->lay.sL - e->lay.top_st);
        d.nadd = 0;
        d.x = nullptr;
        d.y = nullptr;
        d.count = 1 << 30;
        d.err_every = 1;
        good = upload_desc(e) && ok(e, cudaStreamSynchronize(e->stream));
        LaunchSet &s = e->ls;
        s.stream = e->stream;
        s.tests = e->d_desc;
        s.rows = e->d_work;
        s.nrows = (int)P.pairs.size();
        s.cols = e->d_work + P.pairs.size();
        s.ncols = (int)e->NG;
        s.grid_rows = s.nrows;
        s.grid_cols = s.ncols;
        s.row_smem_per_lane = (size_t)P.C * sizeof(longlong2);
        s.col_smem = 2 * (size_t)P.R * e->G * sizeof(longlong2);
        s.G = e->G;
        // twiddles of both plans, split twiddles of a row; t4, osc, w, digits of a column group, its widths
        s.table_smem = ((size_t)2 * P.C + P.R + 4 * (size_t)P.R * e->G) * 16 + ((size_t)2 * P.R * e->G + 15) / 16 * 16;
        good = good && ok(e, cudaDeviceGetAttribute(&e->nsm, cudaDevAttrMultiProcessorCount, device)) &&
               kernels_prepare(s.row_smem_per_lane * 6, s.col_smem, chain_smem(s, e->nsm)) == 0;
        e->chain_cluster = good && chain_in_cluster(s, e->nsm);
        e->chain_grid = good ? chain_grid(s, e->nsm, e->chain_cluster) : 0;
        e->chain_steps = std::max<uint64_t>(32, std::min<uint64_t>(512, kChainDigits / L));
        good = e->chain_grid > 0;
    }
    if (!good) {
        release(e);
        delete e;
        return nullptr;
    }
    return e;
}

// the digits of x into the pinned staging buffer e->h_dig; waits
int kc_fetch_digits(kc_engine *e, const double *x) {
    DeviceGuard dg(e->device);
    launch_col_digits(e->ls, (const double2 *)x);
    if (!check_launch(e)) return e->err;
    if (!ok(e, cudaMemcpyAsync(e->h_dig, e->d_dig, e->lay.L * sizeof(long long), cudaMemcpyDeviceToHost, e->stream)) ||
        !wait_queue(e))
        return e->err;
    return 0;
}

extern "C" {

void kc_engine_free(kc_engine *e) {
    if (!e) return;
    DeviceGuard dg(e->device);
    cudaStreamSynchronize(e->stream);
    {
        Device &dev = g_devices[e->device];
        std::lock_guard<std::mutex> lock(dev.mu);
        dev.busy.erase(std::remove(dev.busy.begin(), dev.busy.end(), e), dev.busy.end());
    }
    release(e);
    delete e;
}

size_t kc_num_doubles(const kc_engine *e) { return e->lay.L; }

double *kc_num_alloc(kc_engine *e) {
    DeviceGuard dg(e->device);
    double *p = nullptr;
    if (!ok(e, cudaMalloc((void **)&p, (size_t)e->lay.L * sizeof(double)))) return nullptr;
    if (!ok(e, cudaMemsetAsync(p, 0, (size_t)e->lay.L * sizeof(double), e->stream))) {
        cudaFree(p);
        return nullptr;
    }
    return p;
}

void kc_num_free(kc_engine *e, double *x) {
    if (!x) return;
    DeviceGuard dg(e->device);
    cudaStreamSynchronize(e->stream);
    cudaFree(x);
}

int kc_from_digits(kc_engine *e, double *x, const int64_t *digits) {
    DeviceGuard dg(e->device);
    const size_t L = e->lay.L;
    if (!wait_queue(e)) return e->err;  // staging buffer reuse
    std::memcpy(e->h_dig, digits, L * sizeof(long long));
    uint64_t mag = 0;  // bit length of the largest digit
    for (size_t j = 0; j < L; j++) mag |= (uint64_t)(digits[j] ^ (digits[j] >> 63));
    const int bits = mag ? 64 - __builtin_clzll(mag) : 1;
    if (!ok(e, cudaMemcpyAsync(e->d_dig, e->h_dig, L * sizeof(long long), cudaMemcpyHostToDevice, e->stream)))
        return e->err;
    launch_col_forward(e->ls, (double2 *)x, false, 0, bits);
    return check_launch(e) ? 0 : e->err;
}

int kc_to_digits(kc_engine *e, const double *x, int64_t *digits) {
    if (kc_fetch_digits(e, x)) return e->err;
    std::memcpy(digits, e->h_dig, e->lay.L * sizeof(long long));
    return 0;
}

int kc_equal(kc_engine *e, const double *a, const double *b) {
    DeviceGuard dg(e->device);
    if (a == b) return 1;
    kc_queue_equal(e, e->stream, a, b, e->d_eq);
    if (!check_launch(e) ||
        !ok(e, cudaMemcpyAsync(e->h_eq, e->d_eq, sizeof(int), cudaMemcpyDeviceToHost, e->stream)) || !wait_queue(e))
        return e->err;
    if (*e->h_eq != 2) return *e->h_eq;
    // the device carry did not settle within its bounds: compare canonical limbs on the host
    std::vector<uint64_t> la(e->lay.nlimbs), lb(e->lay.nlimbs);
    if (kc_get_limbs(e, a, la.data()) || kc_get_limbs(e, b, lb.data())) return e->err ? e->err : -1;
    return la == lb ? 1 : 0;
}

int kc_square(kc_engine *e, double *x, uint64_t count) {
    DeviceGuard dg(e->device);
    if (e->add_c && set_addend(e, 0)) return e->err ? e->err : -1;
    return square_many(e, (double2 *)x, count);
}

int kc_square_add(kc_engine *e, double *x, uint64_t count, int64_t c) {
    DeviceGuard dg(e->device);
    if (set_addend(e, c)) return e->err ? e->err : -1;
    return square_many(e, (double2 *)x, count);
}

int kc_mul(kc_engine *e, double *x, const double *y) {
    DeviceGuard dg(e->device);
    if (e->add_c && set_addend(e, 0)) return e->err ? e->err : -1;
    return product(e, (double2 *)x, (const double2 *)y);
}

int kc_copy(kc_engine *e, double *dst, const double *src) {
    DeviceGuard dg(e->device);
    if (dst == src) return 0;
    return ok(e, cudaMemcpyAsync(dst, src, (size_t)e->lay.L * sizeof(double), cudaMemcpyDeviceToDevice, e->stream))
               ? 0
               : e->err;
}

int kc_add(kc_engine *e, double *x, const double *y) {
    DeviceGuard dg(e->device);
    launch_elementwise(e->stream, (double2 *)x, (const double2 *)y, e->lay.L / 2, 1);
    return check_launch(e) ? 0 : e->err;
}

int kc_sub(kc_engine *e, double *x, const double *y) {
    DeviceGuard dg(e->device);
    launch_elementwise(e->stream, (double2 *)x, (const double2 *)y, e->lay.L / 2, 2);
    return check_launch(e) ? 0 : e->err;
}

double kc_maxerr(kc_engine *e) {
    DeviceGuard dg(e->device);
    if (e->err) return 1.0;
    if (!ok(e, cudaMemcpyAsync(e->h_err, e->d_maxerr, sizeof(unsigned long long), cudaMemcpyDeviceToHost, e->stream)) ||
        !wait_queue(e))
        return 1.0;
    double v;
    std::memcpy(&v, e->h_err, sizeof v);
    return v;
}

void kc_reset_maxerr(kc_engine *e) {
    DeviceGuard dg(e->device);
    ok(e, cudaMemsetAsync(e->d_maxerr, 0, sizeof(unsigned long long), e->stream));
}

void kc_set_roundoff_check(kc_engine *e, uint32_t every) {
    e->err_every = every ? every : 1;
    if (e->desc.err_every != (int)e->err_every) {
        DeviceGuard dg(e->device);
        e->desc.err_every = (int)e->err_every;  // read by chains and graphs
        upload_desc(e);
    }
}

int kc_error(const kc_engine *e) { return e->err; }

int kc_sync(kc_engine *e) {
    DeviceGuard dg(e->device);
    wait_queue(e);
    return e->err;
}

void *kc_stream(kc_engine *e) { return (void *)e->stream; }

void kc_shape(const kc_engine *e, uint32_t *R, uint32_t *C) {
    if (R) *R = e->plan->R;
    if (C) *C = e->plan->C;
}

int kc_group_width(const kc_engine *e) { return e->G; }

int kc_engine_wait_selftest(kc_engine *e, uint64_t wait_cycles) {
    DeviceGuard dg(e->device);
    int nsm = 0;
    if (!ok(e, cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, e->device))) return e->err;
    // the engine's column items without its row items: every column item waits for row items
    // that are not in the queue, so every wait runs out
    LaunchSet s = e->ls;
    s.nrows = 0;
    s.nrows_dev = nullptr;
    s.ncols_dev = nullptr;
    const int grid = squarings_grid(s, nsm);
    const size_t bytes = (kFlowDone + 1) * sizeof(unsigned);
    unsigned *flow = nullptr;
    if (!ok(e, cudaMalloc((void **)&flow, bytes))) return e->err;
    int rc = -1;
    unsigned timed_out = 0;
    if (ok(e, cudaMemsetAsync(flow, 0, bytes, e->stream)) &&
        launch_squarings(s, flow, 0, 1, grid, (long long)wait_cycles) == 0 && check_launch(e) &&
        ok(e, cudaMemcpyAsync(&timed_out, flow + kFlowTimeout, sizeof timed_out, cudaMemcpyDeviceToHost, e->stream)) &&
        ok(e, cudaStreamSynchronize(e->stream)))
        rc = timed_out ? 1 : 0;
    else if (e->err)
        rc = e->err;
    cudaStreamSynchronize(e->stream);
    cudaFree(flow);
    if (rc != 1) return rc;
    // a chain whose CTAs wait for one arrival more than there are, on a scratch number
    ChainCtl c0{0, 0, e->h_timeout}, c1{};
    ChainCtl *ctl = nullptr;
    double *x = kc_num_alloc(e);
    const int emax0 = INT_MIN;
    rc = -1;
    if (x && ok(e, cudaMalloc((void **)&ctl, sizeof(ChainCtl))) &&
        ok(e, cudaMemcpyAsync(ctl, &c0, sizeof c0, cudaMemcpyHostToDevice, e->stream)) &&
        ok(e, launch_chain(e->ls, e->nsm, e->chain_grid, false, (double2 *)x, 0, 1, ctl, 1, e->d_flags, e->chained, (long long)wait_cycles)) &&
        ok(e, cudaMemcpyAsync(&c1, ctl, sizeof c1, cudaMemcpyDeviceToHost, e->stream)) &&
        ok(e, cudaMemcpyAsync(e->d_rexp + e->plan->R, &emax0, sizeof emax0, cudaMemcpyHostToDevice, e->stream)) &&
        ok(e, cudaStreamSynchronize(e->stream)))
        rc = c1.timeout && *(volatile unsigned *)e->h_timeout ? 1 : 0;
    else if (e->err)
        rc = e->err;
    *e->h_timeout = 0;
    cudaFree(ctl);
    if (x) kc_num_free(e, x);
    return rc;
}

}  // extern "C"
