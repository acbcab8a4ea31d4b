// The zero test of two numbers, element-wise operations, and the FP64 probes (see device.h for the
// data layout; the pass kernels are in rows.cu, columns_inverse.cu and columns_forward.cu).
#include <cuda_runtime.h>

#include <mutex>

#include "kernels.h"
#include "passes.cuh"

namespace kg {

// Fold of the top region held in dig[top_t..L-1] plus the carry cy at 2^{s_L}
// (reference src/ctx.c:345-375); returns the amount for digit 0.
__device__ __forceinline__ long long fold_top(const TestDesc &T, long long *dig, long long cy) {
    const int L = T.L, t = T.top_t;
    __int128 H = (__int128)cy << T.top_shift;
    int pos = 0;
    for (int j = t; j < L; j++) {
        H += (__int128)dig[j] << pos;
        pos += T.bits[j];
    }
    const int m = T.top_m;
    const __int128 K = (__int128)T.k;
    __int128 lo = H & (((__int128)1 << m) - 1);
    __int128 hi = H >> m;
    __int128 rem;
    __int128 q = floor_div_inv(hi, T.k, T.k_inv, rem);
    __int128 top = lo + (rem << m);
    const __int128 span = K << m;
    if (2 * top >= span) {
        top -= span;
        q += 1;
    }
    for (int j = t; j + 1 < L; j++) {
        const int b = T.bits[j];
        __int128 qq = (top + ((__int128)1 << (b - 1))) >> b;
        dig[j] = (long long)(top - (qq << b));
        top = qq;
    }
    if (t < L) dig[L - 1] = (long long)top;
    return (long long)q;
}

// Zero test of a - b modulo N for two digit vectors of one test (the digits of two numbers, as
// k_col_digits leaves them): the Gerbicz check's comparison d == x0 * t^(2^B) and the tail's
// x == t, done where the numbers live.  The reference compares canonical limbs on the host
// (src/prp.c:291-296 and :470-474, via kite_get_limbs).
//
// The difference e = a - b is carried exactly as a whole number: the low digits (below top_t)
// are balanced in kEqualThreads chunks, each chunk's carry-out moving to the next chunk round
// by round until none is left; the top region (digits top_t..L-1 with the carry out of the low
// digits) is folded by k*2^n == 1 and re-centred (fold_top), and the fold's amount for digit 0
// rippled in the same way.  Afterwards every low digit is balanced and the top region lies in
// [-k 2^m/2, k 2^m/2), so |e| < N and e == 0 (mod N) exactly when every digit is zero.
// *flag = 1 (equal), 0 (not equal), or 2 when the carry did not settle within its bounds (the
// caller then compares on the host).  a is overwritten; one CTA per test.
constexpr int kEqualThreads = 512;

__device__ __forceinline__ long long ripple(long long *e, const uint8_t *bits, int j0, int j1, long long c) {
    for (int j = j0; j < j1 && c; j++) {
        const int b = bits[j];
        const long long v = e[j] + c;
        c = (v + (1ll << (b - 1))) >> b;
        e[j] = v - (c << b);
    }
    return c;
}

__global__ void __launch_bounds__(kEqualThreads) k_equal_mod_n(const TestDesc *__restrict__ tests, int test,
                                                               long long *__restrict__ a,
                                                               const long long *__restrict__ b, int *flag) {
    __shared__ long long s_out[kEqualThreads];  // carry out of chunk i, not yet moved on
    __shared__ long long s_in0;                  // carry into chunk 0 (from the fold)
    __shared__ long long s_top;                  // carry out of the low digits into the top region
    __shared__ int s_more;
    const TestDesc &T = tests[test];
    const int L = T.L, t = T.top_t, tid = threadIdx.x, nt = blockDim.x;
    for (int j = tid; j < L; j += nt) a[j] -= b[j];
    // chunks of the low digits [0, t): nch chunks of cs digits (the last one may be shorter)
    const int cs = (t + nt - 1) / nt, nch = (t + cs - 1) / cs;
    const int j0 = min(t, tid * cs), j1 = min(t, j0 + cs);
    if (tid == 0) {
        s_in0 = 0;
        s_top = 0;
    }
    __syncthreads();
    // every chunk balanced on its own, from no carry
    long long c = 0;
    if (tid < nch) {
        for (int j = j0; j < j1; j++) {
            const int bw = T.bits[j];
            const long long v = a[j] + c;
            c = (v + (1ll << (bw - 1))) >> bw;
            a[j] = v - (c << bw);
        }
        s_out[tid] = c;
    }
    int settled = 0;
    for (int pass = 0; pass < 64; pass++) {
        // move the carries on until every chunk has absorbed its carry-in; a carry advances at
        // least one chunk per round, so nch + 1 rounds always suffice
        int quiet = 0;
        for (int round = 0; round <= nch + 1; round++) {
            __syncthreads();
            const long long cin = tid == 0 ? s_in0 : (tid < nch ? s_out[tid - 1] : 0);
            const long long to_top = s_out[nch - 1];
            __syncthreads();
            if (tid == 0) {
                s_in0 = 0;
                s_top += to_top;
            }
            long long r = 0;
            if (tid < nch) {
                r = ripple(a, T.bits, j0, j1, cin);
                s_out[tid] = r;
            }
            if (!__syncthreads_or(r != 0)) {
                quiet = 1;
                break;
            }
        }
        if (!quiet) break;  // not settled within the bound: undetermined
        // fold the top region (always once, again whenever a carry reached it)
        if (tid == 0) {
            const long long add = s_top;
            s_top = 0;
            s_more = 0;
            if (pass == 0 || add) {
                long long q;
                if (t < L) {
                    a[t] += add;
                    q = fold_top(T, a, 0);
                } else {
                    q = fold_top(T, a, add);
                }
                s_in0 = q;
                s_more = q != 0;
            }
        }
        __syncthreads();
        if (!s_more) {
            settled = 1;
            break;
        }
    }
    int nonzero = 0;
    for (int j = tid; j < L; j += nt) nonzero |= a[j] != 0;
    nonzero = __syncthreads_or(nonzero);
    if (tid == 0) *flag = settled ? (nonzero ? 0 : 1) : 2;
}

// x op= y element-wise over n complex values: 0 copy, 1 add, 2 sub
__global__ void k_elementwise(double2 *x, const double2 *y, size_t n, int op) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const double2 b = y[i];
        if (op == 0) {
            x[i] = b;
        } else {
            const double2 a = x[i];
            x[i] = op == 1 ? make_double2(a.x + b.x, a.y + b.y) : make_double2(a.x - b.x, a.y - b.y);
        }
    }
}

// ---- host launch wrappers --------------------------------------------------------------------

// The limit is a property of each kernel in the device's context, shared by every engine and
// batch of the process, so it only ever grows: lowering it for a small length would make later
// launches (or captured graphs) of a longer length fail.
int kernels_prepare(size_t row_smem, size_t col_smem, size_t chain_smem) {
    static std::mutex mu;
    static size_t row_hw[kMaxDevices] = {}, col_hw[kMaxDevices] = {}, sq_hw[kMaxDevices] = {};
    static size_t chain_hw[kMaxDevices] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return -1;
    std::lock_guard<std::mutex> lock(mu);
    int rc = 0;
    if (row_smem > row_hw[dev]) {
        rc |= rows_set_smem(row_smem);
        if (!rc) row_hw[dev] = row_smem;
    }
    if (col_smem > col_hw[dev]) {
        rc |= col_inverse_set_smem(col_smem);
        rc |= col_forward_set_smem(col_smem);
        if (!rc) col_hw[dev] = col_smem;
    }
    const size_t sq_smem = squarings_smem(row_smem, col_smem);
    if (sq_smem > sq_hw[dev]) {
        const int r2 = squarings_set_smem(sq_smem);
        if (!r2) sq_hw[dev] = sq_smem;
        rc |= r2;
    }
    if (chain_smem > chain_hw[dev]) {
        const int r2 = chain_set_smem(chain_smem);
        if (!r2) chain_hw[dev] = chain_smem;
        rc |= r2;
    }
    return rc;
}

void launch_equal(cudaStream_t st, const TestDesc *tests, int test, long long *a, const long long *b, int *flag) {
    k_equal_mod_n<<<1, kEqualThreads, 0, st>>>(tests, test, a, b, flag);
}

void launch_elementwise(cudaStream_t st, double2 *x, const double2 *y, size_t n, int op) {
    int grid = (int)((n + 255) / 256);
    if (grid > 4096) grid = 4096;
    k_elementwise<<<grid, 256, 0, st>>>(x, y, n, op);
}

// Dependent DFMA chains: 8 independent chains per thread so the pipe, not latency, limits.
__global__ void k_fp64_probe(double *out, int iters) {
    double a0 = threadIdx.x * 1e-9, a1 = a0 + 1, a2 = a0 + 2, a3 = a0 + 3;
    double a4 = a0 + 4, a5 = a0 + 5, a6 = a0 + 6, a7 = a0 + 7;
    const double m = 0.999999999, c = 1e-12;
    for (int i = 0; i < iters; i++) {
        a0 = fma(a0, m, c); a1 = fma(a1, m, c); a2 = fma(a2, m, c); a3 = fma(a3, m, c);
        a4 = fma(a4, m, c); a5 = fma(a5, m, c); a6 = fma(a6, m, c); a7 = fma(a7, m, c);
    }
    const double s = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
    if (s > 1e300) out[0] = s;
}

// The probe's variants for kc_fp64_probe_rate: CH independent chains per thread of one FP64
// opcode (0 DFMA, 1 DMUL, 2 DADD).
template <int CH, int OP>
__global__ void k_fp64_probe_var(double *out, int iters) {
    double a[CH];
#pragma unroll
    for (int c = 0; c < CH; c++) a[c] = threadIdx.x * 1e-9 + c;
    const double m = 0.999999999, k = 1e-12;
    for (int i = 0; i < iters; i++) {
#pragma unroll
        for (int c = 0; c < CH; c++) a[c] = OP == 0 ? fma(a[c], m, k) : OP == 1 ? a[c] * m : a[c] + k;
    }
    double s = 0;
#pragma unroll
    for (int c = 0; c < CH; c++) s += a[c];
    if (s > 1e300) out[0] = s;
}

int launch_fp64_probe_var(cudaStream_t st, int grid, int block, int iters, int chains, int op, double *out) {
#define KG_PROBE(CH, OP) k_fp64_probe_var<CH, OP><<<grid, block, 0, st>>>(out, iters)
    if (op < 0 || op > 2) return -1;
    switch (chains * 4 + op) {
    case 4 * 4 + 0: KG_PROBE(4, 0); break;
    case 8 * 4 + 0: KG_PROBE(8, 0); break;
    case 16 * 4 + 0: KG_PROBE(16, 0); break;
    case 8 * 4 + 1: KG_PROBE(8, 1); break;
    case 8 * 4 + 2: KG_PROBE(8, 2); break;
    default: return -1;
    }
#undef KG_PROBE
    return 0;
}

void launch_fp64_probe(cudaStream_t st, int grid, int block, int iters, double *out) {
    k_fp64_probe<<<grid, block, 0, st>>>(out, iters);
}

}  // namespace kg
