// Device building blocks: 64-bit fixed-point complex arithmetic and the mixed-radix transform
// over shared memory that the row and column passes run.
//
// Why fixed point.  GB300 issues an FP64 instruction once per 64-76 clocks per SM sub-partition,
// but a 64-bit integer add every two and a 32 x 32 -> 64-bit multiply every four (measured with
// dependent chains at full occupancy).  A complex product of 64-bit fixed-point numbers is
// 12 multiplies and as many adds, about 65 issue clocks, where its FP64 form costs about 280; a
// complex add costs 4 instead of about 150.  The squaring was bound by the FP64 pipe (102 FP64
// instructions per point), so the transforms run in integers, and at no loss of precision: a
// value keeps up to 62 bits under an exponent shared by the row pair or the test.
//
// Representation.  A transform holds complex numbers as two int64.  Its input is scaled so that
// every modulus is at most 2^62 / growth (FftPlan::headroom), where growth bounds what the stages
// can add up, so no data can overflow; what is scaled up again on the way stays below 2^63 by the
// growth of the stages that are left (FftPlan::renorm).  Twiddles are scaled by 2^62 and stored as two signed
// 32-bit limbs a component; a twiddle product keeps the upper 64 bits of 128, so it divides by
// 4, which is the growth of a radix-4 butterfly: twiddled radix-4 stages keep the bound, and the
// values lose half a bit a level against the 62 they start from, as random data grow by sqrt(n)
// and the bound by n.
//
// Every transform is decimation in time (twiddles on the inputs of each butterfly) in Stockham's
// order: a stage reads elements n/P apart and writes its outputs where the next stage reads them in
// turn, from one buffer to another.  Input and output are in natural order, reads of a stage are
// consecutive and need no index arithmetic, and the first and the last stage can read and write
// global memory directly.  Forward uses exp(-2 pi i/n), the inverse its conjugate, and both leave
// the factor 2^-FftPlan::scale.
#pragma once

#include <cuda_runtime.h>

#include "device.h"

namespace kg {

// ---- 64-bit fixed point -----------------------------------------------------------------------

// the upper limb of v = hi32(v) 2^32 + lo32(v) with both limbs signed
__device__ __forceinline__ int lo32(long long v) { return (int)v; }
__device__ __forceinline__ int hi32(long long v) { return (int)(v >> 32) + (int)((unsigned)v >> 31); }
// The 64-bit product of two limbs.  Spelled out, so that it is not joined with the add that follows
// to one multiply-add: that one takes 5.2 clocks a warp and sub-partition (10.4 with a single warp to
// issue), the product and the add 4.25 (6.1).
__device__ __forceinline__ long long mulw(int a, int b) {
#ifdef __CUDA_ARCH__
    long long d;
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(d) : "r"(a), "r"(b));
    return d;
#else
    return (long long)a * b;
#endif
}

// Rounding of a sum of cross products to its upper half.  A twiddle of 1 leaves quarters, and a tie
// that always goes up would leave 1/8 of the last place on the same element (index 0) of every row or
// column of a transform, stage after stage: the next transform gathers that on one element.  So the
// direction of ties is drawn per row and column, from the parity of the index's bits, and turned
// from stage to stage: kHalf up, kHalf - 1 down.
constexpr long long kHalf = 0x80000000ll;
__device__ __forceinline__ int parity(int index) { return __popc(index) & 1; }
__device__ __forceinline__ long long half_of(int odd) { return kHalf - odd; }

__device__ __forceinline__ longlong2 cadd(longlong2 a, longlong2 b) { return make_longlong2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ longlong2 csub(longlong2 a, longlong2 b) { return make_longlong2(a.x - b.x, a.y - b.y); }
// a + i b and a - i b
__device__ __forceinline__ longlong2 caddi(longlong2 a, longlong2 b) { return make_longlong2(a.x - b.y, a.y + b.x); }
__device__ __forceinline__ longlong2 csubi(longlong2 a, longlong2 b) { return make_longlong2(a.x + b.y, a.y - b.x); }
__device__ __forceinline__ longlong2 cshl(longlong2 a, int s) { return make_longlong2(a.x << s, a.y << s); }

// a / 2^s, rounded down after adding less than one last place, as the other component's last bits
// say: no bias.
__device__ __forceinline__ longlong2 cshr(longlong2 a, int s) {
    const long long m = (1ll << s) - 1;
    return make_longlong2((a.x + (a.y & m)) >> s, (a.y + (a.x & m)) >> s);
}
// a 2^s, s of either sign; the caller knows that a left shift does not overflow
__device__ __forceinline__ longlong2 cshift(longlong2 a, int s) {
    return s >= 0 ? cshl(a, s) : cshr(a, min(-s, 60));
}

// v * 2^s, s of either sign; the caller knows that a left shift does not overflow
__device__ __forceinline__ long long shift_by(long long v, int s) {
    return s >= 0 ? v << s : v >> (s < -63 ? 63 : -s);
}

// A real product accumulated as 2^64 p + 2^32 t: the low limbs' product (below a quarter of the
// result's last place, of either sign) is left out.
struct Acc {
    long long p = 0, t;
    __device__ __forceinline__ explicit Acc(long long half = kHalf) : t(half) {}
    __device__ __forceinline__ void mac(int a1, int a0, int b1, int b0) {
        t += mulw(a1, b0);
        t += mulw(a0, b1);
        p += mulw(a1, b1);
    }
    __device__ __forceinline__ long long high() const { return p + (t >> 32); }
    // four times as much, rounded at the last place of that
    __device__ __forceinline__ long long high4() const {
        return (long long)((unsigned long long)p << 2) + ((t - kHalf + (kHalf >> 2)) >> 30);
    }
};

// a * w / 4 and a * conj(w) / 4, w a twiddle {c1, c0, s1, s0} for (c + i s) 2^62
__device__ __forceinline__ longlong2 cmul(longlong2 a, int4 w, long long half) {
    const int x1 = hi32(a.x), x0 = lo32(a.x), y1 = hi32(a.y), y0 = lo32(a.y);
    Acc r(half), i(half);
    r.mac(x1, x0, w.x, w.y);
    r.mac(y1, y0, -w.z, -w.w);
    i.mac(x1, x0, w.z, w.w);
    i.mac(y1, y0, w.x, w.y);
    return make_longlong2(r.high(), i.high());
}
// a * w: cmul without the division by 4
__device__ __forceinline__ longlong2 cmul4(longlong2 a, int4 w) {
    const int x1 = hi32(a.x), x0 = lo32(a.x), y1 = hi32(a.y), y0 = lo32(a.y);
    Acc r, i;
    r.mac(x1, x0, w.x, w.y);
    r.mac(y1, y0, -w.z, -w.w);
    i.mac(x1, x0, w.z, w.w);
    i.mac(y1, y0, w.x, w.y);
    return make_longlong2(r.high4(), i.high4());
}
__device__ __forceinline__ int4 conj_tw(int4 w) { return make_int4(w.x, w.y, -w.z, -w.w); }

// ---- DFTs in registers --------------------------------------------------------------------------

// cos(2 pi r / P) and sin(2 pi r / P) times 2^62, for the odd radices
template <int P>
struct OddRoots;
template <>
struct OddRoots<3> {
    static __device__ constexpr long long c(int r) { return -0x2000000000000000ll; }
    static __device__ constexpr long long s(int r) { return r == 1 ? 0x376cf5d0b09954e7ll : -0x376cf5d0b09954e7ll; }
};
template <>
struct OddRoots<5> {
    static __device__ constexpr long long c(int r) { return r == 1 || r == 4 ? 0x13c6ef372fe94f83ll : -0x33c6ef372fe94f83ll; }
    static __device__ constexpr long long s(int r) {
        const long long v = r == 1 || r == 4 ? 0x3cde1c2688a9febdll : 0x259e4608eab4bbdbll;
        return r > 2 ? -v : v;
    }
};
template <>
struct OddRoots<7> {
    static __device__ constexpr long long c(int r) {
        return r == 1 || r == 6 ? 0x27e741c517dba2d9ll : r == 2 || r == 5 ? -0x0e3dc8718122c135ll : -0x39a9795396b8e1a5ll;
    }
    static __device__ constexpr long long s(int r) {
        const int q = r > 3 ? 7 - r : r;
        const long long v = q == 1 ? 0x320986ea0bbc9617ll : q == 2 ? 0x3e65380ab1d2d1c7ll : 0x1bc4c04d71abc100ll;
        return r > 3 ? -v : v;
    }
};

__device__ __forceinline__ constexpr int limb1(long long v) { return (int)((v + 0x80000000ll) >> 32); }
__device__ __forceinline__ constexpr int limb0(long long v) { return (int)v; }

// Length-P DFT in registers, unnormalised and unscaled.
template <int P, bool INV>
__device__ __forceinline__ void dft(longlong2 *x) {
    if constexpr (P == 2) {
        const longlong2 a = x[0], b = x[1];
        x[0] = cadd(a, b);
        x[1] = csub(a, b);
    } else if constexpr (P == 4) {
        const longlong2 a = cadd(x[0], x[2]), b = csub(x[0], x[2]);
        const longlong2 c = cadd(x[1], x[3]), d = csub(x[1], x[3]);
        x[0] = cadd(a, c);
        x[2] = csub(a, c);
        x[1] = INV ? caddi(b, d) : csubi(b, d);
        x[3] = INV ? csubi(b, d) : caddi(b, d);
    } else {
        // odd P: pair x_m with x_(P-m); y_j = A_j -+ i Z_j, y_(P-j) = A_j +- i Z_j with
        // A_j = x_0 + sum cos(2 pi j m / P) (x_m + x_(P-m)), Z_j = sum sin(..) (x_m - x_(P-m))
        constexpr int h = (P - 1) / 2;
        longlong2 a[h], b[h];
#pragma unroll
        for (int m = 1; m <= h; m++) {
            a[m - 1] = cadd(x[m], x[P - m]);
            b[m - 1] = csub(x[m], x[P - m]);
        }
        const longlong2 x0 = x[0];
        longlong2 y0 = x0;
#pragma unroll
        for (int m = 0; m < h; m++) y0 = cadd(y0, a[m]);
        x[0] = y0;
#pragma unroll
        for (int j = 1; j <= h; j++) {
            Acc ax, ay, zx, zy;
#pragma unroll
            for (int m = 1; m <= h; m++) {
                const int r = (j * m) % P;
                const int c1 = limb1(OddRoots<P>::c(r)), c0 = limb0(OddRoots<P>::c(r));
                const int s1 = limb1(OddRoots<P>::s(r)), s0 = limb0(OddRoots<P>::s(r));
                ax.mac(hi32(a[m - 1].x), lo32(a[m - 1].x), c1, c0);
                ay.mac(hi32(a[m - 1].y), lo32(a[m - 1].y), c1, c0);
                zx.mac(hi32(b[m - 1].x), lo32(b[m - 1].x), s1, s0);
                zy.mac(hi32(b[m - 1].y), lo32(b[m - 1].y), s1, s0);
            }
            const longlong2 A = make_longlong2(x0.x + ax.high4(), x0.y + ay.high4());
            const longlong2 Z = make_longlong2(zx.high4(), zy.high4());
            x[j] = INV ? caddi(A, Z) : csubi(A, Z);
            x[P - j] = INV ? csubi(A, Z) : caddi(A, Z);
        }
    }
}

// a / 4, a half rounded as `half` (half_of) says
__device__ __forceinline__ longlong2 quarter(longlong2 a, long long half) {
    const long long k = half - (kHalf - 2);
    return make_longlong2((a.x + k) >> 2, (a.y + k) >> 2);
}

// How a pass reads the tables: in global memory (the read-only path), or wherever they are (the chain
// keeps its own slices in shared memory); and the digits that the first half of a column pass left for
// the second one, which another CTA may have written unless the chain says otherwise.
struct GlobalTables {
    template <class V>
    static __device__ __forceinline__ V load(const V *p) {
        return __ldg(p);
    }
    template <class V>
    static __device__ __forceinline__ V load_own(const V *p) {
        return __ldcg(p);
    }
};
struct AnyTables {
    template <class V>
    static __device__ __forceinline__ V load(const V *p) {
        return *p;
    }
    template <class V>
    static __device__ __forceinline__ V load_own(const V *p) {
        return *p;
    }
};

// One radix-P butterfly of a stage with twiddle records w^t, t = 1..P-1 (tw).  UNIT: the stage of
// span 1, whose twiddles are 1.  A twiddled butterfly of radix 3, 4, 5 or 7 divides by 4, the others
// do not scale.
template <int P, bool INV, bool UNIT>
__device__ __forceinline__ void butterfly(longlong2 *x, const int4 *tw, long long half) {
    if constexpr (!UNIT) {
        if constexpr (P == 2) {
            const int4 w = tw[0];  // unscaled
            x[1] = cmul4(x[1], INV ? conj_tw(w) : w);
        } else {
            x[0] = quarter(x[0], half);
#pragma unroll
            for (int t = 1; t < P; t++) {
                const int4 w = tw[t - 1];
                x[t] = cmul(x[t], INV ? conj_tw(w) : w, half);
            }
        }
    }
    dft<P, INV>(x);
}

// One stage over 2^LG interleaved sequences, element e of sequence l at (e << LG) + l of the buffers.
// ld(at, e, l) gives the element (at: its index in the source), st(at, e, l, v) takes the result (at:
// its index in the destination).  Bit l of `odd` draws the rounding of sequence l (half_of).
// The loads come first: ld only reads, cook(v, e, l) makes the element of what it read, and pre(e, l)
// reads what st will need besides.  Read where they are used, the first stage of a column inverse waited
// for its P loads from L2 one after the other, and the last one for its P scales: at 256 tests of
// n = 300000 to 700000 the column inverse took 0.133 ms, and 0.100 ms so; the forward 0.096 and 0.087.
template <int P, int LG, bool INV, bool FIRST, class TAB, class LD, class COOK, class PRE, class ST>
__device__ __forceinline__ void run_stage(int n, int span, unsigned magic, const int4 *tw, unsigned odd,
                                          LD &&ld, COOK &&cook, PRE &&pre, ST &&st) {
    const int np = n / P, total = np << LG;
    for (int i = threadIdx.x; i < total; i += blockDim.x) {
        const int l = i & ((1 << LG) - 1), e = i >> LG;
        const int blk = FIRST ? e : (int)(((unsigned long long)(unsigned)e * magic) >> 32);  // e / span
        const int k = FIRST ? 0 : e - blk * span;
        const int o = e + blk * (P - 1) * span;
        int4 w[FIRST || P == 1 ? 1 : P - 1];
        if constexpr (!FIRST) {
#pragma unroll
            for (int t = 0; t < P - 1; t++) w[t] = TAB::load(tw + k * (P - 1) + t);
        }
        decltype(pre(0, 0)) ahead[P];
#pragma unroll
        for (int t = 0; t < P; t++) ahead[t] = pre(o + t * span, l);
        decltype(ld(0, 0, 0)) in[P];
#pragma unroll
        for (int t = 0; t < P; t++) in[t] = ld(i + t * total, e + t * np, l);
        longlong2 x[P];
#pragma unroll
        for (int t = 0; t < P; t++) x[t] = cook(in[t], e + t * np, l);
        if constexpr (P > 1) butterfly<P, INV, FIRST>(x, w, half_of((odd >> l) & 1));
#pragma unroll
        for (int t = 0; t < P; t++) st((((o + t * span) << LG) + l), o + t * span, l, x[t], ahead[t]);
    }
}

// The stage of radix p; the last stage of a short transform may have radix 1.
template <int LG, bool INV, bool FIRST, bool LAST, class TAB, class LD, class COOK, class PRE, class ST>
__device__ __forceinline__ void dispatch_stage(int n, const FftStage &g, const int4 *tw, unsigned odd, LD &&ld, COOK &&cook, PRE &&pre, ST &&st) {
    const int p = g.radix, span = g.span;
    const unsigned magic = g.magic;
    tw += g.off;
#define KG_STAGE(P)                                                          \
    case P:                                                                  \
        run_stage<P, LG, INV, FIRST, TAB>(n, span, magic, tw, odd, ld, cook, pre, st);       \
        break;
    if (p == 4) {
        run_stage<4, LG, INV, FIRST, TAB>(n, span, magic, tw, odd, ld, cook, pre, st);
        return;
    }
    switch (p) {
        KG_STAGE(2)
        KG_STAGE(3)
        KG_STAGE(5)
        KG_STAGE(7)
    default:
        if constexpr (LAST) run_stage<1, LG, INV, FIRST, TAB>(n, span, magic, tw, odd, ld, cook, pre, st);
        break;
    }
#undef KG_STAGE
}

}  // namespace kg
