// The passes of a product as device functions over one work item (see device.h for the layout,
// fixed_fft.cuh for the arithmetic).  The pass kernels (rows.cu, columns_*.cu) and the persistent kernel
// (squarings.cu) run them.
//
//   rows_item         row pass: forward row transforms of a row pair, real-split square (or
//                     product with a second operand), inverse row transforms.  Reference:
//                     src/fast2p.c:545-617 (pass 2), src/fast2p.c:514-543 (split formulas).
//   col_inverse_item  column pass, first half: conj four-step twiddle, inverse column transform,
//                     unweight and scale, round to nearest, track round-off, add constant digits,
//                     balanced carry within each 2G-digit row segment, fold the top region.  Each
//                     segment's carry-out goes to the next segment's slot.  Reference:
//                     src/fast2p.c:376-451.
//   col_forward_item  column pass, second half: absorb the carry-in (the segment's last digit is
//                     the sink, as src/fast2p.c:404-419), reweight, forward column transform,
//                     twiddle.
//   col_digits_item   the digits of a number: conj twiddle, inverse column transform, unweight,
//                     round.
//
// A number in memory is an array of doubles.  The row pass scales a row pair by the exponent of
// its largest component, and leaves its rows as 64-bit fixed-point numbers with one exponent a
// row (TestDesc::rexp, emax) for the column inverse, their only reader.
#pragma once

#include <climits>

#include "fixed_fft.cuh"
#include "kernels.h"

namespace kg {

// Block-wide words of the item in work.
struct ItemCtl {
    unsigned top[2];    // rows_item: largest upper word of |component|, of x and of y
    unsigned mag[2];    //   OR of the upper words of |component| after the forward transform
    unsigned mag_split; //   after the split
    unsigned mag_out;   //   after the inverse transform
    unsigned mid[3];    //   before FftPlan::renorm: the transforms of x and y, and the inverse
};

// The work item's test descriptor, copied into shared memory.  An item reads the descriptor's
// fields (plans, table pointers, sizes) again at every stage, and from shared memory those
// reads stay off the texture path that the tables' own loads queue on.  Every thread of the
// block calls this after the previous item's last barrier; it ends with a barrier.
__device__ __forceinline__ const TestDesc &stage_desc(const TestDesc *tests, int t, TestDesc *s, ItemCtl *ctl) {
    const int4 *src = reinterpret_cast<const int4 *>(tests + t);
    int4 *dst = reinterpret_cast<int4 *>(s);
    for (int i = threadIdx.x; i < (int)(sizeof(TestDesc) / 16); i += blockDim.x) dst[i] = __ldg(src + i);
    if (threadIdx.x == 0) *ctl = ItemCtl{};  // the thread that reads the previous item's last
    __syncthreads();
    return *s;
}

// Zeroes the words for a new item of the same test.  Every thread of the block calls it after the
// previous item's last barrier.
__device__ __forceinline__ void clear_ctl(ItemCtl *ctl) {
    if (threadIdx.x == 0) *ctl = ItemCtl{};
    __syncthreads();
}

// the upper word of |v|, or one less for a negative v
__device__ __forceinline__ unsigned mag32(long long v) {
    const int h = (int)(v >> 32);
    return (unsigned)(h ^ (h >> 31));
}
__device__ __forceinline__ unsigned mag32(longlong2 v) { return mag32(v.x) | mag32(v.y); }
__device__ __forceinline__ int bit_length(unsigned v) { return 32 - __clz((int)v); }

__device__ __forceinline__ void block_or(unsigned v, unsigned *dst) {
    v = __reduce_or_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0 && v) atomicOr(dst, v);
}
__device__ __forceinline__ void block_max(unsigned v, unsigned *dst) {
    v = __reduce_max_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0 && v) atomicMax(dst, v);
}

// the upper word of |d|'s encoding, which orders doubles by magnitude
__device__ __forceinline__ unsigned top_word(longlong2 d) {
    return max((unsigned)(d.x >> 32) & 0x7fffffffu, (unsigned)(d.y >> 32) & 0x7fffffffu);
}
// e with every |component| < 2^e, for a block whose largest upper word is `top` (0: all zero)
__device__ __forceinline__ int top_exponent(unsigned top) { return (int)(top >> 20) - 1022; }
// keeps scales of numbers that are all zero, or far outside what digits can make, in range
__device__ __forceinline__ int clamp_scale(int s) { return max(-900, min(900, s)); }

struct Nothing {};
__device__ __forceinline__ Nothing nothing_ahead(int, int) { return {}; }
__device__ __forceinline__ longlong2 as_read(longlong2 v, int, int) { return v; }

// The whole transform of 2^LG interleaved sequences: the first stage reads first_ld(at, e, l) and
// writes to `to`, the stages then go back and forth between `to` and `alt`, and the last one
// calls last_st(dst, at, e, l, v, last_pre(e, l)), dst being the buffer it may write to (the value
// returned) and last_pre what it reads from the tables, asked for before the stage's own work.
// Long transforms are scaled up to their largest component once more on the way (FftPlan::renorm,
// *mid a zeroed word of the block) by 2^shift, shift >= 0, set before the last stage: data that gather on
// one element have nothing to scale up and are left as they are.  Ends with a barrier.
template <int LG, bool INV, class TAB, class LD, class COOK, class PRE, class ST>
__device__ __forceinline__ longlong2 *transform(const FftPlan &pl, const int4 *tw, longlong2 *to, longlong2 *alt,
                                                unsigned odd, LD &&first_ld, COOK &&cook, PRE &&last_pre, ST &&last_st, unsigned *mid, int &shift) {
    const int n = pl.n, last = pl.ns - 1, renorm = pl.renorm;
    shift = 0;
    dispatch_stage<LG, INV, true, false, TAB>(n, pl.stage[0], tw, odd, first_ld, cook, nothing_ahead,
                                         [&](int at, int, int, longlong2 v, Nothing) { to[at] = v; });
    __syncthreads();
    for (int i = 1; i < last; i++) {
        odd = ~odd;
        const longlong2 *from = to;
        to = alt;
        alt = const_cast<longlong2 *>(from);
        if (renorm) {
            const int sh = i == renorm ? shift : 0;
            const bool track = i + 1 == renorm;
            unsigned mag = 0;
            dispatch_stage<LG, INV, false, false, TAB>(
                n, pl.stage[i], tw, odd, [&](int at, int, int) { return from[at]; },
                [&](longlong2 v, int, int) { return cshl(v, sh); }, nothing_ahead,
                [&](int at, int, int, longlong2 v, Nothing) {
                    to[at] = v;
                    mag |= mag32(v);
                });
            if (track) block_or(mag, mid);
            __syncthreads();
            if (track) shift = max(0, 29 - bit_length(*mid));  // components below 2^61
        } else {
            dispatch_stage<LG, INV, false, false, TAB>(n, pl.stage[i], tw, odd, [&](int at, int, int) { return from[at]; }, as_read, nothing_ahead,
                                                  [&](int at, int, int, longlong2 v, Nothing) { to[at] = v; });
            __syncthreads();
        }
    }
    dispatch_stage<LG, INV, false, true, TAB>(n, pl.stage[last], tw, ~odd, [&](int at, int, int) { return to[at]; }, as_read, last_pre,
                                         [&](int at, int e, int l, longlong2 v, auto p) { last_st(alt, at, e, l, v, p); });
    __syncthreads();
    return alt;
}

// the double with encoding `bits`, times 2^s, rounded to the nearest integer.  The conversion
// runs on the FP64 pipe, which nothing else in a pass uses.
__device__ __forceinline__ long long to_fixed(long long bits, int s) {
    const int h = (int)(bits >> 32);
    if (((h >> 20) & 0x7ff) + s <= 0) return 0;
    return __double2ll_rn(__longlong_as_double(bits + ((long long)s << 52)));
}
// v 2^s as a double
__device__ __forceinline__ double from_fixed(long long v, int s) {
    const long long bits = __double_as_longlong(__ll2double_rn(v));
    return __longlong_as_double(v ? bits + ((long long)s << 52) : 0);
}

// ---- row pass -----------------------------------------------------------------------------------

// 2^64 (re, im) of a b in units that keep two bits more: 4 a b / 2^64.  Components below 2^61.
__device__ __forceinline__ longlong2 mul4(longlong2 a, longlong2 b) {
    const int a1 = hi32(a.x), a0 = lo32(a.x), b1 = hi32(a.y), b0 = lo32(a.y);
    const int c1 = hi32(b.x), c0 = lo32(b.x), d1 = hi32(b.y), d0 = lo32(b.y);
    Acc r, i;
    r.mac(a1, a0, c1, c0);
    // limbs of -b.y, not the negated limbs of b.y: a limb of -2^31 has no negative
    r.mac(b1, b0, hi32(-b.y), lo32(-b.y));
    i.mac(a1, a0, d1, d0);
    i.mac(b1, b0, c1, c0);
    return make_longlong2(r.high4(), i.high4());
}
__device__ __forceinline__ long long rmul4(long long a, long long b) {
    Acc r;
    r.mac(hi32(a), lo32(a), hi32(b), lo32(b));
    return r.high4();
}
// 4 a^2 / 2^64, as (a.x - a.y)(a.x + a.y) and (2 a.x) a.y.  Components below 2^61.
__device__ __forceinline__ longlong2 sqr4(longlong2 a) {
    return make_longlong2(rmul4(a.x - a.y, a.x + a.y), rmul4(2 * a.x, a.y));
}
// Real-split square or product of the pair of points a, b (components below 2^60), times 2^-62.
//   e = a + conj(b), o = -i (a - conj(b)); 4 V_k = e^2 + w o^2 + 2 i e o,
//   4 V_{H-k} = conj(e^2 + w o^2) + 2 i conj(e o); products use e_x e_y + w o_x o_y and
//   e_x o_y + o_x e_y.
// |e|^2 + |o|^2 = 2 (|a|^2 + |b|^2) < 2^123 bounds the results' moduli by 2^62.
template <bool MUL>
__device__ __forceinline__ void split_pair(longlong2 &a, longlong2 &b, int4 w, longlong2 ya, longlong2 yb) {
    const longlong2 e = make_longlong2(a.x + b.x, a.y - b.y);
    const longlong2 o = make_longlong2(a.y + b.y, b.x - a.x);
    longlong2 X, Y;
    if constexpr (!MUL) {
        X = cadd(sqr4(e), cmul4(sqr4(o), w));
        Y = mul4(e, cadd(o, o));
    } else {
        const longlong2 f = make_longlong2(ya.x + yb.x, ya.y - yb.y);
        const longlong2 g = make_longlong2(ya.y + yb.y, yb.x - ya.x);
        X = cadd(mul4(e, f), cmul4(mul4(o, g), w));
        Y = cadd(mul4(e, g), mul4(o, f));
    }
    a = caddi(X, Y);
    b = make_longlong2(X.x + Y.y, Y.x - X.y);
}

// A row pair of a number into `raw` as it is in memory, lane 0 row k_r and lane 1 row R-k_r, and its
// forward transform, from `raw` to `other` and back.  Returns the buffer with the result; `scale` is
// the power of two it was scaled by, *mag the OR of its components' upper words.  Barriers included.
template <class TAB>
__device__ __forceinline__ longlong2 *rows_forward(const TestDesc &T, int2 pr, const double2 *xd, longlong2 *raw,
                                                   longlong2 *other, unsigned odd, unsigned *top, unsigned *mag,
                                                   unsigned *mid, int &scale) {
    const int C = T.C;
    const FftPlan &pl = T.rp;
    const longlong2 *x = reinterpret_cast<const longlong2 *>(xd);
    const longlong2 *xa = x + (size_t)pr.x * C, *xb = x + (size_t)pr.y * C;
    unsigned t = 0;
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
        const longlong2 a = __ldcg(&xa[c]), b = __ldcg(&xb[c]);
        raw[2 * c] = a;
        raw[2 * c + 1] = b;
        t = max(t, max(top_word(a), top_word(b)));
    }
    block_max(t, top);
    __syncthreads();
    // components 2^s below 2^(62 - headroom), the headroom covering the modulus
    const int s = clamp_scale(62 - pl.headroom - top_exponent(*top));
    unsigned m = 0;
    int shift;
    longlong2 *out = transform<1, false, TAB>(
        pl, T.twr, other, raw, odd,
        [&](int at, int, int) { return raw[at]; },
        [&](longlong2 d, int, int) { return make_longlong2(to_fixed(d.x, s), to_fixed(d.y, s)); },
        nothing_ahead,
        [&](longlong2 *dst, int at, int, int, longlong2 v, Nothing) {
            dst[at] = v;
            m |= mag32(v);
        },
        mid, shift);
    block_or(m, mag);
    __syncthreads();
    scale = s - pl.scale + shift;
    return out;
}

// One row pair of one test.  Ends with a barrier after its last global write but thread 0's own.
template <bool MUL, class TAB>
__device__ __forceinline__ void rows_item(const TestDesc &T, int unit, double2 *xd, const double2 *yd, longlong2 *sm,
                                          ItemCtl &ctl) {
    // shared memory: two buffers of two rows, three for a product
    const int C = T.C;
    const FftPlan &pl = T.rp;
    const int2 pr = T.pairs[unit];
    const bool self = pr.x == pr.y;
    const unsigned odd = parity(pr.x) | parity(pr.y) << 1;  // of the lanes' rows
    int sx, sy;
    longlong2 *X = rows_forward<TAB>(T, pr, xd, sm, sm + 2 * C, odd, &ctl.top[0], &ctl.mag[0], &ctl.mid[0], sx);
    longlong2 *other = X == sm ? sm + 2 * C : sm;
    longlong2 *Y = X;
    if constexpr (MUL) {
        Y = rows_forward<TAB>(T, pr, yd, other, sm + 4 * C, odd, &ctl.top[1], &ctl.mag[1], &ctl.mid[1], sy);
        other = Y == other ? sm + 4 * C : other;
    } else {
        sy = sx;
    }
    // split, in place, on components below 2^60
    const int nx = 28 - bit_length(ctl.mag[0]), ny = MUL ? 28 - bit_length(ctl.mag[1]) : nx;
    const int4 *swp = T.sw + (size_t)pr.x * C;
    const int lb = self ? 0 : 1;
    unsigned mag = 0;
    for (int kc = threadIdx.x; kc < C; kc += blockDim.x) {
        // U_k in row k_r pairs with U_{H-k} in row R-k_r, column C-1-k_c; rows 0 and R/2 pair with
        // themselves: k_c with (C-k_c) mod C, resp. C-1-k_c
        const int kb = self && pr.x == 0 ? (kc ? C - kc : 0) : C - 1 - kc;
        if (self && kb < kc) continue;
        const int ia = 2 * kc, ib = 2 * kb + lb;
        longlong2 a = cshift(X[ia], nx), b = cshift(X[ib], nx);
        longlong2 ya = a, yb = b;
        if constexpr (MUL) {
            ya = cshift(Y[ia], ny);
            yb = cshift(Y[ib], ny);
        }
        split_pair<MUL>(a, b, TAB::load(&swp[kc]), ya, yb);
        X[ia] = a;
        if (!self) {
            X[ib] = b;
        } else {  // the second lane repeats the first: it takes part in the scaling
            X[ia + 1] = a;
            if (kb != kc) X[ib] = X[ib + 1] = b;
        }
        mag |= mag32(a) | mag32(b);
    }
    block_or(mag, &ctl.mag_split);
    __syncthreads();
    // inverse, again scaled to the largest component
    const int ns = 62 - pl.headroom - (32 + bit_length(ctl.mag_split));
    longlong2 *x = reinterpret_cast<longlong2 *>(xd);
    longlong2 *oa = x + (size_t)pr.x * C, *ob = x + (size_t)pr.y * C;
    mag = 0;
    int shift;
    transform<1, true, TAB>(
        pl, T.twr, other, X, odd, [&](int at, int, int) { return X[at]; },
        [&](longlong2 v, int, int) { return cshift(v, ns); }, nothing_ahead,
        [&](longlong2 *, int, int e, int l, longlong2 v, Nothing) {
            if (l && self) return;
            (l ? ob : oa)[e] = v;
            mag |= mag32(v);
        },
        &ctl.mid[2], shift);
    block_or(mag, &ctl.mag_out);
    __syncthreads();
    if (threadIdx.x == 0) {
        // rows = stored 2^re: the scales of x and y, the split's shifts and 2^-62, the inverse's
        const int re = 62 - (sx + nx) - (sy + ny) - (ns - pl.scale + shift);
        T.rexp[pr.x] = re;
        T.rexp[pr.y] = re;
        atomicMax(T.emax, re + 32 + bit_length(ctl.mag_out));
    }
}

// ---- column passes ------------------------------------------------------------------------------

// Where the carries find element l of row r of a group of 2^LG columns: a row's columns are turned by
// the row, so that threads that walk along one row each spread over the banks, as those do that walk
// along the columns (the transform's first or last stage, whose other buffer is in plain order).
template <int LG>
__device__ __forceinline__ int turned(int r, int l) {
    return (r << LG) + (l ^ (r & ((1 << LG) - 1)));
}
// bit l: the parity of the index's bits of column l of group g
__device__ __forceinline__ unsigned odd_columns(int g, int lg) {
    return 0x96u ^ (parity(g << lg) ? ~0u : 0u);  // 0..7 has 1, 2, 4 and 7 odd
}

// x / k and its remainder for x < 2^64 and k_inv = floor((2^64 - 1) / k)
__device__ __forceinline__ unsigned long long div_inv(unsigned long long x, unsigned long long k, unsigned long long k_inv,
                                                      unsigned long long &rem) {
    unsigned long long q = __umul64hi(x, k_inv);
    rem = x - q * k;
    for (; rem >= k; rem -= k) q++;  // at most twice
    return q;
}
// floor(h / k) for a signed 128-bit h, in 32-bit digits of |h|; rem = h - k floor(h / k)
__device__ __forceinline__ __int128 floor_div_inv(__int128 h, unsigned long long k, unsigned long long k_inv, __int128 &rem) {
    const bool neg = h < 0;
    const unsigned __int128 a = neg ? (unsigned __int128)(-h) : (unsigned __int128)h;
    unsigned long long r = 0;
    unsigned __int128 q = div_inv((unsigned long long)(a >> 64), k, k_inv, r);
#pragma unroll
    for (int c = 1; c >= 0; c--) {
        const unsigned long long cur = (r << 32) | (unsigned)(a >> (32 * c));
        q = (q << 32) | div_inv(cur, k, k_inv, r);
    }
    __int128 s = (__int128)q;
    rem = (__int128)r;
    if (neg) {
        s = r ? -s - 1 : -s;
        rem = r ? (__int128)(k - r) : 0;
    }
    return s;
}

// The 2G digit widths of the row segment starting at word j0, packed four to a word, in one
// aligned load: j0 is a multiple of 2G (C is a multiple of G), and the table starts on a
// 256-byte boundary.  seg_width(w, i) unpacks width i.
template <int G>
struct SegWidths {
    unsigned w[2 * G / 4];
};

template <int G, class TAB>
__device__ __forceinline__ SegWidths<G> load_segment_widths(const uint8_t *bits, int j0) {
    static_assert(G == 2 || G == 4 || G == 8, "column groups of 2, 4 or 8");
    SegWidths<G> s;
    if constexpr (G == 8) {
        const uint4 v = TAB::load(reinterpret_cast<const uint4 *>(bits + j0));
        s.w[0] = v.x;
        s.w[1] = v.y;
        s.w[2] = v.z;
        s.w[3] = v.w;
    } else if constexpr (G == 4) {
        const uint2 v = TAB::load(reinterpret_cast<const uint2 *>(bits + j0));
        s.w[0] = v.x;
        s.w[1] = v.y;
    } else {
        s.w[0] = TAB::load(reinterpret_cast<const unsigned *>(bits + j0));
    }
    return s;
}

template <int G>
__device__ __forceinline__ int seg_width(const SegWidths<G> &s, int i) {
    return (int)((s.w[i / 4] >> (8 * (i % 4))) & 0xffu);
}

// Fold of the top region (the last digits of the last segment) plus the carry cy at 2^{s_L}
// (reference src/ctx.c:345-375); returns the amount for digit 0.  One thread of the whole test runs it
// while the others wait, so it reads nothing back from memory and divides by k with its reciprocal.
template <int G>
__device__ __forceinline__ long long fold_segment(const TestDesc &T, const SegWidths<G> &bw, long long (&d)[2 * G],
                                                  long long cy) {
    const int first = 2 * G - (T.L - T.top_t);  // the top region's first digit in the segment
    __int128 H = (__int128)cy << T.top_shift;
    int pos = 0;
#pragma unroll
    for (int i = 0; i < 2 * G; i++)
        if (i >= first) {
            H += (__int128)d[i] << pos;
            pos += seg_width(bw, i);
        }
    const int m = T.top_m;
    const __int128 K = (__int128)T.k, span = K << m;
    const __int128 lo = H & (((__int128)1 << m) - 1);
    __int128 r;
    __int128 q = floor_div_inv(H >> m, T.k, T.k_inv, r);
    __int128 top = lo + (r << m);
    if (2 * top >= span) {
        top -= span;
        q += 1;
    }
#pragma unroll
    for (int i = 0; i < 2 * G; i++)
        if (i >= first) {
            if (i == 2 * G - 1) {
                d[i] = (long long)top;
            } else {
                const int b = seg_width(bw, i);
                const __int128 c = (top + ((__int128)1 << (b - 1))) >> b;
                d[i] = (long long)(top - (c << b));
                top = c;
            }
        }
    return (long long)q;
}

// v u 2^-(64 + n) rounded to the nearest integer; frac is the difference to it times 2^32.
__device__ __forceinline__ long long scale_round(long long v, long long u, int n, int &frac) {
    Acc a;
    a.mac(hi32(v), lo32(v), hi32(u), lo32(u));
    a.t -= kHalf;  // the words below the integer are kept, not rounded away
    const long long s = a.high();
    unsigned s0 = (unsigned)a.t, s1 = (unsigned)s;
    int s2 = (int)(s >> 32);
    for (; n >= 32; n -= 32) {
        s0 = s1;
        s1 = (unsigned)s2;
        s2 >>= 31;
    }
    frac = (int)__funnelshift_r(s0, s1, n);
    const long long q = ((long long)(s2 >> n) << 32) | __funnelshift_r(s1, (unsigned)s2, n);
    return q - (frac >> 31);
}

// The scale of a column inverse whose components are below 2^e: conj(t4) divides by 4
__device__ __forceinline__ int col_scale(const FftPlan &pl, int e) {
    return 64 - max(3, pl.headroom) - e;
}

// A thread has a row segment, so what the segments read and write beside the transforms' own layout lies
// by column: 16-byte words of 32 rows side by side.  By rows, each such access touched 32 half-used
// sectors 128 bytes apart: at 256 tests of n = 300000 to 700000 the column forward pass took 0.130 ms,
// and 0.096 ms so.
template <int G, class TAB>
__device__ __forceinline__ void segment_carries(const TestDesc &T, int g, const longlong2 *sm) {
    const int R = T.R, C = T.C;
    constexpr int LG = G == 8 ? 3 : G == 4 ? 2 : 1;
    const int nadd = T.nadd;
    // balanced carry along each row segment (2G digits), constants added first; the carry-out
    // goes to the next segment's slot, the last segment's into the top fold
    for (int r = threadIdx.x; r < R; r += blockDim.x) {
        const int j0 = 2 * (r * C + g * G);
        long long d[2 * G];
        const SegWidths<G> bw = load_segment_widths<G, TAB>(T.segbits, 2 * G * (g * R + r));
#pragma unroll
        for (int l = 0; l < G; l++) {
            const longlong2 p = sm[turned<LG>(r, l)];
            d[2 * l] = p.x;
            d[2 * l + 1] = p.y;
        }
        for (int a = 0; a < nadd; a++) {
            const int at = T.addj[a] - j0;
            if (at < 0 || at >= 2 * G) continue;
#pragma unroll
            for (int i = 0; i < 2 * G; i++)
                if (at == i) d[i] += T.addv[a];
        }
        long long cy = 0;
#pragma unroll
        for (int i = 0; i < 2 * G; i++) {
            const long long v = d[i] + cy;
            const int b = seg_width(bw, i);
            const long long q = (v + (1ll << (b - 1))) >> b;
            d[i] = v - (q << b);
            cy = q;
        }
        const bool top = g == T.NG - 1 && r == R - 1;
        if (top) cy = fold_segment<G>(T, bw, d, cy);
        longlong2 *dst = reinterpret_cast<longlong2 *>(T.dig) + g * G * R + r;
#pragma unroll
        for (int l = 0; l < G; l++) dst[l * R] = make_longlong2(d[2 * l], d[2 * l + 1]);
        T.slot[top ? 0 : g < T.NG - 1 ? (g + 1) * R + r : r + 1] = cy;
    }
}

// What the first stage of a column inverse reads: a component pair, its twiddle, its row's exponent.
struct TurnedIn {
    longlong2 v;
    int4 w;
    int up;
};

// One column group of one test, first half of the column pass.  Ends with a barrier after its
// last global write.
template <int LG, class TAB>
__device__ __forceinline__ void col_inverse_item(const TestDesc &T, int g, int step, const double2 *xd, longlong2 *sm,
                                                 ItemCtl &ctl) {
    const bool track = step % T.err_every == 0;
    const int C = T.C;
    const FftPlan &pl = T.cp;
    const longlong2 *x = reinterpret_cast<const longlong2 *>(xd) + (g << LG);
    const int4 *t4 = T.t4 + (g << LG);
    const int *rexp = T.rexp;
    const int se = col_scale(pl, __ldcg(T.emax));
    // the digits are v osc 2^-(64 + n + shift)
    const int n = se - 4 - pl.scale - T.osc_exp;
    const unsigned odd = odd_columns(g, LG);
    int shift;
    const long long *osc = T.osc + 2 * (g << LG);
    int above = 0, below = 0;  // the largest difference to an integer of either sign
    unsigned big = 0;
    longlong2 *digits = transform<LG, true, TAB>(
        pl, T.twc, sm, sm + (T.R << LG), odd,
        [&](int, int k, int l) { return TurnedIn{__ldcg(&x[k * C + l]), TAB::load(&t4[k * T.pitch + l]), __ldcg(&rexp[k])}; },
        [&](const TurnedIn &in, int k, int l) {
            return cmul(cshift(in.v, in.up + se), conj_tw(in.w), half_of(parity(k) ^ ((odd >> l) & 1)));
        },
        [&](int r, int l) { return TAB::load(reinterpret_cast<const longlong2 *>(osc + 2 * (r * T.pitch + l))); },
        [&](longlong2 *dst, int, int r, int l, longlong2 v, longlong2 o) {
            // unweight, scale and round
            const int m = min((unsigned)(n + shift), 95u);
            int fx, fy;
            v.x = scale_round(v.x, o.x, m, fx);
            v.y = scale_round(v.y, o.y, m, fy);
            above = max(above, max(fx, fy));
            below = min(below, min(fx, fy));
            big |= mag32(v);
            dst[turned<LG>(r, l)] = v;
        },
        &ctl.mid[0], shift);
    const bool short_transform = n + shift < 0;  // the last place is above 1: too short for its data
    segment_carries<1 << LG, TAB>(T, g, digits);
    // |digit| >= 2^51 reports 0.5, as does a transform too short for its data
    // below in unsigned: -1/2 is the lowest int
    unsigned err = track ? max((unsigned)above, 0u - (unsigned)below) : 0;
    if (big >= (1u << 19) || short_transform) err = 0x80000000u;
    err = __reduce_max_sync(0xffffffffu, err);
    if ((threadIdx.x & 31) == 0 && err)
        atomicMax(T.maxerr, (unsigned long long)__double_as_longlong((double)err * (1.0 / 4294967296.0)));
    __syncthreads();
}

template <int G, class TAB>
__device__ __forceinline__ void absorb_carries(const TestDesc &T, int g, bool use_slots, int shift, longlong2 *sm) {
    const int R = T.R;
    constexpr int LG = G == 8 ? 3 : G == 4 ? 2 : 1;
    // absorb the carry-in into the segment's first digits (the last digit takes any rest), reweight
    for (int r = threadIdx.x; r < R; r += blockDim.x) {
        const SegWidths<G> bw = load_segment_widths<G, TAB>(T.segbits, 2 * G * (g * R + r));
        long long cy = use_slots ? __ldcg(&T.slot[g * R + r]) : 0;
        const longlong2 *wv = reinterpret_cast<const longlong2 *>(T.w) + g * G * R + r;
        constexpr int kEarly = G / 2;
        longlong2 we[kEarly];
        long long d[2 * G];
        const longlong2 *src = reinterpret_cast<const longlong2 *>(T.dig) + (use_slots ? g * G * R + r : r * T.C + g * G);
        const int column = use_slots ? R : 1;
#pragma unroll
        for (int l = 0; l < G; l++) {
            const longlong2 p = TAB::load_own(src + l * column);
            d[2 * l] = p.x;
            d[2 * l + 1] = p.y;
        }
#pragma unroll
        for (int l = 0; l < kEarly; l++) we[l] = TAB::load(wv + l * R);
#pragma unroll
        for (int i = 0; i < 2 * G - 1; i++) {
            if (cy) {
                const int b = seg_width(bw, i);
                const long long v = d[i] + cy;
                const long long q = (v + (1ll << (b - 1))) >> b;
                d[i] = v - (q << b);
                cy = q;
            }
        }
        d[2 * G - 1] += cy;
#pragma unroll
        for (int l = 0; l < G; l++) {
            const longlong2 w = l < kEarly ? we[l < kEarly ? l : 0] : TAB::load(wv + l * R);
            const long long a = shift_by(d[2 * l], shift), b = shift_by(d[2 * l + 1], shift);
            Acc x, y;
            x.mac(hi32(a), lo32(a), hi32(w.x), lo32(w.x));
            y.mac(hi32(b), lo32(b), hi32(w.y), lo32(w.y));
            sm[turned<LG>(r, l)] = make_longlong2(x.high(), y.high());
        }
    }
}

// One column group of one test, second half of the column pass: absorb the carry-in, reweight,
// forward column transform, twiddle.  `digit_bits` bounds the digits (T.digit_bits after a
// product).  Ends with a barrier after its last global write.
template <int LG, class TAB>
__device__ __forceinline__ void col_forward_item(const TestDesc &T, int g, double2 *x, bool use_slots, int digit_bits,
                                                 longlong2 *sm, ItemCtl &ctl) {
    const int C = T.C;
    const FftPlan &pl = T.cp;
    // every column inverse that read it is done
    if (g == 0 && threadIdx.x == 0) *T.emax = INT_MIN;
    // digits 2^shift w 2^-3: components below 2^59
    const int shift = 61 - digit_bits - max(0, pl.headroom - 3);
    absorb_carries<1 << LG, TAB>(T, g, use_slots, shift, sm);
    __syncthreads();
    const unsigned odd = odd_columns(g, LG);
    int up;
    const int ex = pl.scale + 2 + 3 - shift;
    double2 *xg = x + (g << LG);
    const int4 *t4 = T.t4 + (g << LG);
    transform<LG, false, TAB>(
        pl, T.twc, sm + (T.R << LG), sm, odd, [&](int, int r, int l) { return sm[turned<LG>(r, l)]; }, as_read,
        [&](int k, int l) { return TAB::load(&t4[k * T.pitch + l]); },
        [&](longlong2 *, int, int k, int l, longlong2 v, int4 w) {
            const int e = k * C + l;
            const longlong2 z = cmul(v, w, half_of(parity(k) ^ ((odd >> l) & 1)));
            xg[e] = make_double2(from_fixed(z.x, ex - up), from_fixed(z.y, ex - up));
        },
        &ctl.mid[0], up);
}

// One column group of one test: its digits.  Ends with a barrier.
template <int LG, class TAB>
__device__ __forceinline__ void col_digits_item(const TestDesc &T, int g, const double2 *xd, long long *dig,
                                                longlong2 *sm, ItemCtl &ctl) {
    const int C = T.C, R = T.R;
    const FftPlan &pl = T.cp;
    const longlong2 *x = reinterpret_cast<const longlong2 *>(xd) + (g << LG);
    const int4 *t4 = T.t4 + (g << LG);
    unsigned top = 0;
    for (int i = threadIdx.x; i < R << LG; i += blockDim.x) {
        const int k = i >> LG, l = i & ((1 << LG) - 1);
        const longlong2 v = __ldcg(&x[k * C + l]);
        sm[i] = v;
        top = max(top, top_word(v));
    }
    block_max(top, &ctl.top[0]);
    __syncthreads();
    const int se = clamp_scale(col_scale(pl, top_exponent(ctl.top[0])));
    const int n = se - 4 - pl.scale - T.idig_exp;
    const unsigned odd = odd_columns(g, LG);
    int shift;
    transform<LG, true, TAB>(
        pl, T.twc, sm + (R << LG), sm, odd,
        [&](int at, int k, int l) { return TurnedIn{sm[at], TAB::load(&t4[k * T.pitch + l]), 0}; },
        [&](const TurnedIn &in, int k, int l) {
            return cmul(make_longlong2(to_fixed(in.v.x, se), to_fixed(in.v.y, se)), conj_tw(in.w),
                        half_of(parity(k) ^ ((odd >> l) & 1)));
        },
        [&](int r, int l) { return __ldg(reinterpret_cast<const longlong2 *>(T.idig + 2 * (r * C + (g << LG) + l))); },
        [&](longlong2 *, int, int r, int l, longlong2 v, longlong2 o) {
            const int j = 2 * (r * C + (g << LG) + l), m = n + shift;
            int f;
            dig[j] = shift_by(scale_round(v.x, o.x, max(0, min(m, 95)), f), max(0, -m));
            dig[j + 1] = shift_by(scale_round(v.y, o.y, max(0, min(m, 95)), f), max(0, -m));
        },
        &ctl.mid[0], shift);
}

}  // namespace kg
