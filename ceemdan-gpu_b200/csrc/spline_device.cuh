// Device primitives of the canonical spline solve shared by the kernels' translation units: exact
// integer-divisor quotients, chunk sweeps over rows and knots, and the partitioned solve of padded
// rows.  Arithmetic order: canon.cuh.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "canon.cuh"
#include "kernels.h"

namespace ceemdan {
namespace {

// Division by a divisor d with y = RN(1/d): div_rcp's quotient (Markstein's correction, correctly
// rounded in its range; tests/spline_div_check.cu); `slow` marks operands outside that range, which
// take the division.
__device__ __forceinline__ double rcp_fast(double a, double d, double y, bool& slow) {
    const double q0 = a * y;
    const double r = fma(-q0, d, a);
    const double q1 = fma(r, y, q0);
    slow = !(fabs(a) > 0x1p-960) || !(fabs(q1) < 0x1p+1000);
    return q1;
}

// ---------------------------------------------------------------------------------------
// chunk primitives of the canonical partitioned solve (rows produced by a functor)
// ---------------------------------------------------------------------------------------
struct ChunkEnds {
    double ga, aa, ba, gb, ab, bb;
};

// End relations of a chunk of `len` rows: top-down elimination gives the last row
// x_b = gb + ab*xL + bb*xR, bottom-up elimination the first row x_a = ga + aa*xL + ba*xR.
// The two sweeps are independent chains and run interleaved.  The pivot reciprocals of the
// top-down sweep are those of the interior's sweep: row k's goes to iw_out(k), where
// chunk_interior_iw takes it from.  (Loops stay rolled: a CTA passes here once, and unrolled
// sweeps spent most of their time fetching instructions, up to 1000 cycles a row.)
template <class Pivot = SplinePivot, class RowFn, class IwOut>
__device__ __forceinline__ ChunkEnds chunk_ends(int len, const RowFn& row, const IwOut& iw_out) {
    const Row wa = row(0), wb = row(len - 1);
    double iw = Pivot::inv(wa.m);
    double iv = Pivot::inv(wb.m);
    double cp = wa.u * iw, gp = wa.r * iw, ap = -wa.l * iw;
    double cq = wb.l * iv, gq = wb.r * iv, bq = -wb.u * iv;
    iw_out(0) = iw;
    Row w = len > 1 ? row(1) : wa, v = len > 1 ? row(len - 2) : wb;
#pragma unroll 1
    for (int k = 1; k < len; ++k) {
        const Row wc = w, vc = v;
        if (k + 1 < len) {  // the next rows load while this row's reciprocals form
            w = row(k + 1);
            v = row(len - 2 - k);
        }
        iw = Pivot::inv(fma(-wc.l, cp, wc.m));
        iv = Pivot::inv(fma(-vc.u, cq, vc.m));
        cp = wc.u * iw;
        gp = fma(-wc.l, gp, wc.r) * iw;
        ap = (-wc.l * ap) * iw;
        cq = vc.l * iv;
        gq = fma(-vc.u, gq, vc.r) * iv;
        bq = (-vc.u * bq) * iv;
        iw_out(k) = iw;
    }
    ChunkEnds e;
    e.gb = gp;
    e.ab = ap;
    e.bb = -wb.u * iw;
    e.ga = gq;
    e.ba = bq;
    e.aa = -wa.l * iv;
    return e;
}

// x(k) <- x(k) - fac(k) x(k+1) from row len-2 down, x(len-1) = xv; loads one row ahead.
template <class X, class Fac>
__device__ __forceinline__ void back_sweep(int len, double xv, const X& x, const Fac& fac) {
    double f = 0.0, g = 0.0;
    if (len > 1) {
        f = fac(len - 2);
        g = x(len - 2);
    }
#pragma unroll 1
    for (int k = len - 2; k >= 0; --k) {
        const double fc = f, gc = g;
        if (k > 0) {
            f = fac(k - 1);
            g = x(k - 1);
        }
        xv = fma(-fc, xv, gc);
        x(k) = xv;
    }
}

// Interior of a chunk whose end relations chunk_ends formed: coupling terms to the right-hand
// side, then canonical Thomas with the reciprocals left in x(k); x(k) receives the solution,
// fac(k) the factors meanwhile (fac(k) may be row k's own u or a slot of it that rows after k do
// not read).
template <class RowFn, class X, class Fac>
__device__ __forceinline__ void chunk_interior_iw(int len, const RowFn& row, double xl, double xr,
                                                  const X& x, const Fac& fac) {
    Row w = row(0);
    double iw = x(0), gp = 0.0;
#pragma unroll 1
    for (int k = 0; k < len; ++k) {
        const Row wc = w;
        const double ic = iw;
        if (k + 1 < len) {
            w = row(k + 1);
            iw = x(k + 1);
        }
        double ri = wc.r;
        if (k == 0) ri = fma(-wc.l, xl, ri);
        if (k == len - 1) ri = fma(-wc.u, xr, ri);
        gp = k == 0 ? ri * ic : fma(-wc.l, gp, ri) * ic;
        fac(k) = wc.u * ic;
        x(k) = gp;
    }
    back_sweep(len, gp, x, fac);
}

// Canonical Thomas on n <= kChunk rows, solution to x(k), factors to fac(k) meanwhile.
template <class Pivot = SplinePivot, class RowFn, class X, class Fac>
__device__ __forceinline__ void thomas_rolled(int n, const RowFn& row, const X& x,
                                              const Fac& fac) {
    Row w = row(0);
    double cp = 0.0, gp = 0.0;
#pragma unroll 1
    for (int k = 0; k < n; ++k) {
        const Row wc = w;
        if (k + 1 < n) w = row(k + 1);
        const double iw = Pivot::inv(k == 0 ? wc.m : fma(-wc.l, cp, wc.m));
        gp = k == 0 ? wc.r * iw : fma(-wc.l, gp, wc.r) * iw;
        cp = wc.u * iw;
        fac(k) = cp;
        x(k) = gp;
    }
    back_sweep(n, gp, x, fac);
}

// Drops the reciprocals it is given.
struct NoIw {
    struct Sink {
        __device__ __forceinline__ void operator=(double) const {}
    };
    __device__ __forceinline__ Sink operator()(int) const { return Sink(); }
};

// Interior of a chunk of `len` rows once its separator values xl, xr are known: coupling
// terms move to the right-hand side, then canonical Thomas; x_k written to out[k*stride].
// kCoupled = false is the plain canonical Thomas (no coupling terms at all).
template <bool kCoupled = true, class Pivot = SplinePivot, class RowFn, class Out>
__device__ __forceinline__ void chunk_interior(int len, const RowFn& row, double xl, double xr,
                                               Out out, int stride) {
    double cp[kChunk], gp[kChunk];
#pragma unroll
    for (int k = 0; k < kChunk; ++k) {
        if (k < len) {
            const Row w = row(k);
            double ri = w.r;
            if (kCoupled && k == 0) ri = fma(-w.l, xl, ri);
            if (kCoupled && k == len - 1) ri = fma(-w.u, xr, ri);
            if (k == 0) {
                const double iw = Pivot::inv(w.m);
                cp[0] = w.u * iw;
                gp[0] = ri * iw;
            } else {
                const double iw = Pivot::inv(fma(-w.l, cp[k - 1], w.m));
                cp[k] = w.u * iw;
                gp[k] = fma(-w.l, gp[k - 1], ri) * iw;
            }
        }
    }
    double xv = 0.0;
#pragma unroll
    for (int k = kChunk - 1; k >= 0; --k) {
        if (k < len) {
            xv = (k == len - 1) ? gp[k] : fma(-cp[k], xv, gp[k]);
            out[k * stride] = xv;
        }
    }
}

// Canonical Thomas on n <= kChunk rows (base case), x written with stride.
template <class Pivot = SplinePivot, class RowFn>
__device__ __forceinline__ void thomas_small(int n, const RowFn& row, double* x, int stride) {
    chunk_interior<false, Pivot>(n, row, 0.0, 0.0, x, stride);
}

// Rows of a tile, knots of a spline: the padded position of in-tile knot m in the shared-memory
// knot arrays, one pad slot after every 16 knots, so that the chunk sweeps (lane p walks the
// knots of chunk p, 16 knots after lane p-1's) read different banks.
__device__ __forceinline__ int kq(int m) { return m + (m >> 4); }

// separators of a tile with c knots (local 0, 16, 32, ... and the last one)
__device__ __forceinline__ int tile_seps(int c) { return c > 0 ? (c + kChunk - 2) / kChunk + 1 : 0; }

// Asynchronous global -> shared copies.
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem));
}
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
// all but the newest group
__device__ __forceinline__ void cp_async_wait_but_one() {
    asm volatile("cp.async.wait_group 1;\n" ::);
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::); }

// The quotient a / d by the division itself, kept out of line of the fast path (a plain
// division in a branch is evaluated unconditionally by the compiler).
__device__ __forceinline__ double div_cold(double a, double d) {
    double q;
    asm volatile("div.rn.f64 %0, %1, %2;" : "=d"(q) : "d"(a), "d"(d));
    return q;
}

// a / d for an integer-valued d in [1, 2^40], from its reciprocal (Markstein's correction as in
// div_rcp; operands outside its range take the division).  The reciprocal is pivot_inv's without
// the check for the all-ones significand, which an integer below 2^52 does not have; measured
// against a table of 1/d in global memory it saves the load and its bounds.
__device__ __forceinline__ double div_int(double a, double d) {
    bool slow;
    double q = rcp_fast(a, d, rcp_raw(d), slow);
    if (slow) q = div_cold(a, d);
    return q;
}

// A segment's coefficients (spline_coefficients) from its length, slope and spline values:
// b = slope - h (2 c0 + c1) / 3, d = (c1 - c0) / (3h).
__device__ __forceinline__ void seg_coeffs_int(double h, double slope, double c0, double c1,
                                               double& b, double& d) {
    const double hq = h * fma(2.0, c0, c1);
    bool slow;
    double qb = rcp_fast(hq, 3.0, kRcp3, slow);
    if (slow) qb = div_cold(hq, 3.0);
    d = div_int(c1 - c0, 3.0 * h);
    b = slope - qb;
}

// Pivots of one chunk inverted by rcp_raw, with one look for the all-ones significand at the end
// (low word -1; once in 2^32 pivots the caller repeats the chunk with pivot_inv).
struct RawPivot {
    bool ones = false;
    __device__ __forceinline__ double inv(double x) {
        ones |= __double2loint(x) == -1;
        return rcp_raw(x);
    }
};
struct CheckedPivot {
    bool ones = false;
    __device__ __forceinline__ double inv(double x) { return pivot_inv(x); }
};

// End relations (chunk_ends: same operations, same order) of the chunk whose knots 0..len+1 sit
// in the padded arrays x, s from the chunk's base on (s[i]: slope of segment i -> i+1).  Each
// sweep loads one new knot and slope per row, a row ahead of its use.
template <class Pivot, class XT>
__device__ __forceinline__ ChunkEnds chunk_ends_sweep(Pivot& pv, const XT* x, const double* s,
                                                      int len) {
    int xt = x[2], xb = x[len - 1];
    // top-down row 0 and bottom-up row len-1
    double lt = (double)(x[1] - x[0]), ut = (double)(xt - x[1]);
    double ub = (double)(x[kq(len + 1)] - x[len]), lb = (double)(x[len] - xb);
    double st = s[1], sb = s[len - 1];
    const double wr0 = 3.0 * (st - s[0]), vr0 = 3.0 * (s[len] - sb);
    const double lf = lt, ul = ub;
    double un = 0.0, lp = 0.0, sn = 0.0, sp = 0.0;  // the next row's
    if (len > 1) {
        const int xn = x[kq(3)], xp = x[len - 2];
        un = (double)(xn - xt);
        xt = xn;
        lp = (double)(xb - xp);
        xb = xp;
        sn = s[2];
        sp = s[len - 2];
    }
    double iw = pv.inv(2.0 * (lt + ut));
    double iv = pv.inv(2.0 * (lb + ub));
    double cp = ut * iw, gp = wr0 * iw, ap = -lt * iw;
    double cq = lb * iv, gq = vr0 * iv, bq = -ub * iv;
#pragma unroll 2
    for (int k = 1; k < len; ++k) {
        lt = ut;
        ut = un;
        ub = lb;
        lb = lp;
        const double wr = 3.0 * (sn - st), vr = 3.0 * (sb - sp);
        st = sn;
        sb = sp;
        if (k + 1 < len) {
            const int xn = x[kq(k + 3)], xp = x[len - 2 - k];
            un = (double)(xn - xt);
            xt = xn;
            lp = (double)(xb - xp);
            xb = xp;
            sn = s[k + 2];
            sp = s[len - 2 - k];
        }
        iw = pv.inv(fma(-lt, cp, 2.0 * (lt + ut)));
        iv = pv.inv(fma(-ub, cq, 2.0 * (lb + ub)));
        cp = ut * iw;
        gp = fma(-lt, gp, wr) * iw;
        ap = (-lt * ap) * iw;
        cq = lb * iv;
        gq = fma(-ub, gq, vr) * iv;
        bq = (-ub * bq) * iv;
    }
    ChunkEnds e;
    e.gb = gp;
    e.ab = ap;
    e.bb = -ul * iw;
    e.ga = gq;
    e.ba = bq;
    e.aa = -lf * iv;
    return e;
}
template <class XT>
__device__ __noinline__ void chunk_ends_checked(ChunkEnds& e, const XT* x, const double* s,
                                                int len) {
    CheckedPivot pv;
    e = chunk_ends_sweep(pv, x, s, len);
}
template <class XT>
__device__ __forceinline__ ChunkEnds chunk_ends_knots(const XT* x, const double* s, int len) {
    RawPivot pv;
    ChunkEnds e = chunk_ends_sweep(pv, x, s, len);
    if (pv.ones) {
        ChunkEnds c;
        chunk_ends_checked(c, x, s, len);
        e = c;
    }
    return e;
}

// One direction of chunk_ends_sweep (same operations, same order; see ends_sweep): top gb, ab, bb to
// out[3..5] and the reciprocals to iwo, else ga, aa, ba to out[0..2].
template <bool top, class Pivot, class XT>
__device__ __forceinline__ void chunk_ends_one(Pivot& pv, const XT* x, const double* s, int len,
                                               double* out, double* iwo) {
    // knots and slopes in the sweep's direction
    auto knot = [&](int i) -> int { return x[kq(top ? i : len + 1 - i)]; };
    auto slope = [&](int i) -> double { return s[top ? i : len - i]; };
    auto length = [](int from, int to) { return (double)(top ? to - from : from - to); };
    auto rhs = [](double s0, double s1) { return 3.0 * (top ? s1 - s0 : s0 - s1); };
    const int x1 = knot(1);
    int xt = knot(2);
    // row k: o the length towards the sweep's start, t towards its end
    double o = length(knot(0), x1), t = length(x1, xt), st = slope(1), tn = 0.0, sn = 0.0;
    const double r0 = rhs(slope(0), st);
    if (len > 1) {
        const int xn = knot(3);
        tn = length(xt, xn);
        xt = xn;
        sn = slope(2);
    }
    double i = pv.inv(2.0 * (o + t));
    if (top) iwo[0] = i;
    double c = t * i, g = r0 * i, f = -o * i;
#pragma unroll 2
    for (int k = 1; k < len; ++k) {
        o = t;
        t = tn;
        const double r = rhs(st, sn);
        st = sn;
        if (k + 1 < len) {
            const int xn = knot(k + 3);
            tn = length(xt, xn);
            xt = xn;
            sn = slope(k + 2);
        }
        i = pv.inv(fma(-o, c, 2.0 * (o + t)));
        c = t * i;
        g = fma(-o, g, r) * i;
        f = (-o * f) * i;
        if (top) iwo[k] = i;
    }
    out[top ? 3 : 0] = g;
    out[top ? 4 : 2] = f;
    out[top ? 5 : 1] = -t * i;
}
template <bool top, class XT>
__device__ __noinline__ void chunk_ends_one_checked(const XT* x, const double* s, int len,
                                                    double* out, double* iwo) {
    CheckedPivot pv;
    chunk_ends_one<top>(pv, x, s, len, out, iwo);
}
template <bool top, class XT>
__device__ __forceinline__ void chunk_ends_half(const XT* x, const double* s, int len, double* out,
                                                double* iwo) {
    RawPivot pv;
    chunk_ends_one<top>(pv, x, s, len, out, iwo);
    if (pv.ones) chunk_ends_one_checked<top>(x, s, len, out, iwo);
}

// Inclusive prefix of v over the warp's lanes.
__device__ __forceinline__ int warp_scan(int v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Rows of a system with one pad slot per 16 (row i at kq(i)): a chunk's rows are consecutive, and
// the lanes that sweep neighbouring chunks read different banks.
struct alignas(16) SepRow {
    double l, m, u, r;
};
__device__ __forceinline__ SepRow load_row(const SepRow* p) {
    const double2 a = reinterpret_cast<const double2*>(p)[0];
    const double2 b = reinterpret_cast<const double2*>(p)[1];
    return SepRow{a.x, a.y, b.x, b.y};
}
__device__ __forceinline__ SepRow sep_row(const Row& w) { return SepRow{w.l, w.m, w.u, w.r}; }
// padded length of n rows
__host__ __device__ __forceinline__ int padded(int n) { return n + (n >> 4) + 1; }

// One direction of chunk_ends (same operations, same order) of len consecutive rows: top the
// top-down sweep, gb, ab, bb to out[3..5] and its reciprocals to iw (unless null), else the bottom-up
// one, ga, aa, ba to out[0..2].  The two directions are different warps' work: a thread that does
// both waits for its own instructions while the warps beside it have nothing to do (on chip, N=2501
// NR=100: 19.5 -> 18.2 us an iteration; with the direction an argument instead of two copies 0.3 us
// slower there and 2 us in k_spline_solve).
template <bool top, class Pivot>
__device__ __forceinline__ void ends_sweep(Pivot& pv, const SepRow* r, int len, double* iw,
                                           double* out) {
    const double* p = reinterpret_cast<const double*>(top ? r : r + len - 1);
    constexpr int step = top ? 4 : -4;
    // the row's coefficient towards the sweep's start and towards its end
    constexpr int io = top ? 0 : 2, it = 2 - io;
    double o = p[io], t = p[it], m = p[1], b = p[3];
    double i = pv.inv(m);
    double c = t * i, g = b * i, f = -o * i;
    if (top && iw) iw[0] = i;
    double on = 0.0, tn = 0.0, mn = 0.0, bn = 0.0;  // the next row's
    if (len > 1) {
        p += step;
        on = p[io], tn = p[it], mn = p[1], bn = p[3];
    }
#pragma unroll 2
    for (int k = 1; k < len; ++k) {
        o = on, t = tn, m = mn, b = bn;
        if (k + 1 < len) {
            p += step;
            on = p[io], tn = p[it], mn = p[1], bn = p[3];
        }
        i = pv.inv(fma(-o, c, m));
        c = t * i;
        g = fma(-o, g, b) * i;
        f = (-o * f) * i;
        if (top && iw) iw[k] = i;
    }
    out[top ? 3 : 0] = g;
    out[top ? 4 : 2] = f;
    out[top ? 5 : 1] = -t * i;
}
template <bool top>
__device__ __noinline__ void ends_rows_checked(const SepRow* r, int len, double* iw, double* out) {
    CheckedPivot pv;
    ends_sweep<top>(pv, r, len, iw, out);
}
template <bool top>
__device__ __forceinline__ void ends_rows(const SepRow* r, int len, double* iw, double* out) {
    RawPivot pv;
    ends_sweep<top>(pv, r, len, iw, out);
    if (pv.ones) ends_rows_checked<top>(r, len, iw, out);
}
// Work item i of the two directions of n chunks: whole warps of one direction.
__device__ __forceinline__ int ends_items(int n) { return 2 * ((n + 31) & ~31); }
__device__ __forceinline__ bool ends_item(int i, int n, int& q) {
    const int half = (n + 31) & ~31;
    q = i < half ? i : i - half;
    return i < half;
}

// Row p of the next level: separator row s between the chunks with end relations e (left) and
// e + 6 (right).
__device__ __forceinline__ SepRow next_row(const SepRow& s, const double* e) {
    return sep_row(reduced_row(Row{s.l, s.m, s.u, s.r}, e[3], e[4], e[5], e[6], e[7], e[8]));
}

// Back substitution x[k] <- x[k] - fac(k) x[k+1], row k's factor in its u.
__device__ __forceinline__ void back_rows(const SepRow* r, double* x, int len, double xv) {
    int k = len - 2;
#pragma unroll 1
    for (; k >= 3; k -= 4) {  // four rows at a time, loaded before the first is needed
        double f[4], g[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            f[i] = r[k - i].u;
            g[i] = x[k - i];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            xv = fma(-f[i], xv, g[i]);
            x[k - i] = xv;
        }
    }
#pragma unroll 1
    for (; k >= 0; --k) {
        xv = fma(-r[k].u, xv, x[k]);
        x[k] = xv;
    }
}

// chunk_interior_iw of len consecutive rows: x holds the reciprocals, then the solution; the rows'
// u is overwritten.
__device__ __forceinline__ void interior_rows(SepRow* r, int len, double xl, double xr,
                                              double* x) {
    SepRow w = load_row(r);
    double ri = fma(-w.l, xl, w.r);
    if (len == 1) ri = fma(-w.u, xr, ri);
    double gp = ri * x[0];
    r[0].u = w.u * x[0];
    x[0] = gp;
    int k = 1;
#pragma unroll 1
    for (; k + 4 < len; k += 4) {  // four rows at a time, loaded before the first is needed
        double l[4], u[4], b[4], iw[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            l[i] = r[k + i].l;
            u[i] = r[k + i].u;
            b[i] = r[k + i].r;
            iw[i] = x[k + i];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            gp = fma(-l[i], gp, b[i]) * iw[i];
            r[k + i].u = u[i] * iw[i];
            x[k + i] = gp;
        }
    }
#pragma unroll 1
    for (; k < len; ++k) {
        w = load_row(r + k);
        ri = w.r;
        if (k == len - 1) ri = fma(-w.u, xr, ri);
        const double iw = x[k];
        gp = fma(-w.l, gp, ri) * iw;
        r[k].u = w.u * iw;
        x[k] = gp;
    }
    back_rows(r, x, len, gp);
}

// Canonical Thomas of n rows, reciprocals formed here.
__device__ __forceinline__ void thomas_rows(SepRow* r, int n, double* x) {
    SepRow w = load_row(r);
    double cp = 0.0, gp = 0.0;
#pragma unroll 1
    for (int k = 0; k < n; ++k) {
        const SepRow a = w;
        if (k + 1 < n) w = load_row(r + k + 1);
        const double iw = pivot_inv(k == 0 ? a.m : fma(-a.l, cp, a.m));
        gp = (k == 0 ? a.r : fma(-a.l, gp, a.r)) * iw;
        cp = a.u * iw;
        r[k].u = cp;
        x[k] = gp;
    }
    back_rows(r, x, n, gp);
}

// cta_partitioned_global<SplinePivot>'s solve on padded rows: n rows at `rows` (u overwritten), solution to the
// padded x; ws: 5 padded(n/16) + 6 (n/16 + 1) doubles and as much again for what is below, at
// most 0.75 n + 64.  Every thread of the group calls it.
struct RowsLevel {
    SepRow* r;
    double* x;
    int n;
};
__device__ __forceinline__ RowsLevel rows_level(int k, int depth, int n, SepRow* rows, double* x,
                                                double* ws) {
    if (k == 0) return RowsLevel{rows, x, n};
    int ro = 0, xo = 0, size = n, mine = 0, mr = 0, mx = 0;
    for (int i = 1; i <= depth; ++i) {
        size = (size - 1) / kChunk;
        if (i == k) {
            mine = size;
            mr = ro;
            mx = xo;
        }
        ro += 4 * padded(size);
        xo += padded(size);
    }
    return RowsLevel{reinterpret_cast<SepRow*>(ws + mr), ws + ro + mx, mine};
}

// The threads that work on one system: a whole CTA, or half of one with a barrier of its own.
struct CtaGroup {
    __device__ __forceinline__ int tid() const { return threadIdx.x; }
    __device__ __forceinline__ int size() const { return blockDim.x; }
    __device__ __forceinline__ void sync() const { __syncthreads(); }
};

template <class Group>
__device__ void partition_rows(const Group& grp, int n, SepRow* rows, double* x, double* ws) {
    const int tid = grp.tid(), size_g = grp.size();
    int depth = 0, all = 0;
    for (int size = n; size > kChunk && depth < 7; ++depth) {
        size = (size - 1) / kChunk;
        all += 5 * padded(size);
    }
    double* ends = ws + all;
#pragma unroll 1
    for (int k = 0; k < depth; ++k) {
        const RowsLevel v = rows_level(k, depth, n, rows, x, ws);
        const RowsLevel o = rows_level(k + 1, depth, n, rows, x, ws);
        for (int i = tid; i < ends_items(o.n + 1); i += size_g) {
            int q;
            const bool top = ends_item(i, o.n + 1, q);
            if (q > o.n) continue;
            const int first = q * kChunk;
            const int len = (q < o.n) ? kChunk - 1 : v.n - first;
            if (top) ends_rows<true>(v.r + kq(first), len, v.x + kq(first), ends + 6 * q);
            else ends_rows<false>(v.r + kq(first), len, nullptr, ends + 6 * q);
        }
        grp.sync();
        for (int p = tid; p < o.n; p += size_g)
            o.r[kq(p)] = next_row(load_row(v.r + kq(p * kChunk + kChunk - 1)), ends + 6 * p);
        grp.sync();
    }
    if (tid == 0) {
        const RowsLevel v = rows_level(depth, depth, n, rows, x, ws);
        thomas_rows(v.r, v.n, v.x);
    }
    grp.sync();
#pragma unroll 1
    for (int k = depth - 1; k >= 0; --k) {
        const RowsLevel v = rows_level(k, depth, n, rows, x, ws);
        const RowsLevel o = rows_level(k + 1, depth, n, rows, x, ws);
        for (int q = tid; q <= o.n; q += size_g) {
            const int first = q * kChunk;
            const int len = (q < o.n) ? kChunk - 1 : v.n - first;
            const double xl = (q > 0) ? o.x[kq(q - 1)] : 0.0;
            const double xr = (q < o.n) ? o.x[kq(q)] : 0.0;
            interior_rows(v.r + kq(first), len, xl, xr, v.x + kq(first));
            if (q < o.n) v.x[kq(first + kChunk - 1)] = xr;
        }
        grp.sync();
    }
}

}  // namespace
}  // namespace ceemdan
