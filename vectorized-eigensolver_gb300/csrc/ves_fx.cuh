// ves_fx.cuh -- the FP64 solver's unitary transformations in 64-bit fixed
// point on the integer pipe.
//
// Why.  GB300 retires 1.9 FP64 FMAs per clock and SM but 25 32x32+64-bit
// integer multiply-adds (IMAD.WIDE).  The Hessenberg reduction and the QR
// sweeps only apply unitary transformations, under which no entry of the
// matrix can grow past ||A||_F, so one scale per matrix is enough and the
// exponent that a floating-point format carries per number is not needed.  A
// complex rotation of a pair of entries takes 36 IMAD.WIDE here: 0.71 pairs
// per clock and SM measured, against 0.14 as 12 FP64 instructions.
//
// Format.  H is held in units of 2^(e-61), 2^e >= ||A||_F, so |entry| <= 2^61;
// Q, Z and the Householder vectors in units of 2^-61, rotation coefficients in
// units of 2^-62.  A product of two such numbers is formed from 32-bit halves
// (signed high half, signed low half), leaving out low x low, and is rounded
// to one unit: an absolute error of about 2^-61 ||A||_F per operation, against
// 2^-53 |entry| in FP64, where the entries of an n x n matrix are of size
// ||A||_F / n: for n <= 64 the fixed-point transformation is the more accurate
// one.  Rotations and reflectors are computed in FP64 (53 bits), as before.
// Sums of products are exact modulo 2^64 until they are rounded, so a result
// does not depend on how a sum is spread over lanes: every kernel that uses
// these routines, with any number of lanes per matrix, gives the same bits.
//
// One scale per matrix means errors relative to the whole matrix.  FP64 can do
// better on a matrix whose rows, columns or blocks differ widely in size, and
// there this form is not used: a matrix goes to the FP64 kernels when a row or
// column has no entry above 2^-9 of the scale, when its Hessenberg form has a
// subdiagonal below 2^-30 of the scale (it is numerically reducible: blocks
// that may differ in size), when a trailing block is small in A and still small
// in the Hessenberg form (fx_blocks), or when it is zero, not finite or of an
// extreme exponent.  The rule uses integer comparisons of the matrix alone, so
// every kernel sends the same matrices the same way.
#pragma once

#include "ves_device.cuh"

namespace ves {

typedef long long i64;

struct fx { int h, l; };  // value = h 2^32 + l, both signed
struct cfx { fx r, i; };
struct cx64 { i64 r, i; };

__device__ __forceinline__ fx fx_split(i64 x)
{
    fx f;
    f.l = (int)x;
    f.h = (int)(x >> 32) + (int)((unsigned)f.l >> 31);
    return f;
}
__device__ __forceinline__ cfx fx_split(cx64 z) { return {fx_split(z.r), fx_split(z.i)}; }
// a b + c as one IMAD.WIDE (written as PTX: from C the compiler also emits
// a multiply and an add, which doubled the instructions of a rotation)
__device__ __forceinline__ i64 wide(int a, int b, i64 c)
{
#ifdef __CUDA_ARCH__
    i64 d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
#else
    return (i64)a * b + c;
#endif
}

// Sum of products in units of (unit a)(unit b): c carries the cross halves
// (weight 2^32) with the rounding constant, a the high halves (weight 2^64).
struct facc { i64 c, a; };
template <int SH> __device__ __forceinline__ facc fx_zero() { return {1LL << (SH - 33), 0}; }
__device__ __forceinline__ void fx_mac(facc &s, fx a, fx b)
{
    s.c = wide(a.h, b.l, s.c);
    s.c = wide(a.l, b.h, s.c);
    s.a = wide(a.h, b.h, s.a);
}
// keeps the cross sum small: |c| < 2^63 holds for 8 products of vectors whose
// norms are at most 2^61 and sqrt(2) 2^61 (4 complex terms)
__device__ __forceinline__ void fx_flush(facc &s)
{
    s.a += s.c >> 32;
    s.c = (i64)(unsigned)s.c;
}
// The sum (t 2^64 + low half of c 2^32) / 2^SH.
template <int SH> __device__ __forceinline__ i64 fx_join(const i64 c, const i64 t)
{
    const unsigned lo = __funnelshift_l((unsigned)c, (unsigned)t, 64 - SH);
    const unsigned hi = __funnelshift_l((unsigned)t, (unsigned)(t >> 32), 64 - SH);
    return (i64)(((unsigned long long)hi << 32) | lo);
}
template <int SH> __device__ __forceinline__ i64 fx_end(const facc s)
{
    return fx_join<SH>(s.c, s.a + (s.c >> 32));
}
// Two and three products, the cross halves first: their carry starts the sum
// of the high halves.
template <int SH> __device__ __forceinline__ i64 fx_dot2(fx a, fx x, fx b, fx y)
{
    i64 c = 1LL << (SH - 33);
    c = wide(a.h, x.l, c);
    c = wide(a.l, x.h, c);
    c = wide(b.h, y.l, c);
    c = wide(b.l, y.h, c);
    i64 t = c >> 32;
    t = wide(a.h, x.h, t);
    t = wide(b.h, y.h, t);
    return fx_join<SH>(c, t);
}
__device__ __forceinline__ i64 fx_dot3(fx a, fx x, fx b, fx y, fx p, fx z)
{
    i64 c = 1LL << 29;
    c = wide(a.h, x.l, c);
    c = wide(a.l, x.h, c);
    c = wide(b.h, y.l, c);
    c = wide(b.l, y.h, c);
    c = wide(p.h, z.l, c);
    c = wide(p.l, z.h, c);
    i64 t = c >> 32;
    t = wide(a.h, x.h, t);
    t = wide(b.h, y.h, t);
    t = wide(p.h, z.h, t);
    return fx_join<62>(c, t);
}

// Matrix and vector accessors, 1-based; element e of a matrix or vector at
// p + e * ST: ST = 1 in shared memory, 32 in a warp's workspace (one matrix
// per lane, a warp's copies of one element contiguous).
template <int ST> struct FxMat {
    longlong2 *p;
    int lda, n;
    __device__ __forceinline__ longlong2 *at(int i, int j) const
    {
        VES_CHECK_IJ(i, j, n);
        return p + ((i - 1) + (j - 1) * lda) * ST;
    }
    __device__ __forceinline__ bool holds(const longlong2 *a, long long reach) const
    {
        return a >= p && reach >= 0 && (a - p) + reach < (long long)lda * n * ST;
    }
    __device__ __forceinline__ cx64 ld(int i, int j) const { const longlong2 v = *at(i, j); return {v.x, v.y}; }
    __device__ __forceinline__ void st(int i, int j, cx64 v) const { *at(i, j) = make_longlong2(v.r, v.i); }
    __device__ __forceinline__ cx<double> ldd(int i, int j) const
    {
        const double2 v = *reinterpret_cast<const double2 *>(at(i, j));
        return mk(v.x, v.y);
    }
    __device__ __forceinline__ void std(int i, int j, cx<double> v) const
    {
        *reinterpret_cast<double2 *>(at(i, j)) = make_double2(v.r, v.i);
    }
};
template <int ST> struct FxVec {
    longlong2 *p;
    __device__ __forceinline__ longlong2 *at(int k) const
    {
        VES_CHECK_I(k);
        return p + (k - 1) * ST;
    }
    __device__ __forceinline__ cx64 ld(int k) const { const longlong2 v = *at(k); return {v.x, v.y}; }
    __device__ __forceinline__ void st(int k, cx64 v) const { *at(k) = make_longlong2(v.r, v.i); }
    __device__ __forceinline__ cx<double> ldd(int k) const
    {
        const double2 v = *reinterpret_cast<const double2 *>(at(k));
        return mk(v.x, v.y);
    }
    __device__ __forceinline__ void std(int k, cx<double> v) const
    {
        *reinterpret_cast<double2 *>(at(k)) = make_double2(v.r, v.i);
    }
};

__device__ __forceinline__ cx<double> fx_d(cx64 z) { return mk((double)z.r, (double)z.i); }
__device__ __forceinline__ i64 fx_abs(i64 x) { return x < 0 ? -x : x; }
__device__ __forceinline__ i64 fx_abs1(cx64 z) { return fx_abs(z.r) + fx_abs(z.i); }
__device__ __forceinline__ int fx_high(cx64 z) { return max(abs((int)(z.r >> 32)), abs((int)(z.i >> 32))); }

// Rotation [c s; -conj(s) c], c real: in FP64, and in units of 2^-62.
struct FxRot {
    double dc;
    cx<double> ds;
    i64 c, sr, si;
};
struct FxCoef {
    fx c, sr, nsr, si, nsi;
    __device__ __forceinline__ FxCoef(i64 ic, i64 isr, i64 isi)
        : c(fx_split(ic)), sr(fx_split(isr)), nsr(fx_split(-isr)), si(fx_split(isi)), nsi(fx_split(-isi))
    {
    }
    __device__ __forceinline__ explicit FxCoef(const FxRot &q) : FxCoef(q.c, q.sr, q.si) {}
    __device__ __forceinline__ FxCoef columns() const  // of the rotation with conj(s)
    {
        FxCoef q(*this);
        q.si = nsi;
        q.nsi = si;
        return q;
    }
};

__device__ __forceinline__ cx64 fx_i(cx<double> z) { return {__double2ll_rn(z.r), __double2ll_rn(z.i)}; }

// The rotation that maps (x0, x1) to (r, 0), from one reciprocal square root:
// with f = |x0|^2, g = |x1|^2, p = 1 / sqrt(f (f + g)): c = f p,
// s = x0 conj(x1) p, r = x0 (f + g) p.
__device__ __forceinline__ FxRot fx_rot(const cx<double> x0, const cx<double> x1, cx<double> &r)
{
    const double one = 4611686018427387904.0;  // 2^62
    const double f = fma(x0.r, x0.r, x0.i * x0.i), g = fma(x1.r, x1.r, x1.i * x1.i);
    const double n2 = f + g, w = f * n2;
    const bool deg = !(w > 1e-280);  // x0 = 0 (or both far below one unit)
    const double p = rsqrt(deg ? fmax(g, 1e-280) : w);
    const double a = deg ? 1.0 : x0.r, b = deg ? 0.0 : x0.i;
    FxRot q;
    q.dc = deg ? 0.0 : f * p;
    q.ds = mk(fma(a, x1.r, b * x1.i) * p, fma(b, x1.r, -(a * x1.i)) * p);
    if (deg && !(g > 1e-280)) { q.dc = 1.0; q.ds = mk(0.0, 0.0); }
    const double np = deg ? g * p : n2 * p;
    r = mk(a * np, b * np);
    const cx64 s = fx_i(cscal(q.ds, one));
    q.c = __double2ll_rn(q.dc * one);
    q.sr = s.r;
    q.si = s.i;
    return q;
}

// Rotate the pair (x1, x2): x1' = c x1 + s x2, x2' = c x2 - conj(s) x1 (rows of
// H; columns of H and Z take the coefficients of conj(s)).
__device__ __forceinline__ void fx_pair(cx64 &x1, cx64 &x2, const FxCoef &q)
{
    const cfx a = fx_split(x1), b = fx_split(x2);
    x1.r = fx_dot3(q.c, a.r, q.sr, b.r, q.nsi, b.i);
    x1.i = fx_dot3(q.c, a.i, q.sr, b.i, q.si, b.r);
    x2.r = fx_dot3(q.c, b.r, q.nsr, a.r, q.nsi, a.i);
    x2.i = fx_dot3(q.c, b.i, q.nsr, a.i, q.si, a.r);
}

// Wilkinson's correction of the shift: t = d - bc / (x + y) for the trailing
// block [a b; c d] (any phases), x = (a - d) / 2, y = sqrt(x^2 + bc) on x's
// side; here bc / (x + y), from x, b, c in units of 2^61 of H.  In FP32: as c
// becomes small the term does too, and an error of 2^-22 of it costs the
// convergence nothing.  Products and sums are written out, so every kernel
// computes the same bits.
__device__ __forceinline__ cx<float> fx_wilkinson(const cx<float> x, const cx<float> b, const cx<float> c)
{
    const cx<float> bc = mk(__fmaf_rn(b.r, c.r, -__fmul_rn(b.i, c.i)), __fmaf_rn(b.i, c.r, __fmul_rn(b.r, c.i)));
    const cx<float> z = mk(__fadd_rn(__fmaf_rn(x.r, x.r, -__fmul_rn(x.i, x.i)), bc.r),
                           __fadd_rn(__fmul_rn(2.f, __fmul_rn(x.r, x.i)), bc.i));
    // sqrt(z): |z| = m |z / m|, m its larger component
    const float m = fmaxf(fabsf(z.r), fabsf(z.i));
    cx<float> y = mk(0.f, 0.f);
    if (m > 0.f) {
        const float im = __frcp_rn(m), u = __fmul_rn(z.r, im), v = __fmul_rn(z.i, im);
        const float az = __fsqrt_rn(__fmaf_rn(u, u, __fmul_rn(v, v)));
        const float h = __fmul_rn(0.5f, __fadd_rn(az, fabsf(u)));  // in [1/2, sqrt 2]
        const float sm = __fsqrt_rn(m), zr = __fsqrt_rn(h), zi = __fmul_rn(__fmul_rn(0.5f, fabsf(v)), __frcp_rn(zr));
        y = u < 0.f ? mk(__fmul_rn(zi, sm), __fmul_rn(zr, sm)) : mk(__fmul_rn(zr, sm), __fmul_rn(zi, sm));
        if (v < 0.f) y.i = -y.i;
    }
    if (__fmaf_rn(x.r, y.r, __fmul_rn(x.i, y.i)) < 0.f) y = mk(-y.r, -y.i);
    const cx<float> w = mk(__fadd_rn(x.r, y.r), __fadd_rn(x.i, y.i));
    const float k = fmaxf(fabsf(w.r), fabsf(w.i));
    if (!(k > 0.f)) return mk(0.f, 0.f);
    const float ik = __frcp_rn(k), wr = __fmul_rn(w.r, ik), wi = __fmul_rn(w.i, ik);
    const float q = __fmul_rn(ik, __frcp_rn(__fmaf_rn(wr, wr, __fmul_rn(wi, wi))));
    return mk(__fmul_rn(__fmaf_rn(bc.r, wr, __fmul_rn(bc.i, wi)), q),
              __fmul_rn(__fmaf_rn(bc.i, wr, -__fmul_rn(bc.r, wi)), q));
}

// For a window of two the shift is the eigenvalue, and one sweep ends it if
// the shift is exact to rounding: two Newton steps on w (w + 2x) = bc, the
// residual in fixed point, take the FP32 value there (2^-22 -> 2^-44 -> units).
__device__ __forceinline__ void fx_wilkinson_2x2(cx64 &w, const cx64 x2, const cx64 b, const cx64 c)
{
    const cfx bf = fx_split(b), cf = fx_split(c);
    const fx nbi = fx_split(-b.i);
    const cx64 bc = {fx_dot2<61>(bf.r, cf.r, nbi, cf.i), fx_dot2<61>(bf.r, cf.i, bf.i, cf.r)};
#pragma unroll 1
    for (int it = 0; it < 2; ++it) {
        const cx64 v = {w.r + x2.r, w.i + x2.i};
        const cfx wf = fx_split(w), vf = fx_split(v);
        const fx nwi = fx_split(-w.i);
        const float rr = (float)(fx_dot2<61>(wf.r, vf.r, nwi, vf.i) - bc.r);
        const float ri = (float)(fx_dot2<61>(wf.r, vf.i, wf.i, vf.r) - bc.i);
        const float k = 0x1p-61f, dr = __fmul_rn(__fadd_rn((float)v.r, (float)w.r), k),
                    di = __fmul_rn(__fadd_rn((float)v.i, (float)w.i), k);
        const float m = fmaxf(fabsf(dr), fabsf(di));
        if (!(m > 0x1p-55f)) return;
        const float im = __frcp_rn(m), ur = __fmul_rn(dr, im), ui = __fmul_rn(di, im);
        const float q = __fmul_rn(im, __frcp_rn(__fmaf_rn(ur, ur, __fmul_rn(ui, ui))));
        const float er = __fmul_rn(__fmaf_rn(rr, ur, __fmul_rn(ri, ui)), q), ei = __fmul_rn(__fmaf_rn(ri, ur, -__fmul_rn(rr, ui)), q);
        if (!(fabsf(er) + fabsf(ei) < 0x1p60f)) return;
        w.r -= __float2ll_rn(er);
        w.i -= __float2ll_rn(ei);
    }
}

// Is the subdiagonal H(K, K-1) = S(K-1) negligible?  The reference's test
// (Toolbox.hpp:810-867: |h| <= ulp (|h_kk| + |h_k-1,k-1|) and the Ahues-
// Tisseur condition, multiplied through by its denominator) in FP32, which
// moves the thresholds by a few 2^-23; anything below half a unit is
// negligible too.  The reference keeps subdiagonals real by a diagonal phase
// similarity: there H(K, K-1) is |s| and H(K-1, K) is turned by the phase of s.
__device__ __forceinline__ float fx_absf(cx<float> z) { return __fsqrt_rn(__fmaf_rn(z.r, z.r, __fmul_rn(z.i, z.i))); }
// x 2^sh in FP32, truncated, without the FP64 pipe (conversions run on it);
// 0 below 2^-126
__device__ __forceinline__ float fx_float(const double x, const int sh)
{
    const int hi = __double2hiint(x), e = ((hi >> 20) & 0x7ff) - 1023 + 127 + sh;
    const int v = (hi & 0x80000000) | (e << 23) | ((hi & 0xfffff) << 3) | (int)((unsigned)__double2loint(x) >> 29);
    return e > 0 ? __int_as_float(v) : 0.f;
}
__device__ __forceinline__ cx<float> fx_float(const cx<double> z, const int sh) { return mk(fx_float(z.r, sh), fx_float(z.i, sh)); }
// (s, d1, d2): S(K-1), H(K-1, K-1), H(K, K).
template <int ST>
__device__ __forceinline__ bool fx_negligible(const FxMat<ST> &H, const FxVec<ST> &S, const int K, const int n,
                                              const cx<double> s, const cx64 d1, const cx64 d2)
{
    const cx<float> sf = fx_float(s, 0);
    const float hk = fx_absf(sf);
    if (hk <= 0.5f) return true;
    float tst = (float)(fx_abs1(d1) + fx_abs1(d2));
    if (tst == 0.f) {
        if (K - 2 >= 1) tst += fx_absf(fx_float(S.ldd(K - 2), 0));
        if (K + 1 <= n) tst += fx_absf(fx_float(S.ldd(K), 0));
    }
    if (hk > 0x1p-52f * tst) return false;
    const cx64 u = H.ld(K - 1, K);
    const float ur = (float)u.r, ui = (float)u.i, ih = __frcp_rn(hk), pr = sf.r * ih, pi = sf.i * ih;
    const float up = fabsf(__fmaf_rn(ur, pr, -__fmul_rn(ui, pi))) + fabsf(__fmaf_rn(ur, pi, __fmul_rn(ui, pr)));
    const float kk = (float)fx_abs1(d2), df = (float)fx_abs1({d1.r - d2.r, d1.i - d2.i});
    return fminf(hk, up) * fmaxf(hk, up) <= 0x1p-52f * fminf(kk, df) * fmaxf(kk, df);
}
template <int ST>
__device__ __forceinline__ bool fx_negligible(const FxMat<ST> &H, const FxVec<ST> &S, const int K, const int n)
{
    return fx_negligible(H, S, K, n, S.ldd(K - 1), H.ld(K - 1, K - 1), H.ld(K, K));
}

// A group of G lanes that owns one matrix: part of a warp (G < 32), a warp, or
// a block of G threads.  Reductions run over RG lanes, in a block of several
// warps redundantly in each of them.
template <int G> struct FxGroup {
    static constexpr int RG = G < 32 ? G : 32;
    int gl, rl, shift;
    unsigned mask;
    __device__ __forceinline__ FxGroup()
    {
        const int lane = threadIdx.x & 31;
        gl = threadIdx.x & (G - 1);
        rl = gl & (RG - 1);
        shift = lane & ~(RG - 1);
        mask = RG == 32 ? FULL : ((1u << (RG & 31)) - 1u) << shift;
    }
    __device__ __forceinline__ void sync() const
    {
        if (G > 32) __syncthreads();
        else if (G > 1) __syncwarp(mask);
    }
    // lanes of the group (from the lowest) with p
    __device__ __forceinline__ unsigned ballot(bool p) const
    {
        return RG == 1 ? (unsigned)p : __ballot_sync(mask, p) >> shift;
    }
    __device__ __forceinline__ bool all(bool p) const { return ballot(!p) << (32 - RG) == 0; }
    // whether a matrix of the warp has p (p is the same on all lanes of a group).  The
    // groups of a warp share its votes in the QR sweeps, so they leave a solve together:
    // all 32 lanes call this.
    __device__ __forceinline__ bool any(bool p) const { return G < 32 ? __any_sync(FULL, p) : p; }
    __device__ __forceinline__ i64 sum(i64 v) const
    {
#pragma unroll
        for (int o = RG / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
        return v;
    }
    __device__ __forceinline__ i64 orr(i64 v) const
    {
#pragma unroll
        for (int o = RG / 2; o > 0; o >>= 1) v |= __shfl_xor_sync(mask, v, o);
        return v;
    }
    __device__ __forceinline__ int maxi(int v) const
    {
#pragma unroll
        for (int o = RG / 2; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(mask, v, o));
        return v;
    }
};

// G lanes that own one matrix in a warp's workspace: the warp holds 32 / G
// matrices, lane l works on matrix l % (32 / G), so that the lanes with one
// index of their groups touch neighbouring matrices.
// Its reductions and syncs are those of the whole warp: all 32 lanes call them.
template <int G> struct FxLanes {
    static constexpr int RG = G, M = 32 / G;
    int gl, rl;
    __device__ __forceinline__ FxLanes() : gl((threadIdx.x & 31) / M), rl(gl) {}
    __device__ __forceinline__ void sync() const { __syncwarp(); }
    template <class T, class F> __device__ __forceinline__ T fold(T v, F f) const
    {
#pragma unroll
        for (int o = M; o < 32; o <<= 1) v = f(v, __shfl_xor_sync(FULL, v, o));
        return v;
    }
    __device__ __forceinline__ bool all(bool p) const
    {
        return fold((int)p, [](int a, int b) { return a & b; });
    }
    __device__ __forceinline__ bool any(bool p) const { return __any_sync(FULL, p); }
    __device__ __forceinline__ i64 sum(i64 v) const
    {
        return fold(v, [](i64 a, i64 b) { return a + b; });
    }
    __device__ __forceinline__ i64 orr(i64 v) const
    {
        return fold(v, [](i64 a, i64 b) { return a | b; });
    }
    __device__ __forceinline__ int maxi(int v) const
    {
        return fold(v, [](int a, int b) { return max(a, b); });
    }
};

template <> struct FxLanes<1> : FxGroup<1> {};

__host__ __device__ __forceinline__ int fx_lda(int n) { return n | 1; }
// 16-byte elements of a matrix's slot in shared memory: H, Z (vectors only),
// and n entries for the reflectors' first elements and the column scales;
// padded so that the slots of a warp's matrices start G elements apart modulo
// 8 (eight lanes' 16-byte accesses fill the banks once).
__host__ __device__ __forceinline__ int fx_slot(int n, int G, bool vec)
{
    int e = (vec ? 2 : 1) * n * fx_lda(n) + n;
    if (G < 8) e += ((G - e % 8) + 8) % 8;
    return e;
}

// Row and column of element e = i - 1 + (j - 1) n, advanced without a division.
struct FxIndex {
    int i, j;
    __device__ __forceinline__ FxIndex(int e, int n) : i(e % n + 1), j(e / n + 1) {}
    __device__ __forceinline__ void next(int step, int n)
    {
        for (i += step; i > n; i -= n) ++j;
    }
};

struct FxOut {
    double *rE, *iE, *rV, *iV, *rT, *iT;
    long long sv, sm;  // element strides of vectors and matrices
};

// Trailing blocks that are large enough for one scale: bit 0, the block of order
// 2, bit 1, of order 4, bit 2, of order n / 2, bit 3, of order n - 1, where row or
// column r of the block that starts there (from its diagonal entry on) has an
// entry of size mt (high half).
//
// A block A(k:n, k:n) far below the rest, beside a strong row and column (a hub
// over near-degenerate levels): FP64 keeps its small eigenvalues to 2^-53 of the
// block if no transformation mixes the block with the strong entries, which is
// when it is small both in A and in the Hessenberg form; an absolute error of
// 2^-61 of the scale is the larger one then (n=8, block of 2^-14: 1e-12 of the
// eigenvalues against 2e-15, of 2^-26: 4e-9).  Where the strong row is not the
// first one, or there are two, or a block becomes small by cancellation only, FP64
// loses as much or more, and the matrix stays here.  The errors meet at a block
// of 2^-6 of the scale.  Blocks of few rows are as small as that by chance in
// large matrices, so their limits follow the entries of a Gaussian matrix, 2^-2.5
// of their size for order 2 (4e-8 of Hermitian ones fall below in A and in H) and
// 2^-0.5 for order 4; measured on 200,000 Gaussian and Hermitian matrices of n = 3
// .. 64: none is refused.
__device__ __forceinline__ int fx_blocks(const int n, const int r, const int mt)
{
    const int c = 32 - __clz(n - 1);  // n <= 2^c
    const int t4 = max(6, 2 + c), m4 = min(4, n - 1), mh = min(max(4, n / 2), n - 1);
    const int s = 30 - min(__clz(mt) - 1, 30);  // 2^s <= mt, or 0
    return (int)(r > n - 2 && s >= 25 - c) | (int)(r > n - m4 && s >= 29 - t4) << 1 | (int)(r > n - mh && s >= 23) << 2 |
           (int)(r > 1 && s >= 29 - t4) << 3;
}
constexpr int kFxBlocks = 7, kFxBlocksInA = 8;

// Functions below that are not inlined keep one copy of their code: the lane
// kernel's warps run out of step, and with everything inlined its code did not
// fit the instruction caches (n=16: 4.0 M/s on one wave, 2.6 M/s on eight).
// ST tells the memory space: 1 = shared, 32 = global.
template <int ST> __device__ __forceinline__ void fx_assume_space(const void *p)
{
#ifdef __CUDA_ARCH__
    if (ST == 1) __builtin_assume(__isShared(p));
    else __builtin_assume(__isGlobal(p));
#endif
}

// Does the graph of A's nonzero entries lead from index 1 to every other?  Where it
// does not (diagonal, triangular, block triangular matrices) the reduction meets a
// zero subdiagonal, at which the matrix would be refused after half the work: n=24 x
// 30,720 block-triangular, eigenvalues only, 23.9 -> 21.2 ms (as in FP64 alone), n=16
// x 100,000 50.0 -> 47.8 (46.8).
// One column's entries for a full matrix.
template <class GR, int ST>
__device__ __forceinline__ bool fx_connected(const GR &gr, const int n, const FxMat<ST> &H)
{
    const i64 all = (i64)(~0ULL >> (64 - n));
    i64 reached = 1, done = 0;
    for (;;) {
        const i64 todo = reached == all ? 0 : reached & ~done;
        if (!gr.any(todo != 0)) break;
        const int r = todo ? __ffsll(todo) : 1;
        i64 to = 0;
        for (int i = gr.rl + 1; i <= n; i += GR::RG) {
            const cx64 x = H.ld(i, r);
            to |= (i64)((x.r | x.i) != 0) << (i - 1);
        }
        reached |= gr.orr(to);
        done |= 1LL << (r - 1);
    }
    return reached == all;
}

// Load A (element e of the column-major matrix at e * s) into H as integers.
// Returns false for a matrix that is left to the FP64 kernels; unit = 2^(e-61);
// blocks: fx_blocks of A.
template <int G, bool kConnected, class GR, int ST>
__device__ __forceinline__ bool fx_load_inline(const GR &gr, const int n, const FxMat<ST> &H, const bool valid,
                                               const double *rA, const double *iA, const long long s, double &unit,
                                               int &blocks)
{
    unit = 1.0;
    int emax = 0;
    FxIndex i0(gr.gl, n);
    for (int e = gr.gl; e < n * n; e += G, i0.next(G, n)) {
        double re = 0.0, im = 0.0;
        if (valid) { re = rA[e * s]; im = iA[e * s]; }
        emax = max(emax, max(__double2hiint(re) & 0x7fffffff, __double2hiint(im) & 0x7fffffff));
        H.std(i0.i, i0.j, mk(re, im));
    }
    gr.sync();
    if (G > 32) {  // each warp reduces over the whole matrix
        for (int e = gr.rl; e < n * n; e += 32) {
            const cx<double> v = H.ldd(e % n + 1, e / n + 1);
            emax = max(emax, max(__double2hiint(v.r) & 0x7fffffff, __double2hiint(v.i) & 0x7fffffff));
        }
    }
    emax = gr.maxi(emax) >> 20;
    const bool range = valid && emax >= 128 && emax <= 1900;
    // ||A||_F^2 from above: |component| < (q + 1) 2^(emax - 1043), q its leading 21 bits
    i64 q2 = 0;
    FxIndex i1(gr.rl, n);
    for (int e = gr.rl; e < n * n; e += GR::RG, i1.next(GR::RG, n)) {
        const cx<double> v = H.ldd(i1.i, i1.j);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int hi = __double2hiint(c ? v.i : v.r) & 0x7fffffff, ex = hi >> 20;
            const int q = ((hi & 0xfffff) | 0x100000) >> min(emax - ex, 31);
            q2 += (i64)(q + 1) * (q + 1);
        }
    }
    q2 = gr.sum(q2);
    const int E = ((64 - __clzll(q2)) + 1) / 2 + emax - 1043;
    gr.sync();  // every warp has read the matrix
    if (range) {
        const double sc = __hiloint2double((61 - E + 1023) << 20, 0);
        unit = __hiloint2double((E - 61 + 1023) << 20, 0);
        FxIndex i2(gr.gl, n);
        for (int e = gr.gl; e < n * n; e += G, i2.next(G, n)) {
            const cx<double> v = H.ldd(i2.i, i2.j);
            H.st(i2.i, i2.j, {__double2ll_rn(v.r * sc), __double2ll_rn(v.i * sc)});
        }
    } else {
        FxIndex i2(gr.gl, n);
        for (int e = gr.gl; e < n * n; e += G, i2.next(G, n)) H.st(i2.i, i2.j, {0, 0});
    }
    gr.sync();
    // every row and column has an entry of at least 2^-9 of the scale
    bool ok = range;
    i64 large = 0;
    for (int r = gr.rl + 1; r <= n; r += GR::RG) {
        int mr = 0, mc = 0, mt = 0;
        for (int j = 1; j <= n; ++j) {
            const int a = fx_high(H.ld(r, j)), b = fx_high(H.ld(j, r));
            mr = max(mr, a);
            mc = max(mc, b);
            if (j >= r) mt = max(mt, max(a, b));
        }
        ok = ok && mr >= (1 << 20) && mc >= (1 << 20);
        large |= fx_blocks(n, r, mt);
    }
    blocks = (int)gr.orr(large);
    if (kConnected) ok = fx_connected(gr, n, H) && ok;
    // A(2:n, 2:n) is only rotated within itself: that it is small is known already
    return gr.all(ok && (blocks & kFxBlocksInA));
}
// One copy beside the kernel's own code, but for the shift-seeded kernel, which has it
// inlined and without fx_connected (a reflector refuses those matrices there): its code
// is the largest, and warps out of step over many waves miss the instruction cache.
// Whole solves, ms: plain n=16 x 1,048,576 266 (inlined 271 .. 274), shift-seeded n=24 x
// 1,048,576 622 (as a function 742; over 3.4 waves, 262,144, no different).
template <int G, class GR, int ST>
__device__ __noinline__ bool fx_load(const GR gr, const int n, const FxMat<ST> H, const bool valid, const double *rA,
                                     const double *iA, const long long s, double &unit, int &blocks)
{
    fx_assume_space<ST>(H.p);
    return fx_load_inline<G, true>(gr, n, H, valid, rA, iA, s, unit, blocks);
}

// Bring the line of p into L2 (no register is held for it).
__device__ __forceinline__ void fx_prefetch(const void *p)
{
#ifdef __CUDA_ARCH__
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
#endif
}

// a -= u (u^H a) for NB vectors a of m entries (vector b at a + b blk), or
// with conj(u) for u (cj): the reflector from the left on columns, or from the
// right on rows.  The first entry of u is u1, the others u[k * ustep].
template <int NB, int ST>
__device__ __noinline__ void fx_reflect(longlong2 *a, const int step, const int blk, const longlong2 *u,
                                        const int ustep, const i64 u1r, const i64 u1i, const int m, const bool cj)
{
    fx_assume_space<ST>(a);
    fx_assume_space<ST>(u);
    facc sr[NB], si[NB];
    longlong2 v[NB], uk = make_longlong2(u1r, u1i);
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        sr[b] = si[b] = fx_zero<61>();
        v[b] = a[b * blk];
    }
    longlong2 *p = a;
    for (int k = 0; k < m; ++k) {
        const cfx f = fx_split(cx64{uk.x, cj ? -uk.y : uk.y});
        const fx nf = fx_split(cj ? uk.y : -uk.y);
        cfx x[NB];
#pragma unroll
        for (int b = 0; b < NB; ++b) x[b] = fx_split(cx64{v[b].x, v[b].y});
        p += step;
        if (k + 1 < m) {  // the next entries
            uk = u[k * ustep];
#pragma unroll
            for (int b = 0; b < NB; ++b) v[b] = p[b * blk];
        }
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            fx_mac(sr[b], f.r, x[b].r);
            fx_mac(sr[b], f.i, x[b].i);
            fx_mac(si[b], f.r, x[b].i);
            fx_mac(si[b], nf, x[b].r);
            if ((k & 3) == 3) { fx_flush(sr[b]); fx_flush(si[b]); }
        }
    }
    cfx nz[NB];
    fx zi[NB];
    p = a;
    uk = make_longlong2(u1r, u1i);
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const i64 zr = fx_end<61>(sr[b]), zm = fx_end<61>(si[b]);
        nz[b] = fx_split(cx64{-zr, -zm});
        zi[b] = fx_split(zm);
        v[b] = p[b * blk];
    }
    for (int k = 0; k < m; ++k) {
        const cfx f = fx_split(cx64{uk.x, cj ? -uk.y : uk.y});
        longlong2 w[NB];
#pragma unroll
        for (int b = 0; b < NB; ++b) w[b] = v[b];
        longlong2 *const p1 = p + step;
        if (k + 1 < m) {
            uk = u[k * ustep];
#pragma unroll
            for (int b = 0; b < NB; ++b) v[b] = p1[b * blk];
        }
#pragma unroll
        for (int b = 0; b < NB; ++b)
            p[b * blk] = make_longlong2(w[b].x + fx_dot2<61>(nz[b].r, f.r, zi[b], f.i),
                                        w[b].y + fx_dot2<61>(nz[b].i, f.r, nz[b].r, f.i));
        p = p1;
    }
}
// vectors gl, gl + G, ... of count in A, kFxReflect at a time; u in H
constexpr int kFxReflect = 4;
template <int G, int ST>
__device__ __forceinline__ void fx_reflect_all(const int gl, const FxMat<ST> &A, longlong2 *a, const int step, const int blk,
                                               int count, const FxMat<ST> &H, const longlong2 *u, const cx64 u1,
                                               const int m, const bool cj)
{
    VES_CHECK_SPAN(A, a, (long long)(count - 1) * blk + (m - 1) * step, count);
    VES_CHECK_SPAN(H, u, (long long)(m - 2) * ST, count);
    constexpr int NB = G > 8 ? 1 : kFxReflect;  // larger groups have one or two vectors per lane
    int v = gl;
    if (NB > 1)
        for (; v + (NB - 1) * G < count; v += NB * G)
            fx_reflect<NB, ST>(a + v * blk, step, G * blk, u, ST, u1.r, u1.i, m, cj);
    for (; v < count; v += G) fx_reflect<1, ST>(a + v * blk, step, 0, u, ST, u1.r, u1.i, m, cj);
}

constexpr i64 kFxMinSub = 1LL << 31;  // 2^-30 of the scale

// Householder reduction to Hessenberg form with Hermitian reflectors
// P = I - u u^H, ||u||^2 = 2 (the subdiagonal comes out complex).  u_k, k >=
// i + 2, stays below the subdiagonal of column i, u_{i+1} in U(i).  ok turns
// false at a subdiagonal that fx_irreducible rejects; the reduction ends where
// no matrix is left for which it is needed (a batch of triangular or
// block-triangular matrices would otherwise pay for it twice).
template <int G, class GR, int ST>
__device__ __forceinline__ void fx_reduce(const GR &gr, const int n, const FxMat<ST> &H, const FxVec<ST> &U, bool &ok)
{
    constexpr int RG = GR::RG;
    const int rs = ST, cs = H.lda * ST;  // steps to the next row, the next column
    for (int i = 1; i <= n - 2; ++i) {
        const cx64 al = H.ld(i + 1, i);
        i64 o = 0;
        for (int k = i + 2 + gr.rl; k <= n; k += RG) { const cx64 x = H.ld(k, i); o |= fx_abs(x.r) | fx_abs(x.i); }
        o = gr.orr(o);
        // squared norm of the entries, to about 2^-55, as a sum of integers
        const int sh = o ? __clzll(o) - 2 : 0;  // |x| << sh < 2^62
        i64 q = 0;
        for (int k = i + 2 + gr.rl; k <= n; k += RG) {
            const cx64 x = H.ld(k, i);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const unsigned long long a = (unsigned long long)fx_abs(c ? x.i : x.r) << sh;
                const unsigned long long hi = __umul64hi(a, a);
                q += (i64)((hi + 4) >> 3);
            }
        }
        q = gr.sum(q);
        double scale = 0.0;  // u_k = x_k scale (units of 2^-61)
        cx64 u1 = {0, 0}, beta = al;
        if (o) {
            // q 2^67 / 2^(2 sh); the sum is unsigned (up to 2^64)
            const double xn2 = (double)(unsigned long long)q * __hiloint2double((67 - 2 * sh + 1023) << 20, 0);
            const double one = 2305843009213693952.0;  // 2^61
            const cx<double> a = fx_d(al);
            const double a2 = fma(a.r, a.r, a.i * a.i), n2 = a2 + xn2;
            const double ra = a2 > 0.0 ? rsqrt(a2) : 0.0;
            const cx<double> ph = a2 > 0.0 ? mk(a.r * ra, a.i * ra) : mk(1.0, 0.0);
            const double nrm = n2 * rsqrt(n2), s = fma(a2, ra, nrm);
            const double r = rsqrt(nrm * s);
            scale = r * one;
            u1 = {__double2ll_rn(ph.r * (s * scale)), __double2ll_rn(ph.i * (s * scale))};
            beta = {-__double2ll_rn(ph.r * nrm), -__double2ll_rn(ph.i * nrm)};
        }
        gr.sync();  // every lane has read column i
        for (int k = i + 2 + gr.gl; k <= n; k += G) {
            const cx64 x = H.ld(k, i);
            H.st(k, i, {__double2ll_rn((double)x.r * scale), __double2ll_rn((double)x.i * scale)});
        }
        if (gr.gl == 0) {
            U.st(i, u1);
            H.st(i + 1, i, beta);
        }
        gr.sync();
        ok = ok && fx_abs1(beta) >= kFxMinSub;
        if (!gr.any(ok)) return;
        const longlong2 *u = H.at(i + 2, i);
        fx_reflect_all<G, ST>(gr.gl, H, H.at(1, i + 1), cs, rs, n, H, u, u1, n - i, true);  // rows of A(:, i+1:n)
        gr.sync();
        fx_reflect_all<G, ST>(gr.gl, H, H.at(i + 1, i + 1), rs, cs, n - i, H, u, u1, n - i, false);  // columns of A(i+1:n, i+1:n)
        gr.sync();
    }
}

// Z = P_1 P_2 ... P_{n-2} from the reflectors.
template <int G, class GR, int ST>
__device__ __forceinline__ void fx_form_q(const GR &gr, const int n, const FxMat<ST> &H, const FxMat<ST> &Z,
                                          const FxVec<ST> &U)
{
    for (int c = gr.gl + 1; c <= n; c += G)
        for (int r = 1; r <= n; ++r) Z.st(r, c, {r == c ? 1LL << 61 : 0, 0});
    gr.sync();
    for (int i = n - 2; i >= 1; --i) {
        fx_reflect_all<G, ST>(gr.gl, Z, Z.at(i + 1, i + 1), ST, Z.lda * ST, n - i, H, H.at(i + 2, i), U.ld(i), n - i, false);
        gr.sync();
    }
}

// No subdiagonal below kFxMinSub, and no trailing block that is small in A
// (blocks) and in its Hessenberg form.
template <int G, class GR, int ST>
__device__ __forceinline__ bool fx_irreducible(const GR &gr, const int n, const FxMat<ST> &H, const int blocks)
{
    bool ok = true;
    for (int k = gr.rl + 2; k <= n; k += GR::RG) ok = ok && fx_abs1(H.ld(k, k - 1)) >= kFxMinSub;
    i64 large = blocks;
    if (gr.any((blocks & kFxBlocks) != kFxBlocks)) {
        for (int r = gr.rl + 1; r <= n; r += GR::RG) {
            int mt = r < n ? fx_high(H.ld(r + 1, r)) : 0;
            for (int j = r; j <= n; ++j) mt = max(mt, fx_high(H.ld(r, j)));
            large |= fx_blocks(n, r, mt);
        }
        large = gr.orr(large);
    }
    return gr.all(ok && (large & kFxBlocks) == kFxBlocks);
}

// Deflate at the bottom of the window [L, I] (the reference's test and sweep
// cap, which moves on) until an eigenvalue needs a sweep; false when none is
// left.  (a0, a1): the vector of the sweep's first rotation, from Wilkinson's
// shift or, at the 10th and 20th sweep, the reference's exceptional ones.
// sp: predicted shifts, in the units of H.  peers: with one lane's scan per lane
// (G = 1) but several lanes per matrix, those lanes.
template <int G, int ST, class SP = NoShiftPredictions>
__device__ __forceinline__ bool fx_next_sweep(const FxGroup<G> &gr, const int n, const FxMat<ST> &H,
                                              const FxVec<ST> &S, const int max_its, int &I, int &L, int &its,
                                              int &status, cx<double> &a0, cx<double> &a1, SP *sp = nullptr,
                                              const unsigned peers = 0)
{
    constexpr int RG = FxGroup<G>::RG;
    for (;;) {
        if (I <= 1) return false;
        if (its > max_its) { status |= ST_ITCAP; --I; L = 1; its = 0; continue; }
        // the largest K in (L, I] whose subdiagonal is negligible, else L
        int K = L;
        if (RG == 1) {  // one lane per matrix: each diagonal entry is read once, one ahead
            cx64 d2 = H.ld(I, I), d1 = L < I ? H.ld(I - 1, I - 1) : d2;
            cx<double> s = L < I ? S.ldd(I - 1) : mk(0.0, 0.0);
            for (int k = I; k > L; --k) {
                const cx64 e2 = d2, e1 = d1;
                const cx<double> es = s;
                if (k - 1 > L) { d1 = H.ld(k - 2, k - 2); s = S.ldd(k - 2); }
                d2 = e1;
                if (fx_negligible(H, S, k, n, es, e1, e2)) { K = k; break; }
            }
        } else for (int top = I; top > L; top -= RG) {
            const int k = top - gr.rl;
            const unsigned b = gr.ballot(k > L && fx_negligible(H, S, k > L ? k : L + 1, n)) &
                               (RG == 32 ? FULL : (1u << (RG & 31)) - 1u);
            if (b) { K = top - (__ffs(b) - 1); break; }
        }
        L = K;
        if (G > 32) __syncthreads();  // the scans have read S
        else if (peers) __syncwarp(peers);
        if (L > 1) S.std(L - 1, mk(0.0, 0.0));  // every lane: the same value
        if (L >= I) {
            if constexpr (SP::kOn) sp->deflated(its);
            --I; L = 1; its = 0;
            continue;
        }
        const cx64 hll = H.ld(L, L);
        a1 = S.ldd(L);
        const cx<double> si = S.ldd(I - 1);
        cx64 t = H.ld(I, I);
        if (its == 10) {
            t = hll;
            t.r += __float2ll_rn(0.75f * fx_absf(fx_float(a1, 0)));
        } else if (its == 20) {
            t.r += __float2ll_rn(0.75f * fx_absf(fx_float(si, 0)));
        } else {
            const cx64 u = H.ld(I - 1, I), d = H.ld(I - 1, I - 1);
            const float k = 0x1p-61f;
            const cx<float> w = fx_wilkinson(mk((float)(d.r - t.r) * (0.5f * k), (float)(d.i - t.i) * (0.5f * k)),
                                             mk((float)u.r * k, (float)u.i * k), fx_float(si, -61));
            cx64 c = {__float2ll_rn(w.r * 0x1p61f), __float2ll_rn(w.i * 0x1p61f)};
            if (L == I - 1) fx_wilkinson_2x2(c, {d.r - t.r, d.i - t.i}, u, fx_i(si));
            t.r -= c.r;
            t.i -= c.i;
        }
        if constexpr (SP::kOn) {
            const cx<double> t0 = fx_d(t);
            cx<double> td = t0;
            sp->template pick<double>(its, I, td, (double)fx_absf(fx_float(si, 0)));
            if (td.r != t0.r || td.i != t0.i) t = fx_i(td);
        }
        a0 = fx_d(cx64{hll.r - t.r, hll.i - t.i});
        ++its;
        return true;
    }
}

// Single-shift QR (reference Toolbox.hpp:690-1031): the same deflation test,
// exceptional shifts and sweep cap as zlahqr_warp, with rotations of real
// cosine, so the subdiagonals stay complex and need no phase fix.  The
// matrices of a warp move in lockstep per sweep, each group with its own
// window [L, I].  kVec = false: the active block only, no Z.
//
// The subdiagonals and the bulge stay in FP64 (S(k) = H(k+1, k)): they
// become small against the matrix as the iteration converges, and the rotation
// that a small pair defines must keep its relative accuracy for the shift to
// reach the end of the window.  With them in fixed point (an absolute
// rounding) the transformations are as accurate, but the subdiagonals stall at
// 2^-46 of the matrix.  Every other entry is only rotated.
//
// The FP64 steps of a rotation are spread over the lanes of a quad: an FP64
// instruction holds a quarter of an SM for 62 cycles however many lanes need
// it, and the chain of them is what a group waits for.  Lanes 0 and 1 of a quad
// work on the real and imaginary part of the pair's first number (and of what
// becomes the next first number), lanes 2 and 3 on the second; the other lanes
// of the group repeat them.  The operations on each value are those of fx_rot
// and of fx_qr_lane.
template <int G, bool kVec, int ST>
__device__ __forceinline__ void fx_qr(const FxGroup<G> &gr, const int n, const FxMat<ST> &H, const FxMat<ST> &Z, const FxVec<ST> &S,
                                      const bool run, const int max_its, int &sweeps, int &status)
{
    static_assert(G >= 4, "the scalar steps are spread over four lanes");
    const int role = gr.gl & 3;
    const bool im = role & 1, second = role >= 2;
    const unsigned mk4 = gr.mask;
    const auto from = [&](double v, int lane) { return __shfl_sync(mk4, v, lane, 4); };
    const double one = 4611686018427387904.0;  // 2^62
    int I = n, L = 1, its = 0;
    bool done = !run || n <= 1;
    for (;;) {
        cx<double> z, a1;
        const bool sweep = !done && fx_next_sweep<G>(gr, n, H, S, max_its, I, L, its, status, z, a1);
        done = !sweep;
        sweeps += sweep;
        double sub = im ? a1.i : a1.r;  // lanes 0, 1: H(K+1, K)
        if (second) z = a1;             // the lane's number of the pair
        int Kmin, Kmax;
        if (G < 32) {
            if (!__any_sync(FULL, sweep)) break;
            Kmin = __reduce_min_sync(FULL, sweep ? L : INT_MAX);
            Kmax = __reduce_max_sync(FULL, sweep ? I - 1 : 0);
        } else {
            if (!sweep) break;
            Kmin = L;
            Kmax = I - 1;
        }
        gr.sync();
        if (G < 32) __syncwarp();
        const int jmax = kVec ? n : I, jmin = kVec ? 1 : L;
        for (int K = Kmin; K <= Kmax; ++K) {
            if (sweep && K >= L && K < I) {
                const cx64 hk = H.ld(K, K);
                const cx<double> nxt = K + 1 < I ? S.ldd(K + 1) : mk(0.0, 0.0);  // H(K+2, K+1)
                const double hc = (double)(im ? hk.i : hk.r);
                const i64 isub = __double2ll_rn(sub);
                // fx_rot
                const double m2 = fma(z.r, z.r, z.i * z.i);
                const double f = from(m2, 0), g = from(m2, 2);
                const double n2 = f + g, w = f * n2;
                const bool deg = !(w > 1e-280);
                const double p = rsqrt(deg ? fmax(g, 1e-280) : w);
                const double x1r = from(z.r, 2), x1i = from(z.i, 2);
                const double a = deg ? 1.0 : from(z.r, 0), b = deg ? 0.0 : from(z.i, 0);
                double v = fma(im ? b : a, x1r, (im ? -a : b) * x1i);  // s / p
                if (second) v = im ? (deg ? g : n2) : f;
                v *= p;  // Re s, Im s, c, n2 p
                if (deg) {
                    if (role == 2) v = g > 1e-280 ? 0.0 : 1.0;
                    if (!second && !(g > 1e-280)) v = 0.0;
                }
                const double np = from(v, 3), dc = from(v, 2);
                const cx<double> ks = mk(from(v, 0), -from(v, 1));  // conj(s)
                const i64 iv = __double2ll_rn(v * one);
                const FxCoef C(__shfl_sync(mk4, iv, 2, 4), __shfl_sync(mk4, iv, 0, 4), __shfl_sync(mk4, iv, 1, 4)),
                    CC = C.columns();
                const double rc = (im ? b : a) * np;  // lanes 0, 1: r
                // lanes 0, 1: x1 = c sub - conj(s) h_kk, H(K+1, K) after the row operation;
                // lanes 2, 3: the bulge conj(s) H(K+2, K+1)
                const double hr = from(hc, 0), hi = from(hc, 1);
                double t = second ? (im ? ks.r : -ks.i) * nxt.i : sub * dc;
                t = fma(second ? (im ? ks.i : ks.r) : (im ? -ks.i : -ks.r), second ? nxt.r : hr, t);
                if (!second) t = fma(im ? -ks.r : ks.i, hi, t);
                const i64 ix1 = __double2ll_rn(t);
                const cx64 sx1 = {__shfl_sync(mk4, ix1, 0, 4), __shfl_sync(mk4, ix1, 1, 4)};
                const cx64 ssub = {__shfl_sync(mk4, isub, 0, 4), __shfl_sync(mk4, isub, 1, 4)};
                gr.sync();  // every lane has read H(K, K) and S
                if (K > L && gr.gl < 2) reinterpret_cast<double *>(S.at(K - 1))[gr.gl] = rc;
                // rows K, K+1 of columns K..jmax; H(K+1, K) is the FP64 subdiagonal
                for (int j = K + gr.gl; j <= jmax; j += G) {
                    cx64 y1 = H.ld(K, j), y2 = H.ld(K + 1, j);
                    if (j == K) y2 = ssub;
                    fx_pair(y1, y2, C);
                    H.st(K, j, y1);
                    if (j > K) H.st(K + 1, j, y2);
                }
                gr.sync();
                // a0 = c x1 + conj(s) h_k+1,k+1; sub = c H(K+2, K+1)
                const cx64 h2 = H.ld(K + 1, K + 1);
                const double xc = (double)(im ? h2.i : h2.r);
                const double xr = from(xc, 0), xi = from(xc, 1);
                double u = (second ? (im ? nxt.i : nxt.r) : t) * dc;
                const double nsub = __shfl_xor_sync(mk4, u, 2, 4);  // lanes 0, 1: from lanes 2, 3
                if (!second) {
                    u = fma(im ? ks.i : ks.r, xr, u);
                    u = fma(im ? ks.r : -ks.i, xi, u);
                    t = u;
                }
                sub = nsub;
                const double other = __shfl_xor_sync(mk4, t, 1, 4);
                z = im ? mk(other, t) : mk(t, other);
                gr.sync();  // every lane has read H(K+1, K+1)
                // columns K, K+1 of H (rows up to K+1), then of Z
                const int nc = K + 2 - jmin;
                for (int q = gr.gl; q < nc + (kVec ? n : 0); q += G) {
                    const bool h = !kVec || q < nc;
                    const int row = h ? K + 1 - q : q - nc + 1;
                    longlong2 *p1 = h ? H.at(row, K) : Z.at(row, K), *p2 = h ? H.at(row, K + 1) : Z.at(row, K + 1);
                    const longlong2 w1 = *p1, w2 = *p2;
                    cx64 y1 = {w1.x, w1.y}, y2 = {w2.x, w2.y};
                    if (q == 0) y1 = sx1;
                    fx_pair(y1, y2, CC);
                    if (q != 0) *p1 = make_longlong2(y1.r, y1.i);
                    *p2 = make_longlong2(y2.r, y2.i);
                }
                if (K == I - 1 && gr.gl < 2) reinterpret_cast<double *>(S.at(I - 1))[gr.gl] = t;
                gr.sync();
            }
            if (G < 32) __syncwarp();
        }
    }
}

// Rotations of the current chunk of a sweep, in shared memory, one set per lane.
// (n=16, one lane per matrix, chunk 4, 8, 16: 277, 274, 260 ms per 1,048,576)
constexpr int kFxChunk = 16;
// k: rotations of a chunk; slots: 16-byte elements per lane, those and (G > 1) the
// lane's rows of the chunk
template <int G> struct FxChunkOf {
    static constexpr int k = G == 1 ? kFxChunk : 8;
    static constexpr int slots = k + (G > 1 ? k / G : 0);
};
constexpr int kFxStream = 2;  // chains streamed together
struct FxChunk {
    longlong2 *cs;  // (c, sr) of rotation k at cs[k * 32]
    i64 *si;
    __device__ __forceinline__ void put(int k, const FxRot &q) const
    {
        VES_CHECK_LT(k, kFxChunk);
        cs[k * 32] = make_longlong2(q.c, q.sr);
        si[k * 32] = q.si;
    }
    __device__ __forceinline__ FxCoef get(int k) const
    {
        VES_CHECK_LT(k, kFxChunk);
        const longlong2 a = cs[k * 32];
        return FxCoef(a.x, a.y, si[k * 32]);
    }
    // G > 1: entry of the lane's row t of the chunk in the column that the next rotation turns
    template <int G> __device__ __forceinline__ longlong2 *row(int t) const
    {
        VES_CHECK_LT(t, FxChunkOf<G>::k / G);
        return cs + (FxChunkOf<G>::k + t) * 32;
    }
};

// Apply ns rotations (c, s at cs[k * 32], si[k * 32]) to NB chains of entries:
// chain b's entries at p + b blk + k step, rotation k on entries k and k + 1,
// from the left or, with conj(s) for s, from the right (col).  The entry that
// two rotations share stays in registers, so each entry is read and written
// once per chunk.
//
// next (nullable): the chains that the caller streams after these; their lines
// are brought into L2 meanwhile.
// One rotation's entries ahead in registers, 16 warps keep 16 KB in flight per
// SM, which against the latency of DRAM is 4.7 TB/s at most; with the lines
// already in L2 the registers cover what is left.
template <int NB>
__device__ __noinline__ void fx_stream(longlong2 *p, const int step, const int blk, const longlong2 *cs, const i64 *si,
                                       const int ns, const bool col, const longlong2 *next, const int next_step)
{
    fx_assume_space<32>(p);
    fx_assume_space<1>(cs);
    fx_assume_space<1>(si);
    cx64 x[NB];
    longlong2 y[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const longlong2 v = p[b * blk];
        x[b] = {v.x, v.y};
        y[b] = p[b * blk + step];
    }
    for (int k = 0; k < ns; ++k) {
        const longlong2 c = cs[k * 32];
        const i64 s = si[k * 32];
        const FxCoef q(c.x, c.y, col ? -s : s);
        longlong2 *const p1 = p + step;
        cx64 z[NB];
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            z[b] = {y[b].x, y[b].y};
            if (k + 1 < ns) y[b] = p1[b * blk + step];  // the next rotation's entries
            if (next) fx_prefetch(next + b * blk);
        }
        if (next) next += next_step;
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            fx_pair(x[b], z[b], q);
            p[b * blk] = make_longlong2(x[b].r, x[b].i);
            x[b] = z[b];
        }
        p = p1;
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) p[b * blk] = make_longlong2(x[b].r, x[b].i);
}
template <int G, int ST>
__device__ __forceinline__ void fx_stream_all(const int gl, const FxMat<ST> &A, longlong2 *p, const int step, const int blk,
                                              int count, const FxChunk &ch, const int ns, const bool col)
{
    VES_CHECK_SPAN(A, p, (long long)(count - 1) * blk + (long long)ns * step, count);
    int b = G == 1 ? 0 : gl;  // chains gl, gl + G, ... of count
    for (; b + kFxStream * G <= count + G - 1; b += kFxStream * G) {
        const bool more = b + 2 * kFxStream * G <= count + G - 1;
        fx_stream<kFxStream>(p + b * blk, step, G * blk, ch.cs, ch.si, ns, col, more ? p + (b + kFxStream * G) * blk : nullptr,
                             more ? step : 0);
    }
    for (; b < count; b += G) fx_stream<1>(p + b * blk, step, blk, ch.cs, ch.si, ns, col, nullptr, 0);
}

// fx_qr for one matrix per lane, or per G lanes of FxLanes, the warp's matrices
// in lockstep per sweep, in its workspace.  The lanes of a matrix compute the
// chain alike and share out the rows and columns.  A sweep runs in chunks of
// FxChunkOf<G>::k rotations: first the chain of rotations, which needs of the
// matrix only the chunk's own columns (the left rotations of the chunk are
// applied to column K + 1 when rotation K is due) and the diagonal; then the
// chunk's rotations are streamed over the rows of Z, the rows above and the
// columns to the right.  A lane whose window does not contain K takes part with
// the identity, which leaves integers unchanged.  The entries see the same
// operations as in fx_qr.
//
// G > 1: every lane reads column K + 1 and S(K + 1) as they were before rotation
// K, so nothing of them may be written before all lanes have read them.  A row's
// owner therefore keeps its entry of column K + 1 in shared memory until rotation
// K + 1 has turned it, column K is written after the barrier that opens rotation
// K, and the diagonal stays in registers to the end of the chunk.
template <int G, bool kVec, int ST, class SP>
__device__ __forceinline__ void fx_qr_lane(const int group_lane, const int n, const FxMat<ST> &H, const FxMat<ST> &Z, const FxVec<ST> &S,
                                           const FxChunk &ch, const bool run, const int max_its, int &sweeps,
                                           int &status, SP *sp)
{
    const FxGroup<1> gr;  // a lane scans its matrix by itself
    constexpr int kChunk = FxChunkOf<G>::k;
    const int rs = ST, cs = n * ST;  // steps to the next row, the next column
    const int gl = G == 1 ? 0 : group_lane;
    unsigned peers = 0;  // the lanes of this matrix
    if (G > 1)
        for (int t = 0; t < G; ++t) peers |= 1u << ((threadIdx.x & (32 / G - 1)) + t * (32 / G));
    int I = n, L = 1, its = 0;
    bool done = !run || n <= 1;
    for (;;) {
        cx<double> a0, a1, sub;
        const bool sweep = !done && fx_next_sweep<1>(gr, n, H, S, max_its, I, L, its, status, a0, a1, sp, peers);
        done = !sweep;
        sub = a1;
        sweeps += sweep;
        if (!__any_sync(FULL, sweep)) break;
        const int Kmin = __reduce_min_sync(FULL, sweep ? L : INT_MAX);
        const int Kmax = __reduce_max_sync(FULL, sweep ? I - 1 : 0);
        cx64 hkk = H.ld(Kmin, Kmin);
        for (int Kc = Kmin; Kc <= Kmax; Kc += kChunk) {
            const int Ke = min(Kc + kChunk - 1, Kmax), ns = Ke - Kc + 1;
            for (int K = Kc; K <= Ke; ++K) {
                const bool act = sweep && K >= L && K < I;
                FxRot R;
                R.dc = 1.0;
                R.ds = mk(0.0, 0.0);
                R.c = 1LL << 62;
                R.sr = R.si = 0;
                if (G > 1) __syncwarp();  // what this rotation writes has been read
                // column K + 1: the chunk's left rotations so far; each row that is done takes
                // rotation K from the right, with its entry of column K
                longlong2 *pc = H.at(Kc, K + 1), *pl = H.at(Kc, K);
                longlong2 v = pc[0], w = G == 1 ? pl[0] : v;
                cx64 x = {v.x, v.y};
                v = pc[rs];
                cx<double> r, nxt = mk(0.0, 0.0);
                if (act) {
                    R = fx_rot(a0, a1, r);
                    if (K + 1 < I) nxt = S.ldd(K + 1);
                }
                ch.put(K - Kc, R);
                const FxCoef C(R), CC = C.columns();
                int turned = K - Kc;
                VES_CHECK_SPAN(H, pc, (K + 1 - Kc) * rs, turned);
                VES_CHECK_SPAN(H, pl, (K - Kc) * rs, turned);
                for (int q = 0; q < turned; ++q) {
                    cx64 y = {v.x, v.y};
                    v = pc[2 * rs];
                    fx_pair(x, y, ch.get(q));
                    if (G == 1) {
                        cx64 z = {w.x, w.y};
                        w = pl[rs];
                        fx_pair(z, x, CC);
                        pl[0] = make_longlong2(z.r, z.i);
                        pc[0] = make_longlong2(x.r, x.i);
                    } else if ((q & (G - 1)) == gl) {  // the rows of a chunk are shared out
                        longlong2 *const row = ch.row<G>(q / G);
                        cx64 z = {row->x, row->y};
                        fx_pair(z, x, CC);
                        pl[0] = make_longlong2(z.r, z.i);
                        *row = make_longlong2(x.r, x.i);
                    }
                    x = y;
                    pc += rs;
                    pl += rs;
                }
                // rows K, K + 1; H(K+1, K) is the FP64 subdiagonal
                cx64 y = {v.x, v.y}, y2 = act ? fx_i(sub) : cx64{0, 0};
                const cx64 h0 = hkk;
                fx_pair(x, y, C);
                fx_pair(hkk, y2, C);
                fx_pair(hkk, x, CC);
                if (((K - Kc) & (G - 1)) == gl) {
                    pl[0] = make_longlong2(hkk.r, hkk.i);
                    *(G == 1 ? pc : ch.row<G>((K - Kc) / G)) = make_longlong2(x.r, x.i);
                }
                if (act) {
                    const cx<double> ks = conj(R.ds);
                    const cx<double> x1 = cnmac(cscal(sub, R.dc), ks, fx_d(h0));  // H(K+1, K) after the row operation
                    if (K > L && gl == 0) S.std(K - 1, r);
                    a0 = cmac(cscal(x1, R.dc), ks, fx_d(y));
                    a1 = cmul(ks, nxt);  // the bulge H(K+2, K)
                    sub = cscal(nxt, R.dc);
                    cx64 z1 = fx_i(x1);
                    fx_pair(z1, y, CC);
                    if (K == I - 1 && gl == 0) S.std(I - 1, a0);
                }
                hkk = y;
                if (G == 1) H.st(K + 1, K + 1, y);
            }
            if (G > 1) {
                __syncwarp();  // column Ke + 1 has been read
                for (int q = gl; q < ns; q += G) *H.at(Kc + q, Ke + 1) = *ch.row<G>(q / G);
                if (gl == 0) H.st(Ke + 1, Ke + 1, hkk);
                __syncwarp();
            }
            // rows above the chunk
            const int r0 = kVec ? 1 : Kmin;
            if (Kc > r0) fx_stream_all<G>(gl, H, H.at(r0, Kc), cs, rs, Kc - r0, ch, ns, true);
            if (kVec) fx_stream_all<G>(gl, Z, Z.at(1, Kc), cs, rs, n, ch, ns, true);
            const int je = kVec ? n : Kmax + 1;
            if (je > Ke + 1) fx_stream_all<G>(gl, H, H.at(Kc, Ke + 2), rs, cs, je - Ke - 1, ch, ns, false);
            if (G > 1) __syncwarp();
        }
    }
}

// T-eigenvectors (ztrevc back substitution) on H converted to FP64, x of
// column k in row k of H's lower triangle; then V = Z X in Z, in FP64.
template <int G, class GR, int ST>
__device__ __forceinline__ void fx_vectors(const GR &gr, const int n, const FxMat<ST> &H, const FxMat<ST> &Z,
                                           const FxVec<ST> &U)
{
    const double ulp = lim<double>::eps();
    const int nsets = (n + G - 1) / G;
    for (int t = 0; t < nsets; ++t) {
        const int ki = t * G + gr.gl + 1, kmax = min(n, (t + 1) * G);
        const bool own = ki <= n;
        const cx<double> tkk = own ? H.ldd(ki, ki) : mk(0.0, 0.0);
        // entries of T are integers: a difference is 0 or at least 1
        const double smin = fmax(ulp * cabs1(tkk), 0.25);
        double s = 1.0;
        if (own)
            for (int k = 1; k < ki; ++k) { const cx<double> v = H.ldd(k, ki); H.std(ki, k, mk(-v.r, -v.i)); }
        for (int j = kmax - 1; j >= 1; --j) {
            if (own && j < ki) {
                cx<double> d = csub(H.ldd(j, j), tkk);
                if (cabs1(d) < smin) d = mk(smin, 0.0);
                cx<double> xj = H.ldd(ki, j);
                // |x_j / d| about to exceed 1e150 (an exponent difference of 498): scale the vector
                const int ex = max(__double2hiint(xj.r) & 0x7fffffff, __double2hiint(xj.i) & 0x7fffffff) >> 20;
                const int ed = max(__double2hiint(d.r) & 0x7fffffff, __double2hiint(d.i) & 0x7fffffff) >> 20;
                if (ex - ed > 497) {
                    const double f = __hiloint2double((1023 - (ex - ed)) << 20, 0);
                    for (int i = 1; i < ki; ++i) H.std(ki, i, cscal(H.ldd(ki, i), f));
                    xj = cscal(xj, f);
                    s *= f;
                }
                const double rd = 1.0 / fma(d.r, d.r, d.i * d.i);
                xj = cscal(cmulc(xj, d), rd);
                H.std(ki, j, xj);
                for (int i = j - 1; i >= 1; --i) H.std(ki, i, cnmac(H.ldd(ki, i), H.ldd(i, j), xj));
            }
        }
        if (own) U.std(ki, mk(s, 0.0));  // scale of the unit entry
    }
    gr.sync();
    for (int r = gr.gl + 1; r <= n; r += 2 * G) {  // two rows of Z at a time, columns n down to 2
        const bool two = r + G <= n;
        const int r2 = two ? r + G : r;
        for (int ki = n; ki >= 2; --ki) {
            const double s = U.ldd(ki).r;
            cx<double> a = cscal(Z.ldd(r, ki), s), b = cscal(Z.ldd(r2, ki), s);
            for (int q = 1; q < ki; ++q) {
                const cx<double> x = H.ldd(ki, q);
                a = cmac(a, Z.ldd(r, q), x);
                if (two) b = cmac(b, Z.ldd(r2, q), x);
            }
            Z.std(r, ki, a);
            if (two) Z.std(r2, ki, b);
        }
    }
    gr.sync();
}

// Predicted shifts of the lane kernel (the learned-shift form).
struct FxNoShifts {
    static constexpr bool kOn = false;
    typedef NoShiftPredictions Picker;
};

// newton64_shifts_lane on the fixed-point Hessenberg matrix (units of H; its
// FP64 subdiagonals in Sub), for two predictions at a time: they share each
// entry's conversion to FP64.  Hf: FP32 copy of H in units of 2^61.  w: 5 n
// elements of scratch (x and x' of the two, the inverse subdiagonals).
__device__ __forceinline__ void fx_newton(const int n, const FxMat<32> &H, const FxVec<32> &Sub, const MatIlv<float> &Hf,
                                          const VecIlv<double> &P, double2 *w, const double maxstep)
{
    const VecIlv<double> X[2] = {{w}, {w + n * 32}}, Inv{w + 4 * n * 32};
    const int lane = threadIdx.x & 31;
    float2 *const f = reinterpret_cast<float2 *>(w - lane + 2 * n * 32) + lane;
    const VecIlv<float> D[2] = {{f}, {f + n * 32}};
    for (int i = 2; i <= n; ++i) Inv.st(i, cinv(Sub.ldd(i - 1)));
    for (int k = 1; k <= n; k += 2) {
        cx<double> s[2], x[2];
        cx<float> sf[2], d[2];
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            s[b] = P.ld(min(k + b, n));
            sf[b] = mk((float)(s[b].r * 0x1p-61), (float)(s[b].i * 0x1p-61));
            x[b] = mk(1.0, 0.0);
            d[b] = mk(0.f, 0.f);
            X[b].st(n, x[b]);
            D[b].st(n, d[b]);
        }
        cx<double> acc[2];
        cx<float> dacc[2];
        for (int i = n; i >= 1; --i) {
            const cx<double> hii = fx_d(H.ld(i, i));
            const cx<float> hf = Hf.ld(i, i);
#pragma unroll
            for (int b = 0; b < 2; ++b) {  // x(i), x'(i) are in x, d
                acc[b] = cmul(csub(hii, s[b]), x[b]);
                dacc[b] = csub(cmul(csub(hf, sf[b]), d[b]), mk((float)x[b].r, (float)x[b].i));
            }
            for (int j = i + 1; j <= n; ++j) {
                const cx<double> h = fx_d(H.ld(i, j));
                const cx<float> g = Hf.ld(i, j);
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    acc[b] = cmac(acc[b], h, X[b].ld(j));
                    dacc[b] = cmac(dacc[b], g, D[b].ld(j));
                }
            }
            if (i == 1) break;
            const cx<double> inv = Inv.ld(i);
            const cx<float> invf = mk((float)(inv.r * 0x1p61), (float)(inv.i * 0x1p61));
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                x[b] = cmul(mk(-acc[b].r, -acc[b].i), inv);
                d[b] = cmul(mk(-dacc[b].r, -dacc[b].i), invf);
                if (cabs1(x[b]) > 1e18) {
                    for (int j = i; j <= n; ++j) {
                        X[b].st(j, cscal(X[b].ld(j), 1e-18));
                        D[b].st(j, cscal(D[b].ld(j), 1e-18f));
                    }
                    x[b] = cscal(x[b], 1e-18);
                    d[b] = cscal(d[b], 1e-18f);
                }
                X[b].st(i - 1, x[b]);
                D[b].st(i - 1, d[b]);
            }
        }
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            if (k + b > n) continue;
            const cx<double> delta = cdiv(acc[b], mk((double)dacc[b].r, (double)dacc[b].i));
            if (!nonfinite(delta.r) && !nonfinite(delta.i) && cabs1(delta) <= maxstep) P.st(k + b, csub(s[b], delta));
        }
    }
}

struct FxShifts {
    static constexpr bool kOn = true;
    typedef ShiftPredictions Picker;
    VecIlv<double> P;   // the matrix's predictions, as given (or polished by the pre-pass)
    MatIlv<float> Hf;   // FP32 copy of H
    longlong2 *scratch;  // 6 n elements, free until Q is formed
    int polish, newton, sweeps_used;
    float gate;
    ShiftPredictions sp;
    // rA, iA (stride s): the matrix; unit: the units of H
    __device__ __forceinline__ ShiftPredictions *prepare(const int n, const FxMat<32> &H, const FxVec<32> &Sub,
                                                         const bool ok, const double *rA, const double *iA,
                                                         const long long s, const double unit)
    {
        double fro2 = 0.0;
        const double iu = 1.0 / unit;  // a power of two
        if (ok) {
            for (int e = 0; e < n * n; ++e) fro2 = fma(iA[e * s], iA[e * s], fma(rA[e * s], rA[e * s], fro2));
            const double scale = sqrt(fro2 / (double)n);
            if (polish > 0 || newton > 0)
                for (int j = 1; j <= n; ++j)
                    for (int i = 1; i <= (j + 1 < n ? j + 1 : n); ++i) {
                        const cx<double> h = i == j + 1 ? Sub.ldd(j) : fx_d(H.ld(i, j));
                        Hf.st(i, j, mk((float)(h.r * 0x1p-61), (float)(h.i * 0x1p-61)));
                    }
            // FP32 steps in units of 2^61 of H, then everything in the units of H
            const double nu = iu * 0x1p-61;
            for (int k = 1; k <= n; ++k) P.st(k, cscal(P.ld(k), nu));
            if (polish > 0) {
                const float tol = (float)(1e-6 * scale * nu), keep = (float)(1e-3 * scale * nu), dup = (float)(1e-5 * scale * nu);
                if (n <= 16) polish_shifts_lane<16>(n, Hf, P, polish, tol, keep, dup);
                else if (n <= 32) polish_shifts_lane<32>(n, Hf, P, polish, tol, keep, dup);
                else polish_shifts_lane<64>(n, Hf, P, polish, tol, keep, dup);
            }
            for (int k = 1; k <= n; ++k) P.st(k, cscal(P.ld(k), 0x1p61));
            if (n >= 2)
                for (int t = 0; t < newton; ++t)
                    fx_newton(n, H, Sub, Hf, P, reinterpret_cast<double2 *>(scratch), 1e-4 * scale * iu);
        }
        sp.S = P;
        sp.n = n;
        sp.sweeps = sweeps_used;
        sp.gate = (double)gate * sqrt(fro2 / (double)n) * iu;
        sp.used = 0;
        sp.current = -1;
        sp.fallbacks = 0;
        return &sp;
    }
};

// The whole solve of one matrix per group, with H, Z (vectors only) and U (n
// entries) its storage.  Returns false (group-uniform) for a valid matrix
// that is left to the FP64 kernels; nothing is written then.
template <int G, bool kVec, class GR, int ST, class SH = FxNoShifts>
__device__ __forceinline__ bool fx_solve(const GR &gr, const int n, const FxMat<ST> &H, const FxMat<ST> &Z,
                                         const FxVec<ST> &U, const bool valid, const double *rA, const double *iA,
                                         const long long s, const FxOut &o, const int max_its, const int vnorm,
                                         int &sweeps, int &status, const FxChunk ch = {}, SH *shifts = nullptr)
{
    double unit;
    int blocks;
    bool ok;
    if constexpr (SH::kOn) ok = fx_load_inline<G, false>(gr, n, H, valid, rA, iA, s, unit, blocks);
    else ok = fx_load<G>(gr, n, H, valid, rA, iA, s, unit, blocks);
    if (gr.any(ok)) fx_reduce<G>(gr, n, H, U, ok);
    if (gr.any(ok)) {
        const bool irreducible = fx_irreducible<G>(gr, n, H, blocks);  // every lane takes part, whatever ok is
        ok = ok && irreducible;
    }
    if (!gr.any(ok)) {
        gr.sync();
        return false;
    }
    typename SH::Picker *sp = nullptr;
    if constexpr (SH::kOn) {
        const FxVec<32> Sub{shifts->scratch + 5 * n * 32};
        for (int k = 1; k < n; ++k) Sub.std(k, fx_d(H.ld(k + 1, k)));
        sp = shifts->prepare(n, H, Sub, ok, rA, iA, s, unit);
    }
    if (kVec) fx_form_q<G>(gr, n, H, Z, U);
    // subdiagonals in FP64 from here on
    for (int k = gr.gl + 1; k < n; k += G) U.std(k, fx_d(H.ld(k + 1, k)));
    gr.sync();
    if constexpr (ST > 1) fx_qr_lane<G, kVec>(gr.gl, n, H, Z, U, ch, ok, max_its, sweeps, status, sp);
    else fx_qr<G, kVec>(gr, n, H, Z, U, ok, max_its, sweeps, status);
    gr.sync();
    if (ok)
        for (int k = gr.gl + 1; k <= n; k += G) {
            const cx<double> e = cscal(fx_d(H.ld(k, k)), unit);
            o.rE[(k - 1) * o.sv] = e.r;
            o.iE[(k - 1) * o.sv] = e.i;
        }
    gr.sync();  // the diagonal is read before it is converted below
    if (kVec) {
        FxIndex ix(gr.gl, n);
        for (int e = gr.gl; e < n * n; e += G, ix.next(G, n)) {
            const cx<double> t = ix.i <= ix.j ? fx_d(H.ld(ix.i, ix.j)) : mk(0.0, 0.0);
            H.std(ix.i, ix.j, t);
            if (ok && o.rT) {
                o.rT[e * o.sm] = t.r * unit;
                o.iT[e * o.sm] = t.i * unit;
            }
            Z.std(ix.i, ix.j, fx_d(Z.ld(ix.i, ix.j)));
        }
        gr.sync();
        fx_vectors<G>(gr, n, H, Z, U);
        // scale of each column: the units of Z, and the caller's normalisation
        for (int c = gr.gl + 1; c <= n; c += G) {
            double sc = 0x1p-61;
            if (vnorm == 1) {
                double mx = 0.0;
                for (int r = 1; r <= n; ++r) mx = fmax(mx, cabs1(Z.ldd(r, c)));
                sc = mx > 0.0 ? 1.0 / mx : 1.0;
            } else if (vnorm == 2) {
                double s2 = 0.0;
                for (int r = 1; r <= n; ++r) {
                    const cx<double> z = cscal(Z.ldd(r, c), 0x1p-61);
                    s2 = fma(z.i, z.i, fma(z.r, z.r, s2));
                }
                sc = s2 > 0.0 ? 0x1p-61 / sqrt(s2) : 1.0;
            }
            U.std(c, mk(sc, 0.0));
        }
        gr.sync();
        if (ok) {
            FxIndex iv(gr.gl, n);
            for (int e = gr.gl; e < n * n; e += G, iv.next(G, n)) {
                const cx<double> v = cscal(Z.ldd(iv.i, iv.j), U.ldd(iv.j).r);
                o.rV[e * o.sm] = v.r;
                o.iV[e * o.sm] = v.i;
            }
        }
    }
    gr.sync();  // the storage is reused for the next matrix
    return ok;
}

}  // namespace ves
