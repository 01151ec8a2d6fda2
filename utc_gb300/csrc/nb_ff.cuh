// nb_ff.cuh -- float-float (double-single) device arithmetic shared by the
// float-float symmetric kernels for FP64 state (nb_symff.cu, single system;
// nb_batch.cu, batches).  Published techniques: Knuth's two-sum, Dekker's
// fast two-sum, the FMA two-product, Halley's iteration for 1/sqrt.  A
// float-float number is hi + lo with |lo| <= ulp(hi)/2 (about 48 bits).
#pragma once

#include "nb_pair.cuh"

namespace nb {

// All of it works on register pairs (f32x2): two targets per instruction.
__device__ __forceinline__ f2 ff_pack1(float v) { return f2_pack(v, v); }

// Dekker's fast two-sum, exact when |a| >= |b| (or a == 0).
__device__ __forceinline__ void ff_fast_two_sum(f2 a, f2 b, f2 &s, f2 &e)
{
    s = f2_add(a, b);
    e = f2_sub(b, f2_sub(s, a));
}

// r = s - p from grid-split coordinates (x = h + m + l with h, m and l on
// the grids 2^-20, 2^-44 and 2^-68 of the scaled units, |x| < 1), as a
// normalized float-float; p is passed negated.  The three differences are
// exact (each fits 24 bits); A + B is split by Dekker's fast two-sum (|A| >=
// 2^-20 >= |B|, or A == 0) and the low part added once: r to 2^-47 relative,
// exactly when the high parts cancel (close pairs).
__device__ __forceinline__ void ff_diff(f2 sh, f2 sm, f2 sl, f2 nph, f2 npm, f2 npl, f2 &rh, f2 &rl)
{
    const f2 A = f2_add(sh, nph), B = f2_add(sm, npm), C = f2_add(sl, npl);
    f2 s1, e1;
    ff_fast_two_sum(A, B, s1, e1);
    ff_fast_two_sum(s1, f2_add(e1, C), rh, rl);
}

// A float-float sum under way.
struct FFSum {
    f2 h, l;
    __device__ __forceinline__ void clear() { h = l = f2_pack(0.f, 0.f); }
    // += r * w.  The low part takes the two-sum's error and the product's
    // error and cross terms; it stays below a few ulp(h) between two norm()s.
    __device__ __forceinline__ void add_product(f2 rh, f2 rl, f2 wh, f2 wl)
    {
        const f2 p = f2_mul(rh, wh);
        f2 e = f2_fma(rh, wh, f2_neg(p));
        e = f2_fma(rh, wl, e);
        e = f2_fma(rl, wh, e);
        f2 s, t;
        f2_two_sum(h, p, s, t);
        h = s;
        l = f2_add(l, f2_add(t, e));
    }
    __device__ __forceinline__ void add(f2 vh, f2 vl)
    {
        f2 s, t;
        f2_two_sum(h, vh, s, t);
        h = s;
        l = f2_add(l, f2_add(t, vl));
    }
    __device__ __forceinline__ void norm() { ff_fast_two_sum(h, l, h, l); }
    __device__ __forceinline__ void shfl(int from)
    {
        h = f2_shfl(h, from);
        l = f2_shfl(l, from);
    }
    // the sums of the two halves in FP64
    __device__ __forceinline__ void get(double &lo, double &hi) const
    {
        float h0, h1, l0, l1;
        f2_unpack(h, h0, h1);
        f2_unpack(l, l0, l1);
        lo = (double)h0 + (double)l0;
        hi = (double)h1 + (double)l1;
    }
    // both halves together
    __device__ __forceinline__ double fold() const
    {
        double lo, hi;
        get(lo, hi);
        return lo + hi;
    }
};

// m * y for a float-float mass (mh, ml) and y (yh, yl), unnormalized
__device__ __forceinline__ void ff_mul(f2 mh, f2 ml, f2 yh, f2 yl, f2 &ph, f2 &pl)
{
    ph = f2_mul(mh, yh);
    f2 e = f2_fma(mh, yh, f2_neg(ph));
    e = f2_fma(mh, yl, e);
    pl = f2_fma(ml, yh, e);
}

// A chunk body, its grid-split coordinates and mass broadcast into pairs.
struct FFSource {
    f2 xh, yh, zh, mh, xm, ym, zm, ml, xl, yl, zl;
    __device__ __forceinline__ void load(const float4 &H, const float4 &M, const float4 &L)
    {
        xh = ff_pack1(H.x);
        yh = ff_pack1(H.y);
        zh = ff_pack1(H.z);
        mh = ff_pack1(H.w);
        xm = ff_pack1(M.x);
        ym = ff_pack1(M.y);
        zm = ff_pack1(M.z);
        ml = ff_pack1(M.w);
        xl = ff_pack1(L.x);
        yl = ff_pack1(L.y);
        zl = ff_pack1(L.z);
    }
};

// A pair of targets, coordinates and masses negated.
struct FFTarget {
    f2 xh, yh, zh, mh, xm, ym, zm, ml, xl, yl, zl;
    __device__ __forceinline__ void load(const float4 &H0, const float4 &M0, const float4 &L0, const float4 &H1,
                                         const float4 &M1, const float4 &L1)
    {
        xh = f2_pack(-H0.x, -H1.x);
        yh = f2_pack(-H0.y, -H1.y);
        zh = f2_pack(-H0.z, -H1.z);
        mh = f2_pack(-H0.w, -H1.w);
        xm = f2_pack(-M0.x, -M1.x);
        ym = f2_pack(-M0.y, -M1.y);
        zm = f2_pack(-M0.z, -M1.z);
        ml = f2_pack(-M0.w, -M1.w);
        xl = f2_pack(-L0.x, -L1.x);
        yl = f2_pack(-L0.y, -L1.y);
        zl = f2_pack(-L0.z, -L1.z);
    }
};

struct FFPair {
    f2 rxh, rxl, ryh, ryl, rzh, rzl;  // r = x_j - x_i
    f2 wjh, wjl;                      // m_j inv^3 (weight on the target)
    f2 wih, wil;                      // -m_i inv^3 (weight of the reaction)
    f2 yh, yl;                        // inv = 1/sqrt(|r|^2 + eps2)
};

// Pair pieces for a source and a pair of targets, eps2 = eh + el.
template <bool REACT>
__device__ __forceinline__ void ff_pair(const FFSource &s, const FFTarget &t, f2 eh, f2 el, FFPair &o)
{
    ff_diff(s.xh, s.xm, s.xl, t.xh, t.xm, t.xl, o.rxh, o.rxl);
    ff_diff(s.yh, s.ym, s.yl, t.yh, t.ym, t.yl, o.ryh, o.ryl);
    ff_diff(s.zh, s.zm, s.zl, t.zh, t.zm, t.zl, o.rzh, o.rzl);
    // squares as (p, e) with p + e = r^2 to float-float accuracy
    const f2 qx = f2_mul(o.rxh, o.rxh), qy = f2_mul(o.ryh, o.ryh), qz = f2_mul(o.rzh, o.rzh);
    f2 ex = f2_fma(o.rxh, o.rxh, f2_neg(qx)), ey = f2_fma(o.ryh, o.ryh, f2_neg(qy)),
       ez = f2_fma(o.rzh, o.rzh, f2_neg(qz));
    ex = f2_fma(f2_add(o.rxh, o.rxh), o.rxl, ex);
    ey = f2_fma(f2_add(o.ryh, o.ryh), o.ryl, ey);
    ez = f2_fma(f2_add(o.rzh, o.rzh), o.rzl, ez);
    f2 S, t1, t2, t3;
    f2_two_sum(eh, qx, S, t1);
    f2_two_sum(S, qy, S, t2);
    f2_two_sum(S, qz, S, t3);
    const f2 L = f2_add(f2_add(f2_add(el, ex), f2_add(ey, ez)), f2_add(f2_add(t1, t2), t3));
    f2 Dh, Dl;
    ff_fast_two_sum(S, L, Dh, Dl);  // all terms >= 0: |S| >= |L|
    // 1/sqrt(D): the FP32 approximation, one Newton step in FP32 (error
    // near 2^-24, so that u below is near 2^-23 and the roundings that scale
    // with it stay near 2^-47), then one Halley step in float-float
    const f2 ONE = ff_pack1(1.0f);
    float d0, d1;
    f2_unpack(Dh, d0, d1);
    const f2 ya = f2_pack(rsqrt_approx(d0), rsqrt_approx(d1));
    const f2 y0 = f2_fma(f2_mul(ya, ff_pack1(0.5f)), f2_fma(f2_neg(Dh), f2_mul(ya, ya), ONE), ya);
    const f2 q = f2_mul(y0, y0);
    const f2 qe = f2_fma(y0, y0, f2_neg(q));
    const f2 t_ = f2_mul(Dh, q);
    f2 c = f2_fma(Dh, q, f2_neg(t_));
    c = f2_fma(Dh, qe, c);
    c = f2_fma(Dl, q, c);
    const f2 u = f2_sub(f2_sub(ONE, t_), c);  // 1 - t is exact (t near 1)
    const f2 corr = f2_mul(y0, f2_mul(u, f2_fma(ff_pack1(0.375f), u, ff_pack1(0.5f))));
    f2 yh, yl;
    ff_fast_two_sum(y0, corr, yh, yl);
    o.yh = yh;
    o.yl = yl;
    // inv^3 = y^3
    const f2 p2 = f2_mul(yh, yh);
    f2 e2 = f2_fma(yh, yh, f2_neg(p2));
    e2 = f2_fma(f2_add(yh, yh), yl, e2);
    const f2 p3 = f2_mul(p2, yh);
    f2 e3 = f2_fma(p2, yh, f2_neg(p3));
    e3 = f2_fma(p2, yl, e3);
    e3 = f2_fma(e2, yh, e3);
    f2 y3h, y3l;
    ff_fast_two_sum(p3, e3, y3h, y3l);
    // weights (mass as the float-float h + m of its split)
    ff_mul(s.mh, s.ml, y3h, y3l, o.wjh, o.wjl);
    if (REACT) ff_mul(t.mh, t.ml, y3h, y3l, o.wih, o.wil);
}

// A lane's 2 * NP targets with the sums of one chunk.
template <int NP, bool PHI>
struct FFTargets {
    FFTarget t[NP];
    FFSum ax[NP], ay[NP], az[NP], ap[PHI ? NP : 1];

    // body(k): the index of target k of the lane, < 0 for a missing one,
    // which gets zero mass: its reactions are 0
    template <class Body>
    __device__ __forceinline__ void load(const float4 *H, const float4 *M,
                                         const float4 *L, Body body)
    {
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const int i = body(2 * p), j = body(2 * p + 1);
            t[p].load(i >= 0 ? H[i] : zero, i >= 0 ? M[i] : zero, i >= 0 ? L[i] : zero, j >= 0 ? H[j] : zero,
                      j >= 0 ? M[j] : zero, j >= 0 ? L[j] : zero);
        }
    }
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            ax[p].clear();
            ay[p].clear();
            az[p].clear();
            if (PHI) ap[p].clear();
        }
    }
    __device__ __forceinline__ void norm()
    {
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            ax[p].norm();
            ay[p].norm();
            az[p].norm();
            if (PHI) ap[p].norm();
        }
    }
    __device__ __forceinline__ void pull(int p, const FFPair &w)
    {
        ax[p].add_product(w.rxh, w.rxl, w.wjh, w.wjl);
        ay[p].add_product(w.ryh, w.ryl, w.wjh, w.wjl);
        az[p].add_product(w.rzh, w.rzl, w.wjh, w.wjl);
    }
};

// The chunk in sH, sM, sL (32 bodies) on the lane's targets, target side only
// (a chunk inside the targets' own row block).  self(k): the chunk position of
// target k itself, or a value outside 0..31; its potential term is left out.
template <int NP, bool PHI, class Self>
__device__ __forceinline__ void ff_chunk_pull(FFTargets<NP, PHI> &T, const float4 *sH, const float4 *sM,
                                              const float4 *sL, f2 eh, f2 el, Self self)
{
#pragma unroll 1
    for (int j = 0; j < 32; ++j) {
        FFSource s;
        s.load(sH[j], sM[j], sL[j]);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            FFPair w;
            ff_pair<false>(s, T.t[p], eh, el, w);
            T.pull(p, w);
            if (PHI) {
                f2 vh, vl;
                ff_mul(s.mh, s.ml, w.yh, w.yl, vh, vl);
                float h0, h1, l0, l1;
                f2_unpack(vh, h0, h1);
                f2_unpack(vl, l0, l1);
                if (j == self(2 * p)) h0 = l0 = 0.f;
                if (j == self(2 * p + 1)) h1 = l1 = 0.f;
                T.ap[p].add(f2_pack(h0, h1), f2_pack(l0, l1));
            }
        }
        T.norm();
    }
}

// The reactions on the 32 chunk bodies (x, y, z and the potential) while the
// lane's targets gather theirs: at step r lane l works on chunk body
// (l + r) mod 32 and hands its reaction, one half per target of a pair, to
// lane l - 1; lane l ends with the reaction on chunk body l.  The sums are
// renormalized every second (targets) and fourth step (reactions): after every
// one costs 11 of 196 operations more (313 against 329 G interactions/s at
// N = 16384, 337 without any).  The two halves of a reaction are chains half as long as
// one chain over both targets, and the errors are the smaller for it (force
// error over |a| + mean|a|, rms over 2000 bodies, Plummer / cube / dense cores:
// 1.6e-15 / 1.9e-15 / 1.4e-15 against 1.75e-15 / 1.94e-15 / 1.53e-15 with one
// chain renormalized after every term).
struct FFReact {
    FFSum x, y, z, p;
};

template <int NP, bool PHI>
__device__ __forceinline__ void ff_chunk_react(FFTargets<NP, PHI> &T, FFReact &F, const float4 *sH, const float4 *sM,
                                               const float4 *sL, int lane, f2 eh, f2 el)
{
    F.x.clear();
    F.y.clear();
    F.z.clear();
    F.p.clear();
    const int from = (lane + 1) & 31;
#pragma unroll 4
    for (int r = 0; r < 32; ++r) {
        const int idx = (lane + r) & 31;
        FFSource s;
        s.load(sH[idx], sM[idx], sL[idx]);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            FFPair w;
            ff_pair<true>(s, T.t[p], eh, el, w);
            T.pull(p, w);
            F.x.add_product(w.rxh, w.rxl, w.wih, w.wil);
            F.y.add_product(w.ryh, w.ryl, w.wih, w.wil);
            F.z.add_product(w.rzh, w.rzl, w.wih, w.wil);
            if (PHI) {
                f2 vh, vl;
                ff_mul(s.mh, s.ml, w.yh, w.yl, vh, vl);
                T.ap[p].add(vh, vl);
                ff_mul(f2_neg(T.t[p].mh), f2_neg(T.t[p].ml), w.yh, w.yl, vh, vl);
                F.p.add(vh, vl);
            }
        }
        if (r % 2 == 1) T.norm();
        if (r % 4 == 3) {
            F.x.norm();
            F.y.norm();
            F.z.norm();
            if (PHI) F.p.norm();
        }
        F.x.shfl(from);
        F.y.shfl(from);
        F.z.shfl(from);
        if (PHI) F.p.shfl(from);
    }
}

// binary exponent e of a non-negative double given by its bits, with
// 2^(e-1) <= v < 2^e; 0 for zero, subnormal, infinite or NaN values
__device__ __forceinline__ int ff_exponent(unsigned long long bits)
{
    const int field = (int)((bits >> 52) & 0x7ff);
    return (field == 0 || field == 0x7ff) ? 0 : field - 1022;
}


}  // namespace nb
