// nb_vjp.cuh -- the packed FP32 pair loops of the symmetric vector-Jacobian
// product, shared by nb_adjoint.cu (single system) and nb_batch.cu (batches).
// The algebra is that of nb_adjoint.cu; as in nb_pair.cuh a lane's targets
// are held as register pairs and every operation is one f32x2 instruction for
// two of them.
//
// 34 operations and one MUFU per pair, of which 20 read three registers: 88
// operand reads, 44 cycles at two reads a cycle (nb_pair.cuh), are the floor
// without operand reuse; the scalar loop ran at 52, held up by its 36 issue
// slots as well, this one at 47.  sym_vjp_kernel, 10 targets per lane, GB300:
// N = 16384 162 us against 178, N = 65536 2.47 ms against 2.74 (rotation loop
// unrolled twice 164 us, four times 168; 8 targets per lane 164, 12 183).
#pragma once

#include "nb_pair.cuh"

namespace nb {

// A chunk body and its g, broadcast into pairs.
struct VjpSource {
    f2 x, y, z, m, gx, gy, gz;
    __device__ __forceinline__ void load(const float4 &s, const float4 &g)
    {
        x = f2_pack(s.x, s.x);
        y = f2_pack(s.y, s.y);
        z = f2_pack(s.z, s.z);
        m = f2_pack(s.w, s.w);
        gx = f2_pack(g.x, g.x);
        gy = f2_pack(g.y, g.y);
        gz = f2_pack(g.z, g.z);
    }
};

// The sums of one body (pairs: two bodies, or two halves of one reaction):
// P = sum inv^3 g, q = sum inv^3 m, Q = sum c r, w = sum inv^3 r.g
struct VjpSums {
    f2 Px, Py, Pz, q, Qx, Qy, Qz, w;
    __device__ __forceinline__ void clear() { Px = Py = Pz = q = Qx = Qy = Qz = w = f2_pack(0.f, 0.f); }
    __device__ __forceinline__ void shfl(int from)
    {
        Px = f2_shfl(Px, from);
        Py = f2_shfl(Py, from);
        Pz = f2_shfl(Pz, from);
        q = f2_shfl(q, from);
        Qx = f2_shfl(Qx, from);
        Qy = f2_shfl(Qy, from);
        Qz = f2_shfl(Qz, from);
        w = f2_shfl(w, from);
    }
};

// m P - q g - 3 Q
__device__ __forceinline__ float3 vjp_out(float m, float gx, float gy, float gz, float Px, float Py, float Pz, float q,
                                          float Qx, float Qy, float Qz)
{
    return make_float3(fmaf(m, Px, fmaf(-q, gx, -3.f * Qx)), fmaf(m, Py, fmaf(-q, gy, -3.f * Qy)),
                       fmaf(m, Pz, fmaf(-q, gz, -3.f * Qz)));
}

// A lane's 2 * NP targets: positions negated, masses, g, and their sums.
template <int NP>
struct VjpTargets {
    f2 px[NP], py[NP], pz[NP], m[NP], gx[NP], gy[NP], gz[NP];
    VjpSums s[NP];

    // target t of the lane is at(t) with g at gat(t); zeros for a missing one,
    // whose terms are then 0
    template <class At, class Gat>
    __device__ __forceinline__ void load(At at, Gat gat)
    {
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const float4 a = at(2 * p), b = at(2 * p + 1), g = gat(2 * p), h = gat(2 * p + 1);
            px[p] = f2_pack(-a.x, -b.x);
            py[p] = f2_pack(-a.y, -b.y);
            pz[p] = f2_pack(-a.z, -b.z);
            m[p] = f2_pack(a.w, b.w);
            gx[p] = f2_pack(g.x, h.x);
            gy[p] = f2_pack(g.y, h.y);
            gz[p] = f2_pack(g.z, h.z);
            s[p].clear();
        }
    }

    // the pair term of source b and target pair p; reactions into R if REACT
    template <bool REACT>
    __device__ __forceinline__ void pair(int p, const VjpSource &b, f2 EPS2, VjpSums &R)
    {
        const f2 rx = f2_add(b.x, px[p]), ry = f2_add(b.y, py[p]), rz = f2_add(b.z, pz[p]);
        f2 d2 = f2_fma(rx, rx, EPS2);
        d2 = f2_fma(ry, ry, d2);
        d2 = f2_fma(rz, rz, d2);
        float lo, hi;
        f2_unpack(d2, lo, hi);
        const f2 inv = f2_pack(rsqrt_approx(lo), rsqrt_approx(hi));
        const f2 inv2 = f2_mul(inv, inv);
        const f2 inv3 = f2_mul(inv2, inv);
        const f2 inv5 = f2_mul(inv3, inv2);
        const f2 rgj = f2_fma(rz, b.gz, f2_fma(ry, b.gy, f2_mul(rx, b.gx)));
        const f2 rgk = f2_fma(rz, gz[p], f2_fma(ry, gy[p], f2_mul(rx, gx[p])));
        const f2 c = f2_mul(inv5, f2_fma(m[p], rgj, f2_neg(f2_mul(b.m, rgk))));
        VjpSums &t = s[p];
        t.Px = f2_fma(inv3, b.gx, t.Px);
        t.Py = f2_fma(inv3, b.gy, t.Py);
        t.Pz = f2_fma(inv3, b.gz, t.Pz);
        t.q = f2_fma(inv3, b.m, t.q);
        t.Qx = f2_fma(c, rx, t.Qx);
        t.Qy = f2_fma(c, ry, t.Qy);
        t.Qz = f2_fma(c, rz, t.Qz);
        t.w = f2_fma(inv3, rgj, t.w);
        if (REACT) {
            const f2 nc = f2_neg(c);
            R.Px = f2_fma(inv3, gx[p], R.Px);
            R.Py = f2_fma(inv3, gy[p], R.Py);
            R.Pz = f2_fma(inv3, gz[p], R.Pz);
            R.q = f2_fma(inv3, m[p], R.q);
            R.Qx = f2_fma(nc, rx, R.Qx);
            R.Qy = f2_fma(nc, ry, R.Qy);
            R.Qz = f2_fma(nc, rz, R.Qz);
            R.w = f2_fma(inv3, rgk, R.w);
        }
    }

    // (out, dm) of the two targets of pair p
    __device__ __forceinline__ void out(int p, float4 &a, float4 &b) const
    {
        const VjpSums &t = s[p];
        float mm[2], g[3][2], P[3][2], q[2], Q[3][2], w[2];
        f2_unpack(m[p], mm[0], mm[1]);
        f2_unpack(gx[p], g[0][0], g[0][1]);
        f2_unpack(gy[p], g[1][0], g[1][1]);
        f2_unpack(gz[p], g[2][0], g[2][1]);
        f2_unpack(t.Px, P[0][0], P[0][1]);
        f2_unpack(t.Py, P[1][0], P[1][1]);
        f2_unpack(t.Pz, P[2][0], P[2][1]);
        f2_unpack(t.q, q[0], q[1]);
        f2_unpack(t.Qx, Q[0][0], Q[0][1]);
        f2_unpack(t.Qy, Q[1][0], Q[1][1]);
        f2_unpack(t.Qz, Q[2][0], Q[2][1]);
        f2_unpack(t.w, w[0], w[1]);
        const float3 u = vjp_out(mm[0], g[0][0], g[1][0], g[2][0], P[0][0], P[1][0], P[2][0], q[0], Q[0][0], Q[1][0],
                                 Q[2][0]);
        const float3 v = vjp_out(mm[1], g[0][1], g[1][1], g[2][1], P[0][1], P[1][1], P[2][1], q[1], Q[0][1], Q[1][1],
                                 Q[2][1]);
        a = make_float4(u.x, u.y, u.z, -w[0]);
        b = make_float4(v.x, v.y, v.z, -w[1]);
    }
};

// The chunk in sC, sG (32 bodies) on the lane's targets, target side only (a
// chunk inside the targets' own row block).
template <int NP>
__device__ __forceinline__ void vjp_chunk_pull(VjpTargets<NP> &T, const float4 *sC, const float4 *sG, f2 EPS2)
{
    VjpSums none;
#pragma unroll 1
    for (int j = 0; j < 32; ++j) {
        VjpSource b;
        b.load(sC[j], sG[j]);
#pragma unroll
        for (int p = 0; p < NP; ++p) T.template pair<false>(p, b, EPS2, none);
    }
}

// The chunk's bodies against the lane's targets, each unordered pair once, the
// chunk body's sums rotating through the warp as in chunk_react (nb_pair.cuh);
// r8 gets the eight reaction sums on chunk body `lane` (P, q, Q, w).
template <int NP>
__device__ __forceinline__ void vjp_chunk_react(VjpTargets<NP> &T, const float4 *sC, const float4 *sG, int lane,
                                                f2 EPS2, float r8[8])
{
    VjpSums R;
    R.clear();
    const int from = (lane + 1) & 31;
#pragma unroll 8
    for (int r = 0; r < 32; ++r) {
        const int idx = (lane + r) & 31;
        VjpSource b;
        b.load(sC[idx], sG[idx]);
#pragma unroll
        for (int p = 0; p < NP; ++p) T.template pair<true>(p, b, EPS2, R);
        R.shfl(from);
    }
    r8[0] = f2_fold(R.Px);
    r8[1] = f2_fold(R.Py);
    r8[2] = f2_fold(R.Pz);
    r8[3] = f2_fold(R.q);
    r8[4] = f2_fold(R.Qx);
    r8[5] = f2_fold(R.Qy);
    r8[6] = f2_fold(R.Qz);
    r8[7] = f2_fold(R.w);
}

// (out, dm) of a chunk body from its reaction sums
__device__ __forceinline__ float4 vjp_reaction(const float4 &b, const float4 &g, const float r8[8])
{
    const float3 o = vjp_out(b.w, g.x, g.y, g.z, r8[0], r8[1], r8[2], r8[3], r8[4], r8[5], r8[6]);
    return make_float4(o.x, o.y, o.z, r8[7]);
}

}  // namespace nb
