// nb_pair.cuh -- the packed FP32 pair loops shared by the symmetric kernels
// (nb_sym.cu, single system; nb_batch.cu, batches).
//
// A lane's targets are held as NP register pairs (targets 2p and 2p + 1 of
// the lane in the halves of pair p), so that every pair-term operation is one
// sm_100+ f32x2 instruction (FADD2 / FMUL2 / FFMA2) for two targets; the chunk
// body is broadcast into pairs once per rotation step and reused for all NP
// pairs.  Per pair of targets: 16 packed operations and two MUFU.RSQ.
//
// What bounds the loop: register-file reads.  An SM sub-partition reads two
// 32-bit operands (one 64-bit operand) per cycle and lane, measured on GB300
// as 1.0 cycle per operation for add, multiply and a*a+c, and 1.4 to 1.7 for
// an FMA with three different register operands (the reuse cache serves a
// weight that two neighbouring FMAs share).  The six accumulating FMAs of a
// pair read three operands each: 37 operand cycles against 32 pipe cycles per
// pair of targets, so 18.5 cycles per pair and warp (4140 G interactions/s
// at 2.07 GHz) are the floor of this arithmetic without operand reuse.
// Measured, force kernel, N = 65536, 16 targets per lane: 4002 G
// interactions/s, against 3578 for the scalar loop that it replaced, whose 17
// issue slots per pair left no room for the operand stalls (the packed loop
// issues 9); 4 warps x 20 targets at N = 262144: 3965 against 3574;
// compensated 1 x 12 (ordered reactions, chunk_react) at N = 131072: 3624 against
// 3166.  Timed beside it (the loop alone, 16
// targets, 4022): the reaction folded to a scalar before each shuffle 3926,
// the chunk stored as duplicated pairs in shared memory 3929, the reaction
// added through shared memory 3887, packed differences with scalar
// accumulation 3770, two chunk bodies per pair instead of two targets 4016
// (12 targets, 244 registers), 18 targets per lane 4002, 20 targets 3910.
#pragma once

#include "nb_internal.cuh"

namespace nb {

// A lane's 2 * NP targets: positions and masses negated (r = q + (-p); the
// reaction on the chunk body points along -r), and their acceleration sums.
template <int NP>
struct PairTargets {
    f2 px[NP], py[NP], pz[NP], nm[NP], ax[NP], ay[NP], az[NP];

    // target t of the lane (0 <= t < 2 NP) is at(t): its (x, y, z, m), or
    // zeros for a missing one, whose reactions are then 0
    template <class At>
    __device__ __forceinline__ void load(At at)
    {
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const float4 a = at(2 * p), b = at(2 * p + 1);
            px[p] = f2_pack(-a.x, -b.x);
            py[p] = f2_pack(-a.y, -b.y);
            pz[p] = f2_pack(-a.z, -b.z);
            nm[p] = f2_pack(-a.w, -b.w);
        }
        clear();
    }
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int p = 0; p < NP; ++p) ax[p] = ay[p] = az[p] = f2_pack(0.f, 0.f);
    }
    // the sums of target t as (x, y, z, 0)
    __device__ __forceinline__ float4 sum(int t) const
    {
        float x[2], y[2], z[2];
        f2_unpack(ax[t >> 1], x[0], x[1]);
        f2_unpack(ay[t >> 1], y[0], y[1]);
        f2_unpack(az[t >> 1], z[0], z[1]);
        return make_float4(x[t & 1], y[t & 1], z[t & 1], 0.f);
    }
};

// r = q - p and inv = 1 / (|r|^2 + eps2)^(1/2) for a pair of targets
struct PairTerm {
    f2 rx, ry, rz, inv;
};

template <int NP>
__device__ __forceinline__ PairTerm pair_term(const PairTargets<NP> &t, int p, f2 X, f2 Y, f2 Z, f2 EPS2)
{
    PairTerm o;
    o.rx = f2_add(X, t.px[p]);
    o.ry = f2_add(Y, t.py[p]);
    o.rz = f2_add(Z, t.pz[p]);
    f2 d2 = f2_fma(o.rx, o.rx, EPS2);
    d2 = f2_fma(o.ry, o.ry, d2);
    d2 = f2_fma(o.rz, o.rz, d2);
    float lo, hi;
    f2_unpack(d2, lo, hi);
    o.inv = f2_pack(rsqrt_approx(lo), rsqrt_approx(hi));
    return o;
}

template <int NP>
__device__ __forceinline__ void pair_add(PairTargets<NP> &t, int p, const PairTerm &r, f2 w)
{
    t.ax[p] = f2_fma(r.rx, w, t.ax[p]);
    t.ay[p] = f2_fma(r.ry, w, t.ay[p]);
    t.az[p] = f2_fma(r.rz, w, t.az[p]);
}

// The pull of one source of mass M on target pair p, where no reaction shares
// the term.  The weight is (M inv) inv^2: inv^3 alone is subnormal from
// distances of 4.4e12 on (zero from 1.2e15) and overflows below 1.4e-13, also at
// the self pair of a softening that small, where 0 * inf would be NaN, while
// the mass keeps the products of this order normal (bodies of 1e30 at 1e18).
// As many multiplications as M inv^3; small_step_kernel with 8 targets is 2 to 3
// % slower for the other schedule (N = 7000 21.3 us with M inv^3, 21.9), with 4, 6
// and 10 it is not.
template <int NP>
__device__ __forceinline__ void pair_pull(PairTargets<NP> &t, int p, const PairTerm &r, f2 M)
{
    const f2 inv2 = f2_mul(r.inv, r.inv);
    pair_add(t, p, r, f2_mul(inv2, f2_mul(r.inv, M)));
}

// The pull of the 32 chunk bodies in sC on the lane's targets (a chunk inside
// the targets' own row block: both orders of each pair occur there).
template <int NP>
__device__ __forceinline__ void chunk_pull(PairTargets<NP> &t, const float4 *sC, f2 EPS2)
{
#pragma unroll 1
    for (int j = 0; j < 32; ++j) {
        const float4 q = sC[j];
        const f2 X = f2_pack(q.x, q.x), Y = f2_pack(q.y, q.y), Z = f2_pack(q.z, q.z), M = f2_pack(q.w, q.w);
#pragma unroll
        for (int p = 0; p < NP; ++p) pair_pull(t, p, pair_term(t, p, X, Y, Z, EPS2), M);
    }
}

__device__ __forceinline__ f2 f2_shfl(f2 v, int from)
{
    float lo, hi;
    f2_unpack(v, lo, hi);
    return f2_pack(__shfl_sync(0xffffffffu, lo, from), __shfl_sync(0xffffffffu, hi, from));
}

__device__ __forceinline__ float f2_fold(f2 v)
{
    float lo, hi;
    f2_unpack(v, lo, hi);
    return lo + hi;
}

// The chunk's bodies against the lane's targets, each unordered pair once: at
// step r lane l pairs its targets with chunk body (l + r) mod 32 and carries
// that body's reaction (one half per target of a pair, folded at the end),
// passed on to lane l - 1 after the step.  Returns the reaction on chunk body
// l from the warp's targets.
//
// ORDERED (the compensated kernel): the reaction is one sum over the targets in
// their order.  A compensated step's state has twice the digits of its pair
// terms, so the rounding of a 384-term sum in FP32 shows in its results: the
// order is part of them (two chains folded at the end moved them by 1e-8 where
// the forces are large).  Six scalar FMAs take the place of three packed
// ones: two steps at N = 131071 take 10196 us, 10029 with the two chains, 11490
// with the scalar loop.
template <int NP, bool ORDERED = false>
__device__ __forceinline__ float3 chunk_react(PairTargets<NP> &t, const float4 *sC, int lane, f2 EPS2)
{
    f2 fx = f2_pack(0.f, 0.f), fy = fx, fz = fx;
    float3 f = make_float3(0.f, 0.f, 0.f);  // ORDERED
    const int from = (lane + 1) & 31;
#pragma unroll 8
    for (int r = 0; r < 32; ++r) {
        const float4 q = sC[(lane + r) & 31];
        const f2 X = f2_pack(q.x, q.x), Y = f2_pack(q.y, q.y), Z = f2_pack(q.z, q.z), M = f2_pack(q.w, q.w);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const PairTerm o = pair_term(t, p, X, Y, Z, EPS2);
            const f2 inv3 = f2_mul(o.inv, f2_mul(o.inv, o.inv));  // shared by the two weights
            pair_add(t, p, o, f2_mul(M, inv3));
            const f2 ss = f2_mul(t.nm[p], inv3);
            if constexpr (ORDERED) {
                float s0, s1, r0, r1;
                f2_unpack(ss, s0, s1);
                f2_unpack(o.rx, r0, r1);
                f.x = __fmaf_rn(r1, s1, __fmaf_rn(r0, s0, f.x));
                f2_unpack(o.ry, r0, r1);
                f.y = __fmaf_rn(r1, s1, __fmaf_rn(r0, s0, f.y));
                f2_unpack(o.rz, r0, r1);
                f.z = __fmaf_rn(r1, s1, __fmaf_rn(r0, s0, f.z));
            } else {
                fx = f2_fma(o.rx, ss, fx);
                fy = f2_fma(o.ry, ss, fy);
                fz = f2_fma(o.rz, ss, fz);
            }
        }
        if constexpr (ORDERED) {
            f.x = __shfl_sync(0xffffffffu, f.x, from);
            f.y = __shfl_sync(0xffffffffu, f.y, from);
            f.z = __shfl_sync(0xffffffffu, f.z, from);
        } else {
            fx = f2_shfl(fx, from);
            fy = f2_shfl(fy, from);
            fz = f2_shfl(fz, from);
        }
    }
    return ORDERED ? f : make_float3(f2_fold(fx), f2_fold(fy), f2_fold(fz));
}

constexpr int pow2_up(int x) { return x <= 2 ? 2 : x <= 4 ? 4 : x <= 8 ? 8 : 16; }

// Sums v[0..C T) (T targets x C components) over the warp.  While more than
// one target is left the lanes halve them: a lane keeps the half that its bit
// selects and gives the other away, so that the first levels cost C T / 2,
// C T / 4, ... shuffles.  Returns the lane's target; every lane of a target's
// group has its C sums.
template <int T, int C>
__device__ __forceinline__ int warp_sum(float *v, int lane)
{
    int mine = 0, off = 16;
#pragma unroll
    for (int h = T / 2; h >= 1; h /= 2) {
        const bool up = (lane & off) != 0;
        mine = 2 * mine + (up ? 1 : 0);
#pragma unroll
        for (int k = 0; k < C * h; ++k) {
            const float give = up ? v[k] : v[C * h + k], keep = up ? v[C * h + k] : v[k];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, give, off);
        }
        off /= 2;
    }
#pragma unroll
    for (; off >= 1; off /= 2) {
#pragma unroll
        for (int k = 0; k < C; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], off);
    }
    return mine;
}

// Packed two-sum (Knuth): s + e == a + b exactly, s = fl(a + b).
__device__ __forceinline__ void f2_two_sum(f2 a, f2 b, f2 &s, f2 &e)
{
    s = f2_add(a, b);
    const f2 bb = f2_sub(s, a);
    e = f2_add(f2_sub(a, f2_sub(s, bb)), f2_sub(b, bb));
}

}  // namespace nb
