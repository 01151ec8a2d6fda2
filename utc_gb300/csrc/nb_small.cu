// nb_small.cu -- the whole step of a small FP32 system in one launch.
//
// The symmetric kernels need two dependent launches a step (pair terms, then
// the sum of every body's partials), and a small system has few (row, chunk)
// items for 152 SMs: at N = 1024 the pair terms take a third of a microsecond
// of the chip, but the two launches took 7.4 us from a graph and 12.3 us one
// by one.  Here a CTA owns TB bodies for the whole step: its 128 threads split
// the sources, every pair is evaluated from the target's side (both orders
// are evaluated, 12 FP32 operations and one rsqrt each: twice the pair terms,
// but no partial leaves the CTA), the sums are reduced through the warps and
// the CTA's first threads apply the kick / damping / drift.  No scratch, no
// second launch, fixed order of summation: deterministic.  A target's sum
// depends neither on its place in a CTA nor on TB (each thread's sources and the
// tree over the threads are the same), so shards of the targets give the same
// bits.  Direct plans of nb_fast.cu use it for their force launch.
//
// Step time from a replayed graph, GB300, us, against the two launches:
// N = 512 1.7 (6.4), 1024 2.2 (7.1), 2048 3.6 (9.2), 3000 5.4 (12.8), 4099
// 9.0 (16.3), 6000 15.7 (23.7), 8192 28 (32.5).  Bounds: latency below N about
// 2000 (launch, one round of loads, the reduction), above it register-file
// reads (26 operand reads a pair of interactions, nb_pair.cuh) and how evenly
// the CTAs fill the SMs.  128 threads a CTA ran 5 to 30 % ahead of 256 and
// 512; the launch bound of one CTA lets the loop have the registers that it
// asks for (146 for 8 targets, 108 for 4; without it 64, and 3.5 us at
// N = 1024).  With 10 targets three CTAs an SM are asked for: with 172
// registers there were two, and 11.8 us at N = 4099.  Sources per turn of the
// loop: 4, with 6 targets 5 (N = 5000 12.7 us, 13.1 with 4), with 10 targets 3
// (N = 4099 9.0, 9.7 with 4).
#include "nb_pair.cuh"

namespace nb {

constexpr int kSmallThreads = 128;

// pos_new == nullptr: no step, only acc_out; acc_out may be given beside a
// step too.
template <int TB>
__global__ void __launch_bounds__(kSmallThreads, TB == 10 ? 3 : 1) small_step_kernel(const float4 *pos_old,
                                                                   float4 *pos_new,
                                                                   float4 *vel, int n, int lo, int hi, float eps2,
                                                                   float damping, float dt, int kick, float G,
                                                                   float4 *acc_out)
{
    constexpr int NP = TB / 2, TP = pow2_up(TB);
    constexpr int NW = kSmallThreads / 32;
    __shared__ float red[NW][3 * TP];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int t0 = lo + blockIdx.x * TB;
    const float4 pad = make_float4(kPadCoord, kPadCoord, kPadCoord, 0.f);
    const f2 EPS2 = f2_pack(eps2, eps2);
    // A programmatic launch: the blocks come in as those of the previous step's
    // kernel leave, and wait here until that kernel is complete and its
    // writes visible.  It gives its dependents no earlier signal: blocks let
    // in before the SMs are free gather on those that empty first (N = 3000:
    // 6.6 us a step against 5.4; plain launches 5.65).
    pdl_wait();
    // the body that this thread integrates
    const int mine = t0 + tid;
    const bool own = tid < TB && mine < hi;
    float4 p = pad, v = pad;
    if (own) {
        p = pos_old[mine];
        if (pos_new) v = vel[mine];
    }
    PairTargets<NP> T;
    T.load([&](int t) { return t0 + t < n ? pos_old[t0 + t] : make_float4(0.f, 0.f, 0.f, 0.f); });
    float4 nxt = tid < n ? pos_old[tid] : pad;
    constexpr int U = TB == 10 ? 3 : TB == 6 ? 5 : 4;
#pragma unroll(U)
    for (int j = tid; j - tid < n; j += kSmallThreads) {
        const float4 q = nxt;
        const int jn = j + kSmallThreads;
        nxt = jn < n ? pos_old[jn] : pad;
        const f2 X = f2_pack(q.x, q.x), Y = f2_pack(q.y, q.y), Z = f2_pack(q.z, q.z), M = f2_pack(q.w, q.w);
#pragma unroll
        for (int k = 0; k < NP; ++k) pair_pull(T, k, pair_term(T, k, X, Y, Z, EPS2), M);
    }
    float s[3 * TP];
#pragma unroll
    for (int t = 3 * TB; t < 3 * TP; ++t) s[t] = 0.f;
#pragma unroll
    for (int t = 0; t < TB; ++t) {
        const float4 a = T.sum(t);
        s[3 * t] = a.x;
        s[3 * t + 1] = a.y;
        s[3 * t + 2] = a.z;
    }
    const int t = warp_sum<TP, 3>(s, lane);
    if ((lane & (32 / TP - 1)) == 0) {
        red[wid][3 * t] = s[0];
        red[wid][3 * t + 1] = s[1];
        red[wid][3 * t + 2] = s[2];
    }
    __syncthreads();
    if (!own) return;
    float ax = 0.f, ay = 0.f, az = 0.f;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        ax = __fadd_rn(ax, red[w][3 * tid]);
        ay = __fadd_rn(ay, red[w][3 * tid + 1]);
        az = __fadd_rn(az, red[w][3 * tid + 2]);
    }
    if (acc_out) acc_out[mine] = make_float4(ax, ay, az, 0.f);
    if (!pos_new) return;
    const float k = kick == NB_KICK_REFERENCE ? p.w : G;
    v.x = __fadd_rn(v.x, __fmul_rn(__fmul_rn(ax, k), dt));
    v.y = __fadd_rn(v.y, __fmul_rn(__fmul_rn(ay, k), dt));
    v.z = __fadd_rn(v.z, __fmul_rn(__fmul_rn(az, k), dt));
    v.x = __fmul_rn(v.x, damping);
    v.y = __fmul_rn(v.y, damping);
    v.z = __fmul_rn(v.z, damping);
    p.x = __fadd_rn(p.x, __fmul_rn(v.x, dt));
    p.y = __fadd_rn(p.y, __fmul_rn(v.y, dt));
    p.z = __fadd_rn(p.z, __fmul_rn(v.z, dt));
    pos_new[mine] = p;
    vel[mine] = v;
}

// Targets per CTA: few bodies per CTA while the step is a chain of latencies
// (below 2000 bodies), then the choice that leaves the fullest SM the least
// to do: ceil(CTAs / SMs) CTAs of TB bodies each, plus 0.9 of a body's work per
// CTA for its pass over the sources and its reduction, and 3 % more for the
// slower schedule with 8.  6 / 8 / 10 bodies, step us: N = 3000 6.5 / 6.2 / 5.4,
// 4099 10.7 / 9.8 / 9.0, 5000 12.7 / 13.6 / 13.6, 6000 17.0 / 16.3 / 15.7, 7000 21.8 /
// 21.9 / 21.8, 8192 28.2 / 28.5 / 29.3; the force launch of direct plans and their
// integrator: 9001 35.6 / 37.1 / 34.2, 12345 64.0 / 65.7 / 64.7, 16384 106.2 / 107.6 /
// 102.5, 20000 157.2 / 158.3 / 157.6, 24576 233.3 / 235.8 / 231.0.
static int small_targets(int n, int sms)
{
    if (n < 2000) return 4;
    int best = 8;
    float least = 1e30f;
    for (int tb = 6; tb <= 10; tb += 2) {
        const int ctas = (n + tb - 1) / tb;
        const float cost = (float)((ctas + sms - 1) / sms) * ((float)tb + 0.9f) * (tb == 8 ? 1.03f : 1.f);
        if (cost < least) {
            least = cost;
            best = tb;
        }
    }
    return best;
}

int small_step(int n, int lo, int hi, int sms, const float4 *pos_old, float4 *pos_new, float4 *vel, float eps2,
               float damping, float dt, int kick, float G, float4 *acc_out, cudaStream_t s)
{
    if (hi <= lo) return NB_OK;
    const int tb = small_targets(hi - lo, sms);
    auto k = tb == 4 ? small_step_kernel<4> : tb == 6 ? small_step_kernel<6> : tb == 8 ? small_step_kernel<8>
                                                                                       : small_step_kernel<10>;
    return pdl_launch("small_step_kernel launch", k, (unsigned)((hi - lo + tb - 1) / tb), kSmallThreads, s, pos_old, pos_new,
                      vel, n, lo, hi, eps2, damping, dt, kick, G, acc_out);
}

}  // namespace nb
