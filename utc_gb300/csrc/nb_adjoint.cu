// nb_adjoint.cu -- reverse-mode (adjoint) kernels of the nbody step.
//
// No counterpart in the reference (it has no gradients).  The forward step is
// the reference's update (benchapps/nbody/seq/bodysystem.cc:135-182):
//   a_i = sum_j m_j r_ij inv_ij^3,  r_ij = x_j - x_i, inv = (|r|^2+eps2)^-1/2
//   v'  = D (v + k a dt),            k_i = m_i (reference kick) or G
//   x'  = x + v' dt
// Given lx = dL/dx', lv = dL/dv' the step's vector-Jacobian product is
//   mu = lv + dt lx,  dL/dv = D mu,  g_i = D dt k_i mu_i
//   dL/dx_k = lx_k + sum_j K(r_kj) (m_k g_j - m_j g_k),
//             K(r) = inv^3 I - 3 inv^5 r r^T
//   dL/dm_k += -sum_j inv^3 (r_kj . g_j) [through a]
//              + D dt mu_k . a_k          [through k, reference kick only]
// The pair sum is evaluated as
//   out_k = m_k P - q g_k - 3 Q,  P = sum inv^3 g_j,  q = sum inv^3 m_j,
//   Q = sum inv^5 (m_k (r.g_j) - m_j (r.g_k)) r
// (26 FP32 operations and one rsqrt per pair), split stream-K over
// persistent CTAs like the forward force kernel; each CTA segment writes
// (out, dm) to its partial slot and the update kernel sums them in CTA order.
//
// The pair term of out is antisymmetric: with r = x_j - x_k,
//   T_kj = m_k inv^3 g_j - m_j inv^3 g_k - 3 inv^5 (m_k r.g_j - m_j r.g_k) r
// and T_jk = -T_kj, while the mass terms are -inv^3 r.g_j on k and
// +inv^3 r.g_k on j.  sym_vjp_kernel therefore evaluates each unordered pair
// once on the forward symmetric kernel's layout (row blocks x 32-body
// chunks, the chunk rotating through the warp with its accumulated reaction):
// 18 shared operations + 8 per side = 34 FP32 operations and one rsqrt per
// pair, 17 per ordered interaction instead of 26.  Systems of up to 7000 bodies
// take both orders of every pair and a whole reverse step in one launch instead
// (small_vjp_kernel).
#include "nb_vjp.cuh"

namespace nb {

template <int NT, int BPT>
__global__ void __launch_bounds__(NT) vjp_pair_kernel(const float4 *__restrict__ pos,
                                                      const float4 *__restrict__ gbuf, int n,
                                                      float eps2, float4 *__restrict__ partial,
                                                      long long total, int ngroups)
{
    constexpr int TB = NT * BPT;
    __shared__ __align__(16) float4 sP[NT];
    __shared__ __align__(16) float4 sG[NT];
    const int t = threadIdx.x;
    const int c = blockIdx.x;
    long long it = sk_start(c, total, gridDim.x);
    const long long end = sk_start(c + 1, total, gridDim.x);
    const float4 pad = make_float4(kPadCoord, kPadCoord, kPadCoord, 0.f);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);

    while (it < end) {
        const int tb = (int)(it / ngroups);
        const long long tb_first = (long long)tb * ngroups;
        const long long seg_end = end < tb_first + ngroups ? end : tb_first + ngroups;
        const int j0 = (int)(it - tb_first) * kGroup;
        const int j1 = min((int)(seg_end - tb_first) * kGroup, n);

        float px[BPT], py[BPT], pz[BPT], pm[BPT], gx[BPT], gy[BPT], gz[BPT];
        float Px[BPT], Py[BPT], Pz[BPT], Q0[BPT], Q1[BPT], Q2[BPT], q[BPT], dm[BPT];
#pragma unroll
        for (int k = 0; k < BPT; ++k) {
            const int i = tb * TB + t + k * NT;
            const float4 a = i < n ? pos[i] : zero;
            const float4 g = i < n ? gbuf[i] : zero;
            px[k] = a.x; py[k] = a.y; pz[k] = a.z; pm[k] = a.w;
            gx[k] = g.x; gy[k] = g.y; gz[k] = g.z;
            Px[k] = Py[k] = Pz[k] = Q0[k] = Q1[k] = Q2[k] = q[k] = dm[k] = 0.f;
        }
        float4 nxp = (j0 + t < j1) ? pos[j0 + t] : pad;
        float4 nxg = (j0 + t < j1) ? gbuf[j0 + t] : zero;
        for (int jt = j0; jt < j1; jt += NT) {
            __syncthreads();
            sP[t] = nxp;
            sG[t] = nxg;
            __syncthreads();
            if (jt + NT < j1) {
                const int jn = jt + NT + t;
                nxp = jn < j1 ? pos[jn] : pad;
                nxg = jn < j1 ? gbuf[jn] : zero;
            }
            const int cnt = min(NT, j1 - jt);
            const int cnt2 = (cnt + 1) & ~1;  // entries past cnt are zero-mass, zero-g pads
            for (int j = 0; j < cnt2; j += 2) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const float4 s = sP[j + u];
                    const float4 g = sG[j + u];
#pragma unroll
                    for (int k = 0; k < BPT; ++k) {
                        const float rx = s.x - px[k], ry = s.y - py[k], rz = s.z - pz[k];
                        float d2 = fmaf(rx, rx, eps2);
                        d2 = fmaf(ry, ry, d2);
                        d2 = fmaf(rz, rz, d2);
                        const float inv = rsqrt_approx(d2);
                        const float inv2 = inv * inv;
                        const float inv3 = inv2 * inv;
                        const float inv5 = inv3 * inv2;
                        Px[k] = fmaf(inv3, g.x, Px[k]);
                        Py[k] = fmaf(inv3, g.y, Py[k]);
                        Pz[k] = fmaf(inv3, g.z, Pz[k]);
                        q[k] = fmaf(inv3, s.w, q[k]);
                        const float rgj = fmaf(rz, g.z, fmaf(ry, g.y, rx * g.x));
                        const float rgk = fmaf(rz, gz[k], fmaf(ry, gy[k], rx * gx[k]));
                        const float cc = inv5 * fmaf(pm[k], rgj, -(s.w * rgk));
                        Q0[k] = fmaf(cc, rx, Q0[k]);
                        Q1[k] = fmaf(cc, ry, Q1[k]);
                        Q2[k] = fmaf(cc, rz, Q2[k]);
                        dm[k] = fmaf(inv3, rgj, dm[k]);
                    }
                }
            }
        }
        float4 *dst = partial + (size_t)(c + tb) * TB;
#pragma unroll
        for (int k = 0; k < BPT; ++k) {
            const float ox = fmaf(pm[k], Px[k], fmaf(-q[k], gx[k], -3.f * Q0[k]));
            const float oy = fmaf(pm[k], Py[k], fmaf(-q[k], gy[k], -3.f * Q1[k]));
            const float oz = fmaf(pm[k], Pz[k], fmaf(-q[k], gz[k], -3.f * Q2[k]));
            dst[t + k * NT] = make_float4(ox, oy, oz, -dm[k]);
        }
        it = seg_end;
    }
}

// One CTA's share of a row: row block I's targets against the chunks
// [kc0, kc1), target-side sums to dst, reactions to sp.  Not inlined into the
// loop over rows, as sym_row_segment of nb_sym.cu.
template <int W, int BPT>
__device__ __noinline__ void sym_vjp_segment(const float4 *pos, const float4 *gbuf, int n,
                                             float eps2, float4 *dst, float4 *sp, int I, int kc0, int kc1)
{
    constexpr int NP = BPT / 2;
    constexpr int WB = 32 * BPT;
    constexpr int RB = W * WB;
    constexpr int RC = RB / 32;
    __shared__ __align__(16) float4 sC[32];
    __shared__ __align__(16) float4 sG[32];
    __shared__ float sF[8][W][32];
    const int lane = threadIdx.x & 31;
    const int wid = threadIdx.x >> 5;
    const int tbase = I * RB + wid * WB;
    const float4 pad = make_float4(kPadCoord, kPadCoord, kPadCoord, 0.f);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const f2 EPS2 = f2_pack(eps2, eps2);

    VjpTargets<NP> T;
    auto idx = [&](int t) { return tbase + lane + 32 * t; };
    T.load([&](int t) { return idx(t) < n ? pos[idx(t)] : zero; }, [&](int t) { return idx(t) < n ? gbuf[idx(t)] : zero; });
    // the next chunk is read ahead
    float4 nxc = kc0 * 32 + lane < n ? pos[kc0 * 32 + lane] : pad;
    float4 nxg = kc0 * 32 + lane < n ? gbuf[kc0 * 32 + lane] : zero;
#pragma unroll 1
    for (int kc = kc0; kc < kc1; ++kc) {
        const int jb = kc * 32;
        __syncthreads();  // previous chunk: sC/sG and sF reads are done
        if (wid == 0) {
            sC[lane] = nxc;
            sG[lane] = nxg;
        }
        __syncthreads();
        if (wid == 0) {
            nxc = jb + 32 + lane < n ? pos[jb + 32 + lane] : pad;
            nxg = jb + 32 + lane < n ? gbuf[jb + 32 + lane] : zero;
        }
        if (kc < (I + 1) * RC) {
            vjp_chunk_pull(T, sC, sG, EPS2);  // chunk inside the own row block: target side only
            continue;
        }
        float r8[8];
        vjp_chunk_react(T, sC, sG, lane, EPS2, r8);
        if constexpr (W > 1) {
#pragma unroll
            for (int k = 0; k < 8; ++k) sF[k][wid][lane] = r8[k];
            __syncthreads();
            if (wid == 0) {
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    r8[k] = 0.f;
#pragma unroll
                    for (int w = 0; w < W; ++w) r8[k] += sF[k][w][lane];
                }
            }
        }
        if (wid == 0 && jb + lane < n) sp[jb + lane - (I + 1) * RB] = vjp_reaction(sC[lane], sG[lane], r8);
    }
    dst += wid * WB + lane;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        float4 a, b;
        T.out(p, a, b);
        dst[64 * p] = a;
        dst[64 * p + 32] = b;
    }
}

template <int W, int BPT, int MINB>
__global__ void __launch_bounds__(32 * W, MINB) sym_vjp_kernel(const float4 *pos,
                                                               const float4 *gbuf, int n,
                                                               float eps2, float4 *tpart,
                                                               float4 *spart,
                                                               long long total, int nc, int nrb)
{
    pdl_wait();
    constexpr int RB = W * 32 * BPT;
    constexpr int RC = RB / 32;
    const int c = blockIdx.x;
    long long it = sk_start(c, total, gridDim.x);
    const long long end = sk_start(c + 1, total, gridDim.x);
    while (it < end) {
        const int I = sym_row_of(it, nc, RC, nrb);
        const long long rfirst = sym_prefix(I, nc, RC);
        const long long rend = sym_prefix(I + 1, nc, RC);
        const long long seg_end = end < rend ? end : rend;
        sym_vjp_segment<W, BPT>(pos, gbuf, n, eps2, tpart + (size_t)(c + I) * RB, spart + sym_soff(I, n, RB), I,
                                I * RC + (int)(it - rfirst), I * RC + (int)(seg_end - rfirst));
        it = seg_end;
    }
}

// g_i = D dt k_i (lv_i + dt lx_i) for the first reverse step.
__global__ void adj_g_kernel(const float4 *__restrict__ pos, const float4 *__restrict__ lx,
                             const float4 *__restrict__ lv, float4 *__restrict__ gbuf, int n,
                             float damping, float dt, int kick, float G)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float k = kick == NB_KICK_REFERENCE ? pos[i].w : G;
    const float4 x = lx[i], v = lv[i];
    const float f = damping * dt * k;
    gbuf[i] = make_float4(f * fmaf(dt, x.x, v.x), f * fmaf(dt, x.y, v.y), f * fmaf(dt, x.z, v.z), 0.f);
}

// Directed layout: sum the partial slots of the CTAs that covered the body's
// target block (CTA order), then update.
__global__ void adj_update_kernel(const float4 *__restrict__ partial, int n, int tbsize,
                                  long long total, int ngroups, int grid,
                                  const float4 *__restrict__ pos, const float4 *__restrict__ acc,
                                  float4 *__restrict__ lx, float4 *__restrict__ lv,
                                  float *__restrict__ gm, float4 *__restrict__ gbuf, float damping,
                                  float dt, int kick, float G, int want_next_g)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int tb = i / tbsize;
    const int li = i - tb * tbsize;
    const long long first = (long long)tb * ngroups;
    const int c0 = sk_owner(first, total, grid);
    const int c1 = sk_owner(first + ngroups - 1, total, grid);
    float ox = 0.f, oy = 0.f, oz = 0.f, odm = 0.f;
    for (int c = c0; c <= c1; ++c) {
        const float4 q = partial[(size_t)(c + tb) * tbsize + li];
        ox += q.x;
        oy += q.y;
        oz += q.z;
        odm += q.w;
    }
    adj_body_update(i, ox, oy, oz, odm, pos, acc, lx, lv, gm, gbuf, damping, dt, kick, G, want_next_g);
}

// Symmetric layout: target-side slots and the source-side entries of rows
// 0..I-1, then the per-body update.  Four threads share a body (thread q of
// the quad sums slots c0+q, c0+q+4, ... and rows q, q+4, ..., the quad
// combines its sums as (s0 + s1) + (s2 + s3), a fixed order): the row walk of
// the last row blocks is what bounds this kernel.
constexpr int kAdjUpdBlock = 256;

__global__ void __launch_bounds__(kAdjUpdBlock) adj_update_sym_kernel(
    const float4 *tpart, const float4 *spart, int n, int rb, int nc, int nrb,
    long long total, int grid, const float4 *pos, const float4 *acc,
    float4 *lx, float4 *lv, float *gm, float4 *gbuf,
    float damping, float dt, int kick, float G, int want_next_g)
{
    pdl_wait();
    // bodies from the last one down, as in sym_integrate_kernel: the blocks
    // with the longest row walks start first
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int i = n - 1 - (int)(t >> 2), q = (int)(t & 3);
    const bool live = i >= 0;  // dead threads still take part in the shuffles
    float ox = 0.f, oy = 0.f, oz = 0.f, odm = 0.f;
    if (live) {
        const int rc = rb / 32;
        const int I = i / rb;
        const int c0 = sk_owner(sym_prefix(I, nc, rc), total, grid);
        const int c1 = sk_owner(sym_prefix(I + 1, nc, rc) - 1, total, grid);
        const int li = i - I * rb;
        auto add = [&](const float4 &v4) {
            ox += v4.x;
            oy += v4.y;
            oz += v4.z;
            odm += v4.w;
        };
        walk<4>(c0 + q, c1, 4, [&](int c) { return tpart[(size_t)(c + I) * rb + li]; }, add);
        walk<4>(q, I - 1, 4, [&](int r) { return spart[sym_soff(r, n, rb) + (i - (long long)(r + 1) * rb)]; }, add);
    }
#pragma unroll
    for (int m = 1; m <= 2; m <<= 1) {
        ox += __shfl_xor_sync(0xffffffffu, ox, m);
        oy += __shfl_xor_sync(0xffffffffu, oy, m);
        oz += __shfl_xor_sync(0xffffffffu, oz, m);
        odm += __shfl_xor_sync(0xffffffffu, odm, m);
    }
    if (!live || q != 0) return;
    adj_body_update(i, ox, oy, oz, odm, pos, acc, lx, lv, gm, gbuf, damping, dt, kick, G, want_next_g);
}

// A whole reverse step of a small system in one launch, as nb_small.cu does
// forward steps: a CTA owns TB bodies, its threads split the other side of every
// pair, the sums are reduced in the CTA and its first threads update their
// bodies.  The next step's g goes to gnext: other CTAs still read gbuf.
//
// Reverse step, GB300, us, against the symmetric kernels' two launches: N = 700
// 4.8 (14.8), 1376 6.5 (16.1), 3000 12.8 (17.6), 5000 29.4 (39.8), 6000 37.3 (39.1),
// 7000 50.2 (53.1), 9000 77.9 (67.4): the line is at 7000.  Bounds: latency (first
// loads, reduction) below N about 2000, then register-file reads, 26 operations
// for each order of a pair where the symmetric kernel takes 42 for both.  4
// bodies a CTA; 2, 6 and 8 are within 10 % and mostly behind (N = 3000: 13.9,
// 14.4, 14.1).
constexpr int kVjpSmallThreads = 128;
constexpr int kVjpSmallTargets = 4;
constexpr int kVjpSmallBodies = 7000;

template <int TB>
__global__ void __launch_bounds__(kVjpSmallThreads, 1)
    small_vjp_kernel(const float4 *pos, const float4 *gbuf, int n, float eps2, const float4 *acc, float4 *lx, float4 *lv,
                     float *gm, float4 *gnext, float damping, float dt, int kick, float G, int want_next_g)
{
    constexpr int NP = TB / 2, TP = pow2_up(TB), NW = kVjpSmallThreads / 32;
    __shared__ float red[NW][4 * TP];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int t0 = blockIdx.x * TB;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 pad = make_float4(kPadCoord, kPadCoord, kPadCoord, 0.f);
    const f2 EPS2 = f2_pack(eps2, eps2);
    pdl_wait();
    VjpTargets<NP> T;
    T.load([&](int t) { return t0 + t < n ? pos[t0 + t] : zero; }, [&](int t) { return t0 + t < n ? gbuf[t0 + t] : zero; });
    VjpSums none;
    float4 nx = tid < n ? pos[tid] : pad, ng = tid < n ? gbuf[tid] : zero;
    for (int j = tid; j - tid < n; j += kVjpSmallThreads) {
        VjpSource b;
        b.load(nx, ng);
        const int jn = j + kVjpSmallThreads;
        nx = jn < n ? pos[jn] : pad;
        ng = jn < n ? gbuf[jn] : zero;
#pragma unroll
        for (int p = 0; p < NP; ++p) T.template pair<false>(p, b, EPS2, none);
    }
    float s[4 * TP];
#pragma unroll
    for (int k = 4 * TB; k < 4 * TP; ++k) s[k] = 0.f;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        float4 a, b;
        T.out(p, a, b);
        s[8 * p] = a.x;
        s[8 * p + 1] = a.y;
        s[8 * p + 2] = a.z;
        s[8 * p + 3] = a.w;
        s[8 * p + 4] = b.x;
        s[8 * p + 5] = b.y;
        s[8 * p + 6] = b.z;
        s[8 * p + 7] = b.w;
    }
    const int t = warp_sum<TP, 4>(s, lane);
    if ((lane & (32 / TP - 1)) == 0) {
#pragma unroll
        for (int k = 0; k < 4; ++k) red[wid][4 * t + k] = s[k];
    }
    __syncthreads();
    const int i = t0 + tid;
    if (tid >= TB || i >= n) return;
    float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int w = 0; w < NW; ++w) {
#pragma unroll
        for (int k = 0; k < 4; ++k) o[k] += red[w][4 * tid + k];
    }
    adj_body_update(i, o[0], o[1], o[2], o[3], pos, acc, lx, lv, gm, gnext, damping, dt, kick, G, want_next_g);
}

typedef void (*vjp_kernel_t)(const float4 *, const float4 *, int, float, float4 *, long long, int);

static vjp_kernel_t vjp_kernel_for(int block, int bpt)
{
    if (block == 128 && bpt == 2) return vjp_pair_kernel<128, 2>;
    if (block == 128 && bpt == 4) return vjp_pair_kernel<128, 4>;
    if (block == 256 && bpt == 2) return vjp_pair_kernel<256, 2>;
    if (block == 256 && bpt == 4) return vjp_pair_kernel<256, 4>;
    return nullptr;
}

int adj_plan(int n, int block, int bpt, int device, SkPlan *pl)
{
    if (block == 0) block = 256;
    if (bpt == 0) bpt = 4;
    vjp_kernel_t k = vjp_kernel_for(block, bpt);
    if (!k) return set_error(NB_ERR_UNSUPPORTED, "adjoint kernel shape not compiled");
    SkPlan p;
    p.n = n;
    p.block = block;
    p.bpt = bpt;
    p.tbsize = block * bpt;
    p.ntb = (n + p.tbsize - 1) / p.tbsize;
    p.ngroups = (n + kGroup - 1) / kGroup;
    p.total = (long long)p.ntb * p.ngroups;
    int sms = 0, occ = 0;
    NB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    NB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, block, 0));
    if (occ < 1) return set_error(NB_ERR_UNSUPPORTED, "adjoint kernel does not fit on an SM");
    long long grid = (long long)sms * occ;
    if (p.total > 0 && grid > p.total) grid = p.total;
    p.grid = p.total > 0 ? (int)grid : 0;
    p.slots = p.total > 0 ? p.grid + p.ntb - 1 : 0;
    *pl = p;
    return NB_OK;
}

int adj_g(int n, const float4 *pos, const float4 *lx, const float4 *lv, float4 *gbuf, float damping,
          float dt, int kick, float G, cudaStream_t s)
{
    if (n == 0) return NB_OK;
    adj_g_kernel<<<(n + 255) / 256, 256, 0, s>>>(pos, lx, lv, gbuf, n, damping, dt, kick, G);
    NB_LAUNCH_CHECK("adj_g_kernel launch");
    return NB_OK;
}

int adj_vjp(const SkPlan &p, const float4 *pos, const float4 *gbuf, float eps2, float4 *partial,
            cudaStream_t s)
{
    if (p.total == 0) return NB_OK;
    vjp_kernel_t k = vjp_kernel_for(p.block, p.tbsize / p.block);
    if (!k) return set_error(NB_ERR_UNSUPPORTED, "adjoint kernel shape not compiled");
    k<<<p.grid, p.block, 0, s>>>(pos, gbuf, p.n, eps2, partial, p.total, p.ngroups);
    NB_LAUNCH_CHECK("vjp_pair_kernel launch");
    return NB_OK;
}

int adj_update(const SkPlan &p, const float4 *partial, const float4 *pos_prev, const float4 *acc,
               float4 *lx, float4 *lv, float *gm, float4 *gbuf, float damping, float dt, int kick,
               float G, int want_next_g, cudaStream_t s)
{
    if (p.n == 0) return NB_OK;
    adj_update_kernel<<<(p.n + 255) / 256, 256, 0, s>>>(partial, p.n, p.tbsize, p.total, p.ngroups,
                                                       p.grid, pos_prev, acc, lx, lv, gm, gbuf,
                                                       damping, dt, kick, G, want_next_g);
    NB_LAUNCH_CHECK("adj_update_kernel launch");
    return NB_OK;
}

typedef void (*sym_vjp_kernel_t)(const float4 *, const float4 *, int, float, float4 *, float4 *,
                                 long long, int, int);

static sym_vjp_kernel_t sym_vjp_kernel_for(int w, int bpt)
{
    if (w == 1 && bpt == 10) return sym_vjp_kernel<1, 10, 8>;
    if (w == 1 && bpt == 8) return sym_vjp_kernel<1, 8, 8>;
    if (w == 1 && bpt == 12) return sym_vjp_kernel<1, 12, 8>;
    if (w == 4 && bpt == 8) return sym_vjp_kernel<4, 8, 2>;
    if (w == 8 && bpt == 8) return sym_vjp_kernel<8, 8, 1>;
    return nullptr;
}

int sym_vjp_plan(int n, int warps, int bpt, int device, SymPlan *pl)
{
    if (warps == 0 && bpt == 0) {
        // one-warp CTAs x 10 targets (row block 320; the fastest of the
        // shapes timed on GB300 at N = 16384 and 65536), then 4 x 8 (1024),
        // 8 x 8 (2048) while the source-side array is over budget
        static const int shapes[3][2] = {{1, 10}, {4, 8}, {8, 8}};
        int s = 0;
        while (s < 2 && sym_spart_entries(n, shapes[s][0] * 32 * shapes[s][1]) * (long long)sizeof(float4) >
                            kSymSpartBudget)
            ++s;
        warps = shapes[s][0];
        bpt = shapes[s][1];
    }
    sym_vjp_kernel_t k = sym_vjp_kernel_for(warps, bpt);
    if (!k) return set_error(NB_ERR_UNSUPPORTED, "symmetric adjoint kernel shape not compiled");
    SymPlan p;
    p.n = n;
    p.warps = warps;
    p.bpt = bpt;
    p.rb = warps * 32 * bpt;
    p.nc = (n + 31) / 32;
    p.nrb = (n + p.rb - 1) / p.rb;
    p.total = n > 0 ? sym_prefix(p.nrb, p.nc, p.rb / 32) : 0;
    int sms = 0, occ = 0;
    NB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    NB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, 32 * warps, 0));
    if (occ < 1) return set_error(NB_ERR_UNSUPPORTED, "symmetric adjoint kernel does not fit on an SM");
    long long grid = (long long)sms * occ;
    if (p.total > 0 && grid > p.total) grid = p.total;
    p.grid = p.total > 0 ? (int)grid : 0;
    p.slots = p.total > 0 ? p.grid + p.nrb - 1 : 0;
    p.spart_size = sym_spart_entries(n, p.rb);
    p.small = warps == 1 && bpt == 10 && n <= kVjpSmallBodies;
    *pl = p;
    return NB_OK;
}

int small_vjp(int n, const float4 *pos, const float4 *gbuf, float eps2, const float4 *acc, float4 *lx, float4 *lv,
              float *gm, float4 *gnext, float damping, float dt, int kick, float G, int want_next_g, cudaStream_t s)
{
    if (n == 0) return NB_OK;
    return pdl_launch("small_vjp_kernel launch", small_vjp_kernel<kVjpSmallTargets>,
                      (unsigned)((n + kVjpSmallTargets - 1) / kVjpSmallTargets), kVjpSmallThreads, s, pos, gbuf, n, eps2,
                      acc, lx, lv, gm, gnext, damping, dt, kick, G, want_next_g);
}

int sym_vjp(const SymPlan &p, const float4 *pos, const float4 *gbuf, float eps2, float4 *tpart,
            float4 *spart, cudaStream_t s)
{
    if (p.total == 0) return NB_OK;
    sym_vjp_kernel_t k = sym_vjp_kernel_for(p.warps, p.bpt);
    if (!k) return set_error(NB_ERR_UNSUPPORTED, "symmetric adjoint kernel shape not compiled");
    return pdl_launch("sym_vjp_kernel launch", k, p.grid, 32 * p.warps, s, pos, gbuf, p.n, eps2, tpart, spart, p.total,
                      p.nc, p.nrb);
}

int adj_update_sym(const SymPlan &p, const float4 *tpart, const float4 *spart, const float4 *pos_prev,
                   const float4 *acc, float4 *lx, float4 *lv, float *gm, float4 *gbuf, float damping,
                   float dt, int kick, float G, int want_next_g, cudaStream_t s)
{
    if (p.n == 0) return NB_OK;
    const long long threads = 4ll * p.n;  // a quad of threads per body
    return pdl_launch("adj_update_sym_kernel launch", adj_update_sym_kernel,
                      (unsigned)((threads + kAdjUpdBlock - 1) / kAdjUpdBlock), kAdjUpdBlock, s, tpart, spart, p.n, p.rb,
                      p.nc, p.nrb, p.total, p.grid, pos_prev, acc, lx, lv, gm, gbuf, damping, dt, kick, G, want_next_g);
}

}  // namespace nb
