// nb_ics.cu -- seeded initial conditions generated on the GPU.
//
// The reference draws its bodies on the host with the C library's rand()
// (randomizeBodies, benchapps/nbody/seq/nbody.h:89-250; kept bit-exact in
// utc_gb300/task/nbody_init.h for the app).  For large synthetic workloads
// the bodies are drawn here instead, one thread per body, from a
// counter-based generator: stream k of body i of seed s is
//   splitmix64(s ^ splitmix64(i * 256 + k)),  k < 256
// (the SplitMix64 finaliser, Steele, Lea & Flood 2014), so a body's draw does
// not depend on the launch shape or on the other bodies.
//  * uniform cube: positions U[-1,1]^3, velocities U[-vmax,vmax]^3, masses
//    U[0.5,1.5]/n (total mass ~ 1);
//  * Plummer sphere (Aarseth, Henon & Wielen 1974): r = a / sqrt(X^-2/3 - 1)
//    with X uniform in (0, 0.999], speeds q * v_esc(r) with q drawn by
//    rejection from q^2 (1 - q^2)^(7/2), isotropic directions, masses M/n;
//    then the centre of mass and its velocity are moved to the origin
//    (FP64 block sums reduced in order by one block: deterministic);
//  * the reference app's own three configurations (randomizeBodies,
//    benchapps/nbody/seq/nbody.h:89-250) with this generator in place of
//    rand(), a = clusterScale, vmax = velocityScale, masses 1, vel.w = 1:
//    random (positions uniform in the ball of radius s = a max(1, n/1024),
//    velocities uniform in the ball of radius s vmax), shell (a unit
//    direction drawn by rejection from the cube, each coordinate scaled by
//    its own draw from [2.5a, 4a], velocity (pos x axis) a vmax with axis z,
//    or (y, x, 1) normalised when the direction is within 1e-6 of z) and
//    expand (positions uniform in the ball of radius s = a n/1024, or a when
//    s < 1; velocity the same point times s vmax).
//
// The FP64 pipe is what bounds this (1/74 of the FP32 rate on GB300), so FP64
// is kept to what the results need of it:
//  * the rejection tests are decided in FP32 from the leading 24 bits of the
//    draws, outside a band about the boundary that covers every rounding of
//    that; inside the band (about 4 tries in 1e5) the FP64 test decides, so
//    the draws that are taken are those of the FP64 test;
//  * float bodies of a Plummer sphere are computed in float-float arithmetic
//    (48 bits) and rounded once: as close to the FP64 values as FP64
//    arithmetic rounded to float is;
//  * the moments of float bodies are summed, and the centre subtracted, in
//    float-float too, and the centre is divided out once.
// 2^20 bodies, whole call, GB300: Plummer float 102 us (852 with all of it in
// FP64), double 374 (807); shell 127 (380) and 116 (369), random 127 (554).
// What is left of the float sphere is issue (1900 instructions a body, half
// of them the generator's 64-bit arithmetic) and the passes of the moments.
#include <cmath>
#include <type_traits>

#include "nb_internal.cuh"

namespace nb {

__device__ __forceinline__ unsigned long long splitmix64(unsigned long long z)
{
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// stream k of body i: 53 random bits above 11 to be dropped
__device__ __forceinline__ unsigned long long draw64(unsigned long long seed, unsigned long long i, unsigned k)
{
    return splitmix64(seed ^ splitmix64(i * 256ull + k));
}
// a draw as a uniform double in [0, 1)
__device__ __forceinline__ double unit64(unsigned long long h)
{
    return (double)(h >> 11) * (1.0 / 9007199254740992.0);
}
__device__ __forceinline__ double u01(unsigned long long seed, unsigned long long i, unsigned k)
{
    return unit64(draw64(seed, i, k));
}
// its leading 24 bits, below it by less than 2^-24
__device__ __forceinline__ float unit24(unsigned long long h) { return (float)(unsigned)(h >> 40) * 0x1p-24f; }

template <typename V4>
__device__ __forceinline__ V4 mk4(double x, double y, double z, double w)
{
    V4 r;
    r.x = x;
    r.y = y;
    r.z = z;
    r.w = w;
    return r;
}

// A point uniform in the unit ball by rejection from the cube: tries use
// streams k0, k0 + 1, ... (3 per try, 40 tries).  All 40 fail with
// probability 0.476^40 ~ 1e-13; then the last candidate is pulled inside.
// The FP32 coordinates are off by less than 1.3e-7, so |r|^2 near 1 by less
// than 8e-7: outside 1 -+ 2e-6 they decide as the FP64 ones do.
__device__ __forceinline__ void ball_point(unsigned long long seed, unsigned long long id, unsigned k0,
                                           double &x, double &y, double &z, double &len)
{
    // The FP64 point is formed once, after the loop, by all lanes together.
    unsigned long long hx = 0, hy = 0, hz = 0;
    auto form = [&] {
        x = 2.0 * unit64(hx) - 1.0;
        y = 2.0 * unit64(hy) - 1.0;
        z = 2.0 * unit64(hz) - 1.0;
        len = sqrt(x * x + y * y + z * z);
    };
    for (unsigned t = 0; t < 40; ++t) {
        hx = draw64(seed, id, k0 + 3 * t);
        hy = draw64(seed, id, k0 + 3 * t + 1);
        hz = draw64(seed, id, k0 + 3 * t + 2);
        const float fx = fmaf(2.f, unit24(hx), -1.f), fy = fmaf(2.f, unit24(hy), -1.f),
                    fz = fmaf(2.f, unit24(hz), -1.f);
        const float d2 = fmaf(fx, fx, fmaf(fy, fy, fz * fz));
        if (d2 < 1.f - 2e-6f) break;
        if (d2 > 1.f + 2e-6f) continue;
        form();
        if (len <= 1.0) break;
    }
    form();
    if (len <= 1.0) return;
    x *= 0.5 / len;
    y *= 0.5 / len;
    z *= 0.5 / len;
    len = 0.5;
}

// The speed fraction of a Plummer sphere by rejection from g(q) = q^2 (1 -
// q^2)^3.5 (max < 0.1), streams 8 + 2t and 9 + 2t: each try is accepted with
// probability 7 pi / 512 / 0.1 = 0.43, so all 64 tries miss with probability
// ~2e-16.  Returns the accepted draw of q; ok is false if all missed (q is
// then the mode of g, sqrt(2/9)).  FP32: q and y / 0.1 are below the FP64 ones
// by less than 6e-8, g' stays below 0.5 and the roundings below 1e-7, so
// outside +-1e-6 the FP32 test decides as the FP64 one does.
__device__ __forceinline__ unsigned long long plummer_speed(unsigned long long seed, unsigned long long id, bool &ok)
{
    ok = true;
    for (unsigned t = 0; t < 64; ++t) {
        const unsigned long long hq = draw64(seed, id, 8 + 2 * t), hy = draw64(seed, id, 9 + 2 * t);
        const float q = unit24(hq), q2 = q * q, t1 = 1.f - q2;
        const float d = fmaf(q2, t1 * t1 * t1 * sqrtf(t1), -0.1f * unit24(hy));
        if (d > 1e-6f) return hq;
        if (d < -1e-6f) continue;
        const double qq = unit64(hq), yy = 0.1 * unit64(hy), tt = 1.0 - qq * qq;
        if (yy < qq * qq * (tt * tt * tt * sqrt(tt))) return hq;
    }
    ok = false;
    return 0;
}

template <typename V4>
__global__ void ics_kernel(int kind, int n, unsigned long long seed, double a, double G, double M,
                           double vmax, V4 *__restrict__ pos, V4 *__restrict__ vel)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned long long id = (unsigned long long)i;
    if (kind == 2 || kind == 4) {  // reference random / expand
        double x, y, z, len;
        ball_point(seed, id, 8, x, y, z, len);
        double s = a * fmax(1.0, n / 1024.0);
        if (kind == 4) {
            s = a * (n / 1024.0);
            if (s < 1.0) s = a;
            pos[i] = mk4<V4>(x * s, y * s, z * s, 1.0);
            vel[i] = mk4<V4>(x * s * vmax, y * s * vmax, z * s * vmax, 1.0);
            return;
        }
        double vx, vy, vz, vlen;
        ball_point(seed, id, 128, vx, vy, vz, vlen);
        pos[i] = mk4<V4>(x * s, y * s, z * s, 1.0);
        vel[i] = mk4<V4>(vx * s * vmax, vy * s * vmax, vz * s * vmax, 1.0);
        return;
    }
    if (kind == 3) {  // reference shell
        double x, y, z, len;
        ball_point(seed, id, 8, x, y, z, len);
        if (len > 1e-6) {  // one FP64 division instead of three
            const double il = 1.0 / len;
            x *= il;
            y *= il;
            z *= il;
        }
        const double inner = 2.5 * a, outer = 4.0 * a;
        const double px = x * (inner + (outer - inner) * u01(seed, id, 128));
        const double py = y * (inner + (outer - inner) * u01(seed, id, 129));
        const double pz = z * (inner + (outer - inner) * u01(seed, id, 130));
        double ax = 0.0, ay = 0.0, az = 1.0;
        if (1.0 - z < 1e-6) {
            const double il = rsqrt(y * y + x * x + 1.0);
            ax = y * il;
            ay = x * il;
            az = il;
        }
        const double vs = a * vmax;
        pos[i] = mk4<V4>(px, py, pz, 1.0);
        vel[i] = mk4<V4>((py * az - pz * ay) * vs, (pz * ax - px * az) * vs, (px * ay - py * ax) * vs, 1.0);
        return;
    }
    if (kind == 0) {  // uniform cube
        pos[i] = mk4<V4>(2.0 * u01(seed, id, 0) - 1.0, 2.0 * u01(seed, id, 1) - 1.0,
                         2.0 * u01(seed, id, 2) - 1.0, (0.5 + u01(seed, id, 3)) / n);
        vel[i] = mk4<V4>(vmax * (2.0 * u01(seed, id, 4) - 1.0), vmax * (2.0 * u01(seed, id, 5) - 1.0),
                         vmax * (2.0 * u01(seed, id, 6) - 1.0), 1.0);
        return;
    }
    // Plummer sphere
    // x1^(-2/3) as rcbrt(x1)^2, (1 - q^2)^3.5 as t^3 sqrt(t) and
    // (r^2 + a^2)^(-1/4) as rsqrt(sqrt(.)): the same quantities without pow,
    // whose FP64 log/exp dominated the sampler on a part with a slow FP64 pipe
    const double x1 = fmax(0.999 * u01(seed, id, 0), 1e-300);
    const double c1 = rcbrt(x1);
    const double r = a / sqrt(c1 * c1 - 1.0);
    double ct = 2.0 * u01(seed, id, 1) - 1.0;
    double st = sqrt(fmax(0.0, 1.0 - ct * ct));
    double sp, cp;
    sincospi(2.0 * u01(seed, id, 2), &sp, &cp);
    pos[i] = mk4<V4>(r * st * cp, r * st * sp, r * ct, M / n);
    bool ok;
    const unsigned long long hq = plummer_speed(seed, id, ok);
    const double q = ok ? unit64(hq) : 0.4714045207910317;
    const double vesc = sqrt(2.0 * G * M) * rsqrt(sqrt(r * r + a * a));
    ct = 2.0 * u01(seed, id, 3) - 1.0;
    st = sqrt(fmax(0.0, 1.0 - ct * ct));
    sincospi(2.0 * u01(seed, id, 4), &sp, &cp);
    const double v = q * vesc;
    vel[i] = mk4<V4>(v * st * cp, v * st * sp, v * ct, 1.0);
}

// ---------------------------------------------------------------------------
// float bodies of a Plummer sphere in float-float arithmetic
// ---------------------------------------------------------------------------
struct FF {  // h + l, |l| <= ulp(h) / 2
    float h, l;
};
__device__ __forceinline__ FF ff_norm(float h, float l)  // |h| >= |l|
{
    FF r;
    r.h = __fadd_rn(h, l);
    r.l = __fsub_rn(l, __fsub_rn(r.h, h));
    return r;
}
__device__ __forceinline__ FF ff_mul(FF a, FF b)
{
    const float p = __fmul_rn(a.h, b.h);
    float e = __fmaf_rn(a.h, b.h, -p);
    e = __fmaf_rn(a.h, b.l, e);
    return ff_norm(p, __fmaf_rn(a.l, b.h, e));
}
__device__ __forceinline__ FF ff_add(FF a, FF b)
{
    float s, e;
    two_sum(a.h, b.h, s, e);
    return ff_norm(s, __fadd_rn(e, __fadd_rn(a.l, b.l)));
}
__device__ __forceinline__ FF ff_one(float h) { return FF{h, 0.f}; }
// 1/sqrt(a), a > 0: the FP32 value and one Halley step
__device__ __forceinline__ FF ff_rsqrt(FF a)
{
    const float y = rsqrtf(a.h);
    const float q = __fmul_rn(y, y), qe = __fmaf_rn(y, y, -q);
    float u = __fmaf_rn(-a.h, q, 1.f);
    u = __fsub_rn(u, __fmaf_rn(a.h, qe, __fmul_rn(a.l, q)));
    return ff_norm(y, __fmul_rn(y, __fmul_rn(u, __fmaf_rn(0.375f, u, 0.5f))));
}
// sqrt(a), a >= 0
__device__ __forceinline__ FF ff_sqrt(FF a) { return a.h > 0.f ? ff_mul(a, ff_rsqrt(a)) : ff_one(0.f); }
// a^(-1/3), a > 0: the FP32 value and one Halley step, y (1 + e/3 + 2 e^2/9)
// with e = 1 - a y^3
__device__ __forceinline__ FF ff_rcbrt(FF a)
{
    const FF y = ff_one(rcbrtf(a.h));
    const FF t = ff_mul(a, ff_mul(ff_mul(y, y), y));
    const float e = __fsub_rn(__fsub_rn(1.f, t.h), t.l);
    return ff_norm(y.h, __fmul_rn(y.h, __fmul_rn(e, __fmaf_rn(0.22222222f, e, 0.33333333f))));
}
// a draw: the leading 24 bits and the other 29, rounded
__device__ __forceinline__ FF ff_unit(unsigned long long h)
{
    return ff_norm((float)(unsigned)(h >> 40) * 0x1p-24f, (float)((unsigned)(h >> 11) & 0x1fffffffu) * 0x1p-53f);
}
// sin and cos of 2 pi u, 0 <= u <= 1: u to the nearest quarter k / 4, the rest
// |f| <= 1/8 turns by the Taylor series in z = (2 pi f)^2 <= 0.617, their
// leading coefficients in float-float.
__device__ __forceinline__ void ff_sincos_turn(FF u, FF &sn, FF &cs)
{
    const float k = rintf(4.f * u.h);
    float fh, fl;
    two_sum(u.h, -0.25f * k, fh, fl);
    const FF x = ff_mul(ff_norm(fh, __fadd_rn(fl, u.l)), FF{6.2831855f, -1.7484555e-07f});  // 2 pi
    const FF z = ff_mul(x, x);
    float p = fmaf(z.h, fmaf(z.h, fmaf(z.h, -2.5052108e-08f, 2.7557319e-06f), -1.9841270e-04f), 8.3333333e-03f);
    const FF s3 = ff_add(FF{-0.16666667f, 4.9670538e-09f}, ff_mul(z, ff_one(p)));  // -1/6 + z/120 - ...
    const FF sv = ff_add(x, ff_mul(ff_mul(x, z), s3));
    p = fmaf(z.h, fmaf(z.h, fmaf(z.h, -2.7557319e-07f, 2.4801587e-05f), -1.3888889e-03f), 0.f);
    FF c4 = ff_add(FF{0.041666668f, -1.2417635e-09f}, ff_one(p));  // 1/24 - z/720 + ...
    c4 = ff_add(ff_one(-0.5f), ff_mul(z, c4));
    const FF cv = ff_add(ff_one(1.f), ff_mul(z, c4));
    const int q = (int)k & 3;
    const FF a = q & 1 ? cv : sv, b = q & 1 ? sv : cv;  // sin, cos before their signs
    const float sa = q & 2 ? -1.f : 1.f, sb = q == 1 || q == 2 ? -1.f : 1.f;
    sn = FF{sa * a.h, sa * a.l};
    cs = FF{sb * b.h, sb * b.l};
}
// length times the direction of the draws hc (cosine of the polar angle, 2 u -
// 1) and hf (azimuth)
__device__ __forceinline__ float3 ff_sphere(FF len, unsigned long long hc, unsigned long long hf)
{
    const FF u = ff_unit(hc);
    const FF c = ff_add(FF{2.f * u.h, 2.f * u.l}, ff_one(-1.f));
    // sin^2 = 1 - c^2 = 4 u (1 - u)
    const FF w = ff_mul(u, ff_add(ff_one(1.f), FF{-u.h, -u.l}));
    const FF st = ff_mul(len, ff_sqrt(FF{4.f * w.h, 4.f * w.l}));
    FF sn, cs;
    ff_sincos_turn(ff_unit(hf), sn, cs);
    return make_float3(ff_mul(st, cs).h, ff_mul(st, sn).h, ff_mul(len, c).h);
}

// vs = sqrt(2 G M)
__global__ void __launch_bounds__(256) ics_plummer_f32_kernel(int n, unsigned long long seed, FF a, FF vs, float m,
                                                              float4 *__restrict__ pos, float4 *__restrict__ vel)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned long long id = (unsigned long long)i;
    const FF u = ff_unit(draw64(seed, id, 0));
    FF r = ff_one(0.f);
    if (u.h > 0.f) {  // r = a / sqrt((0.999 u)^(-2/3) - 1)
        const FF c = ff_rcbrt(ff_mul(u, FF{0.99900001f, -1.2874603e-08f}));
        r = ff_mul(a, ff_rsqrt(ff_add(ff_mul(c, c), ff_one(-1.f))));
    }
    const float3 p = ff_sphere(r, draw64(seed, id, 1), draw64(seed, id, 2));
    bool ok;
    const unsigned long long hq = plummer_speed(seed, id, ok);
    const FF q = ok ? ff_unit(hq) : FF{0.47140452f, -1.8663626e-09f};
    const FF w = ff_rsqrt(ff_add(ff_mul(r, r), ff_mul(a, a)));  // (r^2 + a^2)^(-1/2)
    const float3 v = ff_sphere(ff_mul(q, ff_mul(vs, ff_sqrt(w))), draw64(seed, id, 3), draw64(seed, id, 4));
    pos[i] = make_float4(p.x, p.y, p.z, m);
    vel[i] = make_float4(v.x, v.y, v.z, 1.f);
}

// ---------------------------------------------------------------------------
// the centre of the (equal) masses and its velocity, moved to zero
// ---------------------------------------------------------------------------
// Each thread sums bodies i, i + grid, ... (float bodies as two-sums, doubles in
// FP64), a block its threads by a tree, and one block of 6 x 128 threads the
// blocks; always in the same order.
constexpr int kIcsBlock = 256;
constexpr int kIcsFinal = 128;

template <typename V4>
__global__ void __launch_bounds__(kIcsBlock) ics_moments_kernel(int n, const V4 *__restrict__ pos,
                                                                const V4 *__restrict__ vel, double *__restrict__ part)
{
    __shared__ double red[6][kIcsBlock];
    double sum[6];
    if constexpr (sizeof(V4) == sizeof(float4)) {
        float h[6] = {0, 0, 0, 0, 0, 0}, l[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll 4
        for (int i = blockIdx.x * kIcsBlock + threadIdx.x; i < n; i += gridDim.x * kIcsBlock) {
            const float4 p = pos[i], v = vel[i];
            const float x[6] = {p.x, p.y, p.z, v.x, v.y, v.z};
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                float e;
                two_sum(h[q], x[q], h[q], e);
                l[q] += e;
            }
        }
#pragma unroll
        for (int q = 0; q < 6; ++q) sum[q] = (double)h[q] + (double)l[q];
    } else {
#pragma unroll
        for (int q = 0; q < 6; ++q) sum[q] = 0.0;
        for (int i = blockIdx.x * kIcsBlock + threadIdx.x; i < n; i += gridDim.x * kIcsBlock) {
            const V4 p = pos[i], v = vel[i];
            sum[0] += p.x;
            sum[1] += p.y;
            sum[2] += p.z;
            sum[3] += v.x;
            sum[4] += v.y;
            sum[5] += v.z;
        }
    }
    for (int q = 0; q < 6; ++q) red[q][threadIdx.x] = sum[q];
    __syncthreads();
    for (int w = kIcsBlock / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w)
            for (int q = 0; q < 6; ++q) red[q][threadIdx.x] += red[q][threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x < 6) part[(size_t)blockIdx.x * 6 + threadIdx.x] = red[threadIdx.x][0];
}

// out[q]: what is subtracted, as a double or (float bodies) a float-float.  The
// mean over the bodies, all of mass m; with masses that are not positive the
// mass-weighted sum itself.
template <typename S>
__global__ void __launch_bounds__(6 * kIcsFinal)
    ics_moments_final(const double *__restrict__ part, int nblocks, int n, double m, S *__restrict__ out)
{
    __shared__ double red[6][kIcsFinal];
    const int q = threadIdx.x / kIcsFinal, j = threadIdx.x % kIcsFinal;
    double s = 0;
#pragma unroll 8
    for (int b = j; b < nblocks; b += kIcsFinal) s += part[(size_t)b * 6 + q];
    red[q][j] = s;
    __syncthreads();
    for (int w = kIcsFinal / 2; w > 0; w >>= 1) {
        if (j < w) red[q][j] += red[q][j + w];
        __syncthreads();
    }
    if (j != 0) return;
    s = m > 0 ? red[q][0] / n : red[q][0] * m;
    if constexpr (std::is_same<S, FF>::value) {
        out[q].h = (float)s;
        out[q].l = (float)(s - (double)out[q].h);
    } else {
        out[q] = s;
    }
}

__device__ __forceinline__ double ics_shift(double x, double s) { return x - s; }
__device__ __forceinline__ float ics_shift(float x, FF s)  // x - s, rounded once
{
    float h, e;
    two_sum(x, -s.h, h, e);
    return __fadd_rn(h, __fsub_rn(e, s.l));
}

template <typename V4, typename S>
__global__ void ics_recenter_kernel(int n, V4 *__restrict__ pos, V4 *__restrict__ vel, const S *__restrict__ shift)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    V4 p = pos[i], v = vel[i];
    p.x = ics_shift(p.x, shift[0]);
    p.y = ics_shift(p.y, shift[1]);
    p.z = ics_shift(p.z, shift[2]);
    v.x = ics_shift(v.x, shift[3]);
    v.y = ics_shift(v.y, shift[4]);
    v.z = ics_shift(v.z, shift[5]);
    pos[i] = p;
    vel[i] = v;
}

template <typename V4>
static int ics_launch(int kind, int n, unsigned long long seed, double a, double G, double M,
                      double vmax, V4 *pos, V4 *vel, double *scratch, cudaStream_t s)
{
    const int blocks = (n + kIcsBlock - 1) / kIcsBlock;
    // float-float: factors well inside the float range (others in FP64)
    const double vs = std::sqrt(2.0 * G * M);
    auto fits = [](double x) { return x >= 0x1p-40 && x <= 0x1p40; };
    bool done = false;
    if constexpr (sizeof(V4) == sizeof(float4)) {
        if (kind == 1 && fits(a) && fits(vs)) {
            const FF fa = {(float)a, (float)(a - (double)(float)a)}, fv = {(float)vs, (float)(vs - (double)(float)vs)};
            ics_plummer_f32_kernel<<<blocks, kIcsBlock, 0, s>>>(n, seed, fa, fv, (float)(M / n), pos, vel);
            done = true;
        }
    }
    if (!done) ics_kernel<V4><<<blocks, kIcsBlock, 0, s>>>(kind, n, seed, a, G, M, vmax, pos, vel);
    NB_LAUNCH_CHECK("ics_kernel launch");
    if (kind == 1) {
        int dev = 0, sms = 0;
        NB_CUDA(cudaGetDevice(&dev));
        NB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        const int mb = blocks < 4 * sms ? blocks : 4 * sms;
        const double m = sizeof(V4) == sizeof(float4) ? (double)(float)(M / n) : M / n;
        ics_moments_kernel<V4><<<mb, kIcsBlock, 0, s>>>(n, pos, vel, scratch + 8);
        NB_LAUNCH_CHECK("ics_moments_kernel launch");
        typedef typename std::conditional<sizeof(V4) == sizeof(float4), FF, double>::type S;
        S *shift = reinterpret_cast<S *>(scratch);
        ics_moments_final<S><<<1, 6 * kIcsFinal, 0, s>>>(scratch + 8, mb, n, m, shift);
        NB_LAUNCH_CHECK("ics_moments_final launch");
        ics_recenter_kernel<V4, S><<<blocks, kIcsBlock, 0, s>>>(n, pos, vel, shift);
        NB_LAUNCH_CHECK("ics_recenter_kernel launch");
    }
    return NB_OK;
}

size_t ics_scratch_doubles(int n) { return 8 + 7 * (size_t)((n + kIcsBlock - 1) / kIcsBlock); }

}  // namespace nb

extern "C" int nb_ics_generate(int kind, int n, unsigned long long seed, double a, double G,
                               double M, double vmax, int precision, void *pos_dev, void *vel_dev,
                               void *scratch_dev, void *stream)
{
    if (kind < 0 || kind > 4)
        return nb::set_error(NB_ERR_INVALID,
                             "nb_ics_generate: kind is 0 (cube), 1 (Plummer), 2 (random), 3 (shell) or 4 (expand)");
    if (n < 0 || n > NB_MAX_BODIES) return nb::set_error(NB_ERR_INVALID, "nb_ics_generate: n must be in [0, 2^30]");
    if (precision != NB_F32 && precision != NB_F64)
        return nb::set_error(NB_ERR_INVALID, "nb_ics_generate: precision is NB_F32 or NB_F64");
    if (n == 0) return NB_OK;
    if (!pos_dev || !vel_dev || (kind == 1 && !scratch_dev))
        return nb::set_error(NB_ERR_INVALID, "nb_ics_generate: NULL buffer");
    if (!(a > 0) || !std::isfinite(G) || !std::isfinite(M) || !std::isfinite(vmax))
        return nb::set_error(NB_ERR_INVALID, "nb_ics_generate: bad parameters");
    cudaStream_t s = (cudaStream_t)stream;
    if (precision == NB_F32)
        return nb::ics_launch<float4>(kind, n, seed, a, G, M, vmax, (float4 *)pos_dev, (float4 *)vel_dev,
                                      (double *)scratch_dev, s);
    return nb::ics_launch<double4>(kind, n, seed, a, G, M, vmax, (double4 *)pos_dev, (double4 *)vel_dev,
                                   (double *)scratch_dev, s);
}

extern "C" size_t nb_ics_scratch_bytes(int n) { return nb::ics_scratch_doubles(n) * sizeof(double); }
