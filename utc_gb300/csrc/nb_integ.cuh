// nb_integ.cuh -- the FP64 integrators' common part (nb_sym64.cu, one system;
// nb_batch.cu, batches): partials summed by 4 or 8 warps, then the reference's kick /
// damping / drift in its order with unfused IEEE operations
// (bodysystem.cc:135-182), or the bare acceleration.
#pragma once

#include "nb_internal.cuh"

namespace nb {

constexpr int kIntegSlices = 8;  // warps of a block of 32 bodies

// Called by every thread of a block of S warps (S >= 4); lane l of every warp
// works on body i (its own value of i, < 0 for none).  sum(q, add) passes the
// partials of slice q to add in a fixed order; the slices are added in slice
// order.  scale(component, acc): the sum in the state's units.  acc_out != nullptr
// takes the bare acceleration (w: the sums' fourth component) and nothing is
// stepped.
//
// Memory and the narrow FP64 pipe's additions bound it; for small systems the
// chain of FP64 operations after the sums, which is why each component has a
// warp of its own and fetches its old state first (one system, N = 1000: 9.2 us
// with one warp doing all of it and 64-bit divisions for the slots, now 6.5;
// a batch of 27 systems of 189 to 812 bodies: 11.6 us with one thread per body,
// now 6.7).
template <int S, class Sum, class Scale>
__device__ __forceinline__ void integrate64(int i, Sum sum, Scale scale, const double4 *pos_old, double4 *pos_new,
                                            double4 *vel, double damping, double dt, int kick, double G,
                                            double4 *acc_out)
{
    __shared__ double red[4][S][32];
    const int lane = threadIdx.x & 31, q = threadIdx.x >> 5;
    const bool want_w = acc_out != nullptr;
    // what the warp's component q needs after the sums
    const size_t e = 4 * (size_t)(i < 0 ? 0 : i) + q;
    double xo = 0.0, m = 0.0, v = 0.0;
    if (q < 4 && i >= 0 && !acc_out) {
        xo = reinterpret_cast<const double *>(pos_old)[e];
        m = pos_old[i].w;
        if (q < 3) v = reinterpret_cast<const double *>(vel)[e];
    }
    double ax = 0.0, ay = 0.0, az = 0.0, aw = 0.0;
    if (i >= 0)
        sum(q, [&](const double4 &p) {
            ax = __dadd_rn(ax, p.x);
            ay = __dadd_rn(ay, p.y);
            az = __dadd_rn(az, p.z);
            if (want_w) aw = __dadd_rn(aw, p.w);
        });
    red[0][q][lane] = ax;
    red[1][q][lane] = ay;
    red[2][q][lane] = az;
    red[3][q][lane] = aw;
    __syncthreads();
    // warp q goes on with component q of the 32 bodies: x, y, z, and w (the
    // potential, or what the step carries along)
    if (q > 3 || i < 0) return;
    double a = red[q][0][lane];
#pragma unroll
    for (int k = 1; k < S; ++k) a = __dadd_rn(a, red[q][k][lane]);
    a = scale(q, a);
    if (acc_out) {
        reinterpret_cast<double *>(acc_out)[e] = a;
        return;
    }
    if (q < 3) {
        const double k = kick == NB_KICK_REFERENCE ? m : G;
        v = __dadd_rn(v, __dmul_rn(__dmul_rn(a, k), dt));
        v = __dmul_rn(v, damping);
        reinterpret_cast<double *>(vel)[e] = v;
        xo = __dadd_rn(xo, __dmul_rn(v, dt));
    }
    reinterpret_cast<double *>(pos_new)[e] = xo;  // component 3: the mass
}

}  // namespace nb
