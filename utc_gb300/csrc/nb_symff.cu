// nb_symff.cu -- FP64-accurate symmetric step in float-float arithmetic
// (NB_F64 with NB_ALGO_SYM).
//
// The app's default state type is double (benchapps/nbody/utc/nbody_main.cc
// FTYPE), and the reference evaluates every ordered pair in FP64
// (benchapps/nbody/cuda/bodysystem_kernel.cu:21-56).  On GB300 the FP64 pipe
// runs at about 1/76 of the FP32 rate (measured: 1.06 TFLOP/s DFMA against
// 78.5 TFLOP/s FFMA), so the FP64 symmetric kernel (nb_sym64.cu) is held to
// some 45 G interactions/s however it is arranged.  This kernel gets FP64
// accuracy from the FP32 pipe instead, with the standard float-float
// (double-single) techniques:
//  * error-free sums: Knuth's two-sum (s + e == a + b exactly) and Dekker's
//    fast two-sum for |a| >= |b|;
//  * error-free products from the FMA: p = a*b, e = fma(a, b, -p);
//  * float-float numbers hi + lo with |lo| <= ulp(hi)/2, about 48 bits.
// Per step, positions and masses are scaled by exact powers of two (the
// largest coordinate and the largest mass into [1/2, 1), found by a
// reduction on the device); each scaled coordinate is split on fixed grids
// into three floats, h (2^-20), m (2^-44) and l (2^-68), h + m + l == x
// exactly for |x| >= 2^-16 and to 2^-69 below that (the mass into a
// float-float).  Per unordered pair (the symmetric layout of nb_sym.cu: row
// blocks of 32*BPT targets per warp x 32-body chunks, the chunk rotating
// through the warp with its reaction):
//  * r = x_j - x_i: the three grid differences are exact; two fast
//    two-sums normalize them to a float-float, to 2^-47 relative and
//    exactly for close pairs -- also far from the origin, where a two-float
//    split of the positions would lose the bits below 2^-49 |x|;
//  * d2 = |r|^2 + eps2 in float-float;
//  * 1/sqrt(d2): the FP32 approximation refined by one FP32 Newton step
//    (to ~2^-24) and one Halley step in float-float, y = y0 (1 + t/2 +
//    3t^2/8) with t = 1 - d2 y0^2 formed from an error-free y0^2 (cubic
//    convergence; the small t keeps the correction's roundings near 2^-47);
//  * inv^3, the weights m_j inv^3 and m_i inv^3, and the six products with
//    r in float-float; target and reaction sums in float-float, renormalized
//    every second and fourth step (nb_ff.cuh).
// Each target's 32-source chunk sum is folded into FP64 accumulators; each
// reaction (one chunk body, the warp's 32*BPT targets) is written as FP64.
// The FP64 integrator of nb_sym64.cu then sums the partials in FP64, undoes
// the scaling and integrates.  The default shape, one warp x 2 targets
// (row blocks of 64 bodies: a triangular array of N^2 / 4 bytes), is kept at
// every size: past N = 185k the array is cut into bands of at most 8 GiB as
// in nb_sym.cu (symff_fold_kernel folds each band in FP64), which ran 9-22 %
// faster on GB300 than growing the row block (scalar pair loop: 315 against
// 288 and 259 G interactions/s at N = 2^19 and 2^20).  185 FP32 operations and
// one approximation per pair, two pairs per f32x2 instruction (nb_ff.cuh): the
// FMA pipe is 81 % busy, issue slots half used; what is left are the third
// operands of some 35 FMAs per pair (register reads, as in nb_pair.cuh).
// N = 16384: 328 G interactions/s (force and split) against 311 for the scalar
// loop; N = 65536: 349 against 326; 16 systems x 4096 in a batch: 311 against
// 272.  Results within a few 1e-15 of the FP64
// oracle (FP64 arithmetic: a few 1e-16), not bit-identical (NB_ALGO_EXACT is).
// Range: the scaled squared distances and eps2 must stay normal floats:
// eps2 >= 2^-100 max|x|^2 and body masses >= 2^-100 of the largest.
#include "nb_ff.cuh"

namespace nb {


// range[0] = bits of max |coordinate|, range[1] = bits of max |mass| (non-
// negative doubles order like their bit patterns); range zeroed beforehand.
__global__ void ff_range_kernel(const double4 *__restrict__ pos, int n, unsigned long long *__restrict__ range)
{
    unsigned long long mc = 0, mm = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double4 q = pos[i];
        const double c = fmax(fabs(q.x), fmax(fabs(q.y), fabs(q.z)));
        const unsigned long long bc = (unsigned long long)__double_as_longlong(c);
        const unsigned long long bm = (unsigned long long)__double_as_longlong(fabs(q.w));
        mc = bc > mc ? bc : mc;
        mm = bm > mm ? bm : mm;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long a = __shfl_xor_sync(0xffffffffu, mc, o);
        const unsigned long long b = __shfl_xor_sync(0xffffffffu, mm, o);
        mc = a > mc ? a : mc;
        mm = b > mm ? b : mm;
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&range[0], mc);
        atomicMax(&range[1], mm);
    }
}

// Scaled split of one body: coordinates x * 2^kx (below 1 in magnitude) on the
// grids H: 2^-20, M: 2^-44, L: 2^-68 (H + M + L == x * 2^kx exactly when
// |x * 2^kx| >= 2^-16, otherwise to 2^-69); the mass m * 2^km as the
// float-float H + M (L unused).  ex = -kx, em = -km; a sum with 1.5 * 2^(52 - g) leaves v rounded to the grid 2^-g.
__device__ __forceinline__ void ff_split_body(const double4 &q, int ex, int em, float4 *H, float4 *M, float4 *L)
{
    auto grid = [](double v, double c) { return __dsub_rn(__dadd_rn(v, c), c); };
    const double v[4] = {mul_pow2(q.x, -ex), mul_pow2(q.y, -ex), mul_pow2(q.z, -ex), mul_pow2(q.w, -em)};
    float h[4], m[4], l[4];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double gh = grid(v[k], 0x1.8p32);   // |gh| <= 1: 21 bits
        const double r1 = v[k] - gh;              // exact, |r1| <= 2^-21
        const double gm = grid(r1, 0x1.8p8);      // 24 bits
        const double r2 = r1 - gm;                // exact, |r2| <= 2^-45
        h[k] = (float)gh;
        m[k] = (float)gm;
        l[k] = (float)grid(r2, 0x1.8p-16);        // 24 bits
    }
    h[3] = __double2float_rn(v[3]);
    m[3] = __double2float_rn(v[3] - (double)h[3]);
    l[3] = 0.f;
    *H = make_float4(h[0], h[1], h[2], h[3]);
    *M = make_float4(m[0], m[1], m[2], m[3]);
    *L = make_float4(l[0], l[1], l[2], l[3]);
}

// Latency bounds these two (some 40 dependent operations of the narrow FP64
// pipe a body): small blocks, so that a small system spreads over many SMs.
// With ldexp and rint in place of the products and sums, in blocks of 256, the
// split took 10.8 us at N = 1000 to 8192; now 4.1 to 4.7.
constexpr int kFFSplitBlock = 64;

__global__ void __launch_bounds__(kFFSplitBlock) ff_split_kernel(const double4 *pos, int n,
                                                                 const unsigned long long *range,
                                                                 float4 *H, float4 *M,
                                                                 float4 *L)
{
    pdl_wait();
    const int i = blockIdx.x * kFFSplitBlock + threadIdx.x;
    if (i >= n) return;
    ff_split_body(pos[i], ff_exponent(range[0]), ff_exponent(range[1]), H + i, M + i, L + i);
}

// Range and split in one launch for small systems: every block finds the
// largest coordinate and mass of all bodies for itself (only their exponents
// are used, so the upper words do), instead of a memset and a reduction of
// their own.  The redundant pass over the bodies costs 0.6 us per 1000 of them
// against 3 us and two launches: 4.8 us at N = 1000, 6.7 at N = 4096, 10.1
// at N = 8192, where the three launches take 3.0 + 4.1 us and the gaps between.
constexpr int kFFFusedBlock = 256;

__global__ void __launch_bounds__(kFFFusedBlock) ff_range_split_kernel(const double4 *pos, int n, unsigned long long *range,
                                                                       float4 *H, float4 *M, float4 *L)
{
    __shared__ unsigned red[2][kFFFusedBlock / 32];
    const int i = blockIdx.x * kFFSplitBlock + threadIdx.x;
    const bool own = threadIdx.x < kFFSplitBlock && i < n;
    pdl_wait();
    const double4 mine = own ? pos[i] : make_double4(0.0, 0.0, 0.0, 0.0);
    auto top = [](double v) { return (unsigned)__double2hiint(v) & 0x7fffffffu; };
    unsigned mc = 0, mm = 0;
    for (int j = threadIdx.x; j < n; j += 8 * kFFFusedBlock) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const double4 q = pos[min(j + k * kFFFusedBlock, n - 1)];  // the last body again past the end
            mc = max(mc, max(top(q.x), max(top(q.y), top(q.z))));
            mm = max(mm, top(q.w));
        }
    }
    mc = __reduce_max_sync(0xffffffffu, mc);
    mm = __reduce_max_sync(0xffffffffu, mm);
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = mc;
        red[1][threadIdx.x >> 5] = mm;
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kFFFusedBlock / 32; ++w) {
        mc = max(mc, red[0][w]);
        mm = max(mm, red[1][w]);
    }
    const unsigned long long rc = (unsigned long long)mc << 32, rm = (unsigned long long)mm << 32;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        range[0] = rc;
        range[1] = rm;
    }
    if (own) ff_split_body(mine, ff_exponent(rc), ff_exponent(rm), H + i, M + i, L + i);
}

// One CTA's share of a row: row block I's targets against the chunks
// [kc0, kc1), target-side sums to dst, reactions to spart.  Not inlined into
// the loop over rows, as sym_row_segment of nb_sym.cu.
// PHI: also the potential sum_j m_j inv (j != i) in the partials' w, the
// reaction's included (energy pass).
template <int W, int BPT, bool PHI>
__device__ __noinline__ void symff_row_segment(const float4 *H, const float4 *Mi,
                                               const float4 *Lo, int n, float eps_h, float eps_l,
                                               double4 *dst, double4 *spart, long long soff, int I, int kc0, int kc1)
{
    constexpr int NP = BPT / 2;
    constexpr int WB = 32 * BPT;
    constexpr int RB = W * WB;
    constexpr int RC = RB / 32;
    __shared__ __align__(16) float4 sH[32], sM[32], sL[32];
    __shared__ double sF[4][W][32];
    const int lane = threadIdx.x & 31;
    const int wid = threadIdx.x >> 5;
    const int tbase = I * RB + wid * WB;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const f2 eh = ff_pack1(eps_h), el = ff_pack1(eps_l);

    FFTargets<NP, PHI> T;
    T.load(H, Mi, Lo, [&](int k) {
        const int i = tbase + lane + 32 * k;
        return i < n ? i : -1;
    });
    double ax[BPT], ay[BPT], az[BPT], aphi[BPT];
#pragma unroll
    for (int k = 0; k < BPT; ++k) ax[k] = ay[k] = az[k] = aphi[k] = 0.0;
#pragma unroll 1
    for (int kc = kc0; kc < kc1; ++kc) {
        const int jb = kc * 32;
        const bool in = jb + lane < n;
        __syncthreads();  // previous chunk: shared reads are done
        if (wid == 0) {
            // padding: far away (scaled coordinates are below 1), no mass
            sH[lane] = in ? H[jb + lane] : make_float4(1.0e6f, 1.0e6f, 1.0e6f, 0.f);
            sM[lane] = in ? Mi[jb + lane] : zero;
            sL[lane] = in ? Lo[jb + lane] : zero;
        }
        __syncthreads();
        T.clear();
        if (kc < (I + 1) * RC) {
            // chunk inside the own row block: directed, target side only
            ff_chunk_pull(T, sH, sM, sL, eh, el, [&](int k) { return tbase + lane + 32 * k - jb; });
        } else {
            FFReact F;
            ff_chunk_react(T, F, sH, sM, sL, lane, eh, el);
            // the reaction on chunk body `lane` from this warp
            double fx = F.x.fold(), fy = F.y.fold(), fz = F.z.fold(), fp = PHI ? F.p.fold() : 0.0;
            if constexpr (W > 1) {
                sF[0][wid][lane] = fx;
                sF[1][wid][lane] = fy;
                sF[2][wid][lane] = fz;
                sF[3][wid][lane] = fp;
                __syncthreads();
                fx = fy = fz = fp = 0.0;
                if (wid == 0) {
#pragma unroll
                    for (int w = 0; w < W; ++w) {
                        fx += sF[0][w][lane];
                        fy += sF[1][w][lane];
                        fz += sF[2][w][lane];
                        fp += sF[3][w][lane];
                    }
                }
            }
            if (wid == 0 && in) spart[soff + (jb + lane - (I + 1) * RB)] = make_double4(fx, fy, fz, fp);
        }
        // fold the chunk's sums into FP64
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            double lo, hi;
            T.ax[p].get(lo, hi);
            ax[2 * p] += lo;
            ax[2 * p + 1] += hi;
            T.ay[p].get(lo, hi);
            ay[2 * p] += lo;
            ay[2 * p + 1] += hi;
            T.az[p].get(lo, hi);
            az[2 * p] += lo;
            az[2 * p + 1] += hi;
            if (PHI) {
                T.ap[p].get(lo, hi);
                aphi[2 * p] += lo;
                aphi[2 * p + 1] += hi;
            }
        }
    }
    dst += wid * WB + lane;
#pragma unroll
    for (int k = 0; k < BPT; ++k) dst[32 * k] = make_double4(ax[k], ay[k], az[k], aphi[k]);
}

// BAND: one band of a banded plan, as in sym_force_kernel: items
// [it0, it0 + total) from row block r0 on, target-side slot c + I - r0,
// source-side entries offset by soff0.
template <int W, int BPT, int MINB, bool PHI, bool BAND = false>
__global__ void __launch_bounds__(32 * W, MINB)
    symff_force_kernel(const float4 *H, const float4 *Mi, const float4 *Lo,
                       int n, double eps2, const unsigned long long *range,
                       double4 *tpart, double4 *spart, long long total, int nc, int nrb,
                       long long it0, int r0, long long soff0)
{
    pdl_wait();
    constexpr int RB = W * 32 * BPT;
    constexpr int RC = RB / 32;
    const int c = blockIdx.x;
    // eps2 in the scaled units (x 2^(2 kx)), as a float-float
    const double e2s = mul_pow2(eps2, -2 * ff_exponent(range[0]));
    const float eh = __double2float_rn(e2s), el = __double2float_rn(e2s - (double)eh);
    long long it = sk_start(c, total, gridDim.x);
    long long end = sk_start(c + 1, total, gridDim.x);
    if constexpr (BAND) {
        it += it0;
        end += it0;
    }
    while (it < end) {
        const int I = sym_row_of(it, nc, RC, nrb);
        const long long rfirst = sym_prefix(I, nc, RC);
        const long long rend = sym_prefix(I + 1, nc, RC);
        const long long seg_end = end < rend ? end : rend;
        symff_row_segment<W, BPT, PHI>(H, Mi, Lo, n, eh, el, tpart + (size_t)(c + I - (BAND ? r0 : 0)) * RB, spart,
                                       sym_soff(I, n, RB) - (BAND ? soff0 : 0), I, I * RC + (int)(it - rfirst),
                                       I * RC + (int)(seg_end - rfirst));
        it = seg_end;
    }
}

typedef void (*symff_kernel_t)(const float4 *, const float4 *, const float4 *, int, double,
                               const unsigned long long *, double4 *, double4 *, long long, int, int, long long,
                               int, long long);

static symff_kernel_t symff_kernel_for(int w, int bpt, bool phi = false, bool band = false)
{
    if (band) {  // banded plans: the one-warp shapes
        if (w == 1 && bpt == 2)
            return phi ? symff_force_kernel<1, 2, 16, true, true> : symff_force_kernel<1, 2, 16, false, true>;
        if (w == 1 && bpt == 4)
            return phi ? symff_force_kernel<1, 4, 8, true, true> : symff_force_kernel<1, 4, 8, false, true>;
        return nullptr;
    }
    if (w == 1 && bpt == 2) return phi ? symff_force_kernel<1, 2, 16, true> : symff_force_kernel<1, 2, 16, false>;
    if (w == 1 && bpt == 4) return phi ? symff_force_kernel<1, 4, 8, true> : symff_force_kernel<1, 4, 8, false>;
    if (w == 4 && bpt == 4) return phi ? symff_force_kernel<4, 4, 2, true> : symff_force_kernel<4, 4, 2, false>;
    if (w == 8 && bpt == 4) return phi ? symff_force_kernel<8, 4, 1, true> : symff_force_kernel<8, 4, 1, false>;
    if (w == 8 && bpt == 8) return phi ? symff_force_kernel<8, 8, 1, true> : symff_force_kernel<8, 8, 1, false>;
    return nullptr;
}

int symff_plan(int n, int warps, int bpt, int device, SymPlan *pl, int bands)
{
    const bool given = warps != 0 || bpt != 0;
    if (!given) {
        // one-warp CTAs x 2 targets (row block 64), its source-side array
        // (32 B entries) in bands where it would pass the budget; without
        // bands 1 x 4 (128), 4 x 4 (512), 8 x 4 (1024), 8 x 8 (2048) take
        // over instead
        static const int shapes[5][2] = {{1, 2}, {1, 4}, {4, 4}, {8, 4}, {8, 8}};
        int s = 0;
        if (bands < 0)
            while (s < 4 && sym_spart_entries(n, shapes[s][0] * 32 * shapes[s][1]) * (long long)sizeof(double4) >
                                kSymSpartBudget)
                ++s;
        warps = shapes[s][0];
        bpt = shapes[s][1];
    }
    SymPlan p;
    p.n = n;
    p.warps = warps;
    p.bpt = bpt;
    p.rb = warps * 32 * bpt;
    p.nc = (n + 31) / 32;
    p.nrb = (n + p.rb - 1) / p.rb;
    p.spart_size = sym_spart_entries(n, p.rb);
    p.band_row[0] = 0;
    p.band_row[1] = p.nrb;
    if (bands >= 0 && n > 0 &&
        (bands > 1 || p.spart_size * (long long)sizeof(double4) > kSymSpartBudget)) {
        long long mx = 0;
        const int k = sym_make_bands(n, p.rb, kSymSpartBudget / (long long)sizeof(double4), bands > 1 ? bands : 0,
                                     p.band_row, &mx);
        if (k == 0)
            return set_error(NB_ERR_UNSUPPORTED, "the float-float source side would need more than 512 bands");
        p.nbands = k;
        p.spart_size = mx;
    }
    const bool band = p.nbands > 1;
    symff_kernel_t k = symff_kernel_for(warps, bpt, false, band);
    if (!k)
        return set_error(NB_ERR_UNSUPPORTED, band ? "float-float symmetric kernel shape not compiled for bands "
                                                    "(one warp x 2 or 4 targets)"
                                                  : "float-float symmetric kernel shape not compiled");
    p.total = n > 0 ? sym_prefix(p.nrb, p.nc, p.rb / 32) : 0;
    int sms = 0, occ = 0;
    NB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    NB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, 32 * warps, 0));
    int occ_phi = 0;  // the energy pass runs on the same plan
    NB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_phi, symff_kernel_for(warps, bpt, true, band),
                                                          32 * warps, 0));
    if (occ_phi < occ) occ = occ_phi;
    if (occ < 1) return set_error(NB_ERR_UNSUPPORTED, "float-float symmetric kernel does not fit on an SM");
    long long grid = (long long)sms * occ;
    if (p.total > 0 && grid > p.total) grid = p.total;
    p.grid = p.total > 0 ? (int)grid : 0;
    p.slots = p.total > 0 ? p.grid + p.nrb - 1 : 0;
    p.sms = sms;
    p.small = p.nbands == 1 && bands <= 1 && n > 0 && n <= kFFSmallBodies && warps == 1 && bpt == 2;
    *pl = p;
    return NB_OK;
}

// After band [r0, r1) of a banded plan: the running per-body sums (x, y, z
// and the potential in w), as sym_fold_kernel does for float partials.
__global__ void __launch_bounds__(256) symff_fold_kernel(const double4 *__restrict__ tpart,
                                                         const double4 *__restrict__ spart,
                                                         double4 *__restrict__ accsum, int n, int rb, int nc,
                                                         long long it0, long long bt, int gb, int r0, int r1,
                                                         long long soff0, int first)
{
    const int i = n - 1 - (int)(blockIdx.x * blockDim.x + threadIdx.x);  // longest walks first
    if (i < 0) return;
    const int I = i / rb;
    if (I < r0) return;  // rows before the band get nothing from it (r0 = 0 for the first band)
    double4 a = first ? make_double4(0.0, 0.0, 0.0, 0.0) : accsum[i];
    if (I < r1) {
        const int rc = rb / 32;
        const int c0 = sk_owner(sym_prefix(I, nc, rc) - it0, bt, gb);
        const int c1 = sk_owner(sym_prefix(I + 1, nc, rc) - 1 - it0, bt, gb);
        const int li = i - I * rb;
        for (int c = c0; c <= c1; ++c) {
            const double4 q = tpart[(size_t)(c + I - r0) * rb + li];
            a.x = __dadd_rn(a.x, q.x);
            a.y = __dadd_rn(a.y, q.y);
            a.z = __dadd_rn(a.z, q.z);
            a.w = __dadd_rn(a.w, q.w);
        }
    }
    const int rend = I < r1 ? I : r1;
#pragma unroll 4
    for (int r = r0; r < rend; ++r) {
        const double4 q = spart[sym_soff(r, n, rb) - soff0 + (i - (long long)(r + 1) * rb)];
        a.x = __dadd_rn(a.x, q.x);
        a.y = __dadd_rn(a.y, q.y);
        a.z = __dadd_rn(a.z, q.z);
        a.w = __dadd_rn(a.w, q.w);
    }
    accsum[i] = a;
}

int ff_scale_split(const double4 *pos, int n, int sms, float4 *H, float4 *M, float4 *L, unsigned long long *range,
                   cudaStream_t s)
{
    if (n == 0) return NB_OK;
    if (n <= kFFFusedBodies)
        return pdl_launch("ff_range_split_kernel launch", ff_range_split_kernel,
                          (unsigned)((n + kFFSplitBlock - 1) / kFFSplitBlock), kFFFusedBlock, s, pos, n, range, H, M, L);
    NB_CUDA(cudaMemsetAsync(range, 0, 2 * sizeof(unsigned long long), s));
    const long long want = (n + 255) / 256, cap = 4ll * (sms > 0 ? sms : 1);
    const long long blocks = want < cap ? want : cap;
    ff_range_kernel<<<(unsigned)blocks, 256, 0, s>>>(pos, n, range);
    NB_LAUNCH_CHECK("ff_range_kernel launch");
    return pdl_launch("ff_split_kernel launch", ff_split_kernel, (unsigned)((n + kFFSplitBlock - 1) / kFFSplitBlock),
                      kFFSplitBlock, s, pos, n, range, H, M, L);
}

// ---------------------------------------------------------------------------
// Small systems: the preparation, then the rest of the step in one launch (the
// layout of nb_small.cu).  A CTA owns two bodies (a pair of the f32x2
// arithmetic), its 128 threads split the sources, every pair is evaluated from
// the target's side (140 operations, 1.5 times the work of the symmetric kernel
// a pair of bodies, but no partial leaves the CTA and no item of 64 x 32 pairs
// has to be found for every warp); the sums are reduced through the warps in
// float-float and across them in FP64.
//
// Step time from a replayed graph, GB300, us, against the symmetric kernels:
// N = 300 5.9 (17.4), 1000 11.8 (19.8), 1500 16.8 (20.8), 2000 25.8 (28.1),
// 2300 31.9 (35.6), 2500 37.7 (36.4), 3000 47.5 (44.2): the line is at 2400.
// Bounds: the chain preparation (3 us) - first loads - reduction while small,
// then the FMA pipe and whole CTAs per SM (1000 bodies: 3.3 CTAs an SM on
// average, 4 on most).  4 bodies a CTA: within 6 % either way; 256 threads: 4
// to 15 % slower.
constexpr int kFFSmallThreads = 128;
constexpr int kFFSmallTargets = 2;

__device__ __forceinline__ void ff_add1(float &h, float &l, float gh, float gl)
{
    float s, e;
    two_sum(h, gh, s, e);
    const float t = __fadd_rn(__fadd_rn(l, gl), e);
    h = __fadd_rn(s, t);
    l = __fsub_rn(t, __fsub_rn(h, s));
}

// Sums (h, l)[0..3 T) over the warp as warp_sum of nb_pair.cuh does: the lanes
// halve the targets while there is more than one, and the lane's target is
// returned.
template <int T>
__device__ __forceinline__ int ff_warp_sum(float *h, float *l, int lane)
{
    int mine = 0, off = 16;
#pragma unroll
    for (int half = T / 2; half >= 1; half /= 2) {
        const bool up = (lane & off) != 0;
        mine = 2 * mine + (up ? 1 : 0);
#pragma unroll
        for (int k = 0; k < 3 * half; ++k) {
            const int o = 3 * half + k;
            const float gh = up ? h[k] : h[o], gl = up ? l[k] : l[o];
            h[k] = up ? h[o] : h[k];
            l[k] = up ? l[o] : l[k];
            ff_add1(h[k], l[k], __shfl_xor_sync(0xffffffffu, gh, off), __shfl_xor_sync(0xffffffffu, gl, off));
        }
        off /= 2;
    }
#pragma unroll
    for (; off >= 1; off /= 2) {
#pragma unroll
        for (int k = 0; k < 3; ++k)
            ff_add1(h[k], l[k], __shfl_xor_sync(0xffffffffu, h[k], off), __shfl_xor_sync(0xffffffffu, l[k], off));
    }
    return mine;
}

template <int TB>
__global__ void __launch_bounds__(kFFSmallThreads, 8 / TB)
    symff_small_kernel(const float4 *H, const float4 *M, const float4 *L, const unsigned long long *range,
                       const double *pos_old, double *pos_new, double *vel, int n, double eps2, double damping,
                       double dt, int kick, double G, double *acc_out)
{
    constexpr int NP = TB / 2, NW = kFFSmallThreads / 32;
    __shared__ double red[NW][3 * TB];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int t0 = blockIdx.x * TB;
    // the component that this thread integrates
    const int body = t0 + (tid >> 2), q = tid & 3;
    const bool own = tid < 4 * TB && body < n;
    const size_t e = 4 * (size_t)body + q;
    pdl_wait();
    const int ex = ff_exponent(range[0]), em = ff_exponent(range[1]);
    double x = 0.0, m = 0.0, v = 0.0;
    if (own && pos_new) {
        x = pos_old[e];
        m = pos_old[e - q + 3];
        if (q < 3) v = vel[e];
    }
    const double e2s = mul_pow2(eps2, -2 * ex);
    const float eh = __double2float_rn(e2s), el = __double2float_rn(e2s - (double)eh);
    const f2 EH = ff_pack1(eh), EL = ff_pack1(el);
    FFTargets<NP, false> T;
    T.load(H, M, L, [&](int k) { return t0 + k < n ? t0 + k : -1; });
    T.clear();
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 h = zero, mi = zero, lo = zero;
    if (tid < n) {
        h = H[tid];
        mi = M[tid];
        lo = L[tid];
    }
    bool odd = false;
#pragma unroll 2
    for (int j = tid; j < n; j += kFFSmallThreads) {
        FFSource s;
        s.load(h, mi, lo);
        const int jn = j + kFFSmallThreads;
        if (jn < n) {
            h = H[jn];
            mi = M[jn];
            lo = L[jn];
        }
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            FFPair w;
            ff_pair<false>(s, T.t[p], EH, EL, w);
            T.pull(p, w);
        }
        if (odd) T.norm();
        odd = !odd;
    }
    T.norm();
    float sh[3 * TB], sl[3 * TB];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        f2_unpack(T.ax[p].h, sh[6 * p], sh[6 * p + 3]);
        f2_unpack(T.ax[p].l, sl[6 * p], sl[6 * p + 3]);
        f2_unpack(T.ay[p].h, sh[6 * p + 1], sh[6 * p + 4]);
        f2_unpack(T.ay[p].l, sl[6 * p + 1], sl[6 * p + 4]);
        f2_unpack(T.az[p].h, sh[6 * p + 2], sh[6 * p + 5]);
        f2_unpack(T.az[p].l, sl[6 * p + 2], sl[6 * p + 5]);
    }
    const int t = ff_warp_sum<TB>(sh, sl, lane);
    if ((lane & (32 / TB - 1)) == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) red[wid][3 * t + k] = (double)sh[k] + (double)sl[k];
    }
    __syncthreads();
    if (!own) return;
    double a = 0.0;
    if (q < 3) {
        a = red[0][3 * (tid >> 2) + q];
#pragma unroll
        for (int w = 1; w < NW; ++w) a = __dadd_rn(a, red[w][3 * (tid >> 2) + q]);
        a = mul_pow2(a, em - 2 * ex);
    }
    if (acc_out) acc_out[e] = a;
    if (!pos_new) return;
    if (q < 3) {
        const double k = kick == NB_KICK_REFERENCE ? m : G;
        v = __dadd_rn(v, __dmul_rn(__dmul_rn(a, k), dt));
        v = __dmul_rn(v, damping);
        vel[e] = v;
        x = __dadd_rn(x, __dmul_rn(v, dt));
    }
    pos_new[e] = x;
}

int symff_small_step(const SymPlan &p, const double4 *pos_old, double4 *pos_new, double4 *vel, double eps2,
                     double damping, double dt, int kick, double G, double4 *acc_out, float4 *split,
                     unsigned long long *range, cudaStream_t s)
{
    if (p.n == 0) return NB_OK;
    float4 *H = split, *M = split + p.n, *L = split + 2 * (size_t)p.n;
    if (int st = ff_scale_split(pos_old, p.n, p.sms, H, M, L, range, s)) return st;
    return pdl_launch("symff_small_kernel launch", symff_small_kernel<kFFSmallTargets>,
                      (unsigned)((p.n + kFFSmallTargets - 1) / kFFSmallTargets), kFFSmallThreads, s, H, M, L, range,
                      (const double *)pos_old, (double *)pos_new, (double *)vel, p.n, eps2, damping, dt, kick, G,
                      (double *)acc_out);
}

int symff_force(const SymPlan &p, const double4 *pos, double eps2, float4 *split, unsigned long long *range,
                double4 *tpart, double4 *spart, double4 *accsum, cudaStream_t s, int phi)
{
    if (p.n == 0) return NB_OK;
    symff_kernel_t k = symff_kernel_for(p.warps, p.bpt, phi != 0, p.nbands > 1);
    if (!k) return set_error(NB_ERR_UNSUPPORTED, "float-float symmetric kernel shape not compiled");
    if (p.nbands > 1 && !accsum) return set_error(NB_ERR_INVALID, "symff_force: a banded plan needs its per-body sums");
    float4 *H = split, *M = split + p.n, *L = split + 2 * (size_t)p.n;
    int st = ff_scale_split(pos, p.n, p.sms, H, M, L, range, s);
    if (st) return st;
    if (p.nbands <= 1) {
        return pdl_launch("symff_force_kernel launch", k, p.grid, 32 * p.warps, s, H, M, L, p.n, eps2, range, tpart,
                          spart, p.total, p.nc, p.nrb, 0, 0, 0);
    }
    const int rc = p.rb / 32;
    for (int b = 0; b < p.nbands; ++b) {
        const int r0 = p.band_row[b], r1 = p.band_row[b + 1];
        const long long it0 = sym_prefix(r0, p.nc, rc), bt = sym_prefix(r1, p.nc, rc) - it0;
        const long long soff0 = sym_soff(r0, p.n, p.rb);
        const int gb = (int)(bt < p.grid ? bt : p.grid);
        k<<<gb, 32 * p.warps, 0, s>>>(H, M, L, p.n, eps2, range, tpart, spart, bt, p.nc, p.nrb, it0, r0, soff0);
        NB_LAUNCH_CHECK("symff_force_kernel launch");
        symff_fold_kernel<<<(p.n + 255) / 256, 256, 0, s>>>(tpart, spart, accsum, p.n, p.rb, p.nc, it0, bt, gb, r0,
                                                            r1, soff0, b == 0);
        NB_LAUNCH_CHECK("symff_fold_kernel launch");
    }
    return NB_OK;
}

}  // namespace nb
