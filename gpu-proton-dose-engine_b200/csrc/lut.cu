// lut.cu -- FP64 depth-LUT builder on the device.
//
// Builds, for every energy layer, the integral depth dose IDD_l(z) (physics.py:328-387,
// normalize=False) and the lateral width sigma_l(z) (physics.py:221-286) at the dose
// grid's depths, plus their central differences in CSDA range for the range-shift
// gradient.  This file is compiled with -fmad=false: products and sums are rounded one
// at a time, in the order the reference's NumPy expressions evaluate them, so the
// tables agree with the reference to the last few ulps of the transcendental functions.
//
// Two steps are restated in a different but equivalent form:
//  * CSDA range table cumulative sum: one thread, sequential, as numpy.cumsum.
//  * Range-straggling convolution.  The reference multiplies the zero-padded rfft of
//    the binned dose (nfft = 16384 >= 2 n_fine) by exp(-2 (pi f sigma_R)^2).  By the
//    Poisson summation formula, irfft of that Gaussian spectrum is h * phi_sigma(k h)
//    summed over periods of nfft*h; all other periods and all frequencies past Nyquist
//    are below 1e-300 for any sigma_R >= 2 h, and the zero padding makes the circular
//    convolution linear.  The device therefore computes the linear convolution
//    smooth[n] = sum_m binned[m] * h * phi(|n-m| h) directly in FP64, truncated at
//    16 sigma_R (kernel weight < 1e-55).  The two agree to FFT round-off (~1e-16 of
//    the peak).
#include <math.h>
#include <stdio.h>

#include <algorithm>

#include "pbd_internal.cuh"
#include "tc_common.cuh"

namespace pbd {
namespace {

// physics.py:42-66
constexpr double kMp = 938.27208816;
constexpr double kMe = 0.51099895000;
constexpr double kKbb = 0.307075;
constexpr double kZA = 10.0 / 18.01528;
constexpr double kI = 75.0 * 1e-6;
constexpr double kRho = 1.0;
constexpr double kX0 = 36.08;
constexpr double kPowerP = 1.77;
constexpr double kHighland = 13.6;
constexpr double kElo = 0.5;
constexpr double kEhi = 400.0;
constexpr double kBohr = kKbb * kZA * kRho * kMe;   // physics.py:151
constexpr int kTableN = 3797;                        // 800 + 899 + 899 + 1199 points
constexpr int kBohrN = 4000;                         // physics.py:154

__device__ double g_etab[kTableN];
__device__ double g_rtab[kTableN];

// numpy.linspace(a, b, n)[k]: k*step + a, the last point set to b exactly.
__device__ __forceinline__ double lin(double a, double b, int n, int k) {
    if (k == n - 1) return b;
    double step = (b - a) / (double)(n - 1);
    return (double)k * step + a;
}

// Energy grid of the range table (physics.py:118-123): four linspace pieces with the
// shared end points 2, 20 and 60 MeV kept once.
__device__ double table_energy(int k) {
    if (k < 800) return lin(kElo, 2.0, 800, k);
    if (k < 1699) return lin(2.0, 20.0, 900, k - 799);
    if (k < 2598) return lin(20.0, 60.0, 900, k - 1698);
    return lin(60.0, kEhi, 1200, k - 2597);
}

// beta_gamma, physics.py:72-77
__device__ __forceinline__ void kinematics(double e, double& beta, double& gam, double& b2) {
    gam = 1.0 + e / kMp;
    b2 = 1.0 - 1.0 / (gam * gam);
    b2 = fmin(fmax(b2, 1e-14), 1.0);
    beta = sqrt(b2);
}

// bethe_bloch_water, physics.py:80-100
__device__ double stopping_power(double e) {
    double beta, gam, b2;
    kinematics(e, beta, gam, b2);
    const double me_mp = kMe / kMp;
    double g2 = gam * gam;
    double tmax = 2.0 * kMe * b2 * g2 / (1.0 + 2.0 * gam * me_mp + me_mp * me_mp);
    double arg = 2.0 * kMe * b2 * g2 * tmax / (kI * kI);
    arg = fmax(arg, 1.0 + 1e-12);
    return kKbb * kZA * kRho / b2 * (0.5 * log(arg) - b2);
}

// scattering_power(model="highland_local") at L = 1, physics.py:202-217
__device__ double highland_local(double e) {
    double beta, gam, b2;
    kinematics(e, beta, gam, b2);
    double pc = sqrt(fmax(gam * gam - 1.0, 0.0)) * kMp;
    double bpc = fmax(beta * pc, 1e-9);
    double q = kHighland / bpc;
    double base = q * q / kX0;
    const double lnl = 0.0;   // log(1)
    return base * (1.0 + 0.038 * lnl) * (1.076 + 0.038 * lnl);
}

// numpy.interp on a strictly increasing table.
__device__ double interp(double x, const double* xp, const double* fp, int n, double left,
                         double right) {
    if (x < xp[0]) return left;
    if (x > xp[n - 1]) return right;
    if (x == xp[n - 1]) return fp[n - 1];
    int lo = 0, hi = n - 1;
    while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (xp[mid] <= x) lo = mid; else hi = mid;
    }
    if (xp[lo] == x) return fp[lo];
    double slope = (fp[lo + 1] - fp[lo]) / (xp[lo + 1] - xp[lo]);
    return slope * (x - xp[lo]) + fp[lo];
}

// numpy.linspace(a, b, n)[k] with its step (b - a) / (n - 1) passed in: the same value as lin().
__device__ __forceinline__ double lin_s(double a, double b, int n, int k, double step) {
    if (k == n - 1) return b;
    return (double)k * step + a;
}

// The interval of x on linspace(a, b, n) that np.interp's search finds, for a <= x <= b:
// estimated from x * (1 / step) and corrected against the grid points themselves, whose values
// fk * step + a (fk = (double)lo kept in step with lo -- integers below 2^53, so fk +- 1 is
// exact) are those lin_s computes.  lo and its grid point x0 on return; x == b gives lo = n - 1,
// x0 = b.  step = (b - a) / (n - 1) and inv ~ 1 / step come from the caller.
__device__ __forceinline__ void locate_lin(double x, double a, double b, int n, double step,
                                           double inv, int& lo_out, double& x0_out) {
    if (x == b) {
        lo_out = n - 1;
        x0_out = b;
        return;
    }
    int lo = (int)((x - a) * inv);
    lo = lo < 0 ? 0 : (lo > n - 2 ? n - 2 : lo);
    double fk = (double)lo;
    double x0 = fk * step + a;
    while (lo > 0 && x0 > x) {
        --lo;
        fk -= 1.0;
        x0 = fk * step + a;
    }
    while (lo < n - 2) {
        const double x1 = lo + 1 == n - 1 ? b : (fk + 1.0) * step + a;
        if (!(x1 <= x)) break;
        ++lo;
        fk += 1.0;
        x0 = x1;
    }
    lo_out = lo;
    x0_out = x0;
}

__device__ __forceinline__ double csda(double e) {
    return interp(e, g_etab, g_rtab, kTableN, g_rtab[0], g_rtab[kTableN - 1]);
}
__device__ __forceinline__ double energy_at_range(double r) {
    double rc = fmin(fmax(r, 0.0), g_rtab[kTableN - 1]);
    return interp(rc, g_rtab, g_etab, kTableN, g_etab[0], g_etab[kTableN - 1]);
}

// _range_table, physics.py:111-127.  Trapezoid steps in parallel, cumulative sum in
// one thread in the order numpy.cumsum adds.
__global__ void range_table_kernel() {
    __shared__ double inv_s[kTableN];
    for (int k = threadIdx.x; k < kTableN; k += blockDim.x) {
        double e = table_energy(k);
        g_etab[k] = e;
        inv_s[k] = 1.0 / stopping_power(e);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double r = 0.0;
        g_rtab[0] = 0.0;
        double e_prev = g_etab[0];
        for (int k = 1; k < kTableN; ++k) {
            double e = g_etab[k];
            r = r + 0.5 * (inv_s[k] + inv_s[k - 1]) * (e - e_prev);
            g_rtab[k] = r;
            e_prev = e;
        }
    }
}

__global__ void csda_kernel(const double* in, double* out, int n, int inverse) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = inverse ? energy_at_range(in[i]) : csda(in[i]);
}

// Per (layer, variant) scalars.  Variant 0 is the nominal build, 1 and 2 are built at
// CSDA range +fd_step and -fd_step.
struct LayerScal {
    double e0, r0, sig_r, zmax, h;
    double step, inv;    // zmax / (n_idd - 1), the curve grid's step, and its reciprocal
    int conv_k;
    int last;            // last bin that can hold dose
};

struct LutDims {
    int n_layers, nvar, nz, n_idd, n_fe;
    double fe_lo, fe_hi;      // Fermi-Eyges fine grid end points
    double fe_step, fe_inv;   // its step and the step's reciprocal
    double fd_step;
};

// Scalars of one (layer, variant) per block: energy, range and sigma_R (physics.py:154-174,
// 310-322).  4000 stopping powers per block, FP64 log and divisions: a block of 512 threads
// keeps the FP64 pipe of its SM busy (with the fills below in the same 256-thread block, one
// block per (layer, variant), the set-up took 78 us for 120 of them; now 14 + 15 us).
constexpr int kScalThreads = 512;

__global__ void __launch_bounds__(kScalThreads)
layer_scal_kernel(pbd_lut_spec spec, LutDims dm, const double* energies, const double* shift,
                  LayerScal* scal) {
    __shared__ double f_bohr[kBohrN];
    __shared__ double red[kScalThreads];
    const int lv = blockIdx.x;
    const int l = lv / dm.nvar, v = lv % dm.nvar;
    const double off = v == 0 ? 0.0 : (v == 1 ? dm.fd_step : -dm.fd_step);
    const double s = (shift ? shift[l] : 0.0) + off;
    const double e_in = energies[l];
    const double e0 = (s == 0.0) ? e_in : energy_at_range(csda(e_in) + s);
    const double r0 = csda(e0);

    // range straggling
    double strag = 0.0;
    if (spec.straggling_model == 0) {
        double acc = 0.0;
        if (e0 > kElo) {
            for (int k = threadIdx.x; k < kBohrN; k += blockDim.x) {
                double e = lin(kElo, e0, kBohrN, k);
                double sp = stopping_power(e);
                double beta, gam, b2;
                kinematics(e, beta, gam, b2);
                f_bohr[k] = kBohr / (fmax(b2, 1e-12) * (sp * sp * sp));
            }
            __syncthreads();
            for (int k = threadIdx.x; k < kBohrN - 1; k += blockDim.x) {
                double de = lin(kElo, e0, kBohrN, k + 1) - lin(kElo, e0, kBohrN, k);
                acc += de * (f_bohr[k + 1] + f_bohr[k]) / 2.0;
            }
        }
        red[threadIdx.x] = acc;
        __syncthreads();
        for (int w = blockDim.x / 2; w > 0; w >>= 1) {
            if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
            __syncthreads();
        }
        strag = sqrt(red[0]);
    } else if (spec.straggling_model == 1) {
        strag = spec.strag_coef * pow(r0, spec.strag_exp);
    }
    if (threadIdx.x != 0) return;
    const double espr = kPowerP * spec.energy_spread * r0;
    const double sig_r = hypot(strag, espr);
    const int n = dm.n_idd;
    const double zmax = r0 + 8.0 * sig_r + 0.2;
    const double h = lin(0.0, zmax, n, 1) - 0.0;
    int kk = 0;
    if (sig_r > 0.0) {
        double kf = ceil(16.0 * sig_r / h);
        kk = kf > (double)(n - 1) ? n - 1 : (int)kf;
    }
    LayerScal sc;
    sc.e0 = e0; sc.r0 = r0; sc.sig_r = sig_r; sc.zmax = zmax; sc.h = h; sc.conv_k = kk;
    sc.step = (zmax - 0.0) / (double)(n - 1);
    sc.inv = 1.0 / sc.step;
    // bin k holds dose only where its near edge k zmax / n lies before the range
    const double kr0 = floor(r0 / (zmax / (double)n)) + 1.0;
    sc.last = kr0 < (double)(n - 1) ? (int)kr0 : n - 1;
    scal[lv] = sc;
}

// The arrays of one (layer, variant): the binned CSDA dose (physics.py:362-370), the Gaussian
// kernel table, and T h of the Fermi-Eyges grid -- the local scattering power (physics.py:
// 259-264) times h = numpy.gradient of the grid.  Block (x: layer and variant, y: a share of
// the entries); one range-table search per bin edge, shared through shared memory by the two
// bins that meet there.  t_fe may be null (depth curves only).
constexpr int kFillThreads = 256;
constexpr int kFillBins = 1024;     // bins per block

__device__ __forceinline__ double fe_h(const LutDims& dm, int j) {
    const int n = dm.n_fe;
    if (j == 0) return lin(dm.fe_lo, dm.fe_hi, n, 1) - lin(dm.fe_lo, dm.fe_hi, n, 0);
    if (j == n - 1) return lin(dm.fe_lo, dm.fe_hi, n, n - 1) - lin(dm.fe_lo, dm.fe_hi, n, n - 2);
    return (lin(dm.fe_lo, dm.fe_hi, n, j + 1) - lin(dm.fe_lo, dm.fe_hi, n, j - 1)) / 2.0;
}

__global__ void __launch_bounds__(kFillThreads)
layer_fill_kernel(pbd_lut_spec spec, LutDims dm, const LayerScal* __restrict__ scal,
                  double* __restrict__ binned, double* __restrict__ ker,
                  double* __restrict__ t_fe) {
    __shared__ double s_e[kFillBins + 1];
    asm volatile("griddepcontrol.wait;" ::: "memory");   // the scalars of this call
    const int lv = blockIdx.x, n = dm.n_idd;
    const LayerScal sc = scal[lv];
    const double r0 = sc.r0, zmax = sc.zmax, h = sc.h;
    double* bin = binned + (size_t)lv * n;
    for (int k0 = blockIdx.y * kFillBins; k0 < n; k0 += gridDim.y * kFillBins) {
        const int nb = min(kFillBins, n - k0);
        __syncthreads();
        for (int q = threadIdx.x; q <= nb; q += kFillThreads) {
            const double ea = lin(0.0, zmax, n + 1, k0 + q);
            s_e[q] = ea < r0 ? energy_at_range(fmax(r0 - ea, 0.0)) : 0.0;
        }
        __syncthreads();
        for (int q = threadIdx.x; q < nb; q += kFillThreads) {
            const double zf = lin(0.0, zmax, n, k0 + q);
            const double fl = exp(-zf / spec.atten_len);
            bin[k0 + q] = fl * (s_e[q] - s_e[q + 1]) / h;
        }
    }
    const int t0 = blockIdx.y * kFillThreads + threadIdx.x, stride = gridDim.y * kFillThreads;
    if (sc.sig_r > 0.0) {
        double* kr = ker + (size_t)lv * n;
        const double c = kInvSqrt2Pi / sc.sig_r;
        for (int k = t0; k <= sc.conv_k; k += stride) {
            double t = (double)k * h;
            kr[k] = h * (c * exp(-(t * t) / (2.0 * sc.sig_r * sc.sig_r)));
        }
    }
    if (t_fe == nullptr) return;
    double* tf = t_fe + (size_t)lv * dm.n_fe;
    for (int i = t0; i < dm.n_fe; i += stride) {
        double zf = lin(dm.fe_lo, dm.fe_hi, dm.n_fe, i);
        double t = 0.0;
        if (zf < r0) {
            double el = energy_at_range(fmax(r0 - zf, 0.0));
            t = highland_local(fmax(el, 1e-3));
        }
        tf[i] = t * fe_h(dm, i);
    }
}

// Range-straggling convolution (see the file comment): smooth[i] = sum_m bin[m] kr[|i - m|]
// over |i - m| <= K, bins outside [0, n) being zero, each output summed in ascending m with
// FMA.  A thread owns kConvB consecutive outputs i0 .. i0 + B - 1 and walks the steps
// s = m - i0 + K = 0 .. 2K + B - 1: at each step one bin (shared by its B outputs) and one
// kernel value kr[|K - s|] (the same for every thread of the block) are read from shared
// memory, and the kernel value is kept in a ring of B registers whose slot is the step
// modulo B -- output b needs the value loaded b steps earlier -- so the unrolled body needs
// no register moves.  Steps run in chunks of kConvChunk whose bins and kernel values are
// staged in shared memory; B is odd so that the threads' strided bin reads do not collide
// in the banks.
constexpr int kConvB = 9;
constexpr int kConvThreads = 128;
constexpr int kConvSeg = kConvB * kConvThreads;          // outputs per block
constexpr int kConvChunk = 112 * kConvB;                 // steps per staged chunk
constexpr int kConvSmem = (kConvSeg + kConvChunk + kConvChunk) * (int)sizeof(double);

__global__ void __launch_bounds__(kConvThreads)
conv_kernel(LutDims dm, const LayerScal* scal, const double* binned, const double* ker,
            double* smooth) {
    extern __shared__ double csm[];
    double* sbin = csm;                                   // kConvSeg + kConvChunk bins
    double* skw = csm + kConvSeg + kConvChunk;            // kConvChunk kernel values
    const int lv = blockIdx.x;
    const int n = dm.n_idd;
    const int s0 = blockIdx.y * kConvSeg;
    const double* bin = binned + (size_t)lv * n;
    double* out = smooth + (size_t)lv * n;
    const LayerScal sc = scal[lv];
    if (sc.sig_r <= 0.0) {
        for (int i = s0 + threadIdx.x; i < min(n, s0 + kConvSeg); i += kConvThreads)
            out[i] = bin[i];
        return;
    }
    const double* kr = ker + (size_t)lv * n;
    const int K = sc.conv_k;
    const int n_steps = 2 * K + kConvB;
    const int i0 = s0 + threadIdx.x * kConvB;             // this thread's first output
    double acc[kConvB], ring[kConvB];
#pragma unroll
    for (int b = 0; b < kConvB; ++b) { acc[b] = 0.0; ring[b] = 0.0; }
    for (int c0 = 0; c0 < n_steps; c0 += kConvChunk) {
        // bins m = s0 - K + c0 + j, j < kConvSeg + kConvChunk; kernel kr[|K - c0 - j|], j < chunk
        __syncthreads();
        for (int j = threadIdx.x; j < kConvSeg + kConvChunk; j += kConvThreads) {
            const int m = s0 - K + c0 + j;
            sbin[j] = (m >= 0 && m < n) ? bin[m] : 0.0;
        }
        for (int j = threadIdx.x; j < kConvChunk; j += kConvThreads) {
            const int t = K - c0 - j;
            const int a = t < 0 ? -t : t;
            skw[j] = a <= K ? kr[a] : 0.0;
        }
        __syncthreads();
        const double* sb = sbin + threadIdx.x * kConvB;   // bin of step c0 + j is sb[j]
        for (int j = 0; j < kConvChunk; j += kConvB) {
#pragma unroll
            for (int q = 0; q < kConvB; ++q) {
                ring[q] = skw[j + q];                     // kr[|K - s|], s = c0 + j + q
                const double bv = sb[j + q];
#pragma unroll
                for (int b = 0; b < kConvB; ++b)
                    acc[b] = __fma_rn(bv, ring[(q - b + kConvB) % kConvB], acc[b]);
            }
        }
    }
#pragma unroll
    for (int b = 0; b < kConvB; ++b)
        if (i0 + b < n) out[i0 + b] = acc[b];
}

// The tables at the requested depths.  A depth needs the smoothed curve at two points of its
// fine grid (np.interp's interval) and the scattering integral at two points of its own, so only
// those are formed, straight from the bins and from T h: 2 nz sums of 2 K + 1 products instead
// of n (the whole 6000-point convolution, 325 us for 120 (layer, variant) pairs at 128 depths)
// and 2 nz instead of n_fe for the integral (120 us); both together take 53 us, bound by the
// loads of the bins and kernel values through L1.
//
// One warp per (layer, variant, depth): the lanes stride over the bins (coalesced; the
// windows of a block's neighbouring depths overlap, so they come from L1) and their sums are
// added by a butterfly.  A block holds kEvalDepths depths of one layer with all its
// variants, which combine into the range derivatives.
//
// With `smooth` given (2 nz points would cost more than the whole curve, see lut_build) the
// curve is read instead of summed.
constexpr int kEvalDepths = 8;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// smooth[n0] and smooth[n0 + 1] of the straggling convolution (see conv_kernel): sums over the
// bins |n - m| <= K.  Bins past the range are zero and are not read; for a depth before the
// range, where the curve is of the peak's order, neither are bins more than 9 sigma_R away, whose
// weights (< 3e-18 of the largest) lie below the sum's last bit.  Past the range, where those
// weights are all there is, the window is the whole one.
__device__ __forceinline__ void conv_two(const LayerScal& sc, int n, const double* __restrict__ bin,
                                         const double* __restrict__ kr, int n0, int lane,
                                         double& f0, double& f1) {
    if (sc.sig_r <= 0.0) {
        f0 = bin[n0];
        f1 = n0 + 1 < n ? bin[n0 + 1] : 0.0;
        return;
    }
    int K = sc.conv_k;
    if (n0 < sc.last) {
        const double k9 = ceil(9.0 * sc.sig_r * sc.inv) + 1.0;
        K = k9 < (double)K ? (int)k9 : K;
    }
    const int m0 = max(0, n0 - K), m1 = min(sc.last, n0 + 1 + K);
    double a0 = 0.0, a1 = 0.0;
#pragma unroll 4
    for (int m = m0 + lane; m <= m1; m += 32) {
        const double b = __ldg(bin + m);
        const int d0 = abs(n0 - m), d1 = abs(n0 + 1 - m);
        a0 = __fma_rn(b, d0 <= K ? __ldg(kr + d0) : 0.0, a0);
        a1 = __fma_rn(b, d1 <= K ? __ldg(kr + d1) : 0.0, a1);
    }
    f0 = warp_sum(a0);
    f1 = warp_sum(a1);
}

// Fermi-Eyges direct scattering integral B(zf_i) = sum_{j<i} (zf_i - zf_j)^2 T_j h_j
// (physics.py:266-270) at the grid points i0 and i0 + 1.
__device__ __forceinline__ void fe_two(const LutDims& dm, const double* __restrict__ th, int i0,
                                       int lane, double& b0, double& b1) {
    const int n = dm.n_fe;
    const double step = dm.fe_step;
    const double z0 = lin_s(dm.fe_lo, dm.fe_hi, n, i0, step);
    const double z1 = lin_s(dm.fe_lo, dm.fe_hi, n, min(i0 + 1, n - 1), step);
    double a0 = 0.0, a1 = 0.0;
#pragma unroll 4
    for (int j = lane; j <= i0; j += 32) {       // j = i0 adds 0 to b0 (and i0 = n - 1 uses b0 only)
        const double zj = (double)j * step + dm.fe_lo, t = __ldg(th + j);
        const double d0 = j < i0 ? z0 - zj : 0.0, d1 = z1 - zj;
        a0 += d0 * d0 * t;
        a1 += d1 * d1 * t;
    }
    b0 = warp_sum(a0);
    b1 = warp_sum(a1);
}

__global__ void __launch_bounds__(kEvalDepths * 3 * 32)
lut_eval_kernel(pbd_lut_spec spec, LutDims dm, const LayerScal* __restrict__ scal,
                const double* __restrict__ binned, const double* __restrict__ ker,
                const double* __restrict__ smooth, const double* __restrict__ t_fe,
                double single_depth, double* idd, double* sigma, double* didd, double* dsig) {
    __shared__ double s_i[3][kEvalDepths], s_s[3][kEvalDepths];
    // The arrays of this call.  They are read through L1's read-only path below (__ldg), which may hold only
    // what was complete when this grid started: so the kernels before it must not trigger its launch
    // (griddepcontrol.launch_dependents), and do not -- it starts as their blocks end.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int nb = (dm.nz + kEvalDepths - 1) / kEvalDepths;      // blocks per layer
    const int l = blockIdx.x / nb, k0 = (blockIdx.x - l * nb) * kEvalDepths;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int v = warp / kEvalDepths, kd = warp % kEvalDepths;
    const int k = k0 + kd;
    if (k < dm.nz) {
        const int lv = l * dm.nvar + v;
        const LayerScal sc = scal[lv];
        const int n = dm.n_idd;
        const double d = spec.depth_scale * (spec.z0 + (double)k * spec.dz);
        const double dz_eval = (dm.nz == 1 && !spec.anchor_surface) ? single_depth : d;
        // depth dose: np.interp on linspace(0, zmax, n), 0 outside
        double out_i = 0.0;
        if (!(d < 0.0 || d > sc.zmax)) {
            int lo = 0;
            double x0 = 0.0, f0, f1;
            locate_lin(d, 0.0, sc.zmax, n, sc.step, sc.inv, lo, x0);
            if (smooth) {
                const double* fp = smooth + (size_t)lv * n;
                f0 = fp[lo];
                f1 = lo + 1 < n ? fp[lo + 1] : 0.0;
            } else {
                conv_two(sc, n, binned + (size_t)lv * n, ker + (size_t)lv * n, lo, lane, f0, f1);
            }
            if (x0 == d) {
                out_i = f0;
            } else {
                const double x1 = lin_s(0.0, sc.zmax, n, lo + 1, sc.step);
                out_i = (f1 - f0) / (x1 - x0) * (d - x0) + f0;
            }
        }
        // lateral width: np.interp on the Fermi-Eyges grid, the end values outside
        double b = 0.0;
        if (!(spec.anchor_surface && d <= 0.0)) {
            const int nf = dm.n_fe;
            const double x = fmin(fmax(dz_eval, dm.fe_lo), dm.fe_hi);
            int lo = 0;
            double x0 = 0.0, b0, b1;
            locate_lin(x, dm.fe_lo, dm.fe_hi, nf, dm.fe_step, dm.fe_inv, lo, x0);
            fe_two(dm, t_fe + (size_t)lv * nf, lo, lane, b0, b1);
            if (x0 == x) {
                b = b0;
            } else {
                const double x1 = lin_s(dm.fe_lo, dm.fe_hi, nf, lo + 1, dm.fe_step);
                b = (b1 - b0) / (x1 - x0) * (x - x0) + b0;
            }
        }
        const double zp = dz_eval / spec.depth_scale;
        const double var = spec.sigma_x0 * spec.sigma_x0
                         + 2.0 * spec.rho0 * spec.sigma_x0 * spec.sigma_theta0 * zp
                         + spec.sigma_theta0 * spec.sigma_theta0 * (zp * zp)
                         + b / (spec.depth_scale * spec.depth_scale);
        if (lane == 0) {
            s_i[v][kd] = out_i;
            s_s[v][kd] = sqrt(fmax(var, 0.0));
        }
    }
    __syncthreads();
    const int t = threadIdx.x, ko = k0 + t;
    if (t < kEvalDepths && ko < dm.nz) {
        const size_t o = (size_t)l * dm.nz + ko;
        idd[o] = s_i[0][t];
        sigma[o] = s_s[0][t];
        if (dm.nvar == 3) {
            if (didd) didd[o] = (s_i[1][t] - s_i[2][t]) / (2.0 * dm.fd_step);
            if (dsig) dsig[o] = (s_s[1][t] - s_s[2][t]) / (2.0 * dm.fd_step);
        }
    }
}

// Heterogeneous media: dose = sum_l IDD_l(WED) * lateral_l per voxel, IDD_l the layer's
// smoothed depth curve evaluated at the voxel's water-equivalent depth with the same
// interpolation as the tables.  Accumulated in FP64, in layer order.
//
// A warp owns 128 consecutive voxels (4 per lane, lanes adjacent) and walks the layers that reach any
// of them, the next layer's lateral values loaded while this one's curve points are gathered; layers
// that reach none (smallest WED above zmax) are neither read nor evaluated.  A voxel counts only where
// its WED lies inside the curve (or is NaN): outside [0, zmax] nothing is added, and a (layer, slice)
// the activity table marked inactive has every WED above zmax, so the unwritten part of a lateral map
// is loaded at most, never used.
//
// Bound by the gathers of curve points through L1 (neighbouring columns differ by the CT's noise) and
// instruction issue.  The interval is the rounded estimate alone, without the correction to np.interp's
// exact choice: the interpolation is continuous, so an estimate one interval off within rounding of a
// knot gives the same value to FP64 rounding.  128^3, 40 layers: 195 us with the corrected interval and
// the lateral values in a ring of bulk copies with a block barrier per layer (90 instructions per voxel
// and layer), 98 us now (L1 gathers about 60).
constexpr int kCmbThreads = 256;
constexpr int kCmbPer = 4;                              // voxels per lane
constexpr int kCmbTile = kCmbThreads * kCmbPer;         // voxels per block
constexpr int kCmbLayers = 128;                         // layers whose scalars are staged at a time

__global__ void __launch_bounds__(kCmbThreads, 4) wed_combine_kernel(
    int n, const LayerScal* __restrict__ scal, const double2* __restrict__ pts,
    const float* __restrict__ lateral, size_t lstride, const double* __restrict__ wed, size_t nvox,
    int n_layers, float* __restrict__ dose, const int* __restrict__ fwd_err) {
    __shared__ double s_zmax[kCmbLayers], s_step[kCmbLayers], s_inv[kCmbLayers];
    const int lane = threadIdx.x & 31;
    const size_t v0 = (size_t)blockIdx.x * kCmbTile + (threadIdx.x >> 5) * (32 * kCmbPer) + lane;
    const double inf = __longlong_as_double(0x7FF0000000000000ll);
    constexpr double kMagic = 6755399441055744.0;       // 1.5 2^52: the sum's low word is the integer
    double d[kCmbPer], acc[kCmbPer], mn = inf;
    size_t at[kCmbPer];
#pragma unroll
    for (int j = 0; j < kCmbPer; ++j) {
        const size_t v = v0 + 32 * j;
        at[j] = v < nvox ? v : nvox - 1;
        d[j] = __ldcs(wed + at[j]);
        if (v >= nvox || d[j] < 0.0) d[j] = inf;        // inside no curve
        mn = d[j] != d[j] ? -inf : fmin(mn, d[j]);      // a NaN takes every layer
        acc[j] = 0.0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    for (int b = 0; b < n_layers; b += kCmbLayers) {
        const int nb = min(kCmbLayers, n_layers - b);
        __syncthreads();
        for (int l = threadIdx.x; l < nb; l += kCmbThreads) {
            s_zmax[l] = scal[b + l].zmax;
            s_step[l] = scal[b + l].step;
            s_inv[l] = scal[b + l].inv;
        }
        __syncthreads();
        auto next = [&](int l) {
            while (l < nb && !(mn <= s_zmax[l])) ++l;
            return l;
        };
        float lat[kCmbPer];
        auto fetch = [&](int l, float* x) {
            const float* p = lateral + (size_t)(b + l) * lstride;
#pragma unroll
            for (int j = 0; j < kCmbPer; ++j) x[j] = __ldcs(p + at[j]);
        };
        int l = next(0);
        if (l < nb) fetch(l, lat);
        while (l < nb) {
            const int ln = next(l + 1);
            float ahead[kCmbPer];
#pragma unroll
            for (int j = 0; j < kCmbPer; ++j) ahead[j] = 0.f;
            if (ln < nb) fetch(ln, ahead);
            const double zm = s_zmax[l], st = s_step[l], inv = s_inv[l];
            const double2* lp = pts + (size_t)(b + l) * n;
            double2 pt[kCmbPer];
            double x[kCmbPer];
#pragma unroll
            for (int j = 0; j < kCmbPer; ++j) {
                const double t = fma(d[j], inv, -0.5) + kMagic;
                const unsigned lo = min((unsigned)__double2loint(t), (unsigned)(n - 1));
                x[j] = fma(kMagic - t, st, d[j]);       // from the interval's left point
                pt[j] = __ldg(lp + lo);
            }
#pragma unroll
            for (int j = 0; j < kCmbPer; ++j) {
                const double idd = fma(pt[j].y, x[j], pt[j].x);
                if (!(d[j] > zm) && idd != 0.0) acc[j] = fma(idd, (double)lat[j], acc[j]);
            }
#pragma unroll
            for (int j = 0; j < kCmbPer; ++j) lat[j] = ahead[j];
            l = ln;
        }
    }
    // a wait of the lateral maps' forward ran out: the whole dose is invalid
    const bool bad = fwd_err && *fwd_err;
#pragma unroll
    for (int j = 0; j < kCmbPer; ++j)
        if (v0 + 32 * j < nvox) __stcs(dose + v0 + 32 * j, bad ? __int_as_float(0x7fc00000) : (float)acc[j]);
}

// Depth dose of a layer's curve {value, slope} at depth d, 0 outside [0, zmax]: the interval is the
// rounded estimate alone, as in the combine (any d, NaN included, gives an index inside the curve);
// scalars as in LayerScal.
struct CurveScal {
    double zmax, step, inv;
};
struct CurvePoint {
    double2 pt;
    double x;                // from the interval's left point
};
__device__ __forceinline__ CurvePoint curve_point(const CurveScal& c, const double2* __restrict__ pts,
                                                  int n, double d) {
    constexpr double kMagic = 6755399441055744.0;
    const double t = fma(d, c.inv, -0.5) + kMagic;
    const unsigned lo = min((unsigned)__double2loint(t), (unsigned)(n - 1));
    return CurvePoint{__ldg(pts + lo), fma(kMagic - t, c.step, d)};
}
__device__ __forceinline__ double curve_value(const CurvePoint& p, double zmax, double d) {
    return d < 0.0 || d > zmax ? 0.0 : fma(p.pt.y, p.x, p.pt.x);
}

// The heterogeneous dose's dL/dD seen by layer l: maps[l * lstride + v] = IDD_l(WED[v]) *
// grad[v] (FP64 product, rounded once to FP32), 0 outside the curve.  The adjoint of layer l
// with this map and depth dose 1 on its active slices is dL/dW_l.  kRange: also, at maps +
// set_stride, dL/dD times the range derivative of the layer's depth dose at the WED,
// (IDD+_l(WED) - IDD-_l(WED)) / (2 h), from the curves at range shifts +h and -h (FP64 difference,
// one FP32 rounding of the product).  Only slices that the layer's activity table (act, act +
// act_stride) marks are written: the adjoint reads no other.
//
// One block per 512 voxels of a slice, two per thread, over the slice's active layers.  Bound by the
// gathers of the curve points through L1 and their latency: both voxels' points of all three curves
// are in flight together.  128^3 x 28 layers, both sets: 497 us as two kernels over every pair with
// a division per curve; 240 us in one pass over the active pairs (about half) with np.interp's exact
// interval; 150 us now, with the estimated interval and the points loaded ahead.
constexpr int kMapThreads = 256, kMapPer = 2;
constexpr int kMapLayers = 128;   // layers staged together

template <bool kRange>
__global__ void __launch_bounds__(kMapThreads) wed_grad_maps_kernel(
    int n, const LayerScal* __restrict__ scal, const double2* __restrict__ pts,
    const LayerScal* __restrict__ scp, const double2* __restrict__ ptp,
    const LayerScal* __restrict__ scm, const double2* __restrict__ ptm,
    const float* __restrict__ grad, const double* __restrict__ wed, size_t nslice, int nz,
    int n_layers, const double* __restrict__ act, size_t act_stride, size_t lstride,
    size_t set_stride, double inv2h, float* __restrict__ maps) {
    __shared__ CurveScal s_c[kRange ? 3 : 1][kMapLayers];
    __shared__ int s_l[kMapLayers];      // active layers of the batch: index, bit 30 / 31: set 0 / 1
    __shared__ int s_n;
    const size_t nb = (nslice + kMapThreads * kMapPer - 1) / (kMapThreads * kMapPer);
    const int z = (int)(blockIdx.x / nb);
    const size_t v0 = (blockIdx.x - z * nb) * (kMapThreads * kMapPer) + threadIdx.x;
    double d[kMapPer], g[kMapPer];
    float* out[kMapPer];
    bool in[kMapPer];
#pragma unroll
    for (int q = 0; q < kMapPer; ++q) {
        const size_t v = v0 + q * kMapThreads;
        in[q] = v < nslice;
        const size_t o = (size_t)z * nslice + (in[q] ? v : 0);
        d[q] = wed[o];
        g[q] = (double)grad[o];
        out[q] = maps + o;
    }
    for (int l0 = 0; l0 < n_layers; l0 += kMapLayers) {
        __syncthreads();
        if (threadIdx.x < 32) {          // the batch's active layers, in layer order
            int cnt = 0;
            for (int b = 0; b < kMapLayers; b += 32) {
                const int l = l0 + b + (int)threadIdx.x;
                unsigned f = 0u;
                if (l < n_layers) {
                    if (act[(size_t)l * nz + z] != 0.0) f |= 1u << 30;
                    if (kRange && act[act_stride + (size_t)l * nz + z] != 0.0) f |= 1u << 31;
                }
                const unsigned bal = __ballot_sync(0xffffffffu, f != 0u);
                if (f) s_l[cnt + __popc(bal & ((1u << threadIdx.x) - 1u))] = (int)(f | (unsigned)l);
                cnt += __popc(bal);
            }
            if (threadIdx.x == 0) s_n = cnt;
        }
        __syncthreads();
        const int na = s_n;
        for (int k = threadIdx.x; k < na; k += kMapThreads) {
            const int l = s_l[k] & 0x3FFFFFFF;
            s_c[0][k] = CurveScal{scal[l].zmax, scal[l].step, scal[l].inv};
            if constexpr (kRange) {
                s_c[1][k] = CurveScal{scp[l].zmax, scp[l].step, scp[l].inv};
                s_c[2][k] = CurveScal{scm[l].zmax, scm[l].step, scm[l].inv};
            }
        }
        __syncthreads();
        for (int k = 0; k < na; ++k) {
            const unsigned f = (unsigned)s_l[k];
            const size_t l = f & 0x3FFFFFFFu;
            // every curve point of the layer in flight together, whichever sets are written
            CurvePoint p[kRange ? 3 : 1][kMapPer];
#pragma unroll
            for (int q = 0; q < kMapPer; ++q) {
                p[0][q] = curve_point(s_c[0][k], pts + l * n, n, d[q]);
                if constexpr (kRange) {
                    p[1][q] = curve_point(s_c[1][k], ptp + l * n, n, d[q]);
                    p[2][q] = curve_point(s_c[2][k], ptm + l * n, n, d[q]);
                }
            }
            if (f & (1u << 30)) {
#pragma unroll
                for (int q = 0; q < kMapPer; ++q)
                    if (in[q]) {             // 0 outside the curve, whatever the gradient there (inf, NaN)
                        const double zm = s_c[0][k].zmax;
                        const bool outside = d[q] < 0.0 || d[q] > zm;
                        out[q][l * lstride] = outside ? 0.f : (float)(curve_value(p[0][q], zm, d[q]) * g[q]);
                    }
            }
            if constexpr (kRange) {
                if (f & (1u << 31)) {
#pragma unroll
                    for (int q = 0; q < kMapPer; ++q) {
                        const double dp = curve_value(p[1][q], s_c[1][k].zmax, d[q]);
                        const double dm = curve_value(p[2][q], s_c[2][k].zmax, d[q]);
                        if (in[q]) out[q][set_stride + l * lstride] = (float)((dp - dm) * inv2h * g[q]);
                    }
                }
            }
        }
    }
}

// Curve points of the smoothed depth curves: {fp[k], slope_k} with slope_k = (fp[k+1] - fp[k])
// / (x[k+1] - x[k]) on the grid linspace(0, zmax, n) -- the operands and the single rounding
// of np.interp's slope (and of lut_eval_kernel) -- and 0 at the last point.  Value and slope share a
// 16-byte load in the combine, which needs no division per voxel.
__global__ void wed_slope_kernel(LutDims dm, const LayerScal* scal, const double* smooth,
                                 double2* pts) {
    const int l = blockIdx.x;
    const int n = dm.n_idd;
    const double zm = scal[l].zmax;
    const double st = (zm - 0.0) / (double)(n - 1);
    const double* fp = smooth + (size_t)l * n;
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        double s = 0.0;
        if (k < n - 1) {
            const double x0 = lin_s(0.0, zm, n, k, st), x1 = lin_s(0.0, zm, n, k + 1, st);
            s = (fp[k + 1] - fp[k]) / (x1 - x0);
        }
        pts[(size_t)l * n + k] = make_double2(fp[k], s);
    }
}

// Per (layer, slice) activity of the heterogeneous dose: 1 when some voxel of the slice has a
// WED inside the layer's depth curve (<= zmax), else 0 (the layer adds nothing there).  One
// block per slice: the slice's smallest WED, then one entry per layer.
constexpr int kActThreads = 1024;

__global__ void __launch_bounds__(kActThreads) wed_activity_kernel(const LayerScal* scal,
                                                                   const LayerScal* scal2,
                                                                   const double* wed,
                                                                   size_t nslice, int nz,
                                                                   int n_layers, double* act) {
    __shared__ double red[kActThreads / 32];
    const int z = blockIdx.x;
    const double* p = wed + (size_t)z * nslice;
    const double inf = __longlong_as_double(0x7FF0000000000000ll);
    // eight independent loads in flight per thread; fmin is exact in any order (NaN ignored)
    double m[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) m[q] = inf;
    size_t v = threadIdx.x;
    for (; v + 7 * (size_t)kActThreads < nslice; v += 8 * (size_t)kActThreads) {
#pragma unroll
        for (int q = 0; q < 8; ++q) m[q] = fmin(m[q], __ldcs(p + v + (size_t)q * kActThreads));
    }
    for (; v < nslice; v += kActThreads) m[0] = fmin(m[0], __ldcs(p + v));
    double t = fmin(fmin(fmin(m[0], m[1]), fmin(m[2], m[3])), fmin(fmin(m[4], m[5]), fmin(m[6], m[7])));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t = fmin(t, __shfl_xor_sync(0xffffffffu, t, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x < 32) {
        t = red[threadIdx.x];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t = fmin(t, __shfl_xor_sync(0xffffffffu, t, o));
        if (threadIdx.x == 0) red[0] = t;
    }
    __syncthreads();
    const double smin = red[0];
    // with a second curve set: active where either set's curve reaches
    for (int l = threadIdx.x; l < n_layers; l += kActThreads) {
        const double zm = scal2 ? fmax(scal[l].zmax, scal2[l].zmax) : scal[l].zmax;
        act[(size_t)l * nz + z] = smin <= zm ? 1.0 : 0.0;
    }
}

// Water-equivalent depth at the voxel centres z_k = oz + k dz along +z (the beam axis):
// the sum of rho * path length from depth 0 (physics.py:421-423 per voxel path), voxel i
// filling [z_i - dz/2, z_i + dz/2] with rho_i, water above the first voxel, path lengths
// clipped at depth 0.  FP64.
//
// A block holds 32 columns and kRuns runs of 8 depths (one per warp): each thread sums its run, the sums
// of the runs above are added through shared memory, 8 kRuns depths at a time; the path lengths, the
// same for every column, come from a table of the pass.  Few columns are bound by the latency of the loads (one
// thread per column, 16 in flight: 128^3 17.8 us, now 6.9), many by FP64 issue, which the sums of the runs
// and warps without a depth of their own add to.  So as many runs as the depths fill, up to 16 below 16,000 columns,
// 4 below 100,000 and 1 (a thread per column) above; the sums' order is the same for any number.  Sixteen for
// every grid, path lengths in each thread, against one thread per column before that and now: 512 x 512 x 64
// 121, 50, 40 us; 512 x 512 x 150 237, 114, 91; 128 x 128 x 1 7.3, 2.3, 2.5; 200 x 200 x 256 48, 68, 35.
constexpr int kRayCols = 32, kRayLen = 8, kRayMaxRuns = 16;

template <int kRuns>
__global__ void __launch_bounds__(kRayCols * kRuns, 32 / kRuns) wed_raytrace_kernel(
    int nz, size_t ncol, double oz, double dz, const float* __restrict__ rho, double* __restrict__ wed) {
    __shared__ double sums[2][kRuns][kRayCols];
    __shared__ double2 s_len[2][kRuns * kRayLen];        // path to each depth's voxel centre and through the voxel
    const int lane = threadIdx.x & 31, run = threadIdx.x >> 5;
    int buf = 0;
    for (size_t c0 = (size_t)blockIdx.x * kRayCols; c0 < ncol; c0 += (size_t)gridDim.x * kRayCols) {
        const size_t c = c0 + lane;
        const bool in = c < ncol;
        double above = fmax(oz - 0.5 * dz, 0.0);         // water above the first voxel
        for (int k0 = 0; k0 < nz; k0 += kRuns * kRayLen) {
            const int kr = k0 + run * kRayLen;
            float r[kRayLen];
#pragma unroll
            for (int q = 0; q < kRayLen; ++q)
                r[q] = in && kr + q < nz ? __ldcs(rho + (size_t)(kr + q) * ncol + c) : 0.f;
            if (threadIdx.x < kRuns * kRayLen) {
                const double zc = oz + (double)(k0 + (int)threadIdx.x) * dz;
                const double lo = fmax(zc - 0.5 * dz, 0.0), mid = fmax(zc, 0.0), hi = fmax(zc + 0.5 * dz, 0.0);
                s_len[buf][threadIdx.x] = make_double2(mid - lo, hi - lo);
            }
            __syncthreads();
            const double2* len = s_len[buf] + run * kRayLen;
            double acc = above;
            if constexpr (kRuns > 1) {
                double sum = 0.0;
#pragma unroll
                for (int q = 0; q < kRayLen; ++q) sum += (double)r[q] * len[q].y;
                sums[buf][run][lane] = sum;
                __syncthreads();
#pragma unroll 4
                for (int w = 0; w < kRuns; ++w) {
                    if (w == run) acc = above;
                    above += sums[buf][w][lane];
                }
            }
            double own = 0.0;
#pragma unroll
            for (int q = 0; q < kRayLen; ++q) {
                const double rr = (double)r[q];
                if (in && kr + q < nz) __stcs(wed + (size_t)(kr + q) * ncol + c, acc + rr * len[q].x);
                acc += rr * len[q].y;
                if (kRuns == 1) own += rr * len[q].y;
            }
            if (kRuns == 1) above += own;
            buf ^= 1;                                    // the next pass's tables: no barrier here
        }
    }
}

// Depth list of the Fermi-Eyges integral (host): its first and last points and size.
struct FeList {
    int n_list;
    double lo, hi, single_depth;
    int n_fine;
};

FeList fe_list(const pbd_lut_spec* s) {
    FeList fl{};
    const int nz = s->nz;
    auto depth = [&](int k) { return s->depth_scale * (s->z0 + (double)k * s->dz); };
    fl.single_depth = 0.0;
    if (!s->anchor_surface) {
        if (nz == 1) {  // physics.py:249-253
            double z1 = depth(0);
            fl.single_depth = z1 > 0 ? z1 : 1e-6;
            fl.lo = 0.0; fl.hi = fl.single_depth; fl.n_list = 2;
        } else {
            fl.lo = depth(0); fl.hi = depth(nz - 1); fl.n_list = nz;
        }
    } else {
        int pos = 0;
        for (int k = 0; k < nz; ++k) pos += depth(k) > 0.0;
        fl.lo = 0.0;
        fl.hi = pos > 0 ? depth(nz - 1) : 1e-6;
        fl.n_list = pos + 1;
    }
    double span = fl.hi - fl.lo;   // physics.py:256-258
    int need = span > 0 ? (int)ceil(span / fmax(s->fe_max_step, 1e-6)) + 1 : 2;
    int a = (fl.n_list - 1) * s->fe_n_sub + 1;
    int nf = a > need ? a : need;
    fl.n_fine = nf > 2 ? nf : 2;
    return fl;
}

int validate_spec(const pbd_lut_spec* s, int n_layers) {
    if (!s) return PBD_ERR_NULL_ARG;
    if (n_layers <= 0 || s->nz <= 0 || s->idd_n_fine < 3 || s->fe_n_sub < 1) return PBD_ERR_BAD_DIM;
    if (!(s->dz > 0.0) || !(s->depth_scale > 0.0) || !(s->atten_len > 0.0) ||
        !(s->fe_max_step > 0.0) || !(s->fd_step >= 0.0) || !(s->sigma_x0 >= 0.0) ||
        !(s->energy_spread >= 0.0))
        return PBD_ERR_BAD_VALUE;
    if (s->straggling_model < 0 || s->straggling_model > 2) return PBD_ERR_BAD_VALUE;
    if (s->idd_n_fine > (1 << 20)) return PBD_ERR_UNSUPPORTED;
    FeList fl = fe_list(s);
    if (fl.n_fine > (1 << 16)) return PBD_ERR_UNSUPPORTED;
    return PBD_OK;
}

// The range table is a constant of the physics: the first call on a device builds it and
// waits for it (once per process and device), so that later calls on any stream find it
// ready.  Inside a stream capture the build is recorded into the graph instead and the
// device is not marked.
bool g_range_built[64];

int ensure_range_table(cudaStream_t st) {
    int dev = 0;
    PBD_TRY(cuda_rc(cudaGetDevice(&dev)));
    if (dev >= 0 && dev < 64 && g_range_built[dev]) return PBD_OK;
    range_table_kernel<<<1, 1024, 0, st>>>();
    PBD_LAUNCH_CHECK();
    count_launch(1);
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    PBD_TRY(cuda_rc(cudaStreamIsCapturing(st, &cs)));
    if (cs == cudaStreamCaptureStatusNone && dev >= 0 && dev < 64) {
        PBD_TRY(cuda_rc(cudaStreamSynchronize(st)));
        g_range_built[dev] = true;
    }
    return PBD_OK;
}

struct LutWs {
    LayerScal* scal;
    double *binned, *ker, *smooth, *t_fe;
};

// Scalars, then the arrays, of every (layer, variant); the fills start as the scalars' blocks
// end (a programmatic dependent).  The first launch is an ordinary one: it must not start while
// an earlier call on the stream still reads the workspace.
int launch_layer_setup(const pbd_lut_spec& spec, const LutDims& dm, const double* energies,
                       const double* shift, const LutWs& w, double* t_fe, cudaStream_t st) {
    const int lvn = dm.n_layers * dm.nvar;
    layer_scal_kernel<<<lvn, kScalThreads, 0, st>>>(spec, dm, energies, shift, w.scal);
    PBD_LAUNCH_CHECK();
    const int parts = std::min((dm.n_idd + kFillBins - 1) / kFillBins, 64);
    PBD_TRY(launch_dependent(layer_fill_kernel, dim3(lvn, parts), dim3(kFillThreads), 0, st, spec,
                             dm, (const LayerScal*)w.scal, w.binned, w.ker, t_fe));
    count_launch(2);
    return PBD_OK;
}

size_t carve_lut(Carve& c, LutWs& w, int n_layers, int nvar, int n_idd, int n_fe) {
    const size_t lv = (size_t)n_layers * nvar;
    w.scal = c.take<LayerScal>(lv);
    w.binned = c.take<double>(lv * n_idd);
    w.ker = c.take<double>(lv * n_idd);
    w.smooth = c.take<double>(lv * n_idd);
    w.t_fe = c.take<double>(lv * n_fe);
    return c.used;
}

}  // namespace

int lut_workspace_bytes(const pbd_lut_spec* s, int n_layers, size_t* bytes) {
    PBD_TRY(validate_spec(s, n_layers));
    if (!bytes) return PBD_ERR_NULL_ARG;
    FeList fl = fe_list(s);
    Carve c(nullptr);
    LutWs w;
    *bytes = carve_lut(c, w, n_layers, s->fd_step > 0 ? 3 : 1, s->idd_n_fine, fl.n_fine) + 256;
    return PBD_OK;
}

int lut_build(const pbd_lut_spec* s, int n_layers, const double* energies, const double* shift,
              double* idd, double* sigma, double* didd, double* dsig, void* ws, size_t ws_bytes,
              cudaStream_t st) {
    PBD_TRY(validate_spec(s, n_layers));
    if (!energies || !idd || !sigma) return PBD_ERR_NULL_ARG;
    if (s->fd_step > 0 && (!didd || !dsig)) return PBD_ERR_NULL_ARG;
    size_t need = 0;
    PBD_TRY(lut_workspace_bytes(s, n_layers, &need));
    if (!ws || ws_bytes < need) return PBD_ERR_WORKSPACE;
    FeList fl = fe_list(s);
    LutDims dm;
    dm.n_layers = n_layers;
    dm.nvar = s->fd_step > 0 ? 3 : 1;
    dm.nz = s->nz;
    dm.n_idd = s->idd_n_fine;
    dm.n_fe = fl.n_fine;
    dm.fe_lo = fl.lo;
    dm.fe_hi = fl.hi;
    dm.fe_step = (fl.hi - fl.lo) / (double)(fl.n_fine - 1);
    dm.fe_inv = 1.0 / dm.fe_step;
    dm.fd_step = s->fd_step;
    Carve c(ws);
    LutWs w;
    carve_lut(c, w, n_layers, dm.nvar, dm.n_idd, dm.n_fe);
    const int lvn = n_layers * dm.nvar;

    PBD_TRY(ensure_range_table(st));
    PBD_TRY(launch_layer_setup(*s, dm, energies, shift, w, w.t_fe, st));
    // A depth's two points cost a warp 2 (2 K + 1) products at about a quarter of the rate of
    // the whole curve's blocked convolution, which forms n of them.  Measured (40 layers x 3
    // variants, n = 6000), points against the whole curve: 375 depths 171 / 435 us, 1024 depths
    // 553 / 706, 1500 depths 927 / 1002; the points grow with the depths, so the curve from there.
    const double* smooth = nullptr;
    if (4LL * dm.nz >= dm.n_idd) {
        conv_kernel<<<dim3(lvn, (dm.n_idd + kConvSeg - 1) / kConvSeg), kConvThreads, kConvSmem,
                      st>>>(dm, w.scal, w.binned, w.ker, w.smooth);
        PBD_LAUNCH_CHECK();
        count_launch(1);
        smooth = w.smooth;
    }
    const long long blocks = (long long)((dm.nz + kEvalDepths - 1) / kEvalDepths) * n_layers;
    if (blocks > 2147483647LL) return PBD_ERR_UNSUPPORTED;
    PBD_TRY(launch_dependent(lut_eval_kernel,
                             dim3((unsigned)blocks),
                             dim3(kEvalDepths * dm.nvar * 32), 0, st, *s, dm,
                             (const LayerScal*)w.scal, (const double*)w.binned,
                             (const double*)w.ker, smooth, (const double*)w.t_fe,
                             fl.single_depth, idd, sigma, didd, dsig));
    count_launch(1);
    return PBD_OK;
}

// The depth-curve blob of the heterogeneous dose: the table builder's nominal-variant
// workspace followed by the curve points {value, slope} (n_layers, n_idd).
static size_t carve_curves(Carve& c, LutWs& w, double2*& pts, int n_layers, int n_idd, int n_fe) {
    carve_lut(c, w, n_layers, 1, n_idd, n_fe);
    pts = c.take<double2>((size_t)n_layers * n_idd);
    return c.used;
}

int lut_curve_workspace(const pbd_lut_spec* s, int n_layers, size_t* bytes) {
    PBD_TRY(validate_spec(s, n_layers));
    if (!bytes) return PBD_ERR_NULL_ARG;
    FeList fl = fe_list(s);
    Carve c(nullptr);
    LutWs w;
    double2* pts = nullptr;
    *bytes = carve_curves(c, w, pts, n_layers, s->idd_n_fine, fl.n_fine) + 256;
    return PBD_OK;
}

static int wed_dims(const pbd_lut_spec* s, int n_layers, const void* ws, size_t ws_bytes,
                    LutDims& dm, LutWs& w, double2*& pts) {
    size_t need = 0;
    PBD_TRY(lut_curve_workspace(s, n_layers, &need));
    if (!ws || ws_bytes < need) return PBD_ERR_WORKSPACE;
    FeList fl = fe_list(s);
    dm.n_layers = n_layers;
    dm.nvar = 1;
    dm.nz = s->nz;
    dm.n_idd = s->idd_n_fine;
    dm.n_fe = fl.n_fine;
    dm.fe_lo = fl.lo;
    dm.fe_hi = fl.hi;
    dm.fe_step = (fl.hi - fl.lo) / (double)(fl.n_fine - 1);
    dm.fe_inv = 1.0 / dm.fe_step;
    dm.fd_step = 0.0;
    Carve c(const_cast<void*>(ws));
    carve_curves(c, w, pts, n_layers, dm.n_idd, dm.n_fe);
    return PBD_OK;
}

int lut_wed_curves(const pbd_lut_spec* s, int n_layers, const double* energies,
                   const double* shift, void* curves, size_t curves_bytes, cudaStream_t st) {
    PBD_TRY(validate_spec(s, n_layers));
    if (!energies) return PBD_ERR_NULL_ARG;
    LutDims dm;
    LutWs w;
    double2* pts = nullptr;
    PBD_TRY(wed_dims(s, n_layers, curves, curves_bytes, dm, w, pts));
    PBD_TRY(ensure_range_table(st));
    PBD_TRY(launch_layer_setup(*s, dm, energies, shift, w, nullptr, st));
    conv_kernel<<<dim3(n_layers, (dm.n_idd + kConvSeg - 1) / kConvSeg), kConvThreads, kConvSmem, st>>>(
        dm, w.scal, w.binned, w.ker, w.smooth);
    PBD_LAUNCH_CHECK();
    wed_slope_kernel<<<n_layers, 256, 0, st>>>(dm, w.scal, w.smooth, pts);
    PBD_LAUNCH_CHECK();
    count_launch(2);
    return PBD_OK;
}

int lut_wed_activity(const pbd_lut_spec* s, int n_layers, const void* curves, size_t curves_bytes,
                     const double* wed, int nz, size_t nslice, double* act, cudaStream_t st,
                     const void* curves2, size_t curves2_bytes) {
    PBD_TRY(validate_spec(s, n_layers));
    if (!wed || !act) return PBD_ERR_NULL_ARG;
    LutDims dm;
    LutWs w;
    double2* pts = nullptr;
    PBD_TRY(wed_dims(s, n_layers, curves, curves_bytes, dm, w, pts));
    const LayerScal* scal2 = nullptr;
    if (curves2) {
        LutDims dm2;
        LutWs w2;
        double2* pts2 = nullptr;
        PBD_TRY(wed_dims(s, n_layers, curves2, curves2_bytes, dm2, w2, pts2));
        scal2 = w2.scal;
    }
    wed_activity_kernel<<<nz, kActThreads, 0, st>>>(w.scal, scal2, wed, nslice, nz, n_layers, act);
    PBD_LAUNCH_CHECK();
    count_launch(1);
    return PBD_OK;
}

int lut_wed_combine(const pbd_lut_spec* s, int n_layers, const float* lateral, size_t lstride,
                    const double* wed, size_t nvox, float* dose, const int* fwd_err,
                    const void* curves, size_t curves_bytes, cudaStream_t st) {
    PBD_TRY(validate_spec(s, n_layers));
    if (!lateral || !wed || !dose) return PBD_ERR_NULL_ARG;
    if (lstride < nvox) return PBD_ERR_BAD_VALUE;
    LutDims dm;
    LutWs w;
    double2* pts = nullptr;
    PBD_TRY(wed_dims(s, n_layers, curves, curves_bytes, dm, w, pts));
    const size_t blocks = (nvox + kCmbTile - 1) / kCmbTile;
    if (blocks > 0x7fffffffu) return PBD_ERR_UNSUPPORTED;
    wed_combine_kernel<<<(unsigned)blocks, kCmbThreads, 0, st>>>(dm.n_idd, w.scal, pts, lateral, lstride, wed,
                                                                 nvox, n_layers, dose, fwd_err);
    PBD_LAUNCH_CHECK();
    count_launch(1);
    return PBD_OK;
}

int lut_wed_grad_maps(const pbd_lut_spec* s, int n_layers, const void* curves,
                      size_t curves_bytes, const void* curves_p, const void* curves_m, double h,
                      const float* grad, const double* wed, int nz, size_t nslice,
                      const double* act, size_t lstride, float* maps, cudaStream_t st) {
    PBD_TRY(validate_spec(s, n_layers));
    if (!grad || !wed || !maps || !act) return PBD_ERR_NULL_ARG;
    const size_t nvox = (size_t)nz * nslice;
    if (lstride < nvox) return PBD_ERR_BAD_VALUE;
    const bool range = curves_p != nullptr;
    if (range && (!curves_m || !(h > 0.0) || !isfinite(h))) return PBD_ERR_BAD_VALUE;
    LutDims dm, dp, dn;
    LutWs w, wp{}, wm{};
    double2 *pts = nullptr, *pp = nullptr, *pm = nullptr;
    PBD_TRY(wed_dims(s, n_layers, curves, curves_bytes, dm, w, pts));
    if (range) {
        PBD_TRY(wed_dims(s, n_layers, curves_p, curves_bytes, dp, wp, pp));
        PBD_TRY(wed_dims(s, n_layers, curves_m, curves_bytes, dn, wm, pm));
    }
    const size_t per = (size_t)kMapThreads * kMapPer;
    const size_t blocks = (nslice + per - 1) / per * (size_t)nz;
    if (blocks > 2147483647u) return PBD_ERR_UNSUPPORTED;
    const size_t act_stride = (size_t)n_layers * nz, set_stride = (size_t)n_layers * lstride;
    const auto kernel = range ? wed_grad_maps_kernel<true> : wed_grad_maps_kernel<false>;
    kernel<<<(unsigned)blocks, kMapThreads, 0, st>>>(
        dm.n_idd, w.scal, pts, wp.scal, pp, wm.scal, pm, grad, wed, nslice, nz, n_layers, act,
        act_stride, lstride, set_stride, range ? 0.5 / h : 0.0, maps);
    PBD_LAUNCH_CHECK();
    count_launch(1);
    return PBD_OK;
}

int lut_wed_raytrace(int nz, int ny, int nx, double oz, double dz, const float* rho, double* wed,
                     cudaStream_t st) {
    if (!rho || !wed) return PBD_ERR_NULL_ARG;
    if (nz <= 0 || ny <= 0 || nx <= 0) return PBD_ERR_BAD_DIM;
    if (!isfinite(oz) || !(dz > 0.0) || !isfinite(dz)) return PBD_ERR_BAD_VALUE;
    const size_t ncol = (size_t)ny * nx;
    const int blocks = (int)std::min<size_t>((ncol + kRayCols - 1) / kRayCols, (size_t)num_sms() * 32);
    // the least power of two of runs that holds every depth; 4 at most from 16,000 columns on, 1 from 100,000
    // (256 x 256 x 128: 4 runs 20 us, 1 25, 16 27; 350 x 350 x 100: 1 run 32, 4 38; 64 x 64 x 256: 16 runs 4.8, 4 8.6)
    const int most = ncol >= 100000 ? 1 : ncol >= 16000 ? 4 : kRayMaxRuns;
    int runs = 1;
    while (runs < most && runs * kRayLen < nz) runs *= 2;
    const auto kernel = runs == 1   ? wed_raytrace_kernel<1>
                        : runs == 2 ? wed_raytrace_kernel<2>
                        : runs == 4 ? wed_raytrace_kernel<4>
                        : runs == 8 ? wed_raytrace_kernel<8>
                                    : wed_raytrace_kernel<kRayMaxRuns>;
    kernel<<<blocks, kRayCols * runs, 0, st>>>(nz, ncol, oz, dz, rho, wed);
    PBD_LAUNCH_CHECK();
    count_launch(1);
    return PBD_OK;
}

int lut_csda(const double* e, double* r, int n, int inverse, cudaStream_t st) {
    if (!e || !r) return PBD_ERR_NULL_ARG;
    if (n < 0) return PBD_ERR_BAD_DIM;
    PBD_TRY(ensure_range_table(st));
    if (n == 0) return PBD_OK;
    csda_kernel<<<(n + 255) / 256, 256, 0, st>>>(e, r, n, inverse);
    PBD_LAUNCH_CHECK();
    count_launch(1);
    return PBD_OK;
}

}  // namespace pbd
