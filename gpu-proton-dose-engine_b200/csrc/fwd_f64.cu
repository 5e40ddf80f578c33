// fwd_f64.cu -- forward dose in FP64: the float64 form of the reference's engine on CUDA
// (engines.torch_separable with dtype=torch.float64, engines.py:223-224, 230-274), for callers
// that need the dose to ~1e-15 rather than ~1e-7.
//
//   D[z,y,x] = sum_l IDD_l(z) / (2 pi s^2) sum_j Gy[y,j] sum_i W_l[j,i] Gx[x,i]
//   Gx[x,i] = exp(-(x_v - xs_i)^2 / (2 s^2)),  s = max(sigma_l(z), 1e-9)
//
// One block per (TY x 64 lateral tile, depth slice), over every layer of the slice: the dose
// tile is summed in registers (layer order, then the spot chunks in order) and written once,
// so no scratch memory, no second pass and a deterministic result.  Per active layer and
// chunk of at most 64 spots the block generates Gx, Gy (distances from FP64 differences) and
// W' = W IDD / (2 pi s^2) in shared memory, forms U[j, x] = sum_i W'[j,i] Gx[x,i] and adds
// D[y, x] += sum_j Gy[y,j] U[j,x], both with FP64 matrix instructions (mma.sync m16n8k4; tcgen05
// has no FP64 kind).
//
// What bounds it is the FP64 pipe (64 products per clock and SM, 36 TFLOP/s measured for FMA and
// for the matrix form alike): about 990,000 products and 15,700 exponentials per (layer, slice)
// of the 128^2 grid with 41 x 41 spots.  Hence
//  * the matrix form: one instruction and three 8-byte shared-memory loads per 512 products.
//    With FMAs and 8 x 4 voxels per thread the same tiles took 918 us (pipe 27 % busy: the loads
//    and their latency filled the rest), with 64 x 64 tiles and 4 x 4 voxels 965 us; now 322 us
//    at 128^3 / 41 x 41 x 40 (6.1 ms against 16.9 at 200^2 x 256 / 61 x 61 x 60);
//  * exp as a table of 2^(j/32) and a degree-6 polynomial: 11 FP64 operations instead of the
//    library's 23;
//  * 64 columns by TY = 128 rows: tiles split along x share none of U, and Gy, which every column
//    tile repeats, is formed twice only;
//  * a spot chunk of the lattice rounded up to 4, which leaves room for two blocks per SM up to
//    44 spots: one block's barriers run under the other's products.
// What is left: a slice's layers run in one block (no scratch to split them over), so the grid
// lasts as long as its longest block, 40 layers of 8 us, in which 8 warps cannot hide all of the
// latency between the barriers (512 threads measured the same, 64-row tiles at three blocks per SM
// 426 us).
#include <math.h>

#include <type_traits>

#include "pbd_internal.cuh"

namespace pbd {
namespace {

constexpr int kTX = 64;            // tile columns
constexpr int kSCMax = 64;         // spots per chunk, at most
constexpr int kThreads = 256;
constexpr int kLayerBatch = 128;   // layers whose scalars are staged together
// Row lengths: 4 (mod 8) doubles, so that the four rows and four columns that 16 lanes of a
// fragment load touch lie in 16 different 8-byte banks.
constexpr int kLDX = kTX + 4;
__host__ __device__ constexpr int ld_y(int ty) { return ty + 4; }
__host__ __device__ constexpr int ld_w(int sc) { return sc % 8 ? sc : sc + 4; }

// doubles of dynamic shared memory for spot chunks of sc (a multiple of 4)
constexpr size_t smem_doubles(int ty, int sc) {
    return (size_t)sc * (2 * kLDX + ld_y(ty) + ld_w(sc));
}

// exp(x) for x <= 0 by table lookup (P. T. P. Tang, Table-driven implementation of the
// exponential function, ACM TOMS 15, 1989): x = (32 k + j) ln 2 / 32 + r, |r| <= ln 2 / 64,
// exp(x) = 2^k 2^(j/32) (1 + (e^r - 1)), e^r - 1 to degree 6 (error r^7 / 5040 < 4e-18), ln 2 / 32 in
// two parts.  Below -708 the result is 0 (the true value is under 4e-308); NaN stays NaN (its low
// word, and with it k, is 0).
__device__ __forceinline__ double exp_neg(double x, const double* tab) {
    constexpr double kMagic = 6755399441055744.0;               // 1.5 2^52: rounds to an integer
    constexpr double kInvLn2_32 = 46.166241308446828384;        // 32 / ln 2
    constexpr double kLn2Hi = 0.69314718055994528623 / 32.0;    // ln 2 rounded to double, / 32
    constexpr double kLn2Lo = 2.3190468138462995584e-17 / 32.0;
    const double t = fma(x, kInvLn2_32, kMagic);
    const int k = __double2loint(t);
    const double kf = t - kMagic;
    double r = fma(kf, -kLn2Hi, x);
    r = fma(kf, -kLn2Lo, r);
    double q = fma(r, 1.0 / 720.0, 1.0 / 120.0);
    q = fma(r, q, 1.0 / 24.0);
    q = fma(r, q, 1.0 / 6.0);
    q = fma(r, q, 0.5);
    const double p = fma(r * r, q, r);
    const double b = tab[k & 31];
    const double v = fma(b, p, b);
    const double e = __hiloint2double(__double2hiint(v) + ((k & ~31) << 15), __double2loint(v));
    return x < -708.0 ? 0.0 : e;
}

// D (16 x 8) += A (16 x 4) B (4 x 8).  Lane (g = lane / 4, t = lane % 4) holds A rows g, g + 8 of
// column t, B row t of column g, D rows g (c[0], c[1]) and g + 8 (c[2], c[3]) of columns 2 t, 2 t + 1.
__device__ __forceinline__ void mma_f64(double (&c)[4], double a0, double a1, double b) {
    asm volatile(
        "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
        "{%0,%1,%2,%3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a0), "d"(a1), "d"(b));
}

// kChunks: the lattice takes more than one spot chunk along x or y (U is then summed over steps and
// stays in registers between them).
template <int TY, bool kChunks>
__global__ void __launch_bounds__(kThreads, 2)
fwd_f64_kernel(pbd_field f, const double* __restrict__ w, const double* __restrict__ idd,
               const double* __restrict__ sigma, double* __restrict__ dose, int SC, int ntx,
               int nty, int first_wave) {
    constexpr int MT = TY / 64;        // 16-row pieces per warp: 4 warps along y, 2 along x
    constexpr int kLDY = ld_y(TY);
    extern __shared__ __align__(16) double sm[];
    double* GxT = sm;                  // [i][x]
    double* U = GxT + SC * kLDX;       // [j][x]
    double* GyT = U + SC * kLDX;       // [j][y]
    double* WT = GyT + SC * kLDY;      // [j][i]
    const int LDW = ld_w(SC);
    __shared__ double s_c[kLayerBatch], s_s[kLayerBatch];
    __shared__ double s_tab[32], s_xs[kSCMax], s_ys[kSCMax];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int wy = (warp & 3) * 16 * MT, wx = (warp >> 2) * 32;   // this warp's part of the tile
    // Slices in depth order, the shallow ones, which see the most layers, first; when the blocks
    // fill the SMs less than twice, the second ones in reverse, so that the SMs with the heaviest
    // first block get the lightest second one.
    const int bi = blockIdx.x < first_wave ? blockIdx.x : gridDim.x - 1 - (blockIdx.x - first_wave);
    const int tile = bi % (ntx * nty), z = bi / (ntx * nty);
    const int x0 = (tile % ntx) * kTX, y0 = (tile / ntx) * TY;
    const int nz = f.nz, nsx = f.n_sx, nsy = f.n_sy;
    // The same grid and lattice along x and y, and the tile's columns among its rows: Gx is a part
    // of Gy, read from there (one chunk only, whose spots are then the same as well).
    const bool shared = !kChunks && f.nx == f.ny && f.ox == f.oy && f.dx == f.dy && nsx == nsy &&
                        f.x0 == f.y0 && f.dx_spot == f.dy_spot && x0 >= y0 && x0 + kTX <= y0 + TY;
    const double* gxt = shared ? GyT + (x0 - y0) : GxT;
    const int ldb = shared ? kLDY : kLDX;
    const double cx = 0.5 * (double)(nsx - 1), cy = 0.5 * (double)(nsy - 1);
    const int gx = tid % kTX, gy = tid % TY;     // the column / row whose factors this thread forms
    const double xv = f.ox + (double)(x0 + gx) * f.dx;
    const double yv = f.oy + (double)(y0 + gy) * f.dy;
    if (tid < 32) s_tab[tid] = exp2((double)tid * 0.03125);
    __syncthreads();

    double acc[MT][4][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[m][n][q] = 0.0;

    // The steps: (active layer l, spot chunk j0, spot chunk i0), in order.  The layers' scalars are
    // staged kLayerBatch at a time, reloaded (a block-wide step) at a new batch.
    auto stage_layers = [&](int l) {
        __syncthreads();
        for (int q = tid; q < kLayerBatch && l + q < f.n_layers; q += kThreads) {
            s_c[q] = idd[(size_t)(l + q) * nz + z];
            s_s[q] = sigma[(size_t)(l + q) * nz + z];
        }
        __syncthreads();
    };
    auto next_active = [&](int l) {
        for (; l < f.n_layers; ++l) {
            if (l % kLayerBatch == 0) stage_layers(l);
            if (s_c[l % kLayerBatch] != 0.0) break;
        }
        return l;
    };
    // asynchronous copy of a step's weights into WT; spots past the chunk (to a multiple of 4) are
    // zero-filled
    auto copy_w = [&](int l, int j0, int i0) {
        const int nj = min(SC, nsy - j0), pj = (nj + 3) & ~3;
        const int ni = min(SC, nsx - i0), pi = (ni + 3) & ~3;
        const double* wl = w + ((size_t)l * nsy + j0) * nsx + i0;
        for (int jj = warp; jj < pj; jj += kThreads / 32)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int ii = lane + 32 * h;
                if (ii < pi) {
                    const bool in = jj < nj && ii < ni;
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(
                                     (unsigned)__cvta_generic_to_shared(&WT[jj * LDW + ii])),
                                 "l"(in ? wl + (size_t)jj * nsx + ii : w), "r"(in ? 8 : 0)
                                 : "memory");
                }
            }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    int l = next_active(0), j0 = 0, i0 = 0;
    if (l < f.n_layers) copy_w(l, 0, 0);
    double u[4][4];                    // U rows 16 m + g (+ 8), columns 8 warp + 2 t (+ 1)
    // spot positions of a step's chunks; past their ends any finite one, whose factors meet zero weights
    // and zero rows of U (an infinite one gives NaN where a width's k2 underflows)
    auto stage_spots = [&](int j0, int i0) {
        const int q = tid & 63, n = (tid < 64 ? nsx - i0 : nsy - j0);
        if (tid < 64) s_xs[q] = q < n ? f.x0 + ((double)(i0 + q) - cx) * f.dx_spot : 0.0;
        else if (tid < 128) s_ys[q] = q < n ? f.y0 + ((double)(j0 + q) - cy) * f.dy_spot : 0.0;
        __syncthreads();
    };
    stage_spots(0, 0);
    while (l < f.n_layers) {
        const double s = fmax(s_s[l % kLayerBatch], 1e-9);
        const double k2 = 1.0 / (2.0 * s * s);
        const double nrm = s_c[l % kLayerBatch] * kInv2Pi / (s * s);
        const int nj = min(SC, nsy - j0), pj = (nj + 3) & ~3;
        const int ni = min(SC, nsx - i0), pi = (ni + 3) & ~3;
        // Gx: its buffer was last read before the barrier that ended the previous step's U
        if (!shared) {
#pragma unroll 4
            for (int ii = tid / kTX; ii < pi; ii += kThreads / kTX) {
                const double d = xv - s_xs[ii];
                GxT[ii * kLDX + gx] = exp_neg(-(d * d) * k2, s_tab);
            }
        }
        __syncthreads();               // every warp is done with the previous step's Gy and U
        if (i0 == 0) {
#pragma unroll 4
            for (int jj = tid / TY; jj < pj; jj += kThreads / TY) {
                const double d = yv - s_ys[jj];
                GyT[jj * kLDY + gy] = exp_neg(-(d * d) * k2, s_tab);
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        // U[j, x] += sum_i W[j,i] Gx[x,i]: warp w forms columns 8 w .. 8 w + 7.  Rows past pj (the
        // last 16-row piece) read the last one and are not stored.
        auto stage1 = [&](auto nm) {
            constexpr int NM = decltype(nm)::value;
            const double* wr[2 * NM];
#pragma unroll
            for (int m = 0; m < 2 * NM; ++m) wr[m] = WT + min(8 * m + g, pj - 1) * LDW + t;
            const double* br = gxt + t * ldb + 8 * warp + g;
#pragma unroll 2
            for (int ii = 0; ii < pi; ii += 4) {
                const double b = br[ii * ldb];
#pragma unroll
                for (int m = 0; m < NM; ++m) mma_f64(u[m], wr[2 * m][ii], wr[2 * m + 1][ii], b);
            }
        };
        if (!kChunks || i0 == 0) {
#pragma unroll
            for (int m = 0; m < 4; ++m)
#pragma unroll
                for (int q = 0; q < 4; ++q) u[m][q] = 0.0;
        }
        if (pj > 48) stage1(std::integral_constant<int, 4>{});
        else if (pj > 32) stage1(std::integral_constant<int, 3>{});
        else if (pj > 16) stage1(std::integral_constant<int, 2>{});
        else stage1(std::integral_constant<int, 1>{});
        const bool whole = !kChunks || i0 + SC >= nsx;       // U has every spot i
        if (whole) {
#pragma unroll
            for (int m = 0; m < 4; ++m)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int j = 16 * m + 8 * h + g;
                    const double sc = j < nj ? nrm : 0.0;        // an infinite nrm leaves the padding 0
                    if (j < pj)
                        *reinterpret_cast<double2*>(&U[j * kLDX + 8 * warp + 2 * t]) =
                            make_double2(sc * u[m][2 * h], sc * u[m][2 * h + 1]);
                }
        }
        __syncthreads();
        // the next step's weights come in while this one's products run
        if (kChunks) {
            i0 += SC;
            if (whole) { i0 = 0; j0 += SC; }
            if (j0 >= nsy) j0 = 0;
        }
        if (!kChunks || (i0 == 0 && j0 == 0)) l = next_active(l + 1);
        if (l < f.n_layers) {
            copy_w(l, j0, i0);
            if (kChunks) stage_spots(j0, i0);
        }
        if (!whole) continue;
        // D[y, x] += sum_j Gy[y,j] U[j,x]
#pragma unroll 2
        for (int jj = 0; jj < pj; jj += 4) {
            const double* gr = &GyT[(jj + t) * kLDY + wy + g];
            const double* ur = &U[(jj + t) * kLDX + wx + g];
            double a[MT][2], b[4];
#pragma unroll
            for (int m = 0; m < MT; ++m) { a[m][0] = gr[16 * m]; a[m][1] = gr[16 * m + 8]; }
#pragma unroll
            for (int n = 0; n < 4; ++n) b[n] = ur[8 * n];
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int n = 0; n < 4; ++n) mma_f64(acc[m][n], a[m][0], a[m][1], b[n]);
        }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int y = y0 + wy + 16 * m + 8 * h + g;
            if (y >= f.ny) continue;
            double* row = dose + ((size_t)z * f.ny + y) * f.nx;
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int x = x0 + wx + 8 * n + 2 * t + q;
                    if (x < f.nx) row[x] = acc[m][n][2 * h + q];
                }
        }
}

template <int TY, bool kChunks>
int launch_ty(const pbd_field* f, const double* w, const double* idd, const double* sigma,
              double* dose, cudaStream_t s) {
    // one opt-in size per kernel (the largest chunk's), the launch's own size per lattice
    int set = 0;
    PBD_TRY(smem_optin((const void*)fwd_f64_kernel<TY, kChunks>,
                       (int)(smem_doubles(TY, kSCMax) * sizeof(double)), 0, &set));
    const int sc = min(kSCMax, (max(f->n_sx, f->n_sy) + 3) / 4 * 4);
    const int ntx = (f->nx + kTX - 1) / kTX, nty = (f->ny + TY - 1) / TY;
    const long long blocks = (long long)ntx * nty * f->nz;
    if (blocks > 2147483647LL) return PBD_ERR_UNSUPPORTED;
    const int sms = num_sms();
    const int first = blocks <= 2LL * sms ? min((int)blocks, sms) : (int)blocks;
    fwd_f64_kernel<TY, kChunks><<<(unsigned)blocks, kThreads, smem_doubles(TY, sc) * sizeof(double), s>>>(
        *f, w, idd, sigma, dose, sc, ntx, nty, first);
    PBD_LAUNCH_CHECK();
    return PBD_OK;
}

}  // namespace

int launch_forward_f64(const pbd_field* f, const double* w, const double* idd,
                       const double* sigma, double* dose, cudaStream_t s) {
    if (f->nz > 65535) return PBD_ERR_UNSUPPORTED;
    // 128-row tiles, unless 64-row ones leave out a quarter or more of the padded rows (grids of
    // 1-64 and 129-192 rows): 64 rows of the 41 x 41 x 40 field take 246 us in 64-row tiles, as
    // many as 128 rows take in 128-row ones less a quarter
    const int p128 = (f->ny + 127) / 128 * 128, p64 = (f->ny + 63) / 64 * 64;
    prof_mark(kProfFwd, 0, s);
    const bool small = 4 * p64 <= 3 * p128, chunks = f->n_sx > kSCMax || f->n_sy > kSCMax;
    const auto launch = small ? (chunks ? launch_ty<64, true> : launch_ty<64, false>)
                              : (chunks ? launch_ty<128, true> : launch_ty<128, false>);
    PBD_TRY(launch(f, w, idd, sigma, dose, s));
    prof_mark(kProfFwd, 1, s);
    return PBD_OK;
}

}  // namespace pbd
