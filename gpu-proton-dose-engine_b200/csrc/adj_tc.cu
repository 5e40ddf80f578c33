// adj_tc.cu -- adjoint of the separable dose on the tensor cores (tcgen05), warp-specialised
// and software-pipelined across (layer, slice) pairs.
//
// Same mathematics as adj_simt.cu.  With G = dL/dD[z] and unnormalised Gaussians of width
// s = sigma_l(z), for every active (layer l, slice z) and 128-column tile of the slice:
//
//   stage 1   Y[m, x] = sum_y A[m, y] G[y, x]        A = [Gy | s Gy']^T, m = 2 j: j, m = 2 j + 1: j'
//             M = 128 (m), N <= 128 (x), K <= 256 (y); A generated into TMEM, G^T in smem
//   stage 2   Q[m, n] = sum_x Y[m, x] B[n, x]        B = [Gx | s Gx'], n = 2 i: i, n = 2 i + 1: i'
//             M = 128 (m), N = 2 N1 (n), K <= 128 (x); Y split back into TMEM, B in smem
//
// P = Q[j, i] gives dL/dW_l += IDD P / (2 pi s^2) and dL/dIDD = <P, W> / (2 pi s^2);
// Q[j, i'] + Q[j', i] gives dL/dsigma = IDD <., W> / (2 pi s^3) (G' = dG/ds = G (d^2/s^2 - 1) / s).
// The Gaussian factors are regenerated per pair; nothing Gaussian is stored in HBM.
//
// Precision.  Every split or TF32 mode runs split FP16: a = hi + lo, hi = fp16(a), lo = fp16(a - hi),
// three products, FP32 accumulation; the BF16 mode runs plain BF16.  Operands are scaled by powers
// of two into FP16's range, all exact: A and B by 2^14 (|s G'| <= 1), each unit's slice G so that
// its largest value lands in [2^14, 2^15), and Y by 2^-(14 + ky), 2^ky >= min(1 + sqrt(2 pi) s / dy, 256),
// the bound on sum_y A.  Distances are formed in voxel units from the spot's integer and
// fractional voxel position, so that a Gaussian's exponent is good to FP32 rounding of its own
// size (from y0 + c dy - ys in FP32 the cancellation cost 1e-6 of it); the cross products go to the
// accumulators first and the large ones last, since the tensor core truncates.
//
// Band.  Past 8 s a factor is below 2^-46 and, scaled, exactly zero in FP16; the 16-voxel groups no
// spot reaches are left out of both stages (N and K), of the generation and of Y's split, and a
// warp whose own spots do not reach a group stores zeros for it.  (10 cm of spots on a 25.6 cm
// grid: 6 of 8 groups, and about half of each warp's own.)
//
// CTA = 8 math warps, a scheduler warp, two MMA warps (one per stage), a weight-copy warp; one
// CTA per SM.
//  * Scheduler warp: units (slice z, column tile, chunk of <= C active layers) from an atomic
//    counter in z-major order; one step per active layer and 128-row tile of the slice (one tile up to
//    128 rows, two up to 256) into a 4-slot ring (full / empty mbarriers).
//  * Weight warp: each pair's W_l into one of two shared-memory buffers, rows of N1 + 4 floats.
//  * Math warps, per pair n, without block barriers:
//      at a unit's first step: G^T of the slice, scaled and split, into smem (the previous unit's
//          last stage 1 is complete: it was waited for before this step)
//      G   A = [Gy | s Gy']^T -> TMEM A[step & 1] (tcgen05.st); arrive on ops1.  A lane owns a row
//          and evaluates its own exponentials, two columns per packed FP32 instruction
//      DR  pair n-1's Q from TMEM: P = Q[j, i] / (2 pi s^2) into the (layer, slice) slot, and the
//          dot products <P, W> and <S, W>, S = Q[j, i'] + Q[j', i], summed over the warp
//      (second row tile: G into the other A buffer; stage 1 accumulates)
//      B   [Gx | s Gx'] -> smem (read by stage 2 only, whose previous use DR waited for)
//      E1  Y of pair n from TMEM, split, back into TMEM A; arrive on ops2
//  * MMA warp 1: stage 1 after ops1 (A from TMEM, "TS" form), commit to mma1.
//    MMA warp 2: stage 2 after ops2 (A = split Y from TMEM), commit to mma2.
//  Stage 2 of pair n-1 runs under G of pair n; stage 1 of pair n under DR and B.
//
// What bounds it: the math warps' phases one after another (G 1250 cycles a pair, DR 1070, E1 830, B
// 510, waits for the MMAs 800 of 5500 on the 128^3 / 41 x 41 x 40 field), not the tensor pipe.
// Straight-line code is fetched anew for every pair at some 10 cycles an instruction, so every
// phase is a rolled loop over 16-column groups: unrolled, with fewer instructions executed, the same
// phases took 7800 cycles.  The adjoint of that field: 90 us before (split BF16 with two columns per
// 27 instructions, unrolled, whole tiles, weights loaded by the math warps), 71 us now, and 20 of its
// gradients' jobs in four fields 1413 -> 990 us; a 200 x 200 x 256 field's (which ran in FP32 on the
// CUDA cores) 12.4 -> 0.83 ms.
//
// dL/dW_l = sum over active slices of IDD * slot P in slice order, and the sums of the warps'
// dot-product partials (dL/dIDD, dL/dsigma), are formed by one follow-up kernel in a fixed
// order (deterministic).  Every wait is bounded (2 s of %globaltimer, or a test limit); a warp
// whose wait runs out sets the error word and leaves, the others' waits then run out in
// turn, and the finalize pass turns the gradients into NaN.
// Lattices up to 64 x 64 spots, slices of at most 256 rows; any number of column tiles.
#include <algorithm>
#include <cuda_fp16.h>
#include <math.h>

#include "pbd_internal.cuh"
#include "tc_common.cuh"

namespace pbd {
namespace {
using namespace tcc;

constexpr int kMathWarps = 8;
constexpr int kMath = 32 * kMathWarps;     // 256 math threads: warpgroups 0 and 1
constexpr int kSchedWarp = kMathWarps;     // warpgroup 2: scheduler, two MMA warps, weight copies
constexpr int kS1Warp = kMathWarps + 1;
constexpr int kWWarp = kMathWarps + 3;
constexpr int kThreads = kMath + 128;
constexpr int kRing = 4;      // step slots (the largest two-tile shape leaves 1 KB of static shared memory)
constexpr uint32_t kCols = 512;
// Register split (setmaxnreg) as in the forward: 8 * 32 * 208 + 4 * 32 * 80 <= 384 * 168.
constexpr int kMathRegs = 208, kCtrlRegs = 80;
constexpr int kLaunchRegsNeeded = (kMath * kMathRegs + 128 * kCtrlRegs + kThreads - 1) / kThreads;
// TMEM columns: A[0] [0,128), A[1] [128,256) (16-bit pairs: hi [0,64), lo [64,128) of each),
// Y [256,384), Q [384, 384 + 2 N1)
constexpr uint32_t kColA = 0, kColY = 256, kColQ = 384;
constexpr uint32_t kLoOff = 64;
constexpr float kOpScale = 16384.0f;       // 2^14, the Gaussians' scale
constexpr int kMaxRowTiles = 2;            // 128-row tiles of a slice
constexpr float kBand = 8.0f;              // Gaussians end at 8 s (exp(-32) = 2^-46)

enum : int { kFirst = 1, kEnd = 4, kPairFirst = 8, kPairEnd = 16 };

struct Step {
    int job, z, l, flags;
    int xt, yt, pair;               // column tile, row tile; pair index of this CTA
    int ya, yb, xa, xb;             // 16-voxel groups of the row tile (K of stage 1) and of the column
                                    // tile (N of stage 1, K of stage 2) within the band
    float nay, nax;                 // -log2(e) dy^2 / (2 s^2), the same for dx
    float by, bx;                   // 2^14 dy^2 / s^2, 2^14 dx^2 / s^2
    float ry, rx;                   // the band in voxels
    float nrm, inv_s, fy;           // 1/(2 pi s^2), 1/s, Y's scale 2^-(14 + ky)
    int ky;
    int nsx, nsy;                   // the job's lattice
    float *slot, *dot_p, *dot_s;    // the pair's P slot and its warps' <P, W> and <S, W> partials
};

struct Params {
    const JobDev* jobs;
    int n_jobs, chunk, cmax, n_units;
    int xtmax;           // column tiles of the widest job
    int* counter;        // [0] unit counter
    int* err;            // error word: set when a bounded wait ran out
    unsigned long long wait_ns;   // limit of every bounded wait
    int hold;            // test of the timeout path: the scheduler publishes no step
    int N1;              // x-lattice padded to 16
    int tiles;           // 128-row tiles whose G^T the shared memory holds (1 or 2)
    int stage;           // each unit's dL/dD slice arrives in a staging buffer: 1 by bulk copy (every job's
                         //    slice 16-byte aligned, nx ny % 4 == 0), 2 by 4-byte cp.async (any other), 0:
                         //    read from global memory (several tiles).  Read from global memory as well,
                         //    a slice of the second kind took 10 us a unit where no other step hid it:
                         //    5 layers of 53 x 53 x 110 in a medium 76 us against 40, and
                         //    117 x 93 x 121 with 33 layers' adjoint 93 us against 86
    uint32_t o_b2, o_w, w_bytes, o_stage;   // shared-memory offsets: B, weights (two buffers), staging
    float give_back;     // 2^-24: the split mode's results are raised by what truncation takes; else 0
    int sym;             // 1: every job is one tile and symmetric in x and y (grid, lattice, origins),
                         //    so B's rows equal the rows G evaluates for A
    int adapt;           // 1 (one job, no explicit schedule): every CTA counts the active pairs T
                         //    and uses units of ceil(T / grid) + 1 layers (chunk, cmax, n_units
                         //    then describe that unit size)
};

// The adjoint's unit decomposition in force (P's, or the one the CTA derived).
struct Units {
    int chunk, cmax, n_units;
};

// mbarriers of a CTA
struct Bars {
    uint64_t *full, *empty;                       // step ring
    uint64_t *ops1, *ops2, *mma1, *mma2;          // operands ready, products done
    uint64_t *sfull, *sfree;                      // staging buffer
    uint64_t *wfull, *wfree;                      // weight buffers [2]
    uint64_t *gmax;                               // the unit's largest |G|: every warp's share is in
};

// Two adjacent K elements as packed 16-bit operands (element 0 in the low half): FP16 hi and
// lo = fp16 of the remainders, or plain BF16.
template <bool kSplit>
__device__ __forceinline__ void split2(f32x2 v, uint32_t& hi, uint32_t& lo) {
    float a, b;
    upk(v, a, b);
    if (kSplit) {
        const __half2 h = __floats2half2_rn(a, b);
        hi = *reinterpret_cast<const uint32_t*>(&h);
        const float2 hf = __half22float2(h);
        float ra, rb;
        upk(fma2(pk(hf.x, hf.y), pk(-1.0f, -1.0f), v), ra, rb);
        const __half2 l = __floats2half2_rn(ra, rb);
        lo = *reinterpret_cast<const uint32_t*>(&l);
    } else {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        hi = *reinterpret_cast<const uint32_t*>(&h);
        lo = 0u;
    }
}

// PAIRS x 2 operand values v = e (A + B dd), e = 2^(dd na), dd = (n + q + f)^2, q = 0, 1, ...: the
// columns of a Gaussian (B = 0) or of s times its derivative (A = -2^14, B = 2^14 d^2 / s^2), n
// the first column's integer distance in voxels, f the fractional part.
template <bool kSplit, int PAIRS>
__device__ __forceinline__ void gauss_row(float n, f32x2 f, f32x2 na, f32x2 A, f32x2 B,
                                          uint32_t* hi, uint32_t* lo) {
    f32x2 n2 = pk(n, n + 1.0f);
    const f32x2 two = pk(2.0f, 2.0f);
#pragma unroll
    for (int k = 0; k < PAIRS; ++k) {
        const f32x2 u = add2(n2, f);
        const f32x2 dd = mul2(u, u);
        float a0, a1;
        upk(mul2(dd, na), a0, a1);
        const f32x2 e = pk(ex2_approx(a0), ex2_approx(a1));
        split2<kSplit>(mul2(e, fma2(dd, B, A)), hi[k], lo[k]);
        n2 = add2(n2, two);
    }
}

// ------------------------------------------------------------------------------------------
// Scheduler warp: units (z, column tile, chunk) -> one step per active layer and row tile.
// ------------------------------------------------------------------------------------------
// 16-voxel groups [a, b) of tile t (128 voxels) of an axis of n voxels that the band around the
// lattice (first and last spot at voxel positions p0, p1, +- r) reaches; at most 8, none: a = b.
__device__ __forceinline__ void band_groups(float p0, float p1, float r, int n, int t, int& a, int& b) {
    const float lo = fmaxf(p0 - r - 128.0f * (float)t, 0.0f);
    const float hi = fminf(p1 + r - 128.0f * (float)t, (float)(min(n - 128 * t, 128) - 1));
    if (!(hi >= lo)) {
        a = b = 0;
        return;
    }
    a = (int)lo >> 4;
    b = ((int)hi >> 4) + 1;
}

__device__ __forceinline__ void scheduler_warp(const Params& P, const Units U, Step* ring,
                                               const Bars& B, uint8_t* smem) {
    const int lane = threadIdx.x & 31;
    const unsigned FULL = 0xffffffffu;
    int k = 0, nu = 0;       // ring pushes; units whose slice was copied into the staging buffer
    int pair = 0;
    bool ok = true;
    auto push = [&](int src, const Step& st) -> bool {
        const int slot = k % kRing, n = k / kRing;
        const bool w = wait_bar(&B.empty[slot], (uint32_t)((n & 1) ^ 1), P.wait_ns);
        if (!__all_sync(FULL, w)) return false;
        if (lane == src) {
            ring[slot] = st;
            tc::mbar_arrive(&B.full[slot]);
        }
        __syncwarp();
        ++k;
        return true;
    };
    // timeout-path test: publish nothing, so that every consumer's first wait runs out
    if (P.hold) return;
    // each CTA starts with unit blockIdx.x; the counter hands out those past the first grid-full
    auto next_unit = [&]() {
        int u = 0;
        if (lane == 0) u = (int)gridDim.x + atomicAdd(P.counter, 1);
        return __shfl_sync(FULL, u, 0);
    };
    for (int u = blockIdx.x; u < U.n_units; u = next_unit()) {
        int v = u;
        const int job = v % P.n_jobs; v /= P.n_jobs;
        const int xt = v % P.xtmax; v /= P.xtmax;
        const int c = v % U.cmax;
        const int z = v / U.cmax;
        const JobDev& J = P.jobs[job];
        const int nz = J.nz, nl = J.nl, nty = J.nty;
        if (z >= nz || xt >= J.ntx) continue;
        const double* idd = J.idd;
        // the unit's depth doses and widths, every load in flight together (kept for <= 64 layers)
        double ivg[2], svg[2];
        auto load = [&](int b, double& iv, double& sv) {
            const int l = b + lane;
            iv = l < nl ? __ldg(idd + (size_t)l * nz + z) : 0.0;
            sv = l < nl ? __ldg(J.sigma + (size_t)l * nz + z) : 1.0;
        };
        load(0, ivg[0], svg[0]);
        load(32, ivg[1], svg[1]);
        auto group = [&](int b, double& iv, double& sv) {
            if (b < 64) {
                iv = b == 0 ? ivg[0] : ivg[1];
                sv = b == 0 ? svg[0] : svg[1];
            } else {
                load(b, iv, sv);
            }
        };
        int tot = 0;
        for (int b = 0; b < nl; b += 32) {
            double iv, sv;
            group(b, iv, sv);
            tot += __popc(__ballot_sync(FULL, iv != 0.0));
        }
        const int r0 = c * U.chunk;
        if (r0 >= tot) continue;   // no chunk c here (slices no layer reaches carry no gradient)
        const int r1 = min(tot, r0 + U.chunk);
        if (P.stage) {
            // the unit's dL/dD slice into the staging buffer, once the math warps have converted
            // the previous unit's copy
            bool w = true;
            if (nu > 0) w = wait_bar(B.sfree, (uint32_t)((nu - 1) & 1), P.wait_ns);
            if (!__all_sync(FULL, w)) { ok = false; break; }
            const uint32_t dst = tc::smem_u32(smem) + P.o_stage;
            if (P.stage == 2) {
                // a slice without 16-byte alignment: coalesced 4-byte copies by all lanes, each of
                // which arrives when its own have landed
                const float* src = J.grad_dose + (size_t)z * J.ny * J.nx;
                const int n = J.nx * J.ny;
#pragma unroll 8
                for (int e = lane; e < n; e += 32)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 4u * (uint32_t)e), "l"(src + e)
                                 : "memory");
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc::smem_u32(B.sfull))
                             : "memory");
            } else if (lane == 0) {
                const uint32_t bytes = (uint32_t)J.nx * (uint32_t)J.ny * 4u;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                                 tc::smem_u32(B.sfull)), "r"(bytes)
                             : "memory");
                asm volatile(
                    "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
                    "[%3];" ::"r"(dst),
                    "l"(J.grad_dose + (size_t)z * J.ny * J.nx), "r"(bytes), "r"(tc::smem_u32(B.sfull))
                    : "memory");
            }
            __syncwarp();
            ++nu;
        }
        // the lattice's first and last spots in voxels (FP32: they only choose the band's groups)
        const float idy = (float)(1.0 / J.dy), idx = (float)(1.0 / J.dx);
        const float hy = 0.5f * (float)(J.nsy - 1) * (float)J.dsy * idy;
        const float hx = 0.5f * (float)(J.nsx - 1) * (float)J.dsx * idx;
        const float cy = (float)(J.sy0 - J.oy) * idy, cx = (float)(J.sx0 - J.ox) * idx;
        const float py0 = cy - hy, py1 = cy + hy, px0 = cx - hx, px1 = cx + hx;
        int rank = 0;
        for (int b = 0; b < nl && rank < r1 && ok; b += 32) {
            const int l = b + lane;
            double iv, sv;
            group(b, iv, sv);
            const bool a = iv != 0.0;
            const unsigned bal = __ballot_sync(FULL, a);
            const int my = rank + __popc(bal & ((1u << lane) - 1u));
            const bool mine = a && my >= r0 && my < r1;
            Step st{};
            int ya[kMaxRowTiles] = {0, 0}, yb[kMaxRowTiles] = {0, 0};
            if (mine) {
                const double s = fmax(sv, 1e-9);
                st.job = job; st.z = z; st.l = l; st.xt = xt;
                st.nsx = J.nsx; st.nsy = J.nsy;
                const size_t per = (size_t)J.nsy * ((J.nsx + 15) / 16 * 16);
                const size_t pr = ((size_t)l * nz + z) * J.ntx + xt, np = (size_t)nl * nz * J.ntx;
                st.slot = J.partial + pr * per;
                st.dot_p = J.partial + np * per + pr * kMathWarps;
                st.dot_s = st.dot_p + np * kMathWarps;
                const double is = 1.0 / s, qy = J.dy * is, qx = J.dx * is;
                const float ivy = (float)s * idy, ivx = (float)s * idx;       // s in voxels
                st.nay = (float)(-0.5 * kLog2e * qy * qy);
                st.nax = (float)(-0.5 * kLog2e * qx * qx);
                st.by = (float)((double)kOpScale * qy * qy);
                st.bx = (float)((double)kOpScale * qx * qx);
                const float ry = kBand * ivy, rx = kBand * ivx;
                st.ry = ry; st.rx = rx;
                st.inv_s = (float)is;
                int e = 0;
                // sum_y A < 1 + sqrt(2 pi) s / dy, and no more than the 256 rows, < 2^e
                (void)frexpf(fminf(1.001f + 2.50663f * ivy, 256.5f), &e);
                st.ky = e;
                st.fy = __int_as_float((127 - 14 - st.ky) << 23);
                band_groups(px0, px1, rx, J.nx, xt, st.xa, st.xb);
#pragma unroll
                for (int t = 0; t < kMaxRowTiles; ++t)
                    if (t < nty) band_groups(py0, py1, ry, J.ny, t, ya[t], yb[t]);
                // a band that misses the tile altogether: one group, of zeros
                if (st.xa >= st.xb) { st.xa = 0; st.xb = 1; }
                if (ya[0] >= yb[0] && ya[1] >= yb[1]) { ya[0] = 0; yb[0] = 1; }
                // The tensor core truncates its FP32 accumulators: a result loses up to 1.2 x 2^-24 of itself
                // per k-step (16-voxel group of the band) that matters to it, as many as the width spans.  Lost
                // in units of 2^-24 on one tile, by width in voxels: a dL/dD of one sign 4 (2), 10 (5), 17 (10),
                // 20 (14), 15 (100); of random sign 3, 4, 4, 4, 3; a single voxel 2 at any; over two row tiles one
                // sign 10 (5), 16 (10), 28 (20), 33 (100).  Half-way between, no further than the band's own
                // groups, is given back: 128 voxels or fewer stay within 1.2e-6 of the largest dL/dW at any
                // width (0.6e-6 to 6 voxels), two row tiles within 2.1e-6.  Without it 1.8e-6 and 3.2e-6.
                const float gy = (float)(yb[0] - ya[0] + yb[1] - ya[1]), gx = (float)(st.xb - st.xa);
                const float lost = 2.0f + 0.6f * (fminf(ivy, 1.25f * gy) + fminf(ivx, 1.25f * gx));
                st.nrm = (float)(kInv2Pi * is * is * (1.0 + (double)(lost * P.give_back)));
            }
            unsigned emit = __ballot_sync(FULL, mine);
            while (emit && ok) {
                const int src = __ffs(emit) - 1;
                emit &= emit - 1u;
                const bool h0 = __shfl_sync(FULL, yb[0] > ya[0] ? 1 : 0, src) != 0;
                const bool h1 = __shfl_sync(FULL, yb[1] > ya[1] ? 1 : 0, src) != 0;
                const int first = __shfl_sync(FULL, my == r0 ? 1 : 0, src) ? kFirst : 0;
                st.pair = pair;
                if (h0) {
                    st.yt = 0; st.ya = ya[0]; st.yb = yb[0];
                    st.flags = first | kPairFirst | (h1 ? 0 : kPairEnd);
                    ok = push(src, st);
                }
                if (h1 && ok) {
                    st.yt = 1; st.ya = ya[1]; st.yb = yb[1];
                    st.flags = (h0 ? 0 : first | kPairFirst) | kPairEnd;
                    ok = push(src, st);
                }
                ++pair;
            }
            rank += __popc(bal);
        }
        if (!ok) break;
    }
    if (ok) {
        Step st{};
        st.flags = kEnd;
        (void)push(0, st);
    }
    // the last staging copy lands before the block exits
    if (nu > 0) (void)wait_bar(B.sfull, (uint32_t)((nu - 1) & 1), P.wait_ns);
    if (!ok && lane == 0) atomicExch(P.err, 1);
}

// ------------------------------------------------------------------------------------------
// Weight warp: W_l of each pair into buffer pair & 1, rows of N1 + 4 floats (16-byte aligned, and
// eight rows' 16-byte pieces in different banks), columns past the lattice zero.
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ void weight_warp(const Params& P, const Step* ring, const Bars& B,
                                            uint8_t* smem) {
    const int lane = threadIdx.x & 31;
    const int ldw = P.N1 + 4;
    int k = 0;
    bool ok = true;
    for (;;) {
        const int slot = k % kRing;
        ok = wait_bar(&B.full[slot], (uint32_t)((k / kRing) & 1), P.wait_ns);
        const int flags = ring[slot].flags, job = ring[slot].job, l = ring[slot].l, p = ring[slot].pair;
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&B.empty[slot]);
        ++k;
        if (!__all_sync(0xffffffffu, ok)) break;
        if (flags & kEnd) break;
        if (!(flags & kPairFirst)) continue;
        if (p >= 2) ok = wait_bar(&B.wfree[p & 1], (uint32_t)(((p >> 1) - 1) & 1), P.wait_ns);
        if (!__all_sync(0xffffffffu, ok)) break;
        const JobDev& J = P.jobs[job];
        const int nsx = J.nsx, nsy = J.nsy, n1 = P.N1;
        const float* w = J.w + (size_t)l * nsy * nsx;
        float* dst = reinterpret_cast<float*>(smem + P.o_w + (uint32_t)(p & 1) * P.w_bytes);
        constexpr int kRows = 12;
        for (int j0 = 0; j0 < nsy; j0 += kRows) {
            float v[kRows][2];
#pragma unroll
            for (int r = 0; r < kRows; ++r)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int j = j0 + r, i = lane + 32 * h;
                    v[r][h] = (j < nsy && i < nsx) ? __ldg(w + (size_t)j * nsx + i) : 0.f;
                }
#pragma unroll
            for (int r = 0; r < kRows; ++r)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int j = j0 + r, i = lane + 32 * h;
                    if (j < nsy && i < n1) dst[j * ldw + i] = v[r][h];
                }
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&B.wfull[p & 1]);
    }
    if (!ok && lane == 0) atomicExch(P.err, 1);
}

// ------------------------------------------------------------------------------------------
// MMA warps.  stage 1: Y = A[b] (TMEM, K = y) x G^T (smem rows x); stage 2: Q = Y split
// (TMEM A[b], K = x) x B^T (smem rows n).  The issue loops are rolled, with descriptors that are
// incremented: unrolled, the straight-line code of both warps is fetched anew for every pair
// (some 190 cycles an MMA, against 64 of the tensor core for N = 128).
// ------------------------------------------------------------------------------------------
template <bool kSplit>
__device__ __forceinline__ void issue_stage(uint32_t d, uint32_t a, uint32_t bh, uint32_t lo_off,
                                            uint32_t plane, uint32_t idesc, int ka, int kb,
                                            uint32_t acc) {
    const uint64_t inc = plane >> 3;                 // two planes, in 16-byte units
    const uint64_t dh0 = tc::smem_desc(bh, plane, 128) + (uint64_t)ka * inc;
    uint64_t dh = dh0;
    uint32_t ac = a + (uint32_t)ka * 8u;
    if (kSplit) {
        uint64_t dl = dh0 + (lo_off >> 4);
#pragma unroll 1
        for (int st = ka; st < kb; ++st) {
            tc::mma_bf16_ts(d, ac, dl, idesc, acc);
            tc::mma_bf16_ts(d, ac + kLoOff, dh, idesc, 1u);
            acc = 1u;
            dh += inc; dl += inc; ac += 8u;
        }
        dh = dh0;
        ac = a + (uint32_t)ka * 8u;
    }
#pragma unroll 1
    for (int st = ka; st < kb; ++st) {
        tc::mma_bf16_ts(d, ac, dh, idesc, acc);
        acc = 1u;
        dh += inc; ac += 8u;
    }
}

template <bool kSplit>
__device__ __forceinline__ void mma_warp(const Params& P, uint32_t sbase, uint32_t tb, int stage,
                                         const Step* ring, const Bars& B) {
    constexpr uint32_t kGt = 128u * 128u * 2u;      // one row tile's hi (or lo) half of G^T
    const int lane = threadIdx.x & 31;
    uint64_t* ops = stage == 1 ? B.ops1 : B.ops2;
    uint64_t* done = stage == 1 ? B.mma1 : B.mma2;
    const uint32_t R2 = 2u * (uint32_t)P.N1;
    const uint32_t b2_lo = kSplit ? R2 * 128u * 2u : 0u;
    const uint32_t fmt = kSplit ? 0u : 1u;
    const uint32_t idesc2 = tc::instr_desc(128, (int)R2, fmt);
    int k = 0, n = 0, steps = 0;
    bool ok = true;
    for (;;) {
        const int slot = k % kRing;
        ok = wait_bar(&B.full[slot], (uint32_t)((k / kRing) & 1), P.wait_ns);
        const Step& st = ring[slot];
        const int flags = st.flags, ya = st.ya, yb = st.yb, xa = st.xa, xb = st.xb, yt = st.yt;
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&B.empty[slot]);
        ++k;
        if (!__all_sync(0xffffffffu, ok)) break;
        if (flags & kEnd) break;
        const uint32_t a = tb + kColA + (uint32_t)(steps & 1) * 128u;
        ++steps;
        if (stage == 2 && !(flags & kPairEnd)) continue;
        ok = wait_bar(ops, (uint32_t)(n & 1), P.wait_ns);
        if (!__all_sync(0xffffffffu, ok)) break;
        tc::fence_after_sync();
        if (lane == 0) {
            if (stage == 1) {
                // columns [16 xa, 16 xb): B rows from 16 xa, D columns from 16 xa
                const uint32_t gt = sbase + (uint32_t)yt * (kSplit ? 2u : 1u) * kGt + (uint32_t)xa * 256u;
                issue_stage<kSplit>(tb + kColY + (uint32_t)(16 * xa), a, gt, kGt,
                                    128u * 16u, tc::instr_desc(128, 16 * (xb - xa), fmt), ya, yb,
                                    (flags & kPairFirst) ? 0u : 1u);
            } else {
                issue_stage<kSplit>(tb + kColQ, a, sbase + P.o_b2,
                                    b2_lo, R2 * 16u, idesc2, xa, xb, 0u);
            }
            tc::commit(done);
        }
        __syncwarp();
        ++n;
    }
    if (!ok && lane == 0) atomicExch(P.err, 1);
    if (n > 0) (void)wait_bar(done, (uint32_t)((n - 1) & 1), P.wait_ns);
}

// ------------------------------------------------------------------------------------------
// DR: a pair's Q (TMEM columns from tq: Q[., i] at 2 i, Q[., i'] at 2 i + 1) -> the pair's P slot and
// this warp's share of the pair's two dot products.
//  * Slot layout: P[j][i] = Q[j, i] pow2 nrm, rows of n1 = nsx rounded up to 16 floats (columns i >= nsx
//    hold 0), so that a j lane writes its 8 columns as two 16-byte stores.
//  * A thread's columns: 8-column chunks c0 = 8 half + 16 t, so that both halves of a lane
//    quadrant drain the same number of chunks.
//  * Every lane sums a0 = sum Q[m, i] W[j, i] and a1 = sum Q[m, i'] W[j, i]: the j lane's a0 is its <P, W>,
//    its a1 and the j' lane's a0 are their <S, W> (the j' lane's a1 is not used).  Rows past the
//    lattice and columns past it hold zeros (zero operand rows).  The follow-up kernel adds the
//    eight warps' partials in warp order.
// ------------------------------------------------------------------------------------------
struct Prev {
    int nsx, nsy, pair;
    float pow2, nrm, inv_s;   // Q -> P: the operands' power of two, taken back first, then 1 / (2 pi s^2); 1 / s
    float *slot, *dot_p, *dot_s;
};

__device__ __forceinline__ void drain_q(const Params& P, const Prev& pr, uint32_t tq, int half,
                                        int jrow, bool deriv, int warp, int lane,
                                        const float* wbuf) {
    const int pnsy = pr.nsy;
    const int n1 = (pr.nsx + 15) / 16 * 16;
    const bool row_ok = jrow < pnsy;
    const int jr = row_ok ? jrow : pnsy - 1;
    float* slot_row = pr.slot + jr * n1;
    const float* wrow = wbuf + jr * (P.N1 + 4);
    float a0 = 0.f, a1 = 0.f;
    // a warp whose 32 rows are all padding (its first row 16 sp >= nsy) owns no entry: it skips
    // the TMEM loads and stores zero partials
    const bool pad = __shfl_sync(0xffffffffu, jrow, 0) >= pnsy;
    const f32x2 p2 = pk(pr.pow2, pr.pow2);
    if (!pad) {
#pragma unroll 1
        for (int c = 8 * half; c < n1; c += 16) {
            uint32_t r[16];
            tc::tmem_ld16(tq + (uint32_t)(2 * c), r);
            const float4 w0 = *reinterpret_cast<const float4*>(wrow + c);
            const float4 w1 = *reinterpret_cast<const float4*>(wrow + c + 4);
            const float wv[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
            tc::tmem_wait_ld();
            float pv[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                float vi, vd;          // the power of two comes off before W goes on: Q times W may overflow
                upk(mul2(pk(__uint_as_float(r[2 * q]), __uint_as_float(r[2 * q + 1])), p2), vi, vd);
                a0 = fmaf(vi, wv[q], a0);
                a1 = fmaf(vd, wv[q], a1);
                pv[q] = pr.nrm * vi;
            }
            if (!deriv && row_ok) {
                float4* o = reinterpret_cast<float4*>(slot_row + c);
                o[0] = make_float4(pv[0], pv[1], pv[2], pv[3]);
                o[1] = make_float4(pv[4], pv[5], pv[6], pv[7]);
            }
        }
    }
    // even lanes carry <P, W>, odd lanes <S, W> (their own and their even neighbour's)
    const float other = __shfl_xor_sync(0xffffffffu, a1, 1);
    float v = deriv ? a0 + other : a0;
#pragma unroll
    for (int o = 16; o > 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) pr.dot_p[warp] = pr.nrm * v;
    if (lane == 1) pr.dot_s[warp] = pr.nrm * pr.inv_s * v;
}

// Symmetric fields: B's rows from A's (this lane's row m, read back from TMEM K chunk by K chunk;
// columns outside the step's range are read but not stored).  Rows j >= N1 have no place in B.
template <bool kSplit>
__device__ __forceinline__ void store_b_sym(const Params& P, uint8_t* smem, uint32_t a, const Step& cur,
                                            int half, int m, int jrow) {
    const uint32_t planeR2 = 2u * (uint32_t)P.N1 * 16u;
    const uint32_t b2_lo = kSplit ? 2u * (uint32_t)P.N1 * 128u * 2u : 0u;
    const uint32_t col = a + (uint32_t)(32 * half);
    const int ga = max(cur.xa - 4 * half, 0), gb = min(cur.xb - 4 * half, 4);
    uint8_t* d = smem + P.o_b2 + (uint32_t)(8 * half + 2 * ga) * planeR2 + (uint32_t)m * 16u;
#pragma unroll 1
    for (int g = ga; g < gb; ++g, d += 2 * planeR2) {
        uint32_t r[8], q[8];
        tc::tmem_ld8(col + (uint32_t)(8 * g), r);
        if (kSplit) tc::tmem_ld8(col + kLoOff + (uint32_t)(8 * g), q);
        tc::tmem_wait_ld();
        if (jrow >= P.N1) continue;
        *reinterpret_cast<uint4*>(d) = make_uint4(r[0], r[1], r[2], r[3]);
        *reinterpret_cast<uint4*>(d + planeR2) = make_uint4(r[4], r[5], r[6], r[7]);
        if (kSplit) {
            *reinterpret_cast<uint4*>(d + b2_lo) = make_uint4(q[0], q[1], q[2], q[3]);
            *reinterpret_cast<uint4*>(d + b2_lo + planeR2) = make_uint4(q[4], q[5], q[6], q[7]);
        }
    }
}

// ------------------------------------------------------------------------------------------
// Math warps.
// ------------------------------------------------------------------------------------------
template <bool kSplit>
__device__ __forceinline__ void math_warps(const Params& P, uint8_t* smem, uint32_t tb,
                                           const Step* ring, const Bars& B, unsigned (*s_gmax)[kMathWarps]) {
    constexpr uint32_t kGt = 128u * 128u * 2u;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int sp = warp & 3, half = warp >> 2;
    const uint32_t lane_base = (uint32_t)(32 * sp) << 16;
    const int m = 32 * sp + lane;          // TMEM lane: row m of A, Y, Q
    const int jrow = m >> 1;               // rows 2 j (Gy) and 2 j + 1 (s Gy') of spot row j
    const bool deriv = (m & 1) != 0;
    const int N1 = P.N1;
    const uint32_t R2 = 2u * (uint32_t)N1, planeR2 = R2 * 16u;
    const uint32_t b2_lo = kSplit ? R2 * 128u * 2u : 0u;
    const int bi = tid & 63, bc = tid >> 6;          // B without symmetry: spot and first 8-voxel chunk

    uint32_t ph2 = 0, n1done = 0;          // parity of mma2's next phase; phases of mma1 waited for
    bool ok = true;
    Prev prev{};
    bool have_prev = false;
    int k = 0, n = 0, nu = 0;              // ring reads, steps, units
    // per unit: this lane's row position (integer and fractional voxels, from this half's first
    // column of row tile 0), its warp's first and last rows, the B spot's, and G's scale
    float un = 0.f, uf = 0.f, wlo = 0.f, whi = 0.f, xn = 0.f, xf = 0.f, xlo = 0.f, xhi = 0.f;
    int eg = 0;
    bool finite = true;

    auto wait_mma1 = [&](uint32_t upto) -> bool {
        while (n1done < upto) {
            if (!wait_bar(B.mma1, n1done & 1u, P.wait_ns)) return false;
            ++n1done;
        }
        return true;
    };

    for (;;) {
        const int slot = k % kRing;
        ok = wait_bar(&B.full[slot], (uint32_t)((k / kRing) & 1), P.wait_ns);
        if (!__all_sync(0xffffffffu, ok)) break;
        // the step stays in its ring slot (read from there, not held in registers) until its last use
        const Step& cur = ring[slot];
        if (cur.flags != kEnd && (cur.job < 0 || cur.job >= P.n_jobs)) ok = false;
        ++k;
        if (!__all_sync(0xffffffffu, ok)) break;
        if (cur.flags & kEnd) break;
        const int nsx = cur.nsx, nsy = cur.nsy;
        const int b = n & 1;

        // ---- unit start: G^T of the slice's column tile (rows x, K = y; zero outside the grid) ----
        if (cur.flags & kFirst) {
            const JobDev& J = P.jobs[cur.job];
            const int nx = J.nx, ny = J.ny, x0 = cur.xt * kTile;
            // the slice from the staging buffer (copied by the scheduler when it claimed the unit) or,
            // with several tiles, from global memory
            const float* g = J.grad_dose + (size_t)cur.z * ny * nx + x0;
            if (P.stage) {
                ok = wait_bar(B.sfull, (uint32_t)(nu & 1), P.wait_ns);
                if (!__all_sync(0xffffffffu, ok)) break;
            }
            // Rolled loops: this code runs once per unit and is fetched anew each time (the slice held in
            // registers and unrolled: 11,500 cycles, rolled: 3900).
            // The largest |G| of the column tile, as bits (a NaN or an infinity is the largest).
            unsigned mx = 0u;
            if (P.stage) {
                const uint4* sv = reinterpret_cast<const uint4*>(smem + P.o_stage);
#pragma unroll 2
                for (int e = tid; e < nx * ny / 4; e += kMath) {
                    const uint4 a = sv[e];
                    mx = max(max(mx, a.x & 0x7FFFFFFFu), max(a.y & 0x7FFFFFFFu, max(a.z & 0x7FFFFFFFu, a.w & 0x7FFFFFFFu)));
                }
                if (tid < (nx * ny & 3))
                    mx = max(mx, reinterpret_cast<const unsigned*>(sv)[(nx * ny & ~3) + tid] & 0x7FFFFFFFu);
            } else {
                const int xw = min(kTile, nx - x0);
#pragma unroll 16
                for (int y = tid >> 7; y < ny; y += 2)
                    if ((tid & 127) < xw) mx = max(mx, __float_as_uint(g[(size_t)y * nx + (tid & 127)]) & 0x7FFFFFFFu);
            }
            mx = __reduce_max_sync(0xffffffffu, mx);
            if (lane == 0) {
                s_gmax[nu & 1][warp] = mx;
                tc::mbar_arrive(B.gmax);
            }
            ok = wait_bar(B.gmax, (uint32_t)(nu & 1), P.wait_ns);
            if (!__all_sync(0xffffffffu, ok)) break;
            mx = s_gmax[nu & 1][0];
#pragma unroll
            for (int q = 1; q < kMathWarps; ++q) mx = max(mx, s_gmax[nu & 1][q]);
            finite = mx < 0x7F800000u;
            int e = 0;
            (void)frexpf(__uint_as_float(mx), &e);        // the largest is below 2^e
            eg = (mx > 0u && finite) ? 15 - e : 0;        // and lands in [2^14, 2^15)
            eg = eg > 126 ? 126 : eg;
            const float gs = __int_as_float((127 + eg) << 23);
            const f32x2 gs2 = pk(gs, gs);
            // one column per thread, every other 8-row chunk
            const int x = tid & 127, yo = tid >> 7;
            const bool xin = x0 + x < nx;
            const float* src = (P.stage ? reinterpret_cast<const float*>(smem + P.o_stage) : g) + (size_t)(8 * yo) * nx + x;
            uint8_t* dst = smem + (uint32_t)yo * 2048u + (uint32_t)x * 16u;
            float nv[8];
            auto fetch = [&](int c) {
                const int left = xin ? ny - 8 * c : 0;       // rows of the chunk inside the grid
#pragma unroll
                for (int q = 0; q < 8; ++q) nv[q] = q < left ? src[(size_t)q * nx] : 0.f;
                src += (size_t)16 * nx;
            };
            fetch(yo);
#pragma unroll 1
            for (int c = yo; c < 16 * P.tiles; c += 2) {
                f32x2 v[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) v[q] = mul2(pk(nv[2 * q], nv[2 * q + 1]), gs2);
                fetch(c + 2);                                // the next chunk's loads, under this one's split
                uint32_t h[4], l[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) split2<kSplit>(v[q], h[q], l[q]);
                *reinterpret_cast<uint4*>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
                if (kSplit) *reinterpret_cast<uint4*>(dst + kGt) = make_uint4(l[0], l[1], l[2], l[3]);
                dst += 4096u + (kSplit && (c & 15) >= 14 ? kGt : 0u);    // past the lo half at a row tile's end
            }
            if (P.stage) {
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(B.sfree);   // the staging buffer is free again
            }
            ++nu;
            // positions in voxels (FP64), split into integer and fraction; the ends of this warp's rows
            // (of its spots, for B) from its lanes
            const double py = (J.sy0 + ((double)jrow - 0.5 * (double)(nsy - 1)) * J.dsy - J.oy) * (1.0 / J.dy) - 64.0 * half;
            const double ry = rint(py);
            un = (float)-ry;
            uf = (float)(ry - py);
            wlo = __shfl_sync(0xffffffffu, (float)py, 0);
            whi = __shfl_sync(0xffffffffu, (float)py, min(30, max(0, 2 * (nsy - 1 - 16 * sp))));
            if (!P.sym) {
                const double px = (J.sx0 + ((double)bi - 0.5 * (double)(nsx - 1)) * J.dsx - J.ox) * (1.0 / J.dx) - (double)x0;
                const double rx = rint(px);
                xn = (float)-rx;
                xf = (float)(rx - px);
                xlo = __shfl_sync(0xffffffffu, (float)px, 0);
                xhi = __shfl_sync(0xffffffffu, (float)px, min(31, max(0, nsx - 1 - 32 * (warp & 1))));
            }
        }

        // ---- G: A = [Gy | s Gy']^T -> TMEM A[b] (row m, y columns [64 half, +64)) ----
        // a warp whose 32 TMEM rows are all padding (m >= 2 nsy) skips G and E1: those rows of
        // every product only ever feed rows of Q that are never read
        const bool pad_warp = 32 * sp >= 2 * nsy;
        if (!pad_warp) {
            const bool valid = jrow < nsy;
            const float fa = valid ? (deriv ? -kOpScale : kOpScale) : 0.f;
            const float fb = valid && deriv ? cur.by : 0.f;
            const f32x2 A2 = pk(fa, fa), B2 = pk(fb, fb), na = pk(cur.nay, cur.nay), f2 = pk(uf, uf);
            const float off = (float)(128 * cur.yt);
            const float base = un + off;
            const float g0 = wlo - cur.ry - off, g1 = whi + cur.ry - off;
            const uint32_t col = tb + lane_base + kColA + (uint32_t)b * 128u + (uint32_t)(32 * half);
            // the step's K range within this half
            const int ga = max(cur.ya - 4 * half, 0), gb = min(cur.yb - 4 * half, 4);
#pragma unroll 1
            for (int g = ga; g < gb; ++g) {
                uint32_t hi[8], lo[8];
                if ((float)(16 * g + 15) >= g0 && (float)(16 * g) <= g1) {
                    gauss_row<kSplit, 8>(base + (float)(16 * g), f2, na, A2, B2, hi, lo);
                } else {                        // past this warp's own band
#pragma unroll
                    for (int q = 0; q < 8; ++q) hi[q] = lo[q] = 0u;
                }
                tc::tmem_st8(col + (uint32_t)(8 * g), hi);
                if (kSplit) tc::tmem_st8(col + kLoOff + (uint32_t)(8 * g), lo);
            }
        }
        // Second row tile: the first one's stage 1 is waited for here, so that no warp arrives twice
        // in one phase of ops1 and no phase of mma1 passes unseen.
        if (!(cur.flags & kPairFirst)) {
            ok = wait_mma1((uint32_t)n);
            if (!__all_sync(0xffffffffu, ok)) break;
        }
        tc::tmem_wait_st();
        if (cur.flags & kFirst) tc::fence_async_smem();     // G^T (B's stores are fenced before ops2)
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(B.ops1);

        if (cur.flags & kPairFirst) {
            // ---- DR: Q of the previous pair -> its P slot and dot products ----
            if (have_prev) {
                ok = ok && wait_bar(B.mma2, ph2, P.wait_ns);
                if (ok) ph2 ^= 1;
                ok = ok && wait_bar(&B.wfull[prev.pair & 1], (uint32_t)((prev.pair >> 1) & 1), P.wait_ns);
                if (!__all_sync(0xffffffffu, ok)) break;
                tc::fence_after_sync();
            }
            // symmetric fields: B = the rows just evaluated.  Stage 2 of the previous pair, the only
            // reader of B, is complete (waited for above, or there is none).
            if (P.sym && !pad_warp)
                store_b_sym<kSplit>(P, smem, tb + lane_base + kColA + (uint32_t)b * 128u, cur, half, m, jrow);
            if (have_prev) {
                drain_q(P, prev, tb + lane_base + kColQ, half, jrow, deriv, warp, lane,
                        reinterpret_cast<const float*>(smem + P.o_w + (uint32_t)(prev.pair & 1) * P.w_bytes));
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&B.wfree[prev.pair & 1]);
            }
            have_prev = false;
        }
        ++n;
        if (!(cur.flags & kPairEnd)) {
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&B.empty[slot]);
            continue;
        }

        // ---- B = [Gx | s Gx'] -> smem (rows 2 i and 2 i + 1, K = x).  Only stage 2 reads it, and the
        // previous pair's stage 2 is complete (DR waited), so one buffer serves. ----
        if (!P.sym && bi < N1) {
            const bool valid = bi < nsx;
            const float fa = valid ? kOpScale : 0.f, fb = valid ? cur.bx : 0.f;
            const f32x2 f2 = pk(xf, xf), na = pk(cur.nax, cur.nax), two = pk(2.0f, 2.0f);
            const f32x2 A2 = pk(fa, fa), Am = pk(-fa, -fa), Bd = pk(fb, fb);
            const float g0 = xlo - cur.rx, g1 = xhi + cur.rx;
            // the spots' 32-lane halves are warps: the same chunks are in the band for a whole warp
            for (int c = bc; c < 16; c += 4) {
                if ((c >> 1) < cur.xa || (c >> 1) >= cur.xb) continue;
                uint32_t h0[4], l0[4], h1[4], l1[4];
                if ((float)(8 * c + 7) >= g0 && (float)(8 * c) <= g1) {
                    f32x2 n2 = pk(xn + (float)(8 * c), xn + (float)(8 * c + 1));
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const f32x2 u = add2(n2, f2);
                        const f32x2 dd = mul2(u, u);
                        float a0, a1;
                        upk(mul2(dd, na), a0, a1);
                        const f32x2 e = pk(ex2_approx(a0), ex2_approx(a1));
                        split2<kSplit>(mul2(e, A2), h0[q], l0[q]);
                        split2<kSplit>(mul2(e, fma2(dd, Bd, Am)), h1[q], l1[q]);
                        n2 = add2(n2, two);
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q) h0[q] = l0[q] = h1[q] = l1[q] = 0u;
                }
                const uint32_t o0 = P.o_b2 + (uint32_t)c * planeR2 + (uint32_t)bi * 32u;
                *reinterpret_cast<uint4*>(smem + o0) = make_uint4(h0[0], h0[1], h0[2], h0[3]);
                *reinterpret_cast<uint4*>(smem + o0 + 16) = make_uint4(h1[0], h1[1], h1[2], h1[3]);
                if (kSplit) {
                    *reinterpret_cast<uint4*>(smem + o0 + b2_lo) = make_uint4(l0[0], l0[1], l0[2], l0[3]);
                    *reinterpret_cast<uint4*>(smem + o0 + b2_lo + 16) = make_uint4(l1[0], l1[1], l1[2], l1[3]);
                }
            }
        }
        // ---- E1: Y of this pair -> split -> TMEM A[b] (row m, x columns [64 half, +64)) ----
        ok = ok && wait_mma1((uint32_t)n);
        if (!__all_sync(0xffffffffu, ok)) break;
        tc::fence_after_sync();
        if (!pad_warp) {
            const int xa = cur.xa - 4 * half, xb = cur.xb - 4 * half;
            const f32x2 f2 = pk(cur.fy, cur.fy);
            const uint32_t col = kColA + (uint32_t)b * 128u + (uint32_t)(32 * half);
#pragma unroll 1
            for (int g = max(xa, 0); g < min(xb, 4); ++g) {
                uint32_t r[16], h[8], l[8];
                tc::tmem_ld16(tb + lane_base + kColY + (uint32_t)(64 * half + 16 * g), r);
                tc::tmem_wait_ld();
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    split2<kSplit>(mul2(pk(__uint_as_float(r[2 * q]), __uint_as_float(r[2 * q + 1])), f2),
                                   h[q], l[q]);
                tc::tmem_st8(tb + lane_base + col + (uint32_t)(8 * g), h);
                if (kSplit) tc::tmem_st8(tb + lane_base + col + kLoOff + (uint32_t)(8 * g), l);
            }
        }
        tc::tmem_wait_st();
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(B.ops2);
        // Q = 2^14 2^eg 2^-(14 + ky) 2^14 Q_true; a slice with a non-finite value gives NaN everywhere
        prev.nsx = nsx; prev.nsy = nsy; prev.pair = cur.pair;
        prev.slot = cur.slot; prev.dot_p = cur.dot_p; prev.dot_s = cur.dot_s;
        const int ex = cur.ky - 14 - eg, e1 = max(ex, -100);       // [-139, 108]
        prev.pow2 = __int_as_float((127 + e1) << 23);
        prev.nrm = finite ? cur.nrm * __int_as_float((127 + ex - e1) << 23) : __int_as_float(0x7fc00000);
        prev.inv_s = cur.inv_s;
        have_prev = true;
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&B.empty[slot]);
    }
    // last pair's Q
    if (ok && have_prev) {
        ok = wait_bar(B.mma2, ph2, P.wait_ns);
        ok = ok && wait_bar(&B.wfull[prev.pair & 1], (uint32_t)((prev.pair >> 1) & 1), P.wait_ns);
        if (__all_sync(0xffffffffu, ok)) {
            tc::fence_after_sync();
            drain_q(P, prev, tb + lane_base + kColQ, half, jrow, deriv, warp, lane,
                    reinterpret_cast<const float*>(smem + P.o_w + (uint32_t)(prev.pair & 1) * P.w_bytes));
        }
    }
    if (!ok && lane == 0) atomicExch(P.err, 1);
}

template <bool kSplit>
__global__ void __launch_bounds__(kThreads, 1) adj_tc_kernel(Params P) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t s_bars[2 * kRing + 11];
    __shared__ Step ring[kRing];
    __shared__ unsigned s_gmax[2][kMathWarps];
    __shared__ uint32_t tmem_base_s;

    Bars B;
    B.full = s_bars; B.empty = s_bars + kRing;
    uint64_t* q = s_bars + 2 * kRing;
    B.ops1 = q; B.ops2 = q + 1; B.mma1 = q + 2; B.mma2 = q + 3; B.sfull = q + 4; B.sfree = q + 5;
    B.wfull = q + 6; B.wfree = q + 8; B.gmax = q + 10;
    const int warp = threadIdx.x >> 5;
    if (warp == 0) {
        tc::tmem_alloc(&tmem_base_s, kCols);
        tc::tmem_relinquish();
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < kRing; ++i) {
            tc::mbar_init(&B.full[i], 1);
            tc::mbar_init(&B.empty[i], kMathWarps + 3);   // math warps, both MMA warps, weight warp
        }
        tc::mbar_init(B.sfull, P.stage == 2 ? 32 : 1);     // the scheduler's lanes, or its expect_tx + bytes
        tc::mbar_init(B.sfree, kMathWarps);
        tc::mbar_init(B.ops1, kMathWarps);
        tc::mbar_init(B.ops2, kMathWarps);
        tc::mbar_init(B.mma1, 1);
        tc::mbar_init(B.mma2, 1);
        for (int i = 0; i < 2; ++i) {
            tc::mbar_init(&B.wfull[i], 1);
            tc::mbar_init(&B.wfree[i], kMathWarps);
        }
        tc::mbar_init(B.gmax, kMathWarps);
        tc::fence_mbar_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    // Launched as a programmatic dependent of the forward: everything above overlaps the
    // forward's last CTAs; nothing below runs before the forward has completed (no-op when
    // there is no such predecessor).
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // the reduce (a programmatic dependent) may be scheduled onto the SMs this grid frees; one
    // CTA per SM here, so it takes no SM that a CTA of this grid still needs
    asm volatile("griddepcontrol.launch_dependents;");
    // Units: the largest unit bounds the balance of the persistent grid (a slice with exactly
    // C active layers is one unit, claimed late), so units just above the mean load per CTA,
    // ceil(T / grid) + 1 layers, balance best (a scheduling model and measurements agree); the
    // job views are visible from here on.
    __shared__ Units s_units;
    __shared__ int s_pairs;
    Units U{P.chunk, P.cmax, P.n_units};
    if (P.adapt) {
        if (threadIdx.x == 0) s_pairs = 0;
        __syncthreads();
        const JobDev& J = P.jobs[0];
        const int ne = J.nz * J.nl;
        int cnt = 0;
#pragma unroll 8
        for (int e = threadIdx.x; e < ne; e += kThreads) cnt += __ldg(J.idd + e) != 0.0 ? 1 : 0;
        cnt = __reduce_add_sync(0xffffffffu, cnt);
        if ((threadIdx.x & 31) == 0) atomicAdd(&s_pairs, cnt);
        __syncthreads();
        if (threadIdx.x == 0) {
            const int g = (int)gridDim.x;
            int c = (s_pairs * P.xtmax + g - 1) / g + 1;
            c = c < 1 ? 1 : (c > kMaxChunkCost ? kMaxChunkCost : c);
            const int cm = (J.nl + c - 1) / c;
            s_units = Units{c, cm, J.nz * cm * P.xtmax};
        }
        __syncthreads();
        U = s_units;
    }

    if (warp >= kMathWarps) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kCtrlRegs));
        if (warp == kSchedWarp) {
            scheduler_warp(P, U, ring, B, smem);
        } else if (warp == kWWarp) {
            weight_warp(P, ring, B, smem);
        } else {
            mma_warp<kSplit>(P, tc::smem_u32(smem), tmem_base_s, warp == kS1Warp ? 1 : 2, ring, B);
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kMathRegs));
        math_warps<kSplit>(P, smem, tmem_base_s, ring, B, s_gmax);
    }

    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (warp == 0) tc::tmem_dealloc(tmem_base_s, kCols);
}

// After the main kernel: dL/dW, the per-pair dot products and dL/dR from the slots, with no
// block waiting on another.  Block (entry chunk, layer l, job): kRedEnt slot entries
// e = j * n1 + i of layer l (n1 = nsx rounded up to 16) times kRedSeg depth segments (a "slice"
// below is one column tile of a slice: slots are (layer, slice, tile)).  The
// layer's IDD column is staged in shared memory with its last active slice ze; segment s of an
// entry sums IDD * P slot over its quarter of [0, ze) in slice order, its slot values arriving
// by asynchronous 4-byte copies (cp.async: kRedB slices per batch, every copy of a batch in
// flight together; inactive slices copy nothing and read 0); the segments' sums are then added
// in segment order and written as dL/dW[l, j, i] (i < nsx).  One more block per layer (the
// last in x) adds, per active slice, the eight warp partials of <P, W> (dL/dIDD) and <S, W>
// (dL/dsigma, times IDD) in warp order and forms dL/dR_l in FP64 (a fixed tree over the
// block); that block of layer 0 sums the loss partials the same way.  Every sum is in a fixed
// order: deterministic.
constexpr int kRedThreads = 256;
constexpr int kRedEnt = 64;                        // entries per block
constexpr int kRedSeg = kRedThreads / kRedEnt;     // depth segments per entry
constexpr int kRedTile = 1024;                     // slices staged per pass
constexpr int kRedB = 16;                          // slices per copy batch

__device__ __forceinline__ double block_sum_fixed(double v, double* red) {
    const int tid = threadIdx.x;
    red[tid] = v;
    __syncthreads();
    for (int w = kRedThreads / 2; w > 0; w >>= 1) {
        if (tid < w) red[tid] += red[tid + w];
        __syncthreads();
    }
    const double r = red[0];
    __syncthreads();
    return r;
}

__global__ void __launch_bounds__(kRedThreads) adj_tc_reduce_kernel(
    const JobDev* __restrict__ jobs, int with_range, int finalize_loss, const int* __restrict__ err) {
    // a programmatic dependent of the adjoint kernel: wait for its slots (no-op otherwise)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const JobDev& J = jobs[blockIdx.z];
    const int ec = blockIdx.x, l = blockIdx.y;
    if (l >= J.nl) return;
    const int nz = J.nz, ntx = J.ntx, nt = nz * ntx, nsx = J.nsx, nsy = J.nsy;
    const int n1 = (nsx + 15) / 16 * 16, per = nsy * n1;
    const int nchunk = (per + kRedEnt - 1) / kRedEnt;   // entry blocks; block nchunk: the dots
    if (ec > nchunk) return;
    const int tid = threadIdx.x, el = tid % kRedEnt, sg = tid / kRedEnt;
    const int e = ec * kRedEnt + el;
    const int ej = e / n1, ei = e - ej * n1;
    const bool own = e < per && ei < nsx;
    const size_t ndots = (size_t)J.nl * nt * kMathWarps;
    const float* slots = J.partial + (size_t)l * nt * per;           // (nz, ntx, per) of layer l
    const float* dots = J.partial + (size_t)J.nl * nt * per;          // (2, nl, nz, ntx, kMathWarps)
    const double* idd = J.idd + (size_t)l * nz;
    const bool bad = *err != 0 || (J.fwd_err != nullptr && *J.fwd_err != 0);
    const float nan = __int_as_float(0x7fc00000);
    __shared__ double red[kRedThreads];
    if (ec == nchunk) {
        // per job: no dL/dR output, or a missing derivative table, contributes nothing (the
        // heterogeneous range gradient's two job sets use one table each)
        const bool rng = with_range && J.grad_range != nullptr;
        double a = 0.0;
        for (int z = tid; z < nz; z += kRedThreads) {
            const double c = idd[z];
            if (c == 0.0) continue;
            const size_t o = (size_t)l * nz + z;
            const float* pa = dots + o * ntx * kMathWarps;
            const float* pb = pa + ndots;
            float sa = 0.f, sb = 0.f;
            for (int t = 0; t < ntx; ++t)
#pragma unroll
                for (int w = 0; w < kMathWarps; ++w) { sa += pa[t * kMathWarps + w]; sb += pb[t * kMathWarps + w]; }
            const float dsg = (float)c * sb;
            J.dc[o] = sa;
            J.dsg[o] = dsg;
            if (rng)
                a += (J.didd_dr ? (double)sa * J.didd_dr[o] : 0.0) +
                     (J.dsig_dr ? (double)dsg * J.dsig_dr[o] : 0.0);
        }
        if (rng) {
            const double r = block_sum_fixed(a, red);
            if (tid == 0) J.grad_range[l] = bad ? nan : (float)r;
        }
        if (finalize_loss && l == 0) {
            double t = 0.0;
            for (int b = tid; b < J.n_loss_part; b += kRedThreads) t += J.loss_part[b];
            const double sum = block_sum_fixed(t, red);
            if (tid == 0) *J.loss = bad ? (double)nan : sum;
        }
        return;
    }

    __shared__ float s_c[kRedTile];
    __shared__ int s_end;
    __shared__ float sbuf[kRedB][kRedThreads];
    __shared__ float s_part[kRedSeg][kRedEnt];
    float acc = 0.f;
    const float* se = slots + (own ? e : 0);
    for (int zt = 0; zt < nt; zt += kRedTile) {
        const int zn = min(kRedTile, nt - zt);
        __syncthreads();   // the previous pass's reads of s_c and s_end are done
        if (tid == 0) s_end = 0;
        for (int z = tid; z < zn; z += kRedThreads) s_c[z] = (float)idd[ntx == 1 ? zt + z : (zt + z) / ntx];
        __syncthreads();
        for (int z = tid; z < zn; z += kRedThreads)
            if (s_c[z] != 0.f) atomicMax(&s_end, z + 1);
        __syncthreads();
        const int ze = s_end;   // slices [0, ze) of the pass hold every active one
        const int q = (ze + kRedSeg - 1) / kRedSeg;
        const int zb = sg * q, zf = min(ze, zb + q);
        for (int z0 = zb; z0 < zf; z0 += kRedB) {
#pragma unroll
            for (int h = 0; h < kRedB; ++h) {
                const int z = z0 + h;
                const bool rd = own && z < zf && s_c[z < zf ? z : zb] != 0.f;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
                                 tc::smem_u32(&sbuf[h][tid])),
                             "l"(se + (size_t)(zt + (rd ? z : 0)) * per), "r"(rd ? 4 : 0)
                             : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
            for (int h = 0; h < kRedB; ++h) {
                const int z = z0 + h;
                const float cf = z < zf ? s_c[z] : 0.f;
                acc = fmaf(cf, sbuf[h][tid], acc);
            }
        }
    }
    s_part[sg][el] = acc;
    __syncthreads();
    if (sg == 0 && own) {
        float g = s_part[0][el];
#pragma unroll
        for (int k = 1; k < kRedSeg; ++k) g += s_part[k][el];
        J.grad_w[((size_t)l * nsy + ej) * nsx + ei] = bad ? nan : g;
    }
}

template <bool kSplit>
int launch_mode(const Params& P0, int max_nsy, cudaStream_t s) {
    // the setmaxnreg split needs the full launch allotment, or its increase never returns
    int max_dyn = 0;
    PBD_TRY(smem_optin((const void*)adj_tc_kernel<kSplit>, -1, kLaunchRegsNeeded, &max_dyn));
    Params P = P0;
    P.give_back = kSplit ? 5.9604644775390625e-8f : 0.f;
    const uint32_t narr = kSplit ? 2u : 1u;
    P.o_b2 = (uint32_t)P.tiles * narr * 128u * 128u * 2u;
    P.o_w = P.o_b2 + narr * 2u * (uint32_t)P.N1 * 128u * 2u;
    P.w_bytes = (uint32_t)align_up((size_t)max_nsy * (P.N1 + 4) * sizeof(float), 16);
    // the staging buffer (one 128 x 128 FP32 slice) after the weights, when it fits
    P.o_stage = (uint32_t)align_up(P.o_w + 2u * P.w_bytes, 128);
    if (P.stage && P.o_stage + 65536u > (size_t)max_dyn) P.stage = 0;
    size_t smem = P.stage ? P.o_stage + 65536u : P.o_stage;
    // >= 116 KiB: one CTA, and its 512 TMEM columns, per SM
    smem = std::max<size_t>(smem, 116u * 1024u);
    if (smem > (size_t)max_dyn) return PBD_ERR_NO_SMEM;
    const int grid = std::max(1, std::min(P.n_units, num_sms()));
    prof_mark(kProfAdj, 0, s);
    PBD_TRY(launch_dependent(adj_tc_kernel<kSplit>, dim3(grid), dim3(kThreads), smem, s, P));
    prof_mark(kProfAdj, 1, s);
    return PBD_OK;
}

}  // namespace

int tc_adjoint_dims(int precision, const pbd_field* f, int* N1) {
    if (f->nx > kTile || f->ny > kTile) return PBD_ERR_UNSUPPORTED;
    return tc_adjoint_dims_tiled(precision, f, N1);
}

int tc_adjoint_dims_tiled(int precision, const pbd_field* f, int* N1) {
    if (precision == PBD_PREC_FP32) return PBD_ERR_UNSUPPORTED;
    // past one tile the FP32 kernel is the way out when the slots would take more than 8 GiB
    if ((f->nx > kTile || f->ny > kTile) && tc_adjoint_slot_elems(f) > ((size_t)2 << 30)) return PBD_ERR_UNSUPPORTED;
    if (f->ny > kMaxRowTiles * kTile || f->n_sy > 64 || f->n_sx > 64) return PBD_ERR_UNSUPPORTED;
    *N1 = (f->n_sx + 15) / 16 * 16;
    return PBD_OK;
}

size_t tc_adjoint_counter_ints(int n_jobs, int max_layers) {
    (void)n_jobs;
    (void)max_layers;
    return 2u;
}

size_t tc_adjoint_slot_elems(const pbd_field* f) {
    // slot rows of nsx rounded up to 16 floats: every job's slots start on a 64-byte boundary
    const size_t per = (size_t)f->n_sy * (size_t)((f->n_sx + 15) / 16 * 16);
    const size_t pairs = (size_t)f->n_layers * f->nz * (size_t)((f->nx + kTile - 1) / kTile);
    return pairs * per + 2u * pairs * kMathWarps;
}

int launch_adjoint_tc(int precision, JobDev* jobs_dev, const JobDev* jobs_host, int n_jobs,
                      int* counter, int* err, int chunk, int with_range, int finalize_loss,
                      int counters_zeroed, cudaStream_t s) {
    Params P{};
    P.jobs = jobs_dev;
    P.n_jobs = n_jobs;
    P.chunk = chunk;
    P.counter = counter;
    P.err = err;
    P.wait_ns = wait_limit_ns();
    P.hold = test_hold();
    // bulk copies of the dL/dD slices need them contiguous and 16-byte aligned, and one tile each
    P.stage = 1;
    P.tiles = 1;
    P.xtmax = 1;
    int cm = 1, nzm = 1, max_l = 1, max_per = 1, max_nsy = 1;
    for (int j = 0; j < n_jobs; ++j) {
        const JobDev& J = jobs_host[j];
        pbd_field f{};
        f.nx = J.nx; f.ny = J.ny;
        f.n_sx = J.nsx; f.n_sy = J.nsy;
        int n1 = 0;
        PBD_TRY(tc_adjoint_dims_tiled(precision, &f, &n1));
        if (((size_t)J.nx * J.ny) % 4 != 0 ||
            (reinterpret_cast<uintptr_t>(J.grad_dose) & 15u) != 0)
            P.stage = 2;
        P.N1 = std::max(P.N1, n1);
        P.tiles = std::max(P.tiles, J.nty);
        P.xtmax = std::max(P.xtmax, J.ntx);
        cm = std::max(cm, (J.nl + chunk - 1) / chunk);
        nzm = std::max(nzm, J.nz);
        max_l = std::max(max_l, J.nl);
        max_nsy = std::max(max_nsy, J.nsy);
        max_per = std::max(max_per, J.nsy * ((J.nsx + 15) / 16 * 16));
    }
    const bool tiled = P.tiles > 1 || P.xtmax > 1;
    if (tiled) P.stage = 0;
    P.cmax = cm;
    // one job and no explicit schedule: the CTAs derive the unit size from the active pairs
    P.adapt = (n_jobs == 1 && schedule_adj_override() == 0) ? 1 : 0;
    P.sym = tiled ? 0 : 1;
    for (int j = 0; j < n_jobs; ++j) {
        const JobDev& J = jobs_host[j];
        if (!(J.nx == J.ny && J.ox == J.oy && J.dx == J.dy && J.nsx == J.nsy && J.sx0 == J.sy0 &&
              J.dsx == J.dsy))
            P.sym = 0;
    }
    const long long units = (long long)nzm * cm * n_jobs * P.xtmax;
    if (units > (1LL << 30)) return PBD_ERR_UNSUPPORTED;
    P.n_units = (int)units;
    if (!counters_zeroed)
        PBD_TRY(cuda_rc(cudaMemsetAsync(counter, 0,
                                        tc_adjoint_counter_ints(n_jobs, max_l) * sizeof(int), s)));
    // grids past one tile ran in FP32 before they ran here: split FP16 for every mode
    if (precision == PBD_PREC_BF16 && !tiled) PBD_TRY(launch_mode<false>(P, max_nsy, s));
    else PBD_TRY(launch_mode<true>(P, max_nsy, s));
    PBD_TRY(launch_dependent(adj_tc_reduce_kernel,
                             dim3((max_per + kRedEnt - 1) / kRedEnt + 1, max_l, n_jobs),
                             dim3(kRedThreads), 0, s, (const JobDev*)jobs_dev, with_range,
                             finalize_loss, (const int*)err));
    count_launch(2);
    return PBD_OK;
}

}  // namespace pbd
