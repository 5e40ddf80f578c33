// fwd_simt.cu -- forward dose on the CUDA cores (FP32 FMA), persistent and load-balanced.
//
// D[z,y,x] = sum_l IDD_l(z) sum_j Gy[y,j] sum_i W_l[j,i] Gx[x,i]   (engines.py:191-197)
//
// Work item = (job, depth slice z, lateral tile of at most 128x128, chunk of <= C active layers).
// For each active layer the CTA generates the Gaussian factors of that (layer, slice)
// in shared memory (never stored in HBM), contracts
//     U[j, x] = sum_i W'[j,i] Gx[x,i]      (W' = W * IDD / (2 pi sigma^2))
//     D[y, x] += sum_j Gy[y,j] U[j,x]
// with D held in registers across the chunk's layers, and writes the chunk's partial
// slice once.  The finalize kernel sums the (at most ceil(L/C)) partials of a slice in
// chunk order -- deterministic -- and fuses the masked quadratic loss and its gradient.
// Items are sorted by cost (longest first) by a device-side scheduler, and a
// persistent grid pulls them from an atomic counter: the deep slices that see few
// layers no longer bound the launch.
#include <algorithm>

#include "pbd_internal.cuh"

namespace pbd {
namespace {

constexpr int NT = 256;
constexpr int SC = kSpotChunk;                      // 64 spots per chunk
// shared memory of a 16 RY x 16 RX tile with spot chunks of scx x scy (128 x 128, 64 x 64 spots: 112 KiB)
constexpr size_t fwd_smem(int ry, int rx, int scx, int scy) {
    return (size_t)(16 * (rx * scx + (rx + ry) * scy) + scx * SC) * sizeof(float);
}
// Spots per chunk of an axis of n: equal parts of at most 64, in fours along x (73 spots as 40 + 33, not 64 + 9).
// Along y, where U's rows come in groups of 16, a cut lies on a group (69 spots as 48 + 21, 80 rows, not 36 + 33,
// 96: 150 x 142 x 130, 73 x 69 spots, 24 layers on every slice 1208 us, now 1171).  Each axis of each job has its
// own.  One size for the launch, from its widest axis, cut 41 spots beside 73 into 40 + 1, each part with its
// own weights, factors and barriers: 128 x 128 x 64, 73 x 41 spots, 10 layers 302 us, now 217; a batch of three
// 41 x 41 fields and a small one of 73 x 73 386, now 306.
__host__ __device__ constexpr int spot_chunk(int n, int group = 4) {
    const int parts = (n + SC - 1) / SC, g = parts > 1 ? group : 4;
    return ((n + parts - 1) / parts + g - 1) / g * g;
}

// Tile sizes per axis, in units of 16 voxels.  An axis of n voxels is cut into ceil(n / 128) tiles of
// equal size, rounded up to one of these: a 150 x 142 slice in four 80 x 80 tiles instead of four
// 128 x 128 ones, of which two thirds were outside the grid.  The kernel is bound by FP32 FMA issue, so
// its time follows the padded area: 150 x 142 x 130, 24 layers of 73 x 69 spots (cut in chunks of 40 and 48
// for the same reason, where 64 + 9 were padded to 128): 1143 us with 128 x 128 tiles and 64-spot chunks, 640
// with these, 605-626 with three blocks to an SM (which small tiles allow and large ones do not: an
// 8 x 8 register tile needs 128 registers).  A grid of 128 keeps its 128 x 128 tile: two of 64 x 128
// would build every factor of the uncut axis twice.  Sums run in the same order whatever the tile.
constexpr int kSizes[] = {4, 5, 6, 8};
int tile_size(int n) {
    const int nt = (n + kTile - 1) / kTile, need = ((n + nt - 1) / nt + 15) / 16;
    for (int r : kSizes)
        if (r >= need) return r;
    return 8;
}

__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Scheduler: one CTA per job.  Items are written to the job's segment of the flat
// item array, bucket-sorted by cost (descending); unused slots get cost 0.
// Activity flags (IDD != 0) of a job staged in shared memory when they fit.
constexpr int kActStage = 40 * 1024;

__device__ __forceinline__ bool active(const JobDev& J, const unsigned char* sact, bool staged,
                                       int l, int z) {
    return staged ? sact[l * J.nz + z] != 0 : J.idd[(size_t)l * J.nz + z] != 0.0;
}

__device__ __forceinline__ bool stage_activity(const JobDev& J, unsigned char* sact) {
    const bool staged = J.nl * J.nz <= kActStage;
    if (staged)
        for (int e = threadIdx.x; e < J.nl * J.nz; e += blockDim.x) sact[e] = J.idd[e] != 0.0;
    __syncthreads();
    return staged;
}

__global__ void fwd_schedule_kernel(JobDev* jobs, FwdItem* items, int chunk) {
    const JobDev J = jobs[blockIdx.x];
    extern __shared__ unsigned char sact[];
    __shared__ int cnt[kMaxChunkCost + 1];
    __shared__ int cur[kMaxChunkCost + 1];
    __shared__ int total;
    const int ntiles = J.ntx * J.nty;
    for (int c = threadIdx.x; c <= kMaxChunkCost; c += blockDim.x) cnt[c] = 0;
    const bool staged = stage_activity(J, sact);
    for (int z = threadIdx.x; z < J.nz; z += blockDim.x) {
        int a = 0;
        for (int l = 0; l < J.nl; ++l) a += active(J, sact, staged, l, z);
        const int nch = (a + chunk - 1) / chunk;
        J.nchunks[z] = nch;
        for (int k = 0; k < nch; ++k) atomicAdd(&cnt[min(chunk, a - k * chunk)], ntiles);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int pos = 0;
        for (int c = chunk; c >= 1; --c) { cur[c] = pos; pos += cnt[c]; }
        total = pos;
    }
    __syncthreads();
    for (int z = threadIdx.x; z < J.nz; z += blockDim.x) {
        int k = 0, in_chunk = 0, lb = 0, last = 0;
        for (int l = 0; l <= J.nl; ++l) {
            const bool act = l < J.nl && active(J, sact, staged, l, z);
            if (act) {
                if (in_chunk == 0) lb = l;
                ++in_chunk;
                last = l;
            }
            if ((act && in_chunk == chunk) || (l == J.nl && in_chunk > 0)) {
                for (int t = 0; t < ntiles; ++t) {
                    const int p = atomicAdd(&cur[in_chunk], 1);
                    FwdItem it;
                    it.job = blockIdx.x; it.z = z; it.ty = t / J.ntx; it.tx = t % J.ntx;
                    it.lb = lb; it.le = last + 1; it.chunk = k; it.cost = in_chunk;
                    items[J.item_base + p] = it;
                }
                ++k;
                in_chunk = 0;
            }
        }
    }
    __syncthreads();
    for (int p = total + threadIdx.x; p < J.max_items; p += blockDim.x) {
        FwdItem it{};
        items[J.item_base + p] = it;
    }
}

// Tile of 16 RY rows x 16 RX columns, RY x RX voxels per thread: the first four of an axis are
// consecutive (one 16-byte load), the others 16 apart past them (R < 8) or four more consecutive
// ones (R = 8).
template <int R>
__device__ __forceinline__ int tcoord(int t, int b) {
    if (b < 4) return 4 * t + b;
    return R == 8 ? 64 + 4 * t + (b - 4) : 64 + t + 16 * (b - 4);
}
template <int R>
__device__ __forceinline__ void tload(const float* row, int t, float (&v)[R]) {
    const float4 a = *reinterpret_cast<const float4*>(row + 4 * t);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    if constexpr (R == 8) {
        const float4 c = *reinterpret_cast<const float4*>(row + 64 + 4 * t);
        v[4] = c.x; v[5] = c.y; v[6] = c.z; v[7] = c.w;
    } else {
#pragma unroll
        for (int b = 4; b < R; ++b) v[b] = row[64 + t + 16 * (b - 4)];
    }
}

// U[j, x] of a spot chunk, a < RJ: rows j = 4 ty + a of a full chunk (RJ = 4, one 16-byte load of W), else
// j = ty + 16 a (the chunk's rows, in groups of 16).
template <int RJ>
__device__ __forceinline__ int urow(int ty, int a) { return RJ == 4 ? 4 * ty + a : ty + 16 * a; }

template <int RJ, int RX>
__device__ __forceinline__ void stage1(const float* WT, const float* GxT, int ni, int ty, int tx,
                                       float (&uacc)[4][RX]) {
#pragma unroll 2
    for (int ii = 0; ii < ni; ++ii) {
        float gb[RX], wa[RJ];
        tload<RX>(GxT + ii * 16 * RX, tx, gb);
        if constexpr (RJ == 4) {
            tload<4>(WT + ii * SC, ty, wa);
        } else {
#pragma unroll
            for (int a = 0; a < RJ; ++a) wa[a] = WT[ii * SC + urow<RJ>(ty, a)];
        }
#pragma unroll
        for (int a = 0; a < RJ; ++a)
#pragma unroll
            for (int b = 0; b < RX; ++b) uacc[a][b] = fmaf(wa[a], gb[b], uacc[a][b]);
    }
}

template <int RJ, int RX>
__device__ __forceinline__ void store_u(float* U, int nj, int ty, int tx, const float (&uacc)[4][RX]) {
#pragma unroll
    for (int a = 0; a < RJ; ++a) {
        if (urow<RJ>(ty, a) >= nj) break;
        float* row = U + urow<RJ>(ty, a) * 16 * RX;
#pragma unroll
        for (int b = 0; b < RX; ++b) row[tcoord<RX>(tx, b)] = uacc[a][b];
    }
}

// Two blocks per SM for the largest tiles' registers, three for tiles up to 80 x 80: the barriers
// and the weights' loads of one block run under the others' products.
template <int RY, int RX>
__global__ void __launch_bounds__(NT, RY * RX <= 25 ? 3 : 2)
fwd_simt_kernel(const JobDev* __restrict__ jobs, const FwdItem* __restrict__ items, int total,
                int* counter, int mx, int my) {
    constexpr int TY = 16 * RY, TX = 16 * RX;
    constexpr int PX = NT / TX, PY = NT / TY;        // spots generated at a time
    extern __shared__ float4 smem4[];
    float* GxT = reinterpret_cast<float*>(smem4);   // [mx i][TX x], mx x my: the largest chunk of any job
    float* GyT = GxT + mx * TX;                      // [my j][TY y]
    float* U = GyT + my * TY;                        // [my j][TX x]
    float* WT = U + my * TX;                         // [mx i][SC j]
    // 1 KB of static shared memory and no more: two blocks with the 112 KiB of the largest tile and chunks
    // then just fill an SM.  With the item index beside it, 4 bytes over, only one fitted: 200 x 200 x 64,
    // 61 x 61 spots, 10 layers 465 us against 370 of 60 x 60; now 305 against 303.
    __shared__ double s_xs[SC], s_ys[SC];
    int& s_item = *reinterpret_cast<int*>(WT);       // between items WT holds nothing
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int gx = tid % TX, gxr = tid / TX, gy = tid % TY, gyr = tid / TY;

    // Each block starts with the item of its index, the counter hands out those past the first grid-full,
    // so that a few items land on as many SMs.  Pulled by whichever block came first, they ran two to an
    // SM on half of the SMs (128 x 128 x 64, 61 x 61 spots, 10 layers 157 us, now 108).
    auto next = [&](int idx) {                       // idx or the first item past it that holds layers
        while (idx < total && items[idx].cost == 0) {
            __syncthreads();
            if (tid == 0) s_item = (int)gridDim.x + atomicAdd(counter, 1);
            __syncthreads();
            idx = s_item;
        }
        return idx;
    };
    for (int it_idx = next(blockIdx.x); it_idx < total;) {
        const FwdItem it = items[it_idx];
        const JobDev& J = jobs[it.job];
        const int nz = J.nz, nx = J.nx, ny = J.ny, nsx = J.nsx, nsy = J.nsy;
        const int z = it.z, y0 = it.ty * TY, x0 = it.tx * TX;
        const int scx = spot_chunk(nsx), scy = spot_chunk(nsy, 16);
        const bool chunks = scx < nsx || scy < nsy;
        // the chunk's spot positions: once per item where the lattice is one chunk
        auto stage_spots = [&](int j0, int i0) {
            if (tid < SC) s_xs[tid] = J.sx0 + ((double)(i0 + tid) - 0.5 * (double)(nsx - 1)) * J.dsx;
            else if (tid < 2 * SC) s_ys[tid - SC] = J.sy0 + ((double)(j0 + tid - SC) - 0.5 * (double)(nsy - 1)) * J.dsy;
            __syncthreads();
        };
        if (!chunks) stage_spots(0, 0);

        float dacc[RY][RX];
#pragma unroll
        for (int a = 0; a < RY; ++a)
#pragma unroll
            for (int b = 0; b < RX; ++b) dacc[a][b] = 0.f;

        for (int l = it.lb; l < it.le; ++l) {
            const double c = J.idd[(size_t)l * nz + z];
            if (c == 0.0) continue;
            const double s = fmax(J.sigma[(size_t)l * nz + z], 1e-9);
            const double a2 = kLog2e / (2.0 * s * s);
            const float nrm = (float)(c * kInv2Pi / (s * s));
            const float* wl = J.w + (size_t)l * nsy * nsx;

            for (int j0 = 0; j0 < nsy; j0 += scy) {
                const int nj = min(scy, nsy - j0);
                float uacc[4][RX];
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int b = 0; b < RX; ++b) uacc[a][b] = 0.f;

                for (int i0 = 0; i0 < nsx; i0 += scx) {
                    const int ni = min(scx, nsx - i0);
                    __syncthreads();
                    if (chunks) stage_spots(j0, i0);
#pragma unroll 4
                    for (int e = tid; e < ni * SC; e += NT) {
                        const int ii = e / SC, jj = e % SC;
                        WT[e] = jj < nj ? nrm * wl[(size_t)(j0 + jj) * nsx + i0 + ii] : 0.f;
                    }
                    // a thread forms the factors of one column (row) of the tile, every PX-th (PY-th) spot
                    if (tid < PX * TX) {
                        const double xv = J.ox + (double)(x0 + gx) * J.dx;
#pragma unroll 4
                        for (int ii = gxr; ii < ni; ii += PX) {
                            const double d = xv - s_xs[ii];
                            GxT[ii * TX + gx] = ex2_approx((float)(-(d * d) * a2));
                        }
                    }
                    if (i0 == 0 && tid < PY * TY) {
                        const double yv = J.oy + (double)(y0 + gy) * J.dy;
#pragma unroll 4
                        for (int jj = gyr; jj < nj; jj += PY) {
                            const double d = yv - s_ys[jj];
                            GyT[jj * TY + gy] = ex2_approx((float)(-(d * d) * a2));
                        }
                    }
                    __syncthreads();
                    // stage 1: U[j, x] += sum_i W'[j,i] Gx[x,i]
                    if (nj > 48) stage1<4, RX>(WT, GxT, ni, ty, tx, uacc);
                    else if (nj > 32) stage1<3, RX>(WT, GxT, ni, ty, tx, uacc);
                    else if (nj > 16) stage1<2, RX>(WT, GxT, ni, ty, tx, uacc);
                    else stage1<1, RX>(WT, GxT, ni, ty, tx, uacc);
                }
                if (nj > 48) store_u<4, RX>(U, nj, ty, tx, uacc);
                else store_u<3, RX>(U, nj, ty, tx, uacc);
                __syncthreads();
                // stage 2: D[y, x] += sum_j Gy[y,j] U[j,x]
#pragma unroll 2
                for (int jj = 0; jj < nj; ++jj) {
                    float ga[RY], ub[RX];
                    tload<RY>(GyT + jj * TY, ty, ga);
                    tload<RX>(U + jj * TX, tx, ub);
#pragma unroll
                    for (int a = 0; a < RY; ++a)
#pragma unroll
                        for (int b = 0; b < RX; ++b) dacc[a][b] = fmaf(ga[a], ub[b], dacc[a][b]);
                }
            }
        }
        // partial slice of this chunk
        const size_t n3 = (size_t)nz * ny * nx;
        float* out = J.partial + (size_t)it.chunk * n3 + (size_t)z * ny * nx;
#pragma unroll
        for (int a = 0; a < RY; ++a) {
            const int y = y0 + tcoord<RY>(ty, a);
            if (y >= ny) continue;
#pragma unroll
            for (int b = 0; b < RX; ++b) {
                const int x = x0 + tcoord<RX>(tx, b);
                if (x < nx) out[(size_t)y * nx + x] = dacc[a][b];
            }
        }
        __syncthreads();
        if (tid == 0) s_item = (int)gridDim.x + atomicAdd(counter, 1);
        __syncthreads();
        it_idx = next(s_item);
    }
}

// Sum of the chunk partials (chunk order), dose out, optional loss + dL/dD.
__global__ void fwd_finalize_kernel(const JobDev* __restrict__ jobs, int with_loss,
                                    const int* __restrict__ err) {
    const JobDev& J = jobs[blockIdx.y];
    const size_t plane = (size_t)J.nx * J.ny;
    const size_t n = plane * J.nz;
    const bool bad = *err != 0;   // a main-kernel wait timed out: make the result NaN
    double lsum = 0.0;
    for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < n;
         v += (size_t)gridDim.x * blockDim.x) {
        const int z = (int)(v / plane);
        const int nch = J.nchunks[z];
        float s = bad ? __int_as_float(0x7fc00000) : 0.f;
        for (int k = 0; k < nch; ++k) s += J.partial[(size_t)k * n + v];
        J.dose[v] = s;
        if (with_loss) {
            const float r = s - J.presc[v];
            const float m = J.mask[v];
            J.grad_dose[v] = 2.f * m * r;
            lsum += (double)m * (double)r * (double)r;
        }
    }
    if (with_loss) {
        __shared__ double red[256];
        red[threadIdx.x] = lsum;
        __syncthreads();
        for (int w = blockDim.x / 2; w > 0; w >>= 1) {
            if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
            __syncthreads();
        }
        if (threadIdx.x == 0) J.loss_part[blockIdx.x] = red[0];
    }
}

using FwdKernel = void (*)(const JobDev*, const FwdItem*, int, int*, int, int);
template <int RY>
FwdKernel pick_rx(int rx) {
    switch (rx) {
        case 4: return fwd_simt_kernel<RY, 4>;
        case 5: return fwd_simt_kernel<RY, 5>;
        case 6: return fwd_simt_kernel<RY, 6>;
        default: return fwd_simt_kernel<RY, 8>;
    }
}
FwdKernel pick_kernel(int ry, int rx) {
    switch (ry) {
        case 4: return pick_rx<4>(rx);
        case 5: return pick_rx<5>(rx);
        case 6: return pick_rx<6>(rx);
        default: return pick_rx<8>(rx);
    }
}

}  // namespace

int launch_slice_schedule(JobDev* jobs_dev, FwdItem* items, int chunk, int n_jobs,
                          cudaStream_t s) {
    fwd_schedule_kernel<<<n_jobs, 256, kActStage, s>>>(jobs_dev, items, chunk);
    PBD_LAUNCH_CHECK();
    return PBD_OK;
}

int fwd_chunk_layers(const pbd_field* f, int precision) {
    // FP32: ~4 layers per item keeps items small next to the ~2 CTAs per SM.  Tensor cores:
    // the pipeline runs across unit boundaries, so larger units only save partial slices
    // (24 measured best, with 4-layer adjoint units, on the 128^3 / 41 x 41 x 40 field;
    // the autotuner refines it per geometry).
    // The split-FP16 forward: 20.  The largest unit bounds the balance (a slice with exactly C
    // active layers is one unit, claimed after the shallow slices), and 20 is just above the
    // clinical field's mean load of 18.4 steps per SM (measured 83.6 us against 90.2 at 24).
    (void)f;
    if (precision == PBD_PREC_FP16X3) return 20;
    return precision == PBD_PREC_FP32 ? 4 : 24;
}

int fwd_plan_sizes(const pbd_field* f, int chunk, size_t* partial_elems, int* items) {
    const int ntx = (f->nx + kTile - 1) / kTile, nty = (f->ny + kTile - 1) / kTile;
    const int max_chunks = (f->n_layers + chunk - 1) / chunk;
    *partial_elems = (size_t)max_chunks * f->nz * f->ny * f->nx;
    const long long it = (long long)f->nz * max_chunks * ntx * nty;
    if (it > (1LL << 30)) return PBD_ERR_UNSUPPORTED;
    *items = (int)it;
    return PBD_OK;
}

int launch_forward(JobDev* jobs_dev, const JobDev* jobs_host, int n_jobs, FwdItem* items,
                   int total_items, int* counter, size_t n_counter_ints, int* err, int chunk,
                   int with_loss, int precision, int poison, void* pack, size_t pack_bytes,
                   cudaStream_t s, const JobPair* inst, JobDev* inst_dst, int* inst_status) {
    const bool tc16 = precision == PBD_PREC_FP16X3;
    if (inst && !tc16) return PBD_ERR_UNSUPPORTED;   // only the split-FP16 pack installs views
    if (precision != PBD_PREC_FP32) {
        // the split-FP16 path clears its unit counter in its pack kernel (no memset node between
        // the job install and the dose kernels) and may install the job views there too
        if (tc16)
            return launch_forward_tc16(jobs_dev, jobs_host, n_jobs, counter, err, chunk,
                                       with_loss, poison, pack, pack_bytes, s, inst, inst_dst,
                                       inst_status);
        PBD_TRY(cuda_rc(cudaMemsetAsync(counter, 0, n_counter_ints * sizeof(int), s)));
        return launch_forward_tc(precision, jobs_dev, jobs_host, n_jobs, counter, err, chunk,
                                 with_loss, poison, s);
    }
    // one tile size per launch, the largest a job needs (the tile counts are the same for all)
    int ry = kSizes[0], rx = kSizes[0], set = 0;
    for (int j = 0; j < n_jobs; ++j) {
        ry = std::max(ry, tile_size(jobs_host[j].ny));
        rx = std::max(rx, tile_size(jobs_host[j].nx));
    }
    // the largest spot chunks of any job size the shared memory
    int mx = 4, my = 4;
    for (int j = 0; j < n_jobs; ++j) {
        mx = std::max(mx, spot_chunk(jobs_host[j].nsx));
        my = std::max(my, spot_chunk(jobs_host[j].nsy, 16));
    }
    const FwdKernel kernel = pick_kernel(ry, rx);
    PBD_TRY(smem_optin((const void*)kernel, (int)fwd_smem(ry, rx, SC, SC), 0, &set));
    PBD_TRY(cuda_rc(cudaMemsetAsync(counter, 0, sizeof(int), s)));
    fwd_schedule_kernel<<<n_jobs, 256, kActStage, s>>>(jobs_dev, items, chunk);
    PBD_LAUNCH_CHECK();
    {
        const size_t smem = fwd_smem(ry, rx, mx, my);
        const int per_sm = ry * rx <= 25 && 3 * (smem + 2048u) <= 228u * 1024u ? 3 : 2;
        const int grid = max(1, min(total_items, per_sm * num_sms()));
        prof_mark(kProfFwd, 0, s);
        kernel<<<grid, NT, smem, s>>>(jobs_dev, items, total_items, counter, mx, my);
        PBD_LAUNCH_CHECK();
        prof_mark(kProfFwd, 1, s);
    }
    int max_blocks = 1;
    for (int j = 0; j < n_jobs; ++j) {
        const size_t n = (size_t)jobs_host[j].nx * jobs_host[j].ny * jobs_host[j].nz;
        max_blocks = max(max_blocks, (int)std::min<size_t>((n + 255) / 256, 4096));
    }
    const int fin_blocks = with_loss ? kLossBlocks : max_blocks;
    fwd_finalize_kernel<<<dim3(fin_blocks, n_jobs), 256, 0, s>>>(jobs_dev, with_loss, err);
    PBD_LAUNCH_CHECK();
    count_launch(3);
    return PBD_OK;
}

}  // namespace pbd
