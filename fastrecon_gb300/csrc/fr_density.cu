// fr_density.cu -- sample-density features for the learned DCF.  No
// counterpart in the reference.
//
// Every sample is binned to its nearest grid cell (floor(x + 0.5) of the
// plan's normalised coordinate, clamped to the grid), the per-cell counts are
// turned into a summed-area table (inclusive prefix sums along x, y, z), and
// the number of samples in the (2r+1)^d box around each sample's cell is read
// from the table with 2^d corner lookups.  Counts are exact integers.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "fr_device.cuh"
#include "fr_internal.h"

namespace fr {
namespace {

constexpr int kMaxRadii = 8;

struct Radii {
    int r[kMaxRadii];
    int n;
};

__device__ __forceinline__ int nearest_cell(float x, int G)
{
    const int c = f2i_ref(floorf(__fadd_rn(x, 0.5f)));
    return min(max(c, 0), G - 1);
}

// Samples per cell.  Every readout crosses the k-space centre, so a few cells
// take one sample of each: counted straight into global memory their atomics
// queue up (20,000 spokes: 110 us, most of it that queue).  A CTA first counts
// in a table of its own (a slot belongs to the first cell that maps to it; the
// cells every readout shares are there from the first readouts on), and adds
// the slots to the grid at the end; cells without a slot go straight there.
// 5.1 M samples on a 320^3 grid: 49 us.
constexpr int kHistThreads = 1024, kHistSlots = 4096;

__global__ void __launch_bounds__(kHistThreads) cell_hist_kernel(const float4 *__restrict__ traj, long long n, int dim,
                                                                 int G, int *hist)
{
    __shared__ int key[kHistSlots], count[kHistSlots];
    for (int i = threadIdx.x; i < kHistSlots; i += kHistThreads) {
        key[i] = -1;
        count[i] = 0;
    }
    __syncthreads();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float4 p = traj[i];
        const int x = nearest_cell(p.x, G), y = nearest_cell(p.y, G), z = dim == 3 ? nearest_cell(p.z, G) : 0;
        const int cell = (z * G + y) * G + x;  // fewer than 2^31 cells
        const unsigned slot = ((unsigned)cell * 2654435761u) >> 20;
        int k = key[slot];
        if (k == -1) {
            k = atomicCAS(&key[slot], -1, cell);
            if (k == -1) k = cell;
        }
        if (k == cell)
            atomicAdd(&count[slot], 1);
        else
            atomicAdd(&hist[cell], 1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kHistSlots; i += kHistThreads)
        if (count[i]) atomicAdd(&hist[key[i]], count[i]);
}
static_assert(kHistSlots == 1 << 12, "the slot is the hash's top 12 bits");

// Inclusive scan along x: one warp per row.
__global__ void scan_x_kernel(int *a, long long rows, int G)
{
    const int lane = threadIdx.x & 31;
    const long long warp = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long r = warp; r < rows; r += nwarps) {
        int *row = a + r * G;
        int carry = 0;
        for (int b = 0; b < G; b += 32) {
            int v = b + lane < G ? row[b + lane] : 0;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, v, d);
                if (lane >= d) v += u;
            }
            v += carry;
            if (b + lane < G) row[b + lane] = v;
            carry = __shfl_sync(0xffffffffu, v, 31);
        }
    }
}

// Inclusive scan along x and y of the planes of a 3D grid in one pass, a CTA
// per plane: thread = x (G <= 1024), the warps' totals through shared memory,
// kRows rows at a time, the next kRows' loads in flight, the column sums in a
// register.  Bound: HBM.  320^3: 197 us as a scan along x and one along y, 78
// us so.  (2D has one plane, and takes the two.)
constexpr int kRows = 8;
__global__ void scan_xy_kernel(int *a, int G)
{
    __shared__ int tot[2][kRows][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5, x = threadIdx.x;
    int *plane = a + (size_t)blockIdx.x * G * G;
    int col = 0, buf = 0, next[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) next[r] = x < G && r < G ? plane[(size_t)r * G + x] : 0;
    for (int y0 = 0; y0 < G; y0 += kRows, buf ^= 1) {
        int v[kRows];
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            v[r] = next[r];
            const int y = y0 + kRows + r;
            next[r] = x < G && y < G ? plane[(size_t)y * G + x] : 0;
        }
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, v[r], d);
                if (lane >= d) v[r] += u;
            }
            if (lane == 31) tot[buf][r][warp] = v[r];
        }
        __syncthreads();  // the other buffer is written only after the next one
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            col += v[r] + __reduce_add_sync(0xffffffffu, lane < min(warp, nw) ? tot[buf][r][lane] : 0);
            if (x < G && y0 + r < G) plane[(size_t)(y0 + r) * G + x] = col;
        }
    }
}

// Inclusive scan along an outer axis: thread per column, sequential along
// the axis (stride `step` elements), consecutive threads on consecutive x,
// kAhead loads in flight.  320^3 along z: 149 us with one in flight, 51 us so.
constexpr int kAhead = 8;
__global__ void scan_outer_kernel(int *a, long long columns, int len, long long step, long long plane)
{
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < columns;
         c += (long long)gridDim.x * blockDim.x) {
        // column c: x = c % step within a plane block, block = c / step
        int *p = a + (c / step) * plane + (c % step);
        int acc = 0;
        for (int k0 = 0; k0 < len; k0 += kAhead) {
            int v[kAhead];
#pragma unroll
            for (int k = 0; k < kAhead; ++k) v[k] = k0 + k < len ? p[(size_t)(k0 + k) * step] : 0;
#pragma unroll
            for (int k = 0; k < kAhead; ++k) {
                acc += v[k];
                if (k0 + k < len) p[(size_t)(k0 + k) * step] = acc;
            }
        }
    }
}

// Samples in the boxes of every radius around a sample's cell, from the table's
// corners.  Two lanes a sample, one for each end of the boxes in x: the two corners of
// a row are 2 r + 1 cells apart, mostly in one 128-byte line, which one load of the
// pair then touches once; four radii's corners in flight.  Bound: the lines a
// load touches, one a cycle and SM.  5.1 M samples, 320^3 table, radii 1, 2, 4, 8:
// 488 us with a thread a sample and eight corners in flight, 398 us so.
// (Whole numbers modulo 2^32: the differences are counts below it.)
constexpr int kBoxRadii = 4;
__global__ void __launch_bounds__(256) box_count_kernel(const float4 *__restrict__ traj, long long n, int dim, int G,
                                                        const int *__restrict__ sat, Radii R, int *__restrict__ counts)
{
    const int upper = threadIdx.x & 1;
    const long long pairs = (long long)gridDim.x * (blockDim.x / 2);
    // all lanes of a warp go round together (the pair meets by a shuffle)
    for (long long b = blockIdx.x * (long long)(blockDim.x / 2) + (threadIdx.x & ~31u) / 2; b < n; b += pairs) {
        const long long i = b + (threadIdx.x & 31) / 2;
        const bool live = i < n;
        const float4 p = live ? traj[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        const int cx = nearest_cell(p.x, G), cy = nearest_cell(p.y, G), cz = dim == 3 ? nearest_cell(p.z, G) : 0;
        for (int k0 = 0; k0 < R.n; k0 += kBoxRadii) {
            unsigned v[kBoxRadii];
#pragma unroll
            for (int k = 0; k < kBoxRadii; ++k) {
                const int r = k0 + k < R.n ? R.r[k0 + k] : 0;
                const int x = upper ? min(cx + r, G - 1) : max(cx - r, 0) - 1;
                const int y0 = max(cy - r, 0) - 1, y1 = min(cy + r, G - 1);
                const int z0 = dim == 3 ? max(cz - r, 0) - 1 : -1, z1 = dim == 3 ? min(cz + r, G - 1) : 0;
                const bool on = live && k0 + k < R.n && x >= 0;  // a corner before the table counts nothing
                auto at = [&](int y, int z) {
                    return on && y >= 0 && z >= 0 ? (unsigned)__ldg(&sat[((size_t)z * G + y) * G + x]) : 0u;
                };
                v[k] = (at(y1, z1) - at(y0, z1)) - (at(y1, z0) - at(y0, z0));
            }
#pragma unroll
            for (int k = 0; k < kBoxRadii; ++k) {
                const unsigned other = __shfl_xor_sync(0xffffffffu, v[k], 1);
                // half of the radii are written by each lane
                if (live && k0 + k < R.n && (k >= kBoxRadii / 2) == (upper != 0))
                    counts[i * R.n + k0 + k] = (int)(upper ? v[k] - other : other - v[k]);
            }
        }
    }
}

// max |k| of the raw coordinates (non-negative floats order like their bits)
__global__ void kmax_kernel(const float4 *__restrict__ traj, long long n, int dim, unsigned *out)
{
    float m = 0.f;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float4 p = traj[i];
        float q = __fmul_rn(p.x, p.x);
        if (dim >= 2) q = __fadd_rn(q, __fmul_rn(p.y, p.y));
        if (dim >= 3) q = __fadd_rn(q, __fmul_rn(p.z, p.z));
        m = fmaxf(m, __fsqrt_rn(q));
    }
    __shared__ unsigned part[32];
    const unsigned w = __reduce_max_sync(0xffffffffu, __float_as_uint(m));  // m >= 0
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = w;
    __syncthreads();
    if (threadIdx.x < 32) {
        const unsigned b = __reduce_max_sync(0xffffffffu, threadIdx.x < blockDim.x / 32 ? part[threadIdx.x] : 0u);
        if (threadIdx.x == 0) atomicMax(out, b);
    }
}

__global__ void features_kernel(const int *__restrict__ counts, const float4 *__restrict__ traj, long long n, int dim,
                                Radii R, const unsigned *kmax_bits, float kmax_given, float *feat)
{
    const float kmax = kmax_bits ? __uint_as_float(*kmax_bits) : kmax_given;
    const int nf = R.n + 1;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        for (int k = 0; k < R.n; ++k) {
            const float side = (float)(2 * R.r[k] + 1);
            const float vol = dim == 3 ? __fmul_rn(__fmul_rn(side, side), side) : __fmul_rn(side, side);
            feat[i * nf + k] = logf(__fdiv_rn((float)counts[i * R.n + k], vol));
        }
        const float4 p = traj[i];
        float q = __fmul_rn(p.x, p.x);
        if (dim >= 2) q = __fadd_rn(q, __fmul_rn(p.y, p.y));
        if (dim >= 3) q = __fadd_rn(q, __fmul_rn(p.z, p.z));
        feat[i * nf + R.n] = logf(__fadd_rn(__fdiv_rn(__fsqrt_rn(q), kmax), 0.0009765625f));
    }
}

int blocks_for(long long n, int threads)
{
    int dev = 0, sms = 132;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return (int)std::max<long long>(1, std::min<long long>((n + threads - 1) / threads, (long long)sms * 16));
}

int sm_count_density()
{
    int dev = 0, sms = 132;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

int make_radii(const int *radii, int nradii, Radii *R)
{
    if (nradii < 1 || nradii > kMaxRadii || !radii) return fail(FR_ERR_INVALID_ARGUMENT, "1 to 8 radii");
    R->n = nradii;
    for (int k = 0; k < nradii; ++k) {
        if (radii[k] < 0 || radii[k] > 4096) return fail(FR_ERR_INVALID_ARGUMENT, "radius out of range");
        R->r[k] = radii[k];
    }
    return FR_OK;
}

}  // namespace

int density_counts_run(fr_plan p, const int *radii, int nradii, int *d_counts, cudaStream_t s)
{
    if (!p->planned) return fail(FR_ERR_NOT_PLANNED, "fr_density_counts called before fr_plan_set_trajectory");
    Radii R;
    int st = make_radii(radii, nradii, &R);
    if (st) return st;
    if (p->n == 0) return FR_OK;
    const int G = (int)p->G;
    const size_t cells = p->dim == 3 ? (size_t)G * G * G : (size_t)G * G;
    if (cells > 0x7FFFFFFFull) return fail(FR_ERR_UNSUPPORTED, "grid too large for the density table");
    if (p->density_sat.reserve(cells * 4)) return FR_ERR_CUDA;
    int *sat = p->density_sat.as<int>();
    FR_CUDA(cudaMemsetAsync(sat, 0, cells * 4, s));
    const long long n = (long long)p->n;
    const float4 *traj = p->traj.as<float4>();
    cell_hist_kernel<<<(int)std::min<long long>((n + kHistThreads - 1) / kHistThreads, sm_count_density()), kHistThreads, 0,
                       s>>>(traj, n, p->dim, G, sat);
    FR_CHECK_LAUNCH("cell_hist_kernel");
    if (p->dim == 3 && G <= 1024) {
        scan_xy_kernel<<<G, (G + 31) & ~31, 0, s>>>(sat, G);
        FR_CHECK_LAUNCH("scan_xy_kernel");
    } else {
        const long long rows = (long long)(cells / G), gz = p->dim == 3 ? G : 1;
        scan_x_kernel<<<blocks_for(rows * 32, 256), 256, 0, s>>>(sat, rows, G);
        FR_CHECK_LAUNCH("scan_x_kernel");
        // y: columns (z, x), stride G, planes of G*G
        scan_outer_kernel<<<blocks_for(gz * G, 128), 128, 0, s>>>(sat, gz * G, G, G, (long long)G * G);
        FR_CHECK_LAUNCH("scan_outer_kernel");
    }
    if (p->dim == 3) {  // z: columns (y, x), stride G*G
        scan_outer_kernel<<<blocks_for((long long)G * G, 128), 128, 0, s>>>(sat, (long long)G * G, G, (long long)G * G, 0);
        FR_CHECK_LAUNCH("scan_outer_kernel");
    }
    box_count_kernel<<<blocks_for(2 * n, 256), 256, 0, s>>>(traj, n, p->dim, G, sat, R, d_counts);
    FR_CHECK_LAUNCH("box_count_kernel");
    return FR_OK;
}

int dcf_features_run(const int *d_counts, const float *d_raw, size_t n, int dim, const int *radii, int nradii,
                     float kmax, float *d_feat, unsigned *d_scratch, cudaStream_t s)
{
    Radii R;
    int st = make_radii(radii, nradii, &R);
    if (st) return st;
    if (n == 0) return FR_OK;
    const float4 *traj = reinterpret_cast<const float4 *>(d_raw);
    const unsigned *kb = nullptr;
    if (!(kmax > 0.f)) {
        FR_CUDA(cudaMemsetAsync(d_scratch, 0, 4, s));
        kmax_kernel<<<std::min(blocks_for((long long)n, 512), sm_count_density() * 4), 512, 0, s>>>(traj, (long long)n, dim, d_scratch);
        FR_CHECK_LAUNCH("kmax_kernel");
        kb = d_scratch;
    }
    features_kernel<<<blocks_for((long long)n, 256), 256, 0, s>>>(d_counts, traj, (long long)n, dim, R, kb, kmax,
                                                                  d_feat);
    FR_CHECK_LAUNCH("features_kernel");
    return FR_OK;
}

}  // namespace fr
