// fr_dcf.cu -- density compensation and degridding.  No counterpart in the
// reference, which reads its DCF from a file (ReconData.cpp:108-121) and has
// no interpolation from the grid back to the samples.
//
//  * fr_dcf_analytic: |k|^p of the raw coordinates (|k| for 2D radial, |k|^2
//    for 3D radial), computed in double like the CPU restatement.
//  * fr_degrid: interpolation of a multi-coil grid at the samples, the adjoint
//    of gridding (same clamped cell range and exact LUT index as the scatter,
//    GridLut.cpp:98-136).  Tile by tile: a part of a tile's cells, all coils,
//    in shared memory, a few lanes per sample.  Kernels wider than 5 cells and
//    trajectories with few samples per tile: a thread per sample and block of
//    coils, the grid read through L1/L2.
//  * Pipe-Menon DCF (Pipe & Menon, MRM 41:179-186, 1999):
//        w <- w / (C w),  C w = degrid(grid(w)),
//    with grid(w) a real-valued tile scatter over the plan's bins, from its
//    tap lists where it has them (shared-memory accumulation, one flush per
//    tile, no global atomics) and the degridding fused with the division.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "fr_device.cuh"
#include "fr_internal.h"

namespace fr {
namespace {

// Weight of a tap at squared distance s2 from the exact LUT-index table
// {thr[k+1], lut[k], lut[k+1], 0}: returns false outside the kernel radius.
__device__ __forceinline__ bool lut_weight(float s2, const float4 *lutS, float smax, float kc, int L, float &w)
{
    if (!(s2 < smax)) return false;
    float a;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(a) : "f"(s2));
    const int k0 = min((int)fmaf(a, kc, 0.25f), L - 1);
    const float4 en = lutS[k0];
    w = s2 >= en.x ? en.z : en.y;
    return true;
}

// -- analytic DCF -----------------------------------------------------------
__global__ void dcf_analytic_kernel(const float4 *__restrict__ traj, long long n, int dim, double power, int mode,
                                    float *__restrict__ out)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float4 p = traj[i];
        double q = __dmul_rn((double)p.x, (double)p.x);
        if (dim >= 2) q = __dadd_rn(q, __dmul_rn((double)p.y, (double)p.y));
        if (dim >= 3) q = __dadd_rn(q, __dmul_rn((double)p.z, (double)p.z));
        const double k = __dsqrt_rn(q);
        const double w = mode == 1 ? k : (mode == 2 ? __dmul_rn(k, k) : pow(k, power));
        out[i] = __double2float_rn(w);
    }
}

// -- degridding ---------------------------------------------------------------
struct DegridParams {
    const float4 *traj;  // normalised
    long long n;
    int dim, G;
    float hw;
    int L;
    float smax, kc;
    const float4 *lut_e;
    const float2 *grid;  // channels x cells
    int channels;
    long long cells;
    int checkerboard;
    float2 *out;         // channels x n
};

template <int CB>
__global__ void __launch_bounds__(256) degrid_kernel(DegridParams P)
{
    extern __shared__ float4 lutS[];
    for (int i = threadIdx.x; i < P.L; i += blockDim.x) lutS[i] = P.lut_e[i];
    __syncthreads();
    const int c0 = blockIdx.y * CB;
    const size_t G = (size_t)P.G;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < P.n;
         i += (long long)gridDim.x * blockDim.x) {
        const float4 p = P.traj[i];
        int xs, xe, ys, ye, zs = 0, ze = 0;
        comp_range(p.x, P.hw, P.G, xs, xe);
        comp_range(p.y, P.hw, P.G, ys, ye);
        if (P.dim == 3) comp_range(p.z, P.hw, P.G, zs, ze);
        float2 acc[CB];
#pragma unroll
        for (int c = 0; c < CB; ++c) acc[c] = make_float2(0.f, 0.f);
        for (int z = zs; z <= ze; ++z) {
            const float dz = P.dim == 3 ? __fsub_rn((float)z, p.z) : 0.f;
            const float dz2 = __fmul_rn(dz, dz);
            for (int y = ys; y <= ye; ++y) {
                const float dy = __fsub_rn((float)y, p.y);
                const float dzy = __fadd_rn(dz2, __fmul_rn(dy, dy));
                const size_t row = ((size_t)z * G + (size_t)y) * G;
                for (int x = xs; x <= xe; ++x) {
                    const float dx = __fsub_rn((float)x, p.x);
                    float w;
                    if (!lut_weight(__fadd_rn(dzy, __fmul_rn(dx, dx)), lutS, P.smax, P.kc, P.L, w)) continue;
                    if (P.checkerboard && ((x + y + z) & 1)) w = -w;
#pragma unroll
                    for (int c = 0; c < CB; ++c) {
                        if (c0 + c < P.channels) {
                            const float2 g = P.grid[(size_t)(c0 + c) * P.cells + row + x];
                            acc[c].x = fmaf(w, g.x, acc[c].x);
                            acc[c].y = fmaf(w, g.y, acc[c].y);
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int c = 0; c < CB; ++c)
            if (c0 + c < P.channels) P.out[(size_t)(c0 + c) * P.n + i] = acc[c];
    }
}

// The cells of a footprint along one axis: clamped range (GridLut.cpp:98-106),
// ends at distance kHW dropped where that is exact (they never pass dk < kHW).
__device__ __forceinline__ void footprint(const DegridParams &P, int trim, float c, int &s, int &e)
{
    comp_range(c, P.hw, P.G, s, e);
    if (trim && s <= e) {
        if (!(fabsf(__fsub_rn((float)s, c)) < P.hw)) ++s;
        if (s <= e && !(fabsf(__fsub_rn((float)e, c)) < P.hw)) --e;
    }
}

// Degridding from shared memory.  A CTA takes one part (`box` cells) of one
// work item's tile and one group of coils: it stages the cells that samples
// starting in the part can reach as [cell][coil] (each value of the grid is
// read from its plane once, not once per tap), collects the item's samples
// that start there, and gives each sample LP lanes, two coils a lane.  Per
// plane of a footprint the lanes share the R x R candidates' geometry, list the
// taps inside the radius, and add weight x cell from the list, in the order of
// degrid_kernel.
// Cells are 4 * odd floats apart, so that staging (lanes along x) covers the
// banks; LP = 8 lanes read one cell's 128 bytes at a time.
// Bound: issue (geometry and list a quarter of it), barriers between scan, staging
// and sums, the shared pipe (a cell row per tap), staging (a part's halo: a
// 4 x 8 x 8 part of 12 coils reads 2.5 times its cells).  1.9 M samples, 12 coils,
// 192^3 grid: 3034 us with a thread per sample and 4 coils gathering from the
// planes through L1, 1166 us so (53 % issue, 51 % of the shared pipe).
struct TileDegrid {
    const unsigned long long *recs;
    const WorkItem *items;
    int tile[3], ntile[3];
    int box[3], nbox[3];  // part of a tile, parts per tile
    int trim;
    int coils;            // coils per group (even)
    int stride;           // floats per staged cell
    const float *lutw;
};
constexpr int kDegridThreads = 512;
constexpr int kDegridRound = 512;    // records looked at between two barriers
__host__ __device__ constexpr int degrid_list(int R) { return ((R * R + 3) & ~3) + 2; }  // list entries per sample

template <int LP, int R>
__global__ void __launch_bounds__(kDegridThreads, 2) degrid_tiles_kernel(DegridParams P, TileDegrid T)
{
    constexpr int S = 32 / LP, NR = (R * R + LP - 1) / LP, LE = degrid_list(R);
    extern __shared__ float4 smd[];
    __shared__ int nq;
    const int B[3] = {T.box[0] + R - 1, T.box[1] + R - 1, P.dim == 3 ? T.box[2] + R - 1 : 1};
    float *blk = reinterpret_cast<float *>(smd);
    int2 *lists = reinterpret_cast<int2 *>(blk + (size_t)B[0] * B[1] * B[2] * T.stride);
    float *thr = reinterpret_cast<float *>(lists + (kDegridThreads / LP) * LE);
    float *lut = thr + P.L;
    // {sample, its footprint: first cell in the part, 6 bits an axis, cells, 3 bits};
    // 2 L floats past thr, so on 8 bytes for odd tables too
    uint2 *queue = reinterpret_cast<uint2 *>(thr + 2 * P.L);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    const WorkItem it = T.items[blockIdx.x];
    const int c0 = blockIdx.z * T.coils, nc = min(T.coils, P.channels - c0);
    int o[3], hi[3];  // first cell of the part, first past it
    {
        const int ty = it.tile / T.ntile[0], tz = ty / T.ntile[1];
        const int t3[3] = {it.tile - ty * T.ntile[0], ty - tz * T.ntile[1], tz};
        int b = blockIdx.y;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const int k = b % T.nbox[d];
            b /= T.nbox[d];
            o[d] = t3[d] * T.tile[d] + k * T.box[d];
            hi[d] = min(o[d] + T.box[d], (t3[d] + 1) * T.tile[d]);
        }
    }
    const int G = P.G, Gz = P.dim == 3 ? P.G : 1;
    bool staged = false;
    const unsigned long long *recs = T.recs + it.begin;
    for (int base = 0; base < it.count; base += kDegridRound) {
        if (tid == 0) nq = 0;
        __syncthreads();
        const int n = min(it.count - base, kDegridRound);
        for (int j = warp * 32; j < n; j += kDegridThreads) {
            bool home = false;
            unsigned sidx = 0u, fp = 0u;
            if (j + lane < n) {
                sidx = (unsigned)recs[base + j + lane];
                const float4 p = P.traj[sidx];
                const float c[3] = {p.x, p.y, p.z};
                int st[3] = {0, 0, 0}, e[3] = {0, 0, 0};
                bool some = true;
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    if (d < P.dim) {
                        footprint(P, T.trim, c[d], st[d], e[d]);
                        some = some && st[d] <= e[d];
                    }
                if (!some) {  // no taps: its untrimmed start is still in exactly one tile
#pragma unroll
                    for (int d = 0; d < 3; ++d)
                        if (d < P.dim) {
                            comp_range(c[d], P.hw, P.G, st[d], e[d]);
                            e[d] = st[d] - 1;
                        }
                }
                home = true;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    home = home && st[d] >= o[d] && st[d] < hi[d];
                    fp |= (unsigned)(st[d] - o[d]) << (6 * d) | (unsigned)(e[d] - st[d] + 1) << (18 + 3 * d);
                }
            }
            const unsigned m = __ballot_sync(0xffffffffu, home);
            int at = 0;
            if (lane == 0 && m) at = atomicAdd(&nq, __popc(m));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (home) queue[at + __popc(m & ((1u << lane) - 1u))] = make_uint2(sidx, fp);
        }
        __syncthreads();
        const int count = nq;
        if (count > 0 && !staged) {
            staged = true;
            for (int i = tid; i < P.L; i += kDegridThreads) {
                thr[i] = P.lut_e[i].x;
                lut[i] = T.lutw[i];
            }
            // a row of the block per 16 lanes, coil after coil; the copies are
            // asynchronous (all of a thread's are in flight at once)
            for (int r = tid >> 4; r < B[1] * B[2]; r += kDegridThreads / 16) {
                const int lz = r / B[1], ly = r - lz * B[1];
                const bool row = o[1] + ly < G && o[2] + lz < Gz;
                for (int lx = tid & 15; lx < B[0]; lx += 16) {
                    const bool in = row && o[0] + lx < G;
                    const float2 *src = P.grid + (size_t)c0 * P.cells +
                                        (in ? ((size_t)(o[2] + lz) * G + (o[1] + ly)) * (size_t)G + (o[0] + lx) : 0);
                    float *dst = blk + (size_t)(r * B[0] + lx) * T.stride;
                    unsigned d = (unsigned)__cvta_generic_to_shared(dst);
                    for (int c = 0; c < T.coils; ++c, d += 8, src += P.cells) {
                        // past the grid or the last coil: nothing is read, zeros are written
                        const bool some = in && c < nc;
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d),
                                     "l"(some ? src : P.grid), "r"(some ? 8 : 0)
                                     : "memory");
                    }
                }
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
        }
        const int l = lane % LP, g = lane / LP;
        const bool mine = 2 * l < T.coils;  // this lane's coils c0 + 2 l, c0 + 2 l + 1
        int2 *list = lists + (warp * S + g) * LE;
        for (int q0 = warp * S; q0 < count; q0 += (kDegridThreads / 32) * S) {
            const bool live = q0 + g < count;
            const uint2 qe = queue[live ? q0 + g : q0];
            const unsigned sidx = qe.x, fp = qe.y;
            const float4 p = P.traj[sidx];
            const int bx = fp & 63, by = (fp >> 6) & 63, bz = (fp >> 12) & 63;
            const int nx = (fp >> 18) & 7, ny = (fp >> 21) & 7, nz = (fp >> 24) & 7;
            // the lane's candidates of a plane: l, l + LP, ... (x fastest)
            float dx2[NR], dy2[NR];
            int off[NR];
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const int k = l + LP * r, iy = k / R, ix = k - iy * R;
                const float dx = __fsub_rn((float)(o[0] + bx + ix), p.x), dy = __fsub_rn((float)(o[1] + by + iy), p.y);
                dx2[r] = ix < nx && iy < ny ? __fmul_rn(dx, dx) : __int_as_float(0x7f800000);
                dy2[r] = __fmul_rn(dy, dy);
                // byte offset in a plane of the block, parity of x + y above
                off[r] = ((by + iy) * B[0] + bx + ix) * T.stride * 4 +
                         (P.checkerboard ? (o[0] + bx + ix + o[1] + by + iy) & 1 : 0);
            }
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
            for (int iz = 0; iz < (P.dim == 3 ? R : 1); ++iz) {
                const int z = o[2] + bz + iz;
                const float dz = P.dim == 3 ? __fsub_rn((float)z, p.z) : 0.f;
                const float dz2 = iz < nz ? __fmul_rn(dz, dz) : __int_as_float(0x7f800000);
                const int plane = (bz + iz) * B[0] * B[1] * T.stride * 4;
                const int zodd = P.checkerboard ? z & 1 : 0;
                int nt = 0;
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    const float s2 = __fadd_rn(__fadd_rn(dz2, dy2[r]), dx2[r]);
                    const bool ok = live && s2 < P.smax;
                    const unsigned m = (__ballot_sync(0xffffffffu, ok) >> (g * LP)) & ((1u << LP) - 1u);
                    if (ok) {
                        float a;
                        asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(a) : "f"(s2));
                        const int k0 = min((int)fmaf(a, P.kc, 0.25f), P.L - 1);
                        const float wt = lut[k0 + (s2 >= thr[k0] ? 1 : 0)];  // thr[L - 1] is +inf
                        list[nt + __popc(m & ((1u << l) - 1u))] =
                            make_int2((off[r] & ~1) + plane, __float_as_int((off[r] ^ zodd) & 1 ? -wt : wt));
                    }
                    nt += __popc(m);
                }
                __syncwarp();
                if (mine) {
                    const char *cell = reinterpret_cast<const char *>(blk + 4 * l);
                    auto add = [&](int at, float w) {
                        const float4 v = *reinterpret_cast<const float4 *>(cell + at);
                        acc.x = fmaf(w, v.x, acc.x);
                        acc.y = fmaf(w, v.y, acc.y);
                        acc.z = fmaf(w, v.z, acc.z);
                        acc.w = fmaf(w, v.w, acc.w);
                    };
                    int k = 0;
#pragma unroll 2
                    for (; k + 2 <= nt; k += 2) {
                        const int4 e = *reinterpret_cast<const int4 *>(list + k);
                        add(e.x, __int_as_float(e.y));
                        add(e.z, __int_as_float(e.w));
                    }
                    if (k < nt) add(list[k].x, __int_as_float(list[k].y));
                }
                __syncwarp();
            }
            if (live && 2 * l < nc) {
                float2 *out = P.out + (size_t)(c0 + 2 * l) * P.n + sidx;
                *out = make_float2(acc.x, acc.y);
                if (2 * l + 1 < nc) out[P.n] = make_float2(acc.z, acc.w);
            }
        }
        __syncthreads();
    }
}

// Samples without a cell in reach have no bin record: their values are zero.
__global__ void __launch_bounds__(256) degrid_outside_kernel(DegridParams P)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < P.n;
         i += (long long)gridDim.x * blockDim.x) {
        const float4 p = P.traj[i];
        int s, e;
        comp_range(p.x, P.hw, P.G, s, e);
        bool out = s > e;
        comp_range(p.y, P.hw, P.G, s, e);
        out = out || s > e;
        if (P.dim == 3) {
            comp_range(p.z, P.hw, P.G, s, e);
            out = out || s > e;
        }
        if (out)
            for (int c = 0; c < P.channels; ++c) P.out[(size_t)c * P.n + i] = make_float2(0.f, 0.f);
    }
}

// -- streaming acquisition: incremental regridding -----------------------------
// The gridded change dcf * (new - old) of the samples [begin, begin + count)
// added into the grid with global atomic adds, and the new values put in the
// old ones' place: a warp per sample, the same cell range, LUT index and
// checkerboard signs as the scatter and the degridding.  A lane per cell of the
// footprint (x fastest: 4 lanes of a row share its sectors), so that the
// weights are computed once for all coils; a lane per coil for the values,
// which the warp broadcasts coil by coil; (re, im) in one 8-byte reduction.
// Bound: the L2's reductions.  12,288 samples, 16 coils, 192^3 grid: 93 us with a
// thread per sample and 4 coils (192 CTAs, scalar adds, and a copy after it),
// 31 us so (with the copy 104 -> 33).
struct UpdateParams {
    DegridParams g;          // geometry, LUT, grid size, checkerboard flag
    float2 *old_k;           // channels x n: the k-space the grid was made from, updated
    const float2 *new_k;     // channels x count: the new values
    const float *dcf;        // n
    float2 *grid;            // channels x cells
    long long begin, count;
};
constexpr int kUpdateWarps = 8;

__device__ __forceinline__ void red_add2(float2 *p, float x, float y)
{
    asm volatile("red.relaxed.gpu.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(x), "f"(y) : "memory");
}

__global__ void __launch_bounds__(kUpdateWarps * 32) grid_update_kernel(UpdateParams U)
{
    extern __shared__ float4 lutS[];
    const DegridParams &P = U.g;
    for (int i = threadIdx.x; i < P.L; i += blockDim.x) lutS[i] = P.lut_e[i];
    __syncthreads();
    const size_t G = (size_t)P.G;
    const int lane = threadIdx.x & 31;
    for (long long i = blockIdx.x * (long long)kUpdateWarps + (threadIdx.x >> 5); i < U.count;
         i += (long long)gridDim.x * kUpdateWarps) {
        const long long sidx = U.begin + i;
        const float4 p = P.traj[sidx];
        const float d = U.dcf[sidx];
        int xs, xe, ys, ye, zs = 0, ze = 0;
        comp_range(p.x, P.hw, P.G, xs, xe);
        comp_range(p.y, P.hw, P.G, ys, ye);
        if (P.dim == 3) comp_range(p.z, P.hw, P.G, zs, ze);
        const int nx = max(xe - xs + 1, 0), ny = max(ye - ys + 1, 0), nz = max(ze - zs + 1, 0);
        const int ncell = nx * ny * nz;
        for (int c0 = 0; c0 < P.channels; c0 += 32) {
            float2 v = make_float2(0.f, 0.f);
            if (c0 + lane < P.channels) {
                const float2 a = U.new_k[(size_t)(c0 + lane) * U.count + i];
                float2 *o = U.old_k + (size_t)(c0 + lane) * P.n + sidx;
                const float2 b = *o;
                v = make_float2(__fmul_rn(d, __fsub_rn(a.x, b.x)), __fmul_rn(d, __fsub_rn(a.y, b.y)));
                *o = a;
            }
            const int nc = min(32, P.channels - c0);
            for (int k0 = 0; k0 < ncell; k0 += 32) {
                const int k = k0 + lane;
                bool ok = k < ncell;
                float w = 0.f;
                float2 *cell = U.grid;
                if (ok) {
                    const int r = k / nx, ix = k - r * nx, iz = r / ny, iy = r - iz * ny;
                    const int x = xs + ix, y = ys + iy, z = zs + iz;
                    const float dx = __fsub_rn((float)x, p.x), dy = __fsub_rn((float)y, p.y);
                    const float dz = P.dim == 3 ? __fsub_rn((float)z, p.z) : 0.f;
                    const float dzy = __fadd_rn(__fmul_rn(dz, dz), __fmul_rn(dy, dy));
                    ok = lut_weight(__fadd_rn(dzy, __fmul_rn(dx, dx)), lutS, P.smax, P.kc, P.L, w);
                    if (P.checkerboard && ((x + y + z) & 1)) w = -w;
                    cell += (size_t)c0 * P.cells + ((size_t)z * G + (size_t)y) * G + (size_t)x;
                }
                for (int c = 0; c < nc; ++c, cell += P.cells) {
                    const float vx = __shfl_sync(0xffffffffu, v.x, c), vy = __shfl_sync(0xffffffffu, v.y, c);
                    if (ok) red_add2(cell, __fmul_rn(w, vx), __fmul_rn(w, vy));
                }
            }
        }
    }
}

// -- real-valued tile scatter of per-sample weights ---------------------------
struct RealGridParams {
    const float4 *traj;
    const unsigned long long *recs;
    const WorkItem *items;
    const SplitTile *splits;
    const float *w;
    const float4 *lut_e;
    float *grid;      // G^d floats
    float *partials;  // nslots x K floats
    int dim, G, L;
    int tile[3], ntile[3], K;
    float smax, kc;
    // the plan's tap lists (grid_real_taps_kernel)
    const unsigned long long *trecs;  // sample | first word << 32 | taps << 40
    const unsigned *taps;
    const float *lutw;  // L weights
    int tap_words;
};

constexpr int kRealWarps = 8;

// The scatter from the plan's tap lists.  A warp holds 32 records, numbers
// their groups of 4 taps by a warp scan and deals them 32 per pass, so that
// every lane has taps to add whatever the records' boxes are (a warp per
// record, as in grid_real_kernel, leaves most lanes without a tap and spends
// its time on the box arithmetic).  A lane's group is one 16-byte load when
// its run starts on a 4-word boundary.  CTAs take work items in turn, so that
// the weights and the cells' grid offsets (`offs`) are staged once, not per
// item: most items are a few hundred records.
// Bound: the shared pipe (table reads at random banks and the float adds,
// which are compare-and-swap loops), 66 % busy; then the tap words' bytes
// (about 170 B a sample).  3.1 M samples on a 320^3 grid: 1353 us with a warp
// per record, 500 us so.  Measured slower: 64-bit fixed-point adds (also
// compare-and-swap here, 654 us), a half-warp per record with a tile copy each
// and no atomics (845 us); two 32-bit fixed-point adds were faster (420 us) but
// hold 38 bits under the item's largest weight, too few for weights of any range.
constexpr int kRealTapWarps = 4;

__global__ void __launch_bounds__(kRealTapWarps * 32) grid_real_taps_kernel(RealGridParams P, int nitems)
{
    extern __shared__ float4 smr[];
    __shared__ int4 table[kRealTapWarps][32];
    float *acc = reinterpret_cast<float *>(smr);
    int *offs = reinterpret_cast<int *>(acc + P.K);
    float *lutw = reinterpret_cast<float *>(offs + P.K);
    const int Tx = P.tile[0], Ty = P.tile[1], Tz = P.tile[2];
    const size_t G = (size_t)P.G;
    const int Gz = P.dim == 3 ? P.G : 1;
    for (int i = threadIdx.x; i < P.K; i += blockDim.x) {
        const int lx = i % Tx, r = i / Tx, ly = r % Ty, lz = r / Ty;
        offs[i] = (lz * P.G + ly) * P.G + lx;  // below 64 * 4096^2
        acc[i] = 0.f;
    }
    for (int i = threadIdx.x; i < P.L; i += blockDim.x) lutw[i] = P.lutw[i];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned cmask = (1u << kTapCellBits) - 1u;
    __syncthreads();
    for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
        const WorkItem it = P.items[item];
        const unsigned long long *trecs = P.trecs + it.begin;
        for (int j0 = warp * 32; j0 < it.count; j0 += kRealTapWarps * 32) {
            const unsigned long long rw = j0 + lane < it.count ? __ldg(trecs + j0 + lane) : 0ull;
            const int nt = (int)((rw >> 40) & 0xFF);
            const int np = (nt + 3) >> 2;
            const unsigned nz = __ballot_sync(0xffffffffu, np > 0);
            int incl = np;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const int excl = incl - np;
            const int total = __shfl_sync(0xffffffffu, incl, 31);
            if (np > 0)
                table[warp][__popc(nz & ((1u << lane) - 1u))] =
                    make_int4((int)(unsigned)rw, (int)(((rw >> 32) & 0xFF) | ((unsigned)nt << 8)), excl,
                              __float_as_int(P.w[(unsigned)rw]));
            __syncwarp();
            int recbase = 0;
            for (int p0 = 0; p0 < total; p0 += 32) {
                // bit i of starts: a record's first group is group p0 + i
                const bool in_pass = np > 0 && excl >= p0 && excl < p0 + 32;
                const unsigned starts = __reduce_or_sync(0xffffffffu, in_pass ? 1u << (excl - p0) : 0u);
                const int cr = recbase + __popc(starts & (0xffffffffu >> (31 - lane))) - 1;
                recbase += __popc(starts);
                if (p0 + lane < total) {
                    const int4 e = table[warp][cr];
                    const int gi = 4 * (p0 + lane - e.z);
                    const int nl = min((e.y >> 8) - gi, 4);
                    const size_t tb = (size_t)(unsigned)e.x * (size_t)P.tap_words + (size_t)((e.y & 0xFF) + gi);
                    unsigned tg[4] = {0u, 0u, 0u, 0u};
                    if ((tb & 3) == 0) {  // slots are multiples of 4 words: the group stays in the slot
                        const uint4 q = __ldg(reinterpret_cast<const uint4 *>(P.taps + tb));
                        tg[0] = q.x;
                        tg[1] = q.y;
                        tg[2] = q.z;
                        tg[3] = q.w;
                    } else {
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (k < nl) tg[k] = __ldg(P.taps + tb + k);
                    }
                    const float v = __int_as_float(e.w);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (k < nl)
                            atomicAdd(&acc[min(tg[k] & cmask, (unsigned)(P.K - 1))],
                                      lutw[min(tg[k] >> kTapCellBits, (unsigned)(P.L - 1))] * v);
                }
            }
            __syncwarp();  // the next batch rewrites the table
        }
        __syncthreads();
        // flush, and zero for the next item
        const int t = it.tile;
        const int ty = t / P.ntile[0], tz = ty / P.ntile[1];
        const int ox = (t - ty * P.ntile[0]) * Tx, oy = (ty - tz * P.ntile[1]) * Ty, oz = tz * Tz;
        float *dst = it.slot >= 0 ? P.partials + (size_t)it.slot * P.K : P.grid + ((size_t)oz * G + oy) * G + ox;
        const bool inside = ox + Tx <= P.G && oy + Ty <= P.G && oz + Tz <= Gz;
        for (int i = threadIdx.x; i < P.K; i += blockDim.x) {
            const float v = acc[i];
            acc[i] = 0.f;
            if (it.slot >= 0) {
                dst[i] = v;
            } else {
                bool in = inside;
                if (!inside) {
                    const int lx = i % Tx, r = i / Tx;
                    in = ox + lx < P.G && oy + r % Ty < P.G && oz + r / Ty < Gz;
                }
                if (in) dst[offs[i]] = v;
            }
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kRealWarps * 32) grid_real_kernel(RealGridParams P)
{
    extern __shared__ float4 smr[];
    float4 *lutS = smr;
    float *acc = reinterpret_cast<float *>(smr + P.L);
    const WorkItem it = P.items[blockIdx.x];
    const int t = it.tile;
    const int ox = (t % P.ntile[0]) * P.tile[0];
    const int oy = ((t / P.ntile[0]) % P.ntile[1]) * P.tile[1];
    const int oz = (t / (P.ntile[0] * P.ntile[1])) * P.tile[2];
    const int Tx = P.tile[0], Ty = P.tile[1], Tz = P.tile[2];
    for (int i = threadIdx.x; i < P.L; i += blockDim.x) lutS[i] = P.lut_e[i];
    for (int i = threadIdx.x; i < P.K; i += blockDim.x) acc[i] = 0.f;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned long long *recs = P.recs + it.begin;
    for (int j = warp; j < it.count; j += kRealWarps) {
        const unsigned long long rec = recs[j];
        const unsigned s = (unsigned)rec;
        const unsigned box = (unsigned)(rec >> 32);
        const int lx0 = box & 63, ly0 = (box >> 6) & 63, lz0 = (box >> 12) & 63;
        const int nx = (box >> 18) & 15, ny = (box >> 22) & 15, nz = (box >> 26) & 15;
        const int ntap = nx * ny * nz;
        if (ntap == 0) continue;
        const float4 p = P.traj[s];
        const float v = P.w[s];
        for (int tt = lane; tt < ntap; tt += 32) {
            const int ix = tt % nx, r = tt / nx, iy = r % ny, iz = r / ny;
            const int lx = lx0 + ix, ly = ly0 + iy, lz = lz0 + iz;
            const float dx = __fsub_rn((float)(ox + lx), p.x);
            const float dy = __fsub_rn((float)(oy + ly), p.y);
            const float dz = P.dim == 3 ? __fsub_rn((float)(oz + lz), p.z) : 0.f;
            const float s2 = __fadd_rn(__fadd_rn(__fmul_rn(dz, dz), __fmul_rn(dy, dy)), __fmul_rn(dx, dx));
            float w;
            if (lut_weight(s2, lutS, P.smax, P.kc, P.L, w)) atomicAdd(&acc[(lz * Ty + ly) * Tx + lx], w * v);
        }
    }
    __syncthreads();
    if (it.slot >= 0) {
        float *dst = P.partials + (size_t)it.slot * P.K;
        for (int i = threadIdx.x; i < P.K; i += blockDim.x) dst[i] = acc[i];
        return;
    }
    const size_t G = (size_t)P.G;
    const int Gz = P.dim == 3 ? P.G : 1;
    for (int i = threadIdx.x; i < P.K; i += blockDim.x) {
        const int lx = i % Tx, r = i / Tx, ly = r % Ty, lz = r / Ty;
        const int gx = ox + lx, gy = oy + ly, gz = oz + lz;
        if (gx < P.G && gy < P.G && gz < Gz && lz < Tz) P.grid[((size_t)gz * G + gy) * G + gx] = acc[i];
    }
}

__global__ void reduce_real_splits_kernel(RealGridParams P)
{
    const SplitTile st = P.splits[blockIdx.x];
    const int t = st.tile;
    const int ox = (t % P.ntile[0]) * P.tile[0];
    const int oy = ((t / P.ntile[0]) % P.ntile[1]) * P.tile[1];
    const int oz = (t / (P.ntile[0] * P.ntile[1])) * P.tile[2];
    const size_t G = (size_t)P.G;
    const int Gz = P.dim == 3 ? P.G : 1;
    const float *base = P.partials + (size_t)st.first_slot * P.K;
    for (int i = threadIdx.x; i < P.K; i += blockDim.x) {
        const int lx = i % P.tile[0], r = i / P.tile[0], ly = r % P.tile[1], lz = r / P.tile[1];
        const int gx = ox + lx, gy = oy + ly, gz = oz + lz;
        if (gx >= P.G || gy >= P.G || gz >= Gz) continue;
        // slot after slot, 8 loads in flight (3.1 M samples, 320^3: 31 -> 10 us)
        float v = 0.f;
        int k = 0;
        for (; k + 8 <= st.nslots; k += 8) {
            float a[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) a[u] = base[(size_t)(k + u) * P.K + i];
#pragma unroll
            for (int u = 0; u < 8; ++u) v = __fadd_rn(v, a[u]);
        }
        for (; k < st.nslots; ++k) v = __fadd_rn(v, base[(size_t)k * P.K + i]);
        P.grid[((size_t)gz * G + gy) * G + gx] = v;
    }
}

// Degrid a real grid at each sample and divide the sample's weight by it.
// XR >= 2 hw bounds the cells along x, whose dx^2 are computed once (+inf past
// the footprint); thresholds and weights are read as single words.
// Bound: the L1 data pipe, for the scattered rows and the weight table.  3.1 M
// samples on a 320^3 grid: 340 us with the table as float4 entries (87 % of the
// pipe), 250 us so.  Measured slower: a row's cells as two aligned float4
// (396 us), the tile's cells staged in shared memory (600 us: staging, and
// half-filled warps at a median of 119 records per tile), the tap lists (361 us).
template <int XR>
__global__ void __launch_bounds__(256) pipe_update_kernel(DegridParams P, int trim, const float *__restrict__ lutw,
                                                          const float *__restrict__ g, float *w)
{
    extern __shared__ float tabs[];  // thr [L] (index k + 1 from thr[k] on), weights [L]
    float *thr = tabs, *lut = tabs + P.L;
    for (int i = threadIdx.x; i < P.L; i += blockDim.x) {
        thr[i] = P.lut_e[i].x;
        lut[i] = lutw[i];
    }
    __syncthreads();
    const size_t G = (size_t)P.G;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < P.n;
         i += (long long)gridDim.x * blockDim.x) {
        const float4 p = P.traj[i];
        int xs, xe, ys, ye, zs = 0, ze = 0;
        footprint(P, trim, p.x, xs, xe);
        footprint(P, trim, p.y, ys, ye);
        if (P.dim == 3) footprint(P, trim, p.z, zs, ze);
        float dx2[XR];
#pragma unroll
        for (int k = 0; k < XR; ++k) {
            const float dx = __fsub_rn((float)(xs + k), p.x);
            dx2[k] = xs + k <= xe ? __fmul_rn(dx, dx) : __int_as_float(0x7f800000);
        }
        float acc = 0.f;
        for (int z = zs; z <= ze; ++z) {
            const float dz = P.dim == 3 ? __fsub_rn((float)z, p.z) : 0.f;
            const float dz2 = __fmul_rn(dz, dz);
            for (int y = ys; y <= ye; ++y) {
                const float dy = __fsub_rn((float)y, p.y);
                const float dzy = __fadd_rn(dz2, __fmul_rn(dy, dy));
                const float *row = g + ((size_t)z * G + (size_t)y) * G + xs;
#pragma unroll
                for (int k = 0; k < XR; ++k) {
                    const float s2 = __fadd_rn(dzy, dx2[k]);
                    if (s2 < P.smax) {
                        float a;
                        asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(a) : "f"(s2));
                        const int k0 = min((int)fmaf(a, P.kc, 0.25f), P.L - 1);
                        const float wt = lut[k0 + (s2 >= thr[k0] ? 1 : 0)];  // thr[L - 1] is +inf
                        acc = fmaf(wt, __ldg(row + k), acc);
                    }
                }
            }
        }
        if (acc > 0.f) w[i] = w[i] / acc;
    }
}

int sm_count()
{
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 132;
    }
    return n;
}

DegridParams degrid_params(fr_plan p)
{
    DegridParams P;
    P.traj = p->traj.as<float4>();
    P.n = (long long)p->n;
    P.dim = p->dim;
    P.G = (int)p->G;
    P.hw = p->hw;
    P.L = p->L;
    P.smax = p->lut_smax;
    P.kc = p->lut_kc;
    P.lut_e = p->lut_e.as<float4>();
    P.cells = p->dim == 3 ? (long long)p->G * p->G * p->G : (long long)p->G * p->G;
    P.checkerboard = (p->flags & FR_PLAN_CHECKERBOARD) ? 1 : 0;
    P.grid = nullptr;
    P.channels = 0;
    P.out = nullptr;
    return P;
}

// Most cells of a footprint along an axis: an open interval of length 2 hw
// holds at most ceil(2 hw); without the exact trim floor(2 hw) + 1, where the
// rounding of c - hw and c + hw (below 2^-11 for grids up to 4096) can add one
// if 2 hw is just below an integer.
int footprint_reach(fr_plan p)
{
    return p->prefilter ? (int)std::ceil(2.0 * p->hw) : (int)std::floor(2.0 * p->hw + 1e-3) + 1;
}

template <int LP, int R>
int launch_degrid_tiles(const DegridParams &P, const TileDegrid &T, dim3 grid, size_t smem, cudaStream_t s)
{
    auto kern = degrid_tiles_kernel<LP, R>;
    FR_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<grid, kDegridThreads, smem, s>>>(P, T);
    FR_CHECK_LAUNCH("degrid_tiles_kernel");
    return FR_OK;
}

// The tiled degridding; -1 where a thread per sample is the better form.  The
// lines are where the two crossed over 1 to 30 coils, 1 k to 5 M samples, widths 3
// to 5 (times: thread per sample / tiled, us):
//  * 3D: from 4 coils (a sample's lanes share its geometry over two coils each: 1
//    coil 240 / 347), with under 8 from 4 M values (4 coils, 192 k samples 78 / 85,
//    2.6 M 2666 / 1460), else from 1 M (16 coils, 19 k samples 35 / 47, 64 k 133 /
//    78: too few CTAs below).  Staging a part is paid by its samples: from 100 per
//    work item (12 coils, 180^3: 67 a tile 589 / 636, 160 a tile 2021 / 880), from
//    40 when 4 coils of the grid are past the L2 cache, whose hits the other form
//    lives on (12 coils, 300^3: 32 a tile 2874 / 2335, 48 a tile 4362 / 2501).
//  * the other widths need more: 3 (fewer taps per staged cell) a grid that is not
//    cached, 6 coils and 150 a tile (12 coils, 144^3 278 / 378; 210^3 1787 /
//    1176), 5 a grid past the cache (16 coils, 144^3 1516 / 1601, 210^3 at 20
//    coils 11164 / 5792); a cached grid 6 coils in groups that fill three
//    quarters of their lanes (17 coils, width 5: 1628 / 1757).
//  * 2D (always cached): from 12 coils (8 coils 56 / 58, 16 coils 97 / 67), 100 k
//    samples (20 coils, 75 k 25 / 44) and 32 k cells (a 90^2 grid sits in L1: 54 /
//    60), width over 3 (53 / 57).
//  * never footprints over 5 cells (the lists), over 1024 table entries, or a
//    tile that leaves no part of at most kDegridBlock bytes.
constexpr size_t kDegridBlock = 96 * 1024;  // two CTAs per SM
bool tiled_degrid_pays(fr_plan p, int R, long long cells, int channels, int pairs, int LP)
{
    const long long n = (long long)p->n, values = n * channels;
    const long long each = n / std::max<long long>(p->nitems_occupied, 1);  // samples per work item
    const bool full = 4 * pairs >= 3 * LP;
    if (R > 5 || p->L > 1024 || values < 1ll << 20) return false;
    if (p->dim == 2) return channels >= 12 && n >= 100000 && cells >= 1 << 15 && R >= 4 && full && each >= 100;
    const long long four = cells * 32;  // bytes of 4 coils of the grid
    const bool cached = four < 100ll << 20, past = four > 190ll << 20;
    if (channels < 4 || (channels < 8 && values < 1ll << 22)) return false;
    if (R <= 3) return !cached && channels >= 6 && each >= 150;
    if (R == 5) return past && each >= 100;
    return past ? each >= 40 : each >= 100 && (!cached || (channels >= 6 && full));
}

int degrid_tiles(fr_plan p, const DegridParams &P, cudaStream_t s)
{
    if (p->nitems_occupied == 0) return -1;
    const int R = footprint_reach(p);
    TileDegrid T;
    T.recs = p->pairs.as<unsigned long long>();
    T.items = p->items.as<WorkItem>();
    T.trim = p->prefilter;
    T.lutw = p->lut_d.as<float>();
    // groups of at most 16 coils, even, of near equal size
    const int groups = (P.channels + 15) / 16;
    T.coils = ((P.channels + groups - 1) / groups + 1) & ~1;
    const int pairs = T.coils / 2, LP = pairs <= 2 ? 2 : pairs <= 4 ? 4 : 8;
    if (!tiled_degrid_pays(p, R, P.cells, P.channels, pairs, LP)) return -1;
    T.stride = 4 * (pairs | 1);
    const int RR = R <= 4 ? 4 : 5;
    long long parts = 1;
    for (int d = 0; d < 3; ++d) {
        T.tile[d] = T.box[d] = p->tile[d];
        T.ntile[d] = p->ntile[d];
        T.nbox[d] = 1;
    }
    auto bytes = [&] {
        size_t b = (size_t)T.stride * 4;
        for (int d = 0; d < p->dim; ++d) b *= (size_t)(T.box[d] + RR - 1);
        return b;
    };
    while (bytes() > kDegridBlock) {  // halve the longest axis, the outermost first
        int d = p->dim - 1;
        for (int k = p->dim - 2; k >= 0; --k)
            if (T.box[k] > T.box[d]) d = k;
        if (T.box[d] <= 2) return -1;
        T.box[d] = (T.box[d] + 1) / 2;
        T.nbox[d] = (T.tile[d] + T.box[d] - 1) / T.box[d];
    }
    for (int d = 0; d < 3; ++d) parts *= T.nbox[d];
    if (parts > 65535 || groups > 65535) return -1;
    const size_t smem = bytes() + (size_t)(kDegridThreads / LP) * degrid_list(RR) * 8 + (size_t)P.L * 8 + kDegridRound * 8;
    const dim3 grid((unsigned)p->nitems_occupied, (unsigned)parts, (unsigned)groups);
    degrid_outside_kernel<<<(int)std::min<long long>((P.n + 255) / 256, (long long)sm_count() * 8), 256, 0, s>>>(P);
    FR_CHECK_LAUNCH("degrid_outside_kernel");
    if (RR == 4) {
        switch (LP) {
        case 2: return launch_degrid_tiles<2, 4>(P, T, grid, smem, s);
        case 4: return launch_degrid_tiles<4, 4>(P, T, grid, smem, s);
        default: return launch_degrid_tiles<8, 4>(P, T, grid, smem, s);
        }
    }
    switch (LP) {
    case 2: return launch_degrid_tiles<2, 5>(P, T, grid, smem, s);
    case 4: return launch_degrid_tiles<4, 5>(P, T, grid, smem, s);
    default: return launch_degrid_tiles<8, 5>(P, T, grid, smem, s);
    }
}

}  // namespace

int dcf_analytic_run(const float *d_traj, size_t n, int dim, float power, float *d_out, cudaStream_t s)
{
    if (n == 0) return FR_OK;
    const int mode = power == 1.f ? 1 : (power == 2.f ? 2 : 0);
    const int blocks = (int)std::min<long long>(((long long)n + 255) / 256, (long long)sm_count() * 8);
    dcf_analytic_kernel<<<blocks, 256, 0, s>>>(reinterpret_cast<const float4 *>(d_traj), (long long)n, dim,
                                               (double)power, mode, d_out);
    FR_CHECK_LAUNCH("dcf_analytic_kernel");
    return FR_OK;
}

int degrid_run(fr_plan p, const float *d_grid, int channels, float *d_out, cudaStream_t s)
{
    if (!p->planned) return fail(FR_ERR_NOT_PLANNED, "fr_degrid called before fr_plan_set_trajectory");
    if (channels <= 0) return fail(FR_ERR_INVALID_ARGUMENT, "channels must be positive");
    if (p->n == 0) return FR_OK;
    DegridParams P = degrid_params(p);
    P.grid = reinterpret_cast<const float2 *>(d_grid);
    P.channels = channels;
    P.out = reinterpret_cast<float2 *>(d_out);
    const int tiled = degrid_tiles(p, P, s);
    if (tiled >= 0) return tiled;
    constexpr int CB = 4;
    const size_t smem = (size_t)P.L * 16;
    if (smem > 48 * 1024)
        FR_CUDA(cudaFuncSetAttribute(degrid_kernel<CB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int bx = (int)std::min<long long>((P.n + 255) / 256, (long long)sm_count() * 8);
    dim3 grid(bx, (channels + CB - 1) / CB);
    degrid_kernel<CB><<<grid, 256, smem, s>>>(P);
    FR_CHECK_LAUNCH("degrid_kernel");
    return FR_OK;
}

int grid_update_run(fr_plan p, float *d_kdata, const float *d_new, size_t begin, size_t count, const float *d_dcf,
                    int channels, float *d_grid, cudaStream_t s)
{
    if (!p->planned) return fail(FR_ERR_NOT_PLANNED, "fr_grid_update called before fr_plan_set_trajectory");
    if (channels <= 0) return fail(FR_ERR_INVALID_ARGUMENT, "channels must be positive");
    if (begin > p->n || count > p->n - begin) return fail(FR_ERR_SIZE_MISMATCH, "sample range exceeds the plan's samples");
    if (count == 0) return FR_OK;
    UpdateParams U;
    U.g = degrid_params(p);
    U.g.channels = channels;
    U.old_k = reinterpret_cast<float2 *>(d_kdata);
    U.new_k = reinterpret_cast<const float2 *>(d_new);
    U.dcf = d_dcf;
    U.grid = reinterpret_cast<float2 *>(d_grid);
    U.begin = (long long)begin;
    U.count = (long long)count;
    const size_t smem = (size_t)U.g.L * 16;
    if (smem > 48 * 1024)
        FR_CUDA(cudaFuncSetAttribute(grid_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int bx = (int)std::min<long long>(((long long)count + kUpdateWarps - 1) / kUpdateWarps, (long long)sm_count() * 32);
    grid_update_kernel<<<bx, kUpdateWarps * 32, smem, s>>>(U);
    FR_CHECK_LAUNCH("grid_update_kernel");
    return FR_OK;
}

int grid_real_run(fr_plan p, const float *d_w, float *d_grid, cudaStream_t s)
{
    if (!p->planned) return fail(FR_ERR_NOT_PLANNED, "plan has no trajectory");
    RealGridParams P;
    P.traj = p->traj.as<float4>();
    P.recs = p->pairs.as<unsigned long long>();
    P.items = p->items.as<WorkItem>();
    P.splits = p->splits.as<SplitTile>();
    P.w = d_w;
    P.lut_e = p->lut_e.as<float4>();
    P.grid = d_grid;
    P.dim = p->dim;
    P.G = (int)p->G;
    P.L = p->L;
    P.K = 1;
    for (int d = 0; d < 3; ++d) {
        P.tile[d] = p->tile[d];
        P.ntile[d] = p->ntile[d];
        P.K *= p->tile[d];
    }
    P.smax = p->lut_smax;
    P.kc = p->lut_kc;
    if (p->nslots > 0 && p->real_partials.reserve((size_t)p->nslots * P.K * 4)) return FR_ERR_CUDA;
    P.partials = p->real_partials.as<float>();
    if (p->nitems == 0) return FR_OK;
    P.trecs = p->trecs.as<unsigned long long>();
    P.taps = p->taps.as<unsigned>();
    P.lutw = p->lut_d.as<float>();
    P.tap_words = p->tap_words;
    const size_t smem = (size_t)P.L * 16 + (size_t)P.K * 4;
    if (smem > 227 * 1024) return fail(FR_ERR_UNSUPPORTED, "tile too large for the real-valued scatter");
    if (p->tap_words > 0) {  // plans without tap lists evaluate each record's box
        const size_t tsmem = (size_t)P.L * 4 + (size_t)P.K * 8;
        if (tsmem > 40 * 1024)
            FR_CUDA(cudaFuncSetAttribute(grid_real_taps_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tsmem));
        int per_sm = 0;
        FR_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, grid_real_taps_kernel, kRealTapWarps * 32, tsmem));
        const long long nb = std::min<long long>(p->nitems, (long long)std::max(per_sm, 1) * sm_count());
        grid_real_taps_kernel<<<(unsigned)nb, kRealTapWarps * 32, tsmem, s>>>(P, (int)p->nitems);
        FR_CHECK_LAUNCH("grid_real_taps_kernel");
    } else {
        if (smem > 48 * 1024)
            FR_CUDA(cudaFuncSetAttribute(grid_real_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        grid_real_kernel<<<(unsigned)p->nitems, kRealWarps * 32, smem, s>>>(P);
        FR_CHECK_LAUNCH("grid_real_kernel");
    }
    if (p->nsplits > 0) {
        reduce_real_splits_kernel<<<(unsigned)p->nsplits, 256, 0, s>>>(P);
        FR_CHECK_LAUNCH("reduce_real_splits_kernel");
    }
    return FR_OK;
}

int dcf_pipe_run(fr_plan p, int iterations, float *d_w, cudaStream_t s)
{
    if (!p->planned) return fail(FR_ERR_NOT_PLANNED, "fr_dcf_pipe called before fr_plan_set_trajectory");
    if (iterations < 0) return fail(FR_ERR_INVALID_ARGUMENT, "iterations must be >= 0");
    if (p->n == 0 || iterations == 0) return FR_OK;
    const size_t cells = p->dim == 3 ? (size_t)p->G * p->G * p->G : (size_t)p->G * p->G;
    if (p->real_grid.reserve(cells * 4)) return FR_ERR_CUDA;
    DegridParams P = degrid_params(p);
    const size_t smem = (size_t)P.L * 8;
    const int trim = p->prefilter, reach = footprint_reach(p);
    auto kern = reach <= 4 ? pipe_update_kernel<4> : reach <= 5 ? pipe_update_kernel<5>
                : reach <= 9 ? pipe_update_kernel<9> : pipe_update_kernel<14>;  // widths up to 13
    if (smem > 48 * 1024)
        FR_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    FR_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 256, smem));
    const int bx = (int)std::min<long long>((P.n + 255) / 256, (long long)sm_count() * std::max(per_sm, 1));  // one wave
    for (int it = 0; it < iterations; ++it) {
        int st = grid_real_run(p, d_w, p->real_grid.as<float>(), s);
        if (st) return st;
        kern<<<bx, 256, smem, s>>>(P, trim, p->lut_d.as<float>(), p->real_grid.as<float>(), d_w);
        FR_CHECK_LAUNCH("pipe_update_kernel");
    }
    return FR_OK;
}

}  // namespace fr
