// fr_image.cu -- image-domain kernels: fftShift, crop, fused crop + SoS.
//
// Replaces the host-side ImageFilter::fftShift / crop / SOS that the
// reference runs even in GPU mode (ImageFilter.cpp:40-53,120-209,231-280;
// cuImageFilter.cpp:40-52).  The SoS kernel reads each coil image once over
// the crop window and reproduces the reference's float arithmetic exactly:
// per channel, in channel order, acc += (re*re - im*(-im)), then sqrt.
#include <cuda_runtime.h>

#include "fr_internal.h"

namespace fr {
namespace {

struct Size3 {
    unsigned x, y, z;
};

// ImageFilter::fftShift (ImageFilter.cpp:231-280) as index arithmetic.  Its
// loops swap plane z with plane z + nz/2 (rows y and y + ny/2 in 2D, handled
// here as planes of one row), position (x, y) of the lower plane with
// (partner(x), partner(y)) of the upper one, x fastest.  Along an even axis
// the partners are a bijection and the swaps disjoint; along an odd axis 0
// and n-1 share the partner n/2, so up to four swaps of one plane pair touch
// the same elements: they form a group, done in the loops' order, and groups
// are independent of each other.
__device__ __forceinline__ unsigned shift_partner(unsigned i, unsigned n)
{
    const unsigned h = n / 2;
    return i < h ? i + h : i - h;
}
// 2 when the swap of index i opens a group (0 and n-1) along this axis
__device__ __forceinline__ int shift_group(unsigned i, unsigned n) { return (n & 1) && n > 1 && i == 0 ? 2 : 1; }

// The element that the loops leave at (x, y, z): its group's swaps traced
// backwards.  s is {x, y, z} sizes ({x, 1, y} in 2D).
__device__ __forceinline__ size_t shift_source(const Size3 &s, unsigned x, unsigned y, unsigned z)
{
    const unsigned hz = s.z / 2;
    bool lower = z < hz;
    const unsigned za = lower ? z : z - hz;
    // untouched: the last plane of an odd count, and the upper planes' last
    // column and row along odd axes
    if (z < 2 * hz && (lower || !(((s.y & 1) && s.y > 1 && y == s.y - 1) || ((s.x & 1) && s.x > 1 && x == s.x - 1)))) {
        unsigned gx = lower ? x : shift_partner(x, s.x), gy = lower ? y : shift_partner(y, s.y);
        if ((s.x & 1) && gx == s.x - 1) gx = 0;
        if ((s.y & 1) && gy == s.y - 1) gy = 0;
        for (int ky = shift_group(gy, s.y) - 1; ky >= 0; --ky)
            for (int kx = shift_group(gx, s.x) - 1; kx >= 0; --kx) {
                const unsigned xx = kx ? s.x - 1 : gx, yy = ky ? s.y - 1 : gy;
                const unsigned bx = shift_partner(xx, s.x), by = shift_partner(yy, s.y);
                const bool at = lower ? x == xx && y == yy : x == bx && y == by;
                if (at) {
                    x = lower ? bx : xx;
                    y = lower ? by : yy;
                    lower = !lower;
                }
            }
        z = lower ? za : za + hz;
    }
    return ((size_t)z * s.y + y) * s.x + x;
}

// sos_mode bit 1: continue the sum already in `out` (coils in slabs);
// bit 2: apply sqrt (/ deapod), else store the plain sum.
// SHIFT: read the images through the fftShift (`sh`: its axes), so that a
// recon of an odd grid needs no pass that moves the images.  Bound by launch and
// read latency: 115^3 grid, 3 coils 7 us with or without SHIFT; the serial shift
// pass in front of it took 5.3 ms (recon 5.74 -> 0.48 ms; 151^2, 5 coils: 230 -> 167 us).
template <bool SHIFT>
__global__ void sos_kernel(const float2 *__restrict__ imgs, int channels, Size3 in, Size3 rec,
                           Size3 off, Size3 sh, const float *__restrict__ deapod, float *__restrict__ out, int sos_mode)
{
    const size_t nout = (size_t)rec.x * rec.y * rec.z;
    const size_t cells = (size_t)in.x * in.y * in.z;
    for (size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x; o < nout;
         o += (size_t)gridDim.x * blockDim.x) {
        unsigned x = (unsigned)(o % rec.x);
        size_t r = o / rec.x;
        unsigned y = (unsigned)(r % rec.y);
        unsigned z = (unsigned)(r / rec.y);
        size_t in_idx;
        if (SHIFT) {
            const bool flat = sh.y != in.y || sh.z != in.z;  // 2D: the rows are the planes
            in_idx = flat ? shift_source(sh, x + off.x, 0, y + off.y) : shift_source(sh, x + off.x, y + off.y, z + off.z);
        } else {
            in_idx = ((size_t)(z + off.z) * in.y + (y + off.y)) * in.x + (x + off.x);
        }
        float acc = (sos_mode & 1) ? out[o] : 0.f;
        for (int c = 0; c < channels; ++c) {
            float2 v = imgs[(size_t)c * cells + in_idx];
            // std::complex<float>: x * conj(x) real part = a*a - b*(-b)
            float re = __fsub_rn(__fmul_rn(v.x, v.x), __fmul_rn(v.y, -v.y));
            acc = __fadd_rn(acc, re);
        }
        float m = acc;
        if (sos_mode & 2) {
            m = __fsqrt_rn(m);
            if (deapod) m = __fdiv_rn(m, deapod[o]);
        }
        out[o] = m;
    }
}

__global__ void crop_kernel(const float2 *__restrict__ imgs, int channels, Size3 in, Size3 rec, Size3 off,
                            float2 *__restrict__ out)
{
    const size_t nout = (size_t)rec.x * rec.y * rec.z;
    const size_t cells = (size_t)in.x * in.y * in.z;
    const size_t total = nout * (size_t)channels;
    for (size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x; o < total;
         o += (size_t)gridDim.x * blockDim.x) {
        size_t c = o / nout;
        size_t v = o - c * nout;
        unsigned x = (unsigned)(v % rec.x);
        size_t r = v / rec.x;
        unsigned y = (unsigned)(r % rec.y);
        unsigned z = (unsigned)(r / rec.y);
        out[o] = imgs[c * cells + ((size_t)(z + off.z) * in.y + (y + off.y)) * in.x + (x + off.x)];
    }
}

// The shift in place: a thread per swap group (see shift_partner), which
// replays the group's one to four swaps in the loops' order.  s is {x, y, z}
// sizes ({x, 1, y} in 2D); groups per axis: the length, less one when odd.
// I: 32-bit group numbers where they do, as in shift_even_kernel.
template <typename I>
__global__ void shift_kernel(float2 *__restrict__ imgs, int channels, Size3 s)
{
    const size_t cells = (size_t)s.x * s.y * s.z;
    const unsigned hz = s.z / 2;
    const unsigned nx = (s.x & 1) && s.x > 1 ? s.x - 1 : s.x, ny = (s.y & 1) && s.y > 1 ? s.y - 1 : s.y;
    const I groups = (I)nx * ny * hz, total = groups * (I)channels;
    for (I o = blockIdx.x * (I)blockDim.x + threadIdx.x; o < total; o += (I)gridDim.x * blockDim.x) {
        const I c = o / groups;
        const I i = o - c * groups;
        const I r = i / nx;
        const unsigned x = (unsigned)(i - r * nx);
        const unsigned z = (unsigned)(ny == 1 ? r : r / ny), y = (unsigned)(r - (I)z * ny);
        float2 *lo = imgs + (size_t)c * cells + (size_t)z * s.y * s.x;
        float2 *hi = lo + (size_t)hz * s.y * s.x;
        for (int ky = 0; ky < shift_group(y, s.y); ++ky)
            for (int kx = 0; kx < shift_group(x, s.x); ++kx) {
                const unsigned xx = kx ? s.x - 1 : x, yy = ky ? s.y - 1 : y;
                const size_t a = (size_t)yy * s.x + xx;
                const size_t b = (size_t)shift_partner(yy, s.y) * s.x + shift_partner(xx, s.x);
                const float2 t = lo[a];
                lo[a] = hi[b];
                hi[b] = t;
            }
    }
}

// The same where x and y are even (or y is 1): disjoint swaps, PER of them in flight
// per thread.  T: cells, or pairs of them (float4, s.x in pairs) where the halves of a
// row start on 16 bytes.  Bound: HBM, or the L2 cache for images that fit; 64-bit
// divisions beside the copies.  The kernel above with 64-bit numbers / pairs, us: 2D
// 1024^2, 4 coils 16.7 / 8.5, 2000^2, 6 coils 78 / 60; 3D 256^3, 6 coils 295 / 237.  Cells,
// 1 / 4 swaps in flight: 2D 1500^2, 8 coils 75 / 56, 3D 192^3, 8 coils 144 / 176.
template <typename T, int PER, typename I>
__global__ void shift_even_kernel(T *__restrict__ imgs, int channels, Size3 s)
{
    const size_t cells = (size_t)s.x * s.y * s.z;
    const unsigned hz = s.z / 2;
    const I half = (I)s.x * s.y * hz, total = half * (I)channels;
    for (I o0 = blockIdx.x * (I)(blockDim.x * PER) + threadIdx.x; o0 < total; o0 += (I)gridDim.x * (blockDim.x * PER)) {
        T *a[PER], *b[PER], va[PER], vb[PER];
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const I o = min(o0 + k * blockDim.x, total - 1);
            const I c = o / half;
            const I i = o - c * half;
            const I r = i / s.x;
            const unsigned x = (unsigned)(i - r * s.x);
            const unsigned z = (unsigned)(s.y == 1 ? r : r / s.y), y = (unsigned)(r - (I)z * s.y);
            T *img = imgs + (size_t)c * cells;
            a[k] = img + ((size_t)z * s.y + y) * s.x + x;
            b[k] = img + ((size_t)(z + hz) * s.y + shift_partner(y, s.y)) * s.x + shift_partner(x, s.x);
        }
#pragma unroll
        for (int k = 0; k < PER; ++k)
            if (o0 + k * blockDim.x < total) {
                va[k] = *a[k];
                vb[k] = *b[k];
            }
#pragma unroll
        for (int k = 0; k < PER; ++k)
            if (o0 + k * blockDim.x < total) {
                *a[k] = vb[k];
                *b[k] = va[k];
            }
    }
}

int blocks_for(size_t n, int threads)
{
    size_t b = (n + threads - 1) / threads;
    if (b > 152 * 64) b = 152 * 64;
    return (int)(b ? b : 1);
}

Size3 size_of(int dim, const unsigned *s)
{
    return Size3{s[0], s[1], dim == 3 ? s[2] : 1u};
}

// The shift's axes: 2D rows are planes of one row.
Size3 shift_axes(int dim, const unsigned *s)
{
    return dim == 3 ? Size3{s[0], s[1], s[2]} : Size3{s[0], 1u, s[1]};
}

int check_crop(int dim, const unsigned *size, const unsigned *rec, Size3 &in, Size3 &r, Size3 &off)
{
    in = size_of(dim, size);
    r = Size3{rec[0], rec[1], dim == 3 ? rec[2] : 1u};
    if (r.x > in.x || r.y > in.y || r.z > in.z)
        return fail(FR_ERR_INVALID_ARGUMENT, "crop size larger than image");  // ImageFilter.cpp:128-131
    off = Size3{(in.x - r.x) / 2, (in.y - r.y) / 2, (in.z - r.z) / 2};
    return FR_OK;
}

}  // namespace

int sos_run(const float *d_imgs, int channels, int dim, const unsigned *size, const unsigned *recon,
            const float *d_deapod, float *d_out, cudaStream_t s, int sos_mode, bool shifted)
{
    Size3 in, r, off;
    int st = check_crop(dim, size, recon, in, r, off);
    if (st) return st;
    size_t nout = (size_t)r.x * r.y * r.z;
    auto kern = shifted ? sos_kernel<true> : sos_kernel<false>;
    kern<<<blocks_for(nout, 256), 256, 0, s>>>(reinterpret_cast<const float2 *>(d_imgs), channels, in, r, off,
                                               shift_axes(dim, size), d_deapod, d_out, sos_mode);
    FR_CHECK_LAUNCH("sos_kernel");
    return FR_OK;
}

int crop_run(const float *d_imgs, int channels, int dim, const unsigned *size, const unsigned *crop,
             float *d_out, cudaStream_t s)
{
    Size3 in, r, off;
    int st = check_crop(dim, size, crop, in, r, off);
    if (st) return st;
    size_t total = (size_t)r.x * r.y * r.z * channels;
    crop_kernel<<<blocks_for(total, 256), 256, 0, s>>>(reinterpret_cast<const float2 *>(d_imgs), channels, in, r,
                                                       off, reinterpret_cast<float2 *>(d_out));
    FR_CHECK_LAUNCH("crop_kernel");
    return FR_OK;
}

int shift_run(float *d_imgs, int channels, int dim, const unsigned *size, cudaStream_t s)
{
    const Size3 sz = shift_axes(dim, size);
    if (sz.z < 2) return FR_OK;  // no plane pair to swap
    const size_t most = (size_t)sz.x * sz.y * (sz.z / 2) * channels;
    const bool even = sz.x % 2 == 0 && (sz.y % 2 == 0 || sz.y == 1);
    const bool pairs = even && sz.x % 4 == 0 && (reinterpret_cast<uintptr_t>(d_imgs) & 15) == 0;
    const int per = even && !pairs && sz.y == 1 ? 4 : 1;
    const int blocks = blocks_for((pairs ? most / 2 : most) / per + 1, 256);
    const bool wide = most + (size_t)blocks * 256 * per > 0xFFFFFFFFull;  // the loop's numbers stay below 2^32
    float2 *cells = reinterpret_cast<float2 *>(d_imgs);
    if (pairs) {
        auto kern = wide ? shift_even_kernel<float4, 1, size_t> : shift_even_kernel<float4, 1, unsigned>;
        kern<<<blocks, 256, 0, s>>>(reinterpret_cast<float4 *>(d_imgs), channels, Size3{sz.x / 2, sz.y, sz.z});
    } else if (per == 4) {
        auto kern = wide ? shift_even_kernel<float2, 4, size_t> : shift_even_kernel<float2, 4, unsigned>;
        kern<<<blocks, 256, 0, s>>>(cells, channels, sz);
    } else if (even) {
        auto kern = wide ? shift_even_kernel<float2, 1, size_t> : shift_even_kernel<float2, 1, unsigned>;
        kern<<<blocks, 256, 0, s>>>(cells, channels, sz);
    } else {
        auto kern = wide ? shift_kernel<size_t> : shift_kernel<unsigned>;
        kern<<<blocks, 256, 0, s>>>(cells, channels, sz);
    }
    FR_CHECK_LAUNCH("shift_kernel");
    return FR_OK;
}

}  // namespace fr

// --------------------------------------------------------------------------
// Deapodization (absent in the reference): the image-domain apodization of
// the gridding kernel, obtained by gridding one unit sample at the FFT origin
// of the shifted image (cell G/2 on every axis) with the same LUT and tap
// rule, transforming it with the same backward FFT, and taking |.|
// normalised to the centre.
// --------------------------------------------------------------------------
namespace fr {
namespace {

__global__ void deapod_seed_kernel(float2 *__restrict__ grid, int dim, int G, float hw, const float *__restrict__ lut,
                                   int L, int reach, int checkerboard)
{
    const int w = 2 * reach + 1;
    const int total = dim == 3 ? w * w * w : w * w;
    const int c0 = G / 2;
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int ix = t % w, iy = (t / w) % w, iz = dim == 3 ? t / (w * w) : reach;
        int dx = ix - reach, dy = iy - reach, dz = iz - reach;
        int x = c0 + dx, y = c0 + dy, z = dim == 3 ? c0 + dz : 0;
        if (x < 0 || y < 0 || z < 0 || x >= G || y >= G || z >= G) continue;
        float fdy = (float)dy, fdz = (float)dz;
        float s = __fadd_rn(__fadd_rn(__fmul_rn(fdz, fdz), __fmul_rn(fdy, fdy)), __fmul_rn((float)dx, (float)dx));
        float dk = __fsqrt_rn(s);
        if (!(dk < hw)) continue;
        int ki = (int)roundf(__fmul_rn(__fdiv_rn(dk, hw), (float)(L - 1)));
        if (ki > L - 1) ki = L - 1;
        float v = lut[ki];
        if (checkerboard && ((x + y + z) & 1)) v = -v;
        grid[((size_t)z * G + y) * G + x] = make_float2(v, 0.f);
    }
}

__global__ void deapod_map_kernel(const float2 *__restrict__ img, Size3 in, Size3 rec, Size3 off,
                                  float *__restrict__ out)
{
    const size_t nout = (size_t)rec.x * rec.y * rec.z;
    const size_t ctr = ((size_t)(in.z / 2) * in.y + in.y / 2) * in.x + in.x / 2;
    const float2 c = img[ctr];
    const float norm = sqrtf(c.x * c.x + c.y * c.y);
    for (size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x; o < nout; o += (size_t)gridDim.x * blockDim.x) {
        unsigned x = (unsigned)(o % rec.x);
        size_t r = o / rec.x;
        unsigned y = (unsigned)(r % rec.y);
        unsigned z = (unsigned)(r / rec.y);
        float2 v = img[((size_t)(z + off.z) * in.y + (y + off.y)) * in.x + (x + off.x)];
        float m = sqrtf(v.x * v.x + v.y * v.y) / norm;
        out[o] = m > 1e-6f ? m : 1e-6f;
    }
}

}  // namespace

int deapod_seed_run(float *d_grid, int dim, int G, float hw, const float *d_lut, int L, int checkerboard,
                    cudaStream_t s)
{
    size_t cells = dim == 3 ? (size_t)G * G * G : (size_t)G * G;
    FR_CUDA(cudaMemsetAsync(d_grid, 0, cells * 8, s));
    int reach = (int)ceilf(hw) + 1;
    deapod_seed_kernel<<<1, 256, 0, s>>>(reinterpret_cast<float2 *>(d_grid), dim, G, hw, d_lut, L, reach,
                                         checkerboard);
    FR_CHECK_LAUNCH("deapod_seed_kernel");
    return FR_OK;
}

int deapod_map_run(const float *d_img, int dim, const unsigned *size, const unsigned *recon, float *d_out,
                   cudaStream_t s)
{
    Size3 in, r, off;
    int st = check_crop(dim, size, recon, in, r, off);
    if (st) return st;
    size_t nout = (size_t)r.x * r.y * r.z;
    deapod_map_kernel<<<blocks_for(nout, 256), 256, 0, s>>>(reinterpret_cast<const float2 *>(d_img), in, r, off,
                                                            d_out);
    FR_CHECK_LAUNCH("deapod_map_kernel");
    return FR_OK;
}

}  // namespace fr

// --------------------------------------------------------------------------
// PILS image operations (ImageFilter.cpp:55-118,170-209) and helpers.
// --------------------------------------------------------------------------
namespace fr {
namespace {

__global__ void real_to_complex_kernel(const float *__restrict__ in, size_t n, float2 *__restrict__ out)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = make_float2(in[i], 0.f);
}

// ImageFilter::lowFilter: r = squared distance to (size/2) in integers,
// idx = (int)((float)r / att * 100.0), coefficient table from the host.
__global__ void low_filter_kernel(float2 *__restrict__ imgs, int channels, Size3 s, float att,
                                  const float *__restrict__ coeff)
{
    const size_t cells = (size_t)s.x * s.y * s.z;
    const size_t total = cells * (size_t)channels;
    const long long x0 = s.x / 2, y0 = s.y / 2, z0 = s.z / 2;
    for (size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x; o < total; o += (size_t)gridDim.x * blockDim.x) {
        size_t v = o % cells;
        long long x = (long long)(v % s.x);
        size_t r0 = v / s.x;
        long long y = (long long)(r0 % s.y);
        long long z = (long long)(r0 / s.y);
        int r = (int)((x - x0) * (x - x0) + (y - y0) * (y - y0) + (z - z0) * (z - z0));
        int idx = (int)((double)__fdiv_rn((float)r, att) * 100.0);
        float2 a = imgs[o];
        if (idx >= 2000) {
            a = make_float2(0.f, 0.f);
        } else {
            float c = coeff[idx];
            a.x = __fmul_rn(a.x, c);
            a.y = __fmul_rn(a.y, c);
        }
        imgs[o] = a;
    }
}

// ImageFilter::normalize: mag = sum over channels of std::norm, each value
// divided by sqrtf(mag).
__global__ void normalize_channels_kernel(float2 *__restrict__ imgs, int channels, size_t cells)
{
    for (size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v < cells; v += (size_t)gridDim.x * blockDim.x) {
        float mag = 0.f;
        for (int c = 0; c < channels; ++c) {
            float2 a = imgs[(size_t)c * cells + v];
            mag = __fadd_rn(mag, __fadd_rn(__fmul_rn(a.x, a.x), __fmul_rn(a.y, a.y)));
        }
        float d = __fsqrt_rn(mag);
        for (int c = 0; c < channels; ++c) {
            float2 a = imgs[(size_t)c * cells + v];
            imgs[(size_t)c * cells + v] = make_float2(__fdiv_rn(a.x, d), __fdiv_rn(a.y, d));
        }
    }
}

// ImageFilter::SOS(map, reconSize): out += data * conj(map) per channel.
__global__ void sos_map_kernel(const float2 *__restrict__ imgs, const float2 *__restrict__ maps, int channels,
                               Size3 in, Size3 rec, Size3 off, float2 *__restrict__ out)
{
    const size_t nout = (size_t)rec.x * rec.y * rec.z;
    const size_t cells = (size_t)in.x * in.y * in.z;
    for (size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x; o < nout; o += (size_t)gridDim.x * blockDim.x) {
        unsigned x = (unsigned)(o % rec.x);
        size_t r = o / rec.x;
        unsigned y = (unsigned)(r % rec.y);
        unsigned z = (unsigned)(r / rec.y);
        size_t in_idx = ((size_t)(z + off.z) * in.y + (y + off.y)) * in.x + (x + off.x);
        float2 acc = make_float2(0.f, 0.f);
        for (int c = 0; c < channels; ++c) {
            float2 a = imgs[(size_t)c * cells + in_idx];
            float2 m = maps[(size_t)c * cells + in_idx];
            float nd = -m.y;  // conj
            float re = __fsub_rn(__fmul_rn(a.x, m.x), __fmul_rn(a.y, nd));
            float im = __fadd_rn(__fmul_rn(a.x, nd), __fmul_rn(a.y, m.x));
            acc.x = __fadd_rn(acc.x, re);
            acc.y = __fadd_rn(acc.y, im);
        }
        out[o] = acc;
    }
}

}  // namespace

int real_to_complex_run(const float *d_in, size_t n, float *d_out, cudaStream_t s)
{
    if (n == 0) return FR_OK;
    real_to_complex_kernel<<<blocks_for(n, 256), 256, 0, s>>>(d_in, n, reinterpret_cast<float2 *>(d_out));
    FR_CHECK_LAUNCH("real_to_complex_kernel");
    return FR_OK;
}

int low_filter_run(float *d_imgs, int channels, int dim, const unsigned *size, float att, const float *d_coeff,
                   cudaStream_t s)
{
    Size3 sz = size_of(dim, size);
    size_t total = (size_t)sz.x * sz.y * sz.z * channels;
    low_filter_kernel<<<blocks_for(total, 256), 256, 0, s>>>(reinterpret_cast<float2 *>(d_imgs), channels, sz, att,
                                                            d_coeff);
    FR_CHECK_LAUNCH("low_filter_kernel");
    return FR_OK;
}

int normalize_channels_run(float *d_imgs, int channels, int dim, const unsigned *size, cudaStream_t s)
{
    Size3 sz = size_of(dim, size);
    size_t cells = (size_t)sz.x * sz.y * sz.z;
    normalize_channels_kernel<<<blocks_for(cells, 256), 256, 0, s>>>(reinterpret_cast<float2 *>(d_imgs), channels,
                                                                    cells);
    FR_CHECK_LAUNCH("normalize_channels_kernel");
    return FR_OK;
}

int sos_map_run(const float *d_imgs, const float *d_maps, int channels, int dim, const unsigned *size,
                const unsigned *recon, float *d_out, cudaStream_t s)
{
    Size3 in, r, off;
    int st = check_crop(dim, size, recon, in, r, off);
    if (st) return st;
    size_t nout = (size_t)r.x * r.y * r.z;
    sos_map_kernel<<<blocks_for(nout, 256), 256, 0, s>>>(reinterpret_cast<const float2 *>(d_imgs),
                                                        reinterpret_cast<const float2 *>(d_maps), channels, in, r,
                                                        off, reinterpret_cast<float2 *>(d_out));
    FR_CHECK_LAUNCH("sos_map_kernel");
    return FR_OK;
}

}  // namespace fr
