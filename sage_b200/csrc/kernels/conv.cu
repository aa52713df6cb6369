// im2col / col2im / direct pooling for NHWC images.
//
// Reference: Im2col::compute (src/ops/conv.rs:289-374) gives each (y, x, c) of the column grid to a
// work-item that loops over the batch and the taps; Col2im::compute (:404-498) is the inverse
// gather-sum.  Here im2col gives a warp to each output pixel (see im2col_kernel) and can write the
// tf32 hi / lo planes of the column matrix for the tensor-core GEMM in the same pass; convolutions
// whose channel count is a multiple of 32 do not come here at all (the GEMM loads image tiles with
// im2col-mode TMA).  pool2d evaluates max/avg pooling
// (conv.rs:143-165: im2col, then a reduction over [KH,KW]) straight from the image without
// materialising the KH*KW-times larger column tensor.  Padded taps count as zeros, and with
// ref_compat the max starts from 0 like the reference's reduce accumulator.
#include <cuda.h>
#include <cuda_runtime.h>

#include "kernels.h"
#include "gemm_tc_device.inc"  // split_tf32_value
#include "gemm_h2_device.inc"  // h2_split2
#include "launch.h"

namespace sage {
const char *map_prelude_text();  // codegen/map_emit.cc
namespace k {

struct ConvP {
    long long n, img_h, img_w, chan, col_h, col_w;
    Window w;
};

// One warp per output pixel: the K = KH*KW*C values of a column row are contiguous in the output and
// C-contiguous runs in the image, so with C % 4 == 0 the lanes move 16-byte chunks and both sides
// coalesce; index arithmetic is 32-bit per chunk and once per pixel.  Outputs: the fp32 column
// tensor (row pitch K) and / or the tf32 hi / lo planes of it (row pitch `pitch` >= K, a multiple of
// 4; pad columns are written as zeros) for the tensor-core GEMM that consumes it.
struct ColOut {
    float *col;       // may be null
    float *hi;        // may be null; lo = hi + plane
    long long plane;
    int pitch;
};

__device__ __forceinline__ void split_pair(float x, float *hi, float *lo) { sage_tc::split_tf32_value(x, hi, lo); }
#define SAGE_COLS_SPLIT split_pair
#define SAGE_COLS_PRE(x0) (x0)
#define SAGE_COLS_POST(x0, x1, x2, x3) (x0)
#include "conv_cols_device.inc"
#include "conv_cols_device_src.h"  // generated by the Makefile: the text of conv_cols_device.inc as kConvColsDeviceSrc

// `share` warps to a pixel where there are few of them (128 pixels of 9 x 512 values, one warp each: 16 blocks, 8 us).
__global__ void __launch_bounds__(256) im2col_kernel(const float *__restrict__ img, ColOut o, ConvP p, long long pixels, int share) {
    grid_dependency_sync();
    const long long warp = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), pix = warp / share;
    const int lane = (threadIdx.x & 31) + 32 * (int)(warp - pix * share), step = 32 * share;
    if (pix >= pixels) return;
    const unsigned per_img = (unsigned)(p.col_h * p.col_w);
    const long long n = pix / per_img;
    const unsigned r = (unsigned)(pix - n * per_img);
    const int oy = (int)(r / (unsigned)p.col_w), ox = (int)(r % (unsigned)p.col_w);
    const int iy0 = oy * p.w.stride_h - p.w.pad_h, ix0 = ox * p.w.stride_w - p.w.pad_w;
    const int C = (int)p.chan, K = p.w.ker_h * p.w.ker_w * C;
    const float *im = img + n * p.img_h * p.img_w * C;
    if ((C & 3) == 0) {
        im2col_quads_of_pixel(im, o.col, o.hi, o.plane, o.pitch, p, pix, iy0, ix0, lane, step);
    } else {
        const int width = o.hi ? o.pitch : K;
        for (int kk = lane; kk < width; kk += step) {
            float v = 0.f;
            if (kk < K) {
                const int tap = kk / C, c = kk - tap * C;
                const int ky = tap / p.w.ker_w, kx = tap - ky * p.w.ker_w;
                const int iy = iy0 + ky * p.w.dil_h, ix = ix0 + kx * p.w.dil_w;
                if (ix >= 0 && ix < p.img_w && iy >= 0 && iy < p.img_h) v = __ldg(im + ((long long)iy * p.img_w + ix) * C + c);
                if (o.col) o.col[pix * K + kk] = v;
            }
            if (o.hi) {
                float h, l;
                split_pair(v, &h, &l);
                o.hi[pix * o.pitch + kk] = h;
                o.hi[pix * o.pitch + kk + o.plane] = l;
            }
        }
    }
}

// Planes of the column matrix when C is not a multiple of 4 (the first convolution of a network: C = 1 or 3,
// K = 49 or 147).  A thread owns 4 consecutive entries of a row (one 16-byte store into each plane), so a
// warp writes 512 contiguous bytes per plane; where an entry comes from (tap, channel) is looked up in a
// table in shared memory, built once per block, instead of being divided out per element.
constexpr int kTapTable = 1024;
__global__ void __launch_bounds__(256) im2col_quads_kernel(const float *__restrict__ img, ColOut o, ConvP p, long long quads) {
    grid_dependency_sync();
    __shared__ int tab_off[kTapTable];   // element offset of entry kk from the pixel's first tap, -1 beyond K
    __shared__ int tab_yx[kTapTable];    // (ky * dil_h) << 16 | (kx * dil_w)
    const int C = (int)p.chan, K = p.w.ker_h * p.w.ker_w * C;
    for (int kk = threadIdx.x; kk < o.pitch; kk += 256) {
        if (kk < K) {
            const int tap = kk / C, c = kk - tap * C;
            const int ky = tap / p.w.ker_w, kx = tap - ky * p.w.ker_w;
            tab_off[kk] = (ky * p.w.dil_h * (int)p.img_w + kx * p.w.dil_w) * C + c;
            tab_yx[kk] = ((ky * p.w.dil_h) << 16) | (kx * p.w.dil_w);
        } else {
            tab_off[kk] = -1;
            tab_yx[kk] = 0;
        }
    }
    __syncthreads();
    const int per_row = o.pitch >> 2;
    const unsigned per_img = (unsigned)(p.col_h * p.col_w);
    for (long long q = (long long)blockIdx.x * 256 + threadIdx.x; q < quads; q += (long long)gridDim.x * 256) {
        const long long pix = q / per_row;
        const int k0 = (int)(q - pix * per_row) << 2;
        const long long n = pix / per_img;
        const unsigned r = (unsigned)(pix - n * per_img);
        const int oy = (int)(r / (unsigned)p.col_w), ox = (int)(r % (unsigned)p.col_w);
        const int iy0 = oy * p.w.stride_h - p.w.pad_h, ix0 = ox * p.w.stride_w - p.w.pad_w;
        const float *base = img + (n * p.img_h * p.img_w + (long long)iy0 * p.img_w + ix0) * C;
        float v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int off = tab_off[k0 + i], yx = tab_yx[k0 + i];
            const int iy = iy0 + (yx >> 16), ix = ix0 + (yx & 0xffff);
            v[i] = (off >= 0 && ix >= 0 && ix < p.img_w && iy >= 0 && iy < p.img_h) ? __ldg(base + off) : 0.f;
        }
        float4 h, l;
        split_pair(v[0], &h.x, &l.x);
        split_pair(v[1], &h.y, &l.y);
        split_pair(v[2], &h.z, &l.z);
        split_pair(v[3], &h.w, &l.w);
        float *d = o.hi + pix * o.pitch + k0;
        *reinterpret_cast<float4 *>(d) = h;
        *reinterpret_cast<float4 *>(d + o.plane) = l;
        if (o.col) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (k0 + i < K) o.col[pix * K + k0 + i] = v[i];
        }
    }
}

// Follows the reference's tap test literally, including dilation_h applied to the x tap and
// dilation_w to the y tap (conv.rs:462-464); identical whenever both dilations are equal.
__global__ void __launch_bounds__(256) col2im_kernel(const float *__restrict__ col, float *__restrict__ img, ConvP p,
                                                     long long total) {
    grid_dependency_sync();
    for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < total;
         g += (long long)gridDim.x * blockDim.x) {
        long long r = g;
        const long long c = r % p.chan; r /= p.chan;
        const long long img_x = r % p.img_w; r /= p.img_w;
        const long long img_y = r % p.img_h; r /= p.img_h;
        const long long n = r;
        const long long xp = img_x + p.w.pad_w, yp = img_y + p.w.pad_h;
        const long long ker_ew = (p.w.ker_w - 1) * p.w.dil_w + 1, ker_eh = (p.w.ker_h - 1) * p.w.dil_h + 1;
        const long long xs = xp < ker_ew ? 0 : (xp - ker_ew) / p.w.stride_w + 1;
        const long long ys = yp < ker_eh ? 0 : (yp - ker_eh) / p.w.stride_h + 1;
        const long long xe = min(xp / p.w.stride_w + 1, p.col_w);
        const long long ye = min(yp / p.w.stride_h + 1, p.col_h);
        const long long col_b = n * p.col_h * p.col_w * p.w.ker_h * p.w.ker_w * p.chan;
        float val = 0.f;
        for (long long cx = xs; cx < xe; ++cx)
            for (long long cy = ys; cy < ye; ++cy) {
                long long kx = xp - cx * p.w.stride_w, ky = yp - cy * p.w.stride_h;
                if (kx % p.w.dil_h == 0 && ky % p.w.dil_w == 0) {
                    kx /= p.w.dil_h;
                    ky /= p.w.dil_w;
                    val += col[col_b + (((cy * p.col_w + cx) * p.w.ker_h + ky) * p.w.ker_w + kx) * p.chan + c];
                }
            }
        img[g] = val;
    }
}

// The same gather with 32-bit index arithmetic and four channels per thread (C % 4 == 0).
__global__ void __launch_bounds__(256) col2im_quads_kernel(const float *__restrict__ col, float *__restrict__ img, ConvP p, long long total) {
    grid_dependency_sync();
    col2im_quads(col, img, nullptr, 0, p, total, nullptr, nullptr, nullptr);
}

// One thread per output pixel and group of 4 channels when C % 4 == 0 (16-byte loads, one 64-bit division per thread), else
// one thread per element.  Nine taps are asked for at a time, then taken in the window's order: tap after tap a thread waited
// for the cache each time (3 x 3 over 256 x 112 x 112 x 64: 358 us and a split pass of 62 -> 264 with pieces).  Large windows
// with few results are pool2d_window_kernel's.  With pieces asked for, 16 threads hold the 64 channels of a group: no split pass reads the result again.
template <int VEC, class I, bool MARK>
__global__ void __launch_bounds__(256) pool2d_kernel(const float *__restrict__ img, float *__restrict__ out, ConvP p,
                                                     long long total, int is_max, int ref_compat, PlaneOut forms) {
    grid_dependency_sync();
    constexpr int U = 9;
    const unsigned cn = (unsigned)(p.chan / VEC);
    const int taps = p.w.ker_w * p.w.ker_h;
    for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < total;
         g += (long long)gridDim.x * blockDim.x) {
        const I pix = (I)g / (I)cn;
        const int c = (int)((I)g - pix * (I)cn) * VEC;
        const unsigned per_img = (unsigned)(p.col_h * p.col_w);
        const I n = pix / (I)per_img;
        const unsigned r = (unsigned)(pix - n * (I)per_img);
        const int oy = (int)(r / (unsigned)p.col_w), ox = (int)(r % (unsigned)p.col_w);
        const int y0 = oy * p.w.stride_h - p.w.pad_h, x0 = ox * p.w.stride_w - p.w.pad_w;
        const float *src = img + (long long)n * p.img_h * p.img_w * p.chan + c;
        const I img_w = (I)p.img_w, chan = (I)p.chan;
        const float init = is_max ? (ref_compat ? 0.f : -INFINITY) : 0.f;
        float acc[VEC];
#pragma unroll
        for (int j = 0; j < VEC; ++j) acc[j] = init;
        // reduce over axes [3,4] = [KH,KW]: the first listed axis (KH) is the inner loop
        int kx = 0, ky = 0;
        for (int t = 0; t < taps; t += U) {
            float v[U][VEC];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int iy = y0 + ky * p.w.dil_h, ix = x0 + kx * p.w.dil_w;
#pragma unroll
                for (int j = 0; j < VEC; ++j) v[u][j] = 0.f;
                if (t + u < taps && ix >= 0 && ix < (int)p.img_w && iy >= 0 && iy < (int)p.img_h) {
                    const float *at = src + ((I)iy * img_w + (I)ix) * chan;
                    if (VEC == 4) {
                        const float4 q = __ldg(reinterpret_cast<const float4 *>(at));
                        v[u][0] = q.x; v[u][1 % VEC] = q.y; v[u][2 % VEC] = q.z; v[u][3 % VEC] = q.w;
                    } else {
                        v[u][0] = __ldg(at);
                    }
                }
                if (++ky == p.w.ker_h) {
                    ky = 0;
                    ++kx;
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (t + u < taps)
#pragma unroll
                    for (int j = 0; j < VEC; ++j) acc[j] = is_max ? fmaxf(acc[j], v[u][j]) : acc[j] + v[u][j];
        }
        if (!is_max) {
#pragma unroll
            for (int j = 0; j < VEC; ++j) acc[j] = acc[j] / (float)(p.w.ker_w * p.w.ker_h);
        }
        const long long at = (long long)pix * p.chan + c;
        if (VEC == 1) {
            out[at] = acc[0];
            continue;
        }
        const float4 o = make_float4(acc[0], acc[1 % VEC], acc[2 % VEC], acc[3 % VEC]);
        if (out) *reinterpret_cast<float4 *>(out + at) = o;
        if (forms.h2) {
            using namespace sage_tc;
            unsigned b = max(max(h2_finite_bits(o.x), h2_finite_bits(o.y)), max(h2_finite_bits(o.z), h2_finite_bits(o.w)));
            const unsigned lanes = 0xffffu << (threadIdx.x & 16);
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) b = max(b, __shfl_xor_sync(lanes, b, off));
            float scale;
            const float f = h2_factor(b, &scale);
            uint2 h, l;
            h2_split2(o.x, o.y, f, &h.x, &l.x);
            h2_split2(o.z, o.w, f, &h.y, &l.y);
            *reinterpret_cast<uint2 *>(forms.h2 + at) = h;
            *reinterpret_cast<uint2 *>(forms.h2 + forms.h2_plane + at) = l;
            if ((threadIdx.x & 15) == 0) forms.h2_scale[at >> 6] = scale;
            if (MARK) {
                unsigned low1 = min(min(h2_low1(o.x), h2_low1(o.y)), min(h2_low1(o.z), h2_low1(o.w)));
#pragma unroll
                for (int off = 8; off > 0; off >>= 1) low1 = min(low1, __shfl_xor_sync(lanes, low1, off));
                if ((threadIdx.x & 15) == 0) forms.h2_marked[at >> 6] = h2_wide(low1, f) ? -scale : scale;
            }
        }
    }
}

// Large windows, few results (the mean over 7 x 7 x 512 at an image model's end): a block has 64 channels of a result, four to a thread,
// its 16 groups of threads share the window's taps, all of a thread's (of 64 at a time) in flight, and meet in shared memory in order.
// A thread to four channels took 7.5 us, six rounds of nine taps each.
__global__ void __launch_bounds__(256) pool2d_window_kernel(const float *__restrict__ img, float *__restrict__ out, ConvP p, int chan_blocks, int is_max, int ref_compat) {
    constexpr int U = 4;
    __shared__ float4 part[16][16];
    grid_dependency_sync();
    const int lane = threadIdx.x & 15, group = threadIdx.x >> 4, taps = p.w.ker_w * p.w.ker_h;
    const long long pix = blockIdx.x / chan_blocks;
    const int c = ((int)(blockIdx.x - pix * chan_blocks) * 16 + lane) * 4;
    const long long per_img = p.col_h * p.col_w, n = pix / per_img;
    const int r = (int)(pix - n * per_img), oy = r / (int)p.col_w, ox = r - oy * (int)p.col_w;
    const int y0 = oy * p.w.stride_h - p.w.pad_h, x0 = ox * p.w.stride_w - p.w.pad_w;
    const float *src = img + n * p.img_h * p.img_w * p.chan + c;
    const float init = is_max ? (ref_compat ? 0.f : -INFINITY) : 0.f;
    float4 acc = make_float4(init, init, init, init);
    auto take = [&](float4 &a, const float4 &v) {
        a.x = is_max ? fmaxf(a.x, v.x) : a.x + v.x;
        a.y = is_max ? fmaxf(a.y, v.y) : a.y + v.y;
        a.z = is_max ? fmaxf(a.z, v.z) : a.z + v.z;
        a.w = is_max ? fmaxf(a.w, v.w) : a.w + v.w;
    };
    if (c < (int)p.chan) {
        for (int t = group; t < taps; t += 16 * U) {
            float4 v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int tap = t + 16 * u, kx = tap / p.w.ker_h, ky = tap - kx * p.w.ker_h, iy = y0 + ky * p.w.dil_h, ix = x0 + kx * p.w.dil_w;
                const bool in = tap < taps && ix >= 0 && ix < (int)p.img_w && iy >= 0 && iy < (int)p.img_h;
                v[u] = in ? __ldg(reinterpret_cast<const float4 *>(src + ((long long)iy * p.img_w + ix) * p.chan)) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (t + 16 * u < taps) take(acc, v[u]);
        }
    }
    part[group][lane] = acc;
    __syncthreads();
    if (group || c >= (int)p.chan) return;
    for (int g = 1; g < 16; ++g) take(acc, part[g][lane]);
    if (!is_max) {
        const float taps_f = (float)taps;
        acc = make_float4(acc.x / taps_f, acc.y / taps_f, acc.z / taps_f, acc.w / taps_f);
    }
    *reinterpret_cast<float4 *>(out + pix * p.chan + c) = acc;
}

static unsigned grid_for(Context &ctx, long long n) {
    long long blocks = (n + 255) / 256;
    long long cap = (long long)ctx.sm_count * 32;
    return (unsigned)(blocks < cap ? blocks : cap);
}

sage_status im2col_planes(Context &ctx, const float *img, long long n, long long img_h, long long img_w, long long chan,
                          long long col_h, long long col_w, const Window &w, float *col, float *hi, long long plane, int pitch) {
    ConvP p{n, img_h, img_w, chan, col_h, col_w, w};
    const long long pixels = n * col_h * col_w;
    ctx.note_launch(ctx.verbose_names && hi ? (col ? "im2col+planes" : "im2col=planes") : "im2col");
    if (ctx.dry() || pixels == 0) return SAGE_OK;
    if (col_h * col_w > 0x7fffffffLL || img_h > 0x7fffffffLL || img_w > 0x7fffffffLL || (long long)w.ker_h * w.ker_w * chan > 0x7fffffffLL ||
        (pixels + 7) / 8 > 0x7fffffffLL)
        return ctx.fail(SAGE_ERR_UNSUPPORTED, "im2col: extents beyond 2^31");
    const bool vec = chan % 4 == 0;
    if (vec && ((col && reinterpret_cast<uintptr_t>(col) % 16) || reinterpret_cast<uintptr_t>(img) % 16 ||
                (hi && (reinterpret_cast<uintptr_t>(hi) % 16 || plane % 4 || pitch % 4))))
        return ctx.fail(SAGE_ERR_INVALID, "im2col: unaligned buffer");
    ColOut o{col, hi, plane, pitch};
    if (!vec && hi && pitch % 4 == 0 && pitch <= kTapTable && reinterpret_cast<uintptr_t>(hi) % 16 == 0 && plane % 4 == 0 &&
        img_w * (long long)w.ker_h * w.dil_h * chan < (1LL << 30) && w.ker_w * w.dil_w < 65536) {
        const long long quads = pixels * (pitch / 4);
        launch_dependent(ctx.pdl, ctx.stream(), im2col_quads_kernel, dim3(grid_for(ctx, quads)), dim3(256), 0, img, o, p, quads);
        return ctx.check_cuda(cudaGetLastError(), "im2col launch");
    }
    int share = 1;
    const long long length = w.ker_h * w.ker_w * chan / (vec ? 4 : 1);  // loads of a pixel
    while (share < 16 && pixels * share < 32LL * ctx.sm_count && length >= 128LL * share) share *= 2;
    launch_dependent(ctx.pdl, ctx.stream(), im2col_kernel, dim3((unsigned)((pixels * share + 7) / 8)), dim3(256), 0, img, o, p, pixels, share);
    return ctx.check_cuda(cudaGetLastError(), "im2col launch");
}

// ---- convolutions with at most 4 input channels (the first layer of an image model: C = 3 or 1).
// A channel run of 12 bytes is below TMA's 16-byte granularity, so the image is first re-laid as tf32 planes of
// [N, H + pad, W + pad, 4] — channels padded to 4, the spatial padding written as zeros.  In that layout the KW taps of one
// filter row are KW * 4 CONTIGUOUS floats, so one output pixel's operand row for tap row ky is a 32-float (128-byte)
// window starting 4 * stride_w floats after its left neighbour's: an "image" of 32-channel pixels that overlap.  The
// implicit-GEMM kernel then runs a (1 x KH) convolution over it; the column matrix is never written.
__global__ void __launch_bounds__(256) pack_small_c_kernel(const float *__restrict__ img, float4 *__restrict__ hi, float4 *__restrict__ lo, long long n,
                                                           int h, int w, int c, int hp, int wp, int pad_h, int pad_w) {
    grid_dependency_sync();
    const long long total = n * hp * (long long)wp;
    for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < total; g += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(g % wp) - pad_w;
        const long long r = g / wp;
        const int y = (int)(r % hp) - pad_h;
        const long long b = r / hp;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (x >= 0 && x < w && y >= 0 && y < h) {
            const float *s = img + ((b * h + y) * (long long)w + x) * c;
            for (int i = 0; i < c; ++i) v[i] = s[i];
        }
        if (!lo) {  // plain fp32: the GEMM splits each tile itself
            hi[g] = make_float4(v[0], v[1], v[2], v[3]);
            continue;
        }
        float4 a, d;
        sage_tc::split_tf32_value(v[0], &a.x, &d.x);
        sage_tc::split_tf32_value(v[1], &a.y, &d.y);
        sage_tc::split_tf32_value(v[2], &a.z, &d.z);
        sage_tc::split_tf32_value(v[3], &a.w, &d.w);
        hi[g] = a;
        lo[g] = d;
    }
}

// The filter [KH, KW, C, OC] as the matching B operand [KH * 32, OC]: row ky * 32 + kx * 4 + c; rows of padded
// channels and of the window's unused tail are zero, so whatever the overlapping operand rows hold there is ignored.
__global__ void __launch_bounds__(256) pack_small_c_filter_kernel(const float *__restrict__ f, float *__restrict__ hi, float *__restrict__ lo,
                                                                  int kh, int kw, int c, int oc) {
    grid_dependency_sync();
    const long long total = (long long)kh * 32 * oc;
    for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < total; g += (long long)gridDim.x * blockDim.x) {
        const int o = (int)(g % oc), row = (int)(g / oc), ky = row / 32, r = row % 32, kx = r / 4, cc = r % 4;
        const float v = (kx < kw && cc < c) ? f[(((long long)ky * kw + kx) * c + cc) * oc + o] : 0.f;
        sage_tc::split_tf32_value(v, &hi[g], &lo[g]);
    }
}

sage_status pack_small_c_image(Context &ctx, const float *img, long long n, long long h, long long w, long long c, long long hp, long long wp,
                               int pad_h, int pad_w, float *hi, long long plane) {
    ctx.note_launch("pack_small_c");
    if (ctx.dry()) return SAGE_OK;
    if (c < 1 || c > 4 || plane % 4 || reinterpret_cast<uintptr_t>(hi) % 16 || h > 0x7fffffffLL || w > 0x7fffffffLL || hp > 0x7fffffffLL || wp > 0x7fffffffLL)
        return ctx.fail(SAGE_ERR_INVALID, "pack_small_c: bad arguments");
    const long long total = n * hp * wp;
    launch_dependent(ctx.pdl, ctx.stream(), pack_small_c_kernel, dim3(grid_for(ctx, total)), dim3(256), 0, img, reinterpret_cast<float4 *>(hi), plane ? reinterpret_cast<float4 *>(hi + plane) : nullptr, n, (int)h, (int)w,
                                                                        (int)c, (int)hp, (int)wp, pad_h, pad_w);
    return ctx.check_cuda(cudaGetLastError(), "pack_small_c launch");
}

sage_status pack_small_c_filter(Context &ctx, const float *filt, int kh, int kw, int c, int oc, float *hi, long long plane) {
    ctx.note_launch("pack_small_c_filter");
    if (ctx.dry()) return SAGE_OK;
    if (kw * 4 > 32 || c > 4) return ctx.fail(SAGE_ERR_INVALID, "pack_small_c_filter: window too wide");
    launch_dependent(ctx.pdl, ctx.stream(), pack_small_c_filter_kernel, dim3(grid_for(ctx, (long long)kh * 32 * oc)), dim3(256), 0, filt, hi, hi + plane, kh, kw, c, oc);
    return ctx.check_cuda(cudaGetLastError(), "pack_small_c_filter launch");
}

// ---- the first convolution on half-precision pieces
constexpr int kAmaxParts = 32;  // blocks per image that look for its largest magnitude, and for its smallest above 0
// Magnitudes more than 2^29 apart: pieces under one scale would not hold 22 bits of each (`low1`: the smaller's bits less 1).
__device__ __forceinline__ bool first_wide(unsigned high, unsigned low1) { return high != 0u && (int)(high >> 23) - (int)((low1 + 1u) >> 23) > 29; }
__global__ void __launch_bounds__(256) first_amax_kernel(const float *__restrict__ img, long long len, int vec, uint2 *__restrict__ parts) {
    __shared__ uint2 warps[8];
    grid_dependency_sync();
    const float *s = img + blockIdx.y * len;
    unsigned m = 0, low1 = 0xffffffffu;  // (0 less 1 is the largest: zeros, infinities and nan do not count)
    if (vec) {
        const float4 *v = reinterpret_cast<const float4 *>(s);
#pragma unroll 4
        for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < len / 4; i += kAmaxParts * 256) {
            const float4 x = __ldg(v + i);
            const unsigned b0 = sage_tc::h2_finite_bits(x.x), b1 = sage_tc::h2_finite_bits(x.y), b2 = sage_tc::h2_finite_bits(x.z), b3 = sage_tc::h2_finite_bits(x.w);
            m = max(m, max(max(b0, b1), max(b2, b3)));
            low1 = min(low1, min(min(b0 - 1u, b1 - 1u), min(b2 - 1u, b3 - 1u)));
        }
    } else {
        for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < len; i += kAmaxParts * 256) {
            const unsigned b = sage_tc::h2_finite_bits(s[i]);
            m = max(m, b);
            low1 = min(low1, b - 1u);
        }
    }
    m = __reduce_max_sync(0xffffffffu, m);
    low1 = __reduce_min_sync(0xffffffffu, low1);
    if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = make_uint2(m, low1);
    __syncthreads();
    if (threadIdx.x < 32) {
        const uint2 p = threadIdx.x < 8 ? warps[threadIdx.x] : make_uint2(0u, 0xffffffffu);
        m = __reduce_max_sync(0xffffffffu, p.x);
        low1 = __reduce_min_sync(0xffffffffu, p.y);
        if (threadIdx.x == 0) parts[blockIdx.y * kAmaxParts + blockIdx.x] = make_uint2(m, low1);
    }
}
// A block takes four rows of the padded image, a thread two neighbouring pixels: 16 bytes of each piece.
__global__ void __launch_bounds__(128) pack_first_kernel(const float *__restrict__ img, unsigned short *__restrict__ hi, long long plane, long long rows, int h, int w, int c, int hp,
                                                         int wp, int pad_h, int pad_w, const uint2 *__restrict__ parts, float *__restrict__ scale) {
    grid_dependency_sync();
    for (int i = 0; i < 4; ++i) {
        const long long r = (long long)blockIdx.x * 4 + i;
        if (r >= rows) return;
        const long long b = r / hp;
        const int y = (int)(r - b * hp) - pad_h;
        float s;
        const uint2 part = __ldg(parts + b * kAmaxParts + (threadIdx.x & 31));
        const unsigned high = __reduce_max_sync(0xffffffffu, part.x), low1 = __reduce_min_sync(0xffffffffu, part.y);
        const float f = sage_tc::h2_factor(high, &s);
        if (y == -pad_h && threadIdx.x == 0) scale[b] = first_wide(high, low1) ? -s : s;
        for (int x2 = threadIdx.x; x2 < wp / 2; x2 += 128) {
            float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (y >= 0 && y < h) {
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int x = 2 * x2 + q - pad_w;
                    if (x < 0 || x >= w) continue;
                    const float *px = img + ((b * h + y) * (long long)w + x) * c;
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (k < c) v[q * 4 + k] = __ldg(px + k);
                }
            }
            uint4 a, l;
            sage_tc::h2_split2(v[0], v[1], f, &a.x, &l.x);
            sage_tc::h2_split2(v[2], v[3], f, &a.y, &l.y);
            sage_tc::h2_split2(v[4], v[5], f, &a.z, &l.z);
            sage_tc::h2_split2(v[6], v[7], f, &a.w, &l.w);
            unsigned short *at = hi + (r * wp + 2 * x2) * 4;
            *reinterpret_cast<uint4 *>(at) = a;
            *reinterpret_cast<uint4 *>(at + plane) = l;
        }
    }
}
// One block per output channel, those that fill up the last 64 included (zeros).
__global__ void __launch_bounds__(128) pack_first_filter_kernel(const float *__restrict__ f, unsigned short *__restrict__ out, float *__restrict__ scale, int kh, int kw, int c, int oc) {
    __shared__ uint2 warps[4];
    grid_dependency_sync();
    const int o = blockIdx.x;
    auto value = [&](int i) {  // k = ky * 32 + kx * 4 + channel
        const int ky = i >> 5, kx = (i >> 2) & 7, cc = i & 3;
        return (o < oc && kx < kw && cc < c) ? f[(((long long)ky * kw + kx) * c + cc) * oc + o] : 0.f;
    };
    unsigned m = 0, low1 = 0xffffffffu;
    for (int i = threadIdx.x; i < kh * 32; i += 128) {
        const unsigned b = sage_tc::h2_finite_bits(value(i));
        m = max(m, b);
        low1 = min(low1, b - 1u);
    }
    m = __reduce_max_sync(0xffffffffu, m);
    low1 = __reduce_min_sync(0xffffffffu, low1);
    if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = make_uint2(m, low1);
    __syncthreads();
    m = max(max(warps[0].x, warps[1].x), max(warps[2].x, warps[3].x));
    low1 = min(min(warps[0].y, warps[1].y), min(warps[2].y, warps[3].y));
    float s;
    const float factor = sage_tc::h2_factor(m, &s);
    if (threadIdx.x == 0) scale[o] = first_wide(m, low1) ? -s : s;
    unsigned short *tile = out + (long long)(o >> 6) * kh * 4096;
    for (int i = threadIdx.x * 2; i < kh * 32; i += 256) {
        unsigned a, l;
        sage_tc::h2_split2(value(i), value(i + 1), factor, &a, &l);
        const int at = ((i >> 3) * 128 + (o & 63)) * 8 + (i & 7);
        *reinterpret_cast<unsigned *>(tile + at) = a;
        *reinterpret_cast<unsigned *>(tile + at + 512) = l;
    }
}

sage_status pack_first_image(Context &ctx, const float *img, long long n, long long h, long long w, long long c, long long hp, long long wp, int pad_h, int pad_w,
                             unsigned short *hi, long long plane, float *scale, unsigned *scratch) {
    if (c < 1 || c > 4 || wp % 2 || plane % 8 || reinterpret_cast<uintptr_t>(hi) % 16 || reinterpret_cast<uintptr_t>(scratch) % 8 || h > 0x7fffffffLL || w > 0x7fffffffLL || hp > 0x7fffffffLL ||
        wp > 0x7fffffffLL || n > 65535 ||
        n * hp / 4 > 0x7ffffff0LL)
        return ctx.fail(SAGE_ERR_INVALID, "pack_first_image: bad arguments");
    ctx.note_launch("pack_small_c");
    ctx.note_launch("pack_small_c");
    if (ctx.dry()) return SAGE_OK;
    const long long len = h * w * c;
    uint2 *parts = reinterpret_cast<uint2 *>(scratch);
    const int vec = len % 4 == 0 && reinterpret_cast<uintptr_t>(img) % 16 == 0;
    launch_dependent(ctx.pdl, ctx.stream(), first_amax_kernel, dim3(kAmaxParts, (unsigned)n), dim3(256), 0, img, len, vec, parts);
    launch_dependent(ctx.pdl, ctx.stream(), pack_first_kernel, dim3((unsigned)((n * hp + 3) / 4)), dim3(128), 0, img, hi, plane, n * hp, (int)h, (int)w, (int)c, (int)hp, (int)wp, pad_h,
                     pad_w, (const uint2 *)parts, scale);
    return ctx.check_cuda(cudaGetLastError(), "pack_first_image launch");
}

sage_status pack_first_filter(Context &ctx, const float *filt, int kh, int kw, int c, int oc, unsigned short *out, float *scale) {
    ctx.note_launch("pack_small_c_filter");
    if (ctx.dry()) return SAGE_OK;
    if (kw > 8 || c > 4) return ctx.fail(SAGE_ERR_INVALID, "pack_first_filter: window too wide");
    return ctx.check_cuda(launch_dependent(ctx.pdl, ctx.stream(), pack_first_filter_kernel, dim3((unsigned)((oc + 63) / 64 * 64)), dim3(128), 0, filt, out, scale, kh, kw, c, oc),
                          "pack_first_filter launch");
}

sage_status im2col(Context &ctx, const float *img, float *col, long long n, long long img_h, long long img_w,
                   long long chan, long long col_h, long long col_w, const Window &w) {
    return im2col_planes(ctx, img, n, img_h, img_w, chan, col_h, col_w, w, col, nullptr, 0, 0);
}

sage_status col2im(Context &ctx, const float *col, float *img, long long n, long long img_h, long long img_w,
                   long long chan, long long col_h, long long col_w, const Window &w) {
    ConvP p{n, img_h, img_w, chan, col_h, col_w, w};
    long long total = n * img_h * img_w * chan;
    ctx.note_launch("col2im");
    if (ctx.dry() || total == 0) return SAGE_OK;
    if (chan % 4 == 0 && reinterpret_cast<uintptr_t>(col) % 16 == 0 && reinterpret_cast<uintptr_t>(img) % 16 == 0 && img_h * img_w <= 0x7fffffffLL &&
        col_h * col_w <= 0x7fffffffLL && w.dil_w >= 1 && w.dil_h >= 1) {
        launch_dependent(ctx.pdl, ctx.stream(), col2im_quads_kernel, dim3(grid_for(ctx, total / 4)), dim3(256), 0, col, img, p, total / 4);
        return ctx.check_cuda(cudaGetLastError(), "col2im launch");
    }
    launch_dependent(ctx.pdl, ctx.stream(), col2im_kernel, dim3(grid_for(ctx, total)), dim3(256), 0, col, img, p, total);
    return ctx.check_cuda(cudaGetLastError(), "col2im launch");
}

// ---- with a map spliced in
bool cols_mappable(const void *a, const void *b, long long img_h, long long img_w, long long chan, long long col_h, long long col_w, const Window &w) {
    return chan % 4 == 0 && reinterpret_cast<uintptr_t>(a) % 16 == 0 && reinterpret_cast<uintptr_t>(b) % 16 == 0 && img_h * img_w <= 0x7fffffffLL && col_h * col_w <= 0x7fffffffLL &&
           w.dil_w >= 1 && w.dil_h >= 1 && (long long)w.ker_h * w.ker_w * chan <= 0x7fffffffLL;
}
static sage_status cols_module(Context &ctx, const char *what, const std::string &expr, int naux, Module **mod) {
    const std::string key = std::string(what) + " " + std::to_string(naux) + "\n" + expr;
    *mod = ctx.module_find(key);
    if (*mod) return SAGE_OK;
    const bool pre = what[0] == 'i';
    std::string src = map_prelude_text();
    src += "struct Window { int ker_w, ker_h, stride_w, stride_h, pad_w, pad_h, dil_w, dil_h; };\n"
           "struct ConvP { long long n, img_h, img_w, chan, col_h, col_w; Window w; };\n"
           "#define SAGE_COLS_SPLIT sg_split_tf32\n#define SAGE_COLS_NAUX " + std::to_string(naux) + "\n";
    src += "#define SAGE_COLS_PRE(x0) (" + (pre ? expr : std::string("x0")) + ")\n#define SAGE_COLS_POST(x0, x1, x2, x3) (" + (pre ? std::string("x0") : expr) + ")\n";
    src += kConvColsDeviceSrc;
    const char *wait = "    asm volatile(\"griddepcontrol.launch_dependents;\" ::: \"memory\");\n    asm volatile(\"griddepcontrol.wait;\" ::: \"memory\");\n";
    if (pre)
        src += std::string("extern \"C\" __global__ void __launch_bounds__(256) sage_im2col(const float *img, float *col, float *hi, const long long plane, const int pitch, const ConvP p, const long long pixels, const int share) {\n") + wait +
               "    const long long warp = (long long)blockIdx.x * 8 + (threadIdx.x >> 5), pix = warp / share;\n"
               "    if (pix >= pixels) return;\n"
               "    const long long per_img = p.col_h * p.col_w, n = pix / per_img;\n"
               "    const int r = (int)(pix - n * per_img), oy = r / (int)p.col_w, ox = r % (int)p.col_w;\n"
               "    im2col_quads_of_pixel(img + n * p.img_h * p.img_w * p.chan, col, hi, plane, pitch, p, pix, oy * p.w.stride_h - p.w.pad_h, ox * p.w.stride_w - p.w.pad_w,\n"
               "                          (int)(threadIdx.x & 31) + 32 * (int)(warp - pix * share), 32 * share);\n}\n";
    else
        src += std::string("extern \"C\" __global__ void __launch_bounds__(256) sage_col2im(const float *col, float *img, float *hi, const long long plane, const ConvP p, const long long total, const float *x1, const float *x2, const float *x3) {\n") + wait +
               "    col2im_quads(col, img, hi, plane, p, total, x1, x2, x3);\n}\n";
    sage_status st = ctx.module_get(src, mod);
    if (!st) ctx.module_remember(key, *mod);
    return st;
}

sage_status im2col_mapped(Context &ctx, const std::string &expr, const float *img, long long n, long long img_h, long long img_w, long long chan, long long col_h, long long col_w, const Window &w,
                          float *col, float *hi, long long plane, int pitch) {
    ConvP p{n, img_h, img_w, chan, col_h, col_w, w};
    const long long pixels = n * col_h * col_w;
    if (!cols_mappable(img, col, img_h, img_w, chan, col_h, col_w, w) || reinterpret_cast<uintptr_t>(hi) % 16 || plane % 4 || pitch % 4 || (pixels * 16 + 7) / 8 > 0x7fffffffLL)
        return ctx.fail(SAGE_ERR_UNSUPPORTED, "im2col: not addressable four channels at a time");
    Module *mod = nullptr;
    sage_status st = cols_module(ctx, "im2col", expr, 0, &mod);
    if (st || pixels == 0) return st;
    int share = 1;
    const long long length = w.ker_h * w.ker_w * chan / 4;  // loads of a pixel
    while (share < 16 && pixels * share < 32LL * ctx.sm_count && length >= 128LL * share) share *= 2;
    long long pix = pixels;
    void *params[8] = {&img, &col, &hi, &plane, &pitch, &p, &pix, &share};
    const uint32_t grid[3] = {(uint32_t)((pixels * share + 7) / 8), 1, 1}, block[3] = {256, 1, 1};
    return ctx.launch(mod, "sage_im2col", grid, block, 0, params, ctx.verbose_names ? (col ? "im2col{map}" : "im2col{map}=planes") : "im2col", true);
}

sage_status col2im_mapped(Context &ctx, const std::string &expr, int naux, const float *const aux[3], const float *col, float *img, float *hi, long long plane, long long n, long long img_h,
                          long long img_w, long long chan, long long col_h, long long col_w, const Window &w) {
    ConvP p{n, img_h, img_w, chan, col_h, col_w, w};
    long long total = n * img_h * img_w * chan / 4;
    if (!cols_mappable(col, img, img_h, img_w, chan, col_h, col_w, w) || reinterpret_cast<uintptr_t>(hi) % 16 || plane % 4) return ctx.fail(SAGE_ERR_UNSUPPORTED, "col2im: not addressable four channels at a time");
    for (int i = 0; i < naux; ++i)
        if (reinterpret_cast<uintptr_t>(aux[i]) % 16) return ctx.fail(SAGE_ERR_UNSUPPORTED, "col2im: not addressable four channels at a time");
    Module *mod = nullptr;
    sage_status st = cols_module(ctx, "col2im", expr, naux, &mod);
    if (st || total == 0) return st;
    const float *x[3] = {aux[0], aux[1], aux[2]};
    void *params[9] = {&col, &img, &hi, &plane, &p, &total, &x[0], &x[1], &x[2]};
    const uint32_t grid[3] = {grid_for(ctx, total), 1, 1}, block[3] = {256, 1, 1};
    return ctx.launch(mod, "sage_col2im", grid, block, 0, params, ctx.verbose_names ? "col2im{map}" : "col2im", true);
}

bool pool2d_writes_pieces(const float *img, long long chan, long long out_h, long long out_w) {
    return chan % 64 == 0 && reinterpret_cast<uintptr_t>(img) % 16 == 0 && out_h * out_w <= 0x7fffffffLL;
}

sage_status pool2d(Context &ctx, bool is_max, const float *img, float *out, long long n, long long img_h,
                   long long img_w, long long chan, long long out_h, long long out_w, const Window &w, const PlaneOut &forms) {
    ConvP p{n, img_h, img_w, chan, out_h, out_w, w};
    long long total = n * out_h * out_w * chan;
    const bool vec = chan % 4 == 0 && reinterpret_cast<uintptr_t>(img) % 16 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0 &&
                     out_h * out_w <= 0x7fffffffLL;
    const long long chan_blocks = (chan + 63) / 64;
    // A window's taps shared between threads: from two rounds of taps on, while the blocks are few enough to run at once.
    const bool window = vec && out && !forms.h2 && w.ker_w * w.ker_h >= 16 && n * out_h * out_w * chan_blocks <= 4LL * ctx.sm_count && img_h <= 0x7fffffffLL && img_w <= 0x7fffffffLL;
    ctx.note_launch(ctx.verbose_names && window ? (is_max ? "max_pool2d[window]" : "avg_pool2d[window]") : is_max ? "max_pool2d" : "avg_pool2d");
    if (ctx.dry() || total == 0) return SAGE_OK;
    if (forms.h2 && !(vec && pool2d_writes_pieces(img, chan, out_h, out_w))) return ctx.fail(SAGE_ERR_INVALID, "pool2d: half-precision pieces need whole groups of channels");
    // 32-bit indices where they reach: two 64-bit divisions were a third of a thread's instructions
    const bool narrow = total < (1LL << 31) && img_h * img_w * chan < (1LL << 31);
    const bool mark = forms.h2 && forms.h2_marked;
    if (window) {
        launch_dependent(ctx.pdl, ctx.stream(), pool2d_window_kernel, dim3((unsigned)(n * out_h * out_w * chan_blocks)), dim3(256), 0, img, out, p, (int)chan_blocks, is_max ? 1 : 0, (int)ctx.opts().ref_compat);
        return ctx.check_cuda(cudaGetLastError(), "pool2d launch");
    }
    auto kernel = narrow ? (mark ? pool2d_kernel<4, unsigned, true> : pool2d_kernel<4, unsigned, false>) : (mark ? pool2d_kernel<4, long long, true> : pool2d_kernel<4, long long, false>);
    if (vec) launch_dependent(ctx.pdl, ctx.stream(), kernel, dim3(grid_for(ctx, total / 4)), dim3(256), 0, img, out, p, total / 4, is_max ? 1 : 0, (int)ctx.opts().ref_compat, forms);
    else launch_dependent(ctx.pdl, ctx.stream(), pool2d_kernel<1, long long, false>, dim3(grid_for(ctx, total)), dim3(256), 0, img, out, p, total, is_max ? 1 : 0, (int)ctx.opts().ref_compat, forms);
    return ctx.check_cuda(cudaGetLastError(), "pool2d launch");
}

}  // namespace k
}  // namespace sage
