// Host side of the half-precision-pieces GEMM (gemm_h2_device.inc) and the kernels that bring fp32 data into its operand
// form.  Reference: Gemm::compute_direct / GemmBatched::compute_direct (src/ops/gemm.rs:176-250, 338-421).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "kernels.h"
#include "launch.h"
// the kernels compiled here store the plain fp32 product
#define SAGE_EPI_OUT 1
#define SAGE_EPI_COLS 0
#include "gemm_tc_device.inc"
#include "gemm_h2_device.inc"
#include "attn_tc_device.inc"  // AttnParams and the tile constants; the kernel itself is only compiled by NVRTC
#include "attn_small_device.inc"
#include "gemm_tc_device_src.h"
#include "gemm_h2_device_src.h"
#include "attn_quads_device_src.h"
#include "attn_rows_device_src.h"
#include "attn_small_device_src.h"
#include "attn_tc_device_src.h"
#include "conv_first_device.inc"
#include "conv_first_device_src.h"

namespace sage {
void *driver_symbol(const char *name);  // runtime/context.cc
const char *map_prelude_text();         // codegen/map_emit.cc
namespace k {

using namespace sage_tc;

namespace {

bool aligned16(const void *p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

// ---------------------------------------------------------------------------------- operand forms
// Flat: 16 lanes hold the 64 floats of a group.  Bound by memory: 4 bytes read, 4.06 written per element.
template <bool MARK>
__global__ void __launch_bounds__(256) split_h2_flat_kernel(const float4 *__restrict__ src, long long n4, uint2 *__restrict__ hi, uint2 *__restrict__ lo,
                                                            float *__restrict__ scale, float *__restrict__ marked) {
    grid_dependency_sync();
    for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < n4; g += (long long)gridDim.x * blockDim.x) {
        const float4 x = src[g];  // n4 is a multiple of 16: the lanes of a group are all here or all gone
        unsigned b = max(max(h2_finite_bits(x.x), h2_finite_bits(x.y)), max(h2_finite_bits(x.z), h2_finite_bits(x.w)));
        const unsigned lanes = 0xffffu << (threadIdx.x & 16);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) b = max(b, __shfl_xor_sync(lanes, b, o));
        float s;
        const float f = h2_factor(b, &s);
        uint2 h, l;
        h2_split2(x.x, x.y, f, &h.x, &l.x);
        h2_split2(x.z, x.w, f, &h.y, &l.y);
        hi[g] = h;
        lo[g] = l;
        if ((threadIdx.x & 15) == 0) scale[g >> 4] = s;
        if (MARK) {
            unsigned low1 = min(min(h2_low1(x.x), h2_low1(x.y)), min(h2_low1(x.z), h2_low1(x.w)));
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) low1 = min(low1, __shfl_xor_sync(lanes, low1, o));
            if ((threadIdx.x & 15) == 0) marked[g >> 4] = h2_wide(low1, f) ? -s : s;
        }
    }
}

struct ViewP {
    const float *src;
    long long nb0, sb0, sb1, ld, cs;  // row and column strides of the source
    long long rows, cols, pitch, plane;
    int row_tiles, col_tiles;
    int vec;  // whole 16-byte loads along the contiguous axis are aligned and inside
};

// Single elements of a 64 x 64 tile, four lines of 64 at a time along whichever axis is contiguous.
__device__ __forceinline__ bool along_columns(const ViewP &v) { return v.cs == 1 || v.ld != 1; }
__device__ __forceinline__ void load_singles(const ViewP &v, const float *s, long long r0, long long c0, float (&x)[16]) {
    const int fast = threadIdx.x & 63, slow = threadIdx.x >> 6;
    const bool columns = along_columns(v);
    const long long r = r0 + (columns ? slow : fast), c = c0 + (columns ? fast : slow), step = columns ? 4 * v.ld : 4 * v.cs;
    const int left = (int)min(columns ? v.rows - r : v.cols - c, 64LL);
    const float *at = s + r * v.ld + c * v.cs;
    const bool in = columns ? c < v.cols : r < v.rows;
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = in && 4 * i < left ? at[i * step] : 0.f;
}
__device__ __forceinline__ void store_singles(const ViewP &v, const float (&x)[16], float (*tile)[65]) {
    const int fast = threadIdx.x & 63, slow = threadIdx.x >> 6;
    float *at = along_columns(v) ? &tile[slow][fast] : &tile[fast][slow];
    const int step = along_columns(v) ? 4 * 65 : 4;
#pragma unroll
    for (int i = 0; i < 16; ++i) at[i * step] = x[i];
}
// A 64 x 64 tile of the view into shared memory, read along whichever axis is contiguous (256 threads).
__device__ __forceinline__ void load_tile(const ViewP &v, const float *s, long long r0, long long c0, float (*tile)[65]) {
    const int t = threadIdx.x;
    if (v.vec && v.cs != 1) {
        const int r4 = (t & 15) * 4, line = t >> 4;
        float4 q[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const long long r = r0 + r4, c = c0 + line + 16 * i;
            q[i] = r < v.rows && c < v.cols ? *reinterpret_cast<const float4 *>(s + r + c * v.cs) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int c = line + 16 * i;
            tile[r4][c] = q[i].x;
            tile[r4 + 1][c] = q[i].y;
            tile[r4 + 2][c] = q[i].z;
            tile[r4 + 3][c] = q[i].w;
        }
    } else {
        float x[16];
        load_singles(v, s, r0, c0, x);
        store_singles(v, x, tile);
    }
}
// A row of the tile per 4 lanes, columns 8 * part .. and 32 + 8 * part .. each: no bank conflicts, and the four lanes' 16-byte
// stores lie side by side
__device__ __forceinline__ void tile_row(const float (*tile)[65], float (&y)[16]) {
    const float *t = tile[threadIdx.x >> 2] + (threadIdx.x & 3) * 8;
#pragma unroll
    for (int i = 0; i < 16; ++i) y[i] = t[(i & 7) + (i & 8) * 4];
}
__device__ __forceinline__ unsigned row_amax(const float (&y)[16]) {
    float m = 0.f;  // (fmaxf passes over nan)
#pragma unroll
    for (int i = 0; i < 16; ++i) m = fmaxf(m, fabsf(y[i]));
    unsigned b = __float_as_uint(m);
    if (b >= 0x7f800000u) {
        b = 0u;
#pragma unroll
        for (int i = 0; i < 16; ++i) b = max(b, h2_finite_bits(y[i]));
    }
    b = max(b, __shfl_xor_sync(0xffffffffu, b, 1));
    return max(b, __shfl_xor_sync(0xffffffffu, b, 2));
}
// ... split and stored at `d`, `left` before the row's end in memory (whole 16-byte pieces, zeros behind the last column).
__device__ __forceinline__ void store_row(const float (&y)[16], float factor, unsigned short *d, long long plane, int left) {
    unsigned h[8], l[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) h2_split2(y[2 * i], y[2 * i + 1], factor, &h[i], &l[i]);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        if (32 * i >= left) break;
        *reinterpret_cast<uint4 *>(d + 32 * i) = make_uint4(h[4 * i], h[4 * i + 1], h[4 * i + 2], h[4 * i + 3]);
        *reinterpret_cast<uint4 *>(d + plane + 32 * i) = make_uint4(l[4 * i], l[4 * i + 1], l[4 * i + 2], l[4 * i + 3]);
    }
}

// Where an operand's pieces go.
struct SplitOut {
    unsigned short *hi;
    float *scale, *ratio;
    float *marked;  // MARK
    unsigned long long *columns;
};
__device__ __forceinline__ unsigned row_low1(const float (&y)[16]) {
    unsigned low1 = 0xffffffffu;
#pragma unroll
    for (int i = 0; i < 16; ++i) low1 = min(low1, h2_low1(y[i]));
    return low1;
}

// A thread's four 16-byte loads of a tile: of one row (its columns contiguous; as tile_row has them), or of four rows and two pairs
// of columns.  `at`: its first one, null for rows outside; `left`: columns from there to the view's end.
template <bool FOUR_ROWS>
__device__ __forceinline__ void load_quads(const float *at, long long cs, int left, float4 (&q)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int step = (FOUR_ROWS ? (i & 1) : (i & 1) * 4) + (i >> 1) * 32;
        q[i] = at && step < left ? *reinterpret_cast<const float4 *>(at + (FOUR_ROWS ? step * cs : step)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}
__device__ __forceinline__ void quads_row(const float4 (&q)[4], float (&y)[16]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        y[4 * i] = q[i].x;
        y[4 * i + 1] = q[i].y;
        y[4 * i + 2] = q[i].z;
        y[4 * i + 3] = q[i].w;
    }
}
__device__ __forceinline__ const float *batch_of(const ViewP &v, unsigned b) {
    return b == 0 ? v.src : v.src + (b / (unsigned)v.nb0) * v.sb1 + (b % (unsigned)v.nb0) * v.sb0;
}

// Operand A: a scale per row and 64 columns.  A block takes `run` tiles side by side, the next one's rows on their way.
template <bool MARK>
__device__ __forceinline__ void split_tiles(const ViewP &v, const SplitOut &o, unsigned block, int run, float (*tile)[65]) {
    const unsigned runs = (unsigned)(v.col_tiles + run - 1) / run, line = block / runs, b = line / (unsigned)v.row_tiles;
    const int first = (int)(block - line * runs) * run, last = min(v.col_tiles, first + run);
    const long long r0 = (long long)(line - b * v.row_tiles) * 64, r = r0 + (threadIdx.x >> 2), at_row = b * v.rows + r;
    const float *s = batch_of(v, b);
    const bool straight = v.vec && v.cs == 1, in = r < v.rows;
    const int c = (threadIdx.x & 3) * 8;
    const float *at = straight && in ? s + r * v.ld + c : nullptr;
    float4 q[4];
    if (straight) load_quads<false>(at ? at + first * 64 : nullptr, 1, (int)v.cols - c - first * 64, q);
    for (int t = first; t < last; ++t) {
        float y[16], scale;
        if (straight) {
            quads_row(q, y);
            if (t + 1 < last) load_quads<false>(at ? at + (t + 1) * 64 : nullptr, 1, (int)v.cols - c - (t + 1) * 64, q);
        } else {
            if (t != first) __syncthreads();
            load_tile(v, s, r0, (long long)t * 64, tile);
            __syncthreads();
            tile_row(tile, y);
        }
        const float f = h2_factor(row_amax(y), &scale);
        [[maybe_unused]] bool wide = false;
        if (MARK) {
            unsigned low1 = row_low1(y);
            low1 = min(low1, __shfl_xor_sync(0xffffffffu, low1, 1));
            wide = h2_wide(min(low1, __shfl_xor_sync(0xffffffffu, low1, 2)), f);
        }
        if (!in) continue;
        if ((threadIdx.x & 3) == 0) {
            o.scale[at_row * v.col_tiles + t] = scale;
            if (MARK) o.marked[at_row * v.col_tiles + t] = wide ? -scale : scale;
        }
        store_row(y, f, o.hi + at_row * v.pitch + t * 64 + c, v.plane, (int)v.pitch - t * 64 - c);
    }
}

// Operand B: a scale per row, and a factor per 64 rows and 64 columns (of K).  A cluster of CTAs shares 64 rows, each with a run of
// their columns.  First look: the largest exponent of every tile, and of every row in it; each row's largest relative to the tiles'
// is then exchanged through distributed shared memory, and the columns are read again, from L2.
// The tile after the present one is on its way in both looks.  With whole 16-byte loads the first look needs neither a transposition
// nor a barrier a tile, and rows that lie across are split before they are turned round, as pairs.
// Keeping the tiles in shared memory between the two looks (one read, 133 KB a CTA) left one block per SM: 4096 x 4096 80 us.
// (Every shuffle and vote below is outside of conditions that differ between a warp's rows.)
constexpr int kFactors = 64;  // of a CTA: K up to 2^15 has one per 64, beyond it `span` tiles share one
struct RowsShared {
    union {
        float tiles[2][64][65];
        uint4 pieces[2][2][64][8];             // [buffer][hi, lo][row]: 16-byte chunks, a row's swizzled by piece_swizzle
        unsigned warp_words[kFactors][8][16];  // first look, four rows to a thread: their exponents, a warp's
    };
    int row_rel[64], cta_top;
    __align__(16) int row_scale[64];                    // biased exponent of a row's scale times 2^14
    __align__(16) unsigned char row_top[kFactors][64];  // biased exponents of the largest elements, 0 for none
    unsigned char tile_top[kFactors];
};
// Writers: sixteen rows four apart, the same chunk; readers: two neighbouring rows, four chunks each.
__device__ __forceinline__ int piece_swizzle(int row) { return ((row >> 2) ^ (row << 2)) & 7; }
// Biased exponent of a magnitude that fmaxf found (it passes over nan), 0 for none (27: 2^-100, as in h2_factor), 255 for inf.
__device__ __forceinline__ unsigned h2_exponent(float m) {
    const unsigned b = __float_as_uint(m);
    return b == 0u ? 0u : max(b >> 23, 27u);
}
__device__ __forceinline__ float largest4(float a, float b, float c, float d) { return fmaxf(fmaxf(fabsf(a), fabsf(b)), fmaxf(fabsf(c), fabsf(d))); }
__device__ __forceinline__ float largest_finite4(float a, float b, float c, float d) {
    return __uint_as_float(max(max(h2_finite_bits(a), h2_finite_bits(b)), max(h2_finite_bits(c), h2_finite_bits(d))));
}
__device__ __forceinline__ bool is_finite(float m) { return m < __uint_as_float(0x7f800000u); }

enum { kRowsAny, kRowsOne, kRowsFour };  // a thread's loads: single elements; 16 bytes of one row; 16 bytes of four rows
template <int LOADS, bool MARK>
__device__ __forceinline__ void split_rows(const ViewP &v, const SplitOut &o, unsigned block, int ctas, int tiles_per_cta, int span, RowsShared &sh) {
    const unsigned group = block / (unsigned)ctas, rank = block - group * ctas, b = group / (unsigned)v.row_tiles;
    const long long r0 = (long long)(group - b * v.row_tiles) * 64;
    const float *s = batch_of(v, b);
    const int first = (int)rank * tiles_per_cta, last = min(v.col_tiles, first + tiles_per_cta), row = threadIdx.x >> 2;
    const int factors = first < last ? (last - first + span - 1) / span : 0;
    const bool row_lane = (threadIdx.x & 3) == 0, row_in = r0 + row < v.rows;
    constexpr bool four = LOADS == kRowsFour, any = LOADS == kRowsAny;
    const int r4 = (threadIdx.x & 15) * 4, line = threadIdx.x >> 4;  // four: this thread's rows, and half its first column
    const int c = four ? line * 2 : (threadIdx.x & 3) * 8, cols = (int)v.cols;
    const float *at = nullptr;
    if (!any) {
        const long long r = r0 + (four ? r4 : row);
        if (r < v.rows) at = s + (four ? r + c * v.cs : r * v.ld + c);
    }
    float4 q[4], next[4];
    float x[16];  // single elements, as they are loaded
    auto load = [&](int t, float4 (&to)[4]) {
        if constexpr (any) load_singles(v, s, r0, (long long)t * 64, x);
        else load_quads<four>(at ? at + (four ? t * 64 * v.cs : (long long)t * 64) : nullptr, v.cs, cols - c - t * 64, to);
    };
    // ---- first look
    load(first, q);
    float m[4] = {0.f, 0.f, 0.f, 0.f};  // four rows' largest, or one's
    for (int t = first, left = span, i = 0; t < last; ++t) {
        float y[16];
        if constexpr (any) {
            store_singles(v, x, sh.tiles[t & 1]);
            if (t + 1 < last) load(t + 1, next);
            __syncthreads();
            tile_row(sh.tiles[t & 1], y);
        } else if (t + 1 < last) {
            load(t + 1, next);
        }
        if constexpr (four) {
            float n[4] = {largest4(q[0].x, q[1].x, q[2].x, q[3].x), largest4(q[0].y, q[1].y, q[2].y, q[3].y), largest4(q[0].z, q[1].z, q[2].z, q[3].z),
                          largest4(q[0].w, q[1].w, q[2].w, q[3].w)};
            if (!is_finite(largest4(n[0], n[1], n[2], n[3]))) {
                n[0] = largest_finite4(q[0].x, q[1].x, q[2].x, q[3].x);
                n[1] = largest_finite4(q[0].y, q[1].y, q[2].y, q[3].y);
                n[2] = largest_finite4(q[0].z, q[1].z, q[2].z, q[3].z);
                n[3] = largest_finite4(q[0].w, q[1].w, q[2].w, q[3].w);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) m[j] = fmaxf(m[j], n[j]);
        } else {
            if constexpr (!any) quads_row(q, y);
            float n = 0.f;
#pragma unroll
            for (int k = 0; k < 16; k += 4) n = fmaxf(n, largest4(y[k], y[k + 1], y[k + 2], y[k + 3]));
            if (!is_finite(n)) {
                n = 0.f;
#pragma unroll
                for (int k = 0; k < 16; k += 4) n = fmaxf(n, largest_finite4(y[k], y[k + 1], y[k + 2], y[k + 3]));
            }
            m[0] = fmaxf(m[0], n);
        }
        if (--left == 0 || t == last - 1) {
            if constexpr (four) {
                unsigned lo = h2_exponent(m[0]) | h2_exponent(m[1]) << 16, hi = h2_exponent(m[2]) | h2_exponent(m[3]) << 16;
                lo = __vmaxu2(lo, __shfl_xor_sync(0xffffffffu, lo, 16));
                hi = __vmaxu2(hi, __shfl_xor_sync(0xffffffffu, hi, 16));
                if ((threadIdx.x & 16) == 0) sh.warp_words[i][threadIdx.x >> 5][threadIdx.x & 15] = __byte_perm(lo, hi, 0x6420);
            } else {
                m[0] = fmaxf(m[0], __shfl_xor_sync(0xffffffffu, m[0], 1));
                m[0] = fmaxf(m[0], __shfl_xor_sync(0xffffffffu, m[0], 2));
                if (row_lane) sh.row_top[i][row] = (unsigned char)h2_exponent(m[0]);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) m[j] = 0.f;
            left = span;
            ++i;
        }
        if (!any && t + 1 < last) {
#pragma unroll
            for (int k = 0; k < 4; ++k) q[k] = next[k];
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < factors * 16; k += 256) {  // a factor to 16 lanes, a word of four rows each
        const int i = k >> 4, word = k & 15;
        unsigned *tops = reinterpret_cast<unsigned *>(sh.row_top[i]) + word, w = 0;
        if constexpr (four) {
#pragma unroll
            for (int p = 0; p < 8; ++p) w = __vmaxu4(w, sh.warp_words[i][p][word]);
            *tops = w;
        } else {
            w = *tops;
        }
        w = __vmaxu4(w, w >> 16);
        w = max(w & 0xffu, (w >> 8) & 0xffu);
        const unsigned lanes = 0xffffu << (threadIdx.x & 16);
#pragma unroll
        for (int d = 8; d > 0; d >>= 1) w = max(w, __shfl_xor_sync(lanes, w, d));
        if (word == 0) sh.tile_top[i] = (unsigned char)w;
    }
    __syncthreads();
    int rel = -1000, all = 0;  // this row's largest exponent relative to its tile's; the largest of all
    for (int i = 0; i < factors; ++i) {
        const int top = sh.tile_top[i], e = sh.row_top[i][row];
        rel = e == 0 ? rel : max(rel, e - top);
        all = max(all, top);
    }
    if (ctas > 1) {
        if (row_lane) sh.row_rel[row] = rel;
        if (threadIdx.x == 0) sh.cta_top = all;
        cluster_sync_all();
        const unsigned rel_at = smem_u32(&sh.row_rel[row]), top_at = smem_u32(&sh.cta_top);
        for (int p = 0; p < ctas; ++p) {
            int d, w;
            asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(d) : "r"(peer_addr(rel_at, p)) : "memory");
            asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(w) : "r"(peer_addr(top_at, p)) : "memory");
            rel = max(rel, d);
            all = max(all, w);
        }
        cluster_sync_all();  // nobody leaves while a peer may still read its shared memory
    }
    int se[4];  // biased exponent of the scale of this thread's row(s), times 2^14
    se[0] = max(rel + all, 27);
    const long long at_row = b * v.rows + r0 + row;
    if (rank == 0 && row_lane && row_in) o.scale[at_row] = __uint_as_float((unsigned)(se[0] - 14) << 23);
    if constexpr (four) {
        if (row_lane) sh.row_scale[row] = se[0];
        __syncthreads();
        const int4 w = *reinterpret_cast<const int4 *>(&sh.row_scale[r4]);
        se[0] = w.x;
        se[1] = w.y;
        se[2] = w.z;
        se[3] = w.w;
    }
    // ---- second look, backwards: the last tile is still in registers (single elements: in its buffer, and the one before it too)
    if (any && last - 3 >= first) load(last - 3, next);
    const int lowest = four ? min(min(se[0], se[1]), min(se[2], se[3])) : se[0];
    const int part = (threadIdx.x & 3) * 8;
    unsigned short *d = o.hi + at_row * v.pitch + part;
    float *ratio = o.ratio + (long long)group * v.col_tiles;
    // 2^f: a tile's factor
    const auto factor_of = [&](int t) {
        const int top = sh.tile_top[span == 1 ? t - first : (t - first) / span];
        return top == 0 ? 0 : max(top - all, -kH2Far);
    };
    [[maybe_unused]] float *marked = MARK ? o.marked + (long long)group * v.col_tiles : nullptr;
    [[maybe_unused]] unsigned long long *columns = MARK ? o.columns + (long long)group * v.col_tiles : nullptr;
    if (MARK) {  // none, before the first thread that finds one
        for (int t = first + threadIdx.x; t < last; t += 256) {
            marked[t] = __uint_as_float((unsigned)(127 + factor_of(t)) << 23);
            columns[t] = 0;
        }
        __syncthreads();
    }
    [[maybe_unused]] const auto mark = [&](int t, unsigned long long rows) {
        atomicOr(reinterpret_cast<unsigned *>(marked + t), 0x80000000u);
        atomicOr(columns + t, rows);
    };
    for (int t = last - 1; t >= first; --t) {
        const int f = factor_of(t);
        if (threadIdx.x == 0) ratio[t] = __uint_as_float((unsigned)(127 + f) << 23);
        float factor[4];
#pragma unroll
        for (int j = 0; j < (four ? 4 : 1); ++j) factor[j] = __uint_as_float((unsigned)(268 - se[j] - f) << 23);  // (se + f: at least the row's largest in this tile)
        const bool far = lowest + f < 27;  // a factor would not be finite: two steps, both exact
        if constexpr (four) {
            if (t > first) load(t - 1, next);
            if (far) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (se[j] + f >= 27) continue;
                    const float up = __uint_as_float((unsigned)(127 + 27 - se[j] - f) << 23);
                    factor[j] = __uint_as_float((unsigned)(268 - 27) << 23);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (j == 0) q[i].x *= up;
                        if (j == 1) q[i].y *= up;
                        if (j == 2) q[i].z *= up;
                        if (j == 3) q[i].w *= up;
                    }
                }
            }
            if (MARK) {
                unsigned rows = h2_wide(min(min(h2_low1(q[0].x), h2_low1(q[1].x)), min(h2_low1(q[2].x), h2_low1(q[3].x))), factor[0]) ? 1u : 0u;
                rows |= h2_wide(min(min(h2_low1(q[0].y), h2_low1(q[1].y)), min(h2_low1(q[2].y), h2_low1(q[3].y))), factor[1]) ? 2u : 0u;
                rows |= h2_wide(min(min(h2_low1(q[0].z), h2_low1(q[1].z)), min(h2_low1(q[2].z), h2_low1(q[3].z))), factor[2]) ? 4u : 0u;
                rows |= h2_wide(min(min(h2_low1(q[0].w), h2_low1(q[1].w)), min(h2_low1(q[2].w), h2_low1(q[3].w))), factor[3]) ? 8u : 0u;
                if (rows) mark(t, (unsigned long long)rows << r4);
            }
            unsigned *hi = reinterpret_cast<unsigned *>(sh.pieces[t & 1][0][r4]), *lo = reinterpret_cast<unsigned *>(sh.pieces[t & 1][1][r4]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const float4 &qa = q[2 * half], &qb = q[2 * half + 1];
                    unsigned h, l;
                    h2_split2(j == 0 ? qa.x : j == 1 ? qa.y : j == 2 ? qa.z : qa.w, j == 0 ? qb.x : j == 1 ? qb.y : j == 2 ? qb.z : qb.w, factor[j], &h, &l);
                    const int word = j * 32 + (((line >> 2) + 4 * half) ^ piece_swizzle(r4 + j)) * 4 + (line & 3);
                    hi[word] = h;
                    lo[word] = l;
                }
            }
            __syncthreads();  // (one a tile: the buffer's next writers have passed the barrier behind these reads)
            if (row_in) {
                const int left = (int)v.pitch - t * 64 - part;  // pitch is a multiple of 8: whole 16-byte pieces, zeros behind the last column
                unsigned short *to = d + t * 64;
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    if (32 * half >= left) break;
                    const int chunk = ((threadIdx.x & 3) + 4 * half) ^ piece_swizzle(row);
                    *reinterpret_cast<uint4 *>(to + 32 * half) = sh.pieces[t & 1][0][row][chunk];
                    *reinterpret_cast<uint4 *>(to + v.plane + 32 * half) = sh.pieces[t & 1][1][row][chunk];
                }
            }
            if (t > first) {
#pragma unroll
                for (int i = 0; i < 4; ++i) q[i] = next[i];
            }
        } else {
            float y[16];
            if constexpr (any) {
                if (t < last - 2) {
                    if (t == last - 3) __syncthreads();  // the two tiles that lay in the buffers have been read
                    store_singles(v, x, sh.tiles[t & 1]);
                    if (t > first) load(t - 1, next);
                    __syncthreads();
                }
                tile_row(sh.tiles[t & 1], y);
            } else {
                quads_row(q, y);
                if (t > first) load(t - 1, q);
            }
            if (far) {
                const float up = __uint_as_float((unsigned)(127 + 27 - se[0] - f) << 23);
                factor[0] = __uint_as_float((unsigned)(268 - 27) << 23);
#pragma unroll
                for (int i = 0; i < 16; ++i) y[i] *= up;
            }
            if (MARK && h2_wide(row_low1(y), factor[0])) mark(t, 1ull << row);
            if (row_in) store_row(y, factor[0], d + t * 64, v.plane, (int)v.pitch - t * 64 - part);
        }
    }
}

// Operand B's blocks (in clusters of `ctas`), then operand A's; a launch may have either kind alone.  A plain product brings both in
// with one launch: the second kernel's start and its first loads no longer follow the first one's end.  Whole calls, us, two kernels
// | one: 997 x 1234 x 777 28.4 | 26.2, 512^3 17 | 14, 12 x (300 x 400 x 500) 39.5 | 31, 1000 x 100 x 5000 52.6 | 39, 8192 x 64 x 1024
// 29.4 | 24.4, 4096^3 (320 MB of traffic in the chain, with the last result on its way out of L2) 388 | 380.
struct SplitPair {
    ViewP a, b;
    SplitOut out_a, out_b;
    unsigned b_blocks, a_blocks;
    int ctas, tiles_per_cta, span, run;
};
template <bool MARK>
__global__ void __launch_bounds__(256, 4) split_h2_kernel(const __grid_constant__ SplitPair p) {
    __shared__ RowsShared sh;
    grid_dependency_sync();
    const unsigned block = blockIdx.x;
    if (block < p.b_blocks) {
        if (!p.b.vec) split_rows<kRowsAny, MARK>(p.b, p.out_b, block, p.ctas, p.tiles_per_cta, p.span, sh);
        else if (p.b.cs == 1) split_rows<kRowsOne, MARK>(p.b, p.out_b, block, p.ctas, p.tiles_per_cta, p.span, sh);
        else split_rows<kRowsFour, MARK>(p.b, p.out_b, block, p.ctas, p.tiles_per_cta, p.span, sh);
    } else if (block - p.b_blocks < p.a_blocks) {
        split_tiles<MARK>(p.a, p.out_a, block - p.b_blocks, p.run, sh.tiles[0]);
    }
}

}  // namespace

sage_status split_h2_flat(Context &ctx, const float *src, long long n, unsigned short *hi, long long plane, float *scale, float *marked) {
    ctx.note_launch(ctx.verbose_names ? "split_h2" : "split_tf32");  // launch lists have one name for an operand's split
    if (ctx.dry()) return SAGE_OK;
    if (!aligned16(src) || !aligned16(hi) || plane % 8 || n % 64) return ctx.fail(SAGE_ERR_INVALID, "split_h2_flat: unaligned");
    long long blocks = (n / 4 + 255) / 256;
    const long long cap = (long long)ctx.sm_count * 16;
    if (blocks > cap) blocks = cap;
    return ctx.check_cuda(launch_dependent(ctx.pdl, ctx.stream(), marked ? split_h2_flat_kernel<true> : split_h2_flat_kernel<false>, dim3((unsigned)(blocks < 1 ? 1 : blocks)), dim3(256), 0,
                                           reinterpret_cast<const float4 *>(src), n / 4, reinterpret_cast<uint2 *>(hi), reinterpret_cast<uint2 *>(hi + plane), scale, marked),
                          "split_h2_flat launch");
}

static long long h2_pitch(long long cols) { return (cols + 7) / 8 * 8; }
static size_t up256(size_t b) { return (b + 255) / 256 * 256; }

// [hi][lo][scales], operand B's [batch][rows] and behind them its factors [batch][row tiles][tiles]
size_t split_h2_bytes(long long batches, long long rows, long long cols, bool whole_rows) {
    const size_t planes = (size_t)(batches * rows * h2_pitch(cols)) * 2 * 2;
    const long long tiles = (cols + 63) / 64;
    return up256(planes) + up256((size_t)(batches * (whole_rows ? rows + (rows + 63) / 64 * tiles : rows * tiles)) * 4);
}

static ViewP view_params(const float *src, const SplitView &v, const H2Split &out) {
    ViewP p{src, v.nb0, v.sb0, v.sb1, v.ld, v.col_stride, v.rows, v.cols, out.pitch, out.plane, (int)((v.rows + 63) / 64), (int)((v.cols + 63) / 64), 0};
    p.vec = (v.col_stride == 1 || v.ld == 1) && aligned16(src) && v.sb0 % 4 == 0 && v.sb1 % 4 == 0 && (v.col_stride == 1 ? v.ld % 4 == 0 && v.cols % 4 == 0 : v.col_stride % 4 == 0 && v.rows % 4 == 0);
    return p;
}
static sage_status split_views(Context &ctx, const float *src_a, const SplitView *va, const H2Split &out_a, const float *src_b, const SplitView *vb, const H2Split &out_b) {
    SplitPair p{};
    long long a_blocks = 0, b_blocks = 0;
    p.ctas = p.tiles_per_cta = p.span = p.run = 1;
    if (va) {
        p.a = view_params(src_a, *va, out_a);
        p.out_a = SplitOut{out_a.hi, out_a.scale, nullptr, out_a.marked, nullptr};
        const long long lines = va->nb0 * va->nb1 * p.a.row_tiles, fill = (long long)ctx.sm_count * 16;
        while (p.run < 8 && lines * p.a.col_tiles >= fill * p.run * 2) p.run *= 2;  // as long as the chip is filled several times over
        a_blocks = lines * ((p.a.col_tiles + p.run - 1) / p.run);
    }
    if (vb) {
        p.b = view_params(src_b, *vb, out_b);
        p.out_b = SplitOut{out_b.hi, out_b.scale, out_b.ratio, out_b.marked, out_b.columns};
        while (p.ctas < 8 && p.ctas * 2 <= p.b.col_tiles) p.ctas *= 2;
        p.tiles_per_cta = (p.b.col_tiles + p.ctas - 1) / p.ctas;
        p.span = (p.tiles_per_cta + kFactors - 1) / kFactors;
        b_blocks = vb->nb0 * vb->nb1 * p.b.row_tiles * p.ctas;
    }
    const long long blocks = b_blocks + (a_blocks + p.ctas - 1) / p.ctas * p.ctas;
    if (blocks > 0x7fffffffLL) return ctx.fail(SAGE_ERR_UNSUPPORTED, "split_h2: extents beyond 2^31 tiles");
    p.a_blocks = (unsigned)a_blocks;
    p.b_blocks = (unsigned)b_blocks;
    const char *name = ctx.verbose_names ? "split_h2" : "split_tf32";  // launch lists have one name for an operand's split
    if (va && vb) ctx.note_part(name);
    ctx.note_launch(name);
    if (ctx.dry()) return SAGE_OK;
    // Long runs of operand B (six tiles of 64 k a CTA and more) are not launched while the kernel before still holds most of the chip:
    // the clusters that come early pile up on the SMs it leaves free, four CTAs to each, and finish last.  us a call in a row of calls,
    // two kernels as they once were | one, launched early | as now: 64 x 768 x 3072 26.6 | 27.4 | 20.7, 64 x 1024 x 4096 34.0 | 35.5 | 26.8,
    // 64 x 2048 x 8192 76.3 | 82.8 | 69.5, 512 x 1024 x 4096 44.4 | 45.6 | 37.2, 128 x 1023 x 4099 51.9 | 63.6 | 41.2, 300 x 770 x 3073
    // 47.9 | 55.5 | 35.0, 4096^3 373 | 372 | 362.  Shorter runs, and a few blocks, are better off early: 64 x 768 x 768 13.0 | 13.7,
    // 1000 x 1001 x 1002 23.5 | 23.8 late, 64 x 64 x 4096 19.0 | 20.7.
    const bool early = ctx.pdl && !(p.tiles_per_cta >= 6 && b_blocks >= 32);
    return ctx.check_cuda(launch_dependent(early, ctx.stream(), p.ctas, out_a.marked || out_b.marked ? split_h2_kernel<true> : split_h2_kernel<false>, dim3((unsigned)blocks), dim3(256), 0, p), "split_h2 launch");
}

sage_status split_h2_rows_at(Context &ctx, const float *src, const SplitView &v, const H2Split &out) { return split_views(ctx, nullptr, nullptr, H2Split(), src, &v, out); }

// The layout of an operand's pieces in `dst` (of split_h2_bytes).
static H2Split split_layout(const SplitView &v, void *dst) {
    H2Split out;
    out.pitch = h2_pitch(v.cols);
    out.plane = v.nb0 * v.nb1 * v.rows * out.pitch;
    out.hi = static_cast<unsigned short *>(dst);
    out.scale = reinterpret_cast<float *>(static_cast<char *>(dst) + up256((size_t)out.plane * 4));
    out.ratio = out.scale + v.nb0 * v.nb1 * v.rows;
    return out;
}

sage_status split_h2_view(Context &ctx, const float *src, const SplitView &v, bool whole_rows, H2Split *out, bool mark) {
    const size_t bytes = split_h2_bytes(v.nb0 * v.nb1, v.rows, v.cols, whole_rows);
    const long long marks = mark ? v.nb0 * v.nb1 * (whole_rows ? (v.rows + 63) / 64 : v.rows) * ((v.cols + 63) / 64) : 0;
    Block *block = ctx.allocator().alloc(bytes + (size_t)marks * (whole_rows ? 12 : 4));
    if (!block) return ctx.fail(SAGE_ERR_OOM, "out of memory for an operand in half-precision pieces");
    *out = split_layout(v, block->ptr);
    out->block = block;
    if (mark) {
        char *at = block->ptr + bytes;  // (a multiple of 256)
        if (whole_rows) out->columns = reinterpret_cast<unsigned long long *>(at);
        out->marked = reinterpret_cast<float *>(at + (whole_rows ? marks * 8 : 0));
    }
    return whole_rows ? split_views(ctx, nullptr, nullptr, H2Split(), src, &v, *out) : split_views(ctx, src, &v, *out, nullptr, nullptr, H2Split());
}

H2Operand h2_operand(const H2Split &s, long long batches, long long rows, long long cols, bool whole_rows) {
    H2Operand o;
    o.hi = s.hi;
    o.plane = s.plane;
    o.ld = s.pitch;
    o.rows = rows;
    o.nb0 = batches;
    o.sb0 = rows * s.pitch;
    o.scale = s.scale;
    o.ratio = s.ratio;
    o.s_row = whole_rows ? 1 : (cols + 63) / 64;
    o.s_b0 = rows * o.s_row;
    return o;
}

// ---------------------------------------------------------------------------------- launcher
typedef CUresult (*PFN_encodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                    const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                    CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
typedef CUresult (*PFN_encodeIm2col)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                     const int *, const int *, cuuint32_t, cuuint32_t, const cuuint32_t *, CUtensorMapInterleave,
                                     CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// Looked up once, by whichever thread is first.
static PFN_encodeTiled encode_tiled() {
    static const PFN_encodeTiled f = reinterpret_cast<PFN_encodeTiled>(driver_symbol("cuTensorMapEncodeTiled"));
    return f;
}
static PFN_encodeIm2col encode_im2col_mode() {
    static const PFN_encodeIm2col f = reinterpret_cast<PFN_encodeIm2col>(driver_symbol("cuTensorMapEncodeIm2col"));
    return f;
}

// dims {k, rows, batch low, batch high, piece}, box {64, box_rows, 1, 1, 1}
static bool encode_operand(PFN_encodeTiled encode, const H2Operand &op, long long k, unsigned box_rows, CUtensorMap *map) {
    const cuuint64_t row_b = (cuuint64_t)op.ld * 2;
    const cuuint64_t dims[5] = {(cuuint64_t)k, (cuuint64_t)op.rows, (cuuint64_t)op.nb0, (cuuint64_t)op.nb1, 2};
    const cuuint64_t strides[4] = {row_b, op.nb0 > 1 ? (cuuint64_t)op.sb0 * 2 : row_b, op.nb1 > 1 ? (cuuint64_t)op.sb1 * 2 : row_b, (cuuint64_t)op.plane * 2};
    const cuuint32_t box[5] = {(cuuint32_t)HK, box_rows, 1, 1, 1}, estr[5] = {1, 1, 1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5, const_cast<unsigned short *>(op.hi), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A row-dependent operand of the expression, in boxes of 128 rows x 32 columns.
static bool encode_residual(PFN_encodeTiled encode, const TcAuxArg &x, long long m, long long n, CUtensorMap *map) {
    const cuuint64_t dims[2] = {(cuuint64_t)n, (cuuint64_t)m}, strides[1] = {(cuuint64_t)x.sr * 4};
    const cuuint32_t box[2] = {32, BM}, estr[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float *>(x.ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// One piece of an NHWC image: im2col mode, 64 channels of 128 output pixels.
static bool encode_im2col(PFN_encodeIm2col encode, const H2Gemm &g, const unsigned short *base, CUtensorMap *map) {
    const cuuint64_t dims[4] = {(cuuint64_t)g.img_c, (cuuint64_t)g.img_w, (cuuint64_t)g.img_h, (cuuint64_t)g.img_n};
    const cuuint64_t strides[3] = {(cuuint64_t)g.img_c * 2, (cuuint64_t)(g.img_w * g.img_c) * 2, (cuuint64_t)(g.img_h * g.img_w * g.img_c) * 2};
    const Window &w = g.win;
    const int lower[2] = {-w.pad_w, -w.pad_h};
    const int upper[2] = {w.pad_w - (w.ker_w - 1) * w.dil_w, w.pad_h - (w.ker_h - 1) * w.dil_h};
    const cuuint32_t estr[4] = {1, (cuuint32_t)w.stride_w, (cuuint32_t)w.stride_h, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<unsigned short *>(base), dims, strides, lower, upper, (cuuint32_t)HK, (cuuint32_t)BM, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// ... and tiled, a window of box_w x box_h pixels, for tap reuse
static bool encode_halo(PFN_encodeTiled encode, const H2Gemm &g, const unsigned short *base, unsigned box_w, unsigned box_h, CUtensorMap *map) {
    const cuuint64_t dims[4] = {(cuuint64_t)g.img_c, (cuuint64_t)g.img_w, (cuuint64_t)g.img_h, (cuuint64_t)g.img_n};
    const cuuint64_t strides[3] = {(cuuint64_t)g.img_c * 2, (cuuint64_t)(g.img_w * g.img_c) * 2, (cuuint64_t)(g.img_h * g.img_w * g.img_c) * 2};
    const cuuint32_t box[4] = {(cuuint32_t)HK, box_w, box_h, 1u}, estr[4] = {1, 1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<unsigned short *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Images below 128 KiB (of fp32) are read through tiled boxes instead of im2col-mode maps or windows kept in shared memory: `rows` whole
// output rows of one image to a tile, or `imgs` whole images where several fit its 128 pixels.
struct BoxPlan {
    int imgs, rows, row_tiles;  // row_tiles: of an image
    long long tiles(const H2Gemm &g) const { return (g.img_n + imgs - 1) / imgs * row_tiles; }
};
static bool box_wanted(const H2Gemm &g) { return g.conv && conv_h2_small(g.img_n, g.img_h, g.img_w, g.img_c); }
static bool box_plan(const H2Gemm &g, BoxPlan *plan) {
    if (g.out_w > BM || (g.out_w - 1) * g.win.stride_w + 1 > 256) return false;
    long long r = BM / g.out_w;
    if (r > g.out_h) r = g.out_h;
    const long long in_reach = 255 / g.win.stride_h + 1;  // the box spans (r - 1) * stride + 1 <= 256 image rows
    if (r > in_reach) r = in_reach;
    long long imgs = r == g.out_h ? BM / (g.out_w * g.out_h) : 1;
    if (imgs > g.img_n) imgs = g.img_n;
    plan->imgs = (int)imgs;
    plan->rows = (int)r;
    plan->row_tiles = (int)((g.out_h + r - 1) / r);
    return true;
}
// ... one piece of the image, the pixels of a tile a stride apart
static bool encode_box(PFN_encodeTiled encode, const H2Gemm &g, const BoxPlan &plan, const unsigned short *base, CUtensorMap *map) {
    const cuuint64_t dims[4] = {(cuuint64_t)g.img_c, (cuuint64_t)g.img_w, (cuuint64_t)g.img_h, (cuuint64_t)g.img_n};
    const cuuint64_t strides[3] = {(cuuint64_t)g.img_c * 2, (cuuint64_t)(g.img_w * g.img_c) * 2, (cuuint64_t)(g.img_h * g.img_w * g.img_c) * 2};
    const Window &w = g.win;
    const cuuint32_t box[4] = {(cuuint32_t)HK, (cuuint32_t)((g.out_w - 1) * w.stride_w + 1), (cuuint32_t)((plan.rows - 1) * w.stride_h + 1), (cuuint32_t)plan.imgs};
    const cuuint32_t estr[4] = {1, (cuuint32_t)w.stride_w, (cuuint32_t)w.stride_h, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<unsigned short *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The limits of im2col-mode tensor maps (as for the tf32 kernel), channels in whole groups.
bool conv_h2_ok(const H2Gemm &g) {
    const Window &w = g.win;
    if (g.img_c < 64 || g.img_c % 64 || g.img_n < 1 || g.img_h < 1 || g.img_w < 1 || g.out_h < 1 || g.out_w < 1 || g.out_h * g.out_w > 0x7fffffffLL) return false;
    if (w.stride_w < 1 || w.stride_w > 8 || w.stride_h < 1 || w.stride_h > 8) return false;
    if (w.pad_w < 0 || w.pad_w > 127 || w.pad_h < 0 || w.pad_h > 127 || w.dil_w < 0 || w.dil_h < 0) return false;
    if (w.pad_w - (w.ker_w - 1) * w.dil_w < -128 || w.pad_h - (w.ker_h - 1) * w.dil_h < -128) return false;
    BoxPlan plan;
    if (box_wanted(g) && !box_plan(g, &plan)) return false;
    return (w.ker_w - 1) * w.dil_w <= 255 && (w.ker_h - 1) * w.dil_h <= 255 && g.img_n * g.img_h * g.img_w <= 0x7fffffffLL;
}

// Tap reuse: the rule of conv_halo_plan in gemm_tcgen05.cu (SAGE_CONV_HALO=0 turns it off, read per launch).
static bool halo_plan(const H2Gemm &g, int *wb, int *rows) {
    const char *env = getenv("SAGE_CONV_HALO");
    const Window &w = g.win;
    if ((env && atoi(env) == 0) || !g.conv || box_wanted(g) || w.stride_w != 1 || w.stride_h != 1 || w.dil_w != 1 || w.dil_h != 1) return false;
    if (w.ker_w * w.ker_h < 2 || g.n > 128 || g.n % 32) return false;
    const long long b = g.out_w + w.ker_w - 1;
    if (b > 128) return false;
    long long r = 128 / b;
    if (r > g.out_h) r = g.out_h;
    if (r * g.out_w < 100 || b * (r + w.ker_h - 1) > 256 || 127 + (w.ker_h - 1) * b + (w.ker_w - 1) > 255) return false;
    if (g.img_n * ((g.out_h + r - 1) / r) > 0x3fffffffLL) return false;
    *wb = (int)b;
    *rows = (int)r;
    return true;
}

static bool pairs_on() {
    static const bool on = !(getenv("SAGE_GEMM_PAIR") && atoi(getenv("SAGE_GEMM_PAIR")) == 0);
    return on;
}

// How the columns are cut: tiles of `bn` columns, the last `narrow` of a row block 192 wide instead (only with bn = 256;
// wide = 0: all of them).  The busiest CTA (pair) decides: a tile costs its width plus a fixed 24 columns' worth.
struct ColumnPlan {
    int bn, wide, narrow;
};
static ColumnPlan plan_columns(const Context &ctx, long long m, long long n, long long batch, int ctas) {
    const long long slots = ctx.sm_count / ctas, row_tiles = (m + BM * ctas - 1) / (BM * ctas) * batch;
    ColumnPlan best{128, 0, 0};
    double best_cost = 1e300;
    auto consider = [&](int bn, long long wide, long long narrow) {
        const long long tw = row_tiles * wide, total = tw + row_tiles * narrow;
        if (total > 0x7fffffffLL) return;
        double worst = 0;
        for (long long i = 0; i < slots && i < total; ++i) {  // pair i gets tiles i, i + slots, ..., the wide ones first
            const long long mine = (total - i + slots - 1) / slots, mine_wide = i < tw ? (tw - i + slots - 1) / slots : 0;
            const double load = (double)mine_wide * (bn + 24) + (double)(mine - mine_wide) * (192 + 24);
            if (load > worst) worst = load;
        }
        if (worst < best_cost * (narrow ? 0.98 : 1.0)) {
            best_cost = worst;
            best = ColumnPlan{bn, (int)wide, (int)narrow};
        }
    };
    for (int bn : {256, 128, 64})
        if (bn == 64 || n > bn / 2) consider(bn, (n + bn - 1) / bn, 0);
    for (long long nn = 1; nn * 192 <= n + 191 && n > 128; ++nn) {
        const long long rest = n - nn * 192, nw = rest > 0 ? (rest + 255) / 256 : 0;
        if (nw * 256 + nn * 192 - n < 192) consider(256, nw, nn);
    }
    return best;
}

// op(A) op(B) of plain fp32 operands: both brought into pieces, K contiguous.  `scratch`: where the pieces go (of
// gemm_h2_scratch_bytes), or null to take them from the allocator.
static SplitView operand_view(const float *, long long rows, long long cols, bool k_contiguous, long long ld, long long batch_stride, long long batch) {
    SplitView v;
    v.nb0 = batch;
    v.sb0 = batch_stride;
    v.rows = rows;
    v.cols = cols;
    v.ld = k_contiguous ? ld : 1;
    v.col_stride = k_contiguous ? 1 : ld;
    return v;
}
size_t gemm_h2_scratch_bytes(const GemmArgs &g) { return split_h2_bytes(g.batch, g.m, g.k, false) + split_h2_bytes(g.batch, g.n, g.k, true); }

sage_status gemm_h2(Context &ctx, const GemmArgs &a, void *scratch) {
    const SplitView va = operand_view(a.a, a.m, a.k, !a.ta, a.lda, a.stride_a, a.batch), vb = operand_view(a.b, a.n, a.k, a.tb, a.ldb, a.stride_b, a.batch);
    Block *block = nullptr;
    if (!scratch) {
        block = ctx.allocator().alloc(gemm_h2_scratch_bytes(a));
        if (!block) return ctx.fail(SAGE_ERR_OOM, "out of memory for the operands in half-precision pieces");
        scratch = block->ptr;
    }
    const H2Split pa = split_layout(va, scratch), pb = split_layout(vb, static_cast<char *>(scratch) + split_h2_bytes(a.batch, a.m, a.k, false));
    sage_status st = split_views(ctx, a.a, &va, pa, a.b, &vb, pb);
    if (!st) {
        H2Gemm g;
        g.m = a.m;
        g.n = a.n;
        g.k = a.k;
        g.batch = a.batch;
        g.a = h2_operand(pa, a.batch, a.m, a.k, false);
        g.b = h2_operand(pb, a.batch, a.n, a.k, true);
        g.c = a.c;
        g.ldc = a.ldc;
        g.sc0 = a.stride_c;
        g.nbc0 = a.batch;
        st = gemm_h2_run(ctx, g);
    }
    if (block) ctx.allocator().free(block);  // stream-ordered: later launches on this stream may reuse it
    return st;
}

// The plain product (no epilogue, fp32 result): compiled with the library, so that an entry point which must not load a
// module at run time can use it.
template <int BN, int CTAS, bool SLICED>
__global__ void __launch_bounds__(SLICED ? 64 + 2 * BN : kThreads, SLICED && BN == 64 ? 2 : 1) gemm_h2_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                                                              const __grid_constant__ CUtensorMap map_b2, const __grid_constant__ H2Params p) {
    gemm_h2_body<BN, CTAS, SLICED>(&map_a, &map_a, &map_b, &map_b2, p);
}
// The dynamic shared memory a kernel may be launched with is a setting of the kernel on a device, shared by all threads: raised once,
// to all there is, never to what one launch needs (a shorter ring asks for less, and could lower it under another thread's launch).
template <int BN, int CTAS, bool SLICED>
static cudaError_t allow_shared_memory(int dev) {
    auto raise = [] {
        cudaFuncAttributes a;
        const cudaError_t e = cudaFuncGetAttributes(&a, gemm_h2_kernel<BN, CTAS, SLICED>);
        return e != cudaSuccess ? e : cudaFuncSetAttribute(gemm_h2_kernel<BN, CTAS, SLICED>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - (int)a.sharedSizeBytes);
    };
    static std::once_flag once[64];
    static cudaError_t result[64];
    if (dev < 0 || dev >= 64) return raise();
    std::call_once(once[dev], [&] { result[dev] = raise(); });
    return result[dev];
}
template <int BN, int CTAS, bool SLICED>
static sage_status launch_plain(Context &ctx, const CUtensorMap &map_a, const CUtensorMap &map_b, const CUtensorMap &map_b2, const H2Params &p, int grid, size_t smem) {
    const sage_status st = ctx.check_cuda(allow_shared_memory<BN, CTAS, SLICED>(ctx.device()), "gemm_h2 shared memory attribute");
    if (st) return st;
    return ctx.check_cuda(launch_dependent(ctx.pdl, ctx.stream(), SLICED ? p.slices : CTAS, gemm_h2_kernel<BN, CTAS, SLICED>, dim3(grid), dim3(SLICED ? 64 + 2 * BN : kThreads), smem, map_a, map_b, map_b2, p), "gemm_h2 launch");
}

// How many clusters of `s` CTAs the chip holds at once: they do not cross a GPC, so fewer than SMs / s.
static int clusters_at_once(const Context &ctx, int s) {
    static std::atomic<int> known[64][9];
    const int dev = ctx.device();
    if (ctx.dry() || dev < 0 || dev >= 64) return ctx.sm_count / s * 9 / 10;
    int n = known[dev][s].load(std::memory_order_relaxed);
    if (n > 0) return n;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)s;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(s * 256));
    cfg.blockDim = dim3(64 + 2 * 128);
    cfg.dynamicSmemBytes = 200 * 1024;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (allow_shared_memory<128, 1, true>(dev) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, gemm_h2_kernel<128, 1, true>, &cfg) != cudaSuccess || n < 1) {
        (void)cudaGetLastError();
        n = ctx.sm_count / s * 9 / 10;
    }
    known[dev][s].store(n, std::memory_order_relaxed);
    return n;
}

// Slices of K (gemm_h2_body's SLICED), or 0, and the width of their tiles.  Microseconds, from launches of one wave timed on
// M 24 .. 3136, N 64 .. 3072, K 512 .. 4608: a K-block takes 0.52 / 0.67 / 0.92 with 64 / 128 / 256 columns (a pair of CTAs
// 0.42 / 0.48 / 0.91, windows kept in shared memory 0.48), and not less than the bytes of all CTAs at 9 TB/s; a tile 3.5 beside
// them, and 5 for operands that depend on the row, which slices fetch in time.  Meeting in shared memory: 1.5 and 1.1 per 128 x
// 64 sums (256 columns: 9, never worth it), timed when the sums were fetched after a barrier; sent, they take up to 2 us less
// (eight slices) or as much (two to four), and the line is left on the safe side.  Slices must promise a fifth: they change the order of summation, and nearer to the
// line than that the estimate says little.
struct SlicePlan {
    int slices, bn;
};
static SlicePlan plan_slices(const Context &ctx, const H2Gemm &g) {
    static const bool enabled = !(getenv("SAGE_GEMM_SPLITK") && atoi(getenv("SAGE_GEMM_SPLITK")) == 0);
    const SlicePlan none{0, 0};
    const long long all_kb = (g.k + HK - 1) / HK;
    if (!enabled || all_kb < 4) return none;
    BoxPlan box{};
    int wb = 0, halo_rows = 0;
    const bool halo = halo_plan(g, &wb, &halo_rows), boxed = box_wanted(g) && box_plan(g, &box);
    const int ctas = (pairs_on() && g.m > BM && !boxed) ? 2 : 1;
    double best = 1e300, whole = 1e300, store = 3.5;
    for (int i = 0; i < g.naux; ++i)
        if (g.aux[i].sr != 0) store = 8.5;
    SlicePlan plan = none;
    if (halo) {
        const long long tiles = (g.img_n * ((g.out_h + halo_rows - 1) / halo_rows) + ctas - 1) / ctas, slots = ctx.sm_count / ctas;
        whole = (double)((tiles + slots - 1) / slots) * ((double)all_kb * 0.48 + store + 3.0);
    }
    for (int w = 0; w < 3; ++w) {
        static const double alone[3] = {0.52, 0.67, 0.92}, paired[3] = {0.42, 0.48, 0.91};
        const int bn = 64 << w;
        if (w > 0 && g.n <= bn / 2) continue;
        const long long cols = (g.n + bn - 1) / bn * g.batch;
        auto block_us = [&](double us, long long busy, int pair) {
            const double bytes = (double)busy * (BM + bn / pair) * HK * 4 / 9e6;
            return us > bytes ? us : bytes;
        };
        if (!halo) {
            const long long tiles = (boxed ? box.tiles(g) : (g.m + BM * ctas - 1) / (BM * ctas)) * cols, slots = ctx.sm_count / ctas, busy = tiles < slots ? tiles : slots;
            const double t = (double)((tiles + slots - 1) / slots) * ((double)all_kb * block_us(ctas == 2 ? paired[w] : alone[w], busy * ctas, ctas) + store);
            if (t < whole) whole = t;
        }
        const long long tiles = (boxed ? box.tiles(g) : (g.m + BM - 1) / BM) * cols;
        for (int s = 2; s <= 8 && bn < 256; ++s) {
            const long long kb = (all_kb + s - 1) / s;
            if (kb < 2 || kb * (s - 1) >= all_kb || tiles > clusters_at_once(ctx, s)) continue;
            const double filled = g.m < BM ? (double)g.m / BM : 1.0;
            const double t = (double)kb * block_us(alone[w], tiles * s, 1) + 5.0 + filled * 1.1 * (1 << w);
            if (t < best) {
                best = t;
                plan = SlicePlan{s, bn};
            }
        }
    }
    return best <= 0.8 * whole ? plan : none;
}

// Does the expression call a function of more than a few instructions?
bool long_expression(const std::string &e) {
    static const char *const kShort[] = {"lit", "abs", "square", "sign", "min", "max", "ceil", "floor", "round", "recip"};
    for (size_t at = e.find("sg_"); at != std::string::npos; at = e.find("sg_", at + 3)) {
        bool is_short = false;
        for (const char *name : kShort) is_short = is_short || e.compare(at + 3, strlen(name), name) == 0;
        if (!is_short) return true;
    }
    return false;
}

sage_status gemm_h2_run(Context &ctx, const H2Gemm &g) {
    const PFN_encodeTiled encode = ctx.dry() ? nullptr : encode_tiled();
    const PFN_encodeIm2col encode_conv = ctx.dry() ? nullptr : encode_im2col_mode();
    if (!ctx.dry() && (!encode || !encode_conv)) return ctx.fail(SAGE_ERR_DEVICE, "cuTensorMapEncode is not available");
    if (g.m < 1 || g.n < 1 || g.k < 1 || g.batch < 1 || g.m > 0x7fffffffLL || g.n > 0x7fffffffLL || g.k > 0x7fffffffLL || g.batch > 0x7fffffffLL)
        return ctx.fail(SAGE_ERR_UNSUPPORTED, "gemm_h2: shape not supported");
    if (g.naux < 0 || g.naux > kMaxAux || (!g.c && !g.c_hi && !g.h_hi)) return ctx.fail(SAGE_ERR_INVALID, "gemm_h2: bad epilogue description");
    if (!g.b.ratio || g.b.rows != g.n) return ctx.fail(SAGE_ERR_INVALID, "gemm_h2: operand B is incomplete");
    if (g.conv && (g.batch != 1 || !conv_h2_ok(g) || g.m != g.img_n * g.out_h * g.out_w || g.k != (long long)g.win.ker_h * g.win.ker_w * g.img_c))
        return ctx.fail(SAGE_ERR_INVALID, "gemm_h2: convolution description does not match the GEMM");
    const SlicePlan cut = plan_slices(ctx, g);
    const bool sliced = cut.slices > 1;
    int halo_wb = 0, halo_r = 0;
    const bool halo = !sliced && halo_plan(g, &halo_wb, &halo_r);
    BoxPlan box{};
    const bool boxed = box_wanted(g) && box_plan(g, &box);
    const int ctas = (pairs_on() && g.m > BM && !sliced && !boxed) ? 2 : 1;
    ColumnPlan cols = sliced ? ColumnPlan{cut.bn, 0, 0} : plan_columns(ctx, boxed ? box.tiles(g) * BM : g.m, g.n, g.batch, ctas);
    if (halo) cols = ColumnPlan{g.n <= 64 ? 64 : 128, 0, 0};  // all output channels in one tile: the window is loaded once
    const int bn = cols.bn;
    const int stage_bytes = halo ? 2 * (bn / ctas) * HK * 2 : 2 * BM * HK * 2 + 2 * (bn / ctas) * HK * 2;
    const long long octets = std::min<long long>(BM / 8, (g.m + 7) / 8);  // of a tile: H2Tasks
    const int region = sliced ? (int)((octets * (bn / 64) + cut.slices - 1) / cut.slices) * cut.slices * 2048 : kEpiWarps * kStageBytesPerWarp;
    const int fixed = halo ? kHaloStages * kHaloStageBytes : 0;
    const long long all_kb = (g.k + HK - 1) / HK, my_kb = sliced ? (all_kb + cut.slices - 1) / cut.slices : all_kb;
    const auto fitting = [&](int beside) { return (int)std::min<long long>((227 * 1024 - 2048 - beside - fixed) / stage_bytes, sliced && my_kb < 8 ? my_kb : 8); };
    // Where a sliced tile's sums meet (H2Tasks).  Beside the operands: sent as each CTA is done with its own.  Over them, once the cluster's
    // products are done, where that keeps a stage of the ring (3 of 128 columns, else 2) and a CTA has K-blocks enough to need
    // it.  Left where they are and fetched, with two slices, or with four and nothing else to load in the store.  us a product
    // in chains of equal 3 x 3 convolutions (channels, pixels, slices; + residual), fetched | beside | over; what is chosen in
    // brackets:  512, 16 x 7 x 7, 4: [21.55] | 22.27 | 21.67, + 22.71 | 22.77 | [22.25];  512, 24 x 7 x 7, 3 +: 27.49 | 27.41 | [26.60];
    // 256, 16 x 14 x 14, 2 +: [22.61] | 23.50 | 22.94;  256, 8 x 14 x 14, 4: [15.47] | 15.77 | 15.71, + 16.63 | 16.30 | [16.28];
    // 128, 8 x 28 x 28, 2 +: [16.62] | 17.01 | 16.97;  128, 6 x 28 x 28, 3: 14.32 | [13.88];  128, 28 x 28, 6: 9.60 | [8.42].
    // Plain products of the same sizes, whose operands come faster, and 64 columns lose by the wait: beside.
    bool row_operands = false;
    for (int i = 0; i < g.naux; ++i) row_operands = row_operands || g.aux[i].sr != 0;
    const bool fetch = sliced && g.conv && bn == 128 && (cut.slices == 2 || (cut.slices == 4 && !row_operands));
    const bool over = fetch || (sliced && g.conv && bn == 128 && my_kb >= 9 && fitting(0) > fitting(region));
    const int staging = over ? 0 : region, stages = fitting(staging);
    const size_t smem = (size_t)fixed + (size_t)stages * stage_bytes + staging + 1024;

    H2Params p{};
    p.sums_at = over ? 0 : stages * stage_bytes;
    p.c = g.c;
    p.c_hi = g.c_hi;
    p.c_plane = g.c_plane;
    p.h_hi = g.h_hi;
    p.h_plane = g.h_plane;
    p.h_scale = g.h_scale;
    p.h_marked = g.h_marked;
    p.ldc = g.ldc;
    p.sc0 = g.sc0;
    p.sc1 = g.sc1;
    p.nbc0 = (int)(g.nbc0 < 1 ? 1 : g.nbc0);
    p.na0 = (int)g.a.nb0;
    p.nb0 = (int)g.b.nb0;
    p.slices = sliced ? cut.slices : 0;
    p.kb_count = (int)my_kb;
    p.a_bcast = (g.a.bcast || g.conv) ? 1 : 0;
    p.b_bcast = g.b.bcast ? 1 : 0;
    p.m = (int)g.m;
    p.n = (int)g.n;
    p.k = (int)g.k;
    p.stages = stages;
    p.tiles_m = (int)((g.m + BM * ctas - 1) / (BM * ctas));
    p.tiles_n = (cols.wide || cols.narrow) ? cols.wide + cols.narrow : (int)((g.n + bn - 1) / bn);
    p.rag_wide = cols.wide;
    p.rag_narrow = cols.narrow;
    p.rag_bn = 192;
    p.num_tiles = (int)((long long)p.tiles_m * p.tiles_n * g.batch);
    p.sa = g.a.scale;
    p.sa_row = g.a.s_row;
    p.sa_b0 = g.a.s_b0;
    p.sa_b1 = g.a.s_b1;
    p.sb = g.b.scale;
    p.sb_batch = p.b_bcast ? 0 : g.b.s_b0;
    p.sb_ratio = g.b.ratio;
    p.status = ctx.status_word_dev;
    if (g.conv) {
        p.conv_cb = (int)(g.img_c / HK);
        p.conv_kw = g.win.ker_w;
        p.conv_q = (int)g.out_w;
        p.conv_pq = (int)(g.out_h * g.out_w);
        p.conv_sw = g.win.stride_w;
        p.conv_sh = g.win.stride_h;
        p.conv_pw = g.win.pad_w;
        p.conv_ph = g.win.pad_h;
        p.conv_dw = g.win.dil_w;
        p.conv_dh = g.win.dil_h;
        p.conv_h = (int)g.img_h;
        p.conv_w = (int)g.img_w;
        p.conv_n = (int)g.img_n;
        p.conv_p = (int)g.out_h;
    }
    if (halo) {
        p.halo_wb = halo_wb;
        p.halo_r = halo_r;
        p.halo_rt = (int)((g.out_h + halo_r - 1) / halo_r);
        p.halo_taps = g.win.ker_h * g.win.ker_w;
        p.halo_box_bytes = 128 * halo_wb * (halo_r + g.win.ker_h - 1);
        p.tiles_m = (int)((g.img_n * p.halo_rt + ctas - 1) / ctas);
        p.num_tiles = p.tiles_m * p.tiles_n;
    }
    if (boxed) {
        if (!g.a.marked || !g.b.marked || !g.b.columns || !g.a_f32 || !g.b_f32) return ctx.fail(SAGE_ERR_INVALID, "gemm_h2: a small convolution without its wide groups");
        p.box_imgs = box.imgs;
        p.box_r = box.rows;
        p.box_rt = box.row_tiles;
        p.box_bytes = (int)(box.imgs * box.rows * g.out_w) * HK * 2;
        p.tiles_m = (int)box.tiles(g);
        p.sa = g.a.marked;
        p.sb_ratio = g.b.marked;
        p.b_columns = g.b.columns;
        p.a_f32 = g.a_f32;
        p.b_f32 = g.b_f32;
        p.b_k = g.b_k;
        p.b_n = g.b_n;
        p.num_tiles = p.tiles_m * p.tiles_n;
    }
    const bool vec = g.n % 4 == 0 && g.ldc % 4 == 0 && g.sc0 % 4 == 0 && g.sc1 % 4 == 0 && (!g.c || aligned16(g.c)) && (!g.c_hi || (aligned16(g.c_hi) && g.c_plane % 4 == 0));
    bool aux_vec = true;
    int rowinv = 0, per_col = 0;
    for (int i = 0; i < g.naux; ++i) {
        TcAux &a = p.aux[i];
        a.ptr = g.aux[i].ptr;
        a.s0 = g.aux[i].s0;
        a.s1 = g.aux[i].s1;
        a.sr = g.aux[i].sr;
        a.sc = g.aux[i].sc;
        if (a.sc != 0 && a.sc != 1) return ctx.fail(SAGE_ERR_INVALID, "gemm_h2: epilogue operand column stride must be 0 or 1");
        if (a.sc == 1) aux_vec = aux_vec && aligned16(a.ptr) && a.s0 % 4 == 0 && a.s1 % 4 == 0 && a.sr % 4 == 0;
        if (a.sr == 0) rowinv |= 1 << i;
        if (a.sc != 0) per_col |= 1 << i;
    }
    p.vec_ok = vec ? 1 : 0;
    if (g.h_hi && (!vec || g.n % 64 || g.ldc % 64 || g.sc0 % 64 || g.sc1 % 64 || !aligned16(g.h_hi) || g.h_plane % 8))
        return ctx.fail(SAGE_ERR_INVALID, "gemm_h2: a result in half-precision pieces needs whole groups of 64 columns");
    const int slots = ctx.sm_count / ctas, grid = sliced ? cut.slices * p.num_tiles : ctas * (p.num_tiles < slots ? p.num_tiles : slots);
    const int threads = sliced ? 64 + 2 * bn : kThreads;

    const int out_mask = (g.c ? 1 : 0) | (g.c_hi ? 2 : 0) | (g.h_hi ? 4 : 0) | (g.h_hi && g.h_marked ? 8 : 0);
    // A residual through shared memory, where the ring behind a CTA's only tile takes it.  us, fetched by the store | this: BERT-base 32 x 128
    // 2790 | 2741, 12 x 128 1414 | 1342, 8 x 200 1783 | 1700, of width 512 16 x 128 (6 layers) 610 | 578, 256 40 x 100 1016 | 930, 1024
    // 20 x 128 (8) 2013 | 1965.  (With the store in a loop, as below, 32 x 128 2849.)
    int res = 0;
    if (!sliced && !g.conv && g.batch == 1 && p.num_tiles <= slots && vec && aux_vec)
        for (int i = g.naux; i-- > 0;)
            if (g.aux[i].sr > 0 && g.aux[i].sc == 1 && g.aux[i].sr < (1LL << 36)) res = i + 1;
    // A store that is worked through once is bound by the fetching of its instructions: its four sub-tiles in a loop, where no operand's
    // rows have to be on their way meanwhile (a residual: 32 x 128 tokens of BERT-base 2850 -> 3117 us).  The same for an expression so
    // long that a tile's four copies of it are slower to fetch than to repeat.  us, unrolled | as chosen: GELU on 6 x 77 tokens 986 | 948,
    // 2 x 64 816 | 768, 12 x 128 1617 | 1502, 32 x 128 3018 | 2968 (only single tiles: 3022); without it 6 x 77 894 | 884, 2 x 64 705 |
    // 700, 12 x 128 1411 | 1406, 16 x 128 of width 512 595 | 599.  Several tiles and a short expression: 32 x 128 2762 | 2786 if rolled.
    const bool roll = !sliced && rowinv == (1 << g.naux) - 1 && (p.num_tiles <= slots || long_expression(g.epilogue));
    char num[96];
    snprintf(num, sizeof num, "gemm_h2 %d %d %d %d %d %d %d %d %d %d %d\n", res, roll ? 1 : 0, bn, ctas, sliced ? 1 : 0, aux_vec ? 1 : 0, (g.conv ? (halo ? 2 : boxed ? 3 : 1) : 0) + (fetch ? 4 : 0), g.naux, rowinv, per_col, out_mask);
    const bool plain = !g.conv && g.naux == 0 && g.epilogue.empty() && out_mask == 1;
    const std::string key = num + g.epilogue;
    Module *mod = plain ? nullptr : ctx.module_find(key);
    if (!plain && !mod) {
        std::string src = map_prelude_text();
        src += "struct __align__(64) CUtensorMap { unsigned long long opaque[16]; };\n";
        auto define = [&](const char *name, int v) { src += std::string("#define ") + name + " " + std::to_string(v) + "\n"; };
        define("SAGE_EPI_ROWINV", rowinv);
        define("SAGE_EPI_COLS", per_col);
        define("SAGE_EPI_OUT", out_mask);
        define("SAGE_EPI_NAUX", g.naux);
        define("SAGE_H2_CONV", g.conv ? (boxed ? 2 : 1) : 0);
        define("SAGE_H2_AUX_VEC", aux_vec ? 1 : 0);
        define("SAGE_H2_HALO", halo ? 1 : 0);
        define("SAGE_H2_FETCH", fetch ? 1 : 0);
        define("SAGE_H2_ROLL", roll ? 1 : 0);
        define("SAGE_H2_RES", res);
        src += "#define SAGE_EPI_EXPR(x0, x1, x2, x3) (" + (g.epilogue.empty() ? std::string("x0") : g.epilogue) + ")\n";
        src += kGemmTcDeviceSrc;
        src += kGemmH2DeviceSrc;
        src += "\nextern \"C\" __global__ void __launch_bounds__(" + std::to_string(threads) + (sliced && bn == 64 ? ", 2)\n" : ", 1)\n") +
               "gemm_tc_h2(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_a2,\n"
               "           const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_b2, const __grid_constant__ sage_tc::H2Params p) {\n"
               "    sage_tc::gemm_h2_body<" + std::to_string(bn) + ", " + std::to_string(ctas) + (sliced ? ", true" : ", false") + ">(&map_a, &map_a2, &map_b, &map_b2, p);\n}\n";
        sage_status st = ctx.module_get(src, &mod);
        if (st) return st;
        ctx.module_remember(key, mod);
    }
    CUtensorMap map_a, map_a2, map_b, map_b2;
    if (!ctx.dry()) {
        auto ok = [](const H2Operand &o) {
            return o.hi && aligned16(o.hi) && o.ld % 8 == 0 && o.ld > 0 && o.plane % 8 == 0 && o.plane > 0 && (o.nb0 == 1 || (o.sb0 % 8 == 0 && o.sb0 > 0)) &&
                   (o.nb1 == 1 || (o.sb1 % 8 == 0 && o.sb1 > 0));
        };
        bool good = ok(g.b) && encode_operand(encode, g.b, g.k, (unsigned)(bn / ctas), &map_b);
        map_b2 = map_b;
        if (cols.narrow) good = good && encode_operand(encode, g.b, g.k, (unsigned)(p.rag_bn / ctas), &map_b2);
        if (!g.conv) {
            good = good && ok(g.a) && encode_operand(encode, g.a, g.k, BM, &map_a);
            map_a2 = map_a;
            if (res) good = good && encode_residual(encode, g.aux[res - 1], g.m, g.n, &map_a2);
        } else {
            good = good && aligned16(g.a.hi) && g.a.plane % 8 == 0;
            if (halo)
                good = good && encode_halo(encode, g, g.a.hi, (unsigned)halo_wb, (unsigned)(halo_r + g.win.ker_h - 1), &map_a) &&
                       encode_halo(encode, g, g.a.hi + g.a.plane, (unsigned)halo_wb, (unsigned)(halo_r + g.win.ker_h - 1), &map_a2);
            else if (boxed)
                good = good && encode_box(encode, g, box, g.a.hi, &map_a) && encode_box(encode, g, box, g.a.hi + g.a.plane, &map_a2);
            else
                good = good && encode_im2col(encode_conv, g, g.a.hi, &map_a) && encode_im2col(encode_conv, g, g.a.hi + g.a.plane, &map_a2);
        }
        if (!good) return ctx.fail(SAGE_ERR_INVALID, "gemm_h2: an operand is not addressable by TMA");
    }
    std::string label;
    if (ctx.verbose_names)
        label = "gemm_tc_h2[" + std::to_string(g.m) + "x" + std::to_string(g.n) + "x" + std::to_string(g.k) + (g.batch > 1 ? "x" + std::to_string(g.batch) : "") + (sliced ? (fetch ? ",fetched" : over ? ",over" : "") + std::string(",slices") + std::to_string(cut.slices) : "") +
                (g.conv ? (halo ? ",conv,taps" : boxed ? ",conv,boxes" : ",conv") : "") + ",bn" + std::to_string(bn) + (cols.narrow ? "/" + std::to_string(cols.wide) + "+" + std::to_string(cols.narrow) + "x192" : "") +
                (ctas == 2 ? ",pair" : "") + (roll && !plain ? ",rolled" : "") + (res ? ",residual" + std::to_string(res - 1) : "") + "]o" + std::to_string(out_mask);
    if (plain) {
        ctx.note_launch(ctx.verbose_names ? label.c_str() : "gemm_tc_3xtf32");
        if (ctx.dry()) return SAGE_OK;
        if (sliced) return bn == 128 ? launch_plain<128, 1, true>(ctx, map_a, map_b, map_b2, p, grid, smem) : launch_plain<64, 1, true>(ctx, map_a, map_b, map_b2, p, grid, smem);
        if (ctas == 2)
            return bn == 256 ? launch_plain<256, 2, false>(ctx, map_a, map_b, map_b2, p, grid, smem)
                   : bn == 128 ? launch_plain<128, 2, false>(ctx, map_a, map_b, map_b2, p, grid, smem) : launch_plain<64, 2, false>(ctx, map_a, map_b, map_b2, p, grid, smem);
        return bn == 256 ? launch_plain<256, 1, false>(ctx, map_a, map_b, map_b2, p, grid, smem)
               : bn == 128 ? launch_plain<128, 1, false>(ctx, map_a, map_b, map_b2, p, grid, smem) : launch_plain<64, 1, false>(ctx, map_a, map_b, map_b2, p, grid, smem);
    }
    const uint32_t gr[3] = {(uint32_t)grid, 1, 1}, bl[3] = {(uint32_t)threads, 1, 1};
    void *params[5] = {&map_a, &map_a2, &map_b, &map_b2, &p};
    // launch lists have one name for a tensor-core product; verbose ones tell the kernels apart
    return ctx.launch(mod, "gemm_tc_h2", gr, bl, (uint32_t)smem, params, ctx.verbose_names ? label.c_str() : "gemm_tc_3xtf32", true, sliced ? cut.slices : ctas);
}

// ---------------------------------------------------------------------------------- the first convolution
// Columns two apart (the descriptor's row pitch), the filter and two stages of rows beside the store's staging, and at least six
// tenths of the 128 pixels of a tile inside the row: below that the gathered operand's full tiles are the better ones.
bool conv_first_ok(int kh, int stride_w, long long out_w) { return stride_w == 2 && kh >= 1 && kh <= 11 && out_w * 10 >= (out_w + 127) / 128 * 128 * 6; }

sage_status conv_first_run(Context &ctx, const H2Gemm &g, const FirstConv &f) {
    if (!conv_first_ok(f.kh, 2, g.out_w) || g.n < 1 || f.wp % 2 || f.img_plane % 8 || !f.img_f32 || !f.filter_f32 || g.naux < 0 || g.naux > kMaxAux || (!g.c && !g.c_hi && !g.h_hi) ||
        g.img_n * g.out_h * ((g.out_w + 127) / 128) > 0x3fffffffLL || g.img_n * g.out_h * g.out_w > 0x7fffffffLL)
        return ctx.fail(SAGE_ERR_INVALID, "conv_first: bad description");
    FirstParams p{};
    p.h.c = g.c;
    p.h.c_hi = g.c_hi;
    p.h.c_plane = g.c_plane;
    p.h.h_hi = g.h_hi;
    p.h.h_plane = g.h_plane;
    p.h.h_scale = g.h_scale;
    p.h.ldc = g.ldc;
    p.h.nbc0 = 1;
    p.h.n = (int)g.n;
    p.h.sa = f.img_scale;
    p.h.sb = f.filter_scale;
    p.h.status = ctx.status_word_dev;
    p.img = f.img;
    p.img_plane = f.img_plane;
    p.filter = f.filter;
    p.hp = (int)f.hp;
    p.wp = (int)f.wp;
    p.kh = f.kh;
    p.dil_h = f.dil_h;
    p.stride_h = f.stride_h;
    p.img_f32 = f.img_f32;
    p.filter_f32 = f.filter_f32;
    p.img_h = (int)f.img_h;
    p.img_w = (int)f.img_w;
    p.chan = f.chan;
    p.kw = f.kw;
    p.pad_h = f.pad_h;
    p.pad_w = f.pad_w;
    p.out_h = (int)g.out_h;
    p.out_w = (int)g.out_w;
    p.segs = (int)((g.out_w + 127) / 128);
    p.tiles_n = (int)((g.n + 63) / 64);
    p.num_tiles = (int)(g.img_n * g.out_h * p.segs);
    const bool vec = g.n % 4 == 0 && g.ldc % 4 == 0 && (!g.c || aligned16(g.c)) && (!g.c_hi || (aligned16(g.c_hi) && g.c_plane % 4 == 0));
    bool aux_vec = true;
    int rowinv = 0, per_col = 0;
    for (int i = 0; i < g.naux; ++i) {
        TcAux &a = p.h.aux[i];
        a.ptr = g.aux[i].ptr;
        a.s0 = a.s1 = 0;
        a.sr = g.aux[i].sr;
        a.sc = g.aux[i].sc;
        if (a.sc != 0 && a.sc != 1) return ctx.fail(SAGE_ERR_INVALID, "conv_first: epilogue operand column stride must be 0 or 1");
        if (a.sc == 1) aux_vec = aux_vec && aligned16(a.ptr) && a.sr % 4 == 0;
        if (a.sr == 0) rowinv |= 1 << i;
        if (a.sc != 0) per_col |= 1 << i;
    }
    p.h.vec_ok = vec ? 1 : 0;
    if (g.h_hi && (!vec || g.n % 64 || g.ldc % 64 || !aligned16(g.h_hi) || g.h_plane % 8)) return ctx.fail(SAGE_ERR_INVALID, "conv_first: a result in half-precision pieces needs whole groups of 64 columns");
    const int staging = kEpiWarps * kStageBytesPerWarp, stage_bytes = f.kh * 2 * kFirstRowBytes, filter_bytes = f.kh * 8192;
    p.stages = (227 * 1024 - 2048 - staging - filter_bytes) / stage_bytes;
    if (p.stages > 4) p.stages = 4;
    const size_t smem = (size_t)filter_bytes + (size_t)p.stages * stage_bytes + staging + 1024;
    long long ctas = ctx.sm_count / p.tiles_n;
    if (ctas < 1) ctas = 1;
    if (ctas > p.num_tiles) ctas = p.num_tiles;
    const int out_mask = (g.c ? 1 : 0) | (g.c_hi ? 2 : 0) | (g.h_hi ? 4 : 0);
    char num[96];
    snprintf(num, sizeof num, "conv_first %d %d %d %d %d\n", aux_vec ? 1 : 0, g.naux, rowinv, per_col, out_mask);
    const std::string key = num + g.epilogue;
    Module *mod = ctx.module_find(key);
    if (!mod) {
        std::string src = map_prelude_text();
        src += "struct __align__(64) CUtensorMap { unsigned long long opaque[16]; };\n";
        auto define = [&](const char *name, int v) { src += std::string("#define ") + name + " " + std::to_string(v) + "\n"; };
        define("SAGE_EPI_ROWINV", rowinv);
        define("SAGE_EPI_COLS", per_col);
        define("SAGE_EPI_OUT", out_mask);
        define("SAGE_EPI_NAUX", g.naux);
        define("SAGE_H2_AUX_VEC", aux_vec ? 1 : 0);
        src += "#define SAGE_EPI_EXPR(x0, x1, x2, x3) (" + (g.epilogue.empty() ? std::string("x0") : g.epilogue) + ")\n";
        src += kGemmTcDeviceSrc;
        src += kGemmH2DeviceSrc;
        src += kConvFirstDeviceSrc;
        src += "\nextern \"C\" __global__ void __launch_bounds__(sage_tc::kThreads, 1)\n"
               "conv_first_h2(const __grid_constant__ sage_tc::FirstParams p) {\n    sage_tc::conv_first_body(p);\n}\n";
        sage_status st = ctx.module_get(src, &mod);
        if (st) return st;
        ctx.module_remember(key, mod);
    }
    std::string label;
    if (ctx.verbose_names) label = "conv_first_h2[" + std::to_string(g.img_n * g.out_h * g.out_w) + "x" + std::to_string(g.n) + "x" + std::to_string(f.kh * 32) + "]o" + std::to_string(out_mask);
    const uint32_t gr[3] = {(uint32_t)(ctas * p.tiles_n), 1, 1}, bl[3] = {(uint32_t)kThreads, 1, 1};
    void *params[1] = {&p};
    // launch lists have one name for a tensor-core product; verbose ones tell the kernels apart
    return ctx.launch(mod, "conv_first_h2", gr, bl, (uint32_t)smem, params, ctx.verbose_names ? label.c_str() : "gemm_tc_3xtf32", true);
}

// ---------------------------------------------------------------------------------- fused attention
bool attention_tc_shape_ok(long long lq, long long lk, long long d, long long batch) {
    if (lq < 1 || lk < 1 || d < 4 || d > 64 || d % 4 || batch < 1) return false;
    if (lq > 0x7fffffffLL || lk > 0x7fffffffLL || batch > 0x7fffffffLL) return false;
    return ((lq + 127) / 128) * batch < 0x7fffffffLL;
}

sage_status attention_tc_run(Context &ctx, const TcAttn &a) {
    const PFN_encodeTiled encode = ctx.dry() ? nullptr : encode_tiled();
    if (!ctx.dry() && !encode) return ctx.fail(SAGE_ERR_DEVICE, "cuTensorMapEncodeTiled is not available");
    if (!attention_tc_shape_ok(a.lq, a.lk, a.d, a.batch)) return ctx.fail(SAGE_ERR_UNSUPPORTED, "attention_tc: shape not supported");
    if (a.naux < 0 || a.naux > kMaxAux || (!a.o && !a.out.hi && !a.out.h2)) return ctx.fail(SAGE_ERR_INVALID, "attention_tc: bad description");
    AttnParams p{};
    p.o = a.o;
    p.o_hi = a.out.hi;
    p.o_plane = a.out.plane;
    p.o_h2 = a.out.h2;
    p.o_h2_plane = a.out.h2_plane;
    p.o_h2_scale = a.out.h2_scale;
    p.ldo = a.ldo;
    p.so0 = a.so0;
    p.so1 = a.so1;
    p.nbo0 = (int)(a.nbo0 < 1 ? 1 : a.nbo0);
    p.nq0 = (int)a.q.nb0;
    p.nk0 = (int)a.k.nb0;
    p.nv0 = (int)a.v.nb0;
    p.nbe0 = (int)(a.nbe0 < 1 ? 1 : a.nbe0);
    p.sq = AttnScale{a.q.scale, a.q.s_off, a.q.s_sb0, a.q.s_sb1, a.q.s_row, a.q.s_shift};
    p.sk = AttnScale{a.k.scale, a.k.s_off, a.k.s_sb0, a.k.s_sb1, a.k.s_row, a.k.s_shift};
    p.sv = AttnScale{a.v.scale, a.v.s_off, a.v.s_sb0, a.v.s_sb1, a.v.s_row, a.v.s_shift};
    p.lq = (int)a.lq;
    p.lk = (int)a.lk;
    p.d = (int)a.d;
    p.tiles_q = (int)((a.lq + kAttnQ - 1) / kAttnQ);
    p.num_tiles = (int)((long long)p.tiles_q * a.batch);
    p.from_zero = ctx.opts().ref_compat ? 1 : 0;
    p.status = ctx.status_word_dev;
    bool aux_vec = true;
    const bool vec = a.d % 4 == 0 && a.ldo % 4 == 0 && a.so0 % 4 == 0 && a.so1 % 4 == 0 && (!a.o || aligned16(a.o)) && (!a.out.hi || (aligned16(a.out.hi) && a.out.plane % 4 == 0));
    int rowinv_mask = 0;  // which operands of the score expression have no row stride: compiled in
    for (int i = 0; i < a.naux; ++i) {
        TcAux &x = p.aux[i];
        x.ptr = a.aux[i].ptr;
        x.s0 = a.aux[i].s0;
        x.s1 = a.aux[i].s1;
        x.sr = a.aux[i].sr;
        x.sc = a.aux[i].sc;
        if (x.sc != 0 && x.sc != 1) return ctx.fail(SAGE_ERR_INVALID, "attention_tc: expression operand column stride must be 0 or 1");
        if (x.sc == 1) aux_vec = aux_vec && aligned16(x.ptr) && x.s0 % 4 == 0 && x.s1 % 4 == 0 && x.sr % 4 == 0;
        if (x.sr == 0) rowinv_mask |= 1 << i;
    }
    p.vec_ok = vec ? 1 : 0;
    p.aux_vec = aux_vec ? 1 : 0;
    if (a.out.h2 && (!vec || a.d != 64 || a.ldo % 64 || a.so0 % 64 || a.so1 % 64 || !aligned16(a.out.h2) || a.out.h2_plane % 8))
        return ctx.fail(SAGE_ERR_INVALID, "attention_tc: a result in half-precision pieces needs whole groups of 64 columns");
    // Few short sequences: attn_small_device.inc.  Up to 16 keys always; up to 32 where its blocks are few, or so many that the other
    // form's tiles, a quarter or less filled, come in rounds; up to 48 where there is hardly anything to do (36 and 24 blocks on 148 SMs).  In between its many small blocks
    // leave the next product's less room to start early.  us a layer of BERT (other form | this one; 12 heads unless said otherwise):
    // 8 tokens x 1 51.98 | 45.76, x 16 55.92 | 51.61, x 64 79.33 | 62.33; 16 x 1 60.64 | 53.92, x 4 44.38 | 43.05, x 64 92.44 | 78.04;
    // 24 x 1 44.38 | 40.79, x 4 50.22 | 49.04, x 8 (96 blocks) [55.67] | 58.69, x 32 74.76 | 70.80; 32 x 1 44.15 | 41.70, x 2 46.12 | 43.79,
    // x 4 [53.22] | 54.74, x 16 [63.72] | 66.46, x 32 (384) 82.15 | 80.91, x 64 113.76 | 102.89, 4 heads x 64 (256) [59.71] | 61.59;
    // 40 x 1 44.82 | 42.77, x 2 (48) [49.46] | 51.95; 48 x 1 45.94 | 42.75, 4 heads x 4 (32) [45.64] | 46.36; 64 x 1 [45.42] | 45.93.
    const long long small_blocks = (a.lq + kSmallQ - 1) / kSmallQ * a.batch;
    const bool few = a.lq <= kSmallQ && a.lk <= 32 ? a.lk <= 16 || small_blocks <= 36 || 2 * small_blocks >= 5 * ctx.sm_count : a.lq <= 2 * kSmallQ && a.lk <= 48 && small_blocks <= 24;
    auto operand_ok = [](const AttnOperand &o) { return o.hi && aligned16(o.hi) && o.ld % 8 == 0 && o.plane % 8 == 0 && o.sb0 % 8 == 0 && o.sb1 % 8 == 0; };
    if (few && (ctx.dry() || (operand_ok(a.q) && operand_ok(a.k) && operand_ok(a.v)))) {
        const int nk = (int)((a.lk + 31) / 32), out_mask = (a.o ? 1 : 0) | (a.out.hi ? 2 : 0) | (a.out.h2 ? 4 : 0);
        AttnSmallParams sp{};
        p.tiles_q = (int)((a.lq + kSmallQ - 1) / kSmallQ);
        sp.h = p;
        auto source = [](const AttnOperand &o) { return AttnSource{o.hi, o.plane, o.ld, o.sb0, o.sb1, (int)o.nb0}; };
        sp.q = source(a.q);
        sp.k = source(a.k);
        sp.v = source(a.v);
        char num[64];
        snprintf(num, sizeof num, "attention_small %d %d %d %d\n", nk, a.naux, rowinv_mask, out_mask);
        const std::string key = num + a.epilogue;
        Module *mod = ctx.module_find(key);
        if (!mod) {
            std::string src = map_prelude_text();
            src += "struct __align__(64) CUtensorMap { unsigned long long opaque[16]; };\n#define SAGE_ATTN_NK " + std::to_string(nk) + "\n";
            src += "#define SAGE_EPI_NAUX " + std::to_string(a.naux) + "\n#define SAGE_EPI_ROWINV " + std::to_string(rowinv_mask) + "\n#define SAGE_EPI_OUT " + std::to_string(out_mask) + "\n";
            src += "#define SAGE_EPI_EXPR(x0, x1, x2, x3) (" + (a.epilogue.empty() ? std::string("x0") : a.epilogue) + ")\n";
            src += kGemmTcDeviceSrc;
            src += kGemmH2DeviceSrc;
            src += kAttnTcDeviceSrc;
            src += kAttnSmallDeviceSrc;
            src += "\nextern \"C\" __global__ void __launch_bounds__(sage_tc::kSmallThreads)\n"
                   "attention_small(const __grid_constant__ sage_tc::AttnSmallParams p) {\n    sage_tc::attn_small_body(p);\n}\n";
            sage_status st = ctx.module_get(src, &mod);
            if (st) return st;
            ctx.module_remember(key, mod);
        }
        std::string label;
        if (ctx.verbose_names) label = "attention_tc_h2[" + std::to_string(a.lq) + "x" + std::to_string(a.lk) + "x" + std::to_string(a.d) + "x" + std::to_string(a.batch) + ",small]";
        const size_t smem = sizeof(float) * ((size_t)kSmallQ * kSmallPitch + (size_t)nk * 32 * (kSmallPitch + 64 + kSmallThreads / 32 * 4));
        const uint32_t gr[3] = {(uint32_t)small_blocks, 1, 1}, bl[3] = {(uint32_t)kSmallThreads, 1, 1};
        void *params[1] = {&sp};
        // launch lists have one name for the fused attention; verbose ones tell the kernels apart
        return ctx.launch(mod, "attention_small", gr, bl, (uint32_t)smem, params, ctx.verbose_names ? label.c_str() : "attention_tc_3xtf32", true);
    }
    // Q, the K / V ring, 1 KiB per softmax warp for turning the output round, and the slack for 1024-byte alignment
    // A thread per row where throughput counts: two tiles and more for every SM, more than three blocks of keys each.  With few
    // tiles and blocks the way through a single tile is what the next kernel waits for (32 x 128 in a BERT-base pass: 2809 us, 2845
    // with it).  Both forms, 12 heads, us a launch (a thread a row | four): 4 blocks 32 x 256: 78 | 93; 6 blocks 32 x 384: 141 | 171;
    // 8 blocks 32 x 512: 230 | 285; 3 blocks 32 x 192: 62 | 74; 2 blocks 32 x 128: 35 | 33, 64 x 128: 58 | 65, 128 x 128: 113 | 126.
    // The line is on the safe side: with 700 tiles and more the form with a thread a row is ahead at two blocks already.
    const bool by_rows = p.num_tiles >= 2 * ctx.sm_count && a.lk > 3 * kAttnKeys;
    const int threads = by_rows ? kRowThreads : kQuadThreads, slots = by_rows ? 2 * ctx.sm_count : ctx.sm_count, grid = p.num_tiles < slots ? p.num_tiles : slots;
    const size_t smem = 2 * (size_t)kAttnQBytes + (size_t)(by_rows ? kRowStages : kQuadStages) * 4 * kAttnKVBytes + (size_t)(threads - 64) * 32 + 1024;
    const int out_mask = (a.o ? 1 : 0) | (a.out.hi ? 2 : 0) | (a.out.h2 ? 4 : 0);
    char num[64];
    snprintf(num, sizeof num, "attention_tc %d %d %d %d\n", by_rows ? 1 : 0, a.naux, rowinv_mask, out_mask);
    const std::string key = num + a.epilogue;  // the rest of the translation unit is fixed text
    Module *mod = ctx.module_find(key);
    if (!mod) {
        std::string src = map_prelude_text();
        src += "struct __align__(64) CUtensorMap { unsigned long long opaque[16]; };\n";
        src += "#define SAGE_EPI_NAUX " + std::to_string(a.naux) + "\n#define SAGE_EPI_ROWINV " + std::to_string(rowinv_mask) + "\n#define SAGE_EPI_OUT " + std::to_string(out_mask) + "\n";
        src += "#define SAGE_EPI_EXPR(x0, x1, x2, x3) (" + (a.epilogue.empty() ? std::string("x0") : a.epilogue) + ")\n";
        src += kGemmTcDeviceSrc;
        src += kGemmH2DeviceSrc;
        src += kAttnTcDeviceSrc;
        src += by_rows ? kAttnRowsDeviceSrc : kAttnQuadsDeviceSrc;
        src += std::string("\nextern \"C\" __global__ void __launch_bounds__(") + (by_rows ? "sage_tc::kRowThreads, 2)\n" : "sage_tc::kQuadThreads, 1)\n") +
               "attention_tc_h2(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,\n"
               "                const __grid_constant__ CUtensorMap map_v, const __grid_constant__ sage_tc::AttnParams p) {\n"
               "    sage_tc::" + (by_rows ? "attn_rows_body" : "attn_body") + "(&map_q, &map_k, &map_v, p);\n}\n";
        sage_status st = ctx.module_get(src, &mod);
        if (st) return st;
        ctx.module_remember(key, mod);
    }
    CUtensorMap map_q, map_k, map_v;
    if (!ctx.dry()) {
        auto map_of = [&](const AttnOperand &o, long long rows, unsigned box, CUtensorMap *map) {
            H2Operand h;
            h.hi = o.hi;
            h.plane = o.plane;
            h.ld = o.ld;
            h.rows = rows;
            h.nb0 = o.nb0;
            h.nb1 = o.nb1;
            h.sb0 = o.sb0;
            h.sb1 = o.sb1;
            return o.hi && aligned16(o.hi) && o.ld % 8 == 0 && o.plane % 8 == 0 && o.sb0 % 8 == 0 && o.sb1 % 8 == 0 && encode_operand(encode, h, a.d, box, map);
        };
        if (!map_of(a.q, a.lq, kAttnQ, &map_q) || !map_of(a.k, a.lk, kAttnKeys, &map_k) || !map_of(a.v, a.lk, kAttnKeys, &map_v))
            return ctx.fail(SAGE_ERR_INVALID, "attention_tc: operand not addressable by TMA");
    }
    std::string label;
    if (ctx.verbose_names)
        label = "attention_tc_h2[" + std::to_string(a.lq) + "x" + std::to_string(a.lk) + "x" + std::to_string(a.d) + "x" + std::to_string(a.batch) + (by_rows ? ",rows]" : "]");
    const uint32_t gr[3] = {(uint32_t)grid, 1, 1}, bl[3] = {(uint32_t)threads, 1, 1};
    void *params[4] = {&map_q, &map_k, &map_v, &p};
    return ctx.launch(mod, "attention_tc_h2", gr, bl, (uint32_t)smem, params, ctx.verbose_names ? label.c_str() : "attention_tc_3xtf32", true, 1);
}

}  // namespace k
}  // namespace sage
