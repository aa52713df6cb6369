// fp32 GEMM on the Blackwell tensor cores: tcgen05.mma (kind::tf32) with TMEM accumulators, operands
// staged by TMA into 128B-swizzled shared memory, 3xTF32 so results stay at fp32 accuracy.
//
// Reference: Gemm::compute_direct / GemmBatched::compute_direct (src/ops/gemm.rs:176-250, 338-421) run
// CLBlast's scalar "XgemmDirect" OpenCL kernel (src/ops/kernels/matmul_direct.opencl:514-709); the
// reference has no tensor-core path at all.  Same contract here: row-major C[M,N] = op(A) * op(B),
// all four transpose modes, strided batches, any M/N/K.
//
// 3xTF32.  Each fp32 operand is split into hi = tf32(a) (round to nearest) and lo = a - hi, and
//   C = A_lo*B_hi + A_hi*B_lo + A_hi*B_hi
// The split lives in two planes next to the tensor.  It is made either by the kernel that produces
// the tensor (the GEMM epilogue and the row kernels can write the planes of their result), or by a
// split pass: split_tf32_flat mirrors a whole allocation element for element, so that every view
// of it that TMA can address (strides that are multiples of 16 bytes) is also a view of the planes;
// split_tf32_view gathers any strided view into compact planes with a row pitch that is a multiple
// of 16 bytes (e.g. K = 147 of the first ResNet convolution).
//
// Accumulation.  The tensor core adds into its fp32 accumulator with truncation, which biases a
// long chain: measured on B200, 3072 chained MMAs (K = 8192) were ~17x less accurate than a plain
// fp32 loop.  So a chain is cut every 128 k: each chunk accumulates in TMEM from zero, and the
// epilogue warps add the finished chunk into fp32 registers with round-to-nearest while the tensor
// core already works on the next chunk in the other TMEM buffer.
//
// The device code is in gemm_tc_device.inc.  It is compiled here with a plain-store epilogue, and
// by NVRTC with the expression of a following elementwise map spliced into the epilogue
// (gemm_tc_run with a non-empty TcGemm::epilogue).
#include <cuda.h>

#include <cmath>
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <vector>

#include "kernels.h"
#include "launch.h"
#include "gemm_tc_device.inc"
#include "gemm_tc_device_src.h"  // generated by the Makefile: the text of gemm_tc_device.inc as kGemmTcDeviceSrc

namespace sage {
void *driver_symbol(const char *name);  // runtime/context.cc
const char *map_prelude_text();         // codegen/map_emit.cc
namespace k {

using namespace sage_tc;

namespace {

template <int BN, int CTAS>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_a2,
               const __grid_constant__ CUtensorMap map_b, const TcParams p) {
    gemm_tc_body<BN, CTAS>(&map_a, &map_a2, &map_b, p);
}

// ---------------------------------------------------------------------------------- operand split
// src: a 4-level strided view (b1, b0, row, col).  dst: [2][nb1*nb0][rows][pitch] with pitch = cols
// rounded up to 4; plane 0 = hi, plane 1 = lo.  Pad columns are written as zeros.
__global__ void __launch_bounds__(256) split_tf32_kernel(const float *__restrict__ src, SplitView v, float *__restrict__ dst, int pitch,
                                                         long long plane_stride) {
    grid_dependency_sync();
    const int groups = pitch >> 2;
    const long long batches = v.nb1 * v.nb0;
    const long long total = batches * v.rows * groups;
    const bool vec_in = v.col_stride == 1 && (v.ld % 4 == 0) && (v.sb0 % 4 == 0) && (v.sb1 % 4 == 0) &&
                        (reinterpret_cast<unsigned long long>(src) % 16 == 0);
    for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < total; g += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(g % groups) * 4;
        const long long rb = g / groups;
        const long long r = rb % v.rows;
        const long long b = rb / v.rows;
        const float *s = src + (b / v.nb0) * v.sb1 + (b % v.nb0) * v.sb0 + r * v.ld + (long long)c * v.col_stride;
        float x[4];
        if (vec_in && c + 4 <= v.cols) {
            const float4 t = *reinterpret_cast<const float4 *>(s);
            x[0] = t.x; x[1] = t.y; x[2] = t.z; x[3] = t.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) x[j] = (c + j < v.cols) ? s[j * v.col_stride] : 0.f;
        }
        float hi[4], lo[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) split_tf32_value(x[j], &hi[j], &lo[j]);
        float *d = dst + (b * v.rows + r) * (long long)pitch + c;
        *reinterpret_cast<float4 *>(d) = make_float4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<float4 *>(d + plane_stride) = make_float4(lo[0], lo[1], lo[2], lo[3]);
    }
}

// n4 groups of 4 consecutive floats; planes laid out like the source.
__global__ void __launch_bounds__(256) split_tf32_flat_kernel(const float4 *__restrict__ src, long long n4, float4 *__restrict__ hi_out,
                                                              float4 *__restrict__ lo_out) {
    grid_dependency_sync();
    for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < n4; g += (long long)gridDim.x * blockDim.x) {
        const float4 x = src[g];
        float4 hi, lo;
        split_tf32_value(x.x, &hi.x, &lo.x);
        split_tf32_value(x.y, &hi.y, &lo.y);
        split_tf32_value(x.z, &hi.z, &lo.z);
        split_tf32_value(x.w, &hi.w, &lo.w);
        hi_out[g] = hi;
        lo_out[g] = lo;
    }
}

unsigned split_grid(const Context &ctx, long long groups) {
    long long blocks = (groups + 255) / 256;
    const long long cap = (long long)ctx.sm_count * 16;
    if (blocks > cap) blocks = cap;
    return (unsigned)(blocks < 1 ? 1 : blocks);
}

bool aligned16(const void *p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

typedef CUresult (*PFN_encodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                    const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                    CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// 5-D tensor map {cols, rows, batch low, batch high, plane} with a {32, box_rows, 1, 1, 1} box
// (K-major) or {32, BK, 1, 1, 1} box (MN-major).
// `blocks` > 0 (MN-major only, see mn_blocked_ok): the contiguous axis is cut into runs of 32, dims {32, rows (k), cols / 32,
// batch low, plane}, and the box {32, BK, blocks, 1, 1} brings the `blocks` 4 KiB sub-tiles of a K-block in with ONE
// load, laid out one after the other exactly as `blocks` separate loads would leave them.
bool encode_map(PFN_encodeTiled encode, const TcOperand &op, unsigned box_rows, bool kmajor, CUtensorMap *map, unsigned blocks = 0) {
    const cuuint64_t row_b = (cuuint64_t)op.ld * 4;
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    static_assert(BK == 32, "K-major tiles are 128-byte swizzled rows of 32 floats");
    const CUtensorMapSwizzle sw = kmajor ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B;
    if (blocks > 0) {
        const cuuint64_t dims[5] = {32, (cuuint64_t)op.rows, (cuuint64_t)(op.cols / 32), (cuuint64_t)op.nb0, 2};
        const cuuint64_t strides[4] = {row_b, 128, op.nb0 > 1 ? (cuuint64_t)op.sb0 * 4 : row_b, (cuuint64_t)op.plane * 4};
        const cuuint32_t box[5] = {32u, (cuuint32_t)BK, blocks, 1, 1};
        return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 5, const_cast<float *>(op.hi), dims, strides, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    }
    const cuuint64_t dims[5] = {(cuuint64_t)op.cols, (cuuint64_t)op.rows, (cuuint64_t)op.nb0, (cuuint64_t)op.nb1, 2};
    // an axis of extent 1 is never stepped along; give it any valid stride
    const cuuint64_t strides[4] = {row_b, op.nb0 > 1 ? (cuuint64_t)op.sb0 * 4 : row_b, op.nb1 > 1 ? (cuuint64_t)op.sb1 * 4 : row_b,
                                   (cuuint64_t)op.plane * 4};
    const cuuint32_t box[5] = {32u, kmajor ? box_rows : (cuuint32_t)BK, 1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 5, const_cast<float *>(op.hi), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// An MN-major operand can be loaded a whole K-block at a time when its contiguous axis is whole runs of 32 floats (the
// cut axis has no ragged end that would read past a row) and one batch axis is enough.
static bool mn_blocked_ok(const TcOperand &op, bool kmajor) {
    static const bool enabled = !(getenv("SAGE_GEMM_BLOCKED_LOAD") && atoi(getenv("SAGE_GEMM_BLOCKED_LOAD")) == 0);
    return enabled && !kmajor && op.cols % 32 == 0 && op.nb1 == 1 && op.cols >= 32;
}

typedef CUresult (*PFN_encodeIm2col)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                     const int *, const int *, cuuint32_t, cuuint32_t, const cuuint32_t *, CUtensorMapInterleave,
                                     CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// im2col-mode map over one plane of an NHWC image: dims {C, W, H, N}; the box is 32 channels of 128
// output pixels.  The pixel-box corners say where a filter window may start: from -pad up to
// (extent + pad - dilation * (taps - 1)) exclusive, walked with the convolution's stride.
bool encode_im2col_map(PFN_encodeIm2col encode, const TcConv &cv, const float *base, CUtensorMap *map) {
    const cuuint64_t dims[4] = {(cuuint64_t)cv.c, (cuuint64_t)cv.w, (cuuint64_t)cv.h, (cuuint64_t)cv.n};
    const cuuint64_t strides[3] = {(cuuint64_t)(cv.sw ? cv.sw : cv.c) * 4, (cuuint64_t)(cv.sh ? cv.sh : cv.w * cv.c) * 4,
                                   (cuuint64_t)(cv.sn ? cv.sn : cv.h * cv.w * cv.c) * 4};
    const int lower[2] = {-cv.win.pad_w, -cv.win.pad_h};
    const int upper[2] = {cv.win.pad_w - (cv.win.ker_w - 1) * cv.win.dil_w, cv.win.pad_h - (cv.win.ker_h - 1) * cv.win.dil_h};
    const cuuint32_t estr[4] = {1, (cuuint32_t)cv.win.stride_w, (cuuint32_t)cv.win.stride_h, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float *>(base), dims, strides, lower, upper, 32u, (cuuint32_t)BM, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tiled map over one plane of an NHWC image, dims {C, W, H, N}, for the tap-reuse convolution: the box is 32 channels
// of a (box_w x box_h) window of one image; coordinates outside the image read as zeros.
bool encode_halo_map(PFN_encodeTiled encode, const TcConv &cv, const float *base, unsigned box_w, unsigned box_h, CUtensorMap *map) {
    const cuuint64_t dims[4] = {(cuuint64_t)cv.c, (cuuint64_t)cv.w, (cuuint64_t)cv.h, (cuuint64_t)cv.n};
    const cuuint64_t strides[3] = {(cuuint64_t)cv.c * 4, (cuuint64_t)(cv.w * cv.c) * 4, (cuuint64_t)(cv.h * cv.w * cv.c) * 4};
    const cuuint32_t box[4] = {32u, box_w, box_h, 1u};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tap reuse (TcParams::a_halo) for a stride-1, undilated convolution with more than one tap: worth it where operand A
// dominates what an SM must take in from L2 (few output channels) and whole output rows fill most of a 128-row tile.
// *wb = positions per output row, *rows = output rows per CTA tile.  SAGE_CONV_HALO=0 turns it off.
static bool conv_halo_plan(const TcConv &cv, long long n_out, int *wb, int *rows) {
    const char *env = getenv("SAGE_CONV_HALO");  // read per launch
    const bool enabled = !(env && atoi(env) == 0);
    const Window &w = cv.win;
    if (!enabled || !cv.on || cv.raw || w.stride_w != 1 || w.stride_h != 1 || w.dil_w != 1 || w.dil_h != 1) return false;
    if (w.ker_w * w.ker_h < 2 || n_out > 128 || n_out % 32) return false;
    if ((cv.sw && cv.sw != cv.c) || (cv.sh && cv.sh != cv.w * cv.c) || (cv.sn && cv.sn != cv.h * cv.w * cv.c)) return false;  // dense NHWC only
    const long long b = cv.out_w + w.ker_w - 1;
    if (b > 128) return false;
    long long r = 128 / b;
    if (r > cv.out_h) r = cv.out_h;
    if (r * cv.out_w < 100) return false;                                  // ~80 % of a tile's rows must be real outputs
    if (b * (r + w.ker_h - 1) > 256) return false;                         // the window is at most 256 pixel rows of shared memory
    if (127 + (w.ker_h - 1) * b + (w.ker_w - 1) > 255) return false;       // ... and the last tap's 128 rows stay inside it
    if (cv.n * ((cv.out_h + r - 1) / r) > 0x3fffffffLL) return false;
    *wb = (int)b;
    *rows = (int)r;
    return true;
}

bool conv_ok(const TcConv &cv) {
    const Window &w = cv.win;
    if (!cv.hi || !aligned16(cv.hi) || cv.plane % 4 || cv.c % 32 || cv.c <= 0 || cv.sw % 4 || cv.sh % 4 || cv.sn % 4) return false;
    if (cv.n < 1 || cv.h < 1 || cv.w < 1 || cv.out_h < 1 || cv.out_w < 1 || cv.out_h * cv.out_w > 0x7fffffffLL) return false;
    if (w.stride_w < 1 || w.stride_w > 8 || w.stride_h < 1 || w.stride_h > 8) return false;          // traversal strides are 3-bit fields
    if (w.pad_w < 0 || w.pad_w > 127 || w.pad_h < 0 || w.pad_h > 127) return false;                  // corners are signed bytes
    const int up_w = w.pad_w - (w.ker_w - 1) * w.dil_w, up_h = w.pad_h - (w.ker_h - 1) * w.dil_h;
    if (up_w < -128 || up_h < -128) return false;
    return (w.ker_w - 1) * w.dil_w <= 255 && (w.ker_h - 1) * w.dil_h <= 255;                         // tap offsets are bytes
}

// `ctas` = 1: 128 x bn tiles, one per SM.  2: 256 x bn tiles, one per SM pair.
int pick_bn(const Context &ctx, long long m, long long n, long long batch, int ctas) {
    const int cands[4] = {256, 192, 128, 64};
    int best = 128;
    double best_cost = 1e300;
    for (int bn : cands) {
        if (bn > 64 && n <= bn / 2) continue;  // mostly padding
        const long long tiles = ((n + bn - 1) / bn) * ((m + BM * ctas - 1) / (BM * ctas)) * batch;
        const long long slots = ctx.sm_count / ctas;
        const long long waves = (tiles + slots - 1) / slots;
        const double cost = (double)waves * (bn + 24);  // +24: per-tile fixed cost in units of columns
        if (cost < best_cost) {
            best_cost = cost;
            best = bn;
        }
    }
    return best;
}

// Ragged columns for a launch that would run 256-wide tiles: should the last `*narrow` column tiles of every row block be
// 192 wide instead?  Tiles are dealt to the CTA pairs round-robin, wide ones first; a 192-wide tile costs 0.78 of a wide
// one (measured per K-block).  Taken when the busiest pair's load drops by 4 % or more.  SAGE_GEMM_RAGGED=0 turns it off.
static bool plan_ragged(long long row_tiles, long long n, long long slots, int *wide, int *narrow) {
    const char *env = getenv("SAGE_GEMM_RAGGED");  // read per launch
    const bool enabled = !(env && atoi(env) == 0);
    if (!enabled || n < 256 + 192 || row_tiles < 1 || slots < 1) return false;
    const double c_wide = 1.0, c_narrow = 0.78;
    auto makespan = [&](long long nw, long long nn) {
        // pair i gets tiles i, i + slots, ...: wide tiles are numbers [0, row_tiles * nw)
        const long long tw = row_tiles * nw, tn = row_tiles * nn, total = tw + tn;
        double worst = 0;
        for (long long i = 0; i < slots && i < total; ++i) {
            const long long mine = (total - i + slots - 1) / slots;                      // tiles of pair i
            const long long mine_wide = i < tw ? (tw - i + slots - 1) / slots : 0;       // ... of which wide
            const double load = mine_wide * c_wide + (mine - mine_wide) * c_narrow;
            if (load > worst) worst = load;
        }
        return worst;
    };
    const long long uniform_tiles = (n + 255) / 256;
    const double base = makespan(uniform_tiles, 0);
    double best = base;
    int best_nn = 0, best_nw = 0;
    for (long long nn = 1; nn * 192 <= n + 191; ++nn) {
        const long long rest = n - nn * 192;
        const long long nw = rest > 0 ? (rest + 255) / 256 : 0;
        if (nw * 256 + nn * 192 - n >= 192) continue;  // a whole tile of padding
        const double t = makespan(nw, nn);
        if (t < best) {
            best = t;
            best_nn = (int)nn;
            best_nw = (int)nw;
        }
    }
    if (best_nn == 0 || best > 0.96 * base) return false;
    *wide = best_nw;
    *narrow = best_nn;
    return true;
}

template <int BN, int CTAS>
sage_status launch_static(Context &ctx, const CUtensorMap &map_a, const CUtensorMap &map_a2, const CUtensorMap &map_b, const TcParams &p,
                          int grid, size_t smem) {
    // per device; the limit covers dynamic + static shared memory, so ask for what is used
    static int attr_set[64] = {0};  // per instantiation and device
    const int dev = ctx.device();
    if (dev < 0 || dev >= 64 || attr_set[dev] != (int)smem) {
        sage_status st = ctx.check_cuda(cudaFuncSetAttribute(gemm_tc_kernel<BN, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                                        "gemm_tc shared memory attribute");
        if (st) return st;
        if (dev >= 0 && dev < 64) attr_set[dev] = (int)smem;
    }
    return ctx.check_cuda(launch_dependent(ctx.pdl, ctx.stream(), CTAS, gemm_tc_kernel<BN, CTAS>, dim3(grid), dim3(kThreads), smem, map_a, map_a2,
                                           map_b, p),
                          "gemm_tc launch");
}

template <int CTAS>
sage_status launch_static_bn(Context &ctx, int bn, const CUtensorMap &map_a, const CUtensorMap &map_a2, const CUtensorMap &map_b,
                             const TcParams &p, int grid, size_t smem) {
    switch (bn) {
    case 256: return launch_static<256, CTAS>(ctx, map_a, map_a2, map_b, p, grid, smem);
    case 192: return launch_static<192, CTAS>(ctx, map_a, map_a2, map_b, p, grid, smem);
    case 128: return launch_static<128, CTAS>(ctx, map_a, map_a2, map_b, p, grid, smem);
    default: return launch_static<64, CTAS>(ctx, map_a, map_a2, map_b, p, grid, smem);
    }
}

// The NVRTC translation unit for one (epilogue expression, operand count, tile width).
constexpr int kRawSplitWarps = 4;  // extra warps of the kernels that split a raw fp32 A operand in shared memory

// The generated lines in front of the device code: they and the tile shape decide the module.
std::string jit_defines(const std::string &expr, int naux, bool row_softmax, bool streamk, bool raw_a, bool halo, bool trace, int rowinv_mask,
                        int cols_mask, int out_mask) {
    std::string s;
    if (row_softmax) s += "#define SAGE_EPI_SOFTMAX 1\n";
    if (streamk) s += "#define SAGE_TC_STREAMK 1\n";
    if (raw_a) s += "#define SAGE_TC_SPLIT_WARPS " + std::to_string(kRawSplitWarps) + "\n";
    if (halo) s += "#define SAGE_TC_HALO 1\n";
    if (trace) s += "#define SAGE_TC_TRACE 1\n";
    s += "#define SAGE_EPI_ROWINV " + std::to_string(rowinv_mask) + "\n";
    s += "#define SAGE_EPI_COLS " + std::to_string(cols_mask) + "\n";
    s += "#define SAGE_EPI_OUT " + std::to_string(out_mask) + "\n";
    s += "struct __align__(64) CUtensorMap { unsigned long long opaque[16]; };\n";
    s += "#define SAGE_EPI_NAUX " + std::to_string(naux) + "\n";
    s += "#define SAGE_EPI_EXPR(x0, x1, x2, x3) (" + expr + ")\n";
    return s;
}

std::string jit_source(const std::string &defines, int bn, int ctas) {
    std::string s = map_prelude_text();
    s += defines;
    s += kGemmTcDeviceSrc;
    s += "\nextern \"C\" __global__ void __launch_bounds__(sage_tc::kThreads, 1)\n"
         "gemm_tc_3xtf32(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_a2,\n"
         "               const __grid_constant__ CUtensorMap map_b, const sage_tc::TcParams p) {\n"
         "    sage_tc::gemm_tc_body<" + std::to_string(bn) + ", " + std::to_string(ctas) + ">(&map_a, &map_a2, &map_b, p);\n}\n";
    return s;
}

}  // namespace

// The smallest products the tiled kernel takes from a caller that must know beforehand (sage_gemm_noalloc).
static bool shape_fills_tiles(long long m, long long n, long long k) { return (m >= 64 || (m >= 16 && k >= 2048)) && n >= 32 && k >= 32; }

static bool shape_within_limits(long long m, long long n, long long k, long long batch) {
    if (m < 1 || n < 1 || k < 1 || batch < 1) return false;
    if (m > 0x7fffffffLL || n > 0x7fffffffLL || k > 0x7fffffffLL || batch > 0x7fffffffLL) return false;
    const long long tiles = ((m + BM - 1) / BM) * ((n + 63) / 64) * batch;
    return tiles < 0x7fffffffLL;
}

bool gemm_tc_shape_ok(long long m, long long n, long long k, long long batch) {
    // Tiny problems are latency-bound and would be mostly TMA padding: leave them to the SIMT kernel.  A short M is
    // worth the padding once there is a weight matrix to stream: the SIMT kernel walks K with one CTA per 128 columns
    // (24 x 768 x 768: 90 us against 12 us here), so the line lies where its K loop outlasts a launch of this kernel.  Up
    // to 4096 outputs its warp-per-output kernel is the faster one (1 x 1000 x 512: 6 us, 16 x 33 x 2047: 8 us).
    if (!shape_fills_tiles(m, n, k) && !(n >= 32 && k >= 128 && n * k >= 65536 && m * n > 4096)) return false;
    return shape_within_limits(m, n, k, batch);
}

bool gemm_tc_supported(const GemmArgs &g) { return shape_fills_tiles(g.m, g.n, g.k) && shape_within_limits(g.m, g.n, g.k, g.batch); }

bool tc_operand_ok(const TcOperand &o) {
    const long long lim = 1LL << 38;  // strides in floats; TMA strides are below 2^40 bytes
    if (!o.hi || !aligned16(o.hi) || o.rows < 1 || o.cols < 1 || o.nb0 < 1 || o.nb1 < 1) return false;
    if (o.ld % 4 || o.ld <= 0 || o.ld >= lim || o.plane % 4 || o.plane <= 0 || o.plane >= lim) return false;
    if (o.nb0 > 1 && (o.sb0 % 4 || o.sb0 <= 0 || o.sb0 >= lim)) return false;
    if (o.nb1 > 1 && (o.sb1 % 4 || o.sb1 <= 0 || o.sb1 >= lim)) return false;
    return o.rows <= 0xffffffffLL && o.cols <= 0xffffffffLL && o.nb0 <= 0xffffffffLL && o.nb1 <= 0xffffffffLL;
}

// ---------------------------------------------------------------------------------- bounded-wait self-test
// One thread waits, with the GEMM kernel's own bounded wait, on an mbarrier that nothing ever
// arrives on.  The wait gives up after its limit (~1 s), records bit 0x100 | 0x40 in the status word
// and the kernel returns normally: the context stays usable.
__global__ void bounded_wait_probe_kernel(unsigned *status) {
    __shared__ __align__(8) unsigned long long bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (!mbar_wait(&bar, 0)) atomicOr(status, 0x100u | 0x40u);
    }
}

sage_status bounded_wait_selftest(Context &ctx) {
    ctx.note_launch("bounded_wait_probe");
    if (ctx.dry()) return SAGE_OK;
    bounded_wait_probe_kernel<<<1, 32, 0, ctx.stream()>>>(ctx.status_word_dev);
    return ctx.check_cuda(cudaGetLastError(), "bounded_wait_probe launch");
}

// The tensor map of an operand without a batch for gemm_group.cu: whole K-blocks of an MN-major operand in one load where that
// can be (*blocked).
bool encode_tc_operand(const TcOperand &op, unsigned box_rows, bool kmajor, bool *blocked, CUtensorMap *map) {
    static const PFN_encodeTiled encode = reinterpret_cast<PFN_encodeTiled>(driver_symbol("cuTensorMapEncodeTiled"));
    if (!encode || !tc_operand_ok(op)) return false;
    *blocked = mn_blocked_ok(op, kmajor) && encode_map(encode, op, 32, false, map, box_rows / 32);
    return *blocked || encode_map(encode, op, kmajor ? box_rows : 32, kmajor, map);
}

// ---------------------------------------------------------------------------------- split launchers
sage_status split_tf32_flat(Context &ctx, const float *src, long long n, float *dst_hi, long long plane) {
    ctx.note_launch("split_tf32");
    if (ctx.dry()) return SAGE_OK;
    if (!aligned16(src) || !aligned16(dst_hi) || plane % 4) return ctx.fail(SAGE_ERR_INVALID, "split_tf32_flat: unaligned");
    const long long n4 = (n + 3) / 4;  // allocations are multiples of 512 bytes, so the last group is readable
    launch_dependent(ctx.pdl, ctx.stream(), split_tf32_flat_kernel, dim3(split_grid(ctx, n4)), dim3(256), 0, reinterpret_cast<const float4 *>(src), n4,
                                                                          reinterpret_cast<float4 *>(dst_hi),
                                                                          reinterpret_cast<float4 *>(dst_hi + plane));
    return ctx.check_cuda(cudaGetLastError(), "split_tf32_flat launch");
}

sage_status split_tf32_view(Context &ctx, const float *src, const SplitView &v, SplitPlanes *out) {
    if (v.rows > 0x7fffffffLL || v.cols > 0x7fffffffLL || v.nb0 * v.nb1 > 0x7fffffffLL)
        return ctx.fail(SAGE_ERR_UNSUPPORTED, "split_tf32: extents beyond 2^31");
    out->rows = (int)v.rows;
    out->cols = (int)v.cols;
    out->batches = (int)(v.nb0 * v.nb1);
    out->pitch = (int)((v.cols + 3) / 4 * 4);
    const long long plane = (long long)out->batches * out->rows * out->pitch;
    out->block = ctx.allocator().alloc((size_t)plane * 2 * sizeof(float));
    if (!out->block) return ctx.fail(SAGE_ERR_OOM, "out of memory for the tf32 operand split");
    out->planes = reinterpret_cast<float *>(out->block->ptr);
    ctx.note_launch("split_tf32");
    if (ctx.dry()) return SAGE_OK;
    launch_dependent(ctx.pdl, ctx.stream(), split_tf32_kernel, dim3(split_grid(ctx, plane / 4)), dim3(256), 0, src, v, out->planes, out->pitch, plane);
    return ctx.check_cuda(cudaGetLastError(), "split_tf32 launch");
}

// ---------------------------------------------------------------------------------- GEMM launcher
static sage_status gemm_tc_launch(Context &ctx, const TcGemm &g);

// Split-K.  A product with few output tiles and a long K (weight gradients: [K'=9C, M=N*OH*OW] x [M, OC])
// would keep a handful of SMs busy for hundreds of K blocks.  It is run instead as a batched GEMM over S
// slices of K, each batch writing its partial product to scratch, followed by a sum over the S partials
// in a fixed order (the result repeats bit for bit).  S divides K, with slices that are multiples of
// 4 floats (TMA strides are multiples of 16 bytes), preferably of the K block.  0 = do not split.
static bool pairs_on() {
    static const bool on = !(getenv("SAGE_GEMM_PAIR") && atoi(getenv("SAGE_GEMM_PAIR")) == 0);
    return on;
}
bool gemm_tc_pairs() { return pairs_on(); }

// Chooses the number of K slices and the tile width together.  Cost model (microseconds, from the
// measured launches): the main loop is bound by operand delivery from L2, ~50 GB/s per SM, i.e. a K block
// of a (BM x bn) tile costs 1.31 us x (BM + bn / ctas) / (BM + 256 / ctas); a tile has ~7 us of fixed cost;
// the sum over the slices reads S x m x n floats at ~3 TB/s plus ~10 us of launch and scratch handling.  A split
// must promise 12 % over the best unsplit choice (the model is only that good).  One case is taken from
// measurement directly: a large product whose waves of tiles are poorly filled (4096^3, such as the weight gradient
// of a 4096 x 4096 layer over 4096 rows: 256 pair tiles on 74
// SM pairs = 3.46 waves, 86 % of 4) runs in two K slices when that fills them (6.92 of 7: 772 -> 622 us
// including the sum, measured while products through sage_gemm ran on these planes too).
static int pick_split_k(Context &ctx, const TcGemm &g, int *bn_out) {
    static const bool enabled = !(getenv("SAGE_GEMM_SPLITK") && atoi(getenv("SAGE_GEMM_SPLITK")) == 0);
    if (!enabled || g.conv.on || g.batch != 1 || g.naux != 0 || !g.epilogue.empty() || g.row_softmax || !g.c || g.c_hi || g.ldc != g.n ||
        g.k < 1024)
        return 0;
    const int ctas = (pairs_on() && g.m > BM) ? 2 : 1;
    const long long units = ctx.sm_count / ctas;
    const int cands[4] = {256, 192, 128, 64};
    {
        const int bn = 256;  // the widest tile moves the fewest operand bytes per FLOP; K slices fill its waves
        const long long tiles = g.n >= 256 ? ((g.m + BM * ctas - 1) / (BM * ctas)) * ((g.n + bn - 1) / bn) : 0;
        const double waves = (double)tiles / (double)units, waves2 = 2.0 * waves;
        auto fill = [](double w) { return w / std::ceil(w); };
        if (waves > 2.0 && waves <= 8.0 && fill(waves2) - fill(waves) > 0.1 && g.k % 64 == 0 && g.k >= 2048) {
            *bn_out = bn;
            return 2;
        }
    }
    double best = 1e300, best_unsplit = 1e300;
    int best_s = 0;
    for (int bn : cands) {
        if (bn > 64 && g.n <= bn / 2) continue;
        const long long tiles = ((g.m + BM * ctas - 1) / (BM * ctas)) * ((g.n + bn - 1) / bn);
        const double t_kb = 1.31 * (BM + bn / ctas) / (double)(BM + 256 / ctas);
        for (long long s = 1; s <= g.k / 256 && s <= 64; ++s) {
            if (g.k % s || (g.k / s) % 4) continue;
            const long long kb = (g.k / s + BK - 1) / BK;
            const long long waves = (tiles * s + units - 1) / units;
            double t = (double)waves * ((double)kb * t_kb + 7.0);
            if (s > 1) t += 10.0 + (double)s * (double)g.m * (double)g.n * 4.0 / 3.0e6;
            if (s == 1 && t < best_unsplit) best_unsplit = t;
            if (t < best) {
                best = t;
                best_s = (int)s;
                *bn_out = bn;
            }
        }
    }
    return best_s >= 2 && best <= 0.88 * best_unsplit ? best_s : 0;
}

int gemm_tc_split_plan(Context &ctx, const TcGemm &g) {
    int bn = 0;
    return pick_split_k(ctx, g, &bn);
}

sage_status gemm_tc_partials(Context &ctx, const TcGemm &g0, Block **partial, int *slices) {
    int bn = 0;
    const int S = pick_split_k(ctx, g0, &bn);
    *partial = nullptr;
    *slices = S;
    if (S < 2) return SAGE_OK;
    const long long ks = g0.k / S, mn = g0.m * g0.n;
    Block *scratch = ctx.allocator().alloc((size_t)S * mn * sizeof(float));
    if (!scratch) return SAGE_OK;
    TcGemm g = g0;
    g.batch = S;
    g.k = ks;
    g.force_bn = bn;
    auto slice = [&](TcOperand &o, bool kmajor) {
        if (kmajor) {  // K is the contiguous axis of the operand as stored
            o.cols = ks;
            o.sb0 = ks;
        } else {
            o.rows = ks;
            o.sb0 = ks * o.ld;
        }
        o.nb0 = S;
        o.nb1 = 1;
        o.sb1 = 0;
        o.bcast = false;
    };
    slice(g.a, g.a_kmajor);
    slice(g.b, g.b_kmajor);
    g.c = reinterpret_cast<float *>(scratch->ptr);
    g.ldc = g.n;
    g.sc0 = mn;
    g.sc1 = 0;
    g.nbc0 = S;
    sage_status st = gemm_tc_launch(ctx, g);
    if (st) ctx.allocator().free(scratch);  // stream-ordered
    else *partial = scratch;
    return st;
}

sage_status gemm_tc_run(Context &ctx, const TcGemm &g0) {
    if (!shape_within_limits(g0.m, g0.n, g0.k, g0.batch)) return ctx.fail(SAGE_ERR_UNSUPPORTED, "gemm_tc: shape not supported");
    Block *scratch = nullptr;
    int S = 0;
    sage_status st = gemm_tc_partials(ctx, g0, &scratch, &S);
    if (st) return st;
    if (!scratch) return gemm_tc_launch(ctx, g0);  // no slices, or no room for the partial products: one pass over K
    Dims outer, inner;
    outer.ndim = 1;
    outer.ext[0] = g0.m * g0.n;
    outer.str[0] = 1;
    inner.ndim = 1;
    inner.ext[0] = S;
    inner.str[0] = g0.m * g0.n;
    st = reduce(ctx, SAGE_F32, 0 /* sum */, reinterpret_cast<float *>(scratch->ptr), outer, inner, g0.c);
    ctx.allocator().free(scratch);  // stream-ordered
    return st;
}

static sage_status gemm_tc_launch(Context &ctx, const TcGemm &g) {
    static PFN_encodeTiled encode = nullptr;
    if (!ctx.dry() && !encode) {
        encode = reinterpret_cast<PFN_encodeTiled>(driver_symbol("cuTensorMapEncodeTiled"));
        if (!encode) return ctx.fail(SAGE_ERR_DEVICE, "cuTensorMapEncodeTiled is not available");
    }
    static PFN_encodeIm2col encode_im2col = nullptr;
    if (g.conv.on && !ctx.dry() && !encode_im2col) {
        encode_im2col = reinterpret_cast<PFN_encodeIm2col>(driver_symbol("cuTensorMapEncodeIm2col"));
        if (!encode_im2col) return ctx.fail(SAGE_ERR_DEVICE, "cuTensorMapEncodeIm2col is not available");
    }
    // hard limits only: whether a shape is worth the tensor cores is the caller's decision (gemm_tc_shape_ok),
    // taken before a product is cut into K slices
    if (g.m < 1 || g.n < 1 || g.k < 1 || g.batch < 1 || g.m > 0x7fffffffLL || g.n > 0x7fffffffLL || g.k > 0x7fffffffLL || g.batch > 0x7fffffffLL)
        return ctx.fail(SAGE_ERR_UNSUPPORTED, "gemm_tc: shape not supported");
    if (g.conv.on && (g.batch != 1 || !g.a_kmajor || g.m != g.conv.n * g.conv.out_h * g.conv.out_w ||
                      g.k != (long long)g.conv.win.ker_h * g.conv.win.ker_w * g.conv.c))
        return ctx.fail(SAGE_ERR_INVALID, "gemm_tc: convolution description does not match the GEMM");
    if (g.naux < 0 || g.naux > kMaxAux || (!g.c && !g.c_hi)) return ctx.fail(SAGE_ERR_INVALID, "gemm_tc: bad epilogue description");
    // CTA pairs for everything with at least two row tiles.  SAGE_GEMM_PAIR=0 turns them off.
    const int ctas = (pairs_on() && g.m > BM) ? 2 : 1;
    int bn = g.force_bn ? g.force_bn : pick_bn(ctx, g.m, g.n, g.batch, ctas);
    if (g.row_softmax) {  // a whole output row in one tile
        if (g.n > 256) return ctx.fail(SAGE_ERR_UNSUPPORTED, "gemm_tc: row softmax needs n <= 256");
        bn = g.n <= 64 ? 64 : g.n <= 128 ? 128 : g.n <= 192 ? 192 : 256;
    }
    int halo_wb = 0, halo_r = 0;
    const bool halo = !g.row_softmax && conv_halo_plan(g.conv, g.n, &halo_wb, &halo_r);
    if (halo) bn = g.n <= 64 ? 64 : 128;  // all output channels in one tile: the window is loaded once
    // per CTA and K-block: its rows of A, its share of B — or, with tap reuse, B alone behind the two window buffers
    const int stage_bytes = halo ? 2 * (bn / ctas) * BK * 4 : 2 * BM * BK * 4 + 2 * (bn / ctas) * BK * 4;
    const int staging = kEpiWarps * kStageBytesPerWarp;  // the epilogue's transposition buffers
    const int fixed_bytes = halo ? kHaloStages * kHaloStageBytes : 0;
    int stages = (227 * 1024 - 2048 - staging - fixed_bytes) / stage_bytes;
    if (stages > 8) stages = 8;
    const size_t smem = (size_t)fixed_bytes + (size_t)stages * stage_bytes + staging + 1024;

    TcParams p;
    p.c = g.c;
    p.c_hi = g.c_hi;
    p.c_plane = g.c_plane;
    p.ldc = g.ldc;
    p.sc0 = g.sc0;
    p.sc1 = g.sc1;
    p.nbc0 = (int)(g.nbc0 < 1 ? 1 : g.nbc0);
    p.na0 = (int)g.a.nb0;
    p.nb0 = (int)g.b.nb0;
    p.a_bcast = g.a.bcast ? 1 : 0;
    p.b_bcast = g.b.bcast ? 1 : 0;
    p.m = (int)g.m;
    p.n = (int)g.n;
    p.k = (int)g.k;
    p.stages = stages;
    p.a_kmajor = g.a_kmajor;
    p.b_kmajor = g.b_kmajor;
    p.a_blocked = (!g.conv.on && mn_blocked_ok(g.a, g.a_kmajor)) ? 1 : 0;
    p.b_blocked = mn_blocked_ok(g.b, g.b_kmajor) ? 1 : 0;
    p.tiles_m = (int)((g.m + BM * ctas - 1) / (BM * ctas));
    p.tiles_n = (int)((g.n + bn - 1) / bn);
    p.rag_wide = p.rag_narrow = 0;
    p.rag_bn = 192;
    if (bn == 256 && !g.conv.on && !g.row_softmax && !g.force_bn) {
        int wide = 0, narrow = 0;
        if (plan_ragged((long long)p.tiles_m * g.batch, g.n, ctx.sm_count / ctas, &wide, &narrow)) {
            p.rag_wide = wide;
            p.rag_narrow = narrow;
            p.tiles_n = wide + narrow;
        }
    }
    p.num_tiles = (int)((long long)p.tiles_m * p.tiles_n * g.batch);
    p.status = ctx.status_word_dev;
    p.softmax_from_zero = ctx.opts().ref_compat ? 1 : 0;
    p.a_im2col = g.conv.on ? 1 : 0;
    p.a_raw = (g.conv.on && g.conv.raw) ? 1 : 0;
    p.conv_cb = g.conv.on ? (int)(g.conv.c / 32) : 1;
    p.conv_kw = g.conv.win.ker_w > 0 ? g.conv.win.ker_w : 1;
    p.conv_q = g.conv.on ? (int)g.conv.out_w : 1;
    p.conv_pq = g.conv.on ? (int)(g.conv.out_h * g.conv.out_w) : 1;
    p.conv_sw = g.conv.win.stride_w;
    p.conv_sh = g.conv.win.stride_h;
    p.conv_pw = g.conv.win.pad_w;
    p.conv_ph = g.conv.win.pad_h;
    p.conv_dw = g.conv.win.dil_w;
    p.conv_dh = g.conv.win.dil_h;
    if (g.conv.on) {
        p.na0 = 1;
        p.a_bcast = 1;
    }
    p.a_halo = halo ? 1 : 0;
    p.halo_wb = halo_wb;
    p.halo_r = halo_r;
    p.halo_rt = halo ? (int)((g.conv.out_h + halo_r - 1) / halo_r) : 1;
    p.halo_taps = g.conv.win.ker_h * g.conv.win.ker_w;
    p.halo_box_bytes = halo ? 128 * halo_wb * (halo_r + g.conv.win.ker_h - 1) : 0;
    p.conv_n = (int)g.conv.n;
    p.conv_p = (int)g.conv.out_h;
    if (halo) {  // an M tile is the halo_r output rows of each of the pair's CTAs
        p.a_im2col = 0;
        p.tiles_m = (int)((g.conv.n * p.halo_rt + ctas - 1) / ctas);
        p.num_tiles = p.tiles_m * p.tiles_n;
    }
    bool vec = g.n % 4 == 0 && g.ldc % 4 == 0 && g.sc0 % 4 == 0 && g.sc1 % 4 == 0 && (!g.c || aligned16(g.c)) &&
               (!g.c_hi || (aligned16(g.c_hi) && g.c_plane % 4 == 0));
    for (int i = 0; i < kMaxAux; ++i) {
        TcAux &a = p.aux[i];
        a.ptr = nullptr;
        a.s0 = a.s1 = a.sr = 0;
        a.sc = 0;
        if (i >= g.naux) continue;
        a.ptr = g.aux[i].ptr;
        a.s0 = g.aux[i].s0;
        a.s1 = g.aux[i].s1;
        a.sr = g.aux[i].sr;
        a.sc = g.aux[i].sc;
        if (a.sc != 0 && a.sc != 1) return ctx.fail(SAGE_ERR_INVALID, "gemm_tc: epilogue operand column stride must be 0 or 1");
        if (a.sc == 1) vec = vec && aligned16(a.ptr) && a.s0 % 4 == 0 && a.s1 % 4 == 0 && a.sr % 4 == 0;
    }
    p.vec_ok = vec ? 1 : 0;
    const int slots = ctx.sm_count / ctas;
    int grid = ctas * (p.num_tiles < slots ? p.num_tiles : slots);
    // Stream-K where whole tiles fill the machine badly (64 pair tiles on 74 SM pairs; 2.6 waves): the CTAs share the
    // (tile, K-block) space evenly and tiles cut between two CTAs are summed through scratch.  Needs a K long enough to
    // cut, and is not worth its fix-ups once there are many waves.  OFF unless SAGE_GEMM_STREAMK=1 (read per launch):
    // measured on B200 it loses — 4096 x 768 x 768: 37.1 -> 43.7 us, 4096 x 3072 x 768: 92.0 -> 95.4 us, 4096 x 768 x
    // 3072: 101.7 -> 104.9 us, the BERT-base step 4.98 -> 5.12 ms.  The K loop is bound by operand delivery per SM, so
    // evening out the K-blocks buys less than the partial tiles (a 128 KiB write and read per CTA, epilogue warps that
    // wait for a neighbour's flag) cost.
    p.sk_on = 0;
    p.sk_partial = nullptr;
    p.sk_flags = nullptr;
    p.sk_epoch = 0;
    {
        const char *env = getenv("SAGE_GEMM_STREAMK");
        const bool enabled = env && atoi(env) != 0;
        const long long num_kb = (g.k + BK - 1) / BK, total = (long long)p.num_tiles * num_kb;
        const double waves = (double)p.num_tiles / (double)slots;
        const bool badly_filled = waves / std::ceil(waves) < 0.92 && p.num_tiles <= 8LL * slots;
        if (enabled && !ctx.dry() && !g.conv.on && !g.row_softmax && p.rag_narrow == 0 && num_kb >= 8 && total >= 6LL * slots && badly_filled) {
            const size_t partial_bytes = (size_t)ctx.sm_count * BM * 256 * sizeof(float);  // one 128 x 256 fp32 tile per CTA at most
            const size_t flag_bytes = (size_t)ctx.sm_count * kEpiWarps * sizeof(unsigned);
            if (!ctx.streamk_block) {
                ctx.streamk_block = ctx.allocator().alloc(partial_bytes + flag_bytes);
                if (ctx.streamk_block) {
                    ctx.streamk_bytes = partial_bytes + flag_bytes;
                    sage_status st = ctx.check_cuda(cudaMemsetAsync(reinterpret_cast<char *>(ctx.streamk_block->ptr) + partial_bytes, 0, flag_bytes, ctx.stream()),
                                                    "stream-K flags");
                    if (st) return st;
                }
            }
            if (ctx.streamk_block) {  // without room for the scratch the product simply runs tile by tile
                p.sk_on = 1;
                p.sk_partial = reinterpret_cast<float *>(ctx.streamk_block->ptr);
                p.sk_flags = reinterpret_cast<unsigned *>(reinterpret_cast<char *>(ctx.streamk_block->ptr) + partial_bytes);
                p.sk_epoch = ++ctx.streamk_epoch;
                grid = ctas * slots;
            }
        }
    }

    // SAGE_GEMM_TRACE=<file> (read per launch): this launch runs the build that counts the cycles its roles wait and work,
    // the host waits for it and appends {m, n, k, batch, bn, ctas, grid, stages} + 16 words per CTA to the file.
    // A measuring aid (`python -m sage_b200.microbench --case gemm_trace`); every launch is then followed by a synchronisation.
    const char *trace_path = ctx.dry() ? nullptr : getenv("SAGE_GEMM_TRACE");
    p.trace = nullptr;
    if (trace_path && *trace_path) {
        const size_t bytes = (size_t)ctx.sm_count * 16 * sizeof(unsigned long long);
        if (!ctx.gemm_trace_block) ctx.gemm_trace_block = ctx.allocator().alloc(bytes);
        if (ctx.gemm_trace_block) {
            p.trace = reinterpret_cast<unsigned long long *>(ctx.gemm_trace_block->ptr);
            sage_status st = ctx.check_cuda(cudaMemsetAsync(p.trace, 0, bytes, ctx.stream()), "GEMM trace buffer");
            if (st) return st;
        }
    }
    auto finish = [&](sage_status st) {
        if (st || !p.trace) return st;
        std::vector<unsigned long long> words((size_t)grid * 16);
        st = ctx.check_cuda(cudaMemcpyAsync(words.data(), p.trace, words.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost, ctx.stream()), "GEMM trace read");
        if (!st) st = ctx.check_cuda(cudaStreamSynchronize(ctx.stream()), "GEMM trace read");
        if (st) return st;
        if (FILE *fp = fopen(trace_path, "ab")) {
            const int header[8] = {(int)g.m, (int)g.n, (int)g.k, (int)g.batch, bn, ctas, grid, stages};
            fwrite(header, sizeof(int), 8, fp);
            fwrite(words.data(), sizeof(unsigned long long), words.size(), fp);
            fclose(fp);
        }
        return st;
    };
    std::string label;  // with verbose names: one profile line per shape
    if (ctx.verbose_names)
        label = "gemm_tc_3xtf32[" + std::to_string(g.m) + "x" + std::to_string(g.n) + "x" + std::to_string(g.k) + (g.batch > 1 ? "x" + std::to_string(g.batch) : "") +
                (g.conv.on ? ",conv" : "") + ",bn" + std::to_string(bn) + (p.rag_narrow ? "+" + std::to_string(p.rag_narrow) + "x192" : "") + (ctas == 2 ? ",pair" : "") + "]";
    int rowinv_mask = 0, cols_mask = 0;  // which epilogue operands have no row stride / a column stride: compiled in
    for (int i = 0; i < g.naux; ++i) {
        if (g.aux[i].sr == 0) rowinv_mask |= 1 << i;
        if (g.aux[i].sc != 0) cols_mask |= 1 << i;
    }
    Module *mod = nullptr;
    // the stream-K paths and the operand-split warps exist only in NVRTC builds
    const bool jit = !g.epilogue.empty() || g.naux > 0 || g.row_softmax || p.sk_on || p.a_raw || halo || p.trace;
    if (jit) {
        const std::string defines = jit_defines(g.epilogue.empty() ? "x0" : g.epilogue, g.naux, g.row_softmax, p.sk_on != 0, p.a_raw != 0, halo,
                                                p.trace != nullptr, rowinv_mask, cols_mask, (g.c ? 1 : 0) | (g.c_hi ? 2 : 0));
        const std::string key = "gemm_tc " + std::to_string(bn) + " " + std::to_string(ctas) + "\n" + defines;
        mod = ctx.module_find(key);
        if (!mod) {
            sage_status st = ctx.module_get(jit_source(defines, bn, ctas), &mod);
            if (st) return st;
            ctx.module_remember(key, mod);
        }
    }
    CUtensorMap map_a, map_a2, map_b;
    if (!ctx.dry()) {
        if (g.conv.on) {
            if (!conv_ok(g.conv)) return ctx.fail(SAGE_ERR_INVALID, "gemm_tc: convolution not addressable by im2col TMA");
            if (halo) {
                const unsigned bh = (unsigned)(halo_r + g.conv.win.ker_h - 1);
                if (!encode_halo_map(encode, g.conv, g.conv.hi, (unsigned)halo_wb, bh, &map_a) ||
                    !encode_halo_map(encode, g.conv, g.conv.hi + g.conv.plane, (unsigned)halo_wb, bh, &map_a2))
                    return ctx.fail(SAGE_ERR_DEVICE, "cuTensorMapEncodeTiled failed");
            } else if (!encode_im2col_map(encode_im2col, g.conv, g.conv.hi, &map_a) ||
                !encode_im2col_map(encode_im2col, g.conv, g.conv.raw ? g.conv.hi : g.conv.hi + g.conv.plane, &map_a2))
                return ctx.fail(SAGE_ERR_DEVICE, "cuTensorMapEncodeIm2col failed");
        } else {
            if (!tc_operand_ok(g.a)) return ctx.fail(SAGE_ERR_INVALID, "gemm_tc: operand not addressable by TMA");
            if (p.a_blocked && !encode_map(encode, g.a, 32, false, &map_a, BM / 32)) p.a_blocked = 0;  // the driver declined the cut axis
            if (!p.a_blocked && !encode_map(encode, g.a, g.a_kmajor ? BM : 32, g.a_kmajor, &map_a)) return ctx.fail(SAGE_ERR_DEVICE, "cuTensorMapEncodeTiled failed");
            map_a2 = map_a;
        }
        if (!tc_operand_ok(g.b)) return ctx.fail(SAGE_ERR_INVALID, "gemm_tc: operand not addressable by TMA");
        if (p.b_blocked && !encode_map(encode, g.b, 32, false, &map_b, (unsigned)(bn / ctas / 32))) p.b_blocked = 0;
        if (!p.b_blocked && !encode_map(encode, g.b, g.b_kmajor ? (unsigned)(bn / ctas) : 32, g.b_kmajor, &map_b))
            return ctx.fail(SAGE_ERR_DEVICE, "cuTensorMapEncodeTiled failed");
        if (p.rag_narrow > 0) {  // the narrow tiles' B box, in the slot the convolutions use for their second plane
            const unsigned rows = (unsigned)(p.rag_bn / ctas);
            const bool ok2 = p.b_blocked ? encode_map(encode, g.b, 32, false, &map_a2, rows / 32)
                                         : encode_map(encode, g.b, g.b_kmajor ? rows : 32, g.b_kmajor, &map_a2);
            if (!ok2) return ctx.fail(SAGE_ERR_DEVICE, "cuTensorMapEncodeTiled failed");
        }
    }
    if (jit) {
        const uint32_t gr[3] = {(uint32_t)grid, 1, 1}, bl[3] = {(uint32_t)(kThreads + (p.a_raw ? 32 * kRawSplitWarps : 0)), 1, 1};
        void *params[4] = {&map_a, &map_a2, &map_b, &p};
        return finish(ctx.launch(mod, "gemm_tc_3xtf32", gr, bl, (uint32_t)smem, params, ctx.verbose_names ? label.c_str() : nullptr, true, ctas));
    }
    ctx.note_launch(ctx.verbose_names ? label.c_str() : "gemm_tc_3xtf32");
    if (ctx.dry()) return SAGE_OK;
    return ctas == 2 ? launch_static_bn<2>(ctx, bn, map_a, map_a2, map_b, p, grid, smem)
                     : launch_static_bn<1>(ctx, bn, map_a, map_a2, map_b, p, grid, smem);
}

sage_status gemm_tcgen05(Context &ctx, const GemmArgs &g) {
    if (!gemm_tc_shape_ok(g.m, g.n, g.k, g.batch)) return SAGE_ERR_UNSUPPORTED;
    return gemm_h2(ctx, g);
}

}  // namespace k
}  // namespace sage
