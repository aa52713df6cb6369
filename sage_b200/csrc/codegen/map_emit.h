// Fused elementwise map kernels: CUDA C emitted from an expression, compiled once by NVRTC and
// cached.  Replaces compile_map + translate_id of the reference (src/ops/map.rs:369-410,
// src/ops/core.rs:113-175).
#pragma once
#include <string>
#include <unordered_map>
#include <vector>

#include "../kernels/kernels.h"

namespace sage {

struct MapOperand {
    int dtype;        // sage_dtype
    const void *ptr;  // device address with the element offset applied
    k::Dims view;     // extents (equal to the output's) + element strides (0 = broadcast)
    // > 1: a contiguous f32 operand that is the sum, in order, of so many tensors `slice_stride` elements apart (a product's K slices)
    int slices = 0;
    long long slice_stride = 0;
};

// Per-operator memo of compiled kernels, the counterpart of CachedAccess
// (src/session/context.rs:146-185): signature of the access pattern -> module.
struct MapCache {
    std::unordered_map<std::string, Module *> by_signature;
    Context *owner = nullptr;
};

// What the emitter decided for one launch (exposed for tests).
struct MapPlan {
    std::string source;
    std::string signature;
    int vec = 1;
    int ndim = 1;
    long long n = 0;
    int planes = 0;
    unsigned long long ext[k::kMaxDims] = {0};
    std::vector<std::vector<long long>> strides;  // per input, collapsed dims
};

// `expr` is a C expression over x0..x{n-1}; helper functions come from the prelude
// (sg_exp, sg_max, ...).  The output is contiguous with `out_ext`.
// `planes`: bit 0, the kernel also writes the tf32 hi / lo split of every (f32) result, laid out like y; bit 1, its
// half-precision pieces (in the vector form only, and for whole groups of 64: else the plan drops the bit); bit 2, and not y.
sage_status map_plan(const std::string &expr, const std::vector<MapOperand> &in, int out_dtype, const void *y,
                     int out_ndim, const long long *out_ext, MapPlan *plan, bool emit_source = true, int planes = 0);

// `out` (f32 results only): operand forms of y to write as well; a tensor-core GEMM that reads y next then needs no
// split pass.
sage_status map_launch(Context &ctx, const std::string &expr, const std::vector<MapOperand> &in, int out_dtype,
                       void *y, int out_ndim, const long long *out_ext, MapCache *cache, const k::PlaneOut &out = k::PlaneOut());

}  // namespace sage
