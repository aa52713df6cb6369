// Several [rows, cols] -> [cols] sums, and sums over whole tensors, together: the gradients of a training step's biases and of its
// LayerNorms' scalars, which nothing of the step reads.
// Reference: one launch of the reduction kernel each, src/ops/reduce.rs:258-325.
//
// One launch each, a sum of [4096, 768] took 8.5 us (1.5 TB/s: start, two rounds of loads, meeting), one of [128, 512] 5 us.  Together
// they are one pass over all the matrices, cut into runs of rows of about equal bytes: a block streams whole rows of a matrix (up
// to 2048 columns of them; threads side by side read neighbouring 16 bytes, eight loads in flight), adds its row groups up in
// shared memory and leaves one partial row; a second, small launch adds the partial rows up in order.  A sum over a whole tensor is
// cut into runs in the same way, each of which leaves one value.  Bound by memory.
// Measurements: at column_sums_run.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "kernels.h"
#include "launch.h"

namespace sage {
namespace k {

namespace {

constexpr int kThreads = 512, kLoads = 8, kMaxGroups = 32;

struct ColumnItem {
    const float *x;
    float *y, *partial;      // partial: [chunks, cols], or null where one block holds all rows
    long long pitch, rows;
    int cols, quads;         // quads: 16-byte loads, four columns to a thread
    int unit0;               // blocks of the first launch before this item's
    int chunks, rows_per_chunk;
    int col_blocks, lanes;   // threads of a row group: a block's columns
    int fin0;                // blocks of the second launch before this item's
};
// (cols = 1: `rows` consecutive floats, quads four at a time)
constexpr int kItems = 96;
struct ColumnParams {
    ColumnItem item[kItems];
    int count, from_zero;
};

template <int VEC>
__device__ __forceinline__ void add_rows(const ColumnItem &it, int chunk, int block, float *part, int from_zero) {
    struct alignas(4 * VEC) Vec {
        float v[VEC];
    };
    const int groups = min(kMaxGroups, kThreads / it.lanes), group = (int)threadIdx.x / it.lanes, lane = (int)threadIdx.x - group * it.lanes;
    const int col = (block * it.lanes + lane) * VEC;
    const bool in = group < groups && col < it.cols;
    const long long r0 = (long long)chunk * it.rows_per_chunk;
    const int left = (int)(min(it.rows, r0 + it.rows_per_chunk) - r0);
    float acc[VEC];
#pragma unroll
    for (int e = 0; e < VEC; ++e) acc[e] = 0.f;
    if (in) {
        const float *base = it.x + r0 * it.pitch + col;
        for (int r = group; r < left; r += groups * kLoads) {
            Vec v[kLoads];
#pragma unroll
            for (int u = 0; u < kLoads; ++u) {
                const int at = r + groups * u;
                if (at < left) {
                    v[u] = *reinterpret_cast<const Vec *>(base + at * it.pitch);
                } else {
#pragma unroll
                    for (int e = 0; e < VEC; ++e) v[u].v[e] = 0.f;
                }
            }
#pragma unroll
            for (int w = 1; w < kLoads; w *= 2)  // pairwise: (0 1) (2 3) ..., then (01 23) ...
#pragma unroll
                for (int u = 0; u + w < kLoads; u += 2 * w)
#pragma unroll
                    for (int e = 0; e < VEC; ++e) v[u].v[e] += v[u + w].v[e];
#pragma unroll
            for (int e = 0; e < VEC; ++e) acc[e] += v[0].v[e];
        }
    }
    if (groups > 1) {  // group by group, in order
        if (in)
#pragma unroll
            for (int e = 0; e < VEC; ++e) part[(int)threadIdx.x * VEC + e] = acc[e];
        __syncthreads();
        if (group == 0 && in)
            for (int g = 1; g < groups; ++g)
#pragma unroll
                for (int e = 0; e < VEC; ++e) acc[e] += part[(g * it.lanes + lane) * VEC + e];
    }
    if (group != 0 || !in) return;
    float *to = it.partial ? it.partial + (long long)chunk * it.cols : it.y;
#pragma unroll
    for (int e = 0; e < VEC; ++e) to[col + e] = !it.partial && from_zero ? 0.f + acc[e] : acc[e];
}

// A run of consecutive floats: neighbouring threads read neighbouring 16 bytes, eight loads in flight.
template <int VEC>
__device__ __forceinline__ void add_run(const ColumnItem &it, int chunk, float *part, int from_zero) {
    struct alignas(4 * VEC) Vec {
        float v[VEC];
    };
    const long long r0 = (long long)chunk * it.rows_per_chunk, left = min(it.rows, r0 + it.rows_per_chunk) - r0;  // (a multiple of VEC)
    const float *base = it.x + r0;
    float acc[VEC];
#pragma unroll
    for (int e = 0; e < VEC; ++e) acc[e] = 0.f;
    for (long long i = (long long)threadIdx.x * VEC; i < left; i += (long long)kThreads * VEC * kLoads) {
        Vec v[kLoads];
#pragma unroll
        for (int u = 0; u < kLoads; ++u) {
            const long long at = i + (long long)u * kThreads * VEC;
            if (at < left) {
                v[u] = *reinterpret_cast<const Vec *>(base + at);
            } else {
#pragma unroll
                for (int e = 0; e < VEC; ++e) v[u].v[e] = 0.f;
            }
        }
#pragma unroll
        for (int w = 1; w < kLoads; w *= 2)
#pragma unroll
            for (int u = 0; u + w < kLoads; u += 2 * w)
#pragma unroll
                for (int e = 0; e < VEC; ++e) v[u].v[e] += v[u + w].v[e];
#pragma unroll
        for (int e = 0; e < VEC; ++e) acc[e] += v[0].v[e];
    }
    float a = acc[0];
#pragma unroll
    for (int e = 1; e < VEC; ++e) a += acc[e];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = a;
    __syncthreads();
    if (threadIdx.x >= 32) return;
    a = threadIdx.x < kThreads / 32 ? part[threadIdx.x] : 0.f;
#pragma unroll
    for (int o = kThreads / 64; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (threadIdx.x) return;
    if (it.partial) it.partial[chunk] = a;
    else it.y[0] = from_zero ? 0.f + a : a;
}

__global__ void __launch_bounds__(kThreads) column_sums_kernel(const __grid_constant__ ColumnParams p) {
    __shared__ float part[kThreads * 4];
    grid_dependency_sync();
    int lo = 0, hi = p.count - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if ((int)blockIdx.x >= p.item[mid].unit0) lo = mid;
        else hi = mid - 1;
    }
    const ColumnItem &it = p.item[lo];
    const int unit = (int)blockIdx.x - it.unit0, chunk = unit / it.col_blocks, block = unit - chunk * it.col_blocks;
    if (it.cols == 1) {
        if (it.quads) add_run<4>(it, chunk, part, p.from_zero);
        else add_run<1>(it, chunk, part, p.from_zero);
        return;
    }
    if (it.quads) add_rows<4>(it, chunk, block, part, p.from_zero);
    else add_rows<1>(it, chunk, block, part, p.from_zero);
}

// 32 columns to a block, eight partial rows at a time, each thread's in order.
__global__ void __launch_bounds__(256) column_sums_partials_kernel(const __grid_constant__ ColumnParams p) {
    __shared__ float part[8][33];
    grid_dependency_sync();
    int lo = 0, hi = p.count - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if ((int)blockIdx.x >= p.item[mid].fin0) lo = mid;
        else hi = mid - 1;
    }
    const ColumnItem &it = p.item[lo];
    if (it.cols == 1) {  // one value a run
        float a = 0.f;
#pragma unroll 4
        for (int r = threadIdx.x; r < it.chunks; r += 256) a += it.partial[r];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if ((threadIdx.x & 31) == 0) part[0][threadIdx.x >> 5] = a;
        __syncthreads();
        if (threadIdx.x) return;
        a = part[0][0];
#pragma unroll
        for (int g = 1; g < 8; ++g) a += part[0][g];
        it.y[0] = p.from_zero ? 0.f + a : a;
        return;
    }
    const int lane = threadIdx.x & 31, group = threadIdx.x >> 5, col = ((int)blockIdx.x - it.fin0) * 32 + lane;
    float acc = 0.f;
    if (col < it.cols) {
        const float *base = it.partial + col;
#pragma unroll 4
        for (int r = group; r < it.chunks; r += 8) acc += base[(long long)r * it.cols];
    }
    part[group][lane] = acc;
    __syncthreads();
    if (group == 0 && col < it.cols) {
#pragma unroll
        for (int g = 1; g < 8; ++g) acc += part[g][lane];
        it.y[col] = p.from_zero ? 0.f + acc : acc;
    }
}

}  // namespace

// us, one launch a sum | together (two launches): 72 sums of a BERT-base step (32 x 128 tokens, 1.36 GB) 700 | 225, of which the pass is
// 214 (0.97 of the measured copy rate); 21 of a ResNet-18 step (128 images of 28 x 28) 147 | 17.  With the 50 sums over [4096, 768] of
// its LayerNorms' scalars (two launches each, 9.4 us) BERT-base's whole step 15990 | 15323.
sage_status column_sums_run(Context &ctx, const std::vector<ColumnSum> &all) {
    for (size_t at = 0; at < all.size(); at += kItems) {
        const size_t n = std::min(all.size() - at, (size_t)kItems);
        if (n == 1) {  // by itself it has kernels of its own
            Dims outer, inner;
            outer.ndim = inner.ndim = 1;
            outer.ext[0] = all[at].cols;
            outer.str[0] = 1;
            inner.ext[0] = all[at].rows;
            inner.str[0] = all[at].pitch;  // (1 for a whole tensor: cols = 1, rows consecutive floats)
            sage_status st = reduce(ctx, SAGE_F32, 0, all[at].x, outer, inner, all[at].y);
            if (st) return st;
            continue;
        }
        double bytes = 0.0;
        for (size_t i = 0; i < n; ++i) bytes += 4.0 * (double)all[at + i].rows * (double)all[at + i].cols;
        // Four blocks an SM where there is little to do (one wave of them is resident), 256 KiB a block where there is much: the partial
        // rows are then a hundredth of what is read.
        const double per_block = std::min(262144.0, std::max(32768.0, bytes / (4.0 * ctx.sm_count)));
        ColumnParams p;
        p.count = (int)n;
        p.from_zero = ctx.opts().ref_compat;
        long long floats = 0, units = 0, fins = 0;
        ColumnParams q;  // the items of the second launch
        q.count = 0;
        q.from_zero = p.from_zero;
        for (size_t i = 0; i < n; ++i) {
            const ColumnSum &s = all[at + i];
            ColumnItem &it = p.item[i];
            it.x = s.x;
            it.y = s.y;
            it.partial = nullptr;
            it.pitch = s.pitch;
            it.rows = s.rows;
            it.cols = (int)s.cols;
            const bool whole = s.cols == 1;
            it.quads = (whole ? s.rows : s.cols) % 4 == 0 && (whole || s.pitch % 4 == 0) && reinterpret_cast<uintptr_t>(s.x) % 16 == 0;
            if (whole) {
                it.col_blocks = it.lanes = 1;
                const long long round = (long long)kThreads * kLoads * 4;  // whole rounds of loads
                it.rows_per_chunk = (int)std::max(round, (long long)(per_block / 4.0) / round * round);
            } else {
                const long long vecs = it.quads ? s.cols / 4 : s.cols;
                it.col_blocks = (int)((vecs + kThreads - 1) / kThreads);
                it.lanes = (int)((vecs + it.col_blocks - 1) / it.col_blocks);
                const int groups = std::min(kMaxGroups, kThreads / it.lanes);
                const double row_bytes = (double)it.lanes * (it.quads ? 16.0 : 4.0);
                long long rows = std::max(1LL, (long long)(per_block / row_bytes));
                rows = std::min(s.rows, (rows + groups * kLoads - 1) / (groups * kLoads) * (groups * kLoads));  // whole rounds of loads
                it.rows_per_chunk = (int)std::min(rows, 1LL << 30);
            }
            it.chunks = (int)((s.rows + it.rows_per_chunk - 1) / it.rows_per_chunk);
            it.unit0 = (int)units;
            units += (long long)it.chunks * it.col_blocks;
            it.fin0 = 0;
            if (it.chunks > 1) {
                floats += (long long)it.chunks * s.cols;
                it.fin0 = (int)fins;
                fins += (s.cols + 31) / 32;
            }
        }
        if (units > 0x7fffffffLL) return ctx.fail(SAGE_ERR_UNSUPPORTED, "column sums: too many rows");
        auto name = [&](size_t i) { return all[at + i].cols == 1 ? "reduce_total" : "reduce_cols"; };
        for (size_t i = 0; i + 1 < n; ++i) ctx.note_part(name(i));
        Block *scratch = floats ? ctx.allocator().alloc((size_t)floats * sizeof(float)) : nullptr;
        if (floats && !scratch) {  // no room for partial rows
            for (size_t i = 0; i < n; ++i) {
                ColumnItem &it = p.item[i];
                it.rows_per_chunk = (int)std::min(it.rows, 1LL << 30);
                if ((long long)it.rows_per_chunk < it.rows) return ctx.fail(SAGE_ERR_OOM, "out of memory for the partial results of a column reduction");
                it.chunks = 1;
                it.unit0 = i ? p.item[i - 1].unit0 + p.item[i - 1].col_blocks : 0;
            }
            units = p.item[n - 1].unit0 + p.item[n - 1].col_blocks;
            fins = 0;
        }
        long long used = 0;
        for (size_t i = 0; i < n; ++i) {
            ColumnItem &it = p.item[i];
            if (it.chunks == 1) continue;
            it.partial = reinterpret_cast<float *>(scratch->ptr) + used;
            used += (long long)it.chunks * it.cols;
            q.item[q.count++] = it;
        }
        sage_status st = SAGE_OK;
        ctx.note_launch(name(n - 1));
        if (!ctx.dry()) st = ctx.check_cuda(launch_dependent(ctx.pdl, ctx.stream(), column_sums_kernel, dim3((unsigned)units), dim3(kThreads), 0, p), "column_sums launch");
        if (!st && fins) {
            ctx.note_launch("reduce_partials");
            if (!ctx.dry()) st = ctx.check_cuda(launch_dependent(ctx.pdl, ctx.stream(), column_sums_partials_kernel, dim3((unsigned)fins), dim3(256), 0, q), "column_sums launch");
        }
        if (scratch) ctx.allocator().free(scratch);  // stream-ordered: reused only by work enqueued after these launches
        if (st) return st;
    }
    return SAGE_OK;
}

sage_status LeafBatch::run_sums(Context &ctx) {
    const sage_status st = column_sums.empty() ? SAGE_OK : column_sums_run(ctx, column_sums);
    column_sums.clear();
    held_by_sums.clear();
    own_bytes_of_sums = 0;
    if (!status) status = st;
    return st;
}

sage_status LeafBatch::run_products(Context &ctx) {
    const sage_status st = products.empty() ? SAGE_OK : gemm_tc_group_run(ctx, products);
    products.clear();
    held.clear();
    own_bytes = 0;
    if (!status) status = st;
    return st;
}

sage_status LeafBatch::run(Context &ctx) {
    const sage_status st = run_products(ctx), sums = run_sums(ctx);
    return st ? st : sums;
}

}  // namespace k
}  // namespace sage
