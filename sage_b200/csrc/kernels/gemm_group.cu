// Several independent products in one launch, on tf32 planes: the weight gradients of a training step, which nothing of the
// step reads and which by themselves have few output tiles and a long K.  (Reference: one XgemmDirect launch each,
// src/ops/gemm.rs:176-250.)
//
// One product after the other, a launch of 768 x 768 x 4096 filled the chip only when its K was cut into eight slices, whose
// partial products were written (19 MB), read back by a launch of their own and cost as much traffic as the operands; one of
// 576 x 64 x 6272 was all start and end (15 us, 7 for the sum).  Together they have tiles for every CTA pair: a CTA pair walks over
// units (a tile and a run of its K), the next unit's operands arriving while the last one's tile is stored, and K is cut only
// as far as the pairs' shares need evening out.  Weight gradients of a BERT-base step (72, 32 x 128 tokens) and of a ResNet-18
// step (20, 128 images of 28 x 28): the figures are at gemm_tc_group_run.
//
// The arithmetic is gemm_tc_body's (gemm_tc_device.inc): 3xTF32, chains of at most 128 k, chains added in fp32 registers.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <memory>
#include <string>
#include <vector>

#include "kernels.h"
#include "launch.h"
#include "gemm_tc_device.inc"

namespace sage {
namespace k {

using namespace sage_tc;

// gemm_tcgen05.cu
bool gemm_tc_pairs();
bool encode_tc_operand(const TcOperand &op, unsigned box_rows, bool kmajor, bool *blocked, CUtensorMap *map);

namespace {

constexpr int kGroupBN = 256;                       // the widest tile; a narrower one takes fewer of the columns
constexpr int kGroupABytes = BM * BK * 4;
constexpr int kKMajorA = 1, kKMajorB = 2, kBlockedA = 4, kBlockedB = 8, kVec = 16;

struct alignas(64) GroupItem {
    CUtensorMap a, b;
    float *c;         // the result, or the first of its slices' partial results (m * n floats apart)
    int ldc, m, n, num_kb, kb_per_slice;
    int unit0;        // units of the items before this one
    int tiles_m, tiles_n;
    short bn, flags;
    int chain;        // K-blocks of an accumulation chain
};
template <int MAX>
struct GroupParams {
    GroupItem item[MAX];
    int count, units, stages, b_bytes;  // b_bytes: a stage's room for one piece of operand B
    unsigned *status;
};

struct GroupUnit {
    int u, i;               // unit, item
    int m0, n0, kb0, kb1, slice;
};
template <class P>
__device__ __forceinline__ void group_locate(const P &p, GroupUnit *g) {  // g->u is set, g->i not behind it
    while (g->i + 1 < p.count && g->u >= p.item[g->i + 1].unit0) ++g->i;
    const GroupItem &it = p.item[g->i];
    const int per_slice = it.tiles_m * it.tiles_n;
    int r = g->u - it.unit0;
    g->slice = r / per_slice;
    r -= g->slice * per_slice;
    g->m0 = (r / it.tiles_n) * (2 * BM);
    g->n0 = (r % it.tiles_n) * it.bn;
    g->kb0 = g->slice * it.kb_per_slice;
    g->kb1 = min(it.num_kb, g->kb0 + it.kb_per_slice);
}

// Roles, barriers and bounded waits as in gemm_tc_body<BN, 2>: CTA pairs, warp 0 loads, warp 1 issues, 16 epilogue warps.
template <int MAX>
__global__ void __launch_bounds__(64 + 32 * kEpiWarps, 1) gemm_tc_group_kernel(const __grid_constant__ GroupParams<MAX> p) {
    extern __shared__ __align__(1024) char smem_raw[];
    __shared__ __align__(8) unsigned long long full_bar[8], empty_bar[8], tmem_full[2], tmem_empty[2];
    __shared__ unsigned tmem_base_slot;
    __shared__ volatile int abort_flag;
    constexpr unsigned TMEM_COLS = 2 * kGroupBN;
    char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const unsigned rank = (unsigned)__shfl_sync(0xffffffffu, (int)cluster_rank(), 0);
    const int pidx = (int)blockIdx.x / 2, npairs = (int)gridDim.x / 2;
    const int stage_bytes = 2 * kGroupABytes + 2 * p.b_bytes;

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tmem_full[b], 1);
            mbar_init(&tmem_empty[b], kEpiWarps * 2);
        }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem_base = tmem_base_slot;
    auto timeout = [&](unsigned where) {
        atomicOr(p.status, 0x100u | where);
        abort_flag = 1;
    };
    if (warp == 1 && rank == 0) {  // the leader addresses both CTAs' accumulators with its own address
        unsigned peer_base = tmem_base;
        if (lane == 0) asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(peer_base) : "r"(peer_addr(smem_u32(&tmem_base_slot), 1)) : "memory");
        if (lane == 0 && peer_base != tmem_base) {
            atomicOr(p.status, 0x200u);
            abort_flag = 1;
        }
        __syncwarp();
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    GroupUnit g;
    g.u = pidx;
    g.i = 0;
    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer (whole warp, one elected lane issues)
        int kbg = 0;
        if (g.u < p.units) {
            group_locate(p, &g);
            if (elect_one()) {
                asm volatile("prefetch.tensormap [%0];" ::"l"(&p.item[g.i].a) : "memory");
                asm volatile("prefetch.tensormap [%0];" ::"l"(&p.item[g.i].b) : "memory");
            }
        }
        __syncwarp();
        asm volatile("griddepcontrol.wait;" ::: "memory");
        bool live = true;
        for (; g.u < p.units && live && !__any_sync(0xffffffffu, abort_flag != 0); g.u += npairs) {
            group_locate(p, &g);
            const GroupItem &it = p.item[g.i];
            {  // the next unit's maps, beside this one's loads
                GroupUnit next = g;
                next.u += npairs;
                if (next.u < p.units) {
                    while (next.i + 1 < p.count && next.u >= p.item[next.i + 1].unit0) ++next.i;
                    if (next.i != g.i && elect_one()) {
                        asm volatile("prefetch.tensormap [%0];" ::"l"(&p.item[next.i].a) : "memory");
                        asm volatile("prefetch.tensormap [%0];" ::"l"(&p.item[next.i].b) : "memory");
                    }
                    __syncwarp();
                }
            }
            const int b_rows = it.bn / 2, m0 = g.m0 + (int)rank * BM, nb = g.n0 + (int)rank * b_rows;
            const bool a_kmajor = it.flags & kKMajorA, b_kmajor = it.flags & kKMajorB, a_blocked = it.flags & kBlockedA, b_blocked = it.flags & kBlockedB;
            for (int kb = g.kb0; kb < g.kb1; ++kb, ++kbg) {
                const int s = kbg % p.stages;
                if (!mbar_wait_warp(&empty_bar[s], ((kbg / p.stages) & 1) ^ 1)) {
                    if (lane == 0) timeout(1);
                    live = false;
                    break;
                }
                char *st = smem + (size_t)s * stage_bytes;
                const unsigned fb = peer_addr(smem_u32(&full_bar[s]), 0);  // both CTAs' loads complete on the leader's barrier
                if (elect_one()) {
                    if (rank == 0) mbar_expect_tx(&full_bar[s], (unsigned)((2 * kGroupABytes + 2 * b_rows * BK * 4) * 2));
                    load_operand<true>(&it.a, st, fb, a_kmajor, a_blocked, BM, m0, kb * BK, 0, 0, 0);
                    load_operand<true>(&it.a, st + kGroupABytes, fb, a_kmajor, a_blocked, BM, m0, kb * BK, 0, 0, 1);
                    load_operand<true>(&it.b, st + 2 * kGroupABytes, fb, b_kmajor, b_blocked, b_rows, nb, kb * BK, 0, 0, 0);
                    load_operand<true>(&it.b, st + 2 * kGroupABytes + p.b_bytes, fb, b_kmajor, b_blocked, b_rows, nb, kb * BK, 0, 0, 1);
                }
                __syncwarp();
            }
        }
        for (int i = kbg > p.stages ? kbg - p.stages : 0; i < kbg; ++i) {  // nothing may still be landing here
            const bool landed = rank == 0 ? mbar_wait_warp(&full_bar[i % p.stages], (i / p.stages) & 1) : mbar_wait_warp(&empty_bar[i % p.stages], (i / p.stages) & 1);
            if (!landed && lane == 0) timeout(2);
        }
    } else if (warp == 1 && rank == 0) {
        // ------------------------------------------------------------------ MMA issuer (whole warp, one elected lane issues)
        const unsigned smem0 = smem_u32(smem);
        int cg = 0, s = 0;
        unsigned s_parity = 0;
        bool ok = !__any_sync(0xffffffffu, abort_flag != 0);
        for (; g.u < p.units && ok; g.u += npairs) {
            group_locate(p, &g);
            const GroupItem &it = p.item[g.i];
            const bool a_kmajor = it.flags & kKMajorA, b_kmajor = it.flags & kKMajorB;
            const unsigned idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((a_kmajor ? 0u : 1u) << 15) | ((b_kmajor ? 0u : 1u) << 16) | ((unsigned)((2 * BM) >> 4) << 24) |
                                   ((unsigned)(it.bn >> 3) << 17);
            // layouts as in gemm_tc_body: K-major rows of 128 bytes, or MN-major blocks of 32 columns
            const unsigned long long a_desc0 = smem_desc(0u, a_kmajor ? 16u : (unsigned)(BK * 128), a_kmajor ? 8u * BK * 4u : 512u, a_kmajor ? 2u : 1u);
            const unsigned long long b_desc0 = smem_desc(0u, b_kmajor ? 16u : (unsigned)(BK * 128), b_kmajor ? 8u * BK * 4u : 512u, b_kmajor ? 2u : 1u);
            const unsigned a_step16 = (a_kmajor ? 32u : 1024u) >> 4, b_step16 = (b_kmajor ? 32u : 1024u) >> 4;
            for (int kb_begin = g.kb0; kb_begin < g.kb1 && ok; kb_begin += it.chain, ++cg) {
                const int buf = cg & 1;
                if (!mbar_wait_warp(&tmem_empty[buf], ((cg >> 1) & 1) ^ 1)) {
                    if (lane == 0) timeout(16);
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned tmem_d = tmem_base + (unsigned)(buf * kGroupBN);
                const int kb_end = min(g.kb1, kb_begin + it.chain);
                for (int kb = kb_begin; kb < kb_end; ++kb) {
                    if (!mbar_wait_warp(&full_bar[s], s_parity)) {
                        if (lane == 0 && !abort_flag) timeout(4);
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const unsigned a_hi = smem0 + (unsigned)(s * stage_bytes), a_lo = a_hi + kGroupABytes;
                    const unsigned b_hi = a_hi + 2 * kGroupABytes, b_lo = b_hi + (unsigned)p.b_bytes;
                    const unsigned long long da_hi0 = a_desc0 + (a_hi >> 4), da_lo0 = a_desc0 + (a_lo >> 4);
                    const unsigned long long db_hi0 = b_desc0 + (b_hi >> 4), db_lo0 = b_desc0 + (b_lo >> 4);
                    if (elect_one()) {
#pragma unroll
                        for (int ks = 0; ks < BK / 8; ++ks) {
                            const unsigned long long da_hi = da_hi0 + ks * a_step16, da_lo = da_lo0 + ks * a_step16;
                            const unsigned long long db_hi = db_hi0 + ks * b_step16, db_lo = db_lo0 + ks * b_step16;
                            umma_tf32_pair(tmem_d, da_lo, db_hi, idesc, (kb > kb_begin || ks > 0) ? 1u : 0u);  // small terms first
                            umma_tf32_pair(tmem_d, da_hi, db_lo, idesc, 1u);
                            umma_tf32_pair(tmem_d, da_hi, db_hi, idesc, 1u);
                        }
                        umma_commit_pair(&empty_bar[s]);
                        if (kb == kb_end - 1) umma_commit_pair(&tmem_full[buf]);
                    }
                    __syncwarp();
                    if (++s == p.stages) {
                        s = 0;
                        s_parity ^= 1u;
                    }
                }
            }
        }
    } else if (warp >= 2) {
        // ------------------------------------------------------------------ epilogue: a quarter of a tile's columns to a warp
        asm volatile("griddepcontrol.wait;" ::: "memory");  // the results may lie where the kernel before this one still reads
        const int q = warp & 3, h = (warp - 2) >> 2;
        float4 *stage = reinterpret_cast<float4 *>(smem + (size_t)p.stages * stage_bytes + (size_t)(warp - 2) * kStageBytesPerWarp);
        const int sub_r = lane >> 2, sub_c = lane & 3;
        float acc[64];
        int cg = 0;
        bool ok = true;
        for (; g.u < p.units && ok; g.u += npairs) {
            group_locate(p, &g);
            const GroupItem &it = p.item[g.i];
            const int part = it.bn / 4, runs = it.bn / 64;  // columns of this warp, in runs of 16
#pragma unroll
            for (int i = 0; i < 64; ++i) acc[i] = 0.f;
            for (int kb = g.kb0; kb < g.kb1; kb += it.chain, ++cg) {
                const int buf = cg & 1;
                ok = mbar_wait_warp(&tmem_full[buf], (cg >> 1) & 1);
                if (!ok) {
                    if (lane == 0 && !abort_flag) timeout(8);
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned taddr = tmem_base + (unsigned)(buf * kGroupBN) + ((unsigned)(q * 32) << 16) + (unsigned)(h * part);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (j >= runs) break;
                    unsigned r[16];
                    tmem_ld16(taddr + j * 16, r);
#pragma unroll
                    for (int i = 0; i < 16; ++i) acc[j * 16 + i] += __uint_as_float(r[i]);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    if (rank == 0) mbar_arrive(&tmem_empty[buf]);
                    else mbar_arrive_remote_tmem(peer_addr(smem_u32(&tmem_empty[buf]), 0));
                }
            }
            if (!ok) break;
            // Sub-tiles of 32 x 16 are turned round through shared memory, as in gemm_tc_body: whole 64-byte row segments.
            const int row0 = g.m0 + (int)rank * BM + q * 32 + sub_r, colb = g.n0 + h * part + sub_c * 4;
            const int rows_left = it.m - row0, cols_left = it.n - colb;
            float *at = it.c + ((long long)g.slice * it.m + row0) * it.ldc + colb;  // (slices lie m rows apart)
            const long long step = 8LL * it.ldc;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (j >= runs) break;
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    stage[lane * 4 + (c ^ ((lane >> 1) & 3))] = make_float4(acc[j * 16 + c * 4], acc[j * 16 + c * 4 + 1], acc[j * 16 + c * 4 + 2], acc[j * 16 + c * 4 + 3]);
                __syncwarp();
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const int r = t * 8 + sub_r;
                    const float4 v = stage[r * 4 + (sub_c ^ ((r >> 1) & 3))];
                    float *to = at + t * step + 16 * j;
                    if (8 * t >= rows_left) continue;
                    if (it.flags & kVec) {
                        if (16 * j + 4 <= cols_left) *reinterpret_cast<float4 *>(to) = v;
                    } else {
                        if (16 * j < cols_left) to[0] = v.x;
                        if (16 * j + 1 < cols_left) to[1] = v.y;
                        if (16 * j + 2 < cols_left) to[2] = v.z;
                        if (16 * j + 3 < cols_left) to[3] = v.w;
                    }
                }
                __syncwarp();
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();  // neither CTA leaves (or frees TMEM) while the other may still touch it
    if (warp == 1) {
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

// ---------------------------------------------------------------------------------- the sums over the slices
struct SliceItem {
    const float *x;
    float *y;
    long long n;      // floats of a slice
    int slices, unit0;
};
constexpr int kSliceItems = 100;
struct SliceParams {
    SliceItem item[kSliceItems];
    int count, from_zero;
};
// A thread owns four consecutive results and keeps up to eight loads in flight; the slices are added in order.
__global__ void __launch_bounds__(256) sum_slices_group_kernel(const __grid_constant__ SliceParams p) {
    grid_dependency_sync();
    int lo = 0, hi = p.count - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if ((int)blockIdx.x >= p.item[mid].unit0) lo = mid;
        else hi = mid - 1;
    }
    const SliceItem &it = p.item[lo];
    const long long i = ((long long)((int)blockIdx.x - it.unit0) * 256 + threadIdx.x) * 4;
    if (i >= it.n) return;
    const float *base = it.x + i;
    if (i + 4 > it.n || it.n % 4) {  // any size: element by element
        for (int e = 0; e < 4 && i + e < it.n; ++e) {
            float a = base[e];
            for (int s = 1; s < it.slices; ++s) a += base[e + s * it.n];
            it.y[i + e] = p.from_zero ? 0.f + a : a;
        }
        return;
    }
    float4 a = *reinterpret_cast<const float4 *>(base);
    for (int s = 1; s < it.slices; s += 8) {
        float4 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = s + u < it.slices ? *reinterpret_cast<const float4 *>(base + (s + u) * it.n) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (s + u >= it.slices) break;
            a.x += v[u].x;
            a.y += v[u].y;
            a.z += v[u].z;
            a.w += v[u].w;
        }
    }
    if (p.from_zero) a = make_float4(0.f + a.x, 0.f + a.y, 0.f + a.z, 0.f + a.w);
    if ((reinterpret_cast<uintptr_t>(it.y) & 15) == 0) {
        *reinterpret_cast<float4 *>(it.y + i) = a;
    } else {
        it.y[i] = a.x;
        it.y[i + 1] = a.y;
        it.y[i + 2] = a.z;
        it.y[i + 3] = a.w;
    }
}

bool aligned16(const void *p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

// Cycles of a K-block of a pair's 256 x bn tile with all pairs at work: its operands, 64 KiB + bn * 256 bytes, from L2 at 57 bytes a
// cycle and pair (72 products of a BERT-base step: 8.1 TB/s).
int kb_cycles(int bn) { return (65536 + bn * 256) / 57; }

// The tensor core truncates when it adds, so the length of a chain is most of the error.  Narrow tiles have time for more drains than
// gemm_tc_body's one in 128 k, and long sums are theirs (error of X^T Y against float64, 25088 x 64 x 64: 9.0e-7 ... 9.4e-7 with
// chains of 128; one launch a product, in slices of 392 k, 8.9e-7 ... 9.1e-7).
int chain_kb(int bn) { return bn <= 128 ? 3 : kChunkKB; }

struct Planned {
    const TcGemm *g;
    int bn, kb, slices, per_slice, tiles_m, tiles_n;
    long long cost;  // cycles of a unit
};

template <int MAX>
sage_status launch_group(Context &ctx, const GroupParams<MAX> &p, int grid, size_t smem) {
    static int attr_set[64] = {0};  // per instantiation and device
    const int dev = ctx.device();
    if (dev < 0 || dev >= 64 || attr_set[dev] < (int)smem) {
        sage_status st = ctx.check_cuda(cudaFuncSetAttribute(gemm_tc_group_kernel<MAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - 1024), "gemm_tc_group shared memory attribute");
        if (st) return st;
        if (dev >= 0 && dev < 64) attr_set[dev] = 227 * 1024 - 1024;
    }
    return ctx.check_cuda(launch_dependent(ctx.pdl, ctx.stream(), 2, gemm_tc_group_kernel<MAX>, dim3(grid), dim3(64 + 32 * kEpiWarps), smem, p), "gemm_tc_group launch");
}

template <int MAX>
sage_status run_items(Context &ctx, std::vector<Planned> &plan, const std::vector<float *> &partial) {
    std::unique_ptr<GroupParams<MAX>> p(new GroupParams<MAX>());
    int units = 0, widest = 64;
    for (const Planned &x : plan) widest = std::max(widest, x.bn);
    for (size_t i = 0; i < plan.size(); ++i) {
        const Planned &x = plan[i];
        const TcGemm &g = *x.g;
        GroupItem &it = p->item[i];
        it.c = partial[i] ? partial[i] : g.c;
        it.ldc = (int)(partial[i] ? g.n : g.ldc);
        it.m = (int)g.m;
        it.n = (int)g.n;
        it.num_kb = x.kb;
        it.kb_per_slice = x.per_slice;
        it.unit0 = units;
        it.tiles_m = x.tiles_m;
        it.tiles_n = x.tiles_n;
        it.bn = (short)x.bn;
        it.chain = chain_kb(x.bn);
        bool a_blocked = true, b_blocked = true;
        if (!encode_tc_operand(g.a, BM, g.a_kmajor, &a_blocked, &it.a) || !encode_tc_operand(g.b, (unsigned)(x.bn / 2), g.b_kmajor, &b_blocked, &it.b))
            return ctx.fail(SAGE_ERR_INVALID, "gemm_tc_group: operand not addressable by TMA");
        it.flags = (short)((g.a_kmajor ? kKMajorA : 0) | (g.b_kmajor ? kKMajorB : 0) | (a_blocked ? kBlockedA : 0) | (b_blocked ? kBlockedB : 0) |
                           (it.n % 4 == 0 && it.ldc % 4 == 0 && aligned16(it.c) ? kVec : 0));
        units += x.slices * x.tiles_m * x.tiles_n;
    }
    p->count = (int)plan.size();
    p->units = units;
    p->b_bytes = widest / 2 * BK * 4;
    const int stage_bytes = 2 * kGroupABytes + 2 * p->b_bytes, staging = kEpiWarps * kStageBytesPerWarp;
    p->stages = std::min(8, (227 * 1024 - 2048 - staging) / stage_bytes);
    p->status = ctx.status_word_dev;
    const int pairs = ctx.sm_count / 2;
    return launch_group<MAX>(ctx, *p, 2 * std::min(units, pairs), (size_t)p->stages * stage_bytes + staging + 1024);
}

}  // namespace

bool gemm_tc_groupable(const TcGemm &g) {
    return gemm_tc_pairs() && !g.conv.on && g.batch == 1 && g.naux == 0 && g.epilogue.empty() && !g.row_softmax && g.c && !g.c_hi && !g.force_bn && g.m >= 1 && g.n >= 32 && g.k >= 32 &&
           g.m <= (1LL << 24) && g.n <= (1LL << 24) && g.k <= (1LL << 28) && g.m * g.n <= 0x7fffffffLL && g.ldc == g.n && g.a.nb0 * g.a.nb1 == 1 && g.b.nb0 * g.b.nb1 == 1;
}

// A CTA pair's share of the work is cut into about eight units or more, so that the pairs' ends lie within an eighth of one another
// whatever the sizes; units of fewer than kMinKB K-blocks are not worth their start.  (A ResNet-18 step: 1061 us; a quarter: 1060, a
// sixteenth: 1062, kMinKB 8: 1071, 24: 1064.)  us in a training step, one launch each and one more for the slices' sum | together:
// 72 products of BERT-base (32 x 128 tokens) 3735 | 2620, which is 797 TFLOP/s of tf32 products (the library's own GEMM: 731-760); 20 of
// ResNet-18 (128 images of 28 x 28) 335 | 90.
sage_status gemm_tc_group_run(Context &ctx, const std::vector<TcGemm> &all) {
    constexpr int kMinKB = 12, kMax = 100, kFew = 12;
    for (size_t at = 0; at < all.size(); at += kMax) {
        const size_t n = std::min(all.size() - at, (size_t)kMax);
        if (n == 1) {
            sage_status st = gemm_tc_run(ctx, all[at]);
            if (st) return st;
            continue;
        }
        std::vector<Planned> plan;
        double total = 0.0;
        const int pairs = ctx.sm_count / 2;
        for (size_t i = 0; i < n; ++i) {
            const TcGemm &g = all[at + i];
            Planned x{};
            x.g = &g;
            long long best = 0;
            for (int bn : {256, 192, 128, 64}) {
                const long long cost = (g.n + bn - 1) / bn * kb_cycles(bn);
                if (!best || cost < best) {
                    best = cost;
                    x.bn = bn;
                }
            }
            x.kb = (int)((g.k + BK - 1) / BK);
            x.tiles_m = (int)((g.m + 2 * BM - 1) / (2 * BM));
            x.tiles_n = (int)((g.n + x.bn - 1) / x.bn);
            x.cost = (long long)x.kb * kb_cycles(x.bn);
            total += (double)x.cost * x.tiles_m * x.tiles_n;
            plan.push_back(x);
        }
        const double most = total / pairs / 8.0;
        long long floats = 0;
        for (Planned &x : plan) {
            long long s = (long long)((double)x.cost / most) + 1;
            s = std::max(1LL, std::min(s, (long long)x.kb / kMinKB));
            x.per_slice = (int)(((x.kb + s - 1) / s + chain_kb(x.bn) - 1) / chain_kb(x.bn) * chain_kb(x.bn));  // whole chains
            x.slices = (x.kb + x.per_slice - 1) / x.per_slice;
            x.cost = (long long)std::min(x.per_slice, x.kb) * kb_cycles(x.bn);
            if (x.slices > 1) floats += x.slices * ((x.g->m * x.g->n + 3) / 4 * 4);
        }
        std::stable_sort(plan.begin(), plan.end(), [](const Planned &a, const Planned &b) { return a.cost > b.cost; });  // the longest first: the ends even out
        Block *scratch = floats ? ctx.allocator().alloc((size_t)floats * sizeof(float)) : nullptr;
        if (floats && !scratch)  // no room for partial results: whole K
            for (Planned &x : plan) {
                x.slices = 1;
                x.per_slice = x.kb;
            }
        std::vector<float *> partial(n, nullptr);
        std::vector<SliceItem> sums;
        long long used = 0;
        int blocks = 0;
        for (size_t i = 0; i < n; ++i) {
            const Planned &x = plan[i];
            if (x.slices == 1) continue;
            const long long mn = x.g->m * x.g->n;
            partial[i] = reinterpret_cast<float *>(scratch->ptr) + used;
            used += x.slices * ((mn + 3) / 4 * 4);
            sums.push_back(SliceItem{partial[i], x.g->c, mn, x.slices, blocks});
            blocks += (int)((mn + 1023) / 1024);
        }
        for (size_t i = 0; i < n; ++i) {
            const TcGemm &g = *plan[i].g;
            std::string label = "gemm_tc_3xtf32";
            if (ctx.verbose_names)
                label += "[" + std::to_string(g.m) + "x" + std::to_string(g.n) + "x" + std::to_string(g.k) + ",group,bn" + std::to_string(plan[i].bn) + ",slices" + std::to_string(plan[i].slices) + "]";
            if (i + 1 < n) ctx.note_part(label.c_str());
            else ctx.note_launch(ctx.verbose_names ? label.c_str() : "gemm_tc_3xtf32");
        }
        sage_status st = SAGE_OK;
        if (!ctx.dry()) st = n <= kFew ? run_items<kFew>(ctx, plan, partial) : run_items<kMax>(ctx, plan, partial);
        if (!st && !sums.empty()) {
            for (size_t i = 0; i + 1 < sums.size(); ++i) ctx.note_part("reduce_slices");
            ctx.note_launch("reduce_slices");
            if (!ctx.dry()) {
                SliceParams p;
                p.count = (int)sums.size();
                p.from_zero = ctx.opts().ref_compat;
                std::copy(sums.begin(), sums.end(), p.item);
                st = ctx.check_cuda(launch_dependent(ctx.pdl, ctx.stream(), sum_slices_group_kernel, dim3((unsigned)blocks), dim3(256), 0, p), "sum_slices_group launch");
            }
        }
        if (scratch) ctx.allocator().free(scratch);  // stream-ordered
        if (st) return st;
    }
    return SAGE_OK;
}

}  // namespace k
}  // namespace sage
