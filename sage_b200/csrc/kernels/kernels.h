// Host launchers of the hand-written (non-JIT) CUDA kernels.  Pointers are raw device
// addresses with the tensor's element offset already applied; strides are in elements.
#pragma once
#include <cstdint>
#include <memory>
#include <string>
#include <vector>

#include "../runtime/runtime.h"

namespace sage {
namespace k {

constexpr int kMaxDims = SAGE_MAX_DIMS;

struct Dims {  // extents + strides of a (sub)space, row-major order of traversal
    int ndim = 0;
    long long ext[kMaxDims] = {0};
    long long str[kMaxDims] = {0};
    long long size() const {
        long long p = 1;
        for (int i = 0; i < ndim; ++i) p *= ext[i];
        return p;
    }
};

// Operand forms of a result that its producer writes beside (or instead of) the fp32 values, for the tensor-core product
// that reads it next: tf32 planes (`hi`, lo `plane` floats further) and half-precision pieces (`h2`, lo `h2_plane` elements
// further, a scale per 64 elements).  Null = not wanted; all are laid out like the fp32 result.
struct PlaneOut {
    float *hi = nullptr;
    long long plane = 0;
    unsigned short *h2 = nullptr;
    long long h2_plane = 0;
    float *h2_scale = nullptr;
    float *h2_marked = nullptr;  // the scales again, negative where a group is wide (gemm_h2_device.inc), for a reader that asks
    bool only = false;           // (maps) the planes are all that is read: no fp32 values
};

// column_sums.cu — several [rows, cols] -> [cols] sums in one pass over all of them (src/ops/reduce.rs:258-325, kind Sum); with one
// column and a pitch of 1 the sum over a whole tensor
struct ColumnSum {
    const float *x = nullptr;
    float *y = nullptr;
    long long rows = 0, cols = 0, pitch = 0;
};
// Is this reduction of floats such a sum?
bool column_sum_of(int dtype, int kind, const void *x, const Dims &outer, const Dims &inner, void *y, ColumnSum *out);
sage_status column_sums_run(Context &ctx, const std::vector<ColumnSum> &all);

// reduce.cu — ReduceOperator / ReduceArgOperator (src/ops/reduce.rs:258-325, 372-431)
sage_status reduce(Context &ctx, int dtype, int kind, const void *x, const Dims &outer, const Dims &inner, void *y);
sage_status reduce_arg(Context &ctx, bool is_max, const float *x, const Dims &outer, long long inner_ext,
                       long long inner_str, uint32_t *y);

// rowops.cu — softmax / log_sum_exp / layer_norm over contiguous rows (src/ops/nn.rs:42-100)
sage_status softmax_rows(Context &ctx, const float *x, float *y, long long rows, long long cols, const PlaneOut &planes = PlaneOut());
// Do the kernels of these rows hold whole 64-element groups per half warp (and so write the half-precision pieces)?
bool rows_write_pieces(const float *x, long long cols);
sage_status lse_rows(Context &ctx, const float *x, float *y, long long rows, long long cols);
sage_status layernorm_rows(Context &ctx, const float *x, float *y, long long rows, long long cols, const float *gamma,
                           int gamma_stride, const float *beta, int beta_stride, float eps, const PlaneOut &planes = PlaneOut());

// index.cu — gather / scatter / strided copy (src/ops/core.rs:571-934)
sage_status gather(Context &ctx, const uint32_t *x, const long long *x_str, const uint32_t *ind, const Dims &ind_dims,
                   int axis, uint32_t *y);
sage_status scatter_add(Context &ctx, const float *x, const long long *x_str, const uint32_t *ind, const Dims &ind_dims,
                        int axis, float *y, const long long *y_str);
// y[translate(g, dims.ext, y_str)] = x[translate(g, dims.ext, dims.str)]
sage_status strided_copy(Context &ctx, const uint32_t *x, const Dims &dims, uint32_t *y, const long long *y_str);

// Uniform::compute / Normal::compute (src/ops/rand.rs:50-140) with the two 32-bit seeds given by the caller.
sage_status rand_fill(Context &ctx, bool normal, float *y, long long n, unsigned seed_x, unsigned seed_y);

// conv.cu — im2col / col2im / direct pooling (src/ops/conv.rs:143-165, 289-498)
struct Window {
    int ker_w, ker_h, stride_w, stride_h, pad_w, pad_h, dil_w, dil_h;
};
sage_status im2col(Context &ctx, const float *img, float *col, long long n, long long img_h, long long img_w,
                   long long chan, long long col_h, long long col_w, const Window &w);
// im2col writing the fp32 column tensor (`col`, row pitch K, may be null) and / or its tf32 planes
// (`hi`, lo `plane` floats further, row pitch `pitch` >= K and a multiple of 4, may be null).
sage_status im2col_planes(Context &ctx, const float *img, long long n, long long img_h, long long img_w, long long chan,
                          long long col_h, long long col_w, const Window &w, float *col, float *hi, long long plane, int pitch);
sage_status col2im(Context &ctx, const float *col, float *img, long long n, long long img_h, long long img_w,
                   long long chan, long long col_h, long long col_w, const Window &w);
// Convolutions with C <= 4: the image as tf32 planes [n, hp, wp, 4] (channels padded to 4, `pad_h` / `pad_w` zero rows /
// columns in front, the rest behind), and the filter [kh, kw, c, oc] as planes [kh * 32, oc] with row ky * 32 + kx * 4 + c.
// plane = 0: write plain fp32 instead of the two planes.
sage_status pack_small_c_image(Context &ctx, const float *img, long long n, long long h, long long w, long long c, long long hp, long long wp,
                               int pad_h, int pad_w, float *hi, long long plane);
sage_status pack_small_c_filter(Context &ctx, const float *filt, int kh, int kw, int c, int oc, float *hi, long long plane);
// The first convolution on half-precision pieces (conv_first_device.inc): the image as [n, hp, wp, 4] in pieces with a scale per image
// (wp even; `parts`: 64 words per image of scratch, 8-byte aligned), the filter as [oc / 64][kh][4][piece][64][8] with a scale per
// channel.  A negative scale: its image or channel spans more than one scale holds.
sage_status pack_first_image(Context &ctx, const float *img, long long n, long long h, long long w, long long c, long long hp, long long wp, int pad_h, int pad_w,
                             unsigned short *hi, long long plane, float *scale, unsigned *parts);
sage_status pack_first_filter(Context &ctx, const float *filt, int kh, int kw, int c, int oc, unsigned short *out, float *scale);
// The same with a map before the column matrix (`expr` over x0, an image's value) or behind the image's gradient (over x0, the gathered
// sum, and x1 ... x3, dense like the image), spliced in: C % 4 == 0 and 16-byte alignment throughout.  Results that are null are not stored.
bool long_expression(const std::string &e);  // calls a function of more than a few instructions (gemm_h2.cu)
bool cols_mappable(const void *a, const void *b, long long img_h, long long img_w, long long chan, long long col_h, long long col_w, const Window &w);
sage_status im2col_mapped(Context &ctx, const std::string &expr, const float *img, long long n, long long img_h, long long img_w, long long chan, long long col_h, long long col_w, const Window &w,
                          float *col, float *hi, long long plane, int pitch);
sage_status col2im_mapped(Context &ctx, const std::string &expr, int naux, const float *const aux[3], const float *col, float *img, float *hi, long long plane, long long n, long long img_h,
                          long long img_w, long long chan, long long col_h, long long col_w, const Window &w);
bool pool2d_writes_pieces(const float *img, long long chan, long long out_h, long long out_w);
sage_status pool2d(Context &ctx, bool is_max, const float *img, float *out, long long n, long long img_h,
                   long long img_w, long long chan, long long out_h, long long out_w, const Window &w, const PlaneOut &forms);

// gemm_simt.cu / gemm_tcgen05.cu — Gemm / GemmBatched (src/ops/gemm.rs:176-250, 338-421)
struct GemmArgs {
    bool ta, tb;
    long long m, n, k;
    const float *a;
    long long lda, stride_a;
    const float *b;
    long long ldb, stride_b;
    float *c;
    long long ldc, stride_c;
    long long batch;
};
// An operand split for 3xTF32: [2 planes (hi, lo)][batches][rows][pitch] floats, rows x cols as the
// operand lies in memory (cols contiguous), pitch = cols rounded up to 4.
struct SplitPlanes {
    Block *block = nullptr;
    float *planes = nullptr;
    int rows = 0, cols = 0, pitch = 0, batches = 0;
};
bool gemm_tc_supported(const GemmArgs &g);

// ---- the general form of the tensor-core GEMM, used by the evaluator's fused GEMM operator.
// A split operand as the tensor core reads it: `rows` x `cols` with cols contiguous, rows `ld` floats
// apart, batch index = b1 * nb0 + b0 at b0 * sb0 + b1 * sb1 floats.  `hi` points at the first
// element of the tf32 high parts; the low parts lie `plane` floats further.  hi must be 16-byte
// aligned and ld, sb0, sb1, plane multiples of 4 (TMA strides are multiples of 16 bytes).
struct TcOperand {
    const float *hi = nullptr;
    long long plane = 0, ld = 0;
    long long rows = 0, cols = 0;
    long long nb0 = 1, nb1 = 1, sb0 = 0, sb1 = 0;
    bool bcast = false;  // one matrix shared by every batch of the GEMM (nb0 = nb1 = 1)
};
bool tc_operand_ok(const TcOperand &o);
// An extra operand of the epilogue expression: element (batch, row, col) of the output reads
// ptr[b0 * s0 + b1 * s1 + row * sr + col * sc] with the output's batch decomposition; sc is 0 or 1.
struct TcAuxArg {
    const float *ptr = nullptr;
    long long s0 = 0, s1 = 0, sr = 0;
    int sc = 0;
};
// Implicit-GEMM convolution: A (one row per output pixel, K over (tap, channel)) is read by im2col-mode
// TMA from the tf32 planes of a contiguous NHWC image; needs C % 32 == 0.
struct TcConv {
    bool on = false;
    const float *hi = nullptr;  // hi plane of the image; lo `plane` floats further
    long long plane = 0;
    long long n = 0, h = 0, w = 0, c = 0, out_h = 0, out_w = 0;
    Window win{};
    // Element strides between pixels, rows and images; 0 = the dense NHWC ones (c, w * c, h * w * c).  A pixel stride
    // below c makes neighbouring pixels overlap (the C <= 4 layout: 32-float windows 4 * stride floats apart).
    long long sw = 0, sh = 0, sn = 0;
    bool raw = false;  // `hi` points at plain fp32 (no lo plane): the kernel splits each tile in shared memory
};
struct TcGemm {
    TcConv conv;             // when conv.on, `a` is ignored
    bool a_kmajor = true, b_kmajor = false;  // is K the contiguous axis of the operand as stored
    long long m = 0, n = 0, k = 0, batch = 1;
    TcOperand a, b;
    float *c = nullptr;      // fp32 result (may be null when only planes are wanted)
    float *c_hi = nullptr;   // hi plane of the result, laid out like c (may be null)
    long long c_plane = 0;   // floats from the hi to the lo plane
    long long ldc = 0, sc0 = 0, sc1 = 0, nbc0 = 1;  // result (batch, row, col) at b0 * sc0 + b1 * sc1 + row * ldc + col
    int naux = 0;
    TcAuxArg aux[3];
    std::string epilogue;    // C expression over x0 (the product) and x1..x3 (aux); empty = x0
    bool row_softmax = false;  // store softmax over each output row of the expression; needs n <= 256 (one tile per row)
    int force_bn = 0;          // tile width chosen by the caller (64 / 128 / 192 / 256); 0 = the launcher's own choice
};
bool gemm_tc_shape_ok(long long m, long long n, long long k, long long batch);
sage_status gemm_tc_run(Context &ctx, const TcGemm &g);
// How many K slices gemm_tc_run would cut this product into (0 = none).  Only products without an epilogue are
// cut; a caller with an epilogue may ask for the plain product and apply the epilogue to the sum itself.
int gemm_tc_split_plan(Context &ctx, const TcGemm &g);
// The K slices' partial products alone, m * n floats apart, in memory of `*partial` (whoever asked frees it), and how many there are.
// Without room for them: SAGE_OK and no memory.
sage_status gemm_tc_partials(Context &ctx, const TcGemm &g, Block **partial, int *slices);
// gemm_group.cu: may this product run beside others in one launch; and that launch (several, where there are very many).
bool gemm_tc_groupable(const TcGemm &g);
sage_status gemm_tc_group_run(Context &ctx, const std::vector<TcGemm> &all);
// Work that nothing of a program reads, put off until launches of one kind can be made together.  `held` keeps alive what it
// reads and writes.
struct LeafBatch {
    std::vector<ColumnSum> column_sums;
    std::vector<TcGemm> products;
    std::vector<std::shared_ptr<void>> held, held_by_sums;
    // Of the operands, what would be gone by now had each launch been made at once: the products' and the sums' kinds run when it passes the limit.
    size_t own_bytes = 0, own_bytes_of_sums = 0;
    static constexpr size_t kMaxOwnBytes = (size_t)128 << 20;
    sage_status status = 0;  // of the launches so far
    bool empty() const { return column_sums.empty() && products.empty(); }
    sage_status run(Context &ctx);  // ... and empties it
    sage_status run_products(Context &ctx);
    sage_status run_sums(Context &ctx);
};
// hi/lo split of `n` consecutive floats into planes laid out like the source (dst_hi[i], dst_hi[plane + i]).
sage_status split_tf32_flat(Context &ctx, const float *src, long long n, float *dst_hi, long long plane);
// hi/lo split of a strided 4-level view (b1, b0, row, col) into compact planes owned by `out`.
struct SplitView {
    long long nb1 = 1, nb0 = 1, rows = 0, cols = 0;
    long long sb1 = 0, sb0 = 0, ld = 0, col_stride = 1;
};
sage_status split_tf32_view(Context &ctx, const float *src, const SplitView &v, SplitPlanes *out);
// ---- gemm_h2.cu: the product over two half-precision pieces per operand (kernels/gemm_h2_device.inc states the
// representation).  Both operands are read with K contiguous: `rows` x `k`, rows `ld` elements apart, batch index =
// b1 * nb0 + b0 at b0 * sb0 + b1 * sb1.  `hi` points at the first hi piece, the lo pieces lie `plane` elements further.
// Operand A has a scale per row and 64 k (`scale` + b0 * s_b0 + b1 * s_b1 + row * s_row + k / 64), operand B one per row
// (`scale` + batch * s_b0 + row) and a factor to it per 64 rows and 64 k (`ratio`: [batch][row / 64][k / 64]).  hi must be 16-byte aligned and ld, sb0, sb1, plane multiples of 8.
struct H2Operand {
    const unsigned short *hi = nullptr;
    long long plane = 0, ld = 0, rows = 0;
    long long nb0 = 1, nb1 = 1, sb0 = 0, sb1 = 0;
    bool bcast = false;
    const float *scale = nullptr;
    long long s_row = 0, s_b0 = 0, s_b1 = 0;
    const float *ratio = nullptr;
    const float *marked = nullptr;               // of a small convolution's operands: A's scales or B's factors with the wide ones negative
    const unsigned long long *columns = nullptr;
};
struct H2Gemm {
    bool conv = false;        // A is the im2col of a contiguous NHWC image (a.hi, a.plane, a.scale) with C % 64 == 0
    long long img_n = 0, img_h = 0, img_w = 0, img_c = 0, out_h = 0, out_w = 0;
    Window win{};
    long long m = 0, n = 0, k = 0, batch = 1;
    H2Operand a, b;
    float *c = nullptr, *c_hi = nullptr;  // result as fp32 and / or as tf32 planes, as in TcGemm
    long long c_plane = 0;
    unsigned short *h_hi = nullptr;       // ... and / or in half-precision pieces: needs n, ldc, sc0, sc1 multiples of 64
    long long h_plane = 0;
    float *h_scale = nullptr;
    float *h_marked = nullptr;
    const float *a_f32 = nullptr, *b_f32 = nullptr;  // a small convolution (conv_h2_small): what the pieces were made from, the filter at
    long long b_k = 0, b_n = 0;                      // [k * b_k + column * b_n]
    long long ldc = 0, sc0 = 0, sc1 = 0, nbc0 = 1;
    int naux = 0;
    TcAuxArg aux[3];
    std::string epilogue;
};
sage_status gemm_h2_run(Context &ctx, const H2Gemm &g);
// The first convolution.  g: result and epilogue, img_n / out_h / out_w, n = output channels; the operands as pack_first_* lay them.
struct FirstConv {
    const unsigned short *img = nullptr, *filter = nullptr;
    long long img_plane = 0, hp = 0, wp = 0;
    int kh = 0, dil_h = 1, stride_h = 1;
    const float *img_f32 = nullptr, *filter_f32 = nullptr;  // what they were made from, contiguous
    long long img_h = 0, img_w = 0;
    int chan = 0, kw = 0, pad_h = 0, pad_w = 0;
    const float *img_scale = nullptr, *filter_scale = nullptr;
};
bool conv_first_ok(int kh, int stride_w, long long out_w);
sage_status conv_first_run(Context &ctx, const H2Gemm &g, const FirstConv &f);
// The whole product of plain fp32 operands.  With `scratch` (gemm_h2_scratch_bytes of device memory, 256-byte aligned)
// nothing is taken from the allocator and K is not cut.
size_t gemm_h2_scratch_bytes(const GemmArgs &g);
sage_status gemm_h2(Context &ctx, const GemmArgs &g, void *scratch = nullptr);
bool conv_h2_ok(const H2Gemm &g);
// Images below 128 KiB (of fp32) are read through tiled boxes, and their wide groups worked out in fp32: both operands' pieces come
// `marked`.
inline bool conv_h2_small(long long n, long long h, long long w, long long c) { return n * h * w * c * 4 < 131072; }
// Pieces of `n` consecutive floats (a multiple of 64), laid out like the source, a scale per 64.
sage_status split_h2_flat(Context &ctx, const float *src, long long n, unsigned short *hi, long long plane, float *scale, float *marked = nullptr);
// Pieces of a strided view (b1, b0, row, col) gathered with its columns contiguous: [batch][rows][pitch], pitch = cols
// rounded up to 8.  `whole_rows`: one scale per row and factors (operand B) instead of one per 64 columns.  `mark`: with
// `marked`, A's scales or B's factors again with the wide ones negative, and of B `columns`, which of a block's 64 are wide.
struct H2Split {
    Block *block = nullptr;
    unsigned short *hi = nullptr;
    float *scale = nullptr, *ratio = nullptr;
    float *marked = nullptr;
    unsigned long long *columns = nullptr;
    long long plane = 0, pitch = 0;
};
size_t split_h2_bytes(long long batches, long long rows, long long cols, bool whole_rows);
sage_status split_h2_view(Context &ctx, const float *src, const SplitView &v, bool whole_rows, H2Split *out, bool mark = false);
// Operand B straight into memory the caller laid out: rows of `out->pitch` at out->hi / out->hi + out->plane, out->scale.
sage_status split_h2_rows_at(Context &ctx, const float *src, const SplitView &v, const H2Split &out);
H2Operand h2_operand(const H2Split &s, long long batches, long long rows, long long cols, bool whole_rows);

// Fused attention: O[batch] = softmax_rows(f(Q[batch] K[batch]^T)) V[batch] in one launch (kernels/attn_tc_device.inc), on
// half-precision pieces.  Q is lq x d, K and V are lk x d per batch, head columns contiguous, every row inside one group:
// its scale is scale[((s_off + b0 * s_sb0 + b1 * s_sb1) >> s_shift) + row * s_row].
// `epilogue` is f over x0 (the score) and x1.. (aux, addressed like a GEMM epilogue operand of the lq x lk score
// matrix, batch cut by `nbe0`).  The result goes to o and / or the forms in `out` like a GEMM's (pieces: d = 64).  d <= 64.
struct AttnOperand {
    const unsigned short *hi = nullptr;
    long long plane = 0, ld = 0, nb0 = 1, nb1 = 1, sb0 = 0, sb1 = 0;
    const float *scale = nullptr;
    long long s_off = 0, s_sb0 = 0, s_sb1 = 0, s_row = 0;
    int s_shift = 0;
};
struct TcAttn {
    long long lq = 0, lk = 0, d = 0, batch = 1;
    AttnOperand q, k, v;
    float *o = nullptr;
    PlaneOut out;
    long long ldo = 0, so0 = 0, so1 = 0, nbo0 = 1;
    int naux = 0;
    TcAuxArg aux[3];
    long long nbe0 = 1;
    std::string epilogue;  // empty = x0
};
bool attention_tc_shape_ok(long long lq, long long lk, long long d, long long batch);
sage_status attention_tc_run(Context &ctx, const TcAttn &a);
// Launches a kernel whose bounded wait runs out (nothing arrives on its barrier): ~1 s, then status bit 0x140.
sage_status bounded_wait_selftest(Context &ctx);
sage_status gemm_simt(Context &ctx, const GemmArgs &g);
// Returns SAGE_ERR_UNSUPPORTED when the shape/alignment cannot go through TMA; the caller
// then uses gemm_simt.
sage_status gemm_tcgen05(Context &ctx, const GemmArgs &g);
sage_status gemm(Context &ctx, const GemmArgs &g);  // picks per ctx.opts().gemm_backend

// optim.cu — Sgd::update / Adam::update (src/optim.rs:42-94, 125-178), many parameters per launch.
// A slot: parameter `p` (n contiguous floats, updated in place), gradient `g`, Adam's moments `m`, `v`
// (updated in place; null for Sgd), and optionally the parameter's whole-storage tf32 planes (`hi`, lo
// `plane` floats further) which receive the split of the new value.  `first` = this parameter's first
// update: Adam stores zero moments then.  `vec` is filled in by the launcher.
constexpr int kOptSlots = 32;
struct OptSlot {
    float *p = nullptr;
    const float *g = nullptr;
    float *m = nullptr, *v = nullptr;
    float *hi = nullptr;
    long long plane = 0, n = 0;
    int first = 0, vec = 0;
};
struct OptSgd {
    float lr = 0.f, weight_decay = 0.f;
};
struct OptAdam {
    float lr = 0.f, beta1 = 0.9f, beta2 = 0.999f, one_minus_beta1 = 0.f, one_minus_beta2 = 0.f, eps = 1e-08f, weight_decay = 0.f;
    float corr1 = 1.f, corr2 = 1.f;  // -(beta1 ^ t) + 1 and -(beta2 ^ t) + 1 for this step's t
};
sage_status sgd_update(Context &ctx, const OptSlot *slots, int count, const OptSgd &k);
sage_status adam_update(Context &ctx, const OptSlot *slots, int count, const OptAdam &k);

}  // namespace k
}  // namespace sage
