// Convolution building blocks.  Reference: src/ops/conv.rs — conv_size :47-59, conv_2d :61-96,
// avg_pool_2d / max_pool_2d :143-165, batch_norm_2d :167-185, im2col :188-226 + kernel :289-374,
// col2im :229-264 + kernel :404-498.  Images are NHWC, filters [KH,KW,C,OC]; every two-element
// parameter is ordered [w, h].
#include "graph.h"

namespace sage {
using namespace ops;

static k::Window window(Pair ker, Pair stride, Pair pad, Pair dil) {
    return k::Window{(int)ker.w, (int)ker.h, (int)stride.w, (int)stride.h, (int)pad.w, (int)pad.h, (int)dil.w, (int)dil.h};
}

static long long conv_size(long long size, long long ker, long long stride, long long pad, long long dil) {
    return (size + 2 * pad - dil * (ker - 1) - 1) / stride + 1;
}

sage_status storage_planes_attach(Context &ctx, Storage &st);  // ops_gemm.cc

struct Im2colOp : Operator {
    Pair ker, stride, pad, dil, col;
    std::string pre;  // C expression over x0 that every value of the image goes through first (a map before the column matrix)
    MapCache maps;
    const char *name() const override { return "im2col"; }
    std::vector<Var> grad(const std::vector<Var> &x, const Var &, const Var &gy) override {
        return {col2im(gy, Pair{x[0].extent(2), x[0].extent(1)}, ker, stride, pad, dil)};
    }
    sage_status compute(const std::vector<Tensor> &x, Context &ctx, Tensor *y) override {
        const bool emit = ctx.hint_emit_planes && emits_planes(), only = emit && ctx.hint_planes_only;
        ctx.hint_emit_planes = ctx.hint_emit_h2 = ctx.hint_planes_only = false;
        sage_status st = Tensor::uninit(ctx, out, y);
        if (st) return st;
        const Array &e = x[0].desc.shape.extents;
        Tensor image = x[0];
        const bool spliced = !pre.empty() && k::cols_mappable(image.ptr(), y->ptr(), e[1], e[2], e[3], col.h, col.w, window(ker, stride, pad, dil));
        if (!pre.empty() && !spliced) {  // an image off the 16-byte grid: the map by itself
            st = Tensor::uninit(ctx, x[0].desc.pristine(), &image);
            if (st) return st;
            st = map_launch(ctx, pre, {MapOperand{SAGE_F32, x[0].ptr(), x[0].dims()}}, SAGE_F32, image.ptr(), (int)e.size(), e.data(), &maps);
            if (st) return st;
        }
        if (!emit && spliced)
            return k::im2col_mapped(ctx, pre, (const float *)x[0].ptr(), e[0], e[1], e[2], e[3], col.h, col.w, window(ker, stride, pad, dil), (float *)y->ptr(), nullptr, 0, 0);
        if (!emit)
            return k::im2col(ctx, (const float *)image.ptr(), (float *)y->ptr(), e[0], e[1], e[2], e[3], col.h, col.w, window(ker, stride, pad, dil));
        st = storage_planes_attach(ctx, *y->data);
        if (st) return st;
        const SplitCache &c = *y->data->split;
        y->data->planes_only = only;
        if (spliced)
            return k::im2col_mapped(ctx, pre, (const float *)x[0].ptr(), e[0], e[1], e[2], e[3], col.h, col.w, window(ker, stride, pad, dil), only ? nullptr : (float *)y->ptr(),
                                    c.planes.planes, c.plane, (int)(ker.h * ker.w * e[3]));
        return k::im2col_planes(ctx, (const float *)image.ptr(), e[0], e[1], e[2], e[3], col.h, col.w, window(ker, stride, pad, dil), only ? nullptr : (float *)y->ptr(), c.planes.planes, c.plane,
                                (int)(ker.h * ker.w * e[3]));
    }
    // the planes lie like the result, whole 16-byte pieces at a time
    bool emits_planes() const { return in[0].shape.extents[3] % 4 == 0 && ker.h * ker.w * in[0].shape.extents[3] <= 0x7fffffffLL; }
};
// Does the column matrix come with its tf32 planes when a product reads it (the forward and the weight gradient of a convolution in a
// training program)?  Split by a pass of their own they were 19 launches of a ResNet-18 step.
bool im2col_op_emits_planes(const Operator &op) {
    const Im2colOp *o = dynamic_cast<const Im2colOp *>(&op);
    return o && o->emits_planes();
}

bool im2col_params(const Operator &op, k::Window *w, long long dims[6]) {
    const Im2colOp *o = dynamic_cast<const Im2colOp *>(&op);
    if (!o || !o->pre.empty() || o->in[0].dtype != SAGE_F32 || !o->in[0].shape.has_default_strides()) return false;
    *w = window(o->ker, o->stride, o->pad, o->dil);
    const Array &e = o->in[0].shape.extents;
    dims[0] = e[0];
    dims[1] = e[1];
    dims[2] = e[2];
    dims[3] = e[3];
    dims[4] = o->col.h;
    dims[5] = o->col.w;
    return true;
}

struct Col2imOp : Operator {
    Pair img, ker, stride, pad, dil;
    std::string post;  // C expression over x0, a value of the image, and x1 ... (inputs 1 ..., laid out like it): the map that follows
    MapCache maps;
    const char *name() const override { return "col2im"; }
    std::vector<Var> grad(const std::vector<Var> &, const Var &, const Var &gy) override {
        return {im2col(gy, ker, stride, pad, dil)};
    }
    sage_status compute(const std::vector<Tensor> &x, Context &ctx, Tensor *y) override {
        const bool emit = ctx.hint_emit_planes && !post.empty(), only = emit && ctx.hint_planes_only;
        ctx.hint_emit_planes = ctx.hint_emit_h2 = ctx.hint_planes_only = false;
        sage_status st = Tensor::uninit(ctx, out, y);
        if (st) return st;
        const Array &e = x[0].desc.shape.extents;  // [N, col_h, col_w, KH, KW, C]
        if (!post.empty()) {
            float *hi = nullptr;
            long long plane = 0;
            if (emit) {
                st = storage_planes_attach(ctx, *y->data);
                if (st) return st;
                hi = y->data->split->planes.planes + y->desc.shape.offset;
                plane = y->data->split->plane;
                y->data->planes_only = only;
            }
            const float *aux[3] = {nullptr, nullptr, nullptr};
            bool aligned = k::cols_mappable(x[0].ptr(), y->ptr(), img.h, img.w, e[5], e[1], e[2], window(ker, stride, pad, dil));
            for (size_t i = 1; i < x.size(); ++i) {
                aux[i - 1] = (const float *)x[i].ptr();
                aligned = aligned && k::cols_mappable(aux[i - 1], nullptr, img.h, img.w, e[5], e[1], e[2], window(ker, stride, pad, dil));
            }
            if (!aligned) {  // an operand off the 16-byte grid: the map by itself
                Tensor sum;
                st = Tensor::uninit(ctx, out, &sum);
                if (!st) st = k::col2im(ctx, (const float *)x[0].ptr(), (float *)sum.ptr(), e[0], img.h, img.w, e[5], e[1], e[2], window(ker, stride, pad, dil));
                if (st) return st;
                std::vector<MapOperand> operands = {MapOperand{SAGE_F32, sum.ptr(), sum.dims()}};
                for (size_t i = 1; i < x.size(); ++i) operands.push_back(MapOperand{SAGE_F32, x[i].ptr(), x[i].dims()});
                y->data->planes_only = false;
                k::PlaneOut forms;
                forms.hi = hi;
                forms.plane = plane;
                return map_launch(ctx, post, operands, SAGE_F32, y->ptr(), out.shape.rank(), out.shape.extents.data(), &maps, forms);
            }
            return k::col2im_mapped(ctx, post, (int)x.size() - 1, aux, (const float *)x[0].ptr(), only ? nullptr : (float *)y->ptr(), hi, plane, e[0], img.h, img.w, e[5], e[1], e[2],
                                    window(ker, stride, pad, dil));
        }
        return k::col2im(ctx, (const float *)x[0].ptr(), (float *)y->ptr(), e[0], img.h, img.w, e[5], e[1], e[2],
                         window(ker, stride, pad, dil));
    }
};

// A map of one operand before a column matrix, as part of it: null where the operand is not laid out like the image or the kernel does not
// take four channels at a time.  (An operand's description does not show every start: a reshaped slice may lie off the 16-byte grid all
// the same, and the map is then worked out by itself.)
std::shared_ptr<Operator> im2col_with_map(const Operator &op, const Operator &map, const std::string &expr) {
    const Im2colOp *o = dynamic_cast<const Im2colOp *>(&op);
    if (!o || !o->pre.empty() || map.in.size() != 1 || k::long_expression(expr)) return nullptr;  // (it is worked out for every tap)
    const TensorDesc &src = map.in[0];
    const Array &e = o->in[0].shape.extents;
    if (src.dtype != SAGE_F32 || src.shape.extents != e || !src.shape.has_default_strides() || src.shape.offset % 4) return nullptr;
    if (!k::cols_mappable(nullptr, nullptr, e[1], e[2], e[3], o->col.h, o->col.w, window(o->ker, o->stride, o->pad, o->dil)) || e[0] * o->col.h * o->col.w > (1LL << 29)) return nullptr;
    auto c = std::make_shared<Im2colOp>(*o);
    c->pre = expr;
    c->in = {src};
    return c;
}
// The map `expr` over (the gathered image, aux ...), as part of the gather.
std::shared_ptr<Operator> col2im_with_map(const Operator &op, const std::string &expr, const std::vector<TensorDesc> &aux, const TensorDesc &out) {
    const Col2imOp *o = dynamic_cast<const Col2imOp *>(&op);
    if (!o || !o->post.empty() || aux.size() > 3 || out.dtype != SAGE_F32 || out.shape.size() != o->out.shape.size()) return nullptr;
    const Array &e = o->in[0].shape.extents;
    if (!o->in[0].shape.has_default_strides() || o->in[0].shape.offset % 4 || !k::cols_mappable(nullptr, nullptr, o->img.h, o->img.w, e[5], e[1], e[2], window(o->ker, o->stride, o->pad, o->dil))) return nullptr;
    for (const TensorDesc &a : aux)
        if (a.dtype != SAGE_F32 || a.shape.extents != out.shape.extents || !a.shape.has_default_strides() || a.shape.offset % 4) return nullptr;
    auto c = std::make_shared<Col2imOp>(*o);
    c->post = expr;
    c->in.resize(1);
    for (const TensorDesc &a : aux) c->in.push_back(a);
    c->out = out.pristine();
    return c;
}
bool col2im_op_emits_planes(const Operator &op) {
    const Col2imOp *o = dynamic_cast<const Col2imOp *>(&op);
    return o && !o->post.empty();
}
bool is_col2im_op(const Operator &op) {
    const Col2imOp *o = dynamic_cast<const Col2imOp *>(&op);
    return o && o->post.empty();
}

Var ops::im2col(const Var &x0, Pair ker, Pair stride, Pair pad, Pair dil) {
    Var x = x0.organize();
    if (x.rank() != 4) shape_fail("im2col: input must be [N,H,W,C]");
    if (x.dtype() != SAGE_F32) shape_fail("im2col: input must be float");
    Pair col{conv_size(x.extent(2), ker.w, stride.w, pad.w, dil.w), conv_size(x.extent(1), ker.h, stride.h, pad.h, dil.h)};
    if (col.w <= 0 || col.h <= 0) shape_fail("im2col: window larger than the padded image");
    auto op = std::make_shared<Im2colOp>();
    op->ker = ker;
    op->stride = stride;
    op->pad = pad;
    op->dil = dil;
    op->col = col;
    op->in = {x.desc};
    op->out = TensorDesc(Array{x.extent(0), col.h, col.w, ker.h, ker.w, x.extent(3)}, x.dtype());
    return Var::from_op(op, {x});
}

Var ops::col2im(const Var &x0, Pair img, Pair ker, Pair stride, Pair pad, Pair dil) {
    Var x = x0.organize();
    if (x.rank() != 6) shape_fail("col2im: input must be [N,OH,OW,KH,KW,C]");
    auto op = std::make_shared<Col2imOp>();
    op->img = img;
    op->ker = ker;
    op->stride = stride;
    op->pad = pad;
    op->dil = dil;
    op->in = {x.desc};
    op->out = TensorDesc(Array{x.extent(0), img.h, img.w, x.extent(5)}, x.dtype());
    return Var::from_op(op, {x});
}

Var ops::conv_2d(const Var &x, const Var &filter, Pair stride, Pair pad, Pair dil) {  // conv.rs:61-96
    if (filter.rank() != 4) shape_fail("conv_2d: filter must be [KH,KW,C,OC]");
    const long long kh = filter.extent(0), kw = filter.extent(1), cin = filter.extent(2), cout = filter.extent(3);
    Var col = im2col(x, Pair{kw, kh}, stride, pad, dil);
    if (col.extent(5) != cin) shape_fail("conv_2d: channel mismatch");
    const long long n = col.extent(0), ch = col.extent(1), cw = col.extent(2);
    Var c2 = view(col, {n * ch * cw, kh * kw * cin});
    Var f2 = view(filter, {kh * kw * cin, cout});
    return view(matmul(c2, f2), {n, ch, cw, cout});
}

sage_status storage_h2_attach(Context &ctx, Storage &st, bool wide);  // ops_gemm.cc

// Pooling as one kernel: the same value as im2col followed by mean / max over [KH,KW], without the
// KH*KW-times larger intermediate.
struct Pool2dOp : Operator {
    bool is_max;
    Pair ker, stride, pad, dil;
    const char *name() const override { return is_max ? "max_pool2d" : "avg_pool2d"; }
    std::vector<Var> grad(const std::vector<Var> &, const Var &, const Var &) override {
        shape_fail("pool2d composite is not differentiated; grad walks the decomposed graph");
    }
    sage_status compute(const std::vector<Tensor> &x, Context &ctx, Tensor *y) override {
        const Array &e = x[0].desc.shape.extents;
        const Array &o = out.shape.extents;
        // an image off the 16-byte grid takes the kernel without pieces; its reader splits the result
        const bool emit_h2 = ctx.hint_emit_h2 && k::pool2d_writes_pieces((const float *)x[0].ptr(), e[3], o[1], o[2]);
        const bool only = emit_h2 && !ctx.hint_emit_planes && ctx.hint_planes_only, wide = ctx.hint_mark_wide;
        ctx.hint_emit_planes = ctx.hint_emit_h2 = ctx.hint_planes_only = ctx.hint_mark_wide = false;
        sage_status st = Tensor::uninit(ctx, out, y);
        if (st) return st;
        k::PlaneOut forms;
        if (emit_h2) {
            st = storage_h2_attach(ctx, *y->data, wide);
            if (st) return st;
            forms.h2 = y->data->h2->pieces.hi;
            forms.h2_plane = y->data->h2->pieces.plane;
            forms.h2_scale = y->data->h2->pieces.scale;
            forms.h2_marked = y->data->h2->pieces.marked;
            y->data->planes_only = only;
        }
        return k::pool2d(ctx, is_max, (const float *)x[0].ptr(), only ? nullptr : (float *)y->ptr(), e[0], e[1], e[2], e[3], o[1], o[2],
                         window(ker, stride, pad, dil), forms);
    }
};
bool pool_op_emits_h2(const Operator &op) {
    const Pool2dOp *p = dynamic_cast<const Pool2dOp *>(&op);
    return p && k::pool2d_writes_pieces(nullptr, p->out.shape.extents[3], p->out.shape.extents[1], p->out.shape.extents[2]);
}

static Var pool(const Var &x, Pair ker, Pair stride, Pair pad, Pair dil, bool is_max) {
    Var col = im2col(x, ker, stride, pad, dil);
    Var y = is_max ? reduce(col, {3, 4}, false, RMax) : mean(col, {3, 4}, false);
    const Var &src = col.origin->inputs[0];  // the organized image
    auto op = std::make_shared<Pool2dOp>();
    op->is_max = is_max;
    op->ker = ker;
    op->stride = stride;
    op->pad = pad;
    op->dil = dil;
    op->in = {src.desc};
    op->out = y.desc.pristine();
    y.origin->composite.reset(new Composite{op, {src}});
    return y;
}

Var ops::avg_pool_2d(const Var &x, Pair ker, Pair stride, Pair pad, Pair dil) { return pool(x, ker, stride, pad, dil, false); }
Var ops::max_pool_2d(const Var &x, Pair ker, Pair stride, Pair pad, Pair dil) { return pool(x, ker, stride, pad, dil, true); }

Var ops::batch_norm_2d(const Var &x, const Var &gamma, const Var &beta, const Var &mean_, const Var &var_, float eps) {
    Var xc = div(sub(x, mean_), unary_map(add(var_, eps), Sqrt));  // conv.rs:181-184
    return add(mul(gamma, xc), beta);
}

}  // namespace sage
