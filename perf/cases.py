"""The work this framework is used for, as cases that can be timed and compared: whole forward passes of the
bundled models, whole training steps, the contraction entry point and fused row graphs, each through the
public Python package, from single small requests to batches that fill the GPU.

  listed()            the cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) the inputs, weights and handles of a program that is about to run the case
  run(state)          one pass; its results are views of device memory, valid until the next pass
  work(case)          the bytes and operations one pass cannot do without
  tolerance(case)     how far two correct implementations at the same precision may differ
"""
import ctypes
import math

import numpy as np
import torch

import sage_b200 as S

VOCAB, MAX_TOKENS = 30522, 512
L = ctypes.c_int64


def bert(name, batch, seq, layers=12, width=768, gelu=False, padded=False):
    return {"name": name, "kind": "bert", "batch": batch, "seq": seq, "layers": layers, "width": width, "gelu": gelu, "padded": padded}


def listed():
    return [
        # One short request to an encoder service: the smallest forward pass, latency and launches.
        bert("bert_base_b1_l24", 1, 24),
        # A handful of requests of an odd length, padded to the longest, with the GELU feed-forward of published encoders.
        bert("bert_base_b6_l77_gelu", 6, 77, gelu=True, padded=True),
        # The framework's headline: the base encoder on 32 sequences of 128 tokens.
        bert("bert_base_b32_l128", 32, 128),
        # Offline encoding of long documents with a large encoder, ragged padding: the largest forward pass.
        bert("bert_large_b32_l512", 32, 512, layers=24, width=1024, padded=True),
        # One picture to an image classifier.
        {"name": "resnet18_b1_224", "kind": "resnet", "batch": 1, "size": 224, "channels": 3},
        # Bulk classification.
        {"name": "resnet18_b256_224", "kind": "resnet", "batch": 256, "size": 224, "channels": 3},
        # Fine-tuning the base encoder: loss, all gradients and an Adam update.
        {"name": "train_bert_base_b32_l128", "kind": "train_bert", "batch": 32, "seq": 128, "layers": 12, "width": 768},
        # The training example: ResNet-18 on 28 x 28 grey pictures, batch 128, Adam.
        {"name": "train_resnet18_b128_28", "kind": "train_resnet", "batch": 128, "size": 28, "channels": 1},
        # A large square product through the op-level entry point, operands as the caller holds them (plain fp32).
        {"name": "gemm_4096", "kind": "gemm", "m": 4096, "n": 4096, "k": 4096, "batch": 1, "ta": False, "tb": False},
        # A small product no dimension of which is a multiple of anything, its second operand transposed.
        {"name": "gemm_997x1234x777_t", "kind": "gemm", "m": 997, "n": 1234, "k": 777, "batch": 1, "ta": False, "tb": True},
        # A loss over a fused elementwise chain and its gradient (maps, row reductions, gather / scatter): small, and
        # well beyond the caches.
        {"name": "cross_entropy_grad_1024x1024", "kind": "rows", "op": "cross_entropy_grad", "rows": 1024, "cols": 1024},
        {"name": "cross_entropy_grad_16384x4096", "kind": "rows", "op": "cross_entropy_grad", "rows": 16384, "cols": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bert", "bert", "resnet", "train_bert", "train_resnet", "gemm", "gemm", "rows"])
    while True:
        if kind == "bert":
            c = {"kind": kind, "batch": _log_int(rng, 1, 128), "seq": _log_int(rng, 8, 512), "layers": rng.choice([4, 6, 12, 24]),
                 "width": rng.choice([256, 512, 768, 1024]), "gelu": rng.random() < 0.5, "padded": rng.random() < 0.5}
            most = work(listed()[3])["flops"]
        elif kind == "resnet":
            c = {"kind": kind, "batch": _log_int(rng, 1, 256), "size": rng.randint(48, 224), "channels": rng.choice([1, 3])}
            most = work(listed()[5])["flops"]
        elif kind == "train_bert":
            c = {"kind": kind, "batch": _log_int(rng, 1, 64), "seq": _log_int(rng, 16, 256), "layers": rng.choice([2, 4, 12]), "width": rng.choice([256, 512, 768])}
            most = work(listed()[6])["flops"]
        elif kind == "train_resnet":
            c = {"kind": kind, "batch": _log_int(rng, 4, 256), "size": rng.randint(28, 64), "channels": rng.choice([1, 3])}
            most = 8 * work(listed()[7])["flops"]
        elif kind == "gemm":
            c = {"kind": kind, "m": _log_int(rng, 16, 8192), "n": _log_int(rng, 16, 8192), "k": _log_int(rng, 16, 8192),
                 "batch": _log_int(rng, 1, 64) if rng.random() < 0.4 else 1, "ta": rng.random() < 0.3, "tb": rng.random() < 0.3}
            if rng.random() < 0.5:  # layers come in round sizes as often as not
                c.update({d: (c[d] + 15) // 16 * 16 for d in "mnk"})
            most = 4 * work(listed()[8])["flops"]
            if c["batch"] * (c["m"] * c["k"] + c["k"] * c["n"] + c["m"] * c["n"]) > 1 << 28:
                continue
        else:
            c = {"kind": kind, "op": rng.choice(["cross_entropy_grad", "softmax", "layer_norm", "log_sum_exp"]), "rows": _log_int(rng, 64, 32768),
                 "cols": _log_int(rng, 64, 16384)}
            most = float(1 << 26) * 40
        if work(c)["flops"] <= most:
            return c


# ------------------------------------------------------------------------------------------ inputs
class _Program:
    """What a program keeps between passes.  One context (one stream, one pool) serves the whole process."""
    context = None

    def __init__(self):
        if _Program.context is None:
            _Program.context = S.Context(0)
        self.ctx, self.views, self.owned = _Program.context, {}, []

    def __del__(self):  # a program that ends gives back its compiled graphs and buffers
        try:
            for t in self.owned:
                t.release()
            self.ctx.clear()
            self.ctx.drop_programs()
        except Exception:
            pass


class _DeviceArray:
    def __init__(self, ptr, shape, strides):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "strides": strides, "typestr": "<f4", "version": 3}


def _view(state, ptr, shape, strides=None):
    """Device memory as a tensor (no copy); the wrapper for an address is made once."""
    key = (ptr, shape, strides)
    t = state.views.get(key)
    if t is None:
        t = torch.as_tensor(_DeviceArray(ptr, shape, strides), device="cuda")
        if len(state.views) > 4096:
            state.views.clear()
        state.views[key] = t
    return t


def _result(state, v):
    """An evaluated (or data) variable as a tensor over its own memory."""
    ptr, n = ctypes.c_void_p(), ctypes.c_size_t()
    state.ctx._ck(S.lib.sage_var_buffer(state.ctx.s, v.h, ctypes.byref(ptr), ctypes.byref(n)))
    return _view(state, ptr.value, v.extents or (1,), tuple(4 * s for s in v.strides) or (4,))


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(g, shape, std=1.0, mean=0.0):
    return (torch.randn(tuple(shape), generator=g, device="cuda") * std + mean).cpu().numpy()


def _integers(g, shape, high):
    return torch.randint(0, high, tuple(shape), generator=g, device="cuda").cpu().numpy().astype(np.uint32)


def _bert_model(state, case, g):
    w = case["width"]
    model = S.Bert(embed_dim=w, num_vocabs=VOCAB, max_num_tokens=MAX_TOKENS, hidden_dim=4 * w, num_layers=case["layers"], num_heads=w // 64,
                   num_classes=2, gelu=int(case.get("gelu", False)), layer_norm_eps=1e-12 if case.get("gelu") else 1e-5)
    params, scalars = model.params(), 0
    for p in params:
        if p.extents == (1,):  # LayerNorm's scale and shift, in turn
            state.ctx.set(p, _normal(g, (1,), 0.05, 1.0 if scalars % 2 == 0 else 0.0))
            scalars += 1
        else:
            state.ctx.set(p, _normal(g, p.extents, 0.02))
    return model, params


def _resnet_model(state, case, g, classes):
    model = S.ResNet18(case["channels"], classes)
    params = model.params()
    for p in params:
        e = p.extents
        fan_in = e[0] * e[1] * e[2] if len(e) == 4 else e[0]
        state.ctx.set(p, _normal(g, e, math.sqrt((2.0 if len(e) == 4 else 1.0) / fan_in) if len(e) > 1 else 0.01))
    return model, params


def _tokens(state, case, g):
    b, l = case["batch"], case["seq"]
    mask = np.ones((b, l), np.float32)
    if case.get("padded"):
        for i, pad in enumerate(_integers(g, (b,), max(l // 4, 1))):
            mask[i, l - int(pad):] = 0
    return state.ctx.var(_integers(g, (b, l), VOCAB)), state.ctx.var(mask)


def _prepare_training(state, case, model, params, logits, classes, g):
    """Loss = mean softmax cross entropy; gradients of every parameter; Adam."""
    state.model, state.params = model, params
    labels = state.ctx.var(_integers(g, (case["batch"], 1), classes))
    state.loss = S.softmax_cross_entropy(logits, labels).mean([0], False)
    state.grads = S.grad_param(state.loss, model)
    state.params = list(state.grads)
    state.targets = list(state.grads.values()) + [state.loss]
    state.opt = S.Adam(1e-4)
    state.opt.init(state.ctx)
    if case["kind"] == "train_bert":
        # Of the many equal encoder layers the first and the last are handed back, with the embeddings and the head.  The
        # gradient of a key projection's bias is left out: softmax ignores it, so it is zero up to rounding.
        n = 4 + 16 * case["layers"]
        shown = list(range(4)) + list(range(4, 20)) + (list(range(n - 16, n)) if case["layers"] > 1 else []) + [n, n + 1]
        shown = [i for i in shown if not (4 <= i < n and (i - 4) % 16 == 1)]
        moved = [i for i in shown if len(state.params[i].extents) == 2]
    else:
        shown = list(range(len(params)))
        moved = [i for i in shown if len(params[i].extents) == 4 and params[i].extents[0] > 1]
    values = list(state.grads.values())
    state.shown = [values[i] for i in shown]
    state.moved = [state.params[i] for i in moved]


def prepare(case, seed):
    state, g = _Program(), _generator(seed)
    ctx, kind = state.ctx, case["kind"]
    state.kind = kind
    if kind == "bert":
        state.model, state.params = _bert_model(state, case, g)
        state.target = state.model.pass_(*_tokens(state, case, g))
    elif kind == "resnet":
        state.model, state.params = _resnet_model(state, case, g, 1000)
        state.target = state.model.pass_(ctx.var(_normal(g, (case["batch"], case["size"], case["size"], case["channels"]))))
    elif kind == "train_bert":
        model, params = _bert_model(state, case, g)
        _prepare_training(state, case, model, params, model.pass_(*_tokens(state, case, g)), 2, g)
    elif kind == "train_resnet":
        model, params = _resnet_model(state, case, g, 10)
        x = ctx.var(_normal(g, (case["batch"], case["size"], case["size"], case["channels"])))
        _prepare_training(state, case, model, params, model.pass_(x), 10, g)
    elif kind == "gemm":
        m, n, k, b = case["m"], case["n"], case["k"], case["batch"]
        a = ctx.tensor(_normal(g, (b, k, m) if case["ta"] else (b, m, k)))
        w = ctx.tensor(_normal(g, (b, n, k) if case["tb"] else (b, k, n), 1.0 / math.sqrt(k)))
        y = ctx.empty((b, m, n))
        state.owned = [a, w, y]
        state.out = (S.lib.sage_buf_ptr(y.buf), (b, m, n))
        state.args = (ctx.h, int(case["ta"]), int(case["tb"]), L(m), L(n), L(k), a.buf, L(0), L(m if case["ta"] else k), L(m * k),
                      w.buf, L(0), L(k if case["tb"] else n), L(k * n), y.buf, L(0), L(n), L(m * n), L(b))
    else:
        r, c = case["rows"], case["cols"]
        x = ctx.var(_normal(g, (r, c)))
        if case["op"] == "cross_entropy_grad":
            y, labels = ctx.var(_normal(g, (r, c))), ctx.var(_integers(g, (r, 1), c))
            loss = S.softmax_cross_entropy(x * y + x * 3.14, labels)
            state.results = [loss, x.grad(loss)]
        elif case["op"] == "softmax":
            state.results = [S.softmax(x, [1])]
        elif case["op"] == "log_sum_exp":
            state.results = [S.log_sum_exp(x, [1])]
        else:
            state.results = [S.layer_norm(x, [1], ctx.var(_normal(g, (1,), 0.05, 1.0)), ctx.var(_normal(g, (1,), 0.05)), 1e-5)]
    return state


# ------------------------------------------------------------------------------------------ one pass
def run(state):
    ctx = state.ctx
    if state.kind in ("bert", "resnet"):
        ctx.clear()
        ctx.eval(state.target)
        return _result(state, state.target)
    if state.kind in ("train_bert", "train_resnet"):
        ctx.clear()
        ctx.eval(*state.targets)
        state.opt.update(state.grads, ctx)
        return {"loss": _result(state, state.loss), "gradients": [_result(state, v) for v in state.shown],
                "updated": [_result(state, v) for v in state.moved]}
    if state.kind == "gemm":
        ctx._ck(S.lib.sage_gemm_strided_batched(*state.args))
        return _view(state, *state.out)
    ctx.clear()
    ctx.eval(*state.results)
    return [_result(state, v) for v in state.results]


# ------------------------------------------------------------------------------------------ bounds
def _bert_work(case):
    t, w, n = case["batch"] * case["seq"], case["width"], case["layers"]
    flops = n * (4 * 2 * t * w * w + 2 * 2 * t * w * 4 * w + 4 * t * case["seq"] * w) + 2 * case["batch"] * w * 2
    weights = n * (4 * (w * w + w) + 8 * w * w + 5 * w + 4) + 2 * w + 4
    return flops, weights, t


def _resnet_work(case, classes):
    def out(h, k, s, p):
        return (h + 2 * p - k) // s + 1
    h, weights, per_image = out(case["size"], 7, 2, 3), 49 * case["channels"] * 64 + 64, 0
    per_image += 2 * h * h * 64 * 49 * case["channels"]
    h, cin = out(h, 3, 2, 1), 64
    for stage, planes in enumerate((64, 128, 256, 512)):
        for block in range(2):
            s = 2 if stage > 0 and block == 0 else 1
            o = out(h, 3, s, 1)
            per_image += 2 * o * o * planes * 9 * (cin + planes)
            weights += 9 * planes * (cin + planes) + 2 * planes
            if s != 1:
                per_image += 2 * o * o * planes * cin
                weights += planes * cin + planes
            h, cin = o, planes
    per_image += 2 * 512 * classes
    weights += 512 * classes + classes
    return case["batch"] * per_image, weights


def work(case):
    kind = case["kind"]
    if kind == "bert":
        flops, weights, t = _bert_work(case)
        return {"bytes": 4 * (weights + (t + case["seq"]) * case["width"] + 2 * t + 2 * case["batch"]), "flops": flops}
    if kind == "resnet":
        flops, weights = _resnet_work(case, 1000)
        return {"bytes": 4 * (weights + case["batch"] * (case["size"] ** 2 * case["channels"] + 1000)), "flops": flops}
    if kind in ("train_bert", "train_resnet"):  # Adam reads and writes parameters and both moments; gradients are written and read
        if kind == "train_bert":
            flops, weights, t = _bert_work(case)
            weights, inputs = weights + (VOCAB + MAX_TOKENS) * case["width"], 2 * t
        else:
            (flops, weights), inputs = _resnet_work(case, 10), case["batch"] * case["size"] ** 2 * case["channels"]
        return {"bytes": 4 * (9 * weights + inputs), "flops": 3 * flops}
    if kind == "gemm":
        m, n, k, b = case["m"], case["n"], case["k"], case["batch"]
        return {"bytes": 4 * b * (m * k + k * n + m * n), "flops": 2 * b * m * n * k}
    r, c = case["rows"], case["cols"]
    if case["op"] == "cross_entropy_grad":
        return {"bytes": 4 * (3 * r * c + 2 * r), "flops": 20 * r * c}
    return {"bytes": 4 * (r * c + (r if case["op"] == "log_sum_exp" else r * c)), "flops": 8 * r * c}


def tolerance(case):
    if case["kind"] == "gemm":  # fp32 products and sums of up to 8192 terms
        return {"rel": 1e-5, "max": 1e-4}
    if case["kind"] == "rows":
        return {"rel": 1e-5, "max": 1e-4}
    if case["kind"] in ("bert", "resnet"):  # fp32 rounding carried through up to 24 layers
        return {"rel": 5e-5, "max": 2e-4}
    # Gradients: a rectifier (or a pooling window) whose input lies within rounding of the switch passes its gradient in
    # one evaluation order and not in another.  A share e of such elements shows as sqrt(e) in the norm, and where a row
    # of an embedding's gradient belongs to one token, as a good part of that row.
    return {"rel": 1e-2, "max": 0.8}
