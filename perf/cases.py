"""The work that a user of llmt_b200 has it do, as cases that can be timed and compared.

A case is a dict: `kind` names the call sequence, the other entries are its sizes and options.
Every kind goes through the public Python entry points on tensors, descriptors and workspaces
that the caller made beforehand, as a training or inference program would.

kind          what it is
linear        Linear forward, y = x W^T + b, optionally through the GELU, one llmt_b200.gemm call
linear_step   a Linear layer's training step: gradients zeroed, forward, dX, dW and dbias
layers_step   the four linear layers of a GPT block (QKV, attention output, MLP up with GELU, MLP
              down): forward of all, then backward of all, dX and dW + dbias of a layer per launch
mlp_step      an MLP chained end to end: forward that keeps the pre-activation, backward through
              the GELU, both dW + dbias
lm_head_loss  the tied LM head with its loss and gradients, the logits never stored
lm_head_fp32  the LM head as separate fp32 calls: logits, cross-entropy, its gradient in place, dX, dW
attn_step     attention, forward and backward, on [B*H, T, hd] head tensors, probabilities kept
attn_packed   attention forward out of the packed QKV projection into merged token rows
attn_fp32     attention forward as separate fp32 calls, heads split and merged by copies
"""
import math

import torch

import llmt_b200 as L
from llmt_b200.dp import GradBucket

VOCAB = 50257
BLOCK_LAYERS = (("qkv", 1, 3, False), ("attn_out", 1, 1, False), ("mlp_fc", 1, 4, True), ("mlp_proj", 4, 1, False))


def listed():
    return [
        # Token-by-token inference: a handful of rows through a projection. All latency.
        dict(name="linear bf16 8 rows", kind="linear", dtype="bf16", m=8, i=768, o=2304, gelu=False),
        # The MLP up-projection of a small batch (4 x 64 tokens) in llmt's own precision.
        dict(name="linear fp32 256", kind="linear", dtype="fp32", m=256, i=768, o=3072, gelu=False),
        # A short batch of uneven sequences through a layer whose widths suit no tile: odd pitches.
        dict(name="linear step bf16 odd", kind="linear_step", dtype="bf16", m=1537, i=771, o=1283, y_fp32=False, bias=True),
        # A block's linear layers with a small micro-batch (4 x 128 tokens): launches count.
        dict(name="layers step 512", kind="layers_step", m=512, c=768),
        # The GPT-2-small training step, 8 x 1024 tokens.
        dict(name="layers step 8192", kind="layers_step", m=8192, c=768),
        # The GPT-2-XL-shaped MLP in training, 8192 tokens on one GPU.
        dict(name="mlp step xl", kind="mlp_step", m=8192, c=1600),
        # The tied LM head with fp32 logits stored, contiguous vocabulary; dX and dW from bf16 dLogits.
        dict(name="lm head logits", kind="linear_step", dtype="bf16", m=8192, i=768, o=VOCAB, y_fp32=True, bias=False),
        # The same layer with its loss in training.
        dict(name="lm head loss", kind="lm_head_loss", m=8192, c=768, v=VOCAB),
        # llmt's own composition of head and loss, all fp32, a small micro-batch.
        dict(name="lm head fp32", kind="lm_head_fp32", m=512, c=768, v=VOCAB),
        # Attention of GPT-2 small in training, B = 8.
        dict(name="attention step 1024", kind="attn_step", b=8, h=12, t=1024, hd=64),
        # A prompt of uneven length through one attention layer.
        dict(name="attention packed 333", kind="attn_packed", b=4, h=12, t=333, hd=64),
        # llmt's naive attention in fp32.
        dict(name="attention fp32 256", kind="attn_fp32", b=4, h=12, t=256, hd=64),
    ]


# ------------------------------------------------------------------------------ drawn cases

def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo, hi):
    """A layer width: mostly what models use, sometimes what nobody planned for."""
    v = _log(rng, lo, hi)
    step = rng.choice((64, 64, 64, 8, 1))
    return max(step, v // step * step)


def _tokens(rng, lo, hi):
    v = _log(rng, lo, hi)
    return v if v < 128 or rng.random() < 0.5 else v // 64 * 64


def _capped(m, per_row, most):
    """Tokens brought down to where m * per_row stays within `most` operations."""
    return max(1, min(m, int(most // per_row)))


def draw(rng):
    kind = rng.choice(("linear", "linear", "linear_step", "linear_step", "layers_step", "layers_step", "mlp_step",
                       "lm_head_loss", "lm_head_fp32", "attn_step", "attn_step", "attn_packed", "attn_fp32"))
    if kind in ("linear", "linear_step"):
        dtype = "fp32" if rng.random() < 0.3 else "bf16"
        i, o = _width(rng, 64, 6400), _width(rng, 64, 6400)
        passes = 1 if kind == "linear" else 3
        most = 6e10 if dtype == "fp32" else 6e11
        m = _capped(_tokens(rng, 1, 16384), 2.0 * passes * i * o, most)
        if kind == "linear":
            return dict(kind=kind, dtype=dtype, m=m, i=i, o=o, gelu=rng.random() < 0.3)
        return dict(kind=kind, dtype=dtype, m=m, i=i, o=o, y_fp32=dtype == "fp32" or rng.random() < 0.2,
                    bias=rng.random() < 0.8)
    if kind == "layers_step":
        c = _width(rng, 256, 1600) // 8 * 8
        return dict(kind=kind, m=_capped(_tokens(rng, 32, 16384), 6.0 * 12 * c * c, 6e11), c=c)
    if kind == "mlp_step":
        c = _width(rng, 256, 1600) // 8 * 8
        return dict(kind=kind, m=_capped(_tokens(rng, 32, 16384), 6.0 * 8 * c * c, 8e11), c=c)
    if kind == "lm_head_loss":
        c, v = _width(rng, 256, 1600) // 8 * 8, rng.choice((VOCAB, VOCAB, _log(rng, 2000, VOCAB)))
        return dict(kind=kind, m=_capped(_tokens(rng, 64, 8192), 8.0 * c * v, 2.2e12), c=c, v=v)
    if kind == "lm_head_fp32":
        c, v = _width(rng, 256, 1024), rng.choice((VOCAB, _log(rng, 2000, VOCAB)))
        return dict(kind=kind, m=_capped(_tokens(rng, 32, 1024), 6.0 * c * v, 1e11), c=c, v=v)
    h, hd = rng.choice((1, 4, 8, 12, 16, 25)), rng.choice((32, 64, 64, 64, 96, 128))
    t = _tokens(rng, 16, 2048)
    most = 6e6 if kind == "attn_fp32" else 1e8
    b = max(1, min(rng.choice((1, 2, 4, 8)), int(most // (h * t * t))))
    if h * b * t * t > most:
        t = int(math.sqrt(most / (h * b)))
    return dict(kind=kind, b=b, h=h, t=t, hd=hd)


# ------------------------------------------------------------------------------ bytes and operations

def work(case):
    """Each input read once and each output written once; two operations per multiply-add."""
    k = case["kind"]
    if k in ("linear", "linear_step"):
        m, i, o = case["m"], case["i"], case["o"]
        e = 4 if case["dtype"] == "fp32" else 2
        if k == "linear":
            return {"bytes": e * (m * i + o * i + m * o) + 4 * o, "flops": 2.0 * m * i * o}
        y = 4 if case["y_fp32"] else e
        return {"bytes": e * (2 * m * i + o * i + m * o) + y * m * o + 4 * (o * i + 2 * o), "flops": 6.0 * m * i * o}
    if k == "layers_step":
        m, c = case["m"], case["c"]
        by = sum(2 * (2 * m * i * c + o * c * i * c + 2 * m * o * c) + 4 * (o * c * i * c + 2 * o * c)
                 for _, i, o, _ in BLOCK_LAYERS)
        return {"bytes": by, "flops": 6.0 * m * 12 * c * c}
    if k == "mlp_step":
        m, c = case["m"], case["c"]
        # x, dy in; y, h, pre, d_pre, dx out; two weights in, two gradients out
        return {"bytes": 2 * (4 * m * c + 3 * m * 4 * c + 8 * c * c) + 4 * (8 * c * c + 2 * 5 * c), "flops": 6.0 * m * 8 * c * c}
    if k == "lm_head_loss":
        m, c, v = case["m"], case["c"], case["v"]
        return {"bytes": 2 * (2 * m * c + v * c + m * v) + 4 * (v * c + 4 * m), "flops": 6.0 * m * c * v}
    if k == "lm_head_fp32":
        m, c, v = case["m"], case["c"], case["v"]
        return {"bytes": 4 * (2 * m * c + 2 * v * c + m * v + 4 * m), "flops": 6.0 * m * c * v}
    b, h, t, hd = case["b"], case["h"], case["t"], case["hd"]
    n = b * h
    if k == "attn_step":
        # q, k, v, dO in; O, dQ, dK, dV, P and dS out
        return {"bytes": 2 * (8 * n * t * hd + 2 * n * t * t) + 4 * n * t, "flops": 12.0 * n * t * t * hd}
    e = 4 if k == "attn_fp32" else 2
    return {"bytes": e * (4 * n * t * hd + n * t * t), "flops": 4.0 * n * t * t * hd}


def tolerance(case):
    """fp32: the order of sums of a few thousand terms. bf16: a result rounded to 2^-9 of itself, once
    (a product) or through a chain of rounded results (attention: P, dS)."""
    if case.get("dtype") == "fp32" or case["kind"] in ("lm_head_fp32", "attn_fp32"):
        return {"rel": 1e-5}
    if case["kind"] in ("attn_step", "attn_packed"):
        return {"rel": 1e-2}
    return {"rel": 5e-3}


# ------------------------------------------------------------------------------ what a program has in hand

def _workspace(desc, nbytes):
    """Gives the descriptor scratch of that size (none where it needs none)."""
    if not nbytes:
        return None
    buf = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    desc.workspace, desc.workspace_bytes = buf.data_ptr(), buf.numel()
    return buf


class _Inputs:
    """Seeded inputs on the GPU: activations N(0, 1), weights N(0, 0.02), gradients N(0, 0.01)."""

    def __init__(self, seed, dtype=torch.bfloat16):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        self.dtype = dtype

    def normal(self, *shape, scale=1.0, dtype=None):
        return torch.randn(*shape, device="cuda", generator=self.gen).mul_(scale).to(dtype or self.dtype)

    def weight(self, o, i):
        return self.normal(o, i, scale=0.02)

    def bias(self, o):
        return self.normal(o, scale=0.02, dtype=torch.float32)

    def targets(self, rows, vocab):
        t = torch.randint(vocab, (rows,), device="cuda", generator=self.gen, dtype=torch.int32)
        mask = (torch.rand(rows, device="cuda", generator=self.gen) >= 0.05).float()  # some padding tokens
        mask[0] = 1.0
        return t, mask


def _empty(*shape, dtype=torch.bfloat16):
    return torch.empty(*shape, dtype=dtype, device="cuda")


def _group(problems):
    g = L.Group(problems)
    g.set_workspaces([torch.empty(n, dtype=torch.uint8, device="cuda") if n else None for n in g.workspace_bytes()])
    return g


def _backward_group(dx, dy, w, x, dw, db, dx_desc=None):
    """dX and dW (+ dbias) of one layer as one launch, gradients accumulated."""
    return _group([(dx_desc or L.make_desc(dx, dy, w, False, False), dx, dy, w),
                   (L.make_desc(dw, dy, x, True, False, beta=1.0, dbias=db, dbias_beta=1.0), dw, dy, x)])


def _gradients(shapes):
    return GradBucket(shapes, "cuda")


def prepare(case, seed):
    s = globals()["_prepare_" + case["kind"]](case, seed)
    s["kind"] = case["kind"]
    return s


def run(state):
    return globals()["_run_" + state["kind"]](state)


def _prepare_linear(case, seed):
    r = _Inputs(seed, torch.float32 if case["dtype"] == "fp32" else torch.bfloat16)
    m, i, o = case["m"], case["i"], case["o"]
    s = dict(x=r.normal(m, i), w=r.weight(o, i), b=r.bias(o), y=_empty(m, o, dtype=r.dtype), gelu=case["gelu"])
    need = L.workspace_bytes(L.make_desc(s["y"], s["x"], s["w"], False, True, bias=s["b"], gelu=s["gelu"]), s["x"], s["w"])
    s["ws"] = torch.empty(need, dtype=torch.uint8, device="cuda") if need else None
    return s


def _run_linear(s):
    L.gemm(s["y"], s["x"], s["w"], False, True, bias=s["b"], gelu=s["gelu"], workspace=s["ws"])
    return s["y"]


def _prepare_linear_step(case, seed):
    fp32 = case["dtype"] == "fp32"
    r = _Inputs(seed, torch.float32 if fp32 else torch.bfloat16)
    m, i, o = case["m"], case["i"], case["o"]
    x, w = r.normal(m, i), r.weight(o, i)
    b = r.bias(o) if case["bias"] else None
    dy = r.normal(m, o, scale=1e-4 if o > 20000 else 0.01)
    y = _empty(m, o, dtype=torch.float32 if case["y_fp32"] else r.dtype)
    dx = _empty(m, i, dtype=r.dtype)
    grads = _gradients({"dw": (o, i), "db": (o,)})
    dw, db = grads.view("dw"), grads.view("db")
    d_fwd = L.make_desc(y, x, w, False, True, bias=b)
    s = dict(x=x, w=w, b=b, dy=dy, y=y, dx=dx, grads=grads, dw=dw, db=db, d_fwd=d_fwd, fp32=fp32)
    s["ws"] = _workspace(d_fwd, L.workspace_bytes(d_fwd, x, w))
    if fp32:
        s["d_dx"] = L.make_desc(dx, dy, w, False, False)
        s["d_dw"] = L.make_desc(dw, dy, x, True, False, beta=1.0, dbias=db if case["bias"] else None, dbias_beta=1.0)
        s["ws_bwd"] = [_workspace(s["d_dx"], L.workspace_bytes(s["d_dx"], dy, w)),
                       _workspace(s["d_dw"], L.workspace_bytes(s["d_dw"], dy, x))]
    else:
        s["bwd"] = _backward_group(dx, dy, w, x, dw, db if case["bias"] else None)
    return s


def _run_linear_step(s):
    s["grads"].zero_()
    L.gemm_desc(s["d_fwd"], s["y"], s["x"], s["w"])
    if s["fp32"]:
        L.gemm_desc(s["d_dx"], s["dx"], s["dy"], s["w"])
        L.gemm_desc(s["d_dw"], s["dw"], s["dy"], s["x"])
    else:
        s["bwd"].run()
    return s["y"], s["dx"], s["dw"], s["db"]


def _prepare_layers_step(case, seed):
    r = _Inputs(seed)
    m, c = case["m"], case["c"]
    spec = [(n, i * c, o * c, gelu) for n, i, o, gelu in BLOCK_LAYERS]
    grads = _gradients({k: v for n, i, o, _ in spec for k, v in ((n + ".dw", (o, i)), (n + ".db", (o,)))})
    layers = []
    for n, i, o, gelu in spec:
        t = dict(x=r.normal(m, i), w=r.weight(o, i), b=r.bias(o), dy=r.normal(m, o, scale=0.01), y=_empty(m, o),
                 dx=_empty(m, i), dw=grads.view(n + ".dw"), db=grads.view(n + ".db"))
        t["d_fwd"] = L.make_desc(t["y"], t["x"], t["w"], False, True, bias=t["b"], gelu=gelu)
        t["ws"] = _workspace(t["d_fwd"], L.workspace_bytes(t["d_fwd"], t["x"], t["w"]))
        t["bwd"] = _backward_group(t["dx"], t["dy"], t["w"], t["x"], t["dw"], t["db"])
        layers.append(t)
    return dict(grads=grads, layers=layers)


def _run_layers_step(s):
    s["grads"].zero_()
    for t in s["layers"]:
        L.gemm_desc(t["d_fwd"], t["y"], t["x"], t["w"])
    for t in reversed(s["layers"]):
        t["bwd"].run()
    return [(t["y"], t["dx"], t["dw"], t["db"]) for t in s["layers"]]


def _prepare_mlp_step(case, seed):
    r = _Inputs(seed)
    m, c = case["m"], case["c"]
    x, w_fc, w_proj, b_fc, b_proj = r.normal(m, c), r.weight(4 * c, c), r.weight(c, 4 * c), r.bias(4 * c), r.bias(c)
    dy = r.normal(m, c, scale=0.01)
    h, pre, d_pre, y, dx = _empty(m, 4 * c), _empty(m, 4 * c), _empty(m, 4 * c), _empty(m, c), _empty(m, c)
    grads = _gradients({"fc.dw": (4 * c, c), "fc.db": (4 * c,), "proj.dw": (c, 4 * c), "proj.db": (c,)})
    g = {k: grads.view(k) for k in ("fc.dw", "fc.db", "proj.dw", "proj.db")}
    d_fc = L.make_desc(h, x, w_fc, False, True, bias=b_fc, gelu=True, save_pre=pre)
    d_proj = L.make_desc(y, h, w_proj, False, True, bias=b_proj)
    d_dpre = L.make_desc(d_pre, dy, w_proj, False, False, gelu_bwd_of=pre)
    s = dict(x=x, w_fc=w_fc, w_proj=w_proj, b_fc=b_fc, b_proj=b_proj, h=h, pre=pre, d_pre=d_pre, y=y, dx=dx, dy=dy,
             grads=grads, g=g, d_fc=d_fc, d_proj=d_proj)
    s["ws"] = [_workspace(d_fc, L.workspace_bytes(d_fc, x, w_fc)), _workspace(d_proj, L.workspace_bytes(d_proj, h, w_proj))]
    s["bwd_proj"] = _backward_group(d_pre, dy, w_proj, h, g["proj.dw"], g["proj.db"], dx_desc=d_dpre)
    s["bwd_fc"] = _backward_group(dx, d_pre, w_fc, x, g["fc.dw"], g["fc.db"])
    return s


def _run_mlp_step(s):
    s["grads"].zero_()
    L.gemm_desc(s["d_fc"], s["h"], s["x"], s["w_fc"])
    L.gemm_desc(s["d_proj"], s["y"], s["h"], s["w_proj"])
    s["bwd_proj"].run()
    s["bwd_fc"].run()
    return s["y"], s["h"], s["pre"], s["d_pre"], s["dx"], s["g"]


def _prepare_lm_head_loss(case, seed):
    r = _Inputs(seed)
    m, c, v = case["m"], case["c"], case["v"]
    pitch = (v + 7) // 8 * 8  # rows of dLogits padded to whole 16-byte groups
    x, w = r.normal(m, c), r.weight(v, c)
    targets, mask = r.targets(m, v)
    dlogits = torch.zeros(m, pitch, dtype=torch.bfloat16, device="cuda")[:, :v]
    logits_like = torch.empty_strided((m, v), (v, 1), dtype=torch.float32, device="meta")
    d_fwd = L.make_desc(logits_like, x, w, False, True)
    d_bwd = L.make_desc(dlogits, x, w, False, True)
    s = dict(x=x, w=w, targets=targets, mask=mask, dlogits=dlogits, d_fwd=d_fwd, d_bwd=d_bwd, dx=_empty(m, c),
             row_nll=_empty(m, dtype=torch.float32), loss=_empty(1, dtype=torch.float32), grads=_gradients({"dw": (v, c)}))
    s["ws"] = _workspace(d_fwd, L.lm_head_ce_workspace_bytes(d_fwd, x, w))
    d_bwd.workspace, d_bwd.workspace_bytes = d_fwd.workspace, d_fwd.workspace_bytes  # the statistics stay there
    s["bwd"] = _backward_group(s["dx"], dlogits, w, x, s["grads"].view("dw"), None)
    return s


def _run_lm_head_loss(s):
    s["grads"].zero_()
    L.lm_head_ce_fwd(s["d_fwd"], None, s["x"], s["w"], s["targets"], s["mask"], s["row_nll"], s["loss"])
    L.lm_head_ce_bwd(s["d_bwd"], s["dlogits"], s["x"], s["w"], s["targets"], s["mask"], 1.0, stats_valid=True)
    s["bwd"].run()
    return s["loss"], s["row_nll"], s["dlogits"], s["dx"], s["grads"].view("dw")


def _prepare_lm_head_fp32(case, seed):
    r = _Inputs(seed, torch.float32)
    m, c, v = case["m"], case["c"], case["v"]
    x, w = r.normal(m, c), r.weight(v, c)
    targets, mask = r.targets(m, v)
    logits, dx = _empty(m, v, dtype=r.dtype), _empty(m, c, dtype=r.dtype)
    grads = _gradients({"dw": (v, c)})
    dw = grads.view("dw")
    s = dict(x=x, w=w, targets=targets, mask=mask, logits=logits, dx=dx, grads=grads, dw=dw,
             row_nll=_empty(m, dtype=r.dtype), loss=_empty(1, dtype=r.dtype),
             d_fwd=L.make_desc(logits, x, w, False, True), d_dx=L.make_desc(dx, logits, w, False, False),
             d_dw=L.make_desc(dw, logits, x, True, False, beta=1.0))
    s["ws"] = [_workspace(s["d_fwd"], L.workspace_bytes(s["d_fwd"], x, w)),
               _workspace(s["d_dx"], L.workspace_bytes(s["d_dx"], logits, w)),
               _workspace(s["d_dw"], L.workspace_bytes(s["d_dw"], logits, x))]
    return s


def _run_lm_head_fp32(s):
    logits = s["logits"]
    s["grads"].zero_()
    L.gemm_desc(s["d_fwd"], logits, s["x"], s["w"])
    L.cross_entropy_fwd(s["loss"], s["row_nll"], logits, s["targets"], s["mask"])
    L.cross_entropy_bwd(logits, logits, s["targets"], s["mask"])
    L.gemm_desc(s["d_dx"], s["dx"], logits, s["w"])
    L.gemm_desc(s["d_dw"], s["dw"], logits, s["x"])
    return s["loss"], s["row_nll"], logits, s["dx"], s["dw"]


def _prepare_attn_step(case, seed):
    r = _Inputs(seed)
    n, t, hd = case["b"] * case["h"], case["t"], case["hd"]
    q, k, v, d_o = r.normal(n, t, hd), r.normal(n, t, hd), r.normal(n, t, hd), r.normal(n, t, hd, scale=0.01)
    p, ds = _empty(n, t, t), _empty(n, t, t)
    o, dq, dk, dv = (_empty(n, t, hd) for _ in range(4))
    a = 1.0 / math.sqrt(hd)
    s = dict(q=q, k=k, v=v, d_o=d_o, p=p, ds=ds, o=o, dq=dq, dk=dk, dv=dv, row_dot=_empty(n, t, dtype=torch.float32))
    s["d_p"] = L.make_desc(p, q, k, False, True, alpha=a)
    s["d_ds"] = L.make_desc(ds, d_o, v, False, True)
    s["ws"] = [_workspace(s["d_p"], L.gemm_softmax_workspace_bytes(s["d_p"], q, k)),
               _workspace(s["d_ds"], L.workspace_bytes(s["d_ds"], d_o, v))]
    s["products"] = {}
    for name, c, x, y, tr, al in (("o", o, p, v, False, 1.0), ("dv", dv, p, d_o, True, 1.0), ("dq", dq, ds, k, False, a),
                                  ("dk", dk, ds, q, True, a)):
        d = L.make_desc(c, x, y, tr, False, alpha=al)
        s["ws"].append(_workspace(d, L.workspace_bytes(d, x, y)))
        s["products"][name] = (d, c, x, y)
    return s


def _run_attn_step(s):
    pr = s["products"]
    L.gemm_softmax_fwd(s["d_p"], s["p"], s["q"], s["k"], True)
    L.gemm_desc(*pr["o"])
    L.gemm_desc(*pr["dv"])
    L.rowdot(s["row_dot"], s["d_o"], s["o"])
    L.gemm_softmax_bwd(s["d_ds"], s["ds"], s["d_o"], s["v"], s["p"], s["row_dot"], True)
    L.gemm_desc(*pr["dq"])
    L.gemm_desc(*pr["dk"])
    return s["p"], s["o"], s["ds"], s["dq"], s["dk"], s["dv"]


def _prepare_attn_packed(case, seed):
    r = _Inputs(seed)
    b, h, t, hd = case["b"], case["h"], case["t"], case["hd"]
    width, pitch = h * hd, (t + 7) // 8 * 8  # rows of P padded to whole 16-byte groups
    qkv, y = r.normal(b, t, 3 * width), _empty(b, t, width)
    p = torch.zeros(b * h, t, pitch, dtype=torch.bfloat16, device="cuda")
    d_p, d_o = L.GemmDesc(), L.GemmDesc()
    for d in (d_p, d_o):
        d.m, d.batch, d.batch_inner, d.dtype_ab, d.dtype_c = t, b * h, h, L.BF16, L.BF16
    # P = softmax(Q K^T / sqrt(hd)): operands are [T, hd] views of the packed rows
    d_p.n, d_p.k, d_p.trans_b, d_p.alpha = t, hd, 1, 1.0 / math.sqrt(hd)
    d_p.lda = d_p.ldb = 3 * width
    d_p.stride_a = d_p.stride_b = hd
    d_p.stride_a_outer = d_p.stride_b_outer = t * 3 * width
    d_p.ldc, d_p.stride_c, d_p.stride_c_outer = pitch, t * pitch, h * t * pitch
    # O = P V, straight into columns of the merged token rows
    d_o.n, d_o.k, d_o.alpha = hd, t, 1.0
    d_o.lda, d_o.stride_a, d_o.stride_a_outer = pitch, t * pitch, h * t * pitch
    d_o.ldb, d_o.stride_b, d_o.stride_b_outer = 3 * width, hd, t * 3 * width
    d_o.ldc, d_o.stride_c, d_o.stride_c_outer = width, hd, t * width
    q, k, v = qkv, qkv[:, :, width:], qkv[:, :, 2 * width:]
    s = dict(qkv=qkv, q=q, k=k, v=v, p=p, y=y, d_p=d_p, d_o=d_o)
    s["ws"] = [_workspace(d_p, L.gemm_softmax_workspace_bytes(d_p, q, k)), _workspace(d_o, L.workspace_bytes(d_o, p, v))]
    return s


def _run_attn_packed(s):
    L.gemm_softmax_fwd(s["d_p"], s["p"], s["q"], s["k"], True)
    L.gemm_desc(s["d_o"], s["y"], s["p"], s["v"])
    return s["p"], s["y"]


def _prepare_attn_fp32(case, seed):
    r = _Inputs(seed, torch.float32)
    b, h, t, hd = case["b"], case["h"], case["t"], case["hd"]
    heads = [_empty(b, h, t, hd, dtype=r.dtype) for _ in range(4)]
    s = dict(qkv=r.normal(b, t, 3 * h * hd), y=_empty(b, t, h * hd, dtype=r.dtype), heads=heads,
             p=_empty(b * h, t, t, dtype=r.dtype))
    q, k, v, o = (x.view(b * h, t, hd) for x in heads)
    s["d_s"] = (L.make_desc(s["p"], q, k, False, True, alpha=1.0 / math.sqrt(hd)), s["p"], q, k)
    s["d_o"] = (L.make_desc(o, s["p"], v, False, False), o, s["p"], v)
    s["ws"] = [_workspace(s["d_s"][0], L.workspace_bytes(s["d_s"][0], q, k)),
               _workspace(s["d_o"][0], L.workspace_bytes(s["d_o"][0], s["p"], v))]
    return s


def _run_attn_fp32(s):
    q, k, v, o = s["heads"]
    L.head_split(q, k, v, s["qkv"])
    L.gemm_desc(*s["d_s"])
    L.softmax_fwd(s["p"], s["p"], True)
    L.gemm_desc(*s["d_o"])
    L.head_merge(s["y"], o)
    return s["p"], s["y"]
