"""The measured cases: what a program built on this library has it do, through its public entry points.

A case is a dict of plain values; ``kind`` names the program that runs it:

``product``   a training step's use of one matrix product: forward, then both gradients
``mlp``       one SGD step of a two-hidden-layer perceptron with softmax cross entropy
``lstm``      forward and backward through time over an LSTM layer
``infer``     forward pass of a stack of fully connected layers whose weights stay in place
``host``      forward and both gradients of one product from pinned host buffers

Every program keeps one context, as a ``primitiv::Device`` object does, with the operand-plane
cache on; it forgets all planes at the start of a pass, because a training step has new inputs
and new weights (``infer`` forgets only what it writes).  Element order is primitiv's: column-major,
minibatch outermost.
"""
import math

import numpy as np
import torch

import primitiv_b200 as pb

MODES = {"fp32": pb.MODE_FP32_3XTF32, "tf32": pb.MODE_TF32, "fp16": pb.MODE_FP16, "fp32_3xfp16": pb.MODE_FP32_3XFP16}
PLANE_CACHE_BYTES = 8 << 30   # what the device class keeps

# numbers of the library's operation enumerations (include/primitiv_b200_ops.h)
NEGATE, EXP, TANH, SIGMOID, MUL_CONST, PRELU = 0, 3, 5, 6, 14, 19
ADD, SUBTRACT, MULTIPLY = 0, 1, 2
RED_SUM, RED_LOGSUMEXP = 0, 1


def listed():
    return [
        # A fully connected layer of a small model over a small minibatch, gradients added to
        # what earlier uses of the weight left: launches and host work count here.
        dict(name="layer_small", kind="product", mode="fp32", di=256, dj=256, dk=64, ba=1, bb=16, accumulate=True),
        # The benchmark's headline: large products, a matrix per minibatch item on either side.
        dict(name="square_batched", kind="product", mode="fp32", di=4096, dj=4096, dk=4096, ba=8, bb=8, accumulate=False),
        # The same in the opt-in fp32-grade mode on the half-precision pipe, at an ordinary size.
        dict(name="square_3xfp16", kind="product", mode="fp32_3xfp16", di=2048, dj=2048, dk=2048, ba=2, bb=2, accumulate=False),
        # Nothing a multiple of anything: vocabulary and feature counts of real data, a matrix
        # per item against one shared by all of them.
        dict(name="ragged_fp32", kind="product", mode="fp32", di=515, dj=1022, dk=387, ba=9, bb=1, accumulate=False),
        # The same in half storage, where no row starts on a 16-byte boundary.
        dict(name="ragged_half", kind="product", mode="fp16", di=1021, dj=765, dk=131, ba=12, bb=12, accumulate=False),
        # Many small products at once in the fast mode (scores and mixes of attention heads).
        dict(name="heads_tf32", kind="product", mode="tf32", di=128, dj=64, dk=128, ba=512, bb=512, accumulate=False),
        # Half storage at full size: a shared weight against a large minibatch.
        dict(name="half_broadcast", kind="product", mode="fp16", di=8192, dj=8192, dk=2048, ba=1, bb=32, accumulate=True),
        # Whole training steps of the perceptron on digit images: a very large minibatch ...
        dict(name="mlp_step_large", kind="mlp", mode="fp32", inputs=784, hidden=1024, classes=10, items=65536),
        # ... and one of the size it is usually trained with.
        dict(name="mlp_step_small", kind="mlp", mode="fp32", inputs=784, hidden=800, classes=10, items=200),
        # The recurrent loop of a sequence model, forward and backward through 50 steps.
        dict(name="lstm_loop", kind="lstm", mode="tf32", inputs=512, hidden=1024, items=64, steps=50),
        # Serving: a few requests through four large layers, half storage.
        dict(name="infer_half", kind="infer", mode="fp16", width=4096, layers=4, items=8),
        # A caller whose data lives in host memory: copies and products in one pipelined call.
        dict(name="host_step", kind="host", mode="fp32", di=1024, dj=1024, dk=1024, ba=16, bb=16),
    ]


def _spread(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _extent(rng, low, high, ragged):
    """A size between the two, spread over its logarithm: any integer, or a multiple of 8."""
    v = _spread(rng, low, high)
    return v if ragged else max(low, v // 8 * 8)


def draw(rng):
    kind = rng.choice(["product"] * 5 + ["mlp", "lstm", "infer", "host"])
    ragged = rng.random() < 0.4
    mode = rng.choice(["fp32", "fp32", "tf32", "fp16", "fp16", "fp32_3xfp16"])
    if kind in ("product", "host"):
        top = 4096 if kind == "product" else 2048
        di, dj, dk = (_extent(rng, 64, top, ragged) for _ in range(3))
        most = 4e11 if kind == "product" else 6e10   # multiply-adds of one direction: far below the largest listed
        batch = max(1, min(_spread(rng, 1, 512 if kind == "product" else 32), int(most / (1.0 * di * dj * dk))))
        ba, bb = rng.choice([(1, batch), (batch, batch), (batch, batch), (batch, 1)])
        case = dict(kind=kind, mode=mode, di=di, dj=dj, dk=dk, ba=ba, bb=bb)
        return dict(case, accumulate=rng.random() < 0.5) if kind == "product" else case
    if kind == "mlp":
        mode = rng.choice(["fp32", "tf32", "fp16"])
        # a sum of losses over more items would not fit half storage
        return dict(kind=kind, mode=mode, inputs=_extent(rng, 64, 1024, ragged), hidden=_extent(rng, 64, 1024, ragged),
                    classes=_spread(rng, 2, 200), items=_extent(rng, 32, 8192 if mode == "fp16" else 65536, ragged))
    if kind == "lstm":
        return dict(kind=kind, mode=rng.choice(["fp32", "tf32", "fp16"]), inputs=_extent(rng, 64, 512, ragged),
                    hidden=_extent(rng, 64, 1024, ragged), items=_extent(rng, 8, 128, ragged), steps=_spread(rng, 4, 50))
    return dict(kind=kind, mode=rng.choice(["fp32", "tf32", "fp16"]), width=_extent(rng, 512, 8192, ragged),
                layers=rng.randint(2, 4), items=_spread(rng, 1, 64))


# ---- shared by the programs ---------------------------------------------------------------------

_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = pb.Context(0)
        _ctx.operand_cache_enable(PLANE_CACHE_BYTES)
    return _ctx


def _storage(mode):
    return torch.float16 if mode == "fp16" else torch.float32


class _Arrays:
    """Device arrays made from one seed."""

    def __init__(self, mode, seed):
        self.type = _storage(mode)
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)

    def normal(self, n, scale=1.0):
        return torch.empty(n, device="cuda", dtype=self.type).normal_(0.0, scale, generator=self.gen)

    def uniform(self, n, low, high):
        return torch.empty(n, device="cuda", dtype=self.type).uniform_(low, high, generator=self.gen)

    def empty(self, n):
        return torch.empty(n, device="cuda", dtype=self.type)

    def full(self, n, value):
        return torch.full((n,), value, device="cuda", dtype=self.type)


class _Pointers:
    """The addresses of named arrays."""

    def __init__(self, arrays):
        for name, t in arrays.items():
            setattr(self, name, t.data_ptr())


# ---- product --------------------------------------------------------------------------------------

def _prepare_product(c, seed):
    m = _Arrays(c["mode"], seed)
    na, nb = c["di"] * c["dj"] * c["ba"], c["dj"] * c["dk"] * c["bb"]
    ny = c["di"] * c["dk"] * max(c["ba"], c["bb"])
    half = c["mode"] == "fp16"
    # half storage: values small enough for sums over a long contraction, as its users scale them
    t = dict(a=m.normal(na, 0.05) if half else m.uniform(na, -1, 1), b=m.normal(nb, 0.05) if half else m.uniform(nb, -1, 1),
             gy=m.normal(ny, 0.05 if half else 1.0), y=m.empty(ny), ga=m.full(na, 0.5), gb=m.full(nb, 0.5))
    return dict(ctx=_context(), mode=MODES[c["mode"]], size=(c["di"], c["dj"], c["dk"], c["ba"], c["bb"]),
                acc=c["accumulate"], t=t, p=_Pointers(t))


def _run_product(s):
    ctx, p, t = s["ctx"], s["p"], s["t"]
    ctx.operand_cache_invalidate()
    ctx.matmul_fw(s["mode"], p.a, p.b, p.y, *s["size"])
    ctx.matmul_bw_ex(s["mode"], p.a, p.b, p.gy, p.ga, p.gb, *s["size"], s["acc"], s["acc"])
    return t["y"], t["ga"], t["gb"]


# ---- host -----------------------------------------------------------------------------------------

def _prepare_host(c, seed):
    s = _prepare_product(dict(c, accumulate=False), seed)
    # pinned host memory, as a data loader hands it over
    t = {k: torch.empty(v.numel(), dtype=v.dtype, pin_memory=True).copy_(v) for k, v in s["t"].items()}
    return dict(s, t=t, p=_Pointers(t))


def _run_host(s):
    ctx, p, t = s["ctx"], s["p"], s["t"]
    ctx.operand_cache_invalidate()
    ctx.matmul_fw_bw_host(s["mode"], p.a, p.b, p.gy, p.y, p.ga, p.gb, *s["size"], False, False)
    return t["y"], t["ga"], t["gb"]


# ---- mlp: h1 = relu(W1.x + b1), h2 = relu(W2.h1 + b2), y = W3.h2 + b3, softmax cross entropy, SGD --------

LEARNING_RATE = 0.1
LOSS_SCALE = 1024.0   # half storage: keeps gradients of a mean over many items clear of subnormal numbers


def _prepare_mlp(c, seed):
    m = _Arrays(c["mode"], seed)
    n, k = c["items"], c["classes"]
    sizes = [c["inputs"], c["hidden"], c["hidden"], k]
    t = dict(x=m.uniform(sizes[0] * n, 0, 1), gx=m.empty(sizes[0] * n))
    for i in (1, 2, 3):
        rows, cols = sizes[i], sizes[i - 1]
        bound = math.sqrt(6.0 / (rows + cols))   # Xavier
        t.update({"w%d" % i: m.uniform(rows * cols, -bound, bound), "gw%d" % i: m.empty(rows * cols),
                  "dw%d" % i: m.empty(rows * cols), "b%d" % i: m.uniform(rows, -0.1, 0.1), "gb%d" % i: m.empty(rows),
                  "db%d" % i: m.empty(rows)})
        for name in ("z", "u", "h", "gz", "gu", "gh") if i < 3 else ("z", "u", "gz", "gu"):
            t["%s%d" % (name, i)] = m.empty(rows * n)
    # log softmax and its gradient
    for name in ("spread", "logp", "nlogp", "gneg", "glogp", "gspread", "e0", "e1", "e2", "e3"):
        t[name] = m.empty(k * n)
    t.update({name: m.empty(n) for name in ("lse", "picked", "gpicked", "glse")}, total=m.empty(1), loss=m.empty(1))
    labels = np.random.default_rng(seed).integers(0, k, n).astype(np.uint32)
    return dict(ctx=_context(), mode=MODES[c["mode"]], n=n, scale=LOSS_SCALE if c["mode"] == "fp16" else 1.0, sizes=sizes,
                labels=labels, ids=labels.ctypes.data, t=t, p=_Pointers(t))


def _run_mlp(s):
    ctx, mode, n, p, t = s["ctx"], s["mode"], s["n"], s["p"], s["t"]
    op, d = ctx.op, s["sizes"]
    k, kn = d[3], d[3] * n
    ctx.operand_cache_invalidate()
    # forward
    ctx.matmul_fw(mode, p.w1, p.x, p.z1, d[1], d[0], 1, 1, n)
    op("b200_binary_fw", mode, ADD, p.z1, p.b1, p.u1, d[1], n, 1, 0, None)
    op("b200_unary_fw", mode, PRELU, p.u1, p.h1, d[1] * n, 0.0, 0, None)
    ctx.matmul_fw(mode, p.w2, p.h1, p.z2, d[2], d[1], 1, 1, n)
    op("b200_binary_fw", mode, ADD, p.z2, p.b2, p.u2, d[2], n, 1, 0, None)
    op("b200_unary_fw", mode, PRELU, p.u2, p.h2, d[2] * n, 0.0, 0, None)
    ctx.matmul_fw(mode, p.w3, p.h2, p.z3, d[3], d[2], 1, 1, n)
    op("b200_binary_fw", mode, ADD, p.z3, p.b3, p.u3, d[3], n, 1, 0, None)
    # loss = mean over the minibatch of -log softmax(u3)[label]
    op("b200_reduce_fw", mode, RED_LOGSUMEXP, p.u3, p.lse, k, 1, n, None)
    op("b200_broadcast_fw", mode, p.lse, p.spread, n, 1, k, None)
    op("b200_binary_fw", mode, SUBTRACT, p.u3, p.spread, p.logp, k, n, 1, 1, None)
    op("b200_unary_fw", mode, NEGATE, p.logp, p.nlogp, kn, 0.0, 0, None)
    op("b200_pick_fw", mode, p.nlogp, s["ids"], n, p.picked, 1, k, 1, n, 1, None)
    op("b200_batch_sum_fw", mode, p.picked, p.total, 1, n, None)
    op("b200_unary_fw", mode, MUL_CONST, p.total, p.loss, 1, 1.0 / n, 0, None)
    # backward through the loss
    op("b200_fill", mode, p.gpicked, n, s["scale"] / n, None)
    op("b200_fill", mode, p.gneg, kn, 0.0, None)
    op("b200_pick_bw", mode, p.gpicked, s["ids"], n, p.gneg, 1, k, 1, n, 1, None)
    op("b200_unary_bw", mode, NEGATE, p.logp, p.nlogp, p.gneg, p.glogp, kn, 0.0, 0, 0, None)
    op("b200_binary_bw", mode, SUBTRACT, p.u3, p.spread, p.logp, p.glogp, p.gu3, p.gspread, k, n, 1, 1, 0, 0, None)
    op("b200_reduce_fw", mode, RED_SUM, p.gspread, p.glse, k, 1, n, None)
    op("b200_broadcast_fw", mode, p.lse, p.e0, n, 1, k, None)
    op("b200_binary_fw", mode, SUBTRACT, p.u3, p.e0, p.e1, k, n, 1, 1, None)
    op("b200_unary_fw", mode, EXP, p.e1, p.e2, kn, 0.0, 0, None)
    op("b200_broadcast_fw", mode, p.glse, p.e0, n, 1, k, None)
    op("b200_binary_fw", mode, MULTIPLY, p.e2, p.e0, p.e3, k, n, 1, 1, None)
    op("b200_inplace_add", mode, p.e3, p.gu3, k, n, n, 1.0, None)
    # backward through the layers
    op("b200_binary_bw", mode, ADD, p.z3, p.b3, p.u3, p.gu3, p.gz3, p.gb3, d[3], n, 1, 0, 0, 0, None)
    ctx.matmul_bw_ex(mode, p.w3, p.h2, p.gz3, p.gw3, p.gh2, d[3], d[2], 1, 1, n, False, False)
    op("b200_unary_bw", mode, PRELU, p.u2, p.h2, p.gh2, p.gu2, d[2] * n, 0.0, 0, 0, None)
    op("b200_binary_bw", mode, ADD, p.z2, p.b2, p.u2, p.gu2, p.gz2, p.gb2, d[2], n, 1, 0, 0, 0, None)
    ctx.matmul_bw_ex(mode, p.w2, p.h1, p.gz2, p.gw2, p.gh1, d[2], d[1], 1, 1, n, False, False)
    op("b200_unary_bw", mode, PRELU, p.u1, p.h1, p.gh1, p.gu1, d[1] * n, 0.0, 0, 0, None)
    op("b200_binary_bw", mode, ADD, p.z1, p.b1, p.u1, p.gu1, p.gz1, p.gb1, d[1], n, 1, 0, 0, 0, None)
    ctx.matmul_bw_ex(mode, p.w1, p.x, p.gz1, p.gw1, p.gx, d[1], d[0], 1, 1, n, False, False)
    # SGD
    rate = LEARNING_RATE / s["scale"]
    for w, gw, dw, b, gb, db, rows, cols in ((p.w1, p.gw1, p.dw1, p.b1, p.gb1, p.db1, d[1], d[0]),
                                             (p.w2, p.gw2, p.dw2, p.b2, p.gb2, p.db2, d[2], d[1]),
                                             (p.w3, p.gw3, p.dw3, p.b3, p.gb3, p.db3, d[3], d[2])):
        op("b200_unary_fw", mode, MUL_CONST, gw, dw, rows * cols, rate, 0, None)
        op("b200_inplace_add", mode, dw, w, rows * cols, 1, 1, -1.0, None)
        op("b200_unary_fw", mode, MUL_CONST, gb, db, rows, rate, 0, None)
        op("b200_inplace_add", mode, db, b, rows, 1, 1, -1.0, None)
    return [t[name] for name in ("loss", "u3", "gx", "gw1", "gb1", "gw2", "gb2", "gw3", "gb3", "w1", "b1", "w2", "b2", "w3", "b3")]


# ---- lstm: u = Wx.x + Wh.h + b; i, f, o = sigmoid, j = tanh of its quarters; c = i*j + f*c; h = o*tanh(c);
# ---- loss = mean over the minibatch of the sum of h^2 over units and steps ----------------------------------------------------------

def _prepare_lstm(c, seed):
    m = _Arrays(c["mode"], seed)
    e, h, n, steps = c["inputs"], c["hidden"], c["items"], c["steps"]
    t = dict(wx=m.uniform(4 * h * e, -0.1, 0.1), wh=m.uniform(4 * h * h, -0.1, 0.1), b=m.full(4 * h, 0.0),
             gwx=m.empty(4 * h * e), gwh=m.empty(4 * h * h), gb=m.empty(4 * h), x=m.normal(e * n * steps), gx=m.empty(e * n * steps),
             h0=m.full(h * n, 0.0), c0=m.full(h * n, 0.0), zero=m.full(1, 0.0), ghh=m.full(h * n, 1.0 / n))
    for name in ("ux", "uh", "s", "u", "gu", "gs", "gux", "guh"):
        t[name] = m.empty(4 * h * n)
    for name in ("si", "sf", "so", "sj", "i", "f", "o", "j", "ij", "fc", "c", "tc", "h"):
        t[name] = m.empty(h * n * steps)
    for name in ("hh", "go", "gtc", "gij", "gfc", "gi", "gf", "gj", "gsi", "gsf", "gso", "gsj", "gh", "gh_prev", "gc", "gc_prev"):
        t[name] = m.empty(h * n)
    t.update(row=m.empty(n), part=m.empty(1), mean=m.empty(1), loss=m.empty(steps))
    return dict(ctx=_context(), mode=MODES[c["mode"]], e=e, h=h, n=n, steps=steps, t=t, p=_Pointers(t), width=t["x"].element_size())


def _run_lstm(s):
    ctx, mode, p, t, w = s["ctx"], s["mode"], s["p"], s["t"], s["width"]
    op, e, hid, n, steps = ctx.op, s["e"], s["h"], s["n"], s["steps"]
    vol, size = hid * n, hid * n * w
    gates = ((p.si, p.i, SIGMOID), (p.sf, p.f, SIGMOID), (p.so, p.o, SIGMOID), (p.sj, p.j, TANH))
    ctx.operand_cache_invalidate()
    for step in range(steps):
        at = step * size
        h_prev, c_prev = (p.h + at - size, p.c + at - size) if step else (p.h0, p.c0)
        ctx.matmul_fw(mode, p.wx, p.x + step * e * n * w, p.ux, 4 * hid, e, 1, 1, n)
        ctx.operand_cache_invalidate(h_prev, size)
        ctx.matmul_fw(mode, p.wh, h_prev, p.uh, 4 * hid, hid, 1, 1, n)
        op("b200_binary_fw", mode, ADD, p.ux, p.uh, p.s, 4 * hid, n, 1, 1, None)
        op("b200_binary_fw", mode, ADD, p.s, p.b, p.u, 4 * hid, n, 1, 0, None)
        for q, (part, gate, f) in enumerate(gates):
            op("b200_slice_fw", mode, p.u, part + at, 1, 4 * hid, hid, q * hid, n, None)
            op("b200_unary_fw", mode, f, part + at, gate + at, vol, 0.0, 0, None)
        op("b200_binary_fw", mode, MULTIPLY, p.i + at, p.j + at, p.ij + at, hid, n, 1, 1, None)
        op("b200_binary_fw", mode, MULTIPLY, p.f + at, c_prev, p.fc + at, hid, n, 1, 1, None)
        op("b200_binary_fw", mode, ADD, p.ij + at, p.fc + at, p.c + at, hid, n, 1, 1, None)
        op("b200_unary_fw", mode, TANH, p.c + at, p.tc + at, vol, 0.0, 0, None)
        op("b200_binary_fw", mode, MULTIPLY, p.o + at, p.tc + at, p.h + at, hid, n, 1, 1, None)
        op("b200_binary_fw", mode, MULTIPLY, p.h + at, p.h + at, p.hh, hid, n, 1, 1, None)
        op("b200_reduce_fw", mode, RED_SUM, p.hh, p.row, hid, 1, n, None)
        op("b200_batch_sum_fw", mode, p.row, p.part, 1, n, None)
        op("b200_unary_fw", mode, MUL_CONST, p.part, p.mean, 1, 1.0 / n, 0, None)
        op("b200_binary_fw", mode, ADD, p.loss + (step - 1) * w if step else p.zero, p.mean, p.loss + step * w, 1, 1, 1, 1, None)
    gh, gc, gh_prev, gc_prev = p.gh, p.gc, p.gh_prev, p.gc_prev
    back = ((p.si, p.i, p.gi, p.gsi, SIGMOID), (p.sf, p.f, p.gf, p.gsf, SIGMOID), (p.so, p.o, p.go, p.gso, SIGMOID),
            (p.sj, p.j, p.gj, p.gsj, TANH))
    for step in range(steps - 1, -1, -1):
        at, later = step * size, int(step < steps - 1)
        h_prev, c_prev = (p.h + at - size, p.c + at - size) if step else (p.h0, p.c0)
        op("b200_binary_bw", mode, MULTIPLY, p.h + at, p.h + at, p.hh, p.ghh, gh, gh, hid, n, 1, 1, later, 1, None)
        op("b200_binary_bw", mode, MULTIPLY, p.o + at, p.tc + at, p.h + at, gh, p.go, p.gtc, hid, n, 1, 1, 0, 0, None)
        op("b200_unary_bw", mode, TANH, p.c + at, p.tc + at, p.gtc, gc, vol, 0.0, 0, later, None)
        op("b200_binary_bw", mode, ADD, p.ij + at, p.fc + at, p.c + at, gc, p.gij, p.gfc, hid, n, 1, 1, 0, 0, None)
        op("b200_binary_bw", mode, MULTIPLY, p.f + at, c_prev, p.fc + at, p.gfc, p.gf, gc_prev, hid, n, 1, 1, 0, 0, None)
        op("b200_binary_bw", mode, MULTIPLY, p.i + at, p.j + at, p.ij + at, p.gij, p.gi, p.gj, hid, n, 1, 1, 0, 0, None)
        for q, (part, gate, g, gpart, f) in enumerate(back):
            op("b200_unary_bw", mode, f, part + at, gate + at, g, gpart, vol, 0.0, 0, 0, None)
            op("b200_slice_bw_ex", mode, gpart, p.gu, 1, 4 * hid, hid, q * hid, 1, n, n, int(q > 0), None)
        op("b200_binary_bw", mode, ADD, p.s, p.b, p.u, p.gu, p.gs, p.gb, 4 * hid, n, 1, 0, 0, later, None)
        op("b200_binary_bw", mode, ADD, p.ux, p.uh, p.s, p.gs, p.gux, p.guh, 4 * hid, n, 1, 1, 0, 0, None)
        ctx.operand_cache_invalidate(p.gux, 4 * size)
        ctx.operand_cache_invalidate(p.guh, 4 * size)
        ctx.matmul_bw_ex(mode, p.wh, h_prev, p.guh, p.gwh, gh_prev, 4 * hid, hid, 1, 1, n, later, False)
        ctx.matmul_bw_ex(mode, p.wx, p.x + step * e * n * w, p.gux, p.gwx, p.gx + step * e * n * w, 4 * hid, e, 1, 1, n, later, False)
        gh, gh_prev, gc, gc_prev = gh_prev, gh, gc_prev, gc
    return [t[name] for name in ("loss", "h", "c", "gx", "gwx", "gwh", "gb")]


# ---- infer: x -> relu(W.x + b), layer after layer ------------------------------------------------------

def _prepare_infer(c, seed):
    m = _Arrays(c["mode"], seed)
    d, n = c["width"], c["items"]
    bound = math.sqrt(6.0 / d)   # keeps the size of the activations from layer to layer
    t = dict(x=m.normal(d * n), z=m.empty(d * n), u=m.empty(d * n))
    for i in range(c["layers"]):
        t.update({"w%d" % i: m.uniform(d * d, -bound, bound), "b%d" % i: m.uniform(d, -0.1, 0.1), "h%d" % i: m.empty(d * n)})
    p = _Pointers(t)
    layers = [(getattr(p, "w%d" % i), getattr(p, "b%d" % i), getattr(p, "h%d" % i)) for i in range(c["layers"])]
    return dict(ctx=_context(), mode=MODES[c["mode"]], d=d, n=n, layers=layers, t=t, p=p, bytes=d * n * t["x"].element_size())


def _run_infer(s):
    ctx, mode, d, n, p = s["ctx"], s["mode"], s["d"], s["n"], s["p"]
    op, x = ctx.op, p.x
    for w, b, h in s["layers"]:
        ctx.operand_cache_invalidate(x, s["bytes"])
        ctx.matmul_fw(mode, w, x, p.z, d, d, 1, 1, n)
        op("b200_binary_fw", mode, ADD, p.z, b, p.u, d, n, 1, 0, None)
        op("b200_unary_fw", mode, PRELU, p.u, h, d * n, 0.0, 0, None)
        x = h
    return s["t"]["h%d" % (len(s["layers"]) - 1)]


# ---- what the runner calls --------------------------------------------------------------------------------

_PREPARE = dict(product=_prepare_product, host=_prepare_host, mlp=_prepare_mlp, lstm=_prepare_lstm, infer=_prepare_infer)
_RUN = dict(product=_run_product, host=_run_host, mlp=_run_mlp, lstm=_run_lstm, infer=_run_infer)


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, seed)
    state["run"] = _RUN[case["kind"]]
    return state


def run(state):
    return state["run"](state)


def work(case):
    c, width = case, 2 if case["mode"] == "fp16" else 4
    if c["kind"] in ("product", "host"):
        na, nb = c["di"] * c["dj"] * c["ba"], c["dj"] * c["dk"] * c["bb"]
        batch = max(c["ba"], c["bb"])
        ny = c["di"] * c["dk"] * batch
        moved = 2 * na + 2 * nb + 2 * ny + ((na + nb) if c.get("accumulate") else 0)
        return dict(bytes=width * moved, flops=6.0 * c["di"] * c["dj"] * c["dk"] * batch)
    if c["kind"] == "mlp":
        weights = c["inputs"] * c["hidden"] + c["hidden"] * c["hidden"] + c["hidden"] * c["classes"]
        biases = 2 * c["hidden"] + c["classes"]
        # inputs and labels in, their gradient and the logits out; weights in and out, their gradients out
        moved = (2 * c["inputs"] + c["classes"]) * c["items"] + 3 * (weights + biases)
        return dict(bytes=width * moved + 4 * c["items"], flops=6.0 * weights * c["items"])
    if c["kind"] == "lstm":
        weights = 4 * c["hidden"] * (c["inputs"] + c["hidden"])
        moved = 2 * weights + (2 * c["inputs"] + 2 * c["hidden"]) * c["items"] * c["steps"]
        return dict(bytes=width * moved, flops=6.0 * weights * c["items"] * c["steps"])
    weights = c["width"] * c["width"] * c["layers"]
    return dict(bytes=width * (weights + c["width"] * (c["layers"] + 2 * c["items"])), flops=2.0 * weights * c["items"])


def tolerance(case):
    # fp32-grade modes: the library's own bound of 1e-5 per product; TF32 and half: 11 bits of
    # mantissa per operand or result.  A value next to a rounding boundary may move by a whole unit,
    # and what passes through several layers or steps carries each one's error on.
    one = {"fp32": 1e-5, "fp32_3xfp16": 1e-5, "tf32": 1e-3, "fp16": 1e-3}[case["mode"]]
    if case["kind"] in ("product", "host"):
        return dict(rel=one)
    deep = {"fp32": 5e-5, "tf32": 5e-3, "fp16": 1e-2}[case["mode"]]
    return dict(rel=deep, max=min(0.5, 100 * deep))
