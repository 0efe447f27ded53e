"""The work whose speed is tracked: one pass of each case is one call (or one
launch of a kept handle) through the package's public entry points.

Families (`"kind"` of a case) and the ranges they stand for:

  call   one TTV on device memory (`ttv` with the low-level argument list, or
         `ttv_array` with torch's row-major convention): orders 2 to 7, 2^8 to
         2^28 elements, cubes, uneven extents, thin contractions of 4 and long
         ones, every mode, first- and last-order layouts, fp32, fp64 and
         bf16-stored A, compensated (default) or plain accumulation
  view   `ttv_view` on a padded, sliced, stepped or transposed torch view
  chain  `ttvs`: every mode but one contracted
  batch  one launch of a kept `Batch` of uneven fp32 problems (16 to 4096)
  host   `ttv_host` on host buffers, page-locked or pageable
  model  the cost model's kernels: loss and gradient of a minibatch, or
         predictions of a shape set's variants
"""
import functools
import math

import torch

import ttv_gb300 as T
from ttv_gb300 import batch as B
from ttv_gb300 import costmodel as CM


def listed():
    return [
        # a call of the size that unit grids and small solvers make: latency alone
        {"name": "array_small_f32", "kind": "call", "entry": "array", "dtype": "f32", "shape": "24x20x16", "q": 2},
        # the smallest configured problem: order 3, 256 in every mode, the middle mode contracted
        {"name": "cube256_f32", "kind": "call", "entry": "ttv", "dtype": "f32", "layout": "first", "acc": 0,
         "values": "uniform", "shape": "256x256x256", "q": 2},
        # the symmetric sweep's order 3 in double precision: odd extents, no row of A on the 16-byte grid
        {"name": "cube645_f64", "kind": "call", "entry": "ttv", "dtype": "f64", "layout": "first", "acc": 0,
         "values": "uniform", "shape": "645x645x645", "q": 2},
        # the asymmetric sweep's order 6: one long mode, contraction over 4
        {"name": "thin4_f32", "kind": "call", "entry": "ttv", "dtype": "f32", "layout": "first", "acc": 0,
         "values": "uniform", "shape": "262144x4x4x4x4x4", "q": 3},
        # the long contraction with bf16-stored A of wide dynamic range
        {"name": "long_bf16a", "kind": "call", "entry": "ttv", "dtype": "bf16a", "layout": "first", "acc": 0,
         "values": "wide", "shape": "16x1048576x16", "q": 2},
        # rows padded for alignment (256 of 264), the middle mode contracted
        {"name": "view_padded_f32", "kind": "view", "dtype": "f32", "shape": "512x512x256", "pad": "0x0x8",
         "step": "1x1x1", "offset": "0x0x0", "perm": "1x2x3", "q": 2},
        # an odd sub-block of a field, transposed, contracted along its strided mode
        {"name": "view_sliced_f64", "kind": "view", "dtype": "f64", "shape": "190x241x251", "pad": "9x8x7",
         "step": "1x1x1", "offset": "3x5x3", "perm": "3x1x2", "q": 2},
        # the multi-vector chain on an order-4 tensor
        {"name": "chain128_f32", "kind": "chain", "dtype": "f32", "shape": "128x128x128x128", "q": 3},
        # the batched configuration: 4096 uneven problems a launch
        {"name": "batch4096_f32", "kind": "batch", "count": 4096, "shapes": 4096, "select": "learned"},
        # a small batch, as one step of a tensor method hands over
        {"name": "batch64_f32", "kind": "batch", "count": 64, "shapes": 64, "select": "learned"},
        # the reference's own calling convention: page-locked host buffers in, host result out
        {"name": "host256_f32", "kind": "host", "dtype": "f32", "layout": "first", "shape": "256x256x256", "q": 2,
         "pinned": True},
        # one minibatch of the cost model's training (forward, loss, backward)
        {"name": "model_grad512", "kind": "model", "op": "grad", "rows": 512},
    ]


# ---------------------------------------------------------------------------
# drawn cases
# ---------------------------------------------------------------------------
def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _int_log(rng, lo, hi):
    return max(lo, min(hi, int(round(_log(rng, lo, hi)))))


def _text(values):
    return "x".join(str(int(v)) for v in values)


def _extents(rng, order, elements):
    """Uneven extents (at least 2) of about `elements` in all, none above 2^22."""
    w = [rng.uniform(0.3, 1.0) for _ in range(order)]
    s = sum(w)
    n = [max(2, min(1 << 22, int(round(elements ** (x / s))))) for x in w]
    while math.prod(n) > elements and max(n) > 2:
        n[n.index(max(n))] -= max(1, max(n) // 8)
    return n


def _draw_call(rng):
    dtype = rng.choice(["f32", "f32", "f64", "bf16a"])
    elements = _log(rng, 1 << 8, 1 << 28)
    form = rng.choice(["cube", "uneven", "uneven", "thin", "long"])
    if form == "thin" and elements >= 1 << 12:
        order = rng.randint(2, 7)
        n = [max(4, int(elements / 4 ** (order - 1)))] + [4] * (order - 1)
        q = rng.randint(1, order)
    elif form == "long" and elements >= 1 << 16:
        lead = rng.choice([1, 2, 16, 24, 64])
        n = [lead, max(64, min(1 << 22, int(elements / lead)))]
        q = 2
        if rng.random() < 0.5:
            n.append(rng.choice([2, 3, 16]))
            n[1] = max(64, n[1] // n[2])
    elif form == "cube":
        order = rng.randint(2, 7)
        n = [max(2, int(elements ** (1.0 / order)))] * order
        q = rng.randint(1, order)
    else:
        order = rng.randint(2, 6)
        n = _extents(rng, order, elements)
        q = rng.randint(1, order)
    entry = "array" if rng.random() < 0.25 else "ttv"
    c = {"kind": "call", "entry": entry, "dtype": dtype, "shape": _text(n), "q": q}
    if entry == "ttv":
        c.update(layout=rng.choice(["first", "last"]), acc=1 if rng.random() < 0.1 else 0,
                 values="wide" if form == "long" else "uniform")
    return c


def _draw_view(rng):
    order = rng.randint(2, 4)
    n = _extents(rng, order, _log(rng, 1 << 12, 1 << 26))
    perm = list(range(1, order + 1))
    if rng.random() < 0.5:
        rng.shuffle(perm)
    aligned = rng.random() < 0.4
    if aligned:
        n[-1] = (n[-1] + 3) // 4 * 4
    step = [1] * order
    if rng.random() < 0.25:
        step[rng.randrange(order)] = 2
    pad = [rng.choice([0, 4, 8, 32] if aligned else [0, 1, 3, 6]) for _ in range(order)]
    off = [0 if aligned else rng.randint(0, p) for p in pad]
    if pad[-1] == 0 and step == [1] * order and perm == sorted(perm):
        pad[-1] = 8
    return {"kind": "view", "dtype": rng.choice(["f32", "f32", "f64"]), "shape": _text(n), "pad": _text(pad),
            "step": _text(step), "offset": _text(off), "perm": _text(perm), "q": rng.randint(1, order)}


def _draw_chain(rng):
    order = rng.randint(3, 6)
    elements = _log(rng, 1 << 14, 1 << 28)
    n = [max(2, int(elements ** (1.0 / order)))] * order if rng.random() < 0.4 else _extents(rng, order, elements)
    return {"kind": "chain", "dtype": rng.choice(["f32", "f32", "f64", "bf16a"]), "shape": _text(n),
            "q": rng.randint(1, order)}


def _draw_batch(rng):
    return {"kind": "batch", "count": _int_log(rng, 16, 3500), "shapes": rng.randrange(1 << 20),
            "select": rng.choice(["learned", "fixed"])}


def _draw_host(rng):
    order = rng.randint(2, 5)
    n = _extents(rng, order, _log(rng, 1 << 10, 1 << 25))
    return {"kind": "host", "dtype": rng.choice(["f32", "f64"]), "layout": rng.choice(["first", "last"]),
            "shape": _text(n), "q": rng.randint(1, order), "pinned": rng.random() < 0.75}


def _draw_model(rng):
    if rng.random() < 0.7:
        return {"kind": "model", "op": "grad", "rows": _int_log(rng, 32, 4096)}
    return {"kind": "model", "op": "predict", "rows": _int_log(rng, 288, 18000)}


def draw(rng):
    return rng.choices([_draw_call, _draw_view, _draw_chain, _draw_batch, _draw_host, _draw_model],
                       [0.42, 0.16, 0.12, 0.14, 0.06, 0.10])[0](rng)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
DT = {"f32": torch.float32, "f64": torch.float64, "bf16a": torch.float32}


def _ints(text):
    return [int(x) for x in text.split("x")]


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(n, g, dtype=torch.float32):
    return torch.rand(n, generator=g, device="cuda", dtype=dtype).mul_(2).sub_(1)


def _values(n, g, case):
    """A's values: uniform in [-1, 1], or N(0, 1) 10^U(-3, 3) (wide dynamic range)."""
    dt = DT[case["dtype"]]
    if case.get("values") == "wide":
        a = torch.randn(n, generator=g, device="cuda", dtype=dt)
        a.mul_(torch.pow(10.0, _uniform(n, g, dt).mul_(3)))
    else:
        a = _uniform(n, g, dt)
    return a.to(torch.bfloat16) if case["dtype"] == "bf16a" else a


def _layout(case):
    p = len(_ints(case["shape"]))
    return list(range(1, p + 1)) if case["layout"] == "first" else list(range(p, 0, -1))


def _meta(case):
    na, pia, q = _ints(case["shape"]), _layout(case), case["q"]
    nc, pic = T.output_shape(na, q), T.output_layout(pia, q)
    return {"q": q, "p": len(na), "na": na, "wa": T.strides(na, pia), "pia": pia, "nb": [na[q - 1]], "nc": nc,
            "wc": T.strides(nc, pic), "pic": pic}


def _view_inputs(case, seed):
    n, pad, step, off = (_ints(case[k]) for k in ("shape", "pad", "step", "offset"))
    g = _gen(seed)
    dt = DT[case["dtype"]]
    base = _uniform(math.prod(m * s + p for m, s, p in zip(n, step, pad)), g, dt)
    base = base.view([m * s + p for m, s, p in zip(n, step, pad)])
    A = base[tuple(slice(o, o + (m - 1) * s + 1, s) for m, s, o in zip(n, step, off))]
    A = A.permute([m - 1 for m in _ints(case["perm"])])
    return A, _uniform(A.shape[case["q"] - 1], g, dt)


def _chain_inputs(case, seed):
    na, q = _ints(case["shape"]), case["q"]
    g = _gen(seed)
    A = _values(math.prod(na), g, case).view(na)
    return A, [_uniform(n, g, DT[case["dtype"]]) for m, n in enumerate(na) if m != q - 1]


@functools.lru_cache(maxsize=16)
def _shapes(count, seed):
    """The batched configuration's problems: orders 3 to 5, extents log-uniform in [8, 512], at
    most 2^22 elements, any mode and layout."""
    return CM.random_shapes(count, seed)


def _batch_inputs(case, seed):
    shapes = _shapes(case["count"], case["shapes"])
    sizes = [math.prod(int(x) for x in na) for na, _, _ in shapes]
    outs = [s // int(na[q - 1]) for s, (na, _, q) in zip(sizes, shapes)]
    g = _gen(seed)
    A = _uniform(sum((s + 63) // 64 * 64 for s in sizes), g)
    return shapes, sizes, outs, A, _uniform(512, g)


def _model_inputs(case, seed):
    n = case["rows"]
    g = _gen(seed)
    x = torch.zeros(n, B.MLP_IN, device="cuda")
    x[:, :B.MLP_FEATURES] = torch.rand(n, B.MLP_FEATURES, generator=g, device="cuda")
    v = torch.randint(0, B.NVARIANT, (n,), generator=g, device="cuda")
    x[torch.arange(n, device="cuda"), B.MLP_FEATURES + v] = 1.0
    y = torch.randn(n, generator=g, device="cuda").mul_(2).add_(4)   # log2 of a cost in microseconds
    return torch.from_numpy(B.init_params(seed)).cuda(), x, y


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "call":
        g = _gen(seed)
        na, q = _ints(case["shape"]), case["q"]
        st["a"] = _values(math.prod(na), g, case)
        st["b"] = _uniform(na[q - 1], g, DT[case["dtype"]])
        if case["entry"] == "array":
            st["a"] = st["a"].view(na)
        else:
            st["m"] = _meta(case)
            st["c"] = torch.empty(math.prod(na) // na[q - 1], device="cuda", dtype=DT[case["dtype"]])
            if case["dtype"] == "bf16a":
                st["a"] = st["a"].view(torch.int16)
            st["dtype"] = {"f32": T.F32, "f64": T.F64, "bf16a": T.BF16A}[case["dtype"]]
            st["opts"] = {"accumulate": T.ACC_PLAIN} if case["acc"] else {}
    elif kind == "view":
        st["a"], st["b"] = _view_inputs(case, seed)
    elif kind == "chain":
        st["a"], st["bs"] = _chain_inputs(case, seed)
    elif kind == "batch":
        shapes, sizes, outs, A, b = _batch_inputs(case, seed)
        st["a"], st["b"] = A, b
        st["c"] = torch.zeros(sum((m + 63) // 64 * 64 for m in outs), device="cuda")
        B.load_cost_model()
        probs = CM.problems_from_arena([(sh, 1) for sh in shapes], A, b, st["c"])
        st["batch"] = B.Batch(probs, select=B.SELECT_LEARNED if case["select"] == "learned" else B.SELECT_HEURISTIC)
    elif kind == "host":
        g = _gen(seed)
        m = st["m"] = _meta(case)
        n, dt = math.prod(m["na"]), DT[case["dtype"]]
        for key, t in (("a", _uniform(n, g, dt)), ("b", _uniform(m["nb"][0], g, dt)),
                       ("c", torch.zeros(n // m["nb"][0], device="cuda", dtype=dt))):
            h = torch.empty(t.numel(), dtype=dt, pin_memory=case["pinned"])
            h.copy_(t)
            st[key] = h
    else:
        st["w"], st["x"], st["y"] = _model_inputs(case, seed)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "call":
        if case["entry"] == "array":
            return T.ttv_array(case["q"], st["a"], st["b"])
        m = st["m"]
        return T.ttv(m["q"], m["p"], st["a"], m["na"], m["wa"], m["pia"], st["b"], m["nb"], st["c"], m["nc"],
                     m["wc"], m["pic"], dtype=st["dtype"], **st["opts"])
    if kind == "view":
        return T.ttv_view(case["q"], st["a"], st["b"])
    if kind == "chain":
        return T.ttvs(case["q"], st["a"], st["bs"])
    if kind == "batch":
        st["batch"].launch()
        return st["c"]
    if kind == "host":
        m = st["m"]
        return T.ttv_host(m["q"], m["p"], st["a"], m["na"], m["wa"], m["pia"], st["b"], m["nb"], st["c"], m["nc"],
                          m["wc"], m["pic"])
    if case["op"] == "grad":
        return B.mlp_loss_grad(st["w"], st["x"], st["y"])
    return B.mlp_predict(st["w"], st["x"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
ESIZE = {"f32": (4, 4), "f64": (8, 8), "bf16a": (2, 4)}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        nbytes = flops = 0
        for na, _, q in _shapes(case["count"], case["shapes"]):
            n, nq = math.prod(int(x) for x in na), int(na[q - 1])
            nbytes += 4 * (n + nq + n // nq)
            flops += 2 * n
        return {"bytes": nbytes, "flops": flops}
    if kind == "model":
        n, macs = case["rows"], B.MLP_IN * 64 + 2 * 64 * 64 + 64
        nbytes = 4 * (n * (B.MLP_IN + 1) + 2 * B.MLP_PARAMS)
        return {"bytes": nbytes, "flops": (6 if case["op"] == "grad" else 2) * macs * n}
    n = _ints(case["shape"])
    if kind == "view":
        n = [n[m - 1] for m in _ints(case["perm"])]
    ea, et = ESIZE[case["dtype"]]
    total, nq = math.prod(n), n[case["q"] - 1]
    if kind == "chain":
        return {"bytes": ea * total + et * sum(n), "flops": 2 * total}
    return {"bytes": ea * total + et * (nq + total // nq), "flops": 2 * total}


# ---------------------------------------------------------------------------
# the same in 64 bits, plain torch
# ---------------------------------------------------------------------------
def _contract(A3, b):
    """sum_i A3[s, i, j] b[i] in fp64, over blocks of s or of j that fit comfortably."""
    S, nq, P = A3.shape
    out = torch.empty(S, P, device=A3.device, dtype=torch.float64)
    w = b.double().view(1, nq, 1)
    sb = max(1, min(S, (1 << 26) // max(1, nq * min(P, 1 << 16))))
    jb = max(1, min(P, (1 << 26) // max(1, nq * sb)))
    for s0 in range(0, S, sb):
        for j0 in range(0, P, jb):
            out[s0:s0 + sb, j0:j0 + jb] = (A3[s0:s0 + sb, :, j0:j0 + jb].double() * w).sum(1)
    return out


def _canonical(na, pia, q):
    k = pia.index(q)
    return (math.prod(na[m - 1] for m in pia[k + 1:]), na[q - 1], math.prod(na[m - 1] for m in pia[:k]))


def exact(case, seed):
    kind = case["kind"]
    if kind == "call" and case["entry"] == "array":
        g = _gen(seed)
        na, q = _ints(case["shape"]), case["q"]
        a = _values(math.prod(na), g, case)
        b = _uniform(na[q - 1], g, DT[case["dtype"]])
        c = _contract(a.view(_canonical(na, list(range(len(na), 0, -1)), q)), b)
        return c.reshape([n for m, n in enumerate(na) if m != q - 1])
    if kind in ("call", "host"):
        g = _gen(seed)
        na, q = _ints(case["shape"]), case["q"]
        a = _values(math.prod(na), g, case)
        b = _uniform(na[q - 1], g, DT[case["dtype"]])
        c = _contract(a.view(_canonical(na, _layout(case), q)), b).reshape(-1)
        return c.cpu() if kind == "host" else c
    if kind == "view":
        A, b = _view_inputs(case, seed)
        q = case["q"]
        other = [m for m in range(A.dim()) if m != q - 1]
        shape = [A.shape[m] for m in other]
        moved = A.permute([q - 1] + other).reshape(1, A.shape[q - 1], -1)
        return _contract(moved, b).reshape(shape)
    if kind == "chain":
        A, bs = _chain_inputs(case, seed)
        na, q = list(A.shape), case["q"]
        for r in range(len(na), 0, -1):   # slowest index last: modes from the fastest down
            if r == q:
                continue
            shape = list(A.shape)
            A = _contract(A.reshape(math.prod(shape[:r - 1]), shape[r - 1], math.prod(shape[r:])),
                          bs[r - 1 if r < q else r - 2]).reshape(shape[:r - 1] + [1] + shape[r:])
        return A.reshape(na[q - 1])
    if kind == "batch":
        shapes, sizes, outs, A, b = _batch_inputs(case, seed)
        c = torch.zeros(sum((m + 63) // 64 * 64 for m in outs), device="cuda", dtype=torch.float64)
        oa = oc = 0
        for (na, pia, q), s, m in zip(shapes, sizes, outs):
            na, pia = [int(x) for x in na], [int(x) for x in pia]
            S, nq, P = _canonical(na, pia, q)
            c[oc:oc + m] = (A[oa:oa + s].view(S, nq, P).double() * b[:nq].double().view(1, nq, 1)).sum(1).view(-1)
            oa += (s + 63) // 64 * 64
            oc += (m + 63) // 64 * 64
        return c
    w, x, y = (t.double() for t in _model_inputs(case, seed))
    w.requires_grad_(case["op"] == "grad")
    at, h = 0, x
    for layer, (i, o) in enumerate(((B.MLP_IN, 64), (64, 64), (64, 64), (64, 1))):
        W, bias = w[at:at + i * o].view(i, o), w[at + i * o:at + i * o + o]
        at += i * o + o
        h = h @ W + bias
        if layer < 3:
            h = torch.relu(h)
    if case["op"] == "predict":
        return h.view(-1)
    loss = 0.5 * (h.view(-1) - y).square().mean()
    (grad,) = torch.autograd.grad(loss, w)
    return loss.detach().view(1), grad
