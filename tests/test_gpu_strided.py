"""The general-stride extension, tlibg_ttv_strided (no reference counterpart:
the drop-in calls keep the reference's dense-only rule).  Natural meaning of
every stride: A's element (i_1..i_p) at a[sum i_r wa[r]], b's i-th at b[i wb],
C's element at c[sum j_r wc[r]].  Truth: numpy fp64 over the same strided
views (as_strided), error max |c - ref| / sum |a b| against the bars 1e-5
(fp32) and 1e-13 (fp64); C's untouched elements (padding) must stay as they
were.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {np.float32: 1e-5, np.float64: 1e-13}


def view(buf, shape, strides):
    return np.lib.stride_tricks.as_strided(buf, shape=shape, strides=[s * buf.itemsize for s in strides])


def padded_strides(na, pia, rng, pad_max=3):
    """Strides of a padded dense tensor in layout pia (each mode's stride at least
    the span of the faster ones)."""
    w = [0] * len(na)
    span = 1
    for m in pia:
        w[m - 1] = span
        span *= na[m - 1] + int(rng.integers(0, pad_max + 1))
    return w


def case(rng, dt, p, max_elems=1 << 18):
    while True:
        na = [int(x) for x in rng.integers(1, 24, p)]
        if np.prod(na) <= max_elems:
            break
    pia = [int(x) + 1 for x in rng.permutation(p)]
    q = int(rng.integers(1, p + 1))
    wa = padded_strides(na, pia, rng)
    nc = [n for m, n in enumerate(na) if m != q - 1]
    pic = [int(x) + 1 for x in rng.permutation(p - 1)]
    wc = padded_strides(nc, pic, rng)
    wb = int(rng.integers(1, 4))
    return na, pia, q, wa, nc, pic, wc, wb


def run_case(engine, torch, dev, rng, dt, na, pia, q, wa, nc, pic, wc, wb):
    p = len(na)
    size_a = 1 + sum((n - 1) * w for n, w in zip(na, wa))
    size_c = 1 + sum((n - 1) * w for n, w in zip(nc, wc))
    nq = na[q - 1]
    abuf = rng.uniform(-1, 1, size_a).astype(dt)
    bbuf = rng.uniform(-1, 1, (nq - 1) * wb + 1).astype(dt)
    cbuf = np.full(size_c, 7.0, dt)
    Av, bv = view(abuf, na, wa).astype(np.float64), view(bbuf, [nq], [wb]).astype(np.float64)
    ref = np.tensordot(Av, bv, axes=([q - 1], [0]))
    absn = np.tensordot(np.abs(Av), np.abs(bv), axes=([q - 1], [0]))
    da, db, dc = (torch.from_numpy(x).to(dev) for x in (abuf, bbuf, cbuf))
    engine.ttv_strided(q, p, da, na, wa, pia, db, [nq], dc, nc, wc, pic, wb=wb)
    torch.cuda.synchronize()
    out = dc.cpu().numpy()
    got = view(out, nc, wc).astype(np.float64)
    err = np.max(np.abs(got - ref) / np.maximum(absn, 1e-300)) if ref.size else 0.0
    # every element C's strides do not address keeps its value
    mask = np.ones(size_c, bool)
    idx = np.zeros(1, np.int64)
    for n, w in zip(nc, wc):
        idx = (idx[:, None] + np.arange(n) * w).ravel()
    mask[idx] = False
    assert (out[mask] == 7.0).all()
    return err


@pytest.mark.parametrize("dt", [np.float32, np.float64], ids=["fp32", "fp64"])
def test_random_padded_views(engine, cuda, dt):
    import torch
    rng = np.random.default_rng(5150 if dt == np.float32 else 5151)
    worst = 0.0
    for t in range(60):
        na, pia, q, wa, nc, pic, wc, wb = case(rng, dt, int(rng.integers(2, 6)))
        err = run_case(engine, torch, cuda, rng, dt, na, pia, q, wa, nc, pic, wc, wb)
        assert err <= TOL[dt], (na, pia, q, wa, nc, pic, wc, wb, err)
        worst = max(worst, err)


def test_long_rows_and_columns(engine, cuda):
    """Row form (q fastest, warp per output) and column form with long contractions."""
    import torch
    rng = np.random.default_rng(77)
    for dt in (np.float32, np.float64):
        for na, pia, q in (([3000, 40], [1, 2], 1), ([40, 3000], [1, 2], 2), ([17, 999, 13], [2, 1, 3], 2),
                           ([1, 5000, 1], [1, 2, 3], 2), ([300, 1, 200], [3, 1, 2], 1)):
            wa = padded_strides(na, pia, rng)
            nc = [n for m, n in enumerate(na) if m != q - 1]
            pic = list(range(1, len(nc) + 1))
            wc = padded_strides(nc, pic, rng)
            err = run_case(engine, torch, cuda, rng, dt, na, pia, q, wa, nc, pic, wc, 2)
            assert err <= TOL[dt], (na, pia, q, dt, err)


def test_dense_strides_match_the_dense_call(engine, orc, cuda):
    import torch
    rng = np.random.default_rng(9)
    for na, pia, q in (([64, 48, 80], [1, 2, 3], 2), ([25, 25, 25, 25], [4, 3, 2, 1], 3), ([7, 300], [2, 1], 2)):
        p = len(na)
        wa = engine.strides(na, pia)
        nc, pic = engine.output_shape(na, q), engine.output_layout(pia, q)
        wc = engine.strides(nc, pic)
        a = rng.uniform(-1, 1, int(np.prod(na))).astype(np.float32)
        b = rng.uniform(-1, 1, na[q - 1]).astype(np.float32)
        da, db = torch.from_numpy(a).to(cuda), torch.from_numpy(b).to(cuda)
        c1 = torch.empty(int(np.prod(nc)), device=cuda)
        c2 = torch.empty_like(c1)
        engine.ttv(q, p, da, na, wa, pia, db, [na[q - 1]], c1, nc, wc, pic, sync=True)
        engine.ttv_strided(q, p, da, na, wa, pia, db, [na[q - 1]], c2, nc, wc, pic)
        P, nq, S = orc.canonical(na, pia, q)
        ref, absn = orc.truth(S, nq, P, a, b)
        assert orc.rel_error(c2.cpu().numpy(), ref, absn) <= 1e-5
        assert orc.rel_error(c1.cpu().numpy(), ref, absn) <= 1e-5


def test_torch_views(engine, cuda):
    """ttv_view: slices, transposes and a strided b, no copy, against torch in fp64."""
    import torch
    g = torch.Generator(device=cuda)
    g.manual_seed(3)
    base = torch.rand(64, 90, 70, generator=g, device=cuda, dtype=torch.float64) * 2 - 1
    bb = torch.rand(300, generator=g, device=cuda, dtype=torch.float64) * 2 - 1
    for A in (base[:, ::2, 5:60], base.transpose(0, 2), base[::3].permute(1, 2, 0), base[10:20, :, ::7]):
        for q in range(1, 4):
            n = A.shape[q - 1]
            b = bb[: 2 * n : 2]
            c = engine.ttv_view(q, A, b)
            ref = torch.tensordot(A, b, dims=([q - 1], [0]))
            absn = torch.tensordot(A.abs(), b.abs(), dims=([q - 1], [0]))
            torch.cuda.synchronize()
            assert c.shape == ref.shape
            assert ((c - ref).abs() / absn.clamp_min(1e-300)).max().item() <= 1e-13


def test_vector_forms(engine, cuda):
    """Views on the 16-byte grid take the 16-byte forms: padded rows contracted
    along the row (row form) and across rows (column form, which takes them when
    the outputs fill the GPU: the 4 x 800 x 800 view), fp32 and fp64, with rows
    long and short, against torch in fp64."""
    import torch
    g = torch.Generator(device=cuda)
    g.manual_seed(11)
    for dt, V in ((torch.float32, 4), (torch.float64, 2)):
        for shape, pad in (((48, 30, 64), 4), ((7, 5, 1000), 8), ((3, 200, 8), 2 * V), ((4, 800, 800), 8)):
            base = torch.rand(shape[0], shape[1], shape[2] + pad, generator=g, device=cuda, dtype=dt) * 2 - 1
            A = base[:, :, :shape[2]]
            for q in (1, 2, 3):
                b = torch.rand(A.shape[q - 1], generator=g, device=cuda, dtype=dt) * 2 - 1
                c = engine.ttv_view(q, A, b)
                ref = torch.tensordot(A.double(), b.double(), dims=([q - 1], [0]))
                absn = torch.tensordot(A.double().abs(), b.double().abs(), dims=([q - 1], [0]))
                bar = 1e-5 if dt == torch.float32 else 1e-13
                assert ((c.double() - ref).abs() / absn.clamp_min(1e-300)).max().item() <= bar, (dt, shape, q)


# memory order of the base (slowest first); the last extent is padded
SPLIT_SHAPES = [(2, 3, 2), (3, 5000, 7), (1, 90000, 4), (30000, 6), (5, 70001), (700, 33, 64), (1300, 1381),
                (4, 3, 100000), (17, 2, 4096), (4099, 3, 5, 8), (2, 400, 640), (61, 16, 500)]


@pytest.mark.parametrize("pad", [1, 4])
@pytest.mark.parametrize("dt", [np.float32, np.float64], ids=["fp32", "fp64"])
@pytest.mark.parametrize("shape", SPLIT_SHAPES, ids=["x".join(map(str, s)) for s in SPLIT_SHAPES])
def test_shared_contractions(engine, orc, cuda, shape, dt, pad):
    """Every way the contracted mode is shared (warps, clusters, segments of the grid), loads of
    one element and of 16 bytes, several rows or columns per thread: every mode of padded views,
    into contiguous and into padded, permuted outputs.  Truth in double-double.  Bars: Kahan's
    two roundings per product and the result's (fp32: 4 x 2^-24); one rounding per product and
    the result's (fp64: 4 x 2^-53), both of sum |a b|."""
    import torch
    tdt = torch.float32 if dt == np.float32 else torch.float64
    g = torch.Generator(device=cuda)
    g.manual_seed(len(shape) * 1000 + shape[-1] + pad)
    base = torch.rand(*shape[:-1], shape[-1] + pad, generator=g, device=cuda, dtype=tdt) * 2 - 1
    A = base[..., :shape[-1]]
    p = len(shape)
    bar = 4 * 2.0 ** -24 if dt == np.float32 else 4 * 2.0 ** -53
    dense = A.contiguous().cpu().numpy().ravel()
    for q in range(1, p + 1):
        b = torch.rand(shape[q - 1], generator=g, device=cuda, dtype=tdt) * 2 - 1
        S, nq, P = int(np.prod(shape[:q - 1])), shape[q - 1], int(np.prod(shape[q:]))
        ref, absn = orc.truth(S, nq, P, dense, b.cpu().numpy())
        oshape = [n for m, n in enumerate(shape) if m != q - 1]
        wide = torch.full([n + 1 for n in reversed(oshape)], 7.0, device=cuda, dtype=tdt)
        out = wide.permute(*range(p - 2, -1, -1))[tuple(slice(0, n) for n in oshape)]
        for c in (engine.ttv_view(q, A, b), engine.ttv_view(q, A, b, out=out)):
            got = c.contiguous().cpu().numpy().ravel()
            assert orc.rel_error(got, ref, absn) <= bar, (shape, q, dt, pad)
        rest = wide.clone()
        rest.permute(*range(p - 2, -1, -1))[tuple(slice(0, n) for n in oshape)].fill_(7.0)
        assert (rest == 7.0).all()


@pytest.mark.parametrize("kind", ["growing", "falling", "zeros", "huge", "tiny", "mixed", "cancelling"])
@pytest.mark.parametrize("row", [True, False], ids=["row", "col"])
def test_fp64_exponent_windows(engine, orc, cuda, kind, row):
    """The fixed-point sums' window: products that outgrow it, fall below it, vanish, sit at the
    ends of the exponent range or cancel; bar: one rounding per product and the result's, of
    sum |a b| (and of the smallest normal number)."""
    import torch
    n, m = 3000, 41
    rng = np.random.default_rng(11)
    a = rng.uniform(-1, 1, (m, n))
    if kind == "growing":
        a *= np.exp2(np.linspace(-300, 300, n))
    elif kind == "falling":
        a *= np.exp2(np.linspace(300, -300, n))
    elif kind == "zeros":
        a[rng.uniform(size=a.shape) < 0.9] = 0.0
        a[5] = 0.0
    elif kind == "huge":
        a *= 2.0 ** 1009
    elif kind == "tiny":
        a *= 2.0 ** -1020
    elif kind == "mixed":
        a *= np.exp2(rng.uniform(-200, 200, a.shape))
    else:
        a[:, 1::2] = -a[:, 0::2]
    b = np.ones(n) if kind == "cancelling" else rng.uniform(-1, 1, n)
    buf = np.zeros((m, n + 3))
    buf[:, :n] = a
    A = torch.from_numpy(buf).to(cuda)[:, :n]
    if not row:
        A = torch.from_numpy(np.ascontiguousarray(buf.T)).to(cuda)[:n].T   # contracted mode strided
        A = torch.nn.functional.pad(A.T, (0, 3))[:, :m].T
    c = engine.ttv_view(2, A, torch.from_numpy(b).to(cuda)).cpu().numpy()
    import fractions
    for i in range(0, m, 5):
        terms = [fractions.Fraction(x) * fractions.Fraction(y) for x, y in zip(a[i], b)]
        exact, absn = sum(terms), sum(abs(t) for t in terms)
        bar = absn * fractions.Fraction(4, 2 ** 53) + n * fractions.Fraction(1, 2 ** 1074)
        assert abs(fractions.Fraction(float(c[i])) - exact) <= bar, (kind, i)


def test_fp64_nonfinite_products(engine, cuda):
    """Infinities and NaNs among the products reach their output and no other."""
    import torch
    a = torch.rand(37, 500, device=cuda, dtype=torch.float64)
    b = torch.rand(500, device=cuda, dtype=torch.float64)
    a[3, 77], a[8, 2], a[20, 499] = float("inf"), float("nan"), float("-inf")
    for A in (torch.nn.functional.pad(a, (0, 3))[:, :500], torch.nn.functional.pad(a.T, (0, 3))[:, :37].T):
        c = engine.ttv_view(2, A, b)
        bad = torch.zeros(37, dtype=torch.bool, device=cuda)
        bad[[3, 8, 20]] = True
        assert not torch.isfinite(c[bad]).any() and torch.isfinite(c[~bad]).all()


def _captured(torch, fn, stream):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        fn()
    return graph


@pytest.mark.parametrize("shape,q", [((2, 700001), 2), ((900001, 3), 1)], ids=["rows", "columns"])
def test_captured_views_need_no_scratch(engine, cuda, shape, q):
    """A view of few outputs, whose eager call allocates scratch for segments of the contraction,
    is captured on a stream that never had any, and replayed on new data after a larger eager call."""
    import torch
    g = torch.Generator(device=cuda)
    g.manual_seed(5)
    base = torch.empty(shape[0], shape[1] + 1, device=cuda)
    A, b = base[:, :shape[1]], torch.empty(shape[q - 1], device=cuda)
    c = torch.empty(shape[2 - q], device=cuda)

    def check():
        ref, absn = torch.mv(A.double() if q == 2 else A.double().T, b.double()), A.double().abs().sum(q - 1)
        assert ((c.double() - ref).abs() <= 4 * 2.0 ** -24 * absn).all()

    def fill():
        base.uniform_(-1, 1, generator=g)
        b.uniform_(-1, 1, generator=g)
        c.fill_(float("nan"))

    fill()
    fresh, s = torch.cuda.Stream(), torch.cuda.Stream()
    before = engine.device_alloc_count()
    engine.ttv_view(q, A, b, out=c, stream=fresh)
    torch.cuda.synchronize()
    assert engine.device_alloc_count() == before + 1
    check()
    graph = _captured(torch, lambda: engine.ttv_view(q, A, b, out=c, stream=s), s)
    assert engine.device_alloc_count() == before + 1
    for _ in range(2):
        fill()
        graph.replay()
        torch.cuda.synchronize()
        check()
        wide = torch.rand(4, 1 << 20, device=cuda)[:, 1:]
        engine.ttv_view(2, wide, wide[0], stream=s)
        torch.cuda.synchronize()


def test_captured_scratch_outlives_its_growth(engine, cuda):
    """A captured split call keeps its scratch when a later call on the stream outgrows it; a split
    plan captured on a stream without scratch runs unsplit."""
    import torch
    g = torch.Generator(device=cuda)
    g.manual_seed(6)

    def problem(P, nq, S, **opts):
        a, b = torch.empty(S, nq, P, device=cuda), torch.empty(nq, device=cuda)
        c = torch.empty(S, P, device=cuda)

        def call():
            engine.ttv(2, 3, a, [P, nq, S], [1, P, P * nq], [1, 2, 3], b, [nq], c, [P, S], [1, P], [1, 2], **opts)

        def fill():
            for t in (a, b):
                t.uniform_(-1, 1, generator=g)
            c.fill_(float("nan"))

        def check():
            ref = torch.einsum("sip,i->sp", a.double(), b.double())
            absn = torch.einsum("sip,i->sp", a.double().abs(), b.double().abs())
            assert ((c.double() - ref).abs() <= 4 * 2.0 ** -24 * absn).all()
        return call, fill, check

    s = torch.cuda.Stream()
    small, fill, check = problem(1024, 512, 1, kind=engine.KIND_COL, split=8)
    large, fill2, check2 = problem(16384, 512, 1, kind=engine.KIND_COL, split=32)
    fill()
    fill2()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        small()
    graph = _captured(torch, small, s)
    before = engine.device_alloc_count()
    with torch.cuda.stream(s):
        large()
    torch.cuda.synchronize()
    assert engine.device_alloc_count() == before + 1
    check2()
    for _ in range(2):
        fill()
        torch.cuda.synchronize()
        graph.replay()
        with torch.cuda.stream(s):
            large()
        torch.cuda.synchronize()
        check()
    shape = next(x for x in ((4, 128, 20000), (12, 64, 3000), (146, 3044, 4)) if engine.plan(2, list(x), [1, 2, 3])["split"] > 1)
    planned, fill, check = problem(*shape)
    graph = _captured(torch, planned, torch.cuda.Stream())
    fill()
    graph.replay()
    torch.cuda.synchronize()
    check()
    assert engine.device_error() == 0


# (outputs, contraction): shared by warps and clusters, and a thread's own; more than 1500 products per SM,
# from where fp64 views are summed in fixed point
FX_SHAPES = [(401, 3000), (60003, 37)]


def _fx_view(torch, a, cuda, form, wide):
    """a's view with the contracted mode second: `row` as its fastest mode, `col` as its slower
    one, on the 16-byte grid (`wide`) and off it."""
    t = torch.from_numpy(np.ascontiguousarray(a if form == "row" else a.T)).to(cuda)
    pad = 2 - t.shape[1] % 2 if wide else 1 + t.shape[1] % 2
    t = torch.nn.functional.pad(t, (0, pad))[:, :t.shape[1]]
    return t if form == "row" else t.T


@pytest.mark.parametrize("wide", [True, False], ids=["vectors", "elements"])
@pytest.mark.parametrize("form", ["row", "col"])
@pytest.mark.parametrize("shape", FX_SHAPES, ids=["shared", "own"])
@pytest.mark.parametrize("kind", ["growing", "falling", "zeros", "negative_zeros", "huge", "tiny", "mixed", "cancelling", "negative"])
def test_fp64_fixed_point_sums(engine, cuda, kind, shape, form, wide):
    """The fixed-point kernels themselves (enough products per SM): moving bases, products below the
    window, zeros of both signs, the ends of the exponent range, cancellation, negative sums.  Bar: one
    rounding per product and the result's, of sum |a b|, and of the smallest number per product."""
    import fractions
    import torch
    m, n = shape
    assert m * n > 1500 * torch.cuda.get_device_properties(0).multi_processor_count and n >= 4
    rng = np.random.default_rng(12)
    a = rng.uniform(-1, 1, (m, n))
    if kind == "growing":
        a *= np.exp2(np.linspace(-300, 300, n))
    elif kind == "falling":
        a *= np.exp2(np.linspace(300, -300, n))
    elif kind in ("zeros", "negative_zeros"):
        a[rng.uniform(size=a.shape) < 0.5] = 0.0 if kind == "zeros" else -0.0
        a[5], a[m - 1] = 0.0, -0.0
        a[7, :-1] = 0.0
    elif kind == "huge":
        a *= 2.0 ** 1009
    elif kind == "tiny":
        a *= 2.0 ** -1020
    elif kind == "mixed":
        a *= np.exp2(rng.uniform(-200, 200, a.shape))
    elif kind == "cancelling":
        a[:, 1:n // 2 * 2:2] = -a[:, 0:n // 2 * 2:2]
    else:
        a = -np.abs(a)
    b = np.ones(n) if kind == "cancelling" else rng.uniform(0.25, 1, n) if kind == "negative" else rng.uniform(-1, 1, n)
    c = engine.ttv_view(2, _fx_view(torch, a, cuda, form, wide), torch.from_numpy(b).to(cuda)).cpu().numpy()
    bs = [fractions.Fraction(y) for y in b]
    for i in sorted({0, 5, 7, m - 1, *range(1, m, 40 if n > 1000 else 600)}):
        terms = [fractions.Fraction(x) * y for x, y in zip(a[i], bs)]
        exact, absn = sum(terms), sum(abs(t) for t in terms)
        bar = absn * fractions.Fraction(4, 2 ** 53) + n * fractions.Fraction(1, 2 ** 1074)
        assert abs(fractions.Fraction(float(c[i])) - exact) <= bar, (kind, i)


@pytest.mark.parametrize("wide", [True, False], ids=["vectors", "elements"])
@pytest.mark.parametrize("form", ["row", "col"])
@pytest.mark.parametrize("shape", FX_SHAPES, ids=["shared", "own"])
def test_fp64_fixed_point_nonfinite(engine, cuda, shape, form, wide):
    """Infinities and NaNs among many products reach their output and no other."""
    import torch
    rng = np.random.default_rng(13)
    m, n = shape
    a, b = rng.uniform(-1, 1, shape), rng.uniform(0.5, 1, n)
    bad = np.zeros(m, bool)
    for i, v in ((3, np.inf), (8, np.nan), (20, -np.inf), (m - 1, np.inf), (m // 2, 1.7e308)):
        a[i, (i * 5) % n] = v
        bad[i] = True
    a[m // 2, :3] = 1.7e308
    c = engine.ttv_view(2, _fx_view(torch, a, cuda, form, wide), torch.from_numpy(b).to(cuda)).cpu().numpy()
    assert (np.isfinite(c) == ~bad).all()
    assert np.abs(c[~bad] - a[~bad] @ b).max() <= 1e-13 * n


def test_fp64_fixed_point_folds_in_time(engine, cuda):
    """A thread's sum of more products than the fixed-point accumulator holds between folds (2^18):
    one row of A broadcast over enough outputs that no two threads share a sum."""
    import fractions
    import torch
    rng = np.random.default_rng(14)
    n, m = (1 << 18) + 1003, 2048 * torch.cuda.get_device_properties(0).multi_processor_count
    a, b = rng.uniform(0.5, 1, n), rng.uniform(0.5, 1, n)
    a[1::2] *= -0.25
    c = engine.ttv_view(2, torch.from_numpy(a).to(cuda).expand(m, n), torch.from_numpy(b).to(cuda))
    terms = [fractions.Fraction(x) * fractions.Fraction(y) for x, y in zip(a, b)]
    exact, absn = sum(terms), sum(abs(t) for t in terms)
    assert (c == c[0]).all()
    assert abs(fractions.Fraction(float(c[0])) - exact) <= absn * fractions.Fraction(4, 2 ** 53)
