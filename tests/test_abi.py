"""The C ABI and the host-side logic, without a GPU.

* libttvgpu.so loads and exports every entry point include/tlibg.h declares;
* invalid calls fail with the reference's exception text, in the reference's
  order of checks (golden errors.json), before any device work;
* valid calls without a device fail loudly (no CPU fallback);
* the metadata helpers reproduce the reference's (golden metadata.json);
* the planner picks the kernel family the layout calls for;
* the C++ drop-in header compiles against the reference's own dispatch and in
  standalone mode, and maps errors to std::runtime_error with the same text;
* ttvs' contraction order bookkeeping (forward / backward / optimal).
"""
import ctypes as C
import json
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GOLDEN = os.path.join(ROOT, "tests", "golden")
HEADER = os.path.join(ROOT, "include", "tlibg.h")


def declared_symbols():
    src = open(HEADER).read()
    src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
    return sorted(set(re.findall(r"\b(tlibg_[a-z0-9_]+)\s*\(", src)))


def test_exports_every_declared_symbol(engine):
    lib = engine.library()
    syms = declared_symbols()
    assert len(syms) >= 14
    for s in syms:
        assert hasattr(lib, s), f"{s} declared in tlibg.h but not exported"


def _call(engine, dtype, q, p, na, wa, pia, nb, nc, wc, pic, a=16, b=32, c=48):
    sizes = engine._sizes
    keep = [sizes(v) for v in (na, wa, pia, nb, nc, wc, pic)]
    o = engine._options()
    return engine.library().tlibg_ttv_ex(dtype, q, p, a, *[engine._p(k) for k in keep[:3]], b,
                                         engine._p(keep[3]), c,
                                         *[engine._p(k) for k in keep[4:]], C.byref(o), None)


def test_invalid_calls_match_reference_messages(engine):
    with open(os.path.join(GOLDEN, "errors.json")) as f:
        cases = json.load(f)
    for case in cases:
        x = case["args"]
        nc = x["nc"] if x["nc"] else []
        for dt in (engine.F32, engine.F64):
            st = _call(engine, dt, x["q"], x["p"], x["na"], x["wa"], x["pia"], x["nb"], nc or [0],
                       x["wc"] or [0], x["pic"] or [0]) if x["p"] != 1 else _order1(engine, dt)
            if case["status"] == 0:
                # valid for the reference: past validation, the engine refuses the stand-in
                # pointers loudly (no device; with a device they are not device memory)
                msg = engine._last_error()
                assert st in (engine.ERR_CUDA, engine.OK) or (
                    st == engine.ERR_ARGUMENT and "device-accessible" in msg), msg
            else:
                assert st == engine.ERR_ARGUMENT
                assert engine._last_error() == case["message"]


def _order1(engine, dt):
    sizes = engine._sizes
    keep = [sizes([3]), sizes([1]), sizes([1]), sizes([3])]
    o = engine._options()
    # C of an order-1 tensor has no modes: nc is an empty range
    return engine.library().tlibg_ttv_ex(dt, 1, 1, 16, *[engine._p(k) for k in keep[:3]], 32,
                                         engine._p(keep[3]), 48, engine._p(sizes([1])),
                                         engine._p(sizes([1])), engine._p(sizes([1])), C.byref(o),
                                         None)


def test_null_pointer_checks(engine):
    na, wa, pia = [2, 3, 4], [1, 2, 6], [1, 2, 3]
    E = "Error in tlib::tensor_times_vector: "
    st = _call(engine, engine.F32, 2, 3, na, wa, pia, [3], [2, 4], [1, 2], [1, 2], a=None)
    assert st == engine.ERR_ARGUMENT
    assert engine._last_error() == E + "pointer to input tensor A should not be zero."
    st = _call(engine, engine.F32, 2, 3, na, wa, pia, [3], [2, 4], [1, 2], [1, 2], c=None)
    assert engine._last_error() == E + "pointer to output tensor C should not be zero."
    lib, o = engine.library(), engine._options()
    st = lib.tlibg_ttv_ex(0, 2, 3, 16, None, engine._p(engine._sizes(wa)),
                          engine._p(engine._sizes(pia)), 32, engine._p(engine._sizes([3])), 48,
                          engine._p(engine._sizes([2, 4])), engine._p(engine._sizes([1, 2])),
                          engine._p(engine._sizes([1, 2])), C.byref(o), None)
    assert st == engine.ERR_ARGUMENT
    assert engine._last_error() == E + "pointer to input tensor shape vector na should not be zero."


def test_non_dense_strides_are_refused(engine):
    # valid (monotone) for the reference, but not dense: outside this engine
    st = _call(engine, engine.F32, 2, 3, [2, 3, 4], [1, 3, 9], [1, 2, 3], [3], [2, 4], [1, 2],
               [1, 2])
    assert st == engine.ERR_UNSUPPORTED
    assert "dense" in engine._last_error()


def test_valid_call_without_device_fails_loudly(engine):
    import torch
    if torch.cuda.is_available():
        pytest.skip("a device is present")
    st = _call(engine, engine.F32, 2, 3, [2, 3, 4], [1, 2, 6], [1, 2, 3], [3], [2, 4], [1, 2],
               [1, 2])
    assert st == engine.ERR_CUDA
    with pytest.raises(engine.DeviceError):
        engine.ttv(2, 3, torch.zeros(24), [2, 3, 4], [1, 2, 6], [1, 2, 3], torch.zeros(3), [3],
                   torch.zeros(8), [2, 4], [1, 2], [1, 2])


def test_metadata_helpers_match_reference(engine):
    with open(os.path.join(GOLDEN, "metadata.json")) as f:
        meta = json.load(f)
    for na, q, nc in meta["output_shape"]:
        assert engine.output_shape(na, q) == nc
    for pia, q, pic in meta["output_layout"]:
        assert engine.output_layout(pia, q) == pic
    for n, pi, w in meta["strides"]:
        assert engine.strides(n, pi) == w
    for p, k, pi in meta["k_order"]:
        assert engine.k_order_layout(p, k) == pi
    for pi in ([1, 2, 3], [3, 1, 2], [2, 4, 1, 3]):
        for m in range(1, len(pi) + 1):
            assert pi[engine.inverse_mode(pi, m) - 1] == m
    with pytest.raises(engine.TTVError, match="input shape is not valid"):
        engine.output_shape([2, 0, 3], 1)
    with pytest.raises(engine.TTVError, match="input layout is not valid"):
        engine.output_layout([1, 1, 3], 1)
    with pytest.raises(engine.TTVError, match="compute_strides"):
        engine.strides([2, 3], [1, 3])


def test_planner_kernel_family(engine):
    # q-fastest rows: aligned -> register row kernel; unaligned rows of 64 or more
    # elements, many of them -> the row-shift kernel (fp32 and fp64), few -> row kernel
    assert engine.plan(1, [64, 32, 16], [1, 2, 3])["kind"] == engine.KIND_ROW
    assert engine.plan(3, [645, 645, 645], [3, 2, 1])["kind"] == engine.KIND_ROW_SHIFT
    assert engine.plan(3, [645, 645, 645], [3, 2, 1], dtype=engine.F64)["kind"] == engine.KIND_ROW_SHIFT
    assert engine.plan(1, [645, 99], [1, 2])["kind"] == engine.KIND_ROW
    assert engine.plan(3, [645, 645, 645], [3, 2, 1], vec=1)["kind"] == engine.KIND_ROW
    assert engine.plan(1, [4001, 9999], [1, 2])["kind"] == engine.KIND_ROW   # copies of b over 48 KB
    # rows that fill few rounds of lane groups are split in two (16384 rows of 16384 over the
    # lane groups of 152 SMs without a device); rows that fill many rounds are not
    assert engine.plan(1, [16384, 16384], [1, 2])["split"] == 2
    assert engine.plan(1, [16384, 16384], [1, 2], dtype=engine.F64)["split"] == 2
    assert engine.plan(1, [4096, 65536], [1, 2])["split"] == 1
    # unaligned fp32 rows under 64 elements: the row-tile kernel; aligned ones the row kernel
    assert engine.plan(3, [25, 25, 25], [3, 2, 1])["kind"] == engine.KIND_ROW_TILE
    assert engine.plan(1, [63, 99], [1, 2])["kind"] == engine.KIND_ROW_TILE
    assert engine.plan(1, [16, 99], [1, 2])["kind"] == engine.KIND_ROW
    assert engine.plan(1, [65, 99], [1, 2])["kind"] == engine.KIND_ROW
    assert engine.plan(3, [25, 25, 25], [3, 2, 1], kind=engine.KIND_STREAM)["kind"] == engine.KIND_STREAM
    # fp64 rows of at most 64 elements: the row-tile kernel (native-DFMA mode keeps the row kernel)
    assert engine.plan(1, [25, 25, 25], [1, 2, 3], dtype=engine.F64)["kind"] == engine.KIND_ROW_TILE
    assert engine.plan(1, [25, 25, 25], [1, 2, 3], dtype=engine.F64)["block"] == 128
    assert engine.plan(1, [32, 9], [1, 2], dtype=engine.F64)["kind"] == engine.KIND_ROW_TILE
    assert engine.plan(1, [33, 9], [1, 2], dtype=engine.F64)["kind"] == engine.KIND_ROW
    # fp64 rows under 8 elements: native DFMA in the row-tile kernel unless the mix is asked for
    pl = engine.plan(1, [5, 999], [1, 2], dtype=engine.F64)
    assert pl["kind"] == engine.KIND_ROW_TILE and pl["accumulate"] == engine.ACC_PLAIN
    assert engine.plan(1, [5, 999], [1, 2], dtype=engine.F64,
                       accumulate=engine.ACC_DOUBLE_FLOAT)["accumulate"] == engine.ACC_COMPENSATED
    assert engine.plan(1, [25, 25, 25], [1, 2, 3], dtype=engine.F64,
                       accumulate=engine.ACC_PLAIN)["kind"] == engine.KIND_ROW
    assert engine.plan(1, [16, 4096], [1, 2], kind=engine.KIND_ROW_TILE)["kind"] == engine.KIND_ROW_TILE
    with pytest.raises(engine.TTVError):
        engine.plan(1, [65, 9], [1, 2], kind=engine.KIND_ROW_TILE)
    with pytest.raises(engine.TTVError):
        engine.plan(2, [16, 9], [1, 2], kind=engine.KIND_ROW_TILE)
    # the TMA-staged column kernel: on request for any prefix P > 1, 288 threads
    pl = engine.plan(2, [645, 33, 7], [1, 2, 3], kind=engine.KIND_COL_BULK)
    assert pl["kind"] == engine.KIND_COL_BULK and pl["block"] == 288 and pl["vec"] == 4
    assert engine.plan(2, [645, 33, 7], [1, 2, 3], dtype=engine.F64, kind=engine.KIND_COL_BULK)["vec"] == 2
    assert engine.plan(2, [645, 33, 7], [1, 2, 3])["kind"] == engine.KIND_COL
    with pytest.raises(engine.TTVError):
        engine.plan(1, [16, 9], [1, 2], kind=engine.KIND_COL_BULK)
    assert engine.plan(1, [645, 645, 645], [1, 2, 3], dtype=engine.F64)["kind"] == engine.KIND_ROW_SHIFT
    # fp64 column kernel: the DFMA / double-float mix by default
    assert engine.plan(2, [64, 32, 16], [1, 2, 3], dtype=engine.F64)["accumulate"] == \
        engine.ACC_COMPENSATED
    assert engine.plan(2, [256, 32, 64], [1, 2, 3])["kind"] == engine.KIND_COL
    # its column form on request
    assert engine.plan(2, [645, 645, 645], [1, 2, 3], kind=engine.KIND_STREAM)["kind"] == \
        engine.KIND_STREAM
    # long rows: the register kernels (q fastest -> row kernel, else column kernel)
    assert engine.plan(1, [16384, 16384], [1, 2])["kind"] == engine.KIND_ROW
    assert engine.plan(2, [16384, 16384], [1, 2])["kind"] == engine.KIND_COL
    # prefix rows not 16-byte aligned: scalar loads (two outputs per thread); the
    # realigning kernel on request
    assert engine.plan(3, [645, 645, 645], [1, 2, 3])["kind"] == engine.KIND_COL
    assert engine.plan(3, [645, 645, 645], [1, 2, 3])["vec"] == 1
    assert engine.plan(3, [645, 645, 645], [1, 2, 3], dtype=engine.F64)["kind"] == engine.KIND_COL
    assert engine.plan(3, [645, 645, 645], [1, 2, 3], kind=engine.KIND_COL_REALIGN)["vec"] == 4
    assert engine.plan(2, [25, 25, 25], [1, 2, 3])["kind"] == engine.KIND_COL
    assert engine.plan(3, [645, 645, 645], [1, 2, 3], dtype=engine.BF16A)["kind"] == engine.KIND_COL
    assert engine.plan(2, [25, 25, 25], [1, 2, 3], kind=engine.KIND_COL_REALIGN)["kind"] == \
        engine.KIND_COL_REALIGN
    with pytest.raises(engine.TTVError, match="realigning column kernel"):
        engine.plan(1, [25, 25, 25], [1, 2, 3], kind=engine.KIND_COL_REALIGN)
    # thin prefix, few outputs, long contraction: several rows per warp step
    assert engine.plan(2, [64, 1 << 22], [1, 2])["kind"] == engine.KIND_COL_THIN
    assert engine.plan(2, [16, 1 << 20, 16], [1, 2, 3])["kind"] == engine.KIND_COL_THIN
    assert engine.plan(2, [64, 1 << 22], [1, 2], dtype=engine.F64)["kind"] == engine.KIND_COL_THIN
    assert engine.plan(2, [16, 16, 1 << 20], [1, 2, 3])["kind"] == engine.KIND_COL   # many outputs
    with pytest.raises(engine.TTVError, match="thin-prefix column kernel"):
        engine.plan(2, [24, 1000], [1, 2], kind=engine.KIND_COL_THIN)
    # forced register kernels
    R, Cn = engine.KIND_ROW, engine.KIND_COL
    assert engine.plan(1, [64, 32, 16], [1, 2, 3], kind=R)["kind"] == R
    assert engine.plan(3, [64, 32, 16], [3, 2, 1], kind=R)["kind"] == R
    pl = engine.plan(2, [256, 256, 256], [1, 2, 3], kind=Cn)
    assert (pl["P"], pl["nq"], pl["S"]) == (256, 256, 256)
    assert pl["vec"] == 4 and pl["accumulate"] == engine.ACC_COMPENSATED
    # odd prefix: scalar loads; fp64: 2 per 16-byte load; bf16: 8
    assert engine.plan(2, [25, 25, 25], [1, 2, 3], kind=Cn)["vec"] == 1
    assert engine.plan(2, [256, 256, 256], [1, 2, 3], dtype=engine.F64, kind=Cn)["vec"] == 2
    assert engine.plan(2, [256, 256, 256], [1, 2, 3], dtype=engine.BF16A, kind=Cn)["vec"] == 8
    with pytest.raises(engine.TTVError, match="streamed kernel"):
        engine.plan(1, [16384, 16384], [1, 2], kind=engine.KIND_STREAM)
    # long contraction with a thin prefix is split, and segments fit the staged b
    pl = engine.plan(2, [64, 1 << 22], [1, 2], kind=Cn)
    assert pl["kind"] == Cn and pl["split"] >= (1 << 22) // 4096
    assert engine.plan(2, [64, 1 << 22], [1, 2], kind=engine.KIND_STREAM)["split"] > 1
    # forced options are honoured or refused
    assert engine.plan(2, [256, 256, 256], [1, 2, 3], kind=Cn, group=2, split=3)["group"] == 2
    with pytest.raises(engine.TTVError):
        engine.plan(1, [256, 256, 256], [1, 2, 3], kind=engine.KIND_COL)


def _compile_cpp(tmp_path, standalone):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ missing")
    import oracle
    ref_inc = oracle.REF_INCLUDE   # the staged reference headers (or TTV_REFERENCE_INCLUDE)
    if not standalone and not os.path.isdir(os.path.join(ref_inc, "tlib")):
        pytest.skip("reference headers absent")
    exe = str(tmp_path / ("kat_sa" if standalone else "kat_ref"))
    cuda_inc = "/usr/local/cuda/include"
    cmd = [gxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"), "-I", cuda_inc,
           os.path.join(ROOT, "tests", "cpp", "ttv_gpu_kat.cpp"), "-o", exe,
           "-L", os.path.join(ROOT, "ttv_gb300"), "-lttvgpu", "-L/usr/local/cuda/lib64",
           "-lcudart", "-Wl,-rpath," + os.path.join(ROOT, "ttv_gb300")]
    if standalone:
        cmd.insert(2, "-DTLIBG_STANDALONE")
    else:
        cmd[3:3] = ["-I", ref_inc, "-fopenmp"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


@pytest.mark.parametrize("standalone", [False, True])
def test_cpp_header_dispatch_and_messages(engine, tmp_path, standalone):
    exe = _compile_cpp(tmp_path, standalone)
    r = subprocess.run([exe, "validate"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "PASSED" in r.stdout


def test_ttvs_contraction_order(engine, monkeypatch):
    """ttvs' mode bookkeeping against the reference's Python tests
    (ttvpy/tests/test.py), with the per-step TTV done by einsum on the CPU."""
    import torch

    def cpu_ttv(q, A, b, **kw):
        return torch.tensordot(A, b, dims=([q - 1], [0]))

    monkeypatch.setattr(engine, "ttv_array", cpu_ttv)
    A = torch.arange(3 * 2 * 4 * 5, dtype=torch.float64).reshape(3, 2, 4, 5)
    for q in range(1, 5):
        dims = [d for d in range(4) if d != q - 1]
        B = [torch.arange(A.shape[d], dtype=torch.float64) for d in dims]
        D = A
        for d, bj in sorted(zip(dims, B), key=lambda t: -t[0]):
            D = torch.tensordot(D, bj, dims=([d], [0]))
        for order in ("forward", "backward", "optimal"):
            Cq = engine.ttvs(q, A, B, order, fused=False)
            assert torch.equal(Cq, D), (q, order)
    with pytest.raises(ValueError, match="multiplication order"):
        engine.ttvs(1, A, B, "sideways")
    with pytest.raises(ValueError, match="number of input vectors"):
        engine.ttvs(1, A, B[:2])


def test_ttvs_entry_point_checks(engine):
    """tlibg_ttvs refuses bad calls with ttvpy's messages before touching memory."""
    import ctypes as C
    lib = engine.library()
    buf = (C.c_float * 64)()
    vec = (C.c_void_p * 3)(C.addressof(buf), C.addressof(buf), C.addressof(buf))

    def call(q, p, na, nbs, pia=None):
        pia = pia or list(range(1, p + 1))
        wa = engine.strides(na, pia) if p else [1]
        keep = [engine._sizes(v) for v in (na or [1], wa, pia or [1], nbs or [1])]
        st = lib.tlibg_ttvs(engine.F32, q, p, C.addressof(buf), engine._p(keep[0]), engine._p(keep[1]),
                            engine._p(keep[2]), vec, engine._p(keep[3]), C.addressof(buf), None)
        return st, engine._last_error()

    assert call(1, 0, [], []) == (engine.ERR_ARGUMENT, "Error calling ttvpy::ttvs: input tensor "
                                  "order should be greater than zero.")
    st, msg = call(5, 4, [2, 3, 4, 5], [2, 3, 4])
    assert st == engine.ERR_ARGUMENT and "contraction mode should be greater than zero" in msg
    st, msg = call(2, 4, [2, 3, 4, 5], [2, 4, 4])
    assert st == engine.ERR_ARGUMENT and msg == ("Error calling ttvpy::ttvs: vector dimension is not "
                                                 "compatible with the dimension of a tensor mode.")
    st, msg = call(1, 1, [7], [])
    assert st == engine.ERR_ARGUMENT and "order 1" in msg
    # a valid call gets as far as the device (none here)
    import torch
    if not torch.cuda.is_available():
        st, msg = call(2, 4, [2, 3, 4, 5], [2, 4, 5])
        assert st in (engine.ERR_CUDA, engine.ERR_ARGUMENT), msg


def test_ttvs_truth_matches_einsum(orc):
    """The oracle's chain truth (Kronecker weights, double-double sum) against
    float64 tensordot chains, for first- and last-order layouts."""
    rng = np.random.default_rng(8)
    na = [5, 3, 4, 6]
    A = rng.uniform(-1, 1, int(np.prod(na)))
    for pia in ([1, 2, 3, 4], [4, 3, 2, 1], [2, 4, 1, 3]):
        # the tensor with layout pia: element (i1..i4) at sum i_r w_r
        wa = orc.strides(na, pia)
        T = np.zeros(na)
        for idx in np.ndindex(*na):
            T[idx] = A[sum(i * w for i, w in zip(idx, wa))]
        for q in range(1, 5):
            bs = [rng.uniform(-1, 1, na[m]) for m in range(4) if m != q - 1]
            D = T
            for d, bj in sorted(zip([m for m in range(4) if m != q - 1], bs), key=lambda t: -t[0]):
                D = np.tensordot(D, bj, axes=([d], [0]))
            ref, absn = orc.ttvs_truth(q, A, na, pia, bs)
            assert np.allclose(ref, D, rtol=0, atol=1e-13), (pia, q)


def test_validate_only_entry_point(engine):
    """tlibg_validate runs the reference's checks on metadata alone."""
    L, sz = engine.library(), engine._sizes
    ok = [sz(v) for v in ([4, 5, 6], [1, 4, 20], [1, 2, 3], [5], [4, 6], [1, 4], [1, 2])]
    assert L.tlibg_validate(2, 3, *[engine._p(k) for k in ok]) == 0
    bad = list(ok)
    bad[3] = sz([7])
    assert L.tlibg_validate(2, 3, *[engine._p(k) for k in bad]) == 1
    assert "contraction dimension of A and B are not equal" in engine._last_error()


def test_undersized_tensors_are_refused_before_launch(engine):
    """Tensors smaller than their layout addresses never reach a kernel; the
    reference's own messages still come first."""
    torch = pytest.importorskip("torch")
    na, pia, q = [4, 5, 6], [1, 2, 3], 2
    wa = engine.strides(na, pia)
    nc, pic = engine.output_shape(na, q), engine.output_layout(pia, q)
    wc = engine.strides(nc, pic)
    a, b, c = torch.zeros(120), torch.zeros(5), torch.zeros(24)
    for small in ("a", "b", "c"):
        args = {"a": a, "b": b, "c": c}
        args[small] = args[small][:-1]
        with pytest.raises(engine.TTVError, match=f"buffer {small} holds"):
            engine.ttv(q, 3, args["a"], na, wa, pia, args["b"], [5], args["c"], nc, wc, pic)
    with pytest.raises(engine.TTVError, match="contraction dimension of A and B are not equal"):
        engine.ttv(q, 3, a[:1], na, wa, pia, b, [4], c, nc, wc, pic)


def test_element_misaligned_pointers_refused(engine):
    """Pointers not aligned to their element type never reach a kernel."""
    sz = engine._sizes
    meta = [sz(v) for v in ([4, 5, 6], [1, 4, 20], [1, 2, 3], [5], [4, 6], [1, 4], [1, 2])]
    L = engine.library()
    o = engine._options()
    for dt, a, b, c in ((engine.F32, 18, 32, 64), (engine.F64, 20, 32, 64), (engine.F64, 64, 36, 64),
                        (engine.F32, 64, 32, 66)):
        st = L.tlibg_ttv_ex(dt, 2, 3, a, *[engine._p(k) for k in meta[:3]], b, engine._p(meta[3]), c,
                            *[engine._p(k) for k in meta[4:]], C.byref(o), None)
        assert st == engine.ERR_UNSUPPORTED, (dt, a, b, c, st)
        assert "aligned to their element sizes" in engine._last_error()


def test_pointer_location_without_device(engine):
    """No device in this process: every pointer is a host pointer; null is unknown."""
    import ctypes
    L = engine.library()
    L.tlibg_pointer_location.argtypes = [ctypes.c_void_p]
    buf = ctypes.create_string_buffer(64)
    assert L.tlibg_pointer_location(None) == -1
    try:
        import torch
        has_gpu = torch.cuda.is_available()
    except ImportError:
        has_gpu = False
    if not has_gpu:
        assert L.tlibg_pointer_location(ctypes.addressof(buf)) == 0


def test_strided_extension_checks(engine):
    """tlibg_ttv_strided's host checks (no device needed): the reference's messages
    for shapes, layouts and monotonic strides; C strides that make two outputs
    share an element, b's zero stride and bf16 storage refused."""
    lib = engine.library()
    def call(na, wa, pia, q, nc, wc, pic, wb=1, dtype=engine.F32):
        keep = [engine._sizes(v) for v in (na, wa, pia, [na[q - 1]], nc, wc, pic)]
        st = lib.tlibg_ttv_strided(dtype, q, len(na), 16, engine._p(keep[0]), engine._p(keep[1]),
                                   engine._p(keep[2]), 32, engine._p(keep[3]), wb, 48, engine._p(keep[4]),
                                   engine._p(keep[5]), engine._p(keep[6]), None)
        return st, engine._last_error()
    # C's strides overlap (both modes stride 1)
    st, msg = call([4, 5, 6], [1, 4, 20], [1, 2, 3], 2, [4, 6], [1, 1], [1, 2])
    assert st == engine.ERR_UNSUPPORTED and "share an element" in msg
    # A's strides not monotonic along its layout: the reference's message
    st, msg = call([4, 5, 6], [20, 4, 1], [1, 2, 3], 2, [4, 6], [1, 4], [1, 2])
    assert st == engine.ERR_ARGUMENT and "stride" in msg
    # b's stride zero
    st, msg = call([4, 5, 6], [1, 4, 20], [1, 2, 3], 2, [4, 6], [1, 4], [1, 2], wb=0)
    assert st == engine.ERR_ARGUMENT and "b's stride" in msg
    # bf16-stored A is not taken here
    st, msg = call([4, 5, 6], [1, 4, 20], [1, 2, 3], 2, [4, 6], [1, 4], [1, 2], dtype=engine.BF16A)
    assert st == engine.ERR_UNSUPPORTED
    # valid padded metadata passes the host checks (then needs a device)
    st, msg = call([4, 5, 6], [1, 5, 40], [1, 2, 3], 2, [4, 6], [1, 7], [1, 2])
    assert st in (engine.ERR_CUDA, engine.ERR_ARGUMENT, engine.OK)
    if st == engine.ERR_ARGUMENT:
        assert "device-accessible" in msg


def _packed(engine, dtype, q, p, ptrs, sizes, words, opts=(0, -1, 0, 0, 0, 0)):
    import struct
    return struct.pack(f"=10Q6q{len(words)}Q", dtype, q, p, *ptrs, *sizes, 0, *opts, *words)


def _outcome(engine, st):
    msg = engine._last_error()
    # past every host check: no device, or (with one) the stand-in pointers refused
    if st in (engine.ERR_CUDA, engine.OK) or (st == engine.ERR_ARGUMENT and "device-accessible" in msg):
        return "passed the checks"
    return st, msg


def _mutated(rng, p):
    """Metadata of an order-p call, valid or with one or two entries spoiled."""
    na = [int(x) for x in rng.integers(1, 6, p)]
    pia = [int(x) + 1 for x in rng.permutation(p)]
    q = int(rng.integers(1, p + 1))
    wa, acc = [0] * p, 1
    for m in pia:
        wa[m - 1], acc = acc, acc * na[m - 1]
    nc = [n for m, n in enumerate(na) if m != q - 1]
    pic = [m - (m > q) for m in pia if m != q]
    wc, acc = [0] * (p - 1), 1
    for m in pic:
        wc[m - 1], acc = acc, acc * nc[m - 1]
    nb = [na[q - 1]]
    lists = [na, wa, pia, nb, nc, wc, pic]
    for _ in range(int(rng.integers(0, 3))):
        v = lists[int(rng.integers(0, 7))]
        v[int(rng.integers(0, len(v)))] = int(rng.choice([0, 1, 2, 3, 7, 1000, 2 ** 33, 2 ** 63]))
    if rng.random() < 0.1:
        q = int(rng.choice([0, p + 1, 2 ** 63]))
    return q, lists


def test_packed_calls_answer_like_the_general_ones(engine):
    """The packed forms give the general calls' status and message on 4000 random calls, valid
    and spoiled, at every dtype, through the dense and the strided entry points."""
    lib = engine.library()
    rng = np.random.default_rng(20)
    big = 2 ** 64 - 1
    seen = set()
    for _ in range(4000):
        p = int(rng.integers(2, 6))
        q, lists = _mutated(rng, p)
        na, wa, pia, nb, nc, wc, pic = lists
        dt = int(rng.integers(0, 4))
        ptrs = [int(x) for x in rng.choice([0, 16, 16, 16, 18, 4096], 3)]
        flat = [x for v in lists for x in v]
        general = _outcome(engine, _call(engine, dt, q, p, *lists, *ptrs))
        packed = _outcome(engine, lib.tlibg_ttv_packed(_packed(engine, dt, q, p, ptrs, (big,) * 3, flat)))
        assert packed == general, (q, lists, dt, ptrs)
        seen.add(general)
        wb = int(rng.choice([0, 1, 3]))
        keep = [engine._sizes(v) for v in lists]
        st = lib.tlibg_ttv_strided(dt, q, p, ptrs[0], *[engine._p(k) for k in keep[:3]], ptrs[1], engine._p(keep[3]),
                                   wb, ptrs[2], *[engine._p(k) for k in keep[4:]], None)
        general = _outcome(engine, st)
        packed = _outcome(engine, lib.tlibg_ttv_strided_packed(
            _packed(engine, dt, q, p, ptrs, (big,) * 3, flat + [wb])))
        assert packed == general, (q, lists, dt, ptrs, wb)
    assert len(seen) > 12


def test_packed_calls_check_buffer_sizes(engine):
    """Sizes are compared with what the layouts address, after the metadata checks; strides whose
    span passes 64 bits count as too large, not as small."""
    lib = engine.library()
    q, p, lists = 1, 3, [[4, 5, 6], [1, 4, 20], [1, 2, 3], [4], [5, 6], [1, 5], [1, 2]]
    flat = [x for v in lists for x in v]
    for dt, (ea, et) in ((0, (4, 4)), (1, (8, 8)), (2, (2, 4))):
        need = [120 * ea, 4 * et, 30 * et]
        for i in range(3):
            short = list(need)
            short[i] -= 1
            st = lib.tlibg_ttv_packed(_packed(engine, dt, q, p, (16, 32, 48), short, flat))
            assert (st, engine._last_error()) == (engine.ERR_ARGUMENT, f"tlibg: buffer {'abc'[i]} holds {short[i]} "
                                                                       f"bytes, its layout addresses {need[i]}")
        assert _outcome(engine, lib.tlibg_ttv_packed(
            _packed(engine, dt, q, p, (16, 32, 48), need, flat))) == "passed the checks"
        # C's strides do not matter to the reference here (q fastest), but the buffer check counts them
        lists2 = [list(v) for v in lists]
        lists2[5] = [2 ** 62, 2 ** 63]
        st = lib.tlibg_ttv_packed(_packed(engine, dt, q, p, (16, 32, 48), need, [x for v in lists2 for x in v]))
        assert st == engine.ERR_ARGUMENT and "buffer c holds" in engine._last_error()


def test_packed_rowmajor_derives_the_metadata(engine):
    """tlibg_ttv_packed_rowmajor answers as the packed call with the metadata helpers' layout."""
    lib = engine.library()
    rng = np.random.default_rng(5)
    for _ in range(400):
        p = int(rng.integers(2, 7))
        na = [int(x) for x in rng.integers(1, 5, p)]
        q = int(rng.integers(1, p + 1))
        pia = list(range(p, 0, -1))
        wa = [int(np.prod(na[r + 1:])) for r in range(p)]
        if rng.random() < 0.2:
            wa[int(rng.integers(0, p))] = int(rng.integers(0, 9))
        nb = na[q - 1] + (1 if rng.random() < 0.1 else 0)
        nc, pic = engine.output_shape(na, q), engine.output_layout(pia, q)
        wc = engine.strides(nc, pic)
        need = [4 * (1 + sum((n - 1) * w for n, w in zip(na, wa))), 4 * nb, 4 * int(np.prod(nc))]
        if rng.random() < 0.2:
            need[int(rng.integers(0, 3))] -= 4
        a = _outcome(engine, lib.tlibg_ttv_packed(
            _packed(engine, 0, q, p, (16, 32, 48), need, [*na, *wa, *pia, nb, *nc, *wc, *pic])))
        b = _outcome(engine, lib.tlibg_ttv_packed_rowmajor(
            _packed(engine, 0, q, p, (16, 32, 48), need, [*na, *wa, nb])))
        assert a == b, (na, q, wa, nb)


def test_python_calls_keep_their_answers(engine):
    """Arguments the packed form does not take (None, floats, longer lists, raw addresses, empty
    tensors) go through the general one: the same errors as before."""
    import torch
    t = torch.zeros(120)
    b, c = torch.zeros(4), torch.zeros(30)
    meta = ([4, 5, 6], [1, 4, 20], [1, 2, 3])
    out = ([5, 6], [1, 5], [1, 2])
    with pytest.raises(engine.TTVError, match="pointer to input tensor shape vector na should not be zero"):
        engine.ttv(1, 3, 16, None, *meta[1:], 32, [4], 48, *out)
    with pytest.raises((engine.DeviceError, engine.TTVError), match="CUDA|device"):
        engine.ttv(1, 3, t, [4.0, 5.0, 6.0], *meta[1:], b, [4], c, *out)
    with pytest.raises((engine.DeviceError, engine.TTVError), match="CUDA|device"):
        engine.ttv(1, 3, t, [4, 5, 6, 9], *meta[1:], b, (4,), c, *out)
    with pytest.raises(engine.TTVError, match="shape vector of A is not valid"):
        engine.ttv(1, 3, torch.zeros(0), [4, 0, 6], *meta[1:], b, [4], c, *out)
    with pytest.raises(engine.TTVError, match="contraction mode should be greater zero"):
        engine.ttv(-1, 3, t, *meta, b, [4], c, *out)
    with pytest.raises(TypeError):
        engine.ttv(1, 3, t, *meta, b, [4], c, *out, no_such_option=1)
    with pytest.raises(engine.TTVError, match="contraction dimension of A and B are not equal"):
        engine.ttv_array(2, torch.zeros(4, 5), torch.zeros(4))


def _general(engine, dtype, P, nq, S):
    pl = engine.plan(2, [P, nq, S], [1, 2, 3], dtype=dtype)
    return pl["kind"], pl["cluster"] > 0


def test_plan_tells_the_two_column_kernels_apart(engine):
    """plan() names the kernels that run: general-stride plans carry their cluster size, and their
    kind, group, vec and split as options are a dense plan's."""
    pl = engine.plan(2, [256, 256, 256], [1, 2, 3])
    assert pl["kind"] == engine.KIND_COL and pl["cluster"] >= 1
    back = engine.plan(2, [256, 256, 256], [1, 2, 3], kind=pl["kind"], group=pl["group"], vec=pl["vec"], split=pl["split"])
    assert back["cluster"] == 0
    assert engine.plan(2, [645, 645, 645], [1, 2, 3])["cluster"] == 0
    assert engine.plan(1, [64, 12], [1, 2], kind=engine.KIND_ROW)["cluster"] == 0


def test_unsplit_rows_leave_the_dense_kernel_only_in_whole_blocks(engine):
    """fp32 rows of a multiple of 64 elements run on the general-stride kernel where every lane's
    loads are whole blocks of four, and on the dense kernel, faster there, where they are not."""
    for nq in (128, 192, 384, 512, 1536, 2048):
        assert _general(engine, engine.F32, 1, nq, (1 << 27) // nq) == (engine.KIND_ROW, True), nq
    for nq in (320, 448, 576, 640, 704, 960, 1088, 1344, 1920):
        assert _general(engine, engine.F32, 1, nq, (1 << 27) // nq) == (engine.KIND_ROW, False), nq


def test_short_contractions_stay_on_the_dense_kernels(engine):
    """A few rows of large column problems: bf16 storage up to 6 rows (over 2 of them only below
    2^26 elements), fp64 up to 8 from 2^22 elements on."""
    for P, nq, S, general in ((32768, 1, 4096, False), (32768, 2, 1024, False), (4096, 4, 2048, False), (4096, 6, 1365, False),
                              (4096, 4, 1 << 15, True), (4096, 8, 2048, True), (4096, 12, 1365, True)):
        assert _general(engine, engine.BF16A, P, nq, S) == (engine.KIND_COL, general), (P, nq, S)
    for P, nq, S, general in ((32768, 1, 512, False), (32768, 3, 170, False), (512, 8, 4096, False), (4096, 5, 819, False),
                              (32768, 3, 10, True), (32768, 4, 8, True)):
        assert _general(engine, engine.F64, P, nq, S) == (engine.KIND_COL, general), (P, nq, S)


def test_thin_prefixes_stay_on_their_kernel_in_one_wave(engine):
    """Slabs that all have a resident CTA, and a few split ones of narrow prefixes: the thin kernel;
    a few rows, long slabs and many slabs: the general-stride kernels."""
    thin, gs = (engine.KIND_COL_THIN, False), (engine.KIND_COL, True)
    for dt, P, nq, S, want in ((engine.F32, 2, 256, 200, thin), (engine.F32, 8, 512, 256, thin), (engine.F32, 16, 64, 200, thin),
                               (engine.F32, 8, 1900, 4, thin), (engine.F32, 64, 4, 200, gs), (engine.F32, 8, 9, 400, gs),
                               (engine.F32, 64, 200, 12, gs), (engine.F32, 16, 5, 3000, gs),
                               (engine.BF16A, 2, 64, 256, thin), (engine.BF16A, 8, 100, 200, thin), (engine.BF16A, 2, 256, 1500, thin),
                               (engine.BF16A, 8, 9, 200, gs), (engine.BF16A, 2, 32, 8000, gs),
                               (engine.F64, 2, 256, 200, thin), (engine.F64, 8, 200, 2, thin), (engine.F64, 8, 700, 2, gs)):
        assert _general(engine, dt, P, nq, S) == want, (dt, P, nq, S)


def test_sizes_past_64_bits_are_told_in_full(engine):
    """Layouts that span more than 64 bits' worth of bytes: the message gives the whole number."""
    lists = [[4, 5, 6], [1, 4, 20], [1, 2, 3], [4], [5, 6], [2 ** 62, 2 ** 63], [1, 2]]
    flat = [x for v in lists for x in v]
    st = engine.library().tlibg_ttv_packed(_packed(engine, 0, 1, 3, (16, 32, 48), (480, 16, 120), flat))
    assert st == engine.ERR_ARGUMENT
    assert engine._last_error() == f"tlibg: buffer c holds 120 bytes, its layout addresses {4 * (1 + 4 * 2 ** 62 + 5 * 2 ** 63)}"


def test_array_call_refuses_modes_as_before(engine):
    """Modes that are no integers or out of range are refused before anything is allocated."""
    import ctypes
    import torch
    A, b = torch.zeros(4, 5), torch.zeros(5)
    with pytest.raises(ctypes.ArgumentError):
        engine.ttv_array(1.0, A, b)
    for q in (-1, 3, 9):
        with pytest.raises((engine.TTVError, ValueError), match="mode"):
            engine.ttv_array(q, A, b)


def test_small_buffers_are_told_before_unsupported_strides(engine):
    """A call that is both too small and not dense is refused for its buffer, as the general form does."""
    na, wa, c = [4, 5, 6], [1, 8, 40], [5, 6]
    flat = [x for v in (na, wa, [1, 2, 3], [4], c, [1, 5], [1, 2]) for x in v]
    need = 4 * (1 + 3 + 4 * 8 + 5 * 40)
    call = engine.library().tlibg_ttv_packed
    assert call(_packed(engine, 0, 1, 3, (16, 32, 48), (480, 16, 120), flat)) == engine.ERR_ARGUMENT
    assert engine._last_error() == f"tlibg: buffer a holds 480 bytes, its layout addresses {need}"
    assert call(_packed(engine, 0, 1, 3, (16, 32, 48), (need, 16, 120), flat)) == engine.ERR_UNSUPPORTED
    assert "dense tensor A" in engine._last_error()
