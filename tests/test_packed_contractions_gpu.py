"""Contractions whose operands the tensor maps cannot describe where they lie: they are gathered into
padded rows first and run on the tensor-core path.  Sizes at the edges of that copy: odd row lengths
in either layout, one element short of and past a 16-byte group, axes made of several loops, affine
positions, odd output rows.  16-bit operands: the tolerance of bf16 contractions; single-precision
operands travel as tf32 pairs and keep the tolerance of single precision."""
import numpy as np
import pytest

from ocannl_b200 import workloads as W
from ocannl_b200.low_level import Affine, Routine, Seq, Set, loops, un
from tests.parity import compare, run_device, run_oracle

pytestmark = pytest.mark.gpu


def _mm(b, m, n, k, prec, a_mmajor, b_nmajor, act):
    r = Routine("packed_%d_%d_%d_%d" % (b, m, n, k))
    x = r.tn("x", prec, [b, k, m] if a_mmajor else [b, m, k], read_only=True)
    w = r.tn("w", prec, [b, k, n] if b_nmajor else [b, n, k], read_only=True)
    bias = r.tn("bias", "single", [n], read_only=True)
    y = r.tn("y", prec, [b, m, n])
    ib, i, j, kk = r.syms(4)
    acc = W.reduce_scope(r, "acc", "single", [(kk, k)], lambda: (x[ib, kk, i] if a_mmajor else x[ib, i, kk],
                                                                 w[ib, kk, j] if b_nmajor else w[ib, j, kk]), orig=(ib, i, j))
    v = acc + bias[j]
    r.body = Seq([loops([(ib, b), (i, m), (j, n)], Set(y, (ib, i, j), un("relu", v) if act else v))])
    return r


def _inputs(ir, k, seed=5):
    g = np.random.default_rng(seed)
    return {t.ident: W.store(t.prec, (g.standard_normal(t.dims) / (np.sqrt(k) if t.ident in ("w", "kernel") else 1.0)).astype(np.float32))
            for t in ir.params() if t.read_only}


@pytest.mark.parametrize("shape", [(1, 333, 77, 131), (3, 129, 255, 33), (2, 64, 65, 519), (1, 300, 9, 1001)])
@pytest.mark.parametrize("a_mmajor,b_nmajor", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("prec", ["bfloat16", "half", "single"])
def test_odd_rows(device, shape, a_mmajor, b_nmajor, prec):
    ir = _mm(*shape, prec, a_mmajor, b_nmajor, act=a_mmajor == b_nmajor)
    inputs = _inputs(ir, shape[3])
    want = run_oracle(ir, inputs)
    got, info = run_device(device, ir, inputs)
    kinds = [s["kind"] for s in info["stages"]]
    assert kinds[-1] == "gemm" and "gathers operands" in info["stages"][0]["note"], info
    tol = dict(rtol=1e-5, atol=2e-6) if prec == "single" else dict(rtol=2e-2, atol=2e-3)
    compare(ir, got, want, only=["y"], **tol)


@pytest.mark.parametrize("cin,cout,kernel,stride", [(3, 40, 3, 1), (8, 17, 5, 2), (16, 32, 3, 1)])
@pytest.mark.parametrize("prec", ["bfloat16", "single"])
def test_convolution_patches(device, cin, cout, kernel, stride, prec):
    """Patches of an image (positions `stride * o + k`) against a kernel: m is (image, row, column),
    k is (kernel row, kernel column, channel)."""
    batch, size = 3, 21
    out = (size - kernel) // stride + 1
    r = Routine("patches_%d_%d_%d_%d" % (cin, cout, kernel, stride))
    x = r.tn("x", prec, [batch, size, size, cin], read_only=True)
    w = r.tn("kernel", prec, [cout, kernel, kernel, cin], read_only=True)
    y = r.tn("y", prec, [batch, out, out, cout])
    ib, oh, ow, co, kh, kw, ci = r.syms(7)
    at = lambda: x[ib, Affine(((stride, oh), (1, kh))), Affine(((stride, ow), (1, kw))), ci]
    acc = W.reduce_scope(r, "acc", "single", [(kh, kernel), (kw, kernel), (ci, cin)], lambda: (w[co, kh, kw, ci], at()), orig=(ib, oh, ow, co))
    r.body = Seq([loops([(ib, batch), (oh, out), (ow, out), (co, cout)], Set(y, (ib, oh, ow, co), un("relu", acc)))])
    if 2 * batch * out * out * cout * kernel * kernel * cin < 4e6:      # below the size the tensor cores are used from
        pytest.skip("small")
    inputs = _inputs(r, kernel * kernel * cin)
    want = run_oracle(r, inputs)
    got, info = run_device(device, r, inputs)
    assert [s["kind"] for s in info["stages"]][-1] == "gemm", info
    tol = dict(rtol=1e-5, atol=2e-6) if prec == "single" else dict(rtol=2e-2, atol=2e-3)
    compare(r, got, want, only=["y"], **tol)


def convolution(batch, size, cin, cout, kh, kw, stride, prec):
    """relu of a `valid` convolution with kh x kw kernels, as the reference lowers it."""
    oh_, ow_ = (size - kh) // stride + 1, (size - kw) // stride + 1
    r = Routine("conv_%d_%d_%d_%dx%d_%d" % (size, cin, cout, kh, kw, stride))
    x = r.tn("x", prec, [batch, size, size, cin], read_only=True)
    w = r.tn("kernel", prec, [cout, kh, kw, cin], read_only=True)
    y = r.tn("y", prec, [batch, oh_, ow_, cout])
    ib, oh, ow, co, i, j, ci = r.syms(7)
    at = lambda: x[ib, Affine(((stride, oh), (1, i))), Affine(((stride, ow), (1, j))), ci]
    acc = W.reduce_scope(r, "acc", "single", [(i, kh), (j, kw), (ci, cin)], lambda: (w[co, i, j, ci], at()), orig=(ib, oh, ow, co))
    r.body = Seq([loops([(ib, batch), (oh, oh_), (ow, ow_), (co, cout)], Set(y, (ib, oh, ow, co), un("relu", acc)))])
    return r


@pytest.mark.parametrize("cin,cout,kh,kw,stride", [(64, 256, 1, 1, 1), (64, 256, 1, 1, 2), (64, 128, 1, 5, 1), (32, 64, 3, 3, 1)])
@pytest.mark.parametrize("prec", ["bfloat16", "single"])
def test_patches_that_lie_on_a_tensor_map(device, cin, cout, kh, kw, stride, prec):
    """Kernels one row high have patches that a tensor map can describe where they lie, overlapping ones among
    them (1 x 5); higher ones do not.  16-bit patches are read there, without a copy; single precision keeps its
    precision whatever the kernel."""
    ir = convolution(8, 40, cin, cout, kh, kw, stride, prec)
    inputs = _inputs(ir, kh * kw * cin)
    want = run_oracle(ir, inputs)
    got, info = run_device(device, ir, inputs)
    kinds = [s["kind"] for s in info["stages"]]
    assert kinds == (["gemm"] if prec == "bfloat16" and kh == 1 else ["generic", "gemm"]), info
    tol = dict(rtol=1e-5, atol=2e-6) if prec == "single" else dict(rtol=2e-2, atol=2e-3)
    compare(ir, got, want, only=["y"], **tol)


@pytest.mark.parametrize("cfg", [dict(batch=8, size=16, cin=8, cout=16), dict(batch=5, size=23, cin=3, cout=33, kernel=5),
                                 dict(batch=40, size=17, cin=8, cout=20, stride=2)])
@pytest.mark.parametrize("prec", ["bfloat16", "single"])
def test_convolution_gradients_by_windows(device, cfg, prec):
    """The input gradient as a contraction per window and a gathering kernel, the kernel gradient as a
    contraction over all positions; strides of one and two, odd images."""
    ir = W.conv2d_update(prec=prec, **cfg)
    inputs = W.conv2d_inputs(prec=prec, **cfg)
    want = run_oracle(ir, inputs)
    got, info = run_device(device, ir, inputs)
    assert any("gathers the windows" in s["note"] for s in info["stages"]), [s["note"] for s in info["stages"]]
    for name in ("y", "loss", "z_grad", "bias_grad", "kernel_grad", "x_padded_grad"):
        w, g = (W.load(prec, a[name]) if a[name].dtype == np.uint16 else a[name] for a in (want, got))
        scale = float(np.abs(w).max())
        np.testing.assert_allclose(g, w, rtol=2e-2 if prec != "single" else 1e-4, atol=(2e-2 if prec != "single" else 1e-5) * scale, err_msg=name)


def test_extreme_values_in_two_parts(device):
    """A two-part product keeps what single precision has: an infinite operand times a finite one is infinite,
    infinity times zero and anything with a NaN is NaN, infinities of either sign in one sum are NaN, and
    values next to the largest float multiply like any other."""
    m, n, k = 130, 77, 333
    ir = _mm(1, m, n, k, "single", False, False, act=False)
    inputs = _inputs(ir, k)
    x, w = inputs["x"].reshape(m, k), inputs["w"].reshape(n, k)
    big = np.finfo(np.float32).max
    x[0, 5], x[1, 332], x[2, 7], x[3, 0] = np.inf, -np.inf, np.nan, np.inf
    x[3, 1] = -np.inf                                # of both signs in one row
    w[4, 5] = 0.0                                    # meets the first infinity
    w[6, 9] = np.inf                                 # an infinity on the other side, and one that meets an infinity
    x[8, 9] = -np.inf
    x[9, :], x[10, :], x[11, :] = 0.0, 0.0, 0.0
    x[9, 3], x[10, 3], x[11, 3] = big, np.nextafter(big, np.float32(0)), -big * np.float32(1 - 2.0 ** -12)
    w[:, 3] = np.random.default_rng(2).uniform(0.1, 0.9, n).astype(np.float32)
    w[12, 3], w[13, 3] = 1.0, 1e-34
    want = run_oracle(ir, inputs)
    got, info = run_device(device, ir, inputs)
    assert info["stages"][-1]["kind"] == "gemm" and "tf32 pairs" in info["stages"][0]["note"], info
    g, w_ = got["y"].reshape(m, n).astype(np.float64), want["y"].reshape(m, n).astype(np.float64)
    assert np.array_equal(np.isnan(g), np.isnan(w_)), np.argwhere(np.isnan(g) != np.isnan(w_))[:4]
    inf = np.isinf(w_) | np.isinf(g)
    assert np.array_equal(g[inf], w_[inf]), (np.argwhere(inf & (g != w_))[:4], g[inf & (g != w_)][:4], w_[inf & (g != w_)][:4])
    fin = np.isfinite(w_)
    assert (np.abs(g[fin] - w_[fin]) <= 2e-6 + 1e-5 * np.abs(w_[fin])).all()


@pytest.mark.parametrize("classes", [4, 8, 10, 16])
def test_classifier_widths(device, classes):
    """Logits that leave through a tensor map (rows of whole 16 bytes) and rows behind them that leave as one
    stretch share a staging tile; rows enough that tiles follow one another."""
    ir = W.mlp_forward(rows=4098, dims=(64, 64, 256, classes), wprec="bfloat16")
    x, onehot = W.mlp_inputs(rows=4098, in_dim=64, classes=classes)
    inputs = dict(W.mlp_params(dims=(64, 64, 256, classes)), x=x, labels=onehot)
    got, _ = run_device(device, ir, inputs)
    compare(ir, got, run_oracle(ir, inputs), rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("size,cin,cout,kernel,stride", [(33, 2, 10, 3, 1), (32, 3, 32, 3, 1), (34, 1, 20, 5, 2), (28, 1, 8, 5, 1), (32, 2, 64, 3, 1)])
def test_small_table(device, size, cin, cout, kernel, stride):
    """Single-precision convolutions whose kernel is a table in shared memory: widths that leave columns over,
    odd numbers of positions, the order of the sum (the same bits as the loops give)."""
    ir = W.conv2d_update(batch=80, size=size, cin=cin, cout=cout, kernel=kernel, stride=stride, prec="single")
    rng = np.random.default_rng(3)
    inputs = {t.ident: rng.standard_normal(t.dims).astype(np.float32) for t in ir.params() if t.ident in ("x", "target", "kernel", "bias")}
    got, info = run_device(device, ir, inputs)
    assert any("table of" in s.get("note", "") for s in info["stages"]), info
    plain, _ = run_device(device, ir, inputs, options="gemm=0")
    assert np.array_equal(got["y"], plain["y"])
    compare(ir, got, run_oracle(ir, inputs), rtol=1e-3, atol=1e-3, only=["y"])


@pytest.mark.parametrize("m,n,k", [(333, 40, 131), (64, 65, 519), (200, 72, 30)])
@pytest.mark.parametrize("a_mmajor", [False, True])
@pytest.mark.parametrize("prec", ["bfloat16", "half", "single"])
@pytest.mark.parametrize("between", [None, "reads", "overwrites"])
def test_operand_gathered_where_it_is_made(device, m, n, k, a_mmajor, prec, between):
    """A pointwise stage makes the operand: its elements are stored and gathered by one kernel, also when another stage reads
    the node in between; not when what it was made from has changed by then and a copy would still have to be made."""
    r = Routine("made_%d_%d_%d" % (m, n, k))
    shape = [k, m] if a_mmajor else [m, k]
    src = r.tn("src", prec, shape)
    scale = r.tn("scale", "single", [shape[1]], read_only=True)
    w = r.tn("w", prec, [n, k], read_only=True)
    x, y, z = r.tn("x", prec, shape), r.tn("y", "single", [m, n]), r.tn("z", "single", shape)
    p, q, s, t, u, v = r.syms(6)
    body = [loops([(p, shape[0]), (q, shape[1])], Set(x, (p, q), un("tanh", src[p, q] * scale[q])))]
    if between == "reads":
        body.append(loops([(s, shape[0]), (t, shape[1])], Set(z, (s, t), x[s, t] + 1.0)))
    elif between == "overwrites":
        body.append(loops([(u, shape[0]), (v, shape[1])], Set(src, (u, v), src[u, v] * 0.5)))
    i, j, kk = r.syms(3)
    acc = W.reduce_scope(r, "acc", "single", [(kk, k)], lambda: (x[kk, i] if a_mmajor else x[i, kk], w[j, kk]), orig=(i, j))
    body.append(loops([(i, m), (j, n)], Set(y, (i, j), acc)))
    r.body = Seq(body)
    g = np.random.default_rng(4)
    inputs = {c.ident: W.store(c.prec, (g.standard_normal(c.dims) / (np.sqrt(k) if c.ident == "w" else 1.0)).astype(np.float32))
              for c in (src, scale, w)}
    want = run_oracle(r, inputs)
    got, info = run_device(device, r, inputs)
    notes = [s["note"] or "" for s in info["stages"]]
    if 2 * m * n * k >= 4e6:
        assert any("gathers operands" in c for c in notes), notes
        lies = prec != "single" and (m if a_mmajor else k) % 8 == 0      # on a tensor map as it is
        assert any("where it is made" in c for c in notes) == (between != "overwrites" and not lies), notes
    tol = dict(rtol=1e-5, atol=4e-6) if prec == "single" else dict(rtol=2e-2, atol=4e-3)
    compare(r, got, want, only=["x", "y", "z"] if between == "reads" else ["x", "y"], **tol)
