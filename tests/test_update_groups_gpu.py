"""Updates of several parameters in one launch, and sums over a whole grid: sizes at which a chain ends in the middle
of a warp or a block, or a step of the grid has one element more or fewer.  Pointwise arithmetic in the order of the
reference's loops: single-precision nodes agree to 1e-6, 16-bit parameters to their roundings.  A sum of n values of one sign in another order is off by less than
n 2^-24 of itself; in trees of 1024 threads over 300 blocks far less, 1e-5 is allowed."""
import numpy as np
import pytest

from ocannl_b200 import backend as bk
from ocannl_b200 import workloads as W
from ocannl_b200.low_level import PREC_BYTES, Routine, Seq, Set, loops
from tests.parity import compare, run_device, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(301, 77, 33, 5), (128, 129, 1, 3), (1000, 64, 16, 2), (90, 91, 92, 10)])
@pytest.mark.parametrize("prec", ["single", "bfloat16", "half"])
@pytest.mark.parametrize("kwargs", [dict(), dict(momentum=0.9, weight_decay=1e-4, nesterov=True)])
def test_updates_in_one_launch(device, dims, prec, kwargs):
    ir = W.mlp_sgd(dims=dims, wprec=prec, **kwargs)
    g = np.random.default_rng(7)
    inputs = {}
    for t in ir.params():
        v = np.float32([0.05]) if t.ident == "learning_rate" else g.standard_normal(t.dims).astype(np.float32)
        inputs[t.ident] = W.store(t.prec, v)
    want = run_oracle(ir, inputs, statics=({}, {}))
    got, info = run_device(device, ir, inputs, statics=({}, {}))
    assert any("in the launch of" in (s["note"] or "") for s in info["stages"]), info
    for t in ir.params():
        if t.prec == "single":
            np.testing.assert_allclose(got[t.ident], want[t.ident], rtol=1e-6, atol=1e-6, err_msg=t.ident)
        else:
            # u: the spacing of the format, twice its rounding.  In each of the two steps the product with the rate, at most
            # 0.05 times the largest delta, is rounded here and not by the oracle, whose compiler contracts it with
            # the subtraction in half precision (u / 2 of the product, all that is left where the two nearly cancel),
            # and the parameter then falls on either side of a rounding boundary (u of it).
            u = 2.0 ** -7 if prec == "bfloat16" else 2.0 ** -10
            w, d = W.load(prec, want[t.ident]).astype(np.float64), W.load(prec, got[t.ident]).astype(np.float64)
            delta = max(np.abs(want[n]).max() for n in (t.ident + "_grad", t.ident + "_sgd_delta") if n in want) + 1.0
            assert np.all(np.abs(w - d) <= u * np.abs(w) * 2 + u * 0.05 * delta), t.ident


@pytest.mark.parametrize("dims", [(1773, 887, 1773, 3), (2049, 1025, 3, 2)])
def test_large_updates_take_ranges_of_the_blocks(device, dims):
    """One chain just below and just above the size from which each has blocks of its own, odd lengths, beside small ones; the
    arithmetic of test_updates_in_one_launch in single precision."""
    ir = W.mlp_sgd(dims=dims, wprec="single", momentum=0.9)
    g = np.random.default_rng(7)
    inputs = {t.ident: np.float32([0.05]) if t.ident == "learning_rate" else g.standard_normal(t.dims).astype(np.float32) for t in ir.params()}
    want = run_oracle(ir, inputs)
    got, info = run_device(device, ir, inputs)
    assert any("in the launch of" in (s["note"] or "") for s in info["stages"]), info
    for t in ir.params():
        np.testing.assert_allclose(got[t.ident], want[t.ident], rtol=1e-6, atol=1e-6, err_msg=t.ident)


@pytest.mark.parametrize("shape", [(1, 32768), (3, 10923), (7, 4683), (296, 1024), (297, 1024), (1, 303103), (5, 606209), (64, 41, 259)])
@pytest.mark.parametrize("op", ["add", "max"])
def test_sum_over_a_grid(device, shape, op):
    r = Routine("grid_%s_%s" % (op, "_".join(map(str, shape))))
    x = r.tn("x", "single", list(shape), read_only=True)
    y = r.tn("y", "single", [1])
    syms = r.syms(len(shape))
    term = lambda: x[tuple(syms)] * x[tuple(syms)]
    r.body = Seq([Set(y, (0,), W.reduce_scope(r, "total", "single", list(zip(syms, shape)), term, op=op))])
    inputs = {"x": np.random.default_rng(3).standard_normal(shape).astype(np.float32)}
    got, info = run_device(device, r, inputs)
    assert "grid-wide" in info["stages"][0]["note"], info
    exact = np.square(inputs["x"].astype(np.float64))
    want = exact.sum() if op == "add" else exact.max()
    assert abs(float(got["y"][0]) - want) <= 1e-5 * want


@pytest.mark.parametrize("off", ["b1", "b2_grad", "w2"])
@pytest.mark.parametrize("kwargs", [dict(), dict(momentum=0.9, weight_decay=1e-4, nesterov=True)])
def test_a_parameter_off_its_boundary(device, off, kwargs):
    """A parameter (or its gradient) an element off the boundary of its pairs: its own update goes element by element, the
    updates that share the launch keep their pairs, and the same bits; its own differ by a rounding of the format at most."""
    ir = W.mlp_sgd(dims=(512, 256, 256, 64), wprec="bfloat16", **kwargs)
    g = np.random.default_rng(5)
    inputs = {t.ident: W.store(t.prec, np.float32([0.05]) if t.ident == "learning_rate" else g.standard_normal(t.dims).astype(np.float32)) for t in ir.params()}
    code = bk.Code(ir)
    outs, pairs = [], []
    for shift in (0, 1):
        places, total = {}, 0
        for t in ir.params():
            total = (total + 255) // 256 * 256
            places[t.ident] = total + (shift * PREC_BYTES[t.prec] if t.ident == off else 0)
            total += t.size_in_bytes + 256
        pool = device.alloc_pool(total)
        rt = bk.Context(device, {t.ident: (pool, places[t.ident], t) for t in ir.params()}).link(code)
        for k, v in inputs.items():
            rt.context.from_host(k, v)
        rt.run()
        device.await_()
        outs.append({t.ident: rt.context.to_host(t.ident) for t in ir.params()})
        stages = rt.info()["stages"]
        assert rt.kernels_per_run() == 1 and len(stages) > 1, stages
        pairs.append({s["kernel"]: "pairs" in (s["note"] or "") for s in stages if "small" not in (s["note"] or "")})
        rt.free()
        device.free_pool(pool)
    code.free()
    own = off.split("_")[0]
    for t in ir.params():
        a, b = outs[0][t.ident], outs[1][t.ident]
        if t.ident.split("_")[0] != own:
            assert np.array_equal(a, b), t.ident
        else:
            np.testing.assert_allclose(W.load(t.prec, b), W.load(t.prec, a), rtol=2.0 ** -7, atol=1e-6, err_msg=t.ident)
    lost = [k for k in pairs[0] if not pairs[1].get(k)]
    listed = off == "w2" or not kwargs      # (small chains of several stages are listed together, without their form)
    assert all(pairs[0].values()) and len(lost) == (1 if listed else 0), pairs
