"""Updates of several parameters in one launch, and sums over a whole grid: sizes at which a chain ends in the middle
of a warp or a block, or a step of the grid has one element more or fewer.  Pointwise arithmetic in the order of the
reference's loops: single-precision nodes agree to 1e-6, 16-bit parameters to their roundings.  A sum of n values of one sign in another order is off by less than
n 2^-24 of itself; in trees of 1024 threads over 300 blocks far less, 1e-5 is allowed."""
import numpy as np
import pytest

from ocannl_b200 import workloads as W
from ocannl_b200.low_level import Routine, Seq, Set, loops
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
