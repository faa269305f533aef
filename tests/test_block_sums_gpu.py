"""Sums that a whole block takes: a single output on either side of 256 and of a whole number of steps of 1024 terms, by
itself, behind the stages whose values it sums, and beside stages that have nothing to do with it; maxima too.  And
accumulations at moving positions that are few, spread over threads instead of a long walk by each.  Sums in another
order: n 2^-24 of a sum of n values of one sign at most, in trees far less; 1e-5."""
import numpy as np
import pytest

from ocannl_b200 import workloads as W
from ocannl_b200.low_level import Routine, Seq, Set, loops, un
from tests.parity import compare, run_device, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5, 51), (16, 16), (1, 257), (31, 33), (32, 32), (25, 41), (128, 64), (3, 1365), (90, 91), (8193, 2), (32767, 1)])
@pytest.mark.parametrize("op", ["add", "max"])
def test_single_outputs(device, shape, op):
    r = Routine("sums_%d_%d_%s" % (shape[0], shape[1], op))
    x = r.tn("x", "single", list(shape), read_only=True)
    e, z = r.tn("e", "single", list(shape)), r.tn("z", "single", list(shape))
    y, mean = r.tn("y", "single", [1]), r.tn("mean", "single", [1])
    i, j, k, l, p, q = r.syms(6)
    m, n = shape
    body = [loops([(i, m), (j, n)], Set(e, (i, j), un("exp", x[i, j]))),
            Set(y, (0,), W.reduce_scope(r, "total", "single", [(k, m), (l, n)], lambda: e[k, l] * e[k, l], op=op)),
            Set(mean, (0,), y[0] / float(m * n)),
            loops([(p, m), (q, n)], Set(z, (p, q), x[p, q] * 3.0))]
    r.body = Seq(body)
    inputs = {"x": np.random.default_rng(1).uniform(-1, 1, shape).astype(np.float32)}
    want = run_oracle(r, inputs)
    for options in (None, "fuse=0"):
        got, info = run_device(device, r, inputs, options=options)
        exact = np.exp(inputs["x"].astype(np.float64)) ** 2
        exact = exact.sum() if op == "add" else exact.max()
        assert abs(float(got["y"][0]) - exact) <= 1e-5 * exact, info
        assert abs(float(got["mean"][0]) - exact / (m * n)) <= 1e-5 * exact / (m * n)
        compare(r, got, want, rtol=1e-6, atol=1e-7, only=["e", "z"])


@pytest.mark.parametrize("batch,size,cin,cout,kernel,stride", [(19, 9, 1, 38, 3, 2), (1, 8, 1, 50, 5, 1), (3, 16, 3, 56, 3, 2), (2, 8, 4, 29, 3, 2), (1, 5, 2, 8, 5, 1)])
def test_few_moving_positions(device, batch, size, cin, cout, kernel, stride):
    ir = W.conv2d_update(batch=batch, size=size, cin=cin, cout=cout, kernel=kernel, stride=stride, prec="single")
    g = np.random.default_rng(2)
    inputs = {t.ident: (g.standard_normal(t.dims) * (0.2 if t.ident == "kernel" else 1.0)).astype(np.float32) for t in ir.params() if t.read_only}
    want = run_oracle(ir, inputs)
    got, info = run_device(device, ir, inputs)
    for t in ir.params():
        w, d = want[t.ident].astype(np.float64), got[t.ident].astype(np.float64)
        assert np.linalg.norm(w - d) <= 2e-5 * np.linalg.norm(w) + 1e-12, (t.ident, info)
