"""Layer norm and softmax over row widths on both sides of the register forms' boundaries: below a warp, one
element short of and past whole warps, the dealt widths, the widest; few rows and many."""
import numpy as np
import pytest

from ocannl_b200 import workloads as W
from ocannl_b200.low_level import Routine, Seq, Set, loops, un
from tests.parity import compare, run_device, run_oracle

pytestmark = pytest.mark.gpu


def _layer_norm_and_softmax(rows, width, prec):
    r = Routine("rows_%d_%d" % (rows, width))
    x = r.tn("x", prec, [rows, width], read_only=True)
    gamma = r.tn("gamma", "single", [width], read_only=True)
    s, c, d, y = r.tn("s", "single", [rows, 1]), r.tn("c", "single", [rows, width]), r.tn("d", "single", [rows, 1]), r.tn("y", prec, [rows, width])
    m, e, z, p = r.tn("m", "single", [rows, 1]), r.tn("e", "single", [rows, width]), r.tn("z", "single", [rows, 1]), r.tn("p", prec, [rows, width])
    red = lambda name, node, row, op, f=lambda v: v: (lambda k: W.reduce_scope(r, name, "single", [(k, width)], lambda: f(node[row, k]), op=op))(r.sym())
    body = []
    i = r.sym(); body.append(loops([(i, rows)], Set(s, (i, 0), red("n_s", x, i, "add"))))
    i, j = r.syms(2); body.append(loops([(i, rows), (j, width)], Set(c, (i, j), x[i, j] - s[i, 0] / float(width))))
    i = r.sym(); body.append(loops([(i, rows)], Set(d, (i, 0), un("sqrt", red("n_d", c, i, "add", lambda v: v * v) + 1e-5))))
    i, j = r.syms(2); body.append(loops([(i, rows), (j, width)], Set(y, (i, j), gamma[j] * (c[i, j] / d[i, 0]))))
    i = r.sym(); body.append(loops([(i, rows)], Set(m, (i, 0), red("n_m", y, i, "max"))))
    i, j = r.syms(2); body.append(loops([(i, rows), (j, width)], Set(e, (i, j), un("exp", y[i, j] - m[i, 0]))))
    i = r.sym(); body.append(loops([(i, rows)], Set(z, (i, 0), red("n_z", e, i, "add"))))
    i, j = r.syms(2); body.append(loops([(i, rows), (j, width)], Set(p, (i, j), e[i, j] / z[i, 0])))
    r.body = Seq(body)
    return r


@pytest.mark.parametrize("width", [31, 32, 33, 63, 64, 95, 96, 128, 129, 200, 384, 512, 640, 1023, 1025])
@pytest.mark.parametrize("rows,prec", [(130, "bfloat16"), (1000, "single")])
def test_row_widths(device, width, rows, prec):
    ir = _layer_norm_and_softmax(rows, width, prec)
    g = np.random.default_rng(width)
    inputs = {"x": W.store(prec, g.standard_normal((rows, width)).astype(np.float32)), "gamma": g.standard_normal(width).astype(np.float32)}
    want = run_oracle(ir, inputs)
    got, _ = run_device(device, ir, inputs)
    tol = dict(rtol=2e-2, atol=2e-2) if prec != "single" else dict(rtol=1e-4, atol=2e-4)      # (row sums of terms of either sign)
    compare(ir, got, want, **tol)
