"""Gradients over a batch, dW[o, i] += dz[b, o] * h[b, i], whose short outer loop stays in registers: the lengths of it that
are combined in one, in several or in a ragged last phase, with columns on either side of a warp and of four of them.  And
the clears before them, several nodes of odd sizes and of each element size in one launch.  Sums of n products in
another order: n 2^-24 of the sum of their magnitudes at most (2^-53 in double precision; sums in 32 bits with an
atomic addition per slice), n = 500; in trees far less, 1e-5 (1e-13) of it."""
import numpy as np
import pytest

from ocannl_b200 import workloads as W
from ocannl_b200.low_level import Routine, Seq, Set, ZeroOut, fma, loops
from tests.parity import run_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("out", [2, 3, 7, 10, 16])
@pytest.mark.parametrize("cols", [2, 31, 130, 514])
@pytest.mark.parametrize("rows", [500])
@pytest.mark.parametrize("prec,grad", [("single", "single"), ("bfloat16", "single"), ("double", "double")])
def test_tiled_outputs(device, out, cols, rows, prec, grad):
    r = Routine("split_%d_%d_%d_%s" % (out, cols, rows, prec))
    dz, h = r.tn("dz", prec, [rows, out], read_only=True), r.tn("h", prec, [rows, cols], read_only=True)
    dw, flag = r.tn("dw", grad, [out, cols]), r.tn("flag", "byte", [7])
    db, e = r.tn("db", grad, [out]), r.tn("e", "half", [3, 5])
    b, o, i, b2, o2 = r.syms(5)
    r.body = Seq([ZeroOut(t) for t in (dw, flag, db, e)] +
                 [loops([(b, rows), (o, out), (i, cols)], Set(dw, (o, i), fma(dz[b, o], h[b, i], dw[o, i]))),
                  loops([(b2, rows), (o2, out)], Set(db, (o2,), db[o2] + dz[b2, o2]))])
    g = np.random.default_rng(5)
    inputs = {"dz": W.store(prec, g.standard_normal((rows, out))), "h": W.store(prec, g.standard_normal((rows, cols)))}
    for t in (dw, flag, db, e):
        inputs[t.ident] = np.full(t.dims, 3, np.uint8) if t.prec == "byte" else W.store(t.prec, np.full(t.dims, 3.0))
    got, info = run_device(device, r, inputs, options="gemm=0")
    assert any("kept in registers" in (s["note"] or "") for s in info["stages"]), info
    z, x = (W.load(prec, inputs[n]).astype(np.float64) for n in ("dz", "h"))
    tol = 1e-13 if grad == "double" else 1e-5
    assert np.all(np.abs(got["dw"] - z.T @ x) <= tol * (np.abs(z).T @ np.abs(x)))
    assert np.all(np.abs(got["db"] - z.sum(0)) <= tol * np.abs(z).sum(0))
    assert not np.any(got["flag"]) and not np.any(W.load("half", got["e"]))
