"""Contractions that do not depend on one another in one launch, each on blocks of its own: equal and different shapes,
epilogues and outputs, slices over clusters, a residual by TMA beside plain stores; and neighbours that do depend on one
another, which keep launches of their own.  Tolerance as for single 16-bit contractions: 2e-2 of outputs of magnitude one."""
import numpy as np
import pytest

from ocannl_b200 import workloads as W
from ocannl_b200.low_level import Routine, Seq, Set, loops, un
from tests.parity import compare, run_device, run_oracle

pytestmark = pytest.mark.gpu


def _contract(r, x, name, m, n, k, prec, out_prec, act, residual=None):
    w = r.tn("w_" + name, prec, [n, k], read_only=True)
    y = r.tn("y_" + name, out_prec, [m, n])
    i, j, kk = r.syms(3)
    v = W.reduce_scope(r, "acc_" + name, "single", [(kk, k)], lambda: (w[j, kk], x[i, kk]), orig=(i, j))
    if residual is not None:
        v = v + residual[i, j]
    return y, loops([(i, m), (j, n)], Set(y, (i, j), un(act, v) if act else v))


def _run(device, r, k, expect):
    g = np.random.default_rng(11)
    inputs = {t.ident: W.store(t.prec, (g.standard_normal(t.dims) / (np.sqrt(k) if t.ident.startswith("w_") else 1.0)).astype(np.float32))
              for t in r.params() if t.read_only}
    want = run_oracle(r, inputs)
    for graph in (False, True):
        got, info = run_device(device, r, inputs, statics=({}, {}, {}), graph=graph)
        assert sum("in the launch of" in (s["note"] or "") for s in info["stages"]) == expect, info
        compare(r, got, want, rtol=2e-2, atol=2e-2, only=[t.ident for t in r.params() if t.ident.startswith("y_")])


@pytest.mark.parametrize("m,n,k", [(100, 128, 256), (37, 264, 1024), (500, 256, 256), (9, 72, 4096)])
@pytest.mark.parametrize("prec", ["bfloat16", "half", "single"])
def test_three_of_a_kind(device, m, n, k, prec):
    if prec == "single" and m < 32:
        pytest.skip("loops")
    r = Routine("grouped_%d_%d_%d" % (m, n, k))
    x = r.tn("x", prec, [m, k], read_only=True)
    r.body = Seq([_contract(r, x, c, m, n, k, prec, prec, None)[1] for c in "qkv"])
    _run(device, r, k, 2)


@pytest.mark.parametrize("prec", ["bfloat16", "half"])
def test_different_shapes(device, prec):
    r = Routine("grouped_mixed")
    x = r.tn("x", prec, [200, 256], read_only=True)
    z = r.tn("z", prec, [77, 256], read_only=True)
    res = r.tn("res", "single", [200, 96], read_only=True)
    a = _contract(r, x, "a", 200, 96, 256, prec, "single", "relu", res)[1]
    b = _contract(r, z, "b", 77, 48, 256, prec, prec, None)[1]
    c = _contract(r, x, "c", 200, 27, 256, prec, "single", "tanh")[1]
    r.body = Seq([a, b, c])
    _run(device, r, 256, 2)


def test_dependent_neighbours(device):
    r = Routine("not_grouped")
    x = r.tn("x", "bfloat16", [100, 256], read_only=True)
    y, a = _contract(r, x, "a", 100, 256, 256, "bfloat16", "bfloat16", "tanh")
    b = _contract(r, y, "b", 100, 128, 256, "bfloat16", "bfloat16", None)[1]
    c = _contract(r, x, "c", 100, 128, 256, "bfloat16", "bfloat16", None)[1]
    r.body = Seq([a, b, c])
    _run(device, r, 256, 1)
