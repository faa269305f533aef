"""Contractions of few rows.  Below 128 rows only the rows that exist are staged, in whole swizzle groups of
eight (k-major) or chunks of 64 16-bit / 32 single-precision elements (m-major): one row short of, on and past
those edges, with an operand that varies with the row.  Tolerance: outputs of magnitude about one, sums in fp32 of
products of 16-bit operands, rounded once (2^-9) on either side of the oracle's rounding; single-precision operands
are read as tf32 (2^-11 each).

Few tiles over a long contraction: the k blocks are shared by a cluster of two or four CTAs, each of which finishes
some of the rows; slices of unequal length, a last k block that is not whole, tiles whose columns end early."""
import numpy as np
import pytest

from ocannl_b200 import workloads as W
from ocannl_b200.low_level import Routine, Seq, Set, loops, un
from tests.parity import compare, run_device, run_oracle

pytestmark = pytest.mark.gpu


def routine(batch, m, n, k, prec, a_mmajor, residual=True):
    r = Routine("few_rows_%d_%d_%d_%d" % (batch, m, n, k))
    x = r.tn("x", prec, [batch, k, m] if a_mmajor else [batch, m, k], read_only=True)
    w = r.tn("w", prec, [n, k], read_only=True)
    bias = r.tn("bias", "single", [n], read_only=True)
    res = r.tn("res", "single", [batch, m, n], read_only=True)
    z = r.tn("z", "single", [batch, m, n])
    y = r.tn("y", prec, [batch, m, n])
    ib, i, j, kk = r.syms(4)
    acc = W.reduce_scope(r, "acc", "single", [(kk, k)], lambda: (w[j, kk], x[ib, kk, i] if a_mmajor else x[ib, i, kk]), orig=(ib, i, j))
    v = acc + bias[j]
    if residual:
        v = v + res[ib, i, j]
    jb, p, q = r.syms(3)
    r.body = Seq([loops([(ib, batch), (i, m), (j, n)], Set(z, (ib, i, j), v)),
                  loops([(jb, batch), (p, m), (q, n)], Set(y, (jb, p, q), un("relu", z[jb, p, q])))])
    return r


def inputs_of(ir, k, seed=3):
    g = np.random.default_rng(seed)
    return {t.ident: W.store(t.prec, (g.standard_normal(t.dims) / (np.sqrt(k) if t.ident == "w" else 1.0)).astype(np.float32))
            for t in ir.params() if t.read_only}


def check(device, ir, k):
    inputs = inputs_of(ir, k)
    want = run_oracle(ir, inputs)
    got, info = run_device(device, ir, inputs)
    assert "tcgen05" in info["stages"][-1]["note"], info
    compare(ir, got, want, rtol=2e-2, atol=2e-2, only=["z", "y"])
    return info["stages"][-1]["note"]


@pytest.mark.parametrize("m", [8, 9, 16, 37, 64, 65, 120, 121, 127, 128, 129])
@pytest.mark.parametrize("batch,n,k", [(1, 264, 512), (2, 40, 520)])
def test_rows_staged(device, m, batch, n, k):
    if batch > 1 and m < 16:
        pytest.skip("rows of a batch: the loops")
    check(device, routine(batch, m, n, k, "bfloat16", False), k)


@pytest.mark.parametrize("m", [64, 72, 120, 128, 136])
@pytest.mark.parametrize("prec", ["bfloat16", "single"])
def test_columns_staged(device, m, prec):
    check(device, routine(1, m, 264, 512, prec, True), 512)


@pytest.mark.parametrize("m,n,k", [(40, 1024, 1024), (37, 264, 4096), (100, 48, 2048), (128, 136, 1032), (129, 520, 1096),
                                   (500, 256, 1024), (500, 304, 1040), (1000, 264, 2048), (300, 72, 1160), (64, 16, 8200)])
@pytest.mark.parametrize("prec", ["bfloat16", "half", "single"])
@pytest.mark.parametrize("residual", [False, True])
def test_k_blocks_over_a_cluster(device, m, n, k, prec, residual):
    note = check(device, routine(1, m, n, k, prec, False, residual), k)
    assert "over a cluster" in note, note


@pytest.mark.parametrize("rows,n", [(33, 10), (37, 10), (200, 27), (1000, 32), (4096, 2)])
def test_row_assignments_over_a_cluster(device, rows, n):
    """The softmax and the mean loss that follow a narrow layer, each row whole in one of the cluster's CTAs."""
    ir = W.mlp_forward(rows=rows, dims=(256, 1024, 1024, n), wprec="bfloat16")
    x, labels = W.mlp_inputs(rows=rows, in_dim=256, classes=n)
    inputs = dict(W.mlp_params(dims=(256, 1024, 1024, n)), x=x, labels=labels)
    want = run_oracle(ir, inputs)
    got, info = run_device(device, ir, inputs)
    assert "over a cluster" in info["stages"][-1]["note"] and "grid-wide sum" in info["stages"][-1]["note"], info
    compare(ir, got, want, rtol=2e-2, atol=2e-2)
