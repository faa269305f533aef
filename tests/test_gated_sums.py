"""Which contractions share their k blocks over a cluster (another order of the sums): none whose result a gate or a comparison
reads, directly, through what is made of it or through a local; the others of the same routine as before.  Plans only, no GPU."""
import pytest

from ocannl_b200 import backend as bk
from ocannl_b200 import workloads as W
from ocannl_b200.low_level import DeclareLocal, GetLocal, Routine, Seq, Set, SetLocal, binop, loops, un, where


def _clusters(ir):
    code = bk.Code(ir)
    try:
        return ["over a cluster" in (s["note"] or "") for s in code.info()["stages"] if s["kind"] == "gemm"]
    finally:
        code.free()


@pytest.mark.parametrize("prec", ["single", "bfloat16"])
def test_training_steps_keep_the_order_of_gated_sums(prec):
    forward = _clusters(W.mlp_forward(rows=200, dims=(784, 1024, 1024, 10), wprec=prec))
    assert forward[1:] == [True, True]
    step = _clusters(W.mlp_train_update(rows=200, dims=(784, 1024, 1024, 10), wprec=prec))
    assert step[:2] == [False, False] and step[2]      # hidden layers: gated; logits: nothing compares them


@pytest.mark.parametrize("use,clustered", [("none", True), ("relu", True), ("gate", False), ("lt", False), ("where", False), ("behind", False), ("value of where", True)])
def test_what_counts_as_a_decision(use, clustered):
    m, n, k = 64, 64, 1024
    r = Routine("decide_" + use.replace(" ", "_"))
    a, b = r.tn("a", "bfloat16", [m, k], read_only=True), r.tn("b", "bfloat16", [n, k], read_only=True)
    c, d, e = r.tn("c", "single", [m, n]), r.tn("d", "single", [m, n]), r.tn("e", "single", [m, n])
    i, j, p, q, s, u, v = r.syms(7)
    body = [loops([(i, m), (j, n)], Set(c, (i, j), W.reduce_scope(r, "acc", "single", [(p, k)], lambda: (a[i, p], b[j, p]))))]
    value = {"none": lambda: c[q, s] * 2.0, "relu": lambda: un("relu", c[q, s]), "gate": lambda: binop("relu_gate", c[q, s], d[q, s]),
             "lt": lambda: binop("lt", c[q, s], d[q, s]), "where": lambda: where(c[q, s], d[q, s], e[q, s]),
             "behind": lambda: un("exp", c[q, s]), "value of where": lambda: where(d[q, s], c[q, s], 0.0)}[use]
    body.append(loops([(q, m), (s, n)], Set(e, (q, s), value())))
    if use == "behind":
        body.append(loops([(u, m), (v, n)], Set(d, (u, v), binop("relu_gate", e[u, v], d[u, v]))))
    r.body = Seq(body)
    assert _clusters(r) == [clustered]


@pytest.mark.parametrize("use,clustered", [("relu", True), ("gate", False), ("gate of product", False), ("lt", False), ("where", False), ("trunc", False), ("not", False),
                                           ("value of gate", True), ("value of where", True)])
@pytest.mark.parametrize("prec", ["single", "bfloat16"])
def test_decisions_on_the_sum_itself(use, clustered, prec):
    """The sum is gated, compared or truncated by the assignment that holds it."""
    m, n, k = 64, 64, 1024
    r = Routine("decide_at_once_" + use.replace(" ", "_"))
    a, b = r.tn("a", "bfloat16", [m, k], read_only=True), r.tn("b", "bfloat16", [n, k], read_only=True)
    c, d, e = r.tn("c", prec, [m, n]), r.tn("d", "single", [m, n], read_only=True), r.tn("e", "single", [m, n], read_only=True)
    i, j, p = r.syms(3)
    s = W.reduce_scope(r, "acc", "single", [(p, k)], lambda: (a[i, p], b[j, p]))
    value = {"relu": lambda: un("relu", s), "gate": lambda: binop("relu_gate", s, d[i, j]), "gate of product": lambda: binop("relu_gate", s * e[i, j], d[i, j]),
             "lt": lambda: binop("lt", s, d[i, j]), "where": lambda: where(binop("lt", s, d[i, j]), d[i, j], e[i, j]), "trunc": lambda: un("trunc", s), "not": lambda: un("not", s),
             "value of gate": lambda: binop("relu_gate", d[i, j], s), "value of where": lambda: where(d[i, j], s, 0.0)}[use]
    r.body = Seq([loops([(i, m), (j, n)], Set(c, (i, j), value()))])
    assert _clusters(r) == [clustered]


@pytest.mark.parametrize("use,clustered", [("plain", True), ("gate", False), ("behind", False), ("two locals", False)])
def test_decisions_on_a_local(use, clustered):
    """The sum's node is read into a local of the loop body, and the local decides."""
    m, n, k = 64, 64, 1024
    r = Routine("decide_local_" + use.replace(" ", "_"))
    a, b = r.tn("a", "bfloat16", [m, k], read_only=True), r.tn("b", "bfloat16", [n, k], read_only=True)
    c, d, e, f = r.tn("c", "single", [m, n]), r.tn("d", "single", [m, n], read_only=True), r.tn("e", "single", [m, n]), r.tn("f", "single", [m, n])
    v, w = r.scope(r.tn("v", "single", [1], mode="virtual")), r.scope(r.tn("w", "single", [1], mode="virtual"))
    i, j, p, q, s, x, y = r.syms(7)
    body = [loops([(i, m), (j, n)], Set(c, (i, j), W.reduce_scope(r, "acc", "single", [(p, k)], lambda: (a[i, p], b[j, p]))))]
    inner = [DeclareLocal(v, False), SetLocal(v, c[q, s] * 2.0)]
    if use == "two locals":
        inner += [DeclareLocal(w, False), SetLocal(w, GetLocal(v) + 1.0)]
    got = GetLocal(w if use == "two locals" else v)
    inner.append(Set(e, (q, s), got * d[q, s] if use in ("plain", "behind") else binop("relu_gate", got, d[q, s])))
    body.append(loops([(q, m), (s, n)], Seq(inner)))
    if use == "behind":
        body.append(loops([(x, m), (y, n)], Set(f, (x, y), binop("relu_gate", e[x, y], d[x, y]))))
    r.body = Seq(body)
    assert _clusters(r) == [clustered]
