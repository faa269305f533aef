"""Which pointwise stages may make a contraction's operand where it is gathered, and that every form of such a stage
compiles: the gathering kernel gives the maker its loops and nothing else.  Plans and compilation, which need no GPU, and
one run of each form."""
import numpy as np
import pytest

from ocannl_b200 import backend as bk
from ocannl_b200 import workloads as W
from ocannl_b200.low_level import Affine, EmbedIndex, Routine, Seq, Set, loops, un
from tests.parity import compare, run_device, run_oracle


def _stages(ir, options=None):
    code = bk.Code(ir, options)      # (compiles every kernel of the routine)
    try:
        return code.info()["stages"]
    finally:
        code.free()


def _made(stages):
    return any("where it is made" in (s["note"] or "") for s in stages)


def _contraction(r, x, body, m, n, k):
    """`body`, which makes x, and y := x w^T behind it."""
    w, y = r.tn("w", x.prec, [n, k], read_only=True), r.tn("y", "single", [m, n])
    i, j, kk = r.syms(3)
    acc = W.reduce_scope(r, "acc", "single", [(kk, k)], lambda: (x[i, kk], w[j, kk]), orig=(i, j))
    r.body = Seq([body, loops([(i, m), (j, n)], Set(y, (i, j), acc))])
    return r


M, N, K = 333, 40, 333      # (rows of 666 or 1332 bytes: not on a tensor map)


@pytest.mark.parametrize("prec", ["bfloat16", "half", "single"])
@pytest.mark.parametrize("outer", [True, False])
@pytest.mark.parametrize("read", ["value", "twice", "not"])
def test_loops_of_one_iteration(built_lib, prec, outer, read):
    """A loop of one iteration that the written node does not carry: a batch or a channel of one."""
    r = Routine("unit_loop_%s" % read)
    src, one = r.tn("src", prec, [1, M, K], read_only=True), r.tn("one", "single", [1, K], read_only=True)
    x = r.tn("x", prec, [M, K])
    p, q, e = r.syms(3)
    value = {"value": lambda: un("tanh", src[e, p, q]), "twice": lambda: src[e, p, q] * one[e, q], "not": lambda: un("tanh", src[0, p, q])}[read]
    nest = [(e, 1), (p, M), (q, K)] if outer else [(p, M), (e, 1), (q, K)]
    stages = _stages(_contraction(r, x, loops(nest, Set(x, (p, q), value())), M, N, K))
    assert stages[-1]["kind"] == "gemm" and _made(stages), stages


STATIC = {"embedded": lambda x, s, p, q: x[p, q] * EmbedIndex(s), "embedded sum": lambda x, s, p, q: x[p, q] * EmbedIndex(Affine(((1, p), (2, s)))),
          "loop embedded": lambda x, s, p, q: x[p, q] * EmbedIndex(Affine(((1, p), (2, q))))}


def _static(form, prec):
    r = Routine("static_" + form.replace(" ", "_"))
    s = r.static_sym(16)
    src, x = r.tn("src", prec, [M, K], read_only=True), r.tn("x", prec, [M, K])
    p, q = r.syms(2)
    return _contraction(r, x, loops([(p, M), (q, K)], Set(x, (p, q), STATIC[form](src, s, p, q))), M, N, K), s


@pytest.mark.parametrize("prec", ["bfloat16", "half", "single"])
@pytest.mark.parametrize("form", list(STATIC))
def test_static_index_in_the_value(built_lib, prec, form):
    """A value that holds a static index keeps its own kernel, which is given the index; loop indices may be folded."""
    stages = _stages(_static(form, prec)[0])
    assert stages[-1]["kind"] == "gemm" and _made(stages) == (form == "loop embedded"), stages


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["bfloat16", "single"])
def test_loops_of_one_iteration_on_the_device(device, prec):
    """Tolerances of the contractions of gathered operands: 2e-2 for 16-bit operands, 1e-5 where they travel in two parts."""
    r = Routine("unit_loop")
    src, one = r.tn("src", prec, [1, M, K], read_only=True), r.tn("one", "single", [1, K], read_only=True)
    x = r.tn("x", prec, [M, K])
    p, q, e = r.syms(3)
    _check(device, _contraction(r, x, loops([(p, M), (e, 1), (q, K)], Set(x, (p, q), src[e, p, q] * one[e, q])), M, N, K), prec)


@pytest.mark.gpu
@pytest.mark.parametrize("form", list(STATIC))
def test_static_index_on_the_device(device, form):
    ir, s = _static(form, "single")
    _check(device, ir, "single", statics=({s: 3}, {s: 11}))


def _check(device, ir, prec, statics=({},)):
    g = np.random.default_rng(6)
    inputs = {t.ident: W.store(t.prec, (g.standard_normal(t.dims) / (np.sqrt(K) if t.ident == "w" else 1.0)).astype(np.float32))
              for t in ir.params() if t.read_only}
    want = run_oracle(ir, inputs, statics=statics)
    got, _ = run_device(device, ir, inputs, statics=statics)
    scale = max(1.0, float(np.abs(W.load(prec, want["x"])).max()) / 4.0)     # (the absolute part is that of operands of unit variance)
    tol = dict(rtol=1e-5, atol=4e-6 * scale) if prec == "single" else dict(rtol=2e-2, atol=4e-3 * scale)
    compare(ir, got, want, only=["x", "y"], **tol)


def test_loop_without_iterations(built_lib):
    r = Routine("empty_loop")
    src, x = r.tn("src", "bfloat16", [M, K], read_only=True), r.tn("x", "bfloat16", [M, K])
    p, q, e = r.syms(3)
    stages = _stages(_contraction(r, x, loops([(p, M), (e, 0), (q, K)], Set(x, (p, q), un("tanh", src[p, q]))), M, N, K))
    assert not _made(stages), stages


def test_a_launch_for_every_statement(built_lib):
    """Without fusion the maker keeps a launch of its own."""
    r = Routine("unfused")
    src, x = r.tn("src", "bfloat16", [M, K], read_only=True), r.tn("x", "bfloat16", [M, K])
    p, q = r.syms(2)
    ir = _contraction(r, x, loops([(p, M), (q, K)], Set(x, (p, q), un("tanh", src[p, q]))), M, N, K)
    assert _made(_stages(ir)) and not _made(_stages(ir, "fuse=0"))
    assert len(_stages(ir, "fuse=0")) == len(_stages(ir)) + 1
