"""Accumulations whose written position moves with several loops, few positions and a long walk: a thread per position adds its
terms in the order of the loops, so that the sums have the bits that one thread gives which walks all loops by itself."""
import numpy as np
import pytest

from ocannl_b200 import backend as bk
from ocannl_b200 import workloads as W
from ocannl_b200.low_level import Affine, Routine, Seq, Set, fma, loops
from tests.parity import compare, run_device, run_oracle

# o, k, f: extents of the position's two symbols and of the loop beside them; c, d: the symbols' factors; first: what is added
FORMS = {"steps of one": dict(o=9, k=5, f=40, c=1, d=1), "steps of two": dict(o=9, k=3, f=41, c=2, d=1), "gaps": dict(o=7, k=2, f=33, c=3, d=1),
         "offset": dict(o=8, k=4, f=30, c=2, d=1, first=3), "spread kernel": dict(o=6, k=4, f=40, c=1, d=2), "both spread": dict(o=6, k=5, f=40, c=2, d=3),
         "backwards": dict(o=9, k=4, f=31, c=1, d=-1, first=3), "kernel outside": dict(o=9, k=3, f=40, c=2, d=1, order="kof"), "other loop outside": dict(o=9, k=3, f=40, c=2, d=1, order="fok"),
         "one position": dict(o=1, k=1, f=300, c=1, d=1), "double": dict(o=9, k=3, f=40, c=2, d=1, prec="double"), "no channels": dict(o=9, k=3, f=40, c=2, d=1, ch=1)}


def _routine(name, o, k, f, c, d, first=0, order="okf", prec="single", ch=3, batch=2):
    r = Routine("positions_" + name.replace(" ", "_"))
    length = first + c * (o - 1) + max(0, d * (k - 1)) + 1 + 2          # two positions that nothing reaches
    t = r.tn("t", prec, [batch, length, ch])
    w, g = r.tn("w", prec, [k, f, ch], read_only=True), r.tn("g", prec, [batch, o, f], read_only=True)
    b, io, ik, jf, ic = r.syms(5)
    at = Affine(((c, io), (d, ik)), first)
    nest = {"o": (io, o), "k": (ik, k), "f": (jf, f)}
    r.body = Seq([loops([(b, batch)] + [nest[s] for s in order] + [(ic, ch)],
                        Set(t, (b, at, ic), fma(w[ik, jf, ic], g[b, io, jf], t[b, at, ic])))])
    return r


def _notes(ir, options=None):
    code = bk.Code(ir, options)
    try:
        return [s["note"] or "" for s in code.info()["stages"]]
    finally:
        code.free()


@pytest.mark.parametrize("form", list(FORMS))
def test_which_accumulations(built_lib, form):
    ir = _routine(form, **FORMS[form])
    assert ["by position" in n for n in _notes(ir)] == [True], _notes(ir)
    assert not any("by position" in n for n in _notes(ir, "bounds=1") + _notes(ir, "coop=0"))


@pytest.mark.parametrize("cfg", [dict(batch=1, size=8, cin=1, cout=50, kernel=5), dict(batch=3, size=16, cin=3, cout=56, kernel=3, stride=2), dict(batch=19, size=9, cin=1, cout=38, kernel=3, stride=2)])
def test_small_convolutions_add_in_a_fixed_order(built_lib, cfg):
    notes = _notes(W.conv2d_update(prec="single", **cfg))
    assert any("by position" in n for n in notes) and not any("scatter" in n for n in notes), notes


@pytest.mark.gpu
@pytest.mark.parametrize("form", list(FORMS))
def test_bits_of_the_loops(device, form):
    ir = _routine(form, **FORMS[form])
    g = np.random.default_rng(8)
    inputs = {t.ident: g.standard_normal(t.dims).astype(np.float64 if t.prec == "double" else np.float32) for t in ir.params()}
    got, _ = run_device(device, ir, inputs, statics=({}, {}))
    loops_, _ = run_device(device, ir, inputs, statics=({}, {}), options="coop=0")
    assert np.array_equal(got["t"], loops_["t"])
    # (the order is the oracle's too; 600 terms of magnitude one, each rounded once or twice)
    compare(ir, got, run_oracle(ir, inputs, statics=({}, {})), rtol=1e-5, atol=1e-4, only=["t"])


@pytest.mark.gpu
@pytest.mark.parametrize("cfg", [dict(batch=1, size=8, cin=1, cout=50, kernel=5), dict(batch=3, size=16, cin=3, cout=56, kernel=3, stride=2), dict(batch=19, size=9, cin=1, cout=38, kernel=3, stride=2)])
def test_input_gradients(device, cfg):
    ir, inputs = W.conv2d_update(prec="single", **cfg), W.conv2d_inputs(prec="single", **cfg)
    want = run_oracle(ir, inputs)
    got, _ = run_device(device, ir, inputs)
    scale = float(np.abs(want["x_padded_grad"]).max())
    np.testing.assert_allclose(got["x_padded_grad"], want["x_padded_grad"], rtol=1e-4, atol=1e-5 * scale)
