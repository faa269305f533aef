"""The limit of a contraction's waits counts its own work, not that of the kernels ahead of it, beside which it is already
set up: a role whose waits have a limit first waits for those kernels, and the one that does not ends with the others."""
import re

import numpy as np
import pytest

from ocannl_b200 import backend as bk
from ocannl_b200 import workloads as W
from ocannl_b200.low_level import Routine, Seq, Set, loops
from tests.parity import run_device, run_oracle

M, N, K = 256, 64, 128


def _behind(steps):
    """A recurrence of `steps` terms, which one thread follows, and a contraction behind it."""
    r = Routine("behind_%d" % steps)
    a, b, t = r.tn("a", "bfloat16", [M, K], read_only=True), r.tn("b", "bfloat16", [N, K], read_only=True), r.tn("terms", "single", [steps], read_only=True)
    s, c = r.tn("s", "single", [1]), r.tn("c", "single", [M, N])
    h, i, j, p = r.syms(4)
    r.body = Seq([loops([(h, steps)], Set(s, (0,), s[0] * 0.5 + t[h])),
                  loops([(i, M), (j, N)], Set(c, (i, j), W.reduce_scope(r, "acc", "single", [(p, K)], lambda: (a[i, p], b[j, p]))))])
    return r


@pytest.mark.parametrize("ir", [_behind(64), W.mlp_forward(rows=37), W.mlp_forward(rows=8192), W.mlp_train_update(rows=8192), W.einsum_gelu(1, 300, 300, 304, "single", "single")],
                         ids=["plain", "clusters", "pairs", "split k", "two parts"])
def test_limits_begin_behind_the_kernels_ahead(built_lib, ir):
    code = bk.Code(ir)
    try:
        sources = [code.source(i) for i, s in enumerate(code.info()["stages"]) if s["kind"] == "gemm"]
    finally:
        code.free()
    assert sources
    for text in sources:
        roles = re.split(r"// -+ (TMA producer|MMA issuer[^\n]*|epilogue|teardown)\n", text[text.index("B200_KERNEL_HEAD(B200_TMAP_PARAM"):])
        assert [x.split()[0] for x in roles[1::2]] == ["TMA", "MMA", "epilogue", "teardown"], roles[1::2]
        producer, issuer, epilogue = roles[2:-1:2]
        for role in (producer, epilogue):
            assert "griddepcontrol.wait" in role[:role.index("b200_wait(")], role[:400]
        # the issuer: accumulators, which are free at first, and operands, whose wait the epilogue's limit ends
        assert re.findall(r"b200_wait(\w*)\((\w+)", issuer) == [("", "bar_acc_empty"), ("_aborted", "bar_full")], issuer


@pytest.mark.gpu
def test_kernels_ahead_may_take_longer_than_the_limit(device, monkeypatch):
    monkeypatch.setenv("B200_NVRTC_FLAGS", "-DB200_WAIT_LIMIT_NS=2000000ull")
    steps = 1 << 23        # a chain of at least eight cycles each: 30 ms and more
    ir = _behind(steps)
    g = np.random.default_rng(3)
    inputs = {t.ident: W.store(t.prec, g.standard_normal(t.dims).astype(np.float32)) for t in ir.params() if t.read_only}
    got, info = run_device(device, ir, inputs)      # (a wait that ran out would be raised here)
    assert [s["kind"] for s in info["stages"]] == ["generic", "gemm"], info
    want = run_oracle(ir, inputs)
    np.testing.assert_allclose(got["s"], want["s"], rtol=1e-5)
    # 128 products of bfloat16 values, exact in single precision, added in another order
    np.testing.assert_allclose(got["c"], want["c"], rtol=1e-5, atol=1e-4)
