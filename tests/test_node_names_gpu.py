"""Nodes called like a name of a kernel's own: pointers, loop positions, staging values.  Whatever the routine calls
its nodes, the kernels read and write those nodes."""
import numpy as np
import pytest

from ocannl_b200 import workloads as W
from tests import test_packed_contractions_gpu as T
from tests.parity import compare, run_device, run_oracle

pytestmark = pytest.mark.gpu


def _renamed(ir, inputs, names):
    for t in ir.tnodes:
        t.ident = names.get(t.ident, t.ident)
    return ir, {names.get(k, k): v for k, v in inputs.items()}


@pytest.mark.parametrize("names", [("v", "p", "acc", "base"), ("row", "v", "shape", "i"), ("rr", "grp", "status", "slot")])
@pytest.mark.parametrize("prec", ["bfloat16", "single"])
def test_gathered_contraction(device, names, prec):
    shape = (2, 65, 77, 333)
    ir = T._mm(*shape, prec, False, True, act=True)
    ir, inputs = _renamed(ir, T._inputs(ir, shape[3]), dict(zip(("x", "w", "bias", "y"), names)))
    want = run_oracle(ir, inputs)
    got, info = run_device(device, ir, inputs)
    assert "gathers operands" in info["stages"][0]["note"] and info["stages"][-1]["kind"] == "gemm", info
    tol = dict(rtol=1e-5, atol=2e-6) if prec == "single" else dict(rtol=2e-2, atol=2e-3)
    compare(ir, got, want, only=[names[3]], **tol)


@pytest.mark.parametrize("keys,options", [(65, "attn=0"), (65, None), (64, None)])
def test_attention(device, keys, options):
    """Separate stages (whose gathering kernel copies the node `v`), the kernel for any rows, the tile kernel."""
    ir = W.attention(2, 8, 65, keys)
    ir, inputs = _renamed(ir, W.attention_inputs(2, 8, 65, keys),
                          {"scores": "x", "max": "mx", "exp_vals": "e", "sum_exp": "sum", "attn": "w", "mask": "row", "q": "p"})
    want = run_oracle(ir, inputs)
    got, info = run_device(device, ir, inputs, options=options)
    assert any("attention" in s["kind"] for s in info["stages"]) == (options is None), info
    compare(ir, got, want, rtol=2e-2, atol=2e-2)


def test_windows_of_a_convolution(device):
    cfg = dict(batch=8, size=16, cin=8, cout=16)
    ir = W.conv2d_update(**cfg)
    ir, inputs = _renamed(ir, W.conv2d_inputs(**cfg), {"x_padded_grad": "sum", "x_padded": "v", "kernel": "p1", "z_grad": "r1"})
    want = run_oracle(ir, inputs)
    got, info = run_device(device, ir, inputs)
    assert any("gathers the windows" in s["note"] for s in info["stages"]), info
    for name in ("y", "kernel_grad", "sum"):
        np.testing.assert_allclose(got[name], want[name], rtol=1e-4, atol=1e-5 * float(np.abs(want[name]).max()), err_msg=name)
