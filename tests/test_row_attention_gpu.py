"""The attention chain with short or odd rows in one kernel: key counts at the
edges of its tiles of 8 and 16, head dimensions of one to eight k steps, fewer queries than a warp takes,
with and without a mask, a row masked throughout, nodes kept or routine-local."""
import numpy as np
import pytest

from ocannl_b200 import workloads as W
from tests.parity import compare, run_device, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,h,s,t,e", [(2, 3, 5, 7, 16), (2, 2, 16, 8, 32), (1, 2, 33, 100, 64), (3, 1, 65, 129, 48),
                                       (1, 1, 200, 255, 32), (2, 1, 30, 256, 128), (1, 4, 17, 31, 112)])
@pytest.mark.parametrize("mode,mask,prec", [("ctx", True, "bfloat16"), ("local", True, "half"), ("ctx", False, "half"), ("local", False, "bfloat16")])
def test_row_attention(device, b, h, s, t, e, mode, mask, prec):
    ir = W.attention(b, h, s, t, prec=prec, mask=mask, row_mode=mode, d_head=e)
    inputs = W.attention_inputs(b, h, s, t, prec=prec, d_head=e)
    if mask:
        inputs["mask"][s // 2] = 0.0        # every key masked: equal weights
    else:
        del inputs["mask"]
    want = run_oracle(ir, inputs)
    got, info = run_device(device, ir, inputs)
    assert any(st["kind"] == "row attention" for st in info["stages"]), info
    compare(ir, got, want, rtol=2e-2, atol=2e-2 if prec == "bfloat16" else 4e-3)


@pytest.mark.parametrize("t", [64, 128, 256])
@pytest.mark.parametrize("mode,prec", [("ctx", "bfloat16"), ("local", "half")])
def test_masked_chunks(device, t, mode, prec):
    """Whole tiles of keys: chunks of 32 keys that are masked for all queries of a warp, rows masked throughout
    alone and 32 together, a single key left in a chunk."""
    s = t + 3
    ir = W.attention(2, 2, s, t, prec=prec, row_mode=mode)
    inputs = W.attention_inputs(2, 2, s, t, prec=prec)
    mask = np.tril(np.ones((s, t)))
    mask[5] = 0.0
    mask[32:64] = 0.0
    mask[70:, t - 33] = 1.0
    inputs["mask"] = mask.reshape(inputs["mask"].shape).astype(inputs["mask"].dtype)
    want = run_oracle(ir, inputs)
    got, info = run_device(device, ir, inputs)
    assert any(st["kind"] == "attention" for st in info["stages"]), info
    compare(ir, got, want, rtol=2e-2, atol=2e-2 if prec == "bfloat16" else 4e-3)


@pytest.mark.parametrize("b,h,s,t,e", [(8, 8, 97, 97, 32), (16, 8, 57, 60, 48), (15, 8, 49, 250, 16), (1, 1, 1, 64, 64), (2, 1, 15, 17, 112)])
@pytest.mark.parametrize("mode,mask,prec", [("ctx", True, "bfloat16"), ("local", True, "half"), ("local", False, "bfloat16")])
def test_warps_that_share_queries(device, b, h, s, t, e, mode, mask, prec):
    """Two warps on 16 queries, one, two, four (one query alone), two of which one has a single key: shares of the keys
    that are empty or masked throughout, output tiles that do not divide by the warps."""
    ir = W.attention(b, h, s, t, prec=prec, mask=mask, row_mode=mode, d_head=e)
    inputs = W.attention_inputs(b, h, s, t, prec=prec, d_head=e)
    if not mask:
        del inputs["mask"]
    else:
        inputs["mask"][s // 2] = 0.0
    # (routine-local nodes would lie on the oracle's stack)
    want = run_oracle(W.attention(b, h, s, t, prec=prec, mask=mask, row_mode="ctx", d_head=e), inputs)
    got, info = run_device(device, ir, inputs)
    assert any(st["kind"] == "row attention" for st in info["stages"]), info
    compare(ir, got, want, rtol=2e-2, atol=2e-2 if prec == "bfloat16" else 4e-3)
