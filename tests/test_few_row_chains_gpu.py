"""Layer norms and softmaxes over fewer than 128 rows: a warp a row in registers, or one block together with what
follows.  The decoder of a single short sequence and classifiers whose loss follows their softmax, on either side of
both limits, against the oracle with the tolerance of 16-bit nodes (2e-2 relative, 2e-2 of values of magnitude one)."""
import pytest

from ocannl_b200 import workloads as W
from tests.parity import compare, run_device, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seq,heads,d_head", [(7, 2, 64), (8, 2, 64), (9, 1, 32), (33, 3, 32), (100, 4, 64), (127, 1, 64), (129, 1, 64)])
@pytest.mark.parametrize("fuse", [None, "fuse=0"])
def test_short_decoder(device, seq, heads, d_head, fuse):
    cfg = dict(layers=1, d_model=heads * d_head, heads=heads, d_head=d_head, d_ff=2 * heads * d_head)
    ir = W.transformer_forward(batch=1, seq=seq, **cfg)
    inputs = dict(W.transformer_params(**cfg), **W.transformer_inputs(batch=1, seq=seq))
    want = run_oracle(ir, inputs)
    got, info = run_device(device, ir, inputs, options=fuse)
    if fuse is None and seq >= 33:
        assert sum("one warp per row" in (s["note"] or "") for s in info["stages"]) >= 2, info
    compare(ir, got, want, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("rows,classes", [(20, 40), (60, 50), (100, 40), (103, 40), (100, 64), (127, 33)])
def test_short_batch_with_loss(device, rows, classes):
    dims = (100, 64, 48, classes)
    ir = W.mlp_forward(rows=rows, dims=dims, wprec="single")
    x, labels = W.mlp_inputs(rows=rows, in_dim=100, classes=classes, xprec="single")
    inputs = dict(W.mlp_params(dims=dims, wprec="single"), x=x, labels=labels)
    want = run_oracle(ir, inputs)
    got, info = run_device(device, ir, inputs)
    # the tolerance of the exact single-precision kernels
    compare(ir, got, want, rtol=1e-5, atol=1e-5)
