"""The query-side backward consumes 128-key tiles in four column groups of 32, one group per warpgroup, two of them half a
branch behind the others; the attention dropout mask is walked along rows there and along columns on the key side.  Sequence lengths
put the last visible key at the edges of those groups and tiles, with one tile, an odd and an even number of them."""
import pytest
import torch

from oracle import diffattn_oracle as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("causal,p", [(False, 0.0), (True, 0.0), (False, 0.25), (True, 0.25)])
@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("n", [31, 33, 64, 65, 97, 128, 129, 255, 257, 385])
def test_gradients_at_tile_edges(d, n, causal, p):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import triton_diff_attn_b200 as pkg
    q1, q2, k1, k2, v, dy = oracle.make_inputs(1, 2, n, d, 900 + n + d)
    lam, seed = torch.tensor([0.5]), 4321
    extra = {"dropout_threshold": pkg.layers.dropout_threshold(p), "dropout_seed": seed} if p else {}
    want = oracle.backward_closed_form(q1, q2, k1, k2, v, lam, dy, 0.2, True, causal=causal, **extra)
    dev = torch.device("cuda", 0)
    leaves = [t.to(dev).requires_grad_(True) for t in (q1, q2, k1, k2, v)]
    y = pkg.MultiheadDiffAttnKernel(*leaves, lam.to(dev), 0.2, True, causal=causal, dropout_p=p, dropout_seed=seed)
    grads = torch.autograd.grad(y, leaves, dy.to(dev))
    pkg.device_status(0)
    for name, g in zip(("dq1", "dq2", "dk1", "dk2", "dv"), grads):
        m = oracle.error_metrics(g.cpu(), want[name])
        # the repository's fp16 bound.  (A single token is left to the parity tests: its score gradients are zero up to the
        # 16-bit rounding of the saved outputs, so they have no relative error.)
        assert m["rel_l2"] <= 1e-3, (name, m)
