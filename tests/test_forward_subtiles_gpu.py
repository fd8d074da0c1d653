"""The forward's two softmax warpgroups per branch take alternate 64-key sub-tiles and hand the running row maximum over to
each other; a sub-tile that raises it rescales the accumulator both of them add to.  The maximum is made to jump (by far
more than 2^8) at chosen sub-tiles: each warpgroup's first, a later one, both in a row, the last of an odd count."""
import pytest
import torch

from oracle import diffattn_oracle as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("n,jumps1,jumps2", [
    (64, [0], [0]),                 # one real sub-tile: the second warpgroup sees masked columns only
    (65, [1], [0]),                 # one visible column in the second warpgroup's only sub-tile
    (129, [1, 2], [2]),             # hand-over in both directions; a single column in the last tile
    (330, [1, 2, 3], [3, 5]),       # consecutive jumps; odd-numbered sub-tiles only
    (448, [2, 4, 6], [6]),          # even-numbered sub-tiles only; the jump in the last real sub-tile
])
def test_running_maximum_changes_hands(d, n, jumps1, jumps2):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import triton_diff_attn_b200 as pkg
    q1, q2, k1, k2, v, _ = oracle.make_inputs(1, 2, n, d, 300 + n + d)
    for k, jumps in ((k1, jumps1), (k2, jumps2)):
        for step, t in enumerate(jumps):
            k[:, :, 64 * t:64 * (t + 1)] *= 4.0 * (step + 1)
    lam = torch.tensor([0.5])
    want = oracle.forward(q1, q2, k1, k2, v, lam, 0.8, True)
    dev = torch.device("cuda", 0)
    leaves = [t.to(dev).requires_grad_(True) for t in (q1, q2, k1, k2, v)]
    y = pkg.MultiheadDiffAttnKernel(*leaves, lam.to(dev), 0.8, True)
    lse1, lse2 = (t.cpu() for t in y.grad_fn.saved_tensors[8:10])
    pkg.device_status(0)
    m = oracle.error_metrics(y.detach().cpu(), want["y"])
    assert m["rel_l2"] <= 1e-3, m                     # the repository's fp16 bound for every forward output
    # scores reach a few hundred: their fp32 rounding (6e-8 relative) and the exp unit's 2^-22 stay below 1e-5 of lse + 1e-3
    assert torch.allclose(lse1, want["lse1"], atol=2e-3, rtol=1e-5)
    assert torch.allclose(lse2, want["lse2"], atol=2e-3, rtol=1e-5)


@pytest.mark.parametrize("scale", [0.0, -0.1, 0.125])
@pytest.mark.parametrize("b,h,n,d", [(1, 2, 128, 64), (1, 3, 384, 32), (4, 40, 128, 64), (2, 40, 256, 64), (1, 2, 384, 128)])
def test_any_softmax_scale(b, h, n, d, scale):
    """The C entry point takes the scale as it is given: 0 (every key alike) and negative scales (that of negated queries) too, also where
    a CTA goes on to a second tile with the first one's running maximum still in shared memory."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import triton_diff_attn_b200 as pkg
    from triton_diff_attn_b200 import _lib
    q1, q2, k1, k2, v, _ = oracle.make_inputs(b, h, n, d, 700 + n + d)
    lam = torch.tensor([0.5])
    factor = scale * d ** 0.5                         # the oracle scales by 1 / sqrt(D)
    want = oracle.forward(q1.double() * factor, q2.double() * factor, k1.double(), k2.double(), v.double(), lam, 0.2, False)
    dev = torch.device("cuda", 0)
    ins = [t.to(dev) for t in (q1, q2, k1, k2, v)]
    saved = [torch.empty_like(ins[4]), torch.empty_like(ins[4])] + [torch.empty((b, h, n), device=dev) for _ in range(3)]
    glam = lam.to(dev)
    p = _lib.new_params()
    pkg.layers._fill_common(p, *ins, glam, 0.2, False, saved)
    p.sm_scale = scale
    _lib.check(_lib.lib.diffattn_fwd(p), "fwd")
    pkg.device_status(0)
    m = oracle.error_metrics(saved[0].cpu(), want["y"])
    # the repository's fp16 bound (with a negative scale the kernel's reference is the first sub-tile's maximum: unnormalised probabilities reach e^6 here, in range)
    assert m["rel_l2"] <= 1e-3, m
    assert torch.allclose(saved[2].cpu().double(), want["lse1"].double(), atol=2e-3, rtol=1e-5)
    assert torch.allclose(saved[3].cpu().double(), want["lse2"].double(), atol=2e-3, rtol=1e-5)
