"""The query-side backward consumes 128-key tiles in four column groups of 32, one group per warpgroup, two of them half a
branch behind the others; the attention dropout mask is walked along rows there and along columns on the key side.  Sequence lengths
put the last visible key at the edges of those groups and tiles, with one tile, an odd and an even number of them."""
import numpy as np
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


@pytest.mark.parametrize("options", [{}, {"causal": True, "bf16": True}, {"p": 0.25}, {"causal": True, "bf16": True, "p": 0.25}])
@pytest.mark.parametrize("b,h,n,d", [(1, 1, 64, 64), (2, 5, 200, 32), (3, 7, 640, 64), (1, 3, 300, 128), (2, 20, 512, 128)])
def test_overlapping_kernels_equal_separate_ones(b, h, n, d, options):
    """In one call the backward's kernels start before the one ahead of them has ended; issued one stage at a time they do not.
    Several calls follow each other on the stream with fresh inputs in the same buffers, smaller and larger than the chip."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import triton_diff_attn_b200 as pkg
    from triton_diff_attn_b200 import _lib
    dev = torch.device("cuda", 0)
    dt = torch.bfloat16 if options.get("bf16") else torch.float16
    ins = [t.to(dev, dt) for t in oracle.make_inputs(b, h, n, d, 77)]
    q1, q2, k1, k2, v, dy = ins
    lam = torch.tensor([0.5], device=dev)
    saved = [torch.empty_like(v), torch.empty_like(v)] + [torch.empty((b, h, n), device=dev) for _ in range(3)]
    grads = [torch.empty_like(t) for t in (q1, q2, k1, k2, v)]
    dlam = torch.zeros(1, device=dev)
    p = _lib.new_params()
    pkg.layers._fill_common(p, q1, q2, k1, k2, v, lam, 0.2, True, saved, options.get("causal", False),
                            pkg.layers.dropout_threshold(options.get("p", 0.0)), 4321)
    ws = torch.empty(_lib.lib.diffattn_workspace_bytes(p), dtype=torch.uint8, device=dev)
    p.dy, p.dlambda, p.workspace, p.workspace_bytes = dy.data_ptr(), dlam.data_ptr(), ws.data_ptr(), ws.numel()
    p.dq1, p.dq2, p.dk1, p.dk2, p.dv = (t.data_ptr() for t in grads)

    def rounds(step):
        out = []
        for i in range(4):
            for t, fresh in zip(ins, oracle.make_inputs(b, h, n, d, 200 + i)):
                t.copy_(fresh)
            _lib.check(_lib.lib.diffattn_fwd(p), "fwd")
            step()
            out += [g.clone() for g in grads]      # right behind the call: whoever follows it must see every gradient complete
        return out

    def separate():
        for stage in (_lib.STAGE_PRE, _lib.STAGE_DKDV, _lib.STAGE_DQ):
            _lib.check(_lib.lib.diffattn_bwd_stages(p, stage), "stage")
            torch.cuda.synchronize()

    want = rounds(separate)
    got = rounds(lambda: _lib.check(_lib.lib.diffattn_bwd(p), "bwd"))
    # dQ waits for dK/dV before it stores, and a CTA of it reads no query rows but its own: dq1, dq2 may lie over q1, q2
    p.dq1, p.dq2 = q1.data_ptr(), q2.data_ptr()
    grads[:2] = [q1, q2]
    got += rounds(lambda: _lib.check(_lib.lib.diffattn_bwd(p), "bwd"))
    pkg.device_status(0)
    assert all(torch.equal(a, w) for a, w in zip(got, want + want))


def _bnhd(t):
    """The same values as a view of [B, N, H, D] storage."""
    return t.transpose(1, 2).contiguous().transpose(1, 2)


def _dlambda_tolerance(want, loosen):
    # the repository's bound for this cancelling sum
    return loosen * max(1e-2 * abs(float(want["dlambda"])), 1e-4 * float(want["e2"].abs().sum()), 2e-3)


@pytest.mark.parametrize("b,h,n,d,causal,p,gain,options", [
    (10, 16, 33, 64, False, 0.0, False, {}),      # one tile per head, just more items than SMs
    (16, 20, 100, 64, True, 0.25, True, {}),      # one tile per head, three rounds
    (5, 16, 200, 32, False, 0.0, True, {}),       # two tiles; head dim 32 (one dV store)
    (5, 20, 385, 64, True, 0.0, False, {}),       # four tiles of unequal cost, backward rounds
    (3, 25, 300, 64, False, 0.25, True, {}),      # an odd number of tiles: the rings change slots from item to item
    (4, 40, 257, 32, True, 0.0, True, {}),        # under a mask all heads are one group
    (2, 80, 129, 64, False, 0.0, True, {}),
    (17, 61, 257, 64, True, 0.0, False, {}),      # heads in three groups, the last one smaller
    (5, 16, 200, 32, False, 0.0, True, {"bf16": True, "lam": -0.4}),
    (16, 20, 100, 64, True, 0.25, True, {"bf16": True}),
    (3, 25, 300, 64, False, 0.25, False, {"bf16": True, "lam": -0.4, "bnhd": True}),
    (5, 20, 385, 64, True, 0.0, False, {"lam": -0.4, "bnhd": True}),
    (3, 25, 300, 64, True, 0.0, True, {"bf16": True}),
    (4, 40, 257, 32, True, 0.0, False, {"bf16": True, "bnhd": True}),
])
def test_several_tiles_per_cta(b, h, n, d, causal, p, gain, options):
    """With more tiles than SMs a CTA works on one tile after the other: outputs and gradients of every head against the oracle."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import triton_diff_attn_b200 as pkg
    loosen, dt = (8, torch.bfloat16) if options.get("bf16") else (1, torch.float16)
    ins = [t.to(dt) for t in oracle.make_inputs(b, h, n, d, 50 + n)]
    q1, q2, k1, k2, v, dy = ins
    # (dropout without the output norm: under a causal mask the first rows keep a key or none, A_1 - lambda A_2 can all but vanish there,
    # and the norm's 1 / rms then amplifies the 16-bit rounding of the operands in any implementation)
    lam, seed, rms = torch.tensor([options.get("lam", 0.5)]), 99, p == 0.0
    g = torch.linspace(0.5, 1.5, 2 * d) if gain else None
    extra = {"dropout_threshold": pkg.layers.dropout_threshold(p), "dropout_seed": seed} if p else {}
    want = oracle.backward_closed_form(q1, q2, k1, k2, v, lam, dy, 0.2, rms, causal=causal, gain=g, **extra)
    dev = torch.device("cuda", 0)
    place = _bnhd if options.get("bnhd") else (lambda t: t)
    leaves = [place(t.to(dev)).requires_grad_(True) for t in (q1, q2, k1, k2, v)]
    glam = lam.to(dev).requires_grad_(True)
    gg = g.to(dev).requires_grad_(True) if gain else None
    for _ in range(2):
        y = pkg.MultiheadDiffAttnKernel(*leaves, glam, 0.2, rms, causal=causal, dropout_p=p, dropout_seed=seed, gain=gg)
        grads = torch.autograd.grad(y, leaves + [glam] + ([gg] if gain else []), place(dy.to(dev)))
    pkg.device_status(0)
    for name, got, ref in [("y", y.detach(), want["y_gained" if gain else "y"])] + [(k, t, want[k]) for k, t in zip(("dq1", "dq2", "dk1", "dk2", "dv"), grads)]:
        # the repository's bound (rel-L2 1e-3 in fp16, 8 times that in bf16), for each head: a wrong tile must not hide among the others
        err = (got.float().cpu() - ref.float()).flatten(2).norm(dim=2)
        assert bool((err <= loosen * 1e-3 * ref.float().flatten(2).norm(dim=2)).all()), (name, float((err / ref.float().flatten(2).norm(dim=2)).max()))
    assert abs(float(grads[5]) - float(want["dlambda"])) <= _dlambda_tolerance(want, loosen)
    if gain:
        assert oracle.error_metrics(grads[6].cpu(), want["dgain"])["rel_l2"] <= loosen * 1e-3


@pytest.mark.parametrize("bf16", [False, True])
def test_core_with_several_tiles_per_cta(bf16):
    """The layer core on head-interleaved projections, more tiles than SMs: gain and lambda vectors included."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import triton_diff_attn_b200 as pkg
    b, h, n, d = 4, 20, 300, 64
    loosen, dt = (8, torch.bfloat16) if bf16 else (1, torch.float16)
    dev = torch.device("cuda", 0)
    ins = [t.to(dt) for t in oracle.make_inputs(b, h, n, d, 61)]
    core = pkg.DiffAttnCore(d, lambda_init=0.2, causal=True, device=dev)
    with torch.no_grad():
        core.gain.copy_(torch.linspace(0.5, 1.5, 2 * d))
        for t in (core.lambda_q1, core.lambda_k1, core.lambda_q2, core.lambda_k2):
            t.copy_(torch.linspace(-0.1, 0.2, d) if t is core.lambda_q1 or t is core.lambda_k1 else torch.linspace(0.1, -0.05, d))
    vec = [t.detach().double().cpu() for t in (core.lambda_q1, core.lambda_k1, core.lambda_q2, core.lambda_k2)]
    e1, e2 = torch.exp((vec[0] * vec[1]).sum()), torch.exp((vec[2] * vec[3]).sum())
    lam = (e1 - e2 + 0.2).reshape(1)
    want = oracle.backward_closed_form(*ins[:5], lam, ins[5], 0.2, True, causal=True, gain=core.gain.detach().cpu())
    leaves = [_bnhd(t.to(dev)).requires_grad_(True) for t in ins[:5]]
    wrt = leaves + [core.lambda_q1, core.lambda_k1, core.lambda_q2, core.lambda_k2, core.gain]
    y = core(*leaves)
    grads = torch.autograd.grad(y, wrt, _bnhd(ins[5].to(dev)))
    pkg.device_status(0)
    for name, got, ref in [("y", y.detach(), want["y_gained"]), ("dgain", grads[9], want["dgain"])] + [
            (k, t, want[k]) for k, t in zip(("dq1", "dq2", "dk1", "dk2", "dv"), grads)]:
        assert oracle.error_metrics(got.cpu(), ref)["rel_l2"] <= loosen * 1e-3, name
    tol = _dlambda_tolerance(want, loosen)
    for got, factor in zip(grads[5:9], (e1 * vec[1], e1 * vec[0], -e2 * vec[3], -e2 * vec[2])):
        assert bool(((got.cpu().double() - float(want["dlambda"]) * factor).abs() <= tol * factor.abs() + 1e-6).all())


@pytest.mark.parametrize("n", [1, 32, 64, 128, 300])
@pytest.mark.parametrize("create_graph", [False, True])
def test_core_lambda_in_one_launch(n, create_graph):
    """lambda and the four vectors' gradients against 64 bits: sums of n products and one exponential in fp32."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import triton_diff_attn_b200 as pkg
    dev = torch.device("cuda", 0)
    gen = torch.Generator().manual_seed(n)
    host = [torch.randn(n, generator=gen) * 0.2 for _ in range(4)]
    ref = [t.double().requires_grad_(True) for t in host]
    want = torch.exp((ref[0] * ref[1]).sum()) - torch.exp((ref[2] * ref[3]).sum()) + 0.8
    wg = torch.autograd.grad(want, ref, torch.tensor(1.7, dtype=torch.float64))
    vec = [torch.nn.Parameter(t.to(dev)) for t in host]
    lam = pkg.layers._core_lambda(vec, 0.8, vec[0].device)
    got = torch.autograd.grad(lam, vec, torch.full((1,), 1.7, device=dev), create_graph=create_graph)
    # n products of at most 1 in magnitude summed in fp32 (n 2^-24), an exponential of |x| < 10 (2^-22), a difference of O(1) terms
    assert abs(float(lam.detach()) - float(want.detach())) <= 1e-5 * (1 + abs(float(want.detach())))
    for a, b in zip(got, wg):
        assert torch.allclose(a.detach().cpu().double(), b, rtol=1e-5, atol=1e-6)
    if create_graph:
        assert all(t is not None for t in torch.autograd.grad(sum(t.sum() for t in got), vec))
    for number in (np.float32(0.75), np.array(0.75), torch.tensor(0.75)):        # whatever float() takes, as in tensor operations
        assert torch.equal(pkg.layers._core_lambda(vec, number, dev), pkg.layers._core_lambda(vec, 0.75, dev))
    half = [t.half().to(dev) for t in host]                      # anything but fp32 goes through tensor operations as before
    assert torch.equal(pkg.layers._core_lambda(half, 0.8, dev), pkg.lambda_from_reparam(*half, 0.8))
