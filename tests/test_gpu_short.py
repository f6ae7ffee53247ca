"""Sequences of one chunk on their own kernels (csrc/causal_short.cu): against the oracle, and against the general kernels, which
the same call reaches when a state is asked for (forward) or the sweeps are called one by one (backward).

Gates: the oracle's 2e-3 / 1e-2 of the other parity tests; between the two paths, whose operands are rounded alike and whose
fp32 sums differ in order, a rounding of the fp16 result (2^-11 relative at worst) and of the operands that a sum's last
bit tips: 6e-4 in the 2-norm."""
import pytest
import torch

from conftest import assert_close
from oracle import rfa_oracle as O
from rfa_b200 import _lib, ops

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30))


@pytest.mark.parametrize("scale", [0.3, 3.0])          # denominators in the clamp, and far out of it
@pytest.mark.parametrize("T", [1, 2, 15, 16, 17, 33, 45, 64, 65, 100, 127, 128, 129])
def test_short_sequences(dev, T, scale):
    BH = 3
    gen = torch.Generator().manual_seed(T)
    q, k = ((torch.rand(T, BH, 128, generator=gen) * scale - 0.1).half() for _ in range(2))
    v, g = (torch.randn(T, BH, 64, generator=gen).half() for _ in range(2))
    f = [t.float() for t in (q, k, v)]
    want, grads = O.causal_forward(*f), O.causal_backward(*f, g.float())
    q, k, v, g = (t.to(dev) for t in (q, k, v, g))
    out, ws, has = ops.causal_fwd_saved(q, k, v)
    got = ops.causal_bwd_saved(q, k, v, g, out, ws, has)
    rows = 1e-2 * max(1.0, float(want.abs().max()))
    assert_close(out, want, "out", mabs=rows)
    # one token out of the clamp has out = v whatever q and k are: its gq and gk are zero, two equal terms of g . out inv z (at most 64 * 16 *
    # 3 / 100 = 30) whose fp16 operands differ by 2^-11 each: 3e-2, and nothing relative
    zero = T == 1 and scale > 1
    for name, a, b in zip(("gq", "gk", "gv"), got, grads):
        if zero and name != "gv":
            assert float(a.abs().max()) < 3e-2
            continue
        assert_close(a, b, name, mabs=1e-2 * max(1.0, float(b.abs().max())))
    assert torch.equal(ops.causal_fwd(q, k, v), out)
    # the general path on the same inputs and the same saved output
    general, _, _ = ops.causal_fwd(q, k, v, return_state=True)
    assert rel(out, general) < 6e-4
    ws2 = ws.clone()
    gq, _ = ops.causal_bwd_q_staged(q, k, v, g, out, None, None, ws2, _lib.WS_DEN, want_total=False)
    gk, gv = ops.causal_bwd_kv(q, k, v, g, None, None, ws2)
    for name, a, b in zip(("gq", "gk", "gv"), got, (gq, gk, gv)):
        if zero and name != "gv":
            continue
        assert rel(a, b) < 6e-4, name


@pytest.mark.parametrize("state_dtype,in_dtype", [(torch.float32, torch.float16), (torch.float16, torch.float16), (torch.float32, torch.float32)])
@pytest.mark.parametrize("B,H", [(130, 8), (41, 27)])          # just over one wave of the one-head-per-CTA kernel; heads that split unevenly
def test_decode_of_many_heads(dev, state_dtype, in_dtype, B, H):
    """The streaming kernel against the general one, which the same call reaches for half of the batch at a time.  A projection
    summed in another order may round a feature to the neighbouring fp16 number (2^-11): 1e-3."""
    gen = torch.Generator().manual_seed(B)
    rnd = lambda *s: torch.randn(*s, generator=gen).to(dev)
    w, (q, k, v) = rnd(H, 64, 64), (rnd(B, H, 64).to(in_dtype) for _ in range(3))
    s, z = (rnd(B, H, 128, 64) * 0.1).to(state_dtype), (rnd(B, H, 128) * 0.1 + 1.0).to(state_dtype)
    s1, z1, s2, z2 = s.clone(), z.clone(), s.clone(), z.clone()
    outs = [ops.decode_step_fused(q, k, v, w, 0.1, s1, z1) for _ in range(2)]
    for i in range(2):
        halves = [ops.decode_step_fused(q[a], k[a], v[a], w, 0.1, s2[a], z2[a]) for a in (slice(0, B // 2), slice(B // 2, B))]
        assert rel(outs[i], torch.cat(halves)) < 1e-3
    assert rel(s1, s2) < 1e-3 and rel(z1, z2) < 1e-3


@pytest.mark.parametrize("head_dim,proj_dim,dtype", [(64, 64, torch.float16), (32, 32, torch.float16), (128, 128, torch.float32), (24, 32, torch.float16)])
def test_layer_decode_step_against_the_differentiable_path(dev, head_dim, proj_dim, dtype):
    """One token through the layer: with gradients recorded it goes through feature map and causal kernel, without through the
    fused decoding step (head_dim 24 is none of its widths, and of no decoding kernel's: refused in both forms)."""
    from rfa_b200 import CausalAttention
    torch.manual_seed(0)
    layer = CausalAttention(embed_dim=4 * head_dim, num_heads=4, head_dim=head_dim, proj_dim=proj_dim, tau=0.5).to(dev).to(dtype)
    w = torch.randn(4, proj_dim, head_dim, device=dev, dtype=dtype)
    plain, recorded = {}, {}
    for _ in range(3):
        x = torch.randn(1, 3, 4 * head_dim, device=dev, dtype=dtype)
        y = layer(x, w, saved_state=recorded)
        recorded = {k: t.detach() for k, t in recorded.items()}
        with torch.no_grad():
            if head_dim == 24:
                with pytest.raises(ValueError, match="head_dim"):
                    layer(x, w, saved_state=plain)
                continue
            assert rel(layer(x, w, saved_state=plain), y) < 4e-3
    if head_dim != 24:
        assert rel(plain["prev_s"], recorded["prev_s"]) < 2e-3 and rel(plain["prev_z"], recorded["prev_z"]) < 2e-3
        assert plain["prev_s"].dtype == torch.float32


@pytest.mark.parametrize("state_dtype,in_dtype", [(torch.float32, torch.float16), (torch.float16, torch.float16), (torch.float32, torch.float32)])
@pytest.mark.parametrize("d", [4, 8, 32, 64, 128])
@pytest.mark.parametrize("D", [8, 16, 24, 32, 40, 48, 56, 64, 72, 128, 136])
def test_fused_decode_of_any_width(dev, D, d, in_dtype, state_dtype):
    """Every way the projection is spread over a CTA's lanes (16 lanes a row at D = 8 down to one from D = 72 on), with D ending inside
    a warp's rows at 40 and 56; against fp64.  fp16 features and state are rounded once (2^-11, 2.9e-4 in the 2-norm) and their errors add up
    over an output's features: 1e-3; fp32: sums of d and 2 D terms, 2e-6."""
    B, H = 2, 3
    gen = torch.Generator().manual_seed(D + d)
    q, k, v = (torch.randn(B, H, d, generator=gen).to(in_dtype) for _ in range(3))
    w = torch.randn(H, D, d, generator=gen)
    s, z = (torch.randn(B, H, 2 * D, d, generator=gen) * 0.1).to(state_dtype), torch.rand(B, H, 2 * D, generator=gen).to(state_dtype)

    def phi(x):
        x = x.double()
        u = torch.einsum("bhd,hkd->bhk", x / (x.norm(dim=-1, keepdim=True) + 1e-3), w.double())
        return 0.1 * torch.cat([u.sin(), u.cos()], dim=-1)
    pq, pk = phi(q), phi(k)
    S, Z = s.double() + pk[..., None] * v.double()[..., None, :], z.double() + pk
    want = torch.einsum("bhk,bhkd->bhd", pq, S) / (pq * Z).sum(-1, keepdim=True).clamp_min(1)
    sg, zg = s.to(dev), z.to(dev)
    out = ops.decode_step_fused(q.to(dev), k.to(dev), v.to(dev), w.to(dev), 0.1, sg, zg)
    gate = 2e-6 if in_dtype == torch.float32 else 1e-3
    assert rel(out.cpu(), want) < gate and rel(sg.cpu(), S) < gate and rel(zg.cpu(), Z) < gate


@pytest.mark.parametrize("proj_dim", [40, 56])
def test_layer_decodes_with_a_proj_dim_that_ends_inside_a_warp(dev, proj_dim):
    """CausalAttention, one token at a time, against the same layer over the whole sequence."""
    from rfa_b200 import CausalAttention
    torch.manual_seed(proj_dim)
    layer = CausalAttention(embed_dim=64, num_heads=2, head_dim=32, proj_dim=proj_dim).to(dev).half()
    x, w = torch.randn(5, 3, 64, device=dev).half(), torch.randn(2, proj_dim, 32, device=dev).half()
    saved = {}
    with torch.no_grad():
        steps = torch.cat([layer(x[t:t + 1], w, saved_state=saved) for t in range(5)])
        assert_close(steps, layer(x, w), "decoded")
