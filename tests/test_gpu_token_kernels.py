"""The token-at-a-time kernels (csrc/generic.cu): what the chunked ones have no room for beside the state, on the causal path and
in the state reduction; and the widest geometries that the chunked ones do take, on the other side of that line.

Against fp64 with the gates of test_gpu_chunked.py: 4e-4 in the 2-norm for fp16 results and three spacings of fp16's
smallest numbers, 2e-6 for the fp32 states."""
import pytest
import torch

from rfa_b200.rfa import RFA
from test_gpu_chunked import inputs, rel

pytestmark = pytest.mark.gpu

TOKEN = [(384, 128), (768, 64), (2048, 8), (1032, 16)]      # the last: chunks would fit, but are built for widths up to 1024
CHUNKED = [(1024, 32), (8, 1024)]


def reference(q, k, v, g):
    d = [t.double() for t in (q, k, v, g)]
    return (RFA.forward_torch(*d[:3]), *RFA.backward_torch(*d))


def state(k, v):
    return torch.einsum("tbk,tbd->bkd", k.double(), v.double()), k.double().sum(0)


@pytest.mark.parametrize("K,d", TOKEN + CHUNKED)
@pytest.mark.parametrize("T,BH", [(1, 1), (37, 2)])
def test_causal(dev, K, d, T, BH):
    from rfa_b200 import ops
    ins = inputs(T, BH, K, d, K + T)
    want = reference(*ins)
    q, k, v, g = (t.to(dev) for t in ins)
    leaves = [t.clone().requires_grad_() for t in (q, k, v)]
    out = RFA.apply(*leaves)                              # from the saved forward
    out.backward(g)
    got = [("out", out), *zip(("gq", "gk", "gv"), [t.grad for t in leaves])]
    got += zip(("gq again", "gk again", "gv again"), ops.causal_bwd(q, k, v, g))
    for (name, a), b in zip(got, want + want[1:]):
        # one token out of the clamp has out = v whatever q and k are, and gq, gk exactly zero: two equal terms of |g . out| inv z, at most
        # 45 * 0.2 = 9, that cancel in fp32 sums of a few hundred products (20 units of 2^-24 each): 1e-5, nothing relative
        if float(b.abs().max()) < 1e-12:
            assert float(a.abs().max()) < 1e-5, name
            continue
        assert rel(a, b, 2.0 ** -24) < 4e-4, name
    _, s, z = ops.causal_fwd(q, k, v, return_state=True)
    S, Z = state(ins[1], ins[2])
    assert rel(s, S) < 2e-6 and rel(z, Z) < 2e-6


@pytest.mark.parametrize("K,d", TOKEN)
def test_carried_states(dev, K, d):
    """A sequence in two parts: the state handed on, the reverse state handed back."""
    from rfa_b200 import ops
    T, BH, cut = 40, 2, 23
    ins = inputs(T, BH, K, d, K)
    want = reference(*ins)
    (q1, k1, v1, g1), (q2, k2, v2, g2) = ([t[part].to(dev) for t in ins] for part in (slice(0, cut), slice(cut, T)))
    o1, s, z = ops.causal_fwd(q1, k1, v1, return_state=True)
    o2 = ops.causal_fwd(q2, k2, v2, s, z)
    assert rel(torch.cat([o1, o2]), want[0], 2.0 ** -24) < 4e-4
    if K * (d + 1) * 8 > 220 * 1024:                      # two states do not fit: the second part's reverse total from fp64
        with pytest.raises(ValueError, match="two of them"):
            ops.causal_bwd_q(q2, k2, v2, g2, s, z, True)
        q, k, v, g = (t.double() for t in ins)
        raw = (q * torch.cumsum(k, 0)).sum(-1, keepdim=True)
        inv = 1 / raw.clamp_min(1)
        gz = -(g * want[0]).sum(-1, keepdim=True) * inv * (raw > 1)
        ds = torch.einsum("tbk,tbd->bkd", q[cut:], (g * inv)[cut:]).float().to(dev)
        dz = (q * gz)[cut:].sum(0).float().to(dev)
        gq2, _, _, ws = ops.causal_bwd_q(q2, k2, v2, g2, s, z, False)
    else:
        gq2, ds, dz, ws = ops.causal_bwd_q(q2, k2, v2, g2, s, z, True)
    gk2, gv2 = ops.causal_bwd_kv(q2, k2, v2, g2, None, None, ws)
    first = ops.causal_bwd(q1, k1, v1, g1, None, None, ds.contiguous(), dz.contiguous())
    for name, a, b, ref in zip(("gq", "gk", "gv"), first, (gq2, gk2, gv2), want[1:]):
        assert rel(torch.cat([a, b]), ref, 2.0 ** -24) < 4e-4, name


@pytest.mark.parametrize("K,d", TOKEN + CHUNKED)
def test_state_reduction(dev, K, d):
    from rfa_b200 import ops
    T, B, H = 150, 2, 2
    _, k, v, _ = inputs(T, B * H, K, d, 3)
    pad = torch.arange(T)[None] >= torch.tensor([T, 70])[:, None]
    s, z = ops.cross_state_fwd(k.view(T, B, H, K).to(dev), v.view(T, B, H, d).to(dev), pad.to(dev))
    live = (~pad).t()[:, :, None, None]
    S, Z = state((k.view(T, B, H, K) * live).view(T, B * H, K), v)
    assert rel(s.view(B * H, K, d), S) < 2e-6 and rel(z.view(B * H, K), Z) < 2e-6
    _, k, v, _ = inputs(1100, 2, K, d, 4)                 # in two runs of tokens
    s, z = ops.state_total(k.to(dev), v.to(dev))
    S, Z = state(k, v)
    assert rel(s, S) < 2e-6 and rel(z, Z) < 2e-6
