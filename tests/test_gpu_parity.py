"""Parity of the sm_100a kernels (called through the C ABI) with the CPU oracle and
with the fixtures produced by the upstream Python sources.

Gate for fp16 kernels against the fp32 oracle on identical fp16-valued inputs:
relative L2 error <= 2e-3 and max abs error <= 1e-2, outputs and all gradients
(REL_L2_TOL / MAX_ABS_TOL in conftest.py).  fp32-state quantities (S, z) are held
to 1e-4 relative."""
import numpy as np
import pytest
import torch

from conftest import assert_close, golden
from oracle import rfa_oracle as O

pytestmark = pytest.mark.gpu


def h16(t):
    return t.half().float()


def feats(T, BH, seed, scale=1.0):
    """phi-like inputs: fp16-valued q,k [T,BH,128], v,g [T,BH,64]."""
    gen = torch.Generator().manual_seed(seed)
    w = torch.from_numpy(O.draw_matrices("orf", 1, 64, 64, seed + 100)).float()
    xq, xk = torch.randn(T, BH, 1, 64, generator=gen), torch.randn(T, BH, 1, 64, generator=gen)
    q = h16(O.random_project(xq, w)).view(T, BH, 128) * scale
    k = h16(O.random_project(xk, w)).view(T, BH, 128) * scale
    v = h16(torch.randn(T, BH, 64, generator=gen))
    g = h16(torch.randn(T, BH, 64, generator=gen))
    return h16(q), h16(k), v, g


# ----------------------------------------------------------------------------- causal
def run_causal(dev, q, k, v, g, **kw):
    from rfa_b200 import ops
    cu = lambda t: None if t is None else t.to(dev)
    qh, kh, vh, gh = (t.half().to(dev) for t in (q, k, v, g))
    out = ops.causal_fwd(qh, kh, vh, cu(kw.get("s0")), cu(kw.get("z0")))
    gq, gk, gv = ops.causal_bwd(qh, kh, vh, gh, cu(kw.get("s0")), cu(kw.get("z0")), cu(kw.get("ds")), cu(kw.get("dz")))
    torch.cuda.synchronize()
    return out, gq, gk, gv


@pytest.mark.parametrize("name", ["causal_fwd_gradcheck", "causal_bwd_gradcheck", "causal_features"])
def test_causal_against_upstream_fixtures(dev, name):
    g = golden(name)
    up = g["g"] if "g" in g else torch.ones_like(g["v"])
    out, gq, gk, gv = run_causal(dev, g["q"], g["k"], g["v"], up)
    assert_close(out, g["attn"], f"{name}.attn")
    if "gq" in g:
        assert_close(gq, g["gq"], f"{name}.gq")
        assert_close(gk, g["gk"], f"{name}.gk")
        assert_close(gv, g["gv"], f"{name}.gv")
        # upstream's own criterion (grad_check.py:13-14): squared difference < 1e-4 everywhere
        for a, b in ((gq, g["gq"]), (gk, g["gk"]), (gv, g["gv"]), (out, g["attn"])):
            assert ((a.float().cpu() - b) ** 2 < 1e-4).all()


@pytest.mark.parametrize("T,BH", [(1, 1), (2, 3), (63, 2), (64, 2), (65, 2), (131, 3), (513, 2), (1100, 2), (2048, 5)])
def test_causal_vs_oracle_shapes(dev, T, BH):
    """Ragged lengths around the chunk size, one-token sequences, and (T >= 1024, few
    heads) the segmented path with its pre-pass + scan."""
    q, k, v, g = feats(T, BH, seed=T * 7 + BH)
    out, gq, gk, gv = run_causal(dev, q, k, v, g)
    ro = O.causal_forward(q, k, v)
    rq, rk, rv = O.causal_backward(q, k, v, g)
    assert_close(out, ro, "out"); assert_close(gq, rq, "gq"); assert_close(gk, rk, "gk"); assert_close(gv, rv, "gv")


@pytest.mark.parametrize("T,BH", [(1, 1), (63, 2), (65, 2), (131, 3), (513, 2), (1100, 2), (2048, 5), (4096, 130)])
def test_causal_saved_output_backward_vs_oracle(dev, T, BH):
    """The backward that reuses the forward's output, raw denominators and segment states (what RFA.apply runs) instead of
    recomputing them: ragged lengths, the segmented plan (T >= 1024 with few heads: also reads q for the segment totals)
    and more heads than SMs."""
    from rfa_b200 import ops
    q, k, v, g = feats(T, BH, seed=T * 5 + BH)
    qh, kh, vh, gh = (t.half().to(dev) for t in (q, k, v, g))
    out, ws, has = ops.causal_fwd_saved(qh, kh, vh)
    gq, gk, gv = ops.causal_bwd_saved(qh, kh, vh, gh, out, ws, has)
    gq2, gk2, gv2 = ops.causal_bwd_saved(qh, kh, vh, gh, out, ws, has)          # the kept workspace survives a backward
    torch.cuda.synchronize()
    heads = slice(0, min(BH, 6))
    ro = O.causal_forward(q[:, heads], k[:, heads], v[:, heads])
    rq, rk, rv = O.causal_backward(q[:, heads], k[:, heads], v[:, heads], g[:, heads])
    assert_close(out[:, heads], ro, "out"); assert_close(gq[:, heads], rq, "gq")
    assert_close(gk[:, heads], rk, "gk"); assert_close(gv[:, heads], rv, "gv")
    assert torch.equal(gq, gq2) and torch.equal(gk, gk2) and torch.equal(gv, gv2)
    rec = ops.causal_bwd(qh, kh, vh, gh)                                           # the recomputing backward agrees
    for name, a, b in zip(("gq", "gk", "gv"), (gq, gk, gv), rec):
        assert_close(a, b.float().cpu(), f"{name} vs recomputing backward", rel=1e-3)


def test_causal_saved_output_backward_with_carries(dev):
    """Saved-output backward of the second part of a split sequence: state carried in, reverse-state total out."""
    from rfa_b200 import ops
    T, BH, cut = 1500, 2, 1100
    q, k, v, g = feats(T, BH, seed=91)
    rq, rk, rv = O.causal_backward(q, k, v, g)
    c = lambda t: t.half().to(dev)
    _, s, z = ops.causal_fwd(c(q[:cut]), c(k[:cut]), c(v[:cut]), return_state=True)
    out2, ws, has = ops.causal_fwd_saved(c(q[cut:]), c(k[cut:]), c(v[cut:]), s, z)
    gq2, dpacked = ops.causal_bwd_q_staged(c(q[cut:]), c(k[cut:]), c(v[cut:]), c(g[cut:]), out2, s, z, ws, has)
    gk2, gv2 = ops.causal_bwd_kv(c(q[cut:]), c(k[cut:]), c(v[cut:]), c(g[cut:]), None, None, ws)
    ds, dz = dpacked[:, :128 * 64].reshape(BH, 128, 64).contiguous(), dpacked[:, 128 * 64:].contiguous()
    gq1, gk1, gv1 = ops.causal_bwd(c(q[:cut]), c(k[:cut]), c(v[:cut]), c(g[:cut]), None, None, ds, dz)
    assert_close(out2, O.causal_forward(q, k, v)[cut:], "out (second part)")
    assert_close(torch.cat([gq1, gq2]), rq, "gq"); assert_close(torch.cat([gk1, gk2]), rk, "gk")
    assert_close(torch.cat([gv1, gv2]), rv, "gv")


def generic_feats(T, BH, K, d, seed):
    gen = torch.Generator().manual_seed(seed)
    q = h16(torch.rand(T, BH, K, generator=gen) * 0.3 - 0.1)
    k = h16(torch.rand(T, BH, K, generator=gen) * 0.3 - 0.1)
    return q, k, h16(torch.randn(T, BH, d, generator=gen)), h16(torch.randn(T, BH, d, generator=gen))


@pytest.mark.parametrize("K,d", [(64, 32), (256, 128), (96, 40), (128, 128)])
def test_other_geometries(dev, K, d):
    """On the chunked kernels (test_gpu_token_kernels.py: what stays on the token-at-a-time ones).  Feature widths / head dims other than 128 / 64 (upstream accepts any K % 16 == 0, d % 8 == 0): causal forward,
    both backward forms (recomputing and RFA.apply's), state carries and the reverse-state total, against the oracle."""
    from rfa_b200 import ops
    from rfa_b200.rfa import RFA
    T, BH, cut = 150, 3, 90
    q, k, v, g = generic_feats(T, BH, K, d, seed=K + d)
    c = lambda t: t.half().to(dev)
    ro = O.causal_forward(q, k, v); rq, rk, rv = O.causal_backward(q, k, v, g)
    out = ops.causal_fwd(c(q), c(k), c(v)); gq, gk, gv = ops.causal_bwd(c(q), c(k), c(v), c(g))
    assert_close(out, ro, "out"); assert_close(gq, rq, "gq"); assert_close(gk, rk, "gk"); assert_close(gv, rv, "gv")
    leaves = [c(t).requires_grad_(True) for t in (q, k, v)]
    RFA.apply(*leaves).backward(c(g))
    for name, leaf, ref in zip(("gq", "gk", "gv"), leaves, (rq, rk, rv)):
        assert_close(leaf.grad, ref, f"RFA.apply {name}")
    # split run: state carried in and out, reverse-state total handed back
    o1, s, z = ops.causal_fwd(c(q[:cut]), c(k[:cut]), c(v[:cut]), return_state=True)
    o2, s2, z2 = ops.causal_fwd(c(q[cut:]), c(k[cut:]), c(v[cut:]), s, z, return_state=True)
    assert_close(torch.cat([o1, o2]), ro, "out (split)")
    rs, rz = O.segment_state(k, v)
    assert_close(s2, rs, "S", rel=1e-4); assert_close(z2, rz, "z", rel=1e-4)
    if (K, d) == (256, 128):      # the reverse-state total needs a second state in shared memory, which does not fit here
        with pytest.raises(ValueError, match="two of them"):
            ops.causal_bwd_q(c(q[cut:]), c(k[cut:]), c(v[cut:]), c(g[cut:]), s, z, True)
        return
    gq2, ds, dz, ws2 = ops.causal_bwd_q(c(q[cut:]), c(k[cut:]), c(v[cut:]), c(g[cut:]), s, z, True)
    gk2, gv2 = ops.causal_bwd_kv(c(q[cut:]), c(k[cut:]), c(v[cut:]), c(g[cut:]), None, None, ws2)
    gq1, gk1, gv1 = ops.causal_bwd(c(q[:cut]), c(k[:cut]), c(v[:cut]), c(g[:cut]), None, None, ds, dz)
    assert_close(torch.cat([gq1, gq2]), rq, "gq (split)"); assert_close(torch.cat([gk1, gk2]), rk, "gk (split)")
    assert_close(torch.cat([gv1, gv2]), rv, "gv (split)")


def test_cross_attention_other_geometry(dev):
    Tq, Ts, B, H, K, d = 70, 45, 2, 3, 64, 32
    q, _, _, _ = generic_feats(Tq, B * H, K, d, seed=1)
    _, k, v, _ = generic_feats(Ts, B * H, K, d, seed=2)
    pq, pk, v = q.view(Tq, B, H, K), k.view(Ts, B, H, K), v.view(Ts, B, H, d)
    g = h16(torch.randn(Tq, B, H, d, generator=torch.Generator().manual_seed(3)))
    pad = torch.arange(Ts)[None] >= torch.tensor([Ts, 20])[:, None]
    attn, s, z, gq, gk, gv = run_cross(dev, pq, pk, v, g, pad)
    rs, rz = O.cross_state(pk, v, pad)
    assert_close(s, rs, "s", rel=1e-4); assert_close(z, rz, "z", rel=1e-4)
    assert_close(attn, O.cross_query(pq, rs, rz), "attn")
    rq, rk, rv = O.cross_backward(pq, pk, v, g, pad)
    assert_close(gq, rq, "g_phi_q"); assert_close(gk, rk, "g_phi_k"); assert_close(gv, rv, "g_v")
    assert (gk.cpu()[pad.T] == 0).all() and (gv.cpu()[pad.T] == 0).all()


def test_module_with_another_head_dim(dev):
    """CausalAttention(head_dim=32, proj_dim=32) end to end (feature map, causal kernel, decode) against its own
    incremental form."""
    from rfa_b200 import CausalAttention
    torch.manual_seed(0)
    mod = CausalAttention(embed_dim=64, num_heads=2, head_dim=32, proj_dim=32, tau=1.0).to(dev)
    w = torch.from_numpy(O.draw_matrices("orf", 2, 32, 32, 9)).float().to(dev)
    x = torch.randn(6, 2, 64, device=dev)
    y = mod(x, w)
    st = {}
    ys = torch.cat([mod(x[i:i + 1], w, saved_state=st) for i in range(6)])
    assert_close(ys, y.detach().float().cpu(), "incremental vs full", rel=4e-3)
    y.sum().backward()
    assert all(p.grad is not None and torch.isfinite(p.grad).all() for p in mod.parameters())


def test_causal_unclamped_large_denominators(dev):
    """Positive features so that q.z >> 1 everywhere except the first tokens."""
    gen = torch.Generator().manual_seed(4)
    T, BH = 300, 2
    q = h16(torch.rand(T, BH, 128, generator=gen) * 0.2)
    k = h16(torch.rand(T, BH, 128, generator=gen) * 0.2)
    v = h16(torch.randn(T, BH, 64, generator=gen)); g = h16(torch.randn(T, BH, 64, generator=gen))
    out, gq, gk, gv = run_causal(dev, q, k, v, g)
    ro = O.causal_forward(q, k, v); rq, rk, rv = O.causal_backward(q, k, v, g)
    assert_close(out, ro, "out"); assert_close(gq, rq, "gq"); assert_close(gk, rk, "gk"); assert_close(gv, rv, "gv")


@pytest.mark.parametrize("T,BH,cut", [(200, 2, 70), (1300, 2, 1100)])
def test_causal_state_carry_in_and_out(dev, T, BH, cut):
    """Second half of a sequence run with (S,z) carried in and (dS,dz) carried back equals
    the unsplit run -- the property the sequence-sharded path relies on."""
    from rfa_b200 import ops
    q, k, v, g = feats(T, BH, seed=33)
    ro = O.causal_forward(q, k, v); rq, rk, rv = O.causal_backward(q, k, v, g)
    c = lambda t: t.half().to(dev)
    o1, s, z = ops.causal_fwd(c(q[:cut]), c(k[:cut]), c(v[:cut]), return_state=True)
    o2, s2, z2 = ops.causal_fwd(c(q[cut:]), c(k[cut:]), c(v[cut:]), s, z, return_state=True)
    assert_close(torch.cat([o1, o2]), ro, "out")
    rs, rz = O.segment_state(k, v)
    assert_close(s2, rs, "state S", rel=1e-4, mabs=1e-2); assert_close(z2, rz, "state z", rel=1e-4, mabs=1e-2)
    # backward: later shard first (no reverse carry), its dS total feeds the earlier shard
    gq2, ds, dz, ws2 = ops.causal_bwd_q(c(q[cut:]), c(k[cut:]), c(v[cut:]), c(g[cut:]), s, z, True)
    gk2, gv2 = ops.causal_bwd_kv(c(q[cut:]), c(k[cut:]), c(v[cut:]), c(g[cut:]), None, None, ws2)
    gq1, gk1, gv1 = ops.causal_bwd(c(q[:cut]), c(k[:cut]), c(v[:cut]), c(g[:cut]), None, None, ds, dz)
    assert_close(torch.cat([gq1, gq2]), rq, "gq"); assert_close(torch.cat([gk1, gk2]), rk, "gk")
    assert_close(torch.cat([gv1, gv2]), rv, "gv")


def test_rfa_autograd_function_and_rfa_cuda_shim(dev):
    import rfa_b200
    rfa_b200.install_aliases()
    import rfa_cuda
    from random_feature_attention.rfa import RFA
    g = golden("causal_features")
    q, k, v = (g[n].half().to(dev).requires_grad_(True) for n in ("q", "k", "v"))
    out = RFA.apply(q, k, v)
    (out.float() * g["g"].to(dev)).sum().backward()
    assert_close(out, g["attn"], "attn"); assert_close(q.grad, g["gq"], "gq")
    assert_close(k.grad, g["gk"], "gk"); assert_close(v.grad, g["gv"], "gv")
    assert_close(rfa_cuda.forward(q.detach(), k.detach(), v.detach()), g["attn"], "rfa_cuda.forward")
    assert_close(RFA.forward_torch(q.detach().float(), k.detach().float(), v.detach().float()), g["attn"],
                 "forward_torch twin", rel=1e-5, mabs=1e-5)
    with pytest.raises(TypeError):
        rfa_cuda.forward(q.detach().float(), k.detach().float(), v.detach().float())


def test_outputs_fully_written(dev):
    """Poison the caching allocator's blocks with NaN first: every output element must be
    written by the kernels (upstream hid this behind torch::zeros)."""
    q, k, v, g = feats(130, 3, seed=5)
    junk = [torch.full((130, 3, 128), float("nan"), dtype=torch.half, device=dev) for _ in range(6)]
    del junk
    out, gq, gk, gv = run_causal(dev, q, k, v, g)
    for t in (out, gq, gk, gv):
        assert torch.isfinite(t).all()


def test_host_pipeline_matches_direct_calls(dev):
    """Upload / compute / download on three streams over two buffer sets: every step's results equal the direct calls."""
    from rfa_b200 import ops
    from rfa_b200.host_pipeline import HostPipelinedRFA
    pipe = HostPipelinedRFA(dev)
    steps = []
    for i in range(5):
        q, k, v, g = feats(300, 3, seed=50 + i)
        hin = [t.half().pin_memory() for t in (q, k, v, g)]
        hout = [torch.empty_like(t).pin_memory() for t in (hin[2], hin[0], hin[1], hin[2])]
        pipe.step(*hin, hout)
        steps.append((hin, hout))
    pipe.join()
    torch.cuda.synchronize()
    for hin, hout in steps:
        dq, dk, dv, dg = (t.to(dev) for t in hin)
        attn, ws, has = ops.causal_fwd_saved(dq, dk, dv)           # the calls the pipeline makes per step
        ref = (attn,) + tuple(ops.causal_bwd_saved(dq, dk, dv, dg, attn, ws, has))
        for a, b in zip(hout, ref):
            assert torch.equal(a, b.cpu())


# ----------------------------------------------------------------------------- feature map
def test_feature_map_against_upstream_fixture(dev):
    from rfa_b200 import utils
    g = golden("feature_map")
    x = g["x"].half().to(dev).requires_grad_(True)
    w = g["w_eff"].to(dev).requires_grad_(True)
    phi = utils.random_project(x=x, random_matrices=w)
    assert phi.dtype == torch.half
    assert_close(phi, g["phi"], "phi", rel=1e-3, mabs=2e-4)
    (phi.float() * g["g_phi"].to(dev)).sum().backward()
    assert_close(x.grad, g["g_x"], "g_x"); assert_close(w.grad, g["g_w"], "g_w", rel=2e-3, mabs=5e-2)
    x32 = g["x"].to(dev)
    assert_close(utils.random_project(x=x32, random_matrices=g["w"].to(dev)), g["phi_plain"], "phi fp32", rel=1e-5, mabs=1e-6)


@pytest.mark.parametrize("dtype,d", [(torch.half, 64), (torch.float32, 64), (torch.half, 32)])
def test_feature_map_with_padding_mask(dev, dtype, d):
    """random_project(key_padding_mask=...) == random_project followed by upstream's masked_fill (forward and gradients),
    on the tensor-core kernel (fp16, 64) and the generic ones."""
    from rfa_b200 import utils
    gen = torch.Generator().manual_seed(d)
    T, B, H = 150, 3, 2
    x = h16(torch.randn(T, B, H, d, generator=gen))
    w = torch.randn(H, d, d, generator=gen)
    gp = h16(torch.randn(T, B, H, 2 * d, generator=gen))
    pad = torch.arange(T)[None] >= torch.tensor([T, 100, 1])[:, None]              # [B, T]
    xd = x.to(dev, dtype).requires_grad_(True); wd = w.to(dev).requires_grad_(True)
    phi = utils.random_project(x=xd, random_matrices=wd, key_padding_mask=pad.to(dev))
    (phi.float() * gp.to(dev)).sum().backward()
    xr = x.clone().requires_grad_(True); wr = w.clone().requires_grad_(True)
    ref = O.random_project(xr, wr).masked_fill(pad.t()[:, :, None, None], 0.0)
    (ref * gp).sum().backward()
    tol = dict(rel=2e-3, mabs=2e-4) if dtype == torch.half else dict(rel=1e-5, mabs=1e-6)
    assert_close(phi, ref.detach(), "phi", **tol)
    assert (phi.float().cpu()[pad.t()] == 0).all() and (xd.grad.float().cpu()[pad.t()] == 0).all()
    assert_close(xd.grad, xr.grad, "g_x", rel=2e-3 if dtype == torch.half else 1e-4, mabs=1e-2)
    assert_close(wd.grad, wr.grad, "g_w", rel=2e-3 if dtype == torch.half else 1e-4, mabs=5e-2)


@pytest.mark.parametrize("rows,H,d,D", [(1, 1, 64, 64), (77, 3, 64, 64), (130, 2, 32, 48), (65, 2, 128, 128), (9, 5, 16, 8)])
def test_feature_map_shapes_fp32(dev, rows, H, d, D):
    from rfa_b200 import ops
    gen = torch.Generator().manual_seed(rows)
    x = torch.randn(rows, H, d, generator=gen) * 2
    x[0, 0] = 0                                             # zero vector: norm 0
    w = torch.randn(H, D, d, generator=gen)
    gp = torch.randn(rows, H, 2 * D, generator=gen)
    phi = ops.feature_map_fwd(x.to(dev), w.to(dev), 0.1)
    gx, gw = ops.feature_map_bwd(x.to(dev), w.to(dev), gp.to(dev), 0.1, True)
    assert_close(phi, O.random_project(x, w), "phi", rel=1e-5, mabs=1e-6)
    rx, rw = O.random_project_backward(x, w, gp)
    assert_close(gx, rx, "g_x", rel=1e-4, mabs=1e-4); assert_close(gw, rw, "g_w", rel=1e-4, mabs=1e-3)


@pytest.mark.parametrize("rows,H", [(1, 1), (130, 3), (1000, 2), (4096, 16)])
def test_feature_map_fp16_tensor_core_path(dev, rows, H):
    """fp16 rows with head_dim = proj_dim = 64 take the tcgen05 kernels (forward and backward); several row tiles per
    CTA, a ragged last tile, a zero vector, and g_W accumulated over all tiles and CTAs of a head."""
    from rfa_b200 import ops
    gen = torch.Generator().manual_seed(rows + H)
    x = h16(torch.randn(rows, H, 64, generator=gen) * 2)
    x[0, 0] = 0
    w = torch.randn(H, 64, 64, generator=gen)
    gp = h16(torch.randn(rows, H, 128, generator=gen))
    phi = ops.feature_map_fwd(x.to(dev).half(), w.to(dev), 0.1)
    gx, gw = ops.feature_map_bwd(x.to(dev).half(), w.to(dev), gp.to(dev).half(), 0.1, True)
    assert phi.dtype == torch.half and gx.dtype == torch.half
    assert_close(phi, O.random_project(x, w), "phi", rel=2e-3, mabs=2e-4)
    rx, rw = O.random_project_backward(x, w, gp)
    assert_close(gx, rx, "g_x"); assert_close(gw, rw, "g_w", rel=2e-3, mabs=5e-2)
    gx2, none = ops.feature_map_bwd(x.to(dev).half(), w.to(dev), gp.to(dev).half(), 0.1, False)
    assert none is None and torch.equal(gx2, gx)


def test_state_total_matches_single_cta_reduction(dev):
    """Partials over runs of tokens (many CTAs per sequence) summed == the one-CTA-per-sequence reduction == oracle."""
    from rfa_b200 import ops
    for T, BH in [(5000, 2), (300, 3), (1, 1)]:
        q, k, v, g = feats(T, BH, seed=T + BH)
        kd, vd = k.to(dev).half(), v.to(dev).half()
        s1, z1 = ops.state_total(kd, vd)
        s0, z0 = ops.cross_state_fwd(kd.view(T, 1, BH, -1), vd.view(T, 1, BH, -1), None)
        rs, rz = O.segment_state(k, v)
        assert_close(s1, rs, "S", rel=1e-4, mabs=1e-3); assert_close(z1, rz, "z", rel=1e-4, mabs=1e-3)
        assert_close(s1, s0.view(BH, 128, 64).cpu(), "S vs single", rel=1e-5, mabs=1e-3)
        assert_close(z1, z0.view(BH, 128).cpu(), "z vs single", rel=1e-5, mabs=1e-3)


def test_effective_matrices_for_all_layers_in_one_launch(dev):
    """Device-resident bank, deterministic picks, sigma / tau applied by the gather kernel: equals upstream's
    sample_random_matrices + build_random_matrices per layer (restated by the oracle), with the gradient reaching sigma."""
    from rfa_b200 import utils
    L, H, D, d = 3, 4, 64, 64
    bank = torch.from_numpy(O.draw_matrices("orf", 40, d, D, 5)).half()
    taus = [0.9, 1.0, 1.3]
    sigmas = [(torch.rand(H, 1, d) + 0.5).to(dev).requires_grad_(True) for _ in range(L)]
    gen = lambda: torch.Generator().manual_seed(11)
    eff = utils.sample_effective_matrices(num_layers=L, num_heads=H, random_matrices=bank.to(dev), taus=taus, sigmas=sigmas,
                                          generator=gen())
    layers = utils.sample_random_matrices(num_layers=L, num_heads=H, random_matrices=bank, generator=gen())
    for l in range(L):
        want = O.build_random_matrices(layers[l].float(), taus[l], sigmas[l].detach().cpu(), True)
        assert_close(eff[l], want, f"layer {l}", rel=1e-6, mabs=1e-6)
    up = torch.randn(L, H, D, d, device=dev)
    (eff * up).sum().backward()
    for l in range(L):
        want = (up[l].cpu() * layers[l].float() / taus[l]).sum(dim=1, keepdim=True)
        assert_close(sigmas[l].grad, want, f"grad sigma {l}", rel=1e-5, mabs=1e-4)
    ev = utils.sample_effective_matrices(num_layers=2, num_heads=H, random_matrices=bank.to(dev), taus=[1.0, 2.0], is_training=False)
    assert_close(ev[1], bank[:H].float() / 2.0, "evaluation: the first H matrices", rel=1e-6, mabs=1e-6)


# ----------------------------------------------------------------------------- decode
def test_decode_against_upstream_fixture(dev):
    from rfa_b200.causal_attention import incremental_rfa
    g = golden("incremental")
    pq, pk, v = (g[n].half().to(dev) for n in ("phi_q", "phi_k", "v"))
    a1, s, z = incremental_rfa(phi_q=pq[:6], phi_k=pk[:6], v=v[:6])               # multi-token: causal kernel + carry
    assert s.dtype == torch.float32
    assert_close(a1, g["attn_a"], "attn_a"); assert_close(z, g["z_a"], "z_a", rel=1e-4)
    outs = []
    for i in range(6, 9):                                                         # one token at a time: decode kernel
        a, s, z = incremental_rfa(phi_q=pq[i:i + 1], phi_k=pk[i:i + 1], v=v[i:i + 1], s=s, z=z)
        outs.append(a)
    assert_close(torch.cat(outs), g["attn_b"], "attn_b")
    assert_close(s, g["s_b"], "s_b", rel=1e-4); assert_close(z, g["z_b"], "z_b", rel=1e-4)


def test_incremental_rfa_is_differentiable_and_reorderable(dev):
    """With autograd recording, incremental_rfa differentiates through outputs AND the carried state (as upstream's plain
    PyTorch loop does): two calls in a row against the oracle's gradients of the whole run; then the beam reorder."""
    from rfa_b200.causal_attention import CausalAttention, incremental_rfa
    T, B, H, cut = 40, 2, 3, 25
    q, k, v, g = feats(T, B * H, seed=12)
    leaves = [t.view(T, B, H, -1).half().to(dev).requires_grad_(True) for t in (q, k, v)]
    pq, pk, pv = leaves
    a1, s, z = incremental_rfa(phi_q=pq[:cut], phi_k=pk[:cut], v=pv[:cut])
    a2, s2, z2 = incremental_rfa(phi_q=pq[cut:], phi_k=pk[cut:], v=pv[cut:], s=s, z=z)
    attn = torch.cat([a1, a2])
    assert_close(attn.view(T, B * H, 64), O.causal_forward(q, k, v), "attn")
    (attn.view(T, B * H, 64).float() * g.to(dev)).sum().backward()
    rq, rk, rv = O.causal_backward(q, k, v, g)
    assert_close(pq.grad.view(T, B * H, 128), rq, "gq"); assert_close(pk.grad.view(T, B * H, 128), rk, "gk")
    assert_close(pv.grad.view(T, B * H, 64), rv, "gv")
    st = {"prev_s": s2.detach(), "prev_z": z2.detach()}
    CausalAttention.reorder_incremental_state(st, torch.tensor([1, 1, 0]))
    assert st["prev_s"].shape[0] == 3 and torch.equal(st["prev_s"][0], s2[1]) and torch.equal(st["prev_z"][2], z2[0])


@pytest.mark.parametrize("state_dtype,in_dtype", [(torch.float32, torch.float16), (torch.float16, torch.float16), (torch.float32, torch.float32)])
def test_decode_steps_vs_oracle(dev, state_dtype, in_dtype):
    from rfa_b200 import ops
    gen = torch.Generator().manual_seed(3)
    B, H, steps = 3, 4, 5
    w = torch.from_numpy(O.draw_matrices("orf", H, 64, 64, 1)).float()
    s = torch.zeros(B, H, 128, 64); z = torch.zeros(B, H, 128)
    sd, zd = s.to(dev, state_dtype), z.to(dev, state_dtype)
    sf, zf = s.to(dev, state_dtype), z.to(dev, state_dtype)
    for i in range(steps):
        q, k, v = (h16(torch.randn(B, H, 64, generator=gen)) for _ in range(3))
        pq, pk = h16(O.random_project(q, w)), h16(O.random_project(k, w))
        ref, s, z = O.incremental_rfa(pq[None], pk[None], v[None], s, z)
        out = ops.decode_step(pq.to(dev, in_dtype), pk.to(dev, in_dtype), v.to(dev, in_dtype), sd, zd)
        outf = ops.decode_step_fused(q.to(dev, in_dtype), k.to(dev, in_dtype), v.to(dev, in_dtype), w.to(dev), 0.1, sf, zf)
        assert_close(out.reshape(1, B, -1), ref, f"step {i}")
        assert_close(outf.reshape(1, B, -1), ref, f"fused step {i}")
    tol = 1e-4 if state_dtype == torch.float32 else 2e-3
    assert_close(sd, s, "S", rel=tol); assert_close(zd, z, "z", rel=tol)
    assert_close(sf, s, "S fused", rel=2e-3); assert_close(zf, z, "z fused", rel=2e-3)


# ----------------------------------------------------------------------------- cross
def run_cross(dev, pq, pk, v, g, pad):
    from rfa_b200.cross_attention import cross_rfa_query, cross_rfa_state
    pq_, pk_, v_ = (t.half().to(dev).requires_grad_(True) for t in (pq, pk, v))
    s, z = cross_rfa_state(pk_, v_, None if pad is None else pad.to(dev))
    attn = cross_rfa_query(pq_, s, z)
    (attn.float() * g.to(dev)).sum().backward()
    return attn, s, z, pq_.grad, pk_.grad, v_.grad


@pytest.mark.parametrize("name", ["cross", "cross_signed"])
def test_cross_against_upstream_fixtures(dev, name):
    g = golden(name)
    pad = g.get("pad")
    attn, s, z, gq, gk, gv = run_cross(dev, g["phi_q"], g["phi_k"], g["v"], g["g"], pad)
    assert_close(attn, g["attn"], "attn")
    if "s" in g:
        assert_close(s, g["s"], "s", rel=1e-4); assert_close(z, g["z"], "z", rel=1e-4)
    assert_close(gq, g["g_phi_q"], "g_phi_q"); assert_close(gk, g["g_phi_k"], "g_phi_k"); assert_close(gv, g["g_v"], "g_v")
    if pad is not None:
        assert (gk.cpu()[pad.T] == 0).all() and (gv.cpu()[pad.T] == 0).all()


@pytest.mark.parametrize("Tq,Ts,B,H", [(1, 1, 1, 1), (70, 129, 2, 3), (200, 64, 3, 2)])
def test_cross_vs_oracle_ragged(dev, Tq, Ts, B, H):
    gen = torch.Generator().manual_seed(Tq + Ts)
    q, _, _, _ = feats(Tq, B * H, seed=Tq)
    _, k, v, _ = feats(Ts, B * H, seed=Ts + 1)
    pq, pk, v = q.view(Tq, B, H, 128), k.view(Ts, B, H, 128), v.view(Ts, B, H, 64)
    g = h16(torch.randn(Tq, B, H, 64, generator=gen))
    lens = torch.randint(1, Ts + 1, (B,), generator=gen)
    lens[0] = Ts
    pad = torch.arange(Ts)[None] >= lens[:, None]
    attn, s, z, gq, gk, gv = run_cross(dev, pq, pk, v, g, pad)
    rs, rz = O.cross_state(pk, v, pad)
    assert_close(s, rs, "s", rel=1e-4); assert_close(z, rz, "z", rel=1e-4)
    assert_close(attn, O.cross_query(pq, rs, rz), "attn")
    rq, rk, rv = O.cross_backward(pq, pk, v, g, pad)
    assert_close(gq, rq, "g_phi_q"); assert_close(gk, rk, "g_phi_k"); assert_close(gv, rv, "g_v")


def test_cross_decode_step_all_layers_in_one_launch(dev):
    from rfa_b200 import ops
    L, B, H, K, d = 3, 2, 4, 128, 64
    gen = torch.Generator().manual_seed(8)
    states, refs = [], []
    pq = h16(torch.rand(L, B, H, K, generator=gen) * 0.3 - 0.1)
    for l in range(L):
        s = torch.randn(B, H, K, d, generator=gen) * (1.0 if l else 40.0)          # layer 0: denominators beyond the clamp
        z = torch.randn(B, H, K, generator=gen) * (1.0 if l else 40.0)
        states.append((s.to(dev), z.to(dev)))
        refs.append(O.cross_query(pq[l][None], s, z))
    out = ops.cross_decode_step(pq.half().to(dev), ops.CrossDecodeStates(states))
    assert_close(out.view(L, 1, B, H * d), torch.stack(refs).view(L, 1, B, H * d), "cross decode step")


# ----------------------------------------------------------------------------- modules
def test_modules_against_upstream_fixture(dev):
    from rfa_b200 import CausalAttention, CrossAttention
    from rfa_b200.cross_attention import CrossAttentionProjectLayer
    g = golden("modules")
    sub = lambda pre: {k[len(pre):]: v for k, v in g.items() if k.startswith(pre)}
    w = g["w"].to(dev)
    mod = CausalAttention(embed_dim=128, num_heads=2, head_dim=64, proj_dim=64, tau=0.9).to(dev)
    mod.load_state_dict(sub("causal."))
    y = mod(g["x"].to(dev), w, key_padding_mask=g["kpm"].to(dev))
    assert_close(y, g["y"], "CausalAttention", rel=4e-3)
    st = {}
    ys = torch.cat([mod(g["x"][i:i + 1].to(dev), w, saved_state=st) for i in range(4)])
    assert_close(ys, g["y_inc"], "incremental", rel=4e-3)
    assert_close(st["prev_s"], g["prev_s"], "prev_s", rel=2e-3); assert_close(st["prev_z"], g["prev_z"], "prev_z", rel=2e-3)
    layer = CrossAttentionProjectLayer(embed_dim=128, num_heads=2, head_dim=64, proj_dim=64, tau=1.1).to(dev)
    layer.load_state_dict(sub("xlayer."))
    dec = CrossAttention(embed_dim=128, num_heads=2, head_dim=64, proj_dim=64, tau=1.1).to(dev)
    dec.load_state_dict(sub("xdec."))
    state = layer(encoder_output=g["enc"].to(dev), random_matrices=w, mask=g["emask"].to(dev))
    assert_close(state.s, g["xs"], "cross s", rel=2e-3); assert_close(state.z, g["xz"], "cross z", rel=2e-3)
    assert_close(dec(g["query"].to(dev), state), g["yq"], "CrossAttention", rel=4e-3)
    # gradients reach every parameter through the kernels
    mod.zero_grad()
    mod(g["x"].to(dev), w).sum().backward()
    assert all(p.grad is not None and torch.isfinite(p.grad).all() for p in mod.parameters())


# ----------------------------------------------------------------------------- argument checking
def test_bad_arguments_are_rejected_without_launching(dev):
    from rfa_b200 import ops
    q = torch.zeros(8, 2, 100, dtype=torch.half, device=dev)
    v = torch.zeros(8, 2, 64, dtype=torch.half, device=dev)
    with pytest.raises(ValueError, match="multiples of 8"):
        ops.causal_fwd(q, q, v)
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        ops.causal_fwd(q.cpu(), q.cpu(), v.cpu())
    q = torch.zeros(0, 2, 128, dtype=torch.half, device=dev)
    assert ops.causal_fwd(q, q, torch.zeros(0, 2, 64, dtype=torch.half, device=dev)).shape == (0, 2, 64)


def test_stream_probe_runs_and_checks_its_arguments(dev):
    """The measurement aid behind bench.py's tile-stream ceiling: streams tiles with no arithmetic."""
    from rfa_b200 import _lib
    lib = _lib.load()
    src = torch.zeros(300, 3, 64 * 4, dtype=torch.half, device=dev)
    dst = torch.zeros(300, 3, 128, dtype=torch.half, device=dev)
    st = torch.cuda.current_stream().cuda_stream
    assert lib.rfa_stream_probe(src.data_ptr(), dst.data_ptr(), 300, 3, 4, 1, st) == 0
    assert lib.rfa_stream_probe(src.data_ptr(), None, 300, 3, 4, 0, st) == 0
    torch.cuda.synchronize()
    assert lib.rfa_stream_probe(src.data_ptr(), None, 300, 3, 4, 1, st) == -1       # a store needs somewhere to go
    assert lib.rfa_stream_probe(src.data_ptr(), dst.data_ptr(), 300, 3, 7, 0, st) == -1


def test_causal_long_sequence_late_tokens(dev):
    """T = 32768 on real features: denominators reach ~7500, g/den ~1e-4 (fp16 subnormal range).  The
    late tokens are where rounding would show first; they are held to the same gate."""
    T, BH = 32768, 1
    q, k, v, g = feats(T, BH, seed=77)
    out, gq, gk, gv = run_causal(dev, q, k, v, g)
    ro = O.causal_forward(q.double(), k.double(), v.double(), block=256)
    rq, rk, rv = O.causal_backward(q.double(), k.double(), v.double(), g.double(), block=256)
    tail = slice(T - T // 8, T)
    for name, a, b in (("out", out, ro), ("gq", gq, rq), ("gk", gk, rk), ("gv", gv, rv)):
        assert_close(a, b, name)
        assert_close(a[tail], b[tail], name + " (last eighth)")


@pytest.mark.parametrize("rows,B,H,masked", [(1, 1, 1, False), (300, 2, 3, True), (2048, 8, 16, True)])
def test_feature_map_pair_equals_two_single_launches(dev, rows, B, H, masked):
    """rfa_feature_map_fwd_pair / _bwd_pair (q and k of one layer in one launch) against the single-array entry points."""
    from rfa_b200 import ops
    gen = torch.Generator().manual_seed(rows + H)
    w = torch.from_numpy(O.draw_matrices("orf", H, 64, 64, 3)).float().to(dev)
    xa, xb = (torch.randn(rows, B, H, 64, generator=gen).half().to(dev) for _ in range(2))
    ga, gb = (torch.randn(rows, B, H, 128, generator=gen).half().to(dev) for _ in range(2))
    mask = (torch.rand(rows, B, generator=gen) < 0.2).to(dev) if masked else None
    pa, pb = ops.feature_map_fwd_pair(xa, xb, w, 0.1, None, mask)
    assert torch.equal(pa, ops.feature_map_fwd(xa, w, 0.1))
    assert torch.equal(pb, ops.feature_map_fwd(xb, w, 0.1, row_mask=mask))
    gxa, gxb, gw = ops.feature_map_bwd_pair(xa, xb, w, ga, gb, 0.1, True, None, mask)
    sa, wa = ops.feature_map_bwd(xa, w, ga, 0.1, True)
    sb, wb = ops.feature_map_bwd(xb, w, gb, 0.1, True, row_mask=mask)
    assert torch.equal(gxa, sa) and torch.equal(gxb, sb)
    assert_close(gw, wa + wb, "g_w of the pair", rel=1e-5, mabs=1e-2)
    # against the oracle as well (float64 reference of the analytic gradient)
    want_a, want_wa = O.random_project_backward(xa.float().cpu(), w.cpu(), ga.float().cpu(), 0.1)
    assert_close(gxa, want_a, "g_x (pair, first array)")


@pytest.mark.parametrize("T,BH,status", [(896, 2, 0), (900, 2, 0), (1000, 37, 0), (1023, 2, 0), (1024, 2, -4), (1024, 70, -4), (1024, 75, 0)])
def test_forward_without_a_workspace(dev, T, BH, status):
    """Below 1024 tokens, or with less than two segments to a wave, none is needed, and one that is there is not used: a forward alone
    runs sequences whole.  Above that one is needed, which is said before anything is launched."""
    import ctypes
    from rfa_b200 import _lib, ops
    q, k, v, _ = (t.half().to(dev) for t in generic_feats(T, BH, 128, 64, 3))
    bare = torch.empty_like(v)
    assert _lib.load().rfa_causal_fwd(*(t.data_ptr() for t in (q, k, v, bare)), None, None, None, None, None, ctypes.c_size_t(0),
                                      T, BH, 128, 64, _lib.stream_of(q)) == status
    if status == 0:
        assert torch.equal(bare, ops.causal_fwd(q, k, v))
        assert_close(bare, O.causal_forward(*(t.float().cpu() for t in (q, k, v))), "out without a workspace")


def test_feature_map_is_bit_stable(dev):
    """Repeated launches on the same inputs: the rows' norms must be read before the stage is refilled (test_gpu_repeat.py launches
    each kernel more often, on tiles of different magnitude)."""
    from rfa_b200 import ops
    gen = torch.Generator().manual_seed(0)
    w = torch.randn(16, 64, 64, generator=gen).to(dev)
    x = torch.randn(1024, 16, 16, 64, generator=gen).half().to(dev)
    g = torch.randn(1024, 16, 16, 128, generator=gen).half().to(dev)
    first, grad = ops.feature_map_fwd(x, w, 0.1), ops.feature_map_bwd(x, w, g, 0.1, True)[0]
    for _ in range(60):
        pa, pb = ops.feature_map_fwd_pair(x, x, w, 0.1)
        single, gx = ops.feature_map_fwd(x, w, 0.1), ops.feature_map_bwd(x, w, g, 0.1, True)[0]
        assert torch.equal(pa, first) and torch.equal(pb, first) and torch.equal(single, first) and torch.equal(gx, grad)
