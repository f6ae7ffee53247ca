"""Projections of a few rows (``rfa_linear_rows``) and the layer's one-token call built on them."""
import ctypes as C

import pytest
import torch

from rfa_b200 import CausalAttention, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 8, 9, 16, 17, 32, 33, 64, 65, 128])
@pytest.mark.parametrize("inner,out", [(1024, 1024), (512, 512), (8, 8), (40, 24), (264, 1000)])
def test_linear_rows(dev, n, inner, out):
    """Every tile shape (1..8, ..16, ..32, more tokens) with whole and ragged tiles of tokens, rows of W and inner index, against fp64:
    the result's rounding to fp16 (2^-11) and fp32 sums of up to 1024 terms (2^-24 sqrt(1024) of their 2-norm)."""
    gen = torch.Generator().manual_seed(n + inner)
    x = torch.randn(n, inner, generator=gen).half()
    ws = [torch.randn(out, inner, generator=gen).half() for _ in range(3)]
    bs = [torch.randn(out, generator=gen).half(), None, torch.randn(out, generator=gen).half()]
    xd, wd, bd = x.to(dev), [w.to(dev) for w in ws], [None if b is None else b.to(dev) for b in bs]
    ys = [torch.full((n, out), float("nan"), device=dev, dtype=torch.float16) for _ in range(3)]
    ptrs = lambda ts: (C.c_void_p * 3)(*[None if t is None else t.data_ptr() for t in ts])
    rm, sigma = torch.randn(3, 16, 24, generator=gen).half(), torch.randn(3, 24, generator=gen).half()
    rmd, sd, eff = rm.to(dev), sigma.to(dev), torch.full((3, 16, 24), float("nan"), device=dev)
    status = _lib.load().rfa_linear_rows(xd.data_ptr(), ptrs(wd), ptrs(bd), ptrs(ys), 3, n, inner, out, rmd.data_ptr(), sd.data_ptr(), 0.5,
                                         eff.data_ptr(), 3, 16, 24, torch.cuda.current_stream().cuda_stream)
    assert status == 0, _lib.last_error()
    for w, b, y in zip(ws, bs, ys):
        want = x.double() @ w.double().t() + (0 if b is None else b.double())
        scale = (x.double().norm(dim=1)[:, None] * w.double().norm(dim=1)[None] + 4) * 2.0 ** -19
        assert ((y.cpu().double() - want).abs() <= want.abs() * 2.0 ** -11 + scale).all()
    assert torch.equal(eff.cpu(), ((sigma[:, None] * rm) / 2).float())


@pytest.mark.parametrize("batch", [1, 33, 128, 129])
@pytest.mark.parametrize("tau,reparam", [(1.0, True), (0.7, True), (1.0, False), (3.0, False)])
def test_layer_call_against_its_modules(dev, batch, tau, reparam):
    """The three-launch call and the same layer module by module (a hook sends it there): outputs and states to the rounding of q, k, v and
    the output to fp16 (2^-11 each; the GEMMs' sums round differently), 129 rows being beyond the launch's range."""
    torch.manual_seed(batch)
    layer = CausalAttention(embed_dim=256, num_heads=4, head_dim=64, proj_dim=64, tau=tau, reparam_proj=reparam).to(dev).half()
    w = torch.randn(4, 64, 64, device=dev).half()
    one, two = {}, {}
    calls = []
    with torch.no_grad():
        for _ in range(3):
            x = torch.randn(1, batch, 256, device=dev).half()
            a = layer(x, w, saved_state=one)
            hook = layer.v_proj.register_forward_hook(lambda *args: calls.append(1))
            b = layer(x, w, saved_state=two)
            hook.remove()
            assert ((a - b).float().norm() / b.float().norm()).item() < 3e-3
    assert len(calls) == 3
    for key in ("prev_s", "prev_z"):
        assert ((one[key] - two[key]).norm() / two[key].norm()).item() < 2e-3


def test_layer_call_takes_what_it_took(dev):
    """Forms the launch does not take go module by module with the old result or refusal: states of another layout, a
    broadcast matrix, autocast, an inner module of another class."""
    torch.manual_seed(0)
    layer = CausalAttention(embed_dim=128, num_heads=2, head_dim=64, proj_dim=64).to(dev).half()
    w, x = torch.randn(2, 64, 64, device=dev).half(), torch.randn(1, 5, 128, device=dev).half()
    rel = lambda a, b: ((a - b).float().norm() / b.float().norm()).item()

    class Doubled(torch.nn.Linear):
        def forward(self, t):
            return 2 * super().forward(t)
    with torch.no_grad():
        base = layer(x, w, saved_state={})
        assert rel(layer(x, w[:1].expand(2, 64, 64), saved_state={}), layer(x, w[:1].repeat(2, 1, 1), saved_state={})) < 3e-3
        s = torch.zeros(5, 2, 64, 128, device=dev).transpose(-1, -2)
        with pytest.raises(ValueError, match="contiguous"):
            layer(x, w, saved_state=dict(prev_s=s, prev_z=torch.zeros(5, 2, 128, device=dev)))
        with torch.autocast("cuda", dtype=torch.float16):
            assert rel(layer(x, w, saved_state={}), base) < 3e-3
        out_proj = layer.out_proj
        layer.out_proj = Doubled(128, 128).to(dev).half()
        layer.out_proj.load_state_dict(out_proj.state_dict())
        assert rel(layer(x, w, saved_state={}), 2 * base) < 3e-3


@pytest.mark.parametrize("heads,batch,eager,captured", [(16, 128, True, True), (32, 32, True, True), (32, 33, True, False), (40, 48, True, False),
                                                        (40, 49, False, False), (64, 16, True, True), (64, 18, True, False), (64, 19, False, False)])
def test_the_largest_batch_of_a_layer_call(dev, monkeypatch, heads, batch, eager, captured):
    """Which batches the launch takes depends on the width, and in a CUDA graph, where the host does not count, on less of it; either way the result is the
    layer's."""
    from rfa_b200 import ops
    torch.manual_seed(heads)
    E = 64 * heads
    layer = CausalAttention(embed_dim=E, num_heads=heads, head_dim=64, proj_dim=64).to(dev).half().requires_grad_(False)
    w, x = torch.randn(heads, 64, 64, device=dev).half(), torch.randn(1, batch, E, device=dev).half()
    took, decode = [], ops.layer_decode

    def seen(*args):
        y = decode(*args)
        took.append(y is not None)
        return y
    monkeypatch.setattr(ops, "layer_decode", seen)
    state = lambda: dict(prev_s=torch.zeros(batch, heads, 128, 64, device=dev), prev_z=torch.zeros(batch, heads, 128, device=dev))
    hook = layer.v_proj.register_forward_hook(lambda *args: None)
    want = layer(x, w, saved_state=state())
    hook.remove()
    assert not took
    got, held = layer(x, w, saved_state=state()), state()
    assert took == [eager]
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        replayed = layer(x, w, saved_state=held)
    assert took == [eager, captured]
    graph.replay()
    for y in (got, replayed):
        assert ((y - want).float().norm() / want.float().norm()).item() < 3e-3
