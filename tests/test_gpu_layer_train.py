"""A layer's training step on native nodes (csrc/layer_train.cu, ``ops.layer_train``): its kernels against fp64, the whole against the
step that goes module by module."""
import ctypes as C

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from rfa_b200 import CausalAttention, _lib, ops

pytestmark = pytest.mark.gpu


class Seen(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


def pointers(tensors):
    return (C.c_void_p * len(tensors))(*[t.data_ptr() for t in tensors])


@pytest.mark.parametrize("rows", [0, 1, 8, 63, 65, 513, 4099])
@pytest.mark.parametrize("count,cols", [(1, 8), (2, 40), (3, 512), (3, 1000)])
def test_column_sums(dev, count, rows, cols):
    """fp32 sums rounded once: 2^-11 of the result and a little of the terms' magnitudes."""
    gen = torch.Generator(dev).manual_seed(rows)
    g = [torch.randn(rows, cols, generator=gen, device=dev).half() for _ in range(count)]
    if rows:
        g[0][rows // 2, 3] = float("inf")
    out = [torch.full((cols,), 7.0, device=dev).half() for _ in range(count)]
    assert _lib.load().rfa_column_sums(C.addressof(pointers(g)), C.addressof(pointers(out)), count, rows, cols, torch.cuda.current_stream().cuda_stream) == 0
    for a, b in zip(out, g):
        want, size = b.double().sum(0), b.double().abs().sum(0)
        fine = want.isfinite()
        assert ((a.double() - want).abs()[fine] <= 2.0 ** -11 * want.abs()[fine] + 2.0 ** -20 * size[fine] + 2.0 ** -25).all()
        assert torch.equal(a.double()[~fine], want[~fine])


@pytest.mark.parametrize("H,D,d", [(1, 8, 8), (3, 64, 64), (5, 40, 24), (2, 128, 128)])
@pytest.mark.parametrize("with_sigma,tau", [(True, 1.0), (True, 0.7), (False, 2.0)])
def test_layer_matrices(dev, H, D, d, with_sigma, tau):
    gen = torch.Generator(dev).manual_seed(D)
    rm, g = torch.randn(H, D, d, generator=gen, device=dev).half(), torch.randn(H, D, d, generator=gen, device=dev)
    sigma = (1 + torch.randn(H, 1, d, generator=gen, device=dev) / 8).half() if with_sigma else None
    T, B = 37, 5
    pad, mask = torch.rand(B, T, generator=gen, device=dev) < 0.5, torch.zeros(T, B, dtype=torch.bool, device=dev)
    w, gs, gr = torch.empty(H, D, d, device=dev), torch.empty(H, 1, d, device=dev).half(), torch.empty_like(rm)
    lib, st, sp = _lib.load(), torch.cuda.current_stream().cuda_stream, sigma.data_ptr() if with_sigma else None
    assert lib.rfa_layer_matrices(rm.data_ptr(), sp, 1 / tau, w.data_ptr(), H, D, d, pad.data_ptr(), mask.data_ptr(), T, B, st) == 0
    assert torch.equal(mask, pad.t())
    want = sigma * rm if with_sigma else rm
    assert torch.equal(w, (want if tau == 1 else want / tau).float())
    assert lib.rfa_layer_matrices_bwd(g.data_ptr(), rm.data_ptr(), sp, 1 / tau, gs.data_ptr() if with_sigma else None, gr.data_ptr(), H, D, d, st) == 0
    scale = (sigma.double() if with_sigma else 1.0) / tau
    near = lambda a, b, size: ((a.double() - b).abs() <= 2.0 ** -11 * b.abs() + 2.0 ** -20 * size + 2.0 ** -25).all()
    assert near(gr, g.double() * scale, (g.double() * scale).abs())
    if with_sigma:
        terms = g.double() * rm.double() / tau
        assert near(gs, terms.sum(1, True), terms.abs().sum(1, True))


def make(dev, heads=8, head_dim=64, proj_dim=64, reparam=True, tau=1.0, seed=0):
    torch.manual_seed(seed)
    layer = CausalAttention(embed_dim=heads * head_dim, num_heads=heads, head_dim=head_dim, proj_dim=proj_dim, reparam_proj=reparam, tau=tau)
    for p in layer.parameters():
        torch.nn.init.normal_(p, 1.0 if p.dim() == 3 else 0.0, 0.1 if p.dim() == 3 else 0.05)
    return layer.to(dev).half(), torch.randn(heads, proj_dim, head_dim, device=dev).half()


def step(layer, x, rm, mask, g, context):
    layer.zero_grad(set_to_none=True)
    x = x.detach().requires_grad_(x.requires_grad)
    rm = rm.detach().requires_grad_(rm.requires_grad)
    with context:
        y = layer(x, rm, key_padding_mask=mask)
    y.backward(g)
    return y, [x.grad, rm.grad] + [p.grad for p in layer.parameters()]


CASES = {"plain": {}, "no mask": dict(mask=False), "tau": dict(tau=0.5), "no sigma": dict(reparam=False), "heads of 32": dict(head_dim=32, proj_dim=32),
         "wide": dict(heads=2, head_dim=96, proj_dim=40), "no bias": dict(drop=("q_proj", "out_proj")), "frozen": dict(freeze=("q_proj", "out_proj.bias", "k_proj.bias")),
         "input only": dict(freeze=("",)), "constant input": dict(x=False), "matrices too": dict(rm=True), "one token": dict(T=1, B=1), "strided gradient": dict(expand=True)}


@pytest.mark.parametrize("kind", CASES)
def test_same_step_as_module_by_module(dev, kind):
    """The output bit for bit; gradients, whose sums take another order and fewer roundings to fp16, within 2^-9 of each array's norm; None
    in the same places."""
    c = dict(CASES[kind])
    T, B = c.pop("T", 45), c.pop("B", 6)
    masked, drop, freeze, need_x, need_rm, expand = (c.pop("mask", True), c.pop("drop", ()), c.pop("freeze", None), c.pop("x", True), c.pop("rm", False),
                                                     c.pop("expand", False))
    layer, rm = make(dev, **c)
    for name in drop:
        getattr(layer, name).bias = None
    if freeze:
        for name, p in layer.named_parameters():
            p.requires_grad_(not any(name.startswith(f) for f in freeze))
    x = torch.randn(T, B, layer.embed_dim, device=dev).half().requires_grad_(need_x)
    rm.requires_grad_(need_rm)
    mask = torch.arange(T, device=dev)[None, :] >= torch.randint((T + 1) // 2, T + 1, (B, 1), device=dev) if masked else None
    g = torch.randn(T, B, layer.embed_dim, device=dev).half()
    if expand:
        g = g[:1, :1].expand(T, B, -1)
    y, grads = step(layer, x, rm, mask, g, torch.enable_grad())
    assert "ProjectBackward" in type(y.grad_fn).__name__ or "ProjectBackward" in y.grad_fn.name()
    y2, grads2 = step(layer, x, rm, mask, g, Seen())
    assert "ProjectBackward" not in y2.grad_fn.name()
    assert torch.equal(y, y2)
    for a, b in zip(grads, grads2):
        assert (a is None) == (b is None)
        if b is not None:
            assert a.dtype == b.dtype and a.shape == b.shape and a.stride() == b.stride()
            assert float((a.double() - b.double()).norm()) <= 2.0 ** -9 * float(b.double().norm()) + 1e-6


def test_gradients_of_gradients_and_changed_weights(dev):
    layer, rm = make(dev)
    x = torch.randn(20, 3, layer.embed_dim, device=dev).half().requires_grad_()
    second = []
    for context in (torch.enable_grad(), Seen()):
        with context:
            y = layer(x, rm)
        gw, gb = torch.autograd.grad(y.float().square().sum(), [layer.out_proj.weight, layer.out_proj.bias], create_graph=True)
        second.append(torch.autograd.grad(gw.float().square().mean() + gb.float().square().mean(), [x, layer.v_proj.weight]))
    for a, b in zip(*second):
        assert float((a.double() - b.double()).norm()) <= 2.0 ** -8 * float(b.double().norm())
    y = layer(x, rm)
    with torch.no_grad():
        layer.v_proj.weight.mul_(2)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.sum().backward()
    y = layer(x.detach(), rm)                             # without the input's gradient the projections' weights are not kept
    with torch.no_grad():
        layer.v_proj.weight.mul_(2)
    y.sum().backward()


def test_what_goes_module_by_module(dev):
    layer, rm = make(dev)
    x = torch.randn(20, 3, layer.embed_dim, device=dev).half().requires_grad_()
    native = lambda y: "ProjectBackward" in y.grad_fn.name()
    assert native(layer(x, rm))
    assert not native(layer(x.transpose(0, 1).contiguous().transpose(0, 1), rm))
    assert native(layer(x, rm, key_padding_mask=torch.zeros(3, 20, dtype=torch.bool, device=dev)))
    assert not native(layer(x, rm, key_padding_mask=torch.zeros(3, 20, dtype=torch.uint8, device=dev)))
    with pytest.raises(AssertionError):
        layer(x, rm, key_padding_mask=torch.zeros(20, 3, dtype=torch.bool, device=dev))
    calls = []
    handle = layer.k_proj.register_forward_hook(lambda *a: calls.append(1))
    assert not native(layer(x, rm)) and calls == [1]
    handle.remove()
    with torch.autocast("cuda", dtype=torch.float16):
        assert not native(layer(x, rm))
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t, lambda t: t):
        layer(x, rm).sum().backward()
    assert packed


@pytest.mark.parametrize("heads,head_dim,proj_dim", [(16, 32, 64), (4, 128, 32), (8, 64, 64)])
def test_matrices_of_another_split_into_heads_are_refused(dev, heads, head_dim, proj_dim):
    """A layer of 8 heads of 64 without sigma: matrices of 16 heads of 32 divide its features too, and are refused as they are module by module."""
    layer = CausalAttention(embed_dim=512, num_heads=8, head_dim=64, proj_dim=64, reparam_proj=False).to(dev).half()
    rm = torch.randn(heads, proj_dim, head_dim, device=dev).half()
    train = lambda: layer(torch.randn(20, 2, 512, device=dev).half().requires_grad_(), rm)
    state = {}

    def decode():
        with torch.no_grad():
            return layer(torch.randn(1, 2, 512, device=dev).half(), rm, saved_state=state)
    for call in (train, decode):
        if heads == 8:
            call()
            continue
        with pytest.raises((AssertionError, ValueError, RuntimeError)):
            call()
        assert not state


def test_a_temperature_that_is_a_tensor(dev):
    """Its gradient, and the results of the number that it holds."""
    torch.manual_seed(0)
    layer, rm = make(dev)
    x = torch.randn(20, 2, 512, device=dev).half()
    layer.tau = 2.0
    want, first = layer(x, rm), layer(x[:1], rm, saved_state={})
    layer.tau = torch.nn.Parameter(torch.tensor(2.0, device=dev))
    got = layer(x, rm)
    got.sum().backward()
    assert layer.tau.grad is not None and torch.isfinite(layer.tau.grad) and layer.tau.grad != 0
    near = lambda a, b: ((a - b).float().norm() / b.float().norm()).item() < 3e-3
    with torch.no_grad():
        assert near(got, want) and near(layer(x, rm), want) and near(layer(x[:1], rm, saved_state={}), first)
