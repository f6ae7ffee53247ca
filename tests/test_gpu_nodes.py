"""The native autograd nodes against the Python functions of the same graph, which a dispatch mode around the call selects (plain
calls take the native ones), and the contexts that must keep the Python ones."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from rfa_b200 import _plain, ops
from rfa_b200.cross_attention import cross_rfa_query, cross_rfa_state
from rfa_b200.rfa import RFA
from rfa_b200.utils import random_project, random_project_pair

pytestmark = pytest.mark.gpu


class Seen(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


def features(gen, dev, *shape):
    return (torch.rand(*shape, generator=gen) * 0.3 - 0.1).half().to(dev)


def case(kind, dev):
    gen = torch.Generator().manual_seed(len(kind))
    n = lambda *s: torch.randn(*s, generator=gen).half().to(dev)
    w = torch.randn(3, 64, 64, generator=gen).to(dev)
    pad = (torch.rand(2, 50, generator=gen) < 0.3).to(dev)
    if kind == "causal":
        return [features(gen, dev, 200, 4, 128), features(gen, dev, 200, 4, 128), n(200, 4, 64)], RFA.apply
    if kind == "features":
        return [n(50, 2, 3, 64), w], lambda x, w: random_project(x=x, random_matrices=w, key_padding_mask=pad)
    if kind == "features_half_matrices":
        return [n(50, 2, 3, 64), w.half()], lambda x, w: random_project(x=x, random_matrices=w)
    if kind == "pair":
        return [n(50, 2, 3, 64), n(50, 2, 3, 64), w], lambda a, b, w: torch.cat(random_project_pair(x_a=a, x_b=b, random_matrices=w, key_padding_mask_b=pad))
    if kind == "pair_one_used":
        return [n(50, 2, 3, 64), n(50, 2, 3, 64), w], lambda a, b, w: random_project_pair(x_a=a, x_b=b, random_matrices=w)[0]
    return ([features(gen, dev, 50, 2, 3, 128), n(50, 2, 3, 64), features(gen, dev, 40, 2, 3, 128)],
            lambda k, v, q: cross_rfa_query(q, *cross_rfa_state(k, v, pad)))


def run(leaves, f, needed, context):
    leaves = [t.detach().clone().requires_grad_(need) for t, need in zip(leaves, needed)]
    with context:
        y = f(*leaves)
    g = torch.randn(y.shape, generator=torch.Generator().manual_seed(1)).to(y)
    y.backward(g)
    return y, [t.grad for t in leaves]


@pytest.mark.parametrize("kind", ["causal", "features", "features_half_matrices", "pair", "pair_one_used", "cross"])
def test_native_nodes_make_the_same_graph(dev, kind):
    """Outputs bit for bit; gradients too, but for g_W, whose CTAs' sums meet in atomics in any order: 1e-6 (fp16 matrices: 2^-11)."""
    leaves, f = case(kind, dev)
    for needed in ([True] * len(leaves), [i == 0 for i in range(len(leaves))], [i == len(leaves) - 1 for i in range(len(leaves))]):
        if kind == "pair_one_used" and needed[0] is False:
            continue
        y, grads = run(leaves, f, needed, torch.enable_grad())
        assert "Python" not in type(y.grad_fn).__name__
        y2, grads2 = run(leaves, f, needed, Seen())
        assert torch.equal(y, y2)
        for need, a, b, leaf in zip(needed, grads, grads2, leaves):
            assert (a is None) == (b is None) == (not need)
            if need:
                assert a.dtype == b.dtype == leaf.dtype and a.shape == leaf.shape
                if leaf.dim() == 3 and leaf.shape[0] == 3:
                    assert float((a - b).float().norm() / b.float().norm().clamp_min(1e-30)) < (2.0 ** -11 if leaf.dtype == torch.float16 else 1e-6)
                else:
                    assert torch.equal(a, b)


def test_hooks_on_saved_tensors_and_a_second_backward(dev):
    leaves, f = case("causal", dev)
    leaves = [t.requires_grad_() for t in leaves]
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(t.shape), t.cpu())[1], lambda t: t.to(dev)):
        y = f(*leaves)
    assert len(packed) == 5                              # q, k, v, the output and the workspace
    a = torch.autograd.grad(y.sum(), leaves, retain_graph=True)
    b = torch.autograd.grad(y.sum(), leaves)
    assert all(torch.equal(s, t) for s, t in zip(a, b))
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(y.sum(), leaves)
    y = f(*leaves)
    with torch.no_grad():
        leaves[1].add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace"):
        y.sum().backward()


def test_refusals_keep_their_types(dev):
    q = torch.zeros(4, 2, 128, device=dev, dtype=torch.half)
    with pytest.raises(TypeError, match="fp16"):
        RFA.apply(q.float(), q, q[..., :64])
    with pytest.raises(AssertionError):
        random_project(x=torch.zeros(4, 1, 2, 64, device=dev), random_matrices=torch.zeros(3, 64, 64, device=dev))
    with torch.autograd.forward_ad.dual_level(), pytest.raises(NotImplementedError, match="jvp"):
        RFA.apply(torch.autograd.forward_ad.make_dual(q, q), q, q[..., :64])
    assert _plain.plain_tensors(q, None) and not _plain.plain_tensors(q.cpu())
    with Seen():
        assert not _plain.plain_tensors(q)


def test_a_compiled_caller_runs(dev):
    leaves, f = case("causal", dev)
    want = f(*leaves)
    assert torch.equal(torch.compile(lambda q, k, v: RFA.apply(q, k, v) * 2, backend="eager")(*leaves), want * 2)
    assert ops.causal_fwd(*leaves).shape == want.shape
