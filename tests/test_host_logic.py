"""Host-side mirrors of upstream's Python helpers, checked on CPU against the oracle
and the upstream-generated fixtures."""
import argparse

import numpy as np
import pytest
import torch

from conftest import golden
from oracle import rfa_oracle as O


def test_matrix_generators_match_upstream_bitwise():
    from rfa_b200 import construct_random_matrices as crm
    g = golden("matrices")
    np.random.seed(1)
    mine = np.stack([crm.orf(head_dim=64, proj_dim=64) for _ in range(4)])
    assert np.array_equal(mine, g["orf_seed1"].numpy())
    np.random.seed(7)
    assert np.array_equal(np.stack([crm.rrf(head_dim=64, proj_dim=64) for _ in range(2)]), g["rrf_seed7"].numpy())
    np.random.seed(11)
    assert np.array_equal(np.stack([crm.orf(head_dim=32, proj_dim=48) for _ in range(2)]), g["orf_wide_seed11"].numpy())


def test_matrix_bank_cli(tmp_path):
    from rfa_b200 import construct_random_matrices as crm
    out = tmp_path / "64_64.npy"
    crm.NUM_MATRICES, keep = 3, crm.NUM_MATRICES
    try:
        crm.main(["prog", "orf", "64", "64", str(out)])
    finally:
        crm.NUM_MATRICES = keep
    bank = np.load(out)
    assert bank.shape == (3, 64, 64)
    assert np.array_equal(bank, O.draw_matrices("orf", 3, 64, 64, 31415))
    assert crm.test(64, 64, bank[0].copy(), num_ites=5) < 0.5     # kernel approximation quality is sane


def test_torch_twins_match_oracle():
    from rfa_b200.rfa import RFA, reverse_cumsum, rfa_debug
    g = golden("causal_bwd_gradcheck")
    q, k, v, up = g["q"], g["k"], g["v"], g["g"]
    assert torch.allclose(RFA.forward_torch(q, k, v), g["attn"], atol=2e-6)
    assert torch.allclose(rfa_debug(q, k, v), g["attn"], atol=2e-6)
    for a, b in zip(RFA.backward_torch(q, k, v, up), (g["gq"], g["gk"], g["gv"])):
        assert torch.allclose(a, b, atol=1e-5)
    x = torch.arange(12.).view(3, 4)
    assert torch.equal(reverse_cumsum(x, 0), torch.flip(torch.cumsum(torch.flip(x, [0]), 0), [0]))


def test_utils_helpers():
    from rfa_b200 import utils
    g = golden("feature_map")
    w = utils.build_random_matrices(g["w"], float(g["tau"]), g["sigma"], True)
    assert torch.allclose(w, g["w_eff"], rtol=1e-6)
    assert torch.equal(utils.build_random_matrices(g["w"], 1.0), g["w"])
    xn, n = utils._normalize(g["x"])
    assert torch.allclose(xn, g["x"] / (g["x"].norm(dim=-1, keepdim=True) + 1e-3))
    bank = torch.arange(10 * 2 * 3.).view(10, 2, 3)
    ev = utils.sample_random_matrices(num_layers=3, num_heads=2, random_matrices=bank, is_training=False)
    assert torch.equal(ev, bank[:2])
    np.random.seed(0)
    tr = utils.sample_random_matrices(num_layers=3, num_heads=2, random_matrices=bank, is_training=True)
    np.random.seed(0)
    idx = np.random.choice(10, size=6, replace=False)
    assert len(tr) == 3 and all(torch.equal(tr[i], bank[idx[2 * i:2 * i + 2]]) for i in range(3))
    p = utils.add_rfa_args(argparse.ArgumentParser())
    a = utils.get_rfa_attr(p.parse_args(["--use-rfa", "--causal-proj-dim", "32"]))
    assert a.use_rfa and a.use_linfa and a.causal_proj_dim == 32 and a.cross_tau is None
    a = utils.get_rfa_attr(argparse.Namespace())
    assert (a.cross_proj_dim, a.causal_tau, a.reparam_proj, a.cuda_causal_rfa) == (64, 1.0, True, True)
    wts = utils.normalize_attn_weights(torch.tensor([[1., 3.], [0., 0.]]))
    assert torch.allclose(wts, torch.tensor([[.25, .75], [0., 0.]]))
    st = utils.CrossAttentionState(torch.zeros(1), torch.zeros(1), [], 1.0)
    assert st.tau == 1.0 and st._fields == ("s", "z", "random_matrices", "tau")


def test_masked_rfa_is_upstreams_quadratic_variant():
    from rfa_b200.causal_attention import masked_rfa
    gen = torch.Generator().manual_seed(0)
    T, B, H = 12, 2, 2
    pq, pk = torch.rand(T, B, H, 16, generator=gen), torch.rand(T, B, H, 16, generator=gen)
    v = torch.randn(T, B, H, 8, generator=gen)
    causal = torch.triu(torch.full((T, T), float("-inf")), 1)
    out = masked_rfa(phi_q=pq, phi_k=pk, v=v, attn_mask=causal)
    # with positive features every row sum exceeds 1e-3, so this equals sum-normalised causal attention
    a = torch.einsum("tbhk,sbhk->bhts", pq, pk) * torch.tril(torch.ones(T, T))
    ref = torch.einsum("bhts,sbhd->tbhd", a / a.sum(-1, keepdim=True), v).reshape(T, B, H * 8)
    assert torch.allclose(out, ref, atol=1e-5)


def test_cpu_list_parsing_for_numa_binding():
    from rfa_b200.host_pipeline import _cpulist, gpu_numa_cpus
    assert _cpulist("0-3,8,10-11\n") == [0, 1, 2, 3, 8, 10, 11]
    assert _cpulist("") == []
    assert gpu_numa_cpus(0, sysfs="/nonexistent") is None       # no GPU / no sysfs entry: nothing to bind to


def test_matrix_sampling_with_a_generator_is_reproducible():
    from rfa_b200.utils import sample_matrix_indices, sample_random_matrices
    mk = lambda: torch.Generator().manual_seed(7)
    a = sample_matrix_indices(num_layers=3, num_heads=4, bank_size=50, generator=mk())
    b = sample_matrix_indices(num_layers=3, num_heads=4, bank_size=50, generator=mk())
    assert torch.equal(a, b) and a.numel() == 12 and len(set(a.tolist())) == 12 and int(a.max()) < 50
    bank = torch.arange(50.).view(50, 1, 1).expand(50, 2, 3).contiguous()
    layers = sample_random_matrices(num_layers=3, num_heads=4, random_matrices=bank, generator=mk())
    assert len(layers) == 3 and torch.equal(torch.cat(layers)[:, 0, 0].long(), a)
    import numpy as np
    np.random.seed(3)
    x = sample_matrix_indices(num_layers=2, num_heads=2, bank_size=9)        # upstream's way: numpy's global RNG
    np.random.seed(3)
    assert x.tolist() == np.random.choice(9, size=4, replace=False).tolist()


def test_staged_tiles_are_released_behind_the_proxy_fence():
    """A stage that TMA refills is given back through ``mbar_release_stage`` (fence, then arrive): an arrive alone does not keep
    the thread's plain reads of the tile in front of the refill.  Where a TMA store has read the stage, the wait for it does."""
    import glob
    import os
    import re
    root = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rfa_b200", "csrc")
    sites = 0
    for path in sorted(glob.glob(os.path.join(root, "*.cu"))):
        lines = open(path).read().splitlines()
        for i, line in enumerate(lines):
            if re.search(r"mbar_release_stage\(&bars\[\w*Empty", line):
                sites += 1
            if re.search(r"mbar_arrive\(&bars\[\w*Empty", line):
                assert "tma_store_wait_read<0>()" in lines[i - 1], f"{os.path.basename(path)}:{i + 1}: {line.strip()}"
    assert sites >= 9


@pytest.mark.parametrize("what", ["x", "sigma"])
def test_one_token_refuses_forward_mode(monkeypatch, what):
    """A tangent reaches the feature map's autograd function, which has no forward-mode rule, instead of being dropped by the
    fused decoding step (a plain kernel call)."""
    import torch.autograd.forward_ad as fw
    from rfa_b200 import CausalAttention, ops
    monkeypatch.setattr(ops, "decode_fused_supported", lambda q, w: True)
    monkeypatch.setattr(ops, "decode_step_fused", lambda q, k, v, w, scale, s, z: v.clone())
    monkeypatch.setattr(ops, "feature_map_fwd", lambda x, w, scale, row_mask=None: torch.cat([x, x], dim=-1))
    layer = CausalAttention(embed_dim=16, num_heads=2, head_dim=8, proj_dim=8)
    x, w = torch.randn(1, 3, 16), torch.randn(2, 8, 8)
    with torch.no_grad():
        assert layer(x, w, saved_state={}).shape == x.shape
        with fw.dual_level():
            if what == "x":
                x = fw.make_dual(x, torch.ones_like(x))
            else:
                sigma = layer.sigma.detach()
                del layer.sigma
                layer.sigma = fw.make_dual(sigma, torch.ones_like(sigma))
            with pytest.raises(NotImplementedError, match="jvp"):
                layer(x, w, saved_state={})


def test_native_calls_leave_the_interpreter_to_other_threads():
    """The tensor-level calls run without the interpreter lock.  The time is that of a strided copy of the input, which
    comes before the call finds that it is on the CPU."""
    import threading
    import time
    from rfa_b200 import ops
    x, w = torch.zeros(64, 1 << 20).t().unsqueeze(1), torch.zeros(1, 8, 64)
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(1e-3)
    threads = torch.get_num_threads()
    torch.set_num_threads(1)
    other = threading.Thread(target=tick)
    other.start()
    try:
        time.sleep(0.02)
        t0 = time.perf_counter()
        with pytest.raises(RuntimeError, match="CUDA tensors only"):
            ops.feature_map_fwd(x, w, 0.1)
        t1 = time.perf_counter()
    finally:
        stop.set()
        other.join()
        torch.set_num_threads(threads)
    seen = [t0] + [t for t in ticks if t0 < t < t1] + [t1]
    assert max(b - a for a, b in zip(seen, seen[1:])) < 0.5 * (t1 - t0), (len(seen), t1 - t0)


@pytest.mark.parametrize("T", [0, 3])
def test_a_state_without_its_denominators_is_refused(T):
    from rfa_b200 import ops
    q, v = torch.zeros(T, 2, 128, dtype=torch.half), torch.zeros(T, 2, 64, dtype=torch.half)
    with pytest.raises(ValueError, match="pair"):
        ops.causal_fwd(q, q, v, torch.zeros(2, 128, 64), None, return_state=True)


def test_a_padding_mask_of_another_size_raises_a_runtime_error():
    from rfa_b200 import ops
    phi, v = torch.zeros(4, 2, 3, 128, dtype=torch.half), torch.zeros(4, 2, 3, 64, dtype=torch.half)
    with pytest.raises(RuntimeError, match="shape"):
        ops.cross_state_fwd(phi, v, torch.zeros(3, 3))
    with pytest.raises(RuntimeError, match="shape"):
        ops.cross_state_bwd(phi, v, torch.zeros(3, 3), torch.zeros(2, 3, 128, 64), torch.zeros(2, 3, 128))


def test_the_native_module_is_rebuilt_for_another_torch(monkeypatch, tmp_path):
    """The command that the import error names has to do something: a module newer than its sources but built for another torch
    is stale."""
    import os
    from rfa_b200 import build
    module, key = tmp_path / "_native.so", tmp_path / "_native.key"
    monkeypatch.setattr(build, "NATIVE", str(module))
    monkeypatch.setattr(build, "NATIVE_KEY", str(key))
    assert build.native_stale()                      # nothing built
    module.write_bytes(b"")
    newest = max(os.path.getmtime(p) for p in (build.NATIVE_SRC, str(module)))
    os.utime(module, (newest + 10, newest + 10))
    assert build.native_stale()                      # built for nobody knows what
    key.write_text(build.native_key())
    assert not build.native_stale()
    monkeypatch.setattr(torch, "__version__", "0.0")
    assert build.native_stale()


def test_what_a_native_short_cut_leaves_to_the_tensor_expressions():
    """CPU tensors, subclasses and every context that wants to see a call: compiling, a transform, a mode, a forward-mode level; a caller
    that is compiled reaches the function as before (here: its refusal of CPU tensors)."""
    import torch.autograd.forward_ad as fw
    from rfa_b200 import _plain
    from rfa_b200.rfa import RFA
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    class Function(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    class Dispatch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))
    assert _plain.plain_context() and not _plain.plain_tensors(torch.zeros(1))
    for context in (Function, Dispatch, fw.dual_level):
        with context():
            assert not _plain.plain_context()
    seen = []
    torch.func.vmap(lambda x: (seen.append(_plain.plain_context()), x)[1])(torch.zeros(2))
    torch.jit.trace(lambda x: (seen.append(_plain.plain_context()), x + 1)[1], torch.zeros(2), check_trace=False)
    assert seen and not any(seen)
    assert torch.compile(lambda x: x + 1 if _plain.plain_context() else x + 2, backend="eager")(torch.zeros(1)).item() == 2
    q = torch.zeros(4, 1, 128, dtype=torch.half)
    with pytest.raises(RuntimeError, match="no CPU path"):
        torch.compile(lambda q, v: RFA.apply(q, q, v) * 2, backend="eager")(q, q[..., :64])


@pytest.fixture
def layer_pass(monkeypatch):
    """A layer, its q, k, v and matrices, in place of whose CUDA tensors CPU ones stand; which of them a pass hands to the kernel."""
    from rfa_b200 import CausalAttention, causal_attention, ops
    monkeypatch.setattr(ops, "fused_forward_supported", lambda *_: True)
    monkeypatch.setattr(causal_attention, "plain_tensors", lambda *_: True)
    layer = CausalAttention(embed_dim=128, num_heads=2, head_dim=64, proj_dim=64).half().requires_grad_(False)
    qkv = list(torch.zeros(3, 5, 1, 2, 64, dtype=torch.half))
    return layer, qkv, torch.zeros(2, 64, 64, dtype=torch.half)


def test_a_layer_pass_keeps_matrices_of_another_device_from_the_kernel(layer_pass):
    """`meta` stands for another GPU: the tensor expressions refuse it, and so does the native call itself, before anything is launched."""
    from rfa_b200._lib import native
    layer, (q, k, v), w = layer_pass
    assert layer._fused_layer_pass(q, k, v, w, None)
    assert not layer._fused_layer_pass(q, k, v, w.to("meta"), None)
    layer.sigma = torch.nn.Parameter(layer.sigma.to("meta"), requires_grad=False)
    assert not layer._fused_layer_pass(q, k, v, w, None)
    for sigma, rm in ((None, w.to("meta")), (layer.sigma, w)):
        with pytest.raises(RuntimeError, match="expected all tensors on cpu, got one on meta"):
            native().causal_fwd_fused_layer(q, k, v, rm, sigma, 1.0, 0.1, None)


def test_a_layer_pass_keeps_matrices_at_odd_addresses_from_the_kernel(layer_pass):
    layer, (q, k, v), w = layer_pass
    odd = lambda t: torch.cat([t.new_zeros(3), t.flatten()])[3:].view(t.shape)
    assert not layer._fused_layer_pass(q, k, v, odd(w), None)
    layer.sigma = torch.nn.Parameter(odd(layer.sigma.data), requires_grad=False)
    assert not layer._fused_layer_pass(q, k, v, w, None)


def test_a_layer_pass_leaves_a_temperature_that_is_a_tensor_to_the_tensor_expressions(layer_pass):
    layer, (q, k, v), w = layer_pass
    assert layer._fused_layer_pass(q, k, v, w, None)
    layer.tau = torch.tensor(2.0)
    assert not layer._fused_layer_pass(q, k, v, w, None)


def test_a_layer_pass_asks_for_no_address_while_it_is_traced(layer_pass, monkeypatch):
    """A tensor that only stands for one while a call is traced or compiled has none."""
    from rfa_b200 import causal_attention
    layer, (q, k, v), w = layer_pass
    monkeypatch.setattr(causal_attention, "plain_tensors", lambda *_: False)
    monkeypatch.setattr(torch.Tensor, "data_ptr", lambda self: pytest.fail("asked for an address"))
    assert not layer._fused_layer_pass(q, k, v, w, None)
