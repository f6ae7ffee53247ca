"""Tensor-level wrappers over the C ABI: allocate outputs, pass raw pointers and
the current stream, turn status codes into exceptions.  No arithmetic happens
here; every function launches kernels from ``librfa_b200.so``.  The calls of the
forward, backward and decoding paths are in ``csrc/torch_ops.cpp``; the rest go
through ctypes.
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch
from torch import Tensor

from . import _lib
from ._lib import check, dtype_code, native, ptr, require_half, stream_of

K_BUILT, D_BUILT = 128, 64      # geometry the attention kernels are built for


def _guard(t: Tensor):
    if not t.is_cuda:
        raise RuntimeError(f"rfa_b200 kernels take CUDA tensors only (there is no CPU path); got a {t.device} tensor")
    return _Guard(t.device)


class _Guard:
    """Make the tensor's device current for the call and, on first use of a device, switch on the status mirror."""

    def __init__(self, device):
        self.ctx = torch.cuda.device(device)
        self.index = device.index if device.index is not None else torch.cuda.current_device()

    def __enter__(self):
        self.ctx.__enter__()
        _lib.watch_device(self.index)
        return self

    def __exit__(self, *a):
        return self.ctx.__exit__(*a)


def _workspace(T: int, BH: int, K: int, d: int, like: Tensor) -> Tuple[Tensor, int]:
    n = _lib.load().rfa_causal_workspace_bytes(T, BH, K, d)
    ws = torch.empty(max(n, 256), dtype=torch.uint8, device=like.device)
    return ws, n


# --------------------------------------------------------------------------- feature map
def feature_map_fwd(x: Tensor, w: Tensor, scale: float, out_dtype: Optional[torch.dtype] = None,
                    row_mask: Optional[Tensor] = None) -> Tensor:
    """x [..., H, d], w [H, D, d] fp32 -> phi [..., H, 2D].  row_mask (one entry per leading index, non-zero = masked):
    those rows get all-zero features."""
    return native().feature_map_fwd(x, w, scale, out_dtype, row_mask)


def feature_map_bwd(x: Tensor, w: Tensor, g_phi: Tensor, scale: float, need_gw: bool,
                    row_mask: Optional[Tensor] = None) -> Tuple[Tensor, Optional[Tensor]]:
    return native().feature_map_bwd(x, w, g_phi, scale, need_gw, row_mask)


def feature_map_pair_supported(x_a: Tensor, x_b: Tensor, w: Tensor) -> bool:
    """Whether the one-launch feature map of two arrays takes these: same shape, fp16, head_dim = proj_dim = 64."""
    return (x_a.shape == x_b.shape and x_a.dtype == x_b.dtype == torch.float16 and x_a.is_cuda and x_b.is_cuda
            and tuple(w.shape[-2:]) == (64, 64))


def feature_map_fwd_pair(x_a: Tensor, x_b: Tensor, w: Tensor, scale: float, row_mask_a: Optional[Tensor] = None,
                         row_mask_b: Optional[Tensor] = None) -> Tuple[Tensor, Tensor]:
    """phi of x_a and of x_b (same shape [..., H, 64], fp16; w [H, 64, 64]) in one launch."""
    return native().feature_map_fwd_pair(x_a, x_b, w, scale, row_mask_a, row_mask_b)


def feature_map_bwd_pair(x_a: Tensor, x_b: Tensor, w: Tensor, g_phi_a: Tensor, g_phi_b: Tensor, scale: float, need_gw: bool,
                         row_mask_a: Optional[Tensor] = None, row_mask_b: Optional[Tensor] = None):
    """Backward of ``feature_map_fwd_pair``: (g_x_a, g_x_b, g_w) with g_w the sum of both arrays' contributions (or None)."""
    return native().feature_map_bwd_pair(x_a, x_b, w, g_phi_a, g_phi_b, scale, need_gw, row_mask_a, row_mask_b)


def gather_random_matrices(bank: Tensor, picks: Tensor, sigma: Optional[Tensor] = None,
                           inv_tau: Optional[Tensor] = None) -> Tensor:
    """bank [N, D, d] (fp16 / fp32, on the device), picks [n] int64 -> [n, D, d] fp32 = sigma[i] * bank[picks[i]] * inv_tau[i]
    (sigma [n, d], inv_tau [n], both optional), one launch."""
    N, D, d = bank.shape
    bank = bank.contiguous()
    picks = picks.to(device=bank.device, dtype=torch.int64).contiguous()
    n = picks.numel()
    out = torch.empty(n, D, d, dtype=torch.float32, device=bank.device)
    if sigma is not None:
        sigma = sigma.to(device=bank.device, dtype=torch.float32).reshape(n, d).contiguous()
    if inv_tau is not None:
        inv_tau = inv_tau.to(device=bank.device, dtype=torch.float32).reshape(n).contiguous()
    bad = torch.zeros(1, dtype=torch.int32, device=bank.device)
    with _guard(bank):
        check(_lib.load().rfa_gather_random_matrices(ptr(bank), dtype_code(bank), N, ptr(picks), n, ptr(sigma), ptr(inv_tau),
                                                     ptr(out), D, d, ptr(bad), stream_of(bank)), "rfa_gather_random_matrices")
    return out, bad


# --------------------------------------------------------------------------- causal
def causal_fwd(q: Tensor, k: Tensor, v: Tensor, s_in: Optional[Tensor] = None, z_in: Optional[Tensor] = None,
               return_state: bool = False):
    """q,k [T,BH,K], v [T,BH,d] fp16 -> out [T,BH,d] (and the final state when asked)."""
    out, s_out, z_out = native().causal_fwd(q, k, v, s_in, z_in, return_state)
    return (out, s_out, z_out) if return_state else out


def causal_bwd(q: Tensor, k: Tensor, v: Tensor, g: Tensor, s_in: Optional[Tensor] = None,
               z_in: Optional[Tensor] = None, ds_in: Optional[Tensor] = None, dz_in: Optional[Tensor] = None):
    require_half(q, k, v, g)
    T, BH, K = q.shape
    d = v.shape[-1]
    q, k, v, g = q.contiguous(), k.contiguous(), v.contiguous(), g.contiguous()
    gq, gk, gv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    if T == 0:
        return gq, gk, gv
    ws, n = _workspace(T, BH, K, d, q)
    with _guard(q):
        check(_lib.load().rfa_causal_bwd(ptr(q), ptr(k), ptr(v), ptr(g), ptr(gq), ptr(gk), ptr(gv), ptr(s_in),
                                         ptr(z_in), ptr(ds_in), ptr(dz_in), ptr(ws), n, T, BH, K, d, stream_of(q)),
              "rfa_causal_bwd")
    return gq, gk, gv


# --------------------------------------------------------------------------- causal, staged (kept workspace / saved output)
STATE_N = K_BUILT * D_BUILT + K_BUILT      # floats of one packed state [S | z]


def causal_fwd_saved(q: Tensor, k: Tensor, v: Tensor, s_in: Optional[Tensor] = None, z_in: Optional[Tensor] = None,
                     ws: Optional[Tensor] = None, ws_has: int = 0):
    """Forward that keeps what the backward can reuse.  Returns (out, workspace, ws_has): the workspace then holds the
    raw denominators and, when the sequence is cut into segments, the states entering each of them.  ``ws`` / ``ws_has``
    hand in a workspace that ``shard_total`` has already filled for the same k, v."""
    out, ws = native().causal_fwd_saved(q, k, v, s_in, z_in, ws, ws_has)
    return out, ws, (_lib.WS_STATES | _lib.WS_DEN if q.shape[0] else 0)


def fused_forward_supported(x: Tensor, w: Tensor) -> bool:
    """Whether ``causal_fwd_fused`` takes these inputs: fp16 vectors of head_dim 64 with proj_dim 64 matrices, and enough
    (batch, head) sequences that one CTA each fills the GPU (the kernel does not cut a sequence into segments)."""
    T, B, H, d = x.shape
    return (x.dtype == torch.float16 and x.is_cuda and d == 64 and tuple(w.shape[-2:]) == (64, 64)
            and (B * H >= 120 or T < 1024))


def causal_fwd_fused(x_q: Tensor, x_k: Tensor, v: Tensor, w: Tensor, scale: float, row_mask: Optional[Tensor] = None,
                     s_in: Optional[Tensor] = None, z_in: Optional[Tensor] = None, return_state: bool = False,
                     save_den: bool = False, *, sigma: Optional[Tensor] = None, tau: Optional[float] = None,
                     pad_mask: Optional[Tensor] = None):
    """Causal RFA forward from the raw per-head vectors: x_q, x_k, v [T, B, H, 64] fp16, w [H, 64, 64] fp32; the features
    scale * [sin | cos]((W x) / (|x| + 1e-3)) of q and k are formed inside the kernel.  row_mask [T, B] (or [T * B]) marks
    padded keys.  Returns out [T, B*H, 64] and, as asked, the final state (s, z) and the workspace holding the raw
    denominators for ``causal_bwd_saved(..., ws_has=WS_DEN)``: (out[, s, z][, ws]).

    With ``tau`` given, w is the layer's own fp16 bank [H, 64, 64], taken as sigma * w / tau (``sigma`` [H, 1, 64] fp16 or None), and
    ``pad_mask`` [B, T] its padding mask: out alone, and no launch but this one."""
    if tau is not None:
        assert row_mask is None and s_in is None and z_in is None and not return_state and not save_den
        return native().causal_fwd_fused_layer(x_q, x_k, v, w, sigma, tau, scale, pad_mask)
    out, s_out, z_out, ws = native().causal_fwd_fused(x_q, x_k, v, w, scale, row_mask, s_in, z_in, return_state, save_den)
    res = (out,)
    if return_state:
        res += (s_out, z_out)
    if save_den:
        res += (ws,)
    return res if len(res) > 1 else out


def causal_bwd_saved(q: Tensor, k: Tensor, v: Tensor, g: Tensor, out: Tensor, ws: Tensor, ws_has: int,
                     s_in: Optional[Tensor] = None, z_in: Optional[Tensor] = None):
    """Backward from the forward's output and kept workspace (``causal_fwd_saved``)."""
    return native().causal_bwd_saved(q, k, v, g, out, ws, ws_has, s_in, z_in)


def shard_total(k: Tensor, v: Tensor, packed: Optional[Tensor] = None):
    """This shard's own [sum k (x) v | sum k], packed [BH, K*d + K] fp32 (into ``packed`` when given, e.g. a slice of an
    all-gather buffer), and the workspace holding the per-segment partial sums for ``causal_fwd_saved``."""
    require_half(k, v)
    T, BH, K = k.shape
    d = v.shape[-1]
    k, v = k.contiguous(), v.contiguous()
    if packed is None:
        packed = torch.empty(BH, K * d + K, dtype=torch.float32, device=k.device)
    if T == 0:
        packed.zero_()
        return packed, None
    ws, _ = _workspace(T, BH, K, d, k)
    with _guard(k):
        check(_lib.load().rfa_causal_shard_total(ptr(k), ptr(v), ptr(packed), ptr(ws), ws.numel(), T, BH, K, d, stream_of(k)),
              "rfa_causal_shard_total")
    return packed, ws


def scan_gathered(gathered: Tensor, rank: int, reverse: bool, K: int = K_BUILT, d: int = D_BUILT):
    """gathered [world, BH, K*d + K] fp32 (every shard's packed total) -> the carry of shard ``rank``: the sum over the
    shards before (``reverse``: after) it, as (s [BH,K,d], z [BH,K])."""
    world, BH, n = gathered.shape
    assert n == K * d + K and gathered.dtype == torch.float32 and gathered.is_contiguous()
    s = torch.empty(BH, K, d, dtype=torch.float32, device=gathered.device)
    z = torch.empty(BH, K, dtype=torch.float32, device=gathered.device)
    with _guard(gathered):
        check(_lib.load().rfa_exclusive_scan_gathered(ptr(gathered), world, rank, int(reverse), ptr(s), ptr(z), BH, K, d,
                                                      stream_of(gathered)), "rfa_exclusive_scan_gathered")
    return s, z


def causal_bwd_q_staged(q, k, v, g, out, s_in, z_in, ws: Tensor, ws_has: int, packed: Optional[Tensor] = None,
                        want_total: bool = True):
    """Forward-direction half of the backward on a kept workspace.  Returns (gq, packed reverse-state total or None)."""
    require_half(q, k, v, g)
    T, BH, K = q.shape
    d = v.shape[-1]
    q, k, v, g = q.contiguous(), k.contiguous(), v.contiguous(), g.contiguous()
    gq = torch.empty_like(q)
    if want_total and packed is None:
        packed = torch.empty(BH, K * d + K, dtype=torch.float32, device=q.device)
    if T == 0:
        if want_total:
            packed.zero_()
        return gq, packed if want_total else None
    with _guard(q):
        check(_lib.load().rfa_causal_bwd_q_staged(ptr(q), ptr(k), ptr(v), ptr(g), ptr(out), ptr(gq), ptr(s_in), ptr(z_in),
                                                  ptr(packed) if want_total else None, ptr(ws), ws.numel(), T, BH, K, d, ws_has,
                                                  stream_of(q)), "rfa_causal_bwd_q_staged")
    return gq, packed if want_total else None


def causal_bwd_q(q, k, v, g, s_in, z_in, want_dseg: bool):
    """Forward-direction half of the backward.  Returns (gq, ds_seg, dz_seg, workspace)."""
    require_half(q, k, v, g)
    T, BH, K = q.shape
    d = v.shape[-1]
    q, k, v, g = q.contiguous(), k.contiguous(), v.contiguous(), g.contiguous()
    gq = torch.empty_like(q)
    if T == 0:      # an empty shard: nothing to launch (empty tensors have no address); its reverse-state total is zero
        zeros = (torch.zeros(BH, K, d, device=q.device), torch.zeros(BH, K, device=q.device)) if want_dseg else (None, None)
        return gq, zeros[0], zeros[1], torch.empty(256, dtype=torch.uint8, device=q.device)
    ds = torch.empty(BH, K, d, dtype=torch.float32, device=q.device) if want_dseg else None
    dz = torch.empty(BH, K, dtype=torch.float32, device=q.device) if want_dseg else None
    ws, n = _workspace(T, BH, K, d, q)
    with _guard(q):
        check(_lib.load().rfa_causal_bwd_q(ptr(q), ptr(k), ptr(v), ptr(g), ptr(gq), ptr(s_in), ptr(z_in), ptr(ds),
                                           ptr(dz), ptr(ws), n, T, BH, K, d, stream_of(q)), "rfa_causal_bwd_q")
    return gq, ds, dz, ws


def causal_bwd_kv(q, k, v, g, ds_in, dz_in, ws: Tensor):
    T, BH, K = q.shape
    d = v.shape[-1]
    q, k, v, g = q.contiguous(), k.contiguous(), v.contiguous(), g.contiguous()
    gk, gv = torch.empty_like(k), torch.empty_like(v)
    if T == 0:
        return gk, gv
    with _guard(q):
        check(_lib.load().rfa_causal_bwd_kv(ptr(q), ptr(k), ptr(v), ptr(g), ptr(gk), ptr(gv), ptr(ds_in), ptr(dz_in),
                                            ptr(ws), ws.numel(), T, BH, K, d, stream_of(q)), "rfa_causal_bwd_kv")
    return gk, gv


# --------------------------------------------------------------------------- cross
def cross_state_fwd(phi_k: Tensor, v: Tensor, pad_mask: Optional[Tensor]) -> Tuple[Tensor, Tensor]:
    """phi_k [T,B,H,K], v [T,B,H,d] fp16, pad_mask [B,T] (non-zero = pad) -> s [B,H,K,d], z [B,H,K] fp32."""
    return native().cross_state_fwd(phi_k, v, pad_mask)


def state_total(phi_k: Tensor, v: Tensor) -> Tuple[Tensor, Tensor]:
    """phi_k [T,BH,K], v [T,BH,d] fp16 -> (sum_t k_t v_t^T [BH,K,d], sum_t k_t [BH,K]) fp32, with enough CTAs per
    sequence to fill the GPU when BH is small (partials over runs of tokens, summed here)."""
    require_half(phi_k, v)
    T, BH, K = phi_k.shape
    d = v.shape[-1]
    phi_k, v = phi_k.contiguous(), v.contiguous()
    if T == 0:      # an empty shard contributes nothing
        return torch.zeros(BH, K, d, device=phi_k.device), torch.zeros(BH, K, device=phi_k.device)
    sms = torch.cuda.get_device_properties(phi_k.device).multi_processor_count
    nseg = max(1, min(sms // max(BH, 1), T // 512))
    s = torch.empty(BH, nseg, K, d, dtype=torch.float32, device=phi_k.device)
    z = torch.empty(BH, nseg, K, dtype=torch.float32, device=phi_k.device)
    with _guard(phi_k):
        check(_lib.load().rfa_state_partials(ptr(phi_k), ptr(v), ptr(s), ptr(z), T, BH, K, d, nseg, stream_of(phi_k)),
              "rfa_state_partials")
    return (s[:, 0], z[:, 0]) if nseg == 1 else (s.sum(dim=1), z.sum(dim=1))


def cross_state_bwd(phi_k: Tensor, v: Tensor, pad_mask: Optional[Tensor], d_s: Tensor, d_z: Tensor):
    return native().cross_state_bwd(phi_k, v, pad_mask, d_s, d_z)


def cross_query_fwd(phi_q: Tensor, s: Tensor, z: Tensor) -> Tensor:
    """phi_q [T,B,H,K] fp16, s [B,H,K,d], z [B,H,K] fp32 -> out [T,B,H,d] fp16."""
    return native().cross_query_fwd(phi_q, s, z)


def cross_query_bwd(phi_q: Tensor, s: Tensor, z: Tensor, g: Tensor):
    return native().cross_query_bwd(phi_q, s, z, g)


# --------------------------------------------------------------------------- decode
def decode_step(phi_q: Tensor, phi_k: Tensor, v: Tensor, s: Tensor, z: Tensor, out: Optional[Tensor] = None) -> Tensor:
    """One token, state updated IN PLACE.  phi_q,phi_k [B,H,K], v [B,H,d]; s [B,H,K,d], z [B,H,K]."""
    return native().decode_step(phi_q, phi_k, v, s, z, out)


def decode_step_fused(q: Tensor, k: Tensor, v: Tensor, w: Tensor, scale: float, s: Tensor, z: Tensor,
                      out: Optional[Tensor] = None) -> Tensor:
    """One token from raw q,k [B,H,d]; w [H,D,d] fp32 contiguous; state updated IN PLACE."""
    return native().decode_step_fused(q, k, v, w, scale, s, z, out)


def decode_fused_supported(q: Tensor, w: Tensor) -> bool:
    """Whether one token can go through ``decode_step_fused`` wherever ``feature_map_fwd`` and ``decode_step`` would take it:
    CUDA, fp16 or fp32, head_dim 4 * 2^m and both widths multiples of 8 up to 128 (the feature map's reach)."""
    D, d = w.shape[-2:]
    return (q.is_cuda and q.dtype in (torch.float16, torch.float32) and d in (8, 16, 32, 64, 128) and D % 8 == 0 and D <= 128
            and w.dim() == 3 and w.shape[0] == q.shape[-2] and d == q.shape[-1])


def layer_decode(x: Tensor, q_proj, k_proj, v_proj, out_proj, random_matrices: Tensor, sigma: Optional[Tensor], tau: float,
                 scale: float, s: Optional[Tensor], z: Optional[Tensor], num_heads: int = 0) -> Optional[Tensor]:
    """One token x [1, B, E] through a layer's projections (``nn.Linear`` modules) and its decoding step in three launches, the
    state updated IN PLACE; None, with nothing done, where the tensors are not ones the kernels take (then: module by module), or the
    matrices are not ``num_heads`` (0: any)."""
    return native().layer_decode(x, q_proj.weight, q_proj.bias, k_proj.weight, k_proj.bias, v_proj.weight, v_proj.bias,
                                 out_proj.weight, out_proj.bias, random_matrices, sigma, tau, scale, s, z, num_heads)


def layer_train(x: Tensor, q_proj, k_proj, v_proj, out_proj, random_matrices: Tensor, sigma: Optional[Tensor], tau: float,
                scale: float, pad_mask: Optional[Tensor]) -> Optional[Tensor]:
    """A layer's pass with gradients, x [T, B, E], as five native autograd nodes (the projections, the random matrices, the features, the
    attention, the output projection); pad_mask [B, T] bool.  None, with nothing done, where the tensors are not ones they take."""
    return native().layer_train(x, q_proj.weight, q_proj.bias, k_proj.weight, k_proj.bias, v_proj.weight, v_proj.bias,
                                out_proj.weight, out_proj.bias, random_matrices, sigma, tau, scale, pad_mask)


class CrossDecodeStates:
    """The cross-attention states of all layers of a decoder, gathered once per sequence for ``cross_decode_step``:
    device arrays of pointers to each layer's ``s [B,H,K,d]`` and ``z [B,H,K]`` (fp32, contiguous).  The states are
    referenced, not copied; keep them alive and unchanged while this object is used."""

    def __init__(self, states):
        self.s = [st[0].contiguous() for st in states]
        self.z = [st[1].contiguous() for st in states]
        for t in self.s + self.z:
            if not t.is_cuda or t.dtype != torch.float32:
                raise TypeError("rfa_b200: cross-attention states must be fp32 CUDA tensors")
        self.L = len(self.s)
        B, H, self.K, self.d = self.s[0].shape
        self.BH = B * H
        dev = self.s[0].device
        self.s_ptrs = torch.tensor([t.data_ptr() for t in self.s], dtype=torch.int64, device=dev)
        self.z_ptrs = torch.tensor([t.data_ptr() for t in self.z], dtype=torch.int64, device=dev)


def cross_decode_step(phi_q: Tensor, states: CrossDecodeStates, out: Optional[Tensor] = None) -> Tensor:
    """phi_q [L, B, H, K] (one token's query features for every layer) -> out [L, B, H, d], one launch for all layers."""
    L, B, H, K = phi_q.shape
    assert (L, B * H, K) == (states.L, states.BH, states.K), (phi_q.shape, states.L, states.BH, states.K)
    phi_q = phi_q.contiguous()
    if out is None:
        out = torch.empty(L, B, H, states.d, dtype=phi_q.dtype, device=phi_q.device)
    with _guard(phi_q):
        check(_lib.load().rfa_cross_decode_step(ptr(phi_q), dtype_code(phi_q), ptr(states.s_ptrs), ptr(states.z_ptrs), ptr(out),
                                                L, B * H, K, states.d, stream_of(phi_q)), "rfa_cross_decode_step")
    return out
