"""The chunked kernels of the geometries other than K = 128, d = 64 (csrc/generic_split.cu, generic_mma.cu) against the PyTorch twins in fp64.

Results are fp16, so that a correct one is within half a unit in the last place of the fp64 value: 2^-11 = 4.9e-4 relative at
worst, 2.9e-4 in the 2-norm of evenly spread significands; the gate is 4e-4 in the 2-norm.  Below fp16's smallest normal number
that is an absolute error instead, and gq of a first token whose denominator is out of the clamp is exactly zero, two
terms of about 0.05 that cancel in 22 bits: three spacings of 6e-8 are allowed to every element.  The carried state is fp32 sums
of exact products, a chunk's from zero: 2e-6."""
import ctypes

import pytest
import torch

from rfa_b200.rfa import RFA

pytestmark = pytest.mark.gpu

GEOMETRIES = [(64, 32), (96, 40), (128, 128), (256, 128), (72, 24), (8, 8), (512, 64)]      # the kernels they reach have chunks of 64 and 32 tokens


def inputs(T, BH, K, d, seed):
    gen = torch.Generator().manual_seed(seed)
    q, k = (torch.rand(T, BH, K, generator=gen) * 0.3 - 0.1 for _ in range(2))
    return [t.half() for t in (q, k, torch.randn(T, BH, d, generator=gen), torch.randn(T, BH, d, generator=gen))]


def rel(a, b, spacing=0.0):
    return float((a.detach().cpu().double() - b).norm() - 3 * spacing * b.numel() ** 0.5) / max(float(b.norm()), 1e-30)


@pytest.mark.parametrize("K,d", GEOMETRIES)
@pytest.mark.parametrize("T,BH", [(1, 1), (15, 3), (64, 2), (65, 2), (131, 2), (700, 2)])
def test_chunked_kernels_against_fp64(dev, K, d, T, BH):
    q, k, v, g = inputs(T, BH, K, d, K + d + T)
    want = RFA.forward_torch(*(t.double() for t in (q, k, v)))
    grads = RFA.backward_torch(*(t.double() for t in (q, k, v, g)))
    leaves = [t.to(dev).requires_grad_() for t in (q, k, v)]
    out = RFA.apply(*leaves)
    out.backward(g.to(dev))
    assert rel(out, want, 2.0 ** -24) < 4e-4
    for name, leaf, ref in zip("qkv", leaves, grads):
        assert rel(leaf.grad, ref, 2.0 ** -24) < 4e-4, name


@pytest.mark.parametrize("K,d", [(64, 32), (96, 40), (256, 128)])
@pytest.mark.parametrize("T", [40, 700])
def test_state_out_and_a_forward_without_workspace(dev, K, d, T):
    from rfa_b200 import _lib, ops
    q, k, v, _ = (t.to(dev) for t in inputs(T, 2, K, d, 5))
    out, s, z = ops.causal_fwd(q, k, v, return_state=True)
    kd, vd = k.cpu().double(), v.cpu().double()
    assert rel(s, torch.einsum("tbk,tbd->bkd", kd, vd)) < 2e-6 and rel(z, kd.sum(0)) < 2e-6
    bare = torch.empty_like(out)                       # no workspace: sequences stay whole
    assert _lib.load().rfa_causal_fwd(*(t.data_ptr() for t in (q, k, v, bare)), None, None, None, None, None,
                                      ctypes.c_size_t(0), T, 2, K, d, _lib.stream_of(q)) == 0
    assert rel(bare, out.cpu().double()) < 4e-4


@pytest.mark.parametrize("K,d,T", [(64, 32, 130), (256, 128, 130), (256, 128, 700), (128, 128, 300)])
def test_results_are_rounded_from_fp32_sums(dev, K, d, T):
    """How many fp16 results are not the fp64 value's rounding shows the error in front of that rounding, which the 2-norm hides.  With
    a relative error of e the share is about 2^12 e: 2e-3 (3e-3 for gq, whose terms cancel) allows 8 (12) units of fp32's last place; chains of
    truncating products had 0.5 % and more in out and gv."""
    gen = torch.Generator("cuda").manual_seed(K + T)
    x = torch.randn(2, T, 8, K // 2, generator=gen, device=dev, dtype=torch.float64)
    w = torch.randn(K // 2, K // 2, generator=gen, device=dev, dtype=torch.float64)
    u = (x / x.norm(dim=-1, keepdim=True)) @ w
    q, k = (0.1 * torch.cat([u.sin(), u.cos()], dim=-1)).half()
    v, g = torch.randn(2, T, 8, d, generator=gen, device=dev).half()
    wide = [t.double() for t in (q, k, v, g)]
    want = (RFA.forward_torch(*wide[:3]), *RFA.backward_torch(*wide))
    leaves = [t.clone().requires_grad_() for t in (q, k, v)]
    out = RFA.apply(*leaves)
    out.backward(g)
    share = [float((a != b.half()).double().mean()) for a, b in zip([out, *(t.grad for t in leaves)], want)]
    assert all(s < gate for s, gate in zip(share, (2e-3, 3e-3, 2e-3, 2e-3))), share


@pytest.mark.parametrize("K,d", [(64, 32), (96, 40), (128, 128)])
@pytest.mark.parametrize("T", [16, 45, 300])
def test_the_reverse_state_is_an_fp32_sum(dev, K, d, T):
    """Sum of q (x) (g / den): each term rounded twice (1 / den and its product with g, 2^-25 in the mean each), then fp32 sums of 8, and of
    those: 9e-8 in the 2-norm at 16 tokens, and the square root of the number of sums more."""
    from rfa_b200 import ops
    q, k, v, g = (t.to(dev) for t in inputs(T, 8, K, d, T))
    _, ds, _, _ = ops.causal_bwd_q(q, k, v, g, None, None, True)
    Q, Kd, G = (t.double() for t in (q, k, g))
    inv = 1 / (Q * torch.cumsum(Kd, 0)).sum(-1, keepdim=True).clamp_min(1)
    want = torch.einsum("tbk,tbd->bkd", Q, G * inv)
    assert float((ds - want).norm() / want.norm()) < 9e-8 * max(1.0, T / 16) ** 0.5


@pytest.mark.parametrize("which", [0, 1, 2])
def test_no_token_sees_a_later_non_finite_one(dev, which):
    """A chunk's masked products multiply zeros with the tokens they mask; an infinity there must not reach earlier outputs."""
    T, cut, K, d = 60, 37, 64, 32
    ins = inputs(T, 2, K, d, 9)
    clean = RFA.forward_cuda(*(t.to(dev) for t in ins[:3]))
    ins[which][cut, :, 3] = float("inf")
    q, k, v, g = (t.to(dev) for t in ins)
    out = RFA.forward_cuda(q, k, v)
    assert torch.isfinite(out[:cut]).all()
    # element by element where an infinity of v shares the chunk: fp32 sums in another order, a neighbouring fp16 number at most
    assert ((out[:cut] - clean[:cut]).abs() <= 2.0 ** -10 * clean[:cut].abs() + 1e-6).all()
    gq, _, _ = RFA.backward_cuda(q, k, v, g)
    assert torch.isfinite(gq[:cut]).all()
    if which == 0:       # q of a token reaches the key gradients of itself and of earlier tokens only
        _, gk, gv = RFA.backward_cuda(q, k, v, g)
        assert torch.isfinite(gk[cut + 1:]).all() and torch.isfinite(gv[cut + 1:]).all()


@pytest.mark.parametrize("K,d", [(64, 32), (96, 40), (72, 24)])
@pytest.mark.parametrize("T", [33, 200])
def test_columns_and_tokens_of_very_different_magnitude(dev, K, d, T):
    """A split operand has one power of two per 16 x 16 block: columns of v and g from 2^-9 to 2^9 and tokens of q and k from 2^-8 to 1
    share blocks, and every column of out and gv (a product with those columns alone) still has fp16's rounding error and no more."""
    q, k, v, g = inputs(T, 2, K, d, T)
    gen = torch.Generator().manual_seed(K)
    tokens = 2.0 ** torch.randint(-8, 1, (T, 1, 1), generator=gen)
    columns = 2.0 ** torch.linspace(-9, 9, d).round()
    q, k, v, g = (q * tokens).half(), (k * tokens.flip(0)).half(), (v * columns).half(), (g * columns.flip(0)).half()
    want = RFA.forward_torch(*(t.double() for t in (q, k, v)))
    gq, gk, gv = RFA.backward_torch(*(t.double() for t in (q, k, v, g)))
    leaves = [t.to(dev).requires_grad_() for t in (q, k, v)]
    out = RFA.apply(*leaves)
    out.backward(g.to(dev))
    for j in range(d):
        assert rel(out[..., j], want[..., j], 2.0 ** -24) < 4e-4 and rel(leaves[2].grad[..., j], gv[..., j], 2.0 ** -24) < 4e-4, j
    assert rel(leaves[0].grad, gq, 2.0 ** -24) < 4e-4 and rel(leaves[1].grad, gk, 2.0 ** -24) < 4e-4


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("rows,H,D,d", [(1, 2, 64, 64), (63, 2, 32, 32), (130, 3, 48, 40), (65, 2, 128, 128), (500, 1, 8, 128), (90, 2, 72, 8)])
def test_feature_map_of_any_width_against_fp64(dev, dtype, rows, H, D, d):
    """csrc/feature_map.cu: 64-row tiles, column blocks of 64, with remainders of both.  fp32: sums of d (D) products, 4e-7 per
    result and 2e-6 for the gradient of the matrices (a sum over rows); fp16: the results' rounding, 4e-4."""
    from rfa_b200.utils import random_project
    gen = torch.Generator().manual_seed(rows + D)
    x, w = torch.randn(rows, 1, H, d, generator=gen).to(dtype), torch.randn(H, D, d, generator=gen)
    g = torch.randn(rows, 1, H, 2 * D, generator=gen).to(dtype)
    xd, wd = x.double().requires_grad_(), w.double().requires_grad_()
    u = torch.einsum("tbhd,hkd->tbhk", xd / (xd.norm(dim=-1, keepdim=True) + 1e-3), wd)
    ref = 0.1 * torch.cat([u.sin(), u.cos()], dim=-1)
    ref.backward(g.double())
    xg, wg = x.to(dev).requires_grad_(), w.to(dev).requires_grad_()
    phi = random_project(x=xg, random_matrices=wg)
    phi.backward(g.to(dev))
    half = dtype == torch.float16
    tc = half and (D, d) == (64, 64)              # the tensor-core kernel, with fp16 operands
    assert rel(phi, ref.detach()) < (2e-3 if tc else 4e-4 if half else 4e-7)
    assert rel(xg.grad, xd.grad) < (2e-3 if tc else 4e-4 if half else 1e-6)
    assert rel(wg.grad, wd.grad) < (2e-3 if tc else 2e-6)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("D,d", [(64, 64), (32, 32), (48, 40), (8, 64), (56, 8)])
@pytest.mark.parametrize("rows,H", [(197 * 16, 3), (197 * 16 + 1, 3), (131, 148), (16, 1000), (9601, 1)])
def test_feature_map_on_split_operands(dev, dtype, rows, H, D, d):
    """csrc/feature_map_mma.cu from more than four groups of 16 rows to an SM on (the first case has one too few): ragged groups,
    shares of unequal length, CTAs with one group, widths that end inside a block of 16 or 32.  Gates as for the other fp32 kernels; a row
    of zeros, one of 1e4 and one with an infinity, whose results are NaN and touch no other row."""
    if dtype == torch.float16 and (D, d) == (64, 64):
        pytest.skip("the tensor-core kernel for fp16 operands")
    from rfa_b200 import ops
    gen = torch.Generator(dev).manual_seed(rows + D)
    x, g = torch.randn(rows, H, d, generator=gen, device=dev).to(dtype), torch.randn(rows, H, 2 * D, generator=gen, device=dev).to(dtype)
    w = torch.randn(H, D, d, generator=gen, device=dev) * 2
    x[3], x[5] = 0, x[5] * 1e4
    mask = torch.rand(rows, generator=gen, device=dev) < 0.2
    mask[3] = mask[5] = False
    xd, wd = x.double().requires_grad_(), w.double().requires_grad_()
    u = torch.einsum("thd,hkd->thk", xd / (xd.norm(dim=-1, keepdim=True) + 1e-3), wd)
    ref = 0.1 * torch.cat([u.sin(), u.cos()], dim=-1) * ~mask[:, None, None]
    ref.backward(g.double())
    ref_gx = torch.nan_to_num(xd.grad)                       # the norm's gradient at a row of zeros
    phi = ops.feature_map_fwd(x, w, 0.1, row_mask=mask)
    gx, gw = ops.feature_map_bwd(x, w, g, 0.1, True, row_mask=mask)
    err = lambda a, b: float((a.double() - b).norm() / b.norm())
    half = dtype == torch.float16
    keep = [i for i in range(rows) if i != 3]
    assert err(phi, ref.detach()) < (4e-4 if half else 4e-7)
    assert err(gx[keep], ref_gx[keep]) < (4e-4 if half else 1e-6) and err(gw, wd.grad) < 2e-6
    assert torch.equal(ops.feature_map_bwd(x, w, g, 0.1, False, row_mask=mask)[0], gx)
    x[7, 0, 0] = float("inf")
    bad = ops.feature_map_fwd(x, w, 0.1, row_mask=mask)
    assert not torch.isfinite(bad[7, 0]).any() or bool(mask[7])
    assert torch.equal(bad[:7], phi[:7]) and torch.equal(bad[8:], phi[8:])
    g[9, 0, 0] = float("inf")
    mask[9] = False
    x[7, 0, 0] = 0
    bx, _ = ops.feature_map_bwd(x, w, g, 0.1, True, row_mask=mask)
    assert not torch.isfinite(bx[9, 0]).any() and torch.equal(bx[16:], gx[16:])
    assert torch.isfinite(bx[:9]).all() and torch.isfinite(bx[10:16]).all()
    assert err(bx[10:16], ref_gx[10:16]) < (4e-4 if half else 1e-6)      # rows that share its 16 are summed element by element


def test_sines_of_every_size(dev):
    """csrc/trig.cuh through the feature map: one product a column, so that u is w to a rounding.  2e-7 absolute up to 8000, where the reduction
    is its own, and beyond, where it is the library's."""
    from rfa_b200 import ops
    n = 4 * 148 * 16 + 16
    w = torch.zeros(1, 64, 8, device=dev)
    w[0, :, 0] = torch.cat([torch.linspace(-10, 10, 32, device=dev), 10 ** torch.linspace(1, 6, 32, device=dev)])
    x = torch.zeros(n, 1, 8, device=dev)
    x[:, 0, 0] = 1e4 * (1 + torch.rand(n, device=dev))
    for rows in (n, 64):
        phi = ops.feature_map_fwd(x[:rows], w, 1.0)[:, 0].double()
        u = (x[:rows, 0, :1].double() / (x[:rows, 0, :1].double() + 1e-3)) * w[0, :, 0].double()
        bound = 2e-7 + 2.0 ** -21 * u.abs()               # u itself is rounded: 22 bits of x and of w
        assert ((phi[:, :64] - u.sin()).abs() <= bound).all() and ((phi[:, 64:] - u.cos()).abs() <= bound).all()


@pytest.mark.parametrize("D,d", [(32, 32), (72, 96), (128, 128)])
@pytest.mark.parametrize("rows,H", [(33, 147), (33, 148), (148 * 64 - 64, 1), (148 * 64 - 63, 1)])
def test_feature_map_backward_in_tiles_of_32_and_64(dev, rows, H, D, d):
    """One SM to a tile of 64 rows is where the backward goes from tiles of 32 to tiles of 64.  fp32 as above; the gradient of the matrices
    is a sum over up to 9409 rows, taken 32 or 64 at a time: 2e-6."""
    from rfa_b200 import ops
    gen = torch.Generator(dev).manual_seed(rows + H)
    x, g = torch.randn(rows, H, d, generator=gen, device=dev), torch.randn(rows, H, 2 * D, generator=gen, device=dev)
    w = torch.randn(H, D, d, generator=gen, device=dev)
    mask = torch.rand(rows, generator=gen, device=dev) < 0.2
    xd, wd = x.double().requires_grad_(), w.double().requires_grad_()
    u = torch.einsum("thd,hkd->thk", xd / (xd.norm(dim=-1, keepdim=True) + 1e-3), wd)
    (0.1 * torch.cat([u.sin(), u.cos()], dim=-1)).backward(g.double() * ~mask[:, None, None])
    gx, gw = ops.feature_map_bwd(x, w, g, 0.1, True, row_mask=mask)
    assert float((gx - xd.grad).norm() / xd.grad.norm()) < 1e-6
    assert float((gw - wd.grad).norm() / wd.grad.norm()) < 2e-6
    assert torch.equal(ops.feature_map_bwd(x, w, g, 0.1, False, row_mask=mask)[0], gx)


@pytest.mark.parametrize("D,d", [(64, 64), (32, 32), (48, 40)])
@pytest.mark.parametrize("step", [1, 3, -3])
def test_feature_map_backward_of_faded_rows(dev, D, d, step):
    """csrc/feature_map_mma.cu: the gradients of 16 neighbouring rows fall by 2^step from row to row, to 2^-45 of the largest; each row of g_x has the
    error that a row by itself has (22 bits of W and of g_u, fp32 sums: 3e-7; 1e-6 allowed), and g_W that of a sum over all rows."""
    from rfa_b200 import ops
    gen = torch.Generator(dev).manual_seed(D + step)
    rows, H = 41, 250
    x, w = torch.randn(rows, H, d, generator=gen, device=dev), torch.randn(H, D, d, generator=gen, device=dev)
    g = torch.randn(rows, H, 2 * D, generator=gen, device=dev)
    g *= 2.0 ** -(torch.arange(rows, device=dev) % 16 * step % 48).float()[:, None, None]
    g[20] = 0
    xd, wd = x.double().requires_grad_(), w.double().requires_grad_()
    u = torch.einsum("thd,hkd->thk", xd / (xd.norm(dim=-1, keepdim=True) + 1e-3), wd)
    (0.1 * torch.cat([u.sin(), u.cos()], dim=-1)).backward(g.double())
    gx, gw = ops.feature_map_bwd(x, w, g, 0.1, True)
    assert (gx[20] == 0).all()
    keep = [i for i in range(rows) if i != 20]
    per_row = (gx.double() - xd.grad).norm(dim=(1, 2))[keep] / xd.grad.norm(dim=(1, 2))[keep]
    assert float(per_row.max()) < 1e-6, per_row
    assert float((gw - wd.grad).norm() / wd.grad.norm()) < 2e-6
    assert torch.equal(ops.feature_map_bwd(x, w, g, 0.1, False)[0], gx)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("D,d", [(64, 64), (32, 32), (48, 40), (64, 24), (56, 8)])
@pytest.mark.parametrize("rows,H", [(3 * 16, 198), (8 * 16 + 3, 132), (222 * 16, 8), (395 * 16 + 1, 3), (1184 * 16 + 5, 1), (33 * 16, 297), (5 * 16, 297), (16, 1000)])
def test_feature_map_around_its_lines(dev, dtype, rows, H, D, d):
    """Both sides of the lines in csrc/feature_map.cu between its kernels and those of feature_map_mma.cu: 4, 8 or 12 groups of 16 rows to an SM,
    more heads than CTAs.  The gates are those of either."""
    test_feature_map_on_split_operands(dev, dtype, rows, H, D, d)


# (K, d, tokens, heads) -> which kernels, chunk, CTAs on an SM: each that the dispatch can reach, with several chunks after one another where it makes any
REACHED = [(8, 8, 131, 150),        # generic_split.cu: 64, three
           (64, 32, 131, 150),      # 64, two
           (64, 96, 131, 148),      # 64, one
           (64, 64, 131, 150),      # 32, three
           (64, 96, 131, 150),      # 32, two
           (128, 128, 131, 150),    # 32, one
           (192, 48, 131, 2),       # 16, two
           (160, 128, 131, 20),     # 16, one, in segments
           (160, 128, 112, 148),    # 16, one, whole
           (160, 128, 128, 148),    # generic_mma.cu from here on: 64, one stage of tiles
           (192, 128, 131, 150),
           (896, 8, 131, 40),       # 32, one stage
           (160, 176, 131, 40),     # 32, two stages
           (208, 208, 70, 40),      # 16, one stage
           (224, 184, 70, 40)]      # 16, two stages


@pytest.mark.parametrize("K,d,T,BH", REACHED)
def test_every_chunked_kernel_against_fp64(dev, K, d, T, BH):
    from rfa_b200 import _lib
    q, k, v, g = (t.to(dev) for t in inputs(T, BH, K, d, K + d + T))
    want = RFA.forward_torch(*(t.double() for t in (q, k, v))).cpu()
    grads = [t.cpu() for t in RFA.backward_torch(*(t.double() for t in (q, k, v, g)))]
    leaves = [t.clone().requires_grad_() for t in (q, k, v)]
    out = RFA.apply(*leaves)
    out.backward(g)
    assert rel(out, want, 2.0 ** -24) < 4e-4
    for name, leaf, ref in zip("qkv", leaves, grads):
        assert rel(leaf.grad, ref, 2.0 ** -24) < 4e-4, name
    bare = torch.empty_like(out)                       # no workspace: sequences stay whole
    assert _lib.load().rfa_causal_fwd(*(t.data_ptr() for t in (q, k, v, bare)), None, None, None, None, None,
                                      ctypes.c_size_t(0), T, BH, K, d, _lib.stream_of(q)) == 0
    assert rel(bare, want, 2.0 ** -24) < 4e-4


@pytest.mark.parametrize("rows", [720, 16])
def test_sines_of_exact_arguments(dev, rows):
    """csrc/trig.cuh (720 rows of 40 heads) and CUDA's sines (16 rows) where u is w to the bit: the normalised entry is 1, values of one octave share a block
    of 16, and 22 significant bits survive the split.  From 2^-6 to 2^20, on both sides of where the reduction becomes the library's,
    every other one next to a multiple of pi / 2.  1.6 units of fp32's last place at 1 and the library's 2: 1.2e-7."""
    from rfa_b200 import ops
    H, D, d = 40, 64, 8
    gen = torch.Generator().manual_seed(rows)
    lowest = 2.0 ** torch.linspace(-6, 19, H * D // 16).double()
    u = (lowest[:, None] * (1 + torch.rand(len(lowest), 16, generator=gen, dtype=torch.double))).view(H, D)
    near = (u[:, ::2] / (torch.pi / 2)).round().clamp_min(1) * (torch.pi / 2)
    u[:, ::2] = torch.where(u[:, ::2] > 1.6, near, u[:, ::2])
    mantissa, exponent = torch.frexp(u)
    u = torch.ldexp((mantissa * 2 ** 22).round() / 2 ** 22, exponent)
    w = torch.zeros(H, D, d, dtype=torch.double)
    w[:, :, 0] = u
    x = torch.zeros(rows, H, d, device=dev)
    x[:, :, 0] = 2.0 ** 40
    phi = ops.feature_map_fwd(x, w.float().to(dev), 1.0).cpu().double()
    assert ((phi[..., :D] - u.sin()).abs() <= 1.2e-7).all() and ((phi[..., D:] - u.cos()).abs() <= 1.2e-7).all()


@pytest.mark.parametrize("K,d", [(64, 32), (96, 40), (128, 128), (160, 128)])
@pytest.mark.parametrize("T", [16, 45])
def test_a_token_beside_a_much_larger_one(dev, K, d, T):
    """Queries of 2^15 and of 2^-14 in one block of 16: each output is divided by its own token's denominator, so that the small one's (which the clamp
    leaves at 1) must not have the error of the large one's weights.  Every token has fp16's rounding error and no more."""
    gen = torch.Generator().manual_seed(K + T)
    q, k = (torch.rand(T, 3, K, generator=gen) * 0.3 + 0.02 for _ in range(2))
    v = torch.randn(T, 3, d, generator=gen) * 1024
    q = q * torch.where(torch.arange(T) % 2 == 0, 2.0 ** 15, 2.0 ** -14)[:, None, None]
    q, k, v = q.half(), k.half(), v.half()
    want = RFA.forward_torch(*(t.double() for t in (q, k, v)))
    out = RFA.forward_cuda(*(t.to(dev) for t in (q, k, v)))
    for t in range(T):
        assert rel(out[t], want[t], 2.0 ** -24) < 4e-4, t


@pytest.mark.parametrize("K,d", [(64, 32), (96, 40), (128, 128), (160, 128)])
@pytest.mark.parametrize("T", [16, 45, 300])
def test_a_column_of_the_reverse_state_beside_a_much_larger_one(dev, K, d, T):
    """As above for every column by itself, with gradients whose columns fall from 2^8 to 2^-14 within a block."""
    from rfa_b200 import ops
    q, k, v, g = inputs(T, 8, K, d, T)
    g = (g * 2.0 ** torch.linspace(8, -14, 16).round().repeat(d // 16 + 1)[:d]).half()
    q, k, v, g = (t.to(dev) for t in (q, k, v, g))
    _, ds, _, _ = ops.causal_bwd_q(q, k, v, g, None, None, True)
    Q, Kd, G = (t.double() for t in (q, k, g))
    inv = 1 / (Q * torch.cumsum(Kd, 0)).sum(-1, keepdim=True).clamp_min(1)
    want = torch.einsum("tbk,tbd->bkd", Q, G * inv)
    error = (ds - want).norm(dim=(0, 1)) / want.norm(dim=(0, 1))
    assert float(error.max()) < 1.2e-7 * max(1.0, T / 16) ** 0.5, error


@pytest.mark.parametrize("K,d,T,B,H", [(64, 96, 200, 2, 2), (192, 48, 200, 2, 2), (192, 48, 16, 3, 1), (160, 128, 64, 2, 2), (160, 128, 300, 2, 2), (64, 64, 150, 50, 3)])
def test_state_reductions_alone(dev, K, d, T, B, H):
    """Sequences that are not cut have a choice of chunks of their own: fp32 sums of exact products, 2e-6, padded keys left out."""
    from rfa_b200 import ops
    gen = torch.Generator(dev).manual_seed(K + T)
    k, v = torch.randn(T, B, H, K, generator=gen, device=dev).half(), torch.randn(T, B, H, d, generator=gen, device=dev).half()
    pad = torch.rand(B, T, generator=gen, device=dev) < 0.3
    s, z = ops.cross_state_fwd(k, v, pad)
    kd = k.double() * ~pad.t()[:, :, None, None]
    assert rel(s, torch.einsum("tbhk,tbhd->bhkd", kd, v.double()).cpu()) < 2e-6 and rel(z, kd.sum(0).cpu()) < 2e-6
