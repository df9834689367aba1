"""Products of a few (token, expert) pairs with a row's weights asked for at once (csrc/moe.cu), and the gated norm
with the row in registers, against float64.

Tolerances: an output is rounded to bfloat16 once (2^-9 of itself), gate and up once each before the gated form's product;
float32 sums of up to 4,096 products of order one add 4096^0.5 * 2^-24, nothing beside that: 2^-7 of the largest output."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def product(x, src_div, w, expert, n, act, gated, limit=0.0, slope=1.0):
    """The experts' product of pairs listed in ``expert`` (x, w on the CPU); one column more than asked for, of NaN."""
    from redline_b200.ops import kernels
    E, pairs = w.shape[0], expert.numel()
    i32 = lambda m: torch.zeros(m, dtype=torch.int32, device=DEV)      # noqa: E731
    tiles = kernels.moe_max_tiles(pairs, E)
    order, te, tb, trw, meta = i32(pairs), i32(tiles), i32(tiles), i32(tiles), i32(4)
    kernels.moe_group(expert.to(DEV), pairs, E, order, te, tb, trw, meta)
    out = torch.full((pairs, n + 1), float("nan"), dtype=x.dtype, device=DEV)
    kernels.moe_gemm(x.to(DEV), src_div, w.to(DEV).reshape(-1, x.shape[1]), out[:, :n], order, te, tb, trw, meta, tiles,
                     act=act, few_pairs=True, gated=gated, limit=limit, slope=slope)
    return out.cpu()


@pytest.mark.parametrize("dtype,k", [(torch.bfloat16, 1024), (torch.bfloat16, 2048), (torch.bfloat16, 2056),
                                     (torch.float32, 512), (torch.float32, 1024), (torch.float32, 516)])
@pytest.mark.parametrize("gated,act", [(False, "silu"), (True, "silu"), (True, "clamped_swish")])
@pytest.mark.parametrize("n,shares,top", [(16, [1], 1), (40, [3, 0, 9, 1], 1), (23, [8, 17, 0, 2, 1], 4), (9, [1, 33, 0, 130], 2)])
def test_streamed_products(dtype, k, gated, act, n, shares, top):
    """Against float64, and bit for bit against the kernel for any length: rows and weights with zeros behind them go there,
    and its sums are these in the same order."""
    from redline_b200.ops import kernels
    E, pairs, limit, slope = len(shares), sum(shares), 1.5, 1.25
    g = torch.Generator().manual_seed(k + n)
    x = torch.randn((pairs + top - 1) // top, k, generator=g).to(dtype)
    w = (torch.randn(E, (2 if gated else 1) * n, k, generator=g) * k ** -0.5).to(dtype)
    expert = torch.tensor([e for e, c in enumerate(shares) for _ in range(c)], dtype=torch.int32)[torch.randperm(pairs, generator=g)]
    code = kernels.ACT_CLAMPED_SWISH if act == "clamped_swish" else kernels.ACT_SILU
    got = product(x, top, w, expert, n, code, gated, limit, slope)
    y = torch.einsum("pk,pnk->pn", x[torch.arange(pairs) // top].double(), w[expert.long()].double())
    if gated:
        gate, up = (v.to(dtype).double() for v in y.split(n, dim=1))
        if act == "clamped_swish":
            gate = gate.clamp(max=limit)
            want = gate * torch.sigmoid(slope * gate) * (up.clamp(-limit, limit) + 1.0)
        else:
            want = torch.nn.functional.silu(gate) * up
    else:
        want = torch.nn.functional.silu(y)
    assert got[:, n].isnan().all()                       # (nothing beside the columns)
    # (float32: sums of k products of order k^-0.5, each rounded, and a few roundings more)
    tol = 2.0 ** -7 if dtype == torch.bfloat16 else (8 + k ** 0.5) * 2.0 ** -24
    assert (got[:, :n].double() - want).abs().max() < tol * want.abs().max()
    more = 256 if dtype == torch.bfloat16 else 128
    pad = lambda t: torch.nn.functional.pad(t, (0, 5 * more))          # noqa: E731
    assert torch.equal(product(pad(x), top, pad(w), expert, n, code, gated, limit, slope)[:, :n], got[:, :n])


def test_streamed_products_of_many_features():
    """An expert whose features are more than the grid has blocks for with four of them each."""
    from redline_b200.ops import kernels
    n, k, rows = 4 * 65535 + 8, 2048, 3
    g = torch.Generator(device=DEV).manual_seed(5)
    x = torch.randn(rows, k, generator=g, device=DEV).to(torch.bfloat16)
    w = torch.empty(2 * n, k, dtype=torch.bfloat16, device=DEV).normal_(0.0, k ** -0.5, generator=g)
    out = torch.empty(rows, n, dtype=torch.bfloat16, device=DEV)
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device=DEV)    # noqa: E731
    kernels.moe_gemm(x, 1, w, out, i32(0, 1, 2), i32(0), i32(0), i32(rows), i32(1, 0, 0, 0), 1, act=kernels.ACT_SILU,
                     few_pairs=True, gated=True)
    gate, up = x.float() @ w[n - 32:n].float().t(), x.float() @ w[2 * n - 32:].float().t()
    want = torch.nn.functional.silu(gate.to(torch.bfloat16).float()) * up.to(torch.bfloat16).float()
    assert (out[:, n - 32:].float() - want).abs().max() < 2.0 ** -7 * want.abs().max()


@pytest.mark.parametrize("dtype,w_dtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16),
                                           (torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("rows,n", [(1, 4), (3, 130), (2, 256), (2, 257), (3, 512), (2, 513), (2, 1024), (2, 1025), (8, 2048),
                                    (2, 2049), (5, 4096), (2, 4100)])
def test_gated_norm(dtype, w_dtype, rows, n):
    from redline_b200.ops import kernels
    g = torch.Generator().manual_seed(n)
    o = torch.randn(rows, n, generator=g)
    gate = torch.randn(rows, n + 8, generator=g).to(dtype)
    w = (1.0 + 0.1 * torch.randn(n, generator=g)).to(w_dtype)
    out = torch.empty(rows, n, dtype=dtype, device=DEV)
    kernels.gated_rmsnorm(o.to(DEV), gate.to(DEV)[:, 4:4 + n], w.to(DEV), out, 1e-6)
    od = o.double()
    want = od * torch.rsqrt((od * od).mean(-1, keepdim=True) + 1e-6) * w.double() * torch.sigmoid(gate[:, 4:4 + n].double())
    # (float32: the norm's factor is off by the sum's error, n^0.5 * 2^-24, the rest by a few roundings)
    tol = (8 + n ** 0.5) * 2.0 ** -24 if dtype == torch.float32 else 2.0 ** -8
    assert ((out.cpu().double() - want).abs() <= tol * want.abs().max()).all()
