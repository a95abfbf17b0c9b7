"""Per-head products on the tensor cores and the rotation alone, against 64 bits: one row, a tile of sixteen and one more, K of
one step and of more steps than warps, columns that end inside a block of 64, tails rotated whole, in part and not at
all, rows that are views of wider ones, and only the rows of sequences that bring one; sizes that other kernels keep."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def turned(x, cos_sin, dims):
    half = dims // 2
    c, s = cos_sin[:, None, :, 0], cos_sin[:, None, :, 1]
    a, b = x[..., :half], x[..., half:dims]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., dims:]], -1)


@pytest.mark.parametrize("dtype,out_dtype", [(torch.float32, torch.bfloat16), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("T,H,K,N,tail,dims,pad", [(1, 3, 16, 8, 0, 0, 0), (16, 2, 128, 512, 64, 64, 4), (17, 4, 512, 128, 0, 0, 0),
                                                   (5, 1, 144, 72, 16, 8, 8), (33, 2, 48, 136, 8, 0, 0), (4, 2, 20, 12, 6, 6, 0)])
def test_products_per_head(dtype, out_dtype, T, H, K, N, tail, dims, pad):
    from allpaca_b200 import ops
    g = torch.Generator().manual_seed(T + K)
    wide = torch.randn(T, H * (K + tail) + pad, generator=g).to(dtype)
    x = wide[:, :H * (K + tail)]
    w = (torch.randn(H, K, N, generator=g) * K ** -0.5).to(torch.bfloat16)
    cs = torch.randn(T, dims // 2, 2, generator=g)
    x3 = x.double().view(T, H, K + tail)
    want = torch.cat([torch.einsum("thk,hkn->thn", x3[..., :K], w.double()), turned(x3[..., K:], cs.double(), dims)], -1)
    lens = [3, 1, 1, 2] + [1] * max(0, T - 7) if T >= 7 else [1] * T
    start = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device=DEV)
    single = torch.cat([torch.full((n,), n == 1) for n in lens])
    for singles in (None, start):
        out = torch.zeros(T, H * (N + tail), dtype=out_dtype, device=DEV)
        ops.head_project(wide.to(DEV)[:, :H * (K + tail)], w.to(DEV), out, H, tail=tail, tail_dims=dims,
                         cos_sin=cs.to(DEV) if dims else None, singles=singles, num_seqs=len(lens))
        rows = torch.ones(T, dtype=torch.bool) if singles is None else single
        got = out.double().cpu().view(T, H, N + tail)
        # bfloat16 stores seven bits: half a unit in the last place is at most 2^-8; 32-bit sums of unit size before
        assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + 2e-6)[rows].all())


@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,H,K,tail,dims", [(1, 1, 4, 8, 8), (37, 3, 128, 64, 64), (9, 2, 24, 32, 16), (6, 2, 64, 12, 0), (5, 2, 10, 6, 6)])
def test_rotation_alone(out_dtype, T, H, K, tail, dims):
    from allpaca_b200 import ops
    g = torch.Generator().manual_seed(T + K)
    x, cs = torch.randn(T, H * (K + tail), generator=g), torch.randn(T, dims // 2, 2, generator=g)
    x3 = x.double().view(T, H, K + tail)
    want = torch.cat([x3[..., :K], turned(x3[..., K:], cs.double(), dims)], -1)
    out = torch.zeros(T, H * (K + tail), dtype=out_dtype, device=DEV)
    ops.head_project(x.to(DEV), None, out, H, tail=tail, tail_dims=dims, cos_sin=cs.to(DEV) if dims else None)
    tol = 2.0 ** -8 if out_dtype == torch.bfloat16 else 2.0 ** -23
    assert bool(((out.double().cpu().view(T, H, -1) - want).abs() <= tol * want.abs() + 1e-6).all())


@pytest.mark.parametrize("K", [16, 272])
def test_inputs_that_bfloat16_does_not_hold(K):
    """32-bit inputs beyond the largest bfloat16 number count as what they are, infinite ones stay infinite, NaN stays NaN, and
    each only in its own row."""
    from allpaca_b200 import ops
    most, inf, nan = torch.finfo(torch.float32).max, float("inf"), float("nan")
    special = [most, -most, inf, -inf, nan, 1.0, 2.0 ** -140]
    x = torch.zeros(len(special), K)
    x[:, K - 3] = torch.tensor(special)
    x[:, 1] = torch.tensor([0.0, 0.0, 1.0, 1.0, 1.0, 1.0, 0.0])
    w = torch.full((1, K, 8), 0.0625).to(torch.bfloat16)
    out = torch.empty(len(special), 8, dtype=torch.bfloat16, device=DEV)
    ops.head_project(x.to(DEV), w.to(DEV), out, 1)
    want = (x.double().sum(1) * 0.0625).to(torch.bfloat16)[:, None].expand(-1, 8)
    assert torch.equal(torch.nan_to_num(out.cpu(), nan=7.0), torch.nan_to_num(want, nan=7.0)), (out[:, 0], want[:, 0])
