"""The gated norm over parts wide enough for a CTA of their own: the narrowest and the widest such part, a width that ends
inside a thread's runs, parts one beside the other, and rows whose stride or width leaves them to the general kernel."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,inner,parts,pad", [(3, 256, 1, 0), (5, 1300, 1, 4), (2, 4096, 1, 0), (9, 3 * 1028, 3, 8),
                                               (4, 4100, 1, 0), (4, 512, 1, 3)])
def test_gate_then_norm_in_wide_parts(dtype, T, inner, parts, pad):
    from allpaca_b200 import ops
    g = torch.Generator().manual_seed(T)
    y, z = torch.randn(T, inner, generator=g), torch.randn(T, inner + pad, generator=g)
    w = (1 + 0.2 * torch.randn(inner, generator=g)).to(dtype)
    v = (y.double() * torch.nn.functional.silu(z[:, :inner].double())).view(T, parts, -1)
    want = (v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5)).reshape(T, inner) * w.double()
    out = torch.empty(T, inner, dtype=dtype, device=DEV)
    ops.gated_group_rmsnorm(y.to(DEV), z.to(DEV)[:, :inner], w.to(DEV), 1e-5, out, parts)
    # bfloat16 stores seven bits: half a unit in the last place is at most 2^-8 of the value; 32-bit: a few roundings of the value and of a sum of squares
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-6
    assert bool(((out.double().cpu() - want).abs() <= tol * want.abs() + 1e-7).all())
