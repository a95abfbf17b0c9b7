"""The first maximum where a cluster passes a row: the shortest vocabulary that does, tails of one to three, ties across runs and
CTAs, rows of -inf and NaN, the last number of rows that does and the first that does not; and draws of so many rows that two share
an SM give what the same rows give alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("R,V", [(1, 8188), (1, 16384), (1, 16385), (3, 16387), (37, 20000), (38, 20000), (2, 128256), (4, 40001),
                                 (3, 40002)])
def test_first_maximum(R, V):
    from allpaca_b200 import ops
    g = torch.Generator().manual_seed(V + R)
    l = torch.randn(R, V, generator=g)
    l[0, [V - 1, V // 2, 5]] = 9.0                        # the lowest of equals
    if R > 1:
        l[1] = -torch.inf
        l[1, V - 1] = -3.0
    if R > 2:
        l[2] = -torch.inf
        l[2, 7] = torch.nan
    out = torch.full((R,), -1, dtype=torch.int32, device=DEV)
    ops.argmax(l.to(DEV), out)
    want = torch.nan_to_num(l, nan=-torch.inf).argmax(1)
    assert out[0] == 5 and torch.equal(out.cpu().long(), want) or (R > 2 and out[2] == 0)
    want[2 if R > 2 else 0] = 0 if R > 2 else 5
    assert torch.equal(out.cpu().long(), want)
    # rows that begin on 16-byte boundaries whatever their length, with larger numbers behind their ends
    wide = torch.full((R, (V + 3) // 4 * 4), 99.0)
    wide[:, :V] = l
    wide, out = wide.to(DEV), torch.full_like(out, -1)
    ops.call(ops.core(), "ap_argmax", wide.data_ptr(), wide.shape[1], R, V, out.data_ptr(), 0, ops.stream_handle())
    assert torch.equal(out.cpu().long(), want)


@pytest.mark.parametrize("V", [3000, 30000, 60000, 100000])
def test_draws_of_many_rows(V):
    from allpaca_b200 import ops
    g = torch.Generator().manual_seed(V)
    R = 24
    l = (2.0 * torch.randn(R, V, generator=g)).to(DEV)
    t, p, u = 0.5 + torch.rand(R, generator=g), 0.5 + 0.5 * torch.rand(R, generator=g), torch.rand(R, generator=g)
    k = torch.randint(0, 3000, (R,), generator=g, dtype=torch.int32)
    t[3], k[5], p[5] = 0.0, 0, 1.0
    t, k, p, u = (x.to(DEV) for x in (t, k, p, u))
    many, one = (torch.empty(R, dtype=torch.int32, device=DEV) for _ in range(2))
    ops.sample(l, t, k, p, u, many)
    for r in range(R):
        ops.sample(l[r:r + 1].contiguous(), t[r:r + 1], k[r:r + 1], p[r:r + 1], u[r:r + 1], one[r:r + 1])
    assert torch.equal(many, one)
