"""top_k by the threads' largest logits first: rows on which that list is short, too long, or not there, against a 64-bit draw."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("V", [5000, 32000, 128256])
@pytest.mark.parametrize("rows", [6, 30])
@pytest.mark.parametrize("k", [1, 40, 2047, 2048])
def test_top_k(V, rows, k):
    from allpaca_b200 import ops
    g = torch.Generator().manual_seed(V + k)
    l = torch.randn(rows, V, generator=g) * 3.0
    l[0] = torch.linspace(5.0, -5.0, V)                     # the largest side by side in a few threads
    l[1] = torch.randint(0, 3, (V,), generator=g).float()   # more equals at the cut than any list holds
    l[2, torch.randperm(V, generator=g)[:-100]] = -torch.inf     # fewer than most k
    l[3] = (torch.randn(V, generator=g) * 60.0).clamp(-400.0, 400.0)    # some further below than exp reaches
    l[4, ::2] = torch.nan
    l[5] = 1.0
    u = torch.rand(rows, generator=g)
    out = torch.full((rows,), -1, dtype=torch.int32, device=DEV)
    temp = torch.ones(rows, device=DEV)
    ops.sample(l.to(DEV), temp, torch.full((rows,), k, dtype=torch.int32, device=DEV), torch.ones(rows, device=DEV), u.to(DEV), out)
    for r in range(rows):
        x = torch.nan_to_num(l[r], nan=-torch.inf)
        ids = torch.sort(x, descending=True, stable=True).indices[:k]
        ids = ids[x[ids] > -torch.inf].sort().values
        w = torch.exp((x[ids] - x.max()).double())
        run = w.cumsum(0)
        at = (ids == int(out[r])).nonzero()
        assert at.numel() == 1, (r, int(out[r]))
        i, want = int(at), float(u[r]) * float(run[-1])
        slack = float(run[-1]) * 2048 * 2.0 ** -24           # up to 2048 additions in 32 bits
        assert float(run[i] - w[i]) - slack <= want <= float(run[i]) + slack
