"""Routing, grouping and adding up at the sizes where they change their ways: one row, the last step of single rows and the first
of four rows to a CTA, outputs that end inside a warp's block of experts and inside 32, 64, 128 and 256, K beyond what is
asked for ahead and inside a run, pairs that fill no warp and many, experts nobody chose, runs of columns and odd widths."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def i32(*shape):
    return torch.empty(*shape, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("T,E,K,top,groups,keep", [(1, 5, 264, 2, 1, 1), (3, 16, 2048, 4, 4, 2), (511, 33, 4104, 3, 1, 1),
                                                   (512, 16, 512, 4, 1, 1), (514, 30, 2312, 16, 3, 2), (513, 65, 72, 1, 1, 1),
                                                   (6, 256, 1024, 8, 8, 3), (515, 129, 256, 2, 1, 1)])
@pytest.mark.parametrize("mode", ["top_softmax", "softmax_all", "sigmoid", "softmax_scores"])
def test_choices_and_shares(T, E, K, top, groups, keep, mode):
    from allpaca_b200 import ops
    g = torch.Generator().manual_seed(T + E)
    h = torch.randn(T, K, generator=g).to(torch.bfloat16)
    router = (torch.randn(E, K, generator=g) * 2.0 * K ** -0.5).to(torch.bfloat16)
    chosen, weight = i32(T, top), torch.empty(T, top, device=DEV)
    ops.moe_route_rows(h.to(DEV), router.to(DEV), None, chosen, weight, mode, groups=groups, keep=keep, scale=2.5)
    z = h.double() @ router.double().T
    s = torch.sigmoid(z) if mode == "sigmoid" else torch.softmax(z, 1)
    by = z.clone()
    if keep < groups:
        best = by.view(T, groups, -1).amax(2)
        kept = torch.zeros_like(best, dtype=torch.bool).scatter_(1, best.topk(keep, 1).indices, True)
        by[~kept.repeat_interleave(E // groups, 1)] = -torch.inf
    got = chosen.cpu().long()
    # ties within a 32-bit sum's error may fall either way; what is chosen is as good as the best and chosen once
    want = by.topk(top, 1).values
    assert float((z.gather(1, got) - want).abs().max()) < 1e-5 and all(len(set(r)) == top for r in got.tolist())
    picked = z.gather(1, got) if mode == "top_softmax" else s.gather(1, got)
    share = torch.softmax(picked, 1) if mode == "top_softmax" else picked / picked.sum(1, keepdim=True) if mode == "softmax_all" else picked
    assert float((weight.double().cpu() - 2.5 * share).abs().max()) < 2e-5


@pytest.mark.parametrize("T,top,E,real", [(1, 1, 1, 1), (5, 3, 40, 40), (700, 4, 32, 30), (33, 2, 256, 256), (300, 16, 17, 0)])
def test_pairs_grouped_by_expert(T, top, E, real):
    from allpaca_b200 import ops
    g = torch.Generator().manual_seed(T)
    chosen = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(T)]).to(torch.int32)
    chosen = torch.where(chosen % 3 == 1, chosen, chosen // 2 * 2).contiguous()       # uneven; experts nobody chose
    pairs = T * top
    perm, place, first = i32(pairs), i32(pairs), i32(E + 1)
    tiles = torch.zeros(ops.moe_max_tiles(pairs, E) + 1, 3, dtype=torch.int32, device=DEV)
    ops.moe_sort(chosen.to(DEV), perm, place, tiles, E, first, real=real)
    perm, place, first, tiles = (t.cpu().long() for t in (perm, place, first, tiles))
    flat = chosen.view(-1).long()
    assert torch.equal(first, torch.cat([torch.zeros(1, dtype=torch.long), torch.bincount(flat, minlength=E).cumsum(0)]))
    assert sorted(perm.tolist()) == list(range(pairs)) and torch.equal(perm[place], torch.arange(pairs))
    assert torch.equal(flat[perm], flat.sort().values)
    want = [(e, r, min(64, int(first[e + 1]) - r)) for e in range(real) for r in range(int(first[e]), int(first[e + 1]), 64)]
    assert [tuple(t) for t in tiles[:int(tiles[-1, 0])].tolist()] == want


@pytest.mark.parametrize("T,top,H", [(1, 1, 4), (7, 3, 1028), (20, 9, 2048), (5, 16, 30), (3, 8, 4100)])
@pytest.mark.parametrize("with_base,unweighted", [(False, False), (True, True)])
def test_results_added_up(T, top, H, with_base, unweighted):
    from allpaca_b200 import ops
    g = torch.Generator().manual_seed(H)
    o, weight = torch.randn(T * top, H, generator=g), torch.rand(T, top, generator=g)
    place, base = torch.randperm(T * top, generator=g).to(torch.int32), torch.randn(T, H, generator=g)
    delta = torch.empty(T, H, device=DEV)
    ops.moe_combine(o.to(DEV), place.to(DEV), weight.to(DEV), delta, unweighted=unweighted, base=base.to(DEV) if with_base else None)
    w = torch.ones_like(weight) if unweighted else weight
    want = (o[place.long()].view(T, top, H).double() * w.double()[:, :, None]).sum(1) + (base.double() if with_base else 0.0)
    # top + 2 roundings of partial sums that stay below 16
    assert float((delta.double().cpu() - want).abs().max()) < (top + 2) * 2.0 ** -20
