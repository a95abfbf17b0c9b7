"""Single rows in bfloat16 with a distance bias behind a window, against the same attention in 64 bits: head counts that
need one and two groups of sixteen, sizes that end inside a block of 32 coordinates or 64 columns, sequences of one key,
of exactly a block and one more, windows that end inside a page, kept first tokens, sink, gate, soft cap and every bias;
the pages that a window has passed hold NaN."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("H,G,D,E,P,window,keep,bias,cap,extras", [
    (16, 4, 128, 128, 16, 512, 0, "log", 0.0, False), (40, 2, 64, 64, 8, 70, 5, "linear", 0.0, True),
    (3, 1, 72, 40, 16, 0, 0, None, 9.0, False), (9, 1, 192, 128, 32, 300, 17, "log", 0.0, True),
    (2, 2, 8, 8, 8, 1, 0, "linear", 0.0, False), (17, 1, 136, 96, 24, 48, 30, None, 0.0, True)])
@pytest.mark.parametrize("known", [True, False])
def test_single_rows(H, G, D, E, P, window, keep, bias, cap, extras, known):
    from allpaca_b200 import ops
    gen = torch.Generator().manual_seed(H + D)
    lens = [1, 16, 17, 333, 1030]
    scale = 2.0 / math.sqrt(D)
    r1, r2 = 0.1 + torch.rand(H, generator=gen), 0.05 + torch.rand(H, generator=gen)
    if bias == "linear":
        r1 = 0.05 * r1
    sink = torch.randn(H, generator=gen) if extras else None
    gate = torch.randn(len(lens), H + 3, generator=gen) if extras else None
    q = torch.randn(len(lens), H, D, generator=gen).to(torch.bfloat16)
    pages, table, want, base = [], [], [], 0
    for s, T in enumerate(lens):
        kv = torch.randn(T, G, D + E, generator=gen).to(torch.bfloat16)
        n = -(-T // P)
        own = torch.full((n, G, P, D + E), float("nan"), dtype=torch.bfloat16)
        dist = (T - 1 - torch.arange(T)).double()
        seen = (dist < window) | (torch.arange(T) < keep) if window else torch.ones(T, dtype=torch.bool)
        row = []
        for b in range(n):
            if bool(seen[b * P:(b + 1) * P].any()):
                own[b] = 0
                own[b, :, :min(P, T - b * P)] = kv[b * P:(b + 1) * P].transpose(0, 1)
                row.append(base + n - 1 - b)
            else:
                row.append(-1)
        pages.append(own.flip(0))
        table.append(row)
        base += n
        k, v = (t.double().repeat_interleave(H // G, 1) for t in (kv[..., :D], kv[..., D:]))
        z = torch.einsum("hd,thd->ht", q[s].double(), k) * scale
        if cap:
            z = cap * torch.tanh(z / cap)
        if bias == "log":
            z = z - r1.double()[:, None] * torch.log1p(r2.double()[:, None] * dist)
        elif bias == "linear":
            z = z - r1.double()[:, None] * dist
        z = z.masked_fill(~seen, -math.inf)
        if sink is not None:
            z = torch.cat([z, sink.double()[:, None]], 1)
        o = torch.einsum("ht,thd->hd", torch.softmax(z, 1)[:, :T], v)
        want.append(o * torch.sigmoid(gate[s, 1:1 + H].double())[:, None] if gate is not None else o)
    width = max(len(r) for r in table)
    out = torch.full((len(lens), H * E), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops.attention_window_bias(
        q.reshape(len(lens), -1).to(DEV), out, torch.cat(pages).to(DEV), i32([r + [-1] * (width - len(r)) for r in table]),
        i32(list(range(len(lens) + 1))), i32([n - 1 for n in lens]), len(lens), H, G, D, E, scale, window,
        r1.to(DEV) if bias else None, r2.to(DEV) if bias == "log" else None, single_rows=True, other_rows=False, bias=bias,
        keep_first=keep, gate=gate.to(DEV)[:, 1:1 + H] if gate is not None else None,
        sink=sink.to(DEV) if sink is not None else None, softcap=cap, max_context=max(lens) if known else 0)
    got, want = out.double().cpu().view(len(lens), H, E), torch.stack(want)
    # seven stored bits: half a unit in the last place is at most 2^-8 of the value; the 32-bit sums before add far less
    assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + 2e-5 * want.abs().max()).all()), \
        float(((got - want).abs() / want.abs().max()).max())
