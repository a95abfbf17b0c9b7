"""The recurrence of many single rows, whose states lie in shared memory whole: against 64 bits, at sizes on both sides of
its rule and at the edges of its blocks of columns."""
import pytest
import torch

from allpaca_b200 import ops

DEV = "cuda:0"
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["head", "channel_delta", "gated_unit"])
@pytest.mark.parametrize("seqs,heads,D,V,lens", [
    (16, 8, 128, 128, None), (15, 8, 128, 128, None), (40, 16, 64, 65, None), (40, 8, 100, 161, None), (300, 1, 36, 256, None),
    (40, 8, 128, 129, (0, 2)),                               # as many rows as sequences, yet not one to each
])
def test_many_single_rows(kind, seqs, heads, D, V, lens):
    gen = torch.Generator().manual_seed(seqs * V + D)
    unit = kind == "gated_unit"
    lengths = [1] * seqs
    if lens:
        lengths[3], lengths[5] = lens
    starts = torch.tensor([0] + lengths).cumsum(0)
    T, G = sum(lengths), max(1, heads // 2)
    rnd = lambda *shape: torch.randn(*shape, generator=gen)
    q, k, v = rnd(T, G, D), rnd(T, G, D) * D ** -0.5, rnd(T, heads, V - unit)
    state = rnd(seqs + 2, heads, D, V)
    slots = torch.randperm(seqs + 2, generator=gen)[:seqs]
    positions = torch.randint(1, 50, (T,), generator=gen)
    positions[int(starts[7])] = 0                            # one that starts here
    beta, raw = rnd(T, heads), rnd(T, heads, D)
    const = torch.rand(heads, generator=gen)

    d = lambda t: t.double()
    want_y, want_s, tol_y, tol_s = torch.zeros(T, heads, V).double(), d(state), torch.zeros(T, heads, V).double(), torch.zeros(state.shape).double()
    for s in range(seqs):
        S = d(state[slots[s]])
        for n, t in enumerate(range(int(starts[s]), int(starts[s + 1]))):
            if n == 0 and positions[t] == 0:
                S = torch.zeros_like(S)
            qq, kk = (d(x[t]).repeat_interleave(heads // G, 0) for x in (q, k))
            vv = d(v[t])
            if unit:
                vv = torch.cat([vv, torch.ones(heads, 1).double()], 1)
            if kind == "channel_delta":
                a = torch.exp(-torch.exp(d(const))[:, None] * torch.nn.functional.softplus(d(raw[t])))[:, :, None]
            else:
                a = d(const)[:, None, None]
            size = S.abs() * a
            S = S * a
            if kind == "channel_delta":
                u = torch.sigmoid(d(beta[t]))[:, None] * (vv - torch.einsum("hdc,hd->hc", S, kk))
                umag = vv.abs() + torch.einsum("hdc,hd->hc", S.abs(), kk.abs())
            else:
                u = vv * (d(const * 0.5)[:, None] if unit else 1.0)
                umag = u.abs()
            S = S + kk[:, :, None] * u[:, None, :]
            size = size + kk.abs()[:, :, None] * umag[:, None, :]
            want_y[t] = torch.einsum("hdc,hd->hc", S, qq) * 0.5
            # sums over D in 32 bits, twice where the write needs one itself, and some ulps of the decays' exponentials
            f = (2 * D + 64) * 2.0 ** -24
            tol_y[t] = f * torch.einsum("hdc,hd->hc", size, qq.abs())
            tol_s[slots[s]] = f * size * 2
        want_s[slots[s]] = S

    cuda = lambda t: t.to(DEV).contiguous()
    i32 = lambda t: t.to(torch.int32).to(DEV)
    st, y = cuda(state), torch.zeros(T, heads * V, device=DEV)
    extra = {"decay": "head", "decay_const": cuda(const)}
    if kind == "channel_delta":
        extra = {"decay": "channel_token", "decay_channel": cuda(raw.flatten(1)), "decay_const": cuda(const), "beta": cuda(beta)}
    elif unit:
        extra = {"decay": "head_ready", "decay_head": cuda(const.expand(T, heads)), "unit_column": True,
                 "write_gate": cuda((const * 0.5).expand(T, heads))}
    ops.linear_scan(cuda(q.flatten(1)), cuda(k.flatten(1)), cuda(v.flatten(1)), y, st, i32(starts), i32(positions), i32(slots), seqs, heads,
                    G, D, V - unit, out_scale=0.5, **extra)
    assert ((y.cpu().double().view(T, heads, V) - want_y).abs() <= tol_y + 1e-30).all()
    assert ((st.cpu().double() - want_s).abs() <= tol_s).all()
