"""The state-space recurrence of steps of many rows, eight tokens at a time, against the recurrence in 64 bits: blocks that a portion
fills and does not, single rows beside portions, states carried from portions to single rows and back, several groups, sizes that are no
whole 16-byte runs, no skip and no bias."""
import pytest
import torch

import plain_viresun as plain
from allpaca_b200.parts import Workspace

pytestmark = pytest.mark.gpu
DEV = "cuda"


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("Hh, E, N, G, bare", [(6, 12, 20, 3, False), (4, 32, 70, 1, False), (32, 64, 128, 1, False), (3, 5, 3, 3, False),
                                               (2, 100, 16, 2, True), (1, 64, 512, 1, False)])
def test_portions_of_many_rows(Hh, E, N, G, bare, monkeypatch):
    from allpaca_b200 import ops
    monkeypatch.setattr(ops.mixers, "ssm_in_blocks", lambda rows, num_seqs, *_: rows > 2 * num_seqs)     # small states as well
    g = torch.Generator().manual_seed(Hh * 10 + N)
    inner = Hh * E
    a_log = torch.log(0.02 + 0.3 * torch.rand(Hh, generator=g))
    dt_bias, d_skip = torch.randn(Hh, generator=g) - 0.5, torch.randn(Hh, generator=g)
    ws = Workspace(torch.device(DEV))
    state = torch.full((3, Hh * N * E + 7), float("nan"), device=DEV)[:, :Hh * N * E].unflatten(1, (Hh, N, E))
    lengths = [150, 77, 24]
    rows = [(torch.randn(n, inner + 2 * G * N, generator=g), torch.randn(n, Hh + 3, generator=g)) for n in lengths]
    got = [[], [], []]
    done = [0, 0, 0]

    def run(takes):
        """takes: rows of sequence 0, 1, 2 in this step (0: not in it); sequence i keeps its state in slot 2 - i."""
        parts = [(i, n) for i, n in enumerate(takes) if n]
        starts, pos, xs, dts = [0], [], [], []
        for i, n in parts:
            a = done[i]
            xs.append(rows[i][0][a:a + n])
            dts.append(rows[i][1][a:a + n])
            pos += range(a, a + n)
            starts.append(starts[-1] + n)
            done[i] += n
        xbc, dt = torch.cat(xs).to(DEV), torch.cat(dts).to(DEV)
        before = xbc.clone()
        y = torch.empty(xbc.shape[0], inner, device=DEV)
        ops.ssm_scan(xbc, dt[:, 3:], None if bare else dt_bias.to(DEV), a_log.to(DEV), None if bare else d_skip.to(DEV), state,
                     i32(starts), i32(pos), i32([2 - i for i, _ in parts]), y, len(parts), Hh, G, N, E, workspace=ws)
        assert torch.equal(xbc, before)
        for j, (i, n) in enumerate(parts):
            got[i].append(y[starts[j]:starts[j + 1]].cpu())
    assert ops.ssm_in_blocks(65, 2, Hh) and not ops.ssm_in_blocks(3, 3, Hh)
    run([64, 1, 0])                  # whole blocks beside a single row
    run([1, 60, 14])                 # a ragged block, and the long one goes on by a single row
    run([1, 1, 1])                   # token after token
    run([84, 15, 9])
    for i, (x, dt) in enumerate(rows):
        raw = dt[:, 3:].double() + (0.0 if bare else dt_bias.double())
        want = plain.ssm_recurrence(x[:, :inner].double().view(-1, Hh, E), x[:, inner:inner + G * N].double().view(-1, G, N),
                                    x[:, inner + G * N:].double().view(-1, G, N), torch.log1p(torch.exp(raw)), a_log.double(),
                                    torch.zeros(Hh).double() if bare else d_skip.double()).reshape(-1, inner)
        # the tolerance of the recurrence token after token (test_viresun_kernels_gpu.py)
        assert float((torch.cat(got[i]).double() - want).abs().max()) <= 2e-5 * float(want.abs().max()), i


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("where", ["value", "key", "query", "step"])
def test_rows_before_one_that_is_not_finite(where, value):
    """A token whose numbers are not finite leaves every earlier row of its portion as it is, those of the same eight among them, and
    the other sequences; the recurrence token after token says which rows those are."""
    from allpaca_b200 import ops
    g = torch.Generator().manual_seed(5)
    Hh, E, N = 4, 32, 64
    inner, lengths, bad = Hh * E, [61, 40], 29
    xbc = torch.randn(sum(lengths), inner + 2 * N, generator=g)
    dt = torch.randn(sum(lengths), Hh, generator=g)
    if where == "step":
        dt[bad, 1] = value
    else:
        xbc[bad, {"value": 3, "key": inner + 5, "query": inner + N + 5}[where]] = value
    a_log, d_skip = torch.log(0.02 + 0.3 * torch.rand(Hh, generator=g)), torch.randn(Hh, generator=g)
    pos = torch.cat([torch.arange(n) for n in lengths]).int().to(DEV)
    assert ops.ssm_in_blocks(sum(lengths), 2, Hh)
    results = []
    for ws in (None, Workspace(torch.device(DEV))):
        state = torch.zeros(2, Hh, N, E, device=DEV)
        y = torch.empty(sum(lengths), inner, device=DEV)
        ops.ssm_scan(xbc.to(DEV), dt.to(DEV), None, a_log.to(DEV), d_skip.to(DEV), state, i32([0, 61, 101]), pos, i32([0, 1]), y, 2,
                     Hh, 1, N, E, workspace=ws)
        results.append((y, state))
    (chain, chain_state), (blocks, blocks_state) = results
    for want, got in ((chain, blocks), (chain_state, blocks_state)):
        finite = torch.isfinite(want)
        assert torch.equal(torch.isfinite(got), finite)
        assert float((got - want)[finite].abs().max()) <= 2e-5 * float(want[finite].abs().max())
    assert bool(torch.isfinite(blocks[:bad]).all()) and not bool(torch.isfinite(blocks[bad]).all())


@pytest.mark.parametrize("E", [32, 5])
def test_rows_of_no_sequence(E):
    """Rows ahead of the first sequence's and behind the last one's stay as they are, in blocks as token after token."""
    from allpaca_b200 import ops
    g = torch.Generator().manual_seed(6)
    Hh, N, T, first, last = 4, 16, 130, 3, 101
    xbc, dt = torch.randn(T, Hh * E + 2 * N, generator=g).to(DEV), torch.randn(T, Hh, generator=g).to(DEV)
    a_log, d_skip = torch.randn(Hh, generator=g).to(DEV), torch.randn(Hh, generator=g).to(DEV)
    pos = (torch.arange(T) - first).int().to(DEV)
    assert ops.ssm_in_blocks(T, 1, Hh)
    results = []
    for ws in (None, Workspace(torch.device(DEV))):
        y = torch.full((T, Hh * E), 7.0, device=DEV)
        ops.ssm_scan(xbc, dt, None, a_log, d_skip, torch.zeros(1, Hh, N, E, device=DEV), i32([first, last]), pos, i32([0]), y, 1, Hh, 1,
                     N, E, workspace=ws)
        results.append(y)
    assert all(bool((y[:first] == 7.0).all()) and bool((y[last:] == 7.0).all()) for y in results)
    assert float((results[0] - results[1]).abs().max()) <= 2e-5 * float(results[0].abs().max())


def test_scratch_of_steps_of_as_many_rows():
    """More sequences in a step of as many rows ask for no other buffers: a larger one would have the engine record its graphs again."""
    from allpaca_b200 import ops
    Hh, E, N, T = 4, 32, 64, 160
    ws, seen = Workspace(torch.device(DEV)), []
    for seqs in (1, 2, 5, 20, 40):
        n = T // seqs
        ops.ssm_scan(torch.randn(T, Hh * E + 2 * N, device=DEV), torch.randn(T, Hh, device=DEV), None, torch.zeros(Hh, device=DEV), None,
                     torch.zeros(seqs, Hh, N, E, device=DEV), i32([n * i for i in range(seqs + 1)]), i32(list(range(n)) * seqs),
                     i32(list(range(seqs))), torch.empty(T, Hh * E, device=DEV), seqs, Hh, 1, N, E, workspace=ws, longest=T)
        seen.append(ws.generation)
    assert len(set(seen)) == 1
