"""Decode attention launched directly behind the kernel of this library that stores ALL of a sequence's keys, as a caller of
the ops may (an engine's step stores the newest only): the result is the same bits as with the device idle in between,
every time.  And who says what to a kernel that may read ahead."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
P, B, N = 16, 3, 700                                      # page, sequences, tokens of each


def i32(x):
    return torch.as_tensor(x, dtype=torch.int32).to(DEV)


def layout():
    blocks = -(-N // P)
    table = i32(torch.randperm(B * blocks, generator=torch.Generator().manual_seed(1)).view(B, blocks))
    positions, token_seq = torch.arange(N).repeat(B), torch.arange(B).repeat_interleave(N)
    return B * blocks, table, i32(positions), i32(token_seq), i32(range(B + 1)), i32([N - 1] * B)


def windowed(pages, table, positions, token_seq, start, last, g):
    from allpaca_b200 import ops
    nh, nkv, D = 8, 2, 64
    cache = torch.zeros(pages, nkv, P, 2 * D, dtype=torch.bfloat16, device=DEV)
    qkv, q = torch.randn(B * N, (nh + 2 * nkv) * D, generator=g).to(DEV), torch.empty(B * N, nh * D, dtype=torch.bfloat16, device=DEV)
    one, out = torch.randn(B, nh * D, generator=g).to(torch.bfloat16).to(DEV), torch.empty(B, nh * D, dtype=torch.bfloat16, device=DEV)

    def store():
        ops.qk_norm_store(qkv, q, cache, positions, token_seq, table, nh, nkv, D, D, 1e-5)

    def attend():
        ops.attention_window_bias(one, out, cache, table, start, last, B, nh, nkv, D, D, D ** -0.5, 0, single_rows=True,
                                  other_rows=False, bias=None, max_context=N)
    return cache, store, attend, out


def latent(pages, table, positions, token_seq, start, last, g):
    from allpaca_b200 import ops
    from allpaca_b200.parts import Workspace
    H, R, rot = 8, 128, 32
    cache, ws = torch.zeros(pages, P, R + rot, dtype=torch.bfloat16, device=DEV), Workspace(torch.device(DEV))
    proj, weight = torch.randn(B * N, R + rot, generator=g).to(DEV), torch.ones(R, device=DEV)
    one = torch.randn(B, H * (R + rot), generator=g).to(torch.bfloat16).to(DEV)
    out = torch.empty(B, H * R, dtype=torch.bfloat16, device=DEV)

    def store():
        ops.latent_prepare(proj, 0, 0, None, None, 0, R, rot, 0, weight, cache, positions, token_seq, table, None, 1e-5)

    def attend():
        ops.latent_decode(one, out, cache, table, start, last, B, H, R + rot, R, 0.1, None, N, ws)
    return cache, store, attend, out


def side_by_side(pages, table, positions, token_seq, start, last, g):
    from allpaca_b200 import ops
    nh, nkv, D = 8, 2, 64
    cache, kept = torch.zeros(pages, 2, nkv, P, D, dtype=torch.bfloat16, device=DEV), []
    qkv, q = torch.randn(B * N, (nh + 2 * nkv) * D, generator=g).to(DEV), torch.empty(B * N, nh * D, dtype=torch.bfloat16, device=DEV)
    one, out = torch.randn(B, nh * D, generator=g).to(torch.bfloat16).to(DEV), torch.empty(B, nh * D, dtype=torch.bfloat16, device=DEV)

    def scratch(name, shape, dtype):
        kept.append(torch.empty(shape, dtype=dtype, device=DEV))
        return kept[-1]

    def store():
        ops.rope_kv_store(qkv, q, cache, positions, token_seq, table, None, 0, nh, nkv, D)

    def attend():
        ops.attention(one, out, cache, table, i32(range(B)), last, nh, nkv, D, D ** -0.5, seq_start=start, query_lens=[1] * B,
                      max_context=N, scratch=scratch)
    return cache, store, attend, out


@pytest.mark.parametrize("kind", [windowed, latent, side_by_side])
def test_attention_waits_for_the_keys(kind):
    from allpaca_b200 import ops
    cache, store, attend, out = kind(*layout(), torch.Generator().manual_seed(2))
    store()
    torch.cuda.synchronize()
    attend()
    torch.cuda.synchronize()
    want = out.clone()
    assert torch.isfinite(want).all() and float(want.abs().max()) > 0
    for _ in range(20):
        cache.zero_()
        out.zero_()
        torch.cuda.synchronize()
        store()
        attend()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    ops.check_kernel_status()


def test_only_options_on_the_host_are_read_ahead(monkeypatch):
    from allpaca_b200 import ops
    plain, seen = ops.call, []
    monkeypatch.setattr(ops, "call", lambda lib, name, *a: (seen.append(a[-2]), plain(lib, name, *a)))
    logits, out = torch.randn(2, 500, device=DEV), torch.empty(2, dtype=torch.int32, device=DEV)
    options = [torch.ones(2), torch.full((2,), 5, dtype=torch.int32), torch.ones(2), torch.tensor([0.2, 0.7])]
    pinned, device = [t.pin_memory() for t in options], [t.to(DEV) for t in options]
    ops.sample(logits, *pinned, out)
    ops.sample(logits, *device, out)
    ops.sample(logits, *pinned[:3], device[3], out)
    torch.cuda.synchronize()
    assert seen == [1, 0, 0]


def test_the_engine_says_that_its_keys_are_settled(tmp_path, monkeypatch):
    """The default is to wait; the engine, whose steps begin in plain stream order, need not."""
    from allpaca_b200 import ops
    from allpaca_b200.config import EngineConfig
    from allpaca_b200.config.presets import preset_config
    from allpaca_b200.engine.batch import BatchEntry
    from allpaca_b200.engine.runner import ModelRunner
    from allpaca_b200.weights.random_model import write_random_model
    write_random_model(str(tmp_path), preset_config("tiny-a"), seed=0, dtype="bfloat16", norm_std=0.02)
    runner = ModelRunner(str(tmp_path), EngineConfig(dtype="bfloat16", page_size=16, num_pages=32, max_num_seqs=4,
                                                     max_num_batched_tokens=64, use_cuda_graphs=False))
    plain, seen = ops.attention, []
    monkeypatch.setattr(ops, "attention", lambda *a, **k: (seen.append(k.get("settled", False)), plain(*a, **k))[1])
    runner.step([BatchEntry("a", list(range(20)), [])])
    runner.step([BatchEntry("a", [3], [0])])
    assert seen and all(seen)
