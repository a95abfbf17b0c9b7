"""A step's metadata fetched by a kernel, and choices that leave their tokens in host memory as well: one number and blocks that
end inside a CTA, the device's tokens in their place; options in pinned memory give the tokens that options on the device give,
whichever kernel draws; what is no pinned memory is refused before anything runs."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("first,n,off,count", [(0, 1, 0, 0), (0, 255, 3, 5), (0, 257, 0, 257), (40, 5000, 5039, 1), (9, 4, 9, 4)])
@pytest.mark.parametrize("indexed", [False, True])
def test_metadata_and_tokens(first, n, off, count, indexed):
    from allpaca_b200 import ops
    g = torch.Generator().manual_seed(n)
    end = first + n
    index = torch.randint(-1, max(count, 1), (count,), generator=g, dtype=torch.int32)
    host = torch.cat([torch.randint(-9, 9, (end,), generator=g, dtype=torch.int32), index]).pin_memory()
    dev = torch.full((end + 3,), 77, dtype=torch.int32, device=DEV)
    tokens = torch.arange(100, 100 + count, dtype=torch.int32, device=DEV)
    ops.stage_step(host, dev, first, n, tokens if count else None, off, count, end if indexed else -1)
    want = torch.full((end + 3,), 77, dtype=torch.int32)
    want[first:end] = host[first:end]
    for i in range(count):
        src = int(index[i]) if indexed else i
        if src >= 0:
            want[off + i] = 100 + src
    assert torch.equal(dev.cpu(), want)


def test_memory_that_is_not_pinned_is_refused():
    from allpaca_b200 import ops
    from allpaca_b200.ops import KernelError
    dev, logits = torch.zeros(4, dtype=torch.int32, device=DEV), torch.zeros(1, 8, device=DEV)
    with pytest.raises(KernelError):
        ops.stage_step(torch.zeros(4, dtype=torch.int32), dev, 0, 4)
    with pytest.raises(KernelError):
        ops.argmax(logits, dev[:1], host=torch.zeros(1, dtype=torch.int32))
    one = torch.ones(1)
    with pytest.raises(KernelError):
        ops.sample(logits, one, torch.ones(1, dtype=torch.int32), one, one, dev[:1])


@pytest.mark.parametrize("method", ["cluster", "rows"])
@pytest.mark.parametrize("R,V", [(1, 50), (5, 4097), (3, 70000)])
def test_options_and_tokens_in_host_memory(method, R, V):
    from allpaca_b200 import ops
    g = torch.Generator().manual_seed(V)
    logits = (3.0 * torch.randn(R, V, generator=g)).to(DEV)
    options = [torch.tensor([0.8, 0.0, 1.3, 1.0, 0.5][:R]), torch.tensor([40, 0, 0, 3, 5000][:R], dtype=torch.int32),
               torch.tensor([0.95, 1.0, 0.5, 1.0, 0.9][:R]), torch.rand(R, generator=g)]
    got = []
    for where in (lambda t: t.to(DEV), lambda t: t.pin_memory()):
        out, host = torch.full((R,), -1, dtype=torch.int32, device=DEV), torch.full((R,), -1, dtype=torch.int32).pin_memory()
        placed = [where(t) for t in options]             # kept until the kernel has read them
        ops.sample(logits, *placed, out, method=method, host=host)
        torch.cuda.synchronize()
        assert torch.equal(out.cpu(), host)
        got.append(host)
    assert torch.equal(got[0], got[1])
    out, host = torch.empty(R, dtype=torch.int32, device=DEV), torch.empty(R, dtype=torch.int32).pin_memory()
    ops.argmax(logits, out, host=host)
    torch.cuda.synchronize()
    assert torch.equal(host.long(), logits.argmax(1).cpu()) and torch.equal(out.cpu(), host)


@pytest.mark.parametrize("budget,chunk", [(24, 8), (40, 24)])
def test_decoding_beside_portions_takes_tokens_from_the_device(tmp_path, budget, chunk):
    """Prompts cut into portions beside rows that decode, requests that a stop token ends while a step with their next row
    is in flight, a pool so small that some are preempted: every reply is what the request gives alone (32-bit rows have
    the same bits in every batch)."""
    from allpaca_b200 import LLM, SamplingParams
    from allpaca_b200.config.presets import preset_config
    from allpaca_b200.weights.random_model import write_random_model
    write_random_model(str(tmp_path), preset_config("tiny-a"), seed=0, dtype="float32", norm_std=0.02)
    g = torch.Generator().manual_seed(budget)
    prompts = [torch.randint(0, 200, (n,), generator=g).tolist() for n in (3, 41, 9, 60, 17, 30, 1, 25)]
    kw = dict(model=str(tmp_path), dtype="float32", page_size=8, max_num_seqs=4, max_num_batched_tokens=budget, prefill_chunk=chunk)
    alone = LLM(max_cache_tokens=1024, **kw)
    free = [alone.generate([p], SamplingParams(max_tokens=14, seed=i))[0].token_ids for i, p in enumerate(prompts)]
    params, want = [], []
    for i, t in enumerate(free):
        stop = t[5] if i % 3 == 1 else None
        params.append(SamplingParams(max_tokens=14, seed=i, stop_token_ids=[] if stop is None else [stop]))
        want.append(t if stop is None else t[:t.index(stop) + 1])
    for tokens in (1024, 120):
        llm = LLM(max_cache_tokens=tokens, **kw)
        assert [o.token_ids for o in llm.generate(prompts, params)] == want
        for o in llm.flush():
            pass
        assert llm.runner.cache.num_running() == 0
        llm.runner.cache.check()


def test_a_refused_step_changes_nothing(tmp_path):
    """A place among the device's tokens that is not there, or one for several rows, or too few tokens: refused before pages are
    taken and before a request has advanced, so that the same step without the fault gives what it would have given."""
    from allpaca_b200.config import EngineConfig
    from allpaca_b200.config.presets import preset_config
    from allpaca_b200.engine.batch import BatchEntry
    from allpaca_b200.engine.runner import ModelRunner
    from allpaca_b200.weights.random_model import write_random_model
    write_random_model(str(tmp_path), preset_config("tiny-a"), seed=0, dtype="float32", norm_std=0.02)
    runner = ModelRunner(str(tmp_path), EngineConfig(dtype="float32", page_size=8, num_pages=32, max_num_seqs=4,
                                                     max_num_batched_tokens=64))
    prompt, tokens = list(range(3, 19)), torch.tensor([5, 9], dtype=torch.int32, device=DEV)
    runner.step([BatchEntry("a", prompt, [])])
    want = runner.step([BatchEntry("b", prompt, []), BatchEntry("a", [9], [0])]).clone()
    runner.finish("a"), runner.finish("b")
    runner.step([BatchEntry("a", prompt, [])])
    state = lambda: (runner.cache.num_tokens("a"), runner.cache.has("b"), runner.cache.num_running(), runner.cache.num_free_pages(0))
    before = state()
    for wrong in (BatchEntry("a", [0], [0], 2), BatchEntry("a", [0], [0], -1), BatchEntry("a", [0, 0], [1], 1)):
        with pytest.raises(ValueError):
            runner.step([BatchEntry("b", prompt, []), wrong], device_tokens=tokens)
        assert state() == before
    for bad in (tokens[:1], tokens.long(), tokens.cpu()):
        with pytest.raises(ValueError):
            runner.step([BatchEntry("b", prompt, []), BatchEntry("a", [0], [0])], device_tokens=bad)
        assert state() == before
    assert torch.equal(runner.step([BatchEntry("b", prompt, []), BatchEntry("a", [0], [0], 1)], device_tokens=tokens), want)


def test_a_sampler_goes_away_after_its_launches():
    from allpaca_b200.sampling import SamplingParams
    from allpaca_b200.sampling.sampler import Sampler
    sampler, logits = Sampler(torch.device(DEV), 4), torch.randn(4, 300, device=DEV)
    torch.cuda._sleep(100_000_000)                       # some 50 ms
    done = sampler.launch(logits, [SamplingParams(max_tokens=1, seed=i) for i in range(4)], [0.1, 0.4, 0.6, 0.9]).event
    assert not done.query()
    del sampler
    assert done.query()
