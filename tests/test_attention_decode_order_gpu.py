"""Decode attention whose CTAs take the longest sequences first: the same bits as in the order of the sequences, whatever
number of key slices, for one more row than a warp holds, two rows to every lane, and lengths that tie."""
import math

import pytest
import torch

from test_kernels_gpu import dev, paged_case, reference_attention, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splits", [1, 2, 3, 8])
@pytest.mark.parametrize("nh,nkv,hd,P", [(32, 8, 64, 16), (32, 8, 128, 16), (40, 2, 64, 16)])
@pytest.mark.parametrize("rows", [24, 33, 64])
def test_longest_first_changes_no_bits(splits, nh, nkv, hd, P, rows, monkeypatch):
    from allpaca_b200 import ops
    lens = [1 + (37 * i * i) % 200 for i in range(rows)]
    lens[rows // 2], lens[-1], lens[3] = 1500, 1500, 700
    decode = [(n, 1) for n in lens]
    case = paged_case(decode, nh, nkv, hd, P, torch.bfloat16, seed=rows)
    scale, kept, got, order = 1.0 / math.sqrt(hd), [], [], 0
    monkeypatch.setattr(ops, "decode_splits", lambda *a, **k: splits)
    plain = ops.call

    def spy(lib, name, *args):
        if name == "ap_attention_decode_tma":           # whatever the rule says
            args = args[:-2] + (order, args[-1])
        return plain(lib, name, *args)
    monkeypatch.setattr(ops, "call", spy)

    def scratch(name, shape, dtype):
        kept.append(torch.empty(shape, dtype=dtype, device="cuda"))
        return kept[-1]
    longest = int(case["positions"].max()) + 1
    for order in (0, 1):
        q = dev(case["q"])
        out = torch.full_like(q, float("nan"))
        ops.attention(q, out, dev(case["cache"]), dev(case["table"]), dev(case["token_seq"]), dev(case["positions"]), nh, nkv, hd,
                      scale, 0, seq_start=dev(case["seq_start"]), query_lens=case["query_lens"], max_context=longest,
                      scratch=scratch, use_tma=True)
        ops.check_kernel_status()
        got.append(out.cpu())
    assert torch.equal(got[0], got[1])
    assert rel_err(got[1], reference_attention(case, decode, nh, hd, None, scale=scale)) < 1.5e-2
