"""Rotation and cache store of steps of many rows (several heads to a thread) against the same rows in steps of few, bit for bit: head
counts that are no multiple of a thread's, pages that a row has not, no rotation, no cache."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nh, nkv, hd, T", [(32, 8, 128, 1025), (5, 1, 64, 1025), (3, 3, 48, 1025), (6, 2, 16, 1025), (13, 2, 256, 1025),
                                            (33, 0, 128, 1225), (3, 2, 80, 8193)])
@pytest.mark.parametrize("pairing", [0, 2])
@pytest.mark.parametrize("form", ["all", "no rotation", "no cache"])
def test_rows_of_a_long_step(nh, nkv, hd, T, pairing, form):
    from allpaca_b200 import ops
    if nkv == 0 and form != "no cache":
        pytest.skip("nothing to store")
    g = torch.Generator(device="cuda").manual_seed(nh + hd)
    P, width = 16, T // 16 + 2
    qkv = torch.randn(T, (nh + 2 * nkv) * hd, generator=g, device="cuda").bfloat16()
    angle = torch.rand(T, hd // 2, generator=g, device="cuda") * 6.28
    cos_sin = torch.stack([angle.cos(), angle.sin()], dim=-1).contiguous() if form != "no rotation" else None
    lengths = [T - 213, 1, 212]
    seq = torch.repeat_interleave(torch.arange(3, device="cuda"), torch.tensor(lengths, device="cuda")).int()
    pos = torch.cat([torch.arange(n, device="cuda") + 5 for n in lengths]).int()
    table = torch.randperm(3 * width, generator=g, device="cuda").view(3, width).int().contiguous()
    table[2, 3] = -1                                          # a page that the window has passed

    def run(cuts):
        q = torch.zeros(T, nh * hd, dtype=torch.bfloat16, device="cuda")
        pages = torch.zeros(3 * width, 2, nkv, P, hd, dtype=torch.bfloat16, device="cuda")
        for a, b in zip(cuts, cuts[1:]):
            ops.rope_kv_store(qkv[a:b], q[a:b], pages if form != "no cache" else None, pos[a:b], seq[a:b], table,
                              cos_sin[a:b] if cos_sin is not None else None, pairing, nh, nkv, hd)
        return q, pages
    many, few = run([0, T]), run(list(range(0, T, 400)) + [T])
    assert torch.equal(many[0], few[0]) and torch.equal(many[1], few[1])
