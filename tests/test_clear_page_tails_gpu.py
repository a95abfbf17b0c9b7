"""Clearing of the slots behind a step's last token on pages that it begins, byte for byte against plain indexing: every width of a store,
planes beyond one per warp, few rows and many, one plane to a run, rows inside a page, pages that are full or that a row has not."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def check(T, runs, outer, P, inner, dtype, offset=0):
    from allpaca_b200 import ops
    g = torch.Generator().manual_seed(T + runs + inner)
    num_pages, width = T + 3, 2
    shape = (runs, num_pages, *outer, P, inner)
    n = 1
    for s in shape:
        n *= s
    size = torch.empty(0, dtype=dtype).element_size()
    flat = torch.randint(1, 120, ((n + offset) * size,), generator=g, dtype=torch.uint8).to(DEV).view(dtype)
    pages = flat[offset:].view(shape)
    want = pages.clone()
    # a row per sequence: the first of a page (in the table's first or second column), inside one, on a page it has not, and with
    # more tokens of the step behind it, up to a full page
    table = torch.randperm(num_pages, generator=g)[:T].view(T, 1).repeat(1, width).int()
    pos = torch.randint(0, width * P, (T,), generator=g).int()
    pos[::2] = pos[::2] // P * P
    behind = torch.randint(1, P + 2, (T,), generator=g).int()
    table[T // 2:T // 2 + 1] = -1
    pos[0], behind[0] = P * (width - 1), 1
    context = pos + behind
    for t in range(T):
        page = int(table[t, int(pos[t]) // P])
        if int(pos[t]) % P == 0 and page >= 0:
            want[:, page].narrow(-2, min(int(behind[t]), P), P - min(int(behind[t]), P)).zero_()
    ops.clear_page_tails(pages, pages.dim() - 2, pos.to(DEV), torch.arange(T, dtype=torch.int32, device=DEV), table.to(DEV), context.to(DEV))
    assert torch.equal(pages.view(torch.uint8), want.view(torch.uint8))
    if offset:
        assert bool((flat[:offset].view(torch.uint8) > 0).all())


# inner and type: stores of 16, 8, 4, 2 bytes and 1, and a run of columns that 16 bytes do not divide
@pytest.mark.parametrize("inner, dtype", [(64, torch.bfloat16), (12, torch.bfloat16), (3, torch.float32), (5, torch.bfloat16),
                                          (7, torch.uint8), (72, torch.bfloat16)])
@pytest.mark.parametrize("T", [1, 2, 17, 64, 65, 130])
def test_widths_and_rows(inner, dtype, T):
    check(T, 3, (2, 5), 16, inner, dtype)


@pytest.mark.parametrize("T, runs, outer", [(3, 6, (2, 24)), (64, 7, (41,)), (70, 5, (2, 8)), (9, 300, ()), (5, 1, (261,)), (130, 67, ())])
def test_more_planes_than_warps(T, runs, outer):
    check(T, runs, outer, 8, 8, torch.bfloat16)


@pytest.mark.parametrize("offset", [1, 2, 4])
def test_pages_that_start_off_a_boundary(offset):
    check(9, 2, (2, 3), 16, 64, torch.bfloat16, offset)


def test_a_plane_of_a_gigabyte():
    from allpaca_b200 import ops
    pages = torch.full((1, 1, 1, 2, 2 ** 29), 7, dtype=torch.uint8, device=DEV)
    one = torch.ones(1, dtype=torch.int32, device=DEV)
    ops.clear_page_tails(pages, 3, one - 1, one - 1, one.view(1, 1) - 1, one)
    assert bool((pages[0, 0, 0, 0] == 7).all()) and not bool(pages[0, 0, 0, 1].any())
