"""The 32-bit product against a 64-bit one at the edges of its two kernels (up to 32 rows, tiles of 64 to 176 rows; a
tile's K over a cluster or over one CTA), and one order of sums for every number of rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ROWS = [1, 4, 5, 8, 9, 16, 17, 24, 25, 32, 33, 64, 65, 96, 97, 128, 129, 173, 257]


# N: one tile, a ragged second one, more tiles than the cluster form is used for; K: less than one block, a ragged last
# block, runs of unequal length, empty runs.  Beyond 32 rows the first six take tiles of 64 and 96 rows, the last ones the others too
@pytest.mark.parametrize("N,K", [(128, 32), (130, 4), (97, 100), (256, 256), (300, 1000), (129, 2052), (38000, 96), (2503, 1000),
                                 (3505, 2052)])
def test_rows_of_any_batch(N, K):
    from allpaca_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(N + K)
    a = torch.randn(max(ROWS), K, generator=g, device="cuda")
    w = torch.randn(N, K, generator=g, device="cuda")
    ref = a.double() @ w.double().T
    # a product and an addition round to 2^-24 of a partial sum; partial sums grow as their square root, so the error of
    # a sum of K unit-variance terms stays below 2^-24 K, its size being sqrt(K)
    bound = 2.0 ** -24 * K + 1e-6
    whole = None
    for M in reversed(ROWS):
        out = torch.full((M + 1, N), 7.0, device="cuda")
        ops.gemm_simt(a[:M], w, out[:M])
        assert torch.all(out[M] == 7.0)
        assert float((out[:M].double() - ref[:M]).abs().max()) <= 8 * bound, M
        if whole is None:
            whole = out[:M].clone()
        assert torch.equal(out[:M], whole[:M]), f"{M} rows: other bits than among {max(ROWS)}"
    ops.check_kernel_status()
