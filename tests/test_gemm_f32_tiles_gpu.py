"""The 32-bit product's tiles beyond 32 rows, each at sizes for which the rule takes it (ragged rows and columns among them), with fewer
blocks of K to a CTA than the operand ring holds and with three times as many: the bits of single rows, which another kernel forms, and the 64-bit
sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# outputs to a thread as rows x 100 + columns; the last ones with several row tiles
@pytest.mark.parametrize("M, N, tile", [(33, 1000, 416), (65, 3505, 616), (65, 2503, 812), (97, 2503, 812), (97, 3505, 816), (129, 2503, 1012), (129, 3505, 1114),
                                        (161, 2503, 1112), (300, 3072, 1012), (353, 3000, 812), (512, 1000, 816), (700, 3072, 1112)])
@pytest.mark.parametrize("K", [260, 2052])
def test_every_tile_has_the_bits_of_single_rows(M, N, tile, K):
    from allpaca_b200 import ops
    assert ops.core().ap_gemm_f32_tile(M, N) == tile
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randn(M, K, generator=g, device="cuda")
    w = torch.randn(N, K, generator=g, device="cuda")
    out = torch.full((M + 1, N), 7.0, device="cuda")
    ops.gemm_simt(a, w, out[:M])
    assert torch.all(out[M] == 7.0)
    # as in test_gemm_f32_gpu.py: sums of K unit-variance terms, rounded to 2^-24 of partial sums
    assert float((out[:M].double() - a.double() @ w.double().T).abs().max()) <= 8 * (2.0 ** -24 * K + 1e-6)
    for r0 in (0, M // 2, M - 3):
        few = torch.empty(3, N, device="cuda")
        ops.gemm_simt(a[r0:r0 + 3], w, few)
        assert torch.equal(few, out[r0:r0 + 3])
    ops.check_kernel_status()
