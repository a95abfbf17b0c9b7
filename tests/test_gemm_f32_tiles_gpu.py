"""The 32-bit product's tiles beyond 32 rows, each at sizes for which the rule takes it (ragged rows and columns among them): the bits of
single rows, which another kernel forms, and the 64-bit sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# outputs to a thread: 4 x 16, 6 x 16, 8 x 12, 8 x 16, 10 x 12, 11 x 14, 11 x 12, then several row tiles
@pytest.mark.parametrize("M, N", [(33, 1000), (65, 2503), (97, 2503), (97, 3505), (129, 2503), (129, 3505), (161, 2503),
                                  (300, 3072), (353, 3000)])
def test_every_tile_has_the_bits_of_single_rows(M, N, K=260):
    from allpaca_b200 import ops
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
