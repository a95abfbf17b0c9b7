"""The experts' products on the tensor cores against 64 bits: experts without rows, with one, with a whole tile of rows and
one more, at averages that choose every tile size; widths that end inside a tile of weight rows and inside a block of K;
gated and not, with shares on the inputs, 32-bit results of the second product; rows behind the last expert stay as they are."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def act(name, g, u, limit, alpha, shift):
    if name == "silu":
        return torch.nn.functional.silu(g) * u
    if name == "relu2":
        return torch.relu(g) ** 2 * u
    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return g * torch.sigmoid(alpha * g) * (u + shift)


@pytest.mark.parametrize("counts", [[0, 1, 16, 3, 0, 17, 1], [31, 0, 33, 5, 1], [64, 0, 65, 1], [128, 129, 0, 1, 300, 257],
                                    [1]])
@pytest.mark.parametrize("gated,name,N,K", [(True, "silu", 200, 136), (True, "clamped_sigmoid", 128, 64),
                                            (False, "relu2", 264, 72), (False, None, 72, 1032)])
def test_products_of_all_experts(counts, gated, name, N, K):
    from allpaca_b200 import ops
    gen = torch.Generator().manual_seed(sum(counts) + N)
    E, behind = len(counts), 5
    pairs = sum(counts) + behind
    a = torch.randn(pairs, K, generator=gen).to(torch.bfloat16)
    w = (torch.randn(E, 2 * N if gated else N, K, generator=gen) * K ** -0.5).to(torch.bfloat16)
    perm = torch.randperm(pairs, generator=gen)
    scale = 0.25 + torch.rand(pairs, generator=gen)
    first = [sum(counts[:e]) for e in range(E + 1)]
    out = torch.full((pairs, N), 7.0, dtype=torch.float32 if name is None else torch.bfloat16, device=DEV)
    scaled = name == "silu"
    ops.moe_products(a.to(DEV), w.to(DEV), out, torch.tensor(first + [pairs], dtype=torch.int32, device=DEV), gated=gated,
                     activation=name, limit=1.5, alpha=1.7, shift=1.0, pair_scale=scale.to(DEV) if scaled else None,
                     perm=perm.to(torch.int32).to(DEV) if scaled else None)
    ops.check_kernel_status()
    got = out.double().cpu()
    assert bool((got[first[-1]:] == 7.0).all())
    for e in range(E):
        rows = slice(first[e], first[e + 1])
        z = a[rows].double() @ w[e].double().T
        if scaled:
            z = z * scale[perm[rows]].double()[:, None]
        g, u = (z[:, :N], z[:, N:]) if gated else (z, torch.ones_like(z))
        want = z if name is None else act(name, g, u, 1.5, 1.7, 1.0)
        # a sum of K products of unit size is off by about K^0.5 units of 2^-24 of its terms; bfloat16 stores seven bits
        tol = 2e-5 + (0.0 if name is None else 2.0 ** -8 * want.abs())
        assert bool(((got[rows] - want).abs() <= tol).all()), (e, float((got[rows] - want).abs().max()))


@pytest.mark.parametrize("rows", [1, 40, 300])
@pytest.mark.parametrize("name", ["silu", "clamped_sigmoid"])
def test_gates_far_below_zero_keep_their_small_results(name, rows):
    """1 + exp(88) is a 32-bit number, so a gate of -88 is no zero: times a large second factor it shows."""
    from allpaca_b200 import ops
    N, K = 64, 64
    gates = torch.tensor([-87.0, -87.5, -88.0, -88.5, -80.0, -40.0, -5.0, 3.0]).repeat(N // 8)
    a, w = torch.zeros(rows, K), torch.zeros(1, 2 * N, K)
    a[:, 0] = 1.0
    w[0, :N, 0], w[0, N:, 0] = gates, 2.0 ** 100
    out = torch.empty(rows, N, dtype=torch.bfloat16, device=DEV)
    ops.moe_products(a.to(torch.bfloat16).to(DEV), w.to(torch.bfloat16).to(DEV), out,
                     torch.tensor([0, rows], dtype=torch.int32, device=DEV), gated=True, activation=name, limit=2.0 ** 101, alpha=1.0)
    ops.check_kernel_status()
    z = gates.double()
    want = (z / (1.0 + torch.exp(-z)) * 2.0 ** 100).expand(rows, N)
    # the exponential is off by some units of 2^-24, bfloat16 stores seven bits
    assert bool(((out.double().cpu() - want).abs() <= (2.0 ** -8 + 1e-5) * want.abs()).all()), (out[0, :8].cpu(), want[0, :8])
