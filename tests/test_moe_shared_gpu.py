"""A shared expert in the routed experts' launches against 64 bits: on the tensor cores (every tile size, sizes of its own wider
and narrower than the routed ones, one row and rows of several tiles) and on the CUDA cores (one to more rows than are held at
once), gated and not; without any routed row too."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def act(name, z, gated):
    if name is None:
        return z
    n = z.shape[1] // 2
    g, u = (z[:, :n], z[:, n:]) if gated else (z, torch.ones_like(z))
    return (torch.nn.functional.silu(g) if name == "silu" else torch.relu(g) ** 2) * u


def near(got, want, rounded):
    # 32-bit sums of unit size; bfloat16 stores seven bits
    tol = 2e-5 + (2.0 ** -8 * want.abs() if rounded else 0.0)
    assert bool(((got.double().cpu() - want).abs() <= tol).all()), float((got.double().cpu() - want).abs().max())


def matrix(g, *shape):
    return (torch.randn(*shape, generator=g) * shape[-1] ** -0.5).to(torch.bfloat16)


@pytest.mark.parametrize("counts,T", [([0, 1, 5], 1), ([20, 3, 33], 17), ([40, 64, 41], 65), ([130, 60, 200], 129), ([0, 0], 33)])
@pytest.mark.parametrize("gated,name,N,K,XN,XK", [(True, "silu", 200, 136, 72, 136), (False, "relu2", 72, 64, 392, 200),
                                                  (False, None, 264, 72, 264, 1032)])
def test_beside_the_products_on_the_tensor_cores(counts, T, gated, name, N, K, XN, XK):
    from allpaca_b200 import ops
    g = torch.Generator().manual_seed(T + N)
    E, pairs = len(counts), max(1, sum(counts))
    a, w = torch.randn(pairs, K, generator=g).to(torch.bfloat16), matrix(g, E, 2 * N if gated else N, K)
    xa, xw = torch.randn(T, XK, generator=g).to(torch.bfloat16), matrix(g, 2 * XN if gated else XN, XK)
    first = [sum(counts[:e]) for e in range(E + 1)]
    dt = torch.float32 if name is None else torch.bfloat16
    out, xout = torch.zeros(pairs, N, dtype=dt, device=DEV), torch.zeros(T, XN, dtype=dt, device=DEV)
    ops.moe_products(a.to(DEV), w.to(DEV), out, torch.tensor(first, dtype=torch.int32, device=DEV), gated=gated, activation=name,
                     shared=(xa.to(DEV), xw.to(DEV), xout))
    ops.check_kernel_status()
    near(xout, act(name, xa.double() @ xw.double().T, gated), name is not None)
    for e in range(E):
        r = slice(first[e], first[e + 1])
        near(out[r], act(name, a[r].double() @ w[e].double().T, gated), name is not None)


@pytest.mark.parametrize("T,top,E", [(1, 1, 3), (3, 2, 5), (9, 2, 4), (19, 1, 2)])
@pytest.mark.parametrize("gated,name,F,K,XF", [(True, "silu", 40, 1288, 24), (False, "relu2", 33, 200, 72)])
def test_beside_the_products_of_few_rows(T, top, E, gated, name, F, K, XF):
    from allpaca_b200 import ops
    g = torch.Generator().manual_seed(T + K)
    pairs, H = T * top, 56
    F8 = (F + 7) // 8 * 8                                 # the second product reads whole 16-byte runs
    h = torch.randn(T, K, generator=g).to(torch.bfloat16)
    w, down = matrix(g, E, 2 * F8 if gated else F8, K), matrix(g, E, H, F8)
    xw, xdown = matrix(g, 2 * XF if gated else XF, K), matrix(g, H, XF)
    chosen = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(T)]).to(torch.int32).to(DEV)
    perm, place = (torch.empty(pairs, dtype=torch.int32, device=DEV) for _ in range(2))
    tiles = torch.zeros(ops.moe_max_tiles(pairs, E) + 1, 3, dtype=torch.int32, device=DEV)
    ops.moe_sort(chosen, perm, place, tiles, E)
    hd, wd, dd = h.to(DEV), w.to(DEV), down.to(DEV)
    y, ys = torch.zeros(pairs, F8, dtype=torch.bfloat16, device=DEV), torch.zeros(T, XF, dtype=torch.bfloat16, device=DEV)
    o, os_ = torch.zeros(pairs, H, device=DEV), torch.zeros(T, H, device=DEV)
    assert ops.moe_rows_taken(hd, wd, pairs, E) and ops.moe_rows_taken(y, dd, pairs, E)
    ops.moe_gate_up(hd, wd, y, perm, top, tiles, name, gated=gated, shared=(hd, xw.to(DEV), ys))
    ops.moe_down(y, dd, o, tiles, shared=(ys, xdown.to(DEV), os_))
    near(ys, act(name, h.double() @ xw.double().T, gated), True)
    near(os_, ys.double().cpu() @ xdown.double().T, False)
    for p, pair in enumerate(perm.cpu().tolist()):
        e = int(chosen.view(-1)[pair])
        near(y[p:p + 1], act(name, h[pair // top][None].double() @ w[e].double().T, gated), True)
        near(o[p:p + 1], y[p:p + 1].double().cpu() @ down[e].double().T, False)


@pytest.mark.parametrize("T", [1, 70])
@pytest.mark.parametrize("gated,name", [(True, "silu"), (False, "relu2")])
def test_a_shared_expert_without_any_pair(T, gated, name):
    """No row goes to a routed expert: the shared one's results are there all the same, in each of the three calls."""
    from allpaca_b200 import ops
    g = torch.Generator().manual_seed(T)
    E, N, K, XN, XK = 3, 40, 64, 72, 128
    xa, xw, xdown = torch.randn(T, XK, generator=g).to(torch.bfloat16), matrix(g, 2 * XN if gated else XN, XK), matrix(g, 48, XN)
    w, down = matrix(g, E, 2 * N if gated else N, K).to(DEV), matrix(g, E, N, K).to(DEV)
    a, none = torch.empty(0, K, dtype=torch.bfloat16, device=DEV), torch.empty(0, dtype=torch.int32, device=DEV)
    y = torch.empty(0, N, dtype=torch.bfloat16, device=DEV)
    first = torch.full((E + 1,), 5, dtype=torch.int32, device=DEV)          # not looked at
    tiles = torch.full((ops.moe_max_tiles(0, E) + 1, 3), 5, dtype=torch.int32, device=DEV)
    want = act(name, xa.double() @ xw.double().T, gated)
    outs = [torch.zeros(T, XN, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    ops.moe_products(a, w, y, first, gated=gated, activation=name, shared=(xa.to(DEV), xw.to(DEV), outs[0]))
    ops.moe_gate_up(a, w, y, none, 1, tiles, name, gated=gated, shared=(xa.to(DEV), xw.to(DEV), outs[1]))
    sums = torch.zeros(T, 48, device=DEV)
    ops.moe_down(a, down, torch.empty(0, N, device=DEV), tiles, shared=(outs[1], xdown.to(DEV), sums))
    ops.check_kernel_status()
    for out in outs:
        near(out, want, True)
    near(sums, outs[1].double().cpu() @ xdown.double().T, False)


@pytest.mark.parametrize("T", [1, 40, 300])
@pytest.mark.parametrize("activation", ["silu", "relu"])
def test_a_gated_feed_forward_held_in_halves(T, activation):
    """What a shared expert runs as where it cannot ride, against 64 bits: the sums stay in 32 bits up to the activation."""
    from allpaca_b200.parts import BuildEnv, Workspace
    from allpaca_b200.parts.base import PartSpec, build
    H, S = 72, 136
    g = torch.Generator().manual_seed(T)
    h = torch.randn(T, H, generator=g).to(torch.bfloat16)
    tensors = {"gate_proj.weight": matrix(g, S, H), "up_proj.weight": matrix(g, S, H), "down_proj.weight": matrix(g, H, S)}
    z, u = (h.double() @ tensors[n].double().T for n in ("gate_proj.weight", "up_proj.weight"))
    mid = (torch.nn.functional.silu(z) if activation == "silu" else torch.relu(z)) * u
    want = mid @ tensors["down_proj.weight"].double().T
    env = BuildEnv(dtype=torch.bfloat16, device=torch.device(DEV), workspace=Workspace(torch.device(DEV)), page_size=16, max_seqs=1)
    part = build("feed_forward", PartSpec("swiglu", {"hidden_size": H, "intermediate_size": S, "activation": activation,
                                                     "halves": True}), env)
    part.load({n: t.to(DEV) for n, t in tensors.items()})
    got = part.forward(h.to(DEV), None)[0].double().cpu()
    # the activation is stored in bfloat16: half a unit in the last place of each of the S terms, whose squares add up
    tol = 6 * 2.0 ** -9 * torch.sqrt((mid ** 2) @ (tensors["down_proj.weight"].double() ** 2).T) + 2e-5
    assert bool(((got - want).abs() <= tol).all()), float(((got - want).abs() / tol).max())
