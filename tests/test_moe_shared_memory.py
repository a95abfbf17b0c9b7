"""A shared expert's matrices are held once: those that ride in the routed experts' launches are the shared part's own."""
import pytest
import torch

from allpaca_b200.parts import BuildEnv, Workspace
from allpaca_b200.parts.base import PartSpec, build


@pytest.mark.parametrize("gated,activation", [(True, "silu"), (False, "relu2")])
def test_shared_matrices_are_held_once(gated, activation):
    H, F, S, E = 32, 16, 24, 4
    env = BuildEnv(dtype=torch.bfloat16, device=torch.device("cpu"), workspace=Workspace(torch.device("cpu")), page_size=16, max_seqs=1)
    part = build("feed_forward", PartSpec("routed_experts", {
        "hidden_size": H, "expert_size": F, "experts": E, "top": 2, "activation": activation, "gated": gated, "router_bias": False,
        "shared": {"size": S}}), env)
    part.load({n: torch.randn(s.shape).to(torch.bfloat16) for n, s in part.weights().items()})
    held = {}

    def walk(o):
        for v in vars(o).values():
            if isinstance(v, torch.Tensor):
                held[v.untyped_storage().data_ptr()] = v.untyped_storage().nbytes()
            elif type(v).__module__.startswith("allpaca_b200.parts") and not isinstance(v, BuildEnv):
                walk(v)
    walk(part)
    numbers = E * H + E * F * H * (3 if gated else 2) + S * H * (3 if gated else 2)
    assert sum(held.values()) == 2 * numbers
    assert part.shared_first is not None and part.shared_down is not None
