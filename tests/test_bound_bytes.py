"""What the parts lay out anew when they are bound counts towards the memory that is left for pages."""

import pytest
import torch

import dizatar_tiny as tiny
from freetoken_b200.models.model import Model
from freetoken_b200.registry import architecture_of
from freetoken_b200.weights import random_state


def bound(config, dtype):                 # the random checkpoint holds bfloat16, whatever it is computed in
    arch = architecture_of(config)
    model = Model(arch.build_plan(arch.read_config(config)))
    tensors = random_state(model.tensor_specs(), 0, "cpu", dtype)
    model.bind(tensors, dtype)
    return model, model.bound_bytes(tensors)


def transposed_keys(config, item, taken=lambda m: True):
    return sum(m["heads"] * m["dim"] * m["kv_rank"] * item for m in (layer["mixer"] for layer in config["layers"]) if taken(m))


def without_experts(config):
    return dict(config, layers=[dict(layer, mlp=None) for layer in config["layers"]])


@pytest.mark.parametrize("config", [without_experts(tiny.DZ_A), without_experts(tiny.DZ_B)])
def test_copies_of_latent_keys_are_counted_and_made_where_they_are_used(config):
    streams = lambda m: m["dim"] % 8 == 0 and (m["dim"] + m["rot_dim"]) % 8 == 0
    for dtype, want in ((torch.float32, transposed_keys(config, 2)), (torch.bfloat16, transposed_keys(config, 2, streams))):
        model, counted = bound(config, dtype)
        held = [t for part in model.leaf_parts() for name, t in vars(part).items() if name == "w_ukt" and t is not None]
        assert sum(t.numel() * t.element_size() for t in held) == want
        folded = [t for part in model.leaf_parts() if type(part).__name__ == "RMSNorm" for t in [part.weight]]
        assert want <= counted <= want + sum(t.numel() * 4 for t in folded)
    assert transposed_keys(tiny.DZ_A, 2, streams) == 0 < transposed_keys(tiny.DZ_B, 2, streams)


def test_tensors_as_they_were_loaded_are_not_counted_again():
    model, counted = bound(without_experts(tiny.DZ_A), torch.bfloat16)
    assert counted < 1024                                  # folded norm weights
    # a router is kept in its bfloat16 terms, a copy
    assert bound(tiny.DZ_A, torch.bfloat16)[1] > counted

    class Holds:
        children = staticmethod(lambda: [])
    part = Holds()
    model.parts = lambda: [part]
    own = torch.zeros(1000, dtype=torch.float32)
    tensors = {"a": torch.zeros(64)}
    part.a, part.view, part.twice, part.rows = tensors["a"], tensors["a"][8:], own, {"x": [own[1:], (own,)]}
    assert model.bound_bytes(tensors) == 4000
