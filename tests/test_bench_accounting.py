"""The byte and FLOP counts that bench.py divides by time are checked against the
tensors the model declares (no device needed)."""
import inspect
import os
import sys
from types import SimpleNamespace

import pytest
import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402
from inferx_b200.parts.feed_forward import MoeFeedForward  # noqa: E402
from inferx_b200.weights.random_model import declared_tensors  # noqa: E402


def _numel(shape):
    n = 1
    for x in shape:
        n *= x
    return n


@pytest.mark.parametrize("cfg", [bench.A27B, bench.Q57B], ids=["a2.7b", "57b-a14b"])
def test_weight_bytes_match_the_declared_tensors(cfg):
    declared = sum(_numel(d.shape) * (2 if d.keep == "param" else 4) for d in declared_tensors(cfg))
    wb = bench.weight_bytes(cfg)
    counted = wb["layers"] * (wb["per_layer_fixed"] + cfg["num_experts"] * wb["per_expert"]) \
        + 2 * wb["head"]
    assert abs(counted - declared) <= 1e-5 * declared


def test_decode_step_bytes_are_weights_used_once_plus_the_live_cache():
    cfg = bench.A27B
    wb = bench.weight_bytes(cfg)
    touched, batch, context = 25.5, 8, 4096
    got = bench.decode_step_bytes(cfg, batch, context, touched)
    kv = batch * context * 2 * cfg["num_key_value_heads"] * cfg["head_dim"] * 2 * cfg["num_hidden_layers"]
    want = wb["layers"] * (wb["per_layer_fixed"] + touched * wb["per_expert"]) + wb["head"] + kv
    assert abs(got - want) <= 1e-4 * want
    assert 19.5e9 < got < 20.5e9          # worked out by hand for this point: about 20.1 GB


def test_prefill_flops_of_the_headline_prompt():
    fl = bench.prefill_flops(bench.A27B, 2048)
    assert 8.8e12 < fl < 8.95e12          # 8.47 TFLOP of products + 0.41 TFLOP of attention


def test_experts_of_a_step_are_counted_however_its_layers_route():
    """One call that selects and makes the tables, that call made of the two others, and tables
    alone: every layer once.  A count of nothing is refused, not divided by."""
    ops = SimpleNamespace()
    ops.moe_dispatch = lambda idx, experts, topk_w=None: (idx, "tables")
    ops.router_dispatch = lambda x, one_call: (
        (None, x, None) if one_call else (None, ops.moe_dispatch(x, 8, topk_w=None)[0], None))
    kept = ops.router_dispatch, ops.moe_dispatch
    chosen = torch.tensor([[0, 3], [3, 5], [0, 5]])
    with bench.counted_experts(ops) as seen:
        assert ops.router_dispatch(chosen, True)[1] is chosen
        ops.router_dispatch(chosen[:1], False)
        assert ops.moe_dispatch(chosen[:, :1], 8)[1] == "tables"
    assert seen == [3, 2, 2] and (ops.router_dispatch, ops.moe_dispatch) == kept
    assert bench.mean_experts(seen) == pytest.approx(7 / 3)
    for nothing in ([], [0, 0]):
        with pytest.raises(RuntimeError):
            bench.mean_experts(nothing)


def test_routing_has_a_line_in_every_table_of_faces():
    """What a mixture layer calls to route is among the faces that are timed and left out."""
    layer = inspect.getsource(MoeFeedForward)
    for table in (bench.breakdown, bench.marginal):
        text = inspect.getsource(table)
        for name in ("router_dispatch", "router_topk", "moe_dispatch"):
            assert f"ops.{name}(" in layer and f'"{name}"' in text
