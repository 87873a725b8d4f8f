"""Whoever records operators and ranges sees a call's: the profiler, and an execution trace without a profiler."""

import contextlib
import json

import pytest
import torch
from torch.profiler import ExecutionTraceObserver, ProfilerActivity, profile

from dist_moe_b200 import _bf16, _call


@contextlib.contextmanager
def _trace(path):
    observer = ExecutionTraceObserver()
    observer.register_callback(str(path))
    observer.start()
    try:
        yield
    finally:
        observer.stop()
        observer.unregister_callback()


@pytest.mark.parametrize("recorder", ["profiler", "execution trace"])
def test_a_recorder_is_noticed(recorder, tmp_path):
    x = torch.zeros(2)
    assert not _call.observed() and _bf16._plain_execution(x)
    with profile(activities=[ProfilerActivity.CPU]) if recorder == "profiler" else _trace(tmp_path / "t.json"):
        assert _call.observed() and not _bf16._plain_execution(x)
        with _call.span("dist_moe_range"):
            pass
    assert not _call.observed() and _bf16._plain_execution(x)
    if recorder == "execution trace":
        assert "dist_moe_range" in {n["name"] for n in json.loads((tmp_path / "t.json").read_text())["nodes"]}


@pytest.mark.gpu
def test_an_execution_trace_holds_operators_and_ranges(tmp_path):
    import dist_moe_b200 as dm
    from tests.test_bf16_layer_gpu import make_case
    from tests.test_metrics_gpu import _step

    T, D, F, K, E = 64, 256, 256, 2, 4
    case = make_case(T, D, F, K, E, seed=43, w_scale=D**-0.5)
    cfg = dm.Config(max_num_local_input_tokens=T, hidden_dim=D, intermediate_dim=F, top_k=K, num_experts=E,
                    max_moe_layers_per_activation_slot=1)
    ctx = dm.create_context(group=None, config=cfg, device=0)
    try:
        with _trace(tmp_path / "t.json"):
            _step(dm, ctx, case)
        names = {n["name"] for n in json.loads((tmp_path / "t.json").read_text())["nodes"]}
        for want in ("dist_moe::bf16_forward", "dist_moe::bf16_backward", "dist_moe_preprocess", "dist_moe_routing",
                     "dist_moe_forward", "dist_moe_recompute", "dist_moe_backward"):
            assert want in names, (want, sorted(n for n in names if n.startswith("dist_moe")))
    finally:
        ctx.close()
