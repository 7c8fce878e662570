"""Schedules that recompute layers in the backward pass run the output head once per microbatch: its forward feeds nothing
but the loss, which the recomputation gives."""
import pytest
import torch

from zorse_b200.config.training_config import parse_pipeline_dict
from zorse_b200.models.layers import HeadLayer
from zorse_b200.trainer import Trainer, TrainerOptions


@pytest.mark.parametrize("schedule", ["zero2", "layer_major", "1f1b"])
def test_the_head_runs_once_and_the_step_is_the_same(monkeypatch, schedule):
    cfg = parse_pipeline_dict({
        "model_name": "tiny_llama", "global_batch_size": 3, "microbatch_size": 1, "sequence_length": 32, "vocab_size": 256,
        "autocast_dtype": "float32", "reduce_dtype": "float32",
        "pipeline_config": [{"gpu_ranks": [0], "num_microbatches_per_rank": [3], "layer_partition": [0, 2],
                             "zero_config": [[0]]}]})
    calls = []
    forward = HeadLayer.forward
    monkeypatch.setattr(HeadLayer, "forward", lambda self, *a, **k: calls.append(0) or forward(self, *a, **k))
    got = []
    for recompute in (False, True):
        tr = Trainer(cfg, TrainerOptions(schedule=schedule, ops="ref", activation_recompute=recompute, model_overrides={"layers": 2}))
        batch = tr.synthetic_batch(5)
        calls.clear()
        losses = [tr.train_step_from_host(batch) for _ in range(2)]
        assert len(calls) == 2 * 3
        got.append((losses, [t for st in tr.stages for u in st.engine.units for t in u.state_tensors().values()]))
    (l0, s0), (l1, s1) = got
    # the same fp32 operations; the three losses are added in the order of the backward pass
    assert l1 == pytest.approx(l0, rel=1e-6)
    for a, b in zip(s0, s1):
        torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-7)
