"""Host side of the data-parallel engine, without a GPU."""
import pytest
import torch


@pytest.mark.parametrize("ctas", [1, 2, 8])
def test_optimizer_launch_takes_its_cap(monkeypatch, ctas):
    """The updates beside backward run with as many CTAs per SM as they were asked to."""
    from mccl_b200 import ops
    from mccl_b200.models import build_decoder
    from mccl_b200.parallel import DDPTrainer
    trainer = DDPTrainer(build_decoder("tiny"), torch.device("cpu"), use_graph=False)
    seen = []
    monkeypatch.setattr(ops, "adamw_step", lambda *a, **k: seen.append(k.get("ctas_per_sm")))
    trainer._adamw(0, 64, ctas)
    assert seen == [ctas]
