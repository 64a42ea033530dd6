"""Optimizer updates during backward on one GPU against one update at the end."""
import pytest
import torch

pytestmark = pytest.mark.gpu


class _Mixed(torch.nn.Module):
    """A decoder whose layer weight is also used by a plain PyTorch operator: that share arrives after the native one's report."""

    def __init__(self, inner):
        super().__init__()
        self.inner = inner

    def forward(self, tokens, targets):
        return self.inner(tokens, targets) + self.inner.blocks[1].up.weight.square().mean()


@pytest.mark.parametrize("name,changes,mixed", [("tiny", {"n_layers": 6}, False), ("tiny", {"n_layers": 6}, True),
                                                ("1.3b", {"vocab": 512, "d_model": 256, "n_layers": 3, "n_heads": 4, "d_ff": 512, "max_seq": 256}, False)])
def test_updates_during_backward(monkeypatch, name, changes, mixed):
    from mccl_b200.models import build_decoder
    from mccl_b200.parallel import DDPTrainer
    dev = torch.device("cuda", 0)
    got = []
    for overlap in ("0", "1"):
        monkeypatch.setenv("MCCL_OVERLAP_ADAMW", overlap)
        torch.manual_seed(0)
        with dev:
            model = build_decoder(name, **changes)
        trainer = DDPTrainer(_Mixed(model) if mixed else model, dev, lr=1e-3, bucket_mb=0.25, last_bucket_mb=0.05)
        ids = torch.randint(0, model.cfg.vocab, (4, 65), device=dev, generator=torch.Generator(dev).manual_seed(1))
        for _ in range(4):
            loss = trainer.step(ids[:, :-1].contiguous(), ids[:, 1:].contiguous())
        torch.cuda.synchronize()
        if overlap == "1":
            assert trainer._local_overlap == (not mixed) and (trainer.opt_stream is not None) == (not mixed)
        got.append((float(loss), trainer.flat_p.clone(), trainer.m.clone()))
    (l0, p0, m0), (l1, p1, m1) = got
    assert abs(l0 - l1) < 2e-2 and (p0 - p1).norm() < 1e-3 * p0.norm() and (m0 - m1).norm() < 3e-2 * m0.norm()


@pytest.mark.parametrize("sizes,tokens", [([(1024, 1024), (3072, 1024), (1024, 1024)], 512), ([(256, 64), (64, 256), (128, 128), (8, 64), (512, 512)], 192), ([(64, 8192), (8192, 8192)], 128)])
def test_weight_gradients_that_share_a_launch(sizes, tokens):
    """Linear layers with gradient buffers, in turn, against each layer's own product."""
    from mccl_b200 import ops
    torch.manual_seed(tokens)
    got, want, ready = [], [], []
    total = 0
    for i, (n, k) in enumerate(sizes):
        x = torch.randn(tokens, k, device="cuda").bfloat16()
        w = torch.nn.Parameter(torch.randn(n, k, device="cuda") * 0.02)
        w._grad_sink = torch.ones(n, k, device="cuda")
        w._grad_ready = lambda i=i: ready.append(i)
        d = torch.randn(tokens, n, device="cuda").bfloat16()
        total = total + (ops.linear(x, w) * d).sum()
        got.append(w)
        want.append(d.float().t() @ x.float() + 1)
    total.backward()
    torch.cuda.synchronize()
    assert sorted(ready) == list(range(len(sizes)))
    for w, r in zip(got, want):
        assert ((w._grad_sink - r).norm() / r.norm()).item() < 1e-2 and w.grad is None


def test_trainers_come_and_go():
    """A dropped trainer is gone at once, and what the garbage collector finds does not disturb the next one's capture."""
    import gc
    import weakref
    from mccl_b200.models import build_decoder
    from mccl_b200.parallel import DDPTrainer
    dev = torch.device("cuda", 0)
    ids = torch.randint(0, 512, (2, 65), device=dev)
    threshold = gc.get_threshold()
    gc.collect()
    gc.set_threshold(20, 2, 2)
    try:
        for _ in range(3):
            with dev:
                model = build_decoder("tiny")
            trainer = DDPTrainer(model, dev, lr=1e-3)
            trainer.cycle = trainer   # one that only the collector frees
            trainer.step(ids[:, :-1].contiguous(), ids[:, 1:].contiguous())
            torch.cuda.synchronize()
    finally:
        gc.set_threshold(*threshold)
    del trainer.cycle
    gone = weakref.ref(trainer)
    del trainer
    assert gone() is None


@pytest.mark.parametrize("name,changes", [("tiny", {"n_layers": 3}), ("1.3b", {"vocab": 512, "d_model": 256, "n_layers": 3, "n_heads": 4, "d_ff": 512, "max_seq": 256})])
def test_a_step_that_failed_in_backward(name, changes):
    """Nothing of it is in the next step's gradients."""
    from mccl_b200.models import build_decoder
    from mccl_b200.parallel import DDPTrainer
    dev = torch.device("cuda", 0)
    ids = torch.randint(0, 512, (4, 65), device=dev)
    tok, tgt = ids[:, :-1].contiguous(), ids[:, 1:].contiguous()
    moments = []
    for fails in (False, True):
        torch.manual_seed(0)
        with dev:
            model = build_decoder(name, **changes)
        trainer = DDPTrainer(model, dev, use_graph=False)
        if fails:
            def stop(*_):
                raise ValueError("on purpose")
            handle = model.blocks[0].register_full_backward_hook(stop)
            with pytest.raises(ValueError):
                trainer.step(tok, tgt)
            handle.remove()
        trainer.step(tok, tgt)
        torch.cuda.synchronize()
        moments.append(trainer.m.clone())
    assert ((moments[0] - moments[1]).norm() / moments[0].norm()).item() < 1e-2
