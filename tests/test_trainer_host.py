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


class _Kept(torch.autograd.Function):
    """Hands a product to a queue in backward, or fails."""

    @staticmethod
    def forward(ctx, x, queue, sink, fail):
        ctx.queue, ctx.sink, ctx.fail = queue, sink, fail
        return x.clone()

    @staticmethod
    def backward(ctx, dy):
        if ctx.fail:
            raise ValueError("on purpose")
        ctx.queue(ctx.sink)
        return dy, None, None, None


@pytest.fixture
def launches(monkeypatch):
    """The queues of weight gradients on the host: what they would launch."""
    import contextlib
    from mccl_b200.ops import native
    seen = []
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: None)
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
    monkeypatch.setattr(native._C, "gemm_group", lambda items, accumulate: seen.append([it[2] for it in items]))
    monkeypatch.setattr(native._C, "decoder_layer_wgrads", lambda items, B, S, H: seen.append([it[0] for it in items]))
    return seen


def _param(awaited, *shape):
    p = torch.nn.Parameter(torch.zeros(*shape))
    p._grad_awaited = awaited
    return p


def _single(sink, awaited=False):
    from mccl_b200.ops import native
    native._products.add(torch.zeros(8, 16), torch.zeros(8, 16), sink, _param(awaited, 16, 16))


def _layer(sink, awaited=False):
    from mccl_b200.ops import native
    params = tuple(_param(awaited, 4) for _ in range(12))
    native._deferred.add((sink, None, None, [torch.zeros(4)] * 12), (1, 8, 1), params, torch.device("cpu"))


@pytest.mark.parametrize("queue", [_single, _layer])
def test_a_failed_backward_leaves_nothing_for_the_next(launches, queue):
    from mccl_b200.ops import native
    x = torch.ones(3, requires_grad=True)
    with pytest.raises(ValueError):
        _Kept.apply(_Kept.apply(x, queue, "lost", True), queue, "stale", False).sum().backward()
    _Kept.apply(_Kept.apply(x, queue, "a", False), queue, "b", False).sum().backward()
    assert launches == [["b", "a"]]
    native.join_wgrad()
    assert launches == [["b", "a"]]
    # a pass inside another one (activation checkpointing) keeps its own
    class Inner(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x):
            return x.clone()

        @staticmethod
        def backward(ctx, dy):
            with torch.enable_grad():
                _Kept.apply(torch.ones(3, requires_grad=True), queue, "inner", False).sum().backward()
            return dy
    launches.clear()
    _Kept.apply(Inner.apply(_Kept.apply(x, queue, "first", False)), queue, "last", False).sum().backward()
    assert launches == [["inner"], ["last", "first"]]


@pytest.mark.parametrize("queue", [_single, _layer])
def test_gradients_that_peers_wait_for_are_not_kept_back(launches, queue):
    x = torch.ones(3, requires_grad=True)
    for name in "abc":
        x = _Kept.apply(x, lambda sink: queue(sink, True), name, False)
    x.sum().backward()
    assert launches == [["c"], ["b"], ["a"]]


@pytest.mark.parametrize("world", [1, 2])
def test_trainer_says_whether_peers_wait(monkeypatch, world):
    import mccl_b200
    from mccl_b200.models import build_decoder
    from mccl_b200.parallel import DDPTrainer, trainer
    backend = type("Backend", (), {"device_comm": lambda self, index: object()})()
    monkeypatch.setattr(trainer.dist, "is_initialized", lambda: world > 1)
    monkeypatch.setattr(trainer.dist, "get_world_size", lambda group=None: world)
    monkeypatch.setattr(trainer.dist, "get_rank", lambda group=None: 0)
    monkeypatch.setattr(mccl_b200, "get_backend", lambda group=None: backend)
    monkeypatch.setattr(DDPTrainer, "_sync_initial_params", lambda self, group: None)
    t = DDPTrainer(build_decoder("tiny"), torch.device("cpu"), use_graph=False)
    assert all(getattr(p, "_grad_awaited", False) == (world > 1) for p in t.model.parameters())


def test_products_wait_by_the_sms_they_may_use(launches, monkeypatch):
    """Half of the tiles that the GPU works on at a time: on 148 SMs, on fewer, and with a cap on the CTAs of products."""
    from mccl_b200.ops import native
    alone = []
    monkeypatch.setattr(native, "_wgrad_gemm", lambda dz, x2, sink: alone.append(sink))

    def queue(sink):   # 4 x 5 tiles
        native._products.add(torch.zeros(8, 1024), torch.zeros(8, 1280), sink, _param(False, 1024, 1280))
    for sms, cap, waits in ((148, 0, True), (148, 88, True), (148, 78, False), (80, 0, True), (78, 0, False)):
        monkeypatch.setattr(native._C, "gemm_sm_count", lambda: sms)
        monkeypatch.setattr(native._C, "gemm_cta_limit", lambda: cap)
        launches.clear()
        alone.clear()
        _Kept.apply(torch.ones(3, requires_grad=True), queue, "a", False).sum().backward()
        assert (launches, alone) == (([["a"]], []) if waits else ([], ["a"])), (sms, cap)
    monkeypatch.setattr(native._C, "gemm_sm_count", lambda: 148)
    monkeypatch.setattr(native._C, "gemm_cta_limit", lambda: 0)
    assert native._products.limits() == (37, 64)
