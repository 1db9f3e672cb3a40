"""The layer calls' workspaces: one per stream, given back, never shared by calls that may run at the same
time.  Results are compared bit for bit with the same call made alone (the layer is deterministic)."""
import gc
import threading
import time

import pytest
import torch

from gpu_utils import DEV

pytestmark = pytest.mark.gpu

E, K, H, I = 8, 2, 512, 256
SIZES = [1, 7, 40, 130, 400]


def _layer(native, seed=0, **kw):
    g = torch.Generator().manual_seed(seed)
    w13 = (torch.randn(E, H, 2 * I, generator=g) * H ** -0.5).to(torch.bfloat16).to(DEV)
    w2 = (torch.randn(E, I, H, generator=g) * I ** -0.5).to(torch.bfloat16).to(DEV)
    return native.XpuFusedMoe(w13, None, None, w2, None, None, K, "silu", E, **kw)


def _call(T, seed=0):
    """(output, hidden states, routing weights, ids) of a call with T tokens."""
    g = torch.Generator().manual_seed(1000 * seed + T)
    w, ids = torch.topk(torch.softmax(torch.randn(T, E, generator=g), -1), k=K, dim=-1)
    return (torch.empty(T, H, dtype=torch.bfloat16, device=DEV),
            torch.randn(T, H, generator=g).to(torch.bfloat16).to(DEV), w.to(DEV), ids.int().to(DEV))


def _alone(native, layer, call):
    out = torch.empty_like(call[0])
    layer.apply(out, *call[1:])
    torch.cuda.synchronize()
    return out


def _in_use():
    gc.collect()
    torch.cuda.synchronize()
    return torch.cuda.memory_allocated()


def test_graphs_replay_beside_other_calls_and_give_their_memory_back(native):
    """Two graphs captured on one stream and replayed at the same time on two others, beside calls made on
    the stream of the capture; their intermediates go with them."""
    layer = _layer(native)
    calls = [_call(T) for T in (400, 130, 40)]
    want = [_alone(native, layer, c) for c in calls]
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        layer.apply(*calls[2])
    before = _in_use()
    graphs = [torch.cuda.CUDAGraph() for _ in range(2)]
    for graph, call in zip(graphs, calls):
        with torch.cuda.graph(graph, stream=side):
            layer.apply(*call)
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(20):
        for c in calls:
            c[0].fill_(float("nan"))
        torch.cuda.synchronize()
        for _ in range(5):
            for graph, stream in zip(graphs, streams):
                with torch.cuda.stream(stream):
                    graph.replay()
            with torch.cuda.stream(side):
                layer.apply(*calls[2])
        torch.cuda.synchronize()
        for c, ref in zip(calls, want):
            assert torch.equal(c[0], ref)
    del graphs, graph
    assert _in_use() == before


def test_other_threads_run_while_a_launch_waits(native):
    """Calls behind a sleeping stream fill its launch queue: the call that then waits for a place must not
    hold the interpreter (what the stream waits for may need it)."""
    layer, call = _layer(native), _call(7)
    layer.apply(*call)
    torch.cuda.synchronize()
    ticks, done = [], threading.Event()

    def tick():
        while not done.is_set():
            ticks.append(time.monotonic())
            time.sleep(0.002)

    other = threading.Thread(target=tick)
    other.start()
    torch.cuda._sleep(10 ** 9)            # cycles: half a second
    for _ in range(500):
        layer.apply(*call)                # several launches each, more than a queue holds
    done.set()
    other.join()
    torch.cuda.synchronize()
    assert max(b - a for a, b in zip(ticks, ticks[1:])) < 0.15


@pytest.mark.parametrize("streams", [1, 3])
def test_threads_and_streams_do_not_meet(native, streams):
    """Threads that call layers of different sizes at the same time, on one stream or on one each."""
    layer = _layer(native)
    calls = [_call(T) for T in SIZES[-3:]]
    want = [_alone(native, layer, c) for c in calls]
    own = [torch.cuda.Stream() for _ in range(streams)]
    failed = []

    def work(i):
        with torch.cuda.stream(own[i % streams]):
            for _ in range(60):
                calls[i][0].fill_(float("nan"))
                layer.apply(*calls[i])
                same = torch.equal(calls[i][0], want[i])
                if not same:
                    failed.append(i)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed


def test_a_stage_hook_may_call_a_layer(native):
    layer, inner, call, other = _layer(native), _layer(native, seed=1), _call(40), _call(400)
    want, want_inner = _alone(native, layer, call), _alone(native, inner, other)
    stages = []

    def hook(stage):
        stages.append(stage)
        inner.apply(*other)

    layer.stage_hook = hook
    layer.apply(*call)
    torch.cuda.synchronize()
    assert stages == ["routing", "permute", "gemm1", "activation", "gemm2", "gather"]
    assert torch.equal(call[0], want) and torch.equal(other[0], want_inner)

    def fail(stage):
        raise ValueError(stage)

    layer.stage_hook = fail
    with pytest.raises(ValueError, match="routing"):
        layer.apply(*call)
    layer.stage_hook = None
    assert torch.equal(_alone(native, layer, call), want)


def test_more_streams_than_workspaces(native):
    """Twelve streams take turns: eight keep a buffer, the least recently used one is given back while its
    stream may still be at work."""
    layer = _layer(native)
    streams = [torch.cuda.Stream() for _ in range(12)]
    calls = [_call(T, seed=i) for i, T in enumerate((SIZES * 3)[:12])]
    want = [_alone(native, layer, c) for c in calls]
    native._WORKSPACE.clear()
    before = _in_use()
    with torch.cuda.stream(streams[0]):
        layer.apply(*calls[0])
    one = _in_use() - before
    assert one > 0
    for _ in range(10):
        for c in calls:
            c[0].fill_(float("nan"))
        torch.cuda.synchronize()
        for _ in range(3):
            for s, c in zip(streams, calls):
                with torch.cuda.stream(s):
                    layer.apply(*c)
        torch.cuda.synchronize()
        for c, ref in zip(calls, want):
            assert torch.equal(c[0], ref)
    kept = _in_use() - before
    native._WORKSPACE.clear()
    assert _in_use() == before
    for s in streams:                     # equal sizes: eight buffers of the twelve streams
        with torch.cuda.stream(s):
            layer.apply(*calls[0])
    assert _in_use() - before == 8 * one and kept > 0
    native._WORKSPACE.clear()


def test_the_last_layer_gives_the_workspaces_back(native):
    call = _call(40)
    gc.collect()
    native._WORKSPACE.clear()
    before = _in_use()
    layers = [_layer(native, seed=s) for s in range(2)]
    weights = _in_use() - before
    for layer in layers:
        layer.apply(*call)
    assert _in_use() > before + weights
    del layer
    layers.pop()
    assert _in_use() > before + weights // 2       # the other layer's call may come next
    layers.pop()
    assert _in_use() == before


def test_setting_an_attribute_of_the_plan_counts_from_the_next_call(native):
    call = _call(40)
    layer, other = _layer(native), _layer(native, seed=1)
    first = _alone(native, layer, call)
    g = torch.Generator().manual_seed(3)
    bias = torch.randn(E, H, generator=g).to(torch.bfloat16).to(DEV)
    for name, value in (("w2", other.w2), ("w2_bias", bias), ("gemm1_clamp_limit", 0.25)):
        fresh = _layer(native)
        setattr(fresh, name, value)               # before its first call: there is no plan yet
        setattr(layer, name, value)
        got = _alone(native, layer, call)
        assert not torch.equal(got, first) and torch.equal(got, _alone(native, fresh, call))
        setattr(layer, name, getattr(_layer(native), name))
        assert torch.equal(_alone(native, layer, call), first)


def test_a_call_looks_at_the_weights_as_they_are(native):
    """Weights that get other memory in place (a reload) are used from the next call on, ones that no longer
    fit are refused."""
    call = _call(40)
    layer = _layer(native)
    first = _alone(native, layer, call)
    w2 = layer.w2.clone()
    layer.w2.data = w2 * 2
    got = _alone(native, layer, call)
    fresh = _layer(native)
    fresh.w2 = w2 * 2
    assert not torch.equal(got, first) and torch.equal(got, _alone(native, fresh, call))
    for wrong in (w2[:, :, :-8].contiguous(), w2[:-1].contiguous(), w2.half(), w2.transpose(1, 2).contiguous().transpose(1, 2)):
        layer.w2.data = wrong
        with pytest.raises(RuntimeError, match="ptr_B|weights of the activation dtype"):
            layer.apply(*call)
    layer.w2.data = w2
    assert torch.equal(_alone(native, layer, call), first)
