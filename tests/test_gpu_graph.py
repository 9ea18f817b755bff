"""A launch recorded in a CUDA graph must stay correct when it is replayed: the tile kernel keeps no state between
launches, and the weight-streaming kernel and the pair kernel's stream-K schedule (the last shape) take the epoch of
their hand-off flags from a counter in the workspace, not from the host.  Each replay runs on new activations written into the captured buffers."""
import pytest
import torch

from sol_execbench_b200_kernels_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(16, 4096, 8192), (8, 8192, 28672), (32, 8192, 28672), (256, 1024, 2048),
                                   (512, 384, 4864), (512, 4096, 14336)])
def test_replayed_graph_equals_eager_calls(shape):
    import sol_execbench_b200_kernels_b200 as pkg

    m, k, n = shape
    dev = torch.device("cuda:0")
    base = W.make_inputs(m, k, n, seed=3, device=dev)
    x = base.x.clone()
    sx = base.scale_x.clone()
    out = torch.empty(m, n, dtype=torch.bfloat16, device=dev)
    args = (x, sx, base.gate_proj_weight, base.scale_gate, base.up_proj_weight, base.scale_up, out)
    pkg.run(*args)                      # first call outside the capture: attributes, descriptors
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        pkg.run(*args)
    for trial in range(4):
        fresh = W.make_inputs(m, k, n, seed=10 + trial, device=dev)
        x.view(torch.uint8).copy_(fresh.x.view(torch.uint8))
        sx.copy_(fresh.scale_x)
        out.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert pkg.last_status()[0] == 0
        want = torch.empty_like(out)
        pkg.run(x, sx, base.gate_proj_weight, base.scale_gate, base.up_proj_weight, base.scale_up, want)
        torch.cuda.synchronize()
        assert torch.equal(out, want), f"replay {trial} of {shape} (plan {pkg.select_plan(m, k, n)})"


def test_replays_and_eager_calls_may_interleave_on_one_workspace():
    import sol_execbench_b200_kernels_b200 as pkg

    m, k, n = 16, 4096, 8192
    dev = torch.device("cuda:0")
    inp = W.make_inputs(m, k, n, seed=5, device=dev)
    out_a = torch.empty(m, n, dtype=torch.bfloat16, device=dev)
    out_b = torch.empty_like(out_a)
    pkg.run(*inp.args(), out_a)
    torch.cuda.synchronize()
    want = out_a.clone()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        pkg.run(*inp.args(), out_b)     # the workspace of this stream exists before the capture
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            pkg.run(*inp.args(), out_b)
        for _ in range(3):
            out_b.zero_()
            graph.replay()
            pkg.run(*inp.args(), out_a)
            graph.replay()
        stream.synchronize()
    torch.cuda.synchronize()
    assert pkg.last_status()[0] == 0
    assert torch.equal(out_a, want) and torch.equal(out_b, want)


def _run_call(m, k, n, plan="auto"):
    """A recorded call, its live input, inputs to put there, and the eager result for each of them."""
    import sol_execbench_b200_kernels_b200 as pkg

    base = W.make_inputs(m, k, n, seed=1, device="cuda:0")
    x = base.x.clone()
    out = torch.empty(m, n, dtype=torch.bfloat16, device="cuda:0")
    feeds = [W.make_inputs(m, k, n, seed=20 + i, device="cuda:0").x for i in range(2)]

    def call(dst=out):
        pkg.run_with_plan(x, base.scale_x, base.gate_proj_weight, base.scale_gate, base.up_proj_weight, base.scale_up, dst, plan)

    return call, x.view(torch.uint8), [f.view(torch.uint8) for f in feeds], out


def _mlp_call(m, k, n):
    import sol_execbench_b200_kernels_b200 as pkg

    g = torch.Generator(device="cuda:0").manual_seed(m)
    weights = []
    for rows, cols in ((n, k), (n, k), (k, n)):
        weights += W.quantize_weight_128x128(torch.randn(rows, cols, generator=g, device="cuda:0") * 0.02)
    x = torch.zeros(m, k, dtype=torch.bfloat16, device="cuda:0")
    feeds = [torch.randn(m, k, generator=g, device="cuda:0").bfloat16() for _ in range(2)]
    out = torch.empty_like(x)
    return (lambda dst=out: pkg.mlp_block(x, *weights, dst)), x, feeds, out


# the kernels that use scratch: weight streaming, the stream-K schedules of the pair and the lone-CTA kernel (whose stamp comes
# from the host and is recorded: a replay must find its flags zeroed), the MLP's steps
_WITH_SCRATCH = [(_run_call, (16, 4096, 8192)), (_run_call, (512, 4096, 14336)), (_run_call, (128, 4096, 14336, "tile_sk")),
                 (_mlp_call, (8, 4096, 11008))]


def _two_graphs(make, shape, pool=None):
    """Two graphs recorded on torch's one capture stream, with the eager results for both of their inputs."""
    calls = [make(*shape), make(*shape)]
    want = []
    for call, x, feeds, out in calls:
        want.append([])
        for feed in feeds:
            x.copy_(feed)
            call()
            want[-1].append(out.clone())
    torch.cuda.synchronize()
    graphs = [torch.cuda.CUDAGraph() for _ in calls]
    for graph, (call, _, _, out) in zip(graphs, calls):
        with torch.cuda.graph(graph, pool=pool):
            early = out + 1  # (intermediates of the graph's pool in front of the calls and behind them)
            call()
            call()           # two calls, one scratch
            out.copy_(out + (early - early))
    return calls, want, graphs


def _feed(calls, i):
    for _, x, feeds, out in calls:
        x.copy_(feeds[i])
        out.zero_()


@pytest.mark.parametrize("make,shape", _WITH_SCRATCH)
@pytest.mark.parametrize("shared_pool", [False, True])
def test_graphs_of_one_stream_replay_in_any_order(make, shape, shared_pool):
    import sol_execbench_b200_kernels_b200 as pkg

    calls, want, graphs = _two_graphs(make, shape, torch.cuda.graph_pool_handle() if shared_pool else None)
    for trial, order in enumerate([(1, 0), (1, 1, 0), (0, 1), (0, 0, 1)]):  # the one recorded second comes first
        _feed(calls, trial % 2)
        for g in order:
            graphs[g].replay()
        torch.cuda.synchronize()
        for (_, _, _, out), w in zip(calls, want):
            assert torch.equal(out, w[trial % 2]), (trial, order)
    del graphs[0]  # its scratch was its own
    _feed(calls, 0)
    graphs[0].replay()
    torch.cuda.synchronize()
    assert torch.equal(calls[1][3], want[1][0])
    assert pkg.last_status()[0] == 0


@pytest.mark.parametrize("make,shape", _WITH_SCRATCH)
def test_graphs_replay_at_once_on_two_streams(make, shape):
    import sol_execbench_b200_kernels_b200 as pkg

    calls, want, graphs = _two_graphs(make, shape)
    side = [torch.cuda.Stream(), torch.cuda.Stream()]
    for trial in range(4):
        _feed(calls, trial % 2)
        torch.cuda.synchronize()
        for _ in range(5):
            for graph, stream in zip(graphs, side):
                with torch.cuda.stream(stream):
                    graph.replay()
        torch.cuda.synchronize()
        for (_, _, _, out), w in zip(calls, want):
            assert torch.equal(out, w[trial % 2]), trial
    assert pkg.last_status()[0] == 0


@pytest.mark.parametrize("make,shape", _WITH_SCRATCH)
def test_an_abandoned_capture_leaves_nothing_behind(make, shape):
    import sol_execbench_b200_kernels_b200 as pkg

    call, x, feeds, out = make(*shape)
    x.copy_(feeds[0])
    call()
    want = out.clone()
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    lost = torch.cuda.CUDAGraph()
    with pytest.raises(RuntimeError, match="abandoned"):
        with torch.cuda.graph(lost, stream=stream):
            call()
            raise RuntimeError("abandoned")
    del lost
    out.zero_()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):  # eager, on the stream that the capture used
        call()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        call()
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    assert pkg.last_status()[0] == 0
