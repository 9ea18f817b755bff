"""Launches move in while the kernel in front still runs and fetch their first weights early.  Here that kernel writes
those weights: the library's own quantiser, which lets its successor in before it has written anything, behind a launch
long enough for the host to queue the whole chain.  What counts has to be what it wrote, in eager calls and in replays."""
import pytest
import torch

from sol_execbench_b200_kernels_b200 import workloads as W

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _busy():
    a = torch.zeros(4096, 4096, dtype=torch.bfloat16, device=DEV)
    return lambda: [a @ a for _ in range(4)]


def _sources(g, shapes, count=2):
    return [[(torch.randn(*s, generator=g, device=DEV) * 0.5).bfloat16() for s in shapes] for _ in range(count)]


def _check(write, call, out, sources, live, want, what):
    """`write` quantises the tensors in `live` into the weights, `call` uses them."""
    import sol_execbench_b200_kernels_b200 as pkg

    busy = _busy()

    def load(src):
        for dst, s in zip(live, src):
            dst.copy_(s)

    load(sources[0])
    write()
    call()  # (first call outside the capture)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        write()
        call()
    for trial in range(12):
        load(sources[trial % 2])
        out.fill_(float("nan"))
        busy()
        if trial % 4 < 2:
            write()
            call()
        else:
            graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want[trial % 2]), (what, trial)
    assert pkg.last_status()[0] == 0


# the streaming, lone-CTA, K-split and CTA-pair kernels, and the pair kernel's stream-K schedule
@pytest.mark.parametrize("plan,m,k,n", [("stream", 16, 4096, 8192), ("tile_dp", 100, 2048, 9472), ("tile_split", 100, 2048, 2304),
                                        ("tile_pair", 300, 2048, 4096), ("tile_pair_sk", 512, 1024, 9600)])
def test_weights_written_by_the_launch_in_front_of_run(plan, m, k, n):
    import sol_execbench_b200_kernels_b200 as pkg

    g = torch.Generator(device=DEV).manual_seed(m)
    x, scale_x, gate, scale_gate, up, scale_up = W.make_inputs(m, k, n, seed=m, device=DEV).args()
    sources = _sources(g, [(n, k), (n, k)])
    want = []
    for src in sources:
        qs = [pkg.quantize_activation(s)[0] for s in src]
        out = torch.empty(m, n, dtype=torch.bfloat16, device=DEV)
        torch.cuda.synchronize()
        pkg.run_with_plan(x, scale_x, qs[0], scale_gate, qs[1], scale_up, out, plan)
        torch.cuda.synchronize()
        want.append(out)
    live = [torch.empty_like(s) for s in sources[0]]
    scratch = torch.empty(n, k // 128, device=DEV)
    out = torch.empty_like(want[0])

    def write():
        pkg.quantize_activation(live[1], q=up, scale=scratch)
        pkg.quantize_activation(live[0], q=gate, scale=scratch)

    _check(write, lambda: pkg.run_with_plan(x, scale_x, gate, scale_gate, up, scale_up, out, plan), out, sources, live, want, plan)


# both steps cut along K; lone CTAs and a cut down projection; lone CTAs and pairs; pairs and a cut down projection
@pytest.mark.parametrize("m,k,n,h", [(8, 2048, 2304, 2048), (8, 1024, 9600, 2048), (512, 2048, 5120, 9600),
                                     (512, 4096, 14336, 2048)])
def test_weights_written_by_the_launch_in_front_of_mlp_block(m, k, n, h):
    """`mlp_block` loads weights into shared memory before the kernels in front of it have ended, on the strength of its
    quantiser having waited for everything earlier."""
    import sol_execbench_b200_kernels_b200 as pkg

    g = torch.Generator(device=DEV).manual_seed(m + n)
    x = torch.randn(m, k, generator=g, device=DEV).bfloat16()
    shapes = [(n, k), (n, k), (h, n)]
    weights, scales = [], []
    for s in shapes:
        q, sc = W.quantize_weight_128x128(torch.randn(*s, generator=g, device=DEV) * 0.02)
        weights.append(q)
        scales.append(sc)
    sources = _sources(g, shapes)
    want = []
    for src in sources:
        qs = [pkg.quantize_activation(s)[0] for s in src]
        torch.cuda.synchronize()
        want.append(pkg.mlp_block(x, qs[0], scales[0], qs[1], scales[1], qs[2], scales[2]))
        torch.cuda.synchronize()
    live = [torch.empty_like(s) for s in sources[0]]
    scratch = [torch.empty(r, c // 128, device=DEV) for r, c in shapes]
    out = torch.empty_like(want[0])

    def write():
        for i in (2, 1, 0):
            pkg.quantize_activation(live[i], q=weights[i], scale=scratch[i])

    def call():
        pkg.mlp_block(x, weights[0], scales[0], weights[1], scales[1], weights[2], scales[2], out)

    _check(write, call, out, sources, live, want, (m, k, n, h))


@pytest.mark.parametrize("m", [100, 300])  # lone CTAs, CTA pairs
def test_weights_written_by_the_launch_in_front_of_the_projection(m):
    """The bf16 projection behind one whose result it takes as its weights."""
    from sol_execbench_b200_kernels_b200 import side_ops

    n, k, inner = 4096, 1024, 256
    g = torch.Generator(device=DEV).manual_seed(m)
    hidden = (torch.randn(m, k, generator=g, device=DEV) * 0.5).bfloat16()
    bias = (torch.randn(n, generator=g, device=DEV) * 0.2).bfloat16()
    b0 = torch.zeros(k, dtype=torch.bfloat16, device=DEV)
    factor = (torch.randn(k, inner, generator=g, device=DEV) * 0.1).bfloat16()
    sources = _sources(g, [(n, inner)])
    want = []
    for (src,) in sources:
        weight = torch.empty(n, k, dtype=torch.bfloat16, device=DEV)
        side_ops.mamba_in_proj(src, factor, b0, weight)
        torch.cuda.synchronize()
        out = torch.empty(m, n, dtype=torch.bfloat16, device=DEV)
        side_ops.mamba_in_proj(hidden, weight, bias, out)
        torch.cuda.synchronize()
        want.append(out)
    live = [torch.empty_like(sources[0][0])]
    weight, out = torch.empty(n, k, dtype=torch.bfloat16, device=DEV), torch.empty_like(want[0])
    _check(lambda: side_ops.mamba_in_proj(live[0], factor, b0, weight),
           lambda: side_ops.mamba_in_proj(hidden, weight, bias, out), out, sources, live, want, m)
    assert side_ops.last_status() == (0, 0)
