"""The launch count that stamps are taken from, around its largest value: no two launches in a row on one scratch share a
stamp (the second would take the first one's partial sums for its own), and 0, which fresh scratch holds, is never one."""
import pytest
import torch

from sol_execbench_b200_kernels_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _scratch(kept):
    from sol_execbench_b200_kernels_b200 import kernel

    return kept[(0, kernel._stream_ptr(torch.device("cuda", 0)), 0)].view(torch.int32)


def _check(call, x, feeds, out, kept, word, launches_per_call):
    import sol_execbench_b200_kernels_b200 as pkg

    want = []
    for feed in feeds:
        x.copy_(feed)
        call()
        want.append(out.clone())
    words = _scratch(kept)
    counts = []
    words[word] = -3  # 0xfffffffd
    for i in range(8):
        x.copy_(feeds[i % 3])
        out.zero_()
        call()
        assert torch.equal(out, want[i % 3]), i
        counts.append(int(words[word]))
    stamps = list(range(-2, 0)) + list(range(1, 32))
    assert counts == stamps[launches_per_call - 1::launches_per_call][:8]
    assert pkg.last_status()[0] == 0


@pytest.mark.parametrize("shape,word", [((16, 4096, 8192), 1022),   # weight streaming
                                        ((512, 4096, 14336), 1020)])  # the pair kernel's stream-K schedule
def test_run(shape, word):
    import sol_execbench_b200_kernels_b200 as pkg
    from sol_execbench_b200_kernels_b200 import kernel

    m, k, n = shape
    feeds = [W.make_inputs(m, k, n, seed=s, device="cuda:0") for s in range(3)]
    x, out = feeds[0].x.clone(), torch.empty(m, n, dtype=torch.bfloat16, device="cuda:0")
    rest = feeds[0].args()[1:]
    _check(lambda: pkg.run(x, *rest, out), x.view(torch.uint8), [f.x.view(torch.uint8) for f in feeds], out, kernel._WORKSPACES,
           word, 1)


def test_mlp_block():
    import sol_execbench_b200_kernels_b200 as pkg
    from sol_execbench_b200_kernels_b200 import kernel

    m, k, n = 8, 4096, 11008  # both steps stream: two launches a call
    g = torch.Generator(device="cuda:0").manual_seed(1)
    weights = []
    for rows, cols in ((n, k), (n, k), (k, n)):
        weights += W.quantize_weight_128x128(torch.randn(rows, cols, generator=g, device="cuda:0") * 0.02)
    feeds = [torch.randn(m, k, generator=g, device="cuda:0").bfloat16() for _ in range(3)]
    x, out = feeds[0].clone(), torch.empty(m, k, dtype=torch.bfloat16, device="cuda:0")
    _check(lambda: pkg.mlp_block(x, *weights, out), x, feeds, out, kernel._MLP_WORKSPACES, 0, 2)
