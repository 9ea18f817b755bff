"""`mlp_block` with up to 16 tokens and large weights: the steps that stream their weights through all SMs, against whole
tiles, which other tests hold against the oracle.  (Small shapes run through the same kernels in the range-checked build,
see test_gpu_bounds_sweep.py.)"""
import pytest
import torch

from sol_execbench_b200_kernels_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _weights(g, k, n, h):
    out = []
    for rows, cols in ((n, k), (n, k), (h, n)):
        out += W.quantize_weight_128x128(torch.randn(rows, cols, generator=g, device="cuda:0") * 0.02)
    return out


# tokens at the edges of the padded 16; K blocks that no range divides, odd ones in the down projection (a last step with
# one tile), ranges longer and shorter than a column block, few and many column blocks
@pytest.mark.parametrize("m,kb,nb,hb", [(1, 32, 112, 32), (8, 33, 147, 29), (15, 64, 225, 64), (16, 41, 111, 40), (16, 8, 224, 160),
                                        (2, 128, 64, 96), (3, 16, 449, 5), (8, 33, 150, 29), (16, 41, 80, 40), (15, 9, 170, 16),
                                        (1, 32, 100, 32), (16, 65, 108, 8)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_streamed_steps_match_whole_tiles(m, kb, nb, hb, dtype):
    import sol_execbench_b200_kernels_b200 as pkg
    from sol_execbench_b200_kernels_b200 import _cabi

    k, n, h = 128 * kb, 128 * nb, 128 * hb
    steps = [_cabi.lib.gu_select_tile_kernel(*step, 2) for step in ((_cabi.OP_MLP_GATEUP, m, k, n), (_cabi.OP_MLP_DOWN, m, n, h))]
    assert _cabi.PLAN_STREAM in steps
    g = torch.Generator(device="cuda:0").manual_seed(m)
    x = torch.randn(m, k + 8, generator=g, device="cuda:0").to(dtype)[:, :k]  # pitched rows
    weights = _weights(g, k, n, h)
    ref = pkg.mlp_block(x, *weights, whole_tiles=True)
    wide = torch.full((m + 1, h + 128), 7.0, dtype=torch.bfloat16, device="cuda:0")
    pkg.mlp_block(x, *weights, wide[:m, :h])
    own = pkg.mlp_block(x, *weights)
    torch.cuda.synchronize()
    assert pkg.last_status()[0] == 0
    # fp32 sums joined in another order: a bf16 rounding of the intermediate flips here and there, and may move an e4m3
    # value by a step (2^-3 relative, on fewer than one in a thousand values)
    rel = float(torch.linalg.vector_norm(own.float() - ref.float()) / torch.linalg.vector_norm(ref.float()))
    assert bool(torch.isfinite(own.float()).all()) and rel <= 2e-3, rel
    assert torch.equal(wide[:m, :h], own)  # the order of the sums is fixed
    assert bool((wide[m] == 7.0).all()) and bool((wide[:, h:] == 7.0).all())


def test_replays_eager_calls_and_streams_keep_their_stamps_apart():
    import sol_execbench_b200_kernels_b200 as pkg

    m, k, n = 5, 4096, 14336
    g = torch.Generator(device="cuda:0").manual_seed(3)
    weights = _weights(g, k, n, k)
    xs = [torch.randn(m, k, generator=g, device="cuda:0").bfloat16() for _ in range(3)]
    want = [pkg.mlp_block(x, *weights).clone() for x in xs]
    live, out = xs[0].clone(), torch.empty_like(want[0])
    pkg.mlp_block(live, *weights, out)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        pkg.mlp_block(live, *weights, out)
    other, other_out = torch.cuda.Stream(), torch.empty_like(out)
    for trial in range(12):
        live.copy_(xs[trial % 3])
        if trial % 4 == 3:
            pkg.mlp_block(live, *weights, out)
        else:
            graph.replay()
        with torch.cuda.stream(other):
            pkg.mlp_block(xs[1], *weights, other_out)
        torch.cuda.synchronize()
        assert torch.equal(out, want[trial % 3]) and torch.equal(other_out, want[1]), trial
    assert pkg.last_status()[0] == 0


def test_small_scratch_is_no_scratch():
    """Through the C entry point: with less than gu_mlp_workspace_bytes() the block runs as without scratch."""
    import ctypes

    import sol_execbench_b200_kernels_b200 as pkg
    from sol_execbench_b200_kernels_b200 import _cabi

    m, k, n = 8, 4096, 14336
    need = _cabi.lib.gu_mlp_workspace_bytes(m, k, n, k)
    assert need > 0
    g = torch.Generator(device="cuda:0").manual_seed(5)
    weights = _weights(g, k, n, k)
    x = torch.randn(m, k, generator=g, device="cuda:0").bfloat16()
    stream = torch.cuda.current_stream().cuda_stream
    ws = torch.empty(need, dtype=torch.uint8, device="cuda:0")
    _cabi.check(_cabi.lib.gu_mlp_workspace_init(ws.data_ptr(), need, stream))
    x_q, mid_q = (torch.empty(m, c, dtype=torch.uint8, device="cuda:0") for c in (k, n))
    x_s, mid_s = (torch.empty(m, c // 128, device="cuda:0") for c in (k, n))

    def call(nbytes, whole=0):
        out = torch.empty(m, k, dtype=torch.bfloat16, device="cuda:0")
        block = _cabi.GuMlp(x.data_ptr(), *[t.data_ptr() for t in weights], x_q.data_ptr(), x_s.data_ptr(), mid_q.data_ptr(),
                            mid_s.data_ptr(), out.data_ptr(), m, k, n, k, k, k, 0, whole)
        _cabi.check(_cabi.lib.gu_mlp_block_ws(ctypes.byref(block), ws.data_ptr(), nbytes, stream))
        return out

    without = call(need - 1)
    assert not ws[:4096].any()
    assert torch.equal(call(need), pkg.mlp_block(x, *weights))
    assert ws[:4096].any()
    assert torch.equal(call(need, whole=1), pkg.mlp_block(x, *weights, whole_tiles=True))
    block = _cabi.GuMlp(x.data_ptr(), *[t.data_ptr() for t in weights], x_q.data_ptr(), x_s.data_ptr(), mid_q.data_ptr(),
                        mid_s.data_ptr(), without.data_ptr(), m, k, n, k, k, k, 0, 0)
    plain = without.clone()
    without.fill_(float("nan"))
    _cabi.check(_cabi.lib.gu_mlp_block(ctypes.byref(block), stream))
    torch.cuda.synchronize()
    assert torch.equal(without, plain)
    assert _cabi.lib.gu_mlp_block_ws(ctypes.byref(block), ws.data_ptr() + 4, need + 16, stream) == _cabi.GU_EINVAL_ALIGN
    assert pkg.last_status()[0] == 0
