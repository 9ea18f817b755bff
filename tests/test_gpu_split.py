"""The K-split kernel (a cluster of CTAs per tile): `run` and `mlp_block` on shapes with few tiles, against the same
operations with whole tiles, which the other tests hold against the oracle."""
import pytest
import torch

from sol_execbench_b200_kernels_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _close(out, ref, rel_limit, what):
    rel = float(torch.linalg.vector_norm(out.float() - ref.float()) / torch.linalg.vector_norm(ref.float()))
    assert bool(torch.isfinite(out.float()).all()) and rel <= rel_limit, (what, rel)


# tokens at the edges of a warp's 32 rows and of the 128-row tile; K blocks that no cluster size divides; one column
# block (8 CTAs) up to as many tiles as still leave two CTAs each (74 on a B200), and one more; fewer K blocks than the
# rule cuts
@pytest.mark.parametrize("m,kb,nb,cut", [
    (1, 33, 1, True), (31, 56, 18, True), (33, 32, 18, True), (128, 35, 13, True), (129, 40, 9, True), (200, 17, 30, True),
    (257, 32, 24, True), (64, 12, 48, True), (5, 64, 25, True), (7, 12, 74, True), (130, 32, 37, True),
    (7, 8, 74, False), (33, 11, 18, False), (7, 12, 75, False), (257, 32, 25, False),
    (200, 13, 30, False), (128, 12, 74, False)])
def test_gateup_cut_along_k(m, kb, nb, cut):
    import sol_execbench_b200_kernels_b200 as pkg
    from sol_execbench_b200_kernels_b200 import _cabi

    k, n = 128 * kb, 128 * nb
    choice = _cabi.lib.gu_select_tile_kernel(_cabi.OP_GATEUP, m, k, n, 1)
    assert choice == _cabi.PLAN_TILE_SPLIT if cut else choice in (_cabi.PLAN_TILE_DP, _cabi.PLAN_TILE_PAIR)
    inp = W.make_inputs(m, k, n, seed=m, device="cuda:0")
    whole = torch.empty(m, n, dtype=torch.bfloat16, device="cuda:0")
    pkg.run_with_plan(*inp.args(), whole, "tile_dp")
    wide = torch.full((m + 1, n + 128), 7.0, dtype=torch.bfloat16, device="cuda:0")
    pkg.run_with_plan(*inp.args(), wide[:m, :n], "tile")
    again = torch.empty_like(whole)
    pkg.run_with_plan(*inp.args(), again, "tile")
    kept = torch.empty_like(whole)
    pkg.run_with_plan(*inp.args(), kept, "tile", whole_tiles=True)
    forced = torch.empty_like(whole)
    pkg.run_with_plan(*inp.args(), forced, "tile_split")
    torch.cuda.synchronize()
    assert pkg.last_status()[0] == 0
    # up to eight fp32 partial sums joined: a bf16 rounding flips where a sum is within 2^-24 * 8 of a tie
    for out in (wide[:m, :n], forced):
        _close(out, whole, 1e-4, (m, k, n))
        assert float((out != whole).float().mean()) <= 5e-3
    # the kernel that the choice names is the one that ran: joined sums round differently somewhere, whole tiles nowhere
    assert not cut or m * n < 1 << 15 or not torch.equal(wide[:m, :n], whole)
    assert cut or torch.equal(wide[:m, :n], whole)
    assert torch.equal(wide[:m, :n], again)  # the order of the sums is fixed
    assert torch.equal(kept, whole)
    assert bool((wide[m] == 7.0).all()) and bool((wide[:, n:] == 7.0).all())


def test_leave_to_cut_is_the_callers():
    """Through the C entry point: no tile is cut without scratch and without `cut_k`; either allows it, with the same bits;
    and `run`, which allows it, takes no scratch for it."""
    import ctypes

    import sol_execbench_b200_kernels_b200 as pkg
    from sol_execbench_b200_kernels_b200 import _cabi, kernel

    m, k, n = 128, 7168, 2304
    args = W.make_inputs(m, k, n, seed=4, device="cuda:0").args()
    stream = torch.cuda.current_stream().cuda_stream
    scratch = torch.zeros(4096, dtype=torch.uint8, device="cuda:0")

    def call(cut_k, ws):
        out = torch.empty(m, n, dtype=torch.bfloat16, device="cuda:0")
        pr = _cabi.GuProblem(*[t.data_ptr() for t in args], out.data_ptr(), m, k, n, n, ws.data_ptr() if ws is not None else None,
                             ws.numel() if ws is not None else 0, _cabi.PLAN_AUTO, cut_k)
        _cabi.check(_cabi.lib.gu_run(ctypes.byref(pr), stream))
        return out

    whole, cut = (torch.empty(m, n, dtype=torch.bfloat16, device="cuda:0") for _ in range(2))
    pkg.run_with_plan(*args, whole, "tile_dp")
    before = dict(kernel._WORKSPACES)
    other = torch.cuda.Stream()
    other.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(other):
        pkg.run(*args, cut)
    torch.cuda.synchronize()
    assert kernel._WORKSPACES == before
    assert not torch.equal(cut, whole)
    assert torch.equal(call(0, None), whole)
    assert torch.equal(call(1, None), cut)
    assert torch.equal(call(0, scratch), cut)
    assert not scratch.any()
    assert pkg.last_status()[0] == 0


def test_forced_split_needs_two_k_blocks():
    import sol_execbench_b200_kernels_b200 as pkg

    inp = W.make_inputs(4, 128, 256, seed=1, device="cuda:0")
    with pytest.raises(ValueError, match="plan"):
        pkg.run_with_plan(*inp.args(), torch.empty(4, 256, dtype=torch.bfloat16, device="cuda:0"), "tile_split")


@pytest.mark.parametrize("m,kb,nb,hb", [(1, 4, 40, 1), (8, 32, 112, 32), (8, 9, 33, 3), (31, 7, 18, 5), (128, 16, 35, 16),
                                        (129, 24, 18, 8), (300, 32, 24, 12), (515, 8, 112, 8), (1, 1, 1, 1)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_mlp_block_cut_along_k(m, kb, nb, hb, dtype):
    import sol_execbench_b200_kernels_b200 as pkg

    k, n, h = 128 * kb, 128 * nb, 128 * hb
    g = torch.Generator(device="cuda:0").manual_seed(m)
    x = torch.randn(m, k + 8, generator=g, device="cuda:0").to(dtype)[:, :k]  # pitched rows
    weights = []
    for rows, cols in ((n, k), (n, k), (h, n)):
        weights += W.quantize_weight_128x128(torch.randn(rows, cols, generator=g, device="cuda:0") * 0.02)
    xq, sx = pkg.quantize_activation(x)
    mid_q = torch.empty(m, n, dtype=torch.float8_e4m3fn, device="cuda:0")
    mid_s = torch.empty(m, nb, device="cuda:0")
    pkg.run_fp8_output(xq, sx, *weights[:4], mid_q, mid_s)
    ref = torch.empty(m, h, dtype=torch.bfloat16, device="cuda:0")
    pkg.blockwise_gemm(mid_q, mid_s, *weights[4:], ref)
    wide = torch.full((m + 1, h + 128), 7.0, dtype=torch.bfloat16, device="cuda:0")
    pkg.mlp_block(x, *weights, wide[:m, :h])
    own = pkg.mlp_block(x, *weights)
    torch.cuda.synchronize()
    assert pkg.last_status()[0] == 0
    # a flipped bf16 rounding may move an e4m3 value of the intermediate by a step (2^-3 relative, on fewer than one in
    # a thousand values)
    _close(own, ref, 2e-3, (m, k, n, h))
    assert torch.equal(wide[:m, :h], own)
    assert bool((wide[m] == 7.0).all()) and bool((wide[:, h:] == 7.0).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_mlp_block_with_whole_tiles_gives_rows_that_do_not_depend_on_the_batch(dtype):
    """512 tokens run on CTA pairs, 300 on lone CTAs, and by itself the library would cut both steps of the smaller calls
    along K."""
    import sol_execbench_b200_kernels_b200 as pkg

    k, n, h = 2048, 2304, 2048
    g = torch.Generator(device="cuda:0").manual_seed(9)
    x = torch.randn(512, k, generator=g, device="cuda:0").to(dtype)
    weights = []
    for rows, cols in ((n, k), (n, k), (h, n)):
        weights += W.quantize_weight_128x128(torch.randn(rows, cols, generator=g, device="cuda:0") * 0.02)
    xq, sx = pkg.quantize_activation(x)
    mid_q = torch.empty(512, n, dtype=torch.float8_e4m3fn, device="cuda:0")
    mid_s = torch.empty(512, n // 128, device="cuda:0")
    pkg.run_fp8_output(xq, sx, *weights[:4], mid_q, mid_s)
    ref = torch.empty(512, h, dtype=torch.bfloat16, device="cuda:0")
    pkg.blockwise_gemm(mid_q, mid_s, *weights[4:], ref)
    for m in (512, 300, 129, 128, 31, 1):
        assert torch.equal(pkg.mlp_block(x[:m], *weights, whole_tiles=True), ref[:m]), m
    assert pkg.last_status()[0] == 0


def test_mlp_block_in_a_graph_and_after_a_weight_update():
    """Weights copied in just before the call have to be the ones that count, in eager calls and in replays.  (A copy never
    lets its successor in early; a kernel that does is in front in test_gpu_overlap.py.)"""
    import sol_execbench_b200_kernels_b200 as pkg

    m, k, n = 8, 2048, 5632
    g = torch.Generator(device="cuda:0").manual_seed(3)
    x = torch.randn(m, k, generator=g, device="cuda:0").bfloat16()
    sets = []
    for _ in range(2):
        s = []
        for rows, cols in ((n, k), (n, k), (k, n)):
            s += W.quantize_weight_128x128(torch.randn(rows, cols, generator=g, device="cuda:0") * 0.02)
        sets.append(s)
    want = [pkg.mlp_block(x, *s).clone() for s in sets]
    live = [t.clone() for t in sets[0]]
    out = torch.empty_like(want[0])
    pkg.mlp_block(x, *live, out)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        pkg.mlp_block(x, *live, out)
    for trial in range(20):
        for dst, src in zip(live, sets[trial % 2]):
            dst.view(torch.uint8).copy_(src.view(torch.uint8))
        if trial % 4 < 2:
            pkg.mlp_block(x, *live, out)
        else:
            graph.replay()
        assert torch.equal(out, want[trial % 2]), trial
    assert pkg.last_status()[0] == 0
