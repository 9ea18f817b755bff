"""Where tiles are cut along K in clusters, pinned on the CPU (148 SMs, so 74 clusters of two CTAs, are assumed there)."""
import pytest

from sol_execbench_b200_kernels_b200 import _cabi


def _choice(op, m, k, n, leave):
    return _cabi.PLAN_NAMES[_cabi.lib.gu_select_tile_kernel(op, m, k, n, leave)]


@pytest.mark.parametrize("m,kb,nb,cut", [
    (128, 56, 18, True), (451, 56, 18, True), (1, 12, 74, True), (128, 32, 74, True),
    (1, 12, 75, False), (129, 32, 37, True), (129, 32, 38, False),  # 74 and 76 tiles
    (1, 11, 74, False), (1, 12, 1, True), (600, 32, 14, True), (600, 32, 15, False),
])
def test_gateup_tiles_cut_in_clusters(m, kb, nb, cut):
    k, n = 128 * kb, 128 * nb
    assert (_choice(_cabi.OP_GATEUP, m, k, n, 1) == "tile_split") == cut
    assert _choice(_cabi.OP_MLP_GATEUP, m, k, n, 1) == ("tile_split" if cut else _choice(_cabi.OP_GATEUP_FP8, m, k, n, 1))
    # without leave to cut, and in a call that never cuts, tiles are whole
    assert _choice(_cabi.OP_GATEUP, m, k, n, 0) in ("tile_dp", "tile_pair")
    assert _choice(_cabi.OP_MLP_GATEUP, m, k, n, 0) == _choice(_cabi.OP_GATEUP_FP8, m, k, n, 0)
    assert _choice(_cabi.OP_GATEUP_FP8, m, k, n, 1) in ("tile_dp", "tile_pair")


@pytest.mark.parametrize("m,k,h,cut", [
    (8, 14336, 4096, True), (515, 14336, 4096, False), (512, 14336, 4096, True), (8, 1536, 37 * 256, True),
    (8, 1536, 74 * 256, True), (8, 1536, 74 * 256 + 128, False), (8, 1536, 73 * 256 + 128, True), (8, 1408, 4096, False),
])
def test_down_projection_tiles_cut_in_clusters(m, k, h, cut):
    assert (_choice(_cabi.OP_MLP_DOWN, m, k, h, 1) == "tile_split") == cut
    assert _choice(_cabi.OP_MLP_DOWN, m, k, h, 0) == _choice(_cabi.OP_GEMM, m, k, h, 1) != "tile_split"


@pytest.mark.parametrize("op,m,kb,tiles,cut", [
    # the faster side of the measurements beside the rule, and the rule's line itself
    ("run", 8, 12, 74, True), ("run", 64, 16, 74, True), ("run", 200, 16, 50, True), ("run", 128, 12, 18, True),
    ("run", 128, 12, 37, False), ("run", 128, 16, 37, True), ("run", 128, 16, 74, False), ("run", 128, 24, 74, True),
    ("run", 256, 16, 74, False), ("run", 256, 24, 74, True), ("run", 128, 19, 74, False), ("run", 128, 20, 74, True),
    ("run", 128, 16, 50, True), ("run", 96, 12, 74, False),
    ("gateup", 128, 12, 37, False), ("gateup", 256, 16, 36, True), ("gateup", 128, 16, 37, False), ("gateup", 128, 24, 37, True),
    ("gateup", 128, 24, 74, False), ("gateup", 128, 32, 74, True), ("gateup", 64, 16, 74, False),
    ("gateup", 64, 24, 74, True), ("gateup", 128, 25, 74, False), ("gateup", 128, 26, 74, True),
    ("down", 256, 24, 74, False), ("down", 256, 56, 74, True), ("down", 8, 12, 74, True), ("down", 128, 80, 74, True),
])
def test_cut_only_where_it_was_the_faster(op, m, kb, tiles, cut):
    col_tiles = tiles // ((m + 127) // 128)
    code = {"run": _cabi.OP_GATEUP, "gateup": _cabi.OP_MLP_GATEUP, "down": _cabi.OP_MLP_DOWN}[op]
    n = col_tiles * (256 if op == "down" else 128)
    assert (_choice(code, m, 128 * kb, n, 1) == "tile_split") == cut


def test_no_scratch_is_asked_for_where_none_is_used():
    lib = _cabi.lib
    for m, k, n in [(128, 7168, 2304), (451, 7168, 2304), (256, 8192, 2048), (1, 4224, 128)]:
        assert _choice(_cabi.OP_GATEUP, m, k, n, 1) == "tile_split"
        for plan in (_cabi.PLAN_AUTO, _cabi.PLAN_TILE, _cabi.PLAN_TILE_SPLIT):
            assert lib.gu_workspace_bytes(m, k, n, plan) == 0


def test_unassigned_ops_and_plans_stay_refused():
    assert _cabi.lib.gu_select_tile_kernel(3, 256, 128, 128, 1) == _cabi.GU_EINVAL_PLAN
    assert _cabi.lib.gu_select_tile_kernel(6, 256, 128, 128, 1) == _cabi.GU_EINVAL_PLAN
    assert _cabi.lib.gu_select_tile_kernel(_cabi.OP_MLP_DOWN, 4, 100, 128, 1) == _cabi.GU_EINVAL_SHAPE
