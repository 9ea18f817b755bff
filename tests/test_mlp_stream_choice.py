"""Which steps of `mlp_block` stream their weights when it has scratch, pinned on the CPU (148 SMs are assumed there)."""
import pytest

from sol_execbench_b200_kernels_b200 import _cabi


def _choice(op, m, k, n, with_workspace):
    return _cabi.PLAN_NAMES[_cabi.lib.gu_select_tile_kernel(op, m, k, n, with_workspace)]


@pytest.mark.parametrize("m,k,n,gateup,down", [
    # the faster side of the measurements beside the rule
    (8, 4096, 11008, True, True), (16, 4096, 11008, True, True), (8, 8192, 28672, True, True), (16, 8192, 28672, True, True),
    (8, 1024, 28672, True, True), (8, 2048, 28672, True, True), (8, 6144, 16384, False, True), (8, 3584, 18944, False, True),
    (8, 8192, 8192, False, True), (16, 4096, 14336, False, True),
    (8, 2048, 5632, False, False), (8, 1024, 4096, False, False), (8, 7168, 2304, False, False),
    (17, 4096, 14336, False, False), (17, 8192, 28672, False, False), (8, 512, 14336, False, False),
    # us of the block with operands that stay out of L2, gate/up in whole tiles / streamed
    (8, 4096, 14336, True, True),    # 40.1 / 39.8
    (8, 5120, 13824, True, True),
    (8, 2048, 14336, False, False),  # 30.1 / 30.7
    (8, 3072, 13824, False, False),  # 34.2 / 34.9
    (16, 2048, 11776, False, False), # 28.3 / 30.0
    (1, 4096, 16384, True, True),    # 42.4 / 42.0
    (8, 4096, 16384, False, True),   # 43.6 / 43.6
    (16, 1024, 32768, False, True),  # 37.4 / 39.7: two rounds of tiles
    (4, 1024, 32768, True, True),    # 35.8 / 34.4
    (16, 4096, 56320, True, True),   # 118 / 114: three
    (8, 8192, 32768, True, True),    # 142 / 135
])
def test_steps_that_stream(m, k, n, gateup, down):
    assert (_choice(_cabi.OP_MLP_GATEUP, m, k, n, 2) == "stream") == gateup
    assert (_choice(_cabi.OP_MLP_DOWN, m, n, k, 2) == "stream") == down
    assert (_cabi.lib.gu_mlp_workspace_bytes(m, k, n, k) > 0) == (gateup or down)
    for leave in (0, 1):  # not without that scratch
        assert _choice(_cabi.OP_MLP_GATEUP, m, k, n, leave) != "stream" != _choice(_cabi.OP_MLP_DOWN, m, n, k, leave)


def test_few_column_blocks_and_refused_shapes():
    assert _choice(_cabi.OP_MLP_DOWN, 1, 28672, 128 * 7, 2) != "stream"
    assert _choice(_cabi.OP_MLP_DOWN, 1, 28672, 128 * 8, 2) == "stream"
    assert _cabi.lib.gu_mlp_workspace_bytes(8, 100, 128, 128) == 0
    assert _cabi.lib.gu_mlp_workspace_bytes(0, 4096, 14336, 4096) == 0
    assert _cabi.lib.gu_select_tile_kernel(_cabi.OP_MLP_DOWN, 8, 100, 128, 2) == _cabi.GU_EINVAL_SHAPE
