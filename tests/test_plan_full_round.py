"""The plan for few tokens where one round of tiles fills the device, pinned to the measured choice."""
import pytest

from sol_execbench_b200_kernels_b200 import _cabi


@pytest.mark.parametrize("m,k,n,plan", [
    (8, 8192, 17920, "tile"), (24, 8192, 17920, "tile"), (1, 7168, 18432, "tile"), (16, 6144, 16384, "tile"),
    (8, 8192, 18944, "tile"), (8, 8192, 18944 + 128, "stream"),     # 148 tiles are one round, 149 are two
    (8, 8192, 126 * 128, "tile"), (8, 8192, 125 * 128, "stream"),   # 85 % of 148 SMs
    (8, 3584, 18944, "stream"), (9, 3584, 18944, "tile"), (1, 5120, 18944, "tile"), (1, 4992, 18944, "stream"),
    (8, 8192, 14336, "stream"), (16, 8192, 28672, "stream"),
])
def test_full_round_of_tiles_beats_streaming(m, k, n, plan):
    assert _cabi.PLAN_NAMES[_cabi.lib.gu_select_plan(m, k, n)] == plan
