"""The projection's lone-CTA kernel (up to 128 rows) with every tile width: the width follows N, a width that is no
multiple of 64 has a last chunk of 32 columns that is stored without TMA, and past 148 x 256 columns a CTA takes more
than one tile."""
import pytest
import torch

from oracle import sideops_oracle as O

pytestmark = pytest.mark.gpu


# N: 64-column tiles, 96 (N ends inside the narrow chunk), 160, 224 (one round exactly), 256 in two rounds
@pytest.mark.parametrize("n", [72, 9480, 20000, 32768, 40008])
@pytest.mark.parametrize("m,k", [(1, 136), (33, 64), (128, 520)])
def test_projection_tile_widths(m, k, n):
    from sol_execbench_b200_kernels_b200 import side_ops

    g = torch.Generator(device="cuda:0").manual_seed(n + m)
    hidden = (torch.randn(m, k, generator=g, device="cuda:0") * 0.5).bfloat16()
    weight = (torch.randn(n, k, generator=g, device="cuda:0") * 0.04).bfloat16()
    bias = (torch.randn(n, generator=g, device="cuda:0") * 0.2).bfloat16()
    wide = torch.full((m + 1, n), 7.0, dtype=torch.bfloat16, device="cuda:0")
    side_ops.mamba_in_proj(hidden, weight, bias, wide[:m])
    torch.cuda.synchronize()
    assert side_ops.last_status() == (0, 0)
    exact = O.mamba_in_proj(hidden, weight, bias, exact=True)
    # one rounding to bf16 (2^-9 relative) of an fp32 sum whose error is far below; twice that as the bound
    err = (wide[:m].double() - exact).abs()
    assert bool((err <= 2.0 ** -8 * exact.abs() + 1e-5).all()), float(err.max())
    assert bool((wide[m] == 7.0).all())
