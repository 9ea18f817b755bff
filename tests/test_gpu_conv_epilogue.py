"""The Mamba projection with the convolution tail in its epilogue (more than 128 rows) against the two separate launches,
which other tests hold against the oracle: row counts at the edges of the 128-row blocks and the 256-row pair tiles,
sequences whose starts lie anywhere in them (odd lengths too, and shorter than the taps), one to many column tiles."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_SHAPES = [(1, 129, 64, 64), (1, 131, 64, 192), (1, 256, 72, 128), (1, 257, 64, 320), (2, 65, 64, 64), (3, 67, 200, 320),
           (130, 1, 64, 64), (130, 2, 64, 64), (65, 3, 64, 128), (40, 5, 64, 128), (5, 129, 72, 64), (1, 500, 64, 2048),
           (2, 200, 136, 9600)]


def _inputs(batch, seq, k, channels):
    g = torch.Generator().manual_seed(batch * 1000 + seq)

    def bf16(*shape, scale=1.0):
        return (torch.randn(*shape, generator=g) * scale).to(torch.bfloat16).to("cuda:0")

    hidden, weight = bf16(batch, seq, k), bf16(2 * channels, k, scale=0.1)
    weight[5] *= 60  # convolutions below -20 too
    mask = (torch.rand(batch, seq, generator=g) > 0.15).to(torch.bfloat16).to("cuda:0")
    return hidden, mask, weight, bf16(2 * channels, scale=0.3), bf16(channels, 1, 4, scale=0.5), bf16(channels, scale=0.5)


def _compare(shape):
    from sol_execbench_b200_kernels_b200 import side_ops

    batch, seq, _, channels = shape
    hidden, mask, weight, bias, conv_w, conv_b = _inputs(*shape)
    before = side_ops.launch_count()
    out, gate = side_ops.mamba_conv1d_with_gating(hidden, mask, weight, bias, conv_w, conv_b)
    assert side_ops.launch_count() == before + 2
    projected = torch.empty(batch, seq, 2 * channels, dtype=torch.bfloat16, device="cuda:0")
    want = torch.full((batch, channels, seq), float("nan"), dtype=torch.bfloat16, device="cuda:0")
    side_ops.mamba_in_proj(hidden, weight, bias, projected)
    side_ops.mamba_conv1d_tail(projected, mask, conv_w, conv_b, want)
    torch.cuda.synchronize()
    code, detail = side_ops.last_status()
    assert code == 0, f"{shape}: device status {code}, detail {detail:#x}"
    want_gate = projected[:, :, channels:].transpose(1, 2)
    assert torch.equal(gate, want_gate) and gate.stride() == want_gate.stride()
    # every output and every gate value is written, whatever the buffers held
    again, buf = torch.full_like(out, float("nan")), torch.full_like(projected, float("nan"))
    side_ops._so.check(side_ops._so.lib.so_mamba_in_proj_conv(
        hidden.data_ptr(), weight.data_ptr(), bias.data_ptr(), buf.data_ptr(), mask.data_ptr(), conv_w.data_ptr(),
        conv_b.data_ptr(), again.data_ptr(), batch, seq, hidden.shape[2], 2 * channels, channels,
        torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert torch.equal(again, out) and torch.equal(buf[:, :, channels:], projected[:, :, channels:])
    # The same operations up to the sigmoid, whose reciprocal is shared by other groups of four values: its last fp32 bit
    # may differ, and a bf16 rounding with it (2^-8 relative, then once more in the product) where it is within 2^-22 of
    # a tie, fewer than one in a thousand.
    off = out != want
    assert bool(torch.isfinite(out.float()).all()) and float(off.float().mean()) <= 1e-3, shape
    if bool(off.any()):
        assert float(((out.float() - want.float()).abs() / want.float().abs().clamp_min(1e-30))[off].max()) <= 2.0 ** -6, shape


@pytest.mark.parametrize("shape", _SHAPES)
def test_fused_tail_matches_the_separate_one(shape):
    _compare(shape)


def test_fused_tail_under_the_range_checked_build():
    lib = os.path.join(ROOT, "sol_execbench_b200_kernels_b200", "libsideops_bounds.so")
    assert os.path.exists(lib), "libsideops_bounds.so is missing: python -m sol_execbench_b200_kernels_b200.build --bounds"
    code = ("import sys; sys.path[:0] = [%r, %r]\n"
            "import sol_execbench_b200_kernels_b200.build as B; B.SIDE_LIB_PATH = B.SIDE_BOUNDS_LIB_PATH\n"
            "import test_gpu_conv_epilogue as T\n"
            "for shape in T._SHAPES: T._compare(shape)\n"
            "from sol_execbench_b200_kernels_b200 import _sideops_cabi\n"
            "assert _sideops_cabi.lib.so_is_range_checked_build() == 1\nprint('all in range')") % (ROOT, os.path.join(ROOT, "tests"))
    proc = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600)
    assert proc.returncode == 0 and "all in range" in proc.stdout, proc.stdout[-2000:] + proc.stderr[-3000:]


def test_a_refused_call_launches_nothing():
    from sol_execbench_b200_kernels_b200 import side_ops

    hidden, mask, weight, bias, conv_w, conv_b = _inputs(2, 100, 64, 64)
    before = side_ops.launch_count()
    for bad in ((hidden, mask[:, :-1], weight, bias, conv_w, conv_b), (hidden, mask, weight, bias, conv_w[:, :, :3], conv_b),
                (hidden, mask, weight, bias, conv_w, conv_b.float()), (hidden[:, :, :-8], mask, weight, bias, conv_w, conv_b),
                (hidden, mask, weight, bias[:-1], conv_w, conv_b), (hidden, mask.cpu(), weight, bias, conv_w, conv_b)):
        with pytest.raises(ValueError):
            side_ops.mamba_conv1d_with_gating(*bad)
    assert side_ops.launch_count() == before


def _bad_channels(conv_b):
    """Single channels whose convolutions are not finite, or below -20, each among ordinary neighbours."""
    for channel, value in ((5, "nan"), (16, "inf"), (17, "-50"), (30, "-inf"), (44, "inf"), (47, "-30"), (63, "nan")):
        conv_b[channel] = float(value)


def _same_where_not_finite(got, want, what):
    got, want = got.float().cpu(), want.float().cpu()
    assert torch.equal(torch.isnan(got), torch.isnan(want)), what
    assert torch.equal(torch.isinf(got), torch.isinf(want)), what
    fine = torch.isfinite(want)
    diff, size = (got - want).abs()[fine], want.abs()[fine]
    bad = diff > 1e-30  # (as in the tests of the tail against its oracle: at most 1e-3 of the values, by two bf16 steps)
    assert int(bad.sum()) <= max(2, 1e-3 * bad.numel()) and bool((diff[bad] <= size[bad] * 2.0 ** -6).all()), what


@pytest.mark.parametrize("batch,seq,channels", [(1, 300, 64), (2, 129, 128), (65, 3, 64), (1, 100, 64)])
def test_values_that_are_not_finite_stay_in_their_channel(batch, seq, channels):
    """Both forms of the tail against the oracle: channels with a NaN, an infinity or convolutions below -20, and one token
    whose activations are NaN (it reaches the three positions after it)."""
    from oracle import sideops_oracle
    from sol_execbench_b200_kernels_b200 import side_ops

    hidden, mask, weight, bias, conv_w, conv_b = _inputs(batch, seq, 64, channels)
    _bad_channels(conv_b)
    hidden[batch - 1, seq // 2] = float("nan")
    out, _ = side_ops.mamba_conv1d_with_gating(hidden, mask, weight, bias, conv_w, conv_b)
    projected = torch.empty(batch, seq, 2 * channels, dtype=torch.bfloat16, device="cuda:0")
    alone = torch.empty_like(out)
    side_ops.mamba_in_proj(hidden, weight, bias, projected)
    side_ops.mamba_conv1d_tail(projected, mask, conv_w, conv_b, alone)
    want = sideops_oracle.mamba_conv1d_tail(projected.cpu(), mask.cpu(), conv_w.cpu(), conv_b.cpu())
    assert bool(torch.isnan(want).any()) and bool(torch.isinf(want).any()) and bool(torch.isfinite(want).any())
    _same_where_not_finite(alone, want, "tail")
    _same_where_not_finite(out, want, "epilogue")
