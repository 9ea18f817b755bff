"""Exhaustive small-shape sweep under the range-checked debug build of the library.

`compute-sanitizer` is not available on the machines these tests run on, so the library carries its own checker:
built with -DGU_BOUNDS=1 (libgateup_bounds.so) every kernel tests each computed TMA coordinate, global index and
ring / accumulator stage index against its extent before using it, records the first violation in the status word
(`gu_last_status` -> GU_EBOUNDS) and skips the access.  This test runs every token count M = 1 ... 129 at
K, N in {128, 256} through every plan that takes the shape — the lone-CTA tile kernel and its stream-K schedule, the
CTA-pair kernel (forced also where the second CTA of a pair has no rows), the K-split kernel and the weight-streaming
kernel — inside that build, with canary rows and columns around the destination, against the CPU oracle; then a few
larger shapes through the pair kernel's stream-K schedule, its FP8-output epilogue and its plain-GEMM mode, the K-split
kernel with up to eight CTAs per tile, and `mlp_block`, whose kernels load weights early.  A process binds one build of
the library, so the sweep runs in a child process.
"""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_SWEEP = r"""
import os, sys
sys.path.insert(0, os.environ["GU_ROOT"])
import sol_execbench_b200_kernels_b200.build as B
B.LIB_PATH = B.BOUNDS_LIB_PATH
import torch
import sol_execbench_b200_kernels_b200 as pkg
from sol_execbench_b200_kernels_b200 import _cabi, workloads as W
from oracle import gateup_oracle as O

assert _cabi.lib.gu_is_range_checked_build() == 1
dev = torch.device("cuda:0")
pkg.last_status(clear=True)
launches = 0
for k in (128, 256):
    for n in (128, 256):
        wide = torch.empty(129 + 2, n + 256, dtype=torch.bfloat16, device=dev)
        for m in range(1, 130):
            inp = W.make_inputs(m, k, n, seed=1000 * k + 10 * n + m)
            ref = O.gateup_blockwise(*inp.args())
            g = inp.to(dev)
            plans = ["tile_dp", "tile_pair", "tile_sk"] + (["stream"] if m <= 64 else []) + (["tile_split"] if k > 128 else [])
            for plan in plans:
                wide.fill_(7.0)
                view = wide[1:m + 1, 128:128 + n]
                pkg.run_with_plan(*g.args(), view, plan)
                launches += 1
                torch.cuda.synchronize()
                code, detail = pkg.last_status()
                assert code == 0, f"M={m} K={k} N={n} {plan}: device status {code}, detail {detail:#x}"
                got = view.float().cpu()
                st = O.error_stats(got, ref)
                # (a stream-K hand-off adds partial sums in another association: single roundings may differ)
                assert st["finite"] and st["rel_l2"] <= 1e-3 and st["max_abs"] <= 2e-2, (m, k, n, plan, st)
                mask = torch.ones_like(wide, dtype=torch.bool)
                mask[1:m + 1, 128:128 + n] = False
                assert bool((wide[mask] == 7.0).all()), f"M={m} K={k} N={n} {plan}: wrote outside the destination"
# larger shapes for what needs many tiles or other epilogues: the pair kernel's stream-K schedule (a tile per cluster
# at least), its FP8-output epilogue and its plain-GEMM mode
for shape in ((512, 128, 4864), (300, 256, 5120), (1100, 128, 2432)):
    inp = W.make_inputs(*shape, seed=sum(shape))
    ref = O.gateup_blockwise(*inp.args())
    g = inp.to(dev)
    m, k, n = shape
    wide = torch.full((m + 2, n + 256), 7.0, dtype=torch.bfloat16, device=dev)
    view = wide[1:m + 1, 128:128 + n]
    pkg.run_with_plan(*g.args(), view, "tile_pair_sk")
    launches += 1
    torch.cuda.synchronize()
    code, detail = pkg.last_status()
    assert code == 0, f"{shape} tile_pair_sk: device status {code}, detail {detail:#x}"
    st = O.error_stats(view.float().cpu(), ref)
    assert st["finite"] and st["rel_l2"] <= 1e-3, (shape, st)
    mask = torch.ones_like(wide, dtype=torch.bool)
    mask[1:m + 1, 128:128 + n] = False
    assert bool((wide[mask] == 7.0).all()), f"{shape} tile_pair_sk: wrote outside the destination"
for shape in ((300, 256, 256), (129, 128, 384)):
    m, k, n = shape
    g = W.make_inputs(*shape, seed=7 + m).to(dev)
    q = torch.zeros(m, n, dtype=torch.uint8, device=dev).view(torch.float8_e4m3fn)
    sc = torch.zeros(m, n // 128, dtype=torch.float32, device=dev)
    pkg.run_fp8_output(*g.args(), q, sc)
    ref = torch.empty(m, n, dtype=torch.bfloat16, device=dev)
    pkg.run_with_plan(*g.args(), ref, "tile_dp")
    c = torch.empty(m, k, dtype=torch.bfloat16, device=dev)
    wq, ws = W.quantize_weight_128x128(torch.randn(k, n, device=dev) * 0.05)
    pkg.blockwise_gemm(q, sc, wq, ws, c)
    launches += 3
    torch.cuda.synchronize()
    code, detail = pkg.last_status()
    assert code == 0, f"{shape} fp8 output / plain GEMM: device status {code}, detail {detail:#x}"
    q_ref, s_ref = W.quantize_activation_1x128(ref.cpu().float())
    assert torch.equal(sc.cpu(), s_ref) and torch.equal(q.cpu().view(torch.uint8), q_ref.view(torch.uint8))
    want = O.gemm_blockwise(q.cpu(), sc.cpu(), wq.cpu(), ws.cpu())
    assert O.error_stats(c, want)["rel_l2"] <= 1e-3
# the K-split kernel: as `run` cuts few tiles (8, 3 and 2 CTAs per tile), and forced with one K block per CTA and with
# more tiles than are resident at once
for shape, plan in (((1, 4224, 128), "tile"), ((31, 7168, 384), "tile"), ((200, 2176, 1280), "tile"), ((64, 1536, 6144), "tile"),
                    ((130, 4096, 4736), "tile"), ((17, 1024, 256), "tile_split"), ((129, 384, 9728), "tile_split")):
    m, k, n = shape
    assert plan != "tile" or _cabi.lib.gu_select_tile_kernel(_cabi.OP_GATEUP, m, k, n, 1) == _cabi.PLAN_TILE_SPLIT, shape
    g = W.make_inputs(*shape, seed=m, device=dev)
    ref = torch.empty(m, n, dtype=torch.bfloat16, device=dev)
    pkg.run_with_plan(*g.args(), ref, "tile_dp")
    wide = torch.full((m + 2, n + 256), 7.0, dtype=torch.bfloat16, device=dev)
    view = wide[1:m + 1, 128:128 + n]
    pkg.run_with_plan(*g.args(), view, plan)
    launches += 2
    torch.cuda.synchronize()
    code, detail = pkg.last_status()
    assert code == 0, f"{shape} {plan}: device status {code}, detail {detail:#x}"
    st = O.error_stats(view.float().cpu(), ref.float().cpu())
    assert st["finite"] and st["rel_l2"] <= 1e-3, (shape, st)
    mask = torch.ones_like(wide, dtype=torch.bool)
    mask[1:m + 1, 128:128 + n] = False
    assert bool((wide[mask] == 7.0).all()), f"{shape} {plan}: wrote outside the destination"
# mlp_block, whole, streamed and cut: (tokens, hidden, intermediate, output); without scratch both steps are cut, or one of
# them; pairs, lone CTAs, an odd count of 128-column output blocks
for m, k, n, h in ((1, 1664, 1536, 128), (33, 2048, 2304, 640), (8, 1024, 9600, 1152), (128, 1536, 2432, 384),
                   (129, 384, 2176, 256), (300, 512, 4992, 2048), (515, 256, 384, 128)):
    x = torch.randn(m, k, device=dev).to(torch.bfloat16)
    ws = [t for r, c in ((n, k), (n, k), (h, n)) for t in W.quantize_weight_128x128(torch.randn(r, c, device=dev) * 0.03)]
    xq, sx = pkg.quantize_activation(x)
    q = torch.zeros(m, n, dtype=torch.uint8, device=dev).view(torch.float8_e4m3fn)
    sc = torch.zeros(m, n // 128, dtype=torch.float32, device=dev)
    pkg.run_fp8_output(xq, sx, *ws[:4], q, sc)
    ref = torch.empty(m, h, dtype=torch.bfloat16, device=dev)
    pkg.blockwise_gemm(q, sc, *ws[4:], ref)
    launches += 3
    # whole tiles; streamed up to 16 tokens (any shape in this build) and cut above; cut along K without that scratch
    scratch_bytes = pkg.kernel._mlp_scratch_bytes
    for whole, scratch in ((True, scratch_bytes), (False, scratch_bytes), (False, lambda *shape: 0)):
        pkg.kernel._mlp_scratch_bytes = scratch
        wide = torch.full((m + 2, h + 256), 7.0, dtype=torch.bfloat16, device=dev)
        view = wide[1:m + 1, 128:128 + h]
        pkg.mlp_block(x, *ws, view, whole_tiles=whole)
        launches += 3
        torch.cuda.synchronize()
        code, detail = pkg.last_status()
        assert code == 0, f"mlp_block {(m, k, n, h)} whole={whole}: device status {code}, detail {detail:#x}"
        st = O.error_stats(view.float().cpu(), ref.float().cpu())
        # (cut: an e4m3 rounding of the intermediate may move a step where a bf16 one flips)
        assert torch.equal(view, ref) if whole else st["finite"] and st["rel_l2"] <= 2e-3, (m, k, n, h, whole, st)
        mask = torch.ones_like(wide, dtype=torch.bool)
        mask[1:m + 1, 128:128 + h] = False
        assert bool((wide[mask] == 7.0).all()), f"mlp_block {(m, k, n, h)}: wrote outside the destination"
    pkg.kernel._mlp_scratch_bytes = scratch_bytes
print(f"swept {launches} launches under the range-checked build: status 0 throughout")
"""


def test_every_small_shape_through_every_plan_under_the_range_checked_build():
    lib = os.path.join(ROOT, "sol_execbench_b200_kernels_b200", "libgateup_bounds.so")
    assert os.path.exists(lib), "libgateup_bounds.so is missing: python -m sol_execbench_b200_kernels_b200.build --bounds"
    proc = subprocess.run([sys.executable, "-c", _SWEEP], env=dict(os.environ, GU_ROOT=ROOT), capture_output=True,
                          text=True, timeout=1500)
    assert proc.returncode == 0, proc.stdout[-2000:] + proc.stderr[-4000:]
    assert "status 0 throughout" in proc.stdout


_PROJ_SWEEP = r"""
import os, sys
sys.path.insert(0, os.environ["GU_ROOT"])
import sol_execbench_b200_kernels_b200.build as B
B.SIDE_LIB_PATH = B.SIDE_BOUNDS_LIB_PATH
import torch
from sol_execbench_b200_kernels_b200 import _sideops_cabi, side_ops

assert _sideops_cabi.lib.so_is_range_checked_build() == 1
dev = torch.device("cuda:0")
side_ops.last_status()
launches = 0
g = torch.Generator().manual_seed(3)
few = [1, 31, 33, 128, 129]
# (small N: 64-column tiles up to 128 rows; the large ones give 96, 128, 160, 192, 224 and 256 columns, and two rounds)
for k in (8, 64, 72, 200):
    for n in (8, 248, 264, 520) + ((9480, 14216, 18952, 23688, 28424, 33160, 40008) if k in (8, 200) else ()):
        weight = (torch.randn(n, k, generator=g) * 0.1).to(torch.bfloat16).to(dev)
        bias = (torch.randn(n, generator=g) * 0.2).to(torch.bfloat16).to(dev)
        for m in few if n > 520 else list(range(1, 131)) + [255, 256, 257, 300, 383, 384, 385, 511, 513]:
            hidden = (torch.randn(m, k, generator=g) * 0.5).to(torch.bfloat16).to(dev)
            buf = torch.full((m + 2, n), 7.0, dtype=torch.bfloat16, device=dev)     # canary rows around the result
            out = buf[1:m + 1]
            side_ops.mamba_in_proj(hidden, weight, bias, out)
            launches += 1
            torch.cuda.synchronize()
            code, detail = side_ops.last_status()
            assert code == 0, f"M={m} K={k} N={n}: device status {code}, detail {detail:#x}"
            exact = hidden.double() @ weight.double().t() + bias.double()
            mags = hidden.double().abs() @ weight.double().abs().t() + bias.double().abs()
            err = (out.double() - exact).abs()
            assert bool((err <= exact.abs() * 2.0 ** -8 + mags * 2.0 ** -16 + 1e-30).all()), (m, k, n, float(err.max()))
            assert bool((buf[0] == 7.0).all()) and bool((buf[m + 1] == 7.0).all()), f"M={m} K={k} N={n}: wrote outside"
print(f"swept {launches} projection launches under the range-checked build: status 0 throughout")
"""


def test_projection_small_shapes_under_the_range_checked_build():
    """The bf16 projection GEMM relies on TMA's out-of-range behaviour for ragged M, K and N (reads give zero, stores
    are clipped): every M = 1 ... 130 and a few around the 256-row pair tile, at K and N that are and are not whole
    tiles, inside the range-checked build of libsideops, with canary rows around the destination."""
    lib = os.path.join(ROOT, "sol_execbench_b200_kernels_b200", "libsideops_bounds.so")
    assert os.path.exists(lib), "libsideops_bounds.so is missing: python -m sol_execbench_b200_kernels_b200.build --bounds"
    proc = subprocess.run([sys.executable, "-c", _PROJ_SWEEP], env=dict(os.environ, GU_ROOT=ROOT), capture_output=True,
                          text=True, timeout=1500)
    assert proc.returncode == 0, proc.stdout[-2000:] + proc.stderr[-4000:]
    assert "status 0 throughout" in proc.stdout


def test_the_regular_library_is_not_the_range_checked_build():
    from sol_execbench_b200_kernels_b200 import _cabi, _sideops_cabi

    assert _cabi.lib.gu_is_range_checked_build() == 0
    assert _sideops_cabi.lib.so_is_range_checked_build() == 0
