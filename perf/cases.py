"""The work that users of this package have it do, as measurable cases: `listed()` names them, `draw(rng)` gives more of
the same ranges.  Everything goes through the public entry points, with weights of the scale that real projections have.

Operations: `gateup` is `run` (the FP8 gate/up projection with SwiGLU), `mlp` is `mlp_block` (quantise, gate/up, down
projection), `mamba` is `mamba_conv1d_with_gating` and `rmsnorm` is `rmsnorm_qk`.
"""
import math

import torch

import sol_execbench_b200_kernels_b200 as gu
from sol_execbench_b200_kernels_b200 import side_ops, workloads

BLOCK = 128
# (K, N) of the gate/up projections that the package's shapes, benchmark and kernel-choice tests name
PROJECTIONS = ((4096, 14336), (8192, 28672), (7168, 18432), (3584, 18944), (2048, 5632), (5120, 13824), (1024, 4096),
               (7168, 2304))
MAX_MACS = 16384 * 7168 * 18432  # of the largest listed case


def listed():
    return [
        # one user's decode step on an 8B-class model: the smallest call, all latency and weight reads
        {"name": "gateup_decode_1", "op": "gateup", "m": 1, "k": 4096, "n": 14336},
        # a decode batch on a 70B-class model: weight streaming
        {"name": "gateup_decode_70b", "op": "gateup", "m": 16, "k": 8192, "n": 28672},
        # a ragged mid-sized batch (a busy decode server, or a short prompt) at the reference's own K and N
        {"name": "gateup_ragged_batch", "op": "gateup", "m": 83, "k": 3584, "n": 18944},
        # a prompt whose length is no multiple of anything, at the reference's own K and N
        {"name": "gateup_prompt_1000", "op": "gateup", "m": 1000, "k": 3584, "n": 18944},
        # the headline prefill
        {"name": "gateup_prefill_8b", "op": "gateup", "m": 4096, "k": 4096, "n": 14336},
        # the largest prefill (the shape that is column-sharded over several GPUs), on one GPU
        {"name": "gateup_prefill_large", "op": "gateup", "m": 16384, "k": 7168, "n": 18432},
        # the whole MLP of a decode step for a handful of users, bf16 activations
        {"name": "mlp_decode_8", "op": "mlp", "m": 8, "k": 4096, "n": 14336, "dtype": "bf16"},
        # the whole MLP for one chunk of a chunked prefill, fp32 activations
        {"name": "mlp_chunk_515", "op": "mlp", "m": 515, "k": 4096, "n": 14336, "dtype": "fp32"},
        # the whole MLP for a prefill batch, bf16 activations
        {"name": "mlp_prefill", "op": "mlp", "m": 4096, "k": 4096, "n": 14336, "dtype": "bf16"},
        # a short prompt through the Mamba block's projection, convolution and gate
        {"name": "mamba_b1_l128", "op": "mamba", "batch": 1, "seq": 128},
        # a batch of two prompts with padding, of a length that is no multiple of a tile
        {"name": "mamba_b2_l1000", "op": "mamba", "batch": 2, "seq": 1000},
        # query / key normalisation of one image with its text tokens
        {"name": "rmsnorm_4608", "op": "rmsnorm", "tokens": 4608, "heads": 48},
    ]


def _log_int(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    op = rng.choice(("gateup", "gateup", "gateup", "mlp", "mlp", "mamba", "rmsnorm"))
    if op == "rmsnorm":
        return {"op": op, "tokens": _log_int(rng, 64, 16384), "heads": rng.choice((16, 24, 48))}
    if op == "mamba":
        batch = rng.choice((1, 1, 2, 3, 4))
        return {"op": op, "batch": batch, "seq": _log_int(rng, 17, 8192 // batch)}
    if rng.random() < 0.5:
        k, n = rng.choice(PROJECTIONS)
    else:
        k, n = BLOCK * _log_int(rng, 8, 64), BLOCK * _log_int(rng, 16, 224)
    # an MLP block multiplies half as much again
    m = _log_int(rng, 1, min(16384, MAX_MACS // (k * n) * 2 // (3 if op == "mlp" else 2)))
    case = {"op": op, "m": m, "k": k, "n": n}
    if op == "mlp":
        case["dtype"] = rng.choice(("bf16", "bf16", "fp32"))
    return case


CHANNELS, HIDDEN = 16384, 8192  # the Mamba block's convolution channels and model width


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _weights(g, rows, cols):
    return workloads.quantize_weight_128x128(torch.randn(rows, cols, generator=g, device="cuda") * 0.02)


def prepare(case, seed):
    op = case["op"]
    g = _generator(seed)
    if op == "gateup":
        m, k, n = case["m"], case["k"], case["n"]
        inputs = workloads.make_inputs(m, k, n, seed=seed, device="cuda")
        return {"op": op, "args": inputs.args(), "output": torch.empty(m, n, dtype=torch.bfloat16, device="cuda")}
    if op == "mlp":
        m, k, n = case["m"], case["k"], case["n"]
        x = torch.randn(m, k, generator=g, device="cuda")
        x = x.to(torch.bfloat16) if case["dtype"] == "bf16" else x
        weights = (*_weights(g, n, k), *_weights(g, n, k), *_weights(g, k, n))
        return {"op": op, "x": x, "weights": weights}
    if op == "mamba":
        batch, seq = case["batch"], case["seq"]
        bf16 = dict(device="cuda", dtype=torch.bfloat16)
        hidden = torch.randn(batch, seq, HIDDEN, generator=g, **bf16)
        mask = torch.ones(batch, seq, **bf16)
        for b in range(1, batch):  # prompts of unequal length, padded on the left
            mask[b, : b * seq // 10] = 0
        weight = torch.empty(2 * CHANNELS, HIDDEN, **bf16).normal_(0, 0.02, generator=g)
        bias = torch.empty(2 * CHANNELS, **bf16).normal_(0, 0.1, generator=g)
        conv_w = torch.empty(CHANNELS, 1, 4, **bf16).normal_(0, 0.5, generator=g)
        conv_b = torch.empty(CHANNELS, **bf16).normal_(0, 0.5, generator=g)
        return {"op": op, "args": (hidden, mask, weight, bias, conv_w, conv_b)}
    tokens, heads = case["tokens"], case["heads"]
    query = torch.randn(1, tokens, heads, 128, generator=g, device="cuda") * 1.5
    key = torch.randn(1, tokens, heads, 128, generator=g, device="cuda") * 0.7 + 0.1
    weight_q = 1.0 + 0.1 * torch.randn(heads, 128, generator=g, device="cuda")
    weight_k = 1.0 + 0.1 * torch.randn(heads, 128, generator=g, device="cuda")
    return {"op": op, "args": (query, key, weight_q, weight_k, 1e-6, torch.empty_like(query), torch.empty_like(key))}


def run(state):
    op = state["op"]
    if op == "gateup":
        gu.run(*state["args"], state["output"])
        return state["output"]
    if op == "mlp":
        return gu.mlp_block(state["x"], *state["weights"])
    if op == "mamba":
        return side_ops.mamba_conv1d_with_gating(*state["args"])
    side_ops.rmsnorm_qk(*state["args"])
    return state["args"][5:]


def work(case):
    op = case["op"]
    if op == "gateup":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": workloads.algorithmic_bytes(m, k, n), "flops": workloads.algorithmic_flops(m, k, n)}
    if op == "mlp":  # activations in, three weights with their scales, bf16 result out; the rest may stay on the chip
        m, k, n = case["m"], case["k"], case["n"]
        weights = 3 * (n * k + 4 * (n // BLOCK) * (k // BLOCK))
        return {"bytes": m * k * (2 if case["dtype"] == "bf16" else 4) + weights + 2 * m * k, "flops": 6 * m * n * k}
    if op == "mamba":  # hidden states, mask, weights and biases in; convolved channels and gate out
        rows = case["batch"] * case["seq"]
        read = 2 * (rows * HIDDEN + rows + 2 * CHANNELS * (HIDDEN + 1) + 5 * CHANNELS)
        return {"bytes": read + 2 * rows * 2 * CHANNELS, "flops": 2 * rows * HIDDEN * 2 * CHANNELS}
    elements = case["tokens"] * case["heads"] * 128
    return {"bytes": 16 * elements + 8 * case["heads"] * 128, "flops": 8 * elements}


def tolerance(case):
    """About four times the largest difference seen between this package and the same formulas in float64 with the
    documented rounding steps (gateup 4e-5 ... 1e-4 and 0.016, mlp 4e-4 and 0.022, mamba 3e-4 and 0.039, rmsnorm 6e-8
    and 2.8e-7): a sum in another order flips a bf16 (or e4m3) rounding here and there."""
    return {"gateup": {"rel": 3e-4, "max": 6e-2}, "mlp": {"rel": 1.6e-3, "max": 9e-2},
            "mamba": {"rel": 1.2e-3, "max": 1.5e-1}, "rmsnorm": {"rel": 2.5e-7, "max": 1.1e-6}}[case["op"]]


def _dequantized(q, scale, rows_per_scale):
    s = scale.double().repeat_interleave(BLOCK, 1)
    return q.float().double() * (s if rows_per_scale == 1 else s.repeat_interleave(rows_per_scale, 0))


def _block_matmul(q, scale, weight, scale_weight):
    return _dequantized(q, scale, 1) @ _dequantized(weight, scale_weight, BLOCK).t()


def _bf16(t):
    return t.float().to(torch.bfloat16).double()


def _swiglu(gate, up):
    gate, up = _bf16(gate), _bf16(up)
    return _bf16(gate * torch.sigmoid(gate)) * up


def _quantized(t):
    t = t.float().reshape(t.shape[0], -1, BLOCK)
    amax = t.abs().amax(-1, keepdim=True).clamp_min(1e-12)
    scale = amax / torch.full_like(amax, 448.0)  # a tensor: by a plain number the GPU would multiply by its reciprocal
    q = (t / scale).clamp(-448.0, 448.0).to(torch.float8_e4m3fn)
    return q.reshape(t.shape[0], -1), scale[:, :, 0]


@torch.no_grad()
def exact(case, seed):
    """The formulas in float64; the roundings between the steps (e4m3 activations, bf16 gate, up, SiLU, convolution and
    sigmoid) are part of the operations and are kept, the last one of a result is not."""
    state = prepare(case, seed)
    op = state["op"]
    if op == "gateup":
        x, scale_x, gate_w, scale_gate, up_w, scale_up = state["args"]
        gate = _block_matmul(x, scale_x, gate_w, scale_gate)
        return _swiglu(gate, _block_matmul(x, scale_x, up_w, scale_up))
    if op == "mlp":
        gate_w, scale_gate, up_w, scale_up, down_w, scale_down = state["weights"]
        x, scale_x = _quantized(state["x"])
        gate = _block_matmul(x, scale_x, gate_w, scale_gate)
        middle, scale_middle = _quantized(_bf16(_swiglu(gate, _block_matmul(x, scale_x, up_w, scale_up))))
        return _block_matmul(middle, scale_middle, down_w, scale_down)
    if op == "mamba":
        hidden, mask, weight, bias, conv_w, conv_b = state["args"]
        batch, seq = mask.shape
        flat = hidden.reshape(batch * seq, HIDDEN).double()
        projected = torch.empty(batch * seq, 2 * CHANNELS, dtype=torch.float64, device="cuda")
        for c in range(0, 2 * CHANNELS, 4096):
            projected[:, c:c + 4096] = flat @ weight[c:c + 4096].double().t() + bias[c:c + 4096].double()
        projected = projected.view(batch, seq, 2 * CHANNELS)
        x = _bf16(_bf16(projected[:, :, :CHANNELS]) * mask.double()[:, :, None])
        taps = conv_w.double().reshape(CHANNELS, 4)
        x = torch.nn.functional.pad(x, (0, 0, 3, 0))
        conv = conv_b.double() + sum(x[:, t:t + seq] * taps[:, t] for t in range(4))
        conv = _bf16(conv)
        out = torch.where((mask >= 0.5)[:, :, None], conv * _bf16(torch.sigmoid(conv)), 0.0)
        return out.transpose(1, 2).contiguous(), projected[:, :, CHANNELS:].transpose(1, 2)
    query, key, weight_q, weight_k, eps = state["args"][:5]

    def norm(t, w):
        t = t.double()
        return t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True) + eps) * w.double()

    return norm(query, weight_q), norm(key, weight_k)
