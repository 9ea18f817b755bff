"""The quick acceptance in front of the checks of `run` and `mlp_block`, against those checks, on stand-ins for CUDA tensors:
it accepts a call only where they do, with the same sizes, and accepts every plain one."""
import itertools

import pytest
import torch

from sol_execbench_b200_kernels_b200 import kernel


class Fake:
    """A CPU tensor that says it is on a CUDA device."""

    def __init__(self, t, index=0, cuda=True):
        self.t, self.index, self.is_cuda = t, index, cuda
        self.device = torch.device("cuda", index) if cuda else torch.device("cpu")

    shape = property(lambda self: self.t.shape)
    dtype = property(lambda self: self.t.dtype)

    def __getattr__(self, name):  # dim, stride, is_contiguous
        return getattr(self.t, name)

    def get_device(self):
        return self.index if self.is_cuda else -1


def _operands(m=3, k=256, n=384):
    kb, nb = k // 128, n // 128
    e4m3 = [torch.zeros(r, c, dtype=torch.uint8).view(torch.float8_e4m3fn) for r, c in ((m, k), (n, k), (n, k))]
    return [e4m3[0], torch.zeros(m, kb), e4m3[1], torch.zeros(nb, kb), e4m3[2], torch.zeros(nb, kb),
            torch.zeros(m, n, dtype=torch.bfloat16)]


def _both(operands):
    quick = kernel._plainly_valid(*operands)
    try:
        full = kernel._validate(*operands)
    except (ValueError, IndexError):
        full = None
    return quick, full


@pytest.mark.parametrize("m,k,n", [(1, 128, 128), (3, 256, 384), (129, 128, 256)])
def test_plain_calls_are_accepted_at_once(m, k, n):
    operands = [Fake(t) for t in _operands(m, k, n)]
    assert _both(operands) == ((m, k, n), (m, k, n))
    wide = torch.zeros(m + 1, n + 64, dtype=torch.bfloat16)
    for view in (wide[:m, :n], wide[1:, 64:]):  # a column slice of a wider buffer
        assert _both(operands[:6] + [Fake(view)]) == ((m, k, n), (m, k, n))


def _variants(t):
    yield Fake(t, index=1)
    yield Fake(t, cuda=False)
    yield Fake(t.t())
    yield Fake(t[None])
    yield Fake(t[:-1])
    yield Fake(t[:, :-1])
    yield Fake(torch.zeros(0, t.shape[1]).to(t.dtype) if t.dtype != torch.float8_e4m3fn else t[:0])
    yield Fake(torch.zeros(t.shape, dtype=torch.float16))
    yield Fake(torch.zeros(t.shape, dtype=torch.float64))
    if t.dtype != torch.float8_e4m3fn:
        yield Fake(torch.zeros(t.shape[0], 2 * t.shape[1], dtype=t.dtype)[:, ::2])
        yield Fake(t[:1].expand(t.shape))
    else:
        yield Fake(torch.zeros(t.shape[0], 2 * t.shape[1], dtype=torch.uint8)[:, ::2].view(torch.uint8).contiguous().view(t.dtype))
        yield Fake(torch.zeros(t.shape[0], 2 * t.shape[1], dtype=torch.uint8).view(t.dtype)[:, :t.shape[1]])


def test_whatever_the_checks_refuse_is_left_to_them():
    base = _operands()
    cases = 0
    for i, j in itertools.product(range(7), range(7)):
        for v, w in itertools.product(_variants(base[i]), _variants(base[j])):
            operands = [Fake(t) for t in base]
            operands[i] = v
            if j != i:
                operands[j] = w
            quick, full = _both(operands)
            assert quick is None or quick == full, (i, j)
            cases += 1
    assert cases > 5000
    for m, k, n in ((3, 200, 384), (3, 256, 400), (3, 64, 384)):  # sizes outside the contract
        ok = [Fake(t) for t in _operands(3, max(128, k // 128 * 128), max(128, n // 128 * 128))]
        ok[0], ok[2], ok[4] = (Fake(torch.zeros(r, k, dtype=torch.uint8).view(torch.float8_e4m3fn)) for r in (m, n, n))
        ok[6] = Fake(torch.zeros(m, n, dtype=torch.bfloat16))
        assert _both(ok) == (None, None)


class _Accepted(Exception):
    pass


def _mlp_operands(m=3, k=256, n=384, h=128):
    out = [torch.zeros(m, k, dtype=torch.bfloat16)]
    for rows, cols in ((n, k), (n, k), (h, n)):
        out += [torch.zeros(rows, cols, dtype=torch.uint8).view(torch.float8_e4m3fn), torch.zeros(rows // 128, cols // 128)]
    return out + [torch.zeros(m, h, dtype=torch.bfloat16)]


def test_mlp_block_refuses_what_its_full_checks_refuse(monkeypatch):
    """`mlp_block` with its quick acceptance and with `_check` on every call: the same calls get past, with the same messages."""
    def layout(*shape):
        raise _Accepted(*shape)

    monkeypatch.setattr(kernel, "_mlp_layout", layout)
    quick = kernel._plain

    def outcome(operands, plain):
        monkeypatch.setattr(kernel, "_plain", plain)
        try:
            kernel.mlp_block(*operands)
        except (_Accepted, ValueError, IndexError) as e:
            return type(e), str(e)

    def both(operands):
        got = outcome(operands, quick), outcome(operands, lambda operands, index: False)
        assert got[0] == got[1] and got[0] is not None
        return got[0][0]

    base = _mlp_operands()
    assert both([Fake(t) for t in base]) is _Accepted
    wide = torch.zeros(4, 192, dtype=torch.bfloat16)
    assert both([Fake(t) for t in base[:7]] + [Fake(wide[1:, 64:])]) is _Accepted
    pitched = Fake(torch.zeros(3, 264)[:, :256])
    assert both([pitched] + [Fake(t) for t in base[1:]]) is _Accepted
    refused = 0
    for i, j in itertools.product(range(8), range(8)):
        for v, w in itertools.product(_variants(base[i]), _variants(base[j])):
            operands = [Fake(t) for t in base]
            operands[i] = v
            if j != i:
                operands[j] = w
            refused += both(operands) is not _Accepted
    assert refused > 5000


def test_packed_arguments_have_the_structures_layout():
    import ctypes

    from sol_execbench_b200_kernels_b200 import _cabi

    problem = tuple(range(1, 14)) + (-3, 7)
    assert bytes(_cabi.GuProblem(*problem)) == _cabi.PROBLEM_ARGS.pack(*problem)
    mlp = tuple(range(1, 19)) + (1, 0)
    assert bytes(_cabi.GuMlp(*mlp)) == _cabi.MLP_ARGS.pack(*mlp)
    assert ctypes.sizeof(_cabi.GuMlp) == _cabi.MLP_ARGS.size
