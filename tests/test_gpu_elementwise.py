"""The elementary functions of the kernels against FP64, at error bounds of their own."""
import ctypes

import pytest
import torch

from solvedelta_b200 import _lib

pytestmark = pytest.mark.gpu
INF, NAN = float("inf"), float("nan")
TINY = 2.0 ** -126   # the smallest normal number


def _apply(function, x):
    x = x.cuda()
    y = torch.empty_like(x)
    _lib.check(_lib.load_diagnostics().sd_debug_elementwise(function, x.data_ptr(), y.data_ptr(), x.numel(),
                                                            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return y.cpu()


def test_exponential():
    gen = torch.Generator().manual_seed(1)
    x = torch.cat([torch.linspace(-87.3, 88.7, 200003), torch.randn(100000, generator=gen),
                   1e-6 * torch.randn(10000, generator=gen), torch.tensor([0.0, 1e-40, -1e-40])])
    want = x.double().exp()
    # 2^-22 of the instruction; the product x log2 e rounded (2^-24 of it) with a rounded constant (half of that):
    # |x log2 e| 1.5 2^-24 in the exponent, times ln 2 in the result
    assert ((_apply(0, x).double() - want).abs() <= want * (2.0 ** -22 + 1.5 * x.double().abs() * 2.0 ** -24)).all()
    edges = _apply(0, torch.tensor([-INF, -200.0, -88.0, 89.0, INF, NAN]))
    assert edges[:3].tolist() == [0.0, 0.0, 0.0] and edges[3:5].tolist() == [INF, INF] and edges[5].isnan()


def test_reciprocal():
    gen = torch.Generator().manual_seed(2)
    x = torch.cat([torch.linspace(1.0, 4.0, 300007), torch.exp2(252.0 * torch.rand(200000, generator=gen) - 126.0)])
    x = torch.cat([x, -x])
    want = 1.0 / x.double()
    assert ((_apply(1, x).double() - want).abs() <= want.abs() * 2.0 ** -23).all()
    edges = _apply(1, torch.tensor([INF, -INF, 0.0, TINY / 2, 2.0 ** 127, NAN]))
    assert edges[:2].tolist() == [0.0, 0.0] and edges[2:4].tolist() == [INF, INF] and edges[4] == 0.0 and edges[5].isnan()


def test_tf32_operand_rounding():
    """To the nearest of ten fraction bits, ties away from zero, as the conversion instruction does it; infinities and the
    NaN that arithmetic returns (0x7fffffff) stay what they are."""
    gen = torch.Generator().manual_seed(3)
    bits = torch.cat([torch.randint(0, 0x7f800000, (400000,), generator=gen), torch.arange(0x3f800000, 0x3f804000)])
    bits = bits.to(torch.int32)
    x = torch.cat([bits, bits | torch.tensor(-2 ** 31, dtype=torch.int32)]).view(torch.float32)
    fraction = torch.frexp(x.double())
    want = torch.ldexp(torch.sign(x.double()) * (fraction.mantissa.abs() * 2048 + 0.5).floor(), fraction.exponent - 11)
    normal = x.abs() >= TINY   # below it the spacing is fixed, not ten bits
    assert torch.equal(_apply(2, x).double()[normal], want.float().double()[normal])
    assert _apply(2, torch.tensor([INF, -INF])).tolist() == [INF, -INF]
    nans = torch.tensor([0x7fffffff, 0x7fc00000, -0x400000, 0x7fbfffff, 0x7f802000], dtype=torch.int32).view(torch.float32)
    assert _apply(2, nans).isnan().all()
