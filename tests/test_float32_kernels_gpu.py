"""The float32 path's product at the sizes where its forms meet, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def K():
    from logssms_b200.ops import kernels
    return kernels


# rows: both sides of the streaming form's and the tiles' limits; features and K: remainders of the tiles, K that is no
# multiple of 4 and rows that start off a 16-byte boundary (4-byte copies), one part of K and several
@pytest.mark.parametrize("M", [1, 2, 3, 4, 7, 8, 9, 16, 17, 32, 33, 64, 65, 129, 300])
@pytest.mark.parametrize("N,Kd,lead", [(1, 4, 0), (66, 100, 4), (64, 1030, 0), (2050, 128, 0), (768, 1024, 1), (1024, 2052, 8)])
def test_gemm_f32_forms(M, N, Kd, lead):
    g = torch.Generator().manual_seed(M * 31 + N)
    wide = torch.randn(M, lead + Kd + 4, generator=g)
    w, b = torch.randn(N, Kd, generator=g), torch.randn(N, generator=g)
    a = wide[:, lead:lead + Kd].double()
    out = K().gemm_f32(wide.cuda()[:, lead:lead + Kd], w.cuda(), b.cuda(), 0.5).cpu().double()
    # K products summed in any order, the bias and the scale: every rounding is at most 2^-24 of the sum of magnitudes
    bound = (Kd + 3) * 2.0 ** -24 * (a.abs() @ w.double().abs().T + b.double().abs()) * 0.5
    assert bool(((out - (a @ w.double().T + b.double()) * 0.5).abs() <= bound).all())
    plain = K().gemm_f32(wide.cuda()[:, lead:lead + Kd], w.cuda()).cpu().double()
    assert bool(((plain - a @ w.double().T).abs() <= 2 * bound).all())
