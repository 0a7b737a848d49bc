"""The float32 path's product and its scan of long portions at the sizes where their forms meet, against float64."""
import pytest
import torch

from plain import falcon_h1_plain as P

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


@pytest.mark.parametrize("shape", [(4, 16, 16, 1), (6, 24, 32, 2), (3, 64, 128, 1), (2, 40, 256, 2), (5, 8, 20, 5)])
@pytest.mark.parametrize("lead", [0, 1])                     # 1: B and C off their 16-byte boundaries
def test_ssm_scan_in_blocks(shape, lead):
    """Portions of one token to several blocks, resumed from a state, with the gate; requests of one launch differ."""
    nh, Pd, N, G = shape
    g = torch.Generator().manual_seed(nh * N + lead)
    inner, C = nh * Pd, nh * Pd + 2 * G * N
    lens, starts = [9, 1, 48, 17, 0, 8], [0, 5, 3, 0, 2, 7]
    T = sum(lens)
    A_log, D = torch.log(1 + 15 * torch.rand(nh, generator=g)), 1 + 0.1 * torch.randn(nh, generator=g)
    dt_bias = 0.5 * torch.randn(nh, generator=g) - 2.0
    wide = torch.randn(T, lead + C + 3, generator=g)
    dt = torch.randn(T, nh, generator=g)
    gate = torch.randn(T, inner + 2, generator=g)[:, :inner]
    before = torch.randn(7, nh, Pd, N, generator=g)
    slots = torch.tensor([6, 1, 0, 4, 2, 3], dtype=torch.int32)
    cu = torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).int()
    state = before.clone().cuda()
    state[[6, 4]] = float("nan")                            # what a portion that starts at 0 finds in its slot is not read
    y = K().ssm_scan(wide.cuda()[:, lead:lead + C], dt.cuda(), A_log.cuda(), dt_bias.cuda(), D.cuda(), state, cu.cuda(),
                     torch.tensor(starts, dtype=torch.int32).cuda(), slots.cuda(), len(lens), nh, Pd, N, G, 0.8,
                     gate.cuda(), 0.6, longest=max(lens)).cpu().double()
    rep = nh // G
    for r, n in enumerate(lens):
        lo = int(cu[r])
        row = wide[lo:lo + n, lead:lead + C].double()
        x, B, Cm = row[:, :inner].reshape(n, nh, Pd), row[:, inner:inner + G * N].reshape(n, G, N), row[:, inner + G * N:].reshape(n, G, N)
        step = P.softplus20(dt[lo:lo + n].double() * 0.8 + dt_bias.double())
        S = before[int(slots[r])].double() if starts[r] else torch.zeros(nh, Pd, N, dtype=torch.float64)
        for t in range(n):
            Bt, Ct = B[t].repeat_interleave(rep, 0), Cm[t].repeat_interleave(rep, 0)
            S = S * torch.exp(-torch.exp(A_log.double()) * step[t])[:, None, None] + (x[t] * step[t][:, None])[..., None] * Bt[:, None]
            want = (S * Ct[:, None]).sum(-1) + D.double()[:, None] * x[t]
            want = want.reshape(-1) * P.silu(gate[lo + t].double() * 0.6)
            assert float((y[lo + t] - want).abs().max() / want.abs().max()) <= 2e-5, (r, t)
        got = state[int(slots[r])].cpu().double()
        assert n == 0 or float((got - S).abs().max() / S.abs().max()) <= 2e-5, r
    assert torch.equal(state[[2, 5]].cpu(), before[[2, 5]])      # a request without tokens, a slot of nobody
