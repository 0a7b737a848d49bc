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


# tiles of 128 x 128 and blocks of 64 values of k: remainders of each, one part of K and several (3, 5, 6 and 7 of them as well: parts
# of 42 and 43, 25 and 26 rows ...), a last wave of a few tiles cut finer, rows off the others' stride
@pytest.mark.parametrize("M,N,Kd,lead", [(33, 1540, 1024, 0), (65, 4100, 132, 4), (128, 130, 4096, 0), (129, 1024, 516, 8), (300, 2049, 260, 0),
                                         (601, 1024, 1536, 0), (129, 1750, 1284, 0), (300, 1000, 2100, 0), (300, 880, 2052, 4),
                                         (601, 4096, 1024, 0)])
def test_gemm_f32_on_the_tensor_cores(M, N, Kd, lead):
    g = torch.Generator().manual_seed(M * 31 + N)
    wide = torch.randn(M, lead + Kd + 4, generator=g) * torch.exp(2 * torch.randn(M, 1, generator=g))
    w, b = torch.randn(N, Kd, generator=g), torch.randn(N, generator=g)
    x, wd = wide.cuda()[:, lead:lead + Kd], w.cuda()
    assert K()._gemm_f32_tc_ok(x, wd)
    a = wide[:, lead:lead + Kd].double()
    # six of the nine products of the operands' three parts are taken: what is left out is below 2^-25 |a w|; the tensor core
    # drops less than 2^-23 of the largest term of each of the sums it makes (17 terms, four sums to a block of k, the small
    # products' 2^-8 of that), the blocks are added up with rounded additions
    bound = ((Kd + 63) // 64 + 8) * 2.0 ** -22 * (a.abs() @ w.double().abs().T + b.double().abs())
    out = K().gemm_f32(x, wd, b.cuda(), 0.5).cpu().double()
    want = (a @ w.double().T + b.double()) * 0.5
    assert bool(((out - want).abs() <= bound).all())
    assert float((out - want).norm() / want.norm()) <= 4e-7        # as the plain form's (1.5e-7 .. 5e-7), far below one part less (2e-6)
    K().check_kernel_errors()


@pytest.mark.parametrize("M,N,Kd,most", [(800, 3072, 12288, 2.1e-7), (129, 12288, 3072, 1.37e-7), (2048, 1280, 3072, 1.28e-7)])
def test_gemm_f32_parts_of_k_are_no_longer_than_they_were(M, N, Kd, most):
    """Each block of 64 values of k is one rounded addition: the error grows with the blocks in a part.  With half to a quarter of the
    parts it is 2.8e-7, 1.5e-7 and 1.5e-7 here, with all of them 1.6e-7, 1.2e-7 and 1.1e-7."""
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w = torch.randn(M, Kd, generator=g, device="cuda"), torch.randn(N, Kd, generator=g, device="cuda")
    assert K()._gemm_f32_tc_ok(x, w)
    want = x.double() @ w.double().T
    assert float((K().gemm_f32(x, w).double() - want).norm() / want.norm()) <= most
    K().check_kernel_errors()


def test_gemm_f32_on_the_tensor_cores_keeps_infinities():
    x, w = torch.ones(70, 1024), torch.ones(1024, 1024)
    x[3, 5], x[4, 6], x[5, 7], x[6, 8] = float("inf"), float("nan"), 3.4e38, 1e-42
    w[9, 5] = -2.0
    w[10, 7] = 1.5
    out = K().gemm_f32(x.cuda(), w.cuda()).cpu()
    want = x.double() @ w.double().T
    want = want.float()                                     # beyond the largest float32: infinity
    assert torch.equal(out.isinf(), want.isinf()) and torch.equal(out.isnan(), want.isnan())
    assert torch.equal(out[want.isinf()], want[want.isinf()])
    fine = want.isfinite()
    assert float(((out - want)[fine] / want[fine]).abs().max()) <= 1e-6


@pytest.mark.parametrize("ea,ew", [(0, 0), (-104, 0), (0, -112), (-118, 10), (-140, 40), (100, -60), (60, 10), (60, 25), (105, -100)])
def test_gemm_f32_on_the_tensor_cores_over_the_range_of_exponents(ea, ew):
    """Values from the smallest float32 (multiples of 2^-149) to sums and values past the kernel's own range keep the precision
    of 32-bit arithmetic: a part of a value must not fall below the smallest number of its format."""
    g = torch.Generator().manual_seed(ea + 200)
    x, w = torch.ldexp(torch.randn(65, 1024, generator=g), torch.tensor(ea)), torch.ldexp(torch.randn(1024, 1024, generator=g), torch.tensor(ew))
    a, b = x.cuda(), w.cuda()
    assert K()._gemm_f32_tc_ok(a, b)
    out, want = K().gemm_f32(a, b).cpu().double(), x.double() @ w.double().T
    if ea < 104 and ea + ew < 75:
        assert float((out - want).norm() / want.norm()) <= 4e-7      # as at ordinary magnitudes
    else:                                                            # one chain of fused multiply-adds
        assert bool(((out - want).abs() <= 1024 * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)).all())
    K().check_kernel_errors()


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


@pytest.mark.parametrize("lens", [[255, 256, 3, 257], [272, 0, 513, 17], [528]])
@pytest.mark.parametrize("nh,Pd,N,G,lead", [(3, 16, 128, 1, 0), (2, 24, 40, 2, 1)])
def test_ssm_scan_in_blocks_past_the_table_of_steps(lens, nh, Pd, N, G, lead):
    """The steps and decays of 256 tokens are made at a time: portions that end before, at and behind that line, or fill it twice."""
    g = torch.Generator().manual_seed(sum(lens) + N)
    inner, C, T, B = nh * Pd, nh * Pd + 2 * G * N, sum(lens), len(lens)
    starts = [5 * (r % 2) for r in range(B)]
    A_log, D = torch.log(1 + 15 * torch.rand(nh, generator=g)), 1 + 0.1 * torch.randn(nh, generator=g)
    dt_bias = 0.5 * torch.randn(nh, generator=g) - 2.0
    wide, dt = torch.randn(T, lead + C + 3, generator=g), torch.randn(T, nh, generator=g)
    gate = torch.randn(T, inner, generator=g)
    before = torch.randn(B + 1, nh, Pd, N, generator=g)
    slots = torch.randperm(B + 1, generator=g)[:B].to(torch.int32)
    cu = torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).int()
    state = before.clone().cuda()
    y = K().ssm_scan(wide.cuda()[:, lead:lead + C], dt.cuda(), A_log.cuda(), dt_bias.cuda(), D.cuda(), state, cu.cuda(),
                     torch.tensor(starts, dtype=torch.int32).cuda(), slots.cuda(), B, nh, Pd, N, G, 0.8, gate.cuda(), 0.6,
                     longest=max(lens)).cpu().double()
    xBC = wide[:, lead:lead + C].double()
    x, Bm, Cm = xBC[:, :inner].reshape(T, nh, Pd), xBC[:, inner:inner + G * N].reshape(T, G, N), xBC[:, inner + G * N:].reshape(T, G, N)
    Bm, Cm = Bm.repeat_interleave(nh // G, 1), Cm.repeat_interleave(nh // G, 1)
    step = P.softplus20(dt.double() * 0.8 + dt_bias.double())
    decay, u = torch.exp(-torch.exp(A_log.double()) * step), x * step[..., None]
    for r, n in enumerate(lens):
        S = before[int(slots[r])].double() if starts[r] else torch.zeros(nh, Pd, N, dtype=torch.float64)
        want = torch.zeros(n, nh, Pd, dtype=torch.float64)
        for i, t in enumerate(range(int(cu[r]), int(cu[r + 1]))):
            S = S * decay[t][:, None, None] + u[t][..., None] * Bm[t][:, None]
            want[i] = (S * Cm[t][:, None]).sum(-1)
        if n == 0:
            continue
        lo = int(cu[r])
        want = ((want + D.double()[:, None] * x[lo:lo + n]).reshape(n, inner) * P.silu(gate[lo:lo + n].double() * 0.6))
        off = (y[lo:lo + n] - want).abs().amax(1) / want.abs().amax(1)
        assert float(off.max()) <= 2e-5, (r, int(off.argmax()))              # the bound of the shorter portions above
        got = state[int(slots[r])].cpu().double()
        assert float((got - S).abs().max() / S.abs().max()) <= 2e-5, r
    idle = sorted(set(range(B + 1)) - {int(s) for s, n in zip(slots, lens) if n})
    assert torch.equal(state[idle].cpu(), before[idle])


@pytest.mark.parametrize("lens", [[1, 4, 5, 2, 33, 3, 0, 16, 17], [1] * 40 + [9], [3] * 12 + [20]])
@pytest.mark.parametrize("nh,Pd,N,lead", [(24, 64, 128, 0), (4, 24, 40, 0), (3, 16, 256, 1)])
def test_ssm_scan_of_few_tokens_beside_longer_portions(lens, nh, Pd, N, lead):
    """Portions up to four tokens skip the blocks, and many of them skip that form: the general form's result either way."""
    g = torch.Generator().manual_seed(sum(lens) + N)
    T, B, inner = sum(lens), len(lens), nh * Pd
    wide, dt = torch.randn(T, lead + inner + 2 * N, generator=g).cuda(), torch.randn(T, nh, generator=g).cuda()
    consts = [torch.rand(nh, generator=g).cuda() for _ in range(3)]
    gate, before = torch.randn(T, inner, generator=g).cuda(), torch.randn(B, nh, Pd, N, generator=g).cuda()
    slots = torch.randperm(B, generator=g).to(torch.int32).cuda()
    cu = torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).int().cuda()
    start = torch.tensor([0 if i % 4 == 1 else 3 for i in range(B)], dtype=torch.int32).cuda()
    results = []
    for longest in (0, max(lens)):
        state = before.clone()
        y = K().ssm_scan(wide[:, lead:], dt, *consts, state, cu, start, slots, B, nh, Pd, N, 1, 0.8, gate, 0.6, longest=longest)
        results.append((y, state))
    for want, got in zip(*results):
        assert float((got - want).abs().max() / want.abs().max()) <= 2e-6          # sums over N in another order: N 2^-24 at most


# a thread per 16-byte piece up to 256, up to four pieces a thread, lengths beyond and no multiple of 4
@pytest.mark.parametrize("H", [4, 64, 124, 128, 132, 1020, 1024, 1028, 4096, 4100, 4098])
@pytest.mark.parametrize("rows", [1, 37])
def test_add_rmsnorm_of_float32_rows(rows, H):
    g = torch.Generator().manual_seed(H)
    x, other, res = (torch.randn(rows, H, generator=g) for _ in range(3))
    w = 1 + 0.1 * torch.randn(H, generator=g)
    (a, b), r = K().add_rmsnorm(x.cuda(), w.cuda(), 1e-5, res.cuda(), other=other.cuda(), in_scales=(0.8, 0.7), out_scales=(1.5, 1.2), in_place=False)
    want = x.double() * 0.8 + other.double() * 0.7 + res.double()
    assert float((r.cpu().double() - want).abs().max()) <= 2.0 ** -22 * float(want.abs().max())
    normed = want / torch.sqrt((want * want).mean(-1, keepdim=True) + 1e-5) * w.double()
    for got, s in ((a, 1.5), (b, 1.2)):                     # some ten roundings and a 32-bit sum of H squares
        assert float((got.cpu().double() - normed * s).abs().max()) <= 4e-6 * float(normed.abs().max())
