"""The decode step's state update (`ssm_step_kernel`) against the token-by-token form, at the sizes where its tiles, its pieces of
16 bytes and its choice of tiles per CTA can go wrong."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("state", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,nh,P,N,G", [(1, 24, 64, 128, 1), (13, 24, 64, 256, 2), (64, 24, 128, 64, 1), (3, 5, 40, 104, 5), (30, 8, 128, 192, 1),
                                        (200, 24, 64, 32, 1), (2, 3, 8, 248, 1)])
def test_ssm_step(B, nh, P, N, G, state):
    from logssms_b200.ops import kernels as k
    g = torch.Generator().manual_seed(B * N + P)
    C, inner = nh * P + 2 * G * N, nh * P
    wide = torch.randn(B, 16 + C + 24, generator=g).to(torch.bfloat16).cuda()
    conv, dt = wide[:, 16:16 + C], torch.randn(B, nh, generator=g).to(torch.bfloat16).cuda()
    A_log, dt_bias, D = torch.rand(nh, generator=g).cuda(), torch.randn(nh, generator=g).cuda(), torch.randn(nh, generator=g).cuda()
    gate = torch.randn(B, inner + 8, generator=g).to(torch.bfloat16).cuda()[:, :inner]
    before = torch.randn(B + 2, nh, P, N, generator=g).to(state).cuda()
    slots = torch.randperm(B + 2, generator=g)[:B].to(torch.int32).cuda()
    lens = torch.ones(B, dtype=torch.int32)
    if B > 2:
        lens[1] = 0                                        # a request without a token keeps its state
    cu = torch.cat([torch.zeros(1, dtype=torch.int32), lens.cumsum(0).int()]).cuda()
    start = torch.tensor([0 if i % 5 == 4 else 3 + i for i in range(B)], dtype=torch.int32).cuda()
    results = []
    for longest in (1, 0):                                 # 0: not known, the general form
        s = before.clone()
        y = k.ssm_scan(conv, dt, A_log, dt_bias, D, s, cu, start, slots, B, nh, P, N, G, 0.8, gate, 0.6, longest=longest)
        results.append((y[:int(cu[-1])].float(), s))
    (y1, s1), (y0, s0) = results
    # the same products and 32-bit sums, those over N in another order where the state is 16-bit; y rounded to bfloat16 twice
    assert torch.equal(s1, s0)
    if state == torch.float32:
        assert torch.equal(y1, y0)
    else:
        assert bool(((y1 - y0).abs() <= 2 * 2.0 ** -7 * torch.maximum(y0.abs(), y0.abs().mean())).all())


@pytest.mark.parametrize("state", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,P,N", [(24, 64, 128), (5, 40, 104), (4, 128, 256), (3, 24, 40)])
def test_a_wrong_longest_loses_no_tokens(nh, P, N, state):
    """`longest` chooses a form: portions of several tokens and of none under `longest=1` give what the general form gives."""
    from logssms_b200.ops import kernels as k
    g = torch.Generator().manual_seed(N + P)
    for lens in ([1, 3, 0, 2, 9], [0, 0, 0]):
        B, T, C, inner = len(lens), max(sum(lens), 1), nh * P + 2 * N, nh * P
        conv, dt = torch.randn(T, C, generator=g).to(torch.bfloat16).cuda(), torch.randn(T, nh, generator=g).to(torch.bfloat16).cuda()
        consts = [torch.rand(nh, generator=g).cuda() for _ in range(3)]
        gate = torch.randn(T, inner, generator=g).to(torch.bfloat16).cuda()
        before = torch.randn(B + 2, nh, P, N, generator=g).to(state).cuda()
        slots = torch.randperm(B + 2, generator=g)[:B].to(torch.int32).cuda()
        cu = torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).int().cuda()
        start = torch.tensor([4, 0, 7, 2, 0][:B], dtype=torch.int32).cuda()
        results = []
        for longest in (1, 0):
            s = before.clone()
            y = k.ssm_scan(conv, dt, *consts, s, cu, start, slots, B, nh, P, N, 1, 0.8, gate, 0.6, longest=longest)
            results.append((y[:sum(lens)].float(), s))
        assert torch.equal(results[0][1], results[1][1])
        # requests of one token: y of the step form, whose sums over N have another order where the state is 16-bit
        (y1, _), (y0, _) = results
        assert bool(((y1 - y0).abs() <= 2 * 2.0 ** -7 * torch.maximum(y0.abs(), y0.abs().mean() if y0.numel() else y0)).all())
        assert bool(torch.equal(y1[1:], y0[1:]))


@pytest.mark.parametrize("dtype,state", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("N", [24, 40, 104, 128])
def test_columns_past_the_states_size_take_no_part_in_an_infinite_input(dtype, state, N):
    """A thread's columns are padded where N is no multiple of them: infinity times a padded column's zero must not enter y."""
    from logssms_b200.ops import kernels as k
    if state == torch.bfloat16 and N == 24:
        N = 40                                             # (a bfloat16 state has the step form from 33 columns on)
    nh, P, T = 3, 32, 1 if dtype == torch.bfloat16 else 20
    g = torch.Generator().manual_seed(N)
    conv = torch.randn(T, nh * P + 2 * N, generator=g)
    conv[:, nh * P:] = conv[:, nh * P:].abs() + 0.1
    conv[T - 1, 5], conv[T - 1, 40] = float("inf"), -float("inf")
    consts = [torch.rand(nh, generator=g).cuda() for _ in range(3)]
    dev = lambda *v: torch.tensor(v, dtype=torch.int32).cuda()
    for longest in (T, 0):
        s = torch.rand(2, nh, P, N, generator=torch.Generator().manual_seed(1)).to(state).cuda()
        y = k.ssm_scan(conv.to(dtype).cuda(), torch.randn(T, nh, generator=torch.Generator().manual_seed(2)).to(dtype).cuda(), *consts, s,
                       dev(0, T), dev(3), dev(1), 1, nh, P, N, 1, 1.0, longest=longest).float().cpu()
        assert y[T - 1, 5] == float("inf") and y[T - 1, 40] == -float("inf")
        assert int((~y.isfinite()).sum()) == 2 and bool((s[1, 0, 5] == float("inf")).all())


@pytest.mark.parametrize("state", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,nh,P,N,G", [(1, 24, 64, 128, 1), (13, 6, 64, 256, 2), (3, 5, 40, 104, 5), (70, 4, 128, 64, 1)])
def test_ssm_step_against_64_bits(B, nh, P, N, G, state):
    from logssms_b200.ops import kernels as k
    g = torch.Generator().manual_seed(B * N + P)
    inner, C = nh * P, nh * P + 2 * G * N
    conv, dt = torch.randn(B, C, generator=g).to(torch.bfloat16), torch.randn(B, nh, generator=g).to(torch.bfloat16)
    A_log, dt_bias, D = torch.rand(nh, generator=g), torch.randn(nh, generator=g), torch.randn(nh, generator=g)
    gate = torch.randn(B, inner, generator=g).to(torch.bfloat16)
    before = torch.randn(B + 1, nh, P, N, generator=g).to(state)
    slots = torch.randperm(B + 1, generator=g)[:B]
    start = [0 if i % 4 == 3 else 2 for i in range(B)]
    got = before.clone().cuda()
    y = k.ssm_scan(conv.cuda(), dt.cuda(), A_log.cuda(), dt_bias.cuda(), D.cuda(), got, torch.arange(B + 1, dtype=torch.int32).cuda(),
                   torch.tensor(start, dtype=torch.int32).cuda(), slots.to(torch.int32).cuda(), B, nh, P, N, G, 0.8, gate.cuda(), 0.6,
                   longest=1).double().cpu()
    rnd = lambda t: t.float().to(torch.bfloat16).double()
    step = torch.nn.functional.softplus(rnd(dt.double() * 0.8) + dt_bias.double())                  # [B, nh]
    x = conv[:, :inner].double().view(B, nh, P)
    Bm, Cm = (conv[:, inner + i * G * N:inner + (i + 1) * G * N].double().view(B, G, N).repeat_interleave(nh // G, 1) for i in (0, 1))
    S = before[slots].double() * (torch.tensor(start) > 0).double()[:, None, None, None]
    rate = (torch.exp(A_log.double()) * step)[..., None, None]                                      # the decay is exp(-rate)
    kept, new = S * torch.exp(-rate), (x * step[..., None])[..., None] * Bm[:, :, None]
    S = kept + new
    out = (S * Cm[:, :, None]).sum(-1) + D.double()[:, None] * x
    want = rnd(rnd(out.reshape(B, inner)) * rnd(torch.nn.functional.silu(rnd(gate.double() * 0.6))))
    # y: a rounding to bfloat16 on the other side of a boundary at each of the last three places, 2^-8 of the value each; the state:
    # a dozen 32-bit roundings and exponentials of two units on the way to each of its two terms (2^-20), the decay's argument
    # among them, whose error counts times its size; a bfloat16 state is rounded once
    assert bool(((y - want).abs() <= 3 * 2.0 ** -8 * torch.maximum(want.abs(), want.abs().mean())).all())
    bound = 2.0 ** -20 * (kept.abs() * (1 + rate) + new.abs()) + (2.0 ** -8 * S.abs() if state == torch.bfloat16 else 0)
    assert bool(((got.cpu()[slots].double() - S).abs() <= bound).all())
    spare = sorted(set(range(B + 1)) - set(slots.tolist()))
    assert torch.equal(got.cpu()[spare], before[spare])
