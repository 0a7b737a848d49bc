"""The few-row product on the tensor cores (`linear_rows_tc.cu`): up to 64 rows, every epilogue, at the edges of its tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def K():
    from logssms_b200.ops import kernels
    return kernels


def rnd(t):
    return t.to(torch.bfloat16).float()


def close(got, want, ulps):
    """Both are rounded to bfloat16 (8 bits) after 32-bit sums: where the two sums lie on either side of a rounding
    boundary they differ by one unit of the last place, 2^-7 of the value at most, once per rounding on the way."""
    bound = ulps * 2.0 ** -7 * torch.maximum(want.abs(), want.abs().mean())
    assert bool(((got.float() - want).abs() <= bound).all())


# rows: edges of the padded sizes 16 / 32 / 48 / 64; features: one short tile, a remainder, whole tiles; k: the smallest, no
# multiple of a block, so many blocks that the ring goes round, a split over 2, 4 and 8 CTAs
@pytest.mark.parametrize("M", [9, 16, 17, 32, 33, 48, 49, 64])
@pytest.mark.parametrize("N,Kd", [(40, 256), (200, 1000), (1030, 1032), (128, 4096), (3352, 320), (20000, 264)])
def test_every_epilogue(M, N, Kd):
    g = torch.Generator().manual_seed(M * 7 + N)
    k = K()
    x = torch.randn(M, Kd + 8, generator=g).to(torch.bfloat16).cuda()[:, :Kd]            # a row-strided view
    w = (torch.randn(N, Kd, generator=g) * 0.05).to(torch.bfloat16).cuda()
    b = torch.randn(N, generator=g).to(torch.bfloat16).cuda()
    acc = (x.double() @ w.double().T).float()
    close(k._rows_tc(x, w, None, k._PLAIN), rnd(acc), 1)
    close(k._rows_tc(x, w, b, k._PLAIN, 0.7), rnd(rnd(acc + b.float()) * 0.7), 2)
    out = k._rows_tc(x, w, None, k._OUT_F32, 0.25)
    assert out.dtype == torch.float32
    close(out, rnd(acc) * 0.25, 1)
    I = N // 2
    gate, up = rnd(rnd(acc[:, :I]) * 0.9), rnd(acc[:, I:2 * I])
    got = k._rows_tc(x, w, None, k._SWIGLU, act_scale=0.9)
    # the gate's two roundings go through silu, whose slope relative to its value is at most about 1 + |gate|
    want = rnd(rnd(torch.nn.functional.silu(gate)) * up)
    bound = 2.0 ** -7 * ((4 + 2 * gate.abs()) * want.abs() + 4 * want.abs().mean())
    assert bool(((got.float() - want).abs() <= bound).all())
    k.check_kernel_errors()


def test_which_products_go_there():
    k = K()
    w = torch.zeros(1280, 3072, dtype=torch.bfloat16, device="cuda")
    rows = lambda n: torch.zeros(n, 3072, dtype=torch.bfloat16, device="cuda")
    assert [k._rows_tc_ok(rows(n), w, None) for n in (8, 9, 32, 33)] == [False, True, True, False]
    assert k._rows_tc_ok(rows(64), w, None, k.ROWS_TC_MAX_F32) and not k._rows_tc_ok(rows(65), w, None, k.ROWS_TC_MAX_F32)
    few = torch.zeros(1024, 1024, dtype=torch.bfloat16, device="cuda")
    assert not k._rows_tc_ok(rows(16)[:, :1024].contiguous(), few, None)
    for n in (9, 32, 64):                                  # and the dispatcher reaches the same kernel
        x = torch.randn(n, 3072, device="cuda").to(torch.bfloat16)
        wn = torch.randn(1280, 3072, device="cuda").to(torch.bfloat16)
        assert torch.equal(k.linear(x, wn, out_scale=0.5, out_f32=True), k._rows_tc(x, wn, None, k._OUT_F32, 0.5))
        if n <= 32:
            assert torch.equal(k.linear_swiglu(x, wn, 0.9), k._rows_tc(x, wn, None, k._SWIGLU, act_scale=0.9))


# the windows come preloaded for up to four taps and sixteen rows per CTA of the cluster; 64 rows in one CTA read them late
@pytest.mark.parametrize("M", [9, 32, 64])
@pytest.mark.parametrize("taps", [2, 4, 6])
@pytest.mark.parametrize("N,first,C", [(300, 100, 130), (3352, 1536, 1792), (40000, 500, 300)])
def test_the_conv_step(M, taps, N, first, C):
    g = torch.Generator().manual_seed(M * 5 + taps)
    k = K()
    Kd = 1032
    x = torch.randn(M, Kd, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(N, Kd, generator=g) * 0.05).to(torch.bfloat16).cuda()
    cw, cb = (torch.randn(C, taps, generator=g) * 0.4).cuda(), (torch.randn(C, generator=g) * 0.1).cuda()
    slots = torch.randperm(M + 3, generator=g)[:M].to(torch.int32).cuda()
    start = torch.tensor([0 if i % 3 == 0 else 5 + i for i in range(M)], dtype=torch.int32).cuda()   # some requests are new
    before = torch.randn(M + 3, C, taps - 1, generator=g).to(torch.bfloat16).cuda()
    ends, scales = (C // 3, C // 2), (1.1, 0.9, 1.3)
    state = before.clone()
    got = k._rows_tc(x, w, None, k._CONV, conv=(cw.data_ptr(), cb.data_ptr(), state.data_ptr(), slots.data_ptr(), start.data_ptr(),
                                                first, first + C, taps, *ends, *scales))
    proj = k._rows_tc(x, w, None, k._PLAIN)
    want_state = before.clone()
    conv = k.causal_conv1d(proj[:, first:first + C], cw, cb, want_state, torch.arange(M + 1, dtype=torch.int32).cuda(), start,
                           slots, M, 1, ends, scales)
    assert torch.equal(got[:, :first], proj[:, :first]) and torch.equal(got[:, first + C:], proj[:, first + C:])
    assert torch.equal(state, want_state)
    close(got[:, first:first + C], conv.float(), 2)
    if M <= 32:                                            # and by the dispatcher
        again = before.clone()
        via = k.linear_conv_step(x, w, None, cw, cb, again, slots, start, first, first + C, ends, scales)
        assert torch.equal(via, got) and torch.equal(again, state)
    k.check_kernel_errors()


@pytest.mark.parametrize("M", [9, 32, 33, 64])
@pytest.mark.parametrize("N,Kd", [(40, 256), (1030, 1032), (3352, 320)])
def test_a_bias_under_every_epilogue_that_takes_one(M, N, Kd):
    """Projections with a bias: float32 output, and the conv step, whose window holds the projection with its bias."""
    g = torch.Generator().manual_seed(M * 11 + N)
    k = K()
    x = torch.randn(M, Kd, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(N, Kd, generator=g) * 0.05).to(torch.bfloat16).cuda()
    b = torch.randn(N, generator=g).to(torch.bfloat16).cuda()
    acc = (x.double() @ w.double().T).float()
    out = k._rows_tc(x, w, b, k._OUT_F32, 0.25)
    assert out.dtype == torch.float32
    close(out, rnd(acc + b.float()) * 0.25, 1)
    first, C, taps = N // 4, N // 2, 4
    cw, cb = (torch.randn(C, taps, generator=g) * 0.4).cuda(), (torch.randn(C, generator=g) * 0.1).cuda()
    slots = torch.randperm(M + 3, generator=g)[:M].to(torch.int32).cuda()
    start = torch.tensor([0 if i % 3 == 0 else 5 + i for i in range(M)], dtype=torch.int32).cuda()
    before = torch.randn(M + 3, C, taps - 1, generator=g).to(torch.bfloat16).cuda()
    ends, scales = (C // 3, C // 2), (1.1, 0.9, 1.3)
    state, want_state = before.clone(), before.clone()
    got = k._rows_tc(x, w, b, k._CONV, conv=(cw.data_ptr(), cb.data_ptr(), state.data_ptr(), slots.data_ptr(), start.data_ptr(),
                                             first, first + C, taps, *ends, *scales))
    proj = k._rows_tc(x, w, b, k._PLAIN)
    conv = k.causal_conv1d(proj[:, first:first + C], cw, cb, want_state, torch.arange(M + 1, dtype=torch.int32).cuda(), start,
                           slots, M, 1, ends, scales)
    assert torch.equal(got[:, :first], proj[:, :first]) and torch.equal(got[:, first + C:], proj[:, first + C:])
    assert torch.equal(state, want_state)
    close(got[:, first:first + C], conv.float(), 2)
    k.check_kernel_errors()
