"""Decode attention whose key ranges are the CTAs of one cluster of up to 16: every number of ranges, used and idle ones."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hq,Hkv,hd", [(8, 2, 64), (6, 2, 128), (12, 2, 128), (4, 1, 32)])
@pytest.mark.parametrize("splits", [2, 8, 9, 13, 16])
def test_ranges_of_a_cluster(Hq, Hkv, hd, splits):
    from logssms_b200.ops import kernels as k
    g = torch.Generator().manual_seed(splits + hd)
    contexts, page = [4200, 2049, 256, 1, 0], 64            # 16 ranges in use, some, one
    B, per = len(contexts), 4200 // page + 1
    kc = torch.randn(B * per, page, Hkv, hd, generator=g).to(torch.bfloat16).cuda()
    vc = torch.randn(B * per, page, Hkv, hd, generator=g).to(torch.bfloat16).cuda()
    bt = torch.randperm(B * per, generator=g).to(torch.int32).view(B, per)
    pos = torch.tensor(contexts, dtype=torch.int32)
    slot = (bt[torch.arange(B), (pos // page).long()] * page + pos % page).to(torch.int32)
    qkv = torch.randn(B, (Hq + 2 * Hkv) * hd, generator=g).to(torch.bfloat16).cuda()
    inv = 1.0 / (1e4 ** (torch.arange(0, hd, 2, dtype=torch.float32) / hd))
    table = k.rope_table(inv.cuda(), 8192)

    def step(v_cache, qkv, n):
        return k.attention_decode_step(qkv, Hq, Hkv, hd, pos.cuda(), slot.cuda(), table, kc.clone(), v_cache.clone(), bt.cuda(),
                                       torch.arange(B, dtype=torch.int32).cuda(), hd ** -0.5, 1.0, splits=n).float()

    one, several = step(vc, qkv, 1), step(vc, qkv, splits)
    # A softmax weight is rounded to bfloat16 relative to its range's maximum: 2^-9 of it either way, so the two results differ
    # by at most 2^-8 of the sum of |weight * value| (the same attention over |v|), and each is rounded once, 2^-8 of itself.
    sizes = qkv.clone()
    sizes[:, (Hq + Hkv) * hd:] = sizes[:, (Hq + Hkv) * hd:].abs()
    bound = 2.0 ** -8 * (1.01 * step(vc.abs(), sizes, 1) + 2 * one.abs())
    assert bool(((several - one).abs() <= bound).all())
    # those roundings have no common sign: a range merged with the wrong factor would show at once
    assert float((several - one).norm() / one.norm()) <= 2.0 ** -6
    k.check_kernel_errors()


def test_how_many_ranges():
    from logssms_b200.ops import kernels as k
    assert k.decode_step_splits(1, 8, 2, 8192) == 16 and k.decode_step_splits(1, 8, 2, 40960) > 16
    assert k.decode_step_splits(8, 8, 2, 8192) == 8
    assert k.decode_step_splits(24, 12, 2, 8192, head_dim=128) == 6 and k.decode_step_splits(48, 12, 2, 8192, head_dim=128) == 1


@pytest.mark.parametrize("Hq,Hkv,hd,page", [(8, 2, 64, 64), (12, 2, 128, 64), (6, 2, 112, 64), (4, 1, 32, 16)])
def test_a_gpu_that_holds_no_cluster_of_so_many_ranges(Hq, Hkv, hd, page):
    """... merges them through global memory: what a launch that is not given a cluster does, for 2 to 16 ranges.  And the question
    whether it holds one is asked per size of the CTAs: a larger head after a smaller one (shared memory grows with it)."""
    from logssms_b200.ops import kernels as k
    g = torch.Generator().manual_seed(hd)
    contexts = [4200, 2049, 256, 1, 0]
    B, per = len(contexts), 4200 // page + 1
    pos = torch.tensor(contexts, dtype=torch.int32)
    for dim in (16 * (hd // 16 - 1) if hd > 64 else hd, hd):
        kc, vc = (torch.randn(B * per, page, Hkv, dim, generator=g).to(torch.bfloat16).cuda() for _ in range(2))
        bt = torch.randperm(B * per, generator=g).to(torch.int32).view(B, per)
        slot = (bt[torch.arange(B), (pos // page).long()] * page + pos % page).to(torch.int32)
        qkv = torch.randn(B, (Hq + 2 * Hkv) * dim, generator=g).to(torch.bfloat16).cuda()
        table = k.rope_table((1.0 / (1e4 ** (torch.arange(0, dim, 2, dtype=torch.float32) / dim))).cuda(), 8192)
        args = lambda: (qkv, Hq, Hkv, dim, pos.cuda(), slot.cuda(), table, kc.clone(), vc.clone(), bt.cuda(),
                        torch.arange(B, dtype=torch.int32).cuda(), dim ** -0.5, 1.0)
        for splits in (2, 9, 13, 16):
            clustered = k.attention_decode_step(*args(), splits=splits).float()
            for most in (0, 8):
                plain = k.attention_decode_step(*args(), splits=splits, cluster_ranges=most).float()
                # the same partial results, merged in 32-bit in another order, rounded once to bfloat16
                assert bool(((plain - clustered).abs() <= 2.0 ** -7 * torch.maximum(clustered.abs(), clustered.abs().mean())).all())
    k.check_kernel_errors()
