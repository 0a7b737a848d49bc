"""The rules that choose between kernels, on the CPU: what each form's measurements hold for is asked for there and nowhere else."""
import pytest
import torch

from logssms_b200.ops import kernels as K


@pytest.mark.parametrize("tokens,heads,kv,limit,dim", [(1, 8, 2, 8192, 64), (1, 8, 2, 300, 64), (2, 6, 2, 8192, 128), (4, 8, 2, 4096, 64), (1, 8, 2, 40960, 64)])
def test_key_ranges_of_a_form_without_clusters_are_not_held_to_a_clusters_size(tokens, heads, kv, limit, dim):
    """float32 engines merge through global memory at every count: as many ranges as fill the GPU (one float32 token, 8 heads over 2,
    8,100 keys: 38.5 us with 16 ranges, 28.9 with 32)."""
    items = tokens * kv * -(-(heads // kv) // 4)
    want = max(1, min((296 if dim > 64 else 160) // items, -(-limit // 256), 256))
    assert K.decode_step_splits(tokens, heads, kv, limit, head_dim=dim, tensor_cores=False) == want
    assert K.decode_step_splits(tokens, heads, kv, limit, head_dim=dim) == min(want, 16 if limit <= 16384 else 32)


def test_key_ranges_of_large_heads_and_wide_groups():
    assert K.decode_step_splits(1, 8, 2, 8192, head_dim=160) == 32          # heads past 128 have no tensor-core form
    assert K.decode_step_splits(1, 40, 2, 8192, head_dim=64) == 26          # neither have groups past 16: 6 items of 8 heads
    assert K.decode_step_splits(8, 8, 2, 8192, tensor_cores=False) == 8     # a dozen items and more: 8 in either form


@pytest.mark.parametrize("limit", [8192, 16384, 40960])
def test_key_ranges_do_not_fall_back_with_the_engines_limit(limit):
    """A captured step knows the engine's limit, not its requests' contexts: a longer limit must not cost the short ones a multiple."""
    assert K.decode_step_splits(1, 8, 2, limit) == (16 if limit <= 16384 else 32)
    assert K.decode_step_splits(1, 12, 2, limit, head_dim=128) == (16 if limit <= 16384 else 32)


@pytest.mark.parametrize("mode,rows,taken", [("auto", 32, "rows"), ("auto", 64, "rows"), ("auto", 65, "library"), ("library", 32, "rows"),
                                             ("library", 33, "library"), ("library", 64, "library"), ("tcgen05", 32, "rows"),
                                             ("tcgen05", 33, "tcgen05"), ("tcgen05", 64, "tcgen05")])
def test_the_kernel_family_asked_for_takes_the_products_past_32_rows(monkeypatch, mode, rows, taken):
    """... those with float32 output (the output head), too."""
    called = []
    result = torch.zeros(rows, 8)
    for name, family in (("_rows_tc", "rows"), ("gemm_tcgen05", "tcgen05"), ("linear_skinny", "streamer"), ("scale", "library")):
        monkeypatch.setattr(K, name, lambda *a, family=family, **kw: (called.append(family), result)[1])
    monkeypatch.setattr(K, "_cuda", lambda *a: None)
    monkeypatch.setattr(K, "GEMM_MODE", mode)
    x, w = torch.zeros(rows, 2048, dtype=torch.bfloat16), torch.zeros(64, 2048, dtype=torch.bfloat16)
    assert K.linear(x, w, out_scale=0.5, out_f32=True) is result and called == [taken]
