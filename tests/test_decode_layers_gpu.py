"""The kernel that runs all layers of a decode step (`kernels.decode_layers`): against the plain model at the edges of its tiles
(keys in tiles of 16 and pages of 64, up to 8 and up to 16 rows, a request's first token, requests that share a CTA's keys or not), and against
the chain of kernels over contexts that many CTAs share."""
import math

import pytest
import torch

from tiny import TINY_D, TOL, make_model_dir, plain_logits, rel_err

# the smallest sizes it takes, and one with heads of 128, three query heads to a key/value head, two groups, three taps, no bias
SMALL = {**TINY_D, "hidden_size": 256, "num_attention_heads": 4, "num_key_value_heads": 2, "head_dim": 64, "intermediate_size": 512,
         "mamba_d_ssm": 256, "mamba_n_heads": 4, "mamba_d_head": 64, "mamba_d_state": 128, "mamba_proj_bias": False,
         "projectors_bias": False, "max_position_embeddings": 8192}
WIDE = {**SMALL, "num_hidden_layers": 3, "hidden_size": 512, "num_attention_heads": 6, "num_key_value_heads": 2, "head_dim": 128,
        "intermediate_size": 768, "mamba_d_ssm": 1792, "mamba_n_heads": 14, "mamba_d_head": 128, "mamba_d_state": 256,
        "mamba_n_groups": 2, "mamba_d_conv": 3, "mamba_conv_bias": False, "tie_word_embeddings": True}
CONFIGS = {"small": SMALL, "wide": WIDE}


def decode(engine, prompts, contexts, steps):
    """Logits [steps][rows, vocab] of decode steps behind contexts of the given lengths (0: the first token of all)."""
    from logssms_b200.engine import StepEntry
    live = [engine.new_request() for _ in contexts]
    begun = [(r, ids[:n]) for r, ids, n in zip(live, prompts, contexts) if n > 0]
    if begun:
        engine.step([StepEntry(r, ids) for r, ids in begun])
    out = []
    for i in range(steps):
        logits = engine.step([StepEntry(r, [ids[n + i]], [0]) for r, ids, n in zip(live, prompts, contexts)])
        out.append(logits.float().cpu().clone())
    for r in live:
        engine.release(r)
    return out


@pytest.fixture
def calls(monkeypatch):
    from logssms_b200.ops import kernels as K
    count, inner = [0], K.decode_layers

    def counted(*args):
        count[0] += 1
        return inner(*args)
    monkeypatch.setattr(K, "decode_layers", counted)
    return count


@pytest.mark.gpu
@pytest.mark.parametrize("config,state,contexts", [
    ("small", "float32", [0]), ("small", "float32", [15, 16, 17]), ("small", "activation", [63, 64, 65, 0, 127]),
    ("small", "float32", [1, 200, 31, 0, 129, 78, 47, 3]), ("wide", "float32", [14, 0]), ("wide", "activation", [31, 32, 33]),
    ("wide", "float32", [0, 1, 2, 260, 15, 64, 111, 95]), ("small", "activation", [7, 0, 30, 100, 64, 1, 16, 250, 47]),
    ("wide", "float32", [3, 77, 15, 0, 128, 200, 31, 5, 64, 17, 90, 33, 1, 140, 48, 63])])
def test_decode_steps_in_one_kernel_equal_the_plain_model(tmp_path, calls, config, state, contexts):
    from logssms_b200.engine import Engine
    from logssms_b200.ops import kernels as K
    raw, steps = CONFIGS[config], 3
    model_dir = make_model_dir(tmp_path / "m", raw, seed=17, dtype=torch.bfloat16)
    g = torch.Generator().manual_seed(len(contexts))
    prompts = [torch.randint(0, raw["vocab_size"], (n + steps,), generator=g).tolist() for n in contexts]
    engine = Engine(model_dir, "bfloat16", max_requests=16, max_seq_len=512, num_pages=80, ssm_state_dtype=state, poison_on_free=True)
    got = decode(engine, prompts, contexts, steps)             # the first step kernel by kernel, then captured, then replayed
    assert calls[0] >= 2
    K.check_kernel_errors()
    for b, (ids, n) in enumerate(zip(prompts, contexts)):
        want = plain_logits(model_dir, ids, "bfloat16")
        for i in range(steps):
            assert rel_err(got[i][b], want[n + i]) < TOL["bfloat16"], (b, i)


@pytest.mark.gpu
def test_layers_of_several_launches_and_fewer_requests_than_the_graph(tmp_path, calls, monkeypatch):
    """Three layers as launches of two and one; then six requests through the graph of eight."""
    from logssms_b200.engine import Engine
    from logssms_b200.ops import kernels as K
    monkeypatch.setattr(K, "_DECODE_LAYERS_MOST", 2)
    model_dir = make_model_dir(tmp_path / "m", WIDE, seed=18, dtype=torch.bfloat16)
    g = torch.Generator().manual_seed(5)
    contexts = [40, 3, 66, 129, 18, 300]
    prompts = [torch.randint(0, WIDE["vocab_size"], (n + 2,), generator=g).tolist() for n in contexts]
    engine = Engine(model_dir, "bfloat16", max_requests=8, max_seq_len=512, num_pages=40)
    assert engine.capture_decode_graphs([8]) == [8] and calls[0] == 2
    got = decode(engine, prompts, contexts, 2)
    assert calls[0] == 2                                        # replayed, filled up with dummy requests
    K.check_kernel_errors()
    for b, (ids, n) in enumerate(zip(prompts, contexts)):
        want = plain_logits(model_dir, ids, "bfloat16")
        for i in range(2):
            assert rel_err(got[i][b], want[n + i]) < TOL["bfloat16"], (b, i)


@pytest.mark.gpu
@pytest.mark.parametrize("config,contexts", [("small", [4000]), ("small", [5, 4090, 700]), ("wide", [2500]), ("wide", [1030, 9, 1500, 64, 1, 900, 333, 2000])])
def test_contexts_that_many_ctas_share_equal_the_chain_of_kernels(tmp_path, calls, monkeypatch, config, contexts):
    """Both paths round where the plain model does, in another order of summation: their difference stays within the tolerance
    that each has against the plain model."""
    from logssms_b200.engine import Engine
    from logssms_b200.ops import kernels as K
    raw = CONFIGS[config]
    model_dir = make_model_dir(tmp_path / "m", raw, seed=19, dtype=torch.bfloat16)
    g = torch.Generator().manual_seed(6)
    prompts = [torch.randint(0, raw["vocab_size"], (n + 2,), generator=g).tolist() for n in contexts]
    results = []
    for fused in (True, False):
        if not fused:
            monkeypatch.setattr(K, "decode_layers_ok", lambda *a: False)
        before = calls[0]
        engine = Engine(model_dir, "bfloat16", max_requests=8, max_seq_len=4160, num_pages=200, use_graphs=False)
        results.append(decode(engine, prompts, contexts, 2))
        assert (calls[0] > before) == fused
    K.check_kernel_errors()
    for a, b in zip(*results):
        assert rel_err(a, b) < TOL["bfloat16"]


@pytest.mark.gpu
@pytest.mark.parametrize("config,state,contexts", [("small", "float32", [0, 17, 64, 130]), ("small", "activation", [63, 0, 300]),
                                                   ("wide", "float32", [14, 0, 200]), ("wide", "activation", [5, 0, 31, 64, 17, 90, 33, 1, 140])])
def test_caches_behind_decode_steps_equal_the_chain_of_kernels(tmp_path, calls, monkeypatch, config, state, contexts):
    """Stored keys and values, conv windows and recurrent states of every layer after four steps, the requests' own and nobody's."""
    from logssms_b200.engine import Engine, StepEntry
    from logssms_b200.ops import kernels as K
    raw, steps = CONFIGS[config], 4
    model_dir = make_model_dir(tmp_path / "m", raw, seed=23, dtype=torch.bfloat16)
    g = torch.Generator().manual_seed(9)
    prompts = [torch.randint(0, raw["vocab_size"], (n + steps,), generator=g).tolist() for n in contexts]
    kept = []
    for fused in (True, False):
        if not fused:
            monkeypatch.setattr(K, "decode_layers_ok", lambda *a: False)
        before = calls[0]
        engine = Engine(model_dir, "bfloat16", max_requests=16, max_seq_len=512, num_pages=80, ssm_state_dtype=state)
        cache, live = engine.cache, [engine.new_request() for _ in contexts]
        engine.step([StepEntry(r, ids[:n]) for r, ids, n in zip(live, prompts, contexts) if n > 0])
        idle = [r for r in range(16) if r not in [q.row for q in live]]
        nobodys = [[cache.states[i][k][idle].clone() for k in ("conv", "ssm")] for i in range(raw["num_hidden_layers"])]
        for i in range(steps):
            engine.step([StepEntry(r, [ids[n + i]], [0]) for r, ids, n in zip(live, prompts, contexts)])
        assert (calls[0] > before) == fused
        K.check_kernel_errors()
        layers = []
        for i in range(raw["num_hidden_layers"]):
            k, v, group = cache.kv(i)
            states = cache.states[i]
            for a, b in zip(nobodys[i], (states["conv"][idle], states["ssm"][idle])):
                assert torch.equal(a, b)
            for r, n in zip(live, contexts):
                pages = torch.as_tensor(cache.groups[group].block_table[r.row][:-(-(n + steps) // 64)]).long().cuda()
                for name, t in (("keys", k[pages].flatten(0, 1)[:n + steps]), ("values", v[pages].flatten(0, 1)[:n + steps]),
                                ("conv", states["conv"][r.row]), ("states", states["ssm"][r.row])):
                    layers.append((i, n, name, t.float().cpu()))
        kept.append(layers)
    for (i, n, name, a), (_, _, _, b) in zip(*kept):
        # both round where the plain model does, in another order of summation
        assert a.shape == b.shape and rel_err(a, b) < TOL["bfloat16"], (i, n, name, rel_err(a, b))


def one_layer(dev="cuda", **changed):
    """A layer of the smallest sizes as the kernel takes it, all products zero and norms one except what `changed` names; its tensors
    and the step's, for one row that is its request's first token."""
    from logssms_b200.ops import kernels as K
    bf = lambda *shape: torch.zeros(shape, dtype=torch.bfloat16)
    t = dict(qkv=bf(512, 256), in_w=bf(256 + 512 + 4, 256), o=bf(256, 256), out=bf(256, 256), gate_up=bf(512, 256), down=bf(256, 256),
             conv_w=torch.zeros(512, 4), conv_b=None, a_log=torch.zeros(4), dt_bias=torch.zeros(4), d=torch.ones(4), ff_norm=torch.ones(256),
             norm=torch.ones(256), conv=bf(2, 512, 3), k=bf(2, 64, 2, 64), v=bf(2, 64, 2, 64), ssm=torch.zeros(2, 4, 64, 128),
             table=torch.tensor([[1]], dtype=torch.int32), at=torch.tensor([64], dtype=torch.int32))
    t.update(changed)
    t = {k: None if v is None else v.to(dev) for k, v in t.items()}
    z = K.StepSizes(hidden=256, heads=4, kv_heads=2, head_dim=64, rotary_dim=64, page_size=64, key_scale=1.0, softmax_scale=0.125,
                    ssm_heads=4, ssm_head_dim=64, state_dim=128, groups=1, taps=4, state_bf16=False, multipliers=(1.0,) * 5,
                    intermediate=256, act_scale=1.0, ff_scale=1.0, attn_in=1.0, attn_out=1.0, ssm_in=1.0, ssm_out=1.0, mixer_eps=0.0,
                    ff_eps=0.0)
    return K.StepLayer(z, tuple(t.values()), 2, torch.ones(64, 64, device=dev)), t


@pytest.mark.gpu
@pytest.mark.parametrize("place", ["gate of the feed-forward", "gate of the mixer", "conv"])
def test_silu_far_below_zero(place):
    """SiLU of -87.5 is -8.8e-37, an ordinary bfloat16; a division whose divisor lies past 2^126 must not lose it."""
    from logssms_b200.ops import kernels as K
    eye = torch.eye(256).bfloat16()
    far, one, lift = torch.full((256, 256), -87.5 / 256).bfloat16(), torch.full((256, 256), 1 / 256).bfloat16(), (2.0 ** 120 * torch.eye(256)).bfloat16()
    silu = -87.5 / (1.0 + math.exp(87.5))
    if place == "gate of the feed-forward":                # h = silu(-87.5) * 1
        layer, t = one_layer(gate_up=torch.cat([far, one]), down=lift)
        want = silu
    else:                                                  # y = D x silu(z): a first token's state is its own, and B and C are zero
        in_w = torch.zeros(256 + 512 + 4, 256).bfloat16()
        in_w[:256], in_w[256:512] = (far, 30 * one) if place == "gate of the mixer" else (30 * one, far)
        taps = torch.zeros(512, 4)
        taps[:, 3] = 1.0
        layer, t = one_layer(in_w=in_w, conv_w=taps, out=lift)
        want = silu * 30.0 / (1.0 + math.exp(-30.0))
    x = torch.ones(1, 256, dtype=torch.bfloat16, device="cuda")
    zero = torch.zeros(1, dtype=torch.int32, device="cuda")
    out, res = K.decode_layers(x, t["norm"], [layer], zero, zero, zero)
    got = (out if place == "gate of the feed-forward" else res).float().cpu()
    K.check_kernel_errors()
    want = want * 2.0 ** 120 + (0.0 if place == "gate of the feed-forward" else 1.0)
    assert float((got - want).abs().max()) <= 2.0 ** -6 * abs(want), (got[0, :4], want)     # up to four roundings to bfloat16


@pytest.mark.gpu
def test_a_profile_times_the_kernel_that_the_steps_run(tmp_path, calls):
    from logssms_b200.engine import LLM
    from logssms_b200.sampling import SamplingParams
    model_dir = make_model_dir(tmp_path / "m", SMALL, seed=22, dtype=torch.bfloat16)
    prompts, sp = [list(range(3, 90)), [7, 8, 9]], SamplingParams(temperature=0.0, max_tokens=5, ignore_eos=True)
    want = [o.token_ids for o in LLM(model_dir, "bfloat16", max_running_requests=2, max_seq_len_override=256, num_pages=8).generate(prompts, sp)]
    before = calls[0]
    llm = LLM(model_dir, "bfloat16", max_running_requests=2, max_seq_len_override=256, num_pages=8, profile=True, nvtx=True)
    try:
        assert [o.token_ids for o in llm.generate(prompts, sp)] == want
        report = llm.engine.profile_report()
    finally:
        LLM(model_dir, "bfloat16", max_running_requests=2, max_seq_len_override=256, num_pages=8)      # switches the profiler off again
    steps = calls[0] - before
    assert steps >= 4 and report["kernels"]["decode_layers.lb_decode_layers"]["launches"] == steps
    assert report["classes"]["layers in one kernel"]["launches"] == steps and report["classes"]["layers in one kernel"]["ms"] > 0


# 145 tiles of 8 features in the first product: of 148 CTAs three have none, and with these contexts two of those attend
NARROW = {**SMALL, "num_hidden_layers": 3, "num_key_value_heads": 1, "max_position_embeddings": 32768}


@pytest.mark.gpu
@pytest.mark.parametrize("most", [1, 2, 64])
def test_ctas_without_tiles_of_the_first_product_in_launches_behind_the_first(tmp_path, calls, monkeypatch, most):
    from logssms_b200.engine import Engine
    from logssms_b200.ops import kernels as K
    model_dir = make_model_dir(tmp_path / "m", NARROW, seed=21, dtype=torch.bfloat16)
    g = torch.Generator().manual_seed(8)
    contexts = [18400, 300]
    prompts = [torch.randint(0, NARROW["vocab_size"], (n + 2,), generator=g).tolist() for n in contexts]
    results = []
    for fused in (True, False):
        if fused:
            monkeypatch.setattr(K, "_DECODE_LAYERS_MOST", most)
        else:
            monkeypatch.setattr(K, "decode_layers_ok", lambda *a: False)
        before = calls[0]
        engine = Engine(model_dir, "bfloat16", max_requests=2, max_seq_len=18560, num_pages=300, use_graphs=False)
        results.append(decode(engine, prompts, contexts, 2))
        assert (calls[0] > before) == fused
    K.check_kernel_errors()
    for a, b in zip(*results):                              # as below: two paths that round where the plain model does
        assert rel_err(a, b) < TOL["bfloat16"]


@pytest.mark.gpu
@pytest.mark.parametrize("polls,roles", [((1 << 16, 0, -1), [0x34]), ((1 << 16, -1, 0), [0x33, 0x35]), ((0, -1, -1), [0x32])])
def test_a_wait_that_runs_out_ends_the_step_with_an_error(tmp_path, calls, monkeypatch, polls, roles):
    """Waits of one kind (keys, weights, the grid barrier) give up at once, with copies in flight: the kernel reports itself and
    ends, and the steps behind it are right.  (A CTA's weights, 70 KB a layer, do not all fit its ring.)"""
    from logssms_b200.engine import Engine, StepEntry
    from logssms_b200.ops import kernels as K
    model_dir = make_model_dir(tmp_path / "m", {**SMALL, "num_hidden_layers": 4, "intermediate_size": 8192}, seed=20, dtype=torch.bfloat16)
    g = torch.Generator().manual_seed(7)
    contexts = [300, 200]
    prompts = [torch.randint(0, SMALL["vocab_size"], (n + 2,), generator=g).tolist() for n in contexts]
    engine = Engine(model_dir, "bfloat16", max_requests=4, max_seq_len=512, num_pages=40, use_graphs=False)
    live = [engine.new_request() for _ in contexts]
    engine.step([StepEntry(r, ids[:n]) for r, ids, n in zip(live, prompts, contexts)])
    K.check_kernel_errors()
    with monkeypatch.context() as m:
        m.setattr(K, "_DECODE_LAYERS_POLLS", polls)
        engine.step([StepEntry(r, [ids[n]], [0]) for r, ids, n in zip(live, prompts, contexts)])
        with pytest.raises(K.KernelError, match="|".join(f"role {r}" for r in roles)):
            K.check_kernel_errors()
    for r in live:
        engine.release(r)
    got = decode(engine, prompts, contexts, 2)
    K.check_kernel_errors()
    assert calls[0] == 3
    for b, (ids, n) in enumerate(zip(prompts, contexts)):
        want = plain_logits(model_dir, ids, "bfloat16")
        for i in range(2):
            assert rel_err(got[i][b], want[n + i]) < TOL["bfloat16"], (b, i)


def test_which_steps_go_through_one_kernel():
    from logssms_b200.ops import kernels as K
    base = dict(hidden=1024, heads=8, kv_heads=2, head_dim=64, rotary_dim=64, page_size=64, key_scale=1.0, softmax_scale=0.125,
                ssm_heads=24, ssm_head_dim=64, state_dim=128, groups=1, taps=4, state_bf16=False, multipliers=(1.0,) * 5,
                intermediate=2048, act_scale=1.0, ff_scale=1.0, attn_in=1.0, attn_out=1.0, ssm_in=1.0, ssm_out=1.0,
                mixer_eps=1e-5, ff_eps=1e-5)
    ok = lambda rows=1, keys=2048, **change: K.decode_layers_ok(rows, K.StepSizes(**{**base, **change}), keys)
    assert ok() and ok(8) and ok(8, 8192) and ok(12, 8192) and ok(16) and not ok(16, 8192) and not ok(17) and not ok(0)
    assert ok(8, hidden=1280, intermediate=3072) and not ok(9, hidden=1280, intermediate=3072)
    for change in ({"hidden": 1000}, {"intermediate": 2080}, {"head_dim": 96}, {"rotary_dim": 32}, {"page_size": 48}, {"page_size": 8},
                   {"state_dim": 64}, {"heads": 18}, {"ssm_heads": 23}, {"taps": 1}, {"hidden": 3072, "intermediate": 12288}):
        assert not ok(**change), change


def test_steps_that_the_chain_of_kernels_does_faster_stay_with_it():
    from logssms_b200.ops import kernels as K
    base = dict(hidden=1024, heads=8, kv_heads=2, head_dim=64, rotary_dim=64, page_size=64, key_scale=1.0, softmax_scale=0.125,
                ssm_heads=24, ssm_head_dim=64, state_dim=128, groups=1, taps=4, state_bf16=False, multipliers=(1.0,) * 5,
                intermediate=2048, act_scale=1.0, ff_scale=1.0, attn_in=1.0, attn_out=1.0, ssm_in=1.0, ssm_out=1.0,
                mixer_eps=1e-5, ff_eps=1e-5)
    ok = lambda rows=1, keys=2048, **change: K.decode_layers_ok(rows, K.StepSizes(**{**base, **change}), keys)
    large = dict(head_dim=128, rotary_dim=128, state_dim=256)
    for rows in (1, 8):                                     # hidden sizes above 2,048, whatever the weights
        assert ok(rows, hidden=2048, intermediate=8192, **large) and not ok(rows, hidden=2304, intermediate=2048, **large)
        assert not ok(rows, hidden=2560, intermediate=6144, **large) and not ok(rows, hidden=3072, intermediate=2048, **large)
    assert ok(1, 98304) and not ok(1, 98305) and ok(8, 12288) and not ok(8, 12289)
    assert ok(8, 1024, kv_heads=4, head_dim=128, rotary_dim=128) and not ok(8, 1025, kv_heads=4, head_dim=128, rotary_dim=128)
    assert ok(2, 8192, kv_heads=8) and not ok(2, 8193, kv_heads=8) and ok(1, 16384, kv_heads=8) and not ok(1, 16385, kv_heads=8)
    assert ok(12, 8192) and ok(13, 3780) and not ok(13, 3781) and ok(16, 3072) and not ok(16, 3073) and not ok(16, 6000)
    assert ok(16, 512, head_dim=128, rotary_dim=128, heads=4) and not ok(16, 513, head_dim=128, rotary_dim=128, heads=4)
    assert ok(9, 910, head_dim=128, rotary_dim=128, heads=4) and not ok(9, 911, head_dim=128, rotary_dim=128, heads=4)
    assert not ok(9, 300, kv_heads=4) and not ok(9, 300, intermediate=2816) and ok(8, 300, intermediate=2816)


def test_every_row_and_key_value_head_has_an_sm():
    """On a part of a GPU with fewer SMs than rows times key/value heads some heads would get no CTA."""
    from logssms_b200.ops import kernels as K
    z = K.StepSizes(hidden=1024, heads=8, kv_heads=2, head_dim=64, rotary_dim=64, page_size=64, key_scale=1.0, softmax_scale=0.125,
                    ssm_heads=24, ssm_head_dim=64, state_dim=128, groups=1, taps=4, state_bf16=False, multipliers=(1.0,) * 5,
                    intermediate=2048, act_scale=1.0, ff_scale=1.0, attn_in=1.0, attn_out=1.0, ssm_in=1.0, ssm_out=1.0, mixer_eps=1e-5,
                    ff_eps=1e-5)
    for rows in (1, 8, 9, 16):
        assert K.decode_layers_ok(rows, z, 512, 2 * rows) and not K.decode_layers_ok(rows, z, 512, 2 * rows - 1)
