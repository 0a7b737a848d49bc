"""Zarisun through the engine: trace replay of tiny random models against the plain implementation in every way of
cutting the same requests, and greedy generation through `LLM.generate`, the scheduler and the command line.

One bin/trace_run process per (configuration, dtype) replays all scenarios through one small page pool with four
request rows, so pages and state slots are used again (freed memory is NaN).  The attentions' queries are scaled up, so
single keys carry the output: one that is missing or surplus at a page border, at a window's edge or far back, or a sink
that is left out, moves the logits far beyond the tolerance."""
import random
import subprocess
import sys

import pytest
import torch

from replay_util import PAGE, Trace, in_portions, mixed, run_trace, tail_decoded, whole
from tiny_zarisun import TOL, ZARI, float32_floor, make_zarisun_dir, plain_logits, row_errors

pytestmark = pytest.mark.gpu

LENGTHS = {"r0": 150, "r1": 97, "r2": 130, "r3": 70, "r4": 3, "r5": 65}
MAX_TOKENS = 8 * PAGE
SCENARIOS = ("whole", "tail", "portions", "mixed", "long_decode", "first_tokens")
_cache: dict = {}


def model_for(tmp, name, dtype, sharp=None):
    # the float32 runs are the sharp ones (sharp scores multiply bfloat16's rounding of the scores themselves)
    return make_zarisun_dir(tmp / "model", ZARI[name], seed=11 + len(name), dtype=torch.float32 if dtype == "float32" else torch.bfloat16,
                            sharp=sharp if sharp is not None else 4.0 if dtype == "float32" else 1.5)


def replayed(tmp_path_factory, name, dtype):
    key = (name, dtype)
    if key in _cache:
        return _cache[key]
    raw = ZARI[name]
    tmp = tmp_path_factory.mktemp(f"zarisun_{name}_{dtype}")
    model_dir = model_for(tmp, name, dtype)
    rng = random.Random(7)
    seqs = {rid: [rng.randrange(raw["vocab"]) for _ in range(n)] for rid, n in LENGTHS.items()}
    want = {rid: plain_logits(model_dir, ids) for rid, ids in seqs.items()}
    # what rounding alone does: the plain implementation with everything in the engine's dtype against itself in float64
    # (in bfloat16 it rounds everything, its recurrences and norms too: only the mean over a request is used; in float32 the
    # worst of several orders of its sums is taken per position, since every position of the engine is held to it)
    floor = {rid: float32_floor(model_dir, ids, want[rid]) if dtype == "float32" else
             row_errors(plain_logits(model_dir, ids, torch.bfloat16), want[rid]) for rid, ids in seqs.items()}
    trace = Trace()
    ids_of: dict[str, str] = {}

    def uid(scn, rid):
        u = f"{scn}:{rid}"
        ids_of[u] = rid
        return u
    for rid, ids in seqs.items():
        whole(trace, uid("whole", rid), ids)
    for rid in ("r0", "r1", "r5"):
        tail_decoded(trace, uid("tail", rid), seqs[rid])
    in_portions(trace, uid("portions", "r0"), seqs["r0"], [7, 2, 16, 3, 33, 2, 64, 5])
    in_portions(trace, uid("portions", "r2"), seqs["r2"], [2, 62, 2, 3, 61])
    in_portions(trace, uid("portions", "r5"), seqs["r5"], [63, 2])
    mixed(trace, {uid("mixed", rid): seqs[rid] for rid in ("r1", "r3", "r4", "r5", "r0", "r2")}, MAX_TOKENS, seed=3)
    mixed(trace, {uid("mixed2", rid): seqs[rid] for rid in ("r3", "r4", "r5", "r1", "r2", "r0")}, MAX_TOKENS, seed=4,
          prompt_fraction=0.3)
    long_ids = seqs["r0"]
    trace.add_step([(uid("long_decode", "r0"), long_ids[:5])])
    for i in range(5, len(long_ids)):
        trace.add_step([(uid("long_decode", "r0"), long_ids[i:i + 1])],
                       end=[uid("long_decode", "r0")] if i == len(long_ids) - 1 else [])
    for n in (1, 2, 3):
        whole(trace, uid(f"first_tokens{n}", "r1"), seqs["r1"][:n])
    assert trace.peak_tokens <= MAX_TOKENS, trace.peak_tokens
    got = run_trace(model_dir, dtype, trace, str(tmp / "out"), MAX_TOKENS, raw["vocab"],
                    extra_args=["--poison", "--max-requests", "4"])
    _cache[key] = (got, want, ids_of, floor)
    return _cache[key]


@pytest.mark.parametrize("scenario", SCENARIOS)
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", ["A", "B", "C", "D", "E", "R1", "R2", "R3", "R5", "R8"])
def test_replay_matches_plain(tmp_path_factory, name, dtype, scenario):
    if name == "C" and dtype == "bfloat16":
        # heads of one value channel: their norm is x / sqrt(x^2 + eps), the sign of x unless x is tiny, and bfloat16 inputs
        # turn that sign where float64 inputs do not; the float32 run covers the sizes of 1
        pytest.skip("a norm over one channel is a sign: no tolerance on bfloat16 inputs holds")
    got, want, ids_of, floor = replayed(tmp_path_factory, name, dtype)
    checked = 0
    for u, rid in ids_of.items():
        if not u.split(":")[0].startswith(scenario):
            continue
        g = got[u]
        assert not torch.isnan(g).any(), f"{u}: positions without logits"
        err = row_errors(g, want[rid][:g.shape[0]])
        # float32: no position may differ by more than 3e-4, or three times what rounding does to the plain model there (the
        # worst of eight orders of summation: 6e-5 to 9e-4 at position 0 of r5 of R1, where a query and a key are orthogonal to
        # 7e-6, from where it reaches fourteen later positions; else 3e-4 stands but for seventeen positions of A, C and E,
        # whose bound is 8e-4 at most).
        # bfloat16 against a float64 oracle: the tolerance is 5e-2 or three times the mean rounding error of the plain model
        # in bfloat16 over the request; a few positions (three, or one in ten) may exceed it by any amount: single positions
        # of a tiny random model are ill-conditioned (a head norm over a few channels of a read-out that nearly cancels, a
        # softmax between two nearly equal keys) and multiply rounding from layer to layer, in the plain model as in the
        # engine, whatever the schedule; a fault of the cache or the batch shows on many positions, and in the float32 runs
        if dtype == "bfloat16":
            tol = torch.full_like(err, max(TOL[dtype], 3 * float(floor[rid].mean())))
        else:
            tol = torch.maximum(torch.full_like(err, TOL[dtype]), 3 * floor[rid][:len(err)])
        bad = err > tol
        allowed = 0 if dtype == "float32" else max(3, len(err) // 10)
        assert int(bad.sum()) <= allowed, \
            f"{name} {dtype} {u}: error {float(err.max()):.3g}, {int(bad.sum())} positions over their tolerance; first bad " \
            f"position {int(bad.nonzero()[0])}"
        checked += 1
    assert checked > 0


def check_greedy(model_dir, dtype, prompt, tokens):
    """How many of the engine's tokens are the plain model's choice after the same tokens; every other one must be nearly
    as good there (in bfloat16 one token of a request may be further off, as single positions of a replay may)."""
    ids, exact, far = list(prompt), 0, 0
    for tok in tokens:
        logits = plain_logits(model_dir, ids)[-1].float()
        best = int(logits.argmax())
        gap = float(logits[best] - logits[tok]) / float(logits.abs().max())
        limit = {"float32": 3e-4, "bfloat16": 5e-2}[dtype]
        far += int(gap > limit)
        assert gap <= limit or (dtype == "bfloat16" and gap <= 4 * limit and far <= 1), \
            f"engine chose {tok}, plain {best} (gap {gap:.3g}) after {len(ids)} tokens"
        exact += int(tok == best)
        ids.append(tok)
    return exact


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", ["A", "B"])
def test_greedy_generation_through_the_scheduler_and_a_small_pool(tmp_path, name, dtype):
    from logssms_b200.engine import LLM
    from logssms_b200.sampling import SamplingParams
    raw = ZARI[name]
    model_dir = model_for(tmp_path, name, dtype, sharp=None if dtype == "float32" else 1.0)
    g = torch.Generator().manual_seed(5)
    prompts = [torch.randint(0, raw["vocab"], (n,), generator=g).tolist() for n in (1, 5, 13, 70, 33)]
    new = 12
    llm = LLM(model_dir, dtype, max_running_requests=3, max_seq_len_override=128, num_pages=4, max_prefill_tokens=24,
              poison_on_free=True)
    outs = llm.generate(prompts, SamplingParams(temperature=0.0, max_tokens=new, ignore_eos=True))
    assert [o.finish_reason for o in outs] == ["length"] * len(prompts)
    exact = sum(check_greedy(model_dir, dtype, p, o.token_ids) for p, o in zip(prompts, outs))
    assert all(len(o.token_ids) == new for o in outs) and exact >= 0.8 * new * len(prompts)
    llm.engine.cache.check_integrity()
    assert not llm.engine.cache.live
    again = llm.generate(prompts[:2], SamplingParams(temperature=0.0, max_tokens=new, ignore_eos=True))
    assert [o.token_ids for o in again] == [o.token_ids for o in outs[:2]]


def test_command_line_generates_from_a_model_folder(tmp_path):
    import os
    model_dir = model_for(tmp_path, "A", "float32")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    cmd = [sys.executable, "-m", "logssms_b200", "--model-path", model_dir, "--dtype", "float32", "--max-seq-len-override", "64",
           "--num-pages", "2", "--max-running-requests", "2", "--temperature", "0", "--max-tokens", "5", "--ignore-eos",
           "--prompt-ids", "5,6,7"]
    run = subprocess.run(cmd, cwd=root, capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]
    ids = [int(t) for t in run.stdout.split()]
    assert len(ids) == 5
    check_greedy(model_dir, "float32", [5, 6, 7], ids)
