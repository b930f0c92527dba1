"""The Dodonex design through the engine against the plain implementation (tests/plain_dodonex.py):
whole prompts, token-by-token decoding, portions down to two tokens, unequal batches, pages and
slots that change hands, the captured decode step, long decoding, and greedy generation through
the entry point and the scheduler.  Small configurations of their own (tests/dodonex_cases.py)."""
import pytest
import torch

import dodonex_cases as cases
import plain_dodonex

pytestmark = pytest.mark.gpu

DTYPES = ["float32", "bfloat16"]


@pytest.mark.parametrize("name", ["P", "Q", "R", "S"])
@pytest.mark.parametrize("dtype", DTYPES)
def test_whole_prompt_and_first_tokens(name, dtype):
    runner = cases.make_runner(name, dtype)
    for length, seed in ((1, 1), (2, 2), (3, 3), (70, 4)):  # the first tokens of a sequence, alone and in a prompt
        ids, want = cases.plain_logits(name, length, seed)
        got = cases.replay(runner, f"w{length}", ids, [length])
        cases.assert_close(got, want, dtype, f"{name} whole {length}")


@pytest.mark.parametrize("name", ["P", "Q", "R"])
@pytest.mark.parametrize("dtype", DTYPES)
def test_prefill_then_token_by_token(name, dtype):
    ids, want = cases.plain_logits(name, 90, 7)
    runner = cases.make_runner(name, dtype)
    got = cases.replay(runner, "d", ids, [50] + [1] * 40)
    cases.assert_close(got, want, dtype, f"{name} decode")
    got = cases.replay(runner, "t", ids[:40], [1] * 40)  # from the very first token on, in the slot just freed
    cases.assert_close(got, want[:40], dtype, f"{name} token by token")


@pytest.mark.parametrize("name", ["P", "Q", "R", "S"])
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("page_size", [8, 16])
def test_portions_of_changing_size(name, dtype, page_size):
    ids, want = cases.plain_logits(name, 150, 9)
    runner = cases.make_runner(name, dtype, page_size=page_size)
    pattern = [7, 2, 5, 3, 16, 2, 9, 1, 4, 33, 2, 6, 17, 8, 15, 1, 2, 2]
    cuts = []
    while sum(cuts) < len(ids):
        cuts.append(min(pattern[len(cuts) % len(pattern)], len(ids) - sum(cuts)))
    got = cases.replay(runner, "c", ids, cuts)
    cases.assert_close(got, want, dtype, f"{name} portions")
    if dtype == "float32":  # the order of every sum depends on the position alone
        whole = cases.replay(runner, "w", ids, [len(ids)])
        assert torch.equal(got, whole)


@pytest.mark.parametrize("dtype", DTYPES)
def test_steps_of_many_tokens(dtype):
    """300 tokens in one step, and 270 behind 30 cached ones: in bfloat16 the per-head products of the
    latent attention run on the tensor cores from 256 tokens on."""
    ids, want = cases.plain_logits("R", 300, 11)
    runner = cases.make_runner("R", dtype)
    cases.assert_close(cases.replay(runner, "a", ids, [300]), want, dtype, "300 tokens")
    cases.assert_close(cases.replay(runner, "b", ids, [30, 270]), want, dtype, "270 behind 30")


def _calls(monkeypatch, *names):
    """How often each of these functions of ``ops`` is called."""
    from torchlet_b200 import ops

    counts = dict.fromkeys(names, 0)
    for name in names:
        def counted(*args, name=name, inner=getattr(ops, name), **kwargs):
            counts[name] += 1
            return inner(*args, **kwargs)

        monkeypatch.setattr(ops, name, counted)
    return counts


def _step(runner, portions):
    """One step of (request, tokens): every position's logits, by request."""
    from torchlet_b200.engine import StepEntry

    logits = runner.step([StepEntry(r, ids, list(range(len(ids)))) for r, ids in portions]).cpu()
    return dict(zip([r for r, _ in portions], logits.split([len(ids) for _, ids in portions])))


@pytest.mark.parametrize("lengths", [(300,), (257, 2, 130), (40, 256)])
def test_whole_prompts_with_expanded_keys(lengths, monkeypatch):
    """Steps of whole prompts on the kernel that expands keys and values, each request then continued behind its cache: one
    token, and a portion, on the latent form."""
    counts = _calls(monkeypatch, "latent_prompt", "latent_attention_mma")
    seqs = [cases.plain_logits("T", n + 34, 60 + n) for n in lengths]
    runner = cases.make_runner("T", "bfloat16", num_pages=80)
    for r in range(len(lengths)):
        runner.admit(r)
    got = _step(runner, [(r, seqs[r][0][:n]) for r, n in enumerate(lengths)])
    assert counts["latent_prompt"] == 3 and counts["latent_attention_mma"] == 0
    for r, n in enumerate(lengths):
        cases.assert_close(got[r], seqs[r][1][:n], "bfloat16", f"prompt {r}")
    for first, last in ((0, 1), (1, 34)):
        got = _step(runner, [(r, seqs[r][0][n + first:n + last]) for r, n in enumerate(lengths)])
        for r, n in enumerate(lengths):
            cases.assert_close(got[r], seqs[r][1][n + first:n + last], "bfloat16", f"request {r} behind its prompt")
    assert counts["latent_prompt"] == 3


@pytest.mark.parametrize("before,tokens", [(30, 270), (1, 300)])
def test_portions_behind_cached_tokens_keep_the_latent_form(before, tokens, monkeypatch):
    counts = _calls(monkeypatch, "latent_prompt")
    ids, want = cases.plain_logits("T", before + tokens, 91)
    got = cases.replay(cases.make_runner("T", "bfloat16"), "a", ids, [before, tokens])
    cases.assert_close(got, want, "bfloat16", f"{tokens} behind {before}")
    assert counts["latent_prompt"] == 0


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("decoders,tokens,chunked", [(2, 96, True), (2, 95, False), (1, 256, True), (1, 255, False), (3, 300, True)])
def test_long_portions_beside_decoding_requests(dtype, decoders, tokens, chunked, monkeypatch):
    """A prompt in one step with requests that decode: their recurrences run on kernels of their own where the portion's goes
    chunk by chunk, and every request continues from the state its kernel left."""
    counts = _calls(monkeypatch, "delta_chunked", "delta_scan")
    seqs = [cases.plain_logits("R", 20, 70 + r) for r in range(decoders)] + [cases.plain_logits("R", tokens + 5, 80)]
    runner = cases.make_runner("R", dtype)
    for r in range(decoders + 1):
        runner.admit(r)
    for r in range(decoders):
        _step(runner, [(r, seqs[r][0][:17])])
    counts["delta_scan"] = counts["delta_chunked"] = 0
    order = [decoders] + list(range(decoders)) if decoders == 2 else list(range(decoders + 1))
    got = _step(runner, [(r, seqs[r][0][:tokens] if r == decoders else seqs[r][0][17:18]) for r in order])
    assert counts["delta_chunked"] == (chunked and dtype == "bfloat16") and counts["delta_scan"] == 1
    for r in range(decoders):
        cases.assert_close(got[r], seqs[r][1][17:18], dtype, f"decoding request {r}")
    cases.assert_close(got[decoders], seqs[decoders][1][:tokens], dtype, "the portion")
    got = _step(runner, [(r, seqs[r][0][tokens:] if r == decoders else seqs[r][0][18:]) for r in order])
    for r in range(decoders + 1):
        cases.assert_close(got[r], seqs[r][1][tokens if r == decoders else 18:], dtype, f"request {r} afterwards")


def test_scratch_memory_of_the_delta_rule_is_that_of_one_token_and_stays():
    """What the first decode step allocates for the recurrence serves every later step of the token budget: a long portion, and
    many that each end in a chunk of a few tokens."""
    from torchlet_b200.engine import StepEntry

    runner = cases.make_runner("R", "bfloat16", slots=20, num_pages=80, budget=512)

    def step(lengths):
        for r, n in enumerate(lengths):
            runner.admit(r)
        runner.step([StepEntry(r, cases.make_ids("R", n, r), []) for r, n in enumerate(lengths)])
        for r in range(len(lengths)):
            runner.finish(r)
        return {key: (t.data_ptr(), t.numel()) for key, t in runner._buffers.items() if key.startswith("delta.")}

    first = step([1])
    for lengths in ([500], [33] * 15, [1, 480, 3], [41] * 12):
        assert step(lengths) == first


@pytest.mark.parametrize("name", ["P", "R"])
@pytest.mark.parametrize("dtype", DTYPES)
def test_unequal_batches_with_pages_and_slots_used_again(name, dtype):
    """Up to three live requests in three slots; the pool holds little more than the live tokens:
    every request later in the list runs in a slot and in pages that another one has left."""
    from torchlet_b200.engine import StepEntry

    lengths = (61, 23, 100, 2, 37, 48)
    seqs = [cases.plain_logits(name, n, 20 + i) for i, n in enumerate(lengths)]
    runner = cases.make_runner(name, dtype, num_pages=26, slots=3, page_size=8)
    at = [0] * len(seqs)
    got = [[] for _ in seqs]
    waiting, live = list(range(len(seqs))), []
    portions = [5, 1, 19, 2, 1, 1, 30, 3, 1, 8]
    turn = 0
    while waiting or live:
        while waiting and len(live) < 3 and runner.cache.num_free_slots:
            need = -(-lengths[waiting[0]] // 8)
            held = sum(-(-lengths[r] // 8) for r in live)
            if held + need > 25:
                break
            r = waiting.pop(0)
            runner.admit(r)
            live.append(r)
        entries, taken = [], []
        for r in live:
            size = min(portions[(turn + 3 * r) % len(portions)], lengths[r] - at[r])
            ids = seqs[r][0]
            entries.append(StepEntry(r, ids[at[r]:at[r] + size], list(range(size))))
            taken.append((r, size))
        logits = runner.step(entries).cpu()
        row = 0
        for r, size in taken:
            got[r].append(logits[row:row + size].clone())
            row += size
            at[r] += size
            if at[r] == lengths[r]:
                runner.finish(r)
                live.remove(r)
        runner.cache.check()
        turn += 1
    for r, (ids, want) in enumerate(seqs):
        cases.assert_close(torch.cat(got[r]), want, dtype, f"{name} request {r}")
    if dtype == "float32":  # each request alone gives the very same numbers
        alone = cases.replay(runner, "alone", seqs[2][0], [lengths[2]])
        assert torch.equal(torch.cat(got[2]), alone)


@pytest.mark.parametrize("name", ["P", "Q"])
@pytest.mark.parametrize("dtype", DTYPES)
def test_captured_decode_step_with_padding_lanes(name, dtype):
    """Three requests decode together in a bucket of four lanes (one is padding) from the captured
    graph; the state of a fourth request, which waits meanwhile, must not be touched by the padding lane."""
    from torchlet_b200.engine import StepEntry

    seqs = [cases.plain_logits(name, n, 40 + i) for i, n in enumerate((33, 12, 25, 30))]
    runner = cases.make_runner(name, dtype, slots=4, cuda_graph=True)
    for r, (ids, _) in enumerate(seqs):
        runner.admit(r)
    for r, (ids, _) in enumerate(seqs):  # prompts without their last 10 tokens; request 3 stays behind
        runner.step([StepEntry(r, ids[:len(ids) - 10], [])])
    got = {r: [] for r in range(3)}
    for k in range(10):
        entries = [StepEntry(r, [seqs[r][0][len(seqs[r][0]) - 10 + k]], [0]) for r in range(3)]
        logits = runner.step(entries).cpu()
        for r in range(3):
            got[r].append(logits[r].clone())
    assert runner.graph_steps == 10
    for r in range(3):
        want = seqs[r][1][-10:]
        cases.assert_close(torch.stack(got[r]), want, dtype, f"{name} graph request {r}")
    ids, want = seqs[3]
    rest = runner.step([StepEntry(3, ids[-10:], list(range(10)))]).cpu()  # its state survived the padding lane
    cases.assert_close(rest, want[-10:], dtype, f"{name} the request that waited")


@pytest.mark.parametrize("dtype", DTYPES)
def test_long_decoding(dtype):
    ids, want = cases.plain_logits("Q", 400, 77)
    runner = cases.make_runner("Q", dtype, num_pages=40, cuda_graph=True)
    got = cases.replay(runner, "long", ids, [20] + [1] * 380)
    assert runner.graph_steps == 380
    cases.assert_close(got, want, dtype, "long decoding")


@pytest.mark.parametrize("dtype", DTYPES)
def test_greedy_generation_through_the_entry_point(tmp_path, dtype):
    import json

    from safetensors.torch import save_file

    from torchlet_b200 import LLM

    name = "P"
    folder = tmp_path / "model"
    folder.mkdir()
    raw = json.loads(json.dumps(cases.CASES[name]))
    for layer in raw["layers"]:
        layer["mixer"].pop("decay_rank", None)  # the loader takes it from the tensor's shape
    (folder / "config.json").write_text(json.dumps(raw))
    w = cases.weights_for(name)
    save_file({k: v.to(torch.bfloat16).contiguous() for k, v in w.items()}, str(folder / "model.safetensors"))
    llm = LLM(folder, max_decode_slots=2, kv_block_size=8, dtype=dtype, max_seq_len=96, max_num_blocks=30,
              max_num_batched_tokens=32)
    prompts = [cases.make_ids(name, n, 60 + i) for i, n in enumerate((5, 40, 17, 1))]  # more requests than slots
    new = 10
    outputs = llm.generate(prompts, max_new_tokens=new)
    assert llm.engine.runner.graph_steps > 0
    cfg = cases.CASES[name]
    for prompt, got in zip(prompts, outputs):
        assert len(got) == new
        ids = list(prompt)
        for token in got:
            logits = plain_dodonex.forward(cfg, w, ids)[-1]
            if dtype == "float32":
                assert token == int(logits.argmax())
            else:  # bfloat16 may flip a near-tie: the token must be within rounding of the best
                assert logits[token] >= logits.max() - cases.TOLERANCE[dtype] * logits.abs().max()
            ids.append(token)
    llm.engine.runner.cache.check()
    assert llm.engine.runner.cache.live_requests() == []


def test_trace_replay_chooses_the_model_by_its_configuration(tmp_path):
    import io
    import json

    import numpy as np
    from safetensors.torch import save_file

    from torchlet_b200.engine import trace

    name = "Q"
    folder = tmp_path / "model"
    folder.mkdir()
    (folder / "config.json").write_text(json.dumps(cases.CASES[name]))
    save_file({k: v.to(torch.bfloat16).contiguous() for k, v in cases.weights_for(name).items()},
              str(folder / "model.safetensors"))
    ids, want = cases.plain_logits(name, 30, 5)
    steps = [{"step": 0, "entries": [{"id": "a", "tokens": ids[:20], "want": [0, 19]}], "end": []},
             {"step": 1, "entries": [{"id": "a", "tokens": ids[20:21], "want": [0]}], "end": []},
             {"step": 2, "entries": [{"id": "a", "tokens": ids[21:], "want": [8]}], "end": ["a"]}]
    out = tmp_path / "out"
    code = trace.main(["--model", str(folder), "--dtype", "float32", "--out", str(out), "--max-tokens", "64"],
                      stdin=io.StringIO("\n".join(json.dumps(s) for s in steps) + "\n"), stdout=io.StringIO())
    assert code == 0
    V = cases.CASES[name]["vocab"]
    got = torch.cat([torch.from_numpy(np.fromfile(out / f"{i}.f32", dtype="<f4").reshape(-1, V)) for i in range(3)])
    cases.assert_close(got, want[[0, 19, 20, 29]], "float32", "trace replay")
