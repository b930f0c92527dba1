"""Each mechanism of the Dodonex design alone: the kernels against the plain functions of
tests/plain_dodonex.py, at sizes of their own, with inputs designed so that a fault shows (one far
key among hundreds, a key at a page's border, stale pages full of NaN, a state that must carry)."""
import math

import numpy as np
import pytest
import torch

import plain_dodonex as plain

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rand(*shape, seed=0, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(*shape, generator=g) * scale


@pytest.mark.parametrize("width,groups", [(96, 3), (64, 1), (120, 5), (4096, 4), (70, 7)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_grouped_rms_norm(width, groups, out_dtype):
    from torchlet_b200 import ops

    x = rand(9, width, seed=1, scale=3.0)
    x[:, :width // groups] *= 50.0  # a part with a scale of its own: one norm over the row would show
    w = 1.0 + rand(width, seed=2, scale=0.2)
    want = plain.group_rms_norm(x.double(), w.double(), 1e-5, groups)
    out = torch.empty(9, width, device=DEV, dtype=out_dtype)
    ops.rms_norm(x.to(DEV), w.to(DEV), 1e-5, out, None, groups)
    tol = 1e-5 if out_dtype == torch.float32 else 1e-2
    assert (out.cpu().double() - want).abs().max() <= tol * want.abs().max()
    rows = torch.tensor([7, 0, 3], dtype=torch.int32, device=DEV)
    some = torch.empty(3, width, device=DEV, dtype=out_dtype)
    ops.rms_norm(x.to(DEV), w.to(DEV), 1e-5, some, rows, groups)
    assert torch.equal(some, out[rows.long()])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_clamped_glu_on_both_sides_of_the_limit(dtype):
    from torchlet_b200 import ops

    inter, limit = 52, 1.3
    gu = rand(11, 2 * inter, seed=3, scale=2.0).to(dtype)  # many values beyond the limit on either side
    g, u = gu[:, :inter].double(), gu[:, inter:].double()
    g = torch.clamp(g, max=limit)
    u = torch.clamp(u, min=-limit, max=limit)
    want = g * torch.sigmoid(1.702 * g) * (u + 1.0)
    out = torch.empty(11, inter, device=DEV, dtype=dtype)
    ops.clamped_glu(gu.to(DEV), out, limit, 1.702)
    tol = 1e-6 if dtype == torch.float32 else 1e-2
    assert (out.cpu().double() - want).abs().max() <= tol * want.abs().max()
    assert (gu[:, :inter] < -limit).any() and (gu[:, :inter] > limit).any()  # the gate is clamped from above only


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_gated_token_embedding_part(dtype):
    from torchlet_b200.config import PartSpec
    from torchlet_b200.parts import TOKEN_INPUTS, build_part

    W, dim, V, layers, layer, m, eps = 72, 12, 50, 3, 1, 0.7, 1e-5
    w = {"side.embed": rand(V, dim * layers, seed=4).bfloat16().float(),
         f"l{layer}.side.gate": rand(dim, W, seed=5, scale=0.3).bfloat16().float(),
         f"l{layer}.side.proj": rand(W, dim, seed=6, scale=0.3).bfloat16().float(),
         f"l{layer}.side.norm": (1 + rand(W, seed=7, scale=0.1)).bfloat16().float()}
    part = build_part(TOKEN_INPUTS, PartSpec("gated_token_embedding", {
        "hidden_size": W, "dim": dim, "eps": eps, "vocab_size": V, "table_name": "side.embed",
        "table_width": dim * layers, "offset": layer * dim}))
    torch_dtype = getattr(torch, dtype)
    part.load(w, f"l{layer}.side.", DEV, torch_dtype)
    ids = torch.randint(0, V, (13,), generator=torch.Generator().manual_seed(8))
    x = rand(13, W, seed=9, scale=2.0)
    cfg = {"token_side": {"dim": dim}, "norm": {"eps": eps}}
    want = x.double() + m * plain.token_side(x.double(), ids, {k: v.double() for k, v in w.items()}, layer, cfg)

    class Ctx:
        tokens = ids.to(DEV, torch.int32)

        def __init__(self):
            self.dtype = torch_dtype

        def buffer(self, name, shape, dt):
            return torch.empty(shape, device=DEV, dtype=dt)

    acc = x.to(DEV)
    part.forward(Ctx(), acc, m)
    tol = 1e-5 if dtype == "float32" else 2e-2
    assert (acc.cpu().double() - want).abs().max() <= tol * want.abs().max()


def delta_weights(W, H, D, rank, seed):
    size = H * D
    names = {"r": (size, W), "k": (size, W), "v": (size, W), "g": (size, W), "a": (size, W), "a.b": (size,),
             "w1": (rank, W), "w2": (size, rank), "w0": (size,), "norm": (size,), "o": (W, size)}
    out = {}
    for i, (name, shape) in enumerate(names.items()):
        t = rand(*shape, seed=seed + i, scale=1.0 if len(shape) == 1 else 1.5 / math.sqrt(shape[-1]))
        out["m." + name] = (1 + 0.1 * t if name == "norm" else t).bfloat16().float()
    return out


@pytest.mark.parametrize("H,D,rank", [(2, 24, 5), (1, 64, 16), (3, 40, 7), (2, 100, 4), (1, 16, 2), (1, 200, 3), (1, 256, 8)])
def test_delta_rule_kernels_carry_the_state(H, D, rank):
    """prepare, scan and finish against the plain recurrence: a sequence in three portions (the
    state must carry), beside another request; then the first slot is used again from zero."""
    from torchlet_b200 import ops

    W, size, eps = 48, H * D, 1e-5
    w = delta_weights(W, H, D, rank, seed=10 * H + D)
    mixer = {"heads": H, "dim": D}
    hs = [rand(n, W, seed=30 + i) for i, n in enumerate((37, 9, 21))]
    fused = torch.cat([w["m." + n] for n in ("r", "k", "v", "g", "a", "w1")]).to(DEV)
    f32 = lambda name: w["m." + name].to(DEV)
    state = torch.full((3, H, D, D), float("nan"), device=DEV)  # a slot is zeroed at admission, not before

    def run(parts):  # parts: list of (slot, h rows); one step
        rows = torch.cat([h for _, h in parts]).to(DEV)
        proj = rows @ fused.T
        T = rows.shape[0]
        gates = torch.empty(T, H * 3 * D, device=DEV)
        ops.delta_prepare(proj, f32("w2").t().contiguous(), f32("w0"), f32("a.b"), gates, H, D, rank)
        indptr = torch.tensor([0] + list(torch.tensor([h.shape[0] for _, h in parts]).cumsum(0)), dtype=torch.int32,
                              device=DEV)
        slots = torch.tensor([s for s, _ in parts], dtype=torch.int32, device=DEV)
        o = torch.empty(T, size, device=DEV)
        ops.delta_scan(proj, gates, indptr, slots, state, o, len(parts), H, D)
        out = torch.empty(T, size, device=DEV)
        ops.delta_finish(o, proj, f32("norm"), out, H, D, eps)
        return (out @ f32("o").T).cpu()

    wd = {k: v.double() for k, v in w.items()}
    want = [plain.general_delta(h.double(), wd, "m.", mixer, eps)[0] for h in hs]
    state[2].zero_(); state[0].zero_()
    a = run([(2, hs[0][:5]), (0, hs[1])])          # two requests of unequal length in one step
    b = run([(2, hs[0][5:7])])                     # a portion of two tokens
    c = run([(-1, hs[1][:1]), (2, hs[0][7:])])     # beside a padding lane, which touches no state
    got0 = torch.cat([a[:5], b, c[1:]])
    scale = want[0].abs().max()
    assert (got0.double() - want[0]).abs().max() <= 2e-5 * scale
    assert (a[5:].double() - want[1]).abs().max() <= 2e-5 * want[1].abs().max()
    assert torch.equal(c[:1], torch.zeros_like(c[:1]))
    state[2].zero_()                               # the slot is used again
    d = run([(2, hs[2])])
    assert (d.double() - want[2]).abs().max() <= 2e-5 * want[2].abs().max()
    assert torch.isnan(state[1]).all()             # the slot nobody had stays untouched


@pytest.mark.parametrize("H,D,stride_pad", [(2, 64, 0), (3, 36, 4), (2, 100, 0), (1, 200, 0), (1, 64, 1)])
def test_delta_scan_gives_the_same_bits_from_few_and_from_many_blocks(H, D, stride_pad):
    """Up to 148 (request, head) pairs several blocks share a head's columns, beyond one block takes them: the same additions, so
    the same bits, for whole chunks of tokens, remainders, single tokens and (odd stride) the copies of one float."""
    from torchlet_b200 import ops

    lens = [19, 1, 8, 33] + [1] * (150 // H)
    size, T = H * D, sum(lens)
    width = 5 * size + stride_pad
    proj = rand(T, width, seed=3).to(DEV)
    gates = torch.rand(T, H, 3, D, generator=torch.Generator().manual_seed(4)) / D
    gates[:, :, 0] = gates[:, :, 0] * D * 0.4 + 0.55  # decays; the others keep the removal below what was there
    gates = gates.view(T, -1).to(DEV)
    start = rand(len(lens), H, D, D, seed=5, scale=0.1).to(DEV)
    slots = torch.arange(len(lens), dtype=torch.int32, device=DEV)

    def run(a, b):  # requests a to b - 1 in one step
        first, count = sum(lens[:a]), sum(lens[a:b])
        indptr = torch.tensor([0] + torch.tensor(lens[a:b]).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
        state, out = start.clone(), torch.full((count, size), float("nan"), device=DEV)
        rows = proj[first:first + count]
        ops.delta_scan(rows, gates[first:first + count], indptr, slots[a:b].contiguous(), state, out, b - a, H, D)
        return out, state

    many, state = run(0, len(lens))
    for r in range(5):
        out, alone = run(r, r + 1)
        assert torch.equal(out, many[sum(lens[:r]):sum(lens[:r + 1])]) and torch.equal(alone[r], state[r])


@pytest.mark.parametrize("H,D,requests", [(4, 64, 1), (40, 64, 2), (5, 128, 8), (75, 32, 4)])
def test_delta_scan_blocks_kept_apart(H, D, requests):
    """Portions of 64 tokens and more take shared memory by how many blocks an SM has: one, two, three, more; the bits are
    those of the same tokens in portions of fewer."""
    from torchlet_b200 import ops

    n, size = 66, H * D
    T = n * requests
    proj = rand(T, 5 * size, seed=3).to(DEV)
    gates = torch.rand(T, H, 3, D, generator=torch.Generator().manual_seed(4)) / D
    gates[:, :, 0] = gates[:, :, 0] * D * 0.4 + 0.55
    gates = gates.view(T, -1).to(DEV)
    state, out = torch.zeros(requests, H, D, D, device=DEV), torch.empty(T, size, device=DEV)
    slots = torch.arange(requests, dtype=torch.int32, device=DEV)
    indptr = torch.arange(0, T + 1, n, dtype=torch.int32, device=DEV)
    ops.delta_scan(proj, gates, indptr, slots, state, out, requests, H, D)
    for r in range(requests):
        again = torch.zeros_like(state)
        for first, last in ((0, 40), (40, n)):
            rows = slice(r * n + first, r * n + last)
            part = torch.empty(last - first, size, device=DEV)
            ops.delta_scan(proj[rows], gates[rows], torch.tensor([0, last - first], dtype=torch.int32, device=DEV), slots[r:r + 1], again, part, 1, H, D)
            assert torch.equal(part, out[rows])
        assert torch.equal(again[r], state[r])


def test_delta_scans_of_two_threads_keep_their_shared_memory():
    """Two engines in two threads launch the same kernel with one and with four blocks an SM, which take unlike amounts of shared
    memory: neither launch is refused, and the bits are those of one thread alone."""
    from concurrent.futures import ThreadPoolExecutor

    from torchlet_b200 import ops

    D, n = 16, 64

    def inputs(H):
        proj, gates = rand(n, 5 * H * D, seed=H).to(DEV), torch.rand(n, H * 3 * D, generator=torch.Generator().manual_seed(H)).to(DEV) / D
        return proj, gates, *(torch.tensor(x, dtype=torch.int32, device=DEV) for x in ([0, n], [0]))

    def launch(H, given, times):
        state, out = torch.zeros(1, H, D, D, device=DEV), torch.empty(n, H * D, device=DEV)
        for _ in range(times):
            state.zero_()
            ops.delta_scan(*given, state, out, 1, H, D)
        return out, state

    heads = (8, 500)  # (a block a head at this head size)
    given = {H: inputs(H) for H in heads}
    want = {H: launch(H, given[H], 1) for H in heads}
    torch.cuda.synchronize()
    with ThreadPoolExecutor(4) as pool:
        jobs = [(H, pool.submit(launch, H, given[H], 2000)) for H in heads * 2]
        for H, job in jobs:
            for a, b in zip(job.result(), want[H]):
                assert torch.equal(a, b)


@pytest.mark.parametrize("lens,H,D,rank,pad", [([8], 1, 64, 16, 0), ([37, 9, 1, 8, 16, 100], 2, 64, 16, 0), ([37, 3], 2, 24, 5, 0),
                                               ([50, 2, 41], 3, 40, 7, 0), ([23], 1, 4, 2, 0), ([300], 2, 64, 64, 3)])
def test_delta_rule_chunk_by_chunk(lens, H, D, rank, pad):
    """Against the recurrence in float64, and no further from it than the token-wise kernels (by a half at most: single
    sums of few terms vary); requests below ``least`` and padding lanes leave state and output to the other kernel."""
    from torchlet_b200 import ops

    size, T, R = H * D, sum(lens), len(lens)
    proj = rand(T, 5 * size + rank + pad, seed=1).to(DEV)[:, :5 * size + rank]
    w2, w0, bias = rand(rank, size, seed=2, scale=rank ** -0.5).to(DEV), rand(size, seed=3).to(DEV), rand(size, seed=4).to(DEV)
    start = rand(R + 1, H, D, D, seed=5, scale=0.3).to(DEV)
    indptr = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    slots = torch.arange(R, dtype=torch.int32, device=DEV)

    def chunked(least, slots):
        state, out = start.clone(), torch.full((T, size), float("nan"), device=DEV)
        chunks = sum(-(-n // ops.delta_chunk_tokens()) for n in lens if n >= least)
        records = torch.full((chunks * H * ops.delta_chunk_record(),), float("nan"), device=DEV)
        ops.delta_chunked(proj, w2, w0, bias, indptr, slots, state, out, records, R, chunks, least, H, D, rank)
        return out, state

    def token_wise(below):
        state, out = start.clone(), torch.full((T, size), float("nan"), device=DEV)
        gates = torch.empty(T, H * 3 * D, device=DEV)
        ops.delta_prepare(proj, w2, w0, bias, gates, H, D, rank)
        ops.delta_scan(proj, gates, indptr, slots, state, out, R, H, D, below=below)
        return out, state

    x = proj.double()
    r, k, v = (x[:, i * size:(i + 1) * size].view(T, H, D) for i in range(3))
    a = torch.sigmoid(x[:, 4 * size:5 * size] + bias.double()).view(T, H, D)
    inner = torch.tanh(x[:, 5 * size:5 * size + rank]) @ w2.double() + w0.double()
    w = torch.exp(-math.exp(-0.5) * torch.sigmoid(inner)).view(T, H, D)
    u = k / torch.sqrt(k.pow(2).sum(-1, keepdim=True) + 1e-6)
    want, ends = [], []
    for q in range(R):
        S = start[q].double()
        for t in range(int(indptr[q]), int(indptr[q + 1])):
            seen = u[t][:, None, :] @ S
            S = w[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :] - (a[t] * u[t])[:, :, None] * seen
            want.append((r[t][:, None, :] @ S).reshape(1, size))
        ends.append(S)
    want, ends = torch.cat(want), torch.stack(ends)
    error = lambda got, right: ((got.double() - right).norm() / right.norm()).item()
    out, state = chunked(1, slots)
    plain_out, plain_state = token_wise(None)
    assert error(out, want) <= max(1.5 * error(plain_out, want), 1e-7)
    assert error(state[:R], ends) <= max(1.5 * error(plain_state[:R], ends), 1e-7)
    assert torch.equal(state[R], start[R])
    # the two kernels side by side share the requests by length
    some, some_state = chunked(9, slots)
    rest, rest_state = token_wise(9)
    for q, n in enumerate(lens):
        rows = slice(int(indptr[q]), int(indptr[q + 1]))
        mine, other = ((some, some_state), (rest, rest_state)) if n >= 9 else ((rest, rest_state), (some, some_state))
        assert torch.equal(mine[0][rows], out[rows] if n >= 9 else plain_out[rows])
        assert torch.isnan(other[0][rows]).all() and torch.equal(other[1][q], start[q])
    padded, padded_state = chunked(1, torch.full_like(slots, -1))
    assert (padded == 0).all() and torch.equal(padded_state, start)


@pytest.mark.parametrize("T,H,N,K,gap", [(1, 1, 8, 64, 0), (129, 3, 72, 64, 8), (300, 4, 256, 192, 0), (257, 5, 520, 128, 24)])
def test_products_by_heads_in_one_launch(T, H, N, K, gap):
    """Against float64 within the rounding of the bfloat16 result; columns between the heads' stay as they were."""
    from torchlet_b200 import ops

    x, w = rand(T, H * K, seed=1).to(DEV).bfloat16(), rand(H, N, K, seed=2).to(DEV).bfloat16()
    step = N + gap
    out = torch.full((T, H * step), 7.0, device=DEV, dtype=torch.bfloat16)
    ops.gemm_tc_heads(x, w, out, step)
    want = torch.einsum("thk,hnk->thn", x.double().view(T, H, K), w.double())
    got = out.view(T, H, step)
    bound = 2.0 ** -8 * want.abs() + K * 2.0 ** -23 * torch.einsum("thk,hnk->thn", x.double().view(T, H, K).abs(), w.double().abs())
    assert ((got[..., :N].double() - want).abs() <= bound).all()
    assert (got[..., N:] == 7.0).all()


@pytest.mark.parametrize("room", [5, 6, 9, 14, 18])
def test_delta_chunks_in_passes_give_the_bits_of_one(room):
    """Records for fewer chunks than the step has: the passes cut every request, continue its state and leave the shorter
    requests and padding lanes alone."""
    from torchlet_b200 import ops

    lens, least, H, D, rank = [37, 9, 3, 70, 16, 1, 8], 8, 2, 40, 5
    size, T, R = H * D, sum(lens), len(lens)
    proj = rand(T, 5 * size + rank, seed=1).to(DEV)
    w2, w0, bias = rand(rank, size, seed=2, scale=rank ** -0.5).to(DEV), rand(size, seed=3).to(DEV), rand(size, seed=4).to(DEV)
    indptr = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    slots = torch.tensor([3, 1, 0, 4, -1, 5, 2], dtype=torch.int32, device=DEV)
    each, floats = np.array([-(-n // 8) for n in lens if n >= least]), H * ops.delta_chunk_record()
    chunks = int(each.sum())
    assert ops.delta_chunk_tokens() == 8 and chunks == 19

    def run(room):
        state, out = rand(6, H, D, D, seed=5, scale=0.3).to(DEV), torch.full((T, size), -1.0, device=DEV)
        records = torch.full((room * floats + 7,), float("nan"), device=DEV)
        passes = ops.delta_chunk_passes(each, room)
        assert len(passes) > (room < chunks)
        ops.delta_chunked(proj, w2, w0, bias, indptr, slots, state, out, records, R, chunks, least, H, D, rank, passes)
        assert torch.isnan(records[room * floats:]).all()
        return out, state

    for a, b in zip(run(room), run(chunks)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("lens,D,V", [([129, 200, 3, 140], 64, 128), ([70, 130, 300], 128, 64)])
def test_whole_prompts_beside_rows_without_a_number(lens, D, V):
    """A key tile reaches into the next request's rows: NaN there stays its own."""
    from torchlet_b200 import ops

    T, H, bf = sum(lens), 2, torch.bfloat16
    queries, keys, k_rot, values = (rand(T, n, seed=i).to(DEV).to(bf) for i, n in enumerate((H * (D + 64), H * D, 64, H * V)))
    ends = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    step = ops.latent_prompt_tokens()
    tile_req, tile_row = (torch.tensor(x, dtype=torch.int32, device=DEV)
                          for x in zip(*[(r, row) for r, n in enumerate(lens) for row in range(0, n, step)]))

    def run():
        out = torch.full((T, H * V), -1.0, device=DEV, dtype=bf)
        ops.latent_prompt(queries, keys, k_rot, values, ends, tile_req, tile_row, tile_req.numel(), out, H, D, 64, V, 0.1)
        assert ops.latent_prompt_error() == 0
        return out

    clean = run()
    for t in (keys, k_rot, values):
        t[lens[0]:lens[0] + lens[1]] = float("nan")
    others = [i for i in range(T) if not lens[0] <= i < lens[0] + lens[1]]
    assert clean.isfinite().all() and torch.equal(run()[others], clean[others])


@pytest.mark.parametrize("R,dims", [(32, 16), (48, 48), (64, 2), (16, 0)])
def test_rows_of_whole_prompts_turn_the_rotated_entries_alone(R, dims):
    from torchlet_b200 import ops

    T, H, D, rank, page_size, bf = 130, 2, 64, 40, 16, torch.bfloat16
    q = rand(T, H * (D + R) + 8, seed=1).to(DEV)[:, 8:]  # (a column range of a wider product)
    pages = rand(10, 1, 1, page_size, rank + R, seed=2).to(DEV).to(bf)
    table = torch.arange(9, 0, -1, dtype=torch.int32, device=DEV)[None]
    inv_freq = (500.0 ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64) / max(dims, 1))).float().to(DEV)
    positions = torch.arange(T, dtype=torch.int32, device=DEV)
    queries, c, k_rot = (torch.empty(T, n, device=DEV, dtype=bf) for n in (H * (D + 64), rank, 64))
    ops.latent_prompt_rows(q, inv_freq, positions, torch.zeros_like(positions), table, pages, page_size, queries, c, k_rot, H, D, R, dims)
    x = q.contiguous().double().view(T, H, D + R)
    want = torch.zeros(T, H, D + 64, dtype=torch.float64, device=DEV)
    want[..., :D + R] = x
    angle = positions.double()[:, None, None] * inv_freq.double()
    a, b = x[..., D:D + dims // 2], x[..., D + dims // 2:D + dims]
    want[..., D:D + dims] = torch.cat((a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()), -1)
    # one rounding to bfloat16, and the float32 angle's own (130 x 2^-24)
    assert ((queries.double().view_as(want) - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all()
    rows = pages[table[0].long()].view(-1, rank + R)[:T]
    assert torch.equal(c, rows[:, :rank]) and torch.equal(k_rot[:, :R], rows[:, rank:]) and not k_rot[:, R:].any()


@pytest.mark.parametrize("lens,H,D,R,V,rank,page_size", [([128], 1, 64, 16, 64, 64, 16), ([257, 2, 130], 2, 128, 64, 128, 72, 8),
                                                          ([129, 300], 3, 64, 32, 128, 40, 16), ([513, 127], 2, 128, 48, 64, 64, 32)])
def test_latent_attention_of_whole_prompts(lens, H, D, R, V, rank, page_size):
    """Rows, expansion and attention against float64 over the bfloat16 cache rows: queries, keys, values and P are rounded to
    bfloat16 once (2^-9 each of a weighted mean, whose weights the rounded scores move by a little more)."""
    from torchlet_b200 import ops

    T, bf = sum(lens), torch.bfloat16
    q = rand(T, H * (D + R), seed=1).to(DEV)
    rows = rand(T, rank + R, seed=2).to(DEV).to(bf)
    uk, uv = rand(H * D, rank, seed=3, scale=rank ** -0.5).to(DEV).to(bf), rand(H * V, rank, seed=4, scale=rank ** -0.5).to(DEV).to(bf)
    inv_freq = (10000.0 ** (-2.0 * torch.arange(R // 2, dtype=torch.float64) / R)).float().to(DEV)
    need = [-(-n // page_size) for n in lens]
    order = torch.randperm(sum(need), generator=torch.Generator().manual_seed(5)) + 1
    pages = torch.full((sum(need) + 1, 1, 1, page_size, rank + R), float("nan"), device=DEV, dtype=bf)
    table = torch.zeros(len(lens), max(need), dtype=torch.int32)
    positions = torch.cat([torch.arange(n) for n in lens]).to(torch.int32)
    token_req = torch.cat([torch.full((n,), r) for r, n in enumerate(lens)]).to(torch.int32)
    at = 0
    for r, n in enumerate(need):
        table[r, :n] = order[at:at + n]
        at += n
    where = table[token_req.long(), (positions // page_size).long()].long()
    pages[where.to(DEV), 0, 0, (positions % page_size).long().to(DEV)] = rows
    indptr = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    step = ops.latent_prompt_tokens()
    tiles = [(r, row) for r, n in enumerate(lens) for row in range(0, n, step)]
    tile_req, tile_row = (torch.tensor(x, dtype=torch.int32, device=DEV) for x in zip(*tiles))
    queries, c, k_rot = (torch.empty(T, n, device=DEV, dtype=bf) for n in (H * (D + 64), rank, 64))
    ops.latent_prompt_rows(q, inv_freq, positions.to(DEV), token_req.to(DEV), table.to(DEV), pages, page_size, queries, c, k_rot, H, D, R, R)
    assert torch.equal(c, rows[:, :rank]) and torch.equal(k_rot[:, :R], rows[:, rank:]) and not k_rot[:, R:].any()
    keys, values = torch.empty(T, H * D, device=DEV, dtype=bf), torch.empty(T, H * V, device=DEV, dtype=bf)
    ops.gemm_tc(c, uk, keys, None, ops.EPI_STORE_BF16)
    ops.gemm_tc(c, uv, values, None, ops.EPI_STORE_BF16)
    out = torch.full((T, H * V), float("nan"), device=DEV, dtype=bf)
    scale = (D + R) ** -0.5
    ops.latent_prompt(queries, keys, k_rot, values, indptr, tile_req, tile_row, len(tiles), out, H, D, R, V, scale)
    assert ops.latent_prompt_error() == 0
    x = q.double().view(T, H, D + R)
    angle = positions.to(DEV).double()[:, None, None] * inv_freq.double()
    a, b = x[..., D:D + R // 2], x[..., D + R // 2:]
    turned = torch.cat((a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()), -1)
    got = queries.double().view(T, H, D + 64)
    assert (got[..., D:D + R] - turned).abs().max() <= 2.0 ** -8 * turned.abs().max() and not got[..., D + R:].any()
    for r, n in enumerate(lens):
        s = slice(int(indptr[r]), int(indptr[r + 1]))
        kept = rows[s].double()
        k = torch.einsum("sc,hdc->hsd", kept[:, :rank], uk.double().view(H, D, rank))
        v = torch.einsum("sc,hvc->hsv", kept[:, :rank], uv.double().view(H, V, rank))
        score = torch.einsum("thd,hsd->hts", x[s, :, :D], k) + torch.einsum("thr,sr->hts", turned[s], kept[:, rank:])
        score = (score * scale).masked_fill(torch.ones(n, n, device=DEV).triu(1).bool(), -math.inf)
        want = (torch.softmax(score, -1) @ v).transpose(0, 1).reshape(n, H * V)
        assert (out[s].double() - want).abs().max() <= 2e-2 * want.abs().max()


def latent_setup(H, rank, rot, page_size, num_pages, dtype):
    pages = torch.full((num_pages, 1, 1, page_size, rank + rot), float("nan"), device=DEV, dtype=dtype)
    return pages


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rank,rot,page_size,far", [(40, 8, 16, 15), (64, 16, 16, 16), (22, 6, 8, 3), (128, 32, 32, 31),
                                                    (24, 4, 16, 0)])
def test_latent_attention_finds_one_far_key(dtype, rank, rot, page_size, far):
    """700 cached rows in shuffled pages of a pool that is otherwise NaN; the query of every head
    points at ONE row far back (at, or next to, a page's border): the output is that row."""
    from torchlet_b200 import ops

    H, n = 3, 700
    dk = rank + rot
    num_pages = -(-n // page_size) + 5
    pages = latent_setup(H, rank, rot, page_size, num_pages, dtype)
    order = torch.randperm(num_pages - 1, generator=torch.Generator().manual_seed(1))[: -(-n // page_size)] + 1
    rows = rand(n, dk, seed=2, scale=0.02)  # every other row scores 60 * N(0, 0.02): far below 60
    rows[far] = rand(dk, seed=3, scale=1.0)
    rows[far] /= rows[far].norm()
    flat = pages.view(num_pages * page_size, dk)
    index = order.repeat_interleave(page_size)[:n] * page_size + torch.arange(n) % page_size
    flat[index.to(DEV)] = rows.to(DEV, dtype)
    table = torch.zeros(2, len(order) + 2, dtype=torch.int32, device=DEV)
    table[1, :len(order)] = order.to(DEV, torch.int32)
    q = (rows[far].to(dtype).float() * 60.0).repeat(H, 1)  # score of the far row: 60 |row|^2, of the others about 0
    q_abs = torch.stack([q, q]).to(DEV, dtype).contiguous()  # two query tokens, the last and one in the middle
    positions = torch.tensor([n - 1, max(far, 350)], dtype=torch.int32, device=DEV)
    token_req = torch.tensor([1, 1], dtype=torch.int32, device=DEV)
    out = torch.empty(2, H * rank, device=DEV, dtype=dtype)
    ops.latent_attention(q_abs.view(2, H * dk), pages, table, token_req, positions, out, 2, H, dk, rank, page_size, 1.0)
    want = rows[far, :rank].to(dtype).float()
    got = out.float().cpu().view(2, H, rank)
    assert torch.isfinite(got).all()
    assert (got - want).abs().max() <= (2e-2 if dtype == torch.bfloat16 else 1e-3)
    # and a query BEFORE the far row must not see it: its output is far from that row
    if far > 0:
        positions = torch.tensor([far - 1, far - 1], dtype=torch.int32, device=DEV)
        ops.latent_attention(q_abs.view(2, H * dk), pages, table, token_req, positions, out, 2, H, dk, rank, page_size, 1.0)
        got = out.float().cpu().view(2, H, rank)
        assert torch.isfinite(got).all() and (got - want).abs().max() > 0.05


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,D,rot,dims,V,rank", [(3, 16, 8, 4, 24, 40), (1, 12, 6, 6, 10, 22), (4, 32, 16, 16, 32, 64)])
def test_latent_attention_kernels_against_expanded_keys_and_values(dtype, H, D, rot, dims, V, rank):
    """prepare, absorb_q, attention and expand_o together against attention over expanded keys and
    values: the latent-space form must give what the per-head keys and values give."""
    from torchlet_b200 import ops

    T, page_size, eps, base, scale, q_rank = 45, 8, 1e-5, 700.0, 0.3, 16
    mixer = {"heads": H, "dim": D, "rot_dim": rot, "vdim": V, "kv_rank": rank, "q_rank": q_rank, "scale": scale,
             "rot": {"base": base, "dims": dims}}
    shapes = {"dq": (q_rank, 56), "dq.norm": (q_rank,), "uq": (H * (D + rot), q_rank), "dkv": (rank + rot, 56),
              "dkv.norm": (rank,), "uk": (H * D, rank), "uv": (H * V, rank), "o": (56, H * V)}
    w = {}
    for i, (name, shape) in enumerate(shapes.items()):
        t = rand(*shape, seed=50 + i, scale=1.0 if len(shape) == 1 else 2.0 / math.sqrt(shape[-1]))
        w["m." + name] = (1 + 0.1 * t if name.endswith("norm") else t).bfloat16().float()
    h = rand(T, 56, seed=70)
    wd = {k: v.double() for k, v in w.items()}
    positions = torch.arange(T)
    kv = plain.latent_kv(h.double(), wd, "m.", mixer, eps, positions)
    want = plain.latent_attention(h.double(), wd, "m.", mixer, eps, positions, kv)

    dev = lambda name, dt=dtype: w["m." + name].to(DEV, dt).contiguous()
    down = (h.to(DEV) @ torch.cat([w["m.dq"], w["m.dkv"]]).to(DEV).T).contiguous()
    num_pages = -(-T // page_size) + 2
    pages = torch.full((num_pages, 1, 1, page_size, rank + rot), float("nan"), device=DEV, dtype=dtype)
    table = torch.arange(num_pages - 1, 0, -1, dtype=torch.int32, device=DEV).view(1, -1).contiguous()  # pages in reverse
    pos = positions.to(DEV, torch.int32)
    req = torch.zeros(T, dtype=torch.int32, device=DEV)
    i = torch.arange(dims // 2, dtype=torch.float64)
    inv_freq = (base ** (-2.0 * i / dims)).float().to(DEV)
    c_q = torch.empty(T, q_rank, device=DEV, dtype=dtype)
    ops.latent_prepare(down, q_rank, rank, rot, dims, dev("dq.norm", torch.float32), dev("dkv.norm", torch.float32),
                       inv_freq, eps, pos, req, table, pages, page_size, c_q, write_kv=True)
    q = (c_q.float() @ dev("uq", torch.float32).T).contiguous()
    q_abs = torch.empty(T, H * (rank + rot), device=DEV, dtype=dtype)
    ops.latent_absorb_q(q, dev("uk"), inv_freq, pos, q_abs, H, D, rot, dims, rank)
    o_lat = torch.empty(T, H * rank, device=DEV, dtype=dtype)
    ops.latent_attention(q_abs, pages, table, req, pos, o_lat, T, H, rank + rot, rank, page_size, scale)
    out = torch.empty(T, H * V, device=DEV, dtype=dtype)
    ops.latent_expand_o(o_lat, dev("uv"), out, H, V, rank)
    got = (out.float() @ dev("o", torch.float32).T).cpu().double()
    tol = 2e-5 if dtype == torch.float32 else 3e-2
    assert (got - want).abs().max() <= tol * want.abs().max()
    # the cache rows themselves: latent and rotated key part
    flat = pages.view(num_pages * page_size, rank + rot).float().cpu()
    where = (table[0].cpu().long()[positions // page_size]) * page_size + positions % page_size
    cached = flat[where].double()
    row_tol = 1e-5 if dtype == torch.float32 else 1e-2
    assert (cached[:, :rank] - kv[0]).abs().max() <= row_tol * kv[0].abs().max()
    assert (cached[:, rank:] - kv[1]).abs().max() <= row_tol * kv[1].abs().max()


@pytest.mark.parametrize("H,rank,rot", [(3, 48, 16), (16, 128, 16), (5, 144, 32), (8, 256, 32), (70, 64, 16), (4, 512, 64)])
def test_tensor_core_latent_attention_equals_the_plain_kernel(H, rank, rot):
    """The mma.sync kernel against the one-warp-a-row kernel on the same cache: prompt portions with
    a cached prefix, single tokens with their keys split over several CTAs, requests of unequal
    length in one step; pages shuffled, the rest of the pool NaN."""
    from torchlet_b200 import ops

    dk, page_size = rank + rot, 16
    assert ops.latent_attention_mma_supported(dk, rank)
    lens = [(130, 37), (0, 5), (700, 1), (63, 66)]  # (cached before, new tokens)
    total = sum(b + q for b, q in lens)
    num_pages = sum(-(-(b + q) // page_size) for b, q in lens) + 3
    pages = torch.full((num_pages, 1, 1, page_size, dk), float("nan"), device=DEV, dtype=torch.bfloat16)
    order = (torch.randperm(num_pages - 1, generator=torch.Generator().manual_seed(5)) + 1).tolist()
    width = max(-(-(b + q) // page_size) for b, q in lens)
    table = torch.zeros(len(lens), width, dtype=torch.int32)
    flat = pages.view(num_pages * page_size, dk)
    for r, (b, q) in enumerate(lens):
        n = -(-(b + q) // page_size)
        mine = [order.pop() for _ in range(n)]
        table[r, :n] = torch.tensor(mine)
        rows = rand(b + q, dk, seed=60 + r, scale=0.5).bfloat16()
        index = torch.tensor(mine).repeat_interleave(page_size)[:b + q] * page_size + torch.arange(b + q) % page_size
        flat[index.to(DEV)] = rows.to(DEV)
    T = sum(q for _, q in lens)
    q_abs = rand(T, H * dk, seed=70, scale=0.6).bfloat16().to(DEV)
    indptr = torch.tensor([0] + torch.tensor([q for _, q in lens]).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    before = torch.tensor([b for b, _ in lens], dtype=torch.int32, device=DEV)
    token_req = torch.cat([torch.full((q,), r, dtype=torch.int32) for r, (_, q) in enumerate(lens)]).to(DEV)
    positions = torch.cat([torch.arange(b, b + q, dtype=torch.int32) for b, q in lens]).to(DEV)
    table = table.to(DEV)
    want = torch.empty(T, H * rank, device=DEV, dtype=torch.bfloat16)
    ops.latent_attention(q_abs, pages, table, token_req, positions, want, T, H, dk, rank, page_size, 0.2)
    tile_req, tile_row = [], []
    for r, (_, q) in enumerate(lens):
        for row in range(0, q * H, 64):
            tile_req.append(r)
            tile_row.append(row)
    got = torch.full_like(want, float("nan"))
    ops.latent_attention_mma(q_abs, pages, table, indptr, before, torch.tensor(tile_req, dtype=torch.int32, device=DEV),
                             torch.tensor(tile_row, dtype=torch.int32, device=DEV), len(tile_req), got, T, H, dk, rank,
                             page_size, 0.2)
    assert torch.isfinite(got.float()).all()
    assert (got.float() - want.float()).abs().max() <= 2e-2 * want.float().abs().max()
    # single tokens, keys split over CTAs (more splits than some requests have key tiles)
    singles = [(700, 1), (5, 1), (64, 1), (255, 1)]
    sel = [0, 1, 3]  # requests of the cache above that are long enough: 167, 5 and 129 tokens hold
    lens1 = [(lens[0][0] + lens[0][1] - 1, 1), (lens[1][0] + lens[1][1] - 1, 1), (lens[3][0] + lens[3][1] - 1, 1), (700, 1)]
    reqs = [0, 1, 3, 2]
    T1 = len(reqs)
    q1 = rand(T1, H * dk, seed=71, scale=0.6).bfloat16().to(DEV)
    table1 = table[torch.tensor(reqs, device=DEV)].contiguous()
    indptr1 = torch.arange(T1 + 1, dtype=torch.int32, device=DEV)
    before1 = torch.tensor([b for b, _ in lens1], dtype=torch.int32, device=DEV)
    req1 = torch.arange(T1, dtype=torch.int32, device=DEV)
    want1 = torch.empty(T1, H * rank, device=DEV, dtype=torch.bfloat16)
    ops.latent_attention(q1, pages, table1, req1, before1, want1, T1, H, dk, rank, page_size, 0.2)
    for splits in (1, 3, 16):
        got1 = torch.full_like(want1, float("nan"))
        ops.latent_attention_mma(q1, pages, table1, indptr1, before1, None, None, T1 * (-(-H // 64)), got1, T1, H, dk,
                                 rank, page_size, 0.2, splits)
        assert torch.isfinite(got1.float()).all(), splits
        assert (got1.float() - want1.float()).abs().max() <= 2e-2 * want1.float().abs().max(), splits


@pytest.mark.parametrize("tokens", [1, 8, 70, 300])
def test_clamped_glu_in_the_epilogue_of_the_product(tokens):
    """gate and up as one tensor-core product whose epilogue clamps and gates, against the plain
    formula on the same bfloat16 operands; many values lie beyond the limit on either side."""
    from torchlet_b200 import ops
    from torchlet_b200.parts import swiglu_bf16

    hidden, inter, limit = 64, 48, 0.9
    x = rand(tokens, hidden, seed=90).bfloat16()
    gate, up = rand(inter, hidden, seed=91, scale=0.3).bfloat16(), rand(inter, hidden, seed=92, scale=0.3).bfloat16()
    g = torch.clamp(x.double() @ gate.double().T, max=limit)
    u = torch.clamp(x.double() @ up.double().T, min=-limit, max=limit)
    want = g * torch.sigmoid(1.702 * g) * (u + 1.0)
    assert (x.double() @ gate.double().T > limit).any() and (x.double() @ up.double().T < -limit).any()
    out = torch.empty(tokens, inter, device=DEV, dtype=torch.bfloat16)
    ops.gemm_tc_glu(x.to(DEV), swiglu_bf16.interleave(gate.to(DEV), up.to(DEV)), out, limit, 1.702)
    assert (out.cpu().double() - want).abs().max() <= 1e-2 * want.abs().max()
