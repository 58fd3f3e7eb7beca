"""Attention over cached latent rows on the tensor cores, at the sizes where it can go wrong, against 64-bit."""
import numpy as np
import pytest
import torch

import fasesun_models as fm
from helpers import relative_error
from tau_rs_b200 import Engine, StepEntry, load_model
from tau_rs_b200.csrc import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads, rank, rot", [(16, 512, 64), (1, 64, 32), (17, 128, 0), (33, 448, 64), (8, 512, 128), (5, 192, 96)])
@pytest.mark.parametrize("window, splits", [(0, 1), (0, 3), (70, 1), (70, 5)])
def test_tensor_core_kernel(heads, rank, rot, window, splits):
    """Heads around a block's 16, latents of one to eight tiles a warp, contexts around its 64 rows, ranges that are empty, a window that begins inside
    a page, sinks, an infinity behind the end of a sequence."""
    torch.manual_seed(heads + rank)
    lengths, width = [1, 63, 64, 65, 130, 300], rank + rot
    stride = 5
    pages = torch.randn(len(lengths) * stride, 64, width, device="cuda").to(torch.bfloat16)
    table = torch.randperm(len(lengths) * stride).view(len(lengths), stride).to(torch.int32).cuda()
    for index, length in enumerate(lengths):
        if length % 64:
            pages[int(table[index, length // 64]), length % 64 :] = float("inf")
    queries = torch.randn(len(lengths), heads, width, device="cuda").to(torch.bfloat16)
    sinks = torch.randn(heads, device="cuda")
    positions = torch.tensor([length - 1 for length in lengths], dtype=torch.int32).cuda()
    sequence = torch.arange(len(lengths), dtype=torch.int32).cuda()
    found = torch.full((len(lengths), heads, rank), float("nan"), device="cuda", dtype=torch.bfloat16)
    scale = width ** -0.5
    kernels.latent_attention(queries, pages, found, sinks, positions, sequence, table, heads, rank, rot, scale, window, splits)
    for index, length in enumerate(lengths):
        rows = pages[table[index].long()].reshape(-1, width)[:length].double()[max(0, length - window) if window else 0 :]
        scores = queries[index].double() @ rows.T * scale
        weights = torch.softmax(torch.cat([scores, sinks.double()[:, None]], dim=1), dim=1)[:, :-1]
        wanted = weights @ rows[:, :rank]
        # One bfloat16 rounding of the result, beside 32-bit sums.
        assert bool(((found[index].double() - wanted).abs() <= 2.0 ** -8 * wanted.abs() + 1e-5).all()), (index, float((found[index].double() - wanted).abs().max()))


@pytest.mark.parametrize("head_dim, value_columns", [(64, 64), (128, 128), (192, 128), (192, 192), (256, 240)])
@pytest.mark.parametrize("n_heads, n_kv_heads, window", [(3, 3, 0), (8, 2, 0), (5, 5, 100)])
def test_prefill_from_swizzled_pages(head_dim, value_columns, n_heads, n_kv_heads, window):
    """Pages whose rows lie as the kernel's tiles do, by bulk copies, against the same pages in order: the same bits; what lies behind a sequence's end is
    never read into a result, columns beyond `value_columns` are left alone."""
    torch.manual_seed(head_dim)
    lengths, stride = [1, 64, 65, 200, 700, 256], 11
    tokens = sum(lengths)
    pages = [torch.randn(len(lengths) * stride, n_kv_heads, 64, head_dim, device="cuda").to(torch.bfloat16) for _ in range(2)]
    table = torch.randperm(len(lengths) * stride).view(len(lengths), stride).to(torch.int32).cuda()
    for index, length in enumerate(lengths):
        if length % 64:
            for page in pages:
                page[int(table[index, length // 64]), :, length % 64 :] = float("nan")
    row = torch.arange(64, device="cuda")
    order = (torch.arange(head_dim // 8, device="cuda")[None, :] ^ (row & 7)[:, None])[:, :, None] * 8 + torch.arange(8, device="cuda")
    turned = [torch.empty_like(page).scatter_(3, order.reshape(64, head_dim).expand_as(page), page) for page in pages]
    queries = torch.randn(tokens, n_heads * head_dim, device="cuda").to(torch.bfloat16)
    bounds = torch.tensor([0] + torch.tensor(lengths).cumsum(0).tolist(), dtype=torch.int32).cuda()
    starts, sinks = torch.zeros(len(lengths), dtype=torch.int32, device="cuda"), torch.randn(n_heads, device="cuda")
    results = []
    for (keys, values), swizzled in ((pages, False), (turned, True)):
        out = torch.full((tokens, n_heads * head_dim), 7.0, device="cuda", dtype=torch.bfloat16)
        kernels.attention_prefill(queries, keys, values, out, bounds, starts, table, n_heads, n_kv_heads, head_dim, head_dim ** -0.5, window, sinks, value_columns, swizzled)
        results.append(out.view(tokens, n_heads, head_dim))
    assert torch.equal(results[0], results[1]) and bool((results[0][:, :, value_columns:] == 7.0).all()) and bool(torch.isfinite(results[0]).all())
    head, index = n_heads - 1, 4
    keys, values = (page[table[index].long(), head // (n_heads // n_kv_heads)].reshape(-1, head_dim)[: lengths[index]].double() for page in pages)
    mine = queries.view(tokens, n_heads, head_dim)[int(bounds[index]) : int(bounds[index + 1]), head].double()
    scores = mine @ keys.T * head_dim ** -0.5
    i, j = torch.arange(lengths[index], device="cuda")[:, None], torch.arange(lengths[index], device="cuda")[None, :]
    scores = scores.masked_fill((j > i) | ((j <= i - window) if window else torch.zeros_like(j > i)), float("-inf"))
    weights = torch.softmax(torch.cat([scores, sinks[head].double().expand(lengths[index], 1)], dim=1), dim=1)[:, :-1]
    wanted = (weights @ values)[:, :value_columns]
    found = results[1][int(bounds[index]) : int(bounds[index + 1]), head, :value_columns].double()
    assert float((found - wanted).norm() / wanted.norm()) < 6e-3      # weights and result rounded to bfloat16
    assert kernels.attention_prefill_status(head_dim) == 0


def test_prefill_into_an_output_that_starts_on_two_bytes():
    """The same bits as into one that starts on four: nothing asks an output for more than its elements' alignment."""
    torch.manual_seed(1)
    pages = [torch.randn(4, 2, 64, 80, device="cuda").to(torch.bfloat16) for _ in range(2)]
    queries, bounds = torch.randn(100, 160, device="cuda").to(torch.bfloat16), torch.tensor([0, 70, 100], dtype=torch.int32).cuda()
    starts, table = torch.tensor([0, 40], dtype=torch.int32).cuda(), torch.arange(4, dtype=torch.int32).cuda().view(2, 2)
    wide, wanted = torch.full((100 * 160 + 2,), 7.0, device="cuda", dtype=torch.bfloat16), torch.empty_like(queries)
    odd = wide[1:-1].view(100, 160)
    for out in (wanted, odd):
        kernels.attention_prefill(queries, *pages, out, bounds, starts, table, 2, 2, 80, 80 ** -0.5, 0)
    assert odd.data_ptr() % 4 == 2 and torch.equal(odd, wanted) and float(wide[0]) == 7.0 and float(wide[-1]) == 7.0


@pytest.mark.parametrize("n_heads, n_kv_heads, window, sink", [(3, 3, 0, True), (8, 2, 0, False), (5, 5, 100, True)])
def test_prefill_of_heads_whose_values_are_narrower(n_heads, n_kv_heads, window, sink):
    """Keys of 192 and values of 128 on the tcgen05 kernel: whole prompts and runs behind cached positions, tiles of 128 queries and pages of 64 keys cut
    anywhere; what lies behind a sequence's end or beside its values is never read into a result."""
    torch.manual_seed(n_heads)
    cached, lengths, stride, key_dim, value_dim = [0, 0, 63, 500, 0, 64], [1, 128, 65, 200, 700, 129], 12, 192, 128
    tokens = sum(lengths)
    keys, values = (torch.randn(len(lengths) * stride, n_kv_heads, 64, key_dim, device="cuda").to(torch.bfloat16) for _ in range(2))
    values[:, :, :, value_dim:] = float("nan")
    table = torch.randperm(len(lengths) * stride).view(len(lengths), stride).to(torch.int32).cuda()
    for index, (before, length) in enumerate(zip(cached, lengths)):
        if (before + length) % 64:
            for page in (keys, values):
                page[int(table[index, (before + length) // 64]), :, (before + length) % 64 :] = float("nan")
    queries = torch.randn(tokens, n_heads * key_dim, device="cuda").to(torch.bfloat16)
    bounds = torch.tensor([0] + torch.tensor(lengths).cumsum(0).tolist(), dtype=torch.int32).cuda()
    starts, sinks = torch.tensor(cached, dtype=torch.int32).cuda(), torch.randn(n_heads, device="cuda") if sink else None
    out = torch.full((tokens, n_heads * value_dim), 7.0, device="cuda", dtype=torch.bfloat16)
    kernels.attention_prefill_tc(queries, keys, values, out, bounds, starts, table, n_heads, n_kv_heads, key_dim, key_dim ** -0.5, window, sinks=sinks, value_dim=value_dim)
    for index, (before, length) in enumerate(zip(cached, lengths)):
        mine, total = slice(int(bounds[index]), int(bounds[index + 1])), before + length
        i, j = torch.arange(before, total, device="cuda")[:, None], torch.arange(total, device="cuda")[None, :]
        hidden = (j > i) | ((j <= i - window) if window else torch.zeros_like(j > i))
        for head in range(n_heads):
            k, v = (page[table[index].long(), head // (n_heads // n_kv_heads)].reshape(-1, key_dim)[:total].double() for page in (keys, values))
            scores = (queries.view(tokens, n_heads, key_dim)[mine, head].double() @ k.T * key_dim ** -0.5).masked_fill(hidden, float("-inf"))
            if sink:
                scores = torch.cat([scores, sinks[head].double().expand(length, 1)], dim=1)
            wanted = torch.softmax(scores, dim=1)[:, :total] @ v[:, :value_dim]
            found = out.view(tokens, n_heads, value_dim)[mine, head].double()
            assert float((found - wanted).norm() / wanted.norm()) < 6e-3, (index, head)      # weights and result rounded to bfloat16
    assert kernels.attention_prefill_tc_status(key_dim) == 0


@pytest.mark.parametrize("splits", [1, 3, 8])
def test_rows_that_were_cached_before_are_read_early(splits):
    """The same bits whether the kernel may ask for the cached rows before the kernels in front of it have finished or not: own rows at every place of a tile."""
    torch.manual_seed(splits)
    lengths, heads, rank, rot, stride = [1, 64, 65, 127, 128, 300, 449], 16, 512, 64, 8
    pages = torch.randn(len(lengths) * stride, 64, rank + rot, device="cuda").to(torch.bfloat16)
    table = torch.randperm(len(lengths) * stride).view(len(lengths), stride).to(torch.int32).cuda()
    queries = torch.randn(len(lengths), heads, rank + rot, device="cuda").to(torch.bfloat16)
    positions, sequence = torch.tensor([length - 1 for length in lengths], dtype=torch.int32).cuda(), torch.arange(len(lengths), dtype=torch.int32).cuda()
    results = []
    for early in (False, True):
        out = torch.empty(len(lengths), heads, rank, device="cuda", dtype=torch.bfloat16)
        kernels.latent_attention(queries, pages, out, torch.zeros(heads, device="cuda"), positions, sequence, table, heads, rank, rot, 0.05, 0, splits, cached_before=early)
        results.append(out)
    assert torch.equal(*results)


def leave_nan_in_shared_memory():
    """The kernel over pages and queries of NaN, four tiles to a block and more blocks than fit the GPU at once: what a later block of it does not write is NaN."""
    heads, rank, rot, tokens = 16, 512, 64, 512
    pages, queries = (torch.full(shape, float("nan"), device="cuda", dtype=torch.bfloat16) for shape in ((4, 64, rank + rot), (tokens, heads, rank + rot)))
    positions, sequence = torch.full((tokens,), 255, dtype=torch.int32, device="cuda"), torch.zeros(tokens, dtype=torch.int32, device="cuda")
    out = torch.empty(tokens, heads, rank, device="cuda", dtype=torch.bfloat16)
    kernels.latent_attention(queries, pages, out, None, positions, sequence, torch.arange(4, dtype=torch.int32, device="cuda")[None], heads, rank, rot, 0.05)
    assert bool(torch.isnan(out).all())


@pytest.mark.parametrize("splits", [2, 4, 8, 16])
@pytest.mark.parametrize("window", [0, 30])
def test_short_contexts_beside_a_long_one_read_nothing_stale(splits, window):
    """Ranges that end before the token's position and whose tile reaches over it: shared memory holds NaN from the run before, the results are those of 64 bits."""
    torch.manual_seed(splits)
    lengths, heads, rank, rot, stride = [*range(1, 18), 20, 35, 64, 65, 66, 100, 146, 218, 354, 2048], 16, 512, 64, 32
    pages = torch.randn(len(lengths) * stride, 64, rank + rot, device="cuda").to(torch.bfloat16)
    table = torch.randperm(len(lengths) * stride).view(len(lengths), stride).to(torch.int32).cuda()
    queries = torch.randn(len(lengths), heads, rank + rot, device="cuda").to(torch.bfloat16)
    positions, sequence = torch.tensor([length - 1 for length in lengths], dtype=torch.int32).cuda(), torch.arange(len(lengths), dtype=torch.int32).cuda()
    results = []
    for early in (False, True):
        leave_nan_in_shared_memory()
        out = torch.empty(len(lengths), heads, rank, device="cuda", dtype=torch.bfloat16)
        kernels.latent_attention(queries, pages, out, None, positions, sequence, table, heads, rank, rot, 0.05, window, splits, cached_before=early)
        results.append(out)
    for index, length in enumerate(lengths):
        rows = pages[table[index].long()].reshape(-1, rank + rot)[:length].double()[-window if window else 0 :]
        weights = torch.softmax(queries[index].double() @ rows.T * 0.05, dim=1)
        wanted = weights @ rows[:, :rank]
        assert float((results[1][index].double() - wanted).abs().max() / wanted.abs().max()) < 6e-3, length      # a result rounded to bfloat16 (2^-9)
    assert torch.equal(*results)


def test_decode_steps_of_unequal_requests_with_stale_shared_memory(tmp_path):
    """`Engine.step` over a long request and short ones: each as by itself, whatever an earlier kernel left in shared memory."""
    cfg = fm.config([fm.latent(heads=16, dim=16, rot_dim=64, vdim=32, q_rank=64, kv_rank=512, mlp=None)], width=128, vocab=64)
    fm.write_model(str(tmp_path), cfg, 5)
    engine = Engine(load_model(str(tmp_path), "bfloat16", "gpu"), 8192)
    prompts, steps = [1100, 83, 85, 19, 2], 12
    requests = [np.random.default_rng(index).integers(0, 64, size=prompt + steps).tolist() for index, prompt in enumerate(prompts)]

    def decode(which):
        slots = [engine.open_sequence() for _ in which]
        engine.step([StepEntry(slot, requests[index][: prompts[index]], [prompts[index] - 1]) for slot, index in zip(slots, which)])
        rows = []
        for step in range(steps):
            leave_nan_in_shared_memory()
            rows.append(engine.step([StepEntry(slot, [requests[index][prompts[index] + step]], [0]) for slot, index in zip(slots, which)]).float().cpu().clone())
        for slot in slots:
            engine.close_sequence(slot)
        return torch.stack(rows)

    together = decode(range(len(prompts)))
    assert bool(torch.isfinite(together).all())
    for index in range(len(prompts)):
        # The contexts are cut into other ranges: 32-bit sums in another order, then roundings to bfloat16.
        assert relative_error(together[:, index], decode([index])[:, 0]) < 2e-2, index


@pytest.mark.parametrize("wide", [False, True])
def test_gates_in_the_prefill_of_narrower_values(wide):
    """Whole tiles, ragged ones and single rows, rows of the gate apart: the results times the sigmoids, rounded once instead of twice."""
    torch.manual_seed(4)
    lengths, n_heads, key_dim, value_dim = [128, 1, 300, 129], 3, 192, 128
    tokens, columns = sum(lengths), n_heads * (value_dim if wide else 1)
    keys, values = (torch.randn(len(lengths) * 5, n_heads, 64, key_dim, device="cuda").to(torch.bfloat16) for _ in range(2))
    queries = torch.randn(tokens, n_heads * key_dim, device="cuda").to(torch.bfloat16)
    gate = torch.randn(tokens, columns + 24, device="cuda").mul(3.0).to(torch.bfloat16)[:, 16 : 16 + columns]
    table, starts = torch.arange(len(lengths) * 5, dtype=torch.int32, device="cuda").view(len(lengths), 5), torch.zeros(len(lengths), dtype=torch.int32, device="cuda")
    bounds = torch.tensor([0] + torch.tensor(lengths).cumsum(0).tolist(), dtype=torch.int32).cuda()
    plain, gated = (torch.full((tokens, n_heads * value_dim), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    for out, given in ((plain, None), (gated, gate)):
        kernels.attention_prefill_tc(queries, keys, values, out, bounds, starts, table, n_heads, n_heads, key_dim, key_dim ** -0.5, 0, value_dim=value_dim, head_gate=given)
    wanted = plain.double() * torch.sigmoid(gate.double()).repeat_interleave(1 if wide else value_dim, 1)
    assert bool(((gated.double() - wanted).abs() <= 2.0 ** -7 * wanted.abs() + 1e-30).all())      # half a step of bfloat16 in either
    assert kernels.attention_prefill_tc_status(key_dim) == 0


@pytest.mark.parametrize("n_heads, rotary, window, gate", [(1, 64, 0, None), (3, 32, 0, "wide"), (5, 0, 100, "head")])
def test_prompts_of_expanded_rows_without_copies(n_heads, rotary, window, gate):
    """Queries, keys and values where the products left them: the same bits as through pages of their own, and the same rows in the cache.  Sequences that begin anywhere in
    their neighbours' tiles; a sequence of NaN stays alone."""
    torch.manual_seed(n_heads)
    lengths, head_dim, rot, rank, value_dim = [1, 128, 65, 63, 200, 700, 2], 128, 64, 512, 128
    tokens, width, bad = sum(lengths), head_dim + rot, 3
    bounds = torch.tensor([0] + torch.tensor(lengths).cumsum(0).tolist(), dtype=torch.int32).cuda()
    positions = torch.cat([torch.arange(length) for length in lengths]).to(torch.int32).cuda()
    sequence = torch.repeat_interleave(torch.arange(len(lengths)), torch.tensor(lengths)).to(torch.int32).cuda()
    projected = torch.randn(tokens, n_heads * width + rank + rot + 8, device="cuda").to(torch.bfloat16)
    expanded = torch.randn(tokens, n_heads * (head_dim + value_dim), device="cuda").to(torch.bfloat16)
    projected[int(bounds[bad]) : int(bounds[bad + 1])] = float("nan")
    expanded[int(bounds[bad]) : int(bounds[bad + 1])] = float("nan")
    weight, frequencies, sinks = torch.rand(rank, device="cuda"), torch.rand(max(rotary // 2, 1), device="cuda"), torch.randn(n_heads, device="cuda")
    factors = None if gate is None else torch.randn(tokens, n_heads * (value_dim if gate == "wide" else 1), device="cuda").to(torch.bfloat16)
    starts, pages = torch.zeros(len(lengths), dtype=torch.int32, device="cuda"), -(-max(lengths) // 64)
    table = torch.arange(len(lengths) * pages, dtype=torch.int32, device="cuda").view(len(lengths), pages)
    results = []
    for in_rows in (False, True):
        own = projected.clone()
        q, down = own[:, : n_heads * width], own[:, n_heads * width : n_heads * width + rank + rot]
        cache, latents = torch.zeros(table.numel(), 64, rank + rot, device="cuda", dtype=torch.bfloat16), torch.empty(tokens, rank + (rot if in_rows else 0), device="cuda", dtype=torch.bfloat16)
        kernels.latent_prepare(down, weight, 1e-6, q, None, cache, frequencies, rotary, positions, sequence, table, n_heads, head_dim, rot, rank, True, latents, in_place=in_rows)
        out = torch.full((tokens, n_heads * value_dim), 7.0, device="cuda", dtype=torch.bfloat16)
        if in_rows:
            assert kernels.prefill_expanded_fits(q, down, head_dim, rot, rank, value_dim)
            kernels.attention_prefill_expanded(q, expanded, latents, out, bounds, starts, n_heads, head_dim, rot, value_dim, 0.05, window, sinks, factors)
        else:
            keys, values = (torch.empty(table.numel(), n_heads, 64, width, device="cuda", dtype=torch.bfloat16) for _ in range(2))
            queries = torch.empty(tokens, n_heads, width, device="cuda", dtype=torch.bfloat16)
            kernels.latent_expand(q, down, expanded, queries, keys, values, frequencies, rotary, positions, sequence, pages, n_heads, head_dim, rot, rank, value_dim)
            kernels.attention_prefill_tc(queries.view(tokens, -1), keys, values, out, bounds, starts, table, n_heads, n_heads, width, 0.05, window, sinks=sinks, value_dim=value_dim,
                                         head_gate=factors)
        results.append((out.view(torch.int16), cache.view(torch.int16), latents[:, :rank].reshape(-1).view(torch.int16)))
    good = torch.arange(len(lengths), device="cuda")[sequence.long()] != bad
    assert torch.equal(results[0][0][good], results[1][0][good]) and bool(torch.isfinite(results[1][0].view(torch.bfloat16)[good].float()).all())
    assert torch.equal(results[0][1], results[1][1]) and torch.equal(results[0][2], results[1][2])
    assert kernels.attention_prefill_tc_status(width) == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows, width, before, behind", [(1, 8, 8, 0), (5, 512, 640, 8), (3, 1000, 3, 2), (130, 1536, 2624, 0)])
def test_norm_of_rows_that_lie_apart(dtype, rows, width, before, behind):
    """A column range of a wider product: the bits of the same rows side by side, by 16 bytes at a time and one by one."""
    torch.manual_seed(width)
    wide, weight = torch.randn(rows, before + width + behind, device="cuda").to(dtype), torch.rand(width, device="cuda")
    apart, out, wanted = wide[:, before : before + width], torch.empty(rows, width, device="cuda", dtype=dtype), torch.empty(rows, width, device="cuda", dtype=dtype)
    kernels.rms_norm(apart, weight, 1e-6, out)
    kernels.rms_norm(apart.contiguous(), weight, 1e-6, wanted)
    if before % 8 == behind % 8 == 0:
        assert torch.equal(out, wanted)
    else:      # summed in another order: a step of the type here and there
        assert bool(((out - wanted).abs().float() <= (2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -20) * wanted.abs().float()).all())
