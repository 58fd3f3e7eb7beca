"""The gated delta rule in chunks and token by token, against the recurrence in 64-bit."""
import pytest
import torch

from tau_rs_b200.csrc import kernels

pytestmark = pytest.mark.gpu


def case(runs, heads, key_heads, dim, vdim, seed, decay=(0.9, 1.0)):
    torch.manual_seed(seed)
    tokens = sum(runs)
    q, k = torch.randn(tokens, key_heads, dim), torch.randn(tokens, key_heads, dim) + 0.3      # keys that are not orthogonal
    q, k = q / q.norm(dim=-1, keepdim=True) * dim ** -0.5, k / k.norm(dim=-1, keepdim=True)
    rows = torch.cat([q.flatten(1), k.flatten(1), torch.randn(tokens, heads * vdim), torch.zeros(tokens, 3)], dim=1).cuda()
    gates = torch.stack([torch.empty(tokens, heads).uniform_(*decay), torch.rand(tokens, heads)], dim=-1).cuda()
    kq = (q * k).sum(-1).cuda()
    state = (torch.randn(len(runs) + 2, heads * vdim * dim) * 0.3).cuda()
    numbers = torch.randperm(len(runs) + 2)[: len(runs)].to(torch.int32).cuda()
    bounds = torch.tensor([0] + torch.tensor(runs).cumsum(0).tolist(), dtype=torch.int32).cuda()
    return rows, gates, kq, state, numbers, bounds


def walk(rows, gates, kq, state, numbers, bounds, heads, key_heads, dim, vdim, longest, shortest=0):
    out, state = torch.empty(rows.shape[0], heads * vdim, device="cuda"), state.clone()
    kernels.delta_rule(rows, 0, key_heads * dim, 2 * key_heads * dim, gates, kq, state, bounds, numbers, out, heads, key_heads, dim, vdim, longest=longest, shortest=shortest)
    torch.cuda.synchronize()
    return out, state


def exact(rows, gates, kq, state, numbers, bounds, heads, key_heads, dim, vdim):
    wide, width = rows.double(), key_heads * dim
    q, k = (wide[:, at : at + width].view(-1, key_heads, dim).repeat_interleave(heads // key_heads, dim=1) for at in (0, width))
    v = wide[:, 2 * width : 2 * width + heads * vdim].view(-1, heads, vdim)
    out, state, gates = torch.zeros(rows.shape[0], heads, vdim, dtype=torch.float64, device="cuda"), state.double(), gates.double()
    for index, slot in enumerate(numbers.tolist()):
        S = state[slot].view(heads, vdim, dim).clone()
        for t in range(int(bounds[index]), int(bounds[index + 1])):
            S = gates[t, :, 0, None, None] * S
            update = gates[t, :, 1, None] * (v[t] - torch.einsum("hvd,hd->hv", S, k[t]))
            S = S + update[:, :, None] * k[t][:, None, :]
            out[t] = torch.einsum("hvd,hd->hv", S, q[t])
        state[slot] = S.reshape(-1)
    return out.view(rows.shape[0], -1), state


def off(found, wanted):
    return float((found.double() - wanted).norm() / wanted.norm())


# One token, a chunk's edges, remainders, several chunks, and runs of very different lengths in one step; key widths of one to eight k-steps, value
# widths around the tiles of 16 and 64 columns.
@pytest.mark.parametrize("runs", [[1], [31], [32], [33, 1], [64, 65, 63], [1, 200, 2, 129], [1500]], ids=str)
@pytest.mark.parametrize("heads, key_heads, dim, vdim", [(4, 2, 128, 128), (2, 2, 64, 17), (3, 1, 16, 70), (2, 1, 48, 16), (2, 2, 96, 1)])
def test_runs_in_chunks(runs, heads, key_heads, dim, vdim):
    """The chunks' sums are 32-bit sums in another order: as close to 64 bits as the token walk, read-outs and states."""
    sizes = dict(heads=heads, key_heads=key_heads, dim=dim, vdim=vdim)
    inputs = case(runs, seed=sum(runs) + dim, **sizes)
    wanted, wanted_state = exact(*inputs, **sizes)
    chunked, chunked_state = walk(*inputs, **sizes, longest=1 << 20)
    walked, walked_state = walk(*inputs, **sizes, longest=1)
    print(f"chunks {off(chunked, wanted):.1e} {off(chunked_state, wanted_state):.1e}, walk {off(walked, wanted):.1e} {off(walked_state, wanted_state):.1e}")
    assert off(chunked, wanted) < 2e-6 and off(chunked_state, wanted_state) < 2e-6      # a few units of 2^-24 per sum
    assert kernels.delta_rule_status(dim) == 0


@pytest.mark.parametrize("runs", [[1] * 40 + [130], [200] + [1] * 33 + [64, 63, 0, 65], [1] * 31 + [64] + [3] * 40 + [100, 1], [0, 65, 0]], ids=lambda runs: f"{len(runs)} runs")
def test_long_runs_in_chunks_beside_single_tokens(runs):
    """Every run by the kernel of its own length, whatever the caller said of the lengths; more sequences than a warp looks at once."""
    sizes = dict(heads=4, key_heads=2, dim=64, vdim=40)
    inputs = case(runs, seed=len(runs), **sizes)
    wanted, wanted_state = exact(*inputs, **sizes)
    for longest, shortest in ((max(runs), min(runs)), (1 << 20, 0), (1 << 20, 1 << 20)):
        found, found_state = walk(*inputs, **sizes, longest=longest, shortest=shortest)
        assert off(found, wanted) < 2e-6 and off(found_state, wanted_state) < 2e-6      # as above
    assert kernels.delta_rule_status(64) == 0


@pytest.mark.parametrize("why", ["limit", "memory"])
def test_without_room_for_chunks_the_runs_are_walked(monkeypatch, why):
    sizes = dict(heads=4, key_heads=2, dim=64, vdim=40)
    inputs = case([300, 1, 90], seed=8, **sizes)
    walked, walked_state = walk(*inputs, **sizes, longest=1)
    chunked, _ = walk(*inputs, **sizes, longest=300)
    if why == "limit":
        monkeypatch.setattr(kernels, "DELTA_MOST_WORKSPACE", 1 << 16)
    else:
        def full(*size, _empty=torch.empty, **options):
            if options.get("dtype") == torch.uint8 and size[0] > 1 << 16:
                raise torch.cuda.OutOfMemoryError
            return _empty(*size, **options)

        monkeypatch.setattr(torch, "empty", full)
    found, found_state = walk(*inputs, **sizes, longest=300)
    assert torch.equal(found, walked) and torch.equal(found_state, walked_state) and not torch.equal(chunked, walked)


def test_gates_that_start_on_four_bytes_are_walked():
    sizes = dict(heads=4, key_heads=2, dim=64, vdim=40)
    rows, gates, *rest = case([100], seed=3, **sizes)
    odd = torch.cat([gates.new_zeros(1), gates.flatten()])[1:].view(gates.shape)
    assert odd.data_ptr() % 8 == 4
    for found, wanted in zip(walk(rows, odd, *rest, **sizes, longest=100), walk(rows, gates, *rest, **sizes, longest=1)):
        assert torch.equal(found, wanted)


@pytest.mark.parametrize("decay", [(0.0, 1e-30), (0.0, 0.0), (1e-4, 0.3), (1.0, 1.0), (-1.0, 1.0), (-0.9, -0.8)])
def test_chunks_under_strong_and_no_decay(decay):
    sizes = dict(heads=2, key_heads=1, dim=64, vdim=40)
    inputs = case([300, 70], seed=9, decay=decay, **sizes)
    wanted, wanted_state = exact(*inputs, **sizes)
    found, found_state = walk(*inputs, **sizes, longest=300)
    walked, walked_state = walk(*inputs, **sizes, longest=1)
    print(f"chunks {off(found, wanted):.1e} {off(found_state, wanted_state):.1e}, walk {off(walked, wanted):.1e} {off(walked_state, wanted_state):.1e}")
    assert off(found, wanted) < 2e-6 and off(found_state, wanted_state) < 2e-6


@pytest.mark.parametrize("what", ["value", "key", "gate", "query"])
def test_what_is_no_number_reaches_no_earlier_token_and_no_other_sequence(what):
    sizes = dict(heads=2, key_heads=2, dim=32, vdim=20)
    inputs = case([100, 90], seed=5, **sizes)
    clean, _ = walk(*inputs, **sizes, longest=100)
    rows, gates = inputs[0], inputs[1]
    if what == "gate":
        gates[50, 0, 1] = float("nan")
    else:
        rows[50, {"value": 2 * 64 + 7, "key": 64 + 3, "query": 3}[what]] = float("inf") if what == "value" else float("nan")
    found, state = walk(*inputs, **sizes, longest=100)
    assert off(found[:50], clean[:50].double()) < 1e-6 and torch.equal(found[100:], clean[100:]) and torch.equal(found[:, 20:], clean[:, 20:])
    mine = found[:100, :20]
    if what == "value":
        assert not torch.isfinite(mine[50:, 7]).any() and bool(torch.isfinite(mine[:, 8:]).all())
    elif what == "query":
        assert not torch.isfinite(mine[50]).any() and bool(torch.isfinite(mine[51:]).all())
    else:
        assert not torch.isfinite(mine[50:]).any()


@pytest.mark.parametrize("dtype, out_dtype", [(torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16), (torch.float32, torch.float32)])
@pytest.mark.parametrize("taps, silu", [(2, True), (3, False), (4, True)])
def test_short_convolution_of_four_channels_and_eight_tokens(dtype, out_dtype, taps, silu):
    """Runs that start and end inside a thread's eight tokens, from a state that is not zero: the same bits as channel by channel (rows that do
    not start on whole pieces)."""
    from types import SimpleNamespace

    torch.manual_seed(taps)
    runs, channels = [5, 1, 2, 600, 3, 290, 1], 1612
    tokens = sum(runs)
    x = torch.randn(tokens, channels, device="cuda").to(dtype)
    apart = torch.zeros(tokens, channels + 1, device="cuda", dtype=dtype)
    apart[:, :channels] = x
    weight, bias = torch.randn(taps, channels, device="cuda"), torch.randn(channels, device="cuda")
    state = torch.randn(len(runs) + 1, taps - 1, channels, device="cuda")
    bounds = torch.tensor([0] + torch.tensor(runs).cumsum(0).tolist(), dtype=torch.int32).cuda()
    step = SimpleNamespace(token_seq=torch.repeat_interleave(torch.arange(len(runs)), torch.tensor(runs)).to(torch.int32).cuda(), cu_seqlens=bounds,
                           seq_slot=torch.randperm(len(runs) + 1)[: len(runs)].to(torch.int32).cuda(), n_seqs=len(runs), all_single=False)
    results = []
    for source in (x, apart[:, :channels]):
        kept, out = state.clone(), torch.empty(tokens, channels, device="cuda", dtype=out_dtype)
        kernels.short_conv(source, weight, bias, kept, step, out, silu=silu, update=True)
        results.append((out, kept))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


@pytest.mark.parametrize("rows, groups, width", [(1, 1, 4), (9, 3, 128), (5, 2, 132), (3, 7, 512), (2, 2, 1024), (700, 16, 128), (700, 2, 1024), (8, 1, 2048)])
@pytest.mark.parametrize("gate_dtype", [None, torch.float32, torch.bfloat16])
@pytest.mark.parametrize("normalize, silu", [(True, True), (False, False)])
def test_gated_norm_in_pieces(rows, groups, width, gate_dtype, normalize, silu):
    torch.manual_seed(rows + width)
    total = groups * width
    values, weight = torch.randn(rows, total, device="cuda"), torch.randn(total, device="cuda")
    gate = None if gate_dtype is None else torch.randn(rows, total + 8, device="cuda").to(gate_dtype)[:, 4 : 4 + total]
    wanted = values.double().view(rows, groups, width)
    if normalize:
        wanted = wanted / torch.sqrt((wanted * wanted).mean(-1, keepdim=True) + 1e-5)
    wanted = wanted.reshape(rows, total) * weight.double()
    if gate is not None:
        wanted = wanted * torch.sigmoid(gate.double()) * (gate.double() if silu else 1.0)
    for out_dtype, bound in ((torch.float32, 1e-6), (torch.bfloat16, 2.0 ** -8)):      # a few 32-bit roundings; one bfloat16 rounding
        out = torch.zeros(rows, total + 4, device="cuda", dtype=out_dtype)
        kernels.gated_group_norm(values, weight, gate, out[:, :total], groups, 1e-5, normalize, silu_gate=silu)
        assert bool(((out[:, :total].double() - wanted).abs() <= bound * wanted.abs() + 1e-30).all()) and not out[:, total:].any()
