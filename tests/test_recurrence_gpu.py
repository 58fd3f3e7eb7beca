"""The kernels of `linear_recurrence` at the sizes where they can go wrong, against the recurrence in 64-bit."""
import pytest
import torch

from tau_rs_b200.csrc import kernels

pytestmark = pytest.mark.gpu


def case(runs, heads, dim, vdim, exponential, silu, seed, slots=None, dtype=torch.bfloat16, forget=3.0):
    """q, k and v side by side, gates or decays, states of the slots, the step's bounds."""
    torch.manual_seed(seed)
    tokens, slots = sum(runs), slots or len(runs) + 2
    columns = heads * (2 * dim + vdim)
    rows = (torch.randn(tokens, columns + (-columns) % 8, device="cuda") * 0.7).to(dtype)
    gates = torch.cat([torch.randn(tokens, heads), forget + torch.randn(tokens, heads)], dim=1).cuda() if exponential else None
    decays = None if exponential else torch.linspace(0.0, 1.0, heads + 1)[1:].pow(0.1).cuda()
    per_head = (vdim + 1) * dim + 1 if exponential else vdim * dim
    state = torch.randn(slots, heads * per_head, device="cuda") * 0.5
    if exponential:
        state.view(slots, heads, per_head)[:, :, -1] = torch.rand(slots, heads, device="cuda")
    numbers = torch.randperm(slots)[: len(runs)].to(torch.int32).cuda()
    bounds = torch.tensor([0] + torch.tensor(runs).cumsum(0).tolist(), dtype=torch.int32).cuda()
    return rows, gates, decays, state, numbers, bounds


def walk(rows, gates, decays, state, numbers, bounds, heads, dim, vdim, exponential, silu, longest=None, shortest=0):
    k_end, v_end = 2 * heads * dim, heads * (2 * dim + vdim)
    out = torch.empty(rows.shape[0], heads * vdim, device="cuda")
    state, gates = state.clone(), None if gates is None else gates.clone()
    kernels.linear_recurrence(rows[:, : heads * dim], rows[:, heads * dim : k_end], rows[:, k_end:v_end], gates, decays, state, bounds, numbers, out, heads, dim, vdim,
                              exponential, 15.0, dim ** -0.5, silu, **({} if longest is None else {"longest": longest}), shortest=shortest)
    torch.cuda.synchronize()
    return out, state


def exact(rows, gates, decays, state, numbers, bounds, heads, dim, vdim, exponential, silu):
    act = (lambda x: x * torch.sigmoid(x)) if silu else (lambda x: x)
    wide = rows.double()
    q = act(wide[:, : heads * dim]).view(-1, heads, dim) * dim ** -0.5
    k = act(wide[:, heads * dim : 2 * heads * dim]).view(-1, heads, dim)
    v = act(wide[:, 2 * heads * dim : heads * (2 * dim + vdim)]).reshape(-1, heads, vdim)
    out, state = torch.zeros(rows.shape[0], heads, vdim, dtype=torch.float64, device="cuda"), state.double()
    if exponential:
        capped = 15.0 * torch.tanh(gates.double() / 15.0)
        log_in, log_forget = capped[:, :heads], torch.nn.functional.logsigmoid(capped[:, heads:])
    for index, slot in enumerate(numbers.tolist()):
        kept = state[slot].view(heads, -1)
        S = kept[:, : vdim * dim].view(heads, vdim, dim).clone()
        if exponential:
            n, m = kept[:, vdim * dim : -1].clone(), kept[:, -1].clone()
        for t in range(int(bounds[index]), int(bounds[index + 1])):
            if exponential:
                m_new = torch.maximum(log_forget[t] + m, log_in[t])
                keep, take = torch.exp(log_forget[t] + m - m_new), torch.exp(log_in[t] - m_new)
                S = keep[:, None, None] * S + v[t][:, :, None] * (take[:, None] * k[t])[:, None, :]
                n, m = keep[:, None] * n + take[:, None] * k[t], m_new
                out[t] = torch.einsum("hvd,hd->hv", S, q[t]) / (torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6)[:, None]
            else:
                S = decays.double()[:, None, None] * S + v[t][:, :, None] * k[t][:, None, :]
                out[t] = torch.einsum("hvd,hd->hv", S, q[t])
        state[slot] = torch.cat([S.reshape(heads, -1), n, m[:, None]], dim=1).reshape(-1) if exponential else S.reshape(-1)
    return out.view(rows.shape[0], -1), state


def off(found, wanted):
    return float((found.double() - wanted).norm() / wanted.norm())


def test_more_blocks_than_the_gpu_holds_at_once_read_the_normaliser_as_it_was():
    """Every block of a (sequence, head) starts from n and m; the one that writes them back must not be seen by those that begin after it."""
    sizes = dict(heads=8, dim=64, vdim=310, exponential=True, silu=False)
    inputs = case([1] * 96, seed=3, **sizes)
    wanted, wanted_state = exact(*inputs, **sizes)
    found, found_state = walk(*inputs, **sizes)
    assert off(found, wanted) < 1e-5 and off(found_state, wanted_state) < 1e-5


# One token, a chunk's edges, remainders, several chunks, and runs of very different lengths in one step; key widths of one to sixteen k-steps;
# value widths around the tile (15 columns beside the normaliser, 16 without).
RUNS = [[31], [32], [33, 1], [64, 65, 63], [1, 200, 2, 129], [700]]


@pytest.mark.parametrize("runs", RUNS, ids=str)
@pytest.mark.parametrize("heads, dim, vdim, exponential, silu", [(2, 256, 47, True, False), (3, 64, 15, True, False), (1, 16, 130, True, False), (3, 128, 32, False, True),
                                                                 (2, 48, 17, False, True), (2, 256, 33, False, False), (5, 96, 1, False, False)])
def test_runs_in_chunks(runs, heads, dim, vdim, exponential, silu):
    """The chunks' sums are 32-bit sums in another order: as close to 64 bits as the token walk, read-outs and states."""
    sizes = dict(heads=heads, dim=dim, vdim=vdim, exponential=exponential, silu=silu)
    inputs = case(runs, seed=sum(runs) + dim, **sizes)
    wanted, wanted_state = exact(*inputs, **sizes)
    chunked, chunked_state = walk(*inputs, **sizes, longest=kernels.RECURRENCE_CHUNKS_FROM)
    walked, walked_state = walk(*inputs, **sizes, longest=1)
    print(f"chunks {off(chunked, wanted):.1e} {off(chunked_state, wanted_state):.1e}, walk {off(walked, wanted):.1e} {off(walked_state, wanted_state):.1e}")
    assert off(chunked, wanted) < 2e-6 and off(chunked_state, wanted_state) < 2e-6      # a few units of 2^-24 per sum
    assert kernels.recurrence_status(dim) == 0


MIXED = [[1] * 40 + [130], [200] + [1] * 33 + [48, 47, 0, 64], [1] * 31 + [64] + [3] * 40 + [100, 1], [0, 49, 0]]


@pytest.mark.parametrize("runs", MIXED, ids=lambda runs: f"{len(runs)} runs")
@pytest.mark.parametrize("heads, dim, vdim, exponential, silu", [(2, 64, 47, True, False), (3, 64, 32, False, True)])
def test_long_runs_in_chunks_beside_single_tokens(runs, heads, dim, vdim, exponential, silu):
    """Every run by the kernel of its own length, whatever the caller said of the lengths; more sequences than a warp looks at once."""
    sizes = dict(heads=heads, dim=dim, vdim=vdim, exponential=exponential, silu=silu)
    inputs = case(runs, seed=len(runs), **sizes)
    wanted, wanted_state = exact(*inputs, **sizes)
    for longest, shortest in ((max(runs), min(runs)), (1 << 20, 0), (1 << 20, 1 << 20)):
        found, found_state = walk(*inputs, **sizes, longest=longest, shortest=shortest)
        assert off(found, wanted) < 2e-6 and off(found_state, wanted_state) < 2e-6      # as above
    assert kernels.recurrence_status(dim) == 0


@pytest.mark.parametrize("why", ["limit", "memory"])
def test_without_room_for_chunks_the_runs_are_walked(monkeypatch, why):
    sizes = dict(heads=2, dim=64, vdim=40, exponential=True, silu=False)
    inputs = case([300, 1, 90], seed=8, **sizes)
    walked, walked_state = walk(*inputs, **sizes, longest=1)
    chunked, _ = walk(*inputs, **sizes, longest=300)
    if why == "limit":
        monkeypatch.setattr(kernels, "RECURRENCE_MOST_WORKSPACE", 1 << 16)
    else:
        def full(*size, _empty=torch.empty, **options):
            if options.get("dtype") == torch.uint8 and size[0] > 1 << 16:
                raise torch.cuda.OutOfMemoryError
            return _empty(*size, **options)

        monkeypatch.setattr(torch, "empty", full)
    found, found_state = walk(*inputs, **sizes, longest=300)
    assert torch.equal(found, walked) and torch.equal(found_state, walked_state) and not torch.equal(chunked, walked)


@pytest.mark.parametrize("forget", [-20.0, 0.0, 12.0])
def test_chunks_under_strong_and_weak_forgetting(forget):
    """Log forget gates near -15 a token (products of gates vanish within a chunk) and near 0 (nothing is forgotten)."""
    sizes = dict(heads=2, dim=64, vdim=40, exponential=True, silu=False)
    inputs = case([300, 70], seed=9, forget=forget, **sizes)
    wanted, wanted_state = exact(*inputs, **sizes)
    found, found_state = walk(*inputs, **sizes, longest=300)
    walked, walked_state = walk(*inputs, **sizes, longest=1)
    print(f"chunks {off(found, wanted):.1e} {off(found_state, wanted_state):.1e}, walk {off(walked, wanted):.1e} {off(walked_state, wanted_state):.1e}")
    assert off(found, wanted) < 1e-5 and off(found_state, wanted_state) < 1e-5


@pytest.mark.parametrize("silu", [False, True])
def test_an_infinite_value_reaches_no_earlier_token_and_no_other_sequence(silu):
    sizes = dict(heads=2, dim=32, vdim=20, exponential=False, silu=silu)
    inputs = case([100, 90], seed=5, **sizes)
    clean, _ = walk(*inputs, **sizes, longest=100)
    inputs[0][50, 2 * 2 * 32 + 7] = float("inf")      # value 7 of head 0
    found, _ = walk(*inputs, **sizes, longest=100)
    assert off(found[:50], clean[:50].double()) < 1e-6 and torch.equal(found[100:], clean[100:])
    assert not torch.isfinite(found[50:100, 7]).any()
    assert off(found[:, 8:], clean[:, 8:].double()) < 1e-6
