"""float32 attention on the tensor cores against its plain statement."""
import numpy as np
import pytest
import torch

import plain_kernels
from tau_rs_b200.csrc import kernels
from test_kernels_gpu import DEVICE, close, paged_setup, randn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_heads,n_kv_heads,head_dim,window", [(8, 2, 128, 0), (3, 3, 64, 0), (4, 1, 128, 50), (4, 2, 64, 130), (2, 1, 128, 3)])
def test_runs_of_tokens(n_heads, n_kv_heads, head_dim, window):
    """Whole prompts, continued runs, single tokens, tiles of 128 queries and pages cut anywhere; what lies behind a sequence's end is never read into a result, and
    an infinite value, whose pieces are not numbers, reaches no query before it."""
    lengths, new_counts = [70, 200, 257, 1, 128, 333], [70, 17, 257, 1, 128, 130]
    keys, values, rows, positions, token_seq = paged_setup(lengths, new_counts, n_kv_heads, head_dim, torch.float32, seed=72, pages=48)
    tokens = positions.shape[0]
    queries = randn(tokens, n_heads * head_dim, dtype=torch.float32, seed=73)
    cu = torch.tensor(np.concatenate([[0], np.cumsum(new_counts)]), dtype=torch.int32, device=DEVICE)
    starts = torch.tensor([l - n for l, n in zip(lengths, new_counts)], dtype=torch.int32, device=DEVICE)
    for index, length in enumerate(lengths):
        for place in range(length, ((length + 63) // 64) * 64):
            keys[int(rows[index, place // 64]), :, place % 64] = float("nan")
            values[int(rows[index, place // 64]), :, place % 64] = float("nan")
    values[int(rows[0, 0]), :, 20] = float("inf")      # position 20 of the first sequence
    found, wanted = torch.full_like(queries, float("nan")), torch.empty(tokens, n_heads * head_dim, dtype=torch.float32)
    kernels.attention_f32_tc(queries, keys, values, found, cu, starts, rows, n_heads, n_kv_heads, head_dim, head_dim ** -0.5, window)
    plain_kernels.attention_generic(queries.cpu(), keys.cpu(), values.cpu(), wanted, positions.cpu(), token_seq.cpu(), rows.cpu(),
                                    n_heads, n_kv_heads, head_dim, head_dim ** -0.5, window)
    reached = slice(20, 70 if not window else min(70, 20 + window))
    assert bool(torch.isinf(found[reached]).all())
    found[reached], wanted[reached] = 0.0, 0.0
    close(found, wanted, torch.float32)
    assert kernels.build.load_library("attention_f32_tc.cu").tau_attention_f32_tc_status() == 0


@pytest.mark.parametrize("n_heads,n_kv_heads,head_dim,window", [(3, 1, 128, 0), (2, 2, 64, 130), (2, 1, 128, 3)])
@pytest.mark.parametrize("ranges", [2, 4, 8])
def test_ranges_of_the_keys(n_heads, n_kv_heads, head_dim, window, ranges):
    """Fewer pages than ranges, ranges in which a query sees nothing, rows that are computed again because one range is not finite."""
    lengths, new_counts = [70, 200, 257, 1, 128, 900], [70, 17, 257, 1, 128, 130]
    keys, values, rows, positions, token_seq = paged_setup(lengths, new_counts, n_kv_heads, head_dim, torch.float32, seed=72, pages=48)
    queries = randn(positions.shape[0], n_heads * head_dim, dtype=torch.float32, seed=73)
    cu = torch.tensor(np.concatenate([[0], np.cumsum(new_counts)]), dtype=torch.int32, device=DEVICE)
    starts = torch.tensor([l - n for l, n in zip(lengths, new_counts)], dtype=torch.int32, device=DEVICE)
    values[int(rows[0, 0]), :, 20] = float("inf")      # position 20 of the first sequence
    found, wanted = torch.full_like(queries, float("nan")), torch.empty(queries.shape, dtype=torch.float32)
    kernels.attention_f32_tc(queries, keys, values, found, cu, starts, rows, n_heads, n_kv_heads, head_dim, head_dim ** -0.5, window, ranges)
    plain_kernels.attention_generic(queries.cpu(), keys.cpu(), values.cpu(), wanted, positions.cpu(), token_seq.cpu(), rows.cpu(),
                                    n_heads, n_kv_heads, head_dim, head_dim ** -0.5, window)
    reached = slice(20, 70 if not window else min(70, 20 + window))
    assert bool(torch.isinf(found[reached]).all())
    found[reached], wanted[reached] = 0.0, 0.0
    close(found, wanted, torch.float32)
    assert kernels.build.load_library("attention_f32_tc.cu").tau_attention_f32_tc_status() == 0
