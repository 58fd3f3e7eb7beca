"""Which lane of the gates' scan writes which chunk: host arithmetic of `recurrence.cu`, no GPU."""
import ctypes

import pytest

from tau_rs_b200.csrc import build


@pytest.mark.parametrize("tokens", [32, 64])
def test_every_chunk_has_one_writer(tokens):
    """Two lanes that write the same chunk start from different maxima, and which of them wins is undefined."""
    library = build.load_library("recurrence.cu", ("TAU_KEY_DIM=16",))
    first, behind = ctypes.c_int(), ctypes.c_int()
    for length in range(2201):
        written = []
        for lane in range(32):
            library.tau_recurrence_gate_piece(length, tokens, lane, ctypes.byref(first), ctypes.byref(behind))
            written += range(first.value, behind.value)
        assert written == list(range(-(-length // tokens))), length      # each chunk once, lanes in the order of the chunks
