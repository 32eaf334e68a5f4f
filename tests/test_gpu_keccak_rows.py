"""Keccak-256 of fixed-width rows read in place, without index pairs."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


# around one and two 136-byte blocks, rows off word boundaries, a ragged last CTA, empty rows
@pytest.mark.parametrize("rows,width", [(1, 0), (3, 1), (129, 7), (1000, 20), (127, 135), (130, 136), (257, 137),
                                        (64, 271), (65, 272), (33, 273)])
def test_rows(gpu_lib, rows, width):
    rng = np.random.default_rng(rows * 1000 + width)
    msgs = rng.integers(0, 256, (rows, width), dtype=np.uint8)
    want = np.frombuffer(b"".join(O.keccak256(m.tobytes()) for m in msgs), np.uint8).reshape(rows, 32)
    assert np.array_equal(gpu_lib.keccak256_rows(msgs), want)
    assert np.array_equal(gpu_lib.keccak256_rows(msgs, chunk=max(1, rows // 3)), want)  # slices of the arrays
    if width:  # columns of a wider array
        wide = rng.integers(0, 256, (rows, width + 5), dtype=np.uint8)
        wide[:, 2:2 + width] = msgs
        assert np.array_equal(gpu_lib.keccak256_rows(wide[:, 2:2 + width]), want)
