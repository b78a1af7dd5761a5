"""The fold of a block's triangles (rust-sloth_gb300/csrc/fold.cuh) walks triangles of up to
1024 samples with the f32 row division of the direct walk (direct_walk): checked against the
integer division for every column count such a triangle can have."""
import numpy as np


def test_reciprocal_row_division_is_exact_at_fold_sizes():
    i = np.arange(0, 1100, dtype=np.int64)
    for cols in range(1, 1101):
        r = np.float32(1.0) / np.float32(cols)
        assert np.array_equal(((i.astype(np.float32) + np.float32(0.5)) * r).astype(np.int64), i // cols), cols
