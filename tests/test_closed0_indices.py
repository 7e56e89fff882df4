"""k_c0_bucket's record index (closed0.cuh) restated in numpy, for face offsets that
overlap (a plan's offsets overwritten after it was made): the faces then count more
corners than the mesh has, and only the check against N keeps the records' index in
their array."""
import numpy as np
import pytest


def _bucket_indices(ptr, ids, nv):
    """(v, column start + arrival rank, column length) per corner, as the kernels form them."""
    n = ids.size
    cnt, rank = np.zeros(nv, np.int64), np.zeros(n, np.int64)
    for b, e in zip(ptr[:-1], ptr[1:]):
        if b < 0 or e > n or e - b < 3:             # rejected by k_c0_faces
            continue
        for c in range(b, e):
            rank[c] = cnt[ids[c]]
            cnt[ids[c]] += 1
    sptr = np.concatenate([[0], np.cumsum(cnt)])
    return sptr[ids] + rank, rank < cnt[ids]


@pytest.mark.parametrize("ptr,inside", [([0, 3, 6, 9, 12], True), ([0, 9, 3, 12, 12], False), ([0, 12, 0, 12, 12], False)])
def test_the_records_index_needs_the_check_against_n(ptr, inside):
    ids = np.array([0, 1, 2, 0, 3, 1, 0, 2, 3, 1, 3, 2])        # a tetrahedron
    index, in_column = _bucket_indices(np.array(ptr), ids, 4)
    assert bool(np.all(index[in_column] < ids.size)) == inside
    kept = in_column & (index < ids.size)                       # the kernel's rule
    assert np.all(index[kept] < ids.size)
    if inside:
        assert kept.all() and np.array_equal(np.sort(index), np.arange(ids.size))
