"""The hop list of a model: duplicates add, terms of amplitude zero are left
out of the streamed form and kept in the per-term form."""

import numpy as np
import pytest

from realspace_exatdiagonalization_py_b200.hamiltonian import _merge_terms


@pytest.mark.parametrize("terms,merged,amps,n_all", [
    ([], [], [], 0),
    ([(1, 2, 0.0), (2, 1, 0j), (1, 3, -0.0)], [], [], 3),
    ([(1, 2, 1.0), (1, 2, 0.5j), (2, 3, 0.0)], [(0, 1)], [1 + 0.5j], 3),
    # a sum that cancels stays: its parts differ at another boundary twist
    ([(1, 2, 1.0), (1, 2, -1.0), (3, 1, 2.0)], [(0, 1), (2, 0)], [0.0, 2.0], 3),
    ([(1, 2, 0.0), (1, 2, 3.0)], [(0, 1)], [3.0], 2),
])
def test_merged_terms(terms, merged, amps, n_all):
    begin, to, amp, _ = _merge_terms(terms, 3)
    got = [(i, int(to[k])) for i in range(3) for k in range(begin[i], begin[i + 1])]
    assert got == merged
    np.testing.assert_array_equal(amp, np.array(amps, dtype=np.complex128))
    assert len(_merge_terms(terms, 3, merge=False)[1]) == n_all
