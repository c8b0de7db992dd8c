"""Batches that reach the streamed Gram-Schmidt kernels (16 to 32 columns, at
least 32,768 orbits, blocks that the tiled reduction does not take, or the
streamed update asked for): the route by the kernels that ran, the result by
what the recurrence has to leave (orthonormal blocks, the projected matrix)."""

from fractions import Fraction

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ring24():
    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200 import models

    m = models.build_heisenberg_second_quantized_model(24, 1.0)
    data = ed.build_ed_data(m, filling_fraction=Fraction(1, 2), symmetry_group=ed.build_translation_group(m.lattice))
    dm, sset = data._device()
    dm.build_projection(sset.sqrt_stab, precisions=(64,))
    return dm, sset


def _kernels(run):
    """Names of the kernels that ``run`` launched."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    with profile(activities=[ProfilerActivity.CUDA]) as p:
        run()
        torch.cuda.synchronize()
    return " ".join(e.key for e in p.key_averages())


# the block bound rounded up to 1, 2, 4 and 8; the fewest and the most columns;
# mixed blocks; slots of one and several per warp
@pytest.mark.parametrize("blocks,slots", [
    ([1] * 16, 16), ([1] * 20, 40), ([3] * 6, 16), ([3] * 10, 21), ([4, 2, 4, 2, 4], 16), ([2, 1] * 8, 12),
    ([5] * 4, 12), ([8] * 4, 8), ([2] * 8, 16), ([4] * 8, 16),
])
@pytest.mark.parametrize("single", [True, False])
@pytest.mark.parametrize("update", [True, False])
def test_streamed_recurrence(ring24, blocks, slots, single, update):
    import torch

    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200.lanczos import LanczosBatch

    dm, sset = ring24
    p = ed.LanczosParams(block=max(blocks), n_slots=slots, single_pass=single, stream_update=update)
    b = LanczosBatch(dm, sset, [i % 24 for i in range(len(blocks))], 1, p, block_sizes=blocks)
    b.load_start(None)
    b.start()
    n = min(slots - 1, 12)  # no restart falls due
    names = _kernels(lambda: b.iterate_span(n, False))
    tiled = not update and len(set(blocks)) == 1 and blocks[0] in (2, 4)
    if names:  # empty where another profiler holds the device's activity interface
        assert ("k_lz_gram_stream" in names) == (not tiled)
        assert ("k_lz_gram_tiles" in names) == tiled
        assert ("k_lz_update_stream" in names) == update
    V = b.V[: n + 1]
    P = b.P.cpu()
    HV = torch.empty_like(V)
    for s in range(n + 1):
        dm.apply_block(sset, b.col_sector, V[s], HV[s], 64)
    for i, (c0, k) in enumerate(zip(b.col0, blocks)):
        Q = torch.cat([V[s][:, c0: c0 + k] for s in range(n + 1)], 1)
        Z = torch.cat([HV[s][:, c0: c0 + k] for s in range(n + 1)], 1)
        G = (Q.conj().T @ Q).cpu()
        # a few ulps per Gram-Schmidt step, sums of 112,720 products, up to 12 steps
        assert (G - torch.eye(G.shape[0], dtype=G.dtype)).abs().max() < 1e-12
        T = (Q.conj().T @ Z).cpu()[:, : n * k]
        # the norm of H is below 24
        assert (T - P[i, : (n + 1) * k, : n * k]).abs().max() < 2e-12 * 24
