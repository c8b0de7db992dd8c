"""One-sector solves beside other work on the same operator: the projection
table they stream is their own, and a solve that leaves no room for it runs
on the fly."""

from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _heisenberg(n):
    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200 import models

    m = models.build_heisenberg_second_quantized_model(n, 1.0)
    return ed.build_ed_data(m, filling_fraction=Fraction(1, 2), symmetry_group=ed.build_translation_group(m.lattice))


def _operator(data, s):
    import realspace_exatdiagonalization_py_b200 as ed

    m = data.second_quantized_model
    dm, sset = data._device()
    basis = ed.Symmetry_Sector_Basis(data.irrep_list[s], data.orbit_catalog, sset, s)
    return ed.MatrixFreeHamiltonian(basis, m.bilinear_terms, m.density_density_terms, None, model=dm)


@pytest.mark.parametrize("precision", [64, 32])
def test_solve_leaves_the_model_as_it_was(precision):
    """No table stays behind: a block of odd leading dimension is still taken,
    and a batch of the other precision finds the weights it asks for."""
    import torch

    import realspace_exatdiagonalization_py_b200 as ed

    data = _heisenberg(16)
    dm, sset = data._device()
    ed.ed_scan_at_irrep_matrixfree(data.irrep_list[0].label, data, nev=2,
                                   params=ed.LanczosParams(precision=precision))
    assert dm.proj is None and dm.c.proj_rowptr is None
    cs = torch.zeros(3, dtype=torch.int32, device="cuda")
    X = torch.randn(data.orbit_catalog.n_orbits, 3, dtype=torch.complex128, device="cuda")
    X *= (sset.member[:, None] >> 0) & 1
    Y = torch.empty_like(X)
    dm.apply_block(sset, cs, X, Y)
    other = 32 if precision == 64 else 64
    ed.solve_sectors_batched(data, [0, 1], nev=2, precision=other, return_vectors=False)
    assert dm.proj[f"w{other}"] is not None


def test_operator_follows_an_update_of_its_catalog():
    """The operator of a solved sector reads the catalog as it is now."""
    import torch

    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200.lanczos import diagonalize_block_matrixfree

    data = _heisenberg(16)
    m, cat = data.second_quantized_model, data.orbit_catalog
    op = _operator(data, 1)
    diagonalize_block_matrixfree(op, op.n, nev=2)
    x = torch.randn(op.n, 2, dtype=torch.complex128, device="cuda")
    before = op.adjoint_device(x, 2)
    ed.update_orbit_stabilizer_phases(cat, ed.build_translation_group(m.lattice, [0.3, 0.0]), m.particle_statistics)
    after = op.adjoint_device(x, 2)
    fresh = ed.DeviceModel(cat, m.bilinear_terms, m.density_density_terms)
    want = ed.MatrixFreeHamiltonian(op.basis, m.bilinear_terms, m.density_density_terms, None,
                                    model=fresh).adjoint_device(x, 2)
    assert (before - want).abs().max().item() > 1e-3
    # the same products, at most in another order: sums of up to 16 hops of size about 5
    assert (after - want).abs().max().item() < 1e-13


def test_solve_where_only_the_basis_fits():
    """Device memory for the basis but not for the table beside it."""
    import torch

    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200.batched import APPLY_ON_THE_FLY

    data = _heisenberg(24)
    dm, _ = data._device()
    label = data.irrep_list[0].label
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    want, _ = ed.ed_scan_at_irrep_matrixfree(label, data, nev=1,
                                             params=ed.LanczosParams(apply_variant=APPLY_ON_THE_FLY))
    peak = torch.cuda.max_memory_reserved()
    table = dm.projection_bytes((64,))
    assert table > 16 << 20
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((peak + (8 << 20)) / total)
    try:
        got, _ = ed.ed_scan_at_irrep_matrixfree(label, data, nev=1)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
        torch.cuda.empty_cache()
    # both converged to 1e-10 of the energy
    np.testing.assert_allclose(got, want, atol=1e-8, rtol=0)


@pytest.mark.parametrize("error", ["memory", "limit"])
def test_solve_without_a_table(monkeypatch, error):
    """The table's two refusals: no memory for it, a model beyond its limits."""
    import torch

    import realspace_exatdiagonalization_py_b200 as ed

    def refuse(self, *a, **k):
        raise torch.cuda.OutOfMemoryError("no room") if error == "memory" else ValueError("beyond the limits")

    data = _heisenberg(16)
    label = data.irrep_list[2].label
    want, vecs = ed.ed_scan_at_irrep_matrixfree(label, data, nev=3)
    monkeypatch.setattr(ed.DeviceModel, "build_projection", refuse)
    got, _ = ed.ed_scan_at_irrep_matrixfree(label, data, nev=3)
    np.testing.assert_allclose(got, want, atol=1e-10, rtol=0)


def test_solves_from_two_threads():
    """Sectors of one model solved at the same time on streams of their own."""
    import threading

    import torch

    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200.lanczos import LanczosParams, _solve_sector

    data = _heisenberg(20)
    dm, sset = data._device()
    for s in range(4):
        sset.rows(s)
    want = [_solve_sector(dm, sset, s, 2, LanczosParams())[0] for s in range(4)]
    torch.cuda.synchronize()
    got, failed = {}, []

    def work(s):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(3):
                    got.setdefault(s, []).append(_solve_sector(dm, sset, s, 2, LanczosParams())[0])
        except Exception as e:  # reported by the main thread
            failed.append((s, e))

    threads = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for s in range(4):
        for v in got[s]:
            np.testing.assert_allclose(v, want[s], atol=1e-10, rtol=0)


@pytest.mark.parametrize("precision", [64, 32])
def test_solve_asks_for_no_memory_figure(monkeypatch, precision):
    """The free-memory query can stall for 100 ms: a solve with a small table
    does without it, and an FP32 one streams its refinement all the same."""
    import torch

    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200.batched import streaming_view

    def query(*a):
        raise AssertionError("free memory asked for")

    data = _heisenberg(16)
    dm, sset = data._device()
    monkeypatch.setattr(torch.cuda, "mem_get_info", query)
    ed.ed_scan_at_irrep_matrixfree(data.irrep_list[0].label, data, nev=2,
                                   params=ed.LanczosParams(precision=precision))
    assert streaming_view(dm, sset, precision).proj["precisions"] == ((64,) if precision == 64 else (32, 64))
