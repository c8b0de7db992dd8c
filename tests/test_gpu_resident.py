"""Solvers that stay resident between calls, beside changes of what they read:
the catalog moved to another flux point in place, the table's weights for the
other precision added."""

from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _model(theta):
    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200 import models

    m = models.build_zero_flux_fermionic_fci_second_quantized_model(
        sample_size=[3, 4], params=dict(models.params_Sun_Gu_Katsura_Sarma))
    ed.update_second_quantized_model_with_twisted_phases(m, twisted_phases_over_2π=theta)
    return m, ed.build_translation_group(m.lattice, theta)


# 5 particles on 12 cells: no symmetric orbits, so the sectors are the same at
# every flux point
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("graph", [True, False])
def test_solver_follows_an_update_of_its_catalog(precision, graph):
    import realspace_exatdiagonalization_py_b200 as ed

    thetas = [[0.1, 0.2], [0.3, 0.05]]
    want = []
    for theta in thetas:
        m, G = _model(theta)
        data = ed.build_ed_data(m, filling_fraction=Fraction(5, 24), symmetry_group=G)
        want.append(ed.solve_sectors_batched(data, [0, 1, 2], nev=3, return_vectors=False))
    assert abs(want[0][0][0][0] - want[1][0][0][0]) > 1e-4
    m, G = _model(thetas[0])
    data = ed.build_ed_data(m, filling_fraction=Fraction(5, 24), symmetry_group=G)
    dm, sset = data._device()
    dm.build_projection(sset.sqrt_stab, precisions=(64, 32))
    sol = ed.BatchedSectorSolver(dm, sset, [0, 1, 2], 3, precision=precision, graph=graph)
    for k in (0, 0, 0, 1, 1, 0):  # the graphs are captured by the second solve
        m, G = _model(thetas[k])
        ed.update_orbit_stabilizer_phases(data.orbit_catalog, G, m.particle_statistics)
        dm.term_amp.copy_(ed.DeviceModel(data.orbit_catalog, m.bilinear_terms, m.density_density_terms).term_amp)
        vals, _ = sol.solve(None, vectors=False)
        for i in range(3):
            # residuals of 1e-10 and below, FP32 products refined in FP64
            np.testing.assert_allclose(vals[i], want[k][i][0], atol=1e-9, rtol=0)


@pytest.mark.parametrize("first,second", [(64, 32), (32, 64)])
def test_table_gains_the_other_precision(first, second):
    """A batch of the other precision adds its weights to the model's table;
    the arrays that the first batch's graphs read stay where they are."""
    import realspace_exatdiagonalization_py_b200 as ed

    m, G = _model([0.1, 0.2])
    data = ed.build_ed_data(m, filling_fraction=Fraction(5, 24), symmetry_group=G)
    dm, sset = data._device()

    def solve(prec):
        res = ed.solve_sectors_batched(data, [0, 1], nev=2, precision=prec, return_vectors=False)
        return np.array([res[s][0] for s in (0, 1)])

    dm.build_projection(sset.sqrt_stab, precisions=(first,))
    want = [solve(first) for _ in range(3)][-1]
    assert dm.proj[f"w{first}"] is not None
    held = {k: dm.proj[k].data_ptr() for k in ("rowptr", "cg", f"w{first}")}
    np.testing.assert_allclose(solve(second), want, atol=1e-9, rtol=0)
    assert dm.proj[f"w{second}"] is not None and set(dm.proj["precisions"]) == {32, 64}
    assert held == {k: dm.proj[k].data_ptr() for k in held}
    # the FP64 refinement of FP32 solves streams the added weights from here on
    np.testing.assert_allclose(solve(first), want, atol=1e-9 if first == 32 else 0, rtol=0)


def test_no_table_beyond_half_the_memory(monkeypatch):
    """The table is not made where it would take more than half the free
    memory, however small it is; the buffers are planned for what is left."""
    import torch

    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200 import models

    m = models.build_zero_flux_bosonic_fci_second_quantized_model(sample_size=[3, 4], params=models.params_DNSheng)
    G = ed.build_translation_group(m.lattice)
    total = torch.cuda.mem_get_info()[1]
    p = ed.LanczosParams(block=1, n_slots=8)
    vals = []
    for share in (1.9, 2.1):
        data = ed.build_ed_data(m, filling_fraction=Fraction(6, 24), symmetry_group=G)
        dm, _ = data._device()
        table = dm.projection_bytes((64,))
        monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (int(share * table), total))
        vals.append(ed.solve_sectors_batched(data, [0], nev=1, params=p, return_vectors=False)[0][0])
        assert (dm.proj is not None) == (share > 2)
    np.testing.assert_allclose(vals[0], vals[1], atol=1e-9, rtol=0)


def test_shared_table_of_other_hops():
    """A table is only shared between models with the same hops."""
    import torch

    import realspace_exatdiagonalization_py_b200 as ed

    m, G = _model([0.1, 0.2])
    data = ed.build_ed_data(m, filling_fraction=Fraction(5, 24), symmetry_group=G)
    dm, sset = data._device()
    dm.build_projection(sset.sqrt_stab, precisions=(64, 32))
    (i, j, t), *rest = m.bilinear_terms
    for terms, shared in [(m.bilinear_terms, True), (rest, False), ([(i, j, 0.0), *rest], False),
                          ([(i, j, 2 * t), *rest], True)]:
        other = ed.DeviceModel(data.orbit_catalog, terms, m.density_density_terms)
        cs = torch.arange(4, dtype=torch.int32, device="cuda")
        X = torch.randn(data.orbit_catalog.n_orbits, 4, dtype=torch.complex128, device="cuda")
        want, got = torch.empty_like(X), torch.empty_like(X)
        other.apply_block(sset, cs, X, want)
        other.build_projection(sset.sqrt_stab, precisions=(64,), share=dm.proj)
        assert (other.proj["cg"] is dm.proj["cg"]) == shared
        other.apply_block(sset, cs, X, got)
        # the same products in another order: sums of up to 60 hops of size about 5
        assert (got - want).abs().max().item() < 1e-12
