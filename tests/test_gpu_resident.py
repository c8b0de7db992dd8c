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
