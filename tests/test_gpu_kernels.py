"""Kernels whose work split depends on the sizes, at the edges of their tiles:
each against the oracle's restatement of the same definition."""

from fractions import Fraction

import numpy as np
import pytest

from oracle import port

pytestmark = pytest.mark.gpu


def _case(family, size, nf, theta=None, species=False):
    """(data, sector set, oracle catalog, perm0, eta) of one lattice."""
    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200 import models

    if family == "heisenberg":
        m = models.build_heisenberg_second_quantized_model(size[0], 1.0)
    elif family == "haldane":
        m = models.build_zero_flux_bosonic_fci_second_quantized_model(sample_size=list(size))
    elif family == "checkerboard":
        m = models.build_zero_flux_fermionic_fci_second_quantized_model(sample_size=list(size))
    else:
        m = models.build_spinful_hubbard_second_quantized_model(list(size), 1.0, 4.0)
    if theta is not None and family != "hubbard":
        ed.update_second_quantized_model_with_twisted_phases(m, twisted_phases_over_2π=list(theta))
    G = ed.build_translation_group(m.lattice, theta)
    sp = models.hubbard_spin_species(m, nf // 2) if species else None
    data = ed.build_ed_data(m, filling_fraction=Fraction(nf, m.lattice.n_site), symmetry_group=G, species=sp)
    perm0, eta = port.group_arrays(G)
    osp = None if sp is None else (sum(1 << (i - 1) for i in sp[0]), sp[1])
    cat = port.catalog(m.lattice.n_site, nf, perm0, eta, m.particle_statistics.name == "FERMIONIC", species=osp)
    return data, ed.SectorSet(data.orbit_catalog, data.irrep_list), cat, perm0, eta


def _vector(n, seed):
    rng = np.random.default_rng(seed)
    c = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    return c / np.linalg.norm(c)


# no particles, one, all sites taken, one empty; several chunks; more than 32
# sites (two sites per lane); fermions and twists with stabilizers
@pytest.mark.parametrize("family,size,nf,theta,sector", [
    ("haldane", (2, 3), 0, None, 0),
    ("haldane", (2, 3), 1, None, 1),
    ("haldane", (2, 3), 11, (0.2, 0.1), 0),
    ("haldane", (2, 3), 12, None, 0),
    ("heisenberg", (13, 1), 6, (0.3, 0.0), 5),
    ("checkerboard", (2, 3), 4, (0.25, 0.4), 2),
    ("checkerboard", (4, 4), 2, None, 9),
    ("checkerboard", (3, 6), 2, (0.1, 0.3), 4),
])
def test_one_body_density_sizes(family, size, nf, theta, sector, monkeypatch):
    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200 import _lib
    from realspace_exatdiagonalization_py_b200 import correlators as cr

    data, sset, cat, perm0, eta = _case(family, size, nf, theta)
    n = data.orbit_catalog.n_site
    fermion = family == "checkerboard"
    s = next(k % len(sset.dims) for k in range(sector, sector + len(sset.dims)) if sset.dims[k % len(sset.dims)])
    basis = ed.Symmetry_Sector_Basis(data.irrep_list[s], data.orbit_catalog, sset, s)
    c = _vector(basis.dim, 3)
    chi = np.asarray(data.irrep_list[s].values, dtype=np.complex128)
    orbits = port.sector_orbits(cat, chi)
    ref = port.obdm_orbitwise(cat, orbits, c, chi, perm0, eta, fermion, n, nf)
    rho = cr.one_body_density_matrix(basis, c)
    # entries are at most nf and sums of at most a few thousand terms
    np.testing.assert_allclose(rho, ref, atol=1e-12, rtol=0)
    np.testing.assert_array_equal(rho, cr.one_body_density_matrix(basis, c))
    # without room for the states' amplitudes: evaluated at every lookup
    lib = _lib.lib()
    monkeypatch.setattr(lib, "rsed_obdm_states_bytes", lambda n: 0)
    np.testing.assert_allclose(cr.one_body_density_matrix(basis, c), ref, atol=1e-12, rtol=0)


# one state, several blocks' worth of ranks, symmetric orbits (the sum over the
# group elements that reach a state), fermions, twists, two species
@pytest.mark.parametrize("family,size,nf,theta,species", [
    ("haldane", (2, 3), 0, None, False),
    ("haldane", (2, 3), 12, (0.2, 0.1), False),
    ("heisenberg", (16, 1), 8, (0.3, 0.0), False),
    ("checkerboard", (2, 3), 4, (0.25, 0.4), False),
    ("hubbard", (2, 3), 6, (0.15, 0.0), True),
])
def test_fock_amplitudes_sizes(family, size, nf, theta, species):
    import realspace_exatdiagonalization_py_b200 as ed

    data, sset, cat, perm0, eta = _case(family, size, nf, theta, species)
    fermion = family in ("checkerboard", "hubbard")
    for s in [k for k, d in enumerate(sset.dims) if d][:3]:
        basis = ed.Symmetry_Sector_Basis(data.irrep_list[s], data.orbit_catalog, sset, s)
        c = _vector(basis.dim, s)
        chi = np.asarray(data.irrep_list[s].values, dtype=np.complex128)
        ref = port.fock_expand(cat, port.sector_orbits(cat, chi), c, chi, perm0, eta, fermion)
        keys = np.array(sorted(ref), dtype=np.uint64)
        m, a = ed.expand_sector_state_to_fock_amplitudes(c, basis, as_dict=False)
        m, a = m.cpu().numpy().view(np.uint64), a.cpu().numpy()
        order = np.argsort(m)
        np.testing.assert_array_equal(m[order], keys)
        # unit vectors: a few ulps of the largest amplitude
        np.testing.assert_allclose(a[order], np.array([ref[int(k)] for k in keys]), atol=1e-14, rtol=0)
        dense = ed.expand_sector_state_to_fock_dense(c, basis).cpu().numpy()
        np.testing.assert_array_equal(dense[dense != 0], a)


def _check_catalog(cat, ref):
    np.testing.assert_array_equal(np.array(cat.representative_mask_list, dtype=np.uint64), ref["reprs"])
    np.testing.assert_array_equal(cat.rep_rank_table, ref["rep_rank"])
    np.testing.assert_array_equal(cat.rep_sym_table, ref["rep_sym"])
    assert [list(x) for x in cat.stabilizer_g_indices_list] == [list(x) for x in ref["stab_g"]]
    # both sides round a double within one ulp of the phase to float32
    a, b = cat.rep_amp_table, np.asarray(ref["rep_amp"], dtype=np.complex64)
    assert np.abs((a - b).view(np.float32)).max() <= 6e-8


# 32-bit and 64-bit images, one and eight ranks per thread (2^20 states and
# more), no particles, all sites taken, |G| that does not divide a block
@pytest.mark.parametrize("family,size,nf,theta", [
    ("haldane", (2, 3), 0, (0.2, 0.1)),
    ("haldane", (2, 3), 12, (0.2, 0.1)),
    ("heisenberg", (13, 1), 6, (0.3, 0.0)),
    ("checkerboard", (3, 3), 4, (0.25, 0.4)),
    ("checkerboard", (4, 4), 3, None),
    ("checkerboard", (3, 6), 3, (0.1, 0.3)),
    ("checkerboard", (3, 6), 6, (0.1, 0.3)),
    ("heisenberg", (23, 1), 11, None),
])
def test_catalog_sizes(family, size, nf, theta):
    data, _, cat, _, _ = _case(family, size, nf, theta)
    _check_catalog(data.orbit_catalog, cat)


def test_catalog_element_without_few_distances():
    """A reflection moves every site by another distance: images bit by bit."""
    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200 import models

    n, nf = 18, 9
    m = models.build_heisenberg_second_quantized_model(n, 1.0)
    ops = [ed.Symmetry_Operation("e", list(range(1, n + 1))), ed.Symmetry_Operation("r", list(range(n, 0, -1)))]
    G = ed.Finite_Symmetry_Group("reflection", ops, identity_idx=0)
    cat = ed.build_symmetry_orbit_catalog(second_quantized_model=m, n_filled=nf, symmetry_group=G,
                                          particle_statistics=m.particle_statistics)
    perm0, eta = port.group_arrays(G)
    _check_catalog(cat, port.catalog(n, nf, perm0, eta, False))


# rows of no, few and many entries (shorter and longer than the lanes of a row
# times their entries in flight), row counts off the block, 1 to 9 vectors in
# both layouts
@pytest.mark.parametrize("n,most,k", [(1, 1, 1), (31, 3, 2), (257, 40, 3), (1000, 90, 4), (1023, 200, 7), (300, 33, 9)])
def test_csr_products(n, most, k):
    import scipy.sparse as sp
    import torch

    from realspace_exatdiagonalization_py_b200.hamiltonian import DeviceCSR

    rng = np.random.default_rng(n)
    per = rng.integers(0, most + 1, n)
    rows = np.repeat(np.arange(n), per)
    cols = rng.integers(0, n, per.sum())
    vals = rng.standard_normal(per.sum()) + 1j * rng.standard_normal(per.sum())
    A = sp.csr_matrix((vals, (rows, cols)), shape=(n, n))
    x = rng.standard_normal((n, k)) + 1j * rng.standard_normal((n, k))
    dev = DeviceCSR(*(torch.from_numpy(a).cuda() for a in (rows, cols, vals)), n)
    tol = 1e-15 * (most + 1) * 20  # ulps of sums of `most` products of size about 10 at most
    xd = torch.from_numpy(x).cuda()
    if not per.sum():  # a matrix without entries has no buffers: refused
        with pytest.raises(ValueError):
            dev.matmat(xd)
        return
    np.testing.assert_allclose(dev.matmat(xd).cpu().numpy(), A @ x, atol=tol, rtol=0)
    np.testing.assert_allclose(dev.matmat(xd.conj()).cpu().numpy(), A @ x.conj(), atol=tol, rtol=0)
    np.testing.assert_allclose(dev.matvec(xd.T.contiguous()).T.cpu().numpy(), A @ x, atol=tol, rtol=0)
    np.testing.assert_allclose(dev.matvec(xd[:, 0].contiguous()).cpu().numpy(), A @ x[:, 0], atol=tol, rtol=0)


# the recurrence's kernels (Gram reduction, update) by what they have to leave:
# orthonormal blocks and the projected matrix V^H H V.  Uniform blocks of 2 and
# 4 on one and many sectors (full and part-filled rows of columns), a mixed
# batch, and a basis below the register forms' size
@pytest.mark.parametrize("n_site,blocks,prec", [
    (20, [2] * 8, 64), (20, [2] * 20, 32), (22, [4] * 3, 64), (22, [4] * 11, 32), (24, [4], 64), (24, [2], 64),
    (22, [4, 2, 4], 64), (16, [4] * 5, 64), (24, [2] * 3, 32), (22, [1] * 4, 64),
])
def test_block_recurrence(n_site, blocks, prec):
    import torch

    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200 import models
    from realspace_exatdiagonalization_py_b200.lanczos import LanczosBatch

    m = models.build_heisenberg_second_quantized_model(n_site, 1.0)
    data = ed.build_ed_data(m, filling_fraction=Fraction(n_site // 2, n_site),
                            symmetry_group=ed.build_translation_group(m.lattice))
    dm, sset = data._device()
    dm.build_projection(sset.sqrt_stab, precisions=(64, 32))
    secs = list(range(len(blocks)))
    b = LanczosBatch(dm, sset, secs, 1, ed.LanczosParams(block=max(blocks), precision=prec), block_sizes=blocks)
    b.load_start(None)
    b.start()
    n = 6
    b.iterate_span(n, False)
    V = b.V[: n + 1]
    P = b.P.cpu()
    HV = torch.empty_like(V)
    for s in range(n + 1):
        dm.apply_block(sset, b.col_sector, V[s], HV[s], 64)
    for i, (c0, k) in enumerate(zip(b.col0, blocks)):
        Q = torch.cat([V[s][:, c0: c0 + k] for s in range(n + 1)], 1)
        Z = torch.cat([HV[s][:, c0: c0 + k] for s in range(n + 1)], 1)
        G = (Q.conj().T @ Q).cpu()
        # a few ulps per Gram-Schmidt step, sums of up to 112,720 products
        assert (G - torch.eye(G.shape[0], dtype=G.dtype)).abs().max() < 2e-13
        T = (Q.conj().T @ Z).cpu()[:, : n * k]
        # the norm of H is below n_site; an FP32 product rounds at 6e-8 of it
        tol = 1e-12 * n_site if prec == 64 else 1e-6 * n_site
        assert (T - P[i, : (n + 1) * k, : n * k]).abs().max() < tol


# the restart at sizes of the register form: groups of instances, part-filled
# groups, instances that do not restart
@pytest.mark.parametrize("n_site,n_inst,block", [(20, 8, 2), (20, 20, 4), (22, 3, 4), (20, 17, 2)])
def test_restart_sizes(n_site, n_inst, block):
    import torch

    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200 import models
    from realspace_exatdiagonalization_py_b200.lanczos import S_RESTART_NB, LanczosBatch

    m = models.build_heisenberg_second_quantized_model(n_site, 1.0)
    data = ed.build_ed_data(m, filling_fraction=Fraction(n_site // 2, n_site),
                            symmetry_group=ed.build_translation_group(m.lattice))
    dm, sset = data._device()
    p = ed.LanczosParams(block=block, n_slots=12)
    b = LanczosBatch(dm, sset, list(range(n_inst)), 2, p)
    g = torch.Generator(device="cuda").manual_seed(3)
    b.V.copy_(torch.randn(b.V.shape, dtype=b.V.dtype, device="cuda", generator=g))
    b.ritz_vec.copy_(torch.randn(b.ritz_vec.shape, dtype=b.V.dtype, device="cuda", generator=g))
    nb_old = [13 - i % 3 for i in range(n_inst)]
    nb_old[1] = 0
    st = b.state.cpu()
    st[:, S_RESTART_NB] = torch.tensor(nb_old, dtype=torch.int32)
    b.state.copy_(st)
    want = b.V.clone()
    K = b.keep * block
    for i in range(n_inst):
        if nb_old[i]:
            c = slice(i * block, (i + 1) * block)
            old = torch.cat([b.V[s][:, c] for s in range(nb_old[i] - 1)], 1)
            new = old @ b.ritz_vec[i, : old.shape[1], :K]
            for s in range(b.keep):
                want[s][:, c] = new[:, s * block: (s + 1) * block]
            want[b.keep][:, c] = b.V[nb_old[i] - 1][:, c]
    b.restart()
    # sums of 48 products of size about 10 in another order
    assert (b.V - want).abs().max() < 1e-11


# fewer and more than 32 sites, fewer orbits than a warp takes, several blocks
@pytest.mark.parametrize("family,size,nf", [
    ("haldane", (2, 3), 0), ("haldane", (2, 3), 12), ("heisenberg", (18, 1), 9), ("checkerboard", (4, 4), 3),
    ("checkerboard", (3, 6), 3), ("checkerboard", (3, 7), 2),
])
def test_density_pairs_sizes(family, size, nf):
    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200 import correlators as cr

    data, sset, cat, _, _ = _case(family, size, nf)
    n = data.orbit_catalog.n_site
    s = next(k for k, d in enumerate(sset.dims) if d)
    basis = ed.Symmetry_Sector_Basis(data.irrep_list[s], data.orbit_catalog, sset, s)
    c = _vector(basis.dim, 5)
    masks = np.array([int(cat["reprs"][o]) for o in port.sector_orbits(cat, np.asarray(data.irrep_list[s].values))],
                     dtype=np.uint64)
    occ = ((masks[:, None] >> np.arange(n, dtype=np.uint64)) & np.uint64(1)).astype(float)
    ref = (occ * (np.abs(c) ** 2)[:, None]).T @ occ
    # sums of weights that add up to 1
    np.testing.assert_allclose(cr.density_pairs(basis, c), ref, atol=1e-14, rtol=0)


# the projection matvec by how the columns pair up: pairs (blocks of 2 and 4),
# pairs broken at one place, single columns, odd counts, more columns than one
# chunk, leading dimensions that do not hold whole segments; bases around the
# sizes where the default route changes, with orbits outside some sectors and
# (all sites taken) rows without a hop.  A non-finite value of x reaches the
# rows that H takes it to and no other.
@pytest.mark.parametrize("n_site,nf,blocks,ld", [
    (16, 8, [2] * 3, 6), (16, 16, [2], 2), (20, 10, [2] * 10, 20), (20, 10, [4] * 17, 68), (20, 10, [2, 1, 2, 2], 8),
    (20, 10, [1] * 5, 6), (24, 12, [2], 2), (24, 12, [2] * 5, 10), (24, 12, [4] * 5, 22), (24, 12, [3] * 3, 10),
    (24, 12, [2, 1, 1, 4], 8), (24, 12, [2] * 33, 68),
])
def test_projection_products(n_site, nf, blocks, ld):
    import torch

    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200 import models

    m = models.build_heisenberg_second_quantized_model(n_site, 1.0)
    data = ed.build_ed_data(m, filling_fraction=Fraction(nf, n_site),
                            symmetry_group=ed.build_translation_group(m.lattice))
    dm, sset = data._device()
    n = sum(blocks)
    cs = torch.tensor([i % sset.n_sectors for i, b in enumerate(blocks) for _ in range(b)], dtype=torch.int32,
                      device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(5)
    X = torch.randn(data.orbit_catalog.n_orbits, ld, dtype=torch.complex128, device="cuda", generator=gen)
    X[:, :n] *= (sset.member[:, None] >> cs[None, :].long()) & 1
    Xf = X.to(torch.complex64)
    want, want32 = torch.zeros_like(X), torch.zeros_like(X)
    dm.apply_block(sset, cs, X, want)  # without a table: on the fly
    dm.apply_block(sset, cs, Xf, want32, 32)
    top = max(1.0, want[:, :n].abs().max().item())
    dm.build_projection(sset.sqrt_stab, precisions=(64, 32))
    try:
        Xn = X.clone()
        Xn[0, 0] = complex("nan")
        Yn = torch.zeros_like(X)
        dm.apply_block(sset, cs, Xn, Yn, 64, 302)
        reached = torch.isnan(Yn[:, :n].real)
        for v in (0, 604, 616, 664):
            Y = torch.zeros_like(X)
            dm.apply_block(sset, cs, X, Y, 64, v)
            # the same products in another order: a few ulps of sums of up to 24 hops
            assert (Y[:, :n] - want[:, :n]).abs().max().item() < 1e-13 * top, v
            assert not Y[:, n:].any()
            dm.apply_block(sset, cs, Xn, Y, 64, v)
            assert torch.equal(torch.isnan(Y[:, :n].real), reached), v
        for v in (0, 408, 608, 632, 664):
            Y = torch.zeros_like(X)
            dm.apply_block(sset, cs, Xf, Y, 32, v)
            assert (Y[:, :n] - want32[:, :n]).abs().max().item() < 2e-6 * top, v
    finally:
        dm.drop_projection()


# the projected eigenproblem at the edges of its 16-row blocks, with clusters,
# exact degeneracies, zero rows (no reflector), decoupled parts and scales at
# which the Sturm minors leave their range.  The matrix is planted in P; a step
# on a basis of zeros but for its last block leaves all but the last block's
# column of it, and the eigen-solve of the full basis follows (no restart: none
# is allowed)
@pytest.mark.parametrize("block,slots,kind", [
    (1, 4, "random"), (1, 15, "random"), (1, 16, "random"), (1, 17, "graded"), (1, 33, "degenerate"),
    (2, 16, "random"), (2, 24, "large"), (2, 24, "small"), (2, 32, "random"), (3, 11, "degenerate"), (3, 16, "random"),
    (4, 12, "decoupled"), (4, 16, "random"), (4, 16, "diagonal"), (4, 16, "degenerate"), (4, 16, "graded"),
])
def test_projected_eigenproblem(block, slots, kind):
    import torch

    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200 import _lib, models
    from realspace_exatdiagonalization_py_b200.lanczos import S_NB, S_STATUS, LanczosBatch

    m = models.build_heisenberg_second_quantized_model(16, 1.0)
    data = ed.build_ed_data(m, filling_fraction=Fraction(1, 2), symmetry_group=ed.build_translation_group(m.lattice))
    dm, sset = data._device()
    b = LanczosBatch(dm, sset, [0, 1], 2, ed.LanczosParams(block=block, n_slots=slots, tol=0.0, max_restarts=0))
    b.load_start(None)
    b.start()
    M = slots * block
    rng = np.random.default_rng(M)
    P = torch.zeros_like(b.P)
    for i in range(2):
        A = rng.standard_normal((M, M)) + 1j * rng.standard_normal((M, M))
        if kind == "diagonal":
            A = np.diag(rng.standard_normal(M))
        elif kind == "degenerate":
            q, _ = np.linalg.qr(A)
            A = (q * np.repeat(np.arange((M + 3) // 4) - 5.0, 4)[:M]) @ q.conj().T
        elif kind == "graded":
            s = 10.0 ** -np.linspace(0, 12, M)
            A = A * s[:, None] * s[None, :]
        elif kind == "decoupled":
            A[: M // 2, M // 2:] = 0
            A[M // 2:, : M // 2] = 0
        elif kind in ("large", "small"):
            A = A * (1e60 if kind == "large" else 1e-60)
        P[i, :M, :M] = torch.from_numpy(A + A.conj().T)
    b.P.copy_(P)
    b.V[slots - 1].copy_(b.V[0])
    b.V[: slots - 1].zero_()
    st = b.state.cpu()
    st[:, S_NB] = slots
    b.state.copy_(st)
    b.iterate_span(1, True)
    if kind == "large":  # the step's own block is nothing beside the planted coupling: reported, not solved
        assert (b.status()[:, S_STATUS] == _lib.RSED_EBREAKDOWN).all()
        return
    K = b.keep * block
    for i in range(2):
        A = b.P[i, :M, :M].cpu().numpy()
        A = 0.5 * (A + A.conj().T)
        assert np.abs(A).max() > 0
        S = b.ritz_vec[i, :M, :K].cpu().numpy()
        th = b.ritz_val[i, :K].cpu().numpy()
        # a backward-stable reduction: a few ulps of the norm per row; the cluster
        # gap of the Gram-Schmidt, 1e-3 of the norm, loses three digits
        scale = np.linalg.norm(A, 2)
        np.testing.assert_allclose(th, np.linalg.eigvalsh(A)[:K], atol=1e-15 * M * scale, rtol=0)
        assert np.abs(A @ S - S * th).max() <= 1e-14 * M * scale
        assert np.abs(S.conj().T @ S - np.eye(K)).max() < 1e-11


# the FP64 refinement (Gram over the restart basis, residuals) of FP32 solves:
# even and odd blocks and bases, a mixed batch, more pairs than one group of
# four, by H's own action on the vectors
@pytest.mark.parametrize("n_site,blocks,nev,keep", [
    (16, [1], 1, 0), (16, [1, 1], 5, 7), (16, [2] * 3, 4, 0), (16, [3, 3], 3, 2), (16, [4, 2, 1], 2, 4), (16, [5], 6, 3),
    (16, [8], 8, 2), (18, [2] * 9, 9, 5), (20, [4] * 2, 4, 4),
])
def test_refinement_blocks(n_site, blocks, nev, keep):
    import torch

    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200 import models
    from realspace_exatdiagonalization_py_b200.lanczos import LanczosBatch

    m = models.build_heisenberg_second_quantized_model(n_site, 1.0)
    data = ed.build_ed_data(m, filling_fraction=Fraction(1, 2), symmetry_group=ed.build_translation_group(m.lattice))
    dm, sset = data._device()
    dm.build_projection(sset.sqrt_stab, precisions=(64, 32))
    slots = min(64 // max(blocks), 2 * (keep or 4) + 8)
    b = LanczosBatch(dm, sset, list(range(len(blocks))), nev,
                     ed.LanczosParams(block=max(blocks), n_slots=slots, keep_blocks=keep, precision=32),
                     block_sizes=blocks)
    b.load_start(None)
    b.start()
    b.run()
    b.rayleigh_ritz()
    U, res, th = b.ritz_vectors_orbit(), b.residuals(), b.ritz_val[:, :nev].cpu().numpy()
    ld = nev + nev % 2
    for i in range(len(blocks)):
        X = torch.zeros(U.shape[2], ld, dtype=torch.complex128, device="cuda")
        X[:, :nev] = U[i].T
        Y = torch.zeros_like(X)
        dm.apply_block(sset, torch.full((nev,), i, dtype=torch.int32, device="cuda"), X, Y)
        R = Y[:, :nev] - X[:, :nev] * torch.from_numpy(th[i]).cuda()
        # rounding of H (norm below n_site) on unit vectors
        assert np.abs(torch.linalg.norm(R, dim=0).cpu().numpy() - res[i]).max() < 1e-13 * n_site
        T = X[:, :nev].conj().T @ Y[:, :nev]
        assert (T - torch.diag(torch.from_numpy(th[i]).cuda())).abs().max().item() < 1e-13 * n_site


# a caller of the C interface may leave columns free: instances of one column in
# places of two or four, between full ones; they read as zero and stay so
@pytest.mark.parametrize("n_site,wide,blocks", [(20, 2, [1, 2] * 6), (20, 4, [4, 2, 3, 1] * 3), (24, 2, [1, 2, 1])])
def test_padded_column_layout(n_site, wide, blocks):
    import torch

    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200 import models
    from realspace_exatdiagonalization_py_b200.lanczos import S_STATUS, LanczosBatch

    m = models.build_heisenberg_second_quantized_model(n_site, 1.0)
    data = ed.build_ed_data(m, filling_fraction=Fraction(1, 2), symmetry_group=ed.build_translation_group(m.lattice))
    dm, sset = data._device()
    dm.build_projection(sset.sqrt_stab, precisions=(64,))
    n_inst, nev = len(blocks), 1
    b = LanczosBatch(dm, sset, list(range(n_inst)), nev, ed.LanczosParams(block=wide, n_slots=12))
    assert b.n_orb * n_inst >= 65536
    b.c.reserved &= ~16  # not packed
    b.inst_b.copy_(torch.tensor(blocks, dtype=torch.int32))
    used = torch.zeros(b.ld, dtype=torch.bool, device="cuda")
    for c0, k in zip(b.col0, blocks):
        used[int(c0): int(c0) + k] = True
    b.load_start(None)
    b.W[:, ~used] = 0
    b.start()
    b.iterate_span(12, True)  # with a restart
    assert not (b.status()[:, S_STATUS] < 0).any()
    assert not b.V[: b.keep + 1][:, :, ~used].any()
    n = b.keep
    HV = torch.empty_like(b.V[: n + 1])
    for s in range(n + 1):
        dm.apply_block(sset, b.col_sector, b.V[s], HV[s], 64)
    for i, (c0, k) in enumerate(zip(b.col0, blocks)):
        Q = torch.cat([b.V[s][:, c0: c0 + k] for s in range(n + 1)], 1)
        Z = torch.cat([HV[s][:, c0: c0 + k] for s in range(n + 1)], 1)
        G = (Q.conj().T @ Q).cpu()
        # a few ulps per Gram-Schmidt step and restart, sums of up to 112,720 products
        assert (G - torch.eye(G.shape[0], dtype=G.dtype)).abs().max() < 2e-13
        # the restart basis holds Ritz vectors
        T = (Q.conj().T @ Z).cpu()[: n * k, : n * k]
        assert (T - torch.diag(b.ritz_val[i, : n * k].cpu())).abs().max() < 1e-12 * n_site


# groups with some, none or only elements of few move distances, in both widths
# of the masks and with one and eight ranks per thread
@pytest.mark.parametrize("n,nf,kind", [
    (12, 6, "dihedral"), (18, 9, "dihedral"), (23, 11, "dihedral"), (23, 11, "reflection"), (18, 9, "shuffled"),
    (23, 11, "shuffled"), (36, 4, "reflection"), (36, 5, "shuffled"), (40, 5, "reflection"), (16, 16, "dihedral"),
])
def test_catalog_of_groups_with_many_distances(n, nf, kind):
    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200 import models

    if kind == "shuffled":  # a cyclic group on relabelled sites
        lab = np.random.default_rng(n).permutation(n)
        perms = [[0] * n for _ in range(n // 2)]
        for s in range(n // 2):
            for i in range(n):  # two cycles of n // 2 sites, a fixed site if n is odd
                c, k = divmod(i, n // 2)
                perms[s][lab[i]] = int(lab[i] if c == 2 else lab[c * (n // 2) + (k + s) % (n // 2)])
    else:
        turns = range(n) if kind == "dihedral" else [0]
        perms = [[(i + s) % n for i in range(n)] for s in turns] + [[(s - 1 - i) % n for i in range(n)] for s in turns]
    m = models.build_heisenberg_second_quantized_model(n, 1.0)
    G = ed.Finite_Symmetry_Group(kind, [ed.Symmetry_Operation(str(s), [v + 1 for v in p])
                                        for s, p in enumerate(perms)], identity_idx=0)
    cat = ed.build_symmetry_orbit_catalog(second_quantized_model=m, n_filled=nf, symmetry_group=G,
                                          particle_statistics=m.particle_statistics)
    perm0, eta = port.group_arrays(G)
    _check_catalog(cat, port.catalog(n, nf, perm0, eta, False))


# the projected eigenproblem where its counts leave their range inside a group
# of eight steps and at scales far from one: tridiagonal matrices of nearly equal
# diagonal entries and couplings from small to below the square root of the
# smallest number, diagonals on the interval's bisection points, large and small
# norms.  Planted as above; with two Gram-Schmidt passes the step takes nothing
# from P, so that its own block stays beside any scale
@pytest.mark.parametrize("block,slots,kind,size", [
    (1, 33, "clusters", 1e-8), (1, 33, "clusters", 1e-20), (2, 24, "clusters", 1e-70), (4, 16, "clusters", 1e-160),
    (4, 16, "clusters", 0.0), (1, 49, "dyadic", 1e-3), (4, 16, "dyadic", 1e-20), (2, 32, "dyadic", 0.0),
    (2, 24, "random", 1e60), (4, 16, "random", 1e100), (1, 20, "random", 1e60),
])
def test_projected_eigenproblem_ranges(block, slots, kind, size):
    import torch

    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200 import _lib, models
    from realspace_exatdiagonalization_py_b200.lanczos import S_NB, S_STATUS, LanczosBatch

    m = models.build_heisenberg_second_quantized_model(16, 1.0)
    data = ed.build_ed_data(m, filling_fraction=Fraction(1, 2), symmetry_group=ed.build_translation_group(m.lattice))
    dm, sset = data._device()
    b = LanczosBatch(dm, sset, [0, 1], 2, ed.LanczosParams(block=block, n_slots=slots, tol=0.0, max_restarts=0,
                                                           single_pass=False))
    b.load_start(None)
    b.start()
    M = slots * block
    rng = np.random.default_rng(M)
    P = torch.zeros_like(b.P)
    for i in range(2):
        if kind == "random":
            A = rng.standard_normal((M, M)) + 1j * rng.standard_normal((M, M))
            A = size * (A + A.conj().T)
        else:
            d = np.full(M, -30.0) if kind == "clusters" else -32.0 + rng.integers(0, 3, M) * 2.0 ** -4
            d[rng.permutation(M)[: M // 8]] = rng.uniform(-20, 20, M // 8)
            A = np.diag(d) + size * (np.diag(np.ones(M - 1), 1) + np.diag(np.ones(M - 1), -1))
        P[i, :M, :M] = torch.from_numpy(A)
    b.P.copy_(P)
    b.V[slots - 1].copy_(b.V[0])
    b.V[: slots - 1].zero_()
    st = b.state.cpu()
    st[:, S_NB] = slots
    b.state.copy_(st)
    b.iterate_span(1, True)
    K = b.keep * block
    for i in range(2):
        A = b.P[i, :M, :M].cpu().numpy()
        A = 0.5 * (A + A.conj().T)
        scale = np.linalg.norm(A, 2)
        assert scale > 20 and int(b.status()[i, S_STATUS]) != _lib.RSED_EBREAKDOWN
        S = b.ritz_vec[i, :M, :K].cpu().numpy()
        th = b.ritz_val[i, :K].cpu().numpy()
        # as for the cases above
        np.testing.assert_allclose(th, np.linalg.eigvalsh(A)[:K], atol=1e-15 * M * scale, rtol=0)
        assert np.abs(A @ S - S * th).max() <= 1e-14 * M * scale
        assert np.abs(S.conj().T @ S - np.eye(K)).max() < 1e-11


# the default route of columns that do not pair up, by the chunks it takes: up to
# 16, 17 to 32, a third chunk, a full 64, more; rows of few and of many hops, small
# and larger bases
@pytest.mark.parametrize("n_site,reach", [(18, 1), (20, 1), (22, 1), (22, 3), (24, 1), (24, 4)])
@pytest.mark.parametrize("n", [5, 16, 17, 21, 22, 32, 33, 40, 49, 64, 65, 100])
def test_projection_products_of_single_columns(n_site, reach, n):
    import torch

    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200 import models

    m = models.build_heisenberg_second_quantized_model(n_site, 1.0)
    data = ed.build_ed_data(m, filling_fraction=Fraction(1, 2), symmetry_group=ed.build_translation_group(m.lattice))
    sset = ed.SectorSet(data.orbit_catalog, data.irrep_list)
    terms = [(i + 1, (i + s * k) % n_site + 1, 0.5 / k) for i in range(n_site) for k in range(1, reach + 1)
             for s in (1, -1)]
    dm = ed.DeviceModel(data.orbit_catalog, terms, m.density_density_terms)
    dm.build_projection(sset.sqrt_stab, precisions=(64, 32))
    cs = torch.arange(n, dtype=torch.int32, device="cuda") % n_site
    ld = n + n % 2
    gen = torch.Generator(device="cuda").manual_seed(7)
    X = torch.randn(data.orbit_catalog.n_orbits, ld, dtype=torch.complex128, device="cuda", generator=gen)
    X[:, :n] *= (sset.member[:, None] >> cs[None, :].long()) & 1
    for prec, x, tol in ((64, X, 1e-13), (32, X.to(torch.complex64), 2e-6)):
        # on the fly, 32 columns at a time
        want = torch.zeros_like(X)
        for c in range(0, n, 32):
            w = min(32, n - c)
            xs = torch.zeros(x.shape[0], w + w % 2, dtype=x.dtype, device="cuda")
            xs[:, :w] = x[:, c: c + w]
            ys = torch.zeros_like(xs, dtype=torch.complex128)
            dm.apply_block(sset, cs[c: c + w].contiguous(), xs, ys, prec, 999)
            want[:, c: c + w] = ys[:, :w]
        Y = torch.zeros_like(X)
        dm.apply_block(sset, cs, x, Y, prec)
        top = max(1.0, want[:, :n].abs().max().item())
        # the same products in another order: a few ulps of sums of up to 50 hops
        assert (Y[:, :n] - want[:, :n]).abs().max().item() < tol * top
        assert not Y[:, n:].any()


# the tiled reduction in three groups (the blocks of a wave do not divide by it)
# and the restart in three: as above
@pytest.mark.parametrize("n_site,n_inst,block", [(20, 18, 4), (22, 24, 4), (22, 17, 4)])
def test_three_groups(n_site, n_inst, block):
    import torch

    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200 import models
    from realspace_exatdiagonalization_py_b200.lanczos import LanczosBatch

    m = models.build_heisenberg_second_quantized_model(n_site, 1.0)
    data = ed.build_ed_data(m, filling_fraction=Fraction(1, 2), symmetry_group=ed.build_translation_group(m.lattice))
    dm, sset = data._device()
    dm.build_projection(sset.sqrt_stab, precisions=(64,))
    p = ed.LanczosParams(block=block)
    b = LanczosBatch(dm, sset, [i % n_site for i in range(n_inst)], 1, p)
    b.load_start(None)
    b.start()
    b.iterate_span(p.n_slots, True)  # up to the restart
    n, K = b.keep, b.keep * block
    HV = torch.empty_like(b.V[:n])
    for s in range(n):
        dm.apply_block(sset, b.col_sector, b.V[s], HV[s], 64)
    for i in range(n_inst):
        c = slice(i * block, (i + 1) * block)
        Q = torch.cat([b.V[s][:, c] for s in range(n)], 1)
        Z = torch.cat([HV[s][:, c] for s in range(n)], 1)
        # a few ulps per Gram-Schmidt step and the restart; the restart basis holds Ritz vectors
        assert ((Q.conj().T @ Q).cpu() - torch.eye(K, dtype=Q.dtype)).abs().max() < 1e-12
        T = (Q.conj().T @ Z).cpu()
        assert (T - torch.diag(b.ritz_val[i, :K].cpu())).abs().max() < 2e-12 * n_site
