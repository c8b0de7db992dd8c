"""The calls of this package that are timed, with their inputs and exact results.

A case is one call of a user's program on one lattice: building a catalog,
moving a catalog to another flux point, applying the Hamiltonian, solving
sectors, and the observables that read the solved states.  Lattices, fillings
and couplings are those of the package's models and tests (16-site Heisenberg
ring to the 32-site Haldane lattice); the seed moves the couplings by up to
10 %, draws the boundary twists and the vectors.

``exact`` restates each result in plain torch with 64-bit arithmetic over the
full fixed-filling space; it uses the package only for the model's term lists
and the lattice geometry.
"""

import math
import random
from fractions import Fraction

import numpy as np
import torch

import realspace_exatdiagonalization_py_b200 as ed
from realspace_exatdiagonalization_py_b200 import models

# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------


def _case(kind, family, a, b, nf, **more):
    c = {"kind": kind, "family": family, "a": a, "b": b, "nf": nf, "flux": False, "sector": 0, "cols": 1, "nev": 4,
         "precision": 64, "block": 0, "slots": 0}
    c.update(more)
    return c


def listed():
    return [
        # one product inside a user's own iterative method on the 24-site
        # checkerboard (892 rows): the smallest call, launch and host latency
        dict(_case("operator", "checkerboard", 3, 4, 4, sector=5), name="operator-24"),
        # the same at the largest size the reference reaches (657,756 rows)
        dict(_case("operator", "haldane", 4, 4, 8, sector=1), name="operator-32"),
        # two columns in each of the 16 sectors: the FP64 product of the
        # refinement and of FP64 block solves
        dict(_case("block", "haldane", 4, 4, 8, cols=2), name="block-32"),
        # the catalog of a new lattice: a small ring, and 10.5 million states
        dict(_case("catalog", "heisenberg", 16, 1, 8, flux=True), name="catalog-16"),
        dict(_case("catalog", "haldane", 4, 4, 8, flux=True), name="catalog-32"),
        # the catalog's copy at the next point of a flux grid
        dict(_case("flux", "haldane", 4, 4, 8, flux=True), name="flux-32"),
        # all 12 sectors of the 24-site checkerboard, as ed_scan solves them
        dict(_case("solve", "checkerboard", 3, 4, 4, nev=6), name="solve-24"),
        # all 16 sectors of the 32-site Haldane lattice, FP32 products and FP64
        # refinement, in the configuration the autotuner picks for this batch
        dict(_case("solve", "haldane", 4, 4, 8, nev=4, precision=32, block=2, slots=12), name="solve-32"),
        # one point of a flux scan: catalog moved, all sectors solved once
        dict(_case("scan", "haldane", 3, 4, 6, nev=3, flux=True), name="scan-24"),
        # the ground state of one sector, as the reference's benchmark asks
        dict(_case("single", "heisenberg", 24, 1, 12, nev=1), name="single-24"),
        # one point of a Chern-number grid: two states expanded, their links
        dict(_case("chern", "haldane", 4, 4, 8, flux=True), name="chern-32"),
        # off-diagonal order and structure factor of one state
        dict(_case("correlators", "haldane", 4, 4, 8, sector=0), name="correlators-32"),
    ]


def _lattices():
    """(family, a, b, nf, states, |G|) of the lattices and fillings in use."""
    out = []
    for n in range(12, 27):
        out.append(("heisenberg", n, 1, n // 2, math.comb(n, n // 2), n))
    cells = [(2, 3), (2, 4), (3, 3), (2, 5), (3, 4), (2, 6), (2, 7), (3, 5), (4, 4)]
    for a, b in cells:
        n = 2 * a * b
        for nf in sorted({a * b // 2, a * b // 3, a * b // 3 + 1, 3, 5}):
            for family in ("haldane", "dnsheng", "checkerboard"):
                out.append((family, a, b, nf, math.comb(n, nf), a * b))
    for a, b in [(2, 3), (2, 4), (3, 3), (2, 5), (3, 4)]:
        for nf in (a * b, a * b - 1, 4, 7):  # up and down electrons as equal as can be
            out.append(("hubbard", a, b, nf, math.comb(a * b, nf // 2) * math.comb(a * b, nf - nf // 2), a * b))
    return out


# states of the catalogs that each kind of call is drawn on; a solve costs
# hundreds of products, so its catalogs are smaller than those of one pass
_RANGE = {"operator": (500, 10_600_000), "block": (2_000, 10_600_000), "catalog": (500, 10_600_000),
          "flux": (500, 10_600_000), "solve": (5_000, 300_000), "scan": (5_000, 300_000), "single": (5_000, 1_500_000),
          "chern": (2_000, 10_600_000), "correlators": (2_000, 10_600_000)}


def draw(rng):
    kind = rng.choice(sorted(_RANGE))
    lo, hi = _RANGE[kind]
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    fits = [x for x in _lattices() if lo <= x[4] <= hi]
    if kind == "scan":  # the spinful Hubbard builder has no twisted form
        fits = [x for x in fits if x[0] != "hubbard"]
    fits.sort(key=lambda x: abs(math.log(x[4] / want)))
    family, a, b, nf, _, _ = rng.choice(fits[:6])
    flux = kind in ("catalog", "flux", "chern", "scan") or (
        family != "hubbard" and kind in ("operator", "correlators") and rng.random() < 0.5)
    more = {"flux": flux, "sector": rng.randrange(8), "nev": rng.randint(1, 6)}
    if kind == "operator":
        more["cols"] = rng.choice([1, 1, 2, 3, 5, 8])
    if kind == "block":
        more["cols"] = rng.randint(1, 4)
    if kind == "solve":
        more["precision"] = rng.choice([32, 64])
        more["block"] = rng.choice([0, 2, 4])
    return _case(kind, family, a, b, nf, **more)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


def _model(case, seed):
    """The case's model at zero flux, couplings moved by the seed."""
    r = random.Random(1000003 * seed + 17)

    def s():
        return r.uniform(0.9, 1.1)

    fam, size = case["family"], [case["a"], case["b"]]
    if fam == "heisenberg":
        return models.build_heisenberg_second_quantized_model(case["a"], s())
    if fam in ("haldane", "dnsheng"):
        if fam == "haldane":  # the flux-grid couplings
            p = {"t": 1.0, "t'": 0.6 * s(), "t''": 0.0, "phi_over_2pi": 0.2, "V1": s(), "V2": 0.0}
        else:
            p = dict(models.params_DNSheng)
            p.update({"t'": p["t'"] * s(), "t''": p["t''"] * s()})
        return models.build_zero_flux_bosonic_fci_second_quantized_model(sample_size=size, params=p)
    if fam == "checkerboard":
        p = dict(models.params_Sun_Gu_Katsura_Sarma)
        p.update({"V1": s(), "V2": 0.0, "V3": 0.0})
        return models.build_zero_flux_fermionic_fci_second_quantized_model(sample_size=size, params=p)
    return models.build_spinful_hubbard_second_quantized_model(size, 1.0, 4.0 * s())


def _theta(case, seed):
    if not case["flux"]:
        return [0.0, 0.0]
    r = random.Random(7919 * seed + 3)
    return [r.uniform(0.05, 0.45), 0.0 if case["family"] == "heisenberg" else r.uniform(0.05, 0.45)]


def _species(case, model):
    return models.hubbard_spin_species(model, case["nf"] - case["nf"] // 2) if case["family"] == "hubbard" else None


def _twisted(case, seed):
    """(model at the case's twist, group)."""
    model, theta = _model(case, seed), _theta(case, seed)
    if any(theta):
        if case["family"] != "hubbard":
            ed.update_second_quantized_model_with_twisted_phases(model, twisted_phases_over_2π=theta)
        return model, ed.build_translation_group(model.lattice, theta)
    return model, ed.build_translation_group(model.lattice)


def _data(case, model, group):
    return ed.build_ed_data(model, filling_fraction=Fraction(case["nf"], model.lattice.n_site), symmetry_group=group,
                            species=_species(case, model))


def _normal(shape, seed, dtype=torch.complex128):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    return torch.randn(shape, dtype=dtype, device="cuda", generator=g)


def _sector(dims, first):
    """The first sector with states, counted from ``first``."""
    n = len(dims)
    return next(k % n for k in range(first, first + n) if dims[k % n])


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "kind": kind}
    if kind == "flux":
        # the grid starts from the untwisted catalog
        model = _model(case, seed)
        base = _data(case, model, ed.build_translation_group(model.lattice))
        st.update(catalog=base.orbit_catalog, statistics=model.particle_statistics,
                  group=ed.build_translation_group(model.lattice, _theta(case, seed)))
        return st
    if kind == "scan":
        model = _model(case, seed)
        base = _data(case, model, ed.build_translation_group(model.lattice))
        theta = _theta(case, seed)
        ed.update_second_quantized_model_with_twisted_phases(model, twisted_phases_over_2π=theta)
        st.update(base=base, model=model, group=ed.build_translation_group(model.lattice, theta))
        return st
    model, group = _twisted(case, seed)
    st.update(model=model, group=group)
    if kind == "catalog":
        return st
    data = _data(case, model, group)
    st["data"] = data
    cat = data.orbit_catalog
    if kind in ("solve", "single"):
        return st
    sset = ed.SectorSet(cat, data.irrep_list)
    if kind == "operator":
        s = _sector(sset.dims, case["sector"])
        basis = ed.build_symmetry_sector_basis(cat, data.irrep_list[s])
        st["op"], n = ed.hamiltonian_linear_operator(basis, model.bilinear_terms, model.density_density_terms, None)
        st["x"] = _normal((n,) if case["cols"] == 1 else (n, case["cols"]), seed)
    elif kind == "block":
        dm = ed.DeviceModel(cat, model.bilinear_terms, model.density_density_terms)
        dm.build_projection(sset.sqrt_stab, precisions=(64,))
        n_cols = case["cols"] * len(data.irrep_list)
        ld = n_cols + n_cols % 2
        sec = torch.arange(n_cols, device="cuda", dtype=torch.int32) // case["cols"]
        X = torch.zeros((cat.n_orbits, ld), dtype=torch.complex128, device="cuda")
        X[:, :n_cols] = _normal((cat.n_orbits, n_cols), seed)
        # rows outside a column's sector hold zero, as in the solver's blocks
        X[:, :n_cols] *= (sset.member[:, None] >> sec[None, :].long()) & 1
        st.update(dm=dm, sset=sset, sec=sec, X=X, Y=torch.zeros_like(X))
    elif kind == "chern":
        secs = [s for s, d in enumerate(sset.dims) if d][:2]
        bases = [ed.Symmetry_Sector_Basis(data.irrep_list[s], cat, sset, s) for s in secs]
        states = _normal((3, len(secs), cat.n_states), seed)
        states /= torch.linalg.vector_norm(states, dim=2, keepdim=True)
        st.update(bases=bases, states=states,
                  vecs=[_normal((b.dim,), seed + 1 + i) / math.sqrt(2 * b.dim) for i, b in enumerate(bases)])
    elif kind == "correlators":
        s = _sector(sset.dims, case["sector"])
        c = _normal((sset.dims[s], 1), seed)
        c /= torch.linalg.vector_norm(c)
        data.ed_scan_res[s] = (np.zeros(1), c.cpu().numpy())
        st["label"] = data.irrep_list[s].label
    return st


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "operator":
        return st["op"](st["x"])
    if kind == "block":
        st["dm"].apply_block(st["sset"], st["sec"], st["X"], st["Y"], 64)
        return st["Y"]
    if kind == "catalog":
        return _catalog_outputs(_data(case, st["model"], st["group"]).orbit_catalog)
    if kind == "flux":
        cat = st["catalog"].clone()
        ed.update_orbit_stabilizer_phases(cat, st["group"], st["statistics"])
        return _catalog_outputs(cat)
    if kind == "solve":
        data = st["data"]
        sectors = list(range(len(data.irrep_list)))
        params = config = None
        if case["slots"]:
            config = ed.SolverConfig((case["block"],) * len(sectors), n_slots=case["slots"])
        elif case["block"]:
            params = ed.LanczosParams(block=case["block"], precision=case["precision"])
        res = ed.solve_sectors_batched(data, sectors, nev=case["nev"], precision=case["precision"], params=params,
                                       config=config, return_vectors=False)
        return [res[s][0] for s in sectors]
    if kind == "scan":
        base, model = st["base"], st["model"]
        cat = base.orbit_catalog.clone()
        ed.update_orbit_stabilizer_phases(cat, st["group"], model.particle_statistics)
        data = ed.Symmetry_Resolved_ED_Data(model, base.n_filled, base.filling_fraction, st["group"],
                                            base.irrep_list, cat, [0] * len(base.irrep_list))
        ed.ed_scan(data, nev=case["nev"], mode="matrixfree")
        return [data.ed_scan_res[s][0] for s in range(len(base.irrep_list))]
    if kind == "single":
        data = st["data"]
        vals, _ = ed.ed_scan_at_irrep_matrixfree(data.irrep_list[0].label, data, nev=case["nev"])
        return vals
    if kind == "chern":
        # slot 0 is the new point, 1 and 2 its finished neighbours
        for i, (c, basis) in enumerate(zip(st["vecs"], st["bases"])):
            ed.expand_sector_state_to_fock_dense(c, basis, out=st["states"][0, i])
        return {"amplitudes": st["states"][0], "links": ed.fock_overlaps(st["states"], [(1, 0), (2, 0)])}
    data, model = st["data"], st["model"]
    more = {"filling_fraction": data.filling_fraction, "ed_data": data}
    return {"odlro": ed.off_diagonal_long_range_order(model, st["label"], **more),
            "structure": ed.static_structure_factor(model, st["label"], **more)[1]}


def _catalog_outputs(cat):
    return {"rep_g": cat.table[:, :2], "alpha": cat.table.view(torch.float32)[:, 2:], "reprs": cat.repr_masks,
            "stabilizers": cat.stab_mask, "offsets": cat.stab_off, "phases": cat.stab_phase}


# ---------------------------------------------------------------------------
# the work a call cannot do without
# ---------------------------------------------------------------------------


def work(case):
    fam, a, b, nf = case["family"], case["a"], case["b"], case["nf"]
    n = a if fam == "heisenberg" else 2 * a * b
    ng = a * b
    if fam == "hubbard":
        states = math.comb(a * b, nf // 2) * math.comb(a * b, nf - nf // 2)
    else:
        states = math.comb(n, nf)
    orbits = states / ng
    # directed terms per site times occupied sites with an empty target
    per_site = {"heisenberg": 2, "haldane": 12, "dnsheng": 12, "checkerboard": 12, "hubbard": 4}[fam]
    hops = nf * per_site * max(n - nf, 0) / (n - 1)
    kind, k = case["kind"], case["cols"]
    if kind == "operator":  # matrix entries and column indexes, x read and y written
        return {"bytes": orbits * (hops * 20 + 8 + 32 * k), "flops": 8 * orbits * hops * k}
    if kind == "block":  # one table for all columns
        return {"bytes": orbits * (hops * 20 + 32 + 32 * k * ng), "flops": 8 * orbits * hops * k * ng}
    if kind == "catalog":  # tables written; every image of every state decided
        return {"bytes": 16 * states + 32 * orbits, "flops": states * nf}
    if kind == "flux":  # tables copied and their phases rewritten
        return {"bytes": 32 * states + 40 * orbits, "flops": 6 * states * nf}
    if kind in ("solve", "scan", "single"):
        # the model's matrix once from the table, and about 60 products of one
        # column per sector with the recurrence's two vectors
        sectors = 1 if kind == "single" else ng
        it = 60 * orbits * (hops * 12 + sectors * 64)
        return {"bytes": 16 * states + it, "flops": 8 * 60 * orbits * hops * sectors}
    if kind == "chern":  # table read, two states written, two neighbours read
        return {"bytes": states * (16 + 2 * 16 + 4 * 16), "flops": states * (2 * 6 * nf + 64)}
    # correlators: every hop of every state between any two sites
    return {"bytes": 16 * states + 48 * orbits, "flops": 8 * states * nf * max(n - nf, 1)}


# ---------------------------------------------------------------------------
# exact results: plain torch over the full fixed-filling space
# ---------------------------------------------------------------------------


def _masks(n, k):
    """All n-bit masks with k bits set, ascending."""
    row = [torch.zeros(1, dtype=torch.int64, device="cuda")] + [None] * k
    for bit in range(n):
        new = list(row)
        for j in range(1, k + 1):
            parts = [p for p in (row[j], row[j - 1] + (1 << bit) if row[j - 1] is not None else None) if p is not None]
            new[j] = torch.cat(parts) if parts else None
        row = new
    return row[k]


def _count(v):
    """Set bits of every entry."""
    out = torch.zeros_like(v)
    for i in range(64):
        if not bool((v >> i).any()):
            break
        out += (v >> i) & 1
    return out


class _Space:
    """The fixed-filling space of a case, its orbits under the translations."""

    def __init__(self, case, model, group):
        self.n, self.nf = model.lattice.n_site, case["nf"]
        self.fermions = model.particle_statistics is ed.Particle_Statistics.FERMIONIC
        self.model = model
        self.perm = [[p - 1 for p in op.perm] for op in group.operations]
        self.eta = np.array([op.perm_phases for op in group.operations], dtype=np.complex128)
        species = _species(case, model)
        if species is None:
            self.masks = _masks(self.n, self.nf)
        else:
            sb, kb = sorted(species[0]), species[1]
            sa = [i for i in range(1, self.n + 1) if i not in sb]
            am, bm = _masks(len(sa), self.nf - kb), _masks(len(sb), kb)
            am = sum(((am >> p) & 1) << (i - 1) for p, i in enumerate(sa))
            bm = sum(((bm >> p) & 1) << (i - 1) for p, i in enumerate(sb))
            self.masks = (am[:, None] | bm[None, :]).reshape(-1)
        self.sorted, self.order = torch.sort(self.masks)
        least = self.masks.clone()
        for g in range(len(self.perm)):
            least = torch.minimum(least, self.image(self.masks, g))
        self.reps = self.masks[least == self.masks]
        self.phases, self.images = [], []
        for g in range(len(self.perm)):
            self.images.append(self.image(self.reps, g))
            self.phases.append(self.phase(self.reps, g))
        self.stab = torch.stack([im == self.reps for im in self.images], 1)
        self.order_of = self.stab.sum(1)
        self._table = None

    def rank(self, m):
        return self.order[torch.searchsorted(self.sorted, m)]

    def image(self, m, g):
        out = torch.zeros_like(m)
        for i, p in enumerate(self.perm[g]):
            out |= ((m >> i) & 1) << p
        return out

    def phase(self, m, g):
        """Product of the site phases of the occupied sites, times the
        fermionic sign of the permutation."""
        ang = torch.zeros(m.shape, dtype=torch.float64, device="cuda")
        odd = torch.zeros_like(m)
        placed = torch.zeros_like(m)
        for i, p in enumerate(self.perm[g]):
            occ = (m >> i) & 1
            ang += occ.double() * float(np.angle(self.eta[g, i]))
            if self.fermions:
                odd += occ * _count(placed >> (p + 1))
                placed |= occ << p
        return torch.polar(1.0 - 2.0 * (odd & 1).double(), ang)

    def table(self):
        """(orbit, group element, amplitude) of every state; the last group
        element that reaches it."""
        if self._table is not None:
            return self._table
        rep = torch.zeros(self.masks.shape, dtype=torch.int64, device="cuda")
        el = torch.zeros_like(rep)
        al = torch.zeros(self.masks.shape, dtype=torch.complex128, device="cuda")
        every = torch.arange(self.reps.numel(), device="cuda")
        for g in range(len(self.perm)):
            at = self.rank(self.images[g])
            rep[at], el[at], al[at] = every, g, self.phases[g]
        self._table = rep, el, al
        return self._table

    def stab_phases(self):
        return torch.stack(self.phases, 1)[self.stab]

    def members(self, chi):
        """Orbits of a sector, ascending."""
        off = (torch.stack(self.phases, 1) - chi[None, :]).abs() > 1e-12
        return torch.nonzero(~(off & self.stab).any(1)).reshape(-1)

    def hops(self, rows):
        """Hops of the states ``rows``: (position in rows, target, amplitude)."""
        merged = {}
        for i, j, t in self.model.bilinear_terms:
            merged[(i - 1, j - 1)] = merged.get((i - 1, j - 1), 0) + complex(t)
        for (i, j), t in merged.items():
            at = torch.nonzero(((rows >> i) & 1 == 1) & ((rows >> j) & 1 == 0)).reshape(-1)
            m = rows[at]
            amp = torch.full(m.shape, t, dtype=torch.complex128, device="cuda")
            if self.fermions:
                lo, hi = min(i, j), max(i, j)
                amp = amp * (1 - 2 * (_count(m & (((1 << (hi - lo - 1)) - 1) << (lo + 1))) & 1)).double()
            yield at, m ^ (1 << i) ^ (1 << j), amp

    def diagonal(self, rows):
        out = torch.zeros(rows.shape, dtype=torch.complex128, device="cuda")
        for i, j, v in self.model.density_density_terms:
            out += complex(v) * (((rows >> (i - 1)) & 1) * ((rows >> (j - 1)) & 1)).to(torch.complex128)
        return out

    def entries(self, chi):
        """(dim, rows, cols, values) pieces of a sector's block: the element
        between orbits r and c is t * sign * alpha * conj(chi(g)) *
        sqrt(|Stab c| / |Stab r|)."""
        rep, el, al = self.table()
        mem = self.members(chi)
        row_of = torch.full((self.reps.numel(),), -1, dtype=torch.int64, device="cuda")
        row_of[mem] = torch.arange(mem.numel(), device="cuda")
        st = self.order_of.double()
        parts = []
        for at, target, amp in self.hops(self.reps[mem]):
            r = self.rank(target)
            c = row_of[rep[r]]
            ok = c >= 0
            v = amp * al[r] * chi.conj()[el[r]] * torch.sqrt(st[rep[r]] / st[mem[at]])
            parts.append((c[ok], at[ok], v[ok]))
        every = torch.arange(mem.numel(), device="cuda")
        parts.append((every, every, self.diagonal(self.reps[mem])))
        return mem, parts

    def expand(self, x, chi, mem):
        """Fock amplitudes of a sector vector, in table order."""
        psi = torch.zeros(self.masks.shape, dtype=torch.complex128, device="cuda")
        pref = x / torch.sqrt(len(self.perm) * self.order_of[mem].double())
        for g in range(len(self.perm)):
            psi[self.rank(self.images[g][mem])] += pref * chi[g].conj() * self.phases[g][mem]
        return psi


def _chis(model, group):
    return [torch.tensor(np.asarray(ir.values, dtype=np.complex128), device="cuda")
            for ir in ed.build_irrep_list(group, model.lattice)]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "scan", "single"):
        return _exact_levels(case, seed)
    if kind == "flux":
        model = _model(case, seed)
        group = ed.build_translation_group(model.lattice, _theta(case, seed))
    else:
        model, group = _twisted(case, seed)
    sp = _Space(case, model, group)
    if kind in ("catalog", "flux"):
        _, _, al = sp.table()
        return {"rep_g": None, "alpha": torch.view_as_real(al), "reprs": None, "stabilizers": None, "offsets": None,
                "phases": sp.stab_phases()}
    chis = _chis(model, group)
    dims = [sp.members(c).numel() for c in chis]
    if kind == "operator":
        s = _sector(dims, case["sector"])
        mem, parts = sp.entries(chis[s])
        x = _normal((mem.numel(),) if case["cols"] == 1 else (mem.numel(), case["cols"]), seed)
        x2 = x.reshape(mem.numel(), -1)
        y = torch.zeros_like(x2)
        for r, c, v in parts:
            y.index_add_(0, r, v[:, None] * x2[c])
        return y.reshape(x.shape)
    if kind == "block":
        return _exact_block(case, sp, chis, seed)
    if kind == "chern":
        secs = [s for s, d in enumerate(dims) if d][:2]
        states = _normal((3, len(secs), sp.masks.numel()), seed)
        states /= torch.linalg.vector_norm(states, dim=2, keepdim=True)
        for i, s in enumerate(secs):
            mem = sp.members(chis[s])
            psi = sp.expand(_normal((mem.numel(),), seed + 1 + i) / math.sqrt(2 * mem.numel()), chis[s], mem)
            psi[psi.abs() <= 1e-12] = 0
            states[0, i] = psi / torch.linalg.vector_norm(psi)
        links = torch.stack([states[p].conj() @ states[0].T for p in (1, 2)])
        return {"amplitudes": states[0], "links": links.cpu().numpy()}
    return _exact_correlators(case, sp, chis, dims, seed)


def _exact_block(case, sp, chis, seed):
    n_cols = case["cols"] * len(chis)
    if sp.reps.numel() * n_cols > 40_000_000:
        return None  # 16 blocks of 10^8 entries: too long in plain torch
    draw_ = _normal((sp.reps.numel(), n_cols), seed)
    Y = torch.zeros((sp.reps.numel(), n_cols + n_cols % 2), dtype=torch.complex128, device="cuda")
    for s, chi in enumerate(chis):
        mem, parts = sp.entries(chi)
        cols = slice(s * case["cols"], (s + 1) * case["cols"])
        x = draw_[mem, cols]
        y = torch.zeros_like(x)
        for r, c, v in parts:  # the adjoint
            y.index_add_(0, c, v.conj()[:, None] * x[r])
        Y[mem, cols] = y
    return Y


def _exact_correlators(case, sp, chis, dims, seed):
    s = _sector(dims, case["sector"])
    chi, n = chis[s], sp.n
    c = _normal((dims[s], 1), seed)
    c = (c / torch.linalg.vector_norm(c))[:, 0]
    mem = sp.members(chi)
    ket = sp.expand(c, chi, mem)
    # the bra of a state as the reference writes it: its orbit's coefficient
    # times sqrt(|Stab| / |G|) and conj(alpha conj(chi(g)))
    rep, el, al = sp.table()
    full = torch.zeros(sp.reps.shape, dtype=torch.complex128, device="cuda")
    full[mem] = c
    bra = full[rep] * torch.sqrt(sp.order_of[rep].double() / len(sp.perm)) * (al * chi.conj()[el]).conj()
    # a state reached by several group elements counts once per element
    rho = torch.zeros((n, n), dtype=torch.complex128, device="cuda")
    weight = torch.zeros(sp.masks.shape, dtype=torch.float64, device="cuda")
    for g in range(len(sp.perm)):
        weight[sp.rank(sp.images[g][mem])] += (c.abs() ** 2) / len(sp.perm)
    kets = torch.zeros_like(ket)
    pref = c / torch.sqrt(len(sp.perm) * sp.order_of[mem].double())
    for g in range(len(sp.perm)):
        kets[sp.rank(sp.images[g][mem])] += pref * chi[g].conj() * sp.phases[g][mem]
    for j in range(n):
        at = torch.nonzero((sp.masks >> j) & 1).reshape(-1)
        rho[j, j] = weight[at].sum()
        for i in range(n):
            if i == j or (case["family"] == "hubbard" and (i - j) % 2):
                continue
            sub = at[(sp.masks[at] >> i) & 1 == 0]
            m = sp.masks[sub]
            v = bra[sp.rank(m ^ (1 << i) ^ (1 << j))].conj() * kets[sub]
            if sp.fermions:
                lo, hi = min(i, j), max(i, j)
                v = v * (1 - 2 * (_count(m & (((1 << (hi - lo - 1)) - 1) << (lo + 1))) & 1)).double()
            rho[i, j] = v.sum()
    occ = torch.stack([((sp.masks >> i) & 1).double() for i in range(n)], 1)
    pair = (occ * weight[:, None]).T @ occ
    pair -= torch.outer(pair.diagonal(), pair.diagonal())
    lat = sp.model.lattice
    A = np.array(lat.brav_vec_list, dtype=np.float64)
    B = 2 * math.pi * np.linalg.inv(A)  # column d: b_d
    pos = np.array([(np.array(cell, dtype=np.float64) + np.array(lat.sub_crys_list[sub - 1])) @ A
                    for cell, sub in lat.site_list])
    pair = pair.cpu().numpy()
    S = []
    for k1 in range(lat.sample_size[0]):
        for k2 in range(lat.sample_size[1]):
            q = B @ np.array([k1 / lat.sample_size[0], k2 / lat.sample_size[1]])
            ph = np.exp(-1j * (pos @ q))
            S.append(float(np.real(ph @ pair @ ph.conj())) / n)
    return {"odlro": rho.cpu().numpy(), "structure": np.array(S)}


def _exact_levels(case, seed):
    model, group = _twisted(case, seed)
    states = work(dict(case, kind="catalog", cols=1))["flops"] / case["nf"]
    if states / len(group.operations) > 2500:
        return None  # dense blocks of every sector would take minutes
    sp = _Space(case, model, group)
    # the levels belong to the sectors of the untwisted translation characters
    out = []
    for s, chi in enumerate(_chis(model, group)):
        if case["kind"] == "single" and s:
            break
        mem, parts = sp.entries(chi)
        A = torch.zeros((mem.numel(), mem.numel()), dtype=torch.complex128, device="cuda")
        for r, c, v in parts:
            A.index_put_((r, c), v, accumulate=True)
        # as the solvers do: the Hermitian part, dense blocks by their upper triangle
        A = (A + A.conj().T) / 2 if mem.numel() > 500 else torch.triu(A) + torch.triu(A, 1).conj().T
        vals = torch.linalg.eigvalsh(A).cpu().numpy()[: case["nev"]] if mem.numel() else np.zeros(0)
        out.append(vals)
    return out[0] if case["kind"] == "single" else out
