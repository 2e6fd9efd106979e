"""The cluster engine (one cluster per first-order 1D/2D system) against the
oracle at the sizes where its cut of the lattice changes: one or several warps
per 1D chain, the last one nearly empty, the widest it takes and one beyond;
2D blocks with full, ragged and single rows, with one and several strips per
block, and every boundary kind across blocks."""
import numpy as np
import pytest

from field_b200.desc import (BOUND_MIRROR1, BOUND_MIRROR2, BOUND_PERIODIC, BOUND_SURFACE, GEOM_CYLINDRICAL, GEOM_FLAT,
                             GEOM_SPHERICAL, Lattice, Molecule, MOL_FREE, MOL_RESTRICTED, MOL_SOLVENT, Segment,
                             SEG_FROZEN, SEG_PINNED, SystemSpec)

pytestmark = pytest.mark.gpu

S, M1, M2, P = BOUND_SURFACE, BOUND_MIRROR1, BOUND_MIRROR2, BOUND_PERIODIC


def system(n, lo, hi, geometry=GEOM_FLAT, N=11):
    """Copolymer with an alternating end, odd and even homopolymers (free and
    restricted), a grafted chain and a solvent, next to a frozen segment."""
    g = len(n)
    pad = [0] * (3 - g)
    lat = Lattice(g, list(n) + pad, list(lo) + pad, list(hi) + pad, geometry=geometry, lam=1 / 6,
                  offset_first_layer=4.0 if geometry != GEOM_FLAT and lo[0] == S else 0.0)
    frozen, pinned = np.zeros(lat.shape), np.zeros(lat.shape)
    for d in range(g):
        at = [slice(None)] * g
        if lo[d] == S:
            at[d] = 0
            frozen[tuple(at)] = 1
        if hi[d] == S:
            at[d] = lat.shape[d] - 1
            frozen[tuple(at)] = 1
    if not frozen.any():
        frozen[tuple([n[d] for d in range(g)])] = 1
    pinned[tuple([1] * g)] = 1
    segs = [Segment("S", SEG_FROZEN, frozen.reshape(-1)), Segment("A"), Segment("B"), Segment("W"),
            Segment("X", SEG_PINNED, pinned.reshape(-1))]
    chi = np.zeros((5, 5))
    for a, b, v in ((0, 1, -0.9), (1, 3, 0.5), (2, 3, 0.3), (1, 2, 0.2)):
        chi[a, b] = chi[b, a] = v
    mols = [Molecule("AB", [(1, N), (2, 2), (1, 1), (2, 1)], MOL_FREE, phibulk=0.02),
            Molecule("h", [(2, N)], MOL_RESTRICTED, theta=0.5), Molecule("e", [(1, N + 1)], MOL_FREE, phibulk=0.01),
            Molecule("g", [(4, 1), (1, 6)], MOL_RESTRICTED, theta=0.2), Molecule("W", [(3, 1)], MOL_SOLVENT)]
    return SystemSpec(lat, segs, chi, mols)


ONE = [((n,), (lo,), (hi,), geo) for n in (3, 125, 126, 127, 208, 209, 313) for lo, hi, geo in
       ((S, M1, GEOM_FLAT), (M2, S, GEOM_FLAT), (M1, M2, GEOM_CYLINDRICAL))]
ONE += [((1664,), (S,), (M1,), GEOM_FLAT), ((1665,), (S,), (M1,), GEOM_FLAT), ((130,), (P,), (P,), GEOM_FLAT),
        ((260,), (S,), (M2,), GEOM_SPHERICAL)]
TWO = [((3, 3), (M1, M1), (M1, M1), GEOM_FLAT), ((4, 5), (M2, M2), (M2, M2), GEOM_FLAT),
       ((17, 33), (P, P), (P, P), GEOM_FLAT), ((33, 31), (S, P), (M2, P), GEOM_FLAT),
       ((16, 64), (M1, S), (M2, S), GEOM_CYLINDRICAL), ((100, 7), (M1, M2), (M1, M1), GEOM_CYLINDRICAL),
       ((7, 300), (M2, M1), (S, M2), GEOM_FLAT), ((131, 129), (M1, P), (M1, P), GEOM_CYLINDRICAL),
       ((40, 520), (M1, M1), (M1, M1), GEOM_FLAT)]


@pytest.mark.parametrize("n,lo,hi,geo", ONE + TWO)
def test_residual_at_the_edges_of_the_cut(n, lo, hi, geo):
    from field_b200.system import System
    from oracle.oracle import Oracle
    spec = system(n, lo, hi, geo)
    s, o = System(spec), Oracle(spec)
    x = np.random.default_rng(3).normal(0, 0.2, s.nvar)
    f, ref = s.residual(x), o.residual(x)
    # 2N products of rounded values a site, N = 12: below 1e-13; the parity tests' bound
    assert np.max(np.abs(f - ref)) <= 1e-11 * np.max(np.abs(ref))
    for i in range(len(spec.segments)):
        p, q = s.phi(i), o.phi(i)
        assert np.max(np.abs(p - q)[spec.lattice.interior_mask()]) <= 1e-11 * max(1.0, np.max(np.abs(q)))
    assert np.array_equal(s.residual(x), f)


@pytest.mark.parametrize("n,m", [((60,), 5), ((230,), 1), ((24, 20), 10), ((24, 20), 16)])
def test_solve_meets_the_oracle(n, m):
    from field_b200.system import System
    from oracle.oracle import Oracle
    spec = system(n, (S,) + (M1,) * (len(n) - 1), (M1,) * len(n))
    spec.molecules = [spec.molecules[0], spec.molecules[4]]
    spec.segments, spec.chi = spec.segments[:4], spec.chi[:4, :4]
    s, o = System(spec), Oracle(spec)
    r = s.solve(tol=1e-11, maxit=3000, m=m, eta=0.1)
    x, rc, it, err = o.solve_diis(np.zeros(o.nvar), 1e-11, 3000, m, 0.1)
    assert r.status == rc
    if rc == 0:
        # both lie within |J^-1| 1e-11 of the solution, |J^-1| of order 1e2
        assert np.max(np.abs(r.x - x)) < 1e-8
        f = o.residual(r.x)
        assert np.linalg.norm(f) < 1e-10


@pytest.mark.parametrize("two,count", [(False, 5), (False, 160), (True, 3), (True, 40)])
def test_uneven_batches_meet_single_solves(two, count):
    from field_b200.batch import BatchSolver
    from field_b200.system import System
    rng = np.random.default_rng(count)
    specs = []
    for _ in range(count):
        n = (int(rng.integers(9, 40)), int(rng.integers(9, 40))) if two else (int(rng.integers(20, 300)),)
        spec = system(n, (S,) + (M1,) * (len(n) - 1), (M1,) * len(n), N=int(rng.integers(3, 30)))
        spec.molecules = [spec.molecules[2], spec.molecules[4]]
        spec.segments, spec.chi = spec.segments[:4], spec.chi[:4, :4]
        specs.append(spec)
    b = BatchSolver(specs, m=6, eta=0.1)
    r = b.solve(np.zeros(b.total), tol=1e-11, maxit=2000)
    xs = b.split(r.x)
    for i in sorted({0, 1, count // 2, count - 1}):
        one = System(specs[i]).solve(tol=1e-11, maxit=2000, m=6, eta=0.1)
        assert one.status == r.status[i]
        if one.status == 0:
            assert np.max(np.abs(one.x - xs[i])) < 1e-8
            g = System(specs[i])
            g.residual(xs[i])
            for k in range(1, 4):
                assert np.max(np.abs(b.phi(i, k) - g.phi(k))) < 1e-8
