"""Lumped second-order steps with a thread per site (step2l_sites) against the
oracle at the edges of their blocks (32 x 4 sites in 2D, 128 in 1D), on flat and
curved lattices, and at the persistence factors 0 and 1 that the general
kernel takes."""
import numpy as np
import pytest

from field_b200.desc import (BOUND_MIRROR1, BOUND_MIRROR2, BOUND_PERIODIC, BOUND_SURFACE, GEOM_CYLINDRICAL, GEOM_FLAT,
                             GEOM_SPHERICAL, Lattice, Molecule, MOL_FREE, MOL_RESTRICTED, MOL_SOLVENT, Segment, SystemSpec)

pytestmark = pytest.mark.gpu

S, M1, M2, P = BOUND_SURFACE, BOUND_MIRROR1, BOUND_MIRROR2, BOUND_PERIODIC


@pytest.mark.parametrize("n,lo,hi,geo", [((4, 32), (M1, P), (M2, P), GEOM_FLAT), ((5, 33), (S, M2), (M1, S), GEOM_FLAT),
                                         ((3, 31), (P, M1), (P, M1), GEOM_FLAT), ((9, 64), (M1, S), (M2, M1), GEOM_CYLINDRICAL),
                                         ((128,), (S,), (M2,), GEOM_FLAT), ((129,), (P,), (P,), GEOM_FLAT),
                                         ((40,), (M1,), (M2,), GEOM_CYLINDRICAL), ((127,), (M1,), (M1,), GEOM_SPHERICAL)])
@pytest.mark.parametrize("persistence", [0.0, 0.35, 1.0])
def test_residual_at_block_edges(n, lo, hi, geo, persistence):
    from field_b200.system import System
    from oracle.oracle import Oracle
    g = len(n)
    pad = [0] * (3 - g)
    lat = Lattice(g, list(n) + pad, list(lo) + pad, list(hi) + pad, geometry=geo, lam=1 / 6, order=2)
    chi = np.array([[0, 0.3, 0.8], [0.3, 0, 0.2], [0.8, 0.2, 0]])
    pf = np.full((3, 3), 0.2)
    pf[0, 0] = persistence
    mols = [Molecule("AB", [(0, 5), (1, 3)], MOL_FREE, phibulk=0.03), Molecule("A", [(0, 4)], MOL_RESTRICTED, theta=0.5),
            Molecule("W", [(2, 1)], MOL_SOLVENT)]
    spec = SystemSpec(lat, [Segment("A"), Segment("B"), Segment("W")], chi, mols, pf=pf)
    s, o = System(spec), Oracle(spec)
    x = np.random.default_rng(5).normal(0, 0.2, s.nvar)
    f, ref = s.residual(x), o.residual(x)
    assert np.max(np.abs(f - ref)) <= 1e-11 * np.max(np.abs(ref))   # the parity tests' bound; N = 8 steps of 5 terms
