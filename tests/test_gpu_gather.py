"""Reverse chain steps that gather (adj_gather_*): the dot-product identity
<w, J v> = <J^T w, v> against the forward mode at tile edges and remainders of
the 3D march (32 x 8 columns, 8 planes), at the smallest lattices and under
every pair of boundaries, where a read maps back inside."""
import numpy as np
import pytest

from field_b200.desc import (BOUND_MIRROR1, BOUND_MIRROR2, BOUND_PERIODIC, BOUND_SURFACE, GEOM_CYLINDRICAL, GEOM_FLAT,
                             Lattice, Molecule, MOL_FREE, MOL_RESTRICTED, MOL_SOLVENT, Segment, SystemSpec)

pytestmark = pytest.mark.gpu

S, M1, M2, P = BOUND_SURFACE, BOUND_MIRROR1, BOUND_MIRROR2, BOUND_PERIODIC
CASES = [((9, 8, 32), (P, P, P), (P, P, P), GEOM_FLAT), ((8, 9, 33), (M1, M2, P), (M2, M1, P), GEOM_FLAT),
         ((17, 7, 31), (M2, M2, M2), (M2, M2, M2), GEOM_FLAT), ((3, 3, 3), (M2, M1, M2), (M1, M2, M2), GEOM_FLAT),
         ((3, 4, 3), (P, M1, P), (P, M1, P), GEOM_FLAT), ((3, 4, 65), (P, P, M1), (P, P, M2), GEOM_FLAT),
         ((12, 13), (S, M2), (M2, S), GEOM_FLAT), ((5, 40), (M1, P), (M2, P), GEOM_CYLINDRICAL),
         ((3, 3), (M2, M2), (M1, M2), GEOM_FLAT), ((40,), (M2,), (M2,), GEOM_FLAT), ((40,), (P,), (P,), GEOM_FLAT),
         ((7,), (M1,), (M2,), GEOM_CYLINDRICAL), ((300,), (S,), (S,), GEOM_FLAT)]


@pytest.mark.parametrize("n,lo,hi,geo", CASES)
def test_dot_product_identity(n, lo, hi, geo):
    from field_b200.system import System
    g = len(n)
    pad = [0] * (3 - g)
    lat = Lattice(g, list(n) + pad, list(lo) + pad, list(hi) + pad, geometry=geo, lam=1 / 6)
    chi = np.array([[0, 0.4, 0.9], [0.4, 0, 0.1], [0.9, 0.1, 0]])
    mols = [Molecule("AB", [(0, 4), (1, 3), (0, 1)], MOL_RESTRICTED, theta=0.3 * np.prod(n)),
            Molecule("h", [(1, 6)], MOL_FREE, phibulk=0.05), Molecule("W", [(2, 1)], MOL_SOLVENT)]
    segs = [Segment("A"), Segment("B"), Segment("W")]
    s = System(SystemSpec(lat, segs, chi, mols))
    rng = np.random.default_rng(7)
    x, v, w = rng.normal(0, 0.2, s.nvar), rng.normal(size=s.nvar), rng.normal(size=s.nvar)
    _, jv = s.jvp(x, v)
    _, jw = s.vjp(x, w)
    # sums of nvar rounded products each: |w| |J v| 1e-16 sqrt(nvar), far below the other tests' 1e-10
    assert abs(w @ jv - jw @ v) <= 1e-10 * np.linalg.norm(w) * np.linalg.norm(jv)
