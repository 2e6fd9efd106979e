"""The plain second-order 3D step with a thread per site (step2_sites) at the
edges of its blocks (32 x 2 x 2 sites) under every pair of boundaries, against
the oracle, and bit for bit against the tangent's own primal step."""
import numpy as np
import pytest

from field_b200.desc import (BOUND_MIRROR1, BOUND_MIRROR2, BOUND_PERIODIC, Lattice, Molecule, MOL_FREE, MOL_RESTRICTED,
                             MOL_SOLVENT, Segment, SystemSpec)

pytestmark = pytest.mark.gpu

M1, M2, P = BOUND_MIRROR1, BOUND_MIRROR2, BOUND_PERIODIC


@pytest.mark.parametrize("n,lo,hi", [((3, 3, 3), (M1, M1, M1), (M1, M1, M1)), ((4, 4, 32), (P, M1, M2), (P, M2, M1)),
                                     ((5, 3, 33), (M2, P, M1), (M1, P, M2)), ((3, 6, 65), (M1, M2, P), (M2, M2, P))])
def test_residual_at_block_edges(n, lo, hi):
    from field_b200.system import System
    from oracle.oracle import Oracle
    chi = np.array([[0, 0.3, 0.8], [0.3, 0, 0.2], [0.8, 0.2, 0]])
    pf = np.full((3, 3), 0.2)
    pf[0, 0], pf[0, 1], pf[1, 0] = 0.5, 0.1, 0.1
    mols = [Molecule("AB", [(0, 5), (1, 4)], MOL_FREE, phibulk=0.03), Molecule("A", [(0, 4)], MOL_RESTRICTED, theta=0.5),
            Molecule("W", [(2, 1)], MOL_SOLVENT)]
    spec = SystemSpec(Lattice(3, n, lo, hi, order=2), [Segment("A"), Segment("B"), Segment("W")], chi, mols, pf=pf)
    s, o = System(spec), Oracle(spec)
    rng = np.random.default_rng(9)
    x = rng.normal(0, 0.2, s.nvar)
    f, ref = s.residual(x), o.residual(x)
    assert np.max(np.abs(f - ref)) <= 1e-11 * np.max(np.abs(ref))   # the parity tests' bound; 9 steps of 5 terms
    fj, _ = s.jvp(x, rng.normal(size=s.nvar))
    assert np.array_equal(fj, f)
