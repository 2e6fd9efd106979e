"""Lattices longer in one gradient than a launch grid is wide in y and z (65535
blocks of 2 to 8 rows or planes): the steps, their tangents and their reverses
take them by the row walks, as they take any other lattice."""
import numpy as np
import pytest

from field_b200.desc import BOUND_MIRROR1, BOUND_PERIODIC, Lattice, Molecule, MOL_FREE, MOL_SOLVENT, Segment, SystemSpec

pytestmark = pytest.mark.gpu

M1, P = BOUND_MIRROR1, BOUND_PERIODIC


# one layer past 65535 blocks of 4 rows or planes (262140), of 2 (131070)
@pytest.mark.parametrize("n,order", [((262141, 3), 1), ((262141, 3), 2), ((3, 262141), 1), ((262141, 3, 3), 1),
                                     ((131071, 3, 3), 1), ((3, 262141, 3), 1), ((131071, 3, 3), 2),
                                     ((3, 131071, 3), 2)])
def test_residual_and_derivatives(n, order):
    from field_b200.system import System
    from oracle.oracle import Oracle
    g = len(n)
    bc = [M1, P, P][:g] + [0] * (3 - g)
    lat = Lattice(g, list(n) + [0] * (3 - g), bc, bc, lam=1 / 6, order=order)
    chi = np.array([[0, 0.5], [0.5, 0]])
    mols = [Molecule("A", [(0, 2), (1, 2)], MOL_FREE, phibulk=0.05), Molecule("W", [(1, 1)], MOL_SOLVENT)]
    spec = SystemSpec(lat, [Segment("A"), Segment("W")], chi, mols)
    s, o = System(spec), Oracle(spec)
    rng = np.random.default_rng(4)
    x, v, w = rng.normal(0, 0.2, s.nvar), rng.normal(size=s.nvar), rng.normal(size=s.nvar)
    f, ref = s.residual(x), o.residual(x)
    assert np.max(np.abs(f - ref)) <= 1e-11 * np.max(np.abs(ref))       # the parity tests' bound
    fj, jv = s.jvp(x, v)
    _, jw = s.vjp(x, w)
    assert np.max(np.abs(fj - ref)) <= 1e-11 * np.max(np.abs(ref))
    # nvar rounded products each side: |w| |J v| 1e-16 sqrt(nvar), below the other tests' 1e-10
    assert abs(w @ jv - jw @ v) <= 1e-10 * np.linalg.norm(w) * np.linalg.norm(jv)
