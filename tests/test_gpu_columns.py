"""The column form of the six-neighbour 3D step (step3d_cols, its tangent and
its reverse) at block edges and remainders: 32 x 4 columns, 4 planes a thread.
Primal against the oracle and, bit for bit, against the marching forms;
tangent against its own primal; reverse by the dot-product identity."""
import numpy as np
import pytest

from field_b200.desc import (BOUND_MIRROR1, BOUND_MIRROR2, BOUND_PERIODIC, Lattice, Molecule, MOL_FREE, MOL_SOLVENT,
                             Segment, SystemSpec)

pytestmark = pytest.mark.gpu

M1, M2, P = BOUND_MIRROR1, BOUND_MIRROR2, BOUND_PERIODIC


@pytest.mark.parametrize("n,lo,hi", [((4, 4, 32), (P, P, P), (P, P, P)), ((5, 5, 33), (M1, M2, P), (M2, M1, P)),
                                     ((3, 3, 3), (M1, M1, M2), (M1, M2, M1)), ((7, 8, 31), (M2, P, M1), (M1, P, M2)),
                                     ((9, 3, 65), (P, M1, M1), (P, M2, M1))])
def test_columns(n, lo, hi):
    from field_b200.system import System
    from oracle.oracle import Oracle
    lat = Lattice(3, n, lo, hi)
    chi = np.array([[0, 0.4, 0.9], [0.4, 0, 0.1], [0.9, 0.1, 0]])
    mols = [Molecule("AB", [(0, 4), (1, 3)], MOL_FREE, phibulk=0.1), Molecule("odd", [(1, 7)], MOL_FREE, phibulk=0.05),
            Molecule("W", [(2, 1)], MOL_SOLVENT)]
    spec = SystemSpec(lat, [Segment("A"), Segment("B"), Segment("W")], chi, mols)
    s, o = System(spec), Oracle(spec)
    rng = np.random.default_rng(11)
    x, v, w = rng.normal(0, 0.2, s.nvar), rng.normal(size=s.nvar), rng.normal(size=s.nvar)
    f, ref = s.residual(x), o.residual(x)
    assert np.max(np.abs(f - ref)) <= 1e-11 * np.max(np.abs(ref))       # the parity tests' bound
    for form in (0, 1, 2):
        m = System(spec)
        m.set_tile_pipelined(form)
        assert np.array_equal(m.residual(x), f)
    fj, jv = s.jvp(x, v)
    assert np.array_equal(fj, f)
    _, jw = s.vjp(x, w)
    assert abs(w @ jv - jw @ v) <= 1e-10 * np.linalg.norm(w) * np.linalg.norm(jv)


def test_the_default_form_can_be_set_again():
    from field_b200 import _native
    from field_b200.configs import melt3d
    from field_b200.system import System
    spec, x = melt3d(n=40, nA=10, nB=10)
    s = System(spec)
    f = s.residual(x)
    s.set_tile(4)
    s.set_tile_pipelined(1)
    assert np.array_equal(s.residual(x), f)
    s.set_tile_pipelined(3)
    assert np.array_equal(s.residual(x), f)
    with pytest.raises(_native.SfgpuError):
        s.set_tile_pipelined(4)
