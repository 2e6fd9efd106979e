"""Cylinders whose blocks take strips of eight rows in the cluster engine and end
in a shorter strip (rows per block not a multiple of eight): lambda of a strip's
rows comes from shared memory there, and only the rows that exist may be read."""
import numpy as np
import pytest

from field_b200 import configs

pytestmark = pytest.mark.gpu


# 16 blocks of 13 and of 9 rows; 198 and 178 columns leave 8 rows a thread
@pytest.mark.parametrize("nx,ny", [(200, 198), (129, 178)])
def test_residual_of_ragged_strips(nx, ny):
    from field_b200.system import System
    from oracle.oracle import Oracle
    spec, x = configs.cyl_micelle(nx=nx, ny=ny)
    s, o = System(spec), Oracle(spec)
    f, ref = s.residual(x), o.residual(x)
    assert np.max(np.abs(f - ref)) <= 1e-11 * np.max(np.abs(ref))       # the parity tests' bound
    inner = spec.lattice.interior_mask()
    for i in range(len(spec.segments)):
        p, q = s.phi(i)[inner], o.phi(i)[inner]
        assert np.max(np.abs(p - q)) <= 1e-11 * max(1.0, np.max(np.abs(q)))


# 4 blocks of 25 rows, 2 of 12
@pytest.mark.parametrize("nx,ny", [(100, 41), (24, 86)])
def test_batches_of_ragged_strips(nx, ny):
    from field_b200.batch import BatchSolver
    from oracle.oracle import Oracle
    insts = [configs.cyl_micelle(nx=nx, ny=ny, nA=8, nB=8, radius=4, seed=40 + i) for i in range(40)]
    b = BatchSolver([s for s, _ in insts], m=10, eta=0.1)
    r = b.solve(np.concatenate([x for _, x in insts]), tol=1e-12, maxit=4000)
    assert r.converged.all()
    for i in (0, 39):
        # the iteration's own |f| at its last step is 1e-12; the oracle's differs by rounding
        assert np.linalg.norm(Oracle(insts[i][0]).residual(b.split(r.x)[i])) < 1e-11
