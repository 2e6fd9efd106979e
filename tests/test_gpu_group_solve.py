"""Pure_DIIS in one launch: a few iterates against the oracle's, the solution where
the kept steps outnumber the variables (their products are then singular, the
elimination gives up and the eigen-decomposition takes over), and a batch whose
every instance converges to what the systems alone converge to."""
import numpy as np
import pytest

from field_b200.desc import (BOUND_MIRROR1, BOUND_SURFACE, Lattice, Molecule, MOL_FREE, MOL_SOLVENT, Segment,
                             SEG_FROZEN, SystemSpec)

pytestmark = pytest.mark.gpu

S, M1 = BOUND_SURFACE, BOUND_MIRROR1


def system(n, N=11):
    """A chain of two segment types next to an adsorbing wall."""
    g = len(n)
    pad = [0] * (3 - g)
    lat = Lattice(g, list(n) + pad, [S] + [M1] * (g - 1) + pad, [M1] * g + pad, lam=1 / 6)
    wall = np.zeros(lat.shape)
    wall[0] = 1
    chi = np.zeros((4, 4))
    for a, b, v in ((0, 1, -0.9), (1, 3, 0.5), (2, 3, 0.3), (1, 2, 0.2)):
        chi[a, b] = chi[b, a] = v
    return SystemSpec(lat, [Segment("S", SEG_FROZEN, wall.reshape(-1)), Segment("A"), Segment("B"), Segment("W")], chi,
                      [Molecule("AB", [(1, N), (2, 2), (1, 1), (2, 1)], MOL_FREE, phibulk=0.02),
                       Molecule("W", [(3, 1)], MOL_SOLVENT)])


# m = 1: x - eta g each time, rounding only.  Otherwise the four kept steps span
# two decades, their products four, so the coefficients carry 1e-16 x 1e4 and
# their errors again the residual's 1e-13: 1e-9
@pytest.mark.parametrize("n,m,maxit,bound", [((230,), 1, 12, 1e-12), ((60,), 5, 4, 1e-9), ((24, 20), 10, 4, 1e-9),
                                             ((200, 31), 10, 4, 1e-9)])
def test_first_iterates(n, m, maxit, bound):
    from field_b200.system import System
    from oracle.oracle import Oracle
    spec = system(n)
    s, o = System(spec), Oracle(spec)
    assert s.one_launch
    r = s.solve(tol=1e-14, maxit=maxit, m=m, eta=0.1)
    x, rc, it, err = o.solve_diis(np.zeros(o.nvar), 1e-14, maxit, m, 0.1)
    assert (r.status, r.iterations) == (rc, it) == (5, maxit)
    assert np.max(np.abs(r.x - x)) <= bound * np.max(np.abs(x))


# 9, 12, 15 and 27 variables, as many steps kept or more
@pytest.mark.parametrize("n,m", [((3,), 16), ((4,), 16), ((5,), 16), ((3, 3), 16), ((60,), 5), ((230,), 1), ((24, 20), 16)])
def test_solution(n, m):
    from field_b200.system import System
    from oracle.oracle import Oracle
    spec = system(n)
    s, o = System(spec), Oracle(spec)
    r = s.solve(tol=1e-11, maxit=3000, m=m, eta=0.1)
    x, rc, it, err = o.solve_diis(np.zeros(o.nvar), 1e-11, 3000, m, 0.1)
    assert r.status == rc == 0
    # both lie within |J^-1| 1e-11 of the solution, |J^-1| of order 1e2
    assert np.max(np.abs(r.x - x)) < 1e-8
    assert np.linalg.norm(o.residual(r.x)) < 1e-10


@pytest.mark.parametrize("two", [False, True])
def test_every_instance_of_a_batch(two):
    from field_b200.batch import BatchSolver
    from field_b200.system import System
    rng = np.random.default_rng(8)
    specs = [system((int(rng.integers(9, 40)), int(rng.integers(9, 40))) if two else (int(rng.integers(20, 300)),),
                    N=int(rng.integers(3, 30))) for _ in range(12)]
    b = BatchSolver(specs, m=6, eta=0.1)
    assert b.cluster
    r = b.solve(np.zeros(b.total), tol=1e-11, maxit=3000)
    assert r.converged.all()
    for spec, x in zip(specs, b.split(r.x)):
        one = System(spec).solve(tol=1e-11, maxit=3000, m=6, eta=0.1)
        assert one.converged
        assert np.max(np.abs(one.x - x)) < 1e-8
