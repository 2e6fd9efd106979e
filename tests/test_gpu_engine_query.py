"""Which path a system or a batch takes is asked from the library, not restated."""
import numpy as np
import pytest

from field_b200 import configs
from field_b200.desc import (BOUND_MIRROR1, BOUND_PERIODIC, Lattice, Molecule, MOL_FREE, MOL_SOLVENT, Segment, SystemSpec)

pytestmark = pytest.mark.gpu


def spec_of(n, bc=BOUND_MIRROR1, N=10, order=1):
    g = len(n)
    b = [bc] * g + [0] * (3 - g)
    lat = Lattice(g, list(n) + [0] * (3 - g), b, b, lam=1 / 6, order=order)
    chi = np.array([[0, 0.5], [0.5, 0]])
    return SystemSpec(lat, [Segment("A"), Segment("W")], chi,
                      [Molecule("A", [(0, N // 2), (1, N - N // 2)], MOL_FREE, phibulk=0.05),
                       Molecule("W", [(1, 1)], MOL_SOLVENT)])


# 512 x 512: more threads a block than the engine has, 1664 layers: its widest 1D chain
@pytest.mark.parametrize("n,bc,order,one", [((100,), BOUND_MIRROR1, 1, True), ((1664,), BOUND_MIRROR1, 1, True),
                                            ((1665,), BOUND_MIRROR1, 1, False), ((100,), BOUND_PERIODIC, 1, False),
                                            ((128, 128), BOUND_MIRROR1, 1, True), ((512, 512), BOUND_MIRROR1, 1, False),
                                            ((40, 40), BOUND_MIRROR1, 2, False), ((8, 8, 8), BOUND_PERIODIC, 1, False)])
def test_launches_follow_the_path_taken(n, bc, order, one):
    from field_b200.batch import launches_per_residual
    from field_b200.system import System
    spec = spec_of(n, bc, order=order)
    s = System(spec)
    assert s.one_launch == one
    assert (launches_per_residual(spec, s) == 1) == one


def test_checkpointed_system_is_not_in_the_engine():
    from field_b200.system import System
    assert not System(spec_of((60,)), checkpoint_stride=3).one_launch


def test_autotune_of_a_clustered_batch_times_its_one_shape():
    from field_b200.batch import BatchSolver
    specs = [configs.flat_adsorption(60, 20, 1e-3, 0.2, -1.0)[0] for _ in range(4)]
    b = BatchSolver(specs, m=5, eta=0.1)
    assert b.cluster > 0
    assert len(b.autotune(np.zeros(b.total), tol=1e-8)) == 1
    p = BatchSolver([spec_of((60,), BOUND_PERIODIC)] * 4, m=5, eta=0.1)
    assert p.cluster == 0
    assert len(p.autotune(np.zeros(p.total), tol=1e-8)) > 1
