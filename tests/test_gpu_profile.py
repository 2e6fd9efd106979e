"""sfgpu_profile_propagator times the step that the lattice's residual runs, on
every lattice that has one, and leaves later evaluations as they were."""
import numpy as np
import pytest

from field_b200.desc import (BOUND_MIRROR1, BOUND_PERIODIC, BOUND_SURFACE, GEOM_CYLINDRICAL, GEOM_FLAT, Lattice, Molecule,
                             MOL_FREE, MOL_SOLVENT, Segment, SystemSpec)

pytestmark = pytest.mark.gpu


def system(n, order, geometry=GEOM_FLAT, **kw):
    from field_b200.system import System
    g = len(n)
    pad = [0] * (3 - g)
    bc = ([BOUND_PERIODIC] * 3 if g == 3 else [BOUND_SURFACE, BOUND_MIRROR1][:g] if geometry == GEOM_FLAT
          else [BOUND_MIRROR1] * g) + pad
    lat = Lattice(g, list(n) + pad, bc, bc, geometry=geometry, lam=1 / 6, order=order)
    chi = np.array([[0, 0.4, 0.9], [0.4, 0, 0.1], [0.9, 0.1, 0]])
    mols = [Molecule("AB", [(0, 9), (1, 8)], MOL_FREE, phibulk=0.02), Molecule("W", [(2, 1)], MOL_SOLVENT)]
    return System(SystemSpec(lat, [Segment("A"), Segment("B"), Segment("W")], chi, mols), **kw)


@pytest.mark.parametrize("n,order,geometry", [((70,), 1, GEOM_FLAT), ((70,), 2, GEOM_FLAT), ((70,), 2, GEOM_CYLINDRICAL),
                                              ((20, 33), 1, GEOM_FLAT), ((20, 33), 2, GEOM_FLAT),
                                              ((20, 33), 2, GEOM_CYLINDRICAL), ((9, 8, 33), 1, GEOM_FLAT),
                                              ((9, 8, 33), 2, GEOM_FLAT)])
def test_profile_times_every_lattice(n, order, geometry):
    s = system(n, order, geometry)
    x = np.random.default_rng(1).normal(0, 0.2, s.nvar)
    f = s.residual(x)
    p = s.profile_propagator(reps=40)
    # a launch takes microseconds at least; forty that never ran take less than that together
    assert p["ms_fwd"] > 5e-4 and p["ms_bwd"] > 5e-4
    assert np.array_equal(s.residual(x), f)


@pytest.mark.parametrize("n,order", [((20, 33), 1), ((9, 8, 33), 1), ((9, 8, 33), 2)])
def test_profile_of_a_checkpointed_chain(n, order):
    """Of 17 slices a stride of 5 keeps 4 checkpoints and 5: the profile stays within them."""
    s = system(n, order, checkpoint_stride=5)
    x = np.random.default_rng(1).normal(0, 0.2, s.nvar)
    f = s.residual(x)
    s.profile_propagator(reps=40)
    s.autotune(reps=3)
    assert np.array_equal(s.residual(x), f)
