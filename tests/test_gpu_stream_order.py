"""The first derivative of a system clears the buffers it takes, on the system's
own stream: work that a program has queued on the default stream neither delays
nor reorders those clears.  The buffers are taken from memory that held NaN."""
import numpy as np
import pytest
import torch

from field_b200.desc import (BOUND_MIRROR1, BOUND_SURFACE, Lattice, Molecule, MOL_FREE, MOL_SOLVENT, Segment,
                             SystemSpec)

pytestmark = pytest.mark.gpu


def spec_of(kind):
    n, N = (60, 50), 40
    order = 2 if kind == "second" else 1
    lat = Lattice(2, n + (0,), [BOUND_SURFACE, BOUND_MIRROR1, 0], [BOUND_SURFACE, BOUND_MIRROR1, 0], lam=1 / 6, order=order)
    chi = np.array([[0, 0.4, 0.9], [0.4, 0, 0.1], [0.9, 0.1, 0]])
    if kind == "dendrimer":
        chain = Molecule("D", [(0, 1), (0, 3), (1, 4)], MOL_FREE, phibulk=0.02, generations=[(2, 3), (1, 2)])
    else:
        chain = Molecule("AB", [(0, N // 2), (1, N - N // 2)], MOL_FREE, phibulk=0.02)
    return SystemSpec(lat, [Segment("A"), Segment("B"), Segment("W")], chi,
                      [chain, Molecule("W", [(2, 1)], MOL_SOLVENT)])


@pytest.mark.parametrize("kind", ["linear", "checkpointed", "second", "dendrimer"])
def test_first_derivative_beside_a_busy_default_stream(kind):
    from field_b200.system import System
    spec = spec_of(kind)
    s = System(spec)
    rng = np.random.default_rng(3)
    x, v, w = rng.normal(0, 0.2, s.nvar), rng.normal(size=s.nvar), rng.normal(size=s.nvar)

    def derivatives(t):
        if kind == "checkpointed":
            t.set_checkpoint(7)
        return [*t.vjp(x, w), *t.jvp(x, v)]

    derivatives(s)
    want = derivatives(s)                # the second time: buffers long cleared
    t = System(spec)
    t.synchronize()
    dirt = torch.full((1 << 27,), float("nan"), dtype=torch.float64, device="cuda")     # 1 GiB
    del dirt
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda._sleep(1_000_000_000)     # half a second of the default stream
    got = derivatives(t)
    assert not torch.cuda.default_stream().query()      # it was still busy
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        # repeated runs differ in the order of FP64 atomic additions only
        assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))
