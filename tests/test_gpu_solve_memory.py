"""Device memory that a solve leaves with its system: Pure_DIIS's vectors stay up
to 16 MiB a system after System.solve, none after a solve of many systems."""
import numpy as np
import pytest
import torch

from field_b200 import configs

pytestmark = pytest.mark.gpu


def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_large_vectors_are_given_back():
    from field_b200.system import System
    torch.zeros(1, device="cuda")
    spec, x0 = configs.cyl_micelle(nx=200, ny=198)
    s = System(spec)
    s.solve(x0, maxit=1, m=1)
    before = free()
    r = s.solve(x0, maxit=12, m=10)                 # 22 vectors: 21 MB
    assert before - free() <= 2 << 20               # the allocator's page
    assert np.array_equal(s.solve(x0, maxit=12, m=10).x, r.x)


def test_many_systems_hold_nothing():
    from field_b200.system import System, solve_diis_many
    insts = [configs.cyl_micelle(nx=100, ny=100, seed=i) for i in range(12)]
    systems = [System(s) for s, _ in insts]
    x0s = [x for _, x in insts]
    solve_diis_many(systems[:1], x0s[:1], maxit=1, m=1)
    before = free()
    many = solve_diis_many(systems, x0s, maxit=12, m=10, threads=4)     # 5 MB each
    assert before - free() <= 4 << 20
    one = System(insts[3][0]).solve(x0s[3], maxit=12, m=10)
    assert np.array_equal(many[3].x, one.x)
