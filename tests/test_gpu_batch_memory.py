"""Device memory of a 1D batch in the cluster engine: one set of stored slices per
chain, in whole warps of sites, and none where the chain fits into shared memory."""
import numpy as np
import pytest
import torch

from field_b200 import configs

pytestmark = pytest.mark.gpu


def used_by(make):
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    obj = make()
    torch.cuda.synchronize()
    return obj, free - torch.cuda.mem_get_info()[0]


def test_one_chain_store_per_instance():
    from field_b200.batch import BatchSolver
    from field_b200.system import System
    torch.zeros(1, device="cuda")
    count, n, N = 48, 400, 4000
    specs = [configs.flat_adsorption(n, N, 1e-3, 0.2, -1.0)[0] for _ in range(count)]
    b, used = used_by(lambda: BatchSolver(specs, m=5, eta=0.1))
    # half a symmetric chain, four warps of 128 sites; a second store of the same
    # chain in lattice vectors would add 402 / 512 of it, the rest is below 20 %
    slices = count * (N // 2) * 512 * 8
    assert slices <= used <= 1.4 * slices
    r = b.solve(np.zeros(b.total), tol=1e-10, maxit=40)
    one = System(specs[0]).solve(tol=1e-10, maxit=40, m=5, eta=0.1)
    # forty iterations of the same sums in another order
    assert np.max(np.abs(b.split(r.x)[7] - one.x)) <= 1e-6 * np.max(np.abs(one.x))
