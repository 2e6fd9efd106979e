"""Bytes the bench's roofline counts for the cluster engine: what a solve moves."""
import numpy as np

from field_b200 import configs
from field_b200.batch import engine_bytes


def test_cylinder_solve():
    spec, _ = configs.cyl_micelle()
    sites, nv, m = 130 * 130, spec.n_itvar(), 10
    assert spec.M == sites
    # no iteration: one evaluation, and the start (x, f read; x and the first step's two vectors written)
    assert engine_bytes(spec, 0, m) == 16 * (40 * sites + nv) + 40 * nv
    # a full memory: 40 slices out and back, x and f, ten steps read twice, four more vectors
    step = engine_bytes(spec, 30, m) - engine_bytes(spec, 29, m)
    assert step == 16 * (40 * sites + nv) + 8 * nv * (2 * m + 4)
    # far below a launch per step, which reads G, the slices and phi again each time
    from field_b200.batch import residual_bytes
    assert 16 * 40 * sites < 0.25 * residual_bytes(spec)


def test_layer_solve_works_on_chip():
    spec, _ = configs.flat_adsorption(100, 100, 1e-3, 0.2, -1.0)
    assert engine_bytes(spec, 100, 5) == 16 * spec.n_itvar()
