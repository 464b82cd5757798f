"""GPU: batches large enough to march (mhy_march.cuh: 1.5 million nodes over
the whole batch) give every instance the bits of its own context, whose small
mesh stages tiles: lines from two cells up, remainders of the segments and of
the 128-point blocks, both precisions, one and two environments, classic and
generalised limiters."""
import numpy as np
import pytest

from mhy_b200 import Batch, Context, gen

pytestmark = pytest.mark.gpu

FIELDS = ("density", "internal_energy", "pressure", "velocity", "node_mass")
SIZES = ((2, 2, 2), (3, 17, 5), (31, 4, 33), (15, 16, 17), (40, 9, 3))


def instances(precision, K, limiter):
    o = gen.Options(precision=precision, projection_limiteur_id=limiter)
    if K == 2:
        small = [gen.two_material(*n, seed=5 + i, options=o) for i, n in enumerate(SIZES)]
        return small + [gen.two_material(116, 115, 115, options=o)]
    small = [gen.sod(*n, lx=n[0] * 0.01, ly=n[1] * 0.01, lz=n[2] * 0.01, jitter=0.02, seed=3 + i, options=o)
             for i, n in enumerate(SIZES)]
    return small + [gen.sod(116, 115, 115, 1.0, 1.0, 1.0, options=o)]


@pytest.mark.parametrize("precision,K,limiter", [(0, 1, 0), (0, 1, 5), (0, 2, 0), (1, 1, 0), (1, 1, 2), (1, 2, 1)])
def test_marching_batch_equals_single_contexts(precision, K, limiter):
    cases = instances(precision, K, limiter)
    if limiter >= 3:                                  # the generalised limiters need 3 cells a direction
        cases = cases[1:]
    b = Batch(cases, device=0)
    b.step(9)                                         # three rotations of the sweep order
    b.synchronize()
    for i, c in enumerate(cases[:-1]):
        g = Context(c, device=0)
        g.step(9)
        g.synchronize()
        for f in FIELDS:
            assert np.array_equal(b.field(i, f), g.field(f)), (i, f)
        assert b.dt(i) == g.dt(), i
        g.close()
