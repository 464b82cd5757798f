"""GPU: the y/z sweeps that march (mhy_march.cuh, 1.5 million nodes and more) in one
context: FP64 bit for bit the oracle's in every form that marches; the mixed form,
which has no bitwise oracle, against the same mesh in two slabs, each below the size
that marches.  Then the large instance of a batch against its own context, and the
sweeps' tunings (lines_per_block sets the length of a marching segment)."""
import numpy as np
import pytest

import mhy_oracle
from mhy_b200 import Batch, Context, CTuning, gen, slabs

pytestmark = pytest.mark.gpu

FIELDS = ("density", "internal_energy", "pressure", "velocity", "node_mass")
SIZE = (116, 115, 115)                                 # 1,574,352 nodes


def large(K=1, **o):
    options = gen.Options(final_time=1e9, **o)
    if K == 2:
        return gen.two_material(*SIZE, options=options)
    return gen.sod(*SIZE, 1.0, 1.0, 1.0, jitter=0.02, seed=3, options=options)


def assert_same(a, b, of=lambda x, f: x.field(f)):
    for f in FIELDS:
        assert np.array_equal(of(a, f), b.field(f)), f


@pytest.mark.parametrize("K,options", [(1, {}), (1, {"projection_limiteur_id": 2}), (1, {"projection_limiteur_id": 5}),
                                       (1, {"schema_csts": 1}), (1, {"ordre_projection": 1}), (1, {"ordre_projection": 3}),
                                       (1, {"conservation_energie_totale": 1}), (2, {})])
def test_fp64_context_bitwise(K, options):
    case = large(K, **options)
    o, g = mhy_oracle.Oracle(case, pow_mode="project"), Context(case, device=0)
    o.step(3)                                          # each direction first, second and last
    g.step(3)
    assert_same(o, g)
    assert o.scalars()["dt"] == g.dt()[0]


@pytest.mark.parametrize("K,options", [(1, {}), (1, {"projection_limiteur_id": 1}), (1, {"projection_limiteur_id": 2}),
                                       (1, {"ordre_projection": 1}), (2, {})])
def test_mixed_context_equals_two_slabs_that_stage(K, options):
    case = large(K, precision=1, **options)
    g = Context(case, device=0)
    g.step(3)
    lay = slabs.layout(case.nz, 2)
    ranks = [slabs.SlabRank(case, lay, r, lambda c: slabs.GpuEngine(c, 0)) for r in range(2)]
    assert all(r.local.nnodes < 1_500_000 for r in ranks)
    slabs.run_local(ranks, 3)
    for f in FIELDS:
        assert np.array_equal(np.concatenate([r.owned_field(f) for r in ranks]), g.field(f)), f
    for r in ranks:
        assert r.eng.ctx.dt() == g.dt()
        r.eng.close()


@pytest.mark.parametrize("options", [{}, {"projection_limiteur_id": 5}, {"ordre_projection": 1}, {"schema_csts": 1},
                                     {"precision": 1}, {"precision": 1, "ordre_projection": 1}])
def test_large_instance_of_a_batch_equals_its_context(options):
    small = gen.sod(31, 4, 33, lx=0.31, ly=0.04, lz=0.33, jitter=0.02, seed=5, options=gen.Options(final_time=1e9, **options))
    case = large(**options)
    b, g = Batch([small, case], device=0), Context(case, device=0)
    b.step(3)
    b.synchronize()
    g.step(3)
    assert_same(b, g, of=lambda x, f: x.field(1, f))
    assert b.dt(1) == g.dt()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("lines", [16, 32])
def test_tunings_give_the_same_bits(lines, precision):
    case = large(precision=precision)
    small = gen.sod(31, 4, 33, lx=0.31, ly=0.04, lz=0.33, jitter=0.02, seed=5,
                    options=gen.Options(final_time=1e9, precision=precision))
    t = CTuning.default()
    for k in (3, 4, 6, 7):                             # the y/z sweeps
        t.lines_per_block[k] = lines
        t.order[k] = 2
    ref, tuned, b = Context(case, device=0), Context(case, device=0), Batch([small, case], device=0)
    ref.step(3)
    b.step(1)                                          # with the default tables first
    for x in (tuned, b):
        x.set_tuning(t)
    tuned.step(3)
    b.step(2)
    b.synchronize()
    assert_same(tuned, ref)
    assert_same(b, ref, of=lambda x, f: x.field(1, f))
