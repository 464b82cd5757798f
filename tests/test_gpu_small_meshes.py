"""GPU: the kernel forms chosen by mesh size, at the sizes where the choice or
its remainders change.  The cycle graph below 131072 cells runs node and cell
sweeps side by side; a batch, which never does, must give the same bits.  The
allocation-free dt runs as one cluster up to 8192 segments of 4 layers, else over
segments of 4 or 8; the value is compared with its definition.  The x sweeps
take rows as one sequence of 28 updated items a warp: rows shorter and longer
than that, against the oracle."""
import numpy as np
import pytest

import mhy_b200
import mhy_oracle
from mhy_b200 import Batch, Context, gen

pytestmark = pytest.mark.gpu

FIELDS = ("density", "internal_energy", "pressure", "velocity", "node_mass")


@pytest.mark.parametrize("options", [{}, {"precision": 1}, {"ordre_projection": 3}, {"projection_limiteur_id": 4}])
@pytest.mark.parametrize("K", [1, 2])
def test_graph_of_a_small_mesh_equals_a_batch(K, options):
    o = gen.Options(**options)
    sizes = ((3, 3, 3), (33, 9, 4), (64, 64, 31), (64, 64, 32))      # the last one is not small
    if K == 1:
        cases = [gen.sod(*n, lx=n[0] * 0.01, ly=n[1] * 0.01, lz=n[2] * 0.01, jitter=0.02, seed=i, options=o)
                 for i, n in enumerate(sizes)]
    else:
        cases = [gen.two_material(*n, seed=i, options=o) for i, n in enumerate(sizes)]
    b = Batch(cases, device=0)
    b.step(12)
    b.synchronize()
    for i, c in enumerate(cases):
        g = Context(c, device=0)
        g.step(12)                                    # each rotation's graph four times
        g.synchronize()
        for f in FIELDS:
            assert np.array_equal(b.field(i, f), g.field(f)), (i, f)
        assert b.dt(i) == g.dt(), i
        g.close()


@pytest.mark.parametrize("n", [(1, 1, 1), (5, 3, 7), (100, 5, 5), (16, 16, 16), (17, 16, 16), (4097, 1, 1), (32, 32, 32),
                               (32, 32, 33), (8193, 1, 3), (1, 1, 4099), (257, 3, 13), (600, 520, 9)])
def test_allocation_free_dt_is_the_minimum_of_its_definition(n):
    torch = pytest.importorskip("torch")
    nx, ny, nz = n
    rng = np.random.default_rng(nx + ny + nz)
    L, cs = rng.uniform(0.5, 2.0, (2, nz, ny, nx))
    v = rng.normal(size=(3, nz + 1, ny + 1, nx + 1))
    speed = np.sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2])
    vmax = np.maximum.reduce([speed[dk:nz + dk, dj:ny + dj, di:nx + di] for dk in (0, 1) for dj in (0, 1) for di in (0, 1)])
    want = (L / (cs + vmax)).min()
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (L, cs, v)]
    out = torch.full((2,), -1.0, dtype=torch.float64, device="cuda")

    def call():
        torch.cuda.synchronize()
        rc = mhy_b200.load().mhy_compute_hydro_dt_noalloc(nx, ny, nz, *(t.data_ptr() for t in dev), 0.3, 1e6, 1e6,
                                                          out.data_ptr(), None)
        torch.cuda.synchronize()
        assert rc == 0
        return out.cpu().numpy()

    assert list(call()) == [want, 0.3 * want]
    dev[0][-1, -1, -1] = -1.0                         # the last cell inverted
    got = call()
    assert np.isnan(got[0]) and got[1] == 0.0


@pytest.mark.parametrize("n", [(2, 5, 3), (3, 2, 2), (27, 3, 4), (28, 9, 2), (29, 4, 5), (56, 3, 3), (61, 7, 2)])
@pytest.mark.parametrize("limiter", [0, 2, 5])
def test_rows_of_any_length_bitwise(n, limiter):
    if limiter >= 3 and min(n) < 3:                   # the generalised limiters need 3 cells a direction
        n = tuple(max(x, 3) for x in n)
    case = gen.sod(*n, lx=n[0] * 0.01, ly=n[1] * 0.01, lz=n[2] * 0.01, jitter=0.02, seed=4,
                   options=gen.Options(projection_limiteur_id=limiter))
    o, g = mhy_oracle.Oracle(case, pow_mode="project"), Context(case, device=0)
    for _ in range(9):                                # three rotations of the sweep order
        o.step(1)
        g.step(1)
    g.synchronize()
    for f in FIELDS:
        assert np.array_equal(o.field(f), g.field(f)), f
    assert o.scalars()["dt"] == g.dt()[0]
