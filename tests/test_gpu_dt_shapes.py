"""GPU: the allocation-free dt on meshes of one layer of cells and on thin columns,
where a thread takes one cell and not a segment of a column: the value against its
definition at the edges of that choice, and the time.  One layer of cells reads two
planes of nodes for its one of cells, 64 bytes a cell, where two layers read 52: it
may take 64/52 of the time of the same number of cells in two layers.  A column of
32000 cells lies in memory as 32000 cells in a row do: it may take twice as long."""
import numpy as np
import pytest

import mhy_b200

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def fields(n, seed=7):
    nx, ny, nz = n
    g = torch.Generator("cuda").manual_seed(seed)
    f64 = dict(dtype=torch.float64, device="cuda", generator=g)
    return (torch.rand(nz, ny, nx, **f64) + 0.5, torch.rand(nz, ny, nx, **f64) + 0.5,
            torch.randn(3, nz + 1, ny + 1, nx + 1, **f64), torch.empty(2, dtype=torch.float64, device="cuda"))


def call(n, L, cs, v, out):
    rc = mhy_b200.load().mhy_compute_hydro_dt_noalloc(*n, L.data_ptr(), cs.data_ptr(), v.data_ptr(), 0.3, 1e6, 1e6,
                                                      out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0


@pytest.mark.parametrize("n", [(64, 64, 1), (91, 91, 1), (8193, 1, 1), (300, 1000, 1), (1, 1, 8192), (1, 1, 8193), (3, 1, 2731),
                               (1, 2, 40000), (2, 2, 2048), (2, 2, 2049), (1, 4, 16384), (4, 1, 16385), (127, 1, 65),
                               (128, 1, 65), (127, 1, 516), (127, 1, 517)])
def test_value_of_one_layer_and_of_thin_columns(n):
    nx, ny, nz = n
    L, cs, v, out = fields(n)
    l, c, w = L.cpu().numpy(), cs.cpu().numpy(), v.cpu().numpy()
    speed = np.sqrt(w[0] * w[0] + w[1] * w[1] + w[2] * w[2])
    vmax = np.maximum.reduce([speed[k:nz + k, j:ny + j, i:nx + i] for k in (0, 1) for j in (0, 1) for i in (0, 1)])
    want = (l / (c + vmax)).min()
    call(n, L, cs, v, out)
    assert out.tolist() == [want, 0.3 * want]
    for at in ((0, 0, 0), (nz - 1, ny - 1, nx - 1), (nz // 2, ny // 2, nx // 2)):
        bad = L.clone()
        bad[at] = -1.0                                # an inverted cell
        call(n, bad, cs, v, out)
        got = out.tolist()
        assert np.isnan(got[0]) and got[1] == 0.0, at


def times(*sizes):
    """The least time of 20 calls of each size, taken in turn."""
    data = [(n, *fields(n)) for n in sizes]
    best = [1e9] * len(data)
    for _ in range(9):
        for i, d in enumerate(data):
            call(*d)
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            for _ in range(20):
                call(*d)
            b.record()
            b.synchronize()
            best[i] = min(best[i], a.elapsed_time(b))
    return best


def test_time_of_one_layer():
    one, two = times((2048, 1024, 1), (1024, 1024, 2))
    assert one < 64 / 52 * two


def test_time_of_a_column():
    column, row = times((1, 1, 32000), (32000, 1, 1))
    assert column < 2.0 * row
