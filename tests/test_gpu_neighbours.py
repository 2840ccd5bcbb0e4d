"""The limiter's neighbour search ahead of its use (the one-thread force pass) against
the lane pass: elements with no neighbour, with fewer and with more than the 32 that
are read ahead.  A batch runs the one-thread pass, a handle of a small mesh the lanes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fan(n):
    """n hexes around a common edge: each has the n - 1 others as neighbours."""
    from fierro_gb300.mesh import HexMesh, box_mesh
    if n == 1:
        return box_mesh(1)
    a = 2.0 * np.pi * np.arange(n) / n
    b = a + np.pi / n
    rings = [np.stack([np.cos(a), np.sin(a)], 1), 1.2 * np.stack([np.cos(b), np.sin(b)], 1)]
    flat = np.concatenate([np.zeros((1, 2))] + rings)
    m = flat.shape[0]
    coords = np.concatenate([np.column_stack([flat, np.full(m, z)]) for z in (0.05, 0.4)])
    i = np.arange(n)
    quad = np.stack([np.zeros(n, dtype=np.int64), 1 + i, 1 + n + i, 1 + (i + 1) % n], 1)
    return HexMesh(np.ascontiguousarray(coords), np.ascontiguousarray(np.concatenate([quad, quad + m], 1)))


@pytest.mark.parametrize("n", [1, 3, 5, 9, 32, 33, 34, 37, 60])
@pytest.mark.parametrize("mode", [0, 1])
def test_fans_of_neighbours(lib_built, n, mode):
    from fierro_gb300 import problems, sgh
    p = problems.noh(mesh=_fan(n), cycles=8)
    st = sgh.setup(p)
    with sgh.Batch([p], fp_mode=mode) as b:
        b.set_state(0, st)
        b.run(8)
        got = b.get_state(0)
    with sgh.SGHSolver(p, fp_mode=mode) as s:
        s.set_state(st)
        s.run(8)
        want = s.get_state()
    for k in want:
        assert np.array_equal(got[k], want[k]), k
    assert np.all(np.isfinite(want["corner_force"]))
