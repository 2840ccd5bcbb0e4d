"""The device topology against the host builder's at the sizes where its sorts and
scans change form (all pairs up to 8,192 items, tiles of 512; one scan block up to
8,192 values), with and without equal sort keys: a checkpoint carries a fingerprint
of the device topology and is refused by a handle whose topology differs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 2, 2), (8, 8, 8), (9, 8, 8), (16, 16, 31), (16, 16, 32), (20, 20, 20),
                                   (33, 16, 16), (40, 40, 40)])
@pytest.mark.parametrize("graded", [False, True])
def test_device_topology_equals_the_host_builders(lib_built, tmp_path, monkeypatch, shape, graded):
    from fierro_gb300 import mesh, problems, sgh
    m = mesh.box_mesh(*shape, jitter=0.0 if graded else 0.1, seed=4, permute=True)
    if graded:
        m.coords[:] = m.coords ** 6  # many centroids and nodes share a Morton cell of 2^-21
    prob = problems.noh(mesh=m, cycles=2)
    path = str(tmp_path / "t.ckpt")
    st = sgh.setup(prob)
    states = {}
    for staged in ("0", "1"):
        monkeypatch.setenv("FIERRO_STAGED_TRANSFERS", staged)
        with sgh.SGHSolver(prob) as s:
            if staged == "0":
                s.set_state(st)
                s.checkpoint(path)
            else:
                s.restart(path)
            states[staged] = s.get_state()
    for k in states["0"]:
        assert np.array_equal(states["0"][k], states["1"][k], equal_nan=True), k
