"""A mesh that the GPU's topology builder turns down goes to the host builder; the batch
is made, and nothing of the refusal is left for later calls to find."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fan_beside_box(spokes, side):
    """`spokes` hexes around a common edge (each has all the others as neighbours) beside
    a box large enough for the mesh to go to the GPU."""
    from fierro_gb300.mesh import HexMesh, box_mesh
    a = 2.0 * np.pi * np.arange(spokes) / spokes
    b = a + np.pi / spokes
    flat = np.concatenate([np.zeros((1, 2)), np.stack([np.cos(a), np.sin(a)], 1),
                           1.2 * np.stack([np.cos(b), np.sin(b)], 1)])
    m = flat.shape[0]
    xyz = np.concatenate([np.column_stack([flat, np.full(m, z)]) for z in (0.05, 0.4)])
    i = np.arange(spokes)
    quad = np.stack([0 * i, 1 + i, 1 + spokes + i, 1 + (i + 1) % spokes], 1)
    box = box_mesh(side, jitter=0.1, seed=1, permute=True)
    return HexMesh(np.ascontiguousarray(np.concatenate([xyz, box.coords + 3.0])),
                   np.ascontiguousarray(np.concatenate([np.concatenate([quad, quad + m], 1),
                                                        box.nodes_in_elem + 2 * m]).astype(box.nodes_in_elem.dtype)))


@pytest.mark.parametrize("why", ["neighbours", "memory"])
def test_a_mesh_turned_down_leaves_no_error(lib_built, monkeypatch, why):
    from fierro_gb300 import problems, sgh
    # 75 neighbours (the GPU's builder takes 64), or an allocation that fails
    m = _fan_beside_box(76 if why == "neighbours" else 8, 24)
    p = problems.noh(mesh=m, cycles=3)
    st = sgh.setup(p)
    with sgh.SGHSolver(problems.noh(4)):  # the context is up, and without errors
        pass
    if why == "memory":
        monkeypatch.setenv("FIERRO_FAIL_ALLOC_AFTER", "0")
    with sgh.Batch([p]) as b:
        assert sgh.lib().fierro_last_error() == b""
        b.set_state(0, st)
        b.run(3)
        got = b.get_state(0)
    monkeypatch.setenv("FIERRO_STAGED_TRANSFERS", "1")
    monkeypatch.delenv("FIERRO_FAIL_ALLOC_AFTER", raising=False)
    with sgh.Batch([p]) as b:
        b.set_state(0, st)
        b.run(3)
        want = b.get_state(0)
    for k in want:
        assert np.array_equal(got[k], want[k]), k
