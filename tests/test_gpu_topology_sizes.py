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


def _batch_error(sgh, problems, monkeypatch, staged):
    monkeypatch.setenv("FIERRO_STAGED_TRANSFERS", staged)
    with pytest.raises(sgh.FierroError) as e:
        sgh.Batch(problems)
    return str(e.value)


@pytest.mark.parametrize("sides", [(24,), (24, 5), (9, 24, 20, 3, 16), (12, 12, 12)])
def test_batch_topologies_by_either_builder(lib_built, monkeypatch, sides):
    """A batch's topologies, shared between the GPU and the host's threads, give the
    staged route's results; a mesh that is refused is refused with the same words."""
    import copy
    from fierro_gb300 import problems, sgh
    ps = [problems.sedov(n, jitter=0.1, seed=n + i, permute=True, cycles=3) for i, n in enumerate(sides)]
    states = [sgh.setup(p) for p in ps]
    got = {}
    for staged in ("0", "1"):
        monkeypatch.setenv("FIERRO_STAGED_TRANSFERS", staged)
        with sgh.Batch(ps) as b:
            for i, st in enumerate(states):
                b.set_state(i, st)
            b.run(3)
            got[staged] = [b.get_state(i) for i in range(len(b))]
    for i, (x, y) in enumerate(zip(got["0"], got["1"])):
        for k in x:
            assert np.array_equal(x[k], y[k]), (i, k)
    for i in range(len(ps)):
        bad = copy.deepcopy(ps)
        bad[i].mesh.nodes_in_elem[17, 3] = bad[i].mesh.num_nodes + 5
        bad[-1].mesh.nodes_in_elem[23, 6] = bad[-1].mesh.nodes_in_elem[23, 1]
        messages = [_batch_error(sgh, bad, monkeypatch, staged) for staged in ("0", "1")]
        assert messages[0] == messages[1] and "instance %d" % i in messages[0], messages
