"""The lane passes of small meshes (sgh_lanes.cuh): bit for bit the
one-thread-per-element passes, which a batch of one instance runs, in both
modes, at element counts around a warp's four, around the sizes where the
force, element and node passes change over, and on a checkpoint between them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# 1, 3, 4, 5, 27, 315 elements; 10000 | 10010 (element pass), 11500 | 11550 (force
# pass), 27 x 30 x 33 elements on 29,512 nodes and 29 x 31 x 31 on 30,720 (node pass)
SHAPES = [(1, 1, 1), (3, 1, 1), (2, 2, 1), (5, 1, 1), (3, 3, 3), (7, 9, 5), (20, 20, 25), (11, 10, 91), (20, 23, 25),
          (21, 22, 25), (27, 30, 33), (29, 31, 31)]


def _deck(shape, cycles=12):
    from fierro_gb300 import mesh, problems
    m = mesh.box_mesh(*shape, length=(1.0, 1.1, 0.9), jitter=0.15, seed=sum(shape), permute=True)
    p = problems.noh(max(shape), mesh=m, cycles=cycles)
    p.materials[0].q2ex = 0.4
    p.fills[0].sie = 0.02
    return p


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("mode", [0, 1])
def test_lanes_equal_the_batch(lib_built, shape, mode):
    from fierro_gb300 import sgh
    p = _deck(shape)
    st = sgh.setup(p)
    with sgh.Batch([p], fp_mode=mode) as b:
        b.set_state(0, st)
        b.run(12)
        want, wt = b.get_state(0), b.time(0)
    with sgh.SGHSolver(p, fp_mode=mode) as s:
        s.set_state(st)
        s.run(12)
        got, gt = s.get_state(), s.time()
    assert (gt[0], gt[1], gt[3]) == wt
    for k in ("node_coords", "node_vel", "elem_den", "elem_pres", "elem_sspd", "elem_sie", "elem_vol", "elem_div",
              "corner_force"):
        assert np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("shape", [(5, 1, 1), (7, 9, 5), (21, 13, 33), (20, 20, 25)])
def test_checkpoint_of_a_lane_handle(lib_built, tmp_path, shape):
    """The file holds one CFL partial per element block, as it always has, and a
    restart from it takes the same time steps."""
    import struct

    from fierro_gb300 import sgh
    p = _deck(shape)
    path = str(tmp_path / "a.ckpt")
    with sgh.SGHSolver(p) as a:
        a.set_state(sgh.setup(p))
        a.run(5)
        a.checkpoint(path)
        a.run(7)
        want, wt = a.get_state(), a.time()
    ne, block = p.mesh.num_elems, 128
    while block > 32 and -(-ne // block) < 304:
        block //= 2
    head = struct.unpack_from("<8sII10q", open(path, "rb").read(), 0)
    assert head[3:5] == (p.mesh.num_nodes, ne) and head[-1] == -(-ne // block)
    with sgh.SGHSolver(p) as b:
        b.restart(path)
        b.run(7)
        got, gt = b.get_state(), b.time()
    assert gt == wt
    for k in want:
        assert np.array_equal(got[k], want[k]), k


# 1 and 3 elements, a warp's eight and one more, 9000 | 9020 (element pass), 11500 | 11504 (force pass)
RZ_SHAPES = [(1, 1), (3, 1), (4, 2), (3, 3), (90, 100), (82, 110), (115, 100), (16, 719)]


def _rz_deck(shape, cycles):
    from fierro_gb300 import mesh, problems
    m = mesh.quad_mesh(*shape, length=(1.0, 1.2), jitter=0.1, seed=sum(shape), permute=True)
    p = problems.noh_rz(max(shape), mesh=m, cycles=cycles)
    p.materials[0].q2ex = 0.4
    p.fills[0].sie = 0.02
    return p


@pytest.mark.parametrize("shape", RZ_SHAPES)
def test_quad_lanes_equal_the_restatement(oracle_built, lib_built, shape):
    """Exact mode, bit for bit against the C restatement; the FMA mode within the
    one-cycle gate of the exact one."""
    from conftest import assert_fields
    from fierro_gb300 import sgh
    from oracle import orc
    p = _rz_deck(shape, 8)
    st = sgh.setup(p)
    o = orc.Oracle(p, variant="crpow")
    o.run_cycles(8)
    ref = o.state()
    with sgh.SGHSolver(p) as s:
        s.set_state(st)
        s.run(1)
        one = sgh.compared_fields(s.get_state())
        s.run(7)
        got = s.get_state()
    flat = sgh.compared_fields(got)
    flat.update(corner_force=got["corner_force"], node_mass=got["node_mass"])
    for k in ("coords", "vel", "den", "pres", "sie", "sspd", "vol", "corner_force", "node_mass"):
        assert np.array_equal(np.asarray(flat[k]).ravel(), np.asarray(ref[k]).ravel()), k
    with sgh.SGHSolver(p, fp_mode=sgh.FP_FMA) as s:
        s.set_state(st)
        s.run(1)
        fma = sgh.compared_fields(s.get_state())
    assert_fields(fma, one, 1e-12, keys=("coords", "vel", "den", "pres", "sie"), label="fma %s" % (shape,))


@pytest.mark.parametrize("shape", [(2, 2, 1), (7, 9, 5), (20, 23, 25), (21, 22, 25)])
@pytest.mark.parametrize("kind", ["hypo", "mixed"])
def test_strength_force_equals_the_restatement(oracle_built, lib_built, shape, kind):
    """Exact mode with a strength model, on both sides of the force pass's
    change-over (11500 | 11550 elements), bit for bit against the C restatement."""
    import copy

    from fierro_gb300 import problems, sgh
    from oracle import orc
    p = problems.with_strength(_deck(shape, 5), "hypo", 3.0)
    if kind == "mixed":  # a gas without strength in half of the box, carried over by the force pass
        gas, f = copy.copy(p.materials[0]), copy.copy(p.fills[0])
        gas.strength = "none"
        p.materials.append(gas)
        f.volume, f.mat_id = "box", 1
        f.x2, f.y2, f.z2 = 0.5, 1.1, 0.9
        p.fills.append(f)
    o = orc.Oracle(p, variant="crpow")
    o.run_cycles(5)
    ref = o.state()
    with sgh.SGHSolver(p) as s:
        s.set_state(sgh.setup(p))
        s.run(5)
        got = s.get_state()
    flat = sgh.compared_fields(got)
    flat.update(corner_force=got["corner_force"])
    for k in ("coords", "vel", "den", "pres", "sie", "sspd", "vol", "corner_force"):
        assert np.array_equal(np.asarray(flat[k]).ravel(), np.asarray(ref[k]).ravel()), k
    for b, k in ((0, "stress0"), (1, "stress")):
        assert np.array_equal(got["elem_stress"][b].ravel(), np.asarray(ref[k]).ravel()), k


@pytest.mark.parametrize("n", [2, 3, 11, 21, 22])
def test_adjoint_on_both_sides_of_the_lane_passes(lib_built, n):
    """8, 27, 1331, 9261 (eight lanes) and 10648 elements (one thread): the replayed
    forces equal the tape bit for bit, and the gradient agrees with automatic
    differentiation of the scheme in plain torch, 64 bits: two evaluations of the
    same derivative, a few hundred roundings a cycle apart over 30 cycles (1e-10)."""
    from perf import cases
    case = dict(kind="adjoint", deck="sedov", n=n, mode="exact", cycles=30, chunk=7)
    state = cases.prepare(case, 5)
    cases.run(state)
    state["solver"].adj_verify(True)
    got = cases.run(state)
    assert state["solver"].adj_stats()["force_mismatches"] == 0
    want = cases.exact(case, 5)
    for k in ("dsie", "dgamma", "dvel"):
        w = want[k].cpu().numpy()
        assert np.linalg.norm(got[k] - w) <= 1e-10 * np.linalg.norm(w), k
    state["solver"].close()


@pytest.mark.parametrize("pieces", [(108,), (23, 41, 5, 7, 2, 30), (24, 1, 3, 4, 76)])
def test_runs_in_graphs_of_several_cycles(lib_built, tmp_path, pieces):
    """A handle that has run for a while launches four cycles at a time: any split of a run
    gives what stepping stage by stage gives, across a restart and a stop at the
    final time too."""
    from fierro_gb300 import sgh
    p = _deck((7, 5, 6), 200)
    st = sgh.setup(p)
    with sgh.SGHSolver(p) as a, sgh.SGHSolver(p) as b:
        a.set_state(st)
        b.set_state(st)
        for n in pieces:
            assert a.run(n) == n
        b.run_stages(2 * sum(pieces))
        want, got = b.get_state(), a.get_state()
        assert a.time() == b.time()
        for k in want:
            assert np.array_equal(got[k], want[k]), k
        a.checkpoint(str(tmp_path / "a"))
        ran = a.run(21)  # up to the deck's final time
        want = a.get_state()
        b.run(70)
        b.restart(str(tmp_path / "a"))
        assert b.run(21) == ran
        got = b.get_state()
        for k in want:
            assert np.array_equal(got[k], want[k]), k
    p.params.time_final = 0.12
    with sgh.SGHSolver(p) as a:
        a.set_state(st)
        ran = a.run(66) + a.run(301)
        assert a.time()[0] >= 0.12 and ran == a.time()[3] < 367 and a.run(9) == 0
