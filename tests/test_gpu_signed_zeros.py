"""Signs of zeros.  The reference's sums begin from 0.0, so a sum of negative zeros is
+0.0: node velocities, positions and divergences carry the restatement's signs bit for
bit in exact mode, and a batch (one thread per element) gives a handle's bits (eight
lanes) in both modes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a, dtype=np.float64).reshape(-1).view(np.int64)


def _deck(shape):
    """Cold gas, no boundary conditions, u = -y with -0.0 on the plane y = 0 and in v
    and w.  One element has no neighbours, so its viscous forces are zeros too: the
    corner forces of a node with a negative normal and a velocity above the Riemann
    velocity are -0.0 in every component that matters."""
    from fierro_gb300 import mesh, problems
    p = problems.noh(mesh=mesh.box_mesh(*shape), cycles=3)
    p.boundaries = []
    p.fills[0].velocity = "cartesian"
    p.fills[0].u = p.fills[0].v = p.fills[0].w = -0.0
    p.fills[0].sie = 0.0
    p.materials[0].csmin = 1.0
    return p


def _rz_deck():
    """A parallelogram that touches the axis at one node, whose normal points inwards:
    there a force of -0.0 stays (no hoop term is added on the axis)."""
    from fierro_gb300 import problems
    from fierro_gb300.mesh import HexMesh
    xy = np.array([[0.0, 0.0], [-2.0, 1.0], [-3.0, 1.125], [-1.0, 0.125]])
    p = problems.noh_rz(mesh=HexMesh(xy, np.array([[0, 1, 2, 3]])), cycles=3)
    p.boundaries = []
    p.fills[0].velocity = "cartesian"
    p.fills[0].u = p.fills[0].v = -0.0
    p.fills[0].sie = 0.0
    p.materials[0].csmin = 1.0
    return p


def _start(sgh, p):
    st = sgh.setup(p)
    v = np.full_like(st["node_vel"], -0.0)
    v[..., 0] = -st["node_coords"][..., 1]
    st["node_vel"][...] = v
    return st


def _oracle(p, st, cycles):
    from oracle import orc
    o = orc.Oracle(p, variant="crpow")
    o.set(orc.ORC_NODE_VEL, st["node_vel"])
    o.run_cycles(cycles)
    return o.state()


KEYS = ("coords", "vel", "div", "sie", "pres", "corner_force")


def _flat(got):
    from fierro_gb300 import sgh
    f = sgh.compared_fields(got)
    f.update(corner_force=got["corner_force"], div=got["elem_div"])
    return f


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 1), (3, 2, 2)])
def test_hex_signs(oracle_built, lib_built, shape):
    from fierro_gb300 import sgh
    p = _deck(shape)
    st = _start(sgh, p)
    ref = _oracle(p, st, 2)
    for mode in (0, 1):
        with sgh.Batch([p], fp_mode=mode) as b:
            b.set_state(0, st)
            b.run(2)
            batch = _flat(b.get_state(0))
        with sgh.SGHSolver(p, fp_mode=mode) as s:
            s.set_state(st)
            s.run(2)
            handle = _flat(s.get_state())
        for k in KEYS:
            assert np.array_equal(_bits(batch[k]), _bits(handle[k])), (mode, k)
            if mode == 0 and k != "corner_force":
                assert np.array_equal(_bits(handle[k]), _bits(ref[k])), k


def test_quad_signs(oracle_built, lib_built):
    from fierro_gb300 import sgh
    p = _rz_deck()
    st = _start(sgh, p)
    ref = _oracle(p, st, 2)
    with sgh.SGHSolver(p) as s:
        s.set_state(st)
        s.run(2)
        got = _flat(s.get_state())
    for k in KEYS:
        assert np.array_equal(_bits(got[k]), _bits(ref[k])), k
