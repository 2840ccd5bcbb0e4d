"""The lane passes against the one-thread-per-element passes of the same handle
(FIERRO_LANES=0), bit for bit in both modes, signs of zeros included: quads, strength
models and hexes at sizes that leave remainders of a warp's elements."""
import copy

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hex(shape, strength):
    from fierro_gb300 import mesh, problems
    m = mesh.box_mesh(*shape, length=(1.0, 1.1, 0.9), jitter=0.15, seed=sum(shape), permute=True)
    p = problems.noh(max(shape), mesh=m, cycles=20)
    p.materials[0].q2ex = 0.4
    p.fills[0].sie = 0.02
    if strength == "none":
        return p
    p = problems.with_strength(p, "hyper" if strength == "hyper" else "hypo", 3.0)
    if strength == "mixed":  # a gas without strength in half of the box
        gas, f = copy.copy(p.materials[0]), copy.copy(p.fills[0])
        gas.strength = "none"
        p.materials.append(gas)
        f.volume, f.mat_id = "box", 1
        f.x2, f.y2, f.z2 = 0.5, 1.1, 0.9
        p.fills.append(f)
    return p


def _quad(shape, strength):
    from fierro_gb300 import mesh, problems
    m = mesh.quad_mesh(*shape, length=(1.0, 1.2), jitter=0.1, seed=sum(shape), permute=True)
    p = problems.noh_rz(max(shape), mesh=m, cycles=20)
    p.materials[0].q2ex = 0.4
    p.fills[0].sie = 0.02
    return problems.with_strength(p, strength, 3.0) if strength != "none" else p


CASES = [(_hex, s, k) for s in ((1, 1, 1), (3, 3, 3), (7, 9, 5), (20, 20, 25)) for k in ("none", "hypo", "mixed", "hyper")]
CASES += [(_quad, s, k) for s in ((1, 1), (3, 1), (4, 2), (3, 3), (31, 17), (90, 100)) for k in ("none", "hypo")]


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("deck,shape,strength", CASES, ids=lambda v: getattr(v, "__name__", str(v)))
def test_lanes_equal_one_thread(lib_built, monkeypatch, mode, deck, shape, strength):
    from fierro_gb300 import sgh
    p = deck(shape, strength)
    st = sgh.setup(p)
    got, times = [], []
    for lanes in ("1", "0"):
        monkeypatch.setenv("FIERRO_LANES", lanes)
        with sgh.SGHSolver(p, fp_mode=mode) as s:
            s.set_state(st)
            s.run(12)
            got.append(s.get_state())
            times.append(s.time())
    assert times[0] == times[1]
    for k in got[0]:
        a, b = (np.ascontiguousarray(g[k]).reshape(-1).view(np.int64) for g in got)
        assert np.array_equal(a, b), k
