"""A batch's states by the transfer kernels against the staged route (host loops
through pinned memory): the same bits in every field, for instances whose sizes
leave remainders of the kernels' blocks, with several materials, arrays left out
and arrays off the 8-byte boundary; a refused state changes nothing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIDES = (1, 2, 5, 7, 11)  # 1 to 1,331 elements; blocks of 64 (forces), 128 (padding) and 256


def _problems():
    from fierro_gb300 import mesh, problems
    ps = [problems.sedov(n, jitter=0.1, seed=n, permute=True, cycles=6) for n in SIDES]
    m = mesh.box_mesh(14, 6, 3, length=(7.0, 3.0, 1.7), jitter=0.1, seed=3, permute=True)
    return ps + [problems.triple_point(m, cycles=6)]


def _shifted(a, by):
    raw = np.zeros(a.nbytes + 16, dtype=np.uint8)
    at = (-raw.ctypes.data) % 8 + by
    out = raw[at:at + a.nbytes].view(a.dtype).reshape(a.shape)
    out[...] = a
    return out


def _run(ps, states, cycles, shift=0):
    from fierro_gb300 import sgh
    states = [{k: _shifted(v, shift) if shift else v for k, v in st.items()} for st in states]
    with sgh.Batch(ps, fp_mode=0) as b:
        for i, st in enumerate(states):
            b.set_state(i, st)
        before = [b.get_state(i) for i in range(len(b))]
        b.run(cycles)
        return before, [b.get_state(i) for i in range(len(b))]


@pytest.mark.parametrize("div", [True, False])
def test_transfer_kernels_equal_the_staged_route(lib_built, monkeypatch, div):
    from fierro_gb300 import sgh
    ps = _problems()
    states = [sgh.setup(p) for p in ps]
    rng = np.random.RandomState(1)
    for st in states:
        st["elem_div"][...] = rng.rand(*st["elem_div"].shape)
        if not div:
            del st["elem_div"]
    got = {}
    for route, staged, shift in (("kernels", "0", 0), ("staged", "1", 0), ("unaligned", "0", 4)):
        monkeypatch.setenv("FIERRO_STAGED_TRANSFERS", staged)
        got[route] = _run(ps, states, 6, shift)
    for route in ("staged", "unaligned"):
        for a, b in zip(got["kernels"], got[route]):
            for i, (x, y) in enumerate(zip(a, b)):
                for k in x:
                    assert np.array_equal(x[k], y[k], equal_nan=True), (route, i, k)


def test_refused_state_changes_nothing(lib_built):
    from fierro_gb300 import sgh
    ps = _problems()
    states = [sgh.setup(p) for p in ps]

    def spoil(st, key, idx, value):
        bad = {k: v.copy() for k, v in st.items()}
        bad[key].reshape(-1)[idx] = value
        for k in ("node_vel", "elem_den"):
            bad[k] += 1.0
        return bad

    with sgh.Batch(ps, fp_mode=0) as b:
        for i, st in enumerate(states):
            b.set_state(i, st)
        for i, st in enumerate(states):
            for key, text in (("elem_mat_id", "material id"), ("elem_vol", "volume"), ("elem_mass", "element mass"),
                              ("node_mass", "node mass"), ("elem_stress", "stress")):
                bad = spoil(st, key, -1, 99 if key in ("elem_mat_id", "elem_stress") else -1.0)
                with pytest.raises(sgh.FierroError, match=text):
                    b.set_state(i, bad)
        after = [b.get_state(i) for i in range(len(b))]
    for i, st in enumerate(states):
        for k in ("node_coords", "node_vel", "node_mass", "elem_den", "elem_pres", "elem_sie", "elem_vol", "elem_mass"):
            assert np.array_equal(after[i][k], st[k]), (i, k)
