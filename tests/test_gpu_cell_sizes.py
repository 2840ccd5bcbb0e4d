"""The force pass's cube root over the exponent range of volumes: cells of 1e-78 to
1e57, among them the 1e-60 at which a single-precision term once left its range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-25, 1e-20, 3e-20, 1e-13, 1e-6, 1.0, 1e6, 1e20])
def test_corner_forces_of_cells_of_any_size(oracle_built, lib_built, scale):
    """Exact mode, one stage, bit for bit against the restatement; the Mach switch is
    below its clamp (speed 1, sound speed about 100), so the length enters the force."""
    from fierro_gb300 import mesh, problems, sgh
    from oracle import orc
    m = mesh.box_mesh(6, 5, 7, jitter=0.1, seed=3, permute=True)
    m.coords *= scale
    p = problems.noh(mesh=m, cycles=1)
    p.boundaries = []
    p.fills[0].sie = 1e4
    p.fills[0].den = 1.0 / scale ** 2  # impedances of order one, above the fuzz
    p.params.dt_start, p.params.dt_min = 1e-4 * scale, 1e-9 * scale
    o = orc.Oracle(p, variant="crpow")
    o.run_stages(1)
    ref = o.state()
    with sgh.SGHSolver(p) as s:
        s.set_state(sgh.setup(p))
        s.run_stages(1)
        got = s.get_state()["corner_force"].reshape(-1, 3)
    assert np.isfinite(ref["corner_force"]).all() and (ref["vol"] > 0.0).all()
    assert np.array_equal(got, ref["corner_force"])
