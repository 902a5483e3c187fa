"""The float64 subcycle loop on grids whose work units are dealt out over all
CTA slots (two rows a unit and up), against the plain loop."""
import pytest

from tests import golden_io as G

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from veris_gb300 import _abi
    return _abi.load()


def prepared(nx, ny, seed, **settings):
    """A moving state with the dynamics preparation done."""
    from veris_gb300 import area_mass, dynamics_routines, dynsolver
    from veris_gb300.state import VerisState
    from veris_gb300.synthetic import config_settings, make_state
    st = VerisState.from_numpy(make_state(nx, ny, seed=seed, init_velocity=0.1, init_stress=500.0, ice_lat=20.0),
                               config_settings("c1_4deg", **settings))
    v = st.variables
    v.SeaIceMassC, v.SeaIceMassU, v.SeaIceMassV = area_mass.SeaIceMass(st)
    v.AreaW, v.AreaS = area_mass.AreaWS(st)
    v.WindForcingX, v.WindForcingY = dynsolver.WindForcingXY(st)
    v.SeaIceStrength = dynamics_routines.SeaIceStrength(st)
    return st


# one strip and many, the last strip one column wide, rows that do not divide,
# fewer rows than slots, as many, and the first sizes with full pieces again
@pytest.mark.parametrize("nx,ny", ((4, 4), (5, 29), (33, 35), (61, 93), (120, 60), (251, 133), (455, 31), (760, 380)))
def test_f64_loop_on_small_grids(lib, nx, ny):
    from veris_gb300.state import Call
    st = prepared(nx, ny, nx + ny)
    c = Call(st)
    n = 7
    ws, wsb = c.workspace(lib.veris_evp_fast_workspace_bytes(c.refs()[0], 8))
    pws, pwsb = c.workspace(lib.veris_evp_workspace_bytes(c.refs()[0], 8))
    ref = c.empty(5)
    assert lib.veris_evp_solver_f64(*c.refs(), n, *[t.data_ptr() for t in ref], pws, pwsb, c.stream) == 0
    first = None
    try:
        for rows in (24, 16, 32):
            assert lib.veris_evp_f64_tile_rows(rows) == 0
            out = c.empty(5)
            assert lib.veris_evp_fast_solver_f64(*c.refs(), n, *[t.data_ptr() for t in out], ws, wsb, c.stream) == 0
            if first is None:
                first = out
            assert all(torch.equal(a, b) for a, b in zip(out, first))
    finally:
        lib.veris_evp_f64_tile_rows(0)
    for a, b in zip(first, ref):
        assert G.rel_err(a.cpu().numpy(), b.cpu().numpy()) <= 1e-10
