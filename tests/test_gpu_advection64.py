"""The two-launch float64 advection against the oracle: grid sizes around a
warp, a walk and a row block, every halo fill, limiter branches and ties,
in-place outputs, and the limiter bounds that it leaves to the separate passes."""
from types import SimpleNamespace

import numpy as np
import pytest

from oracle import veris_oracle as O
from tests import golden_io as G

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
NAMES = ("hIceMean", "hSnowMean", "Area")


def _state(nx, ny, seed, **settings):
    from veris_gb300.synthetic import config_settings, make_state
    a = make_state(nx, ny, seed=seed, init_velocity=0.4, ice_lat=10.0, wet_y_halo=True)
    rng = np.random.default_rng(seed)
    shape = a["iceMask"].shape
    # plateaus (zero slopes), equal and doubled slopes (the limiter's ties), open water
    a["hIceMean"] = np.round(a["hIceMean"] * 4) / 4 * (rng.random(shape) > 0.1)
    a["Area"][:, ny // 2:] = 0.0
    a["uIce"] *= rng.random(shape) > 0.1
    return SimpleNamespace(variables=SimpleNamespace(**a), settings=config_settings("c1_4deg", **settings))


def _compare(st, call=None):
    from veris_gb300.advection import Advection
    from veris_gb300.state import VerisState
    gpu = VerisState.from_numpy(vars(st.variables), st.settings)
    with np.errstate(all="ignore"):
        ref = O.Advection(st)
    for name, a, b in zip(NAMES, (call or Advection)(gpu), ref):
        a = a.cpu().numpy()
        ok = np.isfinite(b)
        assert np.array_equal(ok, np.isfinite(a)), name
        assert G.rel_err(np.where(ok, a, 0.0), np.where(ok, b, 0.0)) <= 1e-13, name   # a dozen roundings of each value


@pytest.mark.parametrize("fill", (dict(), dict(enable_cyclic_x=False), dict(veros_fill=False)), ids=("x", "none", "xy"))
@pytest.mark.parametrize("nx,ny", ((4, 4), (5, 27), (13, 28), (29, 29), (60, 123), (61, 125), (130, 257)))
def test_sizes_and_fills(nx, ny, fill):
    _compare(_state(nx, ny, nx + ny, **fill))


@pytest.mark.parametrize("CrMax", (2.0, 1.5, 0.5))
def test_limiter_bound(CrMax):
    _compare(_state(45, 70, 3, CrMax=CrMax))


def test_walks_of_eight_rows():
    _compare(_state(800, 403, 9))


def test_in_place():
    def call(st):
        from veris_gb300.state import Call
        c = Call(st)
        v = st.variables
        ws, wsb = c.workspace(c.lib.veris_advection_workspace_bytes(c.refs()[0], 8))
        out = [getattr(v, k) for k in NAMES]
        assert c.lib.veris_advection_f64(*c.refs(), *[t.data_ptr() for t in out], ws, wsb, c.stream) == 0
        return out
    _compare(_state(90, 140, 5), call)


def test_tiny_values():
    st = _state(45, 70, 6)
    st.variables.hIceMean[10:20] *= 1e-310
    _compare(st)


def test_non_finite_values_spread_as_in_the_separate_passes():
    """The passes that a limiter bound under 2 takes; the bound does not change where values are finite."""
    from veris_gb300.advection import Advection
    from veris_gb300.state import VerisState
    got = []
    for CrMax in (1.5, 2.0):
        st = _state(45, 70, 6, CrMax=CrMax)
        v = st.variables
        v.hSnowMean[22, 11] = np.inf
        v.hIceMean[30, 33] = np.nan
        v.uIce[35, 12] = np.nan
        got.append([torch.isfinite(t) for t in Advection(VerisState.from_numpy(vars(v), st.settings))])
    assert all(torch.equal(a, b) for a, b in zip(*got)) and not got[0][0].all()
