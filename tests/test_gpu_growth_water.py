"""Growth on warps of open water (their own short form), of ice, and mixed, with
inputs that a zero concentration must still spread, against the oracle."""
import numpy as np
import pytest

from oracle import veris_oracle as O
from tests import golden_io as G

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
OUT = ("hIceMean", "hSnowMean", "Area", "TSurf", "EmPmR", "forc_salt", "Qsw", "Qnet", "SeaIceLoad", "IcePenetSW", "rh")


def _state(ny, **settings):
    from types import SimpleNamespace
    from veris_gb300.synthetic import config_settings, make_state
    a = make_state(40, ny, seed=ny, ice_lat=40.0)
    rng = np.random.default_rng(ny)
    shape = a["iceMask"].shape
    a["TSurf"] = rng.uniform(215.0, 276.0, shape)
    a["ATemp"] = rng.uniform(230.0, 290.0, shape)
    a["SWdown"] = rng.uniform(0.0, 500.0, shape)
    a["Qnet"] = rng.uniform(-300.0, 900.0, shape)
    a["theta"] = rng.uniform(271.0, 274.0, shape)
    a["hSnowMean"] *= rng.integers(0, 2, shape)
    a["os_hIceMean"] = rng.uniform(0, 1e-3, shape) * (rng.random(shape) > 0.9)
    some = rng.random(shape)
    a["Area"][some > 0.95] = 0.0      # thickness without concentration, and the other way round
    a["hIceMean"][some < 0.05] = 0.0
    return SimpleNamespace(variables=SimpleNamespace(**a), settings=config_settings("c1_4deg", **settings))


def _compare(st):
    from veris_gb300.growth import Growth
    from veris_gb300.state import VerisState
    gpu = Growth(VerisState.from_numpy(vars(st.variables), st.settings))
    with np.errstate(all="ignore"):
        ref = O.Growth(st)
    for name, a, b in zip(OUT, gpu, ref):
        a = a.cpu().numpy()
        ok = np.isfinite(b)
        assert np.array_equal(ok, np.isfinite(a)), name
        assert G.rel_err(np.where(ok, a, 0.0), np.where(ok, b, 0.0)) <= 1e-10, name   # the parity of every routine


# rows of whole and broken warps; reference salinity on and off; another number of categories
@pytest.mark.parametrize("ny,settings", ((31, {}), (61, dict(saltIce_ref=4.0)), (124, dict(nITC=3, recip_nITC=1 / 3)),
                                         (124, dict(minTIce=-20.0, wetAlbTemp=-1.0, dtempFrz_dS=-0.05))))
def test_growth(ny, settings):
    _compare(_state(ny, **settings))


# the settings of the six iterations, beyond their range: float64 iterations take over
def test_growth_far_from_the_root():
    st = _state(61)
    st.variables.SWdown *= 1e30
    _compare(st)


# the short form against the general one, which a warp takes when one of its points has ice: the same rounding
# up to contraction and constants formed on the host, and not-a-number in the same places
@pytest.mark.parametrize("name", (None, "precip", "snowfall", "evap", "Qsw", "LWdown", "theta", "Qnet"))
def test_short_form_equals_the_general_one(name):
    from veris_gb300.growth import Growth
    from veris_gb300.state import VerisState
    st = _state(61)
    v = st.variables
    for k in ("hIceMean", "hSnowMean", "Area"):
        getattr(v, k)[3:9] = 0.0
    if name:
        getattr(v, name)[3:9, 5:50] = np.nan
    short = Growth(VerisState.from_numpy(vars(v), st.settings))
    for k, x in (("hIceMean", 1.5), ("Area", 0.9)):
        getattr(v, k)[3:9, ::32] = x
    general = Growth(VerisState.from_numpy(vars(v), st.settings))
    cols = [j for j in range(65) if j % 32]
    for out, a, b in zip(OUT, short, general):
        a, b = (t.cpu().numpy()[3:9][:, cols] for t in (a, b))
        ok = np.isfinite(b)
        assert np.array_equal(ok, np.isfinite(a)), out
        assert G.rel_err(np.where(ok, a, 0.0), np.where(ok, b, 0.0)) <= 1e-12, out
