"""The drop-in's subcycle loop (``veris_evp_auto_solver_f64``) against the plain
loop: every option, states that the folded form covers and states that it
leaves to the plain tile."""
import itertools

import pytest

from tests import golden_io as G
from tests.test_gpu_small_grids import prepared

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
NAMES = ("uIce", "vIce", "sigma1", "sigma2", "sigma12")


@pytest.fixture(scope="module", autouse=True)
def lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from veris_gb300 import _abi
    return _abi.load()


def solve(lib, st, n, which):
    from veris_gb300.state import Call
    c = Call(st)
    g, p, _f = c.refs()
    size = lib.veris_evp_auto_workspace_bytes(g, p) if which == "auto" else lib.veris_evp_workspace_bytes(g, 8)
    ws, wsb = c.workspace(size)
    out = [torch.full(c.shape, float("nan"), dtype=torch.float64, device="cuda") for _ in NAMES]
    fn = lib.veris_evp_auto_solver_f64 if which == "auto" else lib.veris_evp_solver_f64
    assert fn(*c.refs(), n, *[t.data_ptr() for t in out], ws, wsb, c.stream) == 0
    return out


def compare(lib, st, n, tol):
    for name, a, b in zip(NAMES, solve(lib, st, n, "auto"), solve(lib, st, n, "plain")):
        a, b = a.cpu().numpy(), b.cpu().numpy()
        assert G.rel_err(a, b) <= tol, name


OPTIONS = [dict(zip(("useAdaptiveEVP", "noSlip", "basalDragK2", "turn"), v))
           for v in itertools.product((False, True), (True, False), (0.0, 15.0), (False, True))]


# 1e-10: the parity every float64 form of the loop is held to
@pytest.mark.parametrize("opt", OPTIONS)
@pytest.mark.parametrize("nx,ny,fill", ((37, 60, True), (130, 91, False)))
def test_options(lib, nx, ny, fill, opt):
    import math
    o = dict(opt, veros_fill=fill)
    if o.pop("turn"):
        o.update(waterTurnAngle=25.0, sinWat=math.sin(math.radians(25)), cosWat=math.cos(math.radians(25)))
    compare(lib, prepared(nx, ny, 5, **o), 9, 1e-10)


@pytest.mark.parametrize("nx,ny", ((4, 4), (9, 28), (1203, 611)))
def test_sizes(lib, nx, ny):
    compare(lib, prepared(nx, ny, 3), 4, 1e-10)
    compare(lib, prepared(nx, ny, 3, useAdaptiveEVP=True, noSlip=False, use_coastline=True), 3, 1e-10)


def _metric(v):
    v.dxV = v.dxV * torch.linspace(1.0, 1.1, v.dxV.shape[1], dtype=torch.float64, device="cuda")


def _mask(v):
    v.iceMaskU = v.iceMaskU * 0.5


def _curvature(v):
    v.k1AtC = v.k1AtC + 1e-9


def _infinite(v):
    v.WindForcingX[5, 6] = float("inf")


def _nan_on_land(v):
    v.SeaIceStrength[v.iceMask == 0] = float("nan")


# states for the plain tile: the same operations in the same order, so only the
# contraction of products and sums may differ (1e-12), and not-a-number spreads alike
@pytest.mark.parametrize("spoil", (_metric, _mask, _curvature, _infinite, _nan_on_land))
@pytest.mark.parametrize("opt", (dict(), dict(useAdaptiveEVP=True, noSlip=False, basalDragK2=15.0)))
def test_states_left_to_the_plain_tile(lib, spoil, opt):
    st = prepared(70, 45, 8, **opt)
    spoil(st.variables)
    for name, a, b in zip(NAMES, solve(lib, st, 5, "auto"), solve(lib, st, 5, "plain")):
        assert torch.equal(torch.isfinite(a), torch.isfinite(b)), name
        a, b = torch.where(torch.isfinite(a), a, 0.0), torch.where(torch.isfinite(b), b, 0.0)
        assert G.rel_err(a.cpu().numpy(), b.cpu().numpy()) <= 1e-12, name


# limits in which the two forms' algebra parts: the plain loop itself runs
@pytest.mark.parametrize("opt", (dict(deltaMin=0.0), dict(pressReplFac=0), dict(secondOrderBC=True),
                                 dict(basalDragK2=15.0, basalDragU0=0.0), dict(waterIceDrag=-0.001)))
def test_settings_left_to_the_plain_loop(lib, opt):
    st = prepared(70, 45, 8, **opt)
    for name, a, b in zip(NAMES, solve(lib, st, 3, "auto"), solve(lib, st, 3, "plain")):
        assert torch.equal(torch.nan_to_num(a), torch.nan_to_num(b)), name


def test_no_subcycle_copies_the_state_and_captures(lib):
    from veris_gb300.evp_solver import evp_solver
    st = prepared(70, 45, 8)
    for name, a in zip(NAMES, solve(lib, st, 0, "auto")):
        assert torch.equal(a, getattr(st.variables, name))
    eager = evp_solver(st, 6)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = evp_solver(st, 6)
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(out, eager))


@pytest.mark.parametrize("spoil", (None, _metric))
@pytest.mark.parametrize("opt", (dict(), dict(useAdaptiveEVP=True, noSlip=False)))
def test_residuals(lib, spoil, opt):
    """The residual loop against the plain one: the solve to 1e-10, the sums to the
    1e-8 that squared differences of such states leave."""
    from veris_gb300.state import Call
    st = prepared(130, 91, 6, **opt)
    if spoil:
        spoil(st.variables)
    n, res = 6, {}
    for which in ("plain", "auto"):
        c = Call(st)
        g, p, _f = c.refs()
        size = (lib.veris_evp_auto_residual_workspace_bytes(g, p, n) if which == "auto"
                else lib.veris_evp_residual_workspace_bytes(g, 8, n))
        ws, wsb = c.workspace(size)
        out = c.empty(5) + [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(2)]
        fn = lib.veris_evp_auto_residual_solver_f64 if which == "auto" else lib.veris_evp_residual_solver_f64
        assert fn(*c.refs(), n, *[t.data_ptr() for t in out], ws, wsb, c.stream) == 0
        res[which] = [t.cpu().numpy() for t in out]
    for k in range(5):
        assert G.rel_err(res["auto"][k], res["plain"][k]) <= 1e-10
    for k in (5, 6):
        assert abs(res["auto"][k] / res["plain"][k] - 1).max() <= 1e-8
