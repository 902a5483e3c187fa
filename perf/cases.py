"""The work that a user of veris_gb300 has it do, as measurable cases.

Each case is one call through the package's public entry points on a seeded
synthetic state (the kinds, sizes and subcycle counts are those of
``veris_gb300.synthetic.CONFIGS`` and of the tests, and sizes between them):

* ``step``       the drop-in step ``model.step(state)``, float64;
* ``coupled``    ``HostCoupledStep``: a host-resident state uploaded, stepped by
                 the captured engine and downloaded, float64 or float32;
* ``evp``        the drop-in ``evp_solver(state)``, float64, any rheology option;
* ``evp_fast``   ``evp_solver_fast``: the engine's subcycle loop, float64 tiles
                 or the float32 register walk;
* ``evp_adjoint`` the taped reverse mode of the subcycle loop;
* ``advection``, ``growth``, ``growth_adjoint``, ``bulk``: single routines;
* ``ensemble``   batched subcycles of many small domains.

``exact`` restates the same calls in plain float64 torch.
"""
import math
from types import SimpleNamespace

import torch

from veris_gb300 import adjoint, model
from veris_gb300.advection import Advection
from veris_gb300.engine import SeaIceStep
from veris_gb300.ensemble import Ensemble
from veris_gb300.evp_solver import evp_solver, evp_solver_fast
from veris_gb300.growth import Growth
from veris_gb300.heat_flux_MITgcm import bulkf_formula_lanl
from veris_gb300.host import HOST_INPUTS, HOST_OUTPUTS, HostCoupledStep
from veris_gb300.settings import default_settings, with_timesteps
from veris_gb300.state import VerisState

EVP_OUT = ("uIce", "vIce", "sigma1", "sigma2", "sigma12")
ICE = ("hIceMean", "hSnowMean", "Area", "TSurf")


def listed():
    return [
        # one step of the 4-degree setup through the drop-in routines: many small launches
        dict(name="step_4deg", kind="step", nx=90, ny=40, n=120, dt=3600.0),
        # one step of a 1-degree ocean model that keeps its fields on the host
        dict(name="coupled_1deg", kind="coupled", nx=360, ny=180, n=300, dt=3600.0, precision="f64"),
        # the drop-in rheology of the 1-degree model
        dict(name="evp_1deg", kind="evp", nx=360, ny=180, n=60, dt=3600.0),
        # the drop-in rheology with adaptive relaxation, free slip, landfast ice and turned
        # stresses, on a regional grid of odd size
        dict(name="evp_options", kind="evp", nx=443, ny=221, n=30, dt=3600.0, adaptive=True, no_slip=False,
             basal=True, turn=True),
        # subcycles of the quarter-degree step in float64 (the benchmark's workload)
        dict(name="evp_f64_quarterdeg", kind="evp_fast", nx=1440, ny=720, n=25, dt=1800.0, precision="f64"),
        # subcycles of the tenth-degree step in float32: the largest grid
        dict(name="evp_f32_tenthdeg", kind="evp_fast", nx=3600, ny=1800, n=20, dt=600.0, precision="f32"),
        # gradients of the subcycle loop in a 1-degree trajectory
        dict(name="evp_adjoint_1deg", kind="evp_adjoint", nx=360, ny=180, n=30, dt=3600.0, precision="f64"),
        # transport of thickness, snow and concentration at a quarter degree
        dict(name="advection_quarterdeg", kind="advection", nx=1440, ny=720, dt=1800.0),
        # thermodynamics at a quarter degree
        dict(name="growth_quarterdeg", kind="growth", nx=1440, ny=720, dt=1800.0),
        # gradients of the thermodynamics on an odd grid
        dict(name="growth_adjoint", kind="growth_adjoint", nx=721, ny=359, dt=3600.0),
        # the forcing producer over the quarter-degree ocean
        dict(name="bulk_quarterdeg", kind="bulk", nx=1440, ny=720, precision="f64"),
        # an ensemble of small domains of uneven sizes
        dict(name="ensemble_12", kind="ensemble", members=12, n=60, dt=3600.0, sizes=7),
    ]


def draw(rng):
    """Another case of the same kinds: sizes over the listed ranges (log-uniform, odd ones among
    them), subcycle counts so that the work stays below the largest listed case's."""
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("step", "coupled", "evp", "evp_fast", "evp_adjoint", "advection", "growth",
                       "growth_adjoint", "bulk", "ensemble"))
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randint(2, 12), n=log(10, 60), dt=3600.0, sizes=rng.randint(0, 10 ** 6))
    top = {"step": 240, "coupled": 900, "evp": 900, "evp_adjoint": 500}.get(kind, 1440)
    nx = log(64, top)
    ny = max(33, min(nx, int(nx * rng.uniform(0.4, 0.7))))
    c = dict(kind=kind, nx=nx, ny=ny)
    if kind != "bulk":
        c["dt"] = 3600.0 if nx < 800 else 1800.0
    cells = nx * ny
    if kind in ("evp_fast", "evp_adjoint", "coupled", "bulk"):
        c["precision"] = rng.choice(("f64", "f64", "f32"))
    if kind == "evp_fast" and c["precision"] == "f32":
        c["nx"] = log(64, 3600)
        c["ny"] = max(33, c["nx"] // 2 + rng.randint(-15, 0))
        c["dt"] = 3600.0 if c["nx"] < 800 else 600.0
        cells = c["nx"] * c["ny"]
    most = {"step": 120, "coupled": min(300, 18_000_000 // cells), "evp": min(90, 4_000_000 // cells),
            "evp_fast": min(120, (100 if c.get("precision") == "f32" else 20) * 1_000_000 // cells),
            "evp_adjoint": min(40, 2_000_000 // cells)}
    if kind in most:
        c["n"] = log(max(2, most[kind] // 3), max(3, most[kind]))
    if kind == "evp":
        c["adaptive"], c["no_slip"] = rng.random() < 0.25, rng.random() < 0.75
        c["basal"], c["turn"] = rng.random() < 0.3, rng.random() < 0.3
    return c


# ------------------------------------------------------------------- inputs

def _settings(case):
    s = default_settings(pStar=27500.0, cStar=20.0, PlasDefCoeff=2.0)
    with_timesteps(s, case.get("dt", 3600.0), case.get("dt", 3600.0), case.get("n", 1))
    if case.get("adaptive"):
        s.useAdaptiveEVP = True
    if case.get("no_slip") is False:
        s.noSlip = False
    if case.get("basal"):
        s.basalDragK2 = 15.0
    if case.get("turn"):
        s.airTurnAngle = s.waterTurnAngle = 25.0
        s.sinWat, s.cosWat = math.sin(math.radians(25.0)), math.cos(math.radians(25.0))
    return s


def _sx(a, di):
    """a at (i + di, j), periodic over the padded array, as the host model's roll."""
    return torch.roll(a, -di, 0)


def _sy(a, dj):
    return torch.roll(a, -dj, 1)


def _fill(a):
    """The cyclic x halo, a new array."""
    return torch.cat((a[-4:-2], a[2:-2], a[2:4]), 0)


class _Inputs:
    """Seeded fields with the distributions of ``veris_gb300.synthetic.make_state``, on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed))

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.g, device="cuda", dtype=torch.float64)

    def uniform(self, lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, generator=self.g, device="cuda", dtype=torch.float64)

    def smooth(self, std, sigma, nx, ny):
        """Gaussian noise smoothed over ``sigma`` cells, with standard deviation ``std``."""
        f = self.normal(nx, ny)
        kx = torch.fft.fftfreq(nx, device="cuda", dtype=torch.float64)[:, None]
        ky = torch.fft.rfftfreq(ny, device="cuda", dtype=torch.float64)[None, :]
        f = torch.fft.irfft2(torch.fft.rfft2(f) * torch.exp(-2.0 * (math.pi * sigma) ** 2 * (kx ** 2 + ky ** 2)),
                             s=(nx, ny))
        return f * (std / f.std())


def _fields(nx, ny, seed, moving=True, wind=1.0):
    r = _Inputs(seed)
    NX, NY = nx + 4, ny + 4
    like = dict(device="cuda", dtype=torch.float64)
    one = torch.ones(NX, NY, **like)
    degtom = 6370e3 * math.pi / 180.0
    dlat = 160.0 / ny
    yt = -80.0 + (torch.arange(NY, **like) - 1.5) * dlat
    dx, dy = 360.0 / nx * degtom, dlat * degtom
    cost = torch.cos(torch.deg2rad(yt.clamp(-89.5, 89.5)))
    cosu = torch.cos(torch.deg2rad((yt + 0.5 * dlat).clamp(-89.5, 89.5)))

    noise = r.smooth(1.0, max(1.0, nx / 45.0), nx, ny)
    mask = torch.zeros(NX, NY, **like)
    mask[2:-2, 2:-2] = (noise > noise.flatten().kthvalue(max(1, noise.numel() // 4)).values).double()
    mask = _fill(mask)
    mU, mV = _fill(mask * _sx(mask, -1)), _fill(mask * _sy(mask, -1))

    v = {"iceMask": mask, "iceMaskU": mU, "iceMaskV": mV, "maskInC": mask.clone(), "maskInU": mU.clone(),
         "maskInV": mV.clone(), "R_low": r.uniform(50.0, 5000.0, NX, NY) * mask}
    v["fCori"] = (2 * math.pi / 43082.0 * torch.sin(torch.deg2rad(yt)) * one).contiguous()
    for k in ("dxC", "dxU", "dxG", "dxV"):
        v[k] = dx * one
    for k in ("dyC", "dyU", "dyG", "dyV"):
        v[k] = dy * one
    v["rA"] = v["rAu"] = dx * dy * cost * one
    v["rAv"] = dx * dy * cosu * one
    rAz = v["rA"] + _sx(v["rA"], -1)
    v["rAz"] = 0.25 * _sy(rAz, -1)
    for k in ("dxC", "dyC", "dxG", "dyG", "dxU", "dyU", "dxV", "dyV", "rA", "rAu", "rAv", "rAz"):
        v["recip_" + k] = 1.0 / v[k]
    for k in ("k1AtC", "k2AtC", "k1AtZ", "k2AtZ", "Fu", "Fv"):
        v[k] = torch.zeros(NX, NY, **like)

    polar = (yt.abs() > 55.0).double() * one
    h = _fill(torch.exp(math.log(1.5) - 0.125 + 0.5 * r.normal(NX, NY)) * polar * mask)
    v["hIceMean"] = h
    v["Area"] = _fill(torch.clamp(h / 0.5, max=1.0) * r.uniform(0.8, 1.0, NX, NY) * (h > 0))
    v["hSnowMean"] = 0.2 * h
    v["TSurf"] = 273.0 * one
    v["uWind"] = _fill(r.smooth(8.0 * wind, 3.0, NX, NY))
    v["vWind"] = _fill(r.smooth(8.0 * wind, 3.0, NX, NY))
    v["wSpeed"] = torch.sqrt(v["uWind"] ** 2 + v["vWind"] ** 2)
    v["uOcean"] = _fill(r.smooth(0.1, 3.0, NX, NY) * mU)
    v["vOcean"] = _fill(r.smooth(0.1, 3.0, NX, NY) * mV)
    v["theta"] = torch.where(h > 0, -1.8, r.uniform(0.0, 10.0, NX, NY)) + 273.15
    v["ATemp"] = r.uniform(-25.0, 0.0, NX, NY) + 273.15
    v["SWdown"] = r.uniform(0.0, 300.0, NX, NY)
    v["LWdown"] = 250.0 * one
    v["aqh"] = r.uniform(0.3e-3, 2.5e-3, NX, NY)
    v["precip"] = r.uniform(0.0, 3e-8, NX, NY)
    v["snowfall"] = v["precip"] * r.uniform(0.0, 1.0, NX, NY)
    v["evap"] = -r.uniform(0.0, 3e-8, NX, NY)
    v["ocSalt"] = r.uniform(33.0, 35.0, NX, NY)
    v["Qnet"] = r.uniform(-50.0, 150.0, NX, NY)
    v["Qsw"] = -v["SWdown"]
    v["ssh_an"] = _fill(r.smooth(0.1, 3.0, NX, NY))
    v["surfPress"] = _fill(101325.0 + r.smooth(500.0, 3.0, NX, NY))
    scale = 1.0 if moving else 0.0
    v["uIce"] = _fill(scale * r.smooth(0.1, 2.0, NX, NY) * mU)
    v["vIce"] = _fill(scale * r.smooth(0.1, 2.0, NX, NY) * mV)
    for k in ("sigma1", "sigma2"):
        v[k] = scale * r.smooth(500.0, 2.0, NX, NY) * mask
    v["sigma12"] = scale * r.smooth(500.0, 2.0, NX, NY) * mask
    for k in ("runoff", "SeaIceMassC", "SeaIceMassU", "SeaIceMassV", "SeaIceStrength", "AreaW", "AreaS",
              "WindForcingX", "WindForcingY", "os_hIceMean", "os_hSnowMean", "SeaIceLoad", "IcePenetSW",
              "OceanStressU", "OceanStressV", "EmPmR", "saltflux", "forc_salt_surface_ice"):
        v[k] = torch.zeros(NX, NY, **like)
    v["recip_hIceMean"] = 1.0 / torch.sqrt(h ** 2 + 0.01)
    return {k: t.contiguous() for k, t in v.items()}


def _member_shapes(case):
    """Uneven member sizes, nx in 64..512 and ny in 64..384 by 32, as the ensemble workload's."""
    g = torch.Generator()
    g.manual_seed(int(case["sizes"]))
    pick = lambda top: [64 + 32 * int(k) for k in torch.randint(0, (top - 64) // 32 + 1, (case["members"],), generator=g)]
    return list(zip(pick(512), pick(384)))


def _lam(shape, seed, names):
    r = _Inputs(seed + 77)
    return {k: r.normal(*shape) for k in names}


def _air(case, seed):
    """Winds, air and sea states over the ocean, as the forcing kernel of a setup has them."""
    r = _Inputs(seed)
    shape = (case["nx"] + 4, case["ny"] + 4)
    a = [r.smooth(8.0, 3.0, *shape), r.smooth(8.0, 3.0, *shape), r.uniform(-25.0, 25.0, *shape) + 273.15,
         r.uniform(0.3e-3, 1.5e-2, *shape), r.uniform(-1.8, 28.0, *shape) + 273.15]
    if case["precision"] == "f32":
        a = [t.float() for t in a]
    return a + [torch.ones_like(a[0])]


def _with_preparation(v, s):
    w = SimpleNamespace(**v)
    for group in (_mass, _areas, _strength, _wind):
        for k, t in group(w, s).items():
            v[k] = t.contiguous()
            setattr(w, k, v[k])
    return v


def prepare(case, seed):
    kind, s = case["kind"], _settings(case)
    if kind == "bulk":
        return SimpleNamespace(case=case, state=VerisState({}, s), args=_air(case, seed))
    if kind == "ensemble":
        members = []
        for m, (nx, ny) in enumerate(_member_shapes(case)):
            v = _fields(nx, ny, seed * 1009 + m, wind=0.5 + (m % 8) / 7.0)
            members.append(VerisState(v, s))
        ens = Ensemble(members, case["n"])
        ens.set_launch(6, 4)   # 32-row walks, four CTAs per SM: the tuner's choice for such members
        return SimpleNamespace(case=case, ens=ens, members=members)
    v = _fields(case["nx"], case["ny"], seed)
    if kind in ("evp", "evp_fast", "evp_adjoint"):
        _with_preparation(v, s)
    st = SimpleNamespace(case=case, state=VerisState(v, s))
    if kind == "coupled":
        st.host = HostCoupledStep(SeaIceStep(st.state, precision=case["precision"]))
        st.h_in, st.h_out = st.host.host_buffers()
    elif kind == "evp_adjoint":
        st.lam = _lam(st.state.shape, seed, EVP_OUT)
    elif kind == "growth_adjoint":
        st.lam = _lam(st.state.shape, seed, ICE)
    return st


# ---------------------------------------------------------------------- run

def run(st):
    case, kind = st.case, st.case["kind"]
    if kind == "step":
        now = VerisState(dict(vars(st.state.variables)), st.state.settings)
        v = model.step(now).variables
        return {k: getattr(v, k) for k in HOST_OUTPUTS}
    if kind == "coupled":
        return st.host.step(st.h_in, st.h_out)
    if kind == "evp":
        return dict(zip(EVP_OUT, evp_solver(st.state)))
    if kind == "evp_fast":
        form = "smem" if case["precision"] == "f64" else "walk"
        return dict(zip(EVP_OUT, evp_solver_fast(st.state, precision=case["precision"], form=form, rows=0)))
    if kind == "evp_adjoint":
        init, const, drag = adjoint.evp_adjoint(st.state, st.lam, precision=case["precision"], tape=True)
        return {"init": init, "const": const, "drag": drag}
    if kind == "advection":
        return dict(zip(ICE, Advection(st.state)))
    if kind == "growth":
        return dict(zip(_GROWTH_OUT, Growth(st.state)))
    if kind == "growth_adjoint":
        return adjoint.growth_adjoint(st.state, st.lam)
    if kind == "bulk":
        return dict(zip(_BULK_OUT, bulkf_formula_lanl(st.state, *st.args)))
    st.ens.step()
    return [st.ens.state(m) for m in range(len(st.members))]


def work(case):
    """Each input read and each output written once; the arithmetic of the loops."""
    kind = case["kind"]
    cells = (sum(nx * ny for nx, ny in _member_shapes(case)) if kind == "ensemble" else case["nx"] * case["ny"])
    size = 4 if case.get("precision") == "f32" or kind == "ensemble" else 8
    n = case.get("n", 0)
    fields = {"step": 48, "coupled": 48, "evp": 20, "evp_fast": 20, "evp_adjoint": 42, "advection": 11, "growth": 33,
              "growth_adjoint": 23, "bulk": 14, "ensemble": 20}[kind]
    flops = {"step": 1000 + 120 * n, "coupled": 1000 + 120 * n, "evp": 120 * n, "evp_fast": 120 * n,
             "evp_adjoint": 330 * n, "advection": 180, "growth": 700, "growth_adjoint": 1400, "bulk": 500,
             "ensemble": 120 * n}[kind]
    if kind == "coupled":
        size = 8
    return {"bytes": float(cells * fields * size), "flops": float(cells * flops)}


# -------------------------------------------------- the same in plain torch

_GROWTH_OUT = ("hIceMean", "hSnowMean", "Area", "TSurf", "EmPmR", "forc_salt_surface_ice", "Qsw", "Qnet", "SeaIceLoad",
               "IcePenetSW", "recip_hIceMean")
_BULK_OUT = ("flwupa", "flha", "fsha", "df0dT", "ust", "vst", "evp", "ssq", "dEvdT")


def _top(a, b):
    """max(a, b) with a plain number b; its derivative where a > b only."""
    return torch.where(a > b, a, torch.full_like(a, b))


def _sqrt0(x):
    """The square root, with derivative 0 at 0."""
    pos = x > 0
    return torch.where(pos, torch.sqrt(torch.where(pos, x, torch.ones_like(x))), torch.zeros_like(x))


def _pick(where, a, b):
    """One of two plain numbers per point (``torch.where`` of two numbers is float32)."""
    like = dict(dtype=torch.float64, device=where.device)
    return torch.where(where, torch.as_tensor(a, **like), torch.as_tensor(b, **like))


def _mass(v, s):
    m = s.rhoIce * v.hIceMean + s.rhoSnow * v.hSnowMean
    return {"SeaIceMassC": m, "SeaIceMassU": 0.5 * (m + _sx(m, -1)), "SeaIceMassV": 0.5 * (m + _sy(m, -1))}


def _areas(v, s):
    return {"AreaW": 0.5 * (v.Area + _sx(v.Area, -1)), "AreaS": 0.5 * (v.Area + _sy(v.Area, -1))}


def _strength(v, s):
    return {"SeaIceStrength": s.pStar * v.hIceMean * torch.exp(-s.cStar * (1 - v.Area)) * v.iceMask}


def _wind(v, s):
    si, co = math.sin(math.radians(s.airTurnAngle)), math.cos(math.radians(s.airTurnAngle))
    ur = v.uWind - 0.5 * (v.uIce + _sx(v.uIce, 1))
    vr = v.vWind - 0.5 * (v.vIce + _sy(v.vIce, 1))
    sq = ur ** 2 + vr ** 2
    speed = torch.where(sq < s.wSpeedMin ** 2, s.wSpeedMin, torch.sqrt(sq))
    cd = _pick(v.fCori < 0, s.airIceDrag_south, s.airIceDrag) * s.rhoAir * speed
    sg = torch.sign(v.fCori)
    tx, ty = cd * (co * ur - sg * si * vr), cd * (co * vr + sg * si * ur)
    tx = 0.5 * (tx + _sx(tx, -1)) * v.iceMaskU
    ty = 0.5 * (ty + _sy(ty, -1)) * v.iceMaskV
    phi = s.gravity * v.ssh_an + v.surfPress * s.recip_rhoSea
    return {"WindForcingX": tx * v.AreaW - v.SeaIceMassU * v.recip_dxC * (phi - _sx(phi, -1)),
            "WindForcingY": ty * v.AreaS - v.SeaIceMassV * v.recip_dyC * (phi - _sy(phi, -1))}


def _ocean_drag(v, s, u, w, drag):
    dc = _pick(v.fCori < 0, drag[1], drag[0]) * s.rhoSea
    du, dv = (u - v.uOcean) * v.maskInU, (w - v.vOcean) * v.maskInV
    t = 0.25 * ((du + _sx(du, 1)) ** 2 + (dv + _sy(dv, 1)) ** 2)
    return torch.where(dc ** 2 * t > s.cDragMin ** 2, dc * _sqrt0(t), s.cDragMin) * v.iceMask


def _evp(v, s, n, drag=None):
    """``n`` subcycles of the modified EVP rheology."""
    drag = drag or (s.waterIceDrag, s.waterIceDrag_south)
    u, w, s1, s2, s12 = (getattr(v, k) for k in EVP_OUT)
    u0, w0, rdt = u, w, s.recip_deltatDyn
    rsq = 1.0 / s.PlasDefCoeff ** 2
    wet = v.iceMask + _sx(v.iceMask, -1)
    wet = wet + _sy(wet, -1)
    rwet = torch.where(wet > 0, 1.0 / wet, 0.0)
    mz = v.iceMask * _sx(v.iceMask, -1)
    mz = mz * _sy(mz, -1)
    hU, hV = v.iceMaskU - _sy(v.iceMaskU, -1), v.iceMaskV - _sx(v.iceMaskV, -1)
    sg = torch.sign(v.fCori)
    lmU = torch.where(v.SeaIceMassU != 0, 1.0, v.SeaIceMassU)
    lmV = torch.where(v.SeaIceMassV != 0, 1.0, v.SeaIceMassV)
    aC = aZ = bU = bV = None
    for _ in range(n):
        e11 = (_sx(u, 1) - u) * v.recip_dxU * v.maskInC
        e22 = (_sy(w, 1) - w) * v.recip_dyV * v.maskInC
        us, ww = _sy(u, -1), _sx(w, -1)
        e12 = 0.5 * ((u - us) * v.recip_dyU + (w - ww) * v.recip_dxV) * mz
        if s.noSlip:
            e12 = e12 + ((u + us) * v.recip_dyU * hU + (w + ww) * v.recip_dxV * hV)
        c = v.rAz * e12 ** 2
        c = c + _sx(c, 1)
        c = 0.25 * v.recip_rA * (c + _sy(c, 1))
        delta = _sqrt0((e11 + e22) ** 2 + rsq * ((e11 - e22) ** 2 + 4.0 * c))
        zeta = 0.5 * (v.SeaIceStrength * (1 + s.tensileStrFac)) / (delta + s.deltaMin)
        press = (v.SeaIceStrength * (1 - s.pressReplFac)
                 + 2.0 * zeta * delta * s.pressReplFac / (1 + s.tensileStrFac)) * (1 - s.tensileStrFac)
        if s.useAdaptiveEVP:
            fac = s.deltatDyn * 4 * (math.pi * s.aEvpCoeff) ** 2
            aC = torch.sqrt(zeta * fac / v.SeaIceMassC.clamp(min=1e-4) * v.recip_rA) * v.iceMask
            aC = aC.clamp(min=s.aEVPalphaMin)
            aZ = 0.5 * (aC + _sy(aC, -1))
            aZ = 0.5 * (aZ + _sx(aZ, -1))
            bU, bV = 0.5 * (aC + _sx(aC, -1)) * rdt, 0.5 * (aC + _sy(aC, -1)) * rdt
        else:
            aC = aZ = s.evpAlpha
            bU = bV = s.evpBeta * rdt
        z = zeta + _sx(zeta, -1)
        z = rwet * (z + _sy(z, -1))
        s1 = (s1 * (aC - 1) + 2 * zeta * (e11 + e22) - press) / aC * v.iceMask
        s2 = (s2 * (aC - 1) + 0.5 * zeta * (e11 - e22)) / aC * v.iceMask
        s12 = (s12 * (aZ - 1) + 0.5 * z * e12) / aZ
        a, b, d, f = 0.5 * (s1 + s2) * v.dyV, s12 * v.dxV, 0.5 * (s1 - s2) * v.dxU, s12 * v.dyU
        sdx = (a - _sx(a, -1) - b + _sy(b, 1)) * v.recip_rAu
        sdy = (d - _sy(d, -1) - f + _sx(f, 1)) * v.recip_rAv
        cd = _ocean_drag(v, s, u, w, drag)
        cdW, cdS = _sx(cd, -1), _sy(cd, -1)
        du, dv = v.uOcean - u, v.vOcean - w
        turn = sg * s.sinWat * 0.5
        fx = v.WindForcingX + (0.5 * (cd + cdW) * s.cosWat * v.uOcean - turn * (
            cd * 0.5 * (du + _sy(du, 1)) + cdW * 0.5 * (_sx(du, -1) + _sy(_sx(du, -1), 1))) * lmU) * v.AreaW
        fy = v.WindForcingY + (0.5 * (cd + cdS) * s.cosWat * v.vOcean + turn * (
            cd * 0.5 * (dv + _sx(dv, 1)) + cdS * 0.5 * (_sy(dv, -1) + _sx(_sy(dv, -1), 1))) * lmV) * v.AreaS
        fv = v.SeaIceMassC * v.fCori * 0.5 * (w + _sy(w, 1))
        fu = v.SeaIceMassC * v.fCori * 0.5 * (u + _sx(u, 1))
        fx = fx + 0.5 * (fv + _sx(fv, -1))
        fy = fy - 0.5 * (fu + _sy(fu, -1))
        dU = v.SeaIceMassU * (bU + rdt) + v.AreaW * 0.5 * (cd + cdW) * s.cosWat
        dV = v.SeaIceMassV * (bV + rdt) + v.AreaS * 0.5 * (cd + cdS) * s.cosWat
        if s.basalDragK2:
            um, vm = u * v.maskInU, w * v.maskInV
            t = 0.25 * (um ** 2 + _sx(um, 1) ** 2 + vm ** 2 + _sy(vm, 1) ** 2)
            x = 10.0 * (v.hIceMean - v.R_low.abs() * v.Area / s.basalDragK1)
            cb = (s.basalDragK2 / torch.sqrt(t + s.basalDragU0 ** 2) * torch.log(torch.exp(x) + 1.0) * 0.1
                  * torch.exp(-s.cBasalStar * (1.0 - v.Area)))
            cb = torch.where(v.Area > 0.01, cb, 0.0)
            dU = dU + v.AreaW * 0.5 * (cb + _sx(cb, -1))
            dV = dV + v.AreaS * 0.5 * (cb + _sy(cb, -1))
        dU = torch.where(dU == 0, 1.0, dU)
        dV = torch.where(dV == 0, 1.0, dV)
        if not s.noSlip:
            sp = 0.5 * torch.sqrt((u + _sx(u, 1)) ** 2 + (w + _sy(w, 1)) ** 2)
            spU = torch.where(v.AreaW > 0, 0.5 * (sp + _sx(sp, -1)), 0.0)
            spV = torch.where(v.AreaS > 0, 0.5 * (sp + _sy(sp, -1)), 0.0)
            cU = (2 - _sx(v.iceMaskU, -1) - _sx(v.iceMaskU, 1)) * v.iceMaskU
            cV = (2 - _sy(v.iceMaskV, -1) - _sy(v.iceMaskV, 1)) * v.iceMaskV
            dU = dU + v.SeaIceMassU * s.sideDragCoeff * cU / (spU + s.sideDragU0)
            dV = dV + v.SeaIceMassV * s.sideDragCoeff * cV / (spV + s.sideDragU0)
        un = v.iceMaskU * (bU * v.SeaIceMassU * u + v.SeaIceMassU * rdt * u0 + fx + sdx) / dU
        wn = v.iceMaskV * (bV * v.SeaIceMassV * w + v.SeaIceMassV * rdt * w0 + fy + sdy) / dV
        u, w = _fill(un), _fill(wn)
    return {"uIce": u, "vIce": w, "sigma1": s1, "sigma2": s2, "sigma12": s12}


def _ocean_stress(v, s):
    cd = _ocean_drag(v, s, v.uIce, v.vIce, (s.waterIceDrag, s.waterIceDrag_south))
    si, co = math.sin(math.radians(s.waterTurnAngle)), math.cos(math.radians(s.waterTurnAngle))
    du, dv = v.uIce - v.uOcean, v.vIce - v.vOcean
    a, b = cd * 0.5 * (dv + _sy(dv, 1)), cd * 0.5 * (du + _sx(du, 1))
    sg = torch.sign(v.fCori)
    return {"OceanStressU": _fill(0.5 * (cd + _sx(cd, -1)) * co * du - sg * si * 0.5 * (a + _sy(a, -1))),
            "OceanStressV": _fill(0.5 * (cd + _sy(cd, -1)) * co * dv + sg * si * 0.5 * (b + _sx(b, -1)))}


def _flux(s, f, m, t, cfl):
    """Superbee-limited flux through the faces of axis 0."""
    R = (f[1:] - f[:-1]) * m[1:]
    Rjm, Rj, Rjp = R[:-2], R[1:-1], R[2:]
    t, cfl = t[2:-1], cfl[2:-1]
    cr = torch.where(t > 0, Rjm, Rjp)
    near = Rj.abs() * s.CrMax > cr.abs()
    cr = torch.where(near, cr / torch.where(near, Rj, torch.ones_like(Rj)),
                     torch.sign(cr) * s.CrMax * torch.sign(Rj))
    cr = torch.maximum((2 * cr).clamp(max=1.0), cr.clamp(max=2.0)).clamp(min=0.0)
    F = torch.zeros_like(f)
    F[2:-1] = t * (f[2:-1] + f[1:-2]) * 0.5 - t.abs() * ((1 - cr) + cfl * cr) * Rj * 0.5
    return F


def _advect(v, s):
    uT, vT = v.uIce * (v.dyG * v.iceMaskU), v.vIce * (v.dxG * v.iceMaskV)
    cu, cv = (v.uIce * s.deltatTherm * v.recip_dxC).abs(), (v.vIce * s.deltatTherm * v.recip_dyC).abs()
    out = {}
    for k in ICE[:3]:
        f = getattr(v, k)
        F = _fill(_flux(s, f, v.iceMaskU * v.maskInU, uT, cu))
        f = f - s.deltatTherm * v.maskInC * v.recip_rA * (_sx(F, 1) - F)
        G = _fill(_flux(s, f.T, (v.iceMaskV * v.maskInV).T, vT.T, cv.T).T)
        out[k] = (f - s.deltatTherm * v.maskInC * v.recip_rA * (_sy(G, 1) - G)) * v.iceMask
    return out


def _clean_up(v, s):
    h, hs, A = v.hIceMean.clamp(min=0), v.hSnowMean.clamp(min=0), v.Area.clamp(min=0)
    thin = h <= s.hIce_min
    h, hs = torch.where(thin, 0.0, h), torch.where(thin, 0.0, hs)
    A = torch.where((h == 0) & (hs == 0), 0.0, A.clamp(min=s.Area_min)).clamp(max=1.0)
    return {"hIceMean": h, "hSnowMean": hs, "Area": A, "TSurf": torch.where(thin, s.celsius2K, v.TSurf),
            "os_hIceMean": (-v.hIceMean).clamp(min=0), "os_hSnowMean": (-v.hSnowMean).clamp(min=0)}


def _solve4temp(v, s, hI, hS, Tin, TempFrz):
    """Surface temperature by six Newton steps -> (T, flux to the ocean, flux to the air, penetrating)."""
    aa1, aa2, bb1, P = 2663.5, 12.537, 0.622, 100000.0
    cc0 = 10.0 ** aa2
    cc1, cc2 = cc0 * aa1 * bb1 * P * math.log(10.0), cc0 * (1 - bb1)
    d1, d1i = s.dalton * s.cpAir * s.rhoAir, s.dalton * s.lhSublim * s.rhoAir
    Tmelt, zero = s.celsius2K, torch.zeros_like(hI)
    Ta, ug = _top(v.ATemp, s.celsius2K + s.minTAir), _top(v.wSpeed, s.wSpeedMin)
    ice, snow = hI > 0, hS > 0
    em = _pick(snow, s.snowEmiss, s.iceEmiss)
    d3, lw = em * s.stefBoltz, em * _top(v.LWdown, s.minLWdown)
    wet, south = Tin >= Tmelt + s.wetAlbTemp, v.fCori < 0
    aI = torch.where(south, _pick(wet, s.wetIceAlb_south, s.dryIceAlb_south),
                     _pick(wet, s.wetIceAlb, s.dryIceAlb))
    aS = torch.where(south, _pick(wet, s.wetSnowAlb_south, s.drySnowAlb_south),
                     _pick(wet, s.wetSnowAlb, s.drySnowAlb))
    alb = torch.where(hS > s.hCut, aS, torch.where(hS == 0, aI, aI + hS / s.hCut * (aS - aI)))
    pen = torch.where(snow, zero, s.shortwave * torch.exp(-1.5 * hI))
    penSW, absSW = -(1 - alb) * pen * v.SWdown, (1 - alb) * (1 - pen) * v.SWdown
    k = s.iceConduct * s.snowConduct / (s.snowConduct * torch.where(ice, hI, 1.0) + s.iceConduct * hS)

    def fluxes(t):
        svp = 10.0 ** (aa2 - aa1 / t)
        qs = bb1 * svp / (P - (1 - bb1) * svp)
        c3 = 10.0 ** (aa1 / t)
        dqs = cc1 * c3 / ((cc2 - c3 * P) ** 2 * t * t)
        Fia = -lw - absSW + t ** 4 * d3 + d1 * ug * (t - Ta) + d1i * ug * (qs - v.aqh)
        return k * (TempFrz - t), Fia, 4 * d3 * t ** 3 + d1 * ug + d1i * ug * dqs

    T = Tin
    for _ in range(6):
        Fc, Fia, dF = fluxes(T)
        T = T + (Fc - Fia) / (k + dF)
        T = torch.where(T < Tmelt, T, torch.full_like(T, Tmelt))
        T = _top(T, s.celsius2K + s.minTIce)
    Fc, Fia, _ = fluxes(T)
    up = Fc > 0
    return (torch.where(ice, T, Tin), torch.where(ice & up, Fc, zero), torch.where(ice & ~up, Fia, zero),
            torch.where(ice, penSW, zero))


def _growth(v, s):
    qi, qs = 1 / (s.rhoIce * s.lhFusion), 1 / (s.rhoSnow * s.lhFusion)
    keep = ((v.hIceMean != 0) & (v.Area != 0)).double()
    h0, hs0, A0 = v.hIceMean * keep, v.hSnowMean * keep, v.Area * keep
    zero = torch.zeros_like(h0)
    rregA = 1 / torch.sqrt(A0 ** 2 + s.Area_reg)
    hIa = _top(torch.where(h0 > 0, h0 * rregA, zero), 0.05)
    hSa = torch.where(h0 > 0, hs0 * rregA, zero)
    rhIa = A0 / torch.sqrt(h0 ** 2 + s.hIce_reg)
    TempFrz = s.tempFrz + s.dtempFrz_dS * v.ocSalt + s.celsius2K
    sums = [zero, zero, zero, zero]
    for l in range(s.nITC):
        f = (2 * l + 1) * s.recip_nITC
        sums = [a + b for a, b in zip(sums, _solve4temp(v, s, hIa * f, hSa * f, v.TSurf, TempFrz))]
    TSurf = sums[0] * s.recip_nITC
    Fio, Fia, pen = (t * s.recip_nITC * A0 for t in sums[1:])
    cold = (A0 > 0) & (sums[0] / s.nITC < s.celsius2K)
    snowAcc = torch.where(cold, v.snowfall + v.precip, v.snowfall) * s.rhoFresh2rhoSnow
    rain = torch.where(cold, 0.0, v.precip)
    gUnder = torch.where(A0 == 0, zero, Fio * qi)
    melt = -Fia * qs
    allMelt = melt * s.deltatTherm >= hs0
    toSnow = torch.where(allMelt, -hs0 * s.recip_deltatTherm / qs, Fia)
    melt = torch.where(allMelt, hs0 * s.recip_deltatTherm, melt)
    Fia = Fia - toSnow
    gNet = (gUnder + Fia * qi) * rregA
    mltf = 1 + (s.McPheeTaperFac - 1) / (1 + torch.exp((A0 - 0.4) * (7 / 0.4)))
    gML = -s.stantonNr * s.uStarBase * s.rhoSea * s.cpWater * (torch.maximum(v.theta, TempFrz) - TempFrz) * mltf * qi
    gOW = qi * v.Qnet
    dh = gNet * A0 + gOW * (1 - A0) + gML
    dA = torch.where((gOW > 0) & ((A0 > 0) | (dh > 0)), gOW * (1 - A0), 0.5 * rhIa * gOW * (1 - A0))
    dA = dA * _pick((gOW > 0) & ((A0 > 0) | (dh > 0)) & (v.fCori < 0), s.recip_h0_south, s.recip_h0)
    dA = dA + torch.where(gML <= 0, 0.5 * rhIa * gML, zero)
    dA = dA + torch.where((gNet <= 0) & (h0 > 0), 0.5 * rhIa * gNet * A0, zero)
    step = v.iceMask * s.deltatTherm
    A, h, hs = A0 + dA * step, h0 + dh * step, hs0 + (snowAcc - melt) * A0 * step
    A = _top(torch.where(A < 1, A, torch.ones_like(A)), 0.0)
    h, hs = _top(h, 0.0), _top(hs, 0.0)
    alive = ((h != 0) & (A != 0)).double()
    A, h, hs = A * alive, h * alive, hs * alive
    flood = _top((hs * s.rhoSnow + h * s.rhoIce) * s.recip_rhoSea - h, 0.0)
    h, hs = h + flood, hs - flood * s.rhoIce2rhoSnow
    dH = h - h0
    E_out = (A0 * (Fia + Fio + pen) + (1 - A0) * v.Qnet) * s.deltatTherm
    fac = torch.where((v.ocSalt > 0) & (v.ocSalt > s.saltIce_ref), 1 - s.saltIce_ref / v.ocSalt, 1.0)
    fresh = -dH * s.rhoIce2rhoFresh * fac + (hs0 + snowAcc * A0 * s.deltatTherm - hs) / s.rhoFresh2rhoSnow
    salt = ((dH + v.os_hIceMean) * v.ocSalt.clamp(max=s.saltIce_ref) * v.iceMask * s.rhoIce * s.recip_deltatTherm)
    EmPmR = v.iceMask * (((-v.evap - v.precip) * (1 - A0) - rain * A0 - v.runoff - fresh / s.deltatTherm) * s.rhoFresh
                         + (v.os_hIceMean * s.rhoIce + v.os_hSnowMean * s.rhoSnow) * s.recip_deltatTherm)
    return {"hIceMean": h, "hSnowMean": hs, "Area": A, "TSurf": TSurf, "EmPmR": EmPmR,
            "forc_salt_surface_ice": EmPmR * v.ocSalt / s.rhoFresh + salt, "Qsw": pen * A0 + v.Qsw * (1 - A0),
            "Qnet": (E_out - dH / qi) * s.recip_deltatTherm, "SeaIceLoad": h * s.rhoIce + hs * s.rhoSnow,
            "IcePenetSW": pen, "recip_hIceMean": 1 / torch.sqrt(h ** 2 + s.hIce_reg)}


def _step(v, s):
    for part in (_mass, _areas, _wind, _strength, lambda v, s: _evp(v, s, s.nEVPsteps), _ocean_stress, _advect,
                 _clean_up, _growth):
        vars(v).update(part(v, s))
    for k in ("hIceMean", "hSnowMean", "Area", "forc_salt_surface_ice", "Qnet"):
        setattr(v, k, _fill(getattr(v, k)))
    return {k: getattr(v, k) for k in HOST_OUTPUTS}


def _bulk(s, uw, vw, ta, qa, tsf):
    aln, czol = math.log(2.0 / 10.0), 10.0 * s.karman * s.grav
    us = torch.sqrt(uw * uw + vw * vw)
    usm = us.clamp(min=1.0)
    t0 = ta * (1.0 + s.zvir * qa)
    ssq = 3.797915 * torch.exp(s.latvap * (7.93252e-6 - 2.166847e-3 / tsf)) / 1013.0
    dp, dq = ta - tsf + s.gamma_blk * 2.0, qa - ssq
    rdn = s.karman / math.log(10.0 / 0.0005)
    ustar, tstar, qstar = rdn * usm, rdn * dp, rdn * dq
    for _ in range(5):
        x = czol / ustar ** 2 * (tstar / t0 + qstar / (1.0 / s.zvir + qa))
        x = x.abs().clamp(max=10.0) * torch.sign(x)
        st = 0.5 + 0.5 * torch.sign(x)
        xsq = torch.sqrt((1.0 - 16.0 * x).abs()).clamp(min=1.0)
        r = torch.sqrt(xsq)
        heat = 2.0 * torch.log(0.5 * (1.0 + xsq))
        pm = -5.0 * x * st + (1.0 - st) * (2.0 * torch.log(0.5 * (1.0 + r)) + heat - 2.0 * torch.atan(r) + math.pi / 2)
        ph = -5.0 * x * st + (1.0 - st) * heat
        rd, rh = rdn / (1.0 + rdn * (aln - pm) / s.karman), rdn / (1.0 + rdn * (aln - ph) / s.karman)
        ustar, qstar, tstar = rd * usm, rh * dq, rh * dp
    csha, clha = s.rhoAir * s.cpdair * us * rh * rd, s.rhoAir * s.latvap * us * rh * rd
    devdt = clha * ssq * 2.166847e-3 / (tsf * tsf)
    lw = s.ocean_emissivity * s.stefBoltz
    cdn = 2.7e-3 / usm + 0.142e-3 + 0.0764e-3 * usm
    return (lw * tsf ** 4, clha * dq, csha * dp, -4.0 * lw * tsf ** 3 - csha - s.latvap * devdt,
            s.rhoAir * cdn * us * uw, s.rhoAir * cdn * us * vw, -clha * dq / s.latvap, ssq, devdt)


def _gradients(outs, lam, inputs):
    total = sum((outs[k] * lam[k]).sum() for k in lam)
    return [torch.zeros_like(x) if g is None else g
            for x, g in zip(inputs, torch.autograd.grad(total, inputs, allow_unused=True))]


def exact(case, seed):
    kind, s = case["kind"], _settings(case)
    if kind == "bulk":
        return dict(zip(_BULK_OUT, _bulk(s, *[t.double() for t in _air(case, seed)[:5]])))
    if kind == "ensemble":
        out = []
        for m, (nx, ny) in enumerate(_member_shapes(case)):
            v = _with_preparation(_fields(nx, ny, seed * 1009 + m, wind=0.5 + (m % 8) / 7.0), s)
            out.append(_evp(SimpleNamespace(**v), s, case["n"]))
        return out
    v = _fields(case["nx"], case["ny"], seed)
    shape = tuple(v["iceMask"].shape)
    if kind in ("evp", "evp_fast", "evp_adjoint"):
        _with_preparation(v, s)
    w = SimpleNamespace(**v)
    if kind in ("step", "coupled"):
        return _step(w, s)
    if kind in ("evp", "evp_fast"):
        return _evp(w, s, case["n"])
    if kind == "advection":
        return _advect(w, s)
    if kind == "growth":
        return _growth(w, s)
    if kind == "growth_adjoint":
        for k in ICE:
            getattr(w, k).requires_grad_(True)
        g = dict(zip(ICE, _gradients(_growth(w, s), _lam(shape, seed, ICE), [getattr(w, k) for k in ICE])))
        return {**g, "TSurf": None}   # the first guess of a converged iteration: nothing but rounding
    drag = [torch.tensor(c, dtype=torch.float64, device="cuda", requires_grad=True)
            for c in (s.waterIceDrag, s.waterIceDrag_south)]
    for k in EVP_OUT + adjoint.EVP_FIELDS:
        getattr(w, k).requires_grad_(True)
    names = EVP_OUT + adjoint.EVP_FIELDS
    g = _gradients(_evp(w, s, case["n"], drag), _lam(shape, seed, EVP_OUT), [getattr(w, k) for k in names] + drag)
    return {"init": dict(zip(EVP_OUT, g)), "const": dict(zip(adjoint.EVP_FIELDS, g[5:])),
            "drag": {"waterIceDrag": g[-2], "waterIceDrag_south": g[-1]}}
