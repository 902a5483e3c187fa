"""The register walk's own preparation (rounding to float32 on the integer pipe)
and the compiled form that the library takes on grids beyond L2."""
import numpy as np
import pytest

from tests.test_gpu_small_grids import prepared

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


# ice at rest: sigma12 after one subcycle is sigma12 (alpha - 1) / alpha of its float32 value, to the bit
def test_conversion_rounds_to_nearest():
    from veris_gb300.evp_solver import evp_solver_fast
    st = prepared(60, 61, 4)
    v = st.variables
    for k in ("uIce", "vIce"):
        setattr(v, k, torch.zeros_like(v.uIce))
    rng = np.random.default_rng(0)
    f = rng.uniform(1, 2, v.sigma12.numel()).astype(np.float32).astype(np.float64)
    half = 2.0 ** -24                              # half a unit in the last place of [1, 2): ties both ways
    x = (f + half * rng.integers(-1, 2, f.size)) * 2.0 ** rng.integers(-60, 60, f.size)
    x *= rng.choice((-1.0, 1.0), f.size)
    x[:12] = (0.0, -0.0, 1e-320, 1e-42, -3e-39, 1.1754943e-38, 1.1754944e-38, 3e38, 3.5e38, -1e300, np.inf, 2.0 - 2.0 ** -25)
    v.sigma12 = torch.from_numpy(x.reshape(v.sigma12.shape)).cuda()
    got = evp_solver_fast(st, "f32", "walk", n_subcycles=1, rows=0)[4]
    alpha = st.settings.evpAlpha
    want = (v.sigma12.float() * np.float32(alpha - 1.0)) * np.float32(1.0 / alpha)
    assert torch.equal(got, want)


# one grid on each side of the line (3 * 2^19 padded cells)
@pytest.mark.parametrize("nx,ny", ((1600, 800), (1804, 903)))
def test_forms_give_the_same_values_around_the_line(nx, ny):
    from veris_gb300.evp_solver import evp_solver_fast
    st = prepared(nx, ny, 2)
    a = evp_solver_fast(st, "f32", "walk", n_subcycles=4, rows=0)
    for variant, rows in ((2, 0), (3, 23)):
        b = evp_solver_fast(st, "f32", "walk", n_subcycles=4, rows=rows, variant=variant)
        assert all(torch.equal(x, y) for x, y in zip(a, b))
