"""The float64 adjoint sweep with P4 of each subcycle fused with P1 of the one
before it, against segments of one subcycle (the two run apart), on grids on
either side of the counts at which a pass releases its successor early."""
import pytest

from tests.test_gpu_small_grids import lib, prepared  # noqa: F401

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# up to three CTAs of 32 x 4 points per SM, up to six, more; last rows and columns that do not fill one
@pytest.mark.parametrize("nx,ny", ((5, 29), (61, 93), (363, 157), (445, 223), (601, 330)))
@pytest.mark.parametrize("basal", (False, True))
def test_fused_passes_match_separate_ones(lib, nx, ny, basal):  # noqa: F811
    from veris_gb300 import adjoint
    st = prepared(nx, ny, nx + ny, **({"basalDragK2": 15.0} if basal else {}))
    shape = st.variables.uIce.shape
    gen = torch.Generator(device="cuda").manual_seed(nx)
    lam = {k: torch.randn(shape, dtype=torch.float64, device="cuda", generator=gen)
           for k in ("uIce", "vIce", "sigma1", "sigma2", "sigma12")}
    fused = adjoint.evp_adjoint(st, lam, n_subcycles=4, tape=True)
    apart = adjoint.evp_adjoint(st, lam, n_subcycles=4, checkpoint_every=1)
    for a, b in zip(fused[:2], apart[:2]):
        for k in a:
            assert (a[k] - b[k]).abs().max().item() <= 1e-12 * b[k].abs().max().item(), k
    for k, x in fused[2].items():
        assert abs(x - apart[2][k]) <= 1e-12 * abs(apart[2][k]), k
