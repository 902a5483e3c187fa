"""A member's state copied out of the batch workspace, on sizes beside the copy
kernel's (fewer columns than threads, one more than a multiple, more rows than CTAs)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SIZES = ((4, 4), (5, 124), (7, 125), (900, 9), (33, 260))


@pytest.mark.parametrize("n_sub", (0, 1))
def test_initial_and_later_state_of_every_member(n_sub):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from veris_gb300.ensemble import EVP_STATE, Ensemble
    from veris_gb300.evp_solver import evp_solver_fast
    from veris_gb300.state import VerisState
    from veris_gb300.synthetic import config_settings, make_state
    members = [VerisState.from_numpy(make_state(nx, ny, seed=k, init_velocity=0.05, init_stress=500.0),
                                     config_settings("c4_ensemble")) for k, (nx, ny) in enumerate(SIZES)]
    ens = Ensemble(members, max(n_sub, 1))
    if n_sub:
        ens.step()
    for m, st in enumerate(members):
        got = ens.state(m)
        ref = (evp_solver_fast(st, "f32", form="smem", n_subcycles=n_sub) if n_sub else
               [getattr(st.variables, k).float() for k in EVP_STATE])
        for k, r in zip(EVP_STATE, ref):
            assert torch.equal(got[k], r), (m, k)
