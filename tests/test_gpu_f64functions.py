"""The table-driven float64 exponential, logarithm and arctangent of the float64
kernels against NumPy's, over the tables' ranges and the special values beyond
them."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
FUNCTIONS = (np.exp, np.log, np.arctan)


def _run(x):
    from veris_gb300 import _abi
    d = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    out = torch.empty(3 * x.size, dtype=torch.float64, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    assert _abi.load().veris_f64_functions_check(d.data_ptr(), x.size, out.data_ptr(), s) == 0
    return out.cpu().numpy().reshape(3, x.size)


def _edges(points):
    """The points and their neighbouring float64 values."""
    p = np.asarray(points, dtype=np.float64)
    return np.concatenate([p, np.nextafter(p, -np.inf), np.nextafter(p, np.inf)])


# table entry (half a unit), remainder and its series (about one more), NumPy's own (one): 3 units in the last
# place; of 1 where the result is below 1 for the two whose table entry and remainder may cancel
@pytest.mark.parametrize("which,x", (
    (0, np.concatenate([np.random.default_rng(1).uniform(-700, 700, 1 << 18), np.random.default_rng(2).normal(0, 1, 1 << 18),
                        _edges(np.arange(-2048, 2049) * np.log(2) / 1024), _edges([-699.99, 0.0, 1e-300, 699.99])])),
    (1, np.concatenate([np.random.default_rng(3).uniform(1, 8, 1 << 18), 2.0 ** np.random.default_rng(4).uniform(0, 63, 1 << 16),
                        np.abs(_edges(1 + np.arange(0, 1025) / 256)), _edges([1.0, 2.0, 2.0 ** 63])])),
    (2, np.concatenate([np.random.default_rng(5).uniform(1, 3.6, 1 << 18), _edges(1 + np.arange(0, 334) / 128),
                        _edges([1.0, 3.6])])),
), ids=("exp", "log", "atan"))
def test_within_three_units(which, x):
    got, ref = _run(x)[which], FUNCTIONS[which](x)
    unit = np.spacing(np.abs(ref)) if which == 0 else np.spacing(np.maximum(np.abs(ref), 1.0))
    assert (np.abs(got - ref) <= 3 * unit).all()


def test_beyond_the_tables():
    x = np.array([0.0, -0.0, 1.0, -1.0, 0.5, 709.7, 710.0, -745.0, -746.0, 1e300, -1e300, 5e-324, np.inf, -np.inf, np.nan])
    got = _run(x)
    with np.errstate(all="ignore"):
        for k, f in enumerate(FUNCTIONS):
            ref = f(x)
            same = np.isfinite(ref)
            np.testing.assert_allclose(got[k][same], ref[same], rtol=1e-15)
            assert np.array_equal(got[k][~same], ref[~same], equal_nan=True)
