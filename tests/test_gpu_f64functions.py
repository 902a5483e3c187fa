"""The table-driven float64 exponential and psi functions of the float64 kernels
against NumPy's, over the tables' ranges and the special values beyond them."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _psi(s):
    """psi_m and psi_h of the bulk formula at s = 1 - 16 huol."""
    x2 = np.sqrt(s)
    x = np.sqrt(x2)
    h = 2 * np.log(0.5 + 0.5 * x2)
    return 2 * np.log(0.5 + 0.5 * x) + h - 2 * np.arctan(x) + np.pi / 2, h


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


# table entry (half a unit), remainder and its series (about one more), NumPy's own (one): 3 units in the last place
def test_exp_within_three_units():
    x = np.concatenate([np.random.default_rng(1).uniform(-700, 700, 1 << 18), np.random.default_rng(2).normal(0, 1, 1 << 18),
                        _edges(np.arange(-2048, 2049) * np.log(2) / 1024), _edges([-699.99, 0.0, 1e-300, 699.99])])
    ref = np.exp(x)
    assert (np.abs(_run(x)[0] - ref) <= 3 * np.spacing(ref)).all()


# values up to 4.5: half a unit each of the table entry and the last sum (9e-16), NumPy's chain of seven
# operations on terms up to 3.9 (eight half units of 4: 3.6e-15)
def test_psi_over_its_range():
    octaves = 2.0 ** np.repeat(np.arange(8), 33) * (1 + np.tile(np.arange(33) / 32, 8))
    x = np.concatenate([np.random.default_rng(3).uniform(1, 161, 1 << 18),
                        1 + 10.0 ** np.random.default_rng(4).uniform(-16, 2.2, 1 << 16),
                        _edges(octaves), _edges([161.0])])
    x = x[(x >= 1) & (x <= 161)]
    for got, ref in zip(_run(x)[1:], _psi(x)):
        assert (np.abs(got - ref) <= 4.5e-15).all()


def test_beyond_the_tables():
    x = np.array([0.0, -0.0, 1.0, -1.0, 0.5, 709.7, 710.0, -745.0, -746.0, 1e300, -1e300, 5e-324, np.inf, -np.inf, np.nan])
    got = _run(x)
    with np.errstate(all="ignore"):
        ref = np.exp(x)
    same = np.isfinite(ref)
    np.testing.assert_allclose(got[0][same], ref[same], rtol=1e-15)
    assert np.array_equal(got[0][~same], ref[~same], equal_nan=True)
    assert np.isnan(got[1:, -1]).all()
