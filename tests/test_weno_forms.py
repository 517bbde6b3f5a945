"""The WENO5-JS forms of the fp64 and mixed kernels (``weno_side``,
``face_value`` and the bound on the float32 weights), restated in NumPy and
checked against the reference's form (reconstruction/WENO5_JS.py, as the
oracle restates it) on CPU.

Both forms take the four differences of the stencil and the curvature terms
13/3 (d_{i+1/2} - d_{i-1/2})^2 + 16 eps of its three inner cells; the split
fluxes enter doubled (H' = F +- alpha q), so t^2 + D is 16 (eps + IS_k), and
the value is f_j + num / (6 den).

* float64: the weights C_k / e_k^2 scaled by (e_1 e_2 e_3)^2.
* float32: the weights relative to the central stencil's, (e_2 / e_k)^2 with
  the ratio bounded by 6.5e4, so that nothing overflows for |f| < 1e17; both
  sides of a face share one reciprocal.

In real arithmetic both are the reference's weights, the bounded ones but for
less than 1e-8 of a weight: so in float64 they agree with it to round-off and
to 1e-8, and in float32 within float32 round-off of the largest value (the
differences and candidates of a stencil round to a few ulp of it, 1e-6).
"""
import numpy as np
import pytest

from oracle import janc_oracle as jo

CAP = 6.5e4


def _terms(f):
    """t_k, e_k and the differences of a doubled stencil a..e in f's dtype."""
    dt = f.dtype.type
    dmm, dm, dp, dpp = (f[i + 1] - f[i] for i in range(4))

    def curv(x, y):
        s = y - x
        return dt(13 / 3) * s * s + dt(16e-6)
    t = dt(3) * dm - dmm, dm + dp, dt(3) * dp - dpp
    e = [x * x + d for x, d in zip(t, (curv(dmm, dm), curv(dm, dp), curv(dp, dpp)))]
    return t, e, dm, dp


def _side64(f):
    (t1, t2, t3), (e1, e2, e3), dm, dp = _terms(f)
    a1, a2, a3 = (e2 * e3) ** 2, 6 * (e1 * e3) ** 2, 3 * (e1 * e2) ** 2
    return a3 * (t3 + dp) + (a2 * (t2 + dp) + a1 * (2 * t1 - dm)), (a1 + a2) + a3


def _side32(f, cap=CAP):
    dt = f.dtype.type
    (t1, t2, t3), (e1, e2, e3), dm, dp = _terms(f)
    with np.errstate(over="ignore"):  # an infinite ratio is bounded too
        r1, r3 = np.minimum(e2 / e1, dt(cap)), np.minimum(e2 / e3, dt(cap))
    a1, a3 = r1 * r1, dt(3) * (r3 * r3)
    return a3 * (t3 + dp) + (a1 * (dt(2) * t1 - dm) + dt(6) * (t2 + dp)), (a1 + dt(6)) + a3


def _value(side, f):
    num, den = side(f)
    return f[2] + num / (f.dtype.type(6) * den)


def _face32(fp, fm):
    """The mixed kernels' doubled face flux of H'+ cells j-2..j+2 and H'- cells
    j-1..j+3: the right-biased value along the reversed axis, one reciprocal."""
    dt = fp.dtype.type
    nl, dl = _side32(fp)
    nr, dr = _side32(fm[::-1])  # of the mirrored stencil
    return dt(1 / 6) * ((nl * dr + nr * dl) * (dt(1) / (dl * dr))) + (fp[2] + fm[2])


def _stencils(scale, n=20000, seed=0, cells=5):
    rng = np.random.default_rng(seed)
    f = rng.standard_normal((cells, n)) * scale
    smooth = np.linspace(0, 1, cells)[:, None] * rng.standard_normal(n) * scale + scale
    f[:, : n // 4] = smooth[:, : n // 4]  # smooth (linear) stencils
    jump = rng.integers(1, cells, n)
    for i in range(n // 4, n // 2):  # one discontinuity
        f[jump[i]:, i] += 1e3 * scale
    for i in range(n // 2, 5 * n // 8):  # a jump next to constant data
        f[:, i] = scale
        f[jump[i]:, i] += 1e3 * scale
    return f


@pytest.mark.parametrize("scale", [1e-3, 1.0, 1e5, 1e11])
def test_weight_forms_match_the_reference_in_float64(scale):
    f = _stencils(scale)
    ref_L = jo._weno_L(*f)
    ref_R = jo._weno_R(*f)
    top = np.max(np.abs(f), axis=0)
    np.testing.assert_array_less(np.abs(0.5 * _value(_side64, 2 * f) - ref_L), 1e-12 * top + 1e-300)
    # the right-biased value is the left-biased one of the reversed stencil
    np.testing.assert_array_less(np.abs(0.5 * _value(_side64, 2 * f[::-1]) - ref_R), 1e-12 * top + 1e-300)
    np.testing.assert_array_less(np.abs(0.5 * _value(_side32, 2 * f) - ref_L), 1e-8 * top + 1e-300)


@pytest.mark.parametrize("scale", [1e-3, 1.0, 1e5, 1e11])
def test_float32_form_and_face(scale):
    f = _stencils(scale, seed=1, cells=6)
    h = (2 * f).astype(np.float32)
    g = (2 * _stencils(scale, seed=2, cells=6)).astype(np.float32)
    top = np.maximum(np.max(np.abs(f), axis=0), np.max(np.abs(g), axis=0))
    with np.errstate(over="raise", invalid="raise"):
        got = 0.5 * _value(_side32, h[:5]).astype(np.float64)
        face = 0.5 * _face32(h[:5], g[1:]).astype(np.float64)
    assert np.all(np.abs(got - jo._weno_L(*f[:5])) <= 1e-5 * top)
    ref = jo._weno_L(*0.5 * h[:5].astype(np.float64)) + jo._weno_R(*0.5 * g[1:].astype(np.float64))
    assert np.all(np.abs(face - ref) <= 1e-5 * top)


@pytest.mark.parametrize("scale", [1e-4, 1.0, 1e4, 1e9])
def test_the_bound_on_the_ratios(scale):
    """e_2 <= 8/3 (e_1 + e_3) for any data; the bound is reached on either
    side, never on both; and where it is, it moves the value by less than 1e-8
    of the largest entry."""
    f = 2 * _stencils(scale, seed=3)
    (_, _, _), (e1, e2, e3), _, _ = _terms(f)
    assert np.all(e2 <= 8 / 3 * (e1 + e3) * (1 + 1e-12))
    left, right = e2 / e1 >= CAP, e2 / e3 >= CAP
    assert not np.any(left & right)
    if scale >= 1.0:
        assert left.any() and right.any()
    top = np.max(np.abs(f), axis=0)
    moved = np.abs(_value(_side32, f) - _value(lambda x: _side32(x, np.inf), f))
    assert np.all(moved <= 1e-8 * top)


def test_float32_form_stays_finite_to_its_range():
    rng = np.random.default_rng(4)
    f = rng.uniform(-1e17, 1e17, (6, 20000))
    f[:3, ::4] = 1e17
    f[2:, 1::4] = -1e17
    h = f.astype(np.float32)
    with np.errstate(over="raise", invalid="raise"):
        v, face = _value(_side32, h[:5]), _face32(h[:5], h[1:])
    assert np.all(np.isfinite(v)) and np.all(np.isfinite(face))
    assert np.all(np.abs(v - jo._weno_L(*f[:5])) <= 1e-5 * 1e17)
