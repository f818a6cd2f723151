"""The continued fraction's kernel (numerator and denominator advanced without a division per step) against the division per
step in extended precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fraction(a, b, c, w, eta, wigner, ctype, ftype):
    a, b, c, w = (x.astype(ftype) for x in (a, b, c, w))
    sgn = ftype(1 if wigner else -1)
    im = ctype(1j) * (2 * w * ftype(eta))
    g = 1 / (a[-1] + sgn * w * w + im)
    for i in range(len(a) - 2, -1, -1):
        g = 1 / (a[i] + sgn * w * w + im - b[i] * c[i] * g)
    return -g.real + 1j * g.imag if wigner else g


# one step, groups and chunks of steps with remainders, blocks of frequencies with remainders; coefficients far from 1 (squared
# frequencies in Ry) and so large or small that a group of steps leaves the range of a double (division per step)
@pytest.mark.parametrize("n_iter,n_w", [(1, 1), (2, 31), (5, 33), (100, 500), (257, 64), (300, 7)])
@pytest.mark.parametrize("scale", [1e-6, 1.0, 1e90, 1e-90])
@pytest.mark.parametrize("wigner", [False, True])
def test_against_extended_precision(cuda, n_iter, n_w, scale, wigner):
    torch = cuda
    from tdscha_b200 import _native
    rng = np.random.default_rng(n_iter)
    a = scale * (1 + 0.2 * rng.standard_normal(n_iter))
    if wigner:
        a = -a
    b, c = (scale * (0.3 + 0.05 * rng.random(max(n_iter - 1, 1))) for _ in range(2))
    w = np.sqrt(scale) * np.linspace(0.0, 2.0, n_w)
    eta = 0.01 * np.sqrt(scale)
    t = lambda x: torch.as_tensor(x, device="cuda")   # noqa: E731
    gf = torch.zeros(n_w, 2, dtype=torch.float64, device="cuda")
    _native.continued_fraction(t(a), t(b), t(c), t(w), gf, False, 1, eta, wigner, False, 0.0, 1.0)
    got = gf.cpu().numpy()
    got = got[:, 0] + 1j * got[:, 1]
    exact = _fraction(a, b, c, w, eta, wigner, np.clongdouble, np.longdouble)
    plain = _fraction(a, b, c, w, eta, wigner, np.complex128, np.float64)
    top = float(np.abs(exact).max())
    err, err_plain = float(np.abs(got - exact).max()) / top, float(np.abs(plain - exact).max()) / top
    # the same recurrence with the same number of roundings on the way: a few times the error of the division form
    assert err <= 8 * err_plain + 1e-14, (err, err_plain)


def test_zero_denominator_and_infinities_are_those_of_the_division_form(cuda):
    torch = cuda
    from tdscha_b200 import _native
    t = lambda x: torch.as_tensor(np.asarray(x, dtype=float), device="cuda")   # noqa: E731
    gf = torch.zeros(2, 2, dtype=torch.float64, device="cuda")
    # d_2 = 0 at w = 0 without smearing: 1 / 0 + ... is not a number there; at w = 1 all denominators are finite
    _native.continued_fraction(t([1.0, 2.0, 0.0]), t([0.5, 0.5]), t([0.5, 0.5]), t([0.0, 1.0]), gf, False, 1, 0.0, False, False,
                               0.0, 1.0)
    g = gf.cpu().numpy()
    assert not np.isfinite(g[0]).all()
    d = 1 / (0.0 - 1 / (1.0 - 0.25 / -1.0) * 0.25)
    assert abs(g[1, 0] - d) < 1e-14 * abs(d) and g[1, 1] == 0.0
