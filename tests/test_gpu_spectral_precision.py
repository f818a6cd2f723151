"""The imaginary part of the continued fraction (the spectral function) far below the real part: relative to itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fraction(a, b, c, w, eta, wigner):
    a, b, c, w = (x.astype(np.longdouble) for x in (a, b, c, w))
    sgn = np.longdouble(1 if wigner else -1)
    im = np.clongdouble(1j) * (2 * w * np.longdouble(eta))
    g = 1 / (a[-1] + sgn * w * w + im)
    for i in range(len(a) - 2, -1, -1):
        g = 1 / (a[i] + sgn * w * w + im - b[i] * c[i] * g)
    return g


# Below and above the band (a = 1 +- 0.2, b c = 0.1) a step keeps less than a third of the error of the steps before it
# (b c |g|^2), and b c > 0 leaves no cancellation in the imaginary part: a step's roundings (about 8, half an ulp each) add up to
# 1.5 times their number, 6 ulp; 16 ulp allowed.
@pytest.mark.parametrize("n_iter", [2, 9, 100, 300, 1500])
@pytest.mark.parametrize("eta", [1e-2, 1e-4, 1e-9])
@pytest.mark.parametrize("scale", [1e-20, 1e-6, 1.0, 1e26])
@pytest.mark.parametrize("wigner", [False, True])
def test_imaginary_part_outside_the_band(cuda, n_iter, eta, scale, wigner):
    torch = cuda
    from tdscha_b200 import _native
    rng = np.random.default_rng(n_iter)
    a = scale * (1 + 0.2 * (2 * rng.random(n_iter) - 1)) * (-1 if wigner else 1)
    b, c = (scale * (0.3 + 0.02 * rng.random(n_iter - 1)) for _ in range(2))
    w = np.sqrt(scale) * np.concatenate([np.linspace(0.01, 0.15, 21), np.linspace(1.7, 4.0, 43)])
    eta = eta * np.sqrt(scale)
    t = lambda x: torch.as_tensor(x, device="cuda")   # noqa: E731
    gf = torch.zeros(len(w), 2, dtype=torch.float64, device="cuda")
    _native.continued_fraction(t(a), t(b), t(c), t(w), gf, False, 1, eta, wigner, False, 0.0, 1.0)
    exact = _fraction(a, b, c, w, eta, wigner)
    err = np.abs(gf[:, 1].cpu().numpy().astype(np.longdouble) / exact.imag - 1)
    assert float(err.max()) <= 16 * 2.0 ** -53 * 2
