"""The exponential and the reciprocal square root of the Stokes kernels
(csrc/cexp.cuh) argument by argument, against 64-bit-mantissa host values.

Bounds, in u = 2^-53 of the modulus scale exp(re).  Each component of the table
form: the reduced phase is off by two roundings below 2^-5 (u/16 together),
the cosine's series ends before r^8/40320 (u/34), the table's value, the inner
and the outer sum round by u/2 each, the product with the factor by u: 2.7 u.
A real part adds the table of 2^(j/64), its product and the scale's (u each)
and the series' end before x^6/720 (0.31 u): 6.1 u.  Beyond the tables CUDA's
functions: 2 u for exp, 2 u for sine or cosine, two products: 6.1 u as well.
Reciprocal root: the residual's rounding enters by half, the sum rounds once,
the series' end is below 2^-58 for a start within 2^-20: 1.6 u."""
import numpy as np
import pytest

from bem_mececcs_b200 import capi

pytestmark = pytest.mark.gpu
U = 2.0 ** -53
LD = np.longdouble


@pytest.fixture(scope="module")
def ctx():
    c = capi.Context(0)
    yield c
    c.close()


def _around(x):
    """Values, and their neighbours on both sides at several distances."""
    x = np.asarray(x, dtype=float)
    return np.concatenate([x, np.nextafter(x, np.inf), np.nextafter(x, -np.inf), x * (1 + 1e-12), x * (1 - 1e-12)])


def _phases(rng):
    step = np.pi / 64
    k = np.concatenate([np.arange(0, 300), rng.integers(300, 200_000_000, 2000)])
    return np.concatenate([
        _around((k + 0.5) * step),              # both sides of every reduction boundary
        _around(k * step),                      # every table entry
        np.exp(rng.uniform(np.log(1e-12), np.log(9.9e6), 40000)),
        rng.uniform(0.0, 20.0, 40000),
        _around([1e7, 9999999.0, 0.0, np.pi / 2, np.pi, 2 * np.pi]),
        np.exp(rng.uniform(np.log(1.01e7), np.log(1e9), 2000))])  # beyond the tables


def _check(ctx, re, im, scale, bound):
    args = np.stack([re, im, scale], 1)
    out = ctx.math_selftest(0, args)
    mod = np.abs(scale).astype(LD) * np.exp(re.astype(LD))
    worst = []
    for col, f in ((0, np.cos), (1, np.sin)):
        want = scale.astype(LD) * np.exp(re.astype(LD)) * f(im.astype(LD))
        worst.append([float(np.max(np.abs(out[:, c] - want) / mod)) / U for c in (col, col + 2)])
    print("error in u of the modulus (cos, sin): tables", worst[0][0], worst[1][0],
          "CUDA", worst[0][1], worst[1][1])
    assert max(worst[0][0], worst[1][0]) <= bound
    return out


def test_undamped_phase(ctx):
    rng = np.random.default_rng(1)
    im = _phases(rng)
    im = np.concatenate([im, -im])
    scale = np.exp(rng.uniform(np.log(1e-3), np.log(1e3), im.size))
    inside = np.abs(im) < 9.9e6
    _check(ctx, np.zeros(inside.sum()), im[inside], scale[inside], 2.7)
    _check(ctx, np.zeros(im.size), im, scale, 6.1)


def test_small_phases_keep_the_sine_relative(ctx):
    """Below pi/128 the sine is its own series: two roundings and the product's."""
    rng = np.random.default_rng(2)
    im = np.exp(rng.uniform(np.log(1e-30), np.log(np.pi / 128.01), 20000)) * rng.choice([-1.0, 1.0], 20000)
    out = ctx.math_selftest(0, np.stack([0 * im, im, 1 + 0 * im], 1))
    want = np.sin(im.astype(LD))
    assert float(np.max(np.abs((out[:, 1] - want) / want))) <= 2.1 * U


def test_damped(ctx):
    rng = np.random.default_rng(3)
    step = np.log(2.0) / 64
    m = np.arange(-400, 400)
    re = np.concatenate([_around((m + 0.5) * step), _around(m[m != 0] * step), rng.uniform(-699.0, 699.0, 40000),
                         -np.exp(rng.uniform(np.log(1e-12), np.log(50.0), 40000)),
                         _around([-700.0, 700.0, -699.9, 699.9]), rng.uniform(-704.0, -700.0, 500),
                         rng.uniform(700.0, 704.0, 500)])
    im = rng.choice(_phases(rng), re.size) * rng.choice([-1.0, 1.0], re.size)
    _check(ctx, re, im, np.exp(rng.uniform(0.0, np.log(10.0), re.size)), 6.1)


def test_not_finite_and_zero(ctx):
    out = ctx.math_selftest(0, [[0.0, 0.0, 2.0], [0.0, np.nan, 1.0], [np.nan, 1.0, 1.0], [-np.inf, 1.0, 1.0],
                                [-800.0, 1.0, 1.0], [0.0, np.inf, 1.0]])
    assert out[0, 0] == 2.0 and out[0, 1] == 0.0
    assert np.isnan(out[1, :2]).all() and np.isnan(out[2, :2]).all() and np.isnan(out[5, :2]).all()
    assert (out[3, :2] == 0.0).all() and (out[4, :2] == 0.0).all()


def test_reciprocal_root(ctx):
    rng = np.random.default_rng(4)
    x = np.concatenate([np.exp(rng.uniform(np.log(1e-290), np.log(1e290), 100000)),
                        rng.uniform(0.25, 4.0, 200000), _around(2.0 ** np.arange(-900, 900)),
                        np.exp(rng.uniform(np.log(1e-8), np.log(1e8), 100000))])
    out = ctx.math_selftest(1, x)
    want = 1 / np.sqrt(x.astype(LD))
    err = [float(np.max(np.abs(out[:, c] / want - 1))) for c in range(3)]
    print("1/sqrt, error in u:", err[0] / U, "CUDA", err[2] / U, "start 2^", np.log2(err[1]))
    assert err[1] <= 2.0 ** -20
    assert err[0] <= 1.6 * U
