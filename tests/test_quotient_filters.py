"""The arithmetic of the step kernels' two quotient filters (bucket_of and
bond_holds in csrc/dem_kernels.cu), restated in float32: wherever they decide
without dividing, the division decides alike."""
import numpy as np
import pytest

F = np.float32


def _near(x, rng, ulps=4):
    return (x.view(np.int32) + rng.integers(-ulps, ulps + 1, x.shape).astype(np.int32)).view(F)


@pytest.mark.parametrize("seed", range(6))
def test_bucket_of_truncates_like_the_quotient(seed):
    rng = np.random.default_rng(seed)
    n = 1_000_000
    cs = F(2.0) ** rng.uniform(-99, 99, n).astype(F)
    k = np.floor(2.0 ** rng.uniform(0, 25, n)) * rng.choice([-1, 1], n)
    v = _near((k * cs.astype(np.float64)).astype(F), rng)        # quotients beside integers
    half = n // 2
    v[:half] = (rng.normal(0, 300, half) * cs[:half]).astype(F)  # and anywhere
    inv = (F(1.0) / cs).astype(F)
    t = (v * inv).astype(F)
    decided = np.abs(t - np.rint(t)) > (np.abs(t) * F(2.4e-7)).astype(F)
    q = (v / cs).astype(F)
    assert np.array_equal(np.trunc(t[decided]), np.trunc(q[decided]))
    assert 0.4 < decided.mean() < 0.9


@pytest.mark.parametrize("seed", range(6))
def test_bond_holds_only_where_the_tear_test_fails(seed):
    rng = np.random.default_rng(seed)
    n = 1_000_000
    R = (2.0 ** rng.uniform(-12, 12, n)).astype(F)
    A = F(2.0) * R
    I = ((F(2.0) / F(3.0) * R).astype(F) * R).astype(F) * R
    sn, ss = (2.0 ** rng.uniform(-30, 30, (2, n))).astype(F)
    # stresses from far below to just beyond the strengths, by 1 + 2^-24 .. 1 - 1
    s = 1.0 + rng.choice([-1, 1], (2, n)) * 2.0 ** rng.uniform(-25, 0, (2, n))
    X = (rng.random(n) * sn * I).astype(F)
    Fn = ((-sn.astype(np.float64) * s[0] + X.astype(np.float64) / I) * A).astype(F)
    T = np.abs(ss.astype(np.float64) * s[1] * A).astype(F)
    f, x, lim, sh = (Fn * I).astype(F), (X * A).astype(F), ((sn * A).astype(F) * I).astype(F), (ss * A).astype(F)
    room = (F(1e-5) * ((np.abs(f) + np.abs(x)).astype(F) + lim).astype(F)).astype(F)
    holds = (I >= F(1e-12)) & (lim >= F(1e-25)) & (sh >= F(1e-25)) & \
        ((f - x).astype(F) > (room - lim).astype(F)) & (T < (F(0.9999) * sh).astype(F))
    tears = (((Fn / A).astype(F) - (X / I).astype(F)).astype(F) < -sn) | ((T / A).astype(F) > ss)
    assert not np.any(holds & tears)
    assert 0.02 < holds.mean() < 0.9 and tears.mean() > 0.1


def _fma(x, y, z):
    """float32 fused multiply-add: the product is exact in float64, and so is
    the sum here, whose terms cancel (gap_f64 takes residuals of x*y near -z)."""
    return (x.astype(np.float64) * y.astype(np.float64) + z.astype(np.float64)).astype(F)


def _two_sum(x, y):
    s = (x + y).astype(F)
    yy = (s - x).astype(F)
    xx = (s - yy).astype(F)
    return s, ((x - xx).astype(F) + (y - yy).astype(F)).astype(F)


@pytest.mark.parametrize("seed", range(8))
def test_gap_f64_rounds_like_double(seed):
    rng = np.random.default_rng(seed)
    n = 1_000_000
    span = 10.0 ** rng.uniform(-4, 5)
    ax, ay = rng.uniform(-span, span, (2, n)).astype(F)
    ang, d = rng.uniform(0, 2 * np.pi, n), 10.0 ** rng.uniform(-3, 1, n)
    bx, by = (ax + d * np.cos(ang)).astype(F), (ay + d * np.sin(ang)).astype(F)
    dx, dy = ax.astype(np.float64) - bx, ay.astype(np.float64) - by
    L = np.sqrt(dx * dx + dy * dy)
    # lengths from the distance itself, a few roundings off, to twice it
    lh = (L * (1.0 + rng.choice([-1, 1], n) * 2.0 ** rng.uniform(-26, 0, n))).astype(F)
    ll = np.zeros(n, F)
    if seed % 2:  # a sum of two radii in double
        ra = (lh * rng.uniform(0.1, 0.9, n)).astype(F)
        rb = (lh - ra).astype(F)
        lh, ll = _two_sum(ra, rb)
    want = (L - (lh.astype(np.float64) + ll)).astype(F)
    xh, xl = _two_sum(ax, -bx)
    yh, yl = _two_sum(ay, -by)
    px, py = (xh * xh).astype(F), (yh * yh).astype(F)
    ex = (_fma(xh, xh, -px) + (F(2) * (xh * xl).astype(F)).astype(F)).astype(F)
    ey = (_fma(yh, yh, -py) + (F(2) * (yh * yl).astype(F)).astype(F)).astype(F)
    s0, sl = _two_sum(px, py)
    sl = (sl + (ex + ey).astype(F)).astype(F)
    s1 = (s0 + sl).astype(F)
    s2 = (sl - (s1 - s0).astype(F)).astype(F)
    with np.errstate(divide="ignore", invalid="ignore"):
        root = np.sqrt(s1)
        fix = ((_fma(-root, root, s1) + s2).astype(F) * (F(0.5) / root).astype(F)).astype(F)
        g0, gl = _two_sum(root, -lh)
        gl = (gl + (fix - ll).astype(F)).astype(F)
        g, rest = _two_sum(g0, gl)
        err = (root * F(2.4e-13)).astype(F)
        taken = (root > F(1e-9)) & (root < F(1e9)) & ((g + (rest + err).astype(F)).astype(F) == g) & \
            ((g + (rest - err).astype(F)).astype(F) == g)
    assert np.array_equal(g[taken], want[taken])
    assert taken.mean() > 0.5
