"""The room that gap_f64 (csrc/dem_kernels.cu) leaves around its value in pairs
of floats, where the length is far above the distance: two particles that
overlap by nearly all of their radii, a bond compressed to nearly nothing."""
import os
import re

import numpy as np
import pytest

from test_quotient_filters import F, _fma, _two_sum

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _gap(ax, ay, bx, by, lh, ll):
    """gap_f64 restated in float32: its value, whether it is taken, and the
    expression in double rounded once."""
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
        err = (((F(4) * root).astype(F) + np.abs(lh)).astype(F) * F(1.8e-14)).astype(F)
        taken = (root > F(1e-9)) & (root < F(1e9)) & ((g + (rest + err).astype(F)).astype(F) == g) & \
            ((g + (rest - err).astype(F)).astype(F) == g)
    dx, dy = ax.astype(np.float64) - bx, ay.astype(np.float64) - by
    want = (np.sqrt(dx * dx + dy * dy) - (lh.astype(np.float64) + ll)).astype(F)
    return g, taken, want


def _near_ties(n, lo, hi, seed):
    """dx, dy of pairs whose distance less a length of 1 lies beside the middle
    of two floats: dx an odd multiple of 2^-25 between 2^lo and 2^hi, and dy
    so small that the distance is dx + dy^2 / (2 dx)."""
    rng = np.random.default_rng(seed)
    dx = ((np.floor(2.0 ** rng.uniform(24 + lo, 24 + hi, n)) * 2 + 1) * 2.0 ** -25).astype(F)
    dy = np.sqrt(2.0 * dx.astype(np.float64) * 2.0 ** rng.uniform(-56, -43, n)).astype(F)
    return dx, dy


def test_the_source_has_the_room_of_the_restatement():
    src = open(os.path.join(ROOT, "physics-sim_gb300", "csrc", "dem_kernels.cu")).read()
    body = src[src.index("float gap_f64("):]
    assert re.search(r"const float err = \(4\.0f \* root \+ fabsf\(lh\)\) \* 1\.8e-14f;", body[:body.index("\n}\n")])


@pytest.mark.parametrize("lo", range(-16, 1, 2))
def test_near_ties_round_like_double(lo):
    dx, dy = _near_ties(400_000, lo, lo + 2, lo + 50)
    zero = np.zeros_like(dx)
    g, taken, want = _gap(dx, dy, zero, zero, np.ones_like(dx), zero)
    assert np.array_equal(g[taken], want[taken])


@pytest.mark.parametrize("seed", range(8))
def test_long_lengths_round_like_double(seed):
    """Lengths of 2 to 2^16 times the distance, alone and as the sum of two radii."""
    rng = np.random.default_rng(seed)
    n = 1_000_000
    ax, ay = rng.uniform(-1, 1, (2, n)).astype(F)
    ang, d = rng.uniform(0, 2 * np.pi, n), 2.0 ** rng.uniform(-10, 0, n)
    bx, by = (ax + d * np.cos(ang)).astype(F), (ay + d * np.sin(ang)).astype(F)
    lh, ll = (d * 2.0 ** rng.uniform(1, 16, n)).astype(F), np.zeros(n, F)
    if seed % 2:
        ra = (lh * rng.uniform(0.1, 0.9, n)).astype(F)
        lh, ll = _two_sum(ra, (lh - ra).astype(F))
    g, taken, want = _gap(ax, ay, bx, by, lh, ll)
    assert np.array_equal(g[taken], want[taken])
    assert taken.mean() > 0.99
    h = float.fromhex  # one that a room of 2.4e-13 root took wrongly
    one = [np.array([v], F) for v in (h("-0x1.68bd1p-9"), h("0x1.d61094p-7"), h("-0x1.71bbacp-9"),
                                      h("0x1.b8e038p-7"), h("0x1.716844p+0"), 0.0)]
    g, taken, want = _gap(*one)
    assert want[0] == F(h("-0x1.712db6p+0")) and (not taken[0] or g[0] == want[0])


@pytest.mark.gpu
@pytest.mark.parametrize("plain", [0, 1])
def test_deep_overlaps_bit_exact(plain):
    """Pairs of particles that overlap by more than 255/256 of their radii,
    their gaps beside the middle of two floats: the forces are the oracle's."""
    import dem
    import dem_scenes
    import oracle
    from gpu_backend import assert_same_state, copy_scene

    dx, dy = _near_ties(160, -12, -8, 3)
    items = []
    for x, y in zip(dx, dy):
        sc, p, _ = dem_scenes.c0_settle(n=2, seed=1, box=(20.0, 20.0), spacing=3.0)
        sc["pos"][:] = [x, y, 0.0, 0.0]
        sc["radii"][:] = 0.5
        sc["grid"] = dem_scenes.grid_capacity(20.0, 20.0, sc["radii"], 2)
        items.append((sc, dict(p, gravity=0), {"use_f64": True}))
    with dem.Batch([(copy_scene(sc), p, e) for sc, p, e in items], plain_launches=plain) as b:
        b.step(1)
        for k, (sc, p, _) in enumerate(items):
            ref = copy_scene(sc)
            oracle.step(ref, p, 1, use_f64=True)
            assert np.abs(ref["acc"]).max() > 0
            assert_same_state(b.download(k), ref, "pair %d: " % k)
