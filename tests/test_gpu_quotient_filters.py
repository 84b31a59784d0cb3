"""Quotients that are only taken near a decision (bucket_of, bond_holds):
scenes that sit on the decisions, bit for bit with the oracle, which divides
every time."""
import numpy as np
import pytest

import dem
import dem_scenes
import oracle
from gpu_backend import assert_same_state, copy_scene

pytestmark = pytest.mark.gpu

F = np.float32


# the reciprocal of 2 and of 0.5 is exact, of 2.4 and 1/3 it is not; 96 buckets
# put the particles' edges at quotients whose roundings reach the integers
@pytest.mark.parametrize("cell", [2.0, 0.5, 2.4, 1.0 / 3.0])
def test_edges_on_bucket_borders(cell):
    """Pairs of disks whose box edges fall on bucket borders, or one to three
    roundings beside them, and beyond the bucket grid's own edges."""
    rng = np.random.default_rng(int(cell * 100))
    n, w = 1200, 96
    cell = F(cell)
    # on a grid of 96 buckets centred on 0: a left edge at border k of column or row
    k = rng.integers(-1, w + 1, (n // 2, 2))
    r = F(0.45) * cell
    pos = ((k - w / 2.0) * np.float64(cell)).astype(F) + r
    for _ in range(3):
        up = rng.integers(-1, 2, pos.shape)
        pos = np.where(up > 0, np.nextafter(pos, F(1e9)), np.where(up < 0, np.nextafter(pos, F(-1e9)), pos))
    second = pos + (rng.choice([-1, 1], pos.shape) * F(1.2) * r).astype(F)
    sc = dem_scenes.empty_scene(n, [1, 1, 1, 1.0, 1e3, 5e2])
    sc["pos"] = np.stack([pos, second], 1).astype(F).reshape(-1).copy()
    sc["radii"][:] = r
    p = dem_scenes.reference_defaults(n)
    p.update({"hor_bound": float(w * cell + 8 * r), "vert_bound": float(w * cell + 8 * r), "planet_mode": 0,
              "gravity": 0, "dT": 1e-5, "bonds": 0})
    sc["grid"] = (float(cell), 64, w, w)
    ref = copy_scene(sc)
    with dem.Context(copy_scene(sc), p) as ctx:
        for steps in (1, 12):
            ctx.step(steps)
            oracle.step(ref, p, steps)
        assert_same_state(ctx.download(), ref)
        assert ctx.stats()["device_error"] == 0


@pytest.mark.parametrize("which", ["normal", "shear"])
def test_bonds_at_their_strength(which):
    """Strengths within three roundings of the first step's own stress: some
    bonds tear and some hold, the same ones as in the oracle."""
    sc, p, ext = dem_scenes.c1_chains(chains=40, length=32, seed=4)
    n, nb = 40 * 32, sc["bonds"].size // 3
    rng = np.random.default_rng(11)
    vel = sc["vel"].reshape(-1, 2)
    vel[:] = rng.normal(0.0, 20.0, (n, 2))
    sc["fixity"][:] = 0
    p = dict(p, bonds_tear=0)
    first = copy_scene(sc)
    kw = {"bond_lambda": ext["bond_lambda"]}
    oracle.step(first, p, 1, **kw)
    # the stresses of the step in its own arithmetic (bonds k: i, i + 1)
    con = sc["contacts"].reshape(-1, 14, 6)
    own = con[(con[..., 5] >= 0) & (con[..., 1] > con[..., 0])]
    own = own[np.argsort(own[:, 5])]
    i, j = own[:, 0], own[:, 1]
    x = first["pos"].reshape(-1, 2)
    d = x[i] - x[j]
    L = np.sqrt((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]).astype(F)).astype(F)
    blen = sc["bonds"].reshape(-1, 3)[:, 2].copy().view(F)
    A = F(2.0) * (F(ext["bond_lambda"]) * F(1.0))
    stress = np.abs(((-F(1e5) * (L - blen)).astype(F) * A).astype(F) / A).astype(F)
    tan = first["contacts"].reshape(-1, 14, 6)
    shear = np.abs(tan[i][tan[i][..., 1] == j[:, None]][:, 3].copy().view(F) / A).astype(F)
    s = stress if which == "normal" else shear
    k = rng.integers(-3, 4, nb)
    near = (s.view(np.int32) + k).view(F)
    strong = np.full(nb, 1e9, F)
    sn, ss = (near, strong) if which == "normal" else (strong, near)
    p = dict(p, bonds_tear=1, moment_contribution_factor=0.0)
    ref = copy_scene(sc)
    ev, _ = oracle.step(ref, p, 1, bond_sn=sn, bond_ss=ss, **kw)
    with dem.Context(copy_scene(sc), p, bond_sn=sn, bond_ss=ss, **kw) as ctx:
        ctx.step(1)
        assert_same_state(ctx.download(), ref)
        got = ctx.break_events()
    assert np.array_equal(np.sort(got["bond"]), np.sort(ev["bond"]))
    assert 0.05 * nb < np.unique(ev["bond"]).size < 0.95 * nb
