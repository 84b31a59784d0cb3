"""The calls of this library whose speed is measured, over the sizes it is used at.

A case is a dict of plain values; `kind` says which public entry point it goes through:

  frame   Context.step(steps) and the readback into the caller's arrays: one displayed frame of
          the reference's loop (State::update_state after gen_per_frame steps)
  mix     Batch.step(steps) and Batch.download_many of every scene: one frame of a parameter sweep
  cycle   Batch.upload_many, step, download_many: every scene restored from host arrays, advanced
          and read back, as a host that owns the states does
  record  Context.record(steps, selections) and the readback: Advance with Record on
  serve   a served stream: requests submitted, advanced until done, fetched
  bonds   dem_generate_bonds of a packed bed (the caller's host arrays in and out)
  bin     dem_broad_phase_noalloc on the caller's device buffers

Scenes come from the builders of dem_scenes.py (the workloads of the tests and of bench.py), seeded.
`exact` restates the step in numpy, in 64 bits, for the scenes of up to some ten thousand particles.
"""
import ctypes as C
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "physics-sim_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import dem  # noqa: E402
import dem_scenes  # noqa: E402

FP, IP = C.POINTER(C.c_float), C.POINTER(C.c_int32)
FIELDS = ("pos", "radii", "vel", "acc", "rot", "rot_vel", "rot_acc", "forces", "fixity", "del_pos", "del_rot",
          "bonds", "contacts", "material_pointers", "data")
MOST_CELLS = 262144  # DEM_NOALLOC_MAX_CELLS
FRAME = 105  # the reference's default gen_per_frame (settings.rs:322)


def listed():
    return [
        # the smallest worlds: a handful of bonded chains under tension, the size of the reference's own experiments
        {"name": "experiment_128", "kind": "frame", "scene": "chains", "chains": 4, "length": 32, "steps": FRAME},
        # the same kind of run recorded step by step (the reference's exported traces)
        {"name": "record_512", "kind": "record", "scene": "chains", "chains": 8, "length": 64, "steps": FRAME},
        # the granular settle at its configured 4,096 disks: an interactive scene
        {"name": "settle_4096", "kind": "frame", "scene": "settle", "n": 4096, "steps": FRAME},
        # the bonded tensile test at its configured 64 chains of 256
        {"name": "chains_16384", "kind": "frame", "scene": "chains", "chains": 64, "length": 256, "steps": FRAME},
        # a packed bed with the F64 distance branch, an odd particle count
        {"name": "bed_f64_30011", "kind": "frame", "scene": "bed", "n": 30011, "f64": True, "steps": FRAME},
        # a packed bed beyond what ends its steps inside the Simulation kernel
        {"name": "bed_262144", "kind": "frame", "scene": "bed", "n": 262144, "f64": False, "steps": FRAME},
        # the 4 M-particle impact scene: breakage, a projectile of 40 radii, a multi-GB state
        {"name": "impact_4m", "kind": "frame", "scene": "impact", "cols": 1024, "rows": 4096, "steps": FRAME},
        # half of the batched mix of uneven scenes (3.9 M particles), a frame of the batch benchmark
        {"name": "mix_256", "kind": "mix", "scenes": 256, "n_min": 1000, "n_max": 64000, "steps": 280},
        # a small batch restored from the host, stepped and read back
        {"name": "cycle_24", "kind": "cycle", "scenes": 24, "n_min": 1000, "n_max": 16000, "steps": FRAME},
        # requests of uneven sizes and horizons, one of them waiting for admission
        {"name": "serve_4", "kind": "serve", "n_min": 2000, "n_max": 32000, "horizon": 210},
        # bonds of a packed bed, as a scene is set up
        {"name": "bonds_200003", "kind": "bonds", "n": 200003, "max_bonds": 6},
        # cell order and cell table of a million particles, close to the entry's largest grid
        {"name": "bin_1000003", "kind": "bin", "n": 1000003, "gw": 509, "gh": 509},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "mix", "cycle", "record", "serve", "bonds", "bin"])
    if kind in ("frame", "record"):
        small = kind == "record"
        scene = "chains" if small else rng.choice(["settle", "chains", "bed", "impact"])
        c = {"kind": kind, "scene": scene, "steps": rng.choice([35, 70, FRAME, 101]) if not small else rng.randint(20, 140)}
        if scene == "settle":
            c["n"] = _log(rng, 64, 40000)
        elif scene == "chains":
            c.update(chains=_log(rng, 1, 16 if small else 96), length=_log(rng, 8, 64 if small else 300))
        elif scene == "bed":
            c.update(n=_log(rng, 64, 1000000), f64=rng.random() < 0.25)
        else:
            c.update(cols=_log(rng, 96, 1000), rows=_log(rng, 64, 2000))
        return c
    if kind == "mix":
        return {"kind": kind, "scenes": _log(rng, 2, 200), "n_min": _log(rng, 200, 2000), "n_max": _log(rng, 4000, 48000),
                "steps": rng.choice([FRAME, 140, 280])}
    if kind == "cycle":
        return {"kind": kind, "scenes": _log(rng, 1, 64), "n_min": _log(rng, 200, 2000), "n_max": _log(rng, 4000, 32000),
                "steps": rng.choice([35, 70, FRAME])}
    if kind == "serve":
        return {"kind": kind, "n_min": _log(rng, 500, 4000), "n_max": _log(rng, 8000, 40000), "horizon": rng.randint(70, 300)}
    if kind == "bonds":
        return {"kind": kind, "n": _log(rng, 100, 400000), "max_bonds": rng.choice([1, 2, 4, 6, 9])}
    gw = _log(rng, 8, 510)
    return {"kind": kind, "n": _log(rng, 1000, 4000000), "gw": gw, "gh": _log(rng, 8, min(4000, (MOST_CELLS - 1) // gw))}


# ---------------------------------------------------------------- scenes

def _one(c, seed):
    """(scene, params, ext) of a frame or record case."""
    kind = c["scene"]
    if kind == "settle":
        # c0_settle's box (8 units^2 a disk) at this particle count
        side = float(np.ceil(np.sqrt(4.0 * c["n"])))
        return dem_scenes.c0_settle(n=c["n"], seed=seed, box=(side, 2.0 * side))
    if kind == "chains":
        sc, p, ext = dem_scenes.c1_chains(chains=c["chains"], length=c["length"], seed=seed)
        # each chain pulled at its own speed: above the configured 0.1, so that the stretch of one frame
        # stands clear of the rounding of the positions, below what breaks bonds within it
        pull = np.random.default_rng(seed + 1).uniform(0.5, 2.0, c["chains"])
        sc["vel"].reshape(-1, 2)[c["length"] - 1::c["length"], 0] = pull
        return sc, p, ext
    if kind == "bed":
        sc, p, ext = dem_scenes.dense_bed(c["n"], seed=seed)
        ext["use_f64"] = bool(c["f64"])
        return sc, p, ext
    # the layout of the bonded clusters is the builder's default, so that every scene of a case has
    # the same number of bonds; the disks' radii and the bonds' strengths change places by the seed
    sc, p, ext = dem_scenes.c2_impact(cols=c["cols"], rows=c["rows"])
    rng = np.random.default_rng(seed)
    sc["radii"][:-1] = rng.permutation(sc["radii"][:-1])
    for k in ("bond_sn", "bond_ss"):
        ext[k] = rng.permutation(ext[k])
    return sc, p, ext


def _sizes(c):
    """(particles, bonded fraction) of each scene of a batch: sizes spread over the logarithm of
    the range, fractions over [0, 0.5], in an order that mixes them."""
    k = c.get("scenes", 4)
    t = (np.arange(k) + 0.5) / k
    ns = (c["n_min"] * (c["n_max"] / c["n_min"]) ** t).astype(int)
    fr = 0.5 * ((np.arange(k) * 0.6180339887) % 1.0)
    order = np.argsort((np.arange(k) * 0.7548776662) % 1.0, kind="stable")
    return [(int(ns[q]), float(fr[q])) for q in order]


def _items(c, seed):
    return [dem_scenes.c3_mix_scene(n, f, seed * 1009 + q) for q, (n, f) in enumerate(_sizes(c))]


def _joined(items):
    """The scenes' arrays end to end, one array a field, and the scenes as views of them."""
    whole = {f: np.concatenate([it[0][f] for it in items]) for f in FIELDS}
    at = {f: 0 for f in FIELDS}
    views = []
    for sc, _, _ in items:
        v = dict(sc)
        for f in FIELDS:
            v[f] = whole[f][at[f]:at[f] + sc[f].size]
            at[f] += sc[f].size
        views.append(v)
    return whole, views


# ---------------------------------------------------------------- the calls

def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "steps": case.get("steps", 0)}
    if kind in ("frame", "record"):
        sc, p, ext = _one(case, seed)
        s["ctx"] = dem.Context(sc, p, **ext)
        s["scene"] = sc  # the caller's state arrays: read back in place
        if kind == "record":
            s["sel"] = _selection(case)
    elif kind in ("mix", "cycle"):
        items = _items(case, seed)
        whole, views = _joined(items)
        s["batch"] = dem.Batch([(v, p, e) for v, (_, p, e) in zip(views, items)])
        s["whole"] = whole
        if kind == "cycle":
            s["inputs"] = dem.SceneTable(enumerate([it[0] for it in items]))
        s["outputs"] = dem.SceneTable(enumerate(views))
    elif kind == "serve":
        s["items"] = _items(case, seed)
        most = max(it[0]["radii"].size for it in s["items"])
        every = sum(it[0]["radii"].size for it in s["items"])
        # admits all but the last arrival at once
        s["server"] = dem.Server(max_active_particles=max(most, every - 1), max_scenes=64)
        s["horizons"] = [case["horizon"] - 23 * q for q in range(len(s["items"]))]
    elif kind == "bonds":
        sc, _, _ = dem_scenes.dense_bed(case["n"], seed=seed)
        n, most = case["n"], case["max_bonds"]
        # the caller's arrays, for as many bonds as there may be
        s.update(pos=sc["pos"], radii=sc["radii"], max_bonds=most, bonds=np.full(3 * n * most, -1, np.int32),
                 contacts=np.zeros(84 * n, np.int32))
    else:
        n, gw, gh = case["n"], case["gw"], case["gh"]
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        pr = torch.rand((n, 4), generator=g, device="cuda")
        pr[:, 0] = (pr[:, 0] - 0.5) * gw * 2.4
        pr[:, 1] = (pr[:, 1] - 0.5) * gh * 2.4
        pr[:, 2] = 0.8 + 0.4 * pr[:, 2]
        pr[:, 2] *= (torch.rand(n, generator=g, device="cuda") > 1e-3)  # a few unused records
        s.update(pr=pr, n=n, gw=gw, gh=gh,
                 keys=torch.zeros(n, dtype=torch.int32, device="cuda"),
                 order=torch.zeros(n, dtype=torch.int32, device="cuda"),
                 start=torch.zeros(gw * gh + 2, dtype=torch.int32, device="cuda"))
    return s


def run(state):
    kind = state["kind"]
    if kind == "frame":
        state["ctx"].step(state["steps"])
        out = state["ctx"].download(state["scene"])
        return {f: out[f] for f in FIELDS}
    if kind == "record":
        rows = state["ctx"].record(state["steps"], state["sel"])
        out = state["ctx"].download(state["scene"])
        return {"rows": rows, **{f: out[f] for f in FIELDS}}
    if kind in ("mix", "cycle"):
        if kind == "cycle":
            state["batch"].upload_many(state["inputs"])
        state["batch"].step(state["steps"])
        state["batch"].download_many(state["outputs"])
        return state["whole"]
    if kind == "serve":
        sv = state["server"]
        ids = [sv.submit(sc, p, h, borrow=True, **ext)
               for (sc, p, ext), h in zip(state["items"], state["horizons"])]
        done = set()
        while len(done) < len(ids):
            sv.advance(70)
            done.update(sv.poll())
        got = [sv.fetch(i)[0] for i in ids]
        return [{f: g[f] for f in FIELDS} for g in got]
    L = dem.lib()
    if kind == "bonds":
        bonds, contacts, n = state["bonds"], state["contacts"], state["radii"].size
        made = C.c_int64(0)
        rc = L.dem_generate_bonds(state["pos"].ctypes.data_as(FP), state["radii"].ctypes.data_as(FP), n,
                                  state["max_bonds"], -1, bonds.ctypes.data_as(IP), bonds.size // 3, C.byref(made),
                                  contacts.ctypes.data_as(IP))
        if rc != 0:
            raise RuntimeError((L.dem_bondgen_last_error() or b"").decode())
        return {"made": made.value, "bonds": bonds, "contacts": contacts}
    gw, gh = state["gw"], state["gh"]
    rc = L.dem_broad_phase_noalloc(state["pr"].data_ptr(), state["n"], -1.2 * gw, -1.2 * gh, 1.0 / 2.4, gw, gh,
                                   state["keys"].data_ptr(), state["order"].data_ptr(), state["start"].data_ptr(),
                                   torch.cuda.current_stream().cuda_stream)
    if rc != 0:
        raise RuntimeError((L.dem_noalloc_last_error() or b"").decode())
    return {"keys": state["keys"], "order": state["order"], "start": state["start"]}


def _selection(c):
    """The pulled end of every chain, as the tensile experiments select it."""
    sel = np.zeros(c["chains"] * c["length"], np.int32)
    sel[c["length"] - 1::c["length"]] = 1
    return sel


# ---------------------------------------------------------------- what a pass cannot do without

def _counts(c):
    """(particles, unbonded and bonded directed slots) of a case's scenes."""
    if c["kind"] in ("mix", "cycle", "serve"):
        sz = _sizes(c)
        n = sum(k for k, _ in sz)
        chained = sum(int(round(k * f)) // 32 * 32 for k, f in sz)
        return n, 0, chained // 32 * 62
    if c["scene"] == "chains":
        n = c["chains"] * c["length"]
        return n, 0, 2 * (n - c["chains"])
    if c["scene"] == "settle":
        return c["n"], 0, 0
    if c["scene"] == "bed":
        return c["n"], 2 * c["n"], 0  # about half of the four lattice neighbours touch
    n = c["cols"] * c["rows"] + 1
    return n, int(1.5 * n), int(0.55 * n)


def work(case):
    kind = case["kind"]
    if kind == "bonds":
        n = case["n"]
        b = min(2 * n, n * case["max_bonds"])
        # positions and radii in; a contact record of 14 x 6 words a particle and a triple a bond out
        return {"bytes": 12 * n + 336 * n + 12 * b, "flops": 9 * 10 * n}
    if kind == "bin":
        # a record in; a key and an order entry out, and the cell table
        return {"bytes": case["n"] * (16 + 8) + 4 * (case["gw"] * case["gh"] + 2), "flops": 4 * case["n"]}
    n, su, sb = _counts(case)
    steps = case["steps"] if kind != "serve" else case["horizon"] - 34
    # a step reads and writes a particle's state (120 bytes), an unbonded slot's partner and
    # history (12) and a bonded one's (36); the caller's arrays hold 468 bytes a particle
    moved = steps * (120 * n + 12 * su + 36 * sb) + 468 * n * (2 if kind in ("cycle", "serve") else 1)
    return {"bytes": moved, "flops": steps * (110 * n + 70 * su + 110 * sb)}


# ---------------------------------------------------------------- the step in 64 bits

EXACT_MOST = 16_000_000  # particle-steps of one restatement


def exact(case, seed):
    kind = case["kind"]
    if kind in ("bonds", "bin"):
        return None  # whole numbers and raw bits
    n, _, _ = _counts(case)
    if kind in ("frame", "record"):
        if n * case["steps"] > EXACT_MOST or case["scene"] == "impact":
            return None
        sc, p, ext = _one(case, seed)
        sel = np.nonzero(_selection(case))[0] if kind == "record" else None
        return _advance(sc, p, ext, case["steps"], sel)
    horizons = [case["horizon"] - 23 * q for q in range(4)] if kind == "serve" else [case["steps"]] * case["scenes"]
    if n * max(horizons) > EXACT_MOST:
        return None
    got = [_advance(sc, p, ext, h) for (sc, p, ext), h in zip(_items(case, seed), horizons)]
    if any(g is None for g in got):
        return None
    if kind == "serve":
        return got
    return {f: None if got[0][f] is None else np.concatenate([g[f] for g in got]) for f in FIELDS}


def _near(pos, rad, reach):
    """Pairs i < j whose centres are within ra + rb + reach, by cells of that width."""
    cell = 2.0 * rad.max() + reach
    k = np.floor((pos - pos.min(0)) / cell).astype(np.int64) + 1
    w = int(k[:, 0].max()) + 2
    key = k[:, 1] * w + k[:, 0]
    order = np.argsort(key, kind="stable")
    ks = key[order]
    out_i, out_j = [], []
    for off in (0, 1, w - 1, w, w + 1):
        lo = np.searchsorted(ks, ks + off, "left")
        hi = np.searchsorted(ks, ks + off, "right")
        if off == 0:
            lo = np.arange(ks.size) + 1  # each pair of a cell once
        cnt = np.maximum(hi - lo, 0)
        i = np.repeat(np.arange(ks.size), cnt)
        j = np.repeat(lo - (np.cumsum(cnt) - cnt), cnt) + np.arange(cnt.sum())
        a, b = order[i], order[j]
        d = pos[a] - pos[b]
        t = rad[a] + rad[b] + reach
        m = (d * d).sum(1) < t * t
        out_i.append(np.minimum(a, b)[m])
        out_j.append(np.maximum(a, b)[m])
    i, j = np.concatenate(out_i), np.concatenate(out_j)
    o = np.argsort(i * np.int64(pos.shape[0]) + j)
    return i[o], j[o]


def _advance(sc, p, ext, steps, sel=None):
    """`steps` steps of one scene in 64 bits: rectangular walls, uniform gravity, linear contacts,
    parallel bonds that hold (None if one would tear)."""
    f = lambda k: float(np.float32(p[k]))  # noqa: E731
    n = sc["radii"].size
    x = sc["pos"].reshape(-1, 2).astype(np.float64)
    v = sc["vel"].reshape(-1, 2).astype(np.float64)
    r = sc["radii"].astype(np.float64)
    a = np.zeros((n, 2))
    rot, w, al = np.zeros(n), np.zeros(n), np.zeros(n)
    fix = sc["fixity"].reshape(-1, 6)
    kick = (fix[:, :3] == 0).astype(np.float64)
    held = fix[:, :2] == 1
    mat = sc["materials"].astype(np.float64)
    mass = mat[3] * np.pi * r * r
    inertia = 0.5 * mass * r * r
    kn, ks, mu, dt = mat[4] / 2.0, mat[5] / 2.0, f("friction_coefficient"), f("dT")
    wall = np.array([f("hor_bound"), f("vert_bound")]) / 2.0
    g = 9.81 * f("gravity_acc") if p["gravity"] == 1 else 0.0

    nb = sc["bonds"].size // 3 if p["bonds"] == 3 else 0
    con = sc["contacts"].reshape(-1, 6)
    own = con[(con[:, 5] >= 0) & (con[:, 1] > con[:, 0])] if nb else con[:0]
    bi, bj, bk = own[:, 0].astype(np.int64), own[:, 1].astype(np.int64), own[:, 5]
    blen = sc["bonds"].reshape(-1, 3)[bk, 2].copy().view(np.float32).astype(np.float64) if nb else np.zeros(0)
    btf, thb, bond_tf = np.zeros(bi.size), np.zeros(bi.size), np.zeros(bi.size)
    if nb:
        Rb = float(np.float32(ext["bond_lambda"])) * np.minimum(r[bi], r[bj])
        A, I2 = 2.0 * Rb, 2.0 / 3.0 * Rb ** 3
        bkn, bks = f("bond_normal_stiffness"), f("bond_shear_stiffness")
        sn = np.asarray(ext["bond_sn"], np.float64)[bk]
        ss = np.asarray(ext["bond_ss"], np.float64)[bk]
        mcf = f("moment_contribution_factor")

    skin = 0.3 * r.max()
    at = None
    live, live_tf = np.zeros(0, np.int64), np.zeros(0)
    rows = []

    def ends(i, j):
        d = x[i] - x[j]
        L = np.sqrt((d * d).sum(1))
        nx, ny = d[:, 0] / L, d[:, 1] / L
        rx, ry = dx[j, 0] - dx[i, 0], dx[j, 1] - dx[i, 1]
        rt = rx * -ny + ry * nx + (dr[j] * r[j] + dr[i] * r[i])
        return L, nx, ny, rt

    def add(i, j, nx, ny, Fn, ft, Mi, Mj, d0, d1):
        for c, val in ((0, nx * Fn - ny * ft), (1, ny * Fn + nx * ft)):
            F[:, c] += np.bincount(i, val, n) - np.bincount(j, val, n)
        M[:] += np.bincount(i, Mi, n) + np.bincount(j, Mj, n)
        for c, (p_, q_) in enumerate(((d0, d0), (d1, d1), (Mi, Mj))):
            D[:, c] += np.bincount(i, p_, n) + np.bincount(j, q_, n)

    for _ in range(steps):
        half = v + kick[:, :2] * a * dt * 0.5
        hw = w + kick[:, 2] * al * dt * 0.5
        mid, mid_w = half.copy(), hw.copy()
        dx, dr = half * dt, hw * dt
        for c in (1, 0):
            q = x[:, c] + dx[:, c]
            lo = (q - r < -wall[c]) & ~held[:, c]
            hi = (q + r > wall[c]) & ~held[:, c] & ~lo
            half[lo | hi, c] *= -0.5
            x[lo, c] += -wall[c] - (q - r)[lo]
            x[hi, c] -= (q + r)[hi] - wall[c]
        x = x + dx
        rot = rot + dr
        if at is None or ((x - at) ** 2).sum(1).max() > (0.45 * skin) ** 2:
            at = x.copy()
            ci, cj = _near(x, r, skin)
            if nb:  # a bonded pair is no loose contact
                ck = ci * np.int64(n) + cj
                keep = ~np.isin(ck, np.minimum(bi, bj) * np.int64(n) + np.maximum(bi, bj))
                ci, cj = ci[keep], cj[keep]
        F, M, D = np.zeros((n, 2)), np.zeros(n), np.zeros((n, 3))
        d = x[ci] - x[cj]
        t = r[ci] + r[cj]
        on = (d * d).sum(1) < t * t
        i, j = ci[on], cj[on]
        key = i * np.int64(n) + j
        tf = np.zeros(key.size)
        if live.size and key.size:
            pos = np.minimum(np.searchsorted(live, key), live.size - 1)
            same = live[pos] == key
            tf[same] = live_tf[pos[same]]
        L, nx, ny, rt = ends(i, j)
        Fn = (r[i] + r[j] - L) * kn
        tf = np.clip(tf + rt * ks, -Fn * mu, Fn * mu)
        live, live_tf = key, tf
        add(i, j, nx, ny, Fn, tf, -r[i] * tf, -r[j] * tf, Fn, tf)
        if nb:
            L, nx, ny, rt = ends(bi, bj)
            Fn = -bkn * (L - blen) * A
            btf = btf + rt * bks * A
            thb = thb + (dr[bi] - dr[bj])  # the other side's is the negative
            bend = bkn * I2 * thb
            if p["bonds_tear"] == 1 and (np.any(Fn / A - mcf * np.abs(bend) * Rb / I2 < -sn) or
                                         np.any(np.abs(btf) / A > ss)):
                return None
            add(bi, bj, nx, ny, Fn, btf, -bend - btf * r[bi], bend - btf * r[bj], -Fn, btf)
            pressed = L < blen
            Fl = np.where(pressed, (blen - L) * kn, 0.0)
            tl = np.clip(bond_tf + rt * ks, -Fl * mu, Fl * mu)
            bond_tf = np.where(pressed, tl, bond_tf)
            tl = np.where(pressed, tl, 0.0)
            add(bi, bj, nx, ny, Fl, tl, -r[bi] * tl, -r[bj] * tl, Fl, tl)
        F[:, 1] -= g * mass
        a = F / mass[:, None]
        al = M / inertia
        v = half + kick[:, :2] * a * dt * 0.5
        w = hw + kick[:, 2] * al * dt * 0.5
        if sel is not None:
            c = [x[:, 0], x[:, 1], mid[:, 0], mid[:, 1], rot, mid_w, D[:, 0], D[:, 1], D[:, 2], np.zeros(n)]
            rows.append([np.abs(q[sel]).sum() if k == 6 else q[sel].mean() for k, q in enumerate(c)])
    data = np.zeros((n, 7))
    data[:, :3], data[:, 4:6], data[:, 6] = D, mid, mid_w
    out = {"pos": x, "radii": r, "vel": v, "acc": a, "rot": rot, "rot_vel": w, "rot_acc": al,
           "forces": sc["forces"].astype(np.float64), "fixity": None, "del_pos": dx, "del_rot": dr, "bonds": None,
           "contacts": None, "material_pointers": None, "data": data}
    out = {k: None if q is None else q.reshape(-1) for k, q in out.items()}
    if sel is not None:
        out = {"rows": np.array(rows), **out}
    return out
