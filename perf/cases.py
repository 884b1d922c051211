"""The work that users of this engine have it do, as measurable cases: each is one pass through the public entry points
(`Engine`, `Server` of the package), on seeded scenes, sensors, direction tables and weights.

What a program does with the engine, and the case that stands for it:

 - annual or daily radiation and sun hours of a scene already resident: sensors and directions up, one visibility trace,
   one sum per quantity (`daylight`): from a single box of 16 faces to a whole city block;
 - the same with glass or porous slots: transmittance bytes instead of bits (`glass`);
 - reflected light: diffuse and specular paths binned by sky patch (`bounce`);
 - the hourly series of every sensor, the chunk's visibility already traced (`series`);
 - views: closest hits over a field of view or all around, shares, reach and isovists (`views`);
 - a scene's first run: the acceleration structure from host arrays, then a small trace (`first_run`);
 - a mesh read from its file image, checked, triangulated and built on the device (`ingest`);
 - a server with resident scenes and a batch of uneven requests (`serving`).
"""
import importlib

import numpy as np

pkg = importlib.import_module("kit-sim_daylight_gb300")
kgb, workloads = pkg.kgb, pkg.workloads

GROUPS = 6   # view classes: sky, ground, obstruction and three target groups


def listed():
    return [
        # an interactive tool's repeated run on a resident scene: one box, the sun hours of one day
        dict(name="box_day", kind="daylight", scene="box", sensors=16, mf=0, suns=15, quantities=1),
        # the smallest annual study: the same box, every sky patch, its ground mirror and every sun-up hour
        dict(name="box_year", kind="daylight", scene="box", sensors=16, mf=1, suns=4456, quantities=4),
        # a building's facades in a block (odd counts of sensors and directions), a season's hours
        dict(name="facade_season", kind="daylight", scene="block", sensors=12345, mf=2, suns=1001, quantities=2),
        # the sun hours of one day for a whole city block (few directions, many sensors)
        dict(name="block_day", kind="daylight", scene="block", sensors=199000, mf=0, suns=14, quantities=1),
        # the headline annual study: a whole block, 577 patches, ground and sun-up hours, four quantities
        dict(name="block_year", kind="daylight", scene="block", sensors=199000, mf=2, suns=4456, quantities=4),
        # a chunk of a study with windows (20 % glass): transmittance bytes at 2305 patches
        dict(name="glass_year", kind="glass", scene="block", sensors=20011, mf=4, suns=4456, quantities=1),
        # reflected light of a chunk: one diffuse bounce of 1024 paths a sensor, with glass facades
        dict(name="bounce", kind="bounce", scene="block", sensors=20011, mf=4, paths=1024, bounces=1),
        # the hourly irradiance of a chunk at 2305 patches, rows returned to the host
        dict(name="series_year", kind="series", scene="block", sensors=8200, mf=4, steps=4456),
        # the views of some facades (fov 120) against a city of half a million triangles
        dict(name="views_fov120", kind="views", tris=500000, sensors=12000, fov=120, cell=2.0, jitter=True, isovist=0, reach=0),
        # all-around views with isovist volume and reach against two million triangles
        dict(name="views_all_around", kind="views", tris=2000000, sensors=25000, fov=360, cell=2.0, jitter=True, isovist=3, reach=3),
        # a new scene's first run: the tree from host arrays, then the sun hours of a day for some facades
        dict(name="first_run_city", kind="first_run", tris=2000000, sensors=5000, suns=14),
        # an evening of uneven requests on two resident scenes
        dict(name="serving_mix", kind="serving", tris=500000, requests=32),
    ]


def _log(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def draw(rng):
    kind = rng.choice(["daylight", "daylight", "daylight", "glass", "bounce", "series", "views", "views", "first_run", "ingest", "serving"])
    if kind == "daylight":
        c = dict(kind=kind, scene="block", sensors=_log(rng, 100, 199000), mf=rng.choice([0, 1, 2, 4]), suns=_log(rng, 1, 4456), quantities=rng.randint(1, 4))
        while c["sensors"] * _dirs(c) > 1.1e9:
            c["sensors"] //= 2
        return c
    if kind == "glass":
        c = dict(kind=kind, scene="block", sensors=_log(rng, 500, 20011), mf=rng.choice([1, 2, 4]), suns=_log(rng, 14, 4456), quantities=rng.randint(1, 2))
        return c
    if kind == "bounce":
        c = dict(kind=kind, scene="block", sensors=_log(rng, 500, 20011), mf=rng.choice([1, 2, 4]), paths=rng.choice([64, 256, 1024]), bounces=rng.randint(1, 3))
        while c["sensors"] * c["paths"] * c["bounces"] > 20011 * 1024:
            c["sensors"] //= 2
        return c
    if kind == "series":
        return dict(kind=kind, scene="block", sensors=_log(rng, 300, 8200), mf=rng.choice([1, 2, 4]), steps=_log(rng, 24, 4456))
    if kind == "views":
        fov = rng.choice([120, 360])
        c = dict(kind=kind, tris=_log(rng, 50000, 2000000), sensors=_log(rng, 500, 25000), fov=fov, cell=rng.choice([2.0, 3.0, 5.0]),
                 jitter=rng.random() < 0.75, isovist=rng.choice([0, 2, 3]) if fov == 360 else 0, reach=rng.choice([0, 3]))
        return c
    if kind == "first_run":
        return dict(kind=kind, tris=_log(rng, 20000, 2000000), sensors=_log(rng, 100, 5000), suns=_log(rng, 1, 100))
    if kind == "ingest":
        return dict(kind=kind, side=_log(rng, 100, 1000), sensors=1000, suns=14)
    return dict(kind="serving", tris=_log(rng, 100000, 500000), requests=rng.randint(4, 32))


# --------------------------------------------------------------------------------------------------- inputs
def _sun(n, seed):
    """n hourly sun directions (unit, float32) of a mid-European year, the year's hours sampled evenly from a seeded
    start, in the order of time."""
    lat = np.radians(52.5)
    day = np.repeat(np.arange(365), 24)
    hour = np.tile(np.arange(24) + 0.5, 365)
    dec = np.radians(23.45) * np.sin(2 * np.pi * (day - 80) / 365)
    ha = np.radians(15 * (hour - 12))
    up = np.sin(lat) * np.sin(dec) + np.cos(lat) * np.cos(dec) * np.cos(ha)
    east = -np.cos(dec) * np.sin(ha)
    north = np.cos(lat) * np.sin(dec) - np.sin(lat) * np.cos(dec) * np.cos(ha)
    v = np.stack([east, north, up], axis=1)[up > 0]
    first = int(np.random.default_rng(seed).integers(0, len(v)))
    v = np.roll(v, -first, axis=0)
    if n <= 20:
        take = np.arange(n)   # consecutive hours
    else:
        take = (np.arange(n) * (len(v) / n)).astype(np.int64) % len(v)
    return v[np.sort(take)].astype(np.float32)


def _patches(mf):
    return 144 * mf * mf + 1 if mf else 0


def _dirs(case):
    return 2 * _patches(case["mf"]) + case["suns"]


def _directions(mf, suns, seed):
    """The direction table [sky | ground = -sky | sun] and the patches' solid angles."""
    sun = _sun(suns, seed)
    if not mf:
        return sun, np.zeros(0, np.float32)
    sky, omega = workloads.patch_dirs(mf)
    return np.concatenate([sky, -sky, sun]).astype(np.float32), omega


def _weights(case, omega, seed):
    """Per quantity a weight per direction (float32) and whether it is weighted by the cosine: radiation, irradiance and
    illuminance sums over the sky, the ground and the sun, then sun hours."""
    rng = np.random.default_rng(seed + 1)
    P, S = len(omega), case["suns"]
    out = []
    for q in range(case["quantities"]):
        w = np.zeros(2 * P + S, np.float32)
        if q == case["quantities"] - 1:   # sun hours
            w[2 * P:] = 1.0
            out.append((w, False))
            continue
        w[:P] = omega * rng.gamma(2.0, 60.0, P)
        w[P:2 * P] = omega * 12.0
        w[2 * P:] = rng.beta(2.0, 1.5, S) * 800.0
        out.append((w, True))
    return out


def _block(sensors, seed, glass=0.0):
    """A seeded 20 x 20 block of extruded boxes with at least `sensors` sensor faces, its first ones taken."""
    s = workloads.urban_block(seed=seed, target_sensors=int(sensors * 1.03) + 300, glass_share=glass, glass_seed=seed + 1)
    while len(s["P"]) < sensors:
        s = workloads.urban_block(seed=seed, target_sensors=int(len(s["P"]) * 1.3) + sensors, glass_share=glass, glass_seed=seed + 1)
    first = (len(s["P"]) - sensors) // 2
    return dict(s, P=s["P"][first:first + sensors], N=s["N"][first:first + sensors])


def _city(tris, sensors, seed):
    s = workloads.views_city(seed=seed, n_buildings=max(400, tris // 100), target_tris=tris, n_sensors=int(sensors * 1.05) + 400)
    return dict(s, P=s["P"][:sensors], N=s["N"][:sensors])


def _grid_image(side, seed):
    """A .dmesh image: a rolling side x side quad terrain with a slot per face."""
    rng = np.random.default_rng(seed)
    a, b = rng.uniform(0.05, 0.3, 2)
    xs, ys = np.meshgrid(np.arange(side + 1, dtype=np.float64), np.arange(side + 1, dtype=np.float64), indexing="ij")
    P = np.stack([xs.ravel(), ys.ravel(), 2.0 * np.sin(a * xs.ravel()) * np.cos(b * ys.ravel())], 1)
    q = np.arange(side * (side + 1)).reshape(side, side + 1)[:, :side].ravel()
    I = np.stack([q, q + side + 1, q + side + 2, q + 1], 1).astype(np.int32).ravel()
    C = np.full(side * side, 4, np.int32)
    S = (np.arange(side * side) % 3).astype(np.uint16)
    head = b"DLM1" + np.array([1], np.uint32).tobytes() + np.array([len(P), len(C), len(I)], np.uint64).tobytes()
    return np.frombuffer(head + P.tobytes() + C.tobytes() + I.tobytes() + S.tobytes(), np.uint8), P


def _glass_slots():
    return [(0.2, 0, 0, 0), (0.0, 0.64, kgb.tn_from_Tn(0.64), kgb.SLOT_GLASS), (0.2, 0, 0, 0)]


def _requests(case, scenes, seed):
    """Uneven requests, as a mixed stream has them: two in three daylight, the others views. Their sizes follow from the
    case alone, which sensors and hours they ask for from the seed."""
    rng, pick = np.random.default_rng(case["requests"]), np.random.default_rng(seed + 3)
    lg = lambda lo, hi: int(np.exp(rng.uniform(np.log(lo), np.log(hi))))
    out = []
    for k in range(case["requests"]):
        sc = int(rng.integers(0, len(scenes)))
        s = scenes[sc]
        if k % 3 < 2:
            n = min(len(s["P"]), lg(100, 20000))
            D, om = _directions(int(rng.choice([1, 2])), max(1, lg(1, 4400) // 2), int(pick.integers(1 << 30)))
            W = np.zeros((2, len(D)), np.float32)
            W[0, :2 * len(om)] = np.concatenate([om, om]) * 0.1
            W[0, 2 * len(om):] = 0.8
            W[1, 2 * len(om):] = 1.0
            first = int(pick.integers(0, len(s["P"]) - n + 1))
            out.append(dict(scene=sc, P=s["P"][first:first + n], N=s["N"][first:first + n], D=D, W=W))
        else:
            n = min(len(s["P"]), lg(500, 8000))
            first = int(pick.integers(0, len(s["P"]) - n + 1))
            out.append(dict(scene=sc, P=s["P"][first:first + n], N=s["N"][first:first + n], fov=int(rng.choice([120, 360]))))
    return out


# --------------------------------------------------------------------------------------------------- prepare, run
def prepare(case, seed):
    kind = case["kind"]
    lib = pkg.load()
    if kind == "serving":
        scenes = [_city(case["tris"] // (1 + k), 20000, seed + k) for k in range(2)]
        srv = kgb.Server(lib, 60e9)
        ids = [srv.add_scene(s["v"], s["tri"]) for s in scenes]
        grids = {fov: workloads.views_grid(float(fov), 2.0) for fov in (120, 360)}
        return dict(case=case, srv=srv, ids=ids, scenes=scenes, requests=_requests(case, scenes, seed), grids=grids)
    e = pkg.engine()
    st = dict(case=case, e=e)
    if kind in ("daylight", "glass"):
        if case["scene"] == "box":
            s = workloads.box_scene()
            # the box at a seeded place of its site: other coordinates, the same study
            move = np.random.default_rng(seed).uniform(-20, 20, 3).astype(np.float32)
            s = dict(s, v=s["v"] + move, P=s["P"] + move)
        else:
            s = _block(case["sensors"], seed, 0.2 if kind == "glass" else 0.0)
        if kind == "glass":
            e.build(s["v"], s["tri"], s["slot"], _glass_slots(), per_slot=True)
            e.set_slots(_glass_slots())
        else:
            e.build(s["v"], s["tri"])
        D, omega = _directions(case["mf"], case["suns"], seed)
        st.update(P=s["P"], N=s["N"], D=D, W=_weights(case, omega, seed), flags=lib.ray_flags(False, kind == "glass"))
    elif kind == "bounce":
        s = _block(case["sensors"], seed, 0.2)
        e.build(s["v"], s["tri"], s["slot"], _glass_slots(), per_slot=True)
        e.set_slots(_glass_slots())
        D, omega = _directions(case["mf"], 1, seed)
        e.set_scene(s["P"], s["N"], D)
        W = np.random.default_rng(seed).gamma(2.0, 60.0, _patches(case["mf"]) + 1).astype(np.float32)
        st.update(W=W, flags=lib.bounce_flags(False))
    elif kind == "series":
        n, T, P = case["sensors"], case["steps"], _patches(case["mf"])
        s = _block(n, seed)
        e.build(s["v"], s["tri"])
        D, omega = _directions(case["mf"], T, seed)
        e.set_scene(s["P"], s["N"], D)
        e.trace(0, n, lib.ray_flags(False, False))
        Wg = np.zeros(len(D), np.float32)
        Wg[P:2 * P] = omega
        G = e.reduce(n, Wg, True).astype(np.float32)
        rng = np.random.default_rng(seed)
        S = (rng.gamma(2.0, 30.0, (P, T))).astype(np.float32)
        st.update(G=G, S=S, g=rng.uniform(5, 40, T).astype(np.float32), omega=omega, row=np.arange(P, dtype=np.int32), sunVec=D[2 * P:],
                  sunW=(rng.beta(2.0, 1.5, T) * 800).astype(np.float32), out=np.zeros((n, T), np.float32))
    elif kind == "views":
        s = _city(case["tris"], case["sensors"], seed)
        e.build(s["v"], s["tri"])
        e.set_labels(s["label"])
        st.update(P=s["P"], N=s["N"], groundZ=s["groundZ"], none=np.zeros((0, 3), np.float32), flags=lib.bounce_flags(False),
                  grid=workloads.views_grid(float(case["fov"]), case["cell"]))
    elif kind == "first_run":
        s = _city(case["tris"], case["sensors"], seed)
        st.update(v=s["v"], tri=s["tri"], P=s["P"], N=s["N"], D=_sun(case["suns"], seed), flags=lib.ray_flags(False, False))
    elif kind == "ingest":
        image, pts = _grid_image(case["side"], seed)
        rng = np.random.default_rng(seed)
        centre = 0.5 * (pts.min(axis=0) + pts.max(axis=0))
        pick = pts[rng.integers(0, len(pts), case["sensors"])] - centre
        st.update(image=image, centre=centre, P=(pick + [0.3, 0.4, 1.0]).astype(np.float32),
                  N=np.tile(np.array([0, 0, 1], np.float32), (case["sensors"], 1)), D=_sun(case["suns"], seed), flags=lib.ray_flags(False, False))
    return st


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "serving":
        srv, tickets = st["srv"], []
        for r in st["requests"]:
            sc = st["scenes"][r["scene"]]
            if "W" in r:
                tickets.append(srv.submit(st["ids"][r["scene"]], r["P"], r["N"], r["D"], r["W"], [True, False]))
            else:
                nAz, nEl, dAz, rowSin, wRow = st["grids"][r["fov"]]
                world = r["fov"] == 360
                tickets.append(srv.submit_views(st["ids"][r["scene"]], r["P"], r["N"], nAz, nEl, 0.0 if world else -60.0, dAz, rowSin, wRow, GROUPS,
                                                1000.0, reach=[6.0, 20.0, 50.0] if world else [], isoDim=3 if world else 0, label=sc["label"],
                                                world=world, cull=world, groundZ=sc["groundZ"]))
        return [srv.wait(t) for t in tickets]
    e, n = st["e"], case.get("sensors", 0)
    if kind in ("daylight", "glass"):
        e.set_scene(st["P"], st["N"], st["D"])
        e.trace(0, n, st["flags"])
        return [e.reduce(n, w, cos) for w, cos in st["W"]]
    if kind == "bounce":
        e.bounce(0, n, st["flags"], N=case["bounces"], M=case["paths"], mf=case["mf"], north=0.0)
        return e.reduce_dc(n, st["W"])
    if kind == "series":
        P, T = _patches(case["mf"]), case["steps"]
        return e.series(n, P, st["row"], st["omega"], st["S"], st["g"], st["G"], 2 * P, np.arange(T, dtype=np.int32), st["sunVec"], st["sunW"],
                        out=st["out"])
    if kind == "views":
        nAz, nEl, dAz, rowSin, wRow = st["grid"]
        world = case["fov"] == 360
        e.set_scene(st["P"], st["N"], st["none"])
        e.view(0, n, st["flags"], nAz, nEl, 0.0 if world else -case["fov"] / 2, dAz, rowSin, world=world, cull=world, jitter=case["jitter"],
               vground=True, groundZ=st["groundZ"])
        return e.reduce_view(n, wRow, GROUPS, 1000.0, reach=[6.0, 20.0, 50.0][:case["reach"]], isoDim=case["isovist"])
    if kind == "ingest":
        info = e.mesh_read(st["image"], "terrain")
        made, skipped = e.build_meshes([info.id], st["centre"])
        e.mesh_free(info.id)
        e.set_scene(st["P"], st["N"], st["D"])
        e.trace(0, n, st["flags"])
        return [e.download_bits(n), made, skipped]
    e.build(st["v"], st["tri"])   # first_run
    e.set_scene(st["P"], st["N"], st["D"])
    e.trace(0, n, st["flags"])
    return e.download_bits(n)


# --------------------------------------------------------------------------------------------------- work
def work(case):
    """What a pass cannot do without: the inputs and the scene read once and the outputs written once; for every ray (or
    path segment) the arithmetic of one box test and one triangle test; the series' contraction and its sun term."""
    kind, n = case["kind"], case.get("sensors", 0)
    ray = 100.0   # operations: a slab test of a box (18), a watertight triangle test (about 80)
    scene = {"box": 20, "block": 2 * n + 3200}.get(case.get("scene"), case.get("tris", 0))
    if kind in ("daylight", "glass"):
        d, q = _dirs(case), case["quantities"]
        return {"bytes": 48.0 * scene + 24.0 * n + 12.0 * d + q * (4.0 * d + 8.0 * n), "flops": 0.5 * n * d * (ray + 7.0 * q)}
    if kind == "bounce":
        bins = _patches(case["mf"]) + 1
        return {"bytes": 48.0 * scene + 24.0 * n + 4.0 * bins + 8.0 * n, "flops": ray * n * case["paths"] * (1 + case["bounces"])}
    if kind == "series":
        P, T = _patches(case["mf"]), case["steps"]
        return {"bytes": n * (2 * P + T) / 8.0 + 4.0 * P * T + 4.0 * n * T + 16.0 * n, "flops": 2.0 * n * T * (P + 1) + 7.0 * n * T}
    if kind == "views":
        nAz, nEl = workloads.views_grid(float(case["fov"]), case["cell"])[:2]
        rays = float(n) * nAz * nEl
        cols = 3 * GROUPS + 1 + case["reach"] + (1 if case["isovist"] else 0)
        return {"bytes": 48.0 * scene + 24.0 * n + 8.0 * n * cols, "flops": rays * (ray + 10.0)}
    if kind == "ingest":
        faces = case["side"] ** 2
        return {"bytes": 46.0 * faces + 2 * 48.0 * faces + 24.0 * n + n * case["suns"] / 8.0, "flops": 0.5 * n * case["suns"] * ray}
    if kind == "first_run":
        return {"bytes": scene * (12.0 + 8.0 + 48.0) + 24.0 * n + n * case["suns"] / 8.0, "flops": 0.5 * n * case["suns"] * ray}
    rays = case["requests"] * (2 / 3 * 3700 * 1000 + 1 / 3 * 2700 * 7000)   # serving: the requests' mean sizes
    return {"bytes": 48.0 * case["tris"] * 1.5 + case["requests"] * 3200 * 40.0, "flops": rays * ray}


# --------------------------------------------------------------------------------------------------- exact
def exact(case, seed):
    """The box studies in 64 bits, every ray against every triangle (plain numpy). None for the others: their rays times
    their triangles (10^11 and more) take minutes."""
    if case["kind"] != "daylight" or case["scene"] != "box":
        return None
    s = workloads.box_scene()
    move = np.random.default_rng(seed).uniform(-20, 20, 3).astype(np.float32)
    v, P, N = (s["v"] + move).astype(np.float64), (s["P"] + move).astype(np.float64), s["N"].astype(np.float64)
    D, omega = _directions(case["mf"], case["suns"], seed)
    W = _weights(case, omega, seed)
    D = D.astype(np.float64)
    a, b, c = (v[s["tri"][:, k]] for k in range(3))
    e1, e2 = b - a, c - a
    out = [np.zeros(len(P)) for _ in W]
    for i in range(len(P)):
        cos = D @ N[i]
        seen = cos > 0
        for k in range(len(a)):   # Moeller and Trumbore
            h = np.cross(D, e2[k])
            det = h @ e1[k]
            ok = np.abs(det) > 1e-12
            inv = np.where(ok, 1.0 / np.where(ok, det, 1.0), 0.0)
            sv = P[i] - a[k]
            u = (h @ sv) * inv
            q = np.cross(sv, e1[k])
            w = (D @ q) * inv
            t = (e2[k] @ q) * inv
            seen &= ~(ok & (u >= 0) & (w >= 0) & (u + w <= 1) & (t > 1e-4))
        for j, (wt, use) in enumerate(W):
            out[j][i] = np.sum(np.where(seen, np.maximum(cos, 0.0) if use else 1.0, 0.0) * wt.astype(np.float64))
    return out
