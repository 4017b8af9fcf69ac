"""The calls whose time matters to a user of this framework, over the sizes they are made at.

A simulation spends its time in four places, and a host program may take any
of them by itself: the continuous collision queries that choose a time step,
the discrete narrow phase with its contact filter, the sequential-impulse
solve, and the outer step that drives them all.  Each case is one such call
with the scene resident and the call's own inputs and output buffers on the
host, as a C or C++ program has them at the C ABI (for the allocation-free
narrow phase: on the device); outer steps go through the Python layer.

Scenes are the package's own configurations: unit cubes (1), 64-point hulls
(2), mixed shapes sharing meshes (3) and 1,280-triangle noisy icospheres (5).
Meshes and trees are loaded once per process, as a program loads its assets;
the poses and velocities come from the seed.  Output buffers have a capacity
by the scene's size; what a call does not fill stays zero.
"""
import ctypes
import functools

import numpy as np
import torch

import delta2_gb300 as D

# op: the call.  config, nx, ny, nz: the scene's shapes and grid (one static
# ground or box beside them).  spacing: grid pitch in metres.  steps: outer
# steps of a run.  scenes: independent scenes batched in one context.
LISTED = [
    # a handful of fast cubes: what an interactive scene asks each frame; launches and round trips count
    dict(name="ccd_cubes", op="ccd", config=1, nx=2, ny=2, nz=2, spacing=1.12, speed=3.0),
    # the 1,024-hull benchmark step: every broad-phase pair over one outer step
    dict(name="ccd_hulls", op="ccd", config=2, nx=8, ny=8, nz=16, spacing=1.4, speed=0.5),
    # detailed non-convex bodies packed close: millions of triangle pairs in a call
    dict(name="ccd_spheres", op="ccd", config=5, nx=3, ny=2, nz=3, spacing=1.2, speed=0.5),
    # a real-time loop with a fixed memory budget: caller's device buffers, no allocation in the call
    dict(name="np_fixed_cubes", op="np_fixed", config=1, nx=2, ny=2, nz=2, spacing=1.05, speed=0.0),
    # the discrete narrow phase of a packed pile of hulls
    dict(name="np_hulls", op="np", config=2, nx=8, ny=8, nz=16, spacing=1.23, speed=0.0),
    # ... and of a few detailed bodies, a ragged grid
    dict(name="np_spheres", op="np", config=5, nx=3, ny=1, nz=3, spacing=1.2, speed=0.0),
    # the contact filter on a pile's contacts
    dict(name="filter_hulls", op="filter", config=2, nx=7, ny=5, nz=9, spacing=1.23, speed=0.0),
    # the impulse solve of a few touching cubes
    dict(name="solve_cubes", op="solve", config=1, nx=2, ny=2, nz=2, spacing=1.05, speed=0.5),
    # ... and of a pile that is one contact cluster of a thousand bodies
    dict(name="solve_hulls", op="solve", config=2, nx=8, ny=8, nz=16, spacing=1.23, speed=0.5),
    # a short episode of a small scene, reset and stepped
    dict(name="step_cubes", op="step", config=1, nx=2, ny=2, nz=2, spacing=1.05, speed=0.3, steps=3, scenes=1),
    # an outer step of a packed pile
    dict(name="step_hulls", op="step", config=2, nx=8, ny=8, nz=8, spacing=1.23, speed=0.2, steps=1, scenes=1),
    # many independent mixed scenes in one context, as training or parameter sweeps run them
    dict(name="step_batch", op="step", config=3, nx=6, ny=6, nz=3, spacing=1.4, speed=0.5, steps=2, scenes=8),
]


def listed():
    return [dict(c) for c in LISTED]


def draw(rng):
    def log_int(lo, hi):
        return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))

    op = rng.choice(["ccd", "ccd", "np", "np", "np_fixed", "filter", "solve", "solve", "step", "step"])
    config = 1 if op == "np_fixed" else rng.choice([1, 2, 2, 5] if op in ("ccd", "np") else [1, 2, 2])
    if op == "step" and rng.random() < 0.4:
        config = 3
    lim = {1: (4, 4, 4), 2: (8, 8, 16), 3: (6, 6, 3), 5: (3, 2, 3)}[config]
    if op == "np_fixed" or (op == "step" and config == 1):
        lim = (2, 2, 2)
    if op == "solve" and config == 1:
        lim = (3, 2, 2)
    if op == "np" and config == 5:
        lim = (3, 1, 3)
    if op == "step" and config == 2:
        lim = (8, 8, 8)
    if op == "filter" and config == 2:
        lim = (7, 5, 9)
    case = dict(op=op, config=config, nx=log_int(1, lim[0]), ny=log_int(1, lim[1]), nz=log_int(1, lim[2]),
                spacing=round({1: rng.uniform(1.05, 1.2), 2: rng.uniform(1.23, 1.4), 3: rng.uniform(1.4, 1.5),
                               5: 1.2}[config], 3),
                speed=0.0 if op in ("np", "np_fixed", "filter") else round(rng.uniform(0.2, 0.3 if op == "step" else 0.8), 2))
    if case["nx"] * case["ny"] * case["nz"] == 1:  # two bodies at least beside the ground
        case["nx"] = 2
    if op == "step":
        case["steps"] = rng.randint(1, 3) if config == 1 else 1
        case["scenes"] = rng.randint(2, 8) if config == 3 else 1
    return case


# ---------------------------------------------------------------- scenes ---
@functools.lru_cache(maxsize=64)
def _assets(config, nx, ny, nz, spacing):
    return D.make_scene(config, nx=nx, ny=ny, nz=nz, spacing=spacing, speed_sigma=0.0, seed=1)


def _scene(case, seed):
    """The case's grid of bodies with the seed's orientations and velocities.
    Bodies stay apart whatever the seed: hulls and spheres fit the spacing in
    any orientation, cubes are tilted by less than their gap allows."""
    rng = np.random.default_rng([0xD2, seed])
    s = _assets(case["config"], case["nx"], case["ny"], case["nz"], case["spacing"]).copy()
    moving = np.flatnonzero(s.is_static == 0)
    q = rng.standard_normal((len(moving), 4))
    q /= np.linalg.norm(q, axis=1)[:, None]
    half = s.bounding_radius[moving] / np.sqrt(3.0)
    nodes = np.diff(s.mesh_node_off)[s.mesh[moving]]
    cube = nodes == np.diff(_assets(1, 1, 1, 1, 1.5).mesh_node_off)[-1]
    tilt = 0.45 * np.maximum(case["spacing"] - 2 * half, 0.0) / s.bounding_radius[moving]
    axis = q[:, 1:] / np.linalg.norm(q[:, 1:], axis=1)[:, None]
    small = np.concatenate([np.ones((len(moving), 1)), 0.5 * tilt[:, None] * axis], axis=1)
    small /= np.linalg.norm(small, axis=1)[:, None]
    q = np.where(cube[:, None], small, q)
    if case["config"] == 1 or (case["config"] == 2 and case["op"] != "ccd"):  # a pile on the ground, not in the air
        reach = np.where(cube, half + tilt * s.bounding_radius[moving], s.bounding_radius[moving]).max()
        s.cur[moving, 10] += reach + 0.02 - s.cur[moving, 10].min()
    s.cur[moving, 1:5] = q
    s.cur[moving, 11:14] = case["speed"] * rng.standard_normal((len(moving), 3))
    s.fut[...] = s.cur
    s.last[...] = s.cur
    return s


def _capacity(case):
    """Room for a call's body pairs and contacts, by the scene's size."""
    n = case["nx"] * case["ny"] * case["nz"]
    pairs = 14 * n + 16
    per_body = {"ccd": {1: 4000, 2: 1000, 5: 60000}, "np": {1: 800, 2: 400, 5: 30000},
                "filter": {1: 30, 2: 15}, "solve": {1: 30, 2: 15}, "np_fixed": {1: 800}}[case["op"]][case["config"]]
    return pairs, per_body * n


def _ptr(a, t):
    return a.ctypes.data_as(ctypes.POINTER(t))


I32, I64, F64 = ctypes.c_int32, ctypes.c_int64, ctypes.c_double


def _call(rc):
    if rc != 0:
        raise RuntimeError("d2g status %d: %s" % (rc, D.lib().d2g_last_error().decode()))


def prepare(case, seed):
    op = case["op"]
    if op == "step" and case["scenes"] > 1:
        parts = [_scene({**case, "nx": 1 + (case["nx"] - 1 + k) % case["nx"]}, 1000 * seed + k)
                 for k in range(case["scenes"])]
        s, scene_of = D.concat_scenes(parts)
    else:
        s, scene_of = _scene(case, seed), None
    st = {"op": op, "scene": s, "scene_of": scene_of, "case": dict(case)}
    if op != "step":
        cap_pairs, cap = _capacity(case)
    if op == "np_fixed":
        cap = min(cap, D.NOALLOC_MAX_CONTACTS)
        pairs = D.broad_phase(s)
        dev = {k: torch.from_numpy(np.ascontiguousarray(getattr(s, k))).cuda()
               for k in ("mesh_node_off", "nodes", "ntris", "tris", "eps", "inner_eps", "mesh", "fut", "geo_eps")}
        ds = D.DeviceScene(len(s.mesh_node_off) - 1, len(s.ntris), dev["mesh_node_off"].data_ptr(),
                           dev["nodes"].data_ptr(), dev["ntris"].data_ptr(), dev["tris"].data_ptr(),
                           dev["eps"].data_ptr(), dev["inner_eps"].data_ptr(), s.n_bodies, dev["mesh"].data_ptr(),
                           dev["fut"].data_ptr(), dev["geo_eps"].data_ptr())
        st.update(keep=dev, dscene=ds, pairs=pairs, d_pairs=torch.from_numpy(pairs).cuda(),
                  contacts=torch.zeros((cap, 14), dtype=torch.float64, device="cuda"),
                  offsets=torch.zeros(cap_pairs + 1, dtype=torch.int32, device="cuda"))
        return st
    ctx = D.Context(0)
    st["ctx"] = ctx
    ctx.set_scene(s.copy())
    if scene_of is not None:
        ctx.set_scenes(scene_of)
    if op == "step":
        st["out"] = s.copy()
        return st
    st.update(contacts=np.zeros((cap, 14)), offsets=np.zeros(cap_pairs + 1, np.int32), counters=np.zeros(4, np.int64))
    if op == "ccd":
        # the first outer step's queries: futures projected over last_dt
        s.last_dt = np.minimum(2.0 * s.last_dt, np.float64(np.float32(s.opt_dt)))
        s.fut[:, 8:11] = s.cur[:, 8:11] + s.last_dt[:, None] * s.cur[:, 11:14]
        st["pairs"] = D.broad_phase(s)
        st["max_time"] = np.minimum(s.last_dt[st["pairs"][:, 0]], s.last_dt[st["pairs"][:, 1]])
    elif op == "np":
        st["pairs"] = D.broad_phase(s)
    elif op == "filter":
        st["pairs"] = D.broad_phase(s)
        st["raw"], st["raw_off"], _ = ctx.compare_trees_full(st["pairs"])
    elif op == "solve":
        # every contact cluster of the scene: particles, step, filtered
        # contacts, contacts per body pair, no warm start
        clusters = ctx.separate_clusters(ctx.broad_phase_device(s))
        ctx.set_bodies(s)
        raw, off, _ = ctx.compare_trees_full(np.concatenate([c[1] for c in clusters]).reshape(-1, 2))
        kept, koff = ctx.filter_contacts(raw, off)
        inter = np.cumsum([0] + [len(c[1]) for c in clusters])
        count = np.diff(koff)
        st.update(parts=np.array([g for c in clusters for g in c[0]], np.int32),
                  part_off=np.cumsum([0] + [len(c[0]) for c in clusters]).astype(np.int32),
                  step=np.full(len(clusters), np.float64(np.float32(s.opt_dt))), kept=np.ascontiguousarray(kept),
                  con_off=np.ascontiguousarray(koff[inter], dtype=np.int32),
                  pair_count=np.repeat(count, count).astype(np.int32), warm=np.full(len(kept), np.nan),
                  status=np.zeros(s.n_bodies, np.int32), iterations=np.zeros((s.n_bodies, 2), np.int32),
                  impulses=np.zeros(cap), bodies=np.zeros((cap, 2), np.int32), out=s.copy())
        if len(kept) > cap:
            raise RuntimeError("more contacts than the capacity")
    return st


def run(st):
    op, L = st["op"], D.lib()
    if op == "np_fixed":
        D.compare_trees_full_noalloc(st["dscene"], st["d_pairs"].data_ptr(), len(st["pairs"]),
                                     st["contacts"].data_ptr(), len(st["contacts"]), st["offsets"].data_ptr(),
                                     torch.cuda.current_stream().cuda_stream)
        return {"contacts": st["contacts"], "offsets": st["offsets"]}
    ctx, s = st["ctx"], st["scene"]
    if op == "ccd":
        _call(L.d2g_compare_trees_full_continuous(ctx.h, _ptr(st["pairs"], I32), _ptr(st["max_time"], F64),
                                                  len(st["pairs"]), _ptr(st["contacts"], F64), len(st["contacts"]),
                                                  _ptr(st["offsets"], I32), _ptr(st["counters"], I64)))
        return {"contacts": st["contacts"], "offsets": st["offsets"], "counters": st["counters"]}
    if op == "np":
        _call(L.d2g_compare_trees_full(ctx.h, _ptr(st["pairs"], I32), len(st["pairs"]), _ptr(st["contacts"], F64),
                                       len(st["contacts"]), _ptr(st["offsets"], I32), _ptr(st["counters"], I64)))
        return {"contacts": st["contacts"], "offsets": st["offsets"], "counters": st["counters"]}
    if op == "filter":
        _call(L.d2g_filter_contacts(ctx.h, _ptr(st["raw"], F64), _ptr(st["raw_off"], I32), len(st["raw_off"]) - 1,
                                    F64(0.0), _ptr(st["contacts"], F64), len(st["contacts"]), _ptr(st["offsets"], I32)))
        return {"contacts": st["contacts"], "offsets": st["offsets"]}
    ctx.set_bodies(s)
    if op == "solve":
        rc = L.d2g_solve_clusters(ctx.h, len(st["step"]), _ptr(st["part_off"], I32), _ptr(st["parts"], I32),
                                  _ptr(st["step"], F64), _ptr(st["kept"], F64), _ptr(st["con_off"], I32),
                                  _ptr(st["pair_count"], I32), _ptr(st["warm"], F64), F64(s.gravity_z),
                                  _ptr(st["status"], I32), _ptr(st["iterations"], I32), _ptr(st["impulses"], F64),
                                  _ptr(st["bodies"], I32))
        if rc != 1:  # 1: a cluster was rejected, which is a result
            _call(rc)
        ctx.get_bodies(st["out"])
        return {"status": st["status"], "iterations": st["iterations"], "impulses": st["impulses"],
                "bodies": st["bodies"], "fut": st["out"].fut}
    if st["scene_of"] is not None:
        ctx.set_scenes(st["scene_of"])
    ctx.world_configure(s)
    ctx.world_step(st["case"]["steps"])
    o = ctx.get_bodies(st["out"])
    return {"cur": o.cur, "fut": o.fut, "last": o.last, "last_dt": o.last_dt, "sleep_steps": o.sleep_steps,
            "sleeping": o.sleeping}


# ------------------------------------------------------------------ work ---
def work(case):
    """What a pass cannot do without, by the case's sizes: the trees' node
    buckets of the bodies involved and the states read, the contacts (112
    bytes) or states written; and per contact the 64-bit operations of the
    primitive tests that give it (~600 for a triangle distance's features,
    ~1,500 for a continuous test) or, per sweep of the solve, of its impulse
    update (~120).  Contacts per neighbouring pair are those the
    configurations give (cubes ~40, hulls ~30, noisy spheres ~20,000)."""
    n = case["nx"] * case["ny"] * case["nz"] * case.get("scenes", 1)
    nodes = {1: 5, 2: 36, 3: 40, 5: 713}[case["config"]]
    pairs = max(1.0, 3.0 * n - case["nx"] * case["ny"])
    per_pair = {1: 40, 2: 30, 3: 30, 5: 20000}[case["config"]]
    if case["op"] == "ccd" and case["config"] == 2:
        per_pair = 4
    con = pairs * per_pair
    trees, states = 720.0 * nodes * n, 400.0 * n
    op = case["op"]
    if op == "ccd":
        return {"bytes": trees + states + 112 * con, "flops": 1500 * con}
    if op in ("np", "np_fixed"):
        return {"bytes": trees + states + 112 * con, "flops": 600 * con}
    if op == "filter":
        return {"bytes": 112 * con + 112 * pairs * 6, "flops": 60 * con}
    kept = pairs * 6
    solve = {"bytes": 112 * kept + 2 * states, "flops": 120.0 * kept * 200}
    if op == "solve":
        return solve
    k = case["steps"]
    return {"bytes": k * (trees + 2 * states + 224 * con), "flops": k * (2100 * con + solve["flops"])}


# ----------------------------------------------------------------- exact ---
def _dot(a, b):
    return (a * b).sum(-1)


def _project(T, p):
    """Point p on triangle T's plane, and whether it falls inside (single-precision barycentrics, as specified)."""
    v0, v1 = T[:, 1] - T[:, 0], T[:, 2] - T[:, 0]
    n = np.cross(v0, v1)
    length = np.linalg.norm(n, axis=1)
    n = n / np.where(length > 0, length, 1.0)[:, None]
    on = p - _dot(p - T[:, 0], n)[:, None] * n
    return on, _inside(T, on)


def _inside(T, on):
    v0, v1, v2 = T[:, 1] - T[:, 0], T[:, 2] - T[:, 0], on - T[:, 0]
    d00, d01, d11, d20, d21 = (x.astype(np.float32) for x in (_dot(v0, v0), _dot(v0, v1), _dot(v1, v1), _dot(v2, v0),
                                                              _dot(v2, v1)))
    den = d00 * d11 - d01 * d01
    v = (d11 * d20 - d01 * d21) / den
    w = (d00 * d21 - d01 * d20) / den
    u = ((np.float32(1) - v) - w).astype(np.float64)
    v = v.astype(np.float64)
    return (0 < u) & (u < 1) & (0 < v) & (v < 1) & (u + v < 1)


def _on_segment(A, B, p):
    d = B - A
    t = np.clip(_dot(p - A, d) / _dot(d, d), 0, 1)[:, None]
    return A * (1 - t) + B * t


def _triangle_distance(A, B):
    """Distance and closest points of triangles A, B [n, 3 vertices, 3]."""
    n = len(A)
    P, Q, best = np.zeros((n, 3)), np.zeros((n, 3)), np.full(n, np.inf)

    def take(p, q, d, ok):
        nonlocal best
        ok = ok & (d < best)
        P[ok], Q[ok] = p[ok], q[ok]
        best = np.where(ok, d, best)

    for i in range(3):
        on, inside = _project(A, B[:, i])
        take(on, B[:, i], np.linalg.norm(on - B[:, i], axis=1), inside)
    for i in range(3):
        on, inside = _project(B, A[:, i])
        take(A[:, i], on, np.linalg.norm(on - A[:, i], axis=1), inside)
    for i in range(3):
        SA, SB = A[:, i], A[:, (i + 1) % 3]
        for j in range(3):
            EA, EB = B[:, j], B[:, (j + 1) % 3]
            d = EB - EA
            dd = _dot(d, d)
            a = SA - (_dot(SA - EA, d) / dd)[:, None] * d
            b = SB - (_dot(SB - EA, d) / dd)[:, None] * d
            same = (a == b).all(1)
            t = _dot(EA - a, b - a) / _dot(b - a, b - a)
            t = np.clip(np.where(same, 0.0, t), 0, 1)[:, None]
            q = _on_segment(EA, EB, SA * (1 - t) + SB * t)
            p = _on_segment(SA, SB, q)
            take(p, q, np.linalg.norm(q - p, axis=1), np.ones(n, bool))
    for T, O in ((A, B), (B, A)):
        v0, v1 = T[:, 1] - T[:, 0], T[:, 2] - T[:, 0]
        m = np.cross(v0, v1)
        m = m / np.linalg.norm(m, axis=1)[:, None]
        for j in range(3):
            s, e = O[:, j], O[:, (j + 1) % 3]
            p1, p2 = _dot(T[:, 0] - s, m), _dot(e - s, m)
            ok = np.abs(p2) > np.finfo(np.float64).eps
            t = np.where(ok, p1 / np.where(ok, p2, 1.0), 0.0)
            ok &= (0 < t) & (t < 1)
            ok &= _inside(T, s + (e - s) * t[:, None])
            x = s * (1 - t)[:, None] + e * t[:, None]
            P[ok] = Q[ok] = x[ok]
    return np.linalg.norm(P - Q, axis=1), P, Q


def _narrow_phase(s, pairs):
    """compareTreesFull of every pair: contacts in pair order, breadth-first within a pair."""
    q = s.fut[:, 1:5]
    w, x, y, z = q.T
    R = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                  2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                  2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], 1).reshape(-1, 3, 3)
    pos = s.fut[:, 8:11]
    pid = np.arange(len(pairs))
    na, nb = s.mesh_node_off[s.mesh[pairs[:, 0]]], s.mesh_node_off[s.mesh[pairs[:, 1]]]
    search = (s.geo_eps[pairs[:, 0]] + s.geo_eps[pairs[:, 1]]).astype(np.float32).astype(np.float64)
    tris = s.tris.reshape(-1, 8, 3, 3)
    centre = tris.mean(2)
    radius = np.linalg.norm(tris - centre[:, :, None], axis=3).max(2)
    recs, rec_pair = [], []
    while len(pid):
        a, b = pairs[pid, 0], pairs[pid, 1]
        ca = np.einsum("nij,nkj->nki", R[a], centre[na]) + pos[a][:, None]
        cb = np.einsum("nij,nkj->nki", R[b], centre[nb]) + pos[b][:, None]
        gap = np.linalg.norm(ca[:, :, None] - cb[:, None], axis=3) - radius[na][:, :, None] - radius[nb][:, None]
        thr = (search[pid][:, None, None] + s.eps[na][:, :, None]) + s.eps[nb][:, None]
        k = np.arange(8)
        near = (k[None, :, None] < s.ntris[na][:, None, None]) & (k[None, None] < s.ntris[nb][:, None, None])
        e, ta, tb = np.nonzero(near & (gap < thr + 1e-6))
        hits = np.zeros(len(pid), np.int64)
        leaf = (s.nodes[na, 2] == 0) & (s.nodes[nb, 2] == 0)
        for lo in range(0, len(e), 200000):
            E, i, j = e[lo:lo + 200000], ta[lo:lo + 200000], tb[lo:lo + 200000]
            A = np.einsum("nij,nvj->nvi", R[a[E]], tris[na[E], i]) + pos[a[E]][:, None]
            B = np.einsum("nij,nvj->nvi", R[b[E]], tris[nb[E], j]) + pos[b[E]][:, None]
            d, P, Q = _triangle_distance(A, B)
            hit = d < thr[E, i, j]
            np.add.at(hits, E[hit], 1)
            f = hit & leaf[E]
            E, i, j = E[f], i[f], j[f]
            recs.append(np.column_stack([P[f], Q[f], s.geo_eps[a[E]] + s.eps[na[E], i], s.geo_eps[b[E]] + s.eps[nb[E], j],
                                         s.inner_eps[na[E], i], s.inner_eps[nb[E], j], np.zeros(len(E)), a[E], b[E],
                                         np.zeros(len(E))]))
            rec_pair.append(pid[E])
        nxt = []
        for r in np.flatnonzero((hits > 0) & ~leaf):
            A, B = s.nodes[na[r]], s.nodes[nb[r]]
            down_a = A[2] != 0 and (B[2] == 0 or A[3] < B[3])
            for ch in range((A if down_a else B)[1]):
                nxt.append((pid[r], A[0] + ch, nb[r]) if down_a else (pid[r], na[r], B[0] + ch))
        nxt = np.array(nxt, np.int64).reshape(-1, 3)
        pid, na, nb = nxt[:, 0], nxt[:, 1], nxt[:, 2]
    rec = np.concatenate(recs) if recs else np.zeros((0, 14))
    return rec[np.argsort(np.concatenate(rec_pair), kind="stable")] if recs else rec


def _filter(contacts, offsets):
    out = []
    for g in range(len(offsets) - 1):
        c = contacts[offsets[g]:offsets[g + 1]]
        c = c[np.lexsort((np.linalg.norm(c[:, 0:3] - c[:, 3:6], axis=1), c[:, 6] + c[:, 7]))]
        mid, near, kept = (c[:, 0:3] + c[:, 3:6]) / 2, c[:, 6] + c[:, 7], []
        for i in range(len(c)):
            if not kept or (np.linalg.norm(mid[kept] - mid[i], axis=1) >= near[i]).all():
                kept.append(i)
        out.append(c[kept])
    return np.concatenate(out) if out else np.zeros((0, 14))


def exact(case, seed):
    """The narrow phase and the filter in plain numpy.  A continuous query (ten
    Newton iterations of every edge pair, a traversal that depends on them),
    the solve (up to a thousand ordered sweeps over every contact) and an
    outer step that chains them have no such form: sweep by sweep in Python
    they take minutes."""
    if case["op"] not in ("np", "np_fixed", "filter"):
        return None
    n = case["nx"] * case["ny"] * case["nz"]
    if case["config"] == 5 and n > 4:  # over a million triangle pairs
        return None
    if case["op"] == "filter":
        st = prepare(case, seed)
        contacts = _filter(st["raw"], st["raw_off"])
    else:
        s = _scene(case, seed)
        contacts = _narrow_phase(s, D.broad_phase(s))
    cap = _capacity(case)[1]
    out = np.zeros((min(cap, D.NOALLOC_MAX_CONTACTS) if case["op"] == "np_fixed" else cap, 14))
    out[:len(contacts)] = contacts
    return {"contacts": out, "offsets": None, "counters": None}
