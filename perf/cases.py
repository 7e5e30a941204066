"""Performance cases of the collision-detection path, through its public entry points.

Each case is one call (or one step) that a program makes:

* ``query``   one primitive query through the single-call entry points;
* ``rows``    a batch of swept primitive rows resident in device memory;
* ``host``    the same batch in host memory, copied in and out by the call;
* ``mesh``    one step of a mesh: new positions from the host, broad and narrow
              phase, the colliding stencils read back;
* ``narrow``  the narrow phase on given candidate stencils;
* ``self``    the self distance of a mesh at new positions.

The primitive rows are those of ``workloads.primitive_batch`` (starts uniform in
the unit cube, normal motion, a fifth of the rows near-degenerate), made on the
GPU because the largest batches hold 10 million of them.  The meshes come from
``collisiondetection_gb300.workloads``.
"""
import math

import numpy as np
import torch

import collisiondetection_gb300 as ccd
from collisiondetection_gb300 import workloads

KIND = {"vf": ccd.VERTEX_FACE, "ee": ccd.EDGE_EDGE, "ve": ccd.VERTEX_EDGE, "vv": ccd.VERTEX_VERTEX}
POINTS = {"vf": 4, "ee": 4, "ve": 3, "vv": 2}
ETA = 1e-6
MOST_COLLISIONS = 16_384

_context = None


def context():
    """The program's one device context (buffers and stream), kept between calls."""
    global _context
    if _context is None:
        _context = ccd.Context(0)
    return _context


def listed():
    return [
        # One query of a program that tests primitives one at a time: latency only.
        {"name": "query_ee", "what": "query", "kind": "ee"},
        # The contacts of a small scene: a few thousand rows, bound by the slowest root solve.
        {"name": "rows_vf_4096", "what": "rows", "kind": "vf", "n": 4096, "per_row_eta": False},
        # An ordinary batch of odd size with a thickness of its own for each row.
        {"name": "rows_ee_65537", "what": "rows", "kind": "ee", "n": 65537, "per_row_eta": True},
        # The benchmark's two batches: 10 million rows of each kind.
        {"name": "rows_vf_10m", "what": "rows", "kind": "vf", "n": 10_000_000, "per_row_eta": False},
        {"name": "rows_ee_10m", "what": "rows", "kind": "ee", "n": 10_000_000, "per_row_eta": False},
        # Vertex-edge rows, the sub-tests of the narrow-phase chain.
        {"name": "rows_ve_1m", "what": "rows", "kind": "ve", "n": 1_000_003, "per_row_eta": False},
        # A batch whose rows and results live in host memory: copies and kernels.
        {"name": "host_vf_500k", "what": "host", "kind": "vf", "n": 500_000, "per_row_eta": False},
        # Two colliding level-3 icospheres: 2,560 faces, 70,000 candidate stencils.
        {"name": "mesh_two_spheres", "what": "mesh", "scene": "spheres", "size": 3, "step": 0},
        # A 256 x 256 sheet that has come to rest on a level-6 icosphere: 211,970 faces, few contacts.
        {"name": "mesh_cloth_212k", "what": "mesh", "scene": "cloth", "size": 256, "step": 25},
        # Independent meshes of very different sizes in one call.
        {"name": "mesh_uneven_24", "what": "mesh", "scene": "uneven", "size": 24, "step": 0},
        # The narrow phase on candidate stencils that the program holds (two icospheres, 10,240 faces).
        {"name": "narrow_spheres", "what": "narrow", "scene": "spheres", "size": 4, "step": 0},
        # The self distance of a scene, as a step-size control asks for it.
        {"name": "self_two_spheres", "what": "self", "scene": "spheres", "size": 3, "step": 0},
    ]


def draw(rng):
    def size(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi)))) | (rng.random() < 0.7)

    what = rng.choice(["query", "rows", "rows", "rows", "host", "mesh", "mesh", "narrow", "self"])
    if what == "query":
        return {"what": "query", "kind": rng.choice(["vf", "ee", "ve", "vv"]), "variant": rng.randrange(1000)}
    if what == "rows":
        return {"what": "rows", "kind": rng.choice(["vf", "ee", "vf", "ee", "ve", "vv"]), "n": size(200, 8_000_000),
                "per_row_eta": rng.random() < 0.4}
    if what == "host":
        return {"what": "host", "kind": rng.choice(["vf", "ee"]), "n": size(1000, 1_000_000), "per_row_eta": rng.random() < 0.4}
    if what == "narrow":
        return {"what": "narrow", "scene": "spheres", "size": rng.randint(2, 4), "step": rng.randint(1, 99)}
    if what == "self":
        scene = rng.choice(["spheres", "cloth"])
        return {"what": "self", "scene": scene, "size": rng.randint(2, 4) if scene == "spheres" else rng.randint(24, 128),
                "step": rng.randint(10, 30)}
    scene = rng.choice(["spheres", "cloth", "cloth", "uneven"])
    n = {"spheres": rng.randint(2, 4), "cloth": size(16, 256), "uneven": rng.randint(2, 24)}[scene]
    return {"what": "mesh", "scene": scene, "size": n, "step": rng.randint(10, 40)}


# ---------------------------------------------------------------- primitive rows
def _dot(a, b):
    return (a * b).sum(-1, keepdim=True)


def _unit(a):
    return a / a.norm(dim=-1, keepdim=True).clamp_min(1e-300)


def _coplanar(kind, s, e, g):
    """The four points within 1e-9 of one plane at the start and at the end."""
    for p in (s, e):
        if kind == "vf":
            n, origin, moved = _unit(torch.linalg.cross(p[:, 2] - p[:, 1], p[:, 3] - p[:, 1])), p[:, 1].clone(), (0,)
        else:
            origin = p[:, 0].clone()
            n, moved = _unit(torch.linalg.cross(p[:, 1] - origin, 0.5 * (p[:, 2] + p[:, 3]) - origin)), (2, 3)
        side = 2.0 * torch.randint(0, 2, (len(p), 1), generator=g, device=p.device, dtype=p.dtype) - 1.0
        for j in moved:
            p[:, j] += (1e-9 * side - _dot(p[:, j] - origin, n)) * n


def _parallel(kind, s, e, g):
    """A vertex moving within 1e-9 of a face's plane; two edges parallel to 1e-9."""
    noise = lambda a: torch.randn(a.shape, generator=g, device=a.device, dtype=a.dtype)  # noqa: E731
    if kind == "ee":
        for p in (s, e):
            p[:, 3] = p[:, 2] + (p[:, 1] - p[:, 0]) + 1e-9 * noise(p[:, 0])
        return
    move = e[:, 1] - s[:, 1]
    e[:, 2], e[:, 3] = s[:, 2] + move, s[:, 3] + move
    n = _unit(torch.linalg.cross(s[:, 2] - s[:, 1], s[:, 3] - s[:, 1]))
    off = 2e-9 * torch.rand((len(s), 1), generator=g, device=s.device, dtype=s.dtype) - 1e-9
    s[:, 0] += (off - _dot(s[:, 0] - s[:, 1], n)) * n
    w = 0.1 * noise(move)
    e[:, 0] = s[:, 0] + move + w - _dot(w, n) * n + 1e-9 * noise(move)


def _tangent(kind, s, e, g):
    """The first point moved so that the coplanarity cubic has a double root in [0, 1]."""
    t = torch.rand((len(s), 1), generator=g, device=s.device, dtype=s.dtype)
    for _ in range(3):
        v = e - s
        x = s + t[:, :, None] * v
        if kind == "vf":  # (x0 - x1) . ((x2 - x1) x (x3 - x1))
            a, b, da, db = x[:, 2] - x[:, 1], x[:, 3] - x[:, 1], v[:, 2] - v[:, 1], v[:, 3] - v[:, 1]
            r, dr = x[:, 0] - x[:, 1], v[:, 0] - v[:, 1]
        else:  # (x0 - x1) . ((x1 - x3) x (x3 - x2)): the plane through the first edge along the second
            a, b, da, db = x[:, 1] - x[:, 3], x[:, 3] - x[:, 2], v[:, 1] - v[:, 3], v[:, 3] - v[:, 2]
            r, dr = x[:, 0] - x[:, 1], v[:, 0] - v[:, 1]
        c = torch.linalg.cross(a, b)
        dc = torch.linalg.cross(da, b) + torch.linalg.cross(a, db)
        f, fp = _dot(r, c), _dot(dr, c) + _dot(r, dc)
        gf, gp = torch.cat([c, t * c], 1), torch.cat([dc, c + t * dc], 1)
        m00, m01, m11 = _dot(gf, gf), _dot(gf, gp), _dot(gp, gp)
        det = m00 * m11 - m01 * m01
        det = torch.where(det.abs() > 1e-300, det, torch.full_like(det, math.inf))
        l0, l1 = (m01 * fp - m11 * f) / det, (m01 * f - m00 * fp) / det
        d = l0 * gf + l1 * gp
        s[:, 0] += d[:, :3]
        e[:, 0] = s[:, 0] + v[:, 0] + d[:, 3:]


def make_rows(kind, n, seed, device="cuda"):
    """(n, width) rows of the swept primitive `kind`, made from the seed alone."""
    g = torch.Generator(device=device).manual_seed(1_000_003 * seed + KIND[kind])
    k = POINTS[kind]
    opt = {"generator": g, "device": device, "dtype": torch.float64}
    s = torch.rand((n, k, 3), **opt)
    e = s + 0.1 * torch.randn((n, k, 3), **opt)
    near = torch.randperm(n, generator=g, device=device)[: round(0.2 * n)]
    if len(near) and k == 4:
        for build, ids in zip((_coplanar, _parallel, _tangent), torch.tensor_split(near, 3)):
            a, b = s[ids], e[ids]
            if len(ids):
                build(kind, a, b, g)
            s[ids], e[ids] = a, b
    elif len(near) and kind == "ve":  # the vertex within 1e-9 of the edge's line at both ends
        for p in (s, e):
            at = 2.0 * torch.rand((len(near), 1), **opt) - 0.5
            p[near, 0] = p[near, 1] + at * (p[near, 2] - p[near, 1]) + 1e-9 * torch.randn((len(near), 3), **opt)
    elif len(near):  # two vertices that meet to 1e-9
        at = torch.rand((len(near), 1), **opt)
        v = e[near, 0] - s[near, 0]
        s[near, 0] = s[near, 1] + at * (e[near, 1] - s[near, 1]) + 1e-9 * torch.randn((len(near), 3), **opt) - at * v
        e[near, 0] = s[near, 0] + v
    return torch.cat([s.reshape(n, -1), e.reshape(n, -1)], 1).contiguous()


def make_eta(case, seed):
    if not case.get("per_row_eta"):
        return torch.full((1,), ETA, dtype=torch.float64, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(7 + seed)
    return 10.0 ** (-7.0 + 3.0 * torch.rand(case["n"], generator=g, device="cuda", dtype=torch.float64))


def make_query(case, seed):
    """A row whose features meet, so that the whole test runs."""
    rows = make_rows(case["kind"], 512, 31 * seed + case.get("variant", 0), device="cpu").numpy()
    k = POINTS[case["kind"]]
    # Each feature turns and moves through the common centre: they meet unless they are parallel edges.
    row = rows[seed % 512].copy()
    start, end = row.reshape(2, k, 3)
    half = k // 2 if case["kind"] in ("ee", "vv") else 1
    for part in (slice(0, half), slice(half, k)):
        turn = end[part] - start[part]
        end[part] = start[part] - 1.7 * (start[part].mean(0) - start.mean(0)) + (turn - turn.mean(0))
    return row


# ---------------------------------------------------------------- meshes
def scene(case, seed):
    """(faces, qstart, qend, instances) of a mesh case."""
    size, step = case["size"], case["step"]
    if case["scene"] == "spheres":
        q0, q1, f = workloads.two_spheres(1000 * seed + step, level=size)
        return f, q0, q1, None
    if case["scene"] == "cloth":
        level = max(1, min(6, int(round(math.log(max(2 * size * size / 60.0, 4.0)) / math.log(4.0)))))
        q0, q1, f = workloads.sheet_on_sphere(size, level, seed, step)
        return f, q0, q1, None
    f, frames, vo, fo = workloads.uneven_batch(size, lo=200.0, hi=1e5, seed=seed)
    return f, frames[0], frames[1], (vo, fo)


def prepare(case, seed):
    what = case["what"]
    state = {"case": case, "ctx": context()}
    if what == "query":
        state["row"] = make_query(case, seed)
    elif what == "rows":
        n = case["n"]
        state["rows"], state["eta"] = make_rows(case["kind"], n, seed), make_eta(case, seed)
        state["hit"] = torch.zeros(n, dtype=torch.uint8, device="cuda")
        state["t"] = torch.full((n,), math.nan, dtype=torch.float64, device="cuda")
    elif what == "host":
        state["rows"] = make_rows(case["kind"], case["n"], seed).cpu().numpy()
        state["eta"] = make_eta(case, seed).cpu().numpy()
    else:
        f, q0, q1, inst = scene(case, seed)
        state["mesh"] = ccd.Mesh(state["ctx"], f, q0, q1, instances=inst)
        state["q0"], state["q1"] = q0, q1
        if what == "narrow":  # a fixed number of the step's candidates, taken round again where there are fewer
            held = 16 * 4 ** (case["size"] + 2)
            vf, ee = state["mesh"].broadphase(ccd.BROADPHASE_KDOP13, ETA)
            state["vf"], state["ee"] = np.resize(vf, (held, 4)), np.resize(ee, (held, 4))
        elif what == "mesh":  # where the program keeps a step's collisions, -1 past the last one
            state["found"] = [np.full((MOST_COLLISIONS, 4), -1, np.int32), np.full(MOST_COLLISIONS, -1.0),
                              np.full((MOST_COLLISIONS, 4), -1, np.int32), np.full(MOST_COLLISIONS, -1.0)]
    torch.cuda.synchronize()  # the context has a stream of its own
    return state


def run(state):
    case, ctx = state["case"], state["ctx"]
    what = case["what"]
    if what == "query":
        return ctx.single(KIND[case["kind"]], state["row"], ETA)
    if what == "rows":
        rows, eta, hit, t = state["rows"], state["eta"], state["hit"], state["t"]
        ctx.prim_batch_device(KIND[case["kind"]], case["n"], rows.data_ptr(), eta.data_ptr(), eta.numel(),
                              hit.data_ptr(), t.data_ptr())
        return hit, t
    if what == "host":
        return ctx.prim_batch(KIND[case["kind"]], state["rows"], state["eta"])
    mesh = state["mesh"]
    if what == "self":
        return mesh.self_distance(state["q1"])
    if what == "narrow":
        return mesh.narrowphase(state["vf"], ETA, state["ee"], ETA)
    mesh.set_positions(state["q0"], state["q1"])
    for kept, new in zip(state["found"], mesh.detect(ccd.BROADPHASE_KDOP13, ETA, ETA)):
        kept[: len(new)] = new
        kept[len(new):] = -1
    return state["found"]


def work(case):
    """Bytes that the inputs and outputs hold; for primitive rows also the FP64 operations of the tests themselves,
    priced at the mean of the rows that an exact sign test leaves undecided (a tenth of the vertex-face rows and a
    fifth of the edge-edge rows, some 4,000 operations each)."""
    what = case["what"]
    if what in ("query", "rows", "host"):
        n = case.get("n", 1)
        row = 48 * POINTS[case["kind"]] + 9 + (8 if case.get("per_row_eta") else 0)
        share = {"vf": 0.1, "ee": 0.2, "ve": 0.05, "vv": 0.0}[case["kind"]]
        ops = 4000.0 * (1.0 if what == "query" else share)
        return {"bytes": float(n * row), "flops": n * (ops + 300.0)}
    size = case["size"]
    if case["scene"] == "spheres":
        faces = 40 * 4 ** size
    elif case["scene"] == "cloth":
        faces = 3.3 * size * size
    else:
        faces = 15_000.0 * size
    # Faces, and start and end positions of half as many vertices, read once.
    return {"bytes": faces * (12.0 + 0.5 * 48.0), "flops": faces * 26.0 * 5.0}


# ---------------------------------------------------------------- 64-bit values
def _polymul(a, b):
    out = np.zeros(a.shape[:-1] + (a.shape[-1] + b.shape[-1] - 1,))
    for i in range(a.shape[-1]):
        out[..., i:i + b.shape[-1]] += a[..., i:i + 1] * b
    return out


def _pdot(a, b):
    """Dot product of moving vectors, (n, 3, degree + 1) with ascending powers of time."""
    return _polymul(a, b).sum(1)


def _pcross(a, b):
    c = [_polymul(a[:, (i + 1) % 3], b[:, (i + 2) % 3]) - _polymul(a[:, (i + 2) % 3], b[:, (i + 1) % 3]) for i in range(3)]
    return np.stack(c, 1)


def _at(p, t):
    """Values at times t (n, m) of the polynomials p (n, degree + 1) or (n, k, degree + 1)."""
    p = p.reshape(len(p), -1, p.shape[-1])
    v = np.zeros((len(p), p.shape[1], t.shape[1]))
    for k in range(p.shape[-1] - 1, -1, -1):
        v = v * t[:, None] + p[:, :, k, None]
    return v


def _real_parts(p):
    p = p / np.abs(p).max(1, keepdims=True).clip(1e-300)
    lead = np.where(np.abs(p[:, -1:]) > 1e-13, p[:, -1:], 1e-13)
    comp = np.zeros((len(p), p.shape[1] - 1, p.shape[1] - 1))
    comp[:, np.arange(1, comp.shape[1]), np.arange(comp.shape[1] - 1)] = 1.0
    comp[:, :, -1] = -p[:, :-1] / lead
    return np.linalg.eigvals(comp).real


def _tests(kind, rows):
    """What has to hold while the features touch: sign polynomials (>= 0) and the distance, as moving vectors c and n
    with |c| <= eta |n|."""
    x = rows.reshape(len(rows), 2, -1, 3)
    p = [np.stack([x[:, 0, j], x[:, 1, j] - x[:, 0, j]], -1) for j in range(x.shape[2])]
    if kind == "vf":
        q, sides = p[0], []
        for a, b, c in ((1, 3, 2), (2, 1, 3), (3, 2, 1)):
            u, v = p[b] - p[a], p[c] - p[a]
            # The normal as a point moving on a line, from its start and the velocities' normal, as the test takes it.
            n = np.stack([np.cross(u[..., 0], v[..., 0]), np.cross(u[..., 1], v[..., 1])], -1)
            sides.append(_pdot(q - p[a], _pcross(n, u)))
        n = _pcross(p[2] - p[1], p[3] - p[1])
        return sides, _pdot(q - p[1], n)[:, None], n
    if kind == "ee":
        q0, p0, q1, p1 = p
        e, f = p0 - q0, p1 - q1

        def between(g, h, d):
            return _polymul(_pdot(h, g), _pdot(d, g)) - _polymul(_pdot(g, g), _pdot(d, h))

        n = _pcross(e, f)
        sides = [between(f, e, q0 - q1), between(f, -e, p0 - q1), between(e, f, q1 - q0), between(e, -f, p1 - q0)]
        return sides, _pdot(p0 - p1, n)[:, None], n
    if kind == "ve":
        q, a, b = p
        return [_pdot(b - a, q - a), _pdot(b - a, b - q)], _pcross(b - a, q - a), b - a
    one = np.zeros((len(rows), 1, 1))
    return [], p[0] - p[1], one + 1.0


def _contact_times(kind, rows, eta):
    """First time in [0, 1] at which every test of a row holds; NaN where there is none."""
    sides, c, n = _tests(kind, rows)
    eta = np.broadcast_to(eta, (len(rows),))[:, None]
    gap = _pdot(c, c)
    reach = eta * eta * _pdot(n, n)
    gap[:, : reach.shape[1]] -= reach

    def excess(t):
        v, w = _at(c, t), _at(n, t)
        return np.sqrt((v * v).sum(1)) - eta * np.sqrt((w * w).sum(1))

    times = [np.zeros((len(rows), 1)), _real_parts(gap)]
    # The distance's roots come in close pairs: their polynomial's roots are refined on |c| - eta |n| itself.
    r, h = times[1], 1e-7
    for _ in range(4):
        slope = (excess(r + h) - excess(r - h)) / (2.0 * h)
        step = excess(r) / np.where(slope == 0.0, np.inf, slope)
        r = r - np.clip(step, -0.01, 0.01)
    times += [r] + [_real_parts(s) for s in sides]
    t = np.sort(np.concatenate(times, 1), 1)
    ok = (t >= 0.0) & (t <= 1.0)
    size = np.abs(c).max((1, 2))[:, None]
    ok &= excess(t) <= 1e-13 * size + 1e-9 * eta * np.abs(n).max((1, 2))[:, None]
    for s in sides:
        ok &= _at(s, t)[:, 0] >= -1e-13 * np.abs(s).max(1, keepdims=True)
    if kind == "ee":  # parallel edges are left to the vertex-edge tests
        ok &= np.sqrt((_at(n, t) ** 2).sum(1)) >= 1e-8
    first = np.where(ok.any(1), np.argmax(ok, 1), 0)
    return np.where(ok.any(1), t[np.arange(len(t)), first], np.nan)


def _to_segment(p, a, b):
    """Vector from p to the closest point of segment ab."""
    d = b - a
    u = ((_dot(p - a, d)) / _dot(d, d).clamp_min(1e-300)).clamp(0.0, 1.0)
    return a + u * d - p


def _shortest(vectors):
    """The shortest of several vectors, row by row."""
    v = torch.stack(vectors, -2)
    best = v.norm(dim=-1).argmin(-1)
    return torch.take_along_dim(v, best[..., None, None], -2).squeeze(-2)


def _to_face(p, a, b, c):
    """Vector from p to the closest point of triangle abc."""
    n = torch.linalg.cross(b - a, c - a)
    nn = _dot(n, n)
    h = _dot(a - p, n) / nn * n
    f = p + h
    inside = nn > 0.0
    for u, v in ((a, b), (b, c), (c, a)):
        inside = inside & (_dot(torch.linalg.cross(v - u, f - u), n) >= 0.0)
    edges = _shortest([_to_segment(p, a, b), _to_segment(p, b, c), _to_segment(p, c, a)])
    return torch.where(inside, h, edges)


def _between_edges(a, b, c, d):
    """Vector from the closest point of segment ab to that of segment cd."""
    u, v, w = b - a, d - c, a - c
    uu, uv, vv, uw, vw = _dot(u, u), _dot(u, v), _dot(v, v), _dot(u, w), _dot(v, w)
    det = uu * vv - uv * uv
    safe = torch.where(det > 0.0, det, torch.ones_like(det))
    s, t = (uv * vw - vv * uw) / safe, (uu * vw - uv * uw) / safe
    inside = (det > 1e-14 * uu * vv) & (s >= 0.0) & (s <= 1.0) & (t >= 0.0) & (t <= 1.0)
    ends = _shortest([_to_segment(a, c, d), _to_segment(b, c, d), -_to_segment(c, a, b), -_to_segment(d, a, b)])
    return torch.where(inside, c + t * v - a - s * u, ends)


def _self_distance(q, faces):
    """The least distance between features of faces that share no vertex."""
    x = torch.from_numpy(q).cuda().reshape(-1, 3)
    f = torch.from_numpy(np.asarray(faces, np.int64)).cuda()
    nv, nf = len(x), len(f)
    on = torch.zeros((nf, nv), device="cuda")
    on.scatter_(1, f, 1.0)
    apart = (on @ on.T == 0.0).float()
    edge = torch.unique(torch.cat([f[:, [0, 1]], f[:, [1, 2]], f[:, [2, 0]]]).sort(1).values, dim=0)
    of = ((on[:, edge[:, 0]] * on[:, edge[:, 1]]) > 0.0).float()  # faces by edges
    v, g = torch.nonzero(on.T @ apart > 0.0, as_tuple=True)
    e, h = torch.nonzero(torch.triu(of.T @ apart @ of > 0.0), as_tuple=True)
    best = math.inf
    for at in range(0, len(v), 1 << 21):
        i, j = v[at:at + (1 << 21)], f[g[at:at + (1 << 21)]]
        best = min(best, float(_to_face(x[i], x[j[:, 0]], x[j[:, 1]], x[j[:, 2]]).norm(dim=1).min()))
    for at in range(0, len(e), 1 << 21):
        i, j = edge[e[at:at + (1 << 21)]], edge[h[at:at + (1 << 21)]]
        best = min(best, float(_between_edges(x[i[:, 0]], x[i[:, 1]], x[j[:, 0]], x[j[:, 1]]).norm(dim=1).min()))
    return best


def exact(case, seed):
    """Contact times of single queries and small batches, and the self distance of small scenes.
    Hit flags, stencil lists and counts are whole values."""
    what = case["what"]
    if what == "query":
        return None, float(_contact_times(case["kind"], make_query(case, seed)[None], ETA)[0])
    if what in ("rows", "host") and case["n"] <= 20_000:
        rows = make_rows(case["kind"], case["n"], seed).cpu().numpy()
        return None, _contact_times(case["kind"], rows, make_eta(case, seed).cpu().numpy())
    if what == "self" and case["scene"] == "spheres" and case["size"] <= 3:
        f, _, q1, _ = scene(case, seed)
        return _self_distance(q1, f), None, None
    return None
