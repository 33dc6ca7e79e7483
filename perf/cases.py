"""The workloads whose speed this repository is judged by, as calls a user's program makes.

Each case is one pass through the public Python binding of the C ABI (kamisimulator_b200.vbd.Solver and
bake_sdf, kamisimulator_b200.autograd): a frame of a device-resident loop, a frame of the plugin's host
loop, several steps of a batch of grooms, a differentiated rollout, or the set-up pass over a body mesh.
Handles run as they are created: no case names a tile shape.

``exact`` restates the step (colour2 and jacobi, wind, substeps, connection springs, SDF pass), its
gradient by autograd and the signed distance of the bake in 64 bits with plain torch.
"""
import math

import numpy as np
import torch

from kamisimulator_b200 import autograd, synth, vbd

GRAVITY = (0.0, 0.0, -9.81)
RADIUS, DENSITY, DAMPING, DECAY = 40e-6, 1300.0, 1e-6, 0.05
WIND_OFF = (0.0, 1.0, 0.7, 0.4, 3.0)
WIND_ON = (40.0, 1.0, 0.7, 0.4, 3.0)  # the reference solver's default wind
K_TIE = 40.0  # stiffness of a connection spring


def _frame(name, strands, vmin, vmax, itr, dt, substeps=1, wind=0, schedule="colour2", sdf=0, scene="groom", seg=2e-3,
           state=0):
    return dict(name=name, kind="frame", strands=strands, vmin=vmin, vmax=vmax, itr=itr, dt=dt, substeps=substeps,
                wind=wind, schedule=schedule, sdf=sdf, scene=scene, seg=seg, state=state)


def listed():
    return [
        # the reference's cantilever harness, one internal step a frame: the smallest call, all latency
        _frame("cantilever_64x32", 64, 32, 32, 10, 1 / 60, scene="rods", seg=5e-3),
        # an ordinary uneven groom: several strands a tile, wind, three substeps, head collision, and a
        # checkpoint of the whole state after each frame
        _frame("groom_2k_uneven_wind", 2000, 8, 64, 20, 1 / 40, substeps=3, wind=1, sdf=96, state=1),
        # the headline groom, device resident: one step and the positions and velocities a frame
        _frame("groom_10k_x64", 10000, 64, 64, 20, 1 / 120, sdf=128),
        # the same groom through the plugin's frame: Hair up, step, Hair down in page-locked host arrays
        dict(name="plugin_frame_10k_x64", kind="hair", strands=10000, vmin=64, vmax=64, row=64, itr=20, dt=1 / 120,
             sdf=128),
        # the reference kernels' own order of updates, on strands of two tile sizes
        _frame("jacobi_3k_x96", 3000, 96, 96, 10, 1 / 240, schedule="jacobi", sdf=96),
        # many uneven grooms in one handle, the head turning: four frames a call
        dict(name="batch_12_grooms", kind="batch", grooms=12, smin=200, smax=3000, vmin=16, vmax=128, itr=20,
             dt=1 / 120, steps=4, sdf=128),
        # the reference solver's default settings: 1 mm segments, 32 iterations, wind, head, 42 substeps of
        # 4e-4 s a 1/60 s frame: the largest
        _frame("default_settings_6k", 6000, 100, 300, 32, 1 / 60, substeps=42, wind=1, sdf=128, seg=1e-3),
        # strands glued to their neighbours: connection springs, on the sweep form
        _frame("tied_rods_4k_x64", 4000, 64, 64, 20, 1 / 120, scene="tied", seg=2e-3),
        # hair-hair collision: five substeps of 4e-4 s with detection in each
        dict(name="hair_hair_2k_x48", kind="hairhair", strands=2000, vmin=48, vmax=48, itr=20, substeps=5),
        # a differentiated rollout: per-strand stiffness scales to positions and back
        dict(name="adjoint_2k_x48", kind="adjoint", strands=2000, vmin=48, vmax=48, itr=10, dt=1 / 120, frames=12,
             every=10, sdf=96),
        # the body's distance grid from a triangle mesh, once a scene
        dict(name="sdf_bake_64", kind="bake", nx=64, ny=64, nz=64, subdivisions=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "hair", "batch", "default", "tied", "hairhair", "adjoint", "bake"])
    if kind == "frame":
        vmax = rng.randint(9, 128)
        vmin = rng.choice([vmax, rng.randint(4, vmax)])
        strands = _log(rng, 48, min(12000, 700000 // vmax))
        jac = rng.random() < 0.2
        sub = 1 if jac else rng.choice([1, 1, 2, 3])
        c = _frame("", strands, vmin, vmax, rng.choice([8, 10, 20, 30]), (1 / 240 if jac else 1 / 120) * sub,
                   substeps=sub, wind=int(rng.random() < 0.4), schedule="jacobi" if jac else "colour2",
                   sdf=rng.choice([0, 96, 128]), state=int(rng.random() < 0.3))
    elif kind == "hair":
        vmax = rng.randint(12, 64)
        c = dict(kind="hair", strands=_log(rng, 200, 10000), vmin=rng.randint(4, vmax), vmax=vmax,
                 row=vmax + rng.randint(0, 8), itr=rng.choice([10, 20]), dt=1 / 120, sdf=rng.choice([0, 96, 128]))
    elif kind == "batch":
        smax = _log(rng, 100, 2500)
        c = dict(kind="batch", grooms=rng.randint(2, 12), smin=max(16, smax // 10), smax=smax, vmin=rng.randint(4, 32),
                 vmax=rng.randint(48, 128), itr=rng.choice([10, 20]), dt=1 / 120, steps=rng.randint(1, 6),
                 sdf=rng.choice([0, 96, 128]))
    elif kind == "default":
        vmin = rng.randint(20, 160)
        c = _frame("", _log(rng, 150, 4000), vmin, vmin + rng.randint(70, 140), 32, 4e-4 * rng.randint(4, 41) * 0.999,
                   wind=1, sdf=128, seg=1e-3)
        c["substeps"] = math.ceil(c["dt"] / 4e-4)
    elif kind == "tied":
        v = rng.randint(10, 160)
        c = _frame("", _log(rng, 32, min(4000, 300000 // v)), v, v, rng.choice([10, 20]), 1 / 120, scene="tied")
    elif kind == "hairhair":
        vmax = rng.randint(16, 48)
        c = dict(kind="hairhair", strands=_log(rng, 150, 2000), vmin=rng.choice([vmax, rng.randint(8, vmax)]),
                 vmax=vmax, itr=rng.choice([10, 20]), substeps=rng.randint(1, 6))
    elif kind == "adjoint":
        vmax = rng.randint(16, 100)
        c = dict(kind="adjoint", strands=_log(rng, 48, 2000), vmin=rng.choice([vmax, rng.randint(8, vmax)]), vmax=vmax,
                 itr=rng.choice([10, 20]), dt=1 / 120, frames=rng.randint(8, 14), every=rng.choice([4, 10]),
                 sdf=rng.choice([0, 96]))
    else:
        c = dict(kind="bake", nx=rng.randint(20, 64), ny=rng.randint(20, 64), nz=rng.randint(20, 64),
                 subdivisions=rng.randint(2, 5))
    c.pop("name", None)
    return c


# ---- inputs -----------------------------------------------------------------------------------------

_grids = {}


def _sphere(n):
    if n == 0:
        return None
    if n not in _grids:  # a head 5 mm under the roots: strands meet it where they fall, not at the first frame
        _grids[n] = synth.sphere_sdf(n, radius=0.085)
    return _grids[n]


def _swing(rng, g):
    """Velocities of strands turning about their roots, up to a few radians a second."""
    sb = np.asarray(g.strand_begin, np.int64)
    of = np.repeat(np.arange(g.num_strands), np.diff(sb))
    w = rng.normal(0.0, 1.5, (g.num_strands, 3))[of]
    return np.cross(w, g.positions.astype(np.float64) - g.positions[sb[:-1]][of]).astype(np.float32)


def _groom(case, rng):
    """(groom, velocities, connection_index) of one groom of a case; its strands' vertex counts are the
    case's own, so that every seed gives outputs of one shape."""
    if case.get("scene", "groom") == "groom":
        lens = np.random.default_rng([case["strands"], case["vmin"], case["vmax"]])
        g = synth.groom_strands(rng, lens.integers(case["vmin"], case["vmax"] + 1, case["strands"]),
                                seg_len=case.get("seg", 2e-3))
        return g, _swing(rng, g), None
    # rods along +x of uneven stiffness
    g = synth.cantilever(case["strands"], case["vmax"], segment=case["seg"], spacing=1e-2 if case["scene"] == "rods" else 2e-3)
    g.strand_young[:] = np.exp(rng.uniform(0.0, math.log(5.0), g.num_strands))
    conn = None
    if case["scene"] == "tied":  # tips of neighbours glued to each other, every fifth rod's middle to the next one's
        conn = np.full(g.num_vertices, -1, np.int32)
        tip, mid = np.asarray(g.strand_begin[1:]) - 1, np.asarray(g.strand_begin[:-1]) + case["vmax"] // 2
        a = np.arange(0, g.num_strands - 1, 2)
        conn[tip[a]], conn[tip[a + 1]] = tip[a + 1], tip[a]
        b = np.arange(0, g.num_strands - 1, 5)
        conn[mid[b]] = mid[b + 1]
    return g, _swing(rng, g) * np.float32(0.3), conn


def _settings(case):
    k = case["kind"]
    st = dict(gravity=GRAVITY, radius=RADIUS, density=DENSITY, damping=DAMPING, velocity_decay=DECAY,
              num_itr=case["itr"], sdf=_sphere(case.get("sdf", 0)))
    if k == "hairhair":
        # the radius and barrier that the solver derives from a 40 um curve radius
        st.update(max_h=4e-4, radius=2e-6, barrier_thickness=7.6e-5, hair_hair=True, sdf=_sphere(96))
    elif k == "frame":
        st.update(max_h=4e-4 if case["seg"] == 1e-3 else case["dt"] / case["substeps"],
                  wind=WIND_ON if case["wind"] else WIND_OFF, schedule=case["schedule"])
    else:
        st.update(max_h=case["dt"])
    return st


def _grooms(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] != "batch":
        return [_groom(case, rng)]
    out, size = [], np.random.default_rng([case["grooms"], case["smin"], case["smax"]])
    for _ in range(case["grooms"]):
        s = int(round(math.exp(size.uniform(math.log(case["smin"]), math.log(case["smax"])))))
        out.append(_groom(dict(case, strands=s), rng))
    return out


def _yaw(frame, dt):
    return synth.head_rotation((frame + 1) * dt) + (0.0, 0.0, 0.0)


def _mesh(case, seed):
    """A closed, bumpy head-sized mesh and the box of its grid."""
    rng = np.random.default_rng(seed)
    v, t = synth.icosphere(case["subdivisions"], 0.09)
    v = v.astype(np.float64)
    u = v / np.linalg.norm(v, axis=1, keepdims=True)
    bump = np.zeros(len(v))
    for _ in range(6):
        k = rng.normal(0.0, 2.5, 3)
        bump += rng.uniform(0.0, 0.03) * np.cos(u @ k + rng.uniform(0.0, 2 * math.pi))
    v = (v * (1.0 + bump)[:, None] * np.array([1.0, 1.1, 1.2])).astype(np.float32)
    lo, hi = synth.mesh_bounds(v)
    return v, t, tuple(a - 0.02 for a in lo), tuple(a + 0.02 for a in hi)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind == "bake":
        v, t, lo, hi = _mesh(case, seed)
        s.update(vertices=v, triangles=t, lo=lo, hi=hi)
        return s
    gs = _grooms(case, seed)
    many = kind == "batch"
    solver = vbd.Solver([g for g, _, _ in gs] if many else gs[0][0], device=0,
                        velocities=[v for _, v, _ in gs] if many else gs[0][1],
                        connection_index=[c for _, _, c in gs] if many else gs[0][2], **_settings(case))
    s.update(solver=solver, frame=0)
    n = solver.num_vertices
    if many or (kind == "frame" and case["state"]):
        s["out"] = torch.empty(solver.state_size() // 4, dtype=torch.float32, device="cuda")
    elif kind in ("frame", "hairhair"):
        s["x"] = torch.empty((n, 3), dtype=torch.float32, device="cuda")
        if _renders(case):
            s["q"] = torch.empty((n, 4), dtype=torch.float32, device="cuda")
        else:
            s["v"] = torch.empty((n, 3), dtype=torch.float32, device="cuda")
    if kind == "hairhair" or (kind == "frame" and case["schedule"] == "jacobi"):
        s["x0"] = torch.from_numpy(gs[0][0].positions).cuda()
        s["v0"] = torch.from_numpy(gs[0][1]).cuda()
    if kind == "hair":
        solver.set_hair_layout(case["strands"], case["row"])
        s["x"] = torch.zeros((case["strands"], case["row"], 3), dtype=torch.float32, pin_memory=True)
        s["v"] = torch.zeros((case["strands"], case["row"], 3), dtype=torch.float32, pin_memory=True)
        solver.download_hair(s["x"], s["v"])
    if kind == "adjoint":
        g = gs[0][0]
        rng = np.random.default_rng([seed, 1])
        s["unit"] = torch.from_numpy(solver.get_rest_darboux()).cuda()
        s["strand_of"] = torch.from_numpy(np.repeat(np.arange(g.num_strands), np.diff(g.strand_begin))).cuda()
        s["init"] = torch.from_numpy(solver.get_state()).cuda()
        scale, w = _adjoint_inputs(rng, g)
        s["scale"] = torch.from_numpy(scale).cuda().requires_grad_()
        s["w"] = torch.from_numpy(w).cuda()
    return s


def _adjoint_inputs(rng, g):
    """Stiffness scales and d loss / d x: each strand off its target by an offset that grows to its tip."""
    sb = np.asarray(g.strand_begin, np.int64)
    of = np.repeat(np.arange(g.num_strands), np.diff(sb))
    along = (np.arange(g.num_vertices) - sb[of]) / np.diff(sb)[of]
    w = rng.normal(0.0, 1.0, (g.num_strands, 3))[of] * along[:, None]
    return rng.uniform(0.5, 2.0, g.num_strands).astype(np.float32), w.astype(np.float32)


def run(s):
    kind = s["kind"]
    if kind == "bake":
        g = vbd.bake_sdf(s["vertices"], s["triangles"], (s["nx"], s["ny"], s["nz"]), s["lo"], s["hi"])
        return {"phi": g.phi, "grad": g.grad}
    solver = s["solver"]
    if kind == "adjoint":
        s["scale"].grad = None
        x = autograd.rollout_positions(s["scale"], solver, s["unit"], s["strand_of"], s["init"], s["frames"], s["dt"],
                                       s["every"])
        (x * s["w"]).sum().backward()
        return {"x": x.detach(), "grad": s["scale"].grad}
    if kind == "hair":  # UploadHair, SolveNextStep, DownloadHair
        solver.step_hair(s["dt"], s["x"], s["v"], s["x"], s["v"])
        return {"x": s["x"], "v": s["v"]}
    if kind == "batch":
        turn = np.array([_yaw(s["frame"] + j, s["dt"]) for j in range(s["steps"])], np.float32)
        s["frame"] += s["steps"]
        solver.batch_step(s["dt"], s["steps"], body_transforms=turn)
        return _state(solver, s["out"])
    if "x0" in s:  # the program sets the hair before the frame (UploadHair from device memory)
        solver.set_positions_velocities(s["x0"], s["v0"])
    solver.step(4e-4 * s["substeps"] if kind == "hairhair" else s["dt"])
    if "out" in s:
        return _state(solver, s["out"])
    if "q" in s:
        solver.get_positions_velocities(s["x"], None)
        return {"x": s["x"], "q": solver.get_orientations(s["q"])}
    solver.get_positions_velocities(s["x"], s["v"])
    return {"x": s["x"], "v": s["v"]}


def _renders(case):
    """Loops at the reference's substep of 4e-4 s take positions and material frames, as a renderer does: an
    FP32 velocity there is dx / h, a position's last bit divided by 4e-4 s, and carries few digits."""
    return case["kind"] == "hairhair" or (case["kind"] == "frame" and case["seg"] == 1e-3)


def _state(solver, out):
    parts = solver.split_state(solver.get_state_into(out))
    return {k: parts[k] for k in ("x", "v", "v_last", "q")}


def work(case):
    """Bytes: the state and constants of each vertex read once, the state written once, a step call (the
    host arrays where the call works on them).  Operations: the step's own arithmetic per vertex and
    iteration with its 3x3 block inverted in closed form, 220 FP32 operations; twice more for its adjoint."""
    kind = case["kind"]
    if kind == "bake":
        nodes, tris = case["nx"] * case["ny"] * case["nz"], 20 * 4 ** case["subdivisions"]
        # the nodes written once, the mesh read once; a distance takes at least one triangle's test a node
        return {"bytes": 16 * nodes + 48 * tris, "flops": 45 * nodes}
    strands = case.get("strands", 0)
    if kind == "batch":
        strands = case["grooms"] * (case["smax"] - case["smin"]) / math.log(case["smax"] / case["smin"])
    v = strands * 0.5 * (case["vmin"] + case["vmax"])
    it = case["itr"] * case.get("substeps", 1) * case.get("steps", 1) * case.get("frames", 1)
    if kind == "hair":
        return {"bytes": (160 + 48) * v, "flops": 220 * v * it}
    if kind == "adjoint":
        return {"bytes": 160 * v * case["frames"], "flops": 3 * 220 * v * it}
    return {"bytes": 160 * v, "flops": 220 * v * it}


# ---- 64-bit restatement -------------------------------------------------------------------------------


def _f32(a):
    return float(np.float32(a))


def _mul(l, r):
    lx, ly, lz, lw = l.unbind(-1)
    rx, ry, rz, rw = r.unbind(-1)
    return torch.stack([lw * rx + rw * lx + ly * rz - ry * lz, lw * ry + rw * ly + lz * rx - rz * lx,
                        lw * rz + rw * lz + lx * ry - rx * ly, lw * rw - lx * rx - ly * ry - lz * rz], -1)


def _conj(q):
    return q * q.new_tensor([-1.0, -1.0, -1.0, 1.0])


def _axis(q):  # q e_x q*
    x, y, z, w = q.unbind(-1)
    return torch.stack([w * w + x * x - y * y - z * z, 2 * (x * y + w * z), 2 * (x * z - w * y)], -1)


def _turn(q, v):
    u = q[:3].expand_as(v)
    a = q[3] * v + torch.cross(u, v, dim=-1)
    return q[3] * a + torch.cross(u, a, dim=-1) + (v * u).sum(-1, keepdim=True) * u


def _norm(v):
    return (v * v).sum(-1, keepdim=True).clamp_min(1e-60).sqrt()


class _Rods:
    """Strands padded to [S, L] (L even); even and odd vertices are the slices [:, 0::2] and [:, 1::2]."""

    def __init__(self, groom, vel, conn, st, dev):
        sb = np.asarray(groom.strand_begin, np.int64)
        n = np.diff(sb)
        S, L = len(n), int(n.max() + n.max() % 2)
        at = sb[:-1, None] + np.arange(L)[None]
        ok = np.arange(L)[None] < n[:, None]
        at[~ok] = 0
        self.at, self.ok, self.L = torch.from_numpy(at).to(dev), torch.from_numpy(ok).to(dev), L
        d = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=dev)  # noqa: E731
        pad = lambda a: d(a)[self.at] * (self.ok[..., None] if a.ndim == 2 else self.ok)  # noqa: E731
        self.x0, self.v0 = pad(groom.positions), pad(vel)
        k = torch.arange(L, device=dev)[None]
        nn = torch.from_numpy(n).to(dev)[:, None]
        self.hn, self.hp, self.hno = k + 1 < nn, (k > 0) & self.ok, k + 2 < nn
        self.root = (k == 0) & self.ok
        r, rho = _f32(st["radius"]), _f32(st["density"])
        seg = self.nxt(self.x0) - self.x0
        ln = torch.where(self.hn, _norm(seg)[..., 0], torch.ones_like(self.x0[..., 0]))
        lsum = torch.where(self.hn, ln, 0 * ln) + torch.where(self.hp, self.prv(ln), 0 * ln)
        mass = lsum * (r * r * math.pi * rho * 0.5)
        self.free = self.ok & ~self.root
        self.mass = torch.where(self.free, mass, torch.ones_like(mass))
        half = (seg / ln[..., None] + seg.new_tensor([1.0, 0.0, 0.0])) * 0.5
        hl = (half * half).sum(-1, keepdim=True)
        half = torch.where(hl > 0, half / hl.clamp_min(1e-60).sqrt(), half.new_tensor([0.0, 1.0, 0.0]).expand_as(half))
        q = torch.stack([0 * ln, -half[..., 2], half[..., 1], half[..., 0]], -1)
        q = torch.where(self.hn[..., None], q, self.prv(q))
        ident = q.new_tensor([0.0, 0.0, 0.0, 1.0]).expand_as(q)
        self.q0 = torch.where(self.ok[..., None], q, ident)
        young, dev_ = d(groom.strand_young)[:, None], d(groom.strand_dev)[:, None]
        mm = r * 1000.0
        ks = young * math.pi * mm * mm
        rq = _mul(_conj(self.q0), self.nxt(self.q0))
        self.qr = rq / _norm(rq) * (ks * dev_ * mm * mm * 0.25 / (ln * ln))[..., None]
        self.kk = ks / ln
        self.dd = torch.where(self.hn, self.kk / ln, 0 * ln)
        self.kn = torch.where(self.hn, self.kk, 0 * ln)
        self.st = st
        self.g = d([_f32(a) for a in st["gravity"]])
        self.wind = [_f32(a) for a in st.get("wind", WIND_OFF)]
        self.damp, self.decay = _f32(st["damping"]), _f32(st["velocity_decay"])
        self.tie = None
        if conn is not None and (np.asarray(conn) >= 0).any():
            flat = np.full(groom.num_vertices, -1, np.int64)
            flat[at[ok]] = np.arange(S * L).reshape(S, L)[ok]
            c = np.asarray(conn, np.int64)
            own = np.nonzero(c >= 0)[0]
            own = own[np.asarray(self.free.cpu()).reshape(-1)[flat[own]]]  # pinned vertices do not move
            self.tie = torch.from_numpy(flat[own]).to(dev), torch.from_numpy(flat[c[own]]).to(dev)
        sdf = st.get("sdf")
        self.sdf = sdf
        if sdf is not None:
            self.grid = torch.cat([d(sdf.grad).reshape(-1, 3), d(sdf.phi).reshape(-1, 1)], 1)
            lo, hi = np.asarray(sdf.grid_min, np.float32), np.asarray(sdf.grid_max, np.float32)
            self.lo, self.cell = d(lo), d((hi - lo) / np.asarray(sdf.dims, np.float32))

    def nxt(self, a):
        return torch.cat([a[:, 1:], torch.zeros_like(a[:, :1])], 1)

    def prv(self, a):
        return torch.cat([torch.zeros_like(a[:, :1]), a[:, :-1]], 1)

    def flat(self, a):
        out = a.new_zeros((int(self.ok.sum()),) + a.shape[2:])
        return out.index_put((self.at[self.ok],), a[self.ok])

    def predict(self, x, v, vl, h, last_h, time):
        ext = self.g.expand_as(x)
        if self.wind[0] != 0.0:
            peak, fy, fz, ft, sharp = self.wind
            c = torch.where(x[..., 1] > 0, torch.cos(2 * math.pi * (fy * x[..., 1] + ft * time)), 0 * x[..., 1])
            c = c * torch.cos(2 * math.pi * (fz * x[..., 2].abs() + ft * time))
            w = peak * (torch.sign(c) * c ** sharp).clamp_min(0.0)
            ext = ext + torch.stack([w, 0 * w, 0 * w], -1)
        dx = h * v
        y = dx + h * h * ext
        s = (((v - vl) / last_h * ext).sum(-1, keepdim=True) / (ext * ext).sum(-1, keepdim=True)).clamp(0.0, 1.0)
        m = self.free[..., None]
        return torch.where(m, dx + h * h * s * ext, dx), torch.where(m, y, v)

    def substep(self, x, v, vl, q, qr, h, last_h, time):
        jac = self.st.get("schedule") == "jacobi"
        damp = self.damp / h
        dx, y = self.predict(x, v, vl, h, last_h, time)
        e = torch.where(self.hn[..., None], self.nxt(x) - x, 0 * x)
        a = torch.where(self.free, self.mass / (h * h), 0 * self.mass)
        dp, kp = self.prv(self.dd), self.prv(self.kn)
        s = (self.dd + dp) * (1 + damp)
        f0 = a[..., None] * y + self.dd[..., None] * e - dp[..., None] * self.prv(e)
        if self.tie is not None:
            own, to = self.tie
            add = torch.zeros_like(s).reshape(-1)
            add[own] = K_TIE * (1 + damp)
            s = s + add.reshape(s.shape)
            pull = torch.zeros_like(x).reshape(-1, 3)
            pull[own] = K_TIE * (x.reshape(-1, 3)[own] - x.reshape(-1, 3)[to])
            f0 = f0 - pull.reshape(x.shape)
        ss = torch.where(self.free, s, torch.ones_like(s))
        sa = torch.where(self.free, 1 / ss, 0 * s)[..., None]
        sb = torch.where(self.free, 1 / (ss + 3 * a), 0 * s)[..., None]
        qn = torch.where(self.hno[..., None], qr, 0 * qr)
        qp = torch.where(self.hp[..., None], self.prv(qr), 0 * qr)
        upd = self.hn
        half = lambda t: (t[:, 0::2].contiguous(), t[:, 1::2].contiguous())  # noqa: E731
        c3 = lambda t: half(t[..., None])  # noqa: E731
        F0, DD, DP, KN, KP, AS, SA, SB = half(f0), c3(self.dd), c3(dp), c3(self.kn), c3(kp), c3(a + s), half(sa), half(sb)
        VE, M2 = half(-2 * self.kk[..., None] * e), c3(-2 * self.kk)
        QN, QP, UP = half(_conj(qn)), half(qp), c3(upd)
        DX, Q = list(half(dx)), list(half(q))

        def near(pair, c):  # (previous, next) values of colour c's vertices
            other = pair[1 - c]
            return (self.prv(other), other) if c == 0 else (other, self.nxt(other))

        def position(c, DX, Q, tied):
            p, n = near(DX, c)
            dq = _axis(Q[c])
            dqp = near((_axis(Q[0]) if c else dq, dq if c else _axis(Q[1])), c)[0]
            f = F0[c] + DD[c] * n + DP[c] * p - AS[c] * DX[c] - KN[c] * dq + KP[c] * dqp
            if tied is not None:
                f = f + tied[c]
            m = f.mean(-1, keepdim=True)
            return DX[c] + SA[c] * (f - m) + SB[c] * m

        def orientation(c, DX, Q):
            qprev, qnext = near(Q, c)
            V = VE[c] + M2[c] * (near(DX, c)[1] - DX[c])
            b = 0
            for P in (_mul(qprev, QP[c]), _mul(qnext, QN[c])):
                b = b + torch.where((Q[c] * P).sum(-1, keepdim=True) > 0, 1.0, -1.0).to(P.dtype) * P
            bq, bw = b[..., :3], b[..., 3:]
            pq = bw * V + torch.cross(V, bq, dim=-1)
            pw = -(V * bq).sum(-1, keepdim=True)
            r = torch.cat([pw, pq[..., 2:3], -pq[..., 1:2], -pq[..., 0:1]], -1) + (_norm(V) + _norm(b)) * b
            r = torch.where(UP[c], r, Q[c])
            return torch.where(UP[c], r / _norm(r), Q[c])

        for _ in range(self.st["num_itr"]):
            tied = None
            if self.tie is not None:  # the partners' displacements as the iteration starts
                own, to = self.tie
                now = torch.stack(DX, 2).reshape(-1, 3)
                t = torch.zeros_like(now)
                t[own] = K_TIE * now[to]
                tied = half(t.reshape(x.shape))
            if jac:
                DX = [position(0, DX, Q, tied), position(1, DX, Q, tied)]
                Q = [orientation(0, DX, Q), orientation(1, DX, Q)]
            else:
                DX[0] = position(0, DX, Q, tied)
                DX[1] = position(1, DX, Q, tied)
                Q[0] = orientation(0, DX, Q)
                Q[1] = orientation(1, DX, Q)
                DX, Q = list(DX), list(Q)
        dx = torch.stack(DX, 2).reshape(x.shape)
        q = torch.stack(Q, 2).reshape(q.shape)
        nv = torch.where(self.free[..., None], dx / h * (1 - self.decay * h), v)
        return x + dx, nv, v, q

    def collide(self, x, v, rot, tr):
        nx, ny, nz = self.sdf.dims
        rot = x.new_tensor([_f32(a) for a in rot])
        lp = _turn(_conj(rot), x - x.new_tensor([_f32(a) for a in tr])) - self.lo
        idx = torch.trunc(lp.detach() / self.cell + 0.5).long()
        top = torch.tensor([nx, ny, nz], device=x.device)
        hit = ((idx >= 0) & (idx < top)).all(-1) & self.ok & ~self.root
        u = lp / self.cell - (idx.to(x.dtype) - 0.5)
        res = 0
        for corner in range(8):
            o = torch.tensor([corner & 1, corner >> 1 & 1, corner >> 2], device=x.device)
            c = idx + o
            inside = (c < top).all(-1, keepdim=True)
            c = torch.minimum(c, top - 1).clamp_min(0)
            val = self.grid[c[..., 0] + nx * (c[..., 1] + ny * c[..., 2])]
            val = torch.cat([torch.where(inside, val[..., :3], 0 * val[..., :3]), val[..., 3:]], -1)
            res = res + torch.where(o > 0, u, 1 - u).prod(-1, keepdim=True) * val
        n = res[..., :3] / _norm(res[..., :3])
        phi = res[..., 3:] - _f32(self.sdf.threshold)
        hit = hit[..., None] & (phi < 0)
        speed = _norm(v)
        nv = v - (v / speed * n).sum(-1, keepdim=True) * n
        return torch.where(hit, x - phi * n, x), torch.where(hit & (speed >= 1e-6), nv, v)

    def advance(self, state, qr, dt, rot=(0.0, 0.0, 0.0, 1.0), tr=(0.0, 0.0, 0.0)):
        x, v, vl, q, last_h, time = state
        dt, max_h = np.float32(dt), np.float32(self.st["max_h"])
        n = max(1, int(math.ceil(dt / max_h)))
        h = float(np.float32(dt / np.float32(n)))
        for _ in range(n):
            x, v, vl, q = self.substep(x, v, vl, q, qr, h, last_h, time)
        if self.sdf is not None:
            x, v = self.collide(x, v, rot, tr)
        return x, v, vl, q, h, float(np.float32(time) + dt)

    def start(self):
        return self.x0, self.v0, torch.zeros_like(self.v0), self.q0, _f32(self.st["max_h"]), 0.0


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "bake":
        return _exact_bake(case, seed, dev)
    if kind == "hairhair":
        return None
    st = _settings(case)
    outs = []
    if kind == "adjoint":
        return _exact_adjoint(case, seed, st, dev)
    with torch.no_grad():
        for g, v, conn in _grooms(case, seed):
            r = _Rods(g, v, conn, st, dev)
            s = r.start()
            for j in range(case.get("steps", 1)):
                s = r.advance(s, r.qr, case["dt"], *((_yaw(j, case["dt"])[:4],) if kind == "batch" else ()))
            if kind == "hair":
                x = s[0].new_zeros((case["strands"], case["row"], 3))
                vv = x.clone()
                L = min(r.L, case["row"])
                x[:, :L] = (s[0] * r.ok[..., None])[:, :L]
                vv[:, :L] = (s[1] * r.ok[..., None])[:, :L]
                return {"x": x, "v": vv}
            outs.append([r.flat(a) for a in s[:4]])
            del r, s
        cat = [torch.cat(a) for a in zip(*outs)]
    got = dict(zip(("x", "v", "v_last", "q"), cat))
    keep = ("x", "q") if _renders(case) else got if kind == "batch" or case["state"] else ("x", "v")
    return {k: got[k] for k in keep}


def _exact_adjoint(case, seed, st, dev):
    from torch.utils.checkpoint import checkpoint

    g, v, _ = _grooms(case, seed)[0]
    r = _Rods(g, v, None, st, dev)
    scale, w = _adjoint_inputs(np.random.default_rng([seed, 1]), g)
    scale = torch.tensor(scale, dtype=torch.float64, device=dev, requires_grad=True)
    qr = r.qr * scale[:, None, None]
    s = r.start()
    for _ in range(case["frames"]):
        def frame(x, v, vl, q, qr, last_h=s[4], time=s[5]):
            return r.advance((x, v, vl, q, last_h, time), qr, case["dt"])
        s = checkpoint(frame, *s[:4], qr, use_reentrant=False)
    x = r.flat(s[0])
    (x * torch.from_numpy(w).to(dev).double()).sum().backward()
    return {"x": x.detach(), "grad": scale.grad}


def _exact_bake(case, seed, dev):
    v, t, lo, hi = _mesh(case, seed)
    dims = (case["nx"], case["ny"], case["nz"])
    tri = torch.from_numpy(v.astype(np.float64)).to(dev)[torch.from_numpy(t.astype(np.int64)).to(dev)]
    a, b, c = tri.unbind(1)
    lo32, hi32 = np.asarray(lo, np.float32), np.asarray(hi, np.float32)
    ds = ((hi32 - lo32) / np.asarray(dims, np.float32)).astype(np.float64)
    ax = [torch.as_tensor(float(lo32[k]) + ds[k] * np.arange(dims[k]), device=dev) for k in range(3)]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    p = torch.stack([x, y, z], -1).reshape(-1, 3)
    out = torch.empty(p.shape[0], dtype=torch.float64, device=dev)
    n = torch.cross(b - a, c - a, dim=-1)
    nn = (n * n).sum(-1)
    dot = lambda m, k: (m * k).sum(-1)  # noqa: E731
    step = max(1, (1 << 25) // tri.shape[0])
    for i in range(0, p.shape[0], step):
        q = p[i:i + step, None]
        pa, pb, pc = a - q, b - q, c - q
        best = torch.full(pa.shape[:2], math.inf, dtype=torch.float64, device=dev)
        inside = torch.ones_like(best, dtype=torch.bool)
        for u, w in ((pa, b - a), (pb, c - b), (pc, a - c)):
            f = (-dot(u, w) / dot(w, w)).clamp(0.0, 1.0)
            best = torch.minimum(best, ((u + f[..., None] * w) ** 2).sum(-1))
            inside &= dot(torch.cross(w.expand_as(u), -u, dim=-1), n) >= 0
        plane = dot(pa, n) ** 2 / nn
        best = torch.where(inside, plane, best).amin(1).sqrt()
        la, lb, lc = pa.norm(dim=-1), pb.norm(dim=-1), pc.norm(dim=-1)
        num = dot(pa, torch.cross(pb, pc, dim=-1))
        den = la * lb * lc + dot(pa, pb) * lc + dot(pb, pc) * la + dot(pc, pa) * lb
        turns = torch.atan2(num, den).sum(1) / (2 * math.pi)  # the winding number: 1 inside, 0 outside
        out[i:i + step] = torch.where(turns.abs() > 0.5, -best, best)
    return {"phi": out.reshape(dims[2], dims[1], dims[0]), "grad": None}
