"""Performance cases of the cloth step: what a user's program calls, over the sizes it is used at.

  listed()            the named cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) meshes, solver or tree handle and inputs, as a program has them before a call
  run(state)          one pass through the public entry points
  work(case)          bytes and floating-point operations one pass cannot do without
  exact(case, seed)   the first pass in 64 bits, for the case whose result is a smooth function of
                      its inputs (the hanging sheet).  Frames with contact or stiff bending branch
                      on float comparisons, and tree builds order integer codes: a 64-bit program
                      has another result there, not a more exact one.
"""
import ctypes
import heapq

import numpy as np
import torch

from xrtailor_gb300 import ClothSolver, Lbvh, _lib, diff, scenes

# Frames of a stepping case before the cloth starts over (drop, first contact, folds); the body
# walks its motion forwards and backwards over the same span, so it never jumps.
EPISODE = 24
BONES = 24


def listed():
    return [
        # a small banner pinned along its top edge, no obstacle: the smallest frame, one launch
        # after the other; positions stay on the device (a renderer reads them there)
        dict(name="banner_31x23", kind="hang", nx=31, ny=23, substeps=4, iterations=25),
        # the 64 x 64 sheet on the icosphere, self-collision on, every frame read to the host
        dict(name="sheet_64x64", kind="drop", nx=64, ny=64, substeps=10, iterations=10),
        # the garment on the skinned body: LRA, bending, contact; every frame read to the host
        dict(name="garment_256x256", kind="body", nx=256, ny=256, substeps=20, iterations=15),
        # an odd-sized garment with the FEM fabric on the same body
        dict(name="fem_garment_121x95", kind="fem", nx=121, ny=95, substeps=10, iterations=10),
        # a large folded sheet falling onto a ground plane: self-contact and bandwidth
        dict(name="folds_768x701", kind="folds", nx=768, ny=701, substeps=10, iterations=10),
        # 24 garments of uneven sizes, each on its own body, in one launch per phase
        dict(name="batch_24", kind="batch", count=24, sizes=4, tile=1024),
        # obstacle trees rebuilt inside a host application's frame, on its own buffers
        dict(name="tree_icosphere_1280", kind="tree", n=1280, shape="sphere"),
        dict(name="tree_body_13776", kind="tree", n=13776, shape="body"),
        # the 1024 x 1024 sheet's tree: build, refit to moved vertices, box queries
        dict(name="tree_sheet_1024", kind="requery", nx=1024, ny=1024, queries=1000),
        # one gradient of a loss on a short rollout of a few sheets
        dict(name="gradient_6x96x96", kind="gradient", count=6, n=96, frames=6),
        # the impact-zone collision step of a sheet crossing the sphere
        dict(name="impact_zone_96", kind="impact", n=96),
        # face pairs, proximity repulsion and impact tests of a rumpled sheet on the sphere
        dict(name="repulsion_150", kind="repulsion", n=150),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["hang", "drop", "body", "fem", "folds", "batch", "tree", "requery",
                       "gradient", "impact", "repulsion"])
    if kind == "hang":
        return dict(kind=kind, nx=_log(rng, 9, 120), ny=_log(rng, 9, 90),
                    substeps=rng.randint(1, 8), iterations=rng.randint(5, 40))
    if kind == "drop":
        return dict(kind=kind, nx=_log(rng, 20, 200), ny=_log(rng, 20, 200),
                    substeps=rng.randint(4, 12), iterations=rng.randint(4, 12))
    if kind == "body":
        return dict(kind=kind, nx=_log(rng, 60, 300), ny=_log(rng, 60, 260),
                    substeps=rng.randint(8, 20), iterations=rng.randint(6, 15))
    if kind == "fem":
        return dict(kind=kind, nx=_log(rng, 30, 160), ny=_log(rng, 30, 160),
                    substeps=rng.randint(4, 10), iterations=rng.randint(4, 10))
    if kind == "folds":
        return dict(kind=kind, nx=_log(rng, 250, 768), ny=_log(rng, 250, 700),
                    substeps=rng.randint(4, 10), iterations=rng.randint(5, 10))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(3, 24), sizes=rng.randint(5, 1 << 16),
                    tile=rng.choice([256, 512, 1024]))
    if kind == "tree":
        return dict(kind=kind, n=_log(rng, 2, 65536), shape="soup")
    if kind == "requery":
        return dict(kind=kind, nx=_log(rng, 100, 1000), ny=_log(rng, 100, 1000),
                    queries=_log(rng, 50, 1000))
    if kind == "gradient":
        return dict(kind=kind, count=rng.randint(1, 6), n=_log(rng, 24, 96),
                    frames=rng.randint(1, 6))
    if kind == "impact":
        return dict(kind=kind, n=_log(rng, 24, 96))
    return dict(kind=kind, n=_log(rng, 24, 150))


# ---- what a program has in hand ------------------------------------------------------------------

def _triangle_soup(case, seed):
    """(n, 9) float32 triangles: an icosphere's, the body's at a pose, or scattered small ones."""
    if case["shape"] == "sphere":
        m = scenes.icosphere(3, 0.3, center=np.random.default_rng(seed).uniform(-0.2, 0.2, 3))
        return m.positions[m.triangles].reshape(-1, 9)
    if case["shape"] == "body":
        b = scenes.TubeBody(seed=seed)
        return b.pose(0.25)[b.triangles].reshape(-1, 9)
    rng = np.random.default_rng(seed)
    c = rng.uniform(-1.0, 1.0, (case["n"], 1, 3))
    return (c + rng.normal(0.0, 0.01, (case["n"], 3, 3))).reshape(-1, 9).astype(np.float32)


def _hanging(case, seed):
    cloth = scenes.rect_cloth(case["nx"], case["ny"], 1.0, 0.7, jitter=1e-3, seed=seed)
    cloth.fixed_indices = np.arange(case["nx"], dtype=np.uint32)
    v0 = np.random.default_rng(seed + 1).normal(0.0, 0.05, cloth.positions.shape)
    v0[:case["nx"]] = 0.0
    return cloth, v0.astype(np.float32)


HANG = dict(stretch_compliance=1e-6, solve_bending=0, enable_self_collision=0,
            num_collision_passes=1)


def _stepping(case, solver, x_init, v_init=None, motion=None, to_host=False):
    v = np.zeros_like(x_init) if v_init is None else v_init
    return dict(kind="step", solver=solver, x=x_init, v=v, motion=motion, to_host=to_host, frame=0,
                reset=case["kind"] != "hang")


def _body_motion(bodies, device):
    """Joint transforms of EPISODE frames at 60 fps, all bodies' joints one after the other: host
    arrays, or device tensors for a batch."""
    t = np.stack([np.concatenate([b.joint_transforms(f / 60.0) for b in bodies]).reshape(-1)
                  for f in range(EPISODE)]).astype(np.float32)
    return torch.from_numpy(t).cuda() if device else t


def _skin(solver, bodies):
    """Binds every body's vertices to its own bones (numbered across the bodies)."""
    parts = [b.skin() for b in bodies]
    rest = np.concatenate([p[0] for p in parts])
    joints = np.concatenate([p[2] + BONES * k for k, p in enumerate(parts)]).astype(np.uint32)
    weights = np.concatenate([p[3] for p in parts])
    solver.set_obstacle_skinning(rest, np.arange(len(rest) + 1, dtype=np.uint32), joints, weights,
                                 BONES * len(bodies))


def _state_of(solver):
    """The resident positions and velocities (V x 4) as tensors on the solver's own buffers; each
    tensor keeps its Buffer, and so the solver, alive."""
    x, v, _ = solver.device_state()
    n = solver.sizes().num_vertices

    class Buffer:
        def __init__(self, ptr):
            self.solver = solver
            self.__cuda_array_interface__ = dict(shape=(n, 4), typestr="<f4", data=(ptr, False),
                                                 version=3)
    return torch.as_tensor(Buffer(x), device="cuda"), torch.as_tensor(Buffer(v), device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("hang", "drop", "body", "fem", "folds"):
        return _prepare_frame(case, seed)
    if kind == "batch":
        return _prepare_batch(case, seed)
    if kind == "tree":
        d = torch.from_numpy(_triangle_soup(case, seed)).cuda()
        n = d.shape[0]
        i32 = dict(dtype=torch.int32, device="cuda")
        out = dict(morton=torch.empty(n, **i32), objects=torch.empty(n, **i32),
                   nodes=torch.empty(2 * n - 1, 4, **i32),
                   boxes=torch.empty(2 * n - 1, 6, dtype=torch.float32, device="cuda"),
                   internal_escape=torch.empty(n - 1, **i32), leaf_escape=torch.empty(n, **i32))
        return dict(kind="tree", lib=_lib.load(), prims=d, out=out)
    if kind == "requery":
        m = scenes.rect_cloth(case["nx"], case["ny"], 2.0, 2.0, jitter=1e-4, seed=seed)
        rng = np.random.default_rng(seed)
        p = m.positions
        p[:, 1] = 0.05 * np.sin(5.0 * p[:, 0] + rng.uniform(0, 6)) * np.sin(4.0 * p[:, 2])
        x = torch.from_numpy(p).cuda()
        tri = torch.from_numpy(m.triangles.astype(np.int64)).cuda()
        moved = x + torch.tensor([0.002, -0.003, 0.001], device="cuda")
        c = p[rng.integers(0, len(p), case["queries"])]
        half = rng.uniform(0.001, 0.006, (case["queries"], 1))
        boxes = np.concatenate([c - half, c + half], 1).astype(np.float32)
        return dict(kind="requery", tree=Lbvh(), prims=x[tri].reshape(-1, 9).contiguous(),
                    pred=moved[tri].reshape(-1, 9).contiguous(), boxes=boxes,
                    slots=np.arange(256, dtype=np.uint32))
    if kind == "gradient":
        return _prepare_gradient(case, seed)
    return _prepare_contact(case, seed)


def _prepare_frame(case, seed):
    kind, nx, ny = case["kind"], case["nx"], case["ny"]
    steps = dict(num_substeps=case["substeps"], num_iterations=case["iterations"])
    if kind == "hang":
        cloth, v0 = _hanging(case, seed)
        s = ClothSolver(scenes._params(**steps, **HANG))
        s.add_cloth(cloth)
        s.start()
        s.set_state(None, v0)
        return _stepping(case, s, cloth.positions, v0)
    passes = dict(num_collision_passes=min(10, case["substeps"] * case["iterations"]))
    if kind == "drop":
        cloth = scenes.rect_cloth(nx, ny, 1.0, (ny - 1) / (nx - 1), origin=(0.0, 0.4, 0.0),
                                  jitter=1e-3, seed=seed)
        cloth.fixed_indices = np.array([0, nx - 1], np.uint32)
        s = ClothSolver(scenes._params(stretch_compliance=1e-8, bend_compliance=1e-6, **steps,
                                       **passes))
        s.add_cloth(cloth, particle_diameter=2e-3 * 64 / nx)
        s.add_obstacle(scenes.icosphere(3, 0.3, center=(0.5, 0.0, 0.5)))
        s.start()
        return _stepping(case, s, cloth.positions, to_host=True)
    if kind == "folds":
        rng = np.random.default_rng(seed)
        cloth = scenes.rect_cloth(nx, ny, 2.0, 2.0, origin=(-1.0, 0.0, -1.0), jitter=1e-4,
                                  seed=seed)
        p = cloth.positions.astype(np.float64)
        k, ph = rng.uniform(2, 6, 2), rng.uniform(0, 2 * np.pi, 2)
        p[:, 1] = (0.02 + 0.3 * (p[:, 0] + 1.0)
                   + 0.05 * np.sin(k[0] * p[:, 0] + ph[0]) * np.sin(k[1] * p[:, 2] + ph[1]))
        cloth.positions = p.astype(np.float32)
        s = ClothSolver(scenes._params(stretch_compliance=1e-8, bend_compliance=1e-6, **steps,
                                       **passes))
        s.add_cloth(cloth, particle_diameter=1e-3)
        s.add_obstacle(scenes.ground_plane(64, 6.0, height=-0.05))
        s.start()
        return _stepping(case, s, cloth.positions)
    # a garment on the body, draped from above and held at two corners
    body = scenes.TubeBody(seed=seed)
    depth = (ny - 1) / (nx - 1)
    cloth = scenes.rect_cloth(nx, ny, 1.0, depth, origin=(-0.5, body.height + 0.05, -0.5 * depth),
                              jitter=1e-3, seed=seed)
    cloth.fixed_indices = cloth.attached_indices = np.array([0, nx - 1], np.uint32)
    s = ClothSolver(scenes._params(stretch_compliance=1e-8, bend_compliance=1e-6, **steps,
                                   **passes))
    if kind == "fem":
        s.set_fem_material()
    s.add_cloth(cloth)
    s.add_obstacle(body.mesh)
    s.start()
    _skin(s, [body])
    return _stepping(case, s, cloth.positions, motion=_body_motion([body], False),
                     to_host=kind == "body")


def _prepare_batch(case, seed):
    """Garments of seeded uneven sizes (2,000 to 100,000 vertices, log-uniform; aspect 0.5 to 2),
    each with its own body and stretch compliance."""
    rng = np.random.default_rng(seed)
    s = ClothSolver(scenes._params(**scenes.BATCHED_PARAMS))
    s.set_tile_vertices(case["tile"])
    bodies, starts, comp = [], [], []
    for k, (nx, ny) in enumerate(scenes.batched_grid_dims(case["count"], case["sizes"])):
        body = scenes.TubeBody(seed=seed + k)
        depth = (ny - 1) / (nx - 1)
        cloth = scenes.rect_cloth(nx, ny, 1.0, depth,
                                  origin=(-0.5, body.height + 0.05, -0.5 * depth), jitter=1e-3,
                                  seed=seed + k)
        cloth.fixed_indices = cloth.attached_indices = np.array([0, nx - 1], np.uint32)
        s.add_instance(cloth, body.mesh)
        bodies.append(body)
        starts.append(cloth.positions)
        edges = nx * (ny - 1) + ny * (nx - 1) + (nx - 1) * (ny - 1)
        comp.append(np.full(edges, 10.0 ** rng.uniform(-9, -5), np.float32))
    s.set_compliance(0, np.concatenate(comp))
    s.start()
    _skin(s, bodies)
    return _stepping(case, s, np.concatenate(starts), motion=_body_motion(bodies, True))


def _prepare_gradient(case, seed):
    inst = scenes.diff_batch(case["count"], case["n"], seed=seed)
    s = ClothSolver(scenes._params(**scenes.DIFF_PARAMS))
    for d in inst:
        s.add_instance(d.cloth, d.sphere)
    s.start()
    x0 = np.concatenate([d.cloth.positions for d in inst])
    cat = lambda name: torch.from_numpy(np.concatenate([getattr(d, name) for d in inst]))  # noqa: E731
    leaves = [torch.from_numpy(x0), cat("velocity"), cat("mass"), cat("stretch_compliance"),
              cat("bend_compliance")]
    target = torch.from_numpy(x0) + torch.tensor([0.0, -0.05, 0.0])
    return dict(kind="gradient", solver=s, frames=case["frames"], target=target,
                leaves=[t.requires_grad_(True) for t in leaves])


def _prepare_contact(case, seed):
    n = case["n"]
    s = ClothSolver(scenes._params(num_substeps=2, num_iterations=3, solve_bending=0,
                                   num_collision_passes=2, enable_self_collision=0))
    cloth = scenes.grid_cloth(n, 1.0, origin=(0.0, 0.35, 0.0), jitter=1e-3, seed=seed)
    cloth.fixed_indices = scenes.two_corner_pins(n)
    s.add_cloth(cloth)
    s.add_obstacle(scenes.icosphere(2, 0.3, center=(0.5, 0.0, 0.5)))
    s.start()
    s.fixed_update(4)
    pred = s.host_positions()
    if case["kind"] == "impact":  # every vertex over the sphere's cap crosses it in the step
        pred[:, 1] -= 0.12
        return dict(kind="impact", solver=s, pred=pred)
    noise = np.random.default_rng(seed).normal(0.0, 0.2 / n, pred.shape)  # a fifth of an edge
    return dict(kind="repulsion", solver=s, pred=(pred + noise).astype(np.float32))


# ---- one pass -------------------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "step":
        return _run_frame(state)
    if kind == "tree":
        o, d = state["out"], state["prims"]
        p = lambda t: ctypes.c_void_p(t.data_ptr() or None)  # noqa: E731
        _lib.check(state["lib"].xrt_lbvh_build_noalloc(
            p(d), None, d.shape[0], 0.0, p(o["morton"]), p(o["objects"]), p(o["nodes"]),
            p(o["boxes"]), p(o["internal_escape"]), p(o["leaf_escape"]),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream or None)))
        return o
    if kind == "requery":
        t, d = state["tree"], state["prims"]
        t.build_device(d.data_ptr(), d.shape[0])
        t.refit_device(state["pred"].data_ptr())
        counts, cands = t.query(2, state["boxes"])
        return counts, np.where(state["slots"] < counts[:, None], cands, 0)
    if kind == "gradient":
        x, v = diff.rollout(state["solver"], state["frames"], *state["leaves"])
        loss = ((x - state["target"]) ** 2).sum()
        return (x.detach(), v.detach()) + torch.autograd.grad(loss, state["leaves"])
    s = state["solver"]
    s.set_predicted(state["pred"])
    if kind == "impact":
        stats = s.collision_step()
        return s.predicted(), stats["passes"], stats["impacts"], stats["solves"]
    s.cloth_bvh_build()
    s.obstacle_bvh_update_ccd()
    pairs = s.update_pairs(1e-6)
    s.proximity_solve(1e-4, 0.25)
    impacts = s.check_impacts(1e-4)
    return s.predicted(), pairs, impacts


def _run_frame(state):
    s, f = state["solver"], state["frame"]
    if state["reset"] and f and f % EPISODE == 0:  # the next take of the same drop
        s.set_state(state["x"], state["v"])
    if state["motion"] is not None:
        k = f % (2 * EPISODE)
        m = state["motion"][k if k < EPISODE else 2 * EPISODE - 1 - k]
        if isinstance(m, torch.Tensor):
            s.set_joint_transforms_device(m.data_ptr())
        else:
            s.set_joint_transforms(m)
    s.fixed_update()
    state["frame"] = f + 1
    if state["to_host"]:
        return s.host_positions(), s.host_velocities()
    return _state_of(s)


# ---- what a pass cannot do without -----------------------------------------------------------------

def _frame_work(nx, ny, substeps, iterations, bend=True, collide=True, obstacle=0):
    """A frame's state and records once, and the projections' arithmetic.  Per substep and vertex
    12 operations of integration; per iteration 45 per stretch constraint, 230 per bend element,
    30 per vertex and kept neighbor (about 4) of the particle collision."""
    V = nx * ny
    E = nx * (ny - 1) + ny * (nx - 1) + (nx - 1) * (ny - 1)
    B = E - 2 * (nx - 1) - 2 * (ny - 1) if bend else 0
    flops = substeps * (12 * V + iterations * (45 * E + 230 * B + (120 * V if collide else 0)))
    return 100 * V + 16 * E + 24 * B + 84 * obstacle, flops


def work(case):
    kind = case["kind"]
    if kind in ("hang", "drop", "body", "fem", "folds"):
        faces = dict(hang=0, drop=1280, body=13776, fem=13776, folds=2 * 63 * 63)[kind]
        b, f = _frame_work(case["nx"], case["ny"], case["substeps"], case["iterations"],
                           bend=kind != "hang", collide=kind != "hang", obstacle=faces)
        return dict(bytes=b, flops=f)
    if kind == "batch":
        parts = [_frame_work(nx, ny, 10, 10, obstacle=13776)
                 for nx, ny in scenes.batched_grid_dims(case["count"], case["sizes"])]
        return dict(bytes=sum(p[0] for p in parts), flops=sum(p[1] for p in parts))
    if kind == "tree":  # triangles in; codes, order, nodes, boxes and escapes out
        return dict(bytes=case["n"] * (36 + 8 + 32 + 48 + 8), flops=60 * case["n"])
    if kind == "requery":  # triangles, their moved copy, the boxes of both passes
        n = 2 * (case["nx"] - 1) * (case["ny"] - 1)
        return dict(bytes=n * (36 + 36 + 2 * 64) + case["queries"] * 200, flops=100 * n)
    if kind == "gradient":  # every frame forward, again, and backward (about twice a forward)
        b, f = _frame_work(case["n"], case["n"], 10, 10, collide=False, obstacle=1280)
        k = case["count"] * case["frames"]
        return dict(bytes=4 * b * k, flops=4 * f * k)
    n = case["n"]
    if kind == "impact":  # about 10 passes of pairs and impact tests
        return dict(bytes=10 * 400 * n * n, flops=10 * 20000 * n * n)
    return dict(bytes=1000 * n * n, flops=8000 * n * n)


# ---- the hanging sheet in 64 bits --------------------------------------------------------------------

def _edges(tri):
    """Edges in order of first appearance over the faces, oriented as there."""
    seen, out = set(), []
    for f in tri.tolist():
        for k in range(3):
            a, b = f[k], f[(k + 1) % 3]
            key = (min(a, b), max(a, b))
            if key not in seen:
                seen.add(key)
                out.append((a, b))
    return np.array(out)


def _first_free(used):
    k = 0
    while used >> k & 1:
        k += 1
    return k


def _sweeps(edges, nv, tile=256):
    """The order constraints are projected in: tiles of consecutive vertices by tile color, and
    inside a tile by local color (both greedy, first free color); one array of edges per sweep."""
    tile_of = edges.min(1) // tile
    tiles = {}
    for e, t in enumerate(tile_of.tolist()):
        tiles.setdefault(t, []).append(e)
    vertex_mask = [0] * nv
    sweeps = []
    for t in sorted(tiles):
        foot = np.unique(edges[tiles[t]]).tolist()
        used = 0
        for v in foot:
            used |= vertex_mask[v]
        tc = _first_free(used)
        for v in foot:
            vertex_mask[v] |= 1 << tc
        mask = dict.fromkeys(foot, 0)
        for e in tiles[t]:
            a, b = edges[e].tolist()
            lc = _first_free(mask[a] | mask[b])
            mask[a] |= 1 << lc
            mask[b] |= 1 << lc
            heapq.heappush(sweeps, (tc, lc, e))
    by_color = {}
    while sweeps:
        tc, lc, e = heapq.heappop(sweeps)
        by_color.setdefault((tc, lc), []).append(e)
    return [np.array(v) for v in by_color.values()]


def exact(case, seed):
    if case["kind"] != "hang":
        return None
    cloth, v0 = _hanging(case, seed)
    x = cloth.positions.astype(np.float64)
    v = v0.astype(np.float64)
    edges = _edges(cloth.triangles)
    sweeps = _sweeps(edges, len(x))
    rest = np.linalg.norm(x[edges[:, 0]] - x[edges[:, 1]], axis=1)
    w = np.ones(len(x))
    w[:case["nx"]] = 0.0
    dt = 1.0 / 60.0 / case["substeps"]
    alpha = HANG["stretch_compliance"] / (dt * dt)
    for _ in range(case["substeps"]):
        start = x.copy()
        v[w > 0] += np.array([0.0, -9.8, 0.0]) * dt
        x = x + v * dt
        lam = np.zeros(len(edges))
        for _ in range(case["iterations"]):
            for s in sweeps:
                i, j = edges[s, 0], edges[s, 1]
                d = x[i] - x[j]
                n = np.linalg.norm(d, axis=1)
                dl = (-(n - rest[s]) - alpha * lam[s]) / (w[i] + w[j] + alpha)
                dl[(w[i] + w[j]) == 0.0] = 0.0
                lam[s] += dl
                c = d * (dl / (n + 1e-6))[:, None]
                x[i] += c * w[i][:, None]
                x[j] -= c * w[j][:, None]
        v = (x - start) / dt * (1.0 - 0.98 * dt)
    pad = lambda a: np.concatenate([a, np.zeros((len(a), 1))], 1)  # noqa: E731
    return pad(x), pad(v)
