"""What this framework is timed on: the calls its users make, at the sizes they make them.

A case is a plain dict. Its "kind" says which public entry points a pass goes through:

  solver   Solver.Step(steps), then what a frame or a checkpoint reads back (GetParticlePositions or get_state)
  batch    Batch.step(steps) of many independent 2D scenes, then every scene's positions
  train    Mlp.train(steps) of the learned return map, then its parameters
  render   Solver.render() of the current particles
  sample   sample_shapes() of a snow shape

A solver, a batch and a network keep their state from one pass to the next, as they do in a program that steps frame
after frame. Inputs come from the seed alone.
"""
import math

import numpy as np
import torch

from mpm_snow_sim2d_b200 import Solver, _lib, scenes
from mpm_snow_sim2d_b200.batch import Batch
from mpm_snow_sim2d_b200.mlp import DEFAULT_WEIGHTS, MIXED_WEIGHTS, N_PARAMS, OFF, Mlp, normalization
from mpm_snow_sim2d_b200.sampling import ball, box, sample_shapes

REFERENCE_MIN_DIST = float(np.float32(15.0) / np.cbrt(np.float32(3000.0)))


def listed():
    solver = dict(kind="solver", stencil="cubic", boundary="friction", plasticity="exact", returns="positions")
    return [
        # the interactive viewer: one step and the positions of a small scene, where launches and latency count
        dict(solver, name="viewer_2d_128", scene="blocks", dim=2, W=128, ppc=4, blocks=3, steps=1, returns="state"),
        # one output frame (33 steps, 1/30 s at the reference's time step) of the 512^2 scene of eight blocks
        dict(solver, name="frame_2d_512", scene="blocks", dim=2, W=512, ppc=8, blocks=8, steps=33),
        # the same grid at 27 particles per cell: the largest 2D scene
        dict(solver, name="frame_2d_512_dense", scene="blocks", dim=2, W=512, ppc=27, blocks=8, steps=33),
        # the reference's own 3D scene as its two snowballs meet: few particles, their mass and volume per particle
        dict(solver, name="frame_3d_reference", scene="reference", dim=3, W=200, ppc=1, blocks=2, steps=33,
             returns="state"),
        # the headline workload: a snowball above a resting slab, 1.65M particles
        dict(solver, name="frame_3d_slab_128", scene="slab", dim=3, W=128, ppc=8, blocks=2, steps=33),
        # the largest workload: two snowballs colliding, 3.8M particles, most of the work in plastic flow
        dict(solver, name="frame_3d_collision_256", scene="collision", dim=3, W=256, ppc=8, blocks=2, steps=33),
        # the headline workload on the quadratic stencil
        dict(solver, name="frame_3d_quadratic_128", scene="slab", dim=3, W=128, ppc=8, blocks=2, steps=33,
             stencil="quadratic"),
        # a collision with the learned return map
        dict(solver, name="frame_3d_learned_128", scene="collision", dim=3, W=128, ppc=8, blocks=2, steps=33,
             plasticity="learned"),
        # the batched workload: 256 scenes of 2k to 64k particles, a data set's worth of steps
        dict(kind="batch", name="batch_2d_256", scenes=256, steps=100),
        # training the learned return map, at the batch size the shipped weights were trained with
        dict(kind="train", name="train_return_map", steps=16, batch=16384, pairs=200000),
        # one picture of the headline workload at the reference's window size
        dict(kind="render", name="render_3d_slab", scene="slab", dim=3, W=128, ppc=8, width=1200, height=600,
             point_size=1.0),
        # filling one of the reference's snowballs when a scene is set up
        dict(kind="sample", name="sample_3d_ball", dim=3, shape="ball", size=15.0, min_dist=REFERENCE_MIN_DIST,
             rounds=30),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choices(["2d", "3d", "batch", "train", "render", "sample"], [30, 40, 10, 8, 6, 6])[0]
    steps = int(round(_log(rng, 1, 33)))
    solver = dict(kind="solver", plasticity="exact", stencil=rng.choice(["cubic", "cubic", "quadratic"]),
                  boundary=rng.choice(["friction", "friction", "sticky"]), steps=steps)
    if kind == "2d":
        return dict(solver, scene="blocks", dim=2, W=int(round(_log(rng, 64, 512))), ppc=int(round(_log(rng, 2, 27))),
                    blocks=rng.randint(1, 8), returns=rng.choice(["positions", "state"]))
    if kind == "3d":
        scene = rng.choice(["slab", "collision", "reference"])
        if scene == "reference":
            return dict(solver, scene=scene, dim=3, W=rng.randint(80, 240), ppc=rng.randint(1, 8), blocks=2,
                        returns="state")
        W = int(round(_log(rng, 32, 128 if scene == "slab" else 256)))
        c = dict(solver, scene=scene, dim=3, W=W, ppc=rng.randint(4, 8), blocks=2, returns="positions")
        if scene == "collision" and c["stencil"] == "cubic" and rng.random() < 0.4:
            c.update(plasticity="learned", W=min(W, 160))
        return c
    if kind == "batch":
        return dict(kind="batch", scenes=int(round(_log(rng, 8, 256))), steps=int(round(_log(rng, 1, 100))))
    if kind == "train":
        return dict(kind="train", steps=rng.randint(1, 16), batch=int(round(_log(rng, 1000, 20000))),
                    pairs=rng.randint(20000, 300000))
    if kind == "render":
        return dict(kind="render", scene=rng.choice(["slab", "collision"]), dim=3, W=rng.randint(32, 128),
                    ppc=rng.randint(4, 8), width=rng.randint(320, 1920), height=rng.randint(240, 1080),
                    point_size=round(rng.uniform(1.0, 4.0), 2))
    dim, shape = rng.choice([2, 3]), rng.choice(["ball", "box"])
    return dict(kind="sample", dim=dim, shape=shape, size=round(rng.uniform(6.0, 15.0), 3),
                min_dist=round(rng.uniform(0.2, 0.4) if dim == 2 else rng.uniform(0.8, 1.4), 4), rounds=30)


# ---------------------------------------------------------------------------------------------------------------------
# Inputs

MATERIAL = scenes.MATERIAL
MARGIN = scenes.MARGIN


def _ball(rng, center, radius, n):
    """n points uniform in a ball (a disk in 2D)."""
    d = len(center)
    u = rng.standard_normal((n, d))
    u *= (radius * rng.random(n) ** (1.0 / d) / np.sqrt((u * u).sum(1)))[:, None]
    return u + np.asarray(center)


def _block_sides(case):
    """Sides of the blocks (fractions of the domain): a tenth of it on average, all of them within 0.09 of its area."""
    k = case["blocks"]
    s = np.linspace(0.05, 0.15, k) if k > 1 else np.array([0.15])
    return s * min(1.0, math.sqrt(0.09 / float((s * s).sum())))


def _count(case):
    """Particles of a solver's scene."""
    W, ppc = case["W"], case["ppc"]
    if case["scene"] == "blocks":
        return int(sum(round((s * W) ** 2 * ppc) for s in _block_sides(case)))
    if case["scene"] == "slab":
        m = MARGIN / W
        return int(round(4 / 3 * math.pi * (0.12 * W) ** 3 * ppc)) + int(round((1 - 2 * m) ** 2 * 0.1 * W ** 3 * ppc))
    if case["scene"] == "collision":
        return 2 * int(round(4 / 3 * math.pi * (0.15 * W) ** 3 * ppc))
    return 2 * 8800 * ppc


def _physical(case, seed):
    """Positions and velocities on the unit domain (in cells for the reference's scene)."""
    rng = np.random.Generator(np.random.PCG64(seed))
    W, ppc, kind = case["W"], case["ppc"], case["scene"]
    if kind == "blocks":  # squares placed apart, that fall and turn (their corners at about the speed of the fall)
        sides = rng.permutation(_block_sides(case))
        while True:
            boxes = []
            for s in sorted(sides, reverse=True):
                for _ in range(400):
                    lo = rng.uniform((MARGIN + 2) / W, 1 - (MARGIN + 2) / W - s, 2)
                    if all(np.any(lo + s <= b) or np.any(lo >= b + t) for b, t in boxes):
                        boxes.append((lo, s))
                        break
            if len(boxes) == len(sides):
                break
        pos, vel = [], []
        for lo, s in boxes:
            p = s * rng.random((int(round((s * W) ** 2 * ppc)), 2))
            spin = rng.uniform(1.0, 2.0) * rng.choice([-1.0, 1.0]) / s
            pos.append(lo + p)
            vel.append(np.array([0.0, -1.0]) + spin * (p - 0.5 * s)[:, ::-1] * np.array([-1.0, 1.0]))
        pos, vel = np.concatenate(pos), np.concatenate(vel)
        return pos, vel + rng.uniform(-0.1, 0.1, pos.shape)
    n = _count(case)
    if kind == "slab":  # a snowball falling towards a slab that rests on the floor
        m = MARGIN / W
        nb = int(round(4 / 3 * math.pi * (0.12 * W) ** 3 * ppc))
        top = _ball(rng, (0.5, 0.7, 0.5), 0.12, nb)
        low = np.array([m, m, m]) + rng.random((n - nb, 3)) * np.array([1 - 2 * m, 0.1, 1 - 2 * m])
        vel = np.zeros((n, 3))
        vel[:nb, 1] = -3.0
        return np.concatenate([top, low]), vel
    if kind == "collision":  # two snowballs about to touch, closing at 6
        r, gap = 0.15, 2.0 / W
        a = _ball(rng, (0.5 - r - gap / 2, 0.5, 0.5), r, n // 2)
        b = _ball(rng, (0.5 + r + gap / 2, 0.5, 0.5), r, n // 2)
        vel = np.zeros((n, 3))
        vel[: n // 2, 0], vel[n // 2:, 0] = 3.0, -3.0
        return np.concatenate([a, b]), vel
    # the reference's scene (200 x 100 x 100 cells, radius 15, speed 40) as its snowballs meet, each turning
    k = W / 200.0
    r, c = 15.0 * k, np.array([W / 2.0, W / 4.0, W / 4.0])
    off = np.array([r + 0.75, -5.0 * k, 0.0])
    pos, vel = [], []
    for sign in (-1.0, 1.0):
        p = _ball(rng, c + sign * off, r, n // 2)
        spin = rng.uniform(0.4, 0.8, 3) * (40.0 * k / r) * sign
        pos.append(p)
        vel.append(np.array([-sign * 40.0 * k, 0.0, 0.0]) + np.cross(spin, p - (c + sign * off)))
    return np.concatenate(pos), np.concatenate(vel)


def _scene(case, seed):
    """The scene in the framework's units (cells)."""
    W, dim, ppc = case["W"], case["dim"], case["ppc"]
    pos, vel = _physical(case, seed)
    n = pos.shape[0]
    form = _lib.FORMULATION_MLS_QUADRATIC if case.get("stencil") == "quadratic" else _lib.FORMULATION_MLS
    bound = _lib.BOUNDARY_STICKY if case.get("boundary") == "sticky" else _lib.BOUNDARY_FRICTION
    f32 = lambda a: np.ascontiguousarray(a, np.float32)  # noqa: E731
    if case["scene"] == "reference":
        R = scenes.REFERENCE_DEFAULT
        total = 4 / 3 * math.pi * (R["radius"] * W / 200.0) ** 3
        volume = np.where(np.arange(n) < n // 2, 1.0, 1.02) * (total / (n // 2))
        return scenes.Scene(
            name="reference", dim=3, width=W, height=W // 2, depth=W // 2, border_margin=R["margin"],
            delta_time=R["delta_time"], gravity=R["gravity"], friction=R["friction"], theta_c=R["theta_c"],
            theta_s=R["theta_s"], xi=R["xi"], nu=R["nu"], youngs=R["youngs"], rho=R["rho"], steps=case.get("steps", 0),
            position=f32(pos), velocity=f32(vel), volume=f32(volume), mass=f32(volume * R["rho"] / 100.0),
            formulation=form, boundary=bound)
    dx = 1.0 / W
    rho = MATERIAL["rho_phys"] * dx * dx * 100.0
    volume = np.full(n, 1.0 / ppc, np.float32)
    dt = 1e-4 * 128.0 / W if dim == 2 else 5e-5 * min(1.0, 256.0 / W)
    return scenes.Scene(
        name=case["scene"], dim=dim, width=W, height=W, depth=W if dim == 3 else 0, border_margin=MARGIN,
        delta_time=dt, gravity=-9.8 / dx, friction=scenes.FRICTION, theta_c=MATERIAL["theta_c"],
        theta_s=MATERIAL["theta_s"], xi=MATERIAL["xi"], nu=MATERIAL["nu"], youngs=MATERIAL["youngs"], rho=rho,
        steps=case.get("steps", 0), position=f32(pos / dx), velocity=f32(vel / dx), volume=volume,
        mass=f32(volume * np.float32(rho) / np.float32(100.0)), formulation=form, boundary=bound)


def _batch_sizes(index):
    """Grid side, block sides (cells), particles per cell and material of scene `index`: the ranges of the batched
    workload (sides 64-256, 1-4 blocks, 2k-64k particles in at most a third of the domain)."""
    rng = np.random.Generator(np.random.PCG64(1004 + index))
    W = int(round(math.exp(rng.uniform(math.log(64), math.log(256)))))
    blocks, ppc = int(rng.integers(1, 5)), int(rng.integers(4, 9))
    youngs, nu = float(rng.uniform(1e5, 2e5)), float(rng.uniform(0.15, 0.3))
    n = math.exp(rng.uniform(math.log(2000), math.log(min(64000, 0.3 * W * W * ppc))))
    return W, np.sqrt(np.maximum(rng.dirichlet(np.full(blocks, 4.0)) * n / ppc, 4.0)), ppc, youngs, nu


def _batch_scenes(case, seed):
    out = []
    for i in range(case["scenes"]):
        W, sides, ppc, youngs, nu = _batch_sizes(i)
        rng = np.random.Generator(np.random.PCG64([seed, i]))
        boxes = []
        while len(boxes) < len(sides):
            boxes = []
            for s in sorted(sides, reverse=True):
                for _ in range(100):
                    lo = rng.uniform(MARGIN + 2, W - (MARGIN + 2) - s, 2)
                    if all(np.any(lo + s <= b) or np.any(lo >= b + t) for b, t in boxes):
                        boxes.append((lo, s))
                        break
                else:
                    break
        pos = np.concatenate([lo + s * rng.random((int(round(s * s * ppc)), 2)) for lo, s in boxes])
        vel = (np.array([0.0, -1.0]) + rng.uniform(-0.1, 0.1, pos.shape)) * W
        rho = MATERIAL["rho_phys"] / W / W * 100.0
        volume = np.full(pos.shape[0], 1.0 / ppc, np.float32)
        out.append(scenes.Scene(
            name=f"batch_{i}", dim=2, width=W, height=W, depth=0, border_margin=MARGIN, delta_time=1e-4 * 128.0 / W,
            gravity=-9.8 * W, friction=scenes.FRICTION, theta_c=MATERIAL["theta_c"], theta_s=MATERIAL["theta_s"],
            xi=MATERIAL["xi"], nu=nu, youngs=youngs, rho=rho, steps=case["steps"],
            position=np.ascontiguousarray(pos, np.float32), velocity=np.ascontiguousarray(vel, np.float32),
            volume=volume, mass=(volume * np.float32(rho) / np.float32(100.0)).astype(np.float32)))
    return out


def _pairs(case, seed):
    """Return-map pairs as the solver logs them: a trial F a little outside the elastic band, and its projection."""
    rng = np.random.Generator(np.random.PCG64(seed))
    n = case["pairs"]

    def rotations():
        q = rng.standard_normal((n, 4))
        w, x, y, z = (q / np.linalg.norm(q, axis=1)[:, None]).T
        return np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w), 2 * (x * y + z * w),
                         1 - 2 * (x * x + z * z), 2 * (y * z - x * w), 2 * (x * z - y * w), 2 * (y * z + x * w),
                         1 - 2 * (x * x + y * y)], 1).reshape(n, 3, 3)

    v = rotations()
    a = rng.uniform(-0.15, 0.15, (n, 3))  # the polar rotation: small turns about a random axis
    k = np.zeros((n, 3, 3))
    k[:, 0, 1], k[:, 0, 2], k[:, 1, 2] = -a[:, 2], a[:, 1], -a[:, 0]
    k[:, 1, 0], k[:, 2, 0], k[:, 2, 1] = a[:, 2], -a[:, 1], a[:, 0]
    r = np.linalg.solve(np.eye(3) - 0.5 * k, np.eye(3) + 0.5 * k)
    s = rng.uniform(0.965, 1.015, (n, 3))
    s[:, 0] = np.where(rng.random(n) < 0.6, rng.uniform(0.965, 0.975, n), rng.uniform(1.0075, 1.015, n))
    c = np.clip(s, 0.975, 1.0075)
    jp = rng.uniform(0.9, 1.05, n)
    u = r @ v
    out = np.empty((n, 20), np.float32)
    out[:, :9] = (u * s[:, None, :] @ v.transpose(0, 2, 1)).reshape(n, 9)
    out[:, 9] = jp
    out[:, 10:19] = (u * c[:, None, :] @ v.transpose(0, 2, 1)).reshape(n, 9)
    out[:, 19] = jp * (s / c).prod(1)
    return out


def _init_params(seed):
    rng = np.random.Generator(np.random.PCG64(seed + 77))
    p = np.zeros(N_PARAMS, np.float32)
    for name, rows, cols, used_r, used_c, gain in (("W1", 64, 16, 64, 10, 1.0), ("W2", 64, 64, 64, 64, 1.0),
                                                   ("W3", 64, 64, 64, 64, 1.0), ("W4", 16, 64, 10, 64, 0.1)):
        w = np.zeros((rows, cols), np.float32)
        w[:used_r, :used_c] = gain * math.sqrt(3.0 / used_c) * rng.uniform(-1, 1, (used_r, used_c))
        off, size = OFF[name]
        p[off:off + size] = w.ravel()
    return p


LEARNING_RATE, WEIGHT_DECAY = 4e-3, 1e-4


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("solver", "render"):
        s = Solver.from_scene(_scene(case, seed))
        net = None
        if case.get("plasticity") == "learned":  # the weights shipped for collisions
            net = Mlp.load(MIXED_WEIGHTS)
            s.set_plasticity(_lib.PLASTIC_MLP, net, 1e-3)
        return dict(case=case, solver=s, net=net)
    if kind == "batch":
        return dict(case=case, batch=Batch(_batch_scenes(case, seed)))
    if kind == "train":
        pairs = _pairs(case, seed)
        net = Mlp()
        net.set_params(_init_params(seed))
        net.set_normalization(*normalization(pairs))
        net.load_pairs(pairs)
        return dict(case=case, net=net, seed=seed % 65536)
    c = [case["size"] + 5.0] * case["dim"]
    shape = ball(c, case["size"]) if case["shape"] == "ball" else box(c, [case["size"]] * case["dim"])
    return dict(case=case, shape=shape, seed=seed)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "solver":
        s = state["solver"]
        s.Step(case["steps"])
        if case["returns"] == "positions":
            return s.GetParticlePositions()
        st = s.get_state()
        return dict(position=st.position, velocity=st.velocity, affine_b=st.affine_b, elastic_f=st.elastic_f,
                    plastic_det=st.plastic_det)
    if kind == "batch":
        b = state["batch"]
        b.step(case["steps"])
        return np.concatenate([b.positions(k) for k in range(case["scenes"])])
    if kind == "train":
        net = state["net"]
        loss = net.train(case["steps"], case["batch"], LEARNING_RATE, WEIGHT_DECAY, seed=state["seed"])
        return dict(params=net.params(), loss=loss)
    if kind == "render":
        return state["solver"].render(width=case["width"], height=case["height"], point_size=case["point_size"])
    # the scene's particle array has room for the largest number of samples
    pos, owner = sample_shapes(case["dim"], [state["shape"]], case["min_dist"], state["seed"], case["rounds"])
    room = _cells(case)
    position, of = np.zeros((room, case["dim"]), np.float32), np.full(room, -1, np.int32)
    position[: pos.shape[0]], of[: pos.shape[0]] = pos, owner
    return dict(count=pos.shape[0], position=position, owner=of)


def _cells(case):
    """Background cells a sampled shape can touch: it holds no more samples than these."""
    return math.ceil(2 * case["size"] / (case["min_dist"] / math.sqrt(case["dim"])) + 2) ** case["dim"]


# ---------------------------------------------------------------------------------------------------------------------
# Work

def _solver_work(n, nodes, dim, points, steps, whole):
    """Each step reads and writes what the next one needs of a particle (x, F_E, J_p) and the sums and velocities of
    the nodes in use; v and B are written once, and what comes back once. Operations: the stencil's sums, both ways,
    and the deformation, band test and stress."""
    carried, rest = 4 * (dim + dim * dim + 1), 4 * (dim + dim * dim)
    node = 2 * 8 * (1 + dim) + 2 * 4 * dim
    per = points * (4 * (1 + dim) + 4 * (dim + dim * dim)) + (150 if dim == 2 else 450)
    out = 4 * (2 * dim + 2 * dim * dim + 1) if whole else 4 * dim
    return dict(bytes=n * (2.0 * carried * steps + rest + out) + nodes * float(node) * steps, flops=float(n) * per * steps)


def work(case):
    kind = case["kind"]
    if kind == "solver":
        n, dim = _count(case), case["dim"]
        points = (3 if case["stencil"] == "quadratic" else 4) ** dim
        return _solver_work(n, n / max(case["ppc"], 1), dim, points, case["steps"], case["returns"] == "state")
    if kind == "batch":
        sizes = [_batch_sizes(i) for i in range(case["scenes"])]
        n = sum(round(t * t * s[2]) for s in sizes for t in s[1])
        nodes = sum(float((s[1] ** 2).sum()) for s in sizes)
        return _solver_work(n, nodes, 2, 16, case["steps"], False)
    if kind == "train":
        macs = 10 * 64 + 2 * 64 * 64 + 64 * 10
        return dict(bytes=case["steps"] * (case["batch"] * 80.0 + N_PARAMS * 4 * 7),
                    flops=case["steps"] * case["batch"] * 6.0 * macs)
    if kind == "render":
        n, px = _count(case), case["width"] * case["height"]
        return dict(bytes=n * 12.0 + px * 3.0, flops=n * 40.0)
    return dict(bytes=_cells(case) * 16.0, flops=_cells(case) * case["rounds"] * 60.0)


# ---------------------------------------------------------------------------------------------------------------------
# The same in 64 bits, in plain torch

def _eigen(S):
    """Eigenvectors and eigenvalues of symmetric matrices (n, d, d), by cyclic Jacobi rotations."""
    d = S.shape[-1]
    S = S.clone()
    V = torch.eye(d, dtype=S.dtype, device=S.device).expand_as(S).clone()
    for _ in range(1 if d == 2 else 5):
        for p in range(d):
            for q in range(p + 1, d):
                th = 0.5 * torch.atan2(2 * S[:, p, q], S[:, q, q] - S[:, p, p])
                c, s = torch.cos(th)[:, None], torch.sin(th)[:, None]
                for M, rows in ((S, False), (S, True), (V, False)):
                    a, b = (M[:, p, :], M[:, q, :]) if rows else (M[:, :, p], M[:, :, q])
                    na, nb = c * a - s * b, s * a + c * b
                    a.copy_(na)
                    b.copy_(nb)
    return V, torch.diagonal(S, dim1=1, dim2=2)


class _Sim64:
    """The MLS step over one or many scenes side by side: scene constants per particle and per node."""

    def __init__(self, scs, device):
        f64 = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=device)  # noqa: E731
        self.dim = d = scs[0].dim
        self.quad = scs[0].formulation == _lib.FORMULATION_MLS_QUADRATIC
        self.sticky = scs[0].boundary == _lib.BOUNDARY_STICKY
        cat = lambda name: f64(np.concatenate([getattr(s, name) for s in scs]))  # noqa: E731
        self.x, self.v, self.m, self.vol = cat("position"), cat("velocity"), cat("mass"), cat("volume")
        n = self.x.shape[0]
        self.B = torch.zeros((n, d, d), dtype=torch.float64, device=device)
        self.F = torch.eye(d, dtype=torch.float64, device=device).expand(n, d, d).clone()
        self.J = torch.ones(n, dtype=torch.float64, device=device)
        self.R = self.F.clone()
        counts = torch.tensor([s.count for s in scs], device=device)
        dims = np.array([[s.width, s.height, s.depth][:d] for s in scs], np.int64)
        nodes = (dims + 1).prod(1)
        first = np.concatenate([[0], np.cumsum(nodes)])
        self.nodes = int(first[-1])

        def each(get, of):
            v = [float(np.float32(get(s))) for s in scs]
            return v[0] if len(set(v)) == 1 else torch.repeat_interleave(f64(v), of)

        of_nodes = torch.as_tensor(nodes, device=device)
        self.dt, self.dt_n = each(lambda s: s.delta_time, counts), each(lambda s: s.delta_time, of_nodes)
        self.g_n, self.mu, self.margin = each(lambda s: s.gravity, of_nodes), float(np.float32(scs[0].friction)), float(scs[0].border_margin)
        self.tc, self.ts, self.xi = (float(np.float32(a)) for a in (scs[0].theta_c, scs[0].theta_s, scs[0].xi))
        youngs, nu = (lambda s: float(np.float32(s.youngs))), (lambda s: float(np.float32(s.nu)))
        self.mu0 = each(lambda s: youngs(s) / (2 * (1 + nu(s))), counts)
        self.la0 = each(lambda s: youngs(s) * nu(s) / ((1 + nu(s)) * (1 - 2 * nu(s))), counts)
        per = lambda a: torch.repeat_interleave(torch.as_tensor(a, device=device), counts, 0)  # noqa: E731
        one = len(scs) == 1
        stride = np.ones_like(dims)
        for k in range(1, d):
            stride[:, k] = stride[:, k - 1] * (dims[:, k - 1] + 1)
        self.stride = [int(stride[0, k]) if one else per(stride[:, k]) for k in range(d)]
        self.first = 0 if one else per(first[:-1])
        self.ext_n = [float(dims[0, k]) if one else torch.repeat_interleave(f64(dims[:, k]), of_nodes) for k in range(d)]
        self.ext = [float(dims[0, k]) if one else per(dims[:, k]).double() for k in range(d)]
        idx = [np.unravel_index(np.arange(nn), tuple((e + 1)[::-1])) for nn, e in zip(nodes, dims)] if not one else None
        if one:
            ax = [torch.arange(int(e) + 1, dtype=torch.float64, device=device) for e in dims[0]]
            self.loc = [g.reshape(-1) for g in torch.meshgrid(*ax[::-1], indexing="ij")][::-1]
        else:
            self.loc = [f64(np.concatenate([i[d - 1 - k] for i in idx])) for k in range(d)]

    def stencil(self):
        """Per axis: first node and the S weights and offsets x_i - x_p."""
        S = 3 if self.quad else 4
        base, w, off = [], [], []
        for k in range(self.dim):
            x = self.x[:, k]
            b = torch.floor(x - 0.5) if self.quad else torch.floor(x) - 1
            base.append(b.long())
            o = torch.stack([b + j - x for j in range(S)])
            a = o.abs()
            if self.quad:
                w.append(torch.where(a < 0.5, 0.75 - a * a, 0.5 * (1.5 - a).clamp(min=0) ** 2))
            else:
                w.append(torch.where(a < 1, 0.5 * a ** 3 - a * a + 2 / 3, (2 - a).clamp(min=0) ** 3 / 6))
            off.append(o)
        return S, base, w, off

    def neighbours(self, S, base, w, off):
        for j in range(S ** self.dim):
            at = [(j // S ** k) % S for k in range(self.dim)]
            idx, wt, d = self.first, 1.0, []
            for k, o in enumerate(at):
                idx = idx + (base[k] + o) * self.stride[k]
                wt = wt * w[k][o]
                d.append(off[k][o])
            yield idx, wt, torch.stack(d, 1)

    def step(self):
        d, dinv = self.dim, 4.0 if self.quad else 3.0
        dt = self.dt if isinstance(self.dt, float) else self.dt[:, None, None]
        F, J = self.F, self.J
        h = torch.exp(self.xi * (1 - J))
        je = torch.linalg.det(F) if d == 2 else (F[:, 0] * torch.linalg.cross(F[:, 1], F[:, 2])).sum(1)
        sig = (2 * self.mu0 * h)[:, None, None] * ((F - self.R) @ F.mT)
        sig = sig + (self.la0 * h * (je - 1) * je)[:, None, None] * torch.eye(d, dtype=F.dtype, device=F.device)
        A = dinv * (self.m[:, None, None] * self.B - dt * self.vol[:, None, None] * sig)
        S, base, w, off = self.stencil()
        mass = torch.zeros(self.nodes, dtype=F.dtype, device=F.device)
        mom = torch.zeros((self.nodes, d), dtype=F.dtype, device=F.device)
        mv = self.m[:, None] * self.v
        for idx, wt, o in self.neighbours(S, base, w, off):
            mass.index_add_(0, idx, wt * self.m)
            mom.index_add_(0, idx, wt[:, None] * (mv + (A * o[:, None, :]).sum(2)))
        vc, vf = self.grid(mass, mom)
        nv = torch.zeros_like(self.v)
        nB = torch.zeros_like(self.B)
        dx = torch.zeros_like(self.x)
        dt1 = self.dt if isinstance(self.dt, float) else self.dt[:, None]
        for idx, wt, o in self.neighbours(S, base, w, off):
            wv = wt[:, None] * vf[idx]
            nv += wv
            nB += wv[:, :, None] * o[:, None, :]
            dx += wt[:, None] * (o + dt1 * vc[idx])
        self.x, self.v, self.B = self.x + dx, nv, nB
        Fh = F + dt * dinv * (nB @ F)
        V, e = _eigen(Fh.mT @ Fh)
        s = e.clamp(min=1e-12).sqrt()
        c = s.clamp(1 - self.tc, 1 + self.ts)
        self.F = (Fh @ V * (c / s)[:, None, :]) @ V.mT
        self.R = (Fh @ V / s[:, None, :]) @ V.mT
        self.J = J * (s / c).prod(1)

    def grid(self, mass, mom):
        d, m = self.dim, self.margin
        use = mass >= 1e-6
        vel = torch.where(use[:, None], mom / mass.clamp(min=1e-300)[:, None], 0.0)
        vel[:, 1] += torch.where(use, self.g_n * self.dt_n * torch.ones_like(mass), 0.0)
        if self.sticky:
            wall = torch.zeros_like(use)
            for k in range(d):
                wall |= (self.loc[k] < m) | (self.loc[k] > self.ext_n[k] - m)
            vel = torch.where(wall[:, None], 0.0, vel)
            return vel, vel
        planes = [(0, -1), (1, 1), (0, 1), (1, -1)] if d == 2 else [(0, -1), (0, 1), (1, -1), (1, 1), (2, -1), (2, 1)]
        vc, hits = vel.clone(), []
        for a, ns in planes:
            p = m if ns > 0 else self.ext_n[a] - m
            delta = ns * (self.loc[a] + self.dt_n * vc[:, a] - p) - (ns * (self.loc[a] - p)).clamp(max=0.0)
            hit = use & (delta < 0)
            vc[:, a] -= torch.where(hit, delta / self.dt_n * ns, 0.0)
            hits.append(hit)
        vf = vc.clone()
        push = self.mu * (vc - vel).square().sum(1).sqrt()
        for (a, ns), hit in zip(planes, hits):
            vt = vc.clone()
            vt[:, a] = vc[:, a] - vf[:, a]
            tn = vt.square().sum(1).sqrt()
            on = hit & (tn > 1e-7)
            vf -= torch.where(on, torch.minimum(tn, push) / tn.clamp(min=1e-300), 0.0)[:, None] * vt
        return vc, vf


def _hash(x):
    """The 32-bit mixing the training kernel draws its rows with."""
    x = x & 0xFFFFFFFF
    x = x ^ (x >> 16)
    x = (x * 0x7FEB352D) & 0xFFFFFFFF
    x = x ^ (x >> 15)
    x = ((x & 0xFFFF) * 0x846CA68B + (((x >> 16) * 0x846CA68B & 0xFFFF) << 16)) & 0xFFFFFFFF
    return x ^ (x >> 16)


def _train64(case, seed):
    dev = torch.device("cuda")
    raw = _pairs(case, seed)
    mi, si, mo, so = (torch.as_tensor(a.astype(np.float64), device=dev) for a in normalization(raw))
    pairs = torch.as_tensor(raw, device=dev).double()
    eye = torch.eye(3, dtype=torch.float64, device=dev).reshape(9)
    X = (torch.cat([pairs[:, :9] - eye, pairs[:, 9:10].log()], 1) - mi) / si
    T = (torch.cat([pairs[:, 10:19] - pairs[:, :9], pairs[:, 19:20].log() - pairs[:, 9:10].log()], 1) - mo) / so
    w = torch.as_tensor(_init_params(seed).astype(np.float64), device=dev)
    decay, used = torch.zeros_like(w), torch.ones_like(w)
    shapes = dict(W1=(64, 16), W2=(64, 64), W3=(64, 64), W4=(16, 64), b1=(64,), b2=(64,), b3=(64,), b4=(16,))
    part = lambda t, k: t[OFF[k][0]:OFF[k][0] + OFF[k][1]].view(shapes[k])  # noqa: E731
    for k in ("W1", "W2", "W3", "W4"):
        part(decay, k).fill_(1.0)
    part(used, "W1")[:, 10:] = 0
    part(used, "W4")[10:] = 0
    part(used, "b4")[10:] = 0
    m1, m2, losses = torch.zeros_like(w), torch.zeros_like(w), []
    rows = torch.arange(case["batch"], device=dev)
    f32 = lambda a: float(np.float32(a))  # noqa: E731
    for it in range(case["steps"]):
        sd = (seed % 65536 * 2654435761 + it) & 0xFFFFFFFF
        at = ((_hash(sd ^ _hash(rows)) << 20) ^ _hash(rows * 2654435761 + sd)) % case["pairs"]
        w.requires_grad_(True)
        y = X[at]
        for k in ("1", "2", "3"):
            y = torch.nn.functional.gelu(y @ part(w, "W" + k)[:, : y.shape[1]].T + part(w, "b" + k), approximate="tanh")
        y = (y @ part(w, "W4").T + part(w, "b4"))[:, :10]
        loss = (y - T[at]).square().sum() / case["batch"]
        (g,) = torch.autograd.grad(loss, w)
        w = w.detach()
        g = g * used
        losses.append(float(loss.detach()))
        frac = it / (case["steps"] - 1) if case["steps"] > 1 else 0.0
        lr = f32(LEARNING_RATE) * (0.05 + 0.475 * (1 + math.cos(math.pi * frac)))
        b1, b2 = f32(0.9), f32(0.999)
        m1, m2 = b1 * m1 + (1 - b1) * g, b2 * m2 + (1 - b2) * g * g
        w = w - lr * f32(WEIGHT_DECAY) * decay * w
        w = w - lr * (m1 / (1 - b1 ** (it + 1))) / ((m2 / (1 - b2 ** (it + 1))).sqrt() + 1e-8)
    return dict(params=w, loss=np.array(losses))


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _train64(case, seed)
    if kind == "batch":
        scs = _batch_scenes(case, seed)
    elif kind == "solver" and case["plasticity"] == "exact":
        scs = [_scene(case, seed)]
    else:  # pictures are bytes, samples are draws of a hash, and the learned map's network is 16-bit by design
        return None
    sim = _Sim64(scs, torch.device("cuda"))
    for _ in range(case["steps"]):
        sim.step()
    if kind == "batch" or case["returns"] == "positions":
        return sim.x
    return dict(position=sim.x, velocity=sim.v, affine_b=sim.B, elastic_f=sim.F, plastic_det=sim.J)
