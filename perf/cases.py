"""The work a user of this framework has it do, as cases that can be timed.

Scenes are blocks of fluid in a box (spacing about h/2, h = 0.1), the shapes of
``scenes.py`` and ``bench.py``, in a state as a running scene has it: the
lattice slightly compressed, every coordinate off its lattice place by up to a
fifth of the spacing, a smooth flow of about 1 m/s with some noise.  One pass of
a simulation case uploads that state from page-locked host memory, takes
``steps`` steps and reads positions and velocities back, as a program that owns
the state does every frame (``bench.py`` times its end-to-end figure this way).

``exact`` evaluates the same equations in 64 bits with torch, from the
published equations (Macklin & Mueller 2013 as the package's header states
them, and the reference's kernels for REF_COMPAT).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import __graft_entry__

H = 0.1
SPACING = 0.05
WALL = 0.25 * H


def listed():
    return [
        # The reference's own scenario files hold 27 to 9,261 particles; its
        # dam is 1,000: the smallest real scene, all launches and latency.
        {"name": "paper_1k", "kind": "sim", "mode": "paper", "nx": 10, "ny": 10, "nz": 10, "steps": 8},
        # The framework's small configuration (32,768 particles, 1.6 x 1.6 x 3.2 box).
        {"name": "paper_32k", "kind": "sim", "mode": "paper", "nx": 32, "ny": 32, "nz": 32, "steps": 4},
        # An ordinary interactive scene of ragged size with the wave wall moving.
        {"name": "paper_152k_wave", "kind": "sim", "mode": "paper", "nx": 61, "ny": 47, "nz": 53, "steps": 2,
         "wave": 0.004},
        # The headline configuration: 1,048,576 particles.
        {"name": "paper_1m", "kind": "sim", "mode": "paper", "nx": 128, "ny": 128, "nz": 64, "steps": 2},
        # The large configuration: 4,194,304 particles, two blocks about to collide.
        {"name": "paper_4m", "kind": "sim", "mode": "paper", "nx": 256, "ny": 128, "nz": 128, "steps": 1},
        # A scene in the reference's own equations, small and at the headline size.
        {"name": "ref_32k", "kind": "sim", "mode": "ref", "nx": 32, "ny": 32, "nz": 32, "steps": 2},
        {"name": "ref_1m", "kind": "sim", "mode": "ref", "nx": 128, "ny": 128, "nz": 64, "steps": 1},
        # A set of independent scenes advanced together, every scene read back.
        {"name": "batch_24", "kind": "batch", "scenes": 24, "n_min": 4096, "n_max": 131072, "mix": 7, "steps": 4},
        # Requests of uneven size and length through the server, to the last result.
        {"name": "serve_10", "kind": "serve", "scenes": 10, "n_min": 8192, "n_max": 65536, "mix": 11, "steps_min": 3,
         "steps_max": 9},
        # The neighbour operators on device arrays: the radix sort of cell keys ...
        {"name": "sort_pairs_1m", "kind": "sort", "n": 1000003, "bits": 18},
        # ... and hash, counting sort by cell and cell ranges of the large scene.
        {"name": "cells_4m", "kind": "cells", "nx": 256, "ny": 128, "nz": 128},
        # A frame of a scene drawn to an image in host memory.
        {"name": "render_152k", "kind": "render", "nx": 61, "ny": 47, "nz": 53, "width": 1280, "height": 720},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_dims(rng, lo, hi):
    n = _log_uniform(rng, lo, hi)
    ax, az = rng.uniform(0.5, 2.0), rng.uniform(0.5, 2.0)
    base = (n / (ax * az)) ** (1.0 / 3.0)
    return [max(2, int(round(v))) for v in (base * ax, base, base * az)]


def draw(rng):
    kind = rng.choice(["paper", "paper", "paper", "paper", "ref", "batch", "serve", "sort", "cells", "render"])
    if kind in ("paper", "ref"):
        nx, ny, nz = _draw_dims(rng, 500, 3500000 if kind == "paper" else 700000)
        n = nx * ny * nz
        case = {"kind": "sim", "mode": kind, "nx": nx, "ny": ny, "nz": nz,
                "steps": 1 if n > (1000000 if kind == "paper" else 200000) else rng.randint(1, 4)}
        if kind == "paper" and rng.random() < 0.4:
            case["wave"] = round(rng.uniform(-0.005, 0.005), 4)
        return case
    if kind == "batch":
        return {"kind": "batch", "scenes": rng.randint(3, 16), "n_min": 1000, "n_max": _log_uniform(rng, 8000, 131072),
                "mix": rng.randint(0, 10 ** 6), "steps": rng.randint(2, 4)}
    if kind == "serve":
        return {"kind": "serve", "scenes": rng.randint(3, 14), "n_min": 2000, "n_max": _log_uniform(rng, 8000, 65536),
                "mix": rng.randint(0, 10 ** 6), "steps_min": 2, "steps_max": rng.randint(3, 9)}
    if kind == "sort":
        return {"kind": "sort", "n": _log_uniform(rng, 1000, 8000000), "bits": rng.randint(8, 27)}
    nx, ny, nz = _draw_dims(rng, 1000, 4000000 if kind == "cells" else 1000000)
    if kind == "cells":
        return {"kind": "cells", "nx": nx, "ny": ny, "nz": nz}
    return {"kind": "render", "nx": nx, "ny": ny, "nz": nz, "width": rng.randint(160, 1920), "height": rng.randint(120, 1080)}


# ---------------------------------------------------------------- inputs --
def _scene(dims, ref, seed):
    """Box, cells and state (float32, n x 4 positions and velocities) of one scene."""
    double = dims[0] >= 200 and not ref  # two blocks at opposite x ends
    blocks = [(dims[0] // 2, dims[1], dims[2])] * 2 if double else [tuple(dims)]
    margin = 2.0 * H if ref else WALL
    ext = [(d - 1) * SPACING + 2 * margin for d in blocks[0]]
    # a box as the configurations have it: twice the block along z (x for two
    # blocks), half as high again; the floor and three walls touch the block
    cells = [max(4, int(math.ceil(f * e / H))) for f, e in zip((2.0, 1.0, 1.0) if double else (1.25, 1.5, 2.0), ext)]
    box = [c * H for c in cells]
    g = torch.Generator().manual_seed(int(seed) * 7919 + 17)
    s = 0.985 * SPACING
    parts = []
    for q, (nx, ny, nz) in enumerate(blocks):
        i = torch.arange(nx, dtype=torch.float32).view(nx, 1, 1).expand(nx, ny, nz)
        j = torch.arange(ny, dtype=torch.float32).view(1, ny, 1).expand(nx, ny, nz)
        k = torch.arange(nz, dtype=torch.float32).view(1, 1, nz).expand(nx, ny, nz)
        p = torch.stack([i, j, k], -1).reshape(-1, 3) * s + margin
        if q == 1:
            p[:, 0] += box[0] - 2 * margin - (nx - 1) * s
        parts.append(p)
    p = torch.cat(parts)
    n = p.shape[0]
    phase = 2 * math.pi * torch.rand(3, generator=g)
    v = torch.stack([torch.sin(2.1 * p[:, 1] + phase[0]), 0.7 * torch.sin(1.7 * p[:, 2] + phase[1]) - 0.3,
                     torch.sin(1.9 * p[:, 0] + phase[2])], -1)
    v += 0.1 * (torch.rand(n, 3, generator=g) - 0.5)
    p += (0.4 * SPACING) * (torch.rand(n, 3, generator=g) - 0.5)
    for a in range(3):
        p[:, a].clamp_(margin, box[a] - margin)
    pos = torch.cat([p, torch.zeros(n, 1)], 1).contiguous()
    vel = torch.cat([v, torch.full((n, 1), 1000.0 * SPACING ** 3)], 1).contiguous()
    return box, cells, pos, vel


def _params(pbf, box, cells, ref):
    p = pbf.scenes.base_params(tuple(box), tuple(cells), pbf.MODE_REF_COMPAT if ref else pbf.MODE_PAPER)
    return p


def _mix(case, seed):
    """(dims, steps) of each scene of a batch or of a request stream."""
    rng = np.random.default_rng(case["mix"])
    out = []
    for _ in range(case["scenes"]):
        n = math.exp(rng.uniform(math.log(case["n_min"]), math.log(max(case["n_min"] + 1, case["n_max"]))))
        ax, az = rng.uniform(0.5, 2.0, size=2)
        base = (n / (ax * az)) ** (1.0 / 3.0)
        dims = [max(2, int(round(v))) for v in (base * ax, base, base * az)]
        steps = case["steps"] if "steps" in case else int(rng.integers(case["steps_min"], case["steps_max"] + 1))
        out.append((dims, steps))
    return out


def _keys(case, seed):
    g = torch.Generator().manual_seed(int(seed) + 5)
    top = (1 << case["bits"]) - (1 << max(0, case["bits"] - 3))  # a grid rarely fills its key range
    # cell keys of particles kept nearly sorted from the step before
    base = torch.arange(case["n"], dtype=torch.float64) * (top / case["n"])
    off = torch.randn(case["n"], generator=g, dtype=torch.float64) * max(4.0, top / 64.0)
    return (base + off).clamp_(0, top - 1).to(torch.int32)


def prepare(case, seed):
    pbf = __graft_entry__.load_package()
    kind = case["kind"]
    if kind == "sort":
        keys = _keys(case, seed).cuda()
        n = case["n"]
        size = pbf.op_sort_scratch_bytes(n, case["bits"])
        return {"kind": kind, "pbf": pbf, "n": n, "bits": case["bits"], "keys": keys, "out_keys": torch.empty_like(keys),
                "out_vals": torch.empty_like(keys), "size": size,
                "scratch": torch.empty(max(16, size), dtype=torch.uint8, device="cuda")}
    if kind == "batch":
        mix = _mix(case, seed)
        made = [_scene(dims, False, seed + 31 * i) for i, (dims, _) in enumerate(mix)]
        solver = _params(pbf, (1.6, 1.6, 1.6), (16, 16, 16), False)
        b = pbf.Batch(solver, len(made), sum(m[2].shape[0] for m in made), sum(int(np.prod(m[1])) for m in made))
        ids = [b.add_scene(_params(pbf, m[0], m[1], False), pbf.particles_from_state(m[2].numpy(), m[3].numpy()))
               for m in made]
        return {"kind": kind, "batch": b, "ids": ids, "steps": case["steps"]}
    if kind == "serve":
        mix = _mix(case, seed)
        made = [_scene(dims, False, seed + 31 * i) for i, (dims, _) in enumerate(mix)]
        solver = _params(pbf, (1.6, 1.6, 1.6), (16, 16, 16), False)
        server = pbf.Server(solver, 2 << 30, max_scenes=64)
        todo = [(_params(pbf, m[0], m[1], False), pbf.particles_from_state(m[2].numpy(), m[3].numpy()), steps)
                for m, (_, steps) in zip(made, mix)]
        return {"kind": kind, "server": server, "todo": todo}
    dims = (case["nx"], case["ny"], case["nz"])
    ref = case.get("mode") == "ref"
    box, cells, pos, vel = _scene(dims, ref, seed)
    prm = _params(pbf, box, cells, ref)
    n = pos.shape[0]
    if kind == "cells":
        ncells = int(np.prod(cells))
        size = pbf.op_sort_cells_scratch_bytes(n, ncells)
        i32 = lambda k: torch.empty(k, dtype=torch.int32, device="cuda")  # noqa: E731
        # particle order of a running scene: by the cell of the step before
        was = [torch.clamp(((pos[:, a] - vel[:, a] / 120.0) / H).long(), 0, cells[a] - 1) for a in range(3)]
        order = torch.argsort(was[0] + cells[0] * (was[1] + cells[1] * was[2]), stable=True)
        return {"kind": kind, "pbf": pbf, "prm": prm, "n": n, "ncells": ncells, "pos": pos[order].cuda(), "hash": i32(n),
                "off": i32(ncells + 1), "skeys": i32(n), "perm": i32(n), "ranges": i32(2 * ncells),
                "size": size, "scratch": torch.empty(max(16, size), dtype=torch.uint8, device="cuda")}
    sim = pbf.Simulation(prm, pbf.particles_from_state(pos.numpy(), vel.numpy()))
    sim.init()
    sim.initCells()
    if kind == "render":
        sim.set_state(torch.cat([pos[:, :3], vel[:, :3].norm(dim=1, keepdim=True)], 1).numpy(), vel.numpy())
        return {"kind": kind, "sim": sim, "width": case["width"], "height": case["height"]}
    if "wave" in case:
        sim.setWaveGenerator(case["wave"])
    return {"kind": kind, "sim": sim, "steps": case["steps"], "pos": pos.pin_memory(), "vel": vel.pin_memory(),
            "out_pos": torch.empty_like(pos).pin_memory(), "out_vel": torch.empty_like(vel).pin_memory()}


# ------------------------------------------------------------------ a pass --
def run(state):
    kind = state["kind"]
    if kind == "sim":
        sim = state["sim"]
        sim.set_state_async(state["pos"].data_ptr(), state["vel"].data_ptr())
        sim.step(state["steps"], sync=False)
        sim.dump_data_async(state["out_pos"].data_ptr(), state["out_vel"].data_ptr())
        return state["out_pos"], state["out_vel"]
    if kind == "batch":
        state["batch"].step(state["steps"], sync=False)
        return [state["batch"].dump_scene(i) for i in state["ids"]]
    if kind == "serve":
        server = state["server"]
        ids = [server.submit(p, ps, steps) for p, ps, steps in state["todo"]]
        server.run_until_idle()
        return [server.result(i) for i in ids]
    if kind == "render":
        return state["sim"].render(None, state["width"], state["height"])
    pbf, n = state["pbf"], state["n"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "sort":
        pbf.op_sort_pairs(state["keys"].data_ptr(), None, n, state["bits"], state["out_keys"].data_ptr(),
                          state["out_vals"].data_ptr(), state["scratch"].data_ptr(), state["size"], stream)
        return state["out_keys"], state["out_vals"]
    pbf.op_cell_hash(state["prm"], state["pos"].data_ptr(), n, state["hash"].data_ptr(), stream)
    pbf.op_sort_cells(state["hash"].data_ptr(), n, state["ncells"], state["off"].data_ptr(), state["skeys"].data_ptr(),
                      state["perm"].data_ptr(), state["scratch"].data_ptr(), state["size"], stream)
    pbf.op_find_cells(state["off"].data_ptr(), state["ncells"], state["ranges"].data_ptr(), stream)
    return state["hash"], state["off"], state["skeys"], state["perm"], state["ranges"]


def work(case):
    kind = case["kind"]
    if kind == "sort":  # keys in, keys and values out
        return {"bytes": 12 * case["n"], "flops": 0}
    # About 33 neighbours within h at the rest density; a pair costs about 25
    # operations in each of the passes of a step (4 lambda, 4 delta-p, and in
    # the paper's equations vorticity and XSPH; one XSPH pass in the reference's).
    paper, ref = 33 * 25 * 10, 33 * 25 * 9
    if kind in ("batch", "serve"):
        mix = _mix(case, 0)
        n = [math.prod(d) for d, _ in mix]
        return {"bytes": 64 * sum(n), "flops": paper * sum(k * s for k, (_, s) in zip(n, mix))}
    n = case["nx"] * case["ny"] * case["nz"]
    if kind == "cells":  # positions in; hash, sorted keys, permutation, offsets and ranges out
        ncells = int(np.prod(_scene_cells((case["nx"], case["ny"], case["nz"]))))
        return {"bytes": 28 * n + 12 * ncells, "flops": 6 * n}
    if kind == "render":
        return {"bytes": 16 * n + 3 * case["width"] * case["height"], "flops": 40 * n}
    return {"bytes": 64 * n, "flops": (ref if case["mode"] == "ref" else paper) * n * case["steps"]}


def _scene_cells(dims):
    double = dims[0] >= 200
    ext = [(d - 1) * SPACING + 2 * WALL for d in ((dims[0] // 2,) + tuple(dims[1:]) if double else dims)]
    return [max(4, int(math.ceil(f * e / H))) for f, e in zip((2.0, 1.0, 1.0) if double else (1.25, 1.5, 2.0), ext)]


# ----------------------------------------------------- the same in 64 bits --
DT = float(np.float32(1.0 / 120.0))
GRAVITY = float(np.float32(-9.81))


def _f32(v):
    return float(np.float32(v))


class _Cells:
    """Particles sorted by cell; `dims`, `low` and `length` are per axis."""

    def __init__(self, p, low, length, dims):
        self.low, self.length, self.dims = low, length, dims
        c = [torch.clamp(((p[:, a] - low[a]) / length[a]).trunc().long(), 0, dims[a] - 1) for a in range(3)]
        key = c[0] + dims[0] * (c[1] + dims[1] * c[2])
        self.order = torch.argsort(key, stable=True)
        count = torch.bincount(key, minlength=int(np.prod(dims)))
        self.start = torch.cumsum(count, 0) - count
        self.count = count
        self.most = int(count.max())

    def candidates(self, p):
        """Index tensors (i, j) of every particle i and the particles j of the
        27 cells around i's place `p`, one rank of one cell at a time."""
        c = [((p[:, a] - self.low[a]) / self.length[a]).trunc().long() for a in range(3)]
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    x, y, z = c[0] + dx, c[1] + dy, c[2] + dz
                    inside = ((x >= 0) & (x < self.dims[0]) & (y >= 0) & (y < self.dims[1]) & (z >= 0) &
                              (z < self.dims[2]))
                    cell = torch.where(inside, x + self.dims[0] * (y + self.dims[1] * z), 0)
                    count = torch.where(inside, self.count[cell], 0)
                    start = self.start[cell]
                    for m in range(self.most):
                        i = torch.nonzero(count > m).squeeze(1)
                        if i.numel() == 0:
                            break
                        yield i, self.order[start[i] + m]


def _pairs(cells, p, h2):
    """All ordered pairs (i, j), 0 < |p_i - p_j|^2 < h2."""
    left, right = [], []
    for i, j in cells.candidates(p):
        r2 = (p[i] - p[j]).square().sum(1)
        keep = (r2 > 1e-30) & (r2 < h2)
        left.append(i[keep].int())
        right.append(j[keep].int())
    return torch.cat(left), torch.cat(right)


def _paper_steps(pos, vel, box, cells, steps, wave, chunk=1 << 24):
    dev = "cuda"
    h = float(np.float32(np.float32(box[0]) - np.float32(0)) / np.float32(cells[0]))
    h2, poly6, spiky = h * h, 315.0 / (64.0 * math.pi * h ** 9), 45.0 / (math.pi * h ** 6)
    w_self = 315.0 / (64.0 * math.pi * h ** 3)
    rho0, eps, k = _f32(1.0 / SPACING ** 3), 600.0, _f32(0.1) * h * h
    den = h2 - (_f32(0.2) * h) ** 2
    c_xsph, c_vort = _f32(0.01), _f32(0.0005)
    lo = [_f32(WALL) + (wave if a == 0 else 0.0) for a in range(3)]
    hi = [_f32(_f32(box[a]) - _f32(WALL)) for a in range(3)]
    length = [_f32(_f32(box[a]) / cells[a]) for a in range(3)]
    x, v, mass = pos[:, :3].to(dev).double(), vel[:, :3].to(dev).double(), vel[:, 3:].to(dev).double()
    n = x.shape[0]

    def total(left, value):  # sum of the pairs' values at their first particle
        return torch.zeros((n,) + value.shape[1:], dtype=value.dtype, device=dev).index_add_(0, left, value)

    def over_pairs(i, j, f, widths):
        sums = [torch.zeros((n, w), dtype=torch.float64, device=dev) for w in widths]
        for at in range(0, i.numel(), chunk):
            a, b = i[at:at + chunk].long(), j[at:at + chunk].long()
            r = p[a] - p[b]
            r2 = r.square().sum(1, keepdim=True)
            near = r2 < h2
            rl = r2.sqrt()
            grad = torch.where(near, -spiky * (h - rl).square() / rl, 0.0) * r
            for s, value in zip(sums, f(a, b, r2, near, grad)):
                s.index_add_(0, a, value)
        return sums

    for _ in range(steps):
        v = v.clone()
        v[:, 1] += DT * GRAVITY
        d = DT * v
        p = x + d
        i, j = _pairs(_Cells(p, (0.0, 0.0, 0.0), length, cells), p, h2)
        for it in range(4):
            rho, g, s = over_pairs(i, j, lambda a, b, r2, near, grad: (
                torch.where(near, poly6 * (h2 - r2) ** 3, 0.0), grad, grad.square().sum(1, keepdim=True)), (1, 3, 1))
            rho = rho + w_self
            lam = -(rho / rho0 - 1.0) / ((g.square().sum(1, keepdim=True) + s) / rho0 ** 2 + eps)
            dp, = over_pairs(i, j, lambda a, b, r2, near, grad: (
                (lam[a] + lam[b] - k * ((h2 - r2) / den) ** 12) * grad,), (3,))
            d = d + dp / rho0
            p = x + d
            for a in range(3):
                p[:, a].clamp_(lo[a], hi[a])
            d = p - x
        u = d / DT
        omega, xsph = over_pairs(i, j, lambda a, b, r2, near, grad: (
            torch.linalg.cross(grad / rho[b], u[b] - u[a]),
            torch.where(near, poly6 * (h2 - r2) ** 3, 0.0) / rho[b] * (u[b] - u[a])), (3, 3))
        size = omega.norm(dim=1, keepdim=True)
        eta, = over_pairs(i, j, lambda a, b, r2, near, grad: ((size[b] - size[a]) / rho[b] * grad,), (3,))
        length_eta = eta.norm(dim=1, keepdim=True)
        eta = torch.where(length_eta > 0, eta / length_eta.clamp_min(1e-300), 0.0)
        v = u + DT * c_vort * torch.linalg.cross(eta, omega) + c_xsph * xsph
        x = p
    return torch.cat([x, v.norm(dim=1, keepdim=True)], 1), torch.cat([v, mass], 1)


def _six(v):
    return float(np.float32(float("%#.6g" % v)))


def _ref_steps(pos, vel, box, cells, steps):
    """The reference's equations: no s_corr and no vorticity, density without
    the self term, walls h inside the box; a particle sees what the 27 cells
    around its present place held at the start of the step."""
    dev = "cuda"
    hf = np.float32(box[0]) / np.float32(cells[0])
    h, h2 = _six(hf), _six(float(hf) ** 2)
    poly6 = _six(315.0 / (64.0 * math.pi * float(hf) ** 9))
    spiky = _six(45.0 / (math.pi * float(hf) ** 6))
    dt, rho0 = _six(DT), _six(_f32(1.0 / SPACING ** 3))
    top = [_six(_f32(box[a])) for a in range(3)]
    length = [_six(np.float32(box[a]) / np.float32(cells[a])) for a in range(3)]
    x, v, mass = pos[:, :3].to(dev).double(), vel[:, :3].to(dev).double(), vel[:, 3:].to(dev).double()
    n = x.shape[0]
    for _ in range(steps):
        v = v.clone()
        v[:, 1] += dt * GRAVITY
        p = x + dt * v
        grid = _Cells(p, (0.0, 0.0, 0.0), length, cells)
        for _ in range(4):
            i, j = (t.long() for t in _pairs(grid, p, h2))
            r = p[i] - p[j]
            r2 = r.square().sum(1, keepdim=True)
            rl = r2.sqrt()
            grad = r / rl * spiky * (h - rl).square()
            z = lambda w: torch.zeros((n, w), dtype=torch.float64, device=dev)  # noqa: E731
            rho = z(1).index_add_(0, i, poly6 * (h2 - r2) ** 3)
            size = z(1).index_add_(0, i, grad.norm(dim=1, keepdim=True)) + z(3).index_add_(0, i, grad).norm(
                dim=1, keepdim=True)
            lam = -(rho / rho0 - 1.0) / (size.square() / rho0 ** 2 + 10000.0)
            p = p + z(3).index_add_(0, i, -(lam[i] + lam[j]) * grad) / rho0
            for a in range(3):
                p[:, a].clamp_(h, top[a] - h)
        v = (p - x) / dt
        i, j = (t.long() for t in _pairs(grid, p, h2))
        r2 = (p[i] - p[j]).square().sum(1, keepdim=True)
        v = v + 0.01 * torch.zeros_like(v).index_add_(0, i, (v[j] - v[i]) / rho[j] * poly6 * (h2 - r2) ** 3)
        x = p
    return torch.cat([x, v.norm(dim=1, keepdim=True)], 1), torch.cat([v, mass], 1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "sort":
        keys = _keys(case, seed)
        order = torch.argsort(keys, stable=True)
        return keys[order], order.int()
    if kind in ("batch", "serve"):
        out = []
        for q, (dims, steps) in enumerate(_mix(case, seed)):
            box, cells, pos, vel = _scene(dims, False, seed + 31 * q)
            out.append(_paper_steps(pos, vel, box, cells, steps, 0.0))
        return out
    if kind == "sim":
        dims = (case["nx"], case["ny"], case["nz"])
        ref = case["mode"] == "ref"
        box, cells, pos, vel = _scene(dims, ref, seed)
        if ref:
            return _ref_steps(pos, vel, box, cells, case["steps"])
        return _paper_steps(pos, vel, box, cells, case["steps"], _f32(case.get("wave", 0.0)))
    return None  # whole numbers and bytes
