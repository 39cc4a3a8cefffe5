"""The timed work of the scatter step: its whole calls and its stages, over the sizes that a reconstruction meets.

Sizes are those of the package's own workloads (``citrus_gb300/workloads.py``: 32^3 cells with one group, 64^3 cells
with eight, 24 x 24 x 16 with twelve, the mixed-precision configuration with sixteen) and odd ones between them.
``exact`` gives the same results in 64 bits from plain torch; direction sets, libraries and densities are inputs.
"""

import functools
import math

import numpy as np
import torch

from citrus_gb300.batched import batched_view_steps
from citrus_gb300.citrus_step import CitrusState, citrus_view_step
from citrus_gb300.cross_sections import BONE, WATER, spectral_library
from citrus_gb300.geometry import ConeGeometry, Grid
from citrus_gb300.learned import HigherOrderProposal, mse
from citrus_gb300.responses import ideal_counting_response, no_grid
from citrus_gb300.scatter_solver import ScatterSolver, SolverConfig
from citrus_gb300.state_store import StateStore
from citrus_gb300.workloads import bremsstrahlung_spectrum, monoenergetic_library

DEVICE = "cuda"
BOX_CM = 25.6          # longest edge of the volume
EXACT_ELEMENTS = 6e9   # ray segments that exact() walks at most


def _scene(kind, rows, cols, slices, groups, order, polar, azimuthal, panel_rows, panel_channels, curved=True, q=1,
           precision="fp32"):
    return {"kind": kind, "rows": rows, "cols": cols, "slices": slices, "groups": groups, "order": order,
            "polar": polar, "azimuthal": azimuthal, "panel_rows": panel_rows, "panel_channels": panel_channels,
            "curved": curved, "q": q, "precision": precision}


def listed():
    return [
        # one view of a small monoenergetic scan, primary included: many short launches, where latency counts
        dict(_scene("step", 32, 32, 32, 1, 3, 4, 12, 64, 64, curved=False), name="view_step_32"),
        # two views of one warm outer iteration of a circular scan at its ordinary size, swept together
        dict(_scene("batch", 64, 64, 64, 8, 5, 6, 20, 192, 256), views=2, name="outer_iteration_64"),
        # the collapsed-cone image of one view at that size, the signal alone, as every outer iteration projects it
        dict(_scene("image", 64, 64, 64, 8, 5, 6, 20, 192, 256), signal_only=True, name="image_signal_64"),
        # all images (fluences and the signal per group) of an odd volume on a flat panel, two points per cell axis
        dict(_scene("image", 22, 27, 19, 5, 3, 4, 8, 61, 83, curved=False, q=2), signal_only=False,
             name="image_full_odd"),
        # one accumulator sweep of the scattering source at the ordinary size
        dict(_scene("sweep", 64, 64, 64, 8, 5, 6, 20, 192, 256), name="sweep_64"),
        # the same with sixteen groups, P7 and 240 directions, its products on the tensor cores
        dict(_scene("sweep", 64, 64, 48, 16, 7, 10, 24, 192, 256, precision="bf16x3"), name="sweep_p7_bf16x3"),
        # uncollided fluence, sampling correction and sweep source of one view, one point per cell
        dict(_scene("first", 64, 64, 64, 8, 5, 6, 20, 192, 256), name="first_collision_64"),
        # the same on an odd volume with two points per cell axis
        dict(_scene("first", 23, 29, 17, 5, 3, 4, 12, 61, 83, curved=False, q=2), name="first_collision_refined"),
        # the primary of one view on a large panel, four rays per pixel
        dict(_scene("primary", 128, 128, 96, 16, 7, 10, 24, 384, 512), samples=2, name="primary_panel"),
        # one view's accumulator into its float16 slot and back, as a scan whose views do not all stay resident does
        dict(_scene("state", 64, 64, 64, 8, 5, 6, 20, 192, 256), name="state_store_64"),
        # the learned start of one view
        dict(_scene("predict", 48, 48, 32, 12, 5, 6, 28, 192, 256), name="proposal_predict"),
        # forward and backward of one training batch of the learned start
        dict(_scene("train", 24, 24, 16, 12, 5, 6, 28, 192, 256), batch=4, name="proposal_train"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "batch", "image", "image", "sweep", "sweep", "first", "first", "primary", "state",
                       "predict", "train"])
    while True:
        rows, cols, slices = (_log_int(rng, 12, 64) for _ in range(3))
        groups = rng.choice([1, 2, 3, 5, 6, 8, 11, 12, 16])
        order = rng.choice([1, 3, 5, 7])
        polar = rng.choice([n for n in (2, 4, 6, 8, 10) if n >= order + 1])
        azimuthal = rng.choice([n for n in (8, 12, 16, 20, 24) if n >= 2 * order + 1])
        if rows * cols * slices * groups * polar * azimuthal <= 64 ** 3 * 8 * 120:
            break
    case = _scene(kind, rows, cols, slices, groups, order, polar, azimuthal, _log_int(rng, 32, 192),
                  _log_int(rng, 32, 256), rng.random() < 0.6, 1, "fp32")
    if kind == "batch":
        case["views"] = rng.choice([1, 2])
    elif kind == "image":
        case["signal_only"] = rng.random() < 0.7
    elif kind == "sweep":
        case["precision"] = rng.choice(["fp32", "bf16x3"])
    elif kind == "primary":
        case.update({k: _log_int(rng, 24, 128) for k in ("rows", "cols", "slices")}, samples=rng.choice([1, 2]),
                    panel_rows=_log_int(rng, 64, 384), panel_channels=_log_int(rng, 64, 512))
    elif kind in ("predict", "train"):
        step = 8
        case.update({k: step * _log_int(rng, 2, 6 if kind == "predict" else 3) for k in ("rows", "cols", "slices")},
                    groups=rng.choice([8, 12]))
        if kind == "train":
            case["batch"] = rng.choice([1, 2, 4])
    if kind in ("step", "image", "first") and rows * cols * slices <= 20000 and rng.random() < 0.5:
        case["q"] = 2
    return case


# ---- what a program keeps ---------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=8)
def _library(groups, order):
    if groups == 1:
        return monoenergetic_library(60.0, [0.206, 0.315], [0.923, 0.611], 0.85, order)
    edges = np.linspace(140.0, 20.0, groups + 1) if groups > 12 else np.linspace(120.0, 30.0, groups + 1)
    return spectral_library(edges, bremsstrahlung_spectrum(kvp=float(edges[0]), seed=0), [WATER, BONE],
                            legendre_order=order)


def _cell(case):
    return BOX_CM / max(case["rows"], case["cols"], case["slices"])


def _grid(case):
    """The fine grid: the points of the quadrature, whose spacing is the fine voxel."""
    q = case["q"]
    return Grid((case["rows"] * q, case["cols"] * q, case["slices"] * q), _cell(case) / q)


def _geometry(case):
    pitch = 0.16 * 256 / case["panel_channels"]
    return ConeGeometry(100.0, 150.0, case["panel_rows"], case["panel_channels"], pitch, pitch,
                        use_curved_detector=bool(case["curved"]))


@functools.lru_cache(maxsize=3)
def _solver(items):
    case = dict(items)
    cell = _cell(case)
    config = SolverConfig(num_groups=case["groups"], legendre_order=case["order"], num_polar=case["polar"],
                          num_azimuthal=case["azimuthal"], transport_cell_cm=cell,
                          quadrature_point_spacing_cm=cell / case["q"], moment_precision=case["precision"])
    return ScatterSolver(_library(case["groups"], case["order"]), config, _geometry(case),
                         detector=ideal_counting_response(), grid_response=no_grid(), device=DEVICE,
                         primary_samples_per_pixel_axis=case.get("samples"))


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed) & 0x7FFFFFFF)


def _uniform(gen, shape, lo, hi):
    return torch.rand(*shape, generator=gen, device=DEVICE) * (hi - lo) + lo


def _densities(grid, seed):
    """[2, R, C, S] float32 water and bone: a water ellipsoid in air with three bone rods, noise of half a percent."""
    rng = np.random.default_rng(seed)
    dx, dy, dz = grid.deltas
    x, y, z = ((torch.arange(n, device=DEVICE, dtype=torch.float64) - (n - 1) / 2) * d
               for n, d in ((grid.shape[1], dx), (grid.shape[0], dy), (grid.shape[2], dz)))
    x, y, z = x[None, :, None], y[:, None, None], z[None, None, :]
    ex, ey, ez = grid.extent
    a, b, c = (rng.uniform(0.36, 0.46) * e for e in (ex, ey, 1.5 * ez))
    body = (x / a) ** 2 + (y / b) ** 2 + (z / c) ** 2 < 1.0
    rods = torch.zeros_like(body)
    for _ in range(3):
        r, t = rng.uniform(0.2, 0.6), rng.uniform(0, 2 * math.pi)
        rods |= ((x - a * r * math.cos(t)) ** 2 + (y - b * r * math.sin(t)) ** 2 < rng.uniform(0.8, 1.8) ** 2) & body
    noise = _uniform(_generator(seed + 1), (2, *grid.shape), 0.995, 1.005)
    water = torch.where(body & ~rods, 1.0, 0.0012) * ~rods
    return (torch.stack([water.float(), rods.float() * 1.85]) * noise).contiguous()


def _angle(seed):
    return float(np.random.default_rng(seed + 2).uniform(0, 2 * math.pi))


def _accumulator(case, seed):
    """[G, N_sh, 4, R, C, S] collided fluence in the sweep's cell-major storage: a positive scalar flux that falls off
    from the middle of the volume, anisotropic and linear parts of a tenth."""
    shape = (case["rows"], case["cols"], case["slices"])
    G, N = case["groups"], (case["order"] + 1) ** 2
    gen = _generator(seed + 3)
    storage = torch.rand(N, *shape, G, 4, generator=gen, device=DEVICE).sub_(0.5).mul_(0.2)
    storage[0, ..., 0] += 1.0
    for a, n in enumerate(shape):
        t = (torch.arange(n, device=DEVICE) + 0.5) / n * 2 - 1
        storage *= torch.exp(-t * t).view([-1 if b == a + 1 else 1 for b in range(6)])
    return storage.mul_(1e-5).permute(4, 0, 5, 1, 2, 3)


def _uncollided(case, seed):
    """[G, ...] a fluence at the points as the focal spot's rays leave it: inverse square, thinned through the body."""
    grid = _grid(case)
    src = _source(_angle(seed))
    p = _centers(grid)
    d = ((p - src) ** 2).sum(-1).sqrt()
    depth = (15.0 + d - 100.0).clamp_min(0.0)
    mu = torch.linspace(0.15, 0.3, case["groups"], device=DEVICE, dtype=torch.float64)
    noise = _uniform(_generator(seed + 4), (case["groups"], *grid.shape), 0.9, 1.1)
    return (torch.exp(-mu[:, None, None, None] * depth) / (d * d)).float() * noise / case["groups"]


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind}
    if kind in ("predict", "train"):
        G, shape = case["groups"], (case["rows"], case["cols"], case["slices"])
        net = HigherOrderProposal(2, G, seed=seed % 1000, device=DEVICE)
        gen = _generator(seed)
        rho = torch.stack([_densities(Grid(shape, _cell(case)), seed + 10 * b)
                           for b in range(case.get("batch", 1))])
        first = _uniform(gen, (rho.shape[0], G, *shape), 0.5, 1.5) * (rho.sum(1, keepdim=True) + 0.1)
        state["proposal"] = net
        if kind == "predict":
            state.update(rho=rho[0].contiguous(), first=first[0].contiguous())
        else:
            state.update(x=torch.cat([rho, first / first.mean()], 1).contiguous(),
                         target=(0.5 * first).contiguous())
        return state
    if kind == "state":
        acc = _accumulator(case, seed)
        state.update(accumulator=acc, store=StateStore(1, acc.shape, DEVICE, location="gpu"))
        return state
    grid = _grid(case)
    solver = _solver(tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "kind", "views"))))
    fields = solver.material_fields(_densities(grid, seed), grid)
    state.update(solver=solver, fields=fields, angle=_angle(seed))
    if kind == "step":
        state["collided"] = _accumulator(case, seed)
    elif kind == "batch":
        state["angles"] = [state["angle"] + 2 * math.pi * v / 60 for v in range(case["views"])]
        state["collided"] = [_accumulator(case, seed + 100 * v) for v in range(case["views"])]
    elif kind == "sweep":
        state["phi"] = _accumulator(case, seed)
    elif kind == "image":
        state["uncollided"] = _uncollided(case, seed)
        state["moments"] = solver.multiple_collision_source_moments(fields, _accumulator(case, seed))
        state["signal_only"] = case["signal_only"]
    return state


def run(state):
    kind = state["kind"]
    if kind == "predict":
        return state["proposal"].predict(state["rho"], state["first"])
    if kind == "train":
        net = state["proposal"].net
        y = net.forward(state["x"], keep=True)
        loss, grad = mse(y, state["target"])
        net.backward(grad)
        return {"y": y, "loss": loss, "gradients": net.gradients()}
    if kind == "state":
        state["store"].put(0, state["accumulator"])
        return state["store"].get(0)
    solver, fields, angle = state["solver"], state["fields"], state["angle"]
    if kind == "step":
        scatter, primary, new = citrus_view_step(solver, CitrusState(collided_moments=state["collided"]), fields,
                                                 angle)
        return {"scatter": scatter, "primary": primary, "collided": new.collided_moments}
    if kind == "batch":
        states = [CitrusState(collided_moments=c) for c in state["collided"]]
        signals, _, new = batched_view_steps(solver, states, fields, state["angles"], batch=0)
        return {"scatter": signals, "collided": [s.collided_moments for s in new]}
    if kind == "sweep":
        return solver.transport_sweep(fields, solver.scatter_moment_source(fields, state["phi"]))
    if kind == "image":
        return solver.scatter_image(fields, angle, state["uncollided"], state["moments"],
                                    signal_only=state["signal_only"])
    if kind == "primary":
        return solver.primary(fields, angle)
    uncollided = solver.uncollided_fluence(fields, angle)
    ctx = solver.sweep_context(fields.grid_coarse)
    source = solver.first_collision_moment_source(fields, angle, uncollided, ctx)
    return {"uncollided": uncollided, "source": source(ctx.direction_indices(0, ctx.directions_per_octant))}


def work(case):
    """Bytes and operations that the path cannot do without: inputs read once, outputs written once; a multiply-add is
    two operations; a ray step is one multiply-add per material."""
    kind, G, N_sh = case["kind"], case["groups"], (case["order"] + 1) ** 2
    N = case["rows"] * case["cols"] * case["slices"]
    V, D, P = N * case["q"] ** 3, case["polar"] * case["azimuthal"], case["panel_rows"] * case["panel_channels"]
    K = 512                                                    # panel-facing directions of the image's cone set
    span = (case["rows"] + case["cols"] + case["slices"]) / 2  # voxels along a ray
    accumulator = 4.0 * N_sh * N * 4 * G
    transfer = 4.0 * G * G * (case["order"] + 1) * N
    pairs = G * (G + 1) / 2.0
    moments = {"bytes": accumulator * 2 + transfer, "flops": 2.0 * pairs * N_sh * 4 * N}
    products = 4.0 * D * N_sh * 4 * G * N + 40.0 * D * N * G   # expansion and accumulation, and the cell solves
    image = 2.0 * K * (2 * span * N + V * (2 * pairs + N_sh * G) + P * span * case["q"] * G)
    first = 2.0 * V * (2 * span * case["q"] + 2 * G * 16 + D * 2 * pairs)
    if kind in ("predict", "train"):
        B, levels, macs, params = case.get("batch", 1), (32, 64, 128, 256), 0.0, 0.0
        for i, c in enumerate(levels):
            c_in = 2 + G if i == 0 else levels[i - 1]
            up = levels[i + 1] if i + 1 < len(levels) else None
            weights = 27.0 * (c_in * c + c * c + (0 if up is None else (c + up) * c + c * c))
            macs += weights * N / 8 ** i
            params += weights
        passes = 1 if kind == "predict" else 3
        return {"bytes": 4.0 * B * N * (2 + 2 * G) + 2 * params * (1 if passes == 1 else 4), "flops":
                2.0 * B * macs * passes}
    if kind == "state":
        return {"bytes": accumulator / 4 + accumulator + 2 * accumulator / 8, "flops": 0.0}
    if kind == "sweep":
        return {"bytes": moments["bytes"], "flops": moments["flops"] + products}
    if kind == "image":
        images = 1 if case["signal_only"] else 3 * G + 1
        return {"bytes": 4.0 * (V * (2 + G) + N * (2 + G + G * N_sh) + P * images), "flops": image}
    if kind == "first":
        return {"bytes": 4.0 * (2 * N + 2 * V + G * V + 4 * D * N * G), "flops": first}
    if kind == "primary":
        rays = P * case["samples"] ** 2
        return {"bytes": 4.0 * (2 * V + P * (3 * G + 1)), "flops": 2.0 * rays * (2 * span + 2 * 16 * G)}
    views = case.get("views", 1)
    return {"bytes": views * (moments["bytes"] + 4.0 * P), "flops": views * (moments["flops"] + products + image + first)}


# ---- the same results in 64 bits ----------------------------------------------------------------------------------

def _f64(a):
    return torch.as_tensor(np.ascontiguousarray(a) if isinstance(a, np.ndarray) else a, dtype=torch.float64,
                           device=DEVICE)


def _source(angle):
    return _f64([math.sin(angle) * 100.0, math.cos(angle) * 100.0, 0.0])


def _centers(grid):
    dx, dy, dz = grid.deltas
    x, y, z = ((torch.arange(n, device=DEVICE, dtype=torch.float64) - (n - 1) / 2) * d
               for n, d in ((grid.shape[1], dx), (grid.shape[0], dy), (grid.shape[2], dz)))
    return torch.stack(torch.broadcast_tensors(x[None, :, None], y[:, None, None], z[None, None, :]), -1)


def _pixels(case, angle, n=1):
    """[Rd n, Cd n, 3] centres of the (sub-)pixels, and the panel's centre and normal toward the source."""
    geo = _geometry(case)
    u = (torch.arange(case["panel_channels"] * n, device=DEVICE, dtype=torch.float64) + 0.5) / n
    v = (torch.arange(case["panel_rows"] * n, device=DEVICE, dtype=torch.float64) + 0.5) / n
    u = (u - case["panel_channels"] / 2) * geo.delta_det_channel
    v = (v - case["panel_rows"] / 2) * geo.delta_det_row
    c, s = math.cos(angle), math.sin(angle)
    u_hat, v_hat, n_hat, pc = _f64([c, -s, 0]), _f64([0, 0, 1]), _f64([s, c, 0]), _f64([-50.0 * s, -50.0 * c, 0])
    u, v = u[None, :, None], v[:, None, None]
    if not case["curved"]:
        return pc + u * u_hat + v * v_hat, pc, n_hat
    g = u / 150.0
    return (pc + 150.0 * torch.sin(g) * u_hat + 300.0 * torch.sin(g / 2) ** 2 * n_hat + v * torch.cos(g) * v_hat, pc,
            n_hat)


def _panel_distance(case, angle, p, w):
    """Distance from points p along w to the panel."""
    if not case["curved"]:
        _, pc, n_hat = _pixels(dict(case, panel_rows=1, panel_channels=1), angle)
        return ((pc - p) @ n_hat) / (w @ n_hat)
    d = (p - _source(angle))[..., :2]
    a, b = (w[..., :2] ** 2).sum(-1), (d * w[..., :2]).sum(-1)
    disc = b * b - a * ((d * d).sum(-1) - 150.0 ** 2)
    return torch.where(disc >= 0, (-b + disc.clamp_min(0).sqrt()) / a, torch.full_like(disc, math.inf))


def _integrals(volume, starts, ends, grid):
    """[C, R] line integrals of volume [C, rows, cols, slices]: every plane crossing of a ray, sorted."""
    flat = volume.reshape(volume.shape[0], -1)
    lo = _f64([-e / 2 for e in grid.extent])
    delta, n = _f64(grid.deltas), (grid.shape[1], grid.shape[0], grid.shape[2])
    stride = (grid.shape[2], grid.shape[1] * grid.shape[2], 1)
    hi = lo + delta * _f64(n)
    out = []
    for p0, p1 in zip(starts.split(1 << 18), ends.split(1 << 18)):
        d = p1 - p0
        nz = d != 0
        inv = 1.0 / torch.where(nz, d, torch.ones_like(d))
        t1, t2 = (lo - p0) * inv, (hi - p0) * inv
        inside = (p0 >= lo) & (p0 <= hi)
        big = torch.full_like(d, math.inf)
        a_lo = torch.where(nz, torch.minimum(t1, t2), torch.where(inside, -big, big)).amax(-1).clamp_min(0)
        a_hi = torch.where(nz, torch.maximum(t1, t2), torch.where(inside, big, -big)).amin(-1).clamp_max(1)
        hit = a_hi > a_lo
        a_lo, a_hi = a_lo.where(hit, torch.zeros_like(a_lo))[:, None], a_hi.where(hit, torch.zeros_like(a_hi))[:, None]
        cuts = [a_lo, a_hi]
        for a in range(3):
            t = (lo[a] + delta[a] * torch.arange(1, n[a], device=DEVICE) - p0[:, a:a + 1]) * inv[:, a:a + 1]
            cuts.append(torch.minimum(torch.maximum(t.where(nz[:, a:a + 1], a_lo), a_lo), a_hi))
        cuts = torch.cat(cuts, 1).sort(1)[0]
        seg, mid = cuts[:, 1:] - cuts[:, :-1], 0.5 * (cuts[:, 1:] + cuts[:, :-1])
        index = torch.zeros(mid.shape, dtype=torch.int64, device=DEVICE)
        for a in range(3):
            i = torch.floor((p0[:, a:a + 1] + mid * d[:, a:a + 1] - lo[a]) / delta[a]).clamp(0, n[a] - 1)
            index += i.long() * stride[a]
        seg = seg * d.norm(dim=-1, keepdim=True)
        out.append(torch.stack([(f[index] * seg).sum(1) for f in flat]))
    return torch.cat(out, 1)


def _harmonics(L, omega):
    """[K, (L+1)^2] real orthonormal spherical harmonics, polar axis z, no Condon-Shortley phase."""
    x, y, z = omega.unbind(-1)
    legendre = {}                               # derivatives of Legendre polynomials: P_l^m / sin^m
    for m in range(L + 1):
        legendre[m, m] = torch.full_like(z, float(np.prod(np.arange(2 * m - 1, 0, -2.0)) if m else 1.0))
        for l in range(m + 1, L + 1):
            lower = legendre[l - 2, m] if l - 2 >= m else torch.zeros_like(z)
            legendre[l, m] = ((2 * l - 1) * z * legendre[l - 1, m] - (l + m - 1) * lower) / (l - m)
    power = (x + 1j * y)[:, None] ** torch.arange(L + 1, device=DEVICE)
    cols = []
    for l in range(L + 1):
        for k in range(-l, l + 1):
            m = abs(k)
            norm = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - m) / math.factorial(l + m)
                             * (1 if m == 0 else 2))
            cols.append(norm * legendre[l, m] * (power[:, m].imag if k < 0 else power[:, m].real))
    return torch.stack(cols, -1)


def _transfer(library, rho, L):
    """[G_in, G_out, L+1, ...] Legendre transfer moments, zero for upscatter as the library has it."""
    return torch.einsum("mabl,m...->abl...", _f64(library.mu_s_l[..., :L + 1]), rho)


def _scatter_moments(case, library, rho, phi):
    """T[g, n] = sum_g' transfer[g', g, l(n)] phi[g', n] of phi [G, N_sh, (4,) R, C, S]."""
    t = _transfer(library, rho, case["order"])
    out = torch.empty_like(phi)
    for l in range(case["order"] + 1):
        s = slice(l * l, (l + 1) ** 2)
        if phi.dim() == 6:
            for c in range(4):
                out[:, s, c] = torch.einsum("ab...,an...->bn...", t[:, :, l], phi[:, s, c])
        else:
            out[:, s] = torch.einsum("ab...,an...->bn...", t[:, :, l], phi[:, s])
    return out


def _coarse(case, rho):
    q, (R, C, S) = case["q"], (case["rows"], case["cols"], case["slices"])
    return rho.view(-1, R, q, C, q, S, q).mean((2, 4, 6))


def _transmission(library, path):
    """[G, ...] sum over a group's fine energies of w exp(-mu . path)."""
    out = torch.zeros(library.num_groups, *path.shape[1:], device=DEVICE, dtype=torch.float64)
    mu = _f64(library.fine_mu_t)
    for e, (w, g) in enumerate(zip(library.fine_weight, library.fine_group)):
        out[int(g)] += float(w) * torch.exp(-torch.einsum("m,m...->...", mu[:, e], path))
    return out


def _exact_uncollided(case, library, rho, angle):
    grid, src = _grid(case), _source(angle)
    p = _centers(grid).reshape(-1, 3)
    path = _integrals(rho, src.expand_as(p), p, grid)
    d = p - src
    t = _panel_distance(case, angle, src.expand_as(p), d)
    _, pc, n_hat = _pixels(case, angle)
    u_hat = _f64([math.cos(angle), -math.sin(angle), 0.0])
    geo, hit = _geometry(case), src + t[:, None] * d
    if case["curved"]:
        depth = -((hit - src) @ n_hat)
        u, v = 150.0 * torch.atan2((hit - src) @ u_hat, depth), 150.0 * hit[:, 2] / depth
    else:
        u, v = (hit - pc) @ u_hat, hit[:, 2]
    lit = ((t > 0) & (u.abs() <= geo.delta_det_channel * case["panel_channels"] / 2)
           & (v.abs() <= geo.delta_det_row * case["panel_rows"] / 2))
    return (_transmission(library, path) * (lit / (d * d).sum(-1))).view(-1, *grid.shape)


def _first_source(library, rho, phi, u, w):
    """[G, ...] first-collision source into direction w of fluence phi whose rays run along u."""
    table = library.mu_s_eta                                            # [M, G_in, G_out, nodes]
    pos = ((u @ w).clamp(-1, 1) + 1) / 2 * (table.shape[-1] - 1)
    i = pos.floor().clamp(0, table.shape[-1] - 2)
    f, i = pos - i, i.long()
    out = torch.zeros_like(phi)
    table = _f64(table)
    for g_in in range(phi.shape[0]):
        for g_out in range(g_in, phi.shape[0]):
            t = table[:, g_in, g_out]
            out[g_out] += ((t[:, i] * (1 - f) + t[:, i + 1] * f) * rho).sum(0) * phi[g_in]
    return out


def _exact_first(case, library, quadrature, rho, phi, angle):
    """A function of a direction's index: [G, 4, cells] corrected first-collision moments (mean and x, y, z slopes)."""
    grid = _grid(case)
    d = _centers(grid) - _source(angle)
    u = d / d.norm(dim=-1, keepdim=True)
    omega, weight = _f64(quadrature.omega), quadrature.weight
    I0, I1, I2 = (torch.zeros_like(phi) for _ in range(3))
    for w, k in zip(omega, weight):
        s, mu = _first_source(library, rho, phi, u, w) * float(k), u @ w
        I0 += s
        I1 += s * mu
        I2 += s * mu * mu
    E0, E1 = torch.einsum("mabl,m...,a...->lb...", _f64(library.mu_s_l[..., :2]), rho, phi)
    c = torch.where(E0 > 0, E1 / E0, torch.zeros_like(E0))
    den = I2 - c * I1
    beta = torch.where((E0 > 0) & (den.abs() > 1e-12 * I0.abs()), (c * I0 - I1) / den, torch.zeros_like(I0)).clamp(-1, 1)
    d0 = I0 + beta * I1
    scale = torch.where(d0 > 0, E0 / d0, torch.ones_like(d0))
    q, (R, C, S) = case["q"], (case["rows"], case["cols"], case["slices"])
    t = (2 * torch.arange(q, device=DEVICE, dtype=torch.float64) + 1) / q - 1
    unit = 1.0 / (t * t).mean() if q > 1 else 0.0

    def moments(k):
        s = _first_source(library, rho, phi, u, omega[k]) * scale * (1 + beta * (u @ omega[k]))
        s = s.view(-1, R, q, C, q, S, q)
        return torch.stack([s.mean((2, 4, 6))] + [(s * t.view([-1 if a == ax else 1 for a in range(7)])).mean((2, 4, 6))
                                                  * unit for ax in (4, 2, 6)], 1)

    return moments


def _exact_sweep(case, library, quadrature, rho_coarse, source):
    """[G, N_sh, 4, R, C, S] moments of the swept angular fluence; ``source(k)`` gives [G, 4, R, C, S] of direction k.
    The linear-discontinuous cell: mean and slopes from the source and the three upstream neighbours."""
    G, shape = case["groups"], (case["rows"], case["cols"], case["slices"])
    N_sh = (case["order"] + 1) ** 2
    cell = _cell(case)
    mu = torch.einsum("mg,mijk->ijkg", _f64(library.mu_t), rho_coarse)
    omega, Y = _f64(quadrature.omega), _harmonics(case["order"], _f64(quadrature.omega))
    phi = torch.zeros(N_sh, *shape, G, 4, device=DEVICE, dtype=torch.float64)
    codes = (quadrature.omega < 0) @ np.array([4, 2, 1])
    axes = (1, 0, 2)                                       # x: columns, y: rows, z: slices
    for code in range(8):
        ks = np.nonzero(codes == code)[0]
        flip = [a for a, bit in zip(axes, (4, 2, 1)) if code & bit]
        m = mu.flip(flip).contiguous().view(-1, G)
        i, j, k = (a.reshape(-1) for a in torch.meshgrid(*(torch.arange(n, device=DEVICE) for n in shape),
                                                         indexing="ij"))
        plane, stride = i + j + k, (shape[2], shape[1] * shape[2], 1)
        order = plane.argsort()
        bounds = np.concatenate([[0], np.cumsum(torch.bincount(plane).cpu().numpy())])
        for part in np.array_split(ks, max(1, -(-len(ks) * m.numel() * 64 // 2 ** 32))):
            psi = torch.stack([source(d).permute(2, 3, 4, 0, 1).flip(flip) for d in part])
            psi = psi.reshape(len(part), -1, G, 4).contiguous()
            c = omega[part].abs() / cell                                           # [d, 3]
            s = [-1.0 if code & bit else 1.0 for bit in (4, 2, 1)]
            for b0, b1 in zip(bounds[:-1], bounds[1:]):
                at = order[b0:b1]
                S, mt = psi[:, at], m[at]
                bar, up = [], []
                for a, (pos, ax) in enumerate(zip((j, i, k), axes)):
                    inner = (pos[at] > 0).double()[None, :, None, None]
                    x = psi[:, (at - stride[a]).clamp_min(0)] * inner
                    up.append(x)
                    bar.append(x[..., 0] + s[a] * x[..., a + 1])
                ca = [c[:, a][:, None, None] for a in range(3)]
                r0 = S[..., 0] + sum(ca[a] * bar[a] for a in range(3))
                r = [S[..., a + 1] - 3 * s[a] * ca[a] * bar[a]
                     + sum(ca[b] * up[b][..., a + 1] for b in range(3) if b != a) for a in range(3)]
                total = ca[0] + ca[1] + ca[2] + mt
                dd = [total + 2 * ca[a] for a in range(3)]
                p0 = ((r0 - sum(s[a] * ca[a] * r[a] / dd[a] for a in range(3)))
                      / (total + 3 * sum(ca[a] ** 2 / dd[a] for a in range(3))))
                psi[:, at] = torch.stack([p0] + [(r[a] + 3 * s[a] * ca[a] * p0) / dd[a] for a in range(3)], -1)
            psi = psi.view(len(part), *shape, G, 4).flip([a + 1 for a in flip])
            weights = Y[part] * _f64(quadrature.weight[part])[:, None]
            phi += (weights.t() @ psi.reshape(len(part), -1)).view(phi.shape)
            del psi
    return phi.permute(4, 0, 5, 1, 2, 3)


def _expansion(case, quadrature, T):
    """``source(k)`` of scattering moments T [G, N_sh, 4, R, C, S]."""
    Y = _harmonics(case["order"], _f64(quadrature.omega))
    return lambda k: torch.einsum("n,gn...->g...", Y[k], T)


def _box_blur(image, width, axis):
    """image [G, Rd, Cd] averaged over a window of ``width`` pixels along an axis, cut at the edges."""
    n = image.shape[axis]
    edge = torch.arange(n, device=DEVICE, dtype=torch.float64)
    half = 0.5 * max(float(width), 1e-3)
    lo, hi = (edge + 0.5 - half).clamp(0, n)[:, None], (edge + 0.5 + half).clamp(0, n)[:, None]
    w = (torch.minimum(hi, edge + 1) - torch.maximum(lo, edge)).clamp_min(0) / (hi - lo)
    return (w @ image.transpose(axis, -2)).transpose(axis, -2) if axis != 2 else image @ w.t()


def _exact_image(case, library, cone, rho, phi, T, angle):
    """fluence, planar fluence and signal per group [G, Rd, Cd] of the collapsed-cone directions."""
    grid, q, G = _grid(case), case["q"], case["groups"]
    coarse = grid.coarsen(q)
    rho_c = _coarse(case, rho)
    mu_c = torch.einsum("mg,m...->g...", _f64(library.mu_t), rho_c)
    pix, pc, n_hat = _pixels(case, angle)
    src, points = _source(angle), _centers(grid)
    d = points - src
    u = d / d.norm(dim=-1, keepdim=True)
    height = (points - pc) @ n_hat
    centers = _centers(coarse).reshape(-1, 3)
    to_axis = (src - pix[0]) * _f64([1, 1, 0])
    normals = to_axis / to_axis.norm(dim=-1, keepdim=True) if case["curved"] else n_hat.expand_as(pix[0])
    diagonal = math.sqrt(sum(e * e for e in grid.extent))
    half = 0.5 * diagonal * (1 + 1e-6) + 1e-6
    t = torch.arange(q, device=DEVICE, dtype=torch.float64) - (q - 1) / 2
    geo = _geometry(case)
    Y = _harmonics(case["order"], _f64(cone.omega))
    out = torch.zeros(3, G, *pix.shape[:2], device=DEVICE, dtype=torch.float64)
    spread = lambda x: x.repeat_interleave(q, -3).repeat_interleave(q, -2).repeat_interleave(q, -1)  # noqa: E731
    for k, w in enumerate(_f64(cone.omega)):
        cos = float(-(w @ n_hat))
        if cos <= 0:
            continue
        far = _panel_distance(case, angle, centers, w).clamp(0, diagonal)
        path = _integrals(rho_c, centers, centers + far[:, None] * w, coarse).view(2, *coarse.shape)
        tau = spread(torch.einsum("mg,m...->g...", _f64(library.mu_t), path))
        dx, dy, dz = grid.deltas
        off = (w[1] * dy * t)[:, None, None] + (w[0] * dx * t)[None, :, None] + (w[2] * dz * t)[None, None, :]
        off = off.repeat(coarse.shape)
        total = _first_source(library, rho, phi, u, w) + spread(torch.einsum("n,gn...->g...", Y[k], T))
        emission = total * torch.exp(-(tau - spread(mu_c) * off).clamp_min(0))
        flat = pix.reshape(-1, 3)
        near = flat - (flat @ w)[:, None] * w
        image = _integrals(emission, near - half * w, near + half * w, grid).view(G, *pix.shape[:2])
        mean = float((emission.sum(0) * height).sum() / emission.sum())
        image = _box_blur(image, mean * cone.cell_width[k, 0] / geo.delta_det_channel, 2)
        image = _box_blur(image, mean * cone.cell_width[k, 1] / geo.delta_det_row, 1)
        local = float(cone.weight[k]) * (-(normals @ w)).clamp(0, 1)
        out[0] += float(cone.weight[k]) * image
        out[1] += local * image
    out[2] = out[1]                              # the ideal counting response: one per photon
    return out


def _exact_primary(case, library, rho, angle):
    n, src, grid = case.get("samples", 1), _source(angle), _grid(case)
    pix = _pixels(case, angle, n)[0]
    flat = pix.reshape(-1, 3)
    T = _transmission(library, _integrals(rho, src.expand_as(flat), flat, grid)).view(-1, *pix.shape[:2])
    T = T.view(T.shape[0], case["panel_rows"], n, case["panel_channels"], n).mean((2, 4))
    pix, _, n_hat = _pixels(case, angle)
    d = pix - src
    d2 = (d * d).sum(-1)
    to_axis = (src - pix) * _f64([1, 1, 0])
    normal = to_axis / to_axis.norm(dim=-1, keepdim=True) if case["curved"] else n_hat
    planar = T / d2 * (-(d * normal).sum(-1) / d2.sqrt())
    return {"fluence": T / d2, "planar_fluence": planar, "signal_per_group": planar, "signal": planar.sum(0)}


def _exact_network(state):
    """Output (with the parameters that require gradients) of the network in 64 bits on its bfloat16 weights."""
    net = state["proposal"].net
    w = {n: v.double().requires_grad_() for n, v in net.bf16_weights().items()}
    b = {n: layer.bias.double().requires_grad_() for n, layer in net.layers.items()}
    conv = lambda n, x: torch.nn.functional.conv3d(x, w[n], b[n], padding=w[n].shape[-1] // 2)  # noqa: E731
    relu, levels = torch.relu, net.levels

    def forward(x):
        skips = []
        for i in range(levels):
            h = x if i == 0 else torch.nn.functional.avg_pool3d(skips[-1], 2)
            skips.append(relu(conv(f"enc{i}b", relu(conv(f"enc{i}a", h)))))
        top = skips[-1]
        for i in reversed(range(levels - 1)):
            up = torch.nn.functional.interpolate(top, scale_factor=2, mode="nearest")
            top = relu(conv(f"dec{i}b", relu(conv(f"dec{i}a", torch.cat([skips[i], up], 1)))))
        return conv("out", top)

    return forward, w, b


def exact(case, seed):
    kind = case["kind"]
    N = case["rows"] * case["cols"] * case["slices"]
    V, P = N * case["q"] ** 3, case["panel_rows"] * case["panel_channels"]
    span = case["rows"] + case["cols"] + case["slices"]
    if kind in ("step", "image") and 512.0 * span * (N + P * case["q"]) * (1 + case["groups"] / 4) > EXACT_ELEMENTS:
        return None
    if kind == "batch":
        return None
    state = prepare(case, seed)
    if kind == "state":
        acc = state["accumulator"].double()
        acc[:, :, 1:] = 0
        return acc
    if kind in ("predict", "train"):
        forward, w, b = _exact_network(state)
        if kind == "predict":
            first = state["first"].double()
            s = first.mean()
            return forward(torch.cat([state["rho"].double(), first / s])[None])[0].detach() * s
        y = forward(state["x"].double())
        loss = ((y - state["target"].double()) ** 2).mean()
        loss.backward()
        gradients = {}
        for n in w:
            gradients[n + ".weight"], gradients[n + ".bias"] = w[n].grad, b[n].grad
        return {"y": y.detach(), "loss": loss.detach(), "gradients": gradients}
    library, angle, solver = _library(case["groups"], case["order"]), state["angle"], state["solver"]
    rho = _densities(_grid(case), seed).double()
    if kind == "primary":
        return _exact_primary(case, library, rho, angle)
    quadrature = solver.sweep_quadrature()
    rho_c = _coarse(case, rho)
    if kind == "sweep":
        T = _scatter_moments(case, library, rho_c, state["phi"].double())
        return _exact_sweep(case, library, quadrature, rho_c, _expansion(case, quadrature, T))
    if kind == "image":
        T = state["moments"].double()
        images = _exact_image(case, library, solver.cone_quadrature(_grid(case), angle), rho,
                              state["uncollided"].double(), T, angle)
        signal = images[2].sum(0)
        return {"signal": signal} if case["signal_only"] else {
            "fluence": images[0], "planar_fluence": images[1], "signal_per_group": images[2], "signal": signal}
    phi_uc = _exact_uncollided(case, library, rho, angle)
    first = _exact_first(case, library, quadrature, rho, phi_uc, angle)
    if kind == "first":
        order = np.argsort((quadrature.omega < 0) @ np.array([4, 2, 1]), kind="stable")
        source = torch.stack([first(int(k)).permute(2, 3, 4, 0, 1).contiguous() for k in order])
        return {"uncollided": phi_uc, "source": source}
    T = _scatter_moments(case, library, rho_c, state["collided"].double())
    scatter = _expansion(case, quadrature, T)
    collided = _exact_sweep(case, library, quadrature, rho_c, lambda k: first(k) + scatter(k))
    T = _scatter_moments(case, library, rho_c, collided[:, :, 0])
    images = _exact_image(case, library, solver.cone_quadrature(_grid(case), angle), rho, phi_uc, T, angle)
    return {"scatter": images[2].sum(0), "primary": _exact_primary(case, library, rho, angle)["signal"],
            "collided": collided}
