"""The work that users of this framework have it do, as cases for timing.

What a program does with this library is: build a brick grid around a wing, create a system on it,
and then, on that one system, run simulations (one per inflow), solve pressure systems, apply the
operator, or use the brick-local network.  The grid and the system are what such a program keeps,
so they are made once per grid and solver setting here; the inputs of a pass (the inflow profile
and speed, right-hand sides, vectors, network samples) come from the seed alone.

Kinds of case:
  run        one simulation on a kept system: inflow profile, freestream initialisation with its first
             projection, `steps` time steps with the surface loads after each, and the velocity and
             pressure fields read back -- one point of a sweep over inflows
  mac        the same with the staggered MAC momentum mode; faces and pressure are read back
  solve      one cold pressure solve to 1e-8 with host vectors
  apply      the pressure operator on device vectors (the inner call of a caller's own solver)
  net        the brick-local network as a preconditioner, on every brick of the grid
  gradients  the network's forward and backward pass on a training batch of bricks

Settings of a system:
  tuned      what the benchmark runs: composite multigrid cycle in FP32 with FP16 stage
             coefficients, delayed CGS2, no recycled vectors, extrapolated start, autotuned launches
  default    the library's defaults: the reference's FP64 cycle, CGS2, three recycled vectors
  fp64       the composite cycle with everything in FP64
"""
from __future__ import annotations

import ctypes
import dataclasses
import math

import numpy as np
import torch

from paracfd_b200 import MG_CYCLE_COMPOSITE, MG_FP32, MOMENTUM_CELL, MOMENTUM_MAC, CompositeSystem, capi, learned_parameter_count
from paracfd_b200.workloads import WORKLOADS

SETTINGS = {
    "tuned": dict(mg_precision=MG_FP32, mg_cycle=MG_CYCLE_COMPOSITE, mg_stage_sweeps=4, mg_stage_chebyshev=20,
                  gmres_delayed=1, gmres_recycle=-1, mg_stage_fp16=1),
    "default": dict(),
    "fp64": dict(mg_cycle=MG_CYCLE_COMPOSITE, gmres_delayed=1, gmres_recycle=-1),
}


# ---- cases -------------------------------------------------------------------------------------
def listed():
    slab = dict(workload="naca0012_slab", levels=1, aoa=4.0, surface_band=0.25)
    glider = dict(workload="paraglider16m", aoa=8.0, surface_band=0.25)
    wing = dict(workload="naca4412_wing", levels=3, aoa=6.0, surface_band=0.1)
    return [
        # a quick look at a section: one level, 65 k cells, where every launch shows
        dict(name="run_slab_65k", kind="run", setting="tuned", h=1 / 16, steps=10, **slab),
        # the single-level 128 x 64 x 64 configuration, straight out of the box
        dict(name="run_slab_524k_default", kind="run", setting="default", h=1 / 32, steps=10, **slab),
        # a paraglider on a design-study grid, 1.1 M cells on three levels
        dict(name="run_paraglider_1m", kind="run", setting="tuned", h=0.25, levels=3, steps=10,
             **dict(glider, surface_band=0.5)),
        # one point of the angle sweep: a wing on three levels, 4.2 M cells
        dict(name="run_wing_4m", kind="run", setting="tuned", h=0.05, steps=10, **wing),
        # the headline grid: the paraglider on four levels, 16 M cells
        dict(name="run_paraglider_16m", kind="run", setting="tuned", h=0.125, levels=4, steps=10, **glider),
        # the staggered momentum mode on the design-study grid
        dict(name="run_mac_1m", kind="mac", setting="tuned", h=0.25, levels=3, steps=10, **dict(glider, surface_band=0.5)),
        # one pressure system from a caller's own time step, the library's defaults
        dict(name="solve_paraglider_1m_default", kind="solve", setting="default", h=0.25, levels=3,
             **dict(glider, surface_band=0.5)),
        # the same call with the FP64 composite cycle on a grid of no round size
        dict(name="solve_wing_fp64", kind="solve", setting="fp64", h=0.083, **wing),
        # the operator inside a caller's own solver: the smallest grid, then the large one
        dict(name="apply_slab_65k", kind="apply", setting="default", h=1 / 16, **slab),
        dict(name="apply_paraglider_5m", kind="apply", setting="default", h=0.125, levels=3, **glider),
        # the learned preconditioner: applied to a grid, and one training batch of 64 bricks
        dict(name="net_paraglider_1m", kind="net", setting="tuned", h=0.25, levels=3, **dict(glider, surface_band=0.5)),
        dict(name="gradients_64", kind="gradients", setting="default", h=1 / 16, bricks=64, **slab),
    ]


def draw(rng):
    kind = rng.choice(["run", "run", "run", "mac", "solve", "solve", "apply", "net", "gradients"])
    workload = rng.choice(["naca0012_slab", "naca4412_wing", "paraglider16m"])
    # the grid's base cell over the range each geometry is used with (log-uniform), in 1e-4 m
    lo, hi = {"naca0012_slab": (1 / 64, 1 / 12), "naca4412_wing": (0.05, 0.2), "paraglider16m": (0.125, 0.5)}[workload]
    case = dict(kind=kind, workload=workload, h=round(math.exp(rng.uniform(math.log(lo), math.log(hi))), 4),
                levels=1 if workload == "naca0012_slab" else rng.choice([2, 3, 3, 4] if workload == "paraglider16m" else [2, 3]),
                aoa=8.0 if workload == "paraglider16m" else round(rng.uniform(-4.0, 11.0), 2))
    case["surface_band"] = round(rng.uniform(0.1, 0.4) if workload == "paraglider16m" else rng.uniform(0.03, 0.12), 3)
    if case["levels"] == 4:                 # no larger than the 16 M-cell grid
        case.update(h=round(max(case["h"], 0.16), 4), surface_band=min(case["surface_band"], 0.25))
    case["setting"] = rng.choice(["tuned", "default", "fp64"]) if kind == "solve" else rng.choice(["tuned", "tuned", "default"])
    if kind in ("run", "mac"):
        case["steps"] = rng.randint(3, 12)
        if case["setting"] != "tuned":      # several times the cost of a tuned step: stay below the largest listed case
            case["h"] = round(max(case["h"], 1.6 * lo), 4)
            case["steps"] = min(case["steps"], 4)
            case["levels"] = min(case["levels"], 3)
    if kind == "gradients":
        case.update(h=0.0625, workload="naca0012_slab", levels=1, bricks=round(math.exp(rng.uniform(0.0, math.log(512)))))
    return case


# ---- grids and systems, kept as a program keeps them ---------------------------------------------
_grids: dict = {}
_systems: dict = {}


def _spec(case):
    return dataclasses.replace(WORKLOADS[case["workload"]], base_cell_size=case["h"], max_levels=case["levels"], aoa=case["aoa"],
                               surface_refinement_distance=case["surface_band"])


def _key(case):
    return tuple(case[k] for k in ("workload", "h", "levels", "aoa", "surface_band"))


class Grid:
    """A built grid with numpy views of its topology."""

    def __init__(self, case):
        self.spec = _spec(case)
        self.built = self.spec.build()
        self.topology = self.built.topology
        self.n = self.built.storage_size
        self.cells = self.built.leaf_cells
        self.active = self.built.active.astype(bool)


def _grid(case) -> Grid:
    key = _key(case)
    if key not in _grids:
        if sum(g.n for g in _grids.values()) > 60_000_000:      # a program has a few grids open, not dozens
            _grids.clear()
        _grids[key] = Grid(case)
    return _grids[key]


def _system(case) -> CompositeSystem:
    """The system of a grid and setting; in the MAC mode with its face links, for the network with
    its weights: what is set once and kept with the system."""
    kind = case["kind"]
    key = (_key(case), case["setting"], kind if kind in ("mac", "net", "gradients") else "")
    if key not in _systems:
        if sum(s.storage_size for s in _systems.values()) > 60_000_000:
            _systems.clear()
        grid = _grid(case)
        system = CompositeSystem(grid.topology, momentum_min_volume_fraction=grid.spec.min_volume_fraction,
                                 **SETTINGS[case["setting"]])
        if case["setting"] == "tuned":
            system.set_initial_guess(1)
            system.autotune(10)
        if kind == "mac":       # every face away from the near-surface band: all same-side links open
            system.set_mac_links(*[np.full(system.faces, 0x3F, np.uint8) for _ in range(3)])
        if kind in ("net", "gradients"):
            system.set_learned_parameters(_network())
        _systems[key] = system
    return _systems[key]


def _array(pointer, *shape):
    return np.ctypeslib.as_array(pointer, shape=(int(np.prod(shape)),)).reshape(shape)


def _level_bricks(grid, level):
    """(level view, covered flag per brick)."""
    lev = grid.topology.levels[level]
    return lev, (_array(lev.flags, lev.brick_count) & capi.BRICK_COVERED) != 0


# ---- inputs from the seed --------------------------------------------------------------------------
def _inflow(grid, system, speed, rng):
    """A gusting X-min profile: the freestream with a few smooth modes of at most 2 % each."""
    slots, bs = system.inflow_layout(), system.brick_size
    origins = np.concatenate([_array(l.origin, l.brick_count, 3) for l in grid.topology.levels[:grid.topology.level_count]])
    h = np.concatenate([np.full(l.brick_count, l.h) for l in grid.topology.levels[:grid.topology.level_count]])
    cell = np.arange(bs) + 0.5
    y = (origins[slots, 1][:, None, None] + h[slots][:, None, None] * cell[None, None, :]).repeat(bs, 1)
    z = (origins[slots, 2][:, None, None] + h[slots][:, None, None] * cell[None, :, None]).repeat(bs, 2)
    profile = np.full(y.shape, float(speed))
    for _ in range(3):
        ky, kz, phase = rng.uniform(0.2, 1.5), rng.uniform(0.2, 1.5), rng.uniform(0, 2 * np.pi)
        profile += speed * rng.uniform(0.005, 0.02) * np.sin(ky * y + kz * z + phase)
    return np.ascontiguousarray(profile.reshape(-1), np.float32)


def _pressure_field(grid, rng):
    """A pressure-like field: a handful of smooth modes of the domain and 1 % of cell-scale content."""
    centroid = _array(grid.topology.centroid, grid.n, 3)
    extent = np.array([hi - lo for lo, hi in zip(grid.topology.domain_lo, grid.topology.domain_hi)])
    p = 0.01 * rng.standard_normal(grid.n)
    for _ in range(4):
        k = rng.uniform(0.5, 4.0, 3) * np.pi / extent
        p += rng.uniform(0.3, 1.0) * np.sin(centroid @ k + rng.uniform(0, 2 * np.pi))
    return np.where(grid.active, p, 0.0)


def _network():
    """Network parameters as they are initialised (He-normal), flat."""
    rng = np.random.default_rng(20261203)
    shapes = [(27, co, ci) for _, _, co, sources in LAYERS for ci in sources]
    parts = [rng.standard_normal(s).ravel() * math.sqrt(2.0 / (s[0] * s[2])) for s in shapes]
    parts.append(rng.standard_normal(16) * math.sqrt(2.0 / 16))
    flat = np.concatenate(parts).astype(np.float32)
    assert flat.size == learned_parameter_count()
    return flat


def _bricks(count, rng):
    """Training samples: smooth brick residuals with noise, scaled to unit RMS, 8 % of the cells solid."""
    g = np.linspace(0.0, 1.0, 8)
    z, y, x = np.meshgrid(g, g, g, indexing="ij")
    a, b = rng.uniform(0, 6, (2, count, 1, 1, 1))
    q = np.sin(3 * x + a) * np.cos(2 * y + b) + 0.3 * rng.standard_normal((count, 8, 8, 8))
    mask = rng.random((count, 512)) > 0.08
    q = q.reshape(count, 512) * mask
    q /= np.sqrt((q * q).sum(1, keepdims=True) / np.maximum(mask.sum(1, keepdims=True), 1))
    # the library keeps the network's input in BF16: hand it values that are BF16 already
    q = torch.from_numpy(q).to(torch.bfloat16).to(torch.float32).numpy()
    target = 0.2 * rng.standard_normal((count, 512)) * mask
    return np.stack([q, mask.astype(np.float32)], axis=-1), target.astype(np.float32)


# ---- prepare / run -----------------------------------------------------------------------------------
def prepare(case, seed):
    rng = np.random.default_rng([seed, 20261203])
    grid, system = _grid(case), _system(case)
    state = dict(case=case, system=system)
    kind = case["kind"]
    if kind in ("run", "mac"):
        state["speed"] = grid.spec.speed * rng.uniform(0.95, 1.05)
        state["flow"] = grid.spec.case
        state["inflow"] = _inflow(grid, system, state["speed"], rng)
    elif kind == "solve":
        state["b"] = _operator(grid, _pressure_field(grid, rng))
    elif kind == "apply":
        state["p"] = torch.from_numpy(_pressure_field(grid, rng)).cuda()
        state["out"] = torch.zeros(grid.n, dtype=torch.float64, device="cuda")
    elif kind == "net":
        state["r"] = torch.from_numpy(np.where(grid.active, rng.standard_normal(grid.n), 0.0)).cuda()
        state["z"] = torch.zeros(grid.n, dtype=torch.float64, device="cuda")
    else:
        state["inputs"], state["targets"] = _bricks(case["bricks"], rng)
    torch.cuda.synchronize()
    return state


def run(state):
    case, system = state["case"], state["system"]
    kind = case["kind"]
    if kind in ("run", "mac"):
        system.set_momentum_mode(MOMENTUM_MAC if kind == "mac" else MOMENTUM_CELL)
        system.configure(speed=state["speed"], **state["flow"])
        system.set_inflow(state["inflow"])
        system.initialize()
        forces = []
        for _ in range(case["steps"]):
            system.step()
            # the MAC mode's loads are the pressure's only: its wall model keeps no patch forces
            loads = system.loads(include_viscous=kind == "run")
            forces.append(loads["total_force"])
        fields = system.get_state() if kind == "run" else system.get_faces()
        # forces as the FP32 field values that they are sums of
        return dict(fields=list(fields), pressure=system.get_pressure_shadow(), forces=np.array(forces, np.float32))
    if kind == "solve":
        x, result = system.solve(state["b"], 1e-8, 600)
        return dict(x=x, converged=result["converged"])
    lib = capi.load()
    if kind == "apply":
        capi.check(lib.pcfd_pressure_apply_device(system.handle, ctypes.c_void_p(state["p"].data_ptr()),
                                                  ctypes.c_void_p(state["out"].data_ptr()), 0))
        return state["out"]
    if kind == "net":
        capi.check(lib.pcfd_learned_apply_device(system.handle, ctypes.c_void_p(state["r"].data_ptr()),
                                                 ctypes.c_void_p(state["z"].data_ptr())))
        return state["z"]
    loss, zhat, gradients = system.learned_evaluate(state["inputs"], state["targets"])
    return dict(loss=loss, zhat=zhat, gradients=gradients)


def work(case):
    if case["kind"] == "gradients":
        # 41.6 MFLOP per brick forward, twice that backward; samples in, outputs and gradients out
        return {"bytes": case["bricks"] * 512 * 16 + 2 * 4 * 179728, "flops": 3 * 41.6e6 * case["bricks"]}
    grid = _grid(case)
    t, cells = grid.topology, grid.cells
    if case["kind"] in ("run", "mac"):
        # per step the velocity (3 FP32) and the pressure (FP64) read and written once
        return {"bytes": float(cells) * 40 * (case["steps"] + 1), "flops": 0.0}
    edges = t.coarse_fine.count + t.embedded.count + t.regular.count
    weights = int(t.gradient_offset[t.gradient_node_count]) if t.gradient_node_count else 0
    # vector in, vector out, one byte of face openings per cell, the compact edges and the gradient stencil
    operator = 17.0 * cells + 60.0 * edges + 28.0 * weights
    if case["kind"] == "net":
        bricks = sum(int((~_level_bricks(grid, l)[1]).sum()) for l in range(t.level_count))
        return {"bytes": 17.0 * cells, "flops": 41.6e6 * bricks}
    return {"bytes": operator, "flops": 14.0 * cells + 20.0 * edges + 7.0 * weights}


# ---- 64-bit values in plain numpy / torch ---------------------------------------------------------------
def _structured(grid, p):
    """The 7-point part: (operator on p, its diagonal), covered bricks and inactive cells zero."""
    t = grid.topology
    out, diagonal = np.zeros(grid.n), np.zeros(grid.n)
    cut_all = _array(t.cut_face_mask, grid.n)
    for level in range(t.level_count):
        lev, covered = _level_bricks(grid, level)
        first, count = lev.level_offset, lev.brick_count
        span = slice(first, first + count * 512)
        shape = (count, 8, 8, 8)                      # brick, z, y, x
        P = p[span].reshape(shape)
        A = grid.active[span].reshape(shape) & ~covered[:, None, None, None]
        C = cut_all[span].reshape(shape)
        O, D = out[span].reshape(shape), diagonal[span].reshape(shape)
        neighbours = _array(lev.neighbors, count, 6)
        for axis in range(3):
            def at(s, axis=axis):
                index = [slice(None)] * 4
                index[3 - axis] = s
                return tuple(index)
            lo, hi = at(slice(0, 7)), at(slice(1, 8))
            open_ = A[lo] & A[hi] & ((C[lo] >> axis) & 1 == 0)
            flux = np.where(open_, lev.h * (P[lo] - P[hi]), 0.0)
            O[lo] += flux
            O[hi] -= flux
            D[lo] += lev.h * open_
            D[hi] += lev.h * open_
            a = np.nonzero((neighbours[:, 2 * axis + 1] >= 0) & ~covered)[0]
            b = neighbours[a, 2 * axis + 1]
            keep = ~covered[b]
            a, b = a[keep], b[keep]
            last, front = at(7)[1:], at(0)[1:]
            open_ = A[a][(slice(None),) + last] & A[b][(slice(None),) + front] & ((C[a][(slice(None),) + last] >> axis) & 1 == 0)
            flux = np.where(open_, lev.h * (P[a][(slice(None),) + last] - P[b][(slice(None),) + front]), 0.0)
            O[(a,) + last] += flux
            O[(b,) + front] -= flux
            D[(a,) + last] += lev.h * open_
            D[(b,) + front] += lev.h * open_
        if t.pressure_outlet_xmax:
            outlet = np.nonzero(((_array(lev.flags, count) & capi.BRICK_XMAX) != 0) & ~covered)[0]
            O[outlet, :, :, 7] += np.where(A[outlet, :, :, 7], 2.0 * lev.h * P[outlet, :, :, 7], 0.0)
            D[outlet, :, :, 7] += 2.0 * lev.h * A[outlet, :, :, 7]
    return out, diagonal


def _edges(grid):
    """The compact edges as arrays: lower, upper, two-point coefficient, area, gradient nodes, correction, weight."""
    t = grid.topology
    parts = []
    for c in (t.coarse_fine, t.embedded):
        if not c.count:
            continue
        coarse, fine, forward = _array(c.coarse_dof, c.count), _array(c.fine_dof, c.count), _array(c.direction, c.count) > 0
        area, factor, normal = (_array(x, c.count) for x in (c.open_area, c.orthogonal_gradient_factor, c.normal_distance))
        factor = np.where(factor > 0, factor, np.where(normal > 0, 1.0 / np.where(normal > 0, normal, 1.0), 0.0))
        parts.append((np.where(forward, coarse, fine), np.where(forward, fine, coarse), area * factor, area, c))
    c = t.regular
    if c.count:
        area = _array(c.open_area, c.count)
        parts.append((_array(c.lower_dof, c.count), _array(c.upper_dof, c.count), area * _array(c.two_point_delta, c.count), area, c))
    for lower, upper, coefficient, area, c in parts:
        keep = (lower >= 0) & (upper >= 0) & (lower != upper)
        keep &= grid.active[np.where(keep, lower, 0)] & grid.active[np.where(keep, upper, 0)]
        yield (lower[keep], upper[keep], coefficient[keep], area[keep], _array(c.lower_gradient_node, c.count)[keep],
               _array(c.upper_gradient_node, c.count)[keep], _array(c.nonorthogonal_correction, c.count, 3)[keep],
               _array(c.upper_gradient_weight, c.count)[keep])


def _operator(grid, p):
    """A p: the 7-point part, the compact two-point edges, the gauges and the WLS correction."""
    t = grid.topology
    out, _ = _structured(grid, p)
    gradient = None
    if t.gradient_node_count:
        nodes = t.gradient_node_count
        offset = _array(t.gradient_offset, nodes + 1)
        nnz = int(offset[-1])
        node = np.repeat(np.arange(nodes), np.diff(offset))
        d = p[_array(t.gradient_neighbour, nnz)] - p[_array(t.gradient_dof, nodes)][node]
        w = _array(t.gradient_weight, nnz, 3)
        gradient = np.stack([np.bincount(node, w[:, a] * d, nodes) for a in range(3)], 1)
    for lower, upper, coefficient, area, ln, un, correction, weight in _edges(grid):
        flux = coefficient * (p[lower] - p[upper])
        if gradient is not None:
            has = (ln >= 0) & (un >= 0)
            mean = (1.0 - weight)[:, None] * gradient[np.where(has, ln, 0)] + weight[:, None] * gradient[np.where(has, un, 0)]
            flux = flux - np.where(has, area * (correction * mean).sum(1), 0.0)
        out += np.bincount(lower, flux, grid.n) - np.bincount(upper, flux, grid.n)
    if t.gauge_count:
        dof = _array(t.gauge_dof, t.gauge_count)
        out += np.bincount(dof, _array(t.gauge_coefficient, t.gauge_count) * p[dof], grid.n)
    return np.where(grid.active, out, 0.0)


def _diagonal(grid):
    _, diagonal = _structured(grid, np.zeros(grid.n))
    for lower, upper, coefficient, *_ in _edges(grid):
        diagonal += np.bincount(lower, coefficient, grid.n) + np.bincount(upper, coefficient, grid.n)
    if grid.topology.gauge_count:
        dof = _array(grid.topology.gauge_dof, grid.topology.gauge_count)
        diagonal += np.bincount(dof, _array(grid.topology.gauge_coefficient, grid.topology.gauge_count), grid.n)
    return diagonal


# the network's layers: name, cells per side, output channels, input channels per source
LAYERS = (("enc0", 8, 16, (16,)), ("enc1", 4, 32, (16,)), ("bott", 2, 64, (32,)), ("dec1", 4, 32, (64, 32)), ("dec0", 8, 16, (32, 16)))


def _net(flat, x):
    """The network in FP64 on x [bricks, 2, 8, 8, 8]; flat: FP64 parameters; returns [bricks, 512]."""
    weights, o = {}, 0
    for name, _, co, sources in LAYERS:
        parts = []
        for ci in sources:
            parts.append(flat[o:o + 27 * co * ci].reshape(3, 3, 3, co, ci).permute(3, 4, 0, 1, 2))
            o += 27 * co * ci
        weights[name] = torch.cat(parts, 1)
    f = torch.nn.functional
    x = f.pad(x, (0, 0, 0, 0, 0, 0, 0, 14))
    e0 = f.relu(f.conv3d(x, weights["enc0"], padding=1))
    e1 = f.relu(f.conv3d(f.avg_pool3d(e0, 2), weights["enc1"], padding=1))
    b = f.relu(f.conv3d(f.avg_pool3d(e1, 2), weights["bott"], padding=1))
    up = lambda v: f.interpolate(v, scale_factor=2, mode="nearest")      # noqa: E731
    d1 = f.relu(f.conv3d(torch.cat([up(b), e1], 1), weights["dec1"], padding=1))
    d0 = f.relu(f.conv3d(torch.cat([up(d1), e0], 1), weights["dec0"], padding=1))
    return torch.einsum("bczyx,c->bzyx", d0, flat[o:o + 16]).reshape(x.shape[0], 512)


def exact(case, seed):
    """FP64 values without this library's kernels: the operator, solutions, the network.  A whole
    time step has no plain restatement that is quick enough here."""
    kind = case["kind"]
    if kind in ("run", "mac"):
        return None
    rng = np.random.default_rng([seed, 20261203])
    if kind == "gradients":
        flat = torch.from_numpy(_network()).double().requires_grad_()
        inputs, targets = (torch.from_numpy(v).double() for v in _bricks(case["bricks"], rng))
        mask = inputs[..., 1]
        zhat = _net(flat, inputs.permute(0, 2, 1).reshape(-1, 2, 8, 8, 8))
        loss = (((zhat - targets) * mask) ** 2).sum() / mask.sum()
        loss.backward()
        return dict(loss=float(loss), zhat=zhat.detach(), gradients=flat.grad)
    grid = _grid(case)
    if kind == "solve":
        return dict(x=_pressure_field(grid, rng), converged=True)
    if kind == "apply":
        return _operator(grid, _pressure_field(grid, rng))
    flat = torch.from_numpy(_network()).double().cuda()
    r = np.where(grid.active, rng.standard_normal(grid.n), 0.0)
    diagonal = _diagonal(grid)
    q = np.where(grid.active & (diagonal > 0), r / np.where(diagonal > 0, diagonal, 1.0), 0.0)
    z = np.zeros(grid.n)
    for level in range(grid.topology.level_count):
        lev, covered = _level_bricks(grid, level)
        rows = lev.level_offset + np.nonzero(~covered)[0][:, None] * 512 + np.arange(512)[None, :]
        for part in np.array_split(rows, max(1, len(rows) // 256)):
            m = torch.from_numpy(grid.active[part].astype(np.float64)).cuda()
            v = torch.from_numpy(q[part]).cuda()
            scale = ((v * v).sum(1, keepdim=True) / m.sum(1, keepdim=True).clamp(min=1.0)).sqrt()
            scale = torch.where(scale > 0, scale, torch.ones_like(scale))
            x = torch.stack([v / scale, m], 1).reshape(-1, 2, 8, 8, 8)
            z[part] = (scale * _net(flat, x) * m).cpu().numpy()
    return z
