"""The small multigrid levels as one cluster launch, against the FP64 oracle restatements of both
cycles, at the sizes where the launch's shape changes: one CTA's levels only, levels spread over
the cluster, a ragged last slice, and hierarchies whose finer levels stay outside it."""
import numpy as np
import pytest

from oracle import port
from paracfd_b200 import MG_CYCLE_COMPOSITE, MG_CYCLE_REFERENCE, MG_FP32, MG_FP64, BuiltTopology, CompositeSystem, capi
from paracfd_b200.geometry import extruded_wing, naca4_section, rotate_section

pytestmark = pytest.mark.gpu

# (levels, base cell, span half-width): stage-1 rows 64 per brick
GRIDS = {
    "one_cta": (1, 1 / 8),            # 12 bricks: 768 rows, all on one CTA
    "ragged": (2, 1 / 8),             # rows that do not divide by the CTAs
    "cluster": (1, 1 / 16),           # 96 bricks: 6,144 rows
}
ABOVE = (3, 1 / 12)                   # 45,888 stage-1 rows: above the launch's row limit


def grid(levels, h):
    vertices, triangles = extruded_wing(rotate_section(naca4_section(12, 48, 1.0), 4.0), -0.6, 0.6)
    return BuiltTopology(vertices, triangles, (-1.0, -1.0, -1.0), (2.0, 1.0, 1.0), h, levels, 8, wing_refinement_distance=0.4,
                         surface_refinement_distance=0.2, wake_length=0.5, wake_radius=0.3)


def rel(a, b, act):
    return np.abs(a - b)[act].max() / np.abs(b[act]).max()


@pytest.mark.parametrize("name", sorted(GRIDS))
@pytest.mark.parametrize("sweeps,ratio", [(6, 30), (1, 30), (3, 8)])
def test_cycles_match_the_oracle(gpu, name, sweeps, ratio):
    built = grid(*GRIDS[name])
    act = built.active.astype(bool)
    r = np.where(act, np.random.default_rng(sweeps).standard_normal(built.storage_size), 0.0)
    oracle = port.PortSystem(built.topology)
    want_reference = oracle.precondition(r)
    oracle.set_composite(sweeps, ratio, 10)
    want = oracle.precondition(r)
    oracle.close()
    with CompositeSystem(built.topology, mg_cycle=MG_CYCLE_REFERENCE, mg_precision=MG_FP64) as s:
        assert rel(s.precondition(r), want_reference, act) <= 1e-12
    options = dict(mg_cycle=MG_CYCLE_COMPOSITE, mg_stage_sweeps=sweeps, mg_stage_chebyshev=ratio)
    with CompositeSystem(built.topology, mg_precision=MG_FP64, **options) as s:
        got = s.precondition(r)
        assert rel(got, want, act) <= 1e-12
        assert np.array_equal(got, s.precondition(r))
    # FP32 storage: some 100 smoothing steps, each rounding at 6e-8 of the largest value
    with CompositeSystem(built.topology, mg_precision=MG_FP32, **options) as s:
        assert rel(s.precondition(r), want, act) <= 1e-4
    # FP16 coefficients perturb the coarse operators by 5e-4: the same solve, at most two iterations more
    b = np.where(act, np.random.default_rng(7).standard_normal(built.storage_size), 0.0)
    iterations = []
    for fp16 in (0, 1):
        with CompositeSystem(built.topology, mg_precision=MG_FP32, mg_stage_fp16=fp16, **options) as s:
            x, result = s.solve(b, 1e-8, 600)
        assert result["converged"]
        iterations.append(result["iterations"])
    assert abs(iterations[0] - iterations[1]) <= 2, iterations
    built.close()


@pytest.mark.parametrize("precision", [MG_FP64, MG_FP32])
@pytest.mark.parametrize("cycle", [MG_CYCLE_REFERENCE, MG_CYCLE_COMPOSITE])
def test_solves_with_finer_levels_outside_the_launch(gpu, cycle, precision):
    """The launch under levels that run on their own: every cycle solves to the true residual of the
    oracle's operator, in no more iterations than the oracle's FP64 restatement of it plus one."""
    built = grid(*ABOVE)
    act = built.active.astype(bool)
    oracle = port.PortSystem(built.topology)
    b = oracle.apply(np.where(act, np.random.default_rng(3).standard_normal(built.storage_size), 0.0))
    if cycle == MG_CYCLE_COMPOSITE:
        oracle.set_composite(6, 30, 10)
    _, want = oracle.solve(b, 1e-8, 600)
    with CompositeSystem(built.topology, mg_cycle=cycle, mg_precision=precision) as s:
        x, got = s.solve(b, 1e-8, 600)
    residual = np.linalg.norm((b - oracle.apply(x))[act]) / np.linalg.norm(b[act])
    oracle.close()
    built.close()
    assert got["converged"] and residual <= 1.01e-8, (got, residual)
    assert got["iterations"] <= want["iterations"] + 1, (got, want)


STAGE_SMOOTH = 2                      # PCFD_PROFILE_STAGE_SMOOTH
MG_CYCLE_CORRECTED = 1


@pytest.mark.parametrize("precision,bound", [(MG_FP64, 1e-12), (MG_FP32, 1e-4)])
@pytest.mark.parametrize("cycle", [MG_CYCLE_REFERENCE, MG_CYCLE_CORRECTED, MG_CYCLE_COMPOSITE])
def test_cycles_match_their_separate_launches(gpu, cycle, precision, bound):
    """Every cycle against itself in launches of its own, each level with its own weights (the lattice
    corrections of the corrected cycle count 1.5 times): bounds as for the oracle."""
    built = grid(*GRIDS["ragged"])
    act = built.active.astype(bool)
    r = np.where(act, np.random.default_rng(6).standard_normal(built.storage_size), 0.0)
    with CompositeSystem(built.topology, mg_cycle=cycle, mg_precision=precision) as s:
        start = s.launch_count()
        together = s.precondition(r)
        middle = s.launch_count()
        s.profile_begin(STAGE_SMOOTH, 64)
        apart = s.precondition(r)
        s.profile_end(64)
        assert s.launch_count() - middle > middle - start + 4       # the levels did run apart
    assert rel(together, apart, act) <= bound
    built.close()


@pytest.mark.parametrize("fp16", [0, 1])
def test_coarsest_level_without_inverse_keeps_its_precision(gpu, fp16):
    """Without an outlet the coarsest operator is singular: no inverse, and its couplings stay FP32
    also with FP16 stages (rounded to FP16 they would not add up to the diagonal, here by 2.4e-4 a
    sweep).  The launch against the same cycle in launches of its own, which a profiled first stage
    takes: equal to FP32 rounding, as above.  The cell size is no power of two, so FP16 rounds."""
    built = grid(1, 1 / 12)
    closed = capi.Topology.from_buffer_copy(built.topology)
    closed.pressure_outlet_xmax = 0
    act = built.active.astype(bool)
    r = np.where(act, np.random.default_rng(5).standard_normal(built.storage_size), 0.0)
    with CompositeSystem(closed, mg_cycle=MG_CYCLE_COMPOSITE, mg_precision=MG_FP32, mg_stage_fp16=fp16) as s:
        together = s.precondition(r)
        s.profile_begin(STAGE_SMOOTH, 64)
        apart = s.precondition(r)
        assert len(s.profile_end(64)) > 0
    assert rel(together, apart, act) <= 1e-4
    built.close()
