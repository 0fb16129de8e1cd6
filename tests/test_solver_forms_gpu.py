"""The forms that the operator, the fine multigrid level, the Krylov recurrence and the learned
network take by size and by what a grid holds, against the oracle restatements.

Bounds.  Operator: a row sums at most some 60 FP64 terms, each within the row's largest value up to
the geometry factors, so 1e-12 of the largest output.  Preconditioner on grids of millions of cells:
some 100 dependent FP64 smoothing steps and coarse sums of 1e4 terms, 1e-11 of the largest value;
with FP32 storage each step rounds at 6e-8, so 1e-4.  Solves: the true residual to the requested
one, and at most one column more than the oracle's restatement."""
import ctypes as C

import numpy as np
import pytest

from oracle import port, unet
from paracfd_b200 import MG_CYCLE_COMPOSITE, MG_CYCLE_REFERENCE, MG_FP32, MG_FP64, BuiltTopology, CompositeSystem, capi
from paracfd_b200.geometry import extruded_wing, naca4_section, rotate_section

pytestmark = pytest.mark.gpu


def grid(levels, h):
    vertices, triangles = extruded_wing(rotate_section(naca4_section(12, 48, 1.0), 4.0), -0.6, 0.6)
    return BuiltTopology(vertices, triangles, (-1.0, -1.0, -1.0), (2.0, 1.0, 1.0), h, levels, 8, wing_refinement_distance=0.4,
                         surface_refinement_distance=0.2, wake_length=0.5, wake_radius=0.3)


WIDTH = {"face_centroid": 3, "nonorthogonal_correction": 3}


def split_connections(built, embedded, gauges, fragments):
    """A copy of the topology with the last `embedded` coarse-fine edges as embedded ones, gauges on
    `gauges` active cells, and `fragments` extra DOFs behind the bricks, each joined to two cells
    without gradient nodes.  The geometry need not be a real cut: the operator is linear in it."""
    t = capi.Topology.from_buffer_copy(built.topology)
    keep, rng = [built], np.random.default_rng(embedded + gauges + fragments)
    S = t.storage_size

    def put(owner, field, array, ctype):
        array = np.ascontiguousarray(array)
        keep.append(array)
        setattr(owner, field, array.ctypes.data_as(C.POINTER(ctype)))

    act = np.flatnonzero(built.active)
    edges, n = t.coarse_fine, t.coarse_fine.count
    joined = rng.choice(act, (2, fragments), replace=False).astype(np.int64)
    pairs = [(joined[0], S + np.arange(fragments)), (joined[1], S + np.arange(fragments))]
    extra = {"coarse_dof": np.concatenate([p[0] for p in pairs]), "fine_dof": np.concatenate([p[1] for p in pairs]),
             "lower_gradient_node": -np.ones(2 * fragments), "upper_gradient_node": -np.ones(2 * fragments),
             "direction": np.ones(2 * fragments), "axis": rng.integers(0, 3, 2 * fragments)}
    for name, ctype in capi.Connections._fields_[1:]:
        scalar, width = ctype._type_, WIDTH.get(name, 1)
        values = np.ctypeslib.as_array(getattr(edges, name), shape=(n * width,))[(n - embedded) * width:] if n else np.zeros(0, scalar)
        more = extra.get(name, rng.uniform(0.01, 0.02, 2 * fragments * width))
        put(t.embedded, name, np.concatenate([values, more.astype(values.dtype)]), scalar)
    t.coarse_fine.count = n - embedded
    t.embedded.count = embedded + 2 * fragments
    for name, width, value in (("active", 1, 1), ("cut_face_mask", 1, 0), ("volume", 1, 1e-4), ("centroid", 3, 0.0)):
        old = np.ctypeslib.as_array(getattr(t, name), shape=(S * width,))
        put(t, name, np.concatenate([old, np.full(fragments * width, value, old.dtype)]), getattr(t, name)._type_)
    if t.freestream_connected:
        old = np.ctypeslib.as_array(t.freestream_connected, shape=(S,))
        put(t, "freestream_connected", np.concatenate([old, np.ones(fragments, np.uint8)]), C.c_uint8)
    aggregate = np.ctypeslib.as_array(t.preconditioner_aggregate, shape=(S,))
    put(t, "preconditioner_aggregate", np.concatenate([aggregate, aggregate[joined[0]]]).astype(np.int32), C.c_int32)
    t.storage_size = S + fragments
    put(t, "gauge_dof", np.sort(rng.choice(act, gauges, replace=False)).astype(np.int32), C.c_int32)
    put(t, "gauge_coefficient", rng.uniform(0.01, 0.1, gauges), C.c_double)
    t.gauge_count = gauges
    t._keep = keep
    active = np.concatenate([built.active, np.ones(fragments, np.uint8)]).astype(bool)
    return t, active


@pytest.mark.parametrize("levels,h,embedded,gauges,fragments", [
    (1, 1 / 16, 0, 0, 0),           # no compact edges: the brick kernel alone
    (1, 1 / 8, 0, 3, 0),            # gauges only
    (3, 1 / 8, 0, 0, 0),            # both sums of a row in one launch
    (2, 1 / 16, 1000, 0, 7),        # embedded edges, DOFs behind the bricks
    (2, 1 / 16, 129, 5, 1),         # with gauges: two launches for the two sums
])
def test_operator_forms(gpu, levels, h, embedded, gauges, fragments):
    import torch
    built = grid(levels, h)
    topology, active = split_connections(built, embedded, gauges, fragments) if embedded or gauges else (
        built.topology, built.active.astype(bool))
    n = topology.storage_size
    p = np.where(active, np.random.default_rng(n).standard_normal(n), 0.0)
    oracle = port.PortSystem(topology)
    lib = capi.load()
    with CompositeSystem(topology) as s:
        for orthogonal in (0, 1):
            want = oracle.apply(p, bool(orthogonal))
            for offset in (0, 1):       # 1: vectors off 16 bytes, the per-brick kernel
                x = torch.zeros(n + offset, dtype=torch.float64, device="cuda:0")
                x[offset:] = torch.from_numpy(p)
                outs = [torch.full((n + offset,), np.nan, dtype=torch.float64, device="cuda:0") for _ in range(2)]
                torch.cuda.synchronize()
                for call, out in zip((lib.pcfd_pressure_apply_device, lib.pcfd_pressure_apply_device_noalloc), outs):
                    for _ in range(2):
                        capi.check(call(s.handle, C.c_void_p(x.data_ptr() + 8 * offset), C.c_void_p(out.data_ptr() + 8 * offset), orthogonal))
                s.synchronize()
                got = [o.cpu().numpy()[offset:][active] for o in outs]
                assert np.array_equal(got[0], got[1])
                assert np.abs(got[0] - want[active]).max() <= 1e-12 * np.abs(want[active]).max(), (orthogonal, offset)
    oracle.close()
    built.close()


@pytest.mark.parametrize("embedded,gauges,fragments", [(0, 0, 0), (129, 5, 1)])
def test_captured_operator(gpu, embedded, gauges, fragments):
    """The allocation-free operator in a CUDA graph on the caller's stream, chained launches included:
    replayed on new values, the bits of a direct call."""
    import torch
    built = grid(3, 1 / 8)
    topology, active = split_connections(built, embedded, gauges, fragments) if gauges else (built.topology, built.active.astype(bool))
    n, lib, stream, handle = topology.storage_size, capi.load(), torch.cuda.Stream(), C.c_void_p()
    capi.check(lib.pcfd_system_create(C.byref(topology), C.byref(capi.Options(stream=stream.cuda_stream)), C.byref(handle)))
    p, out, direct = (torch.zeros(n, dtype=torch.float64, device="cuda:0") for _ in range(3))

    def apply(to):
        capi.check(lib.pcfd_pressure_apply_device_noalloc(handle, C.c_void_p(p.data_ptr()), C.c_void_p(to.data_ptr()), 0))
    torch.cuda.synchronize()
    apply(direct)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        apply(out)
    for seed in (1, 2):
        p.copy_(torch.from_numpy(np.where(active, np.random.default_rng(seed).standard_normal(n), 0.0)))
        torch.cuda.synchronize()
        for _ in range(2):
            graph.replay()
        torch.cuda.synchronize()
        apply(direct)
        torch.cuda.synchronize()
        assert np.abs(direct.cpu().numpy()[active]).max() > 0
        assert torch.equal(out, direct)
    del graph
    lib.pcfd_system_destroy(handle)
    built.close()


@pytest.mark.parametrize("levels,h,embedded,gauges,fragments", [
    (1, 1 / 16, 0, 3, 0),           # gauges on a grid without compact edges
    (2, 1 / 16, 1000, 0, 7),        # DOFs behind the bricks
    (2, 1 / 16, 129, 5, 1),         # all three kinds of deferred row
])
@pytest.mark.parametrize("cycle", [MG_CYCLE_REFERENCE, MG_CYCLE_COMPOSITE])
def test_fine_level_forms(gpu, cycle, levels, h, embedded, gauges, fragments):
    """Deferred rows of embedded edges, gauges and DOFs behind the bricks in every fine-level pass, twice:
    the second application finds the buffers as the first left them."""
    built = grid(levels, h)
    topology, active = split_connections(built, embedded, gauges, fragments)
    n = topology.storage_size
    oracle = port.PortSystem(topology)
    if cycle == MG_CYCLE_COMPOSITE:
        oracle.set_composite(6, 30, 10)
    for precision, bound in ((MG_FP64, 1e-11), (MG_FP32, 1e-4)):
        with CompositeSystem(topology, mg_cycle=cycle, mg_precision=precision) as s:
            for seed in (1, 2):
                r = np.where(active, np.random.default_rng(seed).standard_normal(n), 0.0)
                want = oracle.precondition(r)
                assert np.abs(s.precondition(r) - want)[active].max() <= bound * np.abs(want[active]).max(), (precision, seed)
    oracle.close()
    built.close()


@pytest.mark.parametrize("cycle", [MG_CYCLE_REFERENCE, MG_CYCLE_COMPOSITE])
def test_fine_level_of_a_large_grid(gpu, cycle):
    """More than 4,096 bricks: the two pre-sweeps as two launches, deferred rows of both levels; the
    fields come back by the threaded download (22 MB, a ragged last piece)."""
    built = grid(2, 1 / 40)
    act = built.active.astype(bool)
    assert act.sum() > 4096 * 512
    r = np.where(act, np.random.default_rng(1).standard_normal(built.storage_size), 0.0)
    oracle = port.PortSystem(built.topology)
    if cycle == MG_CYCLE_COMPOSITE:
        oracle.set_composite(6, 30, 10)
    want, applied = oracle.precondition(r), oracle.apply(r)
    oracle.close()
    for precision, bound in ((MG_FP64, 1e-11), (MG_FP32, 1e-4)):
        with CompositeSystem(built.topology, mg_cycle=cycle, mg_precision=precision) as s:
            assert np.abs(s.precondition(r) - want)[act].max() <= bound * np.abs(want[act]).max(), precision
            assert np.abs(s.apply(r) - applied)[act].max() <= 1e-12 * np.abs(applied[act]).max()
    built.close()


@pytest.mark.parametrize("delayed", [0, 1])
@pytest.mark.parametrize("restart,recycle", [(24, 3), (9, 1), (8, -1), (1, 2)])
def test_krylov_column_counts(gpu, delayed, restart, recycle):
    """Every number of columns a pass over the basis can hold, from one to restart + recycled pairs,
    over several cycles and a second solve that starts from recycled pairs.  Delayed: the dot pass of
    grids up to 16,384 bricks (the pass of larger ones below)."""
    built = grid(2, 1 / 16)
    act = built.active.astype(bool)
    oracle = port.PortSystem(built.topology)
    with CompositeSystem(built.topology, mg_cycle=MG_CYCLE_REFERENCE, gmres_restart=restart, gmres_recycle=recycle,
                         gmres_delayed=delayed) as s:
        for seed in (1, 2):
            b = oracle.apply(np.where(act, np.random.default_rng(seed).standard_normal(built.storage_size), 0.0))
            x, got = s.solve(b, 1e-9, 2000)
            residual = np.linalg.norm((b - oracle.apply(x))[act]) / np.linalg.norm(b[act])
            assert got["converged"] and residual <= 1.01e-9, (got, residual)
            if restart == 24 and seed == 1:
                _, want = oracle.solve(b, 1e-9, 2000)
                assert got["iterations"] <= want["iterations"] + 1, (got, want)
    oracle.close()
    built.close()


@pytest.fixture(scope="module")
def large(gpu):
    built = grid(2, 1 / 64)
    act = built.active.astype(bool)
    assert act.sum() > 16384 * 512          # above: the dot pass whose warps share an item's entries
    yield built, act
    built.close()


def test_delayed_columns_of_a_large_grid(large):
    """The dot pass in each of its groupings (up to 2, 4, 8, 16 and 23 vectors before a column) against
    the three-pass form: after as many columns both have the minimiser over the same space.  The
    sums' rounding, 1e-16 of a column, grows at each orthogonalisation by the column's length before
    over after it, some 3 on average: at most 1e-8 of the solution after 24 columns, so 1e-7."""
    built, act = large
    columns, found = (1, 3, 4, 5, 6, 9, 10, 17, 18, 24), []
    for delayed in (0, 1):
        with CompositeSystem(built.topology, mg_cycle=MG_CYCLE_REFERENCE, gmres_recycle=-1, gmres_delayed=delayed) as s:
            b = s.apply(np.where(act, np.random.default_rng(4).standard_normal(built.storage_size), 0.0))
            solves = [s.solve(b, 1e-14, n) for n in columns]
            found.append([x[act] for x, _ in solves])
            assert [got["iterations"] for _, got in solves] == list(columns)
    for n, want, got in zip(columns, *found):
        assert np.abs(got - want).max() <= 1e-7 * np.abs(want).max(), n
    assert len({x.tobytes() for x in found[1]}) == len(columns)       # every column moved the solution


@pytest.mark.parametrize("restart,recycle", [(24, 3), (5, 2)])
def test_delayed_solves_of_a_large_grid(large, restart, recycle):
    """Two solves, the second from recycled pairs, to the true residual (the operator is checked above)
    in the columns of the three-pass form: rounding moves the last column of a cycle at most."""
    built, act = large
    iterations = []
    for delayed in (0, 1):
        with CompositeSystem(built.topology, mg_cycle=MG_CYCLE_REFERENCE, gmres_restart=restart, gmres_recycle=recycle,
                             gmres_delayed=delayed) as s:
            for seed in (4, 5):
                b = s.apply(np.where(act, np.random.default_rng(seed).standard_normal(built.storage_size), 0.0))
                x, got = s.solve(b, 1e-9, 2000)
                residual = np.linalg.norm((b - s.apply(x))[act]) / np.linalg.norm(b[act])
                assert got["converged"] and residual <= 1.01e-9, (got, residual)
                iterations.append(got["iterations"])
    for want, got in zip(iterations[:2], iterations[2:]):
        assert abs(want - got) <= 1 + want // restart, iterations


@pytest.mark.parametrize("n", [2, 5, 149, 301])
def test_network_sample_counts(gpu, n):
    """Forward and gradients where the samples do not fill a tile, a stage or the grid of CTAs."""
    rng = np.random.default_rng(n)
    mask = (rng.random((n, 512)) > 0.08).astype(np.float64)
    xin, _ = unet.prepare(rng.standard_normal((n, 512)), rng.uniform(0.5, 2.0, (n, 512)), mask)
    target = (rng.standard_normal((n, 512)) * 0.2 * mask).astype(np.float32)
    inputs = np.stack([xin[..., 0].reshape(n, 512), xin[..., 1].reshape(n, 512)], axis=-1).astype(np.float32)
    params = unet.flatten(unet.init_params(11)).astype(np.float32)
    tensors = unet.unflatten(params.astype(np.float64))
    want, _ = unet.forward(tensors, xin)
    _, want_grads = unet.loss_and_grads(tensors, xin, target.astype(np.float64), mask)
    built = grid(1, 1 / 8)
    with CompositeSystem(built.topology, mg_cycle=MG_CYCLE_COMPOSITE) as s:
        s.set_learned_parameters(params)
        _, zhat, grads = s.learned_evaluate(inputs, target)
    built.close()
    # BF16 activations and pre-activation gradients on both sides, FP32 against FP64 sums
    assert np.linalg.norm(zhat.ravel() - want.ravel()) <= 1e-2 * np.linalg.norm(want)
    got = unet.unflatten(grads.astype(np.float64))
    for name, _ in unet.param_shapes():
        assert np.linalg.norm(got[name] - want_grads[name]) <= 3e-2 * np.linalg.norm(want_grads[name]), name
