"""Device memory that runs out while a call sets itself up: the call reports it, the next one sets up
again, and its results are those of a system that never failed.  The failure is an error code: a
child process preloads a cudaMalloc that answers "out of memory" once (native/failing_malloc.c)."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

OUT_OF_MEMORY = 5                     # PCFD_OUT_OF_MEMORY
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def systems():
    from paracfd_b200 import BuiltTopology, CompositeSystem
    from paracfd_b200.geometry import extruded_wing, naca4_section, rotate_section
    vertices, triangles = extruded_wing(rotate_section(naca4_section(12, 48, 1.0), 4.0), -0.6, 0.6)
    built = BuiltTopology(vertices, triangles, (-1.0, -1.0, -1.0), (2.0, 1.0, 1.0), 0.125, 2, 8, wing_refinement_distance=0.3,
                          surface_refinement_distance=0.1, wake_length=0.5, wake_radius=0.3)
    while True:
        with CompositeSystem(built.topology) as s:
            yield s


def retried(arm, call):
    """call() with the 1st, 2nd, ... allocation failing, until none does: an error, then the result."""
    from paracfd_b200 import capi
    s = systems()
    want = call(next(s))
    for n in range(1, 100):
        system = next(s)
        arm(n)
        try:
            got = call(system)
        except capi.PcfdError as error:
            assert error.status == OUT_OF_MEMORY, error
            arm(0)
            again = call(system)
            assert all(np.array_equal(a, b) for a, b in zip(want, again)), n
        else:
            arm(0)
            assert n > 1 and all(np.array_equal(a, b) for a, b in zip(want, got)), n
            return n - 1
    raise AssertionError("allocations without end")


def mac(s):
    rng = np.random.default_rng(3)
    faces = [rng.uniform(-1.0, 1.0, s.faces).astype(np.float32) for _ in range(3)]
    s.set_faces(*faces)
    s.set_mac_links(*[np.full(s.faces, 0x3F, np.uint8)] * 3)
    s.mac_advect(0.01)
    return s.get_faces()


def network(s):
    """Two sizes, so that the second enlarges what the first left, then the first again."""
    rng = np.random.default_rng(4)
    out = []
    for n in (2, 5, 2):
        inputs = np.stack([rng.standard_normal((n, 512)), np.ones((n, 512))], axis=-1).astype(np.float32)
        out.append(s.learned_evaluate(inputs, rng.standard_normal((n, 512)).astype(np.float32))[1])
    return out


def network_smaller_after_failure(arm):
    """A larger batch that does not fit leaves the smaller one's buffers usable."""
    from paracfd_b200 import capi
    rng = np.random.default_rng(5)
    batch = {n: np.stack([rng.standard_normal((n, 512)), np.ones((n, 512))], axis=-1).astype(np.float32) for n in (2, 5)}
    made, failures = systems(), 0
    s = next(made)
    evaluate = lambda n: s.learned_evaluate(batch[n], np.zeros((n, 512), np.float32))[1]      # noqa: E731
    want = evaluate(2)
    for n in range(1, 100):
        arm(n)
        try:
            evaluate(5)
        except capi.PcfdError as error:
            assert error.status == OUT_OF_MEMORY, error
            failures += 1
            arm(0)
            assert np.array_equal(evaluate(2), want), n
        else:
            arm(0)
            return failures
    raise AssertionError("allocations without end")


@pytest.mark.gpu
@pytest.mark.parametrize("check", ["mac", "network", "network smaller"])
def test_set_up_after_a_failed_allocation(gpu, tmp_path, check):
    library = str(tmp_path / "libfailing_malloc.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", os.path.join(ROOT, "tests", "native", "failing_malloc.c"), "-o", library, "-ldl"],
                   check=True)
    run = subprocess.run([sys.executable, os.path.abspath(__file__), check], capture_output=True, text=True, timeout=200, cwd=ROOT,
                         env=dict(os.environ, LD_PRELOAD=library, PYTHONPATH=ROOT))
    assert run.returncode == 0 and int(run.stdout.split()[-1]) >= 5, run.stdout + run.stderr


if __name__ == "__main__":
    arm = C.CDLL(None).failing_malloc_arm
    checks = {"mac": lambda: retried(arm, mac), "network": lambda: retried(arm, network),
              "network smaller": lambda: network_smaller_after_failure(arm)}
    print(checks[sys.argv[1]]())
