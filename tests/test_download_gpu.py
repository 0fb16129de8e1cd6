"""Large read-backs on the streams and threads that a program may use: the same bytes."""
import ctypes as C
import threading

import numpy as np
import pytest

from paracfd_b200 import BuiltTopology, CompositeSystem, capi
from paracfd_b200.geometry import extruded_wing, naca4_section, rotate_section

pytestmark = pytest.mark.gpu

PER_THREAD = 2                          # cudaStreamPerThread


def on_stream(topology, stream):
    system = CompositeSystem.__new__(CompositeSystem)
    system._lib, system._topology, system.handle = capi.load(), topology, C.c_void_p()
    options = capi.Options(stream=stream)
    capi.check(system._lib.pcfd_system_create(C.byref(topology), C.byref(options), C.byref(system.handle)))
    system.storage_size = topology.storage_size
    return system


def test_read_backs_follow_the_callers_stream(gpu):
    """1.2 M cells, 9.4 MB a vector: a product right after it was enqueued, from the thread that made
    the system and from a fresh one, on the thread's own stream and on one of the library's."""
    vertices, triangles = extruded_wing(rotate_section(naca4_section(12, 48, 1.0), 4.0), -0.6, 0.6)
    built = BuiltTopology(vertices, triangles, (-1.0, -1.0, -1.0), (2.0, 1.0, 1.0), 1 / 48, 1, 8)
    n = built.storage_size
    assert 8 * n > 8 << 20
    inputs = [np.where(built.active, np.random.default_rng(seed).standard_normal(n), 0.0) for seed in range(3)]
    results = []
    for stream in (None, PER_THREAD):
        with on_stream(built.topology, stream) as s:
            here, there = [s.apply(p) for p in inputs], []
            thread = threading.Thread(target=lambda: there.extend(s.apply(p) for p in inputs))
            thread.start()
            thread.join()
            results += [here, there]
    built.close()
    for other in results[1:]:
        for a, b in zip(results[0], other):
            assert np.array_equal(a, b)
