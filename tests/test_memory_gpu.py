"""Device memory of calls that come and go (string_vext_b200/csrc/memory.cu)."""
import threading

import numpy as np
import pytest
import torch

from string_vext_b200 import synth
from string_vext_b200.orientation import normalized_directors
from string_vext_b200.system import VextSystem, release_memory

pytestmark = pytest.mark.gpu


def directors(n):
    return normalized_directors(np.random.default_rng(n).normal(size=(n, 3)))


def test_systems_dropped_beside_another_threads_capture():
    """A thread makes and drops systems while another one captures a graph
    thread-locally: the capture goes on, and the fields are right."""
    case, axes = synth.small_field(), directors(20)
    with VextSystem(case) as system:
        expected = system.field(12, axes)["orientation_K"]
    x = torch.ones(1 << 20, device="cuda")
    torch.cuda.synchronize()
    inside, done = threading.Event(), threading.Event()
    seen = []

    def drop_systems():
        try:
            inside.wait(30)
            for _ in range(3):
                with VextSystem(case) as system:
                    seen.append(system.field(12, axes)["orientation_K"])
        except Exception as error:   # shown below
            seen.append(error)
        finally:
            done.set()

    thread = threading.Thread(target=drop_systems)
    thread.start()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        y = x * 2
        inside.set()
        assert done.wait(60)
        z = y + 1
    thread.join()
    graph.replay()
    torch.cuda.synchronize()
    assert bool((z == 3).all())
    assert len(seen) == 3
    for field in seen:
        np.testing.assert_array_equal(field, expected)


def test_release_memory_gives_back_what_dropped_systems_held():
    case, axes = synth.full_field(), directors(64)
    release_memory()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(2):
        with VextSystem(case) as system:
            kept = system.field(40, axes)["orientation_K"]
        assert free - torch.cuda.mem_get_info()[0] > 50 << 20   # kept for the next one
        release_memory()
        assert abs(free - torch.cuda.mem_get_info()[0]) < 16 << 20
    with VextSystem(case) as system:
        release_memory()   # what is in use stays
        np.testing.assert_array_equal(system.field(40, axes)["orientation_K"], kept)
        release_memory()
        np.testing.assert_array_equal(system.field(40, axes)["orientation_K"], kept)
