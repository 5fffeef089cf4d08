"""Device memory of calls that come and go (string_vext_b200/csrc/memory.cu)."""
import threading
from contextlib import contextmanager

import numpy as np
import pytest
import torch

from string_vext_b200 import _lib, synth
from string_vext_b200.orientation import normalized_directors
from string_vext_b200.system import VextBatch, VextPoseBatch, VextSystem, release_memory

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


def test_pose_list_build_scratch():
    """4 KB of scratch per pose bin (0.75 A between lattice planes) beside the
    lists, which a cell without images in reach of most bins keeps small."""
    rng = np.random.default_rng(9)
    edge, n = 45.0, 12
    case = synth.make_case([edge] * 3, [90.0] * 3, rng.random((n, 3)),
                           np.full(n, 3.0), np.full(n, 40.0), synth.GUEST_A, 6.0)
    release_memory()
    free = torch.cuda.mem_get_info()[0]
    with VextSystem(case) as system:
        batch = VextPoseBatch([system], [4])
        held = free - torch.cuda.mem_get_info()[0]
        batch.close()
    bins = round(edge / 0.75) ** 3
    listed = 4 / 3 * np.pi * (6.0 + 0.8 + 0.7) ** 3 * n / edge ** 3
    assert held < bins * (4096 + 200 + 32 * 1.5 * listed) + (64 << 20)


# ---- scratch of the faster sums that cannot be had: the plainer ones serve

@contextmanager
def hog(leave):
    """Hold all device memory but `leave` bytes."""
    torch.cuda.synchronize()
    release_memory()
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        torch.cuda.synchronize()
        held.untyped_storage().resize_(0)
        torch.cuda.empty_cache()


def outputs(size, n_axes):
    shape = (n_axes,) + (size,) * 3
    return (torch.empty(shape, dtype=torch.float32, device="cuda"),
            torch.empty(shape + (6,), dtype=torch.float32, device="cuda"))


def exact_adjoint(system, size, axes):
    shape = (len(axes),) + (size,) * 3
    e = torch.empty(shape, dtype=torch.float64, device="cuda")
    g = torch.empty(shape + (6,), dtype=torch.float64, device="cuda")
    system.field_adjoint_device(size, axes, None, None, e, g, mode=_lib.VEXT_MODE_FP64_PLAIN)
    torch.cuda.synchronize()
    return e.cpu().numpy(), g.cpu().numpy()


def assert_mixed(e, g, exact):
    ex, gx = exact
    err = np.abs(e - ex) - 1.2e-7 * np.abs(ex)
    neg = ex <= 0
    assert err[neg].max(initial=0) < 1e-4
    assert (err / np.maximum(np.abs(ex), 1))[~neg].max(initial=0) < 1e-6
    if g is not None:
        err = np.linalg.norm(g - gx, axis=-1) / np.maximum(np.linalg.norm(gx, axis=-1), 1.0)
        assert err.max() < 1e-5


@pytest.fixture(scope="module")
def fine_field():
    size, axes = 40, directors(64)
    with VextSystem(synth.small_field()) as system:
        return size, axes, exact_adjoint(system, size, axes)


def test_adjoint_field_without_room_for_site_sums(fine_field):
    size, axes, exact = fine_field
    e, g = outputs(size, len(axes))
    with VextSystem(synth.small_field()) as system:
        with hog(500 << 20):
            system.field_adjoint_device(size, axes, e, g)
            torch.cuda.synchronize()
            assert_mixed(e.cpu().numpy(), g.cpu().numpy(), exact)
        for pinned in (False, True):   # with room again
            assert_mixed(*system.field_adjoint(size, axes, pinned=pinned), exact)


@pytest.mark.parametrize("pinned", [False, True])
def test_host_adjoint_without_room_for_site_sums(fine_field, pinned):
    size, axes, exact = fine_field
    with VextSystem(synth.small_field()) as system:
        with hog(640 << 20):
            assert_mixed(*system.field_adjoint(size, axes, pinned=pinned), exact)


def test_batch_without_room_for_site_sums(fine_field):
    size, axes, exact = fine_field
    outs = [outputs(size, len(axes)) for _ in range(2)]
    with VextSystem(synth.small_field()) as a, VextSystem(synth.small_field()) as b, \
            hog(500 << 20):
        batch = VextBatch([a, b], size, axes, [o[0] for o in outs],
                          gradients=[o[1] for o in outs])
        assert batch.info()["cta_shape"] != "64-site clusters"
        batch.run()
        batch.check()
        torch.cuda.synchronize()
        for e, g in outs:
            assert_mixed(e.cpu().numpy(), g.cpu().numpy(), exact)
        batch.close()


def test_field_without_room_for_site_sums(fine_field):
    size, axes, exact = fine_field
    with VextSystem(synth.small_field()) as system:
        with hog(260 << 20):
            small = system.field(20, axes)["orientation_K"]
            for _ in range(2):
                assert_mixed(system.field(size, axes)["orientation_K"], None, exact)
            np.testing.assert_array_equal(system.field(20, axes)["orientation_K"], small)


def test_adjoint_without_room_for_expansions():
    size, axes = 4, directors(10600)   # an evaluation matrix of 1 GB
    rng = np.random.default_rng(8)
    kind = rng.integers(0, 4, 8)
    case = synth.make_case([4.0, 4.2, 3.9], [90.0, 90.0, 90.0], rng.random((8, 3)),
                           synth.TYPE_TABLE[kind, 1], synth.TYPE_TABLE[kind, 0],
                           synth.GUEST_A, 12.8)
    with VextSystem(case) as system:
        exact = exact_adjoint(system, size, axes)
        e, g = outputs(size, len(axes))
        with hog(600 << 20):
            system.field_adjoint_device(size, axes, e, g)
            torch.cuda.synchronize()
        assert_mixed(e.cpu().numpy(), g.cpu().numpy(), exact)
