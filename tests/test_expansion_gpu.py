"""Fields whose far inner pairs are summed by local expansion (dense cells on
fine grids) against the plain FP64 kernels, at sizes that leave partial
blocks, partial tiles of poses and of regions, one director past a block of
64, and guests with off-center sites (which keep both sites of the whole
shell).  The bars are the mixed mode's: 1e-4 K where E <= 0, 1e-6 relative
above, gradients 1e-5 relative (floor 1 K/A)."""
import numpy as np
import pytest
import torch

from string_vext_b200 import _lib, synth
from string_vext_b200.orientation import normalized_directors
from string_vext_b200.system import VextBatch, VextSystem

pytestmark = pytest.mark.gpu


def dense_case(guest=synth.GUEST_A, masses=None):
    rng = np.random.default_rng(61)
    n = 220
    kind = rng.integers(0, 4, n)
    case = synth.make_case([11.0, 12.0, 10.0], [80.0, 95.0, 100.0], rng.random((n, 3)),
                           synth.TYPE_TABLE[kind, 1], synth.TYPE_TABLE[kind, 0], guest, 12.8)
    if masses:
        case["guest_mass"], case["total_mass"] = np.array(masses), float(sum(masses))
    return case


def small_case(masses=None):
    case = synth.small_field()
    if masses:
        case["guest_mass"], case["total_mass"] = np.array(masses), float(sum(masses))
    return case


def directors(n):
    return normalized_directors(np.random.default_rng(n).normal(size=(n, 3)))


def assert_energy(got, exact, storage=0.0):
    err = np.abs(got - exact) - storage * np.abs(exact)
    neg = exact <= 0
    assert err[neg].max(initial=0) < 1e-4
    assert (err / np.maximum(np.abs(exact), 1))[~neg].max(initial=0) < 1e-6


def assert_gradient(got, exact):
    err = np.linalg.norm(got - exact, axis=-1) / np.maximum(np.linalg.norm(exact, axis=-1), 1.0)
    assert err.max() < 1e-5


def exact_adjoint(system, size, axes):
    shape = (len(axes),) + (size,) * 3
    e = torch.empty(shape, dtype=torch.float64, device="cuda")
    g = torch.empty(shape + (6,), dtype=torch.float64, device="cuda")
    system.field_adjoint_device(size, axes, None, None, e, g, mode=_lib.VEXT_MODE_FP64_PLAIN)
    torch.cuda.synchronize()
    return e.cpu().numpy(), g.cpu().numpy()


@pytest.mark.parametrize("masses", [None, (15.0, 25.0)])
@pytest.mark.parametrize("maker,size,n_axes", [
    (dense_case, 13, 64), (dense_case, 16, 33), (dense_case, 21, 65), (dense_case, 24, 41),
    (small_case, 20, 64)])   # accessible poses (E <= 0); expansions in the forward field
def test_fields_with_expansions_match_fp64(maker, size, n_axes, masses):
    axes = directors(n_axes)
    shape = (n_axes,) + (size,) * 3
    with VextSystem(maker(masses=masses)) as system:
        ex, gx = exact_adjoint(system, size, axes)
        e = torch.empty(shape, dtype=torch.float32, device="cuda")
        g = torch.empty(shape + (6,), dtype=torch.float32, device="cuda")
        e64 = torch.empty(shape, dtype=torch.float64, device="cuda")
        system.field_adjoint_device(size, axes, e, g, e64)
        torch.cuda.synchronize()
        assert_energy(e64.cpu().numpy(), ex)
        assert_gradient(g.cpu().numpy().astype(np.float64), gx)
        # the host entries: device scratch, page-locked and pageable outputs
        for pinned in (False, True):
            he, hg = system.field_adjoint(size, axes, pinned=pinned)
            np.testing.assert_array_equal(he, e.cpu().numpy())
            np.testing.assert_array_equal(hg, g.cpu().numpy())
        for cb in (8, 16):
            out = system.field(size, axes, energy=True, centers_per_region=cb)
            assert_energy(out["energy"].T.reshape(shape), ex)
            # a second call (plan kept) and other directors in between: same bits
            system.field(size, directors(7), centers_per_region=cb)
            again = system.field(size, axes, centers_per_region=cb)
            np.testing.assert_array_equal(again["orientation_K"], out["orientation_K"])


def test_batch_mixes_systems_with_and_without_expansions():
    """A dense framework with both guests on shared lists beside a dilute one
    (direct sums) in one batch, forward and forward + adjoint, replayed."""
    size, axes = 18, directors(64)
    cases = [dense_case(), dense_case(synth.GUEST_B), synth.small_field()]
    systems = [VextSystem(c) for c in cases]
    shape = (64,) + (size,) * 3
    for adjoint in (False, True):
        outs = [torch.empty(shape, dtype=torch.float32, device="cuda") for _ in systems]
        grads = [torch.empty(shape + (6,), dtype=torch.float32, device="cuda")
                 for _ in systems] if adjoint else None
        batch = VextBatch(systems, size, axes, outs, gradients=grads)
        seen = []
        for _ in range(2):
            batch.run()
            batch.check()
            torch.cuda.synchronize()
            seen.append([t.cpu().numpy() for t in outs + (grads or [])])
        for a, b in zip(*seen):
            np.testing.assert_array_equal(a, b)
        for k, system in enumerate(systems):
            ex, gx = exact_adjoint(system, size, axes)
            assert_energy(seen[0][k].astype(np.float64), ex, storage=1.2e-7)
            if adjoint:
                assert_gradient(seen[0][3 + k].astype(np.float64), gx)
        batch.close()
    for s in systems:
        s.close()


@pytest.mark.parametrize("size,n_axes", [(30, 96), (33, 70)])
def test_page_locked_outputs_by_slabs(size, n_axes):
    """Outputs of 50 MB and more leave by slabs of grid planes while the next
    slab computes (33 planes in four slabs, the last block of them partial):
    the same bits as the device entry, twice, also into a second buffer."""
    axes = directors(n_axes)
    shape = (n_axes,) + (size,) * 3
    with VextSystem(synth.small_field()) as system:
        e = torch.empty(shape, dtype=torch.float32, device="cuda")
        g = torch.empty(shape + (6,), dtype=torch.float32, device="cuda")
        system.field_adjoint_device(size, axes, e, g)
        torch.cuda.synchronize()
        kept = []
        for _ in range(2):
            kept.append(system.field_adjoint(size, axes, pinned=True))
            np.testing.assert_array_equal(kept[-1][0], e.cpu().numpy())
            np.testing.assert_array_equal(kept[-1][1], g.cpu().numpy())
