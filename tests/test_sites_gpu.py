"""Fields summed site by site in clusters (fine grids) against the plain FP64
kernels and against the sum pose by pose: idle places in the last cluster
(17 and 33 directors), blocks cut by the grid's edge, skewed and flat cells,
sites wrapping around a short axis, guests with off-center sites, other near
radii and a site on top of a framework atom.  The bars are the mixed mode's:
1e-4 K where E <= 0, 1e-6 relative above, gradients 1e-5 relative (floor 1
K/A); float32 outputs are rounded on top of it."""
import numpy as np
import pytest
import torch

from string_vext_b200 import _lib, synth
from string_vext_b200.orientation import normalized_directors
from string_vext_b200.physics import body_offsets
from string_vext_b200.system import VextBatch, VextSystem

pytestmark = pytest.mark.gpu

CELLS = {"skewed": ([14.0, 12.0, 13.0], [75.0, 85.0, 115.0], 90),
         "flat": ([16.0, 15.0, 3.6], [90.0, 90.0, 120.0], 60),
         "sparse": ([9.0, 11.0, 8.0], [90.0, 90.0, 90.0], 12),
         "dilute": ([9.0, 11.0, 8.0], [90.0, 90.0, 90.0], 4),
         "dense": ([11.0, 12.0, 10.0], [80.0, 95.0, 100.0], 220)}


def directors(n):
    return normalized_directors(np.random.default_rng(n).normal(size=(n, 3)))


def make_case(cell, masses=None, guest=synth.GUEST_A, extra=None):
    lengths, angles, n = CELLS[cell]
    rng = np.random.default_rng(n)
    frac = rng.random((n, 3))
    if extra is not None:
        frac[0] = extra
    kind = rng.integers(0, 4, n)
    case = synth.make_case(lengths, angles, frac, synth.TYPE_TABLE[kind, 1],
                           synth.TYPE_TABLE[kind, 0], guest, 12.8)
    if masses:
        case["guest_mass"], case["total_mass"] = np.array(masses), float(sum(masses))
    return case


def assert_energy(got, exact, storage=0.0):
    err = np.abs(got - exact) - storage * np.abs(exact)
    neg = exact <= 0
    assert err[neg].max(initial=0) < 1e-4
    assert (err / np.maximum(np.abs(exact), 1))[~neg].max(initial=0) < 1e-6


def assert_gradient(got, exact):
    err = np.linalg.norm(got - exact, axis=-1) / np.maximum(np.linalg.norm(exact, axis=-1), 1.0)
    assert err.max() < 1e-5


def adjoint(system, size, axes, **options):
    shape = (len(axes),) + (size,) * 3
    exact = options.get("mode") == _lib.VEXT_MODE_FP64_PLAIN
    e = None if exact else torch.empty(shape, dtype=torch.float32, device="cuda")
    g = None if exact else torch.empty(shape + (6,), dtype=torch.float32, device="cuda")
    e64 = torch.empty(shape, dtype=torch.float64, device="cuda")
    g64 = torch.empty(shape + (6,), dtype=torch.float64, device="cuda") if exact else None
    system.field_adjoint_device(size, axes, e, g, e64, g64, **options)
    torch.cuda.synchronize()
    return e64.cpu().numpy(), (g64 if exact else g).cpu().numpy().astype(np.float64)


def check(case, size, axes, **options):
    with VextSystem(case) as system:
        ex, gx = adjoint(system, size, axes, mode=_lib.VEXT_MODE_FP64_PLAIN)
        e, g = adjoint(system, size, axes, **options)
        assert_energy(e, ex)
        assert_gradient(g, gx)
        out = system.field(size, axes, energy=True, **options)
        assert_energy(out["energy"].T.reshape(ex.shape), ex)
        # pose by pose: regions of eight grid centers
        e8, g8 = adjoint(system, size, axes, centers_per_region=8, **options)
        neg = ex <= 0
        assert np.abs(e - e8)[neg].max(initial=0) < 2e-4
        # batches, replayed; this call does go by sites
        shape = e.shape
        outs = [torch.empty(shape, dtype=torch.float32, device="cuda") for _ in range(2)]
        grads = [torch.empty(shape + (6,), dtype=torch.float32, device="cuda") for _ in range(2)]
        for adj in (False, True):
            with VextSystem(make_case("sparse")) as other:
                batch = VextBatch([system, other], size, axes, outs,
                                  gradients=grads if adj else None, **options)
                assert batch.info()["cta_shape"] == "64-site clusters"
                for _ in range(2):
                    batch.run()
                batch.check()
                torch.cuda.synchronize()
                assert_energy(outs[0].cpu().numpy().astype(np.float64), ex, storage=1.2e-7)
                if adj:
                    assert_gradient(grads[0].cpu().numpy().astype(np.float64), gx)
                batch.close()


@pytest.mark.parametrize("masses", [None, (15.0, 25.0)])
@pytest.mark.parametrize("cell,size,n_axes", [
    ("skewed", 25, 17), ("skewed", 24, 64), ("flat", 27, 33), ("sparse", 16, 50)])
def test_fields_by_sites_match_fp64(cell, size, n_axes, masses):
    check(make_case(cell, masses), size, directors(n_axes))


@pytest.mark.parametrize("masses", [None, (15.0, 25.0)])
@pytest.mark.parametrize("size,n_axes", [(19, 17), (23, 33), (18, 96)])
def test_expansions_at_sites(size, n_axes, masses):
    """Local expansions by matrix product: partial tiles of sites and regions."""
    check(make_case("dense", masses), size, directors(n_axes))


def test_batch_of_both_routes():
    """A system by sites beside a dilute one by poses in one batch."""
    size, axes = 20, directors(40)
    shape = (40,) + (size,) * 3
    with VextSystem(make_case("skewed")) as a, VextSystem(make_case("dilute")) as b:
        exact = [adjoint(s, size, axes, mode=_lib.VEXT_MODE_FP64_PLAIN) for s in (a, b)]
        for adj in (False, True):
            outs = [torch.empty(shape, dtype=torch.float32, device="cuda") for _ in range(2)]
            grads = [torch.empty(shape + (6,), dtype=torch.float32, device="cuda")
                     for _ in range(2)]
            batch = VextBatch([a, b], size, axes, outs, gradients=grads if adj else None)
            assert batch.info()["cta_shape"] != "64-site clusters"
            for _ in range(2):
                batch.run()
            batch.check()
            torch.cuda.synchronize()
            for k, (ex, gx) in enumerate(exact):
                assert_energy(outs[k].cpu().numpy().astype(np.float64), ex, storage=1.2e-7)
                if adj:
                    assert_gradient(grads[k].cpu().numpy().astype(np.float64), gx)
            batch.close()


@pytest.mark.parametrize("r_split", [6.0, 8.5])
def test_other_near_radii(r_split):
    check(make_case("skewed", guest=synth.GUEST_B), 20, directors(32), r_split=r_split)


def test_site_on_an_atom():
    """A site within the contact floor of an atom."""
    size, axes = 23, directors(24)
    case = make_case("skewed")
    offset = body_offsets(case)[1]
    center = (np.array([3, 7, 11]) + 0.5) / size
    frac = center + offset * axes[5] @ np.linalg.inv(case["cell"]) + 1e-3
    check(make_case("skewed", extra=frac % 1.0), size, axes)
