"""Calls that are summed pose by pose although finer ones go site by site:
local expansions in forward + adjoint, page-locked outputs by slabs of work
items, and String paths too long for the cooperative loop, which iterate by
graphs.  The bars are the mixed mode's: 1e-4 K where E <= 0, 1e-6 relative
above, gradients 1e-5 relative (floor 1 K/A); the String iteration is held to
its CPU restatement as in the other String tests."""
import numpy as np
import pytest
import torch

from oracle import oracle, string_oracle
from string_vext_b200 import _lib, synth
from string_vext_b200.orientation import normalized_directors
from string_vext_b200.string_path import euler_from_quaternions, run_string
from string_vext_b200.system import VextBatch, VextSystem

pytestmark = pytest.mark.gpu


def directors(n):
    return normalized_directors(np.random.default_rng(n).normal(size=(n, 3)))


def random_case(lengths, angles, n, masses=None):
    rng = np.random.default_rng(n)
    kind = rng.integers(0, 4, n)
    case = synth.make_case(lengths, angles, rng.random((n, 3)), synth.TYPE_TABLE[kind, 1],
                           synth.TYPE_TABLE[kind, 0], synth.GUEST_A, 12.8)
    if masses:
        case["guest_mass"], case["total_mass"] = np.array(masses), float(sum(masses))
    return case


def dense(masses=None):
    return random_case([11.0, 12.0, 10.0], [80.0, 95.0, 100.0], 220, masses)


def dilute():
    return random_case([9.0, 11.0, 8.0], [90.0, 90.0, 90.0], 4)


def layered(masses=None):
    case = synth.full_field()
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


@pytest.mark.parametrize("masses", [None, (15.0, 25.0)])
@pytest.mark.parametrize("maker,size,n_axes,options", [
    (dense, 13, 64, {"centers_per_region": 8}), (dense, 16, 33, {"centers_per_region": 8}),
    (dense, 21, 65, {"centers_per_region": 8}), (layered, 21, 25, {})])
def test_adjoint_expansions_pose_by_pose(maker, size, n_axes, options, masses):
    axes = directors(n_axes)
    with VextSystem(maker(masses)) as system:
        ex, gx = adjoint(system, size, axes, mode=_lib.VEXT_MODE_FP64_PLAIN)
        e, g = adjoint(system, size, axes, **options)
        assert_energy(e, ex)
        assert_gradient(g, gx)
        # a batch of it, replayed
        out = torch.empty(e.shape, dtype=torch.float32, device="cuda")
        grad = torch.empty(g.shape, dtype=torch.float32, device="cuda")
        batch = VextBatch([system], size, axes, [out], gradients=[grad], **options)
        assert batch.info()["cta_shape"] != "64-site clusters"
        for _ in range(2):
            batch.run()
        batch.check()
        torch.cuda.synchronize()
        assert_energy(out.cpu().numpy().astype(np.float64), ex, storage=1.2e-7)
        assert_gradient(grad.cpu().numpy().astype(np.float64), gx)
        batch.close()


@pytest.mark.parametrize("maker,size,n_axes,options", [
    (dilute, 41, 90, {}), (dense, 33, 70, {"centers_per_region": 8})])
def test_slabs_pose_by_pose(maker, size, n_axes, options):
    """Page-locked outputs of two and more slabs, without and with local
    expansions (which the first slab evaluates for all): the device entry's
    bits, twice, and the FP64 values."""
    axes = directors(n_axes)
    shape = (n_axes,) + (size,) * 3
    with VextSystem(maker()) as system:
        ex, gx = adjoint(system, size, axes, mode=_lib.VEXT_MODE_FP64_PLAIN)
        e = torch.empty(shape, dtype=torch.float32, device="cuda")
        g = torch.empty(shape + (6,), dtype=torch.float32, device="cuda")
        system.field_adjoint_device(size, axes, e, g, **options)
        torch.cuda.synchronize()
        for _ in range(2):
            he, hg = system.field_adjoint(size, axes, pinned=True, **options)
            np.testing.assert_array_equal(he, e.cpu().numpy())
            np.testing.assert_array_equal(hg, g.cpu().numpy())
        assert_energy(he.astype(np.float64), ex, storage=1.2e-7)
        assert_gradient(hg.astype(np.float64), gx)


@pytest.mark.parametrize("n_images", [296, 297, 400])
def test_long_paths_match_cpu_restatement(n_images):
    """The longest path of the cooperative loop and paths by graphs, plain and
    checked iterations."""
    case, frac, quat, _, _ = synth.string_path()
    path = np.column_stack([frac, np.mod(euler_from_quaternions(quat), 2 * np.pi)])
    at = np.linspace(0, len(path) - 1, n_images)
    low = np.minimum(at.astype(int), len(path) - 2)
    s = path[low] + (at - low)[:, None] * (path[low + 1] - path[low])
    with VextSystem(case) as system:
        gpu, e_gpu, res = run_string(system, s, mode=_lib.VEXT_MODE_FP64, direction=3,
                                     max_iterations=4, check_every=2, conv_trans_percent=0.0)
    ref = s.copy()
    for _ in range(4):
        ref = string_oracle.iteration(case, ref, direction=3)[0]
    assert res["iterations"] == 4 and not res["converged"]
    np.testing.assert_allclose(gpu[:, :3], ref[:, :3], rtol=0, atol=1e-10)
    np.testing.assert_allclose(gpu[:, 3:], ref[:, 3:], rtol=0, atol=1e-9)
    np.testing.assert_allclose(e_gpu, string_oracle.pose_energy(case, gpu), rtol=1e-10, atol=1e-8)


def test_adjoint_into_host_memory_beside_other_calls():
    """Device-pointer calls into page-locked memory (both outputs or one) keep
    their results when the next call of the system starts before they end, and
    device outputs are as before afterwards."""
    size, axes, other = 33, directors(70), directors(24)
    shape = (len(axes),) + (size,) * 3
    options = {"centers_per_region": 8}
    with VextSystem(dense()) as system:
        ex, gx = adjoint(system, size, axes, mode=_lib.VEXT_MODE_FP64_PLAIN)
        first = adjoint(system, size, axes, **options)
        system.field(size, other, **options)   # scratch and lists in place
        for pin_energy, pin_gradient in ((True, True), (False, True), (True, False)):
            e = torch.empty(shape, dtype=torch.float32, pin_memory=pin_energy,
                            device="cpu" if pin_energy else "cuda")
            g = torch.empty(shape + (6,), dtype=torch.float32, pin_memory=pin_gradient,
                            device="cpu" if pin_gradient else "cuda")
            for _ in range(2):
                system.field_adjoint_device(size, axes, e, g, **options)
                system.field(size, other, **options)
                torch.cuda.synchronize()
                assert_energy(e.cpu().numpy().astype(np.float64), ex, storage=1.2e-7)
                assert_gradient(g.cpu().numpy().astype(np.float64), gx)
        for a, b in zip(adjoint(system, size, axes, **options), first):
            np.testing.assert_array_equal(a, b)


def test_expansions_of_more_than_four_million_regions():
    """More region tiles than one of the smaller grid dimensions holds."""
    size, axes = 324, directors(32)
    case = random_case([36.0] * 3, [90.0] * 3, 1100)
    with VextSystem(case) as system:
        out = torch.empty((len(axes),) + (size,) * 3, dtype=torch.float32, device="cuda")
        system.field_device(size, axes, out, centers_per_region=8)
        torch.cuda.synchronize()
        rng = np.random.default_rng(5)
        o = rng.integers(0, len(axes), 2000)
        at = rng.integers(0, size, (2000, 3))
        at[:8] = [[i, j, k] for i in (0, size - 1) for j in (0, size - 1) for k in (0, size - 1)]
        got = out[tuple(torch.from_numpy(x).cuda() for x in (o, *at.T))].cpu().numpy()
    exact = oracle.pose_energy_grad(case, (at + 0.5) / size @ case["cell"], axes[o])[0]
    assert_energy(got.astype(np.float64), exact, storage=1.2e-7)


@pytest.mark.parametrize("n_axes", [10600, 10800, 1900000])
def test_many_directors_on_a_small_grid(n_axes):
    """Directors up to and beyond what an expansion's evaluation matrix holds."""
    size, axes = 4, directors(n_axes)
    case = random_case([4.0, 4.2, 3.9], [90.0, 90.0, 90.0], 8)
    with VextSystem(case) as system:
        e = torch.empty((n_axes,) + (size,) * 3, dtype=torch.float32, device="cuda")
        g = torch.empty(tuple(e.shape) + (6,), dtype=torch.float32, device="cuda")
        free = torch.cuda.mem_get_info()[0]
        system.field_adjoint_device(size, axes, e, g)
        torch.cuda.synchronize()
        assert free - torch.cuda.mem_get_info()[0] < 2 << 30
        rng = np.random.default_rng(6)
        o = rng.integers(0, n_axes, 500)
        at = rng.integers(0, size, (500, 3))
        where = tuple(torch.from_numpy(x).cuda() for x in (o, *at.T))
        got, grad = e[where].cpu().numpy(), g[where].cpu().numpy()
    exact, gc, gu = oracle.pose_energy_grad(case, (at + 0.5) / size @ case["cell"], axes[o])
    gu = gu - (gu * axes[o]).sum(1)[:, None] * axes[o]
    assert_energy(got.astype(np.float64), exact, storage=1.2e-7)
    assert_gradient(grad.astype(np.float64), np.concatenate([gc, gu], 1))


def test_lists_follow_the_directors():
    """Few directors are summed on lists without classes for expansions, whose
    regions cut by the grid's edge are smaller; many ones on lists with them;
    either way the same call gives the same bits again."""
    size = 25
    with VextSystem(dense()) as system:
        seen = {}
        for n_axes in (4, 64, 4, 64):
            out = system.field(size, directors(n_axes), centers_per_region=16)["orientation_K"]
            entries = system.last_stats["list_entries"]
            if n_axes in seen:
                np.testing.assert_array_equal(out, seen[n_axes][0])
                assert entries == seen[n_axes][1]
            seen[n_axes] = out, entries
        assert seen[4][1] < seen[64][1]
        exact = system.field(size, directors(4), energy=True,
                             mode=_lib.VEXT_MODE_FP64)["energy"].T.reshape(seen[4][0].shape)
        assert_energy(seen[4][0].astype(np.float64), exact, storage=1.2e-7)


def slab(lengths, angles, n, thickness, guest, seed):
    rng = np.random.default_rng(seed)
    frac = rng.random((n, 3))
    frac[:, 2] *= thickness
    kind = rng.integers(0, 4, n)
    return synth.make_case(lengths, angles, frac, synth.TYPE_TABLE[kind, 1],
                           synth.TYPE_TABLE[kind, 0], guest, 12.8)


def test_expansions_no_less_accurate_than_pairs():
    """Six slab frameworks, half of their poses at E <= 0: the rms errors there,
    by expansion pose by pose, are on average no larger than those of the sum over
    pairs (1.70e-5 K), and so is the largest error (1.58e-4 K: beyond 1e-4 K, as
    FP32 pair terms near 5 A add up in such frameworks)."""
    tilted = [85.0, 95.0, 100.0]
    runs = [(slab([9.0, 10.0, 14.0], [90.0, 90.0, 110.0], 40, 0.35, synth.GUEST_A, 40), size, n)
            for size, n in ((21, 65), (24, 41))]
    for guest in (synth.GUEST_A, synth.GUEST_B):
        runs.append((slab([12.0, 12.0, 20.0], tilted, 90, 0.4, guest, 28), 28, 64))
        runs.append((slab([18.0, 17.0, 26.0], tilted, 300, 0.4, guest, 40), 40, 32))
    rms, worst = [], []
    for case, size, n_axes in runs:
        axes = directors(n_axes)
        with VextSystem(case) as system:
            exact = adjoint(system, size, axes, mode=_lib.VEXT_MODE_FP64_PLAIN)[0]
            err = (adjoint(system, size, axes, centers_per_region=8)[0] - exact)[exact <= 0]
        rms.append(np.sqrt((err ** 2).mean()))
        worst.append(np.abs(err).max())
    assert np.mean(rms) <= 1.70e-5
    assert max(worst) <= 1.58e-4
