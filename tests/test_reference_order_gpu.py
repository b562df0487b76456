"""Lattices that track in the reference's element order in the default build (most of their elements have no
form in csrc/fastmaps.cuh) through the plain kernel, batches, the server and the adjoint.

Results: a batch or server round that holds such a lattice beside others gives each lattice the bits of
the plain kernel. Time: the same kernel code inline in the batch kernel as in the plain one, so a batch
of one such lattice takes what the plain kernel takes with the same shape; 1.35 allows for the work queue
and the clocks (an out-of-line call per element took 1.65 and more)."""
import importlib
import time

import numpy as np
import pytest

from conftest import load_abi

pytestmark = pytest.mark.gpu
lib = importlib.import_module("bmad-ecosystem_b200.lib")
rings = importlib.import_module("bmad-ecosystem_b200.rings")
abi = load_abi()
E = abi.default_element
AP = dict(x1_limit=0.02, x2_limit=0.02, y1_limit=0.01, y2_limit=0.01)


@pytest.fixture(scope="module")
def ctx():
    c = lib.Context(0)
    yield c
    c.close()


def thin_ring(rare=False, cells=50):
    """A ring with a thin multipole after every element, two after drifts."""
    eles, p = rings.ring(cells)
    out = []
    for e in eles:
        if rare and e.key == abi.QUADRUPOLE:
            e.fringe_type = abi.FRINGE_FULL
        out.append(e)
        if e.key != abi.RFCAVITY:
            out += [E(abi.AB_MULTIPOLE, b_pole={2: 1e-3, 3: -2e-2}, **AP)] * (2 if e.key == abi.DRIFT else 1)
    rings.set_ref_time(out, p)
    return out, p


LATTICES = {"thin": lambda: thin_ring(), "plain": lambda: rings.ring(50), "thin_rare": lambda: thin_ring(True, 20),
            "perturbed": lambda: rings.perturbed_ring(20, seed=3)}


def bunch(name, p, n):
    vec = rings.matched_gaussian(rings.ring(50)[0], n, seed=len(name), scale=3.0)
    vec[0, ::5] += 0.025        # outside the first element's aperture
    vec[1, 1::7] += 3e-3        # lost within a few cells
    return lib.HostBunch.from_vec(vec, p)


def plain(ctx, lat, b, turns):
    lib.track_bunch(ctx, lat, b, n_turns=turns)
    return b


def same(got, want, name):
    assert np.any(want.state != abi.ALIVE)          # losses are part of it
    for k in ("state", "ix_ele", "ix_turn", "location"):
        assert np.array_equal(getattr(got, k), getattr(want, k)), (name, k)
    assert np.array_equal(got.vec, want.vec) and np.array_equal(got.beta, want.beta), name


@pytest.mark.parametrize("names", [("thin",), ("plain", "thin"), ("thin_rare", "perturbed", "thin", "plain")])
@pytest.mark.parametrize("block,ctas", [(None, None), (64, 4), (64, 12), (128, 0), (128, 5), (256, 3), (512, 1)])
def test_batch_gives_the_plain_kernels_bits(ctx, names, block, ctas):
    n, turns, per = 700, 5, 2
    made = {k: LATTICES[k]() for k in names}
    lats = {k: lib.Lattice(ctx, *made[k]) for k in names}
    batch = lib.Batch(ctx, [lats[k] for k in names], [n] * len(names))
    batch.set_tuning(turns_per_launch=per, **({} if block is None else dict(block=block, ctas_per_sm=ctas)))
    for v, k in enumerate(names):
        batch.upload(v, bunch(k, made[k][1], n))
    batch.track(turns)
    ctx.set_tuning(block=128, ctas_per_sm=0, turns_per_launch=per, compact=1)
    for v, k in enumerate(names):
        got = bunch(k, made[k][1], n)
        batch.download(v, got)
        same(got, plain(ctx, lats[k], bunch(k, made[k][1], n), turns), k)
    ctx.set_tuning(turns_per_launch=0, compact=0)
    batch.close()


def test_server_gives_the_plain_kernels_bits(ctx):
    n, turns = 700, 4
    made = {k: LATTICES[k]() for k in sorted(LATTICES)}
    lats = {k: lib.Lattice(ctx, *made[k]) for k in made}
    srv = lib.Server(ctx, max_particles=1 << 16)
    jobs = {}
    for k in made:
        b = bunch(k, made[k][1], n)
        jobs[k] = (b, srv.submit(lats[k], b, turns))
    for k, (b, i) in jobs.items():
        srv.wait(i)
    srv.close()
    for k, (b, _) in jobs.items():
        # the server runs its own number of turns a launch, over which z and t alone are summed differently
        want = plain(ctx, lats[k], bunch(k, made[k][1], n), turns)
        same(b, want, k)


def test_adjoint_of_a_lattice_in_the_reference_order(ctx):
    from test_adjoint_cpu import host_loss_grad, ring_params
    from test_adjoint_gpu import _load_ha
    eles, p = rings.ring(20)
    out = []
    for e in eles:
        out.append(e)
        if e.key != abi.RFCAVITY:
            out += [E(abi.RFCAVITY, l=0.0, voltage=1e3, rf_frequency=5e8, **AP)] * (2 if e.key == abi.DRIFT else 1)
    rings.set_ref_time(out, p)
    vec = rings.matched_gaussian(eles, 40, seed=2)
    _, names = ring_params(out)
    loss_h, grad_h, _, _ = host_loss_grad(_load_ha(), out, p, vec, 4, 2)
    loss_g, grad_g = lib.loss_grad(ctx, lib.Lattice(ctx, out, p), lib.HostBunch.from_vec(vec, p), 4,
                                   [i for i, _ in names], checkpoint_every=2)
    assert abs(loss_g - loss_h) <= 1e-10 * abs(loss_h)
    quads = np.array([k == "k1" for _, k in names])
    for fam in (quads, ~quads):  # the tolerance of tests/test_adjoint_gpu.py
        assert np.max(np.abs(grad_g[fam] - grad_h[fam])) <= 1e-8 * np.max(np.abs(grad_h[fam]))


def best_ms(ctx, f, reps=7):
    out = []
    for _ in range(reps):
        ctx.synchronize()
        t = time.perf_counter()
        f()
        ctx.synchronize()
        out.append(1e3 * (time.perf_counter() - t))
    return min(out)


def test_batch_keeps_the_plain_kernels_speed(ctx):
    import ctypes
    n, turns = 4096, 6
    eles, p = thin_ring()
    lat = lib.Lattice(ctx, eles, p)
    batch = lib.Batch(ctx, [lat], [n])
    batch.set_tuning(block=128, ctas_per_sm=4)
    batch.upload(0, bunch("x", p, n))
    view = batch.view(0)
    ctx.set_tuning(block=128, ctas_per_sm=4, stage_smem=0, turns_per_launch=0, compact=0)

    def direct():
        lib.check(lib.load().bmadgpu_track_bunch_device(ctx.handle, lat.handle, ctypes.byref(view), 0, lat.n_ele, 0,
                                                        turns, None))
    batch.track(turns)  # the losses of the first turns, out of both timings
    t_plain = best_ms(ctx, direct)
    t_batch = best_ms(ctx, lambda: batch.track(turns))
    batch.close()
    assert t_batch <= 1.35 * t_plain, (t_batch, t_plain)
