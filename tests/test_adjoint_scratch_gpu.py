"""bmadgpu_loss_grad with less device memory than its preferred plan takes: every fallback (smaller chunks of
turns, checkpoints every K turns, slabs of particles) gives the bits of the preferred plan, and a call
succeeds with the memory that the per-particle sweep took (checkpoints, turn starts of a segment, element
inputs, strength derivatives)."""
import ctypes
import importlib

import numpy as np
import pytest

from conftest import load_abi
from test_adjoint_cpu import ring_params

pytestmark = pytest.mark.gpu
lib = importlib.import_module("bmad-ecosystem_b200.lib")
rings = importlib.import_module("bmad-ecosystem_b200.rings")
abi = load_abi()


def setup(n, lost):
    eles, p = rings.ring(20)
    vec = rings.matched_gaussian(eles, n, seed=5)
    if lost:
        vec[0, ::7] += 0.025
    return eles, p, vec, [i for i, _ in ring_params(eles)[1]]


def least(n, n_ele, turns, every, slots):
    return 8 * n * (6 + 1 + 7 * -(-turns // every) + 7 * every + 7 * n_ele + slots + 1) + 4 * n


@pytest.mark.parametrize("n,turns,lost", [(40, 24, False), (300, 11, True), (1000, 3, False)])
@pytest.mark.parametrize("every", [1, 3, 5, 100])
def test_every_plan_gives_the_same_bits(n, turns, lost, every):
    ctx = lib.Context(0)
    so = lib.load()
    so.bmadgpu_selftest_scratch_limit.argtypes = [ctypes.c_void_p, ctypes.c_int64]
    eles, p, vec, at = setup(n, lost)
    lat = lib.Lattice(ctx, eles, p)

    def grad():
        return lib.loss_grad(ctx, lat, lib.HostBunch.from_vec(vec, p), turns, at, checkpoint_every=every)

    launches = ctx.launch_count
    loss, want = grad()
    launches = ctx.launch_count - launches
    plans, limit = {launches}, 8 * least(n, len(eles), turns, 1, len(at)) + (turns + 8) * 64 * 8 * n * len(eles)
    refused = False
    while not refused:
        lib.check(so.bmadgpu_selftest_scratch_limit(ctx.handle, limit))
        launches = ctx.launch_count
        try:
            got_loss, got = grad()
        except lib.BmadGpuError as ex:
            assert ex.code == abi.ENOMEM
            refused = True
            assert limit < least(n, len(eles), turns, every, len(at))
            break
        plans.add(ctx.launch_count - launches)
        assert got_loss == loss
        assert np.array_equal(got, want), limit
        limit = int(limit / 1.3)
    assert len(plans) >= (4 if turns > 3 else 2)       # the limits did reach several plans
    lib.check(so.bmadgpu_selftest_scratch_limit(ctx.handle, 0))
    assert grad()[0] == loss
    lat.close()
    ctx.close()
