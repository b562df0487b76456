"""The launch shape: by the particle count until the caller or the autotuner pins one, whatever else of the
tuning is set; the same results for every shape of the rule."""
import ctypes
import importlib

import numpy as np
import pytest

from conftest import load_abi

pytestmark = pytest.mark.gpu
lib = importlib.import_module("bmad-ecosystem_b200.lib")
rings = importlib.import_module("bmad-ecosystem_b200.rings")
abi = load_abi()


@pytest.fixture()
def ctx():
    c = lib.Context(0)
    yield c
    c.close()


def test_other_fields_leave_the_rule_on(ctx):
    first = ctx.get_tuning()
    assert first["automatic"] == 1
    ctx.set_tuning(turns_per_launch=4, compact=1)
    assert ctx.get_tuning() == dict(first, turns_per_launch=4, compact=1)
    ctx.set_tuning(stage_smem=0)
    assert ctx.get_tuning()["automatic"] == 1
    ctx.set_tuning(block=128, ctas_per_sm=4)
    assert ctx.get_tuning()["automatic"] == 0
    ctx.set_tuning(turns_per_launch=0)
    assert ctx.get_tuning()["automatic"] == 0
    ctx.set_tuning(**first)
    assert ctx.get_tuning() == first


def test_a_structure_filled_in_by_hand_pins_its_shape(ctx):
    t = lib.Tuning(256, 2, 1, 0, 0)
    lib.check(lib.load().bmadgpu_ctx_set_tuning(ctx.handle, ctypes.byref(t)))
    assert ctx.get_tuning()["automatic"] == 0


def test_autotune_pins_what_it_chose(ctx):
    import torch
    eles, p = rings.ring(20)
    lat = lib.Lattice(ctx, eles, p)
    vec = rings.matched_gaussian(eles, 2000, seed=1)
    v, beta = torch.from_numpy(vec).cuda(), torch.from_numpy(lib.HostBunch.from_vec(vec, p).beta).cuda()
    state = torch.ones(2000, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    best = lib.autotune(ctx, lat, abi.Bunch(2000, v.data_ptr(), beta.data_ptr(), None, state.data_ptr(), None, None, None))
    assert ctx.get_tuning() == dict(best, automatic=0)


@pytest.mark.parametrize("row", [4, 8])
@pytest.mark.parametrize("extra", [0, 1])
def test_sizes_at_the_edges_of_the_rule(ctx, row, extra):
    n = row * 64 * ctx.sm_count + extra
    eles, p = rings.ring(8)
    lat = lib.Lattice(ctx, eles, p)
    vec = rings.matched_gaussian(eles, n, seed=5, scale=3.0)
    vec[0, ::9] += 0.025
    got, want = lib.HostBunch.from_vec(vec, p), lib.HostBunch.from_vec(vec, p)
    lib.track_bunch(ctx, lat, got, n_turns=2)
    ctx.set_tuning(block=128, ctas_per_sm=4)
    lib.track_bunch(ctx, lat, want, n_turns=2)
    assert np.any(want.state != abi.ALIVE)
    for k in ("vec", "beta", "state", "ix_ele", "ix_turn", "location"):
        assert np.array_equal(getattr(got, k), getattr(want, k)), k
