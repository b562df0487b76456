"""The default build's element forms on the GPU at the edges of their ranges, the core selection and the
turn-parallel adjoint at the sizes where their kernels' tiles end.

Tolerances: an element's coordinates within 16 units in the last place of the largest term they are made
of (tests/test_fastmaps_cpu.py); a selection exactly numpy's stable order; the gradient as close to the
host build's as at larger sizes (1e-8 of a family's largest component, tests/test_adjoint_gpu.py)."""
import importlib

import numpy as np
import pytest

from conftest import load_abi
from helpers import oracle_track
from test_fastmaps_cpu import EDGES, ELEMENTS, ULP

pytestmark = pytest.mark.gpu
lib = importlib.import_module("bmad-ecosystem_b200.lib")
rings = importlib.import_module("bmad-ecosystem_b200.rings")
abi = load_abi()


@pytest.fixture(scope="module")
def ctx():
    c = lib.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("name", sorted(EDGES))
def test_edges_of_the_ranges(ctx, name):
    ele, i, values = EDGES[name]
    eles = [ELEMENTS[ele]]
    p = abi.electron_param(3e9)
    rings.set_ref_time(eles, p)
    vec = np.zeros((6, len(values)))
    vec[i] = values
    b = lib.HostBunch.from_vec(vec, p)
    lib.track_bunch(ctx, lib.Lattice(ctx, eles, p), b, n_turns=1)
    o = oracle_track(eles, p, vec, 1)
    for k in ("state", "ix_ele", "location"):
        assert np.array_equal(getattr(b, k), o[k]), k
    m = o["state"] == abi.ALIVE
    # the oracle is itself within the same distance of the map
    assert np.all(np.abs(b.vec[:, m] - o["vec"][:, m]) <= 32 * ULP * np.maximum(np.abs(o["vec"][:, m]), 0.1))


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 1024, 1025, 100003])
def test_core_selection_sizes(ctx, n):
    import torch
    rng = np.random.default_rng(n)
    keys = rng.exponential(2.0, n)
    keys[rng.random(n) < 0.3] = 1.5          # ties
    keys[rng.random(n) < 0.1] = 1e100        # dead
    order = np.argsort(keys, kind="stable")
    for n_cut in sorted({1, max(1, n // 3), max(1, n // 2), n}):
        got = lib.select_smallest(ctx, torch.from_numpy(keys).cuda(), n_cut)
        if keys[order[n_cut - 1]] > 1e99:
            assert got is None
            continue
        want = np.zeros(n, np.int32)
        want[order[:n_cut]] = abi.ALIVE
        assert np.array_equal(got, want), n_cut


@pytest.mark.parametrize("n,turns", [(1, 1), (1, 3), (33, 2), (129, 5)])
def test_adjoint_sizes(ctx, n, turns):
    from test_adjoint_cpu import host_loss_grad, ring_params
    from test_adjoint_gpu import _load_ha, gpu_loss_grad
    eles, p = rings.ring(50)
    vec = rings.matched_gaussian(eles, n, seed=9)
    _, names = ring_params(eles)
    loss_g, grad_g = gpu_loss_grad(ctx, eles, p, vec, turns, 2, [i for i, _ in names])
    loss_h, grad_h, _, _ = host_loss_grad(_load_ha(), eles, p, vec, turns, 2)
    assert abs(loss_g - loss_h) <= 1e-10 * abs(loss_h)
    quads = np.array([k == "k1" for _, k in names])
    for fam in (quads, ~quads):
        assert np.max(np.abs(grad_g[fam] - grad_h[fam])) <= 1e-8 * np.max(np.abs(grad_h[fam]))
