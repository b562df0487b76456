"""Which element order a lattice tracks in (default build): the forms of csrc/fastmaps.cuh up to a third of
elements without one, above it the reference's, seen in the bits of a tracked orbit against the one-turn
matrix's, which is always tracked in the reference's order."""
import importlib

import numpy as np
import pytest

from conftest import load_abi

pytestmark = pytest.mark.gpu
lib = importlib.import_module("bmad-ecosystem_b200.lib")
rings = importlib.import_module("bmad-ecosystem_b200.rings")
abi = load_abi()


@pytest.mark.parametrize("thin,reference", [(80, False), (89, False), (94, True), (120, True), (150, True)])
def test_order_by_the_share_of_elements_without_a_form(thin, reference):
    ctx = lib.Context(0)
    eles, p = rings.ring(20)          # 180 elements with a form and a cavity without one
    out = []
    for i, e in enumerate(eles):
        out.append(e)
        if i < thin:
            out.append(abi.default_element(abi.AB_MULTIPOLE, b_pole={2: 1e-3}))
    share = (thin + 1) / len(out)
    assert (share > 1 / 3) == reference
    rings.set_ref_time(out, p)
    lat = lib.Lattice(ctx, out, p)
    orbits = rings.matched_gaussian(eles, 16, seed=3).T
    equal = []
    for orbit in orbits:
        _, end = lib.one_turn_matrix(ctx, lat, orbit)
        b = lib.HostBunch.from_vec(orbit[:, None], p)
        lib.track_bunch(ctx, lat, b, n_turns=1)
        equal.append(np.array_equal(b.vec[:, 0], end))
    assert all(equal) if reference else not any(equal)
    lat.close()
    ctx.close()
