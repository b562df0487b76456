"""bmadgpu_one_turn_matrix gives the same matrix whether or not the orbit after the turn is asked for."""
import ctypes
import importlib

import numpy as np
import pytest

from conftest import load_abi

pytestmark = pytest.mark.gpu
lib = importlib.import_module("bmad-ecosystem_b200.lib")
rings = importlib.import_module("bmad-ecosystem_b200.rings")
abi = load_abi()


@pytest.mark.parametrize("rf_on", [True, False])
def test_matrix_does_not_depend_on_the_outputs_asked_for(rf_on):
    ctx = lib.Context(0)
    lat = lib.Lattice(ctx, *rings.perturbed_ring(30, seed=2))
    orbit = np.array([1e-4, -2e-5, 5e-5, 1e-5, 1e-4, 2e-4])
    with_end, _ = lib.one_turn_matrix(ctx, lat, orbit, rf_on=rf_on)
    mat = np.zeros(36)
    D = ctypes.POINTER(ctypes.c_double)
    lib.check(lib.load().bmadgpu_one_turn_matrix(ctx.handle, lat.handle, orbit.ctypes.data_as(D), int(rf_on), None,
                                                 mat.ctypes.data_as(D)))
    assert np.array_equal(mat.reshape(6, 6), with_end)
    lat.close()
    ctx.close()
