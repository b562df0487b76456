"""The correctly rounded build's tables hold no entries that only the default build's element forms read
(its kernels stage them in shared memory, where their size costs resident CTAs): 16-byte headers, a bend of
26 entries, no frame block beside the pitched misalignment."""
import ctypes
import importlib

import pytest

from conftest import load_abi

lib = importlib.import_module("bmad-ecosystem_b200.lib")
rings = importlib.import_module("bmad-ecosystem_b200.rings")
abi = load_abi()


def table_bytes(math, eles, p):
    lib.set_math(math)
    try:
        arr, out = abi.element_array(eles), ctypes.c_int64()
        lib.check(lib.load().bmadgpu_lattice_check(arr, len(arr), ctypes.byref(p), None, ctypes.byref(out)))
        return out.value
    finally:
        lib.set_math("fast")


E = abi.default_element


@pytest.mark.parametrize("ele,fewer", [
    (E(abi.DRIFT, l=1.0), 16),
    (E(abi.QUADRUPOLE, l=0.4, k1=0.8, x_offset=1e-4), 16),
    (E(abi.SBEND, l=1.5, g=0.04), 16 + 8 * 20),
    (E(abi.QUADRUPOLE, l=0.4, k1=0.8, x_pitch=1e-3), 16 + 8 * 36),
])
def test_one_element(ele, fewer):
    p = abi.electron_param(3e9)
    assert table_bytes("cr", [ele], p) == table_bytes("fast", [ele], p) - fewer


def test_ring():
    eles, p = rings.perturbed_ring(200, seed=1)
    assert table_bytes("cr", eles, p) <= table_bytes("fast", eles, p) - 16 * len(eles)
