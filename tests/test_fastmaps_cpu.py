"""The element forms of the default build (csrc/fastmaps.cuh), compiled for the host, against the same
maps in quadruple precision (csrc/hostcheck_quad.cpp) and against the reference's operand order.

A form may not be further from the quadruple-precision map than the reference's order is (rms over the
bunch, per coordinate): the comparison allows a quarter more plus one unit in the last place of the
coordinate's rms, 2^-52, which covers the statistics of a thousand particles and coordinates that are
exact in one of the two. On either side of a form's range both paths have to agree with the map."""
import ctypes
import importlib
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, load_abi
from helpers import oracle_track

abi = load_abi()
rings = importlib.import_module("bmad-ecosystem_b200.rings")
ULP = 2.0 ** -52


def _lib(name):
    path = os.path.join(ROOT, "bmad-ecosystem_b200", "_build", name)
    if not os.path.exists(path):
        subprocess.check_call(["make", "-s", "-C", os.path.join(ROOT, "bmad-ecosystem_b200", "csrc"), "hostcheck-lib"])
    return ctypes.CDLL(path)


def _bunch(vec, p):
    n = vec.shape[1]
    pc = p.p0c * (1 + vec[5])
    beta = np.ascontiguousarray(np.where(vec[5] == 0, p.p0c / p.e_tot, pc / np.sqrt(pc * pc + p.mass ** 2)))
    d = dict(vec=np.array(vec, order="C", copy=True), beta=beta, state=np.ones(n, np.int32),
             ix_ele=np.full(n, -1, np.int32), ix_turn=np.full(n, -1, np.int32), location=np.zeros(n, np.int32))
    return d, abi.Bunch(n, d["vec"].ctypes.data, beta.ctypes.data, None, d["state"].ctypes.data,
                        d["ix_ele"].ctypes.data, d["ix_turn"].ctypes.data, d["location"].ctypes.data)


def fast(eles, p, vec, turns=1):
    d, b = _bunch(vec, p)
    arr = abi.element_array(eles)
    assert _lib("libbmadgpu_hostcheck_fast.so").bmadgpu_hostcheck_fast_track(
        arr, len(arr), ctypes.byref(p), ctypes.byref(b), turns) == 0
    return d


def quad(eles, p, vec, turns=1):
    _, b = _bunch(vec, p)
    arr = abi.element_array(eles)
    hi, lo = np.zeros_like(vec), np.zeros_like(vec)
    P = ctypes.c_void_p
    assert _lib("libbmadgpu_hostquad.so").bmadgpu_hostcheck_quad_track(
        arr, len(arr), ctypes.byref(p), ctypes.byref(b), turns, hi.ctypes.data_as(P), lo.ctypes.data_as(P)) == 0
    return hi, lo


def compare(eles, p, vec, turns=1):
    f, o = fast(eles, p, vec, turns), oracle_track(eles, p, vec, turns)
    for k in ("state", "ix_ele", "ix_turn", "location"):
        assert np.array_equal(f[k], o[k]), k
    hi, lo = quad(eles, p, vec, turns)
    m = o["state"] == abi.ALIVE
    rms = np.maximum(np.sqrt(np.mean(hi[:, m] ** 2, axis=1)), 1e-300)

    def err(r):
        return np.sqrt(np.mean(((r["vec"][:, m] - hi[:, m]) - lo[:, m]) ** 2, axis=1)) / rms

    ef, eo = err(f), err(o)
    assert np.all(ef <= 1.25 * eo + ULP), (ef, eo)
    return ef, eo


AP = dict(x1_limit=0.02, x2_limit=0.02, y1_limit=0.01, y2_limit=0.01)
E = abi.default_element
ELEMENTS = {
    "drift": E(abi.DRIFT, l=2.5, **AP),
    "drift_entrance": E(abi.DRIFT, l=2.5, aperture_at=abi.BOTH_ENDS, **AP),
    "elliptical": E(abi.DRIFT, l=1.0, aperture_type=abi.APERTURE_ELLIPTICAL, x1_limit=0.004, x2_limit=0.006,
                    y1_limit=0.002, y2_limit=0.003),
    "quad_f": E(abi.QUADRUPOLE, l=0.4, k1=0.8, **AP),
    "quad_d": E(abi.QUADRUPOLE, l=0.4, k1=-0.8, x_offset=3e-5, y_offset=-2e-5, tilt=1e-2, **AP),
    "quad_zero": E(abi.QUADRUPOLE, l=0.4, k1=0.0, **AP),
    "quad_multipoles": E(abi.QUADRUPOLE, l=0.4, k1=0.8, b_pole={2: 1e-3, 3: -2e-4}, a_pole={2: 5e-4}, **AP),
    "sextupole": E(abi.SEXTUPOLE, l=0.2, k2=12.0, **AP),
    "sextupole_steps": E(abi.SEXTUPOLE, l=0.2, k2=12.0, x_offset=5e-5, tilt=-1e-2, num_steps=4, **AP),
    "octupole": E(abi.OCTUPOLE, l=0.3, k3=200.0, **AP),
    "kicker": E(abi.KICKER, l=0.3, hkick=1e-5, vkick=2e-5, b_pole={0: 0.2, 1: 3.0}, num_steps=3, tilt=-0.05, **AP),
    "monitor": E(abi.MONITOR, l=0.2, x_offset=1e-4, **AP),
    "bend": E(abi.SBEND, l=1.5, g=2 * np.pi / 100 / 1.5, fringe_type=abi.FRINGE_NONE, **AP),
    "bend_fringe": E(abi.SBEND, l=1.5, g=-2 * np.pi / 100 / 1.5, **AP),
    "bend_one_edge": E(abi.SBEND, l=1.0, g=0.05, fringe_at=abi.EXIT_END, ref_tilt=0.3, **AP),
    "bend_edges": E(abi.SBEND, l=1.0, g=0.05, e1=0.03, e2=-0.02, fint=0.5, hgap=0.02, **AP),
    "bend_dg": E(abi.SBEND, l=1.0, g=0.05, dg=2e-3, **AP),
    "bend_large": E(abi.SBEND, l=1.0, g=0.95, **AP),
    "bend_too_large": E(abi.SBEND, l=1.0, g=1.3, **AP),
    "quad_pitched": E(abi.QUADRUPOLE, l=0.4, k1=-0.8, x_pitch=-2e-3, y_pitch=1e-3, z_offset=-0.01, y_offset=1e-4,
                      tilt=0.1, **AP),
    "sextupole_pitched": E(abi.SEXTUPOLE, l=0.6, k2=1.0, tilt=0.52, num_steps=10, x_offset=2e-3, y_pitch=1e-3,
                           z_offset=0.02, **AP),
    "bend_offsets": E(abi.SBEND, l=1.0, g=0.03, e1=0.02, x_offset=1e-3, y_offset=-5e-4, x_pitch=2e-4, y_pitch=-1e-4,
                      z_offset=0.01, roll=-0.01, ref_tilt=0.2, **AP),
}
ELEMENTS.update({"multipoles_%d" % n: E(abi.SEXTUPOLE, l=0.2, k2=-18.0, b_pole={k: 3.0 * (-7) ** k for k in range(3, n)},
                                        **AP) for n in range(4, 14)})


@pytest.mark.parametrize("name", sorted(ELEMENTS))
def test_element_forms_are_as_close_as_the_reference_order(name):
    eles = [ELEMENTS[name]]
    p = abi.electron_param(3e9)
    rings.set_ref_time(eles, p)
    compare(eles, p, rings.matched_gaussian(rings.ring(50)[0], 1000, seed=11, scale=3.0))


@pytest.mark.parametrize("ring", ["plain", "multipoles", "perturbed"])
def test_rings_are_as_close_as_the_reference_order(ring):
    eles, p = {"plain": lambda: rings.ring(50), "perturbed": lambda: rings.perturbed_ring(50, seed=3),
               "multipoles": lambda: rings.ring(100, fringe=True, multipole_sigma=1e-4)}[ring]()
    compare(eles, p, rings.matched_gaussian(rings.ring(50)[0], 300, seed=5, scale=3.0))


# (element, coordinate swept, values across the edge of the form's range)
EDGES = {
    "px_2^-6": ("drift", 1, (1 + np.linspace(-1e-3, 1e-3, 41)) * 2.0 ** -6),          # (px^2 + py^2)/rel^2 = 2^-12
    "px_bend": ("bend", 1, (1 + np.linspace(-1e-2, 1e-2, 41)) * 2.0 ** -6),
    "pz_quarter": ("bend", 5, np.linspace(0.2499, 0.2501, 41)),
    "pz_minus": ("quad_f", 5, np.linspace(-0.2501, -0.2499, 41)),
    "x_bend": ("bend_large", 0, np.linspace(1e-3, 4e-3, 41)),                           # L_c^2/L_c0^2 - 1 = 2^-8
    "orbit_1e-9": ("bend", 1, np.linspace(0.9e-9, 1.1e-9, 41)),
    "x_aperture": ("drift", 0, np.linspace(0.0199, 0.0201, 41)),
}


@pytest.mark.parametrize("name", sorted(EDGES))
def test_edges_of_the_ranges(name):
    ele, i, values = EDGES[name]
    eles = [ELEMENTS[ele]]
    p = abi.electron_param(3e9)
    rings.set_ref_time(eles, p)
    vec = np.zeros((6, len(values)))
    vec[i] = values
    f, o = fast(eles, p, vec), oracle_track(eles, p, vec, 1)
    for k in ("state", "ix_ele", "location"):
        assert np.array_equal(f[k], o[k]), k
    hi, lo = quad(eles, p, vec)
    m = o["state"] == abi.ALIVE
    # either path: a few rounding errors of the largest term a coordinate is made of (the length, or the
    # bend's sagitta), as the reference's order itself
    scale = np.maximum(np.abs(hi[:, m]), 0.1)
    assert np.all(np.abs((f["vec"][:, m] - hi[:, m]) - lo[:, m]) <= 16 * ULP * scale)


@pytest.mark.parametrize("k1", [3.0, 3.1, 3.125, 3.2, -3.1, -3.2, 40.0])
def test_strong_quadrupoles(k1):
    """|k| step^2 across 1/2 (l = 0.4: k1 = 3.125), where the series gives way to the libm's functions."""
    eles = [E(abi.QUADRUPOLE, l=0.4, k1=k1)]
    p = abi.electron_param(3e9)
    rings.set_ref_time(eles, p)
    compare(eles, p, rings.matched_gaussian(rings.ring(50)[0], 1000, seed=2))
