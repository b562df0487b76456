"""Elements of negative and zero length through the element forms of the default build (csrc/fastmaps.cuh),
compiled for the host, against the oracle and, for the straight ones, the maps in quadruple precision.

Tolerances: compare() of test_fastmaps_cpu.py, a form no further from the quadruple-precision map than the
reference's order is; where a bend has no form the two orders are the same code up to the tilt, so a
coordinate is within 16 units in the last place of the largest term it is made of, as at the edges of the
ranges there (the arc of a bend of negative length is (2 pi - angle)/g, up to 126 m here)."""
import numpy as np
import pytest

from conftest import load_abi
from helpers import oracle_track
from test_fastmaps_cpu import AP, E, ULP, compare, fast, rings

abi = load_abi()

STRAIGHT = {
    "drift": dict(key=abi.DRIFT),
    "quad_f": dict(key=abi.QUADRUPOLE, k1=0.8),
    "quad_d_misaligned": dict(key=abi.QUADRUPOLE, k1=-0.8, x_offset=3e-5, y_offset=-2e-5, tilt=1e-2),
    "sextupole": dict(key=abi.SEXTUPOLE, k2=12.0),
    "sextupole_steps": dict(key=abi.SEXTUPOLE, k2=12.0, num_steps=3),
    "quad_pitched": dict(key=abi.QUADRUPOLE, k1=0.8, x_pitch=1e-3, y_pitch=-5e-4),
}


@pytest.mark.parametrize("length", [-0.4, 0.0])
@pytest.mark.parametrize("name", sorted(STRAIGHT))
def test_straight_elements(name, length):
    eles = [E(l=length, **STRAIGHT[name], **AP)]
    p = abi.electron_param(3e9)
    rings.set_ref_time(eles, p)
    compare(eles, p, rings.matched_gaussian(rings.ring(50)[0], 1000, seed=4, scale=3.0))


BENDS = {
    "sector": dict(g=0.05, fringe_type=abi.FRINGE_NONE),
    "sector_negative_g": dict(g=-0.05, fringe_type=abi.FRINGE_NONE),
    "fringes": dict(g=0.05),
    "edges": dict(g=0.05, e1=0.03, e2=-0.02, fint=0.5, hgap=0.02),
    "one_edge": dict(g=0.05, fringe_at=abi.EXIT_END, ref_tilt=0.3),
    "dg": dict(g=0.05, dg=2e-3),
    "offsets": dict(g=0.03, x_offset=1e-3, y_offset=-5e-4, roll=-0.01, fringe_type=abi.FRINGE_NONE),
}


@pytest.mark.parametrize("length", [-1.0, -0.2])
@pytest.mark.parametrize("name", sorted(BENDS))
def test_bends_of_negative_length(name, length):
    eles = [E(abi.SBEND, l=length, **BENDS[name])]
    p = abi.electron_param(3e9)
    rings.set_ref_time(eles, p)
    vec = rings.matched_gaussian(rings.ring(50)[0], 500, seed=8, scale=3.0)
    vec[1, :3] = 0.0155, 0.0157, 0.03        # either side of the momentum series' range
    f, o = fast(eles, p, vec), oracle_track(eles, p, vec, 1)
    for k in ("state", "ix_ele", "location"):
        assert np.array_equal(f[k], o[k]), k
    m = o["state"] == abi.ALIVE
    scale = np.maximum(np.max(np.abs(o["vec"][:, m]), axis=0), 0.1)
    assert np.all(np.abs(f["vec"][:, m] - o["vec"][:, m]) <= 16 * ULP * scale)
