"""The work that performance is measured on: one entry per way this framework is used, through its
public entry points, from a per-element call on a few hundred particles to a million particles around
a 1801-element ring, and the draws that spread over the ranges between.

Rings, beams and sizes are those of the repository's own workloads (rings.py, bench.py): FODO rings of
50 to 200 cells, matched Gaussian bunches, dynamic-aperture and frequency-map grids. Turn counts are a
few turns of one launch, not the thousands of a long run: the time of a run is proportional to them,
and over many turns the rounding of any two correct programs drifts apart.
"""
import ctypes
import importlib
import math

import numpy as np
import torch
import torch.utils.checkpoint

abi = importlib.import_module("bmad-ecosystem_b200.abi")
lib = importlib.import_module("bmad-ecosystem_b200.lib")
rings = importlib.import_module("bmad-ecosystem_b200.rings")

HOOK_ELEMENTS = {"drift": 0, "quadrupole": 1, "sbend": 3, "sextupole": 5}  # index in the FODO cell


def listed():
    return [
        # The track1_bunch hook of an unmodified Bmad program: one element, host arrays, a small bunch.
        {"name": "hook_quadrupole", "kind": "hook", "ring": "plain", "cells": 50, "element": "quadrupole", "n": 1000},
        # Set-up of every long-term run: closed orbit, one-turn matrices and periodic Twiss.
        {"name": "optics_50", "kind": "optics", "ring": "perturbed", "cells": 50},
        # The small benchmark ring: 10,000 particles, host arrays in and out.
        {"name": "ltt_50_10k", "kind": "track_host", "ring": "plain", "cells": 50, "n": 10000, "turns": 10,
         "scale": 1.0, "moments": False},
        # The same with the per-turn moment sums of long-term tracking, 100,000 particles.
        {"name": "ltt_50_moments", "kind": "track_host", "ring": "plain", "cells": 50, "n": 100000, "turns": 8,
         "scale": 3.0, "moments": True},
        # The 1801-element ring with sextupole multipoles and bend fringes, an odd particle count that
        # fills the chip once or twice, on the device.
        {"name": "track_200_50k", "kind": "track_device", "ring": "multipole", "cells": 200, "n": 50021, "turns": 4,
         "scale": 3.0},
        # The large benchmark ring at its full particle count.
        {"name": "track_200_1m", "kind": "track_device", "ring": "multipole", "cells": 200, "n": 1048576, "turns": 4,
         "scale": 3.0},
        # A ring with pitched quadrupoles and misaligned bends (the kernels for every element form).
        {"name": "track_50_pitched", "kind": "track_device", "ring": "pitched", "cells": 50, "n": 65536, "turns": 6,
         "scale": 3.0},
        # Dynamic-aperture grids of many perturbed rings in one launch, uneven particle counts.
        {"name": "batch_24", "kind": "batch", "ring": "perturbed", "cells": 50, "variants": 24, "n_min": 1024,
         "n_max": 16384, "turns": 8},
        # A burst of requests of mixed rings, sizes and turn counts through the server.
        {"name": "serve_8", "kind": "serve", "ring": "perturbed", "cells": 100, "jobs": 8, "n_min": 256,
         "n_max": 32768, "turns": 16},
        # Gradient of the tracking loss with respect to every quadrupole and sextupole strength.
        {"name": "grad_50_4k", "kind": "grad", "ring": "plain", "cells": 50, "n": 4096, "turns": 32, "every": 16},
        # A frequency map of a grid of starting amplitudes.
        {"name": "fma_50_1k", "kind": "fma", "ring": "perturbed", "cells": 50, "n": 1024, "turns": 128},
        # Bunch statistics and core emittances of a large bunch, as the averages output takes them.
        {"name": "stats_1m", "kind": "stats", "ring": "plain", "cells": 50, "n": 1000000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["hook", "optics", "track_host", "track_host", "track_device", "track_device", "track_device",
                       "batch", "serve", "grad", "fma", "stats"])
    if kind == "hook":
        return {"kind": kind, "ring": "plain", "cells": 50, "element": rng.choice(sorted(HOOK_ELEMENTS)),
                "n": _log(rng, 100, 100000)}
    if kind == "optics":
        ring = rng.choice(["plain", "perturbed", "multipole"])  # offsets on more cells can leave no closed orbit
        return {"kind": kind, "ring": ring, "cells": 50 if ring == "perturbed" else rng.randint(50, 200)}
    if kind == "track_host":
        return {"kind": kind, "ring": rng.choice(["plain", "multipole", "perturbed"]), "cells": rng.randint(50, 100),
                "n": _log(rng, 200, 200000), "turns": rng.randint(1, 10), "scale": rng.choice([1.0, 3.0]),
                "moments": rng.random() < 0.5}
    if kind == "track_device":
        return {"kind": kind, "ring": rng.choice(["plain", "multipole", "perturbed", "pitched"]),
                "cells": rng.randint(50, 200), "n": _log(rng, 1000, 500000), "turns": rng.randint(1, 6),
                "scale": rng.choice([1.0, 3.0])}
    if kind == "batch":
        return {"kind": kind, "ring": "perturbed", "cells": 50, "variants": rng.randint(3, 32), "n_min": 1024,
                "n_max": _log(rng, 2048, 32768), "turns": rng.randint(2, 8)}
    if kind == "serve":
        return {"kind": kind, "ring": "perturbed", "cells": rng.randint(50, 200), "jobs": rng.randint(2, 10),
                "n_min": 256, "n_max": _log(rng, 1024, 32768), "turns": rng.randint(4, 16)}
    if kind == "grad":
        return {"kind": kind, "ring": "plain", "cells": rng.randint(50, 80), "n": _log(rng, 200, 8192),
                "turns": rng.randint(2, 32), "every": rng.choice([4, 8, 16])}
    if kind == "fma":
        return {"kind": kind, "ring": "perturbed", "cells": 50, "n": _log(rng, 100, 4000),
                "turns": rng.choice([64, 96, 100, 128])}
    return {"kind": kind, "ring": "plain", "cells": 50, "n": _log(rng, 1000, 2000000)}


# ---- inputs ---------------------------------------------------------------------------------------

def _ring(case, seed):
    """(elements, param) of the case's ring."""
    kind, cells = case["ring"], case["cells"]
    if kind == "plain":
        return rings.ring(cells)
    if kind == "multipole":
        return rings.ring(cells, fringe=True, multipole_sigma=1e-4, multipole_seed=seed)
    eles, p = rings.perturbed_ring(cells, seed=seed)
    if kind == "pitched":
        rng = np.random.default_rng(seed + 1)
        for e in eles:
            if e.key == abi.QUADRUPOLE:
                e.x_pitch, e.y_pitch = rng.normal(0.0, 1e-4, 2)
                e.z_offset = rng.normal(0.0, 1e-4)
            elif e.key == abi.SBEND:
                e.x_offset, e.y_offset = rng.normal(0.0, 50e-6, 2)
    return eles, p


def _bunch(case, seed, eles, n):
    return rings.matched_gaussian(rings.ring(case["cells"])[0], n, seed=seed, scale=case.get("scale", 1.0))


def _beta(vec, p):
    return lib.HostBunch.from_vec(vec, p).beta


def _jobs(case, seed):
    """[(elements, param, vec)] of the variants of a batch or the requests of a serving burst."""
    count = case.get("variants", case.get("jobs"))
    size, rng = np.random.default_rng(case["n_max"] + count), np.random.default_rng(seed)  # sizes: the case's own
    out = []
    for k in range(count):
        n = int(round(math.exp(size.uniform(math.log(case["n_min"]), math.log(case["n_max"])))))
        cells = case["cells"] if case["kind"] == "batch" or k % 2 else 50
        eles, p = rings.perturbed_ring(cells, seed=int(rng.integers(1 << 30)))
        if case["kind"] == "batch":
            vec = rings.da_grid(n, r_max=0.005 + 0.001 * rng.random())
        else:
            vec = rings.matched_gaussian(rings.ring(cells)[0], n, seed=int(rng.integers(1 << 30)))
        out.append((eles, p, vec))
    return out


def _job_turns(case, k):
    return max(1, case["turns"] - 3 * (k % 4))


def _strength_elements(eles):
    return [i for i, e in enumerate(eles) if e.key in (abi.QUADRUPOLE, abi.SEXTUPOLE)]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind, "ctx": lib.Context(0)}
    if kind in ("batch", "serve"):
        jobs = _jobs(case, seed)
        lats = [lib.Lattice(s["ctx"], e, p) for e, p, _ in jobs]
        if kind == "batch":
            s["batch"] = lib.Batch(s["ctx"], lats, [v.shape[1] for _, _, v in jobs])
            s["start"] = lib.concat_bunches([lib.HostBunch.from_vec(v, p) for _, p, v in jobs])
            s["bunch"] = lib.concat_bunches([lib.HostBunch.from_vec(v, p) for _, p, v in jobs])
        else:
            s["server"] = lib.Server(s["ctx"], max_particles=1 << 20, record_mib=64)
            s["lats"], s["vecs"] = lats, [v for _, _, v in jobs]
            s["betas"] = [_beta(v, p) for _, p, v in jobs]
            s["bunches"] = [lib.PinnedBunch(v, b) for v, b in zip(s["vecs"], s["betas"])]
        return s
    eles, p = _ring(case, seed)
    s["param"] = p
    s["lat"] = lib.Lattice(s["ctx"], eles, p)
    n = case.get("n", 0)
    if kind == "hook":
        s["vec"] = _bunch(dict(case, scale=3.0), seed, eles, n)
        s["beta"] = _beta(s["vec"], p)
    elif kind in ("track_host", "grad"):
        s["vec"] = _bunch(case, seed, eles, n)
        s["beta"] = _beta(s["vec"], p)
        if kind == "grad":
            s["param_ele"] = _strength_elements(eles)
            s["bunch"] = lib.HostBunch(s["vec"], s["beta"])
    elif kind in ("track_device", "stats"):
        vec = _bunch(case, seed, eles, n)
        s["stream"] = torch.cuda.ExternalStream(s["ctx"].stream)
        s["vec"] = torch.from_numpy(vec).cuda()
        s["beta"] = torch.from_numpy(_beta(vec, p)).cuda()
        if kind == "stats":
            s["t"] = torch.from_numpy(np.random.default_rng(seed).normal(0.0, 1e-11, n)).cuda()
            s["state"] = torch.ones(n, dtype=torch.int32, device="cuda")
            s["state"][seed % 7::17] = abi.LOST_POS_X
    elif kind == "fma":
        s["offsets"] = _fma_offsets(case, seed)
        s["setup"] = lib.fma_setup(s["ctx"], s["lat"])
    return s


def _fma_offsets(case, seed):
    off = rings.fma_grid(case["n"], x_max=0.003, y_max=0.0015).T.copy()
    return off * (0.9 + 0.1 * np.random.default_rng(seed).random())


# ---- one pass -------------------------------------------------------------------------------------

def _arrays(b):
    return {"vec": b.vec, "beta": b.beta, "state": b.state, "ix_ele": b.ix_ele, "ix_turn": b.ix_turn,
            "location": b.location}


def run(s):
    case, kind, ctx = s["case"], s["kind"], s["ctx"]
    if kind == "hook":
        b = lib.HostBunch(s["vec"], s["beta"])
        lib.track1_bunch(ctx, s["lat"], b, HOOK_ELEMENTS[case["element"]])
        return _arrays(b)
    if kind == "optics":
        orbit, mat, _ = lib.closed_orbit(ctx, s["lat"])
        mat_off, end = lib.one_turn_matrix(ctx, s["lat"], orbit, rf_on=False)
        tw = lib.twiss_from_mat6(mat_off, orbit)
        return {"orbit": orbit, "mat": mat, "mat_off": mat_off, "end": end,
                "twiss": np.array([tw[k] for k in ("beta_a", "alpha_a", "phi_a", "beta_b", "alpha_b", "phi_b",
                                                   "eta_x", "etap_x")])}
    if kind == "track_host":
        b = lib.HostBunch(s["vec"], s["beta"])
        mom = lib.track_bunch(ctx, s["lat"], b, n_turns=case["turns"], moments=case["moments"])
        out = _arrays(b)
        if case["moments"]:
            out["moments"] = mom
        return out
    if kind == "track_device":
        with torch.cuda.stream(s["stream"]):
            vec, beta = s["vec"].clone(), s["beta"].clone()
            n = beta.numel()
            state = torch.ones(n, dtype=torch.int32, device="cuda")
            ix_ele, ix_turn = torch.full_like(state, -1), torch.full_like(state, -1)
            location = torch.zeros_like(state)
            view = abi.Bunch(n, vec.data_ptr(), beta.data_ptr(), None, state.data_ptr(), ix_ele.data_ptr(),
                             ix_turn.data_ptr(), location.data_ptr())
            lib.check(lib.load().bmadgpu_track_bunch_device(ctx.handle, s["lat"].handle, ctypes.byref(view), 0,
                                                            s["lat"].n_ele, 0, case["turns"], None))
        return {"vec": vec, "beta": beta, "state": state, "ix_ele": ix_ele, "ix_turn": ix_turn, "location": location}
    if kind == "batch":
        s["batch"].upload(-1, s["start"])
        s["batch"].track(case["turns"])
        s["batch"].download(-1, s["bunch"])
        return _arrays(s["bunch"])
    if kind == "serve":
        ids = []
        for k, b in enumerate(s["bunches"]):
            b.vec[:], b.beta[:], b.state[:] = s["vecs"][k], s["betas"][k], abi.ALIVE
            b.ix_ele[:], b.ix_turn[:], b.location[:] = -1, -1, 0
            ids.append(s["server"].submit(s["lats"][k], b, _job_turns(case, k)))
        for i in ids:
            s["server"].wait(i)
        return {"vec": np.concatenate([b.vec for b in s["bunches"]], axis=1),
                "beta": np.concatenate([b.beta for b in s["bunches"]]),
                "state": np.concatenate([b.state for b in s["bunches"]])}
    if kind == "grad":
        loss, grad = lib.loss_grad(ctx, s["lat"], s["bunch"], case["turns"], s["param_ele"], case["every"])
        return {"loss": loss, "grad": grad}
    if kind == "fma":
        orbit, norm, tunes = s["setup"]
        q, status, turn_lost, ix_ele = lib.fma(ctx, s["lat"], s["offsets"], case["turns"], orbit=orbit, norm=norm,
                                               tunes=tunes)
        return {"tunes": q[:, [0, 1, 3, 4]], "status": status, "turn_lost": turn_lost, "ix_ele": ix_ele}
    view = abi.Bunch(s["beta"].numel(), s["vec"].data_ptr(), s["beta"].data_ptr(), s["t"].data_ptr(),
                     s["state"].data_ptr(), None, None, None)
    bd = lib.bunch_stats(ctx, s["lat"], view)
    core = lib.bunch_core_emit(ctx, s["lat"], view)
    return {"n_live": int(bd["n_live"]), "centroid": bd["centroid"], "sigma": bd["sigma"], "skew": bd["skew"],
            "kurt": bd["kurt"], "emit": bd["emit"], "core_emit": core}


# ---- what one pass cannot do without --------------------------------------------------------------

# FP64 operations of one particle through one element of each ring (an operation is one addition,
# multiplication, division, root or transcendental call of the maps), from the operation-counting
# host build: 50-cell rings 65, with multipoles and fringes 219; offsets and tilts add about 8.
OPS = {"plain": 65.0, "perturbed": 73.0, "multipole": 219.0, "pitched": 110.0}
STATE_BYTES = 2 * (7 * 8 + 4 * 4)  # a particle's coordinates, beta and loss record, in and out


def work(case):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        count = case.get("variants", case.get("jobs"))
        mean = (case["n_max"] - case["n_min"]) / math.log(case["n_max"] / case["n_min"])
        cells = case["cells"] if kind == "batch" else 0.5 * (case["cells"] + 50)
        turns = case["turns"] if kind == "batch" else sum(_job_turns(case, k) for k in range(count)) / count
        n = count * mean
        return {"bytes": n * STATE_BYTES, "flops": n * turns * 9 * cells * OPS["perturbed"]}
    ops = OPS[case["ring"]]
    n_ele = 9 * case["cells"] + 1
    n = case.get("n", 0)
    if kind == "hook":
        return {"bytes": n * STATE_BYTES, "flops": n * ops}
    if kind == "optics":
        return {"bytes": 25.0 * STATE_BYTES, "flops": 25.0 * 4 * n_ele * ops}
    if kind == "grad":
        # the turns forward once and the reverse sweep's own forward and adjoint operations
        return {"bytes": n * STATE_BYTES, "flops": 4.0 * n * case["turns"] * n_ele * ops}
    if kind == "fma":
        return {"bytes": n * (6 * 8 + 6 * 8 + 16), "flops": n * case["turns"] * n_ele * ops}
    if kind == "stats":
        # one read of the bunch; 63 sums, then the core's amplitudes (27 products) and sums
        return {"bytes": n * 60.0, "flops": n * 250.0}
    return {"bytes": n * STATE_BYTES, "flops": n * case["turns"] * n_ele * ops}


# ---- the same by plain torch in 64 bits ---------------------------------------------------------------

class _Tracker:
    """The element maps of these rings (drift, quadrupole, exact sector bend with its fringe, thin-kick
    sextupole with multipoles, RF cavity, rectangular apertures) on arrays of particles. Element values
    are numbers, or arrays with one entry per particle where particles belong to different rings."""

    def __init__(self, p):
        self.p0c, self.m, self.e0 = p.p0c, p.mass, p.e_tot
        self.b0 = p.p0c / p.e_tot

    def drift(self, v, L):
        x, px, y, py, z, pz = v
        rel = 1 + pz
        a, b = px / rel, py / rel
        ps = torch.sqrt(1 - (a * a + b * b))
        so = -(a * a + b * b) / (1 + ps)  # ps - 1
        return x + L * a / ps, px, y + L * b / ps, py, z + L * (self.dbeta(pz) + so / ps), pz

    def dbeta(self, pz):
        """beta(pz) / beta0 - 1."""
        q = self.m * self.m * (2 * pz + pz * pz) / ((self.p0c * (1 + pz)) ** 2 + self.m * self.m)
        return q / (1 + torch.sqrt(1 + q))

    def quad(self, v, k, L):
        x, px, y, py, z, pz = v
        rel = 1 + pz
        k = k / rel
        s = torch.sqrt(torch.abs(k))
        ct, st, ch, sh = torch.cos(s * L), torch.sin(s * L) / s, torch.cosh(s * L), torch.sinh(s * L) / s
        f = k > 0
        cx, sx = torch.where(f, ct, ch), torch.where(f, st, sh)
        cy, sy = torch.where(f, ch, ct), torch.where(f, sh, st)
        z = z + (-k) * (L - cx * sx) / 4 * x * x + k * sx * sx / (2 * rel) * x * px - (cx * sx + L) / (4 * rel * rel) * px * px
        z = z + k * (L - cy * sy) / 4 * y * y - k * sy * sy / (2 * rel) * y * py - (cy * sy + L) / (4 * rel * rel) * py * py
        z = z + L * self.dbeta(pz)
        return cx * x + sx / rel * px, -k * sx * rel * x + cx * px, cy * y + sy / rel * py, k * sy * rel * y + cy * py, z, pz

    def bend(self, v, g, L, fringe):
        if fringe:
            v = self.edge(v, g)
        x, px, y, py, z, pz = v
        a = g * L
        ca, sa, hs = math.cos(a), math.sin(a), math.sin(a / 2)
        sinc, cosc = sa / a, 2 * hs * hs / (a * a)
        rel = 1 + pz
        pt = torch.sqrt(rel * rel - py * py)
        gp = g / pt
        phi = torch.asin(px / pt)
        cp, sp = torch.cos(a + phi), torch.sin(a + phi)
        h = (1 + g * x) * L * sinc
        alpha = 2 * h * sp - gp * h * h
        xi = alpha / (torch.sqrt(cp * cp + gp * alpha) + cp)
        lu, lv = xi, L * sinc + x * sa
        lc = torch.sqrt(lu * lu + lv * lv)
        hp = a + phi - torch.atan2(lu, lv)
        lp = lc * hp / torch.sin(hp)
        near = torch.abs(hp) < 1e-8
        lp = torch.where(near, lc, lp)
        v = (x * ca - L * L * g * cosc + xi, pt * torch.sin(phi + a - 2 * hp), y + py * lp / pt, py,
             z + L * (1 + self.dbeta(pz)) - rel * lp / pt, pz)
        return self.edge(v, -g) if fringe else v

    def edge(self, v, g):
        """The second-order hard-edge fringe of a bend with upright faces."""
        x, px, y, py, z, pz = v
        rel = 1 + pz
        return (x + g * y * y / (2 * rel), px, y, py - g * px * y / rel, z - g * px * y * y / (2 * rel * rel), pz)

    def kick(self, v, b):
        x, px, y, py, z, pz = v
        re, im, kx, ky = torch.ones_like(x), torch.zeros_like(x), 0.0, 0.0
        for n in range(1, max(b) + 1):
            re, im = re * x - im * y, re * y + im * x
            if n in b:
                kx, ky = kx + b[n] * re, ky + b[n] * im
        return x, px - kx, y, py + ky, z, pz

    def cavity(self, v, volt, freq):
        x, px, y, py, z, pz = v
        beta = self.b0 * (1 + self.dbeta(pz))
        dE = volt * torch.sin(2 * math.pi * freq * z / (beta * abi.C_LIGHT))
        pc = (1 + pz) * self.p0c
        E = pc / beta
        q = (2 * E * dE + dE * dE) / (pc * pc)
        pz1 = pz + (1 + pz) * q / (1 + torch.sqrt(1 + q))
        return x, px, y, py, z * ((1 + pz1) * self.p0c / (E + dE)) / beta, pz1

    def element(self, v, e):
        """e: a dict of the element's kind and values."""
        if e["kind"] == "drift":
            return self.drift(v, e["l"])
        if e["kind"] == "bend":
            return self.bend(v, e["g"], e["l"], e["fringe"])
        if e["kind"] == "cavity":
            return self.cavity(v, e["voltage"], e["f"])
        mis = "tilt" in e
        if mis:
            v = (v[0] - e["dx"], v[1], v[2] - e["dy"], v[3], v[4], v[5])
            v = self.rotate(v, e["c"], e["s"])
        if e["kind"] == "quad":
            v = self.quad(v, e["k"], e["l"])
        else:
            half = {n: 0.5 * c for n, c in e["b"].items()}
            v = self.kick(self.drift(self.kick(v, half), e["l"]), half)
        if mis:
            v = self.rotate(v, e["c"], -e["s"])
            v = (v[0] + e["dx"], v[1], v[2] + e["dy"], v[3], v[4], v[5])
        return v

    @staticmethod
    def rotate(v, c, s):
        return c * v[0] + s * v[2], c * v[1] + s * v[3], -s * v[0] + c * v[2], -s * v[1] + c * v[3], v[4], v[5]

    def track(self, v, ring, turns, alive=None, after_turn=None):
        """The particles where they are after the turns, or where they left the aperture."""
        alive = torch.ones_like(v[0], dtype=torch.bool) if alive is None else alive
        for _ in range(turns):
            for e in ring:
                w = self.element(v, e)
                v = tuple(torch.where(alive, a, b) for a, b in zip(w, v))
                alive = alive & (torch.abs(v[0]) <= rings.APERTURE_X) & (torch.abs(v[2]) <= rings.APERTURE_Y)
            if after_turn:
                after_turn(v, alive)
        return v


def _values(eles, sizes=None):
    """The ring as dicts for _Tracker; eles: one element list, or one per ring with sizes particles each."""
    lists = eles if sizes else [eles]

    def val(get):
        u = [get(es) for es in lists]
        if all(a == u[0] for a in u):
            return u[0]
        return torch.cat([torch.full((n,), a, dtype=torch.float64, device="cuda") for a, n in zip(u, sizes)])

    out = []
    for i, e in enumerate(lists[0]):
        if e.key == abi.DRIFT:
            d = {"kind": "drift", "l": e.l}
        elif e.key == abi.SBEND:
            d = {"kind": "bend", "l": e.l, "g": e.g, "fringe": e.fringe_type != abi.FRINGE_NONE}
        elif e.key == abi.RFCAVITY:
            d = {"kind": "cavity", "voltage": e.voltage, "f": e.rf_frequency}
        else:
            if e.key == abi.QUADRUPOLE:
                d = {"kind": "quad", "l": e.l, "k": val(lambda es: es[i].k1)}
            else:
                b = {2: val(lambda es: es[i].k2 * es[i].l / 2 + es[i].b_pole[2] * es[i].k2 * es[i].l)}
                for n in range(3, 11):
                    if e.b_pole[n] != 0:
                        b[n] = e.b_pole[n] * e.k2 * e.l
                d = {"kind": "sext", "l": e.l, "b": b}
            if any(es[i].x_offset or es[i].y_offset or es[i].tilt for es in lists):
                d.update(tilt=True, dx=val(lambda es: es[i].x_offset), dy=val(lambda es: es[i].y_offset),
                         c=val(lambda es: math.cos(es[i].tilt)), s=val(lambda es: math.sin(es[i].tilt)))
        out.append(d)
    return out


def _coords(vec):
    return tuple(torch.from_numpy(np.ascontiguousarray(vec)).cuda().unbind(0))


def _final(t, v):
    none = {"state": None, "ix_ele": None, "ix_turn": None, "location": None}
    return {"vec": torch.stack(v), "beta": t.b0 * (1 + t.dbeta(v[5])), **none}


def exact(case, seed):
    kind = case["kind"]
    if case["ring"] == "pitched" or kind in ("optics", "fma"):
        return None
    if kind == "batch":
        jobs = _jobs(case, seed)
        t = _Tracker(jobs[0][1])
        ring = _values([e for e, _, _ in jobs], [v.shape[1] for _, _, v in jobs])
        vec = np.concatenate([v for _, _, v in jobs], axis=1)
        end = _final(t, t.track(_coords(vec), ring, case["turns"]))
        # the batch layout: each variant's [6, n] block after the one before
        cut = np.cumsum([v.shape[1] for _, _, v in jobs])[:-1].tolist()
        end["vec"] = torch.cat([b.reshape(-1) for b in torch.tensor_split(end["vec"], cut, dim=1)]).reshape(6, -1)
        return end
    if kind == "serve":
        parts = []
        jobs = _jobs(case, seed)
        if sum(_job_turns(case, k) * len(e) for k, (e, _, _) in enumerate(jobs)) > 40000:
            return None
        for k, (eles, p, vec) in enumerate(jobs):
            t = _Tracker(p)
            parts.append(_final(t, t.track(_coords(vec), _values(eles), _job_turns(case, k))))
        return {"vec": torch.cat([q["vec"] for q in parts], dim=1), "beta": torch.cat([q["beta"] for q in parts]),
                "state": None}
    eles, p = _ring(case, seed)
    t = _Tracker(p)
    n = case["n"]
    if kind == "hook":
        vec = _bunch(dict(case, scale=3.0), seed, eles, n)
        return _final(t, t.track(_coords(vec), _values(eles)[HOOK_ELEMENTS[case["element"]]:][:1], 1))
    vec = _bunch(case, seed, eles, n)
    if kind in ("track_host", "track_device"):
        if len(eles) * case["turns"] * max(1.0, n / 2e5) > 30000:
            return None
        if case.get("moments"):
            return _exact_moments(t, vec, _values(eles), case["turns"])
        return _final(t, t.track(_coords(vec), _values(eles), case["turns"]))
    if kind == "grad":
        return _exact_grad(t, vec, eles, case["turns"])
    return _exact_stats(vec, seed, n)


def _exact_moments(t, vec, ring, turns):
    rows = []

    def sums(v, alive):
        v = [torch.where(alive, a, 0.0) for a in v]
        m = [alive.double().sum()] + [a.sum() for a in v]
        rows.append(torch.stack(m + [(v[i] * v[j]).sum() for i in range(6) for j in range(i, 6)]))

    end = _final(t, t.track(_coords(vec), ring, turns, after_turn=sums))
    return {**end, "moments": torch.stack(rows)}


def _exact_grad(t, vec, eles, turns):
    if turns * len(eles) > 3600:
        return None
    ring = _values(eles)
    at = _strength_elements(eles)
    k = torch.tensor([eles[i].k1 if eles[i].key == abi.QUADRUPOLE else eles[i].k2 for i in at], dtype=torch.float64,
                     device="cuda", requires_grad=True)

    def turn(k, *v):
        for j, e in enumerate(ring):
            if j in where:
                kj = k[where[j]]
                e = dict(e, k=kj) if e["kind"] == "quad" else dict(e, b={2: kj * e["l"] / 2})
            v = t.element(v, e)
        return v

    where = {i: j for j, i in enumerate(at)}
    v = _coords(vec)
    for _ in range(turns):
        v = torch.utils.checkpoint.checkpoint(turn, k, *v, use_reentrant=False)
    if bool(((v[0].abs() > rings.APERTURE_X) | (v[2].abs() > rings.APERTURE_Y)).any()):
        return None
    loss = (v[0] * v[0] + v[2] * v[2]).mean()
    loss.backward()
    return {"loss": loss.detach(), "grad": k.grad}


def _exact_stats(vec, seed, n):
    live = np.ones(n, bool)
    live[seed % 7::17] = False
    v = vec[:, live]
    a = v.mean(axis=1)
    d = v - a[:, None]
    sig = d @ d.T / v.shape[1]
    m3, m4 = (d ** 3).mean(axis=1), (d ** 4).mean(axis=1)
    s = np.sqrt(np.diag(sig))
    return {"n_live": None, "centroid": a, "sigma": sig.reshape(36), "skew": (m3 / s ** 3)[[0, 2, 4]],
            "kurt": (m4 / s ** 4)[[0, 2, 4]] - 3, "emit": None, "core_emit": None}
