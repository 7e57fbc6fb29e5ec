"""Nodes whose populations from behind faces have no closed sums: inlets and
outlets normal to x, y and z, edges and corners of faces of different kinds,
lattices one node thick between two walls, and walls beside interior solids.

The step takes whole rows of inlet or outlet nodes nine populations in turn,
and lists the others, half a warp a node; sizes around the tiles, so that a
tile has no, one and many such nodes (more than a pass of the block's half
warps), with a correction of the relaxation time, and in 16-bit storage.

Tolerance, derived before the first run: that of the parity tests, the larger
of 1e-5 and 4 times the oracle's own FP32 error, after 3 steps.  16-bit: as in
test_gpu_ghost_phi.py (one step against an FP32 lattice from the same stored
values: 1e-6 of a field's largest value and less than a unit in the last place).
"""
import numpy as np
import pytest

import oracle
from entropicthreadsafe_b200 import capi
from entropicthreadsafe_b200.solver import Lattice
from helpers import field_errors
from test_gpu_tiles import MODES, state

pytestmark = pytest.mark.gpu

P, B, V, I, O, PR = capi.BC_PERIODIC, capi.BC_BOUNCEBACK, capi.BC_VELOCITY, capi.BC_INLET, capi.BC_OUTLET, capi.BC_PRESSURE
FACES = {
    "xio": [I, O, P, P, P, P], "yio": [P, P, I, O, P, P], "zio": [P, P, P, P, I, O],
    "xyio": [I, O, O, I, P, P], "mixed": [V, O, V, PR, I, V], "boxv": [V] * 6, "xbyv": [B, B, V, V, P, P],
    "bio": [B, B, B, B, I, O], "zv": [P, P, P, P, V, B], "box": [B] * 6,
}
BC_U = [[0.01, -0.005, 0.008], [0.0, 0.02, -0.01], [0.02, 0.004, -0.006], [0.003, 0.0, 0.01], [-0.03, 0.01, 0.002], [0.03, 0.0, 0.004]]


def params(mode, faces, precision=capi.PREC_FP32):
    return capi.make_params(mode=MODES[mode], precision=precision, tau_a=0.7, tau_b=0.7 if mode == "phase" else 0.9,
                            sigma=0.0 if mode == "single" else 0.01, beta=0.7, grad_threshold=1e-4, force=(1e-5, -2e-6, 3e-6),
                            bc=FACES[faces], bc_u=BC_U, bc_phi=[0.2, 0.4, 0.6, 0.3, 0.5, 0.8], wall_phi_mode=1)


def inlet_planes(mode, dims, faces):
    """u, v, w, phi of every inlet face: smooth, different per face"""
    out = {}
    for face, kind in enumerate(FACES[faces]):
        if kind != I:
            continue
        a, b = [d for k, d in enumerate(dims) if k != face // 2]
        y, x = np.meshgrid(np.arange(b), np.arange(a), indexing="ij")
        pl = np.zeros((4, b, a), np.float32)
        for k in range(3):
            pl[k] = 0.01 * np.cos(2 * np.pi * x / a + k + face) * np.sin(np.pi * (y + 0.5) / b)
        t = np.tanh((0.3 * min(a, b) - np.hypot(x - a / 3, y - b / 3)) / 2.0)
        pl[3] = 0.5 * (1.0 + t) if mode == "phase" else t
        out[face] = pl
    return out


def set_up(x, inlets, iso, dtau):
    for face, planes in inlets.items():
        x.set_inlet(face, planes)
    if iso is not None:
        (x.set_isfluid if hasattr(x, "set_isfluid") else x.set_solid_mask)(iso)
    if dtau is not None:
        x.set_tau_correction(dtau)


CASES = [(m, d, f, "") for m in ("colour", "phase", "single") for d, f in (
    ((61, 15, 9), "xio"), ((100, 13, 9), "yio"), ((45, 29, 7), "zio"), ((31, 8, 8), "xyio"), ((61, 15, 11), "mixed"),
    ((96, 30, 12), "mixed"), ((33, 7, 20), "boxv"), ((104, 40, 6), "xbyv"), ((90, 20, 8), "bio"), ((40, 12, 1), "zv"), ((1, 20, 15), "xbyv"))]
CASES += [("colour", (61, 15, 9), "xio", "tau"), ("colour", (61, 15, 11), "mixed", "tau"), ("colour", (45, 29, 7), "zio", "tau")]
CASES += [(m, (61, 15, 11), f, "solid") for m in ("colour", "phase", "single") for f in ("mixed", "box", "boxv", "yio")]


@pytest.mark.parametrize("mode,dims,faces,extra", CASES, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else v)
def test_general_faces_match_oracle(mode, dims, faces, extra):
    nx, ny, nz = dims
    p, f, inlets = params(mode, faces), state(mode, dims, 7), inlet_planes(mode, dims, faces)
    rng = np.random.default_rng(2)
    iso = (rng.random((nz, ny, nx)) > 0.06).astype(np.uint8) if extra == "solid" else None
    dtau = rng.uniform(-0.05, 0.2, (nz, ny, nx)).astype(np.float32) if extra == "tau" else None
    res = []
    for fp64 in (True, False):
        o = oracle.Oracle(p, nx, ny, nz, fp64=fp64)
        set_up(o, inlets, iso, dtau)
        o.set_moments({k: np.asarray(v, np.float64) for k, v in f.items()})
        o.step(3)
        res.append(o.get_moments())
        o.close()
    with Lattice(p, nx, ny, nz) as lat:
        set_up(lat, inlets, iso, dtau)
        lat.upload_moments(f)
        lat.step(3)
        res.append(lat.download())
    for r in res:
        if mode == "single":   # phi is held at 1; the oracle's phase-field step moves its own
            r["phi"] = np.ones_like(r["phi"])
        if iso is not None:    # fluid nodes
            for k in capi.FIELDS:
                r[k] = np.where(iso == 1, r[k], 1.0 if k == "rho" else 0.0)
    o64, o32, gpu = res
    eg, e32 = field_errors(gpu, o64), field_errors(o32, o64)
    bad = {k: (eg[k], e32[k]) for k in eg if eg[k] > max(1e-5, 4.0 * e32[k])}
    assert not bad, bad


@pytest.mark.parametrize("mode", ("colour", "phase", "single"))
@pytest.mark.parametrize("dims,faces", [((61, 15, 9), "xio"), ((100, 13, 9), "yio"), ((61, 15, 11), "mixed"), ((96, 30, 12), "mixed")],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else v)
def test_general_faces_in_bf16(mode, dims, faces):
    nx, ny, nz = dims
    inlets = inlet_planes(mode, dims, faces)
    out = []
    stored = state(mode, dims, 7)
    for precision in (capi.PREC_BF16, capi.PREC_FP32):
        with Lattice(params(mode, faces, precision), nx, ny, nz) as lat:
            set_up(lat, inlets, None, None)
            lat.upload_moments(stored)
            if precision == capi.PREC_BF16:
                stored = lat.download()
            lat.step(1)
            lat.synchronize()
            out.append(lat.download())
    for k in capi.FIELDS:
        a, b = (v[k].astype(np.float64) - (1.0 if k == "rho" else 0.0) for v in out)
        tol = 2.0 ** -7 * np.abs(b) + 1e-6 * np.abs(b).max() + (2.0 ** -23 if k == "rho" else 0.0)
        assert np.all(np.abs(a - b) <= tol), (k, float((np.abs(a - b) - tol).max()))
