"""Ghost phi given per face (wall_phi_mode 0, the default, and inlet faces) at
the edges of the step kernel's tiles.

A tile reads phi in whole 16-byte chunks of a row or node by node, and ghost
nodes behind a non-periodic face are computed; rows of whole chunks and not,
tiles whose rim lies behind a wall in y beside tiles that have whole chunks,
edges of faces of different ghost phi, and an inlet with walls beside it.

FP32 tolerance, derived before the first run: that of the parity tests, the
larger of 1e-5 and 4 times the oracle's own FP32 error, after 4 steps.

16-bit storage: one step, against an FP32 lattice that starts from the same
stored values.  Both compute in FP32 (1e-6 of a field's largest value); the
16-bit store then rounds a value to one of its two neighbours, less than a
unit in the last place away (2^-7 of a value in bf16, 2^-10 in fp16), and
rho = 1 + d is returned to FP32 precision (2^-23).  Scaled fp16 takes its
scales from the uploaded fields (the largest value at 2^9 to 2^10 of 65504);
where the moving walls drive a moment beyond that range the step must say so.
"""
import math

import numpy as np
import pytest

from entropicthreadsafe_b200 import capi
from entropicthreadsafe_b200.solver import Lattice, TslbError
from helpers import field_errors, run_gpu, run_oracle
from test_gpu_tiles import MODES, WALLS, state

pytestmark = pytest.mark.gpu

P, B, I, O = capi.BC_PERIODIC, capi.BC_BOUNCEBACK, capi.BC_INLET, capi.BC_OUTLET
GHOST_WALLS = dict(WALLS, ywalls=[P, P, B, B, P, P], inlet=[P, P, B, B, I, O])
BC_U = [[0.01, -0.005, 0.008], [0.0, 0.02, -0.01], [0.02, 0.004, -0.006], [0, 0, 0], [-0.03, 0.01, 0.002], [0.03, 0.0, 0.004]]

CASES = [
    ("phase", (96, 96, 6), "ywalls"), ("phase", (68, 17, 8), "ywalls"), ("phase", (96, 20, 12), "box"),
    ("phase", (128, 64, 5), "ydrag"), ("phase", (104, 13, 6), "duct"), ("phase", (104, 33, 6), "xdrag"),
    ("phase", (101, 17, 9), "box"), ("phase", (96, 30, 8), "inlet"), ("phase", (45, 14, 10), "inlet"),
    ("colour", (96, 20, 12), "ywalls"), ("colour", (128, 64, 5), "box"), ("colour", (101, 17, 9), "box"),
    ("colour", (104, 13, 6), "duct"), ("colour", (72, 7, 33), "ydrag"), ("colour", (104, 33, 6), "xdrag"),
    ("colour", (96, 30, 8), "inlet"), ("colour", (45, 14, 10), "inlet"),
]


def params(mode, walls, wall_phi_mode, precision=capi.PREC_FP32):
    bc_phi = [0.2, -0.6, 0.9, -0.3, 0.5, -0.8]
    if mode == "phase":
        bc_phi = [0.5 * (1.0 + v) for v in bc_phi]
    return capi.make_params(mode=MODES[mode], precision=precision, tau_a=0.7, tau_b=0.7 if mode == "phase" else 0.9, sigma=0.01,
                            beta=0.7, grad_threshold=1e-4, force=(1e-5, -2e-6, 3e-6), bc=GHOST_WALLS[walls], bc_u=BC_U,
                            bc_phi=bc_phi, wall_phi_mode=wall_phi_mode)


def inlet_planes(mode, dims):
    """u, v, w, phi of the plane z = 0: a normal flow with a patch of the other phase."""
    nx, ny, _ = dims
    y, x = np.meshgrid(np.arange(ny), np.arange(nx), indexing="ij")
    pl = np.zeros((4, ny, nx), np.float32)
    pl[0] = 0.004 * np.cos(2 * np.pi * x / nx)
    pl[2] = 0.02 * np.sin(np.pi * (y + 0.5) / ny)
    t = np.tanh((0.3 * min(nx, ny) - np.hypot(x - nx / 3, y - ny / 3)) / 2.0)
    pl[3] = 0.5 * (1.0 + t) if mode == "phase" else t
    return {capi.FACE_ZM: pl}


@pytest.mark.parametrize("wall_phi_mode", (0, 1))
@pytest.mark.parametrize("mode,dims,walls", CASES, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else v)
def test_ghost_phi_matches_oracle(mode, dims, walls, wall_phi_mode):
    p = params(mode, walls, wall_phi_mode)
    f = state(mode, dims, 7)
    inlet = inlet_planes(mode, dims) if walls == "inlet" else None
    gpu, _ = run_gpu(p, f, 4, inlet)
    o64, _ = run_oracle(p, f, 4, fp64=True, inlet=inlet)
    o32, _ = run_oracle(p, f, 4, fp64=False, inlet=inlet)
    eg, e32 = field_errors(gpu, o64), field_errors(o32, o64)
    bad = {k: (eg[k], e32[k]) for k in eg if eg[k] > max(1e-5, 4.0 * e32[k])}
    assert not bad, bad


def beyond_range(uploaded, after):
    """a value beyond the largest scaled fp16 one, 65504 / scale with scale = 2^floor(log2(2^10 / largest uploaded))"""
    for k in capi.FIELDS:
        a, b = uploaded[k].astype(np.float64), after[k].astype(np.float64)
        if k == "rho":
            a, b = a - 1.0, b - 1.0
        e = min(24, max(-8, math.floor(math.log2(1024.0 / np.abs(a).max()))))
        if np.abs(b).max() > 65504.0 / 2.0 ** e:
            return True
    return False


@pytest.mark.parametrize("prec", ("bf16", "fp16s"))
@pytest.mark.parametrize("mode,dims,walls", [c for c in CASES if c[2] in ("box", "ydrag", "inlet")],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else v)
def test_ghost_phi_in_16_bit_storage(mode, dims, walls, prec):
    precision, unit = (capi.PREC_BF16, 2.0 ** -7) if prec == "bf16" else (capi.PREC_FP16S, 2.0 ** -10)
    inlet = inlet_planes(mode, dims) if walls == "inlet" else {}
    nx, ny, nz = dims
    with Lattice(params(mode, walls, 0, precision), nx, ny, nz) as lat:
        for face, planes in inlet.items():
            lat.set_inlet(face, planes)
        lat.upload_moments(state(mode, dims, 7))
        stored = lat.download()
        ref, _ = run_gpu(params(mode, walls, 0), stored, 1, inlet)
        lat.step(1)
        if prec == "fp16s" and beyond_range(state(mode, dims, 7), ref):
            with pytest.raises(TslbError) as err:
                lat.synchronize()
            assert err.value.code == capi.ERR_NAN
            return
        lat.synchronize()
        got = lat.download()
    for k in capi.FIELDS:
        a, b = got[k].astype(np.float64), ref[k].astype(np.float64)
        if k == "rho":
            a, b = a - 1.0, b - 1.0
        tol = unit * np.abs(b) + 1e-6 * np.abs(b).max() + (2.0 ** -23 if k == "rho" else 0.0)
        assert np.all(np.abs(a - b) <= tol), (k, float((np.abs(a - b) - tol).max()))
