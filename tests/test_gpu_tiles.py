"""The step kernel at the edges of its tiles, against the FP64 oracle.

Sizes around the tile width (30 target columns of a 32-lane warp), the row
counts of both block sizes (6 and 14 target rows), rows of whole 16-byte
chunks and not, a periodic axis inside one warp (nx <= 32), and the closed
sums of walls at faces, edges and corners, for every wall kind that has one.

Tolerance, derived before the first run: that of the parity tests, the larger
of 1e-5 and 4 times the oracle's own FP32 error, after 4 steps.
"""
import numpy as np
import pytest

from entropicthreadsafe_b200 import capi, workloads
from helpers import field_errors, run_gpu, run_oracle

pytestmark = pytest.mark.gpu

MODES = {"colour": capi.MODE_COLOUR, "phase": capi.MODE_PHASEFIELD, "single": capi.MODE_SINGLE}
P, B, V, PR = capi.BC_PERIODIC, capi.BC_BOUNCEBACK, capi.BC_VELOCITY, capi.BC_PRESSURE
WALLS = {
    "periodic": [P] * 6,
    "box": [B] * 6,                       # faces, edges and corners of bounce-back
    "couette": [P] * 4 + [V, V],          # one velocity face
    "duct": [B, B, P, P, V, PR],          # a pressure face, edges of mixed kinds
    "ydrag": [P, P, V, B, P, P],          # velocity and bounce-back normal to y
    "xdrag": [V, PR, P, P, B, B],         # normal to x
}

CASES = [
    ("colour", (100, 40, 30), "periodic"), ("colour", (101, 17, 9), "box"), ("colour", (64, 30, 40), "couette"),
    ("colour", (31, 8, 8), "periodic"), ("colour", (32, 16, 20), "periodic"), ("colour", (33, 9, 7), "box"),
    ("colour", (7, 5, 4), "periodic"), ("colour", (70, 33, 12), "duct"), ("colour", (61, 15, 11), "ydrag"),
    ("colour", (104, 13, 6), "xdrag"), ("colour", (160, 29, 140), "couette"),
    ("phase", (100, 40, 30), "periodic"), ("phase", (96, 20, 12), "box"), ("phase", (9, 9, 9), "box"),
    ("phase", (45, 14, 10), "couette"), ("phase", (72, 7, 33), "ydrag"),
    ("single", (100, 40, 30), "box"), ("single", (31, 31, 5), "periodic"), ("single", (62, 28, 17), "duct"),
    ("single", (90, 15, 9), "xdrag"),
]


def state(mode, dims, seed):
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    f = workloads.empty_fields(nx, ny, nz)
    for k in ("u", "v", "w"):
        f[k][:] = rng.normal(0, 0.02, f[k].shape)
    for k in ("pxx", "pxy", "pxz", "pyy", "pyz", "pzz"):
        f[k][:] = rng.normal(0, 1e-4, f[k].shape)
    f["rho"][:] = 1.0 + rng.normal(0, 1e-3, f["rho"].shape)
    if mode == "single":
        f["phi"][:] = 1.0
    else:
        # an interface through the whole lattice, tilted so that it crosses every face
        z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
        t = np.tanh((np.sin(2 * np.pi * (x / nx + 0.3)) + 0.7 * np.cos(2 * np.pi * y / ny) + 0.5 * np.sin(2 * np.pi * z / nz)) * 1.5)
        f["phi"][:] = 0.5 * (1.0 + t) if mode == "phase" else t
    return f


@pytest.mark.parametrize("mode,dims,walls", CASES, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else v)
def test_tile_edges_match_oracle(mode, dims, walls):
    bc_u = [[0.01, -0.005, 0.008], [0.0, 0.02, -0.01], [0.02, 0.004, -0.006], [0, 0, 0], [-0.03, 0.01, 0.002], [0.03, 0.0, 0.004]]
    p = capi.make_params(mode=MODES[mode], tau_a=0.7, tau_b=0.7 if mode == "phase" else 0.9, sigma=0.0 if mode == "single" else 0.01,
                         beta=0.7, grad_threshold=1e-4, force=(1e-5, -2e-6, 3e-6), bc=WALLS[walls], bc_u=bc_u,
                         bc_phi=[0.2] * 6, wall_phi_mode=1)
    f = state(mode, dims, 7)
    gpu, _ = run_gpu(p, f, 4)
    o64, _ = run_oracle(p, f, 4, fp64=True)
    o32, _ = run_oracle(p, f, 4, fp64=False)
    if mode == "single":   # phi is held at 1; the oracle's phase-field step moves its own
        assert np.all(gpu["phi"] == 1.0)
        o64["phi"], o32["phi"] = gpu["phi"], gpu["phi"]
    eg, e32 = field_errors(gpu, o64), field_errors(o32, o64)
    bad = {k: (eg[k], e32[k]) for k in eg if eg[k] > max(1e-5, 4.0 * e32[k])}
    assert not bad, bad


@pytest.mark.parametrize("prec", ["bf16", "fp16s"])
@pytest.mark.parametrize("dims", [(45, 9, 8), (104, 13, 6), (30, 16, 12)], ids=lambda d: "x".join(map(str, d)))
def test_16_bit_rows(prec, dims):
    """16-bit storage, rows of whole chunks and not: one step stays within the
    rounding of the stored values.  The upload rounds each value to a unit in
    the last place (2^-8 of bf16, 2^-11 of fp16) at most and the step's store
    once more; the step itself is within a factor 2 of the identity in them:
    4 units of the largest value of a field."""
    f = state("colour", dims, 3)
    for k in ("pxx", "pxy", "pxz", "pyy", "pyz", "pzz"):
        f[k][:] = 0.0
    f["rho"][:] = 1.0
    unit = 2.0 ** -8 if prec == "bf16" else 2.0 ** -11
    out = {}
    for name, pr in (("fp32", capi.PREC_FP32), (prec, capi.PREC_BF16 if prec == "bf16" else capi.PREC_FP16S)):
        p = capi.make_params(mode=capi.MODE_COLOUR, precision=pr, tau_a=0.9, tau_b=0.8, sigma=0.01, beta=0.7, grad_threshold=1e-3,
                             bc=[P, P, P, P, B, B], bc_phi=[-1.0] * 6, wall_phi_mode=1)
        out[name], _ = run_gpu(p, f, 1)
    vmax = max(float(np.abs(out["fp32"][k]).max()) for k in ("u", "v", "w"))
    for k in ("u", "v", "w", "phi"):
        a, b = out[prec][k].astype(np.float64), out["fp32"][k]
        scale = vmax if k != "phi" else 1.0
        assert float(np.abs(a - b).max()) <= 4 * unit * scale, k
