"""Rows of whole 16-byte chunks on a periodic x axis: every tile reads them in
chunks, wrapped whole, also where the axis is shorter than the 40 nodes that a
tile reads of a row, or lies in one warp.  FP32 against the oracle, with the
parity tests' tolerance (the larger of 1e-5 and 4 times the oracle's own FP32
error, 3 steps); 16-bit storage against an FP32 lattice from the same stored
values, one step (1e-6 of a field's largest value and less than a unit in the
last place, as in test_gpu_ghost_phi.py)."""
import numpy as np
import pytest

from entropicthreadsafe_b200 import capi
from entropicthreadsafe_b200.solver import Lattice
from helpers import field_errors, run_gpu, run_oracle
from test_gpu_tiles import MODES, state

pytestmark = pytest.mark.gpu

P, B = capi.BC_PERIODIC, capi.BC_BOUNCEBACK


def params(mode, yz, precision=capi.PREC_FP32):
    return capi.make_params(mode=MODES[mode], precision=precision, tau_a=0.7, tau_b=0.7 if mode == "phase" else 0.9,
                            sigma=0.0 if mode == "single" else 0.01, beta=0.7, grad_threshold=1e-4, force=(1e-5, -2e-6, 3e-6),
                            bc=[P, P] + ([B] * 4 if yz == "walls" else [P] * 4), bc_phi=[0.3] * 6, wall_phi_mode=0)


@pytest.mark.parametrize("yz", ("periodic", "walls"))
@pytest.mark.parametrize("nx", (4, 8, 12, 32, 36, 40, 60, 64, 92))
@pytest.mark.parametrize("mode", ("colour", "phase", "single"))
def test_fp32_matches_oracle(mode, nx, yz):
    p, f = params(mode, yz), state(mode, (nx, 9, 7), 7)
    gpu, _ = run_gpu(p, f, 3)
    o64, _ = run_oracle(p, f, 3, fp64=True)
    o32, _ = run_oracle(p, f, 3, fp64=False)
    if mode == "single":   # phi is held at 1; the oracle's phase-field step moves its own
        o64["phi"], o32["phi"] = gpu["phi"], gpu["phi"]
    eg, e32 = field_errors(gpu, o64), field_errors(o32, o64)
    bad = {k: (eg[k], e32[k]) for k in eg if eg[k] > max(1e-5, 4.0 * e32[k])}
    assert not bad, bad


@pytest.mark.parametrize("prec", ("bf16", "fp16s"))
@pytest.mark.parametrize("nx", (8, 16, 32, 40, 64, 72))
@pytest.mark.parametrize("mode", ("colour", "phase", "single"))
def test_16_bit_matches_fp32_from_the_same_values(mode, nx, prec):
    precision, unit = (capi.PREC_BF16, 2.0 ** -7) if prec == "bf16" else (capi.PREC_FP16S, 2.0 ** -10)
    with Lattice(params(mode, "periodic", precision), nx, 9, 7) as lat:
        lat.upload_moments(state(mode, (nx, 9, 7), 7))
        stored = lat.download()
        lat.step(1)
        got = lat.download()
    ref, _ = run_gpu(params(mode, "periodic"), stored, 1)
    for k in capi.FIELDS:
        a, b = got[k].astype(np.float64), ref[k].astype(np.float64)
        if k == "rho":
            a, b = a - 1.0, b - 1.0
        tol = unit * np.abs(b) + 1e-6 * np.abs(b).max() + (2.0 ** -23 if k == "rho" else 0.0)
        assert np.all(np.abs(a - b) <= tol), (k, float((np.abs(a - b) - tol).max()))
