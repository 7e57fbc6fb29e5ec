"""Diagnostics of 16-bit states, whose nodes are read two at a time where the
fields allow it, against FP64 sums of the downloaded moments: even and odd
node counts, fewer nodes than a block's threads and several blocks.

Tolerance, derived before the first run: the download rounds 1 + (rho - 1) to
FP32, so a node of the sum of rho is off by at most 6e-8; the other sums add
products of exact values and of that rho, off by 6e-8 of the sum of their
magnitudes; twice that is allowed.
"""
import numpy as np
import pytest

from entropicthreadsafe_b200 import capi, workloads
from entropicthreadsafe_b200.solver import Lattice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", ((3, 3, 3), (9, 7, 5), (8, 6, 4), (33, 31, 29), (64, 48, 40)))
@pytest.mark.parametrize("prec", (capi.PREC_BF16, capi.PREC_FP16S))
def test_sums_match_downloaded_moments(dims, prec):
    nx, ny, nz = dims
    rng = np.random.default_rng(nx)
    p = capi.default_params()
    p.mode, p.precision = capi.MODE_COLOUR, prec
    f = workloads.empty_fields(nx, ny, nz)
    f["rho"] = (1 + 0.01 * rng.standard_normal((nz, ny, nx))).astype(np.float32)
    for k in ("u", "v", "w"):
        f[k] = (0.05 * rng.standard_normal((nz, ny, nx))).astype(np.float32)
    f["phi"] = rng.uniform(-1, 1, (nz, ny, nx)).astype(np.float32)
    with Lattice(p, nx, ny, nz) as lat:
        lat.upload_moments(f)
        d, g = lat.reduce(), lat.download()
    r, u, v, w, phi = (np.asarray(g[k], np.float64) for k in ("rho", "u", "v", "w", "phi"))
    n, eps = nx * ny * nz, 1.2e-7
    kin = 0.5 * r * (u * u + v * v + w * w)
    assert abs(d["mass"] - r.sum()) <= eps * n
    assert abs(d["mass_a"] - (0.5 * r * (1 + phi)).sum()) <= eps * n
    assert abs(d["kinetic"] - kin.sum()) <= eps * kin.sum()
