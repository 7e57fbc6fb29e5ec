"""Gradient of the training kernel at the sizes where its split can go wrong,
against the FP64 closure oracle with the kernel's BF16 rounding points: one
row, one whole tile, a tile and a row, and more tiles than the GPU holds CTAs,
so that a CTA takes several.

Tolerance, derived before the first run: that of the gradient test of one
size, relative L2 error per parameter block <= 2e-3 (single BF16 roundings
that fall the other way), loss within 1e-4.
"""
import numpy as np
import pytest

from oracle import closure_oracle as co
from test_gpu_closure import BLOCKS, closure_with, random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", (1, 128, 129, 40000))
def test_gradient_by_number_of_tiles(n):
    p, mu, sd, dm, F, t, a = random_case(7, n)
    with closure_with(p, mu, sd, dm) as c:
        g, loss = c.gradient(F, t, a)
    lo, ge = co.loss_and_grad(p, mu, sd, dm, F, t, a, emulate=True)
    assert abs(loss - lo) <= 1e-4 * lo, (loss, lo)
    for name, b, e in BLOCKS:
        err = np.linalg.norm(g[b:e].astype(np.float64) - ge[b:e]) / np.linalg.norm(ge[b:e])
        assert err <= 2e-3, (name, err)
