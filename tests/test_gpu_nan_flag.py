"""A moment that is not a number is reported by the step that meets it, in every
storage type: a single NaN of the uploaded state reaches the stored moments of
its node's neighbours, and 16-bit storage checks its range before rounding."""
import numpy as np
import pytest

from entropicthreadsafe_b200 import capi
from entropicthreadsafe_b200.solver import Lattice, TslbError
from test_gpu_tiles import MODES, state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field", ("rho", "w", "pyz", "phi"))
@pytest.mark.parametrize("precision", (capi.PREC_FP32, capi.PREC_BF16, capi.PREC_FP16S), ids=("fp32", "bf16", "fp16s"))
@pytest.mark.parametrize("mode", ("colour", "phase", "single"))
def test_nan_is_reported(mode, precision, field):
    nx, ny, nz = dims = (45, 9, 8)
    f = state(mode, dims, 7)
    p = capi.make_params(mode=MODES[mode], precision=precision, tau_a=0.7, tau_b=0.7, sigma=0.0 if mode == "single" else 0.01)
    if mode == "single" and field == "phi":
        field = "u"   # phi is held at 1 there
    with Lattice(p, nx, ny, nz) as lat:
        lat.upload_moments(f)
        lat.step(1)
        lat.synchronize()   # nothing to report
        f[field][4, 5, 31] = np.nan
        lat.upload_moments(f)
        lat.step(1)
        with pytest.raises(TslbError) as err:
            lat.synchronize()
    assert err.value.code == capi.ERR_NAN
