"""Lattices beyond what the step's 32-bit node numbers reach are refused, with a
message, before any device call; the limit is one device's, not a slabbed lattice's."""
import ctypes

import pytest

from entropicthreadsafe_b200 import build, capi


@pytest.fixture(scope="module")
def lib():
    build.build()
    return capi.lib()


def create(lib, nx, ny, nz):
    p = capi.default_params()
    h = ctypes.c_void_p()
    rc = lib.tslb_create(ctypes.addressof(p), nx, ny, nz, ctypes.byref(h))
    msg = lib.tslb_last_error(None) or b""
    if h.value:
        lib.tslb_destroy(h)
    return rc, msg


@pytest.mark.parametrize("dims", ((2048, 2048, 1024), (65536, 32768, 1), (65536, 65536, 1), (1, 1, 2 ** 31 - 1), (2, 2 ** 30, 3)))
def test_too_large_is_refused(lib, dims):
    rc, msg = create(lib, *dims)
    assert rc == capi.ERR_ARG and b"too large" in msg
    p = capi.default_params()
    n = dims[0] * dims[1] * dims[2]
    rc = lib.tslb_step_noalloc(ctypes.addressof(p), *dims, ctypes.c_void_p(1 << 20), ctypes.c_void_p(1 << 50), (n + 31) // 32 * 32, None)
    assert rc == capi.ERR_ARG and b"too large" in lib.tslb_last_error(None)


@pytest.mark.parametrize("dims", ((2048, 2048, 1023), (46340, 46340, 1)))
def test_largest_is_not_refused_for_its_size(lib, dims):
    rc, msg = create(lib, *dims)
    assert rc != capi.ERR_ARG, msg   # (no device, or not enough memory)


def test_slab_of_a_larger_lattice(lib):
    p = capi.default_params()
    h = ctypes.c_void_p()
    rc = lib.tslb_create_slab(ctypes.addressof(p), 64, 64, 2 ** 21, 64, 128, ctypes.byref(h))
    assert rc != capi.ERR_ARG, lib.tslb_last_error(None)
    if h.value:
        lib.tslb_destroy(h)
