"""Entry points of the library that answer without a device: handles and argument checks."""
import ctypes as C

import pytest

from torchsso import _native as nat


def description(**kwargs):
    d = nat.FactorDesc()
    d.n, d.c, d.h, d.w, d.sn, d.sc = 4, 8, 1, 1, 8, 1
    d.kh = d.kw = d.stride_h = d.stride_w = d.dil_h = d.dil_w = 1
    d.out, d.ldo = 4096, 8
    for k, v in kwargs.items():
        setattr(d, k, v)
    return d


def test_factor_op_handles():
    lib = nat.lib()

    def refused(rc):
        return rc == -1 and b'unknown handle' in lib.sso_last_error()
    d = description()
    a, b = (lib.sso_factor_op_create(C.byref(d), 0) for _ in range(2))
    assert a > 0 and b > 0 and a != b
    assert lib.sso_factor_op_run(a, None, None, 1.0, 0.0, None, 0, None) == -1      # no input
    assert lib.sso_factor_op_destroy(a) == 0
    for h in (a, 0, -5, b + 1000, 1 << 62):          # destroyed, or never given out
        assert refused(lib.sso_factor_op_run(h, 4096, None, 1.0, 0.0, None, 0, None))
        assert refused(lib.sso_factor_op_destroy(h))
    assert lib.sso_factor_op_destroy(b) == 0


@pytest.mark.parametrize('bad', [{'n': 0}, {'kh': 0}, {'ldo': 7}, {'out': None}, {'kw': 2}])
def test_factor_op_refuses_a_bad_description(bad):
    assert nat.lib().sso_factor_op_create(C.byref(description(**bad)), 0) < 0


def test_factor_scratch_grows_with_the_problem_and_has_an_end():
    size = nat.lib().sso_factor_workspace_bytes
    assert size(1 << 31, 16384, nat.IMPL_TCGEN05) < 1 << 31
    for impl in (nat.IMPL_AUTO, nat.IMPL_TCGEN05):
        assert size(1, 1, impl) > 65536
        for rows, d in ((1, 300), (128, 4097), (100000, 64)):
            assert size(rows, d, impl) >= size(rows, d, nat.IMPL_TMA)


@pytest.mark.parametrize('rows,cols,fits', [(5000, 300, True), (20000, 64, True), (128, 2000, True), (1568, 4608, False)])
def test_factor_without_allocation_goes_by_the_partial_tiles(rows, cols, fits):
    """What is refused for its size is refused before the device is asked for anything."""
    lib = nat.lib()
    rc = lib.sso_factor_syrk_noalloc(None, nat.F32, rows, cols, cols, 1, 0, None, 1.0, 0.0, None, cols, nat.IMPL_AUTO, None)
    assert rc < 0 and (b'built-in scratch' not in lib.sso_last_error()) == fits
