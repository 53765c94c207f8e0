"""The automatic shots per CTA, read through the plan's configuration on the host."""
import ctypes

import pytest

from test_capi import lib  # noqa: F401  (module fixture: the built library)
from test_schedule import _plan


@pytest.mark.parametrize("nz,nx,nabc,shots,cpml,spc", [
    (400, 1200, 30, 1, False, 1), (400, 1200, 30, 8, False, 4), (400, 1200, 30, 8, True, 3),
    (400, 1200, 30, 32, False, 11), (1000, 3000, 40, 16, False, 8), (88, 200, 20, 40, False, 2),
    (100, 200, 20, 16, False, 1), (200, 500, 20, 12, False, 2)])
def test_automatic_shots_per_cta(lib, nz, nx, nabc, shots, cpml, spc):  # noqa: F811
    """Equal groups that fill the GPU with as little per-group work as that allows."""
    h = _plan(lib, nz, nx, nabc, 4, shots)
    if cpml:
        assert lib.gb_plan_set_absorbing(h, 1, ctypes.c_float(3000.0)) == 0
    v = [ctypes.c_int() for _ in range(5)]
    assert lib.gb_plan_get_config(h, *[ctypes.byref(x) for x in v]) == 0
    assert v[1].value == spc
    lib.gb_plan_destroy(h)
