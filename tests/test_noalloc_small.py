"""vk_block_solve_noalloc around the sizes up to which a system is solved in one
launch (32 species, 8 layers, 48 values): both sides of each limit, one layer and
one species, failures reported and forgotten.

Tolerance: 100 n eps cond(A) max|x|, as in test_noalloc_shapes.py."""
import numpy as np
import pytest

from test_noalloc_shapes import _call, _check, _system
from vulcan_gb300 import capi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module', autouse=True)
def built():
    from vulcan_gb300 import _build
    _build.build()


@pytest.mark.parametrize('nz,n', [(1, 1), (2, 1), (8, 1), (9, 1), (1, 31), (1, 32), (1, 33), (2, 24), (2, 25),
                                  (3, 16), (3, 17), (4, 12), (4, 13), (8, 6), (8, 7)])
def test_sizes(nz, n):
    _check(*_system(nz, n, 100 * nz + n))


@pytest.mark.parametrize('nz,n', [(1, 3), (3, 16), (8, 6)])
def test_failures(nz, n):
    D, lo, up, b = _system(nz, n, n)
    for j in range(nz):
        bad = D.copy()
        bad[j, 0, n - 1] = np.nan
        assert _call(bad, lo, up, b)[0] == capi.VK_ENAN
    bad = D.copy()
    bad[0] = 0.0
    assert _call(bad, lo, up, b)[0] == capi.VK_ESINGULAR
    rc, x = _call(D, lo, up, b)
    assert rc == capi.VK_OK and np.isfinite(x).all()


def test_result_may_replace_the_right_hand_side():
    import ctypes as C
    import torch
    for nz, n in ((8, 6), (9, 6)):
        D, lo, up, b = _system(nz, n, 5)
        _, x = _call(D, lo, up, b)
        t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (D, lo, up, b)]
        p = [C.c_void_p(a.data_ptr()) for a in t]
        assert capi.lib().vk_block_solve_noalloc(nz, n, *p, p[3], None) == 0
        np.testing.assert_array_equal(t[3].cpu().numpy(), x)
