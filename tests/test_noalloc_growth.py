"""vk_block_solve_noalloc on systems that an elimination from the top spoils: a
block (or one row of it) of the upper half that is nearly singular by itself, which
its couplings to the layer below make harmless from the bottom.  The
two-sided elimination would answer with the digits that the growth costs; such a
system is solved from the bottom.  Clusters and single CTAs, three layers on.

Tolerance: 100 n eps cond(A) max|x|, as for every well-conditioned system
(cond(A) is at most a few hundred here)."""
import numpy as np
import pytest

from test_noalloc_shapes import EPS, _call, _dense, _system

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module', autouse=True)
def built():
    from vulcan_gb300 import _build
    _build.build()


@pytest.mark.parametrize('nz,n', [(3, 5), (5, 31), (4, 33), (5, 40), (9, 69), (3, 160)])
@pytest.mark.parametrize('where', ['top', 'inside', 'row'])
@pytest.mark.parametrize('tiny', [1e-5, 1e-10, 1e-15])
def test_growth_from_the_top(nz, n, where, tiny):
    D, lo, up, b = _system(nz, n, 100 * nz + n)
    j = nz - 1 if where != 'inside' else max(nz - 2, 1)
    if where == 'row':
        D[j, n // 2] = 0.0
        D[j, :, n // 2] = 0.0
        D[j, n // 2, n // 2] = tiny
    else:
        D[j] = tiny * np.eye(n)
    lo[j], up[j - 1] = 1.0 + 0.1 * lo[j], 1.0 + 0.1 * up[j - 1]
    A = _dense(D, lo, up)
    cond = np.linalg.cond(A)
    assert cond < 1e4
    ref = np.linalg.solve(A, b.ravel()).reshape(b.shape)
    rc, x = _call(D, lo, up, b)
    assert rc == 0
    assert np.abs(x - ref).max() <= 100 * n * EPS * cond * np.abs(ref).max()
