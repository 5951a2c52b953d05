"""vk_block_solve_noalloc at the sizes where its kernels can go wrong: one to
five layers (an empty half, no second neighbour), blocks below, at and above
the smallest that a cluster shares and the largest one (a cluster's messages
no longer fit), odd sizes (blocks that start off a 16-byte boundary); and
systems that the two-sided elimination cannot start from the top.

Tolerance: 100 n eps cond(A) max|x|, the bound of a Gaussian elimination whose
growth stays moderate (the blocks are diagonally dominant or well conditioned);
cond(A) from the dense matrix.  A repeated call gives the same bits."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


@pytest.fixture(scope='module', autouse=True)
def built():
    from vulcan_gb300 import _build
    _build.build()


def _system(nz, n, seed):
    rng = np.random.default_rng(seed)
    D = 0.5 * rng.standard_normal((nz, n, n)) / n + np.eye(n) * (2.0 + rng.random((nz, 1, n)))
    lo, up, b = (rng.standard_normal((nz, n)) * s for s in (0.4, 0.4, 1.0))
    return D, lo, up, b


def _dense(D, lo, up):
    nz, n = lo.shape
    A = np.zeros((nz * n, nz * n))
    for j in range(nz):
        s = slice(j * n, (j + 1) * n)
        A[s, s] = D[j]
        if j > 0:
            A[s, (j - 1) * n:j * n] = np.diag(lo[j])
        if j + 1 < nz:
            A[s, (j + 1) * n:(j + 2) * n] = np.diag(up[j])
    return A


def _call(D, lo, up, b):
    import torch
    from vulcan_gb300 import capi
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (D, lo, up, b)]
    x = torch.full_like(t[3], float('nan'))
    torch.cuda.synchronize()
    nz, n = lo.shape
    rc = capi.lib().vk_block_solve_noalloc(nz, n, *[C.c_void_p(a.data_ptr()) for a in t],
                                           C.c_void_p(x.data_ptr()), None)
    return rc, x.cpu().numpy()


def _check(D, lo, up, b):
    A = _dense(D, lo, up)
    ref = np.linalg.solve(A, b.ravel()).reshape(b.shape)
    # the outermost couplings are not read
    lo, up = lo.copy(), up.copy()
    lo[0] = np.nan
    up[-1] = np.nan
    rc, x = _call(D, lo, up, b)
    assert rc == 0
    tol = 100 * b.shape[1] * EPS * np.linalg.cond(A) * np.abs(ref).max()
    assert np.abs(x - ref).max() <= tol
    np.testing.assert_array_equal(_call(D, lo, up, b)[1], x)


@pytest.mark.parametrize('nz,n', [(1, 1), (1, 40), (2, 7), (3, 31), (2, 32), (4, 33), (5, 69),
                                  (40, 17), (70, 38), (3, 150), (3, 160)])
def test_sizes(nz, n):
    _check(*_system(nz, n, 100 * nz + n))


@pytest.mark.parametrize('nz,n', [(2, 5), (4, 33), (5, 40)])
def test_singular_top_block_is_solved_from_the_bottom(nz, n):
    D, lo, up, b = _system(nz, n, nz + n)
    D[-1] = 0.0
    lo[-1], up[-2] = 1.0 + 0.1 * lo[-1], 1.0 + 0.1 * up[-2]
    _check(D, lo, up, b)


def test_singular_and_nan_blocks_are_refused():
    from vulcan_gb300 import capi
    for n in (12, 40):
        D, lo, up, b = _system(5, n, n)
        bad = D.copy()
        bad[0] = 0.0
        assert _call(bad, lo, up, b)[0] == capi.VK_ESINGULAR
        for j in (0, 2, 4):
            bad = D.copy()
            bad[j, 1, 2] = np.nan
            assert _call(bad, lo, up, b)[0] == capi.VK_ENAN
        assert _call(D, lo, up, b)[0] == capi.VK_OK
