"""The mixed path's FP32 block inverses (k_lu32, vk_get_lu32) against NumPy in 64
bits: layer by layer, the scaled block less the Schur terms of the neighbours the
two-sided elimination comes from (the device's own FP32 inverses, so errors do not
add up over the layers), inverted in FP64.  The workload's own mixing, whose Schur
terms are tiny at this step, and one as fast as the step.  Both halves, the middle layer with its
two terms and without a lower half's; networks on both sides of every register tiling's
edge (48, 64, 72, 96, 128, 160 species), every tiling that holds the block.

Tolerance: forming a block costs at most 6 roundings of |D| + |S|, S the Schur terms
(couplings 2, product 2, difference 2), which the inverse carries as |G| (|D| + |S|) |G|;
an elimination of moderate growth adds a few more of |G| |D'| |G|: 16 u max(|G| (|D| + |S|) |G|),
u = 2^-24 (one in NumPy's FP32 stays below 2)."""
import os

import numpy as np
import pytest

from conftest import GOLDEN
from test_synthnet import ATOMS, BUILD
from vulcan_gb300 import batch, capi, configs, synthnet
from vulcan_gb300.network import Network

pytestmark = pytest.mark.gpu
R_ROS = 1. + 1. / 2. ** 0.5
# species of the network: synthnet.generate's ni, n_rev, seed
NETS = {17: (17, 17, 1), 48: (48, 48, 1), 49: (50, 49, 1), 64: (66, 64, 3), 65: (66, 65, 1), 72: (73, 72, 2),
        73: (75, 73, 3), 96: (96, 288, 1), 97: (97, 291, 1), 128: (128, 384, 1), 129: (129, 387, 1),
        160: (160, 480, 1)}


@pytest.fixture(scope='module', autouse=True)
def built():
    from vulcan_gb300 import _build
    _build.build()


def _network(species):
    if species == 69:
        return Network.from_npz(os.path.join(GOLDEN, 'net_NCHO_photo.npz'))
    ni, n_rev, seed = NETS[species]
    path = synthnet.generate(os.path.join(BUILD, 'syn%d' % species), seed=seed, ni=ni, n_rev=n_rev, n_photo=8,
                             name='SYN%d' % species)
    net = Network.from_file(path, use_photo=True)
    assert net.ni == species
    return net


def _scaled(jv, dA, dt, rows, cols, n):
    """(R, S, R D S in FP32) of a layer's block, as k_prep32 forms them."""
    D = np.zeros((n, n))
    D[rows, cols] = jv
    i = np.arange(n)
    D[i, i] += 1.0 / (R_ROS * dt) - dA
    r = 2.0 ** -np.frexp(np.abs(D).max(axis=1))[1]
    s = 2.0 ** -np.frexp(np.abs(r[:, None] * D).max(axis=0))[1]
    return r, s, (r[:, None] * D * s).astype(np.float32).astype(float)


def _column_check(G, blocks, dB, dC):
    nz, n = dB.shape
    mid = nz // 2
    worst = share = 0.0
    for j in range(nz):
        r, s, D = blocks[j]
        S = np.zeros((n, n))
        B = D.copy()
        for side in ([-1] if j < mid else [1] if j > mid else [-1, 1]):
            k = j + side
            if not 0 <= k < nz:
                continue
            out, back = (dC[j], dB[k]) if side < 0 else (dB[j], dC[k])
            term = (r * out * blocks[k][1])[:, None] * G[k].astype(float) * (blocks[k][0] * back * s)
            B -= term
            S += np.abs(term)
        ref = np.linalg.inv(B)
        tol = 16 * 2.0 ** -24 * (np.abs(ref) @ (np.abs(D) + S) @ np.abs(ref)).max()
        worst = max(worst, np.abs(G[j] - ref).max() / tol)
        share = max(share, S.max() / np.abs(D).max())
    return worst, share


@pytest.mark.parametrize('species', [69] + sorted(NETS))
def test_factors(species):
    from vulcan_gb300.solver import ColumnBatch, GPUNetwork, Ros2Handle
    net = _network(species)
    items = []
    for fast in (False, True):
        for nz in (2, 7, 8):
            specs = configs.config4_columns(sorted(net.photo_index()), ncols=1, nz=nz)
            it = batch.build_items(specs, net)
            if fast:                         # exchange between layers at 1e8 / s (1 / dt)
                specs[0].Kzz = 1e8 * it[0]['col'].dzi ** 2
                it = batch.build_items(specs, net)
            items += it
    gn = GPUNetwork(net, ATOMS)
    b = ColumnBatch(items, net.ni)
    h = Ros2Handle(gn, b.ncols, b.L, precision=capi.VK_PREC_MIXED)
    h.set_columns(b)
    rows, cols = gn.jac_pattern()
    n, dt = net.ni, 1e-8
    for variant in [-1] + [t for t, cap in enumerate(capi.LU32_TILING_CAP) if cap >= n]:
        h.set_launch(capi.VK_TUNE_LU32, 0, variant)
        h.attempt(dt)
        assert h.refine_stats()[1] == 0
        jv, dA, dB, dC = h.lhs()
        G = np.empty((b.L, n * n), dtype=np.float32)
        capi.check(capi.lib().vk_get_lu32(h.h, capi.ptr(G, capi.C.c_float)), h.h)
        G = G.reshape(b.L, n, n)
        for c in range(b.ncols):
            o, e = b.off[c], b.end[c]
            blocks = [_scaled(jv[l], dA[l], dt, rows, cols, n) for l in range(o, e)]
            worst, share = _column_check(G[o:e], blocks, dB[o:e], dC[o:e])
            assert worst <= 1.0, (variant, c)
            assert c < 3 or share > 0.01
    h.close()
