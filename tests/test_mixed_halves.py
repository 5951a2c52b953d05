"""The mixed path's factorisation (k_lu32) and refinement (k_refine) work on
the two halves of a column at once: columns of two to seven layers (an empty
half, halves of one layer), block sizes at the edges of the register tilings
(38 to 150 species), the same column alone and in batches, and every register
tiling that holds the block.

Tolerance: the per-attempt bar of the parity tests (1e-10 in the floor metric:
the refinement ends at the FP64 solution); between batch sizes and tilings,
bit for bit."""
import os

import numpy as np
import pytest

from conftest import GOLDEN
from helpers import atm_from_column, floor_err
from oracle import ros2 as O
from test_two_sided_solve import _item
from vulcan_gb300 import capi
from vulcan_gb300.network import Network

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module', autouse=True)
def built():
    from vulcan_gb300 import _build
    _build.build()


def _attempt(net, atoms, items, dt, variant=-1):
    from vulcan_gb300.solver import ColumnBatch, GPUNetwork, Ros2Handle
    b = ColumnBatch(items, net.ni)
    h = Ros2Handle(GPUNetwork(net, atoms), len(items), b.L, precision=capi.VK_PREC_MIXED)
    h.set_columns(b)
    h.set_launch(capi.VK_TUNE_LU32, 0, variant)
    out = h.attempt(dt)
    stats = h.refine_stats()
    h.close()
    return b.split(out['sol']), out['delta'], stats


@pytest.mark.parametrize('name,nz', [('CHO_thermo', 2), ('CHO_thermo', 3), ('CHO_thermo', 4),
                                     ('CHO_photo_lowT', 7), ('NCHO_earth_photo', 6),
                                     ('TiSNCHO_photo', 5), ('SNCHO_DMS_photo_Tsai2024', 4),
                                     ('SYN150_photo', 5)])
def test_short_columns_and_block_sizes(name, nz):
    path = os.path.join(GOLDEN, 'net_%s.npz' % name)
    net = Network.from_npz(path)
    spec, it = _item(net, name, nz)
    dt = 1e-8
    sols, _, (sweeps, fallbacks) = _attempt(net, spec.atom_list, [it], dt)
    assert sweeps >= 1 and fallbacks == 0
    on = O.OracleNet.from_npz(path, spec.atom_list)
    r = O.ros2_attempt(on, it['y'], it['ymix'], dt, it['k'], atm_from_column(it['col']), O.Flags(),
                       O.Tol(), 'banded')
    assert floor_err(sols[0], r.sol, it['col'].n_0) <= 1e-10


@pytest.mark.parametrize('name', ['CHO_thermo', 'NCHO_thermo'])
def test_batch_size_and_tiling_do_not_change_a_column(name):
    net = Network.from_npz(os.path.join(GOLDEN, 'net_%s.npz' % name))
    items = [_item(net, name, nz, seed=nz) for nz in (9, 14, 21)]
    atoms = items[0][0].atom_list
    items = [it for _, it in items]
    fits = [t for t, cap in enumerate(capi.LU32_TILING_CAP) if cap >= net.ni]
    ref = None
    for ncols, variant in [(3, -1), (90, -1), (330, -1)] + [(3, t) for t in fits]:
        sols, delta, _ = _attempt(net, atoms, [items[c % 3] for c in range(ncols)], 1e-7, variant)
        if ref is None:
            ref = (sols, delta)
        for c in range(ncols):
            np.testing.assert_array_equal(sols[c], ref[0][c % 3])
            assert delta[c] == ref[1][c % 3]
