"""k_rates takes tiles of one, two or four layers by the number of layers: the
right-hand side of the same columns alone (one layer a tile), in a small batch
(two) and in a large one (four) -- with ragged ends, tiles that span columns
and the boundary fluxes -- is the same bit for bit, and so is an attempt in
which only some columns take part."""
import os

import numpy as np
import pytest

from conftest import GOLDEN
from test_two_sided_solve import _item
from vulcan_gb300 import capi
from vulcan_gb300.network import Network

pytestmark = pytest.mark.gpu
NZ = (9, 14, 21, 3)


@pytest.fixture(scope='module', autouse=True)
def built():
    from vulcan_gb300 import _build
    _build.build()


def _handle(net, atoms, items):
    from vulcan_gb300.solver import ColumnBatch, GPUNetwork, Ros2Handle
    b = ColumnBatch(items, net.ni)
    h = Ros2Handle(GPUNetwork(net, atoms), len(items), b.L)
    h.set_columns(b)
    return b, h


@pytest.mark.parametrize('name', ['CHO_thermo', 'NCHO_thermo', 'SYN150_photo'])
def test_tile_size_does_not_change_a_layer(name):
    net = Network.from_npz(os.path.join(GOLDEN, 'net_%s.npz' % name))
    items = [_item(net, name, nz, seed=nz) for nz in NZ]
    atoms = items[0][0].atom_list
    items = [it for _, it in items]
    ref = None
    for ncols in (4, 40, 170):                   # 47, 470 and about 2000 layers
        b, h = _handle(net, atoms, [items[c % 4] for c in range(ncols)])
        f = b.split(h.rhs(flags=capi.VK_F_MOLDIFF | capi.VK_F_TOPFLUX | capi.VK_F_BOTFLUX))
        sol = b.split(h.attempt(1e-8)['sol'])
        h.close()
        if ref is None:
            ref = (f, sol)
        for c in range(ncols):
            np.testing.assert_array_equal(f[c], ref[0][c % 4])
            np.testing.assert_array_equal(sol[c], ref[1][c % 4])
