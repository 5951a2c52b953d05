"""Attempts in which only some columns of a batch take part (vk_run: columns that
have taken their steps wait for those whose steps were rejected): each column
ends as it does alone, bit for bit.  Alone its layers are tiles of one and
eight CTAs share its blocks; in the batches tiles of two and four layers mix running
and waiting columns, and blocks are shared by four, two, the long halves' pairs or
not at all."""
import os

import numpy as np
import pytest

from conftest import GOLDEN
from test_two_sided_solve import _item
from vulcan_gb300 import capi, configs
from vulcan_gb300.network import Network

pytestmark = pytest.mark.gpu
NZ = (9, 14, 21, 3)
DT = (1e-10, 1e-3, 1e-8, 1e-1, 1e-10)      # start steps: none to many rejections


@pytest.fixture(scope='module', autouse=True)
def built():
    from vulcan_gb300 import _build
    _build.build()


def _run(net, atoms, items, dt, precision):
    from vulcan_gb300.solver import ColumnBatch, GPUNetwork, Ros2Handle, ctrl_from
    b = ColumnBatch(items, net.ni)
    h = Ros2Handle(GPUNetwork(net, atoms), len(items), b.L, precision=precision)
    h.set_columns(b)
    h.set_atom_ini(np.stack([it['atom_ini'] for it in items]))
    h.set_clock(dt=np.asarray(dt), t=0.0, count=1)
    h.run(ctrl_from(None, gs=configs.GS, Rp=configs.RP), max_steps=3, timeout_s=100)
    st = h.state()
    tries = h.counters()[:, 0].copy()
    h.close()
    return b.split(st['y']), st['dt'], st['t'], tries


@pytest.mark.parametrize('precision', [capi.VK_PREC_FP64, capi.VK_PREC_MIXED])
@pytest.mark.parametrize('ncols', [15, 33, 50, 170])
def test_a_column_ends_as_alone(ncols, precision):
    net = Network.from_npz(os.path.join(GOLDEN, 'net_NCHO_thermo.npz'))
    items = [_item(net, 'NCHO_thermo', nz, seed=nz) for nz in NZ]
    atoms = items[0][0].atom_list
    items = [it for _, it in items]
    kinds = [(c % 4, c % 5) for c in range(ncols)]
    y, dt, t, tries = _run(net, atoms, [items[i] for i, _ in kinds], [DT[d] for _, d in kinds], precision)
    assert tries.max() > tries.min()
    alone = {}
    for c, (i, d) in enumerate(kinds):
        if (i, d) not in alone:
            alone[i, d] = _run(net, atoms, [items[i]], [DT[d]], precision)
        a = alone[i, d]
        np.testing.assert_array_equal(y[c], a[0][0])
        assert (dt[c], t[c], tries[c]) == (a[1][0], a[2][0], a[3][0])
