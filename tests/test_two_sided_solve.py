"""The two-sided FP64 block solve at the sizes where it can go wrong: columns
of two to seven layers (an empty half, halves of one layer), block sizes around
the warp and even/odd edges (38 to 150 species), and the same column alone and
in batches whose blocks are shared by eight, four, two CTAs or one: the result
does not depend on how many share it.

Tolerance: the per-attempt bar of the parity tests (1e-10 in the floor metric,
these early steps are well conditioned); between batch sizes, bit for bit."""
import os

import numpy as np
import pytest

from conftest import GOLDEN
from helpers import atm_from_column, floor_err
from oracle import ros2 as O
from vulcan_gb300 import batch, configs
from vulcan_gb300.network import Network

pytestmark = pytest.mark.gpu
ATOMS = ['H', 'O', 'C', 'He', 'N']


@pytest.fixture(scope='module', autouse=True)
def built():
    from vulcan_gb300 import _build
    _build.build()


def _item(net, name, nz, seed=3):
    rng = np.random.default_rng(seed)
    pco = configs.log_p_grid(nz)
    J = None
    if net.use_photo:
        J = configs.photo_J_profile(rng, pco, sorted(net.photo_index()))
    atoms = [a for a in ATOMS if {'N': 'N2', 'He': 'He'}.get(a, 'H2') in net.species]
    mix = {s: x for s, x in configs.solar_mix(with_n='N2' in net.species).items() if s in net.species}
    spec = configs.ColumnSpec(network=name, use_photo=net.use_photo, pco=pco,
                              Tco=configs.linear_logp_T(pco, 2000., 1000.),
                              Kzz=np.full(nz - 1, 1e8), const_mix=mix, atom_list=atoms,
                              conver_ignore=[], photo_J=J)
    return spec, batch.build_items([spec], net)[0]


def _attempt(net, atoms, items, dt):
    from vulcan_gb300.solver import ColumnBatch, GPUNetwork, Ros2Handle
    b = ColumnBatch(items, net.ni)
    h = Ros2Handle(GPUNetwork(net, atoms), len(items), b.L)
    h.set_columns(b)
    out = h.attempt(dt)
    h.close()
    return b.split(out['sol']), out['delta']


@pytest.mark.parametrize('name,nz', [('CHO_thermo', 2), ('CHO_thermo', 3), ('CHO_thermo', 4),
                                     ('CHO_photo_lowT', 7), ('NCHO_earth_photo', 6),
                                     ('TiSNCHO_photo', 5), ('SNCHO_DMS_photo_Tsai2024', 4),
                                     ('SYN150_photo', 5)])
def test_short_columns_and_block_sizes(name, nz):
    path = os.path.join(GOLDEN, 'net_%s.npz' % name)
    net = Network.from_npz(path)
    spec, it = _item(net, name, nz)
    dt = 1e-8
    sols, delta = _attempt(net, spec.atom_list, [it], dt)
    on = O.OracleNet.from_npz(path, spec.atom_list)
    r = O.ros2_attempt(on, it['y'], it['ymix'], dt, it['k'], atm_from_column(it['col']), O.Flags(),
                       O.Tol(), 'banded')
    assert floor_err(sols[0], r.sol, it['col'].n_0) <= 1e-10
    if r.delta > 0:
        assert abs(delta[0] / r.delta - 1) <= 1e-6


@pytest.mark.parametrize('name', ['CHO_thermo', 'NCHO_thermo', 'TiSNCHO_photo', 'SYN150_photo'])
def test_batch_size_does_not_change_a_column(name):
    net = Network.from_npz(os.path.join(GOLDEN, 'net_%s.npz' % name))
    items = [_item(net, name, nz, seed=nz) for nz in (9, 14, 21)]
    atoms = items[0][0].atom_list
    items = [it for _, it in items]
    ref = None
    for ncols in (3, 15, 33, 50, 75, 90):
        sols, delta = _attempt(net, atoms, [items[c % 3] for c in range(ncols)], 1e-7)
        if ref is None:
            ref = (sols, delta)
        for c in range(ncols):
            np.testing.assert_array_equal(sols[c], ref[0][c % 3])
            assert delta[c] == ref[1][c % 3]
