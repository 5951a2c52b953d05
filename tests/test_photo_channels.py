"""Photolysis channels that name one rate: each has its J, and the rate is the last
one's -- channels that one thread, one pass or two passes of the J kernel hold, at the
layer counts of both its forms."""
import os

import numpy as np
import pytest

from conftest import GOLDEN
from vulcan_gb300 import batch, configs, photo
from vulcan_gb300.network import Network

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('ncols', [1, 20])
def test_the_last_channel_of_a_rate_counts(ncols):
    from vulcan_gb300 import _build
    _build.build()
    net = Network.from_npz(os.path.join(GOLDEN, 'net_NCHO_photo.npz'))
    t = photo.PhotoTables.from_fixture(np.load(os.path.join(GOLDEN, 'golden_c1rt.npz')))
    specs = [configs.config1(sorted(net.photo_index()), nz=131, seed=5)] * ncols
    items = batch.build_items(specs[:1], net) * ncols
    # the first 40 channels twice more, scaled: 128 channels for 48 rates
    t.ch_sp, t.ch_br = list(t.ch_sp), list(t.ch_br)
    nch = len(t.ch_sp)
    for f in (2.0, 3.0):
        t.ch_sp += t.ch_sp[:40]
        t.ch_br += t.ch_br[:40]
        t.cross_J = np.concatenate([t.cross_J, f * t.cross_J[:40]])
    h, b = batch.make_batch_handle(net, items, specs[0].atom_list)
    photo.attach(h, t, net)
    pidx = net.photo_index()
    last = {(s, r): c for c, (s, r) in enumerate(zip(t.ch_sp, t.ch_br))}
    for _ in range(3):
        h.photo_update()
        _, _, J = h.photo_get()
        k = h.k()
        for key, c in last.items():
            np.testing.assert_array_equal(k[:, pidx[key] - 1], J[:, c] * t.f_diurnal)
    lit = J[:, :40] > 1e-300                 # the three channels of a rate differ
    assert lit.any() and np.all(J[:, nch:nch + 40][lit] > 1.9 * J[:, :40][lit])
    assert min(last.values()) == 40 and max(last.values()) == nch + 79
    h.close()
