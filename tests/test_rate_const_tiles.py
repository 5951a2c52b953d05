"""vk_compute_k takes one layer or four at a time by the number of layers, and
the pairs of a large network in several chunks: a batch large enough for tiles
of four (ragged columns, a last tile that is not full) against the host
restatement, and against the same columns alone (one layer at a time), bit for
bit.

Tolerance: that of the rate-constant tests (2e-12: exp / pow / log of two math
libraries, more where exp's argument is large)."""
import os

import numpy as np
import pytest

from helpers import network
from test_rate_consts import ATOMS
from vulcan_gb300 import batch, configs, synthnet
from vulcan_gb300.network import Network

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module', autouse=True)
def built():
    from vulcan_gb300 import _build
    _build.build()


def _k(net, items):
    h, b = batch.make_batch_handle(net, items, ATOMS)
    h.set_rate_params(net)
    h.compute_k()
    k = h.k()
    h.close()
    return k


def _check(net, items, repeat):
    host = np.concatenate([it['k'].T for it in items])
    one = _k(net, items)
    np.testing.assert_allclose(one, host, rtol=2e-12, atol=1e-290)
    many = _k(net, items * repeat)
    assert many.shape[0] >= 4 * 152
    np.testing.assert_array_equal(many, np.concatenate([one] * repeat))


def test_thermo_network():
    net = network('c2')
    items = batch.build_items(configs.config2_columns(ncols=3, seed=7, nz_range=(30, 61)), net)
    _check(net, items, 15)


def test_synthetic_network_in_chunks():
    d = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), '_build', 'tests', 'syn150')
    net = Network.from_file(synthnet.generate(d), use_photo=True)
    items = batch.build_items(configs.config4_columns(sorted(net.photo_index()), ncols=2, nz=41), net)
    _check(net, items, 16)
