"""The radiative-transfer kernels where their layer tiles are ragged: columns
whose layer counts are no multiple of 8 or 16, tiles that straddle columns and
slot gaps, a masked update that must leave the other columns alone, and batches
on both sides of the line between the four- and the sixteen-layer J kernels.

Tolerances: those of the parity tests (tau 1e-13, J 1e-10 relative)."""
import os

import numpy as np
import pytest

from conftest import GOLDEN
from oracle import photo as OP
from vulcan_gb300 import batch, configs, photo
from vulcan_gb300.network import Network

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('nzs,slotted', [([5, 13, 24], False), ([5, 13, 24], True), ([9], False),
                                         ([131] * 19 + [17], False)])
def test_ragged_columns_and_masks(nzs, slotted):
    from vulcan_gb300 import _build, capi
    _build.build()
    net = Network.from_npz(os.path.join(GOLDEN, 'net_NCHO_photo.npz'))
    t = photo.PhotoTables.from_fixture(np.load(os.path.join(GOLDEN, 'golden_c1rt.npz')))
    rng = np.random.default_rng(len(nzs))
    specs = [configs.config1(sorted(net.photo_index()), nz=nz, seed=5) for nz in nzs]
    items = batch.build_items(specs, net)
    for it in items:
        x = np.maximum(it['ymix'], 10. ** rng.uniform(-14, -6, it['ymix'].shape))
        it['ymix'] = x / x.sum(axis=1, keepdims=True)
        it['y'] = it['ymix'] * it['col'].n_0[:, None]
    h, b = batch.make_batch_handle(net, items, specs[0].atom_list, slot_cap=max(nzs) + 3 if slotted else 0)
    photo.attach(h, t, net)
    mask = np.zeros(len(nzs), dtype=np.int32)
    mask[0] = 1
    h.photo_update(mask)
    _, _, J0 = h.photo_get()
    capi.check(capi.lib().vk_photo_reset(h.h), h.h)
    h.photo_update()
    tau, af, J = h.photo_get()
    np.testing.assert_array_equal(J0[b.off[0]:b.end[0]], J[b.off[0]:b.end[0]])
    h.close()
    sp = {s: i for i, s in enumerate(net.species)}
    ab, sc = [sp[s] for s in t.absp_sp], [sp[s] for s in t.scat_sp]
    for c in sorted({0, len(nzs) // 2, len(nzs) - 1}):
        it, nz, nb = items[c], nzs[c], len(t.bins)
        want = OP.compute_tau(it['y'], it['col'].dz, ab, t.cross, sc, t.cross_scat)
        aflux, _, _ = OP.compute_flux(want, it['ymix'], ab, t.cross, sc, t.cross_scat, t.sflux_top, t.bins,
                                      t.sl_angle, t.edd, np.zeros((nz + 1, nb)), np.zeros((nz + 1, nb)))
        wJ = OP.compute_J(aflux, t.cross_J, t.weights()).T
        o = b.off[c]
        np.testing.assert_allclose(tau[o + c:o + c + nz + 1], want, rtol=1e-13, atol=0)
        big = np.abs(wJ).max(axis=0)
        assert np.all(np.abs(J[o:o + nz] - wJ) <= 1e-10 * (np.abs(wJ) + 1e-12 * big))
