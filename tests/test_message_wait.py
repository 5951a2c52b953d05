"""A CTA of the FP64 factorisation that waits in vain for another CTA's message
ends its column with VK_ETIMEOUT, stores nothing of the void block and leaves the
kernel with its whole cluster: with a wait limit of no polls every shared block
gives up, in clusters of eight, four and two CTAs and in the kernel that shares
only the long half-columns.  The handle then solves as a new one does."""
import os

import numpy as np
import pytest

from conftest import GOLDEN
from test_two_sided_solve import _item
from vulcan_gb300 import capi, configs
from vulcan_gb300.network import Network

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module', autouse=True)
def built():
    from vulcan_gb300 import _build
    _build.build()


# (CTAs that share a block: 8, 4, 2; 50 columns: the 32 longest halves in pairs)
@pytest.mark.parametrize('name,ncols', [('NCHO_thermo', 1), ('NCHO_thermo', 3), ('NCHO_thermo', 15),
                                        ('NCHO_thermo', 33), ('NCHO_thermo', 50), ('SYN150_photo', 2)])
def test_a_message_that_never_comes(name, ncols):
    from vulcan_gb300.solver import ColumnBatch, GPUNetwork, Ros2Handle, ctrl_from
    net = Network.from_npz(os.path.join(GOLDEN, 'net_%s.npz' % name))
    items = [_item(net, name, nz, seed=nz) for nz in (9, 14, 21)]
    atoms = items[0][0].atom_list
    items = [items[c % 3][1] for c in range(ncols)]
    b = ColumnBatch(items, net.ni)
    ctrl = ctrl_from(None, gs=configs.GS, Rp=configs.RP)

    def handle():
        h = Ros2Handle(GPUNetwork(net, atoms), ncols, b.L)
        h.set_columns(b)
        h.set_atom_ini(np.stack([it['atom_ini'] for it in items]))
        return h

    def run(h):
        h.set_columns(b)
        h.run(ctrl, max_steps=2, timeout_s=100)
        return h.state()['y']

    h = handle()
    ref = run(h)
    h.close()
    h = handle()
    for _ in range(2):
        h.set_wait_limit(0)
        with pytest.raises(capi.VkError) as e:
            run(h)
        assert e.value.code == capi.VK_ETIMEOUT
        h.set_wait_limit()
        np.testing.assert_array_equal(run(h), ref)
    h.close()


@pytest.mark.parametrize('precision', [capi.VK_PREC_FP64, capi.VK_PREC_MIXED])
def test_an_attempt_reports_it(precision):
    from vulcan_gb300.solver import ColumnBatch, GPUNetwork, Ros2Handle
    net = Network.from_npz(os.path.join(GOLDEN, 'net_NCHO_thermo.npz'))
    spec, it = _item(net, 'NCHO_thermo', 14)
    b = ColumnBatch([it], net.ni)
    h = Ros2Handle(GPUNetwork(net, spec.atom_list), 1, b.L, precision=precision)
    h.set_columns(b)
    h.set_route(1e-9)                            # mixed: this step is solved in FP64
    ref = h.attempt(1e-8)
    h.set_wait_limit(0)
    with pytest.raises(capi.VkError) as e:
        h.attempt(1e-8)
    assert e.value.code == capi.VK_ETIMEOUT
    h.set_wait_limit()
    np.testing.assert_array_equal(h.attempt(1e-8)['sol'], ref['sol'])
    h.close()


@pytest.mark.parametrize('ncols', [1, 50])
def test_ctas_per_sm_leave_the_sharing_as_it_is(ncols):
    """A number of CTAs per SM (a tuning file's, say) does not take from the long halves
    of a batch the CTAs they share: with no polls allowed it fails like the default."""
    from vulcan_gb300.solver import ColumnBatch, GPUNetwork, Ros2Handle
    net = Network.from_npz(os.path.join(GOLDEN, 'net_NCHO_thermo.npz'))
    items = [_item(net, 'NCHO_thermo', nz, seed=nz) for nz in (9, 14, 21)]
    b = ColumnBatch([items[c % 3][1] for c in range(ncols)], net.ni)
    h = Ros2Handle(GPUNetwork(net, items[0][0].atom_list), ncols, b.L)
    h.set_columns(b)
    ref = h.attempt(1e-8)
    for ctas in (1, 2, 4):
        h.set_launch(capi.VK_TUNE_LU64, ctas)
        h.set_launch(capi.VK_TUNE_SWEEP64, ctas)
        np.testing.assert_array_equal(h.attempt(1e-8)['sol'], ref['sol'])
        h.set_wait_limit(0)
        with pytest.raises(capi.VkError) as e:
            h.attempt(1e-8)
        assert e.value.code == capi.VK_ETIMEOUT
        h.set_wait_limit()
    h.close()


def test_limit_is_checked():
    from vulcan_gb300.solver import GPUNetwork, Ros2Handle
    net = Network.from_npz(os.path.join(GOLDEN, 'net_CHO_thermo.npz'))
    h = Ros2Handle(GPUNetwork(net, ['H', 'O', 'C']), 1, 10)
    with pytest.raises(capi.VkError) as e:
        h.set_wait_limit(1 << 23)
    assert e.value.code == capi.VK_EINVAL
    h.close()
