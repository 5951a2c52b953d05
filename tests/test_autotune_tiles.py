"""The autotuner measures each launch once: LU32 variants that come to the same
register tiling are not told apart by noise."""
import os
import re

import pytest

from test_autotune import FakeHandle
from vulcan_gb300 import _build, autotune, capi


def test_tiles_are_those_of_the_kernel():
    with open(os.path.join(_build.CSRC, 'vk_lu32.cu')) as f:
        src = f.read()
    caps = re.search(r'kTileCap\[6\] = \{([^}]*)\}', src).group(1)
    assert tuple(int(c) for c in caps.split(',')) == autotune.LU32_TILES
    caps = re.search(r'kVariantCap\[6\] = \{([^}]*)\}', src).group(1)
    assert tuple(int(c) for c in caps.split(',')) == capi.LU32_TILING_CAP


@pytest.mark.parametrize('ni,tiles', [(41, {48, 96, 128, 160}), (69, {72, 96, 128, 160}), (100, {128, 160}),
                                      (112, {128, 160}), (150, {160})])
def test_each_launch_is_measured_once(ni, tiles):
    tried = []

    class Handle(FakeHandle):
        def set_launch(self, kernel, ctas_per_sm=0, variant=-1):
            super().set_launch(kernel, ctas_per_sm, variant)
            if kernel == capi.VK_TUNE_LU32 and ctas_per_sm:
                tried.append((ctas_per_sm, autotune.lu32_tile(ni, variant)))

    autotune.tune(Handle(ni, lambda k, c, v: 0.0 if c == 0 else 1.0), 1e-3, repeats=1, kernels=('lu32',))
    assert sorted(tried) == sorted((c, t) for c in autotune.CTAS_PER_SM for t in tiles)
