"""ss_kokkos_icp_noalloc at the ends of what its fixed scratch holds: the most
pixels in the longest and the flattest image, where the quotient tables of
columns and rows are largest, bit for bit as ss_kokkos_icp."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("rows,cols", [(12, 25600), (25600, 12), (13, 23630), (480, 640)])
def test_noalloc_scratch_holds_every_shape(rows, cols, kind):
    from superscanner_gb300 import kokkos_icp
    from superscanner_gb300.icp import kokkos_icp_noalloc
    i, j = np.mgrid[0:rows, 0:cols]
    d = (1000 + 200 * np.sin(i / 7.0) + 200 * np.cos(j / 9.0)).astype(np.uint16)
    dev = torch.from_numpy(d.view(np.int16)).cuda()
    intr = (0.9 * max(rows, cols), 0.9 * max(rows, cols), cols / 2 - 0.5, rows / 2 - 0.5)
    tx = np.eye(4)
    tx[:3, 3] = 0.2 / intr[0], 0.1 / intr[1], 0.004
    a, b = (fn(dev, dev, tx, np.eye(4), kind, intr) for fn in (kokkos_icp, kokkos_icp_noalloc))
    assert np.isfinite(a[0]).all() and a[1] < 0.05  # 0 where the pair, one image, comes back to itself
    assert np.array_equal(a[0], b[0]) and a[1] == b[1]
