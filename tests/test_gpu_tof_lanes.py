"""TOF projections with the timing bins over the lanes (csrc/tof.cu) against the oracle at the edges of their rule: lines of
1 to 16 axial positions (17: the grouped kernels), timing bins that fill a lane's groups or leave one over, and the most
that fit (24 a lane, 96 an element; more: the grouped kernels)."""
import dataclasses

import numpy as np
import pytest

from stir_b200 import _abi
from stir_b200 import geometry as G

pytestmark = pytest.mark.gpu

# rings, timing bins
CASES = [(1, 3), (2, 5), (3, 96), (3, 97), (5, 32), (8, 4), (11, 33), (16, 31), (16, 48), (16, 49), (17, 9)]


@pytest.mark.parametrize("rings,bins", CASES)
def test_tof_matches_oracle(rings, bins, cuda_device):
    import torch
    from oracle.oracle import Oracle
    from stir_b200.projectors import RayTracingProjector
    sc = G.Scanner(rings, 64, 100.0, 0.0, 4.0, float(np.float32(np.pi * 100.0 / 64)), 0.0, 400.0, 1400.0 / bins, bins)
    pdi = dataclasses.replace(G.ProjDataInfoCTI(sc, 1, min(rings - 1, 2), 32, 9), tof_mash_factor=1)
    img = G.ImageGeometry(2 * rings - 1, 15, 15, (2.0, 6.0, 6.0))
    proj = RayTracingProjector(pdi, img, device=cuda_device)
    orc = Oracle(proj.geometry)
    x = np.random.default_rng(1).uniform(0.5, 1.5, img.shape).astype(np.float32)
    xd = proj.image_to_device_layout(torch.from_numpy(x).cuda())
    # a float sum of n non-negative products in two orders: each addition rounds by at most 2^-24 of the running value, with
    # either sign, 0.6 of that on average; 6 standard deviations of both sides' sum.  Rows of at most 3 x 4 x 15 elements; a
    # voxel meets up to 3 tangential positions a view, 5 segments and 2 axial positions of each, with every timing bin
    def bound(n):
        return 6 * 0.6 * 2.0 ** -24 * (2 * n) ** 0.5
    lines = 32 * 3 * 5 * 2
    for subset in [(0, 1), (1, 3)]:
        got = proj.projdata_from_device_layout(proj.forward_dev(xd, subset_num=subset[0], num_subsets=subset[1])).cpu().numpy()
        ref = orc.forward(x, *subset)
        assert np.all(np.abs(got - ref) <= bound(180) * np.abs(ref) + 1e-12)
        y = np.random.default_rng(2).uniform(0.5, 1.5, proj.projdata_size).astype(np.float32)
        _check_back(proj, orc, y, subset, bound(lines * bins))
    # one timing bin at a time, so that none hides behind the others: the ends of the data and of the kernel's passes
    per = proj.projdata_size // bins
    passes = -(-bins // 32)
    size = -(-bins // passes)
    size = next(s for s in (8, 16, 20, 24, 32) if s >= size)
    for k in sorted({0, 1, bins // 2, bins - 1} | {b for p in range(1, passes) for b in (p * size - 1, p * size) if b < bins}):
        y = np.zeros(proj.projdata_size, np.float32)
        y[k * per:(k + 1) * per] = np.random.default_rng(3 + k).uniform(0.5, 1.5, per)
        _check_back(proj, orc, y, (0, 1), bound(lines))


def _check_back(proj, orc, y, subset, tolerance):
    import torch
    yd = proj.projdata_to_device_layout(torch.from_numpy(y).cuda())
    ref = orc.back(y, *subset)
    for mode in (_abi.BACKPROJECT_ATOMIC, _abi.BACKPROJECT_DETERMINISTIC):
        got = proj.image_from_device_layout(proj.back_dev(yd, subset_num=subset[0], num_subsets=subset[1], mode=mode)).cpu().numpy()
        assert np.all(np.abs(got - ref) <= tolerance * np.abs(ref) + 1e-6 * ref.max())
