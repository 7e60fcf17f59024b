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
    # sums of n non-negative products, each side at most n roundings of 2^-24: rows of at most 3 x 4 x 15 elements, and
    # for a voxel at most 2 lines a view and ring pair with every timing bin
    nf, nb = 180, 2 * 32 * rings * 5 * bins
    for subset in [(0, 1), (1, 3)]:
        got = proj.projdata_from_device_layout(proj.forward_dev(xd, subset_num=subset[0], num_subsets=subset[1])).cpu().numpy()
        ref = orc.forward(x, *subset)
        assert np.all(np.abs(got - ref) <= 2 * nf * 2.0 ** -24 * np.abs(ref) + 1e-12)
        y = np.random.default_rng(2).uniform(0.5, 1.5, proj.projdata_size).astype(np.float32)
        yd = proj.projdata_to_device_layout(torch.from_numpy(y).cuda())
        ref = orc.back(y, *subset)
        for mode in (_abi.BACKPROJECT_ATOMIC, _abi.BACKPROJECT_DETERMINISTIC):
            got = proj.image_from_device_layout(proj.back_dev(yd, subset_num=subset[0], num_subsets=subset[1],
                                                              mode=mode)).cpu().numpy()
            assert np.all(np.abs(got - ref) <= 2 * nb * 2.0 ** -24 * np.abs(ref) + 1e-6 * ref.max())
