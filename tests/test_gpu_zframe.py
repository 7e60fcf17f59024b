"""z-frame projections (csrc/zframe.cu) against the oracle at the sizes where they can go wrong: planes at and beside the
lanes' 32, 64 and 128, rows of several chains (two rays per bin, span 1, a truncated last segment), rectangular images,
several axial samplings per plane; and infinite values."""
import numpy as np
import pytest

from stir_b200 import _abi
from stir_b200 import geometry as G

pytestmark = pytest.mark.gpu


def _geometry(rings, span, delta, dets=64, tang=21, nz=None, ny=23, nx=23, rays=1, planes_per_ring=2, vxy=4.1):
    sc = G.Scanner(rings, dets, 100.0, 0.0, 4.0, float(np.float32(np.pi * 100.0 / dets)))
    pdi = G.ProjDataInfoCTI(sc, span, delta, dets // 2, tang)
    nz = nz or planes_per_ring * (rings - 1) + 1
    img = G.ImageGeometry(nz, ny, nx, (4.0 / planes_per_ring, vxy, vxy))
    return pdi, img, rays


CASES = {
    "one plane": _geometry(1, 1, 0),
    "31 planes": _geometry(16, 3, 10),
    "33 planes": _geometry(17, 3, 16),
    "63 planes": _geometry(32, 11, 27),
    "65 planes": _geometry(33, 11, 32),
    "127 planes": _geometry(64, 11, 60, dets=32, tang=11, ny=11, nx=11),
    "129 planes": _geometry(65, 11, 60, dets=32, tang=11, ny=11, nx=11),
    "two rays": _geometry(12, 5, 11, rays=2),
    "two rays, 63 planes": _geometry(32, 9, 31, rays=2),
    "span 1": _geometry(9, 1, 8),
    "span 1, one plane a ring": _geometry(9, 1, 8, planes_per_ring=1),
    "span 1, 4 planes a ring": _geometry(9, 1, 5, planes_per_ring=4),
    "truncated segment": _geometry(20, 5, 8),
    "rectangular": _geometry(11, 3, 7, ny=19, nx=31),
    "sparse chains": _geometry(59, 7, 41, dets=32, tang=11, ny=61, nx=60, vxy=1.1, rays=2),
    "even image": _geometry(10, 7, 9, ny=24, nx=24, tang=24),
}


@pytest.fixture(scope="module", params=list(CASES), ids=list(CASES))
def case(request, cuda_device):
    from oracle.oracle import Oracle
    from stir_b200.projectors import RayTracingProjector
    pdi, img, rays = CASES[request.param]
    proj = RayTracingProjector(pdi, img, num_tangential_LORs=rays, device=cuda_device)
    return pdi, img, proj, Oracle(proj.geometry)


def _bound(orc):
    """Relative error of a float sum of n non-negative products against another order of the same sum: each of the n additions
    rounds by at most half a unit (2^-24 of the running value), with either sign, 0.6 of that on average; 6 standard deviations
    of both sides' sum.  n: the longest row (up to 3 planes a column), and for a voxel the lines through it: two tangential
    positions a view, and up to four axial positions of each segment within a plane of it."""
    g = orc.geometry
    n = max(3 * (g.nx + g.ny), 2 * 4 * g.num_views * (2 * g.max_segment_num + 1))
    return 6 * 0.6 * 2.0 ** -24 * (2 * n) ** 0.5


@pytest.mark.parametrize("subset", [(0, 1), (1, 4)])
def test_forward_and_back_match_oracle(case, subset):
    import torch
    pdi, img, proj, orc = case
    x = np.random.default_rng(3).uniform(0.5, 1.5, img.shape).astype(np.float32)
    xd = proj.image_to_device_layout(torch.from_numpy(x).cuda())
    got = proj.projdata_from_device_layout(proj.forward_dev(xd, subset_num=subset[0], num_subsets=subset[1])).cpu().numpy()
    ref = orc.forward(x, *subset)
    assert np.all(np.abs(got - ref) <= _bound(orc) * np.abs(ref) + 1e-12)
    y = np.random.default_rng(4).uniform(0.5, 1.5, proj.projdata_size).astype(np.float32)
    yd = proj.projdata_to_device_layout(torch.from_numpy(y).cuda())
    ref = orc.back(y, *subset)
    for mode in (_abi.BACKPROJECT_ATOMIC, _abi.BACKPROJECT_DETERMINISTIC):
        got = proj.image_from_device_layout(proj.back_dev(yd, subset_num=subset[0], num_subsets=subset[1],
                                                          mode=mode)).cpu().numpy()
        # fixed point: at most one unit of the grid (2^-40 of the largest sum and less) a line's part, within the slack
        assert np.all(np.abs(got - ref) <= _bound(orc) * np.abs(ref) + 1e-6 * ref.max() * (mode != _abi.BACKPROJECT_ATOMIC))
    assert proj.device_status() == 0


def test_infinite_values_reach_their_rows_only(case):
    """An infinite voxel makes the lines through it infinite and no others NaN; an infinite datum its row's voxels."""
    import torch
    pdi, img, proj, orc = case
    x = np.random.default_rng(5).uniform(0.5, 1.5, img.shape).astype(np.float32)
    x[img.nz // 2, img.ny // 2, img.nx // 2 + 2] = np.inf
    xd = proj.image_to_device_layout(torch.from_numpy(x).cuda())
    got = proj.projdata_from_device_layout(proj.forward_dev(xd)).cpu().numpy()
    ref = orc.forward(x)
    assert not np.isnan(got).any() and np.array_equal(np.isinf(got), np.isinf(ref))
    y = np.random.default_rng(6).uniform(0.5, 1.5, proj.projdata_size).astype(np.float32)
    y[proj.projdata_size // 3] = np.inf
    yd = proj.projdata_to_device_layout(torch.from_numpy(y).cuda())
    got = proj.image_from_device_layout(proj.back_dev(yd)).cpu().numpy()
    ref = orc.back(y)
    assert not np.isnan(got).any() and np.array_equal(np.isinf(got), np.isinf(ref))


def test_calls_on_two_streams(cuda_device):
    """Two streams project through one projector at once: every call has padded images of its own."""
    import torch
    from stir_b200.projectors import RayTracingProjector
    pdi, img, _ = CASES["63 planes"]
    proj = RayTracingProjector(pdi, img, device=cuda_device)
    xs = [torch.rand(proj.device_image_shape, device="cuda", generator=torch.Generator("cuda").manual_seed(k))
          for k in range(2)]
    ref = [proj.forward_dev(x) for x in xs]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    outs = [[proj.empty_projdata() for _ in range(8)] for _ in range(2)]
    torch.cuda.synchronize()
    for r in range(8):
        for k in range(2):
            proj.forward_dev(xs[k], out=outs[k][r], stream=streams[k])
    torch.cuda.synchronize()
    for k in range(2):
        for o in outs[k]:
            assert torch.equal(o, ref[k])


# Calls with so few items that warps share them: one of many subsets, paths of 20 to 250 columns, with 1, 2 and
# 4 planes a lane, two rays, several chain groups, 16 warps an item; and the number of subsets
SHARED = {
    "1 plane a lane": (_geometry(8, 3, 7, dets=96, tang=40, ny=90, nx=90, vxy=2.00), 12),
    "1 plane, 16 warps": (_geometry(8, 3, 4, dets=96, tang=12, ny=200, nx=200, vxy=0.90), 24),
    "1 plane, two rays": (_geometry(9, 3, 7, dets=96, tang=40, ny=84, nx=90, vxy=2.00, rays=2), 12),
    "1 plane, span 1": (_geometry(8, 1, 7, dets=96, tang=40, ny=85, nx=85, vxy=2.12), 12),
    "2 planes": (_geometry(21, 5, 17, dets=96, tang=40, ny=80, nx=80, vxy=2.25), 12),
    "2 planes, two rays": (_geometry(23, 7, 17, dets=96, tang=30, ny=90, nx=71, vxy=2.54, rays=2), 12),
    "4 planes": (_geometry(40, 7, 30, dets=96, tang=30, ny=91, nx=91, vxy=1.98), 12),
    "4 planes, two rays": (_geometry(45, 11, 40, dets=96, tang=20, ny=72, nx=72, vxy=2.50, rays=2), 12),
    "4 planes, 8 warps": (_geometry(50, 11, 16, dets=96, tang=8, ny=190, nx=190, vxy=0.95), 24),
    "shorter than the parts": (_geometry(8, 3, 7, dets=96, tang=40, ny=19, nx=19), 12),
}


@pytest.mark.parametrize("name", list(SHARED))
def test_items_shared_by_warps(name, cuda_device):
    import torch
    from oracle.oracle import Oracle
    from stir_b200.projectors import RayTracingProjector
    from stir_b200.subsets import basic_views_in_subset
    (pdi, img, rays), nsub = SHARED[name]
    # at most 8 symmetry operations and 3 chain groups a path: fewer items than half the warps that the GPU runs at a time
    # (148 x 16), so that two warps share an item where a path has ten records
    paths = len(basic_views_in_subset(pdi.num_views, 3, 1, nsub)) * (pdi.num_tangential_poss // 2 + 1)
    assert paths * 8 * 3 <= 148 * 16 // 2 and min(img.nx, img.ny) >= 19
    proj = RayTracingProjector(pdi, img, num_tangential_LORs=rays, device=cuda_device)
    orc = Oracle(proj.geometry)
    x = np.random.default_rng(9).uniform(0.5, 1.5, img.shape).astype(np.float32)
    xd = proj.image_to_device_layout(torch.from_numpy(x).cuda())
    y = np.random.default_rng(10).uniform(0.5, 1.5, proj.projdata_size).astype(np.float32)
    yd = proj.projdata_to_device_layout(torch.from_numpy(y).cuda())
    for subset in (1, 0):
        got = proj.projdata_from_device_layout(proj.forward_dev(xd, subset_num=subset, num_subsets=nsub)).cpu().numpy()
        ref = orc.forward(x, subset, nsub)
        assert np.all(np.abs(got - ref) <= _bound(orc) * np.abs(ref) + 1e-12)
        ref = orc.back(y, subset, nsub)
        for mode in (_abi.BACKPROJECT_ATOMIC, _abi.BACKPROJECT_DETERMINISTIC):
            got = proj.image_from_device_layout(proj.back_dev(yd, subset_num=subset, num_subsets=nsub, mode=mode)).cpu().numpy()
            assert np.all(np.abs(got - ref) <= _bound(orc) * np.abs(ref) + 1e-6 * ref.max() * (mode != _abi.BACKPROJECT_ATOMIC))
    # infinite voxels and data stay in their rows
    x[img.nz // 2, img.ny // 2, img.nx // 2 + 2] = np.inf
    got = proj.projdata_from_device_layout(proj.forward_dev(proj.image_to_device_layout(torch.from_numpy(x).cuda()),
                                                            subset_num=1, num_subsets=nsub)).cpu().numpy()
    ref = orc.forward(x, 1, nsub)
    assert not np.isnan(got).any() and np.array_equal(np.isinf(got), np.isinf(ref))


@pytest.mark.parametrize("name", ["1 plane a lane", "1 plane, span 1", "2 planes, two rays", "4 planes"])
def test_batched_frames_of_shared_items(name, cuda_device):
    """Batched deterministic frames whose items are shared by warps equal their own reconstructions bit for bit, and float ones
    up to the rounding of the back projection's sums."""
    import torch
    from stir_b200.batch import BatchedOSMAPOSL
    from stir_b200.osmaposl import OSMAPOSLReconstruction
    from stir_b200.projectors import RayTracingProjector
    (pdi, img, rays), _ = SHARED[name]
    proj = RayTracingProjector(pdi, img, num_tangential_LORs=rays, device=cuda_device)
    gen = torch.Generator("cuda").manual_seed(13)
    x0 = torch.rand(proj.device_image_shape, device="cuda", generator=gen) + 0.5
    y = proj.forward_dev(x0) * (0.5 + torch.rand(proj.projdata_size, device="cuda", generator=gen))
    add = torch.full_like(y, float(y.mean()))
    for mode in (_abi.BACKPROJECT_DETERMINISTIC, _abi.BACKPROJECT_ATOMIC):
        def recon(n):
            return OSMAPOSLReconstruction(proj, y, additive=add, num_subsets=6, num_subiterations=n, back_projection_mode=mode)
        own, ref = recon(4).set_up(), proj.empty_image().fill_(1.0)
        own.reconstruct(ref)
        batch, xs = BatchedOSMAPOSL(), []
        for n in (4, 4, 2):
            r = recon(n)
            r.sensitivities = own.sensitivities
            xs.append(proj.empty_image().fill_(1.0))
            batch.add(r, xs[-1])
        batch.set_config(kernels=_abi.BATCH_KERNELS_PATHS)
        batch.reconstruct()
        torch.cuda.synchronize()
        batch.close()
        for x in xs[:2]:
            if mode == _abi.BACKPROJECT_DETERMINISTIC:
                assert torch.equal(x, ref)
            else:
                assert float((x - ref).norm() / ref.norm()) <= 4 * 1e-6  # four steps of at most 1e-6 each


def test_forward_sums_are_short(cuda_device):
    """The rounding of the forward sums against 64-bit sums of the same rows: steep paths of about 180 columns, where a sum over
    the whole path, in products of 32 columns, has a relative error of 1.2e-7 (2-norm).  A sum of n values of one size rounds
    n times, by 0.3 of 2^-23 of its running value: sqrt(n / 3) 0.3 2^-23 of the sum if the whole path is one, and with s
    segments 1 / sqrt(s) of 1 / sqrt(s) of that, beside sqrt(s / 3) for adding them: 0.8 2^-24 of about 30 additions (the
    folds and the crossed planes), s = 4, and 0.6 2^-24 for the last rounding and the products'."""
    import torch
    from oracle.oracle import Oracle
    from stir_b200.projectors import RayTracingProjector
    sc = G.Scanner(64, 192, 328.0, 0.0, 4.06, float(np.float32(np.pi * 328.0 / 192)))
    pdi = G.ProjDataInfoCTI(sc, 11, 60, 96, 101)
    img = G.ImageGeometry(127, 172, 172, (2.03, 4.18, 4.18))
    proj = RayTracingProjector(pdi, img, device=cuda_device)
    orc = Oracle(proj.geometry)
    rng = np.random.default_rng(8)
    x = rng.uniform(0.5, 1.5, img.shape).astype(np.float32)
    got = proj.forward_dev(proj.image_to_device_layout(torch.from_numpy(x).cuda())).cpu().numpy()
    x64, g, first = x.astype(np.float64), proj.geometry, 0
    mine, exact = [], []
    for seg in range(-pdi.max_segment_num, pdi.max_segment_num + 1):  # the device layout: [segment][view][tangential][axial]
        nax, ntang = pdi.get_num_axial_poss(seg), pdi.num_tangential_poss
        for _ in range(60):
            view, t, ax = (int(rng.integers(n)) for n in (pdi.num_views, ntang, nax))
            coords, values = orc.row(seg, view, ax, t + pdi.min_tangential_pos_num)
            z, y, xx = coords[:, 0] - g.min_z, coords[:, 1] - g.min_y, coords[:, 2] - g.min_x
            mine.append(got[first + (view * ntang + t) * nax + ax])
            inside = (z >= 0) & (z < img.nz)
            exact.append((x64[z[inside], y[inside], xx[inside]] * values[inside]).sum())
        first += pdi.num_views * ntang * nax
    error = np.linalg.norm(np.array(mine) - np.array(exact)) / np.linalg.norm(exact)
    assert error <= 1.5 * 2.0 ** -24, error


@pytest.mark.parametrize("rays,span", [(1, 1), (2, 3)])
def test_back_sums_are_short(rays, span, cuda_device):
    """The rounding of a voxel's float sum where a path's rows fall into several groups of chains, against the fixed-point sums
    (whose own error is below 3e-8).  Adding N values of one size rounds N times, by 0.3 of 2^-23 of the running value: 0.3
    2^-23 sqrt(N / 3) of the sum (2-norm over the voxels).  One addition a view and column crossed makes N = 1.3 x the views;
    one a group two to three times as many."""
    import torch
    from stir_b200.projectors import RayTracingProjector
    sc = G.Scanner(8, 288, 300.0, 0.0, 4.0, float(np.float32(np.pi * 300.0 / 288)))
    proj = RayTracingProjector(G.ProjDataInfoCTI(sc, span, 7, 144, 64), G.ImageGeometry(15, 64, 64, (2.0, 4.0, 4.0)),
                               num_tangential_LORs=rays, device=cuda_device)
    y = torch.rand(proj.projdata_size, device="cuda", generator=torch.Generator("cuda").manual_seed(11))
    exact = proj.back_dev(y, mode=_abi.BACKPROJECT_DETERMINISTIC).double()
    got = proj.back_dev(y).double()
    error = float((got - exact).norm() / exact.norm())
    assert error <= 0.3 * 2.0 ** -23 * (1.3 * 144 / 3) ** 0.5, error


@pytest.mark.parametrize("case", ["padded images", "image sums"])
def test_captured_calls(case, cuda_device):
    """Calls captured into a graph allocate nothing: the graph can be instantiated twice, which allocation nodes forbid."""
    import torch
    from stir_b200.projectors import RayTracingProjector
    rt = pytest.importorskip("cuda.bindings.runtime")
    if case == "padded images":  # 109 of 128 planes, 1.5 million columns walked
        sc = G.Scanner(55, 192, 200.0, 0.0, 4.0, float(np.float32(np.pi * 200.0 / 192)))
        pdi, img = G.ProjDataInfoCTI(sc, 11, 30, 96, 101), G.ImageGeometry(109, 71, 71, (2.0, 4.0, 4.0))
    else:  # three chain groups
        sc = G.Scanner(8, 96, 100.0, 0.0, 4.0, float(np.float32(np.pi * 100.0 / 96)))
        pdi, img = G.ProjDataInfoCTI(sc, 1, 7, 48, 40), G.ImageGeometry(15, 40, 40, (2.0, 4.0, 4.0))
    proj = RayTracingProjector(pdi, img, device=cuda_device)
    gen = torch.Generator("cuda").manual_seed(12)
    x = torch.rand(proj.device_image_shape, device="cuda", generator=gen)
    y = torch.rand(proj.projdata_size, device="cuda", generator=gen)
    want = proj.forward_dev(x), proj.back_dev(y)
    out, back = proj.empty_projdata(), proj.empty_image()
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()

    def ok(r):
        assert r[0] == rt.cudaError_t.cudaSuccess, r[0]
        return r[1] if len(r) == 2 else None

    ok(rt.cudaStreamBeginCapture(stream.cuda_stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal))
    proj.forward_dev(x, out=out, stream=stream)
    proj.back_dev(y, out=back, stream=stream)
    graph = ok(rt.cudaStreamEndCapture(stream.cuda_stream))
    execs = [ok(rt.cudaGraphInstantiate(graph, 0)) for _ in range(2)]
    for e in execs:
        out.zero_()
        back.zero_()
        torch.cuda.synchronize()
        ok(rt.cudaGraphLaunch(e, stream.cuda_stream))
        stream.synchronize()
        assert torch.equal(out, want[0])
        # two float sums of a voxel in another order: at most 1.3 x 96 views x 3 groups of one size each
        assert float((back - want[1]).norm() / want[1].norm()) <= 2 * 0.3 * 2.0 ** -23 * (1.3 * 96) ** 0.5
    for e in execs:
        ok(rt.cudaGraphExecDestroy(e))
    ok(rt.cudaGraphDestroy(graph))
