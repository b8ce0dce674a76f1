"""The Siddon pair by detector columns (untilted detectors) against the FP64
oracle: sizes at the edges of its groups of 4 columns and 32 rows, rays that
enter or leave through the top and bottom, miss the volume or pass beside it,
a detector running downwards, anisotropic voxels; and calls on two streams,
which share the plan's volume copy."""
import numpy as np
import pytest

from fdk_cuda_impl_b200.geometry import CircularScan, VolumeGrid
from tests import cases as K

pytestmark = pytest.mark.gpu

# A length's two ends are FP32 distances below 128 mm from the middle of the ray:
# rms 2.2e-6 mm each, 3.1e-6 of a voxel a millimetre wide, which is the relative
# error of a backprojection of white noise.  A projection averages it over its
# segments (16 and more, of values that differ by a half), beside its FP32 sum
BP_TOL = 3.1e-6
FP_TOL = 6e-7

CASES = [
    # views, nu, nv, pixel u, pixel v, (nx, ny, nz), voxel, flipped
    (9, 1, 1, 2.0, 2.0, (5, 4, 1), (1.0, 1.0, 1.0), False),
    (12, 7, 33, 2.0, 2.0, (16, 19, 3), (1.0, 1.0, 1.0), False),
    (11, 30, 65, 4.0, 4.0, (21, 30, 12), (1.0, 1.2, 0.9), True),
    (10, 65, 129, 1.1, 1.3, (37, 29, 30), (0.8, 0.9, 1.1), False),
    (8, 40, 40, 1.6, 6.0, (24, 24, 90), (1.0, 1.0, 0.7), False),
    (8, 40, 40, 1.6, 30.0, (24, 24, 90), (1.0, 1.0, 0.2), False),  # climbs a voxel a segment: ray by ray
]


@pytest.mark.parametrize("case", CASES)
def test_siddon_pair_matches_oracle(oracle, cuda_device, case):
    import torch
    from fdk_cuda_impl_b200.projectors import JosephPlan
    views, nu, nv, pu, pv, n, vox, flipped = case
    scan = CircularScan(views, views, 500.0, 1000.0, nu, nv, pu, pv, start_angle_rad=0.05)
    grid = VolumeGrid(*n, vox, (0.4, -0.7, 0.2))
    table = scan.views()
    if flipped:
        table["detS"][:, :3] += (nv - 1) * table["detV"][:, :3]
        table["detV"][:, :3] *= -1
    vol = K.oracle_volume(oracle, grid)
    x, y = oracle.uniform(grid.shape, 0.0, 1.0, 3), oracle.normal((views, nv, nu), 4)
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    plan = JosephPlan(table, nu, nv, grid)
    fp, bp = plan.forward_siddon(xd), plan.backproject_siddon(yd)
    ref_fp, ref_bp = oracle.siddon_fp(table, nu, nv, vol, x), oracle.siddon_bp(table, nu, nv, vol, y)
    assert K.rel_rmse(fp.cpu().numpy(), ref_fp) <= FP_TOL
    assert K.rel_rmse(bp.cpu().numpy(), ref_bp) <= BP_TOL
    twice = plan.forward_siddon(xd, fp.clone(), accumulate=True)
    assert K.rel_rmse(twice.cpu().numpy(), 2 * ref_fp) <= FP_TOL
    both = plan.backproject_siddon(yd, bp.clone(), accumulate=True)
    assert K.rel_rmse(both.cpu().numpy(), 2 * ref_bp) <= BP_TOL
    # two streams in turn
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    out = []
    for i in range(6):
        with torch.cuda.stream(streams[i % 2]):
            out.append(plan.forward_siddon(xd) if i % 3 else plan.backproject_siddon(yd))
    torch.cuda.synchronize()
    for i, o in enumerate(out):
        assert K.rel_rmse(o.cpu().numpy(), ref_fp if i % 3 else ref_bp) <= BP_TOL
    # a captured call
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        gp, gb = plan.forward_siddon(xd), plan.backproject_siddon(yd)
    graph.replay()
    torch.cuda.synchronize()
    assert K.rel_rmse(gp.cpu().numpy(), ref_fp) <= FP_TOL
    assert K.rel_rmse(gb.cpu().numpy(), ref_bp) <= BP_TOL
    # a voxel that no ray of a missing column reads does not leak into it
    if n[0] > 20:
        bad = xd.clone()
        bad[:, 0, 0] = float("nan")
        hit = plan.forward_siddon((xd * 0 + 1) * (~torch.isfinite(bad)))
        assert torch.isfinite(plan.forward_siddon(bad)[hit == 0]).all()
    plan.close()


@pytest.mark.parametrize("n", [21, 48, 75])
def test_infinite_values_stay_where_rays_cross(cuda_device, n):
    # infinite pixels make infinite exactly the voxels that their rays cross,
    # infinite voxels the pixels whose rays cross them; no NaN (infinity times a
    # length of zero), no -inf (a length below zero)
    import torch
    from fdk_cuda_impl_b200.projectors import JosephPlan
    scan = CircularScan(9, 9, 500.0, 1000.0, n + 5, n, 300.0 / n, 280.0 / n, start_angle_rad=0.03)
    grid = VolumeGrid(n, n + 3, n - 7, (128.0 / n,) * 3, (0.4, -0.7, 0.2))
    plan = JosephPlan(scan.views(), n + 5, n, grid)

    def check(apply, data):
        one = apply(data)
        inf = apply(torch.where(data > 0, torch.inf, 0.0))
        assert float(one.min()) >= 0 and float(one.max()) > 0
        assert not torch.isnan(inf).any() and float(inf.min()) >= 0
        assert torch.equal(one != 0, torch.isinf(inf))

    for k in range(9):
        y = torch.zeros(plan.proj_shape, device="cuda")
        y[k] = 1.0
        check(plan.backproject_siddon, y)
    for at in [(n // 2 - 3, n // 2, n // 2), (n // 3, n // 4, n // 2), (n // 2, n // 2, n // 5)]:
        x = torch.zeros(grid.shape, device="cuda")
        x[tuple(slice(i - 1, i + 2) for i in at)] = 1.0
        check(plan.forward_siddon, x)
    plan.close()
