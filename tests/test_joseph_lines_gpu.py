"""The Joseph line projector (axial-column scans) against the slab projector,
which takes the same samples with the same weights (YKB_JOSEPH_BP=gather keeps
it): both round a sample to FP32 and add in FP64, so they differ by the FP32
rounding of a result.  Sizes at the edges of its groups of 8 detector columns,
32-row warps, 4-slice batches and 16-byte z quads; rows closer and farther than
a voxel; views from below (the detector's rows run downwards); a small detector
that sees part of the volume."""
import numpy as np
import pytest

from fdk_cuda_impl_b200.geometry import CircularScan, VolumeGrid
from tests import cases as K

pytestmark = pytest.mark.gpu

CASES = [
    # views, nu, nv, pixel u, pixel v, (nx, ny, nz), voxel, flipped
    (9, 1, 1, 2.0, 2.0, (5, 4, 1), (1.0, 1.0, 1.0), False),
    (12, 7, 31, 2.0, 2.0, (16, 19, 3), (1.0, 1.0, 1.0), False),
    (11, 8, 32, 3.0, 3.0, (33, 30, 21), (1.0, 1.2, 0.9), True),
    (10, 65, 33, 1.1, 1.3, (37, 41, 30), (0.8, 0.9, 1.1), False),
    (8, 40, 97, 1.6, 0.2, (24, 24, 40), (1.0, 1.0, 1.0), True),     # rows a tenth of a voxel apart
    (8, 40, 24, 1.6, 9.0, (24, 24, 120), (1.0, 1.0, 1.0), False),   # rows 4.5 voxels apart
    (8, 24, 130, 1.6, 14.0, (20, 20, 900), (1.0, 1.0, 1.0), False),  # 7 voxels: the 304-float window
    (6, 30, 500, 1.6, 1.6, (40, 36, 420), (1.0, 1.0, 1.0), False),
    (8, 24, 130, 1.6, 26.0, (20, 20, 1700), (1.0, 1.0, 1.0), False),  # 13: no window, the slab projector
]


@pytest.mark.parametrize("case", CASES)
def test_line_projector_matches_slab_projector(oracle, cuda_device, monkeypatch, case):
    import torch
    from fdk_cuda_impl_b200.projectors import JosephPlan
    views, nu, nv, pu, pv, n, vox, flipped = case
    scan = CircularScan(views, views, 500.0, 1000.0, nu, nv, pu, pv, start_angle_rad=0.05)
    grid = VolumeGrid(*n, vox, (0.4, -0.7, 0.2))
    table = scan.views()
    if flipped:
        table["detS"][:, :3] += (nv - 1) * table["detV"][:, :3]
        table["detV"][:, :3] *= -1
    x = torch.from_numpy(oracle.uniform(grid.shape, 0.0, 1.0, 3)).cuda()
    lines = JosephPlan(table, nu, nv, grid)
    monkeypatch.setenv("YKB_JOSEPH_BP", "gather")
    slabs = JosephPlan(table, nu, nv, grid)
    a, b = lines.forward(x), slabs.forward(x)
    assert torch.isfinite(a).all() and float(b.abs().max()) > 0
    assert K.rel_rmse(a.cpu().numpy(), b.cpu().numpy()) <= 2e-7
    twice = lines.forward(x, a.clone(), accumulate=True)
    assert K.rel_rmse(twice.cpu().numpy(), 2 * b.cpu().numpy()) <= 2e-7
    # a second volume through the same plan: nothing stays of the first
    y = torch.from_numpy(oracle.uniform(grid.shape, -1.0, 1.0, 4)).cuda()
    lines.forward(y)
    assert torch.equal(lines.forward(x), a)
    if x.numel() < 50000:
        ref = oracle.joseph_fp(table, nu, nv, K.oracle_volume(oracle, grid), x.cpu().numpy())
        assert K.rel_rmse(a.cpu().numpy(), ref) <= 1e-5
    lines.close()
    slabs.close()


@pytest.mark.parametrize("case", CASES + [(90, 50, 40, 1.7, 1.7, (34, 35, 33), (1.0, 1.0, 1.0), False)])
def test_line_backprojector_matches_gather(oracle, cuda_device, monkeypatch, case):
    # lines formed in runs (rows closer than a voxel) or by splatting, and views
    # split over CTAs for volumes of few blocks; the voxel gather applies the
    # same weights: two FP32 summation orders of at most a few hundred terms
    import torch
    from fdk_cuda_impl_b200.projectors import JosephPlan
    views, nu, nv, pu, pv, n, vox, flipped = case
    scan = CircularScan(views, views, 500.0, 1000.0, nu, nv, pu, pv, start_angle_rad=0.05)
    grid = VolumeGrid(*n, vox, (0.4, -0.7, 0.2))
    table = scan.views()
    if flipped:
        table["detS"][:, :3] += (nv - 1) * table["detV"][:, :3]
        table["detV"][:, :3] *= -1
    y = torch.from_numpy(oracle.normal((views, nv, nu), 7)).cuda()
    lines = JosephPlan(table, nu, nv, grid)
    monkeypatch.setenv("YKB_JOSEPH_BP", "gather")
    gather = JosephPlan(table, nu, nv, grid)
    a, b = lines.adjoint(y), gather.adjoint(y)
    assert torch.isfinite(a).all() and float(b.abs().max()) > 0
    assert K.rel_rmse(a.cpu().numpy(), b.cpu().numpy()) <= 1e-6
    assert torch.equal(lines.adjoint(y), a)
    both = lines.adjoint(y, b.clone(), accumulate=True)
    assert K.rel_rmse(both.cpu().numpy(), 2 * b.cpu().numpy()) <= 1e-6
    # where no ray passes both are exactly zero
    assert torch.equal(lines.adjoint(torch.zeros_like(y)), torch.zeros_like(b))
    lines.close()
    gather.close()


@pytest.mark.parametrize("runs", [True, False])
def test_infinite_rays_stay_infinite(cuda_device, runs):
    # A^T of infinite rays: infinite exactly where their weights are not zero, no
    # NaN (v - v w of an infinite v), with rows closer than a voxel (lines formed
    # in runs) and farther apart.  Rays through voxel centres have a weight of
    # zero times infinity: the offsets keep them off
    import torch
    from fdk_cuda_impl_b200.projectors import JosephPlan
    pix = 0.9 if runs else 3.1
    scan = CircularScan(8, 8, 500.0, 1000.0, 40, 36, 1.7, pix, start_angle_rad=0.05)
    grid = VolumeGrid(33, 30, 28, (1.0, 1.0, 1.0), (0.4, -0.7, 0.23))
    plan = JosephPlan(scan.views(), 40, 36, grid)
    for k in range(8):
        y = torch.zeros(plan.proj_shape, device="cuda")
        y[k, 3:33:3, 2:38:5] = 1.0
        one, inf = plan.adjoint(y), plan.adjoint(torch.where(y > 0, torch.inf, 0.0))
        assert not torch.isnan(inf).any()
        assert torch.equal(one != 0, torch.isinf(inf))
    plan.close()


@pytest.mark.parametrize("case", [CASES[i] for i in (2, 5, 6, 7)])
def test_samples_past_a_narrow_window(oracle, cuda_device, monkeypatch, case):
    # YKB_JOSEPH_FP_WINDOW=64 leaves CTAs of these cases (windows of 96 to 304)
    # one too narrow for their rays; their samples then come from the volume, the
    # same to the bit
    import torch
    from fdk_cuda_impl_b200.projectors import JosephPlan
    views, nu, nv, pu, pv, n, vox, flipped = case
    scan = CircularScan(views, views, 500.0, 1000.0, nu, nv, pu, pv, start_angle_rad=0.05)
    grid = VolumeGrid(*n, vox, (0.4, -0.7, 0.2))
    x = torch.from_numpy(oracle.uniform(grid.shape, 0.0, 1.0, 3)).cuda()
    plan = JosephPlan(scan.views(), nu, nv, grid)
    expected = plan.forward(x)
    plan.close()
    monkeypatch.setenv("YKB_JOSEPH_FP_WINDOW", "64")
    narrow = JosephPlan(scan.views(), nu, nv, grid)
    assert torch.equal(narrow.forward(x), expected)
    narrow.close()


def test_plan_without_room_for_its_table(oracle, cuda_device):
    # with the GPU's memory taken but for what the plan cannot do without, the
    # rays' heights are read from the ray records: the same results to the bit
    import torch
    from fdk_cuda_impl_b200.projectors import JosephPlan
    views, det = 80, 256
    scan = CircularScan(views, views, 500.0, 1000.0, det, det, 0.9, 0.9, start_angle_rad=0.05)
    grid = VolumeGrid(128, 128, 120, (1.0, 1.0, 1.0))
    x = torch.from_numpy(oracle.uniform(grid.shape, 0.0, 1.0, 3)).cuda()
    y = torch.from_numpy(oracle.normal((views, det, det), 7)).cuda()
    plan = JosephPlan(scan.views(), det, det, grid)
    full = plan.workspace_bytes()
    a, b = plan.forward(x), plan.adjoint(y)
    a2, b2 = torch.empty_like(a), torch.empty_like(b)
    plan.close()
    table = 8 * views * det * det
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    taken = torch.empty(free - (full - table // 2), dtype=torch.uint8, device="cuda")
    try:
        plan = JosephPlan(scan.views(), det, det, grid)
        assert plan.workspace_bytes() == full - table
        assert torch.equal(plan.forward(x, a2), a)
        assert torch.equal(plan.adjoint(y, b2), b)
        plan.close()
    finally:
        del taken
        torch.cuda.empty_cache()
