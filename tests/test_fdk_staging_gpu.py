"""The staged backprojection's edges against the FP64 oracle: the row pairs of
the filter epilogue across its 127-row tiles and views, and columns of tilted
and untilted detectors over full, short and single z tiles.  Bound: the FP32
form's 1e-5 (interpolation weights in FP32, sums of at most 48 views)."""
import numpy as np
import pytest

from fdk_cuda_impl_b200.geometry import CircularScan, RampFilter, VolumeGrid
from tests import cases as K

pytestmark = pytest.mark.gpu
FP32_TOL = 1e-5


def _run(oracle, scan, grid, monkeypatch, **options):
    import torch
    from fdk_cuda_impl_b200.projectors import FdkPlan, JosephPlan
    views, nu, nv = scan.views(), scan.channels, scan.rows
    p = oracle.uniform((len(views), nv, nu), 0.5, 1.5, 4)
    plan = FdkPlan(views, nu, nv, scan.scan_range, grid, RampFilter(), **options)
    got = plan.execute(torch.from_numpy(p).cuda()).cpu().numpy()
    plan.check()
    plan.close()
    vol = K.oracle_volume(oracle, grid)
    ref = oracle.fdk(views, nu, nv, scan.scan_range, vol, oracle.filter_struct(1), p)
    assert K.rel_rmse(got, ref) <= FP32_TOL
    jp = JosephPlan(views, nu, nv, grid)
    pseudo = jp.backproject_pseudo(torch.from_numpy(p).cuda()).cpu().numpy()
    jp.check()
    jp.close()
    assert K.rel_rmse(pseudo, oracle.pseudo_bp(views, nu, nv, vol, p)) <= FP32_TOL


@pytest.mark.parametrize("nu,nv", [(17, 1), (33, 2), (48, 126), (49, 127), (64, 128), (80, 129)])
def test_row_pairs_across_filter_tiles(oracle, cuda_device, monkeypatch, nu, nv):
    scan = CircularScan(7, 7, 500.0, 1000.0, nu, nv, 1.6, 1.6)
    _run(oracle, scan, VolumeGrid(24, 20, 18, (1.0, 1.0, 1.0)), monkeypatch)


@pytest.mark.parametrize("tilt", [(0.0, 0.0, 0.0), (0.006, -0.004, 0.008), (0.06, 0.05, -0.07)])
@pytest.mark.parametrize("nz", [1, 33, 64, 69])
def test_columns_over_z_tiles(oracle, cuda_device, monkeypatch, tilt, nz):
    scan = CircularScan(20, 20, 400.0, 800.0, 64, 90, 1.7, 1.9, tilt_rad=tilt,
                        offset_unv_mm=(0.8, 0.0, -1.1))
    _run(oracle, scan, VolumeGrid(35, 33, nz, (1.1, 0.9, 1.2), (1.0, -0.5, 0.6)), monkeypatch)


@pytest.mark.parametrize("tilt", [(0.0, 0.0, 0.0), (0.006, -0.004, 0.008)])
@pytest.mark.parametrize("n,nz,views", [(16, 1, 3), (31, 21, 48), (64, 33, 90), (96, 130, 24)])
def test_split_views_match_one_job_a_tile(oracle, cuda_device, monkeypatch, n, nz, views, tilt):
    # volumes of few tiles split their views into jobs whose sums are added
    # afterwards; the bounds-checked kernel (YKB_FDK_BP_PATH=global) sums every
    # view in one thread from detector coordinates that it rounds to FP32: up
    # to 7.6e-6 px (below 128 px) on white-noise rows, 1e-5 of their size.
    # Also adding to a volume 4 bytes off a 16-byte boundary
    import torch
    from fdk_cuda_impl_b200.projectors import FdkPlan
    scan = CircularScan(views, views, 400.0, 800.0, 70, 90, 3.0 * n / 64, 3.0 * n / 64, tilt_rad=tilt)
    grid = VolumeGrid(n, n + 1, nz, (1.0, 1.0, 1.0))
    p = torch.from_numpy(oracle.uniform((views, 90, 70), 0.5, 1.5, 5)).cuda()
    split = FdkPlan(scan.views(), 70, 90, scan.scan_range, grid, RampFilter())
    monkeypatch.setenv("YKB_FDK_BP_PATH", "global")
    one = FdkPlan(scan.views(), 70, 90, scan.scan_range, grid, RampFilter())
    a, b = split.execute(p), one.execute(p)
    assert K.rel_rmse(a.cpu().numpy(), b.cpu().numpy()) <= 2e-5
    assert torch.equal(a, split.execute(p))
    flat = torch.full((a.numel() + 1,), 2.0, device="cuda")
    shifted = flat[1:].view(a.shape)
    shifted.copy_(b)
    split.execute(p[:views // 2], shifted, clear=False)
    split.execute(p[views // 2:], shifted, view_offset=views // 2, clear=False)
    split.check()
    assert flat[0].item() == 2.0
    assert K.rel_rmse(shifted.cpu().numpy(), 2.0 * b.cpu().numpy()) <= 2e-5
    split.close()
    one.close()


@pytest.mark.parametrize("views,nu,nv,n,nz", [(8, 64, 48, 40, 32), (16, 96, 64, 64, 48)])
def test_column_terms_round_once(oracle, cuda_device, monkeypatch, views, nu, nv, n, nz):
    # plain rows and the pseudo-matched weight: u and v of a column are rounded to
    # FP32 once, below 64 px (rms 2^-18 / sqrt(12) = 1.1e-6 px each).  Uniform rows
    # in 0.5 .. 1.5 differ by 0.41 rms from pixel to pixel: 1.1e-6 x 0.41 x sqrt(2)
    # of a view's value, averaged over the views, beside the FP32 sum's
    # 2^-24 sqrt(views) / 3.  Several roundings a coordinate exceed it
    import torch
    from fdk_cuda_impl_b200.projectors import FdkPlan, JosephPlan
    bound = ((1.1e-6 * 0.41 * 2 ** 0.5) ** 2 / views + (2.0 ** -24 / 3) ** 2 * views) ** 0.5
    scan = CircularScan(views, views, 500.0, 1000.0, nu, nv, 300.0 / nu, 300.0 / nu,
                        start_angle_rad=0.1, offset_unv_mm=(0.8, 0.0, -1.1))
    grid = VolumeGrid(n, n + 3, nz, (128.0 / n,) * 3, (0.3, -0.2, 0.1))
    table, vol = scan.views(), K.oracle_volume(oracle, grid)
    p = oracle.uniform((views, nv, nu), 0.5, 1.5, 4)
    pd = torch.from_numpy(p).cuda()
    jp = JosephPlan(table, nu, nv, grid)
    pseudo = jp.backproject_pseudo(pd).cpu().numpy()
    jp.check()
    jp.close()
    assert K.rel_rmse(pseudo, oracle.pseudo_bp(table, nu, nv, vol, p)) <= bound
    monkeypatch.setenv("YKB_FDK_BP_PATH", "rows")
    plan = FdkPlan(table, nu, nv, scan.scan_range, grid, RampFilter())
    rows = plan.backproject(pd).cpu().numpy()
    plan.check()
    plan.close()
    assert K.rel_rmse(rows, oracle.fdk_backproject(table, nu, nv, scan.scan_range, vol, p)) <= bound


@pytest.mark.parametrize("nu,nv,views", [(300, 64, 60), (391, 64, 120), (200, 128, 60)])
def test_filtered_rows_do_not_depend_on_the_batches(oracle, cuda_device, nu, nv, views):
    # one tile width a plan: a view's rows come out the same to the bit alone, in
    # batches and with all the others
    import torch
    from fdk_cuda_impl_b200.projectors import FdkPlan
    scan = CircularScan(views, views, 500.0, 1000.0, nu, nv, 0.8, 0.8)
    plan = FdkPlan(scan.views(), nu, nv, scan.scan_range, VolumeGrid.cube(16, 1.0), RampFilter())
    p = torch.from_numpy(oracle.uniform((views, nv, nu), 0.5, 1.5, 4)).cuda()
    whole = plan.filter(p)
    for n in (1, 7):
        parts = [plan.filter(p[k:k + n].contiguous(), view_offset=k) for k in range(0, views, n)]
        assert torch.equal(torch.cat(parts), whole)
    plan.check()
    plan.close()
