"""Measured cases: the reconstructions and projections that programs run on this package.

Every case is one call (or one short sequence of calls, where a program makes
them together) of the public torch layer on a flat-panel cone-beam scan of
source-to-isocentre 500 mm and source-to-detector 1000 mm around an object of
about 128 mm:

  kind "fdk"        one reconstruction: FdkPlan.execute, or execute_host from
                    pinned projections to a pinned volume
  kind "joseph"     one gradient step of 1/2 |A x - b|^2 through the
                    differentiable Joseph pair
  kind "operators"  FP_Siddon, BP_Siddon_RayDriven and BP_FDK_PseudoMatched of
                    one projector plan
  kind "cgls"       a CGLS reconstruction

The per-view geometry is a float32 table built here, as a program with a
calibrated scanner has one; `exact` uses the same table.
"""
import math

import numpy as np
import torch

from fdk_cuda_impl_b200.autograd import project
from fdk_cuda_impl_b200.geometry import RampFilter, VolumeGrid
from fdk_cuda_impl_b200.projectors import FdkPlan, JosephPlan
from fdk_cuda_impl_b200.recon import cgls

SID, SDD = 500.0, 1000.0
START = 0.1  # rad: no view at 45 degrees, where the main axis of a Joseph ray is a tie
VIEW = np.dtype([(f, "<f4", 4) for f in ("src", "detS", "detU", "detV", "angle")])


def _fdk(name, n, views, det, vox, pix, **options):
    case = {"name": name, "kind": "fdk", "nx": n[0], "ny": n[1], "nz": n[2], "vox": vox,
            "views": views, "nu": det[0], "nv": det[1], "pix": pix, "degrees": 360.0,
            "tilted": False, "filter": "ramlak", "cutoff": 0.5, "precision": "fp32",
            "input": "f32", "host": False, "batches": 1}
    case.update(options)
    return case


def _pair(name, kind, n, views, det, vox, pix, **options):
    case = {"name": name, "kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "vox": vox,
            "views": views, "nu": det[0], "nv": det[1], "pix": pix, "degrees": 360.0,
            "tilted": False}
    case.update(options)
    return case


def listed():
    return [
        # a preview or a region of interest: launches and too few tiles for the
        # GPU's SMs decide
        _fdk("fdk-64", (64, 64, 48), 60, (96, 64), 2.0, 3.2),
        # a quick look at half resolution
        _fdk("fdk-128", (128, 128, 128), 180, (192, 128), 1.0, 1.6),
        # a short scan of a C-arm, odd sizes throughout, arriving in three batches
        _fdk("fdk-short-ragged", (243, 251, 197), 241, (391, 333), 0.5, 0.8, degrees=215.0,
             filter="hann", cutoff=0.45, batches=3),
        # a calibrated scanner: the detector is tilted by a fraction of a degree
        _fdk("fdk-tilted", (256, 256, 256), 180, (384, 384), 0.5, 0.8, tilted=True),
        # the ordinary full reconstruction, projections on the GPU
        _fdk("fdk-512", (512, 512, 512), 720, (768, 768), 0.25, 0.4),
        # the same from host memory to host memory, as a scanner's console runs it
        _fdk("fdk-512-host", (512, 512, 512), 720, (768, 768), 0.25, 0.4, host=True),
        # the largest: high resolution from projections stored in BF16
        _fdk("fdk-1024-bf16", (1024, 1024, 1024), 1440, (1536, 1536), 0.125, 0.2,
             filter="shepplogan", precision="bf16", input="bf16"),
        # one step of a learned or iterative reconstruction: small (a training
        # patch), full size, and on a calibrated scanner with odd sizes
        _pair("joseph-64", "joseph", (64, 64, 48), 60, (96, 64), 2.0, 3.2),
        _pair("joseph-256", "joseph", (256, 256, 256), 360, (384, 384), 0.5, 0.8),
        _pair("joseph-tilted", "joseph", (181, 167, 149), 120, (279, 245), 0.7, 1.1, tilted=True),
        # the projectors of simulations and of solvers with an unmatched backprojector
        _pair("operators-256", "operators", (256, 256, 256), 120, (384, 384), 0.5, 0.8),
        # a sparse-view iterative reconstruction, whole
        _pair("cgls-256", "cgls", (256, 256, 256), 90, (384, 384), 0.5, 0.8, iterations=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fdk", "fdk", "fdk", "joseph", "joseph", "operators", "cgls"])
    n = _log_int(rng, 48, 512 if kind == "fdk" else 256)
    shape = (max(40, int(n * rng.uniform(0.85, 1.15))), n, max(24, int(n * rng.uniform(0.4, 1.0))))
    vox = round(128.0 / n * rng.uniform(0.9, 1.1), 4)
    views = _log_int(rng, 48, 720 if kind == "fdk" else 240)
    nu = int(n * rng.uniform(1.2, 1.8)) + rng.randrange(2)
    nv = max(16, int(shape[2] * rng.uniform(1.1, 1.7)))
    # pixels that see the whole object in the fan
    pix = round(2.35 * 1.15 * n * vox / nu * rng.uniform(0.95, 1.1), 4)
    options = {"tilted": rng.random() < 0.25}
    if kind == "fdk":
        options.update(filter=rng.choice(["ramlak", "shepplogan", "hann", "cosine", "hamming"]),
                       cutoff=round(rng.uniform(0.35, 0.5), 3), batches=rng.choice([1, 1, 1, 2, 4]))
        options["precision"] = rng.choice(["fp32", "fp32", "bf16"])
        options["input"] = "bf16" if options["precision"] == "bf16" else "f32"
        if rng.random() < 0.25:
            options["degrees"] = round(rng.uniform(232.0, 250.0), 1)
        elif rng.random() < 0.25:
            options.update(host=True, batches=1)
        case = _fdk("", shape, views, (nu, nv), vox, pix, **options)
    else:
        if kind == "cgls":
            options["iterations"] = rng.randint(2, 8)
        case = _pair("", kind, shape, views, (nu, nv), vox, pix, **options)
    del case["name"]
    return case


# ------------------------------------------------------------------- inputs ---
def _orbit(case):
    """The scan's float32 view table (the detector's v axis along z unless
    tilted; then rotated by a fraction of a degree about each of its axes)."""
    n, nu, nv = case["views"], case["nu"], case["nv"]
    step = math.radians(case["degrees"]) / n
    table = np.zeros(n, dtype=VIEW)
    for i in range(n):
        a = START + i * step
        c, s = math.cos(a), math.sin(a)
        rotation = np.array([[c, -s, 0.0], [s, c, 0.0], [0.0, 0.0, 1.0]])
        u, v, centre = np.array([1.0, 0, 0]), np.array([0, 0, 1.0]), np.array([0, SDD - SID, 0.0])
        if case["tilted"]:
            for x, y, angle in ((1, 2, 0.006), (0, 1, -0.004), (0, 2, 0.008)):
                r = np.eye(3)
                r[x, x] = r[y, y] = math.cos(angle)
                r[x, y], r[y, x] = -math.sin(angle), math.sin(angle)
                u, v = r @ u, r @ v
            centre = centre + 1.3 * u - 0.8 * v
        u, v = case["pix"] * u, case["pix"] * v
        corner = centre - 0.5 * (nu - 1) * u - 0.5 * (nv - 1) * v
        table["src"][i, :3] = rotation @ np.array([0.0, -SID, 0.0])
        table["detS"][i, :3] = rotation @ corner
        table["detU"][i, :3] = rotation @ u
        table["detV"][i, :3] = rotation @ v
        table["angle"][i, 0] = a
    return table


def _voxel(case):
    return float(np.float32(case["vox"]))  # as the grid holds it


def _grid(case):
    return VolumeGrid(case["nx"], case["ny"], case["nz"], (_voxel(case),) * 3)


def _spheres(case, generator, count=6):
    """Centres, radii (mm) and attenuations (1/mm) of an object inside the volume."""
    r = torch.rand((count, 5), generator=generator, dtype=torch.float64)
    size = torch.tensor([case["nx"], case["ny"], case["nz"]], dtype=torch.float64) * case["vox"]
    return (r[:, :3] - 0.5) * 0.6 * size, (0.06 + 0.24 * r[:, 3]) * size.min(), 0.005 + 0.02 * r[:, 4]


def _projections(case, table, seed, dtype):
    """Line integrals of the object's spheres plus detector noise, [views][nv][nu]."""
    generator = torch.Generator().manual_seed(seed)
    spheres = list(zip(*(t.tolist() for t in _spheres(case, generator))))
    device_generator = torch.Generator(device="cuda").manual_seed(seed)
    n, nv, nu = case["views"], case["nv"], case["nu"]
    out = torch.empty((n, nv, nu), dtype=dtype, device="cuda")
    f = {k: torch.from_numpy(table[k][:, :3].astype(np.float64)).cuda() for k in VIEW.names[:4]}
    iu = torch.arange(nu, device="cuda", dtype=torch.float32)[None, None, :]
    iv = torch.arange(nv, device="cuda", dtype=torch.float32)[None, :, None]
    step = max(1, (1 << 26) // (nv * nu))
    for k in range(0, n, step):
        src, d0 = f["src"][k:k + step], (f["detS"] - f["src"])[k:k + step]
        du, dv = f["detU"][k:k + step], f["detV"][k:k + step]

        def dot(a, b):
            return (a * b).sum(1).float()[:, None, None]
        dd = (dot(d0, d0) + iu * (2 * dot(d0, du) + iu * dot(du, du)) +
              iv * (2 * dot(d0, dv) + iv * dot(dv, dv)) + (2 * dot(du, dv)) * iu * iv)
        p = torch.randn((len(src), nv, nu), generator=device_generator, device="cuda").mul_(0.003)
        for centre, radius, value in spheres:
            e = torch.tensor(centre, dtype=torch.float64, device="cuda") - src
            along = dot(e, d0) + iu * dot(e, du) + iv * dot(e, dv)
            half = along.square_().div_(dd).add_(radius ** 2 - dot(e, e)).clamp_min_(0).sqrt_()
            p.add_(half, alpha=2 * value)
        out[k:k + step] = p
    return out


def _volume(case, seed):
    """The object's attenuation on the grid with some texture, [nz][ny][nx]."""
    generator = torch.Generator().manual_seed(seed)
    spheres = zip(*(t.tolist() for t in _spheres(case, generator)))
    device_generator = torch.Generator(device="cuda").manual_seed(seed)
    shape = (case["nz"], case["ny"], case["nx"])
    z, y, x = (((torch.arange(n, device="cuda") - 0.5 * (n - 1)) * case["vox"]) for n in shape)
    out = torch.randn(shape, generator=device_generator, device="cuda").mul_(5e-4)
    for (cx, cy, cz), radius, value in spheres:
        d = (z - cz).square()[:, None, None] + (y - cy).square()[:, None] + (x - cx).square()
        out.add_(d <= radius ** 2, alpha=value)
    return out


def prepare(case, seed):
    table, grid = _orbit(case), _grid(case)
    nu, nv = case["nu"], case["nv"]
    state = {"case": case}
    if case["kind"] == "fdk":
        dtype = torch.bfloat16 if case["input"] == "bf16" else torch.float32
        projections = _projections(case, table, seed, dtype)
        short = case["degrees"] < 360.0
        state["plan"] = FdkPlan(table, nu, nv, math.radians(case["degrees"]), grid,
                                RampFilter.named(case["filter"], cutoff=case["cutoff"]),
                                case["precision"], parker="auto" if short else None,
                                start_angle_rad=float(table["angle"][0, 0]))
        state["volume"] = torch.empty(grid.shape, device="cuda")
        if case["host"]:
            state["projections"] = torch.empty(projections.shape, dtype=dtype, pin_memory=True)
            state["projections"].copy_(projections)
            state["host_volume"] = torch.empty(grid.shape, pin_memory=True)
        else:
            state["projections"] = projections
        return state
    state["plan"] = JosephPlan(table, nu, nv, grid)
    state["projections"] = _projections(case, table, seed, torch.float32)
    if case["kind"] != "cgls":
        state["x"] = _volume(case, seed + 1)
    return state


def run(state):
    case, plan = state["case"], state["plan"]
    if case["kind"] == "fdk":
        projections, volume = state["projections"], state["volume"]
        if case["host"]:
            plan.execute_host(projections, volume, host_out=state["host_volume"])
            # the console's next step reads the host volume
            torch.cuda.current_stream().synchronize()
            return state["host_volume"]
        n, batches = case["views"], case["batches"]
        for b in range(batches):
            lo, hi = n * b // batches, n * (b + 1) // batches
            plan.execute(projections[lo:hi], volume, view_offset=lo, clear=b == 0)
        return volume
    if case["kind"] == "joseph":
        x = state["x"].detach().requires_grad_(True)
        y = project(x, plan)
        loss = 0.5 * (y - state["projections"]).square().sum()
        loss.backward()
        return {"projections": y.detach(), "gradient": x.grad}
    if case["kind"] == "operators":
        return {"siddon_fp": plan.forward_siddon(state["x"]),
                "siddon_bp": plan.backproject_siddon(state["projections"]),
                "pseudo_bp": plan.backproject_pseudo(state["projections"])}
    x, norms = cgls(plan, state["projections"], case["iterations"])
    return {"x": x, "norms": norms}


def work(case):
    voxels = case["nx"] * case["ny"] * case["nz"]
    rays = case["views"] * case["nu"] * case["nv"]
    updates = voxels * case["views"]
    # a ray's samples, one a slice of its main axis, over the object's extent
    samples = rays * 0.5 * (case["nx"] + case["ny"])
    if case["kind"] == "fdk":
        # per update two coordinates, a bilinear sample, a weighted sum; per
        # row a forward and a backward FFT of twice its length
        length = 2.0 * case["nu"]
        flops = 10.0 * updates + rays / case["nu"] * 10.0 * length * math.log2(length)
        return {"bytes": rays * (2 if case["input"] == "bf16" else 4) + 4 * voxels, "flops": flops}
    if case["kind"] == "joseph":
        # reads x and b, writes A x and the gradient
        return {"bytes": 8 * voxels + 8 * rays, "flops": 2 * 12.0 * samples}
    if case["kind"] == "operators":
        return {"bytes": 12 * voxels + 12 * rays, "flops": 2 * 8.0 * samples + 14.0 * updates}
    # CGLS: two more operators start it; every iteration applies the pair
    pairs = case["iterations"] + 1
    return {"bytes": 4 * (2 * voxels + rays), "flops": pairs * 2 * 12.0 * samples}


def tolerance(case):
    if case["kind"] == "fdk":
        if case["precision"] == "bf16":
            # two BF16 parts an operand in the ramp filter
            return {"rel": 1e-3, "max": 2e-2}
        return {"rel": 2e-5, "max": 1e-3}
    if case["kind"] == "cgls":
        return {"rel": 2e-5, "max": 1e-3}
    return {"rel": 5e-6, "max": 5e-4}


# -------------------------------------------------------------------- exact ---
_F8 = {"dtype": torch.float64, "device": "cuda"}


def _vectors(table):
    return [torch.from_numpy(table[f][:, :3].astype(np.float64)) for f in ("src", "detS", "detU", "detV")]


def _sample(image, x, y):
    """Bilinear samples of image [b][rows][columns] at pixel coordinates x, y [b][...]; zero outside."""
    rows, columns = image.shape[-2:]
    at = torch.stack((x * (2.0 / (columns - 1)) - 1.0, y * (2.0 / (rows - 1)) - 1.0), -1)
    b = image.shape[0]
    return torch.nn.functional.grid_sample(image[:, None], at.reshape(b, 1, -1, 2), "bilinear", "zeros",
                                           True).reshape(x.shape)


def _axes(case):
    return [((torch.arange(n, **_F8) - 0.5 * (n - 1)) * _voxel(case)) for n in (case["nx"], case["ny"], case["nz"])]


def _backproject_exact(case, table, images, weight):
    """Sum over the views of weight(view, u, v, P - source) x the bilinear sample of its image."""
    src, s, u, v = _vectors(table)
    x, y, z = _axes(case)
    out = torch.zeros((case["nz"], case["ny"], case["nx"]), **_F8)
    for k in range(case["views"]):
        # P - source = (1/t) (S + u U + v V - source): the pixel's homogeneous coordinates
        m = torch.linalg.inv(torch.stack((u[k], v[k], s[k] - src[k]), 1)).tolist()
        c = src[k].tolist()

        def affine(r):
            return (r[2] * (z - c[2]))[:, None, None] + ((r[1] * (y - c[1]))[:, None] + r[0] * (x - c[0]))
        h = affine(m[2])
        pu, pv = affine(m[0]).div_(h), affine(m[1]).div_(h)
        value = _sample(images[k].double()[None], pu[None], pv[None])[0]
        out += weight(k, pu, pv, h, affine) * value
    return out


def _window(x, kind):
    return {"ramlak": lambda: torch.ones_like(x), "shepplogan": lambda: torch.sinc(0.5 * x),
            "cosine": lambda: torch.cos(0.5 * math.pi * x), "hann": lambda: 0.5 + 0.5 * torch.cos(math.pi * x),
            "hamming": lambda: 0.54 + 0.46 * torch.cos(math.pi * x)}[kind]()


def _fdk_exact(case, table, projections):
    n, nu, nv = case["views"], case["nu"], case["nv"]
    src, s, u, v = _vectors(table)
    angle = table["angle"][:, 0].astype(np.float64)
    scan = float(np.float32(math.radians(case["degrees"])))
    length = 1
    while length < 2 * nu:
        length *= 2
    f = torch.arange(length // 2 + 1, **_F8) / length
    cut = float(np.float32(case["cutoff"]))
    pixel = float(u[0].norm())
    ramp = torch.where(f <= cut, f * _window((f / cut).clamp(max=1.0), case["filter"]) / pixel, torch.zeros_like(f))
    iu, iv = torch.arange(nu, **_F8), torch.arange(nv, **_F8)
    images, base, radial = [], [], []
    for k in range(n):
        normal = torch.linalg.cross(v[k], u[k])
        normal = normal / normal.norm()
        centre = s[k] + 0.5 * (nu - 1) * u[k] + 0.5 * (nv - 1) * v[k] - src[k]
        normal = normal if normal @ centre > 0 else -normal
        sid = float(src[k][:2].norm())
        r = torch.tensor([-src[k][0] / sid, -src[k][1] / sid, 0.0], dtype=torch.float64)
        dsd = float((s[k] - src[k]) @ normal / (r @ normal))
        q = [s[k][c] - src[k][c] + iu[None, :] * u[k][c] + iv[:, None] * v[k][c] for c in range(3)]
        w = dsd / torch.sqrt(q[0] ** 2 + q[1] ** 2 + q[2] ** 2) * (dsd / sid / 2.0)
        if case["degrees"] < 360.0:
            w = w * _parker(case, r, src[k], s[k], u[k], v[k], float(angle[k] - angle[0]), scan)
        rows = torch.fft.rfft(projections[k].double().cuda() * w, n=length) * ramp
        images.append(torch.fft.irfft(rows, n=length)[:, :nu].float() if n * nu * nv > 4e8
                      else torch.fft.irfft(rows, n=length)[:, :nu])
        lo, hi = max(k - 1, 0), min(k + 1, n - 1)
        base.append(sid * sid * (angle[hi] - angle[lo]) / (hi - lo) * 2.0 * math.pi / scan)
        radial.append(r.tolist())
    return _backproject_exact(case, table, images,
                              lambda k, pu, pv, h, affine: base[k] / affine(radial[k]).square_())


def _parker(case, r, src, s, u, v, beta, scan):
    """The short scan's weight of every column (sin^2 ramps), with the range/pi scale."""
    def fan(column):
        d = s + column * u + 0.5 * (case["nv"] - 1) * v - src
        return math.atan2(float(d[0] * r[1] - d[1] * r[0]), float(d[0] * r[0] + d[1] * r[1]))
    edge = max(abs(fan(0.0)), abs(fan(case["nu"] - 1.0)))
    beta %= 2 * math.pi
    out = []
    for column in range(case["nu"]):
        g = fan(float(column))
        value = 0.0
        if 0.0 < beta < 2 * (edge + g):
            value = math.sin(0.25 * math.pi * beta / max(edge + g, 1e-6)) ** 2
        elif 0.0 < beta <= math.pi + 2 * g:
            value = 1.0
        elif 0.0 < beta < math.pi + 2 * edge:
            value = math.sin(0.25 * math.pi * (math.pi + 2 * edge - beta) / max(edge - g, 1e-6)) ** 2
        out.append(value * scan / math.pi)
    return torch.tensor(out, **_F8)


def _joseph_views(case, table):
    """Per view: the main axis and the source and pixel vectors in voxel units."""
    src, s, u, v = _vectors(table)
    for k in range(case["views"]):
        d = s[k] + 0.5 * (case["nu"] - 1) * u[k] + 0.5 * (case["nv"] - 1) * v[k] - src[k]
        axis = int(torch.argmax(d.abs()))
        order = [axis] + [a for a in range(3) if a != axis]
        yield k, order, [(t / _voxel(case))[order].tolist() for t in (src[k], s[k], u[k], v[k])]


def _joseph_rays(case, order, geometry):
    """Sample positions on both minor axes [slices][nv][nu] and the chord of a step [nv][nu]."""
    src, s, u, v = geometry
    n = [(case["nx"], case["ny"], case["nz"])[a] for a in order]
    iu, iv = torch.arange(case["nu"], **_F8)[None, :], torch.arange(case["nv"], **_F8)[:, None]
    d = [s[c] + iu * u[c] + iv * v[c] - src[c] for c in range(3)]
    a1, a2 = d[1] / d[0], d[2] / d[0]
    along = (torch.arange(n[0], **_F8) - 0.5 * (n[0] - 1) - src[0])[:, None, None]
    f1 = along * a1 + (src[1] + 0.5 * (n[1] - 1))
    f2 = along * a2 + (src[2] + 0.5 * (n[2] - 1))
    return f1, f2, _voxel(case) * torch.sqrt(1.0 + a1 * a1 + a2 * a2)


def _joseph_fp_exact(case, table, x):
    out = torch.empty((case["views"], case["nv"], case["nu"]), **_F8)
    volume = x.double().permute(2, 1, 0)  # [x][y][z]
    for k, order, geometry in _joseph_views(case, table):
        f1, f2, chord = _joseph_rays(case, order, geometry)
        slab = volume.permute(order[0], order[2], order[1]).contiguous()  # [main][minor 2][minor 1]
        out[k] = _sample(slab, f1, f2).sum(0) * chord
    return out


def _joseph_bp_exact(case, table, y):
    out = torch.zeros((case["nx"], case["ny"], case["nz"]), **_F8)
    for k, order, geometry in _joseph_views(case, table):
        f1, f2, chord = _joseph_rays(case, order, geometry)
        slices, rows, columns = (out.shape[a] for a in (order[0], order[2], order[1]))
        at = torch.stack((f1 * (2.0 / (columns - 1)) - 1.0, f2 * (2.0 / (rows - 1)) - 1.0), -1)
        value = (y[k].double() * chord).reshape(1, 1, 1, -1).expand(slices, 1, 1, -1).contiguous()
        slab, _ = torch.ops.aten.grid_sampler_2d_backward(
            value, torch.zeros((slices, 1, rows, columns), **_F8), at.reshape(slices, 1, -1, 2), 0, 0, True,
            [True, False])
        back = [0, 0, 0]
        for place, a in enumerate((order[0], order[2], order[1])):
            back[a] = place
        out += slab[:, 0].permute(*back)
    return out.permute(2, 1, 0).contiguous()


def _siddon_segments(case, table, k):
    """Segment lengths [rays][segments] and voxel indices (0 where the length is 0) of one view."""
    src, s, u, v = (t[k].cuda() for t in _vectors(table))
    iu, iv = torch.arange(case["nu"], **_F8)[None, :], torch.arange(case["nv"], **_F8)[:, None]
    lo, hi, cuts, n = 0.0, 1.0, [], (case["nx"], case["ny"], case["nz"])
    d = [(s[c] - src[c] + iu * u[c] + iv * v[c]).reshape(-1, 1) for c in range(3)]
    for c in range(3):
        planes = (torch.arange(n[c] + 1, **_F8) - 0.5 * n[c]) * _voxel(case)
        step = torch.where(d[c].abs() > 1e-8, d[c], torch.full_like(d[c], 1e-8))
        t = (planes - src[c]) / step
        lo = torch.clamp(torch.minimum(t[:, :1], t[:, -1:]), min=lo) if isinstance(lo, float) else torch.maximum(
            lo, torch.minimum(t[:, :1], t[:, -1:]))
        hi = torch.clamp(torch.maximum(t[:, :1], t[:, -1:]), max=hi) if isinstance(hi, float) else torch.minimum(
            hi, torch.maximum(t[:, :1], t[:, -1:]))
        cuts.append(t)
    hi = torch.maximum(hi, lo)
    t = torch.sort(torch.minimum(torch.maximum(torch.cat(cuts, 1), lo), hi), 1).values
    length = t.diff(dim=1)
    middle = t[:, :-1] + 0.5 * length
    index = torch.zeros_like(length, dtype=torch.int64)
    for c in (2, 1, 0):
        i = torch.floor((src[c] + middle * d[c]) / _voxel(case) + 0.5 * n[c]).long().clamp_(0, n[c] - 1)
        index = index * n[c] + i
    scale = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
    return length * scale, index


def _operators_exact(case, table, x, y):
    volume = x.double().reshape(-1)
    fp = torch.empty((case["views"], case["nv"], case["nu"]), **_F8)
    bp = torch.zeros(case["nx"] * case["ny"] * case["nz"], **_F8)
    src, s, u, v = _vectors(table)
    cell = _voxel(case) ** 3 / float(u[0].norm() * v[0].norm())
    scale = []
    for k in range(case["views"]):
        length, index = _siddon_segments(case, table, k)
        fp[k] = (length * volume[index]).sum(1).reshape(case["nv"], case["nu"])
        bp.index_add_(0, index.reshape(-1), (length * y[k].double().reshape(-1, 1)).reshape(-1))
        normal = torch.linalg.cross(v[k], u[k])
        scale.append(cell * float(((s[k] - src[k]) @ normal / normal.norm()).abs()))

    def weight(k, pu, pv, h, affine):
        # |P - source| = L h: the weight voxel x L^3 / (|P - source|^2 plane) / pixel area
        plane = scale[k] / cell
        d = [float(s[k][c] - src[k][c]) + pu * float(u[k][c]) + pv * float(v[k][c]) for c in range(3)]
        return torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2).div_(h.square()).mul_(cell / plane)
    return {"siddon_fp": fp, "siddon_bp": bp.reshape(x.shape),
            "pseudo_bp": _backproject_exact(case, table, y, weight)}


def _cgls_exact(case, table, b):
    b = b.double()
    x, r = torch.zeros((case["nz"], case["ny"], case["nx"]), **_F8), b.clone()
    p = _joseph_bp_exact(case, table, r)
    gamma, norms = float(p.square().sum()), [float(r.norm())]
    for _ in range(case["iterations"]):
        w = _joseph_fp_exact(case, table, p)
        alpha = gamma / float(w.square().sum())
        x += alpha * p
        r -= alpha * w
        z = _joseph_bp_exact(case, table, r)
        new = float(z.square().sum())
        p = z + new / gamma * p
        gamma = new
        norms.append(float(r.norm()))
    return {"x": x, "norms": norms}


def exact(case, seed):
    voxels = case["nx"] * case["ny"] * case["nz"]
    if voxels * case["views"] > (1.2e11 if case["kind"] == "fdk" else 7e9):
        return None  # over about 20 seconds
    table = _orbit(case)
    if case["kind"] == "fdk":
        dtype = torch.bfloat16 if case["input"] == "bf16" else torch.float32
        return _fdk_exact(case, table, _projections(case, table, seed, dtype))
    y = _projections(case, table, seed, torch.float32)
    if case["kind"] == "cgls":
        return _cgls_exact(case, table, y)
    x = _volume(case, seed + 1)
    if case["kind"] == "operators":
        return _operators_exact(case, table, x, y)
    fp = _joseph_fp_exact(case, table, x)
    return {"projections": fp, "gradient": _joseph_bp_exact(case, table, fp - y.double())}
