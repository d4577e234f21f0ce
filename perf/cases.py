"""The calls whose time and results are measured, as a user's program makes them.

Each case is a dict of plain values: which call it is (``kind``), the grid,
the polarizations, the CF supports and oversampling, the number of
visibilities, the arithmetic form and where the records lie.  Inputs are
synthetic: separable CFs (Gaussian times a w-dependent quadratic phase, times
a factor per Mueller element), visibilities with N(0, 1) values, u and v in a
disk of 0.45 grid extents, uniform over its area ("disk") or denser towards
the centre as an array's short baselines are ("core"), CF groups drawn by
|w|.  They are made on the GPU with torch from the seed alone.

The mixed arithmetic form carries FP32 accuracy, so a program that asks for
it keeps its grid as complex64; the FP64 form's grid is taken as it is.
"""
import math

import numpy as np
import torch

import hpg_b200
from hpg_b200 import abi, autograd

C_LIGHT = 299792458.0
GRID_SCALE = 0.0476591
FREQ = 1.4e9

# the full-polarization benchmark's w-plane groups
FULL_POL = "8,12,16,20,24,28,32,32"


def _case(name, kind, **kw):
    c = {"kind": kind, "npol": 1, "nx": 512, "ny": 512, "supports": "7",
         "os": 20, "nvis": 1000, "form": "fp64", "dense": False,
         "screen": False, "uv": "disk", "host": False}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: one short integration's model visibilities,
        # where launches and latency are what it costs
        _case("predict_1pol_1k", "predict"),
        # a dirty image: reset, grid one batch, normalise + FFT + shift
        # (the single-polarization benchmark configuration)
        _case("image_1pol_100k", "image", nvis=100_000),
        # A-projection gridding of a modest batch: phase gradients, narrow
        # odd supports, odd grid sides, short baselines dominating
        _case("grid_2pol_20k_screen", "grid", npol=2, nx=1125, ny=1031,
              supports="5,7,11,15", os=33, nvis=19_999, screen=True,
              uv="core"),
        # residuals of a batch in host memory, as a program that reads a
        # measurement set piece by piece calls it
        _case("residual_4pol_50k_host", "residual", npol=4, nx=2048, ny=2048,
              supports=FULL_POL, os=32, nvis=50_000, form="mixed", dense=True,
              host=True),
        # the major cycle's degrid + grid at the full-polarization benchmark's
        # own size, in its headline form
        _case("cycle_4pol_10M_mixed", "cycle", npol=4, nx=2048, ny=2048,
              supports=FULL_POL, os=128, nvis=10_000_000, form="mixed",
              dense=True),
        # the same step at a tenth of the batch in the reference's arithmetic
        _case("cycle_4pol_1M_fp64", "cycle", npol=4, nx=2048, ny=2048,
              supports=FULL_POL, os=64, nvis=1_000_000, dense=True),
        # and with the compensated FP32 tiles, a batch that leaves tiles thin
        _case("cycle_4pol_400k_comp", "cycle", npol=4, nx=2048, ny=2048,
              supports=FULL_POL, os=64, nvis=400_000, form="comp", dense=True),
        # model visibilities for wide w-projection kernels, two polarizations
        _case("predict_2pol_wide_300k", "predict", npol=2, nx=4096, ny=4096,
              supports="16,24,32,40,48,56,64", os=32, nvis=300_000,
              form="mixed", uv="core"),
        # full-polarization A-projection at the widest support
        _case("cycle_4pol_wide_20k", "cycle", npol=4, nx=2048, ny=2048,
              supports="48,64", os=16, nvis=20_000, dense=True, screen=True),
        # one gradient step of differentiable imaging: D, a loss, D^H
        _case("gradient_2pol_1M", "gradient", npol=2, nx=4096, ny=4096,
              supports="8,16,24,32,40,48,56,64", os=64, nvis=1_000_000),
        # many uneven gridding jobs in one call (side:visibilities)
        _case("batch_2pol_8jobs", "batch", npol=2,
              jobs="256:10000,300:25000,456:60000,640:12000,800:150000,"
                   "1024:400000,1536:90000,2048:700000",
              supports="8,16,32", os=32, nvis=1_447_000, form="mixed"),
        # a new CF set (values on the device) and the batch that uses it
        _case("cf_swap_4pol", "cf_swap", npol=4, nx=1024, ny=1024,
              supports="8,16,24,32", os=48, nvis=10_000, dense=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["predict", "predict", "grid", "grid", "residual",
                       "cycle", "cycle", "cycle", "image", "gradient", "batch",
                       "cf_swap"])
    npol = rng.choice([1, 2, 4])
    dense = npol == 4 and rng.random() < 0.7
    form = rng.choice(["fp64", "mixed", "mixed", "comp"])
    if kind in ("image", "gradient", "cf_swap"):
        form = "fp64"
    if kind in ("predict",) and form == "comp":
        form = "mixed"
    nx, ny = _log_int(rng, 256, 4096), _log_int(rng, 256, 4096)
    if rng.random() < 0.6:
        nx, ny = nx & ~1, ny & ~1
    if npol == 4:
        nx, ny = min(nx, 2048), min(ny, 2048)
    top = min(64, min(nx, ny) // 8)
    if dense:
        top = min(top, 40)
    supports = sorted(_log_int(rng, 4, max(5, top))
                      for _ in range(rng.choice([1, 2, 4, 8])))
    cells = sum((s + 1) ** 2 for s in supports) / len(supports)
    planes = 16 if dense else npol
    # at most 2 GB of CF, and at most a tenth of the largest listed case
    most = min(64, int(math.sqrt(2e9 / (8 * planes * sum((s + 4) ** 2
                                                         for s in supports)))))
    os_ = rng.randint(min(8, most), max(9, most))
    nmax = int(min(3e6, 7.4e10 / (cells * planes * 8)))
    if kind == "residual":
        nmax = min(nmax, 200_000)
    if kind == "image":
        nmax = min(nmax, 500_000)
    if kind == "cf_swap":
        nmax = min(nmax, 50_000)
    if kind == "gradient":
        nmax = min(nmax, 1_000_000)
        dense = False
    c = dict(npol=npol, nx=nx, ny=ny,
             supports=",".join(str(s) for s in supports), os=os_,
             nvis=_log_int(rng, 500, nmax), form=form, dense=dense,
             screen=rng.random() < 0.3 and kind != "gradient",
             uv=rng.choice(["disk", "core"]), host=kind == "residual")
    if kind == "batch":
        sides = [_log_int(rng, max(256, 8 * supports[-1]), 2048) & ~1
                 for _ in range(rng.choice([2, 4, 8]))]
        jobs = [(s, _log_int(rng, 500, max(501, nmax // len(sides))))
                for s in sides]
        c["jobs"] = ",".join("%d:%d" % j for j in jobs)
        c["nvis"] = sum(n for _, n in jobs)
        c["screen"] = False
        c["form"] = rng.choice(["fp64", "mixed"])
    return _case(None, kind, **c)


# ---------------------------------------------------------------------------
# inputs

def _supports(c):
    return [int(s) for s in c["supports"].split(",")]


def _taps(support, os_):
    """Taps of a CF of this support: 2 * radius + 1 of its extent."""
    ext = (support + 4) * os_
    return 2 * (((ext - 4 * os_) // os_) // 2) + 1


def _mueller(c):
    """Index table (rows x polarizations, -1 where inactive) and plane count."""
    n = c["npol"]
    if c["dense"]:
        return [[r * n + v for v in range(n)] for r in range(n)], n * n
    return [[r if r == v else -1 for v in range(n)] for r in range(n)], n


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7fffffff)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _cf_values(c, seed):
    """Extents and one complex64 tensor (x, y, mueller, cube) per group."""
    g = _gen(seed + 7_000_001)
    os_, planes = c["os"], _mueller(c)[1]
    n = c["npol"]
    f = torch.complex(_randn(g, planes), _randn(g, planes)) * 0.1
    diag = [r * n + r for r in range(n)] if c["dense"] else list(range(n))
    f[diag] = 1.0 + 0.05 * f[diag]
    extents, values = [], []
    for k, s in enumerate(_supports(c)):
        ext = (s + 4) * os_
        u = (torch.arange(ext, device="cuda", dtype=torch.float64) -
             ext / 2.0) / os_
        a = torch.exp(-0.5 * (u / max(s / 6.0, 0.5)) ** 2)
        ph = math.pi * 0.02 * (k + 0.3) * u * u
        a = torch.complex(a * torch.cos(ph), a * torch.sin(ph))
        xy = (a[:, None] * a[None, :]).to(torch.complex64)
        v = (xy[:, :, None] * f.to(torch.complex64)).unsqueeze(-1)
        values.append(v.contiguous())
        extents.append((ext, ext, planes, 1))
    return extents, values


def _vis_fields(c, nx, ny, n, seed):
    g = _gen(seed)
    npol, ngroups = c["npol"], len(_supports(c))
    f = {"vis": torch.complex(_randn(g, n, npol), _randn(g, n, npol))
         .to(torch.complex64)}
    f["weights"] = (0.5 + _rand(g, n, npol)).to(torch.float32)
    inv_lambda = FREQ / C_LIGHT
    rmax = 0.45 * min(nx, ny)
    r = _rand(g, n)
    r = rmax * (torch.sqrt(r) if c["uv"] == "disk" else r)
    th = 2 * math.pi * _rand(g, n)
    f["uvw"] = torch.empty(n, 3, device="cuda", dtype=torch.float64)
    f["uvw"][:, 0] = r * torch.cos(th) / (GRID_SCALE * inv_lambda)
    f["uvw"][:, 1] = r * torch.sin(th) / (GRID_SCALE * inv_lambda)
    frac = 2 * _rand(g, n) - 1
    f["uvw"][:, 2] = frac * 0.3 * rmax / (GRID_SCALE * inv_lambda)
    f["group"] = (frac.abs() * ngroups).long().clamp_(max=ngroups - 1)
    if c["screen"]:
        f["phase"] = 2 * math.pi * _rand(g, n) - math.pi
        f["grad"] = (2 * _rand(g, n, 2) - 1) * (0.02 / c["os"])
    else:
        f["phase"] = torch.zeros(n, device="cuda", dtype=torch.float64)
        f["grad"] = torch.zeros(n, 2, device="cuda", dtype=torch.float64)
    return f


def _records(f, npol):
    """The fields as a CUDA uint8 tensor of VisData<npol> records."""
    dt = abi.visdata_dtype(npol)
    n = f["vis"].shape[0]
    rec = torch.zeros(n, dt.itemsize, device="cuda", dtype=torch.uint8)

    def put(name, t):
        b = t.contiguous().view(torch.uint8).reshape(n, -1)
        rec[:, dt.fields[name][1]:dt.fields[name][1] + b.shape[1]] = b

    put("vis", torch.view_as_real(f["vis"]).reshape(n, -1))
    put("weights", f["weights"])
    put("freq", torch.full((n, 1), FREQ, device="cuda", dtype=torch.float64))
    put("phase", f["phase"][:, None])
    put("uvw", f["uvw"])
    cfi = torch.zeros(n, 2, device="cuda", dtype=torch.int32)
    cfi[:, 1] = f["group"].to(torch.int32)
    put("cf_index", cfi)
    put("cf_phase_gradient", f["grad"])
    return rec


def _model(c, nx, ny, seed):
    g = _gen(seed + 3_000_017)
    rows = c["npol"]
    return torch.complex(_randn(g, 1, rows, ny, nx), _randn(g, 1, rows, ny, nx))


class _DeviceArray:
    """A device pointer the gridder gives, for torch.as_tensor.  A tensor
    made from it holds this object, and with it the gridder whose memory it
    is."""

    def __init__(self, gridder, ptr, shape, typestr):
        self.gridder = gridder
        self.__cuda_array_interface__ = {
            "data": (ptr, False), "shape": shape, "typestr": typestr,
            "version": 3}


def _views(g):
    nx, ny, nr, nc = g.grid_size
    grid, _ = g.grid_values_ptr()
    weights, _ = g.grid_weights_ptr()
    return (torch.as_tensor(_DeviceArray(g, grid, (nc, nr, ny, nx), "<c16")),
            torch.as_tensor(_DeviceArray(g, weights, (nc, nr), "<f8")))


def _gridder(c, nx, ny, n, cf):
    idx, _ = _mueller(c)
    g = hpg_b200.Gridder.create(
        device=0, max_visibility_batch_size=n,
        grid_size=(nx, ny, c["npol"], 1), grid_scale=(GRID_SCALE, GRID_SCALE),
        mueller_indexes=idx, conjugate_mueller_indexes=idx)
    if c["form"] != "fp64":
        g.set_precision(abi.PRECISION_MIXED)
    if c["form"] == "comp":
        g.set_tiled_plan(compensated=abi.COMPENSATED_ON)
    if cf is not None:
        torch.cuda.synchronize()
        g.set_convolution_function(cf, on_device=True)
    return g


def _jobs(c):
    if c["kind"] != "batch":
        return [(c["nx"], c["ny"], c["nvis"])]
    return [(int(s), int(s), int(n)) for s, n in
            (j.split(":") for j in c["jobs"].split(","))]


def prepare(case, seed):
    c, kind = case, case["kind"]
    extents, values = _cf_values(c, seed)
    cf = hpg_b200.CFArray(c["os"], extents, values)
    s = {"case": c, "gridders": [], "records": [], "views": []}
    for j, (nx, ny, n) in enumerate(_jobs(c)):
        f = _vis_fields(c, nx, ny, n, seed + 101 * j)
        rec = _records(f, c["npol"])
        g = _gridder(c, nx, ny, n, None if kind == "cf_swap" else cf)
        if kind in ("predict", "residual", "cycle"):
            m = _model(c, nx, ny, seed + 101 * j)
            torch.cuda.synchronize()
            g.set_model(m, on_device=True)
            del m
        if kind == "gradient":
            s["model"] = _model(c, nx, ny, seed).requires_grad_()
            s["observed"] = f["vis"].to(torch.complex128)
        if c["host"]:
            rec = rec.cpu().numpy().reshape(-1).view(abi.visdata_dtype(c["npol"]))
        s["gridders"].append(g)
        s["records"].append(rec)
        s["views"].append(_views(g))
    if kind == "cf_swap":
        s["cf"] = cf
    torch.cuda.synchronize()
    return s


def _grid_of(s, j):
    """Grid and weights of gridder j as the program keeps them."""
    grid, weights = s["views"][j]
    if s["case"]["form"] == "fp64":
        return grid, weights
    s["gridders"][j].fence()
    return grid.to(torch.complex64), weights


def run(state):
    c, kind = state["case"], state["case"]["kind"]
    g, rec = state["gridders"][0], state["records"][0]
    if kind == "predict":
        g.degrid_get_predicted_visibilities(rec, on_device=True)
        return rec[:, :8 * c["npol"]].view(torch.float32)
    if kind == "residual":
        g.reset_grid()
        future = g.degrid_grid_get_residual_visibilities(rec)
        weights = g.grid_weights()
        return {"residual": future.get()["vis"], "weights": weights,
                "grid": _grid_of(state, 0)[0]}
    if kind == "gradient":
        model = state["model"]
        predicted = autograd.degrid(model, g, rec.view(-1))
        r = torch.view_as_real(predicted - state["observed"])
        loss = (r * r).sum()
        grad, = torch.autograd.grad(loss, model)
        return {"loss": loss.detach(), "predicted": predicted.detach(),
                "gradient": grad}
    if kind == "batch":
        for h in state["gridders"]:
            h.reset_grid()
        hpg_b200.grid_visibilities_batch(state["gridders"], state["records"],
                                         on_device=True)
        return [_grid_of(state, j) for j in range(len(state["gridders"]))]
    if kind == "cf_swap":
        g.set_convolution_function(state["cf"], on_device=True)
    g.reset_grid()
    if kind == "cycle":
        g.degrid_grid_visibilities(rec, on_device=True)
    else:
        g.grid_visibilities(rec, on_device=True)
    if kind == "image":
        g.image_grid(norm=float(c["nvis"]))
    return _grid_of(state, 0)


# ---------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    c, kind = case, case["kind"]
    npol = c["npol"]
    idx, planes = _mueller(c)
    cells = [_taps(s, c["os"]) ** 2 for s in _supports(c)]
    mean = sum(cells) / len(cells)
    rec = abi.visdata_dtype(npol).itemsize
    passes = {"predict": 1, "grid": 2, "cf_swap": 2, "batch": 2, "residual": 3,
              "cycle": 3, "image": 4, "gradient": 2}[kind]
    macs = {"residual": 2, "cycle": 2, "gradient": 2}.get(kind, 1)
    nbytes = flops = 0.0
    nfine = 2 * (c["os"] // 2) + 1
    table = nfine ** 2 * sum(cells) * planes * 8.0
    for nx, ny, n in _jobs(c):
        # records and the CF slices of all visibilities, once per operator
        # (a slice's visibilities lie all over the grid, so slices are read
        # again unless the whole table is smaller than the L2)
        ops = 2 if kind == "gradient" else 1
        slices = n * mean * planes * 8.0
        nbytes += ops * (n * rec + (min(slices, table) if table < 126e6
                                    else slices))
        nbytes += passes * nx * ny * npol * 16.0
        flops += macs * n * mean * planes * 8.0
        if kind == "image":
            flops += 5.0 * nx * ny * npol * math.log2(nx * ny)
    if kind == "cf_swap":
        for s, t in zip(_supports(c), cells):
            nbytes += 8.0 * planes * (((s + 4) * c["os"]) ** 2 + nfine ** 2 * t)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same results in 64 bits, plain torch

def _coords(c, nx, ny, f, d):
    """Origin, fine offset and tap count along axis d, per visibility."""
    taps_of = torch.tensor([_taps(s, c["os"]) for s in _supports(c)],
                           device="cuda")
    t = taps_of[f["group"]]
    pos = (GRID_SCALE * f["uvw"][:, d]) * (FREQ / C_LIGHT) + (nx, ny)[d] / 2.0
    at = torch.round(pos)
    fine = torch.round((at - pos) * float(c["os"])).long()
    return at.long() - t // 2, fine, t


def _pieces(c, nx, ny, f, cf, model=None, values=None, grid=None,
            conj_adjoint=False):
    """Visits the visibilities group by group in pieces.  With ``model``,
    returns their predictions; with ``values`` (already phased and scaled),
    adds them into ``grid`` (``conj_adjoint``: with the conjugate of the
    degridding factors, which is the adjoint)."""
    npol, os_ = c["npol"], c["os"]
    idx, planes = _mueller(c)
    n = f["vis"].shape[0]
    x0, fx, taps = _coords(c, nx, ny, f, 0)
    y0, fy, _ = _coords(c, nx, ny, f, 1)
    ok = (x0 >= 0) & (y0 >= 0) & (x0 + taps <= nx) & (y0 + taps <= ny)
    pos_w = f["uvw"][:, 2] > 0
    out = torch.zeros(n, npol, device="cuda", dtype=torch.complex128)
    wsum = torch.zeros(n, planes, device="cuda", dtype=torch.complex128)
    for k in range(len(cf)):
        t = _taps(_supports(c)[k], os_)
        radius = t // 2
        cfk = cf[k][..., 0]
        members = torch.nonzero(ok & (f["group"] == k)).reshape(-1)
        step = max(1, int(2.5e8 // (t * t * planes * 16)))
        ar = torch.arange(t, device="cuda")
        for a in range(0, members.numel(), step):
            i = members[a:a + step]
            xs = (2 + ar)[None, :] * os_ + fx[i][:, None]
            ys = (2 + ar)[None, :] * os_ + fy[i][:, None]
            v = cfk[xs[:, None, :], ys[:, :, None]].to(torch.complex128)
            wsum[i] = v.sum(dim=(1, 2))
            # degridding takes the CF for w > 0 and its conjugate otherwise
            v = torch.where(pos_w[i][:, None, None, None], v, v.conj())
            if c["screen"]:
                g = f["grad"][i]
                phx = (-g[:, 0] * (radius * os_ - fx[i]))[:, None] + \
                    ar[None, :] * (g[:, 0] * os_)[:, None]
                phy = (-g[:, 1] * (radius * os_ - fy[i]))[:, None] + \
                    ar[None, :] * (g[:, 1] * os_)[:, None]
                ph = phx[:, None, :] + phy[:, :, None]
                v = v * torch.polar(torch.ones_like(ph), -ph)[..., None]
            gx = (x0[i][:, None, None] + ar[None, None, :])
            gy = (y0[i][:, None, None] + ar[None, :, None])
            at = gy * nx + gx
            for r in range(npol):
                if model is not None:
                    patch = model[0, r].reshape(-1)[at]
                    for q in range(npol):
                        if idx[r][q] >= 0:
                            out[i, q] += (v[..., idx[r][q]] * patch).sum((1, 2))
                if values is not None:
                    add = torch.zeros_like(v[..., 0])
                    for q in range(npol):
                        if idx[r][q] >= 0:
                            add += v[..., idx[r][q]].conj() * \
                                values[i, q][:, None, None]
                    grid[0, r].view(-1).index_add_(0, at.reshape(-1),
                                                   add.reshape(-1))
    return out, wsum, ok, pos_w


def _exact_one(c, nx, ny, n, seed, cf):
    kind, npol = c["kind"], c["npol"]
    idx, planes = _mueller(c)
    f = _vis_fields(c, nx, ny, n, seed)
    model = None
    if kind in ("predict", "residual", "cycle", "gradient"):
        model = _model(c, nx, ny, seed)
    phasor = torch.polar(torch.ones_like(f["phase"]), f["phase"])[:, None]
    vis = f["vis"].to(torch.complex128)
    if model is not None:
        num, wsum, ok, pos_w = _pieces(c, nx, ny, f, cf, model=model)
        ws = torch.where(pos_w[:, None], wsum, wsum.conj())
        den = torch.zeros_like(num)
        for r in range(npol):
            for q in range(npol):
                if idx[r][q] >= 0:
                    den[:, q] += ws[:, idx[r][q]]
        den = torch.where(den == 0, torch.ones_like(den), den)
        factor = phasor.conj() / den
        pred = num * factor
        if kind == "predict":
            v = torch.where(ok[:, None], pred, vis)
            return torch.view_as_real(v).reshape(n, -1)
        if kind == "gradient":
            pred = torch.where(ok[:, None], pred, torch.zeros_like(pred))
            r = pred - vis
            grad = torch.zeros_like(model)
            _pieces(c, nx, ny, f, cf, values=2 * r * factor.conj(), grid=grad)
            return {"loss": (r.real ** 2 + r.imag ** 2).sum(),
                    "predicted": pred, "gradient": grad}
        vis = torch.where(ok[:, None], vis - pred, vis)
    grid = torch.zeros(1, npol, ny, nx, device="cuda", dtype=torch.complex128)
    scaled = vis * phasor * f["weights"].to(torch.float64)
    _, wsum, ok, _ = _pieces(c, nx, ny, f, cf, values=scaled, grid=grid)
    weights = torch.zeros(1, npol, device="cuda", dtype=torch.float64)
    mag = wsum.abs()
    for r in range(npol):
        for q in range(npol):
            if idx[r][q] >= 0:
                weights[0, r] += (mag[:, idx[r][q]] *
                                  f["weights"][:, q].to(torch.float64) *
                                  ok).sum()
    if kind == "residual":
        return {"residual": vis.cpu().numpy(), "weights": weights.cpu().numpy(),
                "grid": grid}
    if kind == "image":
        grid = grid / weights[:, :, None, None]
        grid = torch.fft.ifft2(grid, norm="forward") / float(c["nvis"])
        grid = torch.roll(grid, (ny // 2, nx // 2), (2, 3))
    return grid, weights


def exact(case, seed):
    c = case
    if work(c)["bytes"] > 2e11:
        return None  # the largest case takes too long this way
    _, cf = _cf_values(c, seed)
    got = [_exact_one(c, nx, ny, n, seed + 101 * j, cf)
           for j, (nx, ny, n) in enumerate(_jobs(c))]
    return got if c["kind"] == "batch" else got[0]
