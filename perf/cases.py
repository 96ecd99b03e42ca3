"""The pressure solve's workloads: what a time loop, a training run or a host
program asks of the library, through the package's own entry points.

Every solve runs to a 1e-10 true relative residual, the tolerance of the 32^3
and 128^3 workloads, so that two solvers' pressures agree to about ten digits
whatever path their iterations took.  Right-hand sides are the k^-11/3 spectral
fields of the Ornstein-Uhlenbeck sequence (uniform noise on the sphere-free
periodic box), masks are seeded non-overlapping spheres.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bluebottle-3.0_gb300"))

import bbpp  # noqa: E402
from bbpp import learned, problems  # noqa: E402

TOL = 1e-10
DEV = "cuda"


def _solve(name, nx, ny, nz, bc, nsph, rad, precision, guess, rhs="spectral", host=False, iso=False):
    c = dict(kind="solve", nx=nx, ny=ny, nz=nz, bc=bc, nsph=nsph, rad=rad, precision=precision, guess=guess, rhs=rhs,
             host=host, iso=iso)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: the 32^3 periodic box without particles; launches and host round trips decide it
        _solve("fp64_32_ppp", 32, 32, 32, "ppp", 0, 0, "fp64", "zero", rhs="uniform"),
        # one solve of the training-set generator: 2000 of these make the learned guess's data
        _solve("fp64_64", 64, 64, 64, "ppn", 128, 4, "fp64", "zero"),
        # the reference's method on a closed box with odd extents: walls on every side, no vector-friendly width
        _solve("fp64_ragged_nnn", 101, 75, 58, "nnn", 24, 6, "fp64", "zero"),
        # the reference's method at its ordinary and at its largest size here
        _solve("fp64_128", 128, 128, 128, "ppn", 64, 8, "fp64", "zero"),
        _solve("fp64_256", 256, 256, 256, "ppn", 1000, 6, "fp64", "zero"),
        # mixed precision through host buffers, as a program without its own device data calls it
        _solve("mixed_host_128", 128, 128, 128, "ppn", 64, 8, "mixed", "zero", host=True),
        # mixed precision on an anisotropic channel whose rows the tensor copies do not take
        _solve("mixed_ragged_pnn", 200, 144, 106, "pnn", 60, 7, "mixed", "zero"),
        # mixed precision in a time loop: from the previous step's pressure, and from the learned guess
        _solve("mixed_256_warm", 256, 256, 256, "ppn", 1000, 6, "mixed", "given"),
        _solve("mixed_256_learned", 256, 256, 256, "ppn", 1000, 6, "mixed", "learned"),
        # the largest: 134M cells, 4000 spheres, from the previous step's pressure
        _solve("mixed_512_warm", 512, 512, 512, "ppn", 4000, 5, "mixed", "given"),
        # one training step's loss and gradients: a batch of four 64^3 samples
        dict(kind="train", name="train_64_b4", n=64, nb=4, nsph=128, rad=4),
        # what a time loop builds around the solve: the particle mask, the right-hand side from u*, the residual of
        # the previous pressure
        dict(kind="build", name="build_256", nx=256, ny=256, nz=256, bc="ppn", nsph=1000, rad=6),
    ]


def draw(rng):
    what = rng.choice(["fp64", "fp64", "mixed", "mixed", "mixed", "train", "build"])
    if what == "train":
        n = rng.choice([32, 48, 64])
        return dict(kind="train", n=n, nb=rng.randint(1, 6), nsph=max(1, 128 * n ** 3 // 64 ** 3), rad=4)

    def extent(lo, hi):
        e = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        grain = rng.choice([1, 1, 2, 4, 32])  # odd ones, and the multiples that grids are often made of
        return max(lo, e // grain * grain)

    if what == "build":
        nx, ny, nz = extent(32, 256), extent(32, 256), extent(32, 256)
    elif rng.random() < 0.4:  # a cube of a common size
        nx = ny = nz = rng.choice([32, 64, 96, 128, 160, 192, 256] if what == "mixed" else [32, 48, 64, 96, 128, 192])
    else:
        hi = 288 if what == "mixed" else 160
        nx = extent(24, hi)
        ny, nz = (min(hi, max(24, int(nx * rng.uniform(0.5, 2.0)))) for _ in range(2))
    rad = rng.choice([4, 5, 6, 8])
    fit = max(0, min(nx, ny, nz) - 2 * rad - 2)
    nsph = int(rng.uniform(0.0, 0.08) * nx * ny * nz / (4.19 * rad ** 3)) if fit else 0
    bc = rng.choice(["ppn", "ppn", "ppp", "nnn", "pnn", "npn", "nnp"])
    if what == "build":
        return dict(kind="build", nx=nx, ny=ny, nz=nz, bc=bc, nsph=max(1, nsph), rad=rad)
    guess = rng.choice(["zero", "zero", "given"])
    if what == "mixed" and nx % 8 == ny % 8 == nz % 8 == 0 and rng.random() < 0.3:
        guess, bc = "learned", "ppn"
    return _solve(None, nx, ny, nz, bc, nsph, rad, what, guess, rhs=rng.choice(["spectral", "spectral", "uniform"]),
                  host=rng.random() < 0.15 and guess != "learned", iso=rng.random() < 0.5)


# ------------------------------------------------------------------ inputs --
def _grid(c):
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    h = 1.0 / max(nx, ny, nz)
    d = (h, h, h) if c.get("iso") else (1.0 / nx, 1.0 / ny, 1.0 / nz)
    return bbpp.Grid.make(nx, ny, nz, *d, problems.bc_tuple(c["bc"]))


def _place(grid, nsph, rad_cells, seed):
    """Non-overlapping spheres of rad_cells finest cells, at least a cell apart and off the walls (no pocket of fluid
    is cut off), by seeded rejection on a cell list.  May place fewer than asked."""
    rng = np.random.RandomState(seed & 0x7FFFFFFF)
    L = np.array([grid.nx * grid.dx, grid.ny * grid.dy, grid.nz * grid.dz])
    h = max(grid.dx, grid.dy, grid.dz)
    r = rad_cells * min(grid.dx, grid.dy, grid.dz)
    per = np.array([grid.bc[0] == bbpp.PERIODIC, grid.bc[2] == bbpp.PERIODIC, grid.bc[4] == bbpp.PERIODIC])
    gap = 2 * r + 2 * h
    lo = np.where(per, 0.0, r + 2 * h)
    hi = np.where(per, L, L - r - 2 * h)
    if np.any(hi <= lo) or np.any(L < 2 * gap):
        return np.zeros((0, 3)), np.zeros(0)
    ncell = np.maximum(1, np.floor(L / gap).astype(int))
    cells, out = {}, []
    for u in rng.random_sample((40 * nsph, 3)):
        if len(out) == nsph:
            break
        p = lo + (hi - lo) * u
        at = np.minimum((p / L * ncell).astype(int), ncell - 1)
        ok = True
        for o in np.ndindex(3, 3, 3):
            q = at + np.array(o) - 1
            if np.any(~per & ((q < 0) | (q >= ncell))):
                continue
            for b in cells.get(tuple(q % ncell), ()):
                d = p - b
                d = np.where(per, d - L * np.round(d / L), d)
                if d @ d < gap * gap:
                    ok = False
                    break
            if not ok:
                break
        if ok:
            cells.setdefault(tuple(at), []).append(p)
            out.append(p)
    return np.array(out).reshape(-1, 3), np.full(len(out), r)


_PLACED = {}


def _spheres(c, grid, seed):
    """The geometry of a case and seed (placing 4000 spheres takes a while: kept for the next state of this seed)."""
    key = (grid.as_tuple(), c["nsph"], c["rad"], seed)
    if key not in _PLACED:
        if len(_PLACED) > 64:
            _PLACED.clear()
        _PLACED[key] = _place(grid, c["nsph"], c["rad"], seed)
    return _PLACED[key]


def _mask(grid, cents, radii):
    """Cells whose centre lies inside a sphere, on the GPU (sphere by sphere boxes, periodic images)."""
    m = torch.zeros(grid.shape, dtype=torch.uint8, device=DEV)
    if not len(radii):
        return m
    n = np.array([grid.nx, grid.ny, grid.nz])
    d = np.array([grid.dx, grid.dy, grid.dz])
    per = np.array([grid.bc[0] == bbpp.PERIODIC, grid.bc[2] == bbpp.PERIODIC, grid.bc[4] == bbpp.PERIODIC])
    w = np.ceil(radii[0] / d).astype(int) + 1
    off = torch.stack(torch.meshgrid(*[torch.arange(-int(k), int(k) + 1, device=DEV) for k in w], indexing="ij"),
                      -1).reshape(-1, 3)
    dt, nt = torch.as_tensor(d, device=DEV), torch.as_tensor(n, device=DEV)
    for k in range(0, len(radii), 512):
        p = torch.as_tensor(cents[k:k + 512], device=DEV)
        idx = torch.floor(p / dt).long()[:, None, :] + off[None]
        dist = ((idx.double() + 0.5) * dt - p[:, None, :]).square().sum(-1).sqrt()
        inside = dist < float(radii[0])
        pt = torch.as_tensor(per, device=DEV)
        inside &= (pt | ((idx >= 0) & (idx < nt))).all(-1)
        q = torch.where(pt, idx % nt, idx)[inside]
        m.view(-1)[q[:, 0] + grid.nx * (q[:, 1] + grid.ny * q[:, 2])] = 1
    return m


def _rhs_fields(c, grid, mask, seed, count):
    """`count` consecutive right-hand sides: zero on solid cells, zero mean over the fluid, unit RMS."""
    if c["rhs"] == "uniform":
        gen = torch.Generator(device=DEV)
        out = []
        for k in range(count):
            gen.manual_seed(seed * 31 + k)
            f = torch.rand(grid.shape, generator=gen, dtype=torch.float64, device=DEV) * 2 - 1
            fluid = mask == 0
            f = torch.where(fluid, f, torch.zeros_like(f))
            out.append(f - fluid * (f.sum() / fluid.sum()))
        return out
    seq = problems.OUSequenceDevice(grid.shape, seed, mask.cpu().numpy())
    out = [seq.field().clone()]
    for _ in range(count - 1):
        out.append(seq.step().clone())
    return out


def _solve_inputs(c, seed, count):
    """Grid, mask tensor (None without spheres) and `count` right-hand sides."""
    grid = _grid(c)
    cents, radii = _spheres(c, grid, seed)
    mask = _mask(grid, cents, radii)
    fields = _rhs_fields(c, grid, mask, seed, count)
    return grid, (mask if len(radii) else None), fields


def _view(t):
    return None if t is None else bbpp.DeviceView.of_tensor(t)


def _prepare_solve(c, seed):
    warm = c["guess"] in ("given", "learned")
    grid, mask, fields = _solve_inputs(c, seed, 2 if warm else 1)
    s = bbpp.Solver(grid)
    st = dict(kind="solve", solver=s, host=c["host"], rhs=fields[-1], mask=mask, guess=c["guess"],
              x=torch.zeros(grid.shape, dtype=torch.float64, device=DEV))
    st["kw"] = dict(tol=TOL, precision=bbpp.FP64 if c["precision"] == "fp64" else bbpp.FP32_IR,
                    guess={"zero": bbpp.GUESS_ZERO, "given": bbpp.GUESS_GIVEN, "learned": bbpp.GUESS_LEARNED}[c["guess"]])
    if warm:  # the time loop's previous pressure: the previous right-hand side's solution
        prev = torch.zeros_like(st["x"])
        torch.cuda.synchronize()
        s.solve(_view(fields[0]), _view(prev), _view(mask), tol=TOL, precision=bbpp.FP32_IR)
        st["prev"] = prev
    if c["guess"] == "learned":
        st["net"] = learned.Net(seed=5)
        # a head of small weights stands for the trained network: its correction is of the size of a warm start's
        st["net"].set_params(st["net"].get_params() * np.float32(0.5))
        st["kw"]["net"] = st["net"]
        st["kw"]["prev"] = st["prev"].data_ptr()
    if c["host"]:
        st["rhs"] = st["rhs"].cpu().numpy()
        st["mask"] = None if mask is None else mask.cpu().numpy()
        st["prev"] = st["prev"].cpu().numpy() if warm else None
    else:
        # the program's own stream, on which it also sets the starting pressure
        st["stream"] = torch.cuda.Stream()
        bbpp.lib().bbpp_set_stream(s.handle, st["stream"].cuda_stream)
    torch.cuda.synchronize()
    return st


def _run_solve(st):
    if st["host"]:
        x, _ = st["solver"].solve_host(st["rhs"], st["mask"], x0=st["prev"], **st["kw"])
        return x
    if st["guess"] == "given":
        with torch.cuda.stream(st["stream"]):
            st["x"].copy_(st["prev"])
    st["solver"].solve(_view(st["rhs"]), _view(st["x"]), _view(st["mask"]), **st["kw"])
    return st["x"]


def _inverse_laplacian(f, h2):
    """The periodic Poisson solution of f by FFT (FP64)."""
    n = f.shape[0]
    k = 2.0 - 2.0 * torch.cos(2 * math.pi * torch.arange(n, dtype=torch.float64, device=DEV) / n)
    lam = (k[:, None, None] + k[None, :, None] + k[None, None, :]) / h2
    lam[0, 0, 0] = 1.0
    hat = torch.fft.fftn(f) / lam
    hat[0, 0, 0] = 0
    return torch.fft.ifftn(hat).real


def _prepare_train(c, seed):
    n, nb = c["n"], c["nb"]
    grid = _grid(dict(nx=n, ny=n, nz=n, bc="ppn"))
    cents, radii = _spheres(c, grid, seed)
    mask = _mask(grid, cents, radii)
    seq = problems.OUSequenceDevice(grid.shape, seed, mask.cpu().numpy())
    h2 = grid.dx * grid.dy
    fluid = (mask == 0).double()
    f0 = seq.field().clone()
    r, prev, tgt = [], [], []
    for _ in range(nb):  # the residual of the previous pressure, that pressure, the correction it needs
        f1 = seq.step().clone()
        r.append((f1 - f0) * fluid)
        prev.append(_inverse_laplacian(f0, h2) * fluid)
        tgt.append(_inverse_laplacian(f1 - f0, h2) * fluid)
        f0 = f1
    st = dict(kind="train", dims=(n, n, n), h2=h2, net=learned.Net(seed=seed % 1000 + 1))
    for name, v in (("r", r), ("prev", prev), ("target", tgt)):
        st[name] = bbpp.DeviceArray.from_host(torch.stack(v).float().cpu().numpy())
    st["mask"] = bbpp.DeviceArray.from_host(mask.cpu().numpy())
    torch.cuda.synchronize()
    return st


def _run_train(st):
    loss, grads = st["net"].loss_grad(st["dims"], st["h2"], st["r"], st["prev"], st["target"], st["mask"])
    return dict(loss=loss, grads=grads)


def _prepare_build(c, seed):
    grid = _grid(c)
    nx, ny, nz = grid.nx, grid.ny, grid.nz
    cents, radii = _spheres(c, grid, seed)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    rnd = lambda *s: torch.randn(s, generator=gen, dtype=torch.float64, device=DEV)  # noqa: E731
    st = dict(kind="build", solver=bbpp.Solver(grid), cents=cents, radii=radii, u=rnd(nz, ny, nx + 1),
              v=rnd(nz, ny + 1, nx), w=rnd(nz + 1, ny, nx), p=rnd(nz, ny, nx) * grid.dx,
              mask=torch.zeros(grid.shape, dtype=torch.uint8, device=DEV),
              rhs=torch.zeros(grid.shape, dtype=torch.float64, device=DEV),
              res=torch.zeros(grid.shape, dtype=torch.float64, device=DEV))
    torch.cuda.synchronize()
    return st


RHO, DT = 1.0, 1e-3


def _run_build(st):
    s = st["solver"]
    s.sphere_mask(st["cents"], st["radii"], _view(st["mask"]))
    s.rhs_div(RHO, DT, _view(st["u"]), _view(st["v"]), _view(st["w"]), _view(st["rhs"]))
    rr, bb = s.residual(_view(st["rhs"]), _view(st["p"]), _view(st["res"]), _view(st["mask"]))
    return dict(mask=st["mask"], rhs=st["rhs"], res=st["res"], rr=rr, bb=bb)


def prepare(case, seed):
    return {"solve": _prepare_solve, "train": _prepare_train, "build": _prepare_build}[case["kind"]](case, seed)


def run(state):
    return {"solve": _run_solve, "train": _run_train, "build": _run_build}[state["kind"]](state)


# -------------------------------------------------------------------- work --
def _iterations(c):
    """About the iterations of a Jacobi PCG to TOL on this machine: CG's bound 0.5 sqrt(kappa) ln(2 / tol) of the longest
    mode (a periodic axis holds half a closed one's wavelength), times 0.25, what the named workloads take of it."""
    ext = [c["nx"], c["ny"], c["nz"]]
    longest = max(e if b == "n" else e / 2 for e, b in zip(ext, c["bc"]))
    return 0.25 * 0.5 * 1.1 * longest * math.log(2 / TOL)


def work(case):
    if case["kind"] == "train":
        # 3x3x3 convolutions of three levels (one multiply-add each of 27 cin cout a voxel), forward and both
        # gradients; the first layer needs no input gradient
        vox = case["n"] ** 3 * case["nb"]
        layers = [(16, 16, 1.0), (16, 32, 1 / 8), (32, 64, 1 / 64), (96, 32, 1 / 8), (48, 16, 1.0)]
        fl = sum(3 * 2 * 27 * a * b * f for a, b, f in layers) * vox
        return {"bytes": 12.0 * vox, "flops": fl}
    n = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "build":
        # u, v, w and the mask in, rhs out; rhs, p and the mask in, the residual out
        return {"bytes": n * (32.0 + 1 + 24 + 1), "flops": n * 20.0}
    it = _iterations(case)
    es = 8 if case["precision"] == "fp64" else 4
    # an iteration reads and writes p, r and x and reads the mask
    return {"bytes": it * n * (6.0 * es + (1 if case["nsph"] else 0)), "flops": it * n * 20.0}


# ------------------------------------------------------------------- exact --
class _Op:
    """(-A) of the 7-point Laplacian in torch FP64: periodic or closed axes, solid cells decoupled."""

    def __init__(self, grid, mask):
        self.c = [1 / grid.dz ** 2, 1 / grid.dy ** 2, 1 / grid.dx ** 2]
        self.per = [grid.bc[4] == bbpp.PERIODIC, grid.bc[2] == bbpp.PERIODIC, grid.bc[0] == bbpp.PERIODIC]
        self.fluid = None if mask is None else (mask == 0)
        diag = torch.zeros(grid.shape, dtype=torch.float64, device=DEV)
        for a in range(3):
            diag += 2 * self.c[a]
            if not self.per[a]:
                diag.select(a, 0).sub_(self.c[a])
                diag.select(a, -1).sub_(self.c[a])
        self.diag = diag

    def __call__(self, p):
        out = self.diag * p
        for a in range(3):
            n = p.shape[a]
            out.narrow(a, 1, n - 1).sub_(p.narrow(a, 0, n - 1), alpha=self.c[a])
            out.narrow(a, 0, n - 1).sub_(p.narrow(a, 1, n - 1), alpha=self.c[a])
            if self.per[a]:
                out.select(a, 0).sub_(p.select(a, n - 1), alpha=self.c[a])
                out.select(a, n - 1).sub_(p.select(a, 0), alpha=self.c[a])
        if self.fluid is not None:
            out *= self.fluid
        return out


def _exact_solve(c, seed):
    """Jacobi CG from zero in FP64 to 1e-13 (the D-weighted mean of the start, zero, is kept: the same member of the
    pressure's one-parameter family; a warm start is itself a solution from zero)."""
    if c["guess"] == "learned" or c["nx"] * c["ny"] * c["nz"] > 300 ** 3:
        return None  # the network's correction moves the mean; the largest takes too long
    grid, mask, fields = _solve_inputs(c, seed, 2 if c["guess"] == "given" else 1)
    b, A = fields[-1], _Op(grid, mask)
    dinv = 1.0 / A.diag
    x = torch.zeros_like(b)
    r = b.clone()
    z = r * dinv
    p = z.clone()
    rz = (r * z).sum()
    bb = float((b * b).sum())
    for q in range(1, 20001):
        Ap = A(p)
        al = rz / (p * Ap).sum()
        x.addcmul_(p, al)
        if q % 50 == 0:
            r = b - A(x)
            if float((r * r).sum()) <= 1e-26 * bb:
                break
        else:
            r.addcmul_(Ap, -al)
        z = r * dinv
        rz1 = (r * z).sum()
        p.mul_(rz1 / rz).add_(z)
        rz = rz1
    return x.cpu().numpy() if c["host"] else x


def _exact_build(c, seed):
    st = _prepare_build(c, seed)
    grid = st["solver"].grid
    st["solver"].close()
    rhs = -(RHO / DT) * ((st["u"][:, :, 1:] - st["u"][:, :, :-1]) / grid.dx + (st["v"][:, 1:] - st["v"][:, :-1]) / grid.dy
                         + (st["w"][1:] - st["w"][:-1]) / grid.dz)
    # the residual entry point keeps the reference's solid rows (an identity row's scale), so it has no value here
    return dict(mask=None, rhs=rhs, res=None, rr=None, bb=float((rhs * rhs).sum()))


def exact(case, seed):
    if case["kind"] == "solve":
        return _exact_solve(case, seed)
    if case["kind"] == "build":
        return _exact_build(case, seed)
    return None
