"""Workloads that stand for what a user of cedar_b200 has it do.

Every case runs one pass through the public entry points: the solver classes of
``cedar_b200.solver``, the differentiable solve of ``cedar_b200.autograd``, or the
kernel entry points of the C ABI that Cedar's kernel registry binds.  Kinds:

* ``host2d``     a small Poisson problem solved from host arrays (latency);
* ``solve2d``    2D solves on device arrays: five-point Poisson with point
                 relaxation, nine-point finite elements with line relaxation, FP64
                 and FP32 cycles inside FP64 refinement;
* ``fcg2d``      strongly heterogeneous diffusion by flexible CG;
* ``solve3d``    3D solves: 27-point finite elements with point or plane
                 relaxation, seven-point Poisson;
* ``batch2d``    many independent 2D problems of several sizes in one mixed batch;
* ``inverse2d``  one gradient step of the inverse-diffusion problem (forward and
                 adjoint solves of a batch, hierarchies set up on the new operators);
* ``kernels2d``  one level of a cycle by kernel calls on Cedar's unpadded rows.

``exact`` gives the same outputs in 64 bits from plain torch: sine transforms for
constant coefficients, a block-tridiagonal factorization for 2D operators,
Jacobi-preconditioned CG for 3D ones.
"""
import ctypes
import math

import numpy as np
import torch

from cedar_b200 import _lib, gallery
from cedar_b200.autograd import solve_log_diffusion_batch
from cedar_b200.config import Config
from cedar_b200.solver import MixedBatchSolver2D, Solver2D, Solver3D

F64 = torch.float64
EDGES = (63, 127, 255, 511, 1023)  # edge sizes of a mixed batch, weights 8:4:2:1:1


def listed():
    return [
        # a small model problem, host buffers in and out: launches and latency
        dict(name="poisson_host_64x48", kind="host2d", nx=64, ny=48),
        # the reference's CPU benchmark size: five-point Poisson, FP64, V(2,1) point relaxation
        dict(name="poisson_511_f64", kind="solve2d", op="poisson", nx=511, ny=511, relax="point",
             precision="fp64", tol=1e-10),
        # nine-point heterogeneous diffusion on a ragged grid: the drop-in FP64 line smoother
        dict(name="lines_1300x900_f64", kind="solve2d", op="hetero", nx=1300, ny=900, relax="line-xy",
             precision="fp64", tol=1e-8),
        # the largest single 2D problem: FP32 cycles inside FP64 refinement
        dict(name="lines_2047_f32ir", kind="solve2d", op="constant", nx=2047, ny=2047, relax="line-xy",
             precision="fp32-ir", tol=1e-10),
        # high-contrast anisotropic diffusion at full size (the benchmark's headline problem)
        dict(name="fcg_2047_f32ir", kind="fcg2d", nx=2047, ny=2047, precision="fp32-ir"),
        # 3D finite elements at full size, the eight-colour point smoother
        dict(name="fe3d_255_point_f32ir", kind="solve3d", op="hetero", nx=255, ny=255, nz=255, relax="point",
             precision="fp32-ir", tol=1e-10),
        # the same smoother in FP64 on a smaller ragged box
        dict(name="fe3d_120x97x75_point_f64", kind="solve3d", op="hetero", nx=120, ny=97, nz=75, relax="point",
             precision="fp64", tol=1e-8),
        # plane relaxation: batched 2D cycles over all planes of a box
        dict(name="fe3d_111x95x79_planes_f32ir", kind="solve3d", op="hetero", nx=111, ny=95, nz=79,
             relax="plane-xyz", precision="fp32-ir", tol=1e-8),
        # seven-point Poisson (the reference's 3D test problem), FP64
        dict(name="poisson3d_200_f64", kind="solve3d", op="poisson", nx=200, ny=200, nz=200, relax="point",
             precision="fp64", tol=1e-8),
        # a work list of independent problems of several sizes, solved together
        dict(name="batch_256_f32ir", kind="batch2d", count=256, sizes_seed=7),
        # one gradient step over a batch: setup, forward, adjoint, coefficient gradient
        dict(name="inverse_8x511", kind="inverse2d", count=8, n=511),
        # one fine level of a cycle through the kernel registry's entry points, unpadded rows
        dict(name="kernels_1000x701_f64", kind="kernels2d", nx=1000, ny=701, nstencil=5, relax="point"),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host2d", "solve2d", "solve2d", "fcg2d", "solve3d", "solve3d", "batch2d", "inverse2d",
                       "kernels2d"])
    if kind == "host2d":
        n = _logint(rng, 33, 200)
        return dict(kind=kind, nx=n, ny=max(33, int(n * rng.uniform(0.6, 1.0))))
    if kind == "solve2d":
        op = rng.choice(["poisson", "hetero", "constant"])
        nx = _logint(rng, 100, 2047)
        # point relaxation of a unit-square problem: steps of similar size in x and y
        ny = int(nx * rng.uniform(0.6, 1.0)) if op == "poisson" else _logint(rng, 100, 2047)
        return dict(kind=kind, op=op, nx=nx, ny=ny,
                    relax="point" if op == "poisson" else "line-xy", precision=rng.choice(["fp64", "fp32-ir"]),
                    tol=1e-8 if op == "hetero" else 1e-10)
    if kind == "fcg2d":
        n = _logint(rng, 400, 2000)
        return dict(kind=kind, nx=n, ny=n, precision=rng.choice(["fp64", "fp32-ir"]))
    if kind == "solve3d":
        op, relax = rng.choice([("hetero", "point"), ("hetero", "point"), ("hetero", "plane-xyz"),
                                ("poisson", "point")])
        hi = 90 if relax == "plane-xyz" else 160
        n = _logint(rng, 31, hi)
        dims = [n] + [max(31, int(n * rng.uniform(0.7, 1.0))) for _ in range(2)]
        rng.shuffle(dims)
        return dict(kind=kind, op=op, nx=dims[0], ny=dims[1], nz=dims[2], relax=relax,
                    precision=rng.choice(["fp64", "fp32-ir"]), tol=1e-8)
    if kind == "batch2d":
        return dict(kind=kind, count=_logint(rng, 16, 256), sizes_seed=rng.randrange(1000))
    if kind == "inverse2d":
        n = _logint(rng, 63, 511)
        return dict(kind=kind, count=rng.randint(1, 8), n=n)
    return dict(kind=kind, nx=_logint(rng, 100, 1500), ny=_logint(rng, 100, 1500), nstencil=rng.choice([3, 5]),
                relax=rng.choice(["point", "line-xy"]))


# ------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1 + seed)
    return g


def _field(shape, ell, sigma, g):
    """Gaussian random field on cell centres (any dimension): white noise shaped by the
    Gaussian covariance of length ell on the doubled box, standard deviation sigma."""
    full = [2 * s for s in shape] if len(shape) == 2 else list(shape)
    h = 1.0 / max(shape)
    k2 = 0.0
    for a, m in enumerate(full):
        freq = torch.fft.rfftfreq if a == len(full) - 1 else torch.fft.fftfreq
        f = freq(m, d=h, device="cuda", dtype=F64) * 2 * math.pi
        k2 = k2 + (f * f).reshape([-1 if b == a else 1 for b in range(len(full))])
    noise = torch.randn(full, generator=g, dtype=F64, device="cuda")
    fld = torch.fft.irfftn(torch.fft.rfftn(noise) * torch.exp(-0.25 * ell * ell * k2), s=full)
    fld = fld[tuple(slice(0, s) for s in shape)]
    fld = fld - fld.mean()
    return (fld * (sigma / fld.std())).contiguous()


def _boxes(shape, count, contrast, g, smin, smax):
    """Factor per cell: ``contrast`` inside ``count`` random boxes."""
    fac = torch.ones(shape, dtype=F64, device="cuda")
    u = torch.rand((count, 2, len(shape)), generator=g, dtype=F64, device="cuda").tolist()
    for size, org in u:
        sl = []
        for s, o, n in zip(size, org, shape):
            w = smin + (smax - smin) * s
            lo = o * (1 - w)
            sl.append(slice(math.ceil(lo * n - 0.5), math.ceil((lo + w) * n - 0.5)))
        fac[tuple(sl)] = contrast
    return fac


def _coefficients2(case, seed):
    """Cell coefficients (kx, ky) of a 2D finite-element operator."""
    nc = (case["ny"] + 1, case["nx"] + 1)
    g = _gen(seed)
    if case["kind"] == "fcg2d":
        k = torch.exp(_field(nc, 1.0 / 32, 2.0, g)) * _boxes(nc, 64, 1e4, g, 1.0 / 64, 1.0 / 8)
        ky = k.clone()
        ky[(torch.arange(nc[0], device="cuda") + 0.5) / nc[0] > 0.5] *= 1e-3
        return k, ky
    if case["op"] == "constant":
        k = torch.ones(nc, dtype=F64, device="cuda")
    else:
        k = torch.exp(_field(nc, 1.0 / 32, 1.0, g))
    return k, k


def _coefficients3(case, seed):
    nc = (case["nz"] + 1, case["ny"] + 1, case["nx"] + 1)
    g = _gen(seed)
    return torch.exp(_field(nc, 1.0 / 16, 1.5, g)) * _boxes(nc, 16, 1e3, g, 1.0 / 32, 1.0 / 8)


def _rhs(case, seed, lo=0.0):
    """b = U[lo, 1] h^d on the interior, zero ghosts; unpadded rows."""
    dims = [case[a] for a in ("nz", "ny", "nx") if a in case]
    h = 1.0 / (dims[-1] + 1)
    g = _gen(seed + 1000003)
    b = torch.zeros([m + 2 for m in dims], dtype=F64, device="cuda")
    inner = tuple(slice(1, m + 1) for m in dims)
    b[inner] = (lo + (1.0 - lo) * torch.rand(dims, generator=g, dtype=F64, device="cuda")) * h ** len(dims)
    return b


def _poisson_rhs(case, seed):
    """A smooth source with noise, h^d (sin sin [sin] + U[-1e-3, 1e-3])."""
    dims = [case[a] for a in ("nz", "ny", "nx") if a in case]
    f = torch.ones([1] * len(dims), dtype=F64, device="cuda")
    for a, m in enumerate(dims):
        s = torch.sin(math.pi * torch.arange(1, m + 1, dtype=F64, device="cuda") / (m + 1))
        f = f * s.reshape([-1 if b == a else 1 for b in range(len(dims))])
    f = f + 2e-3 * (torch.rand(dims, generator=_gen(seed), dtype=F64, device="cuda") - 0.5)
    b = torch.zeros([m + 2 for m in dims], dtype=F64, device="cuda")
    vol = 1.0
    for m in dims:
        vol /= m + 1
    b[tuple(slice(1, m + 1) for m in dims)] = f * vol
    return b


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _padded(t, mult):
    pitch = -(-t.shape[-1] // mult) * mult
    out = torch.zeros(t.shape[:-1] + (pitch,), dtype=F64, device="cuda")
    out[..., :t.shape[-1]] = t
    return out


def _assemble2(kx, ky, pitch):
    ny, nx = kx.shape[0] - 1, kx.shape[1] - 1
    so = torch.zeros((5, ny + 2, pitch), dtype=F64, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(_lib.load().cdr_gpu_fe_assemble_2d_f64(_ptr(kx), _ptr(ky), nx + 1, _ptr(so), nx, ny, pitch,
                                                      ctypes.c_void_p(st)))
    return so


def _operator2(case, seed):
    if case["kind"] in ("solve2d", "host2d") and case.get("op", "poisson") == "poisson":
        return gallery.poisson(case["nx"], case["ny"])
    kx, ky = _coefficients2(case, seed)
    return _assemble2(kx, ky, case["nx"] + 2).cpu().numpy()


def _solver_conf(case):
    if case["kind"] == "host2d":
        return Config({"solver": {"max-iter": 30, "tol": 1e-8}})
    if case["kind"] == "fcg2d":
        levels, m = 1, min(case["nx"], case["ny"])
        while m > 64:
            m = (m - 1) // 2 + 1
            levels += 1
        return Config({"solver": {"relaxation": "line-xy", "tol": 1e-3, "max-iter": 400, "num-levels": levels,
                                  "cycle": {"nrelax-pre": 1, "nrelax-post": 1}},
                       "gpu": {"precision": case["precision"], "krylov": "fcg", "coarse-solve": "inverse",
                               "fcg-replace": 10}})
    return Config({"solver": {"relaxation": case["relax"], "max-iter": 100, "tol": case["tol"]},
                   "gpu": {"precision": case["precision"]}})


def _batch_sizes(case):
    w = np.array([8, 4, 2, 1, 1], dtype=float)
    sizes = np.random.default_rng(case["sizes_seed"]).choice(np.array(EDGES), size=case["count"], p=w / w.sum())
    return [(int(n), int((sizes == n).sum())) for n in sorted(set(sizes.tolist()), reverse=True)]


def _batch_class(n, nb, seed):
    """Coefficients and right-hand sides of nb problems of edge n."""
    sub = dict(kind="solve2d", op="hetero", nx=n, ny=n)
    ks = [_coefficients2(sub, seed + 7919 * (n + 1) + p)[0] for p in range(nb)]
    return ks, [_rhs(sub, seed + 7919 * (n + 1) + p) for p in range(nb)]


def _inverse_inputs(case, seed):
    n, nb = case["n"], case["count"]
    g = _gen(seed)
    th = torch.stack([_field((n + 1, n + 1), 1.0 / 32, 1.0, g) for _ in range(nb)]).to(torch.float32)
    obs = torch.stack([_field((n + 1, n + 1), 1.0 / 32, 1.0, g) for _ in range(nb)])
    f = torch.zeros((nb, n + 2, n + 2), dtype=F64, device="cuda")
    pts = torch.randint(1, n + 1, (nb, 8, 2), generator=g, device="cuda").tolist()
    for p, src in enumerate(pts):
        for i, j in src:
            f[p, j, i] += 1.0
    return th, obs, f


def _level_inputs(case, seed):
    """One level of a hierarchy: operator, right-hand side, interpolation weights,
    a coarse correction; rows unpadded."""
    nx, ny = case["nx"], case["ny"]
    g = _gen(seed)
    if case["nstencil"] == 5:
        so = _assemble2(*_coefficients2(dict(case, op="hetero"), seed), nx + 2)
    else:
        so = torch.from_numpy(gallery.poisson(nx, ny)).cuda()
    nxc, nyc = (nx - 1) // 2 + 1, (ny - 1) // 2 + 1
    # weights near bilinear: 1/2 on edges, 1/4 at cell centres
    ci = torch.zeros((8, nyc + 2, nxc + 2), dtype=F64, device="cuda")
    half = torch.tensor([0.5] * 4 + [0.25] * 4, dtype=F64, device="cuda").reshape(8, 1, 1)
    ci[:, 1:, 1:] = half * (0.8 + 0.4 * torch.rand((8, nyc + 1, nxc + 1), generator=g, dtype=F64, device="cuda"))
    b = _rhs(case, seed)
    xc = torch.zeros((nyc + 2, nxc + 2), dtype=F64, device="cuda")
    xc[1:-1, 1:-1] = 1e-2 * torch.rand((nyc, nxc), generator=g, dtype=F64, device="cuda")
    return so, b, ci, xc


def prepare(case, seed):
    kind = case["kind"]
    if kind == "host2d":
        return dict(kind=kind, solver=Solver2D(_operator2(case, seed), _solver_conf(case)),
                    b=_poisson_rhs(case, seed).cpu().numpy())
    stream = torch.cuda.Stream()
    st = dict(kind=kind, stream=stream)
    if kind in ("solve2d", "fcg2d"):
        poisson = case.get("op") == "poisson"
        st["b"] = _padded(_poisson_rhs(case, seed) if poisson else _rhs(case, seed), 32)
        st["solver"] = Solver2D(_operator2(case, seed), _solver_conf(case), stream=stream.cuda_stream)
        st["n"] = case["nx"] + 2
    elif kind == "solve3d":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        if case["op"] == "poisson":
            so = torch.from_numpy(gallery.poisson3(nx, ny, nz)).cuda()
            pitch, ns, b = nx + 2, 4, _poisson_rhs(case, seed)
        else:
            k = _coefficients3(case, seed)
            pitch, ns, b = -(-(nx + 2) // 8) * 8, 14, _rhs(case, seed, lo=-1.0)
            so = torch.empty((14, nz + 2, ny + 2, pitch), dtype=F64, device="cuda")
            cur = torch.cuda.current_stream().cuda_stream
            _lib.check(_lib.load().cdr_gpu_fe_assemble_3d_f64(_ptr(k), nx + 1, (nx + 1) * (ny + 1), _ptr(so), nx, ny,
                                                              nz, pitch, ctypes.c_void_p(cur)))
        torch.cuda.synchronize()
        st["solver"] = Solver3D(so.data_ptr(), _solver_conf(case), stream=stream.cuda_stream, dims=(nx, ny, nz),
                                pitch=pitch, nstencil=ns)
        st["b"], st["n"] = _padded(b, 8), nx + 2
    elif kind == "batch2d":
        conf = Config({"solver": {"relaxation": "line-xy", "cycle": {"nrelax-pre": 1, "nrelax-post": 1},
                                  "max-iter": 60, "tol": 1e-8}, "gpu": {"precision": "fp32-ir"}})
        classes, st["b"], st["sizes"] = [], [], []
        for n, nb in _batch_sizes(case):
            pitch = -(-(n + 2) // 16) * 16
            ks, bs = _batch_class(n, nb, seed)
            so = torch.stack([_assemble2(k, k, pitch) for k in ks])
            classes.append((so, n, nb, pitch))
            st["b"].append(_padded(torch.stack(bs), 16))
            st["sizes"].append(n + 2)
        torch.cuda.synchronize()
        st["solver"] = MixedBatchSolver2D([(so.data_ptr(), 5, n, n, pitch, nb) for so, n, nb, pitch in classes], conf,
                                          stream=stream.cuda_stream)
        st["x"] = [torch.zeros_like(b) for b in st["b"]]
    elif kind == "inverse2d":
        th, obs, f = _inverse_inputs(case, seed)
        st["theta"], st["f"] = th.requires_grad_(True), f
        st["uobs"] = solve_log_diffusion_batch(obs, f, tol=1e-10, maxiter=80).detach()
    else:
        so, b, ci, xc = _level_inputs(case, seed)
        nx, ny, ns = case["nx"], case["ny"], case["nstencil"]
        st.update(case=case, so=so, b=b, ci=ci, xc=xc, x=torch.zeros_like(b), r=torch.zeros_like(b),
                  bc=torch.zeros_like(xc), norm=torch.zeros(1, dtype=F64, device="cuda"))
        lib = _lib.load()
        st["scratch"] = torch.zeros(lib.cdr_gpu_norm_scratch_bytes(), dtype=torch.uint8, device="cuda")
        cur = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        if case["relax"] == "point":
            st["sor"] = torch.zeros_like(b)
            _lib.check(lib.cdr_gpu_setup_recip_2d_f64(_ptr(so), _ptr(st["sor"]), nx, ny, nx + 2, cur))
        else:
            st["sorx"] = torch.zeros((2, ny + 2, nx + 2), dtype=F64, device="cuda")
            st["sory"] = torch.zeros((2, nx + 2, ny + 2), dtype=F64, device="cuda")
            for d, s in ((_lib.DIR_X, "sorx"), (_lib.DIR_Y, "sory")):
                _lib.check(lib.cdr_gpu_setup_lines_2d_f64(_ptr(so), ns, _ptr(st[s]), nx, ny, nx + 2, ny + 2, d, None,
                                                          cur))
    if "solver" in st and "x" not in st:
        st["x"] = torch.zeros_like(st["b"])
    torch.cuda.synchronize()
    return st


# --------------------------------------------------------------------- pass
def _run_level(st):
    """Zero guess, one smoothing step, residual and its norm, restriction, interpolate-add of
    the coarse correction, one smoothing step: a cycle's visit to one level."""
    lib, c = _lib.load(), st["case"]
    nx, ny, ns, p = c["nx"], c["ny"], c["nstencil"], c["nx"] + 2
    nxc, nyc, pc = (nx - 1) // 2 + 1, (ny - 1) // 2 + 1, (nx - 1) // 2 + 3
    cur = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def smooth(updown):
        if c["relax"] == "point":
            _lib.check(lib.cdr_gpu_relax_point_2d_f64(_ptr(st["so"]), ns, _ptr(st["x"]), _ptr(st["b"]),
                                                      _ptr(st["sor"]), nx, ny, p, updown, cur))
            return
        order = ((_lib.DIR_X, "sorx"), (_lib.DIR_Y, "sory"))
        for d, s in order if updown == _lib.DOWN else order[::-1]:
            _lib.check(lib.cdr_gpu_relax_lines_2d_f64(_ptr(st["so"]), ns, _ptr(st["x"]), _ptr(st["b"]), _ptr(st[s]),
                                                      nx, ny, p, ny + 2, d, updown, 0, cur))

    st["x"].zero_()
    smooth(_lib.DOWN)
    _lib.check(lib.cdr_gpu_residual_2d_f64(_ptr(st["so"]), ns, _ptr(st["x"]), _ptr(st["b"]), _ptr(st["r"]), nx, ny, p,
                                           _ptr(st["norm"]), _ptr(st["scratch"]), cur))
    _lib.check(lib.cdr_gpu_restrict_2d_f64(_ptr(st["ci"]), _ptr(st["r"]), _ptr(st["bc"]), nx, ny, p, nxc, nyc, pc,
                                           cur))
    _lib.check(lib.cdr_gpu_interp_add_2d_f64(_ptr(st["ci"]), _ptr(st["xc"]), _ptr(st["r"]), _ptr(st["so"]),
                                             _ptr(st["x"]), nx, ny, p, nxc, nyc, pc, cur))
    smooth(_lib.UP)
    # ghosts of x are not part of the result: for even sizes the reference's loop writes there too
    return st["x"][1:-1, 1:-1], st["r"][1:-1, 1:-1], st["bc"][1:-1, 1:-1], st["norm"]


def run(st):
    kind = st["kind"]
    if kind == "host2d":
        return st["solver"].solve(st["b"])
    if kind == "kernels2d":
        return _run_level(st)
    if kind == "inverse2d":
        st["theta"].grad = None
        u = solve_log_diffusion_batch(st["theta"], st["f"], tol=1e-10, maxiter=80)
        loss = 0.5 * ((u - st["uobs"]) ** 2).sum()
        loss.backward()
        return u.detach(), loss.detach(), st["theta"].grad
    stream = st["stream"]
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        if kind == "batch2d":
            for x in st["x"]:
                x.zero_()
            st["solver"].solve_device([b.data_ptr() for b in st["b"]], [x.data_ptr() for x in st["x"]])
            out = [x[:, 1:n - 1, 1:n - 1] for x, n in zip(st["x"], st["sizes"])]
        else:
            st["x"].zero_()
            st["solver"].solve_device(st["b"].data_ptr(), st["x"].data_ptr(), st["b"].shape[-1])
            out = st["x"][tuple([slice(1, -1)] * (st["x"].dim() - 1)) + (slice(1, st["n"] - 1),)]
    torch.cuda.current_stream().wait_stream(stream)
    return out


# --------------------------------------------------------------------- work
# Words a point and cycle that a V(2,1) cycle cannot do without on a level: per
# relaxation sweep the operator, b, x in and out and the smoother's factors;
# residual, restriction and interpolate-add alike.
def _cycle(points, dim, ns, relax, precision, npre_post=3):
    word = 8 if precision == "fp64" else 4
    sweep = {"point": ns + 4, "line-xy": 2 * (ns + 3), "plane-xyz": 3 * (ns + 4 + 2 * 9 + 15)}[relax]
    flop = {"point": 4 * ns, "line-xy": 8 * ns, "plane-xyz": 3 * (4 * ns + 60)}[relax]
    levels = 4.0 / 3 if dim == 2 else 8.0 / 7
    transfer = 3.25 + 6.25
    byts = points * word * levels * (npre_post * sweep + (ns + 3) + transfer)
    outer = points * (8 * (ns + 3) + (12 if precision != "fp64" else 0))
    return byts + outer, points * levels * (npre_post * flop + 4 * ns + 30) + points * 4 * ns


def work(case):
    kind = case["kind"]
    byts = flops = 0.0

    def add(cycles, *a):
        nonlocal byts, flops
        b, f = _cycle(*a)
        byts, flops = byts + cycles * b, flops + cycles * f

    if kind == "host2d":
        add(10, case["nx"] * case["ny"], 2, 3, "point", "fp64")
    elif kind == "solve2d":
        cycles = {"poisson": 12, "hetero": 10, "constant": 11}[case["op"]]
        add(cycles, case["nx"] * case["ny"], 2, 3 if case["op"] == "poisson" else 5, case["relax"],
            case["precision"])
    elif kind == "fcg2d":
        points = case["nx"] * case["ny"]
        cycles = 77 * math.sqrt(points) / 2047
        add(cycles, points, 2, 5, "line-xy", case["precision"], 2)
        byts, flops = byts + cycles * points * 8 * 9, flops + cycles * points * 12
    elif kind == "solve3d":
        cycles = {"poisson": 9, "hetero": 40 if case["relax"] == "point" else 8}[case["op"]]
        add(cycles, case["nx"] * case["ny"] * case["nz"], 3, 4 if case["op"] == "poisson" else 14, case["relax"],
            case["precision"])
    elif kind == "batch2d":
        for n, nb in _batch_sizes(case):
            add(10, nb * n * n, 2, 5, "line-xy", "fp32-ir", 2)
    elif kind == "inverse2d":
        points = case["count"] * case["n"] ** 2
        add(2 * 9, points, 2, 5, "line-xy", "fp32-ir")
        byts, flops = byts + points * 8 * 40, flops + points * 400
    else:
        points, ns = case["nx"] * case["ny"], case["nstencil"]
        per = {"point": ns + 4, "line-xy": 2 * (ns + 3)}[case["relax"]]
        byts, flops = points * 8 * (2 * per + ns + 3 + 9.5), points * (10 * ns + 30)
    return {"bytes": byts, "flops": flops}


def tolerance(case):
    kind = case["kind"]
    # A solve stops at a residual tolerance, so two correct ones may differ by what that leaves in
    # the solution: about four times the largest error against exact() that each kind shows.
    if kind == "host2d":
        return {"rel": 2e-9}
    if kind == "solve2d":
        return {"rel": 1e-9 if case["op"] == "hetero" else 1e-10}
    if kind == "fcg2d":
        return {"rel": 2e-5}
    if kind == "solve3d":
        return {"rel": 1e-9 if case["op"] == "poisson" else 2e-7}
    if kind == "batch2d":
        return {"rel": 3e-9}
    if kind == "inverse2d":
        return {"rel": 1e-7}  # the gradient is FP32
    return {"rel": 1e-14}


# -------------------------------------------------------------------- exact
def _sine(m):
    k = torch.arange(1, m + 1, dtype=F64, device="cuda")
    return torch.sin(math.pi * torch.outer(k, k) / (m + 1)) * math.sqrt(2.0 / (m + 1))


def _along(mat, t, axis):
    return torch.movedim(torch.tensordot(mat, t, dims=([1], [axis])), 0, axis)


def _sine_solve(b, fe):
    """Constant-coefficient solve by sine transforms: the Laplacian with its h^d factors, or
    (fe) the bilinear-element operator on square cells."""
    dims = b.shape
    cosv = [torch.cos(math.pi * torch.arange(1, m + 1, dtype=F64, device="cuda") / (m + 1)) for m in dims]
    view = [c.reshape([-1 if x == a else 1 for x in range(len(dims))]) for a, c in enumerate(cosv)]
    if fe:
        k = [2 - 2 * c for c in view]
        m = [(4 + 2 * c) / 6 for c in view]
        lam = k[0] * m[1] + m[0] * k[1]
    else:
        vol = 1.0
        for n in dims:
            vol /= n + 1
        lam = sum((2 - 2 * c) * vol * (n + 1) ** 2 for c, n in zip(view, dims))
    t = b
    for a, n in enumerate(dims):
        t = _along(_sine(n), t, a)
    t = t / lam
    for a, n in enumerate(dims):
        t = _along(_sine(n), t, a)
    return t


def _neighbours(cells, mats):
    """Couplings of finite elements: {offset: tensor over the nodes, ghosts included} from cell
    coefficients and element matrices (one pair per coefficient); offsets in (.., y, x) order."""
    dim = cells[0].dim()
    corners = [tuple((l >> (dim - 1 - a)) & 1 for a in range(dim)) for l in range(2 ** dim)]
    out = {}
    shape = [m + 1 for m in cells[0].shape]
    for p in corners:
        for q in corners:
            off = tuple(y - x for x, y in zip(p, q))
            arr = out.setdefault(off, torch.zeros(shape, dtype=F64, device="cuda"))
            view = arr[tuple(slice(x, x + m) for x, m in zip(p, cells[0].shape))]
            for k, mat in zip(cells, mats):
                view += k * mat(p, q)
    return out


def _k1(p, q):
    return 1.0 if p == q else -1.0


def _m1(p, q):
    return (2.0 if p == q else 1.0) / 6.0


def _fe2(kx, ky):
    return _neighbours([kx, ky], [lambda p, q: _k1(p[1], q[1]) * _m1(p[0], q[0]),
                                  lambda p, q: _m1(p[1], q[1]) * _k1(p[0], q[0])])


def _fe3(k):
    h = 1.0 / k.shape[-1]

    def mat(p, q):
        tot = 0.0
        for d in range(3):
            t = 1.0
            for a in range(3):
                t *= _k1(p[a], q[a]) if a == d else _m1(p[a], q[a])
            tot += t
        return h * tot
    return _neighbours([k], [mat])


def _tri(band, x):
    """(tridiagonal matrices given as (sub, diag, super) rows) @ x, batched over the first axis."""
    lo, d, up = (t.unsqueeze(-1) for t in band)
    y = d * x
    y[:, 1:] += lo[:, 1:] * x[:, :-1]
    y[:, :-1] += up[:, :-1] * x[:, 1:]
    return y


def _block_solve(ops, rhs):
    """Direct solves of a batch of nine-point operators ({offset: (nb, ny, nx)}): block Cholesky
    elimination along y.  rhs (nb, ny, nx, columns)."""
    nb, ny, nx, _ = rhs.shape
    band = lambda dy, j: tuple(ops[(dy, dx)][:, j] for dx in (-1, 0, 1))
    eye = torch.eye(nx, dtype=F64, device="cuda").expand(nb, nx, nx)
    inv, y = [], []
    for j in range(ny):
        S, r = _tri(band(0, j), eye), rhs[:, j]
        if j:
            low = band(-1, j)
            S = S - _tri(low, _tri(low, inv[-1]).transpose(1, 2)).transpose(1, 2)
            r = r - _tri(low, inv[-1] @ y[-1])
        inv.append(torch.cholesky_inverse(torch.linalg.cholesky(0.5 * (S + S.transpose(1, 2)))))
        y.append(r)
    x = [None] * ny
    for j in range(ny - 1, -1, -1):
        r = y[j] if j == ny - 1 else y[j] - _tri(band(1, j), x[j + 1])
        x[j] = inv[j] @ r
    return torch.stack(x, 1)


def _direct2(kxs, kys, rhs):
    """Solutions of finite-element problems of one size; rhs (nb, ny, nx, columns) on the interior."""
    all_ops = [_fe2(kx, ky) for kx, ky in zip(kxs, kys)]
    ops = {o: torch.stack([a[o][1:-1, 1:-1] for a in all_ops]) for o in all_ops[0]}
    if rhs.shape[2] > rhs.shape[1]:  # eliminate along the longer side
        ops = {(dx, dy): a.transpose(1, 2) for (dy, dx), a in ops.items()}
        return _block_solve(ops, rhs.transpose(1, 2)).transpose(1, 2)
    return _block_solve(ops, rhs)


def _cg3(ops, b):
    """Jacobi-preconditioned CG with ghost-inclusive arrays, to the attainable accuracy."""
    inner = (slice(1, -1),) * 3
    dims = b.shape
    shift = {o: tuple(slice(1 + a, 1 + a + m - 2) for a, m in zip(o, dims)) for o in ops}
    ops = {o: a[inner].contiguous() for o, a in ops.items()}
    d = ops[(0, 0, 0)]

    def mul(v):
        out = d * v[inner]
        for o, a in ops.items():
            if o != (0, 0, 0):
                out.addcmul_(a, v[shift[o]])
        return out
    x, r = torch.zeros_like(b), b[inner].clone()
    p = torch.zeros_like(b)
    z = r / d
    p[inner] = z
    rz = (r * z).sum()
    stop = 1e-13 * float(r.norm())
    for it in range(20000):
        q = mul(p)
        a = rz / (p[inner] * q).sum()
        x[inner] += a * p[inner]
        r -= a * q
        if it % 50 == 49 and float(r.norm()) < stop:
            break
        z = r / d
        rz, old = (r * z).sum(), rz
        p[inner] = z + (rz / old) * p[inner]
    return x[inner]


def _exact_level(case, seed):
    so, b, ci, xc = _level_inputs(case, seed)
    ns = case["nstencil"]
    ny, nx = case["ny"], case["nx"]
    J, I = torch.meshgrid(torch.arange(1, ny + 1, device="cuda"), torch.arange(1, nx + 1, device="cuda"),
                          indexing="ij")
    x = torch.zeros_like(b)
    at = lambda t, dj=0, di=0: t[1 + dj:ny + 1 + dj, 1 + di:nx + 1 + di]
    cx = {(0, -1): at(so[1]), (0, 1): at(so[1], 0, 1), (-1, 0): at(so[2]), (1, 0): at(so[2], 1)}
    if ns == 5:
        cx.update({(-1, -1): at(so[3]), (-1, 1): at(so[4], 0, 1), (1, -1): at(so[4], 1), (1, 1): at(so[3], 1, 1)})

    def offsum(skip=()):
        t = at(b).clone()
        for o, a in cx.items():
            if o not in skip:
                t += a * at(x, *o)
        return t

    def point(down):
        if ns == 5:
            masks = [(J % 2 == a) & (I % 2 == c) for a, c in ((1, 1), (1, 0), (0, 1), (0, 0))]
        else:
            masks = [(I + J) % 2 == a for a in (0, 1)]
        for m in masks if down else masks[::-1]:
            at(x).copy_(torch.where(m, offsum() / at(so[0]), at(x)))

    def lines(dirx, down):
        diag, off = at(so[0]), at(so[1] if dirx else so[2])
        if not dirx:
            diag, off = diag.T, off.T
        m = diag.shape[1]
        for par in ((0, 1) if down else (1, 0)):
            r = offsum(((0, -1), (0, 1)) if dirx else ((-1, 0), (1, 0)))
            r = (r if dirx else r.T).clone()
            d = diag.clone()
            for i in range(1, m):
                e = off[:, i] / d[:, i - 1]
                d[:, i] -= e * off[:, i]
                r[:, i] += e * r[:, i - 1]
            r[:, m - 1] /= d[:, m - 1]
            for i in range(m - 2, -1, -1):
                r[:, i] = (r[:, i] + off[:, i + 1] * r[:, i + 1]) / d[:, i]
            sol = r if dirx else r.T
            at(x).copy_(torch.where((J if dirx else I) % 2 == par, sol, at(x)))

    def smooth(down):
        if case["relax"] == "point":
            point(down)
        else:
            for dirx in ((True, False) if down else (False, True)):
                lines(dirx, down)

    smooth(True)
    r = torch.zeros((2 * (xc.shape[0]) + 2, 2 * xc.shape[1] + 2), dtype=F64, device="cuda")
    r[1:ny + 1, 1:nx + 1] = offsum() - at(so[0]) * at(x)
    L, R, A, B, SW, NW, NE, SE = ci
    nyc, nxc = xc.shape[0] - 2, xc.shape[1] - 2
    fine = lambda dj, di: r[1 + dj:1 + dj + 2 * nyc:2, 1 + di:1 + di + 2 * nxc:2]
    co = lambda t, dj=0, di=0: t[1 + dj:nyc + 1 + dj, 1 + di:nxc + 1 + di]
    bc = (co(NE) * fine(-1, -1) + co(A) * fine(-1, 0) + co(NW, 0, 1) * fine(-1, 1) + co(R) * fine(0, -1) + fine(0, 0)
          + co(L, 0, 1) * fine(0, 1) + co(SE, 1) * fine(1, -1) + co(B, 1) * fine(1, 0) + co(SW, 1, 1) * fine(1, 1))
    # x += P xc + r/c: cells (jc, ic) from 1, fine (2 jc - 1, 2 ic - 1); one more row for even sizes
    xw = torch.zeros_like(r)
    xw[1:ny + 1, 1:nx + 1] = at(x)
    e = torch.zeros_like(r)
    s0 = lambda t: t[1:, 1:]
    q, qw, qs, qsw = xc[1:, 1:], xc[1:, :-1], xc[:-1, 1:], xc[:-1, :-1]
    my, mx = q.shape
    e[1:1 + 2 * my:2, 1:1 + 2 * mx:2] = q
    e[1:1 + 2 * my:2, 0:2 * mx:2] = s0(L) * qw + s0(R) * q
    e[0:2 * my:2, 1:1 + 2 * mx:2] = s0(B) * qs + s0(A) * q
    e[0:2 * my:2, 0:2 * mx:2] = s0(SW) * qsw + s0(NW) * qw + s0(NE) * q + s0(SE) * qs
    corr = torch.zeros_like(r)
    corr[1:ny + 1, 1:nx + 1] = r[1:ny + 1, 1:nx + 1] / at(so[0])
    corr[1::2, 1::2] = 0.0  # coarse points take the correction alone
    x[1:ny + 1, 1:nx + 1] = (xw + e + corr)[1:ny + 1, 1:nx + 1]
    smooth(False)
    rr = r[1:ny + 1, 1:nx + 1]
    return at(x).clone(), rr, bc, rr.norm().reshape(1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "host2d" or (kind in ("solve2d", "solve3d") and case["op"] == "poisson"):
        b = _poisson_rhs(case, seed)
        sol = _sine_solve(b[(slice(1, -1),) * b.dim()], False)
        if kind == "host2d":
            full = torch.zeros_like(b)
            full[1:-1, 1:-1] = sol
            return full.cpu().numpy()
        return sol
    if kind == "solve2d" and case["op"] == "constant":
        return _sine_solve(_rhs(case, seed)[1:-1, 1:-1], True)
    if kind in ("solve2d", "fcg2d"):
        short, tall = sorted((case["nx"], case["ny"]))
        if short > 1000:
            return None  # the elimination takes too long
        kx, ky = _coefficients2(case, seed)
        return _direct2([kx], [ky], _rhs(case, seed)[None, 1:-1, 1:-1, None])[0, :, :, 0].contiguous()
    if kind == "solve3d":
        if case["nx"] * case["ny"] * case["nz"] > 4e6:
            return None  # too many CG iterations
        return _cg3(_fe3(_coefficients3(case, seed)), _rhs(case, seed, lo=-1.0))
    if kind == "batch2d":
        out = []
        for n, nb in _batch_sizes(case):
            if n > 255:
                out.append(None)  # the eliminations take too long
                continue
            ks, bs = _batch_class(n, nb, seed)
            sols = []
            for p in range(0, nb, 32):
                rhs = torch.stack(bs[p:p + 32])[:, 1:-1, 1:-1, None]
                sols.append(_direct2(ks[p:p + 32], ks[p:p + 32], rhs)[..., 0])
            out.append(torch.cat(sols))
        return out
    if kind == "inverse2d":
        if case["n"] > 300:
            return None  # the eliminations take too long
        th, obs, f = _inverse_inputs(case, seed)
        fi = f[:, 1:-1, 1:-1, None]
        k, ko = torch.exp(th.to(F64)), torch.exp(obs)
        u = torch.zeros_like(f)
        u[:, 1:-1, 1:-1] = _direct2(k, k, fi)[..., 0]
        uo = torch.zeros_like(f)
        uo[:, 1:-1, 1:-1] = _direct2(ko, ko, fi)[..., 0]
        lam = torch.zeros_like(f)
        lam[:, 1:-1, 1:-1] = _direct2(k, k, (u - uo)[:, 1:-1, 1:-1, None])[..., 0]
        grad = torch.zeros_like(k)
        m = k.shape[1]
        corners = [(a, c) for a in (0, 1) for c in (0, 1)]
        for p in corners:
            for q in corners:
                e = _k1(p[1], q[1]) * _m1(p[0], q[0]) + _m1(p[1], q[1]) * _k1(p[0], q[0])
                grad -= e * lam[:, p[0]:p[0] + m, p[1]:p[1] + m] * u[:, q[0]:q[0] + m, q[1]:q[1] + m]
        return u, 0.5 * ((u - uo) ** 2).sum(), (grad * k).to(torch.float32)
    return _exact_level(case, seed)
