"""End-to-end parity of the GPU BoxMG solver with the reference's golden output and
the CPU oracle.  Bar (from the hot-path specification): the plain FP64 path
reproduces the per-iteration relative residual history within 1e-12 and the
solution within 1e-10 relative; the FP32-cycle + FP64-refinement path reaches
the same tolerance and reports its error against the FP64 oracle."""
import json
import os

import numpy as np
import pytest

from cedar_b200 import gallery as G
from cedar_b200 import problems as P
from cedar_b200.config import Config
from tests.golden.make_fixtures import build_case

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), "golden")
HIST_TOL = 1e-12


def gpu_solver(so, relax, **kw):
    from cedar_b200.solver import Solver2D
    conf = {"solver": {"relaxation": relax, "cycle": {"nrelax-pre": kw.get("nrelax_pre", 2),
                                                      "nrelax-post": kw.get("nrelax_post", 1)},
                       "max-iter": kw.get("maxiter", 10), "tol": kw.get("tol", 1e-8),
                       "num-levels": kw.get("num_levels", -1)},
            "gpu": {"precision": kw.get("precision", "fp64"), "graph": kw.get("graph", True),
                    "line-solve": kw.get("line_solve", "sequential")}}
    return Solver2D(so, Config(conf))


def assert_history(h_gpu, h_ref):
    assert len(h_gpu) == len(h_ref)
    d = np.abs(np.asarray(h_gpu) - np.asarray(h_ref))
    assert (d <= HIST_TOL * np.maximum(1.0, np.abs(h_ref))).all(), (h_gpu, h_ref)


def rel(x, y):
    return np.linalg.norm((x - y).ravel()) / np.linalg.norm(y.ravel())


@pytest.mark.parametrize("graph", [True, False])
def test_readme_golden_history(oracle, graph):
    g = json.load(open(os.path.join(GOLD, "readme_poisson400.json")))
    so = G.poisson(400, 400)
    b = G.poisson_rhs_sin2pi(400, 400)
    s = gpu_solver(so, "point", nrelax_pre=1, nrelax_post=1, maxiter=10, tol=1e-10, num_levels=7, graph=graph)
    x = s.solve(b)
    assert [float("%.6g" % v) for v in s.history] == g["history"]
    err = oracle.inf_norm(np.ascontiguousarray(G.poisson_exact_sin2pi(400, 400) - x))
    assert float("%.6g" % abs(err)) == g["solution_norm_abs"]
    o = oracle.Solver(so, relax="point", nrelax_pre=1, nrelax_post=1, maxiter=10, tol=1e-10, num_levels=7)
    xo, ho = o.solve(b)
    assert_history(s.history, ho)
    assert rel(x, xo) < 1e-10


def test_fixture_histories(oracle):
    fx = json.load(open(os.path.join(GOLD, "oracle_histories.json")))
    for case in fx["cases"]:
        so, b, kw = build_case(case)
        s = gpu_solver(so, kw["relax"], nrelax_pre=kw["nrelax_pre"], nrelax_post=kw["nrelax_post"],
                       maxiter=kw["maxiter"], tol=kw["tol"])
        x = s.solve(b)
        assert_history(s.history, case["history"])
        o = oracle.Solver(so, **kw)
        xo, ho = o.solve(b)
        assert rel(x, xo) < 1e-10, case["name"]


@pytest.mark.parametrize("n,relax", [(511, "point"), (255, "line-xy"), (200, "line-xy")])
def test_larger_parity(oracle, n, relax):
    if relax == "point":
        so, b = P.poisson_noise(n)
        kw = dict(nrelax_pre=2, nrelax_post=1, maxiter=15, tol=1e-10)
    else:
        so, b = P.hetero_diffusion(n)
        kw = dict(nrelax_pre=2, nrelax_post=1, maxiter=6, tol=1e-10)
    s = gpu_solver(so, relax, **kw)
    x = s.solve(b)
    o = oracle.Solver(so, relax=relax, **kw)
    xo, ho = o.solve(b)
    assert_history(s.history, ho)
    assert rel(x, xo) < 1e-10


@pytest.mark.parametrize("n", [127, 200])
def test_scan_line_solve_within_rounding_envelope(oracle, n):
    """The parallel-scan line substitutions change only rounding: on the ill-conditioned
    heterogeneous problem (coefficient contrast ~1e11) the history stays within the
    spread between two FP64 builds of the oracle itself (with and without FMA)."""
    so, b = P.hetero_diffusion(n)
    kw = dict(nrelax_pre=2, nrelax_post=1, maxiter=6, tol=1e-10)
    s = gpu_solver(so, "line-xy", line_solve="scan", **kw)
    s.solve(b)
    xo, ho = oracle.Solver(so, relax="line-xy", **kw).solve(b)
    xf, hf = oracle.Solver(so, relax="line-xy", variant="fma", **kw).solve(b)
    envelope = max(np.abs(hf - ho).max(), 1e-12 * max(1.0, ho.max()))
    assert np.abs(s.history - ho).max() <= 10 * envelope, (s.history - ho, hf - ho)


@pytest.mark.parametrize("n", [127, 256])
def test_fp32_ir_reaches_tolerance(oracle, n):
    so, b = P.hetero_diffusion(n, sigma=1.0, n_incl=0, aniso=1.0)
    s64 = gpu_solver(so, "line-xy", maxiter=30, tol=1e-10)
    x64 = s64.solve(b)
    s32 = gpu_solver(so, "line-xy", maxiter=30, tol=1e-10, precision="fp32-ir")
    x32 = s32.solve(b)
    assert s32.history[-1] < 1e-10
    assert s32.iters <= s64.iters + 2
    o = oracle.Solver(so, relax="line-xy", maxiter=30, tol=1e-10)
    xo, ho = o.solve(b)
    assert rel(x64, xo) < 1e-10
    # FP32 preconditioner, FP64 residual: the error against the FP64 oracle is at the tolerance level
    assert rel(x32, xo) < 1e-8


def test_device_buffers_match_host(oracle):
    import torch
    so, b = P.poisson_noise(127)
    s = gpu_solver(so, "point", maxiter=8, tol=1e-12)
    xh = s.solve(b)
    pitch = 160
    bd = torch.zeros((129, pitch), dtype=torch.float64, device="cuda")
    bd[:, :129] = torch.from_numpy(b).cuda()
    xd = torch.zeros_like(bd)
    s.solve_device(bd.data_ptr(), xd.data_ptr(), pitch)
    np.testing.assert_array_equal(xd[:, :129].cpu().numpy(), xh)
    # one vcycle from zero equals the oracle's vcycle
    xv = torch.zeros_like(bd)
    s.vcycle_device(bd.data_ptr(), xv.data_ptr(), pitch)
    o = oracle.Solver(so, relax="point", maxiter=8, tol=1e-12)
    xo = np.zeros_like(b)
    o.vcycle(xo, b)
    assert rel(xv[:, :129].cpu().numpy(), xo) < 1e-13


def test_setup_arrays_match_oracle(oracle):
    """Interpolation weights and Galerkin operators of every level: same bits as the oracle."""
    so, b = P.hetero_diffusion(65)
    s = gpu_solver(so, "line-xy", maxiter=2)
    o = oracle.Solver(so, relax="line-xy", maxiter=2)
    for l in range(1, s.nlevels):
        np.testing.assert_array_equal(s.level_array(l, "ci"), o.level_array(l, "ci"))
        np.testing.assert_array_equal(s.level_array(l, "so"), o.level_array(l, "so"))


@pytest.mark.parametrize("relax,ns,n", [("line-xy", 5, 255), ("point", 3, 200), ("line-x", 5, 130), ("point", 5, 97)])
def test_fused_coarse_cycle_is_bitwise_the_separate_kernels(relax, ns, n):
    """The fused coarse cycle (levels of at most 64x64 in one launch) performs the
    operations of the separate kernels in sequential-substitution mode: the FP64
    solve is bit-identical with and without it."""
    from cedar_b200.config import Config
    from cedar_b200.solver import Solver2D
    if ns == 5:
        so, b = P.hetero_diffusion(n, sigma=1.0, n_incl=4, contrast=100.0, aniso=0.5)
    else:
        so, b = P.poisson_noise(n)
    xs, hs = [], []
    for fuse in (64, 0):
        conf = Config({"solver": {"relaxation": relax, "max-iter": 8, "tol": 1e-14},
                       "gpu": {"line-solve": "sequential", "fuse-coarse": fuse}})
        s = Solver2D(so, conf)
        xs.append(s.solve(b))
        hs.append(s.history.copy())
    assert np.array_equal(xs[0], xs[1])
    assert np.array_equal(hs[0], hs[1])


def test_fused_coarse_cycle_fp32():
    from cedar_b200.config import Config
    from cedar_b200.solver import Solver2D
    so, b = P.hetero_diffusion(255, sigma=1.0, n_incl=4, contrast=100.0, aniso=0.5)
    its = []
    for fuse in (64, 0):
        s = Solver2D(so, Config({"solver": {"relaxation": "line-xy", "max-iter": 30, "tol": 1e-10},
                                 "gpu": {"precision": "fp32-ir", "fuse-coarse": fuse}}))
        s.solve(b)
        assert s.history[-1] < 1e-10
        its.append(s.iters)
    assert abs(its[0] - its[1]) <= 1


@pytest.mark.parametrize("nx,ny", [(61, 63), (63, 64), (65, 66), (94, 51), (127, 30)])
@pytest.mark.parametrize("levels", [-1, 2])
def test_fused_coarse_cycle_line_edges(nx, ny, levels):
    """Fused levels whose lines end around a warp's 32 positions, and coarsest levels whose band is
    wider than a warp (two levels): FP64 bits of the separate kernels, FP32 to the tolerance in as
    many cycles."""
    from cedar_b200 import gallery as G
    from cedar_b200.config import Config
    from cedar_b200.solver import Solver2D
    rng = np.random.default_rng(nx + ny)
    k = np.exp(rng.standard_normal((ny + 1, nx + 1)))
    so = G.fe_hetero(k, k)
    b = np.zeros((ny + 2, nx + 2))
    b[1:-1, 1:-1] = rng.uniform(0, 1, size=(ny, nx))
    out = {}
    for fuse in (64, 0):
        for prec in ("fp64", "fp32-ir"):
            s = Solver2D(so, Config({"solver": {"relaxation": "line-xy", "max-iter": 30, "tol": 1e-9,
                                                "num-levels": levels},
                                     "gpu": {"precision": prec, "line-solve": "sequential", "fuse-coarse": fuse}}))
            out[fuse, prec] = s.solve(b), s.history.copy()
    assert np.array_equal(out[64, "fp64"][0], out[0, "fp64"][0])
    assert np.array_equal(out[64, "fp64"][1], out[0, "fp64"][1])
    assert out[64, "fp32-ir"][1][-1] < 1e-9
    assert abs(len(out[64, "fp32-ir"][1]) - len(out[0, "fp32-ir"][1])) <= 1


@pytest.mark.parametrize("relax,ns", [("line-xy", 5), ("point", 3)])
def test_fcycle_fp64_matches_oracle(oracle, relax, ns):
    """solver.cycle.type = "f" (cycle::fcycle): with the sequential line
    substitutions every operation follows the oracle's F-cycle, so the
    iterates are identical; like the reference, every iteration restarts the
    F-cycle from zero and gives the same x."""
    from cedar_b200.solver import Solver2D
    from cedar_b200 import gallery as G
    n = 63
    if ns == 5:
        so, b = P.hetero_diffusion(n, sigma=1.0, n_incl=4, contrast=100.0, aniso=0.5)
    else:
        so = G.diag_diffusion(n, n, 1.0, 0.5)
        b = np.zeros((n + 2, n + 2))
        b[1:-1, 1:-1] = np.random.default_rng(3).random((n, n)) / (n + 1) ** 2
    conf = Config({"solver": {"relaxation": relax, "max-iter": 3, "tol": 0.0, "cycle": {"type": "f"}},
                   "gpu": {"line-solve": "sequential"}})
    s = Solver2D(so, conf)
    x = s.solve(b)
    x_ref, h_ref = oracle.Solver(np.ascontiguousarray(so), relax=relax, maxiter=3, tol=0.0, cycle="f").solve(b)
    assert np.array_equal(x, x_ref)
    assert np.abs(s.history - h_ref).max() <= 1e-12 * h_ref.max()


def test_fcycle_fp32_ir_converges_in_fewer_cycles():
    """The F-cycle (FP32 cycle, FP64 refinement) on a heterogeneous problem:
    converges, in no more cycles than the V-cycle (each F-cycle also visits
    the coarse levels first).  Default launch shapes, so the run is fixed."""
    from cedar_b200.solver import Solver2D
    so, b = P.hetero_diffusion(255, sigma=1.0, n_incl=4, contrast=100.0, aniso=0.5)
    its = {}
    for cyc in ("v", "f"):
        s = Solver2D(so, Config({"solver": {"relaxation": "line-xy", "max-iter": 60, "tol": 1e-8,
                                            "cycle": {"type": cyc}},
                                 "gpu": {"precision": "fp32-ir", "autotune": False}}))
        s.solve(b)
        assert s.history[-1] < 1e-8, cyc
        its[cyc] = s.iters
    assert its["f"] <= its["v"]


def test_line_tuner_on_a_stream_that_cannot_be_captured():
    """Without graphs a solver on the legacy default stream's handle, which refuses captures, is set up
    with tuned line kernels and solves as on a stream of its own.  The launch counter takes the
    tuner's launches as they run: three times two sweeps per candidate."""
    from cedar_b200 import _lib
    from cedar_b200.solver import Solver2D
    lib = _lib.load()
    legacy = 1  # cudaStreamLegacy
    out = []
    for stream, nx in ((legacy, 203), (0, 203), (legacy, 205)):
        so, b = P.hetero_diffusion(nx, sigma=1.0, n_incl=4, contrast=100.0, aniso=0.5)
        counts = []
        for tune in (True, False):
            conf = Config({"solver": {"relaxation": "line-xy", "max-iter": 5, "tol": 1e-14},
                           "gpu": {"graph": False, "autotune": tune}})
            before = lib.cdr_gpu_launch_count()
            s = Solver2D(so, conf, stream=stream)
            counts.append(lib.cdr_gpu_launch_count() - before)
            out.append((nx, s.solve(b), s.history.copy()))
        assert (counts[0] - counts[1]) % 6 == 0
        assert counts[0] > counts[1] or (stream, nx) == (0, 203)  # shapes are tuned once per process
    for nx, x, h in out[1:]:
        if nx == 203:
            assert np.array_equal(x, out[0][1]) and np.array_equal(h, out[0][2])
