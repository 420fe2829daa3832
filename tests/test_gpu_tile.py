"""Kernels with several elements per warp.  FP64 (spoc_tile.cu) against the
CPU oracle, bit for bit: every tabulated degree and variant on a mesh
large enough for them whose element and face counts are not multiples of a
tile, and an odd element count
at an odd mode count (fields aligned to 8 bytes only).  Mixed precision
(spoc_mixed_tile.cu) against the one-element-per-warp kernels, which sum every
chain in the same order: also bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O
from spoc_b200 import api
from spoc_b200 import workloads as W

RULES = {3: (12, 4), 4: (25, 5), 5: (27, 6), 6: (33, 7), 7: (42, 9)}


def problem(nc, variant, n, odd=False):
    """A problem with random state and wind; odd: one wall element refined, so
    that the mesh has an odd number of elements."""
    ng, ngf = RULES[nc]
    cfg = W.Config("tile", variant, nc, ng, ngf, n, jitter=0.2, beta=2.0e-11, mu0=100.0, mb0=1.0e-3,
                   seed=nc, ic="gauss8")
    p = W.build_problem(cfg)
    if odd:
        wall = int(np.nonzero(p.mesh.bdl)[0][p.mesh.bdl.sum() // 2])
        inn, x, y = W.refine(p.mesh.inn - 1, p.mesh.xgr, p.mesh.ygr, np.arange(p.mesh.ne) == wall)
        inn = api.fix_mesh(inn + 1, x.size)
        p.mesh = api.build_mesh(inn, x, y, nc, cfg.f0, cfg.beta)
    rng = np.random.default_rng(100 * nc + n)
    shape = (p.mesh.ne, p.T.nm)
    p.u, p.v, p.h = (rng.normal(size=shape) for _ in range(3))
    p.w0, p.z0 = (1.0e-4 * rng.normal(size=shape) for _ in range(2))
    p.hb = np.zeros(shape)
    p.hb[:, 0] = cfg.depth
    p.hb += rng.normal(size=shape)
    p.fc = p.mesh.fc
    return p


def check(p):
    c, T, m = p.cfg, p.T, p.mesh
    OT = O.Tables(c.nc, c.ng, c.ngf, T.wi, T.xi, T.yi, T.wif, T.tif)
    OM = O.Mesh(m.inn, m.xgr, m.ygr, c.nc, c.f0, c.beta)
    s = W.make_solver(p)
    got = s.cal_var(p.u, p.v, p.h)
    ref = O.cal_var(c.variant, OT, OM, p.u, p.v, p.h, OM.fc, p.w0, p.z0, p.hb, c.mu0, c.mb0, c.g0)
    for g, r in zip(got, ref):
        assert np.array_equal(g, r), f"right-hand side: max |d| = {np.abs(g - r).max():.3e}"
    dt = 1.0e-3
    s.set_state(p.u, p.v, p.h)
    s.rk4_steps(dt, 2)
    u, v, h = p.u.copy(), p.v.copy(), p.h.copy()
    O.rk4(c.variant, OT, OM, u, v, h, OM.fc, p.w0, p.z0, p.hb, c.mu0, c.mb0, c.g0, dt, 2)
    for g, r in zip(s.get_state(), (u, v, h)):
        assert np.array_equal(g, r), f"two steps: max |d| = {np.abs(g - r).max():.3e}"


@pytest.mark.gpu
@pytest.mark.parametrize("variant", ["lin", "fs", "ns", "inv"])
@pytest.mark.parametrize("nc", sorted(RULES))
def test_ragged_mesh_bitwise(gpu_lib, nc, variant):
    # linear runs of up to 20 elements per SM take the multi-step kernel
    p = problem(nc, variant, 41 if variant == "lin" else 37)
    assert p.mesh.ne % 4 and p.mesh.nf % 16
    check(p)


@pytest.mark.gpu
@pytest.mark.parametrize("nc,n", [(4, 35), (5, 37)])
def test_odd_element_count_bitwise(gpu_lib, nc, n):
    p = problem(nc, "fs", n, odd=True)
    assert p.mesh.ne % 2 == 1
    check(p)


@pytest.mark.gpu
@pytest.mark.parametrize("variant", ["fs", "ns", "inv"])
@pytest.mark.parametrize("nc,n", [(3, 2), (3, 34), (4, 13), (5, 9), (5, 25), (6, 2), (6, 24), (6, 34)])
def test_small_mesh_one_launch_bitwise(gpu_lib, nc, n, variant):
    """Small meshes: all steps of a call in one cooperative launch, with one
    warp per block, the most of either instance, and idle warps."""
    check(problem(nc, variant, n))


@pytest.mark.gpu
@pytest.mark.parametrize("variant", ["fs", "ns", "inv"])
@pytest.mark.parametrize("nc", sorted(RULES))
def test_mixed_ragged_mesh_matches_one_element_kernels(gpu_lib, nc, variant):
    p = problem(nc, variant, 41)
    assert p.mesh.ne % 4 == 2
    p.u, p.v, p.h = 0.1 * p.u, 0.1 * p.v, 0.1 * p.h
    out = []
    for path in ("auto", "generic"):
        s = W.make_solver(p, "mixed")
        s.set_kernel_path(path)
        rhs = s.cal_var(p.u, p.v, p.h)
        s.set_state(p.u, p.v, p.h)
        s.rk4_steps(1.0e-3, 2)
        out.append([*rhs, *s.get_state()])
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("variant", ["fs", "ns", "inv"])
@pytest.mark.parametrize("nc", sorted(RULES))
def test_adjoint_ragged_mesh_matches_one_element_kernels(gpu_lib, nc, variant):
    """Adjoint right-hand side and steps (spoc_adjoint_tile.cu) against
    spoc_adjoint.cu, which sums in the same order: bit for bit."""
    p = problem(nc, variant, 37)
    x = [0.1 * f for f in (p.u, p.v, p.h)]
    b = [np.random.default_rng(nc).normal(size=p.u.shape) for _ in range(3)]
    out = []
    for path in ("auto", "generic"):
        s = W.make_solver(p)
        s.set_kernel_path(path)
        out.append([*s.adj_rhs(x, b), *s.adj_steps(x, b, 1.0e-3, 2)])
    for g, r in zip(*out):
        assert np.isfinite(g).all() and np.array_equal(g, r), f"max |d| = {np.abs(g - r).max():.3e}"


@pytest.mark.gpu
@pytest.mark.parametrize("weight", [0, 3])
def test_ensemble_blocks_help_other_members(gpu_lib, weight):
    """One block per SM for members whose tiles exceed a first round, dealt so
    that some members' blocks finish early and take other members' tiles."""
    ps = [problem(nc, "fs", n) for nc, n in ((3, 50), (6, 41), (4, 13), (5, 60))]
    alone, mem = [], []
    for p in ps:
        p.u, p.v, p.h = 0.1 * p.u, 0.1 * p.v, 0.1 * p.h
        for out in (alone, mem):
            out.append(W.make_solver(p, "mixed"))
            out[-1].set_state(p.u, p.v, p.h)
    for s in alone:
        s.rk4_steps(1.0e-3, 3)
    ens = api.Ensemble(mem)
    ens.configure(1, weight)
    ens.steps([1.0e-3] * len(ps), 3)
    for a, b in zip(alone, mem):
        for x, y in zip(a.get_state(), b.get_state()):
            assert np.isfinite(x).all() and np.array_equal(x, y)
