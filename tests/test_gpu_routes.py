"""The kernels behind one call differ with the mesh's size, the entry point and
the stream; these tests take the routes that the tests of the entry points on
small meshes leave out.

  per stage     one launch per kernel and stage (spoc_profile_rk4), which a run
                on a small mesh does in one launch
  step graph    host-array runs long enough to replay it, with other step sizes
                between, pinned and pageable, packed and strided
  fused         the FMA form of the several-element kernels
  non-finite    reported by the several-element kernels, the handle usable after
  chained       the linear mixed kernel launched behind the one before it
  ensemble      both kernels of small ensembles
"""
import numpy as np
import pytest

from oracle import oracle as O
from spoc_b200 import api
from spoc_b200 import workloads as W
from test_gpu_parity import oracle_for, rel_mass_diff
from test_gpu_tile import RULES, problem

VARIANTS = ["lin", "fs", "ns", "inv"]


def oracle_steps(p, OM, OT, dt, n):
    c = p.cfg
    x = [p.u.copy(), p.v.copy(), p.h.copy()]
    O.rk4(c.variant, OT, OM, *x, OM.fc, p.w0, p.z0, p.hb, c.mu0, c.mb0, c.g0, dt, n)
    return x


@pytest.mark.gpu
@pytest.mark.parametrize("variant", VARIANTS)
@pytest.mark.parametrize("nc,n", [(3, 5), (4, 6), (5, 5), (6, 5), (6, 34), (7, 5)])
def test_per_stage_kernels_of_small_meshes_bitwise(gpu_lib, nc, n, variant):
    p = problem(nc, variant, n)
    OT, OM = oracle_for(p)
    s = W.make_solver(p)
    s.set_state(p.u, p.v, p.h)
    s.profile_rk4(1.0e-3, 2)
    for g, r in zip(s.get_state(), oracle_steps(p, OM, OT, 1.0e-3, 2)):
        assert np.array_equal(g, r), f"max |d| = {np.abs(g - r).max():.3e}"


@pytest.mark.gpu
@pytest.mark.parametrize("stream", [0, 1], ids=["own", "legacy"])
@pytest.mark.parametrize("pinned", [False, True], ids=["pageable", "pinned"])
@pytest.mark.parametrize("strided", [False, True], ids=["packed", "strided"])
@pytest.mark.parametrize("nc,variant,n,precision", [(4, "fs", 37, "fp64"), (5, "lin", 61, "fp64"),
                                                    (7, "ns", 37, "fp64"), (3, "inv", 41, "fp64_fma")])
def test_host_runs_match_resident_runs(gpu_lib, nc, variant, n, precision, strided, pinned, stream):
    """Runs of 8 steps and more replay the step graph between their first and last
    step; the shorter ones and another step size do not disturb it."""
    import torch
    p = problem(nc, variant, n)
    nm, ld = p.T.nm, 45 if strided else p.T.nm
    x = []
    for f in (p.u, p.v, p.h):
        a = torch.full((p.mesh.ne, ld), 7.0, dtype=torch.float64)
        a = a.pin_memory() if pinned else a
        a.numpy()[:, :nm] = f
        x.append(a.numpy())
    s, ref = W.make_solver(p, precision), W.make_solver(p, precision)
    if stream:
        s.set_stream(stream)
    ref.set_state(p.u, p.v, p.h)
    for dt, steps in ((1.0e-3, 9), (1.0e-3, 3), (2.0e-3, 4), (1.0e-3, 8), (3.0e-3, 10), (3.0e-3, 1)):
        s.rk4_steps_host(*x, dt, steps)
        ref.rk4_steps(dt, steps)
        for a, b, c in zip(x, ref.get_state(), s.get_state()):
            assert np.array_equal(a[:, :nm], b) and np.array_equal(b, c), (dt, steps)
            assert (a[:, nm:] == 7.0).all()
    if stream:
        s.set_stream(0)


@pytest.mark.gpu
@pytest.mark.parametrize("variant", VARIANTS)
@pytest.mark.parametrize("nc", sorted(RULES))
def test_fused_several_element_kernels_within_tolerance(gpu_lib, nc, variant):
    """The bounds of the small meshes' test: the mass solves amplify the one-ulp
    differences of the loads by up to 8e4 (degree 7)."""
    p = problem(nc, variant, 41 if variant == "lin" else 37)
    OT, OM = oracle_for(p)
    c = p.cfg
    s = W.make_solver(p, "fp64_fma")
    ref = O.cal_var(c.variant, OT, OM, p.u, p.v, p.h, OM.fc, p.w0, p.z0, p.hb, c.mu0, c.mb0, c.g0)
    assert rel_mass_diff(OT, OM, s.cal_var(p.u, p.v, p.h), ref) < 1e-8
    s.set_state(p.u, p.v, p.h)
    s.rk4_steps(1.0e-3, 1)
    assert rel_mass_diff(OT, OM, s.get_state(), oracle_steps(p, OM, OT, 1.0e-3, 1)) < 1e-11


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("precision", ["fp64", "fp64_fma", "mixed"])
@pytest.mark.parametrize("nc,variant,n", [(3, "ns", 37), (4, "fs", 37), (5, "lin", 61), (7, "inv", 37)])
def test_non_finite_state_is_reported_on_large_meshes(gpu_lib, nc, variant, n, precision, bad):
    p = problem(nc, variant, n)
    x = [0.1 * f for f in (p.u, p.v, p.h)]
    s = W.make_solver(p, precision)
    good = s.cal_var(*x)
    for e in (0, p.mesh.ne // 2, p.mesh.ne - 1):
        y = [a.copy() for a in x]
        y[e % 3][e, p.T.nm - 1] = bad
        with pytest.raises(api.SpocError) as ei:
            s.cal_var(*y)
        assert ei.value.code == 3
        s.set_state(*y)
        with pytest.raises(api.SpocError) as ei:
            s.rk4_steps(1.0e-3, 2)
        assert ei.value.code == 3
    for a, b in zip(s.cal_var(*x), good):
        assert np.isfinite(a).all() and np.array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("nc,n", [(3, 9), (3, 41), (4, 9), (5, 13), (6, 20), (6, 25), (7, 9), (7, 25)])
def test_chained_mixed_linear_steps_match_single_launches(gpu_lib, nc, n):
    p = problem(nc, "lin", n)
    x = [0.1 * f for f in (p.u, p.v, p.h)]
    s, ref = W.make_solver(p, "mixed"), W.make_solver(p, "mixed")
    for h in (s, ref):
        h.set_state(*x)
    s.rk4_steps(1.0e-3, 3)
    ref.profile_rk4(1.0e-3, 3)  # timed between its launches
    for a, b in zip(s.get_state(), ref.get_state()):
        assert np.isfinite(a).all() and np.array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("layout", [(4, 2), (4, 0), (1, 3)])
@pytest.mark.parametrize("members", [[(5, 4), (6, 5)], [(3, 4), (5, 6), (6, 9)], [(3, 4), (3, 7)], [(4, 4), (3, 4)],
                                     [(3, 24), (4, 24), (5, 24), (6, 24)], [(6, 30), (3, 5)]])
def test_small_ensembles_match_members_run_alone(gpu_lib, members, layout):
    """Either ensemble kernel, a pass of its blocks or several."""
    ps = [problem(nc, "fs", n) for nc, n in members]
    alone, mem = [], []
    for p in ps:
        for out in (alone, mem):
            out.append(W.make_solver(p, "mixed"))
            out[-1].set_state(0.1 * p.u, 0.1 * p.v, 0.1 * p.h)
    for s in alone:
        s.rk4_steps(1.0e-3, 5)
    ens = api.Ensemble(mem)
    ens.configure(*layout)
    ens.steps([1.0e-3] * len(ps), 2, graph=False)
    ens.steps([1.0e-3] * len(ps), 3)
    for a, b in zip(alone, mem):
        for x, y in zip(a.get_state(), b.get_state()):
            assert np.isfinite(x).all() and np.array_equal(x, y)
