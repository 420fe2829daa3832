"""Host side of the library on a stand-in for the CUDA runtime (fake_cudart.cpp):
what it allocates, captures, launches and clears, and what it does when a call
fails.  Kernels do nothing there, so no values are looked at."""
import os
import subprocess
import sys
import textwrap
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
CUDA = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))

PRELUDE = """
import ctypes as C
import sys
import numpy as np
from spoc_b200 import api, workloads as W
fake = C.CDLL(None)
fake.fake_limit.argtypes = fake.fake_largest.argtypes = [C.c_size_t]
fake.fake_held.restype = C.c_size_t
fake.fake_filled.argtypes, fake.fake_filled.restype = [C.c_size_t], C.c_void_p
fake.fake_ran.restype = C.c_char_p
def kernels(call, *a):
    # names of the kernels a call launches, in order
    import re
    fake.fake_ran()
    call(*a)
    return re.findall(r"\\d((?:k|kf|kt|kx|ka|k16)_[a-z0-9_]+)", fake.fake_ran().decode())
RULES = {3: (12, 4), 4: (25, 5), 5: (27, 6), 6: (33, 7), 7: (42, 9)}
def problem(nc, variant, n):
    ng, ngf = RULES[nc]
    return W.build_problem(W.Config("host", variant, nc, ng, ngf, n, jitter=0.2, beta=2.0e-11, mu0=100.0,
                                    mb0=1.0e-3, seed=nc, ic="gauss8"))
def bytes_needed(p, variant):
    # the handle's fields and mesh records, without the operators
    n, ne, nf, g = p.mesh.ne * p.T.nm, p.mesh.ne, p.mesh.nf, p.T.ngf
    words = 22 * n + 3 * ne + 2 * nf + 7 * ne
    if variant != "lin":
        words += 12 * n + 6 * g * nf
    return 8 * words + 4 * (7 * ne + 4 * nf)
def error_of(call, *a):
    try:
        call(*a)
    except api.SpocError as e:
        return e.code
    return 0
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    """Runs a program in a process whose CUDA runtime is the stand-in."""
    so = tmp_path_factory.mktemp("fake") / "libfake_cudart.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", str(CUDA / "include"),
                    str(HERE / "fake_cudart.cpp"), "-o", str(so)], check=True)

    def go(program):
        r = subprocess.run([sys.executable, "-c", PRELUDE + textwrap.dedent(program)], cwd=HERE.parent,
                           env=dict(os.environ, LD_PRELOAD=str(so)), capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr

    return go


@pytest.mark.parametrize("variant", ["fs", "lin"])
@pytest.mark.parametrize("call", ["cal_var", "rk4_steps"])
def test_tile_counters_are_cleared_with_a_reported_wait_limit(host, variant, call):
    """A launch whose operators did not arrive in time leaves the tile counters
    wherever they were; the call that reports it leaves them zero for the next."""
    host(f"""
    p = problem(4, {variant!r}, 45)
    s = W.make_solver(p)
    s.set_state(p.u, p.v, p.h)
    flag = C.c_int.from_address(fake.fake_filled(4))
    counters = (C.c_uint * 6).from_address(fake.fake_filled(24))
    call = (lambda: s.rk4_steps(1.0, 1)) if {call!r} == "rk4_steps" else (lambda: s.cal_var(p.u, p.v, p.h))
    call()
    flag.value = 2
    counters[:] = [5, 3, 0, 7, 11, 2]
    assert error_of(call) == 2
    assert list(counters) == [0] * 6 and flag.value == 0
    call()
    """)


def test_short_host_runs_keep_the_step_graph_of_another_step_size(host):
    """Runs on the caller's arrays replay the step graph from eight steps on, and
    from three where the graph held is theirs; a short run with another step
    size neither captures one nor drops the one held."""
    host("""
    p = problem(4, "fs", 45)
    s = W.make_solver(p)
    x = [np.ascontiguousarray(a) for a in (p.u, p.v, p.h)]
    def graphs(dt, steps):
        g, l = fake.fake_graphs(), fake.fake_graph_launches()
        s.rk4_steps_host(*x, dt, steps)
        return fake.fake_graphs() - g, fake.fake_graph_launches() - l
    assert graphs(1.0, 7) == (0, 0)
    assert graphs(1.0, 8) == (1, 5)   # first and last step apart, one before the capture
    assert graphs(2.0, 4) == (0, 0)
    assert graphs(2.0, 7) == (0, 0)
    assert graphs(1.0, 5) == (0, 3)
    assert graphs(1.0, 3) == (0, 1)
    assert graphs(1.0, 2) == (0, 0)
    """)


@pytest.mark.parametrize("variant,n", [("fs", 45), ("lin", 60)])
def test_host_runs_on_a_stream_that_cannot_be_captured(host, variant, n):
    """cudaStreamLegacy cannot be captured: runs on the caller's arrays are plain
    launches there, however long."""
    host(f"""
    p = problem(4, {variant!r}, {n})
    s = W.make_solver(p)
    s.set_stream(1)
    x = [np.ascontiguousarray(a) for a in (p.u, p.v, p.h)]
    for steps in (7, 8, 20):
        assert error_of(s.rk4_steps_host, *x, 1.0, steps) == 0
    assert fake.fake_graphs() == 0
    """)


@pytest.mark.parametrize("nc,variant,n", [(4, "fs", 45), (7, "inv", 30), (5, "fs", 20), (3, "lin", 20)])
def test_handle_takes_no_more_memory_than_its_buffers(host, nc, variant, n):
    """A handle fits where its buffers do, in one piece or in pieces of their
    sizes; what one too large leaves behind does not reach the next."""
    host(f"""
    p = problem({nc}, {variant!r}, {n})
    need, operators = bytes_needed(p, {variant!r}), 2 << 20
    s = W.make_solver(p)
    assert need <= fake.fake_held() <= need + operators, (need, fake.fake_held())
    s.close()
    assert fake.fake_held() == 0
    fake.fake_limit(need + operators)
    s = W.make_solver(p)
    s.cal_var(p.u, p.v, p.h)
    s.close()
    fake.fake_limit(1 << 40)
    fake.fake_largest(8 * max(4 * p.mesh.ne * p.T.nm, 6 * p.T.ngf * p.mesh.nf) + operators)
    s = W.make_solver(p)
    s.cal_var(p.u, p.v, p.h)
    s.close()
    fake.fake_limit(need - 4096)
    assert error_of(W.make_solver, p) == 6
    assert fake.fake_held() == 0
    """)


def test_gradient_buffers_fit_in_pieces_of_their_sizes(host):
    host("""
    p = problem(4, "ns", 45)
    s = W.make_solver(p)
    n = p.mesh.ne * p.T.nm
    before = fake.fake_held()
    # the largest buffers are the 4 (3 ne) ngf side values
    fake.fake_largest(8 * 12 * p.mesh.ne * p.T.ngf + 4096)
    s.set_observations(np.array([1], np.int32), np.ones((1, p.T.nm)), np.array([2], np.int32), np.ones((1, 1)))
    s.bwd_window((p.u, p.v, p.h), 1.0, 4, 3)
    work = 8 * (82 * n + 7 * 3 * p.mesh.ne * p.T.ngf)
    assert fake.fake_held() - before <= work + 3 * 8 * 3 * n + (2 << 20), (fake.fake_held() - before, work)
    """)


@pytest.mark.parametrize("nc,variant,n", [(5, "lin", 50), (7, "fs", 32)])
def test_kernels_that_need_less_memory_run_where_there_is_none_for_the_others(host, nc, variant, n):
    """A handle whose fields fit is made, without what the kernels with several
    elements per warp need beside them; the same for the gradient's buffers."""
    host(f"""
    p = problem({nc}, {variant!r}, {n})
    s = W.make_solver(p)
    full = fake.fake_held()
    launches = fake.fake_launches()
    s.cal_var(p.u, p.v, p.h)
    tile = fake.fake_launches() - launches
    s.close()
    fake.fake_limit(full - 4096)
    s = W.make_solver(p)
    launches = fake.fake_launches()
    s.cal_var(p.u, p.v, p.h)
    assert (tile, fake.fake_launches() - launches) == ((2, 1) if {variant!r} == "lin" else (5, 3)), (tile, fake.fake_launches() - launches)
    s.rk4_steps(1.0, 3)
    s.close()
    fake.fake_limit(1 << 40)
    s = W.make_solver(p)
    before = fake.fake_held()
    s.adj_rhs((p.u, p.v, p.h), (p.u, p.v, p.h))
    full = fake.fake_held()
    s.close()
    if {variant!r} != "lin":
        s = W.make_solver(p)
        fake.fake_limit(full - 4096)
        s.adj_rhs((p.u, p.v, p.h), (p.u, p.v, p.h))
    """)


@pytest.mark.parametrize("nc", [3, 4, 5, 6, 7])
def test_meshes_of_the_gpu_tests_take_the_kernels_they_are_for(host, nc):
    """On 148 SMs the meshes of test_gpu_tile.py and test_gpu_routes.py run the
    several-element kernels, the one-launch kernels and the one-element kernels
    they are sized for."""
    host(f"""
    nc = {nc}
    def state(p):
        return p.u, p.v, p.h
    def steps(s, p):
        s.set_state(*state(p))
        return s.rk4_steps(1.0, 1)
    for precision in ("fp64", "fp64_fma"):
        for variant in ("fs", "ns", "inv"):
            p = problem(nc, variant, 37)
            s = W.make_solver(p, precision)
            right = ["kt_faces", "kt_qphase", "kt_nlvol", "kt_faces", "kt_tendency"]
            assert kernels(s.cal_var, *state(p)) == right
            assert kernels(steps, s, p) == 4 * right
            assert kernels(s.profile_rk4, 1.0, 1) == 4 * right
        p = problem(nc, "lin", 41)
        assert kernels(W.make_solver(p, precision).cal_var, *state(p)) == ["kt_faces", "kt_linear"]
    p = problem(nc, "lin", 61)
    assert kernels(steps, W.make_solver(p), p) == 4 * ["kt_faces", "kt_linear"]
    for variant in ("fs", "ns", "inv"):
        p = problem(nc, variant, 37)
        s = W.make_solver(p)
        ran = kernels(s.adj_rhs, state(p), state(p))
        assert [k for k in ran if k.startswith("ka_")] == ["ka_tend", "ka_faces", "ka_nlvol", "ka_qphase", "ka_faces"]
        s.set_kernel_path("generic")
        assert not any(k.startswith(("ka_", "kt_", "kf_")) for k in kernels(s.adj_rhs, state(p), state(p)))
        p = problem(nc, variant, 41)
        s = W.make_solver(p, "mixed")
        mixed = lambda: [k for k in kernels(s.cal_var, *state(p)) if k.startswith(("kx_vol", "kx_tend"))]
        assert mixed() == ["kx_vol_tile", "kx_tend_tile"]
        s.set_kernel_path("generic")
        assert mixed() == ["kx_vol", "kx_tend"]
        p = problem(nc, variant, 5)
        s = W.make_solver(p)
        per_stage = kernels(s.profile_rk4, 1.0, 1)
        assert len(per_stage) == (20 if nc < 7 else 12) and all(k.startswith("kf_") for k in per_stage), per_stage
        assert kernels(s.cal_var, *state(p)) == (["kf_nl_steps"] if nc < 7 else per_stage[:3])
    """)


def test_ensemble_kernel_follows_the_members_sizes(host):
    """Ensembles whose members fit one pass of their blocks take the kernel with
    one element per warp where that is the faster (148 SMs, one block each here)."""
    host("""
    def ens(*members):
        ps = [problem(nc, "fs", n) for nc, n in members]
        mem = [W.make_solver(p, "mixed") for p in ps]
        for p, s in zip(ps, mem):
            s.set_state(p.u, p.v, p.h)
        e = api.Ensemble(mem)
        ran = kernels(lambda: e.steps([1.0] * len(ps), 1, graph=False))
        return {k for k in ran if k.startswith("kx_ens")}
    small, tile = {"kx_ens_small"}, {"kx_ens_stage"}
    assert ens((5, 4), (6, 5)) == ens((3, 4), (5, 6), (6, 9)) == ens((6, 24)) == small
    assert ens((6, 25)) == ens((3, 12), (6, 25)) == tile
    assert ens((4, 4), (3, 4)) == ens((4, 20)) == tile
    assert ens((3, 4), (3, 6)) == ens((3, 24)) == small and ens((3, 25)) == tile
    """)
