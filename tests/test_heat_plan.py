"""The plan of a heat cycle (csrc/heat_plan.h, plain C++) from weakly coupled to steady-state rows."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "i3elvis_b200", "csrc")


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    src = d / "plan.cpp"
    src.write_text('#include "heat_plan.h"\n'
                   'extern "C" int plan(const double *q, const double *qall, int n, double w, double rtol, int *sweeps)\n'
                   '{ const i3g::HeatPlan P = i3g::heat_plan(q, qall, n, w, rtol); *sweeps = P.sweeps; return P.last; }\n'
                   'extern "C" double rate(double q, double w) { return i3g::heat_sweep_rate(q, w); }\n')
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(d / "plan.so")], check=True)
    L = C.CDLL(str(d / "plan.so"))
    L.plan.argtypes = [C.POINTER(C.c_double), C.POINTER(C.c_double), C.c_int, C.c_double, C.c_double, C.POINTER(C.c_int)]
    L.rate.argtypes, L.rate.restype = [C.c_double, C.c_double], C.c_double

    def run(q, w=1.0, rtol=1e-10, qall=None):
        s = C.c_int()
        last = L.plan((C.c_double * len(q))(*q), (C.c_double * len(q))(*(qall or q)), len(q), w, rtol, C.byref(s))
        return last, s.value
    run.rate = L.rate
    return run


def test_steady_rows_keep_every_level_and_all_sweeps(plan):
    """rho cp / dt far below the neighbour coefficients, zero or not a number: the whole hierarchy with 16
    sweeps on the coarsest level, also where q / (1 + q) rounds to 1."""
    for q in (1e3, 1e8, 1e15, 1e16, 1e17, 1e200, np.inf, np.nan):
        assert plan([q, q, q]) == (2, 16), q
        assert plan([q]) == (0, 16), q


def test_damping_outside_the_convergent_range_takes_all_sweeps(plan):
    for w in (0.0, -1.0, 2.0, 2.5, np.nan):
        assert plan([0.5, 0.1], w=w) == (0, 16), w
        assert plan([9.0, 0.1], w=w) == (1, 16), w


def test_weak_coupling_stays_on_level_0(plan):
    # q = 0.1: a sweep leaves (0.1 / 1.1)^2 = 0.0083 of the error, 1e-10 needs 4.8 of them
    assert plan([0.1, 0.02]) == (0, 5)
    assert plan([0.0, 0.0]) == (0, 2)
    assert plan([1.0, 0.25]) == (0, 12)
    assert plan([1.0]) == (0, 16)
    # coarser levels: down to the first with q <= 1, which reduces its error by 1e-3
    assert plan([4.0, 1.0, 0.25]) == (1, 5)
    assert plan([1e3, 250.0, 60.0]) == (2, 16)


def test_narrow_outer_cells_ask_for_sweeps_of_a_coarse_level(plan):
    q = [1.8, 0.45]
    assert plan(q) == (1, 3)
    assert plan(q, qall=[1.8, 1.8]) == (1, 3)      # a quarter of their error in one sweep
    q = [36.0, 9.0, 2.3, 0.6]
    assert plan(q, qall=[36.0] * 4) == (3, 6)      # (36 / 37)^2 = 0.947 a sweep
    q = [120.0, 30.0, 7.5, 1.9, 0.5]
    assert plan(q, qall=[120.0] * 5) == (4, 16)
    assert plan([0.5, 0.2], qall=[0.5, np.inf]) == (0, 11)   # level 0 has no cells of another kind


@pytest.mark.parametrize("w", [0.5, 0.9, 1.0, 1.2, 1.6])
def test_rate_is_that_of_the_relaxed_matrix(plan, w):
    """Red-black relaxation of the 1-D rows (1 + q) x_i - q/2 (x_i-1 + x_i+1) on a ring, whose Jacobi radius
    is q / (1 + q): the spectral radius of the sweep's matrix equals the plan's rate."""
    n, q = 16, 3.0
    J = np.zeros((n, n))
    for i in range(n):
        J[i, (i + 1) % n] = J[i, (i - 1) % n] = q / 2 / (1 + q)
    S = np.eye(n)
    for colour in (0, 1):
        step = np.eye(n)
        step[colour::2] = ((1 - w) * np.eye(n) + w * J)[colour::2]
        S = step @ S
    assert abs(max(abs(np.linalg.eigvals(S))) - plan.rate(q, w)) < 1e-6
