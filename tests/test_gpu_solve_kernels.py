"""GPU: each kernel of the pressure solve runs where its tests mean it to, as
ntcfd_solve_plan reports it, and the two that no other size reaches are held
against the rest: the resident kernel's exchange on rows that share a warp or
leave lanes over, and the half-sweep kernels (rows of more than 234 cells) in
each of their uses -- step graph, eager launches, moving body, solves without
sweeps, adjoint solves with queued bodies.

Tolerances are those of the same comparisons elsewhere: 1e-12 for two paths of
one step or against the oracle (60 sweeps of at most an ulp; 60 ulp of 1 in a last
change of 1e-5 or more, 1e-9), 1e-9 for the gradients of two paths.
"""
import math

import numpy as np
import pytest

import test_gpu_adjoint as adjoint
import test_gpu_march as march
import test_gpu_resident_deep as deep
import test_gpu_resident_thin as thin
from conftest import interior, rel_l2
from ntustcfdlab_b200 import abi, cases
from ntustcfdlab_b200.abi import (FP64, MIXED, SOLVE_HALF_SWEEPS, SOLVE_MARCH, SOLVE_RESIDENT, SOLVE_RESIDENT_DEEP,
                                  SOR_RESIDENT, SOR_STREAMING, f4, make_params)
from ntustcfdlab_b200.solver import Solver, gridder_equal

pytestmark = pytest.mark.gpu

CAVITY = {"North": ("Dirichlet", "no-slip", "no-slip")}


def _plan(n, precision, path):
    with Solver(make_params(*n, Re=100.0, dt=1e-3, precision=precision, sor_path=path), gridder_equal(*n, 1.0, 1.1, 0.9)) as s:
        return s.solve_plan()


@pytest.mark.parametrize("precision", [FP64, MIXED])
def test_the_kernels_of_the_tests_sizes(precision):
    for n in deep.SIZES:
        assert _plan(n, precision, SOR_RESIDENT)["kernel"] == SOLVE_RESIDENT_DEEP, n
        assert _plan(n, precision, SOR_STREAMING)["kernel"] == SOLVE_MARCH, n
    for n in march.SIZES:
        assert _plan(n, precision, SOR_STREAMING)["kernel"] == SOLVE_MARCH, n
    for n in [n for p, n in thin.CASES if p == precision]:
        plan = _plan(n, precision, SOR_RESIDENT)
        assert plan["kernel"] == SOLVE_RESIDENT, n
        assert _plan(n, precision, SOR_STREAMING)["kernel"] == (SOLVE_HALF_SWEEPS if n[0] > 234 else SOLVE_MARCH), n
    assert any(2 * _plan(n, p, SOR_RESIDENT)["nbj"] > n[1] for p, n in thin.CASES if p == precision)


# rows side by side on a warp (two to four) and rows that leave lanes over; d and 1/diag on the chip, d
# alone, neither
NARROW = [(FP64, (33, 116, 150)), (FP64, (16, 200, 200)), (FP64, (17, 200, 300)), (FP64, (33, 134, 264)), (FP64, (48, 150, 150)),
          (FP64, (48, 192, 187)), (FP64, (62, 150, 170)), (MIXED, (17, 200, 300)), (MIXED, (21, 150, 150)),
          (MIXED, (40, 100, 100)), (MIXED, (47, 192, 187)), (MIXED, (63, 160, 180))]


@pytest.mark.parametrize("precision,n", NARROW)
def test_narrow_rows_hand_over_twice_a_sweep(precision, n):
    plan = _plan(n, precision, SOR_RESIDENT)
    assert plan["kernel"] == SOLVE_RESIDENT and plan["nbj"] * plan["nbk"] > 1
    kw = dict(mixed_cycle=5, check_every=1 if n[0] % 2 else 5, itmax=60, zeta=1e-3)
    march._same(march._solve(n, precision, SOR_STREAMING, SOR_STREAMING, **kw),
                march._solve(n, precision, SOR_RESIDENT, SOR_RESIDENT, **kw))


# ---- the half-sweep kernels
LONG = (236, 7, 6)


def _long(precision, n=LONG, **kw):
    s = Solver(make_params(*n, Re=100.0, dt=f4(1e-3), precision=precision, sor_path=SOR_STREAMING, bc=CAVITY, **kw),
               gridder_equal(*n, 6.0, 1.1, 0.9))
    assert s.solve_plan()["kernel"] == SOLVE_HALF_SWEEPS
    return s


def _state(s, seed):
    rng = np.random.default_rng(seed)
    return [np.asfortranarray(0.3 * rng.standard_normal(s.halo_shape)) for _ in range(4)]


@pytest.mark.parametrize("sweeps", [1, 7])
def test_half_sweeps_match_the_oracle(orc, sweeps):
    with _long(FP64, zeta=0.0, itmax=sweeps) as s:
        o = orc.Oracle(make_params(*LONG, Re=100.0, dt=f4(1e-3), bc=CAVITY, zeta=0.0, itmax=sweeps),
                       gridder_equal(*LONG, 6.0, 1.1, 0.9))
        o.initial_conditions()
        st = _state(s, 5)
        s.set_state(*st)
        for k, a in zip("uvwp", st):
            o.set(k, a)
        s.boundary_conditions()
        o.boundary_conditions()
        info, _ = s.step(2)
        o.step(2, forced=[sweeps, sweeps])
        assert [i.sor_iters for i in info] == [sweeps, sweeps]
        for k, a in zip("uvwp", s.get_state()):
            assert rel_l2(interior(a), interior(o.get(k))) <= 1e-12, k


@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("cycle,every", [(4, 1), (6, 3)])
def test_half_sweeps_eager_graph_and_resident_agree(precision, cycle, every):
    out = []
    for eager in (0, 1):
        with _long(precision, eager=eager, mixed_cycle=cycle, check_every=every) as s:
            s.set_state(*_state(s, 6))
            s.boundary_conditions()
            info, rc = s.step(3)
            assert rc == 0
            out.append((s.get_state(), [(i.sor_iters, i.dc_cycles, i.launches) for i in info]))
    assert out[0][1] == out[1][1]
    for a, b in zip(out[0][0], out[1][0]):
        np.testing.assert_array_equal(a, b)
    p = make_params(*LONG, Re=100.0, dt=f4(1e-3), precision=precision, sor_path=SOR_RESIDENT, bc=CAVITY, mixed_cycle=cycle,
                    check_every=every)
    with Solver(p, gridder_equal(*LONG, 6.0, 1.1, 0.9)) as s:
        s.set_state(*_state(s, 6))
        s.boundary_conditions()
        info, _ = s.step(3)
        assert [(i.sor_iters, i.dc_cycles) for i in info] == [q[:2] for q in out[0][1]]
        for a, b in zip(s.get_state(), out[0][0]):
            assert rel_l2(interior(a), interior(b)) <= 1e-12


@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("eager", [0, 1])
def test_half_sweep_solve_without_sweeps_leaves_p(precision, eager):
    with _long(precision, itmax=0, eager=eager) as s:
        st = _state(s, 5)
        s.set_state(*st)
        info, rc = s.step(1)
        assert rc == abi.NTCFD_NOT_CONVERGED and info[0].sor_iters == 0
        np.testing.assert_array_equal(interior(s.get_state()[3]), interior(st[3]))


@pytest.mark.parametrize("eager", [0, 1])
def test_half_sweeps_with_a_moving_body(eager):
    """The moving-body graph around the half-sweep loops against the one around the resident kernel."""
    n, start = (235, 20, 24), 2
    bc = {"West": ("periodic",) * 3, "East": ("periodic",) * 3, "South": ("Neumann",) * 3, "North": ("Neumann",) * 3,
          "Back": ("Dirichlet",) * 3, "Front": ("Neumann",) * 3}
    t = 2.0 * math.pi * np.arange(41) / 40 + 0.0137
    z, y = 0.5 + 0.61 * np.cos(t), 0.31 * np.sin(t)
    z[-1], y[-1] = z[0], y[0]
    got = []
    for path in (SOR_STREAMING, SOR_RESIDENT):
        p = make_params(*n, Re=300.0, dt=f4(1e-3), bc=bc, bc_value={"Back": (0.0, 0.0, 1.0)}, lx=6.0, sor_path=path,
                        eager=eager)
        with Solver(p, gridder_equal(*n, 6.0, 3.0, 4.0)) as s:
            assert s.solve_plan()["kernel"] == (SOLVE_HALF_SWEEPS if path == SOR_STREAMING else SOLVE_RESIDENT)
            s.set_dynamic_aoa(z, y, 5.0, 2.0, 1.2137, 1.5071, start)
            s.boundary_conditions()
            info, rc = s.step(4)
            assert rc == 0 and info[0].aoa == 0.0 and info[3].aoa > 5.0
            got.append((s.get_state(), s.get_mask(), [(i.sor_iters, i.aoa) for i in info]))
    (a, ma, ia), (b, mb, ib) = got
    assert ia == ib and ma.any()
    np.testing.assert_array_equal(ma, mb)
    for x, q in zip(a, b):
        assert rel_l2(interior(x), interior(q)) <= 1e-12


def test_half_sweep_adjoint_equals_the_resident_one():
    def case(path):
        return cases.cylinder_crossflow(236, 12, 16, 6.0, 6.0, 8.0, zc=2.55, yc=3.1, D=1.3, Re=100.0, dt=0.01, U=1.0,
                                        theta_deg=5.0, steps=adjoint.K, precision=FP64, zeta=1e-12, itmax=200000, sor_path=path)

    c = case(SOR_RESIDENT)
    state = adjoint.initial_state(c)
    force = cases.body_force_c4((236, 12, 16), scale=1e-2)
    r = adjoint.run_adjoint(c, state, force)
    with Solver(case(SOR_STREAMING).params, c.grid) as s:
        assert s.solve_plan()["kernel"] == SOLVE_HALF_SWEEPS
    q = adjoint.run_adjoint(case(SOR_STREAMING), state, force)
    assert abs(q["dJ_dU"] - r["dJ_dU"]) <= 1e-9 * abs(r["dJ_dU"])
    assert adjoint._rel(q["dJ_df"], r["dJ_df"]) <= 1e-9
