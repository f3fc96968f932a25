"""MHD without non-conservative terms (noncons = 0) does not pay for them: its volume kernel forms neither of
their line sums.  Both right-hand sides run on the same state with launches alternating, and the fastest of
each counts; the sums' share of the kernel is 7 to 14 %, of which half is required."""
import numpy as np
import pytest

import fluxo_b200 as fb
from fluxo_b200.solver import profile, set_profiling
from fluxo_b200.workloads import mhd_orszag_tang_state

pytestmark = pytest.mark.gpu


def volume_us(op):
    profile(op, 3)
    op.dg_time_derivative(0.0)
    return profile(op, 3)[0] * 1e3


@pytest.mark.parametrize("N,elems,vf", [(5, 16, 12), (7, 12, 10)])
def test_no_time_for_absent_terms(gpu_lib, N, elems, vf):
    mesh = fb.box_mesh(N, (elems,) * 3, (0,) * 3, (2 * np.pi,) * 3)
    U = mhd_orszag_tang_state(mesh["Elem_xGP"], kappa=5 / 3)
    ops = []
    for nc in (0, 1):
        op = fb.DGOperator(N=N, eqn=2, riemann=10, volume_flux=vf, kappa=5 / 3, noncons=nc, ini_exact_func=0)
        op.set_mesh(mesh)
        op.set_state(U)
        op.glm_ch = 1.0
        set_profiling(op, True)
        ops.append(op)
    times = np.array([[volume_us(op) for op in ops] for _ in range(20)])
    off, on = times[3:].min(axis=0)
    assert off <= 0.96 * on, (off, on)
    for op in ops:
        op.close()
