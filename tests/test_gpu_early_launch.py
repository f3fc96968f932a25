"""Early launches (launch_k, csrc/common.cuh) of a solve's kernels against the same solve without them: a batch
of one instance launches the same kernels in the same shapes without the launch attribute.  The bits agree on
both sides of the sizes where the rule changes (200 k and 2^20 nodes), and on a mesh of less than a wave of
blocks, where a successor that comes up too early slows its predecessor down, they cost no time."""
import time

import numpy as np
import pytest

import fluxo_b200 as fb
from fluxo_b200.batch import Batch
from fluxo_b200.workloads import fourier_state

pytestmark = pytest.mark.gpu
BOX = dict(xmin=(0.0, 0.0, 0.0), xmax=(2.0, 2.0, 2.0))


def case(N, elems, eqn):
    mesh = fb.box_mesh(N, elems, BOX["xmin"], BOX["xmax"])
    U = fourier_state(mesh["Elem_xGP"], BOX["xmin"], BOX["xmax"], np.random.default_rng(N))
    kw = dict(N=N, eqn=eqn, riemann=44, volume_flux=5, ini_exact_func=0, cfl_scale=0.5, dfl_scale=0.4)
    if eqn == 1:
        kw.update(mu0=0.002, lifting=1, lifting_var=3)
    cfg = fb.make_cfg(**kw)
    op = fb.DGOperator(cfg=cfg)
    op.set_mesh(mesh)
    op.set_state(U)
    b = Batch()
    return op, b, b.add(mesh, U, 0.0, 1e30, cfg=cfg), U


@pytest.mark.parametrize("N,elems,eqn", [
    (3, (2, 2, 2), 1), (3, (14, 14, 15), 0), (3, (15, 15, 14), 0), (3, (16, 16, 16), 0), (3, (32, 32, 16), 0), (3, (32, 32, 17), 0),
    (7, (8, 8, 6), 1), (7, (8, 8, 7), 1), (7, (16, 16, 8), 1), (7, (16, 16, 9), 1)])
def test_same_bits(gpu_lib, N, elems, eqn):
    op, b, i, _ = case(N, elems, eqn)
    t, n, err = op.time_disc(0.0, 1e30, 3)
    assert err == 0 and n == 3
    b.run(3)
    assert np.array_equal(op.get_state(), b.get_state(i))
    op.close()


@pytest.mark.parametrize("N,elems", [(1, 16), (5, 5), (7, 5)])
def test_no_time_lost_below_a_wave(gpu_lib, N, elems):
    op, b, i, U = case(N, (elems,) * 3, 1)
    steps, best = 20, [1e9, 1e9]
    for _ in range(12):
        op.set_state(U)
        t0 = time.perf_counter()
        assert op.time_disc(0.0, 1e30, steps)[1:] == (steps, 0)
        t1 = time.perf_counter()
        b.set_state(i, U)
        t2 = time.perf_counter()
        assert b.run(steps) == 1
        best = [min(best[0], t1 - t0), min(best[1], time.perf_counter() - t2)]
    assert best[0] <= 1.15 * best[1], [x / steps * 1e6 for x in best]
    op.close()
