"""The volume kernel's launch shape follows from a solve's configuration and size alone (vol_shape_rule,
csrc/vol_shapes.h): not from which solve of the process came first, nor from a timing.  A small solve before a
large one leaves the large one's shape and bits as they are, and an instance of a batch runs the shape that it
runs alone whatever else is in the batch."""
import numpy as np
import pytest

import fluxo_b200 as fb
from fluxo_b200.batch import Batch
from fluxo_b200.solver import set_volume_shape, volume_shape
from fluxo_b200.workloads import fourier_state

pytestmark = pytest.mark.gpu
BOX = dict(xmin=(0.0, 0.0, 0.0), xmax=(2.0, 2.0, 2.0))


def inputs(N, eqn, elems):
    mesh = fb.box_mesh(N, elems, BOX["xmin"], BOX["xmax"])
    U = fourier_state(mesh["Elem_xGP"], BOX["xmin"], BOX["xmax"], np.random.default_rng(N))
    kw = dict(N=N, eqn=eqn, riemann=44, volume_flux=5, ini_exact_func=0)
    if eqn == 1:
        kw.update(mu0=0.002, lifting=1, lifting_var=3)
    return mesh, U, fb.make_cfg(**kw)


def steps(N, eqn, elems):
    """(shape used, state after two steps) of a solve alone."""
    mesh, U, cfg = inputs(N, eqn, elems)
    op = fb.DGOperator(cfg=cfg)
    op.set_mesh(mesh)
    op.set_state(U)
    op.time_disc(0.0, 1e30, 2)
    out = op.get_state()
    op.close()
    return volume_shape(N, 5, eqn == 1)[1], out


# N, eqn, elements of a small and a large solve, the shapes of both
CASES = [(3, 0, (2, 2, 2), (16, 16, 16), 2, 1), (3, 0, (15, 16, 17), (16, 16, 16), 2, 1),
         (3, 1, (2, 2, 2), (16, 16, 16), 2, 2), (3, 1, (2, 2, 2), (26, 26, 25), 2, 1),
         (5, 0, (2, 2, 2), (12, 12, 12), 2, 0), (5, 1, (7, 9, 1), (4, 4, 4), 2, 0),
         (7, 1, (1, 1, 1), (8, 8, 8), 0, 0), (4, 1, (2, 2, 2), (10, 10, 10), 0, 0), (6, 0, (1, 1, 2), (6, 6, 6), 0, 0)]


@pytest.mark.parametrize("N,eqn,small,large,i_small,i_large", CASES)
def test_order_of_solves(gpu_lib, N, eqn, small, large, i_small, i_large):
    set_volume_shape(N, 5, eqn == 1, -1)
    assert volume_shape(N, 5, eqn == 1)[1] == -1
    a = steps(N, eqn, small)
    b = steps(N, eqn, large)
    assert (a[0], b[0]) == (i_small, i_large)
    set_volume_shape(N, 5, eqn == 1, -1)
    b2 = steps(N, eqn, large)
    a2 = steps(N, eqn, small)
    assert (a2[0], b2[0]) == (i_small, i_large)
    assert np.array_equal(a[1], a2[1]) and np.array_equal(b[1], b2[1])


@pytest.mark.parametrize("N,eqn,small,large,i_small,i_large", CASES[:6])
def test_batch_of_both(gpu_lib, N, eqn, small, large, i_small, i_large):
    b = Batch()
    ids = []
    for elems in (small, large, small):
        mesh, U, cfg = inputs(N, eqn, elems)
        ids.append(b.add(mesh, U, 0.0, 1e30, cfg=cfg))
    b.run(2)
    assert b.info()[0] == (2 if i_small != i_large else 1)  # groups
    for i, elems in zip(ids, (small, large, small)):
        assert np.array_equal(b.get_state(i), steps(N, eqn, elems)[1])
