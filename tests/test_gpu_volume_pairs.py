"""The volume and lifting kernels at the sizes where their schedules can go wrong: every launch shape of the
volume kernel (N+1 = 4, 6, 8: two nodes of a line per thread or one; odd N+1), each pinned in turn, on
element counts that leave a partly filled last block, every volume flux, BR1 and BR2, and states whose
neighbouring nodes lie on both sides of the logarithmic mean's series limit ((b-a)/(b+a))^2 = 1e-4.
Tolerance: relative L2 <= 1e-12 against the CPU oracle (64-bit sums of at most 3 (N+1) <= 24 pair fluxes per
node in another order, a few 1e-15 each, which cancel to a hundredth of their size or more)."""
import numpy as np
import pytest

import fluxo_b200 as fb
from fluxo_b200.solver import set_volume_shape, volume_shape
from oracle.oracle import OracleCase

pytestmark = pytest.mark.gpu
REF = ((1.2, 0.1, 0.0, 0.1, 0.9, 1.0, 1.0, 1.0), (1.1, 0.2, -0.1, 0.2, 0.6, 1.0, 1.0, 1.0))
CUBE = dict(NGeo=2, deform_amp=0.1, xmin=(-1, -1, -1), xmax=(1, 1, 1))


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def every_shape(N, eqn, elems, lift, vf, noise):
    """The right-hand side of every launch shape of the volume kernel against the oracle's."""
    c = OracleCase(N=N, nElems=elems, ini_exact_func=2, riemann=44, volume_flux=vf, eqn=eqn, mu0=0.01 if eqn else 0.0,
                   lifting=lift, lifting_var=3, **CUBE)
    U = c.get_U()
    U = U * (1 + noise * np.random.default_rng(N + 10 * vf).standard_normal(U.shape))
    c.set_U(U)
    ref = c.dg_time_derivative(0.0)
    p = c.params
    op = fb.DGOperator(N=N, eqn=eqn, riemann=44, volume_flux=vf, lifting=lift, lifting_var=3, mu0=p.mu0, kappa=p.kappa,
                       R=p.R, Pr=p.Pr, etaBR2=p.etaBR2, ini_exact_func=2)
    op.set_mesh(c.mesh())
    op.set_state(U)
    try:
        for i in range(volume_shape(N, vf, eqn == 1)[0]):
            set_volume_shape(N, vf, eqn == 1, i)
            op.dg_time_derivative(0.0)
            assert rel(op.get_ut(), ref) <= 1e-12, "shape %d" % i
    finally:
        set_volume_shape(N, vf, eqn == 1, -1)
    op.close()


@pytest.mark.parametrize("vf,noise", [(5, 0.0), (5, 0.007), (5, 0.1), (32, 0.007), (10, 0.007), (7, 0.007), (2, 0.1)])
@pytest.mark.parametrize("N,elems,lift", [(2, (3, 3, 1), 1), (3, (3, 3, 1), 2), (4, (3, 1, 1), 1), (5, (3, 1, 1), 2),
                                          (6, (1, 2, 1), 1), (7, (1, 2, 1), 1), (7, (1, 2, 1), 2)])
def test_navier_stokes(gpu_lib, N, elems, lift, vf, noise):
    every_shape(N, 1, elems, lift, vf, noise)


@pytest.mark.parametrize("vf", [0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 32])
@pytest.mark.parametrize("N,elems", [(1, (17, 1, 1)), (2, (3, 3, 1)), (3, (5, 1, 1)), (3, (7, 1, 1)), (4, (3, 1, 1)),
                                     (5, (3, 1, 1)), (6, (1, 1, 1)), (7, (1, 1, 1))])
def test_euler_every_flux(gpu_lib, N, elems, vf):
    every_shape(N, 0, elems, 1, vf, 0.03)


@pytest.mark.parametrize("vf,nc,glm,noise", [(10, 1, 1, 0.007), (10, 2, 0, 0.03), (12, 3, 1, 0.007), (0, 1, 1, 0.02),
                                             (1, 0, 0, 0.02)])
@pytest.mark.parametrize("N,elems", [(2, (3, 3, 1)), (3, (3, 1, 1)), (4, (3, 1, 1)), (5, (3, 1, 1)), (6, (1, 2, 1)),
                                     (7, (1, 2, 1))])
def test_resistive_mhd(gpu_lib, N, elems, vf, nc, glm, noise):
    c = OracleCase(eqn=3, N=N, nElems=elems, kappa=5 / 3, mhd_ref_state=REF, ini_exact_func=201, ini_center=(0, 0, 0),
                   ini_halfwidth=0.4, ini_amplitude=0.1, glm_ch=0.7, volume_flux=vf, riemann=10, noncons=nc, nc_glm=glm,
                   eta=0.01, mu0=0.01, lifting=1 + N % 2, lifting_var=3, **CUBE)
    rng = np.random.default_rng(N)
    U = c.get_U()
    U = U * (1 + noise * rng.standard_normal(U.shape))
    U[..., 8] = 0.05 * rng.standard_normal(U[..., 8].shape)
    c.set_U(U)
    ref = c.dg_time_derivative(0.0)
    p = c.params
    op = fb.DGOperator(N=N, eqn=3, riemann=10, volume_flux=vf, lifting=p.lifting, lifting_var=3, kappa=p.kappa, Pr=p.Pr,
                       mu0=p.mu0, etaBR2=p.etaBR2, ini_exact_func=1, mu_0=p.mu_0, eta=p.eta, glm_scale=p.glm_scale,
                       glm_scr=p.glm_scr, noncons=nc, nc_glm=glm)
    op.set_mesh(c.mesh())
    op.set_state(U)
    op.glm_ch = 0.7
    op.dg_time_derivative(0.0)
    assert rel(op.get_ut(), ref) <= 1e-12
    op.close()
