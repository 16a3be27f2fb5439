"""The two forms of the Lp Newton step: the five-unknown form that a phase without non-Schmid terms
takes, and the general one, each against the oracle and against each other on the same material."""
import numpy as np
import pytest

from damask_b200 import synthetic, workloads
from damask_b200.grid import SpectralBasic

from conftest import rel, rel_pv

pytestmark = pytest.mark.gpu

# the oracle's and the kernels' orders of sums agree to 1e-11 in these fields (see test_gpu_parity)
TOL = 1e-9


def bcc_12(nonschmid=None):
    p = workloads.bcc_24()
    for name in ('N_sl', 'dot_gamma_0_sl', 'n_sl', 'a_sl', 'h_0_sl_sl', 'xi_0_sl', 'xi_inf_sl'):
        setattr(p, name, getattr(p, name)[:1])
    p.a_nonschmid = list(nonschmid or [])
    return p


def sweep(make, phase, cells, F, num):
    rve = synthetic.voronoi_rve(cells, workloads.SIZE_1MM, 5, 3)
    s = make(rve.cells, rve.size, rve.material, rve.quaternions, phase, num)
    out = []
    for dt in (1.0, 0.5):                      # the second sweep starts from the first one's Lp
        P, *_, status = s.constitutive_response(F, dt)
        assert status == 0
        out.append(P)
    out += [s.get_field(k) for k in ('F_p', 'L_p', 'S', 'F_e', 'xi_sl', 'gamma_sl')]
    counts = s.iteration_counts() if hasattr(s, 'iteration_counts') else None
    s.close()
    return out, counts


def deformation(n, strain, seed=1):
    F = np.eye(3) + np.diag([strain, -0.375 * strain, -0.375 * strain])
    return np.tile(F.reshape(-1, order='F'), (n, 1)) + 0.05 * strain * np.random.default_rng(seed).normal(size=(n, 9))


@pytest.mark.parametrize('option', ['integer n', 'other n', 'kept Jacobian', 'line search'])
@pytest.mark.parametrize('cells,phase', [((1, 1, 1), 'fcc12'), ((5, 5, 5), 'bcc24'), ((3, 43, 1), 'fcc12'),
                                         ((13, 5, 3), 'bcc48'), ((8, 6, 4), 'bcc24')])
def test_forms_against_oracle(gpu, oracle_lib, cells, phase, option):
    """Voxel counts around a block (1, 125, 129, 195, 192) and the options of the Newton iteration."""
    ph = {'fcc12': workloads.fcc_al, 'bcc24': workloads.bcc_24, 'bcc48': workloads.bcc_48}[phase]()
    num = workloads.numerics_default()
    # beyond 4e-3 a voxel's Newton iteration may stall (and the voxel take a substep) by its last bit
    strain = 2e-3
    if option == 'other n':
        ph.n_sl = [15.5] * len(ph.N_sl)
    elif option == 'kept Jacobian':
        num.f_update_jacobi_Lp = 2             # the first Jacobian is kept: it converges near yield only
        strain = 6e-4
    elif option == 'line search':
        num.r_linesearch_Lp = 0.3
    F = deformation(int(np.prod(cells)), strain)
    a, _ = sweep(SpectralBasic, ph, cells, F, num)
    b, _ = sweep(oracle_lib.OracleSpectralBasic, ph, cells, F, num)
    for x, y in zip(a, b):
        assert rel(x, y) < TOL and rel_pv(x, y) < TOL


@pytest.mark.parametrize('cells', [(4, 8, 4), (7, 7, 3)])
def test_general_form_on_a_schmid_material(gpu, cells):
    """Non-Schmid coefficients of 1e-18 select the general form (they change zero entries of P_nS) and
    leave the resolved shears what they are to 1e-18: both forms take the same iterations to the
    same fields up to their rounding."""
    num = workloads.numerics_default()
    F = deformation(int(np.prod(cells)), 4e-3)
    a, ca = sweep(SpectralBasic, bcc_12(), cells, F, num)
    b, cb = sweep(SpectralBasic, bcc_12([1e-18] * 6), cells, F, num)
    assert np.array_equal(ca, cb)
    for x, y in zip(a, b):
        assert rel(x, y) < 1e-10 and rel_pv(x, y) < 1e-10
    # coefficients that are given but zero keep the five-unknown form
    c, cc = sweep(SpectralBasic, bcc_12([0.0] * 6), cells, F, num)
    assert np.array_equal(ca, cc) and all(np.array_equal(x, y) for x, y in zip(a, c))
