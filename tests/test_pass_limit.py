"""The limit of a voxel's stress integrations in one evaluation, in each form that an evaluation takes.

The sweeps here end by themselves after a dozen integrations; a low limit ends them earlier.  Numerics
under which a voxel would go on without end (r_cutback >= 1) are not run.
"""
import ctypes as C

import numpy as np
import pytest

from damask_b200 import _lib, synthetic, workloads
from damask_b200.config import SolutionStruct
from damask_b200.grid import SpectralBasic, SpectralPolarization

SMALL, BEYOND = (2, 2, 2), (64, 37, 32)      # one launch; voxel lists (more than two blocks per SM)


def solver(cells, num=None, cls=SpectralBasic):
    rve = synthetic.voronoi_rve(cells, workloads.SIZE_1MM, 2, 0)
    return cls(rve.cells, rve.size, rve.material, rve.quaternions, workloads.fcc_al(), num or workloads.numerics_default())


@pytest.mark.gpu
@pytest.mark.parametrize('cells', [SMALL, BEYOND])
def test_sweep_ends_at_the_limit(gpu, cells):
    """One Newton iteration is allowed, so that every integration fails and the substep shrinks to its
    floor: 0.9^k > 0.3 for k < 12, twelve integrations a voxel."""
    num = workloads.numerics_default()
    num.N_iter_Lp_max, num.r_cutback, num.r_cutback_min = 1, 0.9, 0.3
    s = solver(cells, num)
    if cells is BEYOND:
        s.set_tuning(3, 4)                       # four lists
    F = np.tile((np.eye(3) + np.diag([5e-3, -2e-3, -2e-3])).reshape(-1), (s.N, 1))
    before = s.get_field('P')
    assert s.constitutive_response(F, 1.0)[-1] == 2
    assert np.all(s.iteration_counts()[:, 0] == 12)
    for limit in (11, 1):
        s.set_pass_limit(limit)
        with pytest.raises(_lib.DamaskError, match='constitutive passes did not terminate'):
            s.constitutive_response(F, 1.0)
        assert np.array_equal(s.get_field('P'), before)
    s.set_pass_limit(12)
    assert s.constitutive_response(F, 1.0)[-1] == 2
    with pytest.raises(_lib.DamaskError):
        s.set_pass_limit(0)
    s.close()


def step(s):
    s.forward(False, True, 1.0, 1.0, 1.0, workloads.tension_x(1.0, 1)[0])
    s.materialpoint_forward()


@pytest.mark.gpu
@pytest.mark.parametrize('cells,cls', [(SMALL, SpectralBasic), (BEYOND, SpectralBasic), (SMALL, SpectralPolarization)])
def test_solution_ends_at_the_limit(gpu, cells, cls):
    """The first increment of a tension test takes two state iterations and more in yielding voxels."""
    s = solver(cells, cls=cls)
    step(s)
    s.set_pass_limit(1)
    with pytest.raises(_lib.DamaskError, match='constitutive passes did not terminate'):
        s.solution()
    s.close()


@pytest.mark.gpu
def test_batch_ends_at_the_limit(gpu):
    members = [solver(SMALL), solver((4, 4, 4))]
    for s in members:
        s.set_pass_limit(1)
    h = C.c_void_p()
    _lib.check(members[0].lib.dmk_batch_create(C.byref(h), (C.c_void_p * 2)(*[s.ctx.value for s in members]), 2))
    for s in members:
        step(s)
    out = (SolutionStruct * 2)()
    with pytest.raises(_lib.DamaskError, match='constitutive passes did not terminate'):
        _lib.check(members[0].lib.dmk_batch_solution(h, (C.c_int * 2)(0, 1), 2, out))
    members[0].lib.dmk_batch_destroy(h)
    for s in members:
        s.close()
