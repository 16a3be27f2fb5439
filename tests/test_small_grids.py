"""Grids whose evaluations run as one launch, at the limit of that form and beyond it."""
import numpy as np
import pytest

from damask_b200 import synthetic, workloads
from damask_b200.batch import DeviceBatch
from damask_b200.grid import SpectralBasic, run_load_cases

from test_stress_forms import phase_of

pytestmark = pytest.mark.gpu

def at_limit(ns, beyond=0):
    """A grid of the one-launch limit, two resident blocks of 128 threads (64 at 48 systems) on every SM, or one
    layer more."""
    import torch
    sm = torch.cuda.get_device_properties(0).multi_processor_count
    return (sm // 4, 64, (16 if ns <= 24 else 8) + beyond) if sm % 4 == 0 else (sm, 32, (8 if ns <= 24 else 4) + beyond)


@pytest.mark.parametrize('size,phase', [('one', 'fcc12'), ('limit', 'fcc12'), ('beyond', 'fcc12'), ('limit', 'bcc48'),
                                        ('beyond', 'bcc48'), ('small', 'bcc12ns'), ('small', 'bcc24ns'), ('small', 'fcc18'),
                                        ('small', 'fcc15'), ('beyond', 'bcc12ns')])
def test_one_launch_against_the_passes(gpu, size, phase):
    """A batch runs the passes over lists at every size: two increments agree with the context's own."""
    ns = int(phase[3:5])
    cells = {'one': (1, 1, 1), 'small': (7, 6, 5)}.get(size) or at_limit(ns, int(size == 'beyond'))
    h = 1.0e-3 / max(cells)
    rve = synthetic.voronoi_rve(cells, tuple(h * c for c in cells), 7, 2)
    job = (rve, phase_of(phase), workloads.tension_x(60.0, 60), workloads.numerics_default())
    db = DeviceBatch([job], max_increments=2)
    db.run_native()
    s = SpectralBasic(rve.cells, rve.size, rve.material, rve.quaternions, job[1], job[3])
    ref = run_load_cases(s, job[2], max_increments=2)
    assert [r.iterations for r in db.results[0]] == [r.iterations for r in ref]
    assert np.array_equal(s.counters()[1:3], db.solvers[0].counters()[1:3])       # state and Newton iterations
    for name in ('P', 'F', 'F_p', 'L_p', 'xi_sl', 'gamma_sl'):
        a, b = s.get_field(name), db.solvers[0].get_field(name)
        # the transforms' plans may round differently: the bound of the batch tests
        assert np.abs(a - b).max() <= 1e-11 * max(np.abs(b).max(), 1e-300), name
    s.close()
    db.close()


@pytest.mark.parametrize('beyond', [False, True])
def test_failed_sweep_keeps_the_stress(gpu, beyond):
    cells = at_limit(12, 1) if beyond else (2, 2, 2)
    num = workloads.numerics_default()
    rve = synthetic.voronoi_rve(cells, workloads.SIZE_1MM, 2, 0)
    num.N_iter_Lp_max = 1
    s = SpectralBasic(rve.cells, rve.size, rve.material, rve.quaternions, workloads.fcc_al(), num)
    before = s.get_field('P')
    F = np.tile((np.eye(3) + np.diag([5e-3, -2e-3, -2e-3])).reshape(-1), (s.N, 1))
    P, P_av, *_, status = s.constitutive_response(F, 1.0)
    assert status != 0
    assert np.array_equal(P, before) and np.array_equal(s.get_field('P'), before)
    assert np.allclose(P_av, before.mean(0), atol=1e-6)
    s.close()
