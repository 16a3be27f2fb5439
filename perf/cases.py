"""The work that programs using this package have it do, as a fixed list of cases with their inputs.

Every case goes through the package's Python entry points (``damask_b200.grid``, ``.batch``,
``.adjoint``) on seeded synthetic polycrystals, with the materials, loads and numerics of
``damask_b200.workloads`` and of the tests.  ``listed()`` names the cases, ``draw(rng)`` gives more of
the same ranges, ``prepare`` makes what a program holds before the call, ``run`` is one pass.

Kinds of pass:

* ``increment``   one load increment of the basic spectral scheme from a device checkpoint (restore,
  forward, materialpoint_forward, solution, updateCoords) and the read-back of its output fields
  into pinned host memory: the step a simulation repeats;
* ``cutback``     the same increment of the polarization scheme at half the time step after a
  cutback, and its read-back (that scheme has no checkpoints);
* ``batch``       one increment of many small grids in one batch, and their read-back;
* ``gradient``    one step of a parameter fit: the stress curve of a few increments and its gradient
  with respect to the hardening parameters (forward and adjoint, through torch.autograd);
* ``response``    one material-point sweep at a prescribed F (host arrays in and out);
* ``coordinates`` cell-centre and node coordinates of a deformation field.

``exact`` restates the path in torch and numpy, in 64 bits, where it can be given in a few seconds:
the coordinates, the material-point sweep, and the first increment of a load case from the
undeformed state (its reference medium and compliance are elastic, so no consistent tangent of a
plastic state enters).
"""
import math

import numpy as np
import torch

from damask_b200 import adjoint, workloads
from damask_b200.batch import DeviceBatch
from damask_b200.config import Numerics, Phase
from damask_b200.grid import IncrementDriver, SpectralBasic, SpectralPolarization
from damask_b200.synthetic import voronoi_rve

FIELDS = ('F', 'P', 'F_p', 'L_p', 'xi_sl', 'gamma_sl')


# ------------------------------------------------------------------------------------ the cases
def _increment(name, cells, phase, precision, pre, grains, derivative='continuous', load='tension', fields='all'):
    return {'name': name, 'kind': 'increment', 'c0': cells[0], 'c1': cells[1], 'c2': cells[2], 'phase': phase,
            'precision': precision, 'pre': pre, 'grains': grains, 'derivative': derivative, 'load': load,
            'fields': fields}


def listed():
    return [
        # the smallest grid of the batched workload, alone: launches and host round trips
        _increment('increment_fcc_8', (8, 8, 8), 'fcc12', 'fp64', 0, 5),
        # the 16^3 configuration, in plastic flow
        _increment('increment_fcc_16', (16, 16, 16), 'fcc12', 'fp64', 2, 20),
        # a ragged grid with prime edges, the difference-scheme operator, and the 17-grains
        # regression material (non-Schmid terms)
        _increment('increment_bcc12ns_odd', (31, 17, 23), 'bcc12ns', 'fp64', 1, 17, derivative='FWBW_difference'),
        # the 64^3 configuration in its mixed form
        _increment('increment_fcc_64', (64, 64, 64), 'fcc12', 'mixed', 2, 200),
        # the 64^3 cut of the 24-system benchmark, FP64, first increment (elastic-plastic transition)
        _increment('increment_bcc24_64', (64, 64, 64), 'bcc24', 'fp64', 0, 31),
        # all three bcc families under shear, an edge that is not a power of two
        _increment('increment_bcc48_40', (40, 40, 40), 'bcc48', 'fp64', 1, 12, load='shear'),
        # the largest: a 128^3 cut of the 24-system benchmark in flow; a production run writes the
        # fields that its post-processing needs
        _increment('increment_bcc24_128', (128, 128, 128), 'bcc24', 'mixed', 2, 250, fields='output'),
        # the other grid solver, a step repeated after a cutback
        {'name': 'cutback_fcc_32', 'kind': 'cutback', 'c0': 32, 'c1': 32, 'c2': 32, 'phase': 'fcc12', 'grains': 50},
        # serving many small microstructures: RVEs of 8^3 to 24^3 in one batch
        {'name': 'batch_fcc_48', 'kind': 'batch', 'n': 48, 'precision': 'mixed', 'max_edge': 24},
        # a step of a parameter fit, forward and backward
        {'name': 'gradient_fcc_12', 'kind': 'gradient', 'c0': 12, 'c1': 12, 'c2': 12, 'grains': 10, 'increments': 2},
        # material points at a prescribed deformation, host arrays
        {'name': 'response_bcc24_32', 'kind': 'response', 'c0': 32, 'c1': 32, 'c2': 31, 'phase': 'bcc24', 'grains': 60},
        # coordinates of the cells and nodes for a result file
        {'name': 'coordinates_63', 'kind': 'coordinates', 'c0': 63, 'c1': 64, 'c2': 65},
    ]


def _edges(rng, lo, hi, most):
    """Three edges spread over their logarithm, odd ones among them, of at most `most` cells."""
    while True:
        a = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        c = [max(lo, min(hi, int(round(a * rng.choice((1.0, 1.0, 1.0, rng.uniform(0.6, 1.5))))))) for _ in range(3)]
        if c[0] * c[1] * c[2] <= most:
            return c


def draw(rng):
    kind = rng.choice(('increment',) * 6 + ('cutback', 'batch', 'gradient', 'response', 'coordinates'))
    if kind == 'increment':
        phase = rng.choice(('fcc12', 'fcc12', 'bcc24', 'bcc24', 'bcc48', 'bcc12ns'))
        c = _edges(rng, 8, 128, {'fcc12': 1 << 21, 'bcc24': 1 << 20, 'bcc48': 1 << 18, 'bcc12ns': 1 << 20}[phase])
        n = c[0] * c[1] * c[2]
        case = _increment('', c, phase, rng.choice(('fp64', 'mixed')), rng.randrange(3),
                          max(4, min(400, n // rng.choice((200, 1000, 4000)))),
                          rng.choice(('continuous', 'continuous', 'continuous', 'FWBW_difference')),
                          rng.choice(('tension', 'tension', 'shear')), 'all' if n <= 1 << 18 else 'output')
        del case['name']
        return case
    if kind == 'cutback':
        c = _edges(rng, 8, 48, 1 << 17)
        return {'kind': kind, 'c0': c[0], 'c1': c[1], 'c2': c[2], 'phase': rng.choice(('fcc12', 'bcc24')),
                'grains': rng.randrange(5, 100)}
    if kind == 'batch':
        return {'kind': kind, 'n': rng.randrange(4, 65), 'precision': rng.choice(('fp64', 'mixed')),
                'max_edge': rng.choice((12, 16, 24, 32))}
    if kind == 'gradient':
        c = _edges(rng, 6, 16, 1 << 12)
        return {'kind': kind, 'c0': c[0], 'c1': c[1], 'c2': c[2], 'grains': rng.randrange(4, 30),
                'increments': rng.randrange(1, 4)}
    c = _edges(rng, 9, 96, 1 << 19)
    if kind == 'response':
        return {'kind': kind, 'c0': c[0], 'c1': c[1], 'c2': c[2], 'phase': rng.choice(('fcc12', 'bcc24')),
                'grains': rng.randrange(5, 200)}
    return {'kind': kind, 'c0': c[0], 'c1': c[1], 'c2': c[2]}


# ------------------------------------------------------------------------------------ inputs
def _phase(name) -> Phase:
    if name == 'bcc12ns':   # the reference's 17-grains regression material
        return Phase.from_dict({'lattice': 'cI', 'mechanical': {
            'elastic': {'type': 'Hooke', 'C_11': 417.4e9, 'C_12': 242.4e9, 'C_44': 211.1e9},
            'plastic': {'type': 'phenopowerlaw', 'N_sl': [12], 'a_non-Schmid': [[0.1] * 6], 'dot_gamma_0_sl': [0.001],
                        'n_sl': [20], 'a_sl': [2.0], 'xi_0_sl': [405.8e6], 'xi_inf_sl': [872.9e6],
                        'h_0_sl-sl': [563.0e9], 'h_sl-sl': [1, 1.4, 1, 1.4, 1.4, 1.4, 1.4]}}})
    return {'fcc12': workloads.fcc_al, 'bcc24': workloads.bcc_24, 'bcc48': workloads.bcc_48}[name]()


def _cells(case):
    return case['c0'], case['c1'], case['c2']


def _rve(case, seed):
    cells = _cells(case)
    h = workloads.SIZE_1MM[0] / max(cells)     # cubic voxels
    return voronoi_rve(cells, tuple(h * c for c in cells), case['grains'], seed % (1 << 31))


def _batch_edges(case):
    edges = [e for e in (8, 12, 16, 24, 32) if e <= case['max_edge']]
    return [edges[k % len(edges)] for k in range(case['n'])]


def _numerics(case) -> Numerics:
    num = workloads.numerics_default()
    num.derivative = case.get('derivative', 'continuous')
    return num


def _load(case):
    return workloads.simple_shear_xy(100.0, 100) if case.get('load') == 'shear' else workloads.tension_x(100.0, 100)


def _pinned(*shape):
    t = torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    return t.numpy()


def _buffers(solver, fields):
    return {k: _pinned(solver.N, solver.lib.dmk_field_size(solver.ctx, {'xi_sl': 6, 'gamma_sl': 7}.get(k, 0)))
            for k in fields}


def _random_F(case, seed):
    """Deformation gradients of a tensile step with a fluctuation from voxel to voxel, voxel-major."""
    n = case['c0'] * case['c1'] * case['c2']
    F = np.eye(3) + np.diag([2e-3, -0.75e-3, -0.75e-3])
    rng = np.random.default_rng(seed)
    amplitude = 1e-2 if case['kind'] == 'coordinates' else 1e-4
    return F.reshape(1, 9) + amplitude * rng.standard_normal((n, 9))


def prepare(case, seed):
    kind = case['kind']
    st = {'case': dict(case)}
    if kind in ('increment', 'cutback'):
        rve, phase, num, lcs = _rve(case, seed), _phase(case['phase']), _numerics(case), _load(case)
        cls = SpectralBasic if kind == 'increment' else SpectralPolarization
        s = cls(rve.cells, rve.size, rve.material, rve.quaternions, phase, num, precision=case.get('precision', 'fp64'))
        drv = IncrementDriver(s, lcs)
        for _ in range(case.get('pre', 1)):
            drv.step()
        if kind == 'increment':
            s.checkpoint_save(0)
        else:
            s.forward(False, True, 1.0, 1.0, 99.0, lcs[0])      # the attempt that is cut back
            s.materialpoint_forward()
            s.solution()
        st.update(solver=s, driver=drv, at=drv.state(), load=lcs[0],
                  out=_buffers(s, FIELDS if case.get('fields', 'all') == 'all' else ('F', 'P', 'F_p', 'xi_sl')))
    elif kind == 'batch':
        # the batched workload's recipe; the edges go by the case alone, the rest by the seed
        rng, jobs = np.random.default_rng(seed), []
        for edge in _batch_edges(case):
            rve = voronoi_rve((edge,) * 3, workloads.SIZE_1MM, int(rng.integers(5, 101)), int(rng.integers(1 << 31)))
            axis = rng.standard_normal(3)
            lcs = workloads.tension_along(axis / np.linalg.norm(axis), 40.0, 40) if rng.random() < 0.5 else \
                workloads.simple_shear_xy(40.0, 40)
            jobs.append((rve, workloads.fcc_al(), lcs, workloads.numerics_default()))
        db = DeviceBatch(jobs, max_increments=1, precision=case['precision'])
        db.run_native()
        for s in db.solvers:
            s.checkpoint_save(0)
        total, ns = sum(s.N for s in db.solvers), db.solvers[0].n_slip
        st.update(batch=db, out={'F': _pinned(total, 9), 'P': _pinned(total, 9), 'xi_sl': _pinned(total, ns)})
    elif kind == 'gradient':
        num = adjoint.gradient_numerics(workloads.numerics_default())
        seq = adjoint.IncrementSequence(_rve(case, seed), adjoint.gradient_phase(workloads.fcc_al()),
                                        workloads.tension_x(50.0, 50), num, case['increments'], k=2)
        theta = np.array([31.0e6, 63.0e6, 75.0e6, 20.0, 2.25])
        goal = np.zeros((case['increments'], 3, 3))
        goal[:, 0, 0] = 1.0e8
        st.update(seq=seq, theta=theta, goal=torch.from_numpy(goal))
    else:
        phase = _phase(case.get('phase', 'fcc12'))
        rve = _rve({'grains': 4, **case}, seed)
        s = SpectralBasic(rve.cells, rve.size, rve.material, rve.quaternions, phase, workloads.numerics_default())
        F = _random_F(case, seed)
        if kind == 'coordinates':
            s.set_field('F_solver', F)
        else:
            s.checkpoint_save(0)
            st['out'] = _buffers(s, ('F_p', 'L_p', 'xi_sl', 'gamma_sl'))
        st.update(solver=s, F=F)
    return st


# ------------------------------------------------------------------------------------ one pass
def run(state):
    kind = state['case']['kind']
    if kind == 'increment':
        s, d = state['solver'], state['driver']
        s.checkpoint_restore(0)
        d.set_state(state['at'])
        recs = d.step()
        return {**{k: s.get_field(k, out=b) for k, b in state['out'].items()}, 'P_av': recs[-1].P_av}
    if kind == 'cutback':
        s = state['solver']
        s.forward(True, True, 0.5, 1.0, 99.0, state['load'])
        sol = s.solution()
        return {**{k: s.get_field(k, out=b) for k, b in state['out'].items()}, 'P_av': np.array(sol.P_av[:])}
    if kind == 'batch':
        db = state['batch']
        for s in db.solvers:
            s.checkpoint_restore(0)
        db.results = [[] for _ in db.jobs]
        db.run_native()
        at = 0
        for s in db.solvers:
            for k, b in state['out'].items():
                s.get_field(k, out=b[at:at + s.N])
            at += s.N
        return state['out']
    if kind == 'gradient':
        theta = torch.tensor(state['theta'], dtype=torch.float64, requires_grad=True)
        P = adjoint.stress_curve(theta, state['seq'])
        loss = (((P - state['goal']) * 1.0e-8) ** 2).mean()
        loss.backward()
        return {'P_av': P.detach(), 'gradient': theta.grad}
    s = state['solver']
    if kind == 'response':
        s.checkpoint_restore(0)
        P, P_av, C_volAvg, C_minMaxAvg, _ = s.constitutive_response(state['F'], 1.0)
        return {'P': P, 'P_av': P_av, 'C_volAvg': C_volAvg, 'C_minMaxAvg': C_minMaxAvg,
                **{k: s.get_field(k, out=b) for k, b in state['out'].items()}}
    s.update_coords()
    ip, nodes = s.get_coords()
    return {'ip': ip, 'nodes': nodes}


# ------------------------------------------------------------------------------------ work
NS = {'fcc12': 12, 'bcc12ns': 12, 'bcc24': 24, 'bcc48': 48}


def _update(ns):
    """Bytes and FP64 operations of one material-point update: the state before and after it, and
    the operations of 2.4 Newton iterations in each of 2.8 state iterations (the averages of the
    24-system benchmark)."""
    return 8.0 * (4 * 9 + 6 + 2 * ns + 5 * 9 + 6 + 2 * ns), 6.8 * (264 + 56 * ns) + 4.0 * (567 + 135 * ns) + 2.8 * (455 + 86 * ns)


def work(case):
    """An increment takes about ten evaluations of every voxel (each reads and writes its state and
    passes its stress through two transforms) and one consistent tangent."""
    kind = case['kind']
    n = case['c0'] * case['c1'] * case['c2'] if 'c0' in case else sum(e ** 3 for e in _batch_edges(case))
    b, f = _update(NS[case.get('phase', 'fcc12')])
    if kind == 'response':
        return {'bytes': n * (b + 4 * 72.0), 'flops': n * (f + 12e3)}
    if kind == 'coordinates':
        return {'bytes': n * (72.0 + 48.0), 'flops': n * 5.0 * 12 * math.log2(n)}
    evaluations = {'increment': 10, 'cutback': 10, 'batch': 9, 'gradient': 40 * case.get('increments', 1)}[kind]
    spectral_b, spectral_f = 4 * 72.0, 2 * 9 * 2.5 * math.log2(max(n, 2)) + 200
    extra = 0.5e6 * case.get('increments', 0)     # local Jacobians of the adjoint
    return {'bytes': n * (evaluations * (b + spectral_b) + 1000.0),
            'flops': n * (evaluations * (f + spectral_f) + 12e3 + extra)}


def tolerance(case):
    mixed = '_mixed' if case.get('precision') == 'mixed' else ''
    return TOLERANCES.get(case.get('phase', '') + mixed) or TOLERANCES[case['kind'] + mixed]


# Measured: the same increments with the microstructure shifted periodically along x by a distance
# that keeps the first voxel's grain (every transform, average and inner product then adds in another
# order), for the mixed form also against the FP64 form, and the sweeps and coordinates against
# exact(); about four times the largest difference over 30 drawn cases.  In FP64 the fields differ by
# up to 4e-12 (norm) and 4e-11 (largest), unless the last bit decides a voxel's Newton convergence
# test differently: such a voxel and those around it move by up to 5e-8, 1e-9 in the norm, and
# that is what the bounds allow for.  In the mixed form the transforms' 32 bits give up to 5e-7 (norm)
# and 6.5e-5 (largest, L_p of a nearly elastic voxel); with the non-Schmid material, nearly all elastic
# in its first increments, L_p is mostly what the Newton tolerance leaves: 3.2e-5 and 8e-3.  The
# gradient, at solver tolerances of 1e-11, differs by up to 2e-9.
TOLERANCES = {
    'increment': {'rel': 4e-9, 'max': 1e-6},
    'increment_mixed': {'rel': 2e-6, 'max': 3e-4},
    'bcc12ns_mixed': {'rel': 1.3e-4, 'max': 3.3e-2},
    'cutback': {'rel': 4e-9, 'max': 1e-6},
    'batch': {'rel': 4e-9, 'max': 1e-6},
    'batch_mixed': {'rel': 2e-6, 'max': 3e-4},
    'gradient': {'rel': 1e-8, 'max': 2e-8},
    'response': {'rel': 4e-9, 'max': 1e-6},
    'coordinates': {'rel': 3e-14, 'max': 1e-12},
}


# ------------------------------------------------------------------------------------ 64 bits
# The slip systems (direction, plane normal) in the order of the crystal tables, families {111}<110>
# (fcc) and {110}<111>, {112}<111> (bcc).
_FCC = '01-1111 -101111 1-10111 0-1-1-1-11 101-1-11 -110-1-11 0-111-1-1 -10-11-1-1 1101-1-1 011-11-1 10-1-11-1 -1-10-11-1'
_BCC = ('1-11011 1-1110-1 1-11-1-10 -1-110-1-1 -1-11101 -1-11-110 11101-1 111-101 1111-10 -1110-11 -111-10-1 -111110 '
        '1-1121-1 1-11-112 1-11121 -1-112-11 -1-11112 -1-11-121 11111-2 1111-21 111-211 -1111-12 -11112-1 -111211')


def _systems(text):
    rows = []
    for word in text.split():
        out, sign = [], 1
        for ch in word:
            if ch == '-':
                sign = -1
            else:
                out.append(sign * int(ch))
                sign = 1
        rows.append(out)
    return np.array(rows, float)


class _Material:
    """Phase constants as tensors: Schmid matrices, interaction matrix, cubic stiffness."""

    def __init__(self, name, device):
        p = _phase(name)
        rows = _systems(_FCC if name == 'fcc12' else _BCC)
        d = rows[:, :3] / np.linalg.norm(rows[:, :3], axis=1, keepdims=True)
        m = rows[:, 3:] / np.linalg.norm(rows[:, 3:], axis=1, keepdims=True)
        fam = np.repeat(np.arange(len(p.N_sl)), p.N_sl)

        def t(x):
            return torch.as_tensor(np.asarray(x, float), dtype=torch.float64, device=device)
        # the workloads' interaction values: 1 for systems of one plane, 1.4 otherwise
        self.h = t(np.where(np.abs(np.abs(m @ m.T) - 1.0) < 1e-9, 1.0, 1.4))
        self.P = t(d[:, :, None] * m[:, None, :])
        self.dg0, self.n, self.a = (t(np.array(v)[fam]) for v in (p.dot_gamma_0_sl, p.n_sl, p.a_sl))
        self.h0, self.xi0, self.xiinf = (t(np.array(v)[fam]) for v in (p.h_0_sl_sl, p.xi_0_sl, p.xi_inf_sl))
        C = np.zeros((3, 3, 3, 3))
        for i in range(3):
            for j in range(3):
                C[i, i, j, j] = p.C_11 if i == j else p.C_12
                if i != j:
                    C[i, j, i, j] = C[i, j, j, i] = p.C_44
        self.C = t(C)
        self.atol_xi, self.atol_gamma = p.atol_xi, p.atol_gamma

    def shear_rates(self, S, xi):
        """dot_gamma and its derivative with respect to tau of every system."""
        tau = torch.einsum('vij,sij->vs', S, self.P)
        r = tau.abs() / xi
        g = self.dg0 * r ** self.n * torch.sign(tau)
        return g, torch.where(tau == 0, torch.zeros_like(tau), g * self.n / torch.where(tau == 0, torch.ones_like(tau), tau))

    def hardening(self, gabs, xi):
        left = 1.0 - xi / self.xiinf
        return self.h0 * left.abs() ** self.a * torch.sign(left) * (gabs @ self.h.T)


class _Refused(Exception):
    """A voxel needs what this restatement leaves out (a substep)."""


def _norm(x):
    return x.flatten(1).norm(dim=1)


def _stress(mat, num, F, Fp0, xi, Lp, dt):
    """The Newton iteration for Lp of every voxel; returns Lp, S, Fp, P and |dot_gamma|."""
    nv, eye = F.shape[0], torch.eye(3, dtype=F.dtype, device=F.device)
    A = F @ torch.linalg.inv(Fp0)
    Lg, lo, dl = Lp.clone(), Lp.clone(), torch.zeros_like(Lp)
    step, old = torch.ones(nv, dtype=F.dtype, device=F.device), torch.full((nv,), np.inf, dtype=F.dtype, device=F.device)
    So, go = torch.zeros_like(F), torch.zeros_like(xi)
    todo = torch.arange(nv, device=F.device)
    for _ in range(num.N_iter_Lp_max):
        a, L, x = A[todo], Lg[todo], xi[todo]
        Fe = a @ (eye - dt * L)
        S = torch.einsum('ijkl,vkl->vij', mat.C, 0.5 * (Fe.mT @ Fe - eye))
        g, dg = mat.shear_rates(S, x)
        Lc = torch.einsum('vs,sij->vij', g, mat.P)
        R = L - Lc
        nR = _norm(R)
        tol = torch.clamp(num.eps_rel_Lp * torch.maximum(_norm(L), _norm(Lc)), min=num.eps_abs_Lp)
        So[todo], go[todo] = S, g.abs()
        better = nR < old[todo]
        done = nR < tol
        # Newton step where the residual fell, else a shorter step from the last accepted guess
        M = a.mT @ Fe
        Q = torch.einsum('sij,ijkl->skl', mat.P, mat.C)
        B = torch.einsum('vpj,sjb->vspb', M, Q)                 # (M Q_s), the change of tau_s per -dt dLp
        J = torch.einsum('vs,skl,vspb->vklpb', dt * dg, mat.P, B).reshape(-1, 9, 9) + torch.eye(9, dtype=F.dtype, device=F.device)
        new = torch.linalg.solve(J, -R.reshape(-1, 9)).reshape(-1, 3, 3)
        b3 = better[:, None, None]
        old[todo] = torch.where(better, nR, old[todo])
        lo[todo] = torch.where(b3, L, lo[todo])
        dl[todo] = torch.where(b3, new, dl[todo])
        step[todo] = torch.where(better, torch.ones_like(nR), num.r_linesearch_Lp * step[todo])
        nxt = torch.where(b3, L + dl[todo], lo[todo] + step[todo][:, None, None] * dl[todo])
        Lg[todo] = torch.where(done[:, None, None], L, nxt)
        todo = todo[~done]
        if todo.numel() == 0:
            break
    else:
        raise _Refused
    Fi = torch.linalg.inv(Fp0) @ (eye - dt * Lg)
    Fp = torch.linalg.inv(Fi)
    P = F @ Fi @ So @ Fi.mT
    return Lg, So, Fp / torch.linalg.det(Fp)[:, None, None] ** (1.0 / 3.0), P, go


def _sweep(mat, num, F, st, dt):
    """One evaluation of every voxel from the start values Fp0, S0 = 0, xi0 and gamma0 = 0; Lp is the
    warm start and is kept for the next one."""
    ns = st['xi0'].shape[1]
    x0 = torch.cat([st['xi0'], torch.zeros_like(st['xi0'])], 1)
    tol = torch.cat([torch.full((ns,), mat.atol_xi), torch.full((ns,), mat.atol_gamma)]).to(F)
    z = torch.zeros_like(st['xi0'])
    last = torch.cat([mat.hardening(z, st['xi0']), z], 1)
    last2 = torch.zeros_like(last)
    x = x0 + last * dt
    todo = torch.arange(F.shape[0], device=F.device)
    P = torch.zeros_like(F)
    for it in range(1, num.N_iter_state_max + 1):
        Lp, S, Fp, Pn, gabs = _stress(mat, num, F[todo], st['Fp0'][todo], x[todo][:, :ns], st['Lp'][todo], dt)
        st['Lp'][todo], st['Fp'][todo], P[todo] = Lp, Fp, Pn
        rate = torch.cat([mat.hardening(gabs, x[todo][:, :ns]), gabs], 1)
        l1 = last[todo]
        l2 = last2[todo] if it > 1 else torch.zeros_like(l1)
        d01, d12, d22 = (rate * l1).sum(1), ((rate - l1) * (l1 - l2)).sum(1), ((l1 - l2) ** 2).sum(1)
        damp = (torch.minimum(d01, d12) < 0) & (d22 > 0)
        zeta = torch.where(damp, 0.75 + 0.25 * torch.tanh(2.0 + 4.0 * d12 / torch.where(d22 > 0, d22, torch.ones_like(d22))),
                           torch.ones_like(d22))[:, None]
        rate = rate * zeta + l1 * (1.0 - zeta)
        r = x[todo] - x0[todo] - rate * dt
        new = x[todo] - r
        last2[todo], last[todo], x[todo] = l1, rate, new
        conv = (r.abs() <= torch.maximum(tol, num.eps_rel_state * new.abs())).all(1)
        todo = todo[~conv]
        if todo.numel() == 0:
            break
    st['x'] = x
    return P


def _orientations(rve, device):
    q = rve.quaternions
    w, x, y, z = (torch.as_tensor(q[:, k], dtype=torch.float64, device=device) for k in range(4))
    qq = w * w - (x * x + y * y + z * z)
    O = torch.stack([qq + 2 * x * x, 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), qq + 2 * y * y, 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), qq + 2 * z * z], 1).reshape(-1, 3, 3).mT   # passive
    O = O / torch.linalg.det(O)[:, None, None] ** (1.0 / 3.0)
    return O[torch.as_tensor(rve.material, dtype=torch.int64, device=device)]


def _start(mat, rve, device):
    O = _orientations(rve, device)
    n = O.shape[0]
    return {'Fp0': O, 'Fp': O.clone(), 'Lp': torch.zeros_like(O), 'xi0': mat.xi0.expand(n, -1).clone()}


def _columns(T):
    """(n, 3, 3) in the voxel-major column-major layout of the fields."""
    return T.mT.reshape(-1, 9).cpu()


def _outputs(F, P, st, fields):
    ns = st['xi0'].shape[1]
    got = {'F': _columns(F), 'P': _columns(P), 'F_p': _columns(st['Fp']), 'L_p': _columns(st['Lp']),
           'xi_sl': st['x'][:, :ns].cpu(), 'gamma_sl': st['x'][:, ns:].cpu()}
    return {k: got[k] for k in fields}


def _first_increment(case, seed, device):
    """The first increment of the load case: Anderson-accelerated fixed point of the basic scheme."""
    rve, num, mat = _rve(case, seed), _numerics(case), _Material(case['phase'], device)
    cells, size = rve.cells, rve.size
    n = math.prod(cells)
    st = _start(mat, rve, device)
    lc, dt = _load(case)[0], 1.0
    eye = torch.eye(3, dtype=torch.float64, device=device)
    # elastic medium of the undeformed state: crystal stiffness in the sample frame (O^T)
    O = st['Fp0']
    first = torch.einsum('mi,nj,pk,ql,mnpq->ijkl', O[0], O[0], O[0], O[0], mat.C)
    mean = torch.zeros_like(first)
    for part in torch.split(O, 8192):
        mean += torch.einsum('vmi,vnj,vpk,vql,mnpq->ijkl', part, part, part, part, mat.C)
    mean /= n
    # masked compliance over the stress-controlled components
    free = [(i, j) for i in range(3) for j in range(3) if not lc.stress_mask[i, j]]
    S = torch.zeros((3, 3, 3, 3), dtype=torch.float64, device=device)
    if free:
        inv = torch.linalg.inv(torch.stack([torch.stack([mean[i + k] for k in free]) for i in free]))
        for a, i in enumerate(free):
            for b, k in enumerate(free):
                S[i + k] = inv[a, b]
    rate = torch.as_tensor(np.where(lc.deformation_mask, 0.0, lc.deformation), dtype=torch.float64, device=device)
    F_aim = eye + rate * dt
    P_aim, fixed = torch.zeros_like(eye), torch.as_tensor(~lc.stress_mask, device=device)
    # frequencies (the Nyquist frequency of an even edge is zero), arrays indexed [z, y, x]
    def freq(c, L, half):
        k = np.fft.rfftfreq(c, 1.0 / c) if half else np.fft.fftfreq(c, 1.0 / c)
        k = np.where((c % 2 == 0) & (np.abs(k) == c // 2), 0.0, k)
        return torch.as_tensor(2 * np.pi * k / L, dtype=torch.float64, device=device)
    ax, ay, az = freq(cells[0], size[0], True), freq(cells[1], size[1], False), freq(cells[2], size[2], False)
    a = torch.stack(torch.broadcast_tensors(ax[None, None, :], ay[None, :, None], az[:, None, None]), -1)
    K = torch.einsum('ljmk,zyxj,zyxk->zyxlm', first, a, a)
    null = torch.linalg.det(K / mat.C[0, 0, 0, 0]).abs() <= 1e-200
    Ki = torch.linalg.inv(torch.where(null[..., None, None], eye, K))
    Ki = torch.where(null[..., None, None], torch.zeros_like(Ki), Ki)
    sp = [size[i] / cells[i] for i in range(3)]
    rescale = [1.0] * 3                                        # geomSize / scaledGeomSize, 'grid+size'
    lo, hi = sp.index(min(sp)), sp.index(max(sp))
    for j in range(3):
        if j != lo and j != hi:
            rescale = [size[j] / cells[j]] * 3
    w = torch.full((cells[0] // 2 + 1,), 2.0, dtype=torch.float64, device=device)
    w[0] = w[-1] = 1.0
    ar = a * torch.as_tensor(rescale, dtype=torch.float64, device=device)

    F = F_aim.expand(n, 3, 3).clone()
    dX, dR, count, m = {}, {}, 0, num.anderson_m
    Rprev = step = None
    for iteration in range(num.N_iter_max + 1):
        P = _sweep(mat, num, F, st, dt)
        P_av = P.mean(0)
        d = P_av - P_aim
        dF = torch.einsum('ijkl,kl->ij', S, d)
        F_aim = F_aim - dF
        err_BC = float(d[fixed].abs().max()) if bool(fixed.any()) else 0.0
        Ph = torch.fft.rfftn(P.reshape(cells[2], cells[1], cells[0], 3, 3), dim=(0, 1, 2))
        div = torch.einsum('zyxlm,zyxm->zyxl', Ph, ar.to(Ph.dtype))
        err_div = math.sqrt(float((div.abs() ** 2).sum(-1).mul(w).sum())) / n
        u = torch.einsum('zyxlm,zyxm->zyxl', Ki.to(Ph.dtype), torch.einsum('zyxlm,zyxm->zyxl', Ph, a.to(Ph.dtype)))
        G = u[..., :, None] * a.to(Ph.dtype)[..., None, :]
        G[0, 0, 0] = dF.to(Ph.dtype) * n
        R = torch.fft.irfftn(G, s=(cells[2], cells[1], cells[0]), dim=(0, 1, 2)).reshape(n, 3, 3)
        top = float(P_av.abs().max())
        if iteration >= num.N_iter_min and err_div < max(top * num.eps_rel_div, num.eps_abs_div) and \
                err_BC < max(top * num.eps_rel_P, num.eps_abs_P):
            return F, P, st, P_av
        X = F - R
        if count:
            new = (count - 1) % m
            dR[new] = R - Rprev
            slots = [q % m for q in range(count - min(count, m), count)]
            while slots:                 # least squares; the oldest pair goes while it is dependent
                Gm = np.array([[float((dR[i] * dR[j]).sum()) for j in slots] for i in slots])
                low, ok = np.zeros_like(Gm), True
                for i in range(len(slots)):
                    for j in range(i + 1):
                        v = Gm[i, j] - low[i, :j] @ low[j, :j]
                        if i == j and not v > 1e-13 * Gm.diagonal().max():
                            ok = False
                            break
                        low[i, j] = math.sqrt(v) if i == j else v / low[j, j]
                    if not ok:
                        break
                if ok:
                    b = np.array([float((dR[i] * R).sum()) for i in slots])
                    for q, g in zip(slots, np.linalg.solve(low.T, np.linalg.solve(low, b))):
                        X = X - g * (dX[q] - dR[q])
                    break
                slots = slots[1:]
        dX[count % m] = X - F
        Rprev, F, count = R, X, count + 1
    raise _Refused


def _coordinates(case, seed):
    cells = _cells(case)
    h = workloads.SIZE_1MM[0] / max(cells)
    F = _random_F(case, seed).reshape(cells[2], cells[1], cells[0], 3, 3).swapaxes(-1, -2)     # [z, y, x, i, j]
    mean = F.mean((0, 1, 2))
    # the Nyquist frequency of an even edge counts as positive; half spectrum along x
    k = [np.fft.fftfreq(c, 1.0 / c) if i else np.fft.rfftfreq(c, 1.0 / c) for i, c in enumerate(cells)]
    k = [2 * np.pi * np.where(np.abs(v) == c / 2, np.abs(v), v) / (h * c) for c, v in zip(cells, k)]
    a = np.stack(np.broadcast_arrays(k[0][None, None, :], k[1][None, :, None], k[2][:, None, None]), -1)
    a2 = (a * a).sum(-1)
    a2[0, 0, 0] = 1.0
    uh = -1j * np.einsum('zyxij,zyxj->zyxi', np.fft.rfftn(F, axes=(0, 1, 2)), a) / a2[..., None]
    uh[0, 0, 0] = 0.0
    u = np.fft.irfftn(uh, s=cells[::-1], axes=(0, 1, 2))
    grid = np.stack(np.meshgrid(*[np.arange(c + 1.0) for c in cells[::-1]], indexing='ij')[::-1], -1)
    ip = u + (grid[:-1, :-1, :-1] + 0.5) * h @ mean.T
    around = sum(np.roll(u, s, (0, 1, 2)) for s in np.ndindex(2, 2, 2)) / 8.0
    nodes = np.pad(around, ((0, 1),) * 3 + ((0, 0),), mode='wrap') + grid * h @ mean.T
    return {'ip': ip.reshape(-1, 3), 'nodes': nodes.reshape(-1, 3)}


def exact(case, seed):
    kind = case['kind']
    if kind == 'coordinates':
        return _coordinates(case, seed)
    device = torch.device('cuda' if torch.cuda.is_available() else 'cpu')
    try:
        if kind == 'response':
            rve, mat = _rve(case, seed), _Material(case['phase'], device)
            st = _start(mat, rve, device)
            F = torch.as_tensor(_random_F(case, seed), device=device).reshape(-1, 3, 3).mT.contiguous()
            P = _sweep(mat, workloads.numerics_default(), F, st, 1.0)
            got = _outputs(F, P, st, ('P', 'F_p', 'L_p', 'xi_sl', 'gamma_sl'))
            return {**got, 'P_av': P.mean(0).mT.reshape(9).cpu(), 'C_volAvg': None, 'C_minMaxAvg': None}
        if kind == 'increment' and case['pre'] == 0 and case['derivative'] == 'continuous' and \
                case['phase'] in ('fcc12', 'bcc24') and math.prod(_cells(case)) <= 1 << 18:
            F, P, st, P_av = _first_increment(case, seed, device)
            fields = FIELDS if case['fields'] == 'all' else ('F', 'P', 'F_p', 'xi_sl')
            return {**_outputs(F, P, st, fields), 'P_av': P_av.cpu()}
    except _Refused:
        pass
    return None
