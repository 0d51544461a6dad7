"""The work a user of this package has it do, as cases that can be timed.

Every case is one pass through the public entry points: the particle sort with and
without its payload, the steady-state re-sort with the move stage fused in, the DSMC
step, and the move and collision stages on their own.  The sizes are those of the
benchmark configurations (`project_aether_b200/workloads.py`), of the command-line
benchmark's default and of the tests; `draw` spreads over the ranges between them.
"""

import math

import torch

import project_aether_b200 as pa
from project_aether_b200 import ntc_collide, workloads

RUN_SEED = 1234
VHS_EXPONENT = 0.46        # 2 - 2 omega of argon-like gases (omega = 0.77)
VHS_COEFFICIENT = 1.7      # sigma_T g at unit relative speed, thermal speed 1
MAJORANT = VHS_COEFFICIENT * 3.0 ** VHS_EXPONENT
PAIR_SHARE = 0.075         # candidate pairs per particle and step


def _case(name, kind, n, cells, density='uniform', drift=0.0, extent=(1.0, 1.0, 1.0)):
    case = {'kind': kind, 'n': n, 'nx': cells[0], 'ny': cells[1], 'nz': cells[2],
            'ex': extent[0], 'ey': extent[1], 'ez': extent[2], 'density': density, 'drift': drift}
    return dict(case, name=name) if name else case


def listed():
    return [
        # Binning only (permutation, counts, starts): the entry point the reference exports.
        # A unit-test-sized call: all latency and launches.
        _case('sort_5k', 'sort', 5000, (25, 25, 16), extent=(1.0, 1.0, 0.64)),
        # The command-line benchmark's default: few cells with four hundred particles each.
        _case('sort_4m_10k_cells', 'sort', 4_000_000, (25, 25, 16), extent=(1.0, 1.0, 0.64)),
        _case('sort_16m_128', 'sort', 1 << 24, (128, 128, 128), drift=5.0),
        # Binning with the payload in sorted order: the four configurations whose input
        # arrives in random order, from the smallest to the largest that one GPU is given.
        _case('gather_1m_64', 'gather', 1 << 20, (64, 64, 64)),
        _case('gather_16m_128', 'gather', 1 << 24, (128, 128, 128), drift=5.0),
        _case('gather_64m_hypersonic', 'gather', 1 << 26, (256, 128, 128), 'hypersonic'),
        _case('gather_256m_512', 'gather', 1 << 28, (512, 256, 256)),
        # A time-stepping loop's re-sort: the state starts cell-sorted, moves, is sorted again.
        _case('resort_128m_256', 'resort', 1 << 27, (256, 256, 256)),
        # A whole DSMC step: a small simulation with an odd particle count, and a large one.
        _case('step_200k', 'step', 200_003, (32, 32, 16)),
        _case('step_16m_128', 'step', 1 << 24, (128, 128, 128)),
        # The move and collision stages as entry points of their own.
        _case('push_16m', 'push', 1 << 24, (128, 128, 128)),
        _case('collide_16m_128', 'collide', 1 << 24, (128, 128, 128)),
    ]


# Particle counts and particles per cell of each kind of call.
_RANGES = {
    'sort': ((1_000, 30_000_000), (2, 400)),
    'gather': ((3_000, 120_000_000), (2, 400)),
    'resort': ((100_000, 60_000_000), (4, 64)),
    'step': ((20_000, 30_000_000), (4, 64)),
    'push': ((10_000, 60_000_000), (4, 64)),
    'collide': ((20_000, 30_000_000), (4, 64)),
}


def draw(rng):
    kind = rng.choice(('sort', 'sort', 'gather', 'gather', 'gather', 'resort', 'step', 'step',
                       'push', 'collide'))
    (n_lo, n_hi), (ppc_lo, ppc_hi) = _RANGES[kind]
    n = int(math.exp(rng.uniform(math.log(n_lo), math.log(n_hi))))
    density = 'hypersonic' if kind in ('sort', 'gather') and rng.random() < 0.3 else 'uniform'
    if density == 'hypersonic':
        ppc_hi = 64
    per_cell = math.exp(rng.uniform(math.log(ppc_lo), math.log(ppc_hi)))
    cells = min(max(1.0, n / per_cell), float(1 << 25))
    side = cells ** (1.0 / 3.0)
    stretch = rng.uniform(1.0, 2.0)
    nx = max(1, round(side * stretch))
    ny = max(1, round(side))
    nz = max(1, round(cells / (nx * ny)))
    extent = rng.choice(((1.0, 1.0, 1.0), (1.0, 1.0, 0.64), (1.2, 1.0, 0.8)))
    if density == 'hypersonic':
        extent = (1.0,) + extent[1:]
    return _case(None, kind, n, (nx, ny, nz), density, rng.choice((0.0, 0.0, 5.0)), extent)


def _grid(case):
    return pa.CellGrid((0.0, 0.0, 0.0), (case['ex'], case['ey'], case['ez']),
                       (case['nx'], case['ny'], case['nz']))


def _dt(case):
    """About five percent of the particles leave their cell in a step."""
    return 0.021 / max(case['nx'] / case['ex'], case['ny'] / case['ey'], case['nz'] / case['ez'])


def _cell_sorted(grid, x, y, z, velocity):
    """The particles in the order of their cells, as a time step leaves them."""
    cell = torch.zeros(x.numel(), dtype=torch.int32, device=x.device)
    for c, hi, cells in ((z, grid.hi[2], grid.cells[2]), (y, grid.hi[1], grid.cells[1]),
                         (x, grid.hi[0], grid.cells[0])):
        cell = cell * cells + (c * (cells / hi)).to(torch.int32).clamp_(0, cells - 1)
    order = torch.argsort(cell, stable=True)
    sorted_velocity = torch.zeros_like(velocity)
    for k in range(3):
        sorted_velocity[k, :order.numel()] = velocity[k, order]
    return x[order], y[order], z[order], sorted_velocity


def _collision_params(case, seed, step):
    per_cell = case['n'] / (case['nx'] * case['ny'] * case['nz'])
    factor = 2.0 * PAIR_SHARE / (max(per_cell, 1.0) * MAJORANT)
    return pa.CollisionParams(factor, VHS_COEFFICIENT, VHS_EXPONENT, RUN_SEED ^ seed, step)


def prepare(case, seed):
    grid = _grid(case)
    cells = grid.num_cells
    work = workloads.Workload('case', case['n'], grid, case['density'], case['drift'])
    x, y, z, velocity = workloads.make_particles(work, 'cuda', seed=seed)
    state = {'case': case, 'grid': grid, 'seed': seed, 'step': 0}
    kind = case['kind']
    if kind in ('resort', 'step'):
        x, y, z, velocity = _cell_sorted(grid, x, y, z, velocity)
    if kind in ('step', 'collide'):
        state['library'] = ntc_collide.load_library()
        state['sigma'] = torch.full((cells,), MAJORANT, device='cuda')
    if kind == 'step':
        state['particles'] = pa.GpuDsmcState([x, y, z], velocity, state['sigma'], case['n'])
    elif kind == 'collide':
        # The sort's cell starts for uniform particles; the velocities are already "sorted".
        gen = torch.Generator(device='cuda').manual_seed(seed + 1)
        cell = torch.randint(0, cells, (case['n'],), device='cuda', generator=gen)
        start = torch.zeros(cells + 1, dtype=torch.int32, device='cuda')
        start[1:] = torch.cumsum(torch.bincount(cell, minlength=cells), 0)
        state.update(velocity=velocity, start=start,
                     collisions=torch.zeros(cells, dtype=torch.int32, device='cuda'))
    else:
        state.update(positions=(x, y, z), velocity=velocity, sets=[None, None])
    return state


def run(state):
    case, grid = state['case'], state['grid']
    step = state['step']
    state['step'] = step + 1
    seed = workloads.step_seed(RUN_SEED ^ state['seed'], step)
    kind = case['kind']
    if kind == 'sort':
        return tuple(pa.sort_particles_by_cell(*state['positions'], grid, seed))
    if kind == 'gather':
        out = pa.sort_and_gather_particles(*state['positions'], state['velocity'], grid, seed)
        return (*out.order, *out.positions, out.velocity)
    if kind == 'resort':
        # The sorted state of a step is the next step's input; two sets of arrays alternate.
        out = pa.sort_and_gather_particles(*state['positions'], state['velocity'], grid, seed,
                                           out=state['sets'][step % 2],
                                           push=(_dt(case), grid.lo, grid.hi))
        state['sets'][step % 2] = out
        state['positions'], state['velocity'] = out.positions, out.velocity
        return (*out.order, *out.positions, out.velocity)
    if kind == 'step':
        particles = state['particles']
        stats = pa.gpu_dsmc_step(particles, state['library'], grid,
                                 _collision_params(case, state['seed'], step), _dt(case))
        return (*particles.positions, particles.velocity, particles.sigma_g_max,
                stats.cell_counts, stats.collisions)
    if kind == 'push':
        rows = [state['velocity'][k, :case['n']] for k in range(3)]
        pa.fused_particle_push(state['positions'], rows, _dt(case), grid.lo, grid.hi)
        return (*state['positions'], state['velocity'])
    pa.collide(state['library'], state['velocity'], state['start'], state['sigma'],
               state['collisions'], case['n'], _collision_params(case, state['seed'], step))
    return state['velocity'], state['sigma'], state['collisions']


def work(case):
    """Each input read once, each output written once."""
    n, cells = case['n'], case['nx'] * case['ny'] * case['nz']
    return {'bytes': {
        'sort': 12 * n + 8 * n + 8 * cells,
        'gather': 24 * n + 32 * n + 8 * cells,
        'resort': 24 * n + 32 * n + 8 * cells,
        # x and v in and out; majorant in and out, counts and accepted collisions out.
        'step': 24 * n + 24 * n + 16 * cells,
        'push': 24 * n + 24 * n,
        # Velocities in and out, starts in, majorant in and out, accepted collisions out.
        'collide': 12 * n + 12 * n + 16 * cells,
    }[case['kind']], 'flops': 0}


def tolerance(case):
    """The sort and the move are defined to the bit.  The collision stage contains powf, sinf
    and cosf: its pair arithmetic in 32 bits against 64 bits, at the listed share of candidate
    pairs, moves the velocities by 2.8e-8 (2-norm) and by at most 1.7e-6 of their size, and
    turns none of 600,000 acceptances (a turned one would show in the accepted counts)."""
    if case['kind'] in ('step', 'collide'):
        return {'rel': 1.2e-7, 'max': 7e-6, 'differ': 1e-6}
    return 'exact'
