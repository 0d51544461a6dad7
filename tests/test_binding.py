"""The native binding takes the plain form of a call; every other form goes through the Python code
and comes out the same, errors included.  Without a binding that fits, all calls do."""

import os
import subprocess
import sys

import numpy as np
import pytest
import torch

import project_aether_b200 as pa
from project_aether_b200 import _native, ntc_collide

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
N, CELLS = 5_003, (8, 7, 6)
GRID = pa.CellGrid((0., 0., 0.), (1., 1., 0.5), CELLS)


@pytest.fixture(scope='module')
def binding():
    _native.load_library()
    return _native.binding


def _state(device, n=N, seed=0):
    gen = torch.Generator().manual_seed(seed)
    pos = [torch.rand(n, generator=gen).to(device) for _ in range(3)]
    vel = torch.zeros((3, -(-n // 4) * 4))
    vel[:, :n] = torch.randn((3, n), generator=gen)
    return pos, vel.to(device)


def test_host_tensors_and_wrong_types_are_left_to_the_python_code(binding):
    pos, vel = _state('cpu')
    assert binding.sort(*pos, GRID, 1, {}) is None
    assert binding.gather(*pos, vel, GRID, 1, 0, None, None, None, {}) is None
    assert binding.collide(vel, pos[0], pos[0], pos[0], N, 1.0, 1.0, 0.5, 1, 1) is None
    assert binding.sort(1, None, 'x', GRID, 1, {}) is None
    assert binding.sort(*pos, GRID, 1) is None
    with pytest.raises(TypeError):
        binding.bind(1, 2)


def _flat(result):
    if isinstance(result, pa.SortResult):
        return list(result)
    return [*result.order, *result.positions, result.velocity]


def _count_plain(monkeypatch, name):
    """How many calls of `name` the binding takes, from here on."""
    taken = []
    inner = getattr(_native.binding, name)

    class Watched:
        def __getattr__(self, other):
            if other != name:
                return getattr(real, other)

            def call(*args):
                out = inner(*args)
                taken.append(out is not None)
                return out
            return call

    real = _native.binding
    monkeypatch.setattr(_native, 'binding', Watched())
    return taken


def _sort_forms(pos, vel):
    """(positions, grid, seed, whether the call is a plain one)"""
    x, y, z = pos
    wide = torch.stack([x, x], 1)
    yield (x, y, z), GRID, 77, True
    yield (x, y, z), pa.CellGrid([0, 0, 0], [1, 1, 0.5], list(CELLS)), 77, True
    yield (wide[:, 0], y, z), GRID, 77, False
    yield (x.view(-1, 1), y.view(1, -1), z), GRID, 77, False
    yield (x, y, z), pa.CellGrid(np.zeros(3), np.array([1., 1., 0.5]), CELLS), 77, False
    yield (x, y, z), GRID, np.int64(77), False
    yield (x, y, z), type('Grid', (pa.CellGrid,), {})(*GRID), 77, False
    yield tuple(torch.nn.Parameter(t) for t in pos), GRID, 77, True


@pytest.mark.gpu
def test_every_form_of_the_sort_comes_out_the_same(cuda, binding, monkeypatch):
    pos, vel = _state(cuda)
    want = pa.sort_particles_by_cell(*pos, GRID, 77, ix_offset=0, nx_local=CELLS[0])  # not plain
    taken = _count_plain(monkeypatch, 'sort')
    for positions, grid, seed, plain in _sort_forms(pos, vel):
        got = pa.sort_particles_by_cell(*positions, grid, seed)
        assert taken.pop() is plain
        assert isinstance(got, pa.SortResult)
        for g, w in zip(got, want):
            assert g.dtype == w.dtype and g.shape == w.shape and torch.equal(g, w)


@pytest.mark.gpu
@pytest.mark.parametrize('push', [None, (0.01, (0., 0., 0.), (1., 1., 0.5)), (0.01, [0, 0, 0], [1, 1, 0.5]),
                                  (np.float32(0.01), (0., 0., 0.), (1., 1., 0.5))])
def test_every_form_of_the_gather_comes_out_the_same(cuda, binding, monkeypatch, push):
    pos, vel = _state(cuda)
    want = pa.sort_and_gather_particles(*pos, vel, GRID, 5, push=push, ix_offset=0, nx_local=CELLS[0])
    taken = _count_plain(monkeypatch, 'gather')
    plain_push = push is None or isinstance(push[0], float)
    spare = pa.sort_and_gather_particles(*pos, vel, GRID, 9)
    taken.clear()
    strided = torch.zeros((3, 2 * vel.shape[1]), device=cuda)
    strided[:, ::2] = vel
    rows = torch.zeros((3, N + 101), device=cuda)
    rows[:, :N] = vel[:, :N]
    for velocity, plain, extra in ((vel, True, {}), (vel, True, {'path': 2}), (vel, True, {'padded_out': N + 5}),
                                   (vel, True, {'out': spare}), (strided[:, ::2], False, {}), (rows[:, :N], True, {})):
        got = pa.sort_and_gather_particles(*pos, velocity, GRID, 5, push=push, **extra)
        assert taken.pop() is (plain and plain_push)
        flat = _flat(got)
        for k, (g, w) in enumerate(zip(flat, _flat(want))):
            if k == 7:
                assert torch.equal(g[:, :N], w[:, :N]) and not g[:, N:].any()
            else:
                assert g.dtype == w.dtype and torch.equal(g, w)
        if 'out' in extra:
            assert all(g is s for g, s in zip(flat, _flat(spare)))
        else:
            assert not any(t._is_view() for t in flat)


@pytest.mark.gpu
def test_errors_are_those_of_the_python_code(cuda, binding):
    pos, vel = _state(cuda)
    x, y, z = pos
    for bad in ((x.double(), y, z), (x[:-1], y, z), (x.cpu(), y, z), (x, y, None)):
        with pytest.raises(ValueError, match='float32 CUDA'):
            pa.sort_particles_by_cell(*bad, GRID, 1)
    with pytest.raises(ValueError, match='32 bits|bits'):
        pa.sort_particles_by_cell(x, y, z, pa.CellGrid((0., 0., 0.), (1., 1., 1.), (1024, 1024, 64)), 1)
    for bad in (vel.double(), vel[:2], vel[:, :100], vel.cpu()):
        with pytest.raises(ValueError, match='Velocity'):
            pa.sort_and_gather_particles(x, y, z, bad, GRID, 1)
    with pytest.raises(ValueError, match='padded_out'):
        pa.sort_and_gather_particles(x, y, z, vel, GRID, 1, padded_out=N - 1)
    with pytest.raises(ValueError, match='does not match'):
        pa.sort_and_gather_particles(x, y, z, vel, GRID, 1,
                                     out=pa.sort_and_gather_particles(x[1:], y[1:], z[1:], vel, GRID, 1))
    with pytest.raises(AttributeError):
        pa.sort_particles_by_cell(x, y, z, tuple(GRID), 1)
    with pytest.raises(ZeroDivisionError):
        pa.sort_particles_by_cell(x, y, z, pa.CellGrid((0., 0., 0.), (0., 1., 1.), CELLS), 1)


@pytest.mark.gpu
def test_watched_calls_are_left_to_the_python_code(cuda, binding):
    """Modes and transforms that see the operations of a call; the workspace is there."""
    from torch.utils._python_dispatch import TorchDispatchMode
    from project_aether_b200 import particle_sort
    pos, vel = _state(cuda)
    pa.sort_particles_by_cell(*pos, GRID, 1)
    call = lambda *p: binding.sort(*p, GRID, 1, particle_sort._workspaces)
    assert call(*pos) is not None

    class Watch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    with Watch():
        assert call(*pos) is None
    seen = []
    batch = torch.stack([pos[0], pos[0]])

    def one(t):
        seen.append(call(t, pos[1], pos[2]))
        return t
    torch.vmap(one)(batch)
    assert seen == [None]
    assert call(torch._neg_view(pos[0]), pos[1], pos[2]) is None


@pytest.mark.gpu
def test_collide_through_the_binding_equals_the_plain_call(cuda, binding):
    pos, vel = _state(cuda)
    order = pa.sort_particles_by_cell(*pos, GRID, 3)
    library = ntc_collide.load_library()
    params = ntc_collide.CollisionParams(1e-3, 1.0, 0.5, 11, 2)
    results = []
    for p in (params, params._replace(step=np.int64(2))):  # the second is not plain
        v, sigma = vel.clone(), torch.ones(GRID.num_cells, device=cuda)
        accepted = torch.zeros(GRID.num_cells, dtype=torch.int32, device=cuda)
        plain = binding.collide(v.clone(), order.cell_start, sigma.clone(), accepted.clone(), N, *p)
        assert plain is (True if isinstance(p.step, int) else None)
        ntc_collide.collide(library, v, order.cell_start, sigma, accepted, N, p)
        results.append((v, sigma, accepted))
    for a, b in zip(*results):
        assert torch.equal(a, b)


# ---- loading: the library alone serves every call ----

_LOAD = """
import sys, types, warnings
sys.modules['project_aether_b200._binding'] = {module}
warnings.simplefilter('ignore')
from project_aether_b200 import _native, ntc_collide
library = _native.load_library()
assert library is _native.load_library() and library is not None
assert library.AetherSortWorkspaceBytes(1000, 100, 0) > 0
assert _native.binding is None and _native.bound_library is None
try:  # no binding: a call gets as far as the Python code's own checks
    ntc_collide.collide(library, types.SimpleNamespace(dim=lambda: 1), *[None] * 4, ntc_collide.CollisionParams(*[1] * 5))
except ValueError as e:
    assert 'contiguous' in str(e)
"""


def _child(code, **env):
    return subprocess.run([sys.executable, '-c', code], cwd=ROOT, env={**os.environ, **env}, capture_output=True,
                          text=True)


@pytest.mark.parametrize('module', ['None',  # none, or one that does not load
                                    "types.SimpleNamespace(bind=None)",
                                    "types.SimpleNamespace(bind=None, built_for='torch 1.0')"])
@pytest.mark.parametrize('named', [False, True])
def test_the_library_loads_without_a_binding_that_fits(module, named):
    env = {'AETHER_SORT_LIBRARY': _native.LIBRARY_PATH} if named else {}
    done = _child(_LOAD.format(module=module), **env)
    assert done.returncode == 0, done.stderr


def test_the_binding_is_there_before_the_library_it_is_bound_to():
    """Another thread may call at any line of the loading: where it finds the bound library, it finds
    the binding."""
    done = _child("""
import sys
from project_aether_b200 import _native
def look(frame, event, arg):
    if frame.f_code is not _native.load_library.__code__:
        return None
    assert _native.bound_library is None or _native.binding is not None, frame.f_lineno
    return look
sys.settrace(look)
_native.load_library()
sys.settrace(None)
assert _native.binding is not None and _native.bound_library is _native.load_library()
""")
    assert done.returncode == 0, done.stderr


def test_a_binding_for_another_pytorch_is_stale(tmp_path, monkeypatch):
    build = pytest.importorskip('project_aether_b200.build')
    source, target = tmp_path / 'binding.cpp', tmp_path / '_binding.so'
    source.write_text('')
    monkeypatch.setattr(build, 'BINDING', str(target))
    assert build._binding_stale([str(source)])
    target.write_bytes(b'\0' + build.binding_abi().encode() + b'\0')
    assert not build._binding_stale([str(source)])
    target.write_bytes(b'\0' + build.binding_abi().replace('torch ', 'torch 1').encode() + b'\0')
    assert build._binding_stale([str(source)])


def test_the_library_is_built_before_a_binding_that_cannot_be(tmp_path, monkeypatch):
    from project_aether_b200 import build
    ran = []

    def run(cmd, verbose):
        ran.append(cmd[0])
        if 'binding.cpp' in ' '.join(cmd):
            raise RuntimeError('no Python.h')
    monkeypatch.setattr(build, '_run', run)
    monkeypatch.setattr(build, '_nvcc', lambda: 'nvcc')
    with pytest.warns(RuntimeWarning, match='no Python.h'):
        assert build.build(force=True) == build.LIB
    assert ran == ['nvcc', 'g++']
