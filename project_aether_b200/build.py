"""Builds libaether_sort.so for sm_100a with nvcc, and the Python binding, in the package folder.

    python -m project_aether_b200.build [--force] [--verbose]

The library is a plain C-ABI shared object (see include/aether_sort.h); it is
loaded with ctypes and needs no Python headers.  The binding (csrc/binding.cpp) is a
Python extension built against the installed PyTorch, which calls that library.  The
package works without it, with more host time per call.
"""

import argparse
import os
import shutil
import subprocess
import sysconfig
import warnings

import torch

from ._native import binding_abi

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, 'csrc')
LIB = os.path.join(PKG, 'libaether_sort.so')
BINDING = os.path.join(PKG, '_binding.so')
SOURCES = ['api.cu', 'sort_standard.cu', 'sort_bucketed.cu', 'slab_partition.cu', 'particle_push.cu',
           'static_scratch.cu', 'collide.cu']
NVCC_FLAGS = [
    '-O3', '-std=c++17', '-gencode', 'arch=compute_100a,code=sm_100a', '-lineinfo',
    '-Xcompiler', '-fPIC', '-shared', '--use_fast_math=false',
]


def _nvcc() -> str:
    for cand in (shutil.which('nvcc'), '/usr/local/cuda/bin/nvcc'):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError('nvcc not found; the CUDA library cannot be built')


def _binding_stale(sources) -> bool:
    """Also where the binding was built for another PyTorch or Python: its name for what it was
    built for is a text inside it."""
    if _stale(BINDING, sources):
        return True
    with open(BINDING, 'rb') as f:
        return binding_abi().encode() not in f.read()


def _stale(target: str, sources) -> bool:
    if not os.path.exists(target):
        return True
    built = os.path.getmtime(target)
    return any(os.path.getmtime(d) > built for d in sources)


def _run(cmd, verbose: bool) -> None:
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or proc.returncode != 0:
        print(proc.stdout + proc.stderr)
    if proc.returncode != 0:
        raise RuntimeError(f'{cmd[0]} failed:\n' + proc.stderr[-4000:])


def _binding_command():
    root = os.path.dirname(torch.__file__)
    includes = [sysconfig.get_paths()['include'], os.path.join(root, 'include'),
                os.path.join(root, 'include', 'torch', 'csrc', 'api', 'include'),
                os.path.join(os.path.dirname(os.path.dirname(_nvcc())), 'include')]
    return ['g++', '-O2', '-std=c++17', '-fPIC', '-shared',
            f'-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}',
            f'-DAETHER_BUILT_FOR="{binding_abi()}"',
            *(f'-I{d}' for d in includes), '-o', BINDING, os.path.join(CSRC, 'binding.cpp'),
            '-L' + os.path.join(root, 'lib'), '-lc10', '-lc10_cuda', '-ltorch_cpu', '-ltorch_python']


def build(force: bool = False, verbose: bool = False) -> str:
    """Compiles every CUDA source into libaether_sort.so, then the binding; returns the library's path.

    A binding that cannot be built (no Python headers, say) is a warning: the library serves every call
    without it."""
    header = os.path.join(os.path.dirname(PKG), 'include', 'aether_sort.h')
    binding = os.path.join(CSRC, 'binding.cpp')
    kernels = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f != 'binding.cpp']
    if force or _stale(LIB, [*kernels, header]):
        flags = [f for f in NVCC_FLAGS if not f.startswith('--use_fast_math')]
        if verbose:
            flags += ['-Xptxas', '-v']
        _run([_nvcc(), *flags, '-ccbin', 'g++', '-o', LIB] + [os.path.join(CSRC, s) for s in SOURCES], verbose)
    if force or _binding_stale([binding, header]):
        try:
            _run(_binding_command(), verbose)
        except (OSError, RuntimeError) as e:
            warnings.warn(f'the Python binding was not built, calls go through ctypes: {e}', RuntimeWarning)
    return LIB


if __name__ == '__main__':
    ap = argparse.ArgumentParser()
    ap.add_argument('--force', action='store_true')
    ap.add_argument('--verbose', action='store_true')
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose))
