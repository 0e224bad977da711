"""Compile the CUDA backend for sm_100a into pysurf_b200/libpysurf_b200.so (in-tree).

    python -m pysurf_b200.build          # rebuild when a source is newer than the library

nvcc cross-compiles without a GPU, so this runs on any machine with the CUDA toolkit.
"""
from __future__ import annotations

import glob
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
LIBRARY = os.path.join(HERE, 'libpysurf_b200.so')
OBJECTS = os.path.join(HERE, '_build')
# each unit's source and definitions, compiled side by side, the longest first; the sweeps once a dimension
# and kernel
UNITS = [('csrc/sph_sweep_kernels.cu', [f'-DSPH_SWEEP_DIM={dim}', f'-DSPH_SWEEP_KERNEL={kernel}'])
         for dim in (3, 2) for kernel in (1, 0)]
UNITS += [(f'csrc/{name}.cu', []) for name in ('sph_classic_sweeps', 'sph_kernels', 'sph_system', 'sph_noalloc',
                                               'sph_surface', 'sph_merge')]
ARCH = ['-gencode', 'arch=compute_100a,code=sm_100a']
FLAGS = ['-O3', '-lineinfo', '-std=c++17', '-Xcompiler', '-fPIC']


def inputs() -> list:
    files = [os.path.join(HERE, s) for s, _ in UNITS]
    files += glob.glob(os.path.join(HERE, 'csrc', '*.cuh')) + glob.glob(os.path.join(HERE, 'csrc', '*.h'))
    files.append(os.path.join(ROOT, 'include', 'pysurf_b200.h'))
    return files


def stale() -> bool:
    if not os.path.exists(LIBRARY):
        return True
    built = os.path.getmtime(LIBRARY)
    return any(os.path.getmtime(f) > built for f in inputs())


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not stale():
        return LIBRARY
    nvcc = os.environ.get('NVCC', 'nvcc')
    os.makedirs(OBJECTS, exist_ok=True)
    objects, running = [], []
    for k, (source, defines) in enumerate(UNITS):
        objects.append(os.path.join(OBJECTS, f'unit{k}.o'))
        command = [nvcc] + ARCH + FLAGS + defines + ['-c', '-o', objects[-1], os.path.join(HERE, source)]
        if verbose:
            print(' '.join(command), flush=True)
        running.append((command, subprocess.Popen(command, cwd=HERE)))
    failed = [command for command, process in running if process.wait() != 0]
    if failed:
        raise subprocess.CalledProcessError(1, failed[0])
    command = [nvcc] + ARCH + ['-shared', '-o', LIBRARY] + objects
    if verbose:
        print(' '.join(command), flush=True)
    subprocess.check_call(command, cwd=HERE)
    return LIBRARY


if __name__ == '__main__':
    print(build(force='--force' in sys.argv, verbose=True))
