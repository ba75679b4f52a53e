"""Build libkvm_b200.so (sm_100a only) in-tree with nvcc.  `python -m kvm_b200.build [--force] [--verbose]`."""
from __future__ import annotations

import os
import re
import time
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / 'csrc'
LIB = PKG / 'libkvm_b200.so'
CLI = PKG / 'kvm_exec'
NVCC = os.environ.get('NVCC', '/usr/local/cuda/bin/nvcc')
CXX = os.environ.get('CXX', 'g++')
UNITS = ('kvm_exec', 'kvm_static', 'kvm_unit_flat', 'kvm_unit_rows', 'kvm_unit_mm', 'kvm_unit_attn', 'kvm_unit_decode')
# relocatable device code: the op families (kvm_unit_*) are linked into both executor kernels; 96 registers is what those kernels' block sizes leave a thread
FLAGS = ['-gencode', 'arch=compute_100a,code=sm_100a', '-rdc=true', '-maxrregcount=96', '-O3', '-std=c++17', '-lineinfo', '-Xcompiler', '-fPIC',
         '--expt-relaxed-constexpr', '--extended-lambda', '-Xcudafe', '--diag_suppress=177']


def sources(unit):
    """The files a translation unit is made of: its own source and everything it includes."""
    seen, todo = set(), [CSRC / f'{unit}.cu']
    while todo:
        p = todo.pop()
        if p in seen:
            continue
        seen.add(p)
        todo += [(p.parent / m).resolve() for m in re.findall(r'^ *#include "([^"]+)"', p.read_text(), re.M)]
    return seen


def unit_stale(unit) -> bool:
    obj = PKG / f'_{unit}.o'
    return not obj.exists() or any(s.stat().st_mtime > obj.stat().st_mtime for s in sources(unit))


def stale() -> bool:
    if not LIB.exists():
        return True
    return any(unit_stale(u) for u in UNITS) or any((PKG / f'_{u}.o').stat().st_mtime > LIB.stat().st_mtime for u in UNITS)


def build(force: bool = False, verbose: bool = False) -> Path:
    """The translation units (two executor kernels, the op families), compiled side by side, then linked."""
    if not force and not stale():
        return LIB
    objs, procs = [], []
    started = time.time()          # an object counts as built when its compile STARTED: a source edited while nvcc runs stays newer
    for unit in UNITS:
        obj = PKG / f'_{unit}.o'
        objs.append(obj)
        if not force and not unit_stale(unit):
            continue
        cmd = [NVCC, *FLAGS, *(['-Xptxas', '-v'] if verbose else []), '-c', str(CSRC / f'{unit}.cu'), '-o', str(obj)]
        procs.append((cmd, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True)))
    for cmd, p in procs:
        out, err = p.communicate()
        if verbose or p.returncode:
            sys.stderr.write(out + err)
        if p.returncode:
            raise RuntimeError(f'nvcc failed ({p.returncode}): {" ".join(cmd)}')
        os.utime(cmd[-1], (started, started))
    cmd = [NVCC, '-gencode', 'arch=compute_100a,code=sm_100a', '-shared', *map(str, objs), '-o', str(LIB), '-lcudart']
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError(f'link failed ({r.returncode}): {" ".join(cmd)}')
    return LIB


def build_cli(force: bool = False) -> Path:
    """kvm_exec: the command-line runner (host C++ over the C ABI, no CUDA code of its own), next to the library."""
    src = CSRC / 'kvm_cli.cpp'
    if not force and CLI.exists() and CLI.stat().st_mtime >= max(src.stat().st_mtime, LIB.stat().st_mtime if LIB.exists() else 0):
        return CLI
    build(force)
    cmd = [CXX, '-O2', '-std=c++17', str(src), '-o', str(CLI), f'-L{PKG}', '-lkvm_b200', '-Wl,-rpath,$ORIGIN']
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError(f'g++ failed ({r.returncode}): {" ".join(cmd)}')
    return CLI


if __name__ == '__main__':
    print(build(force='--force' in sys.argv, verbose='--verbose' in sys.argv))
    print(build_cli(force='--force' in sys.argv))
