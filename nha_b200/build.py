"""Build recipe of the CUDA library (sm_100a only) and of the host module.

``python -m nha_b200.build`` compiles every ``csrc/*.cu`` with nvcc into
``nha_b200/libnha_b200.so`` and every ``csrc/host/*.cpp`` with g++ against PyTorch
into ``nha_b200/_nha_host.so`` (in-tree, so the built files travel with the
source tree).  There is no other backend and no fallback: if they are
missing and cannot be built, the ops raise.
"""
from __future__ import annotations

import glob
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, 'csrc')
LIB = os.path.join(HERE, 'libnha_b200.so')
HOST = os.path.join(HERE, '_nha_host.so')

NVCC_FLAGS = [
    '-gencode', 'arch=compute_100a,code=sm_100a', '-lineinfo', '-O3', '-std=c++17',
    '--use_fast_math', '-Xcompiler', '-fPIC', '-shared', '-cudart', 'static',
]


def sources():
    return sorted(glob.glob(os.path.join(CSRC, '*.cu')))


def host_sources():
    return sorted(glob.glob(os.path.join(CSRC, 'host', '*.cpp')))


def _older(target, deps) -> bool:
    return not os.path.exists(target) or any(os.path.getmtime(f) > os.path.getmtime(target) for f in deps)


def is_stale() -> bool:
    header = glob.glob(os.path.join(HERE, '..', 'include', '*.h'))
    return _older(LIB, sources() + glob.glob(os.path.join(CSRC, '*.cuh')) + header) \
        or _older(HOST, host_sources() + glob.glob(os.path.join(CSRC, 'host', '*.h')) + header)


def nvcc_path():
    return shutil.which('nvcc') or ('/usr/local/cuda/bin/nvcc' if os.path.exists('/usr/local/cuda/bin/nvcc') else None)


def _host_flags():
    """(compiler, compile flags, link flags) of the host module: PyTorch's headers and libraries, and the CUDA library
    beside it (found through $ORIGIN, so the tree can be moved)."""
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    nvcc = nvcc_path()
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvcc))) if nvcc else '/usr/local/cuda'
    inc = [os.path.join(root, 'include'), os.path.join(root, 'include', 'torch', 'csrc', 'api', 'include'),
           os.path.join(cuda, 'include'), sysconfig.get_paths()['include']]
    abi = int(torch._C._GLIBCXX_USE_CXX11_ABI)
    cflags = ['-O2', '-std=c++17', '-fPIC', '-fvisibility=hidden', f'-D_GLIBCXX_USE_CXX11_ABI={abi}'] + [f'-isystem{d}' for d in inc]
    lib = os.path.join(root, 'lib')
    ldflags = [f'-L{lib}', '-lc10', '-lc10_cuda', '-ltorch', '-ltorch_cpu', '-ltorch_cuda', '-ltorch_python', '-Wl,-rpath,$ORIGIN',
               f'-Wl,-rpath,{lib}']
    return shutil.which('g++') or 'g++', cflags, ldflags


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile the library and the host module if one is missing or older than its sources; return the library's path."""
    if not force and not is_stale():
        return LIB
    nvcc = nvcc_path()
    if nvcc is None:
        raise RuntimeError('nha_b200: nvcc not found and libnha_b200.so is missing or stale; '
                           'there is no fallback implementation')
    objs = []
    # objects and the linked library under names of this process: several ranks that find the library stale at the same
    # time each build their own and the last rename wins, instead of linking each other's half-written objects
    tmp = os.path.join(HERE, 'build', f'p{os.getpid()}')
    os.makedirs(tmp, exist_ok=True)
    procs = []
    for src in sources():
        obj = os.path.join(tmp, os.path.basename(src)[:-3] + '.o')
        objs.append(obj)
        cmd = [nvcc] + [f for f in NVCC_FLAGS if f not in ('-shared',)] + os.environ.get('NHA_B200_NVCC_FLAGS', '').split() \
            + ['-c', src, '-o', obj]
        if verbose:
            cmd.insert(1, '-Xptxas=-v')
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    hobjs = []
    cxx, cflags, ldflags = _host_flags()
    for src in host_sources():
        obj = os.path.join(tmp, os.path.basename(src)[:-4] + '.host.o')
        hobjs.append(obj)
        procs.append((src, subprocess.Popen([cxx] + cflags + ['-c', src, '-o', obj], stdout=subprocess.PIPE, stderr=subprocess.STDOUT,
                                            text=True)))
    for src, p in procs:
        out, _ = p.communicate()
        if verbose and out:
            print(out)
        if p.returncode != 0:
            raise RuntimeError(f'compilation failed on {src}:\n{out}')
    out = f'{LIB}.{os.getpid()}.tmp'
    link = [nvcc, '-shared', '-cudart', 'static', '-gencode', 'arch=compute_100a,code=sm_100a', '-Xlinker', '-soname=libnha_b200.so', '-o', out] + objs
    r = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f'link failed:\n{r.stdout}')
    os.replace(out, LIB)
    out = f'{HOST}.{os.getpid()}.tmp'
    r = subprocess.run([cxx, '-shared', '-o', out] + hobjs + [LIB] + ldflags, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f'link failed:\n{r.stdout}')
    os.replace(out, HOST)
    shutil.rmtree(tmp, ignore_errors=True)
    return LIB


if __name__ == '__main__':
    print(build(force='--force' in sys.argv, verbose='-v' in sys.argv))
