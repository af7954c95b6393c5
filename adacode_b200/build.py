"""In-tree build of the sm_100a shared library (``libadacode_sm100.so``) and of the extension module that calls it
(``_native``).

``python -m adacode_b200.build`` compiles ``csrc/*.cu`` with nvcc for ``sm_100a`` only, and ``csrc/host_path.cpp`` with the
host compiler against the installed torch.  nvcc cross-compiles without a GPU, so this also runs on a CPU-only machine.
"""
from __future__ import annotations

import glob
import os
import subprocess
import sys
import sysconfig

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
ROOT_DIR = os.path.dirname(PKG_DIR)
LIB_PATH = os.path.join(PKG_DIR, 'libadacode_sm100.so')
NVCC_FLAGS = [
    '-gencode', 'arch=compute_100a,code=sm_100a', '-lineinfo', '-O3', '-std=c++17',
    '-Xcompiler', '-fPIC', '-shared',
]


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(PKG_DIR, 'csrc', '*.cu')))


def _stale(path: str, deps: list[str]) -> bool:
    return not os.path.exists(path) or any(os.path.getmtime(p) > os.path.getmtime(path) for p in deps)


def _run(cmd: list[str]) -> str:
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(f'{cmd[0]} failed ({proc.returncode}):\n{proc.stdout}\n{proc.stderr}')
    return proc.stderr


def native_path() -> str:
    """The extension module's file, which no other Python takes for its own."""
    return os.path.join(PKG_DIR, '_native' + sysconfig.get_config_var('EXT_SUFFIX'))


def built_for() -> str:
    """What a module has to be compiled against to be loaded here: it reads torch's objects through torch's headers."""
    import torch
    return f'adacode host path for torch {torch.__version__}'


def _compiled_for_this_torch(path: str) -> bool:
    with open(path, 'rb') as f:
        return built_for().encode() + b'\0' in f.read()


def build_native(force: bool = False) -> str:
    """Compile the extension module if it is missing, older than its sources or made for another torch; return its path."""
    import torch
    source, path = os.path.join(PKG_DIR, 'csrc', 'host_path.cpp'), native_path()
    headers = glob.glob(os.path.join(ROOT_DIR, 'include', '*.h'))
    if not force and not _stale(path, [source, *headers]) and _compiled_for_this_torch(path):
        return path
    torch_dir = os.path.dirname(torch.__file__)
    cuda = os.environ.get('CUDA_HOME', '/usr/local/cuda')
    include = [os.path.join(ROOT_DIR, 'include'), os.path.join(torch_dir, 'include'),
               os.path.join(torch_dir, 'include', 'torch', 'csrc', 'api', 'include'), sysconfig.get_paths()['include'],
               os.path.join(cuda, 'include')]
    _run([os.environ.get('CXX', 'g++'), '-O2', '-std=c++17', '-fPIC', '-shared',
          f'-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}', f'-DADACODE_BUILT_FOR="{built_for()}"',
          *(f'-I{p}' for p in include), source, '-o', path, f'-L{PKG_DIR}', '-l:' + os.path.basename(LIB_PATH),
          '-L' + os.path.join(torch_dir, 'lib'), '-ltorch_python', '-ltorch', '-ltorch_cpu', '-ltorch_cuda', '-lc10', '-lc10_cuda',
          '-L' + os.path.join(cuda, 'lib64'), '-lcudart', '-Wl,-rpath,$ORIGIN'])
    return path


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile the library, then the extension module, where they are missing or older than their sources; return the
    library's path."""
    deps = sources() + glob.glob(os.path.join(ROOT_DIR, 'include', '*.h')) + glob.glob(os.path.join(PKG_DIR, 'csrc', '*.cuh'))
    if force or _stale(LIB_PATH, deps):
        _build_library(verbose)
    build_native(force)
    return LIB_PATH


def _build_library(verbose: bool) -> None:
    nvcc = os.environ.get('NVCC', 'nvcc')
    cmd = [nvcc, *NVCC_FLAGS, '-I', os.path.join(ROOT_DIR, 'include'), '-o', LIB_PATH, *sources()]
    if verbose:
        cmd.insert(1, '-Xptxas')
        cmd.insert(2, '-v')
    log = _run(cmd)
    if verbose:
        sys.stderr.write(log)


if __name__ == '__main__':
    print(build(force='--force' in sys.argv, verbose='-v' in sys.argv))
