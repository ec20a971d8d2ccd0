"""Build ``libfwp.so`` (the C-ABI library) in-tree with nvcc for sm_100a, and ``_fwp_torch.so`` (the host path of
the autograd entry points, plain C++ against PyTorch) beside it.

    python recurrent_fwp_b200/build.py [--force] [--verbose]

Each ``csrc/*.cu`` is compiled to an object file (in parallel) and linked into
``recurrent_fwp_b200/libfwp.so`` with the CUDA runtime linked statically, so the
library has no dependency beyond the driver.  Objects are rebuilt only when a
source or header is newer, ``_fwp_torch.so`` also when it was built against another
PyTorch or Python or by another command.  nvcc cross-compiles without a GPU.
"""
import concurrent.futures
import glob
import os
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, 'csrc')
OBJ = os.path.join(PKG, 'build')
LIB = os.path.join(PKG, 'libfwp.so')
BINDING_SRC = os.path.join(CSRC, 'binding', 'fwp_torch.cpp')
BINDING = os.path.join(PKG, '_fwp_torch.so')
BINDING_STAMP = os.path.join(OBJ, '_fwp_torch.built')
NVCC = os.environ.get('NVCC', '/usr/local/cuda/bin/nvcc')
FLAGS = ['-gencode', 'arch=compute_100a,code=sm_100a', '-lineinfo', '-O3', '-std=c++17',
         '-Xcompiler', '-fPIC', '-Xcompiler', '-fvisibility=hidden']


def _newer(src_list, target):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(s) > t for s in src_list)


def _compile(args):
    src, obj, verbose = args
    cmd = [NVCC] + FLAGS + (['-Xptxas', '-v'] if verbose else []) + ['-c', src, '-o', obj]
    r = subprocess.run(cmd, capture_output=True, text=True)
    return src, r.returncode, r.stdout + r.stderr


def _binding_command():
    """_fwp_torch.so: links libfwp.so (found beside it at run time) and the PyTorch libraries already loaded."""
    import torch
    from torch.utils import cpp_extension
    cmd = [os.environ.get('CXX', 'g++'), '-O2', '-std=c++17', '-fPIC', '-shared', '-fvisibility=hidden',
           '-D_GLIBCXX_USE_CXX11_ABI=%d' % torch._C._GLIBCXX_USE_CXX11_ABI,
           '-I' + sysconfig.get_paths()['include'], '-I' + os.path.join(os.path.dirname(os.path.dirname(NVCC)), 'include')]
    cmd += ['-isystem' + d for d in cpp_extension.include_paths()]
    cmd += [BINDING_SRC, '-o', BINDING, '-L' + PKG, '-l:libfwp.so', '-Wl,-rpath,$ORIGIN']
    cmd += ['-L' + d for d in cpp_extension.library_paths()]
    return cmd + ['-lc10', '-lc10_cuda', '-ltorch_cpu', '-ltorch_cuda', '-ltorch', '-ltorch_python']


def _binding_stamp():
    """What the extension depends on besides its source: it uses PyTorch's C++ interface, which changes with the version."""
    import torch
    return '\n'.join([torch.__version__, str(torch.version.git_version), sys.version] + _binding_command())


def _binding_stale():
    if _newer([BINDING_SRC] + glob.glob(os.path.join(PKG, '..', 'include', '*.h')), BINDING):
        return True
    try:
        with open(BINDING_STAMP) as f:
            return f.read() != _binding_stamp()
    except OSError:
        return True


def _compile_binding():
    r = subprocess.run(_binding_command(), capture_output=True, text=True)
    if r.returncode:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError('the compiler failed on %s' % BINDING_SRC)
    with open(BINDING_STAMP, 'w') as f:
        f.write(_binding_stamp())


def build(force=False, verbose=False):
    os.makedirs(OBJ, exist_ok=True)
    sources = sorted(glob.glob(os.path.join(CSRC, '*.cu')))
    headers = glob.glob(os.path.join(CSRC, '*.cuh')) + glob.glob(os.path.join(PKG, '..', 'include', '*.h'))
    jobs, objs = [], []
    for src in sources:
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + '.o')
        objs.append(obj)
        if force or _newer([src] + headers, obj):
            jobs.append((src, obj, verbose))
    if jobs:
        with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            for src, rc, log in ex.map(_compile, jobs):
                if verbose or rc:
                    sys.stderr.write(log)
                if rc:
                    raise RuntimeError('nvcc failed on %s' % src)
    if jobs or _newer(objs, LIB):
        cmd = [NVCC, '-shared', '-o', LIB] + objs + ['-cudart', 'static',
               '-gencode', 'arch=compute_100a,code=sm_100a', '-Xcompiler', '-fPIC']
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError('link failed')
    if force or _binding_stale():
        _compile_binding()
    return LIB


if __name__ == '__main__':
    print(build(force='--force' in sys.argv, verbose='--verbose' in sys.argv))
