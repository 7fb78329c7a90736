"""Builds libnsa_b200.so (the C-ABI library, nvcc for sm_100a) and _nsa_host.so (the native host side of the PyTorch
operators, g++ against the installed PyTorch) in-tree.

    python -m native_sparse_attention_pytorch_b200.build [--force] [--verbose]
"""
import glob
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, 'csrc')
LIB = os.path.join(HERE, 'libnsa_b200.so')
SOURCES = ['nsa_abi.cu', 'nsa_simt_attend.cu', 'nsa_select.cu', 'nsa_combine.cu', 'nsa_rotary.cu', 'nsa_windows.cu', 'nsa_rmsnorm.cu', 'nsa_decode.cu', 'nsa_layer.cu', 'nsa_gemm.cu', 'nsa_topk_grad.cu', 'nsa_sm100_sel.cu']


HOST_LIB = os.path.join(HERE, '_nsa_host.so')
HOST_SOURCES = ['module.cpp', 'status.cpp', 'selected.cpp', 'rooms.cpp', 'decode.cpp', 'layer.cpp']


def _newest(*dirs):
    paths = [os.path.join(d, f) for d in dirs for f in os.listdir(d)] + [os.path.join(ROOT, 'include', 'nsa_b200.h')]
    return max(os.path.getmtime(p) for p in paths if os.path.isfile(p))


def _fresh(lib, *dirs):
    return os.path.exists(lib) and os.path.getmtime(lib) >= _newest(*dirs)


HOST_STAMP = os.path.join(HERE, 'build', 'host_built_for.txt')


def _built_for():
    """What _nsa_host.so depends on besides its sources: it does not load into another PyTorch or Python."""
    import torch
    return f'PyTorch {torch.__version__} at {os.path.dirname(torch.__file__)}, {sysconfig.get_config_var("SOABI")}\n'


def _host_fresh():
    if not (_fresh(HOST_LIB, CSRC, os.path.join(CSRC, 'host')) and os.path.exists(HOST_STAMP)):
        return False
    with open(HOST_STAMP) as f:
        return f.read() == _built_for()


def _cuda_library(name, package, site, toolkit):
    """The shared library PyTorch itself uses: from NVIDIA's wheels beside it, or from the toolkit it was built with."""
    places = [os.path.join(site, 'nvidia', package, 'lib'), os.path.join(site, 'nvidia', 'cu*', 'lib'), os.path.join(toolkit, 'lib64'),
              os.path.join(toolkit, 'targets', '*', 'lib')]
    for place in places:
        found = sorted(glob.glob(os.path.join(place, name + '.so.[0-9]*'))) or glob.glob(os.path.join(place, name + '.so'))
        if found:
            return min(found, key=len)     # libcublas.so.12 rather than libcublas.so.12.8.4.1
    raise RuntimeError(f'{name}.so was found in none of {places}: _nsa_host.so links against the one PyTorch uses')


def _compile_all(jobs, verbose):
    """jobs: (source name, object, command).  Runs them side by side and returns the objects."""
    procs = [(src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)) for src, _, cmd in jobs]
    failed = None
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode != 0:
            sys.stderr.write(f'--- {src} ---\n{out}\n')
        if p.returncode != 0:
            failed = failed or src
    if failed:
        raise RuntimeError(f'compiling {failed} failed')
    return [obj for _, obj, _ in jobs]


def build(force=False, verbose=False):
    """Compile every kernel file for sm_100a and link the two shared libraries."""
    nvcc = os.environ.get('NVCC', '/usr/local/cuda/bin/nvcc')
    objdir = os.path.join(HERE, 'build')
    os.makedirs(objdir, exist_ok=True)
    includes = ['-I', os.path.join(ROOT, 'include'), '-I', CSRC]
    jobs, host_jobs = [], []
    if force or not _fresh(LIB, CSRC):
        flags = ['-gencode', 'arch=compute_100a,code=sm_100a', '-lineinfo', '-O3', '-std=c++17', '-Xcompiler', '-fPIC',
                 *includes] + (['-Xptxas', '-v'] if verbose else [])
        jobs = [(src, os.path.join(objdir, src.replace('.cu', '.o')),
                 [nvcc, *flags, '-c', os.path.join(CSRC, src), '-o', os.path.join(objdir, src.replace('.cu', '.o'))])
                for src in SOURCES]
    if force or not _host_fresh():
        import torch
        from torch.utils import cpp_extension
        cuda = os.path.dirname(os.path.dirname(nvcc))
        flags = ['-O2', '-std=c++17', '-fPIC', '-fvisibility=hidden', '-DTORCH_API_INCLUDE_EXTENSION_H',
                 f'-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}', *includes,
                 '-isystem', sysconfig.get_paths()['include'], '-isystem', os.path.join(cuda, 'include')]
        for d in cpp_extension.include_paths():
            flags += ['-isystem', d]
        host_jobs = [(src, os.path.join(objdir, 'host_' + src.replace('.cpp', '.o')),
                      ['g++', *flags, '-c', os.path.join(CSRC, 'host', src), '-o', os.path.join(objdir, 'host_' + src.replace('.cpp', '.o'))])
                     for src in HOST_SOURCES]
    objs = _compile_all(jobs + host_jobs, verbose)
    if jobs:
        subprocess.run([nvcc, '-shared', '-o', LIB, *objs[:len(jobs)], '-cudart', 'static',
                        '-gencode', 'arch=compute_100a,code=sm_100a'], check=True)
    if host_jobs:
        import torch
        torch_lib = os.path.join(os.path.dirname(torch.__file__), 'lib')
        # PyTorch's own copies of cuBLAS and the CUDA runtime, which its libraries have loaded by the time this one is
        site, toolkit = os.path.dirname(os.path.dirname(torch.__file__)), os.path.dirname(os.path.dirname(nvcc))
        shared = [_cuda_library('libcublas', 'cublas', site, toolkit), _cuda_library('libcudart', 'cuda_runtime', site, toolkit)]
        subprocess.run(['g++', '-shared', '-o', HOST_LIB, *objs[len(jobs):], '-L', HERE, '-lnsa_b200', '-L', torch_lib, '-ltorch', '-ltorch_cpu',
                        '-ltorch_cuda', '-ltorch_python', '-lc10', '-lc10_cuda', *shared, '-Wl,-rpath,$ORIGIN'], check=True)
        with open(HOST_STAMP, 'w') as f:
            f.write(_built_for())
    return LIB


if __name__ == '__main__':
    print(build(force='--force' in sys.argv, verbose='--verbose' in sys.argv))
