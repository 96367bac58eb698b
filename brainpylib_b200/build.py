"""Compile the CUDA sources under ``csrc/`` into ``libbrainpylib_b200.so`` (in-tree).

and the operators' host path ``csrc/native.cc`` into the extension module ``_native`` (g++, against torch's headers).

Usage: ``python -m brainpylib_b200.build [--force] [--verbose]``

sm_100a only; no fast-math (the just-in-time-connectivity kernels must reproduce the
reference's float arithmetic bit for bit).  ``-Xptxas -v`` output (registers, spills,
shared memory) is written next to the library as ``ptxas_info.txt``.
"""
import concurrent.futures
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, 'csrc')
LIB = os.path.join(HERE, 'libbrainpylib_b200.so')
BUILD_DIR = os.path.join(HERE, 'csrc', 'build')
SOURCES = ['csr_kernels.cu', 'csr_shared_gather.cu', 'csr_shared_scatter.cu', 'csr_shared_events_float.cu', 'csr_shared_events_double.cu', 'cbcsr_kernels.cu', 'cbcsr_build.cu', 'jitconn_kernels.cu', 'jit_matmat.cu', 'jitconn_matmat_versions.cu', 'jitconn_event_v1.cu', 'neuron_kernels.cu', 'scatter_kernels.cu', 'event_info_kernels.cu',
           'exchange_kernels.cu', 'host_steps.cc', 'gpu_ops.cc']
HEADERS = ['abi.h', 'common.cuh', 'spike_scan.cuh', 'row_scatter.cuh', 'cb_scatter.cuh', 'jit_stream.cuh', 'csr_shared.h', 'csr_shared.cuh', 'csr_shared_events.cuh', os.path.join('..', '..', 'include', 'brainpylib_b200.h')]
NVCC = os.environ.get('NVCC', 'nvcc')
FLAGS = ['-O3', '-std=c++17', '-gencode', 'arch=compute_100a,code=sm_100a', '-lineinfo',
         '-Xcompiler', '-fPIC', '-Xptxas', '-v', '-Xcudafe', '--diag_suppress=68']


NATIVE_SOURCE = os.path.join(CSRC, 'native.cc')
NATIVE = os.path.join(HERE, '_native' + sysconfig.get_config_var('EXT_SUFFIX'))
NATIVE_STAMP = os.path.join(BUILD_DIR, 'native_torch.txt')     # the torch that NATIVE was compiled against
CXX = os.environ.get('CXX', 'g++')


def _sources():
  return [s for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]


def _stale(target, deps):
  if not os.path.exists(target):
    return True
  t = os.path.getmtime(target)
  return any(os.path.getmtime(d) > t for d in deps)


def _compile(src, verbose):
  obj = os.path.join(BUILD_DIR, os.path.splitext(src)[0] + '.o')
  deps = [os.path.join(CSRC, src)] + [os.path.join(CSRC, h) for h in HEADERS] + [os.path.abspath(__file__)]
  if not _stale(obj, deps):
    return obj, ''
  cmd = [NVCC] + FLAGS + ['-c', os.path.join(CSRC, src), '-o', obj]
  if verbose:
    print(' '.join(cmd), flush=True)
  p = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
  if p.returncode != 0:
    raise RuntimeError(f'nvcc failed on {src}:\n{p.stdout}')
  return obj, p.stdout


def _native_command():
  import torch
  from torch.utils import cpp_extension
  includes = cpp_extension.include_paths('cuda') + [sysconfig.get_path('include')]
  libs = cpp_extension.library_paths('cuda')
  return ([CXX, '-O2', '-std=c++17', '-shared', '-fPIC', '-fvisibility=hidden', '-w',
           f'-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}'] + [f'-I{d}' for d in includes] +
          [NATIVE_SOURCE, '-o', NATIVE] + [f'-L{d}' for d in libs] +
          ['-lc10', '-lc10_cuda', '-ltorch_cpu', '-ltorch_cuda', '-ltorch', '-ltorch_python', f'-L{HERE}', '-lbrainpylib_b200',
           '-Wl,-rpath,$ORIGIN'])


def _torch_stamp():
  import torch
  return f'{torch.__version__} abi={int(torch._C._GLIBCXX_USE_CXX11_ABI)}\n'


def _native_stale(deps):
  if _stale(NATIVE, deps) or not os.path.exists(NATIVE_STAMP):
    return True
  with open(NATIVE_STAMP) as f:
    return f.read() != _torch_stamp()


def _build_native(force, verbose):
  """The extension module.  Its text depends on the C ABI and on torch's headers and libraries, so it is linked again when
  those change and not when a kernel does.  The object goes to a name of this process first: a reader never sees half a
  file, nor do two builds write one."""
  deps = [NATIVE_SOURCE, os.path.join(CSRC, 'abi.h'), os.path.join(CSRC, HEADERS[-1]), os.path.abspath(__file__)]
  if not force and not _native_stale(deps):
    return
  cmd = _native_command()
  out = f'{NATIVE}.{os.getpid()}.tmp'
  cmd[cmd.index(NATIVE)] = out
  if verbose:
    print(' '.join(cmd), flush=True)
  p = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
  if p.returncode != 0:
    raise RuntimeError(f'{CXX} failed on native.cc:\n{p.stdout}')
  os.replace(out, NATIVE)
  os.makedirs(BUILD_DIR, exist_ok=True)
  with open(NATIVE_STAMP, 'w') as f:
    f.write(_torch_stamp())


def build(force=False, verbose=False):
  """Build the shared library and the extension module if any source is newer.  Returns the library's path."""
  _build_library(force, verbose)
  _build_native(force, verbose)
  return LIB


def _build_library(force, verbose):
  srcs = _sources()
  all_inputs = [os.path.join(CSRC, f) for f in srcs + HEADERS] + [os.path.abspath(__file__)]
  if not force and not _stale(LIB, all_inputs):
    return
  os.makedirs(BUILD_DIR, exist_ok=True)
  if force:
    for s in srcs:
      o = os.path.join(BUILD_DIR, os.path.splitext(s)[0] + '.o')
      if os.path.exists(o):
        os.remove(o)
  with concurrent.futures.ThreadPoolExecutor(max_workers=len(srcs)) as ex:
    results = list(ex.map(lambda s: _compile(s, verbose), srcs))
  objs = [o for o, _ in results]
  # one log per source, replaced whenever that source is recompiled; ptxas_info.txt is their concatenation and so
  # always describes the objects the library is linked from
  for s, (_, log) in zip(srcs, results):
    if log:
      with open(os.path.join(BUILD_DIR, 'ptxas_' + os.path.splitext(s)[0] + '.txt'), 'w') as f:
        f.write(log)
  with open(os.path.join(BUILD_DIR, 'ptxas_info.txt'), 'w') as out:
    for s in srcs:
      part = os.path.join(BUILD_DIR, 'ptxas_' + os.path.splitext(s)[0] + '.txt')
      if os.path.exists(part):
        out.write(open(part).read())
  if force or _stale(LIB, objs):
    cmd = [NVCC, '-shared', '-o', LIB] + objs + ['-gencode', 'arch=compute_100a,code=sm_100a']
    if verbose:
      print(' '.join(cmd), flush=True)
    subprocess.check_call(cmd)


if __name__ == '__main__':
  path = build(force='--force' in sys.argv, verbose='--verbose' in sys.argv or '-v' in sys.argv)
  print(path)
