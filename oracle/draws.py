"""ctypes access to ``libdraws.so``: device checks of the error bounds and the batches of the just-in-time walks.
TEST INFRASTRUCTURE ONLY."""
import ctypes
import os
import subprocess

_HERE = os.path.dirname(os.path.abspath(__file__))
_LIB_PATH = os.path.join(_HERE, 'libdraws.so')
_lib = None


def build():
  """Compile ``libdraws.so`` where it is missing or older than its sources."""
  subprocess.check_call(['make', '-C', _HERE, 'draws'], stdout=subprocess.DEVNULL)
  return _LIB_PATH


def _call(name, *args):
  import torch
  global _lib
  if _lib is None:
    _lib = ctypes.CDLL(build())
  fn = getattr(_lib, f'draws_{name}')
  fn.restype = ctypes.c_int
  rc = fn(*args, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
  if rc != 0:
    raise RuntimeError(f'draws_{name}: {rc}')


def log_error():
  """The largest error of the quick logarithm against the reference's, as a share of the bound that the walks take, over all
  2^32 draws."""
  import torch
  out = torch.zeros(1, dtype=torch.float64, device='cuda')
  _call('log_error', ctypes.c_void_p(out.data_ptr()))
  return float(out)


def batch_mismatches(kind, per_batch, sums, low24, log_p, seed, n_streams, n):
  """``(connections, wrong ones)`` of the streams ``seed ..`` over ``n`` positions, in batches against one connection at a time."""
  import torch
  out = torch.zeros(2, dtype=torch.int64, device='cuda')
  _call('batch_mismatches', kind, per_batch, int(sums), int(low24), ctypes.c_double(log_p), ctypes.c_uint32(seed),
        ctypes.c_uint32(n_streams), ctypes.c_uint32(n), ctypes.c_void_p(out.data_ptr()))
  return tuple(out.tolist())
