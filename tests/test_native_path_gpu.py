"""The native host path: its gradients (C++ nodes, weight gradient in one kernel) against index arithmetic in float64, on
row lengths around the kernel's units of 4 entries and 4..32 lanes, and its second-order gradients."""
import threading
import time

import numpy as np
import pytest
import torch

import cases
import brainpylib_b200 as bpl
from brainpylib_b200 import sparse_ops
from oracle import cpu

pytestmark = pytest.mark.gpu

ROWS = {'mixed': [0, 1, 3, 4, 5, 0, 31, 32, 33, 127, 64, 2], 'short': [1] * 70, 'long': [700, 1, 1024, 513], 'empty': [0, 0]}


def _expected(data, indices, indptr, x, ct, shape, transpose):
  row, col = sparse_ops.csr_to_coo(indices, indptr)
  d, x, ct = data.detach().double(), x.detach().double(), ct.double()
  g_data = x[row] * ct[col] if transpose else x[col] * ct[row]
  g_x = torch.zeros(x.shape[0], dtype=torch.float64, device=x.device)
  g_x.index_add_(0, row if transpose else col, d * (ct[col] if transpose else ct[row]))
  return g_data, g_x


@pytest.mark.parametrize('event', [False, True])
@pytest.mark.parametrize('transpose', [False, True])
@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
@pytest.mark.parametrize('rows', sorted(ROWS))
@pytest.mark.parametrize('offset', [0, 1])     # 1: index array not 16-byte aligned
def test_gradients_of_weights_and_vector(cuda, rows, dtype, transpose, event, offset):
  n_col = 900
  data, indices, indptr, rng = cases.ragged_csr(ROWS[rows], n_col, 3)
  shape = (len(ROWS[rows]), n_col)
  indices = torch.as_tensor(np.concatenate([np.zeros(offset, np.int32), indices])).to(cuda)[offset:]
  indptr = torch.as_tensor(indptr).to(cuda)
  data = torch.as_tensor(data).to(cuda, dtype).requires_grad_(True)
  n_in, n_out = shape if transpose else shape[::-1]
  x = torch.as_tensor(rng.standard_normal(n_in) * (rng.random(n_in) < 0.5)).to(cuda, dtype).requires_grad_(True)
  ct = torch.as_tensor(rng.standard_normal(n_out)).to(cuda, dtype)
  op = bpl.event_csr_matvec if event else bpl.csr_matvec
  y = op(data, indices, indptr, x, shape=shape, transpose=transpose)
  got = torch.autograd.grad(y, (data, x), ct)
  tol = dict(rtol=1e-5, atol=1e-4) if dtype == torch.float32 else dict(rtol=1e-12, atol=1e-11)
  for g, want in zip(got, _expected(data, indices, indptr, x, ct, shape, transpose)):
    torch.testing.assert_close(g.double(), want, **tol)


@pytest.mark.parametrize('event', [False, True])
@pytest.mark.parametrize('transpose', [False, True])
# the three kernels: vector in shared memory, longer vector swept in bands, neither; no rows at all
@pytest.mark.parametrize('n_row,n_col,mean', [(20_000, 3000, 60), (20_000, 60_000, 120), (300, 60_000, 9), (0, 40, 0)])
def test_gradient_of_entries_that_no_row_owns(cuda, n_row, n_col, mean, transpose, event):
  """Arrays with room in front of and behind the matrix: the product does not use it, so its gradient is zero."""
  front, back = 5, 3011
  indptr = torch.arange(front, front + n_row * mean + 1, max(mean, 1), dtype=torch.int32, device=cuda)[:n_row + 1]
  g = torch.Generator(device=cuda).manual_seed(1)
  nse = front + n_row * mean + back
  indices = torch.randint(0, n_col, (nse,), dtype=torch.int32, device=cuda, generator=g)
  data = torch.rand(nse, device=cuda, generator=g).requires_grad_(True)
  x = torch.rand(n_row if transpose else n_col, device=cuda, generator=g)
  op = bpl.event_csr_matvec if event else bpl.csr_matvec
  y = op(data, indices, indptr, x, shape=(n_row, n_col), transpose=transpose)
  ct = torch.rand_like(y)
  junk = torch.full_like(data, float('nan'))
  del junk                               # its memory is the gradient's
  got = torch.autograd.grad(y, data, ct)[0]
  want = torch.zeros_like(got)
  if n_row:
    row = torch.arange(n_row, device=cuda).repeat_interleave(mean)
    col = indices[front:nse - back].long()
    want[front:nse - back] = x[row] * ct[col] if transpose else x[col] * ct[row]
  torch.testing.assert_close(got, want)


@pytest.mark.parametrize('transpose', [False, True])
def test_second_order_gradients(cuda, transpose):
  data, indices, indptr, rng = cases.csr_case((30, 40), 0.3, 11, dtype=np.float64)
  w = torch.as_tensor(data).to(cuda).requires_grad_(True)
  indices, indptr = torch.as_tensor(indices).to(cuda), torch.as_tensor(indptr).to(cuda)
  x = torch.as_tensor(rng.standard_normal(30 if transpose else 40)).to(cuda).requires_grad_(True)
  op = lambda w, x: bpl.csr_matvec(w, indices, indptr, x, shape=(30, 40), transpose=transpose)
  assert torch.autograd.gradcheck(op, (w, x)) and torch.autograd.gradgradcheck(op, (w, x))


@pytest.mark.parametrize('dtype', [np.float32, np.float64])
@pytest.mark.parametrize('homo', [False, True])
# the whole vector in shared memory: few columns, rows of every lane count, the longest vector that fits (4 and 8 bytes),
# one element more (plain kernels); the entry count is no multiple of 4
@pytest.mark.parametrize('n_row,n_col,mean', [(9000, 2000, 333), (300_000, 517, 7), (1201, 57_856, 2500), (1201, 28_928, 2500),
                                              (1201, 57_857, 2500)])
def test_products_with_the_vector_in_shared_memory(cuda, n_row, n_col, mean, homo, dtype):
  rng = np.random.default_rng(17)
  lens = rng.poisson(mean, n_row)
  lens[[0, 5, n_row - 1]] = 0, 3 * mean, 1
  lens[n_row // 2:n_row // 2 + 40] = 0
  lens[1] += (1 - int(lens.sum())) % 4          # 4 k + 1 entries
  data, indices, indptr, rng = cases.ragged_csr(lens, n_col, 19, dtype=dtype)
  data = data[:1] if homo else data
  d = [torch.as_tensor(a).to(cuda) for a in (data, indices, indptr)]
  for transpose in (False, True):
    x = rng.standard_normal(n_row if transpose else n_col).astype(dtype)
    got = bpl.csr_matvec(*d, torch.as_tensor(x).to(cuda), shape=(n_row, n_col), transpose=transpose).cpu().numpy()
    want = cpu.csr_matvec(data, indices, indptr, x, shape=(n_row, n_col), transpose=transpose)
    tol = 1e-5 if dtype == np.float32 else 1e-12
    np.testing.assert_allclose(got, want, rtol=10 * tol, atol=20 * tol * np.sqrt(max(mean, indices.size / n_col)))


@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
@pytest.mark.parametrize('homo', [False, True])
@pytest.mark.parametrize('n_row,n_col,mean', [(80_000, 60_000, 50), (16_000, 60_000, 400), (200_000, 47_000, 9)])
def test_products_that_sweep_a_longer_vector(cuda, n_row, n_col, mean, homo, dtype):
  """One lane, several lanes, less than a unit per row; unsorted rows, empty ones, a ragged end of the arrays."""
  g = torch.Generator(device='cuda').manual_seed(23)
  lens = torch.poisson(torch.full((n_row,), float(mean), device=cuda), generator=g).long()
  lens[torch.tensor([0, 7, n_row - 2], device=cuda)] = torch.tensor([0, 3 * mean + 1, 0], device=cuda)
  lens[1] += (3 - int(lens.sum())) % 8
  indptr = torch.cat([lens.new_zeros(1), lens.cumsum(0)]).int()
  indices = torch.randint(0, n_col, (int(lens.sum()),), dtype=torch.int32, device=cuda, generator=g)
  data = torch.randn(1 if homo else indices.shape[0], dtype=dtype, device=cuda, generator=g).requires_grad_(not homo)
  x = torch.randn(n_col, dtype=dtype, device=cuda, generator=g)
  y = bpl.csr_matvec(data, indices, indptr, x, shape=(n_row, n_col))
  row, col = sparse_ops.csr_to_coo(indices, indptr)
  want = torch.zeros(n_row, dtype=torch.float64, device=cuda).index_add_(0, row, (data.detach() * x[col]).double())
  tol = dict(rtol=1e-5, atol=1e-4) if dtype == torch.float32 else dict(rtol=1e-12, atol=1e-11)
  torch.testing.assert_close(y.detach().double(), want, **tol)
  if not homo:
    ct = torch.randn(n_row, dtype=dtype, device=cuda, generator=g)
    torch.testing.assert_close(torch.autograd.grad(y, data, ct)[0], ct[row] * x[col])


@pytest.mark.parametrize('dtype,bool_events', [(np.float32, True), (np.float32, False), (np.float64, True), (np.float64, False)])
@pytest.mark.parametrize('homo', [False, True])
@pytest.mark.parametrize('n_row,n_col,mean', [(9000, 2001, 333), (150_000, 33, 20), (2000, 1_000_003, 2500), (300, 517, 40),
                                              (5000, 250_000, 40)])
def test_event_gather_over_bits(cuda, n_row, n_col, mean, homo, dtype, bool_events):
  rng = np.random.default_rng(29)
  lens = rng.poisson(mean, n_row)
  lens[[0, 3, n_row - 1]] = 0, 2 * mean, 0
  lens[1] += (3 - int(lens.sum())) % 4
  data, indices, indptr, rng = cases.ragged_csr(lens, n_col, 31, dtype=dtype)
  data = -data[:1] if homo else data
  events = rng.random(n_col) < 0.3
  events = events if bool_events else (events * 2.5).astype(dtype)
  d = [torch.as_tensor(a).to(cuda) for a in (data, indices, indptr, events)]
  got = bpl.event_csr_matvec(*d, shape=(n_row, n_col)).cpu().numpy()
  want = cpu.event_csr_matvec(data, indices, indptr, events, shape=(n_row, n_col))
  if homo and dtype == np.float32:       # the reference counts in float64
    assert got.tobytes() == want.tobytes()
  else:
    tol = 1e-5 if dtype == np.float32 else 1e-12
    np.testing.assert_allclose(got, want, rtol=10 * tol, atol=20 * tol * np.sqrt(mean))


@pytest.mark.parametrize('homo', [True, False])
@pytest.mark.parametrize('bool_events', [True, False])
# events as bytes in shared memory: ragged ends, the most of them, one more (bits); few events
@pytest.mark.parametrize('n_row,n_col,mean', [(40_000, 8203, 60), (30_000, 131_072, 90), (30_000, 131_073, 90),
                                              (60_000, 2003, 64), (60_000, 2003, 63)])
def test_event_gather_over_bytes(cuda, n_row, n_col, mean, homo, bool_events):
  test_event_gather_over_bits(cuda, n_row, n_col, mean, homo, np.float32, bool_events)


@pytest.mark.parametrize('dtype,bool_events', [(np.float32, True), (np.float32, False), (np.float64, True)])
@pytest.mark.parametrize('homo', [False, True])
# small (one launch, columns owned by blocks): the most rows, long rows, many columns; few columns (sums in shared memory);
# few rows (straight from the events): one, a group more than the warps, long pieces
@pytest.mark.parametrize('n_row,n_col,mean', [(90_000, 2001, 250), (300_000, 701, 60), (1, 50, 20), (8192, 129, 9),
                                              (40, 700, 2500), (300, 70_001, 31), (9473, 3000, 8), (262_144, 5000, 7),
                                              (262_145, 5000, 7),
                                              (700, 40_000, 3000)])
def test_event_scatter(cuda, n_row, n_col, mean, homo, dtype, bool_events):
  rng = np.random.default_rng(37)
  lens = rng.poisson(mean, n_row)
  lens[n_row // 2:n_row // 2 + 3] = 0
  data, indices, indptr, rng = cases.ragged_csr(lens, n_col, 41, dtype=dtype)
  data = data[:1] if homo else data
  events = rng.random(n_row) < 0.1
  events[-1] = True
  events = events if bool_events else (events * 2.5).astype(dtype)
  d = [torch.as_tensor(a).to(cuda) for a in (data, indices, indptr, events)]
  for ev, host in ((d[3], events), (torch.zeros_like(d[3]), np.zeros_like(events))):
    got = bpl.event_csr_matvec(d[0], d[1], d[2], ev, shape=(n_row, n_col), transpose=True).cpu().numpy()
    want = cpu.event_csr_matvec(data, indices, indptr, host, shape=(n_row, n_col), transpose=True)
    tol = 1e-5 if dtype == np.float32 else 1e-12
    np.testing.assert_allclose(got, want, rtol=10 * tol, atol=20 * tol * np.sqrt(0.1 * indices.size / n_col + 1))


def test_silent_event_scatter_orders_its_zeros(cuda):
  """No row fires: the zeros must be there for a kernel behind the product that starts as early as it may."""
  n_row, n = 20_000, 3_000_000
  indptr = torch.arange(0, 4 * n_row + 1, 4, dtype=torch.int32, device=cuda)
  indices = torch.randint(0, n, (4 * n_row,), dtype=torch.int32, device=cuda)
  data, silent = torch.rand(4 * n_row, device=cuda), torch.zeros(n_row, dtype=torch.bool, device=cuda)
  params = bpl.LifExpParams(dt=0.1, tau_syn=[5.0], E_rev=[0.0], ext_input=20.0, V_rest=-60.0, V_th=-50.0, V_reset=-60.0, R=1.0,
                            tau=20.0, tau_ref=5.0)
  V, t_last, g = torch.full((n,), -55., device=cuda), torch.full((n,), -1e7, device=cuda), torch.zeros(n, device=cuda)
  spikes, spike_list = torch.empty(n, device=cuda), torch.empty(bpl.spike_list_bytes(n), dtype=torch.uint8, device=cuda)
  for _ in range(20):
    y = torch.full((n,), float('nan'), device=cuda)
    del y                                # its memory is the next result's
    y = bpl.event_csr_matvec(data, indices, indptr, silent, shape=(n_row, n), transpose=True)
    bpl.lif_exp_step(y, g, V, t_last, params, 0.0, spikes=spikes, spike_list=spike_list)
    assert torch.equal(g, torch.zeros_like(g))


@pytest.mark.filterwarnings('ignore')      # the tracer warns of the operators' checks
@pytest.mark.parametrize('op', ['csr', 'event', 'jit', 'jit_event', 'matmat'])
@pytest.mark.parametrize('grad', [False, True])
def test_traced_operators_take_new_inputs(cuda, op, grad):
  """A call recorded by torch.jit.trace runs again on the inputs it is given."""
  if grad and op == 'matmat':
    pytest.skip('no gradient')
  data, indices, indptr, rng = cases.csr_case((30, 40), 0.3, 11)
  data, indices, indptr = (torch.as_tensor(a).to(cuda) for a in (data, indices, indptr))
  conn = dict(conn_prob=0.2, seed=3)
  call = {'csr': lambda x: bpl.csr_matvec(data, indices, indptr, x, shape=(30, 40)),
          'event': lambda x: bpl.event_csr_matvec(data, indices, indptr, x, shape=(30, 40)),
          'jit': lambda x: bpl.matvec_prob_conn_homo_weight(x, 0.5, shape=(50, 40), **conn),
          'jit_event': lambda x: bpl.event_matvec_prob_conn_uniform_weight(x, w_low=0., w_high=1., shape=(50, 40), **conn),
          'matmat': lambda x: bpl.matmat_prob_conn_normal_weight(x.reshape(2, 20), w_mu=0., w_sigma=1., shape=(20, 30), **conn)}[op]
  x, other = (torch.as_tensor((rng.standard_normal(40) * (rng.random(40) < 0.5)).astype(np.float32)).to(cuda) for _ in range(2))
  traced = torch.jit.trace(call, x.clone().requires_grad_(grad), check_trace=False)
  torch.testing.assert_close(traced(other), call(other))


@pytest.mark.parametrize('op', ['csr', 'event', 'jit', 'step'])
def test_other_threads_run_while_the_launch_queue_is_full(cuda, op):
  """More launches than the queue of a stream holds, behind half a second of other work: the calls wait for room, and
  meanwhile a thread that needs the interpreter goes on."""
  data, indices, indptr, rng = cases.csr_case((30, 40), 0.3, 11)
  data, indices, indptr = (torch.as_tensor(a).to(cuda) for a in (data, indices, indptr))
  x = torch.rand(40, device=cuda)
  params = bpl.LifExpParams(dt=0.1, tau_syn=[5.0], E_rev=[0.0], ext_input=20.0, V_rest=-60.0, V_th=-50.0, V_reset=-60.0, R=1.0,
                            tau=20.0, tau_ref=5.0)
  y, g, V, t_last, spikes = (torch.zeros(40, device=cuda) for _ in range(5))
  spike_list = torch.empty(bpl.spike_list_bytes(40), dtype=torch.uint8, device=cuda)
  call = {'csr': lambda: bpl.csr_matvec(data, indices, indptr, x, shape=(30, 40)),
          'event': lambda: bpl.event_csr_matvec(data, indices, indptr, x, shape=(30, 40)),
          'jit': lambda: bpl.matvec_prob_conn_homo_weight(x, 0.5, conn_prob=0.2, shape=(50, 40), seed=3),
          'step': lambda: bpl.lif_exp_step(y, g, V, t_last, params, 0.0, spikes=spikes, spike_list=spike_list)}[op]
  call()
  torch.cuda.synchronize()
  gaps, stop = [], threading.Event()

  def beat():
    last = time.perf_counter()
    while not stop.is_set():
      time.sleep(0.001)
      now = time.perf_counter()
      gaps.append(now - last)
      last = now

  thread = threading.Thread(target=beat)
  thread.start()
  begin = time.perf_counter()
  torch.cuda._sleep(1_000_000_000)
  for _ in range(6000):
    call()
  took = time.perf_counter() - begin
  stop.set()
  thread.join()
  torch.cuda.synchronize()
  if took < 0.3:
    pytest.skip('the queue took every launch')
  assert max(gaps) < 0.15


@pytest.mark.parametrize('n_row,n_col,mean', [(300, 517, 40), (90_000, 2001, 250), (20_000, 9000, 20), (270_000, 5000, 3)])
def test_every_event_scatter_records_the_profile_events(cuda, n_row, n_col, mean):
  """One launch, sums in shared memory, straight from the events, from a list."""
  import ctypes
  from brainpylib_b200 import _lib
  indptr = torch.arange(0, n_row * mean + 1, mean, dtype=torch.int32, device=cuda)
  indices = torch.randint(0, n_col, (n_row * mean,), dtype=torch.int32, device=cuda)
  data, events = torch.rand(n_row * mean, device=cuda), torch.rand(n_row, device=cuda) < 0.1
  before, after = (torch.cuda.Event(enable_timing=True) for _ in range(2))
  before.record(), after.record()        # the events exist from their first record on
  torch.cuda.synchronize()
  idle = before.elapsed_time(after)
  lib = _lib.lib()
  lib.bpl_profile_scatter_events(ctypes.c_void_p(before.cuda_event), ctypes.c_void_p(after.cuda_event))
  try:
    bpl.event_csr_matvec(data, indices, indptr, events, shape=(n_row, n_col), transpose=True)
  finally:
    lib.bpl_profile_scatter_events(None, None)
  torch.cuda.synchronize()
  assert before.elapsed_time(after) != idle


# ---- rows of very different lengths: how long single rows are is not known to the rules, which see the mean only ----
def _skewed(n_row, n_col, lens, dtype, device, seed=43):
  g = torch.Generator(device=device).manual_seed(seed)
  lens = torch.as_tensor(lens, device=device).long()
  indptr = torch.cat([lens.new_zeros(1), lens.cumsum(0)]).int()
  indices = torch.randint(0, n_col, (int(lens.sum()),), dtype=torch.int32, device=device, generator=g)
  return torch.randn(indices.shape[0], dtype=dtype, device=device, generator=g), indices, indptr


def _one_long_row(n_row, nse):
  lens = np.full(n_row, nse // 2 // n_row)
  lens[n_row // 3] += nse // 2
  return lens


def _device_us(call, n=10):
  call()
  best = float('inf')
  for _ in range(5):
    begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    begin.record()
    for _ in range(n):
      call()
    end.record()
    end.synchronize()
    best = min(best, begin.elapsed_time(end) * 1e3 / n)
  return best


@pytest.mark.parametrize('homo', [False, True])
@pytest.mark.parametrize('n_row,n_col', [(4096, 1000), (64, 1000), (1, 30_000)])
def test_small_event_scatter_of_one_long_row(cuda, n_row, n_col, homo):
  """Half of the entries in one row; a wrong list would lose or repeat pieces.  One team alone walked it in 230 us or more."""
  data, indices, indptr = _skewed(n_row, n_col, _one_long_row(n_row, 150_000), torch.float32, cuda)
  weights = torch.full((1,), 0.5, device=cuda) if homo else data
  events = torch.rand(n_row, device=cuda, generator=torch.Generator(device=cuda).manual_seed(2)) < 0.2
  events[n_row // 3] = True
  call = lambda: bpl.event_csr_matvec(weights, indices, indptr, events, shape=(n_row, n_col), transpose=True)
  row, col = sparse_ops.csr_to_coo(indices, indptr)
  want = torch.zeros(n_col, dtype=torch.float64, device=cuda).index_add_(
    0, col, torch.where(events[row], weights.double().expand(indices.shape[0]), 0.))
  torch.testing.assert_close(call().double(), want, rtol=1e-5, atol=1e-4)
  assert _device_us(call) < 100.


def test_event_scatter_of_few_long_rows(cuda):
  """Enough warps for the pieces of the rows (a warp for four of them took twice as long as the list-driven product)."""
  n_row, n_col = 256, 300_000
  data, indices, indptr = _skewed(n_row, n_col, np.full(n_row, 78_125), torch.float32, cuda)
  row, col = sparse_ops.csr_to_coo(indices, indptr)
  events = torch.rand(n_row, device=cuda, generator=torch.Generator(device=cuda).manual_seed(2)) < 0.2
  call = lambda: bpl.event_csr_matvec(data, indices, indptr, events, shape=(n_row, n_col), transpose=True)
  want = torch.zeros(n_col, dtype=torch.float64, device=cuda).index_add_(0, col, torch.where(events[row], data.double(), 0.))
  torch.testing.assert_close(call().double(), want, rtol=1e-5, atol=1e-4)
  assert _device_us(call) < 85.


def _uneven(kind):
  if kind == 'shared':           # a block full of cut rows, one of several warps' worth, two for the block
    n_row, n_col, lens = 150_000, 3000, np.full(150_000, 20)
    block = (np.arange(n_row) // 8) % 148 == 5
    lens[np.flatnonzero(block)[::6][:160]] = 401
    lens[[7, 77_777]] = 30_011, 4099
  elif kind == 'shared_many':    # more rows for a block than it has room for
    n_row, n_col, lens = 150_000, 3000, np.full(150_000, 20)
    lens[np.flatnonzero((np.arange(n_row) // 8) % 148 == 5)[::6][:140]] = 4501
  elif kind == 'shared_few':     # fewer rows than warps, each long
    n_row, n_col, lens = 60, 9001, np.full(60, 8003)
    lens[5] = 0
  elif kind == 'bands':          # a whole block of long rows; one lane per row
    n_row, n_col, lens = 100_000, 60_000, np.full(100_000, 31)
    lens[256:384], lens[70_001] = 499, 59_999
  elif kind == 'bands_teams':    # several lanes per row
    n_row, n_col, lens = 16_000, 60_000, np.full(16_000, 401)
    lens[[3, 9000, 9001]] = 0, 50_003, 5400
  else:                          # plain: vector too long for shared memory, too few rows for the bands
    n_row, n_col, lens = 3000, 300_000, np.full(3000, 33)
    lens[[1, 2999]], lens[100:700] = 250_001, 1500
  return n_row, n_col, lens


@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
@pytest.mark.parametrize('homo', [False, True])
@pytest.mark.parametrize('kind', ['shared', 'shared_many', 'shared_few', 'bands', 'bands_teams', 'plain'])
def test_products_of_rows_of_very_different_lengths(cuda, kind, homo, dtype):
  n_row, n_col, lens = _uneven(kind)
  data, indices, indptr = _skewed(n_row, n_col, lens, dtype, cuda)
  data = data[:1].clone() if homo else data
  row, col = sparse_ops.csr_to_coo(indices, indptr)
  g = torch.Generator(device=cuda).manual_seed(47)
  w = data.double().expand(indices.shape[0])
  tol = dict(rtol=1e-5, atol=1e-3) if dtype == torch.float32 else dict(rtol=1e-12, atol=1e-10)
  for transpose in (False, True):
    n_in, n_out, src, dst = (n_row, n_col, row, col) if transpose else (n_col, n_row, col, row)
    x = torch.randn(n_in, dtype=dtype, device=cuda, generator=g)
    d = data.clone().requires_grad_(not homo)
    y = bpl.csr_matvec(d, indices, indptr, x, shape=(n_row, n_col), transpose=transpose)
    want = torch.zeros(n_out, dtype=torch.float64, device=cuda).index_add_(0, dst, w * x[src].double())
    torch.testing.assert_close(y.detach().double(), want, **tol)
    if not homo:
      ct = torch.randn(n_out, dtype=dtype, device=cuda, generator=g)
      torch.testing.assert_close(torch.autograd.grad(y, d, ct)[0], ct[dst] * x[src])
    events = x > 0.5
    y = bpl.event_csr_matvec(data, indices, indptr, events, shape=(n_row, n_col), transpose=transpose)
    want = torch.zeros(n_out, dtype=torch.float64, device=cuda).index_add_(0, dst, torch.where(events[src], w, 0.))
    torch.testing.assert_close(y.double(), want, **tol)


# Bounds several times above what the calls take, far below what the lanes of single rows would (0.9 to 7 ms).
@pytest.mark.parametrize('n_row,n_col,op,bound', [(100_000, 30_000, 'transposed', 350.), (100_000, 60_000, 'product', 350.),
                                                  (100_000, 60_000, 'gradient', 400.), (20_000, 300_000, 'gradient', 400.)])
def test_time_of_a_product_with_a_long_row(cuda, n_row, n_col, op, bound):
  lens = np.full(n_row, 2_000_000 // n_row)
  lens[n_row // 3] = min(n_col, 250_000)
  data, indices, indptr = _skewed(n_row, n_col, lens, torch.float32, cuda)
  x, xt = torch.rand(n_col, device=cuda), torch.rand(n_row, device=cuda)
  data.requires_grad_(op == 'gradient')
  y = bpl.csr_matvec(data, indices, indptr, x, shape=(n_row, n_col))
  call = {'transposed': lambda: bpl.csr_matvec(data, indices, indptr, xt, shape=(n_row, n_col), transpose=True),
          'product': lambda: bpl.csr_matvec(data, indices, indptr, x, shape=(n_row, n_col)),
          'gradient': lambda: torch.autograd.grad(y, data, xt, retain_graph=True)}[op]
  assert _device_us(call) < bound


def test_a_list_product_right_behind_the_gradient_of_its_weights(cuda):
  """The list product is a launch that may start early: behind the gradient of the weights alone, which it reads as constants, it
  starts when that has finished."""
  n_row, n_col = 40_000, 9001
  data, indices, indptr = _skewed(n_row, n_col, np.random.default_rng(4).poisson(90, n_row), torch.float32, cuda)
  row, col = sparse_ops.csr_to_coo(indices, indptr)
  p = bpl.LifExpParams(dt=0.1, tau_syn=[5.0], E_rev=[0.0])
  zeros, V = torch.zeros(n_row, device=cuda), torch.full((n_row,), -40., device=cuda)
  fired, spikes = bpl.lif_exp_step(zeros.clone(), zeros.clone(), V, torch.full_like(V, -1e7), p, 0.0)
  assert bool((fired > 0).all())
  data.requires_grad_(True)
  for turn in range(5):
    g = torch.Generator(device=cuda).manual_seed(turn)
    x, ct = torch.rand(n_col, device=cuda, generator=g), torch.rand(n_row, device=cuda, generator=g)
    y = bpl.csr_matvec(data, indices, indptr, x, shape=(n_row, n_col))
    out, junk = torch.zeros(n_col, device=cuda), torch.full_like(data, float('nan'))
    del junk                             # its memory is the gradient's
    weights, = torch.autograd.grad(y, data, ct)
    got = bpl.event_csr_matvec_from_list(weights, indices, indptr, spikes, out, shape=(n_row, n_col))
    want = torch.zeros(n_col, dtype=torch.float64, device=cuda).index_add_(0, col, ct.double()[row] * x.double()[col])
    torch.testing.assert_close(got.double(), want, rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize('events', [False, True])
def test_time_of_few_equal_rows(cuda, events):
  """Rows that are longer than a warp's share of all entries, because there are fewer rows than warps, but no longer than the
  others: as fast as a few more rows of as many entries in all (cut and walked twice: 2.0 times the time)."""
  def us(n_row, length, n_col=20_000):
    data, indices, indptr = _skewed(n_row, n_col, np.full(n_row, length), torch.float32, cuda)
    x = torch.rand(n_col, device=cuda)
    fires = x < 0.05
    if events:
      return _device_us(lambda: bpl.event_csr_matvec(data, indices, indptr, fires, shape=(n_row, n_col), transpose=False), 30)
    return _device_us(lambda: bpl.csr_matvec(data, indices, indptr, x, shape=(n_row, n_col)), 30)
  assert us(2000, 6000) < 1.2 * us(2400, 5000)


@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
@pytest.mark.parametrize('n_row,mean', [(30, 3000), (1700, 3000), (2000, 3000), (4800, 1500)])
def test_products_of_few_rows(cuda, n_row, mean, dtype):
  """Rows around the line from which they are cut: twice the mean, one entry less and more, far longer, empty.  Small whole numbers: the
  sums are exact."""
  n_col = 12_001
  rng = np.random.default_rng(mean + n_row)
  lengths = rng.poisson(mean, n_row)
  lengths[[0, 3, 9, 14, n_row // 2, n_row - 1]] = 2 * mean, 2 * mean + 1, 2 * mean - 1, 0, 11_000, 4 * mean
  data, indices, indptr = _skewed(n_row, n_col, lengths, dtype, cuda)
  data = torch.randint(-8, 9, data.shape, device=cuda, generator=torch.Generator(device=cuda).manual_seed(1)).to(dtype)
  row, col = sparse_ops.csr_to_coo(indices, indptr)
  for transpose in (False, True):
    src, dst = (row, col) if transpose else (col, row)
    n_in, n_out = (n_row, n_col) if transpose else (n_col, n_row)
    x = torch.randint(-4, 5, (n_in,), device=cuda, generator=torch.Generator(device=cuda).manual_seed(2)).to(dtype)
    for w in (data, data[:1]):
      want = torch.zeros(n_out, dtype=torch.float64, device=cuda).index_add_(0, dst, w.double() * x.double()[src])
      assert torch.equal(bpl.csr_matvec(w, indices, indptr, x, shape=(n_row, n_col), transpose=transpose).double(), want)
      want = torch.zeros(n_out, dtype=torch.float64, device=cuda).index_add_(0, dst, w.double() * (x > 0).double()[src])
      got = bpl.event_csr_matvec(w, indices, indptr, x > 0, shape=(n_row, n_col), transpose=transpose)
      assert torch.equal(got.double(), want)


@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
@pytest.mark.parametrize('transpose', [False, True])
# vector in shared memory with rows cut for warps and blocks, swept in bands by one lane and by several, neither; aligned or not
@pytest.mark.parametrize('kind', ['shared', 'shared_many', 'bands', 'bands_teams', 'plain'])
@pytest.mark.parametrize('front', [0, 5])
def test_both_gradients_at_once(cuda, kind, front, transpose, dtype):
  """One or two launches for both gradients; entries in front of and behind the matrix have the gradient zero."""
  n_row, n_col, lens = _uneven(kind)
  data, indices, indptr = _skewed(n_row, n_col, lens, dtype, cuda)
  pad = lambda a: torch.cat([a.new_zeros(front), a, a.new_zeros(front)])
  data, indices, indptr = pad(data).requires_grad_(True), pad(indices), indptr + front
  g = torch.Generator(device=cuda).manual_seed(51)
  x = torch.randn(n_row if transpose else n_col, dtype=dtype, device=cuda, generator=g).requires_grad_(True)
  y = bpl.csr_matvec(data, indices, indptr, x, shape=(n_row, n_col), transpose=transpose)
  ct = torch.randn(y.shape[0], dtype=dtype, device=cuda, generator=g)
  junk = [torch.full_like(data, float('nan')), torch.full_like(x, float('nan'))]
  del junk                               # their memory is the gradients'
  g_data, g_x = torch.autograd.grad(y, (data, x), ct)
  inner = slice(front, indices.shape[0] - front)
  want_data, want_x = _expected(data[inner], indices[inner], indptr - front, x, ct, (n_row, n_col), transpose)
  torch.testing.assert_close(g_data[inner], want_data.to(dtype))
  assert not g_data[:front].any() and not g_data[indices.shape[0] - front:].any()
  tol = dict(rtol=1e-5, atol=1e-3) if dtype == torch.float32 else dict(rtol=1e-12, atol=1e-10)
  torch.testing.assert_close(g_x.double(), want_x, **tol)


@pytest.mark.parametrize('homo', [True, False])
@pytest.mark.parametrize('mean', [60, 100, 200, 300, 500])         # 4, 8, 16, 16 and 32 lanes per row
def test_event_gather_of_doubles(cuda, mean, homo):
  test_event_gather_over_bits(cuda, 30_000, 3001, mean, homo, np.float64, True)


# One weight and few events: rows of 64 to 512 go to the plain kernel; 9001 events are too many for that.
@pytest.mark.parametrize('mean', [60, 100, 200, 300, 500])         # 4, 8, 16, 16 and 32 lanes per row
def test_event_gather_of_doubles_with_one_weight(cuda, mean):
  test_event_gather_over_bits(cuda, 30_000, 9001, mean, True, np.float64, True)


@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
@pytest.mark.parametrize('more', [0, 1])           # the longest vector beside which a block has 32 warps; one element more: 24
def test_products_by_more_and_fewer_warps(cuda, more, dtype):
  n_row, n_col = 40_000, 131 * 1024 // dtype.itemsize + more
  data, indices, indptr = _skewed(n_row, n_col, np.random.default_rng(3).poisson(130, n_row), dtype, cuda)
  data.requires_grad_(True)
  g = torch.Generator(device=cuda).manual_seed(9)
  tol = dict(rtol=1e-5, atol=1e-3) if dtype == torch.float32 else dict(rtol=1e-12, atol=1e-10)
  for transpose in (False, True):
    x = torch.randn(n_row if transpose else n_col, dtype=dtype, device=cuda, generator=g).requires_grad_(True)
    y = bpl.csr_matvec(data, indices, indptr, x, shape=(n_row, n_col), transpose=transpose)
    ct = torch.randn(y.shape[0], dtype=dtype, device=cuda, generator=g)
    row, col = sparse_ops.csr_to_coo(indices, indptr)
    src, dst = (row, col) if transpose else (col, row)
    want = torch.zeros_like(y, dtype=torch.float64).index_add_(0, dst, data.detach().double() * x.detach().double()[src])
    torch.testing.assert_close(y.detach().double(), want, **tol)
    for got, want in zip(torch.autograd.grad(y, (data, x), ct), _expected(data, indices, indptr, x, ct, (n_row, n_col), transpose)):
      torch.testing.assert_close(got.double(), want, **tol)


@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
@pytest.mark.parametrize('n_row,mean', [(60_000, 12), (40_000, 30), (30_000, 60), (30_000, 90), (15_000, 300), (9_000, 600), (2_000, 300)])
def test_products_by_lanes_per_row(cuda, n_row, mean, dtype):
  n_col = 3001
  rng = np.random.default_rng(mean)
  lengths = rng.poisson(mean, n_row)
  lengths[rng.integers(0, n_row, n_row // 50)] = 0
  lengths[[1, n_row // 2, n_row - 1]] = 70 * mean, 30_000, 65 * 32          # cut: for the warp, for the block, the last row
  data, indices, indptr = _skewed(n_row, n_col, lengths, dtype, cuda)
  row, col = sparse_ops.csr_to_coo(indices, indptr)
  g = torch.Generator(device=cuda).manual_seed(9)
  eps = torch.finfo(dtype).eps
  for transpose in (False, True):
    src, dst = (row, col) if transpose else (col, row)
    x = torch.randn(n_row if transpose else n_col, dtype=dtype, device=cuda, generator=g)
    for w in (data, data[:1]):
      y = bpl.csr_matvec(w, indices, indptr, x, shape=(n_row, n_col), transpose=transpose)
      terms = w.double() * x.double()[src]
      want, size = (torch.zeros_like(y, dtype=torch.float64).index_add_(0, dst, t) for t in (terms, terms.abs()))
      steps = torch.bincount(dst, minlength=y.shape[0]) + 1
      assert bool(((y.double() - want).abs() <= eps * steps * size).all())          # each term takes part in at most so many sums


@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
@pytest.mark.parametrize('n_row,mean', [(60_000, 12), (40_000, 30), (30_000, 60), (30_000, 90), (15_000, 300), (9_000, 600), (2_000, 300)])
def test_exact_products_by_lanes_per_row(cuda, n_row, mean, dtype):
  n_col = 3001
  rng = np.random.default_rng(mean)
  lengths = rng.poisson(mean, n_row)
  lengths[rng.integers(0, n_row, n_row // 50)] = 0
  lengths[[1, n_row // 2, n_row - 1]] = 70 * mean, 30_000, 65 * 32          # cut: for the warp, for the block, the last row
  _, indices, indptr = _skewed(n_row, n_col, lengths, dtype, cuda)
  row, col = sparse_ops.csr_to_coo(indices, indptr)
  g = torch.Generator(device=cuda).manual_seed(9)
  # small whole numbers, whose sums are exact in any order: one entry lost or taken twice shows
  data = torch.randint(1, 9, indices.shape, device=cuda, generator=g).to(dtype)
  for transpose in (False, True):
    src, dst = (row, col) if transpose else (col, row)
    x = torch.randint(1, 9, (n_row if transpose else n_col,), device=cuda, generator=g).to(dtype)
    for w in (data, data[:1]):
      y = bpl.csr_matvec(w, indices, indptr, x, shape=(n_row, n_col), transpose=transpose)
      want = torch.zeros_like(y, dtype=torch.float64).index_add_(0, dst, w.double() * x.double()[src])
      assert float(want.max()) < 1 << 24 and torch.equal(y.double(), want)
