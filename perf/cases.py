"""The work that users of this library give it, as timed cases.

Every case is one call (or one simulation or training step) through the public operators, on inputs drawn on the
GPU from a seed.  Six kinds of work, with the sizes of this repository's benchmark configurations in the middle of
their ranges:

  event_csr   a stored CSR matrix times a spike vector, the projection of a spiking network.  ``transpose=True`` is the
              forward direction of a simulator (spikes of the pre-synaptic neurons scattered onto their targets),
              ``transpose=False`` its gather form.  One weight per projection or one per synapse, 32- and 64-bit floats,
              boolean or float spikes, rows of equal length or of the ragged lengths that a fixed connection
              probability gives, with or without the prepared storage format (float or fixed-point sums)
  csr         a stored CSR matrix times a dense vector (rate models, currents), both orientations, alone or with the
              gradients of weights and vector, as in training
  jit_event   a connectivity that is generated on the fly instead of stored, times a spike vector, one stream per output
              (``outdim_parallel``) or one per input
  jit_dense   the same with a dense vector, alone or with the gradient of the vector (which walks the streams the
              other way)
  jit_matmat  a dense matrix times an on-the-fly connectivity
  network     one time step of a recurrent network of excitatory and inhibitory neurons: fused neuron update with spike
              list, then one list-driven product per population

Matrices follow the recipes of ``brainpylib_b200/workloads.py``, drawn on the GPU: targets uniform over the
post-synaptic neurons, row lengths fixed or Poisson (as a fixed connection probability gives), spikes Bernoulli.
"""
import math

import torch

import brainpylib_b200 as bpl

_DTYPES = {'float32': torch.float32, 'float64': torch.float64}
_BYTES = {'float32': 4, 'float64': 8}


def listed():
  return [
    # one projection of the 4000-neuron network example: the smallest call, called once per time step
    dict(name='small_scatter', kind='event_csr', n_pre=4000, n_post=4000, degree=80, ragged=True, sort=True, rate=0.05,
         weights='one', dtype='float32', events='bool', transpose=True, storage='csr'),
    # the benchmark workload: a million neurons, 1e9 synapses, 1 % firing; called as the reference is called
    dict(name='million_scatter', kind='event_csr', n_pre=1_000_000, n_post=1_000_000, degree=1000, ragged=False,
         sort=False, rate=0.01, weights='each', dtype='float32', events='float', transpose=True, storage='csr'),
    # the same simulation with the matrix prepared once, as a long run does
    dict(name='million_scatter_prepared', kind='event_csr', n_pre=1_000_000, n_post=1_000_000, degree=1000, ragged=False,
         sort=False, rate=0.01, weights='each', dtype='float32', events='float', transpose=True, storage='prepared'),
    # a medium projection between populations of unequal, odd sizes, in double precision
    dict(name='ragged_scatter_double', kind='event_csr', n_pre=30_011, n_post=20_023, degree=400, ragged=True, sort=True,
         rate=0.02, weights='each', dtype='float64', events='bool', transpose=True, storage='csr'),
    # the gather form over a whole matrix of 1e7 synapses
    dict(name='event_gather', kind='event_csr', n_pre=100_000, n_post=100_000, degree=100, ragged=False, sort=True,
         rate=0.05, weights='each', dtype='float32', events='bool', transpose=False, storage='csr'),
    # matrix times dense vector at the benchmark's size
    dict(name='csr_product', kind='csr', n_row=100_000, n_col=100_000, degree=100, ragged=False, dtype='float32',
         transpose=False, grad=False, storage='csr'),
    # one training step of a sparse layer: product, then the gradients of its weights and of its input
    dict(name='csr_training_step', kind='csr', n_row=60_013, n_col=45_007, degree=80, ragged=True, dtype='float32',
         transpose=False, grad=True, storage='csr'),
    # on-the-fly connectivity, a million neurons, 1e9 connections generated per call
    dict(name='jit_event_rows', kind='jit_event', weights='uniform', n_row=1_000_000, n_col=1_000_000, prob=0.001,
         rate=0.02, outdim_parallel=True),
    # the same network with one stream per input neuron: only the firing ones are walked
    dict(name='jit_event_columns', kind='jit_event', weights='normal', n_row=1_000_000, n_col=1_000_000, prob=0.001,
         rate=0.02, outdim_parallel=False),
    # dense input and its gradient, odd sizes
    dict(name='jit_training_step', kind='jit_dense', weights='homo', n_row=100_003, n_col=80_021, prob=0.005, grad=True,
         outdim_parallel=True),
    # the largest contraction: 256 rows through a 65536 x 65536 connectivity
    dict(name='jit_matmat', kind='jit_matmat', weights='normal', m=256, k=65_536, n=65_536, prob=0.01),
    # one time step of the 3200 + 800 neuron network example: latency and launches
    dict(name='network_step', kind='network', n_exc=3200, n_inh=800, degree=80, storage='csr'),
  ]


def _log(rng, lo, hi):
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
  kind = rng.choice(['event_csr', 'event_csr', 'csr', 'csr', 'jit_event', 'jit_dense', 'jit_matmat', 'network'])
  if kind == 'event_csr':
    n_pre, n_post, degree = _log(rng, 1000, 1_000_000), _log(rng, 1000, 1_000_000), _log(rng, 20, 1000)
    degree = max(1, min(degree, n_post // 4, 100_000_000 // n_pre))
    transpose = rng.random() < 0.75
    storage = rng.choice(['csr', 'csr', 'prepared', 'prepared_fixed']) if transpose else 'csr'
    dtype = 'float32' if storage != 'csr' else rng.choice(['float32', 'float32', 'float32', 'float64'])
    return dict(kind=kind, n_pre=n_pre, n_post=n_post, degree=degree, ragged=rng.random() < 0.5, sort=True,
                rate=math.exp(rng.uniform(math.log(0.002), math.log(0.1))),
                weights='each' if storage != 'csr' else rng.choice(['one', 'each', 'each']), dtype=dtype,
                events=rng.choice(['bool', 'float']), transpose=transpose, storage=storage)
  if kind == 'csr':
    n_row, n_col, degree = _log(rng, 1000, 400_000), _log(rng, 1000, 400_000), _log(rng, 20, 1000)
    degree = max(1, min(degree, n_col // 4, 20_000_000 // n_row))
    grad = rng.random() < 0.5
    dtype = rng.choice(['float32', 'float32', 'float32', 'float64'])
    storage = 'prepared' if dtype == 'float32' and not grad and rng.random() < 0.3 else 'csr'
    return dict(kind=kind, n_row=n_row, n_col=n_col, degree=degree, ragged=rng.random() < 0.5, dtype=dtype,
                transpose=rng.random() < 0.5, grad=grad, storage=storage)
  if kind in ('jit_event', 'jit_dense'):
    n_row, n_col = _log(rng, 3000, 1_000_000), _log(rng, 3000, 1_000_000)
    most = 200_000_000 if kind == 'jit_dense' else 1_000_000_000
    prob = min(_log(rng, 50, 1000) / n_col, 0.2, most / n_row / n_col)
    case = dict(kind=kind, weights=rng.choice(['homo', 'uniform', 'normal']), n_row=n_row, n_col=n_col, prob=prob)
    if kind == 'jit_event':
      return dict(case, rate=math.exp(rng.uniform(math.log(0.005), math.log(0.1))), outdim_parallel=rng.random() < 0.5)
    return dict(case, grad=rng.random() < 0.5, outdim_parallel=rng.random() < 0.5)
  if kind == 'jit_matmat':
    m, k, n = _log(rng, 8, 256), _log(rng, 2000, 65_536), _log(rng, 2000, 65_536)
    return dict(kind=kind, weights=rng.choice(['uniform', 'normal']), m=m, k=k, n=n,
                prob=math.exp(rng.uniform(math.log(0.002), math.log(0.01))))
  n = _log(rng, 4000, 400_000)
  degree = min(_log(rng, 50, 1000), n // 8, 100_000_000 // n)
  return dict(kind=kind, n_exc=n - n // 5, n_inh=n // 5, degree=degree, storage=rng.choice(['csr', 'prepared']))


# ---------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------
def _generator(seed):
  return torch.Generator(device='cuda').manual_seed(int(seed))


def _csr(g, n_row, n_col, degree, ragged, sort, rows=None):
  """``(indices, indptr)`` of ``degree`` entries per row: in every row, or (``ragged``) on average, dealt out to random
  rows of the range ``rows`` (default: all), which gives the lengths of a fixed connection probability."""
  if not ragged:
    indptr = torch.arange(0, n_row * degree + 1, degree, dtype=torch.int32, device='cuda')
    indices = torch.randint(0, n_col, (n_row, degree), dtype=torch.int32, device='cuda', generator=g)
    return (indices.sort(dim=1).values if sort else indices).reshape(-1), indptr
  lo, hi = rows or (0, n_row)
  nse = (hi - lo) * degree
  row = torch.randint(lo, hi, (nse,), device='cuda', generator=g)
  key = (row * n_col + torch.randint(0, n_col, (nse,), device='cuda', generator=g)).sort().values
  indptr = torch.zeros(n_row + 1, dtype=torch.int32, device='cuda')
  indptr[1:] = torch.cumsum(torch.bincount(key // n_col, minlength=n_row), 0)
  return (key % n_col).to(torch.int32), indptr


def _conn_seed(seed):
  return int(seed) * 2_654_435_761 % 100_000_000


def prepare(case, seed):
  return {'event_csr': _prepare_event_csr, 'csr': _prepare_csr, 'jit_event': _prepare_jit_event,
          'jit_dense': _prepare_jit_dense, 'jit_matmat': _prepare_jit_matmat, 'network': _prepare_network}[case['kind']](
            case, seed, _generator(seed))


def _prepare_event_csr(case, seed, g):
  dtype, shape = _DTYPES[case['dtype']], (case['n_pre'], case['n_post'])
  indices, indptr = _csr(g, *shape, case['degree'], case['ragged'], case['sort'])
  if case['weights'] == 'one':
    data = torch.tensor([0.6], dtype=dtype, device='cuda')
  else:
    data = torch.rand(indices.shape[0], dtype=dtype, device='cuda', generator=g)
  n_in = shape[0] if case['transpose'] else shape[1]
  events = torch.rand(n_in, device='cuda', generator=g) < case['rate']
  if case['events'] == 'float':
    events = events.to(dtype)
  prepared = None
  if case['storage'] != 'csr':
    prepared = bpl.prepare_event_csr(data, indices, indptr, shape=shape,
                                     accumulate='fixed' if case['storage'] == 'prepared_fixed' else 'float')
  return dict(kind='event_csr', data=data, indices=indices, indptr=indptr, events=events, shape=shape,
              transpose=case['transpose'], prepared=prepared)


def _prepare_csr(case, seed, g):
  dtype, shape = _DTYPES[case['dtype']], (case['n_row'], case['n_col'])
  indices, indptr = _csr(g, *shape, case['degree'], case['ragged'], True)
  data = torch.randn(indices.shape[0], dtype=dtype, device='cuda', generator=g)
  n_in, n_out = shape[::-1] if not case['transpose'] else shape
  vector = torch.rand(n_in, dtype=dtype, device='cuda', generator=g) * 2 - 1
  state = dict(kind='csr', data=data, indices=indices, indptr=indptr, vector=vector, shape=shape,
               transpose=case['transpose'], prepared=None, cotangent=None)
  if case['storage'] == 'prepared':
    state['prepared'] = bpl.csr_to_column_blocked(data, indices, indptr, shape=shape)
  if case['grad']:
    state['cotangent'] = torch.randn(n_out, dtype=dtype, device='cuda', generator=g)
    data.requires_grad_(True)
    vector.requires_grad_(True)
  return state


def _jit_args(case, seed):
  weights = {'homo': dict(weight=0.05), 'uniform': dict(w_low=-0.1, w_high=0.1), 'normal': dict(w_mu=0., w_sigma=0.01)}
  return dict(weights[case['weights']], conn_prob=case['prob'], seed=_conn_seed(seed))


def _prepare_jit_event(case, seed, g):
  events = torch.rand(case['n_col'], device='cuda', generator=g) < case['rate']
  op = {'homo': bpl.event_matvec_prob_conn_homo_weight, 'uniform': bpl.event_matvec_prob_conn_uniform_weight,
        'normal': bpl.event_matvec_prob_conn_normal_weight}[case['weights']]
  return dict(kind='jit_event', op=op, events=events, args=dict(_jit_args(case, seed), shape=(case['n_row'], case['n_col']),
                                                                outdim_parallel=case['outdim_parallel']))


def _prepare_jit_dense(case, seed, g):
  vector = torch.randn(case['n_col'], device='cuda', generator=g)
  op = {'homo': bpl.matvec_prob_conn_homo_weight, 'uniform': bpl.matvec_prob_conn_uniform_weight,
        'normal': bpl.matvec_prob_conn_normal_weight}[case['weights']]
  cotangent = None
  if case['grad']:
    cotangent = torch.randn(case['n_row'], device='cuda', generator=g)
    vector.requires_grad_(True)
  return dict(kind='jit_dense', op=op, vector=vector, cotangent=cotangent,
              args=dict(_jit_args(case, seed), shape=(case['n_row'], case['n_col']),
                        outdim_parallel=case['outdim_parallel']))


def _prepare_jit_matmat(case, seed, g):
  matrix = torch.randn((case['m'], case['k']), device='cuda', generator=g)
  op = {'uniform': bpl.matmat_prob_conn_uniform_weight, 'normal': bpl.matmat_prob_conn_normal_weight}[case['weights']]
  return dict(kind='jit_matmat', op=op, matrix=matrix, args=dict(_jit_args(case, seed), shape=(case['k'], case['n'])))


def _prepare_network(case, seed, g):
  """Conductance-based neurons around threshold; rows of the other population are empty in each projection."""
  n_exc, n_inh = case['n_exc'], case['n_inh']
  n = n_exc + n_inh
  shape = (n, n)
  projections = []
  for lo, hi, strength in ((0, n_exc, 0.6), (n_exc, n, 6.7)):
    indices, indptr = _csr(g, n, n, case['degree'], True, True, rows=(lo, hi))
    data = torch.rand(indices.shape[0], device='cuda', generator=g).add_(0.5).mul_(strength * 80 / case['degree'])
    if case['storage'] == 'prepared':
      projections.append((None, None, None, bpl.prepare_event_csr(data, indices, indptr, shape=shape)))
    else:
      projections.append((data, indices, indptr, None))
  params = bpl.LifExpParams(dt=0.1, tau_syn=[5.0, 10.0], E_rev=[0.0, -80.0], ext_input=20.0, V_rest=-60.0, V_th=-50.0,
                            V_reset=-60.0, R=1.0, tau=20.0, tau_ref=5.0)
  return dict(kind='network', projections=projections, shape=shape, params=params, t=0.0,
              V=torch.randn(n, device='cuda', generator=g).mul_(2).sub_(55), t_last=torch.full((n,), -1e7, device='cuda'),
              g=torch.zeros((2, n), device='cuda'), y=torch.zeros((2, n), device='cuda'),
              spikes=torch.zeros(n, device='cuda'),
              spike_list=torch.zeros(bpl.spike_list_bytes(n), dtype=torch.uint8, device='cuda'))


# ---------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------
def run(state):
  kind = state['kind']
  if kind == 'event_csr':
    return bpl.event_csr_matvec(state['data'], state['indices'], state['indptr'], state['events'], shape=state['shape'],
                                transpose=state['transpose'], prepared=state['prepared'])
  if kind == 'csr':
    y = bpl.csr_matvec(state['data'], state['indices'], state['indptr'], state['vector'], shape=state['shape'],
                       transpose=state['transpose'], prepared=state['prepared'])
    if state['cotangent'] is None:
      return y
    return [y, *torch.autograd.grad(y, (state['data'], state['vector']), state['cotangent'])]
  if kind == 'jit_event':
    return state['op'](state['events'], **state['args'])
  if kind == 'jit_dense':
    y = state['op'](state['vector'], **state['args'])
    if state['cotangent'] is None:
      return y
    return [y, *torch.autograd.grad(y, state['vector'], state['cotangent'])]
  if kind == 'jit_matmat':
    return state['op'](state['matrix'], **state['args'])
  bpl.lif_exp_step(state['y'], state['g'], state['V'], state['t_last'], state['params'], state['t'],
                   spikes=state['spikes'], spike_list=state['spike_list'])
  for channel, (data, indices, indptr, prepared) in enumerate(state['projections']):
    bpl.event_csr_matvec_from_list(data, indices, indptr, state['spike_list'], state['y'][channel], shape=state['shape'],
                                   prepared=prepared)
  state['t'] += state['params'].dt
  return [state['V'], state['t_last'], state['g'], state['y'], state['spikes']]


# ---------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how exact it is
# ---------------------------------------------------------------------------------------------------------
# Integer and float operations that one generated connection needs, whatever the implementation: the generator's state
# update (about 10), conversion, logarithm, quotient, rounding and position (about 8), test and sum.
_JIT_OPS = 20


def work(case):
  kind = case['kind']
  if kind == 'event_csr':
    size = _BYTES[case['dtype']]
    per_synapse = 6 if case['storage'] != 'csr' else 4 + (size if case['weights'] == 'each' else 0)
    n_in, n_out = (case['n_pre'], case['n_post']) if case['transpose'] else (case['n_post'], case['n_pre'])
    rows = case['n_pre'] * (case['rate'] if case['transpose'] else 1.0)
    active = case['n_pre'] * case['degree'] * case['rate']
    vectors = n_in * (1 if case['events'] == 'bool' else size) + n_out * size
    return dict(bytes=rows * (case['degree'] * per_synapse + 8) + vectors, flops=2 * active)
  if kind == 'csr':
    size = _BYTES[case['dtype']]
    nse, both = case['n_row'] * case['degree'], case['n_row'] + case['n_col']
    per_synapse = 6 if case['storage'] != 'csr' else 4 + size
    total = nse * per_synapse + 4 * case['n_row'] + both * size
    if not case['grad']:
      return dict(bytes=total, flops=2 * nse)
    # both gradients as well: cotangent in, weight and vector gradients out
    return dict(bytes=total + nse * size + both * size, flops=5 * nse)
  if kind == 'jit_event':
    walked = 1.0 if case['outdim_parallel'] else case['rate']
    return dict(bytes=case['n_col'] + 4 * case['n_row'], flops=case['n_row'] * case['n_col'] * case['prob'] * walked * _JIT_OPS)
  if kind == 'jit_dense':
    times = 2 if case['grad'] else 1
    return dict(bytes=times * 4 * (case['n_col'] + case['n_row']),
                flops=times * case['n_row'] * case['n_col'] * case['prob'] * _JIT_OPS)
  if kind == 'jit_matmat':
    connections = case['k'] * case['n'] * case['prob']
    return dict(bytes=4 * case['m'] * (case['k'] + case['n']), flops=connections * (2 * case['m'] + _JIT_OPS))
  # about 0.2 % of the neurons fire in a step; the neuron update reads and writes 13 floats per neuron
  n = case['n_exc'] + case['n_inh']
  return dict(bytes=52 * n + 0.002 * n * (8 * case['degree'] + 8), flops=30 * n + 0.004 * n * case['degree'])


def tolerance(case):
  # sums of up to some thousand products in another order
  return dict(rel=1e-12) if case.get('dtype') == 'float64' else dict(rel=1e-5)
