"""The ways a just-in-time product reads its input and gathers its sums (global memory, event bits, tiles of the vector,
tiles of the output) against the CPU oracle, at sizes around the edges of tiles and of the rules that choose.  The
oracle's logarithm may move single connections (it counts them); so many outputs may differ."""
import ctypes

import numpy as np
import pytest
import torch

import brainpylib_b200 as bpl
from oracle import cpu, draws
from test_native_path_gpu import _device_us

pytestmark = pytest.mark.gpu

KINDS = {'homo': (cpu.W_HOMO, 0., 0.), 'uniform': (cpu.W_UNIFORM, -0.1, 0.2), 'normal': (cpu.W_NORMAL, 0., 0.01)}


def _call(x, kind, prob, shape, rows, event, seed=77):
  kw = dict(conn_prob=prob, shape=shape, seed=seed, outdim_parallel=rows)
  name = ('event_' if event else '') + f'matvec_prob_conn_{kind}_weight'
  op = getattr(bpl, name)
  if kind == 'homo':
    return op(x, 1., **kw)
  return op(x, w_low=-0.1, w_high=0.1, **kw) if kind == 'uniform' else op(x, w_mu=0., w_sigma=0.01, **kw)


def _compare(cuda, x, kind, prob, shape, rows, event):
  k, w1, w2 = KINDS[kind]
  got = _call(torch.as_tensor(x).to(cuda), kind, prob, shape, rows, event).cpu().numpy()
  oracle = cpu.jitconn_event_matvec if event else cpu.jitconn_matvec
  want, info = oracle(x, kind=k, w1=w1, w2=w2, conn_prob=prob, shape=shape, seed=77, outdim_parallel=rows, return_info=True)
  scale = float(np.abs(want).max())
  bad = ~np.isclose(got, want, rtol=2e-5, atol=2e-5 * scale)
  assert bad.sum() <= 2 * info['fragile'], (int(bad.sum()), info['fragile'])


@pytest.mark.parametrize('kind', sorted(KINDS))
@pytest.mark.parametrize('dtype', [np.float32, np.float64])
# one tile, exactly two tiles, one element more than a tile of either type, few rows (read from global memory)
@pytest.mark.parametrize('shape,prob', [((3000, 901), 0.3), ((4000, 58113), 0.01), ((2500, 29057), 0.02), ((70, 40000), 0.01)])
def test_dense_rows(cuda, shape, prob, dtype, kind):
  x = np.random.default_rng(1).standard_normal(shape[1]).astype(dtype)
  _compare(cuda, x, kind, prob, shape, True, False)


@pytest.mark.parametrize('kind', sorted(KINDS))
@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
@pytest.mark.parametrize('shape,prob', [((901, 3000), 0.3), ((58113, 4000), 0.01), ((29057, 2500), 0.02)])
def test_dense_columns(cuda, shape, prob, dtype, kind):
  """Against the same streams (seed + column) a few columns at a time.  (One connection that the oracle moves would shift all
  that follow in its stream.)"""
  x = torch.randn(shape[1], dtype=dtype, generator=torch.Generator().manual_seed(2)).to(cuda)
  got = _call(x, kind, prob, shape, False, False).double()
  want = torch.zeros(shape[0], dtype=torch.float64, device=cuda)
  for lo in range(0, shape[1], 50):
    part = x[lo:lo + 50].contiguous()
    want += _call(part, kind, prob, (shape[0], part.shape[0]), False, False, seed=77 + lo).double()
  torch.testing.assert_close(got, want, rtol=1e-5, atol=1e-5 * float(want.abs().max()))


@pytest.mark.parametrize('kind', sorted(KINDS))
def test_dense_columns_against_the_oracle(cuda, kind):
  _compare(cuda, np.random.default_rng(2).standard_normal(400), kind, 0.4, (501, 400), False, False)


@pytest.mark.parametrize('kind', sorted(KINDS))
# eight lanes per stream and one, on both sides of the lines between them; a single stream; a last block of one stream
@pytest.mark.parametrize('streams,length,prob', [(1, 30_001, 0.01), (17, 3, 0.5), (2369, 901, 0.05), (4737, 500, 0.02),
                                                 (5921, 500, 0.02), (8881, 300, 0.05), (8880, 16_384, 0.001)])
def test_few_and_more_streams(cuda, streams, length, prob, kind):
  rng = np.random.default_rng(6)
  x = rng.standard_normal(length).astype(np.float32)
  _compare(cuda, x, kind, prob, (streams, length), True, False)
  _compare(cuda, x > 1., kind, prob, (streams, length), True, True)
  x = rng.standard_normal(streams).astype(np.float32)
  _compare(cuda, x, kind, prob, (length, streams), False, False)


@pytest.mark.parametrize('kind', sorted(KINDS))
# firing columns of a block: none or one, about as many as are walked by eight lanes each, all
@pytest.mark.parametrize('shape,prob,rate', [((900, 33), 0.1, 0.1), ((900, 33), 0.1, 1.0), ((500, 50_000), 0.02, 0.001),
                                             ((500, 50_000), 0.02, 0.04), ((500, 50_000), 0.02, 0.07)])
def test_event_columns(cuda, shape, prob, rate, kind):
  _compare(cuda, np.random.default_rng(7).random(shape[1]) < rate, kind, prob, shape, False, True)


@pytest.mark.parametrize('kind', sorted(KINDS))
@pytest.mark.parametrize('dtype', [torch.bool, torch.float32, torch.float64])
# events read 16 bytes at a time: fewer than that, ragged ends; several rounds of eight lanes; more columns than the SMs' lists hold
@pytest.mark.parametrize('shape,prob,rate', [((900, 1), 0.2, 1.0), ((900, 15), 0.1, 1.0), ((700, 2371), 0.05, 0.0), ((700, 2371), 0.05, 0.5),
                                             ((900, 40_009), 0.02, 1.0), ((5000, 40_009), 0.004, 0.9), ((300, 1_250_003), 0.02, 0.01)])
@pytest.mark.parametrize('offset', [0, 1])                # 1: events not 16-byte aligned
def test_event_columns_by_chunks(cuda, shape, prob, rate, offset, dtype, kind):
  """Against the dense product of the events as zeros and ones, which walks every column."""
  n_row, n_col = shape
  fires = torch.rand(n_col + offset, generator=torch.Generator().manual_seed(8)) < rate
  x = fires.to(dtype).to(cuda)[offset:]
  got = _call(x, kind, prob, shape, False, True).double()
  want = _call(x.double(), kind, prob, shape, False, False)
  torch.testing.assert_close(got, want, rtol=1e-5, atol=1e-5 * max(float(want.abs().max()), 1e-3))


def test_event_columns_of_a_matrix_without_columns(cuda):
  x = torch.zeros(0, dtype=torch.bool, device=cuda)
  junk = torch.full((501,), float('nan'), device=cuda)
  del junk                                                # its memory is the output's
  assert torch.equal(_call(x, 'uniform', 0.2, (501, 0), False, True), torch.zeros(501, device=cuda))


def test_time_of_event_columns_above_one_list(cuda):
  """A few more columns than lists of 8192 on 148 SMs: no second wave of blocks (1.05 times the time; with it, 1.55)."""
  def us(n_col):
    x = torch.rand(n_col, device=cuda, generator=torch.Generator(device=cuda).manual_seed(4)) < 0.02
    return _device_us(lambda: _call(x, 'normal', 0.001, (1_000_000, n_col), False, True))
  assert us(1_250_000) < 1.25 * us(1_200_000)


def test_time_of_event_columns_of_few_connections(cuda):
  """A stream of less than one connection is walked by one lane, into short outputs as into longer ones."""
  x = torch.rand(4_000_000, device=cuda, generator=torch.Generator(device=cuda).manual_seed(4)) < 0.1
  short, longer = (_device_us(lambda: _call(x, 'normal', 5e-5, (n_row, x.shape[0]), False, True)) for n_row in (3000, 4200))
  assert short < 1.25 * longer


@pytest.mark.parametrize('kind', sorted(KINDS))
@pytest.mark.parametrize('prob', [0.0019, 0.0021])        # 3.9 and 4.3 connections per stream: by one lane, by eight
def test_event_columns_around_the_line_of_connections(cuda, prob, kind):
  test_event_columns_by_chunks(cuda, (2048, 40_009), prob, 0.3, 0, torch.bool, kind)


# the largest number of columns; the first whose last chunk ends less than a round of loads before 2^32
@pytest.mark.parametrize('n_col', [(1 << 32) - 1, (1 << 32) - 16_383])
def test_event_columns_up_to_32_bits(cuda, n_col):
  """Firing columns at both ends and in between, against calls with each of them alone."""
  firing = [0, 8191, 1_000_003, (1 << 31) + 5, n_col - 8195, n_col - 2, n_col - 1]
  x = torch.zeros(n_col, dtype=torch.bool, device=cuda)
  x[firing] = True
  one = torch.ones(1, dtype=torch.bool, device=cuda)
  for kind in sorted(KINDS):
    got = _call(x, kind, 0.2, (501, n_col), False, True).double()
    want = sum(_call(one, kind, 0.2, (501, 1), False, True, seed=(77 + c) % (1 << 32)).double() for c in firing)
    torch.testing.assert_close(got, want, rtol=1e-5, atol=1e-6)


def _ends(n):
  return [*range(3), *range(n // 148 - 2, n // 148 + 2), n // 2, *range(n - 1030, n - 1020), *range(n - 3, n)]


@pytest.mark.parametrize('kind,event,prob', [('homo', True, 0.3), ('uniform', True, 0.3), ('uniform', False, 0.3), ('homo', False, 1e-6)])
def test_rows_up_to_32_bits(cuda, kind, event, prob):
  """The largest number of rows, by events in shared memory, by tiles, by gathers: single rows against calls with each of them alone."""
  n_row, n_col = (1 << 32) - 1, 11
  x = torch.arange(n_col, device=cuda) % 2 == 0 if event else torch.arange(1., n_col + 1., device=cuda)
  got = _call(x, kind, prob, (n_row, n_col), True, event)
  for row in _ends(n_row):
    torch.testing.assert_close(got[row:row + 1], _call(x, kind, prob, (1, n_col), True, event, seed=(77 + row) % (1 << 32)))


@pytest.mark.parametrize('n_row,prob', [(11, 0.02), (11, 1e-6)])        # by tiles, by reductions
def test_columns_up_to_32_bits(cuda, n_row, prob):
  n_col = (1 << 32) - 1
  x = torch.zeros(n_col, device=cuda)
  x[_ends(n_col)] = torch.arange(1., len(_ends(n_col)) + 1., device=cuda)
  got = _call(x, 'uniform', prob, (n_row, n_col), False, False)
  want = sum(_call(x[c:c + 1].clone(), 'uniform', prob, (n_row, 1), False, False, seed=(77 + c) % (1 << 32)) for c in _ends(n_col))
  torch.testing.assert_close(got, want, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize('kind', sorted(KINDS))
@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
def test_one_lane_per_stream_in_tiles(cuda, dtype, kind):
  """More streams than eight lanes each are given to, with too few connections for tiles: reductions and gathers."""
  test_dense_columns(cuda, (29_057, 8881), 0.01, dtype, kind)
  x = np.random.default_rng(1).standard_normal(58_113).astype(str(dtype)[6:])
  _compare(cuda, x, kind, 0.002, (6001, 58_113), True, False)


def _tiles(n, other, prob, size, columns):
  """The lines between the walks (jitconn_kernels.cu) for 148 SMs: whether one lane per stream works in tiles of the output
  (`columns`: n outputs, `other` streams) or of the vector (n inputs)."""
  per_sm, waves = n * other * prob / 148, -(-(-(-other // 148)) // 1024)
  if columns:
    return other > 60 * 148 and 1.8 * per_sm > 0.3 * (size // 4) * per_sm + 0.8 * (size // 4) * n * waves + 5000
  return other > 40 * 148 and 0.75 * per_sm > n * size / 56 * (1 if n * size <= 227 * 1024 else waves) + 2000


@pytest.mark.parametrize('kind', sorted(KINDS))
@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
# one tile, one element more, exactly two and one more, of either type
@pytest.mark.parametrize('n', [29_056, 29_057, 58_112, 58_113, 116_225])
def test_sums_in_tiles_of_the_output(cuda, n, dtype, kind):
  columns, prob, few = 12_001, 0.03, 4000           # `few` columns are too few: eight lanes each, reductions
  assert _tiles(n, columns, prob, dtype.itemsize, True) and few <= 32 * 148
  x = torch.randn(columns, dtype=dtype, generator=torch.Generator().manual_seed(2)).to(cuda)
  got = _call(x, kind, prob, (n, columns), False, False).double()
  want = torch.zeros(n, dtype=torch.float64, device=cuda)
  for lo in range(0, columns, few):
    part = x[lo:lo + few].contiguous()
    want += _call(part, kind, prob, (n, part.shape[0]), False, False, seed=77 + lo).double()
  torch.testing.assert_close(got, want, rtol=1e-5, atol=1e-5 * float(want.abs().max()))


@pytest.mark.parametrize('kind', sorted(KINDS))
@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
@pytest.mark.parametrize('n', [29_057, 58_112, 58_113])
def test_vector_in_tiles(cuda, n, dtype, kind):
  rows, prob, few = 6001, 0.02, 2000                # `few` rows: eight lanes each, or gathers from global memory
  assert _tiles(n, rows, prob, dtype.itemsize, False) and not _tiles(n, few, prob, dtype.itemsize, False)
  x = torch.randn(n, dtype=dtype, generator=torch.Generator().manual_seed(3)).to(cuda)
  got = _call(x, kind, prob, (rows, n), True, False)
  want = torch.cat([_call(x, kind, prob, (min(few, rows - lo), n), True, False, seed=77 + lo) for lo in range(0, rows, few)])
  torch.testing.assert_close(got, want, rtol=1e-5, atol=1e-5 * float(want.abs().max()))


@pytest.mark.parametrize('kind', sorted(KINDS))
@pytest.mark.parametrize('dtype', [np.bool_, np.float32])
# every input fires (full queues), ragged last word, more rows than threads, a mask of the largest size
@pytest.mark.parametrize('shape,prob,rate', [((5000, 1000), 0.1, 1.0), ((2111, 4097), 0.2, 0.1), ((160000, 333), 0.1, 0.02),
                                             ((12000, 1_638_400), 0.0004, 0.3), ((50, 3000), 0.1, 0.2)])
def test_event_rows(cuda, shape, prob, rate, dtype, kind):
  x = (np.random.default_rng(3).random(shape[1]) < rate).astype(dtype)
  _compare(cuda, x, kind, prob, shape, True, True)


@pytest.mark.parametrize('kind,most', [('homo', 227 * 1024), ('uniform', 179 * 1024), ('normal', 147 * 1024)])
@pytest.mark.parametrize('more', [0, 1])
def test_events_as_bytes_and_as_bits(cuda, kind, most, more):
  """The longest event vector that a walk keeps as bytes beside its queues, and the first that it keeps as bits; every input
  fires in half of the vector, so that queues fill."""
  x = np.random.default_rng(8).random(most + more) < 0.05
  x[:most // 2] = True
  _compare(cuda, x, kind, 0.001, (9001, most + more), True, True)


@pytest.mark.parametrize('n_row', [12_001, 160_001])       # 512 threads, 1024
@pytest.mark.parametrize('n_col', [1_269_760, 1_269_761, 1_466_369, 1_638_400])
def test_queues_beside_long_masks(cuda, n_row, n_col):
  """The longest mask beside which 1024 threads have queues for batches of eight, and longer ones with queues of six for 1024 and
  for fewer threads; half of the vector fires, so that they fill."""
  x = np.random.default_rng(10).random(n_col) < 0.05
  x[:n_col // 2] = True
  _compare(cuda, x, 'normal', 1.2e-4 if n_row < 100_000 else 4e-5, (n_row, n_col), True, True)


def test_time_of_event_rows_beside_long_masks(cuda):
  """The masks that leave too little for queues of batches of eight cost no wave of rows (1.05 times the time; with it, 1.25)."""
  def us(n_col):
    x = torch.rand(n_col, device=cuda, generator=torch.Generator(device=cuda).manual_seed(4)) < 0.02
    return _device_us(lambda: _call(x, 'normal', 0.001, (300_000, n_col), True, True))
  assert us(1_300_000) < 1.15 * us(1_250_000)


@pytest.mark.parametrize('prob', [1.22e-5, 1.2e-5])      # the last mean gap whose positions bits keep in 24 bits; one beyond
def test_events_as_bits_far_apart(cuda, prob):
  n = 1_638_400
  assert (n + 8 * 23 / prob < 1 << 24) == (prob == 1.22e-5)
  _compare(cuda, np.random.default_rng(9).random(n) < 0.5, 'homo', prob, (250_000, n), True, True)


@pytest.mark.parametrize('prob', [6e-6, 2e-5, 1.0])      # outside the quick test's range, sparse, every position
def test_probabilities_at_the_ends_of_the_range(cuda, prob):
  shape = (600, 200) if prob == 1.0 else (600, 300_000)
  ev = np.random.default_rng(4).random(shape[1]) < 0.5
  for kind in KINDS:
    _compare(cuda, ev, kind, prob, shape, True, True)
    _compare(cuda, ev.astype(np.float32), kind, prob, shape, True, False)


@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
# X staged in shared memory (many columns: one tile, a ragged last tile, the ring going round), X read from L2 with 32, 64
# and 128 rows per warp
@pytest.mark.parametrize('m,k,n,prob', [(33, 383, 30_000, 0.05), (70, 2500, 25_001, 0.02), (7, 1537, 40_000, 0.1),
                                        (31, 5000, 300, 0.01), (50, 5000, 300, 0.01), (150, 5000, 300, 0.01)])
def test_matmat_from_lists_equals_the_inline_kernel(cuda, m, k, n, prob, dtype):
  from brainpylib_b200 import jitconn_ops
  X = torch.randn(m, k, dtype=dtype, generator=torch.Generator().manual_seed(5)).to(cuda)
  kw = dict(kind='normal', w1=0., w2=0.01, conn_prob=prob, shape=(k, n), seed=11)
  assert torch.equal(jitconn_ops.matmat_raw(X, **kw), jitconn_ops.matmat_raw(X, workspace=False, **kw))


@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
# tiles of 384 (float64: 192) positions, a ring of four: one, one and a position, the whole ring, the first tile behind it
@pytest.mark.parametrize('k', [192, 193, 384, 385, 768, 769, 1536, 1537, 3073])
def test_matmat_at_the_edges_of_tiles(cuda, k, dtype):
  from brainpylib_b200 import jitconn_ops
  X = torch.randn(34, k, dtype=dtype, generator=torch.Generator().manual_seed(6)).to(cuda)
  kw = dict(kind='uniform', w1=-0.1, w2=0.2, conn_prob=0.03, shape=(k, 20_001), seed=12)
  assert torch.equal(jitconn_ops.matmat_raw(X, **kw), jitconn_ops.matmat_raw(X, workspace=False, **kw))


@pytest.mark.parametrize('prob', [0.3, 0.01, 0.001, 5.7e-6])
def test_gaps_of_all_draws(cuda, prob):
  """The two-sided test of a gap rests on measured errors of the logarithms: over all 2^32 draws it gives the reference's gap."""
  from brainpylib_b200 import _lib
  fn = _lib.lib().bpl_jit_gap_mismatches
  fn.argtypes, fn.restype = [ctypes.c_void_p, ctypes.c_double, ctypes.c_void_p], ctypes.c_int
  wrong = torch.zeros(1, dtype=torch.int64, device=cuda)
  assert fn(torch.cuda.current_stream().cuda_stream, float(np.float32(np.log1p(-prob))), wrong.data_ptr()) == 1
  assert int(wrong) == 0


def test_errors_of_the_logarithms(cuda):
  """The bound that the ends of a gap take, over all 2^32 draws: for every probability."""
  assert 0.5 < draws.log_error() < 1


@pytest.mark.parametrize('kind', [0, 1, 2])               # homogeneous, uniform, normal
# batches of event walks (bits: positions in 24 bits, and bytes), of tiles, of the others
@pytest.mark.parametrize('per_batch,sums,low24', [(8, True, True), (8, True, False), (4, True, True), (6, True, False), (4, False, False)])
@pytest.mark.parametrize('prob,n', [(0.9, 3000), (0.01, 40_000), (0.001, 1_638_400), (1.22e-5, 1_638_400)])
def test_batches_of_a_stream(cuda, prob, n, per_batch, sums, low24, kind):
  """Positions and raw draws of batches, bit for bit, against one connection at a time by the reference's expression."""
  connections, wrong = draws.batch_mismatches(kind, per_batch, sums, low24, float(np.float32(np.log1p(-prob))), 77, 20_000, n)
  assert wrong == 0 and connections > 0.8 * 20_000 * n * prob
