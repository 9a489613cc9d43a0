"""GPU: column programs that loop over A (row blocks and row tiles) where they can go wrong:
row counts that are not whole 16-byte units, odd contraction lengths, tiles with idle threads,
batches smaller than a wave, masks, pointer arrays, accumulation, misaligned slots, and
non-finite inputs, which must not reach entries outside A's pattern.

Tolerance against the FP64 oracle: 1e-6 relative L2 norm, the bar of the repository's FP32
chains: sums of at most 3 x 84 products rounded once each give about sqrt(252) * 2^-24 = 9.5e-7
at worst with rounding errors of random sign.
"""
import numpy as np
import pytest

from oracle import cases, harness, multilinear

P = 'pointer_based'
ROWS = {   # name -> (chain builder, variant): row blocks, the planner's own choice
  '56x9': (lambda ns: cases.build('chain_o6', ns), {}),
  '35x9_ptr': (lambda ns: cases.volume_chain(ns, 35, 9, q_addr=P, s_addr=P, out_addr=P), {}),
  '84x9': (lambda ns: cases.mixed_chain(ns, 84, 9), {}),
  '10x9_dense': (lambda ns: cases.build('chain_o3_dense', ns), {}),
  'gemm_24x17x5_add': (lambda ns: cases.plain_gemm(ns, 24, 17, 5, 'strided', 'strided', add=True), {}),
  'gemm_13x7x3_ptr_add': (lambda ns: cases.plain_gemm(ns, 13, 7, 3, P, P, add=True), {'dense': 1}),
  'gemm_1x1x1': (lambda ns: cases.plain_gemm(ns, 1, 1, 1, 'strided', 'strided'), {'dense': 1}),
  'gemm_128x128x2': (lambda ns: cases.plain_gemm(ns, 128, 128, 2, 'strided', P), {}),
  'gemm_20x20x9_sparse': (lambda ns: cases.sparse_dense(ns), {}),
  # in pieces: one input buffer and four rows per thread; two rows, an odd number of blocks
  '84x27': (lambda ns: cases.mixed_chain(ns, 84, 27), {}),
  '21x27_ptr': (lambda ns: cases.volume_chain(ns, 21, 27, s_nnz=60, q_addr=P, s_addr=P, out_addr=P), {}),
  '10x27_one_buffer': (lambda ns: cases.mixed_chain(ns, 10, 27), {'threads': 64, 'buffers': 1}),
  # row tiles
  '84x27_tiles': (lambda ns: cases.mixed_chain(ns, 84, 27), {'threads': 256, 'rm': 12, 'rc': 5, 'te': 6}),
  '35x27_tiles': (lambda ns: cases.volume_chain(ns, 35, 27, s_nnz=60, q_addr=P, s_addr=P, out_addr=P),
                  {'threads': 128, 'rm': 12, 'rc': 6, 'te': 9}),
  '20x27_tiles_odd_groups': (lambda ns: cases.mixed_chain(ns, 20, 27), {'threads': 128, 'rm': 8, 'rc': 9, 'te': 14}),
  'gemm_33x18x40_dense_tiles': (lambda ns: cases.plain_gemm(ns, 33, 18, 40, 'strided', 'strided', add=True), {'dense': 1}),
  'gemm_64x30x32_dense_tiles_ptr': (lambda ns: cases.plain_gemm(ns, 64, 30, 32, P, P), {'dense': 1}),
  '56x32_tiles': (lambda ns: cases.volume_chain(ns, 56, 32, s_nnz=300), {}),
}


def generate(name, more=None):
  from tensorforge_b200.common.basic_types import FloatingPointType
  from tensorforge_b200.common.context import Context, Options
  from tensorforge_b200.generators.generator import Generator
  build, variant = ROWS[name]
  variant = dict(variant, **(more or {}))
  ns = cases.ns_from_module('tensorforge_b200')
  g = Generator(build(ns), Context('sm_100a', 'cuda', FloatingPointType.FLOAT,
                                   Options(variant=dict(variant, strategy='colprog') if variant else None)))
  g.generate()
  return g


def unrolled(name):
  build, _ = ROWS[name]
  from tensorforge_b200.kernels import Context, FP, Generator, Options
  g = Generator(build(cases.ns_from_module('tensorforge_b200')),
                Context('sm_100a', 'cuda', FP['float'], Options(variant={'strategy': 'colprog', 'dense': 0})))
  g.generate()
  return g


@pytest.mark.parametrize('name', ROWS)
def test_planned_as_rows_within_shared_memory(name):
  p = generate(name).get_plan()
  assert p.strategy == 'colprog' and p.params['a_source'] == 'dense'
  assert ('rc' in p.params) == ('tiles' in name)
  assert p.smem_bytes <= 227 * 1024


@pytest.mark.parametrize('m,k,n,density,terms,rows', [
  (56, 56, 9, 1, 1, True), (56, 56, 9, 0.2, 1, False), (18, 61, 9, 1, 1, False), (20, 20, 9, 0.3, 1, True), (81, 62, 9, 0.7, 1, True),
  (56, 56, 9, 0.45, 3, True), (56, 56, 9, 0.2, 3, False), (20, 20, 9, 0.2, 3, True), (84, 84, 9, 0.31, 3, True), (35, 35, 20, 0.45, 3, False),
  (128, 128, 9, 0.25, 6, True)])
def test_rows_where_looping_over_zeros_pays(m, k, n, density, terms, rows):
  from types import SimpleNamespace as NS
  from tensorforge_b200.plan.chains import loops_pay
  term = NS(K=k, A=NS(storage_size=lambda: int(density * m * k)))
  assert loops_pay(NS(M=m, N=n, terms=[term] * terms), 7 if n == 20 else n) == rows


def _arguments(g, lay, mem, flags):
  import torch
  dev, kw = {}, {'flags': None if flags is None else torch.tensor(flags.astype(np.int32), device='cuda')}
  for l in lay:
    dev[l.name] = torch.tensor(mem.buffers[l.name], dtype=torch.float32, device='cuda')
    kw[l.name] = dev[l.name]
    if l.kind == 'strided':
      kw[f'{l.name}_extraOffset'] = l.extra_offset
    elif l.kind == 'ptr':
      kw[l.name] = torch.tensor(dev[l.name].data_ptr() + (l.starts - l.extra_offset) * 4, device='cuda')
      kw[f'{l.name}_extraOffset'] = l.extra_offset
  return dev, kw


@pytest.mark.gpu
@pytest.mark.parametrize('name', ROWS)
def test_rows_match_oracle(name):
  import torch
  from tensorforge_b200.runtime import compile_generator
  g = generate(name)
  k = compile_generator(g)
  for n, masked in ((1, False), (37, True), (1999, True), (6007, False)):
    lay, mem = harness.make_memory(g.descr_list, n, seed=n)
    flags = harness.make_flags(n, 3) if masked else None
    before = {l.name: mem.buffers[l.name].copy() for l in lay}
    dev, kw = _arguments(g, lay, mem, flags)
    k(numElements=n, **kw)
    torch.cuda.synchronize()
    multilinear.evaluate(g.descr_list, mem, n, flags=flags)
    for l in lay:
      got, ref = dev[l.name].double().cpu().numpy(), mem.buffers[l.name]
      assert np.linalg.norm(got - ref) <= 1e-6 * np.linalg.norm(ref), (l.name, n)
      kept = ref == before[l.name]   # inputs, masked elements and the gaps between slots
      assert np.array_equal(got[kept], ref[kept]), (l.name, n)


@pytest.mark.gpu
@pytest.mark.parametrize('name', ['56x9', '35x9_ptr', 'gemm_20x20x9_sparse', '84x27', '21x27_ptr', '35x27_tiles'])
def test_non_finite_inputs_stay_inside_the_pattern(name):
  """The same entries are infinite, NaN or finite as with the unrolled program, which only ever
  touches A's stored entries."""
  import torch
  from tensorforge_b200.runtime import compile_generator
  g, u = generate(name), unrolled(name)
  n = 60
  lay, mem = harness.make_memory(g.descr_list, n, seed=8)
  q = next(l for l in lay if l.kind in ('strided', 'ptr') and l.tensor.direction.name == 'SOURCE')
  out = next(l for l in lay if l.kind != 'shared' and l.tensor.direction.name != 'SOURCE')
  rng = np.random.default_rng(3)
  vol = int(np.prod(q.tensor.shape))
  for e, v in zip(rng.permutation(n)[:12], [np.inf, -np.inf, np.nan] * 4):   # one entry per element
    mem.buffers[q.name][q.starts[e] + rng.integers(vol)] = v
  got = []
  for gen in (g, u):
    dev, kw = _arguments(gen, lay, mem, None)
    compile_generator(gen)(numElements=n, **kw)
    got.append(dev[out.name].double().cpu().numpy())
  torch.cuda.synchronize()
  a, b = got
  assert not np.isfinite(b).all() and np.isfinite(b).any()
  assert np.array_equal(np.isnan(a), np.isnan(b))
  assert np.array_equal(np.where(np.isinf(a), np.sign(a), 0), np.where(np.isinf(b), np.sign(b), 0))
  f = np.isfinite(a)
  assert np.linalg.norm(a[f] - b[f]) <= 2e-6 * np.linalg.norm(b[f])


def sources():
  """Every kernel source the tests above build (for building ahead of time)."""
  return ([generate(n).get_source() for n in ROWS]
          + [unrolled(n).get_source() for n in ('56x9', '35x9_ptr', 'gemm_20x20x9_sparse', '84x27', '21x27_ptr', '35x27_tiles')])
