"""FP64: where row blocks and where column blocks on DMMA run, and the addresses of pointer arrays,
which a warp loads all at once.

GPU tolerance: 1e-12 relative L2 norm, as for every FP64 kernel here.
"""
import numpy as np
import pytest

from oracle import cases, harness, multilinear
from tests.test_grouped_forms import chain

P, S = 'pointer_based', 'strided'
PRODUCTS = [   # m, k, n, add, row blocks
  (8, 66, 9, False, False), (16, 66, 12, False, False), (66, 40, 9, False, True), (121, 8, 9, False, False), (121, 16, 9, False, False),
  (121, 40, 9, False, True), (121, 8, 9, True, True), (41, 12, 9, False, False), (41, 12, 4, False, True), (65, 8, 4, False, False), (65, 8, 3, False, True), (122, 6, 9, False, False),
  (122, 20, 9, False, True), (64, 6, 9, False, True), (56, 56, 9, False, True)]
CASES = {   # pointer arrays: several elements per warp, one warp per eight elements, tiles of many elements
  '8x8x9_chain': lambda ns: _ptr_chain(ns, 8, 9, 3),
  '17x17x6_chain': lambda ns: _ptr_chain(ns, 17, 6, 2),
  '56x56x9': lambda ns: cases.plain_gemm(ns),
  '5x24x4_add': lambda ns: cases.plain_gemm(ns, 5, 24, 4, P, P, add=True),
  '12x3x7': lambda ns: cases.plain_gemm(ns, 12, 31, 7, P, S),
}


def _ptr_chain(ns, b, q, terms):
  return cases.volume_chain(ns, b, q, terms=terms, s_nnz=q, q_addr=P, s_addr=P, out_addr=P)


def _generate(descrs):
  from tensorforge_b200.kernels import Context, FP, Generator, Options
  g = Generator(descrs, Context('sm_100a', 'cuda', FP['double'], Options()))
  g.generate()
  return g


def generate(name):
  return _generate(CASES[name](cases.ns_from_module('tensorforge_b200')))


@pytest.mark.parametrize('m,k,n,add,rows', PRODUCTS)
def test_form_of_a_product(m, k, n, add, rows):
  g = _generate(cases.plain_gemm(cases.ns_from_module('tensorforge_b200'), m, k, n, S, S, add=add))
  assert ('mc' in g.get_plan().params) == rows


@pytest.mark.parametrize('b,q,rows', [(16, 27, False), (24, 20, True), (56, 9, True)])
def test_form_of_a_chain(b, q, rows):
  g = _generate(chain(cases.ns_from_module('tensorforge_b200'), b, q, 0.45))
  assert ('mc' in g.get_plan().params) == rows


@pytest.mark.parametrize('name', CASES)
def test_addresses_before_copies(name):
  """Where a warp takes more than two elements, every pointer array is read before the tile's first copy."""
  g = generate(name)
  assert 'mc' in g.get_plan().params
  text = g.get_source()
  te, threads = g.get_plan().params['tile_elements'], g.get_plan().threads
  assert ('__shfl_sync' in text) == (32 * te > 2 * threads) == (name != '56x56x9')
  if name == '56x56x9':
    return
  fetch = text[text.index('const bool there = '):text.index('// this tile has landed')]
  last = max(i for i in range(len(fetch)) if fetch.startswith('= there ? ', i))
  assert last < fetch.index('copy') and '__shfl_sync' in fetch
  assert -(-te // (threads // 32)) <= 32


@pytest.mark.gpu
@pytest.mark.parametrize('name', CASES)
def test_matches_oracle(name):
  import torch
  from tensorforge_b200.runtime import compile_generator
  g = generate(name)
  k = compile_generator(g)
  for n, masked in ((1, False), (13, True), (1201, True), (5003, False)):
    lay, mem = harness.make_memory(g.descr_list, n, seed=n, dtype=np.float64)
    flags = harness.make_flags(n, 3) if masked else None
    dev, kw = {}, {'numElements': n, 'flags': None if flags is None else torch.tensor(flags.astype(np.int32), device='cuda')}
    for l in lay:
      dev[l.name] = kw[l.name] = torch.tensor(mem.buffers[l.name], device='cuda')
      if l.kind == 'ptr':
        kw[l.name] = torch.tensor(dev[l.name].data_ptr() + (l.starts - l.extra_offset) * 8, device='cuda')
      if l.kind != 'shared':
        kw[f'{l.name}_extraOffset'] = l.extra_offset
    k(**kw)
    torch.cuda.synchronize()
    multilinear.evaluate(g.descr_list, mem, n, flags=flags)
    for l in lay:
      got, ref = dev[l.name].cpu().numpy(), mem.buffers[l.name]
      assert np.linalg.norm(got - ref) <= 1e-12 * np.linalg.norm(ref), (l.name, n)
