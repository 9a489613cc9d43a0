"""Row blocks whose last rows are not whole: stores of four, two or one row at a time, accumulated
or not, aligned or not.

GPU tolerance: 1e-6 relative L2 norm against the FP64 oracle, as for the other row blocks.
"""
import numpy as np
import pytest

from oracle import cases, harness, multilinear

P, S = 'pointer_based', 'strided'
CASES = {f'{m}x{k}x{n}_{c}{"_add" if add else ""}': (m, k, n, c, add)
         for m, k, n in ((10, 13, 9), (22, 22, 12), (14, 20, 11), (9, 9, 9), (13, 24, 3), (12, 16, 5), (2, 70, 4), (3, 50, 2))
         for c, add in ((S, False), (S, True), (P, True))}


def generate(name):
  from tensorforge_b200.kernels import Context, FP, Generator, Options
  m, k, n, c, add = CASES[name]
  g = Generator(cases.plain_gemm(cases.ns_from_module('tensorforge_b200'), m, k, n, c, c, add=add),
                Context('sm_100a', 'cuda', FP['float'], Options(variant={'strategy': 'colprog', 'dense': 1})))
  g.generate()
  return g


@pytest.mark.parametrize('name', CASES)
def test_one_test_per_group_of_rows(name):
  """Accumulated outputs: whether rows exist is asked once for all columns, not between their loads and stores."""
  m, k, n, c, add = CASES[name]
  g = generate(name)
  assert g.get_plan().params['rows'] == 4
  tests = g.get_source().count('if (row + ')
  pieces = 0 if m % 4 == 0 else 2 + 4 if m % 2 == 0 else 4
  assert tests == pieces * (1 if add else n)


@pytest.mark.gpu
@pytest.mark.parametrize('name', CASES)
def test_matches_oracle(name):
  import torch
  from tensorforge_b200.runtime import compile_generator
  g = generate(name)
  k = compile_generator(g)
  for n, masked, offsets in ((1, False, False), (131, True, True), (1999, False, False), (6007, True, False)):
    lay, mem = harness.make_memory(g.descr_list, n, seed=n, extra_offsets=offsets)
    flags = harness.make_flags(n, 3) if masked else None
    before = {l.name: mem.buffers[l.name].copy() for l in lay}
    dev, kw = {}, {'numElements': n, 'flags': None if flags is None else torch.tensor(flags.astype(np.int32), device='cuda')}
    for l in lay:
      dev[l.name] = kw[l.name] = torch.tensor(mem.buffers[l.name], dtype=torch.float32, device='cuda')
      if l.kind != 'shared':
        kw[f'{l.name}_extraOffset'] = l.extra_offset
      if l.kind == 'ptr':
        kw[l.name] = torch.tensor(dev[l.name].data_ptr() + (l.starts - l.extra_offset) * 4, device='cuda')
    k(**kw)
    torch.cuda.synchronize()
    multilinear.evaluate(g.descr_list, mem, n, flags=flags)
    for l in lay:
      got, ref = dev[l.name].double().cpu().numpy(), mem.buffers[l.name]
      assert np.linalg.norm(got - ref) <= 1e-6 * np.linalg.norm(ref), (l.name, n)
      kept = ref == before[l.name]
      assert np.array_equal(got[kept], ref[kept]), (l.name, n)


@pytest.mark.parametrize('m,k,n,rows', [(10, 13, 9, True), (10, 13, 12, False), (20, 25, 12, False), (22, 22, 12, True), (20, 25, 9, True)])
def test_twelve_columns_need_an_even_contraction(m, k, n, rows):
  from tensorforge_b200.kernels import Context, FP, Generator, Options
  g = Generator(cases.plain_gemm(cases.ns_from_module('tensorforge_b200'), m, k, n, S, S), Context('sm_100a', 'cuda', FP['float'], Options()))
  g.generate()
  assert ('rows' in g.get_plan().params) == rows
