"""The unrolled column program's write-back where it branches: accumulated outputs (previous values
are loaded in batches), pointer arrays (groups of 16 or 32 lanes per element, addresses loaded
beforehand), element sizes that are not whole 16-byte units, many small elements per tile, masks,
columns too short for shared memory.

GPU tolerance: 1e-6 relative L2 norm against the FP64 oracle, as for the other FP32 column programs
(at most 24 products and the previous value per sum: sqrt(25) * 2^-24 = 3.0e-7).
"""
import numpy as np
import pytest

from oracle import cases, harness, multilinear

P, S = 'pointer_based', 'strided'
CASES = {f'{m}x{k}x{n}_{c}{"_add" if add else ""}': (m, k, n, c, add)
         for m, k, n in ((24, 17, 20), (35, 20, 3), (9, 11, 13), (33, 24, 1), (8, 8, 4), (16, 8, 128), (6, 12, 9), (8, 8, 3), (12, 5, 2))
         for c in (S, P) for add in (False, True)}


def generate(name):
  from tensorforge_b200.kernels import Context, FP, Generator, Options
  m, k, n, c, add = CASES[name]
  g = Generator(cases.plain_gemm(cases.ns_from_module('tensorforge_b200'), m, k, n, c, c, add=add),
                Context('sm_100a', 'cuda', FP['float'], Options(variant={'strategy': 'colprog', 'dense': 0})))
  g.generate()
  return g


@pytest.mark.parametrize('name', CASES)
def test_form(name):
  m, k, n, c, add = CASES[name]
  g = generate(name)
  text = g.get_source()
  assert g.get_plan().strategy == 'colprog' and 'rows' not in g.get_plan().params
  small = m < 8 or m * n < 32
  assert ('col[i] +=' in text) == (add and small)
  assert ('p[i] + ' in text) == (add and not small)      # a batch of previous values before the first store
  assert ('__shfl_sync' in text) == (c == P and not small)


def test_lanes_of_a_group_hold_the_addresses_of_all_its_elements():
  for threads in (128, 256):
    for n in range(1, threads + 1):
      te = threads // n
      lanes = 32 if 32 * te <= 4 * threads else 16
      assert -(-te * lanes // threads) <= lanes


@pytest.mark.gpu
@pytest.mark.parametrize('name', CASES)
def test_matches_oracle(name):
  import torch
  from tensorforge_b200.runtime import compile_generator
  g = generate(name)
  k = compile_generator(g)
  for n, masked, offsets in ((1, False, False), (131, True, True), (1999, False, False), (6007, True, False), (3001, False, True)):
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
