"""GPU: the FP64 row-block form at the edges of its tiles: rows that are not whole blocks of
eight, contraction lengths that are not whole steps of four, odd slots (8-byte copies), batches
below one group of elements, masks, pointer arrays, accumulation; and the column-block form,
which stays for chains that do not fit, on the same inputs.

Tolerance: 1e-12 relative L2 norm, as for every FP64 kernel here (rounding alone gives 1e-15).
"""
import numpy as np
import pytest

from oracle import cases, harness, multilinear

P = 'pointer_based'
CASES = {
  '56x9': lambda ns: cases.build('chain_o6', ns),
  '35x9_ptr': lambda ns: cases.volume_chain(ns, 35, 9, q_addr=P, s_addr=P, out_addr=P),
  '20x27': lambda ns: cases.mixed_chain(ns, 20, 27),
  '10x9_dense': lambda ns: cases.build('chain_o3_dense', ns),
  'gemm_56x56x9_ptr': lambda ns: cases.plain_gemm(ns),
  'gemm_17x5x3_add': lambda ns: cases.plain_gemm(ns, 17, 5, 3, 'strided', 'strided', add=True),
  'gemm_9x7x4_ptr_add': lambda ns: cases.plain_gemm(ns, 9, 7, 4, P, P, add=True),
}


def generate(name, variant=None):
  from tensorforge_b200.kernels import Context, FP, Generator, Options
  g = Generator(CASES[name](cases.ns_from_module('tensorforge_b200')), Context('sm_100a', 'cuda', FP['double'], Options(variant=variant)))
  g.generate()
  return g


@pytest.mark.parametrize('name', CASES)
def test_plan_fits(name):
  p = generate(name).get_plan()
  assert p.strategy == 'dmma' and 'mc' in p.params
  assert p.smem_bytes <= 227 * 1024 and p.threads <= 1024


@pytest.mark.gpu
@pytest.mark.parametrize('name,variant', [(n, None) for n in CASES] + [('56x9', {'prefetch': 1}), ('gemm_17x5x3_add', {'prefetch': 1})])
def test_matches_oracle(name, variant):
  import torch
  from tensorforge_b200.runtime import compile_generator
  g = generate(name, variant)
  k = compile_generator(g)
  for n, masked in ((1, False), (13, True), (1201, True), (5003, False)):
    lay, mem = harness.make_memory(g.descr_list, n, seed=n, dtype=np.float64)
    flags = harness.make_flags(n, 3) if masked else None
    before = {l.name: mem.buffers[l.name].copy() for l in lay}
    dev, kw = {}, {'flags': None if flags is None else torch.tensor(flags.astype(np.int32), device='cuda')}
    for l in lay:
      dev[l.name] = torch.tensor(mem.buffers[l.name], device='cuda')
      kw[l.name] = dev[l.name]
      if l.kind == 'ptr':
        kw[l.name] = torch.tensor(dev[l.name].data_ptr() + (l.starts - l.extra_offset) * 8, device='cuda')
      if l.kind != 'shared':
        kw[f'{l.name}_extraOffset'] = l.extra_offset
    k(numElements=n, **kw)
    torch.cuda.synchronize()
    multilinear.evaluate(g.descr_list, mem, n, flags=flags)
    for l in lay:
      got, ref = dev[l.name].cpu().numpy(), mem.buffers[l.name]
      assert np.linalg.norm(got - ref) <= 1e-12 * np.linalg.norm(ref), (l.name, n)
      kept = ref == before[l.name]
      assert np.array_equal(got[kept], ref[kept]), (l.name, n)
