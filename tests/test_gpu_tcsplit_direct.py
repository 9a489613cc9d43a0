"""GPU: the direct TF32x3 form of a single product per element where it can go wrong: ragged
last tiles, fewer tiles than teams or stages, one element or one hundred and twenty-eight per
tile, contraction lengths that are not whole MMA steps, tensor memory used to the last column,
slots off the 16-byte grid, masks, accumulation, sparse A.

Tolerance: 1e-6 relative L2 norm against the FP64 oracle, the TF32x3 bar.
"""
import ctypes

import numpy as np
import pytest

from oracle import cases, harness, multilinear

P = 'pointer_based'
CASES = {
  '56x56x9_ptr': lambda ns: cases.plain_gemm(ns),
  '56x56x9': lambda ns: cases.plain_gemm(ns, addr_b='strided', addr_c='strided'),
  '20x20x9_sparse': lambda ns: cases.sparse_dense(ns),
  '64x64x5_add': lambda ns: cases.plain_gemm(ns, 64, 64, 5, 'strided', 'strided', add=True),
  '4x4x1_ptr': lambda ns: cases.plain_gemm(ns, 4, 4, 1, P, P),
  '36x12x100': lambda ns: cases.plain_gemm(ns, 36, 12, 100, 'strided', P),
  '128x20x8': lambda ns: cases.plain_gemm(ns, 128, 20, 8, P, 'strided', add=True),
}
FITS = [c for c in CASES if c != '128x20x8']


def generate(name, variant=None):
  from tensorforge_b200.kernels import Context, FP, Generator, Options
  g = Generator(CASES[name](cases.ns_from_module('tensorforge_b200')),
                Context('sm_100a', 'cuda', FP['float'], Options(precision='tf32x3', variant=variant)))
  g.generate()
  return g


@pytest.mark.parametrize('name', CASES)
def test_plan(name):
  p = generate(name).get_plan()
  assert (p.params.get('form') == 'direct') == (name in FITS)   # 2 x (2 x 24 + 2 x 128) columns are too many
  assert p.smem_bytes <= 227 * 1024


@pytest.mark.gpu
@pytest.mark.parametrize('offsets', [False, True], ids=['aligned', 'offsets'])
@pytest.mark.parametrize('name', FITS)
def test_matches_oracle(name, offsets):
  import torch
  from tensorforge_b200.runtime import compile_generator
  g = generate(name)
  k = compile_generator(g)
  te = g.get_plan().params['te']
  for n, masked in ((1, False), (te + 1, True), (148 * te * 2 + 3, False), (148 * te * 7 + te // 2 + 1, True)):
    n = min(n, 30_000)
    lay, mem = harness.make_memory(g.descr_list, n, seed=n, extra_offsets=offsets)
    flags = harness.make_flags(n, 3) if masked else None
    before = {l.name: mem.buffers[l.name].copy() for l in lay}
    dev, kw = {}, {'flags': None if flags is None else torch.tensor(flags.astype(np.int32), device='cuda')}
    for l in lay:
      dev[l.name] = torch.tensor(mem.buffers[l.name], dtype=torch.float32, device='cuda')
      kw[l.name] = dev[l.name]
      if l.kind == 'ptr':
        kw[l.name] = torch.tensor(dev[l.name].data_ptr() + (l.starts - l.extra_offset) * 4, device='cuda')
      if l.kind != 'shared':
        kw[f'{l.name}_extraOffset'] = l.extra_offset
    k(numElements=n, **kw)
    torch.cuda.synchronize()
    errf = getattr(ctypes.CDLL(k.so_path), f'tfb_kernel_error_{g.get_base_name()}')
    errf.argtypes = [ctypes.c_void_p]
    assert errf(None) == 0
    multilinear.evaluate(g.descr_list, mem, n, flags=flags)
    for l in lay:
      got, ref = dev[l.name].double().cpu().numpy(), mem.buffers[l.name]
      assert np.linalg.norm(got - ref) <= 1e-6 * np.linalg.norm(ref), (l.name, n)
      kept = ref == before[l.name]
      assert np.array_equal(got[kept], ref[kept]), (l.name, n)
