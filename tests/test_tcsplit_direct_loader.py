"""The direct TF32x3 form's loader where a tile mixes elements on and off the 16-byte grid: elements
off it are copied with ordinary stores, which have to be ordered before the warp's arrival and
before later bulk copies into the same stage.

GPU tolerance: 1e-6 relative L2 norm against the FP64 oracle, the TF32x3 bar.
"""
import numpy as np
import pytest

from oracle import cases, harness, multilinear

P = 'pointer_based'
CASES = {
  '56x56x9': lambda ns: cases.plain_gemm(ns, 56, 56, 9, P, P),
  '4x4x1': lambda ns: cases.plain_gemm(ns, 4, 4, 1, P, P),      # 128 elements per tile: several per lane
  '20x20x5_add': lambda ns: cases.plain_gemm(ns, 20, 20, 5, P, P, add=True),
}


def generate(name):
  from tensorforge_b200.kernels import Context, FP, Generator, Options
  g = Generator(CASES[name](cases.ns_from_module('tensorforge_b200')), Context('sm_100a', 'cuda', FP['float'], Options(precision='tf32x3')))
  g.generate()
  return g


@pytest.mark.parametrize('name', CASES)
def test_stores_are_ordered_before_the_arrival(name):
  g = generate(name)
  assert g.get_plan().params['form'] == 'direct'
  text = g.get_source()
  loader = text[text.index('unsigned mine = 0;'):text.index('bulk_load(dst + i')]
  steps = ['] = src[q];', 'fence_proxy_async()', '__syncwarp()', '__reduce_add_sync', 'mbar_arrive_expect_tx', '__syncwarp()']
  at = 0
  for step in steps:
    at = loader.index(step, at) + len(step)


@pytest.mark.gpu
@pytest.mark.parametrize('name', CASES)
@pytest.mark.parametrize('shifts', [(0, 4), (0, 4, 8, 12), (4,)], ids=['every_other', 'one_in_four_aligned', 'none_aligned'])
def test_mixed_alignment(name, shifts):
  """Element i starts shifts[i % len] bytes behind a 16-byte boundary."""
  import torch
  from tensorforge_b200.runtime import compile_generator
  g = generate(name)
  te = g.get_plan().params['te']
  n = min(148 * te * 9 + 5, 30_000)     # every stage of the ring is filled more than once
  lay, mem = harness.make_memory(g.descr_list, n, seed=11, extra_offsets=False)
  dev, kw = {}, {'numElements': n}
  for l in lay:
    if l.kind == 'ptr':   # slots on the 16-byte grid, each element `shift` values behind its slot's start
      slot = -(-l.slot // 4) * 4 + 4
      shift = np.array(shifts)[np.arange(n) % len(shifts)] // 4
      l.starts = np.random.default_rng(2).permutation(n).astype(np.int64) * slot + shift
      mem.buffers[l.name] = np.random.default_rng(3).uniform(-1, 1, n * slot).astype(np.float32).astype(np.float64)
      mem.starts[l.name] = l.starts
    dev[l.name] = kw[l.name] = torch.tensor(mem.buffers[l.name], dtype=torch.float32, device='cuda')
    if l.kind == 'ptr':
      kw[l.name] = torch.tensor(dev[l.name].data_ptr() + l.starts * 4, device='cuda')
  compile_generator(g)(**kw)
  torch.cuda.synchronize()
  multilinear.evaluate(g.descr_list, mem, n)
  for l in lay:
    got, ref = dev[l.name].double().cpu().numpy(), mem.buffers[l.name]
    assert np.linalg.norm(got - ref) <= 1e-6 * np.linalg.norm(ref), l.name
