"""The tiled generator's copies of sub-boxes: a box whose padded shared-memory pitch happens to be
its source's leading dimension is not one run of memory (8 rows out of 12), and is copied column
by column.

GPU tolerance: 1e-5 (FP64: 1e-12) of the output's largest magnitude, as for the other cases of this
generator: at most 36 products of values in [-1, 1] per sum, so at most 36 * 2^-24 = 2.2e-6 of the
sum of magnitudes.
"""
import itertools

import numpy as np
import pytest

from oracle import cases, harness, multilinear

MM, ID = [[0, -1], [-1, 1]], [[0, 1], [0, 1]]


def _sub_rows(ns, rows, ld, lo=0, addr='strided', m=16, n=9, cols=None):
  """C[m, n] = A_e[m, rows] * B_e[lo : lo + rows, 0 : n], B stored with `ld` rows."""
  S, P = ns.Addressing.STRIDED, ns.Addressing.str2addr(addr)
  A, C = ns.Tensor([m, rows], S), ns.Tensor([m, n], S)
  B = ns.Tensor([ld, cols or n], P)
  box = ns.BoundingBox([lo, 0], [lo + rows, n])
  return [ns.MultilinearDescr(ns.SubTensor(C), [ns.SubTensor(A), ns.SubTensor(B, box)], MM, ID)]


def _rank3(ns, rows, ld):
  """C[i, j, l] = A[i, k] B[k, j, l] over the first `rows` rows of B."""
  S = ns.Addressing.STRIDED
  A, B, C = ns.Tensor([13, rows], S), ns.Tensor([ld, 4, 3], S), ns.Tensor([13, 4, 3], S)
  box = ns.BoundingBox([0, 0, 0], [rows, 4, 3])
  return [ns.MultilinearDescr(ns.SubTensor(C), [ns.SubTensor(A), ns.SubTensor(B, box)], [[0, -1], [-1, 1, 2]],
                              [[0, 1], [0, 1, 2]])]


CASES = {
  '8_of_12': (lambda ns: _sub_rows(ns, 8, 12), 'float'),
  '8_of_12_from_4_ptr': (lambda ns: _sub_rows(ns, 8, 12, 4, 'pointer_based'), 'float'),
  '32_of_36': (lambda ns: _sub_rows(ns, 32, 36), 'float'),
  '12_of_12_fewer_columns': (lambda ns: _sub_rows(ns, 12, 12, cols=11), 'float'),
  '4_of_6': (lambda ns: _sub_rows(ns, 4, 6), 'double'),
  '8_of_10_from_2': (lambda ns: _sub_rows(ns, 8, 10, 2), 'double'),
  'rank3_8_of_12': (lambda ns: _rank3(ns, 8, 12), 'float'),
}


def generate(name):
  from tensorforge_b200.kernels import Context, FP, Generator, Options
  build, fp = CASES[name]
  g = Generator(build(cases.ns_from_module('tensorforge_b200')), Context('sm_100a', 'cuda', FP[fp], Options()))
  g.generate()
  return g


def _offsets(sizes, strides):
  return [sum(i * s for i, s in zip(idx, strides)) for idx in itertools.product(*(range(n) for n in sizes))]


@pytest.mark.parametrize('name', CASES)
def test_linear_copies_cover_their_box(name):
  """Where the source copies a region as one run, its box is that run on both sides."""
  from tensorforge_b200.codegen.tiled import Staging
  g = generate(name)
  assert g.get_plan().strategy == 'tiled'
  s = Staging(g.get_chain(), bool(g.get_plan().params['stage_shared']))
  text, runs = g.get_source(), 0
  for r in s.regions:
    if r.kind == 'copy' and f'copy16({r.name} + q * {s.vec}u' in text:
      run = list(range(int(np.prod(r.sizes))))
      assert sorted(_offsets(r.sizes, r.strides)) == run and sorted(_offsets(r.sizes, r.src_strides)) == run, r.op.name
      runs += 1
  assert runs >= (1 if name == '8_of_12' else 0)   # A is whole there


@pytest.mark.gpu
@pytest.mark.parametrize('name', CASES)
@pytest.mark.parametrize('offsets', [False, True], ids=['aligned', 'offsets'])
def test_sub_boxes_match_oracle(name, offsets):
  import torch
  from tensorforge_b200.runtime import compile_generator
  g = generate(name)
  fp = CASES[name][1]
  dtype, tol = (torch.float32, 1e-5) if fp == 'float' else (torch.float64, 1e-12)
  n = 601
  lay, mem = harness.make_memory(g.descr_list, n, seed=5, extra_offsets=offsets, dtype=np.float32 if fp == 'float' else np.float64)
  dev, kw = {}, {'numElements': n}
  for l in lay:
    dev[l.name] = kw[l.name] = torch.tensor(mem.buffers[l.name], dtype=dtype, device='cuda')
    if l.kind in ('strided', 'ptr'):
      kw[f'{l.name}_extraOffset'] = l.extra_offset
    if l.kind == 'ptr':
      kw[l.name] = torch.tensor(dev[l.name].data_ptr() + (l.starts - l.extra_offset) * dev[l.name].element_size(), device='cuda')
  compile_generator(g)(**kw)
  torch.cuda.synchronize()
  multilinear.evaluate(g.descr_list, mem, n, quirks=False)
  for l in lay:
    ref = mem.buffers[l.name]
    assert np.abs(dev[l.name].double().cpu().numpy() - ref).max() <= tol * np.abs(ref).max(), l.name
