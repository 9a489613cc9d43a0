"""GPU: the tiled generator against the FP64 oracle where its tiles, copies and epochs have
edges: extents that are not whole 16-byte units, sub-boxes, transposed and repeated operands,
temporaries, accumulated destinations, sparse operands, higher ranks, several lanes groups.

Tolerance: every result is a sum of at most 84 products of values in [-1, 1] (two such sums
in a row where there is a temporary), so its FP32 rounding error stays below
84 * 2^-24 = 5.0e-6 of the sum of magnitudes, typically ten times less; as in the reference's
suites 1e-5 of the output's largest magnitude is allowed (FP64: 1e-12).
"""
import numpy as np
import pytest

from oracle import cases, harness, multilinear

MM, ID = [[0, -1], [-1, 1]], [[0, 1], [0, 1]]


def _gemm(ns, m, k, n, target=MM, a='strided', b='strided', c='strided', add=False, sparse=None):
  shape = lambda t: [{0: m, 1: n, -1: k}[i] for i in t]
  sa, sb = shape(target[0]), shape(target[1])
  spp = lambda s, side: ns.ListSPP(cases.sparse_pattern(*s, 0.3, 5), tuple(s)) if sparse == side else None
  A = ns.Tensor(sa, ns.Addressing.str2addr(a), spp=spp(sa, 'a'))
  B = ns.Tensor(sb, ns.Addressing.str2addr(b), spp=spp(sb, 'b'))
  C = ns.Tensor([m, n], ns.Addressing.str2addr(c))
  return [ns.MultilinearDescr(ns.SubTensor(C), [ns.SubTensor(A), ns.SubTensor(B)], target, ID, add=add)]


def _two_terms(ns, m=13, q=6):
  """out = A1 B; out += A2 B: B is read again after a stage that wrote global memory."""
  S = ns.Addressing.STRIDED
  A1, A2, B, C = ns.Tensor([m, m], S), ns.Tensor([m, m], S), ns.Tensor([m, q], S), ns.Tensor([m, q], S)
  sub = ns.SubTensor
  return [ns.MultilinearDescr(sub(C), [sub(A1), sub(B)], MM, ID),
          ns.MultilinearDescr(sub(C), [sub(A2), sub(B)], MM, ID, add=True)]


def _written_then_read(ns):
  """C = A B; D += C E with C an output of its own: the second stage reads what the first wrote."""
  S = ns.Addressing.STRIDED
  A, B, E = ns.Tensor([9, 7], S), ns.Tensor([7, 12], S), ns.Tensor([12, 5], ns.Addressing.NONE)
  C, D = ns.Tensor([9, 12], S), ns.Tensor([9, 5], S)
  sub = ns.SubTensor
  return [ns.MultilinearDescr(sub(C), [sub(A), sub(B)], MM, ID),
          ns.MultilinearDescr(sub(D), [sub(C), sub(E)], MM, ID, add=True)]


def _rank4(ns):
  """D[i,j,l,p] = A[k,i] B[j,k,l] c[p]: rank 4, three operands, a transposed and a middle contraction."""
  S = ns.Addressing.STRIDED
  A, B, c = ns.Tensor([6, 11], S), ns.Tensor([5, 6, 3], S), ns.Tensor([2], ns.Addressing.NONE)
  D = ns.Tensor([11, 5, 3, 2], S)
  sub = ns.SubTensor
  return [ns.MultilinearDescr(sub(D), [sub(A), sub(B), sub(c)], [[-1, 0], [1, -1, 2], [3]],
                              [[0, 1], [0, 1, 2], [0]])]


def _two_indices(ns):
  """D[i,j] += A[i,k,l] B[l,k,j] s with both contracted indices in other orders."""
  S = ns.Addressing.STRIDED
  A, B, D = ns.Tensor([8, 5, 3], S), ns.Tensor([3, 5, 7], S), ns.Tensor([8, 7], S)
  s = ns.Tensor([], ns.Addressing.SCALAR)
  sub = ns.SubTensor
  return [ns.MultilinearDescr(sub(D), [sub(A), sub(B), sub(s)], [[0, -1, -2], [-2, -1, 1], []],
                              [[0, 1, 2], [0, 1, 2], []], add=True)]


def _boxes(ns, shape=24):
  BB, S = ns.BoundingBox, ns.Addressing.STRIDED
  A = ns.Tensor([shape, shape], S, BB([2, 4], [21, 15]))
  B = ns.Tensor([shape, shape], S, BB([4, 3], [15, 12]))
  C = ns.Tensor([shape, shape], S, BB([2, 3], [21, 12]))
  return [ns.GemmDescr(False, False, ns.SubTensor(A), ns.SubTensor(B), ns.SubTensor(C))]


def _sparse_reused(ns):
  """T = S1 B; U = S2 T; C = U: sparse boxes and temporaries share memory over their lives."""
  S = ns.Addressing.STRIDED
  sp = lambda seed: ns.ListSPP(cases.sparse_pattern(18, 18, 0.3, seed), (18, 18))
  S1, S2 = ns.Tensor([18, 18], S, spp=sp(1)), ns.Tensor([18, 18], S, spp=sp(2))
  B, C = ns.Tensor([18, 4], S), ns.Tensor([18, 4], S)
  sub = ns.SubTensor
  T = ns.generate_tmp_tensor([sub(S1), sub(B)], MM)
  U = ns.generate_tmp_tensor([sub(S2), sub(T)], MM)
  return [ns.MultilinearDescr(sub(T), [sub(S1), sub(B)], MM, ID),
          ns.MultilinearDescr(sub(U), [sub(S2), sub(T)], MM, ID),
          ns.MultilinearDescr(sub(C), [sub(U)], [[0, 1]], [[0, 1]])]


P = 'pointer_based'
CASES = {
  'odd': lambda ns: _gemm(ns, 33, 9, 11),
  'one_row': lambda ns: _gemm(ns, 1, 5, 3),
  'one_column_k1': lambda ns: _gemm(ns, 17, 1, 1),
  'whole_quads_ptr': lambda ns: _gemm(ns, 32, 20, 12, a=P, b=P, c=P),
  'atb': lambda ns: _gemm(ns, 10, 13, 9, target=[[-1, 0], [-1, 1]]),
  'abt_shared_b': lambda ns: _gemm(ns, 14, 7, 10, target=[[0, -1], [1, -1]], b='none'),
  'wide_shared_a': lambda ns: _gemm(ns, 35, 18, 40, a='none', c=P, add=True),
  'large': lambda ns: _gemm(ns, 84, 84, 30, add=True),
  'sparse_a_add': lambda ns: _gemm(ns, 20, 20, 9, sparse='a', add=True),
  'sparse_b_shared': lambda ns: _gemm(ns, 21, 10, 6, b='none', sparse='b'),
  'two_terms': _two_terms,
  'written_then_read': _written_then_read,
  'rank4': _rank4,
  'two_indices': _two_indices,
  'boxes': _boxes,
  'sparse_reused': _sparse_reused,
  'three_matrices': cases.three_matrices,
}
LANES = {'large': (None, 256), 'odd': (None, 64), 'three_matrices': (None, 128)}
PARAMS = [(name, fp, lanes) for name in CASES for fp in (('float', 'double') if name in ('odd', 'three_matrices', 'rank4') else ('float',))
          for lanes in LANES.get(name, (None,)) if fp == 'float' or lanes is None]


def generate(name, fp, lanes):
  from tensorforge_b200.common.basic_types import FloatingPointType
  from tensorforge_b200.common.context import Context, Options
  from tensorforge_b200.generators.generator import Generator
  ns = cases.ns_from_module('tensorforge_b200')
  variant = {'strategy': 'tiled'}
  if lanes:
    variant['threads_per_element'] = lanes
  ftype = FloatingPointType.FLOAT if fp == 'float' else FloatingPointType.DOUBLE
  g = Generator(CASES[name](ns), Context('sm_100a', 'cuda', ftype, Options(variant=variant)))
  g.generate()
  return g


@pytest.mark.parametrize('name,fp,lanes', PARAMS)
def test_regions_stay_inside_shared_memory(name, fp, lanes):
  """Regions that are live together do not overlap, and the layout fits the planned size."""
  g = generate(name, fp, lanes)
  from tensorforge_b200.codegen.tiled import Staging
  plan = g.get_plan()
  assert plan.strategy == 'tiled'
  s = Staging(g.get_chain(), bool(plan.params['stage_shared']))
  elem = [r for r in s.regions if r.where == 'elem']
  for i, r in enumerate(elem):
    assert r.offset % s.vec == 0 and r.offset + r.volume <= s.per_elem
    for q in elem[:i]:
      together = not (r.last < q.first or q.last < r.first)
      assert not (together and r.offset < q.offset + q.volume and q.offset < r.offset + r.volume)
  assert (s.shared + s.per_elem * plan.params['elements_per_block']) * 16 // s.vec <= plan.smem_bytes <= 227 * 1024


@pytest.mark.gpu
@pytest.mark.parametrize('name,fp,lanes', PARAMS)
def test_tiled_matches_oracle(name, fp, lanes):
  import torch
  from tensorforge_b200.runtime import compile_generator
  g = generate(name, fp, lanes)
  k = compile_generator(g)
  dtype, tol = (torch.float32, 1e-5) if fp == 'float' else (torch.float64, 1e-12)
  for n, masked in ((1, False), (7, True), (1537, True), (4099, False)):
    lay, mem = harness.make_memory(g.descr_list, n, seed=n, dtype=np.float32 if fp == 'float' else np.float64)
    flags = harness.make_flags(n, 3) if masked else None
    dev, kw = {}, {'numElements': n}
    if masked:
      kw['flags'] = torch.tensor(flags.astype(np.int32), device='cuda')
    for l in lay:
      if l.kind == 'scalar':
        kw[l.name] = mem.scalars[l.name]
        continue
      dev[l.name] = torch.tensor(mem.buffers[l.name], dtype=dtype, device='cuda')
      kw[l.name] = dev[l.name]
      if l.kind == 'strided':
        kw[f'{l.name}_extraOffset'] = l.extra_offset
      elif l.kind == 'ptr':
        size = dev[l.name].element_size()
        kw[l.name] = torch.tensor(dev[l.name].data_ptr() + (l.starts - l.extra_offset) * size, device='cuda')
        kw[f'{l.name}_extraOffset'] = l.extra_offset
    k(**kw)
    torch.cuda.synchronize()
    multilinear.evaluate(g.descr_list, mem, n, quirks=False, flags=flags)
    for l in lay:
      if l.kind != 'scalar':   # inputs unchanged, outputs right, nothing written outside the boxes
        ref = mem.buffers[l.name]
        assert np.abs(dev[l.name].double().cpu().numpy() - ref).max() <= tol * max(1e-30, np.abs(ref).max()), (l.name, n)
