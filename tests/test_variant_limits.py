"""Variants asked for through Options that lie outside what a form can run."""
import pytest

from oracle import cases


def plan(descrs, variant, precision='plain', fp='float'):
  from tensorforge_b200.kernels import Context, FP, Generator, Options
  g = Generator(descrs(cases.ns_from_module('tensorforge_b200')), Context('sm_100a', 'cuda', FP[fp], Options(precision=precision, variant=variant)))
  g.generate()
  return g


def _small(ns):
  S, sub = ns.Addressing.STRIDED, ns.SubTensor
  A, B, C = ns.Tensor([4, 5], S), ns.Tensor([5, 3], S), ns.Tensor([4, 3], S)
  return [ns.MultilinearDescr(sub(C), [sub(A), sub(B)], [[0, -1], [-1, 1]], [[0, 1], [0, 1]])]


@pytest.mark.parametrize('lanes,elements', [(32, 64), (32, 33), (32, 32), (64, 64), (1024, 2)])
@pytest.mark.parametrize('fp', ['float', 'double'])
def test_tiled_block_stays_launchable(lanes, elements, fp):
  """At most 1,024 threads per CTA, as the generic generator's plans."""
  p = plan(_small, {'threads_per_element': lanes, 'elements_per_block': elements}, fp=fp).get_plan()
  assert p.strategy == 'tiled' and p.threads <= 1024
  assert p.threads == p.params['threads_per_element'] * p.params['elements_per_block']


@pytest.mark.parametrize('option,value', [('acc', 2), ('bbuf', 2), ('ws', 1), ('te', 4)])
def test_form_b_options_keep_form_b(option, value):
  """Options of operand form B on a single product, for which the direct form is the default."""
  p = plan(cases.plain_gemm, {option: value}, 'tf32x3').get_plan()
  assert p.params['form'] == 'b'
  assert p.params.get(option, value) == value


@pytest.mark.parametrize('variant,form', [({}, 'direct'), ({'strategy': 'tcsplit'}, 'direct'), ({'form': 'direct'}, 'direct'),
                                          ({'form': 'b'}, 'b'), ({'pipe': 2}, None)])
def test_forms_of_a_single_product(variant, form):
  assert plan(cases.plain_gemm, variant, 'tf32x3').get_plan().params.get('form') == form


ROW_VARIANTS = {   # row blocks a part of the terms or columns at a time
  '84x27_two_of_three_terms': (84, 27, {'wterms': 2}),
  '84x27_one_term': (84, 27, {'wterms': 1, 'wcols': 14}),
  '56x9_two_of_three_terms': (56, 9, {'wterms': 2}),
  '20x27_more_terms_than_there_are': (20, 27, {'wterms': 5, 'wcols': 40}),
  '20x27_ten_columns': (20, 27, {'wcols': 10}),
}


def row_variant(name):
  b, q, v = ROW_VARIANTS[name]
  return plan(lambda ns: cases.mixed_chain(ns, b, q), dict(v, strategy='colprog', dense=1))


def sources():
  return [row_variant(n).get_source() for n in ROW_VARIANTS]


@pytest.mark.parametrize('name', ROW_VARIANTS)
def test_row_variants_generate(name):
  p = row_variant(name).get_plan().params
  assert 'rows' in p and 1 <= p['wterms'] <= 3 and 1 <= p['wcols'] <= ROW_VARIANTS[name][1]


@pytest.mark.parametrize('variant', [{'rm': 4}, {'rm': 8}, {'rm': 12, 'rc': 5}, {'rc': 5}, {'rm': 6, 'rc': 5, 'te': 2}, {'rm': 2, 'rc': 5, 'te': 2},
                                     {'rm': 12, 'rc': 1, 'te': 9}, {'rm': 12, 'rc': 5, 'te': 0}], ids=str)
def test_incomplete_row_tiles(variant):
  """A tile that is not named whole is the planner's; one that does not cover its columns is not taken."""
  p = plan(lambda ns: cases.volume_chain(ns, 56, 32, s_nnz=300), variant).get_plan().params
  if 'rm' in p:
    assert p['rm'] % 4 == 0 and p['te'] * 32 <= p['threads'] // -(-56 // p['rm']) * p['rc']


@pytest.mark.parametrize('mc', [0, 1, 9, 40])
def test_fp64_columns_at_a_time(mc):
  p = plan(lambda ns: cases.mixed_chain(ns, 20, 9), {'mc': mc}, fp='double').get_plan().params
  assert 1 <= p.get('mc', 1) <= 9


@pytest.mark.gpu
@pytest.mark.parametrize('name', ROW_VARIANTS)
def test_row_variants_match_oracle(name):
  """1e-6 relative L2 norm against the FP64 oracle, as for the planner's own row blocks."""
  import numpy as np
  import torch
  from oracle import harness, multilinear
  from tensorforge_b200.runtime import compile_generator
  g = row_variant(name)
  n = 707
  lay, mem = harness.make_memory(g.descr_list, n, seed=4)
  dev, kw = {}, {'numElements': n}
  for l in lay:
    dev[l.name] = kw[l.name] = torch.tensor(mem.buffers[l.name], dtype=torch.float32, device='cuda')
    if l.kind == 'strided':
      kw[f'{l.name}_extraOffset'] = l.extra_offset
  compile_generator(g)(**kw)
  torch.cuda.synchronize()
  multilinear.evaluate(g.descr_list, mem, n)
  for l in lay:
    got, ref = dev[l.name].double().cpu().numpy(), mem.buffers[l.name]
    assert np.linalg.norm(got - ref) <= 1e-6 * np.linalg.norm(ref), l.name
