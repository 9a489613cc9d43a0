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
