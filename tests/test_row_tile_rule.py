"""Which chains of more than 28 columns loop over a dense A in row tiles, by pattern and size."""
import pytest

from oracle import cases
from tests.test_grouped_forms import MM, ID, chain


def _product(ns, m, k, n, density):
  S, sub = ns.Addressing.STRIDED, ns.SubTensor
  A = ns.Tensor([m, k], ns.Addressing.NONE, spp=ns.ListSPP(cases.sparse_pattern(m, k, density, 3), (m, k)))
  B, C = ns.Tensor([k, n], S), ns.Tensor([m, n], S)
  return [ns.MultilinearDescr(sub(C), [sub(A), sub(B)], MM, ID)]


@pytest.mark.parametrize('terms,m,k,n,density,tiles', [
  (1, 60, 84, 40, 0.44, False), (1, 100, 100, 64, 0.44, False), (1, 84, 84, 64, 0.54, False), (1, 84, 84, 40, 0.7, True), (1, 60, 84, 32, 0.65, True),
  (1, 100, 100, 32, 0.7, True), (1, 50, 37, 40, 0.95, False), (2, 56, 56, 40, 0.42, False), (2, 56, 56, 32, 0.55, True), (3, 56, 56, 32, 0.45, True),
  (2, 84, 84, 64, 0.46, True), (2, 35, 35, 32, 0.9, True)])
def test_rule(terms, m, k, n, density, tiles):
  from tensorforge_b200.kernels import Context, FP, Generator, Options
  ns = cases.ns_from_module('tensorforge_b200')
  g = Generator(_product(ns, m, k, n, density) if terms == 1 else chain(ns, m, n, density, terms), Context('sm_100a', 'cuda', FP['float'], Options()))
  g.generate()
  p = g.get_plan()
  assert p.strategy == 'colprog' and ('rm' in p.params) == tiles
