"""Chains that read most of their operands once and value by value stay with the generic generator."""
import pytest

from oracle import cases

S = 'strided'


def plan(sizes, k, first, second, lead=0, variant=None, fp='float'):
  """out[sizes] = A[first] B[second], `first` and `second` as target lists; A's box starts at `lead`."""
  from tensorforge_b200.kernels import Context, FP, Generator, Options
  ns = cases.ns_from_module('tensorforge_b200')
  T, sub = ns.Tensor, ns.SubTensor
  ext = lambda t: [sizes[i] if i >= 0 else k[-i - 1] for i in t]
  ea, eb = ext(first), ext(second)
  A = T([e + lead if i < 0 else e for e, i in zip(ea, first)], ns.Addressing.STRIDED)
  B = T([e + lead if i < 0 else e for e, i in zip(eb, second)], ns.Addressing.STRIDED)
  box = lambda t, e: ns.BoundingBox([lead if i < 0 else 0 for i in t], [x + (lead if i < 0 else 0) for x, i in zip(e, t)])
  C = T(list(sizes), ns.Addressing.STRIDED)
  g = Generator([ns.MultilinearDescr(sub(C), [sub(A, box(first, ea)), sub(B, box(second, eb))], [first, second],
                                     [list(range(len(first))), list(range(len(second)))])],
                Context('sm_100a', 'cuda', FP[fp], Options(variant=variant)))
  g.generate()
  return g.get_plan()


@pytest.mark.parametrize('sizes,k,first,second,lead,strategy', [
  ([20, 12], [33], [-1, 0, 1], [-1], 0, 'generic'),      # 7,920 values used once, 33 per column
  ([32, 9], [20], [-1, 0, 1], [-1], 1, 'generic'),       # off the 16-byte grid
  ([20, 12], [32], [-1, 0, 1], [-1], 0, 'tiled'),        # copied in 16-byte pieces
  ([8, 8], [33], [-1, 0, 1], [-1], 0, 'tiled'),          # 64 results
  ([16, 12], [5], [-1, 0, 1], [-1], 0, 'tiled'),         # 960 values
  ([33, 11], [9], [0, -1], [-1, 1], 0, 'tiled'),         # a product: every value used several times
])
def test_rule(sizes, k, first, second, lead, strategy):
  assert plan(sizes, k, first, second, lead).strategy == strategy


def test_asked_for():
  args = ([20, 12], [33], [-1, 0, 1], [-1])
  assert plan(*args, variant={'strategy': 'tiled'}).strategy == 'tiled'
  assert plan(*args, variant={'threads_per_element': 64}).strategy == 'tiled'
  assert plan(*args, fp='double').strategy == 'generic'
