"""Kernels that leave the memory of masked elements alone: a masked element's entry of a pointer
array may be null or stale, so no per-element address is formed before the element's flag is known.

Shown on the generated text: every use of a per-element operand stands in a block, or behind a
`continue`, that depends on the element's flag.
"""
import re

import pytest

from oracle import cases

P = 'pointer_based'


def _long_chain(ns, q, k=128, addr='strided'):
  """out += A1 B R1 + A2 B R2 with more than 16,384 values of A."""
  N, S = ns.Addressing.NONE, ns.Addressing.str2addr(addr)
  sub, mm, ident = ns.SubTensor, [[0, -1], [-1, 1]], [[0, 1], [0, 1]]
  B, out = ns.Tensor([k, q], S), ns.Tensor([128, q], S)
  descrs = []
  for t in range(2):
    A, R = ns.Tensor([128, k], N), ns.Tensor([q, q], S, spp=ns.ListSPP([(i, i) for i in range(q)], (q, q)))
    T = ns.generate_tmp_tensor([sub(A), sub(B)], mm)
    descrs += [ns.MultilinearDescr(sub(T), [sub(A), sub(B)], mm, ident),
               ns.MultilinearDescr(sub(out), [sub(T), sub(R)], mm, ident, add=t > 0)]
  return descrs


CASES = {
  'fp64_chain': (lambda ns: cases.build('chain_o6', ns), 'double', 'mc'),
  'fp64_chain_ptr': (lambda ns: cases.volume_chain(ns, 35, 9, q_addr=P, s_addr=P, out_addr=P), 'double', 'mc'),
  'fp64_product_ptr': (lambda ns: cases.plain_gemm(ns), 'double', 'mc'),
  'row_blocks': (lambda ns: cases.build('chain_o6', ns), 'float', 'rows'),
  'row_blocks_in_pieces_ptr': (lambda ns: cases.volume_chain(ns, 21, 27, s_nnz=60, q_addr=P, s_addr=P, out_addr=P), 'float', 'rows'),
  'row_blocks_odd_add': (lambda ns: cases.plain_gemm(ns, 24, 17, 5, P, P, add=True), 'float', 'rows'),
  'row_blocks_long': (lambda ns: _long_chain(ns, 9), 'float', 'rows'),
  'row_tiles_long': (lambda ns: _long_chain(ns, 40), 'float', 'rc'),
  'row_tiles_long_ptr_odd': (lambda ns: _long_chain(ns, 37, 127, P), 'float', 'rc'),
  'fp64_product_odd_add': (lambda ns: cases.plain_gemm(ns, 17, 5, 3, P, 'strided', add=True), 'double', 'mc'),
}


def generate(name):
  from tensorforge_b200.kernels import Context, FP, Generator, Options
  build, fp, _ = CASES[name]
  g = Generator(build(cases.ns_from_module('tensorforge_b200')), Context('sm_100a', 'cuda', FP[fp], Options()))
  g.generate()
  return g


def unguarded(g):
  """Lines of the kernel that use a per-element operand where no enclosing block and no earlier
  statement of one looked at the element's flag."""
  text = g.get_source()
  names = [t.name for t, _ in g.abi_symbols() if t.addressing.name in ('STRIDED', 'PTR_BASED')]
  use = re.compile(r'\b(' + '|'.join(names) + r')(\[| \+)')
  body = text[text.index('__global__'):text.index('launcher_')]
  guarded, out, seen = [False], [], 0
  for line in body.split('\n')[1:]:
    known = guarded[-1] or re.search(r'flags\[.*\] [!=]= 0u', line) is not None
    if use.search(line) and ' + e0 * ' not in line:   # the start of a strided tile belongs to no element
      seen += 1
      if not known:
        out.append(line.strip())
    if re.search(r'flags\[.*\] == 0u\) continue;', line):
      guarded[-1] = True
    for c in line:
      if c == '{':
        guarded.append(known)
      elif c == '}':
        guarded.pop()
        if not guarded:   # behind the kernel
          return out, seen
  raise AssertionError('no end of the kernel')


@pytest.mark.parametrize('name', CASES)
def test_no_address_without_the_flag(name):
  g = generate(name)
  assert CASES[name][2] in g.get_plan().params
  bad, seen = unguarded(g)
  assert seen >= 2 and not bad, bad
