"""Kernels that leave the memory of masked elements alone: a masked element's entry of a pointer
array may be null or stale, so nothing of it is touched before the element's flag is known.
(FP32 chains that fit the unrolled column program fetch strided operands as whole tiles, as it does.)

Shown on the generated text: every use of a per-element operand stands in a block, or behind a
`continue`, that depends on the element's flag (or on the bits a warp made of the tile's flags), or
in a block for batches without flags. On the GPU masked elements have valid pointers and inputs of
NaN, which must not reach any result; tolerance 1e-6 relative L2 norm against the FP64 oracle (at
most 2 x 128 products and two more per sum: sqrt(258) * 2^-24 = 9.6e-7), FP64 1e-12.
"""
import re

import numpy as np
import pytest

from oracle import cases, harness, multilinear

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
  lines = body.split('\n')
  for line, following in zip(lines[1:], lines[2:] + ['']):
    known = guarded[-1] or 'there ? ' in line or re.search(r'flags\[.*\] [!=]= 0u|if \(flags == nullptr\) |if \(.*live\d\)? >> ', line) is not None
    if re.search(r'live\d = (?!~0u)', line):   # a bit is the flag of an element of the batch
      assert re.search(r'= __ballot_sync\(0xffffffffu, .* < \d+u && .* < (pn|numElements) && flags\[.*\] != 0u\);', line), line
    if 'there = ' in line:
      assert re.search(r'there = pe < pn && \(flags == nullptr \|\| flags\[pe0 \+ pe\] != 0u\);', line), line
    if use.search(line) and ' + e0 * ' not in line:   # the start of a strided tile belongs to no element
      seen += 1
      # an entry of a pointer array may be read, and is then not followed before the flag is known
      entry = re.search(r'\* const s\w+ = \(\w+\[.*\] \+ \w+_extraOffset\);$', line) and re.search(r'flags\[.*\] == 0u\) continue;$', following)
      if not known and not entry:
        out.append(line.strip())
    if re.search(r'if \((flags.*\] == 0u|!\(.*live\d\)? >> .*)\) continue;', line):
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


@pytest.mark.gpu
@pytest.mark.parametrize('name', CASES)
def test_masked_elements_reach_nothing(name):
  import torch
  from tensorforge_b200.runtime import compile_generator
  g = generate(name)
  fp = CASES[name][1]
  np_type, dtype, tol = (np.float32, torch.float32, 1e-6) if fp == 'float' else (np.float64, torch.float64, 1e-12)
  k = compile_generator(g)
  for n, keep in ((1, 0.0), (45, 0.5), (1501, 0.75), (2300, 0.1)):
    lay, mem = harness.make_memory(g.descr_list, n, seed=n, dtype=np_type)
    flags = harness.make_flags(n, 3, keep)
    dev, kw = {}, {'numElements': n, 'flags': torch.tensor(flags.astype(np.int32), device='cuda')}
    clean = {}
    for l in lay:
      clean[l.name] = mem.buffers[l.name].copy()
      if l.kind in ('strided', 'ptr') and l.tensor.direction.name == 'SOURCE':
        for e in np.flatnonzero(flags == 0):
          mem.buffers[l.name][l.starts[e]:l.starts[e] + harness.storage_values(l.tensor)] = np.nan
      dev[l.name] = kw[l.name] = torch.tensor(mem.buffers[l.name], dtype=dtype, device='cuda')
      if l.kind in ('strided', 'ptr'):
        kw[f'{l.name}_extraOffset'] = l.extra_offset
      if l.kind == 'ptr':
        kw[l.name] = torch.tensor(dev[l.name].data_ptr() + (l.starts - l.extra_offset) * dev[l.name].element_size(), device='cuda')
    k(**kw)
    torch.cuda.synchronize()
    mem.buffers.update({name: v.copy() for name, v in clean.items()})
    multilinear.evaluate(g.descr_list, mem, n, flags=flags)
    for l in lay:
      if l.kind in ('strided', 'ptr') and l.tensor.direction.name != 'SOURCE':
        got, ref = dev[l.name].double().cpu().numpy(), mem.buffers[l.name]
        assert np.linalg.norm(got - ref) <= tol * np.linalg.norm(ref), (l.name, n)
        kept = ref == clean[l.name]
        assert np.array_equal(got[kept], ref[kept]), (l.name, n)
