"""Row blocks: every shared-memory load of the K loop, those ahead of its last step among them,
stays inside what the CTA allocates, also where the operand buffers behind A are small.

GPU tolerance: 1e-6 relative L2 norm against the FP64 oracle, as for the other row blocks (sums of
at most 16 products, sqrt(16) * 2^-24 = 2.4e-7).
"""
from types import SimpleNamespace as NS

import numpy as np
import pytest

from oracle import cases, harness, multilinear

CASES = {   # the planner's own choice for these: row blocks of a short product with few columns
  '128x8x1': (128, 8, 1), '100x8x1': (100, 8, 1), '97x8x1': (97, 8, 1), '120x12x1': (120, 12, 1), '128x12x1': (128, 12, 1),
  '128x8x2': (128, 8, 2), '128x4x1': (128, 4, 1), '128x16x1': (128, 16, 1),
}


def generate(name):
  from tensorforge_b200.kernels import Context, FP, Generator, Options
  ns = cases.ns_from_module('tensorforge_b200')
  g = Generator(cases.plain_gemm(ns, *CASES[name], 'strided', 'strided'), Context('sm_100a', 'cuda', FP['float'], Options()))
  g.generate()
  return g


def _last_loads(k, mp, ts, nt, rg, rm, pitch, p):
  """Values behind the start of A's term and of B's element that k_loop's loads reach (its text:
  A at a + (l + 1 .. l + 4) * mp, B at b + l + 2 and b + l + 4, two values each; steps left over)."""
  a = [0] + [(l + d) * mp for l in range(0, k - 3, 4) for d in (1, 2, 3, 4)]
  b = [0] + [l + d for l in range(0, k - 3, 4) for d in (2, 4)]
  if k % 4 >= 2:
    a.append((k // 4 * 4 + 1) * mp)
  if k % 4 == 3:
    a.append((k - 1) * mp)
    b.append(k - 1)
  return (nt - 1) * ts + (rg - 1) * rm + max(a) + rm, (p - 1) * pitch + max(b) + 2


def _shape(m, k, n, terms, r):
  b = NS(name='b', kind='batched')
  make = lambda i: NS(K=k, P=n, A=NS(storage_size=lambda: m * k), B=b,
                      R=NS(name=f'r{i}', kind='batched', storage_size=lambda: r) if r else None)
  return NS(M=m, N=n, terms=[make(i) for i in range(terms)])


def _check(shape, variant):
  from tensorforge_b200.codegen.rowblock import layout, rowblock_params
  p = rowblock_params(shape, variant)
  if p is None:
    return 0
  params, smem = p
  rm, te, nt, t = params['rows'], params['te'], len(shape.terms), shape.terms[0]
  a, buf, off = layout(shape, rm, te)
  rg, pitch = -(-shape.M // rm), -(-t.K // 4) * 4
  last_a, last_b = _last_loads(t.K, rg * rm, t.K * rg * rm, nt, rg, rm, pitch, t.P)
  last_b += a + (params['buffers'] - 1) * buf + (te - 1) * off['b'][1]
  assert 4 * max(last_a, last_b, a + params['buffers'] * buf) <= smem <= 227 * 1024, (shape.M, t.K, shape.N, nt, params, smem)
  return 1


def test_lone_products():
  shapes = [(m, k, n) for m in range(1, 129) for k in range(1, 129) for n in (1, 2, 3, 5, 9, 28)]
  assert sum(_check(_shape(m, k, n, 1, 0), {}) for m, k, n in shapes) > 90_000


@pytest.mark.parametrize('terms', [1, 2, 3, 4])
def test_chains(terms):
  shapes = [(m, k, n, r) for m in range(1, 129, 3) for k in (1, 2, 3, 4, 7, 8, 12, 16, 24, 63, 64, 125, 128)
            for n in (1, 2, 4, 9, 14, 20, 27, 28) for r in {1, n, n * n}]
  assert sum(_check(_shape(m, k, n, terms, r), {}) for m, k, n, r in shapes) > 3_000


@pytest.mark.parametrize('variant', [{'threads': 256}, {'threads': 64, 'buffers': 1}, {'rm': 2}, {'te': 1}], ids=str)
def test_variants(variant):
  shapes = [(m, k, n) for m in (1, 17, 64, 97, 100, 128) for k in (4, 7, 8, 12, 128) for n in (1, 2, 9)]
  assert sum(_check(_shape(m, k, n, 1, r), variant) for m, k, n in shapes for r in (0, n)) > 60


@pytest.mark.parametrize('name', CASES)
def test_kernels_allocate_it(name):
  g = generate(name)
  p = g.get_plan()
  m, k, _ = CASES[name]
  assert 'rows' in p.params and p.params['rows'] == 4
  assert p.smem_bytes >= 4 * (k + 1) * (-(-m // 4) * 4)
  assert f', {p.smem_bytes}, stream>>>' in g.get_source()


@pytest.mark.gpu
@pytest.mark.parametrize('name', CASES)
def test_matches_oracle(name):
  import torch
  from tensorforge_b200.runtime import compile_generator
  g = generate(name)
  for n in (1, 1203):
    lay, mem = harness.make_memory(g.descr_list, n, seed=n)
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
      assert np.linalg.norm(got - ref) <= 1e-6 * np.linalg.norm(ref), (l.name, n)
