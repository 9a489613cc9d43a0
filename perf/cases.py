"""The calls a user of the framework makes, as measurable cases.

A program describes batched tensor operations with the frontend (`Tensor`, `ListSPP`,
`MultilinearDescr`, ...), has the generator emit a kernel for each of them once, and then
calls the launchers on its buffers time step after time step. `prepare` therefore holds
the generated kernel and device buffers, `run` is one launcher call.

The operations are the repository's own workloads: volume chains of a discontinuous
Galerkin solver out_e = sum_t K_t Q_e S_{e,t} (shared sparse K_t, per-element sparse S) at
several basis sizes and quantity counts, batches of small GEMMs (shared or per-element left
operand, strided or through pointer arrays), the three-matrix chain D_e += A_e (B_e C_e),
pointwise nonlinear updates, and mixed-shape batches in one persistent launch.
"""
import math

import numpy as np
import torch

from tensorforge_b200.common.aux import generate_tmp_tensor
from tensorforge_b200.common.basic_types import Addressing, FloatingPointType
from tensorforge_b200.common.context import Context, Options
from tensorforge_b200.common.matrix.boundingbox import BoundingBox
from tensorforge_b200.common.matrix.spp import ListSPP
from tensorforge_b200.common.matrix.tensor import SubTensor, Tensor
from tensorforge_b200.functions import assign, exp, scalar, temp, tensor, ternary
from tensorforge_b200.generators.descriptions import ElementwiseDescr, MultilinearDescr
from tensorforge_b200.generators.generator import Generator
from tensorforge_b200.grouped import GroupedKernel
from tensorforge_b200.runtime import compile_generator

MATMUL = [[0, -1], [-1, 1]]
IDENT = [[0, 1], [0, 1]]

MIXED = [(b, q) for b in (10, 20, 35, 56, 84) for q in (9, 27)]


def _chain(basis, q, nnz, seed, terms=3, density=0.45):
  return {'kind': 'chain', 'basis': basis, 'q': q, 'nnz': nnz, 'seed': seed, 'terms': terms, 'density': density}


def _gemm(m, k, n, a='none', b='strided', c='strided', **more):
  return {'kind': 'gemm', 'm': m, 'k': k, 'n': n, 'a': a, 'b': b, 'c': c, **more}


# name -> operation. `precisions`: the computations it is used with; `most`: the largest
# batch that stays within the work of the largest listed case.
KERNELS = {
  'chain_56x9': dict(_chain(56, 9, 24, 0), precisions=('plain', 'tf32x3', 'bf16x3', 'fp64'), most=150_000),
  'chain_20x27': dict(_chain(20, 27, 72, 3), precisions=('plain', 'tf32x3'), most=150_000),
  'chain_10x9_dense': dict(_chain(10, 9, 81, 1, terms=2, density=1.0), precisions=('plain', 'tf32x3'), most=500_000),
  'gemm_56x56x9_ptr': dict(_gemm(56, 56, 9, b='pointer_based', c='pointer_based'),
                           precisions=('plain', 'tf32x3', 'fp64'), most=300_000),
  'gemm_56x56x9': dict(_gemm(56, 56, 9), precisions=('plain', 'tf32x3'), most=300_000),
  'gemm_24x17x5_add': dict(_gemm(24, 17, 5, add=True), precisions=('plain', 'tf32x3'), most=500_000),
  'gemm_33x9x11_batched': dict(_gemm(33, 9, 11, a='strided'), precisions=('plain',), most=200_000),
  'gemm_20x20x9_sparse_a': dict(_gemm(20, 20, 9, sparse='a'), precisions=('plain', 'tf32x3'), most=500_000),
  'gemm_20x20x9_sparse_a_batched': dict(_gemm(20, 20, 9, a='strided', sparse='a'), precisions=('plain', 'fp64'), most=200_000),
  'gemm_20x20x9_sparse_b': dict(_gemm(20, 20, 9, sparse='b'), precisions=('plain',), most=200_000),
  'gemm_32x32x32_ptr': dict(_gemm(32, 32, 32, 'pointer_based', 'pointer_based', 'pointer_based', form='ab'),
                            precisions=('plain',), most=100_000),
  'gemm_32x32x32_ptr_atb': dict(_gemm(32, 32, 32, 'pointer_based', 'pointer_based', 'pointer_based', form='atb'),
                                precisions=('plain',), most=100_000),
  'gemm_32x32x32_ptr_abt': dict(_gemm(32, 32, 32, 'pointer_based', 'pointer_based', 'pointer_based', form='abt'),
                                precisions=('plain',), most=100_000),
  'three_matrices': {'kind': 'three', 'precisions': ('plain', 'fp64'), 'most': 60_000},
  'update_56x9': {'kind': 'update', 'precisions': ('plain', 'fp64'), 'most': 500_000},
}
for _b, _q in MIXED:
  KERNELS[f'chain_{_b}x{_q}_mixed'] = dict(_chain(_b, _q, round(0.3 * _q * _q), _b * 7 + _q), precisions=('plain',),
                                           most=min(300_000, int(3e10 / (3 * 0.9 * _b * _b * _q + 8 * _b * _q))))


def listed():
  return [
    # the order-6 chain on tensor cores over a large mesh: the headline benchmark
    {'name': 'chain o6 tf32x3 500k', 'kernel': 'chain_56x9', 'precision': 'tf32x3', 'n': 500_000, 'flags': False},
    # one small cluster of a local-time-stepping run: latency and how far few elements spread
    {'name': 'chain o6 plain 300', 'kernel': 'chain_56x9', 'precision': 'plain', 'n': 300, 'flags': False},
    # the same chain in the default precision over an ordinary, ragged partition
    {'name': 'chain o6 plain 100003', 'kernel': 'chain_56x9', 'precision': 'plain', 'n': 100_003, 'flags': False},
    # and in double precision, which most production runs of such solvers use
    {'name': 'chain o6 fp64 60k', 'kernel': 'chain_56x9', 'precision': 'fp64', 'n': 60_000, 'flags': False},
    # a viscoelastic order-4 chain with 27 quantities, part of the elements masked out
    {'name': 'chain 20x27 plain masked 40001', 'kernel': 'chain_20x27', 'precision': 'plain', 'n': 40_001, 'flags': True},
    # 10,000 pointer-array GEMMs: the reference's own batched workload
    {'name': 'gemm 56x56x9 ptr plain 10k', 'kernel': 'gemm_56x56x9_ptr', 'precision': 'plain', 'n': 10_000, 'flags': False},
    # the same on tensor cores over a large batch
    {'name': 'gemm 56x56x9 ptr tf32x3 300k', 'kernel': 'gemm_56x56x9_ptr', 'precision': 'tf32x3', 'n': 300_000, 'flags': False},
    # the largest basis of the mixed-shape workload on its own
    {'name': 'chain 84x27 plain 20k', 'kernel': 'chain_84x27_mixed', 'precision': 'plain', 'n': 20_000, 'flags': False},
    # ten shapes in one persistent launch
    {'name': 'mixed shapes 60k', 'kernel': 'grouped', 'precision': 'plain', 'n': 60_000, 'flags': False},
    # D_e += A_e (B_e C_e): every operand per element, a temporary in between
    {'name': 'three matrices 20k', 'kernel': 'three_matrices', 'precision': 'plain', 'n': 20_000, 'flags': False},
    # per-element 32x32 products through pointer arrays, as generated for a tensor toolkit
    {'name': 'gemm 32x32x32 ptr 50k', 'kernel': 'gemm_32x32x32_ptr', 'precision': 'plain', 'n': 50_000, 'flags': False},
    # a pointwise nonlinear update of every element's block
    {'name': 'update 56x9 200k', 'kernel': 'update_56x9', 'precision': 'plain', 'n': 200_000, 'flags': False},
  ]


def draw(rng):
  """Another call of the same kinds: kernel, precision and batch size (log-uniform), one in five masked."""
  name = rng.choice(sorted(KERNELS) + ['grouped'])
  most = 150_000 if name == 'grouped' else KERNELS[name]['most']
  precision = 'plain' if name == 'grouped' else rng.choice(KERNELS[name]['precisions'])
  n = int(round(math.exp(rng.uniform(math.log(100), math.log(most)))))
  return {'kernel': name, 'precision': precision, 'n': n, 'flags': name != 'grouped' and rng.random() < 0.2}


# ------------------------------------------------------------------ patterns

def _bernoulli(rows, cols, density, seed):
  mask = np.random.default_rng(seed).random((rows, cols)) < density
  return [(int(i), int(j)) for j in range(cols) for i in range(rows) if mask[i, j]]


def _fixed(rows, cols, nnz, seed):
  flat = np.sort(np.random.default_rng(seed).choice(rows * cols, size=nnz, replace=False))
  return sorted([(int(f % rows), int(f // rows)) for f in flat], key=lambda t: (t[1], t[0]))


def _chain_patterns(c):
  """(K patterns, S patterns) of a chain, None where dense; entries in column-major order."""
  ks = [_bernoulli(c['basis'], c['basis'], c['density'], c['seed'] * 1000 + 11 + t) if c['density'] < 1 else None
        for t in range(c['terms'])]
  ss = [_fixed(c['q'], c['q'], c['nnz'], c['seed'] * 1000 + 101 + t) if c['nnz'] < c['q'] ** 2 else None
        for t in range(c['terms'])]
  return ks, ss


def _gemm_pattern(c):
  if c.get('sparse') == 'a':
    return _bernoulli(c['m'], c['k'], 0.3, 5)
  return _bernoulli(c['k'], c['n'], 0.3, 5) if c.get('sparse') == 'b' else None


# ------------------------------------------------------------------ kernels

def _product(dest, ops, add=False, target=MATMUL):
  return MultilinearDescr(SubTensor(dest), [SubTensor(o) for o in ops], target, IDENT, add=add)


def _descriptors(c):
  none, strided, ptr = Addressing.NONE, Addressing.STRIDED, Addressing.PTR_BASED
  if c['kind'] == 'chain':
    b, q = c['basis'], c['q']
    kps, sps = _chain_patterns(c)
    Q, out = Tensor([b, q], strided), Tensor([b, q], strided)
    descrs = []
    for t, (kp, sp) in enumerate(zip(kps, sps)):
      K = Tensor([b, b], none, spp=ListSPP(kp, (b, b)) if kp is not None else None)
      S = Tensor([q, q], strided, spp=ListSPP(sp, (q, q)) if sp is not None else None)
      T = generate_tmp_tensor([SubTensor(K), SubTensor(Q)], MATMUL)
      descrs += [_product(T, [K, Q]), _product(out, [T, S], add=t > 0)]
    return descrs
  if c['kind'] == 'gemm':
    m, k, n = c['m'], c['k'], c['n']
    pat = _gemm_pattern(c)
    form = c.get('form', 'ab')
    A = Tensor([m, k], Addressing.str2addr(c['a']), spp=ListSPP(pat, (m, k)) if c.get('sparse') == 'a' else None)
    B = Tensor([k, n], Addressing.str2addr(c['b']), spp=ListSPP(pat, (k, n)) if c.get('sparse') == 'b' else None)
    C = Tensor([m, n], Addressing.str2addr(c['c']))
    if form == 'ab':
      return [_product(C, [A, B], add=c.get('add', False))]
    T = Tensor([m, n], strided, is_tmp=True)
    if form == 'atb':
      return [_product(T, [A, B], target=[[-1, 0], [-1, 1]]),
              MultilinearDescr(SubTensor(C), [SubTensor(T)], [[0, 1]], [[0, 1]])]
    return [MultilinearDescr(SubTensor(T), [SubTensor(A)], [[0, 1]], [[0, 1]]),
            _product(C, [T, B], target=[[0, -1], [1, -1]])]
  if c['kind'] == 'three':
    D, A = Tensor([56, 9], strided, BoundingBox([0, 0], [56, 9])), Tensor([56, 56], strided, BoundingBox([0, 0], [56, 56]))
    B, C = Tensor([56, 9], strided, BoundingBox([0, 0], [56, 9])), Tensor([9, 9], strided, BoundingBox([0, 0], [9, 9]))
    T = generate_tmp_tensor([SubTensor(B), SubTensor(C)], MATMUL)
    return [_product(T, [B, C]), _product(D, [A, T], add=True)]
  Q, O, s, t = Tensor([56, 9], strided), Tensor([56, 9], strided), Tensor([], Addressing.SCALAR), temp()
  return [ElementwiseDescr([assign(t, tensor(Q) * scalar(s)),
                            assign(tensor(O), ternary(t > 0.0, t * exp(-(t * t)), 0.5 * t))])]


_generated = {}


def _generator(kernel, precision):
  fp = FloatingPointType.DOUBLE if precision == 'fp64' else FloatingPointType.FLOAT
  g = Generator(_descriptors(KERNELS[kernel]),
                Context('sm_100a', 'cuda', fp, Options(precision='plain' if precision == 'fp64' else precision)))
  g.generate()
  return g


def _kernel(kernel, precision):
  """The generated launcher; a program generates it once, before its time loop."""
  if (kernel, precision) not in _generated:
    if kernel == 'grouped':
      made = GroupedKernel([_generator(f'chain_{b}x{q}_mixed', precision) for b, q in MIXED])
    else:
      made = compile_generator(_generator(kernel, precision))
    _generated[kernel, precision] = made
  return _generated[kernel, precision]


# ------------------------------------------------------------------ buffers

def _values(gen, size, dtype):
  return torch.randn(size, generator=gen, device='cuda', dtype=dtype)


def _shared(gen, size, k, dtype):
  """Values of a shared operator matrix, scaled so that products keep the inputs' magnitude."""
  return _values(gen, size, dtype) / math.sqrt(k)


def _pointers(gen, buf, n, volume):
  """Per-element addresses into `buf`, in the scattered order a mesh partition gives."""
  at = torch.randperm(n, generator=gen, device='cuda')
  return buf.data_ptr() + at * (volume * buf.element_size()), at


def _chain_names(c):
  """Parameter names of each term's (K, S): parameters are named in order of first
  appearance, K Q out S | K S | K S."""
  return [('m0', 'm3')] + [(f'm{2 * t + 2}', f'm{2 * t + 3}') for t in range(1, c['terms'])]


def _buffers(c, gen, n, dtype):
  """(launcher arguments by parameter name, buffers by what they are)."""
  if c['kind'] == 'chain':
    b, q = c['basis'], c['q']
    ks, _ = _chain_patterns(c)
    args = {'m1': _values(gen, n * b * q, dtype), 'm2': torch.zeros(n * b * q, device='cuda', dtype=dtype)}
    for (kn, sn), kp in zip(_chain_names(c), ks):
      args[kn] = _shared(gen, len(kp) if kp is not None else b * b, b, dtype)
      args[sn] = _values(gen, n * q * q, dtype) / math.sqrt(q)
    return args, args
  if c['kind'] == 'gemm':
    data, args = {}, {}
    pat = _gemm_pattern(c)
    sizes = {'a': c['m'] * c['k'], 'b': c['k'] * c['n'], 'c': c['m'] * c['n']}
    stored = dict(sizes)
    if c.get('sparse'):
      stored[c['sparse']] = len(pat) if c[c['sparse']] == 'none' else sizes[c['sparse']]
    for name in 'abc':
      if c[name] == 'none':
        data[name] = _shared(gen, stored[name], c['k'], dtype)
      elif name == 'c':
        data[name] = _values(gen, n * sizes[name], dtype) if c.get('add') else torch.zeros(n * sizes[name], device='cuda', dtype=dtype)
      else:
        data[name] = _values(gen, n * stored[name], dtype) / (math.sqrt(c['k']) if name == 'a' else 1)
    for name in 'abc':
      args[name] = data[name]
      if c[name] == 'pointer_based':
        args[name], data[name + '_at'] = _pointers(gen, data[name], n, sizes[name])
    order = {'ab': 'cab', 'atb': 'abc', 'abt': 'acb'}[c.get('form', 'ab')]
    return {f'm{i}': args[x] for i, x in enumerate(order)}, data
  if c['kind'] == 'three':
    data = {'B': _values(gen, n * 504, dtype), 'C': _values(gen, n * 81, dtype) / 3,
            'D': _values(gen, n * 504, dtype), 'A': _values(gen, n * 3136, dtype) / math.sqrt(56)}
    return {f'm{i}': data[x] for i, x in enumerate('BCDA')}, data
  data = {'Q': _values(gen, n * 504, dtype), 's': 0.75, 'O': torch.zeros(n * 504, device='cuda', dtype=dtype)}
  return {f'm{i}': data[x] for i, x in enumerate('QsO')}, data


def _group_counts(n, seed):
  """Element counts of the ten shapes, log-uniform over two decades, summing to about n."""
  raw = np.exp(np.random.default_rng(seed).uniform(0, math.log(200), len(MIXED)))
  return [max(8, int(round(n * r / raw.sum() / 8)) * 8) for r in raw]


def _in_hand(case, seed):
  """Every input of a case, made from the seed alone."""
  gen = torch.Generator(device='cuda')
  gen.manual_seed(seed)
  dtype = torch.float64 if case['precision'] == 'fp64' else torch.float32
  if case['kernel'] == 'grouped':
    return [_buffers(KERNELS[f'chain_{b}x{q}_mixed'], gen, k, dtype)[0]
            for (b, q), k in zip(MIXED, _group_counts(case['n'], 0))]
  args, data = _buffers(KERNELS[case['kernel']], gen, case['n'], dtype)
  flags = (torch.rand(case['n'], generator=gen, device='cuda') < 0.7).to(torch.int32) if case['flags'] else None
  return args, data, flags


def prepare(case, seed):
  kernel = _kernel(case['kernel'], case['precision'])
  if case['kernel'] == 'grouped':
    groups = _in_hand(case, seed)
    counts = _group_counts(case['n'], 0)
    launch = kernel.prepare([dict(a, numElements=k) for a, k in zip(groups, counts)])
    return {'launch': launch, 'groups': groups, 'out': {f'{b}x{q}': a['m2'] for (b, q), a in zip(MIXED, groups)}}
  c = KERNELS[case['kernel']]
  args, data, flags = _in_hand(case, seed)
  args = dict(args, numElements=case['n'], flags=flags)
  out = data[{'chain': 'm2', 'gemm': 'c', 'three': 'D', 'update': 'O'}[c['kind']]]
  return {'kernel': kernel, 'args': args, 'data': data, 'out': out}


def run(state):
  if 'launch' in state:
    state['launch'].launch()
  else:
    state['kernel'](**state['args'])
  return state['out']


# ------------------------------------------------------------------ work and 64-bit results

def _chain_work(c, n):
  ks, ss = _chain_patterns(c)
  b, q = c['basis'], c['q']
  nk = [len(k) if k is not None else b * b for k in ks]
  ns = [len(s) if s is not None else q * q for s in ss]
  return n * (2 * b * q + sum(ns)) + sum(nk), 2 * n * sum(k * q + b * s for k, s in zip(nk, ns))


def work(case):
  n = case['n'] * 0.7 if case['flags'] else case['n']
  fs = 8 if case['precision'] == 'fp64' else 4
  if case['kernel'] == 'grouped':
    parts = [_chain_work(KERNELS[f'chain_{b}x{q}_mixed'], k) for (b, q), k in zip(MIXED, _group_counts(case['n'], 0))]
    return {'bytes': fs * sum(p[0] for p in parts), 'flops': sum(p[1] for p in parts)}
  c = KERNELS[case['kernel']]
  extra = 4 * case['n'] if case['flags'] else 0
  if c['kind'] == 'chain':
    values, flops = _chain_work(c, n)
  elif c['kind'] == 'gemm':
    m, k, w = c['m'], c['k'], c['n']
    pat = _gemm_pattern(c)
    sizes = {'a': m * k, 'b': k * w, 'c': m * w * (2 if c.get('add') else 1)}
    flops = 2 * n * m * k * w
    if pat is not None:
      sizes[c['sparse']] = len(pat)
      flops = 2 * n * len(pat) * (w if c['sparse'] == 'a' else m)
    values = sum(s * (1 if c[x] == 'none' else n) for x, s in sizes.items())
    extra += sum(8 * n for x in 'abc' if c[x] == 'pointer_based')
  elif c['kind'] == 'three':
    values, flops = n * (3136 + 3 * 504 + 81), 2 * n * (56 * 9 * 9 + 56 * 56 * 9)
  else:
    values, flops = n * 2 * 504, n * 504 * 5
  return {'bytes': fs * values + extra, 'flops': flops}


def _dense(values, pattern, rows, cols, n=None):
  """Matrices (n, cols, rows) in 64 bits, i.e. column-major, from values in pattern order."""
  slot = rows * cols
  if n is None:
    values, n = values[None], 1
  else:
    values = values.view(n, -1)
  if pattern is None:
    return values.double().view(n, cols, rows)
  full = torch.zeros(n, slot, dtype=torch.float64, device=values.device)
  at = torch.tensor([j * rows + i for i, j in pattern], device=values.device)
  full[:, at] = values[:, :len(pattern)].double()
  return full.view(n, cols, rows)


def _exact_chain(c, args, n):
  b, q = c['basis'], c['q']
  ks, ss = _chain_patterns(c)
  Q = args['m1'].view(n, q, b)
  out = torch.empty(n, q, b, dtype=torch.float64, device=Q.device)
  for e in range(0, n, 20_000):
    part = torch.zeros_like(out[e:e + 20_000])
    for (kn, sn), kp, sp in zip(_chain_names(c), ks, ss):
      K = _dense(args[kn], kp, b, b)[0]                       # K[l, i]: entry (i, l)
      S = _dense(args[sn].view(n, -1)[e:e + 20_000].reshape(-1), sp, q, q, part.shape[0])   # S[e, j, m]
      part += (S @ Q[e:e + 20_000].double()) @ K
    out[e:e + 20_000] = part
  return out.view(-1)


def exact(case, seed):
  n = case['n']
  if case['kernel'] == 'grouped':
    groups = _in_hand(case, seed)
    return {f'{b}x{q}': _exact_chain(KERNELS[f'chain_{b}x{q}_mixed'], a, k)
            for (b, q), a, k in zip(MIXED, groups, _group_counts(n, 0))}
  c = KERNELS[case['kernel']]
  args, data, flags = _in_hand(case, seed)
  if c['kind'] == 'chain':
    before, out = args['m2'].double(), _exact_chain(c, args, n)
  elif c['kind'] == 'gemm':
    m, k, w = c['m'], c['k'], c['n']
    pat = _gemm_pattern(c)
    at = {x: data.get(x + '_at', slice(None)) for x in 'abc'}
    pa, pb = (pat if c.get('sparse') == x else None for x in 'ab')
    A = _dense(data['a'], pa, m, k, None if c['a'] == 'none' else n)[at['a'] if c['a'] != 'none' else slice(None)]
    B = _dense(data['b'], pb, k, w, n)[at['b']]
    if c.get('form') == 'atb':
      A = A.transpose(1, 2)
    if c.get('form') == 'abt':
      B = B.transpose(1, 2)
    before = data['c'].double()
    out = (B @ A).reshape(-1)
    if c['c'] == 'pointer_based':
      place = torch.empty_like(out).view(n, -1)
      place[at['c']] = out.view(n, -1)
      out = place.view(-1)
      if flags is not None:
        active = torch.empty_like(flags)
        active[at['c']] = flags
        flags = active
    if c.get('add'):
      out = out + before
  elif c['kind'] == 'three':
    A, B = data['A'].double().view(n, 56, 56), data['B'].double().view(n, 9, 56)
    C, before = data['C'].double().view(n, 9, 9), data['D'].double()
    out = before + ((C @ B) @ A).reshape(-1)
  else:
    t = data['Q'].double() * data['s']
    before, out = data['O'].double(), torch.where(t > 0, t * torch.exp(-t * t), 0.5 * t)
  if flags is not None:
    out = torch.where((flags != 0).repeat_interleave(out.numel() // n), out, before)
  return out
