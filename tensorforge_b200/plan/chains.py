"""Shared-left GEMM chains: recognition and plans for the fast generators.

A chain qualifies when it computes, for every batch element e,

    out_e  (+)=  sum_t  A_t * B_{e,t} * R_{e,t}

with A_t shared across the batch (Addressing.NONE, dense or sparse), B_{e,t} batched and
dense, R_{e,t} batched or shared (dense or sparse) or absent, written in the
reference's descriptor form (tensorforge/generators/descriptions.py:14-27):

    T_t  =  A_t x B_t            (temporary, targets [[0,-1],[-1,1]])
    out (+)= T_t x R_t           (targets [[0,-1],[-1,1]], add for t > 0)

or a single `out (+)= A x B`. All operands must span their full shape (bounding box =
shape) so that columns are contiguous. This is the shape of BASELINE configs 0-3
(benchmarks/fused/programs/s3time.cf) and of SeisSol's volume/local kernels.
"""
from dataclasses import dataclass, field
from typing import List, Optional

from ..common.basic_types import DataFlowDirection
from . import Plan, SMEM_LIMIT


@dataclass
class Term:
  A: object          # Operand (shared)
  B: object          # Operand (batched, dense)
  R: Optional[object]  # Operand (batched/shared) or None
  K: int
  P: int


@dataclass
class LeftChain:
  terms: List[Term]
  out: object
  M: int
  N: int
  accumulate: bool   # out_e += ... (previous value read once)
  epilogue: list = field(default_factory=list)   # elementwise stages on the output, per entry


def _full(op):
  t = op.tensor
  return list(t.bbox.lower()) == [0] * len(t.shape) and list(t.bbox.upper()) == list(t.shape)


def _full_ref(stage, ref):
  box = [stage.n_ranges[x] if x >= 0 else stage.k_ranges[-x - 1] for x in ref.target]
  return [l for l, _ in box] == [0] * len(box) and [u for _, u in box] == list(ref.op.shape)


def _is_elementwise(stage):
  return getattr(stage, 'kind', '') == 'elementwise'


def _epilogue_ok(tail, shape):
  """Elementwise stages that can run on the output's registers: over the output's whole
  M x N box, writing the output only, reading the output, scalars and batched dense M x N
  tensors at the same entry (n0 = row, n1 = column)."""
  out = shape.out
  for s in tail:
    if s.sizes != [shape.M, shape.N] or any(o is not out for o in s.written):
      return False
    for acc in s.access.values():
      o = acc.op
      if o.kind in ('scalar', 'data') and not acc.dims:
        continue
      if o.kind != 'batched' or o.sparse or not _full(o) or list(o.shape) != [shape.M, shape.N]:
        return False
      if acc.dims != [0, 1] or acc.base != [0, 0]:
        return False
  return True


def match_left_chain(chain) -> Optional[LeftChain]:
  """The chain's shared-left form, with trailing elementwise stages as an epilogue."""
  st = chain.stages
  k = next((i for i, s in enumerate(st) if _is_elementwise(s)), len(st))
  tail = st[k:]
  st = st[:k]
  if not st or not all(_is_elementwise(s) for s in tail):
    return None
  for s in st:
    if not s.is_matmul():
      return None
    for r in s.ops:
      if r.op.kind == 'tmp':
        continue
      if r.op.kind not in ('shared', 'batched') or not _full(r.op) or not _full_ref(s, r):
        return None
  out = None
  terms = []
  i = 0
  accumulate = False
  while i < len(st):
    s = st[i]
    if s.dest.kind == 'tmp':
      if i + 1 >= len(st):
        return None
      s2 = st[i + 1]
      a, b = s.ops
      t, r = s2.ops
      if t.op is not s.dest or s2.dest.kind != 'batched' or s.add:
        return None
      if r.op.kind == 'tmp':
        return None
      if a.op.kind != 'shared' or b.op.kind != 'batched' or b.op.sparse:
        return None
      # the temporary must not be used anywhere else
      if sum(1 for x in st for y in x.ops if y.op is s.dest) != 1:
        return None
      dest = s2.dest
      term = Term(a.op, b.op, r.op, a.op.shape[1], b.op.shape[1])
      add = s2.add
      i += 2
    else:
      if s.dest.kind != 'batched':
        return None
      a, b = s.ops
      if a.op.kind != 'shared' or b.op.kind != 'batched' or b.op.sparse:
        return None
      dest = s.dest
      term = Term(a.op, b.op, None, a.op.shape[1], b.op.shape[1])
      add = s.add
      i += 1
    if dest.sparse or not _full(dest):
      return None
    if out is None:
      out = dest
      accumulate = add
    elif dest is not out or not add:
      return None
    terms.append(term)
  M, N = out.shape
  for t in terms:
    if t.A.shape[0] != M or t.B.shape[0] != t.K:
      return None
    if t.R is None and t.P != N:
      return None
    if t.R is not None and (t.R.shape[0] != t.P or t.R.shape[1] != N):
      return None
    if t.B is out or t.A is out or t.R is out:
      return None
  shape = LeftChain(terms, out, M, N, accumulate)
  if tail:
    if not _epilogue_ok(tail, shape):
      return None
    shape.epilogue = list(tail)
  return shape


def a_values(term):
  """Consumption order of A_t's nonzeros: column l outer, row i inner.

  Returns [(l, [(i, storage position), ...]), ...] for l = 0..K-1.
  """
  A = term.A
  M, K = A.shape
  if A.sparse:
    look = A.sparse_lookup()
    cols = []
    for l in range(K):
      rows = [(i, look[(i, l)]) for i in range(M) if (i, l) in look]
      cols.append((l, rows))
    return cols
  return [(l, [(i, l * M + i) for i in range(M)]) for l in range(K)]


def r_slots(term):
  """Per output column j: [(m, storage position)] of R_t's nonzeros in column j."""
  R = term.R
  P, N = R.shape
  if R.sparse:
    look = R.sparse_lookup()
    return [[(m, look[(m, j)]) for m in range(P) if (m, j) in look] for j in range(N)]
  return [[(m, j * P + m) for m in range(P)] for j in range(N)]


# Column programs unroll one FMA per nonzero of every A_t into straight-line code. Above
# this many ptxas time grows past a minute per kernel, so such chains go to the generic
# generator where no loop over A fits (row_program below). Measured on B200 (84x84 A at 45 %,
# three terms, 9,533 FMAs per column, 26 s of ptxas, 226 registers, no spills): 2.13e7 against
# 2.30e6 el/s for the generic kernel with 27 quantities and 8.25e7 against 1.04e7 with 9; row
# blocks 3.8e7 and 1.3e8.
COLPROG_MAX_FMAS = 16384
# A 128-thread column program whose shared memory leaves room for only one CTA per SM runs
# with 256 threads instead when that keeps the prefetch stage (same registers per thread,
# twice the warps per SM; 2.0x and 1.9x faster on the two 84-basis chains above).
COLPROG_SMEM_PER_SM = 228 * 1024
# A values as constant-bank FMA operands stay in the immediate-constant cache up to roughly
# this many values. Measured on B200: constant A is fastest for most random chains with at
# most 2,048 values and for the dense 56x56 GEMM (3,136 values: 2.54e8 vs 2.32e8 el/s);
# the order-6 chain (4,253 values over three terms) runs 1.24x faster from shared memory.
COLPROG_CONST_A = 4096


# Variant 'mixed' (not a default): the leading terms whose A values fit this budget stay
# constant-bank FMA operands and the rest move to shared memory. With an odd U pitch it
# brings the order-6 chain's CTA to 72 KB of shared memory and 167 registers, three CTAs per
# SM instead of two -- measured slower (2.61e8 against 2.71e8 el/s), as were the other
# three-CTA forms (2.49e8-2.65e8).
COLPROG_CONST_MIXED = 2048


# Variant keys of the unrolled column program: naming one of them asks for that form.
UNROLLED_KEYS = ('a_source', 'chunk', 'cols', 'rsplit', 'upitch', 'min_blocks', 'prefetch', 'const_terms')


# Column programs with more unrolled FMAs than this run slower than row tiles (56x32 chain, 4,253
# FMAs, 20,000 elements: 504 against 385 us).
UNROLLED_MAX_FMAS = 2048
# Above this many the unrolled code has outgrown the instruction cache and looping over the zeros
# as well pays from a density of 0.3 on.
UNROLLED_FETCH_BOUND = 6000


def loops_pay(shape: LeftChain, columns):
  """Whether looping over a dense A (with `columns` output columns at a time) beats code with one
  FMA per stored value. Measured on B200, unrolled time / row-block time:

    three terms, 9 columns    density 0.2   0.3   0.45  0.6   1
      20x20                           1.19  1.19  1.24  1.21  1.33
      35x35                           0.70  0.78  0.98  1.09  1.64
      56x56                           0.68  0.87  1.10  1.68  2.82
      84x84                           0.72  1.29  1.67
    one term, 9 columns
      56x56                           0.75  0.84  1.05  1.17  1.67
      36x68                           0.62  0.71  0.79  0.94  1.37
      84x84                           0.70  0.89  1.17
      35x35, 10x10, 18x61             below 1.1 at any density (odd K: 4-byte copies)
      20x20, 24x17, 16x16             0.95-1.4 (200,000 elements), 1.4-1.5 (5,000: no A to copy
                                      into the constant bank first); with 12 columns and odd K
                                      0.94-0.96 (20,000 and 60,000)

  At the line of 0.42, two and three terms, 20,000 and 60,000 elements: 28x28 1.08-1.30, 72x72 1.45-1.77.
  With 20 columns (pieces of seven) the ratios of several terms are 0.85-1.0 at 0.45."""
  K = max(t.K for t in shape.terms)
  stored = sum(t.A.storage_size() for t in shape.terms)
  density = stored / sum(shape.M * t.K for t in shape.terms)
  if stored > COLPROG_MAX_FMAS or (stored > UNROLLED_FETCH_BOUND and density >= 0.3):
    return True
  if len(shape.terms) == 1:
    if 128 <= shape.M * K <= 512 and shape.N <= (12 if K % 2 == 0 else 9):
      return True
    return K % 2 == 0 and ((stored >= 1800 and density >= 0.42) or
                           (stored >= (512 if shape.N <= 12 else 1024) and density > 0.9 and K % 4 == 0))
  return shape.M * K <= 512 or density >= (0.42 if columns >= min(9, shape.N) else 0.55)


def row_program(shape: LeftChain, fp_size, variant):
  """(parameters, shared-memory bytes) of a column program that loops over A instead of
  unrolling its nonzeros, or None where the unrolled one is the better (or only) form.

  Row blocks (codegen/rowblock.py) for up to 28 columns. Measured against the unrolled program
  (39,900 elements, us): 84x27 1,019 / 1,684, 56x27 519 / 636, 35x27 329 / 388, 20x27 91 / 103,
  10x27 87 / 142, 84x9 300 / 490, 56x9 156 / 172, 35x9 98 / 96, 20x9 35 / 42, 10x9 27 / 40, one
  56x56x9 product 68 / 117. Row tiles (codegen/coltile.py) for more columns or operands that
  differ between terms, where A is dense or its unrolled program long."""
  if fp_size != 4 or shape.epilogue or any(k in variant for k in UNROLLED_KEYS) or not variant.get('dense', 1):
    return None
  if shape.M > 128 or max(t.K for t in shape.terms) > 128 or shape.N > 128:
    return None
  from ..codegen.coltile import coltile_params
  from ..codegen.rowblock import rowblock_params
  p = rowblock_params(shape, variant) if 'rc' not in variant else None
  if p is not None:
    return p if variant.get('dense') or loops_pay(shape, p[0]['wcols']) else None
  stored = sum(t.A.storage_size() for t in shape.terms)
  dense = sum(shape.M * t.K for t in shape.terms)
  # row tiles against the unrolled program (32 to 100 columns, strided, 20,000 and 60,000 elements): several
  # terms, 56x56x40 at 42 % (2,634 values) 0.80, at 60 % 1.56, 56x56x32 at 45 % (4,253) 1.3, 72x72x64 at
  # 42 % (6,532) 3.1; one product, 60x84 at 42 % 0.81, at 50 % 0.87, 84x84 at 55 % 0.91, at 60 % 1.02, at
  # 70 % 1.04-1.24, 100x100 at 55 % 0.94, at 70 % (7,000) 1.8-3.0; with a short pattern it stays
  # unrolled however full that is (50x37 at 95 % times 37x116, 11,570 elements: 194 us, row tiles 238)
  lone = len(shape.terms) == 1 and shape.terms[0].R is None and shape.terms[0].A.sparse
  least = 0.58 if lone else 0.4 if stored > 3500 else 0.5
  if ('rc' in variant or 'dense' in variant or (stored > UNROLLED_MAX_FMAS and stored >= least * dense) or stored > UNROLLED_FETCH_BOUND
      or (stored > 0.8 * dense and not lone)):
    return coltile_params(shape, variant)
  return None


def is_wide_product(shape: LeftChain, fp_size, variant):
  """One dense product with more columns than row blocks hold: the tiled generator's, whose
  elements need no U phase (20,000 elements: 56x56x40 139 us, row tiles 152, unrolled 209;
  32x32x32 41 / 57 / 64; 84x84x64 448 / 496 / 1,205). Against unrolled programs over 37 shapes from
  4x4 to 128x128 with 32 to 128 columns, 150 to 60,000 elements: 1.0 (20x25x100) to 7.5 times as
  fast, 2.3 on average."""
  return (fp_size == 4 and len(shape.terms) == 1 and shape.terms[0].R is None and not shape.terms[0].A.sparse
          and shape.N > 28 and not shape.epilogue and not variant)


def colprog_plan(chain, shape: LeftChain, fp_size, variant):
  if is_wide_product(shape, fp_size, variant):
    return None
  p = row_program(shape, fp_size, variant)
  if p is not None:
    return Plan('colprog', p[0], p[1], p[0]['threads'], note=f'M={shape.M} N={shape.N} terms={len(shape.terms)}')
  if 'threads' in variant:
    return _colprog_plan(chain, shape, fp_size, variant, variant['threads'])
  p = _colprog_plan(chain, shape, fp_size, variant, 128)
  if p is not None and 2 * (p.smem_bytes + 1024) > COLPROG_SMEM_PER_SM:
    wide = _colprog_plan(chain, shape, fp_size, variant, 256)
    # only where the wider tile keeps the prefetch stage (measured only in that form)
    if wide is not None and wide.params['prefetch'] >= p.params['prefetch']:
      return wide
  return p


def unrolled_fits(shape: LeftChain):
  """Whether the FP32 unrolled column program takes the chain by itself."""
  return _colprog_plan(None, shape, 4, {}, 128) is not None


def _colprog_plan(chain, shape: LeftChain, fp_size, variant, threads):
  from ..codegen.colprog import tile_elements
  chunk = variant.get('chunk', 16)
  sizes = [t.A.storage_size() for t in shape.terms]
  a_total = sum(sizes)
  if 'a_source' in variant:
    a_source = variant['a_source']
  elif a_total <= COLPROG_CONST_A:
    a_source = 'const'
  else:
    a_source = 'smem'
  const_terms = int(variant.get('const_terms', 0))
  if a_source == 'mixed' and 'const_terms' not in variant:
    acc = 0
    for n in sizes:
      if acc + n > COLPROG_CONST_MIXED:
        break
      acc += n
      const_terms += 1
    if const_terms == 0:
      a_source = 'smem'
  vec = 4 if fp_size == 4 else 2
  chunk = max(vec, (chunk + vec - 1) // vec * vec)
  if shape.M > 128 or shape.N > threads:
    return None
  if a_total > COLPROG_MAX_FMAS and variant.get('strategy') != 'colprog':
    return None
  cols = int(variant.get('cols', 1))
  rsplit = int(variant.get('rsplit', 1))
  if rsplit > 1 and (shape.epilogue or threads % rsplit or shape.N > threads // rsplit):
    rsplit = 1   # the elementwise epilogue needs whole columns in one thread
  te = tile_elements(shape, threads // rsplit, cols)
  kmax = max(t.K for t in shape.terms)
  upitch = variant.get('upitch', 'odd' if a_source == 'mixed' else 'vec')
  pitch = (kmax | 1) if upitch == 'odd' else (kmax + vec - 1) // vec * vec + vec
  if a_source == 'const' and a_total * fp_size > 48 * 1024:
    a_source = 'smem'
  n_const = {'const': len(sizes), 'smem': 0}.get(a_source, const_terms)
  a_smem_vals = sum(sizes[n_const:])
  prefetch = int(variant.get('prefetch', 1))
  smem = max(te * shape.N * pitch, te * shape.N * shape.M) * fp_size
  r_staged = sum(te * ((t.R.storage_size() + vec - 1) // vec * vec) for t in shape.terms
                 if t.R is not None and t.R.kind == 'batched') * fp_size
  if a_smem_vals:
    smem += (a_smem_vals + vec) * fp_size
  stage = sum(te * ((op.storage_size() if op.sparse else op.element_volume()) + vec - 1) // vec * vec
              for op in {id(o): o for t in shape.terms for o in (t.B, t.R)
                         if o is not None and o.kind == 'batched'}.values()) * fp_size
  if not prefetch or smem + stage > SMEM_LIMIT:
    prefetch = 0
    smem += r_staged
  else:
    smem += stage
  if smem > SMEM_LIMIT:
    return None
  # __launch_bounds__(128, 2) measured 4-5 % faster on the order-6 chain at every chunk size
  # (2.60e8 -> 2.70e8 el/s at chunk 16); 256-thread CTAs gain nothing from it
  default_mb = 2 if threads == 128 and rsplit == 1 else 0
  params = {'threads': threads, 'chunk': chunk, 'min_blocks': variant.get('min_blocks', default_mb),
            'a_source': a_source, 'prefetch': prefetch}
  if a_source == 'mixed':
    params['const_terms'] = n_const
  if upitch != 'vec':
    params['upitch'] = upitch
  if cols != 1:
    params['cols'] = cols
  if rsplit != 1:
    params['rsplit'] = rsplit
  return Plan('colprog', params,
              smem, threads, note=f'M={shape.M} N={shape.N} terms={len(shape.terms)} tile={te}')


def tcsplit_plan(chain, shape, precision, variant):
  if shape.epilogue:  # elementwise epilogues run on the column programs only
    return None
  from ..codegen import tcsplit
  return tcsplit.plan(chain, shape, precision, variant)


def dmma_plan(chain, shape, variant):
  if shape.epilogue:
    return None
  from ..codegen import dmma, dmma_rows
  p = dmma_rows.plan(shape, variant)
  if p is not None:
    return Plan('dmma', *p, note=f'M={shape.M} N={shape.N} terms={len(shape.terms)}')
  return dmma.plan(chain, shape, variant, SMEM_LIMIT)
