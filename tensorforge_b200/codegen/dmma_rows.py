"""FP64 tensor-core row blocks (DMMA, `mma.sync.m8n8k4.f64`) for shared-left GEMM chains.

    out_e (+)= sum_t (A_t * B_e) * R_{e,t}      (terms sharing the per-element B_e)

A warp owns eight elements and eight rows of their outputs. Its DMMA tiles have the elements
as rows and A's rows as columns, one tile per (term t, column m of B):

    W_t[m](e, i) = sum_l B_e[l, m] * A_t[i, l]      8 elements x 8 rows, K in steps of 4

so that a lane ends up with all its columns m of W_t for one element and two rows, and the
product with R_{e,t} (its pattern unrolled) needs no exchange: no U_t = B_e R_t in shared
memory, no U phase, no staging of the output. Per step of four l a warp loads one fragment
per column of B and one per term of A and issues their product in DMMAs: 5 + 3 loads for 15
DMMAs with the five columns at a time that the order-6 chain takes, where the column-block
form (codegen/dmma.py) loads four for three. B and R of the next tile come in by cp.async
while the current one runs; one barrier per tile.

What bounds it: the DMMA rate (A is dense: 169,344 flops per element of the order-6 chain, at
37.0 TFLOP/s 4.6 ns) and its split into seven row blocks, which leaves two of an SM's four
sub-partitions one warp short of the other two: 314 us for 60,000 elements of the order-6
chain. Measured on B200 against the column-block form, 60,000 elements: that chain 474 -> 393 us,
56x56x9 products through pointer arrays 261 -> 155 us, 20x27 chain 368 -> 263 us, 10x9 dense
chain 54 -> 49 us.

Bank conflicts: element slots and A's columns are 4 (mod 8) doubles long, so the four l and
the elements (or rows) of a half-warp fall on different banks.
"""
from ..plan.chains import match_left_chain
from .colprog import _ColProg, _pad, resident_grid, CP_HELPERS
from .dmma import DMMA_HELPERS

SMEM_PER_CTA = 227 * 1024
SMEM_PER_SM = 228 * 1024
MAX_DOUBLES = 66    # accumulators of W and out per lane


def _slot(n):
  """n doubles rounded up to 4 (mod 8)."""
  return n + (4 - n) % 8


def layout(shape, te):
  """Doubles of A and of one operand buffer; offsets and per-element slots inside the buffer."""
  rb = -(-shape.M // 8)
  t0 = shape.terms[0]
  a = len(shape.terms) * _pad(t0.K, 4) * (8 * rb + 4)
  off = {t0.B.name: (0, _slot(t0.P * t0.K))}
  at = te * off[t0.B.name][1]
  for t in shape.terms:
    if t.R is not None and t.R.name not in off:
      n = _pad(t.R.storage_size(), 4) + 2     # 2 (mod 4): elements' 16-byte loads on different banks
      off[t.R.name] = (at, n)
      at += te * n
  return a, _pad(at, 2), off


def pays(shape, warps):
  """Whether row blocks with `warps` resident warps per SM beat the column-block form.

  Measured on B200, column blocks / row blocks, 20,000 and 60,000 elements. Few warps, because an
  element's operands are large: 8x66x9 (two) 0.65, 16x66x12 (four) 0.69, 20x60x12 (six) 0.85, 32x60x12
  (eight) 1.01, 66x40x9 (ten) 1.03, chains of three terms 16x27 (two) 0.66, 20x27 (three) 0.90, 24x20
  (three) 1.12, 30x20 (four) 1.37. Short contractions into columns that are not whole 16-byte pairs or
  fours, where the column blocks' staged stores win unless the output is accumulated: nine columns,
  121x8 0.55, 121x16 0.68, 121x24 0.89, 77x12 0.81, 41x20 0.86, 25x12 0.75, 13x12 0.84 (odd rows),
  122x6 0.81, 122x12 0.86, 26x12 0.90 (even), 64x6 1.14, 121x40 1.12, 122x20 1.1; four columns 65x8 0.81,
  25x6 0.85, 25x12 0.95, others 0.95-1.2."""
  t, lone = shape.terms[0], shape.terms[0].R is None
  if warps < 3 or (lone and shape.N >= 9 and warps < 8):
    return False
  if lone and shape.N >= 4 and not shape.accumulate:
    short = (24 if shape.N > 4 else 8) if shape.M % 2 else 12 if shape.M % 4 and shape.N > 4 else 0
    return t.K > short
  return True


def plan(shape, variant):
  """(plan parameters, shared-memory bytes, threads), or None where the column-block form stays."""
  from .rowblock import applies
  if any(k in variant for k in ('columns', 'tile_elements', 'nsplit', 'prefetch')) or not applies(shape):
    return None
  nt, P, N = len(shape.terms), shape.terms[0].P, shape.N
  lone = shape.terms[0].R is None
  fits = [mc for mc in range(1, P + 1) if nt * mc * 2 + (0 if lone else 2 * N) <= MAX_DOUBLES]
  if not fits or 2 * N > MAX_DOUBLES:
    return None
  # columns of B at a time: as few passes over A as the accumulators allow, evenly filled
  passes = -(-P // max(fits))
  mc = max(1, min(P, variant.get('mc', -(-P // passes))))
  if lone and mc != P:
    return None
  rb = -(-shape.M // 8)
  regs = _pad(2 * (nt * mc * 2 + (0 if lone else 2 * N)) + 2 * (mc + nt) + 20, 8)
  best = None
  for groups in ((variant['groups'],) if 'groups' in variant else range(1, 17)):
    a, buf, _ = layout(shape, 8 * groups)
    smem, threads = (a + 2 * buf) * 8, 32 * rb * groups
    if smem > SMEM_PER_CTA or not 64 <= threads <= 1024:
      continue
    # most resident warps; among equals the smallest CTAs (10x9, 60,000 elements: three CTAs of
    # four warps 49 us, one of twelve 63)
    warps = min(SMEM_PER_SM // (smem + 1024), 65536 // (regs * threads)) * threads // 32
    if warps and (best is None or warps > best[0]):
      best = (warps, groups, smem, threads)
  if best is None or not ({'mc', 'groups'} & set(variant) or pays(shape, best[0])):
    return None
  _, groups, smem, threads = best
  return {'tile_elements': 8 * groups, 'mc': mc}, smem, threads


class _DmmaRows(_ColProg):
  def __init__(self, chain, shape, plan_, ctx, base):
    self.chain, self.s, self.plan, self.base = chain, shape, plan_, base
    self.ctx, self.T = ctx, 'double'
    self.lines, self.ind = [], 0
    self.TE, self.MC = plan_.params['tile_elements'], plan_.params['mc']
    self.RB = -(-shape.M // 8)
    self.BT = 32 * self.RB * (self.TE // 8)
    self.MP = 8 * self.RB + 4
    t0 = shape.terms[0]
    self.NT, self.P, self.K, self.K4 = len(shape.terms), t0.P, t0.K, _pad(t0.K, 4)
    self.a_total, self.buf, self.off = layout(shape, self.TE)
    self.smem = (self.a_total + 2 * self.buf) * 8

  def _stage_a(self, b):
    BT, M = self.BT, self.s.M
    self.w(f'for (int q = threadIdx.x; q < {self.a_total}; q += {BT}) sA[q] = 0.0;')
    self.w('__syncthreads();')
    for ti, t in enumerate(self.s.terms):
      at = ti * self.K4 * self.MP
      self.w('#pragma unroll 8')
      self.w(f'for (int q = threadIdx.x; q < {t.A.storage_size()}; q += {BT})')
      if t.A.sparse:
        self.w(f'  sA[{at} + aoff_{b}_{ti}[q]] = __ldg({t.A.name} + q);')
      else:
        self.w(f'  sA[{at} + q / {M} * {self.MP} + q % {M}] = __ldg({t.A.name} + q);')

  def _tables(self, b):
    for ti, t in enumerate(self.s.terms):
      if t.A.sparse:
        dst = [0] * t.A.storage_size()
        for (i, l), pos in t.A.sparse_lookup().items():
          dst[pos] = l * self.MP + i
        self.w(f'static __device__ const unsigned short aoff_{b}_{ti}[{len(dst)}] = {{{", ".join(map(str, dst))}}};')

  def _fetch(self, g, buf):
    """cp.async B and R of the tile at group `g` into `buf`, 16 bytes at a time where the address
    allows it. A masked element's memory is not touched, nor its pointer followed: its slot keeps
    what it held, and its rows are computed and dropped."""
    BT = self.BT
    ops = {o.name: o for o in self.chain.operands}
    self.open('')
    self.w(f'const size_t pe0 = ({g}) * 8u, pe1 = last * 8u < numElements ? last * 8u : (size_t)numElements;')
    self.w(f'const unsigned pn = pe1 - pe0 < {self.TE}u ? (unsigned)(pe1 - pe0) : {self.TE}u;')
    # Pointer arrays: warp w takes elements w, w + warps, ... Of more than two, its lanes load all
    # addresses at once, for every operand, before the first copy (8x8x9 chain of three terms, 88
    # elements per tile, 60,000 elements: one after the other 85 us, 39).
    warps, pointers = BT // 32, [n for n in self.off if ops[n].addressing.name == 'PTR_BASED']
    ahead = -(-self.TE // warps) > 2
    if pointers and ahead:
      self.w(f'const unsigned pe = warp + lane * {warps}u;')
      self.w('const bool there = pe < pn && (flags == nullptr || flags[pe0 + pe] != 0u);')
      for name in pointers:
        self.w(f'const unsigned long long at_{name} = there ? reinterpret_cast<unsigned long long>({self._elem_ptr(ops[name], "(pe0 + pe)")}) : 0ull;')
    for name, (at, slot) in self.off.items():
      op = ops[name]
      vals = self.P * self.K if name == self.s.terms[0].B.name else op.storage_size()
      vec = vals % 2 == 0
      n = vals // 2 if vec else vals

      def body(q):
        self.w(f'const double* const x = src + {q}{" * 2u" if vec else ""};')
        self.w(f'double* const y = {buf} + {at} + ei * {slot}u + {q}{" * 2u" if vec else ""};')
        if vec:
          self.w('if ((reinterpret_cast<uintptr_t>(x) & 15u) == 0u) tfb_cp::copy16(y, x);')
          self.w('else { tfb_cp::copy8(y, x); tfb_cp::copy8(y + 1, x + 1); }')
        else:
          self.w('tfb_cp::copy8(y, x);')
      if name in pointers:
        if ahead:
          self.open(f'for (unsigned i = 0; i < {-(-self.TE // warps)}u; ++i)')
          self.w(f'const double* const src = reinterpret_cast<const double*>(__shfl_sync(0xffffffffu, at_{name}, i));')
          self.w('if (src == nullptr) continue;')
          self.w(f'const unsigned ei = warp + i * {warps}u;')
        else:
          self.open(f'for (unsigned ei = warp; ei < pn; ei += {warps}u)')
          self.w(f'const double* const src = {self._elem_ptr(op, "(pe0 + ei)")};')
          self.w('if (flags != nullptr && flags[pe0 + ei] == 0u) continue;')
        self.open(f'for (unsigned q = lane; q < {n}u; q += 32u)')
        body('q')
      else:
        self.open(f'for (unsigned i = threadIdx.x; i < pn * {n}u; i += {BT}u)')
        self.w(f'const unsigned ei = i / {n}u, q = i - ei * {n}u;')
        self.w('if (flags != nullptr && flags[pe0 + ei] == 0u) continue;')
        self.w(f'const double* const src = {self._elem_ptr(op, "(pe0 + ei)")};')
        self.open('')
        body('q')
      self.close()
      self.close()
    self.close()

  def _compute(self):
    s, NT, P, K, K4, N = self.s, self.NT, self.P, self.K, self.K4, self.s.N
    lone = s.terms[0].R is None
    bslot = self.off[s.terms[0].B.name][1]
    self.w(f'const double* const bq = cur + el * {bslot}u + kq;')
    self.w(f'const double* const aq = sA + kq * {self.MP}u + rb * 8u + (lane >> 2);')
    if not lone:
      self.w(f'double o[{N}][2] = {{}};')
    for ti, t in enumerate(s.terms):
      if t.R is not None:
        at, slot = self.off[t.R.name]
        self.w(f'const double2* const rq{ti} = reinterpret_cast<const double2*>(cur + {at} + el * {slot}u);')
    c0 = 0
    while c0 < P:
      mc = min(self.MC, P - c0)
      if not lone:
        self.open('')
      self.w(f'double w[{NT}][{mc}][2] = {{}};')
      steps = K // 4
      for l0, count, head in ((0, steps, True), (steps * 4, 1, False)):
        if head:
          if count == 0:
            continue
          self.w('#pragma unroll 2')
          self.open(f'for (int l = 0; l < {steps * 4}; l += 4)')
          l, ok = 'l', ''
        else:
          if K % 4 == 0:
            continue
          # the last, partial step: lanes past K multiply zeros
          self.open('')
          l, ok = str(l0), f'kq < {K - l0}u ? '
        self.w(f'double a[{NT}], b[{mc}];')
        self.w('#pragma unroll')
        self.w(f'for (int m = 0; m < {mc}; ++m) b[m] = {ok}bq[{l} + ({c0} + m) * {K}]{" : 0.0" if ok else ""};')
        self.w('#pragma unroll')
        self.w(f'for (int t = 0; t < {NT}; ++t) a[t] = aq[(t * {K4} + {l}) * {self.MP}];')
        self.w('#pragma unroll')
        self.w(f'for (int m = 0; m < {mc}; ++m)')
        self.w('#pragma unroll')
        self.w(f'  for (int t = 0; t < {NT}; ++t) tfb_dmma::mma(w[t][m][0], w[t][m][1], b[m], a[t]);')
        self.close()
      if not lone:
        for ti, t in enumerate(s.terms):
          look = t.R.sparse_lookup() if t.R.sparse else {(m, j): j * P + m for j in range(N) for m in range(P)}
          used = sorted((pos, m, j) for (m, j), pos in look.items() if c0 <= m < c0 + mc and j < N)
          self.open('')
          for v in sorted({pos // 2 for pos, _, _ in used}):
            self.w(f'const double2 r{v} = rq{ti}[{v}];')
          for pos, m, j in used:
            for h in (0, 1):
              self.w(f'o[{j}][{h}] = fma(w[{ti}][{m - c0}][{h}], r{pos // 2}.{"xy"[pos % 2]}, o[{j}][{h}]);')
          self.close()
        self.close()
      c0 += mc
    o, M, add = s.out, s.M, s.accumulate
    val = (lambda j, h: f'w[0][{j}][{h}]') if lone else (lambda j, h: f'o[{j}][{h}]')
    self.open('if (e < numElements && (flags == nullptr || flags[e] != 0u))')
    self.w(f'double* const dst = {self._elem_ptr(o, "e")} + rb * 8u + 2u * kq;')
    self.w('const unsigned row = rb * 8u + 2u * kq;')

    def scalar():
      for j in range(N):
        for h in (0, 1):
          self.w((f'if (row + {h}u < {M}u) ' if M % 8 else '') + f'dst[{j * M + h}] {"+=" if add else "="} {val(j, h)};')
    if M % 2 == 0:
      self.open(f'if ({f"row < {M}u && " if M % 8 else ""}(reinterpret_cast<uintptr_t>(dst) & 15u) == 0u)')
      for j in range(N):
        y = f'*reinterpret_cast<double2*>(dst + {j * M})'
        if add:
          self.open('')
          self.w(f'const double2 p = {y};')
          self.w(f'{y} = make_double2(p.x + {val(j, 0)}, p.y + {val(j, 1)});')
          self.close()
        else:
          self.w(f'{y} = make_double2({val(j, 0)}, {val(j, 1)});')
      self.close()
      self.open('else')
      scalar()
      self.close()
    else:
      scalar()
    self.close()

  def emit(self, globals_):
    b, BT = self.base, self.BT
    kname = f'kernel_{b}'
    self.w(CP_HELPERS)
    self.w(DMMA_HELPERS)
    self.w(f'// generated by tensorforge_b200 (strategy: dmma, row blocks, {self.TE} elements per tile, {self.MC} columns at a time)')
    self.w('// meta data:')
    for o in self.chain.operands:
      self.w(f'// {o.tensor.gen_descr()}')
    for st in self.chain.stages:
      self.w(f'// {st.descr}')
    self._tables(b)
    self.w(f'__global__ void __launch_bounds__({BT}) {kname}({", ".join(self.params(globals_))}) {{')
    self.ind += 1
    self.w('extern __shared__ __align__(16) unsigned char tfb_smem_raw[];')
    self.w('double* const sA = reinterpret_cast<double*>(tfb_smem_raw);')
    self.w(f'double *cur = sA + {self.a_total}, *next = cur + {self.buf};')
    self.w(f'const unsigned lane = threadIdx.x & 31u, kq = lane & 3u, warp = threadIdx.x >> 5;')
    self.w(f'const unsigned rb = warp % {self.RB}u, el = warp / {self.RB}u * 8u + (lane >> 2);')
    # Each CTA takes one range of groups of eight elements: the last of its tiles is smaller where
    # the range is odd, and no CTA has more than one group above another. Against whole
    # tiles dealt in turn, order-6 chain: 3,000 elements 38.4 -> 30.2 us, 8,000 69 -> 61, 60,000 397 -> 393.
    self.w('const size_t groups = (numElements + 7u) / 8u, last = groups * (blockIdx.x + 1u) / gridDim.x;')
    self.w('size_t g = groups * blockIdx.x / gridDim.x;')
    self.w('if (g < last)')
    self._fetch('g', 'cur')
    self.w('tfb_cp::commit();')
    self._stage_a(b)
    self.open(f'for (; g < last; g += {self.TE // 8}u)')
    self.w('tfb_cp::wait_all();')
    self.w('__syncthreads();  // this tile has landed, and nobody reads the other buffer any more')
    self.w(f'if (g + {self.TE // 8}u < last)')
    self._fetch(f'g + {self.TE // 8}u', 'next')
    self.w('tfb_cp::commit();')
    self.w('const size_t e = g * 8u + el;')
    # whole warps: the DMMAs need all lanes; rows of missing elements are computed and dropped
    self.open('if (g + el / 8u < last)')
    self._compute()
    self.close()
    self.w('double* const swap = cur;')
    self.w('cur = next;')
    self.w('next = swap;')
    self.close()
    self.w('tfb_cp::wait_all();')
    self.ind -= 1
    self.w('}')
    args = []
    for t, _ in globals_:
      args.append(t.name)
      if t.addressing.name not in ('NONE', 'SCALAR'):
        args.append(f'{t.name}_extraOffset')
    args += ['numElements', 'flags']
    self.plan.smem_bytes = self.smem
    pre = [resident_grid(kname, BT, self.smem),
           '  const size_t groups = (numElements + 7) / 8;',
           f'  {kname}<<<(unsigned)(groups < (size_t)cap ? groups : (size_t)cap), {BT}, {self.smem}, stream>>>({", ".join(args)});',
           '  CHECK_ERR;']
    launch = {'kernel': kname, 'block': BT, 'elements_per_block': self.TE, 'smem': self.smem, 'args': args,
              'pre': '\n'.join(pre), 'launched': True}
    return '\n'.join(self.lines), launch, ''


def emit_dmma_rows(chain, plan_, context, base_name, globals_):
  return _DmmaRows(chain, match_left_chain(chain), plan_, context, base_name).emit(globals_)
