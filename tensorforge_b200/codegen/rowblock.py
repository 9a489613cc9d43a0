"""Row-block programs (CUDA cores, FP32) for shared-left GEMM chains with few columns.

    out_e (+)= sum_t (A_t * B_e) * R_{e,t}

for chains whose terms share the per-element operand B_e. A thread owns RM rows of one
element: it forms its rows of W_t = A_t B_e for all terms t and all P columns of B_e at
once, in registers, multiplies them by R_{e,t} (its pattern unrolled) and writes its rows of
out_e. Nothing is exchanged between threads: no U_t = B_e R_t in shared memory, no barrier
but the one that hands over the next tile's operands, which cp.async brings in while the
current tile runs.

Why this split: the unrolled column program (codegen/colprog.py) is bound by shared
memory. Per 32 output columns of the order-6 chain (56 x 9, three terms, A at 45 %) it
takes 2,340 cycles of an SM's shared-memory pipe for A (a 16-byte load, 2.2 cycles, per four
FMAs) and 750 for writing and re-reading U, 3,090 of its 3,830 cycles; its 4,253 FMAs would
take 1,063. Here A is dense (zeros outside its pattern), so the FMAs take 2,353 cycles at
the nominal rate, but per step of l a thread loads 12 + 9 values for 108 products, and
neighbouring threads are the same rows of two elements: a 16-byte shared load takes the
SM two cycles when lanes i and i ^ 1 (or i ^ 2) share their address for every i, else four.
The bound is the packed FMA's rate: 54 of them take a warp 139 cycles alone (0.78 of
nominal), 165 here. Measured on B200 against the unrolled program: order-6 chain, 100,003
elements 387 -> 369 us; 10,000 56x56x9 products through pointer arrays 63 -> 22.6 us (dense
A there went through the constant bank, at a miss per 16 values); 84 x 9, 39,900 elements
490 -> 300 us; 84 x 27, in pieces, 20,000 elements 958 -> 527 us (its 9,533 unrolled FMAs are
fetched at one instruction per 8 cycles, having outgrown the instruction cache). Batches below
one wave of tiles are spread over all CTAs: 300 elements of the order-6 chain 20.5 -> 15.3 us
a call.

FMAs are packed, two rows per instruction. Zeros and non-finite values: entries outside
A_t's pattern are multiplied as zeros, which adds nothing for finite B. A thread whose W
comes out non-finite (an infinite or NaN entry of B reaches every row of its column) runs
its sums again through the pattern's bits, so absent entries stay absent. The contraction
order is the descriptors' own, (A_t B_e) R_{e,t}.
"""
import math

from ..plan.chains import match_left_chain
from .colprog import _ColProg, _pad, resident_grid, CP_HELPERS

RB_HELPERS = r'''
#ifndef TFB_ROWBLOCK_HELPERS
#define TFB_ROWBLOCK_HELPERS
namespace tfb_rb {
// A's values of one step: a thread's RM (2 or 4) rows of NT terms, TS values apart.
template <int NT, int RM, int TS>
__device__ __forceinline__ void load_a(float2 (&av)[NT][RM / 2], const float* a) {
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    if constexpr (RM == 4) {
      const float4 x = *reinterpret_cast<const float4*>(a + t * TS);
      av[t][0] = make_float2(x.x, x.y);
      av[t][1] = make_float2(x.z, x.w);
    } else {
      av[t][0] = *reinterpret_cast<const float2*>(a + t * TS);
    }
  }
}
template <int P, int PITCH>
__device__ __forceinline__ void load_b(float2 (&bv)[P], const float* b) {
#pragma unroll
  for (int m = 0; m < P; ++m) bv[m] = *reinterpret_cast<const float2*>(b + m * PITCH);
}
// w[t][m] += a[t] * (component H of b[m])
template <int NT, int RM, int P, int H>
__device__ __forceinline__ void step(float2 (&w)[NT][P][RM / 2], const float2 (&av)[NT][RM / 2], const float2 (&bv)[P]) {
#pragma unroll
  for (int m = 0; m < P; ++m) {
    const float bk = H == 0 ? bv[m].x : bv[m].y;
    const float2 bb = make_float2(bk, bk);
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int i = 0; i < RM / 2; ++i) w[t][m][i] = __ffma2_rn(av[t][i], bb, w[t][m][i]);
  }
}
// W += A B over K steps, operands loaded a step (A) and two steps (B) ahead of their use; the
// last ones (K a multiple of 4) load a row behind A and two values behind B that are not used;
// allocated() keeps them inside the shared memory.
template <int NT, int RM, int P, int MP, int TS, int K, int PITCH>
__device__ __forceinline__ void k_loop(float2 (&w)[NT][P][RM / 2], const float* a, const float* b) {
  float2 a0[NT][RM / 2], a1[NT][RM / 2], b0[P], b1[P];
  load_a<NT, RM, TS>(a0, a);
  load_b<P, PITCH>(b0, b);
  int l = 0;
#pragma unroll 1
  for (; l + 4 <= K; l += 4) {
    load_a<NT, RM, TS>(a1, a + (l + 1) * MP);
    load_b<P, PITCH>(b1, b + l + 2);
    step<NT, RM, P, 0>(w, a0, b0);
    load_a<NT, RM, TS>(a0, a + (l + 2) * MP);
    step<NT, RM, P, 1>(w, a1, b0);
    load_a<NT, RM, TS>(a1, a + (l + 3) * MP);
    load_b<P, PITCH>(b0, b + l + 4);
    step<NT, RM, P, 0>(w, a0, b1);
    load_a<NT, RM, TS>(a0, a + (l + 4) * MP);
    step<NT, RM, P, 1>(w, a1, b1);
  }
  if (K % 4 >= 1) step<NT, RM, P, 0>(w, a0, b0);
  if (K % 4 >= 2) {
    load_a<NT, RM, TS>(a1, a + (K / 4 * 4 + 1) * MP);
    step<NT, RM, P, 1>(w, a1, b0);
  }
  if (K % 4 == 3) {
    load_a<NT, RM, TS>(a0, a + (K - 1) * MP);
    load_b<P, PITCH>(b1, b + K - 1);
    step<NT, RM, P, 0>(w, a0, b1);
  }
}
// The sums through A's pattern: bits[(t * K + l) * W ...] holds the rows of step l that exist.
template <int NT, int RM, int P, int MP, int TS, int K, int PITCH, int W>
__device__ __forceinline__ void k_loop_pattern(float2 (&w)[NT][P][RM / 2], const float* a, const float* b,
                                               const unsigned* bits, int row0) {
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int m = 0; m < P; ++m)
#pragma unroll
      for (int i = 0; i < RM / 2; ++i) w[t][m][i] = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int l = 0; l < K; ++l) {
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const unsigned y = row0 < 32 * W ? bits[(t * K + l) * W + (row0 >> 5)] >> (row0 & 31) : 0u;
      const float* x = a + t * TS + l * MP;
#pragma unroll
      for (int m = 0; m < P; ++m) {
        const float bk = b[m * PITCH + l];
#pragma unroll
        for (int i = 0; i < RM / 2; ++i) {
          if ((y >> (2 * i)) & 1u) w[t][m][i].x = fmaf(x[2 * i], bk, w[t][m][i].x);
          if ((y >> (2 * i)) & 2u) w[t][m][i].y = fmaf(x[2 * i + 1], bk, w[t][m][i].y);
        }
      }
    }
  }
}
}  // namespace tfb_rb
#endif
'''

SMEM_PER_CTA = 227 * 1024
SMEM_PER_SM = 228 * 1024
MAX_ACC = 112


def applies(shape):
  """One dense per-element B for all terms; every R per element (or absent in a lone term)."""
  b = shape.terms[0].B
  if any(t.B is not b for t in shape.terms):
    return False
  if any(t.R is None for t in shape.terms) and len(shape.terms) > 1:
    return False
  if any(t.R is not None and (t.R.kind != 'batched' or t.R is b) for t in shape.terms):
    return False
  return shape.M <= 128 and shape.terms[0].K <= 128


def slot(n, rg, lanes):
  """Values from one element's operand to the next's: `n` (a multiple of four), or four more where
  the elements that `lanes` neighbouring threads work on (pairs of elements, 2 rg threads
  each) would meet on the same banks. With 480 values per element, 12x40x12 products, 40,000
  elements, took 61 us, eight elements' loads on one bank."""
  elements = 2 * (-(-lanes // (2 * rg)) + 1)
  return n if 32 // math.gcd(n, 32) >= elements or n % 8 else n + 4


def layout(shape, rm, te):
  """Shared-memory values of A and of one operand buffer, and offsets and slots inside the buffer."""
  rg = -(-shape.M // rm)
  a = _pad(sum(t.K for t in shape.terms) * rg * rm, 4)
  t0 = shape.terms[0]
  pitch = _pad(t0.K, 4)
  off = {t0.B.name: (0, slot(t0.P * pitch, rg, 16))}     # 8-byte loads: half a warp at a time
  at = te * off[t0.B.name][1]
  for t in shape.terms:
    if t.R is not None and t.R.name not in off:
      n = slot(_pad(t.R.storage_size(), 4), rg, 8)       # 16-byte loads: a quarter
      off[t.R.name] = (at, n)
      at += te * n
  return a, at, off


def allocated(shape, rm, a, buf, buffers):
  """Shared-memory values of a CTA: A, the operand buffers and what the K loop loads ahead of its
  last step, a row of A behind A (small buffers do not cover it: one 128x8 times 8x1 product has
  64 values behind A and rows of 128) and two values of B."""
  return a + max(buffers * buf + 4, _pad(shape.M, rm))


def rowblock_params(shape, variant):
  """(plan parameters, shared-memory bytes), or None where the accumulators do not fit.

  RM is 4, one 16-byte piece of a column of A (56x56x9 products, 39,900 elements: 68 us, 73 with
  2 rows, 79 with 8). Where W of all terms and columns does not fit beside the outputs it is
  formed for as many columns of B at a time as leave at most 56 values of W, with RM = 2. All
  terms at once, so that B is loaded once for them: per step 3 + 9/2 8-byte shared loads for 54
  products where one term and 14 columns take 1 + 7 for 28 and four rows of one term and 9
  columns 1 + 9/4 16-byte ones for 36 (84x27 1,019 us, 1,160 and 1,099; 20x27 91, 103 and 104).
  Threads and input buffers by the warps an SM then holds, eight being enough; two buffers
  hide a tile's copies, several CTAs per SM cover each other's with one (10x27: four CTAs of 64
  threads with one buffer 87 us, one of 256 with two 109)."""
  nt, P, N = len(shape.terms), shape.terms[0].P, shape.N
  lone = shape.terms[0].R is None
  if not applies(shape) or N > 28 or lone and 4 * P > MAX_ACC:
    return None
  whole = nt * 4 * P <= MAX_ACC
  rm = variant.get('rm', 4 if whole else 2)
  if rm not in (2, 4):
    return None
  cols = P if whole else max(1, min(P, variant.get('wcols', -(-P // -(-P // max(1, 56 // (rm * nt)))))))
  terms = max(1, min(nt, variant.get('wterms', nt)))
  rg = -(-shape.M // rm)
  regs = terms * rm * cols + (0 if lone or whole else rm * N) + 4 * cols + 2 * rm * terms + 40
  out = None
  for bt in ((variant['threads'],) if 'threads' in variant else (128, 256, 64)):
    for buffers in ((variant['buffers'],) if 'buffers' in variant else (2, 1)):
      te = min(variant.get('te', bt), bt // rg)
      while te > 0:
        a, buf, _ = layout(shape, rm, te)
        smem = 4 * allocated(shape, rm, a, buf, buffers)
        if smem <= SMEM_PER_CTA:
          break
        te -= 1
      if te < 1:
        continue
      ctas = min(SMEM_PER_SM // (smem + 1024), 65536 // (_pad(min(regs, 255), 8) * bt), 32)
      score = (min(ctas * te * rg / 32, 8) * (1 if buffers == 2 else 0.93 if ctas > 1 else 0.9)
               * (1 + 0.03 * min(ctas, 4)))
      if ctas and (out is None or score > out[0] * 1.01):
        out = (score, {'threads': bt, 'rows': rm, 'te': te, 'wcols': cols, 'wterms': terms, 'prefetch': 1, 'a_source': 'dense',
                       'buffers': buffers}, smem)
  return out and out[1:]


class _RowBlock(_ColProg):
  skip_masked = True

  def __init__(self, chain, shape, plan, ctx, base):
    super().__init__(chain, shape, plan, ctx, base)
    self.RM, self.TE = plan.params['rows'], plan.params['te']
    self.RG = -(-shape.M // self.RM)
    self.MP = self.RG * self.RM
    self.W = -(-shape.M // 32)
    self.NT, self.P, self.K = len(shape.terms), shape.terms[0].P, shape.terms[0].K
    self.bpitch = _pad(self.K, 4)
    self.a_total, self.buf, self.off = layout(shape, self.RM, self.TE)
    self.PC, self.buffers = plan.params['wcols'], plan.params['buffers']
    self.NG = plan.params['wterms']   # terms whose W a thread forms at once
    self.smem = 4 * allocated(shape, self.RM, self.a_total, self.buf, self.buffers)
    self.sparse = any(t.A.sparse for t in shape.terms)

  def _tables(self, b):
    """Where each stored value of a sparse A_t goes, and all terms' patterns as row bits per step."""
    bits = [0] * (self.NT * self.K * self.W)
    for ti, t in enumerate(self.s.terms):
      at = ti * self.K * self.MP
      if t.A.sparse:
        dst = [0] * t.A.storage_size()
        for (i, l), pos in t.A.sparse_lookup().items():
          dst[pos] = l * self.MP + i
          bits[(ti * self.K + l) * self.W + (i >> 5)] |= 1 << (i & 31)
        self.w(f'static __device__ const unsigned short aoff_{b}_{ti}[{len(dst)}] = {{{", ".join(map(str, dst))}}};')
      else:
        for l in range(self.K):
          for i in range(self.s.M):
            bits[(ti * self.K + l) * self.W + (i >> 5)] |= 1 << (i & 31)
    if self.sparse:
      self.w(f'static __device__ const unsigned abits_{b}[{len(bits)}] = {{{", ".join(f"{x}u" for x in bits)}}};')

  def _stage_a(self, b):
    s, BT = self.s, self.BT
    self.w(f'for (int q = threadIdx.x; q < {self.a_total // 4}; q += {BT}) reinterpret_cast<float4*>(sA)[q] = make_float4(0.f, 0.f, 0.f, 0.f);')
    self.w('__syncthreads();')
    for ti, t in enumerate(s.terms):
      at = ti * self.K * self.MP
      self.w('#pragma unroll 8')
      self.w(f'for (int q = threadIdx.x; q < {t.A.storage_size()}; q += {BT})')
      if t.A.sparse:
        self.w(f'  sA[{at} + aoff_{b}_{ti}[q]] = __ldg({t.A.name} + q);')
      elif self.MP == s.M:
        self.w(f'  sA[{at} + q] = __ldg({t.A.name} + q);')
      else:
        self.w(f'  sA[{at} + q / {s.M} * {self.MP} + q % {s.M}] = __ldg({t.A.name} + q);')

  def _fetch(self, tile, buf):
    """cp.async a tile's B and R into `buf` (16 bytes at a time where the address allows it)."""
    BT = self.BT
    ops = {o.name: o for o in self.chain.operands}
    self.open('')
    self.w(f'const size_t pe0 = ({tile}) * te;')
    self.w('const unsigned pn = numElements - pe0 < te ? (unsigned)(numElements - pe0) : te;')
    if any(self.skips(ops[name]) and ops[name].addressing.name != 'PTR_BASED' for name in self.off):
      self._live_words(self.TE, '{} < pn')
    for name, (at, ev) in self.off.items():
      op = ops[name]
      dense = name == self.s.terms[0].B.name
      vals, cols, pitch = (self.K, self.P, self.bpitch) if dense else (op.storage_size(), 1, ev)
      vec = vals % 4 == 0
      chunks = vals // 4 if vec else vals

      def body(q, src, dst):
        per = chunks * cols
        if cols > 1:
          self.w(f'const unsigned c = {q} / {chunks}u, r = ({q} - c * {chunks}u){" * 4u" if vec else ""};')
          self.w(f'const float* const x = {src} + c * {vals}u + r;')
          self.w(f'float* const y = {dst} + c * {pitch}u + r;')
        else:
          self.w(f'const float* const x = {src} + {q}{" * 4u" if vec else ""};')
          self.w(f'float* const y = {dst} + {q}{" * 4u" if vec else ""};')
        if vec:
          self.w('if ((reinterpret_cast<uintptr_t>(x) & 15u) == 0u) tfb_cp::copy16(y, x);')
          self.w('else { tfb_cp::copy4(y, x); tfb_cp::copy4(y + 1, x + 1); tfb_cp::copy4(y + 2, x + 2); tfb_cp::copy4(y + 3, x + 3); }')
        else:
          self.w('tfb_cp::copy4(y, x);')
      if op.addressing.name == 'PTR_BASED':
        self.open(f'for (unsigned ei = threadIdx.x >> 5; ei < pn; ei += {BT // 32}u)')
        self.w(f'const float* const src = {self._elem_ptr(op, "(pe0 + ei)")};')
        self.w(self._masked('pe0 + ei'))
        self.open(f'for (unsigned q = threadIdx.x & 31u; q < {chunks * cols}u; q += 32u)')
        body('q', 'src', f'{buf} + {at} + ei * {ev}u')
        self.close()
        self.close()
      else:
        def loop(live):
          self.open(f'for (unsigned i = threadIdx.x; i < pn * {chunks * cols}u; i += {BT}u)')
          self.w(f'const unsigned ei = i / {chunks * cols}u, q = i - ei * {chunks * cols}u;')
          if live:
            self.open(f'if ({live})')
          self.w(f'const float* const src = {self._elem_ptr(op, "(pe0 + ei)")};')
          body('q', 'src', f'{buf} + {at} + ei * {ev}u')
          if live:
            self.close()
          self.close()
        self._flagged(op, loop)
    self.close()

  def _compute(self, b):
    """One thread's rows of one element: W for all terms, times R, to global memory."""
    s, RM, P, NT = self.s, self.RM, self.P, self.NT
    H = RM // 2
    lone = s.terms[0].R is None
    whole = self.PC == P and self.NG == NT
    out = (lambda j, i: f'w[0][{j}][{i}]') if lone else (lambda j, i: f'o[{j}][{i}]')
    self.w(f'const float* const bq = cur + ei * {self.off[s.terms[0].B.name][1]}u;')
    if not lone:
      self.w(f'float2 o[{s.N}][{H}];')
    started = set()
    for t0 in range(0, NT, self.NG):
      ng = min(self.NG, NT - t0)
      for c0 in range(0, P, self.PC):
        pc = min(self.PC, P - c0)
        if not whole:
          self.open('')
        every = [f'for (int t = 0; t < {ng}; ++t)', f'for (int m = 0; m < {pc}; ++m)', f'for (int i = 0; i < {H}; ++i)']
        targs = f'{ng}, {RM}, {pc}, {self.MP}, {self.K * self.MP}, {self.K}, {self.bpitch}'
        args = f'w, sA + {t0 * self.K * self.MP} + rg * {RM}u, bq + {c0 * self.bpitch}'
        self.w(f'float2 w[{ng}][{pc}][{H}];')
        for head in every:
          self.w('#pragma unroll')
          self.w(head)
        self.w('  w[t][m][i] = make_float2(0.f, 0.f);')
        self.w(f'tfb_rb::k_loop<{targs}>({args});')
        if self.sparse:
          # one row of one term tells: a non-finite entry of column m of B reaches every row of W
          self.w('float sum0 = 0.f;  // NaN once a column of B holds a value that is not finite')
          self.w('#pragma unroll')
          self.w(f'for (int m = 0; m < {pc}; ++m) sum0 = fmaf(w[0][m][0].x, 0.f, sum0);')
          self.w(f'if (sum0 != 0.f) tfb_rb::k_loop_pattern<{targs}, {self.W}>({args}, abits_{b} + {t0 * self.K * self.W}, rg * {RM});')
        if not lone:
          for ti in range(t0, t0 + ng):
            self._times_r(ti, ti - t0, c0, pc, out, started)
        if not whole:
          self.close()
    if not lone:
      for j in range(s.N):
        for i in range(H):
          if (j, i) not in started:
            self.w(f'{out(j, i)} = make_float2(0.f, 0.f);')
    o, M, N, add = s.out, s.M, s.N, s.accumulate
    self.w(f'float* const dst = {self._elem_ptr(o, "e")} + rg * {RM}u;')
    if M % RM:
      self.w(f'const unsigned row = rg * {RM}u;')

    def rows(width):
      """Stores of `width` rows at a time; rows past the last one are left out. Accumulated outputs test
      each row once for all columns, so that their previous values are loaded together; others
      store a column's rows one after the other (35x9 chain, 20,000 elements: 50.6 us, row by row 53.6)."""
      def store(j, c):
        v = [f'{out(j, h)}.{x}' for h in range(H) for x in 'xy'][c:c + width]
        at = f'dst{f" + {j * M + c}" if j * M + c else ""}'
        test = f'if (row + {c}u < {M}u) ' if M % RM and not add else ''
        if width == 1:
          self.w(f'{test}dst[{j * M + c}] {"+=" if add else "="} {v[0]};')
        elif add:
          self.w(f'{{ float{width}* const y = reinterpret_cast<float{width}*>({at}); const float{width} p = *y; '
                 f'*y = make_float{width}({", ".join(f"p.{x} + {y}" for x, y in zip("xyzw", v))}); }}')
        else:
          self.w(f'{test}*reinterpret_cast<float{width}*>({at}) = make_float{width}({", ".join(v)});')
      if not add:
        for j in range(N):
          for c in range(0, RM, width):
            store(j, c)
        return
      for c in range(0, RM, width):
        if M % RM:
          self.open(f'if (row + {c}u < {M}u)')
        for j in range(N):
          store(j, c)
        if M % RM:
          self.close()
    wide = RM if M % RM == 0 else 2 if M % 2 == 0 else 1
    if wide > 1:
      self.open(f'if ((reinterpret_cast<uintptr_t>(dst) & {4 * wide - 1}u) == 0u)')
      rows(wide)
      self.close()
      self.open('else')
      rows(1)
      self.close()
    else:
      rows(1)

  def _times_r(self, ti, slot, c0, pc, out, started):
    """out += W_t[columns c0 .. c0 + pc) R_t, with the pattern of R_t unrolled."""
    s, P, t = self.s, self.P, self.s.terms[ti]
    at, ev = self.off[t.R.name]
    look = t.R.sparse_lookup() if t.R.sparse else {(m, j): j * P + m for j in range(s.N) for m in range(P)}
    used = [(pos, m - c0, j) for j in range(s.N) for m in range(c0, c0 + pc)
            for pos in (look.get((m, j)),) if pos is not None]
    self.open('')
    self.w(f'const float* const rq = cur + {at} + ei * {ev}u;')
    if pc == P:
      for v in sorted({pos // 4 for pos, _, _ in used}):
        self.w(f'const float4 r{v} = reinterpret_cast<const float4*>(rq)[{v}];')
    for pos, m, j in used:
      r = f'r{pos // 4}.{"xyzw"[pos % 4]}' if pc == P else f'rq[{pos}]'
      self.w(f'{{ const float x = {r}; const float2 xx = make_float2(x, x);')
      for i in range(self.RM // 2):
        prev = out(j, i) if (j, i) in started else 'make_float2(0.f, 0.f)'
        self.w(f'  {out(j, i)} = __ffma2_rn(w[{slot}][{m}][{i}], xx, {prev});')
        started.add((j, i))
      self.w('}')
    self.close()

  def _mine(self):
    """This thread's element of the tile (`ei`, ~0 where it has none) and row block (`rg`)."""
    paired = self.TE // 2 * 2 * self.RG
    self.w('// neighbouring threads: the same rows of two elements (a last odd element follows)')
    self.w(f'unsigned ei = threadIdx.x / {2 * self.RG}u * 2u + (threadIdx.x & 1u), rg = (threadIdx.x >> 1) % {self.RG}u;')
    if self.TE % 2:
      self.w(f'if (threadIdx.x >= {paired}u) {{ ei = threadIdx.x < {paired + self.RG}u ? {self.TE - 1}u : ~0u; rg = threadIdx.x - {paired}u; }}')
    else:
      self.w(f'if (threadIdx.x >= {paired}u) ei = ~0u;')

  def emit_group_functions(self, globals_, gid):
    """Device functions of one group of a grouped launch (see _ColProg.emit_group_functions)."""
    b = self.base
    self._header()
    self._tables(b)
    decl = self._group_symbols(globals_) + ['const size_t numElements = (size_t)ga.num_elements;',
                                            'const unsigned* const flags = ga.flags;', f'const unsigned te = {self.TE}u;']

    def function(name, params, body):
      self.w(f'__device__ __forceinline__ void group{gid}_{name}(const tfb_group_args& ga, {params}) {{')
      self.ind += 1
      for d in decl:
        self.w(d)
      body()
      self.ind -= 1
      self.w('}')

    def tile():
      which = f'which * {self.buf}u' if self.buffers == 2 else '0u'
      self.w(f'const float* const cur = sA + {self.a_total} + {which};')
      self.w('tfb_cp::wait_all();')
      self.w('__syncthreads();  // this tile has landed, and nobody reads the other buffer any more')
      def fetch():
        self.w('if (next_tile != ~(size_t)0)')
        self._fetch('next_tile', f'(sA + {self.a_total}' + (f' + (which ^ 1u) * {self.buf}u)' if self.buffers == 2 else ')'))
        self.w('tfb_cp::commit();')
      if self.buffers == 2:
        fetch()
      self._mine()
      self.w('const size_t e = tile * te + ei;')
      self.open('if (ei < te && e < numElements && (flags == nullptr || flags[e] != 0u))')
      self._compute(b)
      self.close()
      if self.buffers == 1:
        self.w('__syncthreads();')
        fetch()
    function('stage_a', 'float* sA', lambda: self._stage_a(b))
    function('prefetch', 'size_t tile, float* sA, unsigned which',
             lambda: self._fetch('tile', f'(sA + {self.a_total}' + (f' + which * {self.buf}u)' if self.buffers == 2 else ')')))
    function('tile', 'size_t tile, float* sA, size_t next_tile, unsigned which', tile)
    return '\n'.join(self.lines)

  def _header(self):
    self.w(CP_HELPERS)
    self.w(RB_HELPERS)
    self.w(f'// generated by tensorforge_b200 (strategy: colprog, row blocks of {self.RM}, threads={self.BT}, tile={self.TE} elements)')
    self.w('// meta data:')
    for o in self.chain.operands:
      self.w(f'// {o.tensor.gen_descr()}')
    for st in self.chain.stages:
      self.w(f'// {st.descr}')

  def emit(self, globals_):
    b, BT = self.base, self.BT
    kname = f'kernel_{b}'
    self._header()
    self._tables(b)
    self.w(f'__global__ void __launch_bounds__({BT}) {kname}({", ".join(self.params(globals_))}, unsigned te) {{')
    self.ind += 1
    self.w('extern __shared__ __align__(16) unsigned char tfb_smem_raw[];')
    self.w('float* const sA = reinterpret_cast<float*>(tfb_smem_raw);')
    self.w(f'float* cur = sA + {self.a_total};')
    if self.buffers == 2:
      self.w(f'float* next = cur + {self.buf};')
    self._mine()
    self.w('const size_t numTiles = (numElements + te - 1u) / te;')
    self.w('if (blockIdx.x < numTiles)')
    self._fetch('(size_t)blockIdx.x', 'cur')
    self.w('tfb_cp::commit();')
    self._stage_a(b)
    self.open('for (size_t tile = blockIdx.x; tile < numTiles; tile += gridDim.x)')
    self.w('tfb_cp::wait_all();')
    self.w('__syncthreads();  // this tile has landed, and nobody reads the other buffer any more')
    def fetch(buf):
      self.w('if (tile + gridDim.x < numTiles)')
      self._fetch('tile + gridDim.x', buf)
      self.w('tfb_cp::commit();')
    if self.buffers == 2:
      fetch('next')
    self.w('const size_t e = tile * te + ei;')
    self.open('if (ei < te && e < numElements && (flags == nullptr || flags[e] != 0u))')
    self._compute(b)
    self.close()
    if self.buffers == 2:
      self.w('float* const swap = cur;')
      self.w('cur = next;')
      self.w('next = swap;')
    else:
      self.w('__syncthreads();')
      fetch('cur')
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
           '  // a batch that does not fill one wave of full tiles is spread over all of its CTAs',
           '  const size_t spread = (numElements + cap - 1) / cap;',
           f'  const unsigned te = (unsigned)(spread < {self.TE} ? spread : {self.TE});',
           '  const size_t tiles = (numElements + te - 1) / te;',
           f'  {kname}<<<(unsigned)(tiles < (size_t)cap ? tiles : (size_t)cap), {BT}, {self.smem}, stream>>>({", ".join(args)}, te);',
           '  CHECK_ERR;']
    launch = {'kernel': kname, 'block': BT, 'elements_per_block': self.TE, 'smem': self.smem, 'args': args,
              'pre': '\n'.join(pre), 'launched': True}
    return '\n'.join(self.lines), launch, ''


def emit_rowblock(chain, plan, context, base_name, globals_):
  return _RowBlock(chain, match_left_chain(chain), plan, context, base_name).emit(globals_)
