"""Row-tiled column programs (CUDA cores, FP32) for shared-left GEMM chains.

Same chains, tiles and U phase as the unrolled column program (codegen/colprog.py), with
another K stage: instead of one straight-line FMA per nonzero of A_t, every thread owns an
RM x RC block of the tile's output and loops over l,

    acc[i, c] += A_t[i, l] * U_t[l, c]        (RM rows i, RC flat columns c)

with A_t held densely in shared memory (zeros outside its pattern) and packed FP32 FMAs
(two rows per instruction). Per l a thread loads RM + RC values for RM * RC products.

Why dense pays for sparse A: the unrolled program runs 9,533 FMAs of straight-line code per
column for 84 basis functions. Beyond about 100 KB of code a warp gets an instruction every 8
cycles, however many warps share the pass, because the code no longer stays in the
instruction cache. The loop issues 2.2 times the products (A at 45 %) from a body that does
stay. Measured on B200: 84 x 27 chain, three terms, 20,000 elements 948 -> 644 us; the packed
FMAs take about 60 % of that at the rate they reach alone (0.78 of nominal), the U phase,
which nothing overlaps with one CTA per SM, about a fifth.

Zeros and non-finite values: the unrolled program never multiplies an entry outside A_t's
pattern. 0 * u adds nothing for finite u; for an infinite or NaN u it would. The U phase
therefore notes whether a value of U_t is not finite, and a tile that has one runs its K
stage through the pattern's bits instead. Results are the same bits as the unrolled
program's either way: the sum over l runs in the same order with one fused multiply-add
per product.

Row blocks (codegen/rowblock.py) need neither U phase nor write-back and are faster where
they apply (84 x 27: 526 us); this form is for more than 28 columns and for terms with
different per-element operands (84 x 32, 20,000 elements: 776 us against 1,574 unrolled and
1,558 tiled; 56 x 32: 385 against 504 and 624).
"""
from ..plan.chains import match_left_chain
from .colprog import _ColProg, _pad, resident_grid, CP_HELPERS

CT_HELPERS = r'''
#ifndef TFB_COLTILE_HELPERS
#define TFB_COLTILE_HELPERS
namespace tfb_ct {
// CNT (1..4) steps of the K stage from row `a` (this thread's first quad) of A and the
// 16-byte pieces u of RC columns of U: quads of rows lie QS values apart, steps MP apart.
template <int RM, int RC, int MP, int QS, int CNT>
__device__ __forceinline__ void steps(float2 (&acc)[RC][RM / 2], const float* a, const float4 (&u)[RC]) {
#pragma unroll
  for (int k = 0; k < CNT; ++k) {
    float2 av[RM / 2];
#pragma unroll
    for (int s = 0; s < RM / 4; ++s) {
      const float4 x = *reinterpret_cast<const float4*>(a + k * MP + s * QS);
      av[2 * s] = make_float2(x.x, x.y);
      av[2 * s + 1] = make_float2(x.z, x.w);
    }
#pragma unroll
    for (int j = 0; j < RC; ++j) {
      const float uk = k == 0 ? u[j].x : k == 1 ? u[j].y : k == 2 ? u[j].z : u[j].w;
      const float2 uu = make_float2(uk, uk);
#pragma unroll
      for (int i = 0; i < RM / 2; ++i) acc[j][i] = __ffma2_rn(av[i], uu, acc[j][i]);
    }
  }
}
// The K stage of one term: K steps over the columns at u + uo[j].
template <int RM, int RC, int MP, int QS, int K>
__device__ __forceinline__ void k_stage(float2 (&acc)[RC][RM / 2], const float* a, const float* u, const int (&uo)[RC]) {
  float4 x[RC];
#pragma unroll 1
  for (int l = 0; l < K / 4 * 4; l += 4) {
#pragma unroll
    for (int j = 0; j < RC; ++j) x[j] = *reinterpret_cast<const float4*>(u + uo[j] + l);
    steps<RM, RC, MP, QS, 4>(acc, a + l * MP, x);
  }
  if (K % 4 != 0) {
#pragma unroll
    for (int j = 0; j < RC; ++j) x[j] = *reinterpret_cast<const float4*>(u + uo[j] + K / 4 * 4);
    steps<RM, RC, MP, QS, (K % 4 != 0 ? K % 4 : 1)>(acc, a + K / 4 * 4 * MP, x);
  }
}
// The same through A's pattern (W words of row bits per step; this thread's first row: row0).
template <int RM, int RC, int MP, int QS, int W>
__device__ __forceinline__ void k_stage_pattern(float2 (&acc)[RC][RM / 2], const float* a, const float* u, const int (&uo)[RC],
                                             const unsigned* bits, int row0, int K) {
#pragma unroll 1
  for (int l = 0; l < K; ++l) {
#pragma unroll
    for (int s = 0; s < RM / 4; ++s) {
      const int row = row0 + s * QS;
      const unsigned m = row < 32 * W ? bits[l * W + (row >> 5)] >> (row & 31) : 0u;
      const float* x = a + l * MP + s * QS;
#pragma unroll
      for (int j = 0; j < RC; ++j) {
        const float uk = u[uo[j] + l];
        if (m & 1u) acc[j][2 * s].x = fmaf(x[0], uk, acc[j][2 * s].x);
        if (m & 2u) acc[j][2 * s].y = fmaf(x[1], uk, acc[j][2 * s].y);
        if (m & 4u) acc[j][2 * s + 1].x = fmaf(x[2], uk, acc[j][2 * s + 1].x);
        if (m & 8u) acc[j][2 * s + 1].y = fmaf(x[3], uk, acc[j][2 * s + 1].y);
      }
    }
  }
}
}  // namespace tfb_ct
#endif
'''

SMEM_PER_CTA = 227 * 1024
SMEM_PER_SM = 228 * 1024


def _odd_quads(k):
  """Pitch of k values: whole 16-byte units, an odd number of them (columns that neighbouring
  threads read start on different banks)."""
  q = -(-k // 4)
  return 4 * (q if q % 2 else q + 1)


def smem_values(shape, rm, te):
  """(work, stage, A) values of shared memory of one CTA."""
  mp = -(-shape.M // rm) * rm
  a = sum(t.K * mp for t in shape.terms)
  tc = te * shape.N
  pitch = _odd_quads(max(t.K for t in shape.terms))
  ops = {id(o): o for t in shape.terms for o in (t.B, t.R) if o is not None and o.kind == 'batched'}
  stage = sum(te * _pad(o.storage_size() if o.sparse else o.element_volume(), 4) for o in ops.values())
  return _pad(tc * max(pitch, shape.M), 4), stage, a


def choose(shape, threads):
  """(threads, RM, RC, TE) with the most useful work per issued FMA and resident warp.

  Counts the block's padding rows and columns, the loads that a block smaller than 12 x 5 does
  not amortise, and warps missing from the eight an SM needs. Measured on the 84 x 27 chain
  (39,900 elements, 256 threads): 12 x 5 blocks 1,244 us, 12 x 4 1,284, 12 x 6 (a seventh
  element, a column block three quarters full) 1,376, 8 x 8 1,410, 28 x 2 1,777."""
  M, N = shape.M, shape.N
  best = None
  for bt in threads:
    for rm in (8, 12):
      rg = -(-M // rm)
      cg = bt // rg
      for rc in range(1, 10):
        te = min(cg * rc // N, 64)
        while te > 1 and 4 * sum(smem_values(shape, rm, te)) > SMEM_PER_CTA:
          te -= 1
        smem = 4 * sum(smem_values(shape, rm, te))
        if te < 1 or smem > SMEM_PER_CTA:
          continue
        warps = min(SMEM_PER_SM // (smem + 1024), 65536 // (bt * min(255, rm * rc + 4 * rc + rm + 60))) * bt / 32
        score = te * N / (cg * rc) * M / (rg * rm) * min(1.0, rm * rc / 60) * min(1.0, warps / 8)
        if best is None or score > best[0] * 1.001:
          best = (score, bt, rm, rc, te)
  return best[1:] if best else None


def coltile_params(shape, variant):
  """(plan parameters, shared-memory bytes) of the row-tiled form, or None. A variant may name
  the threads, or the threads and the whole tile (rm, rc, te)."""
  threads = (variant['threads'],) if 'threads' in variant else (256, 128)
  if all(k in variant for k in ('rm', 'rc', 'te')):
    cfg = (threads[0], variant['rm'], variant['rc'], variant['te'])
    rows = max(1, -(-shape.M // max(1, cfg[1])))
    if cfg[1] < 4 or cfg[1] % 4 or not 1 <= cfg[3] * shape.N <= cfg[0] // rows * cfg[2]:
      return None   # quads of rows, and every column of the tile with a thread
  else:
    cfg = choose(shape, threads)
  if cfg is None:
    return None
  smem = 4 * sum(smem_values(shape, cfg[1], cfg[3]))
  if smem > SMEM_PER_CTA:
    return None
  return dict(zip(('threads', 'rm', 'rc', 'te'), cfg), prefetch=1, a_source='dense'), smem


class _ColTile(_ColProg):
  skip_masked = True

  def __init__(self, chain, shape, plan, ctx, base):
    super().__init__(chain, shape, plan, ctx, base)
    self.RM, self.RC, self.TE = (plan.params[k] for k in ('rm', 'rc', 'te'))
    self.prefetch = True
    self.const_terms = 0
    self.term_const = [False] * len(shape.terms)
    self.RS = self.CPT = 1
    self.RG = -(-shape.M // self.RM)
    self.CG = self.BT // self.RG
    self.MP = self.RG * self.RM
    self.TC = self.TE * shape.N
    self.TCT = self.TC
    self.pitch = _odd_quads(self.kmax)
    self.W = -(-shape.M // 32)

  # ------------------------------------------------------------------ layout and tables
  def _layout(self):
    s = self.s
    self.a_base, off = [], 0
    for t in s.terms:
      self.a_base.append(off)
      off += t.K * self.MP
    self.a_const_total, self.a_smem_total, self.a_total = 0, off, off
    work, stage, _ = smem_values(s, self.RM, self.TE)
    self.ubuf_vals = self.work_vals = work
    self.stage_vals, self.stage_off = stage, {}
    self.r_off = {}
    at = work
    for t in s.terms:
      for op in (t.B, t.R):
        if op is not None and op.kind == 'batched' and op.name not in self.stage_off:
          self.stage_off[op.name] = at
          at += self.TE * _pad(op.storage_size() if op.sparse else op.element_volume(), 4)
    self.a_off = work + stage
    self.smem = (work + stage + off) * 4

  def _tables(self, b):
    """Where each stored value of a sparse A_t goes, and the pattern's bits per step."""
    for ti, t in enumerate(self.s.terms):
      if not t.A.sparse:
        continue
      look = t.A.sparse_lookup()
      dst = [0] * t.A.storage_size()
      bits = [0] * (t.K * self.W)
      for (i, l), pos in look.items():
        if i < self.s.M and l < t.K:
          dst[pos] = l * self.MP + i
          bits[l * self.W + (i >> 5)] |= 1 << (i & 31)
      self.w(f'static __device__ const unsigned short aoff_{b}_{ti}[{len(dst)}] = {{{", ".join(map(str, dst))}}};')
      self.w(f'static __device__ const unsigned abits_{b}_{ti}[{len(bits)}] = {{{", ".join(f"{x}u" for x in bits)}}};')

  def _stage_a(self, b):
    """Bring A into shared memory, dense, rows padded to whole thread tiles."""
    s, BT = self.s, self.BT
    self.w(f'for (int q = threadIdx.x; q < {self.a_total // 4}; q += {BT}) reinterpret_cast<float4*>(sA)[q] = make_float4(0.f, 0.f, 0.f, 0.f);')
    self.w('__syncthreads();')
    for ti, t in enumerate(s.terms):
      self.w('#pragma unroll 8')
      if t.A.sparse:
        self.w(f'for (int q = threadIdx.x; q < {t.A.storage_size()}; q += {BT}) '
               f'sA[{self.a_base[ti]} + aoff_{b}_{ti}[q]] = __ldg({t.A.name} + q);')
      elif self.MP == s.M:
        self.w(f'for (int q = threadIdx.x; q < {t.K * s.M}; q += {BT}) sA[{self.a_base[ti]} + q] = __ldg({t.A.name} + q);')
      else:
        self.w(f'for (int q = threadIdx.x; q < {t.K * s.M}; q += {BT}) '
               f'sA[{self.a_base[ti]} + q / {s.M} * {self.MP} + q % {s.M}] = __ldg({t.A.name} + q);')

  def _header(self):
    self.w(CP_HELPERS)
    self.w(CT_HELPERS)
    self.w(f'// generated by tensorforge_b200 (strategy: colprog, threads={self.BT}, {self.RM} x {self.RC} outputs per '
           f'thread, tile={self.TE} elements, dense A from shared memory)')
    self.w('// meta data:')
    for o in self.chain.operands:
      self.w(f'// {o.tensor.gen_descr()}')
    for st in self.chain.stages:
      self.w(f'// {st.descr}')

  # ------------------------------------------------------------------ tile
  def _tile_body(self, b):
    s, BT = self.s, self.BT
    RM, RC, MP, QS = self.RM, self.RC, self.MP, 4 * self.RG
    # neighbouring threads read the same rows of A and every other one the same column of U:
    # a 16-byte shared load takes the SM two cycles when lanes i and i ^ 1 (or i ^ 2) share
    # their address for every i, else four
    if self.CG % 2 == 0:
      self.w(f'const unsigned rg = (threadIdx.x >> 1) % {self.RG}u, cg = threadIdx.x / {2 * self.RG}u * 2u + (threadIdx.x & 1u);')
    else:
      self.w(f'const unsigned rg = threadIdx.x % {self.RG}u, cg = threadIdx.x / {self.RG}u;')
    self.w(f'const bool working = cg < {self.CG}u;')
    self.w(f'const size_t e0 = tile * {self.TE}u;')
    self.w(f'int uo[{RC}];')
    self.w('#pragma unroll')
    self.w(f'for (int j = 0; j < {RC}; ++j) uo[j] = min((int)cg + j * {self.CG}, {self.TC - 1}) * {self.pitch};')
    self.w(f'float2 acc[{RC}][{RM // 2}];')
    self.w('#pragma unroll')
    self.w(f'for (int j = 0; j < {RC}; ++j)')
    self.w('#pragma unroll')
    self.w(f'  for (int i = 0; i < {RM // 2}; ++i) acc[j][i] = make_float2(0.f, 0.f);')
    targs = f'{RM}, {RC}, {MP}, {QS}'
    for ti, t in enumerate(s.terms):
      self.w(f'// term {ti}: A={t.A.name} ({s.M}x{t.K}, {"sparse" if t.A.sparse else "dense"}), '
             f'B={t.B.name}, R={t.R.name if t.R is not None else "-"}')
      last = ti == len(s.terms) - 1
      self.w('int odd = 0;  // a value of U that is not finite')
      self._u_phase(ti, t)
      if t.A.sparse:
        self.w('odd = __syncthreads_or(odd);')
      else:
        self.w('__syncthreads();')
      if last:
        self.w('// the stage is free: fetch the next tile while this K stage runs')
        nxt = getattr(self, 'next_tile', None)
        self.open('if (tile + gridDim.x < numTiles)' if nxt is None else f'if ({nxt} != ~(size_t)0)')
        self._prefetch('tile + gridDim.x' if nxt is None else nxt)
        self.close()
        self.w('tfb_cp::commit();')
      self.open('if (working)')
      call = (f'tfb_ct::k_stage<{targs}, {t.K}>(acc, sA + {self.a_base[ti]} + rg * 4u, ubuf, uo);')
      if t.A.sparse:
        self.w(f'if (odd) tfb_ct::k_stage_pattern<{targs}, {self.W}>(acc, sA + {self.a_base[ti]} + rg * 4u, ubuf, uo, '
               f'abits_{b}_{ti}, rg * 4, {t.K});')
        self.w('else ' + call)
      else:
        self.w(call)
      self.close()
      self.w('__syncthreads();')
      if not last:
        self.open('')   # a scope per term
    for _ in s.terms[1:]:
      self.close()
    self._write()

  def _u_phase(self, ti, t):
    """U_t = B R_t into shared memory; `odd`: whether a value of it is not finite (sparse A_t).
    Elements whose operands are not fetched are left out."""
    # row pairs halve R's loads and need about 1.7 times a single row's time
    two = self.row_pairs(t, -(-self.TE * t.K // self.BT), 1.7)
    self.w(f'{"float2" if two else "float"} sum0[3] = {{}};')

    def note(j):   # three sums of 0 * u, NaN once a value is not finite
      if t.A.sparse:
        self.w(f'sum0[{j % 3}] = ' + (f'__ffma2_rn(u{j}, make_float2(0.f, 0.f), sum0[{j % 3}]);' if two
                                      else f'fmaf(u{j}, 0.f, sum0[{j % 3}]);'))
    (self._u_row_pairs if two else self._u_single)(t, note)
    if t.A.sparse:
      total = ' + '.join(f'sum0[{i}]{c}' for i in range(3) for c in (('.x', '.y') if two else ('',)))
      self.w(f'odd = {total} != 0.f;')

  def _u_single(self, t, note):
    """Odd K: a thread computes one row of an element."""
    s, BT, P, K = self.s, self.BT, t.P, t.K
    self.w('#pragma unroll 2')
    self.open(f'for (unsigned q = threadIdx.x; q < {self.TE * K}u; q += {BT}u)')
    self.w(f'const unsigned ei = q / {K}u, l = q - ei * {K}u;')
    self.open(f'if (e0 + ei < numElements{self._present(t)})')
    self.w(f'float* const urow = ubuf + ei * {s.N * self.pitch}u + l;')
    self.w(f'const float* const bq = ubuf + {self.stage_off[t.B.name]} + ei * {_pad(t.B.element_volume(), 4)}u + l;')
    for m in range(P):
      self.w(f'const float q{m} = bq[{m * K}];')
    if t.R is not None:
      rv = self._r_value(t, 'ei')
      look = t.R.sparse_lookup() if t.R.sparse else None
    for j in range(s.N):
      expr = f'q{j}'
      if t.R is not None:
        expr = '0.f'
        for m in range(P):
          pos = look.get((m, j)) if look is not None else j * P + m
          if pos is not None:
            expr = f'fmaf(q{m}, {rv(pos)}, {expr})'
      self.w(f'const float u{j} = {expr};')
      self.w(f'urow[{j * self.pitch}] = u{j};')
      note(j)
    self.close()
    self.close()

  def _write(self):
    """The tile's output through shared memory, then to global memory with 16-byte stores."""
    s, BT, RM, RC, M, N = self.s, self.BT, self.RM, self.RC, self.s.M, self.s.N
    self.w('// stage the tile, then write it back')
    self.open('if (working)')
    self.w('#pragma unroll')
    self.open(f'for (int j = 0; j < {RC}; ++j)')
    self.w(f'const unsigned c = cg + j * {self.CG}u;')
    self.open(f'if (c < {self.TC}u)')
    self.w('#pragma unroll')
    self.open(f'for (int s = 0; s < {RM // 4}; ++s)')
    self.w(f'const unsigned row = (s * {self.RG}u + rg) * 4u;')
    if M % 4 == 0:
      guard = f'if (row < {M}u) ' if self.MP != M else ''
      self.w(f'{guard}*reinterpret_cast<float4*>(ubuf + c * {M}u + row) = make_float4(acc[j][2 * s].x, acc[j][2 * s].y, '
             'acc[j][2 * s + 1].x, acc[j][2 * s + 1].y);')
    else:
      for v, x in enumerate(('acc[j][2 * s].x', 'acc[j][2 * s].y', 'acc[j][2 * s + 1].x', 'acc[j][2 * s + 1].y')):
        self.w(f'if (row + {v}u < {M}u) ubuf[c * {M}u + row + {v}u] = {x};')
    for _ in range(4):
      self.close()
    self._write_back('ubuf', s.accumulate)

  # ------------------------------------------------------------------ kernels
  def kernel(self, globals_, kname):
    b = kname
    self._layout()
    self._header()
    self._tables(b)
    self.w(f'__global__ void __launch_bounds__({self.BT}) {kname}({", ".join(self.params(globals_))}) {{')
    self.ind += 1
    self.w('extern __shared__ __align__(16) unsigned char tfb_smem_raw[];')
    self.w('float* const ubuf = reinterpret_cast<float*>(tfb_smem_raw);')
    self.w(f'float* const sA = ubuf + {self.a_off};')
    self.w(f'const size_t numTiles = (numElements + {self.TE - 1}u) / {self.TE}u;')
    self.open('if (blockIdx.x < numTiles)')
    self._prefetch('(size_t)blockIdx.x')
    self.close()
    self.w('tfb_cp::commit();')
    self._stage_a(b)
    self.open('for (size_t tile = blockIdx.x; tile < numTiles; tile += gridDim.x)')
    self.w('tfb_cp::wait_all();')
    self.w('__syncthreads();')
    self._tile_body(b)
    self.close()
    self.w('tfb_cp::wait_all();')
    self.ind -= 1
    self.w('}')
    return '\n'.join(self.lines)

  def emit_group_functions(self, globals_, gid):
    """Device functions of one group of a grouped launch (see _ColProg.emit_group_functions)."""
    self.next_tile = 'next_tile'
    self._layout()
    self._header()
    b = f'{self.base}'
    self._tables(b)
    decl = self._group_symbols(globals_) + ['const size_t numElements = (size_t)ga.num_elements;', 'const unsigned* const flags = ga.flags;']

    def function(name, params, body):
      self.w(f'__device__ __forceinline__ void group{gid}_{name}(const tfb_group_args& ga, {params}) {{')
      self.ind += 1
      for d in decl:
        self.w(d)
      body()
      self.ind -= 1
      self.w('}')

    def stage():
      self.w(f'float* const sA = smem + {self.a_off};')
      self._stage_a(b)

    def tile():
      self.w(f'const float* const sA = ubuf + {self.a_off};')
      self.w('tfb_cp::wait_all();  // this tile\'s stage has landed')
      self.w('__syncthreads();')
      self._tile_body(b)
    function('stage_a', 'float* smem', stage)
    function('prefetch', 'size_t tile, float* ubuf, unsigned which', lambda: self._prefetch('tile'))
    function('tile', 'size_t tile, float* ubuf, size_t next_tile, unsigned which', tile)
    return '\n'.join(self.lines)


def emit_coltile(chain, plan, context, base_name, globals_):
  k = _ColTile(chain, match_left_chain(chain), plan, context, base_name)
  kname = f'kernel_{base_name}'
  text = k.kernel(globals_, kname)
  args = []
  for t, _ in globals_:
    args.append(t.name)
    if t.addressing.name not in ('NONE', 'SCALAR'):
      args.append(f'{t.name}_extraOffset')
  args += ['numElements', 'flags']
  plan.smem_bytes = k.smem
  launch = {'kernel': kname, 'block': k.BT, 'elements_per_block': k.TE, 'smem': k.smem, 'args': args,
            'pre': resident_grid(kname, k.BT, k.smem)}
  return text, launch, ''
