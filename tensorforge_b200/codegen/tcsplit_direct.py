"""tcgen05 split-precision generator for a single product per element, out_e (+)= A * B_e.

Form U of codegen/tcsplit.py without its U pass: with no R factor the flat columns (e, j) of
B_e, which lie one after the other in an element, are the tensor memory rows of the MMA's A
operand as they are. Per tile of TE = floor(128 / N) elements:

  * a loader warp copies the elements into a ring of shared-memory stages, one bulk copy per
    tile (strided) or per element (pointer arrays), up to four tiles ahead;
  * two teams of four producer warps take tiles in turn: a lane reads its column of K values,
    splits each into hi + lo and stores both to its team's tensor memory slot;
  * one thread issues the MMAs, hi x [hi | lo] as one of twice the width and lo x hi, into the
    team's main and correction accumulators;
  * two teams of four epilogue warps add main and correction, stage the tile's outputs in
    shared memory and send every element off with one bulk store.

Everything is double buffered (two A slots, two accumulator pairs, two output buffers), so
the four steps of different tiles overlap; teams meet only at mbarriers.

What bounds it: HBM (a 56x56x9 product moves 4,032 bytes and two pointers). Operand form B
(codegen/tcsplit_b.py), which this replaces for K a multiple of 4, put the per-element operand
into shared memory in the MMA's tiled layout, one value at a time, with all warps changing
roles together at barriers. Measured on B200, 300,000 pointer-array 56x56x9 products:
536 -> 260 us (4.7 TB/s; strided 223 us), error against 64 bits 4.7e-7 -> 1.8e-7 (correction products apart).

Waits are bounded as in codegen/tcsplit.py: a wait that runs out records an error code (read
with tfb_kernel_error_<name>), and the CTA ends after its copies in flight and its tensor memory.
"""
from ..plan import Plan
from .. import plan as _plan
from ..plan.chains import match_left_chain
from .tcsplit import HELPERS, _TC, _pad

TEAMS = 2


def layout(shape):
  """Shared-memory offsets (bytes) and tile sizes, or None where the form does not apply."""
  t = shape.terms[0]
  if len(shape.terms) != 1 or t.R is not None or t.K % 4 or shape.M % 4 or shape.N > 128 or shape.M > 128:
    return None
  kp, n_mma = _pad(t.K, 8), _pad(shape.M, 16)
  if TEAMS * (2 * kp + 2 * n_mma) > 512:
    return None
  te = 128 // shape.N
  stage = _pad(te * shape.N * t.K * 4, 128)
  ost = _pad(te * shape.N * shape.M * 4, 128)
  b_bytes = 2 * n_mma * kp * 4
  fixed = _pad(b_bytes, 128) + TEAMS * ost + 256
  stages = min(4, (_plan.SMEM_LIMIT - fixed) // stage)
  if stages < 2:
    return None
  off_stage = _pad(b_bytes, 128)
  off_ost = off_stage + stages * stage
  off_bar = off_ost + TEAMS * ost
  return dict(te=te, kp=kp, n_mma=n_mma, stage=stage, stages=stages, ost=ost, off_stage=off_stage,
              off_ost=off_ost, off_bar=off_bar, total=off_bar + 256)


def direct_plan(shape):
  lay = layout(shape)
  if lay is None:
    return None
  return Plan('tcsplit', {'precision': 'tf32x3', 'form': 'direct', 'te': lay['te'], 'stages': lay['stages']},
              max(lay['total'], 120 * 1024), 32 * (8 * TEAMS + 2),
              note=f'direct: M={shape.M} N={shape.N} K={shape.terms[0].K} tile={lay["te"]}')


class _Direct(_TC):
  def __init__(self, chain, shape, plan_, ctx, base):
    self.chain, self.s, self.plan, self.base = chain, shape, plan_, base
    self.T = ctx.fp_as_str()
    self.lay = layout(shape)
    self.lines, self.ind = [], 0

  def wait(self, bar, parity, code):
    """Wait of a whole warp: it leaves its loop together if a lane's wait runs out."""
    self.w(f'if (!__all_sync(0xffffffffu, tfb_tc::mbar_wait_h(&bars[{bar}], {parity}, {self.WAIT_NS}ull))) '
           f'{{ atomicMax(&tfb_err_{self.base}, {code}u); break; }}')

  def emit(self, globals_):
    s, L, b = self.s, self.lay, self.base
    t = s.terms[0]
    K, M, N, te, kp, n_mma, S = t.K, s.M, s.N, L['te'], L['kp'], L['n_mma'], L['stages']
    kname = f'kernel_{b}'
    nthreads = self.plan.threads
    look = t.A.sparse_lookup() if t.A.sparse else None
    tbl = []
    for n in range(n_mma):
      for k in range(kp):
        inside = n < M and k < K
        tbl.append((k * M + n if look is None else look.get((n, k), -1)) if inside else -1)
    self.w(HELPERS)
    self.w(f'// generated by tensorforge_b200 (strategy: tcsplit, tf32x3 direct, tile={te} elements, smem={L["total"]} B)')
    self.w('// meta data:')
    for o in self.chain.operands:
      self.w(f'// {o.tensor.gen_descr()}')
    for st in self.chain.stages:
      self.w(f'// {st.descr}')
    self.w(f'static __device__ const short bgather_{b}[{len(tbl)}] = {{{", ".join(str(x) for x in tbl)}}};')
    self.w(f'__device__ unsigned tfb_err_{b} = 0u;')
    self.w(f'extern "C" int tfb_kernel_error_{b}(void* stream) {{')
    self.w('  unsigned v = 0, z = 0;')
    self.w('  cudaStream_t st = static_cast<cudaStream_t>(stream);')
    self.w(f'  cudaMemcpyFromSymbolAsync(&v, tfb_err_{b}, sizeof(unsigned), 0, cudaMemcpyDeviceToHost, st);')
    self.w(f'  cudaMemcpyToSymbolAsync(tfb_err_{b}, &z, sizeof(unsigned), 0, cudaMemcpyHostToDevice, st);')
    self.w('  cudaStreamSynchronize(st);')
    self.w('  return (int)v;')
    self.w('}')
    # barriers: stage full / empty, A slot full / empty, accumulators full / empty
    SF, SE = 0, S
    AF, AE = 2 * S, 2 * S + TEAMS
    DF, DE = 2 * S + 2 * TEAMS, 2 * S + 3 * TEAMS
    nbars = 2 * S + 4 * TEAMS
    self.bars = dict(SF=SF, SE=SE, AF=AF, AE=AE, DF=DF, DE=DE)
    self.w(f'__global__ void __launch_bounds__({nthreads}, 1) {kname}({", ".join(self.params(globals_))}) {{')
    self.ind += 1
    self.w('extern __shared__ __align__(1024) unsigned char tfb_smem_raw[];')
    self.w(f'uint64_t* const bars = reinterpret_cast<uint64_t*>(tfb_smem_raw + {L["off_bar"]});')
    self.w(f'unsigned* const tmem_slot = reinterpret_cast<unsigned*>(bars + {nbars});')
    self.w('const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;')
    self.w(f'const size_t numTiles = (numElements + {te - 1}u) / {te}u;')
    # A^T, split into hi and lo, in the canonical no-swizzle K-major layout
    sbo = (kp // 4) * 128
    lo_off = n_mma * kp * 4
    self.open(f'for (int q = threadIdx.x; q < {n_mma * kp}; q += {nthreads})')
    self.w(f'const int n = q / {kp}, k = q - n * {kp};')
    self.w(f'const int src = bgather_{b}[q];')
    self.w(f'const float v = src >= 0 ? {t.A.name}[src] : 0.0f;')
    self.w(f'const unsigned boff = (n >> 3) * {sbo}u + (k / 4) * 128u + (n & 7) * 16u + (k % 4) * 4u;')
    self.w('unsigned hb, lb;')
    self.w('tfb_tc::tf32_split(v, hb, lb);')
    self.w('*reinterpret_cast<unsigned*>(tfb_smem_raw + boff) = hb;')
    self.w(f'*reinterpret_cast<unsigned*>(tfb_smem_raw + {lo_off} + boff) = lb;')
    self.close()
    self.open('if (threadIdx.x == 0)')
    self.w(f'for (int i = 0; i < {S}; ++i) {{ tfb_tc::mbar_init(&bars[{SF} + i], 1u); tfb_tc::mbar_init(&bars[{SE} + i], 4u); }}')
    self.w(f'for (int i = 0; i < {TEAMS}; ++i) {{')
    self.w(f'  tfb_tc::mbar_init(&bars[{AF} + i], 4u); tfb_tc::mbar_init(&bars[{AE} + i], 1u);')
    self.w(f'  tfb_tc::mbar_init(&bars[{DF} + i], 1u); tfb_tc::mbar_init(&bars[{DE} + i], 4u);')
    self.w('}')
    self.w('asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");')
    self.close()
    self.w('if (warp == 0) tfb_tc::tmem_alloc(tmem_slot, 512u);')
    self.w('tfb_tc::fence_proxy_async();')
    self.w('tfb_tc::fence_before();')
    self.w('__syncthreads();')
    self.w('tfb_tc::fence_after();')
    self.w('const unsigned tmem = *tmem_slot;')
    self._mma(sbo, lo_off)
    self._loader()
    self._producers()
    self._epilogue_teams()
    self.w('tfb_tc::fence_before();')
    self.w('__syncthreads();')
    self.open('if (warp == 0)')
    self.w('tfb_tc::fence_after();')
    self.w('tfb_tc::tmem_dealloc(tmem, 512u);')
    self.close()
    self.ind -= 1
    self.w('}')
    args = []
    for tt, _ in globals_:
      args.append(tt.name)
      if tt.addressing.name not in ('NONE', 'SCALAR'):
        args.append(f'{tt.name}_extraOffset')
    args += ['numElements', 'flags']
    pre = ('  int sms = 0;\n'
           '  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);\n'
           '  if (sms > 0 && grid.x > (unsigned)sms) grid.x = (unsigned)sms;')
    launch = {'kernel': kname, 'block': nthreads, 'elements_per_block': te, 'smem': self.plan.smem_bytes, 'args': args,
              'pre': pre}
    return '\n'.join(self.lines), launch, ''

  # team k's A slot: 2 kp columns (hi, lo) from k * 2 kp; accumulators behind both slots
  def _slot(self, k):
    return f'{k} * {2 * self.lay["kp"]}u'

  def _acc(self, k):
    return f'{TEAMS * 2 * self.lay["kp"]}u + {k} * {2 * self.lay["n_mma"]}u'

  def _mma(self, sbo, lo_off):
    """One thread: every tile's products, as soon as its A slot is full and its accumulators free."""
    L, B = self.lay, self.bars
    kp, n_mma = L['kp'], L['n_mma']
    idesc = (1 << 4) | (2 << 7) | (2 << 10) | ((n_mma >> 3) << 17) | ((128 >> 4) << 24)
    wide = (idesc & ~(0x3F << 17)) | (((2 * n_mma) >> 3) << 17)
    self.open(f'if (warp == {8 * TEAMS})')
    self.open('if (lane == 0)')
    self.w('unsigned it = 0;')
    self.open('for (size_t tile = blockIdx.x; tile < numTiles; tile += gridDim.x, ++it)')
    self.w(f'const unsigned k = it % {TEAMS}u, ph = it / {TEAMS}u;')
    for bar, parity, code, when in (('DE', '(ph - 1u) & 1u', 13, 'ph > 0u && '), ('AF', 'ph & 1u', 10, '')):
      self.w(f'if ({when}!tfb_tc::mbar_wait(&bars[{B[bar]}u + k], {parity}, {self.WAIT_LIMIT}ull)) '
             f'{{ atomicMax(&tfb_err_{self.base}, {code}u); break; }}')
    self.w('tfb_tc::fence_after();')
    self.w(f'const unsigned d = tmem + {self._acc("k")};')
    self.open(f'for (int ks = 0; ks < {kp // 8}; ++ks)')
    self.w(f'const unsigned hi = tmem + {self._slot("k")} + ks * 8u, lo = hi + {kp}u;')
    self.w(f'const uint64_t bh = tfb_tc::smem_desc(tfb_tc::smem_u32(tfb_smem_raw) + ks * 256u, 128u, {sbo}u);')
    self.w(f'tfb_tc::mma_tf32(d, hi, bh, {wide}u, ks > 0 ? 1u : 0u);     // hi x [hi | lo]')
    self.w(f'tfb_tc::mma_tf32(d + {n_mma}u, lo, bh, {idesc}u, 1u);')
    self.close()
    self.w(f'tfb_tc::mma_commit(&bars[{B["AE"]}u + k]);')
    self.w(f'tfb_tc::mma_commit(&bars[{B["DF"]}u + k]);')
    self.close()
    self.w('// no MMA is left in flight when the tensor memory goes')
    self.open(f'for (unsigned i = it > {TEAMS}u ? it - {TEAMS}u : 0u; i < it; ++i)')
    self.w(f'if (!tfb_tc::mbar_wait(&bars[{B["DF"]}u + i % {TEAMS}u], (i / {TEAMS}u) & 1u, {self.WAIT_LIMIT}ull)) '
           f'atomicMax(&tfb_err_{self.base}, 14u);')
    self.close()
    self.close()
    self.close()

  def _loader(self):
    """One warp: tile it into stage it % S, once the producers have read what it held."""
    s, L, B = self.s, self.lay, self.bars
    op, te, S = s.terms[0].B, L['te'], L['stages']
    vol = op.element_volume()
    self.open(f'else if (warp == {8 * TEAMS + 1})')
    ahead = op.addressing.name == 'PTR_BASED' and te <= 32

    def pointer(tile):
      """The lane's element of a tile: its address, read a tile ahead of its use."""
      return f'({tile}) * {te}u + lane < numElements && lane < {te}u ? {self._elem_ptr(op, f"(({tile}) * {te}u + lane)")} : nullptr'
    self.w('unsigned it = 0;')
    if ahead:
      self.w(f'const float* following = {pointer("(size_t)blockIdx.x")};')
    self.open('for (size_t tile = blockIdx.x; tile < numTiles; tile += gridDim.x, ++it)')
    self.w(f'const unsigned sl = it % {S}u, ph = it / {S}u;')
    if ahead:
      self.w('const float* const src = following;')
      self.w(f'following = {pointer("tile + gridDim.x")};')
    self.open('if (ph > 0u)')
    self.wait(f'{B["SE"]}u + sl', '(ph - 1u) & 1u', 42)
    self.close()
    self.w(f'float* const dst = reinterpret_cast<float*>(tfb_smem_raw + {L["off_stage"]} + sl * {L["stage"]}u);')
    self.w(f'const size_t e0 = tile * {te}u;')
    self.w(f'const unsigned nv = numElements - e0 < {te}u ? (unsigned)(numElements - e0) : {te}u;')
    if op.addressing.name == 'STRIDED':
      self.w(f'const float* const src = {self._elem_ptr(op, "e0")};')
      self.open('if ((reinterpret_cast<uintptr_t>(src) & 15u) == 0u)')
      self.open('if (lane == 0)')
      self.w(f'tfb_tc::mbar_arrive_expect_tx(&bars[{B["SF"]}u + sl], nv * {vol * 4}u);')
      self.w(f'tfb_tc::bulk_load(dst, src, nv * {vol * 4}u, &bars[{B["SF"]}u + sl]);')
      self.close()
      self.close()
      self.open('else')   # in every tile or in none: elements are whole 16-byte units
      self.w(f'for (unsigned q = lane; q < nv * {vol}u; q += 32u) dst[q] = src[q];')
      self.w('__syncwarp();')
      self.w(f'if (lane == 0) tfb_tc::mbar_arrive(&bars[{B["SF"]}u + sl]);')
      self.close()
    else:
      # one bulk copy per element; an element whose address is not a multiple of 16 bytes is
      # copied by its lane before the warp announces the others' bytes. Those stores are made
      # visible first: to the producers by the warp barrier before lane 0's arrival, which
      # releases them, and to a later bulk copy into the same place by the proxy fence
      elements = 'for (unsigned i = lane; i < nv; i += 32u)'
      self.w('unsigned mine = 0;')
      self.open(elements)
      if not ahead:
        self.w(f'const float* const src = {self._elem_ptr(op, "(e0 + i)")};')
      self.w('if ((reinterpret_cast<uintptr_t>(src) & 15u) == 0u) ++mine;')
      self.open('else')
      self.w(f'for (unsigned q = 0; q < {vol}u; ++q) dst[i * {vol}u + q] = src[q];')
      self.w('tfb_tc::fence_proxy_async();')
      self.close()
      self.close()
      self.w('__syncwarp();')
      self.w('const unsigned aligned = __reduce_add_sync(0xffffffffu, mine);')
      self.w(f'if (lane == 0) tfb_tc::mbar_arrive_expect_tx(&bars[{B["SF"]}u + sl], aligned * {vol * 4}u);')
      self.w('__syncwarp();')
      self.open(elements)
      if not ahead:
        self.w(f'const float* const src = {self._elem_ptr(op, "(e0 + i)")};')
      self.w(f'if ((reinterpret_cast<uintptr_t>(src) & 15u) == 0u) tfb_tc::bulk_load(dst + i * {vol}u, src, {vol * 4}u, &bars[{B["SF"]}u + sl]);')
      self.close()
    self.close()
    self.w('// the last copies have to land before the CTA ends, consumed or not')
    self.open(f'for (unsigned i = it > {S}u ? it - {S}u : 0u; i < it; ++i)')
    self.w(f'if (!tfb_tc::mbar_wait_s(&bars[{B["SF"]}u + i % {S}u], (i / {S}u) & 1u, {self.WAIT_NS}ull)) atomicMax(&tfb_err_{self.base}, 41u);')
    self.close()
    self.close()

  def _producers(self):
    """Team k, one warp per quadrant of tensor memory lanes: a lane's column, split, into slot k."""
    s, L, B = self.s, self.lay, self.bars
    K, N, te, kp, S = s.terms[0].K, s.N, L['te'], L['kp'], L['stages']
    self.open(f'else if (warp < {4 * TEAMS})')
    self.w('const unsigned quad = warp & 3u, k = warp >> 2;')
    self.w('const unsigned row = quad * 32u + lane;')
    self.w(f'const unsigned le = row / {N}u;')
    self.w(f'const unsigned slot = tmem + ((quad * 32u) << 16) + {self._slot("k")};')
    self.w('unsigned ph = 0;')
    self.open(f'for (size_t tile = blockIdx.x + (size_t)k * gridDim.x; tile < numTiles; tile += (size_t)gridDim.x * {TEAMS}u, ++ph)')
    self.w(f'const unsigned it = ph * {TEAMS}u + k, sl = it % {S}u;')
    self.w(f'const size_t el = tile * {te}u + le;')
    self.w(f'const bool active = row < {te * N}u && el < numElements && (flags == nullptr || flags[el] != 0u);')
    self.wait(f'{B["SF"]}u + sl', f'(it / {S}u) & 1u', 40)
    self.w(f'const float* const col = reinterpret_cast<const float*>(tfb_smem_raw + {L["off_stage"]} + sl * {L["stage"]}u) + row * {K}u;')
    self.open('if (ph > 0u)')
    self.wait(f'{B["AE"]}u + k', '(ph - 1u) & 1u', 30)
    self.close()
    self.w('tfb_tc::fence_after();')
    self.w('#pragma unroll')
    self.open(f'for (int c0 = 0; c0 < {kp}; c0 += 16)')
    self.w('float u[16];')
    self.w('#pragma unroll')
    self.open('for (int v = 0; v < 4; ++v)')
    self.w('float4 x = make_float4(0.f, 0.f, 0.f, 0.f);')
    self.w(f'if (active && c0 + 4 * v < {K}) x = *reinterpret_cast<const float4*>(col + c0 + 4 * v);')
    self.w('u[4 * v] = x.x; u[4 * v + 1] = x.y; u[4 * v + 2] = x.z; u[4 * v + 3] = x.w;')
    self.close()
    self.w('unsigned hv[16], lv[16];')
    self.w('#pragma unroll')
    self.open('for (int p = 0; p < 8; ++p)')
    self.w('hv[2 * p] = tfb_tc::tf32_rna(u[2 * p]);')
    self.w('hv[2 * p + 1] = tfb_tc::tf32_rna(u[2 * p + 1]);')
    self.w('const float2 lo = __ffma2_rn(make_float2(__uint_as_float(hv[2 * p]), __uint_as_float(hv[2 * p + 1])), '
           'make_float2(-1.0f, -1.0f), make_float2(u[2 * p], u[2 * p + 1]));')
    self.w('lv[2 * p] = __float_as_uint(lo.x);')
    self.w('lv[2 * p + 1] = __float_as_uint(lo.y);')
    self.close()
    self.w(f'if (c0 + 8 < {kp}) {{ tfb_tc::st_x16(slot + c0, hv); tfb_tc::st_x16(slot + {kp}u + c0, lv); }}')
    self.w(f'else {{ tfb_tc::st_x8(slot + c0, hv); tfb_tc::st_x8(slot + {kp}u + c0, lv); }}')
    self.close()
    self.w('__syncwarp();')
    self.w(f'if (lane == 0) tfb_tc::mbar_arrive(&bars[{B["SE"]}u + sl]);   // the stage has been read')
    self.w('tfb_tc::st_wait();')
    self.w('tfb_tc::fence_before();')
    self.w('__syncwarp();')
    self.w(f'if (lane == 0) tfb_tc::mbar_arrive(&bars[{B["AF"]}u + k]);')
    self.close()
    self.close()

  def _epilogue_teams(self):
    """Team k: accumulators k to shared memory, then one bulk store per element."""
    s, L, B = self.s, self.lay, self.bars
    o, M, N, te, n_mma = s.out, s.M, s.N, L['te'], L['n_mma']
    vol = o.element_volume()
    self.open('else')
    self.w(f'const unsigned quad = warp & 3u, k = (warp - {4 * TEAMS}u) >> 2;')
    self.w(f'const unsigned tid = quad * 32u + lane;')
    self.w(f'const unsigned le = tid / {N}u, lj = tid - le * {N}u;')
    self.w(f'const unsigned acc = tmem + ((quad * 32u) << 16) + {self._acc("k")};')
    self.w(f'float* const ost = reinterpret_cast<float*>(tfb_smem_raw + {L["off_ost"]} + k * {L["ost"]}u);')
    self.w('unsigned ph = 0;')
    self.open(f'for (size_t tile = blockIdx.x + (size_t)k * gridDim.x; tile < numTiles; tile += (size_t)gridDim.x * {TEAMS}u, ++ph)')
    if not s.accumulate:
      # the address, read before the wait for the accumulators
      self.w(f'const size_t ee = tile * {te}u + tid;')
      self.w(f'float* const dst = tid < {te}u && ee < numElements && (flags == nullptr || flags[ee] != 0u) ? {self._elem_ptr(o, "ee")} : nullptr;')
    self.w(f'const bool ok = tfb_tc::mbar_wait_h(&bars[{B["DF"]}u + k], ph & 1u, {self.WAIT_NS}ull);')
    self.w(f'if (!ok) atomicMax(&tfb_err_{self.base}, 20u);')
    if not s.accumulate:
      self.w('tfb_tc::bulk_wait_read();   // this thread\'s earlier stores have read the buffer')
    self.w('// one answer for the team: all of it goes on, or none')
    self.w('__syncwarp();')
    self.w('if (tfb_tc::any_sync(1u + k, 128u, !ok)) break;')
    self.w('tfb_tc::fence_after();')
    self.w(f'const size_t el = tile * {te}u + le;')
    if s.accumulate:
      self.w(f'const bool active = tid < {te * N}u && el < numElements && (flags == nullptr || flags[el] != 0u);')
      self.w(f'float* const col = active ? {self._elem_ptr(o, "el")} + (size_t)lj * {M}u : nullptr;')
    self.w('#pragma unroll')
    self.open(f'for (int r0 = 0; r0 < {M}; r0 += 8)')
    self.w('unsigned dv[8], dc[8];')
    self.w('tfb_tc::ld_x8(acc + r0, dv);')
    self.w(f'tfb_tc::ld_x8(acc + {n_mma}u + r0, dc);')
    self.w('tfb_tc::ld_wait();')
    self.w('float x[8];')
    self.w('#pragma unroll')
    self.w('for (int i = 0; i < 4; ++i) { const float2 v = __fadd2_rn(make_float2(__uint_as_float(dv[2 * i]), __uint_as_float(dv[2 * i + 1])), '
           'make_float2(__uint_as_float(dc[2 * i]), __uint_as_float(dc[2 * i + 1]))); x[2 * i] = v.x; x[2 * i + 1] = v.y; }')
    if s.accumulate:
      self.open('if (active)')
      self.w('#pragma unroll')
      self.w(f'for (int i = 0; i < 8; ++i) if (r0 + i < {M}) col[r0 + i] += x[i];')
      self.close()
    else:
      self.open(f'if (tid < {te * N}u)')
      self.w(f'float4* const y = reinterpret_cast<float4*>(ost + tid * {M}u + r0);')
      self.w('y[0] = make_float4(x[0], x[1], x[2], x[3]);')
      self.w(f'if (r0 + 4 < {M}) y[1] = make_float4(x[4], x[5], x[6], x[7]);')
      self.close()
    self.close()
    self.w('tfb_tc::fence_before();')
    self.w('__syncwarp();')
    self.w(f'if (lane == 0) tfb_tc::mbar_arrive(&bars[{B["DE"]}u + k]);')
    if not s.accumulate:
      self.w('tfb_tc::fence_proxy_async();')
      self.w('tfb_tc::named_sync(1u + k, 128u);')
      self.open('if (dst != nullptr)')
      self.w(f'if ((reinterpret_cast<uintptr_t>(dst) & 15u) == 0u) tfb_tc::bulk_store(dst, ost + tid * {vol}u, {vol * 4}u);')
      self.w(f'else for (unsigned q = 0; q < {vol}u; ++q) dst[q] = ost[tid * {vol}u + q];')
      self.close()
    self.close()
    if not s.accumulate:
      self.w('tfb_tc::bulk_wait();  // the last stores have landed')
    self.close()


def emit_direct(chain, plan_, context, base_name, globals_):
  return _Direct(chain, match_left_chain(chain), plan_, context, base_name).emit(globals_)
