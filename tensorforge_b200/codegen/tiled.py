"""Tiled generator (CUDA cores): chains of contractions over per-element operands.

Covers the descriptor lists that have no shared-left form (plan/chains.py): per-element
left operands, transposed products, temporaries between general contractions, sparse
per-element operands, products of any rank. A group of G lanes owns one batch element:

  * every operand a stage reads is brought into shared memory once per element with
    cp.async (16 bytes where the element's address allows it, else one value at a time),
    compactly stored ones are scattered into their dense box; shared (Addressing.NONE)
    operands are brought in once per CTA;
  * a stage's destination is cut into TX x TY register tiles over its first index and its
    widest other one, one tile per lane. Per contracted index a lane loads TX + TY values
    instead of 2 TX TY, with 16-byte shared-memory loads along whichever of its indices an
    operand stores first; columns are padded to an odd number of 16-byte units, so that
    loads of neighbouring columns fall on different banks;
  * temporaries stay in shared memory, results go to global memory with 16-byte stores.

With G = 32 (the default as long as eight warps fit an SM) a warp owns its element alone:
no CTA barrier, and while some warps of the SM wait for their operands others compute.

What bounds it: the operands' bytes, then shared-memory loads. One element's 32x32x32
product takes 12 KB of HBM traffic and, with 8x4 tiles, 3 x 32 16-byte loads per lane.
Measured on B200 against the generic generator (one lane per destination entry, both
factors of every product loaded from global memory or L1):
32x32x32 through pointer arrays, 50,000 elements: 472 -> 113 us (5.4 TB/s); A^T B of the same
size through a temporary, 16,802 elements: 2,009 -> 57 us; A (B C) + D of 56x56, 56x9 and 9x9
factors, 20,000 elements: 235 -> 72 us (5.2 TB/s), of which operands read along their first
index copied as one run instead of column by column and packed FMAs gave 90 -> 72.

Sums run over the contracted indices in the order the generic generator uses (the first
one fastest) with one fused multiply-add per product, so results are the same bits.
"""
from .generic import GenericEmitter, _align4, _colmajor, _prod, _sparse_box, assign_offsets
from .colprog import CP_HELPERS, resident_grid

SMEM_PER_CTA = 227 * 1024
SMEM_PER_SM = 228 * 1024


def padded_strides(sizes, vec, odd=True):
  """Strides of a shared-memory box: the first extent rounded up to 16 bytes and, between
  columns, to an odd number of 16-byte units (`odd`)."""
  if not sizes:
    return [], vec
  p = -(-sizes[0] // vec) * vec
  if odd and _prod(sizes[1:]) > 1 and (p // vec) % 2 == 0:
    p += vec
  strides, acc = [1], p
  for s in sizes[1:]:
    strides.append(acc)
    acc *= s
  return strides, -(-acc // vec) * vec


class Region:
  """A shared-memory box: `sizes` from `lower` of operand `op`, as read by some stages.

  kind 'copy' (dense operand copied from global memory), 'sparse' (expanded), 'tmp'."""

  def __init__(self, name, op, kind, where, sizes, lower, vec):
    self.name, self.op, self.kind, self.where = name, op, kind, where
    self.sizes, self.lower, self.vec = list(sizes), list(lower), vec
    self.strides, self.volume = padded_strides(self.sizes, vec)
    self.rows_first = True   # every reader takes neighbouring lanes along the first index
    self.first = self.last = None
    self.src_strides, self.src_offset = [], 0
    self.offset = 0

  def unpad(self):
    """Lanes that read along the first index meet no bank twice: whole columns, one after the
    other, which a linear copy fills."""
    self.strides, self.volume = padded_strides(self.sizes, self.vec, False)

  def in_pieces(self):
    """Whether the columns can be copied 16 bytes at a time."""
    vec = self.vec
    return bool(self.sizes) and (self.sizes[0] % vec == 0 and self.src_strides[0] == 1 and self.src_offset % vec == 0
                                 and all(s % vec == 0 for s, n in zip(self.src_strides[1:], self.sizes[1:]) if n > 1))

  def used(self, stage):
    self.first = stage if self.first is None else min(self.first, stage)
    self.last = stage if self.last is None else max(self.last, stage)


class Staging:
  """Shared-memory regions of a chain and which one each operand reference reads.

  Operands are copied at the start of the element, but never ahead of a stage that writes
  global memory: stages between two such writes form an epoch, and what an epoch reads is
  copied at its start. An operand that some stage writes is read from global memory."""

  def __init__(self, chain, stage_shared=True):
    self.chain = chain
    self.vec = 16 // chain.fp.size()
    self.regions = []
    self.of_ref = {}        # (stage, position) -> Region
    self.of_dest = {}       # stage -> Region holding the destination (temporary), or its previous values
    self.epoch_start = {}   # first stage of an epoch -> regions copied there
    written = {id(st.dest) for st in chain.stages}
    by_key, epoch, start = {}, 0, 0
    done = set()
    for si, st in enumerate(chain.stages):
      for ri, ref in enumerate(st.ops):
        r = self._region(ref, st, written, epoch, by_key, stage_shared)
        if r is not None:
          r.used(start if r.kind == 'copy' and r.where == 'elem' else si)
          r.used(si)
          r.rows_first = r.rows_first and bool(ref.target) and ref.target[0] == 0
          self.of_ref[si, ri] = r
      if st.dest.kind == 'tmp':
        r = by_key.get(('tmp', st.dest.name))
        if r is None:
          lower = [l for l, _ in st.n_ranges]
          r = self._add(by_key, ('tmp', st.dest.name), st.dest, 'tmp', 'elem', [u - l for l, u in st.n_ranges], lower)
        r.used(si)
        self.of_dest[si] = r
      else:
        if st.add and id(st.dest) not in done:
          # previous values of an accumulated destination, copied with the inputs
          key = ('add', st.dest.name, si)
          r = self._add(by_key, key, st.dest, 'copy', 'elem', [u - l for l, u in st.n_ranges], [l for l, _ in st.n_ranges])
          self._source(r, st.dest_strides, st.dest_origin)
          r.used(start)
          r.used(si)
          self.of_dest[si] = r
        done.add(id(st.dest))
        epoch, start = epoch + 1, si + 1
    for r in self.regions:
      if r.kind == 'copy' and r.rows_first:
        r.unpad()
    ranges = {r.name: (r.first, r.last) for r in self.regions if r.where == 'elem'}
    sizes = {r.name: _align4(r.volume) for r in self.regions if r.where == 'elem'}
    offsets, self.per_elem = assign_offsets(sizes, ranges)
    self.shared = 0
    for r in self.regions:
      if r.where == 'elem':
        r.offset = offsets[r.name]
        # zeros outside a sparse pattern survive from element to element where nothing else
        # lives in the region's memory
        r.alone = not any(q is not r and q.where == 'elem' and offsets[q.name] < r.offset + sizes[r.name]
                          and r.offset < offsets[q.name] + sizes[q.name] for q in self.regions)
        if r.kind == 'copy':
          self.epoch_start.setdefault(r.first, []).append(r)
      else:
        r.offset = self.shared
        self.shared += _align4(r.volume)

  def _add(self, by_key, key, op, kind, where, sizes, lower):
    r = Region(f'r{len(self.regions)}', op, kind, where, sizes, lower, self.vec)
    by_key[key] = r
    self.regions.append(r)
    return r

  def _source(self, r, strides, origin):
    r.src_strides = list(strides)
    r.src_offset = sum((l - o) * s for l, o, s in zip(r.lower, origin, strides))

  def _region(self, ref, st, written, epoch, by_key, stage_shared):
    o = ref.op
    if o.kind == 'tmp':
      return by_key[('tmp', o.name)]
    if o.kind not in ('batched', 'shared') or (o.kind == 'batched' and id(o) in written):
      return None
    where = 'elem' if o.kind == 'batched' else 'cta'
    if o.sparse:
      key = ('sparse', o.name)
      return by_key.get(key) or self._add(by_key, key, o, 'sparse', where, _sparse_box(o), o.bbox.lower())
    if where == 'cta' and not stage_shared:
      return None
    box = [st.n_ranges[t] if t >= 0 else st.k_ranges[-t - 1] for t in ref.target]
    key = (o.name, tuple(ref.strides), tuple(ref.origin), tuple(box), epoch if where == 'elem' else 0)
    r = by_key.get(key)
    if r is None:
      r = self._add(by_key, key, o, 'copy', where, [u - l for l, u in box], [l for l, _ in box])
      self._source(r, ref.strides, ref.origin)
    return r


class _Access:
  """How one operand reference is read inside a stage's tile."""

  def __init__(self, staging, si, ri, st, vec, vw):
    ref = st.ops[ri]
    self.ref, self.o = ref, ref.op
    self.dim_of = {t: d for d, t in enumerate(ref.target)}
    self.region = staging.of_ref.get((si, ri))
    self.kind = self.o.kind
    box = [st.n_ranges[t] if t >= 0 else st.k_ranges[-t - 1] for t in ref.target]
    if self.region is not None:
      self.strides = self.region.strides
      self.first = [b[0] - l for b, l in zip(box, self.region.lower)]
    else:
      self.strides = list(ref.strides)
      self.first = [b[0] - o for b, o in zip(box, ref.origin)]
    self.const = sum(f * s for f, s in zip(self.first, self.strides))
    # 16-byte loads along the dimension stored first
    aligned = (self.region is not None and len(self.strides) > 0 and self.first[0] % vec == 0
               and len(self.dim_of) == len(ref.target))
    t0 = ref.target[0] if ref.target else None
    self.vec_x = aligned and t0 == 0 and vw == vec
    self.vec_k = aligned and t0 == -1 and -1 in self.dim_of

  def stride(self, t):
    return sum(s for u, s in zip(self.ref.target, self.strides) if u == t)

  def has(self, t):
    return t in self.dim_of


def stage_tile(staging, si, st, lanes):
  """(TX, TY, y index) of stage `si`: rows and columns per lane.

  Least shared-memory and FMA issue time over the rounds the lanes need, from measured
  rates: a warp's 16-byte shared load takes the SM 2-4 cycles, its FMA a quarter of one
  (half of one in FP64)."""
  vec = staging.vec
  ext = [u - l for l, u in st.n_ranges]
  X = ext[0] if ext else 1
  yd = max(range(1, len(ext)), key=lambda d: ext[d]) if len(ext) > 1 else None
  Y = ext[yd] if yd is not None else 1
  rest = _prod(ext) // (X * Y)
  K = max(1, st.k_volume())
  best = None
  for tx in (1, 2, 4, 8, 12, 16):
    if tx > -(-X // vec) * vec:
      continue
    for ty in range(1, 17):
      if ty > Y or tx * ty > (48 if vec == 4 else 24):
        continue
      vw = min(vec, tx)
      if tx % vw:
        continue
      rounds = -(-(-(-X // tx) * -(-Y // ty) * rest) // lanes)
      lds = 0.0
      for ri in range(len(st.ops)):
        a = _Access(staging, si, ri, st, vec, vw)
        if a.kind in ('scalar', 'data'):
          continue
        n = (tx if a.has(0) else 1) * (ty if yd is not None and a.has(yd) else 1)
        lds += 3.0 * n / vec if (a.vec_x or a.vec_k) else 1.2 * n
      cost = rounds * (K * (lds + tx * ty * (0.25 if vec == 4 else 0.5) + 0.5) + 2.0 * tx * ty)
      if best is None or cost < best[0] * 0.999:
        best = (cost, tx, ty)
  return best[1], best[2], yd


def passes_through(chain, s):
  """Whether most of what a chain reads per element is copied value by value and used once, while
  its results occupy most of the generic generator's 256 lanes: shared memory only adds a detour then.
  Measured on B200, generic / tiled, up to 5,000 and from 20,000 elements, first index of the large
  operand contracted or not, boxes off the 16-byte grid: 396 results from 12,704 values 0.30 and 0.36,
  396 from 2,376 0.45 and 0.52, 240 from 7,920 0.44 and 0.43, 160 from 4,028 0.42 and 0.48, 320 from 1,600
  0.81 and 0.78, 264 from 4,240 0.84 and 0.99; but 128 from 1,640 1.38 and 2.58, 122 from 12,423 1.12 and 1.26,
  48 from 2,160 0.82 and 1.01, 20 from 16,632 1.49 and 1.81, and copied in 16-byte pieces 480 from 10,100 1.08 and
  1.04, 512 from 5,204 0.89 and 0.96."""
  copies = [r for r in s.regions if r.where == 'elem' and r.kind != 'tmp']
  values = sum(_prod(r.sizes) for r in copies)
  single = sum(_prod(r.sizes) for r in copies if r.kind == 'copy' and not r.in_pieces())
  size = lambda ranges: _prod([u - l for l, u in ranges])
  products = sum(size(st.n_ranges + st.k_ranges) for st in chain.stages)
  return (values >= 1500 and 2 * single >= values and products <= 1.1 * values
          and max(size(st.n_ranges) for st in chain.stages) >= 140)


def tiled_plan(chain, fp_size, variant):
  """(params, shared-memory bytes) for `chain`, or None where another generator has to take it."""
  if not chain.stages or chain.has_elementwise() or any(st.dest.sparse for st in chain.stages):
    return None
  ranges = {}
  for st in chain.stages:   # no empty index range, and a temporary keeps one shape
    if any(u <= l for l, u in st.n_ranges + st.k_ranges):
      return None
    if st.dest.kind == 'tmp' and ranges.setdefault(id(st.dest), st.n_ranges) != st.n_ranges:
      return None
  for stage_shared in (True, False):
    s = Staging(chain, stage_shared)
    if (s.shared + s.per_elem) * fp_size <= SMEM_PER_CTA:
      break
  else:
    return None

  if not variant and passes_through(chain, s):
    return None

  def resident(lanes, e):
    smem = (s.shared + s.per_elem * e) * fp_size
    if smem > SMEM_PER_CTA:
      return 0
    return min(SMEM_PER_SM // (smem + 1024), 32, 64 // (lanes * e // 32)) * (lanes * e // 32)

  if 'threads_per_element' in variant:
    lanes = variant['threads_per_element']
    if lanes % 32 or not 32 <= lanes <= 1024:
      return None
    elems = min(variant.get('elements_per_block', 1), 1024 // lanes) if lanes == 32 else 1
  else:
    lanes, elems = 32, max((4, 8, 2, 1), key=lambda e: min(24, resident(32, e)))
    while resident(lanes, elems) < 8 and lanes < 256:
      lanes, elems = lanes * 2, 1
  if resident(lanes, elems) == 0:
    return None
  return ({'threads_per_element': lanes, 'elements_per_block': elems, 'stage_shared': int(stage_shared)},
          (s.shared + s.per_elem * elems) * fp_size)


class TiledEmitter(GenericEmitter):
  def __init__(self, chain, plan, context, base_name):
    super().__init__(chain, plan, context, base_name)
    self.st = Staging(chain, bool(plan.params['stage_shared']))
    self.VEC = self.st.vec
    self.VT = 'float4' if self.VEC == 4 else 'double2'
    self.comps = ['x', 'y', 'z', 'w'][:self.VEC]
    self.sync = '__syncwarp()' if self.G == 32 else '__syncthreads()'

  # ---------------------------------------------------------------- tables
  def _tables(self):
    T = self.T
    for o in self.chain.operands:
      if o.kind == 'data' and len(o.shape) > 0:
        vals = [0.0] * max(1, _prod(o.shape))
        if isinstance(o.tensor.data, dict):
          for idx, v in o.tensor.data.items():
            vals[sum(i * s for i, s in zip(idx, _colmajor(list(o.shape))))] = v
        self.w(f'__device__ const {T} data_{o.name}_{self.base}[{len(vals)}] = {{{", ".join(self.lit(v) for v in vals)}}};')
    for r in self.st.regions:
      if r.kind == 'sparse':
        pairs = sorted((pos, sum((i - l) * s for i, l, s in zip(idx, r.lower, r.strides))) for idx, pos in r.op.nonzeros())
        r.pairs = pairs
        r.in_order = all(p == i for i, (p, _) in enumerate(pairs))
        self.w(f'__device__ const unsigned short scat_{r.name}_{self.base}[{max(1, len(pairs))}] = '
               f'{{{", ".join(str(d) for _, d in pairs) or "0"}}};')
        if not r.in_order:
          self.w(f'__device__ const unsigned short spos_{r.name}_{self.base}[{max(1, len(pairs))}] = '
                 f'{{{", ".join(str(p) for p, _ in pairs) or "0"}}};')

  # ---------------------------------------------------------------- copies
  def _fill(self, r, lane, step):
    """Copy region `r` from its operand's element (or the shared operand) with cp.async."""
    VEC, T = self.VEC, self.T
    small = 'copy4' if VEC == 4 else 'copy8'
    src = f'glb_{r.op.name}'
    if r.kind == 'sparse':
      pos = 'i' if r.in_order else f'spos_{r.name}_{self.base}[i]'
      with self.block(f'for (unsigned i = {lane}; i < {len(r.pairs)}u; i += {step})'):
        self.w(f'tfb_cp::{small}({r.name} + scat_{r.name}_{self.base}[i], {src} + {pos});')
      return
    if not r.sizes:   # a rank-0 operand: one value
      self.w(f'if ({lane} == 0u) tfb_cp::{small}({r.name}, {src} + {r.src_offset});')
      return
    inner, cols = r.sizes[0], _prod(r.sizes[1:])

    def address(n, width):
      """Decode chunk `n` of `width` values: (destination, source) offsets."""
      per = inner // width
      self.w(f'const unsigned col = {n} / {per}u, row = ({n} - col * {per}u) * {width}u;' if cols > 1 else
             f'const unsigned row = {n} * {width}u;')
      d, s = ['row'], [f'row * {r.src_strides[0]}u' if r.src_strides[0] != 1 else 'row']
      div = 1
      for k in range(1, len(r.sizes) if cols > 1 else 1):
        part = f'(col / {div}u)' if div > 1 else 'col'
        if k < len(r.sizes) - 1:
          part = f'({part} % {r.sizes[k]}u)'
        d.append(f'{part} * {r.strides[k]}u')
        s.append(f'{part} * {r.src_strides[k]}u')
        div *= r.sizes[k]
      return ' + '.join(d), ' + '.join(s + ([f'{r.src_offset}u'] if r.src_offset else []))

    def scalar():
      with self.block(f'for (unsigned q = {lane}; q < {inner * cols}u; q += {step})'):
        d, s = address('q', 1)
        self.w(f'tfb_cp::{small}({r.name} + {d}, {src} + {s});')
    vector = r.in_pieces()
    if not vector:
      scalar()
      return
    # one run of memory on both sides: equal strides alone do not say so, a box of 8 rows out of
    # 12 has its source's pitch of 12 as its padded one
    linear = r.strides == r.src_strides == _colmajor(r.sizes)
    with self.block(f'if ((reinterpret_cast<uintptr_t>({src}) & 15u) == 0u)'):
      if linear:
        self.w('#pragma unroll 4')
        self.w(f'for (unsigned q = {lane}; q < {inner * cols // VEC}u; q += {step}) '
               f'tfb_cp::copy16({r.name} + q * {VEC}u, {src} + {r.src_offset}u + q * {VEC}u);')
      else:
        with self.block(f'for (unsigned q = {lane}; q < {inner * cols // VEC}u; q += {step})'):
          d, s = address('q', VEC)
          self.w(f'tfb_cp::copy16({r.name} + {d}, {src} + {s});')
    with self.block('else'):
      scalar()

  def _zero(self, r, lane, step):
    with self.block(f'for (unsigned i = {lane}; i < {r.volume}u; i += {step})'):
      self.w(f'{r.name}[i] = {self.lit(0)};')

  # ---------------------------------------------------------------- kernel
  def emit_kernel(self, globals_):
    chain, T, G, E = self.chain, self.T, self.G, self.E
    st = self.st
    self.w(CP_HELPERS)
    self.w(f'// generated by tensorforge_b200 (strategy: tiled, G={G}, E={E})')
    for line in self._meta():
      self.w(line)
    self._tables()
    self.w()
    self.w(f'__global__ void __launch_bounds__({G * E}) kernel_{self.base}({", ".join(self.kernel_params(globals_))}) {{')
    self.ind += 1
    self.w('extern __shared__ __align__(16) unsigned char tfb_smem_raw[];')
    self.w(f'{T}* const tfb_smem = reinterpret_cast<{T}*>(tfb_smem_raw);')
    for o in chain.operands:
      if o.kind == 'data' and len(o.shape) > 0:
        self.w(f'const {T}* const data_{o.name} = data_{o.name}_{self.base};')
      if o.kind == 'shared':
        self.w(f'const {T}* const glb_{o.name} = {o.name};')
    self.w(f'const unsigned slot = threadIdx.x / {G}u, lane = threadIdx.x % {G}u;')
    self.w(f'{T}* const elem_smem = tfb_smem + {st.shared} + slot * {st.per_elem}u;')
    for r in st.regions:
      self.w(f'{T}* const {r.name} = {"elem_smem" if r.where == "elem" else "tfb_smem"} + {r.offset};')
    cta = [r for r in st.regions if r.where == 'cta']
    for r in cta:
      if r.kind == 'sparse':
        self._zero(r, 'threadIdx.x', f'{G * E}u')
    for r in st.regions:
      if r.kind == 'sparse' and r.where == 'elem' and r.alone:
        self._zero(r, 'lane', f'{G}u')
    self.w('__syncthreads();')
    for r in cta:
      self._fill(r, 'threadIdx.x', f'{G * E}u')
    if cta:
      self.w('tfb_cp::commit();')
      self.w('tfb_cp::wait_all();')
      self.w('__syncthreads();')
    with self.block(f'for (size_t tile = blockIdx.x; tile * {E}u < numElements; tile += gridDim.x)'):
      self.w(f'const size_t batchId = tile * {E}u + slot;')
      self.w('bool active = batchId < numElements;')
      self.w('if (active && flags != nullptr) active = flags[batchId] != 0u;')
      for o in chain.operands:
        if o.kind != 'batched':
          continue
        const = 'const ' if o.is_const else ''
        if o.addressing.name == 'STRIDED':
          at = f'{o.name} + batchId * {o.element_volume()}u + {o.name}_extraOffset'
        else:
          at = f'{o.name}[batchId] + {o.name}_extraOffset'
        self.w(f'{const}{T}* const glb_{o.name} = active ? {at} : nullptr;')
      if G == 32:
        # a warp's own element: it skips a masked one without waiting for anybody
        self.w('if (!active) continue;')
      for si, stage in enumerate(chain.stages):
        copies = st.epoch_start.get(si, [])
        sparse = [r for r in st.regions if r.kind == 'sparse' and r.where == 'elem' and r.first == si]
        again = [r for r in sparse if not r.alone]
        if again:
          for r in again:
            self._zero(r, 'lane', f'{G}u')
          self.w(f'{self.sync};')
        if copies or sparse:
          with self.block('if (active)'):
            for r in copies + sparse:
              self._fill(r, 'lane', f'{G}u')
          self.w('tfb_cp::commit();')
          self.w('tfb_cp::wait_all();')
          self.w(f'{self.sync};')
        self.w(f'// stage {si}: {stage.descr}'.replace('\n', ' '))
        with self.block('if (active)'):
          self._emit_tile_stage(si, stage)
        self.w(f'{self.sync};')
    self.ind -= 1
    self.w('}')
    return '\n'.join(self.lines)

  # ---------------------------------------------------------------- stage
  def _emit_tile_stage(self, si, st):
    T, G, VEC = self.T, self.G, self.VEC
    tx, ty, yd = stage_tile(self.st, si, st, G)
    vw = min(VEC, tx)
    ext = [u - l for l, u in st.n_ranges]
    X, Y = (ext[0] if ext else 1), (ext[yd] if yd is not None else 1)
    nx, ny = -(-X // tx), -(-Y // ty)
    rest = [d for d in range(1, len(ext)) if d != yd]
    items = nx * ny * _prod([ext[d] for d in rest])
    acc = [_Access(self.st, si, ri, st, VEC, vw) for ri in range(len(st.ops))]
    self.w(f'// {tx} x {ty} values per lane, {items} tiles')
    self.w(f'if (lane < {items}u) {{' if items <= G else f'for (unsigned d = lane; d < {items}u; d += {G}u) {{')
    self.ind += 1
    d = 'lane' if items <= G else 'd'
    self.w(f'const int xg = (int)({d} % {nx}u);')
    self.w(f'const int yg = (int)({d} / {nx}u{f" % {ny}u" if rest else ""});')
    div = nx * ny
    for k in rest:
      self.w(f'const int z{k} = (int)({d} / {div}u % {ext[k]}u);')
      div *= ext[k]
    # rows: quads of vw rows, nx quads apart; columns ny apart. Quads and columns past the
    # end repeat the last one and are not stored.
    for s in range(tx // vw):
      last = (X - 1) // vw * vw
      row = f'(xg + {s * nx}) * {vw}'
      self.w(f'const int x{s} = {row};' if (nx * (s + 1) - 1) * vw <= last else f'const int x{s} = min({row}, {last});')
    for t in range(ty):
      col = f'yg + {t * ny}'
      self.w(f'const int y{t} = {col};' if ny * (t + 1) <= Y else f'const int y{t} = min({col}, {Y - 1});')

    def row_index(s, v):
      return f'(x{s} + {v})' if X % vw == 0 or v == 0 else f'min(x{s} + {v}, {X - 1})'
    # FP32 products of rows (16-byte pieces) and columns run as packed FMAs, two rows each
    self.packed = (VEC == 4 and vw == VEC and len(acc) == 2 and acc[0].vec_x and not (yd is not None and acc[0].has(yd))
                   and acc[1].kind != 'data' and not acc[1].has(0))
    self.value = (lambda i, t: f'acc[{i // 2 + tx // 2 * t}].{"xy"[i % 2]}') if self.packed else (lambda i, t: f'acc[{i + tx * t}]')
    if self.packed:
      self.w(f'float2 acc[{tx // 2 * ty}];')
    else:
      self.w(f'{T} acc[{tx * ty}];')
    self.w('#pragma unroll')
    self.w(f'for (int i = 0; i < {tx * ty // (2 if self.packed else 1)}; ++i) '
           f'acc[i] = {"make_float2(0.f, 0.f)" if self.packed else self.lit(0)};')
    nk = len(st.k_ranges)
    for a in acc:
      a.name = f'p{acc.index(a)}'
      if a.kind in ('scalar', 'data'):
        continue
      base = a.region.name if a.region is not None else f'glb_{a.o.name}'
      terms = [str(a.const)] + [f'z{k} * {a.stride(k)}' for k in rest if a.has(k)]
      self.w(f'const {T}* const {a.name} = {base} + {" + ".join(terms)};')
    for k in reversed(range(1, nk)):
      lo, up = st.k_ranges[k]
      self.w(f'for (int k{k} = 0; k{k} < {up - lo}; ++k{k}) {{')
      self.ind += 1
    if nk == 0:
      self._tile_products(st, acc, yd, tx, ty, vw, '0', 1, row_index)
    else:
      K = st.k_ranges[0][1] - st.k_ranges[0][0]
      full = K // VEC * VEC
      if full:
        self.w('#pragma unroll 2')
        self.w(f'for (int k0 = 0; k0 < {full}; k0 += {VEC}) {{')
        self.ind += 1
        self._tile_products(st, acc, yd, tx, ty, vw, 'k0', VEC, row_index)
        self.ind -= 1
        self.w('}')
      if K > full:
        with self.block(''):
          self._tile_products(st, acc, yd, tx, ty, vw, str(full), K - full, row_index)
    for _ in range(1, nk):
      self.ind -= 1
      self.w('}')
    self._tile_store(si, st, yd, rest, X, Y, tx, ty, vw, nx, ny)
    self.ind -= 1
    self.w('}')

  def _tile_products(self, st, acc, yd, tx, ty, vw, k0, count, row_index):
    """acc[i + tx * t] += product of the operands, for `count` values of the first contracted index from `k0`."""
    T, VEC, VT = self.T, self.VEC, self.VT
    nk = len(st.k_ranges)

    def fixed(a, k):
      """Offset of the contracted indices, with the first one at `k`."""
      terms = [f'({k}) * {a.stride(-1)}' if a.stride(-1) != 1 else f'({k})'] if a.has(-1) else []
      terms += [f'k{j} * {a.stride(-j - 1)}' for j in range(1, nk) if a.has(-j - 1)]
      return terms

    def place(a, s, v, t):
      out = []
      if a.has(0):
        out.append(f'{row_index(s, v) if v is not None else f"x{s}"} * {a.stride(0)}')
      if yd is not None and a.has(yd):
        out.append(f'y{t} * {a.stride(yd)}')
      return out

    def spots(a):
      """(row, column) combinations a lane needs values of."""
      return [(i, t) for t in (range(ty) if yd is not None and a.has(yd) else (0,))
              for i in (range(tx) if a.has(0) else (0,))]
    vectors = {}
    for a in acc:
      if a.kind in ('scalar', 'data') or not (a.vec_k and count == VEC):
        continue
      for i, t in spots(a):
        n = f'{a.name}v{i}_{t}'
        at = ' + '.join(place(a, i // vw, i % vw, t) + fixed(a, k0)) or '0'
        self.w(f'const {VT} {n} = *reinterpret_cast<const {VT}*>({a.name} + {at});')
        vectors[a.name, i, t] = n
    for kk in range(count):
      if st.k_ranges:
        self.w('{')
        self.ind += 1
      k = k0 if kk == 0 else f'{k0} + {kk}'
      names = {}
      for a in acc:
        if a.kind == 'scalar':
          names[a.name] = lambda i, t, a=a: a.o.name
        elif a.kind == 'data':
          names[a.name] = lambda i, t, a=a: self._data_at(a, st, yd, k, row_index(i // vw, i % vw), f'y{t}')
        elif (a.name, 0, 0) in vectors:
          names[a.name] = lambda i, t, a=a: f'{vectors[a.name, i if a.has(0) else 0, t if yd is not None and a.has(yd) else 0]}.{self.comps[kk]}'
        elif a.vec_x:
          for t in sorted({t for _, t in spots(a)}):
            for s in range(tx // vw):
              at = ' + '.join(place(a, s, None, t) + fixed(a, k)) or '0'
              self.w(f'const {VT} {a.name}x{s}_{t} = *reinterpret_cast<const {VT}*>({a.name} + {at});')
          names[a.name] = lambda i, t, a=a: f'{a.name}x{i // vw}_{t if yd is not None and a.has(yd) else 0}.{self.comps[i % vw]}'
        else:
          for i, t in spots(a):
            at = ' + '.join(place(a, i // vw, i % vw, t) + fixed(a, k)) or '0'
            self.w(f'const {T} {a.name}s{i}_{t} = {a.name}[{at}];')
          names[a.name] = lambda i, t, a=a: f'{a.name}s{i if a.has(0) else 0}_{t if yd is not None and a.has(yd) else 0}'
      for t in range(ty if self.packed else 0):
        b = names[acc[1].name](0, t)
        self.w(f'{{ const float2 bb = make_float2({b}, {b});')
        for i in range(0, tx, 2):
          a = ', '.join(names[acc[0].name](i + h, t) for h in (0, 1))
          self.w(f'  acc[{i // 2 + tx // 2 * t}] = __ffma2_rn(make_float2({a}), bb, acc[{i // 2 + tx // 2 * t}]);')
        self.w('}')
      for t in range(0 if self.packed else ty):
        for i in range(tx):
          prod = ' * '.join(names[a.name](i, t) for a in acc) if acc else self.lit(0)
          self.w(f'acc[{i + tx * t}] += {prod};')
      if st.k_ranges:
        self.ind -= 1
        self.w('}')

  def _data_at(self, a, st, yd, k, row, col):
    exprs = []
    for tgt in a.ref.target:
      lo = (st.n_ranges[tgt] if tgt >= 0 else st.k_ranges[-tgt - 1])[0]
      var = row if tgt == 0 else col if tgt == yd else f'z{tgt}' if tgt > 0 else f'({k})' if tgt == -1 else f'k{-tgt - 1}'
      exprs.append(f'({var} + {lo})')
    return self._data_value(a.o, a.ref, exprs)

  def _tile_store(self, si, st, yd, rest, X, Y, tx, ty, vw, nx, ny):
    T, VEC, VT = self.T, self.VEC, self.VT
    held = self.st.of_dest.get(si)
    if st.dest.kind == 'tmp':
      strides, first, base = held.strides, [0] * len(st.n_ranges), held.name
    else:
      strides = list(st.dest_strides)
      first = [l - o for (l, _), o in zip(st.n_ranges, st.dest_origin)]
      base = f'glb_{st.dest.name}'
    terms = [str(sum(f * s for f, s in zip(first, strides)))] + [f'z{k} * {strides[k]}' for k in rest]
    self.w(f'{T}* const out = {base} + {" + ".join(terms)};')
    if st.add and held is not None and st.dest.kind != 'tmp':
      prior = [f'z{k} * {held.strides[k]}' for k in rest]
      self.w(f'const {T}* const prev = {held.name}{" + " + " + ".join(prior) if prior else ""};')
    sy = strides[yd] if yd is not None else 0
    hy = held.strides[yd] if held is not None and yd is not None else 0

    def guard(s, t):
      g = []
      if (nx * (s + 1) - 1) * vw >= X:
        g.append(f'(xg + {s * nx}) * {vw} < {X}')
      if ny * (t + 1) > Y:
        g.append(f'yg + {t * ny} < {Y}')
      return g

    def value(i, t, at, prev_at):
      v = self.value(i, t)
      if not st.add:
        return v
      return f'{v} + {"prev" if st.dest.kind != "tmp" and held is not None else "out"}[{prev_at if st.dest.kind != "tmp" and held is not None else at}]'

    def emit(vector):
      for t in range(ty):
        for s in range(tx // vw):
          g = guard(s, t)
          self.w((f'if ({" && ".join(g)}) ' if g else '') + '{')
          self.ind += 1
          at, pat = f'x{s} + y{t} * {sy}', f'x{s} + y{t} * {hy}'
          if vector:
            vals = ', '.join(value(s * vw + v, t, f'{at} + {v}', f'{pat} + {v}') for v in range(vw))
            self.w(f'*reinterpret_cast<{VT}*>(out + {at}) = make_{VT}({vals});')
          else:
            for v in range(vw):
              tail = X % vw and v >= X % vw
              self.w((f'if (x{s} + {v} < {X}) ' if tail else '')
                     + f'out[{at} + {v}] = {value(s * vw + v, t, f"{at} + {v}", f"{pat} + {v}")};')
          self.ind -= 1
          self.w('}')
    even = (vw == VEC and all(s % VEC == 0 for s, (l, u) in zip(strides[1:], st.n_ranges[1:]) if u - l > 1)
            and sum(f * s for f, s in zip(first, strides)) % VEC == 0)
    if st.dest.kind == 'tmp':
      # whole quads: rows past the end fall into the padding of the column
      emit(even and (not st.add or X % VEC == 0))
    elif even and X % VEC == 0:
      self.w('if ((reinterpret_cast<uintptr_t>(out) & 15u) == 0u) {')
      self.ind += 1
      emit(True)
      self.ind -= 1
      self.w('} else {')
      self.ind += 1
      emit(False)
      self.ind -= 1
      self.w('}')
    else:
      emit(False)


def emit_tiled(chain, plan, context, base_name, globals_):
  em = TiledEmitter(chain, plan, context, base_name)
  kernel = em.emit_kernel(globals_)
  args = []
  for t, _ in globals_:
    args.append(t.name)
    if t.addressing.name not in ('NONE', 'SCALAR'):
      args.append(f'{t.name}_extraOffset')
  args += ['numElements', 'flags']
  threads, smem = em.G * em.E, plan.smem_bytes
  kname = f'kernel_{base_name}'
  # one wave of resident CTAs walks the elements: shared operands are brought in once per CTA
  launch = {'kernel': kname, 'block': threads, 'elements_per_block': em.E, 'smem': smem, 'args': args,
            'pre': resident_grid(kname, threads, smem)}
  return kernel, launch
