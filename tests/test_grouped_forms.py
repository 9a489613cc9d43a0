"""Mixed-shape launches: which form each group's tile takes, by the density of its shared operands."""
import numpy as np
import pytest

from oracle import cases

MM, ID = [[0, -1], [-1, 1]], [[0, 1], [0, 1]]


def chain(ns, b, q, density, terms=3):
  S, sub = ns.Addressing.STRIDED, ns.SubTensor
  B, out, descrs = ns.Tensor([b, q], S), ns.Tensor([b, q], S), []
  for t in range(terms):
    pattern = cases.sparse_pattern(b, b, density, b + q + t)
    A = ns.Tensor([b, b], ns.Addressing.NONE, spp=ns.ListSPP(pattern, (b, b)))
    R = ns.Tensor([q, q], S, spp=ns.ListSPP(cases.sparse_pattern(q, q, 0.3, t), (q, q)))
    T = ns.generate_tmp_tensor([sub(A), sub(B)], MM)
    descrs += [ns.MultilinearDescr(sub(T), [sub(A), sub(B)], MM, ID), ns.MultilinearDescr(sub(out), [sub(T), sub(R)], MM, ID, add=t > 0)]
  return descrs


def grouped(shapes, **kw):
  from tensorforge_b200.grouped import GroupedKernel
  from tensorforge_b200.kernels import Context, FP, Generator, Options
  ns = cases.ns_from_module('tensorforge_b200')
  return GroupedKernel([Generator(chain(ns, *s), Context('sm_100a', 'cuda', FP['float'], Options())) for s in shapes], **kw)


def forms(gk):
  out = []
  for part in gk.source().split('// generated by tensorforge_b200 (strategy: colprog, ')[1:]:
    head = part[:part.index('\n')]
    out.append('blocks' if 'row blocks' in head else 'tiles' if 'outputs per' in head else 'unrolled')
  return out


@pytest.mark.parametrize('shape,form', [
  ((10, 9, 0.1), 'blocks'), ((20, 27, 0.05), 'blocks'), ((35, 27, 0.1), 'blocks'), ((56, 9, 0.1), 'unrolled'), ((84, 9, 0.15), 'unrolled'),
  ((56, 9, 0.45), 'blocks'), ((84, 27, 0.1), 'unrolled'), ((84, 27, 0.45), 'blocks'), ((56, 27, 0.1), 'unrolled'), ((56, 32, 0.1), 'unrolled'),
  ((35, 32, 0.45), 'unrolled'), ((56, 32, 0.5), 'tiles'), ((20, 32, 0.9), 'tiles')])
def test_form_of_a_group(shape, form):
  assert forms(grouped([shape])) == [form]


def test_where_the_unrolled_program_does_not_fit():
  """100x40 at 28 %: A, B and the R factors of a tile and U take an unrolled program with 256 threads
  past 227 KB, so that the group loops although that is the slower form."""
  from tensorforge_b200.grouped import loops_pay
  from tensorforge_b200.plan import Plan
  from tensorforge_b200.plan.chains import match_left_chain
  from tensorforge_b200.codegen.colprog import _ColProg
  gk = grouped([(100, 40, 0.28), (10, 9, 0.45)])
  g = gk.gens[0]
  shape = match_left_chain(g.get_chain())
  u = _ColProg(g.get_chain(), shape, Plan('colprog', {'threads': 256, 'chunk': 16, 'a_source': 'smem', 'prefetch': 1}), g.get_context(), 'x')
  u._layout()
  assert u.smem > 227 * 1024 and not loops_pay(shape, False)
  assert forms(gk) == ['tiles', 'blocks'] and gk.smem <= 227 * 1024


MIX = [(56, 9, 0.1), (20, 27, 0.1), (56, 32, 0.5), (35, 32, 0.2), (10, 9, 0.45)]


def sources():
  return [grouped(MIX).source()]


@pytest.mark.gpu
def test_all_forms_in_one_launch_match_oracle():
  """1e-6 relative L2 norm against the FP64 oracle, as for the groups alone."""
  import torch
  from oracle import harness, multilinear
  from tensorforge_b200.grouped import launch_noalloc
  gk = grouped(MIX)
  assert sorted(set(forms(gk))) == ['blocks', 'tiles', 'unrolled']
  for noalloc in (False, True):
    sets, mems = [], []
    for gid, g in enumerate(gk.gens):
      n = (301, 0, 97, 555, 1203)[gid]
      lay, mem = harness.make_memory(g.descr_list, max(n, 1), seed=gid)
      flags = harness.make_flags(max(n, 1), gid) if gid % 2 == 0 else None
      kw = {'numElements': n, 'flags': None if flags is None else torch.tensor(flags.astype(np.int32), device='cuda')}
      for l in lay:
        kw[l.name] = torch.tensor(mem.buffers[l.name], dtype=torch.float32, device='cuda')
        if l.kind == 'strided':
          kw[f'{l.name}_extraOffset'] = l.extra_offset
      sets.append(kw)
      mems.append((lay, mem, flags, n))
    if noalloc:
      launch_noalloc(gk, sets)
    else:
      gk.prepare(sets).launch()
    torch.cuda.synchronize()
    for g, kw, (lay, mem, flags, n) in zip(gk.gens, sets, mems):
      if n:
        multilinear.evaluate(g.descr_list, mem, n, flags=flags)
      for l in lay:
        got, ref = kw[l.name].double().cpu().numpy(), mem.buffers[l.name]
        assert np.linalg.norm(got - ref) <= 1e-6 * np.linalg.norm(ref), (g.get_base_name(), l.name)
