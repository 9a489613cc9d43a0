"""Row blocks: the elements whose operands neighbouring threads read lie on different banks of
shared memory, and stay inside the CTA's shared memory."""
import pytest

from tests.test_rowblock_bounds import _shape


def _worst(slot, rg, te, width, active):
  """Most elements that meet on one bank in one transaction of a load of `width` values per lane."""
  lanes, worst = 32 // width, 0
  element = [t // (2 * rg) * 2 + (t & 1) for t in range(active)]
  for first in range(0, active, lanes):
    banks = {}
    for e in set(element[first:first + lanes]):
      if e < te:
        for x in range(width):
          banks.setdefault((e * slot + x) % 32, set()).add(e)
    worst = max([worst] + [len(b) for b in banks.values()])
  return worst


@pytest.mark.parametrize('terms', [1, 2, 3])
def test_elements_on_different_banks(terms):
  """At most two elements on a bank (eight for 12x40x12 products, 480 values per element, before)."""
  from tensorforge_b200.codegen.rowblock import layout, rowblock_params
  checked = 0
  for m in range(1, 129, 3 if terms > 1 else 1):
    for k in (1, 4, 7, 8, 12, 13, 16, 20, 24, 25, 31, 32, 40, 48, 56, 64, 84, 96, 128):
      for n in (1, 2, 3, 4, 6, 8, 9, 12, 16, 20, 27, 28):
        shape = _shape(m, k, n, terms, n * 3 if terms > 1 else 0)
        p = rowblock_params(shape, {})
        if p is None:
          continue
        rm, te = p[0]['rows'], p[0]['te']
        rg = -(-m // rm)
        off = layout(shape, rm, te)[2]
        active = -(-te // 2) * 2 * rg
        assert _worst(off['b'][1], rg, te, 2, active) <= 2, (m, k, n, p)
        if terms > 1 and p[0]['wcols'] == n:
          assert _worst(off['r0'][1], rg, te, 4, active) <= 2, (m, k, n, p)
        assert all(s % 4 == 0 for _, s in off.values())   # 16-byte copies
        checked += 1
  assert checked > 5_000
