"""Held-out scores keep the network's own ranking apart from what the tuner tries."""
from types import SimpleNamespace as NS

import pytest


def _record(default, ms):
  variants = [{'strategy': 'tiled'}, {'strategy': 'generic'}, {'strategy': 'generic'}, {'strategy': 'colprog', 'a_source': 'const'}]
  cb = NS(feats=[[0.], [1.], [2.], [3.]], default=default, variants=variants, spec=NS(index=7))
  return cb, [{'ok': True, 'ms': m} for m in ms]


@pytest.mark.parametrize('default,top1,network', [(0, 0.0, 3.0), (1, 3.0, 3.0)])
def test_planners_untrained_plan_counts_for_the_tuner_only(default, top1, network):
  from tensorforge_b200.tune import heldout
  predict = lambda feats: [{0.: 4., 1.: 1., 2.: 2., 3.: 3.}[f[0]] for f in feats]    # the network ranks the tiled variant last
  row, = heldout.score([_record(default, [1.0, 4.0, 2.0, 3.0])], predict, k=2)
  assert (row['top1'], row['network_top1']) == (top1, network)
  assert row['network_top2'] == 1.0 and row['default'] == [0.0, 3.0][default]
  s = heldout.summary([row], k=2)
  assert s['network_top2']['mean'] == 1.0 and s['top1']['mean'] == top1 and s['chains'] == 1
