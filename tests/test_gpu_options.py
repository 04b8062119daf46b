"""Options that name a default's own value mean the default."""
import pytest

import pumatch_b200 as pm
from pumatch_b200 import patterns as P

pytestmark = pytest.mark.gpu


def test_lane_subtree_max_64_is_the_default():
    """The default's scheme takes a seventh of the time of one candidate per lane here."""
    ctx = pm.Context(0)
    g = pm.GraphPreprocessor.from_host(pm.gen_rmat(16_384, 200_000, seed=3, device=0))
    p = pm.PatternPreprocessor(text=P.to_g(*P.clique(5)), labeled=False)

    def run(lane):
        runs = [ctx.match(g, [p], lane_subtree_max=lane, timeout_ms=60000) for _ in range(3)]
        return runs[0][0], runs[0][1]["set_ops"], min(st["kernel_ms"] for _, st in runs)

    default, named, other = run(0), run(64), run(63)
    assert default[:2] == named[:2] == other[:2]
    assert named[2] < 2 * default[2] < other[2]
    g.close()
    ctx.close()
