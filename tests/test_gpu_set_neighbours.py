"""Lists set right after a rebuild was queued (bcg_rebuild_neighbours returns before
it has run) are the ones that stay."""
import numpy as np
import pytest

from baccolonygrowth_b200 import params
from baccolonygrowth_b200.colony import Colony, packed_colony


@pytest.mark.gpu
def test_set_after_queued_rebuild(gpu):
    n = 60000
    p = params.ensemble_member(n)
    p.max_neighbours = 16
    params.finalize(p)
    col = Colony(p, packed_colony(n, *params.dome_size(n, 1.0 / 20.0, 0.9)))
    want = [np.array([(i + 1) % n], dtype=np.int32) for i in range(n)]
    for _ in range(5):
        for _ in range(4):
            col.rebuild_neighbours()
        col.set_neighbours(want)
        got = col.neighbours()
        assert all(len(g) == 1 and g[0] == w[0] for g, w in zip(got, want))
    col.close()
