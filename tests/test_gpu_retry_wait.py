"""2PL with eight or more transactions a warp: retries wait for the row that made
them abort once there are many of them, so a run takes clearly fewer attempts
than one whose retries always go at once (where few transactions starve the two
were the same)."""
import pytest

import gpu_cc_tb_b200 as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", ["tpl_nw", "tpl_wd"])
def test_dense_groups_wait(scheme):
    rows, n = 1_048_576, 65_536
    with g.Engine(rows) as eng:
        eng.load_txs(g.gen_ycsb(rows, n, 0.5, 0.9, seed=5))
        for wd in (0, 1, 2):
            def aborts(flags):
                return [eng.run(scheme, warp_density=wd, flags=flags)["aborts"] for _ in range(3)]
            assert max(aborts(0)) < 0.9 * min(aborts(g.F_RETRY_IMMEDIATE))
