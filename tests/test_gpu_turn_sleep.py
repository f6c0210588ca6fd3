"""Waiters of the ordered schemes sleep by the writes ahead of them, not by the
accesses: the fewer writes a batch has, the shorter its chain. (With a sleep for
each access a batch at read ratio 0.99 took 0.46 of one at 0.9; by the writes
0.28.)"""
import pytest

import gpu_cc_tb_b200 as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", ["gacco", "gputx"])
def test_time_follows_the_writes(scheme):
    rows, n = 10_485_760, 65_536
    with g.Engine(rows) as eng:
        ms = []
        for ratio in (0.9, 0.99):
            eng.load_txs(g.gen_ycsb(rows, n, 0.8, ratio, seed=5))
            eng.run(scheme)
            ms.append(min(eng.run(scheme)["proc_s"] for _ in range(5)))
        assert ms[1] < 0.37 * ms[0]
