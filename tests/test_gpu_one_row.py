"""The ordering pass over a row that every transaction reads: its time stays with
that of a uniform list of the same length (looking back over the accesses one
tile at a time took fifty times as long), and the result is the same as ever."""
import numpy as np
import pytest

import gpu_cc_tb_b200 as g

pytestmark = pytest.mark.gpu


def test_ordering_pass_over_one_row(oracle):
    rows, n = 200_000, 262_144
    t = np.zeros(n, dtype=g.TX_DTYPE)
    t["request_cnt"] = 16
    t["requests"]["read"] = 1
    rng = np.random.default_rng(3)
    with g.Engine(rows, fill_seed=5, max_batch=n) as eng:
        pre = []
        for keys in (rng.integers(0, rows, (n, 16)), np.full((n, 16), 77)):
            t["requests"]["key"] = keys
            eng.load_txs(t)
            eng.run("gacco", batch_size=n)
            pre.append(min(eng.run("gacco", batch_size=n)["pre_s"] for _ in range(3)))
        init = oracle.fill_table(rows, g.LAYOUT_U64X11, 5)
        _, ref_dg, _ = oracle.replay(init, g.LAYOUT_U64X11, t, None, g.WRITE_FIELD, 1)
        assert np.array_equal(eng.digests(), ref_dg)
    assert pre[1] < 2 * pre[0]
