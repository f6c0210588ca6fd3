"""MVCC readers that walk a row's version chain while writers link newer versions
to it: half the transactions write few hot rows, the others only read them.
Replay of the logged order. Integers: bit-exact."""
import numpy as np
import pytest

import gpu_cc_tb_b200 as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wd", range(6))
@pytest.mark.parametrize("rows,n,write_mode", [
    (24, 1500, g.WRITE_FIELD),
    (40, 1500, g.WRITE_ROWCOPY),
    (600, 6000, g.WRITE_FIELD),
])
def test_chain_under_writers(oracle, rows, n, write_mode, wd):
    rng = np.random.default_rng(rows + wd)
    t = np.zeros(n, dtype=g.TX_DTYPE)
    t["request_cnt"] = np.where(np.arange(n) % 2, 16, 3)
    t["requests"]["key"] = np.argsort(rng.random((n, rows)), axis=1)[:, :16]
    t["requests"]["read"] = (np.arange(n) % 2)[:, None] | (np.arange(16) == 0)
    init = oracle.fill_table(rows, g.LAYOUT_U64X11, 9)
    with g.Engine(rows, fill_seed=9, max_batch=n) as eng:
        eng.load_txs(t)
        res = eng.run("mvcc", warp_density=wd, block_size=8, batch_size=1000, write_mode=write_mode,
                      write_seed=3, flags=g.F_COMMIT_LOG, spin_limit_ns=2_000_000_000, max_active=512)
        assert res["committed"] == n
        order = oracle.commit_order(eng.commit_log())
        ref_t, ref_dg, _ = oracle.replay(init, g.LAYOUT_U64X11, t, order, write_mode, 3)
        assert np.array_equal(eng.dump_table(), ref_t)
        assert np.array_equal(eng.digests(), ref_dg)
