"""MVCC reads its rows at once and then marks its writes at once: replay of the
logged order on hot tables (first attempts and one-at-a-time retries), at every
group size, with a row read and then written by one transaction; the opposite
request order of one row stays refused. Integers: bit-exact."""
import numpy as np
import pytest

import gpu_cc_tb_b200 as g

pytestmark = pytest.mark.gpu


def hot_records(rows, n, seed):
    """1 to 16 distinct ascending keys; some transactions end by writing the row
    that they read last."""
    rng = np.random.default_rng(seed)
    t = np.zeros(n, dtype=g.TX_DTYPE)
    for i in range(n):
        c = int(rng.integers(1, min(16, rows) + 1))
        t[i]["requests"]["key"][:c] = np.sort(rng.choice(rows, c, replace=False))
        t[i]["requests"]["read"][:c] = rng.random(c) < 0.6
        if c < 16 and t[i]["requests"]["read"][c - 1] and rng.random() < 0.3:
            t[i]["requests"]["key"][c] = t[i]["requests"]["key"][c - 1]
            c += 1
        t[i]["request_cnt"] = c
    return t


@pytest.mark.parametrize("scheme", ["mvcc", "slow_mvcc"])
@pytest.mark.parametrize("rows,n,wd,batch,write_mode", [
    (64, 2000, 5, 2000, g.WRITE_FIELD),
    (64, 500, 0, 500, g.WRITE_FIELD),
    (200, 1500, 3, 700, g.WRITE_ROWCOPY),
    (3, 300, 4, 300, g.WRITE_FIELD),
    (20_000, 4000, 5, 1024, g.WRITE_ROWCOPY),
])
def test_mvcc_phases(oracle, scheme, rows, n, wd, batch, write_mode):
    txs = hot_records(rows, n, rows + n)
    init = oracle.fill_table(rows, g.LAYOUT_U64X11, 9)
    with g.Engine(rows, fill_seed=9, max_batch=batch) as eng:
        eng.load_txs(txs)
        res = eng.run(scheme, warp_density=wd, block_size=8, batch_size=batch, write_mode=write_mode,
                      write_seed=3, flags=g.F_COMMIT_LOG, spin_limit_ns=2_000_000_000, max_active=512)
        assert res["committed"] == n
        order = oracle.commit_order(eng.commit_log())
        ref_t, ref_dg, _ = oracle.replay(init, g.LAYOUT_U64X11, txs, order, write_mode, 3)
        assert np.array_equal(eng.dump_table(), ref_t)
        assert np.array_equal(eng.digests(), ref_dg)


def test_mvcc_write_before_read_of_one_row():
    t = np.zeros(1, dtype=g.TX_DTYPE)
    t["request_cnt"] = 2
    t["requests"]["key"][0, :2] = 5
    t["requests"]["read"][0, :2] = (0, 1)
    with g.Engine(64) as eng:
        eng.load_txs(t)
        with pytest.raises(g.GccError) as err:
            eng.run("mvcc", spin_limit_ns=100_000_000)
        assert err.value.status == -4
