"""Silo: pairs of transactions of which each reads what the other writes, without a
commit log (the log's own synchronisation comes exactly between the write locks
and the validation of the reads): every pair's digests and rows must be those of
one of its two serial orders. Integers: bit-exact."""
import numpy as np
import pytest

import gpu_cc_tb_b200 as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, g.F_QUEUE])
@pytest.mark.parametrize("wd", [0, 3, 4, 5])
def test_write_skew(oracle, wd, flags):
    pairs = 20_000
    rows = 16 * pairs
    rng = np.random.default_rng(wd)
    keys = rng.permutation(rows).astype(np.uint32).reshape(pairs, 16)
    t = np.zeros(2 * pairs, dtype=g.TX_DTYPE)
    t["request_cnt"] = 16
    t["requests"]["key"] = np.repeat(keys, 2, axis=0)
    first = rng.random((pairs, 16)) < 0.5  # what the pair's first transaction reads
    t["requests"]["read"][0::2] = first
    t["requests"]["read"][1::2] = ~first
    init = oracle.fill_table(rows, g.LAYOUT_U64X11, 3)
    ids = np.arange(2 * pairs)
    want = [oracle.replay(init, g.LAYOUT_U64X11, t, order, g.WRITE_FIELD, 7)[:2]
            for order in (ids, ids ^ 1)]
    with g.Engine(rows, fill_seed=3, max_batch=2 * pairs) as eng:
        eng.load_txs(t)
        for _ in range(5):
            eng.upload_table(init)
            eng.run("silo", warp_density=wd, flags=flags, write_seed=7,
                    spin_limit_ns=2_000_000_000)
            table, dg = eng.dump_table(), eng.digests()
            ok = np.zeros(pairs, dtype=bool)
            for ref_t, ref_dg in want:
                same = (table[keys] == ref_t[keys]).all(axis=(1, 2))
                ok |= same & (dg.reshape(-1, 2) == ref_dg.reshape(-1, 2)).all(axis=1)
            assert ok.all()
