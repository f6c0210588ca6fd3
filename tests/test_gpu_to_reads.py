"""TO with several requests a lane: all reads of a pass share one fence between
their images and the raises of the rows' read timestamps, and come before the
lane's marks. Replay of the logged order on hot tables at every such group
size, with rows read and then written by one lane. Integers: bit-exact."""
import numpy as np
import pytest

import gpu_cc_tb_b200 as g

pytestmark = pytest.mark.gpu


def hot_records(rows, n, lanes, seed):
    """1 to 15 distinct ascending keys; with `lanes`, some transactions end by
    writing a row that the same lane read."""
    rng = np.random.default_rng(seed)
    t = np.zeros(n, dtype=g.TX_DTYPE)
    for i in range(n):
        c = int(rng.integers(1, min(15, rows) + 1))
        q = t[i]["requests"]
        q["key"][:c] = np.sort(rng.choice(rows, c, replace=False))
        q["read"][:c] = rng.random(c) < 0.7
        if lanes and c >= lanes and q["read"][c - lanes] and rng.random() < 0.5:
            q["key"][c] = q["key"][c - lanes]
            c += 1
        t[i]["request_cnt"] = c
    return t


@pytest.mark.parametrize("ordered_after", [0, 2])
@pytest.mark.parametrize("wd", [0, 1, 2, 3])
@pytest.mark.parametrize("rows,n,layout,write_mode", [
    (64, 1200, g.LAYOUT_U64X11, g.WRITE_FIELD),
    (400, 2000, g.LAYOUT_REF104, g.WRITE_ROWCOPY),
    (20_000, 4000, g.LAYOUT_U64X11, g.WRITE_FIELD),
])
def test_to_reads_together(oracle, rows, n, layout, write_mode, wd, ordered_after):
    txs = hot_records(rows, n, 0 if ordered_after else 1 << wd, rows + wd)
    init = oracle.fill_table(rows, layout, 9)
    with g.Engine(rows, layout=layout, index=g.INDEX_SORTED, fill_seed=9, max_batch=n) as eng:
        eng.upload_table(init)
        eng.load_txs(txs)
        res = eng.run("to", warp_density=wd, block_size=4, batch_size=1500, write_mode=write_mode,
                      write_seed=3, flags=g.F_COMMIT_LOG, spin_limit_ns=2_000_000_000,
                      max_active=1024, ordered_after=ordered_after)
        assert res["committed"] == n
        order = oracle.commit_order(eng.commit_log())
        ref_t, ref_dg, _ = oracle.replay(init, layout, txs, order, write_mode, 3)
        assert np.array_equal(eng.dump_table(), ref_t)
        assert np.array_equal(eng.digests(), ref_dg)
