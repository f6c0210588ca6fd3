"""GaccO / GPUTx hand-off at the sizes where a row's list of accesses crosses
the tiles of the ordering passes: few rows with runs of reads longer than a
tile, runs of writes, repeated keys inside a transaction, empty transactions,
ragged batches. Bit-exact against the oracle's serial execution in the
scheme's order (integers: no tolerance)."""
import numpy as np
import pytest

import gpu_cc_tb_b200 as g

pytestmark = pytest.mark.gpu


def records(rows, n, read_ratio, seed):
    """Records of 0 to 16 requests with uniform keys (repeats allowed)."""
    rng = np.random.default_rng(seed)
    t = np.zeros(n, dtype=g.TX_DTYPE)
    t["request_cnt"] = rng.integers(0, 17, n)
    t["requests"]["key"] = np.sort(rng.integers(0, rows, (n, 16)), axis=1)
    t["requests"]["read"] = rng.random((n, 16)) < read_ratio
    return t


@pytest.mark.parametrize("write_mode", [g.WRITE_FIELD, g.WRITE_ROWCOPY])
@pytest.mark.parametrize("rows,n,read_ratio,wd,batch", [
    (1, 700, 1.0, 5, 700),       # one run of reads over several tiles
    (1, 400, 0.998, 5, 400),     # runs longer than a tile with a write between
    (1, 300, 0.0, 5, 129),       # writes only, ragged last batch
    (3, 640, 0.995, 4, 640),
    (70, 1025, 0.9, 5, 1024),    # a batch of one transaction at the end
    (70, 257, 0.5, 0, 257),      # all requests on one lane
    (5000, 65, 0.9, 3, 64),
])
@pytest.mark.parametrize("scheme", ["gacco", "gputx"])
def test_ordered_edges(oracle, scheme, rows, n, read_ratio, wd, batch, write_mode):
    txs = records(rows, n, read_ratio, 1000 * rows + n)
    init = oracle.fill_table(rows, g.LAYOUT_U64X11, 5)
    order = np.arange(n) if scheme == "gacco" else oracle.gputx_order(txs, rows)[1]
    ref_t, ref_dg, ref_rl = oracle.replay(init, g.LAYOUT_U64X11, txs, order, write_mode, 17,
                                          read_log=True)
    with g.Engine(rows, fill_seed=5, max_batch=batch) as eng:
        eng.load_txs(txs)
        res = eng.run(scheme, warp_density=wd, block_size=4, batch_size=batch,
                      flags=g.F_COMMIT_LOG | g.F_READ_LOG, write_mode=write_mode, write_seed=17,
                      spin_limit_ns=2_000_000_000)
        assert res["committed"] == n
        assert np.array_equal(eng.dump_table(), ref_t)
        assert np.array_equal(eng.digests(), ref_dg)
        assert np.array_equal(oracle.commit_order(eng.commit_log()), order)
        log = eng.read_log()
    live = (np.arange(16) < txs["request_cnt"][:, None]) & (txs["requests"]["read"] == 1)
    assert np.array_equal(log[live][:, :88], ref_rl[live][:, :88])
