"""Small CTAs keep an SM full: the transaction kernel's shared memory goes by the
launch's own threads and groups, so 32 CTAs of one warp (the hardware's limit,
and what 64 registers a thread allow) stay resident at every group size."""
import numpy as np
import pytest

import gpu_cc_tb_b200 as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wd", [2, 3, 5])
@pytest.mark.parametrize("block_size", [1, 2, 5, 32])
def test_resident_transactions(wd, block_size):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows, n = 100_000, 60_000
    off, reqs = g.gen_ycsb_var(rows, n, 0.1, 1.0, min_ops=4, max_ops=8, seed=3)  # reads only
    with g.Engine(rows, max_batch=n) as eng:
        eng.load_var_txs(off, reqs)
        res = eng.run_batches("tpl_nw", [0, n], warp_density=wd, block_size=block_size)
        assert res["committed"] == n
        ctas = 32 // block_size  # an SM holds 1,024 threads of 64 registers
        groups = ctas * sms * block_size * 32 >> wd
        assert eng.batch_active()[0] == min(groups, -(-n // (block_size * 32 >> wd)) * (block_size * 32 >> wd))


@pytest.mark.parametrize("scheme", ["tpl_nw", "tictoc", "gacco"])
@pytest.mark.parametrize("wd", range(6))
@pytest.mark.parametrize("block_size", [1, 3, 32])
def test_metrics_of_every_cta_size(oracle, scheme, wd, block_size):
    """The sums in that memory: every transaction is counted, and what is kept for
    a group is its own."""
    rows, n = 48_000, 3000
    rng = np.random.default_rng(wd)
    t = np.zeros(n, dtype=g.TX_DTYPE)
    t["request_cnt"] = 16
    t["requests"]["key"] = rng.permutation(rows).reshape(n, 16)
    t["requests"]["read"] = rng.random((n, 16)) < 0.5
    init = oracle.fill_table(rows, g.LAYOUT_U64X11, 3)
    ref_t, ref_dg, _ = oracle.replay(init, g.LAYOUT_U64X11, t, None, g.WRITE_FIELD, 5)
    with g.Engine(rows, fill_seed=3, max_batch=n) as eng:
        eng.load_txs(t)
        res = eng.run(scheme, warp_density=wd, block_size=block_size, batch_size=n, write_seed=5)
        assert res["committed"] == n and res["aborts"] == 0
        # (tot_d and its parts: ms a transaction)
        assert 0 < res["mng_d"] <= res["tot_d"] < 1e3 * res["tot_s"]
        assert 0 < res["idx_d"] < res["tot_d"]
        assert 0 < res["lat_p50_us"] <= res["lat_p99_us"] <= 1.1e6 * res["tot_s"]
        assert np.array_equal(eng.dump_table(), ref_t)
        assert np.array_equal(eng.digests(), ref_dg)
