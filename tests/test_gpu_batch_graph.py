"""A captured batched run (GCC_F_GRAPH) is replayed only while everything it
was captured with still holds: a call in between that replaces one of the
engine's buffers, or another ordered_after, makes a new capture. Integers:
bit-exact."""
import numpy as np
import pytest

import gpu_cc_tb_b200 as g

pytestmark = pytest.mark.gpu
SPIN = 2_000_000_000
BATCHES = np.array([0, 300, 1000], dtype=np.uint32)


def disjoint(n, seed):
    """Variable-length transactions without a common row: one result whatever the order."""
    rng = np.random.default_rng(seed)
    reqs = np.zeros(8 * n, dtype=g.REQ_DTYPE)
    reqs["key"] = rng.permutation(8 * n)
    reqs["read"] = rng.random(8 * n) < 0.6
    return np.arange(0, 8 * n + 1, 8, dtype=np.uint32), reqs


@pytest.mark.parametrize("scheme", ["tpl_nw", "mvcc", "slow_silo"])
def test_buffers_replaced_between_graph_runs(oracle, scheme):
    n, rows = 1000, 8000
    off, reqs = disjoint(n, 1)
    init = oracle.fill_table(rows, g.LAYOUT_U64X11, 3)
    more = g.gen_ycsb(rows, 5 * n, 0.1, 1.0, seed=2)  # reads only
    kw = dict(warp_density=4, block_size=8, flags=g.F_GRAPH, spin_limit_ns=SPIN)
    with g.Engine(rows, fill_seed=3, max_batch=512) as eng:
        eng.load_var_txs(off, reqs)
        for seed in (11, 12):
            want_t, want_dg = oracle.replay_var(init, g.LAYOUT_U64X11, off, reqs, np.arange(n),
                                                g.WRITE_FIELD, seed)
            for again in range(2):
                eng.upload_table(init)
                assert eng.run_batches(scheme, BATCHES, write_seed=seed, **kw)["committed"] == n
                assert np.array_equal(eng.digests(), want_dg)
                assert np.array_equal(eng.dump_table(), want_t)
                # larger per-transaction outputs, version store, read log
                eng.run_host("mvcc", more[: (1 + again) * 2 * n], spin_limit_ns=SPIN)
                # more time stamps
                eng.run_batches("tpl_nw", np.arange(0, n + 1, 10 // (1 + again)), spin_limit_ns=SPIN)


def test_ordered_after_makes_a_new_capture():
    """32 distinct keys of 20,000, half of them written, 256 transactions in
    flight: retries that never go one request at a time abort more than twice
    as often as ones that always do, so the number of aborts says which of the
    two a graph run did."""
    n, rows = 4000, 20000
    off, reqs = g.gen_ycsb_var(rows, n, 0.1, 0.5, min_ops=32, max_ops=32, seed=5)
    batches = np.array([0, n], dtype=np.uint32)
    with g.Engine(rows, fill_seed=3, max_batch=n) as eng:
        eng.load_var_txs(off, reqs)

        def aborts(after, flags):
            return [eng.run_batches("tpl_nw", batches, ordered_after=after, flags=flags,
                                    max_active=256, spin_limit_ns=SPIN)["aborts"]
                    for _ in range(3)]

        always, never = aborts(1, 0), aborts(1_000_000, 0)
        assert 1.5 * max(always) < min(never)
        middle = (max(always) * min(never)) ** 0.5
        for after in (1, 1_000_000, 1):
            assert all((a < middle) == (after == 1) for a in aborts(after, g.F_GRAPH))
