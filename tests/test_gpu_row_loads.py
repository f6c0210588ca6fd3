"""The row loads of the transaction kernel: 32-byte loads where 88-byte rows lie
on 32-byte boundaries, 16-byte chunks otherwise (a caller's table may start on
any 16 bytes; 104-byte rows always), at every group size. Bit-exact against the
oracle: disjoint transactions, so every serial order gives the same result."""
import ctypes as C

import numpy as np
import pytest

import gpu_cc_tb_b200 as g

pytestmark = pytest.mark.gpu


def disjoint(n, seed):
    rng = np.random.default_rng(seed)
    t = np.zeros(n, dtype=g.TX_DTYPE)
    t["request_cnt"] = rng.integers(0, 17, n)
    t["requests"]["key"] = rng.permutation(16 * n).astype(np.uint32).reshape(n, 16)
    t["requests"]["read"] = rng.random((n, 16)) < 0.6
    return t


@pytest.mark.parametrize("offset", [0, 16, 32, 48])
def test_caller_table_on_any_16_bytes(oracle, offset):
    import torch

    n = 257
    rows = 16 * n
    txs, init = disjoint(n, offset), oracle.fill_table(rows, g.LAYOUT_U64X11, 3)
    ref_t, ref_dg, _ = oracle.replay(init, g.LAYOUT_U64X11, txs, None, g.WRITE_FIELD, 5)
    fn = g.library().gcc_run_tpl_nw_noalloc
    fn.restype = C.c_int
    fn.argtypes = [C.c_void_p, C.c_uint64, C.c_void_p, C.c_uint64, C.c_void_p, C.c_void_p,
                   C.c_uint64, C.c_void_p, C.POINTER(C.c_uint64), C.POINTER(C.c_uint64)]
    padded = np.zeros((rows, 96), dtype=np.uint8)
    padded[:, :88] = init
    table = torch.zeros(rows * 96 + 64, dtype=torch.uint8, device="cuda")
    table[offset:offset + rows * 96] = torch.from_numpy(padded.reshape(-1)).cuda()
    recs = torch.from_numpy(txs.view(np.uint8).copy()).cuda()
    dig = torch.zeros(n, dtype=torch.int64, device="cuda")
    ab = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert fn(recs.data_ptr(), n, table.data_ptr() + offset, rows, dig.data_ptr(), ab.data_ptr(), 5,
              None, None, None) == 0
    got = table[offset:offset + rows * 96].cpu().numpy().reshape(rows, 96)[:, :88]
    assert np.array_equal(got, ref_t)
    assert np.array_equal(dig.cpu().numpy().view(np.uint64), ref_dg)


@pytest.mark.parametrize("layout", [g.LAYOUT_U64X11, g.LAYOUT_REF104])
@pytest.mark.parametrize("wd", range(6))
@pytest.mark.parametrize("scheme", ["tpl_wd", "to", "mvcc", "silo", "tictoc", "gacco"])
def test_row_loads_by_group_size(oracle, scheme, wd, layout):
    n = 333
    rows = 16 * n
    txs, init = disjoint(n, wd), oracle.fill_table(rows, layout, 4)
    ref_t, ref_dg, ref_rl = oracle.replay(init, layout, txs, None, g.WRITE_ROWCOPY, 6, read_log=True)
    rb = g.row_bytes(layout)
    with g.Engine(rows, layout=layout, index=g.INDEX_SORTED, fill_seed=4, max_batch=n) as eng:
        eng.upload_table(init)
        eng.load_txs(txs)
        eng.run(scheme, warp_density=wd, block_size=2, batch_size=200, flags=g.F_READ_LOG,
                write_mode=g.WRITE_ROWCOPY, write_seed=6, spin_limit_ns=2_000_000_000)
        assert np.array_equal(eng.dump_table(), ref_t)
        assert np.array_equal(eng.digests(), ref_dg)
        log = eng.read_log()
    live = (np.arange(16) < txs["request_cnt"][:, None]) & (txs["requests"]["read"] == 1)
    assert np.array_equal(log[live][:, :rb], ref_rl[live][:, :rb])
