"""The engine's workloads as timed cases: what a program that uses
``gpu_cc_tb_b200`` has in hand (``prepare``), one pass of it through the public
entry points (``run``) and the work of that pass (``work``).

A case is a dict of plain values. ``kind`` names the calls:

  host      records in pinned host memory, gcc_run_host: copies in, batches and
            digest copies out in one call (a client that hands batches over)
  resident  records loaded once, gcc_run, then the read digests
  update    records loaded once (or handed over from the host), gcc_run, then a
            set of read-only transactions whose digests say what the table holds
  uneven    4-64-request transactions in batches of uneven sizes (one captured
            device-queue launch), then the same kind of read-back
  orders    order-entry transactions (extended integer ops) in batches, then a
            read-back
  learned   scheduled batches under heavy contention (predictor, deferral, lock
            plans, online training), then the lock plans that the updated
            frequency table gives
  predict   the contention predictor's forward pass over feature rows
  gradient  its forward and backward pass over a labelled minibatch

Which transaction of two conflicting ones commits first is decided by timing
in every scheme but gacco and gputx, so digests, abort counts and the values
of fields with several writers differ from run to run. Such a case returns
what it must have done whatever the order: the read-back's transactions read
rows that exactly one request of the pass wrote (and some that none did).
``host`` and ``resident`` cases return every digest: their scheme is
deterministic, or they only read, or they are small with hardly a conflict and
``prepare`` ends with a first pass, so that a read finds the same values before
and after the write that the pass repeats.
"""
import numpy as np
import torch

import gpu_cc_tb_b200 as g

SKETCH, N_IN, HID, STRIDE = 64, 66, 128, 72  # predictor: u16 features, 66-128-128-1
OE_W, OE_D, OE_C, OE_I = 64, 10, 3000, 100_000  # order-entry shape of the serving workload


def listed():
    plain = dict(rows=10_485_760, layout=0, index=0, rowcopy=False, queue=False, theta=0.6,
                 read_ratio=0.9, batch=65_536, wd=5, bs=32)
    return [
        # a small request batch from a client: latency, launches, per-call resets
        dict(plain, name="host_256", kind="host", scheme="tpl_nw", rows=1_048_576, tx=256,
             theta=0.1),
        # the configuration that the reference can run on its CPU path: low contention
        dict(plain, name="rows1m_low", kind="update", scheme="tpl_nw", rows=1_048_576, tx=65_536,
             theta=0.1),
        # the benchmark's default line, end to end from host memory (the largest)
        dict(plain, name="bench_tpl_nw", kind="update", scheme="tpl_nw", tx=1_048_576, host=True),
        # optimistic scheme through the device queue, as the benchmark runs it
        dict(plain, name="silo_queue", kind="update", scheme="silo", tx=1_048_576, queue=True),
        # multi-version reads, half reads half writes, last batch ragged
        dict(plain, name="mvcc_ragged", kind="update", scheme="mvcc", tx=100_003, read_ratio=0.5),
        # deterministic batch order, a hot table
        dict(plain, name="gacco_hot", kind="resident", scheme="gacco", tx=131_072, theta=0.8),
        # deterministic ranks in the reference's own format: 104-byte rows, sorted
        # index, whole-row copies, smaller groups and blocks
        dict(plain, name="gputx_ref_format", kind="resident", scheme="gputx", tx=65_537, layout=1,
             index=1, rowcopy=True, wd=4, bs=8),
        # consecutive uneven batches, 4-64 requests each, one persistent launch
        dict(plain, name="uneven_tictoc", kind="uneven", scheme="tictoc", tx=120_000, batches=24,
             theta=0.8, max_active=1184),
        # order entry: new orders and payments over 64 warehouses
        dict(plain, name="orders_tpl_wd", kind="orders", scheme="tpl_wd", tx=100_000, batch=16_384),
        # learned scheduling at the highest contention
        dict(plain, name="learned_hot", kind="learned", scheme="tpl_nw", tx=131_072, theta=0.99),
        # the predictor over one batch of transactions
        dict(name="predict_65536", kind="predict", tx=65_536),
        # one default minibatch forward and backward
        dict(name="gradient_4096", kind="gradient", tx=4096),
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, even over its logarithm."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["host", "host", "resident", "resident", "update", "update", "update", "uneven",
                       "orders", "learned", "predict", "gradient"])
    if kind in ("predict", "gradient"):
        return dict(kind=kind, tx=_log(rng, 1000, 100_000 if kind == "predict" else 20_000))
    c = dict(kind=kind, rows=_log(rng, 500_000, 10_485_760), layout=rng.choice([0, 0, 0, 1]),
             index=rng.choice([0, 0, 1, 2]), rowcopy=rng.random() < 0.25, queue=False,
             theta=round(rng.uniform(0.3, 0.7), 2), read_ratio=rng.choice([0.9, 0.95, 0.8, 0.5]),
             batch=rng.choice([65_536, 65_536, 16_384, 30_000]), wd=rng.choice([5, 5, 4, 3]),
             bs=rng.choice([32, 32, 16, 8]))
    if kind == "host":
        c.update(tx=_log(rng, 1, 4096), rows=_log(rng, 1_048_576, 10_485_760),
                 scheme=rng.choice(["tpl_nw", "tpl_wd", "to", "silo", "tictoc", "gacco"]))
        if c["scheme"] != "gacco":  # hardly a conflict, or reads only
            c.update(theta=0.1, read_ratio=1.0 if c["tx"] > 500 else max(0.9, c["read_ratio"]))
    elif kind == "resident":
        c["scheme"] = rng.choice(["gacco", "gputx", "tpl_nw", "silo", "to", "mvcc"])
        c["tx"] = _log(rng, 5000, 200_000)
        if c["scheme"] not in ("gacco", "gputx"):
            c["read_ratio"] = 1.0
    elif kind == "update":
        c["scheme"] = rng.choice(["tpl_nw", "tpl_wd", "to", "mvcc", "silo", "tictoc", "slow_silo",
                                  "slow_tpl_nw"])
        c["tx"] = _log(rng, 5000, 40_000 if c["scheme"].startswith("slow") else
                       80_000 if c["scheme"] == "mvcc" else 300_000)
        c["theta"] = rng.choice([0.1, c["theta"], c["theta"]])
        c["rows"] = _log(rng, 1_000_000 if c["theta"] < 0.2 else 4_000_000, 10_485_760)
        c["queue"] = c["scheme"] in ("silo", "tictoc") and rng.random() < 0.5
        if c["read_ratio"] < 0.8:
            c["theta"] = min(c["theta"], 0.6)
    elif kind == "uneven":
        c.update(scheme=rng.choice(["tictoc", "silo", "tpl_nw"]), tx=_log(rng, 5000, 60_000),
                 batches=rng.randint(2, 12), layout=0, rows=_log(rng, 4_000_000, 10_485_760),
                 max_active=rng.choice([592, 1184]), wd=5, bs=32, read_ratio=0.9)
    elif kind == "orders":
        c.update(scheme=rng.choice(["tpl_nw", "tpl_wd", "silo", "tictoc"]), tx=_log(rng, 5000, 100_000),
                 layout=0, wd=5, bs=32)
    else:
        c.update(scheme=rng.choice(["tpl_nw", "silo"]), tx=_log(rng, 10_000, 131_072),
                 theta=round(rng.uniform(0.8, 0.99), 2), read_ratio=0.9, layout=0, wd=5, bs=32,
                 batch=65_536, rows=10_485_760)
    # whole-row copies carry one different read through many rows, so only the
    # deterministic schemes give the same table twice
    c["rowcopy"] = c["rowcopy"] and c["scheme"] in ("gacco", "gputx")
    return c


class State:
    """What a program keeps between passes; the scheduler goes before its engine."""

    eng = sched = None

    def __del__(self):
        if self.sched is not None:
            self.sched.close()
        if self.eng is not None:
            self.eng.close()


def _pinned(a):
    t = torch.empty(max(1, a.nbytes), dtype=torch.uint8, pin_memory=True)
    v = t.numpy()[: a.nbytes].view(a.dtype).reshape(a.shape)
    v[...] = a
    return v


def _records(case, seed):
    """gen_ycsb records; the reference's format has its dropped repeats and keys from 1."""
    ref = case["layout"] == 1
    return g.gen_ycsb(case["rows"], case["tx"], case["theta"], case["read_ratio"], seed=seed,
                      dedup=g.DEDUP_DROP if ref else g.DEDUP_RESAMPLE, key_base=1 if ref else 0)


def _probes(case):
    return max(256, min(4096, case["tx"] // 64))


def _read_back(case, rows, keys, writes, seed):
    """Requests of the read-back: 16 distinct rows a transaction, half of them
    (where there are enough) written by exactly one of the requests `keys` /
    `writes`, the others by none."""
    n, rng = 16 * _probes(case), np.random.default_rng(seed)
    count = np.bincount(keys[writes], minlength=rows)
    once = rng.permutation(np.flatnonzero(count == 1))[: n // 2]
    never = np.unique(rng.integers(1, rows, 4 * n))
    never = rng.permutation(never[count[never] == 0])[: n - len(once)]
    r = np.zeros(n, dtype=g.REQ_DTYPE)
    r["read"], r["key"] = 1, rng.permutation(np.concatenate([once, never]))
    return r


def _features(rng, n):
    """Feature rows of n 16-request transactions: sketch counts, writes, hot-key sum."""
    f = np.zeros((n, STRIDE), dtype=np.uint16)
    bins = rng.integers(0, SKETCH, (n, 16))
    np.add.at(f, (np.repeat(np.arange(n), 16), bins.ravel()), 1)
    f[:, 64] = rng.binomial(16, 0.1, n)
    f[:, 65] = np.minimum(16 * 16, rng.gamma(4.0, 8.0, n)).astype(np.uint16)
    return f


def _network(case, seed):
    """Features, labels and He-uniform weights, from the seed alone."""
    rng = np.random.default_rng(seed)
    f = _features(rng, case["tx"])
    hot = f[:, 65].astype(np.float64) + 4.0 * f[:, 64] + rng.normal(0.0, 6.0, len(f))
    y = (hot > 40.0).astype(np.uint8)
    parts = []
    for fan, shape in ((N_IN, (N_IN, HID)), (0, (HID,)), (HID, (HID, HID)), (0, (HID,)),
                       (2 * HID, (HID,)), (0, (1,))):
        a = np.sqrt(6.0 / fan) if fan else 0.05
        parts.append(rng.uniform(-a, a, shape).astype(np.float32).ravel())
    return f, y, np.concatenate(parts)


def prepare(case, seed):
    s = State()
    s.case, kind = case, case["kind"]
    if kind in ("predict", "gradient"):
        s.feat, s.labels, w = _network(case, seed)
        s.eng = g.Engine(4096)
        s.sched = g.Scheduler(s.eng, minibatch=4096, seed=1)
        s.sched.set_weights(w)
        return s
    s.knobs = dict(warp_density=case["wd"], block_size=case["bs"], batch_size=case["batch"],
                   write_seed=seed + 1)
    if kind == "orders":
        s.desc = g.order_entry_desc(OE_W, OE_D, OE_C, OE_I)
        off, reqs, _, lay = g.gen_order_entry(s.desc, case["tx"], seed=seed)
        s.rows = lay["rows"]
    else:
        s.rows = case["rows"]
    s.eng = g.Engine(s.rows, layout=case["layout"], index=case["index"] if kind != "orders" else 2,
                     fill_seed=seed + 2, max_batch=case["batch"])
    if kind in ("host", "resident", "update"):
        s.knobs["write_mode"] = g.WRITE_ROWCOPY if case["rowcopy"] else g.WRITE_FIELD
        s.knobs["flags"] = g.F_QUEUE if case["queue"] else 0
        txs = _records(case, seed)
        s.host = kind == "host" or case.get("host", False)
        if s.host:
            s.txs, s.digests = _pinned(txs), _pinned(np.zeros(len(txs), np.uint64))
        else:
            s.eng.load_txs(txs)
        if kind == "update":
            q = txs["requests"][np.arange(16) < txs["request_cnt"][:, None]]
            back = _read_back(case, s.rows, q["key"], q["read"] == 0, seed + 3)
            s.eng.load_var_txs(np.arange(0, len(back) + 1, 16), back)
        else:
            _pass(s)
    elif kind == "learned":
        s.eng.load_txs(_records(case, seed))
        s.sched = g.Scheduler(s.eng, seed=seed % 1000 + 1)
        s.knobs["write_mode"] = g.WRITE_FIELD
    else:  # uneven, orders: read-back with 16-request records from the host
        s.knobs["flags"] = g.F_GRAPH
        n = case["tx"]
        if kind == "uneven":
            off, reqs = g.gen_ycsb_var(s.rows, n, case["theta"], case["read_ratio"], 4, 64, seed=seed)
            s.mode, s.knobs["max_active"] = g.BATCHES_QUEUE, case["max_active"]
            size = np.exp(np.random.default_rng(seed).uniform(0.0, np.log(64.0), case["batches"]))
            cut = np.round(np.cumsum(size) / size.sum() * (n - case["batches"])).astype(np.int64)
            s.batches = np.concatenate([[0], cut + np.arange(1, case["batches"] + 1)]).astype(np.uint32)
        else:
            s.eng.oe_fill(s.desc, seed + 2)
            s.knobs["flags"] |= g.F_EXT_OPS
            s.mode = g.BATCHES_SEQUENTIAL
            s.batches = np.append(np.arange(0, n, case["batch"]), n).astype(np.uint32)
        s.eng.load_var_txs(off, reqs)
        s.txs = np.zeros(_probes(case), dtype=g.TX_DTYPE)
        s.txs["request_cnt"] = 16
        s.txs["requests"] = _read_back(case, s.rows, reqs["key"], reqs["read"] != 1,
                                       seed + 3).reshape(-1, 16)
        s.txs = _pinned(s.txs)
        s.digests = _pinned(np.zeros(len(s.txs), np.uint64))
    return s


def _pass(s):
    if s.host:
        s.eng.run_host(s.case["scheme"], s.txs, s.digests, **s.knobs)
        return s.digests
    s.eng.run(s.case["scheme"], **s.knobs)
    return s.eng.digests()


def run(s):
    kind, scheme = s.case["kind"], s.case.get("scheme")
    if kind == "predict":
        return s.sched.predict(s.feat)
    if kind == "gradient":
        grad, loss = s.sched.gradient(s.feat, s.labels)
        return {"grad": grad, "loss": loss}
    if kind in ("host", "resident"):
        return {"digests": _pass(s)}
    if kind == "learned":
        r = s.sched.run(scheme, **s.knobs)
        return {"committed": r["committed"],
                "lock_plans": s.sched.lock_plans(0, min(s.case["tx"], s.case["batch"]))}
    if kind == "update":
        if s.host:
            r = s.eng.run_host(scheme, s.txs, s.digests, **s.knobs)
        else:
            r = s.eng.run(scheme, **s.knobs)
        s.eng.run_batches("tpl_nw", [0, _probes(s.case)])
    else:
        r = s.eng.run_batches(scheme, s.batches, s.mode, **s.knobs)
        s.eng.run_host("tpl_nw", s.txs, s.digests)
        return {"committed": r["committed"], "table": s.digests}
    return {"committed": r["committed"], "table": s.eng.digests()}


def _distinct(rows, theta, n):
    """Expected number of distinct rows among n Zipf(theta) draws over `rows` keys."""
    edge = np.unique(np.round(np.geomspace(1, rows + 1, 4000)))
    mid, width = np.sqrt(edge[:-1] * (edge[1:] - 1)), np.diff(edge)
    p = mid ** -theta
    p /= (p * width).sum()
    return float((width * -np.expm1(n * np.log1p(-np.minimum(p, 0.5)))).sum())


def work(case):
    n = case["tx"]
    if case["kind"] in ("predict", "gradient"):
        mults = N_IN * HID + HID * HID + HID
        par = 4 * (N_IN * HID + HID + HID * HID + HID + HID + 1)
        if case["kind"] == "predict":
            return {"bytes": n * (2 * N_IN + 4) + par / 2, "flops": 2.0 * n * mults}
        return {"bytes": n * (2 * N_IN + 1) + 1.5 * par, "flops": 2.0 * n * (2 * mults + HID * HID + HID)}
    row = g.row_bytes(case["layout"])
    if case["kind"] == "orders":  # half new orders (34 requests on average), half payments (4)
        ops, reads, writes = 19.0, 6.5, 12.5
        rows, theta = OE_W * (1 + OE_D * (1 + OE_C) + OE_I) + OE_I, 0.1
    else:
        ops = 34.0 if case["kind"] == "uneven" else 16.0
        reads, writes = ops * case["read_ratio"], ops * (1.0 - case["read_ratio"])
        rows, theta = case["rows"], case["theta"]
    # records in, rows read (each distinct one once), fields or rows written, digests out
    put = row if case.get("rowcopy") else 8
    b = n * (8 + 8 * ops + 8) + row * _distinct(rows, theta, n * reads) + put * _distinct(
        rows * (1 if case.get("rowcopy") else 10), theta, n * writes)
    if case["kind"] not in ("host", "resident", "learned"):
        b += _probes(case) * (16 * (8 + row) + 16)
    # a 64-bit mix of every word read (about 8 operations each)
    return {"bytes": b, "flops": n * reads * row / 8 * 8.0}


def exact(case, seed):
    if case["kind"] not in ("predict", "gradient"):
        return None
    f, y, w = _network(case, seed)
    w = torch.from_numpy(w).to(torch.bfloat16).to(torch.float64).numpy()
    cut = np.cumsum([N_IN * HID, HID, HID * HID, HID, HID])
    w1, b1, w2, b2, w3, b3 = np.split(w, cut)
    w1, w2 = w1.reshape(N_IN, HID), w2.reshape(HID, HID)
    x = f[:, :N_IN].astype(np.float64) / 16.0
    h1 = np.maximum(x @ w1 + b1, 0.0)
    h2 = np.maximum(h1 @ w2 + b2, 0.0)
    z = h2 @ w3 + b3
    p = 1.0 / (1.0 + np.exp(-z))
    if case["kind"] == "predict":
        return p
    loss = np.mean(np.maximum(z, 0.0) + np.log1p(np.exp(-np.abs(z))) - y * z)
    dz = (p - y) / len(y)
    d2 = dz[:, None] * w3 * (h2 > 0.0)
    d1 = (d2 @ w2.T) * (h1 > 0.0)
    grad = np.concatenate([(x.T @ d1).ravel(), d1.sum(0), (h1.T @ d2).ravel(), d2.sum(0), h2.T @ dz,
                           [dz.sum()]])
    return {"grad": grad, "loss": loss}
