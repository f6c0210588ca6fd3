// cc_kernel.cuh -- the YCSB transaction kernel under each concurrency-control
// scheme, written for sm_100a.
//
// Reference behaviour followed (gCCTB paths):
//   transaction loop + retry          benchmark/ycsb.cu:21-111
//   2PL no-wait / wait-die             include/twopl.cuh:59-382
//   timestamp ordering                 include/to.cuh:57-271
//   MVCC                               include/mvcc.cuh:61-297
//   Silo                               include/silo.cuh:70-339
//   TicToc                             include/tictoc.cuh:67-369
//   GaccO ordered hand-off             include/gacco.cuh:49-176
//   GPUTx rank execution               include/gputx.cuh:58-146
//   latch ("slow_") variants           include/slow_*.cuh, runtime.cuh:91-109
//
// B200 design (not a translation of the reference):
//   * persistent CTAs; a group of G = 2^warp_density lanes owns one
//     transaction at a time and takes the next from an ordered ticket;
//   * the G lanes split the transaction's requests: op i belongs to lane
//     i % G, so index probes, lock/timestamp operations and row copies of
//     different requests are in flight together (the reference runs them one
//     by one on lane 0); group-wide decisions are ballots;
//   * rows move with 16-byte L2 loads/stores (rows are 16-byte aligned);
//   * every wait is bounded by `spin_limit_ns` of %globaltimer and raises
//     GCC_ETIMEOUT instead of hanging.
//
// Commit rules are the reference's. Differences that fix reference bugs are
// listed where they occur (Silo commit timestamp, MVCC base-row update and
// version-store stride, GPUTx same-rank conflicts).
#pragma once
#include <cooperative_groups.h>
#include <type_traits>
#include "gcc_common.cuh"

namespace gcc {

namespace cg = cooperative_groups;


enum Scheme : int {
    S_TPL_NW = 0, S_TPL_WD, S_TO, S_MVCC, S_SILO, S_TICTOC, S_GACCO, S_GPUTX,
    S_SLOW_TPL_NW, S_SLOW_TPL_WD, S_SLOW_TO, S_SLOW_MVCC, S_SLOW_SILO,
    S_SLOW_TICTOC, S_COUNT
};

enum AttemptStatus : int { kCommit = 0, kAbort = 1, kGiveUp = 2 };

// Where a bounded wait gave up (Counters::err_where).
enum WaitSite : unsigned {
    W_LATCH = 1, W_TPL_WD, W_TO_READ, W_MVCC_READ, W_SILO_READ, W_TICTOC_READ,
    W_TICTOC_EXT, W_TURN, W_RETRY, W_QUEUE = 11, W_STARVE
};

// ---------------------------------------------------------------------------
// A group of G lanes of one warp working on one transaction.
// ---------------------------------------------------------------------------
template <int G>
struct Group {
    unsigned mask;  // lanes of this group within the warp
    int base;       // first lane of the group
    int glane;      // lane within the group
    GCC_D Group() {
        int lane = threadIdx.x & 31;
        base = lane & ~(G - 1);
        glane = lane & (G - 1);
        mask = (G == 32) ? 0xFFFFFFFFu : (((1u << G) - 1u) << base);
    }
    GCC_D bool any(bool p) const { return __any_sync(mask, p); }
    GCC_D void sync() const { __syncwarp(mask); }
    template <class T>
    GCC_D T bcast(T v, int src) const { return __shfl_sync(mask, v, src, G); }
    GCC_D unsigned long long sum(unsigned long long v) const {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o, G);
        return v;
    }
    GCC_D unsigned long long maxv(unsigned long long v) const {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) {
            unsigned long long u = __shfl_xor_sync(mask, v, o, G);
            v = u > v ? u : v;
        }
        return v;
    }
    GCC_D uint32_t orv(uint32_t v) const { return __reduce_or_sync(mask, v); }
    GCC_D unsigned long long orv(unsigned long long v) const {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) v |= __shfl_xor_sync(mask, v, o, G);
        return v;
    }
};

// Per-transaction lane state: lane owns ops i = glane + k*G, k < K, of a
// transaction of at most MO requests.
template <int G_, int MO>
struct TxOps {
    static constexpr int G = G_;
    static constexpr int MAXOPS = MO;
    static constexpr int K = (MO + G - 1) / G;
    static constexpr bool kExt = MO > kMaxOps;  // extended ops (var-length only)
    uint32_t n;                // requests in the transaction
    uint32_t valid;            // bit k: op k exists
    uint32_t isread;           // bit k: op k reads
    using Mask = std::conditional_t<(MO > 32), unsigned long long, uint32_t>;
    Mask readmask;             // group-wide: bit i set if op i reads
    uint32_t row[K];
    // one request a lane: the field and value its write stores (FIELD mode),
    // computed before the attempt so that no row is held for it
    uint32_t wfield;
    unsigned long long wval;
    // 1 + the request that failed in the last aborted 2PL / TO attempt (0:
    // none); the next one-at-a-time attempt visits it after the others
    // (unless GCC_F_REQUEST_ORDER)
    mutable uint32_t obst_op;
    uint32_t turn_ns;   // ordered schemes: sleep for each access ahead
    uint32_t attempts;  // aborted ones so far
    bool crowded;       // many starving transactions at the last abort (see await_row)
};

// Bounded wait helper: true once `limit` ns have passed since `t0`.
GCC_D bool expired(uint64_t t0, uint64_t limit) { return gtimer() - t0 > limit; }
// Pause inside a wait loop so that diverged lanes of the same warp (another
// transaction's group, possibly the one being waited for) get issue slots.
GCC_D void wait_pause() { __nanosleep(20); }

// ---------------------------------------------------------------------------
// Row images: digest, read log, rowcopy scratch, writes.
// ---------------------------------------------------------------------------
constexpr int kMaxChunks = 7;  // 16-byte chunks cover up to 14 words (112 B)

GCC_D size_t slot_of(const KParams &p, uint64_t unit, uint32_t i) {
    return ((size_t)unit * p.slot_ops + i) * p.wslot;
}
// Read a row image from `src` (L2 loads), folding its words into the digest
// term `dt` of op i and copying it to the rowcopy scratch slot and the read
// log when those exist. Where a lane has one or two requests (K), loads of an
// image are issued together before the first is used: chunk by chunk each
// one's L2 round trip came after the one before. Rows of 11 words on 32-byte
// boundaries (the u64 layout) are three 32-byte loads, i.e. one L2 request per
// sector; others move in 16-byte chunks, four together with one request a
// lane. Lanes with more requests have no registers left for that (64 with
// 1,024-thread CTAs) and go chunk by chunk. Measured: see ycsb_kernel.
template <int K>
GCC_D void read_image(const KParams &p, const uint64_t *src, uint32_t tx, uint64_t pos,
                      uint32_t i, unsigned long long &dt) {
    ulonglong2 *sc = p.scratch ? (ulonglong2 *)(p.scratch + slot_of(p, pos, i)) : nullptr;
    ulonglong2 *lg = p.read_log ? (ulonglong2 *)(p.read_log + slot_of(p, tx, i)) : nullptr;
    auto keep = [&](int c, unsigned long long x, unsigned long long y) {
        if (sc) __stcg(sc + c, make_ulonglong2(x, y));
        if (lg) __stcg(lg + c, make_ulonglong2(x, y));
    };
    // the digest's terms, each word's tag counted up
    unsigned long long tag = (unsigned long long)(i * 16u + 1u) * kDigestStep;
    auto fold = [&](unsigned long long w) {
        dt += splitmix64(w ^ tag);
        tag += kDigestStep;
    };
    if (K <= 2 && p.wide) {
        Sector s[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) s[c] = ld_cg32(src + 4 * c);
#pragma unroll
        for (int k = 0; k < 11; ++k) fold(s[k / 4].w[k % 4]);
        if (sc || lg) {
#pragma unroll
            for (int c = 0; c < 6; ++c) keep(c, s[c / 2].w[c % 2 * 2], s[c / 2].w[c % 2 * 2 + 1]);
        }
        return;
    }
    constexpr int kTogether = K == 1 ? 4 : 1;
    const ulonglong2 *s = (const ulonglong2 *)src;
#pragma unroll
    for (int h = 0; h < kMaxChunks; h += kTogether) {
        ulonglong2 v[kTogether];
#pragma unroll
        for (int j = 0; j < kTogether; ++j)
            if (h + j < kMaxChunks && 2 * (h + j) < (int)p.words) v[j] = __ldcg(s + h + j);
#pragma unroll
        for (int j = 0; j < kTogether; ++j) {
            const int c = h + j;
            if (c < kMaxChunks && 2 * c < (int)p.words) {
                fold(v[j].x);
                if (2 * c + 1 < (int)p.words) fold(v[j].y);
                keep(c, v[j].x, v[j].y);
            }
        }
    }
}
GCC_D void copy_image(const KParams &p, uint64_t *dst, const uint64_t *src) {
#pragma unroll
    for (int c = 0; c < kMaxChunks; ++c)
        if (2 * c < (int)p.words)
            __stcg((ulonglong2 *)dst + c, __ldcg((const ulonglong2 *)src + c));
}
// Last read op before op i (program order), -1 if none.
GCC_D int rowcopy_src(unsigned long long readmask, uint32_t i) {
    unsigned long long m = readmask & ((1ull << i) - 1ull);
    return m ? 63 - __clzll((long long)m) : -1;
}
// Extended write op (a request whose `read` word is negative, see
// gcc_engine.h GCC_OP_*): an integer read-modify-write of row fields, or an
// insert of a fresh row. Runs with the row held exclusively by the
// transaction (2PL lock, OCC write lock at commit, TO uncommitted mark,
// ordered turn); read-modify-writes fold the row image they read into the
// digest like a read.
GCC_D unsigned long long apply_ext(const KParams &p, uint64_t *r, uint32_t tx, uint32_t i,
                                  uint32_t w) {
    const uint32_t op = (w >> 28) & 7u, f = (w >> 24) & 15u, v = w & 0xFFFFFFu;
    const uint32_t fmax = op == GCC_OP_STOCK ? 6u : (op == GCC_OP_PAY ? 7u : 9u);
    if (op < GCC_OP_ADD || op > GCC_OP_INSERT || f > fmax || p.words != 11u) {
        set_error(p.ctr, GCC_EFORMAT, 0);
        return 0ull;
    }
    if (op == GCC_OP_INSERT) {
        __stcg((unsigned long long *)(r + 1), (unsigned long long)tx);
        __stcg((unsigned long long *)(r + 2), (unsigned long long)v);
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k)
            __stcg((unsigned long long *)(r + 3 + k),
                   (unsigned long long)hash3(p.write_seed, tx, 1024ull + i * 8ull + k));
        return 0ull;
    }
    unsigned long long dt = 0;
    read_image<4>(p, r, tx, 0, i, dt);
    unsigned long long *fw = (unsigned long long *)(r + 1 + f);
    const unsigned long long a = __ldcg(fw);
    if (op == GCC_OP_ADD) {
        __stcg(fw, a + v);
    } else if (op == GCC_OP_SUB) {
        __stcg(fw, a - v);
    } else if (op == GCC_OP_STOCK) {
        const unsigned long long q = v & 0xFFu, remote = (v >> 8) & 1u;
        __stcg(fw, a >= q + 10u ? a - q : a - q + 91u);
        __stcg(fw + 1, __ldcg(fw + 1) + q);
        __stcg(fw + 2, __ldcg(fw + 2) + 1u);
        __stcg(fw + 3, __ldcg(fw + 3) + remote);
    } else if (op == GCC_OP_PAY) {
        __stcg(fw, a - v);
        __stcg(fw + 1, __ldcg(fw + 1) + v);
        __stcg(fw + 2, __ldcg(fw + 2) + 1u);
    }
    return dt;
}

// Apply write op i of tx to `row` (GCC_WRITE_FIELD or GCC_WRITE_ROWCOPY, or
// an extended op when the run enables them). Extended ops exist only in the
// variable-length kernels (EXT): the 16-request kernels keep their registers.
template <class TX>
GCC_D void apply_write(const KParams &p, const TX &s, uint32_t row, uint32_t tx, uint64_t pos,
                       uint32_t i, unsigned long long &dg) {
    uint64_t *r = row_ptr(p, row);
    if (TX::kExt && p.ext_ops) {
        const int32_t w = p.txs ? __ldg(&p.txs[tx].requests[i].read)
                                : __ldg(&p.reqs[p.tx_off[tx] + i].read);
        if (w < 0) {
            dg += apply_ext(p, r, tx, i, (uint32_t)w);
            return;
        }
    }
    if (p.write_mode == GCC_WRITE_FIELD) {
        const uint32_t f = TX::K == 1 ? s.wfield : write_field(p.write_seed, tx, i);
        const unsigned long long v = TX::K == 1 ? s.wval : write_value(p.write_seed, tx, i);
        __stcg((unsigned long long *)(r + 1 + f), v);
        return;
    }
    int src = rowcopy_src(s.readmask, i);
    if (src < 0) {
#pragma unroll
        for (int c = 0; c < kMaxChunks; ++c)
            if (2 * c < (int)p.words) __stcg((ulonglong2 *)r + c, make_ulonglong2(0ull, 0ull));
    } else {
        copy_image(p, r, p.scratch + slot_of(p, pos, (uint32_t)src));
    }
}

// ---------------------------------------------------------------------------
// Retry timing of 2PL: an aborted attempt releases everything it held and
// tries again at once. When many transactions starve (past starve_limit
// attempts), at least one in kCrowdShare of those in flight, the lane whose
// request failed first polls that row's word (plain loads, short sleeps) until
// it looks compatible, at most kObstacleWaitNs, so that retries are not spent
// against the same conflict; from the kWaitFrom-th attempt on. The lock
// requests themselves keep the scheme's rule (e.g. no-wait: a conflicting
// request aborts). Measured, 10,485,760 rows, r 0.9, M tx/s, always waiting /
// never / this rule:
//   tpl_nw theta 0.6 118 / 153 / 151,  0.8 2.9 / 1.9 / 8.1,
//   tpl_nw theta 0.99 with 256 in flight 1.02 / 0.54 / 1.06,
//   tpl_wd theta 0.8 3.1 / 1.7 / 9.9,  theta 0.99, 256: 1.30 / 0.53 / 1.33
// (a writer that waits for a free word of a read row misses the moments in
// which it is free; under heavy contention retries at once keep every row of
// the others' ways locked). From 2, 12, 16, 30 attempts: within 5 %; one in
// 100: 146 at theta 0.6.
// ---------------------------------------------------------------------------
// Where eight or more transactions share a warp (warp_density 0 to 2) each of
// their attempts holds up the others' instructions, and retries at once cost
// more: they wait from the kWaitFromShared-th attempt on whoever starves.
// 65,536 transactions, r 0.9, tpl_nw, ms at warp_density 0 / 1 / 2, always
// waiting / only while many starve / this rule:
//   10,485,760 rows  theta 0.5  1.5 / 0.9 / 0.6   1.4 / 0.8 / 0.5   1.5 / 0.8 / 0.55
//                    theta 0.6  4.3 / 2.4 / 1.5   6.4 / 2.5 / 1.3   4.5 / 2.3 / 1.4
//                    theta 0.7  21 / 11 / 6.6     45 / 24 / 9.2     22 / 12 / 7.0
//   1,048,576 rows   theta 0.4  2.1 / 1.3 / 0.7   1.9 / 1.0 / 0.5   2.0 / 1.0 / 0.6
//                    theta 0.6  12 / 6.2 / 3.6    30 / 14 / 5.1     12 / 6.1 / 3.6
// (from the 6th or 16th attempt: within 10 %.)
constexpr uint32_t kWaitFromShared = 10;
constexpr uint32_t kWaitFrom = 6;
constexpr uint32_t kCrowdShare = 64;
constexpr uint64_t kObstacleWaitNs = 50000;
// want_zero: wait for the word to be 0; otherwise wait until (word & mask) == 0
GCC_D void await_row(const KParams &p, uint32_t row, unsigned long long mask, bool want_zero) {
    if (row == kNoRow || (p.flags & GCC_F_RETRY_IMMEDIATE)) return;
    const uint64_t t0 = gtimer();
    const uint64_t lim = p.spin_limit_ns < kObstacleWaitNs ? p.spin_limit_ns : kObstacleWaitNs;
    while (true) {
        unsigned long long w = ld_cg(p.meta + row);
        if (want_zero ? w == 0ull : (w & mask) == 0ull) return;
        if (gtimer() - t0 > lim) return;
        __nanosleep(64);
    }
}

// ---------------------------------------------------------------------------
// Latches of the slow_* variants (runtime.cuh:91-109), bounded.
// ---------------------------------------------------------------------------
GCC_D bool latch_acquire(const KParams &p, uint32_t row) {
    // CAS spin as in latch_lock (include/runtime.cuh:91-96), bounded. (A
    // test-and-test-and-set spin on a plain load starved diverged holder
    // lanes of the same warp here; every CAS attempt keeps the spinning path
    // stalled on L2 long enough for the holder to run its release.)
    unsigned *l = p.latch + row;
    if (atomicCAS(l, 0u, 1u) == 0u) { fence_acq_rel(); return true; }
    uint64_t t0 = gtimer();
    while (true) {
        if (atomicCAS(l, 0u, 1u) == 0u) { fence_acq_rel(); return true; }
        if (expired(t0, p.spin_limit_ns) || error_raised(p.ctr)) {
            set_error(p.ctr, GCC_ETIMEOUT, W_LATCH);
            return false;
        }
    }
}
GCC_D void latch_release(const KParams &p, uint32_t row) {
    fence_acq_rel();
    atomicExch(p.latch + row, 0u);
}

// Warp-aggregated timestamp allocation among the group leaders that arrive
// together (one atomic per warp instead of one per transaction).
GCC_D unsigned long long alloc_ts(Counters *c) {
    cg::coalesced_group act = cg::coalesced_threads();
    unsigned long long base = 0;
    if (act.thread_rank() == 0) base = atomicAdd(&c->ts, (unsigned long long)act.size());
    base = act.shfl(base, 0);
    return base + act.thread_rank();
}

// Per-attempt leader-side timing accumulators.
struct Clocks {
    unsigned long long ts, wait;
};

// An attempt works through its requests in stages: the group tries every
// request of a stage's mask (bit k: the lane's k-th) until all are done, one
// fails, or the bounded wait runs out. All stages of an attempt go through one
// inlined copy of `op(k)`, which returns an OpResult. `pre(pending)`, if there
// is one, goes before them: it takes requests off the mask and returns the
// stage's state bits (2: one failed).
enum OpResult : int { O_DONE = 0, O_FAIL = 1, O_RETRY = 2, O_ERR = 3, O_LOOKED = 4 };
struct Waiting {
    bool any = false;
    uint64_t t0 = 0;   // first wait of the attempt
    long long clk = 0;
};
struct NoPre {
    GCC_D uint32_t operator()(uint32_t &) const { return 0u; }
};
template <int G, int K, class OP, class PRE = NoPre>
GCC_D int run_stage(const KParams &p, const Group<G> &g, uint32_t pending, Waiting &w, unsigned site,
                    OP op, PRE pre = PRE{}) {
    while (true) {
        uint32_t st = pre(pending);  // 1: pending, 2: failed, 4: error
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (!((pending >> k) & 1u) || (st & 6u)) continue;
            const int r = op(k);
            if (r == O_DONE) pending &= ~(1u << k);
            else if (r == O_FAIL) st |= 2u;
            else if (r == O_ERR) st |= 4u;
        }
        if (pending) st |= 1u;
        st = g.orv(st);
        if (st & 4u) return O_ERR;
        if (st & 2u) return O_FAIL;
        if (!st) return O_DONE;
        if (!w.any) { w.any = true; w.t0 = gtimer(); w.clk = clock64(); }
        wait_pause();
        if (g.any(expired(w.t0, p.spin_limit_ns) || error_raised(p.ctr))) {
            if (g.glane == 0) set_error(p.ctr, GCC_ETIMEOUT, site);
            return O_ERR;
        }
    }
}
// The stage of request i alone.
template <int G>
GCC_D uint32_t only(const Group<G> &g, uint32_t i) {
    return g.glane == (int)(i % G) ? 1u << (i / G) : 0u;
}

// ===========================================================================
// 2PL no-wait / wait-die (twopl.cuh:233-322; slow_twopl.cuh:238-331)
// ===========================================================================
// One request of the fast variants: a speculative reader increment, or the
// exclusive word into a free one. `again`: the request waited already, so a
// reader looks before it increments. (With several requests a lane (K) the
// branch-free form costs more in spilled registers than it saves.)
template <bool WD, int K>
GCC_D int tpl_request(const KParams &p, uint32_t row, uint32_t tx, bool rd, bool again) {
    unsigned long long *m = p.meta + row;
    if (WD && again && rd) {
        const unsigned long long w = ld_cg(m);
        if (w & tpl::kExcl) return tpl::holder(w) < tx ? O_FAIL : O_RETRY;
    }
    const unsigned long long old = atom_lock_acq<(K == 1)>(m, rd, tpl::excl_word(tx));
    if (rd ? !(old & tpl::kExcl) : old == 0ull) return O_DONE;
    if (rd) atomicAdd(m, ~0ull);  // undo the speculative reader increment
    if (!WD || !(old & tpl::kExcl)) return O_FAIL;  // (shared holders: a writer dies)
    return tpl::holder(old) < tx ? O_FAIL : O_RETRY;
}
// Latch variants: plain read/modify/write of the same word under a latch.
template <bool WD>
GCC_D int slow_tpl_lock(const KParams &p, uint32_t row, uint32_t tx, bool shared) {
    if (!latch_acquire(p, row)) return O_ERR;
    volatile unsigned long long *m = p.meta + row;
    unsigned long long w = *m;
    int r;
    if (shared) {
        if (!(w & tpl::kExcl)) { *m = w + 1ull; r = O_DONE; }
        else r = (!WD || tpl::holder(w) < tx) ? O_FAIL : O_RETRY;
    } else {
        if (w == 0ull) { *m = tpl::excl_word(tx); r = O_DONE; }
        else if (!WD || !(w & tpl::kExcl)) r = O_FAIL;
        else r = tpl::holder(w) < tx ? O_FAIL : O_RETRY;
    }
    latch_release(p, row);
    return r;
}
// The fast variants' releases are plain reductions: the caller has fenced
// (once for all lanes) where rows were read or written under the locks.
template <bool SLOW>
GCC_D bool tpl_unlock(const KParams &p, uint32_t row, bool shared) {
    if (!SLOW) {
        if (shared) atomicAdd(p.meta + row, ~0ull);
        else atomicAnd(p.meta + row, tpl::kReaders);
        return true;
    }
    if (shared) {
        if (!latch_acquire(p, row)) return false;
        volatile unsigned long long *m = p.meta + row;
        *m = *m - 1ull;
        latch_release(p, row);
    } else {
        // the exclusive holder is the only writer of the word
        // (slow_twopl.cuh:333-338 stores without the latch)
        fence_acq_rel();
        atomicExch(p.meta + row, 0ull);
    }
    return true;
}

template <bool WD, bool SLOW, int K>
GCC_D int tpl_lock(const KParams &p, uint32_t row, uint32_t tx, bool rd, bool again) {
    return SLOW ? slow_tpl_lock<WD>(p, row, tx, rd) : tpl_request<WD, K>(p, row, tx, rd, again);
}

// First attempts take all locks at once (one ballot decides); after
// ordered_after failed attempts a retry takes them one request at a time,
// so that competing transactions cannot keep aborting each other. Both
// apply the scheme's rule: a conflict means abort (no-wait) or wait-or-die
// by transaction age (wait-die). Which locks a transaction takes and the
// rule applied to each never change; only the order of the acquisitions:
//   * by default a one-at-a-time retry takes every lock but one at once and
//     then the one whose request failed in the previous attempt: that lock
//     is contended, and taken last it is held the shortest time (taken in
//     request order, the reference's order, the hottest key of a Zipf
//     dataset comes first and is held while 15 more locks are taken one by
//     one, which made each writer of the hottest row cost ~15 us);
//   * GCC_F_REQUEST_ORDER and the latch variants keep request (= ascending
//     key) order (a latch variant's retries taking 15 latches at once kept
//     a starving transaction of a small hot table from ever committing);
//   * a lock plan (p.plan, set by the scheduler from its key-frequency
//     table) lists the hot requests: the others are taken at once, then the
//     hot ones one at a time, the hottest last.
template <int G, bool WD, bool SLOW, class TX>
GCC_D int attempt_tpl(const KParams &p, const Group<G> &g, const TX &s, uint32_t tx,
                      uint64_t pos, unsigned long long &dg, Clocks &ck, bool ordered) {
    constexpr int K = TX::K;
    uint32_t held = 0;
    uint32_t obst = kNoRow;         // row whose lock request failed
    bool obst_x = false;            // ... and whether it was an exclusive request
    uint32_t obst_i = 0xFFFFFFFFu;  // ... and its request index
    Waiting w;
    // planned: this attempt locks the requests outside the plan at once, then
    // the plan's requests in plan order; late bit k: op glane + k * G is planned
    bool planned = false;
    unsigned long long pl = 0;
    uint32_t late = 0;
    if constexpr (TX::MAXOPS == kMaxOps) {
        if (ordered && p.plan != nullptr) {
            planned = true;
            pl = __ldg(p.plan + tx);
        } else if (!SLOW && ordered && !(p.flags & GCC_F_REQUEST_ORDER) && s.obst_op) {
            // a one-entry plan: the request that failed last time, last
            planned = true;
            const unsigned long long i = s.obst_op - 1u;
            pl = (1ull << i) | (1ull << 16) | (i << 20);
        }
        if (planned) {
#pragma unroll
            for (int k = 0; k < K; ++k)
                if ((plan_mask(pl) >> (g.glane + k * G)) & 1u) late |= 1u << k;
        }
    }
    // Stages: the requests that go at once, then (ordered) one after another,
    // then whatever a plan did not list, as a plan only orders. A conflict
    // fails the attempt (no-wait) or, under wait-die, a younger holder makes
    // the request wait.
    uint32_t pending = ordered && !planned ? 0u : s.valid & ~late;
    const uint32_t n_seq = !ordered ? 0u : planned ? plan_count(pl) : s.n;
    int r = O_DONE;
    for (uint32_t j = 0;; ++j) {
        r = run_stage<G, K>(p, g, pending, w, W_TPL_WD, [&](int k) -> int {
            const bool rd = (s.isread >> k) & 1u;
            const int q = tpl_lock<WD, SLOW, K>(p, s.row[k], tx, rd, w.any);
            if (q == O_DONE) held |= 1u << k;
            else if (q == O_FAIL) {
                obst = s.row[k];
                obst_x = !rd;
                obst_i = (uint32_t)(g.glane + k * G);
            }
            return q;
        });
        if (r != O_DONE || j > n_seq || (j == n_seq && !planned)) break;
        if (j < n_seq) pending = only(g, planned ? plan_op(pl, j) : j) & s.valid & ~held;
        else pending = s.valid & ~held;
    }
    if (w.any) ck.wait += clock64() - w.clk;
    const bool fail = r != O_DONE, err = r == O_ERR;
    if (fail) {
#pragma unroll
        for (int k = 0; k < K; ++k)
            if ((held >> k) & 1u) tpl_unlock<SLOW>(p, s.row[k], (s.isread >> k) & 1u);
        if (err) return kGiveUp;
        if (!SLOW && !(p.flags & GCC_F_REQUEST_ORDER)) {
            const uint32_t fi = __reduce_min_sync(g.mask, obst_i);
            s.obst_op = fi == 0xFFFFFFFFu ? 0u : fi + 1u;
        }
        // an exclusive request waits for a free word, a shared one for the
        // exclusive holder to leave
        if ((s.attempts >= kWaitFrom && s.crowded) || (G <= 4 && s.attempts >= kWaitFromShared))
            await_row(p, obst, tpl::kExcl, obst_x);
        return kAbort;
    }
    // (the fast variants' lock RMWs are acquire operations)
    if (SLOW) fence_acq_rel();
    // Serialization point: every lock is held. The leader's sequence number
    // is ordered after every lane's acquisition and before every lane's
    // release by the two warp syncs (lanes' memory operations are otherwise
    // unordered with respect to each other).
    if (p.flags & GCC_F_COMMIT_LOG) {
        g.sync();
        if (g.glane == 0) {
            p.commit_hi[tx] = atomicAdd(&p.ctr->seq, 1ull);
            p.commit_lo[tx] = 0ull;
        }
        g.sync();
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if (((s.valid & s.isread) >> k) & 1u) {
            read_image<K>(p, row_ptr(p, s.row[k]), tx, pos, (uint32_t)(g.glane + k * G), dg);
        }
    }
    if (p.write_mode == GCC_WRITE_ROWCOPY) g.sync();
#pragma unroll
    for (int k = 0; k < K; ++k)
        if (((s.valid & ~s.isread) >> k) & 1u)
            apply_write(p, s, s.row[k], tx, pos, (uint32_t)(g.glane + k * G), dg);
    fence_acq_rel();  // the rows' reads and writes come before the releases
    bool uerr = false;
#pragma unroll
    for (int k = 0; k < K; ++k)
        if ((s.valid >> k) & 1u) uerr |= !tpl_unlock<SLOW>(p, s.row[k], (s.isread >> k) & 1u);
    return g.any(uerr) ? kGiveUp : kCommit;
}

// ===========================================================================
// Timestamp ordering (to.cuh:104-270; slow_to.cuh:137-238)
// ===========================================================================
// After a row's image was read under the committed word x (wts(x) <= ts) and
// the reader has fenced, so that the image's loads come before the look or the
// raise: make its rts cover ts. The image is of version wts(x) as long as the
// word keeps that wts and stays committed; another reader raising rts meanwhile
// does not change it, so only the raise is tried again, not the read. False: a
// writer came in.
GCC_D bool rts_cover(unsigned long long *m, unsigned long long x, uint64_t ts) {
    const unsigned long long wts = tso::wts(x);
    bool seen = false;  // x was read after the image
    while (!(x & tso::kUnc) && tso::wts(x) == wts) {
        if (tso::rts(x) >= ts) {
            if (seen) return true;
            x = ld_cg(m);
        } else {
            const unsigned long long old = atomicCAS(m, x, tso::make(false, ts, wts));
            if (old == x) return true;
            x = old;
        }
        seen = true;
    }
    return false;
}
// A read (fast variant) is O_LOOKED, with the row's word in x, once it has the
// image: a fence and rts_cover follow.
template <bool SLOW, int K>
GCC_D int to_read(const KParams &p, uint32_t row, uint64_t ts, uint32_t tx, uint64_t pos,
                  uint32_t i, unsigned long long &dt, unsigned long long &x) {
    unsigned long long *m = p.meta + row;
    if (SLOW) {
        if (!latch_acquire(p, row)) return O_ERR;
        x = *(volatile unsigned long long *)m;
        int r;
        if (tso::wts(x) > ts) r = O_FAIL;
        else if (x & tso::kUnc) r = O_RETRY;
        else {
            read_image<K>(p, row_ptr(p, row), tx, pos, i, dt);
            uint64_t rts = tso::rts(x) > ts ? tso::rts(x) : ts;
            *(volatile unsigned long long *)m = tso::make(false, rts, tso::wts(x));
            r = O_DONE;
        }
        latch_release(p, row);
        return r;
    }
    x = ld_acquire(m);
    if (tso::wts(x) > ts) return O_FAIL;
    if (x & tso::kUnc) return O_RETRY;  // wait for the older writer
    read_image<K>(p, row_ptr(p, row), tx, pos, i, dt);
    return O_LOOKED;
}
template <bool SLOW>
GCC_D int to_write(const KParams &p, uint32_t row, uint64_t ts, unsigned long long &prev) {
    unsigned long long *m = p.meta + row;
    if (SLOW) {
        if (!latch_acquire(p, row)) return O_ERR;
        unsigned long long x = *(volatile unsigned long long *)m;
        int r;
        if (tso::rts(x) > ts || tso::wts(x) > ts || (x & tso::kUnc)) r = O_FAIL;
        else { prev = x; *(volatile unsigned long long *)m = tso::make(true, ts, ts); r = O_DONE; }
        latch_release(p, row);
        return r;
    }
    unsigned long long x = ld_cg(m);
    if (tso::rts(x) > ts || tso::wts(x) > ts || (x & tso::kUnc)) return O_FAIL;
    if (atomicCAS(m, x, tso::make(true, ts, ts)) != x) return O_RETRY;
    prev = x;
    return O_DONE;
}

template <int G, bool SLOW, class TX>
GCC_D int attempt_to(const KParams &p, const Group<G> &g, const TX &s, uint32_t tx,
                     uint64_t pos, unsigned long long &dg, Clocks &ck, bool ordered) {
    constexpr int K = TX::K;
    unsigned long long ts = 0;
    if (g.glane == 0) {
        long long c0 = clock64();
        ts = alloc_ts(p.ctr);
        ck.ts += clock64() - c0;
    }
    ts = g.bcast(ts, 0);
    if (ts > tso::kTsMax) {
        if (g.glane == 0) set_error(p.ctr, GCC_EOVERFLOW, 0);
        return kGiveUp;
    }
    uint32_t wrote = 0;
    unsigned long long prev[K];
    Waiting w;
    uint32_t fail_i = 0xFFFFFFFFu;  // request index of this lane's failed op
    // A one-at-a-time retry visits every request but one at once first and
    // then the one that failed in the previous attempt, so a contended row
    // is held uncommitted the shortest time; with the default switch, which lies
    // past the starvation limit, only where starvation control is off or the
    // caller's ordered_after is below that limit. Request order (the reference's)
    // instead under GCC_F_REQUEST_ORDER, in the latch variant, and for a
    // starving transaction: TO's conflicts are timestamp checks, and a
    // starving transaction that reached its contended row last kept meeting
    // younger readers there (one did not commit within the wait bound at
    // theta 0.8). late bit k: op glane + k * G is that one.
    uint32_t late = 0, late_i = 0xFFFFFFFFu;
    if constexpr (TX::MAXOPS == kMaxOps) {
        if (!SLOW && ordered && !(p.flags & GCC_F_REQUEST_ORDER) && s.obst_op) {
            late_i = s.obst_op - 1u;
#pragma unroll
            for (int k = 0; k < K; ++k)
                if ((uint32_t)(g.glane + k * G) == late_i) late |= 1u << k;
        }
    }
    // Stages: all requests at once; on ordered retries one at a time, so two
    // writers cannot keep holding each other's rows uncommitted and aborting
    // each other. A request reads (it waits while an older writer's version is
    // uncommitted) or marks its row uncommitted with this ts.
    const bool split = late_i != 0xFFFFFFFFu;
    uint32_t pending = ordered && !split ? 0u : s.valid & ~late;
    const uint32_t n_seq = !ordered ? 0u : split ? 1u : s.n;
    // A lane with several requests fences once for all its reads of a pass,
    // between their images and the raises, and makes its marks after them; the
    // mark of a row that it still has to read waits for that read, which would
    // otherwise wait for the mark. (A fence for each read took wd 0 from 36 to
    // 14 M tx/s.)
    constexpr bool kTogether = K > 1 && !SLOW;
    uint32_t unread = 0;  // reads that the last pass left
    auto reads_first = [&](uint32_t &left) -> uint32_t {
        uint32_t st = 0;
        if constexpr (kTogether) {
            unsigned long long x[K], dt[K];
            uint32_t looked = 0;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                if (!(((left & s.isread) >> k) & 1u) || st) continue;
                const uint32_t i = g.glane + k * G;
                dt[k] = 0;
                const int q = to_read<SLOW, K>(p, s.row[k], ts, tx, pos, i, dt[k], x[k]);
                if (q == O_LOOKED) looked |= 1u << k;
                else if (q == O_FAIL) { st = 2u; fail_i = i; }
            }
            if (looked) {
                fence_acq_rel();
#pragma unroll
                for (int k = 0; k < K; ++k)
                    if (((looked >> k) & 1u) && rts_cover(p.meta + s.row[k], x[k], ts)) {
                        left &= ~(1u << k);
                        dg += dt[k];
                    }
            }
            unread = left & s.isread;
            g.sync();
        }
        return st;
    };
    auto op = [&](int k) -> int {
        const uint32_t i = g.glane + k * G;
        int q;
        if ((s.isread >> k) & 1u) {
            if (kTogether) return O_RETRY;
            unsigned long long dt = 0, x;
            q = to_read<SLOW, K>(p, s.row[k], ts, tx, pos, i, dt, x);
            if (q == O_LOOKED) {
                fence_acq_rel();
                q = rts_cover(p.meta + s.row[k], x, ts) ? O_DONE : O_RETRY;
            }
            if (q == O_DONE) dg += dt;
        } else {
            if (kTogether && unread) {
#pragma unroll
                for (int j = 0; j < K; ++j)
                    if (((unread >> j) & 1u) && s.row[j] == s.row[k]) return O_RETRY;
            }
            q = to_write<SLOW>(p, s.row[k], ts, prev[k]);
            if (q == O_DONE) wrote |= 1u << k;
        }
        if (q == O_FAIL) fail_i = i;
        return q;
    };
    int r = O_DONE;
    for (uint32_t j = 0;; ++j) {
        r = run_stage<G, K>(p, g, pending, w, W_TO_READ, op, reads_first);
        if (r != O_DONE || j == n_seq) break;
        pending = only(g, split ? late_i : j) & s.valid;
    }
    const bool fail = r != O_DONE, err = r == O_ERR;
    if (!SLOW && fail && !err && !(p.flags & GCC_F_REQUEST_ORDER)) {
        const uint32_t fi = __reduce_min_sync(g.mask, fail_i);
        s.obst_op = fi == 0xFFFFFFFFu ? 0u : fi + 1u;
    }
    if (w.any) ck.wait += clock64() - w.clk;
    if (fail) {
        // restore the words this attempt marked uncommitted (to.cuh:255-270)
#pragma unroll
        for (int k = 0; k < K; ++k)
            if ((wrote >> k) & 1u) atomicExch(p.meta + s.row[k], prev[k]);
        fence_acq_rel();
        return err ? kGiveUp : kAbort;
    }
    // Serialization key: (batch, timestamp); timestamps restart per batch.
    if ((p.flags & GCC_F_COMMIT_LOG) && g.glane == 0) {
        p.commit_hi[tx] = p.batch_st;
        p.commit_lo[tx] = ts;
    }
    if (p.write_mode == GCC_WRITE_ROWCOPY) g.sync();
#pragma unroll
    for (int k = 0; k < K; ++k)
        if ((wrote >> k) & 1u) apply_write(p, s, s.row[k], tx, pos, g.glane + k * G, dg);
    fence_acq_rel();
#pragma unroll
    for (int k = 0; k < K; ++k)
        if ((wrote >> k) & 1u) atomicExch(p.meta + s.row[k], tso::make(false, ts, ts));
    return kCommit;
}

// ===========================================================================
// MVCC (mvcc.cuh:113-297). A transaction reads all its rows at once and then
// marks all rows it writes at once: a reader waits for any uncommitted version
// (as in the reference), but it waits before the transaction holds anything,
// and a write never waits (it fails on a younger read, a younger version or an
// uncommitted one), so the waits cannot form a cycle. One request after the
// other in key order, the reference's form, kept the first rows uncommitted
// for 15 more round trips, which every reader of them waited out. Retries past
// the switch (ordered_after) mark one row at a time in request order, so two
// writers cannot keep failing on each other's marks.
// Measured, 10,485,760 rows, theta 0.6, r 0.5, 100,003 transactions in batches
// of 65,536: 31 -> 11.6 ms a run; r 0.9, 262,144 transactions: 15.3 -> 2.3 ms;
// theta 0.8, r 0.9, 65,536 transactions: 98 -> 11 ms. (The switch to one mark
// at a time after 2, 8, 16 or 64 retries measures the same within 3 %.)
// Two reference defects are not reproduced: the base row is updated at commit
// (mvcc.cuh:143 leaves the copy commented out) and each version owns a full
// row image (mvcc.cuh:142 strides the version data by sizeof(version_node)).
// ===========================================================================
template <bool SLOW, int K>
GCC_D int mvcc_read(const KParams &p, uint32_t row, uint64_t ts, uint32_t tx, uint64_t pos,
                    uint32_t i, unsigned long long &dt) {
    unsigned long long *m = p.meta + row;
    if (SLOW && !latch_acquire(p, row)) return O_ERR;
    const unsigned long long x = SLOW ? *(volatile unsigned long long *)m : ld_acquire(m);
    int r;
    if (x & tso::kUnc) {
        r = O_RETRY;
    } else if (tso::wts(x) <= ts) {
        read_image<K>(p, row_ptr(p, row), tx, pos, i, dt);
        if (!SLOW) {
            fence_acq_rel();
            r = rts_cover(m, x, ts) ? O_DONE : O_RETRY;
        } else {
            if (tso::rts(x) < ts) *(volatile unsigned long long *)m = tso::make(false, ts, tso::wts(x));
            r = O_DONE;
        }
    } else {
        // walk the version chain to the newest version with wts <= ts; a writer
        // may be linking a newer one meanwhile, whose fields come with the
        // acquire of the chain's head
        unsigned node = ld_acquire(p.turn + row);
        unsigned hops = 0;
        while (node != kNoRow && tso::wts(ld_cg(p.ver_ts + node)) > ts && hops < 0x1000000u) {
            node = ld_cg(p.ver_prev + node);
            ++hops;
        }
        if (node == kNoRow || hops >= 0x1000000u) {
            set_error(p.ctr, GCC_EFORMAT, W_MVCC_READ);  // broken chain
            r = O_ERR;
        } else {
            // versions never change once linked, and the row's committed wts is
            // past ts already: no later write can come between, so the word is
            // not looked at again
            read_image<K>(p, p.ver_data + (size_t)node * p.wslot, tx, pos, i, dt);
            r = O_DONE;
        }
    }
    if (SLOW) latch_release(p, row);
    return r;
}

template <int G, bool SLOW, class TX>
GCC_D int attempt_mvcc(const KParams &p, const Group<G> &g, const TX &s, uint32_t tx,
                       uint64_t pos, unsigned long long &dg, Clocks &ck, bool ordered) {
    constexpr int K = TX::K;
    unsigned long long ts = 0;
    if (g.glane == 0) {
        long long c0 = clock64();
        ts = alloc_ts(p.ctr);
        ck.ts += clock64() - c0;
    }
    ts = g.bcast(ts, 0);
    if (ts > tso::kTsMax) {
        if (g.glane == 0) set_error(p.ctr, GCC_EOVERFLOW, 0);
        return kGiveUp;
    }
    uint32_t wrote = 0;
    unsigned long long prev[K];
    bool twice = false;
    Waiting w;
    // Stages: the reads, then the writes, at once or (ordered) one by one.
    uint32_t pending = s.valid & s.isread;
    unsigned long long todo = ~(unsigned long long)s.readmask & (s.n < 64u ? (1ull << s.n) - 1ull : ~0ull);
    int r = O_DONE;
    while (true) {
        r = run_stage<G, K>(p, g, pending, w, W_MVCC_READ, [&](int k) -> int {
            if ((s.isread >> k) & 1u) {
                unsigned long long dt = 0;
                const int q = mvcc_read<SLOW, K>(p, s.row[k], ts, tx, pos, (uint32_t)(g.glane + k * G), dt);
                if (q == O_DONE) dg += dt;
                return q;
            }
            const int q = to_write<SLOW>(p, s.row[k], ts, prev[k]);
            if (q == O_DONE) {
                wrote |= 1u << k;
                twice |= tso::rts(prev[k]) == ts;
            }
            return q;
        });
        if (r != O_DONE || !todo) break;
        if (ordered) {
            pending = only(g, (uint32_t)(__ffsll((long long)todo) - 1));
            todo &= todo - 1ull;
        } else {
            pending = s.valid & ~s.isread;
            todo = 0;
        }
    }
    if (w.any) ck.wait += clock64() - w.clk;
    bool fail = r != O_DONE, err = r == O_ERR;
    // A row that this transaction read and then marked (its own timestamp is
    // the row's rts): the read belongs before the write. A request order that
    // has the write first would have to read its own uncommitted row, which no
    // wait ends; it is refused as it always was.
    if (!fail && g.any(twice)) {
        bool bad = false;
        for (uint32_t i = 0; i < s.n; ++i) {
            if ((s.readmask >> i) & 1ull) continue;
            uint32_t wrow = kNoRow;
#pragma unroll
            for (int k = 0; k < K; ++k)
                if (k == (int)(i / G)) wrow = s.row[k];
            wrow = g.bcast(wrow, (int)(i % G));
#pragma unroll
            for (int k = 0; k < K; ++k)
                bad |= ((s.valid & s.isread) >> k & 1u) && s.row[k] == wrow &&
                       (uint32_t)(g.glane + k * G) > i;
        }
        if (g.any(bad)) {
            if (g.glane == 0) set_error(p.ctr, GCC_ETIMEOUT, W_MVCC_READ);
            fail = err = true;
        }
    }
    if (fail) {
#pragma unroll
        for (int k = 0; k < K; ++k)
            if ((wrote >> k) & 1u) atomicExch(p.meta + s.row[k], prev[k]);
        fence_acq_rel();
        return err ? kGiveUp : kAbort;
    }
    // Serialization key: (batch, timestamp); timestamps restart per batch.
    if ((p.flags & GCC_F_COMMIT_LOG) && g.glane == 0) {
        p.commit_hi[tx] = p.batch_st;
        p.commit_lo[tx] = ts;
    }
    if (p.write_mode == GCC_WRITE_ROWCOPY) g.sync();
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if (!((wrote >> k) & 1u)) continue;
        uint32_t i = g.glane + k * G;
        uint32_t row = s.row[k];
        // push the current base row as the version it replaces, link it,
        // then install the new base row and publish (uncommitted -> 0)
        uint32_t node = (uint32_t)(pos * p.slot_ops + i);
        // (acquire: readers of this version reach the older ones through it)
        const uint32_t older = ld_acquire(p.turn + row);
        copy_image(p, p.ver_data + (size_t)node * p.wslot, row_ptr(p, row));
        p.ver_ts[node] = prev[k];
        p.ver_prev[node] = older;
        fence_acq_rel();
        atomicExch(p.turn + row, node);
        apply_write(p, s, row, tx, pos, i, dg);
        fence_acq_rel();
        atomicExch(p.meta + row, tso::make(false, ts, ts));
    }
    return kCommit;
}

// ===========================================================================
// Silo (silo.cuh:116-338; slow_silo.cuh:188-326). The commit timestamp is
// max(read-set ts, current write-set ts) + 1 as in Silo; the reference takes
// the write-set term from a field Write never sets (silo.cuh:306-310), which
// lets a record's ts repeat and a stale read validate.
// ===========================================================================
template <bool SLOW, int K>
GCC_D int silo_read(const KParams &p, uint32_t row, uint32_t tx, uint64_t pos, uint32_t i,
                    unsigned long long &dt, unsigned long long &ts) {
    unsigned long long *m = p.meta + row;
    if (SLOW) {
        if (!latch_acquire(p, row)) return O_ERR;
        unsigned long long x = *(volatile unsigned long long *)m;
        int r = O_RETRY;
        if (!(x & silo::kLock)) { read_image<K>(p, row_ptr(p, row), tx, pos, i, dt); ts = silo::ts(x); r = O_DONE; }
        latch_release(p, row);
        return r;
    }
    const unsigned long long x = ld_acquire(m);
    if (x & silo::kLock) return O_RETRY;
    read_image<K>(p, row_ptr(p, row), tx, pos, i, dt);
    fence_acq_rel();
    if (ld_cg(m) != x) return O_RETRY;
    ts = silo::ts(x);
    return O_DONE;
}
// No-wait write lock: O_DONE (cur = word before locking), O_FAIL if locked.
template <bool SLOW>
GCC_D int occ_lock(const KParams &p, uint32_t row, unsigned long long lockbit,
                   unsigned long long &cur) {
    unsigned long long *m = p.meta + row;
    if (SLOW) {
        if (!latch_acquire(p, row)) return O_ERR;
        unsigned long long x = *(volatile unsigned long long *)m;
        int r = O_FAIL;
        if (!(x & lockbit)) { *(volatile unsigned long long *)m = x | lockbit; cur = x; r = O_DONE; }
        latch_release(p, row);
        return r;
    }
    // one round trip: setting a set bit changes nothing
    cur = atom_or_acq(m, lockbit);
    return (cur & lockbit) ? O_FAIL : O_DONE;
}

// Lock the write set, no-wait and all at once (silo.cuh:268-281,
// tictoc.cuh:269-282). `cts` accumulates f(word before locking) over the locked
// words.
template <int G, bool SLOW, bool TICTOC, class TX>
GCC_D void occ_lock_writes(const KParams &p, const TX &s, uint32_t writes, uint32_t &held,
                           unsigned long long &cts, bool &fail, bool &err) {
    constexpr int K = TX::K;
    const unsigned long long lockbit = TICTOC ? tictoc::kLock : silo::kLock;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if (!((writes >> k) & 1u) || fail || err) continue;
        unsigned long long cur;
        int r = occ_lock<SLOW>(p, s.row[k], lockbit, cur);
        if (r == O_DONE) {
            held |= 1u << k;
            unsigned long long c = TICTOC ? tictoc::rts(cur) + 1ull : silo::ts(cur);
            cts = cts > c ? cts : c;
        } else if (r == O_FAIL) fail = true;
        else err = true;
    }
}

template <int G, bool SLOW, class TX>
GCC_D int attempt_silo(const KParams &p, const Group<G> &g, const TX &s, uint32_t tx,
                       uint64_t pos, unsigned long long &dg, Clocks &ck) {
    constexpr int K = TX::K;
    unsigned long long rec[K];
    uint32_t reads = s.valid & s.isread, writes = s.valid & ~s.isread;
    uint32_t pending = reads, held = 0;
    bool fail = false, err = false;
    // read phase: consistent snapshots (silo.cuh:223-259)
    uint64_t t0 = gtimer();
    bool first = true;
    long long cw = 0;
    while (true) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (!((pending >> k) & 1u) || err) continue;
            unsigned long long dt = 0;
            int r = silo_read<SLOW, K>(p, s.row[k], tx, pos, g.glane + k * G, dt, rec[k]);
            if (r == O_DONE) { pending &= ~(1u << k); dg += dt; }
            else if (r == O_ERR) err = true;
        }
        bool ge = g.any(err), gp = g.any(pending != 0u);
        if (ge) return kGiveUp;
        if (!gp) break;
        if (first) { first = false; cw = clock64(); }
        wait_pause();
        if (g.any(expired(t0, p.spin_limit_ns) || error_raised(p.ctr))) {
            if (g.glane == 0) set_error(p.ctr, GCC_ETIMEOUT, W_SILO_READ);
            return kGiveUp;
        }
    }
    if (!first) ck.wait += clock64() - cw;
    // validation: lock the write set, no-wait (silo.cuh:268-281)
    unsigned long long cts = 0;
    occ_lock_writes<G, SLOW, false>(p, s, writes, held, cts, fail, err);
    bool gf = g.any(fail), ge = g.any(err);
    if (!gf && !ge) {
        if (SLOW) fence_acq_rel();
        // Serialization point: write set locked (by every lane), read set not
        // yet validated (by any lane). Two transactions that read what the
        // other writes must not both miss the other's lock. The fast variant's
        // lock RMWs are acquire operations whose old values are back, so they
        // are performed at L2, where the looks go; that orders the locking lane
        // only (and a vote orders nothing), the warp sync makes every lane's
        // look come after every lane's RMW, log or no log. A fence here besides
        // (acq_rel or sc, all lanes or one) costs a quarter: theta 0.6 310 -> 230
        // M tx/s.
        g.sync();
        if (p.flags & GCC_F_COMMIT_LOG) {
            if (g.glane == 0) {
                p.commit_hi[tx] = atomicAdd(&p.ctr->seq, 1ull);
                p.commit_lo[tx] = 0ull;
            }
            g.sync();
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (!((reads >> k) & 1u)) continue;
            unsigned long long x = ld_cg(p.meta + s.row[k]);
            if (silo::ts(x) != rec[k] || (x & silo::kLock)) fail = true;
            cts = cts > rec[k] ? cts : rec[k];
        }
        gf = g.any(fail);
    }
    if (gf || ge) {
#pragma unroll
        for (int k = 0; k < K; ++k)
            if ((held >> k) & 1u) atomicAnd(p.meta + s.row[k], ~silo::kLock);
        fence_acq_rel();
        return ge ? kGiveUp : kAbort;
    }
    cts = g.maxv(cts) + 1ull;
    if (p.write_mode == GCC_WRITE_ROWCOPY) g.sync();
#pragma unroll
    for (int k = 0; k < K; ++k)
        if ((writes >> k) & 1u) apply_write(p, s, s.row[k], tx, pos, g.glane + k * G, dg);
    fence_acq_rel();
#pragma unroll
    for (int k = 0; k < K; ++k)
        if ((writes >> k) & 1u) atomicExch(p.meta + s.row[k], cts);
    return kCommit;
}

// ===========================================================================
// TicToc (tictoc.cuh:115-368; slow_tictoc.cuh)
// ===========================================================================
template <bool SLOW, int K>
GCC_D int tictoc_read(const KParams &p, uint32_t row, uint32_t tx, uint64_t pos, uint32_t i,
                      unsigned long long &dt, unsigned long long &wts, unsigned long long &rts) {
    unsigned long long *m = p.meta + row;
    if (SLOW) {
        if (!latch_acquire(p, row)) return O_ERR;
        unsigned long long x = *(volatile unsigned long long *)m;
        int r = O_RETRY;
        if (!(x & tictoc::kLock)) {
            read_image<K>(p, row_ptr(p, row), tx, pos, i, dt);
            wts = tictoc::wts(x); rts = tictoc::rts(x); r = O_DONE;
        }
        latch_release(p, row);
        return r;
    }
    unsigned long long x1 = ld_acquire(m);
    if (x1 & tictoc::kLock) return O_RETRY;
    read_image<K>(p, row_ptr(p, row), tx, pos, i, dt);
    fence_acq_rel();
    if (ld_cg(m) != x1) return O_RETRY;
    wts = tictoc::wts(x1);
    rts = tictoc::rts(x1);
    return O_DONE;
}
// Extend a read version's rts to cover commit_ts (tictoc.cuh:302-340).
template <bool SLOW>
GCC_D int tictoc_extend(const KParams &p, uint32_t row, unsigned long long rwts,
                        unsigned long long cts) {
    unsigned long long *m = p.meta + row;
    for (int tries = 0; tries < 1 << 20; ++tries) {
        if (SLOW && !latch_acquire(p, row)) return O_ERR;
        unsigned long long x = SLOW ? *(volatile unsigned long long *)m : ld_cg(m);
        unsigned long long wts = tictoc::wts(x), rts = tictoc::rts(x);
        int r;
        if (wts != rwts || (rts <= cts && (x & tictoc::kLock))) {
            r = O_FAIL;
        } else if (rts > cts) {
            r = O_DONE;
        } else {
            unsigned long long delta = cts - wts;
            unsigned long long shift = delta - (delta & 0x7FFFull);
            unsigned long long nx = tictoc::make(false, delta - shift, wts + shift);
            if (SLOW) { *(volatile unsigned long long *)m = nx; r = O_DONE; }
            else r = atomicCAS(m, x, nx) == x ? O_DONE : O_RETRY;
        }
        if (SLOW) latch_release(p, row);
        if (r != O_RETRY) return r;
    }
    set_error(p.ctr, GCC_ETIMEOUT, W_TICTOC_EXT);
    return O_ERR;
}

template <int G, bool SLOW, class TX>
GCC_D int attempt_tictoc(const KParams &p, const Group<G> &g, const TX &s, uint32_t tx,
                         uint64_t pos, unsigned long long &dg, Clocks &ck) {
    constexpr int K = TX::K;
    unsigned long long rw[K], rr[K];
    uint32_t reads = s.valid & s.isread, writes = s.valid & ~s.isread;
    uint32_t pending = reads, held = 0;
    bool fail = false, err = false;
    uint64_t t0 = gtimer();
    bool first = true;
    long long cw = 0;
    while (true) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (!((pending >> k) & 1u) || err) continue;
            unsigned long long dt = 0;
            int r = tictoc_read<SLOW, K>(p, s.row[k], tx, pos, g.glane + k * G, dt, rw[k], rr[k]);
            if (r == O_DONE) { pending &= ~(1u << k); dg += dt; }
            else if (r == O_ERR) err = true;
        }
        bool ge = g.any(err), gp = g.any(pending != 0u);
        if (ge) return kGiveUp;
        if (!gp) break;
        if (first) { first = false; cw = clock64(); }
        wait_pause();
        if (g.any(expired(t0, p.spin_limit_ns) || error_raised(p.ctr))) {
            if (g.glane == 0) set_error(p.ctr, GCC_ETIMEOUT, W_TICTOC_READ);
            return kGiveUp;
        }
    }
    if (!first) ck.wait += clock64() - cw;
    unsigned long long cts = 0;
    occ_lock_writes<G, SLOW, true>(p, s, writes, held, cts, fail, err);
    bool gf = g.any(fail), ge = g.any(err);
    if (!gf && !ge) {
#pragma unroll
        for (int k = 0; k < K; ++k)
            if ((reads >> k) & 1u) cts = cts > rw[k] ? cts : rw[k];
        cts = g.maxv(cts);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (!((reads >> k) & 1u) || fail || err) continue;
            if (rr[k] >= cts) continue;
            int r = tictoc_extend<SLOW>(p, s.row[k], rw[k], cts);
            if (r == O_FAIL) fail = true;
            else if (r == O_ERR) err = true;
        }
        gf = g.any(fail);
        ge = g.any(err);
    }
    if (gf || ge) {
#pragma unroll
        for (int k = 0; k < K; ++k)
            if ((held >> k) & 1u) atomicAnd(p.meta + s.row[k], ~tictoc::kLock);
        fence_acq_rel();
        return ge ? kGiveUp : kAbort;
    }
    // Serialization key: (batch, commit_ts, order of validation among equal
    // commit_ts). Within a batch commit_ts <= commits + 1 < 2^32.
    if (p.flags & GCC_F_COMMIT_LOG) {
        g.sync();
        if (g.glane == 0) {
            p.commit_hi[tx] = p.batch_st;
            p.commit_lo[tx] = (cts << 32) | (atomicAdd(&p.ctr->seq, 1ull) & 0xFFFFFFFFull);
        }
        g.sync();
    }
    if (p.write_mode == GCC_WRITE_ROWCOPY) g.sync();
#pragma unroll
    for (int k = 0; k < K; ++k)
        if ((writes >> k) & 1u) apply_write(p, s, s.row[k], tx, pos, g.glane + k * G, dg);
    fence_acq_rel();
#pragma unroll
    for (int k = 0; k < K; ++k)
        if ((writes >> k) & 1u) atomicExch(p.meta + s.row[k], tictoc::make(false, 0, cts));
    return kCommit;
}

// ===========================================================================
// GaccO / GPUTx: deterministic execution in a precomputed order. Each row has
// a list of its accesses in that order and a turn word that counts how many
// of them are done (gacco.cuh:156-175; GPUTx's rank launches become the same
// hand-off over the (rank, tx) order, which also orders same-rank conflicts
// by tx index). A write waits until every access before it is done; a read
// only until the last write before it is, so the reads between two writes of
// a row run together instead of one after another. op_wait is the turn value
// an access waits for (k_access_waits).
//
// The bound is the chain of the hottest row: its accesses alternate between
// one write and one run of reads, and each stage costs the hand-over (release
// add at L2, the waiter's next poll, the row's load or store). What is on that
// path was shortened: write values are computed before the wait, the clock and
// the error flag are looked at once in kWaitChecks polls, and a transaction
// that is far from its turn sleeps in proportion, because hundreds of waiters
// polling one word slow the very release they wait for.
// Measured, gacco, 10,485,760 rows, theta 0.8, r 0.9, batch 65,536: 26.9 ms a
// batch with every access taking its own turn, 2.65 ms now (3.4 with this
// hand-off alone, then row images loaded at once and the sleep by writes).
// ===========================================================================
constexpr unsigned kWaitChecks = 16;
// A transaction with more than kTurnNear accesses ahead of its nearest one
// sleeps kTurnSleepNs for each write among them, taken as the batch's share of
// writes: the reads between two writes run together, so the time to a turn goes
// by the writes ahead: about 4 us for one with the reads after it. A fixed time
// an access (150 ns) fitted read ratio 0.9 and made waiters at 0.95 and above
// sleep past their turn. Measured, gacco, theta 0.8, a batch of 65,536, ms,
// that / 300 / 600 / 900 ns a write:
//   r 0.5 8.7 / 8.8 / 8.7 / 8.7, 0.8 4.65 / 4.8 / 4.7 / 4.7, 0.9 2.75 / 2.75 /
//   2.7 / 2.65, 0.95 2.05 / 1.7 / 1.55 / 1.55, 0.98 1.65 / 1.15 / 0.95 / 0.9,
//   0.99 1.25 / 0.95 / 0.8 / 0.75; without any sleep 19.5 at 0.5, 7.2 at 0.9.
// (Following the pace of the turn seen by each waiter instead: 3.6 at 0.9.)
constexpr uint32_t kTurnNear = 12;
constexpr uint32_t kTurnSleepNs = 900, kTurnSleepMaxNs = 20000;

GCC_D uint32_t turn_sleep_ns(const Counters *c) {
    const float reads = (float)c->acc_reads, writes = (float)c->acc_writes;
    return writes > 0.0f ? (uint32_t)((float)kTurnSleepNs * (writes / (reads + writes))) : 0u;
}

template <int G, class TX>
GCC_D int attempt_ordered(const KParams &p, const Group<G> &g, const TX &s, uint32_t tx,
                          uint64_t pos, unsigned long long &dg, Clocks &ck) {
    constexpr int K = TX::K;
    const bool rowcopy = p.write_mode == GCC_WRITE_ROWCOPY;
    uint32_t wait[K];
#pragma unroll
    for (int k = 0; k < K; ++k)
        wait[k] = ((s.valid >> k) & 1u) ? __ldg(p.op_wait + pos * p.slot_ops + g.glane + k * G) : 0u;
    uint32_t pending = s.valid;
    unsigned long long done_ops = 0;
    uint64_t t0 = 0;
    unsigned polls = 0;
    long long cw = 0;
    while (true) {
        unsigned long long mine = 0;
        uint32_t away = 0xFFFFFFFFu;  // fewest accesses ahead of a pending one
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (!((pending >> k) & 1u)) continue;
            uint32_t i = g.glane + k * G;
            bool rd = (s.isread >> k) & 1u;
            if (!rd && rowcopy) {
                int src = rowcopy_src(s.readmask, i);
                if (src >= 0 && !((done_ops >> src) & 1ull)) { away = 0; continue; }
            }
            // acquire: the accesses this one waits for are visible
            const uint32_t turn = ld_acquire(p.turn + s.row[k]);
            if (turn < wait[k]) {
                away = min(away, wait[k] - turn);
                continue;
            }
            if (rd) {
                read_image<K>(p, row_ptr(p, s.row[k]), tx, pos, i, dg);
            } else {
                apply_write(p, s, s.row[k], tx, pos, i, dg);
            }
            // release: this access comes before those that wait for it
            red_add_rel(p.turn + s.row[k], 1u);
            pending &= ~(1u << k);
            mine |= 1ull << i;
        }
        if (rowcopy) {
            done_ops |= g.orv(mine);
            g.sync();
        }
        if (!g.any(pending != 0u)) break;
        if (polls == 0) {
            t0 = gtimer();
            cw = clock64();
        }
        if (++polls % kWaitChecks == 0 &&
            g.any(expired(t0, p.spin_limit_ns) || error_raised(p.ctr))) {
            if (g.glane == 0) set_error(p.ctr, GCC_ETIMEOUT, W_TURN);
            return kGiveUp;
        }
        away = __reduce_min_sync(g.mask, away);
        if (away > kTurnNear)
            __nanosleep(min((away - kTurnNear) * s.turn_ns, kTurnSleepMaxNs));
        else if (G < 32)
            wait_pause();  // the warp's other groups may hold the turn
    }
    if (polls) ck.wait += clock64() - cw;
    if ((p.flags & GCC_F_COMMIT_LOG) && g.glane == 0) {
        p.commit_hi[tx] = p.batch_st + pos;
        p.commit_lo[tx] = 0ull;
    }
    return kCommit;
}

template <int SCH, int G, class TX>
GCC_D int attempt(const KParams &p, const Group<G> &g, const TX &s, uint32_t tx,
                  uint64_t pos, unsigned long long &dg, Clocks &ck, bool ordered) {
    if constexpr (SCH == S_TPL_NW) return attempt_tpl<G, false, false>(p, g, s, tx, pos, dg, ck, ordered);
    else if constexpr (SCH == S_TPL_WD) return attempt_tpl<G, true, false>(p, g, s, tx, pos, dg, ck, ordered);
    else if constexpr (SCH == S_SLOW_TPL_NW) return attempt_tpl<G, false, true>(p, g, s, tx, pos, dg, ck, ordered);
    else if constexpr (SCH == S_SLOW_TPL_WD) return attempt_tpl<G, true, true>(p, g, s, tx, pos, dg, ck, ordered);
    else if constexpr (SCH == S_TO) return attempt_to<G, false>(p, g, s, tx, pos, dg, ck, ordered);
    else if constexpr (SCH == S_SLOW_TO) return attempt_to<G, true>(p, g, s, tx, pos, dg, ck, ordered);
    else if constexpr (SCH == S_MVCC) return attempt_mvcc<G, false>(p, g, s, tx, pos, dg, ck, ordered);
    else if constexpr (SCH == S_SLOW_MVCC) return attempt_mvcc<G, true>(p, g, s, tx, pos, dg, ck, ordered);
    else if constexpr (SCH == S_SILO) return attempt_silo<G, false>(p, g, s, tx, pos, dg, ck);
    else if constexpr (SCH == S_SLOW_SILO) return attempt_silo<G, true>(p, g, s, tx, pos, dg, ck);
    else if constexpr (SCH == S_TICTOC) return attempt_tictoc<G, false>(p, g, s, tx, pos, dg, ck);
    else if constexpr (SCH == S_SLOW_TICTOC) return attempt_tictoc<G, true>(p, g, s, tx, pos, dg, ck);
    else return attempt_ordered<G>(p, g, s, tx, pos, dg, ck);
}

__host__ __device__ constexpr bool is_tpl(int s) {
    return s == S_TPL_NW || s == S_TPL_WD || s == S_SLOW_TPL_NW || s == S_SLOW_TPL_WD;
}
__host__ __device__ constexpr bool is_ordered(int s) { return s == S_GACCO || s == S_GPUTX; }

// Attempts before retries switch to one request at a time (the caller can
// move the switch of 2PL / TO with gcc_run_params.ordered_after).
// Retries take their requests in parallel like the first attempt: Silo and
// TicToc always; 2PL for the first 15 retries, after which they go one request
// at a time (starting from the request that failed last time, see attempt_tpl;
// in key order under GCC_F_REQUEST_ORDER); TO for the first 129, i.e. until its
// retries go one transaction at a time anyway (from 4 x the default starvation
// limit on; a caller who moves starve_limit may move ordered_after with it):
// while others run, a TO attempt that visits its requests in turn meets younger
// timestamps on every one. MVCC marks its writes one by one from the 8th retry
// on, the ordered schemes never abort. The starvation control bounds the
// cycles that made fully parallel retries livelock. Measured, 10,485,760 rows,
// M tx/s, one at a time from the 16th / 31st / 61st / 131st retry / never:
//   to      theta 0.6 r 0.5            5.1 / 4.7 / 8.7 / 42 / 40
//           theta 0.8 r 0.9            0.9 / 0.8 / 1.0 / 3.0 / 3.0
//           theta 0.99, 512 in flight  0.27 / 0.27 / 0.25 / 0.37 / 0.39
//   tpl_nw  theta 0.6 r 0.5            30 / 29 / 27 / 27 / 27
//           theta 0.8 r 0.9            8.1 / 8.0 / 7.1 / 5.1 / 4.8
//           theta 0.99, 512 in flight  1.00 / 1.05 / 0.94 / 0.64 / 0.64
// The latch variants keep the switch of 2PL.
__host__ __device__ constexpr unsigned ordered_after(int s) {
    return (s == S_SILO || s == S_TICTOC || s == S_SLOW_SILO || s == S_SLOW_TICTOC) ? 0xFFFFFFFFu
           : s == S_TO                                                              ? 130u
           : (is_tpl(s) || s == S_SLOW_TO)                                          ? 16u
           : (s == S_MVCC || s == S_SLOW_MVCC)                                      ? 8u
                                                                                    : 1u;
}

// ===========================================================================
// The persistent transaction kernel. Without contention it is bound by the
// round trips that follow one another in a transaction (ticket, record, index,
// lock word, rows, release; 32 warps an SM do not cover them) and by the L2
// requests behind them, not by DRAM (13 % of its bandwidth) or by issue slots
// (41 % before the changes below). What takes a trip or a request out of the
// chain pays: one 32-byte load per sector, an image's loads issued together,
// both kinds of lock RMW in flight at once, acquire RMWs instead of fences, one
// fence per release for all lanes, the record's slots read beside its count,
// error and admission flags in one load after the previous commit, write values
// hashed before anything is held, sums of the metrics per warp instead of per
// CTA.
// Measured, 10,485,760 rows, r 0.9, wd 5, M tx/s before -> after:
//   theta 0.1  tpl_nw 310 -> 402, to 204 -> 261, silo 341 -> 456, tictoc 335 -> 420
//   theta 0.6  tpl_nw 95 -> 121, tpl_wd 110 -> 148, to 91 -> 174, silo 246 -> 317
// Tried without gain: taking the next ticket (and prefetching its record)
// during the current transaction (-3 ... -10 %), prefetching rows to L2 while
// their locks are on the way (-5 % on tables past the TLB's reach).
// ===========================================================================
// Dynamic shared memory of a CTA: the metric sums, a row per warp, and three
// words per group. By the launch's own size: sized for 1,024 threads they cost
// small CTAs residency (warp_density 0, block_size 1: 7 CTAs an SM instead of
// 32; theta 0.1 103 -> 129 M tx/s).
inline size_t ycsb_shared_bytes(int G, int block) {
    return (size_t)(block / 32 * 8 + block / G * 3) * sizeof(unsigned long long);
}

template <int SCH, int G, int MO = kMaxOps>
__global__ void __launch_bounds__(1024, 1) ycsb_kernel(const __grid_constant__ KParams p) {
    // Block-level histogram and metric sums (flushed once at exit) keep the
    // per-thread register budget for the transaction itself.
    __shared__ unsigned s_hist[kHistBuckets];
    extern __shared__ unsigned long long s_dyn[];  // ycsb_shared_bytes
    unsigned long long(*const s_met)[8] = (unsigned long long(*)[8])s_dyn;  // a row per warp
    // what a group's leader keeps through an attempt: start of the transaction
    // (clock, ns) and of the attempt (not in registers: every lane's count)
    unsigned long long(*const s_begin)[3] = (unsigned long long(*)[3])(s_met + blockDim.x / 32);
    __shared__ uint32_t s_turn_ns;
    if (is_ordered(SCH) && threadIdx.x == 0) s_turn_ns = turn_sleep_ns(p.ctr);
    for (int i = threadIdx.x; i < kHistBuckets; i += blockDim.x) s_hist[i] = 0u;
    for (unsigned i = threadIdx.x; i < blockDim.x / 32 * 8; i += blockDim.x) s_dyn[i] = 0ull;
    __syncthreads();

    const Group<G> g;
    using TX = TxOps<G, MO>;
    constexpr int K = TX::K;

    // Positions come from 32 striped ticket counters (stripe j hands out
    // j, j + 32, j + 64, ... in increasing order, each counter on its own
    // 128-byte line): one same-address atomic per transaction on a single
    // counter was the main latency term at low contention. A group starts on
    // stripe (group id % 32) and moves to the next stripe when its stripe is
    // exhausted. Within a stripe positions are taken in order and a group
    // runs one position at a time, so the lowest unfinished position is
    // always held by a running group (the ordered schemes' hand-off stays
    // live).
    const unsigned gid = (blockIdx.x * blockDim.x + threadIdx.x) / G;
    unsigned stripe = gid % kTicketStripes, tried = 0;
    auto ticket = [&]() { return (uint32_t)atomicAdd(&p.ctr->tickets[stripe * 16], 1ull); };
    uint2 es = make_uint2(0u, 0u);  // leader: {err, starving} after its last transaction
    if (g.glane == 0) es = ld_err_starving(p.ctr);
    while (true) {
        uint32_t pos = 0;
        unsigned stop = 0;
        if (g.glane == 0) {
            // admission pause: while some transaction is starving (it has
            // aborted starve_limit times), start no new transaction, so the
            // contention around it drains and it commits. The pause is
            // advisory: after spin_limit_ns admissions resume regardless.
            if (p.starve_limit && es.y != 0u) {
                const uint64_t tw = gtimer();
                while (true) {
                    es = ld_err_starving(p.ctr);
                    if (es.y == 0u || es.x != 0u || expired(tw, p.spin_limit_ns)) break;
                    __nanosleep(1000);
                }
            }
            pos = ticket() * kTicketStripes + stripe;
            while (pos >= p.batch_n) {
                if (++tried >= kTicketStripes) { stop = 1u; break; }
                stripe = (stripe + 1) % kTicketStripes;
                pos = ticket() * kTicketStripes + stripe;
            }
            // device queue: wait (bounded) until the position is admitted
            if (!stop && p.queue_tail) {
                const uint64_t tq = gtimer();
                while (pos >= *p.queue_tail) {
                    if (error_raised(p.ctr) || expired(tq, p.spin_limit_ns)) {
                        set_error(p.ctr, GCC_ETIMEOUT, W_QUEUE);
                        stop = 1u;
                        break;
                    }
                    __nanosleep(256);
                }
            }
            if (es.x) stop = 1u;
        }
        stop = g.bcast(stop, 0);
        if (stop) break;
        pos = g.bcast(pos, 0);
        const uint32_t tx = p.order ? __ldg(p.order + p.batch_st + pos) : p.batch_st + pos;
        unsigned long long *const sum = s_met[threadIdx.x >> 5];
        unsigned long long *const begin = s_begin[threadIdx.x / G];
        auto add_to = [&](int j, unsigned long long v) {
            if (G == 32) sum[j] += v;  // the warp's only writer
            else atomicAdd(sum + j, v);
        };
        if (g.glane == 0) {
            begin[0] = (unsigned long long)clock64();
            begin[1] = gtimer();
        }

        // ---- requests and index probes --------------------------------
        TX s;
        unsigned long long n64;
        constexpr bool kEarly = MO == kMaxOps && K <= 2;
        int2 rq[kEarly ? K : 1];
        const gcc_ycsb_tx *T = nullptr;
        uint32_t beg = 0;
        if constexpr (MO == kMaxOps) {
            T = p.txs + tx;
            // With a device queue the records of later batches are still
            // being copied in while earlier ones run: read them through L2
            // (a line cached in L1 next to an earlier record could predate
            // the copy).
            n64 = p.queue_tail ? __ldcg((const unsigned long long *)&T->request_cnt)
                               : __ldg(&T->request_cnt);
            // the slots are there whatever the count: no wait for it (where a
            // lane has few, so that they fit its registers)
            if constexpr (kEarly) {
#pragma unroll
                for (int k = 0; k < K; ++k)
                    if (g.glane + k * G < kMaxOps)
                        rq[k] = p.queue_tail ? __ldcg((const int2 *)&T->requests[g.glane + k * G])
                                             : __ldg((const int2 *)&T->requests[g.glane + k * G]);
            }
        } else {
            beg = __ldg(p.tx_off + tx);
            n64 = (unsigned long long)(__ldg(p.tx_off + tx + 1) - beg);
        }
        if (n64 > (unsigned long long)MO) {
            if (g.glane == 0) set_error(p.ctr, GCC_EFORMAT, 0);
            break;
        }
        s.n = (uint32_t)n64;
        s.valid = s.isread = 0;
        s.obst_op = 0;
        s.attempts = 0;
        if (is_ordered(SCH)) s.turn_ns = s_turn_ns;
        s.crowded = false;
        bool miss = false;
        typename TX::Mask myreads = 0;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const uint32_t i = g.glane + k * G;
            s.row[k] = kNoRow;
            if (i < s.n) {
                int2 q;
                if constexpr (kEarly) q = rq[k];
                else if constexpr (MO != kMaxOps) q = __ldg((const int2 *)(p.reqs + beg + i));
                else q = p.queue_tail ? __ldcg((const int2 *)&T->requests[i])
                                      : __ldg((const int2 *)&T->requests[i]);
                s.valid |= 1u << k;
                if (q.x > 0) { s.isread |= 1u << k; myreads |= (typename TX::Mask)1 << i; }
                if constexpr (is_ordered(SCH)) {
                    s.row[k] = __ldg(p.op_row + (uint64_t)pos * p.slot_ops + i);
                } else {
                    s.row[k] = index_find(p, (uint32_t)q.y);
                }
                miss |= s.row[k] == kNoRow;
            }
        }
        s.readmask = g.orv(myreads);
        if (K == 1 && p.write_mode == GCC_WRITE_FIELD && (s.valid & ~s.isread & 1u)) {
            s.wfield = write_field(p.write_seed, tx, g.glane);
            s.wval = write_value(p.write_seed, tx, g.glane);
        }
        if (g.any(miss)) {
            if (g.glane == 0) set_error(p.ctr, GCC_EKEY, 0);
            break;
        }
        if (g.glane == 0) add_to(7, (unsigned long long)clock64() - begin[0]);

        // ---- attempt / retry loop (benchmark/ycsb.cu:51-106) -------------
        unsigned attempts = 0;
        int st = kGiveUp;
        Clocks ck{0, 0};
        unsigned long long dg = 0;
        bool starving = false;
        // (the caller's ordered_from applies to the schemes that switch, 2PL / TO)
        const unsigned ord_from = (p.ordered_from && (is_tpl(SCH) || SCH == S_TO || SCH == S_SLOW_TO))
                                      ? p.ordered_from - 1u : ordered_after(SCH);
        while (true) {
            dg = 0;
            if (g.glane == 0) begin[2] = (unsigned long long)clock64();
            st = attempt<SCH, G>(p, g, s, tx, pos, dg, ck, attempts >= ord_from);
            if (st != kAbort) break;
            s.attempts = ++attempts;
            if (p.starve_limit && attempts == p.starve_limit) {
                starving = true;
                if (g.glane == 0) atomicAdd(&p.ctr->starving, 1u);
            }
            // a starving TO transaction retries in request order (see
            // attempt_to); starving 2PL ones keep the failed lock last, which
            // is what lets the hot rows' writers through
            if constexpr (SCH == S_TO) {
                if (starving) s.obst_op = 0;
            }
            // A transaction still aborting after 4 x starve_limit attempts
            // retries only while it holds the starvation token: the others
            // at that stage wait between attempts, holding nothing, so the
            // holder meets only the in-flight work below that stage, which
            // drains (admissions are paused) or reaches it in turn. One
            // holder at a time guarantees progress for transactions whose
            // retries would otherwise keep invalidating each other.
            if (starving && attempts >= 4u * p.starve_limit) {
                unsigned bad = 0;
                if (g.glane == 0) {
                    const unsigned me = tx + 1u;
                    const uint64_t tw = gtimer();
                    while (true) {
                        const unsigned h = atomicCAS(&p.ctr->starve_token, 0u, me);
                        if (h == 0u || h == me) break;
                        if (error_raised(p.ctr)) { bad = 1; break; }
                        if (expired(tw, p.spin_limit_ns)) {
                            set_error(p.ctr, GCC_ETIMEOUT, W_STARVE);
                            bad = 1;
                            break;
                        }
                        __nanosleep(1000);
                    }
                }
                if (g.bcast(bad, 0)) { st = kGiveUp; break; }
            }
            // After 8 failed attempts, a short random pause (up to
            // backoff_ns, at most a few microseconds) breaks the symmetric
            // retry patterns that lock-step warps can otherwise repeat
            // forever, e.g. two OCC transactions that each read what the
            // other writes and abort on each other's write lock. It is kept
            // short because a batch ends with its slowest transaction. The
            // commit rule is untouched.
            if (p.backoff_ns && attempts >= 8u)
                __nanosleep((unsigned)(hash3(tx, attempts, 0x5ull) % p.backoff_ns));
            unsigned late = 0;
            if (g.glane == 0) {
                add_to(4, (unsigned long long)clock64() - begin[2]);
                es = ld_err_starving(p.ctr);
                late = expired(begin[1], 4ull * p.spin_limit_ns) || es.x;
                if (late) set_error(p.ctr, GCC_ETIMEOUT, W_RETRY);
            }
            if (g.bcast(late, 0)) { st = kGiveUp; break; }
            if (is_tpl(SCH))
                s.crowded = !p.starve_limit ||
                            g.bcast(es.y, 0) * kCrowdShare * G >= gridDim.x * blockDim.x;
        }
        if (starving && g.glane == 0) {
            atomicCAS(&p.ctr->starve_token, tx + 1u, 0u);
            atomicSub(&p.ctr->starving, 1u);
        }
        if (st == kGiveUp) break;
        if (g.glane == 0) es = ld_err_starving(p.ctr);  // for the next one's admission
        dg = g.sum(dg);
        if (g.glane == 0) {
            const long long c_end = clock64();
            p.digest[tx] = dg;
            p.tx_aborts[tx] = attempts;
            if (attempts > 64) atomicMax(&p.ctr->max_attempts, attempts + 1u);
            add_to(0, 1ull);
            add_to(1, attempts);
            if (ck.ts) add_to(2, ck.ts);
            if (ck.wait) add_to(3, ck.wait);
            add_to(5, (unsigned long long)c_end - begin[2]);
            add_to(6, (unsigned long long)c_end - begin[0]);
            atomicAdd(&s_hist[hist_bucket(gtimer() - begin[1])], 1u);
        }
    }

    __syncthreads();
    if (threadIdx.x < 8) {
        Counters *c = p.ctr;
        unsigned long long sum = 0;
        for (unsigned w = 0; w < blockDim.x / 32; ++w) sum += s_met[w][threadIdx.x];
        unsigned long long *dst[8] = {&c->committed, &c->aborts, &c->ts_cycles, &c->wait_cycles,
                                      &c->abort_cycles, &c->mng_cycles, &c->tot_cycles,
                                      &c->idx_cycles};
        if (sum) atomicAdd(dst[threadIdx.x], sum);
    }
    for (int i = threadIdx.x; i < kHistBuckets; i += blockDim.x)
        if (s_hist[i]) atomicAdd(&p.ctr->hist[i], s_hist[i]);
}

// Launch helper implemented once per scheme translation unit.
cudaError_t launch_scheme(int scheme, int G, int grid, int block, const KParams &p,
                          cudaStream_t stream);
int occupancy_blocks(int scheme, int G, int block);

}  // namespace gcc
