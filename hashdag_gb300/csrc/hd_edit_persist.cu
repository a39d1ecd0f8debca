// Batched edits in one persistent launch: every edit of a batch, level by
// level, in a single cooperative kernel whose CTAs (one per SM) move through
// the levels together, with no host round trip and no kernel boundary.
//
// Same per-entry logic, same order of bucket scans and appends, hence the
// same table, as applying the edits one by one (hd_edit.cu): the edit of
// HashDAG::edit_threads (hash_dag.h:255-405) applied in sequence.  The work
// queue is ordered by level: for each edit, top-down levels (classify,
// spawn), then bottom-up levels (candidates, grouping by bucket,
// find-or-add).
//
//  * Levels are small near the root.  A level of at most kSmall entries is
//    processed by CTA 0 alone while the other CTAs wait at the next grid
//    barrier: consecutive small levels, the end of one edit and the start of
//    the next cost one barrier in all, or none when no grid step came
//    between (bottom-up, where an entry costs more: kSmallUp entries).
//  * A big level top-down is one grid phase: each CTA finds the descended
//    entries of its share of the children (per-chunk counts of descend flags
//    were gathered while the level was classified), spawns and classifies
//    them.
//  * A big level bottom-up is two phases: candidates, each put in the queue of
//    the CTA that owns its bucket (bucket modulo CTAs), then every CTA sorts
//    its queue and resolves its bucket runs, a warp each.  When a queue
//    overflows (many candidates of few buckets: a box's faces), it is four:
//    two stable radix passes on the level-local bucket (each CTA sums
//    the digit counts itself; pass-2 counts gathered while pass 1 scatters),
//    then find-or-add, one warp per bucket run; from kRepeatLevel candidates
//    on, the repeats and the runs' starts are marked before it.
//  * Grid barriers are bounded waits: a wait longer than kWaitNs sets
//    HD_ERR_TIMEOUT and every CTA returns; the host reports a batch's and makes
//    a single edit level by level.
//  * Nodes and pages that an edit appends are read by the following edits in
//    the same launch: every table read uses L2-coherent loads.
// The graph-per-edit form (hd_edit_batch.cu) stays as the other batch mode.
#include <algorithm>
#include <cstring>
#include <vector>

#include "hd_chunks.cuh"
#include "hd_edit.cuh"

namespace hd {

namespace {

constexpr uint32_t kPWarps = kPT / 32;
// Entries of a level that CTA 0 handles alone, top-down and bottom-up: a grid
// step costs a barrier (2.4-3.5 us), CTA 0 alone 4 us a level of 200 entries and
// 27 us bottom-up at 1,000 (its 32 warps resolve a bucket run in 1.5-2.5 us).
// Batches of 64 edits of radius 4-48 at 2^12 and 8-512 at 2^15: bottom-up limits
// of 128, 256, 512 and 1,024 give 5.78, 5.69, 5.72, 5.80 and 13.4, 13.4, 13.5,
// 13.7 ms; top-down ones of 256, 512 and 1,024 5.70, 5.68, 5.71 and 13.2, 13.1,
// 13.2 ms.
constexpr uint32_t kSmall = 512, kSmallUp = 256;
constexpr uint32_t kDigits = 512;          // radix digits per pass at most (9 bits)
static_assert(1u << (kMaxSortBits + 2) / 2 <= kDigits, "two passes sort every key");
// Candidates of a big level from which repeats are looked for (a grid step).
constexpr uint32_t kRepeatLevel = 4096;
constexpr unsigned long long kWaitNs = 2000000000ull;

enum : uint32_t { kRun = 0, kDone = 1, kCapacity = 2, kTableError = 3, kEmptyScene = 4, kAborted = 5 };

// What CTA 0 asks of the grid at a barrier.
struct Cmd {
    uint32_t stop, phase, level, deepest, idx, pad[3];
};

// Control block in global memory, reset by the host before a launch.
// stop / idx / phase / level / deepest are CTA 0's own state (stop and idx
// also read by the host after the launch); the other CTAs read the copy CTA 0
// publishes in cmd[k & 1] before barrier k.  CTA 0 runs ahead as soon as it
// leaves a barrier, so it must not change what the others are still about to
// read: it writes the slot of the next barrier, which no CTA reads until
// every CTA has left this one.
struct Ctl {
    unsigned long long arrived; // the grid barrier's word (hd_chunks.cuh)
    uint32_t stop;
    uint32_t idx;       // edit being applied
    uint32_t phase;     // the grid step CTA 0 asks for (kPh*)
    uint32_t level;     // its level
    uint32_t deepest;   // deepest level of the current edit
    uint32_t pad;       // (the commands on 8-byte boundaries)
    Cmd cmd[2];
    uint32_t ncand[HD_MAX_DEPTH]; // big levels: candidates for find-or-add
    uint32_t nruns[HD_MAX_DEPTH]; // big levels: long runs of repeats
    uint32_t nstarts[HD_MAX_DEPTH]; // big levels: listed bucket runs
    uint32_t count[HD_MAX_DEPTH];
    // where a wait ran out: the CTA, its barrier count, the arrivals then and
    // the count it waited for, CTA 0's barrier count, phase, level and edit
    uint32_t diag[8];
    uint32_t bars0; // barriers CTA 0 has passed
    // tests of the timeout path (hd_set_test_barrier_skip): CTA skip_cta - 1
    // returns at once, never arriving (0: none); wait_ns bounds every
    // barrier wait (0: kWaitNs)
    uint32_t skip_cta;
    unsigned long long wait_ns;
    Editor ed;
};

// What one edit of the launch gives back.
struct EditOut {
    EditCounters ctr;
    uint32_t root, pad;
    unsigned long long t_begin, t_end;
};

// The launch's arguments, read where they are needed (a __grid_constant__
// parameter: the level arrays' pointers come from the constant bank).
struct PArgs {
    Ctl* ctl;
    const hd_edit* edits; // the batch, or null: the one edit `one`
    uint32_t n_edits;
    uint32_t hold_root;   // the new root goes to the edit's EditOut only (its colours come first)
    Editor one;
    Level lv[HD_MAX_DEPTH];
    uint32_t cap[HD_MAX_DEPTH];
    uint32_t *keys, *vals, *keys2, *vals2;
    uint32_t* bsum;      // 3 x G: per-chunk descend-flag counts, by level parity
    unsigned long long* queue; // G x kPT: bucket << 32 | entry of the candidates a CTA owns
    uint32_t* queued;    // HD_MAX_DEPTH x G: their numbers, by level
    uint32_t *hist, *hist2; // G x kDigits: a big level's digit counts per chunk
    uint32_t *rows, *rows2; // kDigits: their totals
    uint32_t* same;      // a big level's repeats, a bit per sorted candidate
    FollowerRun* runs;   // its long runs of repeats
    EditOut* out;
    uint32_t* d_root;
};

HD_D unsigned long long now_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
HD_D uint32_t ld_acquire(const uint32_t* p)
{
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
HD_D unsigned long long ld_acquire64(const unsigned long long* p)
{
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// Grid barrier of the cooperative launch with a bounded wait; false when a
// wait ran out or another CTA gave up (the caller returns).  The arrival
// count only grows (the control block starts at zero every launch), so the
// k-th barrier is passed once k x CTAs have arrived: no reset, and no
// generation word for the last CTA to publish after its arrival.  Arrivals and
// the flag of a CTA that gave up are one 64-bit word, which every access to it
// takes whole: an acquire of a word orders nothing behind an atomic of half of
// it.  Bound by L2 round trips: a poll is one acquire, without a pause until it
// has waited long (with two reads and a pause a poll, and a fence after, a grid
// step of almost no work took 2.7-4.3 us, now 2.4-3.5).
HD_D bool grid_sync(Ctl* ctl, uint32_t* err, uint32_t& nbar)
{
    __shared__ uint32_t ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = 1;
        nbar++;
        if (blockIdx.x == 0)
            __stcg(&ctl->bars0, nbar);
        const unsigned long long target = barrier_target(nbar, gridDim.x);
        __threadfence();
        if (barrier_arrivals(atomicAdd(&ctl->arrived, 1ull)) + 1 == target) {
            __threadfence(); // the last to arrive acquires here
        } else {
            unsigned long long t0 = 0;
            uint32_t spins = 0;
            for (;;) {
                const unsigned long long word = ld_acquire64(&ctl->arrived);
                if (barrier_arrivals(word) >= target)
                    break;
                if (barrier_aborted(word)) {
                    ok = 0;
                    break;
                }
                if ((++spins & 255u) == 0) {
                    if (!t0)
                        t0 = now_ns();
                    const unsigned long long set_ns = __ldcg(&ctl->wait_ns);
                    const unsigned long long limit = set_ns ? set_ns : kWaitNs;
                    if (now_ns() - t0 > limit) {
                        if (!barrier_aborted(atomicOr(&ctl->arrived, kBarrierAbort))) {
                            ctl->diag[0] = blockIdx.x;
                            ctl->diag[1] = nbar;
                            ctl->diag[2] = uint32_t(barrier_arrivals(ld_acquire64(&ctl->arrived)));
                            ctl->diag[3] = uint32_t(target);
                            ctl->diag[4] = ld_acquire(&ctl->bars0);
                            ctl->diag[5] = ld_acquire(&ctl->phase);
                            ctl->diag[6] = ld_acquire(&ctl->level);
                            ctl->diag[7] = ld_acquire(&ctl->idx);
                        }
                        set_error(err, kErrTimeout, 0xFFFFFFFEu, blockIdx.x, 0);
                        ok = 0;
                        break;
                    }
                }
                if (spins > 64)
                    __nanosleep(64);
            }
        }
    }
    __syncthreads();
    return ok != 0;
}

// Block-wide exclusive scan (kPT threads) of v; *total = the block's sum.
HD_D uint32_t cta_scan(uint32_t v, uint32_t* total, uint32_t* sm32)
{
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t inc = warp_incl_scan(v);
    if (lane == 31)
        sm32[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const uint32_t s = warp_incl_scan(sm32[lane]);
        sm32[lane] = s;
    }
    __syncthreads();
    const uint32_t base = warp ? sm32[warp - 1] : 0u;
    *total = sm32[kPWarps - 1];
    __syncthreads();
    return base + inc - v;
}

// Top-down: entries [i0, i1) of level L (classified, their descend flags
// set): exclusive positions from `prefix` (descended entries before i0),
// then every child of every descended entry spawned at 8 * exp + c and
// classified; children's descend flags are counted per top-down chunk of
// level L + 1 into cnt_next.  CTA-wide.
HD_D void td_range(const Table& t, const Editor& ed, const Level& lv, const Level& nx, uint32_t L, uint32_t i0,
                   uint32_t i1, uint32_t prefix, uint32_t n_next, uint32_t G, uint32_t* cnt_next, EditCounters* ctr,
                   uint32_t* sm32, uint32_t* list)
{
    const uint32_t lane = threadIdx.x & 31;
    uint32_t run = prefix;
    unsigned long long nodes = 0, voxels = 0;
    for (uint32_t base = i0; base < i1; base += kPT) {
        const uint32_t i = base + threadIdx.x;
        const uint32_t f = i < i1 ? lv.flag[i] : 0u;
        uint32_t total;
        const uint32_t off = cta_scan(f, &total, sm32);
        if (f) {
            lv.exp[i] = run + off;
            list[off] = i;
        }
        __syncthreads();
        // the tile's children, spread over the CTA, warps in lockstep
        const uint32_t nchild = 8 * total;
        for (uint32_t k0 = threadIdx.x & ~31u; k0 < nchild; k0 += kPT) {
            const uint32_t k = k0 + lane;
            const bool act = k < nchild;
            uint32_t fl = 0, ch = 0xFFFFFFFFu;
            if (act) {
                const uint32_t parent = list[k >> 3], c = k & 7;
                const uint32_t at = 8 * (run + (k >> 3)) + c;
                uint32_t x, y, z, old;
                spawn_child(t, lv, nx, parent, c, at, x, y, z, old);
                unsigned long long nn, vv;
                classify_values<true>(t, ed, L + 1, nx, at, x, y, z, old, nn, vv);
                nodes += nn;
                voxels += vv;
                fl = nx.flag[at];
                ch = td_chunk(at, n_next, G);
            }
            // the warp's children are 32 consecutive slots (at = 8 run + k),
            // so they fall in at most two chunks (chunks hold >= 32 slots):
            // one atomic per chunk; flags are 0 or 1
            const uint32_t ch0 = __shfl_sync(0xffffffffu, ch, 0);
            const uint32_t b0 = __ballot_sync(0xffffffffu, act && fl && ch == ch0);
            const uint32_t b1 = __ballot_sync(0xffffffffu, act && fl && ch != ch0);
            if (lane == 0 && b0)
                atomicAdd(cnt_next + ch0, uint32_t(__popc(b0)));
            if (b1 && lane == uint32_t(__ffs(b1) - 1))
                atomicAdd(cnt_next + ch, uint32_t(__popc(b1)));
        }
        run += total;
        __syncthreads();
    }
    warp_add(&ctr->num_nodes, nodes);
    warp_add(&ctr->num_voxels, voxels);
}

// The grid's top-down step of a big level: children [k0, k1) of the level
// (child k: slot k % 8 of the descended entry of rank k / 8) spawned and
// classified, so that the children (and the work of classifying them) spread
// evenly over the CTAs whatever chunks the descended entries fall in.  A CTA
// finds its ranks' entries itself, kListRanks at a time: cnt holds the
// descended entries per chunk of the level, and only the flags of the chunks
// that hold its ranks are scanned (a phase of its own for the ranks, listed in
// global memory, cost 4-5 us a level).  k0 is a multiple of 32, so each warp's
// 32 consecutive children fall in at most two chunks of the next level, whose
// descend flags are counted into cnt_next.
constexpr uint32_t kListRanks = 4096;
HD_D void td_children(const Table& t, const Editor& ed, const Level* lvs, uint32_t L, uint32_t n, uint32_t k0,
                      uint32_t k1, uint32_t n_next, uint32_t G, const uint32_t* cnt, uint32_t* cnt_next,
                      EditCounters* ctr, uint32_t* sm32, uint32_t* list, uint32_t* chunk_end)
{
    const Level lv = lvs[L], nx = lvs[L + 1];
    const uint32_t lane = threadIdx.x & 31;
    unsigned long long nodes = 0, voxels = 0;
    const uint32_t chunk = chunk_len(n, G, kChunkAlign);
    // chunk_end[b]: descended entries in chunks 0 .. b
    for (uint32_t b0 = 0, run = 0; b0 < G; b0 += kPT) {
        const uint32_t b = b0 + threadIdx.x;
        const uint32_t c = b < G ? __ldcg(cnt + b) : 0u;
        uint32_t total;
        const uint32_t before = cta_scan(c, &total, sm32);
        if (b < G)
            chunk_end[b] = run + before + c;
        run += total;
    }
    __syncthreads();
    for (uint32_t r0 = k0 / 8; r0 < k1 / 8; r0 += kListRanks) {
        const uint32_t r1 = min(k1 / 8, r0 + kListRanks);
        // the chunks that hold ranks [r0, r1)
        uint32_t b0 = 0, b1 = 0;
        for (uint32_t base = 0; base < G; base += kPT) {
            const uint32_t b = base + threadIdx.x;
            b0 += __syncthreads_count(b < G && chunk_end[b] <= r0);
            b1 += __syncthreads_count(b < G && (b ? chunk_end[b - 1] : 0u) < r1);
        }
        for (uint32_t b = b0; b < b1; b++) {
            const uint32_t before = b ? chunk_end[b - 1] : 0u;
            const uint32_t i1 = min(n, (b + 1) * chunk);
            uint32_t run = before;
            for (uint32_t base = b * chunk; base < i1 && run < r1; base += kPT) {
                const uint32_t i = base + threadIdx.x;
                const uint32_t f = i < i1 ? lv.flag[i] : 0u;
                uint32_t total;
                const uint32_t rank = run + cta_scan(f, &total, sm32);
                if (f && rank >= r0 && rank < r1) {
                    lv.exp[i] = rank;
                    list[rank - r0] = i;
                }
                run += total;
            }
        }
        __syncthreads();
        const uint32_t ke = 8 * r1;
        for (uint32_t kb = 8 * r0 + (threadIdx.x & ~31u); kb < ke; kb += kPT) {
            const uint32_t k = kb + lane;
            const bool act = k < ke;
            uint32_t fl = 0, ch = 0xFFFFFFFFu;
            if (act) {
                uint32_t x, y, z, old;
                spawn_child(t, lv, nx, list[(k >> 3) - r0], k & 7, k, x, y, z, old);
                unsigned long long nn, vv;
                classify_values<true>(t, ed, L + 1, nx, k, x, y, z, old, nn, vv);
                nodes += nn;
                voxels += vv;
                fl = nx.flag[k];
                ch = td_chunk(k, n_next, G);
            }
            const uint32_t ch0 = __shfl_sync(0xffffffffu, ch, 0);
            const uint32_t b0 = __ballot_sync(0xffffffffu, act && fl && ch == ch0);
            const uint32_t b1 = __ballot_sync(0xffffffffu, act && fl && ch != ch0);
            if (lane == 0 && b0)
                atomicAdd(cnt_next + ch0, uint32_t(__popc(b0)));
            if (b1 && lane == uint32_t(__ffs(b1) - 1))
                atomicAdd(cnt_next + ch, uint32_t(__popc(b1)));
        }
        __syncthreads();
    }
    warp_add(&ctr->num_nodes, nodes);
    warp_add(&ctr->num_voxels, voxels);
}

// ---- tiny levels ----------------------------------------------------------------
// The levels near the root hold a few entries, and an edit of any size passes
// through all of them twice, each step waiting for the one before.  Levels of
// at most kTiny entries that such a level spawned keep their arrays in CTA 0's
// shared memory (the level arrays proper are written at the edit's end, and
// only when its colours will read them), a lane an entry: what is left of a
// level's chain is the table itself, two reads down (a node with its child
// pointers, the old child's count) and two or three up (a bucket's size with
// its filters, a page, a claim).  With the arrays in global memory, nodes read
// word after word, a sort and CTA barriers a level took 1.6 us down and 5-6 us
// up, now 0.9 and 3-4.5: an edit of radius 11 at 2^15 goes from 115 to 86 us.
constexpr uint32_t kTiny = 32;
struct __align__(16) TinyLevel {
    uint32_t x[kTiny], y[kTiny], z[kTiny], old[kTiny], res[kTiny], cnt[kTiny], flag[kTiny], exp[kTiny];
    uint8_t state[kTiny];
};
struct TinyState {
    TinyLevel lv[HD_MAX_DEPTH];
    uint32_t rows[kTiny * kRow]; // the candidates of the level being resolved
    uint32_t sk[kTiny], sv[kTiny], rs[kTiny + 1]; // sorted, and their bucket runs' starts
    uint32_t held;               // bit L: level L is held here
    uint32_t failed;             // an append of the edit failed
    uint32_t list[kTiny];        // descended entries by rank
    uint32_t level, status, runs; // what the warp reports
    uint32_t count[HD_MAX_DEPTH]; // CTA 0's copy of the entry counts
};

// Level L's arrays: the shared ones when it is held there
HD_D Level held_level(const PArgs& a, const TinyState& ts, uint32_t L)
{
    Level l = a.lv[L];
    if ((ts.held >> L) & 1u) {
        TinyLevel& m = const_cast<TinyLevel&>(ts.lv[L]);
        l.x = m.x, l.y = m.y, l.z = m.z, l.old = m.old, l.res = m.res, l.cnt = m.cnt, l.flag = m.flag, l.exp = m.exp;
        l.state = m.state;
    }
    return l;
}

// Top-down, one warp of CTA 0 alone: consecutive held levels whose children
// are at most kTiny (td_range's step: ranks, children spawned and classified).
// A node is read with its 8 possible child pointers at once, a word a lane,
// and each child takes its pointer from the lane that has it.  Returns the
// first level it did not descend from; status 0: the level has more children
// (or is the leaf level), 1: it had no descended entry (it is the deepest), 2:
// its children would exceed their level's capacity.
HD_D uint32_t td_tiny(const Table& t, const Editor& ed, const PArgs& a, TinyState& ts, uint32_t L, EditCounters* ctr,
                      uint32_t& status)
{
    const uint32_t lane = threadIdx.x & 31, leafl = t.g.leaf_level;
    unsigned long long nodes = 0, voxels = 0;
    status = 0;
    while (L < leafl) {
        TinyLevel& m = ts.lv[L];
        const uint32_t fb = __ballot_sync(0xffffffffu, lane < ts.count[L] && m.flag[lane]);
        const uint32_t n_next = 8 * __popc(fb);
        if (n_next == 0) {
            status = 1;
            break;
        }
        if (n_next > a.cap[L + 1]) {
            status = 2;
            break;
        }
        if (n_next > kTiny)
            break;
        if ((fb >> lane) & 1u) {
            const uint32_t rank = __popc(fb & ((1u << lane) - 1u));
            m.exp[lane] = rank;
            ts.list[rank] = lane;
        }
        if (lane == 0) {
            ts.held |= 1u << (L + 1);
            ts.count[L + 1] = n_next;
            a.ctl->count[L + 1] = n_next;
        }
        __syncwarp();
        const uint32_t c = lane & 7;
        const bool act = lane < n_next;
        uint32_t x = 0, y = 0, z = 0, old = kInvalid, head = 0, word = 0;
        if (act) {
            const uint32_t p = ts.list[lane >> 3];
            x = (m.x[p] << 1) | ((c >> 2) & 1);
            y = (m.y[p] << 1) | ((c >> 1) & 1);
            z = (m.z[p] << 1) | (c & 1);
            const uint32_t node = m.old[p];
            if (node != kInvalid) {
                const uint32_t* w = t.sys_cg(node);
                head = __ldcg(w);
                word = __ldcg(w + 1 + c); // (past a smaller node's end: not used)
            }
        }
        const uint32_t from = (lane & ~7u) + popc32(head & ((1u << c) - 1u));
        const uint32_t child = __shfl_sync(0xffffffffu, word, from);
        if ((head >> c) & 1u)
            old = child;
        if (act) {
            TinyLevel& k = ts.lv[L + 1];
            k.x[lane] = x;
            k.y[lane] = y;
            k.z[lane] = z;
            k.old[lane] = old;
            unsigned long long nn, vv;
            classify_values<true>(t, ed, L + 1, held_level(a, ts, L + 1), lane, x, y, z, old, nn, vv);
            nodes += nn;
            voxels += vv;
        }
        __syncwarp(); // the next level reads the flags other lanes wrote
        L++;
    }
    warp_add(&ctr->num_nodes, nodes);
    warp_add(&ctr->num_voxels, voxels);
    return L;
}

// Bottom-up, one warp: candidates of level L (at most kTiny entries, a lane
// each; held or not) into ts.rows, grouped by bucket without a sort: the
// lanes of a bucket know each other, groups are in the order of their first
// lanes, and a group's lanes are in entry order.  Returns the bucket runs.
HD_D uint32_t tiny_candidates(const Table& t, const PArgs& a, TinyState& ts, uint32_t L, uint32_t deepest, uint32_t n)
{
    const uint32_t lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    Level lv = held_level(a, ts, L);
    lv.cand = ts.rows;
    const Level child = L < deepest ? held_level(a, ts, L + 1) : Level{};
    const uint32_t key = lane < n ? candidate_entry<true>(t, L, lv, child, lane) : kNoBucket;
    const uint32_t cb = __ballot_sync(0xffffffffu, key != kNoBucket);
    if (!cb) {
        // entries resolved at once: the level above reads their results on
        // other lanes
        __syncwarp();
        return 0;
    }
    const uint32_t peers = __match_any_sync(0xffffffffu, key) & cb;
    const bool lead = key != kNoBucket && (peers & lt) == 0;
    const uint32_t leads = __ballot_sync(0xffffffffu, lead);
    // candidates of the groups before: their sizes summed at their leaders
    const uint32_t end = warp_incl_scan(lead ? uint32_t(__popc(peers)) : 0u);
    const uint32_t first = __shfl_sync(0xffffffffu, end, key != kNoBucket ? __ffs(peers) - 1 : 0) - __popc(peers);
    if (key != kNoBucket) {
        const uint32_t at = first + __popc(peers & lt);
        ts.sk[at] = key;
        ts.sv[at] = lane;
        if (lead)
            ts.rs[__popc(leads & lt)] = at;
    }
    if (lane == 0)
        ts.rs[__popc(leads)] = __popc(cb);
    __syncwarp();
    return __popc(leads);
}

// Bottom-up candidates of entries [i0, i1) of level L: key = level-local
// bucket, or buckets(L) (sorts last) for entries resolved at once.
HD_D void candidates_range(const Table& t, const Level* lvs, uint32_t L, uint32_t deepest, uint32_t i0, uint32_t i1,
                           uint32_t* keys, uint32_t* vals)
{
    const Level lv = lvs[L];
    const Level child = L < deepest ? lvs[L + 1] : Level{};
    const uint32_t empty = t.g.buckets(L);
    for (uint32_t i = i0 + threadIdx.x; i < i1; i += kPT) {
        const uint32_t b = candidate_entry<true>(t, L, lv, child, i);
        keys[i] = b == kNoBucket ? empty : b;
        vals[i] = i;
    }
}

HD_D void foa_counts(const Table& t, uint32_t L, EditCounters* ctr, unsigned long long foa, unsigned long long added,
                     unsigned long long scanned)
{
    if ((threadIdx.x & 31) == 0 && (foa | added | scanned)) {
        atomicAdd(&ctr->foa, foa);
        atomicAdd(&ctr->added, added);
        atomicAdd(&ctr->scanned, scanned);
        atomicAdd(reinterpret_cast<unsigned long long*>(t.level_nodes + L), added);
    }
}

// Find-or-add of a small level: its bucket runs (starts[r] .. starts[r + 1] of
// the sorted candidates) dealt out to the nw warps in turn.
template <int PW>
HD_D void foa_runs(const Table& t, uint32_t L, const Level& lv, const uint32_t* keys, const uint32_t* vals,
                   const uint32_t* starts, uint32_t runs, uint32_t w, uint32_t nw, uint32_t* page, uint32_t* q,
                   FoaCache& cache, EditCounters* ctr, uint32_t* failed = nullptr)
{
    unsigned long long foa = 0, added = 0, scanned = 0;
    for (uint32_t r = w; r < runs; r += nw) {
        const uint32_t j0 = starts[r], j1 = starts[r + 1];
        if (!foa_segment<PW>(t, L, lv, vals, j0, j1, keys[j0], page, q, cache, foa, added, scanned) && failed)
            *failed = 1;
    }
    foa_counts(t, L, ctr, foa, added, scanned);
}

// Find-or-add over the sorted keys [0, n) of a big level (runs of one bucket
// in entry order; n: its candidates): the positions are split into one chunk
// per warp (ceil(n / nw), at least one) and warp w of nw resolves every run
// that starts in its chunk, so that short runs spread over all the warps.
// The arrays were written in another phase: read from L2.
template <int PW>
HD_D void foa_sorted(const Table& t, uint32_t L, const Level& lv, const uint32_t* keys, const uint32_t* vals,
                     uint32_t n, uint32_t w, uint32_t nw, uint32_t* page, uint32_t* q, FoaCache& cache,
                     EditCounters* ctr)
{
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t empty = t.g.buckets(L);
    unsigned long long foa = 0, added = 0, scanned = 0;
    const uint32_t chunk = n > nw ? (n + nw - 1) / nw : 1u;
    const uint64_t cbeg64 = uint64_t(w) * chunk;
    const uint32_t cbeg = cbeg64 < n ? uint32_t(cbeg64) : n, cend = n - cbeg < chunk ? n : cbeg + chunk;
    for (uint32_t c0 = cbeg; c0 < cend; c0 += 32) {
        const uint32_t j = c0 + lane;
        const bool in = j < cend;
        const uint32_t key = in ? __ldcg(keys + j) : empty;
        const uint32_t prev = (in && j > 0) ? __ldcg(keys + j - 1) : kNoBucket;
        uint32_t starts = __ballot_sync(0xffffffffu, in && key < empty && key != prev);
        while (starts) {
            const uint32_t s = __ffs(starts) - 1;
            starts &= starts - 1;
            const uint32_t j0 = c0 + s;
            const uint32_t bucket = __shfl_sync(0xffffffffu, key, s);
            // the run's end: 128 keys at a time
            uint32_t j1 = j0 + 1;
            for (;;) {
                uint32_t k[4];
#pragma unroll
                for (uint32_t m = 0; m < 4; m++)
                    k[m] = j1 + 32 * m + lane < n ? __ldcg(keys + j1 + 32 * m + lane) : kNoBucket;
                uint32_t same = 128; // keys before the first other one
#pragma unroll
                for (int m = 3; m >= 0; m--) {
                    const uint32_t diff = __ballot_sync(0xffffffffu, k[m] != bucket);
                    same = diff ? 32 * m + __ffs(diff) - 1 : same;
                }
                j1 += same;
                if (same < 128)
                    break;
            }
            foa_segment<PW>(t, L, lv, vals, j0, j1, bucket, page, q, cache, foa, added, scanned);
        }
    }
    foa_counts(t, L, ctr, foa, added, scanned);
}

// Find-or-add of a big level whose repeats are known: its bucket runs, listed
// by their starts in any order, dealt out to the nw warps in turn.
template <int PW>
HD_D void foa_listed(const Table& t, uint32_t L, const Level& lv, const uint32_t* keys, const uint32_t* vals, uint32_t n,
                     const uint32_t* starts, uint32_t runs, uint32_t w, uint32_t nw, uint32_t* page, uint32_t* q,
                     FoaCache& cache, EditCounters* ctr, const Repeats& rep)
{
    unsigned long long foa = 0, added = 0, scanned = 0;
    for (uint32_t r = w; r < runs; r += nw) {
        const uint32_t j0 = __ldcg(starts + r), bucket = __ldcg(keys + j0);
        uint32_t j1 = j0 + 1;
        do
            j1 = end_of_repeats(rep, j1);
        while (j1 < n && __ldcg(keys + j1) == bucket && ++j1 < n);
        j1 = min(j1, n);
        foa_segment<PW>(t, L, lv, vals, j0, j1, bucket, page, q, cache, foa, added, scanned, rep);
    }
    foa_counts(t, L, ctr, foa, added, scanned);
}

// Bit j of `same`: sorted candidate j has the bucket and the words of
// candidate j - 1 (positions [j0, j1), j0 a multiple of 32; n: candidates).
// A flat face of a box gives tens of thousands of equal candidates in one
// bucket; the warp that resolves them then steps over them by these bits, 1,024
// at a time, and leaves their results to the whole grid (fill_runs), where
// it compared and wrote them 32 at a time: the leaf level of a box of radius
// 250 (55,640 candidates) went from 1,063 to 94 us, the edit from 1.96 to 0.53
// ms.
// The bucket runs' starts are listed beside (starts / n_starts, in any order).
HD_D void mark_repeats(const Level& lv, bool leaf, const uint32_t* keys, const uint32_t* vals, uint32_t n, uint32_t j0,
                       uint32_t j1, uint32_t* same, uint32_t* starts, uint32_t* n_starts)
{
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t j = j0 + threadIdx.x; j - threadIdx.x < j1; j += kPT) {
        bool eq = false, start = false;
        if (j < j1) {
            start = j == 0 || __ldcg(keys + j) != __ldcg(keys + j - 1);
            if (!start)
                eq = same_row(lv.cand + kRow * uint64_t(__ldcg(vals + j)),
                              lv.cand + kRow * uint64_t(__ldcg(vals + j - 1)), leaf);
        }
        const uint32_t bits = __ballot_sync(0xffffffffu, eq), sb = __ballot_sync(0xffffffffu, start);
        if (lane == 0 && j < j1)
            same[j >> 5] = bits;
        uint32_t at = 0;
        if (lane == 0 && sb)
            at = atomicAdd(n_starts, uint32_t(__popc(sb)));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (start)
            starts[at + __popc(sb & ((1u << lane) - 1u))] = j;
    }
}

// The results of the long runs of repeats, by every warp of the grid: pieces
// of kPiece positions dealt out over all the runs (32 runs at a time: a lane
// holds one, its pieces counted by a prefix sum).
HD_D void fill_runs(const Level& lv, const uint32_t* vals, const FollowerRun* runs, uint32_t n)
{
    constexpr uint32_t kPiece = 256;
    const uint32_t lane = threadIdx.x & 31, nw = gridDim.x * kPWarps;
    const uint32_t gw = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    for (uint32_t r0 = 0; r0 < n; r0 += 32) {
        uint4 x = make_uint4(0, 0, 0, 0);
        if (r0 + lane < n)
            x = __ldcg(reinterpret_cast<const uint4*>(runs + r0 + lane));
        const uint32_t end = warp_incl_scan((x.y - x.x + kPiece - 1) / kPiece); // pieces up to this run's last
        const uint32_t all = __shfl_sync(0xffffffffu, end, 31);
        for (uint32_t p = gw; p < all; p += nw) {
            const uint32_t r = __popc(__ballot_sync(0xffffffffu, end <= p)); // the run of piece p
            const uint32_t before = r ? __shfl_sync(0xffffffffu, end, r - 1) : 0u;
            const uint32_t b = __shfl_sync(0xffffffffu, x.x, r) + (p - before) * kPiece;
            const uint32_t e = min(b + kPiece, __shfl_sync(0xffffffffu, x.y, r));
            const uint32_t result = __shfl_sync(0xffffffffu, x.z, r);
#pragma unroll
            for (uint32_t k = 0; k < kPiece; k += 32)
                if (b + k + lane < e)
                    lv.res[__ldcg(vals + b + k + lane)] = result;
        }
    }
}

// A CTA alone: sort of n <= kPT items x (bucket << 32 | entry, one a thread: the
// candidates of a small level, or a queue of a big one's) in registers: a bitonic network with lane
// shuffles, and shared memory for the steps across warps (two buffers, so
// one barrier a step; a rank sort, n reads a thread, took 15.6 us at n = 784).
// The sorted buckets and entries go to sk / sv, the starts of the bucket runs
// to rs (one more: their end); returns the number of runs.
HD_D uint32_t small_sort(const Table& t, uint32_t L, uint32_t n, unsigned long long x, unsigned long long* s64,
                         uint32_t* sm32, uint32_t* sk, uint32_t* sv, uint32_t* rs)
{
    const uint32_t empty = t.g.buckets(L);
    const uint32_t i = threadIdx.x, lane = i & 31;
    auto keep = [&](unsigned long long y, uint32_t k, uint32_t j) {
        const bool up = (i & k) == 0, low = (i & j) == 0;
        x = (low == up) == (x < y) ? x : y;
    };
    const bool mine = (i & ~31u) < n; // the other warps hold no candidate
    if (mine)
        for (uint32_t k = 2; k <= 32; k <<= 1)
            for (uint32_t j = k >> 1; j > 0; j >>= 1)
                keep(__shfl_xor_sync(0xffffffffu, x, j), k, j);
    uint32_t n2 = 32, step = 0;
    while (n2 < n)
        n2 <<= 1;
    for (uint32_t k = 64; k <= n2; k <<= 1) {
        for (uint32_t j = k >> 1; j >= 32; j >>= 1) {
            unsigned long long* buf = s64 + (step++ & 1) * kPT;
            if (i < n2)
                buf[i] = x;
            __syncthreads();
            if (i < n2)
                keep(buf[i ^ j], k, j);
        }
        if (i < n2)
            for (uint32_t j = 16; j > 0; j >>= 1)
                keep(__shfl_xor_sync(0xffffffffu, x, j), k, j);
    }
    const uint32_t key = uint32_t(x >> 32);
    const bool cand = i < n && key < empty;
    if (i < n) {
        sk[i] = key;
        sv[i] = uint32_t(x);
    }
    const uint32_t ncand = __syncthreads_count(cand); // also: sk is written
    const bool start = cand && (i == 0 || sk[i - 1] != key);
    uint32_t runs;
    const uint32_t at = cta_scan(start, &runs, sm32);
    if (start)
        rs[at] = i;
    if (i == 0)
        rs[runs] = ncand;
    __syncthreads();
    return runs;
}

// Per digit of the nb chunks' counts (rows of nd): exclusive scan over the
// chunks in place, the total into rows.  A thread a digit and part of the
// chunks would wait for each other; a warp reads 32 digits of a chunk at once
// and 8 chunks ahead (fewer digits, of a level of few buckets: fewer lanes).
HD_D void scan_rows(uint32_t* hist, uint32_t nb, uint32_t nd, uint32_t* rows)
{
    const uint32_t d = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32 + (threadIdx.x & 31);
    if (d >= nd)
        return;
    uint32_t* p = hist + d;
    uint32_t run = 0;
    for (uint32_t c0 = 0; c0 < nb; c0 += 8) {
        uint32_t x[8];
#pragma unroll
        for (uint32_t k = 0; k < 8; k++)
            x[k] = c0 + k < nb ? __ldcg(p + (c0 + k) * nd) : 0u;
#pragma unroll
        for (uint32_t k = 0; k < 8; k++) {
            if (c0 + k < nb)
                p[(c0 + k) * nd] = run;
            run += x[k];
        }
    }
    rows[d] = run;
}

// Stable scatter of chunk `cb` of (keys, vals) by digit (key >> shift) & (nd
// - 1); warps of a tile take their turn in order.  Keys of `empty` and above
// are left out.  hist: the digit counts of every chunk, a row of nd a chunk.
// With up to kSumRows chunks each CTA sums the rows itself (totals and the
// chunks before its own), which spares the scan's phase (2-4 us a pass); more
// rows are scanned (scan_rows, totals in rows): 152 of them summed by every
// CTA took 20 us.
// With hist_next, counts each element's next digit in the chunk (of chunk_next
// positions) its output position falls in, equal ones of a warp with one
// atomic.  (Entries resolved at once, keyed `empty`, were sorted
// along and met in one counter: 55 us of a level of 184,528 entries, now 24.)
HD_D void scatter_chunk(const uint32_t* keys, const uint32_t* vals, uint32_t n, uint32_t nb, uint32_t cb,
                        uint32_t shift, uint32_t nd, uint32_t empty, const uint32_t* hist, const uint32_t* rows,
                        uint32_t* keys_out,
                        uint32_t* vals_out, uint32_t* hist_next, uint32_t next_shift,
                        uint32_t chunk_next, uint32_t* run, uint32_t* sm32)
{
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t chunk = chunk_len(n, nb, kChunkAlign);
    if (nb > kSumRows) {
        const uint32_t d = threadIdx.x;
        const uint32_t r = d < nd ? __ldcg(rows + d) : 0u;
        uint32_t total;
        const uint32_t ex = cta_scan(r, &total, sm32);
        if (d < nd)
            run[d] = ex + __ldcg(hist + cb * nd + d);
        __syncthreads();
    } else {
        uint32_t* sum = run + kDigits;
        for (uint32_t d = threadIdx.x; d < nd; d += kPT)
            run[d] = sum[d] = 0;
        __syncthreads();
        // kPT / nd threads a digit, each every kPT / nd-th row
        const uint32_t d = threadIdx.x & (nd - 1), parts = kPT / nd;
        uint32_t total = 0, before = 0;
#pragma unroll 8
        for (uint32_t c = threadIdx.x / nd; c < nb; c += parts) {
            const uint32_t x = __ldcg(hist + c * nd + d);
            total += x;
            before += c < cb ? x : 0u;
        }
        atomicAdd(sum + d, total);
        atomicAdd(run + d, before);
        __syncthreads();
        uint32_t all;
        const uint32_t ex = cta_scan(threadIdx.x < nd ? sum[threadIdx.x] : 0u, &all, sm32);
        if (threadIdx.x < nd)
            run[threadIdx.x] += ex;
        __syncthreads();
    }
    const uint32_t i0 = cb * chunk, i1 = min(n, i0 + chunk);
    for (uint32_t base = i0; base < i1; base += kPT) {
        const uint32_t i = base + threadIdx.x;
        const uint32_t key = i < i1 ? __ldcg(keys + i) : empty;
        const uint32_t val = i < i1 ? __ldcg(vals + i) : 0u;
        const bool valid = key < empty;
        const uint32_t digit = valid ? (key >> shift) & (nd - 1) : kDigits + lane;
        const uint32_t peers = __match_any_sync(0xffffffffu, digit);
        const uint32_t leader = __ffs(peers) - 1;
        const uint32_t turns = min(kPWarps, (i1 - base + 31) / 32);
        for (uint32_t w = 0; w < turns; w++) {
            if (warp == w) {
                uint32_t b = 0;
                if (valid && lane == leader) {
                    b = run[digit];
                    run[digit] = b + __popc(peers);
                }
                b = __shfl_sync(0xffffffffu, b, leader);
                const uint32_t pos = b + __popc(peers & lt);
                if (valid) {
                    keys_out[pos] = key;
                    vals_out[pos] = val;
                }
                if (hist_next) {
                    const uint32_t at = valid ? pos / chunk_next * nd + ((key >> next_shift) & (nd - 1))
                                              : 0x80000000u + lane;
                    const uint32_t same = __match_any_sync(0xffffffffu, at);
                    if (valid && lane == uint32_t(__ffs(same) - 1))
                        atomicAdd(hist_next + at, uint32_t(__popc(same)));
                }
            }
            __syncthreads();
        }
    }
}

// CTA 0's state between grid steps
enum : uint32_t { kLsBegin = 0, kLsTopDown = 1, kLsBottomUp = 2, kLsFinish = 3 };
// the grid step CTA 0 asks for
enum : uint32_t { kPhNone = 0, kPhTopDown = 1, kPhBottomUp = 2 };

// Bytes of the dynamic shared memory the find-or-add buffers and the small
// sort share (a multiple of 16); the small level's sorted keys and entries
// follow.
HD_HD constexpr size_t persist_smem_core()
{
    return (size_t(kPWarps) * kPage * 4 + size_t(kPWarps) * kFoaQuery * 4 + size_t(kPWarps) * sizeof(FoaCache) >
                    size_t(kPT) * 8 * 2
                ? size_t(kPWarps) * kPage * 4 + size_t(kPWarps) * kFoaQuery * 4 + size_t(kPWarps) * sizeof(FoaCache)
                : size_t(kPT) * 8 * 2) +
           15 & ~size_t(15);
}

struct Smem {
    uint32_t* sk; // a small level's sorted keys and entries (kPT each) and
    uint32_t* sv; // run starts (kPT + 1), past the buffers below (which the
    uint32_t* rs; // find-or-add overwrites)
    uint32_t* page;
    uint32_t* q;
    FoaCache* cache;
    unsigned long long* s64;
    uint32_t* list;
    uint32_t* sm32;
    Editor* ed;
    TinyState* tiny;
};

// CTA 0: the next edit of the batch (or the stop); level 0 classified.
// False when the batch stops.
HD_D bool begin_edit(const Table& t, const PArgs& a, const Smem& sm)
{
    Ctl* ctl = a.ctl;
    const uint32_t G = gridDim.x;
    if (threadIdx.x == 0) {
        const uint32_t idx = ctl->idx;
        uint32_t stop = ctl->stop;
        if (stop == kRun && __ldcg(t.error) != 0)
            stop = kTableError;
        if (stop == kRun && idx >= a.n_edits)
            stop = kDone;
        ctl->stop = stop;
        if (stop == kRun) {
            *sm.ed = a.edits ? make_editor(a.edits[idx]) : a.one;
            ctl->ed = *sm.ed;
            for (uint32_t L = 0; L < HD_MAX_DEPTH; L++)
                ctl->count[L] = ctl->ncand[L] = ctl->nruns[L] = ctl->nstarts[L] = 0;
            ctl->count[0] = 1;
            TinyState& ts = *sm.tiny;
            ts.held = 1;
            ts.failed = 0;
            ts.count[0] = 1;
            ts.lv[0].x[0] = ts.lv[0].y[0] = ts.lv[0].z[0] = 0;
            ts.lv[0].old[0] = __ldcg(a.d_root);
            a.out[idx].ctr = EditCounters{};
            a.out[idx].t_begin = now_ns();
        }
        sm.sm32[32] = stop;
    }
    for (uint32_t k = threadIdx.x; k < 3 * G; k += kPT)
        a.bsum[k] = 0;
    for (uint32_t k = threadIdx.x; k < (t.g.leaf_level + 1) * G; k += kPT)
        a.queued[k] = 0;
    __syncthreads();
    if (sm.sm32[32] != kRun)
        return false;
    if (threadIdx.x == 0) {
        unsigned long long nn, vv;
        classify_entry<true>(t, *sm.ed, 0, held_level(a, *sm.tiny, 0), 0, nn, vv);
        EditCounters* ctr = &a.out[ctl->idx].ctr;
        atomicAdd(&ctr->num_nodes, nn);
        atomicAdd(&ctr->num_voxels, vv);
    }
    __syncthreads();
    return true;
}

// CTA 0, after level 0's find-or-add: the new root, or the stop.
HD_D void finish_edit(const Table& t, const PArgs& a, const Smem& sm)
{
    Ctl* ctl = a.ctl;
    if (a.hold_root) {
        // the colour phase reads the level arrays: a warp a held level
        const TinyState& ts = *sm.tiny;
        const uint32_t L = threadIdx.x >> 5, k = threadIdx.x & 31;
        if (L < HD_MAX_DEPTH && ((ts.held >> L) & 1u) && k < ts.count[L]) {
            const TinyLevel& m = ts.lv[L];
            const Level l = a.lv[L];
            l.x[k] = m.x[k], l.y[k] = m.y[k], l.z[k] = m.z[k], l.old[k] = m.old[k];
            l.res[k] = m.res[k], l.cnt[k] = m.cnt[k], l.flag[k] = m.flag[k], l.exp[k] = m.exp[k];
            l.state[k] = m.state[k];
        }
    }
    if (threadIdx.x == 0) {
        const uint32_t idx = ctl->idx;
        if (__ldcg(t.error) != 0) {
            ctl->stop = kTableError;
        } else {
            const uint32_t r = sm.tiny->lv[0].res[0];
            if (r == kInvalid || r == kNotFound) {
                ctl->stop = kEmptyScene;
            } else {
                if (!a.hold_root)
                    *a.d_root = r;
                a.out[idx].root = r;
                __threadfence();
                a.out[idx].t_end = now_ns();
                ctl->idx = idx + 1;
            }
        }
    }
    __syncthreads();
}

// CTA 0: advances the batch alone from state ls at level L (small levels,
// the end of an edit, the start of the next) until the grid is needed
// (ctl->phase / ctl->level) or the batch stops (ctl->stop).
template <int PW>
HD_D void local_advance(const Table& t, const PArgs& a, uint32_t ls, uint32_t L, const Smem& sm, const uint32_t& nbar)
{
    Ctl* ctl = a.ctl;
    const uint32_t G = gridDim.x, leafl = t.g.leaf_level;
    const uint32_t warp = threadIdx.x >> 5;
    TinyState& ts = *sm.tiny;
    __shared__ bool meet;
    const unsigned long long t_in = now_ns();
    for (;;) {
        if (ls == kLsFinish) {
            // the edit ends; the next one begins at once when every other CTA
            // already waits at the coming barrier (it reads no more of this
            // edit's state) and has not waited a good part of its bound
            finish_edit(t, a, sm);
            if (threadIdx.x == 0) {
                const unsigned long long set_ns = __ldcg(&ctl->wait_ns);
                ctl->phase = kPhNone;
                meet = barrier_arrivals(ld_acquire64(&ctl->arrived)) + 1 < barrier_target(nbar + 1, G) ||
                       now_ns() - t_in > (set_ns ? set_ns : kWaitNs) / 16;
            }
            __syncthreads();
            const bool m = meet;
            __syncthreads();
            if (m)
                return;
            ls = kLsBegin;
        }
        if (ls == kLsBegin) {
            if (!begin_edit(t, a, sm))
                return;
            L = 0;
            ls = kLsTopDown;
        }
        EditCounters* ctr = &a.out[ctl->idx].ctr;
        if (ls == kLsTopDown) {
            while (L < leafl) {
                if ((ts.held >> L) & 1u) {
                    // the held levels: warp 0 alone
                    if (warp == 0) {
                        uint32_t st;
                        const uint32_t L2 = td_tiny(t, *sm.ed, a, ts, L, ctr, st);
                        if ((threadIdx.x & 31) == 0) {
                            ts.level = L2;
                            ts.status = st;
                        }
                    }
                    __syncthreads();
                    L = ts.level;
                    if (ts.status == 2) {
                        if (threadIdx.x == 0)
                            ctl->stop = kCapacity;
                        __syncthreads();
                        return;
                    }
                    if (ts.status == 1 || L >= leafl)
                        break;
                }
                const uint32_t n = ts.count[L];
                if (n > kSmall) {
                    if (threadIdx.x == 0) {
                        ctl->phase = kPhTopDown;
                        ctl->level = L;
                    }
                    __syncthreads();
                    return;
                }
                const Level lv = held_level(a, ts, L), nx = a.lv[L + 1];
                uint32_t f = 0;
                for (uint32_t i = threadIdx.x; i < n; i += kPT)
                    f += lv.flag[i];
                uint32_t total;
                cta_scan(f, &total, sm.sm32);
                if (total == 0)
                    break;
                const uint64_t n_next = 8ull * total;
                if (n_next > a.cap[L + 1]) {
                    if (threadIdx.x == 0)
                        ctl->stop = kCapacity;
                    __syncthreads();
                    return;
                }
                uint32_t* zero = a.bsum + ((L + 2) % 3) * G;
                for (uint32_t k = threadIdx.x; k < G; k += kPT)
                    zero[k] = 0;
                __syncthreads();
                td_range(t, *sm.ed, lv, nx, L, 0, n, 0, uint32_t(n_next), G, a.bsum + ((L + 1) % 3) * G, ctr, sm.sm32,
                         sm.list);
                if (threadIdx.x == 0)
                    ctl->count[L + 1] = ts.count[L + 1] = uint32_t(n_next);
                __syncthreads();
                L++;
            }
            if (threadIdx.x == 0)
                ctl->deepest = L;
            __syncthreads();
            ls = kLsBottomUp;
        }
        if (ls == kLsBottomUp) {
            const uint32_t deepest = ctl->deepest;
            if (threadIdx.x == 0 && __ldcg(t.error) != 0)
                ts.failed = 1; // (after a grid step)
            __syncthreads();
            for (;;) {
                // after a failed append the levels above are not rebuilt
                const bool failed = ts.failed;
                __syncthreads(); // (warp 0 writes the state below)
                if (failed)
                    break;
                if (ts.count[L] <= kTiny) {
                    // one warp passes through the levels of at most one
                    // bucket run; more runs are the CTA's
                    if (warp == 0) {
                        uint32_t l = L, runs;
                        for (;;) {
                            runs = tiny_candidates(t, a, ts, l, deepest, ts.count[l]);
                            if (runs > 1)
                                break;
                            if (runs) {
                                Level lv = held_level(a, ts, l);
                                lv.cand = ts.rows;
                                foa_runs<PW>(t, l, lv, ts.sk, ts.sv, ts.rs, runs, 0, 1, sm.page, sm.q, sm.cache[0], ctr,
                                             &ts.failed);
                                __syncwarp();
                            }
                            if (ts.failed || l == 0 || ts.count[l - 1] > kTiny)
                                break;
                            l--;
                        }
                        if ((threadIdx.x & 31) == 0) {
                            ts.level = l;
                            ts.runs = runs;
                        }
                    }
                    __syncthreads();
                    L = ts.level;
                    if (const uint32_t runs = ts.runs; runs > 1) {
                        Level lv = held_level(a, ts, L);
                        lv.cand = ts.rows;
                        foa_runs<PW>(t, L, lv, ts.sk, ts.sv, ts.rs, runs, warp, kPWarps, sm.page + warp * kPage,
                                     sm.q + warp * kFoaQuery, sm.cache[warp], ctr, &ts.failed);
                        __syncthreads();
                    }
                    if (L == 0)
                        break;
                    L--;
                    continue;
                }
                const uint32_t n = ts.count[L];
                if (n > kSmallUp) {
                    if (threadIdx.x == 0) {
                        ctl->phase = kPhBottomUp;
                        ctl->level = L;
                    }
                    __syncthreads();
                    return;
                }
                candidates_range(t, a.lv, L, deepest, 0, n, a.keys, a.vals);
                __syncthreads();
                const unsigned long long x = threadIdx.x < n ? (uint64_t(a.keys[threadIdx.x]) << 32) | a.vals[threadIdx.x]
                                                             : ~0ull;
                const uint32_t runs = small_sort(t, L, n, x, sm.s64, sm.sm32, sm.sk, sm.sv, sm.rs);
                foa_runs<PW>(t, L, a.lv[L], sm.sk, sm.sv, sm.rs, runs, warp, kPWarps, sm.page + warp * kPage,
                             sm.q + warp * kFoaQuery, sm.cache[warp], ctr, &ts.failed);
                // the CTA barrier makes this level's results (lv.res, appended
                // nodes) visible to CTA 0's next level; the grid barrier
                // (a CTA barrier, then a fence by its thread 0) to the grid
                __syncthreads();
                if (L == 0)
                    break;
                L--;
            }
            ls = kLsFinish;
        }
    }
}

template <int PW>
__global__ void __launch_bounds__(kPT, 1)
    k_edit_persistent(__grid_constant__ const Table t, __grid_constant__ const PArgs a)
{
    {
        const uint32_t skip = __ldcg(&a.ctl->skip_cta);
        if (skip && blockIdx.x == skip - 1)
            return; // a test of the timeout path: this CTA never arrives
    }
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint32_t sm32[40];
    __shared__ Editor ed_s;
    __shared__ uint32_t cnt[kDigits];
    // the foa buffers (pages, queries, caches); the same bytes serve the
    // small sort, the top-down tile list and the scatter's digit runs
    Smem sm;
    sm.page = reinterpret_cast<uint32_t*>(smem_raw);
    sm.q = sm.page + kPWarps * kPage;
    sm.cache = reinterpret_cast<FoaCache*>(sm.q + kPWarps * kFoaQuery);
    sm.s64 = reinterpret_cast<unsigned long long*>(smem_raw);
    sm.sk = reinterpret_cast<uint32_t*>(smem_raw + persist_smem_core());
    sm.sv = sm.sk + kPT;
    sm.rs = sm.sv + kPT;
    sm.list = sm.page;
    sm.sm32 = sm32;
    sm.ed = &ed_s;
    sm.tiny = reinterpret_cast<TinyState*>(sm.rs + kPT + 4);
    uint32_t* run = sm.page;
    Ctl* ctl = a.ctl;
    const uint32_t G = gridDim.x, cta = blockIdx.x;
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t leafl = t.g.leaf_level;
    uint32_t ls = kLsBegin, L = 0;
    __shared__ uint32_t nbar; // barriers this CTA has passed (thread 0)
    if (threadIdx.x == 0)
        nbar = 0;
    __syncthreads();
    for (;;) {
        if (cta == 0) {
            local_advance<PW>(t, a, ls, L, sm, nbar);
            if (threadIdx.x == 0) // the command of the coming barrier
                ctl->cmd[(nbar + 1) & 1] = Cmd{ctl->stop, ctl->phase, ctl->level, ctl->deepest, ctl->idx, {0, 0, 0}};
        }
        if (!grid_sync(ctl, t.error, nbar))
            return;
        // the grid step CTA 0 asked for, decided the same way by every CTA
        __shared__ Cmd cmd;
        if (threadIdx.x == 0) {
            const uint32_t* src = reinterpret_cast<const uint32_t*>(&ctl->cmd[nbar & 1]);
            uint32_t* dst = reinterpret_cast<uint32_t*>(&cmd);
            for (uint32_t k = 0; k < sizeof(Cmd) / 4; k++)
                dst[k] = __ldcg(src + k);
        }
        __syncthreads();
        if (cmd.stop != kRun)
            return;
        uint32_t phase = cmd.phase;
        if (phase == kPhNone) {
            ls = kLsBegin; // an edit ended: CTA 0 starts the next
            continue;
        }
        L = cmd.level;
        uint32_t deepest = cmd.deepest;
        EditCounters* ctr = &a.out[cmd.idx].ctr;
        if (threadIdx.x == 0) {
            const uint32_t* src = reinterpret_cast<const uint32_t*>(&ctl->ed);
            uint32_t* dst = reinterpret_cast<uint32_t*>(&ed_s);
            for (uint32_t k = 0; k < sizeof(Editor) / 4; k++)
                dst[k] = __ldcg(src + k);
        }
        __syncthreads();
        if (phase == kPhTopDown) {
            // one phase per level down to the deepest
            for (;;) {
                const uint32_t n = __ldcg(&ctl->count[L]);
                const uint32_t* cnt_cur = a.bsum + (L % 3) * G;
                uint32_t all = 0;
                for (uint32_t b = threadIdx.x; b < G; b += kPT)
                    all += __ldcg(cnt_cur + b);
                uint32_t ta;
                cta_scan(all, &ta, sm32);
                if (ta == 0)
                    break; // nothing descends: L is the deepest level
                const uint64_t n_next = 8ull * ta;
                if (n_next > a.cap[L + 1]) {
                    if (cta == 0 && threadIdx.x == 0)
                        ctl->stop = kCapacity;
                    return; // every CTA decides this alike
                }
                if (threadIdx.x == 0)
                    a.bsum[((L + 2) % 3) * G + cta] = 0;
                const uint32_t cch = chunk_len(uint32_t(n_next), G, kChunkAlign);
                const uint32_t k0 = min(uint32_t(n_next), cta * cch), k1 = min(uint32_t(n_next), k0 + cch);
                td_children(t, ed_s, a.lv, L, n, k0, k1, uint32_t(n_next), G, cnt_cur, a.bsum + ((L + 1) % 3) * G,
                            ctr, sm32, sm.list, sm.list + kListRanks);
                if (cta == 0 && threadIdx.x == 0)
                    ctl->count[L + 1] = sm.tiny->count[L + 1] = uint32_t(n_next);
                if (!grid_sync(ctl, t.error, nbar))
                    return;
                L++;
                if (L == leafl)
                    break;
            }
            deepest = L;
            if (cta == 0 && threadIdx.x == 0)
                ctl->deepest = L;
            phase = kPhBottomUp;
        }
        // bottom-up, big levels; small ones go back to CTA 0
        while (__ldcg(&ctl->count[L]) > kSmallUp && __ldcg(t.error) == 0) {
            const uint32_t n = __ldcg(&ctl->count[L]);
            const uint32_t nb = sort_chunks(n, G);
            const uint32_t chunk = chunk_len(n, nb, kChunkAlign);
            uint32_t key_bits = 1;
            while ((1u << key_bits) <= t.g.buckets(L))
                key_bits++;
            const uint32_t dbits = (key_bits + 1) / 2, nd = 1u << dbits;
            const uint32_t empty = t.g.buckets(L);
            const bool digits = n > kPT; // a queue may overflow
            // 1. candidates, to their owners, and their pass-1 digit counts
            if (cta < nb) {
                if (digits) {
                    for (uint32_t d = threadIdx.x; d < nd; d += kPT) {
                        cnt[d] = 0;
                        a.hist2[cta * nd + d] = 0;
                    }
                    __syncthreads();
                }
                const uint32_t i0 = cta * chunk, i1 = min(n, i0 + chunk);
                candidates_range(t, a.lv, L, deepest, i0, i1, a.keys, a.vals);
                uint32_t mine = 0;
                for (uint32_t i = i0 + threadIdx.x; i < i1; i += kPT) {
                    const uint32_t key = a.keys[i];
                    if (key < empty) {
                        if (digits)
                            atomicAdd(&cnt[key & (nd - 1)], 1u);
                        mine++;
                        const uint32_t owner = key % G, at = atomicAdd(a.queued + L * G + owner, 1u);
                        if (at < kPT)
                            __stcg(a.queue + owner * kPT + at, uint64_t(key) << 32 | i);
                    }
                }
                if (digits) {
                    mine = __reduce_add_sync(0xffffffffu, mine);
                    if ((threadIdx.x & 31) == 0 && mine)
                        atomicAdd(&ctl->ncand[L], mine);
                    __syncthreads();
                    for (uint32_t d = threadIdx.x; d < nd; d += kPT)
                        a.hist[cta * nd + d] = cnt[d];
                }
            }
            if (!grid_sync(ctl, t.error, nbar))
                return;
            // 2. the CTA's own candidates, unless a queue overflowed.  Each grid
            // step costs 2.4-3.5 us whatever it does: with every level sorted
            // by the grid (four steps and more) a level of 4,816 entries took
            // 33 us, now about 20, and one of 1,216 28 and 18: batches of 64
            // edits, as above, 6.22 -> 5.80 and 15.0 -> 13.6 ms.
            {
                const uint32_t* queued = a.queued + L * G;
                bool over = false;
                for (uint32_t k = threadIdx.x; k < G; k += kPT)
                    over |= __ldcg(queued + k) > kPT;
                if (!__syncthreads_or(over)) {
                    const uint32_t own = __ldcg(queued + cta);
                    const unsigned long long x = threadIdx.x < own ? __ldcg(a.queue + cta * kPT + threadIdx.x) : ~0ull;
                    const uint32_t runs = small_sort(t, L, own, x, sm.s64, sm32, sm.sk, sm.sv, sm.rs);
                    foa_runs<PW>(t, L, a.lv[L], sm.sk, sm.sv, sm.rs, runs, warp, kPWarps, sm.page + warp * kPage,
                                 sm.q + warp * kFoaQuery, sm.cache[warp], ctr);
                    if (!grid_sync(ctl, t.error, nbar))
                        return;
                    L--; // (level 0 holds one entry: never big)
                    continue;
                }
            }
            // the second pass and the find-or-add: candidates only
            const uint32_t ncand = __ldcg(&ctl->ncand[L]);
            const uint32_t nb2 = sort_chunks(ncand, G);
            const uint32_t chunk2 = max(kChunkAlign, chunk_len(ncand, nb2, kChunkAlign));
            // 2. pass 1, pass-2 counts
            if (nb > kSumRows) {
                scan_rows(a.hist, nb, nd, a.rows);
                if (!grid_sync(ctl, t.error, nbar))
                    return;
            }
            if (cta < nb)
                scatter_chunk(a.keys, a.vals, n, nb, cta, 0, nd, empty, a.hist, a.rows, a.keys2, a.vals2, a.hist2,
                              dbits, chunk2, run, sm32);
            if (!grid_sync(ctl, t.error, nbar))
                return;
            // 3. pass 2
            if (nb2 > kSumRows) {
                scan_rows(a.hist2, nb2, nd, a.rows2);
                if (!grid_sync(ctl, t.error, nbar))
                    return;
            }
            if (cta < nb2)
                scatter_chunk(a.keys2, a.vals2, ncand, nb2, cta, dbits, nd, empty, a.hist2, a.rows2, a.keys, a.vals,
                              nullptr, 0, 0, run, sm32);
            if (!grid_sync(ctl, t.error, nbar))
                return;
            // 4. find-or-add, one warp per bucket run
            uint32_t *page = sm.page + warp * kPage, *q = sm.q + warp * kFoaQuery;
            if (ncand >= kRepeatLevel) {
                const uint32_t part = chunk_len(ncand, G, 32);
                const uint32_t p0 = min(ncand, cta * part), p1 = min(ncand, p0 + part);
                mark_repeats(a.lv[L], L == leafl, a.keys, a.vals, ncand, p0, p1, a.same, a.keys2, &ctl->nstarts[L]);
                if (!grid_sync(ctl, t.error, nbar))
                    return;
                const Repeats rep{a.same, (ncand + 31) / 32, a.runs, &ctl->nruns[L]};
                foa_listed<PW>(t, L, a.lv[L], a.keys, a.vals, ncand, a.keys2, __ldcg(&ctl->nstarts[L]), warp * G + cta,
                               G * kPWarps, page, q, sm.cache[warp], ctr, rep);
            } else {
                foa_sorted<PW>(t, L, a.lv[L], a.keys, a.vals, ncand, warp * G + cta, G * kPWarps, page, q,
                               sm.cache[warp], ctr);
            }
            if (!grid_sync(ctl, t.error, nbar))
                return;
            if (const uint32_t nr = __ldcg(&ctl->nruns[L])) {
                fill_runs(a.lv[L], a.vals, a.runs, nr);
                if (!grid_sync(ctl, t.error, nbar))
                    return;
            }
            if (L == 0)
                break; // (level 0 holds one entry: never big)
            L--;
        }
        ls = kLsBottomUp; // CTA 0 continues at L (or finishes the edit on an error)
    }
}

} // namespace

// ---- host side --------------------------------------------------------------------

static size_t persist_smem() { return persist_smem_core() + size_t(kPT) * 4 * 3 + 16 + sizeof(TinyState); }

template <int PW>
static const void* persist_kernel()
{
    return reinterpret_cast<const void*>(k_edit_persistent<PW>);
}

namespace {

// The launch shape of a context, found once: one CTA per SM.
struct PersistShape {
    const void* kern;
    uint32_t grid; // 0: the kernel does not fit on an SM
};

PersistShape persist_shape(hd_ctx* c)
{
    const uint32_t pw = c->tuning.probe_words == 4 ? 2 : c->tuning.probe_words == 2 ? 1 : 0;
    const void* kern = pw == 2 ? persist_kernel<4>() : pw == 1 ? persist_kernel<2>() : persist_kernel<1>();
    if (!c->persist_known[pw]) {
        int dev = 0, sms = 0, per_sm = 0;
        HD_CUDA(cudaGetDevice(&dev));
        HD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        HD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(persist_smem())));
        HD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kPT, persist_smem()));
        c->persist_grid[pw] = per_sm < 1 ? 0u : uint32_t(sms);
        c->persist_known[pw] = true;
    }
    return {kern, c->persist_grid[pw]};
}

// Device buffers of a launch of at most n edits; ctl and out lie in one
// buffer, so that one copy brings the results back.
PArgs persist_args(hd_ctx* c, const PersistLevels& pl, uint32_t grid, uint32_t n)
{
    Scratch& s = c->scratch;
    PArgs a{};
    a.ctl = reinterpret_cast<Ctl*>(s.get<unsigned char>("ep_ctl", sizeof(Ctl) + sizeof(EditOut) * n));
    a.out = reinterpret_cast<EditOut*>(a.ctl + 1);
    for (uint32_t L = 0; L <= c->g.leaf_level; L++) {
        a.lv[L] = pl.lv[L];
        a.cap[L] = pl.caps[L];
    }
    a.keys = pl.keys;
    a.vals = pl.vals;
    a.keys2 = pl.keys2;
    a.vals2 = pl.vals2;
    a.bsum = s.get<uint32_t>("ep_bsum", 3ull * grid);
    a.queue = s.get<unsigned long long>("ep_queue", uint64_t(kPT) * grid);
    a.queued = s.get<uint32_t>("ep_queued", uint64_t(HD_MAX_DEPTH) * grid);
    a.hist = s.get<uint32_t>("ep_hist", uint64_t(kDigits) * grid);
    a.hist2 = s.get<uint32_t>("ep_hist2", uint64_t(kDigits) * grid);
    a.rows = s.get<uint32_t>("ep_rows", kDigits);
    a.rows2 = s.get<uint32_t>("ep_rows2", kDigits);
    uint64_t most = 1;
    for (uint32_t L = 0; L <= c->g.leaf_level; L++)
        most = std::max<uint64_t>(most, pl.caps[L]);
    a.same = s.get<uint32_t>("ep_same", most / 32 + 1);
    a.runs = s.get<FollowerRun>("ep_runs", most / kLongRun + 1);
    a.d_root = c->d_root;
    return a;
}
static_assert(sizeof(Ctl) % alignof(EditOut) == 0, "EditOut follows Ctl");

// The control block at its start; hd_set_test_barrier_skip's hook, for one
// launch only (it switches itself off).  Returns the CTAs to ask for.
uint32_t persist_begin(hd_ctx* c, const PersistShape& shape, const PArgs& a)
{
    cudaStream_t st = c->stream;
    HD_CUDA(cudaMemsetAsync(a.ctl, 0, sizeof(Ctl), st));
    const uint32_t skip = c->test_skip_cta;
    if (!skip)
        return shape.grid;
    const unsigned long long wait = c->test_wait_ns;
    c->test_skip_cta = 0;
    c->test_wait_ns = 0;
    if (skip > shape.grid)
        return 64 * shape.grid; // more than any SM holds: the launch is refused
    HD_CUDA(cudaMemcpyAsync(&a.ctl->skip_cta, &skip, 4, cudaMemcpyHostToDevice, st));
    HD_CUDA(cudaMemcpyAsync(&a.ctl->wait_ns, &wait, 8, cudaMemcpyHostToDevice, st));
    HD_CUDA(cudaStreamSynchronize(st));
    return shape.grid;
}

// False when the device has no room for all CTAs at once (fewer SMs to use
// than it says): nothing was launched.
bool persist_launch(hd_ctx* c, const PersistShape& shape, uint32_t grid, PArgs& a)
{
    void* args[] = {&c->t, &a};
    const cudaError_t e =
        cudaLaunchCooperativeKernel(shape.kern, dim3(grid), dim3(kPT), args, persist_smem(), c->stream);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
        cudaGetLastError();
        return false;
    }
    HD_CUDA(e);
    return true;
}

[[noreturn]] void persist_timeout(hd_ctx* c, const Ctl& fin, uint32_t edit)
{
    check_error(c);
    c->root = read_scalar(c->d_root, c->stream);
    std::string where;
    for (uint32_t k = 0; k < 8; k++)
        where += (k ? " " : "") + std::to_string(fin.diag[k]);
    throw StatusError{HD_ERR_TIMEOUT, "edit " + std::to_string(edit) +
                                          ": a grid barrier of the persistent edit kernel ran out of time "
                                          "(cta, barriers, arrivals, arrivals awaited, cta0 barriers, phase, level, edit: " +
                                          where + ")"};
}

} // namespace

// Applies edits[0..n) in one persistent launch per stretch of the batch (a
// level that would outgrow its bound ends the stretch: that edit takes the
// one-edit path and the next stretch starts after it).
void edit_batch_persistent(hd_ctx* c, const hd_edit* edits, uint32_t n, const PersistLevels& pl, hd_edit* d_edits,
                           std::vector<EditCounters>& ctr, std::vector<float>& dur_ms, std::vector<float>& end_ms,
                           float& device_ms, uint64_t& fallbacks)
{
    cudaStream_t st = c->stream;
    const PersistShape shape = persist_shape(c);
    if (!shape.grid)
        throw StatusError{HD_ERR_STATE, "the persistent edit kernel does not fit on an SM"};
    PArgs a = persist_args(c, pl, shape.grid, n);
    std::vector<unsigned char> back(sizeof(Ctl) + sizeof(EditOut) * n);
    uint32_t done = 0;
    c->batch_applied = 0;
    float elapsed_before = 0.0f;
    while (done < n) {
        const uint32_t m = n - done;
        a.edits = d_edits;
        a.n_edits = m;
        HD_CUDA(cudaMemcpyAsync(d_edits, edits + done, sizeof(hd_edit) * m, cudaMemcpyHostToDevice, st));
        const uint32_t grid = persist_begin(c, shape, a);
        HD_CUDA(cudaEventRecord(c->ev0, st));
        if (!persist_launch(c, shape, grid, a))
            throw CudaError{cudaErrorCooperativeLaunchTooLarge, "the persistent edit kernel's launch"};
        HD_CUDA(cudaEventRecord(c->ev1, st));
        HD_CUDA(cudaMemcpyAsync(back.data(), a.ctl, sizeof(Ctl) + sizeof(EditOut) * m, cudaMemcpyDeviceToHost, st));
        HD_CUDA(cudaStreamSynchronize(st));
        Ctl fin;
        std::memcpy(&fin, back.data(), sizeof(Ctl));
        const EditOut* out = reinterpret_cast<const EditOut*>(back.data() + sizeof(Ctl));
        float launch_ms = 0;
        HD_CUDA(cudaEventElapsedTime(&launch_ms, c->ev0, c->ev1));
        const uint32_t ok = fin.idx;
        for (uint32_t k = 0; k < ok; k++) {
            UndoFrame f;
            f.root = c->root;
            push_undo(c, std::move(f));
            c->root = out[k].root;
            ctr[done + k] = out[k].ctr;
            dur_ms[done + k] = float(double(out[k].t_end - out[k].t_begin) * 1e-6);
            end_ms[done + k] = elapsed_before + float(double(out[k].t_end - out[0].t_begin) * 1e-6);
        }
        elapsed_before += launch_ms;
        done += ok;
        c->batch_applied = done;
        if (barrier_aborted(fin.arrived))
            persist_timeout(c, fin, done);
        if (fin.stop == kDone)
            break;
        if (fin.stop == kTableError || fin.stop == kEmptyScene) {
            const uint32_t err = check_error(c);
            c->root = read_scalar(c->d_root, st);
            if (fin.stop == kEmptyScene)
                throw StatusError{HD_ERR_STATE, "edit " + std::to_string(done) + " would empty the whole scene"};
            throw StatusError{hd_status(err ? err : HD_ERR_CUDA),
                              "edit " + std::to_string(done) + " failed on the device (" + c->err_detail + ")"};
        }
        // capacity: this edit with the level-by-level path, then resume
        c->root = read_scalar(c->d_root, st);
        hd_edit_stats es{};
        edit_by_levels(c, edits[done], &es);
        ctr[done].num_voxels = es.num_voxels;
        ctr[done].num_nodes = es.num_nodes;
        ctr[done].foa = es.find_or_add_calls;
        ctr[done].added = es.nodes_added;
        ctr[done].scanned = es.words_scanned;
        dur_ms[done] = es.device_ms;
        elapsed_before += es.device_ms;
        end_ms[done] = elapsed_before;
        done++;
        c->batch_applied = done;
        fallbacks++;
    }
    device_ms = elapsed_before;
}

bool edit_geometry_persistent(hd_ctx* c, const Editor& ed, const PersistLevels& pl, bool hold_root, EditGeometry& out)
{
    cudaStream_t st = c->stream;
    const PersistShape shape = persist_shape(c);
    if (!shape.grid)
        return false;
    PArgs a = persist_args(c, pl, shape.grid, 1);
    a.n_edits = 1;
    a.hold_root = hold_root;
    a.one = ed;
    if (!persist_launch(c, shape, persist_begin(c, shape, a), a))
        return false;
    if (!hold_root)
        HD_CUDA(cudaEventRecord(c->ev1, st)); // with colours the edit goes on
    struct {
        Ctl ctl;
        EditOut edit;
    } back;
    HD_CUDA(cudaMemcpyAsync(&back, a.ctl, sizeof(back), cudaMemcpyDeviceToHost, st));
    HD_CUDA(cudaStreamSynchronize(st));
    const Ctl& fin = back.ctl;
    if (barrier_aborted(fin.arrived)) {
        check_error(c);
        // CTA 0 may have finished the edit, if its levels were small, and
        // waited for the others only then; else what it appended stays, whole
        // nodes within their buckets' sizes
        if (fin.idx != 1)
            return false;
    }
    if (fin.stop == kCapacity)
        return false;
    if (fin.stop == kEmptyScene)
        throw StatusError{HD_ERR_STATE, "edit would empty the whole scene"};
    if (fin.idx != 1) {
        const uint32_t err = check_error(c);
        throw StatusError{hd_status(err ? err : HD_ERR_CUDA), "edit failed on the device (" + c->err_detail + ")"};
    }
    out.ctr = back.edit.ctr;
    out.root = back.edit.root;
    out.deepest = fin.deepest;
    out.count.assign(fin.count, fin.count + c->g.leaf_level + 1);
    return true;
}

} // namespace hd
