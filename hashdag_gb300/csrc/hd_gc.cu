// Garbage collection on the device: mark-and-compact of the hash table.
//
// Reference: HashDAG::remove_stale_nodes (hash_dag.h:407-547).  Mark: the
// nodes reachable from the root level by level (here as a bitmap over each
// level's virtual range, so the live list comes out sorted by address).
// Rebuild bottom-up: every live node's content is gathered with its children
// remapped, the level's buckets are emptied, the full node is added first
// (add_full_node) and the live nodes are re-appended without a find, in
// increasing old-address order (the reference uses its hash-set order), so a
// reachable full node is kept twice as in the reference.  Pages stay mapped;
// the words past a bucket's new size keep their old contents.  With
// HD_GC_RELEASE_PAGES (no reference counterpart: its poolTop only grows,
// hash_table.h:794-809), the pages wholly past each bucket's new size are
// unmapped, zeroed and put on the table's free list, from which the next
// page claims draw first.
#include <algorithm>
#include <vector>

#include "hd_ctx.h"
#include "hd_table.cuh"

namespace hd {

// Bound by the atomics on the words of widely shared children: every parent
// of a level's full node sets the same bit.  The bit is looked at first (a
// cached read; one from L2 when that copy does not show it, as a stale line
// may not), so that an atomic runs only for a bit not yet seen set: the 12
// mark launches of a 2^14 scene go from 6,959 to 369 us.
__global__ void k_gc_mark(Table t, const uint32_t* __restrict__ live, uint32_t n, uint32_t child_base,
                          uint32_t* bitmap)
{
    HD_GRID_STRIDE(i, n)
    {
        const uint32_t* p = t.sys(live[i]);
        const uint32_t cnt = popc32(p[0] & 0xffu);
        for (uint32_t k = 0; k < cnt; k++) {
            const uint32_t off = p[1 + k] - child_base, bit = 1u << (off & 31);
            uint32_t* w = bitmap + (off >> 5);
            if (!(__ldca(w) & bit) && !(__ldcg(w) & bit))
                atomicOr(w, bit);
        }
    }
}

// A level's live list from its mark bitmap, in two passes over it (16 MB for a
// level of 2^16 buckets of 2,048 words, mostly empty): the bits of each tile of
// kScanTile words, then, with the tiles' sums, the list and the ranks: every
// word that has a bit with the live count before it, for ChildMap.  With the
// counts scanned into an array of their own and added up in place, five passes:
// 470 us a GC of a 2^14 scene, so 183.
__global__ void __launch_bounds__(kScanThreads) k_gc_tile_bits(const uint32_t* __restrict__ bitmap, uint64_t n,
                                                               uint32_t* __restrict__ sums)
{
    const uint64_t base = uint64_t(blockIdx.x) * kScanTile;
    uint32_t bits = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        const uint64_t k = base + uint64_t(i) * kScanThreads + threadIdx.x;
        bits += k < n ? popc32(bitmap[k]) : 0u;
    }
    uint32_t total;
    block_excl_scan(bits, &total);
    if (threadIdx.x == 0)
        sums[blockIdx.x] = total;
}
__global__ void __launch_bounds__(kScanThreads)
    k_gc_list(const uint32_t* __restrict__ bitmap, const uint32_t* __restrict__ before, uint64_t n, uint32_t base,
              uint32_t* __restrict__ list, uint2* __restrict__ ranks)
{
    const uint64_t at = uint64_t(blockIdx.x) * kScanTile + uint64_t(threadIdx.x) * kScanItems;
    uint32_t w[kScanItems], bits = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        w[i] = at + i < n ? bitmap[at + i] : 0u;
        bits += popc32(w[i]);
    }
    uint32_t total;
    uint32_t o = before[blockIdx.x] + block_excl_scan(bits, &total);
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        uint32_t b = w[i];
        if (!b)
            continue;
        ranks[at + i] = make_uint2(b, o);
        while (b) {
            const uint32_t bit = __ffs(b) - 1;
            b &= b - 1;
            list[o++] = base + uint32_t(at + i) * 32 + bit;
        }
    }
}

HD_D uint32_t lower_bound(const uint32_t* v, uint32_t n, uint32_t x)
{
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (v[mid] < x)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// A live node with its children remapped.  A child's index in the live list
// of the level below is its rank in that level's mark bitmap: the live count
// before its bitmap word plus the bits below it in the word.  The two lie side
// by side (ranks): apart, they cost a sector more per child, and the keys of
// the two biggest inner levels of a 2^14 scene 258 and 163 us instead of 199
// and 133.
struct ChildMap {
    const uint2* ranks;
    const uint32_t* new_addr;
    uint32_t base;
};
HD_D uint32_t remapped_node(const Table& t, uint32_t v, bool leaf, const ChildMap& m, uint32_t* c)
{
    const uint32_t* p = t.sys(v);
    c[0] = p[0];
    if (leaf) {
        c[1] = p[1];
        return 2;
    }
    const uint32_t cnt = popc32(c[0] & 0xffu);
#pragma unroll
    for (uint32_t k = 0; k < 8; k++)
        if (k < cnt) {
            const uint32_t off = p[1 + k] - m.base;
            const uint2 w = m.ranks[off >> 5];
            c[1 + k] = m.new_addr[w.y + popc32(w.x & ((1u << (off & 31)) - 1u))];
        }
    return cnt + 1;
}

// ---- dry run: every level's new addresses, before anything changes ----------
// The rebuild of a level re-appends its live nodes with a different order
// and so a different padding: a bucket can need a page it never had.  A
// rebuild that runs out of pages half way cannot be undone, so the GC first
// runs every level's rebuild on scratch bucket sizes (the full node first,
// then the live nodes in increasing old address) and counts the pages it
// would map, and the pages a releasing GC would free.  The addresses stay:
// the rebuild itself then writes every node to its address, node by node in
// parallel, with no order to keep.
// A releasing GC frees a level's pages that lie wholly past their bucket's
// final size before it rebuilds the level, so the same level's buckets can
// take them: re-hashed parents (children remapped) move between buckets, and
// one bucket's growth is met by another's shrinkage.

// The level's full node at the head of its (empty) bucket, on dry sizes.
__global__ void k_gc_dry_full(Table t, uint32_t level, uint32_t* dry_sizes, uint32_t* full_dry)
{
    uint32_t node[9];
    uint32_t n, hash;
    const bool leaf = level == t.g.leaf_level;
    if (leaf) {
        node[0] = node[1] = 0xFFFFFFFFu;
        n = 2;
        hash = hash_leaf(~0ull);
    } else {
        const uint32_t depth = t.g.depth - level;
        const uint32_t voxels = level < t.g.T ? 0u : (1u << (3 * depth));
        node[0] = (voxels << 8) | 0xffu;
        for (int c = 0; c < 8; c++)
            node[1 + c] = full_dry[level + 1];
        n = 9;
        hash = hash_interior(9, node);
    }
    const uint32_t bucket = hash & (t.g.buckets(level) - 1);
    dry_sizes[bucket] = n;
    full_dry[level] = t.g.make_ptr(level, bucket, 0);
}

// Bucket and size of every live node (bucket | words << 24; buckets stay
// below 2^24) and its arrival rank in the bucket, in any order.  staged (or
// null): the nodes, for k_gc_write.
__global__ void k_gc_keys(Table t, uint32_t level, const uint32_t* __restrict__ live, uint32_t n, ChildMap m,
                          uint32_t* __restrict__ keys, uint32_t* __restrict__ rank, uint32_t* __restrict__ counts,
                          uint32_t* __restrict__ staged)
{
    const bool leaf = level == t.g.leaf_level;
    HD_GRID_STRIDE(i, n)
    {
        uint32_t c[9];
        const uint32_t words = remapped_node(t, live[i], leaf, m, c);
        const uint32_t hash = leaf ? hash_leaf(uint64_t(c[0]) | (uint64_t(c[1]) << 32)) : hash_interior(words, c);
        const uint32_t bucket = hash & (t.g.buckets(level) - 1);
        if (staged) {
#pragma unroll
            for (uint32_t k = 0; k < 9; k++)
                if (k < words)
                    staged[9 * i + k] = c[k];
        }
        keys[i] = bucket | (words << 24);
        rank[i] = atomicAdd(counts + bucket, 1u);
    }
}

__global__ void k_gc_group(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ rank,
                           const uint32_t* __restrict__ first, uint32_t n, uint32_t* __restrict__ items)
{
    HD_GRID_STRIDE(i, n) items[first[keys[i] & 0xFFFFFFu] + rank[i]] = uint32_t(i);
}

// A warp per bucket: its items in increasing order, appended one after the
// other to the dry size (append_position), 32 at a time: the sizes' prefix
// sums place every node up to the first that would straddle a page, which
// starts the next page.  Then the bucket's pages: those the rebuild maps
// (unmapped, below the final size) and, releasing, frees (mapped, wholly
// past it).
// Bound by latency (a sort of a few dozen items, dependent shuffles).  When
// the buckets were linked lists that one lane walked and then appended from,
// the 13 dry and 13 real appends of a 2^14 scene took 892 and 2,313 us; the
// groups and these assignments take 372 + 60 us, k_gc_write and k_gc_map 241.
constexpr uint32_t kGcWarps = 2;
__global__ void __launch_bounds__(32 * kGcWarps)
    k_gc_assign(Table t, uint32_t level, const uint32_t* __restrict__ keys, const uint32_t* __restrict__ counts,
                const uint32_t* __restrict__ first, const uint32_t* __restrict__ list, uint32_t* __restrict__ dry_sizes,
                uint32_t* __restrict__ out_addr, uint32_t* __restrict__ overflow, uint32_t release,
                unsigned long long* need, unsigned long long* freed)
{
    __shared__ uint32_t items_s[kGcWarps][kMaxBucketItems];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t* items = items_s[warp];
    const bool leaf = level == t.g.leaf_level;
    const uint32_t nb = t.g.buckets(level), cap = t.g.capacity(level);
    unsigned long long a = 0, f = 0;
    for (uint32_t bucket = blockIdx.x * kGcWarps + warp; bucket < nb; bucket += gridDim.x * kGcWarps) {
        uint32_t cnt = counts[bucket], size = dry_sizes[bucket];
        if (cnt > kMaxBucketItems) {
            if (lane == 0)
                set_error(t.error, kErrBucketFull, 0xFFFFFFFFu, t.g.bucket_global(level, bucket), cnt);
            cnt = 0;
        }
        if (cnt) {
            const uint32_t* src = list + first[bucket];
            if (cnt <= 32) {
                // in registers: a bitonic network over the lanes
                uint32_t x = lane < cnt ? src[lane] : kEmpty;
                for (uint32_t k = 2; k <= 32; k <<= 1)
                    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                        const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
                        x = ((lane & k) == 0) == ((lane & j) == 0) ? min(x, y) : max(x, y);
                    }
                items[lane] = x;
            } else {
                uint32_t n2 = 64;
                while (n2 < cnt)
                    n2 <<= 1;
                for (uint32_t i = lane; i < n2; i += 32)
                    items[i] = i < cnt ? src[i] : kEmpty;
                __syncwarp();
                sort_shared(items, n2);
            }
            __syncwarp();
            for (uint32_t i0 = 0; i0 < cnt; i0 += 32) {
                const uint32_t i = i0 + lane;
                const uint32_t r = i < cnt ? items[i] : 0u;
                const uint32_t n = i < cnt ? (leaf ? 2u : keys[r] >> 24) : 0u;
                const uint32_t inc = warp_incl_scan(n);
                uint32_t done = 0, pos = 0; // words of the items placed so far, this lane's position
                bool placed = n == 0;
                for (;;) {
                    // room in the page the size ends in (512 at a page start);
                    // leaves pack pages exactly (even sizes), so they are
                    // placed like nodes that never straddle
                    const uint32_t room = kPage - (size & (kPage - 1));
                    const bool fits = !placed && (leaf || inc - done <= room);
                    const uint32_t fb = __ballot_sync(0xffffffffu, fits);
                    if (fb) {
                        if (fits) {
                            pos = size + (inc - done) - n;
                            placed = true;
                        }
                        const uint32_t all = __shfl_sync(0xffffffffu, inc, 31 - __clz(fb));
                        size += all - done;
                        done = all;
                    }
                    if (!__any_sync(0xffffffffu, !placed))
                        break;
                    size = (size + kPage - 1) & ~(kPage - 1); // the next node starts a page
                }
                if (i < cnt)
                    out_addr[r] = t.g.make_ptr(level, bucket, pos);
            }
            if (lane == 0) {
                if (size > cap)
                    atomicExch(overflow, 1u);
                dry_sizes[bucket] = size;
            }
        }
        for (uint32_t off = lane * kPage; off < cap; off += 32 * kPage) {
            const bool mapped = t.page_table[t.g.make_ptr(level, bucket, off) >> kPageShift] != 0;
            if (off < size)
                a += !mapped;
            else if (release)
                f += mapped;
        }
        __syncwarp();
    }
    for (int o = 16; o; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        f += __shfl_down_sync(0xffffffffu, f, o);
    }
    if (lane == 0 && a)
        atomicAdd(need, a);
    if (lane == 0 && f)
        atomicAdd(freed, f);
}

// ---- rebuild of a level ---------------------------------------------------------
// The live nodes, children remapped, staged before the level's pages are
// written.
__global__ void k_gc_gather(Table t, uint32_t level, const uint32_t* __restrict__ live, uint32_t n, ChildMap m,
                            uint32_t* __restrict__ content)
{
    const bool leaf = level == t.g.leaf_level;
    HD_GRID_STRIDE(i, n)
    {
        uint32_t c[9];
        const uint32_t words = remapped_node(t, live[i], leaf, m, c);
#pragma unroll
        for (uint32_t k = 0; k < 9; k++)
            if (k < words)
                content[9 * i + k] = c[k];
    }
}

// The buckets' final sizes, with every page below them mapped (after the
// full node's).
__global__ void k_gc_map(Table t, uint32_t level, const uint32_t* __restrict__ dry_sizes, uint32_t n)
{
    HD_GRID_STRIDE(b, uint64_t(t.g.buckets(level)))
    {
        const uint32_t size = dry_sizes[b];
        if (map_pages(t, level, uint32_t(b), 0, size))
            t.bucket_sizes[t.g.bucket_global(level, uint32_t(b))] = size;
        if (b == 0)
            t.level_nodes[level] += n;
    }
}

// Every staged node to its address, and into its page's filter.
__global__ void k_gc_write(Table t, uint32_t level, const uint32_t* __restrict__ content,
                           const uint32_t* __restrict__ addr, uint32_t n)
{
    const bool leaf = level == t.g.leaf_level;
    HD_GRID_STRIDE(i, n)
    {
        uint32_t c[9];
        c[0] = content[9 * i];
        const uint32_t words = leaf ? 2 : total_size(c[0]);
#pragma unroll
        for (uint32_t k = 1; k < 9; k++)
            if (k < words)
                c[k] = content[9 * i + k];
        const uint32_t v = addr[i];
        uint32_t* dst = t.sys_rw(v);
#pragma unroll
        for (uint32_t k = 0; k < 9; k++)
            if (k < words)
                dst[k] = c[k];
        bloom_add(t, v, bloom_bits(c, words), leaf);
    }
}

// Pages wholly past a bucket's final size (`sizes`, the level's buckets)
// go to the free list (one thread per bucket, at most capacity / 512 pages
// each).
__global__ void k_gc_release(Table t, uint32_t level, const uint32_t* __restrict__ sizes)
{
    const Geom& g = t.g;
    uint32_t* free_count = t.pool_top + 1;
    HD_GRID_STRIDE(i, g.buckets(level))
    {
        const uint32_t bucket = uint32_t(i);
        const uint32_t size = sizes[bucket], cap = g.capacity(level);
        for (uint32_t off = (size + kPage - 1) & ~(kPage - 1); off < cap; off += kPage) {
            const uint32_t vp = g.make_ptr(level, bucket, off) >> kPageShift;
            const uint32_t p = t.page_ids[vp];
            if (p) {
                const uint32_t k = atomicAdd(free_count, 1u);
                t.free_pages[k] = p;
                if (t.direct) {
                    t.free_phys[k] = vp + 1;
                    t.page_ids[vp] = 0;
                }
                t.page_table[vp] = 0;
            }
        }
    }
}

// Zeroes the pages [from, to) of the free list and their Bloom filters.
__global__ void k_zero_pages(Table t, uint32_t from, uint32_t to)
{
    const uint64_t n = uint64_t(to - from) * kPage;
    HD_GRID_STRIDE(i, n)
    {
        const uint32_t p = t.free_phys[from + uint32_t(i / kPage)];
        t.pool[uint64_t(p) * kPage + (i % kPage)] = 0;
        if (i % kPage < kPageMeta)
            t.meta[uint64_t(p) * kPageMeta + (i % kPage)] = 0;
    }
}

__global__ void k_gc_remap_roots(const uint32_t* __restrict__ live, uint32_t n, const uint32_t* __restrict__ newaddr,
                                 uint32_t* roots, uint32_t n_roots, uint32_t* d_root)
{
    for (uint32_t i = 0; i < n_roots; i++)
        roots[i] = newaddr[lower_bound(live, n, roots[i])];
    *d_root = roots[0];
}

namespace {
constexpr uint64_t kGcStageBytes = 1ull << 30;
// The rebuild may claim the pages other claims leave as the GC's reserve
// (hd_set_page_reserve); the limit comes back however the GC ends.
struct ReserveOpen {
    hd_ctx* c;
    explicit ReserveOpen(hd_ctx* ctx) : c(ctx) { set_claim_limit(c, true); }
    ~ReserveOpen()
    {
        try {
            set_claim_limit(c, false);
        } catch (...) {
        }
    }
};
} // namespace

// stage: the inner levels' nodes may be staged.  HD_ERR_OOM comes before
// anything changes.
static void gc_run(hd_ctx* c, std::vector<uint32_t>& roots, bool release_pages, bool stage)
{
    cudaStream_t st = c->stream;
    Scratch& s = c->scratch;
    const Geom& g = c->g;
    const uint32_t leafl = g.leaf_level;
    ReserveOpen reserve_open(c);
    uint32_t* d_n = s.get<uint32_t>("gc_n", 4);
    // level 0: the roots, sorted unique
    std::vector<uint32_t> r0(roots.begin(), roots.end());
    std::sort(r0.begin(), r0.end());
    r0.erase(std::unique(r0.begin(), r0.end()), r0.end());
    std::vector<uint32_t*> live(leafl + 1), newaddr(leafl + 1);
    std::vector<uint32_t> nlive(leafl + 1);
    live[0] = s.get<uint32_t>("gc_live_0", r0.size());
    HD_CUDA(cudaMemcpyAsync(live[0], r0.data(), r0.size() * 4, cudaMemcpyHostToDevice, st));
    nlive[0] = uint32_t(r0.size());
    // mark; every level's ranks stay for the remapping
    std::vector<uint2*> ranks(leafl + 1, nullptr);
    uint64_t most_words = 1;
    for (uint32_t L = 1; L <= leafl; L++)
        most_words = std::max<uint64_t>(most_words, (uint64_t(g.buckets(L)) * g.capacity(L) + 31) / 32);
    uint32_t* bitmap = s.get<uint32_t>("gc_bitmap", most_words);
    const uint64_t most_tiles = (most_words + kScanTile - 1) / kScanTile;
    uint32_t* tile_bits = s.get<uint32_t>("gc_tile_bits", most_tiles);
    uint32_t* tile_before = s.get<uint32_t>("gc_tile_before", most_tiles);
    std::vector<uint32_t> bbase(leafl + 1, 0);
    for (uint32_t L = 0; L < leafl; L++) {
        const uint32_t base = g.make_ptr(L + 1, 0, 0);
        const uint64_t range = uint64_t(g.buckets(L + 1)) * g.capacity(L + 1);
        const uint64_t nwords = (range + 31) / 32;
        HD_CUDA(cudaMemsetAsync(bitmap, 0, nwords * 4, st));
        k_gc_mark<<<grid_for(nlive[L], 256), 256, 0, st>>>(c->t, live[L], nlive[L], base, bitmap);
        HD_LAUNCH_CHECK();
        char nm[32];
        snprintf(nm, sizeof(nm), "gc_ranks_%u", L + 1);
        ranks[L + 1] = s.get<uint2>(nm, nwords);
        bbase[L + 1] = base;
        const uint32_t tiles = uint32_t((nwords + kScanTile - 1) / kScanTile);
        k_gc_tile_bits<<<tiles, kScanThreads, 0, st>>>(bitmap, nwords, tile_bits);
        HD_LAUNCH_CHECK();
        exclusive_scan<uint32_t, uint32_t>(s, tile_bits, tile_before, tiles, d_n, st);
        nlive[L + 1] = read_scalar(d_n, st);
        snprintf(nm, sizeof(nm), "gc_live_%u", L + 1);
        live[L + 1] = s.get<uint32_t>(nm, uint64_t(nlive[L + 1]) + 1);
        k_gc_list<<<tiles, kScanThreads, 0, st>>>(bitmap, tile_before, nwords, base, live[L + 1], ranks[L + 1]);
        HD_LAUNCH_CHECK();
    }
    uint32_t maxn = 1, max_buckets = 1;
    for (uint32_t L = 0; L <= leafl; L++) {
        maxn = std::max(maxn, nlive[L]);
        max_buckets = std::max(max_buckets, g.buckets(L));
    }
    auto children = [&](int32_t L) {
        return L < int32_t(leafl) ? ChildMap{ranks[L + 1], newaddr[L + 1], bbase[L + 1]} : ChildMap{};
    };
    // The inner levels' nodes are staged as the dry run remaps them (three
    // dependent reads a child), where that takes kGcStageBytes at most; else, and
    // for the leaves, which have no children, the rebuild gathers a level
    // itself.  With 16 edits before it, the GC of a 2^14 scene took 5.69 ms
    // gathering every level again, 5.19 so (its marks counted by the scan too).
    std::vector<uint32_t*> staged(leafl + 1, nullptr);
    uint64_t inner = 0;
    for (uint32_t L = 0; L < leafl; L++)
        inner += nlive[L];
    if (stage && 36 * inner <= kGcStageBytes) {
        uint32_t* at = s.get<uint32_t>("gc_staged", 9 * inner + 1);
        for (uint32_t L = 0; L < leafl; L++) {
            staged[L] = at;
            at += 9ull * nlive[L];
        }
    }
    uint32_t* dry_all = s.get<uint32_t>("gc_dry_sizes", g.total_buckets);
    // dry run, bottom-up: every node's new address, and the pages every
    // level's rebuild needs against the free pages (and those the levels
    // below free when releasing)
    {
        uint32_t top[2];
        HD_CUDA(cudaMemcpyAsync(top, c->t.pool_top, 8, cudaMemcpyDeviceToHost, st));
        uint32_t* full_dry = s.get<uint32_t>("gc_full_dry", HD_MAX_DEPTH);
        uint32_t* keys = s.get<uint32_t>("gc_keys", maxn);
        uint32_t* rank = s.get<uint32_t>("gc_rank", maxn);
        uint32_t* items = s.get<uint32_t>("gc_items", maxn);
        uint32_t* counts = s.get<uint32_t>("gc_bucket_counts", max_buckets);
        uint32_t* first = s.get<uint32_t>("gc_bucket_first", max_buckets);
        unsigned long long* cnt = s.get<unsigned long long>("gc_dry_cnt", 2 * HD_MAX_DEPTH);
        uint32_t* overflow = s.get<uint32_t>("gc_dry_overflow", HD_MAX_DEPTH);
        HD_CUDA(cudaMemsetAsync(overflow, 0, HD_MAX_DEPTH * 4, st));
        HD_CUDA(cudaMemsetAsync(cnt, 0, 2 * HD_MAX_DEPTH * 8, st));
        HD_CUDA(cudaMemsetAsync(dry_all, 0, g.total_buckets * 4, st));
        for (int32_t L = int32_t(leafl); L >= 0; L--) {
            const uint32_t n = nlive[L], nb = g.buckets(uint32_t(L));
            char nm[32];
            snprintf(nm, sizeof(nm), "gc_new_%d", L);
            newaddr[L] = s.get<uint32_t>(nm, uint64_t(n) + 1);
            uint32_t* dry_sizes = dry_all + g.level_first_bucket(uint32_t(L));
            HD_CUDA(cudaMemsetAsync(counts, 0, uint64_t(nb) * 4, st));
            k_gc_dry_full<<<1, 1, 0, st>>>(c->t, uint32_t(L), dry_sizes, full_dry);
            HD_LAUNCH_CHECK();
            k_gc_keys<<<grid_for(n, 256), 256, 0, st>>>(c->t, uint32_t(L), live[L], n, children(L), keys, rank, counts,
                                                        staged[L]);
            HD_LAUNCH_CHECK();
            exclusive_scan<uint32_t, uint32_t>(s, counts, first, nb, nullptr, st);
            k_gc_group<<<grid_for(n, 256), 256, 0, st>>>(keys, rank, first, n, items);
            HD_LAUNCH_CHECK();
            k_gc_assign<<<grid_for(uint64_t(nb) * 32, 32 * kGcWarps, 152 * 12), 32 * kGcWarps, 0, st>>>(
                c->t, uint32_t(L), keys, counts, first, items, dry_sizes, newaddr[L], overflow + L,
                release_pages ? 1u : 0u, cnt + 2 * L, cnt + 2 * L + 1);
            HD_LAUNCH_CHECK();
        }
        unsigned long long h[2 * HD_MAX_DEPTH];
        uint32_t ovf[HD_MAX_DEPTH];
        HD_CUDA(cudaMemcpyAsync(h, cnt, sizeof(h), cudaMemcpyDeviceToHost, st));
        HD_CUDA(cudaMemcpyAsync(ovf, overflow, sizeof(ovf), cudaMemcpyDeviceToHost, st));
        HD_CUDA(cudaStreamSynchronize(st));
        const uint32_t e = check_error(c); // a bucket of more than kMaxBucketItems
        int64_t avail = int64_t(g.pool_pages) - top[0] + top[1];
        for (int32_t L = int32_t(leafl); L >= 0; L--) {
            if (ovf[L])
                throw StatusError{HD_ERR_BUCKET_FULL, "GC: a rebuilt bucket of level " + std::to_string(L) +
                                                          " would exceed its capacity; the table is unchanged"};
            // releasing: the level's pages past the final sizes are freed
            // before its appends claim
            avail += int64_t(h[2 * L + 1]);
            if (int64_t(h[2 * L]) > avail)
                throw StatusError{HD_ERR_POOL_FULL, "GC: rebuilding level " + std::to_string(L) + " needs " +
                                                        std::to_string(h[2 * L]) + " new pages, " +
                                                        std::to_string(std::max<int64_t>(avail, 0)) +
                                                        " are free; the table is unchanged"};
            avail -= int64_t(h[2 * L]);
        }
        if (e)
            throw StatusError{hd_status(e), "GC: " + c->err_detail + "; the table is unchanged"};
    }
    // rebuild bottom-up
    uint32_t* gathered = s.get<uint32_t>("gc_content", uint64_t(staged[0] ? nlive[leafl] : maxn) * 9);
    uint32_t* d_roots = s.get<uint32_t>("gc_roots", roots.size());
    for (int32_t L = int32_t(leafl); L >= 0; L--) {
        const uint32_t n = nlive[L];
        const uint32_t* dry_sizes = dry_all + g.level_first_bucket(uint32_t(L));
        const uint32_t* content = staged[L];
        if (!content) {
            content = gathered;
            k_gc_gather<<<grid_for(n, 256), 256, 0, st>>>(c->t, uint32_t(L), live[L], n, children(L), gathered);
            HD_LAUNCH_CHECK();
        }
        // empty the level's buckets and their pages' filters, then the
        // full node first
        HD_CUDA(cudaMemsetAsync(c->t.bucket_sizes + g.level_first_bucket(uint32_t(L)), 0,
                                uint64_t(g.buckets(uint32_t(L))) * 4, st));
        bloom_clear_level(c, uint32_t(L));
        HD_CUDA(cudaMemsetAsync(c->t.level_nodes + L, 0, 8, st));
        if (release_pages) {
            // the level's pages past its final bucket sizes (the dry run's),
            // zeroed, serve this level's appends and the levels above
            uint32_t before[2], after[2];
            HD_CUDA(cudaMemcpyAsync(before, c->t.pool_top, 8, cudaMemcpyDeviceToHost, st));
            k_gc_release<<<grid_for(g.buckets(uint32_t(L)), 256), 256, 0, st>>>(c->t, uint32_t(L), dry_sizes);
            HD_LAUNCH_CHECK();
            HD_CUDA(cudaMemcpyAsync(after, c->t.pool_top, 8, cudaMemcpyDeviceToHost, st));
            HD_CUDA(cudaStreamSynchronize(st));
            if (after[1] > before[1]) {
                k_zero_pages<<<grid_for(uint64_t(after[1] - before[1]) * kPage, 256), 256, 0, st>>>(c->t, before[1],
                                                                                                   after[1]);
                HD_LAUNCH_CHECK();
            }
        }
        add_full_nodes(c, uint32_t(L), uint32_t(L));
        k_gc_map<<<grid_for(g.buckets(uint32_t(L)), 256), 256, 0, st>>>(c->t, uint32_t(L), dry_sizes, n);
        HD_LAUNCH_CHECK();
        k_gc_write<<<grid_for(n, 256), 256, 0, st>>>(c->t, uint32_t(L), content, newaddr[L], n);
        HD_LAUNCH_CHECK();
    }
    HD_CUDA(cudaMemcpyAsync(d_roots, roots.data(), roots.size() * 4, cudaMemcpyHostToDevice, st));
    k_gc_remap_roots<<<1, 1, 0, st>>>(live[0], nlive[0], newaddr[0], d_roots, uint32_t(roots.size()), c->d_root);
    HD_LAUNCH_CHECK();
    HD_CUDA(cudaMemcpyAsync(roots.data(), d_roots, roots.size() * 4, cudaMemcpyDeviceToHost, st));
    HD_CUDA(cudaStreamSynchronize(st));
    const uint32_t e = check_error(c);
    if (e)
        throw StatusError{hd_status(e), "garbage collection failed on the device"};
    c->root = roots[0];
    c->edit_head_ready = false;
}

void gc(hd_ctx* c, std::vector<uint32_t>& roots, bool release_pages)
{
    try {
        return gc_run(c, roots, release_pages, true);
    } catch (const StatusError& e) {
        if (e.status != HD_ERR_OOM)
            throw;
    }
    // without what GCs and edits keep for speed
    HD_CUDA(cudaStreamSynchronize(c->stream));
    c->scratch.drop("gc_staged");
    drop_batch_levels(c);
    gc_run(c, roots, release_pages, false);
}

} // namespace hd

extern "C" hd_status hd_gc_ex(hd_ctx* c, uint32_t* extra, uint32_t n, uint32_t flags)
{
    if (!c || (n && !extra) || (flags & ~uint32_t(HD_GC_KEEP_HISTORY | HD_GC_RELEASE_PAGES)))
        return HD_ERR_INVALID;
    try {
        std::vector<uint32_t> roots(1 + n);
        roots[0] = hd::read_scalar(c->d_root, c->stream);
        for (uint32_t i = 0; i < n; i++)
            roots[1 + i] = extra[i];
        if (flags & HD_GC_KEEP_HISTORY) {
            // the roots of the undo / redo frames stay alive and are remapped
            for (auto& f : c->undo)
                roots.push_back(f.root);
            for (auto& f : c->redo)
                roots.push_back(f.root);
        } else {
            // the engine frees its undo history with the GC (engine.cpp:178-185)
            c->undo.clear();
            c->redo.clear();
        }
        hd::gc(c, roots, (flags & HD_GC_RELEASE_PAGES) != 0);
        c->needs_gc = false; // the buckets are rebuilt
        // the remapped extra roots go back to the caller
        for (uint32_t i = 0; i < n; i++)
            extra[i] = roots[1 + i];
        size_t k = 1 + n;
        if (flags & HD_GC_KEEP_HISTORY) {
            for (auto& f : c->undo)
                f.root = roots[k++];
            for (auto& f : c->redo)
                f.root = roots[k++];
        }
        return HD_OK;
    } catch (const hd::StatusError& e) {
        c->err = e.msg;
        return e.status;
    } catch (const hd::CudaError& e) {
        c->err = std::string("CUDA error ") + cudaGetErrorString(e.code) + " in " + e.where;
        return HD_ERR_CUDA;
    }
}

extern "C" hd_status hd_gc(hd_ctx* c, uint32_t* extra, uint32_t n) { return hd_gc_ex(c, extra, n, 0); }
