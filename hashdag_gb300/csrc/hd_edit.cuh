// Edit pipeline, per-entry device logic shared by the one-edit-per-call path
// (hd_edit.cu) and the graph-captured batched path (hd_edit_batch.cu).
//
// Reference: HashDAG::edit_threads (hash_dag.h:255-405), which runs
// HashDagEdits::edit_threaded over the levels above C_colorTreeLevels
// (hash_dag_edits.h:106-333) and edit_leaf below (:335-643); editors
// (hash_dag_editors.h:57-127, :223-313); find_or_add_leaf_node /
// find_or_add_interior_node with their bucket scans (hash_table.h:196-357,
// :470-560).
//
// The recursion becomes two level-synchronous sweeps:
//  * top-down, every level's edit entries (a node path and its old index) are
//    classified as in the reference (untouched, carved away, filled, a leaf
//    to rebuild, or an interior node to descend into); descended entries
//    spawn their 8 children, in child order, so each level's entries stay in
//    depth-first (Morton) order;
//  * bottom-up, every rebuilt node is compared with its old self and, when
//    changed, hashed and resolved by find-or-add.  Candidates of a level are
//    grouped by bucket and each bucket is resolved by one warp, candidates in
//    depth-first order one after the other: the same sequence of bucket scans
//    and appends as the reference's single-threaded depth-first recursion,
//    including its scan rules (a node flush with the bucket tail or the page
//    end is invisible to an equal-size query).
#pragma once

#include "hd_ctx.h"
#include "hd_table.cuh"

namespace hd {

constexpr uint32_t kNoBucket = 0xFFFFFFFFu;


// ---- editors ----------------------------------------------------------------
// SphereEditor / BoxEditor (hash_dag_editors.h:223-313), SpherePaintEditor
// (:315-330) and the copy tool (CopyEditorWithDecompression, :437-609).
struct Editor {
    uint32_t tool;
    float cx, cy, cz, r, r2;
    float bminx, bminy, bminz, bmaxx, bmaxy, bmaxz;
    float paint_r, paint_g, paint_b; // paint target colour
    // copy: source / dest, the source region's corner (copyMin) and size,
    // its occupancy and colours read before the edit (x fastest)
    float srcx, srcy, srcz, dstx, dsty, dstz, minx, miny, minz;
    uint32_t size;
    const uint8_t* values;
    const uint64_t* colors;
    // noise and fill (BufferEditor, :129-221): the buffer's corner
    // (BoxEditorBase::min; minx.. above), its radius (1.5 r for the noise)
    // and per voxel kBufNew (the voxel reads true) | kBufSet (set by the
    // tool); the fill's colour of each set voxel in `colors`
    float buf_r;
    HD_HD bool sphere() const
    {
        return tool == HD_TOOL_SPHERE_ADD || tool == HD_TOOL_SPHERE_REMOVE || tool == HD_TOOL_SPHERE_PAINT;
    }
    HD_HD bool adding() const { return tool == HD_TOOL_SPHERE_ADD || tool == HD_TOOL_BOX_ADD; }
    // is_full / is_empty exist for the sphere and box editors only
    HD_HD bool shortcuts() const { return tool <= HD_TOOL_BOX_ADD; }
};

HD_HD Editor make_editor(const hd_edit& e)
{
    Editor ed{};
    ed.tool = e.tool;
    ed.cx = e.center[0];
    ed.cy = e.center[1];
    ed.cz = e.center[2];
    ed.r = e.radius;
    ed.r2 = e.radius * e.radius;
    float bx = e.center[0], by = e.center[1], bz = e.center[2];
    if (e.tool == HD_TOOL_COPY) {
        // BoxEditorBase(center - source + dest, radius)
        ed.srcx = e.source[0];
        ed.srcy = e.source[1];
        ed.srcz = e.source[2];
        ed.dstx = e.dest[0];
        ed.dsty = e.dest[1];
        ed.dstz = e.dest[2];
        bx = e.center[0] - e.source[0] + e.dest[0];
        by = e.center[1] - e.source[1] + e.dest[1];
        bz = e.center[2] - e.source[2] + e.dest[2];
        ed.minx = e.center[0] - e.radius;
        ed.miny = e.center[1] - e.radius;
        ed.minz = e.center[2] - e.radius;
        ed.size = 2 * uint32_t(ceilf(e.radius));
    }
    float br = e.radius;
    if (e.tool == HD_TOOL_NOISE_ADD || e.tool == HD_TOOL_NOISE_REMOVE)
        br = 1.5f * e.radius; // BufferEditor(dag, center, 1.5f * radius) (:716)
    if (e.tool >= HD_TOOL_NOISE_REMOVE) {
        ed.buf_r = br;
        ed.minx = bx - br;
        ed.miny = by - br;
        ed.minz = bz - br;
        ed.size = 2 * uint32_t(ceilf(br));
    }
    ed.bminx = bx - br;
    ed.bminy = by - br;
    ed.bminz = bz - br;
    ed.bmaxx = bx + br;
    ed.bmaxy = by + br;
    ed.bmaxz = bz + br;
    ed.paint_r = float(e.rgb & 0xFF) / 255.0f;
    ed.paint_g = float((e.rgb >> 8) & 0xFF) / 255.0f;
    ed.paint_b = float((e.rgb >> 16) & 0xFF) / 255.0f;
    return ed;
}

// the copy tool's source index of a destination voxel, or -1 (:585-606)
HD_HD int64_t copy_index(const Editor& e, float px, float py, float pz)
{
    const float qx = ((px - e.dstx) + e.srcx) - e.minx, qy = ((py - e.dsty) + e.srcy) - e.miny,
                qz = ((pz - e.dstz) + e.srcz) - e.minz;
    const uint32_t ix = uint32_t(qx < 0 ? 0.0f : qx), iy = uint32_t(qy < 0 ? 0.0f : qy),
                   iz = uint32_t(qz < 0 ? 0.0f : qz);
    if (ix >= e.size || iy >= e.size || iz >= e.size)
        return -1;
    return int64_t(ix) + int64_t(e.size) * iy + int64_t(e.size) * e.size * iz;
}
// Per-voxel flags of the noise and fill buffers
constexpr uint8_t kBufNew = 1; // BufferEditor::get_value reads true (set, or loaded true)
constexpr uint8_t kBufSet = 2; // EValues::SetTrue

// truncate(float3) (cuda_math.h:80) of a float that may be negative, as the
// reference's x86-64 build converts it: to a 64-bit integer toward zero, then
// its low 32 bits ((-1, 0) gives 0, anything below -1 a huge index)
HD_HD uint32_t trunc_u32(float f) { return uint32_t((long long)f); }

// the buffer index of a voxel, or -1 (BufferEditor::get_new_value, :211-220)
HD_HD int64_t buffer_index(const Editor& e, float px, float py, float pz)
{
    const uint32_t x = trunc_u32(px - e.minx), y = trunc_u32(py - e.miny), z = trunc_u32(pz - e.minz);
    if (x >= e.size || y >= e.size || z >= e.size)
        return -1;
    return int64_t(x) + int64_t(e.size) * y + int64_t(e.size) * e.size * z;
}

// get_new_value of each editor
HD_HD bool new_value(const Editor& e, float px, float py, float pz, bool prev)
{
    if (e.tool >= HD_TOOL_NOISE_REMOVE) {
        // `get_value(p) == EValues::Unknown` compares a bool with 0: a
        // voxel reads true when set or loaded true, else keeps its value
        const int64_t i = buffer_index(e, px, py, pz);
        return (i >= 0 && (e.values[i] & kBufNew)) ? true : prev;
    }
    if (e.tool == HD_TOOL_SPHERE_PAINT)
        return prev;
    if (e.tool == HD_TOOL_COPY) {
        if (prev)
            return prev;
        const int64_t i = copy_index(e, px, py, pz);
        return i < 0 ? prev : e.values[i] != 0;
    }
    return e.adding();
}

HD_D float sqr(float f) { return f * f; }
HD_D float fmax_r(float a, float b) { return a > b ? a : b; }

// SphereEditorBase::should_edit_impl (:112-126) / BoxEditorBase (:76-91)
HD_D bool should_edit_impl(const Editor& e, float mnx, float mny, float mnz, float mxx, float mxy, float mxz)
{
    if (e.sphere()) {
        float dist = e.r2;
        if (e.cx < mnx)
            dist -= sqr(e.cx - mnx);
        else if (e.cx > mxx)
            dist -= sqr(e.cx - mxx);
        if (e.cy < mny)
            dist -= sqr(e.cy - mny);
        else if (e.cy > mxy)
            dist -= sqr(e.cy - mxy);
        if (e.cz < mnz)
            dist -= sqr(e.cz - mnz);
        else if (e.cz > mxz)
            dist -= sqr(e.cz - mxz);
        return dist > 0;
    }
    return !(e.bminx >= mxx || e.bminy >= mxy || e.bminz >= mxz || e.bmaxx <= mnx || e.bmaxy <= mny ||
             e.bmaxz <= mnz || mnx >= e.bmaxx || mny >= e.bmaxy || mnz >= e.bmaxz || mxx <= e.bminx ||
             mxy <= e.bminy || mxz <= e.bminz);
}

// is_full_impl / is_empty_impl (:280-295, :233-252): the region lies inside
// the tool.
HD_D bool inside_tool(const Editor& e, float mnx, float mny, float mnz, float mxx, float mxy, float mxz)
{
    if (e.sphere()) {
        const float a = fmax_r(sqr(mnx - e.cx), sqr(mxx - e.cx));
        const float b = fmax_r(sqr(mny - e.cy), sqr(mxy - e.cy));
        const float c = fmax_r(sqr(mnz - e.cz), sqr(mxz - e.cz));
        return (a + b) + c < e.r2;
    }
    return e.bminx <= mnx && e.bminy <= mny && e.bminz <= mnz && e.bmaxx >= mxx && e.bmaxy >= mxy && e.bmaxz >= mxz;
}

// A candidate's row: its words (zeros past the last), then at kRowBloom its
// filter bits and at kRowSize its word count; 16-byte aligned.
constexpr uint32_t kRow = 12, kRowBloom = 9, kRowSize = 10;

// The voxels of the 4^3 leaf at (x0, y0, z0) whose cubes should_edit_impl
// takes, as leaf bits.  Its terms are per axis, so they are made for the 4
// voxel slabs of each axis: a box is an and of three slab masks, and a sphere
// 64 sums of three squares in should_edit_impl's order (a slab the centre
// lies in takes nothing away).  The leaf level's evaluation, a thread a leaf,
// was bound by 64 whole tests: the children of a level (spawned, classified,
// leaves evaluated) went from 12.4 to 7.9 us for 4,816 of them, from 28 to 10
// us for 184,528.
HD_D uint64_t leaf_edit_mask(const Editor& e, uint32_t x0, uint32_t y0, uint32_t z0)
{
    if (e.sphere()) {
        float sx[4], sy[4], sz[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) {
            const float mnx = float(x0 + k), mny = float(y0 + k), mnz = float(z0 + k);
            const float mxx = mnx + 1.0f, mxy = mny + 1.0f, mxz = mnz + 1.0f;
            sx[k] = e.cx < mnx ? sqr(e.cx - mnx) : e.cx > mxx ? sqr(e.cx - mxx) : 0.0f;
            sy[k] = e.cy < mny ? sqr(e.cy - mny) : e.cy > mxy ? sqr(e.cy - mxy) : 0.0f;
            sz[k] = e.cz < mnz ? sqr(e.cz - mnz) : e.cz > mxz ? sqr(e.cz - mxz) : 0.0f;
        }
        uint32_t half[2] = {0, 0};
#pragma unroll
        for (uint32_t b = 0; b < 64; b++) {
            const uint32_t c1 = b >> 3, c2 = b & 7;
            const float d = ((e.r2 - sx[((c1 >> 2) & 1) * 2 + ((c2 >> 2) & 1)]) -
                             sy[((c1 >> 1) & 1) * 2 + ((c2 >> 1) & 1)]) -
                            sz[(c1 & 1) * 2 + (c2 & 1)];
            half[b >> 5] |= (d > 0 ? 1u : 0u) << (b & 31);
        }
        return uint64_t(half[0]) | (uint64_t(half[1]) << 32);
    }
    auto taken = [](float lo, float hi, float mn) {
        const float mx = mn + 1.0f;
        return !(lo >= mx || hi <= mn || mn >= hi || mx <= lo);
    };
    uint64_t mx = 0, my = 0, mz = 0;
#pragma unroll
    for (uint32_t k = 0; k < 4; k++) {
        // slab k of an axis: the half of the 2^3 blocks (bytes) and of the
        // voxels in a block (bits of a byte)
        mx |= taken(e.bminx, e.bmaxx, float(x0 + k)) ? ((k & 2) ? 0xFFFFFFFF00000000ull : 0x00000000FFFFFFFFull) &
                                                           ((k & 1) ? 0xF0F0F0F0F0F0F0F0ull : 0x0F0F0F0F0F0F0F0Full)
                                                     : 0ull;
        my |= taken(e.bminy, e.bmaxy, float(y0 + k)) ? ((k & 2) ? 0xFFFF0000FFFF0000ull : 0x0000FFFF0000FFFFull) &
                                                           ((k & 1) ? 0xCCCCCCCCCCCCCCCCull : 0x3333333333333333ull)
                                                     : 0ull;
        mz |= taken(e.bminz, e.bmaxz, float(z0 + k)) ? ((k & 2) ? 0xFF00FF00FF00FF00ull : 0x00FF00FF00FF00FFull) &
                                                           ((k & 1) ? 0xAAAAAAAAAAAAAAAAull : 0x5555555555555555ull)
                                                     : 0ull;
    }
    return mx & my & mz;
}

// The leaf after the tool: get_new_value of its edited voxels.
HD_D uint64_t edited_leaf(const Editor& e, uint32_t x0, uint32_t y0, uint32_t z0, uint64_t leaf, uint64_t edited)
{
    if (e.shortcuts()) // sphere and box carve / fill: the same value everywhere
        return e.adding() ? (leaf | edited) : (leaf & ~edited);
    if (e.tool == HD_TOOL_SPHERE_PAINT)
        return leaf;
    uint64_t out = leaf;
    for (uint64_t todo = edited; todo; todo &= todo - 1) {
        const uint32_t b = __ffsll((long long)todo) - 1, c1 = b >> 3, c2 = b & 7;
        const float px = float(x0 + ((c1 >> 2) & 1) * 2 + ((c2 >> 2) & 1));
        const float py = float(y0 + ((c1 >> 1) & 1) * 2 + ((c2 >> 1) & 1));
        const float pz = float(z0 + (c1 & 1) * 2 + (c2 & 1));
        const uint64_t bit = 1ull << b;
        out = new_value(e, px, py, pz, (leaf & bit) != 0) ? (out | bit) : (out & ~bit);
    }
    return out;
}

// ---- per-level entry state ---------------------------------------------------
enum : uint8_t {
    kSkip = 0,      // level-C_colorTreeLevels child the parent never hands to edit_leaf
    kKeep = 1,      // untouched: result = old
    kEmptied = 2,   // carved away (is_empty)
    kFilled = 3,    // filled (is_full): the level's full node
    kLeafEval = 4,  // leaf rebuilt voxel by voxel
    kDescend = 5,   // interior node rebuilt from its children
};

struct Level {
    uint32_t* x;
    uint32_t* y;
    uint32_t* z;
    uint32_t* old;
    uint8_t* state;
    uint32_t* res;   // new index (kInvalid = empty)
    uint32_t* cnt;   // voxel count of the new node (levels >= T)
    uint32_t* flag;  // 1 = descends
    uint32_t* exp;   // exclusive scan of flag
    uint64_t* leaf;  // new leaf masks (leaf level only)
    uint32_t* cand;  // candidate rows, kRow words per entry
    // colours (allocated only when the context has colours)
    uint32_t* ocnt;  // voxel count of the old node (levels >= T)
    uint32_t* cn;    // levels < T: colour node; level T: the slot's leaf reference
    uint32_t* noff;  // offset in the task's new colour sequence (levels >= T)
    uint32_t* ooff;  // offset in the task's old leaf
    uint32_t* task;  // level-T entry the entry belongs to
};

struct EditCounters {
    unsigned long long num_voxels, num_nodes, foa, added, scanned;
};

HD_D void warp_add(unsigned long long* p, unsigned long long v)
{
    // warp-aggregated atomic
    const uint32_t mask = __activemask();
    for (int o = 16; o; o >>= 1)
        v += __shfl_down_sync(mask, v, o);
    if ((threadIdx.x & 31) == __ffs(mask) - 1)
        atomicAdd(p, v);
}

// Reads of a node's words.  CG = false: through the read-only path, for
// kernels during which the table does not change; CG = true: L2-coherent
// loads, for a launch that also appends to the table (the persistent batched
// edits read in one edit the nodes and pages an earlier edit of the same
// launch wrote).
template <bool CG>
struct NodeRead {
    const uint32_t* p;
    HD_D NodeRead(const Table& t, uint32_t v) : p(CG ? t.sys_cg(v) : t.sys(v)) {}
    HD_D uint32_t operator[](uint32_t k) const { return CG ? __ldcg(p + k) : p[k]; }
};

// Top-down classification of entry i of level `level` (edit_threaded /
// edit_leaf early exits); nodes / voxels: its share of the edit counters.
// The entry's path (x, y, z) and old node are given (a caller that has just
// spawned it holds them in registers); classify_entry reads them.
template <bool CG = false>
HD_D void classify_values(const Table& t, const Editor& ed, uint32_t level, const Level& lv, uint32_t i, uint32_t x,
                          uint32_t y, uint32_t z, uint32_t old, unsigned long long& nodes, unsigned long long& voxels)
{
    const uint32_t D = t.g.depth, T = t.g.T, leafl = t.g.leaf_level;
    const uint32_t depth = D - level;
    const float s = float(1u << depth);
    const float mnx = float(x << depth), mny = float(y << depth), mnz = float(z << depth);
    const float mxx = mnx + s, mxy = mny + s, mxz = mnz + s;
    const bool se = should_edit_impl(ed, mnx, mny, mnz, mxx, mxy, mxz);
    uint8_t state;
    uint32_t res = old, cnt = 0;
    nodes = 0;
    voxels = 0;
    if (level < T) {
        // edit_threaded: visited in both passes; no early full/empty exits
        nodes = 2;
        state = se ? kDescend : kKeep;
    } else {
        if (level == T && !se) {
            state = kSkip; // the parent keeps the old child without a visit
        } else {
            nodes = 1;
            if (!se) {
                state = kKeep;
                if (old != kInvalid) {
                    const NodeRead<CG> p(t, old);
                    cnt = level < leafl ? (p[0] >> 8) : popc32(p[0]) + popc32(p[1]);
                }
            } else if (ed.shortcuts() && inside_tool(ed, mnx, mny, mnz, mxx, mxy, mxz)) {
                const uint32_t full_count = 1u << (3 * depth);
                voxels = full_count;
                if (ed.adding()) {
                    state = kFilled;
                    res = t.full_nodes[level];
                    cnt = full_count;
                } else {
                    state = kEmptied;
                    res = kInvalid;
                }
            } else if (level == leafl) {
                state = kLeafEval;
                uint64_t leaf = 0;
                if (old != kInvalid) {
                    const NodeRead<CG> p(t, old);
                    leaf = uint64_t(p[0]) | (uint64_t(p[1]) << 32);
                }
                const uint64_t edited = leaf_edit_mask(ed, x << 2, y << 2, z << 2);
                voxels = popc64(edited);
                leaf = edited_leaf(ed, x << 2, y << 2, z << 2, leaf, edited);
                lv.leaf[i] = leaf;
            } else {
                state = kDescend;
            }
        }
    }
    lv.state[i] = state;
    lv.res[i] = res;
    lv.cnt[i] = cnt;
    lv.flag[i] = state == kDescend;
    if (lv.ocnt && level >= T) {
        uint32_t oc = 0;
        if (old != kInvalid) {
            const NodeRead<CG> p(t, old);
            oc = level < leafl ? (p[0] >> 8) : popc32(p[0]) + popc32(p[1]);
        }
        lv.ocnt[i] = oc;
    }
}

template <bool CG = false>
HD_D void classify_entry(const Table& t, const Editor& ed, uint32_t level, const Level& lv, uint32_t i,
                         unsigned long long& nodes, unsigned long long& voxels)
{
    classify_values<CG>(t, ed, level, lv, i, lv.x[i], lv.y[i], lv.z[i], lv.old[i], nodes, voxels);
}

// A descended entry spawns its 8 children (child order) at 8 * exp[i] on the
// next level.
HD_D void spawn_entry(const Table& t, const Level& lv, const Level& next, uint32_t i)
{
    if (!lv.flag[i])
        return;
    const uint32_t base = 8 * lv.exp[i];
    const uint32_t old = lv.old[i];
    uint32_t mask = 0;
    const uint32_t* p = nullptr;
    if (old != kInvalid) {
        p = t.sys(old);
        mask = p[0] & 0xffu;
    }
    uint32_t k = 1;
    for (uint32_t c = 0; c < 8; c++) {
        next.x[base + c] = (lv.x[i] << 1) | ((c >> 2) & 1);
        next.y[base + c] = (lv.y[i] << 1) | ((c >> 1) & 1);
        next.z[base + c] = (lv.z[i] << 1) | (c & 1);
        next.old[base + c] = (mask & (1u << c)) ? p[k++] : kInvalid;
    }
}

// Child c of descended entry i, written at slot `at` of the next level
// (spawn_entry for one child, with L2-coherent table reads); its path and
// old node are also returned (for classify_values).
HD_D void spawn_child(const Table& t, const Level& lv, const Level& next, uint32_t i, uint32_t c, uint32_t at,
                      uint32_t& x, uint32_t& y, uint32_t& z, uint32_t& child)
{
    const uint32_t old = lv.old[i];
    child = kInvalid;
    if (old != kInvalid) {
        const NodeRead<true> p(t, old);
        const uint32_t mask = p[0] & 0xffu;
        if (mask & (1u << c))
            child = p[child_offset(mask, c)];
    }
    x = (lv.x[i] << 1) | ((c >> 2) & 1);
    y = (lv.y[i] << 1) | ((c >> 1) & 1);
    z = (lv.z[i] << 1) | (c & 1);
    next.x[at] = x;
    next.y[at] = y;
    next.z[at] = z;
    next.old[at] = child;
}

// Bottom-up: the rebuilt content of entry i (kLeafEval / kDescend).  Unchanged
// and emptied nodes resolve at once (kNoBucket); otherwise the content goes
// to lv.cand and the function returns its bucket for find-or-add.
template <bool CG = false>
HD_D uint32_t candidate_entry(const Table& t, uint32_t level, const Level& lv, const Level& child, uint32_t i)
{
    const uint32_t T = t.g.T;
    const uint8_t state = lv.state[i];
    uint4* row = reinterpret_cast<uint4*>(lv.cand + uint64_t(kRow) * i);
    uint32_t hash;
    if (state == kLeafEval) {
        const uint64_t leaf = lv.leaf[i];
        const uint32_t old = lv.old[i];
        uint64_t initial = 0;
        if (old != kInvalid) {
            const NodeRead<CG> p(t, old);
            initial = uint64_t(p[0]) | (uint64_t(p[1]) << 32);
        }
        lv.cnt[i] = popc64(leaf);
        if (leaf == initial) {
            lv.res[i] = old;
            return kNoBucket;
        }
        if (!leaf) {
            lv.res[i] = kInvalid;
            lv.cnt[i] = 0;
            return kNoBucket;
        }
        const uint32_t w[9] = {uint32_t(leaf), uint32_t(leaf >> 32)};
        row[0] = make_uint4(w[0], w[1], 0, 0);
        row[1] = make_uint4(0, 0, 0, 0);
        row[2] = make_uint4(0, bloom_bits(w, 2), 2, 0);
        hash = hash_leaf(leaf);
    } else if (state == kDescend) {
        // the 8 children in three independent reads of each array (all were
        // spawned; old: the spawned child's old node, kInvalid where the old
        // node had none, so the old node itself is not read again), the
        // words hashed as they come: no chain of reads
        const uint32_t base = 8 * lv.exp[i];
        const uint32_t old = lv.old[i];
        uint32_t oc[8], nc[8], cc[8];
        const uint4* po = reinterpret_cast<const uint4*>(child.old + base);
        const uint4* pr = reinterpret_cast<const uint4*>(child.res + base);
        const uint4* pc = reinterpret_cast<const uint4*>(child.cnt + base);
        const uint2 st = *reinterpret_cast<const uint2*>(child.state + base);
#pragma unroll
        for (uint32_t h = 0; h < 2; h++) {
            const uint4 o = po[h], r = pr[h], n = level >= T ? pc[h] : make_uint4(0, 0, 0, 0);
            oc[4 * h] = o.x, oc[4 * h + 1] = o.y, oc[4 * h + 2] = o.z, oc[4 * h + 3] = o.w;
            nc[4 * h] = r.x, nc[4 * h + 1] = r.y, nc[4 * h + 2] = r.z, nc[4 * h + 3] = r.w;
            cc[4 * h] = n.x, cc[4 * h + 1] = n.y, cc[4 * h + 2] = n.z, cc[4 * h + 3] = n.w;
        }
        uint32_t mask = 0, total = 0;
        bool changed = false;
#pragma unroll
        for (uint32_t s = 0; s < 8; s++) {
            const uint32_t cs = ((s < 4 ? st.x : st.y) >> (8 * (s & 3))) & 0xffu;
            nc[s] = cs == kSkip ? oc[s] : nc[s];
            changed |= nc[s] != oc[s];
            if (nc[s] != kInvalid) {
                mask |= 1u << s;
                total += cc[s];
            }
        }
        lv.cnt[i] = total;
        if (!changed) {
            lv.res[i] = old;
            return kNoBucket;
        }
        if (!mask) {
            lv.res[i] = kInvalid;
            lv.cnt[i] = 0;
            return kNoBucket;
        }
        // the children packed to the front: a stable compaction by moves of
        // 4, 2 and 1 slots (a child moves left by the empty slots before it)
        uint32_t w[9], gap[8];
        w[0] = (level >= T ? (total << 8) : 0u) | mask;
#pragma unroll
        for (uint32_t s = 0; s < 8; s++)
            gap[s] = (mask >> s & 1u) ? popc32(~mask & ((1u << s) - 1u)) : 0u;
#pragma unroll
        for (uint32_t m = 1; m <= 4; m <<= 1)
#pragma unroll
            for (uint32_t s = m; s < 8; s++)
                if (gap[s] & m) {
                    nc[s - m] = nc[s];
                    gap[s - m] = gap[s] - m;
                    gap[s] = 0;
                }
        const uint32_t n = 1 + popc32(mask);
#pragma unroll
        for (uint32_t s = 0; s < 8; s++)
            w[1 + s] = s + 1 < n ? nc[s] : 0u;
        row[0] = make_uint4(w[0], w[1], w[2], w[3]);
        row[1] = make_uint4(w[4], w[5], w[6], w[7]);
        row[2] = make_uint4(w[8], bloom_bits(w, n), n, 0);
        hash = hash_interior_words(n, w);
    } else {
        return kNoBucket;
    }
    const uint32_t bucket = hash & (t.g.buckets(level) - 1);
    lv.res[i] = kNotFound; // resolved by find-or-add
    return bucket;
}

HD_D bool same_words(const uint4& a, const uint4& b)
{
    return a.x == b.x && a.y == b.y && a.z == b.z && a.w == b.w;
}
// The same words in two candidates' rows of a level
HD_D bool same_row(const uint32_t* a, const uint32_t* b, bool leaf)
{
    if (leaf) {
        const uint2 x = *reinterpret_cast<const uint2*>(a), y = *reinterpret_cast<const uint2*>(b);
        return x.x == y.x && x.y == y.y;
    }
    const uint4 *p = reinterpret_cast<const uint4*>(a), *q = reinterpret_cast<const uint4*>(b);
    return same_words(p[0], q[0]) && same_words(p[1], q[1]) && p[2].x == q[2].x;
}

// One warp per bucket: the bucket's candidates, in depth-first order, each
// resolved against the bucket as it stands (earlier candidates' appends
// included) and appended when not found.  A per-warp cache remembers, for
// every content already resolved in this bucket, the positions where a copy
// lies (the first match a scan sees, the bucket's last node when it holds
// the content, and the copies appended since): a repeated content then needs
// no new scan, only the visibility rule on those positions.  Runs of
// identical candidates after a found result take that result at once.
constexpr uint32_t kCache = 32;
constexpr uint32_t kCachePos = 3;

struct FoaCache {
    uint32_t words[kCache][9];
    uint32_t bloom[kCache]; // the words' filter bits: looked at first
    uint32_t npos[kCache];
    uint32_t pos[kCache][kCachePos];
};

// A node at bucket position p (a walk position) of size n is compared by the
// reference's interior scan iff p + n < min(S, page end) (leaves: always).
HD_D bool visible(uint32_t p, uint32_t n, uint32_t S, bool leaf)
{
    if (leaf)
        return p + 2 <= S;
    const uint32_t pe = (p & ~(kPage - 1)) + kPage;
    return p + n < (S < pe ? S : pe);
}

// A page's words in the warp's registers and in its shared buffer: load r of
// lane l holds words (32 r + l) PW .. + PW - 1 (PW, the probe width: 1, 2 or
// 4), every load issued before the first is used.  L2-coherent loads: the
// same kernel appends nodes and maps pages.  Words past `used`: whatever the
// page holds there, or zeros.
template <int PW>
HD_D void load_page(const uint32_t* src, uint32_t used, uint32_t (&v)[kPage / 32], uint32_t* page, uint32_t lane)
{
    constexpr uint32_t R = kPage / 32 / PW;
#pragma unroll
    for (uint32_t r = 0; r < R; r++) {
        const uint32_t w = (r * 32 + lane) * PW;
        const bool in = w < used;
        if constexpr (PW == 4) {
            const uint4 x = in ? __ldcg(reinterpret_cast<const uint4*>(src + w)) : make_uint4(0, 0, 0, 0);
            v[4 * r] = x.x, v[4 * r + 1] = x.y, v[4 * r + 2] = x.z, v[4 * r + 3] = x.w;
        } else if constexpr (PW == 2) {
            const uint2 x = in ? __ldcg(reinterpret_cast<const uint2*>(src + w)) : make_uint2(0, 0);
            v[2 * r] = x.x, v[2 * r + 1] = x.y;
        } else {
            v[r] = in ? __ldcg(src + w) : 0u;
        }
    }
#pragma unroll
    for (uint32_t r = 0; r < R; r++) {
        const uint32_t w = (r * 32 + lane) * PW;
        if constexpr (PW == 4)
            *reinterpret_cast<uint4*>(page + w) = make_uint4(v[4 * r], v[4 * r + 1], v[4 * r + 2], v[4 * r + 3]);
        else if constexpr (PW == 2)
            *reinterpret_cast<uint2*>(page + w) = make_uint2(v[2 * r], v[2 * r + 1]);
        else
            page[w] = v[r];
    }
}

// The walk from the page's start meets word `at` (lane 0 walks).
HD_D bool walk_meets(const uint32_t* page, uint32_t at)
{
    uint32_t on = 0;
    if ((threadIdx.x & 31) == 0) {
        uint32_t p = 0;
        while (p < at)
            p += total_size(page[p]);
        on = p == at;
    }
    return __shfl_sync(0xffffffffu, on, 0) != 0;
}

// The first word below `lim` of the staged page at which the n words of q lie,
// on the walk (warp-wide); kNotFound when there is none.  Leaves: at even
// words.  Interiors: `starts`, the page's start bits, says at once that a
// match is on the walk; a match that is no start is walked to.
template <int PW>
HD_D uint32_t match_page(const uint32_t (&v)[kPage / 32], const uint32_t* page, const uint32_t* starts,
                         const uint32_t* q, uint32_t n, uint32_t lim, bool leaf)
{
    const uint32_t lane = threadIdx.x & 31;
    uint32_t m = 0; // the lane's words equal to q[0]
#pragma unroll
    for (uint32_t k = 0; k < kPage / 32; k++)
        m |= (v[k] == q[0] ? 1u : 0u) << k;
    uint32_t best = kNotFound, odd = kNotFound; // the lowest match that is a start, that is not
    while (m) {
        const uint32_t k = __ffs(m) - 1;
        m &= m - 1;
        const uint32_t w = ((k / PW) * 32 + lane) * PW + k % PW;
        if (w >= lim || (leaf && (w & 1)))
            continue;
        bool eq = page[w + 1] == q[1];
        for (uint32_t j = 2; eq && j < n; j++)
            eq = page[w + j] == q[j];
        if (!eq)
            continue;
        if (leaf || ((starts[w >> 5] >> (w & 31)) & 1u))
            best = min(best, w);
        else
            odd = min(odd, w);
    }
    best = __reduce_min_sync(0xffffffffu, best);
    // (no loop over further odd matches: past the first that the walk misses,
    // each is looked at in turn)
    uint32_t first = __reduce_min_sync(0xffffffffu, odd);
    while (first < best) {
        if (walk_meets(page, first))
            return first;
        // the next odd match of any lane, found again from the staged words
        uint32_t next = kNotFound;
        for (uint32_t w = lane; w < lim; w += 32) {
            if (w <= first || ((starts[w >> 5] >> (w & 31)) & 1u))
                continue;
            bool eq = true;
            for (uint32_t j = 0; eq && j < n; j++)
                eq = page[w + j] == q[j];
            if (eq) {
                next = w;
                break;
            }
        }
        first = __reduce_min_sync(0xffffffffu, next);
    }
    return best;
}

// Words of a warp's query buffer: the rows of kRowsAhead candidates, then the
// start bits of the page being scanned.
constexpr uint32_t kRowsAhead = 8;
constexpr uint32_t kFoaQuery = kRow * kRowsAhead + 16;

// Warp-wide scan of the bucket for the first compared position holding q
// (find_leaf_node_in_bucket / find_interior_node_in_bucket); returns the
// bucket position or kNotFound.  *last_match: for interiors, the bucket's
// last node when it holds q (compared by no scan until something follows).
// Three dependent waits at most per scanned page: the size (the caller's)
// and the filters together, then a page with its start bits.  (With the
// pages' lines of 512 filter bits alone, a walk per match and words compared
// from shared memory 32 at a time, 53 buckets of a small level took 25 us;
// with runs dealt out to the warps as well, 7.6.)
template <int PW>
HD_D uint32_t scan_bucket(const Table& t, uint32_t vbase, uint32_t S, const uint32_t* q, uint32_t n, bool leaf,
                          uint32_t may, uint32_t bloom, uint32_t pt_lane, uint32_t* page, uint32_t* starts,
                          uint32_t* last_match, unsigned long long& scanned)
{
    const uint32_t lane = threadIdx.x & 31;
    uint32_t found = kNotFound, staged = kNotFound;
    *last_match = kNotFound;
    // page pi's physical page and whether its filter admits q: the first 32
    // pages' from pt_lane / may (a lane per page)
    auto page_of = [&](uint32_t pi) {
        const uint32_t near = __shfl_sync(0xffffffffu, pt_lane, pi & 31);
        return pi < 32 ? near : t.page_cg((vbase >> kPageShift) + pi);
    };
    auto admits = [&](uint32_t pi) {
        return pi < 32 ? ((may >> pi) & 1u) != 0 : bloom_may_phys(t, page_of(pi), bloom, leaf);
    };
    uint32_t v[kPage / 32];
    auto stage = [&](uint32_t pi, uint32_t used) {
        const uint32_t phys = page_of(pi);
        uint32_t sb = 0;
        if (!leaf && lane < 16)
            sb = __ldcg(t.meta + uint64_t(phys) * kPageMeta + kPageStarts + lane);
        __syncwarp();
        load_page<PW>(t.pool + (uint64_t(phys) << kPageShift), used, v, page, lane);
        if (!leaf && lane < 16)
            starts[lane] = sb;
        __syncwarp();
        staged = pi;
    };
    for (uint32_t pindex = 0; pindex < S && found == kNotFound; pindex += kPage) {
        const uint32_t page_end = S < pindex + kPage ? S : pindex + kPage;
        if (!leaf && pindex + n >= page_end)
            break; // "return 0xFFFFFFFF" of the reference scan
        const uint32_t pi = pindex / kPage;
        if (!admits(pi))
            continue; // the page cannot hold q
        const uint32_t used = page_end - pindex;
        stage(pi, used);
        const uint32_t w = match_page<PW>(v, page, starts, q, n, leaf ? used : used - n, leaf);
        if (w != kNotFound)
            found = pindex + w;
        scanned += found == kNotFound ? used : (found - pindex + n);
    }
    if (!leaf && found == kNotFound && S >= n && ((S - n) & ~(kPage - 1)) == ((S - 1) & ~(kPage - 1))) {
        // the bucket's last node ends at S; it holds q iff it starts at S - n
        // (nodes never straddle a page, so S - n lies in the tail's page,
        // whose used words hold nodes only)
        const uint32_t p = S - n, pi = p / kPage, at = p & (kPage - 1);
        if (admits(pi)) {
            if (staged != pi)
                stage(pi, ((S - 1) & (kPage - 1)) + 1);
            bool ok = lane >= n || page[at + lane] == q[lane];
            ok = __all_sync(0xffffffffu, ok) && ((starts[at >> 5] >> (at & 31)) & 1u);
            if (ok)
                *last_match = p;
        }
    }
    return found;
}

// A run of followers whose results are written after the find-or-add phase
// (hd_edit_persist.cu): positions [begin, end) of the sorted candidates take
// `result`.
struct FollowerRun {
    uint32_t begin, end, result, pad;
};
// The repeats of a level's sorted candidates: bit j set when candidate j has
// the bucket and the words of candidate j - 1; runs longer than kLongRun go
// to the list.
struct Repeats {
    const uint32_t* same; // null: not known
    uint32_t words;
    FollowerRun* runs;
    uint32_t* n_runs;
};
constexpr uint32_t kLongRun = 64;

// The end of the run of set bits from bit j on (warp-wide).
HD_D uint32_t end_of_repeats(const Repeats& rep, uint32_t j)
{
    const uint32_t lane = threadIdx.x & 31;
    uint32_t w0 = j >> 5, below = (1u << (j & 31)) - 1u;
    for (;;) {
        uint32_t word = w0 + lane < rep.words ? __ldcg(rep.same + w0 + lane) : 0u;
        if (lane == 0)
            word |= below;
        below = 0;
        const uint32_t open = __ballot_sync(0xffffffffu, word != 0xffffffffu);
        if (open) {
            const uint32_t l = __ffs(open) - 1;
            const uint32_t at = __shfl_sync(0xffffffffu, word, l);
            return (w0 + l) * 32 + __ffs(~at) - 1;
        }
        w0 += 32;
    }
}

// Resolves the candidates vals[j0..j1) of one bucket (all lanes of a warp):
// each gets its index in lv.res.  page / q / cache: the warp's shared
// buffers.  Returns false when an append failed (the device error word says
// why); the bucket size is written back either way.
template <int PW>
HD_D bool foa_segment(const Table& t, uint32_t level, const Level& lv, const uint32_t* __restrict__ vals, uint32_t j0,
                      uint32_t j1, uint32_t bucket, uint32_t* page, uint32_t* q, FoaCache& cache,
                      unsigned long long& foa, unsigned long long& added, unsigned long long& scanned,
                      const Repeats& rep = Repeats{})
{
    const uint32_t lane = threadIdx.x & 31;
    const bool leaf = level == t.g.leaf_level;
    const uint32_t gb = t.g.bucket_global(level, bucket);
    const uint32_t vbase = t.g.make_ptr(level, bucket, 0);
    // the bucket's page-table entries, lane p holding page p's (the warp owns
    // the bucket for the run: only its own appends map pages here)
    const uint32_t vpage0 = vbase >> kPageShift, cap_pages = t.g.capacity(level) >> kPageShift;
    uint32_t S = __ldcg(t.bucket_sizes + gb);
    uint32_t pt_lane = lane < cap_pages ? t.page_cg(vpage0 + lane) : 0u;
    uint32_t used_entries = 0, next_slot = 0;
    bool failed = false;
    uint32_t j = j0;
    // The rows of kRowsAhead candidates lie in shared memory (with the entry's
    // index in a row's last word), the next kRowsAhead on their way in
    // registers, so that the reads of a row wait for no candidate before it.
    constexpr uint32_t kLoads = kRow * kRowsAhead / 32;
    uint32_t ahead[kLoads], jb = j0, ja = j0;
    uint32_t* starts = q + kRow * kRowsAhead;
    auto load_rows = [&](uint32_t from) {
#pragma unroll
        for (uint32_t m = 0; m < kLoads; m++) {
            const uint32_t k = lane + 32 * m, jj = from + k / kRow, w = k % kRow;
            ahead[m] = 0;
            if (jj < j1) {
                const uint32_t entry = vals[jj];
                ahead[m] = w == kRow - 1 ? entry : lv.cand[kRow * uint64_t(entry) + w];
            }
        }
    };
    load_rows(j0);
    bool staged = false;
    while (j < j1 && !failed) {
        if (!staged || j >= jb + kRowsAhead) {
            if (staged && j - ja >= kRowsAhead) { // a run of repeats was passed over
                ja = j;
                load_rows(ja);
            }
            __syncwarp();
#pragma unroll
            for (uint32_t m = 0; m < kLoads; m++)
                q[lane + 32 * m] = ahead[m];
            __syncwarp();
            staged = true;
            jb = ja;
            ja = jb + kRowsAhead;
            if (ja < j1)
                load_rows(ja);
        }
        const uint32_t* qj = q + kRow * (j - jb);
        const uint32_t n = qj[kRowSize], bloom = qj[kRowBloom], ci = qj[kRow - 1];
        // cache lookup: lane e compares entry e's filter bits, then the lanes
        // a word each of an entry that has them
        uint32_t hb = __ballot_sync(0xffffffffu, lane < used_entries && cache.bloom[lane] == bloom);
        uint32_t e = kCache;
        while (hb && e == kCache) {
            const uint32_t k = __ffs(hb) - 1;
            hb &= hb - 1;
            if (__all_sync(0xffffffffu, lane >= 9 || cache.words[k][lane] == qj[lane]))
                e = k;
        }
        if (e == kCache) {
            // the filters of the bucket's first 32 pages, a lane per page,
            // beside the bucket size (they do not wait for it)
            const uint32_t maybe =
                __ballot_sync(0xffffffffu, lane < cap_pages && bloom_may_phys(t, pt_lane, bloom, leaf));
            uint32_t last_match;
            const uint32_t npages = (S + kPage - 1) / kPage;
            const uint32_t may = npages < 32 ? maybe & ((1u << npages) - 1u) : maybe;
            const uint32_t f =
                scan_bucket<PW>(t, vbase, S, qj, n, leaf, may, bloom, pt_lane, page, starts, &last_match, scanned);
            e = next_slot;
            next_slot = (next_slot + 1) % kCache;
            used_entries = used_entries < kCache ? used_entries + 1 : kCache;
            if (lane < 9)
                cache.words[e][lane] = qj[lane];
            if (lane == 0) {
                cache.bloom[e] = bloom;
                cache.npos[e] = 0;
                if (f != kNotFound)
                    cache.pos[e][cache.npos[e]++] = f;
                else if (last_match != kNotFound)
                    cache.pos[e][cache.npos[e]++] = last_match;
            }
            __syncwarp();
        }
        // the first visible copy, else append (the same on every lane)
        uint32_t result = kNotFound;
        const uint32_t np = cache.npos[e];
        for (uint32_t k = 0; k < np && result == kNotFound; k++)
            if (visible(cache.pos[e][k], n, S, leaf))
                result = cache.pos[e][k];
        const bool appended = result == kNotFound;
        if (appended) {
            uint32_t size = S;
            const uint32_t pos = append_position(size, n, leaf);
            // the pages below the size are mapped: an append that stays in
            // the size's last page reads no page-table entry
            const bool mapped = S > 0 && size <= ((S + kPage - 1) & ~(kPage - 1));
            uint32_t ok = 1;
            if (size > t.g.capacity(level)) {
                if (lane == 0)
                    set_error(t.error, kErrBucketFull, level, bucket, size);
                ok = 0;
            } else if (!mapped) {
                if (lane == 0)
                    ok = map_pages(t, level, bucket, pos, size);
                ok = __shfl_sync(0xffffffffu, ok, 0);
                // refresh the entries of the pages the append reached
                if (ok && lane < cap_pages && lane * kPage < size && lane * kPage + kPage > S)
                    pt_lane = t.page_cg(vpage0 + lane);
            }
            if (ok) {
                const uint32_t near = __shfl_sync(0xffffffffu, pt_lane, (pos >> kPageShift) & 31);
                const uint32_t phys = (pos >> kPageShift) < 32 ? near : t.page_cg(vpage0 + (pos >> kPageShift));
                if (lane < n)
                    __stcg(t.pool + (uint64_t(phys) << kPageShift) + (pos & (kPage - 1)) + lane, qj[lane]);
                if (lane == 0)
                    bloom_add_phys(t, phys, pos & (kPage - 1), bloom, leaf);
                result = pos;
                S = size;
                added++;
            } else {
                failed = true;
            }
            __syncwarp(); // the positions were read by every lane
            if (lane == 0 && ok) {
                if (cache.npos[e] == kCachePos) { // keep the newest copies
                    for (uint32_t k = 1; k < kCachePos; k++)
                        cache.pos[e][k - 1] = cache.pos[e][k];
                    cache.npos[e]--;
                }
                cache.pos[e][cache.npos[e]++] = pos;
            }
        }
        if (lane == 0)
            lv.res[ci] = vbase + result;
        foa++;
        if (failed)
            break;
        j++;
        // a found result holds for the identical candidates that follow
        if (!appended && rep.same) {
            const uint32_t e1 = min(end_of_repeats(rep, j), j1);
            if (e1 - j > kLongRun) {
                if (lane == 0)
                    rep.runs[atomicAdd(rep.n_runs, 1u)] = FollowerRun{j, e1, vbase + result, 0};
            } else {
                for (uint32_t k = j + lane; k < e1; k += 32)
                    lv.res[vals[k]] = vbase + result;
            }
            foa += e1 - j;
            j = e1;
        } else if (!appended && j < j1 &&
                   (j - jb >= kRowsAhead || __all_sync(0xffffffffu, lane >= 9 || qj[kRow + lane] == qj[lane]))) {
            // the next candidate is equal (or not staged): 128 candidates at
            // a time, their reads independent
            for (;;) {
                uint32_t entry[4];
                bool same[4];
#pragma unroll
                for (uint32_t m = 0; m < 4; m++) {
                    const uint32_t jj = j + 32 * m + lane;
                    entry[m] = jj < j1 ? vals[jj] : kNotFound;
                }
#pragma unroll
                for (uint32_t m = 0; m < 4; m++) {
                    same[m] = entry[m] != kNotFound;
                    if (same[m])
                        same[m] = same_row(lv.cand + kRow * uint64_t(entry[m]), qj, leaf);
                }
                uint32_t run = 128;
#pragma unroll
                for (int m = 3; m >= 0; m--) {
                    const uint32_t diff = __ballot_sync(0xffffffffu, !same[m]);
                    run = diff ? 32 * m + __ffs(diff) - 1 : run;
                }
#pragma unroll
                for (uint32_t m = 0; m < 4; m++)
                    if (32 * m + lane < run)
                        lv.res[entry[m]] = vbase + result;
                foa += run;
                j += run;
                if (run < 128)
                    break;
            }
        }
        __syncwarp();
    }
    if (lane == 0)
        __stcg(t.bucket_sizes + gb, S);
    return !failed;
}

// ---- the persistent launch (hd_edit_persist.cu) and its buffers (hd_edit_batch.cu)
// Level arrays sized by upper bounds of their entries, and the sort's arrays.
struct PersistLevels {
    std::vector<Level> lv;
    std::vector<uint32_t> caps;
    uint32_t *keys, *vals, *keys2, *vals2;
};
// The geometry of one edit as the persistent launch leaves it.
struct EditGeometry {
    EditCounters ctr;
    uint32_t root, deepest;
    std::vector<uint32_t> count; // entries per level (0 below the deepest)
};
// The batched forms sort by bucket in two passes of at most 2^9 digits: tables
// of at most 2^17 buckets a level (an entry without a bucket sorts behind
// them).  Edits of others are made level by level.
constexpr uint32_t kMaxSortBits = 17;
inline bool two_pass_sort(const Geom& g) { return g.top_bits <= kMaxSortBits && g.low_bits <= kMaxSortBits; }
// Buffers for one edit, or null when its levels may hold more entries than
// the persistent launch is used for, or have too many buckets.
const PersistLevels* one_edit_levels(hd_ctx* c, const Editor& ed);
// Runs one edit's geometry in one persistent launch; false when the edit is to
// be made level by level: a level outgrew its bound, the device did not take
// the launch, or a grid barrier ran out of time (another stream's kernels held
// SMs for seconds).  The root and the history are then as before; after a
// barrier that ran out the table may hold nodes of the edit already, some of
// which the edit then appends again (no scan compares a bucket's last node).
// hold_root: the root is left for the caller to set.
bool edit_geometry_persistent(hd_ctx* c, const Editor& ed, const PersistLevels& pl, bool hold_root, EditGeometry& out);
// One edit, level by level from the host (hd_edit.cu).
void edit_by_levels(hd_ctx* c, const hd_edit& e, hd_edit_stats* stats);

} // namespace hd
