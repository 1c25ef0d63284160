// k_engine.cu -- the query engine: closest / any hit over the two-level
// hashed stackless BVH with Bezier clipping.
//
// A query runs a few passes of two persistent kernels:
//
// k_collect walks the reference's traversal (BVH::hashIntersect,
// src/rt/BVH.h:178-350, nested through the object level as in
// Context::intersect, src/rt/RayTracer.cu:295-383) -- same stackless key /
// postponed-bit state, same perfect-hash backtracking, same nearer-child-first
// order -- and appends what it meets to the ray's chunk: each patch of a
// leaf with the entry distance of the leaf's box, and markers where it enters
// or leaves an object.  It culls with the ray's best t as known at the start
// of the pass (the ray's extent in the first pass).  When the chunk is full
// the ray parks: its key, postponed bits and node are saved and the next
// pass resumes it.
//
// k_clip and k_subdivide replay the reference's leaf callbacks over the chunk in order: a
// patch whose leaf box starts at or beyond the object's current best t is
// skipped (the reference's `L0 < hit.t` test), any other runs the
// Bezier-clipping search with the current best as hit.distance
// (doBezierClipping, src/Spline_BezierClipping.cu:46-114) and keeps a
// strictly closer hit; leaving an object keeps its hit if it beats the world
// best.  A subtree the reference culls lies behind its box entry, at or
// beyond the best t of that moment, so none of its patches can give a
// strictly closer hit; collecting it anyway changes nothing except for hits
// within the search tolerance of the current best (near-ties).  Any-hit
// queries stop at the first patch that reports a hit; at the end of an
// any-hit launch, lanes without rays share the pending intervals of the long
// searches left in their warp.
//
// Patch BVHs with a walk tree (DevBVH::walkBase) are collected on it instead:
// a tree over the same leaf boxes, split on the longest axis, which needs a
// fraction of the node visits of the reference's y-only splits (23.7 against
// 392 inner nodes per ray of the 1920x1080 frame over 16,384 patches).  A
// ray's list comes out the same, entry by entry:
//   * a chunk culls by a bound that is constant while the ray is inside an
//     object, and the slab test is monotone (a box that contains another is met
//     whenever the other is, entering no later, in FP32 as in the reals), so
//     any tree over the same leaf boxes reaches exactly the leaves whose own
//     box passes the test;
//   * the entry distances are slab tests of the same boxes;
//   * k_order puts an object's patches into the reference traversal's order:
//     of two leaves, the one in the nearer child of their lowest common
//     ancestor in the reference tree comes first.  The ancestor's key is the
//     common prefix of the leaves' heap keys, and the perfect hash finds its
//     node.  (Any-hit answers do not depend on the order.)
//   * an object whose patches do not fit in the chunk sends the ray's list to one
//     of a few long lists; where none is left or that fills too, the object is
//     collected again on the reference tree, which parks the ray exactly where it
//     would have parked.
//
// Both kernels refill lanes one ray (k_collect) or one clip iteration
// (the search kernels) at a time, so heavy-tailed per-ray work does not idle the other
// lanes of a warp, and take rays in id order so a warp's rays stay coherent.
// Rays still unfinished after the configured number of passes are completed
// by k_rest, the inline version of the same search.  Block sizes, grid
// occupancy and the pass count are runtime settings (EngineConfig), chosen by
// the autotuner (cgs_autotune) or set by the caller.
#include <algorithm>
#include <mutex>

#include "kernels.h"

namespace cgs {

namespace {

constexpr int kCollectThreads = 256;   // launch bound; runtime block size 128 or 256
constexpr int kResolveThreads = 128;   // launch bound; runtime block size 64 or 128
constexpr uint32_t kChunk = 64;        // list entries per ray and pass (the most; EngineConfig::queueChunk is the first pass's)
// One collect step appends at most two entries: a leaf's first patch and,
// when that patch ends the leaf and nothing is postponed inside the object,
// the marker that leaves the object.
constexpr uint32_t kMaxAppendsPerStep = 2;
// Backtrack cache: the node indices of the last kRing postponed siblings of
// each lane's ray, in a ring in shared memory.
constexpr uint32_t kRing = 8;
constexpr int kMaxPasses = 8;

// list entry word 0: a patch index, or one of these markers (word 1 = object)
constexpr uint32_t kLeave = 0xFFFFFFFFu, kEnter = 0xFFFFFFFEu, kCont = 0xFFFFFFFDu;
// or, in place of the first entry: the list is long list word 1
constexpr uint32_t kLong = 0xFFFFFFFCu;
constexpr uint32_t kLongList = 256;  // entries of a long list
// ray status
enum : uint32_t { kPending = 0, kTraversed = 1, kFinished = 2 };

struct Eng  // per-ray engine state, SoA over the query's capacity
{
    uint32_t *status, *count;
    uint2* list;  // [cap * kChunk]
    uint32_t *node, *key, *post, *leaf, *tnode, *tkey, *tpost, *tleaf, *jumped;
    int32_t *obj, *lpatch;
    float *leafEntry, *limit, *lt, *lu, *lv;
    // the rays to walk in pass p >= 1 (those that parked in pass p - 1) are
    // queue[p & 1][0 .. ctl[4p + 2]); the rays still parked after the last
    // pass P, for the inline fallback, are queue[P & 1][0 .. ctl[4P + 2]).
    // k_pending builds each in ray order, 256 rays at a time.
    uint32_t* queue[2];
    uint32_t* ctl;  // per pass: collect fetch, resolve fetch, length of the pass's queue
    uint32_t chunk;        // list entries a ray may fill in the first pass; each later pass doubles it (<= kChunk)
    uint32_t packetWidth;  // idle lanes a warp gathers before the traversal refills it
    uint32_t originLast;   // any hit: search candidates whose leaf box holds the ray's origin last
    uint32_t subdivLevels; // subdivision searches: bisection levels a lane runs per resolve round
    // Long lists, for the few rays whose candidates on a walk tree outgrow their
    // chunk: kLongList entries each, taken by *longNext, nlong of them (none left:
    // the ray goes back to the reference tree).  Each query has them all.
    uint2* longs;
    uint32_t nlong;
    uint32_t allMarkers;  // lists keep the markers of objects that the ray meets no patch of (cgs_traverse)
    uint32_t* longNext;
    __device__ __forceinline__ uint2* list_of(uint32_t rid) const
    {
        uint2* l = list + size_t(rid) * kChunk;
        const uint2 first = l[0];
        return first.x == kLong ? longs + size_t(first.y) * kLongList : l;
    }
};

constexpr size_t kWordsPerRay = 2 + 2 * kChunk + 18;
// Long lists of a scratch area for cap rays: 43 bytes a ray, 7% of its scratch (a
// single ray has one: servers of a few KB run too).
constexpr uint32_t long_lists(uint32_t cap) { return cap / 48 + (cap < 32 ? cap : 32); }

Eng carve(uint32_t* base, uint32_t cap)
{
    Eng e;
    uint32_t* p = base;
    auto take = [&](size_t words) { uint32_t* r = p; p += words; return r; };
    e.status = take(cap); e.count = take(cap);
    e.list = reinterpret_cast<uint2*>(take(2ull * cap * kChunk));
    e.node = take(cap); e.key = take(cap); e.post = take(cap); e.leaf = take(cap); e.tnode = take(cap);
    e.tkey = take(cap); e.tpost = take(cap); e.tleaf = take(cap); e.jumped = take(cap);
    e.obj = reinterpret_cast<int32_t*>(take(cap)); e.lpatch = reinterpret_cast<int32_t*>(take(cap));
    e.leafEntry = reinterpret_cast<float*>(take(cap)); e.limit = reinterpret_cast<float*>(take(cap));
    e.lt = reinterpret_cast<float*>(take(cap)); e.lu = reinterpret_cast<float*>(take(cap));
    e.lv = reinterpret_cast<float*>(take(cap));
    e.queue[0] = take(cap); e.queue[1] = take(cap);
    e.ctl = take(4 * (kMaxPasses + 1));
    if (size_t(p - base) % 2) p++;
    e.nlong = long_lists(cap);
    e.longs = reinterpret_cast<uint2*>(take(2ull * e.nlong * kLongList));
    e.longNext = nullptr;
    e.allMarkers = 0;
    return e;
}

// The tree a lane walks: its BVH's index in the scene's BVH table, the first
// node record (of the compressed mirror where `compressed`) and the first leaf
// list word.  indexBase EMPTY: a walk tree, whose leaves name their patch in
// place of a list.
struct BvhRef { uint32_t idx, nodeBase, indexBase; bool compressed; };

template<bool kQ, bool kWalk> __device__ __forceinline__ BvhRef bvh_ref(const DevScene& S, uint32_t idx, bool walk)
{
    const DevBVH& d = S.bvhs[idx];
    const uint32_t walkBase = kWalk ? __ldg(&d.walkBase) : EMPTY;
    const bool w = walk && walkBase != EMPTY;
    // the mirror holds the tree that is walked; a ray sent back to the other reads its exact records
    const bool q = kQ && __ldg(&d.compressed) != 0 && (w || walkBase == EMPTY);
    return BvhRef {idx, q ? __ldg(&d.qnodeBase) : w ? walkBase : __ldg(&d.nodeBase),
                   w ? EMPTY : __ldg(&d.indexBase), q};
}

// Warp-wide refill: every lane in `need` gets the next index from *fetch.
// width > 1: the warp waits until at least `width` of its lanes need one (or
// none is busy) and then refills them together: rays enter the warp in
// packets, which keeps its lanes at similar depths of similar walks.
__device__ __forceinline__ uint32_t warp_fetch(uint32_t* fetch, bool need, uint32_t width = 1, bool busy = false)
{
    unsigned m = __ballot_sync(0xFFFFFFFFu, need);
    if (!m) return EMPTY;
    if (width > 1 && uint32_t(__popc(m)) < width && __ballot_sync(0xFFFFFFFFu, busy)) return EMPTY;
    int leader = __ffs(m) - 1;
    uint32_t base = 0;
    if ((int)lane_id() == leader) base = atomicAdd(fetch, (uint32_t)__popc(m));
    base = __shfl_sync(0xFFFFFFFFu, base, leader);
    unsigned lt = (1u << lane_id()) - 1u;
    return need ? base + __popc(m & lt) : EMPTY;
}

// Where a kernel's warps take their rays.  A pass of the whole query: pass 0
// takes every ray, a later pass the queue of rays that parked; which: 0 the
// traversal's counter, 1 the searches'.  (Everything but m is recomputed from the
// kernel's arguments, so that it holds no registers.)
template<int which> struct PassSource
{
    const Eng& E;
    int pass;
    uint32_t m;
    __device__ __forceinline__ PassSource(const Eng& E, int pass, uint32_t n0, const uint32_t* nDev)
        : E(E), pass(pass), m(pass == 0 ? (nDev ? *nDev : n0) : E.ctl[4 * pass + 2])
    {
    }
    __device__ __forceinline__ uint32_t* fetch() const { return E.ctl + 4 * pass + which; }
    __device__ __forceinline__ uint32_t ray(uint32_t k) const { return pass == 0 ? k : E.queue[pass & 1][k]; }
};
// One warp's own rays: m of them from a queue, or from `base` on.
struct WarpSource
{
    uint32_t* next;
    uint32_t m, base;
    const uint32_t* queue;
    __device__ __forceinline__ uint32_t* fetch() const { return next; }
    __device__ __forceinline__ uint32_t ray(uint32_t k) const { return queue ? queue[k] : base + k; }
};

__device__ __forceinline__ void load_ray(const RaysSoA& r, uint32_t i, float3& o, float3& d, float& tmax)
{
    o = f3(r.ox[i], r.oy[i], r.oz[i]);
    d = f3(r.dx[i], r.dy[i], r.dz[i]);
    tmax = r.tmax ? r.tmax[i] : INFINITY;
}

// ------------------------------------------------------------ collect --
//
// A backtrack goes to the sibling postponed deepest on the current path: the
// one postponed last.  With the backtrack cache on, a step that postpones a
// sibling also pushes its node index on the lane's ring, and a backtrack pops
// it from there while it is still in the ring; otherwise (the ring held more
// than kRing postponed siblings, or the ray was parked since) it looks the
// sibling's key up in the perfect hash as BVH::hashIntersect does.  Both give
// the same node.  `rvalid` counts the entries at the top of the ring that are
// still intact; an object's traversal nests inside the object level's on the
// same ring, since it leaves the object only with nothing postponed.
//
// kQ: read the 32-byte compressed node mirror (one 256-bit load; child boxes
// on an 8-bit grid, widened outward) instead of the exact 64-byte records.
// The decoded boxes contain the exact ones, so the walk meets every leaf the
// exact walk meets (and a few more), with leaf entries no later: the list
// holds the same patches plus some the resolve step then clips or culls.
//
// kWalk: some surface has a walk tree; stores without any run an instance
// without that code.
template<bool kAny, bool kQ, bool kWalk, class Source>
__device__ __forceinline__ void collect_rays(const DevScene& S, const RaysSoA& rays, const Eng& E, int pass, int cache,
                                             const Source& src, uint32_t* ring, LocalCounters& lc, uint32_t& nrays)
{
    // entry s of this lane's ring at ring[s * blockDim.x + threadIdx.x]; the
    // ring's state packs its top slot (bits 0-2) with `rvalid` (bits 3-6)
    uint32_t rstate = 0;
    bool active = false, exhausted = false, jumped = false;
    uint32_t rid = 0, ncand = 0;
    // o, inv, limit: the world ray and its culling bound; co, ci, clim: those
    // of the level walked now (the world's, or the object's local ray and
    // best t), switched where the ray enters or leaves an object
    float3 o = f3(0, 0, 0), inv = f3(0, 0, 0), co = f3(0, 0, 0), ci = f3(0, 0, 0);
    float tmax = 0, limit = 0, clim = 0;
    uint32_t node = 0, key = 1, post = 0, leaf = EMPTY, tnode = 0, tkey = 1, tpost = 0, tleaf = EMPTY;
    float leafEntry = -INFINITY;
    int32_t obj = -1;
    bool walk = true;     // false: the object in hand is walked on the reference tree
    bool hollow = false;  // the list ends with the marker that entered the object in hand
    uint32_t topIdx = 0;  // the ray's object-level BVH (its group's)
    BvhRef B {};  // the BVH walked now; its hash parameters are read at a table lookup
    uint2* list = nullptr;
    uint32_t cap = 0;  // entries that the list in hand holds
    const uint32_t m = src.m;
    for (;;)
    {
        const bool need = !active && !exhausted;
        // a lane the packet rule holds back gets EMPTY (ray counts stay below 2^31)
        const uint32_t idx = warp_fetch(src.fetch(), need, E.packetWidth, active);
        if (need && idx != EMPTY)
        {
            const uint32_t r = idx < m ? src.ray(idx) : 0u;
            if (idx >= m)
                exhausted = true;
            else if (pass == 0 && rays.group && __ldg(rays.group + r) >= S.ngroups)
            {
                // a group outside the store: the ray stays a miss and raises an error bit
                lc.errors |= kErrGroup;
                E.count[r] = 0;
                E.status[r] = kTraversed;
            }
            else if (pass == 0 || E.status[r] == kPending)
            {
                rid = r;
                const uint32_t g = rays.group ? __ldg(rays.group + rid) : 0u;
                active = true;
                float3 d;
                load_ray(rays, rid, o, d, tmax);
                inv = f3(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
                list = E.list + size_t(rid) * kChunk;
                cap = min(kChunk, E.chunk << pass);
                ncand = 0;
                rstate = 0;
                topIdx = __ldg(S.groupTop + g);
                if (pass == 0)
                {
                    node = 0; key = 1; post = 0; leaf = EMPTY; obj = -1; jumped = false;
                    leafEntry = -INFINITY; limit = tmax;
                    co = o; ci = inv; clim = limit;
                    B = bvh_ref<kQ, kWalk>(S, topIdx, false);
                    walk = true;
                    nrays++;
                }
                else
                {
                    node = E.node[rid]; key = E.key[rid]; post = E.post[rid]; leaf = E.leaf[rid];
                    const uint32_t flags = E.jumped[rid];
                    jumped = (flags & 1u) != 0; walk = (flags & 2u) == 0; leafEntry = E.leafEntry[rid]; obj = E.obj[rid];
                    limit = kAny ? tmax : E.limit[rid];
                    co = o; ci = inv; clim = limit;
                    B = bvh_ref<kQ, kWalk>(S, topIdx, false);
                    if (obj >= 0)
                    {
                        tnode = E.tnode[rid]; tkey = E.tkey[rid]; tpost = E.tpost[rid]; tleaf = E.tleaf[rid];
                        const DevObject& O = S.objects[obj];
                        float3 ld; float sinv, lmax;
                        to_local(O, o, d, tmax, co, ld, lmax, sinv);
                        ci = f3(1.0f / ld.x, 1.0f / ld.y, 1.0f / ld.z);
                        clim = kAny ? lmax : E.lt[rid];
                        B = bvh_ref<kQ, kWalk>(S, O.surface, walk);
                        list[ncand++] = make_uint2(kCont, uint32_t(obj));
                        hollow = false;
                    }
                }
            }
        }
        if (__ballot_sync(0xFFFFFFFFu, active || !exhausted) == 0) break;
        if (!active) continue;

        if (ncand + kMaxAppendsPerStep > cap)
        {
            if (kWalk && obj >= 0 && B.indexBase == EMPTY)
            {
                // a full chunk goes on in a long list: a search of all of an
                // object's candidates in the reference order keeps the same
                // hit as one chunk by chunk, which would cull some of them first
                if (cap == kChunk && E.nlong)
                {
                    // (looked at first: the count stops soon after the last)
                    const uint32_t at = *(volatile uint32_t*)E.longNext < E.nlong ? atomicAdd(E.longNext, 1u) : E.nlong;
                    if (at < E.nlong)
                    {
                        uint2* l = E.longs + size_t(at) * kLongList;
                        for (uint32_t k = 0; k < ncand; k++) l[k] = list[k];
                        list[0] = make_uint2(kLong, at);
                        list = l;
                        cap = kLongList;
                        continue;
                    }
                }
                // the object's patches do not fit: collect it again on the
                // reference tree, whose order decides which of them do
                do ncand--; while (list[ncand].x != kEnter);
                ncand++;
                hollow = true;
                walk = false;
                node = 0; key = 1; post = 0; leaf = EMPTY; jumped = false;
                leafEntry = -INFINITY;
                rstate = 0;
                B = bvh_ref<kQ, kWalk>(S, B.idx, false);
                continue;
            }
            // no room for what one step may append: park before this step
            E.node[rid] = node; E.key[rid] = key; E.post[rid] = post; E.leaf[rid] = leaf;
            E.jumped[rid] = (jumped ? 1u : 0u) | (walk ? 0u : 2u); E.leafEntry[rid] = leafEntry; E.obj[rid] = obj;
            E.tnode[rid] = tnode; E.tkey[rid] = tkey; E.tpost[rid] = tpost; E.tleaf[rid] = tleaf;
            E.count[rid] = ncand;
            E.status[rid] = kPending;
            active = false;
            continue;
        }

        bool ascend = false, done = false;
        if (leaf != EMPTY)
        {
            const uint32_t e = __ldg(S.indices + B.indexBase + leaf);
            if (e != EMPTY)
            {
                leaf++;
                if (obj < 0)
                {
                    // descend into object e (Context::intersect's callback)
                    tnode = node; tkey = key; tpost = post; tleaf = leaf;
                    obj = int32_t(e);
                    const DevObject& O = S.objects[e];
                    const float3 d = f3(rays.dx[rid], rays.dy[rid], rays.dz[rid]);
                    float3 ld; float sinv;
                    to_local(O, o, d, tmax, co, ld, clim, sinv);
                    ci = f3(1.0f / ld.x, 1.0f / ld.y, 1.0f / ld.z);
                    B = bvh_ref<kQ, kWalk>(S, O.surface, true);
                    node = 0; key = 1; post = 0; leaf = EMPTY; jumped = false;
                    leafEntry = -INFINITY;
                    list[ncand++] = make_uint2(kEnter, e);
                    hollow = true;
                }
                else
                {
                    list[ncand++] = make_uint2(e, __float_as_uint(leafEntry));
                    hollow = false;
                }
            }
            else
            {
                leaf = EMPTY;
                ascend = true;
            }
        }
        else
        {
            // the node: its compressed record (one 256-bit load) where the BVH
            // has them, else the exact 64-byte record (two); the box tests of
            // an inner node's children, or of a leaf's own box when the leaf
            // was reached through a backtrack
            const float3 ro = co, ri = ci;
            uint32_t left, right;
            float L0 = 0.0f, R0 = 0.0f;
            bool mL = false, mR = false;
            if (kQ && B.compressed)
            {
                uint4 qa, qb;
                ldg256u(S.qnodes + 2ull * (B.nodeBase + node), qa, qb);
                const bool isLeaf = ((qa.w >> 24) & kQNodeLeaf) != 0;
                left = isLeaf ? EMPTY : node + 1;
                right = qb.w;
                if (!isLeaf || jumped) qslab2(qa, qb, ro, ri, L0, mL, R0, mR);
            }
            else
            {
                const float4* q = S.nodes + 4ull * (B.nodeBase + node);
                float4 q0, q1, q2, q3;
                ldg256(q, q0, q1);
                ldg256(q + 2, q2, q3);
                left = __float_as_uint(q3.x);
                right = __float_as_uint(q3.y);
                if (left != EMPTY || jumped) mL = slab(L0, f3(q0.x, q0.y, q0.z), f3(q0.w, q1.x, q1.y), ro, ri);
                if (left != EMPTY) mR = slab(R0, f3(q1.z, q1.w, q2.x), f3(q2.y, q2.z, q2.w), ro, ri);
            }
            if (left == EMPTY)
            {
                // reached through a backtrack: its entry is the slab test of its own box
                if (jumped) leafEntry = L0;
                jumped = false;
                // the leaf's first element and the one after it in the same step: a
                // one-element leaf (the build's element count per leaf) is done here
                uint32_t e0 = right, e1 = EMPTY;
                if (!kWalk || B.indexBase != EMPTY)
                {
                    e0 = __ldg(S.indices + B.indexBase + right);
                    e1 = __ldg(S.indices + B.indexBase + right + 1);
                }
                leaf = right + 1;
                if (e0 == EMPTY)
                {
                    leaf = EMPTY;
                    ascend = true;
                }
                else if (obj < 0)
                {
                    // descend into object e0 (Context::intersect's callback)
                    tnode = node; tkey = key; tpost = post; tleaf = leaf;
                    obj = int32_t(e0);
                    const DevObject& O = S.objects[e0];
                    const float3 d = f3(rays.dx[rid], rays.dy[rid], rays.dz[rid]);
                    float3 ld; float sinv;
                    to_local(O, o, d, tmax, co, ld, clim, sinv);
                    ci = f3(1.0f / ld.x, 1.0f / ld.y, 1.0f / ld.z);
                    B = bvh_ref<kQ, kWalk>(S, O.surface, true);
                    node = 0; key = 1; post = 0; leaf = EMPTY; jumped = false;
                    leafEntry = -INFINITY;
                    list[ncand++] = make_uint2(kEnter, e0);
                    hollow = true;
                }
                else
                {
                    list[ncand++] = make_uint2(e0, __float_as_uint(leafEntry));
                    hollow = false;
                    if (e1 == EMPTY)
                    {
                        leaf = EMPTY;
                        ascend = true;
                    }
                }
            }
            else
            {
                lc.nodes++;
                jumped = false;
                const float lim = clim;
                const bool iL = mL && L0 < lim;
                const bool iR = mR && R0 < lim;
                if (iL || iR) post <<= 1;
                if (iL && iR)
                {
                    post |= 1u;
                    uint32_t other;
                    if (L0 < R0) { key = key << 1; node = left; leafEntry = L0; other = right; }
                    else { key = (key << 1) ^ 1u; node = right; leafEntry = R0; other = left; }
                    if (cache)
                    {
                        const uint32_t top = (rstate + 1u) & (kRing - 1u);
                        ring[top * blockDim.x + threadIdx.x] = other;
                        rstate = top | (min((rstate >> 3) + 1u, kRing) << 3);
                    }
                }
                else if (iL) { key = key << 1; node = left; leafEntry = L0; }
                else if (iR) { key = (key << 1) ^ 1u; node = right; leafEntry = R0; }
                else ascend = true;
            }
        }
        if (ascend)
        {
            if (post == 0)
            {
                if (obj < 0)
                    done = true;
                else
                {
                    // an object without candidates leaves nothing in the list: the search
                    // kernel enters no object in vain and skips rays that miss (2,073,600
                    // primary rays 2.56 -> 2.49 ms)
                    if (hollow && !E.allMarkers) ncand--;
                    else list[ncand++] = make_uint2(kLeave, uint32_t(obj));
                    obj = -1;
                    walk = true;
                    co = o; ci = inv; clim = limit;
                    B = bvh_ref<kQ, kWalk>(S, topIdx, false);
                    node = tnode; key = tkey; post = tpost; leaf = tleaf;
                    leafEntry = -INFINITY;
                }
            }
            else
            {
                const int levels = __ffs(post) - 1;
                post >>= levels;
                key = (key >> levels) ^ 1u;
                post ^= 1u;
                lc.hashLookups++;
                if (rstate >= kRing)
                {
                    const uint32_t top = rstate & (kRing - 1u);
                    node = ring[top * blockDim.x + threadIdx.x];
                    rstate = ((top - 1u) & (kRing - 1u)) | (rstate - kRing) >> 3 << 3;
                }
                else
                {
                    lc.tableReads++;
                    const DevBVH H = S.bvhs[B.idx];
                    node = __ldg(S.tables + H.tableBase + hash_slot(S, H, key));
                }
                jumped = true;
            }
        }
        if (done)
        {
            E.count[rid] = ncand;
            E.status[rid] = kTraversed;
            active = false;
        }
    }
}

template<bool kAny, bool kQ, bool kWalk>
__global__ void __launch_bounds__(kCollectThreads, 4) k_collect(DevScene S, RaysSoA rays, uint32_t n0,
                                                                const uint32_t* nDev, Eng E, int pass, int cache,
                                                                Counters* cnt)
{
    __shared__ uint32_t ring[kRing * kCollectThreads];
    LocalCounters lc;
    uint32_t nrays = 0;
    collect_rays<kAny, kQ, kWalk>(S, rays, E, pass, cache, PassSource<0>(E, pass, n0, nDev), ring, lc, nrays);
    flush_counters(cnt, lc, nrays);
}

// -------------------------------------------------------------- order --
// The lists of a closest-hit pass whose objects were collected on walk trees,
// into the reference traversal's order: one thread per ray, a segment (an
// object's patches) at a time.  What was collected on the reference tree is in
// order and stays.
//
// An insertion sort in place: segments are short (8.6 patches on a ray of the
// 1920x1080 torus frame that hits) and the walk meets them in nearly that order.
// Bound by the latency of the comparisons' loads (hash, node) and the lists'
// scattered lines: 300 us for 2,073,600 rays, held to 64 registers.  (Testing only
// the m - 1 nodes where neighbouring heap keys part and sorting by keys with those
// bits flipped has a third of the tests and took 372 us, its arrays in local memory.)
//
// A long segment is sorted by its warp instead: each patch gets a code with a
// bit per level of the reference tree, 1 where its path takes the child visited
// last, which orders as the traversal does.
constexpr int kOrderThreads = 128;
constexpr uint32_t kLongSegment = 24;

// Whether the reference traversal by the ray (ro, ri) visits the left child of
// the node with heap key `key` first.
__device__ __forceinline__ bool left_first(const DevScene& S, const DevBVH& H, uint32_t key, float3 ro, float3 ri)
{
    const uint32_t node = __ldg(S.tables + H.tableBase + hash_slot(S, H, key));
    const float4* q = S.nodes + 4ull * (H.nodeBase + node);
    float4 q0, q1, q2, q3;
    ldg256(q, q0, q1);
    ldg256(q + 2, q2, q3);
    float L0, R0;
    slab(L0, f3(q0.x, q0.y, q0.z), f3(q0.w, q1.x, q1.y), ro, ri);
    slab(R0, f3(q1.z, q1.w, q2.x), f3(q2.y, q2.z, q2.w), ro, ri);
    return L0 < R0;
}

// Whether leaf a (heap key) comes before leaf b in the reference traversal of
// BVH H by the ray (ro, ri), both of them met: at their lowest common
// ancestor the nearer child goes first, the right one on equal distances.
__device__ __forceinline__ bool visits_first(const DevScene& S, const DevBVH& H, uint32_t a, uint32_t b, float3 ro,
                                             float3 ri)
{
    const int da = __clz(a), db = __clz(b);  // the deeper key has fewer leading zeros
    if (da < db) a >>= db - da; else b >>= da - db;
    const int up = 32 - __clz(a ^ b);
    return left_first(S, H, a >> up, ro, ri) == (((a >> (up - 1)) & 1u) == 0u);
}

// The ray, BVH and keys of an entered object that has a walk tree.
struct OrderSegment
{
    float3 ro, ri;
    DevBVH H;
    const uint32_t* keys;
    __device__ __forceinline__ bool open(const DevScene& S, const RaysSoA& rays, uint32_t rid, uint32_t obj)
    {
        const DevObject& O = S.objects[obj];
        H = S.bvhs[O.surface];
        if (H.walkBase == EMPTY) return false;
        float3 o, d, ld;
        float tmax, lmax, sinv;
        load_ray(rays, rid, o, d, tmax);
        to_local(O, o, d, tmax, ro, ld, lmax, sinv);
        ri = f3(1.0f / ld.x, 1.0f / ld.y, 1.0f / ld.z);
        keys = S.leafKeys + __ldg(S.patchBase + O.surface);
        return true;
    }
};

// The long segments of one ray's list, by a whole warp.
__device__ __forceinline__ void order_long(const DevScene& S, const RaysSoA& rays, uint2* list, uint32_t rid,
                                               uint32_t n)
{
    const uint32_t lane = lane_id();
    for (uint32_t k = 0; k + kLongSegment < n; k++)
    {
        if (list[k].x != kEnter) continue;
        uint32_t end = k + 1;
        while (end < n && list[end].x < kCont) end++;
        OrderSegment G;
        const uint32_t size = end - (k + 1);
        if (size > kLongSegment && G.open(S, rays, rid, list[k].y))
        {
            // ranks by counting smaller codes; up to kLongList entries, 8 a lane
            uint2 e[kLongList / 32];
            uint32_t code[kLongList / 32], rank[kLongList / 32];
#pragma unroll
            for (uint32_t c = 0; c < kLongList / 32; c++)
            {
                const uint32_t at = c * 32 + lane;
                rank[c] = 0;
                code[c] = 0xFFFFFFFFu;
                if (at >= size) continue;
                e[c] = list[k + 1 + at];
                const uint32_t key = __ldg(G.keys + e[c].x);
                const int depth = 31 - __clz(key);
                code[c] = 0;
                for (int l = 0; l < depth; l++)
                {
                    const uint32_t child = key >> (depth - 1 - l);
                    if (left_first(S, G.H, child >> 1, G.ro, G.ri) != ((child & 1u) == 0u)) code[c] |= 0x80000000u >> l;
                }
            }
#pragma unroll
            for (uint32_t c = 0; c < kLongList / 32; c++)
            {
                if (c * 32 >= size) break;
                const uint32_t there = min(32u, size - c * 32);
                for (uint32_t l = 0; l < there; l++)
                {
                    const uint32_t other = __shfl_sync(0xFFFFFFFFu, code[c], int(l));
#pragma unroll
                    for (uint32_t x = 0; x < kLongList / 32; x++) rank[x] += other < code[x] ? 1u : 0u;
                }
            }
            __syncwarp();
#pragma unroll
            for (uint32_t c = 0; c < kLongList / 32; c++)
                if (c * 32 + lane < size) list[k + 1 + rank[c]] = e[c];
            __syncwarp();
        }
        k = end - 1;
    }
}

// Orders one ray's segments; true if it has a long one, which is left.
__device__ __forceinline__ bool order_ray(const DevScene& S, const RaysSoA& rays, const Eng& E, uint32_t rid, uint32_t count)
{
    bool longer = false;
    if (count <= 3) return false;
    uint2* list = E.list_of(rid);
    for (uint32_t k = 0; k + 2 < count; k++)
    {
        if (list[k].x != kEnter) continue;
        // the segment is list[k + 1 .. end): to the object's leave marker or the list's end
        if (list[k + 1].x >= kCont || list[k + 2].x >= kCont) continue;
        OrderSegment G;
        if (!G.open(S, rays, rid, list[k].y)) continue;
        uint32_t j = k + 2;
        for (; j < count && list[j].x < kCont; j++)
        {
            if (j > k + kLongSegment) { longer = true; break; }
            const uint2 e = list[j];
            const uint32_t ke = __ldg(G.keys + e.x);
            uint32_t at = j;
            for (; at > k + 1; at--)
            {
                const uint2 p = list[at - 1];
                if (visits_first(S, G.H, __ldg(G.keys + p.x), ke, G.ro, G.ri)) break;
                list[at] = p;
            }
            if (at != j) list[at] = e;
        }
        k = j - 1;
    }
    return longer;
}
__global__ void __launch_bounds__(kOrderThreads) k_order(DevScene S, RaysSoA rays, uint32_t n0, const uint32_t* nDev,
                                                         Eng E, int pass)
{
    const PassSource<0> src(E, pass, n0, nDev);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < src.m; i += gridDim.x * blockDim.x)
    {
        const uint32_t rid = src.ray(i);
        // the rays left to k_order_long: in the queue that the next k_pending fills
        if (order_ray(S, rays, E, rid, E.count[rid])) E.queue[(pass + 1) & 1][atomicAdd(E.ctl + 4 * pass + 3, 1u)] = rid;
    }
}
// Orders a source's rays 32 at a time, all of their segments, by one warp of several (warp w of nw).
template<class Source>
__device__ __forceinline__ void order_rays(const DevScene& S, const RaysSoA& rays, const Eng& E, const Source& src,
                                           uint32_t w, uint32_t nw)
{
    const uint32_t lane = lane_id();
    for (uint32_t i0 = 32 * w; i0 < src.m; i0 += 32 * nw)
    {
        const uint32_t rid = i0 + lane < src.m ? src.ray(i0 + lane) : 0u;
        const uint32_t count = i0 + lane < src.m ? E.count[rid] : 0u;
        const bool longer = order_ray(S, rays, E, rid, count);
        for (unsigned b = __ballot_sync(0xFFFFFFFFu, longer); b; b &= b - 1)
        {
            const int owner = __ffs(b) - 1;
            const uint32_t r = __shfl_sync(0xFFFFFFFFu, rid, owner), n = __shfl_sync(0xFFFFFFFFu, count, owner);
            __syncwarp();
            order_long(S, rays, E.list_of(r), r, n);
        }
    }
}
// A later pass's rays: few, so in one launch.
__global__ void __launch_bounds__(kOrderThreads) k_order_queue(DevScene S, RaysSoA rays, Eng E, int pass)
{
    order_rays(S, rays, E, PassSource<0>(E, pass, 0, nullptr), (blockIdx.x * blockDim.x + threadIdx.x) / 32,
               gridDim.x * blockDim.x / 32);
}
// The first pass's rays with long segments, a warp each: a kernel of its own, so
// that its registers are not k_order's.
__global__ void __launch_bounds__(kOrderThreads) k_order_long(DevScene S, RaysSoA rays, Eng E, int pass)
{
    const uint32_t m = E.ctl[4 * pass + 3], nw = gridDim.x * blockDim.x / 32;
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) / 32; i < m; i += nw)
    {
        const uint32_t rid = E.queue[(pass + 1) & 1][i];
        order_long(S, rays, E.list_of(rid), rid, E.count[rid]);
    }
}

// ------------------------------------------------------------ resolve --
// The tail of a launch is a few long searches.  A lane left without rays takes
// the bottom (largest) pending interval of a search in its warp that holds
// one or more, and searches it as that search would after popping it: the same
// sub-net, derived from the projected net, and the same cut side.  The
// intervals searched are the same, so the roots found are.  A closest-hit search
// needs the nearest, and of roots at the same distance the first in the search's
// order, so each lane of it keeps a range of order numbers: a lender keeps the
// lower half of its own (what it lends comes last) and the borrower merges its
// root under the first of its range.  The lane that has the ray, the owner, waits
// for its borrowers at the end of the patch's search; an any-hit subdivision, which
// needs one root of any patch, at the end of the ray's list.
//
// A search's limits (iterations, stack entries) hold for the whole of it, in its
// order: the owner adds up the iterations of the parts, and where they pass the
// limit, or where the stack would have held nearly all that fit, it drops what
// the parts found and searches again alone, up to the limit: the patch, or the
// ray's list for any hit.  So no answer depends on which lanes were idle.  (With a
// limit for each lane's part a search that reaches it gave what its warp's idle
// lanes made of it.)
//
// An any-hit clipping search waits for nobody: whichever lane finds a root marks
// the ray occluded (writes of "occluded" never clear it), and each part has the
// limits to itself.  (Waiting: 640,001 shadow rays 1.75 ms for 1.55, a batch of
// renders 6.5 ms for 4.3.)
//
// One warp's lanes that lend or borrow.  (Packed: the L1 cache has what the
// blocks' shared memory leaves, and the searches' stacks live there.)
template<bool kAny> struct Lend
{
    uint32_t sum[32];   // owner: lanes searching for it (bits 0-7), kFound, kOverLimit, iterations of ended parts
    uint32_t who[32];   // a lane's owner (bits 0-7) and the log2 of its range of order numbers
    uint32_t lo[32];    // the range's first
    uint32_t rank[32];  // owner: the order number of the best root merged so far, EMPTY: none
    float t[32], u[32], v[32];  // and the root
};
template<> struct Lend<true> { uint32_t sum[32], who[32]; };
// The stack of a search in parts: one entry more would push a cut side's bit out of its word.
constexpr int kPartsStack = 31;
// kOverLimit: the search's parts together are past the limit, the others are to end.
constexpr uint32_t kKids = 0xFFu, kFound = 0x100u, kOverLimit = 0x200u, kSpentShift = 10;
// What a lane searches: a ray's patch of its own, a patch again and alone, a patch
// with intervals lent (the owner), or an interval borrowed.
enum Role : int { kOwn, kAlone, kLent, kThief };
// Where an owner is.
enum LendEnd { kUnended, kEndedNothing, kEndedRoot, kEndedAgain };
__device__ __forceinline__ bool in_parts(int role) { return role >= kLent; }

// Adds a lane's root to its owner's: the nearest is kept, the first in the
// search's order at equal distances.
__device__ __forceinline__ void lend_merge(Lend<false>& L, uint32_t o, uint32_t rank, const HitSink& sink)
{
    if (L.rank[o] == EMPTY || sink.dist < L.t[o] || (sink.dist == L.t[o] && rank < L.rank[o]))
    {
        L.t[o] = sink.dist; L.u[o] = sink.uv.x; L.v[o] = sink.uv.y; L.rank[o] = rank;
    }
}

// Pairs idle lanes with lanes that have an interval to lend.  src: the lane a
// borrower takes from.
__device__ __forceinline__ void lend_pairs(unsigned idleM, unsigned richM, bool& borrows, bool& lends, int& src)
{
    const unsigned lane = lane_id(), below = (1u << lane) - 1u;
    const int pairs = min(__popc(idleM), __popc(richM));
    const int idleRank = __popc(idleM & below), richRank = __popc(richM & below);
    borrows = ((idleM >> lane) & 1u) && idleRank < pairs;
    lends = ((richM >> lane) & 1u) && richRank < pairs;
    src = borrows ? int(__fns(richM, 0, idleRank + 1)) : int(lane);
}

// Whether a lane of this role may lend once more.
template<bool kAny> __device__ __forceinline__ bool lend_may(const Lend<kAny>& L, int role)
{
    if constexpr (kAny) return role != kAlone;
    else return role == kOwn || (in_parts(role) && (L.who[lane_id()] >> 8) != 0u);
}
// The lender's side of a loan, before its borrower reads the lender's entries.
template<bool kAny> __device__ __forceinline__ void lend_give(Lend<kAny>& L, int& role)
{
    const uint32_t lane = lane_id();
    if (role == kOwn)
    {
        L.sum[lane] = 0;
        L.who[lane] = lane | (31u << 8);
        if constexpr (!kAny) { L.lo[lane] = 0; L.rank[lane] = EMPTY; }
        role = kLent;
    }
    atomicAdd(&L.sum[L.who[lane] & 0xFFu], 1u);
}
// The borrower's: the upper half of the lender's order range.
template<bool kAny> __device__ __forceinline__ void lend_take(Lend<kAny>& L, int src, int& role)
{
    const uint32_t lane = lane_id(), who = L.who[src] - (kAny ? 0u : 1u << 8);
    L.who[lane] = who;
    if constexpr (!kAny)
    {
        L.who[src] = who;
        L.lo[lane] = L.lo[src] + (1u << (who >> 8));
    }
    role = kThief;
}

// A borrower's ray and patch, from lane src (called by the whole warp).
__device__ __forceinline__ void lend_ray(bool borrows, int src, HitSink& sink)
{
    const unsigned long long sp =
        __shfl_sync(0xFFFFFFFFu, (unsigned long long)reinterpret_cast<uintptr_t>(sink.P), src);
    const float3 so = f3(__shfl_sync(0xFFFFFFFFu, sink.o.x, src), __shfl_sync(0xFFFFFFFFu, sink.o.y, src),
                         __shfl_sync(0xFFFFFFFFu, sink.o.z, src));
    const float3 sd = f3(__shfl_sync(0xFFFFFFFFu, sink.d.x, src), __shfl_sync(0xFFFFFFFFu, sink.d.y, src),
                         __shfl_sync(0xFFFFFFFFu, sink.d.z, src));
    const float sdist = __shfl_sync(0xFFFFFFFFu, sink.dist, src);
    if (!borrows) return;
    sink.P = reinterpret_cast<const float4*>(uintptr_t(sp));
    sink.o = so; sink.d = sd; sink.dist = sdist; sink.uv = make_float2(0.0f, 0.0f);
}

// One lane's ray: where it is in its list, and the best hit so far.  Shared by
// the two search kernels below.
template<bool kAny> struct ListWalk
{
    uint32_t rid = 0, k = 0, count = 0, patch = 0;
    int32_t obj = -1, lpatch = -1;
    // any hit with E.originLast: sweep 0 searches the candidates whose leaf box
    // holds the ray's origin (entry <= 0) not, sweep 1 only those
    bool sweep = false;
    float3 o = f3(0, 0, 0), d = f3(0, 0, 1);
    float tmax = 0, lmax = 0, sinv = 1, lt = 0, lu = 0, lv = 0, limit = 0;
    const uint2* list = nullptr;

    // Takes ray r; false if it has nothing to search.
    __device__ __forceinline__ bool take(const RaysSoA& rays, const Eng& E, int pass, uint32_t r, LocalCounters&)
    {
        const uint32_t st = E.status[r];
        count = E.count[r];
        if (count == 0 || st == kFinished) return false;
        rid = r;
        k = 0;
        obj = -1;
        sweep = false;
        load_ray(rays, rid, o, d, tmax);
        limit = kAny ? tmax : (pass == 0 ? tmax : E.limit[rid]);
        list = E.list_of(rid);
        return true;
    }

    // Walks the list -- object markers, patches culled by their leaf entry --
    // to the next patch to search (true, with `sink` set up for it) or the end
    // of the chunk (false).
    __device__ __forceinline__ bool next(const DevScene& S, const Eng& E, HitsSoA& hits, HitSink& sink)
    {
        for (;;)
        {
            if (kAny && k >= count && E.originLast && !sweep)
            {
                sweep = true;  // the candidates whose leaf box holds the origin, last
                k = 0;
                obj = -1;
                continue;
            }
            if (k >= count)
            {
                // end of this pass's chunk: keep what the next pass needs
                if (!kAny)
                {
                    E.limit[rid] = limit;
                    if (obj >= 0) { E.lt[rid] = lt; E.lu[rid] = lu; E.lv[rid] = lv; E.lpatch[rid] = lpatch; }
                }
                return false;
            }
            const uint2 e = list[k++];
            if (e.x == kEnter || e.x == kCont)
            {
                obj = int32_t(e.y);
                float3 ld;
                to_local(S.objects[obj], o, d, tmax, sink.o, ld, lmax, sinv);
                sink.d = ld;
                if (e.x == kEnter || kAny) { lt = lmax; lpatch = -1; lu = 0.0f; lv = 0.0f; }
                else { lt = E.lt[rid]; lu = E.lu[rid]; lv = E.lv[rid]; lpatch = E.lpatch[rid]; }
            }
            else if (e.x == kLeave)
            {
                if (!kAny && lpatch >= 0)
                {
                    const float t = lt * sinv;
                    if (t < limit)
                    {
                        limit = t;
                        hits.t[rid] = t; hits.u[rid] = lu; hits.v[rid] = lv;
                        hits.patch[rid] = lpatch; hits.object[rid] = obj;
                    }
                }
                obj = -1;
            }
            else
            {
                patch = e.x;
                const float entry = __uint_as_float(e.y);
                const bool turn = !kAny || !E.originLast || ((entry <= 0.0f) == sweep);
                if (turn && entry < (kAny ? lmax : lt))
                {
                    const uint32_t surface = S.objects[obj].surface;
                    sink.P = S.patches + 16ull * (__ldg(S.patchBase + surface) + patch);
                    sink.dist = kAny ? lmax : lt;
                    sink.uv = kAny ? make_float2(0.0f, 0.0f) : make_float2(lu, lv);
                    return true;
                }
            }
        }
    }

    // The search of the patch ended with a (closer) root.
    __device__ __forceinline__ void keep(float t, float u, float v) { lt = t; lu = u; lv = v; lpatch = int32_t(patch); }
    __device__ __forceinline__ void occlude(const Eng& E, int32_t* occluded) const
    {
        occluded[rid] = 0;
        E.status[rid] = kFinished;
        E.count[rid] = 0;
    }
    // Any hit: where the ray's borrowers have ended (true), the ray is over or starts its list again.
    __device__ __forceinline__ bool settle(const Eng& E, int32_t* occluded, LendEnd end, bool& have)
    {
        if (end == kUnended) return false;
        if (end == kEndedAgain)
        {
            k = 0;
            obj = -1;
            sweep = false;
            return true;
        }
        have = false;
        if (end == kEndedRoot) occlude(E, occluded);
        else finish(E);
        return true;
    }
    // Closest hit: the sink as next() left it; the patch is to be searched again.
    __device__ __forceinline__ void again(const HitsSoA&, HitSink& sink) const
    {
        sink.dist = lt;
        sink.uv = make_float2(lu, lv);
    }
    // The end of the ray's list.
    __device__ __forceinline__ void finish(const Eng& E) { E.count[rid] = 0; }
};

// One lane's explicit (ray, patch) pair, in place of a ray with its list.
struct PairWalk
{
    uint32_t surface, patches;
    const uint32_t* pids;
    uint32_t rid = 0, patch = 0;
    int32_t obj = -1, lpatch = -1;
    bool searched = false;
    float3 o = f3(0, 0, 0), d = f3(0, 0, 1);
    float lt = 0, lu = 0, lv = 0;

    __device__ __forceinline__ bool take(const RaysSoA& rays, const Eng&, int, uint32_t r, LocalCounters&)
    {
        rid = r;
        patch = __ldg(pids + r);
        searched = false;
        lpatch = -1;
        o = f3(__ldg(rays.ox + r), __ldg(rays.oy + r), __ldg(rays.oz + r));
        d = f3(__ldg(rays.dx + r), __ldg(rays.dy + r), __ldg(rays.dz + r));
        return true;
    }
    __device__ __forceinline__ bool next(const DevScene& S, const Eng&, HitsSoA& hits, HitSink& sink)
    {
        if (!searched && patch < patches)
        {
            searched = true;
            sink = HitSink {S.patches + 16ull * (__ldg(S.patchBase + surface) + patch), o, d, hits.t[rid],
                            make_float2(0.0f, 0.0f)};
            return true;
        }
        if (lpatch >= 0) { hits.t[rid] = lt; hits.u[rid] = lu; hits.v[rid] = lv; }
        hits.patch[rid] = lpatch >= 0 ? 1 : 0;
        return false;
    }
    __device__ __forceinline__ void keep(float t, float u, float v) { lt = t; lu = u; lv = v; lpatch = int32_t(patch); }
    __device__ __forceinline__ void again(const HitsSoA& hits, HitSink& sink) const
    {
        sink.dist = hits.t[rid];
        sink.uv = make_float2(0.0f, 0.0f);
    }
    __device__ __forceinline__ void finish(const Eng&) {}
};

// The clipping searches.  A lane takes a ray, walks its list and searches its
// patches; a search is made of the parts of clip_patch's loop.  The lanes of a
// warp are in different parts most of the time, and a loop that ran every part
// each time round for the lanes that are in it used 8 of 32 threads per
// instruction (4.8 in the FP64 instance).  So each time round the warp runs
// only the part that most of its lanes wait for (the projections and cuts in
// FP64 count as parts of their own); the others wait until theirs gathers
// more.  A lane's sequence of parts, and with it every result, does not depend on that.
// 640,001 shadow rays of the 16,384-patch torus: 1.46 ms, 2.02 ms with all
// parts each time round; 301,111 scattered rays 1.13 ms, before 1.29 ms.
//
// kG64: the search may take the FP64 grazing path (precision levels 3 and 5);
// the other levels run an instance without that code.  The FP32 instances are
// held to 128 registers, four 128-thread blocks per SM.
enum : int { kPartWalk, kPartProject, kPartCut, kPartRoot, kPartBegin64, kPartCut64, kPartMerge, kPartWait, kPartNone };

// What the two search kernels share besides their searches: the ends of searches
// in parts.  `it` is the iterations of a lane's part, above `limit` where it ended
// at one of the search's limits.
// Closest hits: lanes with their part at its end (kPartMerge); the owner's
// patch ends with the last.  Called by the whole warp.
__device__ __forceinline__ LendEnd lend_settle(Lend<false>& L, int& part, int& role, const HitSink& sink, bool found,
                                               uint32_t it, uint32_t limit)
{
    const uint32_t lane = lane_id();
    unsigned m = __ballot_sync(0xFFFFFFFFu, part == kPartMerge);
    while (m)
    {
        for (; m; m &= m - 1)
        {
            if (lane == uint32_t(__ffs(m) - 1))
            {
                const uint32_t o = L.who[lane] & 0xFFu;
                uint32_t sum = L.sum[o] - (role == kThief ? 1u : 0u);
                if (!(sum & kOverLimit))
                {
                    sum += it << kSpentShift;
                    if ((sum >> kSpentShift) > limit) sum |= kOverLimit;
                    if (found) lend_merge(L, o, L.lo[lane], sink);
                }
                L.sum[o] = sum;
                part = role == kThief ? kPartNone : kPartWait;
                if (role == kThief) role = kOwn;
            }
            __syncwarp();
        }
        // the other parts of a search that is past its limit end here
        if (in_parts(role) && part >= kPartProject && part <= kPartRoot && (L.sum[L.who[lane] & 0xFFu] & kOverLimit))
            part = kPartMerge;
        m = __ballot_sync(0xFFFFFFFFu, part == kPartMerge);
    }
    LendEnd end = kUnended;
    if (part == kPartWait && (L.sum[lane] & kKids) == 0)
    {
        end = L.sum[lane] & kOverLimit ? kEndedAgain : L.rank[lane] != EMPTY ? kEndedRoot : kEndedNothing;
        role = kOwn;
        part = kPartWalk;
    }
    __syncwarp();
    return end;
}
// Any hit: a lane's part has ended.
__device__ __forceinline__ void lend_end_part(Lend<true>& L, int& part, int& role, bool found, uint32_t it, uint32_t limit)
{
    uint32_t* sum = &L.sum[L.who[lane_id()] & 0xFFu];
    // (an owner's searches after its first loan are counted together; past the limit the sum stands)
    if ((*(volatile uint32_t*)sum >> kSpentShift) <= limit) atomicAdd(sum, it << kSpentShift);
    if (found) atomicOr(sum, kFound);
    if (role == kThief)
    {
        atomicSub(sum, 1u);
        role = kOwn;
        part = kPartNone;
    }
    else part = found ? kPartWait : kPartWalk;
}
// Any hit: an owner at the end of its list looks whether its borrowers are.
__device__ __forceinline__ LendEnd lend_wait(const Lend<true>& L, int& role, uint32_t limit)
{
    const uint32_t sum = *(const volatile uint32_t*)&L.sum[lane_id()];
    if (sum & kKids) return kUnended;
    if ((sum >> kSpentShift) > limit)
    {
        role = kAlone;
        return kEndedAgain;
    }
    role = kOwn;
    return sum & kFound ? kEndedRoot : kEndedNothing;
}

template<bool kAny, bool kG64, class Source, class Walk>
__device__ __forceinline__ void clip_rays(const DevScene& S, const RaysSoA& rays, const Eng& E, int pass, const Query& q,
                                          HitsSoA& hits, int32_t* occluded, const Source& src, Lend<kAny>& L,
                                          LocalCounters& lc, Walk w)
{
    float4 stack[kClipStack];
    volatile float net0[32];  // kG64: a near-grazing search's projected net
    ClipState c;
    c.b64 = false;
    c.sl = 0;
    c.base = 0;
    HitSink sink {nullptr, f3(0, 0, 0), f3(0, 0, 1), 0.0f, make_float2(0, 0)};
    int part = kPartWalk;
    bool have = false;   // the lane has a ray
    int role = kOwn;
    const float tol2 = below_sqrt(q.tol), tol2graze = kG64 ? below_sqrt(kGrazeTol) : 0.0f;
    const uint32_t m = src.m;
    for (;;)
    {
        if constexpr (!kG64)
        {
            // lanes in none of the searches' parts: one vote while there are none
            const unsigned resting = __ballot_sync(0xFFFFFFFFu, part >= kPartMerge);
            if constexpr (!kAny)
            {
                if (resting && __ballot_sync(0xFFFFFFFFu, part == kPartMerge || part == kPartWait))
                {
                    const LendEnd end = lend_settle(L, part, role, sink, c.found, uint32_t(c.it), kMaxClipIterations);
                    if (end == kEndedRoot) w.keep(L.t[lane_id()], L.u[lane_id()], L.v[lane_id()]);
                    if (end == kEndedAgain)
                    {
                        w.again(hits, sink);
                        clip_begin<kG64>(c, sink, q.tol, 0.0f);
                        part = kPartProject;
                        role = kAlone;
                    }
                }
            }
            const unsigned idleM = resting ? __ballot_sync(0xFFFFFFFFu, part == kPartNone) : 0u;
            if (idleM)
            {
                const bool rich = part >= kPartProject && part <= kPartRoot && c.sl > c.base && c.sl < kPartsStack &&
                                  (kAny || lend_may(L, role));
                const unsigned richM = __ballot_sync(0xFFFFFFFFu, rich);
                if (richM)
                {
                    bool borrows, lends;
                    int src;
                    lend_pairs(idleM, richM, borrows, lends, src);
                    float4 e = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    int bit = 0;
                    if (lends)
                    {
                        // entry i's cut side is bit (sl - i) of the bit stack
                        e = stack[c.base];
                        bit = (c.cutsideStack >> (c.sl - c.base)) & 1;
                        if constexpr (!kAny) lend_give(L, role);
                    }
                    const int base = c.base;
                    if (lends) c.base++;
                    __syncwarp();
                    const float4 se =
                        make_float4(__shfl_sync(0xFFFFFFFFu, e.x, src), __shfl_sync(0xFFFFFFFFu, e.y, src),
                                    __shfl_sync(0xFFFFFFFFu, e.z, src), __shfl_sync(0xFFFFFFFFu, e.w, src));
                    const int sbit = __shfl_sync(0xFFFFFFFFu, bit, src), sbase = __shfl_sync(0xFFFFFFFFu, base, src);
                    lend_ray(borrows, src, sink);
                    if constexpr (kAny)
                    {
                        const uint32_t rid = __shfl_sync(0xFFFFFFFFu, w.rid, src);
                        if (borrows) { w.rid = rid; role = kThief; }
                    }
                    if (borrows)
                    {
                        if constexpr (!kAny) lend_take(L, src, role);
                        c.emin = make_float2(se.x, se.y);
                        c.emax = make_float2(se.z, se.w);
                        c.cutsideStack = sbit; c.sl = sbase; c.base = sbase; c.it = 0; c.tol = q.tol;
                        c.found = false; c.b64 = false; c.fresh = false; c.tposed = false;
                        part = kPartProject;
                    }
                    __syncwarp();
                }
            }
        }
        // the part that most lanes wait for
        int run = kPartNone;
        int most = 0;
#pragma unroll
        for (int p = kPartWalk; p <= (kG64 ? kPartCut64 : kPartRoot); p++)
        {
            const int lanes = __popc(__ballot_sync(0xFFFFFFFFu, part == p));
            if (lanes > most) { most = lanes; run = p; }
        }
        if (run == kPartNone) break;
        if (run == kPartWalk)
        {
            const bool need = part == kPartWalk && !have;
            const uint32_t idx = warp_fetch(src.fetch(), need);
            if (need)
            {
                if (idx < m) have = w.take(rays, E, pass, src.ray(idx), lc);
                else part = kPartNone;
            }
            if (part == kPartWalk && have)
            {
                if (w.next(S, E, hits, sink))
                {
                    lc.candidates++;
                    clip_begin<kG64>(c, sink, q.tol, graze_sin(q.precision));
                    if (!kG64 && !kAny) role = kOwn;
                    part = kG64 && c.b64 ? kPartBegin64 : kPartProject;
                }
                else
                {
                    have = false;
                    w.finish(E);
                }
            }
            continue;
        }
        if (part != run) continue;
        ClipNext next;
        if (run == kPartRoot) next = clip_root(c, stack, sink);
        else
        {
            if (kG64 && run == kPartBegin64)
            {
                clip_begin64(c, sink, net0, &S.objects[w.obj], w.o, w.d);
                next = kClipCut;
            }
            else if (run == kPartProject)
            {
                clip_project<kG64>(c, sink, net0);
                next = kClipCut;
            }
            else
                next = clip_cut<kG64>(c, stack, !kG64 && !kAny && in_parts(role) ? kPartsStack : kClipStack);
            if (next == kClipCut) next = clip_test<kG64>(c, kG64 && c.b64 ? tol2graze : tol2, lc);
        }
        if (kAny && c.found) next = kClipOver;  // an any-hit search ends at its first root
        if (next < kClipOver)
        {
            part = next == kClipRoot ? kPartRoot
                   : next == kClipProject ? kPartProject : kG64 && c.b64 ? kPartCut64 : kPartCut;
            continue;
        }
        if (!kG64 && !kAny && in_parts(role))
        {
            // (a limit's error is raised by the search that runs to it alone)
            if (next == kClipFull) c.it = kMaxClipIterations + 1;
            part = kPartMerge;
            continue;
        }
        part = kPartWalk;
        lc.errors |= limit_error(next);
        if constexpr (kAny)
        {
            if (c.found) { w.occlude(E, occluded); have = false; }
            if (role == kThief) { role = kOwn; part = kPartNone; }
        }
        else if (c.found) w.keep(sink.dist, sink.uv.x, sink.uv.y);
    }
}

template<bool kAny, bool kG64>
__global__ void __launch_bounds__(kResolveThreads, kG64 ? 3 : 4) k_clip(DevScene S, RaysSoA rays, uint32_t n0,
                                                                         const uint32_t* nDev, Eng E, int pass, Query q,
                                                                         HitsSoA hits, int32_t* occluded, Counters* cnt)
{
    __shared__ Lend<kAny> lend[kAny || kG64 ? 1 : kResolveThreads / 32];
    LocalCounters lc;
    clip_rays<kAny, kG64>(S, rays, E, pass, q, hits, occluded, PassSource<1>(E, pass, n0, nDev),
                          lend[kAny || kG64 ? 0 : threadIdx.x / 32], lc, ListWalk<kAny> {});
    flush_counters(cnt, lc, 0);
}

// The subdivision method's searches (at the precision form's levels too: it
// has no FP64 bounds), part by part and with lent intervals as in k_clip.  A
// lane runs E.subdivLevels bisections each time round that the bisections run.
// The pending intervals of this search are the upper halves that its bit trail
// has not reached; the first (largest) one is at the trail's first 0 bit.
// 131,101 rays on a 2,048-patch torus, the longest of 3,429 bisections: 0.91 ms
// a query, 1.81 ms with every part each time round and no lending.
template<bool kAny, class Source, class Walk>
__device__ __forceinline__ void subdivide_rays(const DevScene& S, const RaysSoA& rays, const Eng& E, int pass,
                                               const Query& q, HitsSoA& hits, int32_t* occluded, const Source& src,
                                               Lend<kAny>& L, LocalCounters& lc, Walk w)
{
    ClipState c;
    HitSink sink {nullptr, f3(0, 0, 0), f3(0, 0, 1), 0.0f, make_float2(0, 0)};
    int part = kPartWalk;
    bool have = false;
    int role = kOwn;
    const float tol2 = below_sqrt(q.tol);
    c.sl = 0;
    c.found = false;
    const uint32_t m = src.m;
    for (;;)
    {
        const unsigned resting = __ballot_sync(0xFFFFFFFFu, part >= kPartMerge);
        if constexpr (kAny)
        {
            if (part == kPartWait && w.settle(E, occluded, lend_wait(L, role, kMaxBisections), have))
                part = kPartWalk;
        }
        else if (resting && __ballot_sync(0xFFFFFFFFu, part == kPartMerge || part == kPartWait))
        {
            const LendEnd end = lend_settle(L, part, role, sink, c.found, uint32_t(c.it), kMaxBisections);
            if (end == kEndedRoot) w.keep(L.t[lane_id()], L.u[lane_id()], L.v[lane_id()]);
            if (end == kEndedAgain)
            {
                w.again(hits, sink);
                subdiv_begin(c);
                part = kPartProject;
                role = kAlone;
            }
        }
        const unsigned idleM = resting ? __ballot_sync(0xFFFFFFFFu, part == kPartNone) : 0u;
        if (idleM)
        {
            // level j's bit of the trail is bit k - 1 - j: the first level with a 0 bit
            const uint32_t trail = uint32_t(c.cutsideStack);
            const int k = c.sl, j = k > 0 ? __clz(~(trail << (32 - k))) : 0;
            const bool rich = part >= kPartProject && part <= kPartRoot && j < k && lend_may(L, role);
            const unsigned richM = __ballot_sync(0xFFFFFFFFu, rich);
            if (richM)
            {
                bool borrows, lends;
                int src;
                lend_pairs(idleM, richM, borrows, lends, src);
                uint32_t tu = __float_as_uint(c.emin.x), tv = __float_as_uint(c.emin.y);
                int level = 0;
                if (lends)
                {
                    // the path down to level j, with the upper half there: even levels cut u
                    tu = (tu >> ((k + 1) / 2 - (j + 2) / 2)) | (j % 2 == 0 ? 1u : 0u);
                    tv = (tv >> (k / 2 - (j + 1) / 2)) | (j % 2 == 0 ? 0u : 1u);
                    level = j + 1;
                    c.cutsideStack = int(trail | (1u << (k - 1 - j)));
                    lend_give(L, role);
                }
                __syncwarp();
                const uint32_t su = __shfl_sync(0xFFFFFFFFu, tu, src), sv = __shfl_sync(0xFFFFFFFFu, tv, src);
                const int sk = __shfl_sync(0xFFFFFFFFu, level, src);
                lend_ray(borrows, src, sink);
                if (borrows)
                {
                    lend_take(L, src, role);
                    // every level above is done here: the trail is all ones
                    c.cutsideStack = int(sk < 32 ? (1u << sk) - 1u : 0xFFFFFFFFu);
                    c.sl = sk; c.it = 0; c.fresh = true; c.found = false;
                    c.emin = make_float2(__uint_as_float(su), __uint_as_float(sv));
                    part = kPartProject;
                }
                __syncwarp();
            }
        }
        int run = kPartNone;
        int most = 0;
#pragma unroll
        for (int p = kPartWalk; p <= kPartRoot; p++)
        {
            const int lanes = __popc(__ballot_sync(0xFFFFFFFFu, part == p));
            if (lanes > most) { most = lanes; run = p; }
        }
        if (run == kPartNone) break;
        if (run == kPartWalk)
        {
            const bool need = part == kPartWalk && !have;
            const uint32_t idx = warp_fetch(src.fetch(), need);
            if (need)
            {
                if (idx < m) have = w.take(rays, E, pass, src.ray(idx), lc);
                else part = kPartNone;
                if (kAny) role = kOwn;
            }
            if (part == kPartWalk && have)
            {
                if (w.next(S, E, hits, sink))
                {
                    lc.candidates++;
                    subdiv_begin(c);
                    if (!kAny) role = kOwn;
                    part = kPartProject;
                }
                else if (kAny && role == kLent) part = kPartWait;
                else
                {
                    have = false;
                    w.finish(E);
                }
            }
            continue;
        }
        if (part != run) continue;
        ClipNext next;
        if (run == kPartRoot) next = subdiv_root(c, sink);
        else if (run == kPartProject) { subdiv_project(c, sink); next = kClipCut; }
        else
        {
            next = kClipCut;
            const int levels = int(E.subdivLevels);
            for (int s = 0; s < levels; s++)
            {
                next = subdiv_cut(c, tol2, lc);
                if (next != kClipCut) break;
            }
        }
        if (kAny && c.found) next = kClipOver;  // an any-hit search ends at its first root
        if (next < kClipOver)
        {
            part = next == kClipRoot ? kPartRoot : next == kClipProject ? kPartProject : kPartCut;
            continue;
        }
        if (in_parts(role))
        {
            if constexpr (kAny) lend_end_part(L, part, role, c.found, uint32_t(c.it), kMaxBisections);
            else part = kPartMerge;
            continue;
        }
        part = kPartWalk;
        lc.errors |= limit_error(next);
        if (!c.found) continue;
        if constexpr (kAny) { w.occlude(E, occluded); have = false; }
        else w.keep(sink.dist, sink.uv.x, sink.uv.y);
    }
}

template<bool kAny>
__global__ void __launch_bounds__(kResolveThreads, 4) k_subdivide(DevScene S, RaysSoA rays, uint32_t n0,
                                                                  const uint32_t* nDev, Eng E, int pass, Query q,
                                                                  HitsSoA hits, int32_t* occluded, Counters* cnt)
{
    __shared__ Lend<kAny> lend[kResolveThreads / 32];
    LocalCounters lc;
    subdivide_rays<kAny>(S, rays, E, pass, q, hits, occluded, PassSource<1>(E, pass, n0, nDev),
                         lend[threadIdx.x / 32], lc, ListWalk<kAny> {});
    flush_counters(cnt, lc, 0);
}

// A ray unfinished after the last pass: the inline search from the start.
template<bool kAny>
__device__ __forceinline__ void rest_ray(const DevScene& S, const RaysSoA& rays, const Query& q, HitsSoA& hits,
                                         int32_t* occluded, uint32_t rid, LocalCounters& lc)
{
    float3 o, d; float tmax;
    load_ray(rays, rid, o, d, tmax);
    Query q32 = q;
    q32.precision = search_only(q.precision);  // the polish runs afterwards
    const uint32_t g = rays.group ? rays.group[rid] : 0u;
    if (g >= S.ngroups) return;
    if (kAny)
        occluded[rid] = scene_any(S, g, o, d, tmax, q32, lc) ? 0 : -1;
    else
    {
        HitRecord h {tmax, 0.0f, 0.0f, -1, -1};
        int ob = scene_closest(S, g, o, d, tmax, q32, h, lc);
        hits.t[rid] = ob >= 0 ? h.t : tmax; hits.u[rid] = h.u; hits.v[rid] = h.v;
        hits.patch[rid] = ob >= 0 ? h.patch : -1; hits.object[rid] = ob;
    }
}
template<bool kAny>
__global__ void __launch_bounds__(128) k_rest(DevScene S, RaysSoA rays, Eng E, int passes, Query q, HitsSoA hits,
                                              int32_t* occluded, Counters* cnt)
{
    // the rays still parked after the last pass
    const uint32_t m = E.ctl[4 * passes + 2];
    const uint32_t* queue = E.queue[passes & 1];
    LocalCounters lc;
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    for (uint32_t i = tid; i < m; i += nt)
    {
        const uint32_t rid = queue[i];
        if (E.status[rid] == kPending) rest_ray<kAny>(S, rays, q, hits, occluded, rid, lc);
    }
    flush_counters(cnt, lc, 0);
}

// The queue of parked rays for the next pass, in ray order within each tile
// of 256 rays (the tiles' slices land in the order their blocks claim them),
// so that a packet of consecutive queue positions holds neighbouring rays.
constexpr int kPendingThreads = 256;
__global__ void __launch_bounds__(kPendingThreads) k_pending(const uint32_t* __restrict__ status, uint32_t n0,
                                                             const uint32_t* nDev, uint32_t* queue, uint32_t* len)
{
    const uint32_t n = nDev ? *nDev : n0;
    __shared__ uint32_t offset[kPendingThreads / 32];
    __shared__ uint32_t base;
    const uint32_t w = threadIdx.x / 32, lane = threadIdx.x % 32;
    for (uint32_t t0 = blockIdx.x * kPendingThreads; t0 < n; t0 += gridDim.x * kPendingThreads)
    {
        const uint32_t i = t0 + threadIdx.x;
        const bool p = i < n && status[i] == kPending;
        const unsigned m = __ballot_sync(0xFFFFFFFFu, p);
        if (lane == 0) offset[w] = __popc(m);
        __syncthreads();
        if (threadIdx.x == 0)
        {
            uint32_t sum = 0;
            for (uint32_t k = 0; k < kPendingThreads / 32; k++)
            {
                const uint32_t c = offset[k];
                offset[k] = sum;
                sum += c;
            }
            base = sum ? atomicAdd(len, sum) : 0u;
        }
        __syncthreads();
        if (p) queue[base + offset[w] + __popc(m & ((1u << lane) - 1u))] = i;
        __syncthreads();
    }
}

__device__ __forceinline__ void init_ray(const RaysSoA& rays, HitsSoA& hits, int32_t* occluded, const Eng& E, uint32_t i)
{
    E.count[i] = 0;
    if (occluded) { occluded[i] = -1; return; }
    hits.t[i] = rays.tmax ? rays.tmax[i] : INFINITY;
    hits.u[i] = 0.0f; hits.v[i] = 0.0f; hits.patch[i] = -1; hits.object[i] = -1;
}
__global__ void k_init(RaysSoA rays, uint32_t n0, const uint32_t* nDev, HitsSoA hits, int32_t* occluded, Eng E)
{
    const uint32_t n = nDev ? *nDev : n0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        init_ray(rays, hits, occluded, E, i);
}

// One polish per hit.  The FP64 pipe takes a warp instruction whatever its
// active lanes, and a hit takes one to three mixed steps, a few up to ten full FP64
// ones, each as costly as all its mixed steps: so a warp gathers the hits of the
// rays it sweeps, refills its lanes from them and runs, as in k_clip, the part
// (start, mixed step, full step) that most of its lanes wait for.
// 582,000 hits of 2,073,600 rays: 520 us; 630 us with each batch of 32 hits
// run to the end of its slowest.
constexpr int kPolishThreads = 128;
constexpr uint32_t kPolishList = 64;
__device__ __forceinline__ void polish_rays(const DevScene& S, const RaysSoA& rays, HitsSoA& hits, uint32_t first,
                                            uint32_t end, uint32_t stride, uint32_t* list)
{
    constexpr int kIdle = -1, kStart = -2;  // else a PolishNext
    const uint32_t lane = threadIdx.x % 32, below = (1u << lane) - 1u;
    Polish p;
    double isc = 1.0;
    uint32_t rid = 0, cnt = 0, base = first;  // cnt: hits in the list, warp-uniform
    int part = kIdle;
    for (;;)
    {
        const unsigned idle = __ballot_sync(0xFFFFFFFFu, part == kIdle);
        while (cnt < uint32_t(__popc(idle)) && base < end)
        {
            const uint32_t i = base + lane;
            const bool hit = i < end && hits.object[i] >= 0;
            const unsigned m = __ballot_sync(0xFFFFFFFFu, hit);
            if (hit) list[cnt + __popc(m & below)] = i;
            cnt += __popc(m);
            base += stride;
            __syncwarp();
        }
        // lanes are refilled eight or more at a time, or when none is at work
        const uint32_t take = min(cnt, uint32_t(__popc(idle)));
        if (take >= 8 || (take && idle == 0xFFFFFFFFu))
        {
            if (part == kIdle && uint32_t(__popc(idle & below)) < take)
            {
                rid = list[cnt - 1 - __popc(idle & below)];
                part = kStart;
            }
            cnt -= take;
            __syncwarp();
        }
        const int starts = __popc(__ballot_sync(0xFFFFFFFFu, part == kStart)),
                  steps = __popc(__ballot_sync(0xFFFFFFFFu, part == kPolishStep)),
                  fulls = __popc(__ballot_sync(0xFFFFFFFFu, part == kPolishStep64));
        if (starts + steps + fulls == 0) break;
        if (starts >= steps && starts >= fulls)
        {
            if (part != kStart) continue;
            const HitRecord h {hits.t[rid], hits.u[rid], hits.v[rid], hits.patch[rid], hits.object[rid]};
            polish_start(S, f3(rays.ox[rid], rays.oy[rid], rays.oz[rid]), f3(rays.dx[rid], rays.dy[rid], rays.dz[rid]),
                         h, p, isc);
            part = kPolishStep;
        }
        // full steps wait for half a warp of them, or until nothing else is left
        else if (steps && (steps >= fulls || fulls < 16))
        {
            if (part == kPolishStep) part = polish_step(p);
        }
        else if (part == kPolishStep64)
            part = polish_step64(p);
        if (part == kPolishDone || part == kPolishFailed)
        {
            if (part == kPolishDone && polish_accepted(p))
            {
                hits.t[rid] = narrow(p.T * isc); hits.u[rid] = narrow(p.U); hits.v[rid] = narrow(p.V);
            }
            part = kIdle;
        }
    }
}
__global__ void __launch_bounds__(kPolishThreads) k_polish(DevScene S, RaysSoA rays, uint32_t n0,
                                                           const uint32_t* nDev, HitsSoA hits)
{
    __shared__ uint32_t list[kPolishThreads / 32][kPolishList];
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) / 32, nwarps = gridDim.x * blockDim.x / 32;
    polish_rays(S, rays, hits, warp * 32, nDev ? *nDev : n0, nwarps * 32, list[threadIdx.x / 32]);
}

// ------------------------------------------------------ small queries --
// A whole query in one launch, for ray counts that leave no work to balance: a
// warp takes an even share of the rays through every step -- the passes'
// traversal, order and searches on counters and queues of its own, the inline
// fallback, the polish -- so nothing is shared between warps.  A launch costs the
// host about 6 us, and a query of separate kernels is 11 of them and two
// memsets.  Each ray goes through the same steps, with the same results.
template<bool kAny, bool kG64, bool kSub>
__global__ void __launch_bounds__(32, 8) k_small(DevScene S,
                                                              RaysSoA rays, uint32_t n0,
                                                              const uint32_t* nDev,
                                                              Eng E, int passes, int cache, Query q, HitsSoA hits,
                                                              int32_t* occluded, Counters* cnt)
{
    __shared__ uint32_t ring[kRing * 32], fetch;
    static_assert(kRing * 32 >= kPolishList);
    __shared__ Lend<kAny> lend;
    const uint32_t n = nDev ? *nDev : n0, lane = threadIdx.x;
    const uint32_t share = (n + gridDim.x - 1) / gridDim.x, base = blockIdx.x * share;
    if (base >= n) return;
    const uint32_t mine = min(share, n - base);
    LocalCounters lc;
    uint32_t nrays = 0;
    for (uint32_t i = lane; i < mine; i += 32) init_ray(rays, hits, kAny ? occluded : nullptr, E, base + i);
    WarpSource src {&fetch, mine, base, nullptr};
    for (int p = 0;; p++)
    {
        if (p > 0)
        {
            // the rays still parked, in ray order
            uint32_t* queue = E.queue[p & 1] + base;
            uint32_t m = 0;
            for (uint32_t i0 = 0; i0 < mine; i0 += 32)
            {
                const uint32_t r = base + i0 + lane;
                const bool parked = i0 + lane < mine && E.status[r] == kPending;
                const unsigned b = __ballot_sync(0xFFFFFFFFu, parked);
                if (parked) queue[m + __popc(b & ((1u << lane) - 1u))] = r;
                m += __popc(b);
            }
            src.m = m;
            src.queue = queue;
            if (m == 0) break;
        }
        __syncwarp();
        if (p == passes)
        {
            for (uint32_t i = lane; i < src.m; i += 32) rest_ray<kAny>(S, rays, q, hits, occluded, src.ray(i), lc);
            break;
        }
        if (lane == 0) fetch = 0;
        __syncwarp();
        collect_rays<kAny, false, true>(S, rays, E, p, cache, src, ring, lc, nrays);
        __syncwarp();
        if (!kAny && S.leafKeys)
            order_rays(S, rays, E, src, 0, 1);
        if (lane == 0) fetch = 0;
        __syncwarp();
        if constexpr (kSub) subdivide_rays<kAny>(S, rays, E, p, q, hits, occluded, src, lend, lc, ListWalk<kAny> {});
        else clip_rays<kAny, kG64>(S, rays, E, p, q, hits, occluded, src, lend, lc, ListWalk<kAny> {});
        __syncwarp();
    }
    __syncwarp();
    if (!kAny && polishes(q.precision)) polish_rays(S, rays, hits, base, base + mine, 32, ring);
    flush_counters(cnt, lc, nrays);
}

// Explicit (ray, patch) pairs through the same searches: a warp takes an even
// share of the pairs.  One thread per pair ran a warp at the pace of its longest
// search: 200,003 pairs 99 us, 120 us before.
template<bool kSub>
__global__ void __launch_bounds__(32, 16) k_pairs(DevScene S, RaysSoA rays, uint32_t n, uint32_t surface, uint32_t patches,
                                                  const uint32_t* pids, Query q, int subdivLevels, HitsSoA hits,
                                                  Counters* cnt)
{
    __shared__ uint32_t fetch;
    __shared__ Lend<false> lend;
    const uint32_t lane = threadIdx.x, share = (n + gridDim.x - 1) / gridDim.x, base = blockIdx.x * share;
    if (base >= n) return;
    const WarpSource src {&fetch, min(share, n - base), base, nullptr};
    LocalCounters lc;
    for (uint32_t i = lane; i < src.m; i += 32)
        if (__ldg(pids + base + i) >= patches) lc.errors |= kErrPatchId;
    if (lane == 0) fetch = 0;
    __syncwarp();
    Eng E {};
    E.subdivLevels = uint32_t(subdivLevels);
    PairWalk w {surface, patches, pids};
    if constexpr (kSub) subdivide_rays<false>(S, rays, E, 0, q, hits, nullptr, src, lend, lc, w);
    else clip_rays<false, false>(S, rays, E, 0, q, hits, nullptr, src, lend, lc, w);
    __syncwarp();
    flush_counters(cnt, lc, lane == 0 ? src.m : 0u);
}

int sms()
{
    static const int v = [] {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        return n > 0 ? n : 1;
    }();
    return v;
}

int resident(const void* fn, int threads)
{
    int per = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, threads, 0);
    return sms() * (per > 0 ? per : 1);
}

// Resident blocks per SM of kernel fn at `threads` per block (cached: the
// values depend only on the kernel and the block size).
template<bool kAny, bool kG64, bool kSub> auto* search_kernel()
{
    if constexpr (kSub) return k_subdivide<kAny>;
    else return k_clip<kAny, kG64>;
}

template<bool kAny, bool kG64, bool kSub = false> int per_sm(bool collect, int threads, bool compressed = true)
{
    static const int v[3][2] = {
        {resident((const void*)k_collect<kAny, false, true>, 128) / sms(),
         resident((const void*)k_collect<kAny, false, true>, 256) / sms()},
        {resident((const void*)search_kernel<kAny, kG64, kSub>(), 64) / sms(),
         resident((const void*)search_kernel<kAny, kG64, kSub>(), 128) / sms()},
        {resident((const void*)k_collect<kAny, true, true>, 128) / sms(),
         resident((const void*)k_collect<kAny, true, true>, 256) / sms()}};
    return collect ? v[compressed ? 2 : 0][threads == 256] : v[1][threads == 128];
}

template<bool kAny>
void launch_collect(int grid, int threads, cudaStream_t stream, const DevScene& S, RaysSoA rays, uint32_t n,
                    const uint32_t* nDev, Eng E, int pass, const EngineConfig& c, Counters* cnt)
{
    auto* k = S.leafKeys ? (c.compressedNodes ? k_collect<kAny, true, true> : k_collect<kAny, false, true>)
                         : (c.compressedNodes ? k_collect<kAny, true, false> : k_collect<kAny, false, false>);
    k<<<grid, threads, 0, stream>>>(S, rays, n, nDev, E, pass, c.backtrackCache, cnt);
}

// Up to this many rays a query is one launch of k_small.  Closest hits, us a
// query in one launch / in separate kernels: camera rays of a 16,384-patch torus
// 92 / 229 at 32, 178 / 320 at 2,000, 273 / 365 at 16,000, 306 / 410 at 32,000,
// 528 / 598 at 64,000, 721 / 689 at 120,000; scattered rays of a 60,000-patch
// store 613 / 618 at 64,000; subdivision 552 / 658 at 32,000, 861 / 779 at 64,000.
// Near-grazing rays at the precision form, which end in a few long searches, ms:
// 16,384-patch torus 3.6 / 6.8 at 33, 5.4 / 7.3 at 1,000, 11.3 / 11.8 at 8,000,
// 17.9 / 18.5 at 65,536; a union scene 1.0 / 2.6, 2.2 / 3.5, 4.5 / 3.9, 9.8 / 9.9
// (7.3 / 6.7 at 32,000).
constexpr uint32_t kSmallRays = 65536, kSmallSubdivRays = 32768;

template<bool kAny, bool kG64, bool kSub = false>
void launch(const DevScene& S, RaysSoA rays, uint32_t n, const uint32_t* nDev, Query q, HitsSoA hits,
            int32_t* occluded, Eng E, Counters* cnt, cudaStream_t stream, int& nl)
{
    const EngineConfig c = engine_config();
    if (one_launch(n, kSub ? 1 : 0, kAny, nDev != nullptr) && !c.compressedNodes)
    {
        static const int warps = resident((const void*)k_small<kAny, kG64, kSub>, 32);
        k_small<kAny, kG64, kSub><<<int(std::min<uint32_t>(n, uint32_t(warps))), 32, 0, stream>>>(
            S, rays, n, nDev, E, c.passes, c.backtrackCache, q, hits, occluded, cnt);
        nl++;
        return;
    }
    cudaMemsetAsync(E.ctl, 0, sizeof(uint32_t) * 4 * (kMaxPasses + 1), stream);
    k_init<<<sms() * 4, 256, 0, stream>>>(rays, n, nDev, hits, kAny ? occluded : nullptr, E);
    nl++;
    const int ct = c.collectThreads, rt = c.resolveThreads;
    const int pc = per_sm<kAny, kG64, kSub>(true, ct, c.compressedNodes != 0);
    const int pr = per_sm<kAny, kG64, kSub>(false, rt);
    const int cb = sms() * std::max(1, c.collectOccupancy ? std::min(c.collectOccupancy, pc) : pc);
    const int rb = sms() * std::max(1, c.resolveOccupancy ? std::min(c.resolveOccupancy, pr) : pr);
    const uint32_t warps = (n + 31) / 32;
    const int gc = int(std::min<uint32_t>(uint32_t(cb), warps / (ct / 32) + 1));
    const int gr = int(std::min<uint32_t>(uint32_t(rb), warps / (rt / 32) + 1));
    const int gp = int(std::min<uint32_t>(uint32_t(sms() * 8), (n + kPendingThreads - 1) / kPendingThreads));
    for (int p = 0; p < c.passes; p++)
    {
        if (p > 0)
        {
            k_pending<<<gp, kPendingThreads, 0, stream>>>(E.status, n, nDev, E.queue[p & 1], E.ctl + 4 * p + 2);
            nl++;
        }
        launch_collect<kAny>(gc, ct, stream, S, rays, n, nDev, E, p, c, cnt);
        if (!kAny && S.leafKeys)
        {
            const int blocks = int(std::min<uint32_t>((n + kOrderThreads - 1) / kOrderThreads, uint32_t(sms() * 16)));
            if (p == 0)
            {
                k_order<<<blocks, kOrderThreads, 0, stream>>>(S, rays, n, nDev, E, p);
                k_order_long<<<sms(), kOrderThreads, 0, stream>>>(S, rays, E, p);
                nl++;
            }
            else k_order_queue<<<blocks, kOrderThreads, 0, stream>>>(S, rays, E, p);
            nl++;
        }
        search_kernel<kAny, kG64, kSub>()<<<gr, rt, 0, stream>>>(S, rays, n, nDev, E, p, q, hits, occluded, cnt);
        nl += 2;
    }
    k_pending<<<gp, kPendingThreads, 0, stream>>>(E.status, n, nDev, E.queue[c.passes & 1], E.ctl + 4 * c.passes + 2);
    k_rest<kAny><<<sms() * 4, 128, 0, stream>>>(S, rays, E, c.passes, q, hits, occluded, cnt);
    nl += 2;
    if (!kAny && polishes(q.precision))
    {
        k_polish<<<sms() * 8, kPolishThreads, 0, stream>>>(S, rays, n, nDev, hits);
        nl++;
    }
}

}  // namespace

namespace {
std::mutex gConfigMu;
EngineConfig gConfig;
uint64_t gConfigGen = 1;
}  // namespace

bool one_launch(uint32_t n, int method, bool any, bool deviceCount)
{
    // A render's shadow queue is sized for a ray per sample and light and holds the
    // ones that face it, none at all at most bounce levels: a preview of 319 x 181
    // pixels, two lights and three bounces takes 1.43 ms so, 1.79 ms without the
    // factor; frames of 51,200 to 120,000 samples the same within 3%.
    return n <= (method != 0 ? kSmallSubdivRays : kSmallRays) * (any && deviceCount ? 2 : 1);
}

EngineConfig engine_config()
{
    std::lock_guard<std::mutex> g(gConfigMu);
    return gConfig;
}

uint64_t engine_config_generation()
{
    std::lock_guard<std::mutex> g(gConfigMu);
    return gConfigGen;
}

bool valid_engine_config(const EngineConfig& c)
{
    return c.passes >= 1 && c.passes <= kMaxPasses && (c.collectThreads == 128 || c.collectThreads == 256) &&
           (c.resolveThreads == 64 || c.resolveThreads == 128) && c.collectOccupancy >= 0 && c.collectOccupancy <= 32 &&
           c.resolveOccupancy >= 0 && c.resolveOccupancy <= 32 && (c.backtrackCache == 0 || c.backtrackCache == 1) &&
           (c.compressedNodes == 0 || c.compressedNodes == 1) && c.queueChunk >= 4 &&
           c.queueChunk <= int(kChunk) && c.queueChunk % 4 == 0 && c.packetWidth >= 1 && c.packetWidth <= 32 &&
           (c.rayOrder == 0 || c.rayOrder == 1) && (c.originLast == 0 || c.originLast == 1) &&
           c.subdivLevels >= 1 && c.subdivLevels <= 64;
}

bool set_engine_config(const EngineConfig& c)
{
    if (!valid_engine_config(c)) return false;
    std::lock_guard<std::mutex> g(gConfigMu);
    gConfig = c;
    gConfigGen++;
    return true;
}

size_t engine_words(uint32_t capacity, int)
{
    return size_t(capacity) * kWordsPerRay + 4 * (kMaxPasses + 1) + 64 + 2ull * kLongList * long_lists(capacity);
}

cudaError_t run_query(const DevScene& S, RaysSoA rays, uint32_t n, const uint32_t* nDev, Query q, bool any,
                      HitsSoA hits, int32_t* occluded, uint32_t* scratch, uint32_t capacity, int, Counters* cnt,
                      cudaStream_t stream, int* launches, uint32_t turn)
{
    if (nDev) n = capacity;  // grid sizing only; kernels read *nDev
    if (n == 0) return cudaSuccess;
    if (n > capacity) return cudaErrorInvalidValue;
    if (any) q.precision = 0;  // any-hit searches run at level 0
    if (!any && q.precision == 2)
    {
        // the pure-FP64 search has no traversal / clip split
        if (launches) *launches += 1;
        return launch_query_fp64(S, rays, n, nDev, kTolFP64, hits, cnt, stream);
    }
    Eng E = carve(scratch, capacity);
    {
        const EngineConfig ec = engine_config();
        E.chunk = uint32_t(ec.queueChunk);
        E.packetWidth = uint32_t(ec.packetWidth);
        E.originLast = uint32_t(ec.originLast);
        E.subdivLevels = uint32_t(ec.subdivLevels);
    }
    if (cnt) E.longNext = &cnt->longNext[turn];
    else E.nlong = 0;
    int nl = 0;
    if (any) q.method != 0 ? launch<true, false, true>(S, rays, n, nDev, q, hits, occluded, E, cnt, stream, nl)
                           : launch<true, false>(S, rays, n, nDev, q, hits, occluded, E, cnt, stream, nl);
    else if (q.method != 0) launch<false, false, true>(S, rays, n, nDev, q, hits, occluded, E, cnt, stream, nl);
    else if (graze_sin(q.precision) > 0.0f) launch<false, true>(S, rays, n, nDev, q, hits, occluded, E, cnt, stream, nl);
    else launch<false, false>(S, rays, n, nDev, q, hits, occluded, E, cnt, stream, nl);
    if (launches) *launches += nl;
    return cudaGetLastError();
}

cudaError_t launch_patch_pairs(const DevScene& S, uint32_t surface, uint32_t patches, RaysSoA rays,
                               const uint32_t* patch_ids, uint32_t n, Query q, HitsSoA hits, Counters* counters,
                               cudaStream_t stream)
{
    if (n == 0) return cudaSuccess;
    static const int clip = resident((const void*)k_pairs<false>, 32), subdiv = resident((const void*)k_pairs<true>, 32);
    const bool sub = q.method != 0;
    auto* k = sub ? k_pairs<true> : k_pairs<false>;
    k<<<int(std::min<uint32_t>(n, uint32_t(sub ? subdiv : clip))), 32, 0, stream>>>(
        S, rays, n, surface, patches, patch_ids, q, engine_config().subdivLevels, hits, counters);
    return cudaGetLastError();
}

cudaError_t run_traverse(const DevScene& S, RaysSoA rays, uint32_t n, bool any, uint32_t* scratch, uint32_t capacity,
                         Counters* cnt, cudaStream_t stream, uint32_t* listLengths, int* launches)
{
    if (n == 0) return cudaSuccess;
    if (n > capacity) return cudaErrorInvalidValue;
    Eng E = carve(scratch, capacity);
    {
        const EngineConfig ec = engine_config();
        E.chunk = uint32_t(ec.queueChunk);
        E.packetWidth = uint32_t(ec.packetWidth);
        E.originLast = uint32_t(ec.originLast);
        E.subdivLevels = uint32_t(ec.subdivLevels);
    }
    E.nlong = 0;  // a list of patches and markers as long as a chunk is the entry point's contract
    E.allMarkers = 1;
    cudaMemsetAsync(E.ctl, 0, sizeof(uint32_t) * 4 * (kMaxPasses + 1), stream);
    const EngineConfig c = engine_config();
    const int ct = c.collectThreads;
    const bool cq = c.compressedNodes != 0;
    const int pc = any ? per_sm<true, false>(true, ct, cq) : per_sm<false, false>(true, ct, cq);
    const int cb = sms() * std::max(1, c.collectOccupancy ? std::min(c.collectOccupancy, pc) : pc);
    const int gc = int(std::min<uint32_t>(uint32_t(cb), (n + 31) / 32 / (ct / 32) + 1));
    if (any) launch_collect<true>(gc, ct, stream, S, rays, n, nullptr, E, 0, c, cnt);
    else launch_collect<false>(gc, ct, stream, S, rays, n, nullptr, E, 0, c, cnt);
    if (launches) *launches += 1;
    if (listLengths) cudaMemcpyAsync(listLengths, E.count, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, stream);
    return cudaGetLastError();
}

}  // namespace cgs
