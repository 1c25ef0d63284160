// scene.cu -- the scene store of libcgspline_gb300.so: surfaces, objects and
// groups, the host BVH build, device upload, the perfect-hash build of every
// BVH, and the C ABI entry points that build and inspect a store.
#include <atomic>
#include <bit>
#include <thread>
#include <cmath>
#include <memory>
#include <numeric>
#include <random>

#include "scene_impl.h"

using namespace cgs;

namespace cgs {

// BVH::build / split / wrap (src/rt/BVH.cpp:9-108): top-down median split,
// heap keys (root 1, children 2k and 2k+1), nodes in pre-order, leaves keep
// their box in leftBox and an EMPTY-terminated element list.  The split axis
// comes from the size of a box that is never inflated (src/rt/BVH.cpp:46-52),
// i.e. an empty box whose three extents compare equal, which selects y; the
// partition is std::nth_element with the same comparator, so the topology
// matches the reference built with the same standard library.  With
// CGS_SPLIT_LONGEST the box is the elements' centroid box (the evident intent
// of that code): same rule, same partition, the longest axis.
uint32_t HostBVH::wrap(Element* e, size_t count, uint32_t key)
{
    if (count == 0) emptyLeaf = true;
    Box box;
    size_t idx = indices.size();
    indices.resize(idx + count + 1);
    for (size_t i = 0; i < count; i++) { indices[idx + i] = e[i].index; box.inflate(e[i].bounds); }
    indices[idx + count] = EMPTY;
    keys.push_back(key);
    nodes.push_back({box, Box {}, EMPTY, uint32_t(idx)});
    return uint32_t(nodes.size() - 1);
}

uint32_t HostBVH::split(Element* e, size_t count, uint32_t key)
{
    if (count <= perNode || (key & (1u << 31))) return wrap(e, count, key);
    Box box;
    if (split_mode == CGS_SPLIT_LONGEST)
        for (size_t i = 0; i < count; i++) box.inflate(e[i].centroid);
    float v[3] = {box.hi[0] - box.lo[0], box.hi[1] - box.lo[1], box.hi[2] - box.lo[2]};
    const int dim = v[2] > v[1] ? (v[0] > v[2] ? 0 : 2) : (v[0] > v[1] ? 0 : 1);
    size_t middle = count / 2;
    std::nth_element(e, e + middle, e + count,
                     [=](const Element& a, const Element& b) { return a.centroid[dim] < b.centroid[dim]; });
    keys.push_back(key);
    size_t idx = nodes.size();
    nodes.push_back({});
    uint32_t l = split(e, middle, key << 1);
    uint32_t r = split(e + middle, count - middle, (key << 1) ^ 1u);
    Node& node = nodes[idx];
    node.left = l;
    node.right = r;
    node.leftBox = nodes[l].leftBox;
    node.rightBox = nodes[r].leftBox;
    if (nodes[l].left != EMPTY) node.leftBox.inflate(nodes[l].rightBox);
    if (nodes[r].left != EMPTY) node.rightBox.inflate(nodes[r].rightBox);
    return uint32_t(idx);
}

void HostBVH::build(std::vector<Element>& el)
{
    nodes.clear(); keys.clear(); indices.clear(); emptyLeaf = false;
    nodes.reserve(2 * el.size()); keys.reserve(2 * el.size()); indices.reserve(2 * el.size());
    split(el.data(), el.size(), 1u);
}

// std::mt19937(42) with std::uniform_int_distribution<uint32_t>(0, n) and
// gcd(n, A) == 1 retries (src/rt/PerfectHashFunction.cu:379-400): the 16
// trials' coefficients.
void hash_coefficients(uint32_t n, uint32_t A[16], uint32_t B[16])
{
    std::mt19937 mt(42);
    std::uniform_int_distribution<uint32_t> d(0, n);
    for (int t = 0; t < 16; t++)
    {
        uint32_t a, b, cof;
        do
        {
            a = d(mt);
            if (a == 0) a = 31;
            b = d(mt);
            cof = std::gcd(n, a);
        } while (cof > 1);
        A[t] = a; B[t] = b;
    }
}

// Table capacity: n plus 15 growth steps of max(4, 5% of n)
// (src/rt/PerfectHashFunction.cu:249-251, 481).
uint32_t table_capacity(uint32_t n)
{
    uint32_t step = std::max<uint32_t>(4u, uint32_t(0.05f * float(n)));
    return n + 15u * step;
}

// Displacement table size: the power of two at or below max(2, (n-1)/2)
// (src/rt/PerfectHashFunction.cu:233-248).
uint32_t displ_size(uint32_t n)
{
    int s = int(n - 1) >> 1;
    if (s < 2) s = 2;
    return std::bit_floor(uint32_t(s));
}

}  // namespace cgs

namespace {

DevMaterial to_dev(const cgs_material& m)
{
    DevMaterial d;
    std::memcpy(&d, &m, sizeof d);
    return d;
}

// Runs fn(0) .. fn(n - 1) on the host's cores, in any order; on this thread
// alone where there is little to do, on fewer where no more threads are to be had.
unsigned host_cores() { return std::max(1u, std::min(64u, std::thread::hardware_concurrency())); }
template<class F> void on_host_cores(size_t n, bool parallel, F&& fn)
{
    std::atomic<size_t> next {0};
    auto worker = [&]() { for (size_t w; (w = next.fetch_add(1)) < n;) fn(w); };
    const size_t nt = parallel ? std::min<size_t>(n, host_cores()) : 1;
    std::vector<std::thread> pool;
    pool.reserve(nt);
    try
    {
        for (size_t t = 1; t < nt; t++) pool.emplace_back(worker);
    }
    catch (const std::system_error&) {}
    worker();
    for (auto& th : pool) th.join();
}

// BezierSurface::buildBVH (src/rt/Primitive.cu:199-220): per-patch bounds of
// the 16 projected points and their mean as the centroid, of patches first to last - 1.
void fill_elements(const Surface& s, std::vector<Element>& el, size_t first, size_t last)
{
    for (size_t i = first; i < last; i++)
    {
        Element& e = el[i];
        e.bounds = Box {};
        e.centroid[0] = e.centroid[1] = e.centroid[2] = 0.0f;
        e.index = uint32_t(i);
        const float inv = 1.0f / 16.0f;
        for (int j = 0; j < 16; j++)
        {
            const float* w = &s.points[4ull * s.indices[16ull * i + j]];
            float p[3] = {w[0] / w[3], w[1] / w[3], w[2] / w[3]};
            e.bounds.inflate(p);
            for (int k = 0; k < 3; k++) e.centroid[k] = e.centroid[k] + inv * p[k];
        }
    }
}

// cores: by all of the host's.
std::vector<Element> surface_elements(const Surface& s, bool cores = false)
{
    std::vector<Element> el(s.patchCount());
    const size_t n = el.size(), chunk = cores ? 4096 : std::max<size_t>(n, 1);
    on_host_cores((n + chunk - 1) / chunk, cores,
                  [&](size_t c) { fill_elements(s, el, c * chunk, std::min(n, (c + 1) * chunk)); });
    return el;
}

// `out` takes the tree (its split_mode set by the caller).
void build_surface_bvh(const Surface& s, HostBVH& out)
{
    std::vector<Element> el = surface_elements(s);
    out.build(el);
}

// BezierSurface::bounds(M) (src/rt/Primitive.cu:172-179): the bounds of an
// object's transformed points.
Box object_bounds(const cgs_scene* sc, const Object& ob)
{
    const Surface& s = sc->surfaces[ob.surface];
    const float* M = ob.l2w;
    Box b;
    for (uint32_t idx : s.indices)
    {
        const float* w = &s.points[4ull * idx];
        float x = ((w[0] * M[0] + w[1] * M[4]) + w[2] * M[8]) + w[3] * M[12];
        float y = ((w[0] * M[1] + w[1] * M[5]) + w[2] * M[9]) + w[3] * M[13];
        float z = ((w[0] * M[2] + w[1] * M[6]) + w[2] * M[10]) + w[3] * M[14];
        float ww = ((w[0] * M[3] + w[1] * M[7]) + w[2] * M[11]) + w[3] * M[15];
        float p[3] = {x / ww, y / ww, z / ww};
        b.inflate(p);
    }
    return b;
}

// Scene::buildBVH (src/rt/Scene.cu:218-232) for one group: centroid = box
// centre, element index = the global object id; bounds: one box per object.
void build_group_bvh(const Group& g, const std::vector<Box>& bounds, HostBVH& out)
{
    std::vector<Element> el(g.objects.size());
    for (uint32_t i = 0; i < el.size(); i++)
    {
        const Box& b = bounds[g.objects[i]];
        el[i].index = g.objects[i];
        el[i].bounds = b;
        for (int k = 0; k < 3; k++) el[i].centroid[k] = 0.5f * (b.lo[k] + b.hi[k]);
    }
    out.build(el);
}

// ------------------------------------------------- compressed node mirror --
// A device-only copy of every BVH node in 32 bytes (one 256-bit load, one
// 32-byte sector) next to the exact 64-byte record, for the traversal
// kernel.  The child boxes are stored as 8-bit offsets on a per-axis grid
// (the compressed-wide-BVH encoding of Ylitie, Karras and Laine, HPG 2017,
// for binary nodes):
//
//   words 0-2  origin P (float) per axis
//   word  3    bytes 0-2: e per axis (grid step s = 2^(e-127)); byte 3: flags
//              (bit 0: leaf)
//   words 4-6  per axis the bytes (left lo, left hi, right lo, right hi); a
//              leaf keeps its own box in the left bytes
//   word  7    right child (inner node; the left child is the next node in
//              pre-order) or the leaf's first element index
//
// A byte q stands for the coordinate P + q s.  Every child box is widened on
// the grid by at least one step beyond its exact bounds (lo' <= lo - s,
// hi' >= hi + s), which covers the half-step rounding of the traversal's
// decode, so the decoded boxes contain the exact ones: a ray meets every box
// the exact test meets, at an entry distance no larger than the exact one.
// The traversal then visits the same leaves (and a few more) and finds the
// same hits.  A BVH with a node that has no such record (a non-finite box
// coordinate, an extent no grid of 2^-126..2^127 covers, or a left child
// that does not follow its parent, as a loaded blob may have) is read from
// the exact records only.
constexpr uint32_t kQLeaf = 1u;

__device__ float round_down_float(double x)
{
    float f = float(x);
    if (double(f) > x) f = nextafterf(f, -INFINITY);
    return f;
}

// Grid of one axis of a node covering [lo, hi] with a two-step margin below
// lo and at least two steps above hi inside 255 steps.  False if none.
__device__ bool axis_grid(double lo, double hi, float& P, int& e)
{
    if (!isfinite(lo) || !isfinite(hi) || hi < lo) return false;
    // the smallest e with 250 s >= extent, from the binary exponent of
    // extent / 250 (then checked upward)
    const double extent = hi - lo;
    int e0 = extent > 0.0 ? max(1, ilogb(extent / 250.0) + 127) : 1;
    while (e0 < 254 && ldexp(250.0, e0 - 127) < extent) e0++;
    for (e = e0; e <= 254; e++)
    {
        const double s = ldexp(1.0, e - 127);
        P = round_down_float(lo - 2.0 * s);
        if (!isfinite(P)) return false;
        if ((hi - double(P)) / s <= 253.0) return true;
    }
    return false;
}

// One tree's nodes among a store's: [first, first + count), its records in the
// compressed mirror from qbase on (EMPTY: it has none there), the BVH that they belong to.
struct PackJob { uint32_t first, count, qbase, bvh; };

// A node's 64-byte record on the device: the host's node and padding.
struct NodeRecord { Node node; uint32_t pad[2]; };
static_assert(sizeof(Node) == 56 && sizeof(NodeRecord) == 4 * sizeof(float4));

// The compressed mirror of a store's nodes: a thread per node, all trees in one
// launch (their jobs in ascending order).  failed[bvh] is set where a node has no
// compressed record.  Bound by its launch; on the host, one thread over 120,000
// nodes, it was most of the 8.4 ms that the upload and hash build of a
// 30,000-patch store took (2.0 ms now).
__global__ void k_pack_nodes(const NodeRecord* __restrict__ nodes, const PackJob* __restrict__ jobs, uint32_t njobs,
                             uint32_t total, uint4* qnodes, uint32_t* failed)
{
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < total; g += gridDim.x * blockDim.x)
    {
        const Node n = nodes[g].node;
        const Box &L = n.leftBox, &R = n.rightBox;
        uint32_t lo = 0, hi = njobs;
        while (hi - lo > 1)
        {
            const uint32_t mid = (lo + hi) / 2;
            if (jobs[mid].first <= g) lo = mid; else hi = mid;
        }
        const PackJob J = jobs[lo];
        if (J.qbase == EMPTY) continue;
        const uint32_t i = g - J.first;
        const bool leaf = n.left == EMPTY;
        // the compressed record names only the right child: the left one must follow
        bool ok = leaf || n.left == i + 1;
        uint32_t P[3] = {}, bytes[3] = {}, ex[3] = {};
        for (int a = 0; a < 3 && ok; a++)
        {
            const double blo = leaf ? double(L.lo[a]) : fmin(double(L.lo[a]), double(R.lo[a]));
            const double bhi = leaf ? double(L.hi[a]) : fmax(double(L.hi[a]), double(R.hi[a]));
            float p = 0;
            int e = 0;
            if (!axis_grid(blo, bhi, p, e)) { ok = false; break; }
            const double s = ldexp(1.0, e - 127), pd = double(p);
            const double v[4] = {ceil((double(L.lo[a]) - pd) / s) - 2.0, floor((double(L.hi[a]) - pd) / s) + 2.0,
                                 leaf ? 0.0 : ceil((double(R.lo[a]) - pd) / s) - 2.0,
                                 leaf ? 0.0 : floor((double(R.hi[a]) - pd) / s) + 2.0};
            for (int k = 0; k < 4; k++)
            {
                if (!(v[k] >= 0.0 && v[k] <= 255.0)) ok = false;
                else bytes[a] |= uint32_t(v[k]) << (8 * k);
            }
            P[a] = __float_as_uint(p);
            ex[a] = uint32_t(e);
        }
        if (!ok)
        {
            failed[J.bvh] = 1u;
            for (int a = 0; a < 3; a++) { P[a] = 0; ex[a] = 127; bytes[a] = 0; }
        }
        uint4* w = qnodes + 2ull * (J.qbase + i);
        w[0] = make_uint4(P[0], P[1], P[2], ex[0] | (ex[1] << 8) | (ex[2] << 16) | ((leaf ? kQLeaf : 0u) << 24));
        w[1] = make_uint4(bytes[0], bytes[1], bytes[2], n.right);
    }
}

// Lights of all groups, concatenated; groupLights[g] = (first, count);
// groupEnv[g] = background rgb, ambient rgb.
int upload_lights(cgs_scene* sc)
{
    std::vector<DevLight> hl;
    std::vector<uint2> gl;
    std::vector<float> env;
    for (const Group& g : sc->groups)
    {
        gl.push_back(make_uint2(uint32_t(hl.size()), uint32_t(g.lights.size())));
        for (const auto& l : g.lights) { DevLight d; std::memcpy(&d, &l, sizeof d); hl.push_back(d); }
        for (int k = 0; k < 3; k++) env.push_back(g.background[k]);
        for (int k = 0; k < 3; k++) env.push_back(g.ambient[k]);
    }
    CGS_TRY(sc->dlights.reserve(std::max<size_t>(hl.size(), 1)));
    CGS_TRY(sc->groupLights.reserve(gl.size()));
    CGS_TRY(sc->groupEnv.reserve(env.size()));
    if (!hl.empty()) CGS_TRY(cudaMemcpy(sc->dlights.p, hl.data(), hl.size() * sizeof(DevLight), cudaMemcpyHostToDevice));
    CGS_TRY(cudaMemcpy(sc->groupLights.p, gl.data(), gl.size() * sizeof(uint2), cudaMemcpyHostToDevice));
    CGS_TRY(cudaMemcpy(sc->groupEnv.p, env.data(), env.size() * sizeof(float), cudaMemcpyHostToDevice));
    return CGS_OK;
}

}  // namespace

namespace {

// The longest-axis tree of halves, one element to a leaf (which names it), in
// place: a subtree of n elements has 2 n - 1 nodes, so every node's place in
// pre-order is known beforehand and subtrees can be built by different cores.
struct WalkTree
{
    struct Part { Element* e; size_t count; uint32_t key, at; };
    std::vector<Node>& nodes;
    std::vector<uint32_t>& keys;

    // One node: false for a leaf, else its halves.
    bool split(const Part& p, Part& l, Part& r) const
    {
        keys[p.at] = p.key;
        Node& n = nodes[p.at];
        if (p.count == 1)
        {
            Box box;
            box.inflate(p.e->bounds);
            n = Node {box, Box {}, EMPTY, p.e->index};
            return false;
        }
        Box box;
        for (size_t i = 0; i < p.count; i++) box.inflate(p.e[i].centroid);
        const float v[3] = {box.hi[0] - box.lo[0], box.hi[1] - box.lo[1], box.hi[2] - box.lo[2]};
        const int dim = v[2] > v[1] ? (v[0] > v[2] ? 0 : 2) : (v[0] > v[1] ? 0 : 1);  // as HostBVH::split
        const size_t middle = p.count / 2;
        std::nth_element(p.e, p.e + middle, p.e + p.count,
                         [=](const Element& a, const Element& b) { return a.centroid[dim] < b.centroid[dim]; });
        l = Part {p.e, middle, p.key << 1, p.at + 1};
        r = Part {p.e + middle, p.count - middle, (p.key << 1) ^ 1u, p.at + uint32_t(2 * middle)};
        n = Node {Box {}, Box {}, l.at, r.at};
        return true;
    }
    // An inner node's boxes, its children's being done.
    void join(uint32_t at) const
    {
        Node& n = nodes[at];
        const Node &l = nodes[n.left], &r = nodes[n.right];
        n.leftBox = l.leftBox;
        n.rightBox = r.leftBox;
        if (l.left != EMPTY) n.leftBox.inflate(l.rightBox);
        if (r.left != EMPTY) n.rightBox.inflate(r.rightBox);
    }
    void build(const Part& p) const
    {
        Part l, r;
        if (!split(p, l, r)) return;
        build(l);
        build(r);
        join(p.at);
    }
    // The same by all cores: level by level until there are enough subtrees.
    void build_on_cores(const Part& root) const
    {
        std::vector<Part> parts {root};
        std::vector<uint32_t> inner;
        while (parts.size() < 4 * host_cores())
        {
            std::vector<Part> next(2 * parts.size());
            on_host_cores(parts.size(), true, [&](size_t i) {
                if (!split(parts[i], next[2 * i], next[2 * i + 1])) next[2 * i].count = 0;
            });
            for (const Part& p : parts) if (p.count > 1) inner.push_back(p.at);
            parts.clear();
            for (size_t i = 0; i < next.size(); i += 2)
                if (next[i].count) { parts.push_back(next[i]); parts.push_back(next[i + 1]); }
            if (parts.empty()) break;
        }
        on_host_cores(parts.size(), true, [&](size_t i) { build(parts[i]); });
        for (size_t i = inner.size(); i > 0; i--) join(inner[i - 1]);
    }
};

}  // namespace

// A second tree over a surface's patches for the query engine to walk: the
// same median halves, split on the longest axis.  Halving n elements gives
// the same heap keys in the same pre-order whatever the axis, so a hash table
// of the one tree's keys finds the other's nodes.
void cgs::build_walk_bvh(const Surface& s, HostBVH& out, bool cores)
{
    std::vector<Element> el = surface_elements(s, cores);
    out = HostBVH {};
    out.split_mode = CGS_SPLIT_LONGEST;
    if (el.empty()) return;
    for (const Element& e : el)
        for (int k = 0; k < 3; k++)
            if (!std::isfinite(e.bounds.lo[k]) || !std::isfinite(e.bounds.hi[k])) return;
    if (cores)
    {
        out.nodes.resize(2 * el.size() - 1);
        out.keys.resize(2 * el.size() - 1);
        WalkTree {out.nodes, out.keys}.build_on_cores({el.data(), el.size(), 1u, 0u});
        return;
    }
    // by one core: the nodes in order, each written once (4.5 M patches by 16 cores 172 ms, in place 186 ms)
    out.build(el);
    for (Node& n : out.nodes)
        if (n.left == EMPTY) n.right = out.indices[n.right];  // a leaf names its patch
    out.indices.clear();
}

// The walk trees of a store read from a blob: surfaces side by side, and one
// that has more than a core's share of the patches by all cores before them.
// (One thread takes 1.6 s per million patches.)
void cgs::build_walk_bvhs(cgs_scene* sc)
{
    size_t patches = 0;
    for (const Surface& s : sc->surfaces) patches += s.patchCount();
    std::vector<Surface*> few;
    for (Surface& s : sc->surfaces)
        if (s.patchCount() >= 16384 && size_t(s.patchCount()) * host_cores() > patches) build_walk_bvh(s, s.walk, true);
        else few.push_back(&s);
    std::sort(few.begin(), few.end(), [](const Surface* a, const Surface* b) { return a->patchCount() > b->patchCount(); });
    on_host_cores(few.size(), patches > 250, [&](size_t w) { build_walk_bvh(*few[w], few[w]->walk); });
    on_host_cores(sc->surfaces.size(), patches > 250, [&](size_t i) { check_walk_bvh(sc->surfaces[i]); });
}

// What the walk relies on: both trees have the same keys in the same order and
// one leaf per patch, a patch's leaf box is the same in both, and every inner
// box of the reference tree contains its children (the walk tree's do by
// construction).  Trees built here have it; one read from a blob may not.
void cgs::check_walk_bvh(Surface& s)
{
    const HostBVH &b = s.bvh, &w = s.walk;
    if (w.nodes.empty()) return;
    auto contains = [](const Box& outer, const Box& inner) {
        for (int k = 0; k < 3; k++)
            if (!(outer.lo[k] <= inner.lo[k] && outer.hi[k] >= inner.hi[k])) return false;
        return true;
    };
    bool ok = b.keys == w.keys && b.nodes.size() == 2ull * s.patchCount() - 1;
    std::vector<const Box*> box(s.patchCount(), nullptr);
    for (const Node& n : w.nodes)
        if (n.left == EMPTY) box[n.right] = &n.leftBox;
    for (size_t i = 0; ok && i < b.nodes.size(); i++)
    {
        const Node& n = b.nodes[i];
        if (n.left == EMPTY)
        {
            // one element, not seen before, with its own box
            const uint32_t e = b.indices[n.right];
            ok = e < box.size() && b.indices[n.right + 1] == EMPTY && box[e] &&
                 std::memcmp(box[e], &n.leftBox, sizeof(Box)) == 0;
            if (ok) box[e] = nullptr;
            continue;
        }
        const Node &l = b.nodes[n.left], &r = b.nodes[n.right];
        ok = contains(n.leftBox, l.leftBox) && (l.left == EMPTY || contains(n.leftBox, l.rightBox)) &&
             contains(n.rightBox, r.leftBox) && (r.left == EMPTY || contains(n.rightBox, r.rightBox));
    }
    if (!ok) s.walk = HostBVH {};
}

// Device copy of the store's host state (everything but the hash tables).
int cgs::upload_store(cgs_scene* sc)
{
    const uint32_t nb = sc->nbvh(), ns = uint32_t(sc->surfaces.size());
    std::vector<uint32_t> pbase, pmat, gtop;
    std::vector<DevMaterial> hm;
    std::vector<DevObject> ho;
    std::vector<PackJob> jobs;
    sc->hbvh.assign(nb, DevBVH {});
    sc->tableCap.assign(nb, 0);
    sc->walkTrees = false;
    uint32_t tableCursor = 0, dispCursor = 0, nodeCursor = 0, indexCursor = 0, qCursor = 0;
    for (uint32_t k = 0; k < nb; k++)
    {
        const HostBVH& b = sc->bvh(k);
        DevBVH& d = sc->hbvh[k];
        const uint32_t n = uint32_t(b.nodes.size());
        const bool walk = k < ns && !sc->surfaces[k].walk.nodes.empty();
        d.nodeBase = nodeCursor;
        d.indexBase = indexCursor;
        d.qnodeBase = qCursor;
        d.walkBase = walk ? nodeCursor + n : EMPTY;
        jobs.push_back({nodeCursor, n, walk ? EMPTY : qCursor, k});
        if (walk) jobs.push_back({nodeCursor + n, n, qCursor, k});
        nodeCursor += walk ? 2 * n : n;
        qCursor += n;
        indexCursor += uint32_t(b.indices.size());
        sc->walkTrees = sc->walkTrees || walk;
        d.tableBase = tableCursor;
        d.dispBase = dispCursor;
        sc->tableCap[k] = table_capacity(n);
        tableCursor += sc->tableCap[k];
        dispCursor += displ_size(n);
        d.mask = displ_size(n) - 1;
        d.N = n; d.A = 31; d.B = 19;
        d.Nmagic = fastmod_magic(std::max<uint32_t>(n, 1));
    }
    for (uint32_t g = 0; g < sc->groups.size(); g++) gtop.push_back(ns + g);
    uint32_t patches = 0;
    for (const Surface& s : sc->surfaces)
    {
        pbase.push_back(patches);
        patches += s.patchCount();
    }
    for (const Object& ob : sc->objects)
    {
        DevObject d {};
        std::memcpy(d.w2l, ob.w2l, sizeof d.w2l);
        d.surface = ob.surface;
        d.material = uint32_t(hm.size());
        hm.push_back(to_dev(ob.material));
        if (!ob.patchMaterial.empty())
        {
            d.patchMaterialBase = int32_t(pmat.size());
            uint32_t mbase = uint32_t(hm.size());
            for (const auto& m : ob.materials) hm.push_back(to_dev(m));
            for (uint32_t pm : ob.patchMaterial) pmat.push_back(mbase + pm);
        }
        else
            d.patchMaterialBase = -1;
        ho.push_back(d);
    }
    // The device's arrays in one staging area on the host, filled by its cores:
    // de-indexed patches (16 points each), node records, leaf lists, leaf keys.  They
    // go to their places as they are, so a store needs no more device memory while it
    // is made than afterwards.
    auto place = [cursor = size_t(0)](size_t bytes) mutable {
        const size_t at = cursor;
        cursor = (cursor + bytes + 255) & ~size_t(255);
        return at;
    };
    const size_t oPatches = place(size_t(patches) * 256), oNodes = place(size_t(nodeCursor) * sizeof(NodeRecord)),
                 oList = place(size_t(indexCursor) * 4), oKeys = place(sc->walkTrees ? size_t(patches) * 4 : 0),
                 total = place(0);
    std::unique_ptr<uint8_t[]> stage(new (std::nothrow) uint8_t[std::max<size_t>(total, 1)]);
    if (!stage) return CGS_ERR_OUT_OF_MEMORY;
    uint8_t* h = stage.get();
    // one piece of work is a range of a tree's nodes and of its surface's patches
    struct Piece { uint32_t k, first; };
    constexpr uint32_t kPiece = 8192;
    std::vector<Piece> pieces;
    for (uint32_t k = 0; k < nb; k++)
        for (uint32_t first = 0; first == 0 || first < sc->bvh(k).nodes.size(); first += kPiece) pieces.push_back({k, first});
    on_host_cores(pieces.size(), total > (1u << 20), [&](size_t i) {
        const uint32_t k = pieces[i].k, first = pieces[i].first;
        const HostBVH& b = sc->bvh(k);
        const DevBVH& d = sc->hbvh[k];
        NodeRecord* nodes = reinterpret_cast<NodeRecord*>(h + oNodes);
        const bool walk = d.walkBase != EMPTY;
        const Surface* s = k < ns ? &sc->surfaces[k] : nullptr;
        uint32_t* keys = reinterpret_cast<uint32_t*>(h + oKeys) + (s ? pbase[k] : 0);
        for (size_t j = first; j < std::min<size_t>(b.nodes.size(), first + kPiece); j++)
        {
            nodes[d.nodeBase + j] = NodeRecord {b.nodes[j], {0, 0}};
            if (!walk) continue;
            nodes[d.walkBase + j] = NodeRecord {s->walk.nodes[j], {0, 0}};
            if (b.nodes[j].left == EMPTY) keys[b.indices[b.nodes[j].right]] = b.keys[j];
        }
        if (first == 0)
            std::copy(b.indices.begin(), b.indices.end(), reinterpret_cast<uint32_t*>(h + oList) + d.indexBase);
        if (!s) return;
        // (a tree has up to twice as many nodes as its surface patches: the last piece takes the rest)
        const bool last = size_t(first) + kPiece >= b.nodes.size();
        const uint32_t p0 = std::min(first, s->patchCount()), p1 = last ? s->patchCount() : std::min(first + kPiece, s->patchCount());
        float* out = reinterpret_cast<float*>(h + oPatches) + 64ull * (size_t(pbase[k]) + p0);
        for (size_t j = 16ull * p0; j < 16ull * p1; j++, out += 4) std::memcpy(out, &s->points[4ull * s->indices[j]], 16);
        if (sc->walkTrees && !walk) std::fill(keys + p0, keys + p1, 0u);
    });
    CGS_TRY(sc->patches.reserve(size_t(patches) * 16));
    CGS_TRY(sc->nodes.reserve(4ull * nodeCursor));
    CGS_TRY(sc->qnodes.reserve(2ull * qCursor));
    CGS_TRY(sc->indices.reserve(indexCursor));
    CGS_TRY(sc->tables.reserve(tableCursor));
    CGS_TRY(sc->disps.reserve(dispCursor));
    CGS_TRY(sc->patchBase.reserve(pbase.size()));
    CGS_TRY(sc->patchMaterial.reserve(std::max<size_t>(pmat.size(), 1)));
    CGS_TRY(sc->bvhs.reserve(nb));
    CGS_TRY(sc->groupTop.reserve(gtop.size()));
    CGS_TRY(sc->dobjects.reserve(ho.size()));
    CGS_TRY(sc->materials.reserve(hm.size()));
    CGS_TRY(sc->counters.reserve(1));
    if (sc->walkTrees) CGS_TRY(sc->leafKeys.reserve(patches));
    // the jobs and the flags that they raise, in one small array
    struct Temp
    {
        DBuf<uint32_t> b;
        ~Temp() { b.release(); }
    } temp;
    const size_t jobWords = jobs.size() * sizeof(PackJob) / 4;
    std::vector<uint32_t> jobStage(jobWords + nb, 0u);
    std::memcpy(jobStage.data(), jobs.data(), jobs.size() * sizeof(PackJob));
    CGS_TRY(temp.b.reserve(jobStage.size()));
    uint32_t* dFailed = temp.b.p + jobWords;
    CGS_TRY(cudaMemcpy(temp.b.p, jobStage.data(), jobStage.size() * 4, cudaMemcpyHostToDevice));
    CGS_TRY(cudaMemcpy(sc->nodes.p, h + oNodes, size_t(nodeCursor) * sizeof(NodeRecord), cudaMemcpyHostToDevice));
    k_pack_nodes<<<(nodeCursor + 127) / 128, 128>>>(reinterpret_cast<const NodeRecord*>(sc->nodes.p),
                                                    reinterpret_cast<const PackJob*>(temp.b.p), uint32_t(jobs.size()),
                                                    nodeCursor, sc->qnodes.p, dFailed);
    CGS_TRY(cudaGetLastError());
    CGS_TRY(cudaMemcpy(sc->patches.p, h + oPatches, size_t(patches) * 256, cudaMemcpyHostToDevice));
    CGS_TRY(cudaMemcpy(sc->indices.p, h + oList, size_t(indexCursor) * 4, cudaMemcpyHostToDevice));
    if (sc->walkTrees) CGS_TRY(cudaMemcpy(sc->leafKeys.p, h + oKeys, size_t(patches) * 4, cudaMemcpyHostToDevice));
    CGS_TRY(cudaMemcpy(sc->patchBase.p, pbase.data(), pbase.size() * sizeof(uint32_t), cudaMemcpyHostToDevice));
    if (!pmat.empty())
        CGS_TRY(cudaMemcpy(sc->patchMaterial.p, pmat.data(), pmat.size() * sizeof(uint32_t), cudaMemcpyHostToDevice));
    CGS_TRY(cudaMemcpy(sc->dobjects.p, ho.data(), ho.size() * sizeof(DevObject), cudaMemcpyHostToDevice));
    CGS_TRY(cudaMemcpy(sc->materials.p, hm.data(), hm.size() * sizeof(DevMaterial), cudaMemcpyHostToDevice));
    CGS_TRY(cudaMemcpy(sc->groupTop.p, gtop.data(), gtop.size() * sizeof(uint32_t), cudaMemcpyHostToDevice));
    std::vector<uint32_t> failed(nb);
    CGS_TRY(cudaMemcpy(failed.data(), dFailed, nb * sizeof(uint32_t), cudaMemcpyDeviceToHost));
    for (uint32_t k = 0; k < nb; k++) sc->hbvh[k].compressed = failed[k] ? 0u : 1u;
    CGS_TRY(cudaMemcpy(sc->bvhs.p, sc->hbvh.data(), nb * sizeof(DevBVH), cudaMemcpyHostToDevice));
    int r = upload_lights(sc);
    if (r) return r;
    for (Surface& s : sc->surfaces) s.walk = HostBVH {};  // only the device needs it
    sc->uploaded = true;
    return CGS_OK;
}

namespace {

int upload(cgs_scene* sc) { return upload_store(sc); }

// BVH::buildHashTable (src/rt/BVH.cpp:24-39) for every BVH of the store.
// BVHs of at most kHashBlockMaxKeys keys (most: one per surface) are built
// together, one CTA each, in one launch; those of at most
// kHashGlobalBlockMaxKeys by a cluster of CTAs and a global scratch area each,
// in a launch for each number of buckets; one host round trip reads all these
// launches' results.  Larger BVHs run the multi-launch build one at a time.
int hash_all(cgs_scene* sc, cudaStream_t stream)
{
    const uint32_t nb = sc->nbvh();
    std::vector<uint32_t> small, mid, large;
    uint32_t maxSmall = 1, maxLarge = 1;
    size_t blockKeys = 0;
    uint64_t midScratch = 0;
    for (uint32_t k = 0; k < nb; k++)
    {
        const uint32_t n = uint32_t(sc->bvh(k).keys.size());
        if (n <= kHashBlockMaxKeys) { small.push_back(k); maxSmall = std::max(maxSmall, n); blockKeys += n; }
        else if (n <= kHashGlobalBlockMaxKeys)
        {
            mid.push_back(k);
            blockKeys += n;
            midScratch += hash_block_scratch_words(n) + 1;
        }
        else { large.push_back(k); maxLarge = std::max(maxLarge, n); }
    }
    CGS_TRY(sc->keys.reserve(std::max<size_t>({blockKeys, size_t(maxLarge), 1})));
    std::stable_sort(mid.begin(), mid.end(),
                     [&](uint32_t a, uint32_t b) { return sc->bvh(a).keys.size() > sc->bvh(b).keys.size(); });
    if (!small.empty() || !mid.empty())
    {
        std::vector<uint32_t> hk;
        hk.reserve(blockKeys);
        std::vector<HashJob> jobs(small.size() + mid.size());
        uint64_t scratchCursor = 0;
        for (size_t j = 0; j < jobs.size(); j++)
        {
            const uint32_t k = j < small.size() ? small[j] : mid[j - small.size()];
            const HostBVH& b = sc->bvh(k);
            const uint32_t n = uint32_t(b.keys.size());
            HashJob& J = jobs[j];
            J.keyOff = uint32_t(hk.size());
            J.n = n;
            J.dispOff = sc->hbvh[k].dispBase;
            J.tableOff = sc->hbvh[k].tableBase;
            J.tableCap = sc->tableCap[k];
            J.mask = displ_size(n) - 1;
            J.scratchOff = 0;
            J.pad = 0;
            if (j >= small.size())
            {
                if (scratchCursor > 0xFFFFFFFFull) return CGS_ERR_OUT_OF_MEMORY;
                J.scratchOff = uint32_t(scratchCursor);
                scratchCursor += (hash_block_scratch_words(n) + 2) & ~1ull;  // keep 8-byte alignment
            }
            hash_coefficients(n, J.A, J.B);
            hk.insert(hk.end(), b.keys.begin(), b.keys.end());
        }
        const size_t jobWords = (jobs.size() * sizeof(HashJob) + 3) / 4;
        CGS_TRY(sc->hashJobs.reserve(jobWords + 8 * jobs.size()));
        if (!mid.empty()) CGS_TRY(sc->scratch32.reserve(std::max<uint64_t>(scratchCursor, 1)));
        uint32_t* dJobs = sc->hashJobs.p;
        uint32_t* dOut = sc->hashJobs.p + jobWords;
        CGS_TRY(cudaMemcpyAsync(sc->keys.p, hk.data(), hk.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, stream));
        CGS_TRY(cudaMemcpyAsync(dJobs, jobs.data(), jobs.size() * sizeof(HashJob), cudaMemcpyHostToDevice, stream));
        const HashJob* dj = reinterpret_cast<const HashJob*>(dJobs);
        if (!small.empty())
        {
            CGS_TRY(hash_build_blocks(sc->keys.p, dj, uint32_t(small.size()), maxSmall, sc->disps.p, sc->tables.p,
                                      dOut, stream));
            sc->launches += 1;
        }
        // the mid BVHs' launches: one for each number of buckets, the largest first
        for (size_t i = 0, e = 0; i < mid.size(); i = e)
        {
            const uint32_t maxKeys = uint32_t(sc->bvh(mid[i]).keys.size());
            for (e = i; e < mid.size(); e++)
                if (hash_block_buckets(uint32_t(sc->bvh(mid[e]).keys.size())) != hash_block_buckets(maxKeys)) break;
            CGS_TRY(hash_build_blocks(sc->keys.p, dj + small.size() + i, uint32_t(e - i), maxKeys, sc->disps.p,
                                      sc->tables.p, dOut + 8 * (small.size() + i), stream, sc->scratch32.p,
                                      uint32_t(mid.size())));
            sc->launches += 1;
        }
        std::vector<uint32_t> res(8 * jobs.size());
        CGS_TRY(cudaMemcpyAsync(res.data(), dOut, res.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost, stream));
        CGS_TRY(cudaStreamSynchronize(stream));
        for (size_t j = 0; j < jobs.size(); j++)
        {
            const uint32_t* r = &res[8 * j];
            if (r[0] == 4) return CGS_ERR_HASH_BUCKET_OVERFLOW;
            if (r[0]) return CGS_ERR_HASH_FAILED;
            DevBVH& d = sc->hbvh[j < small.size() ? small[j] : mid[j - small.size()]];
            d.A = r[1]; d.B = r[2]; d.N = r[3]; d.mask = r[4];
            d.Nmagic = fastmod_magic(d.N);
        }
    }
    if (!large.empty())
    {
        size_t w32 = 0, w64 = 0;
        hash_scratch_words(maxLarge, w32, w64);
        CGS_TRY(sc->scratch32.reserve(w32));
        CGS_TRY(sc->scratch64.reserve(w64));
        for (uint32_t k : large)
        {
            const HostBVH& b = sc->bvh(k);
            const uint32_t n = uint32_t(b.keys.size());
            HashScratch hs {};
            hash_scratch_carve(hs, n, sc->scratch32.p, sc->scratch64.p);
            CGS_TRY(cudaMemcpyAsync(sc->keys.p, b.keys.data(), n * sizeof(uint32_t), cudaMemcpyHostToDevice, stream));
            uint32_t A[16], B[16], params[5];
            hash_coefficients(n, A, B);
            DevBVH& d = sc->hbvh[k];
            int r = hash_build_device(sc->keys.p, n, A, B, sc->disps.p + d.dispBase, sc->tables.p + d.tableBase,
                                      sc->tableCap[k], hs, params, stream, &sc->launches);
            if (r == 4) return CGS_ERR_HASH_BUCKET_OVERFLOW;
            if (r < 0) return CGS_ERR_CUDA;
            if (r) return CGS_ERR_HASH_FAILED;
            d.A = params[0]; d.B = params[1]; d.N = params[2]; d.mask = params[3];
            d.Nmagic = fastmod_magic(d.N);
        }
    }
    CGS_TRY(cudaMemcpyAsync(sc->bvhs.p, sc->hbvh.data(), nb * sizeof(DevBVH), cudaMemcpyHostToDevice, stream));
    CGS_TRY(cudaStreamSynchronize(stream));
    sc->hashed = true;
    return CGS_OK;
}

Group& current_group(cgs_scene* s) { return s->groups[s->current]; }

// The exported form of BVH k of a mirrored store (CGS_SPLIT_MIRROR): the
// reference-topology tree, built again on the host, and, once the store is
// hashed, its perfect-hash table from the same device build as the store's
// (cgs_perfect_hash_build) into temporary buffers.  params = A, B, N, mask.
int mirror_export(const cgs_scene* s, uint32_t k, HostBVH& ref, std::vector<uint32_t>& table,
                  std::vector<uint32_t>& disp, uint32_t params[4])
{
    const size_t ns = s->surfaces.size();
    ref.split_mode = CGS_SPLIT_REFERENCE;
    if (k < ns) build_surface_bvh(s->surfaces[k], ref);
    else
    {
        std::vector<Box> bounds(s->objects.size());
        for (uint32_t o : s->groups[k - ns].objects) bounds[o] = object_bounds(s, s->objects[o]);
        build_group_bvh(s->groups[k - ns], bounds, ref);
    }
    if (ref.emptyLeaf) return CGS_ERR_EMPTY_LEAF;
    params[0] = params[1] = params[2] = params[3] = 0;
    table.clear();
    disp.clear();
    if (!s->hashed) return CGS_OK;
    CGS_TRY(cudaSetDevice(s->device));
    const uint32_t n = uint32_t(ref.keys.size());
    const uint32_t dcap = displ_size(n), tcap = table_capacity(n);
    struct Temp
    {
        DBuf<uint32_t> keys, disp, table;
        ~Temp() { keys.release(); disp.release(); table.release(); }
    } d;
    CGS_TRY(d.keys.reserve(n));
    CGS_TRY(d.disp.reserve(dcap));
    CGS_TRY(d.table.reserve(tcap));
    uint32_t p5[5] = {};
    CGS_TRY(cudaMemcpy(d.keys.p, ref.keys.data(), n * sizeof(uint32_t), cudaMemcpyHostToDevice));
    if (int r = cgs_perfect_hash_build(d.keys.p, n, d.disp.p, dcap, d.table.p, tcap, p5, nullptr)) return r;
    if (p5[2] > tcap || size_t(p5[3]) + 1 > dcap) return CGS_ERR_HASH_FAILED;
    table.resize(p5[2]);
    disp.resize(size_t(p5[3]) + 1);
    CGS_TRY(cudaMemcpy(disp.data(), d.disp.p, disp.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost));
    CGS_TRY(cudaMemcpy(table.data(), d.table.p, table.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost));
    for (int j = 0; j < 4; j++) params[j] = p5[j];
    return CGS_OK;
}

bool bvh_index(const cgs_scene* s, int32_t which, uint32_t& k)
{
    if (which >= 0)
    {
        if (uint32_t(which) >= s->surfaces.size()) return false;
        k = uint32_t(which);
        return true;
    }
    uint32_t g = uint32_t(-1 - int64_t(which));
    if (g >= s->groups.size()) return false;
    k = uint32_t(s->surfaces.size()) + g;
    return true;
}

}  // namespace

cgs::DevScene cgs_scene::dev() const
{
    DevScene S {};
    S.patches = patches.p; S.nodes = nodes.p; S.qnodes = qnodes.p; S.indices = indices.p; S.tables = tables.p; S.disps = disps.p;
    S.bvhs = bvhs.p; S.patchBase = patchBase.p; S.leafKeys = walkTrees ? leafKeys.p : nullptr; S.objects = dobjects.p; S.materials = materials.p;
    S.patchMaterial = patchMaterial.p; S.lights = dlights.p;
    S.groupTop = groupTop.p; S.groupLights = groupLights.p; S.groupEnv = groupEnv.p;
    S.nobjects = uint32_t(objects.size()); S.nsurfaces = uint32_t(surfaces.size());
    S.ngroups = uint32_t(groups.size());
    return S;
}

cgs_scene::~cgs_scene()
{
    cudaSetDevice(device);
    patches.release(); nodes.release(); qnodes.release();
    for (auto* b : {&indices, &tables, &disps, &patchBase, &patchMaterial, &keys, &groupTop, &scratch32, &groupStage,
                    &hashJobs, &leafKeys,
                    &engine, &fbStage})
        b->release();
    if (hostStage) cudaFreeHost(hostStage);
    rayStage.release(); hitF.release(); linStage.release(); groupEnv.release();
    groupLights.release(); bvhs.release(); dobjects.release(); materials.release(); dlights.release();
    scratch64.release(); counters.release(); hitI.release();
    slot.release();
    if (finished) cudaEventDestroy(finished);
    if (queryDone) cudaEventDestroy(queryDone);
}

// =========================================================== C ABI ====
extern "C" {

const char* cgs_status_string(int s)
{
    switch (s)
    {
    case CGS_OK: return "ok";
    case CGS_ERR_INVALID_ARGUMENT: return "invalid argument";
    case CGS_ERR_CUDA: return "CUDA error";
    case CGS_ERR_OUT_OF_MEMORY: return "out of device memory";
    case CGS_ERR_NOT_BUILT: return "scene not built";
    case CGS_ERR_HASH_BUCKET_OVERFLOW: return "perfect hash: more than 4 keys in a displacement bucket";
    case CGS_ERR_HASH_FAILED: return "perfect hash: no injective table in 16 trials";
    case CGS_ERR_EMPTY_LEAF: return "BVH: empty leaf";
    case CGS_ERR_BUSY: return "render still in flight";
    case CGS_ERR_DEVICE_LIMIT: return "a kernel hit a stack or iteration limit";
    case CGS_ERR_ADMISSION: return "request exceeds the device-memory budget";
    case CGS_ERR_NOT_FOUND: return "not found";
    case CGS_ERR_CAPACITY: return "input exceeds the fixed capacity of this entry point";
    default: return "unknown status";
    }
}

int cgs_version(void) { return 2; }

int cgs_scene_create(cgs_scene** out, int device)
{
    if (!out) return CGS_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) return CGS_ERR_CUDA;
    CGS_TRY(cudaSetDevice(device));
    auto* s = new (std::nothrow) cgs_scene();
    if (!s) return CGS_ERR_OUT_OF_MEMORY;
    s->device = device;
    s->groups.emplace_back();
    if (cudaEventCreateWithFlags(&s->finished, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&s->queryDone, cudaEventDisableTiming) != cudaSuccess)
    {
        delete s;
        return CGS_ERR_CUDA;
    }
    *out = s;
    return CGS_OK;
}

int cgs_scene_destroy(cgs_scene* s)
{
    if (!s) return CGS_ERR_INVALID_ARGUMENT;
    cudaSetDevice(s->device);
    cudaDeviceSynchronize();
    delete s;
    return CGS_OK;
}

int cgs_scene_add_surface(cgs_scene* s, const float* pts, uint32_t npoints, const uint32_t* idx, uint32_t nidx,
                          uint32_t* sid)
{
    if (!s || !pts || !idx || nidx == 0 || nidx % 16 || npoints == 0) return CGS_ERR_INVALID_ARGUMENT;
    for (uint32_t i = 0; i < nidx; i++) if (idx[i] >= npoints) return CGS_ERR_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> g(s->mu);
    Surface sf;
    sf.points.assign(pts, pts + 4ull * npoints);
    sf.indices.assign(idx, idx + nidx);
    s->surfaces.push_back(std::move(sf));
    s->bvhBuilt = s->uploaded = s->hashed = false;
    if (sid) *sid = uint32_t(s->surfaces.size() - 1);
    return CGS_OK;
}

int cgs_scene_add_group(cgs_scene* s, uint32_t* gid)
{
    if (!s) return CGS_ERR_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> g(s->mu);
    if (current_group(s).touched)
    {
        s->groups.emplace_back();
        s->current = uint32_t(s->groups.size() - 1);
        s->bvhBuilt = s->uploaded = s->hashed = false;
    }
    if (gid) *gid = s->current;
    return CGS_OK;
}

int cgs_scene_add_object(cgs_scene* s, uint32_t surface, const float l2w[16], const float w2l[16],
                         const cgs_material* material, const uint32_t* pm, const cgs_material* mats, uint32_t nm,
                         uint32_t* oid)
{
    if (!s || !l2w || !w2l || !material) return CGS_ERR_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> g(s->mu);
    if (surface >= s->surfaces.size()) return CGS_ERR_INVALID_ARGUMENT;
    Object ob;
    ob.surface = surface;
    ob.group = s->current;
    std::memcpy(ob.l2w, l2w, sizeof ob.l2w);
    std::memcpy(ob.w2l, w2l, sizeof ob.w2l);
    ob.material = *material;
    if (pm)
    {
        if (!mats || nm == 0) return CGS_ERR_INVALID_ARGUMENT;
        uint32_t P = s->surfaces[surface].patchCount();
        ob.patchMaterial.assign(pm, pm + P);
        for (uint32_t v : ob.patchMaterial) if (v >= nm) return CGS_ERR_INVALID_ARGUMENT;
        ob.materials.assign(mats, mats + nm);
    }
    s->objects.push_back(std::move(ob));
    current_group(s).objects.push_back(uint32_t(s->objects.size() - 1));
    current_group(s).touched = true;
    s->bvhBuilt = s->uploaded = s->hashed = false;
    if (oid) *oid = uint32_t(s->objects.size() - 1);
    return CGS_OK;
}

int cgs_scene_set_lights(cgs_scene* s, const cgs_light* lights, uint32_t n)
{
    if (!s || (n && !lights)) return CGS_ERR_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> g(s->mu);
    current_group(s).lights.assign(lights, lights + n);
    current_group(s).touched = true;
    if (!s->uploaded) return CGS_OK;
    CGS_TRY(cudaSetDevice(s->device));
    return upload_lights(s);
}

int cgs_scene_set_environment(cgs_scene* s, const float bg[3], const float amb[3])
{
    if (!s || !bg || !amb) return CGS_ERR_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> g(s->mu);
    Group& gr = current_group(s);
    for (int k = 0; k < 3; k++) { gr.background[k] = bg[k]; gr.ambient[k] = amb[k]; }
    gr.touched = true;
    if (!s->uploaded) return CGS_OK;
    CGS_TRY(cudaSetDevice(s->device));
    return upload_lights(s);
}

int cgs_scene_set_bvh_split(cgs_scene* s, int mode)
{
    if (!s || (mode != CGS_SPLIT_REFERENCE && mode != CGS_SPLIT_LONGEST && mode != CGS_SPLIT_MIRROR))
        return CGS_ERR_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> g(s->mu);
    if (s->splitMode != mode) s->bvhBuilt = s->uploaded = s->hashed = false;
    s->splitMode = mode;
    return CGS_OK;
}

int cgs_bvh_build(cgs_scene* s)
{
    if (!s) return CGS_ERR_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> g(s->mu);
    if (s->objects.empty()) return CGS_ERR_INVALID_ARGUMENT;
    for (const Group& gr : s->groups)
        if (gr.objects.empty()) return CGS_ERR_EMPTY_LEAF;
    // the surfaces' BVHs and walk trees and the objects' bounds are independent:
    // built on all host cores, largest first, each by one thread (the same
    // result as in order); then the groups' BVHs over the bounds
    const size_t ns = s->surfaces.size(), no = s->objects.size(), ng = s->groups.size();
    const bool walk = s->splitMode == CGS_SPLIT_REFERENCE;
    // a mirrored store traverses the longest-axis build
    const int mode = s->splitMode == CGS_SPLIT_MIRROR ? CGS_SPLIT_LONGEST : s->splitMode;
    std::vector<std::pair<uint64_t, size_t>> work;
    uint64_t all = 0;
    for (size_t i = 0; i < ns; i++)
    {
        const uint64_t cost = 4ull * s->surfaces[i].patchCount();
        work.push_back({cost, i});
        if (walk) work.push_back({cost, ns + i});
        s->surfaces[i].walk = HostBVH {};
        all += cost;
    }
    for (size_t o = 0; o < no; o++)
        work.push_back({s->surfaces[s->objects[o].surface].patchCount(), 2 * ns + o});
    std::sort(work.begin(), work.end(), [](const auto& a, const auto& b) { return a.first > b.first; });
    std::vector<Box> bounds(no);
    on_host_cores(work.size(), all > 1000, [&](size_t w) {
        const size_t i = work[w].second;
        if (i < ns)
        {
            s->surfaces[i].bvh.split_mode = mode;
            build_surface_bvh(s->surfaces[i], s->surfaces[i].bvh);
        }
        else if (i < 2 * ns) build_walk_bvh(s->surfaces[i - ns], s->surfaces[i - ns].walk);
        else bounds[i - 2 * ns] = object_bounds(s, s->objects[i - 2 * ns]);
    });
    on_host_cores(ng, ng > 64, [&](size_t g) {
        s->groups[g].top.split_mode = mode;
        build_group_bvh(s->groups[g], bounds, s->groups[g].top);
    });
    for (auto& sf : s->surfaces)
        if (sf.bvh.emptyLeaf) return CGS_ERR_EMPTY_LEAF;
    for (auto& gr : s->groups)
        if (gr.top.emptyLeaf) return CGS_ERR_EMPTY_LEAF;
    s->bvhBuilt = true;
    s->uploaded = s->hashed = false;
    return CGS_OK;
}

int cgs_hash_build(cgs_scene* s, void* stream)
{
    if (!s) return CGS_ERR_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> g(s->mu);
    if (!s->bvhBuilt) return CGS_ERR_NOT_BUILT;
    CGS_TRY(cudaSetDevice(s->device));
    if (!s->uploaded)
    {
        int r = upload(s);
        if (r) return r;
    }
    return hash_all(s, (cudaStream_t)stream);
}

int cgs_scene_build(cgs_scene* s, void* stream)
{
    int r = cgs_bvh_build(s);
    if (r) return r;
    return cgs_hash_build(s, stream);
}

int cgs_scene_footprint(const cgs_scene* s, uint64_t* bytes)
{
    if (!s || !bytes) return CGS_ERR_INVALID_ARGUMENT;
    uint64_t b = 0;
    b += s->patches.bytes() + s->nodes.bytes() + s->qnodes.bytes() + s->indices.bytes() + s->tables.bytes() + s->disps.bytes();
    b += s->patchBase.bytes() + s->patchMaterial.bytes() + s->bvhs.bytes() + s->dobjects.bytes();
    b += s->materials.bytes() + s->dlights.bytes() + s->groupTop.bytes() + s->groupLights.bytes();
    b += s->groupEnv.bytes() + s->leafKeys.bytes();
    *bytes = b;
    return CGS_OK;
}

int cgs_bvh_sizes(const cgs_scene* s, int32_t which, uint32_t sizes[5])
{
    if (!s || !sizes) return CGS_ERR_INVALID_ARGUMENT;
    if (!s->bvhBuilt) return CGS_ERR_NOT_BUILT;
    uint32_t k;
    if (!bvh_index(s, which, k)) return CGS_ERR_INVALID_ARGUMENT;
    if (s->splitMode == CGS_SPLIT_MIRROR)
    {
        HostBVH ref;
        std::vector<uint32_t> table, disp;
        uint32_t params[4];
        if (int r = mirror_export(s, k, ref, table, disp, params)) return r;
        sizes[0] = uint32_t(ref.nodes.size());
        sizes[1] = uint32_t(ref.indices.size());
        sizes[2] = params[2];
        sizes[3] = displ_size(uint32_t(ref.keys.size()));
        sizes[4] = uint32_t(ref.keys.size());
        return CGS_OK;
    }
    const HostBVH& b = s->bvh(k);
    sizes[0] = uint32_t(b.nodes.size());
    sizes[1] = uint32_t(b.indices.size());
    sizes[2] = s->hashed ? s->hbvh[k].N : 0;
    sizes[3] = displ_size(uint32_t(b.keys.size()));
    sizes[4] = uint32_t(b.keys.size());
    return CGS_OK;
}

int cgs_bvh_export(const cgs_scene* s, int32_t which, uint32_t* nodes, uint32_t* keys, uint32_t* indices,
                   uint32_t* table, uint32_t* disp, uint32_t params[4])
{
    if (!s) return CGS_ERR_INVALID_ARGUMENT;
    if (!s->bvhBuilt) return CGS_ERR_NOT_BUILT;
    uint32_t k;
    if (!bvh_index(s, which, k)) return CGS_ERR_INVALID_ARGUMENT;
    HostBVH ref;
    std::vector<uint32_t> mtable, mdisp;
    uint32_t mparams[4] = {};
    const bool mirror = s->splitMode == CGS_SPLIT_MIRROR;
    if (mirror)
        if (int r = mirror_export(s, k, ref, mtable, mdisp, mparams)) return r;
    const HostBVH& b = mirror ? ref : s->bvh(k);
    if (nodes)
        for (size_t i = 0; i < b.nodes.size(); i++)
        {
            const Node& n = b.nodes[i];
            float f[12] = {n.leftBox.lo[0], n.leftBox.lo[1], n.leftBox.lo[2], n.leftBox.hi[0], n.leftBox.hi[1],
                           n.leftBox.hi[2], n.rightBox.lo[0], n.rightBox.lo[1], n.rightBox.lo[2], n.rightBox.hi[0],
                           n.rightBox.hi[1], n.rightBox.hi[2]};
            std::memcpy(nodes + 14 * i, f, sizeof f);
            nodes[14 * i + 12] = n.left;
            nodes[14 * i + 13] = n.right;
        }
    if (keys) std::copy(b.keys.begin(), b.keys.end(), keys);
    if (indices) std::copy(b.indices.begin(), b.indices.end(), indices);
    if (mirror)
    {
        if (s->hashed && table) std::copy(mtable.begin(), mtable.end(), table);
        if (s->hashed && disp) std::copy(mdisp.begin(), mdisp.end(), disp);
        if (params) std::copy(mparams, mparams + 4, params);
    }
    else if (s->hashed)
    {
        CGS_TRY(cudaSetDevice(s->device));
        const DevBVH& d = s->hbvh[k];
        if (table) CGS_TRY(cudaMemcpy(table, s->tables.p + d.tableBase, d.N * sizeof(uint32_t), cudaMemcpyDeviceToHost));
        if (disp) CGS_TRY(cudaMemcpy(disp, s->disps.p + d.dispBase, (d.mask + 1) * sizeof(uint32_t), cudaMemcpyDeviceToHost));
        if (params) { params[0] = d.A; params[1] = d.B; params[2] = d.N; params[3] = d.mask; }
    }
    else if (params)
        params[0] = params[1] = params[2] = params[3] = 0;
    return CGS_OK;
}

int cgs_scene_counters(cgs_scene* s, cgs_counters* out)
{
    if (!s || !out) return CGS_ERR_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> g(s->mu);
    std::memset(out, 0, sizeof *out);
    if (!s->lastCounters) return CGS_OK;
    CGS_TRY(cudaSetDevice(s->device));
    CGS_TRY(cudaStreamSynchronize(s->lastStream));
    Counters c;
    CGS_TRY(cudaMemcpy(&c, s->lastCounters, sizeof c, cudaMemcpyDeviceToHost));
    out->rays = c.rays; out->nodes = c.nodes; out->hash_lookups = c.hashLookups; out->candidates = c.candidates;
    out->iterations = c.iterations; out->device_errors = c.errors; out->kernel_launches = uint64_t(s->launches);
    out->hash_table_reads = c.tableReads;
    return CGS_OK;
}

}  // extern "C"
