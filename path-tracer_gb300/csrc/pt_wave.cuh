// pt_wave.cuh - device building blocks shared by the wavefront kernels of one
// tile (trace_wavefront.cu) and of many jobs (batch.cu): the derived BVH and
// triangle layouts, the queue view, the per-lane traversal state machine and
// warp-aggregated queue appends.
#pragma once

#include <map>
#include <mutex>
#include <type_traits>
#include <utility>

#include "pt_path.cuh"

namespace ptd {

struct Fast {
    const float4* pairs;  // the binary nodes: node i at pairs[2i], pairs[2i+1] (32-byte aligned)
    const float4* packed = nullptr;  // the packed BVH (see PackedRay); null: the scene has none
    const float4* tri4;   // triangle i at tri4[kTriStride i .. kTriStride i + 2] (padded to 48 or 64 bytes)
    const float4* wide = nullptr;  // pt_wide_node i at wide[8i .. 8i+7] (precision form)
    const uint32_t* parent = nullptr;   // binary node -> its parent (root: 0xffffffff)
    const uint32_t* leaf_of = nullptr;  // triangle -> the binary leaf holding it
};


struct Queues {
    float4* o[2];
    float4* d[2];
    float4* T[2];
    float4* hit;
    float4* color;
    float4* so;
    float4* sd;
    float4* sc;
    uint32_t* hit_list;   // slots of the current queue whose ray hit a triangle
    uint32_t* miss_list;  // slots whose ray left the scene
    uint32_t* hit_sorted = nullptr;  // the hit list sorted by key (when the round's kCntSorted != 0)
    // beside the hit list, each filed hit's triangle-bucket sort key (triangle
    // >> key_shift, at most the last bucket), written by the trace kernel so
    // that the sort reads its keys in order instead of gathering the hit
    // records; null: the sort computes the keys itself
    uint32_t* hit_keys = nullptr;
    uint32_t key_shift = 0;
    uint32_t* cnt;  // the counters of every round: kRoundCounters words each, all zeroed before the first
    Counters* rec;  // per path (recording variants)
    int32_t* rec_hits;
};

// The counters of one round (bounce).  Each round has its own, so that no
// launch is needed to clear them between rounds.
constexpr uint32_t kRoundCounters = 8;
constexpr uint32_t kCntRays = 0;         // rays of the round
constexpr uint32_t kCntShadows = 1;      // shadow rays that the shading of the round before queued
constexpr uint32_t kCntFetch = 2;        // rays taken; the next two are filed with the same atomic instruction
constexpr uint32_t kCntHits = 3;         // hit list length
constexpr uint32_t kCntMisses = 4;       // miss list length
constexpr uint32_t kCntShadowFetch = 5;  // shadow rays taken
constexpr uint32_t kCntSorted = 6;       // 1: hit_sorted holds the round's hits
constexpr uint32_t kCntTail = 7;         // hits taken by finish_paths beyond those dealt
// rounds 0 .. max_bounces, and the empty one after the last
constexpr uint32_t kCounterWords = kRoundCounters * (PT_MAX_BOUNCES_LIMIT + 2u);
PTD uint32_t* round_counters(const Queues& q, uint32_t round) { return q.cnt + kRoundCounters * round; }

// the ray queues a round reads and writes (they alternate)
struct Stage {
    float4* o;  // current ray queue
    float4* d;
    float4* T;
    float4* no;  // next ray queue
    float4* nd;
    float4* nT;
};

PTD Stage stage_of(const Queues& q, uint32_t round) {
    const bool odd = (round & 1u) != 0u;
    Stage s;
    s.o = odd ? q.o[1] : q.o[0];
    s.d = odd ? q.d[1] : q.d[0];
    s.T = odd ? q.T[1] : q.T[0];
    s.no = odd ? q.o[0] : q.o[1];
    s.nd = odd ? q.d[0] : q.d[1];
    s.nT = odd ? q.T[0] : q.T[1];
    return s;
}

// Waits until the launch before this one in its stream has finished, when it
// was launched with programmatic stream serialization (else it has already).
PTD void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// launch shapes (overridable at build time for tuning sweeps)
#ifndef PT_EXTEND_THREADS
#define PT_EXTEND_THREADS 128
#endif
// 9 resident blocks of the traversal kernels per SM: 56 registers (the packed
// traversal spills 60 bytes stored, 36 loaded a thread for it, the engine's 80 and
// 40; with 8 blocks of 64 registers it is slower, see PackedRay)
#ifndef PT_EXTEND_MIN_BLOCKS
#define PT_EXTEND_MIN_BLOCKS 9
#endif
// the shading kernel: one resident block of 1024 per SM, at most 64
// registers.  Its grid-stride loop hands consecutive slots of the (sorted)
// hit list to consecutive warps, so a block of 1024 keeps 1024 neighbouring
// hits - the same triangles, attributes and materials - in one SM's L1:
// measured 14 % less shading time than 8 blocks of 128 with the same
// registers
#ifndef PT_SHADE_THREADS
#define PT_SHADE_THREADS 1024
#endif
#ifndef PT_SHADE_MIN_BLOCKS
#define PT_SHADE_MIN_BLOCKS 1
#endif
// node visits of a traversal warp between two looks at its idle lanes, at most
#ifndef PT_STEPS_PER_REFILL
#define PT_STEPS_PER_REFILL 32
#endif
// binary subtrees of at most this many triangles become one leaf of the 8-wide BVH
#ifndef PT_WIDE_LEAF_MERGE
#define PT_WIDE_LEAF_MERGE 0
#endif
constexpr uint32_t kWideLeafMerge = PT_WIDE_LEAF_MERGE;
// 1: the accepted children are collected in slot order and the 8-bit mask is
// permuted to octant order once per node; 0: each child sets its octant-order
// bit directly
#ifndef PT_WIDE_MASK_PERMUTE
#define PT_WIDE_MASK_PERMUTE 1
#endif
// resident blocks per SM the 8-wide traversal kernels are compiled for
#ifndef PT_WIDE_MIN_BLOCKS
#define PT_WIDE_MIN_BLOCKS 8
#endif
// 1: a pixel's samples are consecutive paths of a group / work item
// (camera rays of a warp share their first nodes); 0: sample-major
#ifndef PT_PIXEL_MAJOR
#define PT_PIXEL_MAJOR 1
#endif
constexpr int kExtendThreads = PT_EXTEND_THREADS;
constexpr int kShadeThreads = PT_SHADE_THREADS;
constexpr int kTailThreads = 512;  // one block per SM, 4 warps a scheduler (see finish_paths)
constexpr uint32_t kTailSmemStack = 5;  // its packed stacks' shared entries: 40 KB (3 and 8: the same times)
// entries at the top of each traversal lane's stack kept in shared memory
#ifndef PT_SMEM_STACK
#define PT_SMEM_STACK 8
#endif
constexpr uint32_t kSmemStack = PT_SMEM_STACK;
// the same for the packed traversal (16 bytes an entry)
#ifndef PT_PACKED_SMEM_STACK
#define PT_PACKED_SMEM_STACK 8
#endif
constexpr uint32_t kPackedSmemStack = PT_PACKED_SMEM_STACK;
// the same for the 8-wide traversal kernels
#ifndef PT_WIDE_SMEM_STACK
#define PT_WIDE_SMEM_STACK 8
#endif
constexpr uint32_t kWideSmemStack = PT_WIDE_SMEM_STACK;

// The deferred stack of one traversal lane: 64 entries, the first kShared of
// them in the block's shared memory (one column per thread, so a warp touches
// consecutive words), the others in the lane's local memory.
template <uint32_t kThreads, uint32_t kShared>
struct LaneStack {
    uint2* col;  // &shared[threadIdx.x]; entry i < kShared at col[i * kThreads]
    uint2 deep[64];
    PTD void put(uint32_t i, uint2 e) {
        if (i < kShared)
            col[i * kThreads] = e;
        else
            deep[i & 63u] = e;
    }
    PTD uint2 get(uint32_t i) const {
        if (i < kShared) return col[i * kThreads];
        return deep[i & 63u];
    }
};

// the whole stack in local memory
struct LocalStack {
    uint2 deep[64];
    PTD void put(uint32_t i, uint2 e) { deep[i & 63u] = e; }
    PTD uint2 get(uint32_t i) const { return deep[i & 63u]; }
};

// a 32-byte aligned node (or half a triangle) as one 256-bit load
PTD void load_node(const float4* p, float4& lo, float4& hi) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(lo.x), "=f"(lo.y), "=f"(lo.z), "=f"(lo.w), "=f"(hi.x), "=f"(hi.y), "=f"(hi.z), "=f"(hi.w)
        : "l"(p));
}

// float4s per padded triangle: 64 bytes, one 256-bit and one 128-bit load
constexpr uint32_t kTriStride = 4;
PTD Tri load_tri4(const float4* tri4, uint32_t tri) {
    const float4* p = tri4 + kTriStride * (size_t)tri;
    float4 a, b;
    load_node(p, a, b);
    const float4 c = __ldg(p + 2);
    Tri t;
    t.v0 = mk(a.x, a.y, a.z);
    t.v1 = mk(b.x, b.y, b.z);
    t.v2 = mk(c.x, c.y, c.z);
    return t;
}

PTD float box_test(float4 lo, float4 hi, f3 nod, f3 rcp, float hit_t) {
    const float bmin[3] = {lo.x, lo.y, lo.z}, bmax[3] = {hi.x, hi.y, hi.z};
    return intersect_aabb(bmin, bmax, nod, rcp, hit_t);
}

PTD unsigned lane_id() {
    unsigned l;
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(l));
    return l;
}

// The scene a traversal lane reads: one scene for the whole launch ...
struct OneScene {
    const World& world;
    const Fast& fast;
    PTD const World& w() const { return world; }
    PTD const Fast& f() const { return fast; }
    PTD const float4* packed() const { return fast.packed; }
    PTD const float4* wide() const { return fast.wide; }
    PTD const float4* tri4() const { return fast.tri4; }
};
// ... or each lane its own: a table of Record { World w; Fast f; } and the
// lane's index in it, its two hot pointers kept in registers
template <class Record>
struct LaneScene {
    const Record* table;
    uint32_t index;
    const float4 *boxes, *tris;
    PTD const World& w() const { return table[index].w; }
    PTD const Fast& f() const { return table[index].f; }
    PTD const float4* packed() const { return boxes; }
    PTD const float4* wide() const { return boxes; }
    PTD const float4* tri4() const { return tris; }
};

// When a traversal warp turns from node visits to triangle tests (fewer than
// kVisitKeep / 32 of its busy lanes are at a node) and back (at most
// kTestLeave lanes are at a triangle), and when it looks for new rays (at most
// kRefillAt lanes are busy).
#ifndef PT_VISIT_KEEP
#define PT_VISIT_KEEP 16
#endif
#ifndef PT_TEST_LEAVE
#define PT_TEST_LEAVE 4
#endif
#ifndef PT_REFILL_AT
#define PT_REFILL_AT 20
#endif
// two visits between two looks at the warp's lanes: 10.84 against 11.03 ms a 960x540x16 image of 1M triangles
#ifndef PT_VISIT_TWICE
#define PT_VISIT_TWICE 1
#endif
// the 8-wide traversal turns earlier: its visits cost about 100 instructions whatever the lanes
// (1M triangles, 960x540x16: 12.05 ms with 16, 11.84 with 20, 11.78 with 24, 11.81 with 28)
#ifndef PT_WIDE_VISIT_KEEP
#define PT_WIDE_VISIT_KEEP 24
#endif
#ifndef PT_WIDE_TEST_LEAVE
#define PT_WIDE_TEST_LEAVE 0
#endif
#ifndef PT_WIDE_REFILL_AT
#define PT_WIDE_REFILL_AT 20
#endif

// What a lane of the two-word traversals does next, in `todo`: 0 visit an interior node, > 0
// test that many triangles of a leaf, kFinished: the ray's result is there
// and not filed yet, kIdle: no ray.
constexpr int32_t kFinished = -2, kIdle = -1;

// the largest float below t (t > 0), so that `x < t` is `x <= below(t)`;
// -1 for any other t, which no distance above 0 passes
PTD float below(float t) { return t > 0.0f ? __uint_as_float(__float_as_uint(t) - 1u) : -1.0f; }
PTD float above(float t) { return __uint_as_float(__float_as_uint(t) + 1u); }

// the larger, NaN when one of them is
PTD float max_or_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// A box's entry distance, at least 2^-149, NaN when no plane gives a number, and
// exit distance, at most `limit` (see BinaryRay): the box is accepted when
// *t_near <= *t_far.  (Keeping NaN costs trees on the uploaded nodes up to 1.3 %,
// 1280x720x8 of 18k triangles 4.24 -> 4.27 ms, rays along an axis 11.45 -> 11.61;
// kept in the exit distance instead, 4.28 and 11.66.)
PTD void slabs(float4 lo, float4 hi, f3 rcp, f3 nod, float limit, float* t_near, float* t_far) {
    const float t0x = fma_(lo.x, rcp.x, nod.x), t0y = fma_(lo.y, rcp.y, nod.y), t0z = fma_(lo.z, rcp.z, nod.z);
    const float t1x = fma_(hi.x, rcp.x, nod.x), t1y = fma_(hi.y, rcp.y, nod.y), t1z = fma_(hi.z, rcp.z, nod.z);
    *t_near = max_or_nan(0x1p-149f, max3f(fminf(t0x, t1x), fminf(t0y, t1y), fminf(t0z, t1z)));
    *t_far = min3f(fminf(fmaxf(t0x, t1x), limit), fmaxf(t0y, t1y), fmaxf(t0z, t1z));
}

// What a traversal looks for (the template argument kFind): the closest hit
// (trace.slang:764-884), any hit (614-717), or either by the ray: a ray whose
// light_tri is kClosestRay looks for the closest.
constexpr int kFindClosest = 0, kFindAny = 1, kFindEither = 2;
constexpr int32_t kClosestRay = -2;

// One ray's traversal (closest hit or any hit) on the binary nodes as uploaded: visit() one interior node,
// test() one triangle of a leaf; traverse_queue() decides when each runs.
// The deferred stack holds the (left_first, tri_count) of each node, so a pop
// needs no memory access.  A ray's visits and tests happen in exactly the
// reference's order.  The stack lives outside the object so that its scalar
// state can stay in registers.
//
// The slab test of trace.slang:597-609 accepts a box when t_near <= t_far,
// t_far > 0 and t_near < hit_t.  Here that is one comparison,
// max(t_near, 2^-149) <= min(t_far, below(hit_t)): the same for every value
// (2^-149 is the smallest positive float; with hit_t = 2^-149 no triangle can
// be nearer, whatever is visited).  min and max skip NaN, except the last
// max: when no plane of the box gives a number (a box of NaNs, or a ray without
// any extent), t_near stays NaN and the box is rejected, as by the shader.  Of two
// children entered at or before the origin and at exactly 2^-149 the second is
// visited first, as at a tie.
template <bool kRec, bool kAlpha, int kFind, bool kTri36, class Scene>
struct BinaryRay {
    static constexpr int kVisitKeep = PT_VISIT_KEEP, kTestLeave = PT_TEST_LEAVE, kRefillAt = PT_REFILL_AT;
    Scene sc;
    f3 o, rcp, nod;
    Shear s;
    float limit, hv, hw;  // limit: below(hit_t)
    int32_t hit, light_tri, todo;
    uint32_t lf, sp, idx;
    Rng<kRec> rng;
    Counters c;
    Rec<kRec> rec;

    PTD bool any_hit() const { return kFind == kFindAny || (kFind == kFindEither && light_tri != kClosestRay); }
    PTD explicit BinaryRay(Scene scene) : sc(scene), todo(kIdle) {}
    PTD bool busy() const { return todo >= 0; }
    PTD bool at_node() const { return todo == 0; }
    PTD bool at_leaf() const { return todo > 0; }
    PTD bool finished() const { return todo == kFinished; }
    PTD void set_idle() { todo = kIdle; }

    template <class S>
    PTD void init(f3 origin, f3 dir, float t_max, int32_t light, S&) {
        o = origin;
        rcp = mk(ptd::rcp(dir.x), ptd::rcp(dir.y), ptd::rcp(dir.z));
        s = make_shear(dir, rcp);
        nod = -o * rcp;
        limit = below(t_max);
        hv = hw = 0.0f;
        hit = -1;
        light_tri = light;
        sp = 0u;
        idx = 0u;
        lf = __float_as_uint(__ldg(&sc.f().pairs[0].w));
        todo = __float_as_int(__ldg(&sc.f().pairs[1].w));
        if constexpr (kRec) {
            rec.c = &c;
            rng.rec.c = &c;
            if constexpr (kFind == kFindAny) {
                rec.shadow = true;
                c.shadow_rays += 1;
            } else {
                c.extend_rays += 1;
            }
            enter();
        }
    }
    PTD float hit_t() const { return above(limit); }

    // records the visit of the node about to be processed (trace.slang:793, :637)
    PTD void enter() {
        rec.visit(idx);
        if (todo == 0)
            rec.interior();
        else
            rec.leaf();
    }

    template <class S>
    PTD void pop(S& stack, uint32_t* istack) {
        if (sp == 0u) {
            todo = kFinished;
            return;
        }
        sp -= 1u;
        const uint2 e = stack.get(sp);
        lf = e.x;
        todo = (int32_t)e.y;
        if constexpr (kRec) {
            idx = istack[sp & 63u];
            enter();
        }
    }

    template <class S>
    PTD void visit(S& stack, uint32_t* istack) {
        const float4* p = sc.f().pairs + 2 * (size_t)lf;
        float4 l0, l1, r0, r1;
        load_node(p, l0, l1);
        load_node(p + 2, r0, r1);
        float ln, lx, rn, rx;
        slabs(l0, l1, rcp, nod, limit, &ln, &lx);
        slabs(r0, r1, rcp, nod, limit, &rn, &rx);
        const bool hl = ln <= lx, hr = rn <= rx;
        if (!hl && !hr) {
            pop(stack, istack);
            return;
        }
        const bool go_left = hl && (!hr || ln < rn);
        if (hl && hr) {
            stack.put(sp, make_uint2(__float_as_uint(go_left ? r0.w : l0.w), __float_as_uint(go_left ? r1.w : l1.w)));
            if constexpr (kRec) istack[sp & 63u] = go_left ? lf + 1u : lf;
            sp += 1u;
        }
        if constexpr (kRec) idx = go_left ? lf : lf + 1u;
        lf = __float_as_uint(go_left ? l0.w : r0.w);
        todo = __float_as_int(go_left ? l1.w : r1.w);
        if constexpr (kRec) enter();
    }

    template <class S>
    PTD void test(S& stack, uint32_t* istack) {
        const uint32_t tri = lf;
        lf += 1u;
        todo -= 1;
        bool skip = false;
        if constexpr (kFind != kFindClosest) skip = (int32_t)tri == light_tri;
        if (!skip) {
            rec.tri();
            Tri tv;
            if constexpr (kTri36)
                tv = load_tri(sc.w(), tri);  // the caller's 36-byte triangles
            else
                tv = load_tri4(sc.tri4(), tri);
            float t, v, wb;
            if (triangle_test(tv, o, s, &t, &v, &wb) && t > 0.0f && t <= limit) {
                bool counts = true;
                if constexpr (kAlpha) counts = !passes_through(sc.w(), tri, v, wb, rng);
                if (counts) {
                    if (any_hit()) {
                        hit = 1;
                        todo = kFinished;
                        return;
                    } else {
                        limit = below(t);
                        hit = (int32_t)tri;
                        hv = v;
                        hw = wb;
                    }
                }
            }
        }
        if (todo == 0) pop(stack, istack);
    }
};

// ---------------------------------------------------------------- packed BVH
//
// A pair of child boxes in 32 bytes, one load a visit.  The two children of an
// interior node share its planes: on each side of each axis one child (at
// least) has the parent's plane, so the pair needs six new planes and six bits
// that say whose they are.  In a ray's terms a shared plane adds nothing: the
// children's entry distance is the largest of the parent's entry distance and
// those of their own new near planes, and likewise the exit, so the traversal
// carries the node's two distances instead of its box.  The distances are
// those of the uploaded boxes bit for bit (fma is monotonic in the plane, so
// the largest over the three axes does not change when an axis is replaced by
// the parent's smaller or equal value).
//
// Record of the interior node whose children are l and l + 1, at l / 2 (a
// child pair has one parent): three new minima and the left child's
// reference, three new maxima and the right child's reference.  Reference:
// index << 7 | count << 3 | owners; count 0: an interior node, index = its
// record; 1..14: a leaf, index = its first triangle; 15: an interior node
// whose record holds no planes, only l in its first word (boxes that are not
// exactly the union of their children's, planes out of order or not finite,
// even l), visited from the uploaded nodes.  owners, bit a: in the left
// reference, the new minimum of axis a is the right child's (else the left
// child's); in the right reference the same of the new maximum.
// Entry 0 of the array is the root's box and reference; the records follow.
constexpr uint32_t kPackedMaxLeaf = 14, kPackedPlain = 15;
constexpr uint64_t kPackedMaxNodes = 1ull << 26, kPackedMaxTris = 1ull << 25;  // exclusive: all ones is no index
constexpr uint32_t kRefIdle = 0xffffffffu, kRefFinished = 0xfffffffeu;

PTD bool finite3(float4 v) {
    const float inf = __int_as_float(0x7f800000);
    return fabsf(v.x) < inf && fabsf(v.y) < inf && fabsf(v.z) < inf;
}

// node i's children as six new planes and their owners (false: kPackedPlain)
PTD bool pack_planes(const float4* nodes, uint64_t node_count, uint64_t i, float* plane_lo, float* plane_hi,
                     uint32_t* own_lo, uint32_t* own_hi) {
    const float4 p0 = nodes[2 * i], p1 = nodes[2 * i + 1];
    const uint64_t l = __float_as_uint(p0.w);
    if ((l & 1u) == 0u || l + 1u >= node_count) return false;
    const float4 l0 = nodes[2 * l], l1 = nodes[2 * l + 1], r0 = nodes[2 * l + 2], r1 = nodes[2 * l + 3];
    if (!finite3(l0) || !finite3(l1) || !finite3(r0) || !finite3(r1)) return false;
    const float plo[3] = {p0.x, p0.y, p0.z}, phi[3] = {p1.x, p1.y, p1.z};
    const float llo[3] = {l0.x, l0.y, l0.z}, lhi[3] = {l1.x, l1.y, l1.z};
    const float rlo[3] = {r0.x, r0.y, r0.z}, rhi[3] = {r1.x, r1.y, r1.z};
    *own_lo = *own_hi = 0u;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (!(llo[a] <= lhi[a]) || !(rlo[a] <= rhi[a])) return false;
        if (plo[a] != fminf(llo[a], rlo[a]) || phi[a] != fmaxf(lhi[a], rhi[a])) return false;
        const bool lo_right = llo[a] == plo[a], hi_right = lhi[a] == phi[a];
        plane_lo[a] = lo_right ? rlo[a] : llo[a];
        plane_hi[a] = hi_right ? rhi[a] : lhi[a];
        *own_lo |= (lo_right ? 1u : 0u) << a;
        *own_hi |= (hi_right ? 1u : 0u) << a;
    }
    return true;
}

// reference to node i
PTD uint32_t pack_ref(const float4* nodes, uint64_t node_count, uint64_t i) {
    const uint32_t first = __float_as_uint(nodes[2 * i].w), count = __float_as_uint(nodes[2 * i + 1].w);
    if (count > 0u) return (first << 7) | (count << 3);
    float lo[3], hi[3];
    uint32_t a, b;
    return ((first >> 1) << 7) | (pack_planes(nodes, node_count, i, lo, hi, &a, &b) ? 0u : kPackedPlain << 3);
}

// One thread per node of a tree in which every node is reachable, with at most
// kPackedMaxLeaf triangles a leaf.  (A template, so that both translation
// units may include it.)
template <int kUnused>
__global__ void __launch_bounds__(256) pack_bvh_kernel(const float4* nodes, uint64_t node_count, float4* packed) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= node_count) return;
    if (i == 0u) {
        const float4 a = nodes[0], b = nodes[1];
        packed[0] = make_float4(a.x, a.y, a.z, __uint_as_float(pack_ref(nodes, node_count, 0u)));
        packed[1] = make_float4(b.x, b.y, b.z, 0.0f);
    }
    if (__float_as_uint(nodes[2 * i + 1].w) > 0u) return;
    const uint32_t l = __float_as_uint(nodes[2 * i].w);
    if ((uint64_t)l + 1u >= node_count) return;
    float lo[3] = {__uint_as_float(l), 0.0f, 0.0f}, hi[3] = {0.0f, 0.0f, 0.0f};
    uint32_t own_lo = 0u, own_hi = 0u;
    if (!pack_planes(nodes, node_count, i, lo, hi, &own_lo, &own_hi)) {
        lo[0] = __uint_as_float(l);
        own_lo = own_hi = 0u;
    }
    float4* r = packed + 2 + 2 * (size_t)(l >> 1);
    r[0] = make_float4(lo[0], lo[1], lo[2], __uint_as_float(pack_ref(nodes, node_count, l) | own_lo));
    r[1] = make_float4(hi[0], hi[1], hi[2], __uint_as_float(pack_ref(nodes, node_count, l + 1u) | own_hi));
}

// Adds to *plain (in host memory or on the device) the interior nodes that would
// be records without planes; the nodes may be anything.
template <int kUnused>
__global__ void __launch_bounds__(256) count_plain_kernel(const float4* nodes, uint64_t node_count, uint32_t* plain) {
    __shared__ uint32_t sum;
    if (threadIdx.x == 0u) sum = 0u;
    __syncthreads();
    uint32_t mine = 0u;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < node_count; i += (uint64_t)gridDim.x * blockDim.x) {
        float lo[3], hi[3];
        uint32_t a, b;
        if (__float_as_uint(nodes[2 * i + 1].w) == 0u && !pack_planes(nodes, node_count, i, lo, hi, &a, &b)) mine += 1u;
    }
    if (mine) atomicAdd(&sum, mine);
    __syncthreads();
    if (threadIdx.x == 0u && sum) atomicAdd_system(plain, sum);
}

// bytes of the packed BVH of a tree
constexpr size_t packed_bytes(uint64_t nodes) { return 32 + 32 * (nodes / 2 + 1); }

// v into the left child's distance, or the right child's where `right` is not 0
PTD void route_max(uint32_t right, float v, float& l, float& r) {
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@!p max.f32 %0, %0, %2;\n\t@p max.f32 %1, %1, %2;\n\t}"
        : "+f"(l), "+f"(r)
        : "f"(v), "r"(right));
}
PTD void route_min(uint32_t right, float v, float& l, float& r) {
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@!p min.f32 %0, %0, %2;\n\t@p min.f32 %1, %1, %2;\n\t}"
        : "+f"(l), "+f"(r)
        : "f"(v), "r"(right));
}

// The deferred stack of a packed traversal, 16 bytes an entry (reference,
// entry distance, exit distance): the first kShared entries in shared memory,
// the others in the lane's local memory.  Entry 0 is the end: a popped
// kRefFinished ends the traversal.  Positions are byte offsets in local
// memory (16 an entry).  Everything a visit does with the stack is predicated
// instructions, so that a warp whose lanes push, pop and do neither runs no
// branch for it.
template <uint32_t kThreads, uint32_t kShared>
struct PackedStack {
    static constexpr uint32_t kLast = 16u * (kShared - 1u);  // position of the last shared entry
    uint32_t col;   // shared address of this thread's entry 0; entry i at + i * kThreads * 16
    uint32_t deep;  // local address of entry 0
    float4 entries[66];  // at most 64 deferred nodes (checked at upload) above entry 0
    PTD void bind(const float4* top) {
        // (opaque to the compiler, which otherwise computes the addresses again on every visit)
        asm volatile("mov.u32 %0, %1;" : "=r"(col) : "r"((uint32_t)__cvta_generic_to_shared(top + threadIdx.x)));
        asm volatile("{\n\t.reg .u64 a;\n\tcvta.to.local.u64 a, %1;\n\tcvt.u32.u64 %0, a;\n\t}" : "=r"(deep) : "l"(entries) : "memory");
    }
    PTD void clear() const {
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(col), "r"(kRefFinished) : "memory");
    }
    PTD void pop(uint32_t& sp, uint32_t& ref, float& t_near, float& t_far) const {
        asm volatile(
            "{\n\t.reg .pred s;\n\t.reg .b32 z;\n\tsetp.le.u32 s, %0, %4;\n\t"
            "@s ld.shared.v4.b32 {%1, %2, %3, z}, [%5];\n\t@!s ld.local.v4.b32 {%1, %2, %3, z}, [%6];\n\t"
            "sub.u32 %0, %0, 16;\n\t}"
            : "+r"(sp), "+r"(ref), "+f"(t_near), "+f"(t_far)
            : "n"(kLast), "r"(col + sp * kThreads), "r"(deep + sp)
            : "memory");
    }
    // the end of a visit: on to the nearer accepted child, deferring the other,
    // or to the deferred node at the stack's top
    PTD void descend(uint32_t& sp, uint32_t& ref, float& t_near, float& t_far, uint32_t wl, uint32_t wr, float ln,
                     float lx, float rn, float rx) const {
        asm volatile(
            "{\n\t.reg .pred hl, hr, lt, nr, left, both, any, s, p;\n\t.reg .b32 f0, f1, f2, z;\n\t"
            "setp.le.f32 hl, %6, %7;\n\tsetp.le.f32 hr, %8, %9;\n\tsetp.lt.f32 lt, %6, %8;\n\t"
            "not.pred nr, hr;\n\tor.pred left, nr, lt;\n\tand.pred left, left, hl;\n\t"
            "and.pred both, hl, hr;\n\tor.pred any, hl, hr;\n\t"
            "selp.b32 f0, %5, %4, left;\n\tselp.b32 f1, %8, %6, left;\n\tselp.b32 f2, %9, %7, left;\n\t"
            "setp.lt.and.u32 p, %0, %10, both;\n\t@p st.shared.v4.b32 [%11 + %13], {f0, f1, f2, f0};\n\t"
            "setp.ge.and.u32 p, %0, %10, both;\n\t@p st.local.v4.b32 [%12 + 16], {f0, f1, f2, f0};\n\t"
            "not.pred nr, any;\n\t"
            "setp.le.and.u32 s, %0, %10, nr;\n\t@s ld.shared.v4.b32 {%1, %2, %3, z}, [%11];\n\t"
            "setp.gt.and.u32 s, %0, %10, nr;\n\t@s ld.local.v4.b32 {%1, %2, %3, z}, [%12];\n\t"
            "@any selp.b32 %1, %4, %5, left;\n\t@any selp.b32 %2, %6, %8, left;\n\t@any selp.b32 %3, %7, %9, left;\n\t"
            "@both add.u32 %0, %0, 16;\n\t@nr sub.u32 %0, %0, 16;\n\t}"
            : "+r"(sp), "+r"(ref), "+f"(t_near), "+f"(t_far)
            : "r"(wl), "r"(wr), "f"(ln), "f"(lx), "f"(rn), "f"(rx), "n"(kLast), "r"(col + sp * kThreads),
              "r"(deep + sp), "n"(kThreads * 16u)
            : "memory");
    }
};

// The traversal of BinaryRay on the packed BVH: the same visits and tests in
// the same order.  What it is worth: the uploaded nodes cost two 32-byte loads
// a visit, and a load of 32 scattered lanes is 32 wavefronts of the L1 data
// pipe, which was 79 % busy; here it is 62 %, and the kernel is bound by
// instructions (73 % of the issue slots, ALU pipe 60 %).  The extend launch of
// bounce 1 (1M triangles, 960x540x8): 1.08 ms at first, 1.01 with turns of
// visits and tests, 0.87 packed.  2.1M triangles, 1920x1080x16: extend 31.2 ->
// 25.2 ms, the image 55.2 -> 47.9 ms.  At 56 registers 9 blocks of 128 are
// resident with 8 stack entries in shared memory (16 KB a block); 8 blocks
// with 64 registers: 11.3 against 10.8 ms for a 960x540x16 image of 1M
// triangles, 6 entries: 11.3.  A visit has no branch.  The selection of the near
// and far plane by the ray's direction is done by the multiplier: rp holds the
// positive reciprocals, rn the negative ones, 0 elsewhere, and
// fma(a, rp, fma(b, rn, nod)) is the distance of a or b, with one rounding
// (the other product is an exact 0), which spares the ALU pipe, the busiest
// one (half rate), a select.
template <bool kAlpha, int kFind, class Scene>
struct PackedRay {
    static constexpr int kVisitKeep = PT_VISIT_KEEP, kTestLeave = PT_TEST_LEAVE, kRefillAt = PT_REFILL_AT;
    Scene sc;
    f3 o, rp, rn, nod;
    float limit, hv, hw, tn, tf;  // limit: below(hit_t); tn, tf: the node's entry and exit distances
    int32_t hit, light_tri;
    uint32_t ref, sp;  // sp: position of the stack's top entry
    uint32_t oct;      // bit a: rcp[a] < 0; bits 3..6: visits read the uploaded nodes
    Shear s;
    Rng<false> rng;

    PTD bool any_hit() const { return kFind == kFindAny || (kFind == kFindEither && light_tri != kClosestRay); }
    PTD explicit PackedRay(Scene scene) : sc(scene), ref(kRefIdle) {}
    PTD bool busy() const { return ref < kRefFinished; }
    PTD bool at_node() const { return ((ref | oct) & 0x78u) == 0u; }
    PTD bool at_leaf() const { return ((ref | oct) & 0x78u) != 0u && ref < kRefFinished; }
    PTD bool finished() const { return ref == kRefFinished; }
    PTD void set_idle() { ref = kRefIdle; }
    PTD float hit_t() const { return above(limit); }

    template <class S>
    PTD void init(f3 origin, f3 dir, float t_max, int32_t light, S& stack) {
        o = origin;
        const f3 rcp = mk(ptd::rcp(dir.x), ptd::rcp(dir.y), ptd::rcp(dir.z));
        s = make_shear(dir, rcp);
        nod = -o * rcp;
        rp = mk(rcp.x < 0.0f ? 0.0f : rcp.x, rcp.y < 0.0f ? 0.0f : rcp.y, rcp.z < 0.0f ? 0.0f : rcp.z);
        rn = mk(rcp.x < 0.0f ? rcp.x : 0.0f, rcp.y < 0.0f ? rcp.y : 0.0f, rcp.z < 0.0f ? rcp.z : 0.0f);
        oct = (rcp.x < 0.0f ? 1u : 0u) | (rcp.y < 0.0f ? 2u : 0u) | (rcp.z < 0.0f ? 4u : 0u);
        limit = below(t_max);
        hv = hw = 0.0f;
        hit = -1;
        light_tri = light;
        stack.clear();
        sp = 0u;
        float4 a, b;
        load_node(sc.packed(), a, b);
        ref = __float_as_uint(a.w);
        slabs(a, b, rcp, nod, __int_as_float(0x7f800000), &tn, &tf);
        // an axis without a finite reciprocal (a zero direction component) has no
        // distances that could be carried: such a ray visits the uploaded nodes
        const float inf = __int_as_float(0x7f800000);
        if (!(fabsf(nod.x) < inf && fabsf(nod.y) < inf && fabsf(nod.z) < inf)) oct |= 0x78u;
    }

    template <class S>
    PTD void visit(S& stack, uint32_t*) {
        float4 a, b;
        load_node(sc.packed() + 2 + 2 * (size_t)(ref >> 7), a, b);
        const uint32_t wl = __float_as_uint(a.w), wr = __float_as_uint(b.w);
        // owners of the near and of the far planes
        const uint32_t near_own = (wl & ~oct) | (wr & oct), far_own = (wr & ~oct) | (wl & oct);
        float ln = tn, rn_ = tn, lx = fminf(tf, limit), rx = lx;
        route_max(near_own & 1u, fma_(a.x, rp.x, fma_(b.x, rn.x, nod.x)), ln, rn_);
        route_max(near_own & 2u, fma_(a.y, rp.y, fma_(b.y, rn.y, nod.y)), ln, rn_);
        route_max(near_own & 4u, fma_(a.z, rp.z, fma_(b.z, rn.z, nod.z)), ln, rn_);
        route_min(far_own & 1u, fma_(b.x, rp.x, fma_(a.x, rn.x, nod.x)), lx, rx);
        route_min(far_own & 2u, fma_(b.y, rp.y, fma_(a.y, rn.y, nod.y)), lx, rx);
        route_min(far_own & 4u, fma_(b.z, rp.z, fma_(a.z, rn.z, nod.z)), lx, rx);
        stack.descend(sp, ref, tn, tf, wl, wr, ln, lx, rn_, rx);
    }

    // a visit from the uploaded boxes of the two children
    template <class S>
    PTD void visit_plain(S& stack) {
        const float4* r = sc.packed() + 2 + 2 * (size_t)(ref >> 7);
        uint32_t l = 2u * (ref >> 7) + 1u;
        if ((ref & 0x78u) != 0u) l = __float_as_uint(__ldg(&r[0].x));
        const uint32_t wl = __float_as_uint(__ldg(&r[0].w)), wr = __float_as_uint(__ldg(&r[1].w));
        const float4* p = sc.f().pairs + 2 * (size_t)l;
        float4 l0, l1, r0, r1;
        load_node(p, l0, l1);
        load_node(p + 2, r0, r1);
        const f3 rcp = rp + rn;
        float ln, lx, rn_, rx;
        slabs(l0, l1, rcp, nod, limit, &ln, &lx);
        slabs(r0, r1, rcp, nod, limit, &rn_, &rx);
        stack.descend(sp, ref, tn, tf, wl, wr, ln, lx, rn_, rx);
    }

    // One triangle of the leaf, or a plain visit.  A ray whose every visit is
    // plain runs to its end here: such a ray (an axis-parallel one) can meet
    // thousands of boxes, because its zero axis rejects none, and would hold up
    // the launch's end if each visit waited for a turn of the warp (2.1M
    // triangles, 1344x756x16, camera rays: extend 14.0 ms in turns).
    template <class S>
    PTD void test(S& stack, uint32_t*) {
        do {
            const uint32_t count = (ref >> 3) & 15u;
            if (count == 0u || count == kPackedPlain) {
                visit_plain(stack);
                continue;
            }
            const uint32_t tri = ref >> 7;
            ref += (1u << 7) - (1u << 3);  // the next triangle, one fewer left
            float t, v, wb;
            if (!(kFind != kFindClosest && (int32_t)tri == light_tri) &&
                triangle_test(load_tri4(sc.tri4(), tri), o, s, &t, &v, &wb) && t > 0.0f && t <= limit) {
                bool counts = true;
                if constexpr (kAlpha) counts = !passes_through(sc.w(), tri, v, wb, rng);
                if (counts) {
                    if (any_hit()) {
                        hit = 1;
                        ref = kRefFinished;
                        return;
                    } else {
                        limit = below(t);
                        hit = (int32_t)tri;
                        hv = v;
                        hw = wb;
                    }
                }
            }
            if (count == 1u) stack.pop(sp, ref, tn, tf);
        } while ((oct & 0x78u) != 0u && busy());
    }
};

// Whether the reference's binary traversal (trace.slang:786-884) reaches
// triangle a before triangle b on this ray: in one leaf the lower index
// first; otherwise at their lowest common ancestor the child the traversal
// enters first (the nearer accepted child box, ties to the right).  Used
// only to break exact-t ties the way the reference does (its `t < hit_t`
// keeps the first triangle found).
PTD bool binary_first(const Fast& f, f3 o, f3 d, uint32_t a, uint32_t b) {
    uint32_t la = __ldg(f.leaf_of + a), lb = __ldg(f.leaf_of + b);
    if (la == lb) return a < b;
    const auto depth = [&](uint32_t n) {
        uint32_t k = 0;
        while (n != 0u && k < 64u) {
            n = __ldg(f.parent + n);
            ++k;
        }
        return k;
    };
    uint32_t da = depth(la), db = depth(lb);
    for (; da > db; --da) la = __ldg(f.parent + la);
    for (; db > da; --db) lb = __ldg(f.parent + lb);
    for (uint32_t k = 0; k < 64u; ++k) {
        const uint32_t pa = __ldg(f.parent + la), pb = __ldg(f.parent + lb);
        if (pa == pb) break;
        la = pa;
        lb = pb;
    }
    // la, lb: the two children of the common ancestor, la on a's side
    const uint32_t left = la < lb ? la : lb;
    const f3 rcp = 1.0f / d, nod = -o * rcp;
    const float4* p = f.pairs + 2 * (size_t)left;
    const float inf = __int_as_float(0x7f800000);
    const float dl = box_test(__ldg(p), __ldg(p + 1), nod, rcp, inf);
    const float dr = box_test(__ldg(p + 2), __ldg(p + 3), nod, rcp, inf);
    const bool hl = dl >= 0.0f, hr = dr >= 0.0f;
    const bool go_left = hl && (!hr || dl < dr);
    return (la == left) == go_left;
}

// One ray's traversal of the 8-wide BVH of the precision form
// (include/pt_precision.h), with the interface of BinaryRay: visit() takes a
// node's next child, test() one triangle.  A visit decodes the node's child boxes exactly as the host
// quantised them (origin + q * 2^e: the product exact, one rounding) and runs
// the reference's slab test (trace.slang:597-609) on them; an axis whose
// direction component is zero constrains nothing (the binary test's value is
// then not a bound: 0 * inf).  The accepted children are visited in the
// order of their slots XOR the ray's direction octant (the builder places
// them for that order); the deferred stack holds (node, children still to visit), one
// entry per level.  A leaf's triangles are tested with the reference's
// watertight test, so a hit's (t, v, w) are the binary traversal's for the
// same triangle.  Opaque scenes only.
// One axis of a wide node in the ray's frame.  A child bound q (8 bits) is
// placed into the float v = 1 + q 2^-15 with one byte permute, and its slab
// distance is t = fma(v, a15, c): a15 = 2^(e+15) rcp and c = B - a15 with
// B = fma(origin, rcp, -o rcp), so t = B + q 2^e rcp up to rounding.  The
// near bound (the box minimum when rcp >= 0, else the maximum) uses
// c - eps, the far bound c + eps, with eps = 2^-19 (|B| + |a15| + |o rcp|):
// more than the sum of the rounding errors of this form, of the
// reference's slab test on the binary box (trace.slang:597-609), and of the
// box decode (each at most a few units of 2^-24 of those magnitudes).  So the
// wide interval contains the interval the reference computes for every
// binary node under the child, and a box the reference accepts is accepted.
// An axis the ray does not move along (rcp = 0 here) constrains nothing.
// (The near and far distance of a child as one packed fma measured slower:
// 1920x1080x64 of 2.1M triangles 1514 against 1535 Mrays/s, for its registers.)
struct AxisFrame {
    float a15, c_near, c_far;
    uint32_t near0, near1, far0, far1;  // bound bytes of children 0-3 / 4-7
};
PTD AxisFrame axis_frame(float origin, uint32_t ebyte, float rcp_a, float nod_a, uint32_t lo0, uint32_t lo1,
                         uint32_t hi0, uint32_t hi1) {
    AxisFrame f;
    const bool neg = rcp_a < 0.0f;
    f.near0 = neg ? hi0 : lo0;
    f.near1 = neg ? hi1 : lo1;
    f.far0 = neg ? lo0 : hi0;
    f.far1 = neg ? lo1 : hi1;
    if (rcp_a == 0.0f) {
        const float inf = __int_as_float(0x7f800000);
        f.a15 = 0.0f;
        f.c_near = -inf;
        f.c_far = inf;
        return f;
    }
    const float s15 = __uint_as_float((ebyte + 15u) << 23);  // 2^(e + 15)
    f.a15 = s15 * rcp_a;
    const float b = fmaf(origin, rcp_a, nod_a);
    const float c0 = b - f.a15;
    const float eps = (fabsf(b) + fabsf(f.a15) + fabsf(nod_a)) * 0x1p-19f;
    f.c_near = c0 - eps;
    f.c_far = c0 + eps;
    return f;
}
// v = 1 + q 2^-15 for the bound byte of child i (bytes: 0, q, 0x80, 0x3F)
template <int i>
PTD float bound_v(uint32_t w0, uint32_t w1) {
    return __uint_as_float(__byte_perm(i < 4 ? w0 : w1, 0x3F800000u, 0x7604u | ((unsigned)(i & 3) << 4)));
}

template <int kFind, class Scene>
struct WideRay {
    static constexpr int kVisitKeep = PT_WIDE_VISIT_KEEP, kTestLeave = PT_WIDE_TEST_LEAVE, kRefillAt = PT_WIDE_REFILL_AT;
    Scene sc;
    f3 o, d, rcp, nod;
    Shear s;
    float limit, hv, hw;  // limit: the closest hit's t so far
    int32_t hit, light_tri, todo;  // todo: 0 take the next child of `node`, > 0 triangles of a leaf left to test
    // list: the accepted children still to visit in the current node as a mask
    // in bits 0..7, and the ray's direction octant, bit a set when d[a] < 0, in
    // bits 8..10
    uint32_t node, list, lf, sp;
    Rng<false> rng;  // carried through (no alpha draws in the wide form)

    PTD bool any_hit() const { return kFind == kFindAny || (kFind == kFindEither && light_tri != kClosestRay); }
    PTD explicit WideRay(Scene scene) : sc(scene), todo(kIdle) {}
    PTD bool busy() const { return todo >= 0; }
    PTD bool at_node() const { return todo == 0; }
    PTD bool at_leaf() const { return todo > 0; }
    PTD bool finished() const { return todo == kFinished; }
    PTD void set_idle() { todo = kIdle; }
    PTD float hit_t() const { return limit; }

    template <class S>
    PTD void init(f3 origin, f3 dir, float t_max, int32_t light, S&) {
        o = origin;
        d = dir;
        rcp = 1.0f / d;
        s = make_shear(d, rcp);
        nod = -o * rcp;
        // an axis the ray does not move along: the slab test's 0 * inf is not a
        // bound, so the axis is left unconstrained
        const float inf = __int_as_float(0x7f800000);
        if (fabsf(rcp.x) == inf) { rcp.x = 0.0f; nod.x = 0.0f; }
        if (fabsf(rcp.y) == inf) { rcp.y = 0.0f; nod.y = 0.0f; }
        if (fabsf(rcp.z) == inf) { rcp.z = 0.0f; nod.z = 0.0f; }
        limit = t_max;
        hv = hw = 0.0f;
        hit = -1;
        light_tri = light;
        sp = 0u;
        todo = 0;
        node = 0u;
        const uint32_t oct =
            (__float_as_uint(d.x) >> 31) | ((__float_as_uint(d.y) >> 31) << 1) | ((__float_as_uint(d.z) >> 31) << 2);
        list = children(0u, oct) | (oct << 8);
    }

    // the accepted children of node n as a mask: child slot i sets bit i ^ oct,
    // so the lowest set bit is the next child in the octant order.  A child is
    // accepted when max(near bounds, 0) <= min(far bounds, hit_t): every ray
    // the slab test of trace.slang:597-609 accepts on the binary box (plus the
    // boundary cases t_far = 0 and t_near = hit_t, which change no result)
    PTD uint32_t children(uint32_t n, uint32_t oct) const {
        const float4* p = sc.wide() + 8 * (size_t)n;
        float4 h0, h1, h2, h3;
        load_node(p, h0, h1);
        load_node(p + 2, h2, h3);
        const uint32_t meta = __float_as_uint(h0.w);
        const uint32_t count = meta >> 24;
        const AxisFrame X = axis_frame(h0.x, meta & 0xffu, rcp.x, nod.x, __float_as_uint(h1.x), __float_as_uint(h1.y),
                                       __float_as_uint(h2.z), __float_as_uint(h2.w));
        const AxisFrame Y = axis_frame(h0.y, (meta >> 8) & 0xffu, rcp.y, nod.y, __float_as_uint(h1.z),
                                       __float_as_uint(h1.w), __float_as_uint(h3.x), __float_as_uint(h3.y));
        const AxisFrame Z = axis_frame(h0.z, (meta >> 16) & 0xffu, rcp.z, nod.z, __float_as_uint(h2.x),
                                       __float_as_uint(h2.y), __float_as_uint(h3.z), __float_as_uint(h3.w));
        uint32_t mask = 0u;
        const auto child = [&](auto ic) {
            constexpr int i = decltype(ic)::value;
            const float nx = fmaf(bound_v<i>(X.near0, X.near1), X.a15, X.c_near);
            const float ny = fmaf(bound_v<i>(Y.near0, Y.near1), Y.a15, Y.c_near);
            const float nz = fmaf(bound_v<i>(Z.near0, Z.near1), Z.a15, Z.c_near);
            const float fx = fmaf(bound_v<i>(X.far0, X.far1), X.a15, X.c_far);
            const float fy = fmaf(bound_v<i>(Y.far0, Y.far1), Y.a15, Y.c_far);
            const float fz = fmaf(bound_v<i>(Z.far0, Z.far1), Z.a15, Z.c_far);
#if PT_WIDE_MINMAX3
            const float t_near = max3f(nx, ny, fmaxf(nz, 0.0f));
            const float t_far = min3f(fx, fy, fminf(fz, limit));
#else
            const float t_near = fmaxf(fmaxf(nx, ny), fmaxf(nz, 0.0f));
            const float t_far = fminf(fminf(fx, fy), fminf(fz, limit));
#endif
#if PT_WIDE_MASK_PERMUTE
            if (t_near <= t_far) mask |= 1u << i;
#else
            if ((uint32_t)i < count && t_near <= t_far) mask |= 1u << ((uint32_t)i ^ oct);
#endif
        };
        child(std::integral_constant<int, 0>());
        child(std::integral_constant<int, 1>());
        child(std::integral_constant<int, 2>());
        child(std::integral_constant<int, 3>());
        child(std::integral_constant<int, 4>());
        child(std::integral_constant<int, 5>());
        child(std::integral_constant<int, 6>());
        child(std::integral_constant<int, 7>());
#if PT_WIDE_MASK_PERMUTE
        // slot order -> octant order: bit i moves to bit i ^ oct
        mask &= (1u << count) - 1u;
        if (oct & 1u) mask = ((mask & 0x55u) << 1) | ((mask >> 1) & 0x55u);
        if (oct & 2u) mask = ((mask & 0x33u) << 2) | ((mask >> 2) & 0x33u);
        if (oct & 4u) mask = ((mask & 0x0fu) << 4) | ((mask >> 4) & 0x0fu);
#endif
        return mask;
    }
    // takes the next child of the node: a leaf, or an interior child's own children
    template <class S>
    PTD void visit(S& stack, uint32_t*) {
        if ((list & 0xffu) == 0u) {
            if (sp == 0u) {
                todo = kFinished;
                return;
            }
            sp -= 1u;
            const uint2 e = stack.get(sp);
            node = e.x;
            list = e.y;
        }
        const uint32_t oct = list >> 8;
        const uint32_t k = (uint32_t)(__ffs(list) - 1) ^ oct;
        list &= list - 1u;  // the lowest set bit is in the mask: it is not empty
        const float4* p = sc.wide() + 8 * (size_t)node;
        const uint32_t child = __ldg(reinterpret_cast<const uint32_t*>(p + 4) + k);
        const uint32_t tc = __ldg(reinterpret_cast<const unsigned short*>(p + 6) + k);
        if (tc != 0u) {
            lf = child;
            todo = (int32_t)tc;
            return;
        }
        if ((list & 0xffu) != 0u) {
            stack.put(sp, make_uint2(node, list));
            sp += 1u;
        }
        node = child;
        list = children(child, oct) | (oct << 8);
    }

    // one triangle of the leaf
    template <class S>
    PTD void test(S&, uint32_t*) {
        const uint32_t tri = lf;
        lf += 1u;
        todo -= 1;
        if (kFind != kFindClosest && (int32_t)tri == light_tri) return;
        float t, v, wb;
        if (!triangle_test(load_tri4(sc.tri4(), tri), o, s, &t, &v, &wb)) return;
        if (t > 0.0f && t < limit) {
            if (any_hit()) {
                hit = 1;
                todo = kFinished;
            } else {
                limit = t;
                hit = (int32_t)tri;
                hv = v;
                hw = wb;
            }
        } else if (!any_hit() && t == limit && hit >= 0 && binary_first(sc.f(), o, d, tri, (uint32_t)hit)) {
            // an exact tie: keep the triangle the binary traversal finds first
            hit = (int32_t)tri;
            hv = v;
            hw = wb;
        }
    }
};

// node visits between refills of the 8-wide traversal (its visits are longer), at most
#ifndef PT_WIDE_STEPS_PER_REFILL
#define PT_WIDE_STEPS_PER_REFILL 8
#endif
constexpr uint32_t kStepsPerRefill = PT_STEPS_PER_REFILL;
constexpr uint32_t kWideStepsPerRefill = PT_WIDE_STEPS_PER_REFILL;

// The places of a shading step's next ray and shadow ray in their queues, in
// lane order.
struct Places {
    uint32_t ray, shadow;
};
// One atomic instruction per warp (two lanes, neighbouring words `cnt` and
// `cnt + 1`): atomics on one address leave an L2 slice every 0.65 ns, whatever
// the number of warps.  All 32 lanes.
PTD Places append_warp(uint32_t* cnt, bool ray, bool shadow) {
    const unsigned lane = lane_id();
    const unsigned rays = __ballot_sync(0xffffffffu, ray), shadows = __ballot_sync(0xffffffffu, shadow);
    uint32_t base = 0;
    const uint32_t n = (uint32_t)__popc(lane == 0u ? rays : shadows);
    if (lane < 2u && n) base = atomicAdd(cnt + lane, n);
    const unsigned before = (1u << lane) - 1u;
    return Places{__shfl_sync(0xffffffffu, base, 0) + (uint32_t)__popc(rays & before),
                  __shfl_sync(0xffffffffu, base, 1) + (uint32_t)__popc(shadows & before)};
}
// The same with one atomic instruction per block, for launches whose many
// warps each append little (a hit spread over 16 lanes leaves two per warp).
// All threads of the block; shared: 2 + 2 per warp words.
template <int kThreads>
PTD Places append_block(uint32_t* cnt, bool ray, bool shadow, uint32_t* shared) {
    constexpr uint32_t kWarps = kThreads / 32;
    static_assert(kWarps <= 32, "one lane per warp");
    const unsigned lane = lane_id(), wi = threadIdx.x >> 5;
    const unsigned rays = __ballot_sync(0xffffffffu, ray), shadows = __ballot_sync(0xffffffffu, shadow);
    __syncthreads();  // the last step's places have been read
    if (lane < 2u) shared[2u + 2u * wi + lane] = (uint32_t)__popc(lane == 0u ? rays : shadows);
    __syncthreads();
    uint32_t at_ray = 0, at_shadow = 0, all_rays = 0, all_shadows = 0;
#pragma unroll
    for (uint32_t k = 0; k < kWarps; ++k) {
        if (k == wi) {
            at_ray = all_rays;
            at_shadow = all_shadows;
        }
        all_rays += shared[2u + 2u * k];
        all_shadows += shared[3u + 2u * k];
    }
    if (threadIdx.x < 2u) {
        const uint32_t n = threadIdx.x == 0u ? all_rays : all_shadows;
        shared[threadIdx.x] = n ? atomicAdd(cnt + threadIdx.x, n) : 0u;
    }
    __syncthreads();
    const unsigned before = (1u << lane) - 1u;
    return Places{shared[0] + at_ray + (uint32_t)__popc(rays & before),
                  shared[1] + at_shadow + (uint32_t)__popc(shadows & before)};
}

// sort keys of the hit sort (see sort_count_kernel)
#ifndef PT_SORT_BUCKETS
#define PT_SORT_BUCKETS 4096
#endif
constexpr uint32_t kSortBuckets = PT_SORT_BUCKETS;  // a multiple of 1024, at most 8192 (shared memory)
static_assert(kSortBuckets % 1024 == 0 && kSortBuckets <= 8192, "sort buckets: 1024 .. 8192 in steps of 1024");
constexpr uint32_t kSortPerThread = kSortBuckets / 1024;

// Files finished rays of a round under hits (with their record and sort key) or
// misses, so that the shading kernel runs warps of hits only and warps of
// misses only, and takes the warp's next queue entries: the three reservations
// (hit list, miss list, ray queue) are one atomic instruction of three lanes,
// so a warp waits for memory once.  All 32 lanes, converged; `want` lanes ask
// for entries.  Returns the first entry taken.
template <class Ray>
PTD uint32_t file_and_fetch(const Queues& q, uint32_t* cnt, const Ray& ray, uint32_t slot, uint32_t want) {
    const unsigned lane = lane_id();
    const bool fin = ray.finished(), hit = fin && ray.hit != -1;
    const unsigned hits = __ballot_sync(0xffffffffu, hit), done = __ballot_sync(0xffffffffu, fin);
    const unsigned misses = done & ~hits;
    uint32_t base = 0;
    if (lane < 3u) {
        const uint32_t n = lane == 0u ? want : (uint32_t)__popc(lane == 1u ? hits : misses);
        if (n) base = atomicAdd(cnt + kCntFetch + lane, n);
    }
    const unsigned below_me = (1u << lane) - 1u;
    const uint32_t bh = __shfl_sync(0xffffffffu, base, 1), bm = __shfl_sync(0xffffffffu, base, 2);
    if (hit) {
        q.hit[slot] = make_float4(ray.hit_t(), __int_as_float(ray.hit), ray.hv, ray.hw);
        const uint32_t at = bh + (uint32_t)__popc(hits & below_me);
        q.hit_list[at] = slot;
        if (q.hit_keys) q.hit_keys[at] = min((uint32_t)ray.hit >> q.key_shift, kSortBuckets - 1u);
    } else if (fin) {
        q.miss_list[bm + (uint32_t)__popc(misses & below_me)] = slot;
    }
    return __shfl_sync(0xffffffffu, base, 0);
}

// the entries a shadow warp takes
PTD uint32_t fetch_entries(uint32_t* fetch, uint32_t want) {
    uint32_t base = 0;
    if (lane_id() == 0u && want) base = atomicAdd(fetch, want);
    return __shfl_sync(0xffffffffu, base, 0);
}

// The traversal of a kernel: the 8-wide BVH of the precision form, the packed
// BVH, or the uploaded nodes (recording kernels, pt_trace_noalloc, and scenes
// that the packed form cannot hold).
template <bool kRec, bool kAlpha, int kFind, bool kTri36, bool kWide, bool kPacked, class Scene>
using RayOf = typename std::conditional<
    kWide, WideRay<kFind, Scene>,
    typename std::conditional<kPacked, PackedRay<kAlpha, kFind, Scene>,
                              BinaryRay<kRec, kAlpha, kFind, kTri36, Scene>>::type>::type;

// its stack, with the shared memory of one block
template <uint32_t kThreads, bool kWide, bool kPacked, uint32_t kPackedShared = kPackedSmemStack>
struct BlockStack {
    static constexpr uint32_t kShared = kWide ? kWideSmemStack : kPacked ? kPackedShared : kSmemStack;
    using Lane = typename std::conditional<kPacked, PackedStack<kThreads, kShared>, LaneStack<kThreads, kShared>>::type;
    typename std::conditional<kPacked, float4, uint2>::type top[kShared * kThreads];
    PTD void bind(Lane& lane) {
        if constexpr (kPacked)
            lane.bind(top);
        else
            lane.col = top + threadIdx.x;
    }
};

// 1: in opaque scenes a shading step adds exactly one radiance term to its
// path's colour (the sky at a miss, trace.slang:925; emission at a hit,
// :991; the next-event light of :1204 arrives later through the shadow
// kernel), so the shading kernel starts from zero, and reads and rewrites
// the path's colour only when that term is not zero.  Same bits: the colour
// starts at +0 and is only ever a sum, so it is never -0, and
// colour + (+-0) = colour.  Non-opaque scenes add the unoccluded light in
// the same step (two terms), so they keep the read-modify-write of the
// running colour.
#ifndef PT_COLOR_DELTA
#define PT_COLOR_DELTA 1
#endif
template <bool kAlpha>
constexpr bool kColorDelta = PT_COLOR_DELTA && !kAlpha;

// the path's colour after a shading step: `c` is the new colour, or with
// kColorDelta the term the step added (0 + term)
template <bool kAlpha>
PTD void store_color(float4* color, uint32_t p, f3 c) {
    if constexpr (kColorDelta<kAlpha>) {
        if (c.x != 0.0f || c.y != 0.0f || c.z != 0.0f) {
            const float4 old = color[p];
            color[p] = make_float4(old.x + c.x, old.y + c.y, old.z + c.z, 0.0f);
        }
    } else {
        color[p] = make_float4(c.x, c.y, c.z, 0.0f);
    }
}

// The shading kernels' view of a round's filed results: misses first, padded to
// whole warps, then hits, each hit on 2^spread neighbouring lanes (see
// estimate_e_dielectric).  Entry j of that range maps to a queue slot; the
// first lane of a hit is the one that writes.
struct ShadeRange {
    uint32_t n_hit, n_miss, miss_span, spread;
    const uint32_t* hits;
    // kSpread: hits are spread while the launch's threads allow it
    template <bool kSpread>
    PTD static ShadeRange of(const Queues& q, const uint32_t* cnt) {
        ShadeRange r;
        r.n_hit = cnt[kCntHits];
        r.n_miss = cnt[kCntMisses];
        r.miss_span = (r.n_miss + 31u) & ~31u;
        r.hits = cnt[kCntSorted] ? q.hit_sorted : q.hit_list;
        r.spread = 0u;
        if constexpr (kSpread) {
            const uint32_t threads = gridDim.x * blockDim.x;
            while (r.spread < 4u && r.miss_span + (r.n_hit << (r.spread + 1u)) <= threads) r.spread += 1u;
        }
        return r;
    }
    PTD uint32_t count() const { return miss_span + (n_hit << spread); }
    // queue slot of entry j, or 0xffffffff for the padding after the misses and past the end
    PTD uint32_t slot(const Queues& q, uint32_t j) const {
        if (j < miss_span) return j < n_miss ? q.miss_list[j] : 0xffffffffu;
        const uint32_t k = (j - miss_span) >> spread;
        return k < n_hit ? hits[k] : 0xffffffffu;
    }
    PTD bool leads(uint32_t j) const { return j < miss_span || ((j - miss_span) & ((1u << spread) - 1u)) == 0u; }
};

// The blocks' share of `count` entries, 32 per warp: with more than one turn
// per warp, consecutive blocks take consecutive entries (a block's neighbouring
// hits share its L1); otherwise each block takes an equal run, so that every SM
// gets some.  for (at = first; at < last; at += step): the block's warp wi has
// the entries of turn at + wi when mine(at, wi).
struct BlockTurns {
    uint32_t first, last, step, run;  // in warps of entries
    PTD explicit BlockTurns(uint32_t count) {
        const uint32_t per_block = blockDim.x >> 5;
        last = (count + 31u) >> 5;
        run = per_block;
        step = gridDim.x * per_block;
        if (last <= step) {
            run = (last + gridDim.x - 1u) / gridDim.x;
            step = last;
        }
        first = blockIdx.x * run;
    }
    PTD bool mine(uint32_t at, uint32_t wi) const { return wi < run && at + wi < last; }
};

// ---- hit sorting before shading: a counting sort of the hit list into
// kSortBuckets keys, so that neighbouring lanes shade hits of the same
// material (key mode 0: material index) or of nearby triangles (mode 1:
// triangle index >> shift; triangles are in BVH order, so nearby in space,
// and mostly of one mesh).  Three passes: block histograms into global
// counts; one block scans the counts into bucket offsets (and clears the
// counts for the next bounce); blocks recount their chunk, reserve each
// key's range with one global atomic and scatter.  Skipped (kCntSorted stays
// 0) below min_hits.
constexpr int kSortThreads = 256, kSortItems = 8;

template <int kMode>
PTD uint32_t hit_key(const World& w, const Queues& q, uint32_t slot, uint32_t tri_shift) {
    const uint32_t tri = __float_as_uint(__ldg(&q.hit[slot].y));
    if constexpr (kMode == 0) return attr_material(w, tri) & (kSortBuckets - 1u);
    const uint32_t k = tri >> tri_shift;
    return k < kSortBuckets ? k : kSortBuckets - 1u;
}

template <int kMode>
__global__ void __launch_bounds__(kSortThreads) sort_count_kernel(World w, Queues q, uint32_t round, uint32_t* counts,
                                                                   uint32_t min_hits, uint32_t tri_shift) {
    __shared__ uint32_t hist[kSortBuckets];
    after_previous();
    const uint32_t n = round_counters(q, round)[kCntHits];
    if (n < min_hits) return;
    for (uint32_t i = threadIdx.x; i < kSortBuckets; i += blockDim.x) hist[i] = 0u;
    __syncthreads();
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x)
        atomicAdd(&hist[kMode == 1 && q.hit_keys ? q.hit_keys[j] : hit_key<kMode>(w, q, q.hit_list[j], tri_shift)],
                  1u);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kSortBuckets; i += blockDim.x)
        if (hist[i]) atomicAdd(&counts[i], hist[i]);
}

// one block of 1024 threads, kSortPerThread buckets each
template <int kUnused>
__global__ void __launch_bounds__(1024) sort_scan_kernel(Queues q, uint32_t round, uint32_t* counts,
                                                          uint32_t* offsets, uint32_t min_hits) {
    __shared__ uint32_t part[1024];
    after_previous();
    const uint32_t t = threadIdx.x;
    uint32_t* cnt = round_counters(q, round);
    if (cnt[kCntHits] < min_hits) return;  // kCntSorted stays 0
    uint32_t c[kSortPerThread], sum = 0;
#pragma unroll
    for (uint32_t k = 0; k < kSortPerThread; ++k) {
        c[k] = counts[kSortPerThread * t + k];
        counts[kSortPerThread * t + k] = 0u;
        sum += c[k];
    }
    part[t] = sum;
    __syncthreads();
    for (uint32_t off = 1; off < 1024u; off <<= 1) {
        const uint32_t v = t >= off ? part[t - off] : 0u;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    uint32_t base = part[t] - sum;
#pragma unroll
    for (uint32_t k = 0; k < kSortPerThread; ++k) {
        offsets[kSortPerThread * t + k] = base;
        base += c[k];
    }
    if (t == 0) cnt[kCntSorted] = 1u;
}

template <int kMode>
__global__ void __launch_bounds__(kSortThreads) sort_scatter_kernel(World w, Queues q, uint32_t round,
                                                                     uint32_t* offsets, uint32_t min_hits,
                                                                     uint32_t tri_shift) {
    __shared__ uint32_t hist[kSortBuckets];
    after_previous();
    const uint32_t n = round_counters(q, round)[kCntHits];
    if (n < min_hits) return;
    const uint32_t chunk = kSortThreads * kSortItems;
    for (uint32_t c0 = blockIdx.x * chunk; c0 < n; c0 += gridDim.x * chunk) {
        for (uint32_t i = threadIdx.x; i < kSortBuckets; i += blockDim.x) hist[i] = 0u;
        __syncthreads();
        uint32_t keys[kSortItems], slots[kSortItems];
#pragma unroll
        for (int k = 0; k < kSortItems; ++k) {
            const uint32_t j = c0 + (uint32_t)k * kSortThreads + threadIdx.x;
            keys[k] = 0xffffffffu;
            if (j < n) {
                slots[k] = q.hit_list[j];
                keys[k] = kMode == 1 && q.hit_keys ? q.hit_keys[j] : hit_key<kMode>(w, q, slots[k], tri_shift);
                atomicAdd(&hist[keys[k]], 1u);
            }
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < kSortBuckets; i += blockDim.x)
            if (hist[i]) hist[i] = atomicAdd(&offsets[i], hist[i]);  // this block's range of key i
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kSortItems; ++k)
            if (keys[k] != 0xffffffffu) q.hit_sorted[atomicAdd(&hist[keys[k]], 1u)] = slots[k];
        __syncthreads();
    }
}

// How a launch's warps share a queue: every warp begins with `lanes` entries
// of its own (no atomic; a launch of few rays then takes none at all), the
// rest are taken as lanes fall idle.  All 32 lanes when there are enough rays,
// else as few as share them out, at least 8: a warp of few rays diverges less,
// but each warp costs an atomic when it files them.
#ifndef PT_MIN_SHARE
#define PT_MIN_SHARE 8
#endif
struct QueueShare {
    uint32_t count, first, dealt;  // entries; this warp's first; entries dealt to the warps
    unsigned usable;               // the lanes that take entries
    // a launch drains two queues, the first of `before` entries, this one of
    // `entries`, of `all`: the second begins with the warps that the first's
    // entries leave over
    PTD QueueShare(uint32_t before, uint32_t entries, uint32_t all) : count(entries) {
        const uint32_t per_block = blockDim.x >> 5, warps = gridDim.x * per_block;
        const uint32_t share = min(max((all + warps - 1u) / warps, (uint32_t)PT_MIN_SHARE), 32u);
        usable = share >= 32u ? 0xffffffffu : (1u << share) - 1u;
        // with fewer entries than lanes the warps of a block are far apart in the
        // queue, so that every SM gets some
        const uint32_t wi = threadIdx.x >> 5;
        uint32_t warp = share >= 32u ? blockIdx.x * per_block + wi : wi * gridDim.x + blockIdx.x;
        const uint32_t taken = min((before + share - 1u) / share, warps);
        warp = warp >= taken ? warp - taken : warp + warps - taken;
        first = warp * share;
        dealt = warps * share;
    }
};

// The persistent traversal loop of one warp; every lane holds at most one ray.
// Node visits and triangle tests run in turns: the warp visits nodes while
// enough of its busy lanes are at one, then the lanes that reached a leaf test
// its triangles together.  (On the 1M-triangle scene a ray makes 38 visits and
// 6 tests; with one step of either kind per lane and iteration nearly every
// iteration ran both branches, the test for about 3 lanes.)  Each ray still
// makes its own visits and tests in its own order, so nothing but the
// schedule changes.  The extend launch of bounce 1 (960x540x8): 997 M ->
// 829 M warp instructions at 9.8 -> 14.2 lanes, 1.08 -> 1.01 ms, with the L1
// data pipe now the limit (79 % of its wavefronts: one per lane and load);
// a 960x540x16 image 12.5 -> 11.7 ms, 100k scene in tiles of 512: 31.3 ->
// 29.2 ms, the 16-job engine mix 73.4 -> 68.3 ms.
// start(i) loads queue entry i into the lane's ray; turn(want) runs with the
// warp converged: it files the finished rays and returns the first of `want`
// queue entries.  A warp leaves only when the queue is exhausted and none of
// its lanes is busy, so every entry below `count` is traced once.
template <class Ray, class S, class Start, class Turn>
PTD void traverse_queue(const QueueShare& share, uint32_t max_visits, Ray& ray, S& stack, uint32_t* istack,
                        Start&& start, Turn&& turn) {
    const unsigned lane = lane_id();
    if (share.first >= share.count) return;
    bool exhausted = share.dealt >= share.count;
    if (((share.usable >> lane) & 1u) != 0u && share.first + lane < share.count) start(share.first + lane);
    for (;;) {
        unsigned busy = __ballot_sync(0xffffffffu, ray.busy());
        if (busy == 0u || (!exhausted && __popc(busy) <= Ray::kRefillAt)) {
            const unsigned idle = ~busy & share.usable;
            const uint32_t want = exhausted ? 0u : (uint32_t)__popc(idle);
            const uint32_t base = share.dealt + turn(want);
            if (ray.finished()) ray.set_idle();
            if (exhausted) break;  // nobody is busy, nothing is left
            if ((idle >> lane) & 1u) {
                const uint32_t i = base + (uint32_t)__popc(idle & ((1u << lane) - 1u));
                if (i < share.count) start(i);
            }
            exhausted = base + want >= share.count;
            busy = __ballot_sync(0xffffffffu, ray.busy());
            if (busy == 0u) break;
        }
        const int keep = max(1, (__popc(busy) * Ray::kVisitKeep) >> 5);
        uint32_t visits = 0;
        unsigned m;
        do {
            if (ray.at_node()) ray.visit(stack, istack);
#if PT_VISIT_TWICE
            if (ray.at_node()) ray.visit(stack, istack);
#endif
            m = __ballot_sync(0xffffffffu, ray.at_node());
        } while (__popc(m) >= keep && ++visits < max_visits);
        m = __ballot_sync(0xffffffffu, ray.at_leaf());
        while (m != 0u) {
            if (ray.at_leaf()) ray.test(stack, istack);
            m = __ballot_sync(0xffffffffu, ray.at_leaf());
            if (__popc(m) <= Ray::kTestLeave) break;
        }
    }
}

// The same without a queue: the rays that the warp's lanes hold, to their ends.
template <class Ray, class S>
PTD void traverse_warp(Ray& ray, S& stack) {
    for (;;) {
        const int busy = __popc(__ballot_sync(0xffffffffu, ray.busy()));
        if (busy == 0) return;
        const int keep = max(1, (busy * Ray::kVisitKeep) >> 5), leave = busy >> 3;
        unsigned m;
        do {
            if (ray.at_node()) ray.visit(stack, nullptr);
            if (ray.at_node()) ray.visit(stack, nullptr);
            m = __ballot_sync(0xffffffffu, ray.at_node());
        } while (__popc(m) >= keep);
        m = __ballot_sync(0xffffffffu, ray.at_leaf());
        while (m != 0u) {
            if (ray.at_leaf()) ray.test(stack, nullptr);
            m = __ballot_sync(0xffffffffu, ray.at_leaf());
            if (__popc(m) <= leave) break;
        }
    }
}

// The paths of a round, from the shading of its hits and misses to their ends,
// without a launch between their rounds.  A round of few rays takes as long as
// its longest ray, and the launches of a round of 19,200 paths 33 us; here a
// path waits only for those of its block.
//
// A path has 2 to 16 lanes, as many as leave every path its lanes: they shade
// its hit together (see estimate_e_dielectric), then the first traces its next
// ray while the second traces its shadow ray, whose light is added before the
// next hit's emission, as in the rounds.  A group of lanes takes another path
// of the round when its own ends.  The block shades together: its warps, 4 a
// scheduler, would else each fetch the 40 KB of shading instructions by
// themselves (half of all stalls; 160x120 paths of the room 276 us without the
// barrier, 260 with one of each scheduler's warps, 241 with this one).
// 128 registers, 16 warps an SM; 24 warps of 80 registers were slower.  What a
// warp waits for now, in cycles an instruction: the block's longest ray, at the
// barrier (9.3 of 13.8 in the room, 4.0 of 10.7 in 640x360 of 100k triangles),
// its own loads (0.6, 2.6), fixed latencies (2.0, 2.0), instruction fetch (0.9,
// 0.7); 26 and 33 % of the issue slots.
// `env` gives a path's scene, world and bounces; all threads of the block.
template <bool kAlpha, class Ray, class S, class Env>
PTD void finish_paths(const Env& env, const Queues& q, uint32_t first_round, Ray& ray, S& stack) {
    const Stage st = stage_of(q, first_round);
    uint32_t* const cnt = round_counters(q, first_round);
    const uint32_t hits = cnt[kCntHits], misses = cnt[kCntMisses];
    const uint32_t* list = cnt[kCntSorted] ? q.hit_sorted : q.hit_list;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < misses; j += gridDim.x * blockDim.x) {
        const uint32_t slot = q.miss_list[j];
        const float4 o4 = st.o[slot], d4 = st.d[slot], t4 = st.T[slot];
        const uint32_t path = __float_as_uint(o4.w);
        const float4 c4 = q.color[path];
        PathState ps;
        ps.d = mk(d4.x, d4.y, d4.z);
        ps.throughput = mk(t4.x, t4.y, t4.z);
        ps.prev_pdf = t4.w;
        ps.color = mk(c4.x, c4.y, c4.z);
        shade_miss(env.world(path), first_round, ps);
        q.color[path] = make_float4(ps.color.x, ps.color.y, ps.color.z, 0.0f);
    }
    __syncwarp();
    const unsigned lane = lane_id();
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    uint32_t log2 = 4u;
    while (log2 > 1u && (warps << (5u - log2)) < hits) log2 -= 1u;
    const uint32_t share = 32u >> log2, dealt = warps * share;
    Spread spread;
    spread.log2 = log2;
    spread.index = lane & ((1u << log2) - 1u);
    spread.mask = ((1u << (1u << log2)) - 1u) << (lane - spread.index);
    const bool leads = spread.index == 0u;
    const unsigned leader = lane - spread.index;
    const unsigned before = (1u << leader) - 1u;

    bool has = false, alive = false;
    PathState ps;
    ShadowRay sr;
    sr.valid = false;
    uint32_t path = 0, round = 0, hit = 0;
    float ht = 0.0f, hv = 0.0f, hw = 0.0f;
    Rng<false> rng;
    rng.s = 0u;
    const auto load = [&](uint32_t i) {
        has = alive = i < hits;
        if (!has) return;
        const uint32_t slot = list[i];
        const float4 o4 = st.o[slot], d4 = st.d[slot], t4 = st.T[slot], h4 = q.hit[slot];
        path = __float_as_uint(o4.w);
        const float4 c4 = q.color[path];
        ps.o = mk(o4.x, o4.y, o4.z);
        ps.d = mk(d4.x, d4.y, d4.z);
        ps.throughput = mk(t4.x, t4.y, t4.z);
        ps.prev_pdf = t4.w;
        ps.color = mk(c4.x, c4.y, c4.z);
        rng.s = __float_as_uint(d4.w);
        ht = h4.x;
        hit = __float_as_uint(h4.y);
        hv = h4.z;
        hw = h4.w;
        round = first_round;
    };
    load(((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * share + (lane >> log2));
    bool more = dealt < hits;
    for (;;) {
        if (more) {
            const unsigned idle = __ballot_sync(0xffffffffu, !has && leads);
            const uint32_t want = (uint32_t)__popc(idle);
            if (want != 0u) {
                uint32_t base = 0;
                if (lane == 0u) base = atomicAdd(cnt + kCntTail, want);
                base = dealt + __shfl_sync(0xffffffffu, base, 0);
                if (!has) load(base + (uint32_t)__popc(idle & before));
                more = base + want < hits;
            }
        }
        if (!__syncthreads_or(has)) break;
        __syncwarp();
        if (alive) alive = shade_hit<false, kAlpha, true>(env.world(path), round, env.max_bounces(path), ps, ht, hit, hv, hw, rng, nullptr, &sr, spread);
        __syncwarp();
        round += 1u;
        ray.set_idle();
        const bool shadow = !kAlpha && sr.valid && spread.index == 1u, extend = alive && leads;
        if (extend || shadow) {
            env.enter(ray, path);
            ray.rng.s = rng.s;
            ray.init(extend ? ps.o : sr.o, extend ? ps.d : sr.d, extend ? kFltMax : sr.dist, extend ? kClosestRay : sr.light_tri, stack);
        }
        traverse_warp(ray, stack);
        if constexpr (!kAlpha) {
            const int32_t blocked = __shfl_sync(0xffffffffu, ray.hit, leader + 1u);
            if (sr.valid && blocked != 1) ps.color = ps.color + sr.contribution;
            sr.valid = false;
        }
        const int32_t found = __shfl_sync(0xffffffffu, ray.hit, leader);
        ht = __shfl_sync(0xffffffffu, ray.hit_t(), leader);
        hv = __shfl_sync(0xffffffffu, ray.hv, leader);
        hw = __shfl_sync(0xffffffffu, ray.hw, leader);
        if constexpr (kAlpha) rng.s = __shfl_sync(0xffffffffu, ray.rng.s, leader);
        hit = (uint32_t)found;
        if (alive && found == -1) {
            shade_miss(env.world(path), round, ps);
            alive = false;
        }
        if (has && !alive) {
            if (leads) q.color[path] = make_float4(ps.color.x, ps.color.y, ps.color.z, 0.0f);
            has = false;
        }
        __syncwarp();
    }
}

// no hit sort in a group of at most this many paths: its sorted rounds are the
// first few, and three launches a round cost 795 against 778 us (100k
// triangles, 640x360x1); at 1 M paths 1200 against 1222 (10k, 481x271x8)
constexpr uint32_t kUnsortedPaths = 1u << 18;

// The rounds from which a group's paths are finished by the tail kernel: from
// `first` on when a round has at most `hits` hits, from `always` on in any
// case.  Few paths: a round's launches and its longest ray cost more than the
// better use of lanes gives, from the start.  More: the full rounds go faster
// as launches of their own; after round 4 Russian roulette has ended most
// paths, and open scenes thin out earlier.  The lines lie where these cross
// (us a frame, 8 bounces, 1 to 16 samples a pixel; 152 SMs):
//
//   scene, paths              from 0  from 1  from 2  2^17 hits, 5  never
//   room             65,536      270     273     290            307    391
//   10k, coverage    98,304      466     453     477            499    742
//   100k             98,304      585     586     619            642    866
//   1M               98,304      783     826     883            913  1,218
//   room            131,072      393     387     351            370    424
//   100k            131,072      630     612     640            661    897
//   1M              131,072      925     905     975            992  1,263
//   100k            163,840      684     623     664            685    906
//   10k, coverage   262,144      653     558     580            609    865
//   100k            262,144      882     769     777            798  1,006
//   1M              262,144    1,294   1,161   1,115          1,154  1,443
//   room, 1 sample  327,680      632     590     577            609    583
//   100k            327,680      949     851     825            855  1,088
//   1M              524,288    2,323   1,935   1,778          1,828  1,925
//   room          2,097,152    2,107   1,794   1,604          1,257  1,299
//   1M            2,097,152    6,971   5,171   4,400          3,494  3,699
//   10k, coverage 2,621,440    3,986   2,469   2,193          2,246  2,497
//   room          4,194,304    7,652   6,385   5,470          3,732  3,670
//   1M            4,194,304   14,954  10,894   8,928          6,093  6,228
//
// (2^15 hits and 2^18 instead of 2^17: 481x271x8 of 10k triangles with coverage
// 1205 against 1172, 960x540x4 of 1M 4100 against 3611.)  Groups of over 2^21
// paths overlap with one another.
// Beside other groups the tail's blocks, which fill their SMs at a third of the
// rate, are in the way: four groups of 128x128x16 paths of the room 1605 us
// without it, 2089 with; up to 2^16 paths a group they still gain (four of
// 64x64x16: the room 1133 without, 939 with, 1M triangles 3061, 2397).
struct TailRule {
    uint32_t first = 0xffffffffu, always = 0xffffffffu;
    uint32_t hits = 1u << 17;
    static TailRule of(uint32_t paths, bool alone) {
        TailRule r;
        if (!alone) {
            if (paths <= (1u << 16)) r.first = r.always = 1u;
        } else if (paths <= (1u << 18))
            r.first = r.always = paths <= (1u << 17) ? 0u : 1u;
        else if (paths <= (1u << 21)) {
            r.first = 2u;
            r.always = 5u;
        }
        return r;
    }
};

// A launch that may start while the launch before it in its stream ends (the
// kernel waits for it with after_previous()): 1.4 us from launch to launch
// against 4.1 us for a grid of 1368 blocks.
template <class... P, class... A>
cudaError_t launch_after(void (*kernel)(P...), uint32_t grid, uint32_t block, cudaStream_t stream, A&&... args) {
    cudaLaunchAttribute serial{};
    serial.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    serial.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = stream;
    cfg.attrs = &serial;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// blocks of a kernel that stay resident on an SM of the current device (asked once per kernel and device)
template <class K>
uint32_t resident_blocks(K kernel, int threads) {
    int dev = 0;
    cudaGetDevice(&dev);
    static std::mutex mutex;
    static std::map<std::pair<int, std::pair<const void*, int>>, uint32_t> known;
    std::lock_guard<std::mutex> lock(mutex);
    uint32_t& blocks = known[{dev, {reinterpret_cast<const void*>(kernel), threads}}];
    if (blocks == 0u) {
        int n = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, 0);
        blocks = n > 0 ? (uint32_t)n : 1u;
    }
    return blocks;
}

}  // namespace ptd
