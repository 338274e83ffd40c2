// The BVH as the path kernels traverse it: eight children to a node, a ray to
// eight lanes.
//
// A wide node holds the descendants of a binary node (scene.cuh, BvhNode)
// three levels below it, or its leaves where the tree ends earlier; the
// facets' hyperplanes are stored a second time in leaf order.  Eight lanes
// test a node's children together, then a leaf's facets.
//
// The traversal makes the binary traversal's decisions, so it finds the same
// facet at the same distance bit for bit, equal distances included:
//   - A box lies inside its parent's, and the slab test is monotone in the
//     bounds under rounding, so a ray that misses the parent misses the box:
//     the intermediate boxes need no test.
//   - Children are visited in the binary order: at each of the levels between
//     the side the ray's sign on the split axis asks for comes first.
//   - A box test against a distance d is near <= min(d, far), near and far
//     not depending on d; the binary traversal tests a box when it reaches
//     it, so a stacked child keeps its near, which is compared with the
//     distance of that moment.
//   - Of a leaf's facets the closest one hit counts, the first of several at
//     that distance, as when they are tested one by one; it is stacked with
//     the leaf's near and wins if, when its turn comes, near does not exceed
//     the distance and its own is smaller.  A facet that is not closer than
//     the distance at the time of its test never will be.
//
// Why: rays that enter a mesh's box visit 79 binary nodes and 8 facets on
// average on the 4-space hull of 20,000 points, 209 and 35 on a 5-space hull
// of 6,000 points, where the longest of 100,000 visits 1,483 and 411.  One
// lane per ray walked those as a chain of dependent loads: a launch lasted as
// long as its longest ray (2.4 ms in 5-space, 0.6 to 1.1 ms in 4-space,
// whatever the number of rays), with the other lanes of its warp idle.
#pragma once

#include "scene.cuh"

namespace nbpt
{
inline constexpr int WIDE_LEVELS = 3;
inline constexpr int WIDE = 1 << WIDE_LEVELS;
inline constexpr std::uint32_t WIDE_LEAF = 1u << 31;

// Entries of a ray's stack for trees of this depth: a node leaves at most
// WIDE - 1 children behind per level of wide nodes.
inline constexpr int wide_stack_entries(const int depth)
{
        const int levels = depth < 1 ? 1 : (depth + WIDE_LEVELS - 1) / WIDE_LEVELS;
        return levels * (WIDE - 1) + 1;
}

// Dynamic shared memory of a block of `threads` threads.
template <typename T>
constexpr std::size_t wide_stack_bytes(const int entries, const int threads)
{
        return static_cast<std::size_t>(threads / WIDE) * entries * (2 * sizeof(T) + sizeof(std::uint32_t));
}

// ---------------------------------------------------------------------------
// build, from the binary nodes of one mesh

template <int N, typename T>
__global__ void wide_parents_kernel(const BvhNode<N, T>* __restrict__ nodes, const int count,
                                    std::uint32_t* __restrict__ parents)
{
        const int i = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
        if (i >= count)
        {
                return;
        }
        if (i == 0)
        {
                parents[0] = ~0u;
        }
        if (nodes[i].count == 0)
        {
                parents[i + 1] = static_cast<std::uint32_t>(i);
                parents[nodes[i].offset] = static_cast<std::uint32_t>(i);
        }
}

// The wide node of every binary node that becomes one: the root (`root`) and
// the interior nodes at depths that are multiples of WIDE_LEVELS.
template <int N, typename T>
__global__ void wide_index_kernel(const BvhNode<N, T>* __restrict__ nodes, const int count,
                                  const std::uint32_t* __restrict__ parents, const std::uint32_t root,
                                  unsigned* __restrict__ counter, // [2]: wide nodes, depth of the tree
                                  std::uint32_t* __restrict__ wide_index)
{
        const int i = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
        if (i >= count)
        {
                return;
        }
        if (i == 0)
        {
                wide_index[0] = root;
                return;
        }
        unsigned depth = 0;
        for (std::uint32_t p = parents[i]; p != ~0u; p = parents[p])
        {
                ++depth;
        }
        if (nodes[i].count != 0)
        {
                // read first: few leaves deepen the tree
                if (depth > *static_cast<volatile unsigned*>(counter + 1))
                {
                        atomicMax(counter + 1, depth);
                }
                return;
        }
        if (depth % WIDE_LEVELS == 0)
        {
                wide_index[i] = atomicAdd(counter, 1u);
        }
}

// One thread per child slot of every binary node that becomes a wide one.
template <int N, typename T>
__global__ void wide_children_kernel(const BvhNode<N, T>* __restrict__ nodes, const int count,
                                     const std::uint32_t* __restrict__ parents,
                                     const std::uint32_t* __restrict__ wide_index, const int index_offset,
                                     WideChild<N, T>* __restrict__ children)
{
        const long long thread = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
        const int i = static_cast<int>(thread / WIDE);
        const unsigned slot = static_cast<unsigned>(thread % WIDE);
        if (i >= count)
        {
                return;
        }
        if (i != 0)
        {
                if (nodes[i].count != 0)
                {
                        return;
                }
                int depth = 0;
                for (std::uint32_t p = parents[i]; p != ~0u; p = parents[p])
                {
                        ++depth;
                }
                if (depth % WIDE_LEVELS != 0)
                {
                        return;
                }
        }
        WideChild<N, T> c;
        std::uint32_t at = static_cast<std::uint32_t>(i);
        unsigned meta = slot << WideChild<N, T>::SLOT_SHIFT;
        bool used = true;
        for (int level = 0; level < WIDE_LEVELS; ++level)
        {
                const int bit = WIDE_LEVELS - 1 - level;
                if (nodes[at].count != 0)
                {
                        // a leaf above the last level: in the first slot below it
                        used = used && (slot & ((2u << bit) - 1)) == 0;
                        meta |= WideChild<N, T>::NO_AXIS << WideChild<N, T>::axis_shift(level);
                        continue;
                }
                meta |= static_cast<unsigned>(nodes[at].axis) << WideChild<N, T>::axis_shift(level);
                at = ((slot >> bit) & 1u) != 0 ? nodes[at].offset : at + 1;
        }
        const BvhNode<N, T>& n = nodes[at];
#pragma unroll
        for (int d = 0; d < N; ++d)
        {
                // an unused slot's box is never hit
                c.lo[d] = used ? n.lo[d] : infinity<T>();
                c.hi[d] = used ? n.hi[d] : -infinity<T>();
        }
        c.ref = n.count != 0 ? (WIDE_LEAF | (index_offset + n.offset)) : wide_index[at];
        c.meta = used ? (meta | n.count) : WideChild<N, T>::UNUSED;
        children[static_cast<long long>(wide_index[i]) * WIDE + slot] = c;
}

// The facet of every leaf slot of one mesh.
template <int N, typename T>
__global__ void wide_facets_kernel(const Facet<N, T>* __restrict__ facets, const std::uint32_t* __restrict__ indices,
                                   const int count, const int facet_offset, LeafFacet<N, T>* __restrict__ out)
{
        const int i = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
        if (i >= count)
        {
                return;
        }
        const int f = static_cast<int>(indices[i]) + facet_offset;
        LeafFacet<N, T> r;
        r.simplex = facets[f].simplex;
        r.facet = f;
        out[i] = r;
}

// ---------------------------------------------------------------------------
// queries: eight lanes per ray.  Every lane of the warp calls them, with its
// group's ray; `active` and the results are equal in a group's lanes.

// A group's stack, in dynamic shared memory.
template <typename T>
struct WideStack final
{
        T* near;
        T* distance;        // of a leaf's closest facet
        std::uint32_t* ref; // wide node, or WIDE_LEAF | facet
        int entries;

        // the calling thread's group's, in wide_stack_bytes() of memory
        __device__ static WideStack of_group(unsigned char* const memory, const int entries, const int threads)
        {
                const int groups = threads / WIDE;
                const int group = static_cast<int>(threadIdx.x) / WIDE;
                T* const near = reinterpret_cast<T*>(memory);
                T* const distance = near + groups * entries;
                std::uint32_t* const ref = reinterpret_cast<std::uint32_t*>(distance + groups * entries);
                return {near + group * entries, distance + group * entries, ref + group * entries, entries};
        }
};

template <int N, typename T, int C>
struct GroupQueries final
{
        static constexpr unsigned FULL = 0xffffffffu;

        const SceneQueries<N, T, C>& q;
        const WideStack<T> stack;

        __device__ static unsigned lane()
        {
                return threadIdx.x % WIDE;
        }

        __device__ static unsigned group_shift()
        {
                return threadIdx.x % 32 / WIDE * WIDE;
        }

        // The flat and solid shapes of a query, a shape to a lane: the closest
        // hit before `best`, the first of several at one distance; (ANY) whether
        // there is one, in `kind`.
        template <bool ANY>
        __device__ void shapes(const bool active, const Ray<N, T>& ray, T& best, int& kind, int& index) const
        {
                const DeviceScene<N, T, C>& s = q.s;
                T t = best;
                int shape = -1; // in the order of the tests: flat shapes, then solid ones
                if (active)
                {
                        for (int i = static_cast<int>(lane()); i < s.flat_count + s.solid_count; i += WIDE)
                        {
                                ++q.counters.shapes;
                                if (i < s.flat_count)
                                {
                                        const T x = s.flat[i].shape.intersect(ray);
                                        if (x > 0 && x < t)
                                        {
                                                t = x;
                                                shape = i;
                                        }
                                }
                                else
                                {
                                        const T x = s.solid[i - s.flat_count].shape.intersect_volume(ray, t);
                                        if (x >= 0 && x < t)
                                        {
                                                t = x;
                                                shape = i;
                                        }
                                }
                        }
                }
#pragma unroll
                for (int o = 1; o < WIDE; o <<= 1)
                {
                        const T x = __shfl_xor_sync(FULL, t, o);
                        const int i = __shfl_xor_sync(FULL, shape, o);
                        if (i >= 0 && (shape < 0 || x < t || (x == t && i < shape)))
                        {
                                t = x;
                                shape = i;
                        }
                }
                if (shape >= 0)
                {
                        const bool flat = shape < s.flat_count;
                        kind = static_cast<int>(flat ? HitKind::FLAT : HitKind::SOLID);
                        if constexpr (!ANY)
                        {
                                best = t;
                                index = flat ? shape : shape - s.flat_count;
                        }
                }
        }

        // The meshes of a query: the closest hit before `best`, or (ANY) whether
        // there is one, in `kind`.  ONE: the scene has one mesh at most.
        //
        // A mesh's bound is its root box entry (shapes/mesh.cpp:225-229).  Of
        // several meshes eight bounds are tested at a time, a lane each, and the
        // groups then visit theirs, each in its own order, together; a bound that
        // lies behind a hit found in the meantime has no child before it either
        // (3-space, single precision, 500 meshes: one bound after another, by all
        // lanes of a group, 23.7 ms per pass, so 11.3; path tracing 23.5 and 10.4).
        // Scenes of one mesh are 1 to 2 % faster without the rounds, and path
        // tracing without their code.
        template <bool ANY, bool ONE>
        __device__ void mesh(const bool active, const Ray<N, T>& ray, T& best, int& kind, int& index) const
        {
                const DeviceScene<N, T, C>& s = q.s;
                Vec<N, T> rec;
                unsigned neg = 0;
#pragma unroll
                for (int i = 0; i < N; ++i)
                {
                        rec[i] = (ray.dir[i] == 0) ? infinity<T>() : (1 / ray.dir[i]);
                        if (ray.dir[i] < 0)
                        {
                                neg |= 1u << i;
                        }
                }
                if (ONE || s.mesh_count <= 1)
                {
                        const bool enters = active && s.mesh_count > 0 &&
                                            !(ANY && kind != static_cast<int>(HitKind::NONE)) &&
                                            !(box_volume<N>(s.meshes[0].lo, s.meshes[0].hi, ray, best) < 0);
                        if (__any_sync(FULL, enters))
                        {
                                tree<ANY>(enters, 0, ray, rec, neg, best, kind, index);
                        }
                        return;
                }
                if constexpr (!ONE)
                {
                        unsigned entered = 0; // of the eight meshes before `m`, those not yet visited
                        for (int m = 0;;)
                        {
                                if (!__any_sync(FULL, entered != 0))
                                {
                                        if (m >= s.mesh_count)
                                        {
                                                return;
                                        }
                                        const int mine = m + static_cast<int>(lane());
                                        const bool enters =
                                                active && mine < s.mesh_count &&
                                                !(ANY && kind != static_cast<int>(HitKind::NONE)) &&
                                                !(box_volume<N>(s.meshes[mine].lo, s.meshes[mine].hi, ray, best) < 0);
                                        entered = (__ballot_sync(FULL, enters) >> group_shift()) & 0xffu;
                                        m += WIDE;
                                        continue;
                                }
                                const int next = __ffs(static_cast<int>(entered)) - 1;
                                tree<ANY>(entered != 0, static_cast<std::uint32_t>(m - WIDE + next), ray, rec, neg, best,
                                          kind, index);
                                entered = ANY && kind != static_cast<int>(HitKind::NONE) ? 0 : entered & (entered - 1);
                        }
                }
        }

private:
        // The tree of a mesh, whose root is wide node `root`.
        template <bool ANY>
        __device__ __forceinline__ void tree(const bool enters, const std::uint32_t root, const Ray<N, T>& ray,
                                             const Vec<N, T>& rec, const unsigned neg, T& best, int& kind, int& index) const
        {
                int top = 0;
                if (enters)
                {
                        top = 1;
                        if (lane() == 0)
                        {
                                stack.near[0] = 0;
                                stack.ref[0] = root;
                        }
                }
                __syncwarp();
                while (__any_sync(FULL, top > 0))
                {
                        bool node = false;
                        std::uint32_t ref = 0;
                        while (top > 0 && !node)
                        {
                                --top;
                                if (!(stack.near[top] <= best))
                                {
                                        continue;
                                }
                                ref = stack.ref[top];
                                node = (ref & WIDE_LEAF) == 0;
                                if (!ANY && !node && stack.distance[top] < best)
                                {
                                        best = stack.distance[top];
                                        kind = static_cast<int>(HitKind::FACET);
                                        index = static_cast<int>(ref & ~WIDE_LEAF);
                                }
                        }
                        __syncwarp(); // the entries are read before they are written again
                        children<ANY>(node, ref, ray, rec, neg, best, kind, top);
                }
        }

        // Tests the children of node `ref`, and the facets of those that are
        // leaves, and stacks what is hit, the first to visit on top.  ANY: a
        // facet hit ends the query.
        template <bool ANY>
        __device__ void children(const bool node, const std::uint32_t ref, const Ray<N, T>& ray, const Vec<N, T>& rec,
                                 const unsigned neg, const T best, int& kind, int& top) const
        {
                using W = WideChild<N, T>;
                bool hit = false;
                T near = 0;
                T closest = best;
                std::uint32_t entry = 0;
                unsigned key = 0;
                int facets = 0; // of a leaf child that is hit
                if (node)
                {
                        const W c = q.s.wide[static_cast<long long>(ref) * WIDE + lane()];
                        T far = best;
#pragma unroll
                        for (int i = 0; i < N; ++i)
                        {
                                const bool negative = (neg >> i) & 1u;
                                const T a1 = ((negative ? c.hi[i] : c.lo[i]) - ray.org[i]) * rec[i];
                                const T a2 = ((negative ? c.lo[i] : c.hi[i]) - ray.org[i]) * rec[i];
                                near = slab_max(near, a1);
                                far = slab_min(far, a2);
                        }
                        if (c.meta != W::UNUSED)
                        {
                                ++q.counters.nodes;
                                hit = !(far < near);
                        }
                        // the place in the binary visiting order
                        key = (c.meta >> W::SLOT_SHIFT) & (WIDE - 1);
#pragma unroll
                        for (int level = 0; level < WIDE_LEVELS; ++level)
                        {
                                const unsigned axis = (c.meta >> W::axis_shift(level)) & W::NO_AXIS;
                                key ^= ((neg >> axis) & 1u) << (WIDE_LEVELS - 1 - level);
                        }
                        entry = c.ref;
                        facets = hit && (c.ref & WIDE_LEAF) != 0 ? static_cast<int>(c.meta & W::COUNT_MASK) : 0;
                }
                if (__any_sync(FULL, facets > 0))
                {
                        leaf_facets<ANY>(facets, entry, ray, best, closest, hit);
                }
                if constexpr (ANY)
                {
                        const bool facet = hit && (entry & WIDE_LEAF) != 0;
                        if (((__ballot_sync(FULL, facet) >> group_shift()) & 0xffu) != 0)
                        {
                                kind = static_cast<int>(HitKind::FACET);
                                hit = false;
                                top = 0;
                        }
                }
                const unsigned hits =
                        (__reduce_or_sync(FULL, hit ? 1u << (group_shift() + key) : 0u) >> group_shift()) & 0xffu;
                const int count = __popc(hits);
                if (top + count > stack.entries)
                {
                        // the stacks are as deep as the trees; end the query
                        // rather than write past the stack
                        q.counters.overflows += lane() == 0 ? 1 : 0;
                        top = 0;
                }
                else
                {
                        if (hit)
                        {
                                const int at = top + __popc(hits >> (key + 1));
                                stack.near[at] = near;
                                stack.ref[at] = entry;
                                if constexpr (!ANY)
                                {
                                        stack.distance[at] = closest;
                                }
                        }
                        top += count;
                }
                __syncwarp();
        }

        __device__ T facet_distance(const std::uint32_t slot, const Ray<N, T>& ray, const T best, int& facet) const
        {
                ++q.counters.facets;
                const LeafFacet<N, T> f = q.s.leaf_facets[slot];
                const T t = f.simplex.intersect(ray);
                facet = f.facet;
                return t > 0 && t < best ? t : infinity<T>();
        }

        // The facets of the group's leaf children, `count` of this lane's
        // from slot `entry` on (0: none); leaves `closest`, `entry` and `hit`
        // as the lane would by testing its own one by one.  ANY: `hit` in some
        // lane of the group when a facet is hit.
        //
        // Leaves hold 1 to 3 facets as a rule and few of a warp's 32 children
        // are leaves that are hit.  Where a lane has several they are shared
        // out, a facet to a lane: tested by their own lanes they took as many
        // rounds of nearly empty warps as the largest leaf has facets (5-space
        // job: mesh kernels 5.6 -> 4.8 ms).
        template <bool ANY>
        __device__ void leaf_facets(const int count, std::uint32_t& entry, const Ray<N, T>& ray, const T best, T& closest,
                                    bool& hit) const
        {
                if (!__any_sync(FULL, count > 1))
                {
                        if (count > 0)
                        {
                                int facet;
                                const T t = facet_distance(entry & ~WIDE_LEAF, ray, best, facet);
                                hit = t < best;
                                closest = hit ? t : closest;
                                entry = WIDE_LEAF | static_cast<std::uint32_t>(facet);
                        }
                        return;
                }
                const int me = static_cast<int>(lane());
                int end = count; // of the lane's facets among the group's
#pragma unroll
                for (int o = 1; o < WIDE; o <<= 1)
                {
                        const int x = __shfl_up_sync(FULL, end, o, WIDE);
                        end += me >= o ? x : 0;
                }
                const int begin = end - count;
                const int total = __shfl_sync(FULL, end, WIDE - 1, WIDE);
                const std::uint32_t first_slot = (entry & ~WIDE_LEAF) - static_cast<std::uint32_t>(begin);
                hit = hit && count == 0;
                for (int first = 0; __any_sync(FULL, first < total); first += WIDE)
                {
                        const int j = first + me;
                        int owner = 0;
#pragma unroll
                        for (int o = WIDE / 2; o > 0; o >>= 1)
                        {
                                owner += __shfl_sync(FULL, end, owner + o - 1, WIDE) <= j ? o : 0;
                        }
                        const std::uint32_t slot = __shfl_sync(FULL, first_slot, owner, WIDE);
                        T t = infinity<T>();
                        int facet = 0;
                        if (j < total)
                        {
                                t = facet_distance(slot + static_cast<std::uint32_t>(j), ray, best, facet);
                        }
                        if constexpr (ANY)
                        {
                                if (t < best)
                                {
                                        entry = WIDE_LEAF;
                                        hit = true;
                                }
                        }
                        else
                        {
                                const int stop = min(end, first + WIDE);
                                for (int k = max(begin, first); __any_sync(FULL, k < stop); ++k)
                                {
                                        const T x = __shfl_sync(FULL, t, k, WIDE);
                                        const int f = __shfl_sync(FULL, facet, k, WIDE);
                                        if (k < stop && x < closest)
                                        {
                                                closest = x;
                                                entry = WIDE_LEAF | static_cast<std::uint32_t>(f);
                                                hit = true;
                                        }
                                }
                        }
                }
        }

        // near and far of the slab test: a NaN product, of a zero
        // distance and an infinite reciprocal, changes neither
        __device__ static float slab_max(const float near, const float a)
        {
                return fmaxf(near, a);
        }
        __device__ static double slab_max(const double near, const double a)
        {
                return a > near ? a : near;
        }
        __device__ static float slab_min(const float far, const float a)
        {
                return fminf(far, a);
        }
        __device__ static double slab_min(const double far, const double a)
        {
                return a < far ? a : far;
        }
};

// ---------------------------------------------------------------------------
// queries of a ray per lane, for kernels that keep a path on a lane: the warp
// calls them together.  The lanes test the flat and solid shapes; then the
// rays that may enter a mesh (one in five) go to the warp's four groups, four
// at a time, through shuffles.
//
// MANY: scenes of several meshes, or of so many flat and solid shapes that the
// groups test those as well.  In the queries of a bounce only part of a warp's
// lanes have a ray, and they wait for the one whose ray is blocked last; worth
// the shuffles among more than a hundred shapes (path tracing among 1,000
// parallelotopes, 3-space single and double precision: 21.2 and 35.9 ms, shared
// out 12.5 and 21.2; among 100 7.2 and 11.7, shared out 7.1 and 11.3; among 40
// 4.2 and 7.1, shared out 5.0 and 9.5).  Kernels of their own, since the
// additional code costs the other scenes 2 to 3 % (3-space double).
inline constexpr int SHARED_SHAPES = 128;

template <int N, typename T, int C>
inline bool many_shapes(const DeviceScene<N, T, C>& scene)
{
        return scene.mesh_count > 1 || scene.flat_count + scene.solid_count >= SHARED_SHAPES;
}

template <int N, typename T, int C, bool MANY>
struct WarpQueries final
{
        static constexpr unsigned FULL = 0xffffffffu;

        const SceneQueries<N, T, C>& q;
        const GroupQueries<N, T, C> group;

        struct GroupHit final
        {
                T distance;
                int kind;
                int index;
        };

        // whether the groups test the flat and solid shapes
        __device__ bool share_shapes() const
        {
                return MANY && q.s.flat_count + q.s.solid_count >= SHARED_SHAPES;
        }

        // the meshes, and the flat and solid shapes that are shared out, of the
        // lanes that want them: the closest hit before `best` (ANY: whether there
        // is one), kind NONE without
        template <bool ANY>
        NBPT_CALL GroupHit shared(const bool wants, const Ray<N, T>& ray, const T best) const
        {
                GroupHit mine{best, static_cast<int>(HitKind::NONE), -1};
                const int lane = static_cast<int>(threadIdx.x & 31);
                const int my_group = lane / WIDE;
                unsigned pending = __ballot_sync(FULL, wants);
                while (pending != 0)
                {
                        // group g takes the g-th pending lane
                        unsigned rest = pending;
                        for (int g = 0; g < my_group; ++g)
                        {
                                rest &= rest - 1;
                        }
                        const bool active = rest != 0;
                        const int from = active ? __ffs(static_cast<int>(rest)) - 1 : 0;
                        Ray<N, T> r;
#pragma unroll
                        for (int k = 0; k < N; ++k)
                        {
                                r.org[k] = __shfl_sync(FULL, ray.org[k], from);
                                r.dir[k] = __shfl_sync(FULL, ray.dir[k], from);
                        }
                        T distance = __shfl_sync(FULL, best, from);
                        int kind = static_cast<int>(HitKind::NONE);
                        int index = -1;
                        if (share_shapes())
                        {
                                group.template shapes<ANY>(active, r, distance, kind, index);
                        }
                        group.template mesh<ANY, !MANY>(active, r, distance, kind, index);
                        // back to the ray's lane
                        const int place = __popc(pending & ((1u << lane) - 1));
                        const int to = (place % (32 / WIDE)) * WIDE;
                        const T d = __shfl_sync(FULL, distance, to);
                        const int k = __shfl_sync(FULL, kind, to);
                        const int x = __shfl_sync(FULL, index, to);
                        if (((pending >> lane) & 1u) != 0 && place < 32 / WIDE)
                        {
                                mine = {d, k, x};
                        }
#pragma unroll
                        for (int g = 0; g < 32 / WIDE; ++g)
                        {
                                pending &= pending - 1;
                        }
                }
                return mine;
        }

        // a closest-hit query from an offset origin
        __device__ Hit<N, T> closest(const bool active, const Ray<N, T>& ray, const T max_distance) const
        {
                Hit<N, T> h;
                h.kind = static_cast<int>(HitKind::NONE);
                h.index = -1;
                h.distance = max_distance;
                bool wants = false;
                if (active)
                {
                        ++q.counters.queries;
                        wants = share_shapes();
                        if (!wants)
                        {
                                q.closest_shape(ray, h.distance, h.kind, h.index);
                                wants = q.enters_mesh(ray, h.distance);
                        }
                }
                const GroupHit m = shared<false>(wants, ray, h.distance);
                if (m.kind != static_cast<int>(HitKind::NONE))
                {
                        h.distance = m.distance;
                        h.kind = m.kind;
                        h.index = m.index;
                }
                if (h)
                {
                        h.point = q.hit_point(h, ray);
                }
                return h;
        }

        // an any-hit query from an offset origin
        __device__ bool any(const bool active, const Ray<N, T>& ray, const T max_distance) const
        {
                bool hit = false;
                bool wants = false;
                if (active)
                {
                        ++q.counters.queries;
                        wants = share_shapes();
                        if (!wants)
                        {
                                hit = q.any_shape(ray, max_distance);
                                wants = !hit && q.enters_mesh(ray, max_distance);
                        }
                }
                const GroupHit m = shared<true>(wants, ray, max_distance);
                return hit || m.kind != static_cast<int>(HitKind::NONE);
        }

        // scene_intersect (integrators/com/visibility.h:174-204): a hit whose
        // shading normal faces away from the ray is re-cast up to two more times;
        // `normal`: of the surface the ray leaves, where there is one
        __device__ Hit<N, T> scene_intersect(const bool active, const bool from_surface, const Vec<N, T>& normal,
                                             const Ray<N, T>& from, Normals<N, T>& normals) const
        {
                Ray<N, T> ray = from;
                if (active && from_surface)
                {
                        ray.org = offset_ray_org(normal, from);
                }
                Hit<N, T> h = closest(active, ray, infinity<T>());
                bool recast = false;
                if (active && h)
                {
                        normals = q.compute_normals(h, from.dir);
                        recast = dot(from.dir, normals.shading) > 0;
                }
                const bool moved = recast;
                for (int i = 0; i < 2 && __any_sync(FULL, recast); ++i)
                {
                        if (recast)
                        {
                                ray.org = h.point;
                                ray.org = offset_ray_org(q.geometric_normal(h), ray);
                        }
                        const Hit<N, T> next = closest(recast, ray, infinity<T>());
                        if (recast)
                        {
                                h = next;
                        }
                        recast = recast && static_cast<bool>(h);
                }
                if (moved && h)
                {
                        normals = q.compute_normals(h, from.dir);
                }
                return h;
        }
};
} // namespace nbpt
