// Device-resident scene of the n-D painter and its ray queries.
//
// Layout in HBM (all arrays device pointers, one scene per render job):
//   flat[]      flat (n-1)-parallelotopes (walls, light carriers): hyperplane,
//               N-1 slab planes, bounding box, material, attached light
//   solid[]     solid n-parallelotopes: N slabs, bounding box, material
//   meshes[]    one record per mesh shape: root box
//   wide[]      BVH nodes of eight children (wide_bvh.cuh), from the binary
//               nodes (BvhNode), which the scene keeps for export
//   leaf_facets[] the simplex of every leaf slot
//   facets[]    (n-1)-simplex records (hyperplane + N-1 barycentric planes),
//               material and vertex-normal indices
//   normals[]   mesh vertex normals (for interpolated shading normals)
//   materials[] roughness and the two GGX colours (f0, rho_ss)
//   lights[]    parallelotope and ball lights
//
// The queries follow src/painter/scenes/scene.cpp:70-189 (origin offset,
// closest hit, any hit) and src/painter/shapes/*.cpp (per-shape tests).
#pragma once

#include "bvh_build.h"
#include "core.cuh"
#include "geometry.cuh"
#include "shading.cuh"

#include <cstdint>

namespace nbpt
{
enum class NormalType : int
{
        NONE = 0,
        USE = 1,
        REVERSE = 2
};

template <int N, typename T>
struct alignas(16) FlatShape final
{
        FlatParallelotope<N, T> shape;
        T lo[N];
        T hi[N];
        int material;
        int light; // index into lights[] or -1
};

template <int N, typename T>
struct alignas(16) SolidShape final
{
        SolidParallelotope<N, T> shape;
        T lo[N];
        T hi[N];
        int material;
};

template <int N, typename T>
struct alignas(16) Facet final
{
        Simplex<N, T> simplex; // plane possibly reversed (facet.cpp:113-118)
        int material;
        int normal_type;
        int normals[N];
        unsigned reverse_mask;
};

template <int N, typename T>
struct BvhNode final
{
        T lo[N];
        T hi[N];
        std::uint32_t offset; // leaf: first index slot; interior: second child
        std::uint16_t count;  // 0 for interior nodes
        std::uint16_t axis;
};

// A child of a wide node and a facet in leaf order (wide_bvh.cuh), both read
// with 16-byte loads.
template <int N, typename T>
struct alignas(16) WideChild final
{
        T lo[N];
        T hi[N];
        std::uint32_t ref; // wide node, or WIDE_LEAF | first leaf slot
        // facets of a leaf (0: a node), the slot, and the split axis of each
        // level above the child (NO_AXIS below a leaf that ends early)
        std::uint32_t meta;

        static constexpr std::uint32_t COUNT_MASK = 0xffff;
        static constexpr int SLOT_SHIFT = 16;
        static constexpr std::uint32_t NO_AXIS = 7; // no ray has a sign bit there
        static constexpr std::uint32_t UNUSED = ~0u;

        NBPT_HD static constexpr int axis_shift(const int level)
        {
                return SLOT_SHIFT + 3 + 3 * level;
        }
};

template <int N, typename T>
struct alignas(16) LeafFacet final
{
        Simplex<N, T> simplex;
        int facet; // global facet index
};

template <int N, typename T>
struct MeshShape final
{
        T lo[N];
        T hi[N];
};

template <typename T, int C>
struct alignas(16) Material final
{
        T roughness;
        Color<C> f0;
        Color<C> rho_ss;
};

enum class LightType : int
{
        PARALLELOTOPE = 0,
        BALL = 1
};

template <int N, typename T, int C>
struct alignas(16) Light final
{
        int type;
        Vec<N, T> org;             // parallelotope origin or ball centre
        Vec<N, T> vectors[N - 1]; // parallelotope edges or radius-scaled ball basis
        Vec<N, T> normal;          // emission side
        T pdf;                     // 1 / area
        Color<C> radiance;
        T distribution_pdf; // probability of choosing this light
        double cumulative;  // discrete-distribution cumulative probability
        int shape;          // parallelotope: the flat shape that carries it
        T radius_squared;   // ball: square of the radius
};

enum class ProjectorType : int
{
        PERSPECTIVE = 0,
        PARALLEL = 1
};

template <int N, typename T>
struct Projector final
{
        int type;
        Vec<N, T> org;
        Vec<N, T> dir;            // perspective: scaled camera direction; parallel: unit
        Vec<N, T> axes[N - 1];    // normalised screen axes (parallel: times units per pixel)
        Vec<N - 1, T> screen_org; // -size / 2
        int size[N - 1];

        // src/painter/projectors/perspective_projector.cpp:63-69, parallel_projector.cpp:61-67
        NBPT_HD Ray<N, T> ray(const Vec<N - 1, T>& point) const
        {
                Vec<N - 1, T> sp;
#pragma unroll
                for (int i = 0; i < N - 1; ++i)
                {
                        sp[i] = screen_org[i] + point[i];
                }
                Vec<N, T> screen_dir = axes[0] * sp[0];
#pragma unroll
                for (int i = 1; i < N - 1; ++i)
                {
                        screen_dir.multiply_add(axes[i], sp[i]);
                }
                if (type == static_cast<int>(ProjectorType::PERSPECTIVE))
                {
                        return Ray<N, T>::make(org, dir + screen_dir);
                }
                return Ray<N, T>::make(org + screen_dir, dir);
        }
};

template <int N, typename T, int C>
struct DeviceScene final
{
        const FlatShape<N, T>* flat;
        int flat_count;
        const SolidShape<N, T>* solid;
        int solid_count;
        const MeshShape<N, T>* meshes;
        int mesh_count;
        const WideChild<N, T>* wide; // the root of mesh m is wide node m
        const LeafFacet<N, T>* leaf_facets;
        int wide_stack; // stack entries of a query (wide_stack_entries)
        const Facet<N, T>* facets;
        const Vec<N, T>* normals;
        const Material<T, C>* materials;
        const Light<N, T, C>* lights;
        int light_count;
        Projector<N, T> projector;
        ShadingConstants<T> shading;
        // create_painter's flat_shading: shade with the geometric normal, not
        // the facets' interpolated vertex normals (a painter's copy sets it)
        int flat_shading = 0;
};

// ---------------------------------------------------------------------------
// hits

enum class HitKind : int
{
        NONE = 0,
        FLAT = 1,
        SOLID = 2,
        FACET = 3
};

// A surface intersection: what was hit, at which distance, and the hit point
// computed from the (offset) ray the way SurfaceIntersection does
// (src/painter/objects.h:108-116).
template <int N, typename T>
struct Hit final
{
        int kind;
        int index; // flat/solid shape index or global facet index
        T distance;
        Vec<N, T> point;

        NBPT_HD explicit operator bool() const
        {
                return kind != static_cast<int>(HitKind::NONE);
        }
};

template <int N, typename T>
struct Normals final
{
        Vec<N, T> geometric;
        Vec<N, T> shading;
};

// Statistics counted per query for the roofline: BVH boxes (children of wide
// nodes), facet records and other shapes tested.
struct QueryCounters final
{
        std::uint32_t queries;
        std::uint32_t nodes;
        std::uint32_t facets;
        std::uint32_t shapes;
        std::uint32_t overflows; // queries that ended on a full stack
};

template <int N, typename T, int C>
struct SceneQueries final
{
        const DeviceScene<N, T, C>& s;
        QueryCounters& counters;

        // A closest-hit query (scene.cpp:70-95, 97-123, 161-178) moves the
        // origin off the surface the ray leaves (offset_ray_org), counts itself,
        // and asks the flat and solid shapes, then the meshes (wide_bvh.cuh).
        //
        // The flat and solid shapes: closest hit before `best`.
        __device__ void closest_shape(const Ray<N, T>& ray, T& best, int& kind, int& index) const
        {
                for (int i = 0; i < s.flat_count; ++i)
                {
                        ++counters.shapes;
                        const T t = s.flat[i].shape.intersect(ray);
                        if (t > 0 && t < best)
                        {
                                best = t;
                                kind = static_cast<int>(HitKind::FLAT);
                                index = i;
                        }
                }
                for (int i = 0; i < s.solid_count; ++i)
                {
                        ++counters.shapes;
                        const T t = s.solid[i].shape.intersect_volume(ray, best);
                        if (t >= 0 && t < best)
                        {
                                best = t;
                                kind = static_cast<int>(HitKind::SOLID);
                                index = i;
                        }
                }
        }

        // Whether the ray enters a mesh's bound before `best` (with a
        // smaller distance it enters no other).
        __device__ bool enters_mesh(const Ray<N, T>& ray, const T best) const
        {
                for (int i = 0; i < s.mesh_count; ++i)
                {
                        const MeshShape<N, T>& mesh = s.meshes[i];
                        if (!(box_volume<N>(mesh.lo, mesh.hi, ray, best) < 0))
                        {
                                return true;
                        }
                }
                return false;
        }

        // The hit point of a query, from the (offset) ray.
        __device__ Vec<N, T> hit_point(const Hit<N, T>& hit, const Ray<N, T>& ray) const
        {
                const Vec<N, T> p = ray.point(hit.distance);
                switch (static_cast<HitKind>(hit.kind))
                {
                case HitKind::FLAT:
                        return s.flat[hit.index].shape.plane.project(p);
                case HitKind::SOLID:
                        return s.solid[hit.index].shape.project(p);
                default:
                        return s.facets[hit.index].simplex.plane.project(p);
                }
        }

        // The flat and solid shapes of an any-hit query (scene.cpp:125-133,
        // 180-189).
        __device__ bool any_shape(const Ray<N, T>& ray, const T max_distance) const
        {
                for (int i = 0; i < s.flat_count; ++i)
                {
                        ++counters.shapes;
                        const T t = s.flat[i].shape.intersect(ray);
                        if (t > 0 && t < max_distance)
                        {
                                return true;
                        }
                }
                for (int i = 0; i < s.solid_count; ++i)
                {
                        ++counters.shapes;
                        const T t = s.solid[i].shape.intersect_volume(ray, max_distance);
                        if (t >= 0 && t < max_distance)
                        {
                                return true;
                        }
                }
                return false;
        }

        // ---------------------------------------------------------------
        // surface properties

        __device__ Vec<N, T> geometric_normal(const Hit<N, T>& h) const
        {
                switch (static_cast<HitKind>(h.kind))
                {
                case HitKind::FLAT:
                        return s.flat[h.index].shape.plane.n;
                case HitKind::SOLID:
                        return s.solid[h.index].shape.normal(h.point);
                default:
                        return s.facets[h.index].simplex.plane.n;
                }
        }

        // Interpolated vertex normal of a facet (facet.h:96-126); flat and
        // solid parallelotopes have no shading normal.
        __device__ bool shading_normal(const Hit<N, T>& h, Vec<N, T>& out) const
        {
                if (h.kind != static_cast<int>(HitKind::FACET))
                {
                        return false;
                }
                const Facet<N, T>& f = s.facets[h.index];
                if (f.normal_type == static_cast<int>(NormalType::NONE))
                {
                        out = f.simplex.plane.n;
                        return true;
                }
                T bc[N];
                f.simplex.barycentric(h.point, bc);
                Vec<N, T> r;
                {
                        Vec<N, T> n0 = s.normals[f.normals[0]];
                        if ((f.reverse_mask & 1u) != 0)
                        {
                                n0 = -n0;
                        }
                        r = n0 * bc[0];
                }
#pragma unroll
                for (int i = 1; i < N; ++i)
                {
                        Vec<N, T> ni = s.normals[f.normals[i]];
                        if (((f.reverse_mask >> i) & 1u) != 0)
                        {
                                ni = -ni;
                        }
                        r.multiply_add(ni, bc[i]);
                }
                out = r.normalized();
                return true;
        }

        __device__ int material(const Hit<N, T>& h) const
        {
                switch (static_cast<HitKind>(h.kind))
                {
                case HitKind::FLAT:
                        return s.flat[h.index].material;
                case HitKind::SOLID:
                        return s.solid[h.index].material;
                default:
                        return s.facets[h.index].material;
                }
        }

        __device__ int light(const Hit<N, T>& h) const
        {
                return h.kind == static_cast<int>(HitKind::FLAT) ? s.flat[h.index].light : -1;
        }

        // integrators/com/normals.h:45-64; with flat shading the shading
        // normal is the geometric one, which also ends scene_intersect at its
        // first hit (visibility.h:187-190: the flipped geometric normal never
        // faces the ray)
        __device__ Normals<N, T> compute_normals(const Hit<N, T>& h, const Vec<N, T>& ray_dir) const
        {
                const Vec<N, T> g = geometric_normal(h);
                const bool flip = dot(ray_dir, g) >= 0;
                Normals<N, T> r;
                r.geometric = flip ? -g : g;
                Vec<N, T> sn;
                if (s.flat_shading == 0 && shading_normal(h, sn))
                {
                        r.shading = flip ? -sn : sn;
                }
                else
                {
                        r.shading = r.geometric;
                }
                return r;
        }
};
} // namespace nbpt
