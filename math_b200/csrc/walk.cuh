// Subpath walks of BPT as waves: all paths of a chunk take their k-th bounce
// together.
//
//   walk_begin_kernel   every path: random stream, camera ray, and that
//                       ray's test against the flat and solid shapes;
//   walk_mesh_kernel    the rays that may enter a mesh: BVH traversal;
//   walk_step_kernel    every ray of a list: the bounce at its hit
//                       (Bpt::walk_step), then the next ray and its shape
//                       tests; the rays that go on are packed into the next
//                       list;
//   walk_light_kernel   every path with a connectible camera subpath: the
//                       light sample and the first light ray.
//
// The camera subpaths run to the end first, then the light subpaths, so each
// path consumes its random stream in the reference's order (camera subpath,
// light sample, light subpath; bpt.cpp:267-292), and a bounce's number is the
// wave's.
//
// Why waves: a bounce is short (9 shape tests, 6 BVH nodes and 0.7 facets per
// ray on the 4-space box, about 6 rays per path), but its parts differ from
// lane to lane.  One persistent kernel running whole bounces kept 4-5 of 32
// lanes active, held its code (100 KB) out of the instruction cache and
// spilled at the 32 registers its occupancy needed.  Here a warp holds rays
// of one bounce only, each kernel's code is small, the few rays that reach a
// BVH (one in five) are gathered into full warps of their own, and a list is
// read and written in order.  What it costs is the rays' state through
// memory once per bounce: 68 bytes per ray in 4-space single precision.
#pragma once

#include "kernels.cuh"
#include "wide_bvh.cuh"

namespace nbpt
{
inline constexpr int WALK_THREADS = 128;
inline constexpr int WALK_BLOCKS_PER_SM = 16; // of the grids that stride over a list

// The rays of one wave, in the order they were appended; array k of a vector
// holds component k of every ray.
template <int N, typename T>
struct WalkList final
{
        T* org[N]; // moved off the surface the ray leaves
        T* dir[N];
        T* distance; // of the closest hit found so far
        T* pdf;      // forward pdf of the direction
        float* beta; // throughput, channel 0
        int* index;  // hit shape or facet
        // the path's index in the chunk, the camera bounces on its tape and
        // the kind of the hit (HitKind)
        std::uint32_t* path;
        Pcg* rng;

        static constexpr int PATH_BITS = 24;
        static constexpr int BOUNCE_BITS = 4;

        NBPT_HD static std::uint32_t pack(const std::uint32_t path, const int bounces, const int kind)
        {
                return path | (static_cast<std::uint32_t>(bounces) << PATH_BITS) |
                       (static_cast<std::uint32_t>(kind) << (PATH_BITS + BOUNCE_BITS));
        }

        NBPT_HD static std::uint32_t path_of(const std::uint32_t word)
        {
                return word & ((1u << PATH_BITS) - 1);
        }

        NBPT_HD static int bounces_of(const std::uint32_t word)
        {
                return static_cast<int>((word >> PATH_BITS) & ((1u << BOUNCE_BITS) - 1));
        }

        NBPT_HD static int kind_of(const std::uint32_t word)
        {
                return static_cast<int>(word >> (PATH_BITS + BOUNCE_BITS));
        }

        // bytes of the list's arrays for `capacity` rays (a multiple of 64,
        // which keeps every array 16-byte aligned)
        NBPT_HD static constexpr long long bytes(const long long capacity)
        {
                return capacity * static_cast<long long>(sizeof(Pcg) + (2 * N + 2) * sizeof(T) + 3 * 4);
        }

        // lays the arrays out from `p` (16-byte aligned)
        static WalkList at(unsigned char* p, const long long capacity)
        {
                WalkList l;
                l.rng = reinterpret_cast<Pcg*>(p);
                T* t = reinterpret_cast<T*>(p + capacity * sizeof(Pcg));
                for (int i = 0; i < N; ++i)
                {
                        l.org[i] = t;
                        t += capacity;
                }
                for (int i = 0; i < N; ++i)
                {
                        l.dir[i] = t;
                        t += capacity;
                }
                l.distance = t;
                t += capacity;
                l.pdf = t;
                t += capacity;
                l.beta = reinterpret_cast<float*>(t);
                l.index = reinterpret_cast<int*>(l.beta + capacity);
                l.path = reinterpret_cast<std::uint32_t*>(l.index + capacity);
                return l;
        }

        __device__ Ray<N, T> ray(const long long k) const
        {
                Ray<N, T> r;
#pragma unroll
                for (int i = 0; i < N; ++i)
                {
                        r.org[i] = org[i][k];
                        r.dir[i] = dir[i][k];
                }
                return r;
        }

        __device__ void put_ray(const long long k, const Ray<N, T>& r) const
        {
#pragma unroll
                for (int i = 0; i < N; ++i)
                {
                        org[i][k] = r.org[i];
                        dir[i][k] = r.dir[i];
                }
        }
};

static_assert(TASK_MAX_PATHS <= 1LL << 24 && MAX_PATH_VERTICES <= 15);

// The wave counters of a chunk, zeroed before it: the lengths of the lists
// and of the mesh queues by wave (waves 0 .. D of the camera subpaths, then
// 0 .. D of the light subpaths; the last of either stays empty), and of the
// list of light subpaths.
struct WalkCounters final
{
        static constexpr int WAVES = 2 * (MAX_PATH_VERTICES + 1);
        unsigned rays[WAVES];
        unsigned mesh[WAVES];
        unsigned light;
};

// A list's length, 0 once the painter is cancelled: one value for the whole
// block, whose threads loop over the list together.
__device__ inline unsigned block_count(const unsigned* const count, const unsigned* const cancel)
{
        __shared__ unsigned value;
        if (threadIdx.x == 0)
        {
                value = cancelled(cancel) ? 0 : *count;
        }
        __syncthreads();
        return value;
}

// The next ray of a path, tested against the flat and solid shapes, appended
// to a list and, when it may enter a mesh, to the mesh queue.
template <int N, typename T>
struct WalkAppend final
{
        WalkList<N, T> list;
        unsigned* count;
        std::uint32_t* mesh_queue;
        unsigned* mesh_count;

        __device__ void operator()(BlockAppend<WALK_THREADS>& block, const SceneQueries<N, T, 1>& q, const bool go,
                                   const Ray<N, T>& ray, const std::uint32_t path, const int bounces, const float beta,
                                   const T pdf, const Pcg& g) const
        {
                T distance = infinity<T>();
                int kind = static_cast<int>(HitKind::NONE);
                int index = -1;
                bool mesh = false;
                if (go)
                {
                        ++q.counters.queries;
                        q.closest_shape(ray, distance, kind, index);
                        mesh = q.enters_mesh(ray, distance);
                }
                unsigned slot;
                unsigned mesh_slot;
                block.slots(count, go, slot, mesh_count, mesh, mesh_slot);
                if (!go)
                {
                        return;
                }
                list.put_ray(slot, ray);
                list.distance[slot] = distance;
                list.pdf[slot] = pdf;
                list.beta[slot] = beta;
                list.index[slot] = index;
                list.path[slot] = WalkList<N, T>::pack(path, bounces, kind);
                list.rng[slot] = g;
                if (mesh)
                {
                        mesh_queue[mesh_slot] = slot;
                }
        }
};

template <int N, typename T>
__global__ void __launch_bounds__(WALK_THREADS) walk_begin_kernel(
        const DeviceScene<N, T, 1> scene,
        const long long begin,
        const long long paths,
        const int spp,
        const int max_depth,
        const std::uint32_t seed,
        const std::uint32_t pass,
        const T* __restrict__ points,
        PathVertex<N, T, 1>* __restrict__ vertices,
        const WalkAppend<N, T> append,
        PathStats* __restrict__ stats,
        const unsigned* __restrict__ cancel)
{
        __shared__ BlockAppend<WALK_THREADS> block;
        QueryCounters counters{0, 0, 0, 0};
        const SceneQueries<N, T, 1> q{scene, counters};
        const long long i = blockIdx.x * static_cast<long long>(WALK_THREADS) + threadIdx.x;
        // the paths a cancelled pass does not take keep no tape: the later
        // kernels skip the chunk
        const bool go = i < paths && !cancelled(cancel);
        Ray<N, T> ray;
        Pcg g{0, 0};
        if (go)
        {
                // 32-bit index arithmetic: a chunk's path index and a screen's
                // pixel index fit in 31 bits (the painter's chunk limits and its
                // screen check), and a 64-bit division costs several times a
                // 32-bit one
                const unsigned local_pixel = static_cast<unsigned>(i) / static_cast<unsigned>(spp);
                const int sample = static_cast<int>(static_cast<unsigned>(i) - local_pixel * spp);
                const unsigned p = static_cast<unsigned>(begin) + local_pixel;
                Vec<N - 1, T> point;
                {
                        unsigned rest = p;
#pragma unroll
                        for (int d = 0; d < N - 1; ++d)
                        {
                                const unsigned size = static_cast<unsigned>(scene.projector.size[d]);
                                const unsigned r = rest / size;
                                point[d] = static_cast<T>(static_cast<int>(rest - r * size)) + points[i * (N - 1) + d];
                                rest = r;
                        }
                }
                const std::uint32_t words[4] = {seed, pass, static_cast<std::uint32_t>(p),
                                                static_cast<std::uint32_t>(sample + 1)};
                g = seed_seq_pcg(words, 4);
                Bpt<N, T, 1, true> bpt{q, scene, g, max_depth, vertices + i * 2 * (max_depth + 1), nullptr};
                ray = bpt.camera_start(scene.projector.ray(point)).ray;
        }
        append(block, q, go, ray, static_cast<std::uint32_t>(i), 0, 1.0f, T(1), g);
        add_counters(counters, stats);
}

// Eight lanes per queued ray: the closest hit among the meshes, and the
// re-casts (integrators/com/visibility.h:174-204) for a
// facet whose interpolated normal faces away from the ray; only facets have
// one.  The list then holds the last query's hit and its ray's origin.
template <int N, typename T>
__global__ void __launch_bounds__(WALK_THREADS) walk_mesh_kernel(
        const DeviceScene<N, T, 1> scene,
        const WalkList<N, T> list,
        const std::uint32_t* __restrict__ mesh_queue,
        const unsigned* __restrict__ mesh_count,
        PathStats* __restrict__ stats)
{
        constexpr unsigned GROUPS = WALK_THREADS / WIDE;
        using G = GroupQueries<N, T, 1>;
        extern __shared__ __align__(16) unsigned char stacks[];
        QueryCounters counters{0, 0, 0, 0};
        const SceneQueries<N, T, 1> q{scene, counters};
        const G group{q, WideStack<T>::of_group(stacks, scene.wide_stack, WALK_THREADS)};
        const unsigned count = *mesh_count;
        // the warp's groups loop together
        for (unsigned first = blockIdx.x * GROUPS + threadIdx.x / 32 * (32 / WIDE); first < count;
             first += gridDim.x * GROUPS)
        {
                const unsigned m = first + threadIdx.x % 32 / WIDE;
                const bool active = m < count;
                const unsigned k = active ? mesh_queue[m] : 0;
                Ray<N, T> ray = list.ray(k);
                Hit<N, T> hit;
                hit.distance = list.distance[k];
                hit.kind = static_cast<int>(HitKind::NONE);
                hit.index = -1;
                group.template mesh<false, false>(active, ray, hit.distance, hit.kind, hit.index);
                const bool found = active && hit.kind == static_cast<int>(HitKind::FACET);
                bool recast = false;
                if (found && scene.flat_shading == 0)
                {
                        hit.point = q.hit_point(hit, ray);
                        recast = dot(ray.dir, q.compute_normals(hit, ray.dir).shading) > 0;
                }
                const bool moved = recast;
                for (int i = 0; i < 2 && __any_sync(G::FULL, recast); ++i)
                {
                        Vec<N, T> g;
                        if (recast)
                        {
                                g = q.geometric_normal(hit);
                                ray.org = hit.point;
                        }
                        group_closest(group, recast, g, ray, infinity<T>(), hit);
                        if (recast)
                        {
                                ray.org = offset_ray_org(g, ray);
                        }
                        recast = recast && static_cast<bool>(hit);
                }
                if (G::lane() == 0 && (found || moved))
                {
                        if (moved)
                        {
                                list.put_ray(k, ray);
                        }
                        list.distance[k] = hit.distance;
                        list.index[k] = hit.index;
                        const std::uint32_t word = list.path[k];
                        list.path[k] = WalkList<N, T>::pack(WalkList<N, T>::path_of(word),
                                                            WalkList<N, T>::bounces_of(word), hit.kind);
                }
                __syncwarp();
        }
        add_counters(counters, stats);
}

// One bounce of every ray of a list: bounce `depth` of the camera subpaths
// (CAMERA) or of the light subpaths.
template <int N, typename T, bool CAMERA>
__global__ void __launch_bounds__(WALK_THREADS) walk_step_kernel(
        const DeviceScene<N, T, 1> scene,
        const WalkList<N, T> list,
        const unsigned* __restrict__ list_count,
        const WalkAppend<N, T> append,
        std::uint32_t* __restrict__ light_paths, // CAMERA: the paths whose light subpath follows
        unsigned* __restrict__ light_count,
        const int depth,
        const int max_depth,
        PathVertex<N, T, 1>* __restrict__ vertices,
        Pcg* __restrict__ rng,
        std::uint32_t* __restrict__ tape,
        const int words_per_path,
        unsigned char* __restrict__ valid,
        PathStats* __restrict__ stats,
        const unsigned* __restrict__ cancel)
{
        using B = Bpt<N, T, 1, true>;
        using L = WalkList<N, T>;
        __shared__ BlockAppend<WALK_THREADS> block;
        QueryCounters counters{0, 0, 0, 0};
        const SceneQueries<N, T, 1> q{scene, counters};
        const unsigned count = block_count(list_count, cancel);
        for (unsigned first = blockIdx.x * WALK_THREADS; first < count; first += gridDim.x * WALK_THREADS)
        {
                const unsigned k = first + threadIdx.x;
                bool go = false;
                bool light_follows = false;
                Ray<N, T> next;
                std::uint32_t path = 0;
                int bounces = 0;
                Pcg g{0, 0};
                typename B::Walk w;
                if (k < count)
                {
                        const std::uint32_t word = list.path[k];
                        path = L::path_of(word);
                        bounces = L::bounces_of(word);
                        g = list.rng[k];
                        w.beta = Color<1>::filled(list.beta[k]);
                        w.pdf_forward = list.pdf[k];
                        w.ray = list.ray(k);
                        w.depth = depth;
                        w.camera = CAMERA;
                        Hit<N, T> hit;
                        hit.kind = L::kind_of(word);
                        hit.index = list.index[k];
                        hit.distance = list.distance[k];
                        Normals<N, T> normals;
                        if (hit)
                        {
                                hit.point = q.hit_point(hit, w.ray);
                                normals = q.compute_normals(hit, w.ray.dir);
                        }

                        PathVertex<N, T, 1>* const camera = vertices + path * 2LL * (max_depth + 1);
                        std::uint32_t* const tw = tape + path * static_cast<long long>(words_per_path);
                        B bpt{q, scene, g, max_depth, camera, camera + max_depth + 1};
                        bpt.camera_size = depth + 1;
                        bpt.light_size = depth + 1;
                        bpt.tape.w = tw;
                        bpt.tape.n = CAMERA ? TAPE_HEADER + depth * TAPE_CAMERA_BOUNCE
                                            : TAPE_HEADER + bounces * TAPE_CAMERA_BOUNCE + TAPE_LIGHT_START +
                                                      depth * TAPE_LIGHT_BOUNCE;
                        const int tape_begin = bpt.tape.n;
                        go = bpt.walk_step(w, hit, normals);
                        if (go)
                        {
                                next = w.ray;
                                next.org = offset_ray_org(normals.geometric, w.ray);
                                bounces = CAMERA ? depth + 1 : bounces;
                        }
                        else if constexpr (CAMERA)
                        {
                                using S = typename B::Subpaths;
                                const S r = bpt.camera_outcome();
                                tw[0] = static_cast<std::uint32_t>(bpt.tape.n);
                                tw[1] = r != S::BACKGROUND ? 1u : 0u;
                                tw[2] = static_cast<std::uint32_t>(r == S::CONNECT ? bpt.camera_size : 1);
                                tw[3] = 0;
                                valid[path] = r != S::BACKGROUND ? 1 : 0;
                                rng[path] = g;
                                light_follows = r == S::CONNECT;
                                bounces = depth + (bpt.tape.n != tape_begin ? 1 : 0);
                        }
                        else
                        {
                                tw[0] = static_cast<std::uint32_t>(bpt.tape.n);
                                tw[3] = static_cast<std::uint32_t>(bpt.light_size);
                                rng[path] = g;
                        }
                }
                append(block, q, go, next, path, bounces, w.beta.c[0], w.pdf_forward, g);
                if constexpr (CAMERA)
                {
                        unsigned slot;
                        unsigned unused;
                        block.slots(light_count, light_follows, slot, light_count, false, unused);
                        if (light_follows)
                        {
                                light_paths[slot] = L::pack(path, bounces, 0);
                        }
                }
        }
        add_counters(counters, stats);
}

// The light sample of every path whose light subpath follows, and the
// subpath's first ray.
template <int N, typename T>
__global__ void __launch_bounds__(WALK_THREADS) walk_light_kernel(
        const DeviceScene<N, T, 1> scene,
        const std::uint32_t* __restrict__ light_paths,
        const unsigned* __restrict__ light_count,
        const WalkAppend<N, T> append,
        const int max_depth,
        PathVertex<N, T, 1>* __restrict__ vertices,
        Pcg* __restrict__ rng,
        std::uint32_t* __restrict__ tape,
        const int words_per_path,
        PathStats* __restrict__ stats,
        const unsigned* __restrict__ cancel)
{
        using B = Bpt<N, T, 1, true>;
        using L = WalkList<N, T>;
        __shared__ BlockAppend<WALK_THREADS> block;
        QueryCounters counters{0, 0, 0, 0};
        const SceneQueries<N, T, 1> q{scene, counters};
        const unsigned count = block_count(light_count, cancel);
        for (unsigned first = blockIdx.x * WALK_THREADS; first < count; first += gridDim.x * WALK_THREADS)
        {
                const unsigned k = first + threadIdx.x;
                bool go = false;
                std::uint32_t path = 0;
                int bounces = 0;
                Pcg g{0, 0};
                typename B::Walk w;
                if (k < count)
                {
                        const std::uint32_t word = light_paths[k];
                        path = L::path_of(word);
                        bounces = L::bounces_of(word);
                        g = rng[path];
                        PathVertex<N, T, 1>* const camera = vertices + path * 2LL * (max_depth + 1);
                        std::uint32_t* const tw = tape + path * static_cast<long long>(words_per_path);
                        B bpt{q, scene, g, max_depth, camera, camera + max_depth + 1};
                        bpt.tape.w = tw;
                        bpt.tape.n = TAPE_HEADER + bounces * TAPE_CAMERA_BOUNCE;
                        go = bpt.light_start(w);
                        if (!go)
                        {
                                rng[path] = g;
                        }
                }
                append(block, q, go, w.ray, path, bounces, w.beta.c[0], w.pdf_forward, g);
        }
        add_counters(counters, stats);
}

// The walk kernels of a dimension and precision.
template <int N, typename T>
struct WalkKernels final
{
        decltype(&walk_begin_kernel<N, T>) begin;
        decltype(&walk_mesh_kernel<N, T>) mesh;
        decltype(&walk_step_kernel<N, T, true>) camera_step;
        decltype(&walk_light_kernel<N, T>) light;
        decltype(&walk_step_kernel<N, T, false>) light_step;
};

template <int N, typename T>
inline constexpr WalkKernels<N, T> WALK_KERNELS{&walk_begin_kernel<N, T>, &walk_mesh_kernel<N, T>,
                                                &walk_step_kernel<N, T, true>, &walk_light_kernel<N, T>,
                                                &walk_step_kernel<N, T, false>};

// The device buffers of a chunk's walks.
template <int N, typename T>
struct WalkBuffers final
{
        unsigned char* lists;       // two lists of `capacity` rays
        std::uint32_t* mesh_queue;  // [capacity]
        std::uint32_t* light_paths; // [capacity]
        WalkCounters* counters;
        long long capacity;

        static constexpr long long capacity_for(const long long paths)
        {
                return (paths + 63) / 64 * 64;
        }

        static constexpr long long list_bytes(const long long paths)
        {
                return 2 * WalkList<N, T>::bytes(capacity_for(paths));
        }

        // The list that wave `wave` reads, with its counters: the waves
        // alternate between the two lists.
        WalkAppend<N, T> wave(const int wave) const
        {
                return {WalkList<N, T>::at(lists + (wave & 1) * WalkList<N, T>::bytes(capacity), capacity),
                        counters->rays + wave, mesh_queue, counters->mesh + wave};
        }
};

// The launches of one chunk's walks on `stream`; returns their number.  A
// list's length is known to the device only: every launch after the first
// strides a grid of at most `blocks` blocks over it, and a wave whose list is
// empty costs a few microseconds.
template <int N, typename T>
int launch_walks(const WalkKernels<N, T>& kernels, const WalkBuffers<N, T>& buffers, const DeviceScene<N, T, 1>& scene,
                 const long long begin, const long long paths, const int spp, const int max_depth,
                 const std::uint32_t seed, const std::uint32_t pass, const T* const points,
                 PathVertex<N, T, 1>* const vertices, Pcg* const rng, std::uint32_t* const tape,
                 const int words_per_path, unsigned char* const valid, PathStats* const stats,
                 const unsigned* const cancel, const unsigned blocks, const cudaStream_t stream)
{
        const unsigned first = static_cast<unsigned>((paths + WALK_THREADS - 1) / WALK_THREADS);
        const unsigned grid = first < blocks ? first : blocks;
        unsigned* const light_count = &buffers.counters->light;
        const bool meshes = scene.mesh_count > 0;
        int launches = 1;
        const auto mesh = [&](const WalkAppend<N, T>& w)
        {
                if (meshes)
                {
                        kernels.mesh<<<grid, WALK_THREADS, wide_stack_bytes<T>(scene.wide_stack, WALK_THREADS), stream>>>(scene, w.list, w.mesh_queue, w.mesh_count, stats);
                        ++launches;
                }
        };
        kernels.begin<<<first, WALK_THREADS, 0, stream>>>(scene, begin, paths, spp, max_depth, seed, pass, points,
                                                          vertices, buffers.wave(0), stats, cancel);
        int wave = 0;
        for (int depth = 0; depth < max_depth; ++depth, ++wave)
        {
                const WalkAppend<N, T> in = buffers.wave(wave);
                mesh(in);
                kernels.camera_step<<<grid, WALK_THREADS, 0, stream>>>(
                        scene, in.list, in.count, buffers.wave(wave + 1), buffers.light_paths, light_count, depth,
                        max_depth, vertices, rng, tape, words_per_path, valid, stats, cancel);
                ++launches;
        }
        ++wave;
        kernels.light<<<grid, WALK_THREADS, 0, stream>>>(scene, buffers.light_paths, light_count, buffers.wave(wave),
                                                         max_depth, vertices, rng, tape, words_per_path, stats, cancel);
        ++launches;
        for (int depth = 0; depth < max_depth; ++depth, ++wave)
        {
                const WalkAppend<N, T> in = buffers.wave(wave);
                mesh(in);
                kernels.light_step<<<grid, WALK_THREADS, 0, stream>>>(
                        scene, in.list, in.count, buffers.wave(wave + 1), nullptr, nullptr, depth, max_depth, vertices,
                        rng, tape, words_per_path, valid, stats, cancel);
                ++launches;
        }
        return launches;
}
} // namespace nbpt
