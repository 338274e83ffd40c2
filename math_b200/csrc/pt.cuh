// Path tracing with next-event estimation for one path: the reference
// painter's other integrator (Integrator::PT).
//
// Mirrors src/painter/integrators/pt/{pt.cpp, direct_lighting.cpp} and
// src/painter/integrators/com/surface_sample.cpp, with the parallelotope and
// ball lights' arrive_info (src/painter/lights/parallelotope_light.cpp:92-115,
// ball_light.cpp:90-113).  Russian roulette weighs the path by the
// luminance of all its colour channels, so each thread carries its path's
// full throughput (beta) while it traces.
#pragma once

#include "bpt.cuh"
#include "core.cuh"
#include "geometry.cuh"
#include "kernels.cuh"
#include "scene.cuh"
#include "shading.cuh"

namespace nbpt
{
// std::bernoulli_distribution(p)(engine): one canonical double below p
NBPT_HD bool bernoulli(Pcg& g, const double p)
{
        return canonical<double>(g) < p;
}

// sampling::mis::power_heuristic with one sample each (src/sampling/mis.h:34-58)
template <typename T>
NBPT_HD T power_heuristic(const T f_pdf, const T g_pdf)
{
        const T f = square(1 * f_pdf);
        const T g = square(1 * g_pdf);
        return f / (f + g);
}

// A path longer than this many bounces is cut (Russian roulette ends a path
// with probability at least 0.05 per bounce from the fourth on, so no path
// of the reference gets near it).
inline constexpr int PT_MAX_BOUNCES = 100000;

// One direct-lighting estimate of a bounce, colour-free: its channel c is
// (brdf_c * radiance_c) * scale, brdf_c from the terms (0 when the BRDF's
// own checks fail) and radiance_c the light's.
struct PtEstimate final
{
        BrdfTerms terms;
        float scale;
        int light;
        int zero;
};

// The sampled continuation of a bounce (com::surface_sample): beta_c is
// multiplied by brdf_c * scale.
template <int N, typename T>
struct PtContinuation final
{
        BrdfTerms terms;
        float scale;
        Vec<N, T> l;
};

// Tracing and sampling run on the channel-0 view of the scene (the
// reference's Color::is_black() and usable() look at channel 0 only, so
// every decision is the same); the colour arithmetic runs per channel from
// the recorded BRDF terms, in the reference's operation order.
template <int N, typename T>
struct Pt final
{
        const SceneQueries<N, T, 1>& q;
        const DeviceScene<N, T, 1>& s;
        Pcg& g;
        Bpt<N, T, 1> b; // light samples and visibility

        // LightSource::arrive_info: the light seen from `point` in direction
        // `l`; false when not usable.
        __device__ bool arrive_info(const Light<N, T, 1>& light, const Vec<N, T>& point, const Vec<N, T>& l, T& pdf,
                                    T& distance) const
        {
                if (!(dot(light.normal, point - light.org) > 0))
                {
                        return false;
                }
                const Ray<N, T> ray = Ray<N, T>::make(point, l);
                T t;
                if (light.type == static_cast<int>(LightType::PARALLELOTOPE))
                {
                        t = s.flat[light.shape].shape.intersect(ray);
                        if (!(t > 0))
                        {
                                return false;
                        }
                }
                else
                {
                        // HyperplaneBall::intersect (src/geometry/spatial/hyperplane_ball.h:54-69)
                        Plane<N, T> plane;
                        plane.n = light.normal;
                        plane.d = dot(plane.n, light.org);
                        t = plane.intersect(ray);
                        if (!(t > 0))
                        {
                                return false;
                        }
                        const Vec<N, T> p = ray.point(t);
                        if (!((p - light.org).norm_squared() < light.radius_squared))
                        {
                                return false;
                        }
                }
                const T cos = -dot(ray.dir, light.normal);
                pdf = area_pdf_to_solid_angle_pdf<N>(light.pdf, cos, t);
                distance = t;
                return pdf > 0 && !light.radiance.is_black();
        }

        // sample_light_with_mis (direct_lighting.cpp:59-99); the lights here
        // are area lights (is_delta() false).  The warp calls it together.
        template <typename Warp>
        __device__ bool light_with_mis(const Warp& warp, const bool active, const int k,
                                       const Hit<N, T>& surface, const Vec<N, T>& v, const Normals<N, T>& normals,
                                       PtEstimate& out) const
        {
                const Light<N, T, 1>& light = s.lights[k];
                const Vec<N, T>& n = normals.shading;
                ArriveSample<N, T, 1> sample;
                bool ok = false;
                T n_l = 0;
                Ray<N, T> ray;
                if (active)
                {
                        sample = b.arrive_sample(light, surface.point);
                        ok = sample.usable();
                        if (ok)
                        {
                                n_l = dot(n, sample.l);
                                ok = n_l > 0;
                                ray = Ray<N, T>::make(surface.point, sample.l);
                        }
                }
                if (b.occluded_ray(warp, ok, normals, ray, sample.distance) || !ok)
                {
                        return false;
                }
                const Vec<N, T>& l = sample.l;
                const Material<T, 1>& m = s.materials[q.material(surface)];
                // brdf::f's own checks (brdf.h:146-171), then its terms
                out.zero = (dot(n, v) <= 0 || dot(n, l) <= 0) ? 1 : 0;
                if (!out.zero)
                {
                        out.terms = brdf_terms<N>(s.shading, m.roughness, n, v, l);
                }
                const T pdf = brdf_pdf<N>(s.shading, m.roughness, n, v, l);
                const T weight = power_heuristic(sample.pdf, pdf);
                out.scale = static_cast<float>(weight * n_l / sample.pdf);
                out.light = k;
                return true;
        }

        // sample_surface_with_mis (direct_lighting.cpp:101-147); no shape
        // here is specular.  The warp calls it together.
        template <typename Warp>
        __device__ bool surface_with_mis(const Warp& warp, const bool active, const int k,
                                         const Hit<N, T>& surface, const Vec<N, T>& v, const Normals<N, T>& normals,
                                         PtEstimate& out) const
        {
                const Light<N, T, 1>& light = s.lights[k];
                const Vec<N, T>& n = normals.shading;
                BrdfSample<N, 1, T> sample;
                bool ok = false;
                T n_l = 0;
                T light_pdf = 0;
                T distance = 0;
                Ray<N, T> ray;
                if (active)
                {
                        const Material<T, 1>& m = s.materials[q.material(surface)];
                        sample = brdf_sample_call<N>(g, s.shading, m.roughness, m.f0, m.rho_ss, n, v, &out.terms);
                        ok = sample.pdf > 0 && !sample.brdf.is_black();
                        if (ok)
                        {
                                n_l = dot(n, sample.l);
                                ok = n_l > 0 && arrive_info(light, surface.point, sample.l, light_pdf, distance);
                                ray = Ray<N, T>::make(surface.point, sample.l);
                        }
                }
                if (b.occluded_ray(warp, ok, normals, ray, distance) || !ok)
                {
                        return false;
                }
                const T weight = power_heuristic(sample.pdf, light_pdf);
                out.scale = static_cast<float>(weight * n_l / sample.pdf);
                out.light = k;
                out.zero = 0;
                return true;
        }

        // com::surface_sample (surface_sample.cpp:31-70)
        __device__ bool continuation(const Hit<N, T>& surface, const Vec<N, T>& v, const Normals<N, T>& normals,
                                    PtContinuation<N, T>& out) const
        {
                const Vec<N, T>& n = normals.shading;
                const Material<T, 1>& m = s.materials[q.material(surface)];
                const BrdfSample<N, 1, T> sample =
                        brdf_sample_call<N>(g, s.shading, m.roughness, m.f0, m.rho_ss, n, v, &out.terms);
                if (!(sample.pdf > 0 && !sample.brdf.is_black()))
                {
                        return false;
                }
                if (dot(sample.l, normals.geometric) <= 0)
                {
                        return false;
                }
                const T n_l = dot(n, sample.l);
                if (n_l <= 0)
                {
                        return false;
                }
                out.scale = static_cast<float>(n_l / sample.pdf);
                out.l = sample.l;
                return true;
        }
};

template <typename T, int C>
__device__ float pt_brdf_channel(const BrdfTerms& t, const int zero, const Material<T, C>& m, const int c,
                                 const ShadingConstants<T>& sc)
{
        return zero ? 0.0f : brdf_channel(t, m.f0.c[c], m.rho_ss.c[c], sc.fresnel_a, sc.fresnel_b);
}

// The PT integrator's paths (pt.cpp:113-170), one lane per path at a time
// and one bounce per iteration of a persistent loop: every lane traces one
// ray and processes its hit in each iteration, and a lane whose path ends
// writes it out and takes the next path from a shared counter, so the
// warp's lanes run together however many bounces Russian roulette gives
// their paths.  The warp goes through a bounce as one: at every ray query its
// lanes wait for each other and hand the rays that may enter a mesh to the
// warp's groups of eight (WarpQueries), and the block's warps meet at barriers
// between the parts of a bounce, so that they fetch the same instructions.
// Left to themselves the lanes were at different parts of their bounces, 4 of
// 32 active, with 64 warps per SM at 32 registers to hide it (3-space f64, two
// passes of 1 M paths: 14.6 ms); warps in step each for itself are bound by
// instruction fetch (21.8 ms), blocks of 256 or 512 threads in step are not
// (9.3 ms; 4-space spectral f32, 3 M paths: 20.9 -> 17.0 ms, 22.6 with 512).
// The sample points, the path's ray and its random stream are
// those of the BPT kernels (the same stratified points, seed_seq{seed, pass,
// pixel, sample + 1}); the reference's painter draws them the same way
// whichever integrator it runs (painting.cpp:225-257).  Each lane keeps its
// path's beta (all C channels: in registers for RGB, in the thread's local
// memory for a spectrum) and, for RGB, its colour; a spectrum accumulates in
// the output row.  `estimates` holds 2 * light_count records per thread of
// the grid.
//
// A scene of nothing but a mesh, whose primary rays all look for a facet and
// whose paths mostly end there, spends its time in queries that wait for memory
// and at barriers after the longest of them.  From as many paths on as fill them
// it takes kernels of more blocks per SM (with fewer registers for it), in single
// precision not in step either (IN_STEP), whose warps go on starting paths until
// fewer than PT_REFILL of their lanes are without one that hit something (REFILL).
// 4-space mesh of 20,000 points, 3.4 M paths, 30 % hit, single precision: 2 blocks
// in step 14.3 ms, 4 10.6, 5 10.0, 4 not in step 8.7; double 18.9, with 3 blocks
// 17.0, not in step 20.3; 0.37 M paths 2.2 -> 1.5 and 2.8 -> 2.7; 0.22 M the same.
// Not in 5-space, where hardly a primary ray hits (1.7 M paths 2.3 and 2.5 ms);
// and with walls, which most rays hit, starting anew gains nothing and costs the
// small renders registers (5-space, single precision, 20,000 paths 1.1 -> 1.3).
inline constexpr int PT_THREADS = 256;
inline constexpr int PT_REFILL = 16;
inline constexpr long long PT_MESH_PATHS = 300'000;

template <int N, typename T, int C, bool MANY, bool REFILL, bool IN_STEP>
__device__ __forceinline__ void pt_paths(
        const DeviceScene<N, T, 1>& scene,
        const Material<T, C>* __restrict__ materials,
        const Light<N, T, C>* __restrict__ lights,
        const long long begin,
        const long long end,
        const int spp,
        const std::uint32_t seed,
        const std::uint32_t pass,
        const T* __restrict__ points,
        float* __restrict__ colors,
        float* __restrict__ lum,
        unsigned char* __restrict__ valid,
        PtEstimate* __restrict__ estimates,
        unsigned* __restrict__ next_path,
        PathStats* __restrict__ stats,
        const float* __restrict__ cie_y,
        const unsigned* __restrict__ cancel)
{
        constexpr bool IN_REGISTERS = C <= 4;
        const long long paths = (end - begin) * spp;
        PtEstimate* const est =
                estimates + (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) * 2 * scene.light_count;
        const ShadingConstants<T>& sc = scene.shading;
        QueryCounters counters{0, 0, 0, 0};
        const SceneQueries<N, T, 1> q{scene, counters};
        Pcg g{0, 0};
        extern __shared__ __align__(16) unsigned char stacks[];
        using W = WarpQueries<N, T, 1, MANY>;
        const W warp{q, GroupQueries<N, T, 1>{q, WideStack<T>::of_group(stacks, scene.wide_stack, PT_THREADS)}};
        const Pt<N, T> pt{q, scene, g, Bpt<N, T, 1>{q, scene, g, 0, nullptr, nullptr}};
        Ray<N, T> ray;
        Vec<N, T> gn;
        Color<IN_REGISTERS ? C : 1> reg;
        Color<C> beta;
        constexpr int STARTS = -2;
        int depth = STARTS; // the bounce whose hit is traced next; -1: the primary ray, STARTS: a path to be started
        long long i = -1; // the lane's path; -1 when it takes the next one
        bool done = false;
        const auto take_path = [&]
        {
                i = cancelled(cancel) ? paths : reserve_together(next_path, 1);
                done = i >= paths;
                i = done ? -1 : i;
        };
        const auto start_path = [&]
        {
                // 32-bit index arithmetic: a chunk's path index and a
                // screen's pixel index fit in 31 bits (the painter's chunk
                // limits and its screen check), and a 64-bit division costs
                // several times a 32-bit one
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
                                point[d] = static_cast<T>(static_cast<int>(rest - r * size)) +
                                           points[i * (N - 1) + d];
                                rest = r;
                        }
                }
                ray = scene.projector.ray(point);
                const std::uint32_t words[4] = {seed, pass, static_cast<std::uint32_t>(p),
                                                static_cast<std::uint32_t>(sample + 1)};
                g = seed_seq_pcg(words, 4);
                depth = -1;
        };
        const auto write_background = [&]
        {
#pragma unroll 8
                for (int c = 0; c < C; ++c)
                {
                        colors[i * C + c] = 0.0f;
                }
                lum[i] = 0.0f;
                valid[i] = 0;
        };
        const auto in_step = []
        {
                if constexpr (IN_STEP)
                {
                        __syncthreads();
                }
        };
        while (true)
        {
                Hit<N, T> surface;
                Normals<N, T> normals;
                bool background = false; // written already
                if constexpr (!REFILL)
                {
                        if (i < 0 && !done)
                        {
                                take_path();
                        }
                        if (__syncthreads_and(done ? 1 : 0) != 0)
                        {
                                break;
                        }
                        if (i >= 0 && depth == STARTS)
                        {
                                start_path();
                        }
                        surface = warp.scene_intersect(i >= 0, depth >= 0, gn, ray, normals);
                        __syncthreads();
                        background = i >= 0 && depth < 0 && !surface;
                        if (background)
                        {
                                write_background();
                        }
                }
                else
                {
                        surface.kind = static_cast<int>(HitKind::NONE);
                        bool traced = false;
                        in_step();
                        while (true)
                        {
                                if (i < 0 && !done)
                                {
                                        take_path();
                                }
                                const bool fresh = i >= 0 && !traced;
                                if (fresh && depth == STARTS)
                                {
                                        start_path();
                                }
                                Normals<N, T> found;
                                const Hit<N, T> hit = warp.scene_intersect(fresh, depth >= 0, gn, ray, found);
                                if (fresh)
                                {
                                        surface = hit;
                                        normals = found;
                                        traced = true;
                                        if (depth < 0 && !hit)
                                        {
                                                write_background();
                                                i = -1;
                                                depth = STARTS;
                                                traced = false;
                                        }
                                }
                                if (__popc(__ballot_sync(W::FULL, i < 0 && !done)) < PT_REFILL)
                                {
                                        break;
                                }
                        }
                        if (IN_STEP ? __syncthreads_and(i < 0 && done ? 1 : 0) != 0
                                    : __all_sync(W::FULL, i < 0 && done) != 0)
                        {
                                break;
                        }
                }
                const bool live = i >= 0;
                float* const out = colors + i * C;
                if (live && !background && depth < 0)
                {
                        // the emitted radiance seen by the primary ray
                        // (LightSource::leave_radiance(-dir))
                        const int li = q.light(surface);
                        const bool emits = li >= 0 && dot(-ray.dir, scene.lights[li].normal) > 0;
#pragma unroll 8
                        for (int c = 0; c < C; ++c)
                        {
                                const float e = emits ? lights[li].radiance.c[c] : 0.0f;
                                if constexpr (IN_REGISTERS)
                                {
                                        reg.c[c] = e;
                                }
                                else
                                {
                                        out[c] = e;
                                }
                        }
                        beta = Color<C>::filled(1);
                        depth = 0;
                }

                // one bounce (pt.cpp:68-111); the path ends where the
                // reference's loop breaks
                bool go_on = live && !background && static_cast<bool>(surface);
                const Vec<N, T> v = -ray.dir;
                if (go_on)
                {
                        go_on = !(dot(normals.shading, v) <= 0);
                }
                // direct_lighting (direct_lighting.cpp:150-167): both
                // estimates of every light, summed in that order
                int count = 0;
                for (int k = 0; k < scene.light_count; ++k)
                {
                        count += pt.light_with_mis(warp, go_on, k, surface, v, normals, est[count]) ? 1 : 0;
                        in_step();
                        count += pt.surface_with_mis(warp, go_on, k, surface, v, normals, est[count]) ? 1 : 0;
                        in_step();
                }
                if (go_on)
                {
                        const Material<T, C>& m = materials[q.material(surface)];
                        if (count > 0)
                        {
                                // four channels at a time: a spectrum's row is
                                // read and written 16 bytes at a time
                                constexpr int G = IN_REGISTERS ? 1 : 4;
#pragma unroll 1
                                for (int first = 0; first < C; first += IN_REGISTERS ? C : G)
                                {
                                        constexpr int M = IN_REGISTERS ? C : G;
                                        float sum[M];
#pragma unroll
                                        for (int j = 0; j < M; ++j)
                                        {
                                                sum[j] = 0.0f;
                                        }
                                        for (int e = 0; e < count; ++e)
                                        {
                                                const PtEstimate r = est[e];
                                                const Light<N, T, C>& l = lights[r.light];
#pragma unroll
                                                for (int j = 0; j < M; ++j)
                                                {
                                                        const int c = first + j;
                                                        const float brdf = pt_brdf_channel(r.terms, r.zero, m, c, sc);
                                                        const float x = (brdf * l.radiance.c[c]) * r.scale;
                                                        sum[j] = e == 0 ? x : sum[j] + x;
                                                }
                                        }
                                        if constexpr (IN_REGISTERS)
                                        {
#pragma unroll
                                                for (int j = 0; j < M; ++j)
                                                {
                                                        reg.c[j] += beta.c[j] * sum[j];
                                                }
                                        }
                                        else
                                        {
                                                float4* const row = reinterpret_cast<float4*>(out + first);
                                                float4 o = *row;
                                                o.x += beta.c[first] * sum[0];
                                                o.y += beta.c[first + 1] * sum[1];
                                                o.z += beta.c[first + 2] * sum[2];
                                                o.w += beta.c[first + 3] * sum[3];
                                                *row = o;
                                        }
                                }
                        }

                        PtContinuation<N, T> next;
                        go_on = pt.continuation(surface, v, normals, next);
                        if (go_on)
                        {
#pragma unroll 8
                                for (int c = 0; c < C; ++c)
                                {
                                        beta.c[c] *= pt_brdf_channel(next.terms, 0, m, c, sc) * next.scale;
                                }

                                // terminate (pt.cpp:43-66)
                                if (depth >= 4)
                                {
                                        const float y = luminance(beta, cie_y);
                                        go_on = y > 0;
                                        if (go_on)
                                        {
                                                constexpr float MIN = 0.05f;
                                                constexpr float MAX = 0.95f;
                                                const float x = 1 - y;
                                                const float rr = (x < MIN) ? MIN : ((MAX < x) ? MAX : x);
                                                go_on = !bernoulli(g, rr);
                                                if (go_on)
                                                {
                                                        const float k = 1 - rr;
#pragma unroll 8
                                                        for (int c = 0; c < C; ++c)
                                                        {
                                                                beta.c[c] /= k;
                                                        }
                                                }
                                        }
                                }
                                // after the last bounce the path ends without
                                // the next ray, whose hit the reference never uses
                                if (go_on && ++depth < PT_MAX_BOUNCES)
                                {
                                        ray = Ray<N, T>::make(surface.point, next.l);
                                        gn = normals.geometric;
                                        continue;
                                }
                        }
                }
                if (!live)
                {
                        continue;
                }
                const long long path = i;
                i = -1;
                depth = STARTS;
                if (background)
                {
                        continue;
                }

                // the path is done
                if constexpr (IN_REGISTERS)
                {
#pragma unroll
                        for (int c = 0; c < C; ++c)
                        {
                                out[c] = reg.c[c];
                        }
                        lum[path] = luminance(reg, cie_y);
                        if (!all_finite(reg.c))
                        {
                                atomicAdd(&stats->nonfinite, 1ull);
                        }
                }
                else
                {
                        Color<C> final_color;
#pragma unroll 8
                        for (int c = 0; c < C; ++c)
                        {
                                final_color.c[c] = out[c];
                        }
                        lum[path] = luminance(final_color, cie_y);
                        if (!all_finite(final_color.c))
                        {
                                atomicAdd(&stats->nonfinite, 1ull);
                        }
                }
                valid[path] = 1;
        }
        add_counters(counters, stats);
}

template <int N, typename T, int C, bool MANY>
__global__ void __launch_bounds__(PT_THREADS) pt_paths_kernel(
        const DeviceScene<N, T, 1> scene,
        const Material<T, C>* __restrict__ materials,
        const Light<N, T, C>* __restrict__ lights,
        const long long begin,
        const long long end,
        const int spp,
        const std::uint32_t seed,
        const std::uint32_t pass,
        const T* __restrict__ points,
        float* __restrict__ colors,
        float* __restrict__ lum,
        unsigned char* __restrict__ valid,
        PtEstimate* __restrict__ estimates,
        unsigned* __restrict__ next_path,
        PathStats* __restrict__ stats,
        const float* __restrict__ cie_y,
        const unsigned* __restrict__ cancel)
{
        pt_paths<N, T, C, MANY, false, true>(scene, materials, lights, begin, end, spp, seed, pass, points, colors, lum,
                                             valid, estimates, next_path, stats, cie_y, cancel);
}

// Scenes of one mesh and nothing else (see above).
template <int N, typename T, int C>
__global__ void __launch_bounds__(PT_THREADS, (sizeof(T) == 4 ? 4 : 3)) pt_mesh_paths_kernel(
        const DeviceScene<N, T, 1> scene,
        const Material<T, C>* __restrict__ materials,
        const Light<N, T, C>* __restrict__ lights,
        const long long begin,
        const long long end,
        const int spp,
        const std::uint32_t seed,
        const std::uint32_t pass,
        const T* __restrict__ points,
        float* __restrict__ colors,
        float* __restrict__ lum,
        unsigned char* __restrict__ valid,
        PtEstimate* __restrict__ estimates,
        unsigned* __restrict__ next_path,
        PathStats* __restrict__ stats,
        const float* __restrict__ cie_y,
        const unsigned* __restrict__ cancel)
{
        pt_paths<N, T, C, false, true, sizeof(T) == 8>(scene, materials, lights, begin, end, spp, seed, pass, points,
                                                       colors, lum, valid, estimates, next_path, stats, cie_y, cancel);
}

// The kernels of a dimension, precision and colour, by scene and paths of a
// chunk.
template <int N, typename T, int C>
struct PtKernels final
{
        using Kernel = decltype(&pt_paths_kernel<N, T, C, false>);
        Kernel ordinary;
        Kernel meshes;
        Kernel many;

        Kernel of(const DeviceScene<N, T, 1>& scene, const long long paths) const
        {
                if (many_shapes(scene))
                {
                        return many;
                }
                return scene.flat_count + scene.solid_count == 0 && paths >= PT_MESH_PATHS ? meshes : ordinary;
        }
};

template <int N, typename T, int C>
constexpr PtKernels<N, T, C> pt_kernels()
{
        PtKernels<N, T, C> k{};
        k.ordinary = &pt_paths_kernel<N, T, C, false>;
        k.many = &pt_paths_kernel<N, T, C, true>;
        if constexpr (N == 5)
        {
                k.meshes = k.ordinary;
        }
        else
        {
                k.meshes = &pt_mesh_paths_kernel<N, T, C>;
        }
        return k;
}

template <int N, typename T, int C>
inline constexpr PtKernels<N, T, C> PT_KERNELS = pt_kernels<N, T, C>();
} // namespace nbpt
