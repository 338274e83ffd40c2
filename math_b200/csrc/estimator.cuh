// The painter's per-pixel estimator on the GPU: filtered, trimmed, with the
// reference's exact merge semantics.
//
// Every sample of a source pixel is splatted into its 3^(n-1) neighbours with
// the truncated Gaussian weight (src/painter/pixels/pixel_filter.h:32-70,
// gaussian.h:38-78).  For one (receiving pixel, source pixel) pair the
// weighted samples form a group; the group's two lowest and two highest
// weighted luminances are held out and the rest summed
// (samples/create.cpp:147-250); the group is merged into the receiving
// pixel's state keeping the two lowest and two highest of the union
// (samples/merge.cpp:78-223, com/merge.h:34-233).  Background samples (paths
// that escape at the first hit) keep their own held-out weights.
//
// Which of several equal keys is held out, and the order of the float sums,
// follow the reference step for step: groups are ordered with the same
// insertion-sort and binary-heap selection the reference's sort and
// partial_sort perform, sources are merged into a receiving pixel in
// increasing pixel index, and all sums are in float as the reference keeps
// them.  From the same samples the image is therefore the reference's, bit
// for bit.  Every receiving pixel's groups are merged by one thread or warp, so
// no atomics are needed.
//
// The same merges run with the radiance and weight sums in double (the sum
// type S of the sets): the single-precision trace keeps its per-pixel sums
// in double, so that long renders do not lose the small late contributions
// to float rounding.  Held-out samples are float in both forms.
#pragma once

#include "core.cuh"
#include "group_order.h"

#include <cstdint>

namespace nbpt
{

// largest number of samples per pixel a pass can gather in one group
inline constexpr int MAX_GROUP = 256;

// ---------------------------------------------------------------------------
// sample sets (samples/color.h, samples/background.h)

// S is the type of the sums: float as the reference keeps them (the
// bit-exact mode), or double (the radiance sums of the single-precision
// trace kept in double); held-out entries are float samples in both.
template <int C, typename S = float>
struct ColorSet final
{
        S color_sum[C];
        S weight_sum;
        float colors[HELD_OUT][C];
        float weights[HELD_OUT];
        float contributions[HELD_OUT];
        int count; // held-out entries in use
        int full;  // more than HELD_OUT samples seen: the sums are valid
};

template <typename S = float>
struct BackgroundSet final
{
        S weight_sum;
        float weights[HELD_OUT];
        int count;
        int full;
};

template <int C, typename S = float>
struct PixelState final
{
        ColorSet<C, S> color;
        BackgroundSet<S> background;
};

// A group of one source pixel's samples for one receiving pixel: sample
// indices in the source pixel and their float weights; colours are read
// from global memory and weighted on use (sample.color = weight * colour).
template <int C>
struct ColorGroup final
{
        const float* colors; // the source pixel's sample colours [spp][stride]
        const float* weights;
        const float* lum; // the source pixel's sample luminances
        const int* order;
        int n;
        // channel c of this group is channel c * step + offset of the colours
        // (one thread per pixel: all channels, step 1; one warp per pixel: a
        // lane's channels, step 32 and offset the lane)
        int stride;
        int step;
        int offset;

        NBPT_HD float color(const int k, const int c) const
        {
                const int i = order[k];
                return weights[i] * colors[i * stride + c * step + offset];
        }
};

// create_with_sum (samples/com/create.h:28-55): the sums of a group of more
// than HELD_OUT samples, without those held out, in order.  Eight samples'
// colours are loaded before the first is added, since each is a load whose
// address another load gives (64 channels, 27 groups of 27 samples per pixel:
// with the merges as selections (FullMerge) 12.5 -> 10.3 ms for
// 262,144 pixels).
template <int C, typename S>
__device__ void sum_group(const ColorGroup<C>& g, S (&sum)[C], S& wsum)
{
        constexpr int BATCH = 8;
        const int last = g.n - HELD_OUT / 2;
        for (int first = HELD_OUT / 2; first < last; first += BATCH)
        {
                float w[BATCH];
                float c[BATCH][C];
#pragma unroll
                for (int b = 0; b < BATCH; ++b)
                {
                        const int i = g.order[min(first + b, last - 1)];
                        w[b] = g.weights[i];
#pragma unroll
                        for (int k = 0; k < C; ++k)
                        {
                                c[b][k] = g.colors[i * g.stride + k * g.step + g.offset];
                        }
                }
#pragma unroll
                for (int b = 0; b < BATCH; ++b)
                {
                        if (first + b < last)
                        {
#pragma unroll
                                for (int k = 0; k < C; ++k)
                                {
                                        sum[k] += w[b] * c[b][k];
                                }
                                wsum += w[b];
                        }
                }
        }
}

// ---- merges (com/merge.h) ------------------------------------------------

// Entry accessor over a set or a group, in the set's (sorted) order.
template <int C, typename S>
struct SetView final
{
        const ColorSet<C, S>* s;
        const ColorGroup<C>* g; // when merging a fresh group
        int g_full;
        // group held-out positions: 0, 1 -> order[0], order[1]; 2, 3 -> order[n-2], order[n-1]

        NBPT_HD int count() const
        {
                if (s)
                {
                        return s->full ? HELD_OUT : s->count;
                }
                return g_full ? HELD_OUT : g->n;
        }

        NBPT_HD int group_position(const int k) const
        {
                if (!g_full)
                {
                        return k;
                }
                return k < HELD_OUT / 2 ? k : g->n - HELD_OUT + k;
        }

        NBPT_HD float contribution(const int k) const
        {
                if (s)
                {
                        return s->contributions[k];
                }
                const int i = g->order[group_position(k)];
                return g->weights[i] * g->lum[i];
        }

        NBPT_HD float weight(const int k) const
        {
                if (s)
                {
                        return s->weights[k];
                }
                return g->weights[g->order[group_position(k)]];
        }

        NBPT_HD float color(const int k, const int c) const
        {
                if (s)
                {
                        return s->colors[k][c];
                }
                return g->color(group_position(k), c);
        }
};

template <int C, typename S>
NBPT_HD void copy_entry(ColorSet<C, S>& out, const int to, const SetView<C, S>& from, const int k)
{
#pragma unroll 8
        for (int c = 0; c < C; ++c)
        {
                out.colors[to][c] = from.color(k, c);
        }
        out.weights[to] = from.weight(k);
        out.contributions[to] = from.contribution(k);
}

template <int C, typename S>
NBPT_HD void sum_entry(S* color_sum, S& weight_sum, const SetView<C, S>& from, const int k)
{
#pragma unroll 8
        for (int c = 0; c < C; ++c)
        {
                color_sum[c] += from.color(k, c);
        }
        weight_sum += from.weight(k);
}

// The choice merge_with_sum makes between two full sets, once for all their
// values: of either half the two outermost of the four entries are held out
// and the other two summed, a's before b's, the low half first.  Written out
// as selections: with running indices the sets lay in local memory, a
// dependent access per entry and channel.
struct FullMerge final
{
        bool low_first; // a's entry is the first taken
        bool low_second;
        bool high_first;
        bool high_second;

        template <int C, typename S>
        NBPT_HD FullMerge(const SetView<C, S>& a, const SetView<C, S>& b)
        {
                static_assert(HELD_OUT == 4);
                low_first = a.contribution(0) < b.contribution(0);
                low_second = low_first ? a.contribution(1) < b.contribution(0) : a.contribution(0) < b.contribution(1);
                high_first = a.contribution(3) > b.contribution(3);
                high_second = high_first ? a.contribution(2) > b.contribution(3) : a.contribution(3) > b.contribution(2);
        }

        // a(k), b(k): the values of the entries; out: those held out
        template <typename A, typename B, typename S>
        NBPT_HD void entries(const A& a, const B& b, float* const out, S& sum) const
        {
                const float a0 = a(0);
                const float a1 = a(1);
                const float a2 = a(2);
                const float a3 = a(3);
                const float b0 = b(0);
                const float b1 = b(1);
                const float b2 = b(2);
                const float b3 = b(3);
                out[0] = low_first ? a0 : b0;
                out[1] = low_first ? (low_second ? a1 : b0) : (low_second ? a0 : b1);
                out[3] = high_first ? a3 : b3;
                out[2] = high_first ? (high_second ? a2 : b3) : (high_second ? a3 : b2);
                sum += low_first && low_second ? b0 : (!low_first && !low_second ? a0 : a1);
                sum += !low_first && !low_second ? a1 : b1;
                sum += high_first && high_second ? b3 : (!high_first && !high_second ? a3 : a2);
                sum += !high_first && !high_second ? a2 : b2;
        }
};

// merge_with_sum (com/merge.h:199-233, samples/merge.cpp:109-145)
template <int C, typename S>
NBPT_HD void merge_colors_with_sum(const SetView<C, S>& a, const SetView<C, S>& b, const S* a_sum, S a_wsum,
                                   const S* b_sum, S b_wsum, const bool a_full, const bool b_full,
                                   ColorSet<C, S>& out)
{
        // samples_color_sum / samples_weight_sum (samples/merge.cpp:37-76)
        S sum[C];
        S wsum;
        if (a_full && b_full)
        {
#pragma unroll 8
                for (int c = 0; c < C; ++c)
                {
                        sum[c] = a_sum[c] + b_sum[c];
                }
                wsum = a_wsum + b_wsum;
        }
        else if (a_full)
        {
#pragma unroll 8
                for (int c = 0; c < C; ++c)
                {
                        sum[c] = a_sum[c];
                }
                wsum = a_wsum;
        }
        else if (b_full)
        {
#pragma unroll 8
                for (int c = 0; c < C; ++c)
                {
                        sum[c] = b_sum[c];
                }
                wsum = b_wsum;
        }
        else
        {
#pragma unroll 8
                for (int c = 0; c < C; ++c)
                {
                        sum[c] = 0;
                }
                wsum = 0;
        }

        const int a_size = a.count();
        const int b_size = b.count();
        ColorSet<C, S> r;
        if (a_size == HELD_OUT && b_size == HELD_OUT)
        {
                const FullMerge m(a, b);
#pragma unroll 8
                for (int c = 0; c < C; ++c)
                {
                        float out_c[HELD_OUT];
                        m.entries([&](const int k) { return a.color(k, c); }, [&](const int k) { return b.color(k, c); },
                                  out_c, sum[c]);
#pragma unroll
                        for (int k = 0; k < HELD_OUT; ++k)
                        {
                                r.colors[k][c] = out_c[k];
                        }
                }
                m.entries([&](const int k) { return a.weight(k); }, [&](const int k) { return b.weight(k); }, r.weights,
                          wsum);
                S unused = 0;
                m.entries([&](const int k) { return a.contribution(k); }, [&](const int k) { return b.contribution(k); },
                          r.contributions, unused);
        }
        else
        {
                int ai = 0;
                int bi = 0;
                int i = 0;
                while (i < HELD_OUT / 2 && ai < a_size && bi < b_size)
                {
                        if (a.contribution(ai) < b.contribution(bi))
                        {
                                copy_entry(r, i++, a, ai++);
                        }
                        else
                        {
                                copy_entry(r, i++, b, bi++);
                        }
                }
                while (i < HELD_OUT / 2 && ai < a_size)
                {
                        copy_entry(r, i++, a, ai++);
                }
                while (i < HELD_OUT / 2 && bi < b_size)
                {
                        copy_entry(r, i++, b, bi++);
                }
                const int a_low = ai;
                const int b_low = bi;
                int aj = a_size - 1;
                int bj = b_size - 1;
                int j = HELD_OUT - 1;
                while (j >= HELD_OUT / 2 && aj >= a_low && bj >= b_low)
                {
                        if (a.contribution(aj) > b.contribution(bj))
                        {
                                copy_entry(r, j--, a, aj--);
                        }
                        else
                        {
                                copy_entry(r, j--, b, bj--);
                        }
                }
                while (j >= HELD_OUT / 2 && aj >= a_low)
                {
                        copy_entry(r, j--, a, aj--);
                }
                while (j >= HELD_OUT / 2 && bj >= b_low)
                {
                        copy_entry(r, j--, b, bj--);
                }
                for (int k = a_low; k <= aj; ++k)
                {
                        sum_entry(sum, wsum, a, k);
                }
                for (int k = b_low; k <= bj; ++k)
                {
                        sum_entry(sum, wsum, b, k);
                }
        }
#pragma unroll 8
        for (int c = 0; c < C; ++c)
        {
                r.color_sum[c] = sum[c];
        }
        r.weight_sum = wsum;
        r.count = HELD_OUT;
        r.full = 1;
        out = r;
}

// Merge a fresh group, or the set of one, into a pixel's colour set
// (samples/merge.cpp:198-223).
template <int C, typename S>
NBPT_HD void merge_color_view(ColorSet<C, S>& s, const SetView<C, S>& b, const S* g_sum, const S g_wsum,
                              const bool g_full)
{
        const SetView<C, S> a{&s, nullptr, 0};
        const int a_count = a.count();
        const int b_count = b.count();
        if (a_count + b_count > HELD_OUT)
        {
                merge_colors_with_sum(a, b, s.color_sum, s.weight_sum, g_sum, g_wsum, s.full != 0, g_full, s);
                return;
        }
        if (b_count == 0)
        {
                return;
        }
        if (a_count == 0)
        {
                // the group as created, held-out entries and sums
                ColorSet<C, S> r;
                for (int k = 0; k < b_count; ++k)
                {
                        copy_entry(r, k, b, k);
                }
#pragma unroll 8
                for (int c = 0; c < C; ++c)
                {
                        r.color_sum[c] = g_full ? g_sum[c] : S(0);
                }
                r.weight_sum = g_full ? g_wsum : S(0);
                r.count = b_count;
                r.full = g_full ? 1 : 0;
                s = r;
                return;
        }
        // merge (com/merge.h:235-271): sorted merge of two small sets
        ColorSet<C, S> r;
        int i = 0;
        int ai = 0;
        int bi = 0;
        while (ai < a_count && bi < b_count)
        {
                if (a.contribution(ai) < b.contribution(bi))
                {
                        copy_entry(r, i++, a, ai++);
                }
                else
                {
                        copy_entry(r, i++, b, bi++);
                }
        }
        while (ai < a_count)
        {
                copy_entry(r, i++, a, ai++);
        }
        while (bi < b_count)
        {
                copy_entry(r, i++, b, bi++);
        }
        r.count = a_count + b_count;
        r.full = 0;
        s = r;
}

template <int C, typename S>
NBPT_HD void merge_color_group(ColorSet<C, S>& s, const ColorGroup<C>& g, const S* g_sum, const S g_wsum,
                               const bool g_full)
{
        merge_color_view<C, S>(s, SetView<C, S>{nullptr, &g, g_full ? 1 : 0}, g_sum, g_wsum, g_full);
}

// Background sets: the same merges on weights only.
//
// The set of a group of `n` background weights, weight(k) in order
// (order_group on values).
template <typename S, typename Weight>
NBPT_HD void background_group(BackgroundSet<S>& g, const int n, const Weight& weight)
{
        g.weight_sum = 0;
        g.count = n;
        g.full = n > HELD_OUT ? 1 : 0;
        if (g.full)
        {
                g.weights[0] = weight(0);
                g.weights[1] = weight(1);
                for (int k = 2; k < n - 2; ++k)
                {
                        g.weight_sum += weight(k);
                }
                g.weights[2] = weight(n - 2);
                g.weights[3] = weight(n - 1);
                g.count = HELD_OUT;
                return;
        }
        for (int k = 0; k < n; ++k)
        {
                g.weights[k] = weight(k);
        }
}

// Merges a group's set into a pixel's.
template <typename S>
NBPT_HD void merge_background(BackgroundSet<S>& s, const BackgroundSet<S>& g)
{
        const bool g_full = g.full != 0;
        const float* const held = g.weights;
        const S g_sum = g.weight_sum;
        const int g_count = g.count;
        const int a_count = s.full ? HELD_OUT : s.count;
        if (a_count + g_count > HELD_OUT)
        {
                S wsum;
                if (s.full && g_full)
                {
                        wsum = s.weight_sum + g_sum;
                }
                else if (s.full)
                {
                        wsum = s.weight_sum;
                }
                else if (g_full)
                {
                        wsum = g_sum;
                }
                else
                {
                        wsum = 0;
                }
                float out[HELD_OUT];
                const float* a = s.weights;
                const float* b = held;
                const int a_size = a_count;
                const int b_size = g_count;
                if (a_size == HELD_OUT && b_size == HELD_OUT)
                {
                        int ai = 0;
                        int bi = 0;
                        for (int i = 0; i < HELD_OUT / 2; ++i)
                        {
                                out[i] = (a[ai] < b[bi]) ? a[ai++] : b[bi++];
                        }
                        while (ai < HELD_OUT / 2)
                        {
                                wsum += a[ai++];
                        }
                        while (bi < HELD_OUT / 2)
                        {
                                wsum += b[bi++];
                        }
                        ai = HELD_OUT - 1;
                        bi = HELD_OUT - 1;
                        for (int i = HELD_OUT - 1; i >= HELD_OUT / 2; --i)
                        {
                                out[i] = (a[ai] > b[bi]) ? a[ai--] : b[bi--];
                        }
                        while (ai >= HELD_OUT / 2)
                        {
                                wsum += a[ai--];
                        }
                        while (bi >= HELD_OUT / 2)
                        {
                                wsum += b[bi--];
                        }
                }
                else
                {
                        int ai = 0;
                        int bi = 0;
                        int i = 0;
                        while (i < HELD_OUT / 2 && ai < a_size && bi < b_size)
                        {
                                out[i++] = (a[ai] < b[bi]) ? a[ai++] : b[bi++];
                        }
                        while (i < HELD_OUT / 2 && ai < a_size)
                        {
                                out[i++] = a[ai++];
                        }
                        while (i < HELD_OUT / 2 && bi < b_size)
                        {
                                out[i++] = b[bi++];
                        }
                        const int a_low = ai;
                        const int b_low = bi;
                        int aj = a_size - 1;
                        int bj = b_size - 1;
                        int j = HELD_OUT - 1;
                        while (j >= HELD_OUT / 2 && aj >= a_low && bj >= b_low)
                        {
                                out[j--] = (a[aj] > b[bj]) ? a[aj--] : b[bj--];
                        }
                        while (j >= HELD_OUT / 2 && aj >= a_low)
                        {
                                out[j--] = a[aj--];
                        }
                        while (j >= HELD_OUT / 2 && bj >= b_low)
                        {
                                out[j--] = b[bj--];
                        }
                        for (int k = a_low; k <= aj; ++k)
                        {
                                wsum += a[k];
                        }
                        for (int k = b_low; k <= bj; ++k)
                        {
                                wsum += b[k];
                        }
                }
                for (int k = 0; k < HELD_OUT; ++k)
                {
                        s.weights[k] = out[k];
                }
                s.weight_sum = wsum;
                s.count = HELD_OUT;
                s.full = 1;
                return;
        }
        if (g_count == 0)
        {
                return;
        }
        if (a_count == 0)
        {
                for (int k = 0; k < g_count; ++k)
                {
                        s.weights[k] = held[k];
                }
                s.weight_sum = g_full ? g_sum : S(0);
                s.count = g_count;
                s.full = g_full ? 1 : 0;
                return;
        }
        float out[HELD_OUT];
        int i = 0;
        int ai = 0;
        int bi = 0;
        while (ai < a_count && bi < g_count)
        {
                out[i++] = (s.weights[ai] < held[bi]) ? s.weights[ai++] : held[bi++];
        }
        while (ai < a_count)
        {
                out[i++] = s.weights[ai++];
        }
        while (bi < g_count)
        {
                out[i++] = held[bi++];
        }
        for (int k = 0; k < i; ++k)
        {
                s.weights[k] = out[k];
        }
        s.count = i;
        s.full = 0;
}

template <typename S>
NBPT_HD void merge_background_group(BackgroundSet<S>& s, const float* gw, const int n)
{
        BackgroundSet<S> g;
        background_group(g, n, [&](const int k) { return gw[k]; });
        merge_background(s, g);
}

// ---------------------------------------------------------------------------
// accumulation

template <int N>
struct Screen final
{
        int size[N - 1];
        // a slab of the screen: the receiving pixels are [first, first +
        // pixel_count) in global index, and the sample arrays hold the pixels
        // from source_first on (0 and 0 for the whole screen)
        long long first = 0;
        long long source_first = 0;
};

inline constexpr int neighbours(const int n)
{
        return n == 3 ? 9 : (n == 4 ? 27 : 81);
}

// RGB accumulation of few samples per pixel: a thread per receiving pixel goes
// through its 3^(n-1) source pixels, forms each group and merges it.  Groups
// of one to nine samples take less time to form than to carry through memory
// between the two kernels below (132-152 bytes each), once the screen has
// enough pixels to fill the GPU with threads.  Milliseconds with this kernel /
// with the two, single precision: 3-space 8 M pixels x 1 sample 3.4 / 16.4,
// 160,000 x 9 0.24 / 0.40 and 40,000 x 9 0.125 / 0.125; 4-space 8 M x 1
// 8.8 / 49.7, 157,000 x 8 1.06 / 1.15 and 39,000 x 8 0.40 / 0.31; 5-space
// 2.6 M x 1 9.5 / 55.9.  From sixteen samples on the two are faster at every
// size (3-space 2.5 M x 16 7.1 / 5.9, 5-space 2.6 M x 16 89.9 / 65.1).
//
// The screens where both are about equally fast, but for a single sample per
// pixel (no sums and no order), have some 600 pixels per sample of a pixel's
// neighbourhood: 3-space x 4 15,000 to 20,000, x 9 40,000 to 55,000, 4-space
// x 8 110,000 (single) to 300,000 (double).
template <int N>
inline constexpr bool thread_per_pixel(const long long pixels, const int spp)
{
        return spp == 1 || (spp < 16 && pixels >= 600LL * spp * neighbours(N));
}

// Merge one pass's samples of the 3^(n-1) neighbours into receiving pixel t
// (global index).
template <int N, typename T, int C, typename S>
NBPT_HD void accumulate_pixel(
        const Screen<N>& screen,
        const long long t,
        const int spp,
        const T* __restrict__ points,
        const float* __restrict__ colors,
        const float* __restrict__ lum,
        const unsigned char* __restrict__ valid,
        const T alpha,
        const T exp_radius,
        PixelState<C, S>& st)
{
        int tc[N - 1];
        {
                long long rest = t;
#pragma unroll
                for (int d = 0; d < N - 1; ++d)
                {
                        tc[d] = static_cast<int>(rest % screen.size[d]);
                        rest /= screen.size[d];
                }
        }

        float w[MAX_GROUP];
        int color_order[MAX_GROUP];
        float background[MAX_GROUP];

        // sources in increasing pixel index: the last screen axis outermost
        for (int nb = 0; nb < neighbours(N); ++nb)
        {
                int pc[N - 1];
                bool inside = true;
                {
                        int rest = nb;
#pragma unroll
                        for (int d = 0; d < N - 1; ++d)
                        {
                                pc[d] = tc[d] + (rest % 3) - 1;
                                rest /= 3;
                                inside = inside && pc[d] >= 0 && pc[d] < screen.size[d];
                        }
                }
                if (!inside)
                {
                        continue;
                }
                long long p = 0;
#pragma unroll
                for (int d = N - 2; d >= 0; --d)
                {
                        p = p * screen.size[d] + pc[d];
                }

                // weights (pixel_filter.h:57-69, gaussian.h:66-77) and the
                // selection of colour and background samples (com/select.h:28-47)
                int nc = 0;
                int nbg = 0;
                for (int j = 0; j < spp; ++j)
                {
                        const long long sidx = (p - screen.source_first) * spp + j;
                        const T x0 = (static_cast<T>(tc[0] - pc[0]) + T(0.5)) - points[sidx * (N - 1)];
                        T weight = max_value(T(0), exp(alpha * x0 * x0) - exp_radius);
#pragma unroll
                        for (int d = 1; d < N - 1; ++d)
                        {
                                const T x = (static_cast<T>(tc[d] - pc[d]) + T(0.5)) - points[sidx * (N - 1) + d];
                                weight *= max_value(T(0), exp(alpha * x * x) - exp_radius);
                        }
                        if (!(weight > 0))
                        {
                                continue;
                        }
                        const float wf = static_cast<float>(weight);
                        if (valid[sidx])
                        {
                                w[j] = wf;
                                color_order[nc++] = j;
                        }
                        else
                        {
                                background[nbg++] = wf;
                        }
                }

                if (nc > 0)
                {
                        const float* const source_lum = lum + (p - screen.source_first) * spp;
                        order_group(color_order, nc, [&](const int i) { return w[i] * source_lum[i]; });
                        const ColorGroup<C> g{colors + (p - screen.source_first) * spp * C, w, source_lum, color_order, nc, C, 1, 0};
                        S g_sum[C];
                        S g_wsum = 0;
#pragma unroll 8
                        for (int c = 0; c < C; ++c)
                        {
                                g_sum[c] = 0;
                        }
                        const bool g_full = nc > HELD_OUT;
                        if (g_full)
                        {
                                // create_with_sum (samples/com/create.h:28-55)
                                for (int k = HELD_OUT / 2; k < nc - HELD_OUT / 2; ++k)
                                {
#pragma unroll 8
                                        for (int c = 0; c < C; ++c)
                                        {
                                                g_sum[c] += g.color(k, c);
                                        }
                                        g_wsum += w[color_order[k]];
                                }
                        }
                        merge_color_group(st.color, g, g_sum, g_wsum, g_full);
                }
                if (nbg > 0)
                {
                        // background samples are ordered by value
                        int order[MAX_GROUP];
                        for (int k = 0; k < nbg; ++k)
                        {
                                order[k] = k;
                        }
                        order_group(order, nbg, [&](const int i) { return background[i]; });
                        float sorted[MAX_GROUP];
                        for (int k = 0; k < nbg; ++k)
                        {
                                sorted[k] = background[order[k]];
                        }
                        merge_background_group(st.background, sorted, nbg);
                }
        }
}

template <int N, typename T, int C, typename S>
__global__ void __launch_bounds__(128) accumulate_kernel(
        const Screen<N> screen,
        const long long pixel_count,
        const int spp,
        const T* __restrict__ points,
        const float* __restrict__ colors,
        const float* __restrict__ lum,
        const unsigned char* __restrict__ valid,
        const T alpha,
        const T exp_radius,
        PixelState<C, S>* __restrict__ state)
{
        const long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
        if (t >= pixel_count)
        {
                return;
        }
        PixelState<C, S> st = state[t];
        accumulate_pixel<N, T, C, S>(screen, screen.first + t, spp, points, colors, lum, valid, alpha, exp_radius, st);
        state[t] = st;
}

// RGB accumulation in two kernels: the group of every (source pixel,
// receiving pixel) pair is formed by a thread of its own (group_kernel), then
// every receiving pixel merges its groups in increasing source index
// (merge_groups_kernel).
//
// Forming the groups is nearly all of the work (spp weights of N - 1 filter
// factors each, their ordering and sums, 3^(N-1) times per pixel) and its
// pairs are independent; one thread per pixel did them one after the other,
// which left most of the GPU idle on small screens (4,096 pixels of 81
// samples in 5-space: 10.3 ms) and repeated every factor 3^(N-2) times.  The
// threads of a block share a few sources: a source's factors (three offsets
// per sample and axis) are computed once into shared memory, and a warp's
// lanes read the same samples of the same source.  A group travels as a
// sample set (132-152 bytes).  Those 4,096 pixels now take 0.15 ms to form
// and 0.27 ms to merge, 105,000 of 16 samples 1.2 and 1.4 ms (4.5 before).

// threads of a group_kernel block and the source pixels they share
template <int N>
struct GroupShape final
{
        static constexpr int THREADS = N == 5 ? 256 : 128;
        static constexpr int SOURCES = THREADS / neighbours(N);

        // dynamic shared memory for `sources` source pixels: the filter
        // factors and the samples' order (one byte each, by thread)
        template <typename T>
        static constexpr std::size_t bytes(const int sources, const int spp)
        {
                return static_cast<std::size_t>(spp) * (sources * (N - 1) * 3 * sizeof(T) + THREADS);
        }

        // as many sources as fit in a quarter of an SM's shared memory, at
        // least one (256 samples of 5-space double precision: 87 KB)
        template <typename T>
        static constexpr int sources(const int spp)
        {
                int s = SOURCES;
                while (s > 1 && bytes<T>(s, spp) > 56 * 1024)
                {
                        --s;
                }
                return s;
        }
};

// A thread's column of the shared order array.
struct OrderColumn final
{
        unsigned char* p;
        int stride;

        NBPT_HD unsigned char& operator[](const int i) const
        {
                return p[i * stride];
        }
};

// The sample sets of a group: `nc` colour samples and `nbg` background
// samples of one source pixel, in the order they were taken; weight(j) is
// sample j's.
template <typename S, typename Weight>
__device__ void form_group(const OrderColumn order, const OrderColumn order_bg, const int nc, const int nbg,
                           const Weight& weight, const float* const colors, const float* const lum,
                           PixelState<3, S>& out)
{
        constexpr int C = 3;
        out.color.count = nc < HELD_OUT ? nc : HELD_OUT;
        out.color.full = nc > HELD_OUT ? 1 : 0;
        out.background.count = nbg < HELD_OUT ? nbg : HELD_OUT;
        if (nc > 0)
        {
                order_group(order, nc, [&](const int j) { return weight(j) * lum[j]; });
                S sum[C] = {0, 0, 0};
                S wsum = 0;
                // create_with_sum (samples/com/create.h:28-55)
                for (int k = HELD_OUT / 2; k < nc - HELD_OUT / 2 && nc > HELD_OUT; ++k)
                {
                        const int j = order[k];
                        const float w = weight(j);
#pragma unroll
                        for (int i = 0; i < C; ++i)
                        {
                                sum[i] += w * colors[j * C + i];
                        }
                        wsum += w;
                }
#pragma unroll
                for (int i = 0; i < C; ++i)
                {
                        out.color.color_sum[i] = sum[i];
                }
                out.color.weight_sum = wsum;
                for (int k = 0; k < HELD_OUT && k < nc; ++k)
                {
                        const int j = order[nc > HELD_OUT && k >= HELD_OUT / 2 ? nc - HELD_OUT + k : k];
                        const float w = weight(j);
#pragma unroll
                        for (int i = 0; i < C; ++i)
                        {
                                out.color.colors[k][i] = w * colors[j * C + i];
                        }
                        out.color.weights[k] = w;
                        out.color.contributions[k] = w * lum[j];
                }
        }
        if (nbg > 0)
        {
                // background samples are ordered by value
                order_group(order_bg, nbg, weight);
                BackgroundSet<S> g;
                background_group(g, nbg, [&](const int k) { return weight(order_bg[k]); });
                out.background = g;
        }
}

// Merges a pixel's groups (one per neighbour, in increasing source index,
// the last screen axis outermost) into its state.
template <int N, typename S>
__device__ void merge_groups(const Screen<N>& screen, const int* const tc, const PixelState<3, S>* const groups,
                             PixelState<3, S>& st)
{
        for (int nb = 0; nb < neighbours(N); ++nb)
        {
                int rest = nb;
                bool inside = true;
#pragma unroll
                for (int d = 0; d < N - 1; ++d)
                {
                        const int pc = tc[d] + rest % 3 - 1;
                        rest /= 3;
                        inside = inside && pc >= 0 && pc < screen.size[d];
                }
                if (!inside)
                {
                        continue;
                }
                const PixelState<3, S>& group = groups[nb];
                if (group.color.count > 0)
                {
                        const ColorSet<3, S> g = group.color;
                        merge_color_view<3, S>(st.color, SetView<3, S>{&g, nullptr, 0}, g.color_sum, g.weight_sum,
                                               g.full != 0);
                }
                if (group.background.count > 0)
                {
                        merge_background(st.background, group.background);
                }
        }
}

// Small screens: both steps in one launch, the groups in shared memory.  A
// block takes as many receiving pixels as group_kernel takes sources; a
// thread computes its source's weights itself, since few receiving pixels of
// a block share a source.  Worth it while one block per SM holds the screen:
// the merge runs on a thread per pixel with the block's others idle, and the
// launch and the groups' way through memory are saved (whole renders of one
// pass, two launches against one: 3-space 32^2 x 64 samples 685 -> 675 us,
// 4-space 6^3 x 8 722 -> 658 us, 5-space 4^4 x 16 1,188 -> 1,049 us).
template <int N>
struct SmallScreen final
{
        static constexpr int PIXELS = GroupShape<N>::SOURCES; // per block

        // dynamic shared memory: the groups, then the samples' weights and
        // order by thread
        template <typename S>
        static constexpr std::size_t bytes(const int spp)
        {
                return PIXELS * neighbours(N) * sizeof(PixelState<3, S>) +
                       static_cast<std::size_t>(spp) * GroupShape<N>::THREADS * (sizeof(float) + 1);
        }

        template <typename S>
        static constexpr bool fits(const long long pixels, const int spp, const int sms)
        {
                return pixels <= static_cast<long long>(sms) * PIXELS && bytes<S>(spp) <= 160 * 1024;
        }
};

template <int N, typename T, typename S>
__global__ void __launch_bounds__(GroupShape<N>::THREADS) accumulate_small_kernel(
        const Screen<N> screen,
        const long long pixel_count,
        const int spp,
        const T* __restrict__ points,
        const float* __restrict__ colors,
        const float* __restrict__ lum,
        const unsigned char* __restrict__ valid,
        const T alpha,
        const T exp_radius,
        PixelState<3, S>* __restrict__ state)
{
        constexpr int NB = neighbours(N);
        constexpr int THREADS = GroupShape<N>::THREADS;
        constexpr int PIXELS = SmallScreen<N>::PIXELS;
        extern __shared__ __align__(16) unsigned char group_shared[];
        auto* const groups = reinterpret_cast<PixelState<3, S>*>(group_shared);
        float* const weights = reinterpret_cast<float*>(group_shared + PIXELS * NB * sizeof(PixelState<3, S>));
        unsigned char* const orders = reinterpret_cast<unsigned char*>(weights + static_cast<std::size_t>(spp) * THREADS);
        const auto pixel = [&](const int local, int* const tc)
        {
                const long long t = blockIdx.x * static_cast<long long>(PIXELS) + local;
                long long rest = screen.first + t;
#pragma unroll
                for (int d = 0; d < N - 1; ++d)
                {
                        tc[d] = static_cast<int>(rest % screen.size[d]);
                        rest /= screen.size[d];
                }
                return t;
        };

        const int local = threadIdx.x / NB;
        const int nb = threadIdx.x % NB;
        if (local < PIXELS)
        {
                int tc[N - 1];
                const long long t = pixel(local, tc);
                long long p = 0;
                bool inside = t < pixel_count;
                int offset[N - 1];
                {
                        int rest = nb;
                        int pc[N - 1];
#pragma unroll
                        for (int d = 0; d < N - 1; ++d)
                        {
                                offset[d] = 1 - rest % 3;
                                pc[d] = tc[d] - offset[d];
                                rest /= 3;
                                inside = inside && pc[d] >= 0 && pc[d] < screen.size[d];
                        }
#pragma unroll
                        for (int d = N - 2; d >= 0; --d)
                        {
                                p = p * screen.size[d] + pc[d];
                        }
                }
                if (inside)
                {
                        const long long sample = (p - screen.source_first) * spp;
                        const OrderColumn order{orders + threadIdx.x, THREADS};
                        const OrderColumn order_bg{orders + (spp - 1) * THREADS + threadIdx.x, -THREADS};
                        int nc = 0;
                        int nbg = 0;
                        for (int j = 0; j < spp; ++j)
                        {
                                const T* const v = points + (sample + j) * (N - 1);
                                T weight = 0;
#pragma unroll
                                for (int d = 0; d < N - 1; ++d)
                                {
                                        const T x = (static_cast<T>(offset[d]) + T(0.5)) - v[d];
                                        const T f = max_value(T(0), exp(alpha * x * x) - exp_radius);
                                        weight = d == 0 ? f : weight * f;
                                }
                                if (!(weight > 0))
                                {
                                        continue;
                                }
                                weights[j * THREADS + threadIdx.x] = static_cast<float>(weight);
                                if (valid[sample + j])
                                {
                                        order[nc++] = static_cast<unsigned char>(j);
                                }
                                else
                                {
                                        order_bg[nbg++] = static_cast<unsigned char>(j);
                                }
                        }
                        form_group(order, order_bg, nc, nbg,
                                   [&](const int j) { return weights[j * THREADS + threadIdx.x]; }, colors + sample * 3,
                                   lum + sample, groups[local * NB + nb]);
                }
        }
        __syncthreads();
        if (threadIdx.x < PIXELS)
        {
                int tc[N - 1];
                const long long t = pixel(static_cast<int>(threadIdx.x), tc);
                if (t < pixel_count)
                {
                        PixelState<3, S> st = state[t];
                        merge_groups<N, S>(screen, tc, groups + threadIdx.x * NB, st);
                        state[t] = st;
                }
        }
}

// The groups of the source pixels [source_begin, source_begin +
// source_count) for the receiving pixels [begin, begin + count) (global
// indices); groups: [count][3^(N-1)].
template <int N, typename T, typename S>
__global__ void __launch_bounds__(GroupShape<N>::THREADS) group_kernel(
        const Screen<N> screen,
        const long long begin,
        const long long count,
        const long long source_begin,
        const long long source_count,
        const int sources, // per block
        const int spp,
        const T* __restrict__ points,
        const float* __restrict__ colors,
        const float* __restrict__ lum,
        const unsigned char* __restrict__ valid,
        const T alpha,
        const T exp_radius,
        PixelState<3, S>* __restrict__ groups)
{
        constexpr int NB = neighbours(N);
        constexpr int THREADS = GroupShape<N>::THREADS;
        extern __shared__ __align__(16) unsigned char group_shared[];
        T* const factors = reinterpret_cast<T*>(group_shared); // [source][sample][axis][offset]
        unsigned char* const orders =
                group_shared + static_cast<std::size_t>(sources) * spp * (N - 1) * 3 * sizeof(T); // [sample][thread]

        // pixel_filter.h:57-69, gaussian.h:66-77: the factor of an axis for
        // the receiving pixel one below, at, and one above the source
        const long long first = static_cast<long long>(blockIdx.x) * sources;
        const long long sample_first = (source_begin + first - screen.source_first) * spp;
        const int here = static_cast<int>(min(static_cast<long long>(sources), source_count - first));
        for (int e = threadIdx.x; e < here * spp * (N - 1); e += THREADS)
        {
                const T v = points[sample_first * (N - 1) + e];
#pragma unroll
                for (int o = 0; o < 3; ++o)
                {
                        const T x = (static_cast<T>(o - 1) + T(0.5)) - v;
                        factors[e * 3 + o] = max_value(T(0), exp(alpha * x * x) - exp_radius);
                }
        }
        __syncthreads();

        const int local = threadIdx.x / NB;
        const int nb = threadIdx.x % NB;
        if (local >= here)
        {
                return;
        }
        const long long p = source_begin + first + local;
        // the source is neighbour nb of the receiving pixel: digit d of nb is
        // its offset + 1 along axis d
        long long t = 0;
        int at[N - 1]; // the factors' offsets
        {
                int tc[N - 1];
                long long rest = p;
                int digits = nb;
                bool inside = true;
#pragma unroll
                for (int d = 0; d < N - 1; ++d)
                {
                        const int digit = digits % 3;
                        digits /= 3;
                        tc[d] = static_cast<int>(rest % screen.size[d]) - digit + 1;
                        rest /= screen.size[d];
                        inside = inside && tc[d] >= 0 && tc[d] < screen.size[d];
                        at[d] = d * 3 + 2 - digit;
                }
                if (!inside)
                {
                        return;
                }
#pragma unroll
                for (int d = N - 2; d >= 0; --d)
                {
                        t = t * screen.size[d] + tc[d];
                }
        }
        if (t < begin || t >= begin + count)
        {
                return;
        }

        const long long sample = (p - screen.source_first) * spp;
        const T* const mine = factors + static_cast<std::size_t>(local) * spp * (N - 1) * 3;
        const auto weight = [&](const int j)
        {
                const T* const f = mine + j * ((N - 1) * 3);
                T w = f[at[0]];
#pragma unroll
                for (int d = 1; d < N - 1; ++d)
                {
                        w *= f[at[d]];
                }
                return w;
        };
        const auto weight_float = [&](const int j) { return static_cast<float>(weight(j)); };

        // the selection of colour and background samples (com/select.h:28-47):
        // colour samples from the front of the column, background from its back
        const OrderColumn order{orders + threadIdx.x, THREADS};
        const OrderColumn order_bg{orders + (spp - 1) * THREADS + threadIdx.x, -THREADS};
        int nc = 0;
        int nbg = 0;
        for (int j = 0; j < spp; ++j)
        {
                if (!(weight(j) > 0))
                {
                        continue;
                }
                if (valid[sample + j])
                {
                        order[nc++] = static_cast<unsigned char>(j);
                }
                else
                {
                        order_bg[nbg++] = static_cast<unsigned char>(j);
                }
        }
        form_group(order, order_bg, nc, nbg, weight_float, colors + sample * 3, lum + sample,
                   groups[(t - begin) * NB + nb]);
}

// One thread per receiving pixel: its groups merged in increasing source
// index (the last screen axis outermost).
inline constexpr int MERGE_THREADS = 32;

template <int N, typename S>
__global__ void __launch_bounds__(MERGE_THREADS) merge_groups_kernel(
        const Screen<N> screen,
        const long long begin, // of the receiving pixels, global index
        const long long count,
        const PixelState<3, S>* __restrict__ groups,
        PixelState<3, S>* __restrict__ state) // of the pixels from `begin` on
{
        constexpr int NB = neighbours(N);
        const long long i = blockIdx.x * static_cast<long long>(MERGE_THREADS) + threadIdx.x;
        if (i >= count)
        {
                return;
        }
        int tc[N - 1];
        {
                long long rest = begin + i;
#pragma unroll
                for (int d = 0; d < N - 1; ++d)
                {
                        tc[d] = static_cast<int>(rest % screen.size[d]);
                        rest /= screen.size[d];
                }
        }
        PixelState<3, S> st = state[i];
        merge_groups<N, S>(screen, tc, groups + i * NB, st);
        state[i] = st;
}

// Spectral colours: one warp per receiving pixel.  The lanes compute the
// filter weights of a source's samples in parallel; lane 0 selects and
// orders the group (the scalar part, in shared memory); then every lane runs
// the same merge on the same scalars for its own channels (lane, lane + 32,
// ...), so the merge decisions are the single-thread kernel's and each
// channel's sums are formed in the same order.
template <int N, typename T, int C, typename S>
__global__ void __launch_bounds__(128) accumulate_warp_kernel(
        const Screen<N> screen,
        const long long pixel_count,
        const int spp,
        const T* __restrict__ points,
        const float* __restrict__ colors,
        const float* __restrict__ lum,
        const unsigned char* __restrict__ valid,
        const T alpha,
        const T exp_radius,
        PixelState<C, S>* __restrict__ state)
{
        static_assert(C % 32 == 0);
        constexpr int K = C / 32;
        constexpr int WARPS = 4;
        __shared__ float s_weight[WARPS][MAX_GROUP];
        // the keys of a group's order, which one lane compares (multiplied at each
        // comparison: 10 % longer with 64 or 81 samples, 5-space 5.13 -> 5.69 ms
        // for 10,000 pixels)
        __shared__ float s_contribution[WARPS][MAX_GROUP];
        __shared__ int s_kind[WARPS][MAX_GROUP]; // 0 none, 1 colour, 2 background
        __shared__ int s_order[WARPS][MAX_GROUP];
        __shared__ float s_background[WARPS][MAX_GROUP];
        __shared__ float s_sorted[WARPS][MAX_GROUP];
        __shared__ int s_counts[WARPS][2];

        const int warp = threadIdx.x / 32;
        const int lane = threadIdx.x & 31;
        const long long t = blockIdx.x * static_cast<long long>(WARPS) + warp;
        if (t >= pixel_count)
        {
                return; // the whole warp
        }
        float* const w = s_weight[warp];
        int* const kind = s_kind[warp];
        int* const order = s_order[warp];
        float* const background = s_background[warp];
        float* const sorted = s_sorted[warp];

        // this lane's channels of the pixel state, and its scalars
        PixelState<C, S>& global = state[t];
        ColorSet<K, S> cs;
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
                cs.color_sum[k] = global.color.color_sum[lane + 32 * k];
#pragma unroll
                for (int j = 0; j < HELD_OUT; ++j)
                {
                        cs.colors[j][k] = global.color.colors[j][lane + 32 * k];
                }
        }
        cs.weight_sum = global.color.weight_sum;
#pragma unroll
        for (int j = 0; j < HELD_OUT; ++j)
        {
                cs.weights[j] = global.color.weights[j];
                cs.contributions[j] = global.color.contributions[j];
        }
        cs.count = global.color.count;
        cs.full = global.color.full;
        BackgroundSet<S> bs = global.background;

        int tc[N - 1];
        {
                long long rest = screen.first + t;
#pragma unroll
                for (int d = 0; d < N - 1; ++d)
                {
                        tc[d] = static_cast<int>(rest % screen.size[d]);
                        rest /= screen.size[d];
                }
        }
        int neighbours = 1;
#pragma unroll
        for (int d = 0; d < N - 1; ++d)
        {
                neighbours *= 3;
        }
        for (int nb = 0; nb < neighbours; ++nb)
        {
                int pc[N - 1];
                bool inside = true;
                {
                        int rest = nb;
#pragma unroll
                        for (int d = 0; d < N - 1; ++d)
                        {
                                pc[d] = tc[d] + (rest % 3) - 1;
                                rest /= 3;
                                inside = inside && pc[d] >= 0 && pc[d] < screen.size[d];
                        }
                }
                if (!inside)
                {
                        continue;
                }
                long long p = 0;
#pragma unroll
                for (int d = N - 2; d >= 0; --d)
                {
                        p = p * screen.size[d] + pc[d];
                }
                // weights and selection (pixel_filter.h:57-69, com/select.h:28-47)
                for (int j = lane; j < spp; j += 32)
                {
                        const long long sidx = (p - screen.source_first) * spp + j;
                        const T x0 = (static_cast<T>(tc[0] - pc[0]) + T(0.5)) - points[sidx * (N - 1)];
                        T weight = max_value(T(0), exp(alpha * x0 * x0) - exp_radius);
#pragma unroll
                        for (int d = 1; d < N - 1; ++d)
                        {
                                const T x = (static_cast<T>(tc[d] - pc[d]) + T(0.5)) - points[sidx * (N - 1) + d];
                                weight *= max_value(T(0), exp(alpha * x * x) - exp_radius);
                        }
                        int k = 0;
                        if (weight > 0)
                        {
                                const float wf = static_cast<float>(weight);
                                w[j] = wf;
                                k = valid[sidx] ? 1 : 2;
                                s_contribution[warp][j] = wf * lum[sidx];
                        }
                        kind[j] = k;
                }
                __syncwarp();
                if (lane == 0)
                {
                        int nc = 0;
                        int nbg = 0;
                        for (int j = 0; j < spp; ++j)
                        {
                                if (kind[j] == 1)
                                {
                                        order[nc++] = j;
                                }
                                else if (kind[j] == 2)
                                {
                                        background[nbg++] = w[j];
                                }
                        }
                        const float* const source_lum = lum + (p - screen.source_first) * spp;
                        order_group(order, nc, [&](const int i) { return s_contribution[warp][i]; });
                        if (nbg > 1)
                        {
                                // background samples are ordered by value; reuse
                                // `kind` as the index array of the ordering
                                int* const index = kind;
                                for (int j = 0; j < nbg; ++j)
                                {
                                        index[j] = j;
                                }
                                order_group(index, nbg, [&](const int i) { return background[i]; });
                                for (int j = 0; j < nbg; ++j)
                                {
                                        sorted[j] = background[index[j]];
                                }
                        }
                        else if (nbg == 1)
                        {
                                sorted[0] = background[0];
                        }
                        s_counts[warp][0] = nc;
                        s_counts[warp][1] = nbg;
                }
                __syncwarp();
                const int nc = s_counts[warp][0];
                const int nbg = s_counts[warp][1];
                if (nc > 0)
                {
                        const float* const source_lum = lum + (p - screen.source_first) * spp;
                        const ColorGroup<K> g{colors + (p - screen.source_first) * spp * C, w, source_lum, order, nc, C, 32, lane};
                        S g_sum[K];
                        S g_wsum = 0;
#pragma unroll
                        for (int k = 0; k < K; ++k)
                        {
                                g_sum[k] = 0;
                        }
                        const bool g_full = nc > HELD_OUT;
                        if (g_full)
                        {
                                sum_group(g, g_sum, g_wsum);
                        }
                        merge_color_group(cs, g, g_sum, g_wsum, g_full);
                }
                if (nbg > 0)
                {
                        merge_background_group(bs, sorted, nbg);
                }
                __syncwarp();
        }
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
                global.color.color_sum[lane + 32 * k] = cs.color_sum[k];
#pragma unroll
                for (int j = 0; j < HELD_OUT; ++j)
                {
                        global.color.colors[j][lane + 32 * k] = cs.colors[j][k];
                }
        }
        if (lane == 0)
        {
                global.color.weight_sum = cs.weight_sum;
#pragma unroll
                for (int j = 0; j < HELD_OUT; ++j)
                {
                        global.color.weights[j] = cs.weights[j];
                        global.color.contributions[j] = cs.contributions[j];
                }
                global.color.count = cs.count;
                global.color.full = cs.full;
                global.background = bs;
        }
}

// The same merge with the scalar work of the neighbours done side by side,
// for up to 32 samples per pixel: one warp per receiving pixel; first the
// weights of every neighbour's samples (lanes over samples), then every
// neighbour's group ordered on its own lane, then the groups merged in
// increasing pixel index with the channels across the lanes, as
// accumulate_warp_kernel merges them.
inline constexpr int SMALL_GROUP = 32;

template <int N, typename T, int C, typename S>
__global__ void __launch_bounds__(128) accumulate_warp_small_kernel(
        const Screen<N> screen,
        const long long pixel_count,
        const int spp,
        const T* __restrict__ points,
        const float* __restrict__ colors,
        const float* __restrict__ lum,
        const unsigned char* __restrict__ valid,
        const T alpha,
        const T exp_radius,
        PixelState<C, S>* __restrict__ state)
{
        static_assert(C % 32 == 0);
        constexpr int K = C / 32;
        constexpr int WARPS = 4;
        static_assert(N <= 4, "the shared-memory tables hold 3^(N-1) <= 27 neighbours");
        constexpr int NB = N == 3 ? 9 : 27;
        __shared__ float s_weight[WARPS][NB][SMALL_GROUP];
        __shared__ unsigned char s_kind[WARPS][NB][SMALL_GROUP]; // 0 none, 1 colour, 2 background
        __shared__ unsigned char s_order[WARPS][NB][SMALL_GROUP];
        __shared__ unsigned char s_order_bg[WARPS][NB][SMALL_GROUP];
        __shared__ int s_counts[WARPS][NB][2];
        __shared__ int s_order_int[WARPS][SMALL_GROUP];
        __shared__ float s_sorted[WARPS][SMALL_GROUP];

        const int warp = threadIdx.x / 32;
        const int lane = threadIdx.x & 31;
        const long long t = blockIdx.x * static_cast<long long>(WARPS) + warp;
        if (t >= pixel_count)
        {
                return; // the whole warp
        }

        int tc[N - 1];
        {
                long long rest = screen.first + t;
#pragma unroll
                for (int d = 0; d < N - 1; ++d)
                {
                        tc[d] = static_cast<int>(rest % screen.size[d]);
                        rest /= screen.size[d];
                }
        }
        // neighbour nb's pixel, or -1 outside the screen
        const auto neighbour = [&](const int nb, int* pc) -> long long
        {
                int rest = nb;
                bool inside = true;
#pragma unroll
                for (int d = 0; d < N - 1; ++d)
                {
                        pc[d] = tc[d] + (rest % 3) - 1;
                        rest /= 3;
                        inside = inside && pc[d] >= 0 && pc[d] < screen.size[d];
                }
                if (!inside)
                {
                        return -1;
                }
                long long p = 0;
#pragma unroll
                for (int d = N - 2; d >= 0; --d)
                {
                        p = p * screen.size[d] + pc[d];
                }
                return p;
        };

        // weights and kinds (pixel_filter.h:57-69), lanes over the samples
        for (int nb = 0; nb < NB; ++nb)
        {
                int pc[N - 1];
                const long long p = neighbour(nb, pc);
                if (p < 0 || lane >= spp)
                {
                        continue;
                }
                const int j = lane;
                const long long sidx = (p - screen.source_first) * spp + j;
                const T x0 = (static_cast<T>(tc[0] - pc[0]) + T(0.5)) - points[sidx * (N - 1)];
                T weight = max_value(T(0), exp(alpha * x0 * x0) - exp_radius);
#pragma unroll
                for (int d = 1; d < N - 1; ++d)
                {
                        const T x = (static_cast<T>(tc[d] - pc[d]) + T(0.5)) - points[sidx * (N - 1) + d];
                        weight *= max_value(T(0), exp(alpha * x * x) - exp_radius);
                }
                unsigned char k = 0;
                if (weight > 0)
                {
                        const float wf = static_cast<float>(weight);
                        s_weight[warp][nb][j] = wf;
                        k = valid[sidx] ? 1 : 2;
                }
                s_kind[warp][nb][j] = k;
        }
        __syncwarp();

        // every neighbour's group ordered on its own lane (com/select.h:28-47,
        // samples/com/sort.h:26-46)
        if (lane < NB)
        {
                const int nb = lane;
                int pc[N - 1];
                const long long p = neighbour(nb, pc);
                int nc = 0;
                int nbg = 0;
                if (p >= 0)
                {
                        int order[SMALL_GROUP];
                        int order_bg[SMALL_GROUP];
                        for (int j = 0; j < spp; ++j)
                        {
                                const unsigned char k = s_kind[warp][nb][j];
                                if (k == 1)
                                {
                                        order[nc++] = j;
                                }
                                else if (k == 2)
                                {
                                        order_bg[nbg++] = j;
                                }
                        }
                        const float* const source_lum = lum + (p - screen.source_first) * spp;
                        const float* const w = s_weight[warp][nb];
                        order_group(order, nc, [&](const int i) { return w[i] * source_lum[i]; });
                        order_group(order_bg, nbg, [&](const int i) { return w[i]; });
                        for (int k = 0; k < nc; ++k)
                        {
                                s_order[warp][nb][k] = static_cast<unsigned char>(order[k]);
                        }
                        for (int k = 0; k < nbg; ++k)
                        {
                                s_order_bg[warp][nb][k] = static_cast<unsigned char>(order_bg[k]);
                        }
                }
                s_counts[warp][nb][0] = nc;
                s_counts[warp][nb][1] = nbg;
        }
        __syncwarp();

        // this lane's channels of the pixel state, and its scalars
        PixelState<C, S>& global = state[t];
        ColorSet<K, S> cs;
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
                cs.color_sum[k] = global.color.color_sum[lane + 32 * k];
#pragma unroll
                for (int j = 0; j < HELD_OUT; ++j)
                {
                        cs.colors[j][k] = global.color.colors[j][lane + 32 * k];
                }
        }
        cs.weight_sum = global.color.weight_sum;
#pragma unroll
        for (int j = 0; j < HELD_OUT; ++j)
        {
                cs.weights[j] = global.color.weights[j];
                cs.contributions[j] = global.color.contributions[j];
        }
        cs.count = global.color.count;
        cs.full = global.color.full;
        BackgroundSet<S> bs = global.background;

        int* const order = s_order_int[warp];
        float* const sorted = s_sorted[warp];
        for (int nb = 0; nb < NB; ++nb)
        {
                const int nc = s_counts[warp][nb][0];
                const int nbg = s_counts[warp][nb][1];
                if (nc == 0 && nbg == 0)
                {
                        continue;
                }
                int pc[N - 1];
                const long long p = neighbour(nb, pc);
                const float* const w = s_weight[warp][nb];
                if (lane < nc)
                {
                        order[lane] = s_order[warp][nb][lane];
                }
                if (lane < nbg)
                {
                        sorted[lane] = w[s_order_bg[warp][nb][lane]];
                }
                __syncwarp();
                if (nc > 0)
                {
                        const float* const source_lum = lum + (p - screen.source_first) * spp;
                        const ColorGroup<K> g{colors + (p - screen.source_first) * spp * C, w, source_lum, order, nc, C, 32, lane};
                        S g_sum[K];
                        S g_wsum = 0;
#pragma unroll
                        for (int k = 0; k < K; ++k)
                        {
                                g_sum[k] = 0;
                        }
                        const bool g_full = nc > HELD_OUT;
                        if (g_full)
                        {
                                sum_group(g, g_sum, g_wsum);
                        }
                        merge_color_group(cs, g, g_sum, g_wsum, g_full);
                }
                if (nbg > 0)
                {
                        merge_background_group(bs, sorted, nbg);
                }
                __syncwarp();
        }
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
                global.color.color_sum[lane + 32 * k] = cs.color_sum[k];
#pragma unroll
                for (int j = 0; j < HELD_OUT; ++j)
                {
                        global.color.colors[j][lane + 32 * k] = cs.colors[j][k];
                }
        }
        if (lane == 0)
        {
                global.color.weight_sum = cs.weight_sum;
#pragma unroll
                for (int j = 0; j < HELD_OUT; ++j)
                {
                        global.color.weights[j] = cs.weights[j];
                        global.color.contributions[j] = cs.contributions[j];
                }
                global.color.count = cs.count;
                global.color.full = cs.full;
                global.background = bs;
        }
}

// ---------------------------------------------------------------------------
// image resolve: merge_color / merge_color_alpha (samples/merge_color.cpp:45-177)
// and the RGB of the colour (src/color/color.h rgb32).  The background is
// black: its colour and contribution are 0.

template <int C, typename S>
struct Resolved final
{
        bool has;
        S color[C];
        S color_weight;
        S background_weight;
};

template <int C, typename S>
NBPT_HD Resolved<C, S> resolve_pixel(const PixelState<C, S>& st)
{
        Resolved<C, S> res;
        res.has = false;
        const ColorSet<C, S>& a = st.color;
        const BackgroundSet<S>& b = st.background;
        const int a_size = a.full ? HELD_OUT : a.count;
        const int b_size = b.full ? HELD_OUT : b.count;
        if (a_size + b_size <= HELD_OUT)
        {
                if (a_size == 0 || b_size != 0 || !a.full)
                {
                        return res;
                }
                res.has = true;
#pragma unroll 8
                for (int c = 0; c < C; ++c)
                {
                        res.color[c] = a.color_sum[c];
                }
                res.color_weight = a.weight_sum;
                res.background_weight = 0;
                return res;
        }
        res.has = true;
#pragma unroll 8
        for (int c = 0; c < C; ++c)
        {
                res.color[c] = a.full ? a.color_sum[c] : S(0);
        }
        res.color_weight = a.full ? a.weight_sum : S(0);
        res.background_weight = b.full ? b.weight_sum : S(0);

        const auto a_key = [&](const int i)
        {
                return a.contributions[i];
        };
        const auto b_key = [&](const int i)
        {
                return b.weights[i] * 0.0f;
        };
        const auto sum_a = [&](const int i)
        {
#pragma unroll 8
                for (int c = 0; c < C; ++c)
                {
                        res.color[c] += a.colors[i][c];
                }
                res.color_weight += a.weights[i];
        };
        const auto sum_b = [&](const int i)
        {
                res.background_weight += b.weights[i];
        };
        if (a_size == HELD_OUT && b_size == HELD_OUT)
        {
                int ai = 0;
                int bi = 0;
                for (int i = 0; i < HELD_OUT / 2; ++i)
                {
                        if (a_key(ai) < b_key(bi))
                        {
                                ++ai;
                        }
                        else
                        {
                                ++bi;
                        }
                }
                while (ai < HELD_OUT / 2)
                {
                        sum_a(ai++);
                }
                while (bi < HELD_OUT / 2)
                {
                        sum_b(bi++);
                }
                ai = HELD_OUT - 1;
                bi = HELD_OUT - 1;
                for (int i = HELD_OUT - 1; i >= HELD_OUT / 2; --i)
                {
                        if (a_key(ai) > b_key(bi))
                        {
                                --ai;
                        }
                        else
                        {
                                --bi;
                        }
                }
                while (ai >= HELD_OUT / 2)
                {
                        sum_a(ai--);
                }
                while (bi >= HELD_OUT / 2)
                {
                        sum_b(bi--);
                }
                return res;
        }
        int ai = 0;
        int bi = 0;
        int i = 0;
        while (i < HELD_OUT / 2 && ai < a_size && bi < b_size)
        {
                if (a_key(ai) < b_key(bi))
                {
                        ++ai;
                }
                else
                {
                        ++bi;
                }
                ++i;
        }
        while (i < HELD_OUT / 2 && ai < a_size)
        {
                ++ai;
                ++i;
        }
        while (i < HELD_OUT / 2 && bi < b_size)
        {
                ++bi;
                ++i;
        }
        const int a_low = ai;
        const int b_low = bi;
        int aj = a_size - 1;
        int bj = b_size - 1;
        int j = HELD_OUT - 1;
        while (j >= HELD_OUT / 2 && aj >= a_low && bj >= b_low)
        {
                if (a_key(aj) > b_key(bj))
                {
                        --aj;
                }
                else
                {
                        --bj;
                }
                --j;
        }
        while (j >= HELD_OUT / 2 && aj >= a_low)
        {
                --aj;
                --j;
        }
        while (j >= HELD_OUT / 2 && bj >= b_low)
        {
                --bj;
                --j;
        }
        for (int k = a_low; k <= aj; ++k)
        {
                sum_a(k);
        }
        for (int k = b_low; k <= bj; ++k)
        {
                sum_b(k);
        }
        return res;
}

// The pixel's RGB and premultiplied RGBA (pixel.h:51-88, color.h rgb32); with
// double sums the division by the weight is in double and the colour is then
// rounded to float.
template <int C, typename S>
NBPT_HD void resolve_rgb(const PixelState<C, S>& state, const float* xyz, float* rgb, float* rgba)
{
        const Resolved<C, S> r = resolve_pixel(state);
        float out[3] = {0.0f, 0.0f, 0.0f};
        float out_a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (r.has)
        {
                const S sum = r.color_weight + r.background_weight;
                float color[C];
#pragma unroll 8
                for (int c = 0; c < C; ++c)
                {
                        color[c] = static_cast<float>(r.color[c] / sum);
                }
                float c_rgb[3];
                if constexpr (C == 3)
                {
                        c_rgb[0] = max_value(0.0f, color[0]);
                        c_rgb[1] = max_value(0.0f, color[1]);
                        c_rgb[2] = max_value(0.0f, color[2]);
                }
                else
                {
                        float v[3];
                        for (int k = 0; k < 3; ++k)
                        {
                                const float* f = xyz + k * 64;
                                float s = max_value(0.0f, color[0]) * f[0];
                                for (int c = 1; c < C; ++c)
                                {
                                        s += max_value(0.0f, color[c]) * f[c];
                                }
                                v[k] = s;
                        }
                        c_rgb[0] = max_value(0.0f, 3.2406255f * v[0] + -1.5372080f * v[1] + -0.4986286f * v[2]);
                        c_rgb[1] = max_value(0.0f, -0.9689307f * v[0] + 1.8757561f * v[1] + 0.0415175f * v[2]);
                        c_rgb[2] = max_value(0.0f, 0.0557101f * v[0] + -0.2040211f * v[1] + 1.0569959f * v[2]);
                }
                const bool background_only =
                        !(r.color_weight == sum || (r.color_weight / sum) == 1) &&
                        (r.background_weight == sum || (r.background_weight / sum) == 1);
                if (!background_only)
                {
                        out[0] = c_rgb[0];
                        out[1] = c_rgb[1];
                        out[2] = c_rgb[2];
                }
                if (r.color_weight != 0)
                {
                        out_a[0] = c_rgb[0];
                        out_a[1] = c_rgb[1];
                        out_a[2] = c_rgb[2];
                        out_a[3] = static_cast<float>(r.color_weight / sum);
                }
        }
        rgb[0] = out[0];
        rgb[1] = out[1];
        rgb[2] = out[2];
        if (rgba)
        {
                rgba[0] = out_a[0];
                rgba[1] = out_a[1];
                rgba[2] = out_a[2];
                rgba[3] = out_a[3];
        }
}

template <int C, typename S>
__global__ void resolve_kernel(
        const long long pixel_count,
        const PixelState<C, S>* __restrict__ state,
        const float* __restrict__ xyz, // [3][64] colour matching functions (spectrum only)
        float* __restrict__ rgb,
        float* __restrict__ rgba)
{
        const long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
        if (t >= pixel_count)
        {
                return;
        }
        resolve_rgb<C, S>(state[t], xyz, rgb + t * 3, rgba ? rgba + t * 4 : nullptr);
}
} // namespace nbpt
