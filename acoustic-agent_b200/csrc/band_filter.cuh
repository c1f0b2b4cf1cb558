// The crossover recursion of bandlimit_band_signals (acoustic_agent/steam_rt.py
// :3070-3083, :4131-4212).  A band signal passes one or two eight-pole
// low-passes (bands 1-4: the one at the upper crossover less the one at the
// lower; band 0 the upper alone; band 5 the signal less the lower), each four
// biquad sections in a row that hand on float32-rounded signals:
//
//     y0 = b0*x0 + b1*x1 + b2*x2 - a1*y1 - a2*y2, evaluated left to right.
//
// Included by every translation unit that band-limits signals; each of them is
// compiled with -fmad=false, so the float64 arithmetic rounds operation by
// operation like the reference's and the outputs are its bits.
//
// What bounds it: the order of the operations is fixed, so a section's state
// costs three dependent float64 operations per sample, (v - a1*y1) - a2*y2, of
// 8.3 cycles each (25 cycles), whatever else runs beside it.  Everything that
// is not this chain is therefore taken off it: one block carries kSignals
// signals through all sections, with a warp for each job, in steps of
// kStep samples between block barriers:
//
//   recursion warp s (one per scheduler): section s of every chain, one chain
//       per lane; per sample a load of the input part v, the two products, the
//       two differences, the rounding and a store -- nothing is exchanged
//       between lanes and nothing waits inside a step but the chain itself;
//   input warp(s) s: the input part v = (b0*x0 + b1*x1) + b2*x2 of section s,
//       which does not depend on y, for all samples of a step in parallel;
//   loader warp: the next steps' signals, by cp.async;
//   output warp: the bands from the last section's outputs, coalesced.
//
// Section s runs two steps behind section s - 1 (input part, recursion).  One
// RIR of 96,000 samples (10 chains), or eight of them on eight SMs, takes 1.70 ms
// (35 cycles per sample) against 7.3 ms (150 cycles) for one warp per four bands
// with a lane per section and shuffles between the sections.  The recursion
// warp alone, without the others on its scheduler, runs at 29 cycles.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "common.h"
#include "filter_steps.h"

namespace ac {
namespace {

constexpr int kSections = 4;
// Signals per SM up to which each gets a block of its own.  A wide block (30 chains in the recursion lanes) takes 59
// cycles per sample whatever it carries, a block of one signal 36, or 45 with two of them on an SM, which share the
// float64 and conversion pipes; a third would make it 66.
constexpr int kFilterNarrowPerSm = 2;
constexpr int kFilterLag = 2 * kSections;   // steps between the input part of section 0 and the outputs

// One signal of a block: its band rows, `band_stride` apart (0: all bands share one row), and its outputs [6, n_len].
struct FilterSignal {
    const double *x;
    int64_t band_stride;
    float *out;
    const double *crossover;   // [5 cutoffs][4 sections][5 coefficients]
    int n_len;                 // 0: no signal in this place (the pointers are then another's, and nothing is read)
};

// kShared: the six bands share one input row, so the low-pass at a crossover is one chain for the two bands it
// separates (5 chains per signal instead of 10).
template <int kSignals, bool kShared>
struct FilterShape {
    static constexpr int kChains = kShared ? 5 : 10;
    static constexpr int kInputs = kShared ? 1 : 6;
    static constexpr int kLanes = kSignals * kChains;            // chains of the block
    static constexpr int kWidth = kSignals * kInputs;            // input rows of the block
    static constexpr int kXPitch = kWidth | 1;                   // odd pitches: a column has no bank conflicts
    static constexpr int kYPitch = kLanes | 1;
    static constexpr int kRowsAtOnce = 32 / kLanes;              // lanes of an input warp that share a chain
    static constexpr int kInputWarps = kLanes > 16 ? 2 : 1;      // per section
    // samples between two block barriers: a barrier and the refill of the recursion after it cost about 200 cycles;
    // 64 (36.0 cycles per sample, 39.5 with 32) where two blocks of one signal then still fit an SM's shared memory
    static constexpr int kStep = kSignals == 1 ? 64 : 32;
    static constexpr int kRows = 4 * kStep;   // ring rows: the step being written, the one read and its history
    static constexpr int kThreads = 32 * (kSections * (1 + kInputWarps) + 2);
    static_assert(kLanes <= 32, "one chain per lane");
};

template <int kSignals, bool kShared>
struct FilterSmem {
    using Shape = FilterShape<kSignals, kShared>;
    double x[Shape::kRows][Shape::kXPitch];
    double v[kSections][2][Shape::kStep][Shape::kLanes];
    float y[kSections][Shape::kRows][Shape::kYPitch];
};

__device__ __forceinline__ void cp_async8_zfill(double *dst, const double *src, bool valid) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    const int bytes = valid ? 8 : 0;   // past the end of the signal: zeros, and nothing is read
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(s), "l"(src), "r"(bytes) : "memory");
}

// All warps of the block meet here once per step.
template <int kThreads>
__device__ __forceinline__ void filter_barrier() {
    __syncwarp();
    asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");
}

// The whole block filters `signals[0 .. kSignals)`, which lie in shared memory.
template <int kSignals, bool kShared>
__device__ __forceinline__ void filter_block(const FilterSignal *signals, FilterSmem<kSignals, kShared> &m) {
    using Shape = FilterShape<kSignals, kShared>;
    constexpr int kLanes = Shape::kLanes, kChains = Shape::kChains, kInputs = Shape::kInputs;
    constexpr int kStep = Shape::kStep, kRows = Shape::kRows;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int longest = 0;
#pragma unroll
    for (int j = 0; j < kSignals; ++j) longest = max(longest, signals[j].n_len);
    const int blocks = filter_steps(longest, kStep);
    {   // the history before the first sample is +0.0
        unsigned *words = reinterpret_cast<unsigned *>(&m);
        for (int i = threadIdx.x; i < static_cast<int>(sizeof(m) / 4); i += Shape::kThreads) words[i] = 0u;
    }
    __syncthreads();

    const int input_first = kSections, loader = kSections * (1 + Shape::kInputWarps);
    auto load = [&](int k) {   // loader warp: step k's samples, lane = sample
#pragma unroll
        for (int jh = 0; jh < kSignals * (kStep / 32); ++jh) {
            const int j = jh / (kStep / 32);
            const unsigned n = filter_sample(k, kStep, jh % (kStep / 32) * 32 + lane);
            const FilterSignal sg = signals[j];
            const bool valid = in_signal(n, sg.n_len);
            const double *p = sg.x + (valid ? n : 0u);
#pragma unroll
            for (int b = 0; b < kInputs; ++b)
                cp_async8_zfill(&m.x[n & (kRows - 1)][j * kInputs + b], p + b * sg.band_stride, valid);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (warp == loader) {
        load(0);
        load(1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");   // step 0's samples are there
    }
    filter_barrier<Shape::kThreads>();
    const int steps = blocks + kFilterLag;
    // chain of this lane: signal, cutoff and input row
    const bool recursion = warp < kSections;
    const int slot = recursion ? lane : lane % kLanes;
    const bool has_chain = recursion ? lane < kLanes : lane < Shape::kRowsAtOnce * kLanes;
    const int chain_signal = has_chain ? slot / kChains : 0, chain = has_chain ? slot % kChains : 0;
    const int cutoff = chain < 5 ? chain : chain - 5;
    const int input = kShared ? chain_signal : chain_signal * kInputs + (chain < 5 ? chain : chain - 4);

    if (recursion) {
        const int s = warp;
        const double *co = signals[chain_signal].crossover + cutoff * 20 + s * 5;
        const double a1 = co[3], a2 = co[4];
        double y1 = 0.0, y2 = 0.0;
        for (int i = 0; i < steps; ++i) {
            const int k = i - 1 - 2 * s;
            if (k >= 0 && k < blocks && has_chain) {
                const double *vp = &m.v[s][k & 1][0][lane];
                float *yp = &m.y[s][filter_sample(k, kStep, 0) & (kRows - 1)][lane];
                double v[8], next[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = vp[u * kLanes];
#pragma unroll
                for (int base = 0; base < kStep; base += 8) {
                    if (base + 8 < kStep) {
#pragma unroll
                        for (int u = 0; u < 8; ++u) next[u] = vp[(base + 8 + u) * kLanes];
                    }
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const double y0 = v[u] - a1 * y1 - a2 * y2;
                        y2 = y1;
                        y1 = y0;
                        yp[(base + u) * Shape::kYPitch] = static_cast<float>(y0);
                    }
#pragma unroll
                    for (int u = 0; u < 8; ++u) v[u] = next[u];
                }
            }
            filter_barrier<Shape::kThreads>();
        }
    } else if (warp < loader) {
        const int s = (warp - input_first) / Shape::kInputWarps, part = (warp - input_first) % Shape::kInputWarps;
        const double *co = signals[chain_signal].crossover + cutoff * 20 + s * 5;
        const double b0 = co[0], b1 = co[1], b2 = co[2];
        // a lane takes kRun samples in a row of its chain: each value is loaded and widened once, and all loads of a
        // step are issued before the first of them is used (one after another, a step of them took as long as the
        // recursion itself)
        constexpr int kShare = kStep / Shape::kInputWarps;   // samples of this warp per step
        constexpr int kRun = (kShare + Shape::kRowsAtOnce - 1) / Shape::kRowsAtOnce;
        const int run = lane / kLanes * kRun, first = part * kShare + run;
        for (int i = 0; i < steps; ++i) {
            const int k = i - 2 * s;
            if (k >= 0 && k < blocks && has_chain) {
                const unsigned n = filter_sample(k, kStep, first);
                double *vp = &m.v[s][k & 1][first][slot];
                double x[kRun + 2];   // x[u + 2]: sample n + u
                if (s == 0) {
#pragma unroll
                    for (int u = 0; u < kRun + 2; ++u)
                        x[u] = run + u - 2 < kShare ? m.x[(n + u - 2) & (kRows - 1)][input] : 0.0;
                } else {
                    float f[kRun + 2];
#pragma unroll
                    for (int u = 0; u < kRun + 2; ++u)
                        f[u] = run + u - 2 < kShare ? m.y[s - 1][(n + u - 2) & (kRows - 1)][slot] : 0.0f;
#pragma unroll
                    for (int u = 0; u < kRun + 2; ++u) x[u] = static_cast<double>(f[u]);
                }
                double v[kRun];
#pragma unroll
                for (int u = 0; u < kRun; ++u) v[u] = b0 * x[u + 2] + b1 * x[u + 1] + b2 * x[u];
#pragma unroll
                for (int u = 0; u < kRun; ++u)
                    if (run + u < kShare) vp[u * kLanes] = v[u];
            }
            filter_barrier<Shape::kThreads>();
        }
    } else if (warp == loader) {
        for (int i = 0; i < steps; ++i) {
            load(i + 2);
            asm volatile("cp.async.wait_group 1;" ::: "memory");   // step i + 1's samples are there
            filter_barrier<Shape::kThreads>();
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    } else {
        for (int i = 0; i < steps; ++i) {
            const int k = i - kFilterLag;
            if (k >= 0) {
#pragma unroll
                for (int jh = 0; jh < kSignals * (kStep / 32); ++jh) {
                    const int j = jh / (kStep / 32);
                    const unsigned n = filter_sample(k, kStep, jh % (kStep / 32) * 32 + lane);
                    const FilterSignal sg = signals[j];
                    if (in_signal(n, sg.n_len)) {
                        const double x5 = __ldg(sg.x + 5 * sg.band_stride + n);
                        const float *y = &m.y[kSections - 1][n & (kRows - 1)][j * kChains];
                        const float *lower = kShared ? y : y + 5;   // lower[b - 1]: band b's lower low-pass
                        float *out = sg.out + n;
                        const size_t row = static_cast<size_t>(sg.n_len);
                        out[0] = y[0];
#pragma unroll
                        for (int b = 1; b < 5; ++b) out[b * row] = y[b] - lower[b - 1];
                        out[5 * row] = static_cast<float>(x5 - static_cast<double>(lower[4]));
                    }
                }
            }
            filter_barrier<Shape::kThreads>();
        }
    }
}

// Opts a filter kernel into its dynamic shared memory on the current device.
template <class Kernel>
inline int filter_smem(Kernel kernel, size_t bytes) {
    AC_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)));
    return AC_OK;
}

// Calls launch(std::integral_constant<int, signals per block>, blocks) for a batch of `count` signals.
template <int kWide, class Launch>
inline int with_filter_signals(int count, Launch launch) {
    int device = 0, sms = 0;
    AC_CUDA_TRY(cudaGetDevice(&device));
    AC_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    if (count <= kFilterNarrowPerSm * sms) return launch(std::integral_constant<int, 1>{}, count);
    return launch(std::integral_constant<int, kWide>{}, (count + kWide - 1) / kWide);
}

}  // namespace
}  // namespace ac
