// Late reverberation on the GPU: the sixteen-line FDN impulse response and the
// hybrid late tail of acoustic_agent/steam_rt.py:2235-2640.
//
// ac_fdn_impulse restates _fdn_impulse_kernel (:2235-2327) so that every output
// sample is bit-identical to the reference's float64 kernel: this file is
// compiled with -fmad=false and every expression keeps the reference's
// operation order.  The network is sequential in time, but its feedback runs
// through delay lines of at least AC_FDN_MIN_DELAY samples, so nothing a
// sample computes is needed by the next hundred samples except each biquad's
// own state.  What bounds it is that state, ((S - a1*y1) - a2*y2): three
// dependent float64 operations of 8.3 cycles per sample (25 cycles).  One
// 256-thread block renders one impulse response in steps of S samples, a job
// per warp, one recursion warp per scheduler:
//
//   warps 0-2: the 96 absorptive sections, one per lane, sixteen lines of two
//       bands per warp, each S samples in a row from one column of shared
//       memory to the next (Biquad::run);
//   warp 3: the six sections of the output cascade, a lane each;
//   warp 4: the Hadamard mix and the delay lines' new samples (global memory,
//       L2-resident, coalesced per line), lane i taking sample i of the step
//       (in short steps two lanes a sample, eight lines each);
//   warp 5: the sum of the line outputs and the four all-pass stages (their
//       delays are S or more, so a step's samples are independent);
//   warp 6: the delay lines' next samples;
//   warp 7: the output.
//
// Band b + 1 runs one step behind band b, so a sample's feedback is written in
// the sixth step after its first section's, and the step size is picked to fit
// the shortest delay (fdn_step).  8 impulses of 121,952 samples (48 kHz, S = 64):
// 2.47 ms (43 cycles per sample) against 4.3 ms (76) with shuffles between the
// bands of a line in every sample and a barrier every 32; 256 of 30,000 samples
// (16 kHz, S = 32, two blocks per SM) 1.35 ms against 1.94, 1,184 of them 6.1
// against 8.1, where the shared-memory pipe is 66 % busy.  In short steps what
// bounds it is the mix and the loads, some 700 cycles whatever the step: one
// impulse of 16,000 samples with delays from 144 takes 0.525 ms (S = 16, 64
// cycles per sample), from 128 0.575 (S = 14, 71), against 0.648.  Input parts
// on warps of their own, as in band_filter.cuh, took 44 cycles: they double the
// shared-memory traffic, which with 96 sections is then what bounds the step.
//
// ac_late_tail restates the rest of _render_parametric_fdn_late_reverb
// (:2588-2640): bandlimit_band_signals of the impulse (the crossover filter
// of band_filter.cuh, bit-identical), then one block per (RIR, band)
// measures the traced power at the anchor (_late_tail_start_power,
// :2473-2497), scales the FDN band to the target energy and writes the
// equal-power crossfade.  Its sums run in a fixed order but not numpy's
// pairwise order, so scales agree with the reference to about 1e-15 relative.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include <cuda_runtime.h>

#include "band_filter.cuh"
#include "common.h"

namespace ac {
namespace {

constexpr int kLines = AC_FDN_LINES;
constexpr int kBandSections = 6;
constexpr int kTonePitch = kBandSections + 1;
constexpr int kMinAllpass = 32;   // all-pass delays must exceed this

inline size_t align256(size_t v) { return (v + 255) & ~static_cast<size_t>(255); }

struct FdnJobDev {
    double absorptive[kLines][6][5];
    double tone[6][5];
    int32_t delays[kLines];
    int32_t line_start[kLines];     // offset of each delay line within this job's lines
    int32_t allpass[AC_FDN_ALLPASS];
    int32_t allpass_start[AC_FDN_ALLPASS];  // offsets of the all-pass rings in shared memory
    int32_t num_samples;
    int32_t preroll;
    double *out;
    int64_t pool;                   // offset of this job's delay lines in the workspace pool (doubles)
};

// A delay line as the loader and the mix see it: its offset in the pool, its length, and the position of the first
// sample of their next step.
struct FdnLine {
    int start, delay, pos, pad;
};

// Steps of S samples.  Each buffer is doubled: what one warp writes in a step others read in the next.
template <int S>
struct FdnSmem {
    // columns: the delay lines' samples, then the outputs of bands 0 .. 5, sixteen lines each (an odd pitch: the mix
    // reads rows per lane)
    static constexpr int kPitch = kLines * (1 + kBandSections) + 1;
    double y[2][S][kPitch];
    double t[2][S][kTonePitch];            // [0]: the output of the all-passes, [s + 1]: of tone section s
    FdnLine load_line[kLines], mix_line[kLines];
};

constexpr int kFdnThreads = 256;
// What a sample computes reaches the delay lines in the sixth step after its first section's, and the lines are read
// two steps ahead: the pipeline needs delays of at least kFdnLatency * S samples.
constexpr int kFdnLatency = 9;
// Lanes that share a sample's sixteen lines in the mix and in the loads of the delay lines: with steps of 16 samples or
// fewer two of them take eight lines each (one impulse in steps of 16: 0.525 ms against 0.588, 444 of them 1.35 against
// 1.66).
constexpr int fdn_lanes_per_sample(int step) { return step <= 16 ? 2 : 1; }

// One absorptive or tone section (steam_rt.py:2261-2275, :2312-2325) of one lane, in float64:
//     y0 = b0*x0 + b1*x1 + b2*x2 - a1*y1 - a2*y2, left to right.
// The input part ((b0*x0 + b1*x1) + b2*x2) does not depend on y and is formed four samples ahead, so its products fill
// the gaps of the recursion (v - a1*y1) - a2*y2.
struct Biquad {
    double b0, b1, b2, a1, a2, x1, x2, y1, y2;

    __device__ __forceinline__ void load(const double *c) {
        b0 = c[0]; b1 = c[1]; b2 = c[2]; a1 = c[3]; a2 = c[4];
        x1 = x2 = y1 = y2 = 0.0;
    }

    __device__ __forceinline__ double feed(double x) {
        const double v = b0 * x + b1 * x1 + b2 * x2;
        x2 = x1;
        x1 = x;
        return v;
    }

    __device__ __forceinline__ double step(double v) {
        const double y0 = v - a1 * y1 - a2 * y2;
        y2 = y1;
        y1 = y0;
        return y0;
    }

    // S samples from column xp to column yp of rows kPitch apart.
    template <int S, int kPitch>
    __device__ __forceinline__ void run(const double *xp, double *yp) {
        constexpr int kAhead = S % 4 == 0 ? 4 : 2;
        static_assert(S % kAhead == 0, "whole groups");
        double v[kAhead], x[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) x[u] = xp[u * kPitch];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) v[u] = feed(x[u]);
        // not unrolled whole: the warps run different code, and with straight-line code for a step of 64 samples a full
        // GPU (148 impulses) fell from 47 to 77-112 cycles per sample waiting for instructions
#pragma unroll 4
        for (int base = kAhead; base < S; base += kAhead) {
            double vn[kAhead];
            xp += kAhead * kPitch;
#pragma unroll
            for (int u = 0; u < kAhead; ++u) x[u] = xp[u * kPitch];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                yp[u * kPitch] = step(v[u]);
                vn[u] = feed(x[u]);
            }
            yp += kAhead * kPitch;
#pragma unroll
            for (int u = 0; u < kAhead; ++u) v[u] = vn[u];
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) yp[u * kPitch] = step(v[u]);
    }
};

template <int S>
__global__ void __launch_bounds__(kFdnThreads, 2) fdn_kernel(const FdnJobDev *jobs, double *pool) {
    constexpr int kPitch = FdnSmem<S>::kPitch, kPasses = (S + 31) / 32;
    extern __shared__ __align__(16) unsigned char fdn_smem_raw[];
    FdnSmem<S> &m = *reinterpret_cast<FdnSmem<S> *>(fdn_smem_raw);
    double *ap = reinterpret_cast<double *>(fdn_smem_raw + sizeof(FdnSmem<S>));
    const FdnJobDev &job = jobs[blockIdx.x];
    double *lines = pool + job.pool;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int total = job.preroll + job.num_samples;
    const int blocks = (total + S - 1) / S;
    const int steps = blocks + 13;   // a step's outputs are written 13 steps after its first section
    const int ap_total = job.allpass_start[AC_FDN_ALLPASS - 1] + job.allpass[AC_FDN_ALLPASS - 1];
    for (int i = threadIdx.x; i < ap_total; i += kFdnThreads) ap[i] = 0.0;
    if (threadIdx.x < kLines) {
        const FdnLine line{job.line_start[threadIdx.x], job.delays[threadIdx.x], 0, 0};
        m.load_line[threadIdx.x] = m.mix_line[threadIdx.x] = line;
    }
    __syncthreads();
    // all warps meet here once per step
    auto barrier = [] {
        __syncwarp();
        asm volatile("bar.sync 1, %0;" ::"n"(kFdnThreads) : "memory");
    };
    // the lines of this lane in the mix and the loads, and its sample of a pass
    constexpr int kShare = kLines / fdn_lanes_per_sample(S), kSamples = 32 / fdn_lanes_per_sample(S);
    const int own = lane % kSamples, first_line = lane / kSamples * kShare;
    // sample r of line l in the step that `table` stands at; advance() moves it one step on
    auto offset_of = [&](const FdnLine *table, int l, int r) {
        const FdnLine line = table[l];
        const int p = line.pos + r;
        return line.start + (p >= line.delay ? p - line.delay : p);
    };
    auto advance = [&](FdnLine *table) {
        __syncwarp();
        if (lane < kLines) {
            const int p = table[lane].pos + S;
            table[lane].pos = p >= table[lane].delay ? p - table[lane].delay : p;
        }
        __syncwarp();
    };

    if (warp < 3) {
        // bands 2 * warp and 2 * warp + 1 of the sixteen lines; band b works on step i - b
        const int band = 2 * warp + (lane >> 4), column = band * kLines + (lane & 15);
        Biquad section;
        section.load(job.absorptive[lane & 15][band]);
        barrier();
        for (int i = 0; i < steps; ++i) {
            const int k = i - band;
            if (k >= 0 && k < blocks)
                section.run<S, kPitch>(&m.y[k & 1][0][column], &m.y[k & 1][0][column + kLines]);
            barrier();
        }
    } else if (warp == 3) {
        // tone section `lane`, on step i - 7 - lane
        Biquad section;
        section.load(job.tone[lane < kBandSections ? lane : 0]);
        barrier();
        for (int i = 0; i < steps; ++i) {
            const int k = i - 7 - lane;
            if (lane < kBandSections && k >= 0 && k < blocks)
                section.run<S, kTonePitch>(&m.t[k & 1][0][lane], &m.t[k & 1][0][lane + 1]);
            barrier();
        }
    } else if (warp == 4) {
        // the feedback: a sample per lane, an unnormalised Hadamard butterfly of the line outputs, strides 1, 2, 4, 8,
        // written back with gain 0.25 and the unit impulse at sample 0 (steam_rt.py:2279-2295)
        barrier();
        for (int i = 0; i < steps; ++i) {
            const int k = i - kBandSections;
            if (k >= 0 && k < blocks) {
#pragma unroll 1
                for (int h = 0; h < kPasses; ++h) {
                    const int r = 32 * h + own;
                    double d[kShare] = {};
                    int offset[kShare];   // all addresses before the first store, which a later load would wait for
                    if (r < S) {
#pragma unroll
                        for (int l = 0; l < kShare; ++l) offset[l] = offset_of(m.mix_line, first_line + l, r);
                        const double *row = &m.y[k & 1][r][kBandSections * kLines + first_line];
#pragma unroll
                        for (int l = 0; l < kShare; ++l) d[l] = row[l];
#pragma unroll
                        for (int stride = 1; stride < kShare; stride *= 2)
#pragma unroll
                            for (int a = 0; a < kShare; ++a)
                                if ((a & stride) == 0) {
                                    const double one = d[a], two = d[a + stride];
                                    d[a] = one + two;
                                    d[a + stride] = one - two;
                                }
                    }
                    if constexpr (kShare < kLines) {   // the last stride, between the two lanes of a sample
                        static_assert(kShare * 2 == kLines, "two lanes per sample");
#pragma unroll
                        for (int l = 0; l < kShare; ++l) {
                            const double other = __shfl_xor_sync(0xffffffffu, d[l], kSamples);
                            d[l] = first_line == 0 ? d[l] + other : other - d[l];
                        }
                    }
                    if (r < S) {
                        const double injection = k == 0 && r == 0 ? 1.0 : 0.0;
#pragma unroll
                        for (int l = 0; l < kShare; ++l) lines[offset[l]] = injection + 0.25 * d[l];
                    }
                }
                advance(m.mix_line);
            }
            barrier();
        }
    } else if (warp == 5) {
        // the output of the network, a sample per lane: the line outputs summed in line order, over the line count
        // (steam_rt.py:2297-2300), through the four all-passes
        int apos[AC_FDN_ALLPASS], ap_delay[AC_FDN_ALLPASS], ap_start[AC_FDN_ALLPASS];
#pragma unroll
        for (int s = 0; s < AC_FDN_ALLPASS; ++s) {
            ap_delay[s] = job.allpass[s];
            ap_start[s] = job.allpass_start[s];
            apos[s] = 0;
        }
        barrier();
        for (int i = 0; i < steps; ++i) {
            const int k = i - kBandSections;
            if (k >= 0 && k < blocks) {
#pragma unroll 1
                for (int h = 0; h < kPasses; ++h) {
                    const int r = 32 * h + lane;
                    if (r < S) {
                        const double *row = &m.y[k & 1][r][kBandSections * kLines];
                        double d[kLines], previous[AC_FDN_ALLPASS];
                        int cell[AC_FDN_ALLPASS];
#pragma unroll
                        for (int l = 0; l < kLines; ++l) d[l] = row[l];
#pragma unroll
                        for (int s = 0; s < AC_FDN_ALLPASS; ++s) {
                            const int p = apos[s] + r;
                            cell[s] = ap_start[s] + (p >= ap_delay[s] ? p - ap_delay[s] : p);
                            previous[s] = ap[cell[s]];
                        }
                        double v = 0.0;
#pragma unroll
                        for (int l = 0; l < kLines; ++l) v += d[l];
                        v /= static_cast<double>(kLines);
#pragma unroll
                        for (int s = 0; s < AC_FDN_ALLPASS; ++s) {
                            const double internal = v + 0.5 * previous[s];
                            ap[cell[s]] = internal;
                            v = previous[s] - 0.5 * internal;
                        }
                        m.t[k & 1][r][0] = v;
                    }
                }
#pragma unroll
                for (int s = 0; s < AC_FDN_ALLPASS; ++s) {
                    const int p = apos[s] + S;
                    apos[s] = p >= ap_delay[s] ? p - ap_delay[s] : p;
                }
            }
            barrier();
        }
    } else if (warp == 6) {
        // the delay lines' samples, read two steps ahead (around L1: the mix writes them) and stored to the next step's
        // buffer; sample n of a line is at n mod delay
        double x[kPasses][kShare];
        // one branch around a pass's loads: with a condition per load they followed one another
        auto fetch = [&] {
#pragma unroll
            for (int h = 0; h < kPasses; ++h) {
                const int r = 32 * h + own;
                if (r < S) {
                    int offset[kShare];
#pragma unroll
                    for (int l = 0; l < kShare; ++l) offset[l] = offset_of(m.load_line, first_line + l, r);
#pragma unroll
                    for (int l = 0; l < kShare; ++l) x[h][l] = __ldcg(lines + offset[l]);
                }
            }
            advance(m.load_line);
        };
        auto store = [&](int k) {
#pragma unroll
            for (int h = 0; h < kPasses; ++h) {
                const int r = 32 * h + own;
                if (r < S) {
#pragma unroll
                    for (int l = 0; l < kShare; ++l) m.y[k & 1][r][first_line + l] = x[h][l];
                }
            }
        };
        fetch();
        store(0);
        fetch();
        barrier();
        for (int i = 0; i < steps; ++i) {
            store(i + 1);   // (past the last block: samples that nothing reads)
            fetch();        // of step i + 2
            barrier();
        }
    } else {
        const int preroll = job.preroll;
        double *out = job.out;
        barrier();
        for (int i = 0; i < steps; ++i) {
            const int k = i - 13;
#pragma unroll
            for (int h = 0; h < kPasses; ++h) {
                const int r = 32 * h + lane, n = k * S + r;
                if (r < S && k >= 0 && n >= preroll && n < total) out[n - preroll] = m.t[k & 1][r][kBandSections];
            }
            barrier();
        }
    }
}

// ---- the hybrid tail ------------------------------------------------------

struct LateJobDev {
    const double *traced;
    const double *fdn;
    float *out;
    float *component;
    double *stats;
    float *bands;     // workspace: [6, N] band-limited FDN
    double rt60[6];
    int32_t start[6];
    int32_t end[6];
    int32_t anchor[6];
    int32_t changed_from;
    int32_t num_samples;
    int32_t bin_samples;
    int32_t rate_index;
};

// bandlimit_band_signals(np.repeat(raw_fdn[None, :], 6, axis=0)): every band filters the same impulse.
template <int kSignals>
__global__ void __launch_bounds__(FilterShape<kSignals, true>::kThreads)
    late_band_kernel(const LateJobDev *jobs, int num_jobs, const __grid_constant__ ac_synth_batch_config cfg) {
    extern __shared__ __align__(16) unsigned char filter_smem_raw[];
    __shared__ FilterSignal signals[kSignals];
    if (threadIdx.x < kSignals) {
        const int first = static_cast<int>(blockIdx.x) * kSignals, j = first + threadIdx.x;
        const LateJobDev &job = jobs[j < num_jobs ? j : first];
        signals[threadIdx.x] = FilterSignal{job.fdn, 0, job.bands, cfg.crossover[job.rate_index],
                                            j < num_jobs ? job.num_samples : 0};
    }
    __syncthreads();
    filter_block<kSignals, true>(signals, *reinterpret_cast<FilterSmem<kSignals, true> *>(filter_smem_raw));
}

constexpr int kLateWide = 6;   // tails per filter block in a large batch: 30 chains, one per recursion lane

constexpr int kMixThreads = 256;

// Sum of one value per thread over the block, in a fixed order; every thread gets the total.
__device__ double block_sum(double v, double *scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    double total = 0.0;
    for (int w = 0; w < kMixThreads / 32; ++w) total += scratch[w];
    return total;
}

constexpr double kLn10 = 2.302585092994046;  // the float64 nearest ln(10)

// _late_tail_start_power (steam_rt.py:2473-2497) for one band; every thread gets the result.
__device__ double start_power(const double *x, int n_len, int anchor, double rt60, int fs, int bs, double *scratch,
                              double *bin_energy, int *found_bins, double *found_energy) {
    anchor = anchor < 0 ? 0 : (anchor > n_len ? n_len : anchor);
    const int hi = anchor + bs < n_len ? anchor + bs : n_len;
    double acc = 0.0;
    for (int n = anchor + threadIdx.x; n < hi; n += blockDim.x) acc += x[n] * x[n];
    const double here = block_sum(acc, scratch);
    const double measured = hi > anchor ? here / static_cast<double>(hi - anchor) : 0.0;
    if (anchor <= 0) return measured;
    const int nb = (anchor + bs - 1) / bs;
    __shared__ int s_found;
    if (threadIdx.x == 0) s_found = 0;
    __syncthreads();
    // the last five bins with energy above 1e-18, newest first, a block of bins at a time
    for (int top = nb - 1; top >= 0; top -= kMixThreads) {
        const int i = top - static_cast<int>(threadIdx.x);
        double e = 0.0;
        if (i >= 0) {
            const int end = (i + 1) * bs < anchor ? (i + 1) * bs : anchor;
            for (int n = i * bs; n < end; ++n) e += x[n] * x[n];
        }
        bin_energy[threadIdx.x] = e;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int t = 0; t < kMixThreads && s_found < 5 && top - t >= 0; ++t) {
                if (bin_energy[t] > 1e-18) {
                    found_bins[s_found] = top - t;
                    found_energy[s_found] = bin_energy[t];
                    ++s_found;
                }
            }
        }
        __syncthreads();
        if (s_found >= 5) break;
    }
    const int count = s_found;
    if (count == 0) return measured;
    // median of the decayed estimates (np.median: the middle value, or the mean of the two middle ones)
    const double decay = 6.0 * kLn10 / (rt60 > 0.1 ? rt60 : 0.1);
    double est[5];
    for (int j = 0; j < count; ++j) {
        const double centre = (static_cast<double>(found_bins[j]) + 0.5) * bs;
        double elapsed = (static_cast<double>(anchor) - centre) / static_cast<double>(fs > 1 ? fs : 1);
        elapsed = elapsed > 0.0 ? elapsed : 0.0;
        est[j] = (found_energy[j] / bs) * exp(-decay * elapsed);
    }
    for (int a = 1; a < count; ++a)
        for (int b = a; b > 0 && est[b - 1] > est[b]; --b) {
            const double t = est[b];
            est[b] = est[b - 1];
            est[b - 1] = t;
        }
    const double median = (count & 1) ? est[count / 2] : (est[count / 2 - 1] + est[count / 2]) / 2.0;
    return measured > median ? measured : median;
}

__global__ void __launch_bounds__(kMixThreads) late_mix_kernel(const LateJobDev *jobs,
                                                               const __grid_constant__ ac_synth_batch_config cfg) {
    __shared__ double scratch[kMixThreads / 32];
    __shared__ double bin_energy[kMixThreads];
    __shared__ int found_bins[5];
    __shared__ double found_energy[5];
    const LateJobDev &job = jobs[blockIdx.x / 6];
    const int band = blockIdx.x % 6;
    const int N = job.num_samples;
    const int fs = cfg.sample_rates[job.rate_index];
    const double *x = job.traced + static_cast<int64_t>(band) * N;
    const float *f = job.bands + static_cast<int64_t>(band) * N;
    const double rt60 = job.rt60[band];
    const int s = job.start[band], e = job.end[band];
    double scale = 1.0, power = 0.0, fdn_energy = 0.0;
    if (rt60 > 0.0) {
        const int anchor = job.anchor[band];
        power = start_power(x, N, anchor, rt60, fs, job.bin_samples, scratch, bin_energy, found_bins, found_energy);
        const double decay = 6.0 * kLn10 / (rt60 > 0.1 ? rt60 : 0.1);
        double target = 0.0, unit = 0.0;
        for (int k = threadIdx.x; k < N - anchor; k += blockDim.x) {
            target += power * exp(-decay * static_cast<double>(k) / static_cast<double>(fs));
            const double v = static_cast<double>(f[anchor + k]);
            unit += v * v;
        }
        target = block_sum(target, scratch);
        unit = block_sum(unit, scratch);
        scale = target > 0.0 ? sqrt(target / (unit > 1e-24 ? unit : 1e-24)) : 0.0;
        double acc = 0.0;
        for (int n = s + threadIdx.x; n < N; n += blockDim.x) {
            const double v = static_cast<double>(f[n]) * scale;
            acc += v * v;
        }
        fdn_energy = block_sum(acc, scratch);
    }
    // equal-power crossfade: alpha = np.linspace(1, 0, ramp, endpoint=False) = k * (-1 / ramp) + 1
    const int ramp = e - s > 1 ? e - s : 1;
    const double step = -1.0 / static_cast<double>(ramp);
    float *out = job.out + static_cast<int64_t>(band) * N;
    float *comp = job.component + static_cast<int64_t>(band) * N;
    double traced_tail = 0.0, rendered_tail = 0.0, comp_energy = 0.0;
    int changed = 0;
    for (int n = threadIdx.x; n < N; n += blockDim.x) {
        const double t = x[n];
        double o = t;
        double c = 0.0;
        if (n >= s) {
            double w = 1.0;
            if (n < s + ramp) {
                const double alpha = static_cast<double>(n - s) * step + 1.0;
                if (n < e) o = o * sqrt(alpha);
                w = sqrt(1.0 - alpha);
            }
            c = (static_cast<double>(f[n]) * scale) * w;
            traced_tail += t * t;
        }
        if (n >= e) o = 0.0;
        o = o + c;
        out[n] = static_cast<float>(o);
        comp[n] = static_cast<float>(c);
        if (n >= s) rendered_tail += o * o;
        comp_energy += c * c;
        if (n >= job.changed_from && !(fabs(o - t) <= 1e-12 + 1e-7 * fabs(t))) changed = 1;
    }
    traced_tail = block_sum(traced_tail, scratch);
    rendered_tail = block_sum(rendered_tail, scratch);
    comp_energy = block_sum(comp_energy, scratch);
    changed = __syncthreads_or(changed);
    if (threadIdx.x == 0) {
        double *st = job.stats + band * AC_LATE_STATS;
        st[AC_LATE_SCALE] = scale;
        st[AC_LATE_POWER] = power;
        st[AC_LATE_FDN_ENERGY] = fdn_energy;
        st[AC_LATE_TRACED_TAIL] = traced_tail;
        st[AC_LATE_RENDERED_TAIL] = rendered_tail;
        st[AC_LATE_COMPONENT] = comp_energy;
        st[AC_LATE_CHANGED] = changed ? 1.0 : 0.0;
        st[7] = 0.0;
    }
}

// ---- host side -------------------------------------------------------------

struct FdnLayout {
    size_t jobs, pool, total;
    int64_t pool_doubles;
    int max_allpass_doubles;
    int min_delay, min_allpass;
};

int check_fdn(const ac_fdn_job *jobs, int32_t num_jobs, bool need_buffers, FdnLayout *out) {
    if (num_jobs < 0 || (num_jobs > 0 && !jobs)) return fail(AC_ERR_INVALID, "fdn: null argument");
    if (num_jobs > (1 << 24)) return fail(AC_ERR_CAPACITY, "fdn batch of %d jobs is too large", num_jobs);
    FdnLayout l{};
    l.min_delay = l.min_allpass = 1 << 30;
    for (int32_t j = 0; j < num_jobs; ++j) {
        const ac_fdn_job &job = jobs[j];
        int64_t lines = 0;
        for (int i = 0; i < kLines; ++i) {
            if (job.delays[i] < AC_FDN_MIN_DELAY || job.delays[i] > (1 << 26))
                return fail(AC_ERR_INVALID, "fdn job %d: delay %d of line %d outside [%d, 2^26]", j, job.delays[i], i,
                            AC_FDN_MIN_DELAY);
            lines += job.delays[i];
            l.min_delay = std::min(l.min_delay, job.delays[i]);
        }
        if (lines > 0x7FFFFFFF) return fail(AC_ERR_CAPACITY, "fdn job %d: delay lines too long", j);
        int ap = 0;
        for (int s = 0; s < AC_FDN_ALLPASS; ++s) {
            if (job.allpass_delays[s] <= kMinAllpass || job.allpass_delays[s] > AC_FDN_MAX_ALLPASS)
                return fail(AC_ERR_INVALID, "fdn job %d: all-pass delay %d outside [%d, %d]", j, job.allpass_delays[s],
                            kMinAllpass + 1, AC_FDN_MAX_ALLPASS);
            ap += job.allpass_delays[s];
            l.min_allpass = std::min(l.min_allpass, job.allpass_delays[s]);
        }
        if (job.num_samples < 0 || job.preroll < 0 ||
            static_cast<int64_t>(job.num_samples) + job.preroll > (int64_t{1} << 30))
            return fail(AC_ERR_INVALID, "fdn job %d: bad length (%d + %d)", j, job.preroll, job.num_samples);
        if (need_buffers && job.num_samples > 0 && !job.out) return fail(AC_ERR_INVALID, "fdn job %d: null output", j);
        for (int i = 0; i < kLines * 6 * 5; ++i)
            if (!std::isfinite((&job.absorptive[0][0][0])[i]))
                return fail(AC_ERR_INVALID, "fdn job %d: non-finite absorptive coefficient", j);
        for (int i = 0; i < 6 * 5; ++i)
            if (!std::isfinite((&job.tone[0][0])[i])) return fail(AC_ERR_INVALID, "fdn job %d: non-finite tone coefficient", j);
        l.pool_doubles += lines;
        l.max_allpass_doubles = std::max(l.max_allpass_doubles, ap);
    }
    size_t off = 0;
    l.jobs = off; off = align256(off + static_cast<size_t>(num_jobs) * sizeof(FdnJobDev));
    l.pool = off; off = align256(off + static_cast<size_t>(l.pool_doubles) * sizeof(double));
    l.total = off;
    *out = l;
    return AC_OK;
}

constexpr int kMaxSmem = 227 * 1024;

// The step size of a launch: the largest whose pipeline fits the batch's shortest delay (kFdnLatency steps), whose
// all-pass samples are independent within a step and whose buffers fit shared memory.  A larger step has fewer barriers
// per sample, but a step of 64 takes a whole SM (135 KB), so beyond one impulse per SM a step of 32, two blocks per SM,
// is faster (296 impulses of 48 kHz: 72 cycles per sample against two waves of 47).  A step of 40 would fit the designs
// of 16 kHz, but its mix takes two passes of 32 lanes and it is no faster (54 cycles against 47).  The reference's
// designs have delays of at least 841 samples from 32 kHz up, 361 at 16 kHz, 289 from 7 kHz and 169 at 4.5 kHz; a step of
// 14 meets every accepted delay.  1 / 444 impulses of 16,000 samples, shortest delay 128: 0.575 / 1.39 ms with 14, 0.67 /
// 1.49 with 12, 1.62 / 3.87 with 8, 0.65 / 1.76 with the shuffles and a barrier every 32 samples; delay 144 with a step
// of 16: 0.525 / 1.35.
int fdn_step(const FdnLayout &l, int num_jobs, int sms) {
    const size_t ap = static_cast<size_t>(l.max_allpass_doubles) * sizeof(double);
    auto fits = [&](int step, size_t smem) {
        return kFdnLatency * step <= l.min_delay && step <= l.min_allpass && smem + ap <= kMaxSmem;
    };
    if (num_jobs <= sms && fits(64, sizeof(FdnSmem<64>))) return 64;
    if (fits(32, sizeof(FdnSmem<32>))) return 32;
    if (fits(16, sizeof(FdnSmem<16>))) return 16;
    return 14;
}
static_assert(kFdnLatency * 14 <= AC_FDN_MIN_DELAY && 14 <= kMinAllpass, "a step of 14 meets every accepted design");
static_assert(sizeof(FdnSmem<14>) + AC_FDN_ALLPASS * AC_FDN_MAX_ALLPASS * sizeof(double) <= kMaxSmem, "and fits");

template <int S>
int launch_fdn(const FdnJobDev *jobs, int num_jobs, double *pool, int max_allpass_doubles, cudaStream_t stream) {
    const size_t smem = sizeof(FdnSmem<S>) + static_cast<size_t>(max_allpass_doubles) * sizeof(double);
    // always the same limit: a concurrent call with other all-pass lengths must not lower it
    AC_CUDA_TRY(cudaFuncSetAttribute(fdn_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem));
    fdn_kernel<S><<<num_jobs, kFdnThreads, smem, stream>>>(jobs, pool);
    AC_CUDA_TRY(cudaGetLastError());
    return AC_OK;
}

struct LateLayout {
    size_t jobs, bands, total;
    int64_t band_floats;
};

int check_late(const ac_late_tail_job *jobs, int32_t num_jobs, const ac_synth_batch_config *cfg, bool need_buffers,
               LateLayout *out) {
    if (num_jobs < 0 || (num_jobs > 0 && !jobs) || !cfg) return fail(AC_ERR_INVALID, "late tail: null argument");
    if (cfg->num_rates < 1 || cfg->num_rates > AC_SYNTH_MAX_RATES)
        return fail(AC_ERR_INVALID, "late tail: num_rates must be 1..%d", AC_SYNTH_MAX_RATES);
    if (num_jobs > (1 << 24)) return fail(AC_ERR_CAPACITY, "late tail batch of %d jobs is too large", num_jobs);
    LateLayout l{};
    for (int32_t j = 0; j < num_jobs; ++j) {
        const ac_late_tail_job &job = jobs[j];
        const int N = job.num_samples;
        if (N < 1 || N > (1 << 28)) return fail(AC_ERR_INVALID, "late tail job %d: num_samples %d", j, N);
        if (job.bin_samples < 1) return fail(AC_ERR_INVALID, "late tail job %d: bin_samples must be positive", j);
        if (job.rate_index < 0 || job.rate_index >= cfg->num_rates || cfg->sample_rates[job.rate_index] < 1)
            return fail(AC_ERR_INVALID, "late tail job %d: bad rate_index %d", j, job.rate_index);
        for (int b = 0; b < 6; ++b) {
            if (job.start[b] < 0 || job.start[b] >= N || job.end[b] <= job.start[b] || job.end[b] > N)
                return fail(AC_ERR_INVALID, "late tail job %d band %d: crossfade [%d, %d) outside [0, %d)", j, b,
                            job.start[b], job.end[b], N);
            if (job.anchor[b] < 0 || job.anchor[b] > N)
                return fail(AC_ERR_INVALID, "late tail job %d band %d: anchor %d outside [0, %d]", j, b, job.anchor[b], N);
            if (!std::isfinite(job.rt60[b])) return fail(AC_ERR_INVALID, "late tail job %d: non-finite rt60", j);
        }
        if (job.changed_from < 0) return fail(AC_ERR_INVALID, "late tail job %d: negative changed_from", j);
        if (need_buffers && (!job.traced || !job.fdn || !job.out || !job.fdn_component || !job.stats))
            return fail(AC_ERR_INVALID, "late tail job %d: null buffer", j);
        l.band_floats += static_cast<int64_t>(align256(6 * static_cast<size_t>(N) * sizeof(float)) / sizeof(float));
    }
    size_t off = 0;
    l.jobs = off;  off = align256(off + static_cast<size_t>(num_jobs) * sizeof(LateJobDev));
    l.bands = off; off = align256(off + static_cast<size_t>(l.band_floats) * sizeof(float));
    l.total = off;
    *out = l;
    return AC_OK;
}

}  // namespace
}  // namespace ac

extern "C" int ac_fdn_workspace_size(const ac_fdn_job *jobs, int32_t num_jobs, size_t *bytes) {
    if (!bytes) return ac::fail(AC_ERR_INVALID, "ac_fdn_workspace_size: null argument");
    ac::FdnLayout l;
    const int rc = ac::check_fdn(jobs, num_jobs, false, &l);
    if (rc != AC_OK) return rc;
    *bytes = l.total;
    return AC_OK;
}

extern "C" int ac_fdn_impulse(const ac_fdn_job *jobs, int32_t num_jobs, void *workspace, size_t workspace_bytes,
                              void *host_staging, void *stream_ptr) {
    ac::NvtxRange nvtx_range("ac_fdn_impulse");
    ac::FdnLayout l;
    const int rc = ac::check_fdn(jobs, num_jobs, true, &l);
    if (rc != AC_OK) return rc;
    if (num_jobs == 0) return AC_OK;
    if (!workspace || workspace_bytes < l.total)
        return ac::fail(AC_ERR_CAPACITY, "fdn workspace too small: %zu < %zu", workspace_bytes, l.total);
    cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
    unsigned char *ws = static_cast<unsigned char *>(workspace);
    const size_t table_bytes = static_cast<size_t>(num_jobs) * sizeof(ac::FdnJobDev);
    std::vector<unsigned char> local;
    unsigned char *host = static_cast<unsigned char *>(host_staging);
    if (!host) {
        local.assign(table_bytes, 0);
        host = local.data();
    }
    int64_t pool = 0;
    for (int32_t j = 0; j < num_jobs; ++j) {
        const ac_fdn_job &in = jobs[j];
        ac::FdnJobDev d{};
        std::memcpy(d.absorptive, in.absorptive, sizeof(d.absorptive));
        std::memcpy(d.tone, in.tone, sizeof(d.tone));
        int32_t off = 0;
        for (int i = 0; i < ac::kLines; ++i) {
            d.delays[i] = in.delays[i];
            d.line_start[i] = off;
            off += in.delays[i];
        }
        int32_t ap = 0;
        for (int s = 0; s < AC_FDN_ALLPASS; ++s) {
            d.allpass[s] = in.allpass_delays[s];
            d.allpass_start[s] = ap;
            ap += in.allpass_delays[s];
        }
        d.num_samples = in.num_samples;
        d.preroll = in.preroll;
        d.out = in.out;
        d.pool = pool;
        pool += off;
        std::memcpy(host + j * sizeof(ac::FdnJobDev), &d, sizeof(d));
    }
    AC_CUDA_TRY(cudaMemcpyAsync(ws + l.jobs, host, table_bytes, cudaMemcpyHostToDevice, stream));
    if (!host_staging) AC_CUDA_TRY(cudaStreamSynchronize(stream));  // pageable source must stay alive
    AC_CUDA_TRY(cudaMemsetAsync(ws + l.pool, 0, static_cast<size_t>(l.pool_doubles) * sizeof(double), stream));
    int device = 0, sms = 0;
    AC_CUDA_TRY(cudaGetDevice(&device));
    AC_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    const ac::FdnJobDev *d_jobs = reinterpret_cast<const ac::FdnJobDev *>(ws + l.jobs);
    double *lines = reinterpret_cast<double *>(ws + l.pool);
    switch (ac::fdn_step(l, num_jobs, sms)) {
        case 64: return ac::launch_fdn<64>(d_jobs, num_jobs, lines, l.max_allpass_doubles, stream);
        case 32: return ac::launch_fdn<32>(d_jobs, num_jobs, lines, l.max_allpass_doubles, stream);
        case 16: return ac::launch_fdn<16>(d_jobs, num_jobs, lines, l.max_allpass_doubles, stream);
        default: return ac::launch_fdn<14>(d_jobs, num_jobs, lines, l.max_allpass_doubles, stream);
    }
}

extern "C" int ac_late_tail_workspace_size(const ac_late_tail_job *jobs, int32_t num_jobs,
                                           const ac_synth_batch_config *config, size_t *bytes) {
    if (!bytes) return ac::fail(AC_ERR_INVALID, "ac_late_tail_workspace_size: null argument");
    ac::LateLayout l;
    const int rc = ac::check_late(jobs, num_jobs, config, false, &l);
    if (rc != AC_OK) return rc;
    *bytes = l.total;
    return AC_OK;
}

extern "C" int ac_late_tail(const ac_late_tail_job *jobs, int32_t num_jobs, const ac_synth_batch_config *config,
                            void *workspace, size_t workspace_bytes, void *host_staging, void *stream_ptr) {
    ac::NvtxRange nvtx_range("ac_late_tail");
    ac::LateLayout l;
    const int rc = ac::check_late(jobs, num_jobs, config, true, &l);
    if (rc != AC_OK) return rc;
    if (num_jobs == 0) return AC_OK;
    if (!workspace || workspace_bytes < l.total)
        return ac::fail(AC_ERR_CAPACITY, "late tail workspace too small: %zu < %zu", workspace_bytes, l.total);
    cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
    unsigned char *ws = static_cast<unsigned char *>(workspace);
    const size_t table_bytes = static_cast<size_t>(num_jobs) * sizeof(ac::LateJobDev);
    std::vector<unsigned char> local;
    unsigned char *host = static_cast<unsigned char *>(host_staging);
    if (!host) {
        local.assign(table_bytes, 0);
        host = local.data();
    }
    float *bands = reinterpret_cast<float *>(ws + l.bands);
    int64_t band_off = 0;
    for (int32_t j = 0; j < num_jobs; ++j) {
        const ac_late_tail_job &in = jobs[j];
        ac::LateJobDev d{};
        d.traced = in.traced;
        d.fdn = in.fdn;
        d.out = in.out;
        d.component = in.fdn_component;
        d.stats = in.stats;
        d.bands = bands + band_off;
        band_off += static_cast<int64_t>(ac::align256(6 * static_cast<size_t>(in.num_samples) * sizeof(float)) /
                                         sizeof(float));
        for (int b = 0; b < 6; ++b) {
            d.rt60[b] = in.rt60[b];
            d.start[b] = in.start[b];
            d.end[b] = in.end[b];
            d.anchor[b] = in.anchor[b];
        }
        d.changed_from = in.changed_from;
        d.num_samples = in.num_samples;
        d.bin_samples = in.bin_samples;
        d.rate_index = in.rate_index;
        std::memcpy(host + j * sizeof(ac::LateJobDev), &d, sizeof(d));
    }
    AC_CUDA_TRY(cudaMemcpyAsync(ws + l.jobs, host, table_bytes, cudaMemcpyHostToDevice, stream));
    if (!host_staging) AC_CUDA_TRY(cudaStreamSynchronize(stream));
    const ac::LateJobDev *d_jobs = reinterpret_cast<const ac::LateJobDev *>(ws + l.jobs);
    const int units = 6 * num_jobs;
    const int frc = ac::with_filter_signals<ac::kLateWide>(num_jobs, [&](auto signals, int blocks) -> int {
        constexpr int kSignals = decltype(signals)::value;
        const size_t smem = sizeof(ac::FilterSmem<kSignals, true>);
        const int rc2 = ac::filter_smem(ac::late_band_kernel<kSignals>, smem);
        if (rc2 != AC_OK) return rc2;
        ac::late_band_kernel<kSignals>
            <<<blocks, ac::FilterShape<kSignals, true>::kThreads, smem, stream>>>(d_jobs, num_jobs, *config);
        AC_CUDA_TRY(cudaGetLastError());
        return AC_OK;
    });
    if (frc != AC_OK) return frc;
    ac::late_mix_kernel<<<units, ac::kMixThreads, 0, stream>>>(d_jobs, *config);
    AC_CUDA_TRY(cudaGetLastError());
    return AC_OK;
}
