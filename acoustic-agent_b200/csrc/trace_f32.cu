// Float32 production launches: the warp-uniform scene-scan tracer (trace_fast.cuh).
#include <algorithm>
#include <numeric>
#include <vector>

#include "trace_launch.cuh"

namespace ac {

namespace {

constexpr int kDefaultChunkRays = 32;
// A scene group holds at most this many consecutive jobs, so that (job index mod 1024,
// surface) identifies a (job, surface) pair among the lanes of one warp (hit-count keys).
constexpr int64_t kMaxGroupJobs = 1024;

// Zero words of a job's outputs; the arrays of init_single_kernel.
__host__ __device__ inline size_t output_words(const Job<float> &job) {
    const size_t nb = 2 * static_cast<size_t>(kBands) * job.num_bins;
    return nb * (job.ambisonic_fx ? 5 : 1) + 4 * static_cast<size_t>(job.scene.num_surfaces) + 8;
}

__device__ __forceinline__ void zero_word(const Job<float> &job, size_t i) {
    const size_t nb = 2 * static_cast<size_t>(kBands) * job.num_bins, na = job.ambisonic_fx ? 4 * nb : 0;
    const size_t ns = static_cast<size_t>(job.scene.num_surfaces);
    if (i < nb) job.echogram_fx[i] = 0ull;
    else if (i < nb + na) job.ambisonic_fx[i - nb] = 0ull;
    else if (i < nb + na + ns) job.hit_counts[i - nb - na] = 0ull;
    else if (i < nb + na + 2 * ns) job.contrib_counts[i - nb - na - ns] = 0ull;
    else if (i < nb + na + 4 * ns) job.surface_energy_fx[i - nb - na - 2 * ns] = 0ull;
    else job.counters[i - nb - na - 4 * ns] = 0ull;
}

// A single job's outputs before its trace, in one launch (one memset per array cost a launch each).
__global__ void init_single_kernel(const __grid_constant__ Job<float> job) {
    const size_t first = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
    const size_t step = static_cast<size_t>(gridDim.x) * blockDim.x, total = output_words(job);
    for (size_t i = first; i < total; i += step) zero_word(job, i);
    init_visual(job, first, step);
}

// Cell i of a job's float32 outputs ([6, bins] echogram, [6, 4, bins] ambisonic, [S] surface energies) from the fixed
// point; the ambisonic W channel is the echogram's sums.
__device__ __forceinline__ void finalize_cell(const Job<float> &job, const FinalizeTargets &tg, size_t i, double inv) {
    const size_t bins = static_cast<size_t>(job.num_bins), nb = kBands * bins, na = job.ambisonic_fx ? 4 * nb : 0;
    if (i < nb) {
        if (tg.echogram) tg.echogram[i] = static_cast<float>(fixed_to_double(job.echogram_fx + 2 * i, inv));
    } else if (i < nb + na) {
        const size_t k = i - nb, band = k / (4 * bins), channel = (k - band * 4 * bins) / bins;
        unsigned long long *w = job.ambisonic_fx + 2 * k;
        if (channel == 0) {
            const unsigned long long *e = job.echogram_fx + 2 * (band * bins + (k - band * 4 * bins));
            w[0] = e[0];
            w[1] = e[1];
        }
        if (tg.ambisonic) tg.ambisonic[k] = static_cast<float>(fixed_to_double(w, inv));
    } else if (tg.surface_energy) {
        const size_t k = i - nb - na;
        tg.surface_energy[k] = static_cast<float>(fixed_to_double(job.surface_energy_fx + 2 * k, inv));
    }
}

__device__ __forceinline__ size_t finalize_cells(const Job<float> &job) {
    const size_t nb = static_cast<size_t>(kBands) * job.num_bins;
    return nb * (job.ambisonic_fx ? 5 : 1) + static_cast<size_t>(job.scene.num_surfaces);
}

__global__ void finalize_f32_single_kernel(const __grid_constant__ Job<float> job, FinalizeTargets tg) {
    const double inv = 1.0 / job.energy_scale;
    const size_t total = finalize_cells(job);
    if (blockIdx.x == 0 && threadIdx.x == 0) job.counters[4] = 0ull;   // the work counter: its end depends on the launch's shape
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x)
        finalize_cell(job, tg, i, inv);
}

// A batch job's accumulators in the caller's outputs, where its copies are summed to.
struct ShardTargets {
    unsigned long long *echogram_fx, *ambisonic_fx, *hit_counts, *contrib_counts, *surface_energy_fx;
};

// Each job's copies of its accumulators summed into the caller's outputs (for most jobs they are the outputs).
__global__ void gather_shards_kernel(const Job<float> *jobs, const ShardTargets *targets, int num_jobs) {
    for (int j = blockIdx.y; j < num_jobs; j += gridDim.y) {
        const Job<float> &job = jobs[j];
        if (job.shard_mask == 0) continue;
        const ShardTargets t = targets[j];
        const size_t nb = 2 * static_cast<size_t>(kBands) * job.num_bins, na = job.ambisonic_fx ? 4 * nb : 0;
        const size_t ns = static_cast<size_t>(job.scene.num_surfaces), words = nb + na + 4 * ns;
        for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < words;
             i += static_cast<size_t>(gridDim.x) * blockDim.x) {
            unsigned long long sum = 0ull;   // the copies lie as one array: echogram, ambisonic, hits, contributions, energies
            for (int c = 0; c <= job.shard_mask; ++c) sum += __ldcg(job.echogram_fx + c * job.shard_stride + i);
            if (i < nb) t.echogram_fx[i] = sum;
            else if (i < nb + na) t.ambisonic_fx[i - nb] = sum;
            else if (i < nb + na + ns) t.hit_counts[i - nb - na] = sum;
            else if (i < nb + na + 2 * ns) t.contrib_counts[i - nb - na - ns] = sum;
            else t.surface_energy_fx[i - nb - na - 2 * ns] = sum;
        }
    }
}

// Float32 outputs of every job, from the caller's fixed-point ones.
__global__ void finalize_f32_kernel(const Job<float> *jobs, const FinalizeTargets *targets, const ShardTargets *outputs,
                                    int num_jobs) {
    for (int j = blockIdx.y; j < num_jobs; j += gridDim.y) {
        Job<float> job = jobs[j];
        job.echogram_fx = outputs[j].echogram_fx;
        job.ambisonic_fx = outputs[j].ambisonic_fx;
        job.surface_energy_fx = outputs[j].surface_energy_fx;
        const double inv = 1.0 / job.energy_scale;
        const size_t total = finalize_cells(job);
        for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
             i += static_cast<size_t>(gridDim.x) * blockDim.x)
            finalize_cell(job, targets[j], i, inv);
    }
}

using FastKernel = void (*)(const Job<float>, const FastScene, const FastTable);

template <bool kSingle, bool kVisual, bool kOwnSums, bool kLean>
FastKernel pick_stream(bool philox, bool amb) {
    if (philox)
        return amb ? trace_fast_kernel<kSingle, true, true, kVisual, false, kOwnSums, kLean>
                   : trace_fast_kernel<kSingle, true, false, kVisual, false, kOwnSums, kLean>;
    return amb ? trace_fast_kernel<kSingle, false, true, kVisual, false, kOwnSums, kLean>
               : trace_fast_kernel<kSingle, false, false, kVisual, false, kOwnSums, kLean>;
}

template <bool kSingle, bool kLean>
FastKernel pick_variant(bool philox, bool amb, bool visual, bool own_sums) {
    if (visual)   // batches with visual candidates have no copies
        return kSingle && own_sums ? pick_stream<kSingle, true, kSingle, kLean>(philox, amb)
                                   : pick_stream<kSingle, true, false, kLean>(philox, amb);
    return own_sums ? pick_stream<kSingle, false, true, kLean>(philox, amb)
                    : pick_stream<kSingle, false, false, kLean>(philox, amb);
}

template <bool kSingle>
FastKernel pick_kernel(bool philox, bool amb, bool visual, bool own_sums, bool lean) {
    return lean ? pick_variant<kSingle, true>(philox, amb, visual, own_sums)
                : pick_variant<kSingle, false>(philox, amb, visual, own_sums);
}

// Whether the lean kernels can trace a scene: no boxes in the lockstep scan, no four-wide BVH.
bool scene_is_lean(const FastScene &f) { return f.num_box_clusters == 0 && (f.num_bvh_nodes == 0 || f.bvh_width == 2); }

int fast_grid(FastKernel kernel, int device, int block, size_t smem, int64_t total_rays, int requested) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, smem) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    int grid = requested > 0 ? requested : per_sm * device_sm_count(device);
    const int64_t needed = (total_rays + block - 1) / block;
    if (needed < grid) grid = static_cast<int>(needed > 0 ? needed : 1);
    return grid;
}

// Words of one copy of a batch job's accumulators.
size_t accumulator_words(const ac_job &job) {
    const size_t nb = 2 * static_cast<size_t>(kBands) * job.params.num_bins;
    return nb * (job.params.render_ambisonics ? 5 : 1) + 4 * static_cast<size_t>(job.scene->num_surfaces);
}

// A batch job of a small room gets copies of its accumulators, shared out by block: all its rays deposit into a few
// hundred addresses, whose atomics queue up at L2 (100,000 rays x 50 bounces in the shoebox, 100 bins: 3.77 ms with one
// copy, 1.57 with 4, 0.78 with 16, 0.62 with 32).  Jobs of more than 32 KB of accumulators (some 300 bins and up) or 64
// surfaces spread their deposits over addresses or time and gain nothing, nor do the scenes of a mixed launch, which the
// warps trace side by side: eight of them took 129.0 ms without copies and 129.7 with the code that adds to them.  The
// copies of a launch stay within 8 MB of workspace.
constexpr size_t kShardJobBytes = 32 * 1024, kShardTotalBytes = 8 * 1024 * 1024;
constexpr int64_t kShardSurfaces = 64, kShardGroups = 4;
constexpr int32_t kMaxShards = 32;
constexpr int64_t kShardRays = 2048;   // rays per copy at least

// Copies of each job's accumulators (in launch order); returns their words.
size_t shard_plan(const ac_job *jobs, const std::vector<int32_t> &order, int64_t groups, std::vector<int32_t> *copies) {
    size_t total = 0;
    if (copies) copies->assign(order.size(), 1);
    if (groups > kShardGroups || jobs[order[0]].params.visual_limit > 0) return 0;
    for (size_t k = 0; k < order.size(); ++k) {
        const ac_job &job = jobs[order[k]];
        const size_t bytes = accumulator_words(job) * sizeof(unsigned long long);
        if (bytes > kShardJobBytes || job.scene->num_surfaces > kShardSurfaces) continue;
        int32_t n = 1;
        while (n * groups < kMaxShards && job.params.num_rays > kShardRays * n) n *= 2;
        while (n > 1 && total + n * bytes > kShardTotalBytes) n /= 2;
        if (n == 1) continue;
        if (copies) (*copies)[k] = n;
        total += n * bytes;
    }
    return total / sizeof(unsigned long long);
}

// Workspace layout for a float32 batch (each part 256-aligned):
//   [0] chunk counter | group queue counters u64[G] | ray prefix int64[J+1] | Job<float>[J] |
//   FinalizeTargets[J] | ShardTargets[J] | FastGroup[G] | group ray prefix int64[G+1] | copies of jobs' accumulators
// From the ray prefix to the group prefix it is staged on the host and copied in one transfer; the counters and the
// copies are zeroed on the device.
struct F32Layout {
    size_t queues, prefix, jobs, targets, outputs, groups, group_rays, table_end, shards, total;
};

F32Layout f32_layout(int32_t jobs, int64_t groups, size_t shard_words) {
    F32Layout l{};
    size_t off = 256;
    l.queues = off;       off = align256(off + sizeof(unsigned long long) * static_cast<size_t>(groups));
    l.prefix = off;       off = align256(off + sizeof(int64_t) * (static_cast<size_t>(jobs) + 1));
    l.jobs = off;         off = align256(off + sizeof(Job<float>) * static_cast<size_t>(jobs));
    l.targets = off;      off = align256(off + sizeof(FinalizeTargets) * static_cast<size_t>(jobs));
    l.outputs = off;      off = align256(off + sizeof(ShardTargets) * static_cast<size_t>(jobs));
    l.groups = off;       off = align256(off + sizeof(FastGroup) * static_cast<size_t>(groups));
    l.group_rays = off;   off = align256(off + sizeof(int64_t) * (static_cast<size_t>(groups) + 1));
    l.table_end = off;
    l.shards = off;       off = align256(off + sizeof(unsigned long long) * shard_words);
    l.total = off;
    return l;
}

// Jobs sorted by scene so that each scene's rays form one contiguous range.
std::vector<int32_t> scene_order(const ac_job *jobs, const int32_t *indices, int32_t count) {
    std::vector<int32_t> order(indices, indices + count);
    std::stable_sort(order.begin(), order.end(), [&](int32_t a, int32_t b) {
        return reinterpret_cast<uintptr_t>(jobs[a].scene) < reinterpret_cast<uintptr_t>(jobs[b].scene);
    });
    return order;
}

int64_t count_groups(const ac_job *jobs, const std::vector<int32_t> &order) {
    int64_t groups = 0;
    size_t k = 0;
    while (k < order.size()) {
        const ac_scene_t scene = jobs[order[k]].scene;
        for (int64_t members = 0; k < order.size() && jobs[order[k]].scene == scene && members < kMaxGroupJobs; ++members) ++k;
        ++groups;
    }
    return groups;
}

// Warps per SM that a single job's rays are spread over.  In a small room whose sums lie in global memory the deposits of
// more warps meet at the same addresses: a shoebox (scan) of 10,000 / 20,000 rays, 500 bins, takes 0.406 / 0.678 ms over
// eight, 0.362 / 0.641 over two, a room of 6 boxes with 20,000 / 25,000 rays 0.638 / 0.827 over eight, 0.615 / 0.766 over
// six; larger rooms' deposits are spread out (U room, 20,000 rays 0.498 over eight, 0.515 over six).
int single_warps_per_sm(const ac_scene_s *scene, const FastScene &form, bool own_sums) {
    if (own_sums || scene->num_surfaces > 24) return 8;
    return form.num_bvh_nodes > 0 ? 6 : 2;
}

}  // namespace

int launch_trace_f32(const ac_scene_s *scene, const ac_trace_params *p, const ac_trace_outputs *o, double scale,
                     void *stream_ptr) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
    int entries = 0;
    const FastScene &form = fast_form(scene, p->stack_entries);
    const int rc = launch_stack_entries(p->stack_entries, stack_need(scene, form), &entries);
    if (rc != AC_OK) return rc;
    Job<float> job;
    fill_job<float>(scene, p, o, scale, job);
    AC_CUDA_TRY(cudaSetDevice(scene->device));
    {
        const size_t words = output_words(job) + 3 * static_cast<size_t>(job.visual_limit) * job.num_bounces;
        init_single_kernel<<<static_cast<int>(std::min<size_t>((words + 255) / 256, 1024)), 256, 0, stream>>>(job);
        AC_CUDA_TRY(cudaGetLastError());
    }
    const int block = p->block_size > 0 ? p->block_size : kDefaultBlock;
    if (block % 32 != 0 || block > 256) return fail(AC_ERR_INVALID, "block_size must be a multiple of 32 up to 256");
    const int64_t cells = static_cast<int64_t>(kBands) * p->num_bins * (job.ambisonic_fx ? 4 : 1) + scene->num_surfaces;
    const int64_t sum_bytes = 4 * (4 * cells + 2 * scene->num_surfaces);
    const bool own_sums = sum_bytes <= kSharedSumBytes;
    // beside the sums no deeper stack than the tree uses, so that three blocks still fit an SM (U room, 400 bins, 100,000
    // rays: 0.98 ms with two, 0.72 with three; what lies above the need is never read)
    if (own_sums) entries = std::min(entries, stack_need(scene, form));
    FastTable table{};
    table.lanes = p->grid_blocks > 0 ? 32
                                     : warp_lanes(scene->device, p->num_rays, form.num_bvh_nodes > 0 ? 4 : 16,
                                                  single_warps_per_sm(scene, form, own_sums));
    table.chunk_rays = std::min(kDefaultChunkRays, table.lanes);
    table.chunk_counter = reinterpret_cast<unsigned long long *>(o->counters) + 4;
    const FastKernel kernel = pick_kernel<true>(p->rng_mode == AC_RNG_PHILOX, p->render_ambisonics != 0,
                                                p->visual_limit > 0, own_sums, scene_is_lean(form));
    size_t smem = stack_smem_bytes(entries);
    table.stack_words = static_cast<int32_t>(smem / sizeof(int));
    if (own_sums) {
        table.shared_cells = static_cast<int32_t>(cells);
        smem += static_cast<size_t>(sum_bytes);
        // always the same limit, so that concurrent calls do not lower it for one another
        AC_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(stack_smem_bytes(kBvhStack)) + kSharedSumBytes));
    }
    const int grid = fast_grid(kernel, scene->device, block, smem, spread_rays(p->num_rays, table.lanes), p->grid_blocks);
    kernel<<<grid, block, smem, stream>>>(job, form, table);
    AC_CUDA_TRY(cudaGetLastError());
    const FinalizeTargets tg{o->echogram, job.ambisonic_fx ? o->ambisonic : nullptr, o->surface_energy};
    const size_t results = static_cast<size_t>(kBands) * p->num_bins * 5 + scene->num_surfaces;
    finalize_f32_single_kernel<<<static_cast<int>(std::min<size_t>((results + 255) / 256, 1024)), 256, 0, stream>>>(job, tg);
    AC_CUDA_TRY(cudaGetLastError());
    return AC_OK;
}

size_t batch_workspace_bytes_f32(const ac_job *jobs, const int32_t *indices, int32_t count, const ac_batch_config *,
                                 bool copies) {
    const std::vector<int32_t> order = scene_order(jobs, indices, count);
    const int64_t groups = count_groups(jobs, order);
    return f32_layout(count, groups, copies ? shard_plan(jobs, order, groups, nullptr) : 0).total;
}

int launch_batch_f32(const ac_job *jobs_in, const int32_t *indices, int32_t count, const ac_batch_config *cfg,
                     void *workspace, size_t workspace_bytes, void *host_staging, void *stream_ptr) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
    const int64_t chunk_rays = (cfg && cfg->chunk_rays > 0) ? cfg->chunk_rays : kDefaultChunkRays;
    const std::vector<int32_t> order = scene_order(jobs_in, indices, count);
    const int64_t num_groups = count_groups(jobs_in, order);
    std::vector<int32_t> copies;
    size_t shard_words = shard_plan(jobs_in, order, num_groups, &copies);
    if (f32_layout(count, num_groups, shard_words).total > workspace_bytes) {
        shard_words = 0;
        copies.assign(order.size(), 1);
    }
    const F32Layout l = f32_layout(count, num_groups, shard_words);
    if (workspace_bytes < l.total)
        return fail(AC_ERR_CAPACITY, "batch workspace too small: %zu < %zu", workspace_bytes, l.total);
    std::vector<unsigned char> local;
    unsigned char *host = static_cast<unsigned char *>(host_staging);
    if (!host) {
        local.assign(l.table_end, 0);
        host = local.data();
    }
    int64_t *prefix = reinterpret_cast<int64_t *>(host + l.prefix);
    Job<float> *jobs = reinterpret_cast<Job<float> *>(host + l.jobs);
    FinalizeTargets *targets = reinterpret_cast<FinalizeTargets *>(host + l.targets);
    ShardTargets *outputs = reinterpret_cast<ShardTargets *>(host + l.outputs);
    FastGroup *groups = reinterpret_cast<FastGroup *>(host + l.groups);
    int64_t *group_rays = reinterpret_cast<int64_t *>(host + l.group_rays);
    unsigned long long *shards = reinterpret_cast<unsigned long long *>(static_cast<unsigned char *>(workspace) + l.shards);
    int device = -1, need = 0;
    bool lean = true;
    int64_t total = 0, g = -1;
    const ac_scene_s *current = nullptr;
    for (int32_t k = 0; k < count; ++k) {
        const ac_job &in = jobs_in[order[k]];
        if (device < 0) device = in.scene->device;
        if (in.scene->device != device) return fail(AC_ERR_INVALID, "batch jobs must share one device");
        const FastScene &form = fast_form(in.scene, cfg ? cfg->stack_entries : 0);
        need = std::max(need, stack_need(in.scene, form));
        lean = lean && scene_is_lean(form);
        if (in.scene != current || groups[g].num_jobs >= kMaxGroupJobs) {
            ++g;
            current = in.scene;
            group_rays[g] = total;
            groups[g] = FastGroup{in.scene->f32, form, k, 0};
        }
        groups[g].num_jobs += 1;
        double scale = in.params.energy_scale;
        if (!(scale > 0.0)) scale = choose_energy_scale(in.scene, &in.params);
        fill_job<float>(in.scene, &in.params, &in.outputs, scale, jobs[k]);
        outputs[k] = ShardTargets{jobs[k].echogram_fx, jobs[k].ambisonic_fx, jobs[k].hit_counts, jobs[k].contrib_counts,
                                  jobs[k].surface_energy_fx};
        if (copies[k] > 1) {
            const size_t nb = 2 * static_cast<size_t>(kBands) * jobs[k].num_bins, na = jobs[k].ambisonic_fx ? 4 * nb : 0;
            const size_t ns = static_cast<size_t>(jobs[k].scene.num_surfaces), words = accumulator_words(in);
            jobs[k].shard_mask = copies[k] - 1;
            jobs[k].shard_stride = static_cast<int64_t>(words);
            jobs[k].echogram_fx = shards;
            if (na) jobs[k].ambisonic_fx = shards + nb;
            jobs[k].hit_counts = shards + nb + na;
            jobs[k].contrib_counts = shards + nb + na + ns;
            jobs[k].surface_energy_fx = shards + nb + na + 2 * ns;
            shards += words * static_cast<size_t>(copies[k]);
        }
        if (k > 0 && (jobs[k].rng_mode != jobs[0].rng_mode || jobs[k].render_ambisonics != jobs[0].render_ambisonics ||
                      (jobs[k].visual_limit > 0) != (jobs[0].visual_limit > 0)))
            return fail(AC_ERR_INVALID,
                        "one float32 launch needs one random-stream mode, ambisonics and visual-candidate setting");
        if (in.outputs.scale_out) *in.outputs.scale_out = scale;
        prefix[k] = total;
        jobs[k].ray_begin = total;
        total += in.params.num_rays;
        targets[k] = FinalizeTargets{in.outputs.echogram, in.params.render_ambisonics ? in.outputs.ambisonic : nullptr,
                                     in.outputs.surface_energy};
    }
    int entries = 0;
    const int rc = launch_stack_entries(cfg ? cfg->stack_entries : 0, need, &entries);
    if (rc != AC_OK) return rc;
    prefix[count] = total;
    group_rays[num_groups] = total;
    AC_CUDA_TRY(cudaSetDevice(device));
    unsigned char *ws = static_cast<unsigned char *>(workspace);
    AC_CUDA_TRY(cudaMemcpyAsync(ws + l.prefix, host + l.prefix, l.table_end - l.prefix, cudaMemcpyHostToDevice, stream));
    if (!host_staging) AC_CUDA_TRY(cudaStreamSynchronize(stream));
    AC_CUDA_TRY(cudaMemsetAsync(ws + l.queues, 0, sizeof(unsigned long long) * static_cast<size_t>(num_groups), stream));
    if (shard_words) AC_CUDA_TRY(cudaMemsetAsync(ws + l.shards, 0, sizeof(unsigned long long) * shard_words, stream));
    const Job<float> *d_jobs = reinterpret_cast<const Job<float> *>(ws + l.jobs);
    unsigned long long *counter = reinterpret_cast<unsigned long long *>(ws);
    {
        dim3 zgrid(32, static_cast<unsigned>(std::min<int32_t>(count, 65535)));
        zero_outputs_kernel<float><<<zgrid, 256, 0, stream>>>(d_jobs, count, counter);
        AC_CUDA_TRY(cudaGetLastError());
    }
    const int block = (cfg && cfg->block_size > 0) ? cfg->block_size : kDefaultBlock;
    if (block % 32 != 0 || block > 256) return fail(AC_ERR_INVALID, "block_size must be a multiple of 32 up to 256");
    if (total > 0) {
        FastTable table{};
        table.jobs = d_jobs;
        table.ray_begin = reinterpret_cast<const int64_t *>(ws + l.prefix);
        table.groups = reinterpret_cast<const FastGroup *>(ws + l.groups);
        table.num_jobs = count;
        table.chunk_counter = counter;
        table.group_next = reinterpret_cast<unsigned long long *>(ws + l.queues);
        table.group_ray_begin = reinterpret_cast<const int64_t *>(ws + l.group_rays);
        table.num_groups = static_cast<int32_t>(num_groups);
        table.lanes = cfg && cfg->grid_blocks > 0 ? 32 : warp_lanes(device, total, entries > 0 ? 4 : 16);
        table.chunk_rays = static_cast<int32_t>(table.lanes < 32 ? std::min<int64_t>(chunk_rays, table.lanes) : chunk_rays);
        Job<float> unused;
        std::memset(&unused, 0, sizeof(unused));
        FastScene none{};
        // ac_trace_batch partitions jobs so that one launch has one kernel variant.
        const FastKernel kernel = pick_kernel<false>(jobs[0].rng_mode == AC_RNG_PHILOX, jobs[0].render_ambisonics != 0,
                                                     jobs[0].visual_limit > 0, shard_words > 0, lean);
        const size_t smem = stack_smem_bytes(entries);
        const int grid = fast_grid(kernel, device, block, smem, spread_rays(total, table.lanes), cfg ? cfg->grid_blocks : 0);
        kernel<<<grid, block, smem, stream>>>(unused, none, table);
        AC_CUDA_TRY(cudaGetLastError());
    }
    {
        dim3 fgrid(16, static_cast<unsigned>(std::min<int32_t>(count, 65535)));
        const ShardTargets *d_outputs = reinterpret_cast<const ShardTargets *>(ws + l.outputs);
        if (shard_words) {
            gather_shards_kernel<<<fgrid, 256, 0, stream>>>(d_jobs, d_outputs, count);
            AC_CUDA_TRY(cudaGetLastError());
        }
        finalize_f32_kernel<<<fgrid, 256, 0, stream>>>(d_jobs, reinterpret_cast<const FinalizeTargets *>(ws + l.targets),
                                                       d_outputs, count);
        AC_CUDA_TRY(cudaGetLastError());
    }
    return AC_OK;
}

}  // namespace ac
