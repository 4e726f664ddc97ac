// fr_batch.cu -- gridding of many frames (coils x frames of a dynamic
// acquisition, or several volumes) with uneven sample counts in ONE persistent
// launch, replayable as a captured CUDA graph, and an autotuner for the tile
// shape, bin chunk and coil group.  No counterpart in the reference, which
// grids one dataset per GridLut::execute call (GridLut.cpp:53-78).
//
// Planning: every frame is normalised with its own bounds
// (ReconData::normalizeTraj, ReconData.cpp:201-225) and binned by the
// single-trajectory planner; its normalised samples, bin records, tap lists,
// work items and split tiles are appended to batch-wide arrays, and the items,
// split tiles and tap records are relabelled with their frame and global
// offsets.  Gridding: one sample-major copy of all frames' dcf * k, then a
// persistent scatter kernel that takes (coil group, item) work indices from a
// counter until the batch is done: the tap lanes, or without tap lists (a
// kernel too wide for them, coil groups of 32, tiles too large, refused, more
// than half of the free memory, or sparse frames: lanes_pay) the kernel that evaluates the taps.  Frame f's k-space is the block channels x
// n_f at complex offset channels * offset[f] and its grid the block
// channels x G^d at f * channels * G^d.
// Either way a work item's fixed-point sums have a scale per coil float, from that
// float's sum and largest value in the item: a weak coil keeps its bits beside strong ones.
// 64 frames of 8 k to 49 k samples, 12 coils, 384^2 grids: 1312 us evaluating the
// taps (one CTA of 128 KB per SM), 821 us from the lists.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "fr_internal.h"

using namespace fr;

struct fr_batch_s {
    fr_plan plan = nullptr;  // per-frame planner (tiling, LUT)
    int frames = 0;
    std::vector<long long> off;
    DevBuf frame_off, traj, recs, items, splits, counter;
    DevBuf taps, trecs, runs;  // tap lists of all frames, sample runs of the k-space copy
    int tap_words = 0;         // 0: no tap lists
    int chunk = 0;             // most records per work item
    long long nruns = 0;
    // per-call buffers; a captured graph has its own, which later calls with
    // more channels cannot move
    struct Scratch {
        DevBuf partials, kt, float_inv;
    } direct, captured;
    long long n_total = 0, npairs = 0, nitems = 0, nslots = 0, nsplits = 0;
    int blocks = 0;
    bool ready = false;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    ~fr_batch_s()
    {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        if (plan) fr_plan_destroy(plan);
    }
};

namespace {

__global__ void fixup_items_kernel(WorkItem *it, long long n, long long rec_off, int slot_off, int frame)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        WorkItem w = it[i];
        w.begin += rec_off;
        if (w.slot >= 0) w.slot += slot_off;
        w.pad = frame;
        it[i] = w;
    }
}

__global__ void fixup_splits_kernel(SplitTile *st, long long n, int slot_off, int frame)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        st[i].first_slot += slot_off;
        st[i].pad = frame;
    }
}

// A frame's tap records name samples of the whole batch.
__global__ void append_trecs_kernel(const unsigned long long *__restrict__ src, long long n, unsigned sample_off,
                                    unsigned long long *__restrict__ dst)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = src[i] + sample_off;  // the sample is the low 32 bits: no carry below 2^32 samples
}

// Grow `b` to hold `need` bytes, keeping its first `used` bytes.
int grow_keep(DevBuf &b, size_t used, size_t need, cudaStream_t s)
{
    if (need <= b.bytes && b.ptr) return FR_OK;
    DevBuf grown;
    if (grown.reserve(std::max<size_t>(need, b.bytes + b.bytes / 2))) return FR_ERR_OUT_OF_MEMORY;
    if (used) {
        FR_CUDA(cudaMemcpyAsync(grown.ptr, b.ptr, used, cudaMemcpyDeviceToDevice, s));
        FR_CUDA(cudaStreamSynchronize(s));
    }
    std::swap(b.ptr, grown.ptr);
    std::swap(b.bytes, grown.bytes);
    return FR_OK;
}

int fill_batch_grid(fr_batch b, fr_batch_s::Scratch &sc, int lane_floats, BatchGrid *g)
{
    fr_plan p = b->plan;
    g->dim = p->dim;
    g->G = p->G;
    for (int d = 0; d < 3; ++d) {
        g->tile[d] = p->tile[d];
        g->ntile[d] = p->ntile[d];
    }
    g->coil_group = p->coil_group;
    g->L = p->L;
    g->smax = p->lut_smax;
    g->kc = p->lut_kc;
    g->lut_absmax = p->lut_absmax;
    g->checkerboard = (p->flags & FR_PLAN_CHECKERBOARD) ? 1 : 0;
    g->traj = b->traj.as<float4>();
    g->recs = b->recs.as<unsigned long long>();
    g->items = b->items.as<WorkItem>();
    g->splits = b->splits.as<SplitTile>();
    g->lut_e = p->lut_e.as<float4>();
    g->frame_off = b->frame_off.as<long long>();
    g->nitems = b->nitems;
    g->nsplits = b->nsplits;
    g->n_total = b->n_total;
    g->partials = sc.partials.as<float>();
    g->work_counter = b->counter.as<int>();
    g->blocks = b->blocks;
    g->sum_limit = fixed_sum_limit(b->chunk);
    g->lane_floats = lane_floats;
    if (lane_floats > 0) {
        g->tap_words = b->tap_words;
        g->taps = b->taps.as<unsigned>();
        g->trecs = b->trecs.as<unsigned long long>();
        g->lutw = p->lut_d.as<float>();
        g->runs = b->runs.as<FrameRun>();
        g->nruns = b->nruns;
        g->kt = sc.kt.as<float>();
        g->float_inv = sc.float_inv.as<float>();
        g->err = p->err_dev;
    }
    return FR_OK;
}

// Tap lists and the copy of the k-space are a choice of speed: a buffer for them grows
// only into half of the free memory, and is given up where that runs out all the
// same, so that what fits without them still fits, and its caller's grids too.
int reserve_spare(DevBuf &b, size_t need)
{
    if (need <= b.bytes && b.ptr) return FR_OK;
    b.release();
    return need <= device_bytes_free() / 2 ? b.reserve(need) : fail(FR_ERR_OUT_OF_MEMORY, "no spare device memory");
}

// false: there was nothing to give up.  A captured graph reads the lists and its copy.
bool drop_tap_lists(fr_batch b)
{
    fr_plan p = b->plan;
    if (b->exec || (!b->taps.ptr && !p->taps.ptr && !b->direct.kt.ptr && !b->captured.kt.ptr)) return false;
    b->tap_words = 0;
    p->taps_enabled = false;  // until the next trajectories
    for (DevBuf *d : {&b->taps, &b->trecs, &p->taps, &p->trecs}) d->release();
    for (fr_batch_s::Scratch *sc : {&b->direct, &b->captured}) {
        sc->kt.release();
        sc->float_inv.release();
    }
    return true;
}

// Whether the tap lanes of `floats` coil floats are the faster scatter of this batch: sparse
// frames cost their tiles' clearing and writing, which the evaluating kernel's 16 warps and
// plain coil rows do faster, and the lists' copy and scales come on top. The lines, in
// samples per cell, are where the two crossed (lists / evaluating, us): 2D, 64 frames of
// 384^2, 16 coils 0.028 a cell 566 / 477, 0.056 626 / 593, 0.11 741 / 808; 32 of 256^2, 9 coils
// 0.031 117 / 102, 0.062 128 / 128; 6 coils 0.016 84 / 78, 0.031 95 / 95; 3 coils 0.016 70 / 66,
// 0.031 78 / 81; 3D, 8 frames of 96^3, 16 coils 0.005 308 / 287, 0.018 409 / 404, 0.036
// 467 / 509, 8 coils 0.001 158 / 169.
bool lanes_pay(fr_batch b, int floats)
{
    fr_plan p = b->plan;
    const double cells = (double)b->frames * p->ntiles * p->tile[0] * p->tile[1] * p->tile[2];
    const double line = p->dim == 3 ? (floats > 16 ? 0.0175 : 0.0) : floats > 16 ? 0.075 : floats > 8 ? 0.03 : 0.02;
    return floats > 0 && (double)b->n_total >= line * cells;
}

// The buffers of a call, and whether it takes the tap lists (*lane_floats > 0):
// where their copy of the k-space does not fit, the taps are evaluated.
int ensure_scratch(fr_batch b, fr_batch_s::Scratch &sc, int channels, int *lane_floats)
{
    fr_plan p = b->plan;
    const long long K = (long long)p->tile[0] * p->tile[1] * p->tile[2];
    const size_t part = b->nslots > 0 ? grid_partials_bytes(b->nslots, channels, p->coil_group, K) : 0;
    *lane_floats = b->tap_words > 0 ? batch_lane_floats(K, p->coil_group, p->L, channels) : 0;
    if (!lanes_pay(b, *lane_floats)) *lane_floats = 0;
    if (part > 0 && sc.partials.reserve(part)) {
        if (!drop_tap_lists(b) || sc.partials.reserve(part)) return FR_ERR_OUT_OF_MEMORY;
        *lane_floats = 0;
    }
    const size_t rows = (size_t)std::max<long long>(b->n_total, 1);
    const size_t row = (size_t)(channels + (channels & 1)) * 8;  // bytes
    if (*lane_floats > 0 && (reserve_spare(sc.kt, rows * row) || reserve_spare(sc.float_inv, (size_t)b->nitems * row)))
        *lane_floats = 0;
    return FR_OK;
}

// An error an earlier call's kernels left in the plan's mapped word.
int kernel_error(fr_batch b)
{
    fr_plan p = b->plan;
    if (!p->err_host || !*p->err_host) return FR_OK;
    const int e = *p->err_host;
    *p->err_host = 0;
    return fail(e, e == FR_ERR_DEVICE_TIMEOUT ? "a bulk copy of the scatter never completed (an earlier call)"
                                              : "the plan's tap lists overflowed a sample slot (internal error)");
}

int check_grid_args(fr_batch b, const float *d_kdata, const float *d_dcf, int channels, const float *d_grid)
{
    if (!b || !d_grid) return fail(FR_ERR_INVALID_ARGUMENT, "null argument");
    if (!b->ready) return fail(FR_ERR_NOT_PLANNED, "fr_batch_set_trajectories has not run");
    if (channels <= 0) return fail(FR_ERR_INVALID_ARGUMENT, "channels must be positive");
    if (b->n_total && (!d_kdata || !d_dcf)) return fail(FR_ERR_INVALID_ARGUMENT, "null argument");
    if ((reinterpret_cast<uintptr_t>(d_kdata) & 7) || (reinterpret_cast<uintptr_t>(d_grid) & 7))
        return fail(FR_ERR_INVALID_ARGUMENT, "complex buffers must be 8-byte aligned");
    return FR_OK;
}

}  // namespace

extern "C" {

int fr_batch_create(const fr_plan_desc *desc, fr_batch *out)
{
    if (!out) return fail(FR_ERR_INVALID_ARGUMENT, "null argument");
    *out = nullptr;
    if (!desc) return fail(FR_ERR_INVALID_ARGUMENT, "null argument");
    auto b = new (std::nothrow) fr_batch_s;
    if (!b) return fail(FR_ERR_OUT_OF_MEMORY, "batch");
    fr_plan_desc d = *desc;
    if (d.dim == 2 && d.tile[0] <= 0 && d.tile[1] <= 0) {
        // 64 KB of tile: two CTAs per SM, so that one's zeroing, waits and flush
        // hide behind the other's adds (64 frames, 12 coils: scatter 800 us with 32 x 32 and one CTA, 690 so)
        d.tile[0] = 32;
        d.tile[1] = 16;
    }
    int st = fr_plan_create(&d, &b->plan);
    if (st) {
        delete b;
        return st;
    }
    *out = b;
    return FR_OK;
}

int fr_batch_destroy(fr_batch b)
{
    delete b;
    return FR_OK;
}

int fr_batch_set_trajectories(fr_batch b, const float *d_traj, const size_t *offsets, int frames, void *stream)
{
    if (!b || !offsets || frames < 1) return fail(FR_ERR_INVALID_ARGUMENT, "null argument or no frames");
    if (offsets[0] != 0) return fail(FR_ERR_INVALID_ARGUMENT, "offsets[0] must be 0");
    for (int f = 0; f < frames; ++f)
        if (offsets[f + 1] < offsets[f]) return fail(FR_ERR_INVALID_ARGUMENT, "offsets must be non-decreasing");
    if (offsets[frames] && !d_traj) return fail(FR_ERR_INVALID_ARGUMENT, "null trajectory");
    if (reinterpret_cast<uintptr_t>(d_traj) & 15) return fail(FR_ERR_INVALID_ARGUMENT, "trajectory must be 16-byte aligned");
    cudaStream_t s = (cudaStream_t)stream;
    fr_plan p = b->plan;
    b->ready = false;
    if (b->exec) {
        cudaGraphExecDestroy(b->exec);
        b->exec = nullptr;
    }
    if (b->graph) {
        cudaGraphDestroy(b->graph);
        b->graph = nullptr;
    }
    b->frames = frames;
    b->off.assign(offsets, offsets + frames + 1);
    b->n_total = (long long)offsets[frames];
    auto first = [&] {
        return b->traj.reserve(std::max<long long>(b->n_total, 1) * 16) || b->frame_off.reserve((size_t)(frames + 1) * 8) ||
               b->counter.reserve(256);
    };
    p->taps_enabled = !(p->flags & FR_PLAN_NO_TAP_LISTS);
    if (first() && (!drop_tap_lists(b) || first())) return FR_ERR_OUT_OF_MEMORY;  // (lists of the last trajectories)
    FR_CUDA(cudaMemcpyAsync(b->frame_off.ptr, b->off.data(), (size_t)(frames + 1) * 8, cudaMemcpyHostToDevice, s));
    long long npairs = 0, nitems = 0, nslots = 0, nsplits = 0;
    b->tap_words = 0;
    b->chunk = 0;
    bool taps = b->n_total <= 0x7FFFFFFFll;
    std::vector<FrameRun> runs;
    // true: memory ran out beside the tap lists, which are now given up
    auto without_lists = [&](int st) {
        if (st != FR_ERR_OUT_OF_MEMORY || !drop_tap_lists(b)) return false;
        taps = false;
        return true;
    };
    for (int f = 0; f < frames; ++f) {
        const size_t nf = offsets[f + 1] - offsets[f];
        int st = plan_run(p, d_traj + 4 * offsets[f], nf, s);  // synchronises s
        if (without_lists(st)) st = plan_run(p, d_traj + 4 * offsets[f], nf, s);
        if (st) return st;
        b->chunk = std::max(b->chunk, p->chunk);
        if (nslots + p->nslots > 0x7FFFFFFFll || nitems + p->nitems > 0x7FFFFFFFll)
            return fail(FR_ERR_UNSUPPORTED, "batch too large for 32-bit item indices");
        auto grow = [&] {
            int e = grow_keep(b->recs, (size_t)npairs * 8, (size_t)(npairs + p->npairs) * 8, s);
            if (!e) e = grow_keep(b->items, (size_t)nitems * sizeof(WorkItem), (size_t)(nitems + p->nitems) * sizeof(WorkItem), s);
            if (!e) e = grow_keep(b->splits, (size_t)nsplits * sizeof(SplitTile),
                                  (size_t)(nsplits + std::max<long long>(p->nsplits, 0)) * sizeof(SplitTile), s);
            return e;
        };
        st = grow();
        if (without_lists(st)) st = grow();
        if (st) return st;
        if (nf > 0 && taps) {
            if (p->tap_words > 0 && b->tap_words == 0 && !reserve_spare(b->taps, (size_t)b->n_total * p->tap_words * 4))
                b->tap_words = p->tap_words;
            taps = p->tap_words > 0 && b->tap_words > 0 &&
                   !grow_keep(b->trecs, (size_t)npairs * 8, (size_t)(npairs + p->npairs) * 8, s);
            if (!taps) drop_tap_lists(b);
        }
        if (nf > 0 && taps) {
            FR_CUDA(cudaMemcpyAsync(b->taps.as<unsigned>() + offsets[f] * (size_t)b->tap_words, p->taps.ptr,
                                    nf * (size_t)b->tap_words * 4, cudaMemcpyDeviceToDevice, s));
            if (p->npairs) {
                append_trecs_kernel<<<(int)std::min<long long>((p->npairs + 255) / 256, 1024), 256, 0, s>>>(
                    p->trecs.as<unsigned long long>(), p->npairs, (unsigned)offsets[f],
                    b->trecs.as<unsigned long long>() + npairs);
                FR_CHECK_LAUNCH("append_trecs_kernel");
            }
            for (size_t k = 0; k < nf; k += (size_t)frame_run_samples())
                runs.push_back(FrameRun{(long long)offsets[f], (int)nf, (int)k, f, 0});
        }
        if (nf) FR_CUDA(cudaMemcpyAsync(b->traj.as<float4>() + offsets[f], p->traj.ptr, nf * 16, cudaMemcpyDeviceToDevice, s));
        if (p->npairs)
            FR_CUDA(cudaMemcpyAsync(b->recs.as<unsigned long long>() + npairs, p->pairs.ptr, (size_t)p->npairs * 8,
                                    cudaMemcpyDeviceToDevice, s));
        if (p->nitems) {
            WorkItem *dst = b->items.as<WorkItem>() + nitems;
            FR_CUDA(cudaMemcpyAsync(dst, p->items.ptr, (size_t)p->nitems * sizeof(WorkItem), cudaMemcpyDeviceToDevice, s));
            fixup_items_kernel<<<(int)std::min<long long>((p->nitems + 255) / 256, 1024), 256, 0, s>>>(
                dst, p->nitems, npairs, (int)nslots, f);
            FR_CHECK_LAUNCH("fixup_items_kernel");
        }
        if (p->nsplits) {
            SplitTile *dst = b->splits.as<SplitTile>() + nsplits;
            FR_CUDA(cudaMemcpyAsync(dst, p->splits.ptr, (size_t)p->nsplits * sizeof(SplitTile), cudaMemcpyDeviceToDevice, s));
            fixup_splits_kernel<<<(int)std::min<long long>((p->nsplits + 255) / 256, 1024), 256, 0, s>>>(
                dst, p->nsplits, (int)nslots, f);
            FR_CHECK_LAUNCH("fixup_splits_kernel");
        }
        npairs += p->npairs;
        nitems += p->nitems;
        nslots += p->nslots;
        nsplits += p->nsplits;
    }
    if (!taps || b->tap_words == 0 || b->runs.reserve(std::max<size_t>(runs.size(), 1) * sizeof(FrameRun)))
        drop_tap_lists(b);
    b->nruns = (long long)runs.size();
    if (b->tap_words > 0 && !runs.empty())
        FR_CUDA(cudaMemcpyAsync(b->runs.ptr, runs.data(), runs.size() * sizeof(FrameRun), cudaMemcpyHostToDevice, s));
    FR_CUDA(cudaStreamSynchronize(s));  // the planner's buffers are reused by the next call
    b->npairs = npairs;
    b->nitems = nitems;
    b->nslots = nslots;
    b->nsplits = nsplits;
    const long long K = (long long)p->tile[0] * p->tile[1] * p->tile[2];
    int st = batch_grid_setup(p->dim, K, p->coil_group, p->L, &b->blocks);
    if (st) return st;
    b->ready = true;
    return FR_OK;
}

int fr_batch_stats(fr_batch b, long long *frames, long long *samples, long long *items, long long *slots,
                   int *persistent_ctas)
{
    if (!b) return fail(FR_ERR_INVALID_ARGUMENT, "null argument");
    if (frames) *frames = b->frames;
    if (samples) *samples = b->n_total;
    if (items) *items = b->nitems;
    if (slots) *slots = b->nslots;
    if (persistent_ctas) {
        fr_plan p = b->plan;
        const long long K = (long long)p->tile[0] * p->tile[1] * p->tile[2];
        *persistent_ctas = b->blocks;
        if (b->ready && b->tap_words > 0 && lanes_pay(b, batch_lane_floats(K, p->coil_group, p->L, p->coil_group)))
            return batch_lane_ctas(K, p->coil_group, p->L, persistent_ctas);
    }
    return FR_OK;
}

int fr_batch_grid(fr_batch b, const float *d_kdata, const float *d_dcf, int channels, float *d_grid, void *stream)
{
    int st = check_grid_args(b, d_kdata, d_dcf, channels, d_grid), nf = 0;
    if (st) return st;
    if ((st = kernel_error(b)) || (st = ensure_scratch(b, b->direct, channels, &nf))) return st;
    BatchGrid g;
    fill_batch_grid(b, b->direct, nf, &g);
    return batch_grid_run(g, d_kdata, d_dcf, channels, d_grid, (cudaStream_t)stream);
}

int fr_batch_capture(fr_batch b, const float *d_kdata, const float *d_dcf, int channels, float *d_grid, void *stream)
{
    int st = check_grid_args(b, d_kdata, d_dcf, channels, d_grid), nf = 0;
    if (st) return st;
    if (!stream) return fail(FR_ERR_INVALID_ARGUMENT, "capture needs a created stream, not the legacy default stream");
    if (b->exec) {
        cudaGraphExecDestroy(b->exec);
        b->exec = nullptr;
    }
    if (b->graph) {
        cudaGraphDestroy(b->graph);
        b->graph = nullptr;
    }
    if ((st = kernel_error(b)) || (st = ensure_scratch(b, b->captured, channels, &nf))) return st;
    cudaStream_t s = (cudaStream_t)stream;
    BatchGrid g;
    fill_batch_grid(b, b->captured, nf, &g);
    FR_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    st = batch_grid_run(g, d_kdata, d_dcf, channels, d_grid, s);
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamEndCapture(s, &graph);
    if (st) {
        if (graph) cudaGraphDestroy(graph);
        return st;
    }
    if (e != cudaSuccess) return cuda_fail(e, "cudaStreamEndCapture");
    e = cudaGraphInstantiate(&b->exec, graph, 0);
    if (e != cudaSuccess) {
        cudaGraphDestroy(graph);
        b->exec = nullptr;
        return cuda_fail(e, "cudaGraphInstantiate");
    }
    b->graph = graph;
    return FR_OK;
}

int fr_batch_replay(fr_batch b, void *stream)
{
    if (!b) return fail(FR_ERR_INVALID_ARGUMENT, "null argument");
    if (!b->exec) return fail(FR_ERR_NOT_PLANNED, "no captured graph: call fr_batch_capture first");
    if (const int st = kernel_error(b)) return st;
    FR_CUDA(cudaGraphLaunch(b->exec, (cudaStream_t)stream));
    note_launch();
    return FR_OK;
}

int fr_batch_autotune(const fr_plan_desc *base, const float *d_traj, const size_t *offsets, int frames,
                      const float *d_kdata, const float *d_dcf, int channels, float *d_grid, int repeats,
                      fr_plan_desc *best, float *best_ms, void *stream)
{
    if (!base || !best) return fail(FR_ERR_INVALID_ARGUMENT, "null argument");
    if (repeats < 1) repeats = 3;
    cudaStream_t s = (cudaStream_t)stream;
    struct Cand {
        int t[3];
        int chunk;
        int cg;
    };
    std::vector<Cand> cands;
    const int cgs[3] = {8, 16, 32};
    if (base->dim == 3) {
        const int shapes[][3] = {{8, 8, 8}, {16, 8, 8}, {8, 8, 4}, {16, 8, 4}, {16, 16, 4}};
        for (auto &sh : shapes)
            for (int chunk : {2048, 4096, 8192})
                for (int cg : cgs) cands.push_back({{sh[0], sh[1], sh[2]}, chunk, cg});
    } else {
        const int shapes[][2] = {{16, 16}, {32, 16}, {32, 32}, {64, 32}, {64, 64}};
        for (auto &sh : shapes)
            for (int chunk : {1024, 2048, 4096, 8192})
                for (int cg : cgs) cands.push_back({{sh[0], sh[1], 1}, chunk, cg});
    }
    cudaEvent_t e0, e1;
    FR_CUDA(cudaEventCreate(&e0));
    FR_CUDA(cudaEventCreate(&e1));
    float bestv = 1e30f;
    int found = 0;
    for (const Cand &c : cands) {
        if (c.cg > 8 && c.cg >= 2 * channels) continue;  // a coil group at least twice the coils
        fr_plan_desc d = *base;
        for (int i = 0; i < 3; ++i) d.tile[i] = c.t[i];
        d.chunk = c.chunk;
        d.coil_group = c.cg;
        fr_batch b = nullptr;
        if (fr_batch_create(&d, &b) != FR_OK) continue;  // shape does not fit: skip
        float ms = 1e30f;
        int st = fr_batch_set_trajectories(b, d_traj, offsets, frames, stream);
        if (!st) st = fr_batch_grid(b, d_kdata, d_dcf, channels, d_grid, stream);  // warm-up
        for (int r = 0; !st && r < repeats; ++r) {
            cudaEventRecord(e0, s);
            st = fr_batch_grid(b, d_kdata, d_dcf, channels, d_grid, stream);
            cudaEventRecord(e1, s);
            if (!st && cudaEventSynchronize(e1) == cudaSuccess) {
                float t = 0.f;
                cudaEventElapsedTime(&t, e0, e1);
                ms = std::min(ms, t);
            }
        }
        fr_batch_destroy(b);
        if (st == FR_ERR_CUDA || st == FR_ERR_OUT_OF_MEMORY) {
            cudaEventDestroy(e0);
            cudaEventDestroy(e1);
            return st;
        }
        if (!st && ms < bestv) {
            bestv = ms;
            *best = d;
            found = 1;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (!found) return fail(FR_ERR_UNSUPPORTED, "no tiling candidate ran");
    if (best_ms) *best_ms = bestv;
    return FR_OK;
}

}  // extern "C"
