/*
 * sciddicaT_batch.cu -- an ensemble of independent SCIDDICA-T instances
 * (calibration ensembles, scenarios) advanced together, forward and adjoint.
 * Every instance is the plain program of OpenCAL/examples/cal_sciddicaT
 * (flat boundary, von Neumann, EP 1 outflows + EP 2 width update,
 * OpenCAL-OMP/examples/calomp_sciddicaT/source/sciddicaT.c), each with its
 * own grid size, DEM, source, p_r and p_epsilon.
 *
 * Layout.  The fields of all instances are packed back to back, one
 * allocation per field; instance b occupies [off_b, off_b + rows_b*cols_b)
 * with off_b a multiple of 32 cells (256 bytes).  A device table holds
 * per-instance dimensions and parameters.  Each instance is cut into tiles;
 * the tiles of all instances are numbered in one range.
 *
 * Forward and adjoint: one list of the wet cells of all instances per step
 * (sciddicaT_wet.cuh), two launches per step each way in the recorded
 * evaluation, all steps in one cooperative launch otherwise.  Dry regions cost
 * nothing, and every instance stays bit-identical to a run of its own.
 *
 * Tape.  The forward TAPES each wet cell's elimination set and differences,
 * step after step at offsets the steps chain on the device; the backward
 * walks it in reverse and reads nothing else but lambda.  The tape holds
 * every wet cell of every step, so it grows with the flow's area times T;
 * when it would not fit in device memory the ensemble falls back to sqrt(T)
 * checkpointing: h is stored every K = ceil(sqrt(T)) steps and the backward
 * recomputes one segment at a time from its checkpoint, taping that segment
 * only.  lambda is updated in place, and dL/dp_r and dL/dp_eps are added up,
 * in a fixed order: the gradients repeat bit for bit (the losses, added up
 * with atomics, need not).
 *
 * The tile shape -- the unit of the update and of the gather -- is 32x8 or
 * chosen by a small autotuner (cal_sdt_batch_autotune): each candidate shape
 * times a forward probe with CUDA events and the fastest is kept for the
 * ensemble.
 */
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "sciddicaT_wet.cuh"

namespace sdtb {

using sdtw::Adj;
using sdtw::Dev;
using sdtw::Inst;
using sdtw::T;

constexpr int MAX_INST = 4096;
constexpr long long ALIGN = 32; /* cells */

struct Shape {
    int tw, th;
};
constexpr int NSHAPES = 5;
static const Shape kShapes[NSHAPES] = {{32, 16}, {64, 16}, {64, 32}, {16, 8}, {32, 8}};

struct Batch {
    int B = 0, steps = 0, K = 0, nseg = 0, shape = 4;
    std::vector<Inst> inst;
    std::vector<long long> offs; /* B + 1 (offs[B] = N) */
    Dev d = {};
    Adj a = {};
    double *z_dem = nullptr, *z = nullptr, *h0 = nullptr;
    double* ckpt = nullptr; /* nseg x N, segments only */
    double* loss = nullptr; /* B */
    unsigned long long* words = nullptr; /* of the cooperative launches */
    cudaStream_t st = nullptr;
    /* f is zero everywhere before a run, but after one that gave up (words
     * say so, and k_init clears it) */
    bool flows_clear = false;
    /* the loss + gradient evaluation recorded once as a CUDA graph and
     * replayed every call: tape offsets chained on the device, results
     * copied into pinned host memory (h_out: B losses, 2B gradients, then
     * the tape entries needed and the cooperative launches' error word); valid
     * for the target, the dL/dh0 buffer and what the tape holds (dropped with
     * the tiles and the tape it was recorded with) */
    double* h_out = nullptr; /* pinned: 3B doubles + two long longs */
    cudaGraphExec_t gexec = nullptr;
    const double* g_target = nullptr;
    const double* g_gh0 = nullptr;
    long long graph_launches = 0;
    long long graph_nodes = 0; /* kernel and copy nodes of the recorded evaluation */
    bool use_graph = true;
    /* what the tape holds: the whole rollout (run_full: the backward
     * recomputes nothing) or one sqrt(T) segment at a time.  tape_mode -1
     * chooses by memory: the whole rollout while its tape (plus a quarter)
     * fits in half of the device memory free for it, else segments; 0
     * always segments, 1 always the whole rollout */
    int tape_mode = -1;
    bool run_full = true;
    bool g_full = true;
    long long last_need = 0; /* entries of tape the last evaluation needed */
};

static void drop_graph(Batch& bt)
{
    if (bt.gexec)
        cudaGraphExecDestroy(bt.gexec);
    bt.gexec = nullptr;
}

/* a tape of `cap` entries; false when out of memory.  A recorded evaluation
 * holds the old arrays and the old capacity in its nodes, and the new arrays
 * may lie where some of the old ones did: it goes with them. */
static bool grow_tape(Batch& bt, long long cap)
{
    Dev& d = bt.d;
    drop_graph(bt);
    cudaFree(d.t_entry);
    cudaFree(d.t_elim);
    cudaFree(d.t_diff);
    d.t_entry = nullptr;
    d.t_elim = nullptr;
    d.t_diff = nullptr;
    d.cap = 0;
    if (cudaMalloc(&d.t_entry, (size_t)cap * sizeof(sdtw::Entry)) != cudaSuccess ||
        cudaMalloc(&d.t_elim, (size_t)cap) != cudaSuccess ||
        cudaMalloc(&d.t_diff, (size_t)cap * sizeof(sdtw::D4)) != cudaSuccess) {
        (void)cudaGetLastError();
        cudaFree(d.t_entry);
        cudaFree(d.t_elim);
        d.t_entry = nullptr;
        d.t_elim = nullptr;
        return false;
    }
    d.cap = cap;
    return true;
}

/* re-tile every instance for the current shape; false when out of memory
 * (d.tiles is then NULL, and nothing runs until another shape fits) */
static bool tiles_for(Batch& bt)
{
    Dev& d = bt.d;
    const int tw = kShapes[bt.shape].tw, th = kShapes[bt.shape].th;
    drop_graph(bt); /* the work-list buffers are reallocated */
    std::vector<int> tinst;
    for (int b = 0; b < bt.B; b++) {
        Inst& I = bt.inst[b];
        I.tiles_x = (I.cols + tw - 1) / tw;
        I.tiles_y = (I.rows + th - 1) / th;
        I.tile0 = (int)tinst.size();
        tinst.insert(tinst.end(), (size_t)I.tiles_x * I.tiles_y, b);
    }
    d.ntiles = (int)tinst.size();
    d.lw = d.lh = 0;
    while (1 << d.lw < tw)
        d.lw++;
    while (1 << d.lh < th)
        d.lh++;
    cudaStreamSynchronize(bt.st);
    cudaFree((void*)d.tile_inst);
    cudaFree(d.stamps);
    cudaFree(d.tiles);
    d.tile_inst = nullptr;
    d.stamps = nullptr;
    d.tiles = nullptr;
    bool ok = cudaMalloc((void**)&d.tile_inst, sizeof(int) * tinst.size()) == cudaSuccess &&
              cudaMalloc(&d.stamps, sizeof(int) * tinst.size()) == cudaSuccess &&
              cudaMalloc(&d.tiles, sizeof(int) * std::max<size_t>(1, (size_t)d.ntiles * bt.steps)) == cudaSuccess;
    if (!ok) {
        (void)cudaGetLastError();
        cudaFree(d.tiles);
        d.tiles = nullptr;
        return false;
    }
    cudaMemcpy((void*)d.tile_inst, tinst.data(), sizeof(int) * tinst.size(), cudaMemcpyHostToDevice);
    cudaMemcpy((void*)d.inst, bt.inst.data(), sizeof(Inst) * bt.B, cudaMemcpyHostToDevice);
    return true;
}

/* steps [t0, t1) queued: in one cooperative launch, or, to be recorded,
 * launch by launch */
static void queue_steps(Batch& bt, int t0, int t1, int epoch0, bool taped, bool recorded)
{
    if (recorded)
        sdtw::queue_steps(bt.d, t0, t1, epoch0, taped, bt.st);
    else
        sdtw::launch_steps(bt.d, t0, t1, epoch0, taped, bt.words, bt.st);
}

static void queue_adjoint(Batch& bt, Adj& a, int t0, int t1, bool recorded)
{
    if (recorded)
        sdtw::queue_adjoint(bt.d, a, t0, t1, bt.st);
    else
        sdtw::launch_sweep(bt.d, a, t0, t1, bt.words, bt.st);
}

/* before the first run: no outflows, and no run that gave up */
static void first_state(Batch& bt)
{
    if (bt.flows_clear)
        return;
    cudaMemsetAsync(bt.d.f, 0, (size_t)bt.d.N * sizeof(sdtw::D4), bt.st);
    cudaMemsetAsync(bt.words, 0, sizeof(unsigned long long) * 16 * sdtw::NWORDS, bt.st);
    bt.flows_clear = !sdtw::capturing(bt.st); /* what a caller captures has not run yet */
}

/* The initial state and `steps` steps from it, queued.  keep: h every K
 * steps into the checkpoints; taped: every step onto the tape (toff[0] = 0,
 * need reset). */
static void forward(Batch& bt, int steps, bool keep, bool taped, bool recorded)
{
    Dev& d = bt.d;
    cudaStream_t st = bt.st;
    const size_t offs = sizeof(long long) * (bt.B + 1);
    cudaMemsetAsync(d.stamps, 0, sizeof(int) * d.ntiles, st);
    cudaMemsetAsync(d.counts, 0, sizeof(int) * (bt.steps + 1), st);
    cudaMemsetAsync(d.nlist, 0, sizeof(int) * (bt.steps + 1), st);
    if (taped || keep) {
        cudaMemsetAsync(d.toff, 0, sizeof(long long), st);
        cudaMemsetAsync(d.need, 0, sizeof(long long), st);
    }
    first_state(bt);
    sdtw::k_init<<<sdtw::dense_blocks(d.N), T, offs, st>>>(d, bt.z_dem, bt.h0, bt.z, bt.words);
    cudaMemsetAsync(bt.words, 0, sizeof(unsigned long long) * 16 * sdtw::NWORDS, st);
    for (int t = 0; t < steps; t += keep ? bt.K : steps) {
        const int t1 = std::min(t + (keep ? bt.K : steps), steps);
        if (keep)
            cudaMemcpyAsync(bt.ckpt + (size_t)(t / bt.K) * d.N, d.h, (size_t)d.N * sizeof(double),
                            cudaMemcpyDeviceToDevice, st);
        queue_steps(bt, t, t1, 1, taped, recorded);
    }
    if (steps > 0)
        sdtw::k_clear_flows<<<sdtw::BLOCKS, T, 0, st>>>(d, steps - 1);
}

static void destroy(Batch* bt)
{
    if (bt->st)
        cudaStreamSynchronize(bt->st);
    drop_graph(*bt);
    if (bt->h_out)
        cudaFreeHost(bt->h_out);
    Dev& d = bt->d;
    Adj& a = bt->a;
    void* ptrs[] = {(void*)d.inst, (void*)d.offs, (void*)d.tile_inst, d.h,     d.zh,    d.f,       d.list[0], d.list[1],
                    d.nlist,       d.tiles,       d.counts,           d.stamps, d.t_entry, d.t_elim, d.t_diff,  d.toff,
                    d.need,        a.lam,         a.mu,               a.stamp, a.w,     a.g,       a.grad,    a.part,
                    bt->z_dem,     bt->z,         bt->h0,             bt->ckpt, bt->loss, bt->words};
    for (void* p : ptrs)
        cudaFree(p);
    if (bt->st)
        cudaStreamDestroy(bt->st);
    delete bt;
}

} // namespace sdtb

using sdtb::Batch;

/* Create an ensemble of B instances.  dims[2b], dims[2b+1] = rows, cols;
 * params[2b], params[2b+1] = p_r, p_eps; z_dem, h0: host arrays holding the
 * instances' rows*cols values back to back (row-major, unpadded); `steps`
 * per rollout.  NULL on a bad argument or when device memory runs out. */
extern "C" void* cal_sdt_batch_create(int B, const int* dims, const double* params, const double* z_dem_host,
                                      const double* h0_host, int steps)
{
    if (B <= 0 || B > sdtb::MAX_INST || steps < 0 || !dims || !params || !z_dem_host || !h0_host)
        return nullptr;
    Batch* bt = new Batch();
    bt->B = B;
    bt->steps = steps;
    bt->K = (int)ceil(sqrt((double)(steps > 0 ? steps : 1)));
    bt->nseg = steps > 0 ? (steps + bt->K - 1) / bt->K : 1;
    bt->offs.assign(B + 1, 0);
    for (int b = 0; b < B; b++) {
        sdtb::Inst I;
        memset(&I, 0, sizeof(I));
        I.rows = dims[2 * b];
        I.cols = dims[2 * b + 1];
        if (I.rows <= 0 || I.cols <= 0) {
            delete bt;
            return nullptr;
        }
        I.off = bt->offs[b];
        I.r = params[2 * b];
        I.eps = params[2 * b + 1];
        memcpy(&I.eps_bits, &I.eps, sizeof(double));
        bt->inst.push_back(I);
        const long long n = (long long)I.rows * I.cols;
        bt->offs[b + 1] = bt->offs[b] + (n + sdtb::ALIGN - 1) / sdtb::ALIGN * sdtb::ALIGN;
    }
    sdtw::Dev& d = bt->d;
    d.B = B;
    d.N = bt->offs[B];
    const size_t nb = (size_t)d.N * sizeof(double);
    /* packed cell indices are 32-bit; the adjoint's arrays and the
     * checkpoints come with the first evaluation that needs them */
    bool ok = d.N < 0x7fffffffLL && cudaStreamCreateWithFlags(&bt->st, cudaStreamNonBlocking) == cudaSuccess &&
              cudaMalloc((void**)&d.inst, sizeof(sdtb::Inst) * B) == cudaSuccess &&
              cudaMalloc((void**)&d.offs, sizeof(long long) * (B + 1)) == cudaSuccess &&
              cudaMalloc(&d.counts, sizeof(int) * (steps + 1)) == cudaSuccess &&
              cudaMalloc(&d.nlist, sizeof(int) * (steps + 1)) == cudaSuccess &&
              cudaMalloc(&d.toff, sizeof(long long) * (steps + 1)) == cudaSuccess &&
              cudaMalloc(&d.need, sizeof(long long)) == cudaSuccess &&
              cudaMalloc(&bt->words, sizeof(unsigned long long) * 16 * sdtw::NWORDS) == cudaSuccess &&
              cudaMalloc(&bt->z_dem, nb) == cudaSuccess &&
              cudaMalloc(&bt->z, nb) == cudaSuccess && cudaMalloc(&bt->h0, nb) == cudaSuccess &&
              cudaMalloc(&d.h, nb) == cudaSuccess && cudaMalloc(&d.zh, nb) == cudaSuccess &&
              cudaMalloc(&d.f, (size_t)d.N * sizeof(sdtw::D4)) == cudaSuccess &&
              cudaMalloc(&d.list[0], (size_t)d.N * sizeof(sdtw::Entry)) == cudaSuccess &&
              cudaMalloc(&d.list[1], (size_t)d.N * sizeof(sdtw::Entry)) == cudaSuccess;
    if (ok) {
        d.z = bt->z;
        cudaMemset(d.counts, 0, sizeof(int) * (steps + 1));
        cudaMemcpy((void*)d.offs, bt->offs.data(), sizeof(long long) * (B + 1), cudaMemcpyHostToDevice);
        cudaMemset(bt->z_dem, 0, nb);
        cudaMemset(bt->h0, 0, nb);
        size_t src = 0;
        for (int b = 0; b < B; b++) {
            const size_t n = (size_t)bt->inst[b].rows * bt->inst[b].cols;
            cudaMemcpy(bt->z_dem + bt->offs[b], z_dem_host + src, n * sizeof(double), cudaMemcpyHostToDevice);
            cudaMemcpy(bt->h0 + bt->offs[b], h0_host + src, n * sizeof(double), cudaMemcpyHostToDevice);
            src += n;
        }
        ok = sdtb::tiles_for(*bt) && cudaGetLastError() == cudaSuccess;
    }
    if (!ok) {
        (void)cudaGetLastError();
        fprintf(stderr, "opencal-gb300: cal_sdt_batch_create: out of device memory\n");
        sdtb::destroy(bt);
        return nullptr;
    }
    return bt;
}

extern "C" void cal_sdt_batch_destroy(void* handle)
{
    if (handle)
        sdtb::destroy((Batch*)handle);
}

/* padded cell count and the B + 1 instance offsets of the device layout */
extern "C" long long cal_sdt_batch_cells(void* handle, long long* offsets)
{
    Batch* bt = (Batch*)handle;
    if (offsets)
        memcpy(offsets, bt->offs.data(), sizeof(long long) * (bt->B + 1));
    return bt->d.N;
}

extern "C" void* cal_sdt_batch_stream(void* handle) { return ((Batch*)handle)->st; }
extern "C" int cal_sdt_batch_shape(void* handle) { return ((Batch*)handle)->shape; }

/* replace the per-instance parameters (host array of 2B doubles: p_r, p_eps) */
extern "C" int cal_sdt_batch_set_params(void* handle, const double* params)
{
    Batch* bt = (Batch*)handle;
    for (int b = 0; b < bt->B; b++) {
        bt->inst[b].r = params[2 * b];
        bt->inst[b].eps = params[2 * b + 1];
        memcpy(&bt->inst[b].eps_bits, &bt->inst[b].eps, sizeof(double));
    }
    cudaStreamSynchronize(bt->st);
    return (int)cudaMemcpy((void*)bt->d.inst, bt->inst.data(), sizeof(sdtb::Inst) * bt->B, cudaMemcpyHostToDevice);
}

/* Forward rollout of every instance (`steps` steps); h_T copied into hT (a
 * device array in the padded layout, or NULL).  Asynchronous on the
 * ensemble's stream; hT is NaN when a grid barrier gave up. */
extern "C" int cal_sdt_batch_forward(void* handle, double* hT)
{
    Batch* bt = (Batch*)handle;
    if (!bt->d.tiles)
        return (int)cudaErrorMemoryAllocation;
    sdtb::forward(*bt, bt->steps, false, false, false);
    if (hT)
        sdtw::k_out<<<sdtw::dense_blocks(bt->d.N), sdtw::T, 0, bt->st>>>(bt->d.h, hT, bt->d.N, bt->words);
    return (int)cudaGetLastError();
}

/* Tiles updated by each step of the last rollout: steps + 1 counts, the last
 * 0 (no step).  Synchronises; an error when the rollout gave up at a grid
 * barrier. */
extern "C" int cal_sdt_batch_active_tiles(void* handle, int* out)
{
    Batch* bt = (Batch*)handle;
    cudaStreamSynchronize(bt->st);
    unsigned long long gave_up = 0;
    if (bt->flows_clear)
        cudaMemcpy(&gave_up, bt->words + 16 * 7, sizeof(gave_up), cudaMemcpyDeviceToHost);
    if (gave_up)
        return (int)cudaErrorUnknown;
    return (int)cudaMemcpy(out, bt->d.counts, sizeof(int) * (bt->steps + 1), cudaMemcpyDeviceToHost);
}

namespace sdtb {

/* The whole loss + gradient evaluation queued on the ensemble's stream:
 * forward with the tape or with checkpoints, loss, the reverse sweep (segment
 * by segment where the rollout is not on the tape), dL/dh0, and the losses,
 * gradients and the tape entries needed copied into the pinned h_out.
 * Nothing in it waits for the host, so it can be recorded. */
static void queue_loss_grad(Batch& bt, const double* target, double* g_h0, bool recorded)
{
    Dev& d = bt.d;
    Adj a = bt.a;
    if (!g_h0)
        a.mu = nullptr; /* nothing reads it */
    const size_t nb = (size_t)d.N * sizeof(double), offs = sizeof(long long) * (bt.B + 1);
    cudaStream_t st = bt.st;
    forward(bt, bt.steps, !bt.run_full, bt.run_full, recorded);
    cudaMemsetAsync(bt.loss, 0, bt.B * sizeof(double), st);
    cudaMemsetAsync(a.stamp, 0xff, sizeof(int) * (size_t)d.N, st);
    sdtw::k_loss<<<sdtw::dense_blocks(d.N), T, offs, st>>>(d, a, target, bt.loss);
    if (bt.run_full) {
        queue_adjoint(bt, a, 0, bt.steps, recorded);
    } else {
        for (int s = bt.nseg - 1; s >= 0; s--) {
            const int t0 = s * bt.K, t1 = std::min(t0 + bt.K, bt.steps);
            if (t1 <= t0)
                continue;
            cudaMemcpyAsync(d.h, bt.ckpt + (size_t)s * d.N, nb, cudaMemcpyDeviceToDevice, st);
            cudaMemsetAsync(d.nlist + t0, 0, sizeof(int) * (t1 - t0 + 1), st);
            cudaMemsetAsync(d.counts + t0, 0, sizeof(int) * (t1 - t0), st);
            cudaMemsetAsync(d.toff + t0, 0, sizeof(long long), st);
            sdtw::k_relist<<<sdtw::dense_blocks(d.N), T, offs, st>>>(d, t0);
            queue_steps(bt, t0, t1, bt.steps + 1, true, recorded);
            sdtw::k_clear_flows<<<sdtw::BLOCKS, T, 0, st>>>(d, t1 - 1);
            queue_adjoint(bt, a, t0, t1, recorded);
        }
    }
    if (g_h0)
        sdtw::k_final_grad<<<sdtw::dense_blocks(d.N), T, 0, st>>>(bt.h0, a.lam, a.mu, g_h0, d.N);
    sdtw::queue_grad(d, a, st);
    cudaMemcpyAsync(bt.h_out, bt.loss, bt.B * sizeof(double), cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(bt.h_out + bt.B, a.grad, 2 * bt.B * sizeof(double), cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(bt.h_out + 3 * bt.B, d.need, sizeof(long long), cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(bt.h_out + 3 * bt.B + 1, bt.words + 16 * 7, sizeof(long long), cudaMemcpyDeviceToHost, st);
}

/* arrays that only the gradient needs, allocated by the first call that
 * wants them */
static bool adjoint_arrays(Batch& bt, bool want_mu)
{
    Adj& a = bt.a;
    const size_t n = (size_t)bt.d.N;
    auto need = [](auto** p, size_t count) {
        if (*p)
            return true;
        if (cudaMalloc(p, count * sizeof(**p)) == cudaSuccess)
            return true;
        (void)cudaGetLastError();
        *p = nullptr;
        return false;
    };
    if (!need(&a.w, 2 * n)) /* and the cells' sums */
        return false;
    a.sums = a.w + n;
    return need(&a.lam, n) && need(&a.stamp, n) && need(&a.g, n) && need(&a.grad, 2 * (size_t)bt.B) &&
           need(&a.part, 4 * (size_t)bt.B * sdtw::PARTS) && need(&bt.loss, (size_t)bt.B) &&
           (!want_mu || need(&a.mu, n)) &&
           (bt.run_full || bt.steps == 0 || need(&bt.ckpt, n * bt.nseg));
}

/* One evaluation: as one launch of the recorded graph (recorded again when
 * the target, the dL/dh0 buffer or what the tape holds changed, or when the
 * tiles or the tape were allocated again), or launch by launch.  When the
 * tape was too small the evaluation is discarded, the tape grown to the size
 * the device reported (plus a quarter) and the evaluation run again; a first
 * call, without a tape, runs the forward alone to learn that size.  In the memory-chosen mode a
 * whole-rollout tape that would not fit switches the ensemble to segments.
 * Segments of more than 32 steps (rollouts over 1024 steps) are not
 * recorded: six launches a step would make a graph that costs more to
 * instantiate than the cooperative launches to run. */
static int loss_grad(Batch& bt, const double* target, double* loss_out, double* grad_out, double* g_h0)
{
    Dev& d = bt.d;
    cudaStream_t st = bt.st;
    if (!d.tiles || (!bt.h_out && cudaMallocHost(&bt.h_out, sizeof(double) * (3 * bt.B + 2)) != cudaSuccess))
        return (int)cudaErrorMemoryAllocation;
    for (int attempt = 0; attempt < 5; attempt++) {
        if (!adjoint_arrays(bt, g_h0 != nullptr)) {
            fprintf(stderr, "opencal-gb300: cal_sdt_batch_loss_grad: out of device memory\n");
            return (int)cudaErrorMemoryAllocation;
        }
        const bool measure = bt.run_full && d.cap == 0 && bt.steps > 0;
        if (measure) {
            forward(bt, bt.steps, false, true, false);
            cudaMemcpyAsync(bt.h_out + 3 * bt.B, d.need, sizeof(long long), cudaMemcpyDeviceToHost, st);
            cudaMemcpyAsync(bt.h_out + 3 * bt.B + 1, bt.words + 16 * 7, sizeof(long long), cudaMemcpyDeviceToHost, st);
        } else if (bt.use_graph && bt.steps > 0 && (bt.run_full || bt.K <= 32)) {
            if (!bt.gexec || bt.g_target != target || bt.g_gh0 != g_h0 || bt.g_full != bt.run_full) {
                drop_graph(bt);
                cudaGraph_t graph = nullptr;
                first_state(bt); /* the recording must not hold the one-off clear */
                if (cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) != cudaSuccess)
                    return (int)cudaGetLastError();
                queue_loss_grad(bt, target, g_h0, true);
                cudaError_t e = cudaStreamEndCapture(st, &graph);
                if (e != cudaSuccess || !graph) {
                    (void)cudaGetLastError();
                    return (int)(e != cudaSuccess ? e : cudaErrorUnknown);
                }
                e = cudaGraphInstantiate(&bt.gexec, graph, 0);
                size_t nodes = 0;
                cudaGraphGetNodes(graph, nullptr, &nodes);
                bt.graph_nodes = (long long)nodes;
                cudaGraphDestroy(graph);
                if (e != cudaSuccess)
                    return (int)e;
                bt.g_target = target;
                bt.g_gh0 = g_h0;
                bt.g_full = bt.run_full;
            }
            if (cudaGraphLaunch(bt.gexec, st) != cudaSuccess)
                return (int)cudaGetLastError();
            bt.graph_launches++;
        } else {
            queue_loss_grad(bt, target, g_h0, false);
        }
        if (cudaStreamSynchronize(st) != cudaSuccess) {
            bt.flows_clear = false;
            return (int)cudaGetLastError();
        }
        long long need = 0, gave_up = 0;
        memcpy(&need, bt.h_out + 3 * bt.B, sizeof(need));
        memcpy(&gave_up, bt.h_out + 3 * bt.B + 1, sizeof(gave_up));
        if (gave_up) /* a grid barrier did (the next run clears what it left) */
            return (int)cudaErrorUnknown;
        bt.last_need = need;
        if (!measure && need <= d.cap) {
            if (loss_out)
                memcpy(loss_out, bt.h_out, bt.B * sizeof(double));
            if (grad_out)
                for (int b = 0; b < bt.B; b++) {
                    grad_out[2 * b] = bt.h_out[bt.B + b];
                    grad_out[2 * b + 1] = bt.h_out[2 * bt.B + b];
                }
            return 0;
        }
        const long long cap = std::max<long long>(1, need + need / 4);
        if (bt.run_full && bt.tape_mode < 0) {
            size_t free_b = 0, total_b = 0;
            cudaMemGetInfo(&free_b, &total_b);
            if ((size_t)cap * sdtw::TAPE_BYTES > (free_b + (size_t)d.cap * sdtw::TAPE_BYTES) / 2) {
                bt.run_full = false; /* the segments' tape is about sqrt(T) times smaller */
                continue;
            }
        }
        if (!grow_tape(bt, cap)) {
            if (bt.run_full && bt.tape_mode < 0) {
                bt.run_full = false;
                continue;
            }
            fprintf(stderr, "opencal-gb300: cal_sdt_batch_loss_grad: out of device memory for the tape\n");
            return (int)cudaErrorMemoryAllocation;
        }
    }
    return (int)cudaErrorUnknown;
}

} // namespace sdtb

/* Loss L_b = sum over instance b of (h_T - target)^2 and its gradients:
 * forward, then the adjoint.  target: device array in the padded layout.
 * loss_out[B], grad_out[2B] (dL/dp_r, dL/dp_eps of each instance,
 * interleaved): host arrays; g_h0: device array for dL/dh0 (padded layout),
 * or NULL.  Synchronises. */
extern "C" int cal_sdt_batch_loss_grad(void* handle, const double* target, double* loss_out, double* grad_out,
                                       double* g_h0)
{
    const int rc = sdtb::loss_grad(*(Batch*)handle, target, loss_out, grad_out, g_h0);
    return rc ? rc : (int)cudaGetLastError();
}

/* Pick the fastest tile shape for this ensemble: a forward of `probe_steps`
 * steps per candidate (0: 32x16, 1: 64x16, 2: 64x32, 4: 32x8, the shape until
 * another is chosen), timed with CUDA events after one untimed probe.  (The
 * recorded evaluation launches other kernels; they rank the shapes alike:
 * 100 steps of 64 instances, ms, cooperative 2.17 / 2.65 / 3.33 / 2.11,
 * recorded 2.09 / 2.56 / 3.32 / 2.01.)  Writes the milliseconds to ms[0..2]
 * and ms[4] (ms[3] = 0) and returns the chosen shape, or -1 on a CUDA error.
 * Shape 3 (16x8) is selected by cal_sdt_batch_set_shape. */
extern "C" int cal_sdt_batch_autotune(void* handle, int probe_steps, float* ms)
{
    Batch* bt = (Batch*)handle;
    if (probe_steps > bt->steps)
        probe_steps = bt->steps;
    int best = bt->shape;
    float best_ms = 1e30f;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    for (int s = 0; s < sdtb::NSHAPES; s++)
        if (ms)
            ms[s] = 0.f;
    for (int s : {0, 1, 2, 4}) {
        bt->shape = s;
        if (!sdtb::tiles_for(*bt)) {
            best = -1;
            break;
        }
        sdtb::forward(*bt, probe_steps, false, false, false);
        cudaEventRecord(e0, bt->st);
        sdtb::forward(*bt, probe_steps, false, false, false);
        cudaEventRecord(e1, bt->st);
        cudaEventSynchronize(e1);
        float t = 0.f;
        cudaEventElapsedTime(&t, e0, e1);
        if (ms)
            ms[s] = t;
        if (t < best_ms) {
            best_ms = t;
            best = s;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (best < 0)
        return -1;
    bt->shape = best;
    if (!sdtb::tiles_for(*bt))
        return -1;
    return cudaGetLastError() == cudaSuccess ? best : -1;
}

/* set the tile shape (0: 32x16, 1: 64x16, 2: 64x32, 3: 16x8, 4: 32x8); 0 on
 * success */
extern "C" int cal_sdt_batch_set_shape(void* handle, int shape)
{
    Batch* bt = (Batch*)handle;
    if (shape < 0 || shape >= sdtb::NSHAPES)
        return 1;
    bt->shape = shape;
    return sdtb::tiles_for(*bt) ? 0 : 2;
}

/* 1 (default): cal_sdt_batch_loss_grad runs as one launch of a recorded
 * graph; 0: launch by launch */
extern "C" int cal_sdt_batch_set_graph(void* handle, int on)
{
    Batch* bt = (Batch*)handle;
    bt->use_graph = on != 0;
    return 0;
}

/* What the adjoint's tape holds: -1 (default) the whole rollout while it
 * fits in half of the free device memory, else sqrt(T) segments recomputed
 * from checkpoints; 0 always segments; 1 always the whole rollout.  1 on a
 * bad mode. */
extern "C" int cal_sdt_batch_set_tape(void* handle, int mode)
{
    Batch* bt = (Batch*)handle;
    if (mode < -1 || mode > 1)
        return 1;
    bt->tape_mode = mode;
    bt->run_full = mode != 0;
    return 0;
}

/* info[0] = 1 when the last evaluation taped the whole rollout (0:
 * segments), info[1] = the tape's capacity in bytes, info[2] = the bytes of
 * tape the last evaluation needed */
extern "C" int cal_sdt_batch_tape_info(void* handle, long long* info)
{
    Batch* bt = (Batch*)handle;
    info[0] = bt->run_full ? 1 : 0;
    info[1] = bt->d.cap * (long long)sdtw::TAPE_BYTES;
    info[2] = bt->last_need * (long long)sdtw::TAPE_BYTES;
    return 0;
}

/* graph launches made by cal_sdt_batch_loss_grad so far and the nodes of
 * the recorded evaluation (kernels and copies) */
extern "C" int cal_sdt_batch_graph_stats(void* handle, long long* launches, long long* nodes)
{
    Batch* bt = (Batch*)handle;
    if (launches)
        *launches = bt->graph_launches;
    if (nodes)
        *nodes = bt->graph_nodes;
    return 0;
}
