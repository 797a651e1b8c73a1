/*
 * sciddicaT_adjoint.cu -- reverse-mode adjoint of a SCIDDICA-T rollout
 * (plain mode) of one grid, for calibration.
 *
 * Forward model (one step, every wet cell c, h_c > epsilon):
 *   m = h_c - eps, u_0 = z_c + eps, u_n = z_nb(n) + h_nb(n) (n = 1..4),
 *   A_c = cells left by the minimisation, k_c = |A_c|,
 *   avg_c = (m + sum_{n in A_c} u_n) / k_c,
 *   f_{c,n} = r (avg_c - u_n) for n in A_c, n >= 1, else 0;
 *   h'_x = h_x + sum_n (f_{nb(n), opp(n)} - f_{x,n}).
 * The elimination sets A_c and the wet set are discrete: they are the
 * forward's, frozen, so the derivative is that of the piecewise-linear map
 * the forward actually evaluated.
 *
 * Adjoint of one step, with lambda' = dL/dh_{t+1}:
 *   lf_{c,n} = lambda'_nb(n) - lambda'_c       (0 for absent neighbours'
 *                                               lambda' on a flat grid)
 *   S_c = sum_{n in A_c, n>=1} lf_{c,n},  g_c = (r / k_c) S_c
 *   w_{c,m} = g_c - r lf_{c,m} for m in A_c, m >= 1, else 0
 *   lambda_t(x) = lambda'_x + g_x + sum_d w_{nb(d), opp(d)}
 *   lambda_z(x) += [0 in A_x] g_x + sum_d w_{nb(d), opp(d)}
 *   dL/dr   += sum_c sum_{n in A_c, n>=1} lf_{c,n} (avg_c - u_n)
 *   dL/deps += sum_c S_c r ([0 in A_c] - 1) / k_c
 * and the initialisation z = z_dem - h0 where h0 > 0 adds
 *   dL/dh0 = lambda_0 - [h0 > 0] lambda_z.
 *
 * The steps and their adjoint are the wet-cell list's (sciddicaT_wet.cuh)
 * with one instance, in one cooperative launch each way.  The forward tapes
 * the rollout into a tape that, where memory matters, takes no more of it than
 * checkpoints every K = ceil(sqrt(T)) steps and the states of a segment
 * between two would (kept_tape: a program may hold many rollouts between
 * their forwards and backwards).  The backward first learns what the tape
 * needed.  One that was too small holds the last steps; when running the
 * steps before them again, as often as it takes, costs no more than one
 * forward, the sweep goes on so (1024 x 1024 x 2000 with 0.6 of the tape it
 * needs: 45 -> 54 ms, with a forward into a larger one 65).  Else the forward
 * runs again with a tape that fits, given back after the sweep, or, when that
 * would take more than half of the free device memory, with h stored every K
 * steps, and the sweep then recomputes and tapes one segment at a time.
 */
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "sciddicaT_wet.cuh"

namespace sdtadj {

using sdtw::Adj;
using sdtw::Dev;
using sdtw::Inst;
using sdtw::T;

/* the unit of the update and the gather, as the ensembles' */
constexpr int LW = 5, LH = 3;

struct Work {
    int rows = 0, cols = 0, steps = 0, toroidal = 0, K = 0, nseg = 0;
    double r = 0, eps = 0;
    Dev d = {};
    Adj a = {};
    Inst* inst = nullptr;
    long long* offs = nullptr;
    double *z_dem = nullptr, *z = nullptr, *h0 = nullptr;
    double* ckpt = nullptr; /* segments only */
    char* slab = nullptr;   /* every array of fixed size, one allocation */
    char* tape = nullptr;
    unsigned long long* words = nullptr; /* of the cooperative launches */
    bool want_tape = true, want_segments = false;
    /* the flagged tiles of all steps, which a whole tape needs, would take
     * more than the checkpoints (over a million steps, or 270,000 on a grid
     * of few cells): room for one segment's */
    bool only_segments = false;
    bool flows_clear = false;
    long long kept = 0;  /* entries of the tape kept after a backward */
    long long limit = 0; /* on those (0: none) */
    /* counts the changes of tape and checkpoints; need[1] holds the one that
     * the last forward to run left its record in (a captured forward may run
     * after they were changed) */
    long long record = 0;
};

/* need[1] of a forward that cannot be reversed as it is: captured, or run in
 * part (need[0] is then the part's) */
constexpr long long NOT_TAPED = -1, IN_PART = -2;

__global__ void k_start(long long* toff, long long* tpos, long long* need, long long record)
{
    toff[0] = 0;
    tpos[0] = 0;
    need[0] = 0;
    need[1] = record;
}

__global__ void k_instance(Inst I, long long n, Inst* inst, long long* offs)
{
    inst[0] = I;
    offs[0] = 0;
    offs[1] = n;
}

/* successive arrays of a slab, 256-byte aligned; with base NULL only sizes */
struct Carve {
    char* base;
    size_t at = 0;
    template <typename E>
    void take(E** p, size_t count)
    {
        *p = (E*)(base + at);
        at += (count * sizeof(E) + 255) & ~(size_t)255;
    }
};

static size_t carve(Work& W, char* base)
{
    const size_t n = (size_t)W.rows * W.cols, steps = (size_t)W.steps + 1;
    Dev& d = W.d;
    Adj& a = W.a;
    Carve c{base};
    c.take(&W.inst, 1);
    c.take(&W.offs, 2);
    c.take((int**)&d.tile_inst, d.ntiles);
    c.take(&W.z_dem, n);
    c.take(&W.z, n);
    c.take(&W.h0, n);
    c.take(&d.h, n);
    c.take(&d.zh, n);
    c.take(&d.f, n);
    c.take(&d.list[0], n);
    c.take(&d.list[1], n);
    c.take(&d.nlist, steps);
    c.take(&d.counts, steps);
    c.take(&d.tiles, (size_t)d.ntiles * (W.only_segments ? W.K : steps));
    c.take(&d.stamps, d.ntiles);
    c.take(&d.toff, steps);
    c.take(&d.tpos, steps);
    c.take(&d.need, 2);
    c.take(&W.words, 16 * sdtw::NWORDS);
    c.take(&a.lam, n);
    c.take(&a.mu, n);
    c.take(&a.stamp, n);
    c.take(&a.w, n);
    c.take(&a.g, n);
    c.take(&a.sums, n);
    c.take(&a.part, 4 * sdtw::PARTS);
    c.take(&a.grad, 2);
    d.inst = W.inst;
    d.offs = W.offs;
    d.z = W.z;
    return c.at;
}

/* d with the flagged tiles of the steps from t0 on at the start of d.tiles */
static Dev from_step(const Dev& d, int t0)
{
    Dev s = d;
    s.tiles = (int*)((char*)d.tiles - sizeof(int) * (size_t)t0 * d.ntiles);
    return s;
}

static void drop_tape(Work& W)
{
    cudaFree(W.tape);
    W.tape = nullptr;
    W.d.cap = 0;
    if (!W.ckpt) /* with checkpoints it holds one segment at a time */
        W.record++;
}

/* a tape of `entries` entries, instead of the one there was */
static bool make_tape(Work& W, long long entries)
{
    Dev& d = W.d;
    drop_tape(W);
    for (int pass = 0; pass < 2; pass++) {
        Carve c{W.tape};
        c.take(&d.t_diff, (size_t)entries);
        c.take(&d.t_entry, (size_t)entries);
        c.take(&d.t_elim, (size_t)entries);
        if (pass == 0 && cudaMalloc(&W.tape, c.at) != cudaSuccess) {
            (void)cudaGetLastError();
            W.tape = nullptr;
            return false;
        }
    }
    d.cap = entries;
    return true;
}

/* Entries of the tape a rollout may keep between its forward and its
 * backward: no more bytes than sqrt(T) checkpointing keeps (nseg checkpoints,
 * K + 1 states) or than a 128th of the free memory, and no more than a
 * sixteenth of the cells wet on average need.  (512 x 480 x 400: 81 MB, 2 GB,
 * 268 MB; of 40 flows two fifths of the first is the median need and 1.6 times
 * it the largest.) */
static long long kept_tape(const Work& W)
{
    const long long n = W.d.N;
    size_t free_b = 0, total_b = 0;
    cudaMemGetInfo(&free_b, &total_b);
    const long long states = (long long)(W.nseg + W.K + 1) * n * (long long)sizeof(double);
    const long long bytes = std::max(states, (long long)(free_b / 128));
    const long long entries = std::min(std::min(bytes, (long long)free_b / 8) / (long long)sdtw::TAPE_BYTES,
                                       (n / 16 + 1024) * W.steps);
    return std::max<long long>(1, W.limit > 0 ? std::min(entries, W.limit) : entries);
}

static bool make_checkpoints(Work& W)
{
    if (cudaMalloc(&W.ckpt, (size_t)W.nseg * W.d.N * sizeof(double)) != cudaSuccess) {
        (void)cudaGetLastError();
        W.ckpt = nullptr;
        return false;
    }
    W.record++;
    return true;
}

/* The first `steps` steps of the rollout from h0 and z_dem, queued: taped, or
 * with checkpoints (keep).  A captured one is not taped: its nodes would keep the address of a tape
 * that a backward may allocate again. */
static void queue_forward(Work& W, int steps, bool keep, cudaStream_t st)
{
    Dev d = W.d;
    const size_t n = (size_t)d.N;
    const bool captured = sdtw::capturing(st);
    if (captured)
        d.cap = 0;
    k_start<<<1, 1, 0, st>>>(d.toff, d.tpos, d.need,
                             steps < W.steps ? IN_PART
                                             : ((captured || W.only_segments) && !keep ? NOT_TAPED : W.record));
    cudaMemsetAsync(d.stamps, 0, sizeof(int) * d.ntiles, st);
    cudaMemsetAsync(d.counts, 0, sizeof(int) * (W.steps + 1), st);
    cudaMemsetAsync(d.nlist, 0, sizeof(int) * (W.steps + 1), st);
    const size_t words = sizeof(unsigned long long) * 16 * sdtw::NWORDS;
    if (!W.flows_clear) { /* before the first run: no outflows, and no run that gave up */
        cudaMemsetAsync(d.f, 0, n * sizeof(sdtw::D4), st);
        cudaMemsetAsync(W.words, 0, words, st);
        W.flows_clear = !captured; /* what is captured has not run yet */
    }
    sdtw::k_init<<<sdtw::dense_blocks(d.N), T, 2 * sizeof(long long), st>>>(d, W.z_dem, W.h0, W.z, W.words);
    if (steps == W.steps) /* else a part of a sweep that may have given up already */
        cudaMemsetAsync(W.words, 0, words, st);
    const bool parts = keep || W.only_segments;
    const int per = parts ? W.K : std::max(1, steps);
    for (int t = 0; t < steps; t += per) {
        if (keep)
            cudaMemcpyAsync(W.ckpt + (size_t)(t / per) * n, d.h, n * sizeof(double), cudaMemcpyDeviceToDevice, st);
        Dev part = parts ? from_step(d, t) : d;
        sdtw::launch_steps(part, t, std::min(t + per, steps), 1, !parts, W.words, st);
    }
    if (steps > 0)
        sdtw::k_clear_flows<<<sdtw::BLOCKS, T, 0, st>>>(d, steps - 1);
}

/* need[0]: the largest tape any step sequence asked for since the last
 * forward; need[1]: that forward's record */
static cudaError_t tape_need(Work& W, long long need[2], cudaStream_t st)
{
    cudaMemcpyAsync(need, W.d.need, 2 * sizeof(*need), cudaMemcpyDeviceToHost, st);
    return cudaStreamSynchronize(st);
}

/* The stretches [c, t1) of steps, last first, that a tape too small for all
 * holds one at a time after a forward to t1; none when a step does not fit at
 * all or the forwards would take more than `steps` steps together. */
static std::vector<std::pair<int, int>> stretches(const Work& W, const std::vector<long long>& toff)
{
    std::vector<std::pair<int, int>> out;
    std::vector<long long> base(W.steps);
    long long pos = 0, again = 0;
    for (int t = 0; t < W.steps; t++) {
        const int n = (int)(toff[t + 1] - toff[t]);
        base[t] = sdtw::tape_slot(W.d.cap, true, pos, n);
        if (base[t] < 0)
            return out;
        pos = sdtw::tape_next(true, pos, base[t], n);
    }
    for (int t1 = W.steps, c; t1 > 0; t1 = c) {
        long long end = 0; /* of what lies at the start of the tape since it began again */
        int lap = 0;
        for (c = t1; c > 0; c--) {
            const long long from = base[c - 1], to = from + (toff[c] - toff[c - 1]);
            if (c < t1 && to > base[c]) /* step c began at 0 again */
                lap++;
            if (lap == 2 || (lap == 1 && from < end))
                break;
            if (lap == 0)
                end = std::max(end, to);
        }
        out.push_back(std::make_pair(c, t1));
        again += c;
        if (again > W.steps) {
            out.clear();
            return out;
        }
    }
    return out;
}

static void queue_seed(Work& W, const double* gT, cudaStream_t st)
{
    const size_t b = (size_t)W.d.N * sizeof(double);
    cudaMemcpyAsync(W.a.lam, gT, b, cudaMemcpyDeviceToDevice, st);
    cudaMemcpyAsync(W.a.mu, gT, b, cudaMemcpyDeviceToDevice, st);
    cudaMemsetAsync(W.a.stamp, 0xff, sizeof(int) * (size_t)W.d.N, st);
}

/* the reverse sweep recomputing segments from the checkpoints */
static void queue_segments(Work& W, cudaStream_t st)
{
    const size_t n = (size_t)W.d.N;
    cudaMemsetAsync(W.d.need, 0, sizeof(long long), st);
    for (int s = W.nseg - 1; s >= 0; s--) {
        const int t0 = s * W.K, t1 = std::min(t0 + W.K, W.steps);
        Dev d = from_step(W.d, t0);
        d.tpos = nullptr;
        cudaMemcpyAsync(d.h, W.ckpt + (size_t)s * n, n * sizeof(double), cudaMemcpyDeviceToDevice, st);
        cudaMemsetAsync(d.nlist + t0, 0, sizeof(int) * (t1 - t0 + 1), st);
        cudaMemsetAsync(d.counts + t0, 0, sizeof(int) * (t1 - t0), st);
        cudaMemsetAsync(d.toff + t0, 0, sizeof(long long), st);
        cudaMemsetAsync(d.stamps, 0, sizeof(int) * d.ntiles, st);
        sdtw::k_relist<<<sdtw::dense_blocks(d.N), T, 2 * sizeof(long long), st>>>(d, t0);
        sdtw::launch_steps(d, t0, t1, 1, true, W.words, st);
        sdtw::k_clear_flows<<<sdtw::BLOCKS, T, 0, st>>>(d, t1 - 1);
        sdtw::launch_sweep(d, W.a, t0, t1, W.words, st);
    }
}

} // namespace sdtadj

using sdtadj::Work;

/* Workspace for rollouts of `steps` steps on a rows x cols grid. */
extern "C" void* cal_sdt_adj_create(int rows, int cols, int steps, int toroidal)
{
    Work* W = new Work();
    W->rows = rows;
    W->cols = cols;
    W->steps = steps > 0 ? steps : 0;
    W->toroidal = toroidal;
    W->K = (int)ceil(sqrt((double)(steps > 0 ? steps : 1)));
    W->nseg = (W->steps + W->K - 1) / W->K;
    sdtw::Dev& d = W->d;
    d.B = 1;
    d.N = (long long)rows * cols;
    d.lw = sdtadj::LW;
    d.lh = sdtadj::LH;
    const int tx = (cols + (1 << d.lw) - 1) >> d.lw, ty = (rows + (1 << d.lh) - 1) >> d.lh;
    d.ntiles = tx * ty;
    const double lists = (double)d.ntiles * sizeof(int) * W->steps;
    W->only_segments = lists > 1 << 20 && lists > (double)(W->nseg + W->K + 1) * d.N * sizeof(double);
    const size_t bytes = sdtadj::carve(*W, nullptr);
    if (rows <= 0 || cols <= 0 || d.N >= 0x7fffffffLL || cudaMalloc(&W->slab, bytes) != cudaSuccess) {
        (void)cudaGetLastError();
        fprintf(stderr, "opencal-gb300: cal_sdt_adj_create: out of device memory\n");
        delete W;
        return nullptr;
    }
    sdtadj::carve(*W, W->slab);
    return W;
}

extern "C" void cal_sdt_adj_destroy(void* handle)
{
    Work* W = (Work*)handle;
    if (!W)
        return;
    cudaFree(W->slab);
    cudaFree(W->tape);
    cudaFree(W->ckpt);
    delete W;
}

/* 0: the next forwards leave no tape (no backward is expected; one that
 * comes all the same runs the forward again); 1 (default): they do; 2: they
 * leave checkpoints, and backwards recompute and tape a segment at a time (a
 * workspace that has checkpoints stays with them).  1 on a bad mode. */
extern "C" int cal_sdt_adj_set_tape(void* handle, int mode)
{
    Work* W = (Work*)handle;
    if (mode < 0 || mode > 2)
        return 1;
    W->want_tape = mode == 1;
    W->want_segments = mode == 2;
    return 0;
}

/* The most entries of tape (41 bytes each) that the workspace keeps between a
 * forward and its backward; 0 (default): as the memory allows.  For the
 * tapes allocated from now on. */
extern "C" int cal_sdt_adj_set_tape_limit(void* handle, long long entries)
{
    if (entries < 0)
        return 1;
    ((Work*)handle)->limit = entries;
    return 0;
}

/* Forward rollout on device buffers: init (z = z_dem - h0 where h0 > 0),
 * `steps` steps, h_T into hT; the tape kept for the backward.  May be
 * captured into a graph (nothing is allocated then: without a tape from an
 * earlier forward the backward runs the forward again). */
extern "C" int cal_sdt_adj_forward(void* handle, const double* z_dem, const double* h0, double p_r, double p_eps,
                                   double* hT, void* stream)
{
    Work* W = (Work*)handle;
    cudaStream_t st = (cudaStream_t)stream;
    sdtw::Dev& d = W->d;
    W->r = p_r;
    W->eps = p_eps;
    const size_t b = (size_t)d.N * sizeof(double);
    if ((W->want_segments || W->only_segments) && !W->ckpt && W->steps > 0 && !sdtw::capturing(st) &&
        !sdtadj::make_checkpoints(*W))
        return (int)cudaErrorMemoryAllocation;
    if (W->want_tape && !W->ckpt && !d.cap && W->steps > 0 && !sdtw::capturing(st)) {
        W->kept = sdtadj::kept_tape(*W);
        sdtadj::make_tape(*W, W->kept);
    }
    sdtadj::Inst I;
    memset(&I, 0, sizeof(I));
    I.rows = W->rows;
    I.cols = W->cols;
    I.r = p_r;
    I.eps = p_eps;
    memcpy(&I.eps_bits, &p_eps, sizeof(double));
    I.tiles_x = (W->cols + (1 << d.lw) - 1) >> d.lw;
    I.tiles_y = (W->rows + (1 << d.lh) - 1) >> d.lh;
    I.toroidal = W->toroidal;
    sdtadj::k_instance<<<1, 1, 0, st>>>(I, d.N, W->inst, W->offs);
    cudaMemsetAsync((void*)d.tile_inst, 0, sizeof(int) * d.ntiles, st);
    cudaMemcpyAsync(W->h0, h0, b, cudaMemcpyDeviceToDevice, st);
    cudaMemcpyAsync(W->z_dem, z_dem, b, cudaMemcpyDeviceToDevice, st);
    sdtadj::queue_forward(*W, W->steps, W->ckpt != nullptr, st);
    /* no step: h0 as given, -0 and all */
    sdtw::k_out<<<sdtw::dense_blocks(d.N), sdtadj::T, 0, st>>>(W->steps > 0 ? d.h : W->h0, hT, d.N, W->words);
    return (int)cudaGetLastError();
}

/* Backward: from dL/dh_T (gT) to dL/dh0 (g_h0, device) and dL/dp_r, dL/dp_eps
 * (host doubles; the call synchronises the stream). */
extern "C" int cal_sdt_adj_backward(void* handle, const double* gT, double* g_h0, double* g_r, double* g_eps,
                                    void* stream)
{
    Work* W = (Work*)handle;
    cudaStream_t st = (cudaStream_t)stream;
    sdtw::Dev& d = W->d;
    long long need[2] = {0, 0};
    cudaError_t e = sdtadj::tape_need(*W, need, st);
    if (e == cudaSuccess && need[1] == sdtadj::IN_PART) {
        sdtadj::queue_forward(*W, W->steps, W->ckpt != nullptr, st);
        e = sdtadj::tape_need(*W, need, st);
    }
    if (e != cudaSuccess)
        return (int)e;
    bool segments = W->ckpt != nullptr;
    std::vector<std::pair<int, int>> parts;
    if (!segments && !W->only_segments && need[0] > d.cap && d.cap > 0 && need[1] == W->record) {
        std::vector<long long> toff(W->steps + 1);
        cudaMemcpyAsync(toff.data(), d.toff, sizeof(long long) * toff.size(), cudaMemcpyDeviceToHost, st);
        if ((e = cudaStreamSynchronize(st)) != cudaSuccess)
            return (int)e;
        parts = sdtadj::stretches(*W, toff);
    }
    if (parts.empty()) {
        if (!segments && (W->only_segments || need[0] > d.cap)) {
            size_t free_b = 0, total_b = 0;
            cudaMemGetInfo(&free_b, &total_b);
            segments = W->only_segments ||
                       (size_t)need[0] * sdtw::TAPE_BYTES > (free_b + (size_t)d.cap * sdtw::TAPE_BYTES) / 2 ||
                       !sdtadj::make_tape(*W, need[0]);
            if (segments && !sdtadj::make_checkpoints(*W))
                return (int)cudaErrorMemoryAllocation;
        }
        if (need[1] != W->record)
            sdtadj::queue_forward(*W, W->steps, segments, st);
        parts.push_back(std::make_pair(0, W->steps));
    }
    for (int attempt = 0;; attempt++) {
        sdtadj::queue_seed(*W, gT, st);
        if (!segments) {
            for (const auto& part : parts) {
                if (part.second < W->steps)
                    sdtadj::queue_forward(*W, part.second, false, st);
                sdtw::launch_sweep(d, W->a, part.first, part.second, W->words, st);
            }
            break;
        }
        sdtadj::queue_segments(*W, st);
        if ((e = sdtadj::tape_need(*W, need, st)) != cudaSuccess)
            return (int)e;
        if (need[0] <= d.cap)
            break;
        if (attempt || !sdtadj::make_tape(*W, need[0]))
            return (int)cudaErrorMemoryAllocation;
    }
    sdtw::k_final_grad<<<sdtw::dense_blocks(d.N), sdtadj::T, 0, st>>>(W->h0, W->a.lam, W->a.mu, g_h0, d.N);
    sdtw::queue_grad(d, W->a, st);
    double res[2] = {0.0, 0.0};
    unsigned long long gave_up = 0; /* a grid barrier did */
    cudaMemcpyAsync(res, W->a.grad, sizeof(res), cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(&gave_up, W->words + 16 * 7, sizeof(gave_up), cudaMemcpyDeviceToHost, st);
    e = cudaStreamSynchronize(st);
    if (e == cudaSuccess && gave_up)
        e = cudaErrorUnknown;
    if (d.cap > W->kept)
        sdtadj::drop_tape(*W); /* another backward runs the forward again */
    if (g_r)
        *g_r = res[0];
    if (g_eps)
        *g_eps = res[1];
    return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}
