/*
 * sciddicaT_wet.cuh -- many SCIDDICA-T grids (or one) advanced together over
 * one list of their wet cells, forward and adjoint: the kernels of the
 * ensembles (sciddicaT_batch.cu) and of the single rollout
 * (sciddicaT_adjoint.cu).
 *
 * The flow covers a small part of its grids (calibration ensembles: 1 % of
 * the cells, 8 % of the cells of the tiles that hold some), and a wet cell's
 * FP64 chain is the expensive part, so the unit of work is the wet cell:
 * whatever tiles they lie in, the cells of the list spread evenly over the
 * SMs.  A step is two launches:
 *
 *   k_outflows  one thread per listed wet cell: its outflows into f (zero
 *               everywhere else), and the tiles that hold the cell or a
 *               receiver flagged once (epoch stamps) in the step's tile
 *               list.  With a tape, the cell, its elimination set and the
 *               differences average - u[n] of its kept neighbours go to
 *               entry off + k of the tape.
 *   k_update    the flagged tiles: h in place, z + h beside it, and the next
 *               list (wet cells, and ~c for a cell that dried, whose outflows
 *               the next k_outflows clears); wet cells of other tiles are
 *               carried over.
 *
 * The adjoint of a step reads the tape and lambda alone -- neither h nor z,
 * nothing is restored or minimised again -- and is two launches:
 *
 *   k_coeffs    one thread per taped wet cell: g and the four w (the
 *               formulas of sciddicaT_adjoint.cu) beside the step's stamp,
 *               and its parts of dL/dr and dL/deps;
 *   k_gather    the step's flagged tiles: lambda = lambda + g + the
 *               neighbours' w, in place, in a fixed order (results do not
 *               depend on the order of the list).
 *
 * mu = lambda - lambda_z, kept only when dL/dh0 is wanted: both take the same
 * w, so mu changes only by g at a wet cell that eliminated itself, and
 * dL/dh0 = lambda_0 - [h0 > 0] lambda_z is mu where h0 > 0, lambda elsewhere.
 *
 * Measured against the tile-by-tile step this replaced (fused tiles of 64 x
 * 16 cells with their rings, the adjoint on whole tiles after restoring
 * them), 64 instances of 128..1024 cells a side, 500 steps, us per step:
 * forward 92 -> 16 (k_outflows) + 16 (k_update); reverse 10 + 65 + 29 -> 13
 * (k_coeffs) + 10 (k_gather).  k_outflows is bound by the FP64 pipe (60 % of
 * it over the launch, the rest is its chain of loads), the others by the
 * latency of theirs.
 */
#pragma once

#include "sciddicaT_kernels.cuh"

namespace sdtw {

constexpr int T = 256;
/* 608 blocks: launch cost grows with the blocks, and four resident blocks on
 * each SM keep the FP64 pipes fed (the split step of the single grid,
 * sciddicaT.cu, measured the same) */
constexpr int BLOCKS = 152 * 4;

struct Inst {
    int rows, cols;
    long long off;
    double r, eps;
    long long eps_bits;
    int tiles_x, tiles_y, tile0, toroidal;
};

struct __align__(32) D4 {
    double v[4];
};

/* cell (packed index; ~cell: dried in the previous step) and its instance */
typedef int2 Entry;

struct Dev {
    const Inst* inst;
    const long long* offs; /* B + 1 */
    const int* tile_inst;
    int B, ntiles, lw, lh; /* tiles of 2^lw x 2^lh cells */
    long long N;
    const double* z;
    double* h;
    double* zh; /* z + h */
    D4* f;
    Entry* list[2]; /* list t in list[t & 1] */
    int* nlist;     /* per step: entries of its list */
    int* tiles;     /* per step: ntiles places for its flagged tiles */
    int* counts;    /* per step: flagged tiles */
    int* stamps;    /* per tile: epoch it was flagged in */
    Entry* t_entry; /* tape */
    unsigned char* t_elim;
    D4* t_diff;
    long long cap;   /* its entries */
    long long* toff; /* per step: entries before it; toff[t + 1] chained by step t */
    long long* tpos; /* a tape that starts again from its first entry when a step does not fit behind the one
                      * before (NULL: later steps are left out): per step, where the step before ended */
    long long* need; /* the most entries any rollout or segment asked for */
};

constexpr size_t TAPE_BYTES = sizeof(Entry) + 1 + sizeof(D4); /* per entry */

struct Adj {
    double* lam;
    double* mu; /* or NULL */
    int* stamp; /* per cell: step whose coefficients it holds; -1 before its first */
    D4* w;
    double* g;
    D4* sums;      /* per cell: its parts of dL/dr, dL/deps of all steps (Sum, Sum) */
    double* part;  /* PARTS x 4B: sums of runs of cells */
    double* grad;  /* 2B: dL/dr[0..B), dL/deps[B..2B) */
};
constexpr int PARTS = 64;

/* Kahan's sum: the value is v - c.  The parts of the cells cancel within a
 * step more than those of a cell over the steps, so that plain sums cell by
 * cell lost what sums step by step keep (errors of up to 1.2e-14 where those
 * had 9e-16). */
struct Sum {
    double v, c;
};

static __device__ __forceinline__ bool sum_finite(double v)
{
    return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000; /* on the integer pipe */
}

static __device__ __forceinline__ void sum_add(Sum& s, double x)
{
    const double y = x - s.c, t = s.v + y, c = (t - s.v) - y;
    s.c = sum_finite(t) ? c : 0.0; /* an infinite sum stays one */
    s.v = t;
}

/* a + b with the rounding of a.v + b.v kept whatever their order */
static __device__ __forceinline__ void sum_add(Sum& a, const Sum& b)
{
    const double t = a.v + b.v, z = t - a.v, c = a.c + b.c - ((a.v - (t - z)) + (b.v - z));
    a.c = sum_finite(t) ? c : 0.0;
    a.v = t;
}

/* neighbour q = 0..3 (north, west, east, south) of (i, j); false where a
 * flat grid ends */
static __device__ __forceinline__ bool nbr(const Inst& I, int i, int j, int q, int* a, int* b)
{
    *a = i + (q == 0 ? -1 : (q == 3 ? 1 : 0));
    *b = j + (q == 1 ? -1 : (q == 2 ? 1 : 0));
    if (I.toroidal) {
        *a = sdt::wrapi(*a, I.rows);
        *b = sdt::wrapi(*b, I.cols);
        return true;
    }
    return (unsigned)*a < (unsigned)I.rows && (unsigned)*b < (unsigned)I.cols;
}

/* the n tape entries of a step start here; -1: they do not fit (the
 * evaluation is repeated).  at: where the step before ended, or, when later
 * steps are left out, the entries before */
static __host__ __device__ __forceinline__ long long tape_slot(long long cap, bool again, long long at, int n)
{
    return at + n <= cap ? at : (again && n <= cap ? 0 : -1);
}
/* and the step's end */
static __host__ __device__ __forceinline__ long long tape_next(bool again, long long at, long long base, int n)
{
    return again ? (base >= 0 ? base + n : at) : at + n;
}
static __device__ __forceinline__ long long tape_base(const Dev& d, int t, int n)
{
    return tape_slot(d.cap, d.tpos != nullptr, d.tpos ? d.tpos[t] : d.toff[t], n);
}

static __device__ __forceinline__ int add(int* count, int v) { return atomicAdd(count, v); }
static __device__ __forceinline__ int add(unsigned long long* count, int v)
{
    return (int)(unsigned)atomicAdd(count, (unsigned long long)v);
}

/* the outflows of the n entries of list t, by warp `warp` of `nwarps`; base:
 * where they go on the tape, or -1; ntiles: counter of the flagged tiles */
template <typename C>
static __device__ __forceinline__ void outflows(const Dev& d, int t, int epoch, int n, long long base, C* ntiles,
                                                int warp, int nwarps)
{
    const Entry* list = d.list[t & 1];
    int* tiles = d.tiles + (size_t)t * d.ntiles;
    for (int k = warp * 32 + (threadIdx.x & 31); k < n; k += nwarps * 32) {
        const Entry e = list[k];
        if (base >= 0)
            d.t_entry[base + k] = e;
        if (e.x < 0) {
            const D4 zero = {{0.0, 0.0, 0.0, 0.0}};
            d.f[~e.x] = zero;
            continue;
        }
        const Inst I = d.inst[e.y];
        const int lc = (int)(e.x - I.off);
        const int i = lc / I.cols, j = lc - i * I.cols;
        double u[4];
        /* the cell's tile and its receivers' where they differ, and their
         * stamps, loaded here so that they arrive while the minimisation
         * runs (one after another behind it they added up to 2 us a step) */
        const int own = I.tile0 + (i >> d.lh) * I.tiles_x + (j >> d.lw);
        int rt[4], stamp[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            int a, b;
            const bool in = nbr(I, i, j, q, &a, &b);
            u[q] = in ? d.zh[I.off + (long long)a * I.cols + b] : 0.0; /* an absent neighbour: 0.0 + 0.0 */
            rt[q] = in ? I.tile0 + (a >> d.lh) * I.tiles_x + (b >> d.lw) : own;
            stamp[q] = rt[q] != own ? d.stamps[rt[q]] : epoch;
        }
        const int own_stamp = d.stamps[own];
        D4 diff, f;
        const unsigned elim = sdt::minimise(d.h[e.x], d.z[e.x] + I.eps, u[0], u[1], u[2], u[3], I.eps, diff.v);
#pragma unroll
        for (int q = 0; q < 4; q++)
            f.v[q] = (elim & (2u << q)) ? 0.0 : diff.v[q] * I.r;
        d.f[e.x] = f;
        if (base >= 0) {
            d.t_elim[base + k] = (unsigned char)elim;
            d.t_diff[base + k] = diff;
        }
        /* the tiles the update must visit: the receivers', and the own tile
         * once per distinct tile of the lanes here */
        const bool any = (elim & 0x1eu) != 0x1eu;
        auto flag = [&](int tile) {
            if (atomicExch(d.stamps + tile, epoch) != epoch)
                tiles[add(ntiles, 1)] = tile;
        };
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (!(elim & (2u << q)) && stamp[q] != epoch)
                flag(rt[q]);
        const bool mine = any && own_stamp != epoch;
        const unsigned act = __activemask();
        const unsigned peers = __match_any_sync(act, mine ? own : -1);
        if (mine && (threadIdx.x & 31) == __ffs(peers) - 1)
            flag(own);
    }
}

static __global__ void __launch_bounds__(T) k_outflows(const __grid_constant__ Dev d, int t, int epoch, int taped)
{
    const int n = d.nlist[t];
    long long base = -1;
    if (taped) {
        base = tape_base(d, t, n);
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            const long long end = d.toff[t] + n;
            d.toff[t + 1] = end;
            if (d.tpos)
                d.tpos[t + 1] = tape_next(true, d.tpos[t], base, n);
            if (*d.need < end) /* one step at a time runs */
                *d.need = end;
        }
    }
    /* chunks of 32 entries on consecutive blocks */
    outflows(d, t, epoch, n, base, d.counts + t, (threadIdx.x >> 5) * gridDim.x + blockIdx.x, gridDim.x * (T / 32));
}

/* the update works in groups of T threads: a block of the per-step kernel is
 * one group, a block of the persistent kernels GROUPS that meet at barriers
 * of their own */
template <int NG>
static __device__ __forceinline__ void group_sync()
{
    if (NG == 1)
        __syncthreads();
    else
        asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)(threadIdx.x / T)), "n"(T) : "memory");
}

/* one entry per thread at most onto the next list, one atomic per group */
template <int NG, typename C>
static __device__ __forceinline__ void group_append(bool want, Entry e, Entry* list, C* count)
{
    __shared__ int s_warps[NG][T / 32];
    int* s_warp = s_warps[threadIdx.x / T];
    const int lane = threadIdx.x & 31, warp = (threadIdx.x % T) >> 5;
    const unsigned m = __ballot_sync(0xffffffffu, want);
    if (lane == 0)
        s_warp[warp] = __popc(m);
    group_sync<NG>();
    if (warp == 0) {
        const int v = lane < T / 32 ? s_warp[lane] : 0;
        int incl = v;
#pragma unroll
        for (int o = 1; o < T / 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o)
                incl += y;
        }
        int at = 0;
        if (lane == T / 32 - 1 && incl > 0)
            at = add(count, incl);
        at = __shfl_sync(0xffffffffu, at, T / 32 - 1);
        if (lane < T / 32)
            s_warp[lane] = at + incl - v;
    }
    group_sync<NG>();
    if (want)
        list[s_warp[warp] + __popc(m & ((1u << lane) - 1u))] = e;
    group_sync<NG>(); /* s_warp is reused */
}

/* the update of step t's ntiles flagged tiles and the next list, whose
 * counter is `count`, by group `group` of `ngroups` */
template <int NG, typename C>
static __device__ __forceinline__ void update(const Dev& d, int t, int epoch, int ntiles, int nlist, C* count,
                                              int group, int ngroups)
{
    const int tid = threadIdx.x % T;
    const int* tiles = d.tiles + (size_t)t * d.ntiles;
    const Entry* cur = d.list[t & 1];
    Entry* next = d.list[(t + 1) & 1];
    const int items = ntiles + (nlist + T - 1) / T;
    for (int item = group; item < items; item += ngroups) {
        if (item >= ntiles) {
            /* wet cells of tiles that no flow touched: they stay wet */
            const int k = (item - ntiles) * T + tid;
            bool carry = false;
            Entry e = make_int2(-1, 0);
            if (k < nlist) {
                e = cur[k];
                if (e.x >= 0) {
                    const Inst& I = d.inst[e.y];
                    const int lc = (int)(e.x - I.off);
                    const int i = lc / I.cols, j = lc - i * I.cols;
                    carry = d.stamps[I.tile0 + (i >> d.lh) * I.tiles_x + (j >> d.lw)] != epoch;
                }
            }
            group_append<NG>(carry, e, next, count);
            continue;
        }
        const int tile = tiles[item];
        const int bi = d.tile_inst[tile];
        const Inst I = d.inst[bi];
        const int lt = tile - I.tile0;
        const int ty = lt / I.tiles_x, tx = lt - ty * I.tiles_x;
        for (int q0 = 0; q0 < 1 << (d.lw + d.lh); q0 += T) {
            const int q = q0 + tid;
            const int i = (ty << d.lh) + (q >> d.lw), j = (tx << d.lw) + (q & ((1 << d.lw) - 1));
            bool want = false;
            Entry e = make_int2(-1, bi);
            if (q < 1 << (d.lw + d.lh) && i < I.rows && j < I.cols) {
                const int c = (int)(I.off + (long long)i * I.cols + j);
                const double hc = d.h[c];
                const D4 o = d.f[c];
                double in[4]; /* inflow from neighbour q is its outflow towards here */
#pragma unroll
                for (int s = 0; s < 4; s++) {
                    int a, b;
                    in[s] = nbr(I, i, j, s, &a, &b) ? d.f[I.off + (long long)a * I.cols + b].v[3 - s] : 0.0;
                }
                long long any = 0;
#pragma unroll
                for (int s = 0; s < 4; s++)
                    any |= __double_as_longlong(in[s]) | __double_as_longlong(o.v[s]);
                double hn = hc;
                if (any != 0) {
#pragma unroll
                    for (int s = 0; s < 4; s++)
                        hn += in[s] - o.v[s];
                    d.h[c] = hn;
                    d.zh[c] = d.z[c] + hn;
                }
                const bool wet = sdt::is_wet(hn, I.eps_bits);
                want = wet || sdt::is_wet(hc, I.eps_bits);
                e.x = wet ? c : ~c;
            }
            group_append<NG>(want, e, next, count);
        }
    }
}

static __global__ void __launch_bounds__(T) k_update(const __grid_constant__ Dev d, int t, int epoch)
{
    update<1>(d, t, epoch, d.counts[t], d.nlist[t], d.nlist + t + 1, blockIdx.x, gridDim.x);
}

/* f back to zero after the last step run: the cells wet in step t */
static __global__ void __launch_bounds__(T) k_clear_flows(const __grid_constant__ Dev d, int t)
{
    const int n = d.nlist[t];
    const D4 zero = {{0.0, 0.0, 0.0, 0.0}};
    for (int k = blockIdx.x * T + threadIdx.x; k < n; k += gridDim.x * T) {
        const Entry e = d.list[t & 1][k];
        d.f[e.x < 0 ? ~e.x : e.x] = zero;
    }
}

/* Every cell of every instance, a run of consecutive cells per block, with
 * the instance carried along (offsets in shared memory): fn(c, b, inside)
 * for all lanes of the warp together; inside is false on padding and past
 * the end (b then still names an instance). */
template <typename FN>
static __device__ __forceinline__ void each_cell(const Dev& d, long long* s_offs, FN fn)
{
    for (int k = threadIdx.x; k <= d.B; k += T)
        s_offs[k] = d.offs[k];
    __syncthreads();
    const long long per = ((d.N + gridDim.x - 1) / gridDim.x + T - 1) / T * T;
    const long long c1 = min(d.N, per * (blockIdx.x + 1));
    int b = 0, hi = d.B - 1; /* the last instance that starts at or before the run */
    while (b < hi) {
        const int mid = (b + hi + 1) >> 1;
        if (s_offs[mid] <= per * blockIdx.x)
            b = mid;
        else
            hi = mid - 1;
    }
    for (long long c0 = per * blockIdx.x; c0 < c1; c0 += T) {
        const long long c = c0 + threadIdx.x;
        while (b + 1 < d.B && s_offs[b + 1] <= c)
            b++;
        fn(c, b, c < c1 && c - s_offs[b] < (long long)d.inst[b].rows * d.inst[b].cols);
    }
}

/* z after the initialisation (z_dem - h0 where h0 > 0), h = h0 with -0 made
 * +0 (the first reference step adds 0.0 to every cell), z + h, and list 0.
 * words: of the run before; one that gave up left outflows in f */
static __global__ void __launch_bounds__(T) k_init(const __grid_constant__ Dev d, const double* __restrict__ z_dem,
                                            const double* __restrict__ h0, double* z,
                                            const unsigned long long* words)
{
    extern __shared__ long long s_offs[];
    const bool gave_up = words[16 * 7] != 0;
    each_cell(d, s_offs, [&](long long c, int b, bool inside) {
        bool wet = false;
        if (gave_up && c < d.N) {
            const D4 zero = {{0.0, 0.0, 0.0, 0.0}};
            d.f[c] = zero;
        }
        if (inside) {
            const double hv = h0[c];
            const double zv = hv > 0.0 ? z_dem[c] - hv : z_dem[c];
            const double hc = sdt::plus_zero(hv);
            z[c] = zv;
            d.h[c] = hc;
            d.zh[c] = zv + hc;
            wet = sdt::is_wet(hc, d.inst[b].eps_bits);
        } else if (c < d.N) {
            z[c] = d.h[c] = d.zh[c] = 0.0;
        }
        const unsigned m = __ballot_sync(0xffffffffu, wet);
        if (m) {
            const int lane = threadIdx.x & 31;
            int at = 0;
            if (lane == 0)
                at = atomicAdd(d.nlist, __popc(m));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (wet)
                d.list[0][at + __popc(m & ((1u << lane) - 1u))] = make_int2((int)c, b);
        }
    });
}

/* list t and z + h again from h (a checkpoint just copied into it) */
static __global__ void __launch_bounds__(T) k_relist(const __grid_constant__ Dev d, int t)
{
    extern __shared__ long long s_offs[];
    each_cell(d, s_offs, [&](long long c, int b, bool inside) {
        bool wet = false;
        if (inside) {
            const double hc = d.h[c];
            d.zh[c] = d.z[c] + hc;
            wet = sdt::is_wet(hc, d.inst[b].eps_bits);
        }
        const unsigned m = __ballot_sync(0xffffffffu, wet);
        if (m) {
            const int lane = threadIdx.x & 31;
            int at = 0;
            if (lane == 0)
                at = atomicAdd(d.nlist + t, __popc(m));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (wet)
                d.list[t & 1][at + __popc(m & ((1u << lane) - 1u))] = make_int2((int)c, b);
        }
    });
}

/* The coefficients of step t's wet cells and their parts of dL/dr, dL/deps.
 * A cell adds its parts to sums of its own, which are added up after the last
 * step in a fixed order (k_parts, k_fold), so that the gradients repeat bit
 * for bit whatever order the lists were appended in, and no atomics queue on
 * an instance's two words.  287,000 entries of 64 instances, us a step: all
 * added to one word per instance and sum 48.7, a segmented scan over each warp
 * and 32 copies of the words 15, so 13.3 (11.0 were the sums not compensated). */
static __device__ __forceinline__ void coeffs(const Dev& d, const Adj& a, int t, int n, long long base, int warp,
                                              int nwarps)
{
    for (int k = warp * 32 + (int)(threadIdx.x & 31); k < n; k += nwarps * 32) {
        const Entry e = d.t_entry[base + k];
        const unsigned elim = e.x >= 0 ? d.t_elim[base + k] : 31u;
        const int kk = 5 - __popc(elim);
        if (kk == 0)
            continue;
        const int c = e.x;
        const Inst I = d.inst[e.y];
        const int lc = (int)(c - I.off);
        const int i = lc / I.cols, j = lc - i * I.cols;
        const D4 diff = d.t_diff[base + k];
        const double own = a.lam[c];
        const D4 sums = a.sums[c]; /* counts from the cell's second step on */
        const bool later = a.stamp[c] >= 0;
        Sum sr = {later ? sums.v[0] : 0.0, later ? sums.v[1] : 0.0};
        Sum se = {later ? sums.v[2] : 0.0, later ? sums.v[3] : 0.0};
        double S = 0.0, lf[4], er = 0.0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            lf[q] = 0.0;
            if (!(elim & (2u << q))) {
                int na, nb;
                const bool in = nbr(I, i, j, q, &na, &nb);
                lf[q] = (in ? a.lam[I.off + (long long)na * I.cols + nb] : 0.0) - own;
                S += lf[q];
                er += lf[q] * diff.v[q];
            }
        }
        const double g = cal_div_small(I.r, kk) * S; /* exact division by 1..5 on the integer pipe */
        D4 w;
#pragma unroll
        for (int q = 0; q < 4; q++)
            w.v[q] = (elim & (2u << q)) ? 0.0 : g - I.r * lf[q];
        a.stamp[c] = t;
        a.g[c] = g;
        a.w[c] = w;
        sum_add(sr, er);
        if (elim & 1u) {
            sum_add(se, -cal_div_small(S * I.r, kk));
            if (a.mu)
                a.mu[c] += g;
        }
        const D4 sums1 = {{sr.v, sr.c, se.v, se.c}};
        a.sums[c] = sums1;
    }
}

static __global__ void __launch_bounds__(T) k_coeffs(const __grid_constant__ Dev d, const __grid_constant__ Adj a, int t)
{
    const int n = d.nlist[t];
    const long long base = tape_base(d, t, n);
    if (base >= 0)
        coeffs(d, a, t, n, base, (threadIdx.x >> 5) * gridDim.x + blockIdx.x, gridDim.x * (T / 32));
}

/* Block (p, b): the sums of the p-th run of instance b's cells.  Few cells
 * were ever wet; the rest of the work is the additions that join the
 * threads' sums, on an FP64 pipe that takes some 19 clocks a warp: one warp
 * joins them (64 instances, 84 MB of stamps: in every warp, with 64 runs an
 * instance, 1081 us) */
static __global__ void __launch_bounds__(T) k_parts(const __grid_constant__ Dev d, const __grid_constant__ Adj a)
{
    __shared__ Sum s_sum[2][T];
    const Inst I = d.inst[blockIdx.y];
    const long long n = (long long)I.rows * I.cols, per = (n + PARTS - 1) / PARTS;
    const long long c1 = min(n, per * (blockIdx.x + 1));
    Sum q[2] = {{0.0, 0.0}, {0.0, 0.0}};
    for (long long c0 = per * blockIdx.x; c0 < c1; c0 += 8 * T) {
        int stamp[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const long long c = c0 + u * T + threadIdx.x;
            stamp[u] = c < c1 ? a.stamp[I.off + c] : -1;
        }
#pragma unroll
        for (int h = 0; h < 8; h += 4) {
            D4 v[4];
            bool any = false;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                v[u] = {{0.0, 0.0, 0.0, 0.0}};
                if (stamp[h + u] >= 0) {
                    v[u] = a.sums[I.off + c0 + (h + u) * T + threadIdx.x];
                    any = true;
                }
            }
            if (any) /* in the flow, mostly the whole warp */
#pragma unroll
                for (int u = 0; u < 4; u++)
#pragma unroll
                    for (int k = 0; k < 2; k++) {
                        sum_add(q[k], v[u].v[2 * k]);
                        q[k].c += v[u].v[2 * k + 1];
                    }
        }
    }
    s_sum[0][threadIdx.x] = q[0];
    s_sum[1][threadIdx.x] = q[1];
    __syncthreads();
    const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (k >= 2)
        return;
    Sum v = s_sum[k][lane];
    for (int w = 1; w < T / 32; w++)
        sum_add(v, s_sum[k][w * 32 + lane]);
    for (int o = 16; o > 0; o >>= 1)
        sum_add(v, Sum{__shfl_down_sync(0xffffffffu, v.v, o), __shfl_down_sync(0xffffffffu, v.c, o)});
    if (lane == 0) {
        double* out = a.part + (size_t)blockIdx.x * 4 * d.B + k * d.B + blockIdx.y;
        out[0] = v.v;
        out[2 * d.B] = v.c;
    }
}

/* the instances' dL/dr and dL/deps (n = 2B): their partial sums in a fixed
 * order, a warp each */
static __global__ void __launch_bounds__(T) k_fold(const double* __restrict__ part, double* __restrict__ grad, int n)
{
    const int q = blockIdx.x * (T / 32) + (int)(threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (q >= n)
        return;
    Sum v = {0.0, 0.0};
    for (int p = lane; p < PARTS; p += 32)
        sum_add(v, Sum{part[(size_t)p * 2 * n + q], part[(size_t)p * 2 * n + n + q]});
    for (int o = 16; o > 0; o >>= 1)
        sum_add(v, Sum{__shfl_down_sync(0xffffffffu, v.v, o), __shfl_down_sync(0xffffffffu, v.c, o)});
    if (lane == 0)
        grad[q] = v.v - v.c;
}

/* lambda_t from lambda_{t+1}: every cell whose lambda changes lies in a tile
 * that step t flagged (it kept a neighbour or is one that was kept) */
static __device__ __forceinline__ void gather(const Dev& d, const Adj& a, int t, int ntiles, int group, int ngroups)
{
    const int* tiles = d.tiles + (size_t)t * d.ntiles;
    for (int item = group; item < ntiles; item += ngroups) {
        const int tile = tiles[item];
        const Inst I = d.inst[d.tile_inst[tile]];
        const int lt = tile - I.tile0;
        const int ty = lt / I.tiles_x, tx = lt - ty * I.tiles_x;
        for (int q = threadIdx.x % T; q < 1 << (d.lw + d.lh); q += T) {
            const int i = (ty << d.lh) + (q >> d.lw), j = (tx << d.lw) + (q & ((1 << d.lw) - 1));
            if (i >= I.rows || j >= I.cols)
                continue;
            const long long c = I.off + (long long)i * I.cols + j;
            long long cn[4];
            unsigned have = a.stamp[c] == t ? 16u : 0u;
#pragma unroll
            for (int s = 0; s < 4; s++) {
                int na, nb;
                const bool in = nbr(I, i, j, s, &na, &nb);
                cn[s] = I.off + (long long)na * I.cols + nb;
                if (in && a.stamp[cn[s]] == t)
                    have |= 1u << s;
            }
            if (!have)
                continue;
            double from_nb = 0.0;
#pragma unroll
            for (int s = 0; s < 4; s++) /* x is neighbour 3 - s of its neighbour s */
                if (have & (1u << s))
                    from_nb += a.w[cn[s]].v[3 - s];
            a.lam[c] = a.lam[c] + ((have & 16u) ? a.g[c] : 0.0) + from_nb;
        }
    }
}

static __global__ void __launch_bounds__(T) k_gather(const __grid_constant__ Dev d, const __grid_constant__ Adj a, int t)
{
    if (tape_base(d, t, d.nlist[t]) >= 0)
        gather(d, a, t, d.counts[t], blockIdx.x, gridDim.x);
}

/* ---- all steps in one cooperative launch --------------------------------
 * Launched one after another on a stream, dependent kernels that read their
 * counts from memory start 4.1 us apart at least (1.2 us as nodes of a
 * graph); the phases of a step separated by grid barriers of one block of
 * 1024 threads per SM take 1.45 us each (sciddicaT.cu, sdt2::k_persist), so
 * runs that are not recorded go this way (one grid of 512 x 480, us per step:
 * forward 16 -> 10.8, reverse 15 -> 7.7; 40 instances forward 21 -> 17).  The
 * blocks take every SM's registers, so that kernels of other streams wait for
 * the end of the launch; the recorded form leaves them room between its own. */
constexpr int GROUPS = 4, PT = GROUPS * T;
constexpr unsigned SPIN_LIMIT = 1u << 22;

/* words[16 k]: k = 0, 1, 2 the flagged tiles of steps by t % 3; 3, 4, 5 the
 * next list's entries; 6 arrivals of the plain barrier; counts in the low 32
 * bits, a phase's arrivals in the high 32 (words zero at launch); word 7:
 * not 0 when a wait gave up */
constexpr int NWORDS = 8;

/* End of a phase: the block's arrival on *word, then the wait for all of
 * `rounds` x gridDim.x arrivals (a word counted afresh each use: rounds = 1);
 * bounded, and false for the whole block when it gave up.  *low: the word's
 * low half when complete. */
static __device__ __forceinline__ bool phase_end(unsigned long long* word, unsigned rounds, unsigned long long* err,
                                                 int* low)
{
    __shared__ int s_ok, s_low;
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(word), "l"(1ull << 32) : "memory");
        unsigned long long v = 0;
        int ok = 0;
        for (unsigned polls = 0; polls < SPIN_LIMIT; polls++) {
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(word) : "memory");
            if ((unsigned)(v >> 32) >= rounds * gridDim.x) {
                ok = 1;
                break;
            }
            __nanosleep(20);
        }
        if (!ok)
            atomicExch(err, 1ull);
        s_ok = ok;
        s_low = (int)(unsigned)v;
    }
    __syncthreads();
    *low = s_low;
    return s_ok != 0;
}

/* steps [t0, t1) from list t0 */
static __global__ void __launch_bounds__(PT, 1) k_steps(const __grid_constant__ Dev d, int t0, int t1, int epoch0,
                                                       int taped, unsigned long long* words)
{
    const int warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, nwarps = gridDim.x * (PT / 32);
    const int group = (threadIdx.x / T) * gridDim.x + blockIdx.x, ngroups = gridDim.x * GROUPS;
    int n = d.nlist[t0];
    /* the tape's state lies in shared memory: the two phases leave no
     * register for it */
    __shared__ long long s_at, s_off; /* as for tape_slot; entries so far */
    const bool again = d.tpos != nullptr, first = blockIdx.x == 0 && threadIdx.x == 0;
    if (threadIdx.x == 0 && taped) {
        s_off = d.toff[t0];
        s_at = again ? d.tpos[t0] : s_off;
    }
    __syncthreads();
    for (int t = t0; t < t1; t++) {
        unsigned long long* tword = words + 16 * (t % 3);
        unsigned long long* lword = words + 16 * (3 + t % 3);
        if (first) {
            /* the next step's words, last polled two steps ago */
            words[16 * ((t + 1) % 3)] = 0;
            words[16 * (3 + (t + 1) % 3)] = 0;
        }
        outflows(d, t, epoch0 + t, n, taped ? tape_slot(d.cap, again, s_at, n) : -1, tword, warp, nwarps);
        int ntiles;
        if (!phase_end(tword, 1, words + 16 * 7, &ntiles))
            return;
        if (threadIdx.x == 0 && taped) { /* read again after the next barrier */
            s_at = tape_next(again, s_at, tape_slot(d.cap, again, s_at, n), n);
            s_off += n;
            if (first) {
                d.toff[t + 1] = s_off;
                if (again)
                    d.tpos[t + 1] = s_at;
            }
        }
        update<GROUPS>(d, t, epoch0 + t, ntiles, n, lword, group, ngroups);
        if (first)
            d.counts[t] = ntiles;
        if (!phase_end(lword, 1, words + 16 * 7, &n))
            return;
        if (first)
            d.nlist[t + 1] = n;
    }
    if (taped && first && *d.need < s_off)
        *d.need = s_off;
}

/* the adjoint of steps [t0, t1), last first (steps that did not fit the tape
 * are left out, as by k_coeffs) */
static __global__ void __launch_bounds__(PT, 1) k_sweep(const __grid_constant__ Dev d, const __grid_constant__ Adj a,
                                                       int t0, int t1, unsigned long long* words)
{
    const int warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, nwarps = gridDim.x * (PT / 32);
    const int group = (threadIdx.x / T) * gridDim.x + blockIdx.x, ngroups = gridDim.x * GROUPS;
    unsigned round = 0;
    int unused;
    int n = d.nlist[t1 - 1], ntiles = d.counts[t1 - 1];
    long long base = tape_base(d, t1 - 1, n);
    for (int t = t1 - 1; t >= t0; t--) {
        if (base >= 0)
            coeffs(d, a, t, n, base, warp, nwarps);
        if (!phase_end(words + 16 * 6, ++round, words + 16 * 7, &unused))
            return;
        if (base >= 0)
            gather(d, a, t, ntiles, group, ngroups);
        if (t > t0) { /* known since the forward: loaded before the wait */
            n = d.nlist[t - 1];
            ntiles = d.counts[t - 1];
            base = tape_base(d, t - 1, n);
        }
        if (!phase_end(words + 16 * 6, ++round, words + 16 * 7, &unused))
            return;
    }
}

/* h into the caller's array; NaN everywhere when a wait gave up */
static __global__ void k_out(const double* __restrict__ h, double* __restrict__ out, long long n,
                             const unsigned long long* words)
{
    const bool bad = words[16 * 7] != 0;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x)
        out[c] = bad ? __longlong_as_double(0x7ff8000000000000LL) : h[c];
}

/* lambda_T = 2 (h_T - target), mu_T the same, and the instances' losses */
static __global__ void __launch_bounds__(T) k_loss(const __grid_constant__ Dev d, const __grid_constant__ Adj a,
                                            const double* __restrict__ target, double* loss)
{
    extern __shared__ long long s_offs[];
    double acc = 0.0;
    int cur = -1; /* the instance acc belongs to, the same in every lane */
    auto flush = [&]() {
        double v = acc;
        for (int o = 16; o > 0; o >>= 1)
            v += __shfl_down_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0 && cur >= 0 && v != 0.0)
            atomicAdd(loss + cur, v);
        acc = 0.0;
    };
    each_cell(d, s_offs, [&](long long c, int b, bool inside) {
        const double diff = inside ? d.h[c] - target[c] : 0.0;
        if (c < d.N) {
            a.lam[c] = 2.0 * diff;
            if (a.mu)
                a.mu[c] = 2.0 * diff;
        }
        const int b0 = __shfl_sync(0xffffffffu, b, 0);
        if (__all_sync(0xffffffffu, b == b0)) {
            if (b0 != cur) {
                flush();
                cur = b0;
            }
            acc += diff * diff;
        } else if (diff != 0.0) {
            atomicAdd(loss + b, diff * diff);
        }
    });
    flush();
}

/* dL/dh0 (see the top of the file) */
static __global__ void k_final_grad(const double* __restrict__ h0, const double* __restrict__ lam,
                             const double* __restrict__ mu, double* __restrict__ g_h0, long long n)
{
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x)
        g_h0[c] = h0[c] > 0.0 ? mu[c] : lam[c];
}

static int dense_blocks(long long n)
{
    const long long b = (n + T - 1) / T;
    return (int)(b > 152 * 8 ? 152 * 8 : (b < 1 ? 1 : b));
}

/* steps [t0, t1) queued; epochs are unique per run since the stamps were
 * cleared */
static void queue_steps(const Dev& d, int t0, int t1, int epoch0, bool taped, cudaStream_t st)
{
    for (int t = t0; t < t1; t++) {
        k_outflows<<<BLOCKS, T, 0, st>>>(d, t, epoch0 + t, taped ? 1 : 0);
        k_update<<<BLOCKS, T, 0, st>>>(d, t, epoch0 + t);
    }
}

/* the adjoint of steps [t0, t1), last first */
static void queue_adjoint(const Dev& d, const Adj& a, int t0, int t1, cudaStream_t st)
{
    for (int t = t1 - 1; t >= t0; t--) {
        k_coeffs<<<BLOCKS, T, 0, st>>>(d, a, t);
        k_gather<<<BLOCKS, T, 0, st>>>(d, a, t);
    }
}

/* dL/dr and dL/deps from the cells' sums */
static void queue_grad(const Dev& d, const Adj& a, cudaStream_t st)
{
    k_parts<<<dim3(PARTS, d.B), T, 0, st>>>(d, a);
    k_fold<<<(2 * d.B + T / 32 - 1) / (T / 32), T, 0, st>>>(a.part, a.grad, 2 * d.B);
}

static int sm_count()
{
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    }
    return sms;
}

static bool capturing(cudaStream_t st)
{
    cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(st, &c) == cudaSuccess && c != cudaStreamCaptureStatusNone;
}

/* As queue_steps, queue_adjoint, in one cooperative launch each (words:
 * NWORDS x 16), or like them while a caller captures the stream and where
 * the launch is refused: a process that is given
 * a part of the SMs cannot have a block on each.  (A launch that fails for
 * another reason leaves an error that the plain launches meet again.) */
static void launch_steps(Dev& d, int t0, int t1, int epoch0, bool taped, unsigned long long* words, cudaStream_t st)
{
    if (t1 <= t0)
        return;
    if (capturing(st)) {
        queue_steps(d, t0, t1, epoch0, taped, st);
        return;
    }
    /* word 7, an error of an earlier part of the run, stays */
    cudaMemsetAsync(words, 0, sizeof(unsigned long long) * 16 * 7, st);
    int on = taped ? 1 : 0;
    void* args[] = {&d, &t0, &t1, &epoch0, &on, &words};
    if (cudaLaunchCooperativeKernel((const void*)k_steps, dim3(sm_count()), dim3(PT), args, 0, st) != cudaSuccess) {
        (void)cudaGetLastError();
        queue_steps(d, t0, t1, epoch0, taped, st);
    }
}

static void launch_sweep(Dev& d, Adj& a, int t0, int t1, unsigned long long* words, cudaStream_t st)
{
    if (t1 <= t0)
        return;
    cudaMemsetAsync(words, 0, sizeof(unsigned long long) * 16 * 7, st);
    void* args[] = {&d, &a, &t0, &t1, &words};
    if (cudaLaunchCooperativeKernel((const void*)k_sweep, dim3(sm_count()), dim3(PT), args, 0, st) != cudaSuccess) {
        (void)cudaGetLastError();
        queue_adjoint(d, a, t0, t1, st);
    }
}

} // namespace sdtw
