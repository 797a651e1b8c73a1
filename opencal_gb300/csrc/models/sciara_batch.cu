/*
 * sciara_batch.cu -- SCIARA-fv2 scenarios (one grid or many, each with its
 * own morphology, vents and emission rates) advanced by a split step:
 *
 *   K0 (vents): updateVentsEmission (OpenCAL-OMP/examples/calomp_sciara-fv2/
 *      source/Sciara.cpp:3-16): thickness += rate / Pac * Pclock at each
 *      emitting vent (the last vent listed for a cell wins, as the EP's
 *      get-current-then-set does), temperature = PTvent; a vent cell that
 *      had no lava joins the lava list.
 *   K1 (flows): empiricalFlows + outflowsMin (Sciara.cpp:18-105) for every
 *      cell of the lava list (Slt > 0), one thread each, spread over the
 *      whole GPU -- the power laws, the shear test and the minimisation
 *      are the step's FP64 work.  The eight outflows of list entry k, and
 *      each outflow times the cell's temperature (the product width_update
 *      forms at the receiver, same operands), go to compact slot k; a
 *      per-cell (epoch, slot) map makes them addressable by cell.  A
 *      receiver without lava joins the receiver list once (epoch stamp).
 *   K2 (update): width_update, updateTemperature and the steering's border
 *      reset (Sciara.cpp:106-169, 185-193) at every lava cell and every
 *      receiver, one thread each over the whole GPU, in place: a cell reads
 *      only its own state and the compact outflows; it joins the next lava
 *      list if it still holds lava.  Any other cell has no lava and no
 *      inflow, so it is unchanged (border cells hold 0 from the start).
 *   For the adjoint, K1 leaves its compact slots and K2 what the update's
 *   adjoint needs of every cell it visits on a tape, one entry per visited
 *   cell and step.
 *
 * Arithmetic is the reference's, operation by operation (--fmad=false),
 * except the transcendental forms of sciara_math.cuh (exp10, the shear test
 * without atan / cos, T^3 and cbrt), shared with the device-process program
 * (sciara.cu), which this step reproduces bit for bit.  All scenarios share
 * the physical parameters and the emission schedule's length, so they run
 * the same number of steps (the reference stops when the elapsed time
 * reaches the emission's end).
 *
 * Layout: scenarios packed back to back (offsets padded to 32 cells); per
 * cell Sz, Slt, St, Msl (FP64), Mb (byte), the (epoch, slot) map (8 B), the
 * outflow mask (byte), the receiver stamp (4 B) and a copy of the initial
 * Sz, Slt, St (every run starts from it): 70 B per cell; per list slot (capacity chosen at
 * creation) two lava-list entries, a receiver entry and the outflows
 * (140 B).
 */
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <thread>
#include <vector>

#include "exact_div.cuh"
#include "sciara_math.cuh"

namespace sci2 {

constexpr int T = 256;
constexpr int K1T = 64;
constexpr int BT = 64; /* reverse sweep: entries per block */
constexpr int TW = 32, TH = 16; /* K2 tile; 2 cells per thread */
constexpr int K2_BLOCKS = 152 * 4;
constexpr int MAX_INST = 1024;

struct Phys {
    double Pclock, Pc, Pac, PTsol, PTvent, a, b, c, d, Pcool, Prho, Pepsilon, Psigma, Pcv, rad2;
    double rrad2, w2; /* RN(1 / rad2), Pc * Pc */
    double cool3;     /* 3 Pepsilon Psigma Pclock Pcool / (Prho Pcv Pac) */
    int rad2_recip;   /* x / rad2 by cal_div_recip (its precondition holds) */
};

struct Inst {
    int rows, cols;
    long long off;
    int tiles_x, tiles_y, tile0, pad;
};

/* counts[]: [0] lava list length, [5] K2 ticket, [6] epoch, [7] tiles
 * flagged in this step, [8] lava- or receiver-list overflow flag, [9] tiles
 * flagged in all steps so far, [11] receiver list length, [12] tiles flagged
 * in the previous step, [13] lava cells after the last update */
struct Dev {
    const Inst* inst;
    const long long* offs;
    int B;
    double* Sz;
    double* Slt;
    double* St;
    double* Msl;
    const unsigned char* Mb;
    double* fc;   /* 16 doubles per list slot: f[8], f * St[8]; only those in fmask are written */
    unsigned char* fmask; /* per lava cell: bit k - 1 = neighbour k must add the outflow to it (k_flows) */
    int2* map;    /* per cell: (epoch, slot) */
    int* recv;    /* per cell: epoch in which it was listed as a receiver */
    int* rlist;   /* cells without lava that receive a flow this step */
    int* list;    /* lava cells, tile by tile, row-major within a tile */
    unsigned* mask; /* per tile 16 words: bit j of word r = cell (r, j) holds lava after K2 */
    int* counts;
    int* tflag;
    int* tlist;
    long long ncells;
    int capacity;
    /* vent cells: the vents of one scenario at one cell form a group; per
     * group and phase the vent whose emission takes effect (the last with a
     * positive one, -1: none) and its thickness */
    int ngroups;
    const int* g_cell;    /* packed cell */
    const int* g_eff;     /* ngroups x nphases */
    const double* g_emit; /* ngroups x nphases */
    int nphases;
    unsigned emission_time;
    Phys ph;
};

static __device__ __forceinline__ int locate(const long long* s_offs, int B, long long c)
{
    int lo = 0, hi = B - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (s_offs[mid] <= c)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

/* Moore neighbour k = 0..8 (OpenCAL order: centre, N, W, E, S, NW, SW, SE, NE) */
__device__ __constant__ int kMi[9] = {0, -1, 0, 0, 1, -1, 1, 1, -1};
__device__ __constant__ int kMj[9] = {0, 0, -1, 1, 0, -1, -1, 1, 1};

static __device__ __forceinline__ bool nbr(const Inst& I, int i, int j, int k, long long* c)
{
    const int a = i + kMi[k], b = j + kMj[k];
    if ((unsigned)a >= (unsigned)I.rows || (unsigned)b >= (unsigned)I.cols)
        return false; /* flat boundary */
    *c = I.off + (long long)a * I.cols + b;
    return true;
}

static __device__ __forceinline__ void append(int* list, int* count, int capacity, int* overflow, int value)
{
    const int pos = atomicAdd(count, 1);
    if (pos < capacity)
        list[pos] = value;
    else
        atomicExch(overflow, 1);
}

static __device__ __forceinline__ void flag_tile(const Dev& d, int t, int epoch)
{
    if (d.tflag[t] != epoch && atomicExch(d.tflag + t, epoch) != epoch)
        d.tlist[atomicAdd(d.counts + 7, 1)] = t;
}

/* K0: the lava list of this step, and the vent emission.
 * The list is collected from the lava masks K2 left in the tiles flagged by
 * the previous step (every cell that can hold lava after an update lies in
 * one), tile by tile and row-major within a tile, so that neighbouring list
 * entries are neighbouring cells; the masks are cleared on the way.  Half a
 * warp reads a tile's 16 mask words and reserves the tile's run of list
 * slots with one atomic.  (The first step uses the list the priming kernel
 * built.)  Block 0 also emits at the vents, one thread per scenario; a
 * vent cell that had no lava is appended. */
__global__ void __launch_bounds__(T) k_collect(const __grid_constant__ Dev d, unsigned phase, int rebuild)
{
    if (blockIdx.x == 0) {
        if (threadIdx.x == 0)
            d.counts[13] = 0;
        for (int g = threadIdx.x; g < d.ngroups; g += blockDim.x) {
            const int c = d.g_cell[g];
            const int eff = phase < (unsigned)d.nphases ? d.g_eff[(size_t)g * d.nphases + phase] : -1;
            /* the process reads the current thickness: the cell's vents add
             * to the value before this step's emission, the last positive
             * one wins */
            const double orig = d.Slt[c];
            if (eff >= 0) {
                d.Slt[c] = orig + d.g_emit[(size_t)g * d.nphases + phase];
                d.St[c] = d.ph.PTvent;
                if (!(orig > 0))
                    append(d.list, d.counts + 0, d.capacity, d.counts + 8, c);
            }
        }
    }
    if (!rebuild)
        return;
    const int ntiles = d.counts[12];
    const int lane = threadIdx.x & 31, half = lane >> 4, l = lane & 15;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int item0 = 2 * warp; item0 < ntiles; item0 += 2 * nwarps) {
        const int item = item0 + half;
        unsigned w = 0;
        int t = 0;
        if (item < ntiles) {
            t = d.tlist[item];
            w = d.mask[(size_t)t * 16 + l];
            if (w)
                d.mask[(size_t)t * 16 + l] = 0;
        }
        const int cnt = __popc(w);
        int inc = cnt; /* inclusive scan over the half warp */
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, inc, o, 16);
            if (l >= o)
                inc += v;
        }
        int base = 0;
        if (l == 15 && inc > 0)
            base = atomicAdd(d.counts + 0, inc);
        base = __shfl_sync(0xffffffffu, base, 15, 16);
        if (w) {
            int lo = 0, hi = d.B - 1; /* the tile's instance: largest b with tile0 <= t */
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (d.inst[mid].tile0 <= t)
                    lo = mid;
                else
                    hi = mid - 1;
            }
            const Inst I = d.inst[lo];
            const int lt = t - I.tile0;
            const int ty = lt / I.tiles_x, tx = lt - ty * I.tiles_x;
            const long long row = I.off + (long long)(ty * TH + l) * I.cols + tx * TW;
            int pos = base + inc - cnt;
            while (w) {
                const int bit = __ffs(w) - 1;
                w &= w - 1;
                if (pos < d.capacity)
                    d.list[pos] = (int)(row + bit);
                else
                    atomicExch(d.counts + 8, 1);
                pos++;
            }
        }
    }
}

/* outflowsMin (Sciara.cpp:23-90) at lava cell c, with what its adjoint needs */
struct Flow {
    double h[9], z[9], H[9], f[9];
    double avg, Pr, t;
    long long cn[9];
    unsigned inside, S, F; /* in-grid neighbours, final set, positive outflows */
    int nS;
};

/* The arithmetic of outflowsMin with every FP64 operation that can leave
 * the narrow FP64 pipe moved to the integer pipe, each with identical
 * results (exact_div.cuh): comparisons of non-negative values on the bit
 * patterns; z0 + h0 > z_k + h_k as the sign of their difference (for finite
 * values, a - b > 0 exactly when a > b); the average's division by the set
 * size (1..9) by integer long division; the diagonal altitude's division by
 * rad2 through its reciprocal with Markstein's correction. */
static __device__ __forceinline__ void compute_flows(const Dev& d, const Inst& I, long long c, int i, int j, Flow& F)
{
    double dz[9];
    bool in_set[9];
    const double t = d.St[c];
    F.t = t;
    F.Pr = sci_power_law(d.ph.a, d.ph.b, t);
    const double hc = sci_power_law(d.ph.c, d.ph.d, t);
    const double sz0 = d.Sz[c];
    const bool recip = d.ph.rad2_recip != 0;
    F.inside = 0;
#pragma unroll
    for (int q = 0; q < 9; q++) {
        const bool in = nbr(I, i, j, q, &F.cn[q]);
        F.inside |= (in ? 1u : 0u) << q;
        F.h[q] = in ? d.Slt[F.cn[q]] : 0.0;
        const double sz = in ? d.Sz[F.cn[q]] : 0.0;
        F.H[q] = F.f[q] = dz[q] = 0;
        if (q < 5)
            F.z[q] = sz;
        else
            F.z[q] = sz0 - (recip ? cal_div_recip(sz0 - sz, d.ph.rad2, d.ph.rrad2) : (sz0 - sz) / d.ph.rad2);
    }
    F.H[0] = F.z[0];
    in_set[0] = true;
    const double zh0 = F.z[0] + F.h[0];
#pragma unroll
    for (int q = 1; q < 9; q++) {
        const double Hq = F.z[q] + F.h[q];
        const double dq = zh0 - Hq;
        in_set[q] = cal_pos(dq);
        if (in_set[q]) {
            F.H[q] = Hq;
            dz[q] = dq;
        }
    }
    bool loop;
    double avg;
    int counter;
    do {
        loop = false;
        avg = F.h[0];
        counter = 0;
#pragma unroll
        for (int q = 0; q < 9; q++)
            if (in_set[q]) {
                avg += F.H[q];
                counter++;
            }
        if (counter != 0)
            avg = cal_div_small(avg, counter);
#pragma unroll
        for (int q = 0; q < 9; q++)
            if (in_set[q] && cal_le(avg, F.H[q])) {
                in_set[q] = false;
                loop = true;
            }
    } while (loop);
    /* the last average was formed over the set before the final (empty)
     * round of eliminations: that set is the final one */
    F.avg = avg;
    F.nS = counter;
    F.S = 0;
    F.F = 0;
#pragma unroll
    for (int q = 0; q < 9; q++)
        F.S |= (in_set[q] ? 1u : 0u) << q;
    const double h0 = F.h[0];
    const double h0sq = h0 * h0, rhs = hc * hc * d.ph.w2;
#pragma unroll
    for (int q = 1; q < 9; q++) {
        double fq = 0.0;
        /* sci_shear_exceeded(h0, hc, dz, w): h0 > 0 and h0^2 (w^2 + dz^2) > hc^2 w^2 */
        if (in_set[q] && cal_pos(h0) && cal_gt(h0sq * (d.ph.w2 + dz[q] * dz[q]), rhs))
            fq = F.Pr * (avg - F.H[q]);
        /* empiricalFlows stores only positive outflows; the rest stay 0 */
        if (!cal_pos(fq))
            fq = 0.0;
        F.f[q] = fq;
        if (cal_pos(fq))
            F.F |= 1u << q;
    }
}

/* The tape of a run whose gradient is wanted: per step one entry for every
 * cell K2 visits, in K2's order (the lava list, then the receivers), at
 * consecutive slots from the step's base.  It holds everything the reverse
 * sweep reads, so the sweep neither restores the state nor evaluates the
 * flows, the mixing or the cooling again: 200 bytes an entry, where copying
 * the visited 32 x 16 tiles' state took 12 KB a tile (16 scenarios of
 * 700 x 768, 240 steps: 4.6 GB of tiles).  Lava entries: the sixteen
 * doubles of K1's slot (K2 reads them here too), the power law Pr and the
 * masks; every entry: the update's intermediate values. */
struct Tape {
    int* cell;
    unsigned* mask;      /* lava entries: F | S << 9 | in-grid neighbours << 18 */
    unsigned char* flag; /* E_* */
    double* pr;          /* lava entries */
    double* fc;          /* 16 per entry */
    double* val;         /* NVAL arrays of cap: t, t', h', residual, D, aus, cooled t */
    long long cap;       /* entries; 0: the run is not taped */
    long long* used;     /* entries of the steps so far, counted on past the capacity */
    long long* step_base;
    int* step_lava; /* lava entries of each step */
    int* step_n;    /* all entries */
};
constexpr int NVAL = 7;
constexpr long long EXPONENT = 0x7ff0000000000000LL; /* all ones: infinite or NaN */
constexpr size_t ENTRY_BYTES = sizeof(int) * 2 + 1 + sizeof(double) * (1 + 16 + NVAL);
constexpr unsigned char E_FLOW = 1, E_BORDER = 2, E_LAVA = 4, E_SOLID = 8;

/* where this step's compact slots are: the list's scratch, or the tape
 * while the step's lava entries fit (a run that outgrows the tape is
 * repeated with a larger one); K1 and K2 decide alike */
static __device__ __forceinline__ double* slots_of(const Dev& d, const Tape& tp, int nlava, long long* base)
{
    *base = tp.cap ? *tp.used : 0;
    return tp.cap && *base + nlava <= tp.cap ? tp.fc + 16 * (size_t)*base : d.fc;
}

/* K1: outflows of every lava cell into compact slots.  A receiver without
 * lava joins the receiver list once (epoch stamp), so that K2 visits
 * exactly the lava cells and the cells they flow into.  The tiles of the
 * lava cells and receivers are flagged: they hold every cell that can hold
 * lava after K2 (K0 of the next step collects the list from them). */
__global__ void __launch_bounds__(K1T) k_flows(const __grid_constant__ Dev d, const __grid_constant__ Tape tp)
{
    __shared__ long long s_offs[MAX_INST + 1];
    for (int k = threadIdx.x; k <= d.B; k += blockDim.x)
        s_offs[k] = d.offs[k];
    __syncthreads();
    const int epoch = d.counts[6];
    const int n = min(d.counts[0], d.capacity);
    long long base;
    double* slots = slots_of(d, tp, n, &base);
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int c = d.list[k];
        const Inst I = d.inst[locate(s_offs, d.B, c)];
        const long long lc = c - I.off;
        const int i = (int)(lc / I.cols), j = (int)(lc - (long long)i * I.cols);
        Flow F;
        compute_flows(d, I, c, i, j, F);
        if (slots != d.fc) {
            tp.mask[base + k] = F.F | (F.S << 9) | (F.inside << 18);
            tp.pr[base + k] = F.Pr;
        }
        double* slot = slots + (size_t)k * 16;
        /* a flow that is 0 changes nothing where it arrives (update_cell
         * leaves it out), unless the temperature is not finite: 0 x t is
         * then NaN, in the model's sum of the receiver too */
        const unsigned sent = (__double_as_longlong(F.t) & EXPONENT) == EXPONENT ? 0x1feu : F.F;
        d.fmask[c] = (unsigned char)(sent >> 1);
#pragma unroll
        for (int q = 1; q < 9; q++) {
            if (!((sent >> q) & 1u))
                continue;
            slot[q - 1] = F.f[q];
            slot[8 + q - 1] = F.f[q] * F.t;
            if ((F.F >> q) & (F.inside >> q) & 1u) {
                const int cn = (int)F.cn[q];
                if (!cal_pos(F.h[q]) && d.recv[cn] != epoch && atomicExch(d.recv + cn, epoch) != epoch) {
                    append(d.rlist, d.counts + 11, d.capacity, d.counts + 8, cn);
                    const long long rc = F.cn[q] - I.off;
                    const int ri = (int)(rc / I.cols), rj = (int)(rc - (long long)ri * I.cols);
                    flag_tile(d, I.tile0 + (ri / TH) * I.tiles_x + rj / TW, epoch);
                }
            }
        }
        d.map[c] = make_int2(epoch, k);
        flag_tile(d, I.tile0 + (i / TH) * I.tiles_x + j / TW, epoch);
    }
}

/* width_update and updateTemperature at one cell (Sciara.cpp:106-169):
 * the forward quantities, with the outflows found through the (epoch, slot)
 * map */
struct CellFwd {
    double h, t, sz, in_sum, out_sum, ht, residual, D, hn, tn, aus, st;
    bool flowcond, border, lava, solid;
};

static __device__ __forceinline__ void compute_cell(const Dev& d, const double* slots, const Inst& I, int i, int j,
                                                    long long x, int epoch, CellFwd& Cf)
{
    const int opp[8] = {3, 2, 1, 0, 6, 7, 4, 5};
    Cf.h = d.Slt[x];
    Cf.t = d.St[x];
    Cf.sz = d.Sz[x];
    const int2 me = d.map[x];
    const double* mine = slots + (size_t)me.y * 16;
    const unsigned out = me.x == epoch ? d.fmask[x] : 0u;
    /* which neighbours' flows arrive here, and their slots: most of a cell's
     * eight neighbours send nothing, and a zero added changes nothing, so
     * only the flows there are (and those of a neighbour whose temperature is
     * not finite) get loaded and added (16 scenarios of 700 x
     * 768, us a step: 23.3 with all sixteen loads and 24 additions of a cell
     * amid lava, 21.7 so; k_flows, which then stores no zeros, 34.3 and
     * 31.4) */
    unsigned in = 0;
    int from[9];
#pragma unroll
    for (int n = 1; n < 9; n++) {
        long long cn;
        from[n] = 0;
        if (nbr(I, i, j, n, &cn)) {
            const int2 m = d.map[cn];
            const unsigned f = d.fmask[cn];
            if (m.x == epoch && ((f >> opp[n - 1]) & 1u)) {
                in |= 1u << n;
                from[n] = m.y;
            }
        }
    }
    double flow[9], heat[9], gone[9];
#pragma unroll
    for (int n = 1; n < 9; n++) {
        flow[n] = heat[n] = gone[n] = 0.0;
        if ((in >> n) & 1u) {
            const double* s = slots + (size_t)from[n] * 16;
            flow[n] = s[opp[n - 1]];
            heat[n] = s[8 + opp[n - 1]]; /* inFlow * neigh_t, formed at the source with the same operands */
        }
        if ((out >> (n - 1)) & 1u)
            gone[n] = mine[n - 1];
    }
    double ht = 0, in_sum = 0, out_sum = 0;
#pragma unroll
    for (int n = 1; n < 9; n++) {
        if ((in >> n) & 1u) {
            ht += heat[n];
            in_sum += flow[n];
        }
        if ((out >> (n - 1)) & 1u)
            out_sum += gone[n];
    }
    Cf.ht = ht;
    Cf.in_sum = in_sum;
    Cf.out_sum = out_sum;
    double h_next = Cf.h;
    double t_next = Cf.t;
    h_next += in_sum - out_sum;
    Cf.flowcond = in_sum > 0 || out_sum > 0;
    Cf.residual = 0.0;
    Cf.D = 1.0;
    if (Cf.flowcond) {
        Cf.residual = Cf.h - out_sum;
        Cf.D = Cf.residual + in_sum;
        t_next = (Cf.residual * Cf.t + ht) / Cf.D;
    }
    Cf.hn = h_next;
    Cf.tn = t_next;
    Cf.border = d.Mb[x] != 0;
    Cf.lava = h_next > 0 && !Cf.border;
    Cf.solid = false;
    Cf.aus = 1.0;
    Cf.st = t_next;
    if (Cf.lava) {
        const double nT = t_next;
        Cf.st = sci_cool(nT, h_next, d.ph.Pepsilon, d.ph.Psigma, d.ph.Pclock, d.ph.Pcool, d.ph.Prho, d.ph.Pcv,
                         d.ph.Pac, &Cf.aus);
        Cf.solid = Cf.st <= d.ph.PTsol;
    }
}

/* the step at one cell, in place (the border reset of the steering last);
 * with a tape slot (entry >= 0) the values its adjoint needs go there */
static __device__ __forceinline__ bool update_cell(const Dev& d, const double* slots, const Inst& I, int i, int j,
                                                   int epoch, const Tape& tp, long long entry)
{
    const long long x = I.off + (long long)i * I.cols + j;
    CellFwd Cf;
    compute_cell(d, slots, I, i, j, x, epoch, Cf);
    if (entry >= 0) {
        tp.cell[entry] = (int)x;
        tp.flag[entry] = (unsigned char)((Cf.flowcond ? E_FLOW : 0) | (Cf.border ? E_BORDER : 0) |
                                         (Cf.lava ? E_LAVA : 0) | (Cf.solid ? E_SOLID : 0));
        const double v[NVAL] = {Cf.t, Cf.tn, Cf.hn, Cf.residual, Cf.D, Cf.aus, Cf.st};
#pragma unroll
        for (int q = 0; q < NVAL; q++)
            tp.val[q * tp.cap + entry] = v[q];
    }
    double sh = Cf.hn, st = Cf.tn;
    if (Cf.lava) {
        st = Cf.st;
        if (Cf.solid) {
            d.Sz[x] = Cf.sz + sh;
            d.Msl[x] = d.Msl[x] + sh;
            sh = 0;
            st = d.ph.PTsol;
        }
    }
    if (Cf.border) {
        sh = 0;
        st = 0;
    }
    d.Slt[x] = sh;
    d.St[x] = st;
    return sh > 0;
}

/* K2: width_update, updateTemperature and the border reset at every lava
 * cell and every receiver (the only cells whose state can change: any
 * other cell has no lava and no inflow, so h + (0 - 0) = h and the
 * temperature stays; border cells hold 0 from the start); one thread per
 * cell over the whole GPU; a cell that still holds lava sets its bit in
 * its tile's mask.  The last block to finish advances the step's
 * counters. */
__global__ void __launch_bounds__(K1T) k_update(const __grid_constant__ Dev d, const __grid_constant__ Tape tp,
                                                int step)
{
    __shared__ long long s_offs[MAX_INST + 1];
    for (int k = threadIdx.x; k <= d.B; k += blockDim.x)
        s_offs[k] = d.offs[k];
    __syncthreads();
    const int epoch = d.counts[6];
    const int nl = min(d.counts[0], d.capacity);
    const int n = nl + min(d.counts[11], d.capacity);
    long long base;
    const double* slots = slots_of(d, tp, nl, &base);
    const bool taped = tp.cap && base + n <= tp.cap;
    const int lane = threadIdx.x & 31;
    const int stride = gridDim.x * blockDim.x;
    for (int k0 = blockIdx.x * blockDim.x; k0 < n; k0 += stride) {
        const int k = k0 + threadIdx.x;
        bool lava = false;
        if (k < n) {
            const int c = k < nl ? d.list[k] : d.rlist[k - nl];
            const Inst I = d.inst[locate(s_offs, d.B, c)];
            const long long lc = c - I.off;
            const int i = (int)(lc / I.cols), j = (int)(lc - (long long)i * I.cols);
            lava = update_cell(d, slots, I, i, j, epoch, tp, taped ? base + k : -1);
            if (lava)
                atomicOr(d.mask + (size_t)(I.tile0 + (i / TH) * I.tiles_x + j / TW) * 16 + (i % TH), 1u << (j % TW));
        }
        const unsigned m = __ballot_sync(0xffffffffu, lava);
        if (m && lane == 0)
            atomicAdd(d.counts + 13, __popc(m));
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(reinterpret_cast<unsigned*>(d.counts + 5), 1u) == gridDim.x - 1) {
            if (tp.cap) {
                tp.step_base[step] = base;
                tp.step_lava[step] = nl;
                tp.step_n[step] = n;
                *tp.used = base + n;
            }
            d.counts[9] += d.counts[7];
            d.counts[0] = 0; /* K0 of the next step collects the list from the masks */
            d.counts[5] = 0;
            d.counts[6] = epoch + 1;
            d.counts[12] = d.counts[7];
            d.counts[7] = 0;
            d.counts[11] = 0;
        }
    }
}

/* ---- adjoint of the final-thickness misfit --------------------------------
 * L = sum over every scenario's cells of (Slt_T - target)^2; gradient with
 * respect to every vent's emission rate of every phase.  The forward's
 * discrete decisions are frozen: the minimisation's elimination sets and the
 * shear-resistance test, whether a cell has any flow, whether it holds lava,
 * whether it solidifies, the border mask.  Reverse mode, step by step from
 * the last, over the step's tape entries, one thread each:
 *   B2 (every entry): mixing and cooling backward, in place on the cell's
 *      own adjoints; keeps, per entry, dL/dh' (A_h), dL/dt' / D (A_t) and
 *      t' for the outflow adjoints;
 *   B1 (lava entries): the adjoint of each outflow gathered from the two
 *      cells it connects, then the minimisation backward to the nine cells
 *      it read: the cell's own adjoints directly, its neighbours' through
 *      one FP64 atomic each onto two sums per cell, of the neighbours across
 *      an edge (H = z + h: dL/dh and dL/dz alike) and across a corner
 *      (dL/dz by 1 / sqrt 2); B2 folds a cell's sums into its adjoints; then, by its last block, the emission backward --
 *      dL/drate += dL/dSlt(vent) * Pclock / Pac for the vent whose emission
 *      took effect, the temperature adjoint of the vent cell reset (the
 *      emission overwrote it).
 * Both are bound by the FP64 pipe, and the entries spread over every SM.
 * The sweep before took the visited tiles as its unit (a block per 32 x 16
 * tile, so that the few hundred tiles left SMs idle) and evaluated the flows
 * twice and the cooling once more per step from a restored state; 16
 * scenarios of 700 x 768, 240 steps: 211 us per step in four kernels (ncu:
 * FP64 pipe 57 % on the 88 SMs with tiles). */
struct __align__(32) Mix {
    double Ah, At, tp, unused;
};
struct Adj {
    double* lh;   /* dense: dL/dSlt */
    double* lt;   /* dense: dL/dSt */
    double* lz;   /* dense: dL/dSz */
    double* side; /* dense: dL/dH from the cells across an edge, */
    double* diag; /* and across a corner, not yet in lh and lz */
    Mix* mix;     /* per entry of the step */
    double* grad; /* nvents x nphases, internal vent order */
};

__global__ void __launch_bounds__(BT) k_bcells(const __grid_constant__ Dev d, const __grid_constant__ Tape tp,
                                               const __grid_constant__ Adj a, long long base, int n, int epoch_b)
{
    const int k = blockIdx.x * BT + threadIdx.x;
    if (k >= n)
        return;
    const long long e = base + k;
    const int x = tp.cell[e];
    const unsigned flag = tp.flag[e];
    const double t = tp.val[e], tn = tp.val[tp.cap + e];
    const double side = a.side[x], diag = a.diag[x];
    const double lh = a.lh[x] + (side + diag), lt = a.lt[x];
    const double lz = a.lz[x] + (side + diag * d.ph.rrad2);
    double Lh = lh, Lt = lt; /* adjoints of h', t' */
    if (flag & E_BORDER) {
        Lh = 0.0;
        Lt = 0.0;
    } else if (flag & E_SOLID) {
        Lh = lz; /* Sz += h' */
        Lt = 0.0;
    } else if (flag & E_LAVA) {
        /* st = t' / aus^(1/3), aus = 1 + q, q = cool3 t'^3 / h' */
        const double hn = tp.val[2 * tp.cap + e], aus = tp.val[5 * tp.cap + e], st = tp.val[6 * tp.cap + e];
        const double rh = 1.0 / hn, rt = 1.0 / tn;
        const double q = d.ph.cool3 * (tn * tn * tn) * rh;
        const double dst_daus = -st / (3.0 * aus);
        Lh = lh - lt * (dst_daus * q * rh);
        Lt = lt * ((st + 3.0 * dst_daus * q) * rt);
    }
    Mix m = {Lh, 0.0, tn, 0.0};
    if (flag & E_FLOW) {
        const double residual = tp.val[3 * tp.cap + e], D = tp.val[4 * tp.cap + e];
        m.At = Lt / D;
        Lh = Lh + m.At * (t - tn);
        Lt = m.At * residual;
    }
    a.side[x] = 0.0;
    a.diag[x] = 0.0;
    a.lz[x] = lz;
    a.lh[x] = Lh;
    a.lt[x] = Lt;
    a.mix[k] = m;
    d.map[x] = make_int2(epoch_b, k);
}

__global__ void __launch_bounds__(BT) k_bflows(const __grid_constant__ Dev d, const __grid_constant__ Tape tp,
                                               const __grid_constant__ Adj a, long long base, int nlava, int epoch_b,
                                               unsigned phase)
{
    extern __shared__ long long s_offs[];
    __shared__ int s_last;
    for (int k = threadIdx.x; k <= d.B; k += BT)
        s_offs[k] = d.offs[k];
    __syncthreads();
    /* the entry's values in one round of loads (the kernel is a chain of
     * them), whether the cell had a flow or not */
    const int k0 = blockIdx.x * BT + threadIdx.x;
    const long long e = base + (k0 < nlava ? k0 : 0);
    const unsigned mask = k0 < nlava ? tp.mask[e] : 0u;
    const int x = tp.cell[e];
    const double t = tp.val[e], Pr = tp.pr[e];
    const Mix me = a.mix[e - base];
    const unsigned F = mask & 511u, S = (mask >> 9) & 511u, inside = mask >> 18;
    if (F) { /* no positive outflow: nothing was moved from the cell */
        const int cols = d.inst[locate(s_offs, d.B, x)].cols;
        const double* f = tp.fc + 16 * (size_t)e - 1; /* f[1..8] */
        const double dlog = d.ph.b * 2.302585092994045684;
        int to[8]; /* the receivers' entries, -1: not in the grid */
#pragma unroll
        for (int k = 1; k < 9; k++) {
            to[k - 1] = -1;
            if ((F >> k) & (inside >> k) & 1u) {
                const int2 m = d.map[x + kMi[k] * cols + kMj[k]];
                if (m.x == epoch_b)
                    to[k - 1] = m.y;
            }
        }
        /* v = dL/df[k] from the cell the flow left and the one it reached;
         * f[k] = Pr(t) (avg - H[k]), avg = (h0 + sum_S H) / |S|, so
         * dPr/dt (avg - H[k]) = b ln(10) f[k].  A loop over the flows there
         * are: a cell has one or two, and all eight directions in turn, in
         * a warp whose cells' flows differ, took 23.1 us a step
         * against 20.9 (16 scenarios of 700 x 768).
         * H[k] = z[k] + h[k] for k >= 1, H[0] = z[0];
         * z[k] = sz0 - (sz0 - sz_k) / rad2 for k >= 5. */
        const double inv = d.ph.rrad2;
        const double left = -me.Ah + me.At * (me.tp - t); /* the outflow's part in this cell */
        double lt_add = 0.0, V = 0.0, corner = 0.0; /* sums of v: all, and across corners */
        for (unsigned todo = F; todo; todo &= todo - 1) {
            const int k = __ffs(todo) - 1;
            const double fk = f[k];
            double v = left, at = 0.0;
            int m = -1;
#pragma unroll
            for (int q = 1; q < 9; q++)
                m = q == k ? to[q - 1] : m;
            if (m >= 0) { /* the receiver's inflow, and its heat term f * t */
                const Mix r = a.mix[m];
                v += r.Ah + r.At * (t - r.tp);
                at = r.At;
            }
            if ((inside >> k) & 1u)
                atomicAdd((k < 5 ? a.side : a.diag) + x + kMi[k] * cols + kMj[k], -(v * Pr));
            V += v;
            if (k >= 5)
                corner += v;
            lt_add += (v * dlog + at) * fk;
        }
        const double g = cal_div_small(V * Pr, __popc(S));
        for (unsigned todo = S & inside & 0x1feu; todo && g != 0.0; todo &= todo - 1) {
            const int k = __ffs(todo) - 1;
            atomicAdd((k < 5 ? a.side : a.diag) + x + kMi[k] * cols + kMj[k], g);
        }
        const double corners = g * (double)__popc(S >> 5) - corner * Pr;
        const double lz_own = ((S & 1u) ? g : 0.0) + corners * (1.0 - inv);
        /* no other thread of the launch touches these */
        a.lh[x] += g; /* avg's h[0] */
        a.lt[x] += lt_add;
        a.lz[x] += lz_own;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(reinterpret_cast<unsigned*>(d.counts + 5), 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last)
        return;
    __threadfence();
    for (int q = threadIdx.x; q < d.ngroups; q += BT) {
        const int eff = phase < (unsigned)d.nphases ? d.g_eff[(size_t)q * d.nphases + phase] : -1;
        if (eff >= 0) {
            const int c = d.g_cell[q];
            const double lh = __ldcg(a.lh + c) + (__ldcg(a.side + c) + __ldcg(a.diag + c));
            a.grad[(size_t)eff * d.nphases + phase] += lh * d.ph.Pclock / d.ph.Pac;
            a.lt[c] = 0.0;
        }
    }
    if (threadIdx.x == 0)
        d.counts[5] = 0;
}

/* dL/dSlt_T = 2 (Slt_T - target), the other adjoints 0; per-scenario loss.
 * A block takes one run of consecutive cells, so that a warp's cells are of
 * one scenario but where two meet: its sum is kept in registers and added
 * to the scenario's loss when the scenario changes (one atomic per cell
 * queued them all on a few words: 8.6M cells 1.30 ms). */
__global__ void __launch_bounds__(T) k_bloss(const __grid_constant__ Dev d, const __grid_constant__ Adj a,
                                             const double* tgt, double* loss)
{
    extern __shared__ long long s_offs[];
    for (int k = threadIdx.x; k <= d.B; k += blockDim.x)
        s_offs[k] = d.offs[k];
    __syncthreads();
    const long long per = ((d.ncells + gridDim.x - 1) / gridDim.x + T - 1) / T * T;
    const long long c1 = min(d.ncells, per * (blockIdx.x + 1));
    double acc = 0.0;
    int cur = -1; /* the scenario acc belongs to, the same in every lane */
    auto flush = [&]() {
        double v = acc;
        for (int o = 16; o > 0; o >>= 1)
            v += __shfl_down_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0 && cur >= 0 && v != 0.0)
            atomicAdd(loss + cur, v);
        acc = 0.0;
    };
    for (long long c0 = per * blockIdx.x; c0 < c1; c0 += T) {
        const long long c = c0 + threadIdx.x;
        int b = -1;
        double diff = 0.0;
        if (c < c1) {
            b = locate(s_offs, d.B, c);
            if (c - s_offs[b] < (long long)d.inst[b].rows * d.inst[b].cols)
                diff = d.Slt[c] - tgt[c];
            a.lh[c] = 2.0 * diff;
            a.lt[c] = 0.0;
            a.lz[c] = 0.0;
            a.side[c] = 0.0;
            a.diag[c] = 0.0;
        }
        const int b0 = __shfl_sync(0xffffffffu, b, 0);
        if (__all_sync(0xffffffffu, b == b0 || b < 0)) {
            if (b0 >= 0 && b0 != cur) {
                flush();
                cur = b0;
            }
            acc += diff * diff;
        } else if (b >= 0 && diff != 0.0) {
            atomicAdd(loss + b, diff * diff);
        }
    }
    flush();
}

/* MakeBorder (Sciara.cpp:206-250) on the device, the border reset of the
 * initial state, and the first lava list */
__global__ void k_prime(const __grid_constant__ Dev d)
{
    __shared__ long long s_offs[MAX_INST + 1];
    for (int k = threadIdx.x; k <= d.B; k += blockDim.x)
        s_offs[k] = d.offs[k];
    __syncthreads();
    unsigned char* Mb = const_cast<unsigned char*>(d.Mb);
    for (long long c0 = (long long)blockIdx.x * blockDim.x; c0 < d.ncells; c0 += (long long)gridDim.x * blockDim.x) {
        const long long c = c0 + threadIdx.x;
        bool lava = false;
        if (c < d.ncells) {
            const Inst I = d.inst[locate(s_offs, d.B, c)];
            const long long lc = c - I.off;
            if (lc < (long long)I.rows * I.cols) {
                const int i = (int)(lc / I.cols), j = (int)(lc - (long long)i * I.cols);
                bool border = false;
                if (d.Sz[c] >= 0) {
                    if (i == 0 || i == I.rows - 1 || j == 0 || j == I.cols - 1) {
                        border = true;
                    } else {
                        for (int k = 1; k < 9 && !border; k++) {
                            long long cn;
                            if (nbr(I, i, j, k, &cn) && d.Sz[cn] < 0)
                                border = true;
                        }
                    }
                }
                Mb[c] = border ? 1 : 0;
                if (border) {
                    d.Slt[c] = 0;
                    d.St[c] = 0;
                } else if (cal_d2i(d.Slt[c]) == (long long)0x8000000000000000LL) {
                    d.Slt[c] = 0; /* -0 thickness: the first update would make it +0 */
                }
                lava = !border && d.Slt[c] > 0;
            } else {
                Mb[c] = 0;
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, lava);
        if (m) {
            const int lane = threadIdx.x & 31;
            int base = 0;
            if (lane == 0)
                base = atomicAdd(d.counts + 0, __popc(m));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (lava) {
                const int pos = base + __popc(m & ((1u << lane) - 1u));
                if (pos < d.capacity)
                    d.list[pos] = (int)c;
                else
                    atomicExch(d.counts + 8, 1);
            }
        }
    }
}

struct Batch {
    int B = 0, nvents = 0, nphases = 0;
    unsigned emission_time = 0;
    long long N = 0;
    int ntiles = 0, capacity = 0;
    std::vector<Inst> inst;
    std::vector<long long> offs;
    Dev d;
    double effusion_duration = 0;
    std::vector<int> vent_order; /* internal vent k -> the caller's vent index */
    double *Sz0 = nullptr, *Slt0 = nullptr, *St0 = nullptr; /* the initial state, for every run */
    cudaStream_t st = nullptr;
    void* allocs[32] = {};
    int nalloc = 0;
    bool primed = false;
    /* loss_grad's workspace: kept for the next call while what all handles
     * keep is a small part of the device's memory (keep_work) */
    Tape tp = {};
    Adj adj = {};
    double* tgt = nullptr;  /* target, padded layout */
    double* loss = nullptr; /* B */
    int tape_steps = 0, mix_cap = 0;
    long long tape_limit = 0; /* entries; 0: none */
    long long kept = 0;       /* bytes of the workspace in g_kept */
};

template <typename T>
static bool dalloc(Batch& bt, T** p, size_t bytes)
{
    if (bt.nalloc >= (int)(sizeof(bt.allocs) / sizeof(bt.allocs[0])) || cudaMalloc(p, bytes) != cudaSuccess)
        return false;
    bt.allocs[bt.nalloc++] = *p;
    return true;
}

template <typename T>
static bool walloc(T** p, size_t count)
{
    if (*p)
        return true;
    if (cudaMalloc(p, std::max<size_t>(1, count) * sizeof(T)) == cudaSuccess)
        return true;
    (void)cudaGetLastError();
    *p = nullptr;
    return false;
}

template <typename T>
static void wfree(T** p)
{
    cudaFree(*p);
    *p = nullptr;
}

static void free_tape(Batch& bt)
{
    Tape& tp = bt.tp;
    wfree(&tp.cell);
    wfree(&tp.mask);
    wfree(&tp.flag);
    wfree(&tp.pr);
    wfree(&tp.fc);
    wfree(&tp.val);
    tp.cap = 0;
}

/* a tape for `entries` entries (kept when it is large enough already); false
 * when that is more than the caller allows or the memory holds (what there
 * was is then given up in the second case) */
static bool grow_tape(Batch& bt, long long entries)
{
    Tape& tp = bt.tp;
    if (tp.cap >= entries)
        return true;
    if (bt.tape_limit > 0 && entries > bt.tape_limit)
        return false;
    free_tape(bt);
    const size_t n = (size_t)entries;
    if (walloc(&tp.cell, n) && walloc(&tp.mask, n) && walloc(&tp.flag, n) && walloc(&tp.pr, n) &&
        walloc(&tp.fc, 16 * n) && walloc(&tp.val, NVAL * n)) {
        tp.cap = entries;
        return true;
    }
    free_tape(bt);
    return false;
}

static std::atomic<long long> g_kept{0}; /* bytes that handles keep between calls */

static void free_work(Batch& bt)
{
    free_tape(bt);
    wfree(&bt.tp.used);
    wfree(&bt.tp.step_base);
    wfree(&bt.tp.step_lava);
    wfree(&bt.tp.step_n);
    wfree(&bt.adj.lh);
    wfree(&bt.adj.lt);
    wfree(&bt.adj.lz);
    wfree(&bt.adj.side);
    wfree(&bt.adj.diag);
    wfree(&bt.adj.mix);
    wfree(&bt.adj.grad);
    wfree(&bt.tgt);
    wfree(&bt.loss);
    bt.tape_steps = bt.mix_cap = 0;
    g_kept -= bt.kept;
    bt.kept = 0;
}

/* the workspace stays for the next call while those of all handles together
 * take at most a sixteenth of the device's memory; else it is given back */
static void keep_work(Batch& bt)
{
    size_t free_b = 0, total_b = 0;
    cudaMemGetInfo(&free_b, &total_b);
    const long long bytes = bt.tp.cap * (long long)ENTRY_BYTES + (long long)sizeof(double) * 6 * bt.N +
                            (long long)sizeof(Mix) * bt.mix_cap;
    const long long before = g_kept.fetch_add(bytes - bt.kept);
    const long long all = before + bytes - bt.kept;
    bt.kept = bytes;
    if (all > (long long)(total_b / 16)) {
        cudaStreamSynchronize(bt.st);
        free_work(bt);
    }
}

static void destroy(Batch* bt)
{
    if (bt->st)
        cudaStreamSynchronize(bt->st);
    free_work(*bt);
    for (int k = 0; k < bt->nalloc; k++)
        cudaFree(bt->allocs[k]);
    if (bt->st)
        cudaStreamDestroy(bt->st);
    delete bt;
}

} // namespace sci2

using sci2::Batch;

/* Create B SCIARA-fv2 scenarios.  dims: 2B ints (rows, cols); z0, slt0, st0:
 * the scenarios' morphology, initial thickness and temperature back to back
 * (unpadded, row-major; slt0 / st0 may be NULL for zero); params: the 13
 * physical parameters (Pclock, PTsol, PTvent, Pr(Tsol), Pr(Tvent),
 * Phc(Tsol), Phc(Tvent), Pcool, Prho, Pepsilon, Psigma, Pcv, Pc); vents:
 * vent_inst[v] = scenario, vent_xy[2v..2v+1] = (x, y), in each scenario's
 * vent order; rates: nvents x nphases m^3/s, each phase emission_time
 * seconds.  list_fraction: lava-list capacity as a fraction of all cells,
 * or <= 0 for the default (all cells up to 16M cells, an eighth beyond); a
 * run that needs more reports CAL_ERROR_OUT_OF_MEMORY. */
extern "C" void* cal_sciara_batch_create(int B, const int* dims, const double* z0, const double* slt0,
                                         const double* st0, const double* params, int nvents, const int* vent_inst,
                                         const int* vent_xy, unsigned emission_time, int nphases, const double* rates,
                                         double list_fraction)
{
    if (B <= 0 || B > sci2::MAX_INST || nvents < 0 || nphases < 0 || emission_time == 0)
        return nullptr;
    Batch* bt = new Batch();
    bt->B = B;
    bt->nvents = nvents;
    bt->nphases = nphases;
    bt->emission_time = emission_time;
    bt->offs.assign(B + 1, 0);
    int tiles = 0;
    for (int b = 0; b < B; b++) {
        sci2::Inst I;
        memset(&I, 0, sizeof(I));
        I.rows = dims[2 * b];
        I.cols = dims[2 * b + 1];
        if (I.rows < 3 || I.cols < 3) {
            delete bt;
            return nullptr;
        }
        I.off = bt->offs[b];
        I.tiles_x = (I.cols + sci2::TW - 1) / sci2::TW;
        I.tiles_y = (I.rows + sci2::TH - 1) / sci2::TH;
        I.tile0 = tiles;
        tiles += I.tiles_x * I.tiles_y;
        bt->inst.push_back(I);
        const long long n = (long long)I.rows * I.cols;
        bt->offs[b + 1] = bt->offs[b] + (n + 31) / 32 * 32;
    }
    bt->N = bt->offs[B];
    bt->ntiles = tiles;
    /* default (list_fraction <= 0): every cell up to 16M cells, an eighth
     * beyond (lava covers a small part of a large volcano) */
    if (list_fraction <= 0)
        list_fraction = bt->N <= (16LL << 20) ? 1.0 : 0.125;
    const double frac = list_fraction > 1.0 ? 1.0 : list_fraction;
    bt->capacity = (int)std::min<long long>(bt->N, std::max<long long>(1024, (long long)(frac * bt->N)));
    /* vents: packed cell indices, grouped by scenario in the given order */
    std::vector<int> vcell(nvents), vfirst(B + 1, 0);
    std::vector<double> vrates((size_t)nvents * nphases);
    {
        std::vector<int> order(nvents);
        for (int v = 0; v < nvents; v++)
            order[v] = v;
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return vent_inst[a] < vent_inst[b]; });
        bt->vent_order = order;
        for (int k = 0; k < nvents; k++) {
            const int v = order[k];
            const int b = vent_inst[v];
            const int x = vent_xy[2 * v], y = vent_xy[2 * v + 1];
            if (b < 0 || b >= B || x < 0 || y < 0 || x >= bt->inst[b].cols || y >= bt->inst[b].rows) {
                delete bt;
                return nullptr;
            }
            vcell[k] = (int)(bt->inst[b].off + (long long)y * bt->inst[b].cols + x);
            vfirst[b + 1]++;
            for (int p = 0; p < nphases; p++)
                vrates[(size_t)k * nphases + p] = rates[(size_t)v * nphases + p];
        }
        for (int b = 0; b < B; b++)
            vfirst[b + 1] += vfirst[b];
    }
    /* vent cells (groups) with, per phase, the vent that takes effect */
    std::vector<int> g_cell, g_member, g_mfirst(1, 0), g_eff;
    std::vector<double> g_emit;
    {
        const double Pac = params[12] * params[12], Pclock = params[0];
        for (int b = 0; b < B; b++)
            for (int v = vfirst[b]; v < vfirst[b + 1]; v++) {
                bool lead = true;
                for (int w = vfirst[b]; w < v; w++)
                    if (vcell[w] == vcell[v])
                        lead = false;
                if (!lead)
                    continue;
                g_cell.push_back(vcell[v]);
                for (int w = v; w < vfirst[b + 1]; w++)
                    if (vcell[w] == vcell[v])
                        g_member.push_back(w);
                g_mfirst.push_back((int)g_member.size());
                for (int p = 0; p < nphases; p++) {
                    int eff = -1;
                    double e = 0.0;
                    for (int m = g_mfirst[g_mfirst.size() - 2]; m < g_mfirst.back(); m++) {
                        /* updateVentsEmission's thickness, rate / Pac * Pclock */
                        const double em = vrates[(size_t)g_member[m] * nphases + p] / Pac * Pclock;
                        if (em > 0) {
                            eff = g_member[m];
                            e = em;
                        }
                    }
                    g_eff.push_back(eff);
                    g_emit.push_back(e);
                }
            }
    }
    const int ngroups = (int)g_cell.size();
    sci2::Dev& d = bt->d;
    memset(&d, 0, sizeof(d));
    d.B = B;
    d.ncells = bt->N;
    d.capacity = bt->capacity;
    d.nphases = nphases;
    d.emission_time = emission_time;
    d.ph.Pclock = params[0];
    d.ph.PTsol = params[1];
    d.ph.PTvent = params[2];
    const double Pr_Tsol = params[3], Pr_Tvent = params[4], Phc_Tsol = params[5], Phc_Tvent = params[6];
    d.ph.Pcool = params[7];
    d.ph.Prho = params[8];
    d.ph.Pepsilon = params[9];
    d.ph.Psigma = params[10];
    d.ph.Pcv = params[11];
    d.ph.Pc = params[12];
    d.ph.Pac = d.ph.Pc * d.ph.Pc;
    d.ph.rad2 = sqrt(2.0);
    d.ph.rrad2 = 1.0 / d.ph.rad2;
    d.ph.rad2_recip = cal_recip_exact_ok(d.ph.rad2, d.ph.rrad2) ? 1 : 0;
    d.ph.w2 = d.ph.Pc * d.ph.Pc;
    d.ph.cool3 = 3.0 * d.ph.Pepsilon * d.ph.Psigma * d.ph.Pclock * d.ph.Pcool / (d.ph.Prho * d.ph.Pcv * d.ph.Pac);
    /* evaluatePowerLawParams (Sciara.cpp:199-204), C library log10 */
    d.ph.b = (log10(Pr_Tvent) - log10(Pr_Tsol)) / (d.ph.PTvent - d.ph.PTsol);
    d.ph.a = log10(Pr_Tsol) - d.ph.b * (d.ph.PTsol);
    d.ph.d = (log10(Phc_Tvent) - log10(Phc_Tsol)) / (d.ph.PTvent - d.ph.PTsol);
    d.ph.c = log10(Phc_Tsol) - d.ph.d * (d.ph.PTsol);
    bt->effusion_duration = (double)emission_time * nphases;

    const size_t nb = (size_t)bt->N * sizeof(double);
    bool ok = cudaStreamCreateWithFlags(&bt->st, cudaStreamNonBlocking) == cudaSuccess &&
              sci2::dalloc(*bt, (sci2::Inst**)&d.inst, sizeof(sci2::Inst) * B) &&
              sci2::dalloc(*bt, (long long**)&d.offs, sizeof(long long) * (B + 1)) &&
              sci2::dalloc(*bt, &d.Sz, nb) && sci2::dalloc(*bt, &d.Slt, nb) && sci2::dalloc(*bt, &d.St, nb) &&
              sci2::dalloc(*bt, &d.Msl, nb) && sci2::dalloc(*bt, (unsigned char**)&d.Mb, (size_t)bt->N) &&
              sci2::dalloc(*bt, &d.map, sizeof(int2) * (size_t)bt->N) &&
              sci2::dalloc(*bt, &d.fmask, (size_t)bt->N) &&
              sci2::dalloc(*bt, &d.recv, sizeof(int) * (size_t)bt->N) &&
              sci2::dalloc(*bt, &d.rlist, sizeof(int) * (size_t)bt->capacity) &&
              sci2::dalloc(*bt, &d.list, sizeof(int) * (size_t)bt->capacity) &&
              sci2::dalloc(*bt, &d.mask, sizeof(unsigned) * 16 * (size_t)tiles) &&
              sci2::dalloc(*bt, &d.fc, sizeof(double) * 16 * (size_t)bt->capacity) &&
              sci2::dalloc(*bt, &d.counts, 16 * sizeof(int)) &&
              sci2::dalloc(*bt, &d.tflag, sizeof(int) * (size_t)tiles) &&
              sci2::dalloc(*bt, &d.tlist, sizeof(int) * (size_t)tiles) &&
              sci2::dalloc(*bt, (int**)&d.g_cell, sizeof(int) * std::max(1, ngroups)) &&
              sci2::dalloc(*bt, (int**)&d.g_eff, sizeof(int) * std::max<size_t>(1, g_eff.size())) &&
              sci2::dalloc(*bt, (double**)&d.g_emit, sizeof(double) * std::max<size_t>(1, g_emit.size())) &&
              sci2::dalloc(*bt, &bt->Sz0, nb) && sci2::dalloc(*bt, &bt->Slt0, nb) && sci2::dalloc(*bt, &bt->St0, nb);
    if (!ok) {
        fprintf(stderr, "opencal-gb300: cal_sciara_batch_create: out of device memory\n");
        sci2::destroy(bt);
        return nullptr;
    }
    cudaMemcpy((void*)d.inst, bt->inst.data(), sizeof(sci2::Inst) * B, cudaMemcpyHostToDevice);
    cudaMemcpy((void*)d.offs, bt->offs.data(), sizeof(long long) * (B + 1), cudaMemcpyHostToDevice);
    d.ngroups = ngroups;
    if (nvents) {
        cudaMemcpy((void*)d.g_cell, g_cell.data(), sizeof(int) * ngroups, cudaMemcpyHostToDevice);
        if (!g_eff.empty()) {
            cudaMemcpy((void*)d.g_eff, g_eff.data(), sizeof(int) * g_eff.size(), cudaMemcpyHostToDevice);
            cudaMemcpy((void*)d.g_emit, g_emit.data(), sizeof(double) * g_emit.size(), cudaMemcpyHostToDevice);
        }
    }
    cudaMemset(d.Sz, 0, nb);
    cudaMemset(d.Slt, 0, nb);
    cudaMemset(d.St, 0, nb);
    cudaMemset(d.Msl, 0, nb);
    size_t src = 0;
    for (int b = 0; b < B; b++) {
        const size_t n = (size_t)bt->inst[b].rows * bt->inst[b].cols;
        const long long o = bt->offs[b];
        cudaMemcpy(d.Sz + o, z0 + src, n * sizeof(double), cudaMemcpyHostToDevice);
        if (slt0)
            cudaMemcpy(d.Slt + o, slt0 + src, n * sizeof(double), cudaMemcpyHostToDevice);
        if (st0)
            cudaMemcpy(d.St + o, st0 + src, n * sizeof(double), cudaMemcpyHostToDevice);
        src += n;
    }
    cudaMemcpy(bt->Sz0, d.Sz, nb, cudaMemcpyDeviceToDevice);
    cudaMemcpy(bt->Slt0, d.Slt, nb, cudaMemcpyDeviceToDevice);
    cudaMemcpy(bt->St0, d.St, nb, cudaMemcpyDeviceToDevice);
    if (cudaGetLastError() != cudaSuccess) {
        sci2::destroy(bt);
        return nullptr;
    }
    return bt;
}

extern "C" void cal_sciara_batch_destroy(void* handle)
{
    if (handle)
        sci2::destroy((Batch*)handle);
}

namespace sci2 {

/* the run from the initial state: calRun2D's loop with the stop condition
 * of Sciara.cpp:177-183 (elapsed time >= emission's end).  With a tape the
 * entries of the steps from taped_from on are kept. */
static int forward(Batch* bt, int max_steps, const Tape* tape, int taped_from, std::vector<double>* elapsed_of,
                   int* steps_done, float* ms)
{
    Dev& d = bt->d;
    cudaStream_t st = bt->st;
    const size_t nb = (size_t)bt->N * sizeof(double);
    cudaMemcpyAsync(d.Sz, bt->Sz0, nb, cudaMemcpyDeviceToDevice, st);
    cudaMemcpyAsync(d.Slt, bt->Slt0, nb, cudaMemcpyDeviceToDevice, st);
    cudaMemcpyAsync(d.St, bt->St0, nb, cudaMemcpyDeviceToDevice, st);
    cudaMemsetAsync(d.Msl, 0, nb, st);
    cudaMemsetAsync(d.counts, 0, 16 * sizeof(int), st);
    cudaMemsetAsync(d.map, 0, sizeof(int2) * (size_t)bt->N, st);
    cudaMemsetAsync(d.recv, 0, sizeof(int) * (size_t)bt->N, st);
    cudaMemsetAsync(d.mask, 0, sizeof(unsigned) * 16 * (size_t)bt->ntiles, st);
    cudaMemsetAsync(d.tflag, 0, sizeof(int) * (size_t)bt->ntiles, st);
    const int one = 1;
    cudaMemcpyAsync(d.counts + 6, &one, sizeof(int), cudaMemcpyHostToDevice, st);
    int blocks = (int)std::min<long long>((bt->N + T - 1) / T, 152 * 16);
    k_prime<<<blocks, T, 0, st>>>(d);
    const Tape none = {};
    if (tape)
        cudaMemsetAsync(tape->used, 0, sizeof(long long), st);
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, st);
    double elapsed = 0.0;
    int done = 0;
    for (int step = 1; max_steps <= 0 || step <= max_steps; step++) {
        if (elapsed_of)
            elapsed_of->push_back(elapsed);
        /* the phase as the vent process forms it: (unsigned)(elapsed / emission_time) */
        const unsigned phase = (unsigned)(elapsed / (double)bt->emission_time);
        const Tape& tp = tape && done >= taped_from ? *tape : none;
        k_collect<<<K2_BLOCKS, T, 0, st>>>(d, phase, done > 0);
        k_flows<<<152 * 32, K1T, 0, st>>>(d, tp);
        k_update<<<152 * 32, K1T, 0, st>>>(d, tp, done);
        done++;
        elapsed += d.ph.Pclock;
        if (elapsed >= bt->effusion_duration)
            break;
    }
    cudaEventRecord(e1, st);
    cudaEventSynchronize(e1);
    float t = 0.f;
    cudaEventElapsedTime(&t, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (ms)
        *ms = t;
    if (steps_done)
        *steps_done = done;
    int overflow = 0;
    cudaMemcpy(&overflow, d.counts + 8, sizeof(overflow), cudaMemcpyDeviceToHost);
    if (cudaGetLastError() != cudaSuccess)
        return 3; /* CAL_ERROR_CUDA */
    return overflow ? 2 /* CAL_ERROR_OUT_OF_MEMORY: lava list too small */ : 0;
}

/* steps a run takes (the stop condition's accumulation of the clock) */
static int run_length(const Batch* bt, int max_steps)
{
    double elapsed = 0.0;
    int done = 0;
    for (int step = 1; max_steps <= 0 || step <= max_steps; step++) {
        done++;
        elapsed += bt->d.ph.Pclock;
        if (elapsed >= bt->effusion_duration)
            break;
    }
    return done;
}

} // namespace sci2

/* Run every scenario from its initial state (as created) until the emission ends (or
 * max_steps > 0 steps); the state stays on the device for
 * cal_sciara_batch_read.  steps_done: steps run; ms: device time of the step
 * loop.  0, or a CALError code (CAL_ERROR_OUT_OF_MEMORY = list overflow). */
extern "C" int cal_sciara_batch_run(void* handle, int max_steps, int* steps_done, float* ms)
{
    return sci2::forward((Batch*)handle, max_steps, nullptr, 0, nullptr, steps_done, ms);
}

namespace sci2 {

/* tape entries a run is first given room for: a vent's lava spreads over
 * some 15 cells more each step (10..50 m3/s on 10 m cells), half as many
 * again for receivers and slower lava, at most a quarter of the free memory;
 * a run that visits more is repeated with the size it asked for */
static long long first_tape(const Batch& bt, int steps)
{
    long long sum = 0;
    for (int t = 1; t <= steps; t++)
        sum += std::min<long long>(bt.N, 64 + 24LL * std::max(1, bt.nvents) * t);
    size_t free_b = 0, total_b = 0;
    cudaMemGetInfo(&free_b, &total_b);
    sum = std::max<long long>(4096, std::min<long long>(sum, (long long)(free_b / 4 / ENTRY_BYTES)));
    return bt.tape_limit > 0 ? std::min(sum, bt.tape_limit) : sum;
}

static int loss_grad(Batch* bt, const double* target, int max_steps, double* loss_out, double* grad_out,
                     int* steps_done, long long tape_slots, float* ms, cudaEvent_t e0, cudaEvent_t e1)
{
    constexpr int OOM = 2, CUDA = 3; /* CAL_ERROR_OUT_OF_MEMORY, CAL_ERROR_CUDA */
    Dev& d = bt->d;
    Tape& tp = bt->tp;
    Adj& a = bt->adj;
    cudaStream_t st = bt->st;
    const int steps = run_length(bt, max_steps);
    const size_t ngrad = (size_t)std::max(1, bt->nvents * bt->nphases);
    if (steps > bt->tape_steps) {
        wfree(&tp.step_base);
        wfree(&tp.step_lava);
        wfree(&tp.step_n);
        bt->tape_steps = steps;
    }
    if (!walloc(&tp.used, 1) || !walloc(&tp.step_base, (size_t)bt->tape_steps) ||
        !walloc(&tp.step_lava, (size_t)bt->tape_steps) || !walloc(&tp.step_n, (size_t)bt->tape_steps) ||
        !walloc(&bt->tgt, (size_t)bt->N) || !walloc(&bt->loss, (size_t)bt->B) || !walloc(&a.lh, (size_t)bt->N) ||
        !walloc(&a.lt, (size_t)bt->N) || !walloc(&a.lz, (size_t)bt->N) ||
        !walloc(&a.side, (size_t)bt->N) || !walloc(&a.diag, (size_t)bt->N) || !walloc(&a.grad, ngrad))
        return OOM;
    if (!tp.cap && !grow_tape(*bt, first_tape(*bt, steps)) && !grow_tape(*bt, 1))
        return OOM;
    /* target in the padded layout: an input, copied before the timed region */
    cudaMemsetAsync(bt->tgt, 0, (size_t)bt->N * sizeof(double), st);
    size_t src = 0;
    for (int b = 0; b < bt->B; b++) {
        const size_t n = (size_t)bt->inst[b].rows * bt->inst[b].cols;
        cudaMemcpyAsync(bt->tgt + bt->offs[b], target + src, n * sizeof(double), cudaMemcpyHostToDevice, st);
        src += n;
    }
    std::vector<double> elapsed_of;
    std::vector<int> n;
    int done = 0;
    long long need = 0;
    for (int attempt = 0;; attempt++) {
        elapsed_of.clear();
        cudaEventRecord(e0, st);
        const int rc = forward(bt, max_steps, &tp, 0, &elapsed_of, &done, nullptr);
        if (rc)
            return rc;
        int tiles = 0;
        n.resize(done);
        cudaMemcpy(&need, tp.used, sizeof(need), cudaMemcpyDeviceToHost);
        cudaMemcpy(&tiles, d.counts + 9, sizeof(tiles), cudaMemcpyDeviceToHost);
        cudaMemcpy(n.data(), tp.step_n, sizeof(int) * done, cudaMemcpyDeviceToHost);
        if (tape_slots > 0 && tiles > tape_slots)
            return OOM; /* the caller's limit */
        if (need <= tp.cap || attempt || !grow_tape(*bt, need))
            break;
    }
    const int most = std::max(1, *std::max_element(n.begin(), n.end()));
    if (most > bt->mix_cap) {
        wfree(&a.mix);
        bt->mix_cap = 0;
        if (!walloc(&a.mix, (size_t)most))
            return OOM;
        bt->mix_cap = most;
    }
    /* A run whose tape does not fit is taped and swept a stretch of steps at
     * a time, the last first, each after a forward to its end (no state is
     * kept: a tape of half the size costs two and a half forwards more) */
    const bool stretches = need > tp.cap;
    if (stretches) {
        long long entries = need;
        while (entries > most && !grow_tape(*bt, entries))
            entries /= 2;
        if (!grow_tape(*bt, std::max<long long>(most, entries)))
            return OOM;
    }
    cudaMemsetAsync(bt->loss, 0, sizeof(double) * bt->B, st);
    cudaMemsetAsync(a.grad, 0, sizeof(double) * ngrad, st);
    const size_t offs_bytes = sizeof(long long) * (bt->B + 1);
    std::vector<long long> base(done);
    std::vector<int> nlava(done);
    for (int t1 = done, t0; t1 > 0; t1 = t0) {
        t0 = 0;
        if (stretches) {
            long long room = tp.cap;
            for (t0 = t1; t0 > 0 && n[t0 - 1] <= room; t0--)
                room -= n[t0 - 1];
            const int rc = forward(bt, t1, &tp, t0, nullptr, nullptr, nullptr);
            if (rc)
                return rc;
        }
        if (t1 == done)
            k_bloss<<<(int)std::min<long long>((bt->N + T - 1) / T, 152 * 8), T, offs_bytes, st>>>(d, a, bt->tgt,
                                                                                                   bt->loss);
        cudaMemcpyAsync(&base[t0], tp.step_base + t0, sizeof(long long) * (t1 - t0), cudaMemcpyDeviceToHost, st);
        cudaMemcpyAsync(&nlava[t0], tp.step_lava + t0, sizeof(int) * (t1 - t0), cudaMemcpyDeviceToHost, st);
        cudaStreamSynchronize(st);
        for (int t = t1 - 1; t >= t0; t--) {
            const int epoch_b = -(t + 1);
            const unsigned phase = (unsigned)(elapsed_of[t] / bt->emission_time);
            if (n[t] > 0)
                k_bcells<<<(n[t] + BT - 1) / BT, BT, 0, st>>>(d, tp, a, base[t], n[t], epoch_b);
            /* an emitting vent cell is a lava cell of the step */
            if (nlava[t] > 0)
                k_bflows<<<(nlava[t] + BT - 1) / BT, BT, offs_bytes, st>>>(d, tp, a, base[t], nlava[t], epoch_b,
                                                                           phase);
        }
    }
    cudaEventRecord(e1, st);
    if (stretches) { /* the run's final state */
        const int rc = forward(bt, max_steps, nullptr, 0, nullptr, nullptr, nullptr);
        if (rc)
            return rc;
    }
    std::vector<double> grad(ngrad);
    cudaMemcpyAsync(grad.data(), a.grad, sizeof(double) * ngrad, cudaMemcpyDeviceToHost, st);
    if (loss_out)
        cudaMemcpyAsync(loss_out, bt->loss, sizeof(double) * bt->B, cudaMemcpyDeviceToHost, st);
    cudaStreamSynchronize(st);
    if (ms)
        cudaEventElapsedTime(ms, e0, e1);
    if (steps_done)
        *steps_done = done;
    if (grad_out)
        for (int k = 0; k < bt->nvents; k++)
            for (int p = 0; p < bt->nphases; p++)
                grad_out[(size_t)bt->vent_order[k] * bt->nphases + p] = grad[(size_t)k * bt->nphases + p];
    return cudaGetLastError() == cudaSuccess ? 0 : CUDA;
}

} // namespace sci2

/* The most entries that loss_grad's tape may hold (0, the default: as many as
 * the device memory holds); runs that need more are taped in stretches. */
extern "C" int cal_sciara_batch_set_tape_limit(void* handle, long long entries)
{
    Batch* bt = (Batch*)handle;
    if (entries < 0)
        return 1; /* CAL_ERROR_INVALID_ARGUMENT */
    bt->tape_limit = entries;
    if (entries > 0 && bt->tp.cap > entries) {
        cudaStreamSynchronize(bt->st);
        sci2::free_tape(*bt);
    }
    return 0;
}

/* Loss L_b = sum over scenario b of (Slt_T - target)^2 and its gradient
 * with respect to every emission rate, by the adjoint with the forward's
 * decisions frozen.  target: host array, the scenarios' grids back to back
 * (unpadded); loss_out[B]; grad_out[nvents x nphases] in the caller's vent
 * order.  tape_slots: a limit on the tiles flagged, summed over the steps
 * (0: none); a run that flags more is an error.  The tape grows to the run:
 * when it proves too small the forward runs once more with a tape of the
 * size it asked for, and where that does not fit the steps are taped and
 * swept in stretches.  The state after the call is the run's final one.  0
 * or a CALError code; ms: device time of forward + adjoint. */
extern "C" int cal_sciara_batch_loss_grad(void* handle, const double* target, int max_steps, double* loss_out,
                                          double* grad_out, int* steps_done, long long tape_slots, float* ms)
{
    Batch* bt = (Batch*)handle;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int rc = sci2::loss_grad(bt, target, max_steps, loss_out, grad_out, steps_done, tape_slots, ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) {
        cudaStreamSynchronize(bt->st);
        sci2::free_work(*bt);
    } else {
        sci2::keep_work(*bt);
    }
    return rc;
}

namespace sci2 {

/* Host pages under a result, before the copy into it.  Pages of a freshly
 * allocated array do not exist yet; when the device's copy is the first to
 * touch them, each fault is a round trip of the GPU to the operating system
 * (134 MB: 37-72 ms), while a few host threads map them in a fraction of
 * that.  Every byte written here is overwritten by the copy. */
static void touch_pages(void* dst, size_t bytes)
{
    /* the C library keeps freed blocks below 32 MB mapped for reuse, larger
     * ones come fresh from the system every time */
    constexpr size_t STEP = 4096, MIN_BYTES = 32u << 20;
    const int nthreads = 4;
    if (bytes < MIN_BYTES)
        return;
    volatile char* p = (volatile char*)dst;
    auto share = [=](int k, int n) {
        for (size_t q = bytes / n * k; q < (k + 1 == n ? bytes : bytes / n * (k + 1)); q += STEP)
            p[q] = 0;
    };
    std::vector<std::thread> others;
    int started = 1;
    try {
        others.reserve(nthreads - 1);
        for (; started < nthreads; started++)
            others.emplace_back(share, started, nthreads);
    } catch (...) { /* no more threads: the rest here */
    }
    share(0, nthreads);
    for (int k = started; k < nthreads; k++)
        share(k, nthreads);
    for (std::thread& t : others)
        t.join();
}

} // namespace sci2

/* the scenarios' final Sz, Slt, St, Msl, back to back and unpadded (any may be NULL) */
extern "C" int cal_sciara_batch_read(void* handle, double* z, double* slt, double* st, double* msl)
{
    Batch* bt = (Batch*)handle;
    cudaStreamSynchronize(bt->st);
    double* outs[4] = {z, slt, st, msl};
    const double* src[4] = {bt->d.Sz, bt->d.Slt, bt->d.St, bt->d.Msl};
    for (int q = 0; q < 4; q++) {
        if (!outs[q])
            continue;
        size_t pos = 0, total = 0;
        for (int b = 0; b < bt->B; b++)
            total += (size_t)bt->inst[b].rows * bt->inst[b].cols;
        cudaPointerAttributes at;
        const bool known = cudaPointerGetAttributes(&at, outs[q]) == cudaSuccess;
        if (!known)
            (void)cudaGetLastError();
        if (!known || at.type == cudaMemoryTypeUnregistered)
            sci2::touch_pages(outs[q], total * sizeof(double));
        for (int b = 0; b < bt->B; b++) {
            const size_t n = (size_t)bt->inst[b].rows * bt->inst[b].cols;
            cudaMemcpy(outs[q] + pos, src[q] + bt->offs[b], n * sizeof(double), cudaMemcpyDeviceToHost);
            pos += n;
        }
    }
    return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

/* lava cells of the last step (all scenarios) */
extern "C" int cal_sciara_batch_lava_cells(void* handle)
{
    Batch* bt = (Batch*)handle;
    int c = 0;
    cudaStreamSynchronize(bt->st);
    cudaMemcpy(&c, bt->d.counts + 13, sizeof(int), cudaMemcpyDeviceToHost);
    return c;
}
