// Beam kernels: density deposit of a layer, substep sizes, and the substepped
// Higuera-Cary push of a layer between two plasma planes.  FP64.
#include "common.cuh"

namespace lcb {

// A particle's 25-point stencil is shared by a group of eight lanes, five of
// which take a row of it (along y) each: the layers of a beam are a few
// thousand particles, which would leave most of the chip idle with one thread
// each, and a thread with hundreds of loads or additions in sequence.
constexpr int BEAM_GROUP = 8;

struct LayoutArgs {
    int64_t n;
    int N;
    double h, xi_step, xi_layer;
    const double *x, *y, *xi, *q;
    double *ro0, *ro1;
    int *err;
};

// Beam density deposit (lcode/beam3d/weights.py:108-138, driver :152-163):
// q * w4(x) w4(y) * xi_loc into ro0 and * (1 - xi_loc) into ro1.  Stencil
// points are addressed by the flat index (iy+ky) + N (ix+kx) as in the
// reference; points whose flat index leaves [0, N*N) are skipped and flagged.
// Thread `first` of `threads`.
__device__ __forceinline__ void layout(const LayoutArgs &l, int64_t first, int64_t threads)
{
    const int half_n = l.N / 2, a = (int)(first % BEAM_GROUP);
    const int64_t NN = (int64_t)l.N * l.N;
    if (a >= 5) return;
    for (int64_t k = first / BEAM_GROUP; k < l.n; k += threads / BEAM_GROUP) {
        const double xi_loc = (l.xi_layer - l.xi[k]) / l.xi_step;
        double xl, yl;
        const int ix = cell_of(l.x[k] / l.h + 0.5, half_n, xl);
        const int iy = cell_of(l.y[k] / l.h + 0.5, half_n, yl);
        double wx[5], wy[5];
        weights4(xl, wx);
        weights4(yl, wy);
        const double wxa = a == 0 ? wx[0] : a == 1 ? wx[1] : a == 2 ? wx[2] : a == 3 ? wx[3] : wx[4];
        const double qk = l.q[k];
        bool bad = false;
#pragma unroll
        for (int b = 0; b < 5; b++) {
            const double w = wxa * wy[b];
            const double w0 = w * xi_loc, w1 = w * (1 - xi_loc);
            const int64_t idx = (int64_t)(iy + b - 2) + (int64_t)l.N * (ix + a - 2);
            if (idx < 0 || idx >= NN) { bad = true; continue; }
            atomicAdd(l.ro0 + idx, qk * w0);
            atomicAdd(l.ro1 + idx, qk * w1);
        }
        if (bad && l.err) atomicOr(l.err, LCB_DEVERR_BEAM_STENCIL);
    }
}

__global__ void __launch_bounds__(128) k_beam_deposit(LayoutArgs l)
{
    layout(l, blockIdx.x * (int64_t)blockDim.x + threadIdx.x, (int64_t)gridDim.x * blockDim.x);
}

// Substep size (lcode/beam3d/beam_calculator.py:28-46) and the driver's
// scaling (:111-114).
__global__ void k_beam_substepping(int64_t n, const double *__restrict__ q_m,
                                   const double *__restrict__ pz, double e_sub,
                                   double time_step, double *dt, int64_t *rem)
{
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
         k += (int64_t)gridDim.x * blockDim.x) {
        const double qm = q_m[k], p = pz[k];
        const double max_dt = sqrt(sqrt(1 / (qm * qm) + p * p) / e_sub);
        double d = 1.0;
        // The reference halves without limit; here the substep stops at
        // 2^-20 (a million substeps) so a degenerate q_m cannot stall the
        // push kernel.  Physical beams stop after a few halvings.
        while (d > max_dt && d > 0x1p-20) d /= 2;
        dt[k] = d * time_step;
        rem[k] = (int64_t)(1. / d);
    }
}

// Layers up to this size push with a group of lanes per particle, larger ones
// with one thread each.  A layer step (push, compaction, layout) on a 257
// grid, groups against single threads: 13.6 / 18.6 us for 833 particles, 25.6
// / 31.8 us for 8,333, 78.8 / 76.9 us for 33,333.
constexpr int64_t BEAM_GROUP_MAX = 16384;

struct FieldPair {
    const double *k[6], *k1[6];  // Ex Ey Ez Bx By Bz at plane k and k+1
};

struct PushParams {
    double xi_step, r_max, xi_k, xi_k1, h;
    int N;
};

// One particle's substepped push (lcode/beam3d/move.py:155-273).  Fields are
// weighted with w0 = xi_loc on plane k and w1 = 1 - xi_loc on plane k+1, as
// the reference GPU kernel weights them.  Updates the state in place and
// returns the flags 1 lost | 2 moved | 4 fell; the id is negated when lost.
// G lanes of a warp (1, or BEAM_GROUP with the same particle in all of them;
// `sub`: the lane's place) share the gather, a row of the stencil each, and
// go through the rest together.
template <int G>
__device__ uint8_t push_particle(int sub, const PushParams &P, const FieldPair &F, double qm, double dt,
                                 int64_t &r, int64_t &id, double &x, double &y, double &xi,
                                 double &px, double &py, double &pz, int *err)
{
    const int half_n = P.N / 2;
    const int64_t NN = (int64_t)P.N * P.N;
    const double q = copysign(1.0, qm);
    const double im = 1. / qm;
    bool lost = false, fell = false, bad = false;
    if (r > (int64_t(1) << 20)) {  // bounded work per particle
        r = int64_t(1) << 20;
        if (err) atomicOr(err, LCB_DEVERR_CAPACITY);
    }
    while (r > 0) {
        double gm = sqrt(im * im + px * px + py * py + pz * pz);
        const double xh = x + dt / 2. * (px / gm);
        const double yh = y + dt / 2. * (py / gm);
        const double xih = xi + dt / 2. * (pz / gm - 1);
        if (xih < P.xi_k1) { fell = true; break; }
        if (xh * xh + yh * yh >= P.r_max * P.r_max) {
            x = xh; y = yh; xi = xih;
            lost = true; r = 0;
            break;
        }
        double xl, yl;
        const int ix = cell_of(xh / P.h + 0.5, half_n, xl);
        const int iy = cell_of(yh / P.h + 0.5, half_n, yl);
        const double xi_loc = (xih - P.xi_k) / P.xi_step;
        double wx[5], wy[5];
        weights4(xl, wx);
        weights4(yl, wy);
        double Ex = 0, Ey = 0, Ez = 0, Bx = 0, By = 0, Bz = 0;
        // one row (G > 1: the lane's own), or all five
#pragma unroll
        for (int u = 0; u < (G > 1 ? 1 : 5); u++) {
            const int a = G > 1 ? sub : u;
            const double wxa = a == 0 ? wx[0] : a == 1 ? wx[1] : a == 2 ? wx[2] : a == 3 ? wx[3] : wx[4];
#pragma unroll
            for (int b = 0; b < 5; b++) {
                const double w = wxa * wy[b];
                const double w0 = w * xi_loc, w1 = w * (1 - xi_loc);
                const int64_t idx = (int64_t)(iy + b - 2) + (int64_t)P.N * (ix + a - 2);
                if (a >= 5) continue;
                if (idx < 0 || idx >= NN) { bad = true; continue; }
                Ex += __ldg(F.k[0] + idx) * w0 + __ldg(F.k1[0] + idx) * w1;
                Bx += __ldg(F.k[3] + idx) * w0 + __ldg(F.k1[3] + idx) * w1;
                Ey += __ldg(F.k[1] + idx) * w0 + __ldg(F.k1[1] + idx) * w1;
                By += __ldg(F.k[4] + idx) * w0 + __ldg(F.k1[4] + idx) * w1;
                Ez += __ldg(F.k[2] + idx) * w0 + __ldg(F.k1[2] + idx) * w1;
                Bz += __ldg(F.k[5] + idx) * w0 + __ldg(F.k1[5] + idx) * w1;
            }
        }
        if (G > 1) {
            const unsigned lanes = ((1u << (G & 31)) - 1u) << ((threadIdx.x & 31) / G * G);
#pragma unroll
            for (int o = G / 2; o > 0; o >>= 1) {
                Ex += __shfl_xor_sync(lanes, Ex, o); Bx += __shfl_xor_sync(lanes, Bx, o);
                Ey += __shfl_xor_sync(lanes, Ey, o); By += __shfl_xor_sync(lanes, By, o);
                Ez += __shfl_xor_sync(lanes, Ez, o); Bz += __shfl_xor_sync(lanes, Bz, o);
            }
        }
        const double hd = q * dt / 2.;
        const double pxm = px + hd * Ex, bx = hd * Bx;
        const double pym = py + hd * Ey, by = hd * By;
        const double pzm = pz + hd * Ez, bz = hd * Bz;
        gm = sqrt(im * im + pxm * pxm + pym * pym + pzm * pzm);
        const double bsq = bx * bx + by * by + bz * bz;
        const double bp = bx * pxm + by * pym + bz * pzm;
        const double g2 = gm * gm - bsq;
        gm = sqrt((g2 + sqrt(g2 * g2 + 4 * bsq + 4 * bp * bp)) / 2.);
        const double tx = bx / gm, ty = by / gm, tz = bz / gm;
        const double tp = 1. + tx * tx + ty * ty + tz * tz;
        const double tmn = 1. - tx * tx - ty * ty - tz * tz;
        const double sx = 2. * tx / tp, sy = 2. * ty / tp, sz = 2. * tz / tp;
        const double sp = sx * pxm + sy * pym + sz * pzm;
        px = tx * sp + pxm * tmn / tp + pym * sz - pzm * sy + hd * Ex;
        py = ty * sp + pym * tmn / tp + pzm * sx - pxm * sz + hd * Ey;
        pz = tz * sp + pzm * tmn / tp + pxm * sy - pym * sx + hd * Ez;
        gm = sqrt(im * im + px * px + py * py + pz * pz);
        x = xh + dt / 2. * (px / gm);
        y = yh + dt / 2. * (py / gm);
        xi = xih + dt / 2. * (pz / gm - 1);
        if (x * x + y * y >= P.r_max * P.r_max) { lost = true; r = 0; break; }
        r -= 1;
    }
    if (r == 0 && xi < P.xi_k1) fell = true;
    if (lost) id = -id;
    if (bad && err) atomicOr(err, LCB_DEVERR_BEAM_STENCIL);
    return (uint8_t)((lost ? 1 : 0) | (fell ? 4 : 0) | (!fell && !lost ? 2 : 0));
}

template <int G>
__global__ void __launch_bounds__(128)
k_beam_move(int64_t n, PushParams P, const double *__restrict__ q_m,
            const double *__restrict__ dt_a, FieldPair F, int64_t *rem,
            int64_t *id, double *xa, double *ya, double *xia, double *pxa,
            double *pya, double *pza, uint8_t *flags, int *err)
{
    const int sub = threadIdx.x % G;
    for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G; i < n;
         i += (int64_t)gridDim.x * blockDim.x / G) {
        double x = xa[i], y = ya[i], xi = xia[i], px = pxa[i], py = pya[i], pz = pza[i];
        int64_t r = rem[i], pid = id[i];
        const uint8_t f = push_particle<G>(sub, P, F, q_m[i], dt_a[i], r, pid, x, y, xi, px, py, pz, err);
        if (G > 1) __syncwarp(((1u << (G & 31)) - 1u) << ((threadIdx.x & 31) / G * G));   // all have read it
        if (sub != 0) continue;
        flags[i] = f;
        xa[i] = x; ya[i] = y; xia[i] = xi; pxa[i] = px; pya[i] = py; pza[i] = pz;
        rem[i] = r;
        id[i] = pid;
    }
}

// ---------------------------------------------------------------------------
// Device-resident layer step: push the previous layer (the fresh particles
// of the source slice, with their substep sizes, then the particles that
// fell from the push before) into a staging buffer, then compact it in order
// into the drain (moved), the next fell buffer and the lost buffer.  The fell
// and drain counts live on the device, so the xi loop never waits for the
// host.  Orders match the reference's boolean-mask gathers
// (beam_calculator.py:130-134, data.py:151-178).
// ---------------------------------------------------------------------------
__device__ __forceinline__ double substep(double qm, double pz, double e_sub)
{
    const double max_dt = sqrt(sqrt(1 / (qm * qm) + pz * pz) / e_sub);
    double d = 1.0;
    while (d > max_dt && d > 0x1p-20) d /= 2;
    return d;
}

struct StepArgs {
    lcb_beam_soa src, fin, stage;
    int64_t move_begin, n_fresh;
    const int64_t *fell_in_count;
    int64_t stage_capacity;
    uint8_t *flags;
    double e_sub, time_step;
    PushParams P;
    FieldPair F;
    double *clear;          // plane zeroed by the same grid (the next layout's lower plane)
    int64_t clear_n;
    int64_t *fell_out_count;   // zeroed too (the compaction's blocks check out there)
    int *err;
};

__device__ __forceinline__ void soa_load(const lcb_beam_soa &s, int64_t i, double *v, int64_t &id,
                                         int64_t &rem)
{
    v[0] = s.xi[i]; v[1] = s.x[i]; v[2] = s.y[i]; v[3] = s.px[i]; v[4] = s.py[i];
    v[5] = s.pz[i]; v[6] = s.q_m[i]; v[7] = s.q_norm[i]; v[8] = s.dt[i];
    id = s.id[i];
    rem = s.remaining_steps[i];
}

__device__ __forceinline__ void soa_store(const lcb_beam_soa &s, int64_t i, const double *v,
                                          int64_t id, int64_t rem)
{
    s.xi[i] = v[0]; s.x[i] = v[1]; s.y[i] = v[2]; s.px[i] = v[3]; s.py[i] = v[4];
    s.pz[i] = v[5]; s.q_m[i] = v[6]; s.q_norm[i] = v[7]; s.dt[i] = v[8];
    s.id[i] = id;
    s.remaining_steps[i] = rem;
}

template <int G>
__device__ __forceinline__ void push_stage(const StepArgs &a, int64_t total)
{
    const int sub = threadIdx.x % G;
    for (int64_t t = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G; t < total;
         t += (int64_t)gridDim.x * blockDim.x / G) {
        if (t >= a.stage_capacity) {
            if (a.err) atomicOr(a.err, LCB_DEVERR_CAPACITY);
            break;
        }
        double v[9];
        int64_t id, rem;
        if (t < a.n_fresh) {
            soa_load(a.src, a.move_begin + t, v, id, rem);
            const double d = substep(v[6], v[5], a.e_sub);  // beam_calculator.py:109-114
            v[8] = d * a.time_step;
            rem = (int64_t)(1. / d);
        } else {
            soa_load(a.fin, t - a.n_fresh, v, id, rem);
        }
        const uint8_t f = push_particle<G>(sub, a.P, a.F, v[6], v[8], rem, id, v[1], v[2], v[0], v[3],
                                           v[4], v[5], a.err);
        if (sub == 0) {
            a.flags[t] = f;
            soa_store(a.stage, t, v, id, rem);
        }
    }
}

// The grid is sized by the fresh particles; how many have fallen is known here
// only.  Groups take what the grid can hold of them twice over, which is all of
// a layer whose particles are mostly fresh; more than that go one to a thread
// (a layer step behind the beam, 50,000 fallen particles and none fresh: 54 us,
// with groups and one compacting block 372; all in single threads and one block
// of 1024, 207).  GROUPS false: more fresh particles than groups take.
template <bool GROUPS>
__global__ void __launch_bounds__(128) k_beam_push_stage(StepArgs a)
{
    pdl_wait();
    pdl_trigger();
    if (a.fell_out_count && blockIdx.x == 0 && threadIdx.x == 0) *a.fell_out_count = 0;
    const int64_t threads = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < a.clear_n; t += threads) a.clear[t] = 0.0;
    const int64_t total = a.n_fresh + *a.fell_in_count;
    if (GROUPS && total <= BEAM_GROUP_MAX && total * BEAM_GROUP <= 2 * threads) push_stage<BEAM_GROUP>(a, total);
    else push_stage<1>(a, total);
}

struct CompactArgs {
    lcb_beam_soa stage, drain, fout, lost;
    const uint8_t *flags;
    int64_t n_fresh;
    const int64_t *fell_in_count;
    int64_t stage_capacity;
    int64_t *drain_count, *fell_out_count, *lost_count;
    int64_t drain_capacity, fell_capacity, lost_capacity;
    int *err;
};

// Ordered compaction: a block takes tiles of 256 staged particles and finds
// where a tile's particles go by counting the flags before it itself (a byte
// per particle, from L2), so that the blocks do not wait for one another.
// The counters may only move once every block has read them: the blocks check
// out in the upper bits of fell_out_count (zeroed by the push, or the count of
// the fallen itself where that is updated in place), and the last one writes all
// three.  The grid's other blocks lay out the next layer meanwhile (that
// reads only the source, and the push's grid has cleared ro1).
// For a layer of 8,300 particles one block over all chunks took 34 us and the
// layout another 9 after it.
constexpr int CMP_THREADS = 256, CMP_WARPS = CMP_THREADS / 32;
constexpr int CMP_CHECK_OUT = 40;   // a count is below 2^40

struct FlagCounts { int moved, fell, lost; };

__device__ __forceinline__ void count_word(FlagCounts &c, unsigned w)
{
    c.moved += __popc(w & 0x02020202u);
    c.fell += __popc(w & 0x04040404u);
    c.lost += __popc(w & 0x01010101u);
}

// The block's sums over flags [from, to), the same in every thread.
__device__ FlagCounts count_flags(const uint8_t *flags, int64_t from, int64_t to, int (*red)[3])
{
    FlagCounts c = {0, 0, 0};
    const int tid = threadIdx.x;
    int64_t k = from;
    if (((uintptr_t)(flags + from) & 15) == 0) {
        const int64_t quads = (to - from) / 16;
        const uint4 *q = reinterpret_cast<const uint4 *>(flags + from);
        for (int64_t t = tid; t < quads; t += CMP_THREADS) {
            const uint4 w = q[t];
            count_word(c, w.x); count_word(c, w.y); count_word(c, w.z); count_word(c, w.w);
        }
        k += quads * 16;
    }
    for (k += tid; k < to; k += CMP_THREADS) count_word(c, flags[k]);
    c.moved = __reduce_add_sync(0xffffffffu, c.moved);
    c.fell = __reduce_add_sync(0xffffffffu, c.fell);
    c.lost = __reduce_add_sync(0xffffffffu, c.lost);
    __syncthreads();   // the last sums have been read
    if ((tid & 31) == 0) {
        red[tid >> 5][0] = c.moved; red[tid >> 5][1] = c.fell; red[tid >> 5][2] = c.lost;
    }
    __syncthreads();
    c = {0, 0, 0};
#pragma unroll
    for (int w = 0; w < CMP_WARPS; w++) {
        c.moved += red[w][0]; c.fell += red[w][1]; c.lost += red[w][2];
    }
    return c;
}

__device__ void compact(const CompactArgs &a, int block, int blocks)
{
    __shared__ int red[CMP_WARPS][3], wsum[CMP_WARPS][3];
    __shared__ bool last;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int64_t total = a.n_fresh + (*a.fell_in_count & ((int64_t(1) << CMP_CHECK_OUT) - 1));
    if (total > a.stage_capacity) total = a.stage_capacity;
    const int64_t drain0 = *a.drain_count, lost0 = a.lost_count ? *a.lost_count : 0;
    int64_t om = drain0, of = 0, ol = lost0, counted = 0;   // places of the tile's first ones
    for (int64_t t0 = (int64_t)block * CMP_THREADS; t0 < total; t0 += (int64_t)blocks * CMP_THREADS) {
        const FlagCounts before = count_flags(a.flags, counted, t0, red);
        counted = t0;
        om += before.moved; of += before.fell; ol += before.lost;
        const int64_t t = t0 + tid;
        const uint8_t f = t < total ? a.flags[t] : 0;
        double v[9];
        int64_t id = 0, rem = 0;
        if (f) soa_load(a.stage, t, v, id, rem);
        const unsigned mm = __ballot_sync(0xffffffffu, f & 2), mf = __ballot_sync(0xffffffffu, f & 4),
                       ml = __ballot_sync(0xffffffffu, f & 1), lower = (1u << lane) - 1u;
        if (lane == 0) { wsum[warp][0] = __popc(mm); wsum[warp][1] = __popc(mf); wsum[warp][2] = __popc(ml); }
        __syncthreads();
        int pm = __popc(mm & lower), pf = __popc(mf & lower), pl = __popc(ml & lower);
        for (int w = 0; w < warp; w++) { pm += wsum[w][0]; pf += wsum[w][1]; pl += wsum[w][2]; }
        if (f & 2) {
            if (om + pm < a.drain_capacity) soa_store(a.drain, om + pm, v, id, rem);
            else if (a.err) atomicOr(a.err, LCB_DEVERR_CAPACITY);
        } else if (f & 4) {
            if (of + pf < a.fell_capacity) soa_store(a.fout, of + pf, v, id, rem);
            else if (a.err) atomicOr(a.err, LCB_DEVERR_CAPACITY);
        }
        // (a lost particle that has also fallen goes into both buffers)
        if ((f & 1) && a.lost.id) {
            if (ol + pl < a.lost_capacity) soa_store(a.lost, ol + pl, v, id, rem);
            else if (a.err) atomicOr(a.err, LCB_DEVERR_CAPACITY);
        }
    }
    __syncthreads();   // every thread has read the counters
    if (tid == 0) {
        __threadfence();
        last = atomicAdd(reinterpret_cast<unsigned long long *>(a.fell_out_count), 1ull << CMP_CHECK_OUT) >>
               CMP_CHECK_OUT == (unsigned long long)(blocks - 1);
    }
    __syncthreads();
    if (!last) return;
    const FlagCounts all = count_flags(a.flags, 0, total, red);
    if (tid == 0) {
        const int64_t d = drain0 + all.moved, l = lost0 + all.lost;
        *a.drain_count = d < a.drain_capacity ? d : a.drain_capacity;
        *a.fell_out_count = all.fell < a.fell_capacity ? all.fell : a.fell_capacity;
        if (a.lost_count) *a.lost_count = l < a.lost_capacity ? l : a.lost_capacity;
    }
}

__global__ void __launch_bounds__(CMP_THREADS) k_beam_compact_layout(CompactArgs a, LayoutArgs l, int blocks)
{
    pdl_wait();
    pdl_trigger();
    if ((int)blockIdx.x < blocks) compact(a, blockIdx.x, blocks);
    else layout(l, (int64_t)(blockIdx.x - blocks) * CMP_THREADS + threadIdx.x,
                (int64_t)(gridDim.x - blocks) * CMP_THREADS);
}

static int grid_for(int64_t n, int threads)
{
    int64_t blocks = (n + threads - 1) / threads;
    const int64_t cap = (int64_t)sm_count() * 16;
    if (blocks > cap) blocks = cap;
    return (int)(blocks < 1 ? 1 : blocks);
}

}  // namespace lcb

using namespace lcb;

extern "C" int lcb_beam_deposit(int64_t n, int grid_steps, double h, double xi_step,
                                int64_t layer_idx, const double *x, const double *y,
                                const double *xi, const double *q_norm, double *ro0,
                                double *ro1, int *err, void *stream)
{
    LCB_REQUIRE(n >= 0 && grid_steps >= 5, "bad sizes");
    if (n == 0) return LCB_OK;
    const LayoutArgs l = {n, grid_steps, h, xi_step, -xi_step * (double)layer_idx, x, y, xi, q_norm, ro0, ro1, err};
    k_beam_deposit<<<grid_for(n * BEAM_GROUP, 128), 128, 0, as_stream(stream)>>>(l);
    LCB_LAUNCH_CHECK("k_beam_deposit");
    return LCB_OK;
}

extern "C" int lcb_beam_substepping(int64_t n_fresh, const double *q_m, const double *pz,
                                    double substep_energy, double time_step, double *dt,
                                    int64_t *remaining_steps, void *stream)
{
    LCB_REQUIRE(n_fresh >= 0, "n < 0");
    LCB_REQUIRE(substep_energy > 0, "beam-substepping-energy must be > 0");
    if (n_fresh == 0) return LCB_OK;
    k_beam_substepping<<<grid_for(n_fresh, 128), 128, 0, as_stream(stream)>>>(
        n_fresh, q_m, pz, substep_energy, time_step, dt, remaining_steps);
    LCB_LAUNCH_CHECK("k_beam_substepping");
    return LCB_OK;
}

extern "C" int lcb_beam_move(int64_t n, double xi_step, double r_max,
                             int64_t beam_layer_idx, double h, int grid_steps,
                             const double *q_m, const double *dt,
                             const lcb_fields *fields_k, const lcb_fields *fields_k1,
                             int64_t *remaining_steps, int64_t *id, double *x,
                             double *y, double *xi, double *px, double *py,
                             double *pz, uint8_t *flags, int *err, void *stream)
{
    LCB_REQUIRE(n >= 0 && grid_steps >= 5, "bad sizes");
    LCB_REQUIRE(fields_k && fields_k1, "fields are NULL");
    if (n == 0) return LCB_OK;
    FieldPair F;
    for (int c = 0; c < 6; c++) {
        F.k[c] = fields_k->f[c];
        F.k1[c] = fields_k1->f[c];
        LCB_REQUIRE(F.k[c] && F.k1[c], "field plane %d is NULL", c);
    }
    PushParams P;
    P.xi_step = xi_step; P.r_max = r_max; P.h = h; P.N = grid_steps;
    P.xi_k = (double)beam_layer_idx * (-xi_step);
    P.xi_k1 = (double)(beam_layer_idx + 1) * (-xi_step);
    if (n <= BEAM_GROUP_MAX)
        k_beam_move<BEAM_GROUP><<<grid_for(n * BEAM_GROUP, 128), 128, 0, as_stream(stream)>>>(
            n, P, q_m, dt, F, remaining_steps, id, x, y, xi, px, py, pz, flags, err);
    else
        k_beam_move<1><<<grid_for(n, 128), 128, 0, as_stream(stream)>>>(
            n, P, q_m, dt, F, remaining_steps, id, x, y, xi, px, py, pz, flags, err);
    LCB_LAUNCH_CHECK("k_beam_move");
    return LCB_OK;
}

static bool soa_ok(const lcb_beam_soa &s)
{
    return s.xi && s.x && s.y && s.px && s.py && s.pz && s.q_m && s.q_norm && s.id &&
           s.dt && s.remaining_steps;
}

extern "C" int lcb_beam_step(const lcb_beam_step_args *a, void *stream)
{
    LCB_REQUIRE(a, "args is NULL");
    LCB_REQUIRE(a->grid_steps >= 5 && a->h > 0 && a->xi_step > 0, "bad grid parameters");
    LCB_REQUIRE(a->layout_begin >= 0 && a->layout_end >= a->layout_begin &&
                a->move_begin >= 0 && a->move_end >= a->move_begin, "bad layer slices");
    LCB_REQUIRE(a->substep_energy > 0, "beam-substepping-energy must be > 0");
    LCB_REQUIRE(a->fell_in_count && a->fell_out_count && a->drain_count && a->stage_flags,
                "device counters / flags are NULL");
    LCB_REQUIRE(a->fields_k && a->fields_k1, "fields are NULL");
    LCB_REQUIRE(soa_ok(a->source) && soa_ok(a->fell_in) && soa_ok(a->fell_out) &&
                soa_ok(a->drain) && soa_ok(a->stage), "beam arrays are NULL");
    LCB_REQUIRE(a->move_end - a->move_begin <= a->stage_capacity,
                "stage capacity %lld < fresh layer %lld", (long long)a->stage_capacity,
                (long long)(a->move_end - a->move_begin));
    LCB_REQUIRE(a->ro0 && a->ro1, "density planes are NULL");
    cudaStream_t st = as_stream(stream);
    const int N = a->grid_steps;
    StepArgs s;
    s.src = a->source; s.fin = a->fell_in; s.stage = a->stage;
    s.move_begin = a->move_begin; s.n_fresh = a->move_end - a->move_begin;
    s.fell_in_count = a->fell_in_count;
    s.stage_capacity = a->stage_capacity;
    s.flags = a->stage_flags;
    s.e_sub = a->substep_energy; s.time_step = a->time_step;
    s.P.xi_step = a->xi_step; s.P.r_max = a->r_max; s.P.h = a->h; s.P.N = N;
    s.P.xi_k = (double)(a->layer_idx - 1) * (-a->xi_step);
    s.P.xi_k1 = (double)(a->layer_idx) * (-a->xi_step);
    for (int c = 0; c < 6; c++) {
        s.F.k[c] = a->fields_k->f[c];
        s.F.k1[c] = a->fields_k1->f[c];
        LCB_REQUIRE(s.F.k[c] && s.F.k1[c], "field plane %d is NULL", c);
    }
    s.clear = a->ro1;
    s.clear_n = (int64_t)N * N;
    s.fell_out_count = a->fell_out_count == a->fell_in_count ? nullptr : a->fell_out_count;
    s.err = a->err;
    // at least two blocks per SM, for the plane and for particles that fell
    // (their number is on the device)
    const bool group = s.n_fresh <= BEAM_GROUP_MAX;
    const int pg = grid_for(group ? s.n_fresh * BEAM_GROUP : s.n_fresh, 128), most = 2 * sm_count();
    cudaError_t e = launch_after(group ? k_beam_push_stage<true> : k_beam_push_stage<false>,
                                 dim3(pg > most ? pg : most), dim3(128), 0, st, s);
    if (e != cudaSuccess) return cuda_check(e, "beam push launch");
    count_launch();
    CompactArgs c;
    c.stage = a->stage; c.drain = a->drain; c.fout = a->fell_out; c.lost = a->lost;
    c.flags = a->stage_flags;
    c.n_fresh = s.n_fresh; c.fell_in_count = a->fell_in_count;
    c.stage_capacity = a->stage_capacity;
    c.drain_count = a->drain_count; c.fell_out_count = a->fell_out_count;
    c.lost_count = a->lost.id ? a->lost_count : nullptr;
    c.drain_capacity = a->drain_capacity; c.fell_capacity = a->fell_capacity;
    c.lost_capacity = a->lost_capacity;
    c.err = a->err;
    const int64_t n = a->layout_end - a->layout_begin, o = a->layout_begin;
    const LayoutArgs l = {n, N, a->h, a->xi_step, -a->xi_step * (double)a->layout_idx,
                          a->source.x + o, a->source.y + o, a->source.xi + o, a->source.q_norm + o,
                          a->ro0, a->ro1, a->err};
    // blocks for every tile that the staging buffer can hold, up to two per SM
    // (those without a tile only check out: the number of fallen particles is
    // on the device); as many again at most for the layout
    auto blocks = [&](int64_t threads) {
        const int64_t b = (threads + CMP_THREADS - 1) / CMP_THREADS;
        return (int)(b < most ? b : most);
    };
    const int nc = a->stage_capacity > 0 ? blocks(a->stage_capacity) : 1;
    e = launch_after(k_beam_compact_layout, dim3(nc + blocks(n * BEAM_GROUP)), dim3(CMP_THREADS), 0, st, c, l, nc);
    if (e != cudaSuccess) return cuda_check(e, "beam compaction launch");
    count_launch();
    return LCB_OK;
}
