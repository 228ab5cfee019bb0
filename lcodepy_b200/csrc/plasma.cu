// Plasma particle kernels: free-streaming estimate, fused gather + push, and
// tiled charge/current deposition.  FP64 particles (SoA, coalesced).
#include <type_traits>

#include "common.cuh"

namespace lcb {

// ---------------------------------------------------------------------------
// K1: copy prev -> full and free-stream (lcode/plasma3d/move.py:292-313,
// copy at :337-339).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
k_move_wo_fields(int64_t n, double xi_step, const double *__restrict__ m,
                 const double *__restrict__ xo_p, const double *__restrict__ yo_p,
                 const double *__restrict__ px_p, const double *__restrict__ py_p,
                 const double *__restrict__ pz_p, const double *__restrict__ q_p,
                 double *xo_f, double *yo_f, double *px_f, double *py_f,
                 double *pz_f, double *q_f)
{
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
         k += (int64_t)gridDim.x * blockDim.x) {
        const double mk = m[k], px = px_p[k], py = py_p[k], pz = pz_p[k];
        double xo = xo_p[k], yo = yo_p[k];
        if (mk != 0) {
            const double gm = sqrt(mk * mk + pz * pz + px * px + py * py);
            const double adv = xi_step / (gm - pz);
            xo += px * adv;
            yo += py * adv;
        }
        xo_f[k] = xo; yo_f[k] = yo;
        px_f[k] = px; py_f[k] = py; pz_f[k] = pz;
        q_f[k] = q_p[k];
    }
}

// ---------------------------------------------------------------------------
// K2: fused midpoint gather + two-pass momentum update + advance +
// reflection + absorption (lcode/plasma3d/move.py:169-289).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void reflect(double &x, double b, double &px, double &py, double &pz)
{
    if (x > b)  { x =  2 * b - x; px = py = pz = 0; }
    if (x < -b) { x = -2 * b - x; px = py = pz = 0; }
}

__global__ void __launch_bounds__(256)
k_move_smart(int64_t n, double xi_step, double boundary, double h, int N,
             const double *__restrict__ Exf, const double *__restrict__ Eyf,
             const double *__restrict__ Ezf, const double *__restrict__ Bxf,
             const double *__restrict__ Byf, const double *__restrict__ Bzf,
             const double *__restrict__ x_init, const double *__restrict__ y_init,
             const double *__restrict__ xo_p, const double *__restrict__ yo_p,
             const double *__restrict__ px_p, const double *__restrict__ py_p,
             const double *__restrict__ pz_p, const double *__restrict__ m,
             double *q_f, double *xo_f, double *yo_f, double *px_f,
             double *py_f, double *pz_f, int *err)
{
    const int half_n = N / 2;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
         k += (int64_t)gridDim.x * blockDim.x) {
        const double qk = q_f[k];
        if (qk == 0) continue;
        const double xi0 = x_init[k], yi0 = y_init[k];
        const double opx = px_p[k], opy = py_p[k], opz = pz_p[k];
        double px = opx, py = opy, pz = opz;
        double xh = xi0 + (xo_p[k] + xo_f[k]) / 2;
        double yh = yi0 + (yo_p[k] + yo_f[k]) / 2;
        // The reference zeroes momenta when the midpoint is reflected; the
        // zeroed values only feed gamma in the first pass below.
        if (xh > boundary)  { xh =  2 * boundary - xh; px = py = pz = 0; }
        if (xh < -boundary) { xh = -2 * boundary - xh; px = py = pz = 0; }
        if (yh > boundary)  { yh =  2 * boundary - yh; px = py = pz = 0; }
        if (yh < -boundary) { yh = -2 * boundary - yh; px = py = pz = 0; }

        double xl, yl;
        const int ix = cell_of(xh / h + 0.5, half_n, xl);
        const int iy = cell_of(yh / h + 0.5, half_n, yl);
        double Ex = 0, Ey = 0, Ez = 0, Bx = 0, By = 0, Bz = 0;
        if (ix >= 2 && ix < N - 2 && iy >= 2 && iy < N - 2) {
            double wx[5], wy[5];
            weights4(xl, wx);
            weights4(yl, wy);
#pragma unroll
            for (int a = 0; a < 5; a++) {
                const int row = (ix + a - 2) * N + iy - 2;
#pragma unroll
                for (int b = 0; b < 5; b++) {
                    const double w = wx[a] * wy[b];
                    const int idx = row + b;
                    Ex += __ldg(Exf + idx) * w; Bx += __ldg(Bxf + idx) * w;
                    Ey += __ldg(Eyf + idx) * w; By += __ldg(Byf + idx) * w;
                    Ez += __ldg(Ezf + idx) * w; Bz += __ldg(Bzf + idx) * w;
                }
            }
        } else if (err) {
            atomicOr(err, LCB_DEVERR_PLASMA_STENCIL);
        }
        const double mk = m[k];
        // velocities as p * (1/gamma m): one quotient per pass instead of three
        double gm = sqrt(mk * mk + px * px + py * py + pz * pz);
        double ig = 1.0 / gm;
        double vx = px * ig, vy = py * ig, vz = pz * ig;
        double f = qk * xi_step / (1 - vz);
        double dpx = f * (Ex + vy * Bz - vz * By);
        double dpy = f * (Ey - vx * Bz + vz * Bx);
        double dpz = f * (Ez + vx * By - vy * Bx);
        px = opx + dpx * 0.5; py = opy + dpy * 0.5; pz = opz + dpz * 0.5;

        gm = sqrt(mk * mk + px * px + py * py + pz * pz);
        ig = 1.0 / gm;
        vx = px * ig; vy = py * ig; vz = pz * ig;
        f = qk * xi_step / (1 - vz);
        dpx = f * (Ex + vy * Bz - vz * By);
        dpy = f * (Ey - vx * Bz + vz * Bx);
        dpz = f * (Ez + vx * By - vy * Bx);
        px = opx + dpx * 0.5; py = opy + dpy * 0.5; pz = opz + dpz * 0.5;

        gm = sqrt(mk * mk + px * px + py * py + pz * pz);
        const double adv = xi_step / (gm - pz);
        double xo = xo_p[k] + px * adv;
        double yo = yo_p[k] + py * adv;
        px = opx + dpx; py = opy + dpy; pz = opz + dpz;

        double x = xi0 + xo, y = yi0 + yo;
        if (x > boundary)  { x =  2 * boundary - x; xo = x - xi0; px = py = pz = 0; }
        if (x < -boundary) { x = -2 * boundary - x; xo = x - xi0; px = py = pz = 0; }
        if (y > boundary)  { y =  2 * boundary - y; yo = y - yi0; px = py = pz = 0; }
        if (y < -boundary) { y = -2 * boundary - y; yo = y - yi0; px = py = pz = 0; }
        if (x >= boundary || x <= -boundary || y >= boundary || y <= -boundary) {
            xo = yo = 0; px = py = pz = 0;
            q_f[k] = 0;
        }
        xo_f[k] = xo; yo_f[k] = yo;
        px_f[k] = px; py_f[k] = py; pz_f[k] = pz;
    }
}

// ---------------------------------------------------------------------------
// K3: deposition (lcode/plasma3d/weights.py:151-190, 249-285).
//
// A block owns a TI x TJ tile of one sort's particle lattice (particles are
// created on a lattice, k = s*Np + i*Ns + j, and drift little per xi step, so
// a tile's particles stay in a compact cell window).  Contributions whose
// whole 5x5 stencil lies inside the block's shared-memory window [wx0, wx0+WX)
// x [wy0, wy0+WY) are accumulated there with shared atomics; any other
// particle (a runaway, a lattice that is not a lattice) goes straight to
// global atomics.  The window is then flushed with one global atomic per
// non-zero cell and quantity.  The window origin follows the tile's first
// particle's initial position, with S cells of slack for drift.
//
// FP64 shared atomics retry when two lanes of a warp hit the same address in
// the same instruction.  With two particles per cell along each axis (the
// 2 x 2 per cell lattice) the lanes of a warp are therefore given particles of
// one parity sub-lattice (every other row and column), which sit in distinct
// cells; all 25 stencil points of a warp instruction then differ too.
// ---------------------------------------------------------------------------
constexpr int DEP_TI = 16, DEP_TJ = 32, DEP_THREADS = 256;
constexpr int DEP_NP = DEP_TI * DEP_TJ;
constexpr int DEP_PPT = DEP_NP / DEP_THREADS;
constexpr int DEP_SLACK = 4;
constexpr int DEP_WX = 28, DEP_WY = 44;  // >= tile cells (fineness 1) + 4 + 2*slack

// Tile position (ti, tj) of the q-th particle slot of a block.
__device__ __forceinline__ void tile_slot(int q, bool two_per_cell, int &ti, int &tj)
{
    if (two_per_cell) {
        const int par = q >> 7, w = q & 127;        // 4 parity sub-lattices of 8 x 16
        ti = 2 * (w >> 4) + (par >> 1);
        tj = 2 * (w & 15) + (par & 1);
    } else {
        ti = q / DEP_TJ;
        tj = q % DEP_TJ;
    }
}

// Deposit one particle's 25-point stencil (weights.py:151-190 arithmetic)
// into the block's shared window, or straight into HBM when the stencil
// leaves the window.  dep = false: nothing to deposit.
// Accumulator of the mixed-precision deposit: every contribution is rounded
// to a multiple of 2^-32 and summed as a 64-bit integer, so the sums are
// exact and do not depend on the order of the atomics (an FP32 sum of the
// ~100 contributions a cell receives rounds at the magnitude of the running
// total, which for the electron density is the background ~1, and leaves a
// systematic ~1e-7 error that the background ions then expose).
//
// The rounding is one FMA: v * 2^32 + 1.5 * 2^52 has a unit in the last
// place of exactly 1, so the sum's low mantissa bits are round(v * 2^32) in
// two's complement, read off by subtracting the constant's bit pattern (no
// float-to-integer conversion instruction).  That needs |v| < 2^19 per
// contribution; particles whose values could approach it (|value| / h^2 >=
// 2^20, weights are below 0.36) raise LCB_DEVERR_FIXED_RANGE.  Sums have the
// range +-2^31.
constexpr double FIX_SCALE = 4294967296.0;            // 2^32
constexpr double FIX_INV = 1.0 / 4294967296.0;
constexpr double FIX_MAGIC = 6755399441055744.0;      // 1.5 * 2^52
constexpr double FIX_PARTICLE_LIMIT = 1048576.0;      // 2^20
typedef unsigned long long fix_t;

// round(v * 2^32) from fma(v, 2^32, FIX_MAGIC) (or any x = w * 2^32 * v + FIX_MAGIC)
__device__ __forceinline__ fix_t fix_bits(double x)
{
    return (fix_t)__double_as_longlong(x) - (fix_t)0x4338000000000000ull;
}

template <typename Acc>
__device__ __forceinline__ Acc to_acc(double v) { return Acc(v); }
template <>
__device__ __forceinline__ fix_t to_acc<fix_t>(double v)
{
    return fix_bits(fma(v, FIX_SCALE, FIX_MAGIC));
}

// Particles whose largest contribution could leave the fixed-point rounding
// range set the error word; nothing else changes.
template <typename Acc>
__device__ __forceinline__ void check_range(double, double, double, double, double, int *) {}
template <>
__device__ __forceinline__ void check_range<fix_t>(double dro, double djx, double djy, double djz,
                                                   double ih, int *err)
{
    const double m = fmax(fmax(fabs(dro), fabs(djx)), fmax(fabs(djy), fabs(djz))) * ih * ih;
    if (!(m < FIX_PARTICLE_LIMIT) && err) atomicOr(err, LCB_DEVERR_FIXED_RANGE);
}

template <typename Acc, int WX, int WY>
__device__ __forceinline__ void deposit_one(Acc *sw, Acc *gro, Acc *gjx, Acc *gjy, Acc *gjz,
                                            int N, double h, int wx0, int wy0, bool dep,
                                            int ix, int iy, double xl, double yl,
                                            double dro, double djx, double djy, double djz)
{
    constexpr int WSZ = WX * WY;
    if (!dep) return;
    double wx[5], wy[5];
    weights4(xl, wx);
    weights4(yl, wy);
    // w = (wx / h) (wy / h), with 1/h multiplications for the 30 quotients
    const double ih = 1.0 / h;
#pragma unroll
    for (int b = 0; b < 5; b++) wy[b] *= ih;
    const int lx = ix - 2 - wx0, ly = iy - 2 - wy0;
    const bool inwin = lx >= 0 && lx + 5 <= WX && ly >= 0 && ly + 5 <= WY;
#pragma unroll
    for (int a = 0; a < 5; a++) {
        const double wxa = wx[a] * ih;
#pragma unroll
        for (int b = 0; b < 5; b++) {
            const double w = wxa * wy[b];
            if (inwin) {
                const int c = (lx + a) * WY + ly + b;
                atomicAdd(sw + c, to_acc<Acc>(dro * w));
                atomicAdd(sw + WSZ + c, to_acc<Acc>(djx * w));
                atomicAdd(sw + 2 * WSZ + c, to_acc<Acc>(djy * w));
                atomicAdd(sw + 3 * WSZ + c, to_acc<Acc>(djz * w));
            } else {
                const int64_t c = (int64_t)(ix + a - 2) * N + iy + b - 2;
                atomicAdd(gro + c, to_acc<Acc>(dro * w));
                atomicAdd(gjx + c, to_acc<Acc>(djx * w));
                atomicAdd(gjy + c, to_acc<Acc>(djy * w));
                atomicAdd(gjz + c, to_acc<Acc>(djz * w));
            }
        }
    }
}

template <typename Acc>
__global__ void __launch_bounds__(DEP_THREADS)
k_deposit_tiled(int64_t n_per_sort, int Ns, int N, double h,
                const double *__restrict__ x_init, const double *__restrict__ y_init,
                const double *__restrict__ x_offt, const double *__restrict__ y_offt,
                const double *__restrict__ px_a, const double *__restrict__ py_a,
                const double *__restrict__ pz_a, const double *__restrict__ q_a,
                const double *__restrict__ m_a, Acc *ro, Acc *jx, Acc *jy, Acc *jz,
                int *err)
{
    static_assert(DEP_PPT == 2, "a thread owns two particles");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Acc *sw = reinterpret_cast<Acc *>(smem_raw);  // [4][WX][WY]
    constexpr int WSZ = DEP_WX * DEP_WY;
    const int s = blockIdx.z;
    const int64_t base = (int64_t)s * n_per_sort;
    const int half_n = N / 2;
    const int64_t NN = (int64_t)N * N;
    Acc *gro = ro + s * NN, *gjx = jx + s * NN, *gjy = jy + s * NN, *gjz = jz + s * NN;

    for (int t = threadIdx.x; t < 4 * WSZ; t += blockDim.x) sw[t] = Acc(0);
    // Tiles start on a lattice row whose cell also holds the next row, so
    // that a thread's two particles (slots t and t + DEP_THREADS: lattice
    // rows ti and ti + 1, ti even) usually share a cell; the grid has one
    // spare row of tiles for the shift.
    double dummy;
    int off = 0;
    if (Ns > 1 && cell_of(x_init[base] / h + 0.5, half_n, dummy) !=
                  cell_of(x_init[base + Ns] / h + 0.5, half_n, dummy))
        off = 1;
    const int i0 = blockIdx.y * DEP_TI - off, j0 = blockIdx.x * DEP_TJ;
    const int ir = i0 < 0 ? 0 : i0;
    if (ir >= Ns) return;
    // window origin from the tile's first particle's initial lattice position
    const int64_t k0 = base + (int64_t)ir * Ns + j0;
    const int wx0 = cell_of(x_init[k0] / h + 0.5, half_n, dummy) - 2 - DEP_SLACK;
    const int wy0 = cell_of(y_init[k0] / h + 0.5, half_n, dummy) - 2 - DEP_SLACK;
    // lattice spacing along x: two particles per cell?
    bool two = false;
    if (ir + 1 < Ns) {
        const double d = x_init[k0 + Ns] - x_init[k0];
        two = fabs(2 * d - h) < 0.25 * h;
    }
    __syncthreads();

    bool dep[2];
    double v[2][4], xl[2], yl[2];
    int ix[2], iy[2];
#pragma unroll
    for (int r = 0; r < DEP_PPT; r++) {
        int ti, tj;
        tile_slot(threadIdx.x + r * DEP_THREADS, two, ti, tj);
        const int i = i0 + ti, j = j0 + tj;
        dep[r] = i >= 0 && i < Ns && j < Ns;
        v[r][0] = v[r][1] = v[r][2] = v[r][3] = 0;
        xl[r] = yl[r] = 0;
        ix[r] = iy[r] = -1000;
        if (dep[r]) {
            const int64_t k = base + (int64_t)i * Ns + j;
            const double q = q_a[k];
            if (q == 0) {
                dep[r] = false;
            } else {
                const double m = m_a[k], px = px_a[k], py = py_a[k], pz = pz_a[k];
                const double gm = sqrt(m * m + px * px + py * py + pz * pz);
                const double ig = 1.0 / gm;
                const double dro = q / (1 - pz * ig);
                const double rg = dro * ig;
                v[r][0] = dro; v[r][1] = px * rg; v[r][2] = py * rg; v[r][3] = pz * rg;
                check_range<Acc>(v[r][0], v[r][1], v[r][2], v[r][3], 1.0 / h, err);
                ix[r] = cell_of((x_init[k] + x_offt[k]) / h + 0.5, half_n, xl[r]);
                iy[r] = cell_of((y_init[k] + y_offt[k]) / h + 0.5, half_n, yl[r]);
                if (!(ix[r] >= 2 && ix[r] < N - 2 && iy[r] >= 2 && iy[r] < N - 2)) {
                    if (err) atomicOr(err, LCB_DEVERR_PLASMA_STENCIL);
                    dep[r] = false;
                }
            }
        }
    }
    // FP64: two particles in one cell add their contributions before the
    // shared atomic (one atomic per stencil point and quantity for both)
    const int lx = ix[0] - 2 - wx0, ly = iy[0] - 2 - wy0;
    const bool joint = sizeof(Acc) == sizeof(double) && !std::is_integral<Acc>::value &&
                       dep[0] && dep[1] && ix[0] == ix[1] && iy[0] == iy[1] &&
                       lx >= 0 && lx + 5 <= DEP_WX && ly >= 0 && ly + 5 <= DEP_WY;
    if (joint) {
        double ax[5], ay[5], bx[5], by[5];
        weights4(xl[0], ax); weights4(yl[0], ay);
        weights4(xl[1], bx); weights4(yl[1], by);
        const double ih = 1.0 / h;
#pragma unroll
        for (int b = 0; b < 5; b++) { ay[b] *= ih; by[b] *= ih; }
#pragma unroll
        for (int a = 0; a < 5; a++) {
            const double xa = ax[a] * ih, xb = bx[a] * ih;
#pragma unroll
            for (int b = 0; b < 5; b++) {
                const double wa = xa * ay[b], wb = xb * by[b];
                const int c = (lx + a) * DEP_WY + ly + b;
#pragma unroll
                for (int q = 0; q < 4; q++)
                    atomicAdd(sw + q * WSZ + c, Acc(fma(v[0][q], wa, v[1][q] * wb)));
            }
        }
    } else {
#pragma unroll
        for (int r = 0; r < DEP_PPT; r++)
            deposit_one<Acc, DEP_WX, DEP_WY>(sw, gro, gjx, gjy, gjz, N, h, wx0, wy0, dep[r], ix[r],
                                              iy[r], xl[r], yl[r], v[r][0], v[r][1], v[r][2], v[r][3]);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < WSZ; t += blockDim.x) {
        const int gx = wx0 + t / DEP_WY, gy = wy0 + t % DEP_WY;
        if (gx < 0 || gx >= N || gy < 0 || gy >= N) continue;
        const int64_t c = (int64_t)gx * N + gy;
        const Acc v0 = sw[t], v1 = sw[WSZ + t], v2 = sw[2 * WSZ + t], v3 = sw[3 * WSZ + t];
        if (v0 != Acc(0)) atomicAdd(gro + c, v0);
        if (v1 != Acc(0)) atomicAdd(gjx + c, v1);
        if (v2 != Acc(0)) atomicAdd(gjy + c, v2);
        if (v3 != Acc(0)) atomicAdd(gjz + c, v3);
    }
}

template <typename T>
static size_t deposit_smem_bytes()
{
    return (size_t)4 * DEP_WX * DEP_WY * sizeof(T);
}

// ---------------------------------------------------------------------------
// Fused predictor-corrector stage: K2 (move_smart) followed by K3 (deposit)
// of the same particles, and for the first stage of an xi step K1 (the
// free-streaming estimate) in front (move.py:169-313, weights.py:151-190).
// A block owns a lattice tile of TI x TJ particles.  The six field planes are
// staged in a shared-memory window around the tile for the midpoint gather;
// the moved particles are then sorted by cell (counts, a scan, records of
// their weights and values in shared memory), and their stencils summed in
// registers, a lane taking four cells along x and one quantity, before the
// sums go to HBM: about 16 additions per particle instead of 100 in shared
// memory (mixed precision with one particle per cell: in shared memory all the
// same, see Stage).  Particles whose stencil leaves a window use global memory.
// FP64 (FT = double): FP64 window, weights and sums.  Mixed precision
// (FT = float): coordinates and momenta stay FP64; the gather reads an FP32
// copy of the field window with FP32 weights; the deposit keeps FP64 weights, scales each particle's four
// values by 2^32 / h^2 once, and rounds every contribution to an integer with
// one FMA against FIX_MAGIC, so that the sums are exact.  FP64 sums round as
// they are added, in an order that the atomics decide: they repeat to their last
// bits only, a node's density to 1.0 of 2^-53 rms (0.7 with exact block sums of
// terms in units of 2^-56, which leave currents much smaller than the density
// less exact, and whose price for the cells in registers is 101 -> 125 us).
//
// What bounds it: latency, at the 16 warps per SM that the push's registers
// leave.  Adding every contribution to a shared window with 32-bit integer
// atomics (three words a sum in FP64, two in mixed precision) kept the
// shared-memory pipe 75 % busy and took 145 / 112 us for 929,296 particles
// behind a driver (FP64 / mixed, with the clearing of the planes); this form
// takes 101 / 94 us (with the background's copy folded into the clearing; 107
// before that).  Also measured, at 107 / 94: the contraction on the FP64 matrix
// instructions (121 / 114 us; m8n8k4 runs at a third of the vector rate for
// this shape), columns of cells walked with a sliding sum (119 / 107 us), and
// a deposit kernel of its own (121 / 125 us).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void weights4f(float x, float w[5])
{
    const float x2 = x * x, x3 = x2 * x, x4 = x3 * x;
    const float a = 0.5f - x, b = 0.5f + x;
    const float r6 = 1.0f / 6.0f, r24 = 1.0f / 24.0f;
    w[0] = a * a * a * a * r24;
    w[1] = 19 / 96.f - 11 / 24.f * x + x2 * 0.25f + x3 * r6 - x4 * r6;
    w[2] = 115 / 192.f - 5 / 8.f * x2 + x4 * 0.25f;
    w[3] = 19 / 96.f + 11 / 24.f * x + x2 * 0.25f - x3 * r6 - x4 * r6;
    w[4] = b * b * b * b * r24;
}

__device__ __forceinline__ void weights_of(float x, float w[5]) { weights4f(x, w); }
__device__ __forceinline__ void weights_of(double x, double w[5]) { weights4(x, w); }

// The five weights of a particle whose cell is s (0 or 1) cells past the
// origin of a six-point footprint, as six weights (zero outside).
template <typename W>
__device__ __forceinline__ void shift6(const W w[5], int s, W o[6])
{
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const W keep = k < 5 ? w[k] : W(0), moved = k > 0 ? w[k - 1] : W(0);
        o[k] = s ? moved : keep;
    }
}

// Packed FP32 pairs (sm_100 f32x2 arithmetic): two floats in one 64-bit
// register pair, and an FMA on both lanes.
__device__ __forceinline__ unsigned long long f32x2(float lo, float hi)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack_f32x2(unsigned long long v, float &lo, float &hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma_f32x2(unsigned long long a, unsigned long long b,
                                                        unsigned long long c)
{
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// Field window in shared memory: the six field values of a cell are stored
// together, so that one stencil point of the gather takes vector loads
// (FP32: a float4 of Ex, Ey, Ez, Bx and a float2 of By, Bz; FP64: three
// double2) instead of six scalar ones.  A quarter warp reads eight
// consecutive cells of a row (128 contiguous bytes per load), so rows need
// no padding.
template <typename FT> struct FieldWin;
template <> struct FieldWin<float> {
    static constexpr int bytes_per_cell = 24;
    __device__ static void put(unsigned char *w, int ncell, int c, const float v[6])
    {
        reinterpret_cast<float4 *>(w)[c] = make_float4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<float2 *>(w + 16 * ncell)[c] = make_float2(v[4], v[5]);
    }
    __device__ static void get(const unsigned char *w, int ncell, int c, float v[6])
    {
        const float4 a = reinterpret_cast<const float4 *>(w)[c];
        const float2 b = reinterpret_cast<const float2 *>(w + 16 * ncell)[c];
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y;
    }
};
template <> struct FieldWin<double> {
    static constexpr int bytes_per_cell = 48;
    __device__ static void put(unsigned char *w, int ncell, int c, const double v[6])
    {
        double2 *d = reinterpret_cast<double2 *>(w);
        d[c] = make_double2(v[0], v[1]);
        d[ncell + c] = make_double2(v[2], v[3]);
        d[2 * ncell + c] = make_double2(v[4], v[5]);
    }
    __device__ static void get(const unsigned char *w, int ncell, int c, double v[6])
    {
        const double2 *d = reinterpret_cast<const double2 *>(w);
        const double2 a = d[c], b = d[ncell + c], e = d[2 * ncell + c];
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = e.x; v[5] = e.y;
    }
};

// Midpoint gather of one particle from the window when the stencil fits in
// it, else from the FP64 planes in HBM; weights and sums in FT.
template <typename FT, int WX, int WY>
__device__ __forceinline__ void gather_one(const unsigned char *sf, const double *const *fld, int N,
                                           int wx0, int wy0, int ix, int iy, FT xl, FT yl,
                                           FT F[6])
{
    FT wx[5], wy[5];
    weights_of(xl, wx);
    weights_of(yl, wy);
    const int lx = ix - 2 - wx0, ly = iy - 2 - wy0;
    if (lx >= 0 && lx + 5 <= WX && ly >= 0 && ly + 5 <= WY) {
#pragma unroll
        for (int a = 0; a < 5; a++) {
#pragma unroll
            for (int b = 0; b < 5; b++) {
                const FT w = wx[a] * wy[b];
                FT v[6];
                FieldWin<FT>::get(sf, WX * WY, (lx + a) * WY + ly + b, v);
#pragma unroll
                for (int f = 0; f < 6; f++) F[f] += v[f] * w;
            }
        }
    } else {
#pragma unroll 1
        for (int a = 0; a < 5; a++) {
            const int row = (ix + a - 2) * N + iy - 2;
#pragma unroll
            for (int b = 0; b < 5; b++) {
                const FT w = wx[a] * wy[b];
#pragma unroll
                for (int f = 0; f < 6; f++) F[f] += (FT)__ldg(fld[f] + row + b) * w;
            }
        }
    }
}

// Values (in units of 2^-32, with the 1/h^2 of the weights) whose sums over
// a block's particles stay far inside the integers that fit FIX_MAGIC's
// binade (512 x 2^42 x 0.36 < 2^51); larger ones go straight to HBM.
constexpr double FIX_SHARED_LIMIT = 4398046511104.0;   // 2^42

__device__ __forceinline__ double max_abs4(const double (&v)[4])
{
    return fmax(fmax(fabs(v[0]), fabs(v[1])), fmax(fabs(v[2]), fabs(v[3])));
}

// One particle's deposit into HBM (weights.py:151-190 arithmetic): its
// stencil leaves the window, or its values the range that a block sums (FP64:
// infinities and NaN); sv: its values with the 1/h^2 (mixed: in fixed-point
// units).
template <typename FT, typename Acc>
__device__ __forceinline__ void deposit_direct(Acc *const (&g)[4], int N, int cx, int cy, double xl,
                                               double yl, const double (&sv)[4])
{
    double wx[5], wy[5];
    weights4(xl, wx);
    weights4(yl, wy);
    int64_t row = (int64_t)(cx - 2) * N + cy - 2;
#pragma unroll 1
    for (int a = 0; a < 5; a++) {
#pragma unroll
        for (int b = 0; b < 5; b++) {
            const double w = wx[0] * wy[b];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if constexpr (sizeof(FT) == 4) atomicAdd(g[q] + row + b, fix_bits(fma(sv[q], w, FIX_MAGIC)));
                else atomicAdd(g[q] + row + b, sv[q] * w);
            }
        }
#pragma unroll
        for (int k = 0; k < 4; k++) wx[k] = wx[k + 1];
        row += N;
    }
}

template <typename FT> struct StageAcc;
template <> struct StageAcc<float> { typedef fix_t type; };
template <> struct StageAcc<double> { typedef double type; };

// t = FIX_MAGIC + n, |n| < 2^41, into a sum of shared memory: its low 20 bits to
// an unsigned word, the rest to a signed one (32-bit integer atomics are native
// there, 64-bit ones are not).  Of a block's 512 particles neither word overflows.
__device__ __forceinline__ void shared_fix_add(unsigned *lo, int *hi, double t)
{
    const unsigned w0 = (unsigned)__double2loint(t);
    const unsigned w1 = (unsigned)(__double2hiint(t) - 0x43380000);   // (FIX_MAGIC's low word is zero)
    atomicAdd(lo, w0 & 0xFFFFFu);
    atomicAdd(hi, (int)__funnelshift_r(w0, w1, 20));
}

// Shape of a block of the fused stage: TI x TJ lattice particles, two per
// thread; a window of WX x WY nodes around them.  SHARED: the deposit adds to
// node sums in shared memory (mixed precision), else by cells in registers.
// With one particle per cell along an axis a lane would clear, walk and send 40
// sums for four particles: a mixed stage at 641 takes 80 us by cells, 65 us
// with the sums in shared memory (75 us with three blocks per SM and 80
// registers); at 321 32.3 and 28.5, at 91 19.5 and 18.  With four particles per
// cell the cells win: 105 us against 93 at 513; they also do where a tile's
// particles meet in few cells (all in one: 92 us against 160 at 513, one per
// cell).  FP64 has no exact sums of two words, and stays with the cells.
template <typename FT, int WX_, int WY_, bool SHARED_ = false> struct Stage {
    static constexpr bool SHARED = SHARED_;
    static constexpr int TI = 16, TJ = 32, WX = WX_, WY = WY_;
    static constexpr int NP = TI * TJ, THREADS = NP / 2, WARPS = THREADS / 32;
    static constexpr int WSZ = WX * WY;
    static constexpr int CX = WX - 4, CY = WY - 4, NC = CX * CY;   // cells of the window
    // cells along x that one lane of the deposit sums (4: 107 us a production
    // FP64 stage, 3: 109, 5: 111)
    static constexpr int XU = 4;
    // a particle's record for the deposit: five weights along x, five along
    // y, four values; the cells' columns a record apart (neighbouring lanes
    // write to and read from neighbouring columns, some 40 records away, and
    // shall not meet in a bank)
    static constexpr int RECORD = 14, SLOTS = NP + CY;
    static constexpr size_t field_bytes = (size_t)WSZ * FieldWin<FT>::bytes_per_cell;
    static constexpr size_t rec_bytes = (size_t)SLOTS * RECORD * sizeof(double);
    static constexpr size_t main_bytes = field_bytes > rec_bytes || SHARED ? field_bytes : rec_bytes;
    static constexpr size_t smem = main_bytes + (SHARED ? 8 * WSZ : NC + 1 + WARPS + 4) * sizeof(int);
};

template <typename S, typename FT, bool FIRST>
__global__ void __launch_bounds__(S::THREADS, 2)
k_move_deposit(int64_t n_per_sort, int Ns, int N, int fineness, double h, double xi_step, double boundary,
                  const double *__restrict__ Exf, const double *__restrict__ Eyf,
                  const double *__restrict__ Ezf, const double *__restrict__ Bxf,
                  const double *__restrict__ Byf, const double *__restrict__ Bzf,
                  const double *__restrict__ x_init, const double *__restrict__ y_init,
                  const double *__restrict__ xo_p, const double *__restrict__ yo_p,
                  const double *__restrict__ px_p, const double *__restrict__ py_p,
                  const double *__restrict__ pz_p, const double *__restrict__ q_p,
                  const double *__restrict__ m_a,
                  double *q_f, double *xo_f, double *yo_f, double *px_f, double *py_f,
                  double *pz_f, typename StageAcc<FT>::type *ro, typename StageAcc<FT>::type *jx,
                  typename StageAcc<FT>::type *jy, typename StageAcc<FT>::type *jz, int *err)
{
    // launched after its predecessor's tail (programmatic launch): no global
    // memory access before the wait
    pdl_wait();
    pdl_trigger();
    constexpr bool MIXED = sizeof(FT) == 4;
    typedef typename StageAcc<FT>::type Acc;
    constexpr int WX = S::WX, WY = S::WY, WSZ = S::WSZ, THREADS = S::THREADS;
    constexpr int CX = S::CX, NC = S::NC;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // the field window (FieldWin); after the gather, over it, the particles'
    // records in the order of their cells (SHARED: behind it, the node sums)
    unsigned char *sf = smem_raw;
    double *rec = reinterpret_cast<double *>(smem_raw);
    int *start = reinterpret_cast<int *>(smem_raw + S::main_bytes);   // [NC + 1] first records
    int *wsum = start + NC + 1, *box = wsum + S::WARPS;
    unsigned *sum_lo = reinterpret_cast<unsigned *>(smem_raw + S::main_bytes);   // SHARED: [4][WX][WY]
    int *sum_hi = reinterpret_cast<int *>(sum_lo + 4 * WSZ);
    const int s = blockIdx.z;
    const int64_t base = (int64_t)s * n_per_sort;
    const int half_n = N / 2;
    const int64_t NN = (int64_t)N * N;
    Acc *const g4[4] = {ro + s * NN, jx + s * NN, jy + s * NN, jz + s * NN};
    const double *const fld[6] = {Exf, Eyf, Ezf, Bxf, Byf, Bzf};
    const double ih = 1.0 / h;

    // Lanes take consecutive particles of a lattice row (coalesced loads;
    // neighbours in one cell read the same window values), a thread the rows
    // i and i + 1.  Tiles start on a lattice row whose cell also holds the
    // next row, so that a thread's two rows share a cell: when rows 0 and 1
    // sit in different cells the tiles are shifted up by one row (the grid has
    // one spare row of tiles for it).  The loads are issued for what the
    // package's own lattice needs (a shift with two particles per cell) before
    // the lattice is looked at, and again if it is another one.
    const int row = 2 * (threadIdx.x / S::TJ), j = blockIdx.x * S::TJ + threadIdx.x % S::TJ;
    int64_t kk[2];
    bool live[2], zero_p[2];
    double L_xo0[2], L_yo0[2], L_xi[2], L_yi[2], L_q[2], L_xof[2], L_yof[2];
    double L_m[2], L_px[2], L_py[2], L_pz[2], x0, y0;
    auto load = [&](int off) {
        const int i0 = blockIdx.y * S::TI - off;
#pragma unroll
        for (int p = 0; p < 2; p++) {
            const int i = i0 + row + p;
            live[p] = i >= 0 && i < Ns && j < Ns;
            const int64_t k = kk[p] = base + (int64_t)i * Ns + j;
            L_xo0[p] = L_yo0[p] = L_xi[p] = L_yi[p] = L_q[p] = L_xof[p] = L_yof[p] = 0;
            L_m[p] = L_px[p] = L_py[p] = L_pz[p] = 0;
            if (!live[p]) continue;
            L_xo0[p] = xo_p[k]; L_yo0[p] = yo_p[k];
            L_xi[p] = x_init[k]; L_yi[p] = y_init[k];
            if (FIRST) {
                L_m[p] = m_a[k]; L_px[p] = px_p[k]; L_py[p] = py_p[k]; L_pz[p] = pz_p[k];
                L_q[p] = q_p[k];
            } else {
                L_q[p] = q_f[k]; L_xof[p] = xo_f[k]; L_yof[p] = yo_f[k];
            }
        }
        // the tile's first particle
        const int ir = i0 < 0 ? 0 : i0;
        const int64_t k0 = base + (int64_t)(ir < Ns ? ir : 0) * Ns + blockIdx.x * S::TJ;
        x0 = x_init[k0]; y0 = y_init[k0];
    };
    // the field window, FILL_BATCH cells per thread at a time: the batch's
    // loads are all in flight before the first store to the window
    auto fill = [&](int wx0, int wy0) {
        constexpr int FILL_ITERS = (WSZ + THREADS - 1) / THREADS, FILL_BATCH = 3;
#pragma unroll
        for (int k0 = 0; k0 < FILL_ITERS; k0 += FILL_BATCH) {
            FT v[FILL_BATCH][6];
#pragma unroll
            for (int k = 0; k < FILL_BATCH; k++) {
                const int t = threadIdx.x + (k0 + k) * THREADS;
                const int gx = wx0 + t / WY, gy = wy0 + t % WY;
                const bool in = k0 + k < FILL_ITERS && t < WSZ && gx >= 0 && gx < N && gy >= 0 && gy < N;
                const int64_t g = (int64_t)gx * N + gy;
#pragma unroll
                for (int f = 0; f < 6; f++) v[k][f] = in ? (FT)__ldg(fld[f] + g) : FT(0);
            }
#pragma unroll
            for (int k = 0; k < FILL_BATCH; k++) {
                const int t = threadIdx.x + (k0 + k) * THREADS;
                if (k0 + k < FILL_ITERS && t < WSZ) FieldWin<FT>::put(sf, WSZ, t, v[k]);
            }
        }
    };
    // The window around the tile's first particle: where a lattice centred on
    // the grid with `fineness` particles per cell has it, so that the fields
    // are asked for together with the particles, and where it is, if that is
    // elsewhere.
    double dummy;
    auto origin = [&](double x) { return cell_of(x * ih + 0.5, half_n, dummy) - 2 - DEP_SLACK; };
    const double lat = h / fineness, mid = 0.5 * (Ns - 1);
    const int shift = fineness == 2;
    const double r0x = x_init[base], r1x = Ns > 1 ? x_init[base + Ns] : r0x;
    load(shift);
    const int px = origin((max((int)blockIdx.y * S::TI - shift, 0) - mid) * lat);
    const int py = origin(((int)blockIdx.x * S::TJ - mid) * lat);
    fill(px, py);
    for (int t = threadIdx.x; t < (S::SHARED ? 8 * WSZ : NC + 1); t += blockDim.x) start[t] = 0;
    if (!S::SHARED && threadIdx.x < 4) box[threadIdx.x] = (threadIdx.x & 1) ? -1 : 0x7fffffff;
    const int off = cell_of(r0x * ih + 0.5, half_n, dummy) != cell_of(r1x * ih + 0.5, half_n, dummy);
    if (off != shift) load(off);
    if ((int)blockIdx.y * S::TI - off >= Ns) return;
    const int wx0 = origin(x0), wy0 = origin(y0);
    if (wx0 != px || wy0 != py) fill(wx0, wy0);
    __syncthreads();

    // ---- phase 1: K1 (first stage) and the midpoint of each particle ----
    int ix[2], iy[2];
    FT xlf[2], ylf[2];
#pragma unroll
    for (int p = 0; p < 2; p++) {
        zero_p[p] = false;
        ix[p] = iy[p] = -1000;
        xlf[p] = ylf[p] = FT(0);
        if (!live[p]) continue;
        const int64_t k = kk[p];
        const double xo0 = L_xo0[p], yo0 = L_yo0[p];
        const double qk = L_q[p];
        double xof, yof;
        if (FIRST) {
            const double mk = L_m[p], opx = L_px[p], opy = L_py[p], opz = L_pz[p];
            xof = xo0; yof = yo0;
            if (mk != 0) {
                const double gm = sqrt_nr(mk * mk + opz * opz + opx * opx + opy * opy);
                const double adv = xi_step * rcp_nr(gm - opz);
                xof += opx * adv;
                yof += opy * adv;
            }
            if (qk == 0) {
                xo_f[k] = xof; yo_f[k] = yof;
                px_f[k] = opx; py_f[k] = opy; pz_f[k] = opz;
                q_f[k] = qk;
            }
        } else {
            xof = L_xof[p]; yof = L_yof[p];
        }
        if (qk == 0) { live[p] = false; continue; }
        double xh = L_xi[p] + (xo0 + xof) / 2;
        double yh = L_yi[p] + (yo0 + yof) / 2;
        bool z = false;
        if (xh > boundary)  { xh =  2 * boundary - xh; z = true; }
        if (xh < -boundary) { xh = -2 * boundary - xh; z = true; }
        if (yh > boundary)  { yh =  2 * boundary - yh; z = true; }
        if (yh < -boundary) { yh = -2 * boundary - yh; z = true; }
        zero_p[p] = z;
        double xl, yl;
        ix[p] = cell_of(xh * ih + 0.5, half_n, xl);
        iy[p] = cell_of(yh * ih + 0.5, half_n, yl);
        xlf[p] = (FT)xl; ylf[p] = (FT)yl;
        if (!(ix[p] >= 2 && ix[p] < N - 2 && iy[p] >= 2 && iy[p] < N - 2)) {
            if (err) atomicOr(err, LCB_DEVERR_PLASMA_STENCIL);
            ix[p] = -1000;  // no gather: zero fields, as in the reference's skip
        }
        // the push's mass and momenta, loaded while the gather runs
        if (!FIRST) { L_m[p] = m_a[k]; L_px[p] = px_p[k]; L_py[p] = py_p[k]; L_pz[p] = pz_p[k]; }
    }

    // ---- phase 2: gather ----
    // Three forms, chosen per warp so that a warp runs one of them: when
    // every lane's two particles share a cell (or the lane has none), the
    // 5 x 5 joint form; otherwise lanes whose particles sit in neighbouring
    // cells gather both over one 6 x 6 footprint (each particle's weights
    // zero outside its own 5 x 5), and the rest one particle at a time.  The
    // zero-weight terms leave each particle's sums unchanged.
    FT F0[6] = {0, 0, 0, 0, 0, 0}, F1[6] = {0, 0, 0, 0, 0, 0};
    {
        const int lx = ix[0] - 2 - wx0, ly = iy[0] - 2 - wy0;
        const bool joint = ix[0] >= 0 && ix[0] == ix[1] && iy[0] == iy[1] &&
                           lx >= 0 && lx + 5 <= WX && ly >= 0 && ly + 5 <= WY;
        const int mx = min(ix[0], ix[1]), my = min(iy[0], iy[1]);
        const int px0 = mx - 2 - wx0, py0 = my - 2 - wy0;
        const bool pair = ix[0] >= 0 && ix[1] >= 0 && abs(ix[1] - ix[0]) <= 1 &&
                          abs(iy[1] - iy[0]) <= 1 && px0 >= 0 && px0 + 6 <= WX &&
                          py0 >= 0 && py0 + 6 <= WY;
        const bool idle = ix[0] < 0 && ix[1] < 0;
        if (!__all_sync(0xffffffffu, joint || idle)) {
            if (pair && MIXED) {
                float ax[6], ay[6], bx[6], by[6], t[5];
                weights4f((float)xlf[0], t); shift6(t, ix[0] - mx, ax);
                weights4f((float)ylf[0], t); shift6(t, iy[0] - my, ay);
                weights4f((float)xlf[1], t); shift6(t, ix[1] - mx, bx);
                weights4f((float)ylf[1], t); shift6(t, iy[1] - my, by);
                unsigned long long A[3] = {0ull, 0ull, 0ull}, B[3] = {0ull, 0ull, 0ull};
#pragma unroll
                for (int a = 0; a < 6; a++) {
#pragma unroll
                    for (int b = 0; b < 6; b++) {
                        const float wa = ax[a] * ay[b], wb = bx[a] * by[b];
                        const unsigned long long wa2 = f32x2(wa, wa), wb2 = f32x2(wb, wb);
                        const int c = (px0 + a) * WY + py0 + b;
                        const float4 p = reinterpret_cast<const float4 *>(sf)[c];
                        const float2 q = reinterpret_cast<const float2 *>(sf + 16 * WSZ)[c];
                        const unsigned long long v3[3] = {f32x2(p.x, p.y), f32x2(p.z, p.w),
                                                          f32x2(q.x, q.y)};
#pragma unroll
                        for (int k = 0; k < 3; k++) {
                            A[k] = fma_f32x2(v3[k], wa2, A[k]);
                            B[k] = fma_f32x2(v3[k], wb2, B[k]);
                        }
                    }
                }
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    float lo, hi;
                    unpack_f32x2(A[k], lo, hi); F0[2 * k] = (FT)lo; F0[2 * k + 1] = (FT)hi;
                    unpack_f32x2(B[k], lo, hi); F1[2 * k] = (FT)lo; F1[2 * k + 1] = (FT)hi;
                }
            } else if (pair) {
                FT ax[6], ay[6], bx[6], by[6], t[5];
                weights_of(xlf[0], t); shift6(t, ix[0] - mx, ax);
                weights_of(ylf[0], t); shift6(t, iy[0] - my, ay);
                weights_of(xlf[1], t); shift6(t, ix[1] - mx, bx);
                weights_of(ylf[1], t); shift6(t, iy[1] - my, by);
#pragma unroll
                for (int a = 0; a < 6; a++) {
#pragma unroll
                    for (int b = 0; b < 6; b++) {
                        const FT wa = ax[a] * ay[b], wb = bx[a] * by[b];
                        FT v[6];
                        FieldWin<FT>::get(sf, WSZ, (px0 + a) * WY + py0 + b, v);
#pragma unroll
                        for (int f = 0; f < 6; f++) {
                            F0[f] += v[f] * wa;
                            F1[f] += v[f] * wb;
                        }
                    }
                }
            } else {
                if (ix[0] >= 0)
                    gather_one<FT, WX, WY>(sf, fld, N, wx0, wy0, ix[0], iy[0], xlf[0], ylf[0], F0);
                if (ix[1] >= 0)
                    gather_one<FT, WX, WY>(sf, fld, N, wx0, wy0, ix[1], iy[1], xlf[1], ylf[1], F1);
            }
        } else if (joint && MIXED) {
            // FP32: the window's float4 / float2 of a cell are register pairs
            // (Ex Ey)(Ez Bx)(By Bz), accumulated with packed f32x2 FMAs
            // (per lane the same rounding as the scalar FMAs)
            float ax[5], ay[5], bx[5], by[5];
            weights4f((float)xlf[0], ax); weights4f((float)ylf[0], ay);
            weights4f((float)xlf[1], bx); weights4f((float)ylf[1], by);
            unsigned long long A[3] = {0ull, 0ull, 0ull}, B[3] = {0ull, 0ull, 0ull};
            // stencil rows in a rolled loop, as in the deposit
            int row = lx * WY + ly;
#pragma unroll 1
            for (int a = 0; a < 5; a++) {
#pragma unroll
                for (int b = 0; b < 5; b++) {
                    const float wa = ax[0] * ay[b], wb = bx[0] * by[b];
                    const unsigned long long wa2 = f32x2(wa, wa), wb2 = f32x2(wb, wb);
                    const int c = row + b;
                    const float4 p = reinterpret_cast<const float4 *>(sf)[c];
                    const float2 q = reinterpret_cast<const float2 *>(sf + 16 * WSZ)[c];
                    const unsigned long long v3[3] = {f32x2(p.x, p.y), f32x2(p.z, p.w), f32x2(q.x, q.y)};
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        A[k] = fma_f32x2(v3[k], wa2, A[k]);
                        B[k] = fma_f32x2(v3[k], wb2, B[k]);
                    }
                }
#pragma unroll
                for (int k = 0; k < 4; k++) { ax[k] = ax[k + 1]; bx[k] = bx[k + 1]; }
                row += WY;
            }
#pragma unroll
            for (int k = 0; k < 3; k++) {
                float lo, hi;
                unpack_f32x2(A[k], lo, hi); F0[2 * k] = (FT)lo; F0[2 * k + 1] = (FT)hi;
                unpack_f32x2(B[k], lo, hi); F1[2 * k] = (FT)lo; F1[2 * k + 1] = (FT)hi;
            }
        } else if (joint) {
            FT ax[5], ay[5], bx[5], by[5];
            weights_of(xlf[0], ax); weights_of(ylf[0], ay);
            weights_of(xlf[1], bx); weights_of(ylf[1], by);
            int row = lx * WY + ly;
#pragma unroll 1
            for (int a = 0; a < 5; a++) {
#pragma unroll
                for (int b = 0; b < 5; b++) {
                    const FT wa = ax[0] * ay[b], wb = bx[0] * by[b];
                    FT v[6];
                    FieldWin<FT>::get(sf, WSZ, row + b, v);
#pragma unroll
                    for (int f = 0; f < 6; f++) {
                        F0[f] += v[f] * wa;
                        F1[f] += v[f] * wb;
                    }
                }
#pragma unroll
                for (int k = 0; k < 4; k++) { ax[k] = ax[k + 1]; bx[k] = bx[k + 1]; }
                row += WY;
            }
        }
    }

    // ---- phase 3: push (FP64) and the deposit values ----
    double sv[2][4];
    int cx[2], cy[2];
    double dxl[2], dyl[2];
#pragma unroll
    for (int p = 0; p < 2; p++) {
        cx[p] = -1000; cy[p] = 0; dxl[p] = dyl[p] = 0;
        sv[p][0] = sv[p][1] = sv[p][2] = sv[p][3] = 0;
        if (!live[p]) continue;
        const int64_t k = kk[p];
        const FT *Fp = p ? F1 : F0;
        const double Ex = Fp[0], Ey = Fp[1], Ez = Fp[2], Bx = Fp[3], By = Fp[4], Bz = Fp[5];
        const double mk = L_m[p], qk = L_q[p];
        const double opx = L_px[p], opy = L_py[p], opz = L_pz[p];
        const double xi0 = x_init[k], yi0 = y_init[k];
        double px = opx, py = opy, pz = opz;
        if (zero_p[p]) px = py = pz = 0;
        double gm, dpx, dpy, dpz;
#pragma unroll
        for (int it = 0; it < 2; it++) {
            gm = sqrt_nr(mk * mk + px * px + py * py + pz * pz);
            // f (E + v x B) with v = p / gm and f = q dxi / (1 - vz), as
            // q dxi (gm E + p x B) / (gm - pz): one quotient (algebraically
            // the reference's two, move.py:234-239)
            const double r = qk * xi_step * rcp_nr(gm - pz);
            dpx = r * (gm * Ex + py * Bz - pz * By);
            dpy = r * (gm * Ey - px * Bz + pz * Bx);
            dpz = r * (gm * Ez + px * By - py * Bx);
            px = opx + dpx * 0.5; py = opy + dpy * 0.5; pz = opz + dpz * 0.5;
        }
        gm = sqrt_nr(mk * mk + px * px + py * py + pz * pz);
        const double adv = xi_step * rcp_nr(gm - pz);
        double xo = xo_p[k] + px * adv;
        double yo = yo_p[k] + py * adv;
        px = opx + dpx; py = opy + dpy; pz = opz + dpz;
        double x = xi0 + xo, y = yi0 + yo;
        if (x > boundary)  { x =  2 * boundary - x; xo = x - xi0; px = py = pz = 0; }
        if (x < -boundary) { x = -2 * boundary - x; xo = x - xi0; px = py = pz = 0; }
        if (y > boundary)  { y =  2 * boundary - y; yo = y - yi0; px = py = pz = 0; }
        if (y < -boundary) { y = -2 * boundary - y; yo = y - yi0; px = py = pz = 0; }
        bool absorbed = false;
        if (x >= boundary || x <= -boundary || y >= boundary || y <= -boundary) {
            xo = yo = 0; px = py = pz = 0;
            absorbed = true;
        }
        xo_f[k] = xo; yo_f[k] = yo;
        px_f[k] = px; py_f[k] = py; pz_f[k] = pz;
        if (FIRST || absorbed) q_f[k] = absorbed ? 0.0 : qk;
        if (absorbed) continue;
        const double gd = sqrt_nr(mk * mk + px * px + py * py + pz * pz);
        // q / (1 - pz / gd) and p q / (gd - pz): one quotient (weights.py:
        // 164-168 has two)
        const double r = qk * rcp_nr(gd - pz);
        const double dro = r * gd, djx = r * px, djy = r * py, djz = r * pz;
        if (MIXED) check_range<fix_t>(dro, djx, djy, djz, ih, err);
        const int c_x = cell_of((xi0 + xo) * ih + 0.5, half_n, dxl[p]);
        const int c_y = cell_of((yi0 + yo) * ih + 0.5, half_n, dyl[p]);
        if (!(c_x >= 2 && c_x < N - 2 && c_y >= 2 && c_y < N - 2)) {
            if (err) atomicOr(err, LCB_DEVERR_PLASMA_STENCIL);
            continue;
        }
        cx[p] = c_x; cy[p] = c_y;
        // with the 1/h^2 of the weights; mixed: in units of 2^-32
        const double sc = (MIXED ? FIX_SCALE : 1.0) * ih * ih;
        sv[p][0] = dro * sc; sv[p][1] = djx * sc; sv[p][2] = djy * sc; sv[p][3] = djz * sc;
    }

    // ---- phase 4: deposit ----
    if constexpr (S::SHARED) {
        // Two particles in the same or neighbouring cells share a footprint of
        // 6 x 6 nodes, their terms added before the atomics (each still rounded
        // by itself); any other pair goes one by one.
        const int mx = min(cx[0], cx[1]), my = min(cy[0], cy[1]);
        const int lx = mx - 2 - wx0, ly = my - 2 - wy0;
        if (cx[0] >= 0 && cx[1] >= 0 && abs(cx[1] - cx[0]) <= 1 && abs(cy[1] - cy[0]) <= 1 && lx >= 0 &&
            lx + 6 <= WX && ly >= 0 && ly + 6 <= WY && max_abs4(sv[0]) < FIX_SHARED_LIMIT &&
            max_abs4(sv[1]) < FIX_SHARED_LIMIT) {
            double ax[6], ay[6], bx[6], by[6], t[5];
            weights4(dxl[0], t); shift6(t, cx[0] - mx, ax);
            weights4(dyl[0], t); shift6(t, cy[0] - my, ay);
            weights4(dxl[1], t); shift6(t, cx[1] - mx, bx);
            weights4(dyl[1], t); shift6(t, cy[1] - my, by);
            const bool wide = cy[0] != cy[1];
            int row = lx * WY + ly;
#pragma unroll 1
            for (int a = 0; a < 6; a++) {
#pragma unroll
                for (int b = 0; b < 6; b++) {
                    if (b == 5 && !wide) continue;
                    const double wa = ax[0] * ay[b], wb = bx[0] * by[b];
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        shared_fix_add(sum_lo + q * WSZ + row + b, sum_hi + q * WSZ + row + b,
                                       fma(sv[0][q], wa, fma(sv[1][q], wb, FIX_MAGIC)));
                }
#pragma unroll
                for (int k = 0; k < 5; k++) { ax[k] = ax[k + 1]; bx[k] = bx[k + 1]; }
                row += WY;
            }
        } else {
#pragma unroll
            for (int p = 0; p < 2; p++) {
                if (cx[p] < 0) continue;
                const int px = cx[p] - 2 - wx0, py = cy[p] - 2 - wy0;
                if (!(px >= 0 && px + 5 <= WX && py >= 0 && py + 5 <= WY && max_abs4(sv[p]) < FIX_SHARED_LIMIT)) {
                    deposit_direct<FT>(g4, N, cx[p], cy[p], dxl[p], dyl[p], sv[p]);
                    continue;
                }
                double wx[5], wy[5];
                weights4(dxl[p], wx);
                weights4(dyl[p], wy);
                int row = px * WY + py;
#pragma unroll 1
                for (int a = 0; a < 5; a++) {
#pragma unroll
                    for (int b = 0; b < 5; b++)
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            shared_fix_add(sum_lo + q * WSZ + row + b, sum_hi + q * WSZ + row + b,
                                           fma(sv[p][q], wx[0] * wy[b], FIX_MAGIC));
#pragma unroll
                    for (int k = 0; k < 4; k++) wx[k] = wx[k + 1];
                    row += WY;
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; q++)
            for (int t = threadIdx.x; t < WSZ; t += THREADS) {
                const unsigned lo = sum_lo[q * WSZ + t];
                const int hi = sum_hi[q * WSZ + t];
                if (lo || hi)
                    atomicAdd(g4[q] + (int64_t)(wx0 + t / WY) * N + wy0 + t % WY,
                              (Acc)(((long long)hi << 20) + lo));
            }
        return;
    }
    // Particles whose stencil lies in the window are counted per cell; the
    // others (and, in mixed precision, values outside the window's range) go
    // straight to HBM.
    int cell[2], rank[2];
    int bx0 = WX, bx1 = -1, by0 = WY, by1 = -1;
#pragma unroll
    for (int p = 0; p < 2; p++) {
        cell[p] = -1;
        if (cx[p] < 0) continue;
        const int lx = cx[p] - 2 - wx0, ly = cy[p] - 2 - wy0;
        if (lx >= 0 && lx + 5 <= WX && ly >= 0 && ly + 5 <= WY && max_abs4(sv[p]) < (MIXED ? FIX_SHARED_LIMIT : 1e200)) {
            cell[p] = ly * CX + lx;
            rank[p] = atomicAdd(start + 1 + cell[p], 1);
            bx0 = min(bx0, lx); bx1 = max(bx1, lx);
            by0 = min(by0, ly); by1 = max(by1, ly);
        } else {
            deposit_direct<FT>(g4, N, cx[p], cy[p], dxl[p], dyl[p], sv[p]);
        }
    }
    bx0 = __reduce_min_sync(0xffffffffu, bx0);
    bx1 = __reduce_max_sync(0xffffffffu, bx1);
    by0 = __reduce_min_sync(0xffffffffu, by0);
    by1 = __reduce_max_sync(0xffffffffu, by1);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0 && bx1 >= 0) {
        atomicMin(box, bx0); atomicMax(box + 1, bx1);
        atomicMin(box + 2, by0); atomicMax(box + 3, by1);
    }
    __syncthreads();   // counts complete; the field window is read no more

    // counts -> the cells' first records (start[c + 1] held cell c's count)
    {
        constexpr int E = (NC + THREADS - 1) / THREADS;
        int n[E], sum = 0;
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int c = threadIdx.x * E + e;
            n[e] = c < NC ? start[1 + c] : 0;
            sum += n[e];
        }
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        int at = incl - sum;
#pragma unroll
        for (int w = 0; w < THREADS / 32; w++)
            if (w < warp) at += wsum[w];
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int c = threadIdx.x * E + e;
            at += n[e];
            if (c < NC) start[1 + c] = at;
        }
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < 2; p++) {
        if (cell[p] < 0) continue;
        double w[10];
        weights4(dxl[p], w);
        weights4(dyl[p], w + 5);
        const int ly = cell[p] / CX, k = start[cell[p]] + rank[p] + ly;
        double2 *r = reinterpret_cast<double2 *>(rec + k * S::RECORD);
#pragma unroll
        for (int u = 0; u < 5; u++) r[u] = make_double2(w[2 * u], w[2 * u + 1]);
        r[5] = make_double2(sv[p][0], sv[p][1]);
        r[6] = make_double2(sv[p][2], sv[p][3]);
    }
    __syncthreads();

    // A lane takes XU cells along x and one quantity: the node sums of their
    // particles in registers, then to HBM.  Neighbouring lanes take the four
    // quantities (reading the same records), then the next column; the block's
    // lanes share out the box of cells in use.
    // mixed: a sum starts at FIX_MAGIC, where a unit in the last place is one,
    // so that every term is rounded to an integer as it is added.
    constexpr double ZERO = MIXED ? FIX_MAGIC : 0.0;
    constexpr int XU = S::XU;
    const int cx0 = box[0], nx = box[1] - cx0 + 1, cy0 = box[2], ny = box[3] - cy0 + 1;
    if (ny <= 0) return;
    const int q = threadIdx.x & 3;
    Acc *const gq = q == 0 ? g4[0] : q == 1 ? g4[1] : q == 2 ? g4[2] : g4[3];
    for (int u = threadIdx.x >> 2; u < ny * ((nx + XU - 1) / XU); u += THREADS / 4) {
        const int ux = u / ny, c = cy0 + u - ux * ny, x = cx0 + ux * XU;
        const int *col = start + c * CX + x;
        double acc[XU + 4][5];
#pragma unroll
        for (int a = 0; a < XU + 4; a++)
#pragma unroll
            for (int b = 0; b < 5; b++) acc[a][b] = ZERO;
        int k = col[0];
#pragma unroll
        for (int i = 0; i < XU; i++) {
            const int end = x + i < CX ? col[i + 1] : k;
            for (; k < end; k++) {
                const double *r = rec + (k + c) * S::RECORD;
                double w[10], t[5];
#pragma unroll
                for (int u = 0; u < 5; u++) {
                    const double2 d = reinterpret_cast<const double2 *>(r)[u];
                    w[2 * u] = d.x;
                    w[2 * u + 1] = d.y;
                }
                const double v = r[10 + q], *wx = w;
#pragma unroll
                for (int b = 0; b < 5; b++) t[b] = w[5 + b] * v;
#pragma unroll
                for (int a = 0; a < 5; a++)
#pragma unroll
                    for (int b = 0; b < 5; b++) acc[a + i][b] = fma(wx[a], t[b], acc[a + i][b]);
            }
        }
        Acc *out = gq + (int64_t)(wx0 + x) * N + wy0 + c;
#pragma unroll
        for (int a = 0; a < XU + 4; a++) {
#pragma unroll
            for (int b = 0; b < 5; b++) {
                const double t = acc[a][b];
                if (t != ZERO) {
                    if constexpr (MIXED) atomicAdd(out + b, fix_bits(t));
                    else atomicAdd(out + b, t);
                }
            }
            out += N;
        }
    }
}

template <typename S, typename FT, bool FIRST>
static int launch_move_deposit(const lcb_move_deposit_args *a,
                                    typename StageAcc<FT>::type *const out[4], cudaStream_t st)
{
    const dim3 grid((a->particles_side + S::TJ - 1) / S::TJ,
                    (a->particles_side + 1 + S::TI - 1) / S::TI,   // spare tile row
                    a->n_sorts);
    static std::atomic<unsigned long long> attr{0};
    {
        const cudaError_t e = ensure_smem(k_move_deposit<S, FT, FIRST>, S::smem, attr);
        if (e != cudaSuccess) return cuda_check(e, "move_deposit smem attribute");
    }
    const lcb_plasma_particles &p = a->prev, &f = a->full;
    const cudaError_t e = launch_after(
        k_move_deposit<S, FT, FIRST>, grid, dim3(S::THREADS), S::smem, st,
        a->n_per_sort, a->particles_side, a->grid_steps, a->lattice_fineness, a->h, a->xi_step, a->boundary,
        a->fields[0], a->fields[1], a->fields[2], a->fields[3], a->fields[4], a->fields[5],
        p.x_init, p.y_init, p.x_offt, p.y_offt, p.px, p.py, p.pz, p.q, p.m,
        f.q, f.x_offt, f.y_offt, f.px, f.py, f.pz, out[0], out[1], out[2], out[3], a->err);
    if (e != cudaSuccess) return cuda_check(e, "move_deposit launch");
    return LCB_OK;
}

// Window: the tile's cells (8 x TJ / 2 with two or more particles per cell,
// 16 x TJ with one) + 2 stencil + 4 slack on each side.
template <typename FT>
static int dispatch_move_deposit(const lcb_move_deposit_args *a,
                                      typename StageAcc<FT>::type *const out[4], cudaStream_t st)
{
    typedef Stage<FT, 20, 28> Two;
    typedef Stage<FT, 28, 44, sizeof(FT) == 4> One;
    if (a->lattice_fineness >= 2)
        return a->first ? launch_move_deposit<Two, FT, true>(a, out, st)
                        : launch_move_deposit<Two, FT, false>(a, out, st);
    return a->first ? launch_move_deposit<One, FT, true>(a, out, st)
                    : launch_move_deposit<One, FT, false>(a, out, st);
}

// Fixed-point sums (4 quantities x 2 columns x N*N) to the FP64 outputs;
// columns past n_sorts get the background ions (ro) or zero.  A thread
// takes one node of both columns.
__global__ void k_fix_finish(int64_t plane, int n_sorts, const fix_t *__restrict__ w,
                             const double *__restrict__ ro_initial, double *ro, double *jx,
                             double *jy, double *jz)
{
    pdl_wait();
    double *outs[4] = {ro, jx, jy, jz};
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < plane;
         t += (int64_t)gridDim.x * blockDim.x) {
        double v[8];
#pragma unroll
        for (int qd = 0; qd < 4; qd++) {
            v[2 * qd] = (double)(long long)w[qd * 2 * plane + t] * FIX_INV;
            v[2 * qd + 1] = n_sorts > 1 ? (double)(long long)w[qd * 2 * plane + plane + t] * FIX_INV
                          : ((qd == 0 && ro_initial) ? ro_initial[t] : 0.0);
        }
#pragma unroll
        for (int qd = 0; qd < 4; qd++) {
            outs[qd][t] = v[2 * qd];
            outs[qd][plane + t] = v[2 * qd + 1];
        }
    }
}

// Zero four regions of n 8-byte words each, or set the second half of the
// first to `background` (one kernel in the stream's chain of programmatic
// launches, where a memset or a copy would break it).
__global__ void __launch_bounds__(256) k_zero4(uint64_t *r0, uint64_t *r1, uint64_t *r2, uint64_t *r3,
                                               const uint64_t *background, int64_t n)
{
    pdl_wait();
    pdl_trigger();
    uint64_t *r[4] = {r0, r1, r2, r3};
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n;
         t += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
        for (int q = 0; q < 4; q++)
            r[q][t] = q == 0 && background && t >= n / 2 ? background[t - n / 2] : 0ull;
    }
}

static int grid_for(int64_t n, int threads);

static int zero4(void *r0, void *r1, void *r2, void *r3, int64_t n, cudaStream_t st,
                 const double *background = nullptr)
{
    const cudaError_t e = launch_after(k_zero4, dim3(grid_for(n, 256)), dim3(256), 0, st,
                                       static_cast<uint64_t *>(r0), static_cast<uint64_t *>(r1),
                                       static_cast<uint64_t *>(r2), static_cast<uint64_t *>(r3),
                                       reinterpret_cast<const uint64_t *>(background), n);
    if (e != cudaSuccess) return cuda_check(e, "zero launch");
    count_launch();
    return LCB_OK;
}

// Zero the columns of the fixed-point sums that the deposit adds to (the
// first column of each quantity, both with two sorts).
static int clear_fixed(fix_t *w, size_t plane, int n_sorts, cudaStream_t st)
{
    const int64_t n = (int64_t)(n_sorts > 1 ? 2 : 1) * plane;
    return zero4(w, w + 2 * plane, w + 4 * plane, w + 6 * plane, n, st);
}

static int grid_for(int64_t n, int threads)
{
    int64_t blocks = (n + threads - 1) / threads;
    const int64_t cap = (int64_t)sm_count() * 16;
    if (blocks > cap) blocks = cap;
    return (int)(blocks < 1 ? 1 : blocks);
}

// Mixed-precision deposit: fixed-point sums in the workspace, then one pass
// to the FP64 outputs (background column included).
static int deposit_fixed(int64_t n_per_sort, int n_sorts, int N, double h, int particles_side,
                         const double *x_init, const double *y_init, const double *x_offt,
                         const double *y_offt, const double *px, const double *py,
                         const double *pz, const double *q, const double *m,
                         const double *ro_initial, double *ro, double *jx, double *jy,
                         double *jz, void *workspace, size_t workspace_bytes, int *err,
                         cudaStream_t st)
{
    const size_t plane = (size_t)N * N;
    LCB_REQUIRE(workspace && workspace_bytes >= (size_t)8 * plane * sizeof(fix_t),
                "deposit workspace too small");
    fix_t *w = static_cast<fix_t *>(workspace);
    int rc = clear_fixed(w, plane, n_sorts, st);
    if (rc) return rc;
    cudaError_t e;
    if (n_per_sort > 0) {
        const dim3 grid((particles_side + DEP_TJ - 1) / DEP_TJ,
                        (particles_side + 1 + DEP_TI - 1) / DEP_TI, n_sorts);   // spare tile row
        const size_t sm = deposit_smem_bytes<fix_t>();
        static std::atomic<unsigned long long> attr{0};
        e = ensure_smem(k_deposit_tiled<fix_t>, sm, attr);
        if (e != cudaSuccess) return cuda_check(e, "deposit smem attribute");
        k_deposit_tiled<fix_t><<<grid, DEP_THREADS, sm, st>>>(
            n_per_sort, particles_side, N, h, x_init, y_init, x_offt, y_offt, px, py, pz, q, m,
            w, w + 2 * plane, w + 4 * plane, w + 6 * plane, err);
        LCB_LAUNCH_CHECK("k_deposit_tiled<fixed>");
    }
    e = launch_after(k_fix_finish, dim3(grid_for(plane, 256)), dim3(256), 0, st, (int64_t)plane,
                     n_sorts, (const fix_t *)w, ro_initial, ro, jx, jy, jz);
    if (e != cudaSuccess) return cuda_check(e, "fix finish launch");
    count_launch();
    return LCB_OK;
}

}  // namespace lcb

using namespace lcb;

extern "C" int lcb_plasma_move_wo_fields(
    int64_t n, double xi_step, const double *m, const double *x_offt_prev,
    const double *y_offt_prev, const double *px_prev, const double *py_prev,
    const double *pz_prev, const double *q_prev, double *x_offt_full,
    double *y_offt_full, double *px_full, double *py_full, double *pz_full,
    double *q_full, void *stream)
{
    LCB_REQUIRE(n >= 0, "n < 0");
    if (n == 0) return LCB_OK;
    k_move_wo_fields<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>(
        n, xi_step, m, x_offt_prev, y_offt_prev, px_prev, py_prev, pz_prev,
        q_prev, x_offt_full, y_offt_full, px_full, py_full, pz_full, q_full);
    LCB_LAUNCH_CHECK("k_move_wo_fields");
    return LCB_OK;
}

extern "C" int lcb_plasma_move_smart(
    int64_t n, double xi_step, double boundary, double h, int grid_steps,
    const double *Ex, const double *Ey, const double *Ez, const double *Bx,
    const double *By, const double *Bz, const double *x_init,
    const double *y_init, const double *x_offt_prev, const double *y_offt_prev,
    const double *px_prev, const double *py_prev, const double *pz_prev,
    const double *m, double *q_full, double *x_offt_full, double *y_offt_full,
    double *px_full, double *py_full, double *pz_full, int *err, void *stream)
{
    LCB_REQUIRE(n >= 0 && grid_steps >= 5, "bad sizes n=%lld N=%d", (long long)n, grid_steps);
    if (n == 0) return LCB_OK;
    k_move_smart<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>(
        n, xi_step, boundary, h, grid_steps, Ex, Ey, Ez, Bx, By, Bz, x_init,
        y_init, x_offt_prev, y_offt_prev, px_prev, py_prev, pz_prev, m, q_full,
        x_offt_full, y_offt_full, px_full, py_full, pz_full, err);
    LCB_LAUNCH_CHECK("k_move_smart");
    return LCB_OK;
}

extern "C" size_t lcb_plasma_deposit_workspace_bytes(int grid_steps, int precision)
{
    if (precision == LCB_PREC_MIXED)
        return (size_t)8 * grid_steps * grid_steps * sizeof(fix_t);
    return 0;
}

extern "C" int lcb_plasma_deposit(
    int64_t n_per_sort, int n_sorts, int grid_steps, double h, int particles_side,
    int precision, const double *x_init, const double *y_init,
    const double *x_offt, const double *y_offt, const double *px,
    const double *py, const double *pz, const double *q, const double *m,
    const double *ro_initial, double *ro, double *jx, double *jy, double *jz,
    void *workspace, size_t workspace_bytes, int *err, void *stream)
{
    const int N = grid_steps;
    LCB_REQUIRE(n_sorts >= 1 && n_sorts <= 2, "n_sorts must be 1 or 2");
    LCB_REQUIRE((int64_t)particles_side * particles_side == n_per_sort,
                "n_per_sort (%lld) must be particles_side^2 (%d^2)",
                (long long)n_per_sort, particles_side);
    LCB_REQUIRE(N >= 5, "grid_steps < 5");
    LCB_REQUIRE(precision == LCB_PREC_FP64 || precision == LCB_PREC_MIXED, "bad precision");
    cudaStream_t st = as_stream(stream);
    const size_t plane = (size_t)N * N;
    const size_t bytes = 2 * plane * sizeof(double);
    if (precision == LCB_PREC_MIXED)
        return deposit_fixed(n_per_sort, n_sorts, N, h, particles_side, x_init, y_init, x_offt,
                             y_offt, px, py, pz, q, m, ro_initial, ro, jx, jy, jz, workspace,
                             workspace_bytes, err, st);
    for (double *p : {ro, jx, jy, jz}) {
        cudaError_t e = cudaMemsetAsync(p, 0, bytes, st);
        if (e != cudaSuccess) return cuda_check(e, "memset currents");
    }
    if (n_per_sort > 0) {
        dim3 grid((particles_side + DEP_TJ - 1) / DEP_TJ,
                  (particles_side + 1 + DEP_TI - 1) / DEP_TI, n_sorts);   // spare tile row
        {
            const size_t sm = deposit_smem_bytes<double>();
            static std::atomic<unsigned long long> attr{0};
            const cudaError_t e = ensure_smem(k_deposit_tiled<double>, sm, attr);
            if (e != cudaSuccess) return cuda_check(e, "deposit smem attribute");
            k_deposit_tiled<double><<<grid, DEP_THREADS, sm, st>>>(
                n_per_sort, particles_side, N, h, x_init, y_init, x_offt, y_offt,
                px, py, pz, q, m, ro, jx, jy, jz, err);
            LCB_LAUNCH_CHECK("k_deposit_tiled<double>");
        }
    }
    if (ro_initial) {
        cudaError_t e = cudaMemcpyAsync(ro + plane, ro_initial, plane * sizeof(double),
                                        cudaMemcpyDeviceToDevice, st);
        if (e != cudaSuccess) return cuda_check(e, "copy ro_initial");
    }
    return LCB_OK;
}

extern "C" int lcb_plasma_move_deposit(const lcb_move_deposit_args *a, void *stream)
{
    LCB_REQUIRE(a, "args is NULL");
    const int N = a->grid_steps;
    LCB_REQUIRE(a->n_sorts >= 1 && a->n_sorts <= 2, "n_sorts must be 1 or 2");
    LCB_REQUIRE((int64_t)a->particles_side * a->particles_side == a->n_per_sort,
                "n_per_sort (%lld) must be particles_side^2 (%d^2)",
                (long long)a->n_per_sort, a->particles_side);
    LCB_REQUIRE(N >= 5, "grid_steps < 5");
    LCB_REQUIRE(a->precision == LCB_PREC_FP64 || a->precision == LCB_PREC_MIXED, "bad precision");
    for (int f = 0; f < 6; f++) LCB_REQUIRE(a->fields[f], "field plane %d is NULL", f);
    cudaStream_t st = as_stream(stream);
    const size_t plane = (size_t)N * N;
    if (a->precision == LCB_PREC_MIXED) {
        LCB_REQUIRE(a->workspace && a->workspace_bytes >= lcb_plasma_deposit_workspace_bytes(N, a->precision),
                    "deposit workspace too small");
        fix_t *w = static_cast<fix_t *>(a->workspace);
        const int rc0 = clear_fixed(w, plane, a->n_sorts, st);
        if (rc0) return rc0;
        if (a->n_per_sort > 0) {
            fix_t *const out[4] = {w, w + 2 * plane, w + 4 * plane, w + 6 * plane};
            const int rc = dispatch_move_deposit<float>(a, out, st);
            if (rc) return rc;
            LCB_LAUNCH_CHECK("k_move_deposit<float>");
        }
        const cudaError_t e = launch_after(k_fix_finish, dim3(grid_for(plane, 256)), dim3(256), 0, st,
                                           (int64_t)plane, a->n_sorts, (const fix_t *)w,
                                           a->ro_initial, a->ro, a->jx, a->jy, a->jz);
        if (e != cudaSuccess) return cuda_check(e, "fix finish launch");
        count_launch();
        return LCB_OK;
    }
    {
        // background ions go to the plane that no sort deposits into
        const int rc0 = zero4(a->ro, a->jx, a->jy, a->jz, 2 * (int64_t)plane, st,
                              a->n_sorts == 1 ? a->ro_initial : nullptr);
        if (rc0) return rc0;
    }
    if (a->n_per_sort > 0) {
        double *const out[4] = {a->ro, a->jx, a->jy, a->jz};
        const int rc = dispatch_move_deposit<double>(a, out, st);
        if (rc) return rc;
        LCB_LAUNCH_CHECK("k_move_deposit<double>");
    }
    if (a->ro_initial && a->n_sorts > 1) {
        cudaError_t e = cudaMemcpyAsync(a->ro + plane, a->ro_initial, plane * sizeof(double),
                                        cudaMemcpyDeviceToDevice, st);
        if (e != cudaSuccess) return cuda_check(e, "copy ro_initial");
    }
    return LCB_OK;
}
