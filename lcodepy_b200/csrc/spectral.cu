// Field solver by fast transforms: compute_fields (lcode/plasma3d/fields.py:
// 176-322) for grids whose number of intervals M = N - 1 factors into primes
// up to 13, in four kernels and FP64 throughout (in both precisions).
//
// A DCT-I of a line of N nodes is the discrete Fourier transform of its even
// extension to L = 2 M points, a DST-I (times -i) that of its odd extension.
// An even and an odd extension add up to one line that a reflection takes
// apart again, and a real and an imaginary part hold two of those, so one
// complex transform of length L carries four real ones.  The seven problems
// make two such units per line (S = DST-I, C = DCT-I):
//   unit 0: Ey (rows along y C, along x S), Bx (C, S), Ex (S, C), By (S, C)
//           z = (Ey + Ex) + i (Bx + By) along y
//   unit 1: Bz (C, C), Ez (S, S), Phi (S, S)
//           z = (Bz + Ez) + i Phi along y
// Along y the transform of unit 0 is Z_k = (Ey^ + By^) + i (Bx^ - Ex^), with
// Ey^, Bx^ even and By^, Ex^ odd in k.  Along x, By and Ex are the even ones
// and Ey and Bx the odd ones, so Z_k is already a packed line for the second
// transform: its even part less its odd part, the values of the mirrored
// nodes, is -Z_{L-k}.  For unit 1 it is +Z_{L-k}.  Nothing is taken apart
// between the two directions.  What a complex transform rounds is relative to
// the largest of the numbers that it carries, so each field enters multiplied
// by the power of two that brings its largest right-hand side near one, and
// leaves divided by it: a small field beside a large one keeps its own
// precision.  Phi is not a derivative of the currents as Bz and Ez are, and its
// low modes grow in the solution, so it enters smaller (spectral_solve).  The solver's spectral factor 1 / (lam_x +
// lam_y + shift) is the same for all the fields of a unit and even along the
// line, so it multiplies the packed spectrum as it is.
//
// The four: right-hand sides and each block's largest of every field; rows
// scaled, packed and transformed; transforms of the columns, spectral factor,
// and back; rows back, with the half/full combinations, the Dirichlet edges and
// Bz's mean removal.  One FP64 buffer Z[unit][i][s][k] is transformed in place
// (s = 0: index k, s = 1: index L - k of the line; of the right-hand sides s =
// 0 holds the even fields of node k and s = 1 the odd ones).  The scratch of a 513 grid is 16.8 MB and stays in
// L2.
//
// What bounds it: the inputs and outputs of a 513 grid are 97 MB (15 us at
// 6.45 TB/s), the transforms 0.2 GFLOP of FP64.  As dense products on the
// tensor cores (fields.cu, exact int8 slices) the same solve took 187 us in
// FP64 and 105 us in mixed precision (without Phi), against 50 and 46 us with
// these kernels (inputs that change from call to call): 36 slice products per
// multiply-add and N multiply-adds per node and transform cost more than log N
// FP64 operations on the vector units.  At 129 the solve went from 63 to 32 us
// (four launches instead of eleven), at 331, with the kernels for any length,
// from 84 to 52 us.  Finding the scales costs 0.5 to 1.5 us of each kernel of
// the rows and of the right-hand sides; without them (one rounding size for all
// the fields of a unit) 385 takes 48.3 us instead of 48.9, 451 80.2 instead of
// 81.0, 641 138.6 instead of 141.  The error against 64-bit sums is 6e-16 of each field (dense: 1e-14
// FP64, 1e-6 mixed, at 513).
#include <map>
#include <mutex>

#include "dft.cuh"
#include "spectral.cuh"

namespace lcb {

constexpr int SP_MAX_STAGES = 16;

// Radices of a transform of length L, in order, and where the twiddle
// factors of stage s > 0 start: entry (q - 1) Ns + k is exp(-2 pi i q k /
// (Ns R)), Ns the product of the radices before.
struct DftPlan {
    int L, n;
    int r[SP_MAX_STAGES];
    int off[SP_MAX_STAGES];
    int entries;
};

static void plan_offsets(DftPlan &p)
{
    int ns = p.r[0];
    p.entries = 0;
    p.off[0] = 0;
    for (int s = 1; s < p.n; s++) {
        p.off[s] = p.entries;
        p.entries += (p.r[s] - 1) * ns;
        ns *= p.r[s];
    }
}

// Fewest stages, then the smallest largest radix, by trying the radices from
// large to small.
static void plan_search(int left, int maxr, int depth, int *cur, int &best_n, int &best_max, int *best)
{
    if (left == 1) {
        int m = 0;
        for (int i = 0; i < depth; i++) m = cur[i] > m ? cur[i] : m;
        if (depth < best_n || (depth == best_n && m < best_max)) {
            best_n = depth;
            best_max = m;
            for (int i = 0; i < depth; i++) best[i] = cur[i];
        }
        return;
    }
    if (depth >= best_n || depth >= SP_MAX_STAGES) return;
    static const int radices[] = {16, 13, 12, 11, 10, 9, 8, 7, 6, 5, 4, 3, 2};
    for (int r : radices) {
        if (r > maxr || left % r) continue;
        cur[depth] = r;
        plan_search(left / r, r, depth + 1, cur, best_n, best_max, best);
    }
}

static bool make_plan(int L, DftPlan &p)
{
    int rest = L;
    for (int q : {2, 3, 5, 7, 11, 13})
        while (rest % q == 0) rest /= q;
    if (rest != 1 || L < 2) return false;
    int cur[SP_MAX_STAGES], best[SP_MAX_STAGES], bn = SP_MAX_STAGES + 1, bm = 99;
    plan_search(L, 16, 0, cur, bn, bm, best);
    if (bn > SP_MAX_STAGES) return false;
    p.L = L;
    p.n = bn;
    for (int i = 0; i < bn; i++) p.r[i] = best[i];
    plan_offsets(p);
    return true;
}

static DftPlan reversed(const DftPlan &p)
{
    DftPlan q = p;
    for (int i = 0; i < p.n; i++) q.r[i] = p.r[p.n - 1 - i];
    plan_offsets(q);
    return q;
}

// A line in shared memory has one spare slot behind every eight, so that the
// strided stores of a radix-8 or radix-16 step spread over the banks.
__host__ __device__ constexpr int sp_pad(int i) { return i + (i >> 3); }
// Slots of one line; a multiple of 8 plus 4, so that the two columns of a
// block start half the banks apart.
__host__ __device__ constexpr int sp_line(int L) { return (sp_pad(L) / 8) * 8 + 12; }

// Lengths L = 64 Q with their own kernels: three steps of radix 8, Q, 8 with
// sixteen elements per thread held in registers.
static int fixed_q(int L)
{
    return (L == 128 || L == 256 || L == 512 || L == 1024) ? L / 64 : 0;
}

struct OpsView {
    const double *f[2];        // spectral factors of the two units, N x N, symmetric
    const double2 *tw, *twr;   // twiddle factors of the plan, and of the reversed one
};

static size_t round256(size_t b) { return (b + 255) / 256 * 256; }

// The plan of a grid, found once per size (a solve asks for it on every call).
static bool plan_of(int N, DftPlan &p)
{
    const int L = 2 * (N - 1), q = fixed_q(L);
    if (q) {
        p.L = L; p.n = 3;
        p.r[0] = 8; p.r[1] = q; p.r[2] = 8;
        plan_offsets(p);
        return true;
    }
    static std::mutex mu;
    static std::map<int, DftPlan> plans;   // n = 0: the size has none
    std::lock_guard<std::mutex> lock(mu);
    auto it = plans.find(L);
    if (it == plans.end()) {
        DftPlan made;
        if (!make_plan(L, made)) made.n = 0;
        it = plans.emplace(L, made).first;
    }
    p = it->second;
    return p.n > 0;
}

static OpsView ops_view(const void *ops, int N, const DftPlan &p)
{
    const char *b = static_cast<const char *>(ops);
    const size_t plane = round256((size_t)N * N * sizeof(double));
    OpsView v;
    v.f[0] = reinterpret_cast<const double *>(b);
    v.f[1] = reinterpret_cast<const double *>(b + plane);
    v.tw = reinterpret_cast<const double2 *>(b + 2 * plane);
    v.twr = reinterpret_cast<const double2 *>(b + 2 * plane + round256(p.entries * sizeof(double2)));
    return v;
}

// Bytes of shared memory of the column kernel for lines of any length: two
// buffers for each of its columns.
static size_t any_smem(int L, int cols) { return (size_t)cols * 2 * sp_line(L) * sizeof(double2); }

bool spectral_grid(int N)
{
    if (N < 5 || N % 2 == 0 || N > 8192 || any_smem(2 * (N - 1), 1) > 220 * 1024) return false;
    DftPlan p;
    return plan_of(N, p);
}

size_t spectral_ops_bytes(int N)
{
    DftPlan p;
    if (!plan_of(N, p)) return 0;
    const DftPlan q = reversed(p);
    return 2 * round256((size_t)N * N * sizeof(double)) + round256(p.entries * sizeof(double2)) +
           round256(q.entries * sizeof(double2));
}

// Z[unit][i][s][k], then the column sums of Bz, then the blocks' largest
// exponents and the fields' scales.
__host__ __device__ constexpr int z_pitch(int N) { return N + 1; }
static size_t z_bytes(int N) { return round256((size_t)2 * N * 2 * z_pitch(N) * sizeof(double2)); }
static size_t colsum_bytes(int N) { return round256((size_t)N * sizeof(double)); }

// Most blocks of the right-hand sides' kernel: every block of the rows reads
// what all of them found.  A block has one patch of nodes up to this number of
// patches (grids up to 760 or so), several above; the loop over them costs 4 us
// of 57 at 513, which is why it has an instance of its own.
constexpr int SPR_BLOCKS = 16 * 148;

struct Scales {
    uint2 part[2][SPR_BLOCKS];   // per unit and block: biased exponents (A.x, B.x | A.y, B.y), 16 bits each
    double inv[2][4];            // per unit: what A.x, B.x, A.y, B.y are multiplied by on the way out, halved
};

size_t spectral_work_bytes(int N) { return z_bytes(N) + colsum_bytes(N) + round256(sizeof(Scales)); }

// 4 / h^2 sin^2(k pi / (2 (N - 1)))   (initialization.py:22-24)
__device__ double sp_lam(int k, int N, double h)
{
    const double s = sinpi((double)k / (2.0 * (N - 1)));
    return 4 / (h * h) * (s * s);
}

// The spectral factors: the mixed solver's 1 / (lam + lam + c) for unit 0,
// the Neumann solver's 1 / (lam + lam) for unit 1 (the Dirichlet solver's is
// its interior), with the transforms' norm.  Edges whose transforms vanish
// keep a finite factor.
__global__ void k_spectral_factors(int N, double h, double c, double *f0, double *f1)
{
    const double norm = (2.0 * (N - 1)) * (2.0 * (N - 1));
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < (int64_t)N * N;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int r = (int)(t / N), k = (int)(t % N);
        const double s = sp_lam(r, N, h) + sp_lam(k, N, h);
        f0[t] = (r == 0 && k == 0) ? 0.0 : 1 / (s + c) / norm;
        f1[t] = (r == 0 && k == 0) ? 0.0 : 1 / s / norm;
    }
}

__global__ void k_twiddles(DftPlan p, double2 *tw)
{
    int ns = p.r[0];
    for (int s = 1; s < p.n; s++) {
        const int R = p.r[s], m = ns * R;
        for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < (R - 1) * ns; e += gridDim.x * blockDim.x) {
            const int q = e / ns + 1, k = e % ns;
            const int t = (int)(((int64_t)q * k) % m);
            double sn, cs;
            sincospi(2.0 * t / m, &sn, &cs);
            tw[p.off[s] + e] = make_double2(cs, -sn);
        }
        ns = m;
    }
}

int spectral_ops_build(int N, double h, double c, void *ops, cudaStream_t st)
{
    DftPlan p;
    LCB_REQUIRE(plan_of(N, p), "grid_steps %d has no fast transform", N);
    const DftPlan q = reversed(p);
    const OpsView v = ops_view(ops, N, p);
    const int blocks = (int)(((int64_t)N * N + 255) / 256);
    k_spectral_factors<<<blocks, 256, 0, st>>>(N, h, c, const_cast<double *>(v.f[0]),
                                               const_cast<double *>(v.f[1]));
    LCB_LAUNCH_CHECK("k_spectral_factors");
    k_twiddles<<<(p.L + 255) / 256, 256, 0, st>>>(p, const_cast<double2 *>(v.tw));
    LCB_LAUNCH_CHECK("k_twiddles");
    k_twiddles<<<(p.L + 255) / 256, 256, 0, st>>>(q, const_cast<double2 *>(v.twr));
    LCB_LAUNCH_CHECK("k_twiddles");
    return LCB_OK;
}

// ---------------------------------------------------------------------------
// Right-hand sides (fields.py:112-230).  A block computes patches of 8 x 32
// nodes; the summed half-step densities and the full currents it
// differentiates are staged with a one-node halo in shared memory.  It leaves
// the largest exponent of each field among its patches.  Four blocks per SM:
// the registers of a fifth and sixth hold more of a thread's loads in flight
// (solve at 513: 50.2 us, 54.0 with 48 registers, 56.1 with 40).
// ---------------------------------------------------------------------------
struct SpRhsArgs {
    int N;
    double c, i2h, idxi, irb;                 // shift, 1 / (2 h), 1 / dxi, 1 / beam divisor
    const double *ro_f, *jx_f, *jy_f, *jz_f;  // full currents, n_f planes
    const double *ro_p, *jx_p, *jy_p, *jz_p;  // previous currents, n_p planes
    int n_f, n_p;
    const double *rb_full, *rb_prev;
    const double *Ex, *Ey, *Bx, *By;          // fields (Helmholtz term)
    int with_phi;
};

__device__ __forceinline__ double sp_sum(const double *a, int np, int64_t plane, int64_t i)
{
    return np == 2 ? a[i] + a[i + plane] : a[i];
}

constexpr int SPR_TY = 8, SPR_TX = 32;

// The biased exponents of two values, into a running maximum of 16 bits each
__device__ __forceinline__ void sp_largest(unsigned &m, double v0, double v1)
{
    const unsigned a = (unsigned)__double2hiint(v0) & 0x7ff00000u, b = (unsigned)__double2hiint(v1) & 0x7ff00000u;
    m = __vmaxu2(m, __byte_perm(a, b, 0x7632) >> 4);
}

template <bool MANY>
__global__ void __launch_bounds__(SPR_TX * SPR_TY, 4) k_rhs(SpRhsArgs a, int patches_x, int patches, double2 *Z,
                                                                Scales *sc)
{
    pdl_wait();
    pdl_trigger();
    __shared__ double s_ro[SPR_TY + 2][SPR_TX + 2], s_jz[SPR_TY + 2][SPR_TX + 2];
    __shared__ double s_jx[SPR_TY + 2][SPR_TX + 2], s_jy[SPR_TY + 2][SPR_TX + 2];
    __shared__ unsigned s_w[SPR_TY][4];
    const int N = a.N;
    const int64_t plane = (int64_t)N * N;
    const int tid = threadIdx.y * SPR_TX + threadIdx.x;
    unsigned top[4] = {0, 0, 0, 0};   // (Ey, Ex), (Bx, By), (Bz, Ez), (-, Phi): 16 bits each
    const int block = MANY ? blockIdx.x : blockIdx.y * gridDim.x + blockIdx.x;
    for (int patch = block; MANY ? patch < patches : patch == block; patch += MANY ? gridDim.x : 1) {
        const int i0 = (MANY ? patch / patches_x : blockIdx.y) * SPR_TY - 1;
        const int j0 = (MANY ? patch % patches_x : blockIdx.x) * SPR_TX - 1;
        if (MANY) __syncthreads();   // the last patch has been read
        for (int e = tid; e < (SPR_TY + 2) * (SPR_TX + 2); e += SPR_TX * SPR_TY) {
            const int li = e / (SPR_TX + 2), lj = e % (SPR_TX + 2);
            const int gi = i0 + li, gj = j0 + lj;
            double ro = 0, jz = 0, jx = 0, jy = 0;
            if (gi >= 0 && gi < N && gj >= 0 && gj < N) {
                const int64_t q = (int64_t)gi * N + gj;
                const double rbf = a.rb_full[q] * a.irb, rbp = a.rb_prev[q] * a.irb;
                // (full + rho_beam_full + prev + rho_beam_prev) / 2, fields.py:194-197
                ro = (sp_sum(a.ro_f, a.n_f, plane, q) + rbf + sp_sum(a.ro_p, a.n_p, plane, q) + rbp) / 2;
                jz = (sp_sum(a.jz_f, a.n_f, plane, q) + rbf + sp_sum(a.jz_p, a.n_p, plane, q) + rbp) / 2;
                jx = sp_sum(a.jx_f, a.n_f, plane, q);
                jy = sp_sum(a.jy_f, a.n_f, plane, q);
            }
            s_ro[li][lj] = ro; s_jz[li][lj] = jz; s_jx[li][lj] = jx; s_jy[li][lj] = jy;
        }
        __syncthreads();
        const int li = threadIdx.y + 1, lj = threadIdx.x + 1;
        const int i = i0 + li, j = j0 + lj;
        if (i >= N || j >= N) continue;
        const int64_t t = (int64_t)i * N + j;
        const bool in_x = i >= 1 && i < N - 1, in_y = j >= 1 && j < N - 1, inner = in_x && in_y;
        double dro_dx = 0, dro_dy = 0, djz_dx = 0, djz_dy = 0, bz = 0, ez = 0, phi = 0;
        if (inner) {
            dro_dx = (s_ro[li + 1][lj] - s_ro[li - 1][lj]) * a.i2h;
            dro_dy = (s_ro[li][lj + 1] - s_ro[li][lj - 1]) * a.i2h;
            djz_dx = (s_jz[li + 1][lj] - s_jz[li - 1][lj]) * a.i2h;
            djz_dy = (s_jz[li][lj + 1] - s_jz[li][lj - 1]) * a.i2h;
            const double djx_dy = s_jx[li][lj + 1] - s_jx[li][lj - 1];
            const double djy_dx = s_jy[li + 1][lj] - s_jy[li - 1][lj];
            const double djx_dx = s_jx[li + 1][lj] - s_jx[li - 1][lj];
            const double djy_dy = s_jy[li][lj + 1] - s_jy[li][lj - 1];
            bz = -(djx_dy - djy_dx) * a.i2h;
            ez = -(djx_dx + djy_dy) * a.i2h;
            if (a.with_phi) phi = sp_sum(a.ro_f, a.n_f, plane, t) - sp_sum(a.jz_f, a.n_f, plane, t);
        }
        const double djx_dxi = (sp_sum(a.jx_p, a.n_p, plane, t) - s_jx[li][lj]) * a.idxi;
        const double djy_dxi = (sp_sum(a.jy_p, a.n_p, plane, t) - s_jy[li][lj]) * a.idxi;
        // sources that their transforms do not see (the Dirichlet edges) are zero
        const double ex = in_y ? -(dro_dx - djx_dxi - a.c * a.Ex[t]) : 0.0;
        const double ey = in_x ? -(dro_dy - djy_dxi - a.c * a.Ey[t]) : 0.0;
        const double bx = in_x ? +(djz_dy - djy_dxi + a.c * a.Bx[t]) : 0.0;
        const double by = in_y ? -(djz_dx - djx_dxi - a.c * a.By[t]) : 0.0;
        const int pitch = z_pitch(N);
        double2 *z0 = Z + ((int64_t)i * 2) * pitch + j;
        double2 *z1 = z0 + (int64_t)N * 2 * pitch;
        z0[0] = make_double2(ey, bx);
        z0[pitch] = make_double2(ex, by);
        z1[0] = make_double2(bz, 0.0);
        z1[pitch] = make_double2(ez, phi);
        sp_largest(top[0], ey, ex); sp_largest(top[1], bx, by);
        sp_largest(top[2], bz, ez); sp_largest(top[3], 0.0, phi);
    }
    // the four words over the warp: half of them stay with each half of the
    // lanes, then one with each quarter
    const bool up = threadIdx.x & 16, up2 = threadIdx.x & 8;
    const unsigned a0 = __vmaxu2(top[up ? 2 : 0], __shfl_xor_sync(0xffffffffu, top[up ? 0 : 2], 16));
    const unsigned a1 = __vmaxu2(top[up ? 3 : 1], __shfl_xor_sync(0xffffffffu, top[up ? 1 : 3], 16));
    unsigned m = __vmaxu2(up2 ? a1 : a0, __shfl_xor_sync(0xffffffffu, up2 ? a0 : a1, 8));
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) m = __vmaxu2(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 7) == 0) s_w[threadIdx.y][threadIdx.x >> 3] = m;
    __syncthreads();
    if (tid < 4) {
        unsigned r = s_w[0][tid];
#pragma unroll
        for (int y = 1; y < SPR_TY; y++) r = __vmaxu2(r, s_w[y][tid]);
        reinterpret_cast<unsigned *>(&sc->part[tid >> 1][block])[tid & 1] = r;
    }
}

// What the fields of a unit are multiplied by on the way in (A.x, B.x, A.y,
// B.y), from the blocks' exponents; T threads, `red`: one word pair per warp.
template <int T>
__device__ __forceinline__ void sp_scales(Scales *sc, int unit, int blocks, int phi_shift, bool keep, uint2 *red,
                                          double (&f)[4])
{
    uint2 m = make_uint2(0, 0);
    for (int k0 = threadIdx.x; k0 < blocks; k0 += 8 * T) {
        uint2 p[8];
#pragma unroll
        for (int g = 0; g < 8; g++) p[g] = k0 + g * T < blocks ? sc->part[unit][k0 + g * T] : make_uint2(0, 0);
#pragma unroll
        for (int g = 0; g < 8; g++) {
            m.x = __vmaxu2(m.x, p[g].x);
            m.y = __vmaxu2(m.y, p[g].y);
        }
    }
    constexpr int W = T < 32 ? T : 32;
    constexpr unsigned lanes = T < 32 ? (1u << (T & 31)) - 1u : 0xffffffffu;
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) {
        m.x = __vmaxu2(m.x, __shfl_xor_sync(lanes, m.x, o));
        m.y = __vmaxu2(m.y, __shfl_xor_sync(lanes, m.y, o));
    }
    if (T > 32) {
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < T / 32; w++) {
            m.x = __vmaxu2(m.x, red[w].x);
            m.y = __vmaxu2(m.y, red[w].y);
        }
    }
    const unsigned e4[4] = {m.x & 0xffffu, m.x >> 16, m.y & 0xffffu, m.y >> 16};
#pragma unroll
    for (int q = 0; q < 4; q++) {
        // (a field of zeros or subnormal numbers stays as it is)
        const int e = e4[q] == 0 ? 1023 : min((int)e4[q] + (unit == 1 && q == 3 ? phi_shift : 0), 2045);
        f[q] = __hiloint2double((2046 - e) << 20, 0);
        if (keep && threadIdx.x == 0) sc->inv[unit][q] = 0.5 * __hiloint2double(e << 20, 0);
    }
}

// Nodes j and L - j of a row's line, packed from the fields of node j.
__device__ __forceinline__ void sp_pack(double2 A, double2 B, const double (&f)[4], double2 &zp, double2 &zm)
{
    const double ax = A.x * f[0], bx = B.x * f[1], ay = A.y * f[2], by = B.y * f[3];
    zp = make_double2(ax + bx, ay + by);
    zm = make_double2(ax - bx, ay - by);
}

// ---------------------------------------------------------------------------
// Outputs of one node (i, j) and unit from the line's values z_j and z_{L-j}.
// ---------------------------------------------------------------------------
struct SpOut {
    double *half[7], *full[7];   // Ex Ey Ez Bx By Bz Phi, NULL where not wanted
    const double *prev[6];
    const double *colsum;        // Bz's column sums, N values
};

// Half of what the fields of a unit are multiplied by on the way out, by their
// places (A.x, B.x, A.y, B.y).
__device__ __forceinline__ void sp_inverse(const Scales *sc, int unit, double (&u)[4])
{
#pragma unroll
    for (int q = 0; q < 4; q++) u[q] = sc->inv[unit][q];
}

// G nodes j[0 .. G-1] of row i (live ones: j >= 0).  The previous fields of
// all of them are read before the first store, so that their latencies
// overlap (a store may alias what is read next, as far as the compiler knows).
template <int G>
__device__ __forceinline__ void sp_emit(const SpOut &o, int unit, int N, int i, const int (&j)[G],
                                        const double2 (&zp)[G], const double2 (&zm)[G], double mean,
                                        const double (&u)[4])
{
    const int64_t t0 = (int64_t)i * N;
    const bool edge_x = i == 0 || i == N - 1;
    if (unit == 0) {
        // transverse: the solution is the half-step field, full = 2 half - prev
        constexpr int F[4] = {0, 1, 3, 4};
        double pv[4][G];
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int g = 0; g < G; g++) pv[q][g] = (o.full[F[q]] && j[g] >= 0) ? o.prev[F[q]][t0 + j[g]] : 0.0;
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int g = 0; g < G; g++) {
                if (j[g] < 0) continue;
                const double a = q < 2 ? zp[g].x : zp[g].y, b = q < 2 ? zm[g].x : zm[g].y;
                // Ex and By are the odd parts, Ey and Bx the even ones
                const double s = u[q == 0 ? 1 : q == 1 ? 0 : q];
                const double v = (q == 0 || q == 3) ? s * (a - b) : edge_x ? 0.0 : s * (a + b);
                if (o.full[F[q]]) o.full[F[q]][t0 + j[g]] = 2 * v - pv[q][g];
                if (o.half[F[q]]) o.half[F[q]][t0 + j[g]] = v;
            }
    } else {
        double pe[G], pb[G];
#pragma unroll
        for (int g = 0; g < G; g++) {
            pe[g] = (o.half[2] && j[g] >= 0) ? o.prev[2][t0 + j[g]] : 0.0;
            pb[g] = (o.half[5] && j[g] >= 0) ? o.prev[5][t0 + j[g]] : 0.0;
        }
#pragma unroll
        for (int g = 0; g < G; g++) {
            if (j[g] < 0) continue;
            const int64_t t = t0 + j[g];
            const double ez = edge_x ? 0.0 : u[1] * (zp[g].x - zm[g].x);
            const double bz = u[0] * (zp[g].x + zm[g].x) - mean;
            const double phi = edge_x ? 0.0 : u[3] * (zp[g].y - zm[g].y);
            if (o.full[2]) o.full[2][t] = ez;
            if (o.half[2]) o.half[2][t] = (ez + pe[g]) / 2;
            if (o.full[5]) o.full[5][t] = bz;
            if (o.half[5]) o.half[5][t] = (bz + pb[g]) / 2;
            if (o.half[6]) o.half[6][t] = phi;
            if (o.full[6]) o.full[6][t] = phi;
        }
    }
}

// Sum over all nodes of Bz from its column sums, the same in every block
// (fixed order); `red` holds one double per warp.
__device__ __forceinline__ double sp_total(const double *colsum, int N, double *red)
{
    double s = 0;
    for (int k = threadIdx.x; k < N; k += blockDim.x) s += colsum[k];
    const unsigned lanes = blockDim.x < 32 ? (1u << blockDim.x) - 1u : 0xffffffffu;
    const int width = blockDim.x < 32 ? blockDim.x : 32;
    for (int o = width / 2; o > 0; o >>= 1) s += __shfl_xor_sync(lanes, s, o);
    if (blockDim.x <= 32) return s;
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    s = 0;
    for (int w = 0; w < (int)(blockDim.x + 31) / 32; w++) s += red[w];
    return s;
}

// Weight of column k in the sum over a row's nodes of the values it
// transforms back to.
__device__ __forceinline__ double sp_col_weight(int k, int N)
{
    return k == 0 ? (double)N : k == N - 1 ? 1.0 : (k & 1) ? 0.0 : 2.0;
}

// Element idx of a row's line (slot 0 up to M, the mirrored half in slot 1).
__device__ __forceinline__ double2 row_get(const double2 *row, int pitch, int idx, int M)
{
    return idx <= M ? row[idx] : row[pitch + 2 * M - idx];
}

// ---------------------------------------------------------------------------
// Lines of any length: radices at run time, two shared buffers per line.
// ---------------------------------------------------------------------------
template <int R, typename Ld, typename St>
__device__ __forceinline__ void any_step(int L, int Ns, const double2 *tw, int t, int T, Ld ld, St st)
{
    const int nb = L / R;
    for (int b = t; b < nb; b += T) {
        double2 v[R];
#pragma unroll
        for (int q = 0; q < R; q++) v[q] = ld(b + q * nb);
        const int k = b % Ns;
        if (Ns > 1) {
#pragma unroll
            for (int q = 1; q < R; q++) v[q] = cmul(v[q], __ldg(tw + (q - 1) * Ns + k));
        }
        Dft<R>::run(v);
        const int o = (b / Ns) * Ns * R + k;
#pragma unroll
        for (int q = 0; q < R; q++) st(o + q * Ns, v[q]);
    }
}

template <typename Ld, typename St>
__device__ __forceinline__ void any_dispatch(int R, int L, int Ns, const double2 *tw, int t, int T, Ld ld,
                                             St st)
{
    switch (R) {
    case 2: any_step<2>(L, Ns, tw, t, T, ld, st); break;
    case 3: any_step<3>(L, Ns, tw, t, T, ld, st); break;
    case 4: any_step<4>(L, Ns, tw, t, T, ld, st); break;
    case 5: any_step<5>(L, Ns, tw, t, T, ld, st); break;
    case 6: any_step<6>(L, Ns, tw, t, T, ld, st); break;
    case 7: any_step<7>(L, Ns, tw, t, T, ld, st); break;
    case 8: any_step<8>(L, Ns, tw, t, T, ld, st); break;
    case 9: any_step<9>(L, Ns, tw, t, T, ld, st); break;
    case 10: any_step<10>(L, Ns, tw, t, T, ld, st); break;
    case 11: any_step<11>(L, Ns, tw, t, T, ld, st); break;
    case 12: any_step<12>(L, Ns, tw, t, T, ld, st); break;
    case 13: any_step<13>(L, Ns, tw, t, T, ld, st); break;
    case 16: any_step<16>(L, Ns, tw, t, T, ld, st); break;
    }
}

// The line in `a` through every step of the plan, between buffers a and b;
// returns the buffer that holds the result.  The caller synchronises before.
__device__ __forceinline__ double2 *any_line(const DftPlan &p, const double2 *tw, double2 *a, double2 *b,
                                             int t, int T)
{
    int ns = 1;
    for (int s = 0; s < p.n; s++) {
        const double2 *src = a;
        double2 *dst = b;
        any_dispatch(p.r[s], p.L, ns, tw + p.off[s], t, T, [&](int i) { return src[sp_pad(i)]; },
                     [&](int i, double2 v) { dst[sp_pad(i)] = v; });
        ns *= p.r[s];
        __syncthreads();
        double2 *x = a;
        a = b;
        b = x;
    }
    return a;
}

constexpr int SP_ANY_THREADS = 128;

// DIR 0: forward transform of row (blockIdx.x, unit blockIdx.y) in place;
// DIR 1: back to the nodes, and out.
template <int DIR>
__global__ void __launch_bounds__(SP_ANY_THREADS)
k_rows_any(int N, const __grid_constant__ DftPlan p, const double2 *tw, double2 *Z, SpOut o, Scales *sc, int blocks,
           int phi_shift)
{
    extern __shared__ __align__(16) double2 line[];
    __shared__ double red[SP_ANY_THREADS / 32];
    __shared__ uint2 red2[SP_ANY_THREADS / 32];
    pdl_wait();
    pdl_trigger();
    const int M = N - 1, L = p.L, pitch = z_pitch(N), i = blockIdx.x, unit = blockIdx.y;
    double2 *row = Z + ((int64_t)unit * N + i) * 2 * pitch;
    double2 *a = line, *b = line + sp_line(L);
    if (DIR == 0) {
        // four nodes of a thread on their way at a time, the first ones while
        // the scales are found (451: 83.0 us without, 81.0 with)
        double2 A[4], B[4];
        double f[4];
        for (int r = 0; r <= M; r += 4 * SP_ANY_THREADS) {
            const int j0 = r + threadIdx.x;
#pragma unroll
            for (int g = 0; g < 4; g++) {
                const int j = j0 + g * SP_ANY_THREADS;
                if (j <= M) { A[g] = row[j]; B[g] = row[pitch + j]; }
            }
            if (r == 0) sp_scales<SP_ANY_THREADS>(sc, unit, blocks, phi_shift, i == 0, red2, f);
#pragma unroll
            for (int g = 0; g < 4; g++) {
                const int j = j0 + g * SP_ANY_THREADS;
                if (j > M) continue;
                double2 zp, zm;
                sp_pack(A[g], B[g], f, zp, zm);
                a[sp_pad(j)] = zp;
                if (j > 0 && j < M) a[sp_pad(L - j)] = zm;
            }
        }
    } else {
        for (int idx = threadIdx.x; idx < L; idx += SP_ANY_THREADS)
            a[sp_pad(idx)] = cswap(row_get(row, pitch, idx, M));
    }
    __syncthreads();
    a = any_line(p, tw, a, b, threadIdx.x, SP_ANY_THREADS);
    if (DIR == 0) {
        for (int k = threadIdx.x; k <= M; k += SP_ANY_THREADS) {
            row[k] = a[sp_pad(k)];
            row[pitch + k] = a[sp_pad(k == 0 ? 0 : L - k)];
        }
    } else {
        double u[4];
        sp_inverse(sc, unit, u);
        const double mean = unit == 1 ? sp_total(o.colsum, N, red) / ((double)N * N) * (2 * u[0]) : 0.0;
        for (int j0 = threadIdx.x; j0 <= M; j0 += 4 * SP_ANY_THREADS) {
            int j[4];
            double2 zp[4], zm[4];
#pragma unroll
            for (int g = 0; g < 4; g++) {
                const int jj = j0 + g * SP_ANY_THREADS;
                j[g] = jj <= M ? jj : -1;
                zp[g] = cswap(a[sp_pad(jj <= M ? jj : 0)]);
                zm[g] = cswap(a[sp_pad(jj == 0 || jj > M ? 0 : L - jj)]);
            }
            sp_emit(o, unit, N, i, j, zp, zm, mean, u);
        }
    }
}

// COLS columns per block: transform along x, spectral factor, and back.
template <int COLS>
__global__ void __launch_bounds__(SP_ANY_THREADS)
k_cols_any(int N, const __grid_constant__ DftPlan p, const __grid_constant__ DftPlan pr, const double2 *tw,
           const double2 *twr, const double *f0, const double *f1, double2 *Z, double *colsum)
{
    extern __shared__ __align__(16) double2 line[];
    pdl_wait();
    pdl_trigger();
    constexpr int T = SP_ANY_THREADS / COLS;
    const int M = N - 1, L = p.L, pitch = z_pitch(N), unit = blockIdx.y;
    const int c = threadIdx.x % COLS, t = threadIdx.x / COLS;
    const int kc = blockIdx.x * COLS + c, k = kc < N ? kc : N - 1;
    const bool live = kc < N;
    double2 *a = line + 2 * c * sp_line(L), *b = a + sp_line(L);
    const double sgn = unit == 0 ? -1.0 : 1.0;
    double2 *col = Z + (int64_t)unit * N * 2 * pitch + k;
    const int m1 = (k == 0 || k == M) ? 0 : pitch;   // columns that are their own mirror image
    for (int i = t; i <= M; i += T) {
        const double2 zp = col[(int64_t)i * 2 * pitch], zm = col[(int64_t)i * 2 * pitch + m1];
        a[sp_pad(i)] = zp;
        if (i > 0 && i < M) a[sp_pad(L - i)] = make_double2(sgn * zm.x, sgn * zm.y);
    }
    __syncthreads();
    double2 *x = any_line(p, tw, a, b, t, T);
    const double *f = (unit == 0 ? f0 : f1) + (int64_t)k * N;
    double dc = 0;
    for (int i = t; i < L; i += T) {
        const double2 z = x[sp_pad(i)];
        const double g = f[i <= M ? i : L - i];
        if (i == 0) dc = g * z.x;
        x[sp_pad(i)] = make_double2(g * z.y, g * z.x);
    }
    __syncthreads();
    x = any_line(pr, twr, x, x == a ? b : a, t, T);
    if (!live) return;
    for (int i = t; i <= M; i += T) {
        const double2 zp = cswap(x[sp_pad(i)]), zm = cswap(x[sp_pad(i == 0 ? 0 : L - i)]);
        col[(int64_t)i * 2 * pitch] = zp;
        col[(int64_t)i * 2 * pitch + pitch] = make_double2(sgn * zm.x, sgn * zm.y);
    }
    // sum of the column's N nodes: the line's L values (its zeroth spectral
    // value) with the two end nodes, halved
    if (unit == 1 && t == 0)
        colsum[k] = 0.5 * sp_col_weight(k, N) * (L * dc + x[sp_pad(0)].y + x[sp_pad(M)].y);
}

// ---------------------------------------------------------------------------
// Lines of length L = 64 Q: steps of radix 8, Q, 8; T = L / 16 threads per
// line, a thread's sixteen elements in registers, one shared buffer.
// ---------------------------------------------------------------------------
template <int Q> struct Fix {
    static constexpr int L = 64 * Q, T = 4 * Q, M = 32 * Q, N = M + 1, NB = 16 / Q;
    static constexpr int B = 8 * Q;    // radix-8 butterflies of a step (two per thread)
};

// Element b + q B of a line of length 8 B is one of the first half (up to M =
// 4 B), or else the mirror image of element (B - b) + (7 - q) B.
__device__ __forceinline__ bool fix_direct(int b, int q) { return q < 4 || (q == 4 && b == 0); }

// Second butterfly of a thread in the last step: B - t, so that a thread
// holds both z_j and z_{L-j} (t = 0: B / 2, its own mirror image).
template <int Q> __device__ __forceinline__ int fix_b(int t, int n)
{
    return n == 0 ? t : (t == 0 ? Fix<Q>::B / 2 : Fix<Q>::B - t);
}

// The line of thread t: v[n][q] is element fix_b(t, n) + q B on the way in
// and on the way out.  `sync` is called by every thread of the block.
template <int Q>
__device__ __forceinline__ void fix_line(double2 (&v)[2][8], double2 *s, const double2 *tw, int t)
{
    using F = Fix<Q>;
#pragma unroll
    for (int n = 0; n < 2; n++) {
        Dft<8>::run(v[n]);
        const int o = 9 * fix_b<Q>(t, n);   // sp_pad(8 b)
#pragma unroll
        for (int q = 0; q < 8; q++) s[o + q] = v[n][q];
    }
    __syncthreads();
    double2 w[F::NB][Q];
#pragma unroll
    for (int n = 0; n < F::NB; n++) {
        const int b = t + n * F::T;
#pragma unroll
        for (int q = 0; q < Q; q++) w[n][q] = s[sp_pad(b) + 72 * q];
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < F::NB; n++) {
        const int b = t + n * F::T, k = b & 7;
#pragma unroll
        for (int q = 1; q < Q; q++) w[n][q] = cmul(w[n][q], __ldg(tw + (q - 1) * 8 + k));
        Dft<Q>::run(w[n]);
        const int o = (b >> 3) * 9 * Q + k;   // sp_pad((b / 8) 8 Q + k)
#pragma unroll
        for (int q = 0; q < Q; q++) s[o + 9 * q] = w[n][q];
    }
    __syncthreads();
    const double2 *t3 = tw + (Q - 1) * 8;
#pragma unroll
    for (int n = 0; n < 2; n++) {
        const int b = fix_b<Q>(t, n);
#pragma unroll
        for (int q = 0; q < 8; q++) v[n][q] = s[sp_pad(b) + 9 * Q * q];
#pragma unroll
        for (int q = 1; q < 8; q++) v[n][q] = cmul(v[n][q], __ldg(t3 + (q - 1) * F::B + b));
        Dft<8>::run(v[n]);
    }
}

template <int Q, int DIR>
__global__ void __launch_bounds__(Fix<Q>::T, Q >= 8 ? 512 / Fix<Q>::T : 1)
k_rows_fix(const double2 *tw, double2 *Z, SpOut o, Scales *sc, int blocks,
           int phi_shift)
{
    using F = Fix<Q>;
    __shared__ __align__(16) double2 s[sp_line(F::L)];
    __shared__ double red[(F::T + 31) / 32];
    __shared__ uint2 red2[(F::T + 31) / 32];
    pdl_wait();
    pdl_trigger();
    constexpr int M = F::M, N = F::N, pitch = z_pitch(N);
    const int i = blockIdx.x, unit = blockIdx.y, t = threadIdx.x;
    double2 *row = Z + ((int64_t)unit * N + i) * 2 * pitch;
    double2 v[2][8];
    double u[4], mean = 0;
    if (DIR == 0) {
        // the fields of nodes j = b + q B, which are packed into elements j and
        // L - j = (B - b) + (7 - q) B: a thread's own, as above
        double2 A[2][4], B[2][4], AM, BM;
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int j = fix_b<Q>(t, n) + q * F::B;
                A[n][q] = row[j];
                B[n][q] = row[pitch + j];
            }
        AM = BM = make_double2(0.0, 0.0);
        if (t == 0) { AM = row[M]; BM = row[pitch + M]; }
        sp_scales<F::T>(sc, unit, blocks, phi_shift, i == 0, red2, u);
        double2 m[2][4], zM, mM;
        sp_pack(AM, BM, u, zM, mM);
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int q = 0; q < 4; q++) sp_pack(A[n][q], B[n][q], u, v[n][q], m[n][q]);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            v[1][7 - q] = t > 0 ? m[0][q] : m[1][q];
            v[0][7 - q] = t > 0 ? m[1][q] : q < 3 ? m[0][q < 3 ? q + 1 : 0] : zM;
        }
    } else {
#pragma unroll
        for (int n = 0; n < 2; n++) {
            const int b = fix_b<Q>(t, n);
#pragma unroll
            for (int q = 0; q < 8; q++)
                v[n][q] = cswap(fix_direct(b, q) ? row[b + q * F::B] : row[pitch + F::B - b + (7 - q) * F::B]);
        }
        sp_inverse(sc, unit, u);
        if (unit == 1) mean = sp_total(o.colsum, N, red) / ((double)N * N) * (2 * u[0]);
    }
    fix_line<Q>(v, s, tw, t);
    if (DIR == 0) {
#pragma unroll
        for (int n = 0; n < 2; n++) {
            const int b = fix_b<Q>(t, n);
#pragma unroll
            for (int q = 0; q < 8; q++) {
                if (fix_direct(b, q)) row[b + q * F::B] = v[n][q];
                // (elements 0 and M are their own mirror images)
                if (q >= 4) row[pitch + F::B - b + (7 - q) * F::B] = v[n][q];
                if (q == 0 && b == 0) row[pitch] = v[n][q];
            }
        }
    } else {
        // element q of butterfly b mirrors element 7 - q of butterfly B - b;
        // butterfly 0 (thread 0) element 8 - q of itself, butterfly B / 2
        // element 7 - q of itself
#pragma unroll
        for (int n = 0; n < 2; n++) {
            int j[4];
            double2 zp[4], zm[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                j[q] = fix_b<Q>(t, n) + q * F::B;
                zp[q] = cswap(v[n][q]);
                zm[q] = cswap(t > 0 ? v[1 - n][7 - q] : n == 0 ? v[0][(8 - q) & 7] : v[1][7 - q]);
            }
            sp_emit(o, unit, N, i, j, zp, zm, mean, u);
        }
        if (t == 0) {
            const int j[1] = {M};
            const double2 z[1] = {cswap(v[0][4])};
            sp_emit(o, unit, N, i, j, z, z, mean, u);
        }
    }
}

// Two columns per block, lanes alternating between them (32-byte sectors).
template <int Q>
__global__ void __launch_bounds__(2 * Fix<Q>::T, Q >= 8 ? 512 / (2 * Fix<Q>::T) : 1)
k_cols_fix(const double2 *tw, const double2 *twr, const double *f0, const double *f1, double2 *Z, double *colsum)
{
    using F = Fix<Q>;
    __shared__ __align__(16) double2 s2[2 * sp_line(F::L)];
    pdl_wait();
    pdl_trigger();
    constexpr int M = F::M, L = F::L, N = F::N, pitch = z_pitch(N);
    const int unit = blockIdx.y, c = threadIdx.x & 1, t = threadIdx.x >> 1;
    const int kc = blockIdx.x * 2 + c, k = kc < N ? kc : N - 1;
    const bool live = kc < N;
    double2 *s = s2 + c * sp_line(L);
    const double sgn = unit == 0 ? -1.0 : 1.0;
    double2 *col = Z + (int64_t)unit * N * 2 * pitch + k;
    const int m1 = (k == 0 || k == M) ? 0 : pitch;
    double2 v[2][8];
#pragma unroll
    for (int n = 0; n < 2; n++) {
        const int b = fix_b<Q>(t, n);
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const bool direct = fix_direct(b, q);
            const double2 z = direct ? col[(b + q * F::B) * 2 * pitch]
                                     : col[(F::B - b + (7 - q) * F::B) * 2 * pitch + m1];
            v[n][q] = direct ? z : make_double2(sgn * z.x, sgn * z.y);
        }
    }
    fix_line<Q>(v, s, tw, t);
    const double *f = (unit == 0 ? f0 : f1) + (int64_t)k * N;
    const double dc = f[0] * v[0][0].x;   // used by t = 0
#pragma unroll
    for (int n = 0; n < 2; n++) {
        const int b = fix_b<Q>(t, n);
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const double g = f[fix_direct(b, q) ? b + q * F::B : F::B - b + (7 - q) * F::B];
            v[n][q] = make_double2(g * v[n][q].y, g * v[n][q].x);
        }
    }
    __syncthreads();   // the last step's reads are done
    // the reversed plan's factors are the same (8, Q, 8): as a table of their
    // own they are loaded again instead of being kept in 100 registers
    fix_line<Q>(v, s, twr, t);
    if (!live) return;
#pragma unroll
    for (int n = 0; n < 2; n++) {
        const int b = fix_b<Q>(t, n);
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const double2 z = cswap(v[n][q]), zs = make_double2(sgn * z.x, sgn * z.y);
            if (fix_direct(b, q)) col[(b + q * F::B) * 2 * pitch] = z;
            if (q >= 4) col[(F::B - b + (7 - q) * F::B) * 2 * pitch + pitch] = zs;
            if (q == 0 && b == 0) col[pitch] = zs;
        }
    }
    if (unit == 1 && t == 0)
        colsum[k] = 0.5 * sp_col_weight(k, N) * (L * dc + v[0][0].y + v[0][4].y);
}

template <int Q>
static int solve_fix(const OpsView &v, double2 *Z, double *colsum, const SpOut &o, Scales *sc, int blocks,
                     int phi_shift, cudaStream_t st)
{
    constexpr int N = Fix<Q>::N, T = Fix<Q>::T;
    cudaError_t e = launch_after(k_rows_fix<Q, 0>, dim3(N, 2), dim3(T), 0, st, v.tw, Z, o, sc, blocks, phi_shift);
    if (e != cudaSuccess) return cuda_check(e, "row transforms launch");
    count_launch();
    e = launch_after(k_cols_fix<Q>, dim3((N + 1) / 2, 2), dim3(2 * T), 0, st, v.tw, v.twr, v.f[0], v.f[1], Z,
                     colsum);
    if (e != cudaSuccess) return cuda_check(e, "column transforms launch");
    count_launch();
    e = launch_after(k_rows_fix<Q, 1>, dim3(N, 2), dim3(T), 0, st, v.tw, Z, o, sc, blocks, phi_shift);
    if (e != cudaSuccess) return cuda_check(e, "row transforms back launch");
    count_launch();
    return LCB_OK;
}

template <int COLS>
static int launch_cols_any(int N, const DftPlan &p, const DftPlan &pr, const OpsView &v, double2 *Z,
                           double *colsum, cudaStream_t st)
{
    const size_t sm = any_smem(p.L, COLS);
    static std::atomic<unsigned long long> attr{0};
    cudaError_t e = ensure_smem(k_cols_any<COLS>, 224 * 1024, attr);
    if (e != cudaSuccess) return cuda_check(e, "column transforms smem attribute");
    e = launch_after(k_cols_any<COLS>, dim3((N + COLS - 1) / COLS, 2), dim3(SP_ANY_THREADS), sm, st, N, p, pr,
                     v.tw, v.twr, v.f[0], v.f[1], Z, colsum);
    if (e != cudaSuccess) return cuda_check(e, "column transforms launch");
    count_launch();
    return LCB_OK;
}

template <int DIR>
static int launch_rows_any(int N, const DftPlan &p, const double2 *tw, double2 *Z, const SpOut &o, Scales *sc,
                           int blocks, int phi_shift, cudaStream_t st)
{
    static std::atomic<unsigned long long> attr{0};
    cudaError_t e = ensure_smem(k_rows_any<DIR>, 224 * 1024, attr);
    if (e != cudaSuccess) return cuda_check(e, "row transforms smem attribute");
    e = launch_after(k_rows_any<DIR>, dim3(N, 2), dim3(SP_ANY_THREADS), any_smem(p.L, 1), st, N, p, tw, Z, o,
                     sc, blocks, phi_shift);
    if (e != cudaSuccess) return cuda_check(e, "row transforms launch");
    count_launch();
    return LCB_OK;
}

int spectral_solve(const lcb_compute_fields_args *a, const void *ops, cudaStream_t st)
{
    const int N = a->grid_steps;
    DftPlan p;
    LCB_REQUIRE(plan_of(N, p), "grid_steps %d has no fast transform", N);
    const OpsView v = ops_view(ops, N, p);
    double2 *Z = static_cast<double2 *>(a->workspace);
    char *behind = static_cast<char *>(a->workspace) + z_bytes(N);
    double *colsum = reinterpret_cast<double *>(behind);
    Scales *sc = reinterpret_cast<Scales *>(behind + colsum_bytes(N));

    SpRhsArgs r;
    r.N = N;
    r.c = a->subtraction_coeff;
    // multiplications by reciprocals (at most an ulp from the quotients)
    r.i2h = 1.0 / (2.0 * a->h); r.idxi = 1.0 / a->xi_step; r.irb = 1.0 / a->rho_beam_divisor;
    r.ro_f = a->currents_full.ro; r.jx_f = a->currents_full.jx;
    r.jy_f = a->currents_full.jy; r.jz_f = a->currents_full.jz;
    r.n_f = a->currents_full.n_planes;
    r.ro_p = a->currents_prev.ro; r.jx_p = a->currents_prev.jx;
    r.jy_p = a->currents_prev.jy; r.jz_p = a->currents_prev.jz;
    r.n_p = a->currents_prev.n_planes;
    r.rb_full = a->rho_beam_full; r.rb_prev = a->rho_beam_prev;
    r.Ex = a->fields.f[0]; r.Ey = a->fields.f[1];
    r.Bx = a->fields.f[3]; r.By = a->fields.f[4];
    r.with_phi = (a->out_half.f[6] || a->out_full.f[6]) ? 1 : 0;
    const int patches_x = (N + SPR_TX - 1) / SPR_TX, patches_y = (N + SPR_TY - 1) / SPR_TY;
    const int patches = patches_x * patches_y, rounds = (patches + SPR_BLOCKS - 1) / SPR_BLOCKS;
    const int blocks = (patches + rounds - 1) / rounds;
    const dim3 threads(SPR_TX, SPR_TY);
    cudaError_t e = rounds == 1
        ? launch_after(k_rhs<false>, dim3(patches_x, patches_y), threads, 0, st, r, patches_x, patches, Z, sc)
        : launch_after(k_rhs<true>, dim3(blocks), threads, 0, st, r, patches_x, patches, Z, sc);
    if (e != cudaSuccess) return cuda_check(e, "rhs launch");
    count_launch();

    // The smallest Laplacian eigenvalue lets Phi's solution reach 0.074 W^2 of
    // its right-hand side, W the grid's width, where Bz's and Ez's stay near one
    // times theirs at the plasma's wave numbers: half of that factor (in powers
    // of two) in either direction.
    const double grow = 0.27 * (N - 1) * a->h;
    const int phi_shift = grow > 1 ? (int)lround(fmin(log2(grow), 40.0)) : 0;

    SpOut o;
    for (int f = 0; f < 7; f++) {
        o.half[f] = a->out_half.f[f];
        o.full[f] = a->out_full.f[f];
        if (f < 6) o.prev[f] = a->fields_prev.f[f];
    }
    o.colsum = colsum;
    switch (fixed_q(p.L)) {
    case 2: return solve_fix<2>(v, Z, colsum, o, sc, blocks, phi_shift, st);
    case 4: return solve_fix<4>(v, Z, colsum, o, sc, blocks, phi_shift, st);
    case 8: return solve_fix<8>(v, Z, colsum, o, sc, blocks, phi_shift, st);
    case 16: return solve_fix<16>(v, Z, colsum, o, sc, blocks, phi_shift, st);
    }
    const DftPlan pr = reversed(p);
    int rc = launch_rows_any<0>(N, p, v.tw, Z, o, sc, blocks, phi_shift, st);
    if (rc) return rc;
    // two columns per block read whole 32-byte sectors, but past L = 1100 two of
    // their buffers leave room for two blocks per SM only (whole solves with
    // two columns and with one: L = 768 48 / 52 us, 900 84 / 85, 1152 110 / 107,
    // 1280 175 / 139)
    rc = p.L < 1100 ? launch_cols_any<2>(N, p, pr, v, Z, colsum, st)
                    : launch_cols_any<1>(N, p, pr, v, Z, colsum, st);
    if (rc) return rc;
    return launch_rows_any<1>(N, p, v.tw, Z, o, sc, blocks, phi_shift, st);
}

}  // namespace lcb
