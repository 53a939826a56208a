// Comoving Poisson solve of the FP64 PM step: RHS assembly with the mean
// density removed (Gravity::solve_for_phi + CorrectRhsUsingOffset,
// Source/Gravity/Gravity.cpp:267-315, 1207-1244) and a geometric multigrid
// V-cycle with red-black Gauss-Seidel smoothing on the red-black split layout,
// the GB300-native replacement of the AMReX MLMG solve that
// Gravity::solve_with_MLMG (Gravity.cpp:1318-1416) calls.
//
// GB300 executes FP64 at a small fraction of its FP32 rate, so these kernels
// are written for the fewest FP64 instructions: the right-hand side is kept in
// smoother units (beta = h^2 rhs / 6, one fused multiply-add per Gauss-Seidel
// update), the trilinear prolongation weights are exact constants, and index
// arithmetic uses 3-D launch geometry instead of integer division.  Built with
// --fmad=false: only the explicit fma() calls fuse, in the same places the CPU
// oracle fuses, so both round identically.
#include "pm_cic.cuh"
#include "pm_cluster.cuh"
#include "pm_common.cuh"
#include "pm_sum6.cuh"
#include "pm_tail.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace nyxpm {

namespace {

constexpr int kThreads = 256;
constexpr double kSixth = 1.0 / 6.0;

__constant__ double kProlongW[8] = {0.421875, 0.140625, 0.140625, 0.046875,
                                    0.140625, 0.046875, 0.046875, 0.015625};

inline unsigned blocks_for(long long n, int t = kThreads)
{
    long long b = (n + t - 1) / t;
    return (unsigned)(b < 1 ? 1 : b);
}

__device__ __forceinline__ int wrap1(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

// ---------------------------------------------------------------------------
// RHS: canonical sum of (rho - mass_offset), then
// beta = ((((rho - mass_offset) - mean) * ggrav) * (1/a)) * (h^2/6)
// ---------------------------------------------------------------------------
// one warp per row: 32 strided lane partials, then a halving tree
__global__ void k_rowsum(int n, const double* __restrict__ rho, double mo, double* rows)
{
    pdl_wait();
    pdl_trigger();
    const long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= (long long)n * n) return;
    const double* r = rho + row * n;
    double s = 0.0;
    for (int i = lane; i < n; i += 32) s = s + (r[i] - mo);
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
        const double t = __shfl_down_sync(0xffffffffu, s, off);
        if (lane < off) s = s + t;
    }
    if (lane == 0) rows[row] = s;
}

// The n row sums of each plane in order, one plane per lane, then by whichever block ends
// last the n plane sums in order (ticket wraps to 0).  Two serial chains of n additions:
// the rows are read a 32 x 32 tile at a time, so that only the additions are serial.
// It also sets the norms that the solve collects by maximum to 0.
// (64^3: two launches, the loads in the chains, 5.4 + 4.6 us and the gap; this 6.)
__global__ void __launch_bounds__(32) k_mean(int n, double dx, double L, const double* __restrict__ rows,
                                             double* planes, unsigned* ticket, double* scal, unsigned long long* norms)
{
    __shared__ double tile[32][33];
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x, k0 = blockIdx.x * 32;
    if (blockIdx.x == 0 && lane < 2) norms[lane] = 0;
    double s = 0.0;
    for (int j0 = 0; j0 < n; j0 += 32) {
        double v[32];
#pragma unroll
        for (int p = 0; p < 32; ++p)
            v[p] = k0 + p < n && j0 + lane < n ? rows[(long long)(k0 + p) * n + j0 + lane] : 0.0;
        __syncwarp();
#pragma unroll
        for (int p = 0; p < 32; ++p) tile[p][lane] = v[p];
        __syncwarp();
        const int m = min(32, n - j0);
        for (int j = 0; j < m; ++j) s = s + tile[lane][j];
    }
    if (k0 + lane < n) planes[k0 + lane] = s;
    __threadfence();
    __syncwarp();
    unsigned last = 0;
    if (lane == 0) last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
    if (!__shfl_sync(0xffffffffu, last, 0)) return;
    __threadfence();
    s = 0.0;
    for (int q0 = 0; q0 < n; q0 += 32) {
        const double v = q0 + lane < n ? *(volatile double*)(planes + q0 + lane) : 0.0;
        const int m = min(32, n - q0);
        for (int q = 0; q < m; ++q) s = s + __shfl_sync(0xffffffffu, v, q);
    }
    if (lane == 0) scal[0] = (s * (dx * dx * dx)) / (L * L * L);
}

// the right-hand side and its maximum norm
__global__ void k_make_beta(int n, int split, const double* __restrict__ rho, double mo,
                            const double* __restrict__ scal, double ggrav, double ainv, double k0,
                            double* beta_r, double* beta_b, unsigned long long* norm)
{
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    unsigned long long u = 0;
    if (i < n && j < n) {
        const double mean = scal[0];
        const double v = rho[cidx(i, j, k, n)];
        const double beta = ((((v - mo) - mean) * ggrav) * ainv) * k0;
        *lv_ptr<double>(beta_r, beta_b, n, split, i, j, k) = beta;
        u = absbits(beta);
    }
    block_umax_store(u, norm);
}

// ---------------------------------------------------------------------------
// norms (max is order independent; non-negative doubles compare as their bits)
// ---------------------------------------------------------------------------
// neighbour sum in the oracle's order: x-, x+, y-, y+, z-, z+
__device__ __forceinline__ double nbr_sum(const LevelView& L, int i, int j, int k)
{
    const int n = L.n;
    const int im = i == 0 ? n - 1 : i - 1, ip = i == n - 1 ? 0 : i + 1;
    const int jm = j == 0 ? n - 1 : j - 1, jp = j == n - 1 ? 0 : j + 1;
    const int km = k == 0 ? n - 1 : k - 1, kp = k == n - 1 ? 0 : k + 1;
    double s = *lv_ptr<double>(L.phi_r, L.phi_b, n, L.split, im, j, k) +
               *lv_ptr<double>(L.phi_r, L.phi_b, n, L.split, ip, j, k);
    s = s + *lv_ptr<double>(L.phi_r, L.phi_b, n, L.split, i, jm, k);
    s = s + *lv_ptr<double>(L.phi_r, L.phi_b, n, L.split, i, jp, k);
    s = s + *lv_ptr<double>(L.phi_r, L.phi_b, n, L.split, i, j, km);
    s = s + *lv_ptr<double>(L.phi_r, L.phi_b, n, L.split, i, j, kp);
    return s;
}

// residual in smoother units: beta - (s/6 - phi)
__device__ __forceinline__ double resid_at(const LevelView& L, int i, int j, int k)
{
    const double s = nbr_sum(L, i, j, k);
    const double c = *lv_ptr<double>(L.phi_r, L.phi_b, L.n, L.split, i, j, k);
    const double b = *lv_ptr<double>(L.beta_r, L.beta_b, L.n, L.split, i, j, k);
    return b - fma(s, kSixth, -c);
}

// ||r_beta||_inf of a split level: one thread per (ih, j, k), both cells of the pair
__global__ void k_resnorm_split(LevelView L, unsigned long long* out)
{
    pdl_wait();
    pdl_trigger();
    const int half = L.n >> 1;
    const int ih = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    unsigned long long v = 0;
    if (ih < half && j < L.n) {
        const unsigned long long a = absbits(resid_at(L, 2 * ih, j, k));
        const unsigned long long b = absbits(resid_at(L, 2 * ih + 1, j, k));
        v = a > b ? a : b;
    }
    block_umax_store(v, out);
}

// Two compact cells 2 t2, 2 t2 + 1 of one colour of row (j, k) of a split level whose
// rows hold an even number of them: their neighbour sums from the other colour's array
// (16-byte loads; the two cells share one x neighbour), cell u of the pair being
// i = 4 t2 + 2 u + q.
__device__ __forceinline__ double2 pair_at(const double* a, unsigned at)
{
    return __ldg(reinterpret_cast<const double2*>(a + at));
}

__device__ __forceinline__ unsigned pair_row(unsigned n, unsigned j, unsigned k) { return (j + n * k) * (n >> 1); }

__device__ __forceinline__ double2 pair_sums(int n, const double* __restrict__ other, unsigned t2, int j, int k,
                                             int q, bool on_int)
{
    const unsigned half = (unsigned)n >> 1, ih = 2 * t2;
    const int jm = j == 0 ? n - 1 : j - 1, jp = j == n - 1 ? 0 : j + 1;
    const int km = k == 0 ? n - 1 : k - 1, kp = k == n - 1 ? 0 : k + 1;
    const unsigned r0 = pair_row(n, j, k);
    const double2 c = pair_at(other, r0 + ih);
    const double2 ym = pair_at(other, pair_row(n, jm, k) + ih), yp = pair_at(other, pair_row(n, jp, k) + ih);
    const double2 zm = pair_at(other, pair_row(n, j, km) + ih), zp = pair_at(other, pair_row(n, j, kp) + ih);
    const double e = __ldg(other + r0 + (q ? (ih + 2 == half ? 0u : ih + 2) : (ih == 0 ? half - 1 : ih - 1)));
    const double x0 = q ? c.x : e, x1 = q ? c.y : c.x, x2 = q ? e : c.y;
    const double nb0[6] = {x0, x1, ym.x, yp.x, zm.x, zp.x};
    const double nb1[6] = {x1, x2, ym.y, yp.y, zm.y, zp.y};
    return make_double2(sum6(nb0, on_int), sum6(nb1, on_int));
}

// k_resnorm_split by pairs of each colour
__global__ void __launch_bounds__(256) k_resnorm_split2(LevelView L, unsigned long long* out)
{
    pdl_wait();
    pdl_trigger();
    const int n = L.n;
    const unsigned t2 = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    unsigned long long v = 0;
    if (t2 < (unsigned)n >> 2 && j < n) {
        const unsigned t = pair_row(n, j, k) + 2 * t2;
        const bool on_int = sum6_on_int();
#pragma unroll
        for (int color = 0; color < 2; ++color) {
            const double2 s = pair_sums(n, color ? L.phi_r : L.phi_b, t2, j, k, (j + k + color) & 1, on_int);
            const double2 c = pair_at(color ? L.phi_b : L.phi_r, t), b = pair_at(color ? L.beta_b : L.beta_r, t);
            const unsigned long long r0 = absbits(b.x - fma(s.x, kSixth, -c.x));
            const unsigned long long r1 = absbits(b.y - fma(s.y, kSixth, -c.y));
            v = max(v, max(r0, r1));
        }
    }
    block_umax_store(v, out);
}

// the same over the red cells only: one thread per red cell of the split level
__global__ void k_resnorm_red(int n, const double* __restrict__ phi_r, const double* __restrict__ phi_b,
                              const double* __restrict__ beta_r, unsigned long long* out)
{
    pdl_wait();
    pdl_trigger();
    const int half = n >> 1;
    const int ih = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    unsigned long long v = 0;
    if (ih < half && j < n) {
        const int q = (j + k) & 1;  // the red cell of this pair is i = 2*ih + q
        const int ihm = q ? ih : (ih == 0 ? half - 1 : ih - 1);
        const int ihp = q ? (ih == half - 1 ? 0 : ih + 1) : ih;
        const int jm = j == 0 ? n - 1 : j - 1, jp = j == n - 1 ? 0 : j + 1;
        const int km = k == 0 ? n - 1 : k - 1, kp = k == n - 1 ? 0 : k + 1;
        const long long row = (long long)j + (long long)n * k;
        const long long t = row * half + ih;
        double s = phi_b[row * half + ihm] + phi_b[row * half + ihp];
        s = s + phi_b[((long long)jm + (long long)n * k) * half + ih];
        s = s + phi_b[((long long)jp + (long long)n * k) * half + ih];
        s = s + phi_b[((long long)j + (long long)n * km) * half + ih];
        s = s + phi_b[((long long)j + (long long)n * kp) * half + ih];
        v = absbits(beta_r[t] - fma(s, kSixth, -phi_r[t]));
    }
    block_umax_store(v, out);
}

// k_resnorm_red fused with the red half sweep that opens the next V-cycle: both
// need the same neighbour sum s of each red cell, so one pass gives the norm of
// beta - (s/6 - phi_red) and the next red value fma(s, 1/6, -beta), written to a
// spare red array (adopted only if the solve goes on) -- the same bits as the
// norm pass followed by the sweep
__global__ void k_resnorm_red_sweep(int n, const double* __restrict__ phi_r,
                                    const double* __restrict__ phi_b,
                                    const double* __restrict__ beta_r, double* __restrict__ next_r,
                                    unsigned long long* out)
{
    pdl_wait();
    pdl_trigger();
    const int half = n >> 1;
    const int ih = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    unsigned long long v = 0;
    if (ih < half && j < n) {
        const int q = (j + k) & 1;
        const int ihm = q ? ih : (ih == 0 ? half - 1 : ih - 1);
        const int ihp = q ? (ih == half - 1 ? 0 : ih + 1) : ih;
        const int jm = j == 0 ? n - 1 : j - 1, jp = j == n - 1 ? 0 : j + 1;
        const int km = k == 0 ? n - 1 : k - 1, kp = k == n - 1 ? 0 : k + 1;
        const long long row = (long long)j + (long long)n * k;
        const long long t = row * half + ih;
        double s = phi_b[row * half + ihm] + phi_b[row * half + ihp];
        s = s + phi_b[((long long)jm + (long long)n * k) * half + ih];
        s = s + phi_b[((long long)jp + (long long)n * k) * half + ih];
        s = s + phi_b[((long long)j + (long long)n * km) * half + ih];
        s = s + phi_b[((long long)j + (long long)n * kp) * half + ih];
        const double b = beta_r[t];
        v = absbits(b - fma(s, kSixth, -phi_r[t]));
        next_r[t] = fma(s, kSixth, -b);
    }
    block_umax_store(v, out);
}

// k_resnorm_red_sweep by pairs
__global__ void __launch_bounds__(256) k_resnorm_red_sweep2(int n, const double* __restrict__ phi_r,
                                                            const double* __restrict__ phi_b,
                                                            const double* __restrict__ beta_r,
                                                            double* __restrict__ next_r, unsigned long long* out)
{
    pdl_wait();
    pdl_trigger();
    const unsigned t2 = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    unsigned long long v = 0;
    if (t2 < (unsigned)n >> 2 && j < n) {
        const unsigned t = pair_row(n, j, k) + 2 * t2;
        const double2 s = pair_sums(n, phi_b, t2, j, k, (j + k) & 1, sum6_on_int());
        const double2 c = pair_at(phi_r, t), b = pair_at(beta_r, t);
        const unsigned long long r0 = absbits(b.x - fma(s.x, kSixth, -c.x));
        const unsigned long long r1 = absbits(b.y - fma(s.y, kSixth, -c.y));
        v = max(r0, r1);
        *reinterpret_cast<double2*>(next_r + t) = make_double2(fma(s.x, kSixth, -b.x), fma(s.y, kSixth, -b.y));
    }
    block_umax_store(v, out);
}

__global__ void k_resnorm_nat(LevelView L, unsigned long long* out)
{
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    unsigned long long v = 0;
    if (i < L.n && j < L.n) v = absbits(resid_at(L, i, j, k));
    block_umax_store(v, out);
}

// ---------------------------------------------------------------------------
// red-black Gauss-Seidel half sweep on a split level: one thread per cell of
// the colour being updated; reads the other colour's array, writes this one.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_gsrb(int n, int color, double* __restrict__ mine,
                                              const double* __restrict__ other,
                                              const double* __restrict__ beta)
{
    pdl_wait();
    pdl_trigger();
    const int half = n >> 1;
    const int ih = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    if (ih >= half || j >= n) return;
    const int q = (j + k + color) & 1;  // this cell is i = 2*ih + q
    const int ihm = q ? ih : (ih == 0 ? half - 1 : ih - 1);
    const int ihp = q ? (ih == half - 1 ? 0 : ih + 1) : ih;
    const int jm = j == 0 ? n - 1 : j - 1, jp = j == n - 1 ? 0 : j + 1;
    const int km = k == 0 ? n - 1 : k - 1, kp = k == n - 1 ? 0 : k + 1;
    const long long row = (long long)j + (long long)n * k;
    const long long t = row * half + ih;
    double s = other[row * half + ihm] + other[row * half + ihp];
    s = s + other[((long long)jm + (long long)n * k) * half + ih];
    s = s + other[((long long)jp + (long long)n * k) * half + ih];
    s = s + other[((long long)j + (long long)n * km) * half + ih];
    s = s + other[((long long)j + (long long)n * kp) * half + ih];
    mine[t] = fma(s, kSixth, -beta[t]);
}

// The red half sweep from phi = 0: fma(0, 1/6, -beta) = 0 - beta by the sign bit (+0 for either
// zero), two cells per thread.
__global__ void __launch_bounds__(256) k_gsrb_zero(unsigned pairs, const ulonglong2* __restrict__ beta,
                                                   ulonglong2* __restrict__ phi)
{
    pdl_wait();
    pdl_trigger();
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= pairs) return;
    const ulonglong2 b = __ldg(beta + t);
    auto minus = [](unsigned long long u) { return (u << 1) == 0 ? 0ULL : u ^ (1ULL << 63); };
    phi[t] = make_ulonglong2(minus(b.x), minus(b.y));
}

// k_gsrb by pairs
__global__ void __launch_bounds__(256) k_gsrb2(int n, int color, double* __restrict__ mine,
                                               const double* __restrict__ other,
                                               const double* __restrict__ beta)
{
    pdl_wait();
    pdl_trigger();
    const unsigned t2 = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    if (t2 >= (unsigned)n >> 2 || j >= n) return;
    const unsigned t = pair_row(n, j, k) + 2 * t2;
    const double2 b = pair_at(beta, t);
    const double2 s = pair_sums(n, other, t2, j, k, (j + k + color) & 1, sum6_on_int());
    *reinterpret_cast<double2*>(mine + t) = make_double2(fma(s.x, kSixth, -b.x), fma(s.y, kSixth, -b.y));
}

// a coarse cell's right-hand side and the phi it starts from
__device__ __forceinline__ void restrict_store(const LevelView& Cv, int I, int J, int K, double beta, int open)
{
    *lv_ptr<double>(Cv.beta_r, Cv.beta_b, Cv.n, Cv.split, I, J, K) = beta;
    if (open && ((I + J + K) & 1)) return;
    *lv_ptr<double>(Cv.phi_r, Cv.phi_b, Cv.n, Cv.split, I, J, K) = open ? fma(0.0, kSixth, -beta) : 0.0;
}

// coarse beta = 1/2 of the 8 fine residuals (summed dk, dj, di); coarse phi = 0
// RED = 1 after pre-smoothing (the last half sweep was black): the black
// children's residuals are round-off by construction and count as 0, so the 4 red
// children (di + dj + dk even) are summed in the same (dk, dj, di) order -- half
// the FP64 residual work
// open: the coarse level is smoothed from 0 next, and its opening red half sweep, of black
// neighbours that are 0, is made here in place of a launch (the black half sweep after it
// overwrites the black cells unread): three FP64 steps at 256^3 86.2 -> 85.2 ms
template <int RED>
__global__ void k_restrict(LevelView F, LevelView Cv, int open)
{
    pdl_wait();
    pdl_trigger();
    const int nc = Cv.n;
    const int I = blockIdx.x * blockDim.x + threadIdx.x;
    const int J = blockIdx.y * blockDim.y + threadIdx.y;
    const int K = blockIdx.z;
    if (I >= nc || J >= nc) return;
    double s = 0.0;
#pragma unroll
    for (int dk = 0; dk < 2; ++dk)
#pragma unroll
        for (int dj = 0; dj < 2; ++dj)
#pragma unroll
            for (int di = 0; di < 2; ++di)
                if (!RED || ((di + dj + dk) & 1) == 0)
                    s = s + resid_at(F, 2 * I + di, 2 * J + dj, 2 * K + dk);
    restrict_store(Cv, I, J, K, s * 0.5, open);
}

// k_restrict<1> by pairs: two coarse cells 2 t2, 2 t2 + 1 of a row per thread, whose
// red children in a fine row are the row's red pair 2 t2, 2 t2 + 1
__global__ void __launch_bounds__(256) k_restrict_red2(LevelView F, LevelView Cv, int open)
{
    pdl_wait();
    pdl_trigger();
    const int n = F.n, nc = Cv.n;
    const unsigned t2 = blockIdx.x * blockDim.x + threadIdx.x;
    const int J = blockIdx.y * blockDim.y + threadIdx.y;
    const int K = blockIdx.z;
    if (t2 >= (unsigned)nc >> 1 || J >= nc) return;
    const bool on_int = sum6_on_int();
    double2 acc = make_double2(0.0, 0.0);
#pragma unroll 1
    for (int d = 0; d < 4; ++d) {
        const int j = 2 * J + (d & 1), k = 2 * K + (d >> 1);
        const unsigned t = pair_row(n, j, k) + 2 * t2;
        const double2 b = pair_at(F.beta_r, t), c = pair_at(F.phi_r, t);
        const double2 s = pair_sums(n, F.phi_b, t2, j, k, (j + k) & 1, on_int);
        acc.x = acc.x + (b.x - fma(s.x, kSixth, -c.x));
        acc.y = acc.y + (b.y - fma(s.y, kSixth, -c.y));
    }
    const int I = 2 * (int)t2;
    restrict_store(Cv, I, J, K, acc.x * 0.5, open);
    restrict_store(Cv, I + 1, J, K, acc.y * 0.5, open);
}

// The black children's corrections of two coarse cells of a row per thread, for a split fine
// level of n % 8 == 0 over a split coarse level, when post-smoothing follows (its first half
// sweep overwrites the red cells unread).  Bound by the FP64 pipe: a black child takes eight
// fused multiply-adds and an addition, in the order nearest row and plane first, the x pair
// innermost.  The four black children of a coarse cell (odd dx + dy + dz) have the first product
// in common, two each the second term, so a coarse cell takes 30 instead of 36, the product on
// the integer pipe.  Four steps at 160^3 34.9 -> 30.8 ms, at 256^3 106.3 -> 103.3, against a thread
// for four black cells of a fine row.
__global__ void __launch_bounds__(256) k_prolong_black(LevelView Cv, LevelView F)
{
    pdl_wait();
    pdl_trigger();
    const int nc = Cv.n;
    const unsigned ch = (unsigned)nc >> 1, t2 = blockIdx.x * blockDim.x + threadIdx.x;   // coarse cells 2 t2, 2 t2 + 1
    const int J = blockIdx.y * blockDim.y + threadIdx.y;
    const int K = blockIdx.z;
    if (t2 >= ch || J >= nc) return;
    const int Jr[3] = {J, J == 0 ? nc - 1 : J - 1, J + 1 == nc ? 0 : J + 1};
    const int Kr[3] = {K, K == 0 ? nc - 1 : K - 1, K + 1 == nc ? 0 : K + 1};
    double v[3][4];   // a plane's rows J, J - 1, J + 1 at x = 2 t2 - 1 .. 2 t2 + 2
    auto load = [&](int kk) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const bool even_red = ((Jr[a] + Kr[kk]) & 1) == 0;
            const unsigned row = ((unsigned)Jr[a] + (unsigned)nc * (unsigned)Kr[kk]) * ch;
            const double* ev = (even_red ? Cv.phi_r : Cv.phi_b) + row;
            const double* od = (even_red ? Cv.phi_b : Cv.phi_r) + row;
            v[a][0] = __ldg(od + (t2 == 0 ? ch - 1 : t2 - 1));
            v[a][1] = __ldg(ev + t2);
            v[a][2] = __ldg(od + t2);
            v[a][3] = __ldg(ev + (t2 + 1 == ch ? 0u : t2 + 1));
        }
    };
    double t[2][2][2];   // [cell][dx][dy] after the four terms of the plane K
    load(0);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        double p = mul_on_int(kProlongW[0], v[0][c + 1]);
        if (__double_as_longlong(p) == (long long)(1ULL << 63)) p = 0.0;   // as fma(w, v, 0)
#pragma unroll
        for (int dx = 0; dx < 2; ++dx) {
            const double s = fma(kProlongW[1], v[0][c + 2 * dx], p);
#pragma unroll
            for (int dy = 0; dy < 2; ++dy)
                t[c][dx][dy] = fma(kProlongW[3], v[1 + dy][c + 2 * dx], fma(kProlongW[2], v[1 + dy][c + 1], s));
        }
    }
    const unsigned n = (unsigned)F.n, half = n >> 1;
#pragma unroll
    for (int dz = 0; dz < 2; ++dz) {
        load(1 + dz);
#pragma unroll
        for (int dy = 0; dy < 2; ++dy) {
            const int dx = 1 ^ dy ^ dz;
            double2* f = reinterpret_cast<double2*>(F.phi_b + (2u * J + dy + n * (2u * K + dz)) * half + 2 * t2);
            double s[2];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                double u = fma(kProlongW[4], v[0][c + 1], t[c][dx][dy]);
                u = fma(kProlongW[5], v[0][c + 2 * dx], u);
                u = fma(kProlongW[6], v[1 + dy][c + 1], u);
                s[c] = fma(kProlongW[7], v[1 + dy][c + 2 * dx], u);
            }
            double2 p = *f;
            p.x = p.x + s[0];
            p.y = p.y + s[1];
            *f = p;
        }
    }
}

// k_prolong for a split fine level over a split coarse level with
// half % 4 == 0: four compact columns (eight fine cells) per thread.  The six
// coarse x-neighbours ih0-1 .. ih0+4 of each (J', K') row are a pair plus one
// in each colour array.  Same weighted sums in the same order.
__global__ void k_prolong4(LevelView Cv, LevelView F)
{
    pdl_wait();
    pdl_trigger();
    const int n = F.n, nc = Cv.n;
    const unsigned half = (unsigned)n >> 1, chalf = (unsigned)nc >> 1, h4 = half >> 2;
    const unsigned t4 = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    if (t4 >= h4 || j >= n) return;
    const int J = j >> 1, K = k >> 1;
    const int Js[2] = {J, wrap1((j & 1) ? J + 1 : J - 1, nc)};
    const int Ks[2] = {K, wrap1((k & 1) ? K + 1 : K - 1, nc)};
    const unsigned c2 = 2 * t4;
    double v[2][2][6];
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            const unsigned row = ((unsigned)Js[a] + (unsigned)nc * (unsigned)Ks[b]) * chalf;
            const bool even_red = ((Js[a] + Ks[b]) & 1) == 0;
            const double* ev = even_red ? Cv.phi_r : Cv.phi_b;
            const double* od = even_red ? Cv.phi_b : Cv.phi_r;
            const double2 e01 = __ldg(reinterpret_cast<const double2*>(ev + row + c2));
            const double e2 = __ldg(ev + row + (c2 + 2 == chalf ? 0u : c2 + 2));
            const double2 o01 = __ldg(reinterpret_cast<const double2*>(od + row + c2));
            const double om = __ldg(od + row + (c2 == 0 ? chalf - 1 : c2 - 1));
            v[b][a][0] = om;
            v[b][a][1] = e01.x;
            v[b][a][2] = o01.x;
            v[b][a][3] = e01.y;
            v[b][a][4] = o01.y;
            v[b][a][5] = e2;
        }
    const unsigned t = ((unsigned)j + (unsigned)n * (unsigned)k) * half + 4 * t4;
    const bool even_fine_red = ((j + k) & 1) == 0;
    double* fe = (even_fine_red ? F.phi_r : F.phi_b) + t;
    double* fo = (even_fine_red ? F.phi_b : F.phi_r) + t;
    {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            double se = 0.0;
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    se = fma(kProlongW[0 + 2 * a + 4 * b], v[b][a][r + 1], se);
                    se = fma(kProlongW[1 + 2 * a + 4 * b], v[b][a][r], se);
                }
            fe[r] = fe[r] + se;
        }
    }
    {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            double so = 0.0;
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    so = fma(kProlongW[0 + 2 * a + 4 * b], v[b][a][r + 1], so);
                    so = fma(kProlongW[1 + 2 * a + 4 * b], v[b][a][r + 2], so);
                }
            fo[r] = fo[r] + so;
        }
    }
}

// trilinear cell-centred prolongation of the coarse correction, added to the
// fine phi; one thread per fine pair (2ih, 2ih+1) of a split level (BLACK: the
// black cell of the pair only, as in k_prolong_black)
template <int BLACK>
__global__ void k_prolong(LevelView Cv, LevelView F)
{
    pdl_wait();
    pdl_trigger();
    const int n = F.n, nc = Cv.n, half = n >> 1;
    const int ih = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    if (ih >= half || j >= n) return;
    const int J = j >> 1, K = k >> 1;
    const int Js[2] = {J, wrap1((j & 1) ? J + 1 : J - 1, nc)};
    const int Ks[2] = {K, wrap1((k & 1) ? K + 1 : K - 1, nc)};
    const long long t = ((long long)j + (long long)n * k) * half + ih;
#pragma unroll
    for (int odd = 0; odd < 2; ++odd) {
        const int i = 2 * ih + odd;
        if (BLACK && ((i + j + k) & 1) == 0) continue;
        const int I = ih;
        const int Is[2] = {I, wrap1(odd ? I + 1 : I - 1, nc)};
        double s = 0.0;
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int tt = 0; tt < 2; ++tt)
                    s = fma(kProlongW[tt + 2 * a + 4 * b],
                            *lv_ptr<const double>(Cv.phi_r, Cv.phi_b, nc, Cv.split, Is[tt], Js[a], Ks[b]), s);
        double* p = (((i + j + k) & 1) ? F.phi_b : F.phi_r) + t;
        *p = *p + s;
    }
}

// exact coarsest solve: phi = G * beta (cyclic convolution, y in storage order), one block
__global__ void k_bottom(int nb, const double* __restrict__ G, const double* __restrict__ beta,
                         double* phi)
{
    pdl_wait();
    pdl_trigger();
    __shared__ double r[kMaxBottom * kMaxBottom * kMaxBottom];
    __shared__ double g[kMaxBottom * kMaxBottom * kMaxBottom];
    const int nc = nb * nb * nb;
    for (int t = threadIdx.x; t < nc; t += blockDim.x) {
        r[t] = beta[t];
        g[t] = G[t];
    }
    __syncthreads();
    for (int c = threadIdx.x; c < nc; c += blockDim.x) {
        const int i = c % nb, j = (c / nb) % nb, k = c / (nb * nb);
        double s = 0.0;
        int y = 0;
        for (int yk = 0; yk < nb; ++yk) {
            const int dk = wrap1(k - yk, nb) * nb * nb;
            for (int yj = 0; yj < nb; ++yj) {
                const int djk = dk + wrap1(j - yj, nb) * nb;
                for (int yi = 0; yi < nb; ++yi, ++y) s = fma(g[djk + wrap1(i - yi, nb)], r[y], s);
            }
        }
        phi[c] = s;
    }
}

// the coarse end of an FP64 V-cycle by one CTA (pm_tail.cuh): the arithmetic of
// k_gsrb, k_restrict, k_bottom and k_prolong in the same order, so the same bits
struct TailD {
    int nl;                  // levels in the tail; the last is the bottom (natural layout)
    int nu1, nu2, nb;
    const double* G;
    LevelView lv[kMaxTail];
};

__global__ void __launch_bounds__(kTailThreadsD) k_vcycle_tail_d(TailD A)
{
    pdl_wait();
    pdl_trigger();
    __shared__ double r[kMaxBottom * kMaxBottom * kMaxBottom];
    __shared__ double g[kMaxBottom * kMaxBottom * kMaxBottom];
    vcycle_tail<double>(A.lv, A.nl, A.nu1, A.nu2, A.G, A.nb, r, g, A.nu1 > 0);
}

// A V-cycle, or a whole solve, of small levels by one cluster (pm_cluster.cuh).
// one V-cycle from a zero guess: the right-hand side and the correction of L in global memory
__global__ void __launch_bounds__(kClThreads, 1) k_cluster_vcycle_d(ClArgs<double> A, LevelView L)
{
    extern __shared__ __align__(16) double cl_mem_d[];
    __shared__ ClShared<double> S;
    cl_setup(A, S, cl_mem_d);
    pdl_wait();
    pdl_trigger();
    cl_load_green(A, S);
    cl_load(S.lv[0], L, false);
    cl_open(S.lv[0]);
    cl_barrier();
    cl_vcycle(A, S, cl_mem_d, 2);
    cl_store(S.lv[0], L);
}

// the same with both in natural layout
__global__ void __launch_bounds__(kClThreads, 1) k_cluster_vcycle_nat_d(ClArgs<double> A,
                                                                        const double* __restrict__ beta,
                                                                        double* __restrict__ e)
{
    extern __shared__ __align__(16) double cl_mem_d[];
    __shared__ ClShared<double> S;
    cl_setup(A, S, cl_mem_d);
    pdl_wait();
    pdl_trigger();
    cl_load_green(A, S);
    const ClLevel<double>& L = S.lv[0];
    const int n = L.n, half = n >> 1, total = n * n * L.np;
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int i, j, q;
        cl_split(t, n, n, i, j, q);
        const int black = (i + j + L.p0 + q) & 1, at = (i >> 1) + half * (j + n * q);
        const double b = beta[(size_t)L.p0 * n * n + t];
        (black ? L.beta_b : L.beta_r)[at] = b;
        if (!black) L.phi_r[at] = fma(0.0, kSixth, -b);
    }
    cl_barrier();
    cl_vcycle(A, S, cl_mem_d, 2);
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int i, j, q;
        cl_split(t, n, n, i, j, q);
        e[(size_t)L.p0 * n * n + t] = ((i + j + L.p0 + q) & 1 ? L.phi_b : L.phi_r)[(i >> 1) + half * (j + n * q)];
    }
}

// The V-cycles of a solve from phi (level 0) until ||r||_inf <= rel_tol max(norms[0],
// norms[1]) = rel_tol max(||beta||, ||r0||), with the red-cell norm of mg_solve's loop:
// norms[5] = ||r||, norms[6] = the number of V-cycles.  Every CTA sees the same norms, so
// all leave the loop together.
// zero: phi is 0 on entry, whatever the arrays hold.
__global__ void __launch_bounds__(kClThreads, 1) k_cluster_solve_d(ClArgs<double> A, LevelView L, double rel_tol,
                                                                int max_vcycles, int zero, unsigned long long* norms)
{
    extern __shared__ __align__(16) double cl_mem_d[];
    __shared__ ClShared<double> S;
    cl_setup(A, S, cl_mem_d);
    pdl_wait();
    pdl_trigger();
    const double bnorm = __longlong_as_double((long long)norms[0]);
    const double r0 = zero ? bnorm : __longlong_as_double((long long)norms[1]);
    const double target = rel_tol * (bnorm < r0 ? r0 : bnorm);
    double r = r0;
    int it = 0;
    if (!(r0 <= target)) {
        const ClLevel<double>& F = S.lv[0];
        const int n = F.n, half = n >> 1, total = half * n * F.np;
        cl_load_green(A, S);
        cl_load(F, L, !zero);
        cl_barrier();
        for (it = 1;; ++it) {
            cl_vcycle(A, S, cl_mem_d, zero && it == 1 ? 1 : 0);
            unsigned long long v = 0;
            for (int t = threadIdx.x; t < total; t += blockDim.x) {
                int ih, j, q;
                cl_split(t, half, n, ih, j, q);
                const double s = cl_sum<double>(F.zb, n, q + 1, j, ih, (j + F.p0 + q) & 1);
                v = max(v, absbits(F.beta_r[t] - fma(s, kSixth, -F.phi_r[t])));
            }
            cl_norm_put(S, it & 1, v);
            cl_barrier();
            r = __longlong_as_double((long long)cl_norm_get(S, it & 1));
            if (r <= target || r != r || it >= max_vcycles) break;
        }
        cl_store(F, L);
    } else if (zero) {
        const ClLevel<double>& F = S.lv[0];
        const int plane = F.n * (F.n >> 1);
        for (int t = threadIdx.x; t < plane * F.np; t += blockDim.x) {
            L.phi_r[F.p0 * plane + t] = 0.0;
            L.phi_b[F.p0 * plane + t] = 0.0;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        norms[5] = absbits(r);
        norms[6] = (unsigned long long)it;
    }
}

// g_d(c) = 0.5*((phi_c - phi_{c-e_d})*dxi + (phi_{c+e_d} - phi_c)*dxi), second product fused;
// component-major output; one product on the integer pipe
__global__ void k_grav(LevelView L, double dxi, double* g)
{
    pdl_wait();
    pdl_trigger();
    const int n = L.n;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    if (i >= n || j >= n) return;
    const long long nc = (long long)n * n * n;
    const long long c = cidx(i, j, k, n);
    auto P = [&](int a, int b, int d) {
        return *lv_ptr<const double>(L.phi_r, L.phi_b, n, L.split, a, b, d);
    };
    const double pc = P(i, j, k);
    const int im = i == 0 ? n - 1 : i - 1, ip = i == n - 1 ? 0 : i + 1;
    const int jm = j == 0 ? n - 1 : j - 1, jp = j == n - 1 ? 0 : j + 1;
    const int km = k == 0 ? n - 1 : k - 1, kp = k == n - 1 ? 0 : k + 1;
    auto diff = [&](double m, double p) { return 0.5 * fma(p - pc, dxi, mul_on_int(pc - m, dxi)); };
    g[c] = diff(P(im, j, k), P(ip, j, k));
    g[nc + c] = diff(P(i, jm, k), P(i, jp, k));
    g[2 * nc + c] = diff(P(i, j, km), P(i, j, kp));
}

// the same for a split level, two cells per thread (256^3: 484 -> 415 us)
__global__ void __launch_bounds__(256) k_grav2(int n, const double* __restrict__ phi_r,
                                               const double* __restrict__ phi_b, double dxi, double* __restrict__ g)
{
    pdl_wait();
    pdl_trigger();
    const unsigned half = (unsigned)n >> 1;
    const unsigned ih = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    if (ih >= half || j >= n) return;
    const CellPair P = cell_pair(phi_r, phi_b, n, ih, j, k);
    auto diff = [&](double m, double c, double p) { return 0.5 * fma(p - c, dxi, mul_on_int(c - m, dxi)); };
    const long long nc2 = (long long)n * n * half;
    double2* out = reinterpret_cast<double2*>(g) + ((unsigned)j + (unsigned)n * (unsigned)k) * half + ih;
#pragma unroll
    for (int d = 0; d < 3; ++d)
        out[d * nc2] = make_double2(diff(P.c[2 * d], P.even, P.c[2 * d + 1]),
                                    diff(P.c[6 + 2 * d], P.odd, P.c[7 + 2 * d]));
}

__global__ void k_to_natural(LevelView L, double* out)
{
    const int n = L.n;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    if (i >= n || j >= n) return;
    out[cidx(i, j, k, n)] = *lv_ptr<const double>(L.phi_r, L.phi_b, n, L.split, i, j, k);
}

__global__ void k_from_natural(LevelView L, const double* __restrict__ in)
{
    const int n = L.n;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    if (i >= n || j >= n) return;
    *lv_ptr<double>(L.phi_r, L.phi_b, n, L.split, i, j, k) = in[cidx(i, j, k, n)];
}

// the right-hand side of a correction solve from natural layout; with red, also the red half
// sweep that opens it from phi = 0
__global__ void k_beta_from_natural(LevelView L, const double* __restrict__ in, int red)
{
    pdl_wait();
    pdl_trigger();
    const int n = L.n;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    if (i >= n || j >= n) return;
    const double b = in[cidx(i, j, k, n)];
    *lv_ptr<double>(L.beta_r, L.beta_b, n, L.split, i, j, k) = b;
    if (red && ((i + j + k) & 1) == 0)
        *lv_ptr<double>(L.phi_r, L.phi_b, n, L.split, i, j, k) = fma(0.0, kSixth, -b);
}

// Levels of at least this edge work by pairs of cells, their sums on the integer pipes
// (pm_sum6.cuh): there the FP64 pipe is the bound (four steps at 96^3 12.3 -> 11.5 ms, at 112^3
// 18.3 -> 17.1).  Below, a half sweep is latency: with integer sums on level 64 four 64^3 steps take
// 7.24 ms against 7.10, on level 80 four 160^3 steps 31.1 against 30.5.  Their half sweeps and
// restrictions go by blocks of 128 threads, whose four warps are one on the FP64 pipe and three on the
// integer pipes (256^3: 101.5 ms with 256 threads, 100.2; with 64 106.6).
constexpr int kPairMinEdge = 96;
inline bool by_pairs(const Level& l) { return l.split && l.n >= kPairMinEdge && l.n % 4 == 0; }

nyxpm_status gsrb_sweep(Ctx& c, const Level& l, int fine, int black_only = 0)
{
    const long long half_cells = (long long)l.n * l.n * l.n / 2;
    const bool pairs = by_pairs(l);
    const Geo g = geo3(pairs ? l.n / 4 : l.n / 2, l.n, l.n, pairs ? 128 : 256);
    for (int color = black_only ? 1 : 0; color < 2; ++color) {
        double* mine = color ? l.phi_b : l.phi_r;
        const double* other = color ? l.phi_r : l.phi_b;
        const double* beta = color ? l.beta_b : l.beta_r;
        prof_begin(c);
        launch_pdl(c, pairs ? k_gsrb2 : k_gsrb, dim3(g.grid), dim3(g.block), l.n, color, mine, other, beta);
        prof_end(c, NYXPM_ST_SMOOTH, 24.0 * half_cells, fine);
    }
    return check_launch(c, "gsrb");
}

// One SM issues FP64 at 1/64 of its FP32 rate, so the FP64 form fuses only the
// levels of at most half the FP32 edge (8^3 cells at the default 16): there a
// level's half sweep is a few hundred cells, cheaper on one SM than a launch.
bool tail_fits_d(const Ctx& c, const Box& b, size_t li)
{
    const int edge = c.p.mg_fused_edge / 2;
    return li > 0 && edge > 0 && b.levels[li].n <= edge && b.levels.size() - li >= 2 &&
           b.levels.size() - li <= (size_t)kMaxTail;
}

// whether the levels from li on are taken by one cluster, and how they lie in it.  Below a
// box's finest level only from 16^3 down: a pass over 32^3 takes the FP64 pipes of 16 SMs as long
// as a launch takes all of them and its launch (four steps at 64^3 7.48 ms with level 32 in the
// cluster, 7.19 without; 7.8 with level 16 out too).  A box of up to 32^3 is solved in one
// launch (3.64 ms; its V-cycles by launches down to 16^3 3.82).  Grids of 4 * 2^k and 6 * 2^k
// cells only (cl_layout).
constexpr int kClusterEdgeD = 16;   // (whole boxes: kClEdgeD)

bool cluster_fits_d(Ctx& c, const Box& b, size_t li, ClArgs<double>& A)
{
    if (li > 0 && b.levels[li].n > kClusterEdgeD) return false;
    if (!cl_args<double>(c, b, li, A)) return false;
    if (c.cluster_d < 0) {
        const size_t most = cl_max_bytes<double>();
        c.cluster_d = cl_prepare(k_cluster_vcycle_d, most) && cl_prepare(k_cluster_vcycle_nat_d, most) &&
                      cl_prepare(k_cluster_solve_d, most);
    }
    return c.cluster_d > 0;
}

nyxpm_status vcycle_tail_d(Ctx& c, Box& b, size_t li)
{
    TailD A;
    A.nl = (int)(b.levels.size() - li);
    A.nu1 = c.p.nu1;
    A.nu2 = c.p.nu2;
    A.nb = b.nb;
    A.G = b.G;
    double bytes = 0;
    for (int l = 0; l < A.nl; ++l) {
        const Level& lv = b.levels[li + l];
        A.lv[l] = view(lv);
        const double cells = (double)lv.n * lv.n * lv.n;
        bytes += (l + 1 < A.nl) ? 12.0 * cells * 2 * (c.p.nu1 + c.p.nu2) + 32.0 * cells : 16.0 * cells;
    }
    prof_begin(c);
    launch_pdl(c, k_vcycle_tail_d, dim3(1), dim3(kTailThreadsD), A);
    prof_end(c, NYXPM_ST_SMOOTH, bytes);
    return check_launch(c, "fused coarse V-cycle");
}

// red_done: the opening red half sweep of this level was already made (by
// k_resnorm_red_sweep or the restriction)
nyxpm_status vcycle(Ctx& c, Box& b, size_t li, int red_done = 0)
{
    nyxpm_status st;
    const Level& f = b.levels[li];
    ClArgs<double> ca;
    if (li > 0 && cluster_fits_d(c, b, li, ca)) {
        prof_begin(c);
        launch_cluster(c, k_cluster_vcycle_d, ca.elems * sizeof(double), ca, view(f));
        prof_end(c, NYXPM_ST_SMOOTH, 32.0 * f.n * f.n * f.n);
        return check_launch(c, "cluster V-cycle");
    }
    if (tail_fits_d(c, b, li)) return vcycle_tail_d(c, b, li);
    if (li + 1 == b.levels.size()) {
        prof_begin(c);
        launch_pdl(c, k_bottom, dim3(1), dim3(512), b.nb, b.G, f.beta_r, f.phi_r);
        prof_end(c, NYXPM_ST_BOTTOM, 16.0 * f.n * f.n * f.n);
        return check_launch(c, "bottom");
    }
    const int nu1 = c.p.nu1, nu2 = c.p.nu2;
    for (int s = 0; s < nu1; ++s)
        if ((st = gsrb_sweep(c, f, li == 0, s == 0 && red_done)) != NYXPM_OK) return st;
    const Level& cl = b.levels[li + 1];
    const long long ncc = (long long)cl.n * cl.n * cl.n;
    const long long ncf = (long long)f.n * f.n * f.n;
    const bool quads = f.split && (f.n / 2) % 4 == 0;
    // a coarse level that launches smooth (not the cluster, the tail or the bottom)
    const int open = nu1 > 0 && li + 2 < b.levels.size() && !tail_fits_d(c, b, li + 1) &&
                     !cluster_fits_d(c, b, li + 1, ca);
    {
        const bool pairs = c.p.nu1 > 0 && by_pairs(f);
        const Geo g = geo3(pairs ? cl.n / 2 : cl.n, cl.n, cl.n, pairs ? 128 : 256);
        prof_begin(c);
        if (c.p.nu1 > 0)
            launch_pdl(c, pairs ? k_restrict_red2 : k_restrict<1>, dim3(g.grid), dim3(g.block), view(f), view(cl),
                       open);
        else
            launch_pdl(c, k_restrict<0>, dim3(g.grid), dim3(g.block), view(f), view(cl), open);
        prof_end(c, NYXPM_ST_RESTRICT, 16.0 * ncf + 16.0 * ncc);
    }
    if ((st = check_launch(c, "restrict")) != NYXPM_OK) return st;
    if ((st = vcycle(c, b, li + 1, open)) != NYXPM_OK) return st;
    {
        prof_begin(c);
        const bool black = nu2 > 0;
        if (quads && cl.split) {
            const Geo g = black ? geo3(cl.n / 2, cl.n, cl.n) : geo3(f.n / 8, f.n, f.n);
            launch_pdl(c, black ? k_prolong_black : k_prolong4, dim3(g.grid), dim3(g.block), view(cl), view(f));
        } else {
            const Geo g = geo3(f.n / 2, f.n, f.n);
            if (black) launch_pdl(c, k_prolong<1>, dim3(g.grid), dim3(g.block), view(cl), view(f));
            else launch_pdl(c, k_prolong<0>, dim3(g.grid), dim3(g.block), view(cl), view(f));
        }
        prof_end(c, NYXPM_ST_PROLONG, 16.0 * ncf + 8.0 * ncc);
    }
    if ((st = check_launch(c, "prolong")) != NYXPM_OK) return st;
    for (int s = 0; s < nu2; ++s)
        if ((st = gsrb_sweep(c, f, li == 0)) != NYXPM_OK) return st;
    return NYXPM_OK;
}

// launch ||r_beta||_inf of level 0 into norms[slot] (0 before): all cells, or the red
// cells only after a cycle that ended with a black half sweep
nyxpm_status launch_resnorm(Ctx& c, Box& b, int slot, int red_only)
{
    const Level& l = b.levels[0];
    const long long nc = (long long)l.n * l.n * l.n;
    prof_begin(c);
    if (l.split && red_only) {
        const Geo g = geo3(l.n / 2, l.n, l.n);
        launch_pdl(c, k_resnorm_red, dim3(g.grid), dim3(g.block), l.n, l.phi_r, l.phi_b, l.beta_r, b.norms + slot);
    } else if (l.split) {
        const bool pairs = by_pairs(l);
        const Geo g = geo3(pairs ? l.n / 4 : l.n / 2, l.n, l.n);
        launch_pdl(c, pairs ? k_resnorm_split2 : k_resnorm_split, dim3(g.grid), dim3(g.block), view(l), b.norms + slot);
    } else {
        const Geo g = geo3(l.n, l.n, l.n);
        launch_pdl(c, k_resnorm_nat, dim3(g.grid), dim3(g.block), view(l), b.norms + slot);
    }
    prof_end(c, NYXPM_ST_NORM, (red_only ? 12.0 : 16.0) * nc);
    return check_launch(c, "resnorm");
}

double read_norm(Box& b, int slot)
{
    double v;
    std::memcpy(&v, &b.h_norms[slot], sizeof(v));
    return v;
}

}  // namespace

double beta_scale(const Box& b)
{
    const double h = b.L / b.n;
    return (h * h) * kSixth;
}

nyxpm_status launch_make_rhs(Ctx& c, Box& b, double a)
{
    const int n = b.n;
    const long long nc = (long long)n * n * n;
    const Level& l0 = b.levels[0];
    const double dx = b.L / n;
    const Geo g = geo3(n, n, n);
    prof_begin(c);
    launch_pdl(c, k_rowsum, dim3(blocks_for((long long)n * n * 32)), dim3(kThreads), n, b.rho, b.mass_offset, b.rows);
    launch_pdl(c, k_mean, dim3((n + 31) / 32), dim3(32), n, dx, b.L, b.rows, b.planes,
               reinterpret_cast<unsigned*>(b.scal + kScalTicket), b.scal, b.norms);
    launch_pdl(c, k_make_beta, dim3(g.grid), dim3(g.block), n, l0.split, b.rho, b.mass_offset, b.scal,
               -4.0 * M_PI * c.p.gconst, 1.0 / a, beta_scale(b), l0.beta_r, l0.beta_b, b.norms);
    prof_end(c, NYXPM_ST_RHS, 24.0 * nc);
    c.launches += 2;
    return check_launch(c, "make rhs");
}

nyxpm_status launch_zero_phi(Ctx& c, Box& b)
{
    const Level& l0 = b.levels[0];
    const size_t nc = (size_t)l0.n * l0.n * l0.n;
    if (l0.split) {
        cudaMemsetAsync(l0.phi_r, 0, sizeof(double) * nc / 2, c.stream);
        cudaMemsetAsync(l0.phi_b, 0, sizeof(double) * nc / 2, c.stream);
    } else {
        cudaMemsetAsync(l0.phi_r, 0, sizeof(double) * nc, c.stream);
    }
    return check_launch(c, "zero phi");
}

nyxpm_status mg_solve(Ctx& c, Box& b, int zero_guess, nyxpm_solve_info* info, bool* grav_done)
{
    nyxpm_status st;
    const Level& l0 = b.levels[0];
    const long long nc = (long long)l0.n * l0.n * l0.n;
    post_open(c, b.post);
    // a small box: the whole solve in one cluster launch
    ClArgs<double> ca;
    const bool in_cluster = cluster_fits_d(c, b, 0, ca);
    const int red_only = (c.p.nu2 > 0 && b.levels.size() > 1) ? 1 : 0;
    // The red-cell norm after a V-cycle and the red half sweep that opens the next
    // one share their neighbour sums: k_resnorm_red_sweep makes both, the sweep into
    // the spare red array, which becomes level 0's red array only if the solve
    // goes on (the next V-cycle then starts at its black half sweep).
    Level& L0 = b.levels[0];
    const bool fuse = red_only && c.p.nu1 > 0 && L0.split && b.phi_r_spare;
    // From phi = 0 the residual is beta, whose norm launch_make_rhs left, and the opening red
    // half sweep needs no neighbours, so phi is not zeroed (370 us of a 256^3 solve)
    const bool from_zero = zero_guess && (in_cluster || fuse);
    if (zero_guess && !from_zero && (st = launch_zero_phi(c, b)) != NYXPM_OK) return st;
    // ||r0||_inf
    if (!from_zero && (st = launch_resnorm(c, b, 1, 0)) != NYXPM_OK) return st;
    if (in_cluster) {
        prof_begin(c);
        launch_cluster(c, k_cluster_solve_d, ca.elems * sizeof(double), ca, view(l0), c.p.rel_tol, c.p.max_vcycles,
                       from_zero ? 1 : 0, b.norms);
        prof_end(c, NYXPM_ST_SMOOTH, 0);
        if ((st = check_launch(c, "cluster solve")) != NYXPM_OK) return st;
    }
    post_words(c, b.post, b.norms, 0, in_cluster ? 7 : 2, 1 << 1);
    // the gravity vector follows every solve that ends, converged or not
    if (in_cluster && (st = launch_grav_vector(c, b)) != NYXPM_OK) return st;
    *grav_done = in_cluster;
    if ((st = check_launch(c, "norm read-back")) != NYXPM_OK) return st;
    if ((st = post_wait(c, b.post, "solve sync")) != NYXPM_OK) return st;
    const double bnorm = read_norm(b, 0);
    const double r0 = from_zero ? bnorm : read_norm(b, 1);
    const double target = c.p.rel_tol * std::max(bnorm, r0);
    double r = r0;
    int it = 0;
    nyxpm_status result = NYXPM_OK;
    if (from_zero && !in_cluster && r0 <= target && (st = launch_zero_phi(c, b)) != NYXPM_OK) return st;
    if (in_cluster) {
        r = read_norm(b, 5);
        it = (int)b.h_norms[6];
        if (r != r) {
            c.err = "multigrid residual is NaN";
            return NYXPM_NOT_CONVERGED;
        }
        if (!(r <= target)) {
            result = NYXPM_NOT_CONVERGED;
            c.err = "multigrid reached max_vcycles above tolerance";
        }
    } else if (!(r0 <= target)) {
        bool first = !from_zero;
        if (from_zero) {
            prof_begin(c);
            launch_pdl(c, k_gsrb_zero, dim3(blocks_for(nc / 4)), dim3(kThreads), (unsigned)(nc / 4),
                       reinterpret_cast<const ulonglong2*>(L0.beta_r), reinterpret_cast<ulonglong2*>(L0.phi_r));
            prof_end(c, NYXPM_ST_SMOOTH, 8.0 * nc);
            if ((st = check_launch(c, "opening sweep")) != NYXPM_OK) return st;
        }
        auto iteration = [&]() -> nyxpm_status {
            nyxpm_status s;
            if ((s = vcycle(c, b, 0, fuse && !first ? 1 : 0)) != NYXPM_OK) return s;
            if (fuse) {
                const bool pairs = by_pairs(L0);
                const Geo g = geo3(pairs ? L0.n / 4 : L0.n / 2, L0.n, L0.n);
                prof_begin(c);
                launch_pdl(c, pairs ? k_resnorm_red_sweep2 : k_resnorm_red_sweep, dim3(g.grid), dim3(g.block), L0.n,
                           L0.phi_r, L0.phi_b, L0.beta_r, b.phi_r_spare, b.norms + 1);
                prof_end(c, NYXPM_ST_NORM, 16.0 * nc);
                if ((s = check_launch(c, "red norm + sweep")) != NYXPM_OK) return s;
            } else if ((s = launch_resnorm(c, b, 1, red_only)) != NYXPM_OK) {
                return s;
            }
            post_words(c, b.post, b.norms, 1, 1, 1 << 1);
            return check_launch(c, "norm read-back");
        };
        for (it = 1; it <= c.p.max_vcycles; ++it) {
            // one graph per (opening or later iteration, physical red array)
            const int gi = (first ? 0 : 2) + (L0.phi_r == b.phi_r_alloc ? 0 : 1);
            post_open(c, b.post);
            if ((st = run_iteration(c, b.iter_graph[gi], iteration)) != NYXPM_OK) return st;
            if ((st = post_wait(c, b.post, "solve sync")) != NYXPM_OK) return st;
            r = read_norm(b, 1);
            if (r != r) {
                c.err = "multigrid residual is NaN";
                return NYXPM_NOT_CONVERGED;
            }
            if (r <= target) break;
            if (fuse && it < c.p.max_vcycles) {
                std::swap(L0.phi_r, b.phi_r_spare);
                first = false;
            }
        }
        if (it > c.p.max_vcycles) {
            it = c.p.max_vcycles;
            result = NYXPM_NOT_CONVERGED;
            c.err = "multigrid reached max_vcycles above tolerance";
        }
    }
    b.have_phi = 1;
    if (info) {
        const double inv_k0 = 1.0 / beta_scale(b);
        info->vcycles = it;
        info->inner_vcycles = 0;
        info->resnorm0 = r0 * inv_k0;
        info->resnorm = r * inv_k0;
        info->bnorm = bnorm * inv_k0;
    }
    return result;
}

nyxpm_status launch_grav_vector(Ctx& c, Box& b)
{
    const long long nc = (long long)b.n * b.n * b.n;
    const Geo g = geo3(b.n, b.n, b.n);
    prof_begin(c);
    if (b.levels[0].split) {
        const Geo g2 = geo3(b.n / 2, b.n, b.n);
        launch_pdl(c, k_grav2, dim3(g2.grid), dim3(g2.block), b.n, b.levels[0].phi_r, b.levels[0].phi_b, b.dxi, b.g);
    } else {
        launch_pdl(c, k_grav, dim3(g.grid), dim3(g.block), view(b.levels[0]), b.dxi, b.g);
    }
    prof_end(c, NYXPM_ST_KICK, 32.0 * nc);
    return check_launch(c, "grav vector");
}

nyxpm_status launch_phi_to_natural(Ctx& c, Box& b, double* d_out)
{
    const long long nc = (long long)b.n * b.n * b.n;
    const Geo g = geo3(b.n, b.n, b.n);
    prof_begin(c);
    k_to_natural<<<g.grid, g.block, 0, c.stream>>>(view(b.levels[0]), d_out);
    prof_end(c, NYXPM_ST_GATHER, 16.0 * nc);
    return check_launch(c, "phi to natural");
}

nyxpm_status launch_phi_from_natural(Ctx& c, Box& b, const double* d_in)
{
    const long long nc = (long long)b.n * b.n * b.n;
    const Geo g = geo3(b.n, b.n, b.n);
    prof_begin(c);
    k_from_natural<<<g.grid, g.block, 0, c.stream>>>(view(b.levels[0]), d_in);
    prof_end(c, NYXPM_ST_GATHER, 16.0 * nc);
    return check_launch(c, "phi from natural");
}

nyxpm_status mg_vcycle_zero(Ctx& c, Box& b, const double* beta_nat, double* e_nat)
{
    nyxpm_status st;
    const long long nc = (long long)b.n * b.n * b.n;
    const Geo g = geo3(b.n, b.n, b.n);
    ClArgs<double> ca;
    if (cluster_fits_d(c, b, 0, ca)) {
        prof_begin(c);
        launch_cluster(c, k_cluster_vcycle_nat_d, ca.elems * sizeof(double), ca, beta_nat, e_nat);
        prof_end(c, NYXPM_ST_SMOOTH, 16.0 * nc);
        return check_launch(c, "cluster V-cycle");
    }
    // (black cells are written before they are read)
    const Level& l0 = b.levels[0];
    const int red = l0.split && c.p.nu1 > 0 && !tail_fits_d(c, b, 0) ? 1 : 0;
    prof_begin(c);
    launch_pdl(c, k_beta_from_natural, dim3(g.grid), dim3(g.block), view(l0), beta_nat, red);
    prof_end(c, NYXPM_ST_RHS, 16.0 * nc);
    if (!red && (st = launch_zero_phi(c, b)) != NYXPM_OK) return st;
    if ((st = vcycle(c, b, 0, red)) != NYXPM_OK) return st;
    return launch_phi_to_natural(c, b, e_nat);
}

}  // namespace nyxpm
