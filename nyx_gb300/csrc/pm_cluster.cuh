// V-cycles of small levels by one cluster of 16 CTAs, every level in shared memory.
//
// Why.  On small levels a pass is a few thousand cells: as a launch of its own it takes 1.5
// to 4 us, nearly all of it launch and memory latency, and a V(2,2) cycle has ten passes per
// level.  One CTA is too slow for these levels, and a cluster that passes its values through
// L2 as well.  Here the levels of a V-cycle stay in the CTAs' shared memory: a level is cut
// into slabs of whole z planes, the CTA that owns a plane updates it, the neighbour planes of
// a slab are read from the other CTAs' shared memory, and a hardware cluster barrier stands
// between two passes.  The levels small enough for one CTA (8^3 in FP64, 16^3 in FP32) are
// cycled by the cluster's first CTA (vcycle_solo, pm_tail.cuh) in its shared memory, two
// levels at least, the bottom and a split one: in FP64 the chains 20-10-5 and 28-14-7 have the
// bottom only, and grids of 5 * 2^k and 7 * 2^k cells an edge go by launches at every level.
//
// Measured on GB300 (SM clocks): a cluster barrier 526; a half sweep of 32^3 in FP64 3800,
// against 2.2 us (4500 clocks) of a launch.  FP64 issues at 19 clocks per warp instruction and
// SM, so that a pass over 32^3 takes the FP64 pipes of 16 SMs about as long as a launch over
// the whole chip.  Where the edges lie (launches overlap by programmatic dependent launch):
//   whole boxes             FP64 to 32^3: four steps 3.64 ms, by launches down to 16^3 3.82;
//                           FP32 to 48^3: 3.35 against 3.47; at 64^3 4.08 against 3.83
//   below a finest level    FP64 from 16^3: 64^3 7.10, with level 32 7.48, without any 7.8;
//                           FP32 from 32^3: 128^3 7.50, with level 64 8.28, without level 32 8.60
// (Integer sums, pm_sum6.cuh, lose here: on coarse levels some lane of a warp nearly always
// needs the FP64 additions as well, a 32^3 solve of 0.55 ms took 0.64.)
//
// Every cell's arithmetic is that of the per-pass kernels (k_gsrb, k_restrict<1>,
// k_prolong<1> and their FP32 forms), in the same order, so the bits are theirs.
// Pre- and post-smoothing are both present (nu1, nu2 > 0): the restriction takes the red
// children and the prolongation corrects the black cells.
#pragma once

#include "pm_common.cuh"
#include "pm_tail.cuh"

#include <algorithm>

namespace nyxpm {

constexpr int kClCtas = 16;         // CTAs of the cluster
constexpr int kClThreads = 512;   // a cluster barrier of 16 x 512 threads takes 526 cycles, of 16 x 1024 682
constexpr int kClMaxPlanes = 3;     // planes of a level a CTA owns at most: kClEdgeF / kClCtas
constexpr int kClMaxLevels = 4;     // levels in slabs
constexpr int kClEdgeF = 48;        // largest level taken, FP32 and FP64 (whole boxes; see cluster_fits_f, _d)
constexpr int kClEdgeD = 32;
constexpr int kClSoloF = 16;        // levels up to this edge belong to one CTA
constexpr int kClSoloD = 8;

__device__ __forceinline__ void cl_barrier()
{
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ int cl_rank()
{
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return (int)r;
}

// the address, in CTA rank's shared memory, of what p addresses in this CTA's
template <typename T>
__device__ __forceinline__ T* cl_map(T* p, int rank)
{
    unsigned long long q;
    asm("mapa.u64 %0, %1, %2;" : "=l"(q) : "l"((unsigned long long)p), "r"(rank));
    return reinterpret_cast<T*>(q);
}

// CTA c owns the planes p of a level with p * 16 / n = c: cl_first(c) .. cl_first(c+1) - 1
__host__ __device__ inline int cl_owner(int p, int n) { return p * kClCtas / n; }
__host__ __device__ inline int cl_first(int c, int n) { return (c * n + kClCtas - 1) / kClCtas; }

// The levels of a cluster V-cycle and where they lie in every CTA's shared memory (in
// elements): a slab level's four arrays phi_r, phi_b, beta_r, beta_b of `planes` planes
// each; the staged planes of the coarser level; the one-CTA levels (used in CTA 0 only).
template <typename T>
struct ClArgs {
    int nd, ns;                        // levels in slabs, levels of one CTA (the last is the bottom)
    int nu1, nu2, nb;
    const T* G;
    int n[kClMaxLevels + kMaxTail];    // edges, finest first
    int planes[kClMaxLevels];
    unsigned at[kClMaxLevels + kMaxTail];
    unsigned stage;                    // staged coarse planes (red, then black); CTA 0's scratch
    unsigned elems;                    // dynamic shared memory, elements
};

// dynamic shared memory a cluster kernel may ask for
template <typename T>
constexpr size_t cl_max_bytes() { return (sizeof(T) == 4 ? 216 : 96) * 1024; }

// the levels of a hierarchy of edges n[]; false if they do not fit
template <typename T>
inline bool cl_layout(ClArgs<T>& A, const int* n, int levels)
{
    const int solo = sizeof(T) == 4 ? kClSoloF : kClSoloD, top = sizeof(T) == 4 ? kClEdgeF : kClEdgeD;
    if (levels < 2 || n[0] <= solo || n[0] > top) return false;
    A.nd = A.ns = 0;
    unsigned at = 0, stage = 0;
    for (int l = 0; l < levels; ++l) {
        const int nl = n[l];
        if (nl > solo) {
            if (A.nd == kClMaxLevels || (nl & 1)) return false;
            int planes = 0;
            for (int c = 0; c < kClCtas; ++c) planes = std::max(planes, cl_first(c + 1, nl) - cl_first(c, nl));
            if (planes > kClMaxPlanes) return false;
            A.planes[l] = planes;
            // the coarse planes under a slab and one on each side
            stage = std::max(stage, (unsigned)(planes / 2 + 3) * (nl / 2) * (nl / 2));
            A.nd++;
            A.n[l] = nl;
            A.at[l] = at;
            at += 2u * planes * nl * nl;
        } else {
            if (A.ns == kMaxTail) return false;
            A.ns++;
            A.n[l] = nl;
            A.at[l] = at;
            at += 2u * nl * nl * nl;
        }
    }
    if (A.ns < 2) return false;   // vcycle_solo takes a split level over the bottom
    stage = std::max(stage, (unsigned)(A.n[A.nd] * A.n[A.nd] * A.n[A.nd]) / 2u);
    A.stage = (at + 3u) & ~3u;
    A.elems = A.stage + stage;
    return A.elems * sizeof(T) <= cl_max_bytes<T>();
}

// One slab level as a CTA sees it.  zr, zb, br: the planes p0 - 1 .. p0 + np + 1 (periodic)
// of phi_r, phi_b and beta_r, wherever they lie.
template <typename T>
struct ClLevel {
    int n, p0, np;
    T *phi_r, *phi_b, *beta_r, *beta_b;
    T* zr[kClMaxPlanes + 3];
    T* zb[kClMaxPlanes + 3];
    T* br[kClMaxPlanes + 3];
};

template <typename T>
struct ClShared {
    ClLevel<T> lv[kClMaxLevels];
    SoloLevel<T> solo[kMaxTail];
    unsigned long long part[2][kClCtas];   // the CTAs' norms
    T g[kMaxBottom * kMaxBottom * kMaxBottom];
};

template <typename T>
__device__ __forceinline__ void cl_setup(const ClArgs<T>& A, ClShared<T>& S, T* mem)
{
    const int rank = cl_rank();
    if ((int)threadIdx.x < A.nd) {
        const int l = threadIdx.x, n = A.n[l];
        ClLevel<T>& L = S.lv[l];
        const unsigned plane = (unsigned)n * (n >> 1), arr = plane * A.planes[l];
        L.n = n;
        L.p0 = cl_first(rank, n);
        L.np = cl_first(rank + 1, n) - L.p0;
        L.phi_r = mem + A.at[l];
        L.phi_b = L.phi_r + arr;
        L.beta_r = L.phi_b + arr;
        L.beta_b = L.beta_r + arr;
        for (int q = 0; q < L.np + 3; ++q) {
            const int p = (L.p0 - 1 + q + n) % n, c = cl_owner(p, n);
            const unsigned o = (unsigned)(p - cl_first(c, n)) * plane;
            L.zr[q] = cl_map(L.phi_r + o, c);
            L.zb[q] = cl_map(L.phi_b + o, c);
            L.br[q] = cl_map(L.beta_r + o, c);
        }
    }
    if ((int)threadIdx.x < A.ns)
        S.solo[threadIdx.x] = SoloLevel<T>{A.n[A.nd + threadIdx.x], mem + A.at[A.nd + threadIdx.x]};
    __syncthreads();
}

// t -> (x, y, plane)
__device__ __forceinline__ void cl_split(int t, int nx, int ny, int& x, int& y, int& z)
{
    tail_split3(t, nx, ny, x, y, z);
}

// neighbour sum of the cell at column ih of row j of the own plane q (q = 1 is p0), from
// the planes z of the other colour; odd: the cell's x is 2 ih + 1
template <typename T>
__device__ __forceinline__ T cl_sum(T* const* z, int n, int q, int j, int ih, int odd)
{
    const int half = n >> 1;
    const T* c = z[q] + j * half;
    const int ihm = odd ? ih : (ih == 0 ? half - 1 : ih - 1), ihp = odd ? (ih == half - 1 ? 0 : ih + 1) : ih;
    const int jm = j == 0 ? n - 1 : j - 1, jp = j == n - 1 ? 0 : j + 1;
    T s = c[ihm] + c[ihp];
    s = s + z[q][jm * half + ih];
    s = s + z[q][jp * half + ih];
    s = s + z[q - 1][j * half + ih];
    s = s + z[q + 1][j * half + ih];
    return s;
}

// one half sweep of the own planes.  zero: the other colour is 0 throughout (not read)
template <typename T>
__device__ __forceinline__ void cl_gsrb(const ClLevel<T>& L, int color, bool zero)
{
    const int n = L.n, half = n >> 1, total = half * n * L.np;
    T* mine = color ? L.phi_b : L.phi_r;
    const T* beta = color ? L.beta_b : L.beta_r;
    T* const* z = color ? L.zr : L.zb;
    if (zero) {
        for (int t = threadIdx.x; t < total; t += blockDim.x) mine[t] = tail_fma(T(0), tail_sixth<T>(), -beta[t]);
        return;
    }
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int ih, j, q;
        cl_split(t, half, n, ih, j, q);
        const T s = cl_sum<T>(z, n, q + 1, j, ih, (j + L.p0 + q + color) & 1);
        mine[t] = tail_fma(s, tail_sixth<T>(), -beta[t]);
    }
}

// the same, four cells of a row at a time (half % 4 == 0)
__device__ __forceinline__ void cl_gsrb4(const ClLevel<float>& L, int color, bool zero)
{
    const int n = L.n, half = n >> 1, h4 = half >> 2, total = h4 * n * L.np;
    float4* mine = reinterpret_cast<float4*>(color ? L.phi_b : L.phi_r);
    const float4* beta = reinterpret_cast<const float4*>(color ? L.beta_b : L.beta_r);
    float* const* z = color ? L.zr : L.zb;
    constexpr float sixth = 1.0f / 6.0f;
    if (zero) {
        for (int t = threadIdx.x; t < total; t += blockDim.x) {
            const float4 b = beta[t];
            mine[t] = make_float4(fmaf(0.f, sixth, -b.x), fmaf(0.f, sixth, -b.y), fmaf(0.f, sixth, -b.z),
                                  fmaf(0.f, sixth, -b.w));
        }
        return;
    }
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int t4, j, q;
        cl_split(t, h4, n, t4, j, q);
        const int jm = j == 0 ? n - 1 : j - 1, jp = j == n - 1 ? 0 : j + 1;
        const float* row = z[q + 1] + j * half;
        const float4 zm = *reinterpret_cast<const float4*>(z[q] + j * half + 4 * t4);
        const float4 zp = *reinterpret_cast<const float4*>(z[q + 2] + j * half + 4 * t4);
        const float4 c = *reinterpret_cast<const float4*>(row + 4 * t4);
        const float4 ym = *reinterpret_cast<const float4*>(z[q + 1] + jm * half + 4 * t4);
        const float4 yp = *reinterpret_cast<const float4*>(z[q + 1] + jp * half + 4 * t4);
        const float4 b = beta[t];
        const int odd = (j + L.p0 + q + color) & 1;
        const float e = row[odd ? (4 * t4 + 4 == half ? 0 : 4 * t4 + 4) : (t4 == 0 ? half - 1 : 4 * t4 - 1)];
        const float x0 = odd ? c.x : e, x1 = odd ? c.y : c.x, x2 = odd ? c.z : c.y, x3 = odd ? c.w : c.z,
                    x4 = odd ? e : c.w;
        float4 r;
        r.x = fmaf(((((x0 + x1) + ym.x) + yp.x) + zm.x) + zp.x, sixth, -b.x);
        r.y = fmaf(((((x1 + x2) + ym.y) + yp.y) + zm.y) + zp.y, sixth, -b.y);
        r.z = fmaf(((((x2 + x3) + ym.z) + yp.z) + zm.z) + zp.z, sixth, -b.z);
        r.w = fmaf(((((x3 + x4) + ym.w) + yp.w) + zm.w) + zp.w, sixth, -b.w);
        mine[t] = r;
    }
}

template <typename T>
__device__ __forceinline__ void cl_half_sweep(const ClLevel<T>& L, int color, bool zero)
{
    if constexpr (sizeof(T) == 4) {
        if ((L.n & 7) == 0) return cl_gsrb4(L, color, zero);
    }
    cl_gsrb<T>(L, color, zero);
}

// the red children's residuals of the coarse planes K with fine plane 2K in this slab,
// into the coarse right-hand side (in the slabs of C, with the opening red half sweep of
// the coarse level, or in CTA 0's level at solo)
template <typename T>
__device__ __forceinline__ void cl_restrict(const ClLevel<T>& F, const ClLevel<T>* C, T* solo)
{
    const int n = F.n, half = n >> 1, nc = n >> 1, chalf = nc >> 1;
    const int K0 = (F.p0 + 1) >> 1, nK = ((F.p0 + F.np + 1) >> 1) - K0;
    const int total = nc * nc * nK;
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int I, J, K;
        cl_split(t, nc, nc, I, J, K);
        K += K0;
        T s = T(0);
#pragma unroll
        for (int dk = 0; dk < 2; ++dk)
#pragma unroll
            for (int dj = 0; dj < 2; ++dj) {
                const int j = 2 * J + dj, q = 2 * K + dk - F.p0 + 1;   // the red child is x = 2 I + ((dj + dk) & 1)
                const T sum = cl_sum<T>(F.zb, n, q, j, I, (dj + dk) & 1);
                s = s + (F.br[q][j * half + I] - tail_fma(sum, tail_sixth<T>(), -F.zr[q][j * half + I]));
            }
        const int black = (I + J + K) & 1;
        const unsigned o = (unsigned)(I >> 1) + (unsigned)chalf * J;
        if (C) {
            const int c = cl_owner(K, nc);
            const unsigned at = (unsigned)(K - cl_first(c, nc)) * (nc * chalf) + o;
            const T b = s * T(0.5);
            *cl_map((black ? C->beta_b : C->beta_r) + at, c) = b;
            if (!black) *cl_map(C->phi_r + at, c) = tail_fma(T(0), tail_sixth<T>(), -b);
        } else {
            *cl_map(solo + (2 + black) * (nc * nc * chalf) + K * (nc * chalf) + o, 0) = s * T(0.5);
        }
    }
}

// the same, two coarse cells of a row at a time (half % 4 == 0): their red children in a
// fine row are a pair of the row
__device__ __forceinline__ void cl_restrict2(const ClLevel<float>& F, const ClLevel<float>* C, float* solo)
{
    const int n = F.n, half = n >> 1, nc = n >> 1, chalf = nc >> 1, plane = nc * chalf;
    const int K0 = (F.p0 + 1) >> 1, nK = ((F.p0 + F.np + 1) >> 1) - K0;
    const int total = chalf * nc * nK;
    constexpr float sixth = 1.0f / 6.0f;
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int t2, J, K;
        cl_split(t, chalf, nc, t2, J, K);
        K += K0;
        const int c2 = 2 * t2;
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int dk = 0; dk < 2; ++dk)
#pragma unroll
            for (int dj = 0; dj < 2; ++dj) {
                const int j = 2 * J + dj, q = 2 * K + dk - F.p0 + 1, odd = (dj + dk) & 1;
                const int jm = j == 0 ? n - 1 : j - 1, jp = j == n - 1 ? 0 : j + 1;
                const float* row = F.zb[q] + j * half;
                auto pair = [&](const float* a) { return *reinterpret_cast<const float2*>(a + c2); };
                const float2 c = pair(row), ym = pair(F.zb[q] + jm * half), yp = pair(F.zb[q] + jp * half);
                const float2 zm = pair(F.zb[q - 1] + j * half), zp = pair(F.zb[q + 1] + j * half);
                const float2 b = pair(F.br[q] + j * half), m = pair(F.zr[q] + j * half);
                const float e = row[odd ? (c2 + 2 == half ? 0 : c2 + 2) : (c2 == 0 ? half - 1 : c2 - 1)];
                const float x0 = odd ? c.x : e, x1 = odd ? c.y : c.x, x2 = odd ? e : c.y;
                s0 = s0 + (b.x - fmaf(((((x0 + x1) + ym.x) + yp.x) + zm.x) + zp.x, sixth, -m.x));
                s1 = s1 + (b.y - fmaf(((((x1 + x2) + ym.y) + yp.y) + zm.y) + zp.y, sixth, -m.y));
            }
        // coarse cells 2 t2 (colour of J + K) and 2 t2 + 1, both at compact t2
        const int even_black = (J + K) & 1, o = t2 + chalf * J;
        float *be, *bo;
        int c = 0;
        if (C) {
            c = cl_owner(K, nc);
            const int at = (K - cl_first(c, nc)) * plane + o;
            be = (even_black ? C->beta_b : C->beta_r) + at;
            bo = (even_black ? C->beta_r : C->beta_b) + at;
        } else {
            be = solo + (2 + even_black) * nc * plane + K * plane + o;
            bo = solo + (3 - even_black) * nc * plane + K * plane + o;
        }
        const float b0 = s0 * 0.5f, b1 = s1 * 0.5f;
        *cl_map(be, c) = b0;
        *cl_map(bo, c) = b1;
        if (C) *cl_map(C->phi_r + (K - cl_first(c, nc)) * plane + o, c) = fmaf(0.f, sixth, -(even_black ? b1 : b0));
    }
}

template <typename T>
__device__ __forceinline__ void cl_restrict_any(const ClLevel<T>& F, const ClLevel<T>* C, T* solo)
{
    if constexpr (sizeof(T) == 4) {
        if ((F.n & 7) == 0) return cl_restrict2(F, C, solo);
    }
    cl_restrict<T>(F, C, solo);
}

// the coarse planes a slab's prolongation reads, (p0 >> 1) - 1 on, into this CTA
template <typename T>
__device__ __forceinline__ void cl_stage(const ClLevel<T>& F, const ClLevel<T>* C, T* solo, T* stage, int cap)
{
    const int nc = F.n >> 1, chalf = nc >> 1, plane = nc * chalf;
    if (F.np == 0) return;
    const int Kf = (F.p0 >> 1) - 1, nK = ((F.p0 + F.np - 1) >> 1) + 1 - Kf + 1;
    // whole 16-byte words where a plane is a number of them
    constexpr int kW = 16 / sizeof(T);
    const int w = plane % kW == 0 ? kW : 1, pw = plane / w;
    for (int t = threadIdx.x; t < 2 * nK * pw; t += blockDim.x) {
        int o, k, color;
        cl_split(t, pw, nK, o, k, color);
        const int K = (Kf + k + nc) % nc;
        const T* src;
        if (C) {
            const int c = cl_owner(K, nc);
            src = cl_map((color ? C->phi_b : C->phi_r) + (K - cl_first(c, nc)) * plane + o * w, c);
        } else {
            src = cl_map(solo + color * nc * plane + K * plane + o * w, 0);
        }
        T* dst = stage + color * cap + k * plane + o * w;
        if (w == kW) *reinterpret_cast<float4*>(dst) = *reinterpret_cast<const float4*>(src);
        else *dst = *src;
    }
}

// the staged coarse correction into the black cells of the own planes
template <typename T>
__device__ __forceinline__ void cl_prolong(const ClLevel<T>& F, const T* stage, int cap)
{
    const int n = F.n, half = n >> 1, nc = n >> 1, chalf = nc >> 1, plane = nc * chalf;
    const int Kf = (F.p0 >> 1) - 1, total = half * n * F.np;
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int ih, j, q;
        cl_split(t, half, n, ih, j, q);
        const int k = F.p0 + q;
        const int odd = (j + k + 1) & 1;   // the black cell of the pair is x = 2 ih + odd
        const int J = j >> 1, K = (k >> 1) - Kf;
        const int Js[2] = {J, tail_wrap((j & 1) ? J + 1 : J - 1, nc)};
        const int Ks[2] = {K, (k & 1) ? K + 1 : K - 1};
        const int Is[2] = {ih, tail_wrap(odd ? ih + 1 : ih - 1, nc)};
        T s = T(0);
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int tt = 0; tt < 2; ++tt) {
                    const int I = Is[tt], Kg = Kf + Ks[b];
                    const T v = stage[((I + Js[a] + Kg) & 1) * cap + Ks[b] * plane + Js[a] * chalf + (I >> 1)];
                    s = tail_fma(tail_prolong_w<T>(tt + 2 * a + 4 * b), v, s);
                }
        F.phi_b[t] = F.phi_b[t] + s;
    }
}

// the same, four compact columns of a row at a time (half % 4 == 0, chalf % 2 == 0): the
// six coarse values beside them of each of four coarse rows
__device__ __forceinline__ void cl_prolong4(const ClLevel<float>& F, const float* stage, int cap)
{
    const int n = F.n, half = n >> 1, nc = n >> 1, chalf = nc >> 1, plane = nc * chalf, h4 = half >> 2;
    const int Kf = (F.p0 >> 1) - 1, total = h4 * n * F.np;
    float4* black = reinterpret_cast<float4*>(F.phi_b);
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int t4, j, q;
        cl_split(t, h4, n, t4, j, q);
        const int k = F.p0 + q, c2 = 2 * t4;
        const int odd = (j + k + 1) & 1;   // the black cells are x = 2 ih + odd
        const int J = j >> 1, K = (k >> 1) - Kf;
        const int Js[2] = {J, tail_wrap((j & 1) ? J + 1 : J - 1, nc)};
        const int Ks[2] = {K, (k & 1) ? K + 1 : K - 1};
        float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                const int par = (Js[a] + Kf + Ks[b]) & 1;   // colour of the row's even x
                const float* row = stage + Ks[b] * plane + Js[a] * chalf;
                const float2 e = *reinterpret_cast<const float2*>(row + par * cap + c2);
                const float2 o = *reinterpret_cast<const float2*>(row + (1 - par) * cap + c2);
                // x = ih0 - 1 or ih0 + 4, whichever the black cells reach
                const float z = odd ? row[par * cap + (c2 + 2 == chalf ? 0 : c2 + 2)]
                                    : row[(1 - par) * cap + (c2 == 0 ? chalf - 1 : c2 - 1)];
                const float w[4] = {e.x, o.x, e.y, o.y};
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float side = odd ? (r == 3 ? z : w[r == 3 ? 3 : r + 1])
                                           : (r == 0 ? z : w[r == 0 ? 0 : r - 1]);
                    s[r] = fmaf(tail_prolong_w<float>(2 * a + 4 * b), w[r], s[r]);
                    s[r] = fmaf(tail_prolong_w<float>(1 + 2 * a + 4 * b), side, s[r]);
                }
            }
        float4 p = black[t];
        p.x = p.x + s[0];
        p.y = p.y + s[1];
        p.z = p.z + s[2];
        p.w = p.w + s[3];
        black[t] = p;
    }
}

template <typename T>
__device__ __forceinline__ void cl_prolong_any(const ClLevel<T>& F, const T* stage, int cap)
{
    if constexpr (sizeof(T) == 4) {
        if ((F.n & 7) == 0) return cl_prolong4(F, stage, cap);
    }
    cl_prolong<T>(F, stage, cap);
}

// The opening red half sweep of a level whose correction is 0, in place of one with its
// barrier: each thread takes the cells it has just copied (cl_copy's order).
template <typename T>
__device__ __forceinline__ void cl_open(const ClLevel<T>& L)
{
    const int cnt = L.n * (L.n >> 1) * L.np;
    for (int t = threadIdx.x; t < cnt; t += blockDim.x) L.phi_r[t] = tail_fma(T(0), tail_sixth<T>(), -L.beta_r[t]);
}

// One V-cycle on the slab levels, ending after a cluster barrier.  start: the finest
// level's correction is in place (0), is 0 throughout (1), or has had its opening red half
// sweep from 0 (2), as the coarser ones have from the restriction (ten FP64 steps at 64^3
// 18.65 -> 18.5 ms).
template <typename T>
__device__ __forceinline__ void cl_vcycle(const ClArgs<T>& A, ClShared<T>& S, T* mem, int start)
{
    const int rank = cl_rank();
    for (int l = 0; l < A.nd; ++l) {
        for (int sw = 0; sw < A.nu1; ++sw) {
            if (sw > 0 || (l == 0 && start < 2)) {
                cl_half_sweep<T>(S.lv[l], 0, sw == 0 && start == 1);
                cl_barrier();
            }
            cl_half_sweep<T>(S.lv[l], 1, false);
            cl_barrier();
        }
        const bool last = l + 1 == A.nd;
        cl_restrict_any<T>(S.lv[l], last ? nullptr : &S.lv[l + 1], S.solo[0].base);
        cl_barrier();
    }
    if (rank == 0) vcycle_solo<T>(S.solo, A.ns, A.nu1, A.nu2, S.g, A.nb, mem + A.stage, true);
    cl_barrier();
    for (int l = A.nd - 1; l >= 0; --l) {
        const bool last = l + 1 == A.nd;
        const int nc = A.n[l] >> 1, cap = (A.planes[l] / 2 + 3) * nc * (nc >> 1);
        cl_stage<T>(S.lv[l], last ? nullptr : &S.lv[l + 1], S.solo[0].base, mem + A.stage, cap);
        __syncthreads();
        cl_prolong_any<T>(S.lv[l], mem + A.stage, cap);
        cl_barrier();
        for (int sw = 0; sw < A.nu2; ++sw) {
            cl_half_sweep<T>(S.lv[l], 0, false);
            cl_barrier();
            cl_half_sweep<T>(S.lv[l], 1, false);
            cl_barrier();
        }
    }
}

// CTA 0's copy of the bottom's Green's function (the first barrier of a V-cycle follows)
template <typename T>
__device__ __forceinline__ void cl_load_green(const ClArgs<T>& A, ClShared<T>& S)
{
    if (cl_rank() == 0)
        for (int t = threadIdx.x; t < A.nb * A.nb * A.nb; t += blockDim.x) S.g[t] = A.G[t];
}

// own planes between a split level in global memory and the slab
template <typename T>
__device__ __forceinline__ void cl_copy(T* dst, const T* src, int count)
{
    for (int t = threadIdx.x; t < count; t += blockDim.x) dst[t] = src[t];
}

template <typename T, typename LV>
__device__ __forceinline__ void cl_load(const ClLevel<T>& L, const LV& G, bool with_phi)
{
    const int plane = L.n * (L.n >> 1), cnt = plane * L.np;
    const size_t o = (size_t)L.p0 * plane;
    cl_copy<T>(L.beta_r, G.beta_r + o, cnt);
    cl_copy<T>(L.beta_b, G.beta_b + o, cnt);
    if (with_phi) {
        cl_copy<T>(L.phi_r, G.phi_r + o, cnt);
        cl_copy<T>(L.phi_b, G.phi_b + o, cnt);
    }
}

template <typename T, typename LV>
__device__ __forceinline__ void cl_store(const ClLevel<T>& L, const LV& G)
{
    const int plane = L.n * (L.n >> 1), cnt = plane * L.np;
    const size_t o = (size_t)L.p0 * plane;
    cl_copy<T>(G.phi_r + o, L.phi_r, cnt);
    cl_copy<T>(G.phi_b + o, L.phi_b, cnt);
}

// block maximum of v (all threads), into slot s of every CTA of the cluster
template <typename T>
__device__ __forceinline__ void cl_norm_put(ClShared<T>& S, int s, unsigned long long v)
{
    __shared__ unsigned long long w[32];
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, off));
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        v = threadIdx.x < (blockDim.x >> 5) ? w[threadIdx.x] : 0ULL;
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, off));
        if (threadIdx.x < kClCtas) *cl_map(&S.part[s][cl_rank()], (int)threadIdx.x) = v;
    }
    __syncthreads();
}

// after a cluster barrier: the maximum over the CTAs
template <typename T>
__device__ __forceinline__ unsigned long long cl_norm_get(const ClShared<T>& S, int s)
{
    unsigned long long v = 0;
#pragma unroll
    for (int c = 0; c < kClCtas; ++c) v = max(v, S.part[s][c]);
    return v;
}

// host: A for the levels of b from li on; false if this path does not take them
template <typename T>
inline bool cl_args(const Ctx& c, const Box& b, size_t li, ClArgs<T>& A)
{
    if (c.p.mg_fused_edge <= 0 || c.p.nu1 <= 0 || c.p.nu2 <= 0) return false;
    int n[kClMaxLevels + kMaxTail];
    const size_t levels = b.levels.size() - li;
    if (levels > (size_t)(kClMaxLevels + kMaxTail)) return false;
    for (size_t l = 0; l < levels; ++l) n[l] = b.levels[li + l].n;
    if (!cl_layout<T>(A, n, (int)levels)) return false;
    A.nu1 = c.p.nu1;
    A.nu2 = c.p.nu2;
    A.nb = b.nb;
    A.G = sizeof(T) == 4 ? reinterpret_cast<const T*>(b.Gf) : reinterpret_cast<const T*>(b.G);
    return true;
}

// host: whether a kernel can run here as one cluster with that much dynamic shared memory
template <typename K>
inline bool cl_prepare(K kernel, size_t bytes, int threads = kClThreads)
{
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kClCtas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(kClCtas);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = bytes;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return clusters >= 1;
}

template <typename... KArgs, typename... Args>
inline void launch_cluster(Ctx& c, void (*kernel)(KArgs...), size_t bytes, Args... args)
{
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kClCtas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = c.pdl ? 1 : 0;
    cfg.gridDim = dim3(kClCtas);
    cfg.blockDim = dim3(kClThreads);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = c.stream;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
    if (e != cudaSuccess && c.launch_error == cudaSuccess) c.launch_error = e;   // check_launch reports it
}

}  // namespace nyxpm
