// The coarse end of a V-cycle run by one CTA: every level from the first one of
// at most mg_fused_edge cells per edge (half that in FP64) down to the bottom is smoothed,
// restricted, solved exactly and prolonged by the block, with a block barrier
// between the passes.  It replaces some 20 dependent launches of a few hundred
// to a few thousand cells each per V-cycle.  (One SM is slower than a
// grid-wide launch from 32^3 cells up: 16 is the default edge.)
//
// Each cell's arithmetic is the one of the per-pass kernels (red-black
// Gauss-Seidel, residual + restriction, circulant bottom solve, trilinear
// prolongation + correction), in the same order, so a fused V-cycle gives the
// same bits as the launches it replaces.  The code is templated on the scalar:
// float for the mixed form's inner V-cycles, double for the coarsest levels of
// the FP64 form (whose restriction sums the red children only, as k_restrict<1>).  Loads are plain (not the read-only
// path): the block writes what it reads.
#pragma once

#include "pm_common.cuh"

namespace nyxpm {

constexpr int kMaxTail = 8;
constexpr int kTailThreads = 1024;   // FP32 tail: levels up to 16^3
constexpr int kTailThreadsD = 256;   // FP64 tail: levels up to 8^3 (256 cells per half sweep)

__device__ __forceinline__ int tail_wrap(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

// t -> (x, y, z) with x < nx, y < ny: shifts when both are powers of two
__device__ __forceinline__ void tail_split3(int t, int nx, int ny, int& x, int& y, int& z)
{
    if (((nx & (nx - 1)) | (ny & (ny - 1))) == 0) {
        const int sx = __ffs(nx) - 1, sy = __ffs(ny) - 1;
        x = t & (nx - 1);
        y = (t >> sx) & (ny - 1);
        z = t >> (sx + sy);
    } else {
        const int r = t / nx;
        x = t - r * nx;
        z = r / ny;
        y = r - z * ny;
    }
}

// trilinear weights 27/64, 9/64, 9/64, 3/64, 9/64, 3/64, 3/64, 1/64 at index tt + 2a + 4b
template <typename T>
__device__ __forceinline__ T tail_prolong_w(int idx)
{
    constexpr T w[8] = {T(0.421875), T(0.140625), T(0.140625), T(0.046875),
                        T(0.140625), T(0.046875), T(0.046875), T(0.015625)};
    return w[idx];
}

__device__ __forceinline__ float tail_fma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double tail_fma(double a, double b, double c) { return fma(a, b, c); }
template <typename T>
__device__ __forceinline__ T tail_sixth() { return T(1) / T(6); }

// one red (color 0) or black (1) half sweep of a split level
template <typename T, typename LV>
__device__ __forceinline__ void tail_gsrb(const LV& F, int color)
{
    const int n = F.n, half = n >> 1;
    const int total = half * n * n;
    T* mine = color ? F.phi_b : F.phi_r;
    const T* other = color ? F.phi_r : F.phi_b;
    const T* beta = color ? F.beta_b : F.beta_r;
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int ih, j, k;
        tail_split3(t, half, n, ih, j, k);
        const int q = (j + k + color) & 1;
        const int ihm = q ? ih : (ih == 0 ? half - 1 : ih - 1);
        const int ihp = q ? (ih == half - 1 ? 0 : ih + 1) : ih;
        const int jm = j == 0 ? n - 1 : j - 1, jp = j == n - 1 ? 0 : j + 1;
        const int km = k == 0 ? n - 1 : k - 1, kp = k == n - 1 ? 0 : k + 1;
        const int row = j + n * k;
        T s = other[row * half + ihm] + other[row * half + ihp];
        s = s + other[(jm + n * k) * half + ih];
        s = s + other[(jp + n * k) * half + ih];
        s = s + other[(j + n * km) * half + ih];
        s = s + other[(j + n * kp) * half + ih];
        mine[t] = tail_fma(s, tail_sixth<T>(), -beta[t]);
    }
}

template <typename T, typename LV>
__device__ __forceinline__ T tail_resid(const LV& L, int i, int j, int k)
{
    const int n = L.n;
    const int im = i == 0 ? n - 1 : i - 1, ip = i == n - 1 ? 0 : i + 1;
    const int jm = j == 0 ? n - 1 : j - 1, jp = j == n - 1 ? 0 : j + 1;
    const int km = k == 0 ? n - 1 : k - 1, kp = k == n - 1 ? 0 : k + 1;
    T s = *lv_ptr<T>(L.phi_r, L.phi_b, n, L.split, im, j, k) +
          *lv_ptr<T>(L.phi_r, L.phi_b, n, L.split, ip, j, k);
    s = s + *lv_ptr<T>(L.phi_r, L.phi_b, n, L.split, i, jm, k);
    s = s + *lv_ptr<T>(L.phi_r, L.phi_b, n, L.split, i, jp, k);
    s = s + *lv_ptr<T>(L.phi_r, L.phi_b, n, L.split, i, j, km);
    s = s + *lv_ptr<T>(L.phi_r, L.phi_b, n, L.split, i, j, kp);
    const T c = *lv_ptr<T>(L.phi_r, L.phi_b, n, L.split, i, j, k);
    return *lv_ptr<T>(L.beta_r, L.beta_b, n, L.split, i, j, k) - tail_fma(s, tail_sixth<T>(), -c);
}

// residual of F restricted to the coarse right-hand side; coarse phi = 0.
// red_only: the children with di + dj + dk even only (F ends its pre-smoothing
// with a black half sweep, so the black residuals are round-off)
template <typename T, typename LV>
__device__ __forceinline__ void tail_restrict(const LV& F, const LV& Cv, bool red_only)
{
    const int nc = Cv.n;
    const int total = nc * nc * nc;
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int I, J, K;
        tail_split3(t, nc, nc, I, J, K);
        T s = T(0);
#pragma unroll
        for (int dk = 0; dk < 2; ++dk)
#pragma unroll
            for (int dj = 0; dj < 2; ++dj)
#pragma unroll
                for (int di = 0; di < 2; ++di)
                    if (!red_only || ((di + dj + dk) & 1) == 0)
                        s = s + tail_resid<T>(F, 2 * I + di, 2 * J + dj, 2 * K + dk);
        *lv_ptr<T>(Cv.beta_r, Cv.beta_b, nc, Cv.split, I, J, K) = s * T(0.5);
        *lv_ptr<T>(Cv.phi_r, Cv.phi_b, nc, Cv.split, I, J, K) = T(0);
    }
}

// fine phi += trilinear interpolation of the coarse phi (black: the black fine
// cells only -- the post-smoothing's first half sweep overwrites the red ones
// unread)
template <typename T, typename LV>
__device__ __forceinline__ void tail_prolong(const LV& Cv, const LV& F, bool black)
{
    const int n = F.n, nc = Cv.n, half = n >> 1;
    const int total = half * n * n;
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int ih, j, k;
        tail_split3(t, half, n, ih, j, k);
        const int J = j >> 1, K = k >> 1;
        const int Js[2] = {J, tail_wrap((j & 1) ? J + 1 : J - 1, nc)};
        const int Ks[2] = {K, tail_wrap((k & 1) ? K + 1 : K - 1, nc)};
#pragma unroll
        for (int odd = 0; odd < 2; ++odd) {
            const int i = 2 * ih + odd;
            if (black && ((i + j + k) & 1) == 0) continue;
            const int Is[2] = {ih, tail_wrap(odd ? ih + 1 : ih - 1, nc)};
            T s = T(0);
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int a = 0; a < 2; ++a)
#pragma unroll
                    for (int tt = 0; tt < 2; ++tt)
                        s = tail_fma(tail_prolong_w<T>(tt + 2 * a + 4 * b),
                                     *lv_ptr<const T>(Cv.phi_r, Cv.phi_b, nc, Cv.split, Is[tt], Js[a], Ks[b]),
                                     s);
            T* p = (((i + j + k) & 1) ? F.phi_b : F.phi_r) + t;
            *p = *p + s;
        }
    }
}

// exact bottom solve phi = G (*) beta on the natural nb^3 level (cyclic
// convolution, y in storage order); r and g are kMaxBottom^3 shared arrays
template <typename T, typename LV>
__device__ __forceinline__ void tail_bottom(const LV& B, const T* Gf, int nb, T* r, T* g)
{
    const int nc = nb * nb * nb;
    for (int t = threadIdx.x; t < nc; t += blockDim.x) {
        r[t] = B.beta_r[t];
        g[t] = Gf[t];
    }
    __syncthreads();
    for (int c = threadIdx.x; c < nc; c += blockDim.x) {
        const int i = c % nb, j = (c / nb) % nb, k = c / (nb * nb);
        T s = T(0);
        int y = 0;
        for (int yk = 0; yk < nb; ++yk) {
            const int dk = tail_wrap(k - yk, nb) * nb * nb;
            for (int yj = 0; yj < nb; ++yj) {
                const int djk = dk + tail_wrap(j - yj, nb) * nb;
                for (int yi = 0; yi < nb; ++yi, ++y) s = tail_fma(g[djk + tail_wrap(i - yi, nb)], r[y], s);
            }
        }
        B.phi_r[c] = s;
    }
}

// the V-cycle over lv[0 .. nl-1] (lv[nl-1] the natural bottom) by the calling
// block; lv[0]'s right-hand side is in place and its phi is the initial guess
// red_restrict: restrictions after pre-smoothing sum the red children only
template <typename T, typename LV>
__device__ __forceinline__ void vcycle_tail(const LV* lv, int nl, int nu1, int nu2, const T* Gf,
                                            int nb, T* r, T* g, bool red_restrict)
{
    for (int l = 0; l + 1 < nl; ++l) {
        for (int sw = 0; sw < nu1; ++sw) {
            tail_gsrb<T>(lv[l], 0);
            __syncthreads();
            tail_gsrb<T>(lv[l], 1);
            __syncthreads();
        }
        tail_restrict<T>(lv[l], lv[l + 1], red_restrict && nu1 > 0);
        __syncthreads();
    }
    tail_bottom<T>(lv[nl - 1], Gf, nb, r, g);
    __syncthreads();
    for (int l = nl - 2; l >= 0; --l) {
        tail_prolong<T>(lv[l + 1], lv[l], nu2 > 0);
        __syncthreads();
        for (int sw = 0; sw < nu2; ++sw) {
            tail_gsrb<T>(lv[l], 0);
            __syncthreads();
            tail_gsrb<T>(lv[l], 1);
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------------------
// The same V-cycle with every level in the block's shared memory, for levels of at most
// kSoloSlots blockDim.x compact cells per colour and pre- and post-smoothing (nu1, nu2 >
// 0).  What bounds it is latency and instructions, not arithmetic: a half sweep of 16^3
// is 2048 FP32 updates.  A thread keeps its cells' neighbour offsets in registers over a
// level's sweeps (they are the same for both colours), the red residuals are formed one
// cell per thread before the coarse cells add them up, and the coarse correction is put
// in natural layout once so that the prolongation indexes it without a colour test.
// Measured on GB300 against vcycle_tail on shared memory (SM clocks, 512 and 1024
// threads): 16^3 down to 4^3 in FP32 43,000 -> 19,000, 8^3 down to 4^3 in FP64 30,000 ->
// 19,000.
// ---------------------------------------------------------------------------
constexpr int kSoloSlots = 4;

// the four arrays phi_r, phi_b, beta_r, beta_b of a split level (or phi, beta of the
// natural bottom), one after another
template <typename T>
struct SoloLevel {
    int n;
    T* base;
};

// compact cell t of a level of edge n: t itself and its neighbours' offsets
struct SoloCell {
    int t, xm, xp, ym, yp, zm, zp, odd;
    __device__ __forceinline__ void set(int tt, int n)
    {
        const int half = n >> 1;
        int ih, j, k;
        t = tt;
        tail_split3(tt, half, n, ih, j, k);
        const int row = (j + n * k) * half;
        xm = row + (ih == 0 ? half - 1 : ih - 1);
        xp = row + (ih == half - 1 ? 0 : ih + 1);
        ym = tt + ((j == 0 ? n : 0) - 1) * half;
        yp = tt + (1 - (j == n - 1 ? n : 0)) * half;
        zm = tt + ((k == 0 ? n : 0) - 1) * half * n;
        zp = tt + (1 - (k == n - 1 ? n : 0)) * half * n;
        odd = (j + k) & 1;
    }
    // neighbour sum in the other colour's array a; o: the cell's x is 2 ih + o
    template <typename T>
    __device__ __forceinline__ T sum(const T* a, int o) const
    {
        const T c = a[t], e = a[o ? xp : xm];
        T s = (o ? c : e) + (o ? e : c);
        s = s + a[ym];
        s = s + a[yp];
        s = s + a[zm];
        s = s + a[zp];
        return s;
    }
};

// sweeps red-black sweeps; zero: the level's correction is 0 on entry (not read)
template <typename T>
__device__ __forceinline__ void solo_smooth(const SoloCell (&cell)[kSoloSlots], T* base, int n, int sweeps, bool zero)
{
    const int nh = (n * n * n) >> 1;
    for (int sw = 0; sw < 2 * sweeps; ++sw) {
        const int color = sw & 1;
        T* mine = base + (color ? nh : 0);
        const T* other = base + (color ? 0 : nh);
        const T* beta = base + (color ? 3 : 2) * nh;
#pragma unroll
        for (int s = 0; s < kSoloSlots; ++s) {
            if (cell[s].t >= nh) break;
            const T sum = zero && sw == 0 ? T(0) : cell[s].template sum<T>(other, cell[s].odd ^ color);
            mine[cell[s].t] = tail_fma(sum, tail_sixth<T>(), -beta[cell[s].t]);
        }
        __syncthreads();
    }
}

// lv[0 .. nl-1] in shared memory (lv[nl-1] the natural bottom), lv[0]'s right-hand side in
// place, its correction 0 on entry if zero; g: the bottom's Green's function in shared
// memory; tmp: shared scratch of half as many values as lv[0] has cells
template <typename T>
__device__ __forceinline__ void vcycle_solo(const SoloLevel<T>* lv, int nl, int nu1, int nu2, const T* g, int nb,
                                            T* tmp, bool zero)
{
    SoloCell cell[kSoloSlots];
    for (int l = 0; l + 1 < nl; ++l) {
        const int n = lv[l].n, nh = (n * n * n) >> 1, nc = n >> 1;
        T* base = lv[l].base;
#pragma unroll
        for (int s = 0; s < kSoloSlots; ++s) {
            cell[s].t = nh;
            if ((int)(threadIdx.x + s * blockDim.x) < nh) cell[s].set(threadIdx.x + s * blockDim.x, n);
        }
        solo_smooth<T>(cell, base, n, nu1, zero || l > 0);
        // red residuals, then each coarse cell's four in (dk, dj) order
#pragma unroll
        for (int s = 0; s < kSoloSlots; ++s) {
            if (cell[s].t >= nh) break;
            const int t = cell[s].t;
            tmp[t] = base[2 * nh + t] -
                     tail_fma(cell[s].template sum<T>(base + nh, cell[s].odd), tail_sixth<T>(), -base[t]);
        }
        __syncthreads();
        const bool split = l + 2 < nl;
        const int cc = nc * nc * nc;
        for (int t = threadIdx.x; t < cc; t += blockDim.x) {
            int I, J, K;
            tail_split3(t, nc, nc, I, J, K);
            T s = T(0);
#pragma unroll
            for (int dk = 0; dk < 2; ++dk)
#pragma unroll
                for (int dj = 0; dj < 2; ++dj) s = s + tmp[I + nc * (2 * J + dj + n * (2 * K + dk))];
            const int at = split ? cc + ((I + J + K) & 1) * (cc >> 1) + (I >> 1) + (nc >> 1) * (J + nc * K) : cc + t;
            lv[l + 1].base[at] = s * T(0.5);
        }
        __syncthreads();
    }
    // exact bottom solve phi = G (*) beta (cyclic convolution, y in storage order)
    {
        T* phi = lv[nl - 1].base;
        const int cc = nb * nb * nb;
        const T* r = phi + cc;
        for (int c = threadIdx.x; c < cc; c += blockDim.x) {
            const int i = c % nb, j = (c / nb) % nb, k = c / (nb * nb);
            T s = T(0);
            if (nb == 4) {
#pragma unroll 4
                for (int yjk = 0; yjk < 16; ++yjk) {
                    const int row = 16 * ((k - (yjk >> 2)) & 3) + 4 * ((j - yjk) & 3);
#pragma unroll
                    for (int yi = 0; yi < 4; ++yi) s = tail_fma(g[row + ((i - yi) & 3)], r[4 * yjk + yi], s);
                }
            } else {
                int y = 0;
                for (int yk = 0; yk < nb; ++yk) {
                    const int dk = tail_wrap(k - yk, nb) * nb * nb;
                    for (int yj = 0; yj < nb; ++yj) {
                        const int djk = dk + tail_wrap(j - yj, nb) * nb;
                        for (int yi = 0; yi < nb; ++yi, ++y) s = tail_fma(g[djk + tail_wrap(i - yi, nb)], r[y], s);
                    }
                }
            }
            phi[c] = s;
        }
        __syncthreads();
    }
    for (int l = nl - 2; l >= 0; --l) {
        const int n = lv[l].n, nh = (n * n * n) >> 1, nc = n >> 1, cc = nc * nc * nc;
        T* base = lv[l].base;
        const T* coarse = lv[l + 1].base;
        if (l + 2 < nl) {
            for (int t = threadIdx.x; t < cc; t += blockDim.x) {
                int I, J, K;
                tail_split3(t, nc, nc, I, J, K);
                tmp[t] = coarse[((I + J + K) & 1) * (cc >> 1) + (I >> 1) + (nc >> 1) * (J + nc * K)];
            }
            __syncthreads();
            coarse = tmp;
        }
#pragma unroll
        for (int s = 0; s < kSoloSlots; ++s) {
            cell[s].t = nh;
            if ((int)(threadIdx.x + s * blockDim.x) < nh) {
                cell[s].set(threadIdx.x + s * blockDim.x, n);
                int ih, j, k;
                tail_split3(cell[s].t, nc, n, ih, j, k);
                // the pair's black cell is x = 2 ih + 1 - odd
                const int I1 = tail_wrap(cell[s].odd ? ih - 1 : ih + 1, nc);
                const int J0 = nc * (j >> 1), J1 = nc * tail_wrap((j & 1) ? (j >> 1) + 1 : (j >> 1) - 1, nc);
                const int K0 = nc * nc * (k >> 1), K1 = nc * nc * tail_wrap((k & 1) ? (k >> 1) + 1 : (k >> 1) - 1, nc);
                T v = T(0);
#pragma unroll
                for (int b = 0; b < 2; ++b)
#pragma unroll
                    for (int a = 0; a < 2; ++a) {
                        const T* row = coarse + (a ? J1 : J0) + (b ? K1 : K0);
                        v = tail_fma(tail_prolong_w<T>(2 * a + 4 * b), row[ih], v);
                        v = tail_fma(tail_prolong_w<T>(1 + 2 * a + 4 * b), row[I1], v);
                    }
                base[nh + cell[s].t] = base[nh + cell[s].t] + v;
            }
        }
        __syncthreads();
        solo_smooth<T>(cell, base, n, nu2, false);
    }
}

}  // namespace nyxpm
