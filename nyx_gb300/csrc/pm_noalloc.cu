// nyxpm_deposit_noalloc: the CIC mass density of particles that are already in
// device memory, computed without allocating any device memory.
//
// Who needs it: a host code whose device memory is owned by its own arena
// allocator (an AMReX build reserves most of the GPU in its arena at start-up
// and hands out pieces of it) cannot let a library call cudaMalloc behind its
// back -- the call can fail for lack of free memory or fragment the memory the
// arena manages.  Such a caller passes its own input and output buffers; the
// scratch the counting sort needs lives in a file-scope __device__ array that
// every GPU which loads this library holds until the process exits.
//
// Limits: grid edge n <= 64 (262,144 cells) and at most 262,144 particles, so
// the array is ~10 MiB.  Larger problems go through nyxpm_box_create /
// nyxpm_deposit, which allocate.
//
// The arithmetic (key, sort order, per-key partial sums, cell sums) is that of
// nyxpm_deposit for uniform masses, so both give the same density bit for bit.
// Like nyxpm_deposit it refuses non-finite positions: the key pass counts them,
// and the call reads the count back before it returns.
// Built with --fmad=false like the other FP64 units.
#include "pm_cluster.cuh"
#include "pm_common.cuh"

#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>

namespace nyxpm {

namespace {

constexpr int kNaMaxN = 64;
constexpr long long kNaMaxCells = (long long)kNaMaxN * kNaMaxN * kNaMaxN;
constexpr long long kNaMaxParticles = 262144;
constexpr int kNaScanT = 512, kNaScanIPT = 8, kNaScanTile = kNaScanT * kNaScanIPT;
constexpr long long kNaTiles = (kNaMaxCells + kNaScanTile - 1) / kNaScanTile;

// Up to this many particles and cells the sort is one cluster launch (na_sort), beyond it
// and where the device or the stream cannot place that cluster ten launches over the whole
// chip.  Measured, a call from the host, particles on a lattice: 8^3 77 -> 40 us, 32^3
// 95 -> 61 us, 48^3 112 -> 87 us; 64^3 with 262,144 particles 134 us by launches, 136 by the
// cluster, 155 before the deposit below.
constexpr long long kNaClusterMax = 131072;
// scratch layout, each part rounded up to 256 bytes
constexpr size_t up256(size_t b) { return (b + 255) & ~size_t(255); }
constexpr size_t kOffCount = 0;
constexpr size_t kOffStart = kOffCount + up256(4 * kNaMaxCells);
constexpr size_t kOffTiles = kOffStart + up256(4 * (kNaMaxCells + 1));
constexpr size_t kOffLongCount = kOffTiles + up256(4 * (kNaTiles + 1));
constexpr size_t kOffLongList = kOffLongCount + 256;
constexpr size_t kOffKey = kOffLongList + up256(4 * (kNaMaxParticles / 32 + 2));
constexpr size_t kOffPerm = kOffKey + up256(4 * kNaMaxParticles);
constexpr size_t kOffX = kOffPerm + up256(4 * kNaMaxParticles);
constexpr size_t kOffY = kOffX + up256(8 * kNaMaxParticles);
constexpr size_t kOffZ = kOffY + up256(8 * kNaMaxParticles);
constexpr size_t kScratchBytes = kOffZ + up256(8 * kNaMaxParticles);

// the scratch: every call shares it, and it keeps the last call's contents
static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

// the cluster sort (declared here for its launch attribute)
__global__ void na_sort(int np, int n, double dxi, const double* __restrict__ x, const double* __restrict__ y,
                        const double* __restrict__ z, int* key, int* count, int* start, int* perm, int* long_list,
                        int* long_count, int* bad);

constexpr int kNaThreads = 1024;   // of a CTA of the cluster sort

constexpr int kMaxDevices = 64;
std::mutex g_setup_mutex;
unsigned char* g_scratch_addr[kMaxDevices] = {};
int g_sm_count[kMaxDevices] = {};
int g_cluster[kMaxDevices] = {};   // the device can place the cluster sort: 1 yes, -1 no, 0 not asked yet

// The device address of the scratch on the current device (the host-side name
// of the array is not a device address).  It is looked up again on every call
// whose stream is not capturing -- a device reset reloads the module and may
// move the array -- and the last address found is used while a capture runs.
nyxpm_status scratch_address(cudaStream_t stream, unsigned char** out, int* sm_count, bool* cluster,
                             bool* capturing, char* errbuf, size_t errlen)
{
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        cudaGetLastError();
        if (errbuf && errlen) std::snprintf(errbuf, errlen, "no current CUDA device");
        return NYXPM_NO_DEVICE;
    }
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &cap) != cudaSuccess) {
        cudaGetLastError();
        cap = cudaStreamCaptureStatusNone;
    }
    std::lock_guard<std::mutex> lock(g_setup_mutex);
    if (!g_scratch_addr[dev] || cap == cudaStreamCaptureStatusNone) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            cudaGetLastError();
            if (errbuf && errlen)
                std::snprintf(errbuf, errlen, "cudaGetSymbolAddress of the scratch failed: %s",
                              cudaGetErrorString(e));
            return NYXPM_CUDA_ERROR;
        }
        g_scratch_addr[dev] = static_cast<unsigned char*>(p);
        int sms = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
            cudaGetLastError();
            sms = 1;
        }
        g_sm_count[dev] = sms > 0 ? sms : 1;
        if (!g_cluster[dev])
            g_cluster[dev] = cl_prepare(na_sort, 0, kNaThreads) ? 1 : -1;
        else if (cudaFuncSetAttribute(na_sort, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
            cudaGetLastError();   // (a device reset forgets it) the launch reports it
    }
    *out = g_scratch_addr[dev];
    *sm_count = g_sm_count[dev];
    *cluster = g_cluster[dev] > 0;
    *capturing = cap != cudaStreamCaptureStatusNone;
    return NYXPM_OK;
}

__device__ __forceinline__ int na_key1(double x, double dxi, int n, double* frac)
{
    const double l = fma(x, dxi, 0.5);
    int il;
    const double fl = floor_int(l, &il);
    *frac = l - fl;
    return wrapi(il, n);
}

__global__ void na_zero(int* a, long long cnt)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < cnt) a[t] = 0;
}

// A non-finite coordinate is counted in *bad (the call then refuses the input);
// its key is still a valid cell (the float-to-int conversion saturates and a NaN
// converts to 0), so no access leaves the arrays.
__global__ void na_keys(long long np, int n, double dxi, const double* __restrict__ x,
                        const double* __restrict__ y, const double* __restrict__ z, int* key, int* count,
                        int* bad)
{
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= np) return;
    const double px = x[q], py = y[q], pz = z[q];
    if (!(isfinite(px) && isfinite(py) && isfinite(pz))) atomicAdd(bad, 1);
    double f;
    const int i = na_key1(px, dxi, n, &f);
    const int j = na_key1(py, dxi, n, &f);
    const int k = na_key1(pz, dxi, n, &f);
    const int K = (int)cidx(i, j, k, n);
    key[q] = K;
    atomicAdd(count + K, 1);
}

__device__ __forceinline__ int na_warp_scan(int v)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

__device__ int na_block_scan(int v, int* total)
{
    __shared__ int ws[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int inc = na_warp_scan(v);
    if (lane == 31) ws[w] = inc;
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x >> 5;
        int s = lane < nw ? ws[lane] : 0;
        s = na_warp_scan(s);
        ws[lane] = s;
    }
    __syncthreads();
    const int before = (w > 0 ? ws[w - 1] : 0) + inc - v;
    *total = ws[(blockDim.x >> 5) - 1];
    __syncthreads();
    return before;
}

__global__ void na_scan_reduce(const int* __restrict__ in, int cnt, int* tiles)
{
    const long long base = (long long)blockIdx.x * kNaScanTile + (long long)threadIdx.x * kNaScanIPT;
    int s = 0;
#pragma unroll
    for (int t = 0; t < kNaScanIPT; ++t)
        if (base + t < cnt) s += in[base + t];
    int total;
    na_block_scan(s, &total);
    if (threadIdx.x == 0) tiles[blockIdx.x] = total;
}

__global__ void na_scan_top(int* tiles, int ntiles)
{
    int carry = 0;
    for (int b0 = 0; b0 < ntiles; b0 += blockDim.x) {
        const int i = b0 + threadIdx.x;
        const int v = i < ntiles ? tiles[i] : 0;
        int total;
        const int ex = na_block_scan(v, &total);
        if (i < ntiles) tiles[i] = carry + ex;
        carry += total;
    }
}

__global__ void na_scan_down(const int* __restrict__ in, int cnt, const int* __restrict__ tiles, int* out)
{
    const long long base = (long long)blockIdx.x * kNaScanTile + (long long)threadIdx.x * kNaScanIPT;
    int v[kNaScanIPT];
    int s = 0;
#pragma unroll
    for (int t = 0; t < kNaScanIPT; ++t) {
        v[t] = base + t < cnt ? in[base + t] : 0;
        s += v[t];
    }
    int total;
    int run = na_block_scan(s, &total) + tiles[blockIdx.x];
#pragma unroll
    for (int t = 0; t < kNaScanIPT; ++t) {
        if (base + t < cnt) out[base + t] = run;
        run += v[t];
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) out[cnt] = run;
}

__global__ void na_scatter(long long np, const int* __restrict__ key, const int* __restrict__ start,
                           int* count, int* perm)
{
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= np) return;
    const int K = key[q];
    perm[start[K] + atomicSub(count + K, 1) - 1] = (int)q;
}

// order each key segment by original particle index (so the deposit order, and
// with it the density, does not depend on how the atomics were served)
__global__ void na_fix_short(int nc, const int* __restrict__ start, int* perm, int* long_list,
                             int* long_count)
{
    const int K = blockIdx.x * blockDim.x + threadIdx.x;
    if (K >= nc) return;
    const int s = start[K], len = start[K + 1] - s;
    if (len <= 1) return;
    if (len > 32) {
        long_list[atomicAdd(long_count, 1)] = K;
        return;
    }
    sort_short_segment(perm, s, len);
}

// Long segments: a rank sort by one block per segment (the values are distinct).
// A segment of up to kNaLongSmem entries is ranked from shared memory; a longer
// one (every particle in a few cells) from global memory.
constexpr int kNaLongSmem = 12288;

__global__ void na_fix_long(const int* __restrict__ start, const int* __restrict__ long_list,
                            const int* __restrict__ long_count, int* perm, int* tmp)
{
    __shared__ int sv[kNaLongSmem];
    const int total = *long_count;
    for (int li = blockIdx.x; li < total; li += gridDim.x) {
        const int K = long_list[li];
        const int s = start[K], len = start[K + 1] - s;
        const bool in_smem = len <= kNaLongSmem;
        __syncthreads();
        if (in_smem)
            for (int t = threadIdx.x; t < len; t += blockDim.x) sv[t] = perm[s + t];
        __syncthreads();
        for (int t = threadIdx.x; t < len; t += blockDim.x) {
            const int v = in_smem ? sv[t] : perm[s + t];
            int rank = 0;
            if (in_smem) {
                for (int u = 0; u < len; ++u) rank += sv[u] < v;
            } else {
                for (int u = 0; u < len; ++u) rank += perm[s + u] < v;
            }
            tmp[s + rank] = v;
        }
        __syncthreads();
        for (int t = threadIdx.x; t < len; t += blockDim.x) perm[s + t] = tmp[s + t];
    }
}

__global__ void na_gather(long long np, const int* __restrict__ perm, const double* __restrict__ x,
                          const double* __restrict__ y, const double* __restrict__ z, double* xs,
                          double* ys, double* zs)
{
    const long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= np) return;
    const int q = perm[s];
    xs[s] = x[q];
    ys[s] = y[q];
    zs[s] = z[q];
}

__device__ __forceinline__ void na_add_weights(int q, int n, double dxi,
                                               const double* __restrict__ x,
                                               const double* __restrict__ y,
                                               const double* __restrict__ z, double s[8])
{
    double fx, fy, fz;
    na_key1(x[q], dxi, n, &fx);
    na_key1(y[q], dxi, n, &fy);
    na_key1(z[q], dxi, n, &fz);
    const double sx[2] = {1.0 - fx, fx};
    const double sy[2] = {1.0 - fy, fy};
    const double sz[2] = {1.0 - fz, fz};
#pragma unroll
    for (int cz = 0; cz < 2; ++cz)
#pragma unroll
        for (int cy = 0; cy < 2; ++cy)
#pragma unroll
            for (int cx = 0; cx < 2; ++cx)
                s[cx + 2 * cy + 4 * cz] = s[cx + 2 * cy + 4 * cz] + (sx[cx] * sy[cy]) * sz[cz];
}

// ---------------------------------------------------------------------------
// The whole counting sort by one cluster of 16 CTAs: counts to zero, keys, exclusive
// scan, scatter, segments back in particle order, a cluster barrier between two steps.
// As launches the steps were ten kernels of 2 to 4 us each (their own time and the host's)
// for a few microseconds of work.  The particles are not permuted: the deposit reads them
// through perm.  Same keys, counts and order as the kernels above.
// ---------------------------------------------------------------------------
constexpr int kNaSeg = 512;   // longer segments are ranked by a block

// Corner sums of the keys longer than a warp, a warp each: lane l sums particles l, l + 32,
// ... and an xor butterfly adds the lanes, as nyxpm_deposit sums them.  Key K's sums go to
// heavy[8 slot], slot = count[K] (the counts are zero after the scatter).  perm null: the
// particles are in sorted order.
__device__ __forceinline__ void na_heavy_keys(int warp, int warps, int n, double dxi, const double* x, const double* y,
                                              const double* z, const int* perm, const int* start,
                                              const int* long_list, int longs, int* count, double* heavy)
{
    const int lane = threadIdx.x & 31;
    for (int li = warp; li < longs; li += warps) {
        const int K = long_list[li], e = start[K + 1];
        double s[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        for (int q = start[K] + lane; q < e; q += 32) na_add_weights(perm ? perm[q] : q, n, dxi, x, y, z, s);
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1)
#pragma unroll
            for (int c = 0; c < 8; ++c) s[c] = s[c] + __shfl_xor_sync(0xffffffffu, s[c], off);
        if (lane == 0) {
#pragma unroll
            for (int c = 0; c < 8; ++c) heavy[8 * li + c] = s[c];
            count[K] = li;
        }
    }
}

__global__ void __launch_bounds__(256) na_heavy(int n, double dxi, const double* x, const double* y, const double* z,
                                                const int* start, const int* long_list, const int* long_count,
                                                int* count, double* heavy)
{
    na_heavy_keys((blockIdx.x * 256 + threadIdx.x) >> 5, gridDim.x * 8, n, dxi, x, y, z, nullptr, start, long_list,
                  *long_count, count, heavy);
}

// segment s .. s + len of perm into ascending order, by the calling group of `width`
// threads, t the thread's number in it; tmp: scratch of the same extent
__device__ __forceinline__ void na_rank(const int* perm, int* tmp, int s, int len, int t, int width)
{
    for (int i = t; i < len; i += width) {
        const int v = perm[s + i];
        int rank = 0;
        for (int u = 0; u < len; ++u) rank += perm[s + u] < v;
        tmp[s + rank] = v;
    }
}

__global__ void __launch_bounds__(kNaThreads, 1) na_sort(int np, int n, double dxi, const double* __restrict__ x,
                                                         const double* __restrict__ y, const double* __restrict__ z,
                                                         int* key, int* count, int* start, int* perm, int* long_list,
                                                         int* long_count, int* bad)
{
    __shared__ int part[kClCtas];
    const int rank = cl_rank(), lane = threadIdx.x & 31;
    const int nc = n * n * n, gt = rank * kNaThreads + threadIdx.x;
    constexpr int kAll = kClCtas * kNaThreads;
    for (int c = gt; c < nc; c += kAll) count[c] = 0;
    if (gt == 0) *long_count = 0;
    if (gt == 1) *bad = 0;
    cl_barrier();
    for (int q = gt; q < np; q += kAll) {
        const double px = x[q], py = y[q], pz = z[q];
        if (!(isfinite(px) && isfinite(py) && isfinite(pz))) atomicAdd(bad, 1);
        double f;
        const int K = (int)cidx(na_key1(px, dxi, n, &f), na_key1(py, dxi, n, &f), na_key1(pz, dxi, n, &f), n);
        key[q] = K;
        atomicAdd(count + K, 1);
    }
    cl_barrier();
    // scan: each thread a run of consecutive cells, each CTA a slice
    const int ipt = (nc + kAll - 1) / kAll, c0 = gt * ipt;
    int sum = 0;
    for (int i = 0; i < ipt; ++i)
        if (c0 + i < nc) sum += count[c0 + i];
    int total;
    int run = na_block_scan(sum, &total);
    if (threadIdx.x < kClCtas) *cl_map(&part[rank], (int)threadIdx.x) = total;
    cl_barrier();
    for (int c = 0; c < rank; ++c) run += part[c];
    for (int i = 0; i < ipt; ++i)
        if (c0 + i < nc) {
            start[c0 + i] = run;
            run += count[c0 + i];
        }
    if (gt == 0) start[nc] = np;
    cl_barrier();
    for (int q = gt; q < np; q += kAll) {
        const int K = key[q];
        perm[start[K] + atomicSub(count + K, 1) - 1] = q;
    }
    cl_barrier();
    for (int K = gt; K < nc; K += kAll) {
        const int s = start[K], len = start[K + 1] - s;
        if (len > 32) long_list[atomicAdd(long_count, 1)] = K;
        else if (len > 1) sort_short_segment(perm, s, len);
    }
    cl_barrier();
    const int longs = *(volatile int*)long_count;
    for (int li = gt >> 5; li < longs; li += kAll >> 5) {
        const int s = start[long_list[li]], len = start[long_list[li] + 1] - s;
        if (len > kNaSeg) continue;
        na_rank(perm, key, s, len, lane, 32);
        __syncwarp();
        for (int i = lane; i < len; i += 32) perm[s + i] = key[s + i];
    }
    for (int li = rank; li < longs; li += kClCtas) {
        const int s = start[long_list[li]], len = start[long_list[li] + 1] - s;
        if (len <= kNaSeg) continue;
        __syncthreads();
        na_rank(perm, key, s, len, threadIdx.x, kNaThreads);
        __syncthreads();
        for (int i = threadIdx.x; i < len; i += kNaThreads) perm[s + i] = key[s + i];
    }
    cl_barrier();
    // the ranks' scratch (key) takes the long keys' sums
    na_heavy_keys(gt >> 5, kAll >> 5, n, dxi, x, y, z, perm, start, long_list, longs, count,
                  reinterpret_cast<double*>(key));
}

// Tiles of 8 x 8 x 4 cells, one block each: the eight corner sums of every key of the
// tile's 9 x 9 x 5 window (a long key's from na_heavy_keys), then the cells.  The weights
// are bound by the FP64 pipe, which one thread with a key of 32 particles keeps waiting
// 35 us; so a warp takes 32 keys, numbers their particles densely over its lanes, one lane
// computes one particle's weights into shared memory, and eight lanes per key, one per
// corner, add them in sorted order (k_deposit_keys does the same).  Four planes, not
// eight: 32^3 would be 64 tiles for 152 SMs.  The particles are perm's (null: in place).
constexpr int kTx = 8, kTy = 8, kTz = 4;
constexpr int kKx = kTx + 1, kKy = kTy + 1, kKz = kTz + 1;
constexpr int kNKeys = kKx * kKy * kKz;
constexpr int kDepWarps = 8;

__global__ void __launch_bounds__(32 * kDepWarps) na_deposit(int n, double dxi, double scale,
                                                             const double* __restrict__ x,
                                                             const double* __restrict__ y,
                                                             const double* __restrict__ z,
                                                             const int* __restrict__ perm,
                                                             const int* __restrict__ start,
                                                             const int* __restrict__ slot,
                                                             const double* __restrict__ heavy, double* rho)
{
    __shared__ double part[kNKeys * 8];
    __shared__ double wbuf[kDepWarps][32][8];
    pdl_wait();
    pdl_trigger();
    constexpr unsigned full = 0xffffffffu;
    const int i0 = blockIdx.x * kTx, j0 = blockIdx.y * kTy, k0 = blockIdx.z * kTz;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, corner = lane & 7;
    for (int kl0 = 32 * wid; kl0 < kNKeys; kl0 += 32 * kDepWarps) {
        const int kl = kl0 + lane;
        int b0 = 0, cnt = 0;
        if (kl < kNKeys) {
            const int ki = kl % kKx, kj = (kl / kKx) % kKy, kk = kl / (kKx * kKy);
            const int K = (int)cidx(wrapi(i0 + ki, n), wrapi(j0 + kj, n), wrapi(k0 + kk, n), n);
            b0 = start[K];
            cnt = start[K + 1] - b0;
            const bool longer = cnt > kDepositLanes;
            const double* h = heavy + 8LL * (longer ? slot[K] : 0);
#pragma unroll
            for (int c = 0; c < 8; ++c) part[kl * 8 + c] = longer ? h[c] : 0.0;
            if (longer) cnt = 0;
        }
        const int incl = na_warp_scan(cnt), excl = incl - cnt;
        const int total = __shfl_sync(full, incl, 31);
        __syncwarp();
        for (int base = 0; base < total; base += 32) {
            // the lane whose key holds particle number q: the first whose inclusive count exceeds q
            const int q = base + lane;
            int o = 0;
#pragma unroll
            for (int bit = 16; bit >= 1; bit >>= 1) {
                const int v = __shfl_sync(full, incl, o + bit - 1);
                if (v <= q) o += bit;
            }
            const int ob0 = __shfl_sync(full, b0, o & 31), oex = __shfl_sync(full, excl, o & 31);
            if (q < total) {
                const int s = ob0 + (q - oex), p = perm ? perm[s] : s;
                double fx, fy, fz;
                na_key1(x[p], dxi, n, &fx);
                na_key1(y[p], dxi, n, &fy);
                na_key1(z[p], dxi, n, &fz);
                const double sx[2] = {1.0 - fx, fx};
                const double sy[2] = {1.0 - fy, fy};
                const double sz[2] = {1.0 - fz, fz};
#pragma unroll
                for (int c = 0; c < 8; ++c) wbuf[wid][lane][c] = (sx[c & 1] * sy[(c >> 1) & 1]) * sz[c >> 2];
            }
            __syncwarp();
            // eight rounds of four keys x eight corners
#pragma unroll 1
            for (int r = 0; r < 8; ++r) {
                const int ow = 4 * r + (lane >> 3);
                const int oi = __shfl_sync(full, incl, ow), oe = __shfl_sync(full, excl, ow);
                const int lo = max(oe, base) - base, hi = min(oi, base + 32) - base;
                if (lo < hi) {
                    double a = part[(kl0 + ow) * 8 + corner];
                    for (int t = lo; t < hi; ++t) a = a + wbuf[wid][t][corner];
                    part[(kl0 + ow) * 8 + corner] = a;
                }
            }
            __syncwarp();
        }
    }
    __syncthreads();
    const int cl = threadIdx.x;   // one cell per thread
    const int ci = cl % kTx, cj = (cl / kTx) % kTy, ck = cl / (kTx * kTy);
    const int i = i0 + ci, j = j0 + cj, k = k0 + ck;
    if (i >= n || j >= n || k >= n) return;
    double acc = 0.0;
#pragma unroll
    for (int dk = 0; dk < 2; ++dk)
#pragma unroll
        for (int dj = 0; dj < 2; ++dj)
#pragma unroll
            for (int di = 0; di < 2; ++di) {
                const int kl = (ci + di) + kKx * ((cj + dj) + kKy * (ck + dk));
                acc = acc + part[kl * 8 + (1 - di) + 2 * (1 - dj) + 4 * (1 - dk)];
            }
    rho[cidx(i, j, k, n)] = acc * scale;
}

// the count of non-finite positions above a flag, one store (nothing else to order:
// the deposit's kernels have completed)
__global__ void na_post(const int* __restrict__ bad, unsigned long long* host)
{
    pdl_wait();
    *reinterpret_cast<volatile unsigned long long*>(host) = (unsigned long long)(unsigned)*bad << 32 | 1;
}

static_assert(kTx * kTy * kTz == 32 * kDepWarps, "one cell per thread");

}  // namespace

}  // namespace nyxpm

using namespace nyxpm;

extern "C" nyxpm_status nyxpm_deposit_noalloc(const double* d_x, const double* d_y, const double* d_z,
                                              int64_t np, double mass, int n, double L, double* d_rho,
                                              void* stream, char* errbuf, size_t errlen)
{
    if (errbuf && errlen) errbuf[0] = '\0';
    auto fail = [&](nyxpm_status st, const char* msg) {
        if (errbuf && errlen) std::snprintf(errbuf, errlen, "%s", msg);
        return st;
    };
    if (!d_x || !d_y || !d_z || !d_rho) return fail(NYXPM_INVALID_ARG, "null device pointer");
    if (n < 1 || n > kNaMaxN)
        return fail(NYXPM_INVALID_ARG, "grid edge n must be in [1, 64] (the no-allocation scratch limit)");
    if (np < 1 || np > kNaMaxParticles)
        return fail(NYXPM_INVALID_ARG,
                    "particle count must be in [1, 262144] (the no-allocation scratch limit)");
    if (!(L > 0) || !std::isfinite(L)) return fail(NYXPM_INVALID_ARG, "box length must be positive");
    if (!(mass >= 0) || !std::isfinite(mass)) return fail(NYXPM_INVALID_ARG, "mass must be finite, >= 0");
    unsigned char* base = nullptr;
    int sm_count = 1;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    bool cluster = false, capturing = false;
    const nyxpm_status st = scratch_address(s, &base, &sm_count, &cluster, &capturing, errbuf, errlen);
    if (st != NYXPM_OK) return st;
    int* count = reinterpret_cast<int*>(base + kOffCount);
    int* start = reinterpret_cast<int*>(base + kOffStart);
    int* tiles = reinterpret_cast<int*>(base + kOffTiles);
    int* long_count = reinterpret_cast<int*>(base + kOffLongCount);
    int* bad = long_count + 1;   // non-finite positions seen
    int* long_list = reinterpret_cast<int*>(base + kOffLongList);
    int* key = reinterpret_cast<int*>(base + kOffKey);
    int* perm = reinterpret_cast<int*>(base + kOffPerm);
    double* xs = reinterpret_cast<double*>(base + kOffX);
    double* ys = reinterpret_cast<double*>(base + kOffY);
    double* zs = reinterpret_cast<double*>(base + kOffZ);
    const int nc = n * n * n;
    const double dxi = (double)n / L;
    const double dx = L / n;
    const double scale = mass * (1.0 / (dx * dx * dx));
    const unsigned pb = (unsigned)((np + 255) / 256);
    const unsigned cb = (unsigned)((nc + 255) / 256);
    const dim3 grid((n + kTx - 1) / kTx, (n + kTy - 1) / kTy, (n + kTz - 1) / kTz);
    cudaError_t e = cudaSuccess;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[1];
    bool sorted = false;
    if (cluster && np <= kNaClusterMax && nc <= kNaClusterMax) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = kClCtas;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(kClCtas);
        cfg.blockDim = dim3(kNaThreads);
        cfg.stream = s;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        sorted = cudaLaunchKernelEx(&cfg, na_sort, (int)np, n, dxi, d_x, d_y, d_z, key, count, start, perm, long_list,
                                    long_count, bad) == cudaSuccess;
        if (!sorted) cudaGetLastError();   // this stream cannot place it (an SM partition, say): by launches
    }
    if (sorted) {
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.gridDim = grid;
        cfg.blockDim = dim3(256);
        e = cudaLaunchKernelEx(&cfg, na_deposit, n, dxi, scale, d_x, d_y, d_z, (const int*)perm, (const int*)start,
                               (const int*)count, (const double*)key, d_rho);
    } else {
        const int ntiles = (nc + kNaScanTile - 1) / kNaScanTile;
        // the counts, the long-segment counter and the non-finite count must start at
        // zero: the array keeps whatever the previous call (or an interrupted one) left
        na_zero<<<cb, 256, 0, s>>>(count, nc);
        na_zero<<<1, 32, 0, s>>>(long_count, 2);
        na_keys<<<pb, 256, 0, s>>>(np, n, dxi, d_x, d_y, d_z, key, count, bad);
        na_scan_reduce<<<ntiles, kNaScanT, 0, s>>>(count, nc, tiles);
        na_scan_top<<<1, 1024, 0, s>>>(tiles, ntiles);
        na_scan_down<<<ntiles, kNaScanT, 0, s>>>(count, nc, tiles, start);
        na_scatter<<<pb, 256, 0, s>>>(np, key, start, count, perm);
        na_fix_short<<<cb, 256, 0, s>>>(nc, start, perm, long_list, long_count);
        na_fix_long<<<2 * sm_count, 512, 0, s>>>(start, long_list, long_count, perm, key);
        na_gather<<<pb, 256, 0, s>>>(np, perm, d_x, d_y, d_z, xs, ys, zs);
        na_heavy<<<4 * sm_count, 256, 0, s>>>(n, dxi, xs, ys, zs, start, long_list, long_count, count, (double*)key);
        na_deposit<<<grid, 256, 0, s>>>(n, dxi, scale, xs, ys, zs, nullptr, start, count, (const double*)key, d_rho);
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    else cudaGetLastError();
    if (e != cudaSuccess) {
        if (errbuf && errlen) std::snprintf(errbuf, errlen, "kernel launch failed: %s", cudaGetErrorString(e));
        return NYXPM_CUDA_ERROR;
    }
    // refuse non-finite positions as nyxpm_deposit does: read the count back
    // (into a host variable, no allocation), which waits for the stream.  A
    // stream under capture cannot be waited for: the graph holds the deposit
    // alone, and the check is the caller's (every replay's positions finite).
    if (capturing) return NYXPM_OK;
    // Where the device can write the caller's stack, one kernel writes the count there and
    // the host polls for it (32^3: the call 61 -> 48 us against the copy and the wait); some
    // microseconds only, where the application wants waits that give the CPU away.
    int h_bad = 0, dev = 0, pageable = 0;
    cudaError_t es = cudaGetDevice(&dev);
    if (es == cudaSuccess) es = cudaDeviceGetAttribute(&pageable, cudaDevAttrPageableMemoryAccess, dev);
    if (es == cudaSuccess && pageable) {
        unsigned long long word = 0;
        cfg.gridDim = dim3(1);
        cfg.blockDim = dim3(1);
        cfg.stream = s;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        es = cudaLaunchKernelEx(&cfg, na_post, (const int*)bad, &word);
        if (es == cudaSuccess) {
            cudaError_t q = cudaErrorNotReady;
            int i = 1;
            while (!__atomic_load_n(&word, __ATOMIC_ACQUIRE) && q == cudaErrorNotReady) {
                if (i++ & 4095) continue;
                q = i == 4097 && waits_give_way() ? cudaStreamSynchronize(s) : cudaStreamQuery(s);
                if (q == cudaErrorNotReady) cudaGetLastError();
            }
            // a stream that ended (or failed) first: nothing writes the word any more
            if (q != cudaErrorNotReady) es = cudaStreamSynchronize(s);
            h_bad = (int)(word >> 32);
        }
    } else if (es == cudaSuccess) {
        es = cudaMemcpyAsync(&h_bad, bad, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (es == cudaSuccess) es = cudaStreamSynchronize(s);
    }
    if (es != cudaSuccess) {
        cudaGetLastError();
        if (errbuf && errlen) std::snprintf(errbuf, errlen, "deposit failed: %s", cudaGetErrorString(es));
        return NYXPM_CUDA_ERROR;
    }
    if (h_bad != 0)
        return fail(NYXPM_INVALID_ARG, "non-finite particle position (rho holds no valid density)");
    return NYXPM_OK;
}
