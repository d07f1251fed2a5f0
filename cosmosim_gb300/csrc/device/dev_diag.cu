// dev_diag.cu — FP64 diagnostics and pipe-peak probes.
//
// Direct-sum accelerations of a body sample over all bodies of its system (the formula of
// the reference's test helper, tests/test_physics.c:54-71) and the total
// energy KE + softened PE (tests/test_physics.c:34-52), both in FP64. The
// j range is split over blocks; each block writes its partial sums and a
// second kernel adds them in a fixed order, so results are deterministic.
//
// The probes time long independent FMA chains (8 per thread) and report the
// FP32 and FP64 CUDA-core throughput of this GPU: the denominators for the
// walk kernels, which are bound by those pipes, not by tensor cores or HBM.
#include "dev_fixpair.cuh"
#include "dev_fpint.cuh"
#include "dev_internal.cuh"

namespace {

constexpr int DT = 256;       // threads per block
constexpr int JCHUNKS = 64;   // j-range splits for the direct sum
constexpr int FT = 128;       // threads per block of the energy

// Direct sum of sample idx[k] over bodies of its system, chunk blockIdx.y of `chunks`
// of the bodies: the reference's expression in FP64 throughout, its square root and
// its division correctly rounded on the integer pipes (dev_fpint.cuh), so with the
// compiler's operators' bits. It shares nothing with the walks' pair terms, which it
// checks. Bound by the FP64 pipe: 12 operations a pair (28 with the compiler's
// operators; 4096 of 100k bodies: 9.3 ms against 20.0, the pipe 87% busy).
__global__ void __launch_bounds__(DT) k_direct(const double *__restrict__ x,
                                               const double *__restrict__ y,
                                               const double *__restrict__ z,
                                               const double *__restrict__ m,
                                               const int *__restrict__ gid, int n,
                                               const int *__restrict__ idx, int ns, double G,
                                               double eps2, int chunks,
                                               double *__restrict__ part)
{
    __shared__ double sx[DT], sy[DT], sz[DT], sgm[DT];
    __shared__ int sg[DT];
    const int k = blockIdx.x * DT + threadIdx.x;
    const int chunk = blockIdx.y;
    const int per = (n + chunks - 1) / chunks;
    const int j0 = chunk * per, j1 = min(n, j0 + per);
    // A sample index outside [0, n) reads nothing: its row becomes NaN.
    const int i = (k < ns) ? idx[k] : -1;
    const bool valid = (unsigned)i < (unsigned)n;
    const double xi = valid ? x[i] : 0.0, yi = valid ? y[i] : 0.0, zi = valid ? z[i] : 0.0;
    const int gi = (valid && gid) ? gid[i] : 0; // only bodies of the same system attract
    double ax = 0.0, ay = 0.0, az = 0.0;
    for (int t = j0; t < j1; t += DT) {
        const int j = t + threadIdx.x;
        __syncthreads();
        if (j < j1) {
            sx[threadIdx.x] = x[j];
            sy[threadIdx.x] = y[j];
            sz[threadIdx.x] = z[j];
            sgm[threadIdx.x] = G * ((m[j] <= 0.0) ? 0.0 : m[j]);
            sg[threadIdx.x] = gid ? gid[j] : 0;
        }
        __syncthreads();
        const int cnt = min(DT, j1 - t);
        if (valid) {
            for (int q = 0; q < cnt; q++) {
                if (t + q == i || sg[q] != gi)
                    continue;
                double dx = sx[q] - xi, dy = sy[q] - yi, dz = sz[q] - zi;
                double r2 = dx * dx + dy * dy + dz * dz + eps2;
                double inv = div_rn(1.0, r2 * sqrt_rn(r2));
                double f = sgm[q] * inv;
                ax += f * dx;
                ay += f * dy;
                az += f * dz;
            }
        }
    }
    if (k < ns) {
        if (!valid)
            ax = ay = az = __longlong_as_double(0x7ff8000000000000ll);
        double *p = part + ((size_t)chunk * ns + k) * 3;
        p[0] = ax;
        p[1] = ay;
        p[2] = az;
    }
}

__global__ void k_direct_sum(const double *__restrict__ part, int chunks, int ns,
                             double *__restrict__ out)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= ns)
        return;
    double a[3] = {0.0, 0.0, 0.0};
    for (int c = 0; c < chunks; c++)
        for (int d = 0; d < 3; d++)
            a[d] += part[((size_t)c * ns + k) * 3 + d];
    for (int d = 0; d < 3; d++)
        out[3 * (size_t)k + d] = a[d];
}

// Potential energy: rows of 2 FT bodies (two a thread) against a chunk of `per`
// columns j > i. Differences and sums in FP64, 1/r by integers (pair_inv_r): 4 FP64
// operations a pair, 256 cycles a warp and scheduler, beside about 150 on
// the other pipes: 38.3 ms at 100k bodies, the FP64 pipe 87% busy. With the whole 1/r in FP64 (14 operations,
// and rows not split) 196 ms; with positions and sums in fixed point 28.3 ms, but the
// bits of close pairs near the origin lost to the grid. The block's sum of m_i m_j / r goes to part[c gridDim.x + b] (0 for
// a chunk wholly at or before the rows). The columns are split so that the long
// rows of the first bodies do not keep a few SMs busy at the end.
constexpr int PT_ROWS = 2 * FT;

template <bool MULTI>
__global__ void __launch_bounds__(FT, 6) k_potential(const double *__restrict__ x,
                                                  const double *__restrict__ y,
                                                  const double *__restrict__ z,
                                                  const double *__restrict__ m,
                                                  const int *__restrict__ gid, int n, int per,
                                                  PairEps eps, double *__restrict__ part)
{
    __shared__ double tx[FT], ty[FT], tz[FT], tm[FT];
    __shared__ int tg[FT];
    const int row0 = blockIdx.x * PT_ROWS, j0 = blockIdx.y * per, j1 = min(n, j0 + per);
    const int ia = row0 + threadIdx.x, ib = ia + FT;
    const double xa = ia < n ? x[ia] : 0.0, ya = ia < n ? y[ia] : 0.0, za = ia < n ? z[ia] : 0.0;
    const double xb = ib < n ? x[ib] : 0.0, yb = ib < n ? y[ib] : 0.0, zb = ib < n ? z[ib] : 0.0;
    const int ga = (MULTI && ia < n) ? gid[ia] : 0, gb = (MULTI && ib < n) ? gid[ib] : 0;
    double sa = 0.0, sb = 0.0;
    for (int t = max(j0, row0); t < j1; t += FT) {
        const int j = t + threadIdx.x;
        __syncthreads();
        if (j < j1) {
            tx[threadIdx.x] = x[j];
            ty[threadIdx.x] = y[j];
            tz[threadIdx.x] = z[j];
            tm[threadIdx.x] = (m[j] > 0.0) ? m[j] : 0.0;
            if (MULTI)
                tg[threadIdx.x] = gid[j];
        }
        __syncthreads();
        const int cnt = min(FT, j1 - t);
        for (int q = 0; q < cnt; q++) {
            const bool ta = t + q > ia && (!MULTI || tg[q] == ga),
                       tb = t + q > ib && (!MULTI || tg[q] == gb);
            const double va = pair_inv_r(eps, tx[q] - xa, ty[q] - ya, tz[q] - za);
            const double vb = pair_inv_r(eps, tx[q] - xb, ty[q] - yb, tz[q] - zb);
            sa = fma(tm[q], ta ? va : 0.0, sa);
            sb = fma(tm[q], tb ? vb : 0.0, sb);
        }
    }
    // the block's rows, added in a fixed order
    __syncthreads();
    const double ma = (ia < n && m[ia] > 0.0) ? m[ia] : 0.0, mb = (ib < n && m[ib] > 0.0) ? m[ib] : 0.0;
    tx[threadIdx.x] = ma * sa + mb * sb;
    __syncthreads();
    for (int s = FT / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s)
            tx[threadIdx.x] += tx[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        part[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = tx[0];
}

__global__ void k_energy_reduce(const double *__restrict__ part, int parts, double G,
                                const double *__restrict__ m, const double *__restrict__ vx,
                                const double *__restrict__ vy, const double *__restrict__ vz, int n,
                                double *__restrict__ out)
{
    // one block; fixed-order tree reduction in shared memory
    __shared__ double ske[1024], spe[1024];
    double ke = 0.0, pe = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        double mm = (m[i] > 0.0) ? m[i] : 0.0;
        ke += 0.5 * mm * (vx[i] * vx[i] + vy[i] * vy[i] + vz[i] * vz[i]);
    }
    for (int i = threadIdx.x; i < parts; i += blockDim.x)
        pe += part[i];
    ske[threadIdx.x] = ke;
    spe[threadIdx.x] = pe;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            ske[threadIdx.x] += ske[threadIdx.x + s];
            spe[threadIdx.x] += spe[threadIdx.x + s];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[0] = ske[0];
        out[1] = -G * spe[0];
    }
}

template <typename T>
__global__ void k_fma_probe(T *out, int iters, T a, T b)
{
    T x0 = (T)threadIdx.x * (T)1e-3, x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3;
    T x4 = x0 + 4, x5 = x0 + 5, x6 = x0 + 6, x7 = x0 + 7;
    for (int i = 0; i < iters; i++) {
        x0 = x0 * a + b;
        x1 = x1 * a + b;
        x2 = x2 * a + b;
        x3 = x3 * a + b;
        x4 = x4 * a + b;
        x5 = x5 * a + b;
        x6 = x6 * a + b;
        x7 = x7 * a + b;
    }
    out[blockIdx.x * blockDim.x + threadIdx.x] = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
}

} // namespace

extern "C" int csgd_direct_forces(csgd_t *d, const int *host_idx, int ns, double G,
                                  double softening, double *host_out)
{
    if (ns <= 0)
        return CSG_OK;
    if (ns > d->n || !host_idx)
        return CSG_ERR_BAD_ARG;
    for (int k = 0; k < ns; k++)
        if (host_idx[k] < 0 || host_idx[k] >= d->n)
            return CSG_ERR_BAD_ARG;
    // one allocation: partial sums, result, sample
    const size_t doubles = 3 * (size_t)ns * (JCHUNKS + 1);
    double *part = nullptr;
    if (csgd_malloc((void **)&part, sizeof(double) * doubles + sizeof(int) * (size_t)ns) !=
        cudaSuccess) {
        cudaGetLastError();
        return CSG_ERR_NOMEM;
    }
    double *out = part + 3 * (size_t)ns * JCHUNKS;
    int *didx = (int *)(part + doubles);
    cudaStream_t s = d->stream;
    cudaMemcpyAsync(didx, host_idx, sizeof(int) * (size_t)ns, cudaMemcpyHostToDevice, s);
    const dim3 grid((ns + DT - 1) / DT, JCHUNKS);
    { k_direct<<<grid, DT, 0, s>>>(d->x, d->y, d->z, d->m, d->gid, d->n, didx, ns, G, softening * softening, JCHUNKS, part); d->launches++; }
    { k_direct_sum<<<csgd_grid(ns, 256), 256, 0, s>>>(part, JCHUNKS, ns, out); d->launches++; }
    cudaMemcpyAsync(host_out, out, sizeof(double) * 3 * (size_t)ns, cudaMemcpyDeviceToHost, s);
    const int rc = csgd_sync(d);
    cudaFree(part);
    return rc;
}

extern "C" int csgd_energy(csgd_t *d, double G, double softening, double *ke, double *pe)
{
    const int n = d->n;
    if (n <= 0) {
        *ke = *pe = 0.0;
        return CSG_OK;
    }
    // columns a chunk: at least 2048, at most 32 chunks (their partial sums)
    const int per = n / 32 > 2048 ? (n + 31) / 32 : 2048;
    const int chunks = (n + per - 1) / per;
    const dim3 grid((n + PT_ROWS - 1) / PT_ROWS, chunks);
    const int parts = (int)grid.x * chunks;
    double *part = nullptr;
    if (csgd_malloc((void **)&part, sizeof(double) * ((size_t)parts + 2)) != cudaSuccess) {
        cudaGetLastError();
        return CSG_ERR_NOMEM;
    }
    double *out = part + parts;
    cudaStream_t s = d->stream;
    const PairEps eps = pair_eps(softening);
    if (d->n_gal > 1)
        k_potential<true><<<grid, FT, 0, s>>>(d->x, d->y, d->z, d->m, d->gid, n, per, eps, part);
    else
        k_potential<false><<<grid, FT, 0, s>>>(d->x, d->y, d->z, d->m, d->gid, n, per, eps, part);
    d->launches++;
    { k_energy_reduce<<<1, 1024, 0, s>>>(part, parts, G, d->m, d->vx, d->vy, d->vz, n, out); d->launches++; }
    double h[2] = {0.0, 0.0};
    cudaMemcpyAsync(h, out, sizeof(h), cudaMemcpyDeviceToHost, s);
    const int rc = csgd_sync(d);
    *ke = h[0];
    *pe = h[1];
    cudaFree(part);
    return rc;
}

// FP32 and FP64 FMA throughput (TFLOP/s, 2 flop per FMA) of the current device.
extern "C" CSG_EXPORT int csg_measure_fp_peaks(double *fp32_tflops, double *fp64_tflops)
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        return CSG_ERR_NO_DEVICE;
    }
    const int blocks = sms * 8, threads = 256;
    const size_t nthr = (size_t)blocks * threads;
    float *o32 = nullptr;
    double *o64 = nullptr;
    cudaStream_t s;
    if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess)
        return CSG_ERR_CUDA;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    int rc = CSG_OK;
    if (csgd_malloc((void **)&o32, nthr * sizeof(float)) != cudaSuccess ||
        csgd_malloc((void **)&o64, nthr * sizeof(double)) != cudaSuccess) {
        rc = CSG_ERR_NOMEM;
    } else {
        const int it32 = 8192, it64 = 512;
        float best32 = 1e30f, best64 = 1e30f, ms = 0.f;
        for (int rep = 0; rep < 3; rep++) {
            cudaEventRecord(e0, s);
            k_fma_probe<float><<<blocks, threads, 0, s>>>(o32, it32, 0.999999f, 1e-7f);
            cudaEventRecord(e1, s);
            cudaEventSynchronize(e1);
            cudaEventElapsedTime(&ms, e0, e1);
            best32 = ms < best32 ? ms : best32;
            cudaEventRecord(e0, s);
            k_fma_probe<double><<<blocks, threads, 0, s>>>(o64, it64, 0.999999, 1e-7);
            cudaEventRecord(e1, s);
            cudaEventSynchronize(e1);
            cudaEventElapsedTime(&ms, e0, e1);
            best64 = ms < best64 ? ms : best64;
        }
        *fp32_tflops = 2.0 * 8.0 * it32 * (double)nthr / (best32 * 1e-3) / 1e12;
        *fp64_tflops = 2.0 * 8.0 * it64 * (double)nthr / (best64 * 1e-3) / 1e12;
        if (cudaGetLastError() != cudaSuccess)
            rc = CSG_ERR_CUDA;
    }
    cudaFree(o32);
    cudaFree(o64);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaStreamDestroy(s);
    return rc;
}

// ---- direct sum without allocation -----------------------------------------
//
// Callers that cannot allocate device memory — code inside an engine or
// renderer that owns a fixed GPU budget and its own allocator, a real-time
// thread that must not block on cudaMalloc/cudaFree (both can synchronise the
// device) — can still run the FP64 direct-sum check on buffers they already
// hold. Its scratch (per-chunk partial sums) lives in the file-scope array
// below instead of cudaMalloc'd memory: 16 chunks x 4096 bodies x 3 doubles =
// 1.5 MiB, held by every GPU that loads the library until the process exits.
// All calls share that array, so calls that overlap on the GPU race; every
// call overwrites each partial it later reads, so nothing needs clearing.

constexpr int NOALLOC_CHUNKS = 16;
constexpr int NOALLOC_MAX_SAMPLE = 4096;
constexpr int NOALLOC_MAX_DEVICES = 64;

static __device__ __align__(256) double g_noalloc_partials[NOALLOC_CHUNKS * NOALLOC_MAX_SAMPLE * 3];

#include <mutex>

namespace {

std::mutex g_noalloc_mutex;
double *g_noalloc_ptr[NOALLOC_MAX_DEVICES];

} // namespace

// The device address of the scratch array on the current device, looked up
// once per device (the first call on a device does it, so that call should
// come before any stream capture on that device). The address belongs to the
// device's primary context: after a cudaDeviceReset the cached address is
// stale, so a process that resets a device must not call the entry point on
// it again.
static int noalloc_scratch(double **ptr)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) {
        cudaGetLastError();
        return CSG_ERR_NO_DEVICE;
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_noalloc_partials) != cudaSuccess || !p) {
            cudaGetLastError();
            return CSG_ERR_CUDA;
        }
        g_noalloc_ptr[dev] = (double *)p;
    }
    *ptr = g_noalloc_ptr[dev];
    return CSG_OK;
}

extern "C" CSG_EXPORT int csg_direct_forces_noalloc(const double *x, const double *y,
                                                    const double *z, const double *mass,
                                                    const int *sys, int n, const int *idx, int m,
                                                    double G, double softening, double *out,
                                                    void *stream)
{
    if (n < 0 || m < 0 || m > NOALLOC_MAX_SAMPLE)
        return CSG_ERR_BAD_ARG;
    if (m == 0)
        return CSG_OK;
    if (!x || !y || !z || !mass || !idx || !out || n == 0)
        return CSG_ERR_BAD_ARG;
    double *part = nullptr;
    int rc = noalloc_scratch(&part);
    if (rc)
        return rc;
    cudaStream_t s = (cudaStream_t)stream;
    const dim3 grid((m + DT - 1) / DT, NOALLOC_CHUNKS);
    k_direct<<<grid, DT, 0, s>>>(x, y, z, mass, sys, n, idx, m, G, softening * softening, NOALLOC_CHUNKS, part);
    k_direct_sum<<<(m + 255) / 256, 256, 0, s>>>(part, NOALLOC_CHUNKS, m, out);
    if (cudaGetLastError() != cudaSuccess)
        return CSG_ERR_CUDA;
    return CSG_OK;
}

// ---- integer-pipe division and square root: self-check ----------------------
//
// div_rn and sqrt_rn (dev_fpint.cuh) against the compiler's correctly rounded
// operators, bit for bit, on n seeded operand pairs of several kinds: operands
// of moderate exponents, arbitrary bit patterns (zeros, subnormals,
// infinities, NaNs, exponents near the fast path's bounds), integer operands
// over small odd divisors (exact quotients and ties), power-of-two divisors,
// signed zeros and SPH-like distances and smoothing lengths.

namespace {

__device__ __forceinline__ unsigned long long xs_next(unsigned long long &s)
{
    s ^= s << 13;
    s ^= s >> 7;
    s ^= s << 17;
    return s;
}

__device__ __forceinline__ double rand_moderate(unsigned long long &s, int span)
{
    const unsigned long long r = xs_next(s);
    const long long e = 1023 + (long long)(r % (unsigned long long)(2 * span + 1)) - span;
    return __longlong_as_double((long long)((r & (1ull << 63)) | ((unsigned long long)e << 52) |
                                            (xs_next(s) & fpint::MANT)));
}

__global__ void k_check_div_sqrt(unsigned long long seed, long long n, unsigned long long *out)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    unsigned long long bad_div = 0, bad_sqrt = 0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        unsigned long long s = (seed ^ ((unsigned long long)i * 0x9E3779B97F4A7C15ull)) | 1ull;
        xs_next(s);
        xs_next(s);
        double a, b;
        switch ((unsigned)(xs_next(s) % 8)) {
        case 0:
        case 1:
            a = rand_moderate(s, 60);
            b = rand_moderate(s, 60);
            break;
        case 2:
            a = __longlong_as_double((long long)xs_next(s));
            b = __longlong_as_double((long long)xs_next(s));
            break;
        case 3: {
            const unsigned sh = 11 + (unsigned)(xs_next(s) % 40);
            a = (double)(long long)(xs_next(s) >> sh);
            const double odd[6] = {3.0, 5.0, 7.0, 9.0, 11.0, 1.0 + (double)(xs_next(s) & 255) * 2.0};
            b = odd[xs_next(s) % 6] * ((xs_next(s) & 1) ? 1.0 : -1.0);
            break;
        }
        case 4:
            a = rand_moderate(s, 500);
            b = __longlong_as_double((long long)((unsigned long long)(1023 + (long long)(xs_next(s) % 1001) - 500)
                                                 << 52));
            break;
        case 5:
            a = (xs_next(s) & 1) ? 0.0 : -0.0;
            b = rand_moderate(s, 1000);
            break;
        case 6: // exponents near the fast path's limits
            a = rand_moderate(s, 1022);
            b = rand_moderate(s, 1022);
            break;
        default: { // distances, smoothing lengths, densities of the SPH passes
            const double r = (double)(xs_next(s) >> 11) * 0x1p-53 * 4.0;
            const double h = 0.01 + (double)(xs_next(s) >> 11) * 0x1p-53;
            a = (xs_next(s) & 1) ? r * r : r;
            b = (xs_next(s) & 1) ? h : h * h * h * 3.141592653589793;
            break;
        }
        }
        if (__double_as_longlong(div_rn(a, b)) != __double_as_longlong(__ddiv_rn(a, b)))
            bad_div++;
        const double x = (xs_next(s) & 3) ? fabs(a) : a;
        if (__double_as_longlong(sqrt_rn(x)) != __double_as_longlong(__dsqrt_rn(x)))
            bad_sqrt++;
    }
    if (bad_div)
        atomicAdd(&out[0], bad_div);
    if (bad_sqrt)
        atomicAdd(&out[1], bad_sqrt);
}

} // namespace

extern "C" CSG_EXPORT int csg_check_div_sqrt(int64_t n, uint64_t seed, int64_t *div_mismatches,
                                             int64_t *sqrt_mismatches)
{
    if (n < 0 || !div_mismatches || !sqrt_mismatches)
        return CSG_ERR_BAD_ARG;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        return CSG_ERR_NO_DEVICE;
    }
    unsigned long long *out = nullptr;
    if (csgd_malloc((void **)&out, 2 * sizeof(unsigned long long)) != cudaSuccess) {
        cudaGetLastError();
        return CSG_ERR_NOMEM;
    }
    unsigned long long h[2] = {0, 0};
    int rc = CSG_OK;
    if (cudaMemset(out, 0, sizeof(h)) != cudaSuccess)
        rc = CSG_ERR_CUDA;
    if (!rc && n > 0) {
        k_check_div_sqrt<<<sms * 8, 256>>>((unsigned long long)seed, (long long)n, out);
        if (cudaGetLastError() != cudaSuccess)
            rc = CSG_ERR_CUDA;
    }
    if (!rc && cudaMemcpy(h, out, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess)
        rc = CSG_ERR_CUDA;
    cudaFree(out);
    *div_mismatches = (int64_t)h[0];
    *sqrt_mismatches = (int64_t)h[1];
    return rc;
}
