// psx_kernels.cu -- single-stage kernels behind the drop-in entry points
// of include/peasoup_b200.h (one launch per call, asynchronous).
//
// Layout conventions: time series are float[N]; complex spectra are
// interleaved float pairs (cufftComplex); all grids are grid-stride loops
// sized to a multiple of the SM count (psx::grid_for).
#include <cuda.h>
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <fstream>
#include <mutex>
#include <sstream>
#include <string>
#include <vector>
#include "psx_common.cuh"
#include "psx_device.cuh"
#include "psx_stages.cuh"

namespace psx {

static thread_local std::string g_err;

void set_error(const char* fmt, ...)
{
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_err = buf;
}

void clear_error() { g_err.clear(); }

cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t s)
{
    static std::mutex mu;
    static cudaMemPool_t pools[64] = {nullptr};
    static bool tried[64] = {false};
    int dev = 0;
    cudaMemPool_t pool = nullptr;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64) {
        std::lock_guard<std::mutex> lock(mu);
        if (!tried[dev]) {
            tried[dev] = true;
            cudaMemPoolProps props{};
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = dev;
            cuuint64_t keep = 64ull << 20;
            if (cudaMemPoolCreate(&pools[dev], &props) != cudaSuccess) {
                pools[dev] = nullptr;
            } else if (cudaMemPoolSetAttribute(pools[dev], cudaMemPoolAttrReleaseThreshold,
                                               &keep) != cudaSuccess) {
                cudaMemPoolDestroy(pools[dev]);
                pools[dev] = nullptr;
            }
        }
        pool = pools[dev];
    }
    if (pool && cudaMallocFromPoolAsync(p, bytes, pool, s) == cudaSuccess) return cudaSuccess;
    (void)cudaGetLastError();  // no pool (or one a device reset took): the default one
    return cudaMallocAsync(p, bytes, s);
}

int sm_count()
{
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (!cached[dev]) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
            n = 148;
        cached[dev] = n;
    }
    return cached[dev];
}

// ------------------------------------------------------------------ resample
// Each thread writes four consecutive outputs with one 128-bit store; the
// reads are a near-unit-stride gather that L1/L2 coalesce.
template <bool CENTRED>
__global__ void __launch_bounds__(256) k_resample(const float* __restrict__ in,
                                                  float* __restrict__ out,
                                                  size_t n, double k, double size,
                                                  const double* __restrict__ ktab,
                                                  size_t out_pitch)
{
    const unsigned t = blockIdx.y;
    if (ktab) k = ktab[t];
    float* o = out + (size_t)t * out_pitch;
    const size_t n4 = n / 4;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < n4; q += stride) {
        const unsigned long long i0 = 4ull * q;
        float4 v;
        if (CENTRED) {
            double s2 = size * 0.5;
            v.x = gather_at(in, resample_index(i0 + 0, k, s2), n);
            v.y = gather_at(in, resample_index(i0 + 1, k, s2), n);
            v.z = gather_at(in, resample_index(i0 + 2, k, s2), n);
            v.w = gather_at(in, resample_index(i0 + 3, k, s2), n);
        } else {
            const double id = (double)i0;  // exact (n < 2^32)
            v.x = resampleII_read(in, id, k, size, (unsigned)n);
            v.y = resampleII_read(in, id + 1.0, k, size, (unsigned)n);
            v.z = resampleII_read(in, id + 2.0, k, size, (unsigned)n);
            v.w = resampleII_read(in, id + 3.0, k, size, (unsigned)n);
        }
        reinterpret_cast<float4*>(o)[q] = v;
    }
    // tail (n not a multiple of 4)
    if (blockIdx.x == 0 && threadIdx.x < (n & 3)) {
        const unsigned long long i = 4ull * n4 + threadIdx.x;
        o[i] = CENTRED ? gather_at(in, resample_index(i, k, size * 0.5), n)
                       : resampleII_read(in, (double)i, k, size, (unsigned)n);
    }
}

double accel_fact(float acc, float tsamp)
{
    // reference src/kernels.cu:361: float product, double divide
    float at = acc * tsamp;
    return (double)at / (2 * 299792458.0);
}

int launch_resample(const float* d_in, float* d_out, size_t n, const double* d_ktab,
                    double k, int ntrials, size_t out_pitch, bool centred, cudaStream_t s)
{
    if (!d_in || !d_out || n == 0 || n >= (size_t(1) << 32) || ntrials <= 0) {
        set_error("resample: bad arguments (1 <= n < 2^32)");
        return PSX_ERR_INVALID;
    }
    const unsigned threads = 256;
    dim3 grid(grid_for((n + 3) / 4, threads, 8), (unsigned)ntrials);
    if (centred)
        k_resample<true><<<grid, threads, 0, s>>>(d_in, d_out, n, k, (double)n, d_ktab, out_pitch);
    else
        k_resample<false><<<grid, threads, 0, s>>>(d_in, d_out, n, k, (double)n, d_ktab, out_pitch);
    return launch_status("resample kernel");
}

// ------------------------------------------------------------------- forming
// way 0 amplitude, way 1 interbinned amplitude.  Each thread forms two
// bins from one 128-bit load of two complex values; bin 2q-1 comes from
// the neighbouring lane (or a cached scalar load at warp edges).
template <int WAY>
__global__ void __launch_bounds__(256) k_form(const float* __restrict__ X,
                                              float* __restrict__ out, size_t nbins)
{
    const size_t npairs = nbins / 2;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < npairs; q += stride) {
        const float4 v = reinterpret_cast<const float4*>(X)[q];
        float2 r;
        if (WAY == 0) {
            r.x = amplitude(v.x, v.y);
            r.y = amplitude(v.z, v.w);
        } else {
            float rl = 0.f, il = 0.f;
            if (q > 0) {
                rl = X[4 * q - 2];
                il = X[4 * q - 1];
            }
            r.x = interbin(v.x, v.y, rl, il);
            r.y = interbin(v.z, v.w, v.x, v.y);
        }
        reinterpret_cast<float2*>(out)[q] = r;
    }
    if ((nbins & 1) && blockIdx.x == 0 && threadIdx.x == 0) {
        const size_t k = nbins - 1;
        const float re = X[2 * k], im = X[2 * k + 1];
        if (WAY == 0) {
            out[k] = amplitude(re, im);
        } else {
            const float rl = k ? X[2 * k - 2] : 0.f, il = k ? X[2 * k - 1] : 0.f;
            out[k] = interbin(re, im, rl, il);
        }
    }
}

// -------------------------------------------------------------- dereddening
__global__ void __launch_bounds__(256) k_scrunch5(const float* __restrict__ in, size_t count,
                                                  float* __restrict__ out)
{
    if (count < 5) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            float r = 0.f;
            if (count == 1) r = in[0];
            else if (count == 2) r = 0.5f * (in[0] + in[1]);
            else if (count == 3) r = med3(in[0], in[1], in[2]);
            else if (count == 4) r = med4(in[0], in[1], in[2], in[3]);
            if (count) out[0] = r;
        }
        return;
    }
    const size_t oc = count / 5;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < oc; i += stride) {
        const float* p = in + 5 * i;
        out[i] = med5(p[0], p[1], p[2], p[3], p[4]);
    }
}

// The median spliced from its three levels (median_at); with X given the
// spectrum is divided by the median in place (bins 0..4 zeroed), otherwise the
// median itself is written.
__global__ void __launch_bounds__(256) k_median_apply(MedianLevels L, size_t nbins,
                                                      float* __restrict__ median_out,
                                                      float* __restrict__ X, size_t x_stride = 0,
                                                      size_t m_stride = 0)
{
    if (blockIdx.y) {  // row blockIdx.y of a batch (strides in floats)
        L.m5 += (size_t)blockIdx.y * m_stride;
        L.m25 += (size_t)blockIdx.y * m_stride;
        L.m125 += (size_t)blockIdx.y * m_stride;
        if (X) X += (size_t)blockIdx.y * x_stride;
    }
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < nbins; k += stride) {
        const float m = median_at(L, (unsigned)k);
        if (median_out) median_out[k] = m;
        if (X) {
            cuComplex* c = reinterpret_cast<cuComplex*>(X);
            if (k < 5)
                c[k] = make_cuComplex(0.0, 0.0);
            else
                c[k] = cuCdivf(c[k], make_cuComplex(m, 0.0));
        }
    }
}

__global__ void __launch_bounds__(256) k_divide_c_by_f(float* __restrict__ X,
                                                       const float* __restrict__ f, size_t nbins)
{
    cuComplex* c = reinterpret_cast<cuComplex*>(X);
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < nbins; k += stride) {
        if (k < 5)
            c[k] = make_cuComplex(0.0, 0.0);
        else
            c[k] = cuCdivf(c[k], make_cuComplex(f[k], 0.0));
    }
}

__global__ void __launch_bounds__(256) k_stretch(const float* __restrict__ in, unsigned in_count,
                                                 float* __restrict__ out, size_t out_count,
                                                 float step)
{
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < out_count; i += stride)
        out[i] = stretch_at(in, in_count, (unsigned)i, step);
}

size_t median_scratch_bytes(size_t nbins)
{
    auto up = [](size_t v) { return (v + 63) / 64 * 64; };
    return sizeof(float) * (up(nbins / 5 + 1) + up(nbins / 25 + 1) + up(nbins / 125 + 1));
}

static float stretch_step(size_t in_count, size_t out_count)
{
    // reference src/kernels.cu:1016: float(in_count-1)/(out_count-1)
    return (float)(in_count - 1) / (float)(out_count - 1);
}

MedianLevels median_levels(size_t nbins, double bin_width, float b5, float b25, float* scratch)
{
    auto up = [](size_t v) { return (v + 63) / 64 * 64; };
    // reference dereddener.hpp:48-49: (int)(boundary / bin_width)
    const int pos5 = (int)((double)b5 / bin_width), pos25 = (int)((double)b25 / bin_width);
    MedianLevels L;
    L.m5 = scratch;
    L.m25 = scratch + up(nbins / 5 + 1);
    L.m125 = L.m25 + up(nbins / 25 + 1);
    L.n5 = (unsigned)(nbins / 5);
    L.n25 = L.n5 / 5;
    L.n125 = L.n25 / 5;
    L.step5 = stretch_step(L.n5, nbins);
    L.step25 = stretch_step(L.n25, nbins);
    L.step125 = stretch_step(L.n125, nbins);
    L.pos5 = (unsigned)(pos5 < 0 ? 0 : (size_t)pos5 > nbins ? nbins : pos5);
    L.pos25 = (unsigned)(pos25 < 0 ? 0 : (size_t)pos25 > nbins ? nbins : pos25);
    if (L.pos25 < L.pos5) L.pos25 = L.pos5;
    return L;
}

// The three median-of-5 levels of the amplitudes of a complex spectrum X
// (AMP), or of the powers X as they are, in one pass: a CTA takes groups of
// 125 bins (5 * 25) at a time, so every value of the 5-, 25- and 125-bin levels
// it writes is formed from its own bins; the levels stop where the reference's floor(count / 5)
// stops them.  The amplitudes themselves are never written.  (One launch in
// place of three for the powers: at 2^20 bins on B200 6.4 us of three
// latency-bound kernels became 3.7.)
constexpr int kScrGroups = 16;  // 125-bin groups per CTA step

template <bool AMP>
__global__ void __launch_bounds__(256) k_scrunch3(const float* __restrict__ X,
                                                  float* __restrict__ m5, size_t n5,
                                                  float* __restrict__ m25, size_t n25,
                                                  float* __restrict__ m125, size_t n125,
                                                  size_t x_stride = 0, size_t m_stride = 0)
{
    // row blockIdx.y of a batch: its spectrum and its scratch (strides in floats)
    X += (size_t)blockIdx.y * x_stride;
    m5 += (size_t)blockIdx.y * m_stride;
    m25 += (size_t)blockIdx.y * m_stride;
    m125 += (size_t)blockIdx.y * m_stride;
    constexpr int kStep = kScrGroups * 125;  // bins of a CTA step, a multiple of 4
    __shared__ __align__(16) float buf[kStep];
    __shared__ float s5[kScrGroups * 25];
    __shared__ float s25[kScrGroups * 5];
    const bool vec = (reinterpret_cast<uintptr_t>(X) & 15u) == 0;
    const size_t ngroups = (n5 + 24) / 25;  // groups holding any 5-level value
    for (size_t g0 = (size_t)blockIdx.x * kScrGroups; g0 < ngroups;
         g0 += (size_t)gridDim.x * kScrGroups) {
        // the step's bins through shared memory (reading five neighbours per
        // thread straight from X touches every line five times)
        const size_t e0 = g0 * 125;
        const int cnt = (int)min((size_t)kStep, 5 * n5 - e0);
        int done = 0;
        if (vec) {
            if constexpr (AMP) {
                done = cnt & ~1;
                const float4* x4 = reinterpret_cast<const float4*>(X + 2 * e0);
#pragma unroll 4
                for (int i = threadIdx.x; i < cnt / 2; i += blockDim.x) {
                    const float4 z = x4[i];
                    reinterpret_cast<float2*>(buf)[i] =
                        make_float2(amplitude(z.x, z.y), amplitude(z.z, z.w));
                }
            } else {
                done = cnt & ~3;
                const float4* x4 = reinterpret_cast<const float4*>(X + e0);
#pragma unroll 2
                for (int i = threadIdx.x; i < cnt / 4; i += blockDim.x)
                    reinterpret_cast<float4*>(buf)[i] = x4[i];
            }
        }
        for (int i = done + threadIdx.x; i < cnt; i += blockDim.x)
            buf[i] = AMP ? amplitude(X[2 * (e0 + i)], X[2 * (e0 + i) + 1]) : X[e0 + i];
        __syncthreads();
        for (int i = threadIdx.x; i < kScrGroups * 25; i += blockDim.x) {
            const size_t j = g0 * 25 + i;  // 5-level index
            float v = 0.f;
            if (j < n5) {
                const float* a = buf + 5 * i;
                v = med5(a[0], a[1], a[2], a[3], a[4]);
                m5[j] = v;
            }
            s5[i] = v;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < kScrGroups * 5; i += blockDim.x) {
            const size_t j = g0 * 5 + i;
            float v = 0.f;
            if (j < n25) {
                const float* q = s5 + 5 * i;
                v = med5(q[0], q[1], q[2], q[3], q[4]);
                m25[j] = v;
            }
            s25[i] = v;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < kScrGroups; i += blockDim.x) {
            const size_t j = g0 + i;
            if (j < n125) {
                const float* q = s25 + 5 * i;
                m125[j] = med5(q[0], q[1], q[2], q[3], q[4]);
            }
        }
        __syncthreads();
    }
}

namespace {

// The stretch, splice and division of launch_running_median once the three
// levels are in the scratch.
int median_apply(size_t nbins, double bin_width, float b5, float b25, float* d_median, float* d_X,
                 float* m5, cudaStream_t s)
{
    const MedianLevels L = median_levels(nbins, bin_width, b5, b25, m5);
    k_median_apply<<<grid_for(nbins, 256), 256, 0, s>>>(L, nbins, d_median, d_X);
    return launch_status("median apply kernel");
}

}  // namespace

int launch_running_median_spectrum(float* d_X, size_t nbins, double bin_width, float b5,
                                   float b25, void* d_scratch, cudaStream_t s)
{
    if (!d_X || !d_scratch || nbins < 125 || nbins > 0xffffffffu) {
        set_error("running median: bad arguments (nbins=%zu)", nbins);
        return PSX_ERR_INVALID;
    }
    auto up = [](size_t v) { return (v + 63) / 64 * 64; };
    float* m5 = static_cast<float*>(d_scratch);
    float* m25 = m5 + up(nbins / 5 + 1);
    float* m125 = m25 + up(nbins / 25 + 1);
    const size_t n5 = nbins / 5, n25 = n5 / 5, n125 = n25 / 5;
    const size_t ngroups = (n5 + 24) / 25;
    const unsigned grid = (unsigned)std::min<size_t>((ngroups + kScrGroups - 1) / kScrGroups,
                                                     (size_t)sm_count() * 8);
    k_scrunch3<true><<<grid, 256, 0, s>>>(d_X, m5, n5, m25, n25, m125, n125);
    PSX_TRY(launch_status("amplitude + scrunch kernel"));
    return median_apply(nbins, bin_width, b5, b25, nullptr, d_X, m5, s);
}

int launch_running_median(const float* d_powers, size_t nbins, double bin_width, float b5,
                          float b25, float* d_median, float* d_X, void* d_scratch,
                          cudaStream_t s)
{
    if (!d_powers || !d_scratch || nbins < 125 || nbins > 0xffffffffu) {
        set_error("running median: bad arguments (nbins=%zu)", nbins);
        return PSX_ERR_INVALID;
    }
    auto up = [](size_t v) { return (v + 63) / 64 * 64; };
    float* m5 = static_cast<float*>(d_scratch);
    float* m25 = m5 + up(nbins / 5 + 1);
    float* m125 = m25 + up(nbins / 25 + 1);
    const size_t n5 = nbins / 5, n25 = n5 / 5, n125 = n25 / 5;
    const size_t ngroups = (n5 + 24) / 25;
    const unsigned grid = (unsigned)std::min<size_t>((ngroups + kScrGroups - 1) / kScrGroups,
                                                     (size_t)sm_count() * 8);
    k_scrunch3<false><<<grid, 256, 0, s>>>(d_powers, m5, n5, m25, n25, m125, n125);
    PSX_TRY(launch_status("scrunch kernel"));
    return median_apply(nbins, bin_width, b5, b25, d_median, d_X, m5, s);
}

// ------------------------------------------------------------------- zapping
// Bins [low, high) of a birdie (reference src/kernels.cu, zap kernel).
__device__ __forceinline__ bool zap_range(float freq, float width, float bin_width, unsigned nbins,
                                          int& low_bin, int& high_bin)
{
    low_bin = __float2int_rd((freq - width) / bin_width);
    high_bin = __float2int_ru((freq + width) / bin_width);
    if (low_bin < 0) low_bin = 0;
    if (low_bin >= (int)nbins) return false;
    if (high_bin >= (int)nbins) high_bin = (int)nbins - 1;
    return true;
}

// One warp per birdie; lanes stride the birdie's bin range.
__global__ void k_zap(float* __restrict__ X, const float* __restrict__ freqs,
                      const float* __restrict__ widths, float bin_width, unsigned nbirdies,
                      unsigned nbins, size_t x_stride = 0)
{
    X += (size_t)blockIdx.y * x_stride;  // row blockIdx.y of a batch
    const unsigned warp = (blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const unsigned lane = threadIdx.x & 31;
    if (warp >= nbirdies) return;
    int low_bin, high_bin;
    if (!zap_range(freqs[warp], widths[warp], bin_width, nbins, low_bin, high_bin)) return;
    float2* c = reinterpret_cast<float2*>(X);
    for (int k = low_bin + (int)lane; k < high_bin; k += 32) c[k] = make_float2(1.0f, 0.0f);
}

int launch_zap(float* d_X, const float* d_freqs, const float* d_widths, float bin_width,
               size_t nbirdies, size_t nbins, cudaStream_t s)
{
    if (nbirdies == 0) return PSX_OK;
    if (!d_X || !d_freqs || !d_widths) {
        set_error("zap: null pointer");
        return PSX_ERR_INVALID;
    }
    const unsigned T = 256;
    const unsigned blocks = (unsigned)((nbirdies * 32 + T - 1) / T);
    k_zap<<<blocks, T, 0, s>>>(d_X, d_freqs, d_widths, bin_width, (unsigned)nbirdies,
                               (unsigned)nbins);
    return launch_status("zap kernel");
}

// ---------------------------------------------------------------- reductions
// Deterministic two-level sum of x and x^2 (double accumulators): each
// block writes its partials, one block adds them in fixed order.
template <class Src>
__global__ void __launch_bounds__(256) k_sum_partials(Src src, size_t first, size_t n,
                                                      double2* __restrict__ partials)
{
    double s = 0.0, s2 = 0.0;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = first + (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const double v = src(i);
        s += v;
        s2 += v * v;
    }
    for (int o = 16; o; o >>= 1) {
        s += __shfl_down_sync(0xffffffffu, s, o);
        s2 += __shfl_down_sync(0xffffffffu, s2, o);
    }
    __shared__ double sh[2][8];
    const int w = threadIdx.x / 32;
    if ((threadIdx.x & 31) == 0) {
        sh[0][w] = s;
        sh[1][w] = s2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int i = 0; i < (int)(blockDim.x / 32); ++i) {
            a += sh[0][i];
            b += sh[1][i];
        }
        partials[blockIdx.x] = make_double2(a, b);
    }
}

// The reference's float statistics {mean, rms, std, mean*scale, std*scale} of
// `count` values with sums a and (of squares) b, computed exactly as its host
// code does (stats.hpp:20-31 and src/kernels.cu:443,458), without contraction.
__device__ __forceinline__ void write_stats(double a, double b, double count,
                                            float* __restrict__ stat, float scale)
{
    const float cnt = (float)count;
    const float mean = __fdiv_rn((float)a, cnt);
    const float rms = sqrtf(__fdiv_rn((float)b, cnt));
    const float sd = sqrtf(__fsub_rn(__fmul_rn(rms, rms), __fmul_rn(mean, mean)));
    stat[0] = mean;
    stat[1] = rms;
    stat[2] = sd;
    stat[3] = __fmul_rn(mean, scale);
    stat[4] = __fmul_rn(sd, scale);
}

// Adds `nparts` partials (one warp, fixed order); writes the totals to sums[0..1]
// and, when stat != nullptr, the statistics of write_stats.
__global__ void k_finish_stats(const double2* __restrict__ partials, int nparts, double count,
                               double* __restrict__ sums, float* __restrict__ stat, float scale,
                               size_t part_stride = 0, size_t sums_stride = 0,
                               size_t stat_stride = 0)
{
    if (blockIdx.x != 0 || threadIdx.x >= 32) return;
    // row blockIdx.y of a batch (strides in elements)
    partials += (size_t)blockIdx.y * part_stride;
    sums += (size_t)blockIdx.y * sums_stride;
    if (stat) stat += (size_t)blockIdx.y * stat_stride;
    double a, b;
    warp_sum_partials(partials, nparts, a, b);
    if (threadIdx.x != 0) return;
    sums[0] = a;
    sums[1] = b;
    if (stat) write_stats(a, b, count, stat, scale);
}

struct PlainSrc {
    const float* x;
    __device__ double operator()(size_t i) const { return (double)x[i]; }
};

struct InterbinSrc {
    const float* X;
    __device__ double operator()(size_t k) const
    {
        const float re = X[2 * k], im = X[2 * k + 1];
        const float rl = k ? X[2 * k - 2] : 0.f, il = k ? X[2 * k - 1] : 0.f;
        return (double)interbin(re, im, rl, il);
    }
};

// Block sum of (a, b) pairs into partials[blockIdx.x] (fixed order).
template <int NT>
__device__ __forceinline__ void block_partials(double s, double s2, double2* __restrict__ partials)
{
    for (int o = 16; o; o >>= 1) {
        s += __shfl_down_sync(0xffffffffu, s, o);
        s2 += __shfl_down_sync(0xffffffffu, s2, o);
    }
    __shared__ double sh[2][NT / 32];
    const int w = threadIdx.x / 32;
    if ((threadIdx.x & 31) == 0) {
        sh[0][w] = s;
        sh[1][w] = s2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int i = 0; i < NT / 32; ++i) {
            a += sh[0][i];
            b += sh[1][i];
        }
        partials[blockIdx.x] = make_double2(a, b);
    }
}

__device__ __forceinline__ void acc4(float4 v, double& s, double& s2)
{
    const double a = v.x, b = v.y, c = v.z, d = v.w;
    s += (a + b) + (c + d);
    s2 += (a * a + b * b) + (c * c + d * d);
}

constexpr int kVecThreads = 512;

// Partial sums of x and x^2 over [0, n) with 128-bit loads (x 16-byte
// aligned); the n % 4 tail is added by block 0.  With `copy` set, x is also
// written there (16-byte aligned), fusing the copy of a series into its
// first pass; with `state` set, block 0 starts the baseline loop state
// (state[0] = 1 active, state[1] = 0 passes).
__global__ void __launch_bounds__(kVecThreads) k_partials_v4(const float* __restrict__ x, size_t n,
                                                             double2* __restrict__ partials,
                                                             float* __restrict__ copy,
                                                             unsigned* __restrict__ state,
                                                             size_t x_stride = 0,
                                                             size_t part_stride = 0,
                                                             size_t state_stride = 0)
{
    // row blockIdx.y of a batch (strides in elements; no copy in a batch)
    x += (size_t)blockIdx.y * x_stride;
    partials += (size_t)blockIdx.y * part_stride;
    if (state) state += (size_t)blockIdx.y * state_stride;
    if (state && blockIdx.x == 0 && threadIdx.x == 0) {
        state[0] = 1u;
        state[1] = 0u;
    }
    double s = 0.0, s2 = 0.0;
    const size_t n4 = n / 4, stride = (size_t)gridDim.x * blockDim.x;
    const float4* x4 = reinterpret_cast<const float4*>(x);
    float4* c4 = reinterpret_cast<float4*>(copy);
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < n4; q += stride) {
        const float4 v = x4[q];
        if (copy) c4[q] = v;
        acc4(v, s, s2);
    }
    if (blockIdx.x == 0 && threadIdx.x < n - 4 * n4) {
        const float v = x[4 * n4 + threadIdx.x];
        if (copy) copy[4 * n4 + threadIdx.x] = v;
        s += (double)v;
        s2 += (double)v * v;
    }
    block_partials<kVecThreads>(s, s2, partials);
}

// One pass of the device-side baseline loop (reference src/kernels.cu:
// 463-479) in one kernel.  While *flag_in says the loop goes on, every CTA
// forms the float mean of the previous pass's partials (float sum / float
// count; the same fixed-order sum in every CTA), subtracts it, and, while
// |mean| > 5e-7 n, writes its partials of the new x to part_out; CTA 0
// records the decision in *flag_out and counts the pass.  Flags and
// partials alternate between passes, so no CTA reads what this pass writes.
// With fin_flag set (the last pass) the final decision and the pass count
// are copied there and to fin_passes.
__global__ void __launch_bounds__(kVecThreads) k_baseline_pass_v4(
    float* __restrict__ x, size_t n, double count, const double2* __restrict__ part_in,
    int nparts, double2* __restrict__ part_out, const unsigned* __restrict__ flag_in,
    unsigned* __restrict__ flag_out, unsigned* __restrict__ passes,
    unsigned* __restrict__ fin_flag, unsigned* __restrict__ fin_passes, size_t x_stride = 0,
    size_t part_stride = 0, size_t flag_stride = 0)
{
    if (blockIdx.y) {  // row blockIdx.y of a batch (strides in elements)
        const size_t r = blockIdx.y;
        x += r * x_stride;
        part_in += r * part_stride;
        part_out += r * part_stride;
        flag_in += r * flag_stride;
        flag_out += r * flag_stride;
        passes += r * flag_stride;
        if (fin_flag) fin_flag += r * flag_stride;
        if (fin_passes) fin_passes += r * flag_stride;
    }
    __shared__ float s_mean;
    __shared__ int s_go;
    if (*flag_in == 0u) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            *flag_out = 0u;
            if (fin_flag) {
                *fin_flag = 0u;
                *fin_passes = *passes;
            }
        }
        return;
    }
    if (threadIdx.x < 32) {
        double a, b;
        warp_sum_partials(part_in, nparts, a, b);
        if (threadIdx.x == 0) {
            const float mean = __fdiv_rn((float)a, (float)count);
            s_mean = mean;
            s_go = (fabsf(mean) > 5e-7 * count) ? 1 : 0;
        }
    }
    __syncthreads();
    const float m = s_mean;
    const bool sum = s_go != 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const unsigned np = *passes + 1u;
        *passes = np;
        *flag_out = sum ? 1u : 0u;
        if (fin_flag) {
            *fin_flag = sum ? 1u : 0u;
            *fin_passes = np;
        }
    }
    if (m == 0.0f) return;
    double s = 0.0, s2 = 0.0;
    const size_t n4 = n / 4, stride = (size_t)gridDim.x * blockDim.x;
    float4* x4 = reinterpret_cast<float4*>(x);
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < n4; q += stride) {
        float4 v = x4[q];
        v.x -= m;
        v.y -= m;
        v.z -= m;
        v.w -= m;
        x4[q] = v;
        if (sum) acc4(v, s, s2);
    }
    if (blockIdx.x == 0 && threadIdx.x < n - 4 * n4) {
        const float v = x[4 * n4 + threadIdx.x] - m;
        x[4 * n4 + threadIdx.x] = v;
        s += (double)v;
        s2 += (double)v * v;
    }
    if (sum) block_partials<kVecThreads>(s, s2, part_out);
}

// Partial sums of the interbinned amplitude of the complex spectrum X over
// bins [0, nbins): two bins per thread from one 128-bit load, the previous
// bin's pair from a 64-bit load; the odd last bin is added by block 0.
__global__ void __launch_bounds__(kVecThreads) k_interbin_partials_v4(const float* __restrict__ X,
                                                                      size_t nbins,
                                                                      double2* __restrict__ partials,
                                                                      size_t x_stride = 0,
                                                                      size_t part_stride = 0)
{
    X += (size_t)blockIdx.y * x_stride;  // row blockIdx.y of a batch
    partials += (size_t)blockIdx.y * part_stride;
    double s = 0.0, s2 = 0.0;
    const size_t npairs = nbins / 2, stride = (size_t)gridDim.x * blockDim.x;
    const float4* X4 = reinterpret_cast<const float4*>(X);
    const float2* X2 = reinterpret_cast<const float2*>(X);
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < npairs; q += stride) {
        const float4 v = X4[q];
        const float2 l = q ? X2[2 * q - 1] : make_float2(0.f, 0.f);
        const double a = interbin(v.x, v.y, l.x, l.y);
        const double b = interbin(v.z, v.w, v.x, v.y);
        s += a + b;
        s2 += a * a + b * b;
    }
    if ((nbins & 1) && blockIdx.x == 0 && threadIdx.x == 0) {
        const size_t k = nbins - 1;
        const float2 l = k ? X2[k - 1] : make_float2(0.f, 0.f);
        const double a = interbin(X[2 * k], X[2 * k + 1], l.x, l.y);
        s += a;
        s2 += a * a;
    }
    block_partials<kVecThreads>(s, s2, partials);
}

int reduction_blocks() { return sm_count() * 2; }

// The means of the baseline loop are sums over fixed pieces of the series,
// one warp to a piece, added in one order: the 16 pieces of a group, then the
// groups, 32 apart to a lane.  A mean then depends on the samples alone and
// not on the rows that share its launch, the CTAs of a row or the address of
// the series, and with it the dereddened series of a DM trial, bit for bit.
// 512 pieces up to 2^21 samples, one to a warp of a 16-CTA cluster; 2048, four
// to such a warp, up to 2^23, the longest row a cluster takes; 4096 above,
// where the series come from HBM (2^26 samples, whole search: 7151 us on B200
// with 2048 pieces, 7106 with 4096; 12 series of 2^23: 2300 and 2455).
constexpr size_t kMeanShort = (size_t)1 << 21, kMeanMedium = (size_t)1 << 23;
constexpr unsigned kMeanGroup = 16;
inline unsigned mean_pieces(size_t n)
{
    return n <= kMeanShort ? 512u : n <= kMeanMedium ? 2048u : 4096u;
}

__device__ __forceinline__ double warp_total(double v, int width)
{
    for (int o = width / 2; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Adds (x - m0) - m1 (x - 0 is x) over pieces first + k W, k < K, of
// `pieces` to this lane's s[k].  Piece v holds the runs of 128 samples
// v, v + pieces, ..., four consecutive samples to a lane; the n % 4 last
// samples go to piece 0.
template <int K>
__device__ __forceinline__ void piece_sums(const float* __restrict__ x, size_t n, unsigned pieces,
                                           unsigned first, unsigned W, float m0, float m1,
                                           double (&s)[K])
{
    const unsigned lane = threadIdx.x & 31;
    const size_t n4 = n / 4, steps = n4 / 32 / pieces;
    auto less = [&](float v) { return (double)((v - m0) - m1); };
    auto run = [&](auto load) {
        auto add = [&](double& t, const float* p) {
            const float4 v = load(p);
            t += (less(v.x) + less(v.y)) + (less(v.z) + less(v.w));
        };
        const size_t step = (size_t)pieces * 128;
        const unsigned next = W * 128;
        const float* p = x + ((size_t)first * 32 + lane) * 4;
#pragma unroll (8 / K)
        for (size_t j = 0; j < steps; ++j, p += step)  // eight loads in flight
#pragma unroll
            for (int k = 0; k < K; ++k) add(s[k], p + k * next);
#pragma unroll
        for (int k = 0; k < K; ++k)
            if ((steps * pieces + first + k * W) * 32 + lane < n4) add(s[k], p + k * next);
    };
    if ((reinterpret_cast<uintptr_t>(x) & 15u) == 0)
        run([](const float* p) { return *reinterpret_cast<const float4*>(p); });
    else
        run([](const float* p) { return make_float4(p[0], p[1], p[2], p[3]); });
    if (first == 0 && lane < n - 4 * n4) s[0] += less(x[4 * n4 + lane]);
}

// The device-side baseline loop (reference src/kernels.cu:463-479) without
// writing the series: every pass finds the float mean that the reference
// would subtract next, from the sums of the series less the means found so
// far (the subtraction itself, in the same order and so with the same
// roundings, is done by the transform's loads).  Pass 0 (FIRST) sums the
// series; pass p forms mean p - 1 from the previous pass's group sums and,
// while |mean| > 5e-7 n, sums again.  A CTA sums one group of pieces.  Row
// blockIdx.y of a batch; `cnt` as Slot::d_count (16 words a row: [2] still
// active after the last pass, [3] passes, [6 + p] pass p's flag), `means` 4
// floats a row.
constexpr int kMeanGroupThreads = 32 * kMeanGroup;

template <bool FIRST>
__global__ void __launch_bounds__(kMeanGroupThreads) k_baseline_means(
    const __grid_constant__ SeriesRows rows, size_t n, double* __restrict__ sums, size_t sum_stride,
    unsigned* __restrict__ cnt, float* __restrict__ means, int pass, int last)
{
    const float* x = rows.p[blockIdx.y];
    unsigned* c = cnt + 16 * blockIdx.y;
    float* m = means + 4 * blockIdx.y;
    const unsigned groups = gridDim.x, lane = threadIdx.x & 31, warp = threadIdx.x / 32;
    double* out = sums + (size_t)blockIdx.y * sum_stride;  // two halves: passes alternate
    const double* in = out + ((pass - 1) & 1) * groups;
    out += (pass & 1) * groups;
    double s[1] = {0.0};
    const unsigned first = blockIdx.x * kMeanGroup + warp, pieces = groups * kMeanGroup;
    const bool one = blockIdx.x == 0 && threadIdx.x == 0;
    if constexpr (FIRST) {
        if (one) {
            c[6] = 1u;
            for (int k = 0; k < 4; ++k) m[k] = 0.f;
        }
        piece_sums<1>(x, n, pieces, first, 0, 0.f, 0.f, s);
    } else {
        // (mean p - 1 is read by nobody else in this pass: every CTA forms it)
        const bool active = c[6 + pass - 1] != 0u;
        if (!active) {
            if (one) {
                c[6 + pass] = 0u;
                if (last) c[2] = 0u;
            }
            return;
        }
        __shared__ float s_mean;
        if (warp == 0) {
            double t = 0.0;
            for (unsigned g = lane; g < groups; g += 32) t += in[g];
            t = warp_total(t, 32);
            if (lane == 0) s_mean = __fdiv_rn((float)t, (float)(double)n);
        }
        __syncthreads();
        const float mean = s_mean;
        const bool more = fabsf(mean) > 5e-7 * (double)n;
        if (one) {
            m[pass - 1] = mean;
            c[6 + pass] = more ? 1u : 0u;
            c[3] = (unsigned)pass;
            if (last) c[2] = more ? 1u : 0u;
        }
        if (!more || last) return;
        if (pass > 1)
            piece_sums<1>(x, n, pieces, first, 0, m[0], mean, s);
        else
            piece_sums<1>(x, n, pieces, first, 0, mean, 0.f, s);
    }
    __shared__ double sh[kMeanGroup];
    s[0] = warp_total(s[0], 32);
    if (lane == 0) sh[warp] = s[0];
    __syncthreads();
    if (warp == 0) {
        const double t = warp_total(lane < kMeanGroup ? sh[lane] : 0.0, kMeanGroup);
        if (lane == 0) out[blockIdx.x] = t;
    }
}
static_assert(kBaselineMeans == 3, "the third mean needs no sum after it");

// The same loop in one launch: a cluster of CTAs per row sums, K pieces to a
// warp, exchanges its group sums through distributed shared memory and goes
// round again while the mean is above the threshold.  Clusters of 16 (8 for
// more than 8 rows up to 2^21 samples, where 16 would take two waves); a few
// SMs read a long row slower than the whole device, so fewer than 4 rows take
// it up to 2^21 samples, 4 and more up to 2^23.  A call of 1, 12 and 48 DM
// trials on B200 (us; four launches, one with clusters of 8, of 16): 2^19:
// 171/162/164, 513/397/379, 1225/744/793; 2^20: 173/170/164, 614/508/494,
// 1797/1370/1346; 2^21: 178/187/176, 887/808/777, 2828/2497/2416; 2^22:
// 231/300/258, 1428/1435/1356, 5093/5001/4872.  (With sums per CTA; pieces of
// their own per warp take the same within 1 %, and the four launches at 2^23
// 4 % less of a 12-DM call, 2355 against 2455.)
constexpr int kMeanThreads = 1024;
inline unsigned mean_ctas(int rows, size_t n) { return rows > 8 && n <= kMeanShort ? 8u : 16u; }
inline size_t mean_max_samples(int rows) { return rows < 4 ? kMeanShort : kMeanMedium; }

template <int K>
__global__ void __launch_bounds__(kMeanThreads) k_baseline_means_cluster(
    const __grid_constant__ SeriesRows rows, size_t n, unsigned* __restrict__ cnt,
    float* __restrict__ means)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const float* x = rows.p[blockIdx.y];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x / 32;
    const unsigned W = cl.num_blocks() * (kMeanThreads / 32), pieces = K * W;
    __shared__ double warp_sum[K][kMeanThreads / 32];
    __shared__ double part[kBaselineMeans][2 * K];  // this CTA's group sums of each pass
    static_assert(kMeanThreads / 32 == 2 * kMeanGroup, "two groups to the warps of a CTA");
    float m[kBaselineMeans] = {0.f, 0.f, 0.f};
    int pass = 0;
    bool more = true;
#pragma unroll
    for (int p = 0; p < kBaselineMeans; ++p) {
        if (!more) break;  // the same in every thread of the cluster
        double s[K] = {};
        piece_sums<K>(x, n, pieces, cl.block_rank() * (kMeanThreads / 32) + warp, W, m[0], m[1], s);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            s[k] = warp_total(s[k], 32);
            if (lane == 0) warp_sum[k][warp] = s[k];
        }
        __syncthreads();
        if (warp < K) {
            const double t = warp_total(warp_sum[warp][lane], kMeanGroup);
            if (lane % kMeanGroup == 0) part[p][2 * warp + lane / kMeanGroup] = t;
        }
        cl.sync();
        // group g is half g % 2 of the warps that CTA (g / 2) % CTAs ran its
        // k = g / 2 / CTAs on
        double total = 0.0;
        for (unsigned g = lane; g < pieces / kMeanGroup; g += 32)
            total += *cl.map_shared_rank(&part[p][2 * (g / 2 / cl.num_blocks()) + g % 2],
                                         g / 2 % cl.num_blocks());
        total = warp_total(total, 32);
        m[p] = __fdiv_rn((float)total, (float)(double)n);
        more = fabsf(m[p]) > 5e-7 * (double)n;
        pass = p + 1;
    }
    if (cl.block_rank() == 0 && threadIdx.x == 0) {
        unsigned* c = cnt + 16 * blockIdx.y;
        c[2] = more ? 1u : 0u;
        c[3] = (unsigned)pass;
        for (int k = 0; k < kBaselineMeans; ++k) means[4 * blockIdx.y + k] = m[k];
    }
    cl.sync();  // no CTA leaves while another reads its partial sums
}

// Launches the cluster form with K pieces to a warp; false where this device
// does not run such clusters (asked once per device and K: 16 is above the
// portable 8).
template <int K>
static bool mean_cluster(cudaLaunchConfig_t cfg, const SeriesRows& rows, size_t n, unsigned* d_cnt,
                         float* d_means, int* rc)
{
    static std::mutex mu;
    static int table[64] = {};  // 1 yes, 2 no
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!table[dev]) {
            int fit = 0;
            const bool ok = cudaFuncSetAttribute(k_baseline_means_cluster<K>,
                                                 cudaFuncAttributeNonPortableClusterSizeAllowed,
                                                 1) == cudaSuccess &&
                            cudaOccupancyMaxActiveClusters(&fit, k_baseline_means_cluster<K>,
                                                           &cfg) == cudaSuccess && fit > 0;
            (void)cudaGetLastError();
            table[dev] = ok ? 1 : 2;
        }
        if (table[dev] != 1) return false;
    }
    *rc = cuda_status(cudaLaunchKernelEx(&cfg, k_baseline_means_cluster<K>, rows, n, d_cnt, d_means),
                      "baseline mean kernel");
    return true;
}

int launch_baseline_means(const SeriesRows& rows, int nrows, size_t n, double2* d_parts,
                          size_t part_stride, unsigned* d_cnt, float* d_means, cudaStream_t s,
                          int* launches)
{
    const unsigned pieces = mean_pieces(n);
    if (n <= mean_max_samples(nrows)) {
        const unsigned ctas = mean_ctas(nrows, n);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(ctas, nrows);
        cfg.blockDim = dim3(kMeanThreads);
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim = {ctas, 1, 1};
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int rc = PSX_OK;
        bool ran = false;
        switch (pieces / (ctas * (kMeanThreads / 32))) {
        case 1: ran = mean_cluster<1>(cfg, rows, n, d_cnt, d_means, &rc); break;
        case 2: ran = mean_cluster<2>(cfg, rows, n, d_cnt, d_means, &rc); break;
        default: ran = mean_cluster<4>(cfg, rows, n, d_cnt, d_means, &rc); break;
        }
        if (ran) {
            ++*launches;
            return rc;
        }
    }
    const dim3 grid(pieces / kMeanGroup, nrows);
    double* sums = reinterpret_cast<double*>(d_parts);
    if (part_stride < grid.x) {  // (a row's two halves, in double2)
        set_error("baseline means: partial sums of a row hold %zu entries", part_stride);
        return PSX_ERR_INVALID;
    }
    *launches += 1 + kBaselineMeans;
    k_baseline_means<true><<<grid, kMeanGroupThreads, 0, s>>>(rows, n, sums, 2 * part_stride, d_cnt,
                                                              d_means, 0, 0);
    for (int pass = 1; pass <= kBaselineMeans; ++pass)
        k_baseline_means<false><<<grid, kMeanGroupThreads, 0, s>>>(
            rows, n, sums, 2 * part_stride, d_cnt, d_means, pass, pass == kBaselineMeans);
    return launch_status("baseline mean kernels");
}

// Median levels of `rows` amplitude spectra (strides in floats).
int launch_scrunch_rows(const float* d_amp, size_t stride, int rows, size_t nbins, float* d_scratch,
                        size_t scratch_stride, cudaStream_t s)
{
    auto up = [](size_t v) { return (v + 63) / 64 * 64; };
    float* m25 = d_scratch + up(nbins / 5 + 1);
    float* m125 = m25 + up(nbins / 25 + 1);
    const size_t n5 = nbins / 5, n25 = n5 / 5, n125 = n25 / 5, ngroups = (n5 + 24) / 25;
    const unsigned grid = (unsigned)std::min<size_t>((ngroups + kScrGroups - 1) / kScrGroups,
                                                     (size_t)sm_count() * 8);
    k_scrunch3<false><<<dim3(grid, rows), 256, 0, s>>>(d_amp, d_scratch, n5, m25, n25, m125, n125,
                                                       stride, scratch_stride);
    return launch_status("scrunch kernel (rows)");
}

// k_finish_stats for many partials: 32 warps, each a fixed run of them.
__global__ void __launch_bounds__(1024) k_finish_stats_wide(const double2* __restrict__ partials,
                                                            int nparts, double count,
                                                            float* __restrict__ stat, float scale,
                                                            size_t part_stride, size_t stat_stride)
{
    partials += (size_t)blockIdx.y * part_stride;
    stat += (size_t)blockIdx.y * stat_stride;
    __shared__ double2 sh[32];
    const int w = threadIdx.x / 32, per = (nparts + 31) / 32;
    const int p0 = min(nparts, w * per), np = min(nparts, p0 + per) - p0;
    double a, b;
    warp_sum_partials(partials + p0, np, a, b);
    if ((threadIdx.x & 31) == 0) sh[w] = make_double2(a, b);
    __syncthreads();
    if (threadIdx.x >= 32) return;
    warp_sum_partials(sh, 32, a, b);
    if (threadIdx.x == 0) write_stats(a, b, count, stat, scale);
}

int launch_finish_stats_rows(const double2* d_partials, int nparts, size_t part_stride, int rows,
                             size_t count, float* d_stat, size_t stat_stride, float scale,
                             cudaStream_t s)
{
    k_finish_stats_wide<<<dim3(1, rows), 1024, 0, s>>>(d_partials, nparts, (double)count, d_stat,
                                                       scale, part_stride, stat_stride);
    return launch_status("statistics kernel (rows)");
}

// Bits of the bins that k_zap sets (the same ranges), for kernels that zap
// as they go.
__global__ void k_zap_mask(unsigned* __restrict__ mask, const float* __restrict__ freqs,
                           const float* __restrict__ widths, float bin_width, unsigned nbirdies,
                           unsigned nbins)
{
    const unsigned warp = (blockIdx.x * blockDim.x + threadIdx.x) / 32;
    if (warp >= nbirdies) return;
    int lo, hi;
    if (!zap_range(freqs[warp], widths[warp], bin_width, nbins, lo, hi)) return;
    for (int k = lo + (int)(threadIdx.x & 31); k < hi; k += 32)
        atomicOr(mask + (k >> 5), 1u << (k & 31));
}

int launch_zap_mask(unsigned* d_mask, const float* d_freqs, const float* d_widths, float bin_width,
                    size_t nbirdies, size_t nbins, cudaStream_t s)
{
    PSX_CUDA(cudaMemsetAsync(d_mask, 0, (nbins + 31) / 32 * sizeof(unsigned), s));
    if (nbirdies == 0) return PSX_OK;
    k_zap_mask<<<(unsigned)((nbirdies * 32 + 255) / 256), 256, 0, s>>>(
        d_mask, d_freqs, d_widths, bin_width, (unsigned)nbirdies, (unsigned)nbins);
    return launch_status("zap mask kernel");
}

int launch_partials_v4(const float* d_x, size_t n, double2* d_partials, float* d_copy,
                       unsigned* d_state, cudaStream_t s)
{
    k_partials_v4<<<reduction_blocks(), kVecThreads, 0, s>>>(d_x, n, d_partials, d_copy, d_state);
    return launch_status("partial sums kernel");
}

int launch_baseline_pass_v4(float* d_x, size_t n, const double2* d_part_in, double2* d_part_out,
                            const unsigned* d_flag_in, unsigned* d_flag_out, unsigned* d_passes,
                            unsigned* d_fin_flag, unsigned* d_fin_passes, cudaStream_t s)
{
    const int nb = reduction_blocks();
    k_baseline_pass_v4<<<nb, kVecThreads, 0, s>>>(d_x, n, (double)n, d_part_in, nb, d_part_out,
                                                  d_flag_in, d_flag_out, d_passes, d_fin_flag,
                                                  d_fin_passes);
    return launch_status("baseline pass kernel");
}

int launch_interbin_stats_v4(const float* d_X, size_t nbins, double2* d_partials, double* d_sums,
                             float* d_stat, float scale, cudaStream_t s)
{
    const int nb = reduction_blocks();
    k_interbin_partials_v4<<<nb, kVecThreads, 0, s>>>(d_X, nbins, d_partials);
    k_finish_stats<<<1, 32, 0, s>>>(d_partials, nb, (double)nbins, d_sums, d_stat, scale);
    return launch_status("interbin statistics kernels");
}

// ---- row-batched prologue stages (the grouped prologue of the engine)
int launch_partials_rows(const float* d_x, size_t n, size_t x_stride, int rows,
                         double2* d_partials, size_t part_stride, unsigned* d_state,
                         size_t state_stride, cudaStream_t s)
{
    if (rows < 1 || rows > 65535) {
        set_error("partial sums: bad row count %d", rows);
        return PSX_ERR_INVALID;
    }
    k_partials_v4<<<dim3(reduction_blocks(), rows), kVecThreads, 0, s>>>(
        d_x, n, d_partials, nullptr, d_state, x_stride, part_stride, state_stride);
    return launch_status("partial sums kernel (rows)");
}

int launch_baseline_pass_rows(float* d_x, size_t n, size_t x_stride, int rows,
                              const double2* d_part_in, double2* d_part_out, size_t part_stride,
                              const unsigned* d_flag_in, unsigned* d_flag_out,
                              unsigned* d_passes, unsigned* d_fin_flag, unsigned* d_fin_passes,
                              size_t flag_stride, cudaStream_t s)
{
    const int nb = reduction_blocks();
    k_baseline_pass_v4<<<dim3(nb, rows), kVecThreads, 0, s>>>(
        d_x, n, (double)n, d_part_in, nb, d_part_out, d_flag_in, d_flag_out, d_passes, d_fin_flag,
        d_fin_passes, x_stride, part_stride, flag_stride);
    return launch_status("baseline pass kernel (rows)");
}

int launch_running_median_spectrum_rows(float* d_X, size_t x_stride, int rows, size_t nbins,
                                        double bin_width, float b5, float b25, void* d_scratch,
                                        size_t scratch_stride_floats, cudaStream_t s)
{
    if (!d_X || !d_scratch || nbins < 125 || nbins > 0xffffffffu) {
        set_error("running median: bad arguments (nbins=%zu)", nbins);
        return PSX_ERR_INVALID;
    }
    auto up = [](size_t v) { return (v + 63) / 64 * 64; };
    float* m5 = static_cast<float*>(d_scratch);
    float* m25 = m5 + up(nbins / 5 + 1);
    float* m125 = m25 + up(nbins / 25 + 1);
    const size_t n5 = nbins / 5, n25 = n5 / 5, n125 = n25 / 5;
    const size_t ngroups = (n5 + 24) / 25;
    const unsigned grid = (unsigned)std::min<size_t>((ngroups + kScrGroups - 1) / kScrGroups,
                                                     (size_t)sm_count() * 8);
    k_scrunch3<true><<<dim3(grid, rows), 256, 0, s>>>(d_X, m5, n5, m25, n25, m125, n125, x_stride,
                                                      scratch_stride_floats);
    PSX_TRY(launch_status("amplitude + scrunch kernel (rows)"));
    const MedianLevels L = median_levels(nbins, bin_width, b5, b25, m5);
    k_median_apply<<<dim3(grid_for(nbins, 256), rows), 256, 0, s>>>(
        L, nbins, nullptr, d_X, x_stride, scratch_stride_floats);
    return launch_status("median apply kernel (rows)");
}

int launch_zap_rows(float* d_X, size_t x_stride, int rows, const float* d_freqs,
                    const float* d_widths, float bin_width, size_t nbirdies, size_t nbins,
                    cudaStream_t s)
{
    if (nbirdies == 0) return PSX_OK;
    if (!d_X || !d_freqs || !d_widths) {
        set_error("zap: null pointer");
        return PSX_ERR_INVALID;
    }
    const unsigned T = 256;
    const unsigned blocks = (unsigned)((nbirdies * 32 + T - 1) / T);
    k_zap<<<dim3(blocks, rows), T, 0, s>>>(d_X, d_freqs, d_widths, bin_width, (unsigned)nbirdies,
                                          (unsigned)nbins, x_stride);
    return launch_status("zap kernel (rows)");
}

int launch_interbin_stats_rows(const float* d_X, size_t x_stride, int rows, size_t nbins,
                               double2* d_partials, size_t part_stride, double* d_sums,
                               size_t sums_stride, float* d_stat, size_t stat_stride, float scale,
                               cudaStream_t s)
{
    const int nb = reduction_blocks();
    k_interbin_partials_v4<<<dim3(nb, rows), kVecThreads, 0, s>>>(d_X, nbins, d_partials, x_stride,
                                                                  part_stride);
    k_finish_stats<<<dim3(1, rows), 32, 0, s>>>(d_partials, nb, (double)nbins, d_sums, d_stat,
                                                scale, part_stride, sums_stride, stat_stride);
    return launch_status("interbin statistics kernels (rows)");
}

int launch_partials(const float* d_x, size_t n, double2* d_partials, cudaStream_t s)
{
    k_sum_partials<PlainSrc><<<reduction_blocks(), 256, 0, s>>>(PlainSrc{d_x}, 0, n, d_partials);
    return launch_status("partial sums kernel");
}

int launch_stats(const float* d_x, bool interbinned, size_t first, size_t n, double2* d_partials,
                 double* d_sums, float* d_stat, float scale, cudaStream_t s)
{
    const unsigned T = 256;
    const int nb = reduction_blocks();
    if (!interbinned && (reinterpret_cast<uintptr_t>(d_x + first) & 15u) == 0)
        k_partials_v4<<<nb, kVecThreads, 0, s>>>(d_x + first, n - first, d_partials, nullptr,
                                                 nullptr);
    else if (interbinned)
        k_sum_partials<InterbinSrc><<<nb, T, 0, s>>>(InterbinSrc{d_x}, first, n, d_partials);
    else
        k_sum_partials<PlainSrc><<<nb, T, 0, s>>>(PlainSrc{d_x}, first, n, d_partials);
    k_finish_stats<<<1, 32, 0, s>>>(d_partials, nb, (double)(n - first), d_sums, d_stat, scale);
    return launch_status("statistics kernels");
}

// ------------------------------------------------------------- element-wise
// Four values per thread from one 128-bit load where x is 16-byte aligned
// (VEC), the n % 4 last ones by block 0.
template <bool VEC>
__global__ void __launch_bounds__(256) k_normalise(float* __restrict__ x, float mean, float sigma,
                                                   size_t n)
{
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const size_t first = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if constexpr (VEC) {
        float4* x4 = reinterpret_cast<float4*>(x);
        for (size_t q = first; q < n / 4; q += stride) {
            float4 v = x4[q];
            v.x = normalise(v.x, mean, sigma);
            v.y = normalise(v.y, mean, sigma);
            v.z = normalise(v.z, mean, sigma);
            v.w = normalise(v.w, mean, sigma);
            x4[q] = v;
        }
        const size_t i = n / 4 * 4 + first;
        if (blockIdx.x == 0 && i < n) x[i] = normalise(x[i], mean, sigma);
    } else {
        for (size_t i = first; i < n; i += stride) x[i] = normalise(x[i], mean, sigma);
    }
}

__global__ void k_sub_scalar(float* __restrict__ x, size_t n, const float* __restrict__ v)
{
    const float m = *v;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) x[i] -= m;
}

__global__ void k_fill(float* __restrict__ x, size_t n, float value, size_t x_stride = 0)
{
    x += (size_t)blockIdx.y * x_stride;  // row blockIdx.y of a batch
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) x[i] = value;
}

template <class T>
__global__ void k_convert(const T* __restrict__ in, float* __restrict__ out, size_t n)
{
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        out[i] = static_cast<float>(in[i]);
}

int launch_sub_scalar(float* d_x, size_t n, const float* d_v, cudaStream_t s)
{
    if (n == 0) return PSX_OK;
    k_sub_scalar<<<grid_for(n, 256), 256, 0, s>>>(d_x, n, d_v);
    return launch_status("subtract kernel");
}

int launch_fill(float* d_x, size_t n, float value, cudaStream_t s)
{
    if (n == 0) return PSX_OK;
    k_fill<<<grid_for(n, 256), 256, 0, s>>>(d_x, n, value);
    return launch_status("fill kernel");
}

int launch_fill_rows(float* d_x, size_t n, size_t x_stride, int rows, float value,
                     cudaStream_t s)
{
    if (n == 0) return PSX_OK;
    dim3 grid(grid_for(n, 256), rows);
    k_fill<<<grid, 256, 0, s>>>(d_x, n, value, x_stride);
    return launch_status("fill kernel (rows)");
}

// Mean of d_x[0..n) in float as the reference forms it (float sum / float
// count), from a double-accumulated sum; written to d_mean.
__global__ void k_mean_from_sums(const double* __restrict__ sums, double count,
                                 float* __restrict__ d_mean)
{
    *d_mean = __fdiv_rn((float)sums[0], (float)count);
}

int remove_baseline_pass(float* d_x, size_t n, double2* d_partials, double* d_sums,
                         float* d_mean, cudaStream_t s)
{
    const unsigned T = 256;
    const int nb = reduction_blocks();
    k_sum_partials<PlainSrc><<<nb, T, 0, s>>>(PlainSrc{d_x}, 0, n, d_partials);
    k_finish_stats<<<1, 32, 0, s>>>(d_partials, nb, (double)n, d_sums, nullptr, 0.f);
    k_mean_from_sums<<<1, 1, 0, s>>>(d_sums, (double)n, d_mean);
    k_sub_scalar<<<grid_for(n, T), T, 0, s>>>(d_x, n, d_mean);
    return launch_status("baseline kernels");
}

// ----------------------------------------------------------- harmonic sums
struct FoldPtrs {
    float* p[5];
};

// Adds the fractions m/2^H (odd m, in the reference's order) of the bins
// i + 32 k, k < K, to val: 32 m / 2^H is whole for H <= 5, so the K reads of
// a fraction are one computed index and constant distances from it.
template <int H, int K>
__device__ __forceinline__ void add_fractions(const float* __restrict__ in, unsigned i, int take,
                                              float (&val)[K])
{
#pragma unroll
    for (int r = 0; r < (1 << (H - 1)); ++r) {
        const unsigned m = H == 2 ? (r == 0 ? 3u : 1u) : 2u * r + 1u;  // fold 2 adds 3/4 first
        const float* p = in + frac_index<H>(i, m);
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (k < take) val[k] += p[(size_t)k * (32u * m >> H)];
    }
}

// The running sums in the reference's order (src/kernels.cu:41-96): a warp
// takes 32 K consecutive bins, lane l the bins l + 32 k.  Bound by the loads'
// L1 wavefronts (one or two per 32 reads) where the spectrum fills the
// device, and by a lane's chain of reads below that: two bins to a lane up to
// kHsLongBins, four above.  Measured on B200 (us, 5 folds; one bin per thread
// with every index formed anew, K = 2, 4): 24,577 bins 4.48, 4.29, 5.60;
// 131,073: 5.19, 4.77, 6.14; 262,145: 7.36, 5.47, 6.40; 524,289: 11.9, 7.81,
// 7.33; 2^20: 22.3, 12.8, 10.4; 2^22: 82.8, 46.7, 36.6.
constexpr size_t kHsLongBins = (size_t)3 << 17;

template <int NH, int K>
__global__ void __launch_bounds__(256) k_harmonic_sum(const float* __restrict__ in, FoldPtrs out,
                                                      unsigned n)
{
    const unsigned warps = gridDim.x * (blockDim.x / 32);
    const unsigned nw = n / (32 * K) + (n % (32 * K) != 0);
    for (unsigned w = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; w < nw; w += warps) {
        const unsigned i = w * (32 * K) + (threadIdx.x & 31);
        // bins of this lane inside the spectrum
        const int take = i >= n ? 0 : (int)min((unsigned)K, (n - 1 - i) / 32 + 1);
        float val[K];
#pragma unroll
        for (int k = 0; k < K; ++k) val[k] = k < take ? in[i + 32 * k] : 0.f;
        auto put = [&](float* o, auto scale) {
#pragma unroll
            for (int k = 0; k < K; ++k)
                if (k < take) o[i + 32 * k] = val[k] * scale;
        };
        add_fractions<1>(in, i, take, val);
        put(out.p[0], rsqrt(2.0));
        if constexpr (NH > 1) {
            add_fractions<2>(in, i, take, val);
            put(out.p[1], 0.5f);  // exact, as the double product is
        }
        if constexpr (NH > 2) {
            add_fractions<3>(in, i, take, val);
            put(out.p[2], rsqrt(8.0));
        }
        if constexpr (NH > 3) {
            add_fractions<4>(in, i, take, val);
            put(out.p[3], 0.25f);
        }
        if constexpr (NH > 4) {
            add_fractions<5>(in, i, take, val);
            put(out.p[4], rsqrt(32.0));
        }
    }
}

// ------------------------------------------------------------- compaction
// Order-preserving stream compaction of (i, x[i]) with x[i] > thresh over
// [start, n) in two kernels.  The bins are cut into one run per CTA (at most
// kPeakRuns, a multiple of 256 bins each) and every run into one part per
// warp.  The first kernel counts per part and per run; in the second a CTA
// adds the counts of the runs before its own and its warps write their
// parts.  Values above a threshold are rare, so most warps read their bins
// once, in the first kernel.  (Counting per 4096 bins, a one-thread scan over
// the tiles and a write that read every tile again took 7 + 10 + 9 us at 2^21
// bins on B200, this 3.6 + 3.7.)
constexpr int kPeakRuns = 1024;
constexpr int kPeakWarps = 8;
constexpr int kPeakInts = kPeakRuns * (1 + kPeakWarps) + 1;  // scratch: runs, parts, total

// The spectra of one launch (grid y): a fold-by-fold search of a trial's
// harmonic sums is one pair of launches and one read-back.
constexpr int kPeakSpectra = 8;
struct PeakJobs {
    const float* x[kPeakSpectra];
    int start[kPeakSpectra], n[kPeakSpectra], run[kPeakSpectra];
    int* counts[kPeakSpectra];  // kPeakInts - 1 of scratch
    int* total[kPeakSpectra];
    int* idx[kPeakSpectra];
    float* val[kPeakSpectra];
};

__global__ void __launch_bounds__(32 * kPeakWarps) k_peaks_count(const __grid_constant__ PeakJobs job,
                                                                 float thresh)
{
    const int sp = blockIdx.y, run = job.run[sp], start = job.start[sp], n = job.n[sp];
    const float* __restrict__ x = job.x[sp];
    int* __restrict__ counts = job.counts[sp];
    const int runs = (int)(((long long)n - start + run - 1) / run);
    if ((int)blockIdx.x >= runs) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x / 32, part = run / kPeakWarps;
    const long long a = start + (long long)blockIdx.x * run + (long long)warp * part;
    const int len = (int)max(0LL, min((long long)part, (long long)n - a));
    const float* p = x + a;
    int c = 0;
#pragma unroll 8
    for (int k = lane; k < len; k += 32) c += p[k] > thresh;
    c = __reduce_add_sync(0xffffffffu, c);
    __shared__ int sh[kPeakWarps];
    if (lane == 0) {
        sh[warp] = c;
        counts[runs + blockIdx.x * kPeakWarps + warp] = c;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int w = 0; w < kPeakWarps; ++w) t += sh[w];
        counts[blockIdx.x] = t;
    }
}

__global__ void __launch_bounds__(32 * kPeakWarps) k_peaks_write(const __grid_constant__ PeakJobs job,
                                                                 float thresh, int cap)
{
    const int sp = blockIdx.y, run = job.run[sp], start = job.start[sp], n = job.n[sp];
    const float* __restrict__ x = job.x[sp];
    const int* __restrict__ counts = job.counts[sp];
    int* __restrict__ idx = job.idx[sp];
    float* __restrict__ val = job.val[sp];
    const int runs = (int)(((long long)n - start + run - 1) / run);
    if ((int)blockIdx.x >= runs) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x / 32, part = run / kPeakWarps;
    const int own = counts[blockIdx.x];
    const bool last = (int)blockIdx.x == runs - 1;
    if (own == 0 && !last) return;
    __shared__ int sh[kPeakWarps];
    int c = 0;  // hits of the runs before this one
    for (int k = threadIdx.x; k < (int)blockIdx.x; k += blockDim.x) c += counts[k];
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) sh[warp] = c;
    __syncthreads();
    int pos = 0;
    for (int w = 0; w < kPeakWarps; ++w) pos += sh[w];
    if (last && threadIdx.x == 0) *job.total[sp] = pos + own;
    const int* parts = counts + runs + blockIdx.x * kPeakWarps;
    for (int w = 0; w < warp; ++w) pos += parts[w];
    int left = parts[warp];
    const long long a = start + (long long)blockIdx.x * run + (long long)warp * part;
    const int len = (int)max(0LL, min((long long)part, (long long)n - a));
    for (int k = 0; k < len && left > 0; k += 32) {
        const int i = k + lane;
        const float v = i < len ? x[a + i] : 0.f;
        const bool hit = i < len && v > thresh;
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (hit) {
            const int at = pos + __popc(m & ((1u << lane) - 1));
            if (at < cap) {
                idx[at] = (int)(a + i);
                val[at] = v;
            }
        }
        pos += __popc(m);
        left -= __popc(m);
    }
}

// Bins per run of [start, n): at least 2048, so that a short spectrum's few
// CTAs have work.
static int peak_run(long long bins)
{
    const long long run = (bins + kPeakRuns - 1) / kPeakRuns;
    return (int)(((run < 2048 ? 2048 : run) + 255) / 256 * 256);
}

// Both kernels over the first `count` spectra of the job (all with n > start).
static int launch_peaks(PeakJobs& job, int count, float thresh, int cap, cudaStream_t s)
{
    unsigned g = 1;
    for (int k = 0; k < count; ++k) {
        const long long bins = (long long)job.n[k] - job.start[k];
        job.run[k] = peak_run(bins);
        g = std::max(g, (unsigned)((bins + job.run[k] - 1) / job.run[k]));
    }
    const dim3 grid(g, (unsigned)count);
    k_peaks_count<<<grid, 32 * kPeakWarps, 0, s>>>(job, thresh);
    k_peaks_write<<<grid, 32 * kPeakWarps, 0, s>>>(job, thresh, cap);
    return launch_status("compaction kernels");
}

// One spectrum; `scratch` holds kPeakInts ints, its last one the total.
static int launch_peaks(const float* d_spec, int n, int start, float thresh, int* scratch,
                        int* d_idx, float* d_val, int cap, cudaStream_t s)
{
    PeakJobs job{};
    job.x[0] = d_spec;
    job.start[0] = start;
    job.n[0] = n;
    job.counts[0] = scratch;
    job.total[0] = scratch + kPeakInts - 1;
    job.idx[0] = d_idx;
    job.val[0] = d_val;
    return launch_peaks(job, 1, thresh, cap, s);
}

}  // namespace psx

using namespace psx;

// =================================================================== C ABI
extern "C" {

const char* psx_last_error(void) { return psx::g_err.c_str(); }

const char* psx_status_string(int st)
{
    switch (st) {
    case PSX_OK: return "ok";
    case PSX_ERR_INVALID: return "invalid argument";
    case PSX_ERR_CUDA: return "CUDA error";
    case PSX_ERR_CUFFT: return "cuFFT error";
    case PSX_ERR_ALLOC: return "allocation failed";
    case PSX_ERR_OVERFLOW: return "output buffer too small";
    case PSX_ERR_UNSUPPORTED: return "unsupported";
    case PSX_ERR_IO: return "I/O error";
    case PSX_ERR_BUSY: return "busy";
    default: return "unknown status";
    }
}

const char* psx_version(void) { return "peasoup_b200 0.1 (sm_100a)"; }

int psx_resampleII(const float* d_in, float* d_out, size_t size, float acc, float tsamp,
                   psx_stream_t stream)
{
    clear_error();
    return launch_resample(d_in, d_out, size, nullptr, accel_fact(acc, tsamp), 1, size, false,
                           cs(stream));
}

int psx_resample(const float* d_in, float* d_out, size_t size, float acc, float tsamp,
                 psx_stream_t stream)
{
    clear_error();
    return launch_resample(d_in, d_out, size, nullptr, accel_fact(acc, tsamp), 1, size, true,
                           cs(stream));
}

int psx_resampleII_batch(const float* d_in, float* d_out, size_t size, const float* h_accs,
                         int ntrials, float tsamp, psx_stream_t stream)
{
    clear_error();
    if (!h_accs || ntrials <= 0 || ntrials > 65535) {
        set_error("resampleII_batch: bad trial list");
        return PSX_ERR_INVALID;
    }
    std::vector<double> k(ntrials);
    for (int t = 0; t < ntrials; ++t) k[t] = accel_fact(h_accs[t], tsamp);
    double* d_k = nullptr;
    PSX_CUDA(scratch_alloc((void**)&d_k, sizeof(double) * ntrials, cs(stream)));
    int rc = cuda_status(cudaMemcpyAsync(d_k, k.data(), sizeof(double) * ntrials,
                                         cudaMemcpyHostToDevice, cs(stream)),
                         "resampleII_batch copy");
    if (rc == PSX_OK)
        rc = launch_resample(d_in, d_out, size, d_k, 0.0, ntrials, size, false, cs(stream));
    cudaFreeAsync(d_k, cs(stream));
    // the host vector must outlive the copy
    if (rc == PSX_OK) rc = cuda_status(cudaStreamSynchronize(cs(stream)), "resampleII_batch");
    return rc;
}

int psx_form_power_series(const float* d_fseries, float* d_out, size_t nbins, int way,
                          psx_stream_t stream)
{
    clear_error();
    if (!d_fseries || !d_out || nbins == 0 || (way != 0 && way != 1)) {
        set_error("form_power_series: bad arguments");
        return PSX_ERR_INVALID;
    }
    const unsigned T = 256;
    const unsigned g = grid_for(nbins / 2 + 1, T);
    if (way == 0)
        k_form<0><<<g, T, 0, cs(stream)>>>(d_fseries, d_out, nbins);
    else
        k_form<1><<<g, T, 0, cs(stream)>>>(d_fseries, d_out, nbins);
    return launch_status("form kernel");
}

int psx_median_scrunch5(const float* d_in, size_t count, float* d_out, psx_stream_t stream)
{
    clear_error();
    if (!d_in || !d_out || count == 0) {
        set_error("median_scrunch5: bad arguments");
        return PSX_ERR_INVALID;
    }
    k_scrunch5<<<grid_for(count / 5 + 1, 256), 256, 0, cs(stream)>>>(d_in, count, d_out);
    return launch_status("scrunch kernel");
}

int psx_linear_stretch(const float* d_in, size_t in_count, float* d_out, size_t out_count,
                       psx_stream_t stream)
{
    clear_error();
    if (!d_in || !d_out || in_count == 0 || out_count < 2 || in_count > 0xffffffffu ||
        out_count > 0xffffffffu) {
        set_error("linear_stretch: bad arguments");
        return PSX_ERR_INVALID;
    }
    k_stretch<<<grid_for(out_count, 256), 256, 0, cs(stream)>>>(
        d_in, (unsigned)in_count, d_out, out_count, stretch_step(in_count, out_count));
    return launch_status("stretch kernel");
}

size_t psx_running_median_scratch_bytes(size_t nbins) { return median_scratch_bytes(nbins); }

int psx_running_median(const float* d_powers, size_t nbins, double bin_width, float b5,
                       float b25, float* d_median, void* d_scratch, psx_stream_t stream)
{
    clear_error();
    if (!d_median) {
        set_error("running_median: null output");
        return PSX_ERR_INVALID;
    }
    return launch_running_median(d_powers, nbins, bin_width, b5, b25, d_median, nullptr,
                                 d_scratch, cs(stream));
}

int psx_divide_c_by_f(float* d_fseries, const float* d_f, size_t nbins, psx_stream_t stream)
{
    clear_error();
    if (!d_fseries || !d_f || nbins == 0) {
        set_error("divide_c_by_f: bad arguments");
        return PSX_ERR_INVALID;
    }
    k_divide_c_by_f<<<grid_for(nbins, 256), 256, 0, cs(stream)>>>(d_fseries, d_f, nbins);
    return launch_status("divide kernel");
}

int psx_deredden(float* d_fseries, const float* d_powers, size_t nbins, double bin_width,
                 float b5, float b25, void* d_scratch, psx_stream_t stream)
{
    clear_error();
    if (!d_fseries) {
        set_error("deredden: null spectrum");
        return PSX_ERR_INVALID;
    }
    return launch_running_median(d_powers, nbins, bin_width, b5, b25, nullptr, d_fseries,
                                 d_scratch, cs(stream));
}

int psx_zap_birdies(float* d_fseries, const float* d_freqs, const float* d_widths,
                    float bin_width, size_t nbirdies, size_t nbins, psx_stream_t stream)
{
    clear_error();
    return launch_zap(d_fseries, d_freqs, d_widths, bin_width, nbirdies, nbins, cs(stream));
}

int psx_read_zaplist(const char* path, float* h_freqs, float* h_widths, size_t cap, size_t* n)
{
    clear_error();
    if (!path || !n) {
        set_error("read_zaplist: null argument");
        return PSX_ERR_INVALID;
    }
    std::ifstream f(path);
    if (!f.good()) {
        set_error("zap list %s could not be opened", path);
        return PSX_ERR_IO;
    }
    // birdiezapper.hpp:35-46: whitespace-separated "freq width" per line,
    // blank lines skipped, numbers parsed as atof does.
    std::string line;
    size_t k = 0;
    while (std::getline(f, line)) {
        std::istringstream ss(line);
        std::string a, b;
        if (!(ss >> a)) continue;
        if (!(ss >> b)) {
            set_error("zap list %s: line without a width: '%s'", path, line.c_str());
            return PSX_ERR_IO;
        }
        if (h_freqs && k < cap) {
            h_freqs[k] = (float)atof(a.c_str());
            h_widths[k] = (float)atof(b.c_str());
        }
        ++k;
    }
    *n = k;
    if (h_freqs && k > cap) {
        set_error("zap list has %zu entries, buffer holds %zu", k, cap);
        return PSX_ERR_OVERFLOW;
    }
    return PSX_OK;
}

int psx_stats(const float* d_x, size_t n, size_t first, float* h_mean, float* h_rms,
              float* h_std, psx_stream_t stream)
{
    clear_error();
    if (!d_x || n <= first) {
        set_error("stats: bad arguments");
        return PSX_ERR_INVALID;
    }
    cudaStream_t s = cs(stream);
    void* scratch = nullptr;
    const int nb = reduction_blocks();
    const size_t bytes = sizeof(double2) * nb + 2 * sizeof(double) + 8 * sizeof(float);
    PSX_CUDA(scratch_alloc(&scratch, bytes, s));
    double2* part = static_cast<double2*>(scratch);
    double* sums = reinterpret_cast<double*>(part + nb);
    float* stat = reinterpret_cast<float*>(sums + 2);
    int rc = launch_stats(d_x, false, first, n, part, sums, stat, 1.0f, s);
    float h[5] = {0, 0, 0, 0, 0};
    if (rc == PSX_OK)
        rc = cuda_status(cudaMemcpyAsync(h, stat, sizeof h, cudaMemcpyDeviceToHost, s), "stats copy");
    cudaFreeAsync(scratch, s);
    if (rc == PSX_OK) rc = cuda_status(cudaStreamSynchronize(s), "stats");
    if (rc == PSX_OK) {
        if (h_mean) *h_mean = h[0];
        if (h_rms) *h_rms = h[1];
        if (h_std) *h_std = h[2];
    }
    return rc;
}

int psx_normalise(float* d_x, float mean, float sigma, size_t n, psx_stream_t stream)
{
    clear_error();
    if (!d_x) {
        set_error("normalise: null pointer");
        return PSX_ERR_INVALID;
    }
    if (n == 0) return PSX_OK;
    if ((reinterpret_cast<uintptr_t>(d_x) & 15u) == 0)
        k_normalise<true><<<grid_for((n + 3) / 4, 256), 256, 0, cs(stream)>>>(d_x, mean, sigma, n);
    else
        k_normalise<false><<<grid_for(n, 256), 256, 0, cs(stream)>>>(d_x, mean, sigma, n);
    return launch_status("normalise kernel");
}

int psx_remove_baseline(float* d_x, size_t n, int* h_passes, psx_stream_t stream)
{
    clear_error();
    if (!d_x || n == 0) {
        set_error("remove_baseline: bad arguments");
        return PSX_ERR_INVALID;
    }
    cudaStream_t s = cs(stream);
    const int nb = reduction_blocks();
    void* scratch = nullptr;
    PSX_CUDA(scratch_alloc(&scratch, sizeof(double2) * 2 * nb + 2 * sizeof(double) + 64, s));
    double2* part = static_cast<double2*>(scratch);
    double* sums = reinterpret_cast<double*>(part + 2 * nb);
    float* d_mean = reinterpret_cast<float*>(sums + 2);
    unsigned* flags = reinterpret_cast<unsigned*>(d_mean + 2);  // as Slot::d_count of the search
    int rc = PSX_OK, count = 0;
    float mean = 0.f;
    bool more = true;
    // reference src/kernels.cu:467-477: do { subtract mean } while
    // (|mean| > 5e-7 n), leaving after the 102nd pass at most.  A series
    // rarely needs more than two passes: those run without the host (three
    // kernels and one read-back, where a pass of its own takes four kernels
    // and a read-back), the loop goes on from there.
    if ((reinterpret_cast<uintptr_t>(d_x) & 15u) == 0) {
        unsigned h[2] = {0, 0};
        rc = launch_partials_v4(d_x, n, part, nullptr, flags + 4, s);
        for (int pass = 0; pass < 2 && rc == PSX_OK; ++pass)
            rc = launch_baseline_pass_v4(d_x, n, part + pass * nb, part + (1 - pass) * nb,
                                         pass ? flags + 6 : flags + 4, flags + 6 + pass, flags + 5,
                                         pass ? flags + 2 : nullptr, pass ? flags + 3 : nullptr, s);
        if (rc == PSX_OK)
            rc = cuda_status(cudaMemcpyAsync(h, flags + 2, sizeof h, cudaMemcpyDeviceToHost, s),
                             "baseline copy");
        if (rc == PSX_OK) rc = cuda_status(cudaStreamSynchronize(s), "baseline");
        more = h[0] != 0;
        count = (int)h[1];
    }
    while (more && rc == PSX_OK) {
        rc = remove_baseline_pass(d_x, n, part, sums, d_mean, s);
        if (rc != PSX_OK) break;
        rc = cuda_status(cudaMemcpyAsync(&mean, d_mean, sizeof(float), cudaMemcpyDeviceToHost, s),
                         "baseline copy");
        if (rc == PSX_OK) rc = cuda_status(cudaStreamSynchronize(s), "baseline");
        if (rc != PSX_OK) break;
        if (count++ > 100) break;
        more = std::fabs(mean) > 5e-7 * (double)n;
    }
    cudaFreeAsync(scratch, s);
    if (h_passes) *h_passes = count;
    return rc;
}

int psx_fill(float* d_x, size_t n, float value, psx_stream_t stream)
{
    clear_error();
    if (!d_x && n) {
        set_error("fill: null pointer");
        return PSX_ERR_INVALID;
    }
    return launch_fill(d_x, n, value, cs(stream));
}

int psx_convert_u8_f32(const uint8_t* d_in, float* d_out, size_t n, psx_stream_t stream)
{
    clear_error();
    if (!d_in || !d_out) {
        set_error("convert: null pointer");
        return PSX_ERR_INVALID;
    }
    if (!n) return PSX_OK;
    k_convert<uint8_t><<<grid_for(n, 256), 256, 0, cs(stream)>>>(d_in, d_out, n);
    return launch_status("convert kernel");
}

int psx_convert_i8_f32(const int8_t* d_in, float* d_out, size_t n, psx_stream_t stream)
{
    clear_error();
    if (!d_in || !d_out) {
        set_error("convert: null pointer");
        return PSX_ERR_INVALID;
    }
    if (!n) return PSX_OK;
    k_convert<int8_t><<<grid_for(n, 256), 256, 0, cs(stream)>>>(d_in, d_out, n);
    return launch_status("convert kernel");
}

int psx_harmonic_sum(const float* d_in, float* const* h_out_ptrs, size_t n, int nharms,
                     psx_stream_t stream)
{
    clear_error();
    if (!d_in || n == 0 || n > 0x7fffffffu || nharms < 0 || nharms > 5 ||
        (nharms && !h_out_ptrs)) {
        set_error("harmonic_sum: bad arguments (nharms must be 0..5)");
        return PSX_ERR_INVALID;
    }
    if (nharms == 0) return PSX_OK;
    FoldPtrs o{};
    for (int h = 0; h < nharms; ++h) {
        if (!h_out_ptrs[h]) {
            set_error("harmonic_sum: null output %d", h);
            return PSX_ERR_INVALID;
        }
        o.p[h] = h_out_ptrs[h];
    }
    cudaStream_t s = cs(stream);
    auto go = [&](auto two, auto four) {
        if (n <= kHsLongBins)
            two<<<grid_for((n + 1) / 2, 256), 256, 0, s>>>(d_in, o, (unsigned)n);
        else
            four<<<grid_for((n + 3) / 4, 256), 256, 0, s>>>(d_in, o, (unsigned)n);
    };
    switch (nharms) {
    case 1: go(k_harmonic_sum<1, 2>, k_harmonic_sum<1, 4>); break;
    case 2: go(k_harmonic_sum<2, 2>, k_harmonic_sum<2, 4>); break;
    case 3: go(k_harmonic_sum<3, 2>, k_harmonic_sum<3, 4>); break;
    case 4: go(k_harmonic_sum<4, 2>, k_harmonic_sum<4, 4>); break;
    default: go(k_harmonic_sum<5, 2>, k_harmonic_sum<5, 4>); break;
    }
    return launch_status("harmonic sum kernel");
}

int psx_find_peaks(const float* d_spec, int n, int start, float thresh, int* d_idx,
                   float* d_val, int cap, int* h_count, psx_stream_t stream)
{
    clear_error();
    if (!d_spec || !h_count || (cap > 0 && (!d_idx || !d_val))) {
        set_error("find_peaks: bad arguments");
        return PSX_ERR_INVALID;
    }
    if (start < 0) start = 0;
    *h_count = 0;
    if (n <= start) return PSX_OK;
    cudaStream_t s = cs(stream);
    int* scratch = nullptr;
    PSX_CUDA(scratch_alloc((void**)&scratch, sizeof(int) * kPeakInts, s));
    int rc = launch_peaks(d_spec, n, start, thresh, scratch, d_idx, d_val, cap, s);
    int total = 0;
    if (rc == PSX_OK)
        rc = cuda_status(cudaMemcpyAsync(&total, scratch + kPeakInts - 1, sizeof(int),
                                         cudaMemcpyDeviceToHost, s), "find_peaks copy");
    cudaFreeAsync(scratch, s);
    if (rc == PSX_OK) rc = cuda_status(cudaStreamSynchronize(s), "find_peaks");
    if (rc != PSX_OK) return rc;
    *h_count = total;
    if (total > cap) {
        set_error("find_peaks: %d values above threshold, buffer holds %d", total, cap);
        return PSX_ERR_OVERFLOW;
    }
    return PSX_OK;
}

int psx_find_peaks_host(const float* const* d_specs, const int* n, const int* start, int nspec,
                        float thresh, int* h_idx, float* h_val, int cap, int* h_counts,
                        psx_stream_t stream)
{
    clear_error();
    if (!d_specs || !n || !start || nspec < 1 || nspec > kPeakSpectra || !h_counts || cap < 0 ||
        (cap > 0 && (!h_idx || !h_val))) {
        set_error("find_peaks_host: bad arguments (1 to %d spectra)", kPeakSpectra);
        return PSX_ERR_INVALID;
    }
    for (int k = 0; k < nspec; ++k)
        if (!d_specs[k]) {
            set_error("find_peaks_host: null spectrum %d", k);
            return PSX_ERR_INVALID;
        }
    cudaStream_t s = cs(stream);
    // the counts and the first kFirst peaks of every spectrum come back in
    // one copy: per spectrum [total, idx[kFirst], val[kFirst]]
    constexpr int kFirst = 512, kRow = 1 + 2 * kFirst;
    PeakJobs job{};
    int which[kPeakSpectra], count = 0;
    for (int k = 0; k < nspec; ++k) {
        h_counts[k] = 0;
        const int st = std::max(0, start[k]);
        if (n[k] <= st) continue;
        which[count] = k;
        job.x[count] = d_specs[k];
        job.start[count] = st;
        job.n[count] = n[k];
        ++count;
    }
    if (!count) return PSX_OK;
    int* scratch = nullptr;
    PSX_CUDA(scratch_alloc((void**)&scratch,
                           sizeof(int) * (size_t)count * (kPeakInts - 1 + kRow), s));
    int* back = scratch + (size_t)count * (kPeakInts - 1);  // the rows read back
    for (int c = 0; c < count; ++c) {
        job.counts[c] = scratch + (size_t)c * (kPeakInts - 1);
        job.total[c] = back + c * kRow;
        job.idx[c] = job.total[c] + 1;
        job.val[c] = reinterpret_cast<float*>(job.idx[c] + kFirst);
    }
    int h[kPeakSpectra * kRow];
    int rc = launch_peaks(job, count, thresh, kFirst, s);
    if (rc == PSX_OK)
        rc = cuda_status(cudaMemcpyAsync(h, back, sizeof(int) * (size_t)count * kRow,
                                         cudaMemcpyDeviceToHost, s), "find_peaks_host copy");
    cudaFreeAsync(scratch, s);
    if (rc == PSX_OK) rc = cuda_status(cudaStreamSynchronize(s), "find_peaks_host");
    if (rc != PSX_OK) return rc;
    int most = 0;
    for (int c = 0; c < count; ++c) most = std::max(most, h_counts[which[c]] = h[c * kRow]);
    if (most > cap) {
        set_error("find_peaks_host: %d values above threshold, buffer holds %d", most, cap);
        return PSX_ERR_OVERFLOW;
    }
    for (int c = 0; c < count; ++c) {
        const int k = which[c], total = h_counts[k];
        int* oi = h_idx + (size_t)k * cap;
        float* ov = h_val + (size_t)k * cap;
        if (total <= kFirst) {
            std::memcpy(oi, h + c * kRow + 1, sizeof(int) * total);
            std::memcpy(ov, h + c * kRow + 1 + kFirst, sizeof(float) * total);
            continue;
        }
        // more than came back: this spectrum again, into a buffer of its size
        PSX_CUDA(scratch_alloc((void**)&scratch, sizeof(int) * (kPeakInts + 2 * (size_t)total), s));
        int* d_idx = scratch + kPeakInts;
        float* d_val = reinterpret_cast<float*>(d_idx + total);
        rc = launch_peaks(job.x[c], job.n[c], job.start[c], thresh, scratch, d_idx, d_val, total, s);
        if (rc == PSX_OK)
            rc = cuda_status(cudaMemcpyAsync(oi, d_idx, sizeof(int) * total,
                                             cudaMemcpyDeviceToHost, s), "find_peaks_host copy");
        if (rc == PSX_OK)
            rc = cuda_status(cudaMemcpyAsync(ov, d_val, sizeof(float) * total,
                                             cudaMemcpyDeviceToHost, s), "find_peaks_host copy");
        cudaFreeAsync(scratch, s);
        if (rc == PSX_OK) rc = cuda_status(cudaStreamSynchronize(s), "find_peaks_host");
        if (rc != PSX_OK) return rc;
    }
    return PSX_OK;
}

}  // extern "C"

// ------------------------------------------------- peak finding, no allocation
// psx_find_peaks_noalloc runs the two compaction kernels of psx_find_peaks
// with their counts in a fixed device array instead of memory from
// cudaMallocAsync.  It serves callers that may not allocate device memory
// while they search: hosts that have handed the whole of a GPU's memory to
// their own pool or to another framework, hosts that forbid allocation
// after start-up so that memory use cannot grow during a run, and code
// running where an allocation could block or fail at a bad moment.
//
// The array g_peak_tile_scratch is compiled into this library: every GPU
// that loads the library holds its 256 KiB (+ 4 bytes) until the process
// exits.  A call may scan at most 2^28 bins (n - start), the documented limit
// of the entry point (one count per 4096 bins would fill the array; the
// kernels need kPeakInts ints of it).  All calls on a device share the one
// array and it keeps the last call's contents; nothing in it needs to start
// at zero, because k_peaks_count writes every count a call uses before
// k_peaks_write reads it.  Calls whose GPU work overlaps (other streams, other host
// threads) race on the array and give wrong results.
namespace psx {
namespace {

constexpr int kNoAllocMaxTiles = 65536;
constexpr long long kNoAllocMaxBins = (long long)kNoAllocMaxTiles * 4096;
static_assert(kPeakInts <= kNoAllocMaxTiles + 1, "static scratch");
constexpr int kNoAllocMaxDevices = 64;

// Device-side storage.  In host code this name is only a handle for the
// runtime's symbol lookup, never a pointer that can be dereferenced or
// passed to a kernel.
static __device__ __align__(256) int g_peak_tile_scratch[kNoAllocMaxTiles + 1];

std::mutex g_peak_scratch_mu;
int* g_peak_scratch_addr[kNoAllocMaxDevices] = {nullptr};

// The device address of g_peak_tile_scratch on the current device, looked
// up once per device (the first call on each device does it, with that
// device current) and cached.
int peak_scratch_address(int** out)
{
    int dev = -1;
    PSX_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNoAllocMaxDevices) {
        set_error("find_peaks_noalloc: device ordinal %d outside 0..%d", dev,
                  kNoAllocMaxDevices - 1);
        return PSX_ERR_UNSUPPORTED;
    }
    std::lock_guard<std::mutex> lock(g_peak_scratch_mu);
    if (!g_peak_scratch_addr[dev]) {
        void* p = nullptr;
        PSX_CUDA(cudaGetSymbolAddress(&p, g_peak_tile_scratch));
        if (!p) {
            set_error("find_peaks_noalloc: no device address for the scratch array");
            return PSX_ERR_CUDA;
        }
        g_peak_scratch_addr[dev] = static_cast<int*>(p);
    }
    *out = g_peak_scratch_addr[dev];
    return PSX_OK;
}

}  // namespace
}  // namespace psx

extern "C" int psx_find_peaks_noalloc(const float* d_spec, int n, int start, float thresh,
                                      int* d_idx, float* d_val, int cap, int* h_count,
                                      psx_stream_t stream)
{
    clear_error();
    if (!d_spec || !h_count || (cap > 0 && (!d_idx || !d_val))) {
        set_error("find_peaks_noalloc: bad arguments");
        return PSX_ERR_INVALID;
    }
    if (start < 0) start = 0;
    *h_count = 0;
    if (n <= start) return PSX_OK;
    if ((long long)n - start > kNoAllocMaxBins) {
        set_error("find_peaks_noalloc: %lld bins to scan, the static scratch holds at most %lld "
                  "(use psx_find_peaks)", (long long)n - start, kNoAllocMaxBins);
        return PSX_ERR_INVALID;
    }
    int* scratch = nullptr;
    int rc = peak_scratch_address(&scratch);
    if (rc != PSX_OK) return rc;
    cudaStream_t s = cs(stream);
    rc = launch_peaks(d_spec, n, start, thresh, scratch, d_idx, d_val, cap, s);
    int total = 0;
    if (rc == PSX_OK)
        rc = cuda_status(cudaMemcpyAsync(&total, scratch + kPeakInts - 1, sizeof(int),
                                         cudaMemcpyDeviceToHost, s), "find_peaks_noalloc copy");
    if (rc == PSX_OK) rc = cuda_status(cudaStreamSynchronize(s), "find_peaks_noalloc");
    if (rc != PSX_OK) return rc;
    *h_count = total;
    if (total > cap) {
        set_error("find_peaks_noalloc: %d values above threshold, buffer holds %d", total, cap);
        return PSX_ERR_OVERFLOW;
    }
    return PSX_OK;
}
