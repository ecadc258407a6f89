// psx_dedisp.cu -- direct incoherent dedispersion of SIGPROC sample rows
// into device-resident series: the producer of the search's input.
//
// The reference calls the external dedisp library through Dedisperser
// (include/transforms/dedisperser.hpp:13-188) and copies every dedispersed
// series back to the host, from where each Worker copies one series at a
// time to the device again (src/pipeline_multi.cu:474-505, 166-170).  Here
// the sample rows are unpacked once into a channel-major layout in HBM and
// the dedispersed block is written where the search reads it.
//
// Arithmetic (the published direct algorithm; dedisp itself is absent):
//   delay_c  = 4.15e3/tsamp * (f_c^-2 - fch1^-2)   samples per unit DM
//   D(d, c)  = round-half-even(float(dm_d * delay_c))
//   sum[d,t] = sum over live channels of x_c[t + D(d, c)]  (exact integer)
//   out[d,t] = sum, or (sum - nchans*m/2) * 1/(m*sqrt(nchans)) + 1/2.
//
// Layout.  cm[c][t]: one row of `pitch` samples (u8 for 1..8-bit input, u16
// for 16-bit) per channel, so that every (channel, time window) a CTA needs
// is one contiguous run.  A CTA owns 8 DM trials (one per warp) and 512
// output samples; per channel it stages the window the 8 trials need,
// [t0 + min D, t0 + 512 + max D), with cp.async in double-buffered chunks of
// channels, then each lane adds 16 outputs per channel from shared memory:
// two aligned 32-bit loads, one funnel shift, and (8-bit samples) two byte
// permutes into packed 16-bit accumulators.  Consecutive CTAs take the same
// time tile for successive DM blocks, so the window is read from HBM once
// and from L2 after that.  Where the DM trials of a block share most of their
// relative shifts, subband sums formed once serve all of them instead
// (k_dedisperse_tree, below, with the rule at kDedispWeights).
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <new>
#include <vector>

#include "psx_common.cuh"

namespace psx {
namespace {

constexpr int kDdThreads = 256;
constexpr int kDdWarps = 8;    // DM trials per CTA
constexpr int kDdTile8 = 1024; // output samples per CTA, 1..8-bit samples
constexpr int kDdTile16 = 512; // output samples per CTA, 16-bit samples
inline int dd_tile(int elem) { return elem == 1 ? kDdTile8 : kDdTile16; }
constexpr int kUpRows = 64;    // unpack tile: samples
constexpr int kUpThreads = 256;
constexpr float kDmConst = 4.15e3f;
constexpr size_t kDdMaxSmem = 220 * 1024;  // dynamic shared memory of a launch at most

template <int NBITS> struct Sample { using T = uint8_t; };
template <> struct Sample<16> { using T = uint16_t; };

// A SIGPROC row: below 8 bits the first channel sits in the least significant
// bits of its byte; 16-bit samples are little-endian.
//
// Rows [r0, r0 + nrows) of the packed input (rows[0] is row r0) become
// columns of cm; columns [r0 + nrows, r0 + ncols) are zeroed.  One CTA per
// 64 samples x the channels of 64 bytes of a row (64 channels at 16 bits);
// every store is 16 bytes.  r0 and ncols' rounding to 64 stay inside the
// pitch.
//
// A thread takes one 32-bit word of four consecutive rows, splits it into
// bytes of one channel class each (1, 2 or 4 bits: shift and mask) and turns
// 4 channels x 4 samples around with eight byte permutes, so the tile is
// written a word (four samples of a channel) at a time.  The words of a
// channel are XOR-ed by the row word's index, so that neither side's accesses
// meet in a bank more than twice.  Where rows do not start on 4-byte
// boundaries (vec 0) the words are put together from bytes.  (Writing the
// tile a byte at a time, 64 samples x 64 channels, took 146 us for 2^22
// samples x 64 channels of 8 bits on B200 and 234 for 400,000 x 1024 of 4
// bits; this takes 121 and 136, 4.5 TB/s.)
template <int NBITS>
struct UnpackTile {
    static constexpr int kElem = NBITS == 16 ? 2 : 1;
    static constexpr int kWords = NBITS == 16 ? 32 : 16;         // of a row's segment
    static constexpr int kPer = 32 / NBITS;                      // channels of a word
    static constexpr int kChans = kWords * kPer;
    static constexpr int kChanWords = kUpRows * kElem / 4;       // of a channel's samples
};

template <int NBITS>
__global__ void __launch_bounds__(kUpThreads) k_unpack_chanmajor(
    const uint8_t* __restrict__ rows, size_t row_bytes, size_t nrows, size_t r0, size_t ncols,
    int nchans, typename Sample<NBITS>::T* __restrict__ cm, size_t pitch, int vec)
{
    using U = UnpackTile<NBITS>;
    __shared__ __align__(16) uint32_t tile[U::kChans * U::kChanWords];
    const size_t col0 = (size_t)blockIdx.x * kUpRows;
    const int c0 = blockIdx.y * U::kChans;
    const size_t seg = (size_t)c0 * NBITS / 8;  // first byte of the CTA's part of a row
    constexpr int kRows = NBITS == 16 ? 2 : 4;  // rows of a thread's step: one word of samples
    const int words = (int)min((size_t)U::kWords, (row_bytes - seg + 3) / 4);
    bool turned = false;
    if constexpr (NBITS == 16) {
        // Two rows a step give a thread four steps: for a whole tile of rows
        // of whole words all their loads first (400,000 x 64 on B200: 28.8 us
        // step by step, 18.7; 40,000 x 64: 6.1, 4.1).
        if (vec && words == U::kWords && col0 + kUpRows <= nrows) {
            constexpr int kSteps = (kUpRows / kRows) * U::kWords / kUpThreads;
            const int q = threadIdx.x % U::kWords, g0 = threadIdx.x / U::kWords;
            const uint8_t* p = rows + (col0 + kRows * g0) * row_bytes + seg + 4 * q;
            const size_t step = (size_t)(kRows * (kUpThreads / U::kWords)) * row_bytes;
            uint32_t w[kSteps][kRows];
#pragma unroll
            for (int j = 0; j < kSteps; ++j)
#pragma unroll
                for (int r = 0; r < kRows; ++r)
                    w[j][r] = *reinterpret_cast<const uint32_t*>(p + j * step + r * row_bytes);
            uint32_t* t = tile + (q * U::kPer) * U::kChanWords;
#pragma unroll
            for (int j = 0; j < kSteps; ++j) {
                const int at = (g0 + j * (kUpThreads / U::kWords)) ^ (q & (U::kChanWords - 1));
                t[at] = __byte_perm(w[j][0], w[j][1], 0x5410);
                t[U::kChanWords + at] = __byte_perm(w[j][0], w[j][1], 0x7632);
            }
            turned = true;
        }
    }
    for (int i = threadIdx.x; !turned && i < (kUpRows / kRows) * words; i += blockDim.x) {
        const int q = i % words, g = i / words;  // row word, group of rows
        const size_t byte = seg + 4 * (size_t)q;
        uint32_t w[kRows];
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            const size_t rr = col0 + kRows * g + r;
            w[r] = 0;
            if (rr < nrows && byte < row_bytes) {
                const uint8_t* p = rows + rr * row_bytes + byte;
                if (vec) {
                    w[r] = *reinterpret_cast<const uint32_t*>(p);
                } else {
                    for (int k = 0; k < 4; ++k)
                        if (byte + k < row_bytes) w[r] |= (uint32_t)p[k] << (8 * k);
                }
            }
        }
        uint32_t* t = tile + (q * U::kPer) * U::kChanWords;
        const int at = g ^ (q & (U::kChanWords - 1));
        if constexpr (NBITS == 16) {
            t[at] = __byte_perm(w[0], w[1], 0x5410);
            t[U::kChanWords + at] = __byte_perm(w[0], w[1], 0x7632);
        } else {
            // class k: channels k, k + kPer/4, ... of the word, one per byte
            constexpr int kClasses = U::kPer / 4;
            constexpr uint32_t kMask = 0x01010101u * ((1u << NBITS) - 1u);
#pragma unroll
            for (int k = 0; k < kClasses; ++k) {
                uint32_t b[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) b[r] = NBITS == 8 ? w[r] : (w[r] >> (NBITS * k)) & kMask;
                const uint32_t l0 = __byte_perm(b[0], b[1], 0x5140), l1 = __byte_perm(b[2], b[3], 0x5140);
                const uint32_t h0 = __byte_perm(b[0], b[1], 0x7362), h1 = __byte_perm(b[2], b[3], 0x7362);
                // byte j of a word holds its channel j * kClasses + k
                t[(0 * kClasses + k) * U::kChanWords + at] = __byte_perm(l0, l1, 0x5410);
                t[(1 * kClasses + k) * U::kChanWords + at] = __byte_perm(l0, l1, 0x7632);
                t[(2 * kClasses + k) * U::kChanWords + at] = __byte_perm(h0, h1, 0x5410);
                t[(3 * kClasses + k) * U::kChanWords + at] = __byte_perm(h0, h1, 0x7632);
            }
        }
    }
    __syncthreads();
    constexpr int kPer16 = U::kChanWords / 4;  // 16-byte stores per channel
    constexpr int kVec = 16 / U::kElem;        // samples of one
    const int chans = min(U::kChans, nchans - c0);
    for (int i = threadIdx.x; i < chans * kPer16; i += blockDim.x) {
        const int c = i / kPer16, v = i % kPer16, x = (c / U::kPer) & (U::kChanWords - 1);
        if (col0 + (size_t)v * kVec >= ncols) continue;
        // words 4 v + 0..3 lie at (4 v + j) ^ x: one 16-byte group, its words XOR-ed
        uint4 w = *reinterpret_cast<const uint4*>(tile + c * U::kChanWords + ((4 * v) ^ (x & ~3)));
        if (x & 1) w = make_uint4(w.y, w.x, w.w, w.z);
        if (x & 2) w = make_uint4(w.z, w.w, w.x, w.y);
        *reinterpret_cast<uint4*>(cm + (size_t)(c0 + c) * pitch + r0 + col0 + (size_t)v * kVec) = w;
    }
}

struct DedispArgs {
    const void* cm;
    size_t pitch;           // samples per channel row of cm
    const int* chan;        // [nlive] channel row of each live channel
    const int* lo;          // [ngroups * nlive] window start after t0 (samples)
    const int* off;         // [ndm_pad * nlive] D(d, c) - lo(group of d, c)
    int nlive, ndm, nblk, cc, lwin, group;
    float* out;
    size_t out_pitch, nout;
    float mid, scale;
    int raw;
    int p8, p16;            // channels a byte / a 16-bit sum holds at the input's largest value
    unsigned tile0;         // first output tile of the launch
};

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem)
{
    unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ uint32_t lds32(uint32_t addr)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(v) : "r"(addr));
    return v;
}
template <int OFF>
__device__ __forceinline__ uint32_t lds32o(uint32_t addr)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1+%2];\n" : "=r"(v) : "r"(addr), "n"(OFF));
    return v;
}

__device__ __forceinline__ float map_sum(unsigned s, float mid, float scale, int raw)
{
    float v = (float)s;
    if (!raw) v = __fadd_rn(__fmul_rn(__fsub_rn(v, mid), scale), 0.5f);
    return v;
}

template <typename T, bool FLUSH, bool SMALL>
__global__ void __launch_bounds__(kDdThreads) k_dedisperse(DedispArgs a)
{
    extern __shared__ __align__(16) uint8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int blk = blockIdx.x % a.nblk;
    constexpr int kTile = sizeof(T) == 1 ? kDdTile8 : kDdTile16;
    const size_t t0 = (size_t)(a.tile0 + blockIdx.x / a.nblk) * kTile;
    const int d = blk * kDdWarps + warp;
    const int nwin = kDdWarps / a.group;
    const int gw = warp / a.group;
    const int gbase = blk * kDdWarps / a.group;
    const int win_bytes = a.lwin * (int)sizeof(T);
    const int stage_bytes = a.cc * nwin * win_bytes;
    int* s_off = reinterpret_cast<int*>(smem + 2 * stage_bytes);  // [2][8][cc]
    const int nq = (a.nlive + a.cc - 1) / a.cc;

    auto load_chunk = [&](int q, int st) {
        for (int w = warp; w < a.cc * nwin; w += kDdWarps) {
            int j = w / nwin, g = w % nwin, i = q * a.cc + j;
            if (i >= a.nlive) continue;
            const uint8_t* src = static_cast<const uint8_t*>(a.cm) +
                ((size_t)a.chan[i] * a.pitch + t0 + a.lo[(size_t)(gbase + g) * a.nlive + i]) * sizeof(T);
            uint8_t* dst = smem + st * stage_bytes + w * win_bytes;
            for (int p = lane; p < win_bytes / 16; p += 32) cp_async16(dst + 16 * p, src + 16 * p);
        }
        for (int k = threadIdx.x; k < kDdWarps * a.cc; k += kDdThreads) {
            int ww = k / a.cc, j = k % a.cc, i = q * a.cc + j, dd = blk * kDdWarps + ww;
            s_off[(st * kDdWarps + ww) * a.cc + j] =
                (i < a.nlive && dd < a.ndm) ? a.off[(size_t)dd * a.nlive + i] : 0;
        }
        cp_async_commit();
    };

    const bool active = d < a.ndm;
    float* out = a.out + (size_t)(active ? d : 0) * a.out_pitch;

    if constexpr (sizeof(T) == 1) {
        // lane: outputs t0 + 4*lane + 128*k + {0..3}, k = 0..7, as packed
        // 16-bit pairs; with more channels than a pair holds (p16: 257 at
        // 8 bits) a pair is flushed into 32-bit sums before it can overflow.
        // SMALL (samples of at most 4 bits): the four bytes of a word are
        // summed as they stand, p8 channels at a time (17 at 4 bits, 85 at
        // 2, 255 at 1), before they are spread into the 16-bit pairs.
        constexpr int kUnits = kDdTile8 / 128;
        uint32_t acc[2 * kUnits];
        uint32_t a8[SMALL ? kUnits : 1];
#pragma unroll
        for (int k = 0; k < (SMALL ? kUnits : 1); ++k) a8[k] = 0;
        int since8 = 0;
        // 32-bit sums behind the packed pairs, in shared memory (touched once
        // per 257 channels): s_full[k * 256 + thread], after the offsets
        uint32_t* s_full = reinterpret_cast<uint32_t*>(
            smem + 2 * stage_bytes + 2 * kDdWarps * a.cc * (int)sizeof(int));
#pragma unroll
        for (int k = 0; k < 2 * kUnits; ++k) acc[k] = 0;
        if constexpr (FLUSH) {
#pragma unroll
            for (int k = 0; k < 4 * kUnits; ++k) s_full[k * kDdThreads + threadIdx.x] = 0;
        }
        int since = 0;
        const uint32_t s_base = (uint32_t)__cvta_generic_to_shared(smem);
        const uint32_t s_offs = s_base + 2u * stage_bytes + (uint32_t)warp * a.cc * 4u;
        const uint32_t wstep = (uint32_t)(nwin * win_bytes);
        load_chunk(0, 0);
        for (int q = 0; q < nq; ++q) {
            if (q + 1 < nq) { load_chunk(q + 1, (q + 1) & 1); cp_async_wait<1>(); }
            else cp_async_wait<0>();
            __syncthreads();
            const int st = q & 1;
            const int nj = min(a.cc, a.nlive - q * a.cc);
            if (active) {
                if constexpr (SMALL) {
                    if (since8 + nj > a.p8) {
#pragma unroll
                        for (int k = 0; k < kUnits; ++k) {
                            acc[2 * k] += __byte_perm(a8[k], 0, 0x4140);
                            acc[2 * k + 1] += __byte_perm(a8[k], 0, 0x4342);
                            a8[k] = 0;
                        }
                        since8 = 0;
                    }
                    since8 += nj;
                }
                if constexpr (FLUSH) {
                    if (since + nj > a.p16) {
                        if constexpr (SMALL) {
#pragma unroll
                            for (int k = 0; k < kUnits; ++k) {
                                acc[2 * k] += __byte_perm(a8[k], 0, 0x4140);
                                acc[2 * k + 1] += __byte_perm(a8[k], 0, 0x4342);
                                a8[k] = 0;
                            }
                            since8 = nj;
                        }
#pragma unroll
                        for (int k = 0; k < 2 * kUnits; ++k) {
                            s_full[(2 * k) * kDdThreads + threadIdx.x] += acc[k] & 0xffffu;
                            s_full[(2 * k + 1) * kDdThreads + threadIdx.x] += acc[k] >> 16;
                            acc[k] = 0;
                        }
                        since = 0;
                    }
                    since += nj;
                }
                uint32_t wa = s_base + (uint32_t)(st * stage_bytes + gw * win_bytes) + 4u * lane;
                const uint32_t oa = s_offs + (uint32_t)st * kDdWarps * a.cc * 4u;
#pragma unroll 2
                for (int j = 0; j < nj; ++j, wa += wstep) {
                    const int o = (int)lds32(oa + 4u * j);
                    const uint32_t ad = wa + (uint32_t)(o & ~3);
                    const uint32_t sh = (uint32_t)(o & 3) << 3;
#define PSX_DD_STEP(k)                                                            \
                    {                                                             \
                        uint32_t v = __funnelshift_r(lds32o<128 * (k)>(ad),       \
                                                     lds32o<128 * (k) + 4>(ad), sh); \
                        if constexpr (SMALL) {                                    \
                            a8[(k)] += v;                                         \
                        } else {                                                  \
                            acc[2 * (k)] += __byte_perm(v, 0, 0x4140);            \
                            acc[2 * (k) + 1] += __byte_perm(v, 0, 0x4342);        \
                        }                                                         \
                    }
                    PSX_DD_STEP(0)
                    PSX_DD_STEP(1)
                    PSX_DD_STEP(2)
                    PSX_DD_STEP(3)
                    PSX_DD_STEP(4)
                    PSX_DD_STEP(5)
                    PSX_DD_STEP(6)
                    PSX_DD_STEP(7)
#undef PSX_DD_STEP
                }
            }
            __syncthreads();
        }
        if (!active) return;
        if constexpr (SMALL) {
#pragma unroll
            for (int k = 0; k < kUnits; ++k) {
                acc[2 * k] += __byte_perm(a8[k], 0, 0x4140);
                acc[2 * k + 1] += __byte_perm(a8[k], 0, 0x4342);
            }
        }
#pragma unroll
        for (int k = 0; k < kUnits; ++k) {
            uint32_t s0 = acc[2 * k] & 0xffffu, s1 = acc[2 * k] >> 16;
            uint32_t s2 = acc[2 * k + 1] & 0xffffu, s3 = acc[2 * k + 1] >> 16;
            if constexpr (FLUSH) {
                s0 += s_full[(4 * k) * kDdThreads + threadIdx.x];
                s1 += s_full[(4 * k + 1) * kDdThreads + threadIdx.x];
                s2 += s_full[(4 * k + 2) * kDdThreads + threadIdx.x];
                s3 += s_full[(4 * k + 3) * kDdThreads + threadIdx.x];
            }
            size_t t = t0 + 4 * lane + 128 * k;
            float4 v = make_float4(map_sum(s0, a.mid, a.scale, a.raw),
                                   map_sum(s1, a.mid, a.scale, a.raw),
                                   map_sum(s2, a.mid, a.scale, a.raw),
                                   map_sum(s3, a.mid, a.scale, a.raw));
            if (t + 3 < a.nout) {
                *reinterpret_cast<float4*>(out + t) = v;
            } else {
                if (t < a.nout) out[t] = v.x;
                if (t + 1 < a.nout) out[t + 1] = v.y;
                if (t + 2 < a.nout) out[t + 2] = v.z;
            }
        }
    } else {
        // 16-bit samples: lane outputs t0 + 2*lane + 64*k + {0, 1}, k = 0..7
        uint32_t full[16] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
        load_chunk(0, 0);
        for (int q = 0; q < nq; ++q) {
            if (q + 1 < nq) { load_chunk(q + 1, (q + 1) & 1); cp_async_wait<1>(); }
            else cp_async_wait<0>();
            __syncthreads();
            const int st = q & 1;
            const int nj = min(a.cc, a.nlive - q * a.cc);
            if (active) {
                const uint8_t* wbase = smem + st * stage_bytes + gw * win_bytes;
                const int* offs = s_off + (st * kDdWarps + warp) * a.cc;
                for (int j = 0; j < nj; ++j) {
                    const uint32_t* w = reinterpret_cast<const uint32_t*>(wbase + j * nwin * win_bytes);
                    const int o = offs[j] + 2 * lane;
                    const int sh = (o & 1) * 16;
                    const int wi = o >> 1;
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        uint32_t v = __funnelshift_r(w[wi + 32 * k], w[wi + 32 * k + 1], sh);
                        full[2 * k] += v & 0xffffu;
                        full[2 * k + 1] += v >> 16;
                    }
                }
            }
            __syncthreads();
        }
        if (!active) return;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            size_t t = t0 + 2 * lane + 64 * k;
            float2 v = make_float2(map_sum(full[2 * k], a.mid, a.scale, a.raw),
                                   map_sum(full[2 * k + 1], a.mid, a.scale, a.raw));
            if (t + 1 < a.nout) *reinterpret_cast<float2*>(out + t) = v;
            else if (t < a.nout) out[t] = v.x;
        }
    }
}

// ---------------------------------------------------------------------------
// Shared partial sums.  The shifts of neighbouring DM trials differ by almost
// the same amount in neighbouring channels: over S consecutive live channels
// (a subband) the relative shifts D(d, c) - D(d, c0) of a block of up to 32 DM
// trials take only a few distinct values (2 per pair of channels, 4 to 6 per
// four at survey spacing).  So a CTA first forms, once per distinct vector
// ("pattern") of relative shifts, the subband's own series
//   Y[i] = sum over the S channels of x_c[t0 + smin + i + D(d,c) - D(d,c0)],
// and each DM trial then adds one Y per subband instead of S channels.  The
// sums are integers, so the result is the direct kernel's bit for bit.
//
// Layout.  A tile is 4Q outputs (2Q for 16-bit samples), Q = 256.  A staged
// channel window is rearranged in shared memory into words
// (x[i], x[i+Q], x[i+2Q], x[i+3Q]) ((x[i], x[i+Q]) for 16-bit samples), and a
// pattern's Y is kept in the same arrangement: for 1..4-bit samples the same
// words (the sum of four channels fits a byte), for 8-bit samples pairs of
// words ((y[i], y[i+2Q]), (y[i+Q], y[i+3Q])) of 16-bit sums, for 16-bit
// samples pairs (y[i], y[i+Q]) of 32-bit sums.  Every shift is then a whole
// number of words, so no load needs a funnel shift and a warp's loads are
// consecutive.
//
// Bound: the shared-memory port (71 % of its wavefronts at 8 bits, 64 % at 4;
// 45 % of the shared-memory ones the second level's, 2 bytes per output,
// subband and DM trial) and issue (67 %, 69 %).  Measured on B200 (us, the whole call, channel by channel and so):
// 256 DM trials x 2^22 samples x 64 channels, 8 bits: 6311, 3033; 100 x
// 400,000 x 1024, 4 bits: 3408, 1680.  Subbands of 8 channels have three times the
// patterns; blocks of 64 DM trials leave half the warps.
constexpr int kTrQ = 256;      // words of a row per (DM trial, YE or YO)
constexpr int kTrWords = kTrQ / 32;
// 16 warps of at most 64 registers, two CTAs to an SM (8 warps of 4 DM trials
// each, the same work in half the warps, took 3407 us against 3162)
constexpr int kTrThreads = 512;
constexpr int kTrWarps = 16;
constexpr int kTrMaxDms = 32;  // DM trials per CTA: at most 2 per warp
constexpr int kTrMinDms = 8;   // fewer take the direct form (kDedispWeights)
// sample classes: 8-bit bytes (their sums need 16 bits at once), 1..4-bit
// bytes (a subband's sum fits a byte), 16-bit samples (32-bit sums)
enum { kTr8 = 0, kTrSmall = 1, kTr16 = 2 };
constexpr int kTrS = 4;        // channels per subband
constexpr int kTrRec = 8;      // ints of a pattern's record (32-byte aligned)
inline int tr_tile(int el) { return el == 1 ? 4 * kTrQ : 2 * kTrQ; }

struct TreeArgs {
    const void* cm;
    size_t pitch;
    const int4* chan;  // [nblk * nlive] channel row, window start after t0 (samples),
                       // first planar word in the stage, planar words / 4
    int rawlen, pmax;  // words of the stage's windows, patterns of a stage at most
    const int* dmrow;  // [ndm] output row of each DM trial in block order
    const int* pstart; // [nblk * nq + 1] first pattern of (block, stage)
    const int4* pat;   // [2 * patterns] planar word of each channel's source; first
                       // group of 32 Y elements in the stage, groups
    const int* gtot;   // [nblk * nq] groups of a stage
    const int* yoff;   // [nblk * nq * (cc/S) * 16 DPW] Y element of a trial
    int nlive, ndm, ndb, nblk, cc, nq, zero, zlen, plen, gmax;
    float* out;
    size_t out_pitch, nout;
    float mid, scale;
    int raw;
    int p16;           // channels a 16-bit sum holds at the input's largest value
    int p8s;           // subbands a byte holds (1..4-bit samples)
    unsigned tile0;    // first output tile of the launch
};

// A warp's Y offsets of one subband.
template <int DPW>
__device__ __forceinline__ int2 yoffs(const int* p)
{
    if constexpr (DPW == 2) return *reinterpret_cast<const int2*>(p);
    return make_int2(p[0], p[0]);
}

template <int MODE, int DPW, bool FLUSH>
__global__ void __launch_bounds__(kTrThreads, 2) k_dedisperse_tree(TreeArgs a)
{
    constexpr int S = kTrS, W = kTrWords;
    constexpr int kSlots = kTrWarps * DPW, kElem = MODE == kTr16 ? 2 : 1;
    constexpr int kParts = MODE == kTr16 ? 2 : 4;      // outputs of one planar word
    constexpr int kYWords = MODE == kTrSmall ? 1 : 2;  // words of one Y element
    extern __shared__ __align__(16) uint32_t tsm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int blk = blockIdx.x % a.nblk;
    const size_t t0 = (size_t)(a.tile0 + blockIdx.x / a.nblk) * (kParts * kTrQ);
    const int nsb = a.cc / S;       // subbands per stage
    uint32_t* raw = tsm;            // the next stage's windows as they are in cm
    uint32_t* pl = raw + a.rawlen;  // planar words of the stage's channels, zeros at a.zero
    uint32_t* ysm = pl + a.plen;    // Y of the stage's patterns
    int4* s_pat = reinterpret_cast<int4*>(ysm + a.gmax * 32 * kYWords);  // [2][pmax][2]
    int* s_yoff = reinterpret_cast<int*>(s_pat + 4 * a.pmax);            // [2][nsb][kSlots]
    // a window's words after its planar ones' first part; its place in raw
    // follows from its place among the planar words
    constexpr int kMore = MODE == kTr16 ? kTrQ / 2 : 3 * kTrQ / 4;
    auto raw_at = [&](int c, const int4& ch) {
        return raw + (MODE == kTr16 ? ch.z / 2 : ch.z / 4) + c * (kMore + 4);
    };

    // A stage's windows and tables, asynchronously.
    auto load_stage = [&](int q) {
        const int nch = min(a.cc, a.nlive - q * a.cc), bq = blk * a.nq + q;
        for (int c = warp; c < nch; c += kTrWarps) {
            const int4 ch = a.chan[(size_t)blk * a.nlive + q * a.cc + c];
            const uint32_t* w = reinterpret_cast<const uint32_t*>(
                static_cast<const uint8_t*>(a.cm) + ((size_t)ch.x * a.pitch + t0 + ch.y) * kElem);
            uint32_t* d = raw_at(c, ch);
            const int n = (MODE == kTr16 ? 2 * ch.w : ch.w) + kMore;
            for (int p = 4 * lane; p < n; p += 128) cp_async16(d + p, w + p);
        }
        const int p0 = a.pstart[bq], np = a.pstart[bq + 1] - p0;
        int4* dp = s_pat + (q & 1) * 2 * a.pmax;
        for (int k = threadIdx.x; k < 2 * np; k += kTrThreads) cp_async16(dp + k, a.pat + 2 * (size_t)p0 + k);
        int* dy = s_yoff + (q & 1) * nsb * kSlots;
        const int* sy = a.yoff + (size_t)bq * nsb * kSlots;
        for (int k = threadIdx.x; k < nsb * (kSlots / 4); k += kTrThreads) cp_async16(dy + 4 * k, sy + 4 * k);
        cp_async_commit();
    };
    // Windows -> planar words, four consecutive words per step.
    auto to_planar = [&](int q) {
        const int nch = min(a.cc, a.nlive - q * a.cc);
        for (int c = warp; c < nch; c += kTrWarps) {
            const int4 ch = a.chan[(size_t)blk * a.nlive + q * a.cc + c];
            const uint32_t* w = raw_at(c, ch);
            uint4* d = reinterpret_cast<uint4*>(pl + ch.z);
            for (int p = lane; p < ch.w; p += 32) {
                uint4 v;
                if constexpr (MODE == kTr16) {
                    const uint2 a0 = reinterpret_cast<const uint2*>(w)[p];
                    const uint2 b0 = reinterpret_cast<const uint2*>(w)[p + kTrQ / 4];
                    v.x = __byte_perm(a0.x, b0.x, 0x5410);
                    v.y = __byte_perm(a0.x, b0.x, 0x7632);
                    v.z = __byte_perm(a0.y, b0.y, 0x5410);
                    v.w = __byte_perm(a0.y, b0.y, 0x7632);
                } else {
                    const uint32_t w0 = w[p], w1 = w[p + kTrQ / 4];
                    const uint32_t w2 = w[p + kTrQ / 2], w3 = w[p + 3 * kTrQ / 4];
                    const uint32_t l0 = __byte_perm(w0, w1, 0x5140), l1 = __byte_perm(w2, w3, 0x5140);
                    const uint32_t h0 = __byte_perm(w0, w1, 0x7362), h1 = __byte_perm(w2, w3, 0x7362);
                    v.x = __byte_perm(l0, l1, 0x5410);
                    v.y = __byte_perm(l0, l1, 0x7632);
                    v.z = __byte_perm(h0, h1, 0x5410);
                    v.w = __byte_perm(h0, h1, 0x7632);
                }
                d[p] = v;
            }
        }
    };

    // packed 16-bit sums (32-bit for 16-bit samples): the pairs' first
    // words, then their second words
    uint32_t acc[DPW][2 * W];
#pragma unroll
    for (int j = 0; j < DPW; ++j)
#pragma unroll
        for (int k = 0; k < 2 * W; ++k) acc[j][k] = 0;
    // the warp's DM trials in the block: neighbours, which may read the same
    // Y, or (1..4 bits, whose loop has no registers left to compare) 16 apart,
    // so that a block that is not full leaves no warp without one
    constexpr int kStep = MODE == kTrSmall ? kTrWarps : 1;
    const int s0 = MODE == kTrSmall ? warp : DPW * warp;
    const int d0 = blk * a.ndb + s0;
    const int dend = min(a.ndm, (blk + 1) * a.ndb);
    bool flushed = false;
    int since = 0;
    // f(output of trial j after t0 + lane, sum) over the warp's outputs
    auto each_of = [&](int j, auto in, auto f) {
#pragma unroll
        for (int k = 0; k < 2 * W; ++k) {
            const int t = 32 * (k % W) + (k < W ? 0 : kTrQ);
            if constexpr (MODE == kTr16) {
                if (in(t)) f(t, acc[j][k]);
            } else {
                if (in(t)) f(t, acc[j][k] & 0xffffu);
                if (in(t + 2 * kTrQ)) f(t + 2 * kTrQ, acc[j][k] >> 16);
            }
        }
    };
    auto each = [&](int j, auto f) {
        if (t0 + kParts * kTrQ <= a.nout) {
            each_of(j, [](int) { return true; }, f);
        } else {
            const int left = (int)(a.nout - t0) - lane;  // the last tile
            each_of(j, [&](int t) { return t < left; }, f);
        }
    };

    for (int k = threadIdx.x; k < a.zlen; k += kTrThreads) pl[a.zero + k] = 0;
    load_stage(0);
    cp_async_wait<0>();
    __syncthreads();
    to_planar(0);
    for (int q = 0; q < a.nq; ++q) {
        const int bq = blk * a.nq + q, nch = min(a.cc, a.nlive - q * a.cc);
        const int np = a.pstart[bq + 1] - a.pstart[bq], ng = a.gtot[bq];
        __syncthreads();
        if (q + 1 < a.nq) load_stage(q + 1);
        // the patterns' series: every warp takes an equal run of the stage's
        // ng groups of 32 elements, starting inside pattern p
        {
            const int4* sp = s_pat + (q & 1) * 2 * a.pmax;
            int g = ng * warp / kTrWarps;
            const int gend = ng * (warp + 1) / kTrWarps;
            int p = -1;
            for (int b0 = 0; b0 < np; b0 += 32) {
                const bool at = b0 + lane < np && sp[2 * (b0 + lane) + 1].x <= g;
                p += __popc(__ballot_sync(0xffffffffu, at));
            }
            while (g < gend) {
                const int4 src = sp[2 * p], rec = sp[2 * p + 1];
                const int n = min(rec.x + rec.y, gend) - g, k = 32 * (g - rec.x) + lane;
                const uint32_t* x0 = pl + src.x + k;
                const uint32_t* x1 = pl + src.y + k;
                const uint32_t* x2 = pl + src.z + k;
                const uint32_t* x3 = pl + src.w + k;
                uint32_t* y = ysm + (32 * g + lane) * kYWords;
#pragma unroll 8
                for (int m = 0; m < n; ++m) {
                    const uint32_t v0 = x0[32 * m], v1 = x1[32 * m], v2 = x2[32 * m],
                                   v3 = x3[32 * m];
                    if constexpr (MODE == kTrSmall) {
                        y[32 * m] = v0 + v1 + v2 + v3;
                    } else if constexpr (MODE == kTr8) {
                        // whole words summed modulo 2^32; the odd bytes' sums
                        // taken out of that leave the even bytes' (both < 2^16)
                        const uint32_t all = v0 + v1 + v2 + v3;
                        const uint32_t o = __byte_perm(v0, 0, 0x4341) + __byte_perm(v1, 0, 0x4341) +
                                           __byte_perm(v2, 0, 0x4341) + __byte_perm(v3, 0, 0x4341);
                        reinterpret_cast<uint2*>(y)[32 * m] = make_uint2(all - o * 256u, o);
                    } else {
                        reinterpret_cast<uint2*>(y)[32 * m] =
                            make_uint2((v0 & 0xffffu) + (v1 & 0xffffu) + (v2 & 0xffffu) + (v3 & 0xffffu),
                                       (v0 >> 16) + (v1 >> 16) + (v2 >> 16) + (v3 >> 16));
                    }
                }
                g += n;
                ++p;
            }
        }
        cp_async_wait<0>();
        __syncthreads();
        // the planar words are free: the next stage's go in beside the sums
        if (q + 1 < a.nq) to_planar(q + 1);
        if constexpr (FLUSH) {
            // before a 16-bit sum can overflow: the sums so far go to the
            // output rows as whole floats (exact: checked on the host)
            if (since + nch > a.p16) {
#pragma unroll
                for (int j = 0; j < DPW; ++j) {
                    if (d0 + j * kStep < dend) {
                        float* o = a.out + (size_t)a.dmrow[d0 + j * kStep] * a.out_pitch + t0 + lane;
                        each(j, [&](int t, uint32_t v) {
                            o[t] = flushed ? o[t] + (float)v : (float)v;
                        });
                    }
#pragma unroll
                    for (int k = 0; k < 2 * W; ++k) acc[j][k] = 0;
                }
                flushed = true;
                since = 0;
            }
            since += nch;
        }
        // one Y per subband and DM trial
        // (1..4 bits: tested below, per trial)
        const int nb = MODE == kTrSmall || d0 < dend ? (nch + S - 1) / S : 0;
        const int* sy = s_yoff + (q & 1) * nsb * kSlots + s0;
        if constexpr (MODE == kTrSmall) {
            // bytes as they stand while they cannot overflow
#pragma unroll
            for (int j = 0; j < DPW; ++j) {
                if (d0 + j * kStep >= dend) continue;
                for (int b0 = 0; b0 < nb; b0 += a.p8s) {
                    uint32_t a8[W];
#pragma unroll
                    for (int k = 0; k < W; ++k) a8[k] = 0;
                    const int b1 = min(nb, b0 + a.p8s);
#pragma unroll 2
                    for (int b = b0; b < b1; ++b) {
                        const uint32_t* y = ysm + sy[b * kSlots + j * kStep] + lane;
#pragma unroll
                        for (int k = 0; k < W; ++k) a8[k] += y[32 * k];
                    }
#pragma unroll
                    for (int k = 0; k < W; ++k) {
                        acc[j][k] += __byte_perm(a8[k], 0, 0x4240);
                        acc[j][W + k] += __byte_perm(a8[k], 0, 0x4341);
                    }
                }
            }
        } else {
            // A warp's two trials are neighbours and read the same Y where
            // their offsets agree (18 % of them at survey spacing).  Not
            // unrolled: two subbands at a time spilled registers.
            const uint2* y2 = reinterpret_cast<const uint2*>(ysm) + lane;
#pragma unroll 1
            for (int b = 0; b < nb; ++b) {
                const int2 off = yoffs<DPW>(sy + b * kSlots);
                uint2 v[W];
#pragma unroll
                for (int k = 0; k < W; ++k) v[k] = y2[off.x + 32 * k];
#pragma unroll
                for (int k = 0; k < W; ++k) {
                    acc[0][k] += v[k].x;
                    acc[0][W + k] += v[k].y;
                }
                if constexpr (DPW == 2) {
                    if (off.y != off.x) {
#pragma unroll
                        for (int k = 0; k < W; ++k) v[k] = y2[off.y + 32 * k];
                    }
#pragma unroll
                    for (int k = 0; k < W; ++k) {
                        acc[1][k] += v[k].x;
                        acc[1][W + k] += v[k].y;
                    }
                }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < DPW; ++j) {
        if (d0 + j * kStep >= dend) continue;
        float* o = a.out + (size_t)a.dmrow[d0 + j * kStep] * a.out_pitch + t0 + lane;
        each(j, [&](int t, uint32_t v) {
            if constexpr (FLUSH) {
                if (flushed) v += (uint32_t)o[t];
                o[t] = map_sum(v, a.mid, a.scale, a.raw);
            } else if constexpr (MODE == kTr16) {
                o[t] = map_sum(v, a.mid, a.scale, a.raw);
            } else {
                // a 16-bit whole number to float without the conversion unit
                float f = __uint_as_float(0x4b000000u | v) - 8388608.0f;
                if (!a.raw) f = __fadd_rn(__fmul_rn(__fsub_rn(f, a.mid), a.scale), 0.5f);
                o[t] = f;
            }
        });
    }
}

size_t round_up(size_t x, size_t m) { return (x + m - 1) / m * m; }

}  // namespace

// When the shared sums are taken: predicted time over the direct form's below
// one.  Of a full device, as a share of the direct form's (2Q words of shared
// memory per DM trial and channel, DM trials in eights): the words of the
// patterns' series (S + 2 each), one Y per subband and DM trial, a stage's
// fixed time over its channels and DM trials, and what a CTA takes beside its
// channels.  Of a device that is not full: an SM runs the CTAs of a launch two
// (direct: four) at a time, and a lone shared-sum CTA takes 1.2 to 1.5 halves
// of a pair's time, the direct form half to one CTA's time over its CTAs'.
// The weights are least squares of the measured times (B200, kernel alone,
// 2, 8 and 16 bits x 16 to 1024 channels x 8 to 100 DM trials of up to 20 to
// 150 x 50 to 1200 CTAs, 8400 pairs, prediction within 12 % RMS): taken so,
// 0.3 % of the pairs are more than 3 % slower than the direct form, against
// 4 % with one line through the words and one through the CTAs.  Some of
// those measured (us, direct and shared; channels, DM trials up to DM, bits):
// 64, 32 to 60, 2: 18.5 and 28.7 at 74 CTAs, 71.8 and 65.9 at 400; 64, 32 to
// 60, 8: 20.4 and 30.9 at 74, 35.0 and 31.7 at 148; 64, 32 to 90, 8: 83.9 and
// 94.5 at 400; 1024, 32 to 60, 8: 307 and 264 at 74; 1024, 20 to 150, 8: 998
// and 774 at 400.  Of 692 other lists of 8 to 400 DM trials (uneven spacing,
// channels left out, 1 to 16 bits), 6 are more than 3 % slower so than with
// the direct form, 1.16 times at most; of 189 lists of 2 to 7, 24, up to 1.42
// times: those take the direct form.
struct DedispWeights {
    double patterns, sums, stage, channel, odd, fill;
};
constexpr DedispWeights kDedispWeights[3] = {
    {1.07, 0.73, 46.0, 2.1, 0.26, 0.5},   // kTr8
    {1.07, 0.86, 59.0, 2.6, 0.22, 0.5},   // kTrSmall
    {0.95, 0.68, 58.0, 0.75, 0.48, 1.0},  // kTr16
};

// The second factor of that prediction, for the CTAs of both launches.
inline double dedisp_occupancy(int kind, double ctas, double direct_ctas)
{
    const DedispWeights& w = kDedispWeights[kind];
    const double sms = sm_count(), n = std::ceil(ctas / sms);
    return (n + (std::fmod(n, 2.0) != 0.0 ? w.odd : 0.0)) / ctas /
           ((std::ceil(direct_ctas / sms) + w.fill) / direct_ctas);
}

// Shift tables and launch shape of one form for one class of samples.
struct DedispTables {
    // kRated: only `rate`, at least, known so far; kNotTaken: the direct form instead
    enum State { kNew, kRated, kBuilt, kNotTaken };
    State state = kNew;
    bool uploaded = false;
    int kind = 0;           // sample class (direct: any of this width)
    int elem = 0;           // bytes a sample
    int nlive = 0, ndm_pad = 0, nblk = 0, group = 8, lwin = 0, cc = 0;
    size_t ngroups = 0, max_lo = 0;
    size_t flush_bytes = 0;             // shared 32-bit sums above 257 channels
    // shared-partial-sum form (k_dedisperse_tree): 0 = the direct kernel,
    // else S; DM trials in order of DM, ndb per block, dpw per warp
    double rate = 0.0;      // predicted time of a full device over the direct form's
    int tree = 0, dpw = 0, ndb = 0, nq = 0, zero = 0, zlen = 0, plen = 0, gmax = 0, pmax = 0, rawlen = 0,
        tile = 0;
    size_t tab_row = 0, tab_ps = 0, tab_gt = 0, tab_pat = 0, tab_yoff = 0;  // in h_tab
    std::vector<int> h_tab;
    int* d_tab = nullptr;
    size_t tab_cap = 0;

    // a stage's windows: the planar words' samples once, and per channel
    // the parts after the first
    static int raw_words(int c, int pm, int more, int el) { return pm / (el == 1 ? 4 : 2) + c * (more + 4); }

    static size_t tree_bytes(int raw, int plen, int gmax, int yw, int pmax, int trials)
    {
        return 4ull * ((size_t)raw + plen + 32ull * gmax * yw + 2ull * pmax * kTrRec + 2ull * trials);
    }

    size_t smem_bytes() const
    {
        if (tree)
            return tree_bytes(rawlen, plen, gmax, kind == kTrSmall ? 1 : 2, pmax,
                              cc / kTrS * kTrWarps * dpw);
        return 2ull * cc * (kDdWarps / group) * lwin * elem + 2ull * kDdWarps * cc * sizeof(int) +
               flush_bytes;
    }
};

}  // namespace psx

using namespace psx;

struct psx_dedisp_plan {
    size_t nchans = 0;
    float tsamp = 0, fch1 = 0, foff = 0;
    std::vector<float> delays, dms;
    std::vector<int> live;  // 1 = channel summed
    // Derived tables: the shared-sum form's by sample class, then the direct
    // form's by sample width.  Every one a call has needed is kept until the
    // DM list or the channels change, so that calls which need different ones
    // in turn (a short output after long ones, files of another sample width)
    // do not build and upload them each time: 0.9 ms of host time at 1024
    // channels x 100 DM trials, 9 ms at 4096 x 300.
    DedispTables sets[5];
    DedispTables* t = nullptr;          // the call's
    size_t scratch_limit = 4ull << 30;  // bytes of channel-major samples
    void* d_cm = nullptr;
    size_t cm_cap = 0;
    uint8_t* d_stage = nullptr;
    size_t stage_cap = 0;
    cudaStream_t copy_stream = nullptr;
    cudaEvent_t ev_copied[2] = {nullptr, nullptr};
    cudaEvent_t ev_used[2] = {nullptr, nullptr};

    size_t max_delay() const
    {
        if (dms.empty() || nchans == 0) return 0;
        float dm_max = dms[0];
        for (float v : dms) dm_max = std::max(dm_max, v);
        float prod = dm_max * delays[nchans - 1];
        return (size_t)std::floor((double)prod + 0.5);
    }

    void changed()
    {
        for (DedispTables& x : sets) x.state = DedispTables::kNew;
    }

    // Takes the tables for one class of samples and nout outputs, building
    // them where this DM list has not needed them yet.
    int take_tables(int kind, size_t nout)
    {
        const int el = kind == kTr16 ? 2 : 1;
        if (dms.empty()) {
            set_error("psx_dedisp: no DM list set");
            return PSX_ERR_INVALID;
        }
        DedispTables &shared = sets[kind], &direct = sets[3 + (el == 2)];
        const double tiles = (double)((nout + tr_tile(el) - 1) / tr_tile(el));
        const double direct_ctas = tiles * (double)((dms.size() + kDdWarps - 1) / kDdWarps);
        const size_t blocks = (dms.size() + kTrMaxDms - 1) / kTrMaxDms;
        const double full = dedisp_occupancy(kind, tiles * (double)blocks, direct_ctas);
        std::vector<int> chans, shift;
        // The rate of a list is not looked at (0.4 ms of host time at 1024
        // channels x 100 DM trials) where it had to be below a half: less than
        // half the device's SMs have a CTA then, and little is to be gained.
        if (dms.size() >= kTrMinDms && full < 2.0 &&
            (shared.state == DedispTables::kNew ||
             (shared.state == DedispTables::kRated && shared.rate * full < 1.0))) {
            shared.kind = kind;
            shared.elem = el;
            shared.uploaded = false;
            shifts(&chans, &shift);
            shared.nlive = (int)chans.size();
            shared.state = shared.nlive > 0 ? build_tree(shared, chans, shift, full)
                                            : DedispTables::kNotTaken;
        }
        t = shared.state == DedispTables::kBuilt && shared.rate * full < 1.0 ? &shared : &direct;
        if (t->state == DedispTables::kBuilt) return PSX_OK;
        if (shift.empty()) shifts(&chans, &shift);
        direct.kind = kind;
        direct.elem = el;
        direct.uploaded = false;
        PSX_TRY(build_direct(direct, chans, shift));
        direct.state = DedispTables::kBuilt;
        return PSX_OK;
    }

    // Channels summed, and the shift of every (DM trial, such channel).
    void shifts(std::vector<int>* chans, std::vector<int>* shift) const
    {
        for (size_t c = 0; c < nchans; ++c)
            if (live[c]) chans->push_back((int)c);
        const size_t nlive = chans->size(), ndm = dms.size();
        shift->resize(ndm * std::max<size_t>(nlive, 1));
        for (size_t d = 0; d < ndm; ++d)
            for (size_t i = 0; i < nlive; ++i) {
                float p = dms[d] * delays[(*chans)[i]];
                (*shift)[d * nlive + i] = (int)std::nearbyint(p);
            }
    }

    // Shift tables and the window shape of the direct form.
    int build_direct(DedispTables& T, const std::vector<int>& chans, const std::vector<int>& shift)
    {
        const int el = T.elem;
        const int nlive = T.nlive = (int)chans.size();
        const int ndm = (int)dms.size();
        const int ndm_pad = T.ndm_pad = (int)round_up((size_t)ndm, kDdWarps);
        T.nblk = ndm_pad / kDdWarps;
        const int align = 16 / el;  // window starts on 16-byte boundaries
        T.tile = dd_tile(el);
        T.tree = 0;
        // window shape for groups of G trials: lo = min shift aligned down,
        // lwin covers 512 outputs past the largest shift plus the read-ahead
        auto shape = [&](int G, std::vector<int>* lo_out, int* lwin_out, size_t* max_lo_out) {
            size_t ng = (size_t)ndm_pad / G;
            std::vector<int> lo(ng * std::max(nlive, 1), 0);
            int spread = 0;
            size_t mlo = 0;
            for (size_t g = 0; g < ng; ++g)
                for (int i = 0; i < nlive; ++i) {
                    int mn = INT32_MAX, mx = 0;
                    for (int d = (int)g * G; d < std::min(ndm, (int)(g + 1) * G); ++d) {
                        int s = shift[(size_t)d * nlive + i];
                        mn = std::min(mn, s);
                        mx = std::max(mx, s);
                    }
                    if (mn == INT32_MAX) mn = mx = 0;
                    int l = mn / align * align;
                    lo[g * nlive + i] = l;
                    spread = std::max(spread, mx - l);
                    mlo = std::max(mlo, (size_t)l);
                }
            *lwin_out = (int)round_up((size_t)spread + dd_tile(el) + 8, (size_t)align);
            *max_lo_out = mlo;
            if (lo_out) lo_out->swap(lo);
        };
        std::vector<int> lo8, lo1;
        int lwin8 = 0, lwin1 = 0;
        size_t mlo8 = 0, mlo1 = 0;
        shape(8, &lo8, &lwin8, &mlo8);
        shape(1, &lo1, &lwin1, &mlo1);
        T.group = (lwin8 <= kDdWarps * lwin1) ? 8 : 1;
        std::vector<int>& lo = T.group == 8 ? lo8 : lo1;
        T.lwin = T.group == 8 ? lwin8 : lwin1;
        T.max_lo = T.group == 8 ? mlo8 : mlo1;
        T.ngroups = (size_t)ndm_pad / T.group;
        const int nwin = kDdWarps / T.group;
        T.cc = 0;
        T.flush_bytes = (el == 1 && nlive > 257) ? 4ull * (kDdTile8 / 32) * kDdThreads : 0;
        // with the flush sums, fewer channels per chunk keep 4 CTAs on an SM
        const size_t cap = T.flush_bytes ? 56 * 1024 : 96 * 1024;
        for (int c : {16, 8, 4, 2, 1}) {
            size_t bytes = 2ull * c * nwin * T.lwin * el + 2ull * kDdWarps * c * sizeof(int) +
                           T.flush_bytes;
            if (bytes <= cap || (c == 1 && bytes <= 200 * 1024)) {
                T.cc = c;
                break;
            }
        }
        if (T.cc == 0) {
            set_error("psx_dedisp: DM trials of one block spread over %d samples; "
                      "the shared-memory window does not fit", T.lwin);
            return PSX_ERR_UNSUPPORTED;
        }
        T.h_tab.assign((size_t)nlive + T.ngroups * nlive + (size_t)ndm_pad * nlive, 0);
        std::copy(chans.begin(), chans.end(), T.h_tab.begin());
        std::copy(lo.begin(), lo.begin() + T.ngroups * nlive, T.h_tab.begin() + nlive);
        int* off = T.h_tab.data() + nlive + T.ngroups * nlive;
        for (int d = 0; d < ndm; ++d)
            for (int i = 0; i < nlive; ++i)
                off[(size_t)d * nlive + i] =
                    shift[(size_t)d * nlive + i] - lo[(size_t)(d / T.group) * nlive + i];
        return PSX_OK;
    }

    // Rate and, where the call's CTAs (`full`) want them, tables of the
    // shared-partial-sum form; kNotTaken where the direct kernel is taken
    // whatever the outputs: the series do not fit shared memory, a sum could
    // pass 2^24 where sums are kept as floats, or the patterns are so many (few
    // or widely spaced DM trials) that no number of CTAs makes up for them (see
    // kDedispWeights; its second factor is 0.66 at least).
    DedispTables::State build_tree(DedispTables& T, const std::vector<int>& chans,
                                   const std::vector<int>& shift, double full)
    {
        constexpr int S = kTrS;
        const int el = T.elem, nlive = T.nlive;
        const int ndm = (int)dms.size();
        if (el == 1 && (double)nlive * 255.0 >= 16777216.0) return DedispTables::kNotTaken;
        std::vector<int> order(ndm);
        for (int d = 0; d < ndm; ++d) order[d] = d;
        std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return dms[x] < dms[y]; });
        const int nb_ = (ndm + kTrMaxDms - 1) / kTrMaxDms;
        const int per = (ndm + nb_ - 1) / nb_;       // DM trials per block, evenly
        const int dw = (per + kTrWarps - 1) / kTrWarps, slots = kTrWarps * dw;
        const int blocks = (ndm + per - 1) / per;
        const int nsbt = (nlive + S - 1) / S, align = 16 / el;
        struct Pat {
            int first, lo, groups;  // a trial that has it, smallest reference shift, 32-word groups
        };
        // per (block, channel): window start, planar words / 4
        std::vector<int> lo((size_t)blocks * nlive), quads((size_t)blocks * nlive);
        std::vector<int> np((size_t)blocks * nsbt);
        std::vector<Pat> pats;                       // in (block, subband) order
        std::vector<uint8_t> which((size_t)ndm * nsbt);
        int most = 0;
        size_t mlo = 0, ngroups_ = 0;
        for (int g = 0; g < blocks; ++g) {
            const int e0 = g * per, e1 = std::min(ndm, e0 + per);
            int* l = &lo[(size_t)g * nlive];
            std::vector<int> mx(shift.begin() + (size_t)order[e0] * nlive,
                                shift.begin() + (size_t)(order[e0] + 1) * nlive);
            std::copy(mx.begin(), mx.end(), l);
            for (int e = e0 + 1; e < e1; ++e) {
                const int* v = &shift[(size_t)order[e] * nlive];
                for (int i = 0; i < nlive; ++i) {
                    l[i] = std::min(l[i], v[i]);
                    mx[i] = std::max(mx[i], v[i]);
                }
            }
            for (int i = 0; i < nlive; ++i) {
                l[i] = l[i] / align * align;
                // a multiple of 16 planar words, so that the windows start 16-byte aligned
                const int qd = (int)round_up((size_t)(kTrQ + mx[i] - l[i]), 16) / 4;
                quads[(size_t)g * nlive + i] = qd;
                most = std::max(most, qd);
                mlo = std::max(mlo, (size_t)l[i]);
            }
            for (int b = 0; b < nsbt; ++b) {
                const int c0 = b * S, nc = std::min(S, nlive - c0);
                int first[kTrMaxDms], mn[kTrMaxDms], mxr[kTrMaxDms], n = 0, last = 0;
                for (int e = e0; e < e1; ++e) {
                    const int* v = &shift[(size_t)order[e] * nlive + c0];
                    auto same = [&](int p) {
                        const int* u = &shift[(size_t)order[first[p]] * nlive + c0];
                        for (int c = 1; c < nc; ++c)
                            if (v[c] - v[0] != u[c] - u[0]) return false;
                        return true;
                    };
                    int p = last;
                    if (n == 0 || !same(p))
                        for (p = 0; p < n && !same(p);) ++p;
                    if (p == n) {
                        first[n] = e;
                        mn[n] = mxr[n] = v[0];
                        ++n;
                    }
                    mn[p] = std::min(mn[p], v[0]);
                    mxr[p] = std::max(mxr[p], v[0]);
                    which[(size_t)e * nsbt + b] = (uint8_t)p;
                    last = p;
                }
                np[(size_t)g * nsbt + b] = n;
                for (int p = 0; p < n; ++p) {
                    const int gr = (kTrQ + mxr[p] - mn[p] + 31) / 32;
                    pats.push_back({first[p], mn[p], gr});
                    ngroups_ += gr;
                }
            }
        }
        const DedispWeights& w = kDedispWeights[T.kind];
        auto rate_at = [&](int c) {  // with c channels a stage
            return (w.patterns * (double)ngroups_ * 32 * (S + 2) / (2.0 * kTrQ * nlive * ndm) +
                    w.sums * nsbt / nlive + w.stage / ((double)c * per) + w.channel / nlive) *
                   ndm / (double)round_up((size_t)ndm, kDdWarps);
        };
        T.rate = rate_at(32);
        if (T.rate * full >= 1.0) return DedispTables::kRated;
        // channels per stage: the most that leave two CTAs on an SM
        const int yw = T.kind == kTrSmall ? 1 : 2;
        int c_ = 0, pm = 0, gm = 0, nm = 0;
        const int more = el == 1 ? 3 * kTrQ / 4 : kTrQ / 2;
        for (int c : {32, 16, 8, 4}) {
            if (c > 4 && c / 2 >= nlive) continue;
            pm = gm = nm = 0;
            size_t at = 0;
            for (int g = 0; g < blocks; ++g)
                for (int b0 = 0; b0 < nsbt; b0 += c / S) {
                    int gr = 0, pw = 0, n = 0;
                    for (int b = b0; b < std::min(nsbt, b0 + c / S); ++b)
                        for (int p = 0; p < np[(size_t)g * nsbt + b]; ++p, ++n) gr += pats[at++].groups;
                    nm = std::max(nm, n);
                    for (int i = b0 * S; i < std::min(nlive, b0 * S + c); ++i)
                        pw += 4 * quads[(size_t)g * nlive + i];
                    pm = std::max(pm, pw);
                    gm = std::max(gm, gr);
                }
            // the last group of a pattern may read up to 31 words past a
            // channel's: into the next one's, or the zeros
            const size_t b = DedispTables::tree_bytes(DedispTables::raw_words(c, pm, more, el),
                                                      pm + 4 * most + 32, gm, yw, nm, c / S * slots);
            if (b <= 112 * 1024 || (c == 4 && b <= kDdMaxSmem)) {
                c_ = c;
                break;
            }
        }
        if (!c_) return DedispTables::kNotTaken;
        T.rate = rate_at(c_);
        if (T.rate >= 1.0 / 0.66) return DedispTables::kNotTaken;
        if (T.rate * full >= 1.0) return DedispTables::kRated;
        const int nq_ = (nlive + c_ - 1) / c_, sbs = c_ / S;
        // tables: channel records, output rows, per stage the first pattern
        // and the groups, pattern records, the trials' Y offsets
        T.tab_row = 4 * (size_t)blocks * nlive;
        T.tab_ps = T.tab_row + round_up((size_t)ndm, 4);
        T.tab_gt = T.tab_ps + round_up((size_t)blocks * nq_ + 1, 4);
        T.tab_pat = T.tab_gt + round_up((size_t)blocks * nq_, 4);
        T.tab_yoff = T.tab_pat + pats.size() * kTrRec;
        T.h_tab.assign(T.tab_yoff + (size_t)blocks * nq_ * sbs * slots, 0);
        for (int g = 0; g < blocks; ++g)
            for (int i = 0, at = 0; i < nlive; ++i) {
                if (i % c_ == 0) at = 0;
                int* ch = T.h_tab.data() + 4 * ((size_t)g * nlive + i);
                ch[0] = chans[i];
                ch[1] = lo[(size_t)g * nlive + i];
                ch[2] = at;
                ch[3] = quads[(size_t)g * nlive + i];
                at += 4 * ch[3];
            }
        std::copy(order.begin(), order.end(), T.h_tab.begin() + T.tab_row);
        int* ps = T.h_tab.data() + T.tab_ps;
        int* gt = T.h_tab.data() + T.tab_gt;
        int* yo = T.h_tab.data() + T.tab_yoff;
        size_t at = 0;  // next pattern
        for (int g = 0; g < blocks; ++g) {
            const int e0 = g * per, e1 = std::min(ndm, e0 + per);
            for (int b = 0; b < nsbt; ++b) {
                const int q = b / sbs, c0 = b * S, n = np[(size_t)g * nsbt + b];
                int& gr = gt[g * nq_ + q];
                if (b % sbs == 0) {
                    ps[g * nq_ + q] = (int)at;
                    gr = 0;
                }
                int ybase[kTrMaxDms];
                for (int p = 0; p < n; ++p) {
                    const Pat& pt = pats[at + p];
                    const int* u = &shift[(size_t)order[pt.first] * nlive];
                    int* rec = T.h_tab.data() + T.tab_pat + (at + p) * kTrRec;
                    for (int c = 0; c < S; ++c) {
                        const int i = c0 + c;
                        const int* ch = T.h_tab.data() + 4 * ((size_t)g * nlive + i);
                        rec[c] = i < nlive ? ch[2] + pt.lo + (u[i] - u[c0]) - ch[1]
                                           : pm;  // the zeros
                    }
                    rec[4] = gr;
                    rec[5] = pt.groups;
                    ybase[p] = 32 * gr - pt.lo;
                    gr += pt.groups;
                }
                int* row = yo + (((size_t)g * nq_ + q) * sbs + b % sbs) * slots;
                for (int e = e0; e < e1; ++e)
                    row[e - e0] = ybase[which[(size_t)e * nsbt + b]] +
                                  shift[(size_t)order[e] * nlive + c0];
                // a warp's missing second trial reads what its first one does
                if (e1 - e0 < slots) row[e1 - e0] = row[e1 - e0 - 1];
                at += n;
            }
        }
        ps[blocks * nq_] = (int)at;
        T.tree = S;
        T.dpw = dw;
        T.ndb = per;
        T.nblk = blocks;
        T.cc = c_;
        T.nq = nq_;
        T.zero = pm;
        T.zlen = 4 * most + 32;
        T.plen = T.zero + T.zlen;
        T.gmax = gm;
        T.pmax = nm;
        T.rawlen = DedispTables::raw_words(c_, pm, more, el);
        T.lwin = 4 * most + (el == 1 ? 3 : 1) * kTrQ;
        T.max_lo = mlo;
        T.tile = tr_tile(el);
        return DedispTables::kBuilt;
    }

    ~psx_dedisp_plan()
    {
        for (DedispTables& x : sets)
            if (x.d_tab) cudaFree(x.d_tab);
        if (d_cm) cudaFree(d_cm);
        if (d_stage) cudaFree(d_stage);
        for (int i = 0; i < 2; ++i) {
            if (ev_copied[i]) cudaEventDestroy(ev_copied[i]);
            if (ev_used[i]) cudaEventDestroy(ev_used[i]);
        }
        if (copy_stream) cudaStreamDestroy(copy_stream);
    }
};

namespace {

int grow(void** p, size_t* cap, size_t need, const char* what)
{
    if (*cap >= need) return PSX_OK;
    if (*p) {
        cudaFree(*p);  // synchronises the device: no launch still reads it
        *p = nullptr;
        *cap = 0;
    }
    cudaError_t e = cudaMalloc(p, need);
    if (e != cudaSuccess) {
        cudaGetLastError();
        *p = nullptr;
        set_error("psx_dedisp: cannot allocate %zu bytes for %s: %s", need, what,
                  cudaGetErrorString(e));
        return e == cudaErrorMemoryAllocation ? PSX_ERR_ALLOC : PSX_ERR_CUDA;
    }
    *cap = need;
    return PSX_OK;
}

int check_input(psx_dedisp_plan* p, size_t nsamps, int nbits, float* d_out, size_t out_pitch,
                size_t* nout)
{
    if (!p) {
        set_error("psx_dedisp: null plan");
        return PSX_ERR_INVALID;
    }
    if (nbits != 1 && nbits != 2 && nbits != 4 && nbits != 8 && nbits != 16) {
        set_error("psx_dedisp: %d-bit samples are not supported (1, 2, 4, 8, 16)", nbits);
        return PSX_ERR_UNSUPPORTED;
    }
    if ((p->nchans * (size_t)nbits) % 8 != 0) {
        set_error("psx_dedisp: a row of %zu %d-bit channels is not whole bytes", p->nchans, nbits);
        return PSX_ERR_INVALID;
    }
    size_t md = p->max_delay();
    if (p->dms.empty() || nsamps <= md) {
        set_error("psx_dedisp: %zu samples do not exceed the maximum delay %zu", nsamps, md);
        return PSX_ERR_INVALID;
    }
    if (!d_out || (reinterpret_cast<uintptr_t>(d_out) & 15) || out_pitch % 4 != 0 ||
        out_pitch < nsamps - md) {
        set_error("psx_dedisp: output must be 16-byte aligned with a pitch (multiple of 4) "
                  "of at least %zu floats", nsamps - md);
        return PSX_ERR_INVALID;
    }
    *nout = nsamps - md;
    return PSX_OK;
}

// Tables uploaded and cm sized.  The outputs are made in gulps of *gulp
// samples (a multiple of the CTA tile) so that cm, *pitch samples per
// channel, stays within the plan's scratch limit; one gulp covers the
// whole series when it fits.
int prepare(psx_dedisp_plan* p, size_t nout, int nbits, cudaStream_t st, size_t* gulp,
            size_t* pitch)
{
    const int kind = nbits == 16 ? kTr16 : nbits <= 4 ? kTrSmall : kTr8;
    const int el = nbits == 16 ? 2 : 1;
    PSX_TRY(p->take_tables(kind, nout));
    if (!p->t->uploaded) {
        // Nothing can be allocated or copied from here while the stream is
        // captured: the form whose tables are on the device then, as good as
        // the other but for its time.
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        PSX_CUDA(cudaStreamIsCapturing(st, &capture));
        DedispTables& other = p->t == &p->sets[kind] ? p->sets[3 + (el == 2)] : p->sets[kind];
        if (capture != cudaStreamCaptureStatusNone && other.state == DedispTables::kBuilt &&
            other.uploaded)
            p->t = &other;
    }
    DedispTables& t = *p->t;
    if (!t.uploaded) {
        size_t bytes = t.h_tab.size() * sizeof(int);
        PSX_TRY(grow(reinterpret_cast<void**>(&t.d_tab), &t.tab_cap, std::max<size_t>(bytes, 4),
                     "shift tables"));
        PSX_CUDA(cudaMemcpyAsync(t.d_tab, t.h_tab.data(), bytes, cudaMemcpyHostToDevice, st));
        t.uploaded = true;
    }
    const size_t tile = (size_t)p->t->tile;
    const size_t md = p->max_delay();
    auto pitch_for = [&](size_t g) {
        size_t nt = (g + tile - 1) / tile;
        size_t need = (nt - 1) * tile + p->t->max_lo + (size_t)p->t->lwin;
        return round_up(std::max(need, g + md), kUpRows);
    };
    size_t g = round_up(nout, tile);
    const size_t limit = p->scratch_limit / (p->nchans * (size_t)el);
    if (pitch_for(g) > limit) {
        size_t fixed = pitch_for(tile) - tile;
        g = limit > fixed + tile ? (limit - fixed) / tile * tile : tile;
    }
    *gulp = g;
    *pitch = pitch_for(g);
    return grow(&p->d_cm, &p->cm_cap, *pitch * p->nchans * el, "channel-major samples");
}

template <int NBITS>
int launch_unpack(const uint8_t* rows, size_t nrows, size_t r0, size_t ncols, psx_dedisp_plan* p,
                  size_t pitch, cudaStream_t st)
{
    using T = typename Sample<NBITS>::T;
    size_t row_bytes = p->nchans * NBITS / 8;
    dim3 grid((unsigned)((ncols + kUpRows - 1) / kUpRows),
              (unsigned)((p->nchans + UnpackTile<NBITS>::kChans - 1) / UnpackTile<NBITS>::kChans));
    // word loads when every row starts 4-byte aligned; channels past the
    // last whole word of a row then read as zero and are never stored
    const int vec = (row_bytes % 4 == 0 && (reinterpret_cast<uintptr_t>(rows) & 3) == 0) ? 1 : 0;
    k_unpack_chanmajor<NBITS><<<grid, kUpThreads, 0, st>>>(rows, row_bytes, nrows, r0, ncols,
                                                    (int)p->nchans, static_cast<T*>(p->d_cm), pitch,
                                                    vec);
    return launch_status("k_unpack_chanmajor");
}

int unpack(int nbits, const uint8_t* rows, size_t nrows, size_t r0, size_t ncols,
           psx_dedisp_plan* p, size_t pitch, cudaStream_t st)
{
    switch (nbits) {
        case 1: return launch_unpack<1>(rows, nrows, r0, ncols, p, pitch, st);
        case 2: return launch_unpack<2>(rows, nrows, r0, ncols, p, pitch, st);
        case 4: return launch_unpack<4>(rows, nrows, r0, ncols, p, pitch, st);
        case 8: return launch_unpack<8>(rows, nrows, r0, ncols, p, pitch, st);
        default: return launch_unpack<16>(rows, nrows, r0, ncols, p, pitch, st);
    }
}

// Opts a kernel into kDdMaxSmem: always the same value, since plans in other
// threads launch the same kernel with windows of their own between one
// thread's setting and its launch.
template <class Kernel>
int allow_smem(Kernel kern)
{
    PSX_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kDdMaxSmem));
    return PSX_OK;
}

template <int MODE, bool FLUSH>
int launch_tree(const TreeArgs& a, int dpw, unsigned grid, size_t smem, cudaStream_t st)
{
    auto go = [&](auto kern) -> int {
        PSX_TRY(allow_smem(kern));
        kern<<<grid, kTrThreads, smem, st>>>(a);
        return launch_status("k_dedisperse_tree");
    };
    return dpw == 1 ? go(k_dedisperse_tree<MODE, 1, FLUSH>) : go(k_dedisperse_tree<MODE, 2, FLUSH>);
}

// The shared-partial-sum form (p->t->tree), output tiles [tile0, tile1).
int dedisperse_tree(psx_dedisp_plan* p, int nbits, size_t pitch, size_t nout, float* d_out,
                    size_t out_pitch, int flags, size_t tile0, size_t tile1, cudaStream_t st)
{
    TreeArgs a;
    a.cm = p->d_cm;
    a.pitch = pitch;
    a.chan = reinterpret_cast<const int4*>(p->t->d_tab);
    a.dmrow = p->t->d_tab + p->t->tab_row;
    a.pstart = p->t->d_tab + p->t->tab_ps;
    a.pat = reinterpret_cast<const int4*>(p->t->d_tab + p->t->tab_pat);
    a.gtot = p->t->d_tab + p->t->tab_gt;
    a.yoff = p->t->d_tab + p->t->tab_yoff;
    a.nlive = p->t->nlive;
    a.ndm = (int)p->dms.size();
    a.ndb = p->t->ndb;
    a.nblk = p->t->nblk;
    a.cc = p->t->cc;
    a.nq = p->t->nq;
    a.zero = p->t->zero;
    a.zlen = p->t->zlen;
    a.plen = p->t->plen;
    a.gmax = p->t->gmax;
    a.pmax = p->t->pmax;
    a.rawlen = p->t->rawlen;
    a.out = d_out;
    a.out_pitch = out_pitch;
    a.nout = nout;
    const unsigned m = (1u << nbits) - 1u;
    a.mid = (float)(0.5 * (double)p->nchans * (double)m);
    a.scale = (float)(1.0 / ((double)m * std::sqrt((double)p->nchans)));
    a.raw = (flags & PSX_DEDISP_RAW) ? 1 : 0;
    a.p16 = (int)(65535u / m);
    a.p8s = (int)(255u / m) / kTrS;
    a.tile0 = (unsigned)tile0;
    const size_t nblocks = (tile1 - tile0) * (size_t)p->t->nblk;
    if (nblocks > 0x7fffffffull) {
        set_error("psx_dedisp: %zu blocks exceed one launch", nblocks);
        return PSX_ERR_UNSUPPORTED;
    }
    const size_t smem = p->t->smem_bytes();
    const unsigned grid = (unsigned)nblocks;
    if (nbits == 16) return launch_tree<kTr16, false>(a, p->t->dpw, grid, smem, st);
    const bool flush = p->t->nlive > a.p16;
    if (nbits <= 4)
        return flush ? launch_tree<kTrSmall, true>(a, p->t->dpw, grid, smem, st)
                     : launch_tree<kTrSmall, false>(a, p->t->dpw, grid, smem, st);
    return flush ? launch_tree<kTr8, true>(a, p->t->dpw, grid, smem, st)
                 : launch_tree<kTr8, false>(a, p->t->dpw, grid, smem, st);
}

// Output tiles [tile0, tile1) of nout outputs (tile1 0: all the rest).
int dedisperse(psx_dedisp_plan* p, int nbits, size_t pitch, size_t nout, float* d_out,
               size_t out_pitch, int flags, cudaStream_t st, size_t tile0 = 0, size_t tile1 = 0)
{
    if (!tile1) tile1 = (nout + p->t->tile - 1) / p->t->tile;
    if (p->t->tree)
        return dedisperse_tree(p, nbits, pitch, nout, d_out, out_pitch, flags, tile0, tile1, st);
    DedispArgs a;  // with every channel killed the sums are zero
    a.cm = p->d_cm;
    a.pitch = pitch;
    a.chan = p->t->d_tab;
    a.lo = p->t->d_tab + p->t->nlive;
    a.off = p->t->d_tab + p->t->nlive + p->t->ngroups * p->t->nlive;
    a.nlive = p->t->nlive;
    a.ndm = (int)p->dms.size();
    a.nblk = p->t->nblk;
    a.cc = p->t->cc;
    a.lwin = p->t->lwin;
    a.group = p->t->group;
    a.out = d_out;
    a.out_pitch = out_pitch;
    a.nout = nout;
    unsigned m = (1u << nbits) - 1u;
    a.mid = (float)(0.5 * (double)p->nchans * (double)m);
    a.scale = (float)(1.0 / ((double)m * std::sqrt((double)p->nchans)));
    a.raw = (flags & PSX_DEDISP_RAW) ? 1 : 0;
    a.p8 = (int)(255u / m);
    a.p16 = (int)(65535u / m);
    a.tile0 = (unsigned)tile0;
    size_t nblocks = (tile1 - tile0) * (size_t)p->t->nblk;
    if (nblocks > 0x7fffffffull) {
        set_error("psx_dedisp: %zu blocks exceed one launch", nblocks);
        return PSX_ERR_UNSUPPORTED;
    }
    size_t smem = p->t->smem_bytes();
    const unsigned grid = (unsigned)nblocks;
    if (nbits == 16) {
        PSX_TRY(allow_smem(k_dedisperse<uint16_t, false, false>));
        k_dedisperse<uint16_t, false, false><<<grid, kDdThreads, smem, st>>>(a);
    } else {
        // 8 bits and below: the flush and small-sample variants
        const bool flush = p->t->nlive > a.p16, small = nbits <= 4;
        auto kern = small ? (flush ? k_dedisperse<uint8_t, true, true>
                                   : k_dedisperse<uint8_t, false, true>)
                          : (flush ? k_dedisperse<uint8_t, true, false>
                                   : k_dedisperse<uint8_t, false, false>);
        PSX_TRY(allow_smem(kern));
        kern<<<grid, kDdThreads, smem, st>>>(a);
    }
    return launch_status("k_dedisperse");
}

}  // namespace

extern "C" {

int psx_dedisp_create(size_t nchans, float tsamp, float fch1, float foff, psx_dedisp_plan** out)
{
    clear_error();
    if (!out || nchans == 0 || nchans > (1u << 20) || !(tsamp > 0.0f) || !(fch1 > 0.0f) ||
        !(foff < 0.0f) || !(fch1 + (float)(nchans - 1) * foff > 0.0f)) {
        set_error("psx_dedisp_create: need nchans > 0, tsamp > 0 and a band fch1 > ... > 0 "
                  "with foff < 0");
        return PSX_ERR_INVALID;
    }
    auto* p = new (std::nothrow) psx_dedisp_plan();
    if (!p) return PSX_ERR_ALLOC;
    p->nchans = nchans;
    p->tsamp = tsamp;
    p->fch1 = fch1;
    p->foff = foff;
    p->delays.resize(nchans);
    for (size_t c = 0; c < nchans; ++c) {
        float inv_f = 1.0f / (fch1 + (float)c * foff);
        float inv_0 = 1.0f / fch1;
        float diff = inv_f * inv_f - inv_0 * inv_0;
        p->delays[c] = (float)((double)kDmConst / (double)tsamp * (double)diff);
    }
    p->live.assign(nchans, 1);
    *out = p;
    return PSX_OK;
}

int psx_dedisp_destroy(psx_dedisp_plan* plan)
{
    delete plan;
    return PSX_OK;
}

int psx_dedisp_set_dm_list(psx_dedisp_plan* p, const float* h_dms, size_t n)
{
    clear_error();
    if (!p || (!h_dms && n) || n == 0) {
        set_error("psx_dedisp_set_dm_list: empty list");
        return PSX_ERR_INVALID;
    }
    for (size_t i = 0; i < n; ++i)
        if (!(h_dms[i] >= 0.0f) || !std::isfinite(h_dms[i])) {
            set_error("psx_dedisp_set_dm_list: DM %zu is negative or not finite", i);
            return PSX_ERR_INVALID;
        }
    p->dms.assign(h_dms, h_dms + n);
    p->changed();
    return PSX_OK;
}

int psx_dedisp_generate_dm_list(psx_dedisp_plan* p, float dm_start, float dm_end, float width_us,
                                float tol)
{
    clear_error();
    if (!p || !(dm_start >= 0.0f) || !(tol > 1.0f) || !(width_us >= 0.0f)) {
        set_error("psx_dedisp_generate_dm_list: need dm_start >= 0, tol > 1, width >= 0");
        return PSX_ERR_INVALID;
    }
    // next DM x from the previous p: t^2 + w^2 + a^2 x^2 + b^2 (x - p)^2
    // = tol^2 (t^2 + w^2 + a^2 p^2), times in microseconds; a is the
    // smearing across one channel per unit DM (8.3 us * foff / f_GHz^3) and
    // b = a * nchans / 4 that of a DM step across a quarter of the band
    const double ts = (double)p->tsamp * 1e6;
    const double f = ((double)p->fch1 + ((double)(p->nchans / 2) - 0.5) * (double)p->foff) * 1e-3;
    const double t2 = (double)tol * (double)tol;
    const double a = 8.3 * (double)p->foff / (f * f * f);
    const double a2 = a * a;
    const double b2 = a2 * ((double)(p->nchans * p->nchans) / 16.0);
    const double c = (ts * ts + (double)width_us * (double)width_us) * (t2 - 1.0);
    std::vector<float> list{dm_start};
    while (list.back() < dm_end) {
        double prev = (double)list.back();
        double k = c + t2 * a2 * prev * prev;
        double x = (b2 * prev + std::sqrt(-a2 * b2 * prev * prev + (a2 + b2) * k)) / (a2 + b2);
        list.push_back((float)x);
        if (list.size() > 100000000u || !(list.back() > list[list.size() - 2])) {
            set_error("psx_dedisp_generate_dm_list: the DM step does not advance");
            return PSX_ERR_INVALID;
        }
    }
    p->dms.swap(list);
    p->changed();
    return PSX_OK;
}

size_t psx_dedisp_get_dm_count(const psx_dedisp_plan* p) { return p ? p->dms.size() : 0; }

int psx_dedisp_get_dm_list(const psx_dedisp_plan* p, float* h_out, size_t cap)
{
    clear_error();
    if (!p || !h_out) return PSX_ERR_INVALID;
    if (cap < p->dms.size()) {
        set_error("psx_dedisp_get_dm_list: %zu DMs do not fit in %zu", p->dms.size(), cap);
        return PSX_ERR_OVERFLOW;
    }
    std::copy(p->dms.begin(), p->dms.end(), h_out);
    return PSX_OK;
}

int psx_dedisp_get_delay_table(const psx_dedisp_plan* p, float* h_out)
{
    if (!p || !h_out) return PSX_ERR_INVALID;
    std::copy(p->delays.begin(), p->delays.end(), h_out);
    return PSX_OK;
}

int psx_dedisp_set_killmask(psx_dedisp_plan* p, const int* h_mask)
{
    if (!p) return PSX_ERR_INVALID;
    for (size_t c = 0; c < p->nchans; ++c) p->live[c] = h_mask ? (h_mask[c] != 0) : 1;
    p->changed();
    return PSX_OK;
}

size_t psx_dedisp_get_max_delay(const psx_dedisp_plan* p) { return p ? p->max_delay() : 0; }

int psx_dedisp_set_scratch_limit(psx_dedisp_plan* p, size_t bytes)
{
    if (!p || bytes == 0) return PSX_ERR_INVALID;
    p->scratch_limit = bytes;
    return PSX_OK;
}

int psx_dedisp_execute(psx_dedisp_plan* p, size_t nsamps, const uint8_t* d_in, int nbits,
                       float* d_out, size_t out_pitch, int flags, psx_stream_t stream)
{
    clear_error();
    size_t nout = 0, pitch = 0, gulp = 0;
    PSX_TRY(check_input(p, nsamps, nbits, d_out, out_pitch, &nout));
    if (!d_in) return PSX_ERR_INVALID;
    cudaStream_t st = cs(stream);
    PSX_TRY(prepare(p, nout, nbits, st, &gulp, &pitch));
    const size_t row_bytes = p->nchans * (size_t)nbits / 8;
    const size_t md = p->max_delay();
    for (size_t g0 = 0; g0 < nout; g0 += gulp) {
        const size_t n = std::min(gulp, nout - g0);
        PSX_TRY(unpack(nbits, d_in + g0 * row_bytes, n + md, 0, pitch, p, pitch, st));
        PSX_TRY(dedisperse(p, nbits, pitch, n, d_out + g0, out_pitch, flags, st));
    }
    return PSX_OK;
}

int psx_dedisp_execute_host(psx_dedisp_plan* p, size_t nsamps, const uint8_t* h_in, int nbits,
                            float* d_out, size_t out_pitch, int flags, psx_stream_t stream)
{
    clear_error();
    size_t nout = 0, pitch = 0, gulp = 0;
    PSX_TRY(check_input(p, nsamps, nbits, d_out, out_pitch, &nout));
    if (!h_in) return PSX_ERR_INVALID;
    cudaStream_t st = cs(stream);
    PSX_TRY(prepare(p, nout, nbits, st, &gulp, &pitch));
    const size_t row_bytes = p->nchans * (size_t)nbits / 8;
    const size_t md = p->max_delay();
    // pieces of an eighth of the input (4 to 32 MB: below that a copy is not
    // worth splitting), a multiple of the unpack tile
    const size_t piece = std::min<size_t>(32u << 20, std::max<size_t>(4u << 20,
                                                                      nsamps * row_bytes / 8));
    size_t rows = std::max<size_t>(kUpRows, piece / row_bytes / kUpRows * kUpRows);
    rows = std::min(rows, round_up(std::min(gulp, nout) + md, kUpRows));
    PSX_TRY(grow(reinterpret_cast<void**>(&p->d_stage), &p->stage_cap, 2 * rows * row_bytes,
                 "input staging"));
    if (!p->copy_stream) {
        PSX_CUDA(cudaStreamCreateWithFlags(&p->copy_stream, cudaStreamNonBlocking));
        for (int i = 0; i < 2; ++i) {
            PSX_CUDA(cudaEventCreateWithFlags(&p->ev_copied[i], cudaEventDisableTiming));
            PSX_CUDA(cudaEventCreateWithFlags(&p->ev_used[i], cudaEventDisableTiming));
        }
    }
    // the copy stream starts after what `stream` already holds (the
    // staging buffers may still be read by an earlier call)
    PSX_CUDA(cudaEventRecord(p->ev_used[0], st));
    PSX_CUDA(cudaEventRecord(p->ev_used[1], st));
    size_t k = 0;
    for (size_t g0 = 0; g0 < nout; g0 += gulp) {
        const size_t n_out = std::min(gulp, nout - g0);
        const size_t n_in = n_out + md;
        size_t done = 0;  // output tiles launched
        for (size_t r0 = 0; r0 < n_in; r0 += rows, ++k) {
            const int b = (int)(k & 1);
            const size_t n = std::min(rows, n_in - r0);
            uint8_t* buf = p->d_stage + (size_t)b * rows * row_bytes;
            PSX_CUDA(cudaStreamWaitEvent(p->copy_stream, p->ev_used[b], 0));
            PSX_CUDA(cudaMemcpyAsync(buf, h_in + (g0 + r0) * row_bytes, n * row_bytes,
                                     cudaMemcpyHostToDevice, p->copy_stream));
            PSX_CUDA(cudaEventRecord(p->ev_copied[b], p->copy_stream));
            PSX_CUDA(cudaStreamWaitEvent(st, p->ev_copied[b], 0));
            const bool last = r0 + n >= n_in;
            PSX_TRY(unpack(nbits, buf, n, r0, last ? pitch - r0 : n, p, pitch, st));
            PSX_CUDA(cudaEventRecord(p->ev_used[b], st));
            // The tiles whose samples are all here run beside the next
            // pieces' copies, once they make two waves (two CTAs to an SM).
            // From pinned rows on B200, one after the other against so: 2^22
            // samples x 64 channels of 8 bits to 256 DM trials 7984, 5291 us;
            // 400,000 x 1024 of 4 bits to 100 5344, 4823.
            const size_t tile = (size_t)p->t->tile;
            const size_t ready = last || r0 + n <= md ? 0 : (r0 + n - md) / tile;
            if (last) {
                PSX_TRY(dedisperse(p, nbits, pitch, n_out, d_out + g0, out_pitch, flags, st, done));
            } else if (ready > done && (ready - done) * p->t->nblk >= 4 * (size_t)sm_count()) {
                PSX_TRY(dedisperse(p, nbits, pitch, n_out, d_out + g0, out_pitch, flags, st, done,
                                   ready));
                done = ready;
            }
        }
    }
    return PSX_OK;
}

}  // extern "C"
