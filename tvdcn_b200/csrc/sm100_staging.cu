// Staging around the tensor-core kernels: the layouts they read are made by one kernel in front of them, what they
// leave behind goes back to the caller's layout by another.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "plan.h"
#include "sm100_common.cuh"

namespace tvdcn_b200 {

namespace {

// Padded channel of the staged image -> channel of the caller's tensor, or -1: see GeoHost.
__device__ __forceinline__ int real_channel(int cp, int gran, int gran_pad) {
    if (gran == gran_pad) return cp;
    const int r = cp % gran_pad;
    return r < gran ? cp / gran_pad * gran + r : -1;
}

// ---- one launch for everything a tensor-core kernel needs prepared -------------------------------------
// A call needs up to ten small preparations (image channels-last, packed weights, zeroed accumulators, offsets
// widened to f32, ...).  As launches of their own they cost more than their work on small calls (1.5-2 us of device
// time and about as much of host time each), so they are jobs of one kernel: a block finds its job by its index.

// Largest finite magnitude of a block's values, as float bits, whose order is that of the magnitudes.
__device__ __forceinline__ uint32_t finite_magnitude(float v) {
    const uint32_t m = __float_as_uint(v) & 0x7fffffffu;
    return m < 0x7f800000u ? m : 0u;
}
__device__ void store_block_max(uint32_t m, const StageJob &j, int block) {
    __shared__ uint32_t part[8];
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) m = max(m, part[w]);
        static_cast<unsigned *>(j.part[0])[block] = m;
    }
}
// the same of two pairs of f16 values, as pairs of f16 bits
__device__ __forceinline__ uint32_t max_finite_f16x2(uint32_t m, uint32_t w) {
    w &= 0x7fff7fffu;
    return __vmaxu2(m, w & __vcmpltu2(w, 0x7c007c00u));
}
__device__ __forceinline__ uint32_t f16x2_to_magnitude(uint32_t m) {
    return __float_as_uint(__half2float(__ushort_as_half((unsigned short)max(m & 0xffffu, m >> 16))));
}

// Image [B, C, S] -> [B, S, Cpad], one 64 x 64 tile per block.  16-bit tiles are held as words of two neighbouring
// positions, the words of a channel pair 32 words apart and pairs 65 apart, 32-bit tiles in rows of 65: the
// transposing accesses are free of bank conflicts.
template <bool MAXIMA>
__device__ void stage_image_tile(const StageJob &j, int block, uint32_t *tile) {
    const int C64 = j.c_pad / 64, S64 = (j.S + 63) / 64;
    const int c0 = block % C64 * 64, s0 = block / C64 % S64 * 64;
    const int64_t b = block / C64 / S64;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (j.elem_bytes == 2) {
        const uint16_t *in = static_cast<const uint16_t *>(j.src) + b * j.C * (int64_t)j.S;
        uint32_t *out = reinterpret_cast<uint32_t *>(static_cast<uint16_t *>(j.dst) + b * j.S * (int64_t)j.c_pad);
        if (j.wide) {
            const int v = lane & 7;                                     // 8 positions s0 + 8 v ...
#pragma unroll
            for (int pass = 0; pass < 2; ++pass) {
                const int cl = warp * 8 + (lane >> 3) * 2 + pass;       // one parity per instruction
                const int c = real_channel(c0 + cl, j.gran, j.gran_pad), s = s0 + v * 8;
                uint4 x = make_uint4(0u, 0u, 0u, 0u);
                if (c >= 0 && s < j.S) x = __ldg(reinterpret_cast<const uint4 *>(in + (int64_t)c * j.S + s));
                uint32_t *w = tile + (cl >> 1) * 65 + (cl & 1) * 32 + v * 4;
                w[0] = x.x; w[1] = x.y; w[2] = x.z; w[3] = x.w;
            }
        } else {
            // all loads of a thread before the first store: they are its only latency
            const int s = s0 + 2 * lane;
            uint32_t lo[8], hi[8];
#pragma unroll
            for (int pass = 0; pass < 8; ++pass) {
                const int c = real_channel(c0 + warp * 8 + pass, j.gran, j.gran_pad);
                const uint16_t *p = in + (int64_t)max(c, 0) * j.S + s;
                lo[pass] = c >= 0 && s < j.S ? __ldg(p) : 0;
                hi[pass] = c >= 0 && s + 1 < j.S ? __ldg(p + 1) : 0;
            }
#pragma unroll
            for (int pass = 0; pass < 8; ++pass) {
                const int cl = warp * 8 + pass;
                tile[(cl >> 1) * 65 + (cl & 1) * 32 + lane] = lo[pass] | (hi[pass] << 16);
            }
        }
        __syncthreads();
        const int c = c0 + 2 * lane;
        uint32_t largest = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int s2 = warp * 4 + i;
            const uint32_t a = tile[lane * 65 + s2], bb = tile[lane * 65 + 32 + s2];
            if constexpr (MAXIMA) largest = max_finite_f16x2(max_finite_f16x2(largest, a), bb);
            const int s = s0 + 2 * s2;
            if (s < j.S) out[((int64_t)s * j.c_pad + c) >> 1] = __byte_perm(a, bb, 0x5410);
            if (s + 1 < j.S) out[((int64_t)(s + 1) * j.c_pad + c) >> 1] = __byte_perm(a, bb, 0x7632);
        }
        if constexpr (MAXIMA) store_block_max(f16x2_to_magnitude(largest), j, block);
    } else {
        const uint32_t *in = static_cast<const uint32_t *>(j.src) + b * j.C * (int64_t)j.S;
        uint32_t *out = static_cast<uint32_t *>(j.dst) + b * j.S * (int64_t)j.c_pad;
        const int v = threadIdx.x & 15, r = threadIdx.x >> 4;           // 16 vectors per row, 16 rows per pass
        if (j.wide) {
#pragma unroll
            for (int pass = 0; pass < 4; ++pass) {
                const int cl = pass * 16 + r;
                const int c = real_channel(c0 + cl, j.gran, j.gran_pad), s = s0 + v * 4;
                uint4 x = make_uint4(0u, 0u, 0u, 0u);
                if (c >= 0 && s < j.S) x = __ldg(reinterpret_cast<const uint4 *>(in + (int64_t)c * j.S + s));
                uint32_t *w = tile + cl * 65 + v * 4;
                w[0] = x.x; w[1] = x.y; w[2] = x.z; w[3] = x.w;
            }
        } else {
            const int sl = (warp & 1) * 32 + lane, s = s0 + sl;
            uint32_t x[16];
#pragma unroll
            for (int pass = 0; pass < 16; ++pass) {
                const int c = real_channel(c0 + pass * 4 + (warp >> 1), j.gran, j.gran_pad);
                x[pass] = c >= 0 && s < j.S ? __ldg(in + (int64_t)max(c, 0) * j.S + s) : 0u;
            }
#pragma unroll
            for (int pass = 0; pass < 16; ++pass) tile[(pass * 4 + (warp >> 1)) * 65 + sl] = x[pass];
        }
        __syncthreads();
#pragma unroll
        for (int pass = 0; pass < 4; ++pass) {
            const int sl = pass * 16 + r;
            const int s = s0 + sl, c = c0 + v * 4;
            if (s < j.S) {
                uint4 x;
                x.x = tile[(v * 4 + 0) * 65 + sl];
                x.y = tile[(v * 4 + 1) * 65 + sl];
                x.z = tile[(v * 4 + 2) * 65 + sl];
                x.w = tile[(v * 4 + 3) * 65 + sl];
                *reinterpret_cast<uint4 *>(out + (int64_t)s * j.c_pad + c) = x;
            }
        }
    }
}

// Weights [Cd, csg, K] -> parts of [g][tap][d'][s'] (KS) or [g][tap][s'][d'] (KD), zero in the padding.  A block takes
// up to 32 d x 8 s x all taps through shared memory: per d one contiguous run of the caller's tensor, and 16 bytes per
// thread on the way out.  Rows of the tile have odd length, so the lanes of a warp, which differ in d, meet no bank
// twice.  (Runs are contiguous in padded layouts too: a granule starts at a multiple of 64.)
constexpr int STAGE_WORDS = 64 * 65;
constexpr int PACK_S = 8;
__host__ __device__ inline int pack_d(int K) {   // most d, a power of two, whose tile fits
    int d = 32;
    while (d > 1 && d * (PACK_S * K + 1) > STAGE_WORDS) d >>= 1;
    return d;
}
template <typename TW>
__device__ void pack_weight_tile(const StageJob &j, int block, float *tile) {
    const int D = pack_d(j.K), log_d = 31 - __clz(D), run = PACK_S * j.K, row = run | 1;
    const int ns = j.c_pad / PACK_S, nd = j.cdg_pad / D;
    const int s0 = block % ns * PACK_S, d0 = block / ns % nd * D, grp = block / ns / nd;
    const int s_real = real_channel(s0, j.gran, j.gran_pad);           // C, c_pad: sampled channels of one group
    const int have = s_real < 0 ? 0 : min(PACK_S, j.gran - s0 % j.gran_pad) * j.K;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int dl = warp; dl < D; dl += 8) {
        const TW *in = static_cast<const TW *>(j.src) + (((int64_t)grp * j.cdg + d0 + dl) * j.C + s_real) * j.K;
        const int n = d0 + dl < j.cdg ? have : 0;
#pragma unroll 4
        for (int r = lane; r < run; r += 32) tile[dl * row + r] = r < n ? load_acc(in, r) : 0.f;
    }
    __syncthreads();
    // D * K vectors of 8 s (KS), or of 8 consecutive d (KD, D >= 8)
    const bool kd = j.kd && D >= 8;
    const int n_out = kd ? j.K * D : (D * j.K);
    for (int i = threadIdx.x; i < n_out; i += 256) {
        float v[8];
        int64_t o;
        const int tap = i >> log_d;
        const int64_t plane = ((int64_t)grp * j.K + tap) * j.cdg_pad * (int64_t)j.c_pad;
        int step = 1;
        if (kd) {
            const int q = i & (D - 1), sl = q & 7, dl = q & ~7;         // D / 8 vectors for each of 8 s
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = tile[(dl + e) * row + sl * j.K + tap];
            o = plane + (int64_t)(s0 + sl) * j.cdg_pad + d0 + dl;
        } else {
            const int dl = i & (D - 1);
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = tile[dl * row + e * j.K + tap];
            o = plane + (j.kd ? (int64_t)s0 * j.cdg_pad + d0 + dl : (int64_t)(d0 + dl) * j.c_pad + s0);
            step = j.kd ? j.cdg_pad : 1;
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            if (j.part[q] == nullptr) break;
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if constexpr (std::is_same<TW, __half>::value) {
                    w[e] = pack2(v[2 * e], v[2 * e + 1], __half());
                } else {
                    w[e] = pack2(v[2 * e], v[2 * e + 1], __nv_bfloat16());
                    v[2 * e] -= __uint_as_float(w[e] << 16);
                    v[2 * e + 1] -= __uint_as_float(w[e] & 0xffff0000u);
                }
            }
            uint16_t *out = static_cast<uint16_t *>(j.part[q]) + o;
            if (step == 1) {
                *reinterpret_cast<uint4 *>(out) = make_uint4(w[0], w[1], w[2], w[3]);
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) out[(int64_t)e * step] = (uint16_t)(w[e / 2] >> (16 * (e & 1)));
            }
        }
    }
}

constexpr int ZERO_BYTES = 256 * 16 * 16;     // per block
__device__ void zero_range(const StageJob &j, int block) {
    const int64_t n = j.n, at = (int64_t)block * ZERO_BYTES;            // bytes, a multiple of 4
    char *p = static_cast<char *>(j.dst) + at;
    const int64_t m = min(n - at, (int64_t)ZERO_BYTES);
    if (j.wide) {
        for (int64_t i = threadIdx.x; i < m / 16; i += 256) reinterpret_cast<uint4 *>(p)[i] = make_uint4(0u, 0u, 0u, 0u);
        if (threadIdx.x < m % 16 / 4) reinterpret_cast<uint32_t *>(p)[m / 16 * 4 + threadIdx.x] = 0u;
    } else {
        for (int64_t i = threadIdx.x; i < m / 4; i += 256) reinterpret_cast<uint32_t *>(p)[i] = 0u;
    }
}

constexpr int WIDEN_ELEMS = 256 * 8;          // per block
template <bool MAXIMA>
__device__ void widen_range(const StageJob &j, int block) {
    const int64_t end = min(j.n, ((int64_t)block + 1) * WIDEN_ELEMS);
    float *out = static_cast<float *>(j.dst);
    uint32_t largest = 0;
    for (int64_t i = (int64_t)block * WIDEN_ELEMS + threadIdx.x; i < end; i += 256) {
        const float v = j.dtype == DT_F16 ? __half2float(__ldg(static_cast<const __half *>(j.src) + i))
                                          : __bfloat162float(__ldg(static_cast<const __nv_bfloat16 *>(j.src) + i));
        out[i] = v;
        if constexpr (MAXIMA) largest = max(largest, finite_magnitude(v));
    }
    if constexpr (MAXIMA)
        if (j.part[0] != nullptr) store_block_max(largest, j, block);
}
// The maxima alone, of f32 values.
__device__ void max_range(const StageJob &j, int block) {
    const int64_t first = (int64_t)block * WIDEN_ELEMS + threadIdx.x;
    float v[WIDEN_ELEMS / 256];               // all loads in flight together
#pragma unroll
    for (int k = 0; k < WIDEN_ELEMS / 256; ++k)
        v[k] = first + k * 256 < j.n ? __ldg(static_cast<const float *>(j.src) + first + k * 256) : 0.f;
    uint32_t largest = 0;
#pragma unroll
    for (int k = 0; k < WIDEN_ELEMS / 256; ++k) largest = max(largest, finite_magnitude(v[k]));
    store_block_max(largest, j, block);
}

// Rows of S 16-bit values -> rows c_pad apart (a multiple of 8), so that TMA can read them.
constexpr int PITCH_VECS = 256 * 4;           // 8-value vectors per block
__device__ void pitch_range(const StageJob &j, int block) {
    const int vecs = j.c_pad / 8;
    const int64_t total = j.n * vecs, end = min(total, ((int64_t)block + 1) * PITCH_VECS);
    for (int64_t i = (int64_t)block * PITCH_VECS + threadIdx.x; i < end; i += 256) {
        const int64_t row = i / vecs;
        const int e0 = (int)(i - row * vecs) * 8;
        const uint16_t *in = static_cast<const uint16_t *>(j.src) + row * j.S + e0;
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t lo = e0 + 2 * k < j.S ? __ldg(in + 2 * k) : 0;
            const uint32_t hi = e0 + 2 * k + 1 < j.S ? __ldg(in + 2 * k + 1) : 0;
            w[k] = lo | (hi << 16);
        }
        *reinterpret_cast<uint4 *>(static_cast<uint16_t *>(j.dst) + row * j.c_pad + e0) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// RESIDENT blocks per SM.  Copies of large images are bound by bytes in flight: eight blocks of 32 registers moved 537 MB in
// 451 us (two calls' staging) where five of 48 took 523.  The unaligned paths keep 16 loads per thread in flight and spill
// with 32 registers, and a launch that is resident as a whole either way gains nothing.
constexpr int STAGE_RESIDENT = 5;             // what 48 registers allow
// MAXIMA: with the jobs that take maxima (a branch in the image path of every call cost 1 us of a 154 us training step).
template <int RESIDENT, bool MAXIMA>
__global__ void __launch_bounds__(256, RESIDENT) stage_kernel(const __grid_constant__ StageList list) {
    __shared__ uint32_t tile[STAGE_WORDS];
    ptx::allow_dependents();
    if (blockIdx.x == 0 && threadIdx.x == 0) ptx::publish(list.status);
    int q = 0, first = 0;
    while (q + 1 < list.n && (int)blockIdx.x >= list.job[q].end_block) first = list.job[q++].end_block;
    const StageJob &j = list.job[q];
    const int block = (int)blockIdx.x - first;
    switch (j.kind) {
        case STAGE_IMAGE: stage_image_tile<MAXIMA>(j, block, tile); break;
        case STAGE_PACK: {
            float *f = reinterpret_cast<float *>(tile);
            if (j.dtype == DT_F32) pack_weight_tile<float>(j, block, f);
            else if (j.dtype == DT_F16) pack_weight_tile<__half>(j, block, f);
            else pack_weight_tile<__nv_bfloat16>(j, block, f);
            break;
        }
        case STAGE_ZERO: zero_range(j, block); break;
        case STAGE_WIDEN: widen_range<MAXIMA>(j, block); break;
        case STAGE_PITCH: pitch_range(j, block); break;
        case STAGE_MAX:
            if constexpr (MAXIMA) max_range(j, block);
            break;
    }
}

// ---- f32 channels-last accumulator -> caller's layout ---------------------------------------------------
// [B, S, Cpad] f32 (+ bias[c]) -> [B, C, S], one 64 x 64 tile per block; wide: S a multiple of 4, aligned output
template <typename TO>
__global__ void __launch_bounds__(256) from_channels_last_kernel(const float *__restrict__ src,
                                                                 const float *__restrict__ bias, TO *__restrict__ dst,
                                                                 int C, int c_pad, int gran, int gran_pad, int S,
                                                                 int wide) {
    __shared__ float tile[64 * 65];
    ptx::grid_dependency_wait();
    const int c64 = c_pad / 64, s64 = (S + 63) / 64;
    const int c0 = (int)blockIdx.x % c64 * 64, s0 = (int)blockIdx.x / c64 % s64 * 64;
    const int64_t b = (int)blockIdx.x / c64 / s64;
    const float *in = src + b * S * (int64_t)c_pad;
    TO *out = dst + b * C * (int64_t)S;
    const int v = threadIdx.x & 15, r = threadIdx.x >> 4;
#pragma unroll
    for (int pass = 0; pass < 4; ++pass) {
        const int sl = pass * 16 + r;
        const int s = s0 + sl;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (s < S) x = __ldg(reinterpret_cast<const float4 *>(in + (int64_t)s * c_pad + c0 + v * 4));
        float *w = tile + sl * 65 + v * 4;
        w[0] = x.x; w[1] = x.y; w[2] = x.z; w[3] = x.w;
    }
    __syncthreads();
    if (wide) {
#pragma unroll
        for (int pass = 0; pass < 4; ++pass) {
            const int cl = pass * 16 + r;
            const int c = real_channel(c0 + cl, gran, gran_pad), s = s0 + v * 4;
            if (c >= 0 && s < S) {
                const float bv = bias != nullptr ? __ldg(bias + c) : 0.f;
                float x[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) x[k] = tile[(v * 4 + k) * 65 + cl] + bv;
                TO *o = out + (int64_t)c * S + s;
                if constexpr (sizeof(TO) == 4) {
                    *reinterpret_cast<float4 *>(o) = make_float4(x[0], x[1], x[2], x[3]);
                } else {
                    TO y[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) store_acc(y, k, x[k]);
                    *reinterpret_cast<uint2 *>(o) = *reinterpret_cast<const uint2 *>(y);
                }
            }
        }
    } else {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
        for (int pass = 0; pass < 16; ++pass) {
            const int cl = pass * 4 + (warp >> 1), sl = (warp & 1) * 32 + lane;
            const int c = real_channel(c0 + cl, gran, gran_pad), s = s0 + sl;
            if (c >= 0 && s < S)
                store_acc(out, (int64_t)c * S + s, tile[sl * 65 + cl] + (bias != nullptr ? __ldg(bias + c) : 0.f));
        }
    }
}

// ---- dense tensor: channel sums and / or 16-bit parts -----------------------------------------------------
// [B, C, P] read once: PARTS > 0 writes the value's bf16 parts with rows `pitch` apart (a multiple of 8), sum_out
// receives the sum over batch and space per channel.  grid (C, splits): with one block per channel a 64-channel
// tensor kept 64 of 148 SMs busy.  The partial sums of a channel are added in a fixed order by its last block.
constexpr int SUM_THREADS = 256, SUM_BLOCKS = 4;   // SUM_BLOCKS resident per SM
template <typename T, int PARTS>
__global__ void __launch_bounds__(SUM_THREADS, SUM_BLOCKS)
dense_pass_kernel(const T *__restrict__ src, uint2 *__restrict__ p0, uint2 *__restrict__ p1, uint2 *__restrict__ p2,
                  int B, int C, int P, int pitch, int wide, float *__restrict__ partial, unsigned *__restrict__ done,
                  void *__restrict__ sum_out, int sum_dtype) {
    // vectors of 16 bytes where only sums are taken, of 4 values where parts are written; UN of them in flight
    constexpr int V = PARTS == 0 && sizeof(T) == 2 ? 8 : 4, UN = 4;
    __shared__ float red[SUM_THREADS / 32];
    __shared__ bool last;
    const int c = blockIdx.x;
    const int nv = (P + V - 1) / V;
    const int64_t total = (int64_t)B * nv, per = (total + gridDim.y - 1) / gridDim.y;
    const int64_t begin = blockIdx.y * per, end = min(total, begin + per);
    float sum = 0.f;
    // (image, vector in its row) of this thread's next vector, stepped instead of divided
    int64_t i = begin + threadIdx.x;
    int64_t b = i / nv;
    int r = (int)(i - b * nv);
    const int step_b = SUM_THREADS / nv, step_r = SUM_THREADS % nv;
    while (i < end) {
        float f[UN][V];
        int64_t o[UN];
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const bool on = i < end;
            const int e0 = r * V;
            const T *in = src + (b * C + c) * (int64_t)P + e0;
            o[u] = on ? (b * C + c) * (int64_t)pitch + e0 : -1;
            if (wide) {
                if constexpr (V * sizeof(T) == 16) {
                    const uint4 x = on ? __ldg(reinterpret_cast<const uint4 *>(in)) : make_uint4(0u, 0u, 0u, 0u);
                    const T *y = reinterpret_cast<const T *>(&x);
#pragma unroll
                    for (int k = 0; k < V; ++k) f[u][k] = to_acc(y[k]);
                } else {
                    const uint2 x = on ? __ldg(reinterpret_cast<const uint2 *>(in)) : make_uint2(0u, 0u);
                    const T *y = reinterpret_cast<const T *>(&x);
#pragma unroll
                    for (int k = 0; k < V; ++k) f[u][k] = to_acc(y[k]);
                }
            } else {
#pragma unroll
                for (int k = 0; k < V; ++k) f[u][k] = on && e0 + k < P ? load_acc(in, k) : 0.f;
            }
            i += SUM_THREADS;
            b += step_b;
            r += step_r;
            if (r >= nv) { r -= nv; ++b; }
        }
#pragma unroll
        for (int u = 0; u < UN; ++u) {
#pragma unroll
            for (int k = 0; k < V; ++k) sum += f[u][k];
            if constexpr (PARTS > 0) {
                if (o[u] >= 0) {
                    uint32_t a[PARTS], bb[PARTS];
                    split_pair<PARTS, __nv_bfloat16>(f[u][0], f[u][1], a);
                    split_pair<PARTS, __nv_bfloat16>(f[u][2], f[u][3], bb);
                    p0[o[u] / 4] = make_uint2(a[0], bb[0]);
                    if constexpr (PARTS > 1) p1[o[u] / 4] = make_uint2(a[1], bb[1]);
                    if constexpr (PARTS > 2) p2[o[u] / 4] = make_uint2(a[2], bb[2]);
                }
            }
        }
    }
    if (sum_out == nullptr) return;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        float v = 0.f;
        for (int w = 0; w < SUM_THREADS / 32; ++w) v += red[w];
        partial[(int64_t)c * gridDim.y + blockIdx.y] = v;
        __threadfence();
        last = atomicAdd(&done[c], 1u) + 1u == gridDim.y;
    }
    __syncthreads();
    if (last && threadIdx.x == 0) {
        __threadfence();
        float v = 0.f;
        for (unsigned y = 0; y < gridDim.y; ++y) v += *const_cast<volatile float *>(partial + (int64_t)c * gridDim.y + y);
        if (sum_dtype == DT_F16) store_acc(static_cast<__half *>(sum_out), c, v);
        else if (sum_dtype == DT_BF16) store_acc(static_cast<__nv_bfloat16 *>(sum_out), c, v);
        else store_acc(static_cast<float *>(sum_out), c, v);
    }
}

}  // namespace

// ---- host side ----------------------------------------------------------------------------------------------
StageJob *Stager::add(int kind, int64_t blocks) {
    if (blocks <= 0) return nullptr;
    if (list_.n == StageList::MAX || blocks_ + blocks > 0x7fffffff) {
        error_ = cudaErrorInvalidValue;
        return nullptr;
    }
    StageJob &j = list_.job[list_.n++];
    memset(&j, 0, sizeof(j));
    blocks_ += blocks;
    j.kind = kind;
    j.end_block = (int)blocks_;
    return &j;
}

static bool aligned(const void *p, size_t a) { return reinterpret_cast<uintptr_t>(p) % a == 0; }

void Stager::image(const void *src, void *dst, const GeoHost &h, int elem_bytes, unsigned *maxima) {
    StageJob *j = add(STAGE_IMAGE, image_blocks(h));
    if (j == nullptr) return;
    j->src = src; j->dst = dst; j->part[0] = maxima;
    j->C = h.Cs_r; j->c_pad = h.Cs; j->gran = h.gran; j->gran_pad = h.gran_pad;
    j->S = h.S;
    j->elem_bytes = elem_bytes;
    j->wide = h.S % (16 / elem_bytes) == 0 && aligned(src, 16);
    // Row B*S of the staged image is all zeros: corners that fall outside the image (and the positions past the
    // end of the last tile) read it, so that an Inf or NaN elsewhere in the image cannot leak into results that
    // the reference computes without touching that pixel (0 x Inf = NaN).
    zero(static_cast<char *>(dst) + (size_t)h.B * h.S * h.Cs * elem_bytes, (int64_t)h.Cs * elem_bytes);
}

void Stager::pack(const void *weight, void *const *parts, const GeoHost &h, int dtype, int n_parts, bool kd) {
    const int cdg_pad = h.Cd / h.groups, csg_pad = h.Cs / h.groups;
    StageJob *j = add(STAGE_PACK, (int64_t)h.groups * (cdg_pad / pack_d(h.K)) * (csg_pad / PACK_S));
    if (j == nullptr) return;
    j->src = weight;
    for (int q = 0; q < n_parts; ++q) j->part[q] = parts[q];
    j->dtype = dtype;
    j->kd = kd;
    j->C = h.Cs_r / h.groups; j->c_pad = csg_pad; j->gran = h.gran; j->gran_pad = h.gran_pad;
    j->cdg = h.Cd_r / h.groups; j->cdg_pad = cdg_pad;
    j->K = h.K;
}

void Stager::zero(void *dst, int64_t bytes) {
    StageJob *j = add(STAGE_ZERO, (bytes + ZERO_BYTES - 1) / ZERO_BYTES);
    if (j == nullptr) return;
    j->dst = dst;
    j->n = bytes;
    j->wide = aligned(dst, 16);
}

int64_t Stager::widen_blocks(int64_t n) { return (n + WIDEN_ELEMS - 1) / WIDEN_ELEMS; }

void Stager::widen(const void *src, void *dst, int dtype, int64_t n, unsigned *maxima) {
    StageJob *j = add(STAGE_WIDEN, widen_blocks(n));
    if (j == nullptr) return;
    j->src = src; j->dst = dst; j->part[0] = maxima;
    j->dtype = dtype;
    j->n = n;
}

void Stager::max_abs(const void *src, unsigned *maxima, int64_t n) {
    StageJob *j = add(STAGE_MAX, widen_blocks(n));
    if (j == nullptr) return;
    j->src = src; j->part[0] = maxima;
    j->n = n;
}

void Stager::pitch(const void *src, void *dst, int64_t rows, int P, int pitch) {
    StageJob *j = add(STAGE_PITCH, (rows * (pitch / 8) + PITCH_VECS - 1) / PITCH_VECS);
    if (j == nullptr) return;
    j->src = src; j->dst = dst;
    j->n = rows;
    j->S = P; j->c_pad = pitch;
}

cudaError_t Stager::launch(const Status &status, cudaStream_t stream) {
    if (error_ != cudaSuccess) return error_;
    if (list_.n == 0) return cudaSuccess;
    list_.status = status;
    LaunchScope scope("stage", stream);
    bool wide = true, maxima = false;
    for (int q = 0; q < list_.n; ++q) {
        const StageJob &j = list_.job[q];
        wide = wide && (j.kind != STAGE_IMAGE || j.wide);
        maxima = maxima || (j.kind != STAGE_PACK && j.part[0] != nullptr);
    }
    const bool eight = wide && blocks_ > 148 * STAGE_RESIDENT;
    auto *kernel = eight ? (maxima ? stage_kernel<8, true> : stage_kernel<8, false>)
                         : (maxima ? stage_kernel<STAGE_RESIDENT, true> : stage_kernel<STAGE_RESIDENT, false>);
    kernel<<<(unsigned)blocks_, 256, 0, stream>>>(list_);
    return cudaGetLastError();
}

cudaError_t launch_from_channels_last_bias(const float *src, const float *bias, void *dst, int dst_dtype, const GeoHost &h,
                                           cudaStream_t stream) {
    const int64_t blocks = (int64_t)h.B * ((h.S + 63) / 64) * (h.Cs / 64);
    if (blocks > 0x7fffffff) return cudaErrorInvalidValue;
    const int wide = h.S % 4 == 0 && aligned(dst, 16);
    LaunchScope scope("from_channels_last", stream);
    auto run = [&](auto *out) {
        using TO = typename std::remove_pointer<decltype(out)>::type;
        return launch_dependent<from_channels_last_kernel<TO>>(dim3((unsigned)blocks), 256u, 0, stream, src, bias, out, h.Cs_r,
                                                               h.Cs, h.gran, h.gran_pad, h.S, wide);
    };
    if (dst_dtype == DT_F32) return run((float *)dst);
    if (dst_dtype == DT_BF16) return run((__nv_bfloat16 *)dst);
    if (dst_dtype == DT_F16) return run((__half *)dst);
    return cudaErrorInvalidValue;
}

// Blocks per channel: one wave of resident blocks at most (five per channel instead of two, 1280 blocks where 1184 are
// resident, took 22 us instead of 11 for 51 MB), but at least 8 vectors for every thread.
static int sum_splits(int B, int C, int P) {
    const int64_t vecs = (int64_t)B * ((P + 3) / 4);
    return (int)std::max<int64_t>(1, std::min<int64_t>(vecs / (SUM_THREADS * 8), 148 * SUM_BLOCKS / C));
}
int64_t dense_sum_scratch_floats(int B, int C, int P) { return (int64_t)C * sum_splits(B, C, P); }

cudaError_t launch_dense_pass(const void *src, int dtype, int n_parts, void *const *parts, int B, int C, int P, int pitch,
                              float *partial, unsigned *done, void *sum_out, int sum_dtype, cudaStream_t stream) {
    const dim3 grid((unsigned)C, (unsigned)sum_splits(B, C, P));
    const int wide = P % (dtype == DT_F32 ? 4 : 8) == 0 && aligned(src, 16);
    LaunchScope scope(n_parts == 0 ? "channel_sum" : (sum_out != nullptr ? "split_f32_channel_sum" : "split_f32"), stream);
    auto run = [&](auto *in, auto np) {
        using T = typename std::remove_const<typename std::remove_pointer<decltype(in)>::type>::type;
        constexpr int N = decltype(np)::value;
        dense_pass_kernel<T, N><<<grid, SUM_THREADS, 0, stream>>>(
            in, N > 0 ? (uint2 *)parts[0] : nullptr, N > 1 ? (uint2 *)parts[1] : nullptr,
            N > 2 ? (uint2 *)parts[2] : nullptr, B, C, P, pitch, wide, partial, done, sum_out, sum_dtype);
        return cudaGetLastError();
    };
    if (dtype == DT_F32 && n_parts == 0) return run((const float *)src, std::integral_constant<int, 0>());
    if (dtype == DT_F32 && n_parts == 2) return run((const float *)src, std::integral_constant<int, 2>());
    if (dtype == DT_F32 && n_parts == 3) return run((const float *)src, std::integral_constant<int, 3>());
    if (dtype == DT_F16 && n_parts == 0) return run((const __half *)src, std::integral_constant<int, 0>());
    if (dtype == DT_BF16 && n_parts == 0) return run((const __nv_bfloat16 *)src, std::integral_constant<int, 0>());
    return cudaErrorInvalidValue;
}

}  // namespace tvdcn_b200
