// Pieces shared by the tcgen05 kernels: the sampling plan of a tile, the swizzled shared-memory tile
// layout the producers write, tensor-map creation, layout staging kernels.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <type_traits>
#include <utility>

#include "common.cuh"
#include "kernels.h"
#include "sm100_ptx.cuh"

namespace tvdcn_b200 {

template <int DIM>
inline Geo<DIM> geo_from_host(const GeoHost &h) {
    Geo<DIM> g;
    g.B = h.B; g.Cs = h.Cs; g.Cd = h.Cd; g.groups = h.groups; g.og = h.og; g.mg = h.mg; g.K = h.K;
    g.S = h.S; g.P = h.P;
    g.csg = h.Cs / h.groups;
    g.cdg = h.Cd / h.groups;
    g.cs_per_og = h.og > 0 ? h.Cs / h.og : h.Cs;
    g.cs_per_mg = h.mg > 0 ? h.Cs / h.mg : h.Cs;
    g.Cd_r = h.Cd_r;
    g.cdg_r = h.Cd_r / h.groups;
    g.BP = (long long)h.B * h.P;
    for (int a = 0; a < DIM; ++a) {
        g.img[a] = h.img[a]; g.grid[a] = h.grid[a]; g.ker[a] = h.ker[a];
        g.stride[a] = h.stride[a]; g.pad[a] = h.pad[a]; g.dil[a] = h.dil[a];
    }
    return g;
}

template <int MODE>
struct Mode {
    static constexpr bool F32 = MODE == TC_SPLIT || MODE == TC_F32_WIDE;       // type of image, weight and dense tensor
    static constexpr bool HALF = MODE == TC_F16 || MODE == TC_F16_WIDE;
    static constexpr bool BLEND_F32 = MODE >= TC_SPLIT;                        // corners are blended in f32
    static constexpr int COL_PARTS = MODE == TC_F32_WIDE ? 3 : (MODE >= TC_SPLIT ? 2 : 1);
    static constexpr int MAT_PARTS = MODE == TC_F32_WIDE ? 3 : (MODE == TC_SPLIT ? 2 : 1);
    static constexpr bool LOW_ACC = F32;                                       // the small products have accumulators
    using T16 = typename std::conditional<HALF, __half, __nv_bfloat16>::type;  // type of the operands
};
constexpr int TILE_POS = 128;       // grid positions per tile = TMEM lanes
constexpr int CHUNK_C = 64;         // channels per K chunk = one 128-byte swizzle row of 16-bit values
constexpr int A_TILE_BYTES = TILE_POS * 128;

// Byte offset of 16-byte chunk `chunk` (0..7) of row `row` inside a 128-byte-swizzled tile.
__device__ __forceinline__ uint32_t sw128_offset(int row, int chunk) {
    return (uint32_t)row * 128u + (uint32_t)((chunk ^ (row & 7)) << 4);
}

// Decoded grid position of one thread.
template <int DIM>
struct PosInfo {
    bool valid;
    int b, p;
    int base[DIM];  // grid * stride - pad per axis
};

template <int DIM>
__device__ __forceinline__ void decode_in_image(const Geo<DIM> &g, PosInfo<DIM> &pi) {
    int r = pi.p;
#pragma unroll
    for (int a = DIM - 1; a >= 0; --a) {
        const int c = r % g.grid[a];
        r /= g.grid[a];
        pi.base[a] = c * g.stride[a] - g.pad[a];
    }
}

template <int DIM>
__device__ __forceinline__ PosInfo<DIM> decode_position(const Geo<DIM> &g, long long idx) {
    PosInfo<DIM> pi;
    pi.valid = idx < g.BP;
    const int i = pi.valid ? (int)idx : 0;             // fewer than 2^31 positions
    pi.b = i / g.P;
    pi.p = i - pi.b * g.P;
    decode_in_image<DIM>(g, pi);
    return pi;
}

// ---- sampling plan ------------------------------------------------------------------------------------
// One slot per (position, tap): for each of the NC = 2^DIM corners of the cell where the corner's 64-channel row
// starts in the channels-last image, in 16-byte units, then for each corner its interpolation weight times the mask
// -- as a packed 16-bit pair (w, w) where the corners are blended in 16 bits, else as f32 bits.  Rows and weights are
// apart so that a producer reads the weights only when it blends: they would hold NC registers per position in flight.
// Out-of-image corners point at the row of zeros behind the image with weight 0, so the producers load
// unconditionally.
template <int NC>
__device__ __forceinline__ void load_slot_half(uint32_t (&out)[NC], const uint32_t *p) {
    if constexpr (NC == 2) {
        const uint2 x = *reinterpret_cast<const uint2 *>(p);
        out[0] = x.x; out[1] = x.y;
    } else {
#pragma unroll
        for (int c = 0; c < NC; c += 4) {
            const uint4 x = *reinterpret_cast<const uint4 *>(p + c);
            out[c] = x.x; out[c + 1] = x.y; out[c + 2] = x.z; out[c + 3] = x.w;
        }
    }
}
template <int NC>
__device__ __forceinline__ void store_slot_half(uint32_t *p, const uint32_t (&v)[NC]) {
    if constexpr (NC == 2) {
        *reinterpret_cast<uint2 *>(p) = make_uint2(v[0], v[1]);
    } else {
#pragma unroll
        for (int c = 0; c < NC; c += 4) *reinterpret_cast<uint4 *>(p + c) = make_uint4(v[c], v[c + 1], v[c + 2], v[c + 3]);
    }
}

// Offsets and mask of one (position, tap, groups): loaded early, turned into plan entries later, so that the
// global-memory latency overlaps the sampling of the previous chunk.
template <int DIM>
struct RawCoords {
    float off[DIM];
    float m;
};

// The power of two of a ColumnRange, 2^15 / (bounds of the two maxima); the 128 planner threads, thread t among them,
// take part and all get it.  It is the planners' work because they have the loads of their first coordinates to wait for
// meanwhile.  part: 8 words of shared memory; BAR: a named barrier of theirs.
template <int BAR>
__device__ __forceinline__ float column_scale(const ColumnRange &r, int t, uint32_t *part) {
    constexpr int U = 4;
    uint32_t m[2] = {0u, 0u};
    for (int i0 = t; i0 < max(r.n_img, r.n_mask); i0 += 128 * U) {
        uint32_t a[U], b[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const int i = i0 + 128 * k;
            a[k] = i < r.n_img ? __ldg(r.img + i) : 0u;
            b[k] = i < r.n_mask ? __ldg(r.mask + i) : 0u;
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
            m[0] = max(m[0], a[k]);
            m[1] = max(m[1], b[k]);
        }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        m[q] = __reduce_max_sync(0xffffffffu, m[q]);
        if ((t & 31) == 0) part[q * 4 + (t >> 5)] = m[q];
    }
    asm volatile("bar.sync %0, 128;" ::"n"(BAR) : "memory");
    int e = 15;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const uint32_t v = max(max(part[q * 4], part[q * 4 + 1]), max(part[q * 4 + 2], part[q * 4 + 3]));
        // a normal value is below 2^(biased exponent - 126); zero and subnormals: as if 1, they need no factor
        if (v >= 0x00800000u) e -= (int)(v >> 23) - 126;
    }
    return __uint_as_float((uint32_t)(127 + min(max(e, -120), 120)) << 23);
}
__device__ __forceinline__ float inverse_of_power_of_two(float v) {
    return __uint_as_float((254u << 23) - __float_as_uint(v));
}

template <int MODE>
__device__ __forceinline__ uint32_t encode_weight(float w) {
    if constexpr (Mode<MODE>::BLEND_F32) {
        return __float_as_uint(w);
    } else if constexpr (MODE == TC_F16) {
        const __half2 h = __float2half2_rn(w);
        return *reinterpret_cast<const uint32_t *>(&h);
    } else {
        const __nv_bfloat162 h = __float2bfloat162_rn(w);
        return *reinterpret_cast<const uint32_t *>(&h);
    }
}

// Kernel coordinates of a tap (axis 0 outermost).
template <int DIM>
__device__ __forceinline__ void tap_coords(const Geo<DIM> &g, int tap, int (&tc)[DIM]) {
    int r = tap;
#pragma unroll
    for (int a = DIM - 1; a >= 0; --a) {
        tc[a] = r % g.ker[a];
        r /= g.ker[a];
    }
}

// Writes the plan slot of one position and tap, whose kernel coordinates are tc (the divisions by the kernel extents were
// a quarter of the instructions of a slot, and a planner thread makes slots back to back).  row_scale = Cs * element
// size / 16; weight_scale: see ColumnRange.
template <int DIM, int MODE>
__device__ __forceinline__ void build_plan_at(const Geo<DIM> &g, const PosInfo<DIM> &pi, const RawCoords<DIM> &rc,
                                              bool deformable, const int (&tc)[DIM], uint32_t row_scale,
                                              uint32_t *slot, float weight_scale = 1.f) {
    constexpr int NC = 1 << DIM;
    int fl[DIM];
    float fr[DIM];
#pragma unroll
    for (int a = 0; a < DIM; ++a) {
        const int base = pi.base[a] + tc[a] * g.dil[a];
        if (deformable) {
            const float pos = (float)base + rc.off[a];
            const float f = floorf(pos);
            fl[a] = (int)f;
            fr[a] = pos - f;
        } else {
            fl[a] = base;
            fr[a] = 0.f;
        }
    }
    uint32_t rows[NC], ws[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        bool ok = pi.valid && (deformable || c == 0);
        int flat = 0;
        float w = MODE == TC_F16_WIDE ? rc.m * weight_scale : rc.m;
#pragma unroll
        for (int a = 0; a < DIM; ++a) {
            const int bit = (c >> (DIM - 1 - a)) & 1;
            const int i = (int)((unsigned)fl[a] + (unsigned)bit);
            ok = ok && ((unsigned)i < (unsigned)g.img[a]);
            flat = flat * g.img[a] + i;
            w *= bit ? fr[a] : (1.f - fr[a]);
        }
        // out-of-image corners read the row of zeros that follows the staged image
        rows[c] = (uint32_t)(ok ? pi.b * g.S + flat : g.B * g.S) * row_scale;
        ws[c] = encode_weight<MODE>(ok ? w : 0.f);
    }
    store_slot_half<NC>(slot, rows);
    store_slot_half<NC>(slot + NC, ws);
}

__device__ __forceinline__ void unpack8(const uint4 &v, float (&f)[8], __nv_bfloat16) {
    const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[2 * i] = __uint_as_float(u[i] << 16);
        f[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
    }
}
__device__ __forceinline__ void unpack8(const uint4 &v, float (&f)[8], __half) {
    const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 p = __half22float2(*reinterpret_cast<const __half2 *>(&u[i]));
        f[2 * i] = p.x;
        f[2 * i + 1] = p.y;
    }
}
__device__ __forceinline__ uint32_t pack2(float a, float b, __nv_bfloat16) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ uint32_t pack2(float a, float b, __half) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}

// acc (+)= w * v on packed 16-bit pairs (the blend of 16-bit data stays in its own precision: the result is
// rounded to that precision for the tensor core anyway)
template <typename T16>
__device__ __forceinline__ uint32_t fma2(uint32_t w, uint32_t v, uint32_t acc) {
    if constexpr (std::is_same<T16, __half>::value) {
        const __half2 r = __hfma2(*reinterpret_cast<const __half2 *>(&w), *reinterpret_cast<const __half2 *>(&v),
                                  *reinterpret_cast<const __half2 *>(&acc));
        return *reinterpret_cast<const uint32_t *>(&r);
    } else {
        const __nv_bfloat162 r = __hfma2(*reinterpret_cast<const __nv_bfloat162 *>(&w),
                                         *reinterpret_cast<const __nv_bfloat162 *>(&v),
                                         *reinterpret_cast<const __nv_bfloat162 *>(&acc));
        return *reinterpret_cast<const uint32_t *>(&r);
    }
}
template <typename T16>
__device__ __forceinline__ uint32_t mul2(uint32_t w, uint32_t v) {
    if constexpr (std::is_same<T16, __half>::value) {
        const __half2 r = __hmul2(*reinterpret_cast<const __half2 *>(&w), *reinterpret_cast<const __half2 *>(&v));
        return *reinterpret_cast<const uint32_t *>(&r);
    } else {
        const __nv_bfloat162 r = __hmul2(*reinterpret_cast<const __nv_bfloat162 *>(&w),
                                         *reinterpret_cast<const __nv_bfloat162 *>(&v));
        return *reinterpret_cast<const uint32_t *>(&r);
    }
}

// A value as PARTS 16-bit parts of decreasing magnitude: part k is what rounding leaves of the first k.
template <int PARTS, typename T16>
__device__ __forceinline__ void split_pair(float a, float b, uint32_t (&out)[PARTS]) {
#pragma unroll
    for (int k = 0; k < PARTS; ++k) {
        out[k] = pack2(a, b, T16());
        if (k + 1 < PARTS) {
            if constexpr (std::is_same<T16, __half>::value) {
                const float2 r = __half22float2(*reinterpret_cast<const __half2 *>(&out[k]));
                a -= r.x;
                b -= r.y;
            } else {
                a -= __uint_as_float(out[k] << 16);
                b -= __uint_as_float(out[k] & 0xffff0000u);
            }
        }
    }
}

// Samples `nvpos` virtual positions x 64 channels into 128-byte-swizzled tiles (row = position).  Virtual
// position v belongs to sub-tile v / pos_per_sub (tiles `sub_bytes` apart, each with its own first channel
// chan16[sub], in 16-byte units) and is row v % pos_per_sub of it.  plan + v * 2 * NC is its slot;
// the parts of a column (see the modes) are tiles `part_bytes` apart.
// All NT threads take part; each keeps the loads of IB positions in flight together so that global-memory
// latency is overlapped.  nvpos must be a multiple of (NT / lanes-per-position) * IB.
//   16-bit data: 8 lanes x 8 channels per position; f32 data: 16 lanes x 4 channels.
template <int NC, int MODE, int NT, int IB>
__device__ __forceinline__ void produce_tiles(uint8_t *tiles, uint32_t part_bytes, uint32_t sub_bytes, int pos_per_sub,
                                              int nvpos, const uint4 *__restrict__ img16, const uint32_t *chan16,
                                              const uint32_t *plan, int tid) {
    using M = Mode<MODE>;
    using T16 = typename M::T16;
    constexpr int LPP = M::F32 ? 16 : 8;
    constexpr int PPI = NT / LPP;
    const int part = tid & (LPP - 1);
    const int psub = tid / LPP;
    for (int v0 = 0; v0 < nvpos; v0 += PPI * IB) {
        uint4 v[IB][NC];
#pragma unroll
        for (int i = 0; i < IB; ++i) {
            const int vp = v0 + i * PPI + psub;
            const uint4 *src = img16 + chan16[(v0 + i * PPI) / pos_per_sub] + part;
            uint32_t rows[NC];
            load_slot_half<NC>(rows, plan + vp * 2 * NC);
#pragma unroll
            for (int c = 0; c < NC; ++c) v[i][c] = __ldg(src + rows[c]);
        }
#pragma unroll
        for (int i = 0; i < IB; ++i) {
            const int vp = v0 + i * PPI + psub;
            const int sub = (v0 + i * PPI) / pos_per_sub;
            const int pos = vp - sub * pos_per_sub;
            uint8_t *dst = tiles + (size_t)sub * sub_bytes;
            uint32_t w[NC];
            load_slot_half<NC>(w, plan + vp * 2 * NC + NC);
            if constexpr (!M::BLEND_F32) {
                uint4 o;
                o.x = mul2<T16>(w[0], v[i][0].x);
                o.y = mul2<T16>(w[0], v[i][0].y);
                o.z = mul2<T16>(w[0], v[i][0].z);
                o.w = mul2<T16>(w[0], v[i][0].w);
#pragma unroll
                for (int c = 1; c < NC; ++c) {
                    o.x = fma2<T16>(w[c], v[i][c].x, o.x);
                    o.y = fma2<T16>(w[c], v[i][c].y, o.y);
                    o.z = fma2<T16>(w[c], v[i][c].z, o.z);
                    o.w = fma2<T16>(w[c], v[i][c].w, o.w);
                }
                *reinterpret_cast<uint4 *>(dst + sw128_offset(pos, part)) = o;
            } else if constexpr (!M::F32) {
                float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const float wf = __uint_as_float(w[c]);
                    float f[8];
                    unpack8(v[i][c], f, T16());
#pragma unroll
                    for (int k = 0; k < 8; ++k) acc[k] = fmaf(wf, f[k], acc[k]);
                }
                uint32_t p[4][M::COL_PARTS];
#pragma unroll
                for (int k = 0; k < 4; ++k) split_pair<M::COL_PARTS, T16>(acc[2 * k], acc[2 * k + 1], p[k]);
#pragma unroll
                for (int q = 0; q < M::COL_PARTS; ++q)
                    *reinterpret_cast<uint4 *>(dst + q * part_bytes + sw128_offset(pos, part)) =
                        make_uint4(p[0][q], p[1][q], p[2][q], p[3][q]);
            } else {
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const float wf = __uint_as_float(w[c]);
                    acc[0] = fmaf(wf, __uint_as_float(v[i][c].x), acc[0]);
                    acc[1] = fmaf(wf, __uint_as_float(v[i][c].y), acc[1]);
                    acc[2] = fmaf(wf, __uint_as_float(v[i][c].z), acc[2]);
                    acc[3] = fmaf(wf, __uint_as_float(v[i][c].w), acc[3]);
                }
                uint32_t p01[M::COL_PARTS], p23[M::COL_PARTS];
                split_pair<M::COL_PARTS, T16>(acc[0], acc[1], p01);
                split_pair<M::COL_PARTS, T16>(acc[2], acc[3], p23);
                const uint32_t off = sw128_offset(pos, part >> 1) + (uint32_t)(part & 1) * 8u;
#pragma unroll
                for (int q = 0; q < M::COL_PARTS; ++q)
                    *reinterpret_cast<uint2 *>(dst + q * part_bytes + off) = make_uint2(p01[q], p23[q]);
            }
        }
    }
}

// a / b where b is often 1: a division costs a kernel's first instructions some hundred cycles
__host__ __device__ __forceinline__ int div_often_one(int a, int b) { return b == 1 ? a : a / b; }

// ---- host helpers ---------------------------------------------------------------------------------
// Launches a kernel as a dependent of the one before it in the stream (see ptx::allow_dependents).  The kernel is granted
// all dynamic shared memory there is once per device, not its launch's share on every launch (host time, and two threads
// would overwrite each other's grant).
template <auto Kern, typename... Args>
inline cudaError_t launch_dependent(dim3 grid, unsigned block, size_t smem, cudaStream_t stream, const Args &...args) {
    static std::atomic<uint64_t> granted{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev < 64 ? 1ull << dev : 0;
    if ((granted.load(std::memory_order_acquire) & bit) == 0) {
        cudaFuncAttributes fa;
        e = cudaFuncGetAttributes(&fa, Kern);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(Kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - (int)fa.sharedSizeBytes);
        if (e != cudaSuccess) return e;
        granted.fetch_or(bit, std::memory_order_acq_rel);
    }
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, Kern, args...);
}

// 16-bit tiled tensor map with 128-byte swizzle; dims innermost first.  Returns false when the driver
// entry point is unavailable or rejects the description.
bool make_tensor_map_16bit(CUtensorMap *map, const void *base, int rank, const uint64_t *dims,
                           const uint64_t *strides_bytes /* rank-1 entries */, const uint32_t *box);
// The maps of an operand's parts, all of one shape; unused entries repeat the first.
inline bool make_part_maps(CUtensorMap *maps /* 3 */, const void *const *parts, int n, int rank, const uint64_t *dims,
                           const uint64_t *strides_bytes, const uint32_t *box) {
    for (int k = 0; k < n; ++k)
        if (!make_tensor_map_16bit(&maps[k], parts[k], rank, dims, strides_bytes, box)) return false;
    for (int k = n; k < 3; ++k) maps[k] = maps[0];
    return true;
}

template <typename F>
inline cudaError_t with_mode(int mode, F &&f) {
    switch (mode) {
        case TC_BF16: return f(std::integral_constant<int, TC_BF16>());
        case TC_F16: return f(std::integral_constant<int, TC_F16>());
        case TC_SPLIT: return f(std::integral_constant<int, TC_SPLIT>());
        case TC_BF16_WIDE: return f(std::integral_constant<int, TC_BF16_WIDE>());
        case TC_F16_WIDE: return f(std::integral_constant<int, TC_F16_WIDE>());
        case TC_F32_WIDE: return f(std::integral_constant<int, TC_F32_WIDE>());
    }
    return cudaErrorInvalidValue;
}

}  // namespace tvdcn_b200
