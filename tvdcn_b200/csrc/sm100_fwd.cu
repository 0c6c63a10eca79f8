// Tensor-core "sample -> GEMM" kernel (tcgen05 / TMEM).
//
//   dense[b, d, p] = bias[d] + sum_{tap, s'} W[d, s', tap] * mask * sample(img[b, s], pos(b, og(s), tap, p))
//
// It is an implicit GEMM  D[128 positions x BN dense channels] += A[128 x 64] * B[BN x 64]^T  over K chunks
// of 64 channels of one kernel tap.  The A tile (the im2col columns of the reference,
// tvdcn/csrc/ops/cuda/deform_conv2d_common_kernels.cu:138-192) is never written to global memory: sixteen
// producer warps sample a channels-last copy of the image straight into the 128-byte-swizzled shared
// memory layout the tensor core reads.  The B tile (weights packed per tap) arrives by TMA.  One thread
// issues tcgen05.mma with the accumulator in tensor memory; the producer warps then read it back
// (tcgen05.ld: lane = position) and store NCHW with the bias added, so the reference's output_buf
// transpose and bias pass (tvdcn/csrc/ops/cuda/deform_conv2d_kernel.cpp:371-380) are gone too.
//
// Work is cut into chunk-sized units ordered tile by tile; the grid has at most one CTA per SM and each takes an equal,
// contiguous range of units.  So a CTA runs through its tiles without starting over (2048 tiles x 8 groups of 5 chunks
// were 16384 CTAs whose start-up and epilogue outlasted their main loops), the SMs finish together where the tiles make
// 5.3 waves, and a handful of tiles with long reductions is spread over the chip, two CTAs to a tile.  A tile that several CTAs share
// is summed from partial results in the workspace by whichever of them arrives last, in a fixed order; nobody waits.
//
// Warp roles (896 threads): warps 0-15 producers, 16-19 planners, 20-23 epilogue, 24 MMA issue + TMEM owner, 25 TMA,
// 26-27 idle.  The planners turn sampling coordinates into plan entries a few chunks ahead; the epilogue of a tile runs
// under the main loop of the next one where tensor memory holds two sets of accumulators.
#include <algorithm>
#include <type_traits>

#include "plan.h"
#include "sm100_common.cuh"

namespace tvdcn_b200 {

// How the chunk units of a launch are shared out.  The same arithmetic on host and device.
struct FwdWork {
    int n_tiles, tiles_y;   // position tiles x tiles_y; tile t covers positions t / tiles_y, (group, dense tile) t % tiles_y
    int n_chunks;           // units per tile: taps x 64-channel chunks
    int ctas;
    int whole;              // no tile is shared
    int halves;             // every tile of an odd number of chunks is shared by two CTAs, 2 t (one chunk more) and 2 t + 1
    int base, extra;        // CTA c has `base` units (whole: tiles), the first `extra` CTAs (halves: the even ones) one more

    // First unit of CTA c.  A piece of one chunk is not worth its trip through the workspace: it stays with its neighbour.
    // (32-bit arithmetic: every role of every CTA starts with it.)
    __host__ __device__ int bound(int c) const {
        const int b = c * base + (halves ? (c + 1) >> 1 : (c < extra ? c : extra));
        if (whole) return b * n_chunks;
        const int r = b % n_chunks;
        return r == 1 ? b - 1 : (r == n_chunks - 1 ? b + 1 : b);
    }
    // the CTA that has a unit
    __host__ __device__ int owner(int unit) const {
        if (halves) return 2 * unit / n_chunks;
        const int wide = extra * (base + 1);
        int c = unit < wide ? unit / (base + 1) : extra + (unit - wide) / base;
        if (c + 1 < ctas && bound(c + 1) <= unit) ++c;     // the neighbour's, after its bound was moved by one
        if (bound(c) > unit) --c;
        return c;
    }
};

// Chunks in the order the CTA takes them: tap innermost, so the taps of one 64-channel chunk sample the same slab of the
// image, which then stays in L1 for all of them; then the chunk, the (group, dense tile), the positions.
struct ChunkIter {
    int tap, cc, y, x;
    __device__ __forceinline__ void start(const FwdWork &w, int unit, int taps) {
        const int tile = unit / w.n_chunks, j = unit - tile * w.n_chunks;
        x = div_often_one(tile, w.tiles_y);
        y = tile - x * w.tiles_y;
        cc = j < taps ? 0 : j / taps;
        tap = j - cc * taps;
    }
    // returns whether a new tile begins
    __device__ __forceinline__ bool next(int taps, int chunks, int tiles_y) {
        if (++tap < taps) return false;
        tap = 0;
        if (++cc < chunks) return false;
        cc = 0;
        if (++y == tiles_y) {
            y = 0;
            ++x;
        }
        return true;
    }
};

template <int DIM>
struct FwdParams {
    Geo<DIM> g;
    const void *img_cl;     // [B, S, Cs], data type of the problem
    const float *offset;    // may be null
    const float *mask;      // may be null
    const float *bias;      // may be null
    ColumnRange range;      // TC_F16_WIDE
    void *out;              // [B, Cd, P], data type of the problem
    Status status;
    float *partial;         // partial sums of shared tiles: two [bn / 4][128] float4 per CTA (null: no tile is shared)
    unsigned *arrived;      // per tile, zeroed
    FwdWork work;
    int bn;                 // dense channels per tile: 64, 128 or 256
    int stages;
};

namespace {

constexpr int PRODUCER_WARPS = 16;
constexpr int PRODUCERS = PRODUCER_WARPS * 32;
// Producer groups: group q samples chunks j with j % groups == q.  Two groups for 16-bit data (three stages: one
// group's gathers are in flight while the other blends); one group of all 16 warps for f32 data, whose two stages
// would otherwise make each group wait for the MMA of its own previous chunk.
__host__ __device__ constexpr int producer_groups_of(int mode) {
    return mode == TC_SPLIT || mode == TC_F32_WIDE ? 1 : 2;
}
constexpr int PLANNER_WARPS = 4;                  // one planner thread per tile position
constexpr int PLAN_BUFS = 4;
// The warpgroups re-divide the registers at kernel start (launch: 72 each, 7 x 72 = 504): the producers, who keep the
// gathers of several positions in flight, take FWD_REGS_PRODUCER, the others give up what that costs:
// 4 x 88 + 56 + 64 + 32 = 504.
constexpr int EPI_WARP0 = PRODUCER_WARPS + PLANNER_WARPS;
constexpr int EPI_WARPS = 4;                      // one per quarter of the TMEM lanes
constexpr int MMA_WARP = EPI_WARP0 + EPI_WARPS;
constexpr int TMA_WARP = MMA_WARP + 1;
constexpr int FWD_THREADS = (TMA_WARP + 3) * 32;
static_assert(FWD_THREADS == 896, "seven warpgroups");
constexpr int FWD_REGS_PRODUCER = 88, FWD_REGS_PLANNER = 56, FWD_REGS_EPILOGUE = 64, FWD_REGS_ISSUE = 32;
constexpr int FWD_MAX_TAPS = 512;                 // taps whose kernel coordinates a CTA tabulates (more: SIMT kernels)

template <int DIM, int MODE>
__global__ void __launch_bounds__(FWD_THREADS, 1)
dcn_fwd_tc_kernel(const FwdParams<DIM> P, const __grid_constant__ CUtensorMap tmap0,
                  const __grid_constant__ CUtensorMap tmap1, const __grid_constant__ CUtensorMap tmap2) {
    constexpr int NC = 1 << DIM;
    using M = Mode<MODE>;
    constexpr int CPARTS = M::COL_PARTS, MPARTS = M::MAT_PARTS;
    constexpr int PGROUPS = producer_groups_of(MODE);
    constexpr int GROUP_WARPS = PRODUCER_WARPS / PGROUPS;
    constexpr int GROUP_THREADS = GROUP_WARPS * 32;
    using T16 = typename M::T16;
    const Geo<DIM> &g = P.g;

    extern __shared__ uint8_t smem_raw[];
    // align by offset, not by integer round-trip, so that the compiler keeps these as shared-memory pointers
    uint8_t *smem = smem_raw + ((1024u - (ptx::smem_u32(smem_raw) & 1023u)) & 1023u);
    const int S = P.stages;
    const int BN = P.bn;
    const uint32_t a_stage_bytes = A_TILE_BYTES * CPARTS;
    const uint32_t b_part_bytes = (uint32_t)BN * 128u;
    const uint32_t b_stage_bytes = b_part_bytes * MPARTS;
    uint8_t *sA = smem;
    uint8_t *sB = sA + (size_t)S * a_stage_bytes;
    uint32_t *plan = reinterpret_cast<uint32_t *>(sB + (size_t)S * b_stage_bytes);   // slots [PLAN_BUFS][128][2 NC]
    uint64_t *bars = reinterpret_cast<uint64_t *>(plan + PLAN_BUFS * 2 * NC * TILE_POS);
    uint64_t *full_a = bars;
    uint64_t *full_b = bars + S;
    uint64_t *empty = bars + 2 * S;
    uint64_t *acc_full = bars + 3 * S;      // [2] MMA -> epilogue: a tile's (or a piece's) sums are complete
    uint64_t *acc_empty = acc_full + 2;     // [2] epilogue -> MMA
    uint64_t *acc_last = acc_empty + 2;     // MMA -> producers: the sums of the CTA's last piece are complete
    uint64_t *plan_full = acc_last + 1;
    uint64_t *plan_empty = plan_full + PLAN_BUFS;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(plan_empty + PLAN_BUFS);
    uint32_t *last_flags = tmem_slot + 1;     // [2] epilogue warps, producers: this CTA brought the last piece

    // kernel coordinates of every tap, so that the planners do not divide by the kernel extents per chunk
    __shared__ int16_t tap_tab[FWD_MAX_TAPS * DIM];
    for (int tp = threadIdx.x; tp < g.K; tp += FWD_THREADS) {
        int tc[DIM];
        tap_coords<DIM>(g, tp, tc);
#pragma unroll
        for (int a = 0; a < DIM; ++a) tap_tab[tp * DIM + a] = (int16_t)tc[a];
    }
    // TC_F16_WIDE: the factor of the sums, written by the planners before their first plan and read behind a tile's last MMA
    __shared__ float out_scale;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_n = g.cdg / BN, chunks = g.csg / CHUNK_C;
    const FwdWork &W = P.work;
    const int n_chunks = W.n_chunks;
    const int unit0 = W.bound((int)blockIdx.x);
    const int n_local = W.bound((int)blockIdx.x + 1) - unit0;
    // f32 data: the tensor core's f32 accumulation rounds toward zero, so the error of one accumulator grows
    // with the number of MMAs added into it.  Chunks go round-robin into NACC accumulators for the products of the
    // leading parts (one chain near 80 MMAs, 4 per chunk, where half of tensor memory holds that many), all smaller products
    // into one more; the epilogue adds them (round to nearest).  Two-part operands whose 12 MMAs per chunk make no
    // chain longer than 250 keep one accumulator for everything: short reductions feel every extra TMEM read.
    int NACC = 1, acc_sets = 1;
    if (M::LOW_ACC && (MODE != TC_SPLIT || n_chunks > 20)) {
        acc_sets = 2;
        while (acc_sets * 2 * BN <= 256 && (acc_sets - 1) * 20 < n_chunks) acc_sets *= 2;
        NACC = acc_sets - 1;
    }
    const bool low_acc = acc_sets > 1;
    const uint32_t low_col = (uint32_t)(NACC * BN);   // accumulator of the small products
    const uint32_t set_cols = (uint32_t)(acc_sets * BN);
    const int acc_bufs = set_cols <= 256 ? 2 : 1;     // sets of accumulators: the epilogue reads one, the MMA fills the other
    const uint32_t ncols = set_cols * (uint32_t)acc_bufs;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            ptx::mbar_init(&full_a[s], GROUP_WARPS);
            ptx::mbar_init(&full_b[s], 1);
            ptx::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            ptx::mbar_init(&acc_full[b], 1);
            ptx::mbar_init(&acc_empty[b], EPI_WARPS);
        }
        ptx::mbar_init(acc_last, 1);
        for (int b = 0; b < PLAN_BUFS; ++b) {
            ptx::mbar_init(&plan_full[b], PLANNER_WARPS);
            ptx::mbar_init(&plan_empty[b], GROUP_WARPS);
        }
        ptx::fence_mbar_init();
    }
    if (warp == TMA_WARP && lane == 0) {
        ptx::prefetch_tmap(&tmap0);
        if (MPARTS > 1) ptx::prefetch_tmap(&tmap1);
        if (MPARTS > 2) ptx::prefetch_tmap(&tmap2);
    }
    if (warp == MMA_WARP) {
        ptx::tmem_alloc(tmem_slot, ncols);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    ptx::grid_dependency_wait();     // nothing above reads what an earlier kernel wrote

    constexpr uint32_t ESZ = M::F32 ? 4 : 2;
    const uint4 *img16 = reinterpret_cast<const uint4 *>(P.img_cl);

    constexpr int CW = 16;                            // dense channels the epilogue handles at a time
    // n consecutive dense channels of one position, from channel col0 of the tile
    auto store_block = [&](const PosInfo<DIM> &pi, int y, auto &v, int col0) {
        constexpr int N = sizeof(v) / sizeof(float);
        if (!pi.valid) return;
        const int grp = y / tiles_n, dl0 = y % tiles_n * BN + col0;      // first dense channel within the group
        const int d0 = grp * g.cdg_r + dl0, n = min(N, g.cdg_r - dl0);
        using TO = typename std::conditional<M::F32, float, T16>::type;
        TO *out = static_cast<TO *>(P.out) + ((int64_t)pi.b * g.Cd_r + d0) * (int64_t)g.P + pi.p;
        if constexpr (MODE == TC_F16_WIDE) {
            const float factor = out_scale;
#pragma unroll
            for (int e = 0; e < N; ++e) v[e] *= factor;
        }
        if (n == N) {
#pragma unroll
            for (int e = 0; e < N; ++e) {
                store_acc(out, 0, P.bias != nullptr ? v[e] + __ldg(P.bias + d0 + e) : v[e]);
                out += g.P;
            }
        } else {                                      // the group ends inside this block of columns
#pragma unroll
            for (int e = 0; e < N; ++e)
                if (e < n) store_acc(out, (int64_t)e * g.P, P.bias != nullptr ? v[e] + __ldg(P.bias + d0 + e) : v[e]);
        }
    };
    // The pieces of a shared tile added in the order of the CTAs: columns 4 q .. 4 q + 3 of position `row` for
    // q = q0, q0 + step, ..., QN of them at a time.
    auto sum_pieces = [&](int tile, int row, int q0, int step, auto qn) {
        constexpr int QN = decltype(qn)::value;
        const int first = tile * n_chunks;
        const int c0 = W.owner(first), c1 = W.owner(first + n_chunks - 1);
        const PosInfo<DIM> pi = decode_position<DIM>(g, (long long)(tile / W.tiles_y) * TILE_POS + row);
        const size_t piece_size = (size_t)(BN / 4) * TILE_POS;
        // the first CTA's piece is in its second slot where it came to the tile from an earlier one
        const float4 *base = reinterpret_cast<const float4 *>(P.partial) + row;
        const size_t slot0 = (size_t)c0 * 2 + (W.bound(c0) < first ? 1 : 0);
        for (int q = q0; q < BN / 4; q += step * QN) {
            float4 sum[QN];
#pragma unroll
            for (int k = 0; k < QN; ++k) sum[k] = __ldcg(base + slot0 * piece_size + (size_t)(q + k * step) * TILE_POS);
#pragma unroll 2
            for (int c = c0 + 1; c <= c1; ++c) {
#pragma unroll
                for (int k = 0; k < QN; ++k) {
                    const float4 v = __ldcg(base + (size_t)c * 2 * piece_size + (size_t)(q + k * step) * TILE_POS);
                    sum[k].x += v.x;
                    sum[k].y += v.y;
                    sum[k].z += v.z;
                    sum[k].w += v.w;
                }
            }
#pragma unroll
            for (int k = 0; k < QN; ++k) {
                float f[4] = {sum[k].x, sum[k].y, sum[k].z, sum[k].w};
                store_block(pi, tile % W.tiles_y, f, (q + k * step) * 4);
            }
        }
    };
    // A tile's (or piece's) sums, `len` chunks of it, leave tensor memory: to the output, or to the workspace where the tile
    // is shared -- whoever brings the last piece there adds them all.  4 * parts warps, this one being of quad `part`; a warp
    // whose wait ran out (!ok) passes the barriers with the others, which have no time limit, and does nothing else.
    auto finish_piece = [&](bool ok, int tile, int len, bool first_unit, int buf, int part, auto parts_c, bool last_piece, auto barrier) {
        constexpr int parts = decltype(parts_c)::value;
        uint32_t *last_flag = last_flags + (last_piece ? 1 : 0);
        const int row = (warp & 3) * 32 + lane;               // position in the tile = TMEM lane
        const int y = tile % W.tiles_y;
        const uint32_t t_lane = tmem_base + (uint32_t)buf * set_cols + ((uint32_t)((warp & 3) * 32) << 16);
        const PosInfo<DIM> pi = decode_position<DIM>(g, (long long)(tile / W.tiles_y) * TILE_POS + row);
        const bool shared_tile = len < n_chunks;
        // this CTA's piece: in its first slot where it begins with the CTA's first unit, else in its second
        float4 *mine = shared_tile ? reinterpret_cast<float4 *>(P.partial) + ((size_t)blockIdx.x * 2 + (first_unit ? 0 : 1)) * (BN / 4) * TILE_POS
                                   : nullptr;
        for (int cb = ok ? part : BN / CW; cb < BN / CW; cb += parts) {
            float v[CW];
            uint32_t raw[CW];
            ptx::tmem_ld_32x16(t_lane + (uint32_t)(cb * CW), raw);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < CW; ++e) v[e] = __uint_as_float(raw[e]);
            for (int a = 1; a < acc_sets; ++a) {
                if (a < NACC && a >= len) continue;           // never written
                ptx::tmem_ld_32x16(t_lane + (uint32_t)(a * BN + cb * CW), raw);
                ptx::tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < CW; ++e) v[e] += __uint_as_float(raw[e]);
            }
            if (shared_tile) {
#pragma unroll
                for (int e = 0; e < CW / 4; ++e)
                    mine[(cb * (CW / 4) + e) * TILE_POS + row] = make_float4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]);
            } else {
                store_block(pi, y, v, cb * CW);
            }
        }
        if (!last_piece) {
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&acc_empty[buf]);
        }
        if (shared_tile) {
            const int first = tile * n_chunks;
            const int others = W.owner(first + n_chunks - 1) - W.owner(first);
            barrier();
            if (part == 0 && row == 0) {
                __threadfence();
                *last_flag = atomicAdd(&P.arrived[tile], 1u) == (unsigned)others ? 1u : 0u;
                __threadfence();
            }
            barrier();
            if (ok && *last_flag != 0) sum_pieces(tile, row, part, parts, std::integral_constant<int, 4>());
            barrier();
        }
    };
    // The pieces of this CTA, in order; the last one is the producers' (they are through by then, and four times as many as
    // the epilogue warps), the others are handled under the main loop of the next.
    const int first_tile = unit0 / n_chunks, last_tile = (unit0 + n_local - 1) / n_chunks;

    if (warp < PRODUCER_WARPS) {
        // ------------------------------------------------------------------ producers
        ptx::reg_inc<FWD_REGS_PRODUCER>();
        bool ok = true;
        // Two groups of producer warps take alternate chunks, so that one group's loads are in flight while the
        // other blends and stores: the load/store pipe stays busy instead of idling between phases.
        const int pgroup = warp / GROUP_WARPS;
        const int tg = (int)threadIdx.x % GROUP_THREADS;
        ChunkIter it;
        it.start(W, unit0 + pgroup, g.K);
        for (int i = pgroup; i < n_local; i += PGROUPS) {
            const int s = i % S, r = i / S;
            const int pbuf = i % PLAN_BUFS;
            if (ok && !ptx::mbar_wait(&plan_full[pbuf], (uint32_t)((i / PLAN_BUFS) & 1))) {
                ptx::report(P.status, 105);
                ok = false;
            }
            if (ok && !ptx::mbar_wait(&empty[s], (uint32_t)((r & 1) ^ 1))) {
                ptx::report(P.status, 101);
                ok = false;
            }
            ok = __all_sync(0xffffffffu, ok);  // keep the warp converged for the __syncwarp below
            if (!ok) break;
            uint8_t *a_tiles = sA + (size_t)s * a_stage_bytes;
            const uint32_t c16 = (uint32_t)(div_often_one(it.y, tiles_n) * g.csg + it.cc * CHUNK_C) * ESZ / 16u;
            produce_tiles<NC, MODE, GROUP_THREADS, (NC >= 8 ? 2 : 4)>(a_tiles, A_TILE_BYTES, 0u, TILE_POS, TILE_POS, img16, &c16,
                                                                      plan + pbuf * TILE_POS * 2 * NC, tg);
            ptx::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                ptx::mbar_arrive(&full_a[s]);
                ptx::mbar_arrive(&plan_empty[pbuf]);
            }
#pragma unroll
            for (int k = 0; k < PGROUPS; ++k) it.next(g.K, chunks, W.tiles_y);
        }
        const int before = last_tile - first_tile, buf = before % acc_bufs;
        // (a barrier of its own: tiles of one chunk are made faster than summed, and two pieces before acc_full looks alike)
        ok = ok && ptx::mbar_wait(acc_last, 0);
        ok = __all_sync(0xffffffffu, ok);  // tcgen05.ld is a whole-warp instruction
        if (!ok && lane == 0) ptx::report(P.status, 108);
        ptx::tc_fence_after();
        const int len = before == 0 ? n_local : unit0 + n_local - last_tile * n_chunks;
        finish_piece(ok, last_tile, len, before == 0, buf, warp >> 2, std::integral_constant<int, PRODUCER_WARPS / 4>(), true,
                     [] { asm volatile("bar.sync 2, %0;" ::"n"(PRODUCERS) : "memory"); });
    } else if (warp >= EPI_WARP0 && warp < MMA_WARP) {
        // ------------------------------------------------------------------ epilogue: one thread per position
        ptx::reg_dec<FWD_REGS_EPILOGUE>();
        bool ok = true;
        int buf = 0;
        uint32_t phase = 0;
        for (int tile = first_tile; tile < last_tile; ++tile) {
            if (ok) {
                ok = ptx::mbar_wait(&acc_full[buf], phase);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok && lane == 0) ptx::report(P.status, 102);
            }
            ptx::tc_fence_after();
            finish_piece(ok, tile, tile == first_tile ? (tile + 1) * n_chunks - unit0 : n_chunks, tile == first_tile, buf, 0,
                         std::integral_constant<int, 1>(), false, [] { asm volatile("bar.sync 1, 128;" ::: "memory"); });
            if (++buf == acc_bufs) {
                buf = 0;
                phase ^= 1u;
            }
        }
    } else if (warp == MMA_WARP) {
        // ------------------------------------------------------------------ MMA issue
        ptx::reg_dec<FWD_REGS_ISSUE>();
        if (lane == 0) {
            const uint32_t idesc = ptx::instr_desc_f16(M::HALF ? 0 : 1, TILE_POS, BN, 0, 0);
            bool ok = true;
            // ring position, phase and accumulator are stepped, and the descriptors of a stage derived from those of
            // stage 0 by an addition: this single thread must not spend longer on bookkeeping than on issuing MMAs
            const uint64_t a_desc0 = ptx::smem_desc_sw128(ptx::smem_u32(sA), 16, 1024);
            const uint64_t b_desc0 = ptx::smem_desc_sw128(ptx::smem_u32(sB), 16, 1024);
            int s = 0, acc_i = 0, buf = 0, j = 0;             // j: chunk of the current piece
            uint32_t phase = 0, acc_phase = 1;
            int left = n_local > 0 ? min(n_chunks - unit0 % n_chunks, n_local) : 0;   // chunks of the piece to go
            uint32_t acc0 = tmem_base;
            for (int i = 0; i < n_local && ok; ++i) {
                if (j == 0 && !ptx::mbar_wait(&acc_empty[buf], acc_phase)) {
                    ptx::report(P.status, 107);
                    ok = false;
                    break;
                }
                const bool got_b = ptx::mbar_wait(&full_a[s], phase) && ptx::mbar_wait(&full_b[s], phase);
                if (!got_b) {
                    ptx::report(P.status, 103);
                    ok = false;
                    break;
                }
                ptx::tc_fence_after();
                const uint64_t a_hi = a_desc0 + (uint64_t)((uint32_t)s * (a_stage_bytes >> 4));
                const uint64_t b_hi = b_desc0 + (uint64_t)((uint32_t)s * (b_stage_bytes >> 4));
                const uint32_t d_tmem = acc0 + (uint32_t)(acc_i * BN);
                const uint32_t low_tmem = low_acc ? acc0 + low_col : d_tmem;
#pragma unroll
                for (int k4 = 0; k4 < 4; ++k4) {
                    ptx::mma_f16(d_tmem, a_hi + 2 * k4, b_hi + 2 * k4, idesc, (j >= NACC || k4 > 0) ? 1u : 0u);
                    uint32_t low_on = (!low_acc || j > 0 || k4 > 0) ? 1u : 0u;
                    // products of parts ca + cb < parts of the finer operand; larger sums are below its last bit
#pragma unroll
                    for (int ca = 0; ca < CPARTS; ++ca)
#pragma unroll
                        for (int cb = 0; cb < MPARTS; ++cb)
                            if (ca + cb > 0 && ca + cb < CPARTS) {
                                ptx::mma_f16(low_tmem, a_hi + (uint64_t)(ca * (A_TILE_BYTES >> 4) + 2 * k4),
                                             b_hi + (uint64_t)(cb * (b_part_bytes >> 4) + 2 * k4), idesc, low_on);
                                low_on = 1u;
                            }
                }
                ptx::mma_commit(&empty[s]);
                if (++s == S) {
                    s = 0;
                    phase ^= 1u;
                }
                if (++acc_i == NACC) acc_i = 0;
                ++j;
                if (--left == 0) {                            // the piece is complete
                    ptx::mma_commit(i + 1 < n_local ? &acc_full[buf] : acc_last);
                    j = 0;
                    acc_i = 0;
                    left = min(n_chunks, n_local - i - 1);
                    acc0 += set_cols;
                    if (++buf == acc_bufs) {
                        buf = 0;
                        acc_phase ^= 1u;
                        acc0 = tmem_base;
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp == TMA_WARP) {
        // ------------------------------------------------------------------ TMA: weight tiles
        ptx::reg_dec<FWD_REGS_ISSUE>();
        if (lane == 0) {
            int s = 0, last_s = -1;
            uint32_t e_phase = 1, last_phase = 0;
            ChunkIter it;
            it.start(W, unit0, g.K);
            for (int i = 0; i < n_local; ++i) {
                if (!ptx::mbar_wait(&empty[s], e_phase)) {
                    ptx::report(P.status, 104);
                    break;
                }
                uint8_t *b_dst = sB + (size_t)s * b_stage_bytes;
                ptx::mbar_arrive_expect_tx(&full_b[s], b_stage_bytes);
                const int c0 = it.cc * CHUNK_C, grp = div_often_one(it.y, tiles_n), n0 = (it.y - grp * tiles_n) * BN;
                ptx::tma_load_4d(b_dst, &tmap0, &full_b[s], c0, n0, it.tap, grp);
                if (MPARTS > 1) ptx::tma_load_4d(b_dst + b_part_bytes, &tmap1, &full_b[s], c0, n0, it.tap, grp);
                if (MPARTS > 2) ptx::tma_load_4d(b_dst + 2 * b_part_bytes, &tmap2, &full_b[s], c0, n0, it.tap, grp);
                it.next(g.K, chunks, W.tiles_y);
                last_s = s;
                last_phase = e_phase ^ 1u;
                if (++s == S) {
                    s = 0;
                    e_phase ^= 1u;
                }
            }
            // never leave with a copy still in flight into this CTA's shared memory
            if (last_s >= 0) ptx::mbar_wait(&full_b[last_s], last_phase);
        }
        __syncwarp();
    }

    if (warp > TMA_WARP) ptx::reg_dec<FWD_REGS_ISSUE>();   // the two idle warps of the last warpgroup

    if (warp >= PRODUCER_WARPS && warp < EPI_WARP0) {
        // ------------------------------------------------------------------ planners: one thread per position
        ptx::reg_dec<FWD_REGS_PLANNER>();
        // run ahead of the producers: coordinates -> plan slots
        const int t = threadIdx.x - PRODUCERS;
        const bool deformable = P.offset != nullptr;
        const uint32_t row_scale = (uint32_t)g.Cs * ESZ / 16u;
        // Offsets / mask of chunk i + 2 are requested while chunk i is planned: their latency stays off the critical path
        // (one planner thread has nothing else in flight).  Both chunks are stepped by counting: a planner thread runs
        // one dependent instruction chain, so every division in it costs the whole CTA; positions and groups change
        // with the tile or the channel chunk only.
        struct Cursor {
            ChunkIter it;
            int ogi, mgi;
        };
        auto groups_of = [&](Cursor &c) {
            const int chan0 = div_often_one(c.it.y, tiles_n) * g.csg + c.it.cc * CHUNK_C;
            c.ogi = g.og > 1 ? chan0 / g.cs_per_og : 0;
            c.mgi = g.mg > 1 ? chan0 / g.cs_per_mg : 0;
        };
        Cursor fetch_c;
        ChunkIter cur_c;
        fetch_c.it.start(W, unit0, g.K);
        cur_c = fetch_c.it;
        groups_of(fetch_c);
        PosInfo<DIM> pi = decode_position<DIM>(g, (long long)cur_c.x * TILE_POS + t);
        // the fetched position's offset / mask addresses differ per chunk by a multiple of P only
        const float *off_base, *mask_base;
        auto bases_of = [&](const PosInfo<DIM> &p) {
            off_base = (P.offset != nullptr && p.valid) ? P.offset + (int64_t)p.b * g.og * g.K * DIM * (int64_t)g.P + p.p : nullptr;
            mask_base = (P.mask != nullptr && p.valid) ? P.mask + (int64_t)p.b * g.mg * g.K * (int64_t)g.P + p.p : nullptr;
        };
        bases_of(pi);
        auto fetch = [&](RawCoords<DIM> &rc) {
#pragma unroll
            for (int a = 0; a < DIM; ++a)
                rc.off[a] = off_base != nullptr
                                ? __ldg(off_base + (int64_t)((fetch_c.ogi * g.K + fetch_c.it.tap) * DIM + a) * g.P) : 0.f;
            rc.m = mask_base != nullptr ? __ldg(mask_base + (int64_t)(fetch_c.mgi * g.K + fetch_c.it.tap) * g.P) : 1.f;
            const int x = fetch_c.it.x;
            fetch_c.it.next(g.K, chunks, W.tiles_y);
            if (fetch_c.it.tap == 0) groups_of(fetch_c);
            if (fetch_c.it.x != x) bases_of(decode_position<DIM>(g, (long long)fetch_c.it.x * TILE_POS + t));
        };
        // Plans chunk i from `cur` and requests the coordinates of chunk i + 2 into `fill`.  The three coordinate
        // sets rotate by name (the loop below is unrolled by three), never by assignment: copying a set whose loads
        // are still in flight would wait for them and put their latency back on the critical path.
        float col_scale = 1.f;
        auto step = [&](int i, const RawCoords<DIM> &cur, RawCoords<DIM> &fill) -> bool {
            const int pbuf = i % PLAN_BUFS;
            if (i + 2 < n_local) fetch(fill);
            bool ok = ptx::mbar_wait(&plan_empty[pbuf], (uint32_t)(((i / PLAN_BUFS) & 1) ^ 1));
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) {
                if (lane == 0) ptx::report(P.status, 106);
                return false;
            }
            uint32_t *slot = plan + (pbuf * TILE_POS + t) * 2 * NC;
            int tc[DIM];
#pragma unroll
            for (int a = 0; a < DIM; ++a) tc[a] = tap_tab[cur_c.tap * DIM + a];
            build_plan_at<DIM, MODE>(g, pi, cur, deformable, tc, row_scale, slot, col_scale);
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&plan_full[pbuf]);
            const int x = cur_c.x;
            cur_c.next(g.K, chunks, W.tiles_y);
            if (cur_c.x != x) pi = decode_position<DIM>(g, (long long)cur_c.x * TILE_POS + t);
            return true;
        };
        RawCoords<DIM> r0, r1, r2;
        if (n_local > 0) fetch(r0);
        if (n_local > 1) fetch(r1);
        if constexpr (MODE == TC_F16_WIDE) {
            __shared__ uint32_t scale_part[8];
            col_scale = column_scale<3>(P.range, t, scale_part);
            if (t == 0) out_scale = inverse_of_power_of_two(col_scale);
        }
        int i = 0;
        bool ok = true;
        for (; ok && i + 2 < n_local; i += 3) ok = step(i, r0, r2) && step(i + 1, r1, r0) && step(i + 2, r2, r1);
        if (ok && i < n_local) ok = step(i, r0, r2);
        if (ok && i + 1 < n_local) ok = step(i + 1, r1, r0);
    }

    ptx::tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) ptx::tmem_dealloc(tmem_base, ncols);
}

}  // namespace

bool make_tensor_map_16bit(CUtensorMap *map, const void *base, int rank, const uint64_t *dims,
                           const uint64_t *strides_bytes, const uint32_t *box) {
    typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static EncodeFn encode = nullptr;
    if (encode == nullptr) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess ||
            qres != cudaDriverEntryPointSuccess || fn == nullptr)
            return false;
        encode = (EncodeFn)fn;
    }
    cuuint32_t ones[5] = {1, 1, 1, 1, 1};
    const CUresult rc = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void *>(base),
                               (const cuuint64_t *)dims, (const cuuint64_t *)strides_bytes, (const cuuint32_t *)box,
                               ones, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return rc == CUDA_SUCCESS;
}

// ---- launcher -----------------------------------------------------------------------------------------
size_t fwd_tc_smem_bytes(int dim, int mode, int bn, int stages) {
    const size_t stage = (size_t)A_TILE_BYTES * mode_col_parts(mode) + (size_t)bn * 128 * mode_mat_parts(mode);
    const size_t plan = (size_t)PLAN_BUFS * (1 << dim) * TILE_POS * 8;
    return 1024 + stages * stage + plan + (3 * stages + 5 + 2 * PLAN_BUFS) * 8 + 16;
}

// statically allocated shared memory of the kernel (tap table), which counts against the same 227 KB
static size_t fwd_static_smem(int dim) { return (size_t)FWD_MAX_TAPS * dim * sizeof(int16_t) + 128; }

static bool fwd_work(const GeoHost &h, int mode, int bn, bool may_share, FwdWork *w) {
    const long long tiles_x = ((long long)h.B * h.P + TILE_POS - 1) / TILE_POS, tiles_y = h.groups * ((h.Cd / h.groups) / bn);
    w->n_chunks = h.K * (h.Cs / h.groups / CHUNK_C);
    const long long units = tiles_x * tiles_y * w->n_chunks;
    if (units > 0x7fffffffLL) return false;
    w->n_tiles = (int)(tiles_x * tiles_y);
    w->tiles_y = (int)tiles_y;
    // Sharing tiles evens out the last wave, or spreads few tiles over the chip: each SM then takes units / SMs chunks
    // instead of whole tiles.  What it costs, in chunks: a piece of 128 x bn sums goes to the workspace, and whoever comes last
    // reads all of a tile's.  Two CTAs per tile (`halves`) end with their only piece, which their 16 producer warps take out
    // together; in equal ranges of units most CTAs also begin with the rest of a tile, which falls to the four epilogue
    // warps.  (Halves cut by equal ranges drift against the tiles where their chunks are odd: 37 tiles of 27 chunks of 256
    // bf16 channels took 56 us, cut exactly 38, whole 39.)  A chunk of f32 data takes twice the time, so it counts half.
    // Fitted to 1700 calls of 1 to 600 tiles of 4 to 72 chunks, each timed both ways: these lines lose 0.1 % against the better
    // side on average and 10 % at worst (8 chunks for all, 16 with 256 channels: 1.0 % and 28 %).  Microseconds, whole /
    // shared, 37 tiles of 36 chunks of 64, 128, 256 channels: bf16 43 / 33, 45 / 37, 46 / 41; f32 67 / 45, 73 / 51, 80 / 59; 150
    // tiles of 36 chunks: bf16 74 / 54, 77 / 58, 78 / 67; f32 124 / 80, 129 / 91, 157 / 117.
    constexpr int HALVES[2][3] = {{6, 6, 11}, {3, 3, 5}}, RANGES[2][3] = {{7, 12, 22}, {4, 5, 11}};   // [f32][64, 128, 256 channels]
    const long long sms = 148;
    const long long shared = std::min(sms, std::min(units / 3, 2LL * w->n_tiles));
    const bool two_each = shared == 2LL * w->n_tiles;
    int cost = (two_each ? HALVES : RANGES)[mode_f32(mode)][bn / 128];
    // Beyond five tiles per SM the last wave is a small part, and CTAs that are out of step with one another lose something in
    // every tile: 1050 tiles of 27 chunks, whole / shared: bf16 219 / 211 (64 channels), 227 / 223, 237 / 239 (256); f32 377 / 364, 475 / 509,
    // 625 / 641; of 9 chunks (a gain of 8): bf16 84 / 91, 93 / 100, 120 / 127, f32 140 / 137, 160 / 160, 201 / 205.
    if (w->n_tiles > 5 * sms) cost = bn == 256 || (mode_f32(mode) && bn == 128) ? 1 << 20 : std::max(cost, 10);
    const long long whole_time = (w->n_tiles + sms - 1) / sms * w->n_chunks;
    w->whole = !may_share || w->n_chunks < 3 || shared < 2 || whole_time <= (units + shared - 1) / std::max(shared, 1LL) + cost;
    w->halves = !w->whole && two_each && w->n_chunks % 2 != 0;       // (an even number is halved by equal ranges)
    w->ctas = (int)(w->whole ? std::max(1LL, std::min<long long>(sms, w->n_tiles)) : shared);   // 1: an empty batch, planned but not launched
    const long long items = w->whole ? w->n_tiles : units;
    w->base = (int)(items / w->ctas);
    w->extra = (int)(items % w->ctas);
    return true;
}

// Picks the dense-channel tile and the pipeline depth; returns false when the shape is not covered
// or has 2^31 units of work or more.
bool fwd_tc_config(const GeoHost &h, int mode, int *bn, int *stages) {
    const int cdg = h.Cd / h.groups;
    // widest tile of dense channels first (the sampled tile is produced once per CTA, so a wider tile divides the
    // sampling work), then the deepest pipeline that fits
    int n = 0, s = 0;
    for (int cand_n : {256, 128, 64}) {
        if (cdg % cand_n != 0) continue;
        for (int cand : {3, 2})
            if (fwd_tc_smem_bytes(h.dim, mode, cand_n, cand) + fwd_static_smem(h.dim) <= 227 * 1024) { s = cand; break; }
        if (s != 0) { n = cand_n; break; }
    }
    FwdWork work;
    if (n == 0 || !fwd_work(h, mode, n, false, &work)) return false;
    *bn = n;
    *stages = s;
    return true;
}

template <int DIM, int MODE>
cudaError_t launch_fwd_tc_t(const GeoHost &h, const FwdParams<DIM> &P, const CUtensorMap *maps, cudaStream_t stream) {
    const size_t smem = fwd_tc_smem_bytes(DIM, MODE, P.bn, P.stages);
    LaunchScope scope("dcn_fwd_tc", stream);
    return launch_dependent<dcn_fwd_tc_kernel<DIM, MODE>>(dim3((unsigned)P.work.ctas), FWD_THREADS, smem, stream, P, maps[0],
                                                          maps[1], maps[2]);
}

// Bytes of the partial sums and number of arrival counters that a launch needs in its workspace (0: no tile is shared).
void fwd_tc_workspace(const GeoHost &h, int mode, int bn, size_t *partial_bytes, size_t *counters) {
    FwdWork w;
    *partial_bytes = *counters = 0;
    if (!fwd_work(h, mode, bn, true, &w) || w.whole) return;
    *partial_bytes = (size_t)w.ctas * 2 * bn * TILE_POS * sizeof(float);
    *counters = (size_t)w.n_tiles;
}

// img_cl: channels-last sampled image in the problem's data type; w_parts: weights packed [g][tap][d'][s'], one
// 16-bit tensor per part of the mode; h: padded geometry; partial / arrived: see fwd_tc_workspace, arrived zeroed (partial null: every tile has one CTA).
cudaError_t launch_sample_gemm_tc(const GeoHost &h, int mode, const void *img_cl, void *const *w_parts,
                                  const float *offset, const float *mask, const float *bias, const ColumnRange &range,
                                  void *out, float *partial, unsigned *arrived, const Status &status, cudaStream_t stream) {
    const int cdg = h.Cd / h.groups, csg = h.Cs / h.groups;
    int bn = 0, stages = 0;
    if (!fwd_tc_config(h, mode, &bn, &stages)) return cudaErrorInvalidConfiguration;
    FwdWork work;
    if (!fwd_work(h, mode, bn, partial != nullptr, &work)) return cudaErrorInvalidConfiguration;
    CUtensorMap maps[3];
    const uint64_t dims[4] = {(uint64_t)csg, (uint64_t)cdg, (uint64_t)h.K, (uint64_t)h.groups};
    const uint64_t strides[3] = {(uint64_t)csg * 2, (uint64_t)csg * cdg * 2, (uint64_t)csg * cdg * h.K * 2};
    const uint32_t box[4] = {CHUNK_C, (uint32_t)bn, 1, 1};
    if (!make_part_maps(maps, w_parts, mode_mat_parts(mode), 4, dims, strides, box)) return cudaErrorInvalidValue;
    auto run = [&](auto dimc) -> cudaError_t {
        constexpr int DIM = decltype(dimc)::value;
        FwdParams<DIM> P;
        P.g = geo_from_host<DIM>(h);
        P.img_cl = img_cl;
        P.offset = offset;
        P.mask = mask;
        P.bias = bias;
        P.range = range;
        P.out = out;
        P.status = status;
        P.bn = bn;
        P.stages = stages;
        P.partial = partial;
        P.arrived = arrived;
        P.work = work;
        return with_mode(mode, [&](auto m) { return launch_fwd_tc_t<DIM, decltype(m)::value>(h, P, maps, stream); });
    };
    if (h.dim == 1) return run(std::integral_constant<int, 1>());
    if (h.dim == 2) return run(std::integral_constant<int, 2>());
    if (h.dim == 3) return run(std::integral_constant<int, 3>());
    return cudaErrorInvalidValue;
}

}  // namespace tvdcn_b200
