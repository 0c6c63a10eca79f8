// Tensor-core "GEMM -> scatter" kernel (tcgen05 / TMEM) with pixel-owned aggregation.
//
//   col[k | b, p] = sum_{d in group} W[d, k] * dense[b, d, p],   k = (tap, sampled channel)
// consumed straight out of tensor memory, never stored in global memory:
//   img_grad[b, s, corner]   += col * mask * corner weight                      (scatter)
//   grad_offset[b, og, tap, axis, p] += col * mask * d sample / d axis          (needs the sampled image)
//   grad_mask[b, mg, tap, p]         += col * sample                            (needs the sampled image)
//
// Replaces addmm_ + compute_grad_offset + compute_grad_mask + col2im of the reference's backward loop
// (tvdcn/csrc/ops/cuda/deform_conv2d_kernel.cpp:519-598) and addmm_ + col2im of the transposed forward
// (tvdcn/csrc/ops/cuda/deform_conv_transpose2d_kernel.cpp:333-362): the column buffer is never written.
//
// Work is cut into *units*: (tile of 128 grid positions, 64-channel chunk, batch of TB taps), ordered tile by tile.  The
// grid has one CTA per SM (see launch_dgrad_t) and each takes an equal, contiguous range of units: nothing but a CTA's first unit waits
// for its operands (start-up was 12 k of 36 k cycles per tile for short 1-d reductions), and the SMs finish together
// whatever the number of tiles.
//   GEMM   D[128 positions (TMEM lanes) x TB*32 columns] over the dense channels of the group, two of them (slabs of 32
//          channels) per unit.
//          A = the dense tile [128 pos][cdg], read once per tile from the caller's [B, Cd, P] tensor (thread =
//              position, coalesced), converted to 16-bit (f32 data: bf16 parts) and kept in TENSOR MEMORY
//              (tcgen05.st; the MMA reads A from TMEM, so shared memory carries only B); later tiles are loaded by the
//              finishing warps as soon as the old tile's last MMA is through;
//          B = weights packed [g][tap][s'][d'], one TMA box {64 d', 32 s', TB taps} per reduction chunk (ring);
//          D = a ring of up to four accumulators in the TMEM columns behind A.
//   plan   Four planner warps (thread = position) turn the unit's offsets / mask into one entry per PAIR of bilinear corners
//          that are neighbours along the image's last axis (rows of the even and of the odd one, their weights x mask) and GROUP
//          THE ENTRIES BY PIXEL: a counting sort by the left pixel modulo SC_SLOTS (shared-memory integer atomics + prefix sum).
//   gather Twelve warps copy the unit's columns TMEM -> shared memory ([128 pos][TB*64] f32); then 8 lanes per entry (8 channels
//          each) walk equal spans of the pixel-grouped entry list.  An entry's column values are read once for both of its pixels:
//          they go into the running sums of the even and of the odd pixel (which leave the SM as red.global.add.v4.f32 when the
//          pixel changes, instead of once per corner), and into the dot products <col, image row of the pixel> that the
//          coordinate gradients need.  The image rows stay in registers while the pixel does.
//   finish Four warps turn the dots of a unit into grad_offset / grad_mask, and load dense tiles.
//
// What bounds it: the gather loop, by issue slots, instruction fetch and the latency of its shared-memory reads in about equal parts
// (45-50 % of issue slots, 50 % of the load/store data pipe; its twelve warps are few because each needs 100 registers).  Hence the
// form of the loop: two entries per iteration and no more (a loop of four, 6 KB of code beside the planners' and finishers' straight
// lines, took 574 instead of 551 us at 128 x 256 x 28 x 28 bf16, 4 groups of offsets), columns and entries read ahead, one
// branch per flush.  Before, one entry per corner, 4 channels per lane and the columns staged in two halves: 799 us there, 850 f32,
// 64 x 512 x 4096 1-d f32 1907, 8 x 64 x 16 x 56 x 56 3-d f32 4147; now 531, 670, 1165, 2589.  (16 gather warps have
// no registers to read columns ahead: 586 us, and 768 with the spills of trying.)
//
// Warp roles (768 threads): 0-3 finish, 4-15 gather, 16-19 planners, 20 MMA issue + TMEM owner, 21 TMA, 22-23 idle
// (they complete the last warpgroup for the register hand-over).
#include <algorithm>
#include <type_traits>

#include "plan.h"
#include "sm100_common.cuh"

namespace tvdcn_b200 {

template <int DIM>
struct DgradParams {
    Geo<DIM> g;
    const void *dense;      // [B, Cd, P] in the problem's data type, the caller's layout
    const void *img_cl;     // sampled image, channels-last (16-bit or f32); null when no coordinate gradient is wanted
    const float *offset;    // may be null
    const float *mask;      // may be null
    float *img_grad_cl;     // [B*S, Cs] f32, accumulated into; may be null
    float *goff;            // f32, accumulated into; may be null
    float *gmask;           // f32, accumulated into; may be null
    Status status;
    int rc;                 // reduction chunks: cdg / 64
    int tb;                 // taps per batch
    int nbatch;             // ceil(K / tb)
    int nacc;               // accumulators in the TMEM ring
    int b_stages;
    int tiles_x;            // position tiles
    int n_units;            // units per (position tile, group): (csg / 64) * nbatch
    int total_units;
    int block[DIM];         // volumes: the grid is taken in blocks of this extent (the last of a row, strip or slab may be smaller)
};

namespace {

constexpr int SC_FINISH_WARPS = 4;
constexpr int SC_GATHER_WARPS = 12;
constexpr int SC_WORK_WARPS = SC_FINISH_WARPS + SC_GATHER_WARPS;
constexpr int SC_LOAD_WARPS = 16;                                 // these load the first dense tile
constexpr int SC_PLAN_WARP0 = SC_WORK_WARPS;
constexpr int SC_PLAN_WARPS = 4;                                  // one planner thread per tile position
constexpr int SC_MMA_WARP = SC_PLAN_WARP0 + SC_PLAN_WARPS;
constexpr int SC_TMA_WARP = SC_MMA_WARP + 1;
constexpr int SC_THREADS = (SC_TMA_WARP + 3) * 32;                // two idle warps complete the last warpgroup
static_assert(SC_THREADS == 768, "six warpgroups");
// Registers per thread after the warpgroups have rebalanced them (launch: 80 each for 6 warpgroups = 480 x 128):
// 3 x 104 (gather) + 72 (planners) + 64 (finish) + 32 (MMA / TMA) = 480.
constexpr int SC_REGS_LAUNCH = 65536 / SC_THREADS / 8 * 8;
constexpr int SC_REGS_GATHER = 104, SC_REGS_PLAN = 72, SC_REGS_FINISH = 64, SC_REGS_ISSUE = 32;
static_assert(SC_GATHER_WARPS * SC_REGS_GATHER + SC_PLAN_WARPS * SC_REGS_PLAN + SC_FINISH_WARPS * SC_REGS_FINISH + 4 * SC_REGS_ISSUE <=
                  SC_THREADS / 32 * SC_REGS_LAUNCH, "an increase beyond the launch's registers waits for ever");
template <int N>
__device__ __forceinline__ void take_registers() {
    if constexpr (N >= SC_REGS_LAUNCH) ptx::reg_inc<N>();
    else ptx::reg_dec<N>();
}
constexpr int SC_GROUPS = SC_GATHER_WARPS * 4;                    // 8-lane groups walking the entry list
constexpr int SC_SLAB = 32;                                       // channels per pass
constexpr int SC_PLAN_SLACK = SC_GROUPS * 2 + 8;                  // padding of the spans to a multiple of two; read-ahead
// Slots of the counting sort.  A tile's entries lie around its positions, so rows that share a slot are rare; where
// they do, their entries interleave and the pixel's running sum leaves the SM more often, nothing else.
constexpr int SC_SLOTS = 2048, SC_SLOT_WORDS = SC_SLOTS + SC_SLOTS / 32 * 4;
constexpr int SC_TMEM_COLS = 512;
constexpr int SC_SLEEP_NS = 32;                                   // back-off of the long waits (64 to 512 measured equal)
constexpr int SC_MAX_TAPS = 512;                                  // taps whose kernel coordinates a CTA tabulates

// most taps per batch: shared memory holds the columns of one batch and the entry lists of two (volumes: three taps leave
// room for two stages of weights, and still gain over two taps with four: 8 x 64 x 16 x 56 x 56 f32 2822 -> 2644 us)
__host__ __device__ constexpr int sc_tb_max(int dim) { return dim == 1 ? 4 : 3; }

__device__ __forceinline__ uint64_t pack_f32x2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

template <int SIZE>
__device__ __forceinline__ uint64_t row_at(uint64_t base, uint32_t px) {
    uint64_t r;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(px), "n"(SIZE), "l"(base));
    return r;
}

// Where px != cur: adds the sums `v` (4 + 4 channels, 32 apart) to the row at `addr` and starts them anew.  One branch for all of
// it: the compiler wraps every predicated reduction in a branch of its own.  No "memory" clobber: nothing in this kernel reads
// what the reductions write, and the shared-memory loads around them must stay free to move.
__device__ __forceinline__ void flush_sums(uint32_t px, uint32_t cur, uint64_t addr, float (&v)[8]) {
    if (px != cur) {
        asm volatile(
            "red.global.add.v4.f32 [%8], {%0, %1, %2, %3};\n\t"
            "red.global.add.v4.f32 [%8 + 128], {%4, %5, %6, %7};\n\t"
            ::"f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "l"(addr));
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = 0.f;
    }
}
// Weight of what adds nothing to its pixel: one outside of the image, or an entry that pads the list.  The former's pixel offset is that
// of the place next to its real neighbour in memory, an ordinary pixel, so that running sums go on under it.  (With rows of waste
// behind the image every such entry cost a flush, and in calls without offsets each entry lacks a pixel: backward kernel 64 x 64 x 56 x
// 56 f32 525 us, now 207; 2 x 64 x 16 x 56 x 56 818, now 355; with offsets 128 x 256 x 28 x 28 f32 662, now 670, bf16 527, now 531.)  No product of two floats has
// these bits (a NaN result is 0x7fffffff).  A weight of zero would not do: zero times an infinite column is NaN.
constexpr uint32_t SC_NO_WEIGHT = 0xffffffffu;
// sum += weight x column
__device__ __forceinline__ void add_weighted(float (&sum)[8], uint32_t weight, const uint64_t (&c)[4]) {
    const uint64_t ww = pack_f32x2(__uint_as_float(weight), __uint_as_float(weight));
#pragma unroll
    for (int k = 0; k < 4; ++k) unpack_f32x2(fma_f32x2(ww, c[k], pack_f32x2(sum[2 * k], sum[2 * k + 1])), sum[2 * k], sum[2 * k + 1]);
}
// Where px != was: loads 4 + 4 channels, 32 apart, of 16-bit (4 words) or f32 (8 words) data.
template <int IW>
__device__ __forceinline__ void load_row(uint32_t px, uint32_t was, uint32_t (&v)[IW], uint64_t addr) {
    if constexpr (IW == 4)
        asm volatile(
            "{\n\t"
            ".reg .pred q;\n\t"
            "setp.ne.u32 q, %5, %6;\n\t"
            "@q ld.global.nc.v2.u32 {%0, %1}, [%4];\n\t"
            "@q ld.global.nc.v2.u32 {%2, %3}, [%4 + 64];\n\t"
            "}\n" : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]) : "l"(addr), "r"(px), "r"(was));
    else
        asm volatile(
            "{\n\t"
            ".reg .pred q;\n\t"
            "setp.ne.u32 q, %9, %10;\n\t"
            "@q ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%8];\n\t"
            "@q ld.global.nc.v4.u32 {%4, %5, %6, %7}, [%8 + 128];\n\t"
            "}\n" : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7])
            : "l"(addr), "r"(px), "r"(was));
}

__device__ __forceinline__ void planner_barrier() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// Sampling geometry of one (position, tap): floor and fraction per axis, mask value.
template <int DIM>
struct TapGeometry {
    int fl[DIM];
    float fr[DIM];
    float mval;
};

// Position number idx of the launch: images one after the other; volumes in blocks of 4 x 4 x 8, each row by row.  A tile of whole
// rows of a volume has many pixels around it, and the more there are, the fewer entries share one: blocks take 8 x 64 x 16 x 56 x 56 f32
// (offsets of sigma 1) from 3150 to 2820 us, 4 x 64 x 16 x 40 x 40 from 787 to 744 (sigma 0.5) and 949 to 842 (3), 128 x 6 x 60 x 90 bf16
// from 533 to 398.  (8 x 16 in 2-d gains 10 % on images 160 wide and nothing on those below 100, and its arithmetic in the
// planners cost narrow ones up to 5 %.)
template <int DIM>
__device__ __forceinline__ PosInfo<DIM> decode_blocked(const DgradParams<DIM> &P, long long idx) {
    const Geo<DIM> &g = P.g;
    if constexpr (DIM < 3) {
        return decode_position<DIM>(g, idx);
    } else {
        PosInfo<DIM> pi;
        pi.valid = idx < g.BP;
        const int i = pi.valid ? (int)idx : 0;             // fewer than 2^31 positions
        pi.b = i / g.P;
        int r = i - pi.b * g.P;
        int first[DIM], ext[DIM], size = g.P;              // size: positions of what is being cut (image, slab, strip)
#pragma unroll
        for (int a = 0; a < DIM; ++a) {
            const int line = size / g.grid[a];            // positions per unit of length along this axis
            const int blk = r / (line * P.block[a]);
            first[a] = blk * P.block[a];
            ext[a] = min(P.block[a], g.grid[a] - first[a]);
            r -= line * first[a];
            size = line * ext[a];
        }
        int c[DIM];
#pragma unroll
        for (int a = DIM - 1; a > 0; --a) {
            const int q = r / ext[a];
            c[a] = first[a] + r - q * ext[a];
            r = q;
        }
        c[0] = first[0] + r;
        pi.p = 0;
#pragma unroll
        for (int a = 0; a < DIM; ++a) {
            pi.p = pi.p * g.grid[a] + c[a];
            pi.base[a] = c[a] * g.stride[a] - g.pad[a];
        }
        return pi;
    }
}

// Pair q of the 2^(DIM - 1) pairs of corners that are neighbours along the last axis: pixel row of the left one (of the
// place left of the image where only the right one lies in it), which of the two are in the image, their weights.  key: the
// left one's slot in the counting sort: its place where every row begins with one place more (which keeps pairs across an edge
// apart from others), modulo the slots; in volumes, whose planes would meet there, some bits of each coordinate, as many as a
// tile reaches.
template <int DIM>
__device__ __forceinline__ void pair_of(const Geo<DIM> &g, const PosInfo<DIM> &pi, const TapGeometry<DIM> &tg,
                                        bool deformable, int q, uint32_t &left, uint32_t &key, bool &ok_l, bool &ok_r, float &w_l,
                                        float &w_r) {
    bool ok = deformable || q == 0;
    int flat = 0;
    float w = 1.f;
    unsigned row_y = 0, row_z = 0;
#pragma unroll
    for (int a = 0; a < DIM - 1; ++a) {
        const int bit = (q >> (DIM - 2 - a)) & 1;
        const int i = (int)((unsigned)tg.fl[a] + (unsigned)bit);
        row_z = row_y;
        row_y = (unsigned)i;
        ok = ok && ((unsigned)i < (unsigned)g.img[a]);
        flat = flat * g.img[a] + i;
        w *= bit ? tg.fr[a] : (1.f - tg.fr[a]);
    }
    const unsigned i = (unsigned)tg.fl[DIM - 1];
    ok_l = ok && i < (unsigned)g.img[DIM - 1];
    ok_r = ok && deformable && i + 1u < (unsigned)g.img[DIM - 1];
    unsigned row = (unsigned)pi.b;
#pragma unroll
    for (int a = 0; a < DIM - 1; ++a) row *= (unsigned)g.img[a];
    row += (unsigned)flat;
    left = row * (unsigned)g.img[DIM - 1] + i;
    if constexpr (DIM < 3) key = left + row + 1u;
    else key = ((i + 1u) & 15u) | (row_y & 15u) << 4 | ((unsigned)pi.b * (unsigned)g.img[0] + row_z & 7u) << 8;
    key &= SC_SLOTS - 1;
    w_l = w * (1.f - tg.fr[DIM - 1]);
    w_r = w * tg.fr[DIM - 1];
}

// Byte offsets of the dynamic shared memory regions (after alignment to 1024).
struct ScLayout {
    uint32_t b_stage, plan_buf, col, plan, info, pos, cnt, taps, misc, bars, total;
    int n, col_stride, max_entries;
};
__host__ __device__ inline ScLayout sc_layout(int dim, int tb, int b_stages) {
    ScLayout L;
    L.n = tb * SC_SLAB;
    L.col_stride = 2 * L.n + 4;                   // words; = 4 mod 32, so that the row-per-lane stores spread over the banks
    L.max_entries = TILE_POS * tb << (dim - 1);
    L.b_stage = (uint32_t)(L.n * 128);             // one 16-bit part (hi or lo) of one reduction chunk
    // per entry {pixel offset even, odd, weight even, odd} and a word (col index | dot slot << 16), with room for the padding
    // of the groups' spans and the read-ahead of the last group; then two dot products per entry (+ two for the padding entries)
    L.plan_buf = (uint32_t)((L.max_entries + SC_PLAN_SLACK) * 20 + (2 * L.max_entries + 4) * 4);
    uint32_t o = 0;
    o += (uint32_t)b_stages * L.b_stage;
    L.col = o;  o += (uint32_t)(TILE_POS * L.col_stride * 4);
    L.plan = o; o += 2 * L.plan_buf;
    L.info = o; o += 4 * 16;                      // of four units: first channel, first tap, offset group, mask group
    L.pos = o;  o += 4 * TILE_POS * 8;            // and per position of the tile: image (or -1), position in it
    L.cnt = o;  o += SC_SLOT_WORDS * 4;
    L.taps = o; o += SC_MAX_TAPS * 4;             // kernel coordinates of every tap, ten bits per axis
    L.misc = o; o += 64;                          // scan partial sums [4], wait flag, entry counts [2], TMEM slot
    L.bars = o; o += (uint32_t)(18 + 2 * b_stages) * 8;
    L.total = o;
    return L;
}

// The units of a CTA in order.  1-d and 2-d: a CTA's tiles follow one another, so it finds its neighbourhood of the image
// in the caches.  3-d: that neighbourhood spans planes and 148 of them do not fit L2 (tiles one after the other: 8 x 64 x 16 x 56 x 56
// bf16 2573 instead of 2289 us, 2 x 64 x 16 x 56 x 56 f32 732 instead of 695), so the CTAs take neighbouring tiles at the same time: ranges
// run down the columns of a matrix of tiles with one column per CTA, filled row by row.  (One CTA per tile: the same order.)
struct UnitIter {
    int x, grp, chunk, batch;   // position tile, group, 64-channel chunk, tap batch
    int order;                  // the tile's place in that order
};
template <int DIM>
__device__ __forceinline__ void locate_tile(const DgradParams<DIM> &P, UnitIter &u) {
    int tile = u.order;
    if constexpr (DIM == 3) {
        const int tiles = P.tiles_x * P.g.groups, cols = (int)gridDim.x, rows = (tiles + cols - 1) / cols;
        const int full = tiles - cols * (rows - 1);    // columns that have all rows
        int c, r;
        if (u.order < full * rows) {
            c = u.order / rows;
            r = u.order - c * rows;
        } else {
            const int o = u.order - full * rows;
            c = o / (rows - 1);
            r = o - c * (rows - 1);
            c += full;
        }
        tile = r * cols + c;
    }
    u.grp = tile < P.tiles_x ? 0 : tile / P.tiles_x;
    u.x = tile - u.grp * P.tiles_x;
}
template <int DIM>
__device__ __forceinline__ UnitIter first_unit(const DgradParams<DIM> &P, int unit) {
    UnitIter u;
    u.order = unit / P.n_units;
    const int r = unit - u.order * P.n_units;
    u.chunk = r / P.nbatch;
    u.batch = r - u.chunk * P.nbatch;
    locate_tile(P, u);
    return u;
}
// Returns whether a new tile begins.  (Behind the last unit of the launch there is none: its position stays as it is.)
template <int DIM>
__device__ __forceinline__ bool next_unit(const DgradParams<DIM> &P, UnitIter &u) {
    if (++u.batch < P.nbatch) return false;
    u.batch = 0;
    if (++u.chunk < P.g.csg / CHUNK_C) return false;
    u.chunk = 0;
    if (++u.order < P.tiles_x * P.g.groups) locate_tile(P, u);
    return true;
}

// what is wanted: the scattered image, the coordinate gradients (grad_offset and / or grad_mask), both
enum { SC_SCATTER = 1, SC_COORD = 2 };

template <int DIM, int MODE, int WANT>
__global__ void __launch_bounds__(SC_THREADS, 1)
dcn_dgrad_tc_kernel(const DgradParams<DIM> P, const __grid_constant__ CUtensorMap tmap_b_hi,
                    const __grid_constant__ CUtensorMap tmap_b_lo, const __grid_constant__ CUtensorMap tmap_b_lo2) {
    constexpr bool SCATTER = (WANT & SC_SCATTER) != 0, COORD = (WANT & SC_COORD) != 0;
    constexpr int NC = 1 << DIM, NP = NC / 2;           // corners of a cell, pairs of them
    using M = Mode<MODE>;
    constexpr int PARTS = M::MAT_PARTS;                 // 16-bit parts of the dense tile and of the weights
    constexpr int ACCS = MODE == TC_F32_WIDE ? 2 : 1;   // accumulators of a pass: leading / small products
    constexpr int TBM = sc_tb_max(DIM);
    using T16 = typename M::T16;
    const Geo<DIM> &g = P.g;

    extern __shared__ uint8_t smem_raw[];
    // align by offset, not by integer round-trip, so that the compiler keeps these as shared-memory pointers
    uint8_t *smem = smem_raw + ((1024u - (ptx::smem_u32(smem_raw) & 1023u)) & 1023u);
    const int RC = P.rc, TB = P.tb, BS = P.b_stages, NACC = P.nacc;
    const ScLayout L = sc_layout(DIM, TB, BS);
    const int N = L.n;
    const int a_cols = g.cdg / 2;                       // TMEM columns of one 16-bit copy of the dense tile
    const uint32_t acc_col0 = (uint32_t)(a_cols * PARTS);
    uint8_t *sB = smem;
    float *col = reinterpret_cast<float *>(smem + L.col);
    uint32_t *cnt = reinterpret_cast<uint32_t *>(smem + L.cnt);
    uint32_t *misc = reinterpret_cast<uint32_t *>(smem + L.misc);
    uint32_t *scan_part = misc;          // [4]
    uint32_t *wait_flag = misc + 4;
    uint32_t *n_entries = misc + 6;      // [2]
    uint32_t *tmem_slot = misc + 8;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L.bars);
    uint64_t *a_first = bars;            // dense tile of the CTA's first unit is in TMEM / of every later tile
    uint64_t *a_next = bars + 1;
    uint64_t *b_full = bars + 2;
    uint64_t *b_empty = b_full + BS;
    uint64_t *t_full = b_empty + BS;     // [4] MMA -> gather warps: accumulator complete
    uint64_t *t_empty = t_full + 4;      // [4] gather warps -> MMA: accumulator read out
    uint64_t *col_full = t_empty + 4;    // gather warps: the unit's columns are in shared memory
    uint64_t *plan_full = col_full + 1;  // [2] planners -> gather warps
    uint64_t *plan_done = plan_full + 2; // [2] gather warps -> themselves, finishing warps, planners: through with the unit's columns and entries
    uint64_t *fin_done = plan_done + 2;  // [2] finishing warps -> gather warps: the dots of the unit have been used
    uint64_t *a_free = fin_done + 2;     // MMA -> finishing warps: the last MMA on the dense tile is through
    uint32_t *tap_tab = reinterpret_cast<uint32_t *>(smem + L.taps);
    const int plan_words = L.max_entries + SC_PLAN_SLACK;
    auto plan_ent = [&](int pb) { return reinterpret_cast<uint4 *>(smem + L.plan + (size_t)pb * L.plan_buf); };
    auto plan_meta = [&](int pb) { return reinterpret_cast<uint32_t *>(plan_ent(pb) + plan_words); };
    auto plan_dot = [&](int pb) { return reinterpret_cast<float *>(plan_meta(pb) + plan_words); };

    // of unit j: what its finalisation reads outlives its plan
    auto info_of = [&](int j) { return reinterpret_cast<int4 *>(smem + L.info) + (j & 3); };
    auto pos_of = [&](int j) { return reinterpret_cast<int2 *>(smem + L.pos) + (j & 3) * TILE_POS; };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // this CTA's units
    const int unit0 = (int)((long long)P.total_units * blockIdx.x / gridDim.x);
    const int n_units = (int)((long long)P.total_units * (blockIdx.x + 1) / gridDim.x) - unit0;
    const int n_pass = 2 * n_units;
    const bool deformable = P.offset != nullptr;
    if (threadIdx.x == 0) {
        ptx::mbar_init(a_first, SC_LOAD_WARPS);
        ptx::mbar_init(a_next, SC_FINISH_WARPS);
        ptx::mbar_init(a_free, 1);
        for (int s = 0; s < BS; ++s) {
            ptx::mbar_init(&b_full[s], 1);
            ptx::mbar_init(&b_empty[s], 1);
        }
        for (int q = 0; q < 4; ++q) {
            ptx::mbar_init(&t_full[q], 1);
            ptx::mbar_init(&t_empty[q], SC_GATHER_WARPS);
        }
        ptx::mbar_init(col_full, SC_GATHER_WARPS);
        for (int i = 0; i < 2; ++i) {
            ptx::mbar_init(&plan_full[i], SC_PLAN_WARPS);
            ptx::mbar_init(&plan_done[i], SC_GATHER_WARPS);
            ptx::mbar_init(&fin_done[i], SC_FINISH_WARPS);
        }
        ptx::fence_mbar_init();
    }
    for (int tp = threadIdx.x; tp < g.K; tp += SC_THREADS) {
        int tc[DIM];
        tap_coords<DIM>(g, tp, tc);
#pragma unroll
        for (int a = 1; a < DIM; ++a) tc[0] |= tc[a] << (10 * a);
        tap_tab[tp] = (uint32_t)tc[0];
    }
    if (warp == SC_TMA_WARP && lane == 0) {
        ptx::prefetch_tmap(&tmap_b_hi);
        if (PARTS > 1) ptx::prefetch_tmap(&tmap_b_lo);
        if (PARTS > 2) ptx::prefetch_tmap(&tmap_b_lo2);
    }
    if (warp == SC_MMA_WARP) {
        ptx::tmem_alloc(tmem_slot, SC_TMEM_COLS);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    ptx::grid_dependency_wait();     // nothing above reads what an earlier kernel wrote

    // ---- pieces shared by the planners (which build a unit's entry list) and the finishing warps (which turn its dot
    // products into coordinate gradients); both map thread -> position of the tile
    // {first channel, first tap, offset group, mask group} of a unit
    auto describe = [&](const UnitIter &u) {
        const int chan0 = u.grp * g.csg + u.chunk * CHUNK_C;
        return make_int4(chan0, u.batch * TB, g.og > 1 ? chan0 / g.cs_per_og : 0, g.mg > 1 ? chan0 / g.cs_per_mg : 0);
    };
    // offsets and mask of this position for the taps of one unit, as loaded (all loads in flight together)
    struct RawUnit {
        float off[TBM][DIM];
        float m[TBM];
    };
    // (This and the gradients below run once per unit beside the gather loop, which is short of issue slots and instruction cache: one
    // pointer and strides, no address from scratch, one body for all taps.  Half the code it was: 554 -> 543 us at 128 x 256 x 28 x 28.)
    auto load_unit = [&](const PosInfo<DIM> &pi, const int4 &info, RawUnit &ru) {
        const int n = pi.valid ? min(TB, g.K - info.y) : 0;
        const float *po = P.offset + (((int64_t)pi.b * g.og + info.z) * g.K + info.y) * DIM * (int64_t)g.P + pi.p;
        const float *pm = P.mask + (((int64_t)pi.b * g.mg + info.w) * g.K + info.y) * (int64_t)g.P + pi.p;
#pragma unroll
        for (int t = 0; t < TBM; ++t) {
#pragma unroll
            for (int a = 0; a < DIM; ++a) {
                ru.off[t][a] = (t < n && deformable) ? __ldg(po) : 0.f;
                po += g.P;
            }
            ru.m[t] = (t < n && P.mask != nullptr) ? __ldg(pm) : 1.f;
            pm += g.P;
        }
    };
    auto geometry = [&](const PosInfo<DIM> &pi, const RawUnit &ru, int t, int tap) -> TapGeometry<DIM> {
        TapGeometry<DIM> tg;
        const uint32_t tc = tap_tab[tap];
#pragma unroll
        for (int a = 0; a < DIM; ++a) {
            const int base = pi.base[a] + (int)(tc >> (10 * a) & 1023u) * g.dil[a];
            if (deformable) {
                const float pos = (float)base + ru.off[t][a];
                const float f = floorf(pos);
                tg.fl[a] = (int)f;
                tg.fr[a] = pos - f;
            } else {
                tg.fl[a] = base;
                tg.fr[a] = 0.f;
            }
        }
        tg.mval = ru.m[t];
        return tg;
    };

    // combines the dot products of a finished unit (an entry has two: even pixel row, odd one) into the coordinate gradients of its
    // (position, tap)s
    auto finalize = [&](const PosInfo<DIM> &pi, int pt, const int4 &info, int pb, const RawUnit &ru) {
        const int n = pi.valid ? min(TB, g.K - info.y) : 0;
        float *po = P.goff + (((int64_t)pi.b * g.og + info.z) * g.K + info.y) * DIM * (int64_t)g.P + pi.p;
        float *pm = P.gmask + (((int64_t)pi.b * g.mg + info.w) * g.K + info.y) * (int64_t)g.P + pi.p;
        const float2 *dots = reinterpret_cast<const float2 *>(plan_dot(pb)) + pt * TB * NP;
#pragma unroll 1
        for (int t = 0; t < n; ++t) {
            RawUnit one;                                     // (a loop, not TBM copies of its body: the registers are picked by selects)
#pragma unroll
            for (int k = 0; k < TBM; ++k) {
                if (k == 0 || k == t) {
#pragma unroll
                    for (int a = 0; a < DIM; ++a) one.off[0][a] = ru.off[k][a];
                    one.m[0] = ru.m[k];
                }
            }
            TapGeometry<DIM> tg = geometry(pi, one, 0, info.y + t);
            // A cell outside of the image has no gradients, whatever its fractions are: those of an infinite offset are NaN.  (Us, 128 x 256 x 28 x
            // 28 bf16 / 8 x 64 x 160 x 160 bf16 / 4 x 64 x 16 x 56 x 56 coordinate gradients f32: selects of the results, behind the contraction, 547 /
            // 301 / 1026; leaving the body here 527 / 271 / 1053; selects of the fractions 531 / 275 / 1020.)
            bool inside = true;
#pragma unroll
            for (int a = 0; a < DIM; ++a) inside = inside && (unsigned)tg.fl[a] + 1u <= (unsigned)g.img[a];
#pragma unroll
            for (int a = 0; a < DIM; ++a) tg.fr[a] = inside ? tg.fr[a] : 0.f;
            // the dots at the corners of the cell, then contracted axis by axis, the last one first: with the weights, and with (-1, 1) for
            // the axis whose derivative it is
            float val[NC], der[DIM][NC];
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                uint32_t left, key;
                bool okl, okr;
                float wl, wr;
                pair_of<DIM>(g, pi, tg, deformable, q, left, key, okl, okr, wl, wr);
                const float2 e = dots[q];
                const bool odd = (left & 1u) != 0u;
                val[2 * q] = okl ? (odd ? e.y : e.x) : 0.f;
                val[2 * q + 1] = okr ? (odd ? e.x : e.y) : 0.f;
            }
            dots += NP;
#pragma unroll
            for (int a = DIM - 1; a >= 0; --a) {
                const float f = tg.fr[a], f1 = 1.f - f;
#pragma unroll
                for (int i = 0; i < (1 << a); ++i) {
                    der[a][i] = val[2 * i + 1] - val[2 * i];
                    val[i] = fmaf(f, val[2 * i + 1], f1 * val[2 * i]);
#pragma unroll
                    for (int a2 = a + 1; a2 < DIM; ++a2) der[a2][i] = fmaf(f, der[a2][2 * i + 1], f1 * der[a2][2 * i]);
                }
            }
            if (P.goff != nullptr) {
#pragma unroll
                for (int a = 0; a < DIM; ++a) {
                    atomicAdd(po, tg.mval * der[a][0]);
                    po += g.P;
                }
            }
            if (P.gmask != nullptr) atomicAdd(pm, val[0]);
            pm += g.P;
        }
    };

    // ------------------------------------------------------------------ dense tile -> tensor memory
    // Thread = position (its TMEM lane); `loaders` warps per lane quarter split the channels in units of 16 (8 TMEM
    // columns), this warp being number `part` of them.
    auto load_dense = [&](const UnitIter &u, int part, int loaders, uint64_t *bar) {
        constexpr int U = 2;                            // units (of 16 loads) in flight per thread
        const int q = warp & 3;
        const PosInfo<DIM> pa = decode_blocked<DIM>(P, (long long)u.x * TILE_POS + q * 32 + lane);
        const uint32_t t_lane = tmem_base + ((uint32_t)(q * 32) << 16);
        const int64_t base = ((int64_t)pa.b * g.Cd_r + (int64_t)u.grp * g.cdg_r) * g.P + pa.p;
        const int n_units_a = g.cdg / 16;
        using TD = typename std::conditional<M::F32, float, uint16_t>::type;
        using TV = typename std::conditional<M::F32, float, uint32_t>::type;
        const TD *dense = static_cast<const TD *>(P.dense) + base;
        for (int u0 = part; u0 < n_units_a; u0 += U * loaders) {
            TV v[U][16];
#pragma unroll
            for (int h = 0; h < U; ++h) {
                const int c0 = (u0 + h * loaders) * 16;
                const int n = pa.valid ? g.cdg_r - c0 : 0;      // channels past the group's end are zeros
                const TD *src = dense + (int64_t)c0 * g.P;
                if (n >= 16) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[h][i] = (TV)__ldg(src + (int64_t)i * g.P);
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[h][i] = i < n ? (TV)__ldg(src + (int64_t)i * g.P) : (TV)0;
                }
            }
            __syncwarp();                                       // tcgen05.st is a whole-warp instruction
#pragma unroll
            for (int h = 0; h < U; ++h) {
                if (u0 + h * loaders >= n_units_a) break;
                const uint32_t t_col = t_lane + (uint32_t)((u0 + h * loaders) * 8);
                uint32_t part16[8];
                if constexpr (M::F32) {
#pragma unroll
                    for (int k = 0; k < PARTS; ++k) {           // v keeps what the parts so far leave
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            part16[i] = pack2(v[h][2 * i], v[h][2 * i + 1], __nv_bfloat16());
                            v[h][2 * i] -= __uint_as_float(part16[i] << 16);
                            v[h][2 * i + 1] -= __uint_as_float(part16[i] & 0xffff0000u);
                        }
                        ptx::tmem_st_32x8(t_col + (uint32_t)(k * a_cols), part16);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) part16[i] = v[h][2 * i] | (v[h][2 * i + 1] << 16);
                    ptx::tmem_st_32x8(t_col, part16);
                }
            }
        }
        ptx::tmem_st_wait();
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(bar);
    };

    if (warp < SC_WORK_WARPS) {
        if (warp < SC_FINISH_WARPS) {
            // -------------------------------------------------------------- finishing warps: coordinate gradients, dense tiles
            load_dense(first_unit(P, unit0), warp >> 2, SC_LOAD_WARPS / 4, a_first);   // before registers are handed over
            take_registers<SC_REGS_FINISH>();
            const int row = warp * 32 + lane;
            // this thread's position in the tile of unit j
            auto position = [&](int j) {
                const int2 at = pos_of(j)[row];
                PosInfo<DIM> pi;
                pi.valid = at.x >= 0;
                pi.b = max(at.x, 0);
                pi.p = at.y;
                decode_in_image<DIM>(g, pi);
                return pi;
            };
            // The gather warps are through with unit j: its dot products become gradients.
            auto finish_unit = [&](int j) -> bool {
                bool good = ptx::mbar_wait_backoff<SC_SLEEP_NS>(&plan_done[j & 1], (uint32_t)((j >> 1) & 1));
                good = __all_sync(0xffffffffu, good);
                if (!good) {
                    if (lane == 0) ptx::report(P.status, 308);
                    return false;
                }
                const PosInfo<DIM> pi = position(j);
                RawUnit ru;
                load_unit(pi, *info_of(j), ru);
                finalize(pi, row, *info_of(j), j & 1, ru);
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&fin_done[j & 1]);
                return true;
            };
            // The next tile is loaded as soon as the old one's last MMA is through.  With four accumulators the MMAs run two units ahead of the
            // gather warps, with two one unit: while those walk unit j, that moment comes for tiles that end with unit j + lead.
            const int lead = NACC >= 4 ? 2 : (NACC >= 2 ? 1 : 0);
            int next_tile = P.n_units - unit0 % P.n_units;       // first unit of the next tile to be loaded
            UnitIter u = first_unit(P, unit0);
            uint32_t phase = 0;
            bool ok = true;
            for (int j = 0; j < n_units && ok; ++j) {
                if (COORD && j > 0) ok = finish_unit(j - 1);
                for (; ok && next_tile < n_units && next_tile - 1 - lead <= j; next_tile += P.n_units) {
                    ok = ptx::mbar_wait_backoff<SC_SLEEP_NS>(a_free, phase);
                    phase ^= 1u;
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) {
                        if (lane == 0) ptx::report(P.status, 309);
                        break;
                    }
                    ptx::tc_fence_after();
                    ++u.order;
                    locate_tile(P, u);
                    load_dense(u, 0, 1, a_next);
                }
            }
            if (COORD && ok) finish_unit(n_units - 1);   // the last unit
        } else {
            // -------------------------------------------------------------- gather warps
            if (warp < SC_LOAD_WARPS) load_dense(first_unit(P, unit0), warp >> 2, SC_LOAD_WARPS / 4, a_first);
            take_registers<SC_REGS_GATHER>();
            // An 8-lane group walks its span of the pixel-grouped entry list; lane l8 owns channels 4 l8 .. 4 l8 + 3 and
            // 32 + 4 l8 .. of the chunk, so that the 8 lanes' 16-byte accesses to columns and sums are contiguous.  An entry is a
            // pair of neighbouring pixels, so it reads its column values once for both; the one with the even row number adds into the
            // sums `ev`, the other into `od`, each with a pixel of its own that changes every second step along an image row.
            // (A warp's four spans lie a quarter of the list apart: at its ends, where the pixels have few entries, every entry costs a flush,
            // and a warp with such spans only is the one that all wait for: 543 -> 531 us, f32 709 -> 678.)
            const int gid = (lane >> 3) * SC_GATHER_WARPS + warp - SC_FINISH_WARPS;
            const int l8 = lane & 7;
            using TI = typename std::conditional<M::F32, float, T16>::type;
            constexpr int IW = M::F32 ? 8 : 4;              // words of an image row per lane
            struct Rows {
                uint32_t ev[IW], od[IW];
            };
            // Columns of a unit, TMEM -> shared: a warp reads the lanes of its quarter, the warps of a quarter share the columns out in
            // blocks of 16.
            const int q = warp & 3, part = (warp - SC_FINISH_WARPS) >> 2;
            float *col_row = col + (q * 32 + lane) * L.col_stride;
            int aq = 0;
            uint32_t t_phase = 0;
            bool ok = true;
            for (int j = 0; j < n_units && ok; ++j) {
                const int pb = j & 1;
                if (j > 0) ok = ptx::mbar_wait(&plan_done[pb ^ 1], (uint32_t)(((j - 1) >> 1) & 1));   // the columns of the unit before have been used
                for (int slab = 0; slab < 2; ++slab) {
                    ok = ok && ptx::mbar_wait(&t_full[aq], t_phase);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) {
                        if (lane == 0) ptx::report(P.status, 301);
                        break;
                    }
                    ptx::tc_fence_after();
                    const uint32_t src = tmem_base + ((uint32_t)(q * 32) << 16) + acc_col0 + (uint32_t)(aq * ACCS * N);
                    for (int blk = part; blk < 2 * TB; blk += SC_GATHER_WARPS / 4) {
                        uint32_t raw[16];
                        ptx::tmem_ld_32x16(src + (uint32_t)(blk * 16), raw);
                        ptx::tmem_ld_wait();
                        if constexpr (ACCS == 2) {
                            uint32_t low[16];
                            ptx::tmem_ld_32x16(src + (uint32_t)(N + blk * 16), low);
                            ptx::tmem_ld_wait();
#pragma unroll
                            for (int e = 0; e < 16; ++e)
                                raw[e] = __float_as_uint(__uint_as_float(raw[e]) + __uint_as_float(low[e]));
                        }
                        float *dst = col_row + (blk >> 1) * CHUNK_C + slab * SC_SLAB + (blk & 1) * 16;
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            *reinterpret_cast<uint4 *>(dst + 4 * e) =
                                make_uint4(raw[4 * e], raw[4 * e + 1], raw[4 * e + 2], raw[4 * e + 3]);
                    }
                    ptx::tc_fence_before();
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive(&t_empty[aq]);
                    if (++aq == NACC) {
                        aq = 0;
                        t_phase ^= 1u;
                    }
                }
                if (!ok) break;
                if (lane == 0) ptx::mbar_arrive(col_full);
                ok = ptx::mbar_wait(&plan_full[pb], (uint32_t)((j >> 1) & 1));
                if (COORD && j >= 2) ok = ok && ptx::mbar_wait(&fin_done[pb], (uint32_t)(((j >> 1) & 1) ^ 1));
                ok = ok && ptx::mbar_wait(col_full, (uint32_t)(j & 1));
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) {
                    if (lane == 0) ptx::report(P.status, 306);
                    break;
                }
                const int span = (int)n_entries[pb];     // entries per group, padded: a multiple of 2
                const uint4 *my_ent = plan_ent(pb) + gid * span;
                const uint2 *my_meta = reinterpret_cast<const uint2 *>(plan_meta(pb) + gid * span);
                float *p_dot = plan_dot(pb);
                const float4 *colb = reinterpret_cast<const float4 *>(col) + l8;
                const uint32_t chan = (uint32_t)(info_of(j)->x + l8 * 4);
                // opaque: the compiler would take the sums of base, channel and row apart and add six times
                uint64_t img_c = reinterpret_cast<uint64_t>(reinterpret_cast<const TI *>(P.img_cl) + chan);
                uint64_t gimg_c = reinterpret_cast<uint64_t>(P.img_grad_cl + chan);
                asm volatile("" : "+l"(img_c), "+l"(gimg_c));

                float ev[8], od[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) ev[k] = od[k] = 0.f;
                auto fetch_rows = [&](Rows &rows, const uint4 &e, uint32_t was_ev, uint32_t was_od) {
                    if constexpr (COORD) {
                        load_row<IW>(e.x, was_ev, rows.ev, row_at<sizeof(TI)>(img_c, e.x));
                        load_row<IW>(e.y, was_od, rows.od, row_at<sizeof(TI)>(img_c, e.y));
                    }
                };
                // this lane's share of <column, image row>
                auto dot = [&](const uint64_t (&c)[4], const uint32_t (&row)[IW]) -> float {
                    uint64_t d = 0;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        uint64_t iv;
                        if constexpr (M::F32) {
                            iv = pack_f32x2(__uint_as_float(row[2 * k]), __uint_as_float(row[2 * k + 1]));
                        } else if constexpr (M::HALF) {
                            const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&row[k]));
                            iv = pack_f32x2(f.x, f.y);
                        } else {
                            iv = pack_f32x2(__uint_as_float(row[k] << 16), __uint_as_float(row[k] & 0xffff0000u));
                        }
                        d = k == 0 ? mul_f32x2(c[k], iv) : fma_f32x2(c[k], iv, d);
                    }
                    return __uint_as_float((uint32_t)d) + __uint_as_float((uint32_t)(d >> 32));
                };
                // Adds weight x column to the sums, which were those of the pixels of `prev` and are now those of e's.  The test of the weights, us:
                // f32 data, one branch for entries that have both pixels, 8 x 64 x 16 x 56 x 56 2629, 128 x 256 x 28 x 28 676; a branch for each
                // pixel 2737, 680; bf16 2406, 576 and 2306, 531 (predicated multiply-adds 2456, 580).
                auto add = [&](const uint4 &prev, const uint4 &e, const uint64_t (&c)[4]) {
                    if constexpr (M::F32) {
                        flush_sums(e.x, prev.x, row_at<4>(gimg_c, prev.x), ev);
                        flush_sums(e.y, prev.y, row_at<4>(gimg_c, prev.y), od);
                        if (max(e.z, e.w) != SC_NO_WEIGHT) {
                            add_weighted(ev, e.z, c);
                            add_weighted(od, e.w, c);
                        } else {
                            if (e.z != SC_NO_WEIGHT) add_weighted(ev, e.z, c);
                            if (e.w != SC_NO_WEIGHT) add_weighted(od, e.w, c);
                        }
                    } else {
                        flush_sums(e.x, prev.x, row_at<4>(gimg_c, prev.x), ev);
                        if (e.z != SC_NO_WEIGHT) add_weighted(ev, e.z, c);
                        flush_sums(e.y, prev.y, row_at<4>(gimg_c, prev.y), od);
                        if (e.w != SC_NO_WEIGHT) add_weighted(od, e.w, c);
                    }
                };
                // One entry, the one before it being `prev`; its image rows are in `rows`, which then receives those of `next`.
                auto load_columns = [&](uint64_t (&c)[4], uint32_t meta) {
                    const float4 a = colb[meta & 0xffffu], b = colb[(meta & 0xffffu) + 8];
                    c[0] = pack_f32x2(a.x, a.y);
                    c[1] = pack_f32x2(a.z, a.w);
                    c[2] = pack_f32x2(b.x, b.y);
                    c[3] = pack_f32x2(b.z, b.w);
                };
                auto step = [&](const uint4 &prev, const uint4 &e, const uint64_t (&c)[4], Rows &rows, const uint4 &next, float &d_ev, float &d_od) {
                    if constexpr (COORD) {
                        d_ev = dot(c, rows.ev);
                        d_od = dot(c, rows.od);
                    }
                    fetch_rows(rows, next, e.x, e.y);
                    if constexpr (SCATTER) add(prev, e, c);
                };
                // sums over the 8 lanes of the four dots of two entries at once: after the exchanges lane (b2 b1 b0) holds dot 2 b2 + b1
                auto reduce = [&](const float (&d)[4], uint32_t m0, uint32_t m1) {
                    if constexpr (COORD) {
                        const bool h4 = (l8 & 4) != 0, h2 = (l8 & 2) != 0;
                        float k0 = h4 ? d[2] : d[0], k1 = h4 ? d[3] : d[1];
                        k0 += __shfl_xor_sync(0xffffffffu, h4 ? d[0] : d[2], 4);
                        k1 += __shfl_xor_sync(0xffffffffu, h4 ? d[1] : d[3], 4);
                        float k = h2 ? k1 : k0;
                        k += __shfl_xor_sync(0xffffffffu, h2 ? k0 : k1, 2);
                        k += __shfl_xor_sync(0xffffffffu, k, 1);
                        if ((l8 & 1) == 0) p_dot[((h4 ? m1 : m0) >> 16) + (h2 ? 1 : 0)] = k;
                    }
                };
                if (span > 0) {
                    uint4 A = my_ent[0], B = my_ent[1], C, D;
                    // image rows: f32 data has registers for one entry's, 16-bit data for two
                    Rows ra, rb;
                    Rows &rn = M::F32 ? ra : rb;
                    fetch_rows(ra, A, ~A.x, ~A.y);
                    if constexpr (!M::F32) fetch_rows(rb, B, ~B.x, ~B.y);
                    uint4 last = A;     // the running pixels start as the first entry's: no flush before anything was summed
                    // Entries are read two ahead, their columns one, past the end of the span: still inside the list's slack.
                    uint64_t ca[4], cb[4];
                    uint2 m = my_meta[0];
                    load_columns(ca, m.x);
#pragma unroll 1
                    for (int it = 0; it < span; it += 2) {
                        float d[4];
                        const uint2 m2 = my_meta[(it >> 1) + 1];
                        C = my_ent[it + 2];
                        load_columns(cb, m.y);
                        step(last, A, ca, ra, M::F32 ? B : C, d[0], d[1]);
                        D = my_ent[it + 3];
                        load_columns(ca, m2.x);
                        step(A, B, cb, rn, M::F32 ? C : D, d[2], d[3]);
                        reduce(d, m.x, m.y);
                        last = B;
                        A = C;
                        B = D;
                        m = m2;
                    }
                    if constexpr (SCATTER) {
                        flush_sums(~last.x, last.x, row_at<4>(gimg_c, last.x), ev);
                        flush_sums(~last.y, last.y, row_at<4>(gimg_c, last.y), od);
                    }
                }
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&plan_done[pb]);
            }
        }
    } else if (warp < SC_MMA_WARP) {
        // ------------------------------------------------------------------ planners
        take_registers<SC_REGS_PLAN>();
        const int pt = threadIdx.x - SC_PLAN_WARP0 * 32;
        const int pw = warp - SC_PLAN_WARP0;
        UnitIter u = first_unit(P, unit0);
        PosInfo<DIM> pi = decode_blocked<DIM>(P, (long long)u.x * TILE_POS + pt);
        const uint32_t colq_row = (uint32_t)(pt * (L.col_stride / 4));
        const uint32_t pixels = (uint32_t)g.B * (uint32_t)g.S;
        const uint32_t padding = blockIdx.x % pixels * (uint32_t)g.Cs;   // where entries that pad the list add nothing: not one row for all

        // four words of padding behind every 32: a thread's 16 slots then meet those of its seven neighbours in no bank
        auto word_of = [](uint32_t slot) { return slot + (slot >> 5) * 4u; };
        // one thread waits, all learn the result: the named barrier must always see all 128 threads
        auto wait_all = [&](uint64_t *bar, uint32_t parity) -> bool {
            if (pt == 0) *wait_flag = ptx::mbar_wait_backoff<SC_SLEEP_NS>(bar, parity) ? 1u : 0u;
            planner_barrier();
            const bool r = *wait_flag != 0u;
            planner_barrier();
            return r;
        };
        auto build = [&](const int4 &info, int j, const RawUnit &ru) {
            const int t0 = info.y, pb = j & 1;
            if (pt == 0) *info_of(j) = info;
            pos_of(j)[pt] = make_int2(pi.valid ? pi.b : -1, pi.p);
            {
                uint4 *c4 = reinterpret_cast<uint4 *>(cnt + word_of(pt * 16));
#pragma unroll
                for (int i = 0; i < 4; ++i) c4[i] = make_uint4(0u, 0u, 0u, 0u);
            }
            planner_barrier();
            // pass 1: every entry's rank within its slot; all atomics of a thread are independent
            constexpr bool AGAIN = TBM * NP > 8;            // pass 2 works pixels and weights out again: there are no registers to keep them
            constexpr int KEPT = AGAIN ? 1 : TBM * NP;
            uint32_t left[KEPT];
            uint32_t slot[TBM * NP];                        // slot, then (12 bits up) the rank in it; two top bits: left, right pixel in the image
            float wl[KEPT], wr[KEPT];
#pragma unroll
            for (int t = 0; t < TBM; ++t) {
                const bool live = t < TB && t0 + t < g.K && pi.valid;
                const TapGeometry<DIM> tg = geometry(pi, ru, t, t0 + t);
#pragma unroll
                for (int q = 0; q < NP; ++q) {
                    const int i = t * NP + q, k = AGAIN ? 0 : i;
                    bool okl, okr;
                    uint32_t key;
                    pair_of<DIM>(g, pi, tg, deformable, q, left[k], key, okl, okr, wl[k], wr[k]);
                    wl[k] *= tg.mval;
                    wr[k] *= tg.mval;
                    slot[i] = key | ((live && okl) ? 1u << 30 : 0u) | ((live && okr) ? 1u << 31 : 0u);
                }
            }
#pragma unroll
            for (int i = 0; i < TBM * NP; ++i)
                if ((slot[i] >> 30) != 0u) slot[i] |= atomicAdd(&cnt[word_of(slot[i] & (SC_SLOTS - 1))], 1u) << 12;
            planner_barrier();
            // exclusive prefix sum of the slot counts, in place (16 slots per thread)
            uint32_t total;
            {
                uint32_t v[16];
                uint32_t s = 0;
                uint4 *c4 = reinterpret_cast<uint4 *>(cnt + word_of(pt * 16));
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint4 x = c4[i];
                    v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
                    s += x.x + x.y + x.z + x.w;
                }
                uint32_t inc = s;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t o = __shfl_up_sync(0xffffffffu, inc, d);
                    if (lane >= d) inc += o;
                }
                if (lane == 31) scan_part[pw] = inc;
                planner_barrier();
                uint32_t run = inc - s;
                total = 0;
#pragma unroll
                for (int w = 0; w < SC_PLAN_WARPS; ++w) {
                    const uint32_t part = scan_part[w];
                    if (w < pw) run += part;
                    total += part;
                }
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    const uint32_t a = run + v[i], b = a + v[i + 1], c = b + v[i + 2];
                    c4[i >> 2] = make_uint4(run, a, b, c);
                    run = c + v[i + 3];
                }
            }
            // entries per gather group: a multiple of 2; the list is padded with entries that add nothing
            const uint32_t span = ((total + SC_GROUPS * 2 - 1) / (SC_GROUPS * 2)) * 2;
            if (pt == 0) n_entries[pb] = span;
            planner_barrier();
            // pass 2: every entry goes to (start of its slot) + (its rank)
            uint4 *ent = plan_ent(pb);
            uint32_t *e_meta = plan_meta(pb);
#pragma unroll
            for (int t = 0; t < TBM; ++t) {
                TapGeometry<DIM> tg;
                if constexpr (AGAIN) tg = geometry(pi, ru, t, t0 + t);
#pragma unroll
                for (int q = 0; q < NP; ++q) {
                    const int i = t * NP + q, k = AGAIN ? 0 : i;
                    const uint32_t both = slot[i] >> 30;
                    if (both != 0u) {
                        if constexpr (AGAIN) {
                            bool okl, okr;
                            uint32_t key;
                            pair_of<DIM>(g, pi, tg, deformable, q, left[0], key, okl, okr, wl[0], wr[0]);
                            wl[0] *= tg.mval;
                            wr[0] *= tg.mval;
                        }
                        const uint32_t at = cnt[word_of(slot[i] & (SC_SLOTS - 1))] + (slot[i] >> 12 & 0xfffu);
                        // (not behind the last pixel nor, where left is -1, before the first)
                        const uint32_t pl = min(left[k], left[k] + 1u) * (uint32_t)g.Cs;
                        const uint32_t pr = min(left[k] + 1u, pixels - 1u) * (uint32_t)g.Cs;
                        const bool odd = (left[k] & 1u) != 0u;
                        const uint32_t a = (both & 1u) ? __float_as_uint(wl[k]) : SC_NO_WEIGHT;
                        const uint32_t b = (both & 2u) ? __float_as_uint(wr[k]) : SC_NO_WEIGHT;
                        ent[at] = odd ? make_uint4(pr, pl, b, a) : make_uint4(pl, pr, a, b);
                        e_meta[at] = (colq_row + (uint32_t)(t * (CHUNK_C / 4))) | ((uint32_t)((pt * TB + t) * NC + 2 * q) << 16);
                    }
                }
            }
            // padding entries up to the end of the last span and the words the read-ahead of the last group touches
            const uint32_t n_words = span * SC_GROUPS + 4;
            for (uint32_t i = total + pt; i < n_words; i += 128) {
                ent[i] = make_uint4(padding, padding, SC_NO_WEIGHT, SC_NO_WEIGHT);
                e_meta[i] = (uint32_t)(2 * L.max_entries) << 16;
            }
            planner_barrier();
            if (lane == 0) ptx::mbar_arrive(&plan_full[pb]);
        };

        bool ok = true;
        RawUnit ru, ru_next;
        int4 info = describe(u);
        load_unit(pi, info, ru);
        ru_next = ru;
        for (int j = 0; j < n_units && ok; ++j) {
            const int pb = j & 1;
            if (j >= 2) {
                ok = wait_all(&plan_done[pb], (uint32_t)(((j >> 1) & 1) ^ 1));
                if (!ok) {
                    if (pt == 0) ptx::report(P.status, 307);
                    break;
                }
            }
            // the next unit's offsets and mask travel while this unit is built
            UnitIter u_next = u;
            const bool next_new = next_unit(P, u_next);
            PosInfo<DIM> pi_next = pi;
            if (next_new) pi_next = decode_blocked<DIM>(P, (long long)u_next.x * TILE_POS + pt);
            const int4 info_next = describe(u_next);
            if (j + 1 < n_units) load_unit(pi_next, info_next, ru_next);
            build(info, j, ru);
            ru = ru_next;
            u = u_next;
            pi = pi_next;
            info = info_next;
        }
    } else if (warp == SC_MMA_WARP) {
        // ------------------------------------------------------------------ MMA issue
        take_registers<SC_REGS_ISSUE>();
        if (lane == 0) {
            const uint32_t idesc = ptx::instr_desc_f16(M::HALF ? 0 : 1, TILE_POS, N, 0, 0);
            bool ok = true, new_tile = true;
            UnitIter u = first_unit(P, unit0);
            // ring position and phase are stepped, never divided: a division by the run-time ring depth per stage
            // costs this single thread more than the stage's MMAs
            int s = 0, aq = 0;
            uint32_t b_phase = 0, t_phase = 1, a_phase = 0;
            const uint64_t b_desc0 = ptx::smem_desc_sw128(ptx::smem_u32(sB), 16, 1024);
            for (int jp = 0; jp < n_pass && ok; ++jp) {
                if ((jp & 1) == 0) {
                    if (new_tile) {
                        ok = jp == 0 ? ptx::mbar_wait(a_first, 0) : ptx::mbar_wait(a_next, a_phase);
                        if (jp > 0) a_phase ^= 1u;
                        if (!ok) {
                            ptx::report(P.status, 302);
                            break;
                        }
                        ptx::tc_fence_after();
                    }
                    new_tile = next_unit(P, u);
                }
                if (!ptx::mbar_wait_backoff<SC_SLEEP_NS>(&t_empty[aq], t_phase)) {
                    ptx::report(P.status, 303);
                    ok = false;
                    break;
                }
                ptx::tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc_col0 + (uint32_t)(aq * ACCS * N);
                // f32 data: the parts of a weight chunk are stages of their own; part b meets the dense parts a with
                // a + b < PARTS (two parts: hi x hi, lo x hi; hi x lo)
                for (int st = 0; st < RC * PARTS && ok; ++st) {
                    const int rc = st / PARTS, part = st % PARTS;
                    if (!ptx::mbar_wait(&b_full[s], b_phase)) {
                        ptx::report(P.status, 304);
                        ok = false;
                        break;
                    }
                    // no tcgen05 fence here: the stage was filled by TMA (async proxy, like the MMA's own reads) and
                    // the fence would wait for the MMAs in flight to drain, once per stage
                    // descriptor of the stage = descriptor of stage 0 + its byte distance / 16; one K = 16 step further
                    // is 32 bytes inside the swizzled rows (+ 2), 8 TMEM columns of A
                    const uint64_t b_desc = b_desc0 + (uint64_t)((uint32_t)s * (L.b_stage >> 4));
                    const uint32_t a_hi = tmem_base + (uint32_t)(rc * 32);
                    // the products of one weight part with the dense parts PA0 ... PA1 - 1, into accumulator d
                    auto products = [&](uint32_t d, auto pa0, auto pa1, bool open) {
#pragma unroll
                        for (int k4 = 0; k4 < 4; ++k4)
#pragma unroll
                            for (int pa = decltype(pa0)::value; pa < decltype(pa1)::value; ++pa) {
                                const uint32_t a_k = a_hi + (uint32_t)(pa * a_cols + k4 * 8);
                                if (k4 == 0 && pa == decltype(pa0)::value)
                                    ptx::mma_f16_ts(d, a_k, b_desc, idesc, open ? 0u : 1u);
                                else
                                    ptx::mma_f16_ts_acc(d, a_k, b_desc + (uint64_t)(2 * k4), idesc);
                            }
                    };
                    using std::integral_constant;
                    const bool open = rc == 0;
                    if constexpr (ACCS == 1) {
                        if (part == 0)
                            products(d_tmem, integral_constant<int, 0>(), integral_constant<int, PARTS>(), open);
                        else
                            products(d_tmem, integral_constant<int, 0>(), integral_constant<int, 1>(), false);
                    } else {
                        const uint32_t d_low = d_tmem + (uint32_t)N;
                        if (part == 0) {
                            products(d_tmem, integral_constant<int, 0>(), integral_constant<int, 1>(), open);
                            products(d_low, integral_constant<int, 1>(), integral_constant<int, 3>(), open);
                        } else if (part == 1) {
                            products(d_low, integral_constant<int, 0>(), integral_constant<int, 2>(), false);
                        } else {
                            products(d_low, integral_constant<int, 0>(), integral_constant<int, 1>(), false);
                        }
                    }
                    ptx::mma_commit(&b_empty[s]);
                    if (++s == BS) {
                        s = 0;
                        b_phase ^= 1u;
                    }
                }
                if (ok) ptx::mma_commit(&t_full[aq]);
                // the tile's last pass, and another tile follows
                if (ok && (jp & 1) && new_tile && jp + 1 < n_pass) ptx::mma_commit(a_free);
                if (++aq == NACC) {
                    aq = 0;
                    t_phase ^= 1u;
                }
            }
        }
        __syncwarp();
    } else if (warp == SC_TMA_WARP) {
        // ------------------------------------------------------------------ TMA: weight ring
        take_registers<SC_REGS_ISSUE>();
        if (lane == 0) {
            int s = 0, last_s = -1;
            uint32_t e_phase = 1, last_phase = 0;
            bool ok = true;
            UnitIter u = first_unit(P, unit0);
            for (int jp = 0; jp < n_pass && ok; ++jp) {
                const int t0 = u.batch * TB, grp = u.grp;
                const int s0 = u.chunk * CHUNK_C + (jp & 1) * SC_SLAB;
                for (int st = 0; st < RC * PARTS; ++st) {
                    const int rc = st / PARTS, part = st % PARTS;
                    if (!ptx::mbar_wait_backoff<SC_SLEEP_NS>(&b_empty[s], e_phase)) {
                        ptx::report(P.status, 305);
                        ok = false;
                        break;
                    }
                    ptx::mbar_arrive_expect_tx(&b_full[s], L.b_stage);
                    ptx::tma_load_4d(sB + (size_t)s * L.b_stage, part == 0 ? &tmap_b_hi : (part == 1 ? &tmap_b_lo : &tmap_b_lo2), &b_full[s], rc * 64, s0,
                                     t0, grp);
                    last_s = s;
                    last_phase = e_phase ^ 1u;
                    if (++s == BS) {
                        s = 0;
                        e_phase ^= 1u;
                    }
                }
                if (!ok) break;
                if (jp & 1) next_unit(P, u);
            }
            // no copy may still be in flight when the CTA's shared memory is released
            if (last_s >= 0) ptx::mbar_wait(&b_full[last_s], last_phase);
        }
        __syncwarp();
    } else {
        take_registers<SC_REGS_ISSUE>();   // the two idle warps of the last warpgroup
    }

    ptx::tc_fence_before();
    __syncthreads();
    if (warp == SC_MMA_WARP) ptx::tmem_dealloc(tmem_base, SC_TMEM_COLS);
}

size_t dgrad_smem_bytes(int dim, int tb, int b_stages) {
    return 1024 + sc_layout(dim, tb, b_stages).total;
}

template <int DIM, int MODE>
cudaError_t launch_dgrad_t(const DgradParams<DIM> &P, const CUtensorMap *maps, cudaStream_t stream) {
    const size_t smem = dgrad_smem_bytes(DIM, P.tb, P.b_stages);
    const bool coord = P.goff != nullptr || P.gmask != nullptr;
    // One CTA per SM, except for f32 volumes of many tiles, whose costs differ so much that the hardware's scheduling beats equal
    // ranges, once a tile has units enough to outweigh a CTA's start-up.  64 channels, us, ranges / one CTA per tile.  Backward kernel, f32,
    // 27 taps (nine units): 392 tiles 328 / 355, 784 668 / 701, 1568 1388 / 1330, 3136 2769 / 2597; 18 taps (six) 1568 871 / 904, 6272 3783 /
    // 3531, the transposed one 3164 / 2924; 8 taps (three) 1568 480 / 502, 2352 723 / 742, 6272 1934 / 1931, transposed with stride 2 2744
    // 1039 / 951; 6 taps (two) 1568 383 / 418, 2352 611 / 617; one tap 132 / 205, 179 / 293.  So the lines are at ten tiles per SM and three
    // units.  The scatter alone: 27 taps 1568 744 / 822, 8 taps 277 / 344, but with stride 2 2744 887 / 768; 6 taps 1568 209 / 279, one tap 99 / 154.
    // 16-bit data, with its shorter start-up but also shorter tiles: 27 taps 784 601 / 678, 3136 2348 / 2479, 8 taps 2744 662 / 758.
    const int tiles = P.total_units / P.n_units;
    const bool one_per_tile = DIM == 3 && Mode<MODE>::F32 && P.n_units >= 3 && tiles >= 10 * 148;
    const dim3 grid((unsigned)(one_per_tile ? tiles : std::min(P.total_units, 148)));
    LaunchScope scope("dcn_dgrad_tc", stream);
    auto run = [&](auto want) {
        return launch_dependent<dcn_dgrad_tc_kernel<DIM, MODE, decltype(want)::value>>(grid, SC_THREADS, smem, stream, P, maps[0],
                                                                                       maps[1], maps[2]);
    };
    if (!coord) return run(std::integral_constant<int, SC_SCATTER>());
    if (P.img_grad_cl == nullptr) return run(std::integral_constant<int, SC_COORD>());
    return run(std::integral_constant<int, SC_SCATTER | SC_COORD>());
}

}  // namespace

// Position tiles, and the units they are cut into (per tile and group, and in all); false from 2^31 units on.
static bool dgrad_units(const GeoHost &h, int tb, int *tiles_x, int *per_tile, int *total) {
    const long long tx = ((long long)h.B * h.P + TILE_POS - 1) / TILE_POS;
    const long long n = (long long)(h.Cs / h.groups / CHUNK_C) * ((h.K + tb - 1) / tb), all = tx * h.groups * n;
    if (all > 0x7fffffffLL) return false;
    *tiles_x = (int)tx;
    *per_tile = (int)n;
    *total = (int)all;
    return true;
}

// Taps per batch, accumulator ring and weight-ring depth that fit tensor memory and shared memory; false when
// nothing fits (the dense tile of one group must fit tensor memory beside one accumulator) or the work is too much.
bool dgrad_tc_config(const GeoHost &h, int mode, int *tb, int *nacc, int *b_stages) {
    const int K = h.K, a_cols = (h.Cd / h.groups / 2) * mode_mat_parts(mode);
    for (int cand = std::min(sc_tb_max(h.dim), K); cand >= 1; --cand) {
        // equal batches: the fewest batches of at most `cand` taps
        const int nb = (K + cand - 1) / cand;
        const int t = (K + nb - 1) / nb;
        const int n = t * SC_SLAB;
        const int acc = std::min(4, (SC_TMEM_COLS - a_cols) / (n * (mode == TC_F32_WIDE ? 2 : 1)));
        if (acc < 1) continue;
        for (int st = 4; st >= 2; --st)
            if (dgrad_smem_bytes(h.dim, t, st) <= 227 * 1024) {
                int tiles, per_tile, total;
                if (!dgrad_units(h, t, &tiles, &per_tile, &total)) return false;
                *tb = t;
                *nacc = acc;
                *b_stages = st;
                return true;
            }
    }
    return false;
}

// dense: [B, Cd_r, P] in the problem's data type; w_parts: weights packed [g][tap][s'][d'], one 16-bit tensor per part;
// img_cl: sampled image channels-last (needed for goff / gmask); accumulation targets are f32 and initialised by
// the caller.
cudaError_t launch_gemm_scatter_tc(const GeoHost &h, int mode, const void *dense, void *const *w_parts,
                                   const void *img_cl, const float *offset, const float *mask, float *img_grad_cl, float *goff, float *gmask, const Status &status, cudaStream_t stream) {
    const int cdg = h.Cd / h.groups, csg = h.Cs / h.groups;
    int tb = 0, nacc = 0, bs = 0, tiles_x = 0, n_units = 0, total = 0;
    if (!dgrad_tc_config(h, mode, &tb, &nacc, &bs) || !dgrad_units(h, tb, &tiles_x, &n_units, &total))
        return cudaErrorInvalidConfiguration;
    const int nbatch = (h.K + tb - 1) / tb;
    CUtensorMap maps[3];
    {
        const uint64_t dims[4] = {(uint64_t)cdg, (uint64_t)csg, (uint64_t)h.K, (uint64_t)h.groups};
        const uint64_t strides[3] = {(uint64_t)cdg * 2, (uint64_t)cdg * csg * 2, (uint64_t)cdg * csg * h.K * 2};
        const uint32_t box[4] = {64, (uint32_t)SC_SLAB, (uint32_t)tb, 1};
        if (!make_part_maps(maps, w_parts, mode_mat_parts(mode), 4, dims, strides, box)) return cudaErrorInvalidValue;
    }
    auto run = [&](auto dimc) -> cudaError_t {
        constexpr int DIM = decltype(dimc)::value;
        DgradParams<DIM> P;
        P.g = geo_from_host<DIM>(h);
        P.dense = dense;
        P.img_cl = img_cl;
        P.offset = offset;
        P.mask = mask;
        P.img_grad_cl = img_grad_cl;
        P.goff = goff;
        P.gmask = gmask;
        P.status = status;
        P.rc = cdg / 64;
        P.tb = tb;
        P.nbatch = nbatch;
        P.nacc = nacc;
        P.b_stages = bs;
        P.tiles_x = tiles_x;
        P.n_units = n_units;
        P.total_units = total;
        for (int a = 0; a < DIM; ++a) P.block[a] = std::min(h.grid[a], a == DIM - 1 ? 8 : 4);
        // 16-bit data: nothing is rounded between the MMA and the results, there is no wide mode of its own
        switch (mode) {
            case TC_BF16: case TC_BF16_WIDE: return launch_dgrad_t<DIM, TC_BF16>(P, maps, stream);
            case TC_F16: case TC_F16_WIDE: return launch_dgrad_t<DIM, TC_F16>(P, maps, stream);
            case TC_SPLIT: return launch_dgrad_t<DIM, TC_SPLIT>(P, maps, stream);
            case TC_F32_WIDE: return launch_dgrad_t<DIM, TC_F32_WIDE>(P, maps, stream);
        }
        return cudaErrorInvalidValue;
    };
    if (h.dim == 1) return run(std::integral_constant<int, 1>());
    if (h.dim == 2) return run(std::integral_constant<int, 2>());
    if (h.dim == 3) return run(std::integral_constant<int, 3>());
    return cudaErrorInvalidValue;
}

}  // namespace tvdcn_b200
