// Engine choice per GEMM-shaped primitive and workspace layout.
#include "plan.h"

#include <algorithm>

namespace tvdcn_b200 {

namespace {
struct Bump {
    size_t off = 0;
    size_t take(size_t bytes) {
        const size_t at = off;
        off = align_up(off + bytes);
        return at;
    }
};
// A granule of channels padded by more than this runs on the SIMT kernels.  A tensor-core kernel's time does not depend on how
// much of the 64 channels is real, a SIMT kernel's is proportional to it.  SIMT / tensor us at 4 x 128 x 128, 3 x 3 (f32; bf16),
// forward and backward: 4 channels 45 / 75, 171 / 241; 43 / 57, 176 / 203.  8 channels 74 / 76, 303 / 240; 70 / 58, 315 / 203.
// 12 channels 105 / 76, 343 / 240; 99 / 58, 357 / 203.
constexpr int MAX_CHANNEL_PADDING = 8;
bool is16(int dt) { return dt == DT_F16 || dt == DT_BF16; }

int gcd(int a, int b) { return b == 0 ? a : gcd(b, a % b); }
int round_up(int v, int m) { return (v + m - 1) / m * m; }

// Shape conditions shared by all tensor-core kernels, on the padded geometry: rows of the channels-last image are
// indexed in 32 bits, and padding must not outweigh what the tensor cores gain.
const char *tc_common(const tvdcn_problem *p, const GeoHost &g) {
    if (p->engine == TVDCN_ENGINE_SIMT) return "SIMT engine requested";
    if (p->dtype == TVDCN_F64) return "f64 has no tensor-core kind";
    const int csg = g.Cs / g.groups;
    if (g.K > 512) return "more than 512 kernel taps (the tensor-core kernels tabulate tap coordinates)";
    if (g.gran_pad > MAX_CHANNEL_PADDING * g.gran) return "too few sampled channels share their groups";
    if (((long long)g.B * g.S + 1) * g.Cs >= (1LL << 31) || (long long)g.B * g.P >= (1LL << 31))
        return "sampled image has 2^31 elements or more (32-bit element offsets)";
    if ((long long)g.Cd * csg * g.K >= (1LL << 31)) return "weight has 2^31 elements or more";
    return nullptr;
}

// The shapes whose 16-bit columns and two-part f32 operands the tolerances of these data types were set for: no
// padding, f32 offsets.  Everything else used to run on the SIMT kernels and keeps their precision (wide modes).
bool unpadded(const tvdcn_problem *p, const GeoHost &g) {
    return g.gran_pad == g.gran && g.Cd == g.Cd_r && p->aux_dtype == TVDCN_F32;
}
int mode_of(int dtype, bool wide) {
    if (dtype == DT_F32) return wide ? TC_F32_WIDE : TC_SPLIT;
    if (dtype == DT_F16) return wide ? TC_F16_WIDE : TC_F16;
    return wide ? TC_BF16_WIDE : TC_BF16;
}

// Calls that the tensor-core kernels take but the SIMT kernels finish sooner.  Figures: SIMT / tensor us, one granule.
bool simt_is_faster(const tvdcn_problem *p, const GeoHost &g, bool backward) {
    const int gran = g.gran, pad = g.gran_pad, cdg = g.Cd_r / g.groups;
    const long long n = (long long)g.B * g.P * (g.Cs_r / gran);     // positions of all granules
    const bool f32 = p->dtype == TVDCN_F32;
    if (backward)
        // 8 channels, f32.  1-d: 32000 positions 103 / 80, 120000 207 / 242, 400000 581 / 765, but 8 -> 64 channels 799 / 748; transposed
        // 2-d: 32400 267 / 263, 65536 448 / 526, 262144 1753 / 2184, 3-d: 102400 4561 / 5203, but 1-d 480000 956 / 840.  10 channels:
        // 720 / 773, 608 / 526.
        return f32 && pad > 7 * gran && n > 32768 && (p->transposed ? g.dim > 1 && cdg <= 64 : g.dim == 1 && cdg <= 32);
    if (!p->transposed)
        // One tap, 102400 positions: f32 16 channels 32 / 39, 24 channels 49 / 41; bf16 31 / 33, 47 / 35; 8 -> 64 channels 35 / 39, 8 -> 128
        // 60 / 59.  f32, 1-d, five taps: 8 channels 23 / 31 at 32000 positions, 785 / 867 at 1.6 million, 10 channels 29 / 31 and
        // 971 / 869, 8 -> 64 channels at 400000 238 / 222.
        return (g.K == 1 && pad >= 4 * gran && cdg <= 64) || (f32 && g.dim == 1 && pad > 7 * gran && cdg <= 32);
    // The transposed forward has the widest accumulator to zero, scatter into and turn back.  2-d, 4 x 4 taps, 8 channels: f32
    // 1000 positions 20 / 20, 5000 29 / 33, 65536 173 / 201, 262144 632 / 930; bf16 5000 31 / 31, 65536 179 / 191, 262144 644 / 921;
    // 10 channels, bf16: 65536 224 / 190, 131044 427 / 383, 262144 829 / 921; 11 channels: 939 / 919.
    if (pad > 6 * gran && cdg <= 64 && n > (f32 ? 4096 : 65536)) return true;
    // f32, 1-d, up to one wave of SIMT blocks of one or two reduction steps (four taps, 330 positions, 8 -> 16 channels 16.4 / 18.5,
    // 16 -> 16 18.4 / 18.4; 8 -> 16, 9400 positions 18.4 / 20.5): they are through before the tensor path's three kernels
    // have started up.  16-bit data, whose SIMT sums are converted by a kernel of their own, 18.5 / 16.4; 2-d, 16 taps, 22.5 / 20.5.
    const long long blocks = ((long long)g.B * g.P + 63) / 64 * g.groups * (((long long)g.Cs_r / g.groups * g.K + 63) / 64);
    return f32 && g.dim == 1 && cdg <= 16 && blocks <= 148 && pad != gran;
}

// f32 data on the tensor cores: one accumulator may take about 2400 MMAs before the round-toward-zero error of
// the f32 accumulation (~2e-8 of the result per MMA) eats half of the 1e-4 budget.  Longer reductions stay on the
// SIMT kernel.
bool chain_ok(int mode, const GeoHost &g, int bn) {
    if (!mode_f32(mode)) return true;
    const int nacc = std::min(4, 512 / std::max(bn, 1));
    const long long chain = (long long)g.K * (g.Cs / g.groups / 64) * 12 / nacc;
    return chain <= 2400;
}

void take_parts(size_t (&at)[3], Bump &b, int parts, size_t elems) {
    for (int q = 0; q < parts; ++q) at[q] = b.take(elems * 2);
}
size_t packed_elems(const GeoHost &g) { return (size_t)g.Cd * (g.Cs / g.groups) * g.K; }

// 16-bit offset / mask / bias reach the tensor-core kernels as f32
void take_aux(Plan &pl, Bump &b, const tvdcn_problem *p, const GeoHost &g, bool bias) {
    if (!is16(p->aux_dtype)) return;
    if (g.og > 0) pl.off32 = b.take((size_t)g.B * g.og * g.K * g.dim * g.P * sizeof(float));
    if (g.mg > 0) pl.mask32 = b.take((size_t)g.B * g.mg * g.K * g.P * sizeof(float));
    if (bias) pl.bias32 = b.take((size_t)p->out_channels * sizeof(float));
}

// The staged sampled image comes first in both plans, and the maxima of its blocks (maxima: a kernel of the call has the
// wide f16 mode) next: a backward call that is told to reuse the forward call's staging (TVDCN_FLAG_REUSE_STAGED_INPUT)
// finds them at the same offsets of the same workspace.
void take_image(Plan &pl, Bump &b, const tvdcn_problem *p, const GeoHost &g, bool maxima) {
    pl.img_cl = b.take(((size_t)g.B * g.S + 1) * g.Cs * (p->dtype == TVDCN_F32 ? 4 : 2));   // + one row of zeros
    if (!maxima) return;
    pl.n_img_max = (int)Stager::image_blocks(g);
    pl.img_max = b.take((size_t)pl.n_img_max * sizeof(unsigned));
    if (g.mg == 0) return;
    pl.n_mask_max = (int)Stager::widen_blocks((int64_t)g.B * g.mg * g.K * g.P);
    pl.mask_max = b.take((size_t)pl.n_mask_max * sizeof(unsigned));
}

// buffers of the sample -> GEMM kernel besides the staged image (no partial sums: no tile is shared)
void take_sample_buffers(Plan &pl, Bump &b, const GeoHost &g, int bn, bool share_tiles) {
    take_parts(pl.w_pack, b, mode_mat_parts(pl.mode), packed_elems(g));
    if (!share_tiles) return;
    size_t partial = 0;
    fwd_tc_workspace(g, pl.mode, bn, &partial, &pl.sg_counters);
    if (partial > 0) {
        pl.sg_partial = b.take(partial);
        pl.sg_arrived = b.take(pl.sg_counters * sizeof(unsigned));
    }
}

// buffers of the GEMM -> scatter kernel
void take_scatter_buffers(Plan &pl, Bump &b, const GeoHost &g, bool scatter) {
    take_parts(pl.w_pack_kd, b, mode_mat_parts(pl.mode), packed_elems(g));
    if (scatter) pl.img_grad_cl = b.take((size_t)g.B * g.S * g.Cs * sizeof(float));
}
}  // namespace

GeoHost tc_geometry(const GeoHost &g) {
    GeoHost t = g;
    int gran = gcd(g.Cs, g.Cs / g.groups);
    if (g.og > 0) gran = gcd(gran, g.Cs / g.og);
    if (g.mg > 0) gran = gcd(gran, g.Cs / g.mg);
    t.gran = gran;
    t.gran_pad = round_up(gran, 64);
    t.Cs_r = g.Cs;
    t.Cd_r = g.Cd;
    const long long cs = (long long)g.Cs / gran * t.gran_pad, cd = (long long)g.groups * round_up(g.Cd / g.groups, 64);
    t.Cs = (int)std::min<long long>(cs, 0x7fffffff);
    t.Cd = (int)std::min<long long>(cd, 0x7fffffff);
    return t;
}

Plan plan_forward(const tvdcn_problem *p, bool share_tiles) {
    Plan pl;
    const GeoHost g = tc_geometry(make_geo_host(p));
    Bump b;
    const char *why = tc_common(p, g);
    if (why == nullptr && p->engine == TVDCN_ENGINE_AUTO && simt_is_faster(p, g, false)) why = "the SIMT kernels are faster";
    pl.wide = !unpadded(p, g);
    pl.mode = mode_of(p->dtype, pl.wide);
    int bn = 0, st = 0, gbufs = 0;
    if (why == nullptr && !p->transposed) {
        if (fwd_tc_config(g, pl.mode, &bn, &st) && chain_ok(pl.mode, g, bn)) {
            pl.tensor = pl.tc_sg = true;
            take_image(pl, b, p, g, pl.mode == TC_F16_WIDE);
            take_sample_buffers(pl, b, g, bn, share_tiles);
            take_aux(pl, b, p, g, true);
        } else {
            why = "no tile configuration fits (or too many work units, or too long an f32 accumulation chain)";
        }
    } else if (why == nullptr) {
        if (dgrad_tc_config(g, pl.mode, &bn, &gbufs, &st)) {
            pl.tensor = pl.tc_gs = true;
            take_scatter_buffers(pl, b, g, true);
            take_aux(pl, b, p, g, true);
        } else {
            why = "no tile configuration fits (or too many work units)";
        }
    }
    if (why != nullptr) {
        pl.why_not = why;
        if (p->transposed && is16(p->dtype)) pl.img_acc = b.take((size_t)g.B * g.Cs_r * g.S * sizeof(float));
    }
    pl.total = b.off;
    return pl;
}

Plan plan_backward(const tvdcn_problem *p, bool want_input, bool want_weight, bool want_offset, bool want_mask) {
    Plan pl;
    const GeoHost g = tc_geometry(make_geo_host(p));
    Bump b;
    const char *why = tc_common(p, g);
    if (why == nullptr && p->engine == TVDCN_ENGINE_AUTO && simt_is_faster(p, g, true)) why = "the SIMT kernels are faster";
    pl.wide = !unpadded(p, g);
    pl.mode = mode_of(p->dtype, pl.wide);
    pl.mode_sw = mode_of(p->dtype, pl.wide || g.P % 8 != 0);
    want_offset = want_offset && g.og > 0;
    want_mask = want_mask && g.mg > 0;
    if (why == nullptr) {
        int bn = 0, sg_bn = 0, st = 0, ns = 0, mt = 0, gbufs = 0;
        // which primitives run on the tensor cores
        // transposed backward: grad_input is a sample -> GEMM over grad_output
        pl.tc_sg = p->transposed && want_input && fwd_tc_config(g, pl.mode, &sg_bn, &st) &&
                   chain_ok(pl.mode, g, sg_bn);
        pl.tc_sw = want_weight && wgrad_tc_config(g, pl.mode_sw, &ns, &mt, &st);
        // conv: scatter into grad_input + coordinate gradients; transposed: coordinate gradients only
        const bool scatter = !p->transposed && want_input;
        pl.tc_gs = (scatter || want_offset || want_mask) &&
                   dgrad_tc_config(g, pl.mode, &bn, &gbufs, &st);
        pl.tensor = pl.tc_sg || pl.tc_sw || pl.tc_gs;
        if (pl.tensor) {
            take_image(pl, b, p, g, (pl.tc_sg && pl.mode == TC_F16_WIDE) || (pl.tc_sw && pl.mode_sw == TC_F16_WIDE));
            take_aux(pl, b, p, g, false);
        }
        if (pl.tc_sg) take_sample_buffers(pl, b, g, sg_bn, true);
        if (pl.tc_sw) {
            // f32 data is split into 16-bit parts; 16-bit rows are copied only where TMA cannot read them
            pl.dense_pitch = round_up(g.P, 8);
            const int parts = p->dtype == TVDCN_F32 ? mode_mat_parts(pl.mode_sw) : (g.P % 8 != 0 ? 1 : 0);
            take_parts(pl.dense, b, parts, (size_t)g.B * g.Cd_r * pl.dense_pitch);
        }
        if (pl.tc_gs) take_scatter_buffers(pl, b, g, scatter);
        if (!pl.tensor) pl.why_not = "no tensor-core kernel covers the requested gradients for this shape";
    } else {
        pl.why_not = why;
    }
    if (is16(p->dtype)) {
        if (!p->transposed && want_input && !pl.tc_gs) pl.img_acc = b.take((size_t)g.B * g.Cs_r * g.S * sizeof(float));
    }
    // 16-bit data accumulates the weight gradient in f32; the tensor-core kernel accumulates (any data type) into
    // a staged layout that a small kernel turns into the caller's afterwards
    if (want_weight && (is16(p->dtype) || pl.tc_sw))
        pl.gw_acc = b.take((size_t)g.Cd_r * ((pl.tc_sw ? g.Cs : g.Cs_r) / g.groups) * g.K * sizeof(float));
    if (is16(p->aux_dtype)) {
        if (want_offset) pl.goff_acc = b.take((size_t)g.B * g.og * g.K * g.dim * g.P * sizeof(float));
        if (want_mask) pl.gmask_acc = b.take((size_t)g.B * g.mg * g.K * g.P * sizeof(float));
    }
    // bias gradient: the sum of grad_output (the dense tensor of the conv, the sampled image of the transposed conv)
    if (pl.tensor) {
        const int c = p->transposed ? g.Cs_r : g.Cd_r, n = p->transposed ? g.S : g.P;
        pl.sum_partial = b.take((size_t)dense_sum_scratch_floats(g.B, c, n) * sizeof(float));
        pl.sum_done = b.take((size_t)c * sizeof(unsigned));
    }
    pl.total = b.off;
    return pl;
}

}  // namespace tvdcn_b200
