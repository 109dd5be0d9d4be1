// Mamba-1 fused selective-scan forward for sm_100a.
// Host side of the fused forward: argument validation, TMA descriptors, variant
// selection, the time-segment plan and launch.  The kernels live in
// m1_fwd_kernel.cuh (all sizes) and m1_fwd16_kernel.cuh (warp roles, d_state 9 .. 16).
#include <algorithm>

#include "m1_fwd16_kernel.cuh"

namespace mb200 {

constexpr int kMaxSegments = 64;

// Time segments of sscan_fwd_kernel when it was lent a workspace (see launch_fwd): the count with the least estimated
// time, which it returns in *us.  In one piece a step takes 0.1155 us with one CTA per SM and 0.137 with two; both passes of a cut take
// kCut[2 x] with x CTAs per SM on average (d_state 16; f32 takes 1.03 times as long), a piece
// costs its steps and 16 more for its pipeline to fill, and the call 8 us with two more launches.  Beyond 1.15 CTAs
// per SM one piece is as fast, and under 192 steps (1 x 128 x 2560 whole 17.6, in four 18.9).  Fitted to 300
// measured shapes of 64 to 4096 steps: half of the estimates are within 5 %, and the counts chosen take 0.8 % longer
// than the best that was measured on average, 9 % at most.  Whole and as cut here, bf16 and f32 in us: 1 x 1021 x
// 1536 118 and 31, 129 and 32; 2 x 192 x 1536 25 and 20, 27 and 19; 4 x 512 x 1536 61 and 51, 66 and 53.
// From 1536 steps on the pieces are long whatever their number, and their number goes by what was measured: eight
// from 0.7 CTAs per SM on (0.85 x 2048 steps 207 us, 16: 209; 1.1: 253, 261), else 16 (0.65: 168, eight 171; 0.32 x
// 4096: 174, eight 183), or as many as fill the chip (0.03 x 2048: 24 in 64, 35 in 16).
constexpr int kFwdMaxPerSm = 9, kFwdMaxCtas = 170;
constexpr int kFwdMaxPieces = 12 * 148;  // of all CTAs together, by either rule
static long long fwd_ctas(int B, int D, int N) {  // of four consumer warps, one a scheduler
    int lpc = 1;
    while (8 * lpc < N) lpc *= 2;
    const int cw = lpc >= 16 ? 8 : 4, dt = cw * (32 / lpc);
    return static_cast<long long>(B) * ((D + dt - 1) / dt) * (cw / 4);
}
static size_t fwd_ws_bytes(int B, int D, int N, int segs, size_t* o_sum, size_t* o_h0, size_t* o_c0) {
    auto al = [](size_t v) { return (v + 255) & ~size_t(255); };
    size_t off = al(sizeof(float) * static_cast<size_t>(B) * segs * D * N);
    *o_sum = off;
    off += al(sizeof(float) * static_cast<size_t>(B) * segs * D);
    *o_h0 = off;
    off += al(sizeof(float) * static_cast<size_t>(B) * D * N);
    *o_c0 = off;
    off += al(sizeof(float) * static_cast<size_t>(B) * D * kKMax);
    return off;
}
static bool fwd_ws_holds(long long bytes, int B, int D, int N, int segs) {
    size_t o1, o2, o3;
    return bytes > 0 && fwd_ws_bytes(B, D, N, segs, &o1, &o2, &o3) <= static_cast<size_t>(bytes);
}
// `lent`: bytes of the workspace.  Where they do not hold the count that was wanted, it is one that they do hold, and
// *us what that takes (1 x 1021 x 1536 with 4 KB is walked whole, and not in the 31 us of sixteen segments); whole: 0.
static int fwd_segments(int B, int T, int D, int N, long long lent, double* us) {
    static const double kCut[2 * kFwdMaxPerSm + 2] = {0.175, 0.180, 0.191, 0.221, 0.239, 0.275, 0.312, 0.395, 0.429, 0.460,
                                                      0.508, 0.536, 0.568, 0.619, 0.669, 0.712, 0.753, 0.806, 0.860, 0.860};
    const long long ctas = fwd_ctas(B, D, N);
    // whole: three CTAs share an SM, 0.165 us a step together
    const long long rounds = ctas / (3 * 148), rest = ctas % (3 * 148);
    const double whole = rounds * (3.2 + 0.165 * T) + (rest ? 3.2 + T * (rest <= 148 ? 0.1155 : rest <= 296 ? 0.137 : 0.165) : 0.0);
    *us = 0.0;
    if (lent <= 0 || ctas > kFwdMaxCtas || T < 192) return 1;
    const int blocks = (T + 31) / 32;
    auto cut = [&](int s) {
        const int per = (blocks + s - 1) / s;
        const double x = 2.0 * ctas * s / 148, f = x - static_cast<int>(x);
        const double* at = kCut + std::min(static_cast<int>(x), 2 * kFwdMaxPerSm);
        return 8 + (32 * per + 16) * (x < 2 * kFwdMaxPerSm ? at[0] + f * (at[1] - at[0]) : at[0] * x / (2 * kFwdMaxPerSm));
    };
    int best = 1;
    double least = whole;
    if (T >= 1536) {
        const double w = ctas / 148.0;
        best = w >= 0.7 ? 8 : std::min({std::max(16, static_cast<int>(2.6 / w) + 1), blocks, kMaxSegments});
    } else {
        for (int s = 2; s <= kMaxSegments && s <= blocks && ctas * s <= kFwdMaxPerSm * 148; ++s)
            if (cut(s) < least) {
                least = cut(s);
                best = s;
            }
    }
    while (best > 1 && !fwd_ws_holds(lent, B, D, N, best)) best /= 2;
    if (best > 1) *us = cut(best);
    return best;
}
// What sscan_fwd_kernel (d_state 9 .. 16) takes in one piece, in us: kWhole[f32][plain][0] and a step by CTAs per SM,
// three, without a gate four of f32; the CTAs past full waves run beside the end of the last one.  plain: rows of B and C
// that no tensor map describes, brought by one warp's loads.  Means of rates in progression and general ones, which lie
// 12 % below and above them in 16-bit storage, 6 % in f32.
static double fwd_whole_us(bool f32, bool gated, bool plain, int T, long long ctas) {
    static const double kWhole[2][2][5] = {{{4.4, 0.102, 0.123, 0.161}, {9.0, 0.121, 0.190, 0.235}},
                                           {{4.2, 0.118, 0.1395, 0.175, 0.210}, {6.0, 0.180, 0.262, 0.275, 0.360}}};
    static const double kTail[4] = {0.83, 0.93, 0.96, 1.0};
    const double* at = kWhole[f32][plain];
    double base = at[0];
    if (!f32 && T <= 64) base = T <= 32 ? (plain ? 5.5 : 4.2) : (plain ? 11.0 : 4.9);  // one chunk, two
    const int per = f32 && !gated ? 4 : 3;
    const long long full = ctas / (per * 148), rest = ctas % (per * 148);
    const int k = static_cast<int>((rest + 147) / 148);
    return full * (base + at[per] * T) + (rest ? at[k] * T * (full ? kTail[k - 1] : 1.0) + (full ? 0.0 : base) : 0.0);
}

// The kernel by warp roles: how a call is laid out and what that takes, in us, by storage (16-bit, f32).  One CTA has an
// SM to itself (three at two consumer warps).  Whole: w0 + w1 a step and round of CTAs; cut, where all pieces run side by
// side: c0 + c1 a step of a piece, both passes, + cs a segment, whose states every CTA chains.  Steps are those of whole
// chunks, which the kernel walks whatever the length (34 steps of 16-bit storage take what 64 do).  Means of rates in
// progression and general ones, which lie 6 % below and above them (cut 8 %).  Fitted to 2400 shapes of 16 to 8192 steps
// (as CUDA graphs): nine in ten of the estimates are within 3 % of either kind (cut 5 %).
struct Fwd16Kind {
    int ns, workers, helpers, stages;
    double w0, w1[2], c0, c1[2], cs;
};
static const Fwd16Kind kFwd16Kinds[] = {{4, 2, 2, 3, 4.2, {0.0600, 0.0680}, 6.6, {0.1000, 0.1130}, 0.27},
                                        {4, 4, 4, 4, 3.8, {0.0680, 0.0800}, 6.1, {0.1140, 0.1337}, 0.27},
                                        {4, 5, 4, 4, 4.6, {0.0822, 0.0984}, 7.0, {0.1443, 0.1662}, 0.26},
                                        {4, 6, 4, 4, 4.7, {0.0850, 0.0999}, 7.1, {0.1474, 0.1690}, 0.26},
                                        {4, 8, 4, 4, 4.4, {0.1020, 0.1184}, 6.8, {0.1754, 0.1986}, 0.30},
                                        {8, 6, 4, 4, 5.8, {0.1491, 0.1640}, 9.9, {0.2700, 0.2900}, 0.50}};
// Two consumer warps, two or three CTAs an SM: the base and a step.
static const double kFwd16Shared[2][3] = {{4.8, 0.0845, 0.0972}, {4.2, 0.0930, 0.1080}};
struct Fwd16Plan {
    const Fwd16Kind* kind = nullptr;  // null: sscan_fwd_kernel
    int segs = 1;
};

struct FwdTable {
    FwdVariant v[3][kMaxFwdVariants];
    int n[3];
};

// Built once, under the thread-safe initialisation of a function-local static.
static const FwdTable& fwd_table() {
    static const FwdTable table = [] {
        FwdTable t;
        memset(&t, 0, sizeof(t));
        t.n[MAMBA_B200_F32] = fwd_variants_f32(t.v[MAMBA_B200_F32]);
        t.n[MAMBA_B200_F16] = fwd_variants_f16(t.v[MAMBA_B200_F16]);
        t.n[MAMBA_B200_BF16] = fwd_variants_bf16(t.v[MAMBA_B200_BF16]);
        return t;
    }();
    return table;
}

// The smallest one that holds N states.
static const FwdVariant* fwd_variant(int dtype, int N) {
    const FwdTable& tab = fwd_table();
    for (int i = 0; i < tab.n[dtype]; ++i)
        if (tab.v[dtype][i].ns * tab.v[dtype][i].lpc >= N) return &tab.v[dtype][i];
    return nullptr;
}

// Built once, like the other table.
struct Fwd16Tables {
    Fwd16Table t[3];
};
static const Fwd16Tables& fwd16_tables() {
    static const Fwd16Tables tables = [] {
        Fwd16Tables t;
        fwd16_f32(&t.t[MAMBA_B200_F32]);
        fwd16_f16(&t.t[MAMBA_B200_F16]);
        fwd16_bf16(&t.t[MAMBA_B200_BF16]);
        return t;
    }();
    return tables;
}

int m1_fwd_configure(Ctx* c) {
    for (int dt = 0; dt < 3; ++dt)
        for (int i = 0; i < 2; ++i)
            for (int f = 0; f < 6; ++f)
                MB200_CUDA_CHECK(c, cudaFuncSetAttribute(reinterpret_cast<const void*>(fwd16_tables().t[dt].fn[i][f]),
                                                         cudaFuncAttributeMaxDynamicSharedMemorySize, kF16MaxSmem));
    const FwdTable& t = fwd_table();
    for (int dt = 0; dt < 3; ++dt)
        for (int i = 0; i < t.n[dt]; ++i)
            for (int f = 0; f < 16; ++f)
                if (t.v[dt][i].fn[f] && t.v[dt][i].smem <= 227 * 1024)
                    MB200_CUDA_CHECK(c, cudaFuncSetAttribute(
                                            reinterpret_cast<const void*>(t.v[dt][i].fn[f]),
                                            cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            static_cast<int>(t.v[dt][i].smem)));
    return MAMBA_B200_OK;
}

// Segment hand-over: slot s of seg_states arrives holding the state segment s
// leaves when started from zero (segment 0: from the real entering state) and
// leaves holding the true state at the end of segment s, i.e. the one segment
// s + 1 starts from.  A segment's decay is exp(a * sum of its deltas): the carry
// costs one exp2 per state and segment.  Bound by the latency of its loads, so eight segments' are
// requested together (32 segments of 1 x 1536 x 16: 3.2 us, one by one 6.1).
__global__ void sscan_seg_carry_kernel(float* seg_states, const float* seg_sumdl, const float* a_neg,
                                       int B, int S, int D, int N) {
    const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (i >= static_cast<long long>(B) * D * N) return;
    const int n = static_cast<int>(i % N);
    const int d = static_cast<int>((i / N) % D);
    const int b = static_cast<int>(i / (static_cast<long long>(N) * D));
    const float a2 = a_neg[static_cast<long long>(d) * N + n] * kLog2e;
    float* st = seg_states + (static_cast<long long>(b) * S * D + d) * N + n;
    const float* sums = seg_sumdl + static_cast<long long>(b) * S * D + d;
    const long long DN = static_cast<long long>(D) * N;
    float run = st[0];
    for (int s0 = 1; s0 + 1 < S; s0 += 8) {
        float h[8], q[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int s = s0 + k + 1 < S ? s0 + k : s0;
            h[k] = st[s * DN];
            q[k] = sums[static_cast<long long>(s) * D];
        }
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (s0 + k + 1 < S) {
                run = fmaf(ex2(a2 * q[k]), run, h[k]);
                st[(s0 + k) * DN] = run;
            }
    }
}

// The layout with the least estimate, if that is at most 0.95 of `us`, what sscan_fwd_kernel is estimated to take.
// Against that kernel alone, 2400 shapes of 16 to 8192 steps with and without a workspace, both kinds of rates: 25 % less
// time on average, six calls in a thousand more than 2 % more, 11 % at most.  Rates in progression decide where the line
// lies: they help the other kernel more, so that at the border they are even and general ones gain a tenth.  8 x 2048 x
// 1536 with general rates 284 -> 196 us, 2 x 8192 x 5120 with progressions 757 -> 640, 16 x 2048 x 1536 363 -> 339, 1 x
// 1021 x 1536 32.0 -> 28.5, 4 x 512 x 256 19.7 -> 15.5.  Under 24 steps the shorter prologue of the other kernel wins (12 x
// 9 x 144 4.5 us, here 5.8), with 34 to 36 steps of 16-bit storage its shorter chunks of rows do (14 x 37 x 2416 15.3, here
// 19.8), in f32 without a gate its four CTAs an SM (10 x 544 x 3096 110, here 127), and past three rounds of CTAs its three
// (19 x 33 x 5360 32, here 59).
static Fwd16Plan fwd16_plan(const Fwd16Table& t, bool f32, int B, int T, int D, int N, double us, long long workspace_bytes) {
    Fwd16Plan best;
    if (T < 24) return best;
    us *= 0.95;
    for (const Fwd16Kind& k : kFwd16Kinds) {
        const int steps = t.steps[k.ns == 8], chunks = (T + steps - 1) / steps, dt = 4 * k.ns * k.workers;
        const long long ctas = static_cast<long long>(B) * ((D + dt - 1) / dt);
        double c = ((ctas + 147) / 148) * (k.w0 + k.w1[f32] * chunks * steps);
        if (k.workers == 2 && ctas > 148) c = kFwd16Shared[f32][0] + kFwd16Shared[f32][ctas > 2 * 148 ? 2 : 1] * chunks * steps;
        // a tile that reaches past the channels stores element by element, which progressions leave no time for
        if (k.ns == 8 && !f32 && D % dt != 0) c *= 1.06;
        if (c < us && ctas <= 3 * 148) {
            us = c;
            best = {&k, 1};
        }
        if (T < 192) continue;
        for (int s = 2; ctas * s <= 148 && s <= 32; ++s) {
            const int per = (chunks + s - 1) / s, segs = (chunks + per - 1) / per;
            if (segs != s || per * steps < 32 || !fwd_ws_holds(workspace_bytes, B, D, N, s)) continue;
            c = k.c0 + k.c1[f32] * per * steps + k.cs * s;
            if (c < us) {
                us = c;
                best = {&k, s};
            }
        }
    }
    return best;
}

// How a call is laid out that both kernels can take (no conv, d_state 9 .. 16, x, delta and z by TMA); segs: of the
// general kernel, with `us` from fwd_segments, which is for 16-bit storage and B and C by TMA.
static Fwd16Plan fwd16_choose(int dtype, int B, int T, int D, int N, bool gated, bool plain, int segs, double us, long long lent) {
    const bool f32 = dtype == MAMBA_B200_F32;
    us += 0.17 * std::max(0, segs - 18);  // the kernel between the passes
    us = segs > 1 ? us * (plain ? 1.3 : 1.0) * (f32 ? 1.03 : 1.0) : fwd_whole_us(f32, gated, plain, T, fwd_ctas(B, D, N));
    return fwd16_plan(fwd16_tables().t[dtype], f32, B, T, D, N, us, lent);
}

static bool overlaps(const void* a, size_t na, const void* b, size_t nb) {
    const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
    return a && b && x < y + nb && y < x + na;
}

// The caller's workspace, divided for `segs` time segments.
struct SegmentBuffers {
    float *states, *sums, *ssm, *conv;
};
static SegmentBuffers segment_buffers(const mamba_b200_sscan_fwd_args& a, int segs) {
    size_t o_sum, o_h0, o_c0;
    fwd_ws_bytes(a.B, a.D, a.N, segs, &o_sum, &o_h0, &o_c0);
    unsigned char* ws = static_cast<unsigned char*>(a.workspace);
    return {reinterpret_cast<float*>(ws), reinterpret_cast<float*>(ws + o_sum), reinterpret_cast<float*>(ws + o_h0),
            reinterpret_cast<float*>(ws + o_c0)};
}
static void launch_seg_carry(cudaStream_t stream, const mamba_b200_sscan_fwd_args& a, const SegmentBuffers& w, int segs) {
    const long long n = static_cast<long long>(a.B) * a.D * a.N;
    sscan_seg_carry_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, stream>>>(w.states, w.sums, a.a_neg, a.B, segs, a.D,
                                                                                      a.N);
}

// The call by warp roles.  q.f holds what both kernels need, and the tensor maps of this one's tiles after fwd16_maps.
static bool fwd16_maps(Ctx* c, const mamba_b200_sscan_fwd_args& a, const Fwd16Table& t, const Fwd16Plan& plan, Fwd16Params* q) {
    const Fwd16Kind& k = *plan.kind;
    const int steps = t.steps[k.ns == 8], dt = 4 * k.ns * k.workers;
    auto tile = [&](CUtensorMap* map, const void* base, long long ld, int cols, int box) {
        return make_tmap_3d(c, map, a.dtype, base, ld, cols, a.T, a.B, box, steps);
    };
    q->dt = dt;
    if (!tile(&q->f.tm_x, a.x, a.ld_x, a.D, dt) || !tile(&q->f.tm_dl, a.delta, a.ld_delta, a.D, dt) ||
        (a.z_mode && !tile(&q->f.tm_z, a.z, a.ld_z, a.D, dt)))
        return false;
    if (tile(&q->f.tm_b, a.Bm, a.ld_bc, a.N, a.N)) q->f.tma_mask |= kTmaB;
    if (tile(&q->f.tm_c, a.Cm, a.ld_bc, a.N, a.N)) q->f.tma_mask |= kTmaC;
    return true;
}
static int launch_fwd16(Ctx* c, cudaStream_t stream, const mamba_b200_sscan_fwd_args& a, const Fwd16Table& t, const Fwd16Plan& plan,
                        Fwd16Params& q) {
    const Fwd16Kind& k = *plan.kind;
    const int i = k.ns == 8, steps = t.steps[i], dt = q.dt;
    q.stages = k.stages;
    while (t.smem[i](dt, q.stages) > kF16MaxSmem) --q.stages;
    // a helper goes to the scheduler (warp % 4) that has the least to do
    int load[4] = {}, warps = k.workers;
    for (int w = 0; w < k.workers; ++w) {
        q.consumers |= 1u << w;
        load[w % 4] += 2;
    }
    for (int h = 0; h < k.helpers; ++h) {
        int best = -1;
        for (int w = k.workers; w < k.workers + 8; ++w)
            if (!(q.helpers >> w & 1) && (best < 0 || load[w % 4] < load[best % 4])) best = w;
        q.helpers |= 1u << best;
        load[best % 4] += 1;
        warps = std::max(warps, best + 1);
    }
    const int threads = 32 * (warps + 1);  // and the producer
    q.vec_y = reinterpret_cast<uintptr_t>(a.y) % (2 * dtype_size(a.dtype)) == 0 && a.ld_y % 2 == 0;
    auto aligned = [](const void* ptr) { return reinterpret_cast<uintptr_t>(ptr) % 16 == 0; };
    q.vec_state = a.N == 16 && aligned(a.ssm_state) && aligned(a.chunk_states) && q.f.cs_ld_b % 4 == 0 && q.f.cs_ld_k % 4 == 0;

    const int flags = (a.delta_softplus ? 1 : 0) | (a.z_mode ? 2 : 0);
    const size_t smem = t.smem[i](dt, q.stages);
    dim3 grid((a.D + dt - 1) / dt, a.B, plan.segs);
    if (plan.segs > 1) {
        const int chunks = (a.T + steps - 1) / steps;
        q.f.seg_chunks = (chunks + plan.segs - 1) / plan.segs;
        const SegmentBuffers w = segment_buffers(a, plan.segs);
        q.f.seg_states = w.states;
        q.f.seg_sumdl = w.sums;
        Fwd16Params q1 = q;
        q1.f.ssm_copy = w.ssm;
        t.fn[i][4 + (flags & 1)]<<<grid, threads, smem, stream>>>(q1);
        MB200_CUDA_CHECK(c, cudaGetLastError());
        q.f.ssm_in = w.ssm;  // the last segment writes the caller's state while others may still be starting
    }
    t.fn[i][flags]<<<grid, threads, smem, stream>>>(q);
    MB200_CUDA_CHECK(c, cudaGetLastError());
    return MAMBA_B200_OK;
}

static int launch_fwd(Ctx* c, cudaStream_t stream, const mamba_b200_sscan_fwd_args& a, long long cs_ld_b = 0,
                      long long cs_ld_k = 0) {
    if (!dtype_ok(a.dtype)) return fail(c, MAMBA_B200_ERR_ARG, "sscan_fwd: bad dtype %d", a.dtype);
    if (a.B < 0 || a.T < 0 || a.D <= 0 || a.N <= 0)
        return fail(c, MAMBA_B200_ERR_ARG, "sscan_fwd: bad dims B=%d T=%d D=%d N=%d", a.B, a.T, a.D, a.N);
    if (a.N > 256) return fail(c, MAMBA_B200_ERR_SHAPE, "sscan_fwd: d_state %d > 256", a.N);
    if (a.B == 0 || a.T == 0) return MAMBA_B200_OK;
    if (a.B > 65535) return fail(c, MAMBA_B200_ERR_SHAPE, "sscan_fwd: batch %d > 65535", a.B);
    if (!a.x || !a.delta || !a.Bm || !a.Cm || !a.a_neg || !a.Dp || !a.y)
        return fail(c, MAMBA_B200_ERR_ARG, "sscan_fwd: null required pointer");
    if (a.z_mode < 0 || a.z_mode > 2 || (a.z_mode && !a.z))
        return fail(c, MAMBA_B200_ERR_ARG, "sscan_fwd: z_mode %d with z=%p", a.z_mode, a.z);
    if (a.conv_w && (!a.conv_b || a.K < 1 || a.K > kKMax))
        return fail(c, MAMBA_B200_ERR_SHAPE, "sscan_fwd: d_conv %d outside 1..%d or null bias", a.K, kKMax);
    if (a.ld_x < a.D || a.ld_delta < a.D || a.ld_y < a.D || a.ld_bc < a.N ||
        (a.z_mode && a.ld_z < a.D) || (a.u_out && a.ld_u < a.D))
        return fail(c, MAMBA_B200_ERR_ARG, "sscan_fwd: a row stride is smaller than its row");
    const size_t es = dtype_size(a.dtype);
    auto misaligned = [&](const void* ptr) { return (reinterpret_cast<uintptr_t>(ptr) % es) != 0; };
    if (misaligned(a.x) || misaligned(a.delta) || misaligned(a.Bm) || misaligned(a.Cm) ||
        misaligned(a.y) || (a.z && misaligned(a.z)) || (a.u_out && misaligned(a.u_out)))
        return fail(c, MAMBA_B200_ERR_ARG, "sscan_fwd: pointer not aligned to its element size");
    // With the conv fused, a chunk re-reads the rows of x just before it: y (or u_out)
    // written over x would be read back as input.
    const size_t span_x = (static_cast<size_t>(a.B) * a.T - 1) * a.ld_x * es + a.D * es;
    if (a.conv_w && (overlaps(a.x, span_x, a.y, (static_cast<size_t>(a.B) * a.T - 1) * a.ld_y * es + a.D * es) ||
                     (a.u_out && overlaps(a.x, span_x, a.u_out,
                                          (static_cast<size_t>(a.B) * a.T - 1) * a.ld_u * es + a.D * es))))
        return fail(c, MAMBA_B200_ERR_ARG, "sscan_fwd: with the conv fused, y and u_out must not overlap x");

    const FwdVariant* v = fwd_variant(a.dtype, a.N);
    if (!v) return fail(c, MAMBA_B200_ERR_SHAPE, "sscan_fwd: no variant for d_state %d", a.N);
    if (a.chunk_states && (a.save_stride <= 0 || a.save_stride % 32 != 0 || a.save_stride > 64))
        return fail(c, MAMBA_B200_ERR_ARG, "sscan_fwd: save_stride %d must be 32 or 64", a.save_stride);

    FwdParams p;
    memset(&p, 0, sizeof(p));
    p.x = a.x; p.dl = a.delta; p.z = a.z_mode ? a.z : nullptr; p.bm = a.Bm; p.cm = a.Cm;
    p.y = a.y; p.u_out = a.conv_w ? a.u_out : nullptr;
    p.ld_x = a.ld_x; p.ld_dl = a.ld_delta; p.ld_z = a.ld_z; p.ld_bc = a.ld_bc; p.ld_y = a.ld_y;
    p.ld_u = a.ld_u;
    p.a_neg = a.a_neg; p.Dp = a.Dp; p.conv_w = a.conv_w; p.conv_b = a.conv_b;
    p.conv_state = a.conv_w ? a.conv_state : nullptr;
    p.ssm_state = a.ssm_state; p.chunk_states = a.chunk_states;
    p.conv_in = p.conv_state; p.ssm_in = p.ssm_state;
    p.B = a.B; p.T = a.T; p.D = a.D; p.N = a.N; p.K = a.conv_w ? a.K : 0;
    p.z_mode = a.z_mode;
    p.save_stride = a.chunk_states ? a.save_stride : 1;
    if (a.chunk_states) {  // default: dense [B, ceil(T / stride), D, N]
        p.cs_ld_k = cs_ld_k ? cs_ld_k : static_cast<long long>(a.D) * a.N;
        p.cs_ld_b = cs_ld_b ? cs_ld_b : p.cs_ld_k * ((a.T + a.save_stride - 1) / a.save_stride);
    }
    p.status = c->d_status;
    const long long lent = a.workspace ? a.workspace_bytes : 0;
    double us = 0.0;
    int segs = fwd_segments(a.B, a.T, a.D, a.N, lent, &us);
    const bool ws_aligned = reinterpret_cast<uintptr_t>(a.workspace) % 256 == 0;
    if (segs > 1 && !ws_aligned) return fail(c, MAMBA_B200_ERR_ARG, "sscan_fwd: workspace must be 256-byte aligned");
    // d_state 9 .. 16 without the conv, channels that TMA can bring: by warp roles where that is estimated to be faster
    auto fits = [&](const void* base, long long ld, int cols, int box) {
        return tmap_3d_fits(c, a.dtype, base, ld, cols, a.T, box, v->tc);
    };
    if (v->ns * v->lpc == 16 && !a.conv_w && fits(a.x, a.ld_x, a.D, v->dt) && fits(a.delta, a.ld_delta, a.D, v->dt) &&
        (!a.z_mode || fits(a.z, a.ld_z, a.D, v->dt))) {
        const Fwd16Table& t16 = fwd16_tables().t[a.dtype];
        const bool plain = !fits(a.Bm, a.ld_bc, a.N, a.N) || !fits(a.Cm, a.ld_bc, a.N, a.N);
        const Fwd16Plan plan = fwd16_choose(a.dtype, a.B, a.T, a.D, a.N, a.z_mode != 0, plain, segs, us, ws_aligned ? lent : 0);
        Fwd16Params q;
        if (plan.kind) {
            memset(&q, 0, sizeof(q));
            q.f = p;
            if (fwd16_maps(c, a, t16, plan, &q)) return launch_fwd16(c, stream, a, t16, plan, q);
        }
    }

    unsigned m = 0;
    const int xrows = a.conv_w ? v->tc + kHaloRows : v->tc;
    if (make_tmap_3d(c, &p.tm_x, a.dtype, a.x, a.ld_x, a.D, a.T, a.B, v->dt, xrows)) m |= kTmaX;
    if (make_tmap_3d(c, &p.tm_dl, a.dtype, a.delta, a.ld_delta, a.D, a.T, a.B, v->dt, v->tc)) m |= kTmaDl;
    if (a.z_mode && make_tmap_3d(c, &p.tm_z, a.dtype, a.z, a.ld_z, a.D, a.T, a.B, v->dt, v->tc)) m |= kTmaZ;
    if (make_tmap_3d(c, &p.tm_b, a.dtype, a.Bm, a.ld_bc, a.N, a.T, a.B, a.N, v->tc)) m |= kTmaB;
    if (make_tmap_3d(c, &p.tm_c, a.dtype, a.Cm, a.ld_bc, a.N, a.T, a.B, a.N, v->tc)) m |= kTmaC;
    p.tma_mask = m;

    const int flags = (a.delta_softplus ? 1 : 0) | (a.z_mode ? 2 : 0) | (a.conv_w ? 4 : 0);
    FwdKernelFn fn = v->fn[flags];
    FwdKernelFn fn_state = v->fn[8 | (flags & 5)];
    if (!fn || !fn_state || v->smem > 227 * 1024)
        return fail(c, MAMBA_B200_ERR_SHAPE, "sscan_fwd: no kernel for dtype %d flags %d d_state %d",
                    a.dtype, flags, a.N);

    // Time segments.  When batch x channel tiles leave warp schedulers idle
    // (small-batch prefill) and the caller lent a workspace, the sequence is cut
    // into S segments that run side by side: a first launch walks segments
    // 0 .. S-2 for their leaving states only (segment s > 0 from a zero state,
    // keeping the sum of its deltas), a small kernel chains them into the true
    // entering states, and the second launch runs every segment in full.
    const int tiles = (a.D + v->dt - 1) / v->dt;
    const int nchunks = (a.T + v->tc - 1) / v->tc;
    dim3 grid(tiles, a.B, 1);
    if (segs > 1) {
        p.seg_chunks = (nchunks + segs - 1) / segs;
        segs = (nchunks + p.seg_chunks - 1) / p.seg_chunks;
    }
    if (segs > 1) {
        grid.z = segs;
        FwdParams p1 = p;
        const SegmentBuffers w = segment_buffers(a, segs);
        p.seg_states = p1.seg_states = w.states;
        p.seg_sumdl = p1.seg_sumdl = w.sums;
        p1.ssm_copy = w.ssm;  // the state-only pass also keeps the entering states for the second pass
        p1.conv_copy = p.K ? w.conv : nullptr;
        fn_state<<<grid, v->threads, v->smem, stream>>>(p1);
        MB200_CUDA_CHECK(c, cudaGetLastError());
        launch_seg_carry(stream, a, w, segs);
        MB200_CUDA_CHECK(c, cudaGetLastError());
        // segment 0 of the second pass reads the copies: the last segment overwrites the
        // caller's state arrays while other segments may still be starting
        p.ssm_in = p1.ssm_copy;
        p.conv_in = p1.conv_copy;
    }
    fn<<<grid, v->threads, v->smem, stream>>>(p);
    MB200_CUDA_CHECK(c, cudaGetLastError());
    return MAMBA_B200_OK;
}

}  // namespace mb200

using namespace mb200;

extern "C" MAMBA_B200_API long long mamba_b200_sscan_fwd_workspace_bytes(int B, int T, int D, int N) {
    if (B <= 0 || T <= 0 || D <= 0 || N <= 0 || N > 256) return 0;
    // room for every batch up to B and length up to T, whose counts of segments may be larger
    size_t o1, o2, o3, most = 0;
    for (int b = 1; b <= B; ++b) {
        const long long ctas = fwd_ctas(b, D, N);
        if (ctas > kFwdMaxCtas) b = B;
        const long long segs = ctas > kFwdMaxCtas ? 1 : std::min<long long>({kFwdMaxPieces / ctas, (T + 31) / 32, kMaxSegments});
        most = std::max(most, fwd_ws_bytes(b, D, N, static_cast<int>(segs), &o1, &o2, &o3));
    }
    return static_cast<long long>(most);
}

extern "C" MAMBA_B200_API int mamba_b200_sscan_fwd_layout(int dtype, int B, int T, int D, int N, int z_mode, long long workspace_bytes,
                                                            int* out) {
    if (!out || !dtype_ok(dtype) || B <= 0 || T <= 0 || D <= 0 || N <= 0 || N > 256) return MAMBA_B200_ERR_ARG;
    const FwdVariant* v = fwd_variant(dtype, N);
    double us = 0.0;
    int segs = fwd_segments(B, T, D, N, workspace_bytes, &us);
    Fwd16Plan plan;
    if (v->ns * v->lpc == 16)
        plan = fwd16_choose(dtype, B, T, D, N, z_mode != 0, N * dtype_size(dtype) % 16 != 0, segs, us, workspace_bytes);
    if (!plan.kind) {
        const int chunks = (T + v->tc - 1) / v->tc, per = (chunks + segs - 1) / segs;
        segs = (chunks + per - 1) / per;
    }
    out[0] = plan.kind ? plan.kind->ns : 0;
    out[1] = plan.kind ? plan.kind->workers : 0;
    out[2] = plan.kind ? plan.segs : segs;
    return MAMBA_B200_OK;
}

extern "C" MAMBA_B200_API int mamba_b200_sscan_fwd(void* handle, void* stream, const mamba_b200_sscan_fwd_args* args) {
    Ctx* c = static_cast<Ctx*>(handle);
    if (!c) return MAMBA_B200_ERR_ARG;
    if (!args) return fail(c, MAMBA_B200_ERR_ARG, "sscan_fwd: null args");
    return launch_fwd(c, static_cast<cudaStream_t>(stream), *args);
}

extern "C" MAMBA_B200_API int mamba_b200_ssm_scan_fwd_nosave(void* handle, void* stream, int dtype, float* h,
                                              void* y_out, const void* delta, const void* u,
                                              const void* B, const void* C, const float* a_neg,
                                              const float* D, int batch, int T, int d_inner,
                                              int d_state) {
    Ctx* c = static_cast<Ctx*>(handle);
    if (!c) return MAMBA_B200_ERR_ARG;
    mamba_b200_sscan_fwd_args a;
    memset(&a, 0, sizeof(a));
    a.dtype = dtype; a.B = batch; a.T = T; a.D = d_inner; a.N = d_state;
    a.x = u; a.ld_x = d_inner; a.delta = delta; a.ld_delta = d_inner; a.delta_softplus = 0;
    a.Bm = B; a.Cm = C; a.ld_bc = d_state; a.z_mode = 0;
    a.a_neg = a_neg; a.Dp = D; a.ssm_state = h; a.y = y_out; a.ld_y = d_inner;
    return launch_fwd(c, static_cast<cudaStream_t>(stream), a);
}

extern "C" MAMBA_B200_API int mamba_b200_ssm_scan_fwd_save(void* handle, void* stream, int dtype, float* h,
                                                           void* y_out, float* h_saved, const void* delta,
                                                           const void* u, const void* B, const void* C,
                                                           const float* a_neg, const float* D, int batch, int T,
                                                           int d_inner, int d_state) {
    Ctx* c = static_cast<Ctx*>(handle);
    if (!c) return MAMBA_B200_ERR_ARG;
    if (!h_saved) return fail(c, MAMBA_B200_ERR_ARG, "ssm_scan_fwd_save: null h_saved");
    mamba_b200_sscan_fwd_args a;
    memset(&a, 0, sizeof(a));
    a.dtype = dtype; a.B = batch; a.T = T; a.D = d_inner; a.N = d_state;
    a.x = u; a.ld_x = d_inner; a.delta = delta; a.ld_delta = d_inner; a.delta_softplus = 0;
    a.Bm = B; a.Cm = C; a.ld_bc = d_state; a.z_mode = 0;
    a.a_neg = a_neg; a.Dp = D; a.ssm_state = h; a.y = y_out; a.ld_y = d_inner;
    // rows 0, 32, 64, ... of h_saved [batch, T+1, d_inner, d_state]
    a.chunk_states = h_saved; a.save_stride = 32;
    const long long row = static_cast<long long>(d_inner) * d_state;
    return launch_fwd(c, static_cast<cudaStream_t>(stream), a, row * (static_cast<long long>(T) + 1), 32 * row);
}
