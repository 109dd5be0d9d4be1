// Mamba-1 selective-scan forward, d_state 9 .. 16, no fused conv: the kernel by warp roles.
//
// A CTA owns (sample b, a tile of DT channels, a time segment) and walks its steps in chunks of TC.  A chunk goes
// through a ring of stages in shared memory; the roles meet on mbarriers only:
//
//   producer  (1 thread): TMA brings the x / delta / z / B / C tiles (full[s]);
//   helpers             : before the recurrence (delta, delta * u) of every row in f32, a 16-byte word for two channels,
//                         and zero-padded f32 rows of B and C (ready[s]); after it y = (y + D u) * gate, whole sectors
//                         to global memory (empty[s]);
//   consumers           : LPC lanes own two neighbouring channels, NS states of each, in registers for the whole
//                         sequence: h = exp(delta a) h + (delta u) B, y = <h, C>, nothing else; y takes the place of
//                         the delta it was made of (done[s]).
//
// Rows past the end have delta = delta * u = 0 there, which leaves the state as it is: the consumers know no ragged
// chunk.  The words of a row hold channels 0, 4, 8 ... (and their neighbours) first, then 2, 6 ...: a helper lane has
// four neighbouring channels (64 bits of 16-bit storage) and reaches both words without bank conflicts.
//
// What bounds it, at 8 x 2048 x 1536 in bf16 with general rates (284 us by sscan_fwd_kernel, 196 here; with rates in
// arithmetic progression 231 and 172): with 5.2 consumer warps an SM the latency of a step, 90 of 190 cycles of which
// are issue slots; then the MUFU pipe (98 cycles a step) and shared-memory bandwidth.  A 128-bit shared load takes four
// cycles of the SM's return path whether or not its lanes ask for the same words, so B and C cost a cycle per channel
// and step where a lane has one channel (204 us), half where it has two.  Four states a lane: eight (16 x 2048 x 1536
// 342 us) need fewer instructions and loads, but leave one warp a scheduler below 256 channels an SM (8 x 2048 x 1536
// 260 us); they take all of the 128 registers that 512 threads leave and spill 8 bytes.  Elementwise work in the consumers, as sscan_fwd_kernel has it, would put its latency into the chain of
// every step and its registers into every lane.  Tried and not kept: packing over the two channels (B and C twice in
// shared memory, 30 % slower); a fourth of the exponentials by a polynomial on the FMA pipe (196 -> 206 us);
// chunks unrolled in full (instruction fetch: 141 -> 190 us at four consumer warps).
#pragma once
#include "m1_fwd_kernel.cuh"

namespace mb200 {

constexpr int kF16Threads = 512;  // most threads of a CTA
constexpr int kF16MaxStages = 4;
constexpr int kF16BarBytes = 128;  // four mbarriers a stage
constexpr size_t kF16MaxSmem = 227 * 1024;

struct Fwd16Params {
    FwdParams f;
    int dt, stages;               // channels of a CTA, stages of the ring
    unsigned consumers, helpers;  // which warps are (bit = warp); the last one of the CTA is the producer's
    int vec_state;                // rows of states are 16 aligned floats
    int vec_y;                    // rows of y start on a multiple of two elements
};

// A stage's layout for dt channels, dt a multiple of 8.
template <typename Tact, int TC>
struct Fwd16Stage {
    static __host__ __device__ constexpr size_t al(size_t v) { return (v + 127) & ~size_t(127); }
    static __host__ __device__ constexpr size_t act(int dt) { return al(sizeof(Tact) * TC * dt); }
    static constexpr size_t RAW_BC = sizeof(Tact) * TC * 16;  // room for d_state 16, a multiple of 128
    static constexpr size_t WIDE = sizeof(float) * TC * 16;
    // (delta, delta * u) words, f32 rows of B and of C, then the landed tiles: a consumer that asks for a row ahead
    // reads past the end of the first three, not of the stage
    static __host__ __device__ constexpr size_t off_wide(int dt) { return 8 * TC * static_cast<size_t>(dt); }
    static __host__ __device__ constexpr size_t off_x(int dt) { return off_wide(dt) + 2 * WIDE; }
    static __host__ __device__ constexpr size_t off_dl(int dt) { return off_x(dt) + act(dt); }
    static __host__ __device__ constexpr size_t off_z(int dt) { return off_dl(dt) + act(dt); }
    static __host__ __device__ constexpr size_t off_rb(int dt) { return off_z(dt) + act(dt); }
    static __host__ __device__ constexpr size_t bytes(int dt) { return off_rb(dt) + 2 * RAW_BC; }
    // ring, D of the channels, mbarriers
    static __host__ __device__ constexpr size_t smem(int dt, int stages) {
        return stages * bytes(dt) + al(sizeof(float) * dt) + kF16BarBytes;
    }
};

// Four adjacent storage elements, aligned to four.
__device__ __forceinline__ void ld_quad(const float* src, float2* v) {
    const float4 w = *reinterpret_cast<const float4*>(src);
    v[0] = make_float2(w.x, w.y);
    v[1] = make_float2(w.z, w.w);
}
template <typename Th>
__device__ __forceinline__ void ld_quad(const Th* src, float2* v) {
    const uint2 w = *reinterpret_cast<const uint2*>(src);
    v[0] = unpack2<Th>(w.x);
    v[1] = unpack2<Th>(w.y);
}
// softplus_sel and silu_sel of two values.  For 16-bit storage the larger of v and ln(1 + e^min(v, 20)) takes the
// place of a choice at 20: below it they differ by less than a rounding where v is the larger one.
template <bool HALF>
__device__ __forceinline__ float2 softplus2(float2 v) {
    if constexpr (HALF) {
        const float2 m = mul2(make_float2(fminf(v.x, 20.0f), fminf(v.y, 20.0f)), splat2(kLog2e));
        const float2 e = add2(make_float2(ex2(m.x), ex2(m.y)), splat2(1.0f));
        const float2 r = mul2(make_float2(lg2(e.x), lg2(e.y)), splat2(kLn2));
        return make_float2(fmaxf(r.x, v.x), fmaxf(r.y, v.y));
    } else {
        return make_float2(softplusf_fast(v.x), softplusf_fast(v.y));
    }
}
template <bool HALF>
__device__ __forceinline__ float2 silu2(float2 v) {
    if constexpr (HALF) {
        const float2 w = mul2(v, splat2(0.5f));
        float2 t;
        asm("tanh.approx.f32 %0, %1;" : "=f"(t.x) : "f"(w.x));
        asm("tanh.approx.f32 %0, %1;" : "=f"(t.y) : "f"(w.y));
        return mul2(v, fma2(t, splat2(0.5f), splat2(0.5f)));
    } else {
        return make_float2(siluf_fast(v.x), siluf_fast(v.y));
    }
}

__device__ __forceinline__ void warp_arrive(uint64_t* bar, int lane) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, int* status) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, status));
}

// A place in the ring of stages: its index and the parity of the phase of its barriers, counted up without divisions
// (with them a chunk cost 1300 cycles more than its work).
struct RingPlace {
    int s = 0;
    uint32_t parity = 0;
    __device__ __forceinline__ void next(int stages) {
        if (++s == stages) {
            s = 0;
            parity ^= 1;
        }
    }
};

// The exponent of a decay, a times delta.  ex2.approx comes out low, by 5e-9 of its value on average from -0.002 to
// -0.0001 and by 1.6e-8 to 2.7e-8 from -0.5 to -0.004.  A state that decays slowly gathers that over every step of a piece:
// in f32 it was the largest part of the error, and grew with the piece.  The constant centres it at no cost and leaves
// ex2(0) = 1.  Distance from 64 bits in f32, y and the state, without it and with it: 1 x 1000 x 1536 whole 1.62e-6 and
// 8.2e-7, 4.0e-6 and 1.9e-6; 2 x 300 x 1536 in pieces 9.1e-7 and 5.9e-7, 1.22e-6 and 7.3e-7 (sscan_fwd_kernel, whose pieces
// are shorter: 6.4e-7 and 7.2e-7).  From 8e-9 to 1.4e-8 the sums differ by a fifth, 2.7e-8 is no better than none.  In
// 16-bit storage softplus is 1e-5 off and this is nothing.
template <bool HALF>
__device__ __forceinline__ float2 exponent(float2 delta, float2 a) {
    if constexpr (HALF) return mul2(delta, a);
    else return fma2(delta, a, splat2(1.2e-8f));
}

// FLAGS: bit0 softplus on delta, bit1 gate present, bit3 state-only pass (as sscan_fwd_kernel).
template <typename Tact, int NS, int TC, int FLAGS>
__global__ void __launch_bounds__(kF16Threads, 1)
sscan_fwd16_kernel(const __grid_constant__ Fwd16Params q) {
    using Stage = Fwd16Stage<Tact, TC>;
    constexpr bool kSoftplus = (FLAGS & 1) != 0, kStateOnly = (FLAGS & 8) != 0;
    constexpr bool kGate = (FLAGS & 2) != 0 && !kStateOnly;
    constexpr bool kHalf = sizeof(Tact) == 2;
    constexpr int LPC = 16 / NS, CHW = 64 / LPC;
    extern __shared__ __align__(128) unsigned char smem[];
    const FwdParams& p = q.f;
    const int DT = q.dt, W = __popc(q.consumers), HW = __popc(q.helpers), S = q.stages;
    const size_t stage_bytes = Stage::bytes(DT);
    float* dskip = reinterpret_cast<float*>(smem + S * stage_bytes);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + S * stage_bytes + Stage::al(sizeof(float) * DT));
    uint64_t* ready = full + kF16MaxStages;
    uint64_t* done = ready + kF16MaxStages;
    uint64_t* empty = done + kF16MaxStages;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned before_me = (1u << warp) - 1u;
    const int b = blockIdx.y, d0 = blockIdx.x * DT;
    const int T = p.T, D = p.D, N = p.N;
    const int nchunks_all = (T + TC - 1) / TC;
    const int seg = blockIdx.z, nseg = gridDim.z;
    const int c_begin = p.seg_chunks > 0 ? min(nchunks_all, seg * p.seg_chunks) : 0;
    const int c_end = (p.seg_chunks > 0 && seg + 1 < nseg) ? min(nchunks_all, (seg + 1) * p.seg_chunks) : nchunks_all;
    const int nch = c_end - c_begin;
    if (kStateOnly && seg == nseg - 1) return;  // nothing follows the last segment

    if (tid == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&ready[s], HW);
            mbar_init(&done[s], W);
            mbar_init(&empty[s], HW);
        }
        fence_barrier_init();
    }
    for (int i = tid; i < DT; i += blockDim.x) dskip[i] = d0 + i < D ? p.Dp[d0 + i] : 0.0f;
    __syncthreads();
    auto stage = [&](int s) { return smem + s * stage_bytes; };

    // =========================== producer ===========================
    if (warp == static_cast<int>(blockDim.x / 32) - 1) {
        if (lane != 0) return;
        const bool tma_b = (p.tma_mask & kTmaB) != 0, tma_c = !kStateOnly && (p.tma_mask & kTmaC) != 0;
        const uint32_t tx = sizeof(Tact) * TC * ((kGate ? 3 : 2) * DT + ((tma_b ? 1 : 0) + (tma_c ? 1 : 0)) * N);
        RingPlace to;
        int issued = 0;
        for (; issued < nch; ++issued, to.next(S)) {
            if (issued >= S && !mbar_wait(&empty[to.s], to.parity ^ 1, p.status)) break;
            unsigned char* st = stage(to.s);
            uint64_t* bar = &full[to.s];
            const int t0 = (c_begin + issued) * TC;
            mbar_expect_tx(bar, tx);
            tma_load_3d(st + Stage::off_dl(DT), &p.tm_dl, bar, d0, t0, b);
            tma_load_3d(st + Stage::off_x(DT), &p.tm_x, bar, d0, t0, b);
            if (tma_b) tma_load_3d(st + Stage::off_rb(DT), &p.tm_b, bar, 0, t0, b);
            if (tma_c) tma_load_3d(st + Stage::off_rb(DT) + Stage::RAW_BC, &p.tm_c, bar, 0, t0, b);
            if (kGate) tma_load_3d(st + Stage::off_z(DT), &p.tm_z, bar, d0, t0, b);
        }
        // The last copies land before the CTA may leave, also after a wait that gave up: what was not waited for
        // above are the last S of them.
        for (int k = max(0, issued - S); k < issued; ++k) mbar_wait(&full[k % S], (k / S) & 1, p.status);
        return;
    }

    // =========================== helpers ===========================
    if (q.helpers >> warp & 1) {
        // An item is two rows of four neighbouring channels; a thread's items are the same in every chunk.
        const int quarter = DT / 4, step = HW * 32, htid = __popc(q.helpers & before_me) * 32 + lane;
        const int drp = step / quarter, dcp = step % quarter, rp0 = htid / quarter, cp0 = htid % quarter;
        const bool silu = p.z_mode == 1;
        const bool wide = q.vec_y && d0 + DT <= D;  // every row of the tile is whole words of y
        auto items = [&](auto&& f) {
            int rp = rp0, cp = cp0;
            while (rp < TC / 2) {
                f(rp, cp);
                rp += drp;
                cp += dcp;
                if (cp >= quarter) {
                    cp -= quarter;
                    ++rp;
                }
            }
        };
        // B and C rows of the chunk as zero-padded f32: a thread has eight states of a row of B or of C at a time, from
        // the landed tiles, or from rows that no tensor map describes
        constexpr int kRows = (kStateOnly ? 1 : 2) * TC;
        auto widen = [&](unsigned char* st, int c) {
            float* wide = reinterpret_cast<float*>(st + Stage::off_wide(DT));
            const int nv = T - (c_begin + c) * TC;
            for (int i = htid; i < 2 * kRows; i += step) {
                const int r = (i >> 1) % TC, n0 = (i & 1) * 8;
                const bool is_c = !kStateOnly && i >= 2 * TC;
                const bool landed = (p.tma_mask & (is_c ? kTmaC : kTmaB)) != 0;
                const Tact* row = landed ? reinterpret_cast<const Tact*>(st + Stage::off_rb(DT) + (is_c ? Stage::RAW_BC : 0)) + r * N
                                         : static_cast<const Tact*>(is_c ? p.cm : p.bm) +
                                               (static_cast<long long>(b) * T + (c_begin + c) * TC + r) * p.ld_bc;
                float v[8];
                if (N == 16 && landed) {
                    float2 w[4];
                    ld_quad(row + n0, w);
                    ld_quad(row + n0 + 4, w + 2);
#pragma unroll
                    for (int j = 0; j < 8; ++j) v[j] = j & 1 ? w[j / 2].y : w[j / 2].x;
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) v[j] = (n0 + j < N && r < nv) ? to_f(row[n0 + j]) : 0.0f;
                }
                float4* out = reinterpret_cast<float4*>(wide + i * 8);  // B's rows, then C's
                out[0] = make_float4(v[0], v[1], v[2], v[3]);
                out[1] = make_float4(v[4], v[5], v[6], v[7]);
            }
        };
        // before the recurrence; WHOLE: no row of the chunk is past the end
        auto before = [&](auto whole_tag, unsigned char* st, int c) {
            constexpr bool WHOLE = decltype(whole_tag)::value;
            const int nv = T - (c_begin + c) * TC;
            items([&](int rp, int cp) {
                const Tact* xs = reinterpret_cast<const Tact*>(st + Stage::off_x(DT)) + 2 * rp * DT + 4 * cp;
                const Tact* ds = reinterpret_cast<const Tact*>(st + Stage::off_dl(DT)) + 2 * rp * DT + 4 * cp;
                float4* dst = reinterpret_cast<float4*>(st) + rp * DT + cp;  // a row: DT / 2 words
                float2 x[2][2], dl[2][2], du[2][2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    ld_quad(ds + i * DT, dl[i]);
                    ld_quad(xs + i * DT, x[i]);
                }
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const bool in = WHOLE || 2 * rp + i < nv;
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        if (kSoftplus) dl[i][k] = softplus2<kHalf>(dl[i][k]);
                        du[i][k] = mul2(dl[i][k], x[i][k]);
                        if (!in) dl[i][k] = du[i][k] = splat2(0.0f);
                    }
                }
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int k = 0; k < 2; ++k)
                        dst[(2 * i + k) * quarter] = make_float4(dl[i][k].x, dl[i][k].y, du[i][k].x, du[i][k].y);
            });
        };
        // after it; WHOLE: every row and channel of the tile is written, two elements to a store
        auto after = [&](auto whole_tag, unsigned char* st, int c) {
            constexpr bool WHOLE = decltype(whole_tag)::value;
            const int t0 = (c_begin + c) * TC, nv = T - t0;
            Tact* yg = static_cast<Tact*>(p.y) + (static_cast<long long>(b) * T + t0) * p.ld_y + d0;
            items([&](int rp, int cp) {
                const Tact* xs = reinterpret_cast<const Tact*>(st + Stage::off_x(DT)) + 2 * rp * DT + 4 * cp;
                const Tact* zs = reinterpret_cast<const Tact*>(st + Stage::off_z(DT)) + 2 * rp * DT + 4 * cp;
                const float4* src = reinterpret_cast<const float4*>(st) + rp * DT + cp;
                float2 x[2][2], z[2][2];
                float2 y[2][2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    if (kGate) ld_quad(zs + i * DT, z[i]);
                    ld_quad(xs + i * DT, x[i]);
                }
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int k = 0; k < 2; ++k) y[i][k] = *reinterpret_cast<const float2*>(src + (2 * i + k) * quarter);
                const float4 dk = *reinterpret_cast<const float4*>(dskip + 4 * cp);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    float2 v[2];
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        v[k] = fma2(k ? make_float2(dk.z, dk.w) : make_float2(dk.x, dk.y), x[i][k], y[i][k]);
                        if (kGate) v[k] = mul2(v[k], silu ? silu2<kHalf>(z[i][k]) : z[i][k]);
                    }
                    const int row = 2 * rp + i, dc = 4 * cp;
                    Tact* dst = yg + row * p.ld_y + dc;
                    if (WHOLE) {
                        st_pair(dst, v[0]);
                        st_pair(dst + 2, v[1]);
                    } else if (row < nv) {
                        const float o[4] = {v[0].x, v[0].y, v[1].x, v[1].y};
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (d0 + dc + k < D) dst[k] = from_f<Tact>(o[k]);
                    }
                }
            });
        };
        RingPlace in, out;
        for (int c = 0; c <= nch; ++c) {
            if (c < nch) {
                if (!warp_wait(&full[in.s], in.parity, p.status)) return;
                widen(stage(in.s), c);
                if (T - (c_begin + c) * TC >= TC) before(std::true_type{}, stage(in.s), c);
                else before(std::false_type{}, stage(in.s), c);
                warp_arrive(&ready[in.s], lane);
                in.next(S);
            }
            if (c >= 1) {
                if (!warp_wait(&done[out.s], out.parity, p.status)) return;
                if (!kStateOnly) {
                    if (wide && T - (c_begin + c - 1) * TC >= TC) after(std::true_type{}, stage(out.s), c - 1);
                    else after(std::false_type{}, stage(out.s), c - 1);
                }
                warp_arrive(&empty[out.s], lane);
                out.next(S);
            }
        }
        return;
    }

    // =========================== consumers ===========================
    if (!(q.consumers >> warp & 1)) return;  // left free to even the schedulers out
    const int part = lane % LPC, pos = __popc(q.consumers & before_me) * (CHW / 2) + lane / LPC;  // states, pair of channels
    const int d = d0 + 4 * (pos % (DT / 4)) + 2 * (pos / (DT / 4));
    const int n0 = part * NS;
    // h of either channel by pairs of states; a_neg * log2(e) by pairs of channels, which (delta, delta) multiplies as
    // it comes: the exponentials put their results wherever they are wanted
    float2 h[2][NS / 2], a2[NS], a_inc;
    bool progression = true;
    {
        const float* h0 = seg == 0 && p.ssm_in ? p.ssm_in + static_cast<long long>(b) * D * N : nullptr;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float av[NS], hv[NS];
#pragma unroll
            for (int j = 0; j < NS; ++j) {
                const bool ok = d + i < D && n0 + j < N;
                const long long at = static_cast<long long>(d + i) * N + n0 + j;
                av[j] = ok ? p.a_neg[at] * kLog2e : 0.0f;
                if (fabsf(av[j]) > 3e38f) av[j] = copysignf(3e38f, av[j]);  // 0 * infinity in the rows past the end
                hv[j] = (ok && h0) ? h0[at] : 0.0f;
                if (kStateOnly && seg == 0 && ok && p.ssm_copy) p.ssm_copy[static_cast<long long>(b) * D * N + at] = hv[j];
            }
            const float inc = av[1] - av[0];  // a[n] = a[n0] + (n - n0) * inc to 4 ulp (a NaN is none)
            if (i) a_inc.y = inc;
            else a_inc.x = inc;
#pragma unroll
            for (int j = 2; j < NS; ++j)
                if (!(fabsf(av[j] - fmaf(static_cast<float>(j), inc, av[0])) <= 4.8e-7f * fabsf(av[j]))) progression = false;
#pragma unroll
            for (int j = 0; j < NS; ++j) {
                if (i) a2[j].y = av[j];
                else a2[j].x = av[j];
                if (j & 1) h[i][j / 2] = make_float2(hv[j - 1], hv[j]);
            }
        }
    }
    // The state that enters a later segment: h = exp(a * sum of its deltas) h + what it leaves from zero, over the
    // segments before this one (the first of which started from the real state).  Every CTA does this for itself, from
    // L2, a few segments' loads at a time: with a launch of its own between the passes it took 3 us more.
    if (!kStateOnly && seg > 0) {
        const long long row = static_cast<long long>(D) * N;
        const float* left = p.seg_states + static_cast<long long>(b) * nseg * row + static_cast<long long>(d) * N + n0;
        const float* sums = p.seg_sumdl + static_cast<long long>(b) * nseg * D + d;
        constexpr int U = NS == 8 ? 2 : 4;
        for (int s0 = 0; s0 < seg; s0 += U) {
            float w[U][2][NS], dl[U][2];
#pragma unroll
            for (int k = 0; k < U; ++k) {
                const int s = min(s0 + k, seg - 1);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const bool ok = d + i < D;
                    dl[k][i] = ok ? sums[static_cast<long long>(s) * D + i] : 0.0f;
                    if (N == 16 && ok) {
#pragma unroll
                        for (int v = 0; v < NS; v += 4) {
                            const float4 f = *reinterpret_cast<const float4*>(left + s * row + i * 16 + v);
                            w[k][i][v] = f.x, w[k][i][v + 1] = f.y, w[k][i][v + 2] = f.z, w[k][i][v + 3] = f.w;
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < NS; ++j) w[k][i][j] = ok && n0 + j < N ? left[s * row + i * N + j] : 0.0f;
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < U; ++k)
                if (s0 + k < seg) {
#pragma unroll
                    for (int i = 0; i < 2; ++i)
#pragma unroll
                        for (int j = 0; j < NS; ++j) {
                            float& x = j & 1 ? h[i][j / 2].y : h[i][j / 2].x;
                            x = s0 + k ? fmaf(ex2((i ? a2[j].y : a2[j].x) * dl[k][i]), x, w[k][i][j]) : w[k][i][j];
                        }
                }
        }
    }
    const bool geo = __all_sync(0xffffffffu, progression);
    float2 sum_dl = splat2(0.0f);

    auto chunk = [&](auto geo_tag, unsigned char* st) {
        constexpr bool GEO = decltype(geo_tag)::value;
        constexpr int RB = 4;  // rows of the loop's body: longer ones wait for their instructions
        const int row_words = DT / 2;
        float4* pp = reinterpret_cast<float4*>(st) + pos;
        const float4* Bp = reinterpret_cast<const float4*>(st + Stage::off_wide(DT)) + part * (NS / 4);
        constexpr int kToC = TC * 4;  // from a word of B to that of C
        // Two rows are in work: the operands and decays of the next one between the recurrence of this one, state by
        // state, so that neither the MUFU nor the FMA pipe waits for the other.
        struct Row {
            float4 w, b[NS / 4], c[NS / 4];
            float2 e[2][NS / 2], r[2];
        };
        auto operands = [&](Row& q, const float4* from) {
#pragma unroll
            for (int v = 0; v < NS / 4; ++v) {
                q.b[v] = from[v];
                if (!kStateOnly) q.c[v] = from[kToC + v];
            }
        };
        auto decay = [&](Row& q, int j) {  // of states 2 j and 2 j + 1 of both channels
            const float2 dl = make_float2(q.w.x, q.w.y);
            if (GEO) {
                if (j == 0) {
                    const float2 xe = exponent<kHalf>(dl, a2[0]), xr = exponent<kHalf>(dl, a_inc);
                    const float2 r = make_float2(ex2(xr.x), ex2(xr.y)), r2 = mul2(r, r);
                    q.e[0][0].x = ex2(xe.x);
                    q.e[1][0].x = ex2(xe.y);
                    q.e[0][0].y = q.e[0][0].x * r.x;
                    q.e[1][0].y = q.e[1][0].x * r.y;
                    q.r[0] = splat2(r2.x);
                    q.r[1] = splat2(r2.y);
                } else {
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        if (j == 2) q.r[i] = mul2(q.r[i], q.r[i]);
                        q.e[i][j] = mul2(q.e[i][j == 1 ? 0 : j - 2], q.r[i]);
                    }
                }
            } else {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const float2 x = exponent<kHalf>(dl, a2[2 * j + k]);
                    if (k) q.e[0][j].y = ex2(x.x), q.e[1][j].y = ex2(x.y);
                    else q.e[0][j].x = ex2(x.x), q.e[1][j].x = ex2(x.y);
                }
            }
        };
        // Sums over the pair's lanes: lane `part` gets that of row part of the four (and, with two lanes, part + 2).
        // y goes where all lanes of the pair have read delta.
        auto half_sum = [&](float2 lo, float2 hi, int bit) {
            const bool up = part & bit;
            const float2 keep = up ? hi : lo, send = up ? lo : hi;
            return add2(keep, make_float2(__shfl_xor_sync(0xffffffffu, send.x, bit), __shfl_xor_sync(0xffffffffu, send.y, bit)));
        };
        auto finish = [&](const float2* yp, float4* to, bool store) {
            if constexpr (LPC == 4) {
                const float2 v = half_sum(half_sum(yp[0], yp[2], 2), half_sum(yp[1], yp[3], 2), 1);
                if (store) *reinterpret_cast<float2*>(to) = v;
            } else {
                const float2 v = half_sum(yp[0], yp[1], 1), w = half_sum(yp[2], yp[3], 1);
                if (store) *reinterpret_cast<float2*>(to) = v;
                if (store) *reinterpret_cast<float2*>(to + 2 * row_words) = w;
            }
        };
        Row rows[RB + 1];
        float2 yp[RB] = {};  // of the rows before these: their sums wait for no one while these rows are in work
        float4 w_next = pp[row_words];
        rows[0].w = pp[0];
        operands(rows[0], Bp);
#pragma unroll
        for (int j = 0; j < NS / 2; ++j) decay(rows[0], j);
#pragma unroll 1
        for (int r0 = 0; r0 < TC; r0 += RB) {
            float2 yn[RB];
            if (!kStateOnly) finish(yp, pp + (part - RB) * row_words, r0 > 0);
#pragma unroll
            for (int k = 0; k < RB; ++k) {
                const Row& q = rows[k];
                Row& nx = rows[k + 1];
                nx.w = w_next;
                w_next = pp[(k + 2) * row_words];
                operands(nx, Bp + (k + 1) * 4);
                float2 y[2];
#pragma unroll
                for (int j = 0; j < NS / 2; ++j) {
                    const float4 bv = q.b[j / 2], cv = q.c[j / 2];
                    const float2 b2 = j & 1 ? make_float2(bv.z, bv.w) : make_float2(bv.x, bv.y);
                    const float2 c2 = j & 1 ? make_float2(cv.z, cv.w) : make_float2(cv.x, cv.y);
                    decay(nx, j);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        h[i][j] = fma2(q.e[i][j], h[i][j], mul2(splat2(i ? q.w.w : q.w.z), b2));
                        if (!kStateOnly) y[i] = j ? fma2(h[i][j], c2, y[i]) : mul2(h[i][j], c2);
                    }
                }
                if (kStateOnly) sum_dl = add2(sum_dl, make_float2(q.w.x, q.w.y));
                else yn[k] = make_float2(y[0].x + y[0].y, y[1].x + y[1].y);
            }
            rows[0] = rows[RB];
#pragma unroll
            for (int k = 0; k < RB; ++k) yp[k] = yn[k];
            pp += RB * row_words;
            Bp += RB * 4;
        }
        if (!kStateOnly) finish(yp, pp + (part - RB) * row_words, true);
    };

    // the states of this lane to rows of N floats at dst
    auto put = [&](float* dst) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (d + i >= D) continue;
            float* to = dst + static_cast<long long>(d + i) * N + n0;
            if (q.vec_state) {
#pragma unroll
                for (int v = 0; v < NS / 4; ++v)
                    *reinterpret_cast<float4*>(to + 4 * v) = make_float4(h[i][2 * v].x, h[i][2 * v].y, h[i][2 * v + 1].x, h[i][2 * v + 1].y);
            } else {
#pragma unroll
                for (int j = 0; j < NS; ++j)
                    if (n0 + j < N) to[j] = j & 1 ? h[i][j / 2].y : h[i][j / 2].x;
            }
        }
    };
    RingPlace at;
    int to_save = p.save_stride - (c_begin * TC) % p.save_stride;  // steps to the next saved state, save_stride: now
    float* saved = p.chunk_states ? p.chunk_states + b * p.cs_ld_b + (c_begin * TC + p.save_stride - 1) / p.save_stride * p.cs_ld_k : nullptr;
    for (int c = 0; c < nch; ++c) {
        const int s = at.s;
        if (!warp_wait(&ready[s], at.parity, p.status)) return;
        at.next(S);
        if (!kStateOnly && saved) {
            if (to_save == p.save_stride) {
                put(saved);
                saved += p.cs_ld_k;
            }
            to_save -= TC;
            if (to_save == 0) to_save = p.save_stride;
        }
        if (geo) chunk(std::true_type{}, stage(s));
        else chunk(std::false_type{}, stage(s));
        warp_arrive(&done[s], lane);
    }
    if (kStateOnly) {
        put(p.seg_states + (static_cast<long long>(b) * nseg + seg) * D * N);
        if (part == 0) {
            float* to = p.seg_sumdl + (static_cast<long long>(b) * nseg + seg) * D;
            if (d < D) to[d] = sum_dl.x;
            if (d + 1 < D) to[d + 1] = sum_dl.y;
        }
    } else if (p.ssm_state && seg == nseg - 1) {
        put(p.ssm_state + static_cast<long long>(b) * D * N);
    }
}

typedef void (*Fwd16KernelFn)(const Fwd16Params);

// Steps of a chunk: the tiles of f32 storage fill the stages twice as fast.
template <typename Tact>
constexpr int fwd16_steps() {
    return sizeof(Tact) == 4 ? 16 : 32;
}

// By lanes' states (4, 8) and flags: 0 .. 3 softplus / gate, 4 and 5 the state-only passes.
struct Fwd16Table {
    Fwd16KernelFn fn[2][6];
    int steps[2];
    size_t (*smem[2])(int channels, int stages);
};
template <typename Tact, int NS>
static void fill_fwd16(Fwd16Table* t, int i) {
    constexpr int TC = fwd16_steps<Tact>();
    t->steps[i] = TC;
    t->smem[i] = [](int channels, int stages) { return Fwd16Stage<Tact, TC>::smem(channels, stages); };
    t->fn[i][0] = sscan_fwd16_kernel<Tact, NS, TC, 0>;
    t->fn[i][1] = sscan_fwd16_kernel<Tact, NS, TC, 1>;
    t->fn[i][2] = sscan_fwd16_kernel<Tact, NS, TC, 2>;
    t->fn[i][3] = sscan_fwd16_kernel<Tact, NS, TC, 3>;
    t->fn[i][4] = sscan_fwd16_kernel<Tact, NS, TC, 8>;
    t->fn[i][5] = sscan_fwd16_kernel<Tact, NS, TC, 9>;
}
template <typename Tact>
static void build_fwd16(Fwd16Table* t) {
    fill_fwd16<Tact, 4>(t, 0);
    fill_fwd16<Tact, 8>(t, 1);
}
void fwd16_f32(Fwd16Table* t);
void fwd16_f16(Fwd16Table* t);
void fwd16_bf16(Fwd16Table* t);

}  // namespace mb200
