// Mamba-3 SISO SSD scan (trapezoidal recurrence) forward for sm_100a.
//
// Two kernels behind one entry point:
//  * m3_ssd_fwd_tc_kernel — chunked form on the 5th-generation tensor cores
//    (tcgen05.mma, accumulators in TMEM) for 16-bit storage, headdim 64,
//    d_state 128: per (sample, head) one CTA walks 128-step chunks and keeps
//    the running state S^T [N x hd] f32 resident in TMEM, so the entering states
//    never touch HBM (the reference writes [B, chunks, nh, hd, N] f32 of them).
//    Per chunk: G = Q K^T, decay/causal mask in registers, Y1 = M V,
//    Y2 = Q S_in^T, S^T <- exp(dA_end) S^T + K^T (w o V).
//    With a carried state the same kernel starts from it (CARRY).
//  * m3_ssd_seq_kernel — the sequential definition (eight rows p per warp, state in
//    registers) for every other shape / dtype, and for carried windows that are short or f16.
#include <string.h>

#include <type_traits>

#include "common.cuh"
#include "internal.h"
#include "m3_tc.cuh"

namespace mb200 {

struct M3Params {
    // tensor-core kernel: Q (or Cn), K (or Bn) and x as [128 x 64] swizzled sub-tile maps
    CUtensorMap tm_q, tm_k, tm_v;
    CUtensorMap tm_adt, tm_dt, tm_trap;  // [B,T,nh] f32, boxes of 4 heads x 129 rows
    int sc_tma;                          // 1: the three maps above are valid (nheads % 4 == 0)
    int wide_y;                          // 1: y rows leave as 256-bit stores
    const void *x, *K, *Q;
    const float *dt, *trap, *adt, *Dh;
    void* y;
    float *ssm_state, *k_state, *v_state;  // in/out (may be null: zero in, not written)
    int B, T, nh, hd, N;
    int carry_in;  // 1: the state buffers hold a state to continue from
    // Optional: K and Q built inside the tensor-core kernel from the group-level
    // B / C after BCNorm, the per-head biases and RoPE (Bn == nullptr: K, Q are read).
    const void *Bn, *Cn;            // [B,T,ng,N] storage dtype
    const float *b_bias, *c_bias;   // [nh,N]
    const float* angle_vel;         // [B,T,n_angles]: tanh(angles_raw) * pi
    float* angle_state;             // [B,nh,n_angles] in/out (may be null: zero in, not written)
    int ng, n_angles;
    int* status;
};

// ---------------------------------------------------------------------------
// Sequential definition, src/mamba3_siso/cpu/forward.rs:85-138 / kernels/mamba3_ssd.cu:229-348:
//   h = alpha h + (beta v_prev) k_prev + (gamma x) k ;  y = <h, q> + D x
// A warp owns R rows p of one (sample, head); its lanes split the state index (n = lane + 32 i),
// so the state, K and Q move as whole 128-byte rows and no block barrier is needed.  The dot
// products of a step are reduced by a halving butterfly that leaves row r in one lane group.
// With few heads the chain of one step bounds it (0.37 us a step at 1 x 4 heads of 64 x 128; loads
// are requested PF steps ahead), with many the issue slots (1.5 us at 8 x 32 heads); one thread per
// row with 128 states in registers and two block barriers a step, which it replaces, took 8 us.
// grid (nh, B, ceil(hd / rows of a CTA)).
// ---------------------------------------------------------------------------
template <typename Tact, int NI, int R, bool PART>  // PART: the last 32 states are not all there
__global__ void __launch_bounds__(256) m3_ssd_seq_kernel(const M3Params p) {
    constexpr int PF = 4;  // steps requested ahead
    const int h = blockIdx.x, b = blockIdx.y, lane = threadIdx.x & 31;
    const int N = p.N, hd = p.hd, nh = p.nh, T = p.T;
    const int p0 = (blockIdx.z * (blockDim.x >> 5) + (threadIdx.x >> 5)) * R;
    const long long bh = static_cast<long long>(b) * nh + h;
    // lane -> output row of this warp after the butterfly: R == 8: bits 4..2, R == 2: bit 4
    const int rl = R == 8 ? ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1) : (lane >> 4) & 1;
    const bool rok = p0 + rl < hd;
    const bool writer = rok && (R == 8 ? (lane & 3) == 0 : (lane & 15) == 0);
    bool nok[NI];
#pragma unroll
    for (int i = 0; i < NI; ++i) nok[i] = lane + 32 * i < N;
    float st[R][NI], kp[NI], vp[R];
#pragma unroll
    for (int i = 0; i < NI; ++i) kp[i] = 0.0f;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        vp[r] = 0.0f;
#pragma unroll
        for (int i = 0; i < NI; ++i) st[r][i] = 0.0f;
    }
    if (p.carry_in) {
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (p0 + r < hd) {
                vp[r] = p.v_state[bh * hd + p0 + r];
#pragma unroll
                for (int i = 0; i < NI; ++i)
                    if (nok[i]) st[r][i] = p.ssm_state[(bh * hd + p0 + r) * N + lane + 32 * i];
            }
#pragma unroll
        for (int i = 0; i < NI; ++i)
            if (nok[i]) kp[i] = p.k_state[bh * N + lane + 32 * i];
        __syncthreads();  // the CTA's warps have read k_state before one of them overwrites it
    }
    if (p0 >= hd) return;
    const Tact* xb = static_cast<const Tact*>(p.x) + static_cast<long long>(b) * T * nh * hd + h * hd + p0 + rl;
    const Tact* Kb = static_cast<const Tact*>(p.K) + (static_cast<long long>(b) * T * nh + h) * N + lane;
    const Tact* Qb = static_cast<const Tact*>(p.Q) + (static_cast<long long>(b) * T * nh + h) * N + lane;
    Tact* yb = static_cast<Tact*>(p.y) + static_cast<long long>(b) * T * nh * hd + h * hd + p0 + rl;
    const float Dv = p.Dh[h];
    Tact kr[PF][NI], qr[PF][NI], xr[PF];
    float sa[PF], sd[PF], sg[PF];
    auto request = [&](int t, int s) {
        if (t >= T) return;
        const long long th = (static_cast<long long>(b) * T + t) * nh + h;
        const long long kq = static_cast<long long>(t) * nh * N;
        sa[s] = p.adt[th]; sd[s] = p.dt[th]; sg[s] = p.trap[th];
#pragma unroll
        for (int i = 0; i < NI; ++i)
            if (nok[i]) {
                kr[s][i] = Kb[kq + 32 * i];
                qr[s][i] = Qb[kq + 32 * i];
            }
        if (rok) xr[s] = xb[static_cast<long long>(t) * nh * hd];
    };
#pragma unroll
    for (int s = 0; s < PF; ++s) request(s, s);
    for (int tb = 0; tb < T; tb += PF) {
#pragma unroll
        for (int s = 0; s < PF; ++s) {
            const int t = tb + s;
            if (t < T) {
                const float alpha = ex2(sa[s] * kLog2e);
                const float beta = alpha * sd[s] * (1.0f - sg[s]), gamma = sg[s] * sd[s];
                const float xv = rok ? to_f(xr[s]) : 0.0f;
                float k[NI], q[NI], acc[R];
#pragma unroll
                for (int i = 0; i < NI; ++i) {
                    k[i] = nok[i] ? to_f(kr[s][i]) : 0.0f;
                    q[i] = nok[i] ? to_f(qr[s][i]) : 0.0f;
                }
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int src = R == 8 ? ((r >> 2) & 1) * 16 + ((r >> 1) & 1) * 8 + (r & 1) * 4 : r * 16;
                    const float xb_r = __shfl_sync(0xffffffffu, xv, src);
                    const float bv = beta * vp[r], gx = gamma * xb_r;
                    acc[r] = 0.0f;
#pragma unroll
                    for (int i = 0; i < NI; ++i) {
                        if (PART && !nok[i]) continue;  // (an infinite x would make a NaN of the zeros there)
                        st[r][i] = fmaf(alpha, st[r][i], fmaf(bv, kp[i], gx * k[i]));
                        acc[r] = fmaf(st[r][i], q[i], acc[r]);
                    }
                    vp[r] = xb_r;
                }
#pragma unroll
                for (int i = 0; i < NI; ++i) kp[i] = k[i];
                request(t + PF, s);
                // halving butterfly over the lanes: R sums, one per lane group
                int m = 16;
#pragma unroll
                for (int w = R / 2; w >= 1; w >>= 1, m >>= 1) {
                    const bool up = (lane & m) != 0;
#pragma unroll
                    for (int r = 0; r < w; ++r) {
                        const float give = up ? acc[r] : acc[r + w], keep = up ? acc[r + w] : acc[r];
                        acc[r] = keep + __shfl_xor_sync(0xffffffffu, give, m);
                    }
                }
                float y = acc[0];
#pragma unroll
                for (int mm = R == 8 ? 2 : 8; mm >= 1; mm >>= 1) y += __shfl_xor_sync(0xffffffffu, y, mm);
                if (writer) yb[static_cast<long long>(t) * nh * hd] = from_f<Tact>(fmaf(Dv, xv, y));
            }
        }
    }
    if (gridDim.z == 1 && threadIdx.x < 32 && p.k_state) {
#pragma unroll
        for (int i = 0; i < NI; ++i)
            if (nok[i]) p.k_state[bh * N + lane + 32 * i] = kp[i];
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (p0 + r < hd) {
            if (p.ssm_state)
#pragma unroll
                for (int i = 0; i < NI; ++i)
                    if (nok[i]) p.ssm_state[(bh * hd + p0 + r) * N + lane + 32 * i] = st[r][i];
            if (p.v_state && lane == 0) p.v_state[bh * hd + p0 + r] = vp[r];
        }
}

// k_state after the window when several CTAs share a (sample, head): any of them may still be
// reading the entering k_state when another has finished.
template <typename Tact>
__global__ void m3_seq_kstate_kernel(const M3Params p) {
    const int h = blockIdx.x, b = blockIdx.y;
    const Tact* kl = static_cast<const Tact*>(p.K) + ((static_cast<long long>(b) * p.T + p.T - 1) * p.nh + h) * p.N;
    for (int n = threadIdx.x; n < p.N; n += blockDim.x)
        p.k_state[(static_cast<long long>(b) * p.nh + h) * p.N + n] = to_f(kl[n]);
}

// ---------------------------------------------------------------------------
// tcgen05 / TMEM chunked kernel.  hd = 64, N = 128, chunk = 128, 256 threads.
// ---------------------------------------------------------------------------
namespace tc {

constexpr int CS = 128, HD = 64, NS = 128;
// Shared-memory operand tiles are 128-byte-swizzled [rows x 64] sub-tiles (m3_tc.cuh); TMA
// lands Q, K and V in that form.  One CTA per SM.  Q, K and V are double-buffered: the
// copies of chunk c + 1 are issued (one thread, five boxes) before chunk c is touched, so a
// whole chunk of work hides their latency -- with single buffers, two CTAs per SM and
// 16-byte asynchronous copies, 7.6 of the 11.5 us a chunk took were spent waiting for its
// tiles.  M has its own tile; one more tile holds w o V for the state update and then the
// 16-bit copy of the new state for the next chunk's Y2; then f32 vectors, barriers.
constexpr uint32_t kQ0 = 0, kK0 = 65536, kV0 = 131072, kQKStride = 32768, kVStride = 16384;
constexpr uint32_t kM = 163840, kVw = 196608, kS = 196608;
// carried state: one Q, K and V buffer; remainders of M, w o V (two) and the state copy behind them
constexpr uint32_t kCarryK = 32768, kCarryV = 65536, kMlo = 81920, kVwLo = 114688, kSlo = kVwLo, kVwRest = 131072;
static_assert(kVwRest + 16384 <= kM, "carry layout");
// f32 dA[128], scale[128], gamma[128], dA*log2(e)[128], dt[128] per chunk, two sets: a chunk's
// set is written while slower threads may still read the previous chunk's
constexpr uint32_t kVec = 212992, kVecSet = 5 * 128;
// K / Q generation: the angle entering the chunk, f64 [64]; this head's B / C biases [2][128]
constexpr uint32_t kCarry = kVec + 2 * kVecSet * 4, kBias = kCarry + 64 * 8;
// per-row adt, dt, trap of a chunk (dt and trap with the row after it), two buffers,
// filled by 4-byte asynchronous copies
// [3][129 rows][4 heads] f32; a TMA destination has to start on a 128-byte boundary
constexpr uint32_t kStage = kBias + 2 * 128 * 4, kStageArr = 17 * 128;
static_assert(kStage % 128 == 0 && kStageArr >= 129 * 16, "scalar staging");
constexpr uint32_t kBar = kStage + 3 * kStageArr + 16, kTmemSlot = kBar + 48;
constexpr uint32_t kTot = kTmemSlot + 8;  // SEG: log2 of the decay over this CTA's chunks
constexpr uint32_t kSmem = kTmemSlot + 16;
constexpr uint32_t kLoc = kM;             // SEG: f32 local state [128 n][64 p], before M is used
// TMEM columns: G; Y1; Y2; S^T.
constexpr uint32_t cG = 0, cY1 = 256, cY2 = 320, cS = 384, kTmemCols = 512;

// LEAN: two CTAs per SM, so that one's tensor-core and copy waits (3000 of a chunk's 7300 cycles) are the other's time.
// One buffer for Q, K and V, asked for again when the last MMA of a chunk is done; M over the Q tile, Y1 over G, which
// have been read by then.  8 x 4096 steps x 32 heads of 64 x 128: 250 -> 195 us (0.63 of the measured HBM rate), the same
// bits.  What is left is the chain of a chunk, 11600 cycles long with the copies in it.  Two CTAs leave 128 registers a
// thread: 76 bytes of each spill (carried windows 116).  Not kept: the next chunk's tiles brought into L2 ahead (201 us),
// V on a barrier of its own and another warp for the copies (196).
// Carried windows (CARRY) do this too, although they have five more operand tiles: the remainders take turns in the tiles
// of the first products (S_lo after S, M_lo after M, the second and third part of w o V after the first), five MMA groups
// a chunk for two, whose waits are the other CTA's time.  Y2 takes its rows' decay in tensor memory and M V on top, which
// leaves G readable.  The state's sums keep their order, and its bits.  8 x 256 steps x 32 heads: 62 -> 47 us with inputs
// that are new to the caches.
namespace lean {
constexpr uint32_t kK0 = 32768, kV0 = 65536, kVw = 81920, kVec = 98304, kStage = kVec + 2 * kVecSet * 4;
static_assert(kStage % 128 == 0, "scalar staging");
constexpr uint32_t kBar = kStage + 3 * kStageArr + 16, kTmemSlot = kBar + 48, kSmem = kTmemSlot + 16;
static_assert(2 * (kSmem + 1024) <= 228 * 1024, "two CTAs per SM");
constexpr uint32_t cY2 = 128, cS = 192, kTmemCols = 256;
}  // namespace lean

// GEN: build the K and Q tiles of a chunk in the kernel instead of reading them:
//   K[t,h,:] = rope(Bn[t,g,:] + b_bias[h,:], angle[t,h,:]),  Q likewise from Cn / c_bias,
//   angle[t,h,a] = (angle_in[h,a] + sum_{s<=t} angle_vel[s,a] * dt[s,h]) mod 2 pi
// (src/mamba3_siso/cpu/forward.rs:336-375; kernels/mamba3_ops.cu:279-310, :400-440,
// :575-640).  The in-chunk sums run in f32 (shuffle scans over the rows), the angle
// entering a chunk is carried in f64.
//
// CARRY: continue from ssm_state / k_state / v_state.  In the shifted form the state that enters
// is S = h + dt_0 (1 - trap_0) k_prev v_prev^T, so it is loaded into TMEM and the first chunk is
// a chunk like any other.  A carried state is kept to f32 accuracy as the sequential definition
// keeps it (K, Q and V are 16-bit inputs and exact): w o V, which the state is made of, is three
// bf16 values, f32's 24 bits, with a product each; M and the state copy, which only y is made of,
// are two, 2^-17 of each term against the 2^-9 that y is rounded to.  The further tiles take the
// room of the second Q / K / V buffers: Q of the next chunk is requested when the first MMA group
// has read it, K and V when the second has.  8 x 256 steps x 32 heads of 64 x 128: 62 us, 47 as LEAN (393
// by the sequential kernel).  The state's error against 64 bits there is 1.1e-6 (sequentially 3.2e-6),
// over 1 x 1000 steps 6.2e-7 (5.4e-7; 2.5e-6 with w o V of two values).  bf16 only: f16's range
// does not hold the remainders (x of 1e-3 left an error of 4e-3) nor products beyond 65504, so a
// carried f16 window is the sequential kernel's.
//
// SEG: the chunks of a (sample, head) are divided over the CTAs of a thread-block cluster, for shapes
// with fewer (sample, head) pairs than SMs.  Every CTA but the last first walks its chunks for the state
// alone (K, V, one product a chunk) from zero; the CTAs then read one another's local states and decays
// through distributed shared memory, which gives each the exact state entering its chunks, and walk them
// in full.
template <typename Th, bool GEN, bool CARRY, bool SEG, bool LEAN>
__global__ void __launch_bounds__(256, LEAN ? 2 : 1) m3_ssd_fwd_tc_kernel(const __grid_constant__ M3Params p) {
    static_assert(!LEAN || !(GEN || SEG), "the other forms need the room");
    constexpr bool TURNS = CARRY && LEAN;  // the remainders' products take turns in the tiles of the first ones
    constexpr uint32_t kK0 = LEAN ? lean::kK0 : tc::kK0, kV0 = LEAN ? lean::kV0 : tc::kV0, kM = LEAN ? kQ0 : tc::kM;
    constexpr uint32_t kVw = LEAN ? lean::kVw : tc::kVw, kS = kVw, kVec = LEAN ? lean::kVec : tc::kVec;
    constexpr uint32_t kStage = LEAN ? lean::kStage : tc::kStage, kBar = LEAN ? lean::kBar : tc::kBar;
    constexpr uint32_t kTmemSlot = LEAN ? lean::kTmemSlot : tc::kTmemSlot, kTmemCols = LEAN ? lean::kTmemCols : tc::kTmemCols;
    constexpr uint32_t cY1 = LEAN ? cG : tc::cY1, cY2 = LEAN ? lean::cY2 : tc::cY2, cS = LEAN ? lean::cS : tc::cS;
    constexpr uint32_t kQKStride = LEAN ? 0 : tc::kQKStride, kVStride = LEAN ? 0 : tc::kVStride;  // to the second buffer
    constexpr uint32_t kQKBytes = tc::kQKStride, kVBytes = tc::kVStride;
    extern __shared__ __align__(1024) unsigned char smem[];
    // two threads per step: thread (row, half) owns row `row` of the chunk (TMEM lane
    // `row`) and half of that row's columns in every elementwise stage
    const int tid = threadIdx.x & 127, half = threadIdx.x >> 7, warp = (threadIdx.x >> 5) & 3;
    const int lane = threadIdx.x & 31, wfull = threadIdx.x >> 5;
    const int nrank = SEG ? static_cast<int>(gridDim.x) / p.nh : 1, rank = SEG ? blockIdx.x % nrank : 0;
    const int h = SEG ? blockIdx.x / nrank : blockIdx.x, b = blockIdx.y;
    const int T = p.T, nh = p.nh;
    // headdim <= 64 and d_state <= 128 (multiples of 8): the tiles keep their full
    // size and the missing columns are zero-filled, so every product is unchanged.
    const int hdv = p.hd, nsv = p.N;
    constexpr uint32_t fmt = std::is_same<Th, __nv_bfloat16>::value ? 1u : 0u;
    float* vec = reinterpret_cast<float*>(smem + kVec);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kBar);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + kTmemSlot);
    const uint32_t sbase = smem_u32(smem);

    uint64_t* full = bars + 2;  // tiles of buffer 0 / 1 have landed (TMA)
    if (threadIdx.x == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        mbar_init(&full[0], 1);
        mbar_init(&full[1], 1);
        mbar_init(bars + 4, 1);
        fence_barrier_init();
    }
    double* carry = reinterpret_cast<double*>(smem + kCarry);
    float* bias_sm = reinterpret_cast<float*>(smem + kBias);
    if (GEN) {
        if (threadIdx.x < 64) {
            const int a = threadIdx.x;
            const float v = (a < p.n_angles && p.angle_state)
                                ? p.angle_state[(static_cast<long long>(b) * nh + h) * p.n_angles + a] : 0.0f;
            carry[a] = static_cast<double>(v);
        }
        const float* bsrc = half ? p.c_bias : p.b_bias;
        bias_sm[half * 128 + tid] = tid < nsv ? bsrc[static_cast<long long>(h) * nsv + tid] : 0.0f;
    }
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tslot;
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>(warp * 32) << 16);  // this warp's 32 lanes

    const Th* xg = static_cast<const Th*>(p.x);
    Th* yg = static_cast<Th*>(p.y);
    const Th* Kg = static_cast<const Th*>(p.K);
    const float Dv = p.Dh[h];
    const int nchunks = (T + CS - 1) / CS;
    // this CTA's chunks; every chunk walked (in either pass) has a number j of its own, which the two-deep
    // buffers and barrier phases go by: j0 is that of chunk c_lo in the full pass
    const int per_rank = SEG ? (nchunks + nrank - 1) / nrank : nchunks;
    const int c_lo = SEG ? min(nchunks, rank * per_rank) : 0, c_hi = SEG ? min(nchunks, c_lo + per_rank) : nchunks;
    const bool state_pass = SEG && c_lo < c_hi && c_hi < nchunks;
    const int j0 = state_pass ? c_hi - c_lo : 0;
    bool ok = true;

    // Per-row scalars of chunk c into stage `st`: inclusive cumsum of adt, scale, gamma.
    // Per-row adt, dt, trap of the next chunk (dt and trap with the row after it) are staged in
    // shared memory while the current chunk runs.  As register loads they were drained by every
    // proxy fence of the chunk (0.18 ms of 0.45 ms at 32 heads, where they are 128-byte-strided
    // words); a fence waits for 4-byte asynchronous copies too.  TMA copies are not waited for:
    // with nheads % 4 == 0 one thread fetches [129 rows x 4 heads] boxes; otherwise the copies
    // are issued where the next fence is furthest away.
    uint64_t* scf = bars + 4;
    const int hcol = h & 3;
    auto stage_scalars = [&](int c) {
        if (c >= c_hi) return;
        if (p.sc_tma) {
            if (threadIdx.x == 0) {
                mbar_expect_tx(scf, 3 * 129 * 16);
                tma_load_3d(smem + kStage, &p.tm_adt, scf, h & ~3, c * CS, b);
                tma_load_3d(smem + kStage + kStageArr, &p.tm_dt, scf, h & ~3, c * CS, b);
                tma_load_3d(smem + kStage + 2 * kStageArr, &p.tm_trap, scf, h & ~3, c * CS, b);
            }
        } else {
            if (threadIdx.x <= CS) {
                float* st = reinterpret_cast<float*>(smem + kStage) + threadIdx.x * 4 + hcol;
                const int t = c * CS + threadIdx.x;
                const long long th = (static_cast<long long>(b) * T + t) * nh + h;
                if (t < T) {
                    cp_async4(st, p.adt + th);
                    cp_async4(st + kStageArr / 4, p.dt + th);
                    cp_async4(st + 2 * kStageArr / 4, p.trap + th);
                } else {
                    st[0] = st[kStageArr / 4] = st[2 * kStageArr / 4] = 0.0f;
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
    };
    auto scalars = [&](int j) {
        const int st = j & 1;
        float* dA = vec + st * kVecSet;
        float* scl = dA + 128;
        float* gam = dA + 256;
        if (p.sc_tma) {
            ok = mbar_wait(scf, j & 1, p.status) && ok;
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();  // every thread's staged words of this chunk are in shared memory
        }
        const float* stg = reinterpret_cast<const float*>(smem + kStage) + hcol;
        const float a = stg[tid * 4], dtr = stg[kStageArr / 4 + tid * 4], g = dtr * stg[2 * kStageArr / 4 + tid * 4];
        const float s = g + stg[kStageArr / 4 + tid * 4 + 4] * (1.0f - stg[2 * kStageArr / 4 + tid * 4 + 4]);
        float run = a;
#pragma unroll
        for (int m = 1; m < 32; m <<= 1) {
            const float o = __shfl_up_sync(0xffffffffu, run, m);
            if (lane >= m) run += o;
        }
        // warp totals in the 112 spare bytes behind the first staging array
        float* wtot = reinterpret_cast<float*>(smem + kStage + 129 * 16);
        if (lane == 31) wtot[warp] = run;
        gam[tid] = g;
        scl[tid] = s;
        if (GEN) dA[512 + tid] = dtr;
        __syncthreads();
        const float w0 = wtot[0], w1 = wtot[1], w2 = wtot[2];
        const float off = (warp > 0 ? w0 : 0.0f) + (warp > 1 ? w1 : 0.0f) + (warp > 2 ? w2 : 0.0f);
        dA[tid] = run + off;
        dA[384 + tid] = (run + off) * kLog2e;
        // (the barrier ahead of the first MMA group publishes these rows)
    };


    // K and Q tiles of chunk c from the group-level rows (GEN only): TMA lands the raw Bn / Cn
    // rows of this head's group in the K / Q tiles and gen_apply rewrites them in place.
    // Thread (lane, warp w) owns the 16-byte pieces j = w and w + 8 of the rows lane,
    // lane + 32, lane + 64, lane + 96.  The angle of (row, a) is the angle entering the chunk
    // (f64, shared memory) plus an inclusive sum over the rows: a warp shuffle scan inside each
    // block of 32 rows and a running prefix over the four blocks, which the same thread owns.
    // this thread's angle velocities of the chunk that gen_apply rewrites next (loaded a
    // chunk ahead, like the per-row scalars)
    float4 velr[4][2];
    auto load_vel = [&](int c) {
        const int t0 = c * CS, nv = min(CS, T - t0), na = p.n_angles;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int j = wfull + 8 * q, row = lane + 32 * i;
                velr[i][q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (c < nchunks && 4 * j < na && row < nv)
                    velr[i][q] = __ldg(reinterpret_cast<const float4*>(
                        p.angle_vel + (static_cast<long long>(b) * T + t0 + row) * na + 4 * j));
            }
    };
    auto gen_apply = [&](int c, int buf) {
        const int t0 = c * CS, nv = min(CS, T - t0);
        const int na = p.n_angles;
        constexpr double kTwoPi64 = 6.283185307179586, kInvTwoPi64 = 0.15915494309189535;
        const bool rot0 = 4 * wfull < na, rot1 = 4 * (wfull + 8) < na;
        float ang[4][2][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = lane + 32 * i;
            const float dtr = row < nv ? vec[(c & 1) * kVecSet + 512 + row] : 0.0f;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                ang[i][q][0] = velr[i][q].x * dtr; ang[i][q][1] = velr[i][q].y * dtr;
                ang[i][q][2] = velr[i][q].z * dtr; ang[i][q][3] = velr[i][q].w * dtr;
            }
        }
        // inclusive sums over the 32 rows of each block: every value advances together
#pragma unroll
        for (int m = 1; m < 32; m <<= 1) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    if (q ? rot1 : rot0) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float o = __shfl_up_sync(0xffffffffu, ang[i][q][e], m);
                            if (lane >= m) ang[i][q][e] += o;
                        }
                    }
        }
        // entering angle + the blocks before; the chunk's total goes into the f64 carry
#pragma unroll
        for (int q = 0; q < 2; ++q)
            if (q ? rot1 : rot0) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int a = 4 * (wfull + 8 * q) + e;
                    const double cin = carry[a];
                    float run = static_cast<float>(cin), tot = 0.0f;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float bt = __shfl_sync(0xffffffffu, ang[i][q][e], 31);
                        ang[i][q][e] += run;
                        run += bt;
                        tot += bt;
                    }
                    double sacc = cin + static_cast<double>(tot);
                    sacc -= kTwoPi64 * floor(sacc * kInvTwoPi64);
                    __syncwarp();
                    if (lane == 0) carry[a] = sacc;
                }
            }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = lane + 32 * i;
            const bool rok = row < nv;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int j = wfull + 8 * q;
                const bool rot = q ? rot1 : rot0;
                float sn[4], cs[4];
                if (rot) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        // to [-pi, pi] before the fast sine / cosine
                        float x = ang[i][q][e];
                        const float turns = rintf(x * 0.15915494309189535f);
                        x = fmaf(turns, -6.2831854820251465f, x);
                        x = fmaf(turns, 1.7484555e-7f, x);
                        __sincosf(x, &sn[e], &cs[e]);
                    }
                }
                if (8 * j < nsv && rok) {
#pragma unroll
                    for (int which = 0; which < 2; ++which) {
                        uint4* pp = reinterpret_cast<uint4*>(smem + (which ? kQ0 : kK0) + buf * kQKStride +
                                                             sw_chunk(row, j));
                        const uint4 raw = *pp;
                        const uint32_t rw[4] = {raw.x, raw.y, raw.z, raw.w};
                        const float4 b0 = *reinterpret_cast<const float4*>(bias_sm + which * 128 + 8 * j);
                        const float4 b1 = *reinterpret_cast<const float4*>(bias_sm + which * 128 + 8 * j + 4);
                        const float bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
                        uint32_t ow[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float2 f = unpack2<Th>(rw[e]);
                            float v0 = f.x + bv[2 * e], v1 = f.y + bv[2 * e + 1];
                            if (rot) {
                                const float r0 = cs[e] * v0 - sn[e] * v1, r1 = sn[e] * v0 + cs[e] * v1;
                                v0 = r0; v1 = r1;
                            }
                            ow[e] = pack2<Th>(v0, v1);
                        }
                        *pp = make_uint4(ow[0], ow[1], ow[2], ow[3]);
                    }
                }
            }
        }
    };

    // One elected thread issues the five boxes of a chunk (Q and K: two 64-column sub-tiles
    // each, V: one); rows past the end of the sequence and columns past the head's width
    // arrive as zeros.
    auto issue_carry_q = [&](int c) {
        if (threadIdx.x == 0) {
            mbar_expect_tx(&full[0], kQKBytes);
#pragma unroll
            for (int sub = 0; sub < 2; ++sub)
                tma_load_4d(smem + kQ0 + sub * kSwSub, &p.tm_q, &full[0], 64 * sub, h, c * CS, b);
        }
    };
    auto issue_carry_kv = [&](int c) {
        if (threadIdx.x == 0) {
            mbar_expect_tx(&full[1], kQKBytes + kVBytes);
#pragma unroll
            for (int sub = 0; sub < 2; ++sub)
                tma_load_4d(smem + kCarryK + sub * kSwSub, &p.tm_k, &full[1], 64 * sub, h, c * CS, b);
            tma_load_4d(smem + kCarryV, &p.tm_v, &full[1], 0, h, c * CS, b);
        }
    };
    auto issue_kv = [&](int c, int j) {  // state pass
        if (threadIdx.x == 0) {
            const int buf = j & 1, t0 = c * CS;
            mbar_expect_tx(&full[buf], kQKBytes + kVBytes);
#pragma unroll
            for (int sub = 0; sub < 2; ++sub)
                tma_load_4d(smem + kK0 + buf * kQKStride + sub * kSwSub, &p.tm_k, &full[buf], 64 * sub, h, t0, b);
            tma_load_4d(smem + kV0 + buf * kVStride, &p.tm_v, &full[buf], 0, h, t0, b);
        }
    };
    auto issue_tiles = [&](int c, int j) {
        if (threadIdx.x == 0) {
            const int buf = LEAN ? 0 : j & 1, t0 = c * CS;
            const int hq = GEN ? h / (nh / p.ng) : h;
            mbar_expect_tx(&full[buf], 2 * kQKBytes + kVBytes);
#pragma unroll
            for (int sub = 0; sub < 2; ++sub) {
                tma_load_4d(smem + kQ0 + buf * kQKStride + sub * kSwSub, &p.tm_q, &full[buf], 64 * sub, hq, t0, b);
                tma_load_4d(smem + kK0 + buf * kQKStride + sub * kSwSub, &p.tm_k, &full[buf], 64 * sub, hq, t0, b);
            }
            tma_load_4d(smem + kV0 + buf * kVStride, &p.tm_v, &full[buf], 0, h, t0, b);
        }
    };
    // 16-bit copy of this thread's state row (and the remainders): the B operand of Y2
    uint32_t s_lo[TURNS ? 16 : 1], m_lo[TURNS ? 2 : 1][16];  // TURNS: remainders that wait for their turn
    auto copy_state = [&](const float* sv) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            uint32_t w[4], lo[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                w[i] = pack2<Th>(sv[8 * j + 2 * i], sv[8 * j + 2 * i + 1]);
                if (CARRY) {
                    const float2 r = unpack2<Th>(w[i]);
                    lo[i] = pack2<Th>(sv[8 * j + 2 * i] - r.x, sv[8 * j + 2 * i + 1] - r.y);
                }
            }
            *reinterpret_cast<uint4*>(smem + kS + sw_chunk(tid, half * 4 + j)) = make_uint4(w[0], w[1], w[2], w[3]);
            if constexpr (TURNS) {
#pragma unroll
                for (int i = 0; i < 4; ++i) s_lo[4 * j + i] = lo[i];
            } else if (CARRY) {
                *reinterpret_cast<uint4*>(smem + kSlo + sw_chunk(tid, half * 4 + j)) =
                    make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
        }
    };
    // the carried state as this thread's row: h + dt_0 (1 - trap_0) k_prev v_prev^T
    auto carried_state = [&](float* sv) {
        const long long bh = static_cast<long long>(b) * nh + h, th0 = static_cast<long long>(b) * T * nh + h;
        const float kc = tid < nsv ? p.dt[th0] * (1.0f - p.trap[th0]) * p.k_state[bh * nsv + tid] : 0.0f;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            const int pp = half * 32 + i;
            sv[i] = pp < hdv && tid < nsv ? fmaf(kc, p.v_state[bh * hdv + pp], p.ssm_state[(bh * hdv + pp) * nsv + tid])
                                          : 0.0f;
        }
    };
    // and as what the first chunk walked in full starts from
    auto enter_state = [&]() {
        float sv[32];
        carried_state(sv);
        tmem_st32(lane_addr + cS + half * 32, sv);
        copy_state(sv);
        fence_proxy_async();
    };
    // w o V of chunk j (and its remainders; TURNS: which of the three): the B operand of the state update
    auto weigh_v = [&](const float* dA, const float* scl, int nv, uint32_t tV, int turn) {
        const float wt = tid < nv ? ex2((dA[nv - 1] - dA[tid]) * kLog2e) * scl[tid] : 0.0f;
#pragma unroll
        for (int jj = half * (HD / 16); jj < (half + 1) * (HD / 16); ++jj) {
            const uint4 v = *reinterpret_cast<const uint4*>(smem + tV + sw_chunk(tid, jj));
            uint32_t w4[4] = {v.x, v.y, v.z, v.w}, lo[4], rest[4];
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) {
                const float2 f = unpack2<Th>(w4[q4]);
                w4[q4] = pack2<Th>(f.x * wt, f.y * wt);
                if (CARRY) {
                    const float2 hi = unpack2<Th>(w4[q4]), r = make_float2(f.x * wt - hi.x, f.y * wt - hi.y);
                    lo[q4] = pack2<Th>(r.x, r.y);
                    const float2 mid = unpack2<Th>(lo[q4]);
                    rest[q4] = pack2<Th>(r.x - mid.x, r.y - mid.y);
                }
            }
            if (TURNS && turn > 0) {
#pragma unroll
                for (int q4 = 0; q4 < 4; ++q4) w4[q4] = turn == 1 ? lo[q4] : rest[q4];
            }
            *reinterpret_cast<uint4*>(smem + kVw + sw_chunk(tid, jj)) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
            if (CARRY && !TURNS) {
                *reinterpret_cast<uint4*>(smem + kVwLo + sw_chunk(tid, jj)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                *reinterpret_cast<uint4*>(smem + kVwRest + sw_chunk(tid, jj)) = make_uint4(rest[0], rest[1], rest[2], rest[3]);
            }
        }
    };
    auto decay_state = [&](float e_end) {  // S^T row `tid` (state index n = tid) *= exp(dA_end)
        float sv[32];
        tmem_ld32(lane_addr + cS + half * 32, sv);
#pragma unroll
        for (int i = 0; i < 32; ++i) sv[i] *= e_end;
        tmem_st32(lane_addr + cS + half * 32, sv);
    };
    auto update_state = [&](uint32_t tK, bool accumulate) {  // S^T += K^T (w o V); one thread
        const uint32_t idS = instr_desc(fmt, 1, 1, 64);
#pragma unroll
        for (int k = 0; k < CS / 16; ++k)  // M = n, N = p, K = t
            mma(tmem + cS, desc_sw_mn(sbase + tK, k), desc_sw_mn(sbase + kVw, k), idS, accumulate || k > 0);
        if (CARRY && !TURNS) {
#pragma unroll
            for (int k = 0; k < CS / 16; ++k)
                mma(tmem + cS, desc_sw_mn(sbase + tK, k), desc_sw_mn(sbase + kVwLo, k), idS, true);
#pragma unroll
            for (int k = 0; k < CS / 16; ++k)
                mma(tmem + cS, desc_sw_mn(sbase + tK, k), desc_sw_mn(sbase + kVwRest, k), idS, true);
        }
    };

    if constexpr (SEG) {
        float tot = 0.0f;  // sum of dA over this CTA's chunks
        if (state_pass) {
            if (CARRY && rank == 0) {
                float sv[32];
                carried_state(sv);
                tmem_st32(lane_addr + cS + half * 32, sv);
            }
            if (CARRY) issue_carry_kv(c_lo);
            else issue_kv(c_lo, 0);
            stage_scalars(c_lo);
            for (int c = c_lo; c < c_hi; ++c) {
                const int j = c - c_lo, nv = min(CS, T - c * CS);
                const uint32_t tK = CARRY ? kCarryK : kK0 + (j & 1) * kQKStride;
                const uint32_t tV = CARRY ? kCarryV : kV0 + (j & 1) * kVStride;
                const float* dA = vec + (j & 1) * kVecSet;
                if (!CARRY && c + 1 < c_hi) issue_kv(c + 1, j + 1);
                scalars(j);
                ok = mbar_wait(CARRY ? &full[1] : &full[j & 1], CARRY ? j & 1 : (j >> 1) & 1, p.status) && ok;
                __syncthreads();  // the per-row vectors of every row
                stage_scalars(c + 1);
                weigh_v(dA, dA + 128, nv, tV, 0);
                const bool have = c > c_lo || (CARRY && rank == 0);
                if (have) decay_state(ex2(dA[nv - 1] * kLog2e));
                tot += dA[nv - 1];
                fence_proxy_async();
                fence_before();
                __syncthreads();
                if (threadIdx.x == 0) {
                    fence_after();
                    update_state(tK, have);
                    commit(&bars[1]);
                }
                ok = mbar_wait(&bars[1], j & 1, p.status) && ok;
                fence_after();
                if (CARRY && c + 1 < c_hi) issue_carry_kv(c + 1);
            }
        }
        // the full pass's first tiles travel while the states are exchanged
        if (c_lo < c_hi) {
            if (CARRY) {
                issue_carry_q(c_lo);
                issue_carry_kv(c_lo);
            } else {
                issue_tiles(c_lo, j0);
            }
            stage_scalars(c_lo);
        }
        if (state_pass) {
            float sv[32];
            tmem_ld32(lane_addr + cS + half * 32, sv);
#pragma unroll
            for (int i = 0; i < 8; ++i)
                *reinterpret_cast<float4*>(smem + kLoc + tid * 256 + half * 128 + i * 16) =
                    make_float4(sv[4 * i], sv[4 * i + 1], sv[4 * i + 2], sv[4 * i + 3]);
            if (threadIdx.x == 0) *reinterpret_cast<float*>(smem + kTot) = tot * kLog2e;
        }
        cluster_sync();
        if (c_lo < c_hi && rank > 0) {
            float sv[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) sv[i] = 0.0f;
            float between = 0.0f;  // log2 of the decay of the CTAs between q and this one
            for (int q = rank - 1; q >= 0; --q) {
                const float f = ex2(between);
                const uint32_t src = cluster_addr(sbase + kLoc + tid * 256 + half * 128, q);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 v = ld_cluster4(src + i * 16);
                    sv[4 * i] = fmaf(f, v.x, sv[4 * i]);
                    sv[4 * i + 1] = fmaf(f, v.y, sv[4 * i + 1]);
                    sv[4 * i + 2] = fmaf(f, v.z, sv[4 * i + 2]);
                    sv[4 * i + 3] = fmaf(f, v.w, sv[4 * i + 3]);
                }
                between += ld_cluster1(cluster_addr(sbase + kTot, q));
            }
            tmem_st32(lane_addr + cS + half * 32, sv);
            copy_state(sv);
            fence_proxy_async();  // (published by the barriers ahead of the first MMA group)
        }
        // ahead of the barrier: past it the CTA of the last chunk may already replace the carried state in place
        if (CARRY && rank == 0) enter_state();
        cluster_sync();  // nobody reads this CTA's shared memory any more
    } else {
        if (CARRY && !LEAN) {
            issue_carry_q(0);
            issue_carry_kv(0);
        } else {
            issue_tiles(0, 0);
        }
        stage_scalars(0);
        if (GEN) load_vel(0);
        if (CARRY) enter_state();
    }

    for (int c = c_lo; c < c_hi; ++c) {
        const int i0 = c - c_lo, j = j0 + i0;
        const int t0 = c * CS, nv = min(CS, T - t0);
        const bool row_ok = tid < nv;
        const float* dA = vec + (j & 1) * kVecSet;
        const float* scl = dA + 128;
        const float* gam = dA + 256;
        const uint32_t tQ = kQ0 + (CARRY ? 0u : (j & 1) * kQKStride);
        const uint32_t tK = CARRY && !LEAN ? kCarryK : kK0 + (j & 1) * kQKStride;
        const uint32_t tV = CARRY && !LEAN ? kCarryV : kV0 + (j & 1) * kVStride;
        // ---- 1. copies of the next chunk's tiles into the other buffers (their last readers,
        //         the MMAs of chunk c - 1, have completed); per-row scalars; this chunk's tiles ----
        if (!CARRY && !LEAN && c + 1 < c_hi) issue_tiles(c + 1, j + 1);
        scalars(j);
        if (LEAN) {
            ok = mbar_wait(&full[0], j & 1, p.status) && ok;
        } else if (CARRY) {
            ok = mbar_wait(&full[0], i0 & 1, p.status) && ok;
            ok = mbar_wait(&full[1], j & 1, p.status) && ok;
        } else {
            ok = mbar_wait(&full[j & 1], (j >> 1) & 1, p.status) && ok;
        }
        if (GEN) {
            gen_apply(c, c & 1);
            fence_proxy_async();  // the rewritten K / Q pieces, before the tensor core reads them
        }
        fence_before();
        __syncthreads();
        // A proxy fence waits for this thread's outstanding asynchronous copies (measured:
        // 1500 cycles when the staged scalars were issued ahead of one), so they start here,
        // with the MMA wait and the mask stage between them and the next fence.
        stage_scalars(c + 1);
        // ---- 2. G = Q K^T (and Y2 = Q S_in^T for c > 0) ----
        if (threadIdx.x == 0) {
            fence_after();
            const uint32_t idG = instr_desc(fmt, 0, 0, 128), idY = instr_desc(fmt, 0, 1, 64);
#pragma unroll
            for (int k = 0; k < NS / 16; ++k)
                mma(tmem + cG, desc_sw_k(sbase + tQ, k), desc_sw_k(sbase + tK, k), idG, k > 0);
            if (CARRY || c > 0) {
#pragma unroll
                for (int k = 0; k < NS / 16; ++k)  // N = p, K = n
                    mma(tmem + cY2, desc_sw_k(sbase + tQ, k), desc_sw_mn(sbase + kS, k), idY, k > 0);
            }
            if (CARRY && !LEAN) {
#pragma unroll
                for (int k = 0; k < NS / 16; ++k)
                    mma(tmem + cY2, desc_sw_k(sbase + tQ, k), desc_sw_mn(sbase + kSlo, k), idY, true);
            }
            commit(&bars[0]);
        }
        ok = mbar_wait(&bars[0], TURNS ? 0 : i0 & 1, p.status) && ok;
        fence_after();
        if constexpr (TURNS) {  // Y2 += Q S_lo, S_lo where the state copy was
#pragma unroll
            for (int q = 0; q < 4; ++q)
                *reinterpret_cast<uint4*>(smem + kS + sw_chunk(tid, half * 4 + q)) =
                    make_uint4(s_lo[4 * q], s_lo[4 * q + 1], s_lo[4 * q + 2], s_lo[4 * q + 3]);
            fence_proxy_async();
            fence_before();
            __syncthreads();
            if (threadIdx.x == 0) {
                fence_after();
                const uint32_t idY = instr_desc(fmt, 0, 1, 64);
#pragma unroll
                for (int k = 0; k < NS / 16; ++k)
                    mma(tmem + cY2, desc_sw_k(sbase + tQ, k), desc_sw_mn(sbase + kS, k), idY, true);
                commit(&bars[0]);
            }
            ok = mbar_wait(&bars[0], 1, p.status) && ok;
            fence_after();
        }
        if (CARRY && !LEAN && c + 1 < c_hi) issue_carry_q(c + 1);
        // ---- 3. decay / causal mask -> M (over the Q tile); w o V (over the old state
        //         copy); rescale the running state ----
        {
            weigh_v(dA, scl, nv, tV, 0);
            const float* dAl = dA + 384;  // dA * log2(e)
            const float dAlt = dAl[tid], gt = gam[tid];
            // One 32-column block of row `tid`.  Blocks left of the diagonal block need no
            // mask; rows and columns past the end of the sequence need none either (their
            // V rows are zero and their y rows are never stored).
            auto mask_block = [&](auto diag_tag, int q4) {
                constexpr bool DIAG = decltype(diag_tag)::value;
                float g[32];
                tmem_ld32(lane_addr + cG + q4 * 32, g);
                uint32_t packed[16], rest[16];
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    const float4 da4 = *reinterpret_cast<const float4*>(dAl + q4 * 32 + i);
                    const float4 sc4 = *reinterpret_cast<const float4*>(scl + q4 * 32 + i);
                    const float dav[4] = {da4.x, da4.y, da4.z, da4.w}, scv[4] = {sc4.x, sc4.y, sc4.z, sc4.w};
                    float m[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        float v = g[i + u] * scv[u] * ex2(dAlt - dav[u]);
                        if (DIAG) {
                            const int s = q4 * 32 + i + u;
                            if (s > tid) v = 0.0f;
                            else if (s == tid) v = fmaf(g[i + u], gt, Dv);
                        }
                        m[u] = v;
                    }
                    packed[i / 2] = pack2<Th>(m[0], m[1]);
                    packed[i / 2 + 1] = pack2<Th>(m[2], m[3]);
                    if (CARRY) {
                        const float2 r0 = unpack2<Th>(packed[i / 2]), r1 = unpack2<Th>(packed[i / 2 + 1]);
                        rest[i / 2] = pack2<Th>(m[0] - r0.x, m[1] - r0.y);
                        rest[i / 2 + 1] = pack2<Th>(m[2] - r1.x, m[3] - r1.y);
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    *reinterpret_cast<uint4*>(smem + kM + sw_chunk(tid, q4 * 4 + j)) =
                        make_uint4(packed[4 * j], packed[4 * j + 1], packed[4 * j + 2], packed[4 * j + 3]);
                if constexpr (TURNS) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        if (q4 & 1) m_lo[1][j] = rest[j];
                        else m_lo[0][j] = rest[j];
                    }
                } else if (CARRY) {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        *reinterpret_cast<uint4*>(smem + kMlo + sw_chunk(tid, q4 * 4 + j)) =
                            make_uint4(rest[4 * j], rest[4 * j + 1], rest[4 * j + 2], rest[4 * j + 3]);
                }
            };
            if constexpr (TURNS) {
#pragma unroll
                for (int j = 0; j < 16; ++j) m_lo[0][j] = m_lo[1][j] = 0;
            }
            for (int q4 = 2 * half; q4 < 2 * half + 2; ++q4) {
                if (q4 > warp) {  // wholly above the diagonal for every row of this warp
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        *reinterpret_cast<uint4*>(smem + kM + sw_chunk(tid, q4 * 4 + j)) = make_uint4(0, 0, 0, 0);
                        if (CARRY && !TURNS)
                            *reinterpret_cast<uint4*>(smem + kMlo + sw_chunk(tid, q4 * 4 + j)) = make_uint4(0, 0, 0, 0);
                    }
                } else if (q4 == warp) {
                    mask_block(std::true_type{}, q4);
                } else {
                    mask_block(std::false_type{}, q4);
                }
            }
            if (CARRY || c > 0) decay_state(ex2(dA[nv - 1] * kLog2e));
            if constexpr (TURNS) {  // Y2 takes its rows' decay here and M V on top
                const float e_t = ex2(dA[tid] * kLog2e);
                float y2[32];
                tmem_ld32(lane_addr + cY2 + half * 32, y2);
#pragma unroll
                for (int i = 0; i < 32; ++i) y2[i] *= e_t;
                tmem_st32(lane_addr + cY2 + half * 32, y2);
            }
        }
        fence_proxy_async();
        fence_before();
        __syncthreads();
        // register loads issued here have the longest run before the next proxy fence
        if (GEN) load_vel(c + 1);
        // ---- 4. Y1 = M V ;  S^T += K^T (w o V) ----
        if (threadIdx.x == 0) {
            fence_after();
            const uint32_t idY = instr_desc(fmt, 0, 1, 64);
#pragma unroll
            for (int k = 0; k < CS / 16; ++k)  // N = p, K = s
                mma(tmem + (TURNS ? cY2 : cY1), desc_sw_k(sbase + kM, k), desc_sw_mn(sbase + tV, k), idY, TURNS || k > 0);
            if (CARRY && !TURNS) {
#pragma unroll
                for (int k = 0; k < CS / 16; ++k)
                    mma(tmem + cY1, desc_sw_k(sbase + kMlo, k), desc_sw_mn(sbase + tV, k), idY, true);
            }
            update_state(tK, CARRY || c > 0);
            commit(&bars[1]);
        }
        ok = mbar_wait(&bars[1], (TURNS ? 3 * j : j) & 1, p.status) && ok;
        fence_after();
        if constexpr (TURNS) {
            // the remainders' turns: M_lo V and K^T (w o V)_lo, then K^T (w o V)_rest
#pragma unroll
            for (int turn = 1; turn < 3; ++turn) {
                weigh_v(dA, scl, nv, tV, turn);
                if (turn == 1) {
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        *reinterpret_cast<uint4*>(smem + kM + sw_chunk(tid, half * 8 + q)) =
                            make_uint4(m_lo[q / 4][4 * (q % 4)], m_lo[q / 4][4 * (q % 4) + 1], m_lo[q / 4][4 * (q % 4) + 2],
                                       m_lo[q / 4][4 * (q % 4) + 3]);
                }
                fence_proxy_async();
                fence_before();
                __syncthreads();
                if (threadIdx.x == 0) {
                    fence_after();
                    const uint32_t idY = instr_desc(fmt, 0, 1, 64);
                    if (turn == 1) {
#pragma unroll
                        for (int k = 0; k < CS / 16; ++k)
                            mma(tmem + cY2, desc_sw_k(sbase + kM, k), desc_sw_mn(sbase + tV, k), idY, true);
                    }
                    update_state(tK, true);
                    commit(&bars[1]);
                }
                ok = mbar_wait(&bars[1], (3 * j + turn) & 1, p.status) && ok;
                fence_after();
            }
        }
        if (CARRY && !LEAN && c + 1 < c_hi) issue_carry_kv(c + 1);
        if (LEAN && c + 1 < c_hi) issue_tiles(c + 1, j + 1);
        // ---- 5. epilogue: y row; 16-bit copy of the new state for the next chunk ----
        {
            const float e_t = ex2(dA[tid] * kLog2e);
            const int q2 = half;
            float y1[32], y2[32];
            if (TURNS) {
                tmem_ld32(lane_addr + cY2 + q2 * 32, y1);
            } else if (CARRY || c > 0) {
                tmem_ld32x2(lane_addr + cY1 + q2 * 32, y1, lane_addr + cY2 + q2 * 32, y2);
#pragma unroll
                for (int i = 0; i < 32; ++i) y1[i] = fmaf(e_t, y2[i], y1[i]);
            } else {
                tmem_ld32(lane_addr + cY1 + q2 * 32, y1);
            }
            uint4 yo[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                yo[j] = make_uint4(pack2<Th>(y1[8 * j], y1[8 * j + 1]), pack2<Th>(y1[8 * j + 2], y1[8 * j + 3]),
                                   pack2<Th>(y1[8 * j + 4], y1[8 * j + 5]), pack2<Th>(y1[8 * j + 6], y1[8 * j + 7]));
            float sv[32];
            tmem_ld32(lane_addr + cS + q2 * 32, sv);
            if (c + 1 < c_hi) {
                copy_state(sv);
            } else if (c + 1 == nchunks && p.ssm_state) {  // final state [b, h, p, n], n = tid
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (q2 * 32 + i < hdv && tid < nsv)
                        p.ssm_state[((static_cast<long long>(b) * nh + h) * hdv + q2 * 32 + i) * nsv + tid] = sv[i];
            }
            fence_proxy_async();  // the state copy, before the next chunk's Y2 reads it
            // y rows leave after the fence: a proxy fence waits for the thread's outstanding
            // global stores too, and the next one is most of a chunk away
            if (row_ok) {
                Th* yrow = yg + (static_cast<long long>(b) * T + t0 + tid) * nh * hdv + h * hdv + q2 * 32;
                if (p.wide_y) {  // headdim a multiple of 16, y 32-byte aligned
#pragma unroll
                    for (int j = 0; j < 4; j += 2)
                        if (q2 * 32 + 8 * j < hdv) store32b(yrow + 8 * j, yo[j], yo[j + 1], true);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (q2 * 32 + 8 * j < hdv) *reinterpret_cast<uint4*>(yrow + 8 * j) = yo[j];
                }
            }
        }
        // no barrier here: the next chunk writes the other set of per-row vectors, and every tile,
        // TMEM column and the state copy it touches is ordered by its own barriers
    }
    fence_before();
    __syncthreads();
    fence_after();
    // last inputs of the window (kernels/mamba3_chunked.cu:289-330)
    if (c_lo < c_hi && c_hi == nchunks) {
        const long long last = static_cast<long long>(b) * T + (T - 1);
        if (GEN) {
            // the last K row is still in its tile; fold the last chunk's sums into the angle
            const int lr = T - 1 - (nchunks - 1) * CS;
            if (p.k_state && half == 0 && tid < nsv)
                p.k_state[(static_cast<long long>(b) * nh + h) * nsv + tid] =
                    to_f(*reinterpret_cast<const Th*>(smem + kK0 + ((nchunks - 1) & 1) * kQKStride +
                                                     sw_chunk(lr, tid >> 3) + (tid & 7) * 2));
            if (p.angle_state && threadIdx.x < p.n_angles)
                p.angle_state[(static_cast<long long>(b) * nh + h) * p.n_angles + threadIdx.x] =
                    static_cast<float>(carry[threadIdx.x]);
        } else if (p.k_state && half == 0 && tid < nsv)
            p.k_state[(static_cast<long long>(b) * nh + h) * nsv + tid] = to_f(Kg[(last * nh + h) * nsv + tid]);
        if (p.v_state && half == 0 && tid < hdv)
            p.v_state[(static_cast<long long>(b) * nh + h) * hdv + tid] = to_f(xg[last * nh * hdv + h * hdv + tid]);
    }
    __syncthreads();
    if (threadIdx.x < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    (void)ok;
}

}  // namespace tc

// CTAs of a cluster that share one (sample, head), by estimated time: a chunk takes one CTA `full` us
// undivided, `pair` in a cluster of two and `many` in a larger one; the exchange takes `fixed` a rank.  A wave
// is one CTA per SM, less what clusters of 4 and 8 cannot place.  A division that gains less than 5 % is not
// taken.
int m3_cluster_ranks(int heads, int nchunks, double full, double pair, double many, double fixed) {
    int best = 1;
    double cost = static_cast<double>((heads + 147) / 148) * nchunks * full;
    const int cap[4] = {148, 148, 144, 128};
    for (int i = 1; i < 4; ++i) {
        const int r = 1 << i, per = (nchunks + r - 1) / r;
        if (r > nchunks) break;
        const double c = static_cast<double>((heads * r + cap[i] - 1) / cap[i]) * (per * (r == 2 ? pair : many) + r * fixed);
        if (c < 0.95 * cost) {
            cost = c;
            best = r;
        }
    }
    return best;
}

// Two CTAs per SM (LEAN) or one: 5.9 us a chunk for both together against 3.7 for one, which has its next tiles on the
// way while it works.  16 chunks of 64 x 128 in us, one / two per SM: 152 pairs 127 and 99, 256 131 and 104, 296 148
// and 132, 352 191 and 188, 384 192 and 193, 440 220 and 223, 464 284 and 232, 512 256 and 198, 592 309 and 264, 896 443
// and 362.  So one wave of one CTA per SM stays, and three nearly full ones.
static bool m3_two_per_sm(int pairs) { return pairs > 148 && (pairs <= 360 || pairs > 3 * 148); }

// The same for carried windows, in us: 152 pairs x 256 steps 49 and 42, 256 62 and 47, 512 121 and 90; x 1024 steps 123
// and 108, 126 and 110, 247 and 214; in the third wave of one CTA per SM, 384 pairs, 91 and 86 x 256 but 186 and 202 x
// 1024, so there only up to two chunks.  256 pairs x 21 steps 33 and 23.
static bool m3_two_carried_per_sm(int pairs, int nchunks) {
    return pairs > 148 && (pairs <= 2 * 148 || pairs > 3 * 148 || nchunks <= 2);
}

cudaError_t launch_cluster(const void* fn, dim3 grid, dim3 block, size_t smem, cudaStream_t st, int ranks, void** args) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at;
    memset(&at, 0, sizeof(at));
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = ranks;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, fn, args);
}

int m3_configure(Ctx* c) {
    const void* fns[8] = {reinterpret_cast<const void*>(tc::m3_ssd_fwd_tc_kernel<__nv_bfloat16, false, false, false, false>),
                          reinterpret_cast<const void*>(tc::m3_ssd_fwd_tc_kernel<__half, false, false, false, false>),
                          reinterpret_cast<const void*>(tc::m3_ssd_fwd_tc_kernel<__nv_bfloat16, true, false, false, false>),
                          reinterpret_cast<const void*>(tc::m3_ssd_fwd_tc_kernel<__half, true, false, false, false>),
                          reinterpret_cast<const void*>(tc::m3_ssd_fwd_tc_kernel<__nv_bfloat16, false, true, false, false>),
                          reinterpret_cast<const void*>(tc::m3_ssd_fwd_tc_kernel<__nv_bfloat16, false, false, true, false>),
                          reinterpret_cast<const void*>(tc::m3_ssd_fwd_tc_kernel<__half, false, false, true, false>),
                          reinterpret_cast<const void*>(tc::m3_ssd_fwd_tc_kernel<__nv_bfloat16, false, true, true, false>)};
    for (const void* fn : fns)
        MB200_CUDA_CHECK(c, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, tc::kSmem));
    const void* lean_fns[3] = {reinterpret_cast<const void*>(tc::m3_ssd_fwd_tc_kernel<__nv_bfloat16, false, true, false, true>),
                               reinterpret_cast<const void*>(tc::m3_ssd_fwd_tc_kernel<__nv_bfloat16, false, false, false, true>),
                               reinterpret_cast<const void*>(tc::m3_ssd_fwd_tc_kernel<__half, false, false, false, true>)};
    for (const void* fn : lean_fns) {
        MB200_CUDA_CHECK(c, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, tc::lean::kSmem));
        MB200_CUDA_CHECK(c, cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    }
    return MAMBA_B200_OK;
}

// Eight rows a warp share one K / Q load and one butterfly; two rows a warp when that leaves
// fewer than eight warps per SM (the step's chain, not the arithmetic, is then the time).
template <typename Tact, int NI, int R, bool PART>
static void launch_seq_rows(const M3Params& p, cudaStream_t st) {
    const int warps = min(8, (p.hd + R - 1) / R);
    const dim3 grid(p.nh, p.B, (p.hd + R * warps - 1) / (R * warps));
    m3_ssd_seq_kernel<Tact, NI, R, PART><<<grid, warps * 32, 0, st>>>(p);
    if (grid.z > 1 && p.k_state) m3_seq_kstate_kernel<Tact><<<dim3(p.nh, p.B), 128, 0, st>>>(p);
}
template <typename Tact>
static void launch_seq(const M3Params& p, int sms, cudaStream_t st) {
    const bool few = static_cast<long long>(p.B) * p.nh * ((p.hd + 7) / 8) < 8LL * sms, part = p.N % 32 != 0;
#define MB200_SEQ(NI, R)                                               \
    do {                                                               \
        if (part) launch_seq_rows<Tact, NI, R, true>(p, st);           \
        else launch_seq_rows<Tact, NI, R, false>(p, st);               \
    } while (0)
    if (few) {
        if (p.N <= 32) MB200_SEQ(1, 2);
        else if (p.N <= 64) MB200_SEQ(2, 2);
        // (96 states in three pieces: 36 us for 24 at 1 x 64 steps x 4 heads)
        else if (p.N < 128) launch_seq_rows<Tact, 4, 2, true>(p, st);
        else launch_seq_rows<Tact, 4, 2, false>(p, st);
    } else if (p.N <= 32) MB200_SEQ(1, 8);
    else if (p.N <= 64) MB200_SEQ(2, 8);
    else if (p.N <= 96) MB200_SEQ(3, 8);  // (8 x 64 steps x 32 heads, 96 states: 59 us for 93 in four pieces)
    else MB200_SEQ(4, 8);
#undef MB200_SEQ
}

}  // namespace mb200

using namespace mb200;

// A carried window of at most this many steps takes the sequential kernel: a 128-row chunk costs the tensor-core kernel the
// same time whether it holds 1 step or 128 (15 us at 4 heads, 22 at 150 to 296 pairs, 41 to 45 at 297 to 592), and the
// sequential kernel reaches that after 30 steps at 4 heads and 18 to 21 at 150 to 296 pairs of 48 x 128.  At 64 x 128 it
// does after 12 to 17 (16 steps of 256 pairs 28 and 23 us, 20 of 512 66 and 45), but it keeps an infinite input to its own
// step and row, where 0 * infinity in the chunk's masked products reaches all of them: the line stays for every size.
constexpr int kCarrySeqSteps = 20;

extern "C" MAMBA_B200_API int mamba_b200_m3_ssd_fwd(void* handle, void* stream,
                                                    const mamba_b200_m3_ssd_args* ap) {
    Ctx* c = static_cast<Ctx*>(handle);
    if (!c) return MAMBA_B200_ERR_ARG;
    if (!ap) return fail(c, MAMBA_B200_ERR_ARG, "m3_ssd_fwd: null args");
    const mamba_b200_m3_ssd_args& a = *ap;
    if (!dtype_ok(a.dtype)) return fail(c, MAMBA_B200_ERR_ARG, "m3_ssd_fwd: bad dtype %d", a.dtype);
    if (a.B < 0 || a.T < 0 || a.nh <= 0 || a.hd <= 0 || a.N <= 0)
        return fail(c, MAMBA_B200_ERR_ARG, "m3_ssd_fwd: bad dims");
    if (a.hd > 1024 || a.N > 128)
        return fail(c, MAMBA_B200_ERR_SHAPE, "m3_ssd_fwd: headdim %d > 1024 or d_state %d > 128", a.hd, a.N);
    if (a.B == 0 || a.T == 0) return MAMBA_B200_OK;
    if (a.B > 65535) return fail(c, MAMBA_B200_ERR_SHAPE, "m3_ssd_fwd: batch %d > 65535", a.B);
    const bool gen = a.Bn != nullptr;
    if (!a.x || (!gen && (!a.K || !a.Q)) || !a.dt || !a.trap || !a.adt || !a.Dh || !a.y)
        return fail(c, MAMBA_B200_ERR_ARG, "m3_ssd_fwd: null required pointer");
    if (gen) {
        if (!a.Cn || !a.b_bias || !a.c_bias || a.ng <= 0 || a.nh % a.ng != 0 || a.n_angles < 0 ||
            (a.n_angles > 0 && !a.angle_vel))
            return fail(c, MAMBA_B200_ERR_ARG, "m3_ssd_fwd: K/Q generation needs Bn, Cn, both biases, ngroups "
                                                "dividing nheads and angle_vel when n_angles > 0");
        if (a.n_angles % 4 != 0 || 2 * a.n_angles > a.N)
            return fail(c, MAMBA_B200_ERR_SHAPE, "m3_ssd_fwd: n_angles %d must be a multiple of 4 and <= d_state / 2",
                        a.n_angles);
    }
    if (a.carry_in && (!a.ssm_state || !a.k_state || !a.v_state))
        return fail(c, MAMBA_B200_ERR_ARG, "m3_ssd_fwd: carry_in needs all three state buffers");
    M3Params p;
    memset(&p, 0, sizeof(p));
    p.x = a.x; p.K = a.K; p.Q = a.Q; p.dt = a.dt; p.trap = a.trap; p.adt = a.adt; p.Dh = a.Dh; p.y = a.y;
    p.ssm_state = a.ssm_state; p.k_state = a.k_state; p.v_state = a.v_state;
    p.B = a.B; p.T = a.T; p.nh = a.nh; p.hd = a.hd; p.N = a.N; p.carry_in = a.carry_in;
    p.Bn = a.Bn; p.Cn = a.Cn; p.b_bias = a.b_bias; p.c_bias = a.c_bias; p.angle_vel = a.angle_vel;
    p.angle_state = a.angle_state; p.ng = a.ng; p.n_angles = a.n_angles;
    p.status = c->d_status;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
    bool tensor_core = a.dtype != MAMBA_B200_F32 && a.hd <= tc::HD && a.hd % 8 == 0 && a.N <= tc::NS &&
                       a.N % 8 == 0 && (!a.carry_in || (!gen && a.dtype == MAMBA_B200_BF16 && a.T > kCarrySeqSteps)) &&
                       !a.force_sequential && al16(a.x) && al16(a.y) &&
                       (gen ? al16(a.Bn) && al16(a.Cn) && al16(a.angle_vel) : al16(a.K) && al16(a.Q));
    // the tile maps; when the driver refuses one (no encoder, a stride beyond its range) the
    // sequential kernel takes the call
    tensor_core = tensor_core &&
                  make_tmap_head_tile(c, &p.tm_q, a.dtype, gen ? a.Cn : a.Q, a.N, gen ? a.ng : a.nh, a.T, a.B) &&
                  make_tmap_head_tile(c, &p.tm_k, a.dtype, gen ? a.Bn : a.K, a.N, gen ? a.ng : a.nh, a.T, a.B) &&
                  make_tmap_head_tile(c, &p.tm_v, a.dtype, a.x, a.hd, a.nh, a.T, a.B);
    if (gen && !tensor_core)
        return fail(c, MAMBA_B200_ERR_SHAPE, "m3_ssd_fwd: K/Q generation runs on the tensor-core path only (16-bit "
                                              "storage, headdim <= 64, d_state <= 128, multiples of 8, no carried "
                                              "state, 16-byte aligned tensors)");
    if (tensor_core) {
        p.wide_y = a.hd % 16 == 0 && reinterpret_cast<uintptr_t>(a.y) % 32 == 0;
        p.sc_tma = a.nh % 4 == 0 &&
                   make_tmap_3d(c, &p.tm_adt, MAMBA_B200_F32, a.adt, a.nh, a.nh, a.T, a.B, 4, 129) &&
                   make_tmap_3d(c, &p.tm_dt, MAMBA_B200_F32, a.dt, a.nh, a.nh, a.T, a.B, 4, 129) &&
                   make_tmap_3d(c, &p.tm_trap, MAMBA_B200_F32, a.trap, a.nh, a.nh, a.T, a.B, 4, 129);
        dim3 grid(a.nh, a.B);
        const bool bf = a.dtype == MAMBA_B200_BF16;
        // bf16, 64 x 128: 4 heads x 4096 steps 44 us (one CTA each: 123), 24 x 2048 34 (63), 64 x 4096 91 (124);
        // continued from a state 4 x 4096 62 us
        const int nchunks = (a.T + tc::CS - 1) / tc::CS;
        // Pairs that two CTAs per SM take are not divided, whose costs are one CTA's: 180 pairs continued over 4096 steps 535
        // us in clusters of four, 352 undivided; 150 x 16384 from zero 1023 and 825.
        const int pairs = a.B * a.nh;
        const bool two = !gen && (a.carry_in ? m3_two_carried_per_sm(pairs, nchunks) : m3_two_per_sm(pairs));
        const int ranks = gen || two ? 1 : a.carry_in ? m3_cluster_ranks(pairs, nchunks, 5.5, 6.6, 6.6, 3.2)
                                                      : m3_cluster_ranks(pairs, nchunks, 3.7, 5.15, 5.15, 2.6);
        if (ranks > 1) {
            const void* fn = bf ? (a.carry_in ? reinterpret_cast<const void*>(tc::m3_ssd_fwd_tc_kernel<__nv_bfloat16, false, true, true, false>)
                                              : reinterpret_cast<const void*>(tc::m3_ssd_fwd_tc_kernel<__nv_bfloat16, false, false, true, false>))
                                : reinterpret_cast<const void*>(tc::m3_ssd_fwd_tc_kernel<__half, false, false, true, false>);
            void* args[1] = {&p};
            MB200_CUDA_CHECK(c, launch_cluster(fn, dim3(a.nh * ranks, a.B), dim3(256), tc::kSmem, st, ranks, args));
        } else if (two && a.carry_in) {
            tc::m3_ssd_fwd_tc_kernel<__nv_bfloat16, false, true, false, true><<<grid, 256, tc::lean::kSmem, st>>>(p);
        } else if (two) {
            if (bf) tc::m3_ssd_fwd_tc_kernel<__nv_bfloat16, false, false, false, true><<<grid, 256, tc::lean::kSmem, st>>>(p);
            else tc::m3_ssd_fwd_tc_kernel<__half, false, false, false, true><<<grid, 256, tc::lean::kSmem, st>>>(p);
        } else if (bf) {
            if (gen) tc::m3_ssd_fwd_tc_kernel<__nv_bfloat16, true, false, false, false><<<grid, 256, tc::kSmem, st>>>(p);
            else if (a.carry_in) tc::m3_ssd_fwd_tc_kernel<__nv_bfloat16, false, true, false, false><<<grid, 256, tc::kSmem, st>>>(p);
            else tc::m3_ssd_fwd_tc_kernel<__nv_bfloat16, false, false, false, false><<<grid, 256, tc::kSmem, st>>>(p);
        } else {
            if (gen) tc::m3_ssd_fwd_tc_kernel<__half, true, false, false, false><<<grid, 256, tc::kSmem, st>>>(p);
            else tc::m3_ssd_fwd_tc_kernel<__half, false, false, false, false><<<grid, 256, tc::kSmem, st>>>(p);
        }
    } else {
        if (a.dtype == MAMBA_B200_F32) launch_seq<float>(p, c->sm_count, st);
        else if (a.dtype == MAMBA_B200_F16) launch_seq<__half>(p, c->sm_count, st);
        else launch_seq<__nv_bfloat16>(p, c->sm_count, st);
    }
    MB200_CUDA_CHECK(c, cudaGetLastError());
    return MAMBA_B200_OK;
}
