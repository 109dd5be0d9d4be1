// One decode step (one token per sequence) through every layer of a Mamba-1 backbone in one
// launch: residual + RMSNorm, in_proj, conv step + SiLU, x_proj, dt_proj, softplus, SSM step, gate,
// out_proj, and for the language model the embedding row, the tied head and the greedy choice.
// Replaces the per-layer launch sequence of GpuMambaBackbone::step
// (src/mamba_ssm/gpu/inference.rs:1515-1855, :1062-1215) and GpuMambaLM's decode step
// (src/module/gpu_lm.rs:560-679).
//
// A token needs every weight once and little arithmetic, so what a launch per operator costs is
// the launches: 198 of them, replayed from a graph, took 0.64 ms a token for the 130m architecture
// at batch 8 (bf16), and 590 us a step for three layers of d_model 128 without a graph; the weights
// at HBM speed are 0.04 ms.  Here the grid (one CTA per SM) stays resident and the CTAs hand one
// another four things a layer:
//   1  act = rmsnorm(residual)  (every CTA for itself);  x | z = act W_in;  u = silu(conv(x))      -> u
//   2  slices of x_proj: u W_x over a range of channels                              -> partial sums
//   3  delta, SSM step, gate for the channels of phase 1                                        -> y
//   4  residual += y W_out                                                               -> residual
// What is left is latency and instructions: every phase starts when the slowest CTA of the one before
// has handed over, and its code runs once a layer, so nothing hides it.  Hence:
// - What is handed over travels as 8-byte words of a 4-byte value and the tag of its layer, and the
//   reader loads until the tag is right.  There is no barrier of the grid, no fence and no counter: a
//   hand-over is one store and one load.  (Four barriers a layer, with release, poll and first read,
//   took 10,000 of a layer's 24,700 cycles.)  A word may be overwritten a layer later because whoever
//   writes it then needs, through the chain of phases, something that its every reader made from it.
// - Channels stay with a CTA from phase 1 to 3: u, z and the states are its own.
// - A seventeenth warp asks for all operands (TMA tiles of the four weights, bulk copies of the small
//   ones) as soon as their room is free; the sixteen others never wait for HBM.
// - Index arithmetic is done once per launch, packet counts are template arguments, and the products
//   take the weights as the M side of mma.sync m16n8k16 (a tile of x beside its tile of z) with eight
//   sequences as N, so a warp issues about 900 instructions a layer where it issued 2,800.
// Loops stay rolled: code that outgrows the instruction cache takes longer than it saves.  Measured
// (before: the same split with four barriers): 0.286 ms a token of the 130m architecture at batch 8
// (0.336), of which 0.025 are the head; 30 us a step of three layers of d_model 128 (38).
// Arithmetic: mma.sync for 16-bit storage (tcgen05's 128-row tiles would be mostly padding at these
// batch sizes and the products are not what takes the time), FMA for f32.  Sums are f32 in a fixed
// order: two runs are bit-identical.
#include <string.h>

#include <type_traits>

#include "common.cuh"
#include "internal.h"

namespace mb200 {
namespace dec {

constexpr int kThreads = 512, kWarps = 16;  // compute threads; one more warp asks for the operands
constexpr int kN = 16, kK = 4;          // d_state and d_conv of this kernel
constexpr int kMaxDm = 1024, kMaxB = 64, kMaxKSlice = 384, kMaxKs = 4;
constexpr long long kHeadAhead = 64ll << 20;  // bytes of the head's table asked for ahead of it
constexpr int kMaxPolls = 1 << 21;      // a poll is about a microsecond's L2 round trip

struct Params {
    CUtensorMap tm_in, tm_out, tm_x, tm_dt;  // W_in, W_out, W_x, W_dt of all layers: [L, K, columns]
    const void* lp;                     // compute-dtype arena
    const float *master, *a_neg;        // f32 arena, [L, di, N]
    long long lstride;                  // elements from one layer to the next (both arenas)
    long long o_in, o_cw, o_cb, o_x, o_dtw, o_dtb, o_D, o_out, o_normf, o_emb;
    float *conv, *ssm;                  // [L, Bcap, di, K], [L, Bcap, di, N]
    float* res;                         // [B, dm] residual stream; an element is its phase-4 thread's own
    // what CTAs hand one another: 8-byte words, a 4-byte value and the tag of its layer
    uint2 *u_x, *y_x;                   // [B, di]: two 16-bit values or one f32 a word
    uint2* p_x;                         // [ks, B, ncg * 8] partial sums of x_proj
    uint2* r_x;                         // [B, dm] residual stream
    uint4* a_x;                         // [B, ncta] best logit and its index
    unsigned* ctl;                      // [0] tags used so far, [1] CTAs done (zero between launches), [2] polls a
                                        // wait may take (zero: kMaxPolls)
    void* out;                          // backbone: rmsnorm(residual) in the compute dtype
    int *next_ids, *tokens;             // LM: ids in / next ids out; tokens[b * tok_ld] = id taken in
    long long tok_ld;
    void* logits;                       // LM: [B, V]
    int B, Bcap, dm, di, dr, xd, L, V;
    float eps, inv_dm;
    // in_proj / out_proj: column tiles per CTA (in_proj: of x, and as many of z), padded K, and how they lie in shared memory: chunks of
    // c tiles (odd, so that rows of c * 16 bytes meet different banks), ka rows each, from TMA boxes of br rows
    int t1, c1, kp1, ka1, br1;
    int t4, c4, kp4, ka4, br4;
    int ncg, ks, kslice, nch;           // x_proj: column groups, K slices; channels per CTA
    int brx, brd, x_tma, dt_tma;        // rows of a W_x and a W_dt box; whether the two come by TMA
    uint32_t s_w1, s_w4, s_act, s_red, s_wx, s_wd, s_norm, s_conv, s_uz, s_a;
    int* status;
};

__device__ __forceinline__ void cp16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp4(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
template <typename Th>
__device__ __forceinline__ void mma16816(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    if constexpr (std::is_same<Th, __nv_bfloat16>::value)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                     "{%0,%1,%2,%3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                     "{%0,%1,%2,%3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Words with their tags: 64-bit accesses are single, so a word is either wholly there or not at all.
__device__ __forceinline__ void put(uint2* dst, uint32_t v, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(dst), "l"(static_cast<unsigned long long>(tag) << 32 | v) : "memory");
}
__device__ __forceinline__ uint4 get2(const void* src) {
    unsigned long long a, b;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(src) : "memory");
    return make_uint4(static_cast<uint32_t>(a), static_cast<uint32_t>(a >> 32), static_cast<uint32_t>(b), static_cast<uint32_t>(b >> 32));
}
__device__ __forceinline__ float4 ldcg4(const float* p) { return __ldcg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// 32 values per lane summed over the warp; lane L keeps the sum of value L.
__device__ __forceinline__ float sum32(float* v, int lane) {
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) {
        const bool up = (lane & m) != 0;
#pragma unroll
        for (int r = 0; r < m; ++r) {
            const float give = up ? v[r] : v[r + m], keep = up ? v[r + m] : v[r];
            v[r] = keep + __shfl_xor_sync(0xffffffffu, give, m);
        }
    }
    return v[0];
}
// argmax order of the reference's greedy choice: larger value, then lower index; a NaN wins.
__device__ __forceinline__ bool better(float v, int i, float bv, int bi) {
    const bool vn = v != v, bn = bv != bv;
    if (vn != bn) return vn;
    if (vn) return i < bi;
    return v > bv || (v == bv && i < bi);
}

template <typename Tact>
struct Step {
    static constexpr bool H = sizeof(Tact) == 2;
    static constexpr int TW = 16 / sizeof(Tact);  // columns of a tile (16 bytes)
    static constexpr int LW = H ? 3 : 2;          // log2 of it
    static constexpr int BT = H ? 16 : 8;         // sequences per pass of a projection
    static constexpr int E = 4 / sizeof(Tact);    // values of an exchanged word
    static constexpr int PP = H ? 4 : 2;          // pairs of column tiles of a pass
    const Params& p;
    unsigned char* sm;
    const int tid, lane, warp, cta, ncta;
    bool alive = true;
    unsigned base_tag = 0;
    float* pair;     // sums that two warps of a row exchange
    uint64_t* bars;  // landed: W_in, W_out, W_x, small operands; then free: the same
    volatile int* dead;  // [1]: polls a wait may take (in shared memory, read after a miss: in a register it cost 3 %)

    __device__ Step(const Params& p_, unsigned char* sm_, float* pair_, uint64_t* bars_, int* dead_)
        : p(p_), sm(sm_), tid(threadIdx.x), lane(threadIdx.x & 31), warp(threadIdx.x >> 5), cta(blockIdx.x),
          ncta(gridDim.x), pair(pair_), bars(bars_), dead(dead_) {}

    __device__ const Tact* lp(int l, long long off) const { return static_cast<const Tact*>(p.lp) + l * p.lstride + off; }
    __device__ const float* mf(int l, long long off) const { return p.master + l * p.lstride + off; }
    __device__ unsigned tag_of(int l) const { return base_tag + 2 + l; }  // l = -1: the stream that enters
    // Which parts of the phases this CTA has: the first CTAs own channels (phases 1 and 3), phases 2 and 4 are
    // dealt from the last CTA down.
    __device__ int channels() const { return max(0, min(p.nch, p.di - cta * p.nch)); }
    __device__ int unit0() const { return ncta - 1 - cta; }
    __device__ bool has_unit() const { return unit0() < p.ncg * p.ks; }
    __device__ int out_tile() const { return (ncta - 1 - cta) * p.t4; }
    __device__ int out_tiles() const { return max(0, min(p.t4, p.dm / TW - out_tile())); }

    // ---- barriers of the compute warps; after meet() every thread knows whether some wait ran out ----
    __device__ void sync() { asm volatile("bar.sync 0, %0;" ::"n"(kThreads) : "memory"); }
    __device__ void meet() {
        uint32_t all;
        asm volatile(
            "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, 0, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
            : "=r"(all) : "r"(static_cast<uint32_t>(alive)), "n"(kThreads) : "memory");
        alive = all != 0;
    }
    enum Bar { kWIn, kWOut, kWX, kSmall, kFree };  // bars[kFree + x]: the room of x may be written again
    __device__ void landed(Bar b, int l) { alive = mbar_wait(&bars[b], l & 1, p.status) && alive; }
    __device__ void release(Bar b) {
        if (tid == 0) mbar_arrive(&bars[kFree + b]);
    }

    // ---- N packets of two words, at src + min(j + i * step, last), loaded until each has its tag.  Called by
    //      whole warps.  After a miss one lane asks for its first packet alone until it is there: all of them
    //      asked for again and again would load the L2 that the other CTAs write through. ----
    template <int N>
    __device__ void take(const uint4* src, int j, int step, int last, uint32_t tag, uint4 (&v)[N]) {
        for (int it = 0;;) {
            uint32_t miss = 0;
#pragma unroll
            for (int i = 0; i < N; ++i) v[i] = get2(src + min(j + i * step, last));
#pragma unroll
            for (int i = 0; i < N; ++i) miss |= (v[i].y ^ tag) | (v[i].w ^ tag);
            if (!__any_sync(0xffffffffu, miss != 0)) break;
            const int polls = dead[1];
            if (lane == 0)
                while ((v[0].y != tag || v[0].w != tag) && ++it < polls) v[0] = get2(src + min(j, last));
            it = __shfl_sync(0xffffffffu, it, 0) + 1;
            if (it >= polls || !alive) {
                alive = false;
                if (lane == 0) atomicCAS(p.status, kStatusOk, kStatusBarrierTimeout);
                break;
            }
        }
    }
    // element `at` of [B, di] to the other CTAs; in 16-bit storage the lane GAP further on has the next one of
    // the word.  Called by whole warps.
    template <int GAP>
    __device__ void publish(uint2* dst, int at, Tact v, bool on, unsigned tag) {
        if constexpr (H) {
            const uint32_t own = *reinterpret_cast<const unsigned short*>(&v), next = __shfl_down_sync(0xffffffffu, own, GAP);
            if (on && (at & 1) == 0) put(dst + at / 2, own | next << 16, tag);
        } else if (on) {
            put(dst + at, __float_as_uint(v), tag);
        }
    }

    // ================= the seventeenth warp: operands of a layer, asked for as soon as their room is free =================
    __device__ void ask_tiles(const CUtensorMap* map, Bar b, uint32_t dst, int l, int first, int per, int sets, int c, int ka, int br) {
        const int kb = ka / br, chunks = per / c * sets;
        if (lane == 0) mbar_expect_tx(&bars[b], static_cast<uint32_t>(chunks) * ka * c * 16);
        __syncwarp();
#pragma unroll 1
        for (int j = lane; j < chunks * kb; j += 32) {
            const int q = j / kb, k = (j - q * kb) * br, q0 = q < per / c ? q : q - per / c;
            tma_load_3d(sm + dst + static_cast<uint32_t>(q * ka + k) * c * 16, map, &bars[b],
                        (first + q0 * c) * TW + (q == q0 ? 0 : p.di), k, l);
        }
    }
    __device__ void ask_x(int l) {
        if (lane == 0) {
            mbar_expect_tx(&bars[kWX], static_cast<uint32_t>(p.kslice) * 8 * sizeof(Tact));
            for (int k = 0; k < p.kslice; k += p.brx)
                tma_load_3d(sm + p.s_wx + k * 8 * sizeof(Tact), &p.tm_x, &bars[kWX], unit0() % p.ncg * 8, unit0() / p.ncg * p.kslice + k, l);
        }
    }
    // norm weights; conv windows [B][channels], taps and bias; W_dt's columns; A, D and dt's bias of the channels
    __device__ void ask_small(int l) {
        const int n = channels(), d0 = cta * p.nch, db = (p.dr + p.brd - 1) / p.brd;
        unsigned char* cv = sm + p.s_conv;
        if (lane == 0)
            mbar_expect_tx(&bars[kSmall], p.dm * 4 + (p.B + 1) * n * 16 + n * (4 + kN * 4 + 4 + static_cast<int>(sizeof(Tact))) +
                                              (p.dt_tma ? db * p.brd * p.nch * static_cast<int>(sizeof(Tact)) : 0));
        __syncwarp();
        if (lane == 0) bulk_load(sm + p.s_norm, mf(l, 0), p.dm * 4, &bars[kSmall]);
        if (lane == 1) bulk_load(cv + p.B * p.nch * 16, mf(l, p.o_cw) + d0 * kK, n * 16, &bars[kSmall]);
        if (lane == 2) bulk_load(cv + (p.B + 1) * p.nch * 16, mf(l, p.o_cb) + d0, n * 4, &bars[kSmall]);
        unsigned char* am = sm + p.s_a;
        if (lane == 3) bulk_load(am, p.a_neg + (static_cast<long long>(l) * p.di + d0) * kN, n * kN * 4, &bars[kSmall]);
        if (lane == 4) bulk_load(am + p.nch * kN * 4, mf(l, p.o_D) + d0, n * 4, &bars[kSmall]);
        if (lane == 5) bulk_load(am + p.nch * (kN + 1) * 4, lp(l, p.o_dtb) + d0, n * sizeof(Tact), &bars[kSmall]);
        for (int b = lane; b < p.B; b += 32)
            bulk_load(cv + b * p.nch * 16, p.conv + ((static_cast<long long>(l) * p.Bcap + b) * p.di + d0) * kK, n * 16, &bars[kSmall]);
        if (p.dt_tma && lane < db)
            tma_load_3d(sm + p.s_wd + lane * p.brd * p.nch * sizeof(Tact), &p.tm_dt, &bars[kSmall], d0, lane * p.brd, l);
    }
    // the states of layer l, which the scan loads itself, into L2
    __device__ void hint(int l) {
        const int ch0 = cta * p.nch, n = channels();
        if (l >= p.L || n <= 0) return;
        for (int b = lane; b < p.B; b += 32)
            l2_prefetch_bulk(p.ssm + ((static_cast<long long>(l) * p.Bcap + b) * p.di + ch0) * kN, n * kN * 4);
    }
    __device__ void ask_in(int l) { ask_tiles(&p.tm_in, kWIn, p.s_w1, l, cta * p.t1, p.t1, 2, p.c1, p.ka1, p.br1); }
    __device__ void ask_out(int l) { ask_tiles(&p.tm_out, kWOut, p.s_w4, l, out_tile(), p.t4, 1, p.c4, p.ka4, p.br4); }
    // false when the compute warps have given up (or never come)
    __device__ bool freed(Bar b, int l) {
        for (int it = 0; it < (1 << 12); ++it) {
            if (mbar_wait(&bars[kFree + b], l & 1, nullptr, 1 << 10)) return true;
            if (*dead) return false;
        }
        return false;
    }
    // A quarter of this CTA's tiles of the head, into L2 under each of the last four layers, whose weights leave
    // HBM nine tenths idle.  Beyond kHeadAhead they would only push one another out.
    static constexpr int kHeadRows = H ? 16 : 4;  // of a tile
    __device__ void hint_head(int l) {
        const int quarter = l - (p.L - 4);
        if (!p.next_ids || quarter < 0) return;
        const long long row = static_cast<long long>(p.dm) * sizeof(Tact);
        for (int t = lane;; t += 32) {
            const long long r = (static_cast<long long>(t) * ncta + cta) * kHeadRows + quarter * (kHeadRows / 4);
            if (r >= p.V || r * row > kHeadAhead) return;
            l2_prefetch_bulk(static_cast<const Tact*>(p.lp) + p.o_emb + r * p.dm,
                             static_cast<uint32_t>(min(static_cast<long long>(kHeadRows / 4), p.V - r) * row));
        }
    }
    __device__ void feed() {
        const bool in = channels() > 0, x = has_unit() && p.x_tma, out = out_tiles() > 0;
        if (in) ask_in(0);
        if (in) ask_small(0);
        if (x) ask_x(0);
        if (out) ask_out(0);
        hint(0);
        hint(1);
        int n_in = 1, n_small = 1, n_x = 1, n_out = 1;  // asked for so far
        for (int l = 0; l < p.L - 1; ++l) {
            if (in) {
                if (!freed(kWIn, l)) break;
                ask_in(l + 1);
                ++n_in;
            }
            if (x) {
                if (!freed(kWX, l)) break;
                ask_x(l + 1);
                ++n_x;
            }
            hint(l + 2);
            hint_head(l + 1);
            if (in) {
                if (!freed(kSmall, l)) break;
                ask_small(l + 1);
                ++n_small;
            }
            if (out) {
                if (!freed(kWOut, l)) break;
                ask_out(l + 1);
                ++n_out;
            }
        }
        // everything has to land in this CTA's memory while it is this CTA's
        if (in) mbar_wait(&bars[kWIn], (n_in - 1) & 1, nullptr, 1 << 16);
        if (in) mbar_wait(&bars[kSmall], (n_small - 1) & 1, nullptr, 1 << 16);
        if (x) mbar_wait(&bars[kWX], (n_x - 1) & 1, nullptr, 1 << 16);
        if (out) mbar_wait(&bars[kWOut], (n_out - 1) & 1, nullptr, 1 << 16);
    }

    // ================= compute warps =================
    // ---- rows b0 .. b0+bt of rmsnorm(stream) * w as the A operand, the stream from the phase 4 of a layer; two
    //      warps a row, N pairs of columns a lane ----
    template <int N>
    __device__ void norm_rows_n(const float* w, int b0, int bt, int kp, unsigned tag) {
        Tact* act = reinterpret_cast<Tact*>(sm + p.s_act);
        const int ld = kp + TW, j = lane + 32 * (warp & 1);
#pragma unroll 1
        for (int r = warp >> 1; r < bt; r += kWarps / 2) {
            uint4 v[N];
            take<N>(reinterpret_cast<const uint4*>(p.r_x + (b0 + r) * p.dm), j, 64, p.dm / 2 - 1, tag, v);
            float ss = 0.0f;
#pragma unroll
            for (int i = 0; i < N; ++i) {
                if (j + 64 * i >= p.dm / 2) v[i].x = v[i].z = 0;
                const float a = __uint_as_float(v[i].x), b = __uint_as_float(v[i].z);
                ss = fmaf(a, a, fmaf(b, b, ss));
            }
#pragma unroll
            for (int m = 16; m >= 1; m >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, m);
            if (lane == 0) pair[warp] = ss;
            asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp >> 1)) : "memory");
            ss = pair[warp & ~1] + pair[warp | 1];
            float inv = rsqrtf(fmaf(ss, p.inv_dm, p.eps));
            if (!(inv > 0.0f && inv <= 1e20f)) inv = 1.0f;  // rms not finite or below 1e-20: the norm operator's guard
            Tact* row = act + r * ld + 2 * j;
#pragma unroll
            for (int i = 0; i < N; ++i)
                if (j + 64 * i < p.dm / 2) {
                    const float2 g = *reinterpret_cast<const float2*>(w + 2 * j + 128 * i);
                    st_pair(row + 128 * i, make_float2(__uint_as_float(v[i].x) * inv * g.x, __uint_as_float(v[i].z) * inv * g.y));
                }
            if ((warp & 1) == 0 && p.dm + lane < kp) act[r * ld + p.dm + lane] = from_f<Tact>(0.0f);  // kp - dm < 32
            if (r + kWarps / 2 < bt) asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp >> 1)) : "memory");  // (`pair` is read)
        }
    }
    __device__ void norm_rows(const float* w, int b0, int bt, int kp, unsigned tag) {
        const int n = (p.dm + 127) / 128;
        if (n <= 1) norm_rows_n<1>(w, b0, bt, kp, tag);
        else if (n <= 2) norm_rows_n<2>(w, b0, bt, kp, tag);
        else if (n <= 4) norm_rows_n<4>(w, b0, bt, kp, tag);
        else if (n <= 6) norm_rows_n<6>(w, b0, bt, kp, tag);
        else norm_rows_n<kMaxDm / 128>(w, b0, bt, kp, tag);
    }
    // ---- rows of y (from phase 3 of the layer) as the A operand; two warps a row ----
    template <int N>
    __device__ void load_rows_n(int kp, int b0, int bt, unsigned tag) {
        Tact* act = reinterpret_cast<Tact*>(sm + p.s_act);
        const int ld = kp + TW, n = p.di / (2 * E), np = kp / (2 * E), j1 = lane + 32 * (warp & 1);
#pragma unroll 1
        for (int r = warp >> 1; r < bt; r += kWarps / 2)
#pragma unroll 1
            for (int j = j1; j - j1 < np; j += N * 64) {
                uint4 v[N];
                take<N>(reinterpret_cast<const uint4*>(p.y_x + (b0 + r) * (p.di / E)), j, 64, n - 1, tag, v);
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    const int q = j + 64 * i;
                    if (q < np) *reinterpret_cast<uint2*>(act + r * ld + q * 2 * E) = q < n ? make_uint2(v[i].x, v[i].z) : make_uint2(0, 0);
                }
            }
    }
    __device__ void load_rows(int b0, int bt, unsigned tag) {
        const int n = (p.kp4 / (2 * E) + 63) / 64;
        if (n <= 1) load_rows_n<1>(p.kp4, b0, bt, tag);
        else if (n <= 2) load_rows_n<2>(p.kp4, b0, bt, tag);
        else if (n <= 4) load_rows_n<4>(p.kp4, b0, bt, tag);
        else if (n <= 6) load_rows_n<6>(p.kp4, b0, bt, tag);
        else load_rows_n<8>(p.kp4, b0, bt, tag);
    }

    // ---- out[b][column] = act W for n <= PP pairs of column tiles; pair i is tile a0 + i * da and tile b0 + i * db
    //      of the CTA's (the second clamped to the last one there is).  The warps split K; partials in s_red. ----
    static constexpr int RP = H ? 160 : 32;  // floats of a part: [8 rows, 20 apart][16 columns] / [8 rows][4 columns]
    __device__ static int parts_log(int n) { return H ? (n > 2 ? 2 : n > 1 ? 3 : 4) : n > 1 ? 2 : 3; }  // log2 of the K parts
    __device__ void project(uint32_t wofs, int kp, int ka, int cw, int ta, int da, int tb, int db, int last, int n, int rows) {
        float* red = reinterpret_cast<float*>(sm + p.s_red);
        const int ld = kp + TW;
        if constexpr (H) {
            const int lg = parts_log(n), i = warp >> lg, part = warp & ((1 << lg) - 1), groups = rows > 8 ? 2 : 1;
            if (i >= n) return;
            // lanes 0-7 and 16-23 hold rows of the first tile of the pair, the others of the second
            const int tile = (lane & 8) ? min(tb + i * db, last) : ta + i * da, q = cw == 1 ? tile : tile / cw;
            const int kr = (lane & 7) + ((lane & 16) >> 1);  // K row of this lane's ldmatrix address
            uint32_t arow = smem_u32(sm + wofs) + static_cast<uint32_t>((q * ka + kr + part * 32) * cw + tile - q * cw) * 16;
            uint32_t brow = smem_u32(sm + p.s_act) + (min(lane & 7, rows - 1) * ld + (lane >> 3) * 8 + part * 32) * 2;
            const uint32_t brow2 = (min(8 + (lane & 7), rows - 1) - min(lane & 7, rows - 1)) * ld * 2;
            float c[4][4];  // two accumulators for each group of eight rows
#pragma unroll
            for (int e = 0; e < 4; ++e) c[0][e] = c[1][e] = c[2][e] = c[3][e] = 0.0f;
            const uint32_t ahalf = 256 * cw, astep = (512u * cw) << lg, bstep = 64u << lg;
            const int units = kp / 32;
            // three units of 32 at a time, all their loads ahead of the products
#pragma unroll 1
            for (int u = part; u < units; u += 3 << lg, arow += 3 * astep, brow += 3 * bstep) {
                uint32_t a[3][8], b[3][4];
                const int m = min(3, (units - u + (1 << lg) - 1) >> lg);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const uint32_t o = k < m ? k : 0;
                    ldmatrix_x4_trans(arow + o * astep, a[k]);
                    ldmatrix_x4_trans(arow + o * astep + ahalf, a[k] + 4);
                    ldmatrix_x4(brow + o * bstep, b[k]);
                }
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    if (k < m) {
                        mma16816<Tact>(c[0], a[k][0], a[k][1], a[k][2], a[k][3], b[k][0], b[k][1]);
                        mma16816<Tact>(c[1], a[k][4], a[k][5], a[k][6], a[k][7], b[k][2], b[k][3]);
                    }
                if (groups == 2) {
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                        if (k < m) {
                            ldmatrix_x4(brow + brow2 + k * bstep, b[k]);
                            mma16816<Tact>(c[2], a[k][0], a[k][1], a[k][2], a[k][3], b[k][0], b[k][1]);
                            mma16816<Tact>(c[3], a[k][4], a[k][5], a[k][6], a[k][7], b[k][2], b[k][3]);
                        }
                }
            }
            float* o = red + warp * (2 * RP) + (lane & 3) * 40 + (lane >> 2);
            o[0] = c[0][0] + c[1][0]; o[20] = c[0][1] + c[1][1]; o[8] = c[0][2] + c[1][2]; o[28] = c[0][3] + c[1][3];
            if (groups == 2) {
                o += RP;
                o[0] = c[2][0] + c[3][0]; o[20] = c[2][1] + c[3][1]; o[8] = c[2][2] + c[3][2]; o[28] = c[2][3] + c[3][3];
            }
        } else {
            const float* act = reinterpret_cast<const float*>(sm + p.s_act);
            // a warp has one tile and a part of K
            const int lg = parts_log(n), t = warp >> lg, part = warp & ((1 << lg) - 1);
            float acc[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) acc[i] = 0.0f;
            const int tile = (t & 1) ? min(tb + (t >> 1) * db, last) : ta + (t >> 1) * da, q = tile / cw;
            const float4* w = reinterpret_cast<const float4*>(sm + wofs) + q * ka * cw + (tile - q * cw);
#pragma unroll 1
            for (int k = part * 32 + lane; k < kp; k += 32 << lg) {
                const float4 wv = w[k * cw];
#pragma unroll
                for (int b = 0; b < 8; ++b) {
                    const float a = act[min(b, rows - 1) * ld + k];
                    acc[4 * b] = fmaf(a, wv.x, acc[4 * b]);
                    acc[4 * b + 1] = fmaf(a, wv.y, acc[4 * b + 1]);
                    acc[4 * b + 2] = fmaf(a, wv.z, acc[4 * b + 2]);
                    acc[4 * b + 3] = fmaf(a, wv.w, acc[4 * b + 3]);
                }
            }
            red[warp * RP + lane] = sum32(acc, lane);
        }
    }
    // the sum of output (pair i, second: column c of its second tile, row b)
    __device__ float total(int n, int i, bool second, int b, int c) const {
        const float* o = reinterpret_cast<const float*>(sm + p.s_red);
        const int lg = parts_log(n);
        constexpr int D = H ? 2 * RP : RP;  // from part to part
        if constexpr (H) o += (i << lg) * D + (b >> 3) * RP + (b & 7) * 20 + (second ? 8 : 0) + c;
        else o += ((2 * i + (second ? 1 : 0)) << lg) * D + b * 4 + c;
        float s = (o[0] + o[D]) + (o[2 * D] + o[3 * D]);
        if (lg >= 3) s += (o[4 * D] + o[5 * D]) + (o[6 * D] + o[7 * D]);
        if (lg >= 4) s += ((o[8 * D] + o[9 * D]) + (o[10 * D] + o[11 * D])) + ((o[12 * D] + o[13 * D]) + (o[14 * D] + o[15 * D]));
        return s;
    }
    // rows of a pass as a power of two: 8 or 16
    __device__ static int row_log(int rows) { return rows > 8 ? 4 : 3; }

    // ---- phase 1: this CTA's x and z columns; u goes to phase 2, u and z stay for phase 3 ----
    __device__ void in_proj(int l) {
        const int n = channels();
        if (n <= 0) return;
        const float4* win_s = reinterpret_cast<const float4*>(sm + p.s_conv);
        const float4* tap_s = win_s + p.B * p.nch;
        const float* cb_s = reinterpret_cast<const float*>(tap_s + p.nch);
        float2* uz = reinterpret_cast<float2*>(sm + p.s_uz);
        landed(kSmall, l);
#pragma unroll 1
        for (int b0 = 0; b0 < p.B; b0 += BT) {
            const int bt = min(BT, p.B - b0), rl = row_log(bt);
            norm_rows(reinterpret_cast<const float*>(sm + p.s_norm), b0, bt, p.kp1, tag_of(l - 1));
            if (b0 == 0) landed(kWIn, l);
            meet();
            if (!alive) return;
#pragma unroll 1
            for (int t0 = 0; t0 < p.t1; t0 += PP) {
                const int tn = min(PP, p.t1 - t0);
                project(p.s_w1, p.kp1, p.ka1, p.c1, t0, 1, p.t1 + t0, 1, 2 * p.t1 - 1, tn, bt);
                sync();
                if (t0 + PP >= p.t1 && b0 + BT >= p.B) release(kWIn);
                // columns, rows, pairs on consecutive threads, whole warps
#pragma unroll 1
                for (int i = tid; i < tn << (LW + rl); i += kThreads) {
                    const int c = i & (TW - 1), b = (i >> LW) & ((1 << rl) - 1), q = i >> (LW + rl), cc = (t0 + q) * TW + c;
                    const int d = cta * p.nch + cc, at = b0 + b;
                    const bool on = b < bt && cc < n;
                    Tact u = from_f<Tact>(0.0f);
                    if (on) {
                        // the projection leaves in the storage dtype, as the x | z halves do elsewhere
                        const float v = to_f(from_f<Tact>(total(tn, q, false, b, c))), z = to_f(from_f<Tact>(total(tn, q, true, b, c)));
                        const float4 win = win_s[at * p.nch + cc], cw = tap_s[cc];
                        const float acc = fmaf(v, cw.w, fmaf(win.w, cw.z, fmaf(win.z, cw.y, fmaf(win.y, cw.x, cb_s[cc]))));
                        u = from_f<Tact>(siluf_fast(acc));
                        uz[at * p.nch + cc] = make_float2(to_f(u), z);
                        *reinterpret_cast<float4*>(p.conv + ((static_cast<long long>(l) * p.Bcap + at) * p.di + d) * kK) =
                            make_float4(win.y, win.z, win.w, v);
                    }
                    publish<1>(p.u_x, at * p.di + d, u, on, tag_of(l));
                }
                if (t0 + PP < p.t1 || b0 + BT < p.B) sync();
            }
        }
    }

    // ---- phase 2: partial sums of x_proj over a slice of channels, eight columns a unit ----
    // W_x where TMA does not take it: asynchronous 4-byte copies where a row starts on 4 bytes, else plain loads
    __device__ void x_weights(int l, int unit) {
        if (l >= p.L || unit >= p.ncg * p.ks) return;
        Tact* w2 = reinterpret_cast<Tact*>(sm + p.s_wx);
        const int k0 = (unit / p.ncg) * p.kslice, c0 = (unit % p.ncg) * 8, nk = min(p.kslice, p.di - k0);
        const Tact* w = lp(l, p.o_x) + static_cast<long long>(k0) * p.xd + c0;
        constexpr int PR = 8 / E;  // copies of a row
        if (p.xd % E == 0) {
            const int c = tid % PR;
            if (c0 + c * E < p.xd)
#pragma unroll 1
                for (int k = tid / PR; k < nk; k += kThreads / PR)
                    cp4(smem_u32(w2 + k * 8 + c * E), w + static_cast<long long>(k) * p.xd + c * E);
        } else {
            const int c = tid & 7;
#pragma unroll 1
            for (int k = tid >> 3; k < nk; k += kThreads / 8)
                if (c0 + c < p.xd) w2[k * 8 + c] = w[static_cast<long long>(k) * p.xd + c];
        }
        cp_wait_all();
    }
    __device__ void x_proj(int l) {
        if (!has_unit()) return;
        Tact* us = reinterpret_cast<Tact*>(sm + p.s_act);
        const int uld = p.kslice + TW;
#pragma unroll 1
        for (int unit = unit0(); unit < p.ncg * p.ks; unit += ncta) {
            if (unit >= ncta) {  // (W_x comes by TMA only where a CTA has one unit)
                sync();
                x_weights(l, unit);
            }
            const int s = unit / p.ncg, k0 = s * p.kslice, g = unit - s * p.ncg;
#pragma unroll 1
            for (int b0 = 0; b0 < p.B; b0 += BT) {
                const int bt = min(BT, p.B - b0);
                constexpr int CH = H ? 32 : 64, N = 3;  // threads a row, packets a thread
                static_assert(CH * N * 2 * E >= kMaxKSlice && kThreads / CH >= (H ? 16 : 8), "slice");
                const int b = tid / CH, j = tid % CH, nj = p.kslice / (2 * E), have = min(nj, (p.di - k0) / (2 * E));
                if (b < bt) {
                    uint4 v[N];
                    take<N>(reinterpret_cast<const uint4*>(p.u_x + ((b0 + b) * p.di + k0) / E), j, CH, have - 1, tag_of(l), v);
#pragma unroll
                    for (int i = 0; i < N; ++i) {
                        const int q = j + i * CH;
                        if (q < nj) *reinterpret_cast<uint2*>(us + b * uld + q * 2 * E) = q < have ? make_uint2(v[i].x, v[i].z) : make_uint2(0, 0);
                    }
                }
                if (b0 == 0 && p.x_tma) landed(kWX, l);
                meet();
                if (!alive) return;
                uint2* out = p.p_x + (static_cast<long long>(s) * p.B + b0) * (p.ncg * 8) + g * 8;
                float* red = reinterpret_cast<float*>(sm + p.s_red);
                if constexpr (H) {
                    const int steps = p.kslice / 16, groups = bt > 8 ? 2 : 1;
                    static_assert(kMaxKSlice / 16 <= 2 * kWarps, "two K steps a warp");
                    if (warp < steps) {
                        float c[2][4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) c[0][e] = c[1][e] = 0.0f;
                        // (the second tile of the pair is the first one again, its sums go nowhere)
                        uint32_t arow = smem_u32(sm + p.s_wx) + (warp * 16 + (lane & 7) + ((lane & 16) >> 1)) * 16;
                        // matrices: rows 0-7 of K 0-7, 8-15, then rows 8-15
                        uint32_t brow = smem_u32(us) + (min((lane & 7) + ((lane & 16) >> 1), bt - 1) * uld + warp * 16 + (lane & 8)) * 2;
#pragma unroll 1
                        for (int k = warp; k < steps; k += kWarps, arow += kWarps * 256, brow += kWarps * 32) {
                            uint32_t a[4], bb[4];
                            ldmatrix_x4_trans(arow, a);
                            ldmatrix_x4(brow, bb);
                            mma16816<Tact>(c[0], a[0], a[1], a[2], a[3], bb[0], bb[1]);
                            if (groups == 2) mma16816<Tact>(c[1], a[0], a[1], a[2], a[3], bb[2], bb[3]);
                        }
                        float* o = red + warp * 128 + (lane & 3) * 16 + (lane >> 2);
                        o[0] = c[0][0]; o[8] = c[0][1];
                        if (groups == 2) { o[64] = c[1][0]; o[72] = c[1][1]; }
                    }
                    sync();
                    if (b0 + BT >= p.B && unit == unit0()) release(kWX);
                    if (tid < 8 * bt) {
                        float sum = red[tid], sum2 = 0.0f;
#pragma unroll
                        for (int w = 1; w < kWarps; ++w)
                            if (w < steps) (w & 1 ? sum2 : sum) += red[w * 128 + tid];
                        sum += sum2;
                        put(out + (tid >> 3) * p.ncg * 8 + (tid & 7), __float_as_uint(sum), tag_of(l));
                    }
                } else {
                    const int c = tid & 7, b = (tid >> 3) & 7, part = tid >> 6;
                    const float *ur = reinterpret_cast<const float*>(us) + min(b, bt - 1) * uld, *wr = reinterpret_cast<const float*>(sm + p.s_wx) + c;
                    float acc = 0.0f;
#pragma unroll 4
                    for (int k = part; k < p.kslice; k += 8) acc = fmaf(ur[k], wr[k * 8], acc);
                    red[tid] = acc;
                    sync();
                    if (b0 + BT >= p.B && unit == unit0()) release(kWX);
                    if (part == 0 && b < bt)
                        put(out + b * p.ncg * 8 + c,
                            __float_as_uint(((red[tid] + red[tid + 64]) + (red[tid + 128] + red[tid + 192])) +
                                            ((red[tid + 256] + red[tid + 320]) + (red[tid + 384] + red[tid + 448]))),
                            tag_of(l));
                }
                if (b0 + BT < p.B) sync();
            }
        }
        if (!p.x_tma) {
            if (unit0() + ncta < p.ncg * p.ks) sync();
            x_weights(l + 1, unit0());  // (published by the barriers ahead of the next use)
        }
    }

    // ---- phase 3: delta, SSM step, gate; four lanes (four states each) per (sequence, channel) ----
    __device__ void dt_weights(int l) {  // where TMA does not take W_dt
        const int n = channels();
        if (l >= p.L || n <= 0) return;
        const Tact* w = lp(l, p.o_dtw) + cta * p.nch;
        Tact* wd = reinterpret_cast<Tact*>(sm + p.s_wd);
#pragma unroll 1
        for (int i = tid; i < p.dr * n; i += kThreads) {
            const int r = i / n, c = i - r * n;
            wd[r * p.nch + c] = w[static_cast<long long>(r) * p.di + c];
        }
    }
    __device__ float4 load_state(int l, int b, int c) const {
        return ldcg4(p.ssm + ((static_cast<long long>(l) * p.Bcap + b) * p.di + cta * p.nch + c) * kN + 4 * (tid & 3));
    }
    __device__ void do_task(int l, int b, int c, bool on, float4 h0) {
        const Tact* wd = reinterpret_cast<const Tact*>(sm + p.s_wd) + c;
        const int j = tid & 3, d = cta * p.nch + c;
        const float* xr = reinterpret_cast<const float*>(sm + p.s_act) + b * p.xd;
        const float* am = reinterpret_cast<const float*>(sm + p.s_a);
        const float4 a = *reinterpret_cast<const float4*>(am + c * kN + 4 * j);
        const float D = am[p.nch * kN + c], dtb = to_f(reinterpret_cast<const Tact*>(am + p.nch * (kN + 1))[c]);
        float dl = 0.0f;
#pragma unroll 4
        for (int r = j; r < p.dr; r += 4) dl = fmaf(xr[r], to_f(wd[r * p.nch]), dl);
        dl += __shfl_xor_sync(0xffffffffu, dl, 1);
        dl += __shfl_xor_sync(0xffffffffu, dl, 2);
        dl = softplusf_fast(dl + dtb);
        const float2 uz = reinterpret_cast<const float2*>(sm + p.s_uz)[b * p.nch + c];
        const float du = dl * uz.x, dk = dl * kLog2e;
        const float* Bv = xr + p.dr + 4 * j;
        const float* Cv = Bv + kN;
        float4 h;
        h.x = fmaf(ex2(dk * a.x), h0.x, du * Bv[0]);
        h.y = fmaf(ex2(dk * a.y), h0.y, du * Bv[1]);
        h.z = fmaf(ex2(dk * a.z), h0.z, du * Bv[2]);
        h.w = fmaf(ex2(dk * a.w), h0.w, du * Bv[3]);
        float y = fmaf(h.x, Cv[0], fmaf(h.y, Cv[1], fmaf(h.z, Cv[2], h.w * Cv[3])));
        y += __shfl_xor_sync(0xffffffffu, y, 1);
        y += __shfl_xor_sync(0xffffffffu, y, 2);
        publish<4>(p.y_x, b * p.di + d, from_f<Tact>(fmaf(D, uz.x, y) * siluf_fast(uz.y)), on && j == 0, tag_of(l));
        if (on) *reinterpret_cast<float4*>(p.ssm + ((static_cast<long long>(l) * p.Bcap + b) * p.di + d) * kN + 4 * j) = h;
    }
    // (b, c) of this thread's first task and first pair of x_proj columns: the same in every layer
    struct Place { int b, c, row, col; };
    __device__ void scan(int l, const Place& at) {
        const int n = channels();
        if (n <= 0) return;
        const int tasks = p.B * n, q0 = tid >> 2;
        float4 h = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (q0 < tasks) h = load_state(l, at.b, at.c);
        float* xs = reinterpret_cast<float*>(sm + p.s_act);
        const int per = p.ncg * 4, pairs = p.B * per;  // pairs of columns of all rows
        int row = at.row, col = at.col;
#pragma unroll 1
        for (int i0 = tid; i0 - lane < pairs; i0 += kThreads) {
            if (i0 != tid) {
                row = i0 / per;
                col = 2 * (i0 - row * per);
            }
            float a = 0.0f, c = 0.0f;
#pragma unroll 1
            for (int s0 = 0; s0 < p.ks; s0 += kMaxKs) {
                uint4 v[kMaxKs];
                const int me = s0 * pairs + min(i0, pairs - 1);
                take<kMaxKs>(reinterpret_cast<const uint4*>(p.p_x) + me, 0, pairs, (p.ks - 1 - s0) * pairs, tag_of(l), v);
#pragma unroll
                for (int q = 0; q < kMaxKs; ++q)
                    if (s0 + q < p.ks) {
                        a += __uint_as_float(v[q].x);
                        c += __uint_as_float(v[q].z);
                    }
            }
            if (i0 < pairs && col < p.xd) xs[row * p.xd + col] = a;
            if (i0 < pairs && col + 1 < p.xd) xs[row * p.xd + col + 1] = c;
        }
        meet();
        if (!alive) return;
        int b = at.b, c = at.c;
#pragma unroll 1
        for (int q = q0, r = 0; r < tasks; q += kThreads / 4, r += kThreads / 4) {
            if (r > 0) {
                b = q < tasks ? q / n : 0;
                c = q < tasks ? q - b * n : 0;
                if (q < tasks) h = load_state(l, b, c);
            }
            if (q - lane / 4 < tasks) do_task(l, b, c, q < tasks, h);  // whole warps
        }
    }

    // ---- phase 4 ----
    // element i of a pass's outputs of phase 4: n pairs of tiles from t0 on, 1 << rl rows
    __device__ bool out_element(int i, int t0, int b0, int bt, int rl, int& q, bool& second, int& b, int& c, int& d) const {
        c = i & (TW - 1);
        b = (i >> LW) & ((1 << rl) - 1);
        second = (i >> (LW + rl)) & 1;
        q = i >> (LW + rl + 1);
        const int tile = t0 + 2 * q + (second ? 1 : 0);
        d = (out_tile() + tile) * TW + c;
        return b < bt && tile < out_tiles();
    }
    // the stream that enters, as its phase-4 threads keep it; the first element stays in a register
    __device__ void enter(float& own) {
        const int n = out_tiles();
#pragma unroll 1
        for (int b0 = 0; b0 < p.B && n > 0; b0 += BT) {
            const int bt = min(BT, p.B - b0), rl = row_log(bt);
#pragma unroll 1
            for (int t0 = 0; t0 < n; t0 += 2 * PP)
#pragma unroll 1
                for (int i = tid; i < min(PP, (n - t0 + 1) / 2) << (LW + rl + 1); i += kThreads) {
                    int q, b, c, d;
                    bool second;
                    if (!out_element(i, t0, b0, bt, rl, q, second, b, c, d)) continue;
                    const int at = (b0 + b) * p.dm + d;
                    float v = 0.0f;
                    if (p.next_ids) {
                        const int id = p.next_ids[b0 + b];
                        if (id >= 0 && id < p.V) v = to_f(static_cast<const Tact*>(p.lp)[p.o_emb + static_cast<long long>(id) * p.dm + d]);
                        p.res[at] = v;
                    } else {
                        v = p.res[at];
                    }
                    if (i == tid && t0 == 0 && b0 == 0) own = v;
                    put(p.r_x + at, __float_as_uint(v), tag_of(-1));
                }
        }
    }
    __device__ void out_proj(int l, float& own) {
        const int n = out_tiles();
        if (n <= 0) return;
#pragma unroll 1
        for (int b0 = 0; b0 < p.B; b0 += BT) {
            const int bt = min(BT, p.B - b0), rl = row_log(bt);
            load_rows(b0, bt, tag_of(l));
            if (b0 == 0) landed(kWOut, l);
            meet();
            if (!alive) return;
#pragma unroll 1
            for (int t0 = 0; t0 < n; t0 += 2 * PP) {
                const int tn = min(PP, (n - t0 + 1) / 2);
                project(p.s_w4, p.kp4, p.ka4, p.c4, t0, 2, t0 + 1, 2, p.t4 - 1, tn, bt);
                sync();
                if (t0 + 2 * PP >= n && b0 + BT >= p.B) release(kWOut);
#pragma unroll 1
                for (int i = tid; i < tn << (LW + rl + 1); i += kThreads) {
                    int q, b, c, d;
                    bool second;
                    if (!out_element(i, t0, b0, bt, rl, q, second, b, c, d)) continue;
                    const int at = (b0 + b) * p.dm + d;
                    const bool kept = i == tid && t0 == 0 && b0 == 0;
                    const float v = (kept ? own : __ldcg(p.res + at)) + total(tn, q, second, b, c);
                    if (kept) own = v;
                    put(p.r_x + at, __float_as_uint(v), tag_of(l));
                    if (!kept || l == p.L - 1) p.res[at] = v;
                }
                if (t0 + 2 * PP < n || b0 + BT < p.B) sync();
            }
        }
    }

    // ---- tied head: logits[b][v] = act . emb[v]; the best (value, index) of this CTA per sequence ----
    __device__ void head() {
        const Tact* emb = static_cast<const Tact*>(p.lp) + p.o_emb;
        Tact* lg = static_cast<Tact*>(p.logits);
        float* rv = reinterpret_cast<float*>(sm + p.s_red);
        int* ri = reinterpret_cast<int*>(rv + kWarps * 32);
        constexpr int HB = H ? 32 : 8;  // sequences per pass over the table
        const int ld = p.kp1 + TW;
        for (int b0 = 0; b0 < p.B; b0 += HB) {
            const int bt = min(HB, p.B - b0);
            sync();
            norm_rows(p.master + p.o_normf, b0, bt, p.kp1, tag_of(p.L - 1));
            meet();
            if (!alive) return;
            if constexpr (H) {
                const int g = lane >> 2, q = lane & 3, nt = (bt + 7) / 8;
                float bv[4][2];
                int bi[4][2];
#pragma unroll
                for (int t = 0; t < 4; ++t)
#pragma unroll
                    for (int e = 0; e < 2; ++e) { bv[t][e] = -INFINITY; bi[t][e] = 0x7fffffff; }
                const Tact* ar = reinterpret_cast<const Tact*>(sm + p.s_act) + g * ld + 8 * q;
                const int nb = p.kp1 / 32;
                // U blocks of 32 columns of a 16-row tile are requested while the U before them are multiplied;
                // the walk goes on into the warp's next tile, so 2 U to 4 U loads a lane are always in flight
                constexpr int U = 3;
                const int stride = ncta * kWarps;
                int lt = warp * ncta + cta, lk = 0;  // what is requested next (a round's tiles go around the CTAs first)
                auto request = [&](uint4 (*x)[2]) {
                    if (lt * 16 < p.V) {
                        const Tact* w0 = emb + static_cast<long long>(min(lt * 16 + g, p.V - 1)) * p.dm + 8 * q;
                        const Tact* w1 = emb + static_cast<long long>(min(lt * 16 + g + 8, p.V - 1)) * p.dm + 8 * q;
#pragma unroll
                        for (int i = 0; i < U; ++i) {
                            x[i][0] = x[i][1] = make_uint4(0, 0, 0, 0);
                            if ((lk + i) * 32 + 8 * q < p.dm) {
                                x[i][0] = __ldg(reinterpret_cast<const uint4*>(w0 + (lk + i) * 32));
                                x[i][1] = __ldg(reinterpret_cast<const uint4*>(w1 + (lk + i) * 32));
                            }
                        }
                        lk += U;
                        if (lk >= nb) { lk = 0; lt += stride; }
                    }
                };
                float c[4][4];
                auto multiply = [&](int kb, uint4 (*x)[2]) {
#pragma unroll
                    for (int i = 0; i < U; ++i)
                        if (kb + i < nb) {
#pragma unroll
                            for (int t = 0; t < 4; ++t)
                                if (t < nt) {
                                    const uint4 a = *reinterpret_cast<const uint4*>(ar + t * 8 * ld + (kb + i) * 32);
                                    mma16816<Tact>(c[t], x[i][0].x, x[i][1].x, x[i][0].y, x[i][1].y, a.x, a.y);
                                    mma16816<Tact>(c[t], x[i][0].z, x[i][1].z, x[i][0].w, x[i][1].w, a.z, a.w);
                                }
                        }
                };
                uint4 xa[U][2], xb[U][2];
                bool first = true;
                request(xa);
                for (int tile = warp * ncta + cta; tile * 16 < p.V; tile += stride) {
                    const int v0 = tile * 16 + g, v1 = v0 + 8;
#pragma unroll
                    for (int t = 0; t < 4; ++t)
#pragma unroll
                        for (int e = 0; e < 4; ++e) c[t][e] = 0.0f;
                    for (int kb = 0; kb < nb; kb += U, first = !first) {
                        if (first) { request(xb); multiply(kb, xa); }
                        else { request(xa); multiply(kb, xb); }
                    }
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        if (t < nt)
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const int v = e < 2 ? v0 : v1, b = t * 8 + 2 * q + (e & 1);
                                if (v < p.V && b < bt) {
                                    const Tact o = from_f<Tact>(c[t][e]);
                                    lg[static_cast<long long>(b0 + b) * p.V + v] = o;
                                    if (better(to_f(o), v, bv[t][e & 1], bi[t][e & 1])) { bv[t][e & 1] = to_f(o); bi[t][e & 1] = v; }
                                }
                            }
                }
#pragma unroll
                for (int t = 0; t < 4; ++t)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
#pragma unroll
                        for (int m = 4; m <= 16; m <<= 1) {
                            const float ov = __shfl_xor_sync(0xffffffffu, bv[t][e], m);
                            const int oi = __shfl_xor_sync(0xffffffffu, bi[t][e], m);
                            if (better(ov, oi, bv[t][e], bi[t][e])) { bv[t][e] = ov; bi[t][e] = oi; }
                        }
                        if (g == 0) { rv[warp * 32 + t * 8 + 2 * q + e] = bv[t][e]; ri[warp * 32 + t * 8 + 2 * q + e] = bi[t][e]; }
                    }
            } else {
                const float* act = reinterpret_cast<const float*>(sm + p.s_act);
                float bv = -INFINITY;
                int bi = 0x7fffffff;
                for (int tile = warp * ncta + cta; tile * 4 < p.V; tile += ncta * kWarps) {
                    float acc[32];
#pragma unroll
                    for (int i = 0; i < 32; ++i) acc[i] = 0.0f;
                    for (int k = 4 * lane; k < p.dm; k += 128) {
                        float4 w[4];
#pragma unroll
                        for (int r = 0; r < 4; ++r)
                            w[r] = __ldg(reinterpret_cast<const float4*>(
                                reinterpret_cast<const float*>(emb) + static_cast<long long>(min(tile * 4 + r, p.V - 1)) * p.dm + k));
#pragma unroll
                        for (int b = 0; b < 8; ++b) {
                            const float4 a = *reinterpret_cast<const float4*>(act + b * ld + k);
#pragma unroll
                            for (int r = 0; r < 4; ++r)
                                acc[4 * b + r] = fmaf(a.x, w[r].x, fmaf(a.y, w[r].y, fmaf(a.z, w[r].z, fmaf(a.w, w[r].w, acc[4 * b + r]))));
                        }
                    }
                    const float o = sum32(acc, lane);
                    const int v = tile * 4 + (lane & 3), b = lane >> 2;
                    if (v < p.V && b < bt) {
                        lg[static_cast<long long>(b0 + b) * p.V + v] = from_f<Tact>(o);
                        if (better(o, v, bv, bi)) { bv = o; bi = v; }
                    }
                }
#pragma unroll
                for (int m = 1; m <= 2; m <<= 1) {
                    const float ov = __shfl_xor_sync(0xffffffffu, bv, m);
                    const int oi = __shfl_xor_sync(0xffffffffu, bi, m);
                    if (better(ov, oi, bv, bi)) { bv = ov; bi = oi; }
                }
                if ((lane & 3) == 0) { rv[warp * 32 + (lane >> 2)] = bv; ri[warp * 32 + (lane >> 2)] = bi; }
            }
            sync();
            if (tid < bt) {
                float v = rv[tid];
                int i = ri[tid];
                for (int w = 1; w < kWarps; ++w)
                    if (better(rv[w * 32 + tid], ri[w * 32 + tid], v, i)) { v = rv[w * 32 + tid]; i = ri[w * 32 + tid]; }
                uint2* o = reinterpret_cast<uint2*>(p.a_x + static_cast<long long>(b0 + tid) * ncta + cta);
                put(o, __float_as_uint(v), tag_of(p.L));
                put(o + 1, static_cast<uint32_t>(i), tag_of(p.L));
            }
        }
    }
    __device__ void choose() {
        for (int b = cta; b < p.B; b += ncta)
            if (warp == 0) {
                float v = -INFINITY;
                int i = 0x7fffffff;
                for (int c0 = 0; c0 < ncta; c0 += 4 * 32) {
                    uint4 q[4];
                    take<4>(p.a_x + static_cast<long long>(b) * ncta, c0 + lane, 32, ncta - 1, tag_of(p.L), q);
#pragma unroll
                    for (int k = 0; k < 4; ++k)  // (the last one again past the end: it wins nothing twice)
                        if (better(__uint_as_float(q[k].x), static_cast<int>(q[k].z), v, i)) {
                            v = __uint_as_float(q[k].x);
                            i = static_cast<int>(q[k].z);
                        }
                }
#pragma unroll
                for (int m = 16; m >= 1; m >>= 1) {
                    const float ov = __shfl_xor_sync(0xffffffffu, v, m);
                    const int oi = __shfl_xor_sync(0xffffffffu, i, m);
                    if (better(ov, oi, v, i)) { v = ov; i = oi; }
                }
                if (lane == 0 && alive) {
                    if (p.tokens) p.tokens[b * p.tok_ld] = p.next_ids[b];
                    p.next_ids[b] = i;
                }
            }
    }
    __device__ void final_norm() {  // one row per CTA and pass, through the A-operand tile
        for (int b = cta; b < p.B; b += ncta) {
            norm_rows(p.master + p.o_normf, b, 1, p.kp1, tag_of(p.L - 1));
            meet();
            if (!alive) return;
            const Tact* act = reinterpret_cast<const Tact*>(sm + p.s_act);
            for (int k = tid; k < p.dm; k += kThreads) static_cast<Tact*>(p.out)[static_cast<long long>(b) * p.dm + k] = act[k];
            sync();
        }
    }

    __device__ void run() {
        const volatile unsigned* ctl = p.ctl;
        base_tag = ctl[0];
        float own = 0.0f;
        enter(own);
        const int n = channels(), per = p.ncg * 4;
        Place at;
        at.b = n > 0 && (tid >> 2) < p.B * n ? (tid >> 2) / n : 0;
        at.c = n > 0 && (tid >> 2) < p.B * n ? (tid >> 2) - at.b * n : 0;
        at.row = tid / per;
        at.col = 2 * (tid - at.row * per);
        if (!p.x_tma) {
            // columns past the last are never filled: their sums are handed over, though nobody reads them
            for (int i = tid; i < p.kslice * 8; i += kThreads) reinterpret_cast<Tact*>(sm + p.s_wx)[i] = from_f<Tact>(0.0f);
            sync();
            x_weights(0, unit0());
        }
        if (!p.dt_tma) dt_weights(0);
        if (!p.x_tma || !p.dt_tma) sync();
#pragma unroll 1
        for (int l = 0; l < p.L; ++l) {
            in_proj(l);
            if (!alive) break;
            x_proj(l);
            if (!alive) break;
            scan(l, at);
            if (!alive) break;
            sync();  // the operands of the scan and of phase 1 have been read
            release(kSmall);
            if (!p.dt_tma) dt_weights(l + 1);
            out_proj(l, own);
            if (!alive) break;
        }
        if (alive && p.next_ids) {
            head();
            if (alive) choose();
        } else if (alive) {
            final_norm();
        }
        meet();
        if (!alive) *dead = 1;
        // the last CTA to get here (all have read the tag base) hands the next launch tags of its own; a CTA that
        // has given up counts like any other, or the next launch would take this one's words for its own
        if (tid == 0) {
            __threadfence();
            if (atomicAdd(p.ctl + 1, 1u) == static_cast<unsigned>(ncta) - 1) {
                p.ctl[0] = base_tag + p.L + 2;
                p.ctl[1] = 0;
            }
        }
    }
};

template <typename Tact>
__global__ void __launch_bounds__(kThreads + 32, 1) decode_step_kernel(const __grid_constant__ Params p) {
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ float pair[kWarps];
    __shared__ int dead[2];
    __shared__ __align__(8) uint64_t bars[8];
    if (threadIdx.x == 0) {
        for (int i = 0; i < 8; ++i) mbar_init(&bars[i], 1);
        dead[0] = 0;
        const unsigned limit = *reinterpret_cast<const volatile unsigned*>(p.ctl + 2);
        dead[1] = limit > 0 && limit < static_cast<unsigned>(kMaxPolls) ? static_cast<int>(limit) : kMaxPolls;
        fence_barrier_init();
    }
    __syncthreads();
    Step<Tact> s(p, sm, pair, bars, dead);
    if (threadIdx.x >= kThreads) s.feed();
    else s.run();
}

}  // namespace dec

int decode_configure(Ctx* c) {
    const void* fns[3] = {reinterpret_cast<const void*>(dec::decode_step_kernel<float>),
                          reinterpret_cast<const void*>(dec::decode_step_kernel<__half>),
                          reinterpret_cast<const void*>(dec::decode_step_kernel<__nv_bfloat16>)};
    for (const void* fn : fns)
        MB200_CUDA_CHECK(c, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - 1024));
    return MAMBA_B200_OK;
}

// Splits the phases over the CTAs and lays out shared memory and the workspace.  Returns the
// number of CTAs, or 0 when the kernel does not take this model: d_state 16 and d_conv 4 (every
// Mamba-1 checkpoint), d_model a multiple of 8 up to 1024 (16-byte rows; a row of the residual in
// one warp's registers), at most 64 sequences (beyond that a library GEMM per projection has
// enough work), and two projection tiles that fit shared memory beside the operand rows.
static int plan(int sms, const mamba_b200_decode_args& a, dec::Params& p, long long* ws_bytes, uint32_t* smem) {
    using namespace dec;
    if (a.N != kN || a.K != kK || a.d_model % 8 != 0 || a.d_model < 8 || a.d_model > kMaxDm || a.B < 1 || a.B > kMaxB ||
        a.d_inner % 16 != 0 || a.dt_rank < 1 || a.dt_rank > 1024 || a.n_layers < 1)
        return 0;
    const bool half = a.dtype != MAMBA_B200_F32;
    const int es = half ? 2 : 4, tw = 16 / es, bt = half ? 16 : 8;
    p.B = a.B; p.dm = a.d_model; p.di = a.d_inner; p.dr = a.dt_rank; p.xd = a.dt_rank + 2 * kN; p.L = a.n_layers;
    p.kp1 = (p.dm + 31) / 32 * 32;
    p.kp4 = (p.di + 31) / 32 * 32;
    p.ncg = (p.xd + 7) / 8;
    const int tiles1 = p.di / tw, tiles4 = p.dm / tw;
    int grid = tiles1 > kMaxKs * p.ncg ? tiles1 : kMaxKs * p.ncg;
    if (grid > sms || a.vocab > 0) grid = sms;
    auto tiles = [](int n, int g, int kp, int& per, int& c, int& ka, int& br) {
        per = (n + g - 1) / g;
        for (c = per; c % 2 == 0;) c /= 2;
        const int boxes = (kp + 255) / 256;
        br = ((kp + boxes - 1) / boxes + 7) / 8 * 8;
        ka = br * boxes;
    };
    tiles(tiles1, grid, p.kp1, p.t1, p.c1, p.ka1, p.br1);
    tiles(tiles4, grid, p.kp4, p.t4, p.c4, p.ka4, p.br4);
    if (p.c1 * tw > 256 || p.c4 * tw > 256) return 0;
    p.nch = p.t1 * tw;
    if (p.nch > 256) return 0;
    // enough slices to use the CTAs, few enough that adding them up stays short
    int ks = grid / p.ncg;
    ks = ks < 1 ? 1 : ks > kMaxKs ? kMaxKs : ks;
    int sl = ((p.di + ks - 1) / ks + 15) / 16 * 16;
    if (sl > kMaxKSlice) sl = kMaxKSlice;
    p.kslice = sl;
    p.ks = (p.di + sl - 1) / sl;
    p.brx = sl > 256 ? sl / 2 : sl;
    const int dboxes = (p.dr + 255) / 256;
    p.brd = ((p.dr + dboxes - 1) / dboxes + 7) / 8 * 8;
    auto up = [](long long v) { return (v + 15) / 16 * 16; };
    const int rows = p.B < bt ? p.B : bt, hrows = half ? (p.B < 8 ? 8 : p.B < 32 ? (p.B + 7) / 8 * 8 : 32) : 8;
    long long act = static_cast<long long>(rows) * ((p.kp4 > p.kp1 ? p.kp4 : p.kp1) + tw) * es;
    if (a.vocab > 0) {
        const long long h = static_cast<long long>(hrows) * (p.kp1 + tw) * es;
        act = act > h ? act : h;
    }
    const long long us = static_cast<long long>(bt) * (p.kslice + tw) * es, xs = static_cast<long long>(p.B) * p.xd * 4;
    act = act > us ? act : us;
    act = act > xs ? act : xs;
    auto up128 = [](long long v) { return (v + 127) / 128 * 128; };
    long long o = 0;
    p.s_w1 = o; o += up128(2LL * p.t1 * p.ka1 * 16);
    p.s_w4 = o; o += up128(static_cast<long long>(p.t4) * p.ka4 * 16);
    p.s_wx = o; o += up128(static_cast<long long>(p.kslice) * 8 * es);
    p.s_wd = o; o += up128(static_cast<long long>(dboxes) * p.brd * p.nch * es);
    p.s_act = o; o += up(act);
    p.s_red = o; o += up(half ? kWarps * 2 * 160 * 4 : kWarps * 2 * 32 * 4);
    p.s_norm = o; o += up(static_cast<long long>(p.dm) * 4);
    p.s_conv = o; o += up(static_cast<long long>(p.nch) * (16LL * (p.B + 1) + 4));
    p.s_uz = o; o += up(8LL * p.B * p.nch);
    p.s_a = o; o += up(p.nch * (kN * 4 + 4 + es));
    if (o > 227 * 1024 - 1024) return 0;
    *smem = static_cast<uint32_t>(o);
    const long long Bl = p.B;
    *ws_bytes = 256 + 2 * up(Bl * p.di * 2 * es) + up(8 * Bl * p.dm) + up(64LL * p.ks * Bl * p.ncg) + 16 * Bl * sms;
    return grid;
}

}  // namespace mb200

using namespace mb200;

extern "C" MAMBA_B200_API long long mamba_b200_decode_workspace_bytes(void* handle, const mamba_b200_decode_args* a) {
    Ctx* c = static_cast<Ctx*>(handle);
    if (!c || !a || !dtype_ok(a->dtype)) return 0;
    dec::Params p;
    memset(&p, 0, sizeof(p));
    long long ws = 0;
    uint32_t smem = 0;
    return plan(c->sm_count, *a, p, &ws, &smem) ? ws : 0;
}

extern "C" MAMBA_B200_API int mamba_b200_decode_step(void* handle, void* stream, const mamba_b200_decode_args* ap) {
    Ctx* c = static_cast<Ctx*>(handle);
    if (!c) return MAMBA_B200_ERR_ARG;
    if (!ap) return fail(c, MAMBA_B200_ERR_ARG, "decode_step: null args");
    const mamba_b200_decode_args& a = *ap;
    if (!dtype_ok(a.dtype)) return fail(c, MAMBA_B200_ERR_ARG, "decode_step: bad dtype %d", a.dtype);
    const bool lm = a.next_ids != nullptr;
    if (!a.lp || !a.master || !a.a_neg || !a.conv_state || !a.ssm_state || !a.residual || !a.workspace ||
        (lm ? !a.logits || a.vocab < 1 : !a.out))
        return fail(c, MAMBA_B200_ERR_ARG, "decode_step: null required pointer");
    if (a.batch_capacity < a.B) return fail(c, MAMBA_B200_ERR_ARG, "decode_step: state holds %d sequences, %d given", a.batch_capacity, a.B);
    dec::Params p;
    memset(&p, 0, sizeof(p));
    long long ws = 0;
    uint32_t smem = 0;
    const int grid = plan(c->sm_count, a, p, &ws, &smem);
    if (!grid) return fail(c, MAMBA_B200_ERR_SHAPE, "decode_step: this model or batch is not taken (see mamba_b200_decode_workspace_bytes)");
    if (a.workspace_bytes < ws) return fail(c, MAMBA_B200_ERR_ARG, "decode_step: workspace %lld < %lld bytes", a.workspace_bytes, ws);
    const void* al[8] = {a.lp, a.master, a.a_neg, a.conv_state, a.ssm_state, a.residual, a.workspace, lm ? a.logits : a.out};
    for (int i = 0; i < 7; ++i)
        if (reinterpret_cast<uintptr_t>(al[i]) & 15) return fail(c, MAMBA_B200_ERR_ARG, "decode_step: pointer %d is not 16-byte aligned", i);
    const long long offs[] = {a.layer_stride, a.o_in_proj, a.o_conv_w, a.o_conv_b, a.o_dt_proj_b, a.o_d_param, a.o_out_proj, a.o_norm_f, lm ? a.o_embedding : 0};
    for (long long v : offs)
        if (v % 8 != 0) return fail(c, MAMBA_B200_ERR_ARG, "decode_step: arena offsets must be multiples of 8 elements");
    p.lp = a.lp; p.master = a.master; p.a_neg = a.a_neg; p.lstride = a.layer_stride;
    p.o_in = a.o_in_proj; p.o_cw = a.o_conv_w; p.o_cb = a.o_conv_b; p.o_x = a.o_x_proj; p.o_dtw = a.o_dt_proj_w;
    p.o_dtb = a.o_dt_proj_b; p.o_D = a.o_d_param; p.o_out = a.o_out_proj; p.o_normf = a.o_norm_f; p.o_emb = a.o_embedding;
    p.conv = a.conv_state; p.ssm = a.ssm_state; p.res = a.residual; p.Bcap = a.batch_capacity;
    p.out = a.out; p.next_ids = a.next_ids; p.tokens = a.tokens; p.tok_ld = a.tokens_ld; p.logits = a.logits;
    p.V = lm ? a.vocab : 0;
    p.eps = a.eps;
    p.inv_dm = 1.0f / static_cast<float>(a.d_model);
    p.status = c->d_status;
    const int es = static_cast<int>(dtype_size(a.dtype));
    auto up = [](long long v) { return (v + 15) / 16 * 16; };
    unsigned char* w = static_cast<unsigned char*>(a.workspace);
    p.ctl = reinterpret_cast<unsigned*>(w); w += 256;
    p.u_x = reinterpret_cast<uint2*>(w); w += up(static_cast<long long>(p.B) * p.di * 2 * es);
    p.y_x = reinterpret_cast<uint2*>(w); w += up(static_cast<long long>(p.B) * p.di * 2 * es);
    p.r_x = reinterpret_cast<uint2*>(w); w += up(8LL * p.B * p.dm);
    p.p_x = reinterpret_cast<uint2*>(w); w += up(64LL * p.ks * p.B * p.ncg);
    p.a_x = reinterpret_cast<uint4*>(w);
    const unsigned char* lp8 = static_cast<const unsigned char*>(a.lp);
    const int tw = 16 / es;
    if (!make_tmap_stack(c, &p.tm_in, a.dtype, lp8 + p.o_in * es, 2 * p.di, p.dm, p.L, p.lstride, p.c1 * tw, p.br1) ||
        !make_tmap_stack(c, &p.tm_out, a.dtype, lp8 + p.o_out * es, p.dm, p.di, p.L, p.lstride, p.c4 * tw, p.br4))
        return fail(c, MAMBA_B200_ERR_CUDA, "decode_step: the weight tensor maps were refused");
    // rows of W_x or W_dt that do not start on 16 bytes are copied by the compute warps
    p.x_tma = p.ncg * p.ks <= grid && make_tmap_stack(c, &p.tm_x, a.dtype, lp8 + p.o_x * es, p.xd, p.di, p.L, p.lstride, 8, p.brx);
    p.dt_tma = make_tmap_stack(c, &p.tm_dt, a.dtype, lp8 + p.o_dtw * es, p.di, p.dr, p.L, p.lstride, p.nch, p.brd);
    int steps = lm && a.steps > 1 ? a.steps : 1;
    const void* fn = a.dtype == MAMBA_B200_F32   ? reinterpret_cast<const void*>(dec::decode_step_kernel<float>)
                     : a.dtype == MAMBA_B200_F16 ? reinterpret_cast<const void*>(dec::decode_step_kernel<__half>)
                                                 : reinterpret_cast<const void*>(dec::decode_step_kernel<__nv_bfloat16>);
    for (int i = 0; i < steps; ++i) {
        void* args[1] = {&p};
        MB200_CUDA_CHECK(c, cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(dec::kThreads + 32), args, smem, static_cast<cudaStream_t>(stream)));
        if (p.tokens) ++p.tokens;
    }
    return MAMBA_B200_OK;
}
