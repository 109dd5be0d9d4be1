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
// at HBM speed are 0.04 ms.  Here the grid (one CTA per SM) stays resident and meets at four
// barriers a layer:
//   1  act = rmsnorm(residual)  (every CTA for itself);  x | z = act W_in;  u = silu(conv(x))
//   2  slices of x_proj: u W_x over a range of channels  (partial sums, added by their readers)
//   3  delta, SSM step, gate for a range of channels
//   4  residual += y W_out
// A CTA owns the same column tiles (16 bytes wide) of W_in and W_out in every layer and asks for
// the next layer's by TMA as soon as it has finished with this layer's, so weights stream from HBM
// under the other three phases; the small operands of a phase are read a phase or a layer ahead.
// Measured: 0.335 ms a token (130m, batch 8), 38 us a step (d_model 128).  What is left is latency:
// a layer is 24,700 cycles, of which a barrier (release, poll) is 1,700 and the first read of what
// another CTA wrote 900, four times each, and the instructions of the phases themselves, which run
// once per layer: with loops unrolled for more loads in flight the code outgrew the instruction
// cache and a layer took 30,000 cycles, so loops stay rolled and sixteen warps share the work.
// Arithmetic: mma.sync m16n8k16 with the batch as M for 16-bit storage (the tile is 8 columns;
// tcgen05's 128-row tiles would be mostly padding at these batch sizes and the products are not
// what takes the time), FMA for f32.  Sums are f32 in a fixed order: two runs are bit-identical.
#include <string.h>

#include <type_traits>

#include "common.cuh"
#include "internal.h"

namespace mb200 {
namespace dec {

constexpr int kThreads = 512, kWarps = 16;
constexpr int kN = 16, kK = 4;          // d_state and d_conv of this kernel
constexpr int kMaxDm = 1024, kMaxB = 64, kMaxKSlice = 192, kMaxKs = 8;
constexpr int kTC = 4;                  // column tiles accumulated together
constexpr int kMaxPolls = 1 << 22;      // a barrier poll is about a microsecond's L2 round trip

struct Params {
    CUtensorMap tm_in, tm_out;          // W_in, W_out of all layers: [L, K, columns]
    const void* lp;                     // compute-dtype arena
    const float *master, *a_neg;        // f32 arena, [L, di, N]
    long long lstride;                  // elements from one layer to the next (both arenas)
    long long o_in, o_cw, o_cb, o_x, o_dtw, o_dtb, o_D, o_out, o_normf, o_emb;
    float *conv, *ssm;                  // [L, Bcap, di, K], [L, Bcap, di, N]
    float* res;                         // [B, dm] residual stream
    float *z, *xpart, *amax_v;          // workspace
    int* amax_i;
    void *u, *y;
    unsigned* bar;                      // [0] arrivals, [1] exits; zero between launches
    void* out;                          // backbone: rmsnorm(residual) in the compute dtype
    int *next_ids, *tokens;             // LM: ids in / next ids out; tokens[b * tok_ld] = id taken in
    long long tok_ld;
    void* logits;                       // LM: [B, V]
    int B, Bcap, dm, di, dr, xd, L, V;
    float eps, inv_dm;
    // in_proj / out_proj: column tiles per CTA, padded K, and how they lie in shared memory: chunks of
    // c tiles (odd, so that rows of c * 16 bytes meet different banks), ka rows each, from TMA boxes of br rows
    int t1, c1, kp1, ka1, br1;
    int t4, c4, kp4, ka4, br4;
    int ncg, ks, kslice, nch;           // x_proj: column groups, K slices; scan channels per CTA
    uint32_t s_w1, s_w4, s_act, s_red, s_wx, s_wd, s_norm, s_conv;
    int* status;
};

__device__ __forceinline__ void cp16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp4(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void l2_prefetch(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x2_trans(uint32_t addr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr));
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
// Data that other CTAs of this launch write: read past L1.
__device__ __forceinline__ float4 ldcg4(const float* p) { return __ldcg(reinterpret_cast<const float4*>(p)); }
template <typename Tact>
__device__ __forceinline__ Tact ldcg_raw(const Tact* p) {
    if constexpr (sizeof(Tact) == 4) {
        return __ldcg(p);
    } else {
        const unsigned short w = __ldcg(reinterpret_cast<const unsigned short*>(p));
        return *reinterpret_cast<const Tact*>(&w);
    }
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
    static constexpr int BT = H ? 16 : 8;         // sequences per pass of a projection
    const Params& p;
    unsigned char* sm;
    const int tid, lane, warp, cta, ncta;
    unsigned epoch = 0;
    bool alive = true;
    int* flag;
    uint64_t* bars;  // W_in and W_out tiles have landed

    __device__ Step(const Params& p_, unsigned char* sm_, int* flag_, uint64_t* bars_)
        : p(p_), sm(sm_), tid(threadIdx.x), lane(threadIdx.x & 31), warp(threadIdx.x >> 5), cta(blockIdx.x),
          ncta(gridDim.x), flag(flag_), bars(bars_) {}

    __device__ const Tact* lp(int l, long long off) const { return static_cast<const Tact*>(p.lp) + l * p.lstride + off; }
    __device__ const float* mf(int l, long long off) const { return p.master + l * p.lstride + off; }

    // ---- grid barrier in two halves; what needs no other CTA's data goes in between ----
    __device__ void arrive() {
        __syncthreads();
        epoch += ncta;
        if (tid == 0) {  // the release covers what the CTA's other threads wrote before the block barrier
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p.bar) : "memory");
        }
    }
    __device__ void wait() {
        if (tid == 0) {
            unsigned v = 0;
            int it = 0;
            do {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p.bar) : "memory");
            } while (v < epoch && ++it < kMaxPolls);
            *flag = v >= epoch;
            if (v < epoch) atomicCAS(p.status, kStatusOk, kStatusBarrierTimeout);
        }
        __syncthreads();
        alive = *flag != 0;
    }

    // ---- weights of a projection: this CTA's column tiles, landed by TMA ----
    __device__ void fetch(const CUtensorMap* map, uint64_t* bar, uint32_t dst, int l, int tiles, int per, int c, int ka, int br) {
        const int first = cta * per;
        if (tid != 0 || l >= p.L || first >= tiles) return;  // (another thread would slow the release down: 1100 -> 2500 cycles)
        mbar_expect_tx(bar, static_cast<uint32_t>(per / c) * ka * c * 16);
        for (int q = 0; q < per / c; ++q)
            for (int k = 0; k < ka; k += br)
                tma_load_3d(sm + dst + static_cast<uint32_t>(q * ka + k) * c * 16, map, bar, (first + q * c) * TW, k, l);
    }
    __device__ void fetch_in(int l) { fetch(&p.tm_in, &bars[0], p.s_w1, l, 2 * p.di / TW, p.t1, p.c1, p.ka1, p.br1); }
    __device__ void fetch_out(int l) { fetch(&p.tm_out, &bars[1], p.s_w4, l, p.dm / TW, p.t4, p.c4, p.ka4, p.br4); }

    // ---- what phase 1 of layer l reads besides: norm weights; conv windows, taps and bias of the
    //      CTA's x columns (window rows [B][columns], then taps, then bias) ----
    __device__ int x_columns() const { return max(0, min(p.t1 * TW, p.di - cta * p.t1 * TW)); }
    __device__ void fetch_small(int l) {
        if (l >= p.L) return;
        const int n = x_columns(), d0 = cta * p.t1 * TW, cols = p.t1 * TW;
        const uint32_t cv = smem_u32(sm + p.s_conv);
        if (warp >= 8) {
            const uint32_t dst = smem_u32(sm + p.s_norm);
#pragma unroll 1
            for (int k = tid - 8 * 32; k < p.dm / 4; k += kThreads / 2) cp16(dst + k * 16, mf(l, 0) + 4 * k);
        } else if (warp == 7) {
#pragma unroll 1
            for (int c = lane; c < n; c += 32) {
                cp16(cv + (p.B * cols + c) * 16, mf(l, p.o_cw) + (d0 + c) * kK);
                if ((c & 3) == 0) cp16(cv + (p.B + 1) * cols * 16 + c * 4, mf(l, p.o_cb) + d0 + c);
            }
        } else {
#pragma unroll 1
            for (int b = warp; b < p.B; b += 7)
#pragma unroll 1
                for (int c = lane; c < n; c += 32)
                    cp16(cv + (b * cols + c) * 16, p.conv + ((static_cast<long long>(l) * p.Bcap + b) * p.di + d0 + c) * kK);
        }
    }
    // the lines of layer l that phases 1-3 of this CTA read, into L2; a warp per kind
    __device__ void hint(int l) {
        if (l >= p.L) return;
        const int ch0 = cta * p.nch, n = min(p.nch, p.di - ch0), m = x_columns(), d0 = cta * p.t1 * TW;
        if (warp == 1 && n > 0) {
#pragma unroll 1
            for (int b = lane; b < p.B; b += 32)
                l2_prefetch_bulk(p.ssm + ((static_cast<long long>(l) * p.Bcap + b) * p.di + ch0) * kN, n * kN * 4);
        } else if (warp == 2 && n > 0) {
            if (lane == 0) l2_prefetch_bulk(p.a_neg + (static_cast<long long>(l) * p.di + ch0) * kN, n * kN * 4);
            if (lane == 1) l2_prefetch(mf(l, p.o_D) + ch0);
            if (lane == 2) l2_prefetch(lp(l, p.o_dtb) + ch0);
            if (lane == 3 && m > 0) l2_prefetch_bulk(mf(l, p.o_cw) + d0 * kK, m * kK * 4);
            if (lane == 4 && m > 0) l2_prefetch(mf(l, p.o_cb) + d0);
            if (lane == 5) l2_prefetch(mf(l, 0) + min(p.dm - 1, cta * 32));
        } else if (warp == 3 && n > 0) {
#pragma unroll 1
            for (int i = lane; i < p.dr; i += 32) l2_prefetch(lp(l, p.o_dtw) + static_cast<long long>(i) * p.di + ch0);
        } else if (warp == 4 && m > 0) {
#pragma unroll 1
            for (int b = lane; b < p.B; b += 32)
                l2_prefetch_bulk(p.conv + ((static_cast<long long>(l) * p.Bcap + b) * p.di + d0) * kK, m * kK * 4);
        } else if (warp >= 8 && cta < p.ncg * p.ks) {
            const int k0 = (cta / p.ncg) * p.kslice, g = cta % p.ncg, i = tid - 8 * 32;
            if (i < min(p.kslice, p.di - k0)) l2_prefetch(lp(l, p.o_x) + static_cast<long long>(k0 + i) * p.xd + g * 8);
        }
    }

    // ---- rows b0 .. b0+bt of rmsnorm(stream) * w as the A operand, a row per warp ----
    template <bool IDS>
    __device__ void norm_rows(const float* w, int b0, int bt, int kp) {
        Tact* act = reinterpret_cast<Tact*>(sm + p.s_act);
        const int ld = kp + TW;
        constexpr int NV = kMaxDm / 128;
#pragma unroll 1
        for (int r = warp; r < bt; r += kWarps) {
            float4 v[NV];
            const Tact* er = nullptr;
            const float* src = p.res + static_cast<long long>(b0 + r) * p.dm + 4 * lane;
            if (IDS) {
                const int id = p.next_ids[b0 + r];
                if (id >= 0 && id < p.V)
                    er = static_cast<const Tact*>(p.lp) + p.o_emb + static_cast<long long>(id) * p.dm + 4 * lane;
            }
            float ss = 0.0f;
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                v[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (128 * i + 4 * lane < p.dm) {
                    if (!IDS) {
                        v[i] = ldcg4(src + 128 * i);
                    } else if (er) {
                        const float2 a = ld_pair(er + 128 * i), b = ld_pair(er + 128 * i + 2);
                        v[i] = make_float4(a.x, a.y, b.x, b.y);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < NV; ++i)
                if (128 * i < p.dm)
                    ss = fmaf(v[i].x, v[i].x, fmaf(v[i].y, v[i].y, fmaf(v[i].z, v[i].z, fmaf(v[i].w, v[i].w, ss))));
#pragma unroll
            for (int m = 16; m >= 1; m >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, m);
            float inv = rsqrtf(fmaf(ss, p.inv_dm, p.eps));
                if (!(inv > 0.0f && inv <= 1e20f)) inv = 1.0f;  // rms not finite or below 1e-20: the norm operator's guard
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const int k = 128 * i + 4 * lane;
                if (k < p.dm) {
                    const float4 g = *reinterpret_cast<const float4*>(w + k);
                    st_pair(act + r * ld + k, make_float2(v[i].x * inv * g.x, v[i].y * inv * g.y));
                    st_pair(act + r * ld + k + 2, make_float2(v[i].z * inv * g.z, v[i].w * inv * g.w));
                }
            }
            if (p.dm + lane < kp) act[r * ld + p.dm + lane] = from_f<Tact>(0.0f);  // kp - dm < 32
        }
    }
    // rows of `src` (K columns, written by other CTAs) as the A operand: a row per warp, eight loads in flight
    __device__ void load_rows(const Tact* src, int K, int kp, int b0, int bt) {
        Tact* act = reinterpret_cast<Tact*>(sm + p.s_act);
        const int ld = kp + TW, per = kp / TW;
#pragma unroll 1
        for (int r = warp; r < bt; r += kWarps)
#pragma unroll 1
            for (int j0 = lane; j0 < per; j0 += 256) {
                uint4 v[8];
                const Tact* row = src + static_cast<long long>(b0 + r) * K + j0 * TW;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    v[i] = make_uint4(0, 0, 0, 0);
                    if ((j0 + 32 * i) * TW < K) v[i] = __ldcg(reinterpret_cast<const uint4*>(row + 32 * i * TW));
                }
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (j0 + 32 * i < per) *reinterpret_cast<uint4*>(act + r * ld + (j0 + 32 * i) * TW) = v[i];
            }
    }

    // ---- out[b][tile][col] = act W for up to kTC tiles; the warps split K, partials in s_red.  Loops stay
    //      rolled: a layer's worth of code runs once per layer and has to stay in the instruction cache ----
    __device__ void project(uint32_t wofs, int kp, int ka, int cw, int tile0, int n, int rows) {
        float* red = reinterpret_cast<float*>(sm + p.s_red);
        const int ld = kp + TW;
        if constexpr (H) {
            float c[kTC][4];
#pragma unroll
            for (int t = 0; t < kTC; ++t)
#pragma unroll
                for (int i = 0; i < 4; ++i) c[t][i] = 0.0f;
            const uint32_t arow = smem_u32(sm + p.s_act) + (min(lane & 15, rows - 1) * ld + (lane >> 4) * 8) * 2;
            uint32_t brow[kTC];
            int q = tile0 / cw, w = tile0 - q * cw;
#pragma unroll
            for (int t = 0; t < kTC; ++t) {
                brow[t] = smem_u32(sm + wofs) + static_cast<uint32_t>(((q * ka + (lane & 15)) * cw + w) * 16);
                if (++w == cw) { w = 0; ++q; }
            }
#pragma unroll 1
            for (int s = warp; s < kp / 16; s += kWarps) {
                uint32_t a[4], b[kTC][2];
                ldmatrix_x4(arow + s * 32, a);
#pragma unroll
                for (int t = 0; t < kTC; ++t)
                    if (t < n) ldmatrix_x2_trans(brow[t] + static_cast<uint32_t>(s * 256 * cw), b[t]);
#pragma unroll
                for (int t = 0; t < kTC; ++t)
                    if (t < n) mma16816<Tact>(c[t], a[0], a[1], a[2], a[3], b[t][0], b[t][1]);
            }
            const int g = lane >> 2, e = lane & 3;
#pragma unroll
            for (int t = 0; t < kTC; ++t)
                if (t < n) {
                    float* o = red + (warp * kTC + t) * (BT * TW);
                    *reinterpret_cast<float2*>(o + g * TW + 2 * e) = make_float2(c[t][0], c[t][1]);
                    *reinterpret_cast<float2*>(o + (g + 8) * TW + 2 * e) = make_float2(c[t][2], c[t][3]);
                }
        } else {
            const float* act = reinterpret_cast<const float*>(sm + p.s_act);
            if (warp * 32 >= kp) return;  // total() knows
#pragma unroll 1
            for (int t = 0; t < n; ++t) {
                float acc[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) acc[i] = 0.0f;
                const int q = (tile0 + t) / cw;
                const float4* w = reinterpret_cast<const float4*>(sm + wofs) + q * ka * cw + (tile0 + t - q * cw);
#pragma unroll 1
                for (int k = warp * 32 + lane; k < kp; k += kThreads) {
                    const float4 wv = w[k * cw];
#pragma unroll
                    for (int b = 0; b < BT; ++b) {
                        const float a = act[min(b, rows - 1) * ld + k];
                        acc[4 * b] = fmaf(a, wv.x, acc[4 * b]);
                        acc[4 * b + 1] = fmaf(a, wv.y, acc[4 * b + 1]);
                        acc[4 * b + 2] = fmaf(a, wv.z, acc[4 * b + 2]);
                        acc[4 * b + 3] = fmaf(a, wv.w, acc[4 * b + 3]);
                    }
                }
                red[(warp * kTC + t) * (BT * TW) + lane] = sum32(acc, lane);
            }
        }
    }
    __device__ float total(int t, int b, int c, int kp) const {
        const float* o = reinterpret_cast<const float*>(sm + p.s_red) + t * (BT * TW) + b * TW + c;
        const int parts = H ? kWarps : min(kWarps, kp / 32);
        float s = o[0];
#pragma unroll
        for (int w = 1; w < kWarps; ++w)
            if (H || w < parts) s += o[w * kTC * BT * TW];
        return s;
    }

    // ---- phase 1 ----
    __device__ void in_proj(int l) {
        const int tiles = 2 * p.di / TW, first = cta * p.t1, n = min(p.t1, tiles - first);
        if (n <= 0) return;
        const int cols = p.t1 * TW;
        const float4* win_s = reinterpret_cast<const float4*>(sm + p.s_conv);
        const float4* tap_s = win_s + p.B * cols;
        const float* cb_s = reinterpret_cast<const float*>(tap_s + cols);
#pragma unroll 1
        for (int b0 = 0; b0 < p.B; b0 += BT) {
            const int bt = min(BT, p.B - b0);
            if (l == 0 && p.next_ids) norm_rows<true>(reinterpret_cast<const float*>(sm + p.s_norm), b0, bt, p.kp1);
            else norm_rows<false>(reinterpret_cast<const float*>(sm + p.s_norm), b0, bt, p.kp1);
            __syncthreads();
            if (b0 == 0) alive = mbar_wait(&bars[0], l & 1, p.status) && alive;
#pragma unroll 1
            for (int t0 = 0; t0 < n; t0 += kTC) {
                const int tn = min(kTC, n - t0);
                project(p.s_w1, p.kp1, p.ka1, p.c1, t0, tn, bt);
                __syncthreads();
                // TW columns x BT rows of a tile on consecutive threads (rows past the batch idle)
#pragma unroll 1
                for (int i = tid; i < tn * BT * TW; i += kThreads) {
                    const int c = i % TW, b = (i / TW) % BT, t = i / (TW * BT);
                    if (b >= bt) continue;
                    const int cc = (t0 + t) * TW + c, d = first * TW + cc;
                    // the projection leaves in the storage dtype, as the x | z halves do elsewhere
                    const float v = to_f(from_f<Tact>(total(t, b, c, p.kp1)));
                    if (d < p.di) {
                        const float4 win = win_s[(b0 + b) * cols + cc], cw = tap_s[cc];
                        const float acc = fmaf(v, cw.w, fmaf(win.w, cw.z, fmaf(win.z, cw.y, fmaf(win.y, cw.x, cb_s[cc]))));
                        *reinterpret_cast<float4*>(p.conv + ((static_cast<long long>(l) * p.Bcap + b0 + b) * p.di + d) * kK) =
                            make_float4(win.y, win.z, win.w, v);
                        static_cast<Tact*>(p.u)[static_cast<long long>(b0 + b) * p.di + d] = from_f<Tact>(siluf_fast(acc));
                    } else {
                        p.z[static_cast<long long>(b0 + b) * p.di + d - p.di] = v;
                    }
                }
                if (t0 + kTC < n || b0 + BT < p.B) __syncthreads();
            }
        }
    }

    // ---- phase 2: partial sums of x_proj over a slice of channels, eight columns a unit ----
    // (asynchronous 4-byte copies where a row of W_x starts on 4 bytes, plain loads otherwise)
    __device__ void x_weights(int l, int unit) {
        if (l >= p.L || unit >= p.ncg * p.ks) return;
        Tact* w2 = reinterpret_cast<Tact*>(sm + p.s_wx);
        const int k0 = (unit / p.ncg) * p.kslice, c0 = (unit % p.ncg) * 8, nk = min(p.kslice, p.di - k0);
        const Tact* w = lp(l, p.o_x) + static_cast<long long>(k0) * p.xd + c0;
        constexpr int E = 4 / sizeof(Tact), PR = 8 / E;  // elements of a copy, copies of a row
        if (p.xd % E == 0) {
            const int c = tid % PR;
            if (c0 + c * E < p.xd)
#pragma unroll 1
                for (int k = tid / PR; k < nk; k += kThreads / PR)
                    cp4(smem_u32(w2 + k * 8 + c * E), w + static_cast<long long>(k) * p.xd + c * E);
        } else {
            constexpr int NI = kMaxKSlice / (kThreads / 8);
            Tact v[NI];
            const int c = tid & 7;
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const int k = (tid >> 3) + kThreads / 8 * i;
                if (k < nk && c0 + c < p.xd) v[i] = w[static_cast<long long>(k) * p.xd + c];
            }
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const int k = (tid >> 3) + kThreads / 8 * i;
                if (k < nk && c0 + c < p.xd) w2[k * 8 + c] = v[i];
            }
        }
    }
    __device__ void x_proj(int l) {
        const Tact* w2 = reinterpret_cast<const Tact*>(sm + p.s_wx);
        Tact* us = reinterpret_cast<Tact*>(sm + p.s_act);
        float* red = reinterpret_cast<float*>(sm + p.s_red);
        const int uld = p.kslice + TW;
        for (int unit = cta; unit < p.ncg * p.ks; unit += ncta) {
            if (unit != cta) {
                __syncthreads();
                x_weights(l, unit);
                cp_wait_all();
            }
            const int s = unit / p.ncg, k0 = s * p.kslice, g = unit - s * p.ncg;
    #pragma unroll 1
        for (int b0 = 0; b0 < p.B; b0 += BT) {
                const int bt = min(BT, p.B - b0);
                constexpr int CH = kThreads / BT;  // a thread per 16-byte piece of the slice
                static_assert(CH * TW >= kMaxKSlice, "slice");
                {
                    const int b = tid / CH, k = (tid % CH) * TW;
                    if (k < p.kslice) {
                        uint4 v = make_uint4(0, 0, 0, 0);
                        if (b < bt && k0 + k < p.di)
                            v = __ldcg(reinterpret_cast<const uint4*>(static_cast<const Tact*>(p.u) +
                                                                      static_cast<long long>(b0 + b) * p.di + k0 + k));
                        *reinterpret_cast<uint4*>(us + b * uld + k) = v;
                    }
                }
                __syncthreads();
                float* out = p.xpart + (static_cast<long long>(s) * p.B + b0) * p.xd + g * 8;
                if constexpr (H) {
                    float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                    const uint32_t arow = smem_u32(us) + ((lane & 15) * uld + (lane >> 4) * 8) * 2;
                    const uint32_t brow = smem_u32(w2) + (lane & 15) * 16;
                    static_assert(kMaxKSlice / 16 <= kWarps, "a K step per warp");
                    const int k = warp;
                    if (k < p.kslice / 16) {
                        uint32_t a[4], b[2];
                        ldmatrix_x4(arow + k * 32, a);
                        ldmatrix_x2_trans(brow + k * 256, b);
                        mma16816<Tact>(c, a[0], a[1], a[2], a[3], b[0], b[1]);
                    }
                    float* o = red + warp * 128 + (lane >> 2) * 8 + 2 * (lane & 3);
                    *reinterpret_cast<float2*>(o) = make_float2(c[0], c[1]);
                    *reinterpret_cast<float2*>(o + 64) = make_float2(c[2], c[3]);
                    __syncthreads();
                    if (tid < 128) {
                        float sum = red[tid];
                        const int parts = p.kslice / 16;
#pragma unroll
                        for (int w = 1; w < kMaxKSlice / 16; ++w)
                            if (w < parts) sum += red[w * 128 + tid];
                        const int b = tid >> 3, cc = tid & 7;
                        if (b < bt && g * 8 + cc < p.xd) out[static_cast<long long>(b) * p.xd + cc] = sum;
                    }
                } else {
                    const int c = tid & 7, b = (tid >> 3) & 7, part = tid >> 6;
                    const float *ur = reinterpret_cast<const float*>(us) + b * uld, *wr = reinterpret_cast<const float*>(w2) + c;
                    float acc = 0.0f;
#pragma unroll 4
                    for (int k = part; k < p.kslice; k += 8) acc = fmaf(ur[k], wr[k * 8], acc);
                    red[tid] = acc;
                    __syncthreads();
                    if (part == 0 && b < bt && g * 8 + c < p.xd)
                        out[static_cast<long long>(b) * p.xd + c] =
                            ((red[tid] + red[tid + 64]) + (red[tid + 128] + red[tid + 192])) +
                            ((red[tid + 256] + red[tid + 320]) + (red[tid + 384] + red[tid + 448]));
                }
                if (b0 + BT < p.B) __syncthreads();
            }
        }
    }

    // ---- phase 3: delta, SSM step, gate; four lanes (four states each) per (sequence, channel) ----
    __device__ void dt_weights(int l) {  // nch is even, so are di and the 4-byte alignment of a row's start
        const int ch0 = cta * p.nch, n = min(p.nch, p.di - ch0);
        if (l >= p.L || n <= 0) return;
        constexpr int E = 4 / sizeof(Tact);
        const Tact* w = lp(l, p.o_dtw) + ch0;
        Tact* wd = reinterpret_cast<Tact*>(sm + p.s_wd);
        const int per = n / E;
#pragma unroll 1
        for (int c = lane; c < per; c += 32)
#pragma unroll 1
            for (int r = warp; r < p.dr; r += kWarps)
                cp4(smem_u32(wd + r * p.nch + c * E), w + static_cast<long long>(r) * p.di + c * E);
    }
    // what a quad needs of its (sequence, channel) that is ready before the x_proj sums are
    struct Task {
        float4 h, a;
        float z, D;
        Tact u, dtb;  // as loaded: a conversion here would wait for the load
        int b, c;
    };
    __device__ void load_task(int l, int q, int n, Task& t) {
        if (q >= p.B * n) return;
        t.b = q / n;
        t.c = q - t.b * n;
        const int d = cta * p.nch + t.c, j = tid & 3;
        const long long bd = static_cast<long long>(t.b) * p.di + d;
        t.h = ldcg4(p.ssm + ((static_cast<long long>(l) * p.Bcap + t.b) * p.di + d) * kN + 4 * j);
        t.a = __ldg(reinterpret_cast<const float4*>(p.a_neg + (static_cast<long long>(l) * p.di + d) * kN) + j);
        t.u = ldcg_raw(static_cast<const Tact*>(p.u) + bd);
        t.z = __ldcg(p.z + bd);
        t.dtb = lp(l, p.o_dtb)[d];
        t.D = __ldg(mf(l, p.o_D) + d);
    }
    __device__ void do_task(int l, int q, int n, const Task& t) {
        const Tact* wd = reinterpret_cast<const Tact*>(sm + p.s_wd);
        const float* xs = reinterpret_cast<const float*>(sm + p.s_act);
        const int j = tid & 3;
        const bool on = q < p.B * n;
        const int b = on ? t.b : 0, c = on ? t.c : 0, d = cta * p.nch + c;
        const float* xr = xs + b * p.xd;
        float dl = 0.0f;
#pragma unroll 4
        for (int r = j; r < p.dr; r += 4) dl = fmaf(xr[r], to_f(wd[r * p.nch + c]), dl);
        dl += __shfl_xor_sync(0xffffffffu, dl, 1);
        dl += __shfl_xor_sync(0xffffffffu, dl, 2);
        dl = softplusf_fast(dl + to_f(t.dtb));
        const float u = to_f(t.u), du = dl * u, dk = dl * kLog2e;
        const float* Bv = xr + p.dr + 4 * j;
        const float* Cv = Bv + kN;
        float4 h;
        h.x = fmaf(ex2(dk * t.a.x), t.h.x, du * Bv[0]);
        h.y = fmaf(ex2(dk * t.a.y), t.h.y, du * Bv[1]);
        h.z = fmaf(ex2(dk * t.a.z), t.h.z, du * Bv[2]);
        h.w = fmaf(ex2(dk * t.a.w), t.h.w, du * Bv[3]);
        float y = fmaf(h.x, Cv[0], fmaf(h.y, Cv[1], fmaf(h.z, Cv[2], h.w * Cv[3])));
        y += __shfl_xor_sync(0xffffffffu, y, 1);
        y += __shfl_xor_sync(0xffffffffu, y, 2);
        if (on) {
            *reinterpret_cast<float4*>(p.ssm + ((static_cast<long long>(l) * p.Bcap + b) * p.di + d) * kN + 4 * j) = h;
            if (j == 0)
                static_cast<Tact*>(p.y)[static_cast<long long>(b) * p.di + d] = from_f<Tact>(fmaf(t.D, u, y) * siluf_fast(t.z));
        }
    }
    __device__ void scan(int l, int n, Task& t) {
        if (n <= 0) return;
        float* xs = reinterpret_cast<float*>(sm + p.s_act);
        const long long slice = static_cast<long long>(p.B) * p.xd;
        const int sums = p.B * p.xd;
#pragma unroll 1
        for (int i0 = tid; i0 < sums; i0 += 2 * kThreads) {  // up to 16 loads in flight
            float v[2][kMaxKs];
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int q = 0; q < kMaxKs; ++q)
                    v[u][q] = q < p.ks && i0 + u * kThreads < sums ? __ldcg(p.xpart + q * slice + i0 + u * kThreads) : 0.0f;
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (i0 + u * kThreads < sums) {
                    float s = v[u][0];
#pragma unroll
                    for (int q = 1; q < kMaxKs; ++q) s += v[u][q];
#pragma unroll 1
                    for (int q = kMaxKs; q < p.ks; ++q) s += __ldcg(p.xpart + q * slice + i0 + u * kThreads);
                    xs[i0 + u * kThreads] = s;
                }
        }
        __syncthreads();
        const int tasks = p.B * n;
#pragma unroll 1
        for (int q = tid >> 2, r = 0; r < tasks; q += kThreads / 4, r += kThreads / 4) {
            do_task(l, q, n, t);
            load_task(l, q + kThreads / 4, n, t);
        }
    }

    // ---- phase 4 ----
    __device__ float stream_at(int l, int b, int d) const {
        if (l > 0 || !p.next_ids) return __ldcg(p.res + static_cast<long long>(b) * p.dm + d);
        const int id = p.next_ids[b];
        return id >= 0 && id < p.V ? to_f(static_cast<const Tact*>(p.lp)[p.o_emb + static_cast<long long>(id) * p.dm + d]) : 0.0f;
    }
    // this thread's first output of phase 4, read ahead of the barrier
    __device__ float out_base(int l) const {
        const int c = tid % TW, b = (tid / TW) % BT, t = tid / (TW * BT), first = cta * p.t4;
        return t < p.t4 && (first + t) * TW + c < p.dm && b < p.B ? stream_at(l, b, (first + t) * TW + c) : 0.0f;
    }
    __device__ void out_proj(int l, float base) {
        const int tiles = p.dm / TW, first = cta * p.t4, n = min(p.t4, tiles - first);
        if (n <= 0) return;
#pragma unroll 1
        for (int b0 = 0; b0 < p.B; b0 += BT) {
            const int bt = min(BT, p.B - b0);
            load_rows(static_cast<const Tact*>(p.y), p.di, p.kp4, b0, bt);
            __syncthreads();
            if (b0 == 0) alive = mbar_wait(&bars[1], l & 1, p.status) && alive;
#pragma unroll 1
            for (int t0 = 0; t0 < n; t0 += kTC) {
                const int tn = min(kTC, n - t0);
                project(p.s_w4, p.kp4, p.ka4, p.c4, t0, tn, bt);
                __syncthreads();
#pragma unroll 1
                for (int i = tid; i < tn * BT * TW; i += kThreads) {
                    const int c = i % TW, b = (i / TW) % BT, t = i / (TW * BT), d = (first + t0 + t) * TW + c;
                    if (b >= bt) continue;
                    if (i != tid || t0 > 0 || b0 > 0) base = stream_at(l, b0 + b, d);
                    p.res[static_cast<long long>(b0 + b) * p.dm + d] = base + total(t, b, c, p.kp4);
                }
                if (t0 + kTC < n || b0 + BT < p.B) __syncthreads();
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
            __syncthreads();
            norm_rows<false>(p.master + p.o_normf, b0, bt, p.kp1);
            __syncthreads();
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
                int lt = cta * kWarps + warp, lk = 0;  // what is requested next
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
                for (int tile = cta * kWarps + warp; tile * 16 < p.V; tile += stride) {
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
                for (int tile = cta * kWarps + warp; tile * 4 < p.V; tile += ncta * kWarps) {
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
            __syncthreads();
            if (tid < bt) {
                float v = rv[tid];
                int i = ri[tid];
                for (int w = 1; w < kWarps; ++w)
                    if (better(rv[w * 32 + tid], ri[w * 32 + tid], v, i)) { v = rv[w * 32 + tid]; i = ri[w * 32 + tid]; }
                p.amax_v[static_cast<long long>(b0 + tid) * ncta + cta] = v;
                p.amax_i[static_cast<long long>(b0 + tid) * ncta + cta] = i;
            }
        }
    }
    __device__ void choose() {
        for (int b = cta; b < p.B; b += ncta)
            if (warp == 0) {
                float v = -INFINITY;
                int i = 0x7fffffff;
                for (int c = lane; c < ncta; c += 32) {
                    const float ov = __ldcg(p.amax_v + static_cast<long long>(b) * ncta + c);
                    const int oi = __ldcg(p.amax_i + static_cast<long long>(b) * ncta + c);
                    if (better(ov, oi, v, i)) { v = ov; i = oi; }
                }
#pragma unroll
                for (int m = 16; m >= 1; m >>= 1) {
                    const float ov = __shfl_xor_sync(0xffffffffu, v, m);
                    const int oi = __shfl_xor_sync(0xffffffffu, i, m);
                    if (better(ov, oi, v, i)) { v = ov; i = oi; }
                }
                if (lane == 0) {
                    if (p.tokens) p.tokens[b * p.tok_ld] = p.next_ids[b];
                    p.next_ids[b] = i;
                }
            }
    }
    __device__ void final_norm() {  // one row per CTA and pass, through the A-operand tile
        for (int b = cta; b < p.B; b += ncta) {
            norm_rows<false>(p.master + p.o_normf, b, 1, p.kp1);
            __syncthreads();
            const Tact* act = reinterpret_cast<const Tact*>(sm + p.s_act);
            for (int k = tid; k < p.dm; k += kThreads) static_cast<Tact*>(p.out)[static_cast<long long>(b) * p.dm + k] = act[k];
            __syncthreads();
        }
    }

    __device__ void run() {
        if (tid == 0) {
            mbar_init(&bars[0], 1);
            mbar_init(&bars[1], 1);
            fence_barrier_init();
        }
        // rows of a short last slice are never filled: they meet zeros, so they must not be NaN
        for (int i = tid; i < p.kslice * 8; i += kThreads) reinterpret_cast<Tact*>(sm + p.s_wx)[i] = from_f<Tact>(0.0f);
        __syncthreads();
        fetch_in(0);
        fetch_out(0);
        fetch_small(0);
        x_weights(0, cta);
        dt_weights(0);
        hint(1);
        const int n3 = min(p.nch, p.di - cta * p.nch);
        int l = 0;
#pragma unroll 1
        for (; l < p.L; ++l) {
            cp_wait_all();
            __syncthreads();
            in_proj(l);
            arrive();
            fetch_in(l + 1);
            cp_wait_all();
            wait();
            if (!alive) break;
            x_proj(l);
            arrive();
            x_weights(l + 1, cta);
            Task task;
            load_task(l, tid >> 2, n3, task);
            hint(l + 2);
            wait();
            if (!alive) break;
            scan(l, n3, task);
            arrive();
            const float base = out_base(l);
            dt_weights(l + 1);
            wait();
            if (!alive) break;
            out_proj(l, base);
            arrive();
            fetch_out(l + 1);
            fetch_small(l + 1);
            wait();
            if (!alive) break;
        }
        if (!alive) {  // a wait ran out: the copies in flight still have to land in this CTA's memory
            cp_wait_all();
            mbar_wait(&bars[0], (l + 1) & 1, nullptr, 1 << 12);
            mbar_wait(&bars[1], l & 1, nullptr, 1 << 12);
        }
        if (!alive) return;
        if (p.next_ids) {
            head();
            arrive();
            wait();
            if (!alive) return;
            choose();
        } else {
            final_norm();
        }
        // the last CTA to get here (all have left every barrier) makes the counters ready for the next launch
        if (tid == 0) {
            __threadfence();
            if (atomicAdd(p.bar + 1, 1u) == static_cast<unsigned>(ncta) - 1) {
                p.bar[0] = 0;
                p.bar[1] = 0;
            }
        }
    }
};

template <typename Tact>
__global__ void __launch_bounds__(kThreads, 1) decode_step_kernel(const __grid_constant__ Params p) {
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ int flag;
    __shared__ __align__(8) uint64_t bars[2];
    Step<Tact> s(p, sm, &flag, bars);
    s.run();
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
    const int tiles1 = 2 * p.di / tw, tiles4 = p.dm / tw;
    int grid = tiles1 < sms ? tiles1 : sms;
    if (a.vocab > 0) grid = sms;
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
    p.nch = ((p.di + grid - 1) / grid + 1) / 2 * 2;
    p.ncg = (p.xd + 7) / 8;
    // enough slices to use the CTAs, few enough that adding them up stays short
    int ks = grid / p.ncg;
    ks = ks < 1 ? 1 : ks > 8 ? 8 : ks;
    int sl = ((p.di + ks - 1) / ks + 15) / 16 * 16;
    if (sl > kMaxKSlice) sl = kMaxKSlice;
    p.kslice = sl;
    p.ks = (p.di + sl - 1) / sl;
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
    p.s_w1 = o; o += up128(static_cast<long long>(p.t1) * p.ka1 * 16);
    p.s_w4 = o; o += up128(static_cast<long long>(p.t4) * p.ka4 * 16);
    p.s_act = o; o += up(act);
    p.s_red = o; o += up(static_cast<long long>(kWarps) * kTC * bt * tw * 4);
    p.s_wx = o; o += static_cast<long long>(p.kslice) * 16 * (es / 2);
    p.s_wd = o; o += up(static_cast<long long>(p.dr) * p.nch * es);
    p.s_norm = o; o += up(static_cast<long long>(p.dm) * 4);
    p.s_conv = o; o += up(static_cast<long long>(p.t1) * tw * (16LL * (p.B + 1) + 4));
    if (o > 227 * 1024 - 1024) return 0;
    *smem = static_cast<uint32_t>(o);
    const long long Bl = p.B;
    *ws_bytes = 256 + up(Bl * p.di * 4) + up(static_cast<long long>(p.ks) * Bl * p.xd * 4) + 2 * up(Bl * p.di * es) +
                2 * up(Bl * sms * 4);
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
    const long long offs[] = {a.layer_stride, a.o_in_proj, a.o_conv_w, a.o_conv_b, a.o_out_proj, a.o_norm_f, lm ? a.o_embedding : 0};
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
    p.bar = reinterpret_cast<unsigned*>(w); w += 256;
    p.z = reinterpret_cast<float*>(w); w += up(static_cast<long long>(p.B) * p.di * 4);
    p.xpart = reinterpret_cast<float*>(w); w += up(static_cast<long long>(p.ks) * p.B * p.xd * 4);
    p.u = w; w += up(static_cast<long long>(p.B) * p.di * es);
    p.y = w; w += up(static_cast<long long>(p.B) * p.di * es);
    p.amax_v = reinterpret_cast<float*>(w); w += up(static_cast<long long>(p.B) * c->sm_count * 4);
    p.amax_i = reinterpret_cast<int*>(w);
    const unsigned char* lp8 = static_cast<const unsigned char*>(a.lp);
    const int tw = 16 / es;
    if (!make_tmap_stack(c, &p.tm_in, a.dtype, lp8 + p.o_in * es, 2 * p.di, p.dm, p.L, p.lstride, p.c1 * tw, p.br1) ||
        !make_tmap_stack(c, &p.tm_out, a.dtype, lp8 + p.o_out * es, p.dm, p.di, p.L, p.lstride, p.c4 * tw, p.br4))
        return fail(c, MAMBA_B200_ERR_CUDA, "decode_step: the weight tensor maps were refused");
    int steps = lm && a.steps > 1 ? a.steps : 1;
    const void* fn = a.dtype == MAMBA_B200_F32   ? reinterpret_cast<const void*>(dec::decode_step_kernel<float>)
                     : a.dtype == MAMBA_B200_F16 ? reinterpret_cast<const void*>(dec::decode_step_kernel<__half>)
                                                 : reinterpret_cast<const void*>(dec::decode_step_kernel<__nv_bfloat16>);
    for (int i = 0; i < steps; ++i) {
        void* args[1] = {&p};
        MB200_CUDA_CHECK(c, cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(dec::kThreads), args, smem, static_cast<cudaStream_t>(stream)));
        if (p.tokens) ++p.tokens;
    }
    return MAMBA_B200_OK;
}
