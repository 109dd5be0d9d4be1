// f32 products of a few rows of activations with a weight matrix, and the weight gradient that belongs to
// them: what a training step or prefill of a few dozen tokens does in f32.
//   op 0  C[M,N] = A[M,K] B[K,N] (+ bias)        forward
//   op 1  C[M,N] = A[M,K] B[N,K]^T               gradient of the activations; tied head
//   op 2  C[M,N] += A[K,M]^T B[K,N]              gradient of the weights (K rows of activations)
// With M = 32 a weight is used 32 times per load, so the bound is HBM and the FMA pipe alike: 9.4 MB of
// in_proj at 768 x 3072 are 1.5 us of HBM and 2 us of FMA, after which comes a launch's latency.  The
// library's f32 kernels leave most SMs without a tile at such sizes.  32 rows, measured: 768 x 3072 8.6 us
// (library 14.5), 1536 x 768 7.9 (18.1), 1536 x 80 7.7 (17.9); transposed 9.2 (15.0), 8.4 (17.3), 8.2
// (16.7); gradient 6.3 (8.8), 4.1 (5.9), 2.9 (4.0).
//
// ops 0 and 1: a CTA of 128 threads has 32 rows x 64 columns, a 4 x 4 block per thread, and a part of K; the
// parts of a tile form a cluster and add their blocks through distributed shared memory, in rank order, so
// the result does not depend on scheduling.  Tiles of 32 K steps come by cp.async, three stages.  Where a part
// has more than 256 steps the running sums are added to a second set every 256: in one chain the product over a
// vocabulary (32 x 50280 x 768) was 1.4e-6 from the exact one, with two 3.1e-7, the library's 9.3e-7 (150 us in
// one chain, 171 in two; transposed 174 and 156).
// op 2: a CTA of 256 threads has 64 x 64 of C, requested before the products so that its read, which is
// what the call costs, overlaps them.
#include <string.h>

#include "common.cuh"
#include "internal.h"

namespace mb200 {
namespace sg {

constexpr int BM = 32, BN = 64, BK = 32, LA = BK + 4, STAGES = 3;

struct Params {
    const float *a, *b, *bias;
    float* c;
    long long lda, ldb, ldc;
    int M, N, K, kper;  // kper: K steps of a part, a multiple of BK
};

template <bool VEC>
__device__ __forceinline__ void copy4(float* dst, const float* src, int have) {  // four values, `have` of them there
    if (VEC) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(have > 0 ? 16 : 0) : "memory");
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst + i)), "l"(src + (i < have ? i : 0)), "r"(i < have ? 4 : 0)
                         : "memory");
    }
}

template <int OP, bool VEC, bool LONG>  // LONG: a part of K has more than 256 steps
__global__ void __launch_bounds__(128) rows_kernel(const Params p) {
    constexpr int LB = OP == 0 ? BN : LA, WB = OP == 0 ? BK * BN : BN * LA, WA = BM * LA;
    extern __shared__ __align__(16) float sm[];  // [STAGES][A | B]
    uint32_t parts, rank;
    asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(parts));
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int tid = threadIdx.x, n0 = static_cast<int>(blockIdx.x / parts) * BN, m0 = blockIdx.y * BM;
    const int k0 = min(p.K, static_cast<int>(rank) * p.kper), k1 = min(p.K, k0 + p.kper), steps = (k1 - k0 + BK - 1) / BK;
    auto fetch = [&](int s) {
        if (s < steps) {
            float* A = sm + (s % STAGES) * (WA + WB);
            float* B = A + WA;
            const int k = k0 + s * BK;
#pragma unroll
            for (int i = 0; i < BM * BK / 4 / 128; ++i) {
                const int r = (tid + 128 * i) / (BK / 4), c = (tid + 128 * i) % (BK / 4) * 4;
                const bool on = m0 + r < p.M;
                const int have = on ? min(4, k1 - k - c) : 0;
                copy4<VEC>(A + r * LA + c, have > 0 ? p.a + (m0 + r) * p.lda + k + c : p.a, have);
            }
#pragma unroll
            for (int i = 0; i < BN * BK / 4 / 128; ++i) {
                int r, c, have;
                const float* src;
                if (OP == 0) {
                    r = (tid + 128 * i) / (BN / 4), c = (tid + 128 * i) % (BN / 4) * 4;
                    have = k + r < k1 ? min(4, p.N - n0 - c) : 0;
                    src = p.b + (k + r) * p.ldb + n0 + c;
                } else {
                    r = (tid + 128 * i) / (BK / 4), c = (tid + 128 * i) % (BK / 4) * 4;
                    have = n0 + r < p.N ? min(4, k1 - k - c) : 0;
                    src = p.b + (n0 + r) * p.ldb + k + c;
                }
                copy4<VEC>(B + r * LB + c, have > 0 ? src : p.b, have);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int s = 0; s < STAGES - 1; ++s) fetch(s);
    const int tx = tid & 15, ty = tid >> 4;  // rows ty + 8 i; columns 4 tx + j (op 0) or tx + 16 j (op 1)
    float acc[4][4], sum[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = sum[i][j] = 0.0f;  // (sum: LONG)
    for (int s = 0; s < steps;) {
        const int top = LONG ? min(steps, s + 8) : steps;
        for (; s < top; ++s) {
            asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
            __syncthreads();
            fetch(s + STAGES - 1);
            const float* A = sm + (s % STAGES) * (WA + WB);
            const float* B = A + WA;
#pragma unroll
            for (int k = 0; k < BK; k += 4) {
                float4 a[4], b[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(A + (ty + 8 * i) * LA + k);
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    b[j] = *reinterpret_cast<const float4*>(OP == 0 ? B + (k + j) * LB + 4 * tx : B + (tx + 16 * j) * LB + k);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float av[4] = {a[i].x, a[i].y, a[i].z, a[i].w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float bv[4] = {b[j].x, b[j].y, b[j].z, b[j].w};
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            if (OP == 0) acc[i][q] = fmaf(av[j], bv[q], acc[i][q]);
                            else acc[i][j] = fmaf(av[q], bv[q], acc[i][j]);
                        }
                    }
                }
            }
        }
        if (LONG) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    sum[i][j] += acc[i][j];
                    acc[i][j] = 0.0f;
                }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) sm[(ty + 8 * i) * BN + (OP == 0 ? 4 * tx + j : tx + 16 * j)] = LONG ? sum[i][j] : acc[i][j];
    if (parts > 1) cluster_sync();
    else __syncthreads();
    // this rank's rows of the sum
    const int per = BM / static_cast<int>(parts);
    for (int i = tid; i < per * BN; i += 128) {
        const int r = static_cast<int>(rank) * per + i / BN, c = i % BN;
        float s = 0.0f;
        if (parts > 1) {
            const uint32_t at = smem_u32(sm + r * BN + c);
            for (uint32_t q = 0; q < parts; ++q) s += ld_cluster1(cluster_addr(at, static_cast<int>(q)));
        } else {
            s = sm[r * BN + c];
        }
        if (m0 + r < p.M && n0 + c < p.N) p.c[(m0 + r) * p.ldc + n0 + c] = s + (p.bias ? p.bias[n0 + c] : 0.0f);
    }
    if (parts > 1) cluster_sync();  // nobody reads this CTA's shared memory any more
}

template <bool VEC, bool TALL>  // TALL: grid.x counts the tiles of rows
__global__ void __launch_bounds__(256) grad_kernel(const Params p) {
    constexpr int BC = 64;
    __shared__ __align__(16) float A[BK][BC], B[BK][BC];
    const int tid = threadIdx.x, m0 = (TALL ? blockIdx.x : blockIdx.y) * BC, n0 = (TALL ? blockIdx.y : blockIdx.x) * BC, tx = tid & 15, ty = tid >> 4;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
    float* c = p.c + (m0 + 4 * ty) * p.ldc + n0 + 4 * tx;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (m0 + 4 * ty + i < p.M) {
            if (VEC) {
                if (n0 + 4 * tx < p.N) {
                    const float4 v = *reinterpret_cast<const float4*>(c + i * p.ldc);
                    acc[i][0] = v.x; acc[i][1] = v.y; acc[i][2] = v.z; acc[i][3] = v.w;
                }
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (n0 + 4 * tx + j < p.N) acc[i][j] = c[i * p.ldc + j];
            }
        }
    for (int k = 0; k < p.K; k += BK) {
        if (k) __syncthreads();
#pragma unroll
        for (int i = 0; i < BK * BC / 4 / 256; ++i) {
            const int r = (tid + 256 * i) / (BC / 4), q = (tid + 256 * i) % (BC / 4) * 4;
            const int ha = k + r < p.K ? min(4, p.M - m0 - q) : 0, hb = k + r < p.K ? min(4, p.N - n0 - q) : 0;
            copy4<VEC>(&A[r][q], ha > 0 ? p.a + (k + r) * p.lda + m0 + q : p.a, ha);
            copy4<VEC>(&B[r][q], hb > 0 ? p.b + (k + r) * p.ldb + n0 + q : p.b, hb);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
#pragma unroll 8
        for (int t = 0; t < BK; ++t) {
            const float4 a = *reinterpret_cast<const float4*>(&A[t][4 * ty]), b = *reinterpret_cast<const float4*>(&B[t][4 * tx]);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (m0 + 4 * ty + i < p.M) {
            if (VEC) {
                if (n0 + 4 * tx < p.N)
                    *reinterpret_cast<float4*>(c + i * p.ldc) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (n0 + 4 * tx + j < p.N) c[i * p.ldc + j] = acc[i][j];
            }
        }
}

}  // namespace sg

}  // namespace mb200

using namespace mb200;

extern "C" MAMBA_B200_API int mamba_b200_sgemm_rows(void* handle, void* stream, int op, const float* a, long long lda, const float* b,
                                                    long long ldb, const float* bias, float* out, long long ldc, int M, int N, int K) {
    Ctx* c = static_cast<Ctx*>(handle);
    if (!c) return MAMBA_B200_ERR_ARG;
    if (op < 0 || op > 2 || M < 0 || N < 0 || K < 0) return fail(c, MAMBA_B200_ERR_ARG, "sgemm_rows: op %d, %d x %d x %d", op, M, N, K);
    if (M == 0 || N == 0 || (op == 2 && K == 0)) return MAMBA_B200_OK;
    if (!out || (K > 0 && (!a || !b))) return fail(c, MAMBA_B200_ERR_ARG, "sgemm_rows: null required pointer");
    if (op == 2 && bias) return fail(c, MAMBA_B200_ERR_ARG, "sgemm_rows: a gradient takes no bias");
    sg::Params p;
    p.a = a; p.b = b; p.bias = bias; p.c = out; p.lda = lda; p.ldb = ldb; p.ldc = ldc; p.M = M; p.N = N; p.K = K;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    auto al = [](const void* q, long long ld) { return reinterpret_cast<uintptr_t>(q) % 16 == 0 && ld % 4 == 0; };
    if (op == 2) {
        p.kper = 0;
        // a row's groups of four are whole where both sides are multiples of four
        const bool vec = al(a, lda) && al(b, ldb) && al(out, ldc) && M % 4 == 0 && N % 4 == 0;
        // tiles of columns side by side; of rows where there are too many for the other dimension (a vocabulary)
        dim3 grid((N + 63) / 64, (M + 63) / 64);
        const bool tall = grid.y > 65535;
        if (tall) grid = dim3(grid.y, grid.x);
        if (grid.y > 65535) return fail(c, MAMBA_B200_ERR_SHAPE, "sgemm_rows: a gradient of %d x %d", M, N);
        if (vec && !tall) sg::grad_kernel<true, false><<<grid, 256, 0, st>>>(p);
        else if (vec) sg::grad_kernel<true, true><<<grid, 256, 0, st>>>(p);
        else if (!tall) sg::grad_kernel<false, false><<<grid, 256, 0, st>>>(p);
        else sg::grad_kernel<false, true><<<grid, 256, 0, st>>>(p);
        MB200_CUDA_CHECK(c, cudaGetLastError());
        return MAMBA_B200_OK;
    }
    const int tiles = (N + sg::BN - 1) / sg::BN, rows = (M + sg::BM - 1) / sg::BM;
    if (rows > 65535) return fail(c, MAMBA_B200_ERR_SHAPE, "sgemm_rows: %d rows", M);
    // parts of K until there are two CTAs for every SM (more only adds to the sums: 64 rows, 768 x 3072 took
    // 15.3 us with four, 13.4 with two, 18.5 with one), none shorter than two tiles
    int parts = 1;
    while (parts < 8 && static_cast<long long>(tiles) * rows * parts < 2 * 148 && K >= parts * 4 * sg::BK) parts *= 2;
    p.kper = ((K + parts - 1) / parts + sg::BK - 1) / sg::BK * sg::BK;
    const bool vec = al(a, lda) && al(b, ldb) && K % 4 == 0 && (op == 1 || N % 4 == 0);
    const bool lng = p.kper > 8 * sg::BK;
#define MB200_ROWS(OP, VEC) {reinterpret_cast<const void*>(sg::rows_kernel<OP, VEC, false>), reinterpret_cast<const void*>(sg::rows_kernel<OP, VEC, true>)}
    const void* fns[4][2] = {MB200_ROWS(0, false), MB200_ROWS(0, true), MB200_ROWS(1, false), MB200_ROWS(1, true)};
#undef MB200_ROWS
    const size_t smem = sizeof(float) * sg::STAGES * (sg::BM * sg::LA + (op == 0 ? sg::BK * sg::BN : sg::BN * sg::LA));
    static_assert(sizeof(float) * sg::STAGES * (sg::BM * sg::LA + sg::BN * sg::LA) <= 48 * 1024, "within what needs no opt-in");
    void* args[1] = {&p};
    MB200_CUDA_CHECK(c, launch_cluster(fns[op * 2 + (vec ? 1 : 0)][lng ? 1 : 0], dim3(tiles * parts, rows), dim3(128), smem, st, parts, args));
    return MAMBA_B200_OK;
}
