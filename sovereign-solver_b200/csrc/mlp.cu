// mlp.cu -- the learned warm start's network on the tensor cores: a
// 2-hidden-layer ReLU MLP (n_in -> hidden -> hidden -> n_out) whose forward
// and backward passes are BF16 GEMMs with FP32 accumulation on tcgen05
// (k_gemm_tn), trained with Adam on FP32 master weights.
//
// One GEMM form covers every product: C[M x N] = A[M x K] * B[N x K]^T with
// both operands K-contiguous (row-major A and B), fused epilogue (bias, ReLU,
// a ReLU-derivative mask or the loss's derivative; FP32, BF16 and transposed
// BF16 outputs). The weight gradients dY^T H take their operands from the
// transposed outputs of the GEMMs that made them, the input gradients dY W the
// weights' transposed copies (k_transpose, when the weights change).
//
// Forward (batch B):  H1 = relu(X W1^T + b1), H2 = relu(H1 W2^T + b2),
//                     Y = H2 W3^T + b3.
// Loss:               L = sum (Y - T)^2 / (B n_out).
// Backward:           dY = 2 (Y - T) / (B n_out); dW3 = dY^T H2, db3 = sum_b dY;
//                     dZ2 = (dY W3) * [H2 > 0]; dW2 = dZ2^T H1; db2 = sum_b dZ2;
//                     dZ1 = (dZ2 W2) * [H1 > 0]; dW1 = dZ1^T X; db1 = sum_b dZ1.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <random>
#include <string>
#include <vector>

#include "../../include/pdhg_b200.h"
#include "pass.cuh"
#include "tcgen05.cuh"

namespace pdhg {
namespace {

using bf16 = __nv_bfloat16;

constexpr int kGemmThreads = kBlock;
constexpr long long kSpinLimit = 1LL << 24;  // bounded mbarrier waits

struct GemmArgs {
    int M, N, K;
    const bf16* A;
    int lda;
    const bf16* B;
    int ldb;
    const float* bias;  // N, or null
    int relu;
    const bf16* mask;   // M x N: output * [mask > 0], or null
    int ldm;
    // The output is the loss's derivative 2 (v - target) scale at v = the
    // product, or null; row r's target is row idx[r] (idx null: r) of N. Each
    // CTA's share of the loss (v - target)^2 scale to part[its tile].
    const float* target;
    const int32_t* idx;
    float scale;
    double* part;
    float* out32;       // M x N, or null
    int ld32;
    bf16* out16;        // M x N, or null
    int ld16;
    bf16* out16t;       // N x M: the transposed output, or null
    int ldt;
    int* err;           // set when a bounded wait gives up
    int vec;            // 1: every row of bias / mask / target / outputs starts 16-byte aligned
};
// One launch over the tiles of up to two products, the second's after tiles0.
struct GemmPair {
    GemmArgs g[2];
    int tiles0;
};

// 16-byte asynchronous global -> shared copy (cp.async, no register staging);
// src_bytes = 0 writes zeros and reads nothing.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(tc::smem_u32(smem)),
                 "l"(gmem), "r"(src_bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Rows [r0, r0 + ROWS) x K-elements [k0, k0 + 64) of a matrix of `rows` x K
// into a staged tile, zeros outside.
template <int ROWS>
__device__ __forceinline__ void stage_rows(bf16* dst, const bf16* src, int ld, int r0, int rows, int k0, int K) {
#pragma unroll
    for (int c = threadIdx.x; c < ROWS * (tc::kTileK / 8); c += kGemmThreads) {
        const int row = c >> 3, kc = (c & 7) * 8;
        const int gr = r0 + row, gk = k0 + kc;
        const bool in = gr < rows && gk < K;
        cp_async16(dst + tc::tile_offset(row, kc), in ? src + static_cast<size_t>(gr) * ld + gk : src, in ? 16 : 0);
    }
}

// C = A B^T on one 128 x BN tile: the K loop keeps STAGES slices of A (128 x
// 64) and B (BN x 64) in shared memory (core-matrix layout, see tcgen05.cuh)
// or on their way there in 16-byte asynchronous copies; one thread issues each
// slice's four 16-deep MMAs into the TMEM accumulator and commits them to the
// slice's mbarrier, which is waited on before the slice is overwritten. The
// epilogue reads the accumulator with tcgen05.ld, one TMEM lane (= output row)
// per thread, 32 columns at a time; the second four warps take every other 32.
//
// Bound: the latency of one CTA's chain (slice, MMAs, epilogue); a product of
// the network (256 x 512 x 512) is 0.1 us of the tensor cores. So all of its
// slices are in flight at once, and the tiles are as narrow as keeps the grid
// within the SMs (gemm). One slice at a time on 128-column tiles, with the
// transposes, the loss and the column sums in launches of their own, the
// gradients of 256 rows through 64 -> 512 -> 512 -> 512 took 536 us with their
// copies, 25 launches; 294 us in 8, as programmatic dependents, the same bits.
template <int BN, int STAGES>
__global__ void __launch_bounds__(kGemmThreads) k_gemm_tn(const __grid_constant__ GemmPair pair) {
    extern __shared__ __align__(1024) unsigned char dyn[];
    __shared__ __align__(8) uint64_t bar[STAGES];
    __shared__ uint32_t tmem_base;
    __shared__ double loss_part[kGemmThreads / 32];
    constexpr int kA = tc::kTileM * tc::kTileK, kB = BN * tc::kTileK;
    bf16* const slices = reinterpret_cast<bf16*>(dyn);  // A's and B's of stage 0, of stage 1, ...
    const bool second = static_cast<int>(blockIdx.x) >= pair.tiles0;
    const GemmArgs& g = pair.g[second ? 1 : 0];
    const int tile = static_cast<int>(blockIdx.x) - (second ? pair.tiles0 : 0);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tiles_m = (g.M + tc::kTileM - 1) / tc::kTileM;
    const int m0 = tile % tiles_m * tc::kTileM, n0 = tile / tiles_m * BN;
    const int rounds = (g.K + tc::kTileK - 1) / tc::kTileK;
    if (warp == 0) {
        tc::tmem_alloc(&tmem_base, BN);
        tc::tmem_relinquish();
    }
    if (tid == 0) {
        for (int i = 0; i < STAGES; ++i) tc::mbar_init(&bar[i], 1);
        tc::fence_mbar_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    // The next launch may start only now that this CTA holds its TMEM columns:
    // its CTAs take columns and then wait for this grid, so one of this grid's
    // that still waited for columns beside them would never get any.
    pass_begin();
    const uint32_t tmem = tmem_base;
    constexpr uint32_t idesc = tc::instr_desc_bf16(BN);
    const uint32_t base = tc::smem_u32(slices);
    auto stage = [&](int r) {
        if (r < rounds) {
            bf16* at = slices + (r % STAGES) * (kA + kB);
            stage_rows<tc::kTileM>(at, g.A, g.lda, m0, g.M, r * tc::kTileK, g.K);
            stage_rows<BN>(at + kA, g.B, g.ldb, n0, g.N, r * tc::kTileK, g.K);
        }
        cp_async_commit();
    };
    auto wait = [&](int r) {  // for round r's MMAs, bounded; the same answer for the CTA
        long long spins = 0;
        bool timed_out = false;
        while (!tc::mbar_try_wait(&bar[r % STAGES], static_cast<uint32_t>((r / STAGES) & 1)))
            if (++spins > kSpinLimit) {
                timed_out = true;
                break;
            }
        return __syncthreads_or(timed_out) == 0;
    };
    pass_wait();  // the operands are the kernel before's
    for (int r = 0; r < STAGES - 1; ++r) stage(r);
    bool ok = true;
    int issued = 0;
    for (int r = 0; r < rounds; ++r) {
        const int next = r + STAGES - 1;
        if (next >= STAGES && next < rounds) ok = wait(next - STAGES);
        if (!ok) break;
        stage(next);
        cp_async_wait<STAGES - 1>();  // round r's copies have landed
        tc::fence_proxy_async_smem();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after_sync();
            const uint32_t a = base + static_cast<uint32_t>(r % STAGES) * 2u * (kA + kB), b = a + 2u * kA;
#pragma unroll
            for (int s = 0; s < tc::kTileK / 16; ++s)
                tc::mma_bf16(tmem, tc::smem_desc(a + s * 2 * tc::kChunkBytes),
                             tc::smem_desc(b + s * 2 * tc::kChunkBytes), idesc, (r > 0 || s > 0) ? 1u : 0u);
            tc::mma_commit(&bar[r % STAGES]);
        }
        ++issued;
    }
    if (ok) ok = wait(rounds - 1);  // the commits arrive in order
    tc::fence_after_sync();
    double loss = 0.0;
    if (!ok) {
        if (tid == 0) *reinterpret_cast<volatile int*>(g.err) = 1;
        cp_async_wait<0>();
        if (issued > 0) wait(issued - 1);  // one more bounded chance for the MMAs in flight
    } else {
        const int row = m0 + (warp & 3) * 32 + lane;
        for (int cb = (warp >> 2) * 32; cb < BN; cb += kGemmThreads / 128 * 32) {
            float v[32];
            tc::tmem_load32(tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + cb, v);
            if (row >= g.M) continue;
            const int c0 = n0 + cb;
            const float* trow = nullptr;
            if (g.target != nullptr) trow = g.target + static_cast<size_t>(g.idx != nullptr ? g.idx[row] : row) * g.N;
            if (g.vec && c0 + 32 <= g.N) {
                // a thread's 32 columns are contiguous in its row: 16-byte
                // loads of bias and mask, all issued before they are used,
                // and 16-byte stores
                if (g.bias != nullptr) {
                    const float4* b4 = reinterpret_cast<const float4*>(g.bias + c0);
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const float4 b = b4[q];
                        v[4 * q] += b.x;
                        v[4 * q + 1] += b.y;
                        v[4 * q + 2] += b.z;
                        v[4 * q + 3] += b.w;
                    }
                }
                if (g.relu)
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.f);
                if (g.mask != nullptr) {
                    const uint4* m4 = reinterpret_cast<const uint4*>(g.mask + static_cast<size_t>(row) * g.ldm + c0);
                    uint4 mk[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) mk[q] = m4[q];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const bf16* mb = reinterpret_cast<const bf16*>(&mk[q]);
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            if (!(__bfloat162float(mb[j]) > 0.f)) v[8 * q + j] = 0.f;
                    }
                }
                if (trow != nullptr) {
                    const float4* t4 = reinterpret_cast<const float4*>(trow + c0);
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const float4 t = t4[q];
                        const float tv[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const float d = v[4 * q + u] - tv[u];
                            v[4 * q + u] = 2.f * d * g.scale;
                            loss += static_cast<double>(d) * d * g.scale;
                        }
                    }
                }
                if (g.out32 != nullptr) {
                    float4* o4 = reinterpret_cast<float4*>(g.out32 + static_cast<size_t>(row) * g.ld32 + c0);
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        o4[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                }
                if (g.out16 != nullptr) {
                    uint4* o4 = reinterpret_cast<uint4*>(g.out16 + static_cast<size_t>(row) * g.ld16 + c0);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        uint4 w;
                        bf16* wb = reinterpret_cast<bf16*>(&w);
#pragma unroll
                        for (int j = 0; j < 8; ++j) wb[j] = __float2bfloat16_rn(v[8 * q + j]);
                        o4[q] = w;
                    }
                }
                if (g.out16t != nullptr)  // a warp's 32 rows of a column are 64 contiguous bytes
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        g.out16t[static_cast<size_t>(c0 + j) * g.ldt + row] = __float2bfloat16_rn(v[j]);
                continue;
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                const int col = c0 + j;
                if (col >= g.N) continue;
                float x = v[j];
                if (g.bias != nullptr) x += g.bias[col];
                if (g.relu) x = fmaxf(x, 0.f);
                if (g.mask != nullptr &&
                    !(__bfloat162float(g.mask[static_cast<size_t>(row) * g.ldm + col]) > 0.f))
                    x = 0.f;
                if (trow != nullptr) {
                    const float d = x - trow[col];
                    x = 2.f * d * g.scale;
                    loss += static_cast<double>(d) * d * g.scale;
                }
                if (g.out32 != nullptr) g.out32[static_cast<size_t>(row) * g.ld32 + col] = x;
                if (g.out16 != nullptr)
                    g.out16[static_cast<size_t>(row) * g.ld16 + col] = __float2bfloat16_rn(x);
                if (g.out16t != nullptr)
                    g.out16t[static_cast<size_t>(col) * g.ldt + row] = __float2bfloat16_rn(x);
            }
        }
    }
    if (g.target != nullptr) {  // the same for the CTA
        __syncwarp();
        for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
        if (lane == 0) loss_part[warp] = loss;
    }
    tc::fence_before_sync();
    __syncthreads();
    if (g.target != nullptr && tid == 0) {
        double s = 0.0;
        for (int w = 0; w < kGemmThreads / 32; ++w) s += loss_part[w];
        g.part[tile] = s;
    }
    if (warp == 0) tc::tmem_dealloc(tmem, BN);
}

// out[c * ldo + r] = in[r * ldi + c] for an R x C BF16 matrix (32 x 32 tiles).
__global__ void k_transpose(const bf16* in, int ldi, bf16* out, int ldo, int R, int C) {
    __shared__ bf16 t[32][33];
    const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
    for (int i = threadIdx.y; i < 32; i += 8) {
        const int r = r0 + i, c = c0 + threadIdx.x;
        if (r < R && c < C) t[i][threadIdx.x] = in[static_cast<size_t>(r) * ldi + c];
    }
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += 8) {
        const int c = c0 + i, r = r0 + threadIdx.x;
        if (r < R && c < C) out[static_cast<size_t>(c) * ldo + r] = t[threadIdx.x][i];
    }
}

__global__ void k_to_bf16(const float* in, bf16* out, int64_t n) {
    const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (t < n) out[t] = __float2bfloat16_rn(in[t]);
}

// Rows idx[0..B) (idx null: 0..B) of src (S x d, FP32) in BF16: dst (B x d)
// and, unless null, its transposed copy (d x B). 32 x 32 tiles, all along the
// grid's x: of rows or of inputs there may be more than its y takes (65,535).
__global__ void k_gather_rows(const float* src, int d, const int32_t* idx, int B, bf16* dst, bf16* dst_t) {
    __shared__ bf16 t[32][33];
    pass_begin();
    pass_wait();
    const int rb = (B + 31) / 32;
    const int r0 = static_cast<int>(blockIdx.x) % rb * 32, c0 = static_cast<int>(blockIdx.x) / rb * 32;
    const int c = c0 + threadIdx.x;
    for (int i = threadIdx.y; i < 32; i += 8) {
        const int r = r0 + i;
        if (r >= B || c >= d) continue;
        const bf16 v = __float2bfloat16_rn(src[static_cast<int64_t>(idx != nullptr ? idx[r] : r) * d + c]);
        dst[static_cast<size_t>(r) * d + c] = v;
        t[i][threadIdx.x] = v;
    }
    if (dst_t == nullptr) return;
    __syncthreads();
    const int r = r0 + threadIdx.x;
    for (int i = threadIdx.y; i < 32; i += 8)
        if (r < B && c0 + i < d) dst_t[static_cast<size_t>(c0 + i) * B + r] = t[threadIdx.x][i];
}

// db[j] = sum_b dZ[b, j] for up to three dZ (B x N), and the loss from its
// parts, in one launch: CTA c takes 32 columns of one matrix, staged 256 rows
// at a time so that the loads are all in flight; each column is then one
// thread's sum in row order. The last CTA adds the loss's parts in order.
// (One thread per column, each row's load waiting for the one before: 20 us
// for 256 rows; staged 3 us.)
struct ColSums {
    const float* dz[3];
    float* db[3];
    int N[3], first[4];  // first[i]: matrix i's first CTA; first[3]: the loss's
    int B;
    const double* part;
    int n_part;
    double* loss;
};
constexpr int kColRows = 256;
__global__ void __launch_bounds__(256) k_colsums(const __grid_constant__ ColSums a) {
    __shared__ float st[kColRows][33];
    pass_begin();
    pass_wait();
    const int b = static_cast<int>(blockIdx.x), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (b == a.first[3]) {
        if (warp != 0) return;
        double s = 0.0;
        for (int i = 0; i < a.n_part; i += 32) {
            const double v = i + lane < a.n_part ? a.part[i + lane] : 0.0;
            for (int q = 0; q < 32; ++q) s += __shfl_sync(0xffffffffu, v, q);
        }
        if (lane == 0) *a.loss = s;
        return;
    }
    const int k = b >= a.first[2] ? 2 : b >= a.first[1] ? 1 : 0;
    const int N = a.N[k], j = (b - a.first[k]) * 32 + lane;
    const float* __restrict__ dz = a.dz[k];
    float s = 0.f;
    for (int r0 = 0; r0 < a.B; r0 += kColRows) {
        const int rows = min(kColRows, a.B - r0);
#pragma unroll 8
        for (int r = warp; r < rows; r += 8)
            if (j < N) st[r][lane] = __ldcg(dz + static_cast<size_t>(r0 + r) * N + j);
        __syncthreads();
        if (warp == 0)
#pragma unroll 16
            for (int r = 0; r < rows; ++r) s += st[r][lane];
        __syncthreads();
    }
    if (warp == 0 && j < N) a.db[k][j] = s;
}

// Adam (bias-corrected) on FP32 master weights; refreshes the BF16 copy.
__global__ void k_adam(float* w, const float* g, float* m, float* v, bf16* w16, int64_t n,
                       float lr, float b1, float b2, float eps, float c1, float c2) {
    const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (t >= n) return;
    const float gt = g[t];
    const float mt = b1 * m[t] + (1.f - b1) * gt;
    const float vt = b2 * v[t] + (1.f - b2) * gt * gt;
    m[t] = mt;
    v[t] = vt;
    const float wt = w[t] - lr * (mt / c1) / (sqrtf(vt / c2) + eps);
    w[t] = wt;
    if (w16 != nullptr) w16[t] = __float2bfloat16_rn(wt);
}

inline int blocks(int64_t n, int t) { return static_cast<int>((n + t - 1) / t); }

template <int BN>
constexpr int kStageBytes = 2 * (tc::kTileM + BN) * tc::kTileK;

// Once per device (the caller's current one), before its first GEMM.
cudaError_t init_gemm() {
    constexpr auto smem = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(k_gemm_tn<32, 8>, smem, 8 * kStageBytes<32>);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_gemm_tn<64, 8>, smem, 8 * kStageBytes<64>);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_gemm_tn<128, 6>, smem, 6 * kStageBytes<128>);
    return e;
}

template <int BN, int STAGES>
cudaError_t run_gemm(const GemmPair& p, int tiles, int rounds, bool early, cudaStream_t s) {
    return launch_pass_smem(k_gemm_tn<BN, STAGES>, tiles, early, s, std::min(rounds, STAGES) * kStageBytes<BN>, p);
}

// Host checks of the GEMM's layout contract, then one launch of one or two
// products (h null: one; early: see launch_pass). The tiles are 32 columns wide while that gives no more
// CTAs than the GPU has SMs, then 64, then 128: a wider tile reads A less often,
// a narrower one leaves fewer SMs idle (256 x 512 x 512: 8 CTAs of 128 columns,
// 32 of 32).
int gemm(const GemmArgs& g, const GemmArgs* h, bool early, int sms, cudaStream_t s) {
    GemmPair p{};
    int rounds = 0, tiles[3] = {};
    auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
    for (int i = 0; i < (h != nullptr ? 2 : 1); ++i) {
        GemmArgs& a = p.g[i] = i == 0 ? g : *h;
        if (a.M < 1 || a.N < 1 || a.K < 8 || a.K % 8 != 0 || a.lda % 8 != 0 || a.ldb % 8 != 0 || !al16(a.A) ||
            !al16(a.B))
            return PDHG_ERR_INVALID_ARGUMENT;
        a.vec = al16(a.bias) && (a.mask == nullptr || (al16(a.mask) && a.ldm % 8 == 0)) &&
                (a.target == nullptr || (al16(a.target) && a.N % 4 == 0)) &&
                (a.out32 == nullptr || (al16(a.out32) && a.ld32 % 4 == 0)) &&
                (a.out16 == nullptr || (al16(a.out16) && a.ld16 % 8 == 0)) ? 1 : 0;
        rounds = std::max(rounds, (a.K + tc::kTileK - 1) / tc::kTileK);
        for (int w = 0; w < 3; ++w) {
            const int t = ((a.M + tc::kTileM - 1) / tc::kTileM) * ((a.N + (32 << w) - 1) / (32 << w));
            tiles[w] += t;
        }
    }
    const int w = tiles[0] <= sms ? 0 : tiles[1] <= sms ? 1 : 2;
    p.tiles0 = ((g.M + tc::kTileM - 1) / tc::kTileM) * ((g.N + (32 << w) - 1) / (32 << w));
    const cudaError_t e = w == 0   ? run_gemm<32, 8>(p, tiles[0], rounds, early, s)
                          : w == 1 ? run_gemm<64, 8>(p, tiles[1], rounds, early, s)
                                   : run_gemm<128, 6>(p, tiles[2], rounds, early, s);
    return e == cudaSuccess ? PDHG_OK : PDHG_ERR_BACKEND;
}

void transpose(const bf16* in, int ldi, bf16* out, int ldo, int R, int C, cudaStream_t s) {
    const dim3 grid((C + 31) / 32, (R + 31) / 32);
    k_transpose<<<grid, dim3(32, 8), 0, s>>>(in, ldi, out, ldo, R, C);
}

// CTAs of forward()'s last product (gemm's rule), each with its part of the loss.
int loss_parts(int B, int n_out, int sms) {
    const int tm = (B + tc::kTileM - 1) / tc::kTileM;
    for (int w = 0; w < 2; ++w)
        if (tm * blocks(n_out, 32 << w) <= sms) return tm * blocks(n_out, 32 << w);
    return tm * blocks(n_out, 128);
}

template <class T>
struct Dev {
    T* p = nullptr;
    size_t n = 0;
    Dev() = default;
    Dev(const Dev&) = delete;
    Dev& operator=(const Dev&) = delete;
    ~Dev() {
        if (p != nullptr) cudaFree(p);
    }
    cudaError_t alloc(size_t count) {
        if (p != nullptr) cudaFree(p);
        p = nullptr;
        n = count;
        return count ? cudaMalloc(reinterpret_cast<void**>(&p), sizeof(T) * count) : cudaSuccess;
    }
};

}  // namespace

struct Mlp {
    int device = 0;
    int sms = 0;  // the device's
    int n_in = 0, hidden = 0, n_out = 0, max_batch = 0;
    cudaStream_t stream = nullptr;
    std::string err;
    // parameters, one FP32 block [W1 b1 W2 b2 W3 b3] and its gradient / Adam moments
    int64_t off[6] = {}, cnt[6] = {}, total = 0;
    Dev<float> w, g, m, v;
    Dev<bf16> w16, w2t, w3t;  // BF16 weights, transposed W2 and W3 (for dX products)
    long long adam_t = 0;
    // activations (max_batch rows)
    Dev<bf16> x16, xt, h1, h1t, h2, h2t, dy16, dyt, dz2_16, dz2t, dz1t;
    Dev<float> x32, t32, y32, dy32, dz2_32, dz1_32;
    Dev<double> part;
    // in pinned memory, written by the kernels
    struct Status {
        double loss;
        int err;
    }* status = nullptr;
    // training set on the device
    Dev<float> xs, ts;

    ~Mlp() {
        if (stream != nullptr) cudaStreamDestroy(stream);
        if (status != nullptr) cudaFreeHost(status);
    }
    float* W(int i) { return w.p + off[2 * i]; }
    float* Bv(int i) { return w.p + off[2 * i + 1]; }
    bf16* W16(int i) { return w16.p + off[2 * i]; }
    float* gW(int i) { return g.p + off[2 * i]; }
    float* gB(int i) { return g.p + off[2 * i + 1]; }
};

namespace {

#define MCK(expr)                                                           \
    do {                                                                    \
        cudaError_t e_ = (expr);                                            \
        if (e_ != cudaSuccess) {                                            \
            h.err = std::string(#expr) + ": " + cudaGetErrorString(e_);     \
            return e_ == cudaErrorMemoryAllocation ? PDHG_ERR_OUT_OF_MEMORY \
                                                   : PDHG_ERR_BACKEND;      \
        }                                                                   \
    } while (0)

int check_err(Mlp& h) {
    MCK(cudaStreamSynchronize(h.stream));
    if (h.status->err != 0) {
        h.err = "tensor-core GEMM: an MMA did not complete within its wait limit";
        return PDHG_ERR_BACKEND;
    }
    return PDHG_OK;
}

GemmArgs args(int M, int N, int K, const bf16* A, int lda, const bf16* B, int ldb, int* err) {
    GemmArgs g{};
    g.M = M;
    g.N = N;
    g.K = K;
    g.A = A;
    g.lda = lda;
    g.B = B;
    g.ldb = ldb;
    g.err = err;
    return g;
}

// Refresh the BF16 weights and the transposed copies from the FP32 masters.
void refresh_weights(Mlp& h) {
    k_to_bf16<<<blocks(h.total, 256), 256, 0, h.stream>>>(h.w.p, h.w16.p, h.total);
    transpose(h.W16(1), h.hidden, h.w2t.p, h.hidden, h.hidden, h.hidden, h.stream);
    transpose(h.W16(2), h.hidden, h.w3t.p, h.n_out, h.n_out, h.hidden, h.stream);
}

// Y of the batch in x16, or, for a gradient (t: the targets, row r's at row
// idx[r]), its loss's derivative and, transposed too, the layers' outputs.
int forward(Mlp& h, int B, const float* t, const int32_t* idx) {
    int rc;
    GemmArgs g = args(B, h.hidden, h.n_in, h.x16.p, h.n_in, h.W16(0), h.n_in, &h.status->err);
    g.bias = h.Bv(0);
    g.relu = 1;
    g.out16 = h.h1.p;
    g.ld16 = h.hidden;
    g.out16t = t != nullptr ? h.h1t.p : nullptr;
    g.ldt = B;
    if ((rc = gemm(g, nullptr, true, h.sms, h.stream)) != PDHG_OK) return rc;
    g = args(B, h.hidden, h.hidden, h.h1.p, h.hidden, h.W16(1), h.hidden, &h.status->err);
    g.bias = h.Bv(1);
    g.relu = 1;
    g.out16 = h.h2.p;
    g.ld16 = h.hidden;
    g.out16t = t != nullptr ? h.h2t.p : nullptr;
    g.ldt = B;
    if ((rc = gemm(g, nullptr, true, h.sms, h.stream)) != PDHG_OK) return rc;
    g = args(B, h.n_out, h.hidden, h.h2.p, h.hidden, h.W16(2), h.hidden, &h.status->err);
    g.bias = h.Bv(2);
    g.ld32 = h.n_out;
    if (t == nullptr) {
        g.out32 = h.y32.p;
    } else {
        g.target = t;
        g.idx = idx;
        g.scale = 1.f / static_cast<float>(static_cast<int64_t>(B) * h.n_out);
        g.part = h.part.p;
        g.out32 = h.dy32.p;
        g.out16 = h.dy16.p;
        g.ld16 = h.n_out;
        g.out16t = h.dyt.p;
        g.ldt = B;
    }
    return gemm(g, nullptr, true, h.sms, h.stream);
}

// Gradients into h.g after forward() with targets; the batch's loss to *loss.
int backward(Mlp& h, int B, double* loss) {
    int rc;
    int* err = &h.status->err;
    // layer 3's weights and layer 2's input
    GemmArgs g = args(h.n_out, h.hidden, B, h.dyt.p, B, h.h2t.p, B, err);
    g.out32 = h.gW(2);
    g.ld32 = h.hidden;
    GemmArgs d = args(B, h.hidden, h.n_out, h.dy16.p, h.n_out, h.w3t.p, h.n_out, err);
    d.mask = h.h2.p;
    d.ldm = h.hidden;
    d.out32 = h.dz2_32.p;
    d.ld32 = h.hidden;
    d.out16 = h.dz2_16.p;
    d.ld16 = h.hidden;
    d.out16t = h.dz2t.p;
    d.ldt = B;
    if ((rc = gemm(g, &d, true, h.sms, h.stream)) != PDHG_OK) return rc;
    // layer 2's weights and layer 1's input
    g = args(h.hidden, h.hidden, B, h.dz2t.p, B, h.h1t.p, B, err);
    g.out32 = h.gW(1);
    g.ld32 = h.hidden;
    d = args(B, h.hidden, h.hidden, h.dz2_16.p, h.hidden, h.w2t.p, h.hidden, err);
    d.mask = h.h1.p;
    d.ldm = h.hidden;
    d.out32 = h.dz1_32.p;
    d.ld32 = h.hidden;
    d.out16t = h.dz1t.p;
    d.ldt = B;
    if ((rc = gemm(g, &d, true, h.sms, h.stream)) != PDHG_OK) return rc;
    // layer 1's weights
    g = args(h.hidden, h.n_in, B, h.dz1t.p, B, h.xt.p, B, err);
    g.out32 = h.gW(0);
    g.ld32 = h.n_in;
    if ((rc = gemm(g, nullptr, true, h.sms, h.stream)) != PDHG_OK) return rc;
    ColSums c{};
    const float* dz[3] = {h.dy32.p, h.dz2_32.p, h.dz1_32.p};
    const int n[3] = {h.n_out, h.hidden, h.hidden};
    for (int i = 0; i < 3; ++i) {
        c.dz[i] = dz[i];
        c.db[i] = h.gB(2 - i);
        c.N[i] = n[i];
        c.first[i + 1] = c.first[i] + blocks(n[i], 32);
    }
    c.B = B;
    c.part = h.part.p;
    c.n_part = loss_parts(B, h.n_out, h.sms);
    c.loss = loss;
    return launch_pass(k_colsums, c.first[3] + 1, true, h.stream, c) == cudaSuccess ? PDHG_OK : PDHG_ERR_BACKEND;
}

// The batch's inputs (rows idx, null: in order) in BF16, transposed too for a gradient.
int set_batch(Mlp& h, int B, const float* x, const int32_t* idx, bool gradient) {
    k_gather_rows<<<blocks(B, 32) * blocks(h.n_in, 32), dim3(32, 8), 0, h.stream>>>(
        x, h.n_in, idx, B, h.x16.p, gradient ? h.xt.p : nullptr);
    MCK(cudaGetLastError());
    return PDHG_OK;
}

int upload_batch(Mlp& h, int B, const float* x, const float* t) {
    MCK(cudaMemcpyAsync(h.x32.p, x, sizeof(float) * B * h.n_in, cudaMemcpyHostToDevice, h.stream));
    if (t != nullptr)
        MCK(cudaMemcpyAsync(h.t32.p, t, sizeof(float) * B * h.n_out, cudaMemcpyHostToDevice, h.stream));
    return set_batch(h, B, h.x32.p, nullptr, t != nullptr);
}

bool batch_ok(const Mlp& h, int B) { return B >= 8 && B % 8 == 0 && B <= h.max_batch; }

}  // namespace
}  // namespace pdhg

struct pdhg_mlp {
    pdhg::Mlp h;
};

extern "C" {

int pdhg_mlp_create(int device, int n_in, int hidden, int n_out, int max_batch, pdhg_mlp** out) {
    using namespace pdhg;
    if (out == nullptr) return PDHG_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    if (n_in < 8 || n_in % 8 || hidden < 8 || hidden % 8 || n_out < 8 || n_out % 8 ||
        max_batch < 8 || max_batch % 8)
        return PDHG_ERR_INVALID_ARGUMENT;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev)
        return PDHG_ERR_UNSUPPORTED;
    std::unique_ptr<pdhg_mlp> p(new (std::nothrow) pdhg_mlp());
    if (!p) return PDHG_ERR_OUT_OF_MEMORY;
    Mlp& h = p->h;
    h.device = device;
    h.n_in = n_in;
    h.hidden = hidden;
    h.n_out = n_out;
    h.max_batch = max_batch;
    MCK(cudaSetDevice(device));
    MCK(init_gemm());
    MCK(cudaDeviceGetAttribute(&h.sms, cudaDevAttrMultiProcessorCount, device));
    MCK(cudaStreamCreateWithFlags(&h.stream, cudaStreamNonBlocking));
    const int64_t sizes[6] = {static_cast<int64_t>(hidden) * n_in, hidden,
                              static_cast<int64_t>(hidden) * hidden, hidden,
                              static_cast<int64_t>(n_out) * hidden, n_out};
    int64_t o = 0;
    for (int i = 0; i < 6; ++i) {
        h.off[i] = o;
        h.cnt[i] = sizes[i];
        o += (sizes[i] + 7) / 8 * 8;  // 16-byte aligned BF16 sub-arrays
    }
    h.total = o;
    const size_t B = static_cast<size_t>(max_batch), H = hidden;
    MCK(h.w.alloc(o));
    MCK(h.g.alloc(o));
    MCK(h.m.alloc(o));
    MCK(h.v.alloc(o));
    MCK(h.w16.alloc(o));
    MCK(h.w2t.alloc(H * H));
    MCK(h.w3t.alloc(H * n_out));
    MCK(h.x16.alloc(B * n_in));
    MCK(h.x32.alloc(B * n_in));
    MCK(h.xt.alloc(B * n_in));
    MCK(h.h1.alloc(B * H));
    MCK(h.h1t.alloc(B * H));
    MCK(h.h2.alloc(B * H));
    MCK(h.h2t.alloc(B * H));
    MCK(h.dy16.alloc(B * n_out));
    MCK(h.dyt.alloc(B * n_out));
    MCK(h.dz2_16.alloc(B * H));
    MCK(h.dz2t.alloc(B * H));
    MCK(h.dz1t.alloc(B * H));
    MCK(h.t32.alloc(B * n_out));
    MCK(h.y32.alloc(B * n_out));
    MCK(h.dy32.alloc(B * n_out));
    MCK(h.dz2_32.alloc(B * H));
    MCK(h.dz1_32.alloc(B * H));
    // a batch of fewer rows has narrower tiles, up to one per SM
    MCK(h.part.alloc(std::max(loss_parts(max_batch, n_out, h.sms), h.sms)));
    MCK(cudaHostAlloc(reinterpret_cast<void**>(&h.status), sizeof(Mlp::Status), cudaHostAllocDefault));
    *h.status = Mlp::Status{};
    MCK(cudaMemsetAsync(h.w.p, 0, sizeof(float) * o, h.stream));
    MCK(cudaMemsetAsync(h.m.p, 0, sizeof(float) * o, h.stream));
    MCK(cudaMemsetAsync(h.v.p, 0, sizeof(float) * o, h.stream));
    MCK(cudaStreamSynchronize(h.stream));
    *out = p.release();
    return PDHG_OK;
}

int pdhg_mlp_destroy(pdhg_mlp* p) {
    if (p == nullptr) return PDHG_ERR_INVALID_ARGUMENT;
    cudaSetDevice(p->h.device);
    if (p->h.stream != nullptr) cudaStreamSynchronize(p->h.stream);
    delete p;
    return PDHG_OK;
}

const char* pdhg_mlp_last_error(const pdhg_mlp* p) {
    return p == nullptr ? "null network" : p->h.err.c_str();
}

int64_t pdhg_mlp_param_count(const pdhg_mlp* p) {
    if (p == nullptr) return -1;
    int64_t s = 0;
    for (int i = 0; i < 6; ++i) s += p->h.cnt[i];
    return s;
}

// params: [W1 (hidden x n_in), b1, W2 (hidden x hidden), b2, W3 (n_out x hidden), b3]
int pdhg_mlp_set_params(pdhg_mlp* p, const float* params) {
    using namespace pdhg;
    if (p == nullptr || params == nullptr) return PDHG_ERR_INVALID_ARGUMENT;
    Mlp& h = p->h;
    MCK(cudaSetDevice(h.device));
    int64_t src = 0;
    for (int i = 0; i < 6; ++i) {
        MCK(cudaMemcpyAsync(h.w.p + h.off[i], params + src, sizeof(float) * h.cnt[i],
                            cudaMemcpyHostToDevice, h.stream));
        src += h.cnt[i];
    }
    MCK(cudaMemsetAsync(h.m.p, 0, sizeof(float) * h.total, h.stream));
    MCK(cudaMemsetAsync(h.v.p, 0, sizeof(float) * h.total, h.stream));
    h.adam_t = 0;
    refresh_weights(h);
    MCK(cudaStreamSynchronize(h.stream));
    return PDHG_OK;
}

int pdhg_mlp_get_params(pdhg_mlp* p, float* params) {
    using namespace pdhg;
    if (p == nullptr || params == nullptr) return PDHG_ERR_INVALID_ARGUMENT;
    Mlp& h = p->h;
    MCK(cudaSetDevice(h.device));
    int64_t dst = 0;
    for (int i = 0; i < 6; ++i) {
        MCK(cudaMemcpyAsync(params + dst, h.w.p + h.off[i], sizeof(float) * h.cnt[i],
                            cudaMemcpyDeviceToHost, h.stream));
        dst += h.cnt[i];
    }
    MCK(cudaStreamSynchronize(h.stream));
    return PDHG_OK;
}

int pdhg_mlp_forward(pdhg_mlp* p, int batch, const float* x, float* y) {
    using namespace pdhg;
    if (p == nullptr || x == nullptr || y == nullptr || !batch_ok(p->h, batch))
        return PDHG_ERR_INVALID_ARGUMENT;
    Mlp& h = p->h;
    MCK(cudaSetDevice(h.device));
    int rc = upload_batch(h, batch, x, nullptr);
    if (rc != PDHG_OK) return rc;
    if ((rc = forward(h, batch, nullptr, nullptr)) != PDHG_OK) return rc;
    MCK(cudaMemcpyAsync(y, h.y32.p, sizeof(float) * batch * h.n_out, cudaMemcpyDeviceToHost,
                        h.stream));
    return check_err(h);
}

int pdhg_mlp_gradients(pdhg_mlp* p, int batch, const float* x, const float* t, float* grads,
                       float* loss) {
    using namespace pdhg;
    if (p == nullptr || x == nullptr || t == nullptr || grads == nullptr ||
        !batch_ok(p->h, batch))
        return PDHG_ERR_INVALID_ARGUMENT;
    Mlp& h = p->h;
    MCK(cudaSetDevice(h.device));
    int rc = upload_batch(h, batch, x, t);
    if (rc != PDHG_OK) return rc;
    if ((rc = forward(h, batch, h.t32.p, nullptr)) != PDHG_OK) return rc;
    if ((rc = backward(h, batch, &h.status->loss)) != PDHG_OK) return rc;
    // every section is a multiple of 8 entries (the dimensions are): one block
    MCK(cudaMemcpyAsync(grads, h.g.p, sizeof(float) * h.total, cudaMemcpyDeviceToHost, h.stream));
    rc = check_err(h);
    if (loss != nullptr) *loss = static_cast<float>(h.status->loss);
    return rc;
}

// One Adam step with gradients from outside (parameter order, host FP32):
// the update of data-parallel training, where every replica applies the
// gradients all ranks have averaged. The step counter is the one
// pdhg_mlp_train advances, and the hyper-parameters are its own.
int pdhg_mlp_adam_step(pdhg_mlp* p, const float* grads, float lr) {
    using namespace pdhg;
    if (p == nullptr || grads == nullptr || !(lr > 0.f)) return PDHG_ERR_INVALID_ARGUMENT;
    Mlp& h = p->h;
    MCK(cudaSetDevice(h.device));
    int64_t src = 0;
    for (int i = 0; i < 6; ++i) {
        MCK(cudaMemcpyAsync(h.g.p + h.off[i], grads + src, sizeof(float) * h.cnt[i],
                            cudaMemcpyHostToDevice, h.stream));
        src += h.cnt[i];
    }
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    h.adam_t += 1;
    const float c1 = 1.f - std::pow(b1, static_cast<float>(h.adam_t));
    const float c2 = 1.f - std::pow(b2, static_cast<float>(h.adam_t));
    k_adam<<<blocks(h.total, 256), 256, 0, h.stream>>>(h.w.p, h.g.p, h.m.p, h.v.p, h.w16.p,
                                                      h.total, lr, b1, b2, eps, c1, c2);
    transpose(h.W16(1), h.hidden, h.w2t.p, h.hidden, h.hidden, h.hidden, h.stream);
    transpose(h.W16(2), h.hidden, h.w3t.p, h.n_out, h.n_out, h.hidden, h.stream);
    MCK(cudaStreamSynchronize(h.stream));
    return check_err(h);
}

// Adam over `epochs` passes of shuffled mini-batches of the samples x (S x
// n_in) with targets t (S x n_out); the last incomplete batch of an epoch is
// dropped. epoch_loss (epochs entries, may be NULL) gets each epoch's mean
// batch loss.
int pdhg_mlp_train(pdhg_mlp* p, int64_t samples, const float* x, const float* t, int epochs,
                   int batch, float lr, uint64_t seed, float* epoch_loss) {
    using namespace pdhg;
    if (p == nullptr || x == nullptr || t == nullptr || epochs < 0 || samples < batch ||
        !batch_ok(p->h, batch) || !(lr > 0.f))
        return PDHG_ERR_INVALID_ARGUMENT;
    Mlp& h = p->h;
    MCK(cudaSetDevice(h.device));
    MCK(h.xs.alloc(static_cast<size_t>(samples) * h.n_in));
    MCK(h.ts.alloc(static_cast<size_t>(samples) * h.n_out));
    MCK(cudaMemcpyAsync(h.xs.p, x, sizeof(float) * samples * h.n_in, cudaMemcpyHostToDevice,
                        h.stream));
    MCK(cudaMemcpyAsync(h.ts.p, t, sizeof(float) * samples * h.n_out, cudaMemcpyHostToDevice,
                        h.stream));
    std::mt19937_64 rng(seed);
    std::vector<int32_t> perm(static_cast<size_t>(samples));
    const int steps = static_cast<int>(samples / batch);
    Dev<int32_t> perm_d;
    MCK(perm_d.alloc(static_cast<size_t>(samples)));
    std::vector<double> losses(static_cast<size_t>(steps));
    Dev<double> lsum;
    MCK(lsum.alloc(static_cast<size_t>(steps) + 1));
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    for (int ep = 0; ep < epochs; ++ep) {
        for (int64_t i = 0; i < samples; ++i) perm[i] = static_cast<int32_t>(i);
        std::shuffle(perm.begin(), perm.end(), rng);
        MCK(cudaMemcpyAsync(perm_d.p, perm.data(), sizeof(int32_t) * samples,
                            cudaMemcpyHostToDevice, h.stream));
        for (int sI = 0; sI < steps; ++sI) {
            const int32_t* idx = perm_d.p + static_cast<int64_t>(sI) * batch;
            int rc = set_batch(h, batch, h.xs.p, idx, true);
            if (rc == PDHG_OK) rc = forward(h, batch, h.ts.p, idx);
            if (rc == PDHG_OK) rc = backward(h, batch, lsum.p + sI);
            if (rc != PDHG_OK) return rc;
            h.adam_t += 1;
            const float c1 = 1.f - std::pow(b1, static_cast<float>(h.adam_t));
            const float c2 = 1.f - std::pow(b2, static_cast<float>(h.adam_t));
            k_adam<<<blocks(h.total, 256), 256, 0, h.stream>>>(h.w.p, h.g.p, h.m.p, h.v.p, h.w16.p,
                                                              h.total, lr, b1, b2, eps, c1, c2);
            transpose(h.W16(1), h.hidden, h.w2t.p, h.hidden, h.hidden, h.hidden, h.stream);
            transpose(h.W16(2), h.hidden, h.w3t.p, h.n_out, h.n_out, h.hidden, h.stream);
        }
        MCK(cudaMemcpyAsync(losses.data(), lsum.p, sizeof(double) * steps, cudaMemcpyDeviceToHost,
                            h.stream));
        MCK(cudaStreamSynchronize(h.stream));
        if (epoch_loss != nullptr) {
            double s = 0.0;
            for (double l : losses) s += l;
            epoch_loss[ep] = static_cast<float>(s / steps);
        }
    }
    return check_err(h);
}

// The tensor-core GEMM on its own (test entry): C = A B^T (+ bias, ReLU) with
// A (m x k) and B (n x k) given in FP32 on the host and rounded to BF16, FP32
// accumulation, C (m x n) FP32 on the host. k must be a multiple of 8.
int pdhg_gemm_bf16(int device, int m, int n, int k, const float* a, const float* b,
                   const float* bias, int relu, float* c) {
    using namespace pdhg;
    if (m < 1 || n < 1 || k < 8 || k % 8 || a == nullptr || b == nullptr || c == nullptr)
        return PDHG_ERR_INVALID_ARGUMENT;
    if (cudaSetDevice(device) != cudaSuccess) return PDHG_ERR_UNSUPPORTED;
    int sms = 0;
    if (init_gemm() != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
        return PDHG_ERR_BACKEND;
    Dev<float> a32, b32, c32, bias32;
    Dev<bf16> a16, b16;
    Dev<int> err;
    const size_t na = static_cast<size_t>(m) * k, nb = static_cast<size_t>(n) * k;
    if (a32.alloc(na) || b32.alloc(nb) || c32.alloc(static_cast<size_t>(m) * n) ||
        a16.alloc(na) || b16.alloc(nb) || err.alloc(1) || (bias && bias32.alloc(n)))
        return PDHG_ERR_OUT_OF_MEMORY;
    cudaMemcpy(a32.p, a, sizeof(float) * na, cudaMemcpyHostToDevice);
    cudaMemcpy(b32.p, b, sizeof(float) * nb, cudaMemcpyHostToDevice);
    if (bias) cudaMemcpy(bias32.p, bias, sizeof(float) * n, cudaMemcpyHostToDevice);
    cudaMemset(err.p, 0, sizeof(int));
    k_to_bf16<<<blocks(na, 256), 256>>>(a32.p, a16.p, na);
    k_to_bf16<<<blocks(nb, 256), 256>>>(b32.p, b16.p, nb);
    GemmArgs g = args(m, n, k, a16.p, k, b16.p, k, err.p);
    g.bias = bias ? bias32.p : nullptr;
    g.relu = relu;
    g.out32 = c32.p;
    g.ld32 = n;
    int rc = gemm(g, nullptr, false, sms, nullptr);
    if (rc != PDHG_OK) return rc;
    int e = 0;
    if (cudaMemcpy(&e, err.p, sizeof e, cudaMemcpyDeviceToHost) != cudaSuccess) return PDHG_ERR_BACKEND;
    if (e != 0) return PDHG_ERR_BACKEND;
    if (cudaMemcpy(c, c32.p, sizeof(float) * m * n, cudaMemcpyDeviceToHost) != cudaSuccess)
        return PDHG_ERR_BACKEND;
    return PDHG_OK;
}

}  // extern "C"
