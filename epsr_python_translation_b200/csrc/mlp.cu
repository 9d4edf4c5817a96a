// mlp.cu -- the surrogate network of the delayed-acceptance Monte Carlo: a 1280 -> 128 -> 128
// -> 1 perceptron with SiLU activations, BF16 weights and activations, FP32 accumulation,
// evaluated and trained by one hand-written tcgen05 GEMM kernel with per-layer epilogues.
//
// The GEMM.  One CTA computes a 128 x TN tile D = A_tile . B_tile^T (TN 32, 64 or 128) over a K range
// (split-K over blockIdx.z): one thread streams 128 x 64 BF16 tiles of A and TN x 64 of B into a
// shared-memory ring with TMA (SWIZZLE_128B, K-major), another issues four tcgen05.mma (M = 128, N = TN,
// K = 16) per stage and commits each stage back to its ring slot; the FP32 accumulator lives in TN
// columns of tensor memory.  The matrices are small (a few hundred to a few thousand rows), so what
// bounds a launch is the latency of one tile, not the tensor cores: the ring holds as much of K as
// fits, layers whose epilogue works column by column are cut into 32-column tiles (four times the
// CTAs), and every warp's epilogue is 32 rows x 32 columns held in registers (tcgen05.ld 32x32b), written
// 16 bytes at a time, its column sums formed by a butterfly that halves the columns as it halves the
// rows (31 shuffles for 32 columns).  2,048 rows, us: layer 1 14, layer 2 with the head and its gradients
// 13, its backward pass 14, both weight gradients 12; 59, 62, 44 and 31 with four warps a tile, a row a
// thread and one thread alone at the ring.
// Epilogues:
//   STORE      D as FP32 (the raw product, for tests);
//   ATOMIC     D added into an FP32 matrix (the weight gradients, split over K = samples);
//   BIAS_SILU  z = D + b, h = silu(z): h in BF16 (row-major, and transposed for the weight
//              gradient), z in FP32 when training;
//   HEAD       z = D + b, h = silu(z), y = h . w3 + b3 per row; when training, rows come in
//              pairs (features before/after, after/before) whose antisymmetric part
//              s = (y0 - y1)/2 is fitted to the target: the loss, dL/dy, dz = dL/dy w3 silu'(z)
//              in BF16 (row-major and transposed) and the w3, b3, b2 gradients;
//   SILU_BWD   dz = D silu'(z_saved) (D = dz2 . W2), BF16 transposed, and the b1 gradient.
// Every mbarrier wait is bounded (2 s): on timeout the kernel records status 1 and returns
// after releasing its tensor memory.
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <mutex>

#include "common.cuh"
#include "umma.cuh"

namespace epsr {

using bf16 = __nv_bfloat16;
constexpr int MLP_IN = 1280, MLP_H = 128;
__host__ __device__ constexpr int g_stages(int tn) { return tn == 32 ? 10 : tn == 64 ? 8 : 6; }
__host__ __device__ constexpr int g_threads(int tn) { return 128 * (tn / 32); }
__host__ __device__ constexpr size_t g_stage_bytes(int tn) { return umma::TILE_BYTES + (size_t)tn * umma::TILE_K * 2; }
__host__ __device__ constexpr size_t g_smem(int tn) { return 1024 + g_stages(tn) * g_stage_bytes(tn); }   // + alignment slack

enum Epi : int { EPI_STORE = 0, EPI_ATOMIC = 1, EPI_BIAS_SILU = 2, EPI_HEAD = 3, EPI_SILU_BWD = 4 };

struct GemmArgs {
    int M, N, K, kslices, epi;
    float *out;
    int ldo;
    const float *bias;
    float *z_out;           // [M][N] FP32 pre-activation (BIAS_SILU, training)
    bf16 *h_out;            // [M][N] BF16 activation (BIAS_SILU)
    bf16 *ht_out;           // [N][ldt] BF16 transposed activation (BIAS_SILU, training)
    int ldt;                // leading dimension of the transposed outputs (>= M)
    const float *w3;        // [N] (HEAD)
    const float *b3;        // [1] (HEAD)
    float *y;               // [M] (HEAD)
    const float *target;    // [M/2] antisymmetric targets (HEAD, training), or null
    float gscale;           // dL/dy scale (1 / number of pairs)
    float *loss;            // [1] sum of squared pair errors (HEAD, training)
    float *dw3, *db3, *db;  // gradients (HEAD: w3, b3, b2; SILU_BWD: b1 in db)
    bf16 *dz_out;           // [M][N] BF16 (HEAD, training)
    bf16 *dzt_out;          // [N][ldt] BF16 transposed (HEAD and SILU_BWD, training)
    const float *z_in;      // [M][N] saved pre-activation (SILU_BWD)
    int *status;
};

__device__ __forceinline__ float sigm(float z) { return 1.0f / (1.0f + __expf(-z)); }
__device__ __forceinline__ float silu(float z) { return z * sigm(z); }
__device__ __forceinline__ float dsilu(float z) {
    const float s = sigm(z);
    return s * (1.0f + z * (1.0f - s));
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// s[c] of 32 lanes -> lane c holds the sum of s[c] over the lanes (the pairs of warp_sum)
__device__ __forceinline__ float column_sums(float (&s)[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const float keep = up ? s[i + o] : s[i], send = up ? s[i] : s[i + o];
            s[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return s[0];
}
// 32 floats, 16 bytes at a time where the caller's array is so aligned
__device__ __forceinline__ void load32(float (&d)[32], const float *p) {
    if (((uintptr_t)p & 15) == 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float4 v = __ldg((const float4 *)p + i);
            d[4 * i] = v.x, d[4 * i + 1] = v.y, d[4 * i + 2] = v.z, d[4 * i + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) d[i] = __ldg(p + i);
    }
}
// 32 BF16 of a row, 64 bytes
__device__ __forceinline__ void store_row(bf16 *out, const bf16 (&h)[32]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            w[k] = (uint32_t)__bfloat16_as_ushort(h[8 * i + 2 * k]) | ((uint32_t)__bfloat16_as_ushort(h[8 * i + 2 * k + 1]) << 16);
        ((uint4 *)out)[i] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// CTAs with blockIdx.y >= ny take the second product (its maps, shape and output).
template <int TN>
__global__ void __launch_bounds__(g_threads(TN)) umma_gemm_kernel(const __grid_constant__ CUtensorMap ta0,
                                                                  const __grid_constant__ CUtensorMap tb0, GemmArgs g0,
                                                                  const __grid_constant__ CUtensorMap ta1,
                                                                  const __grid_constant__ CUtensorMap tb1, GemmArgs g1,
                                                                  int ny) {
    constexpr int STAGES = g_stages(TN);
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full[STAGES], empty[STAGES], done;
    __shared__ uint32_t tmem_base;
    __shared__ float sacc[umma::TILE_M];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const bool second = (int)blockIdx.y >= ny;
    const CUtensorMap *ta = second ? &ta1 : &ta0, *tb = second ? &tb1 : &tb0;
    const GemmArgs &g = second ? g1 : g0;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * umma::TILE_M, n0 = ((int)blockIdx.y - (second ? ny : 0)) * TN;
    const int nkb = g.K / umma::TILE_K;
    const int kb0 = (int)((long long)blockIdx.z * nkb / g.kslices);
    const int kb1 = (int)((long long)(blockIdx.z + 1) * nkb / g.kslices);
    const int nk = kb1 - kb0;
    if (warp == 0) {
        umma::tmem_alloc(&tmem_base, TN);
        umma::tmem_relinquish();
    }
    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            umma::mbar_init(&full[s], 1);
            umma::mbar_init(&empty[s], 1);
        }
        umma::mbar_init(&done, 1);
        umma::fence_mbar_init();
    }
    umma::tc_fence_before();
    __syncthreads();
    umma::tc_fence_after();
    const uint32_t tmem = tmem_base;
    auto stage_a = [&](int s) { return smem + (size_t)s * g_stage_bytes(TN); };
    auto stage_b = [&](int s) { return smem + (size_t)s * g_stage_bytes(TN) + umma::TILE_BYTES; };
    if (tid == 32) {          // the ring's producer
        for (int i = 0; i < nk; ++i) {
            const int s = i % STAGES;
            if (i >= STAGES && !umma::mbar_wait(&empty[s], (uint32_t)(i / STAGES - 1) & 1u, g.status)) break;
            umma::mbar_expect_tx(&full[s], (uint32_t)g_stage_bytes(TN));
            umma::tma_load_2d(stage_a(s), ta, (kb0 + i) * umma::TILE_K, m0, &full[s]);
            umma::tma_load_2d(stage_b(s), tb, (kb0 + i) * umma::TILE_K, n0, &full[s]);
        }
    } else if (tid == 0) {    // its consumer
        constexpr uint32_t idesc = umma::idesc_bf16_f32(umma::TILE_M, TN);
        for (int i = 0; i < nk; ++i) {
            const int s = i % STAGES;
            if (!umma::mbar_wait(&full[s], (uint32_t)(i / STAGES) & 1u, g.status)) break;
            umma::tc_fence_after();
            const uint64_t ad = umma::sdesc_sw128(stage_a(s)), bd = umma::sdesc_sw128(stage_b(s));
#pragma unroll
            for (int kk = 0; kk < umma::TILE_K / 16; ++kk)   // 32 bytes (16 BF16) further per K-slice
                umma::mma_bf16(tmem, ad + 2 * kk, bd + 2 * kk, idesc, (i > 0 || kk > 0) ? 1u : 0u);
            umma::mma_commit(&empty[s]);
        }
        umma::mma_commit(&done);
    }
    __syncwarp();
    // this warp's 32 rows (those its tensor-memory lanes hold) and 32 columns
    const int rl = (warp & 3) * 32 + lane, row = m0 + rl, c0 = (warp >> 2) * 32, n = n0 + c0;
    const bool rv = row < g.M;
    float bias[32], w3[32];
    if (g.epi == EPI_BIAS_SILU || g.epi == EPI_HEAD) {   // while the product runs
        load32(bias, g.bias + n);
        if (g.epi == EPI_HEAD) load32(w3, g.w3 + n);
    } else if (g.epi == EPI_SILU_BWD && rv) {
        load32(bias, g.z_in + (size_t)row * g.N + n);
    }
    const bool ok = umma::mbar_wait(&done, 0, g.status) && nk > 0;
    umma::tc_fence_after();
    float v[32];
    if (ok) {
        const uint32_t t = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0;
        float u[16];
        umma::tmem_ld16(t, u);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = u[i];
        umma::tmem_ld16(t + 16, u);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[16 + i] = u[i];
    }
    if (ok && (g.epi == EPI_STORE || g.epi == EPI_ATOMIC)) {
        float *o = g.out + (size_t)row * g.ldo + n;
        if (rv && n + 32 <= g.N && ((uintptr_t)o & 15) == 0) {
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
                if (g.epi == EPI_STORE) *(float4 *)(o + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                else
                    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(o + i), "f"(v[i]), "f"(v[i + 1]),
                                 "f"(v[i + 2]), "f"(v[i + 3])
                                 : "memory");
            }
        } else if (rv) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
                if (n + i < g.N) {
                    if (g.epi == EPI_STORE) o[i] = v[i];
                    else atomicAdd(o + i, v[i]);
                }
        }
    } else if (ok && g.epi == EPI_BIAS_SILU) {
        bf16 h[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            v[i] += bias[i];
            h[i] = __float2bfloat16_rn(silu(v[i]));
        }
        if (rv) {
            store_row(g.h_out + (size_t)row * g.N + n, h);
            if (g.z_out) {
                float4 *z = (float4 *)(g.z_out + (size_t)row * g.N + n);
#pragma unroll
                for (int i = 0; i < 8; ++i) z[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            }
            if (g.ht_out) {
#pragma unroll
                for (int i = 0; i < 32; ++i) g.ht_out[(size_t)(n + i) * g.ldt + row] = h[i];
            }
        }
    } else if (g.epi == EPI_HEAD) {   // TN = 128: the whole row; every warp passes the barriers
        float p[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            v[i] = ok ? v[i] + bias[i] : 0.0f;
            p[i] = silu(v[i]) * w3[i];
        }
        // the row's sum in column order, 32 columns a warp in turn
        for (int k = 0; k < TN / 32; ++k) {
            if (c0 == 32 * k) {
                float acc = k ? sacc[rl] : 0.0f;
#pragma unroll
                for (int i = 0; i < 32; ++i) acc += p[i];
                sacc[rl] = acc;
            }
            __syncthreads();
        }
        const float y = sacc[rl] + *g.b3;
        if (ok && rv && c0 == 0) g.y[row] = y;
        if (ok && g.target) {
            // rows 2p, 2p+1 are the two orders of pair p (adjacent lanes of one warp)
            const float yo = __shfl_xor_sync(0xffffffffu, y, 1);
            const bool even = (lane & 1) == 0;
            const float s = even ? 0.5f * (y - yo) : 0.5f * (yo - y);
            const float diff = rv ? s - g.target[row >> 1] : 0.0f;
            const float gy = rv ? (even ? diff : -diff) * g.gscale : 0.0f;
            if (c0 == 0) {
                const float l = warp_sum((even && rv) ? diff * diff : 0.0f);
                const float gb3 = warp_sum(gy);
                if (lane == 0) {
                    atomicAdd(g.loss, l);
                    atomicAdd(g.db3, gb3);
                }
            }
            bf16 dzb[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                p[i] = gy * silu(v[i]);
                v[i] = gy * w3[i] * dsilu(v[i]);
                dzb[i] = __float2bfloat16_rn(v[i]);
            }
            if (rv) {
                store_row(g.dz_out + (size_t)row * g.N + n, dzb);
#pragma unroll
                for (int i = 0; i < 32; ++i) g.dzt_out[(size_t)(n + i) * g.ldt + row] = dzb[i];
            }
            atomicAdd(g.dw3 + n + lane, column_sums(p));
            atomicAdd(g.db + n + lane, column_sums(v));
        }
    } else if (ok && g.epi == EPI_SILU_BWD) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            v[i] = rv ? v[i] * dsilu(bias[i]) : 0.0f;
            if (rv) g.dzt_out[(size_t)(n + i) * g.ldt + row] = __float2bfloat16_rn(v[i]);
        }
        atomicAdd(g.db + n + lane, column_sums(v));
    }
    umma::tc_fence_before();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(tmem, TN);
}

// ----------------------------------------------------------------- Adam
// Every parameter array in one launch; m and v are laid out as the arrays follow one another.
struct AdamPart {
    float *w, *grad;
    bf16 *wh;      // BF16 copy [n] (or null)
    bf16 *wht;     // BF16 transposed copy of a rows x cols matrix (or null)
    int n, rows, cols;
};
struct AdamArgs {
    AdamPart part[6];
    float *m, *v;
    float lr, b1, b2, eps, c1, c2, wd;
};

__global__ void adam_kernel(AdamArgs a) {
    const int at = blockIdx.x * blockDim.x + threadIdx.x;
    int i = at, k = 0;
    while (k < 6 && i >= a.part[k].n) i -= a.part[k++].n;
    if (k == 6) return;
    const AdamPart &p = a.part[k];
    const float gr = p.grad[i];
    const float m = a.b1 * a.m[at] + (1.0f - a.b1) * gr;
    const float v = a.b2 * a.v[at] + (1.0f - a.b2) * gr * gr;
    a.m[at] = m;
    a.v[at] = v;
    float w = p.w[i];
    w -= a.lr * ((m * a.c1) / (sqrtf(v * a.c2) + a.eps) + a.wd * w);
    p.w[i] = w;
    p.grad[i] = 0.0f;
    if (p.wh) p.wh[i] = __float2bfloat16_rn(w);
    if (p.wht) {
        const int r = i / p.cols, c = i % p.cols;
        p.wht[(size_t)c * p.rows + r] = __float2bfloat16_rn(w);
    }
}

__global__ void to_bf16_kernel(const float *w, bf16 *wh, bf16 *wht, int rows, int cols) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows * cols) return;
    const bf16 h = __float2bfloat16_rn(w[i]);
    if (wh) wh[i] = h;
    if (wht) wht[(size_t)(i % cols) * rows + i / cols] = h;
}

// ----------------------------------------------------------------- host side
namespace {
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
std::mutex g_encode_mu;

int get_encode() {
    std::lock_guard<std::mutex> lk(g_encode_mu);
    if (g_encode) return EPSR_OK;
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
    if (e != cudaSuccess || !fn || q != cudaDriverEntryPointSuccess) {
        epsr_set_error("cuTensorMapEncodeTiled is not available from the driver");
        return EPSR_ERR_CUDA;
    }
    g_encode = (PFN_cuTensorMapEncodeTiled_v12000)fn;
    return EPSR_OK;
}

// Tensor map of a row-major BF16 matrix [rows][cols] (cols contiguous, ld elements between
// rows) read in box_rows x 64 boxes with the 128-byte swizzle.  cols and ld must be multiples of 64
// and the base 16-byte aligned, so every box starts on a 16-byte boundary (x = 64 k); rows
// beyond the matrix read as zero.
int make_map(CUtensorMap *m, const void *base, int64_t rows, int64_t cols, int64_t ld, int box_rows) {
    int rc = get_encode();
    if (rc) return rc;
    if (((uintptr_t)base & 15) || cols % umma::TILE_K || ld % umma::TILE_K || ld < cols || rows <= 0) {
        epsr_set_error("tensor map: base %p must be 16-byte aligned, cols %lld and ld %lld multiples of 64", base,
                       (long long)cols, (long long)ld);
        return EPSR_ERR_ARG;
    }
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {(cuuint32_t)umma::TILE_K, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        epsr_set_error("cuTensorMapEncodeTiled failed (%d) for a %lld x %lld matrix", (int)r, (long long)rows,
                       (long long)cols);
        return EPSR_ERR_CUDA;
    }
    return EPSR_OK;
}

// D[M x N] over K: A [M][lda] and B [N][ldb] row-major BF16 (K contiguous).  The grid covers
// M in tiles of 128 and N in tiles of TN (rows past M of A and past N of B read as zero); K is a
// multiple of 64 and is split into kslices ranges (one CTA each, at least one 64-wide block apiece).
struct Product {
    const void *A;
    int64_t lda;
    const void *B;
    int64_t ldb;
    int M, N, K, kslices;
    GemmArgs g;
};
// one product, or two of the same M and kslices side by side in one launch
template <int TN>
int gemm(Product p, cudaStream_t s, Product *q = nullptr) {
    CUtensorMap t[4];
    Product *both[2] = {&p, q};
    for (int i = 0; i < (q ? 2 : 1); ++i) {
        Product &x = *both[i];
        if (x.M <= 0 || x.N <= 0 || x.K <= 0 || x.K % umma::TILE_K || x.kslices < 1 || x.kslices > x.K / umma::TILE_K) {
            epsr_set_error("umma gemm: bad shape M %d N %d K %d kslices %d", x.M, x.N, x.K, x.kslices);
            return EPSR_ERR_ARG;
        }
        int rc = make_map(&t[2 * i], x.A, x.M, x.K, x.lda, umma::TILE_M);
        if (rc) return rc;
        rc = make_map(&t[2 * i + 1], x.B, x.N, x.K, x.ldb, TN);
        if (rc) return rc;
        x.g.M = x.M;
        x.g.N = x.N;
        x.g.K = x.K;
        x.g.kslices = x.kslices;
    }
    const Product &r = q ? *q : p;
    const int ny = (p.N + TN - 1) / TN;
    EPSR_SMEM_OPTIN(umma_gemm_kernel<TN>);
    dim3 grid((p.M + 127) / 128, ny + (q ? (q->N + TN - 1) / TN : 0), p.kslices);
    EPSR_TIMED("umma_gemm_kernel", s, umma_gemm_kernel<TN><<<grid, g_threads(TN), g_smem(TN), s>>>(
        t[0], t[1], p.g, t[q ? 2 : 0], t[q ? 3 : 1], r.g, ny));
    EPSR_CUDA(cudaGetLastError());
    return EPSR_OK;
}
}  // namespace
}  // namespace epsr

using namespace epsr;

extern "C" int epsr_umma_gemm_f32(const void *a, int32_t m, const void *b, int32_t n, int32_t k, int32_t kslices,
                                  float *out, int32_t ldo, int32_t accumulate, int32_t *status, void *stream) {
    if (!a || !b || !out || !status || ldo < n) {
        epsr_set_error("epsr_umma_gemm_f32: null pointer or ldo < n");
        return EPSR_ERR_ARG;
    }
    GemmArgs g = {};
    g.epi = accumulate ? EPI_ATOMIC : EPI_STORE;
    g.out = out;
    g.ldo = ldo;
    g.status = status;
    return gemm<128>({a, k, b, k, m, n, k, kslices, g}, (cudaStream_t)stream);
}

extern "C" int64_t epsr_mlp_work_bytes(int32_t rows) {
    const int64_t R = ((int64_t)rows + 127) / 128 * 128;
    return 256 * 8 + R * MLP_H * (2 + 4 + 2 + 2 + 2 + 2) + R * 4 * 2 + 4096;
}

namespace {
struct MlpWork {
    bf16 *h1, *h1t, *dz2, *dz2t, *dz1t;
    float *z1, *y, *loss;
};
MlpWork carve(void *work, int R) {
    char *p = (char *)work;
    auto take = [&](size_t b) {
        char *r = p;
        p += (b + 255) & ~(size_t)255;
        return (void *)r;
    };
    MlpWork w;
    w.h1 = (bf16 *)take(sizeof(bf16) * (size_t)R * MLP_H);
    w.h1t = (bf16 *)take(sizeof(bf16) * (size_t)R * MLP_H);
    w.dz2 = (bf16 *)take(sizeof(bf16) * (size_t)R * MLP_H);
    w.dz2t = (bf16 *)take(sizeof(bf16) * (size_t)R * MLP_H);
    w.dz1t = (bf16 *)take(sizeof(bf16) * (size_t)R * MLP_H);
    w.z1 = (float *)take(sizeof(float) * (size_t)R * MLP_H);
    w.y = (float *)take(sizeof(float) * (size_t)R);
    w.loss = (float *)take(sizeof(float) * 8);
    return w;
}

int check_net(const epsr_mlp_t *net, const char *who) {
    if (!net || !net->w1 || !net->b1 || !net->w2 || !net->b2 || !net->w3 || !net->b3 || !net->w1h || !net->w2h ||
        !net->w2th || !net->status) {
        epsr_set_error("%s: null network pointer", who);
        return EPSR_ERR_ARG;
    }
    return EPSR_OK;
}

// the activations in the work area are stored, and read by TMA, 16 bytes at a time
bool work_aligned(const void *work, const char *who) {
    if (((uintptr_t)work & 15) == 0) return true;
    epsr_set_error("%s: work %p must be 16-byte aligned", who, work);
    return false;
}
}  // namespace

extern "C" int epsr_mlp_sync_weights(const epsr_mlp_t *net, void *stream) {
    int rc = check_net(net, "epsr_mlp_sync_weights");
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    to_bf16_kernel<<<(MLP_H * MLP_IN + 255) / 256, 256, 0, s>>>(net->w1, (bf16 *)net->w1h, nullptr, MLP_H, MLP_IN);
    to_bf16_kernel<<<(MLP_H * MLP_H + 255) / 256, 256, 0, s>>>(net->w2, (bf16 *)net->w2h, (bf16 *)net->w2th, MLP_H,
                                                                MLP_H);
    EPSR_CUDA(cudaGetLastError());
    return EPSR_OK;
}

extern "C" int epsr_mlp_forward(const epsr_mlp_t *net, const void *x, int32_t rows, float *y, void *work,
                                int64_t work_bytes, void *stream) {
    int rc = check_net(net, "epsr_mlp_forward");
    if (rc) return rc;
    if (!x || !y || !work || rows <= 0) {
        epsr_set_error("epsr_mlp_forward: null pointer or no rows");
        return EPSR_ERR_ARG;
    }
    if (!work_aligned(work, "epsr_mlp_forward")) return EPSR_ERR_ARG;
    if (work_bytes < epsr_mlp_work_bytes(rows)) {
        epsr_set_error("epsr_mlp_forward: work needs %lld bytes", (long long)epsr_mlp_work_bytes(rows));
        return EPSR_ERR_CAPACITY;
    }
    cudaStream_t s = (cudaStream_t)stream;
    MlpWork w = carve(work, (rows + 127) / 128 * 128);
    GemmArgs g1 = {};
    g1.epi = EPI_BIAS_SILU;
    g1.bias = net->b1;
    g1.h_out = w.h1;
    g1.status = net->status;
    rc = gemm<32>({x, MLP_IN, net->w1h, MLP_IN, rows, MLP_H, MLP_IN, 1, g1}, s);
    if (rc) return rc;
    GemmArgs g2 = {};
    g2.epi = EPI_HEAD;
    g2.bias = net->b2;
    g2.w3 = net->w3;
    g2.b3 = net->b3;
    g2.y = y;
    g2.status = net->status;
    return gemm<128>({w.h1, MLP_H, net->w2h, MLP_H, rows, MLP_H, MLP_H, 1, g2}, s);
}

extern "C" int epsr_mlp_train_step(const epsr_mlp_t *net, const void *x, const void *xt, int64_t ldxt, int32_t row0,
                                   int32_t rows, const float *target, float lr, int32_t step, float *loss_out,
                                   void *work, int64_t work_bytes, void *stream) {
    int rc = check_net(net, "epsr_mlp_train_step");
    if (rc) return rc;
    if (!x || !xt || !target || !work || rows <= 0 || rows % 128 || row0 % 128 || ldxt < row0 + rows || step < 1 ||
        !net->dw1 || !net->m1 || !net->v1) {
        epsr_set_error("epsr_mlp_train_step: null pointer, or rows/row0 not multiples of 128, or ldxt too small");
        return EPSR_ERR_ARG;
    }
    if (!work_aligned(work, "epsr_mlp_train_step")) return EPSR_ERR_ARG;
    if (work_bytes < epsr_mlp_work_bytes(rows)) {
        epsr_set_error("epsr_mlp_train_step: work needs %lld bytes", (long long)epsr_mlp_work_bytes(rows));
        return EPSR_ERR_CAPACITY;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const int R = rows;
    MlpWork w = carve(work, R);
    const bf16 *xr = (const bf16 *)x + (size_t)row0 * MLP_IN;
    float *loss = loss_out ? loss_out : w.loss;
    EPSR_CUDA(cudaMemsetAsync(loss, 0, sizeof(float), s));
    // forward, layer 1: z1 and h1 (row-major for layer 2, transposed for dW2)
    GemmArgs g1 = {};
    g1.epi = EPI_BIAS_SILU;
    g1.bias = net->b1;
    g1.z_out = w.z1;
    g1.h_out = w.h1;
    g1.ht_out = w.h1t;
    g1.ldt = R;
    g1.status = net->status;
    rc = gemm<32>({xr, MLP_IN, net->w1h, MLP_IN, R, MLP_H, MLP_IN, 1, g1}, s);
    if (rc) return rc;
    // forward, layer 2 + head + loss gradient: dz2 (row-major and transposed), dw3, db3, db2
    GemmArgs g2 = {};
    g2.epi = EPI_HEAD;
    g2.bias = net->b2;
    g2.w3 = net->w3;
    g2.b3 = net->b3;
    g2.y = w.y;
    g2.target = target + row0 / 2;
    g2.gscale = 1.0f / (float)(R / 2);
    g2.loss = loss;
    g2.dw3 = net->dw3;
    g2.db3 = net->db3;
    g2.db = net->db2;
    g2.dz_out = w.dz2;
    g2.dzt_out = w.dz2t;
    g2.ldt = R;
    g2.status = net->status;
    rc = gemm<128>({w.h1, MLP_H, net->w2h, MLP_H, R, MLP_H, MLP_H, 1, g2}, s);
    if (rc) return rc;
    // backward through layer 2: dh1 = dz2 . W2 (B = W2^T rows), dz1 = dh1 silu'(z1) transposed, db1
    GemmArgs g3 = {};
    g3.epi = EPI_SILU_BWD;
    g3.z_in = w.z1;
    g3.dzt_out = w.dz1t;
    g3.ldt = R;
    g3.db = net->db1;
    g3.status = net->status;
    rc = gemm<32>({w.dz2, MLP_H, net->w2th, MLP_H, R, MLP_H, MLP_H, 1, g3}, s);
    if (rc) return rc;
    // weight gradients over the R samples: dW1 = dz1^T x (x^T rows are features), dW2 = dz2^T h1
    const int ks = R / 128 < 8 ? R / 128 : 8;
    GemmArgs g4 = {};
    g4.epi = EPI_ATOMIC;
    g4.out = net->dw1;
    g4.ldo = MLP_IN;
    g4.status = net->status;
    GemmArgs g5 = {};
    g5.epi = EPI_ATOMIC;
    g5.out = net->dw2;
    g5.ldo = MLP_H;
    g5.status = net->status;
    // B = x^T restricted to the batch's columns: rows = features, K = samples from row0
    Product dw2 = {w.dz2t, R, w.h1t, R, MLP_H, MLP_H, R, ks, g5};
    rc = gemm<64>({w.dz1t, R, (const bf16 *)xt + row0, ldxt, MLP_H, MLP_IN, R, ks, g4}, s, &dw2);
    if (rc) return rc;
    // Adam (bias-corrected), then the BF16 copies the next forward reads
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f / (1.0f - powf(b1, (float)step)), c2 = 1.0f / (1.0f - powf(b2, (float)step));
    AdamArgs a = {{{net->w1, net->dw1, (bf16 *)net->w1h, nullptr, MLP_H * MLP_IN, MLP_H, MLP_IN},
                   {net->b1, net->db1, nullptr, nullptr, MLP_H, 1, MLP_H},
                   {net->w2, net->dw2, (bf16 *)net->w2h, (bf16 *)net->w2th, MLP_H * MLP_H, MLP_H, MLP_H},
                   {net->b2, net->db2, nullptr, nullptr, MLP_H, 1, MLP_H},
                   {net->w3, net->dw3, nullptr, nullptr, MLP_H, 1, MLP_H},
                   {net->b3, net->db3, nullptr, nullptr, 1, 1, 1}},
                  net->m1, net->v1, lr, b1, b2, 1e-8f, c1, c2, 0.0f};
    constexpr int nparam = MLP_H * MLP_IN + MLP_H * MLP_H + 3 * MLP_H + 1;
    adam_kernel<<<(nparam + 255) / 256, 256, 0, s>>>(a);
    EPSR_CUDA(cudaGetLastError());
    return EPSR_OK;
}
