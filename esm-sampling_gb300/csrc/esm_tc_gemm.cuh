// BF16 GEMM on the 5th-generation tensor cores (tcgen05) for the surrogate MLP: C[M,N] (+)=
// A[M,K] B[N,K]^T with A and B K-major in BF16, the FP32 accumulator in tensor memory (TMEM).
//
// One CTA of 4 warps per 128 x 64 tile of C. Operands are staged through shared memory in the
// canonical no-swizzle K-major layout of tcgen05 (core matrices of 8 rows x 16 bytes; along K the
// core matrices of a row group are 128 bytes apart (the leading-dimension offset), row groups 1024
// bytes apart (the stride-dimension offset)) by 16-byte asynchronous copies, TC_STAGES deep: three tiles
// are on their way while the tensor core multiplies one. (With one tile ahead, through registers, every
// 64 columns of K waited for memory: 1024 x 1024 x 1024 took 75 us.) Rows are padded to 8 elements, so
// every copy is aligned, and the pads are zero. One elected thread issues tcgen05.mma (M = 128, N = 64,
// K = 16, kind::f16, BF16 x BF16 -> FP32) and commits each stage to an mbarrier that releases the
// stage's shared memory. The epilogue reads the accumulator with tcgen05.ld (32 lanes x 32 bits, each
// warp its 32 rows), adds the bias, applies SiLU and writes FP32 and BF16 outputs, 16 bytes at a time
// where the rows allow. Every mbarrier wait is bounded: on time-out the kernel sets *err, frees its
// tensor memory and returns.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace tc {

#define TC_BM 128
#define TC_BN 64
#define TC_BK 64
#define TC_STAGE_A (TC_BM * TC_BK * 2)  // bytes of one A stage
#define TC_STAGE_B (TC_BN * TC_BK * 2)
#define TC_STAGES 4
#define TC_SMEM (TC_STAGES * (TC_STAGE_A + TC_STAGE_B) + 1024)
#define TC_WAIT_LIMIT (1 << 24)

struct GemmTC {
    int M, N, K;
    const __nv_bfloat16 *A;  // A(m, k) at A[m*lda + k]; 16-byte aligned, lda a multiple of 8, zeros from K to
    int lda;                 // the next multiple of 8
    const __nv_bfloat16 *B;  // B(n, k) at B[n*ldb + k], likewise
    int ldb;
    float *C;  // C(m, n) at C[m*ldc + n] (may be null)
    int ldc;
    int accumulate;
    const float *bias;  // per n (may be null)
    int silu;
    __nv_bfloat16 *Cb;  // BF16 copy of the (activated) output (may be null)
    int ldcb;
    int *err;  // set to 1 when a wait ran out
};

__device__ inline uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor: start address, leading- and stride-dimension byte offsets (all
// in units of 16 bytes), the descriptor version 1 of this architecture, no swizzle
__device__ inline uint64_t sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
    d |= (uint64_t)((lbo & 0x3FFFF) >> 4) << 16;
    d |= (uint64_t)((sbo & 0x3FFFF) >> 4) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both K-major, M x N
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ inline bool mbar_wait(uint32_t bar, uint32_t parity) {
    for (int it = 0; it < TC_WAIT_LIMIT; ++it) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// the 16-byte chunk c of a 128-row x 64-column (or 64-row) K-major tile: row and K chunk, and its
// offset in the canonical layout
__device__ inline uint32_t tile_off(int row, int kc) { return (uint32_t)((row >> 3) * 1024 + kc * 128 + (row & 7) * 16); }

// 16 bytes from global to shared memory, zeros when not `valid`
__device__ inline void copy_chunk(uint32_t dst, const void *src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

__global__ void __launch_bounds__(128, 1) k_gemm_tc(GemmTC g) {
    extern __shared__ uint8_t smraw[];
    __shared__ __align__(8) uint64_t mbar[TC_STAGES];
    __shared__ uint32_t tmem_s;
    __shared__ int bad_s;
    uint8_t *sm = (uint8_t *)(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);
    const uint32_t sA = smem_u32(sm), sB = sA + TC_STAGES * TC_STAGE_A;
    int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int m0 = blockIdx.y * TC_BM, n0 = blockIdx.x * TC_BN;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)),
                     "r"(TC_BN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        bad_s = 0;
        for (int s = 0; s < TC_STAGES; ++s)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar[s])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    uint32_t tmem = tmem_s;
    const uint32_t idesc = idesc_bf16(TC_BM, TC_BN);
    int nk = (g.K + TC_BK - 1) / TC_BK;
    auto load = [&](int t) {  // tile t into its stage: A 1024 chunks, B 512 chunks over 128 threads
        const int s = t % TC_STAGES, k0 = t * TC_BK;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            int c = tid + i * 128, r = m0 + (c >> 3), k = k0 + (c & 7) * 8;
            bool v = r < g.M && k < g.K;
            copy_chunk(sA + s * TC_STAGE_A + tile_off(c >> 3, c & 7), v ? g.A + (size_t)r * g.lda + k : g.A, v);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int c = tid + i * 128, r = n0 + (c >> 3), k = k0 + (c & 7) * 8;
            bool v = r < g.N && k < g.K;
            copy_chunk(sB + s * TC_STAGE_B + tile_off(c >> 3, c & 7), v ? g.B + (size_t)r * g.ldb + k : g.B, v);
        }
    };
    bool ok = true;
    // (a group is committed for every tile of the loop, empty ones too, so that the count stands for tiles)
    for (int t = 0; t < TC_STAGES - 1; ++t) {
        if (t < nk) load(t);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int t = 0; t < nk; ++t) {
        const int s = t % TC_STAGES;
        asm volatile("cp.async.wait_group %0;" ::"n"(TC_STAGES - 2) : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (__syncthreads_or(!ok)) {
            ok = false;
            break;
        }
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int kk = 0; kk < TC_BK / 16; ++kk) {
                uint64_t ad = sdesc(sA + s * TC_STAGE_A + kk * 256, 128, 1024);
                uint64_t bd = sdesc(sB + s * TC_STAGE_B + kk * 256, 128, 1024);
                uint32_t acc = (t > 0 || kk > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(
                        tmem),
                    "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_u32(&mbar[s]))
                         : "memory");
        }
        // the stage of tile t - 1 takes tile t + TC_STAGES - 1 once its multiplications have read it
        const int nt = t + TC_STAGES - 1;
        if (t >= 1 && !mbar_wait(smem_u32(&mbar[(t - 1) % TC_STAGES]), (uint32_t)(((t - 1) / TC_STAGES) & 1))) ok = false;
        if (ok && nt < nk) load(nt);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    // the last tile's multiplications complete the accumulator (every wait of a stage before it was made)
    if (ok && nk > 0 && !mbar_wait(smem_u32(&mbar[(nk - 1) % TC_STAGES]), (uint32_t)(((nk - 1) / TC_STAGES) & 1))) ok = false;
    if (!ok) bad_s = 1;
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (!bad_s && nk > 0) {
        int row = m0 + warp * 32 + lane;
        for (int cc = 0; cc < TC_BN; cc += 16) {
            uint32_t r[16];
            uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)cc;
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                "%14, %15}, [%16];"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                  "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                : "r"(taddr));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (row >= g.M) continue;
            const int n1 = n0 + cc;
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                v[j] = __uint_as_float(r[j]);
                if (g.bias && n1 + j < g.N) v[j] += g.bias[n1 + j];
            }
            if (g.C) {
                float *cp = g.C + (size_t)row * g.ldc + n1;
                if (n1 + 16 <= g.N && (g.ldc & 3) == 0 && !g.accumulate) {
#pragma unroll
                    for (int j = 0; j < 16; j += 4) *(float4 *)(cp + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (n1 + j < g.N) cp[j] = g.accumulate ? cp[j] + v[j] : v[j];
                }
            }
            if (g.Cb) {
                __align__(16) __nv_bfloat16 o[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) o[j] = __float2bfloat16(g.silu ? v[j] / (1.f + expf(-v[j])) : v[j]);
                __nv_bfloat16 *bp = g.Cb + (size_t)row * g.ldcb + n1;
                if (n1 + 16 <= g.N && (g.ldcb & 7) == 0) {
                    *(uint4 *)bp = *(const uint4 *)o;
                    *(uint4 *)(bp + 8) = *(const uint4 *)(o + 8);
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (n1 + j < g.N) bp[j] = o[j];
                }
            }
        }
    }
    if (bad_s && tid == 0 && g.err) atomicExch(g.err, 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TC_BN) : "memory");
}

// B[n, k] (K-major) from a row-major [k, n] BF16 matrix: out[n*ldo + k] = in[k*ldi + n], and zeros in out
// from `rows` up to the next multiple of 8
__global__ void k_transpose_bf16(int rows, int cols, const __nv_bfloat16 *in, int ldi, __nv_bfloat16 *out, int ldo) {
    __shared__ __nv_bfloat16 tile[32][33];
    int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        int r = r0 + i, c = c0 + threadIdx.x;
        tile[i][threadIdx.x] = (r < rows && c < cols) ? in[(size_t)r * ldi + c] : __float2bfloat16(0.f);
    }
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        int c = c0 + i, r = r0 + threadIdx.x;
        if (c < cols && r < ((rows + 7) & ~7)) out[(size_t)c * ldo + r] = tile[threadIdx.x][i];
    }
}

}  // namespace tc
