// float32 products for more than a handful of tokens on the 5th-generation tensor cores: y[t, n] = sum_k x[t, k] w[n, k], float32 in and
// out.  Nothing of an operand is left out: its 24 digits are three bfloat16 numbers of eight, x = a + b + c (pico_split3).  Eight of the nine products
// of the parts are tcgen05.mma.kind::f16 (c c, below 2^-30 of x w, is left out), into three sums: a a; a b and b a, below 2^-6 of it; the other five,
// below 2^-12.  The tensor cores cut a sum off where float32 rounds it, so the first leaves them after 64 terms (a product a a has 16 digits:
// mostly nothing is cut off) and is added up in float32; the others stay to the end and are then added.  A sum of one term is its product
// to 2^-28 of it, rounded once, as a multiply-add's; a row of one 1 among noughts gives w bit for bit.
//
// What bounds it: the CUDA cores have 74 TFLOP/s for float32, and the library's product reaches 32 (340 x 2,048 x 1,536, K last: 65 us; here 32) and
// less for few rows; eight bfloat16 products have 200.  A tile is 128 rows of w (the instruction's M) x up to 128 tokens (its N), and K is cut
// into as many parts as fill the chip; the parts are added by a second kernel in a fixed order.  Per block: one warp copies (TMA, 128-byte
// swizzle, 32 k at a time, three stages of 32 KB), eight warps split what came into two stages of 48 KB (rows of 64 bytes in the 64-byte
// swizzle) and drain the accumulators, one thread multiplies.
//
// An infinity has no parts, so where a sum is no number it is computed again with float32 multiply-adds: infinities and NaN are what
// they would be there.
//
// Waits are bounded as in gemm_tcgen05_pair.cu (pico_tf_status).
#include "common.cuh"
#include <cuda.h>

#define TF_BM 128              // rows of w
#define TF_BN 128              // tokens at most
#define TF_BK 32               // k of a stage (128 bytes)
#define TF_STAGES 3            // copies
#define TF_RAW ((TF_BM + TF_BN) * TF_BK * 4)        // a copy: w, then x
#define TF_SPLITS 2            // stages of parts
#define TF_PART ((TF_BM + TF_BN) * TF_BK * 2)       // one part of a stage: w, then x
#define TF_WORKERS 8
#define TF_THREADS (64 + 32 * TF_WORKERS)
#define TF_GROUP 2             // stages whose products a a share a sum
#define TF_WAIT_LIMIT (1 << 16)

__device__ int g_tf_status = 0;        // 0 = fine; 1 = a wait ran out

PICO_API int pico_tf_status(int* out) { return (int)cudaMemcpyFromSymbol(out, g_tf_status, sizeof(int), 0, cudaMemcpyDeviceToHost); }

struct TfArgs {
    const float *x, *w;        // [M, K] (rows ldx apart), [N, K]
    float* out;                // [M, N], or [parts, 2, M, N]
    long long ldx;
    int M, N, K, parts, m_tile;        // m_tile: tokens of a tile, a multiple of 16
};

__device__ __forceinline__ uint32_t tf_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void tf_init(uint64_t* bar, int count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(tf_u32(bar)), "r"(count)); }
__device__ __forceinline__ void tf_arrive(uint64_t* bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(tf_u32(bar)) : "memory"); }
__device__ __forceinline__ bool tf_wait(uint64_t* bar, uint32_t parity, volatile int* abort) {
    for (int i = 0; i < TF_WAIT_LIMIT && !*abort; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n.reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok) : "r"(tf_u32(bar)), "r"(parity) : "memory");
        if (ok) return true;
    }
    g_tf_status = 1;
    *abort = 1;
    return false;
}
__device__ __forceinline__ void tf_load(void* dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n"
                 ::"r"(tf_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(tf_u32(bar)) : "memory");
}
// K-major rows of 64 bytes in the 64-byte swizzle (the chunk of 16 bytes at q lies at q ^ (row / 2 % 4)); sixteen k (32 bytes) an instruction
__device__ __forceinline__ uint64_t tf_desc(uint32_t tile, int k16) {
    return (uint64_t)(((tile + k16 * 32) >> 4) & 0x3fff) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}
__device__ __forceinline__ void tf_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t add) {
    const uint32_t zero = 0;
    asm volatile(
        "{\n.reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n}\n"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(add), "r"(zero) : "memory");
}
__device__ __forceinline__ void tf_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(tf_u32(bar)) : "memory");
}
// 16 columns of two sums, and the wait for them
__device__ __forceinline__ void tf_ld16(uint32_t first, uint32_t second, uint32_t (&r)[16], uint32_t (&s)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n"
        "tcgen05.wait::ld.sync.aligned;\n"
        : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7]), "=&r"(r[8]), "=&r"(r[9]),
          "=&r"(r[10]), "=&r"(r[11]), "=&r"(r[12]), "=&r"(r[13]), "=&r"(r[14]), "=&r"(r[15]), "=&r"(s[0]), "=&r"(s[1]), "=&r"(s[2]),
          "=&r"(s[3]), "=&r"(s[4]), "=&r"(s[5]), "=&r"(s[6]), "=&r"(s[7]), "=&r"(s[8]), "=&r"(s[9]), "=&r"(s[10]), "=&r"(s[11]),
          "=&r"(s[12]), "=&r"(s[13]), "=&r"(s[14]), "=&r"(s[15])
        : "r"(first), "r"(second) : "memory");
}
// y where it is a number, else what float32 multiply-adds give
__device__ __forceinline__ float tf_number(const TfArgs& p, float y, int t, int n) {
    if (y == y) return y;
    const float *a = p.x + (size_t)t * p.ldx, *b = p.w + (size_t)n * p.K;
    y = 0.f;
#pragma unroll 1
    for (int k = 0; k < p.K; ++k) y = fmaf(a[k], b[k], y);
    return y;
}

// Grid (tiles of w, tiles of tokens, parts of K)
__global__ void __launch_bounds__(TF_THREADS, 1)
gemm_f32_tcgen05_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map, const TfArgs p) {
    pdl_launch_dependents();
    extern __shared__ unsigned char tf_dyn[];
    unsigned char* smem = tf_dyn + ((1024u - (tf_u32(tf_dyn) & 1023u)) & 1023u);
    __shared__ uint64_t full[TF_STAGES], empty[TF_STAGES], split[TF_SPLITS], used[TF_SPLITS], sum_full[2], sum_empty[2], done;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * TF_BM, t0 = blockIdx.y * p.m_tile;
    const int nkb = (p.K + TF_BK - 1) / TF_BK, kb0 = (int)((long long)nkb * blockIdx.z / p.parts), nk = (int)((long long)nkb * (blockIdx.z + 1) / p.parts) - kb0;
    unsigned char* parts_s = smem + TF_STAGES * TF_RAW;
    if (threadIdx.x == 0) {
        for (int s = 0; s < TF_STAGES; ++s) {
            tf_init(full + s, 1);
            tf_init(empty + s, TF_WORKERS);
        }
        for (int s = 0; s < TF_SPLITS; ++s) {
            tf_init(split + s, TF_WORKERS);
            tf_init(used + s, 1);
        }
        for (int i = 0; i < 2; ++i) {
            tf_init(sum_full + i, 1);
            tf_init(sum_empty + i, TF_WORKERS);
        }
        tf_init(&done, 1);
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tf_u32(&tmem_slot)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = tmem_slot, tmem_mid = tmem + 2 * TF_BN, tmem_small = tmem + 3 * TF_BN;       // products a a (two sums in turn), a b and b a, the others
    pdl_wait();
    if (warp == 0) {
        if (lane == 0) {
            const uint32_t bytes = (TF_BM + p.m_tile) * TF_BK * 4;
            int kb = 0;
            for (; kb < nk; ++kb) {
                const int s = kb % TF_STAGES;
                if (kb >= TF_STAGES && !tf_wait(empty + s, ((kb / TF_STAGES) - 1) & 1, &abort_s)) break;
                unsigned char* dst = smem + s * TF_RAW;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(tf_u32(full + s)), "r"(bytes) : "memory");
                tf_load(dst, &w_map, (kb0 + kb) * TF_BK, n0, full + s);
                tf_load(dst + TF_BM * TF_BK * 4, &x_map, (kb0 + kb) * TF_BK, t0, full + s);
            }
            // the last copies land before the block leaves, also where an error comes after the last of them was asked for
            for (int i = kb > TF_STAGES ? kb - TF_STAGES : 0; i < kb; ++i) {
                volatile int never = 0;
                tf_wait(full + i % TF_STAGES, (i / TF_STAGES) & 1, &never);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // float32 sums, bfloat16 operands, both K-major, N = m_tile, M = 128
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.m_tile >> 3) << 17) | ((uint32_t)(TF_BM >> 4) << 24);
            for (int kb = 0; kb < nk; ++kb) {
                const int s = kb % TF_SPLITS, group = kb / TF_GROUP, buf = group & 1, within = kb % TF_GROUP;
                if (within == 0 && group >= 2 && !tf_wait(sum_empty + buf, ((group >> 1) - 1) & 1, &abort_s)) break;
                if (!tf_wait(split + s, (kb / TF_SPLITS) & 1, &abort_s)) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t w = tf_u32(parts_s + s * 3 * TF_PART), x = w + TF_BM * TF_BK * 2;
#pragma unroll
                for (int k16 = 0; k16 < TF_BK / 16; ++k16) {
                    uint64_t wd[3], xd[3];
#pragma unroll
                    for (int i = 0; i < 3; ++i) {
                        wd[i] = tf_desc(w + i * TF_PART, k16);
                        xd[i] = tf_desc(x + i * TF_PART, k16);
                    }
                    const uint32_t add = (kb | k16) ? 1u : 0u;
                    tf_mma(tmem + buf * TF_BN, wd[0], xd[0], idesc, (within | k16) ? 1u : 0u);
                    tf_mma(tmem_mid, wd[0], xd[1], idesc, add);
                    tf_mma(tmem_small, wd[1], xd[2], idesc, add);
                    tf_mma(tmem_small, wd[2], xd[1], idesc, 1u);
                    tf_mma(tmem_small, wd[0], xd[2], idesc, 1u);
                    tf_mma(tmem_small, wd[2], xd[0], idesc, 1u);
                    tf_mma(tmem_mid, wd[1], xd[0], idesc, 1u);
                    tf_mma(tmem_small, wd[1], xd[1], idesc, 1u);
                }
                tf_commit(used + s);
                if (within == TF_GROUP - 1 || kb == nk - 1) tf_commit(sum_full + buf);
            }
            // products that nobody waits for any more, after an error, end before the tensor memory is given back
            volatile int never = 0;
            tf_commit(&done);
            tf_wait(&done, 0, &never);
        }
    } else {
        // a worker drains tensor-memory lanes 32 (warp % 4) .. (rows of w) at half of the tokens
        const int worker = warp - 2, half = worker >> 2;
        const uint32_t lanes = (uint32_t)(warp & 3) << 21;
        const bool any = half * 64 < p.m_tile;
        float sum[64];                         // of the products a a
#pragma unroll
        for (int i = 0; i < 64; ++i) sum[i] = 0.f;
        const int groups = (nk + TF_GROUP - 1) / TF_GROUP, rows8 = (TF_BM + p.m_tile) / 8;
        int drained = 0;
        bool ok = true;
        auto drain = [&]() {
            ok = tf_wait(sum_full + (drained & 1), (drained >> 1) & 1, &abort_s);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) return;
            const uint32_t col = tmem + (drained & 1) * TF_BN + lanes + half * 64;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
            for (int c = 0; c < 64; c += 32) {
                if (any) {
                    uint32_t r[16], s[16];
                    tf_ld16(col + c, col + c + 16, r, s);
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        sum[c + i] += __uint_as_float(r[i]);
                        sum[c + 16 + i] += __uint_as_float(s[i]);
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            if (lane == 0) tf_arrive(sum_empty + (drained & 1));
            ++drained;
        };
        // a lane splits eight k of a row: eight rows side by side, which keeps every bank busy once in both swizzles
        const int r8 = lane & 7, q = lane >> 3;
        const uint32_t from0 = r8 * 128 + ((2 * q) ^ r8) * 16, from1 = r8 * 128 + ((2 * q + 1) ^ r8) * 16, to = r8 * 64 + (q ^ (r8 >> 1)) * 16;
        for (int kb = 0; ok && kb < nk; ++kb) {
            const int s = kb % TF_STAGES, sp = kb % TF_SPLITS;
            ok = tf_wait(full + s, (kb / TF_STAGES) & 1, &abort_s) && (kb < TF_SPLITS || tf_wait(used + sp, ((kb / TF_SPLITS) - 1) & 1, &abort_s));
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const unsigned char* from = smem + s * TF_RAW;
            unsigned char* at = parts_s + sp * 3 * TF_PART + to;
#pragma unroll 4
            for (int i = worker; i < rows8; i += TF_WORKERS) {
                const float4 u = *reinterpret_cast<const float4*>(from + i * 1024 + from0), v = *reinterpret_cast<const float4*>(from + i * 1024 + from1);
                uint4 a, b, c;
                pico_split3(u.x, u.y, a.x, b.x, c.x);
                pico_split3(u.z, u.w, a.y, b.y, c.y);
                pico_split3(v.x, v.y, a.z, b.z, c.z);
                pico_split3(v.z, v.w, a.w, b.w, c.w);
                *reinterpret_cast<uint4*>(at + i * 512) = a;
                *reinterpret_cast<uint4*>(at + i * 512 + TF_PART) = b;
                *reinterpret_cast<uint4*>(at + i * 512 + 2 * TF_PART) = c;
            }
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                tf_arrive(empty + s);
                tf_arrive(split + sp);
            }
            // the sums of the group before the last one are long done
            if (kb % TF_GROUP == TF_GROUP - 1 && kb / TF_GROUP > drained) drain();
        }
        while (ok && drained < groups) drain();
        if (ok && any) {
            const int n = n0 + (warp & 3) * 32 + lane;
            const size_t all = (size_t)p.M * p.N;
            float* out = p.out + 2 * blockIdx.z * all + n;             // a part leaves both sums, [2, M, N]
#pragma unroll
            for (int c = 0; c < 64; c += 16) {
                uint32_t r[16], s[16];
                tf_ld16(tmem_mid + lanes + half * 64 + c, tmem_small + lanes + half * 64 + c, r, s);       // (complete with the last group's)
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const int m = half * 64 + c + i, t = t0 + m;
                    const float rest = __uint_as_float(r[i]) + __uint_as_float(s[i]);
                    if (n < p.N && m < p.m_tile && t < p.M) {
                        if (p.parts > 1) {
                            out[(size_t)t * p.N] = sum[c + i];
                            out[all + (size_t)t * p.N] = rest;
                        } else {
                            out[(size_t)t * p.N] = tf_number(p, sum[c + i] + rest, t, n);
                        }
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512));
    }
}

// out = the sum of the parts, one after the other, the products a a apart from the others to the end
__global__ void __launch_bounds__(256)
gemm_f32_sum_kernel(const float* __restrict__ parts, float* __restrict__ out, const TfArgs p) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t all = (size_t)p.M * p.N, i = ((size_t)blockIdx.x * 256 + threadIdx.x) * 4;
    if (i >= all) return;
    float4 v = *reinterpret_cast<const float4*>(parts + i), r = *reinterpret_cast<const float4*>(parts + all + i);
#pragma unroll 4
    for (int z = 1; z < p.parts; ++z) {
        const float4 a = *reinterpret_cast<const float4*>(parts + 2 * z * all + i), b = *reinterpret_cast<const float4*>(parts + (2 * z + 1) * all + i);
        v.x += a.x;
        v.y += a.y;
        v.z += a.z;
        v.w += a.w;
        r.x += b.x;
        r.y += b.y;
        r.z += b.z;
        r.w += b.w;
    }
    const int t = (int)(i / p.N), n = (int)(i % p.N);          // N is a multiple of four
    v.x = tf_number(p, v.x + r.x, t, n);
    v.y = tf_number(p, v.y + r.y, t, n + 1);
    v.z = tf_number(p, v.z + r.z, t, n + 2);
    v.w = tf_number(p, v.w + r.w, t, n + 3);
    *reinterpret_cast<float4*>(out + i) = v;
}

typedef CUresult (*TfEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                               const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static TfEncodeFn tf_encode_fn() {
    static TfEncodeFn fn = []() -> TfEncodeFn {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult st;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &st) == cudaSuccess && st == cudaDriverEntryPointSuccess)
            return (TfEncodeFn)f;
        return nullptr;
    }();
    return fn;
}
static int tf_map(CUtensorMap* map, const void* base, long long rows, int K, long long ld, int box_rows) {
    TfEncodeFn fn = tf_encode_fn();
    if (!fn) return -7;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
    const cuuint32_t box[2] = {TF_BK, (cuuint32_t)box_rows}, one[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -7;
}

// How many parts K is cut into for these sizes: as many as fill the multiprocessors once, each of four stages at least.
PICO_API int pico_gemm_f32_parts(int M, int N, int K) {
    const int nkb = (K + TF_BK - 1) / TF_BK;
    const long long tiles = (long long)((N + TF_BM - 1) / TF_BM) * ((M + TF_BN - 1) / TF_BN);
    long long parts = pico_num_sms() / (tiles > 0 ? tiles : 1);
    if (parts > nkb / 4) parts = nkb / 4;
    return parts < 1 ? 1 : (int)parts;
}

// out [M, N] = x w^T; x [M, K] with rows ldx apart, w [N, K]; K, N, ldx multiples of 4, addresses of 16 bytes.  scratch: 2 * parts * M * N floats
// where pico_gemm_f32_parts gives more than one.
PICO_API int pico_gemm_f32(const float* x, long long ldx, const float* w, float* out, float* scratch, int M, int N, int K, cudaStream_t stream) {
    if (M < 1 || N < 4 || K < 4 || K % 4 || N % 4 || ldx % 4 || (((uintptr_t)x | (uintptr_t)w | (uintptr_t)out | (uintptr_t)scratch) & 15)) return PICO_ERR_SIZE;
    const int m_tiles = (M + TF_BN - 1) / TF_BN;
    if (m_tiles > 65535) return PICO_ERR_SIZE;
    TfArgs a = {};
    a.x = x; a.w = w; a.ldx = ldx; a.M = M; a.N = N; a.K = K;
    a.parts = pico_gemm_f32_parts(M, N, K);
    a.m_tile = ((M + m_tiles - 1) / m_tiles + 15) / 16 * 16;
    a.out = a.parts > 1 ? scratch : out;
    if (!a.out) return PICO_ERR_SIZE;
    CUtensorMap xm, wm;
    int rc = tf_map(&xm, x, M, K, ldx, a.m_tile);
    if (rc) return rc;
    rc = tf_map(&wm, w, N, K, K, TF_BM);
    if (rc) return rc;
    const size_t smem = (size_t)TF_STAGES * TF_RAW + (size_t)TF_SPLITS * 3 * TF_PART + 1024;
    cudaFuncSetAttribute(gemm_f32_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    pico_launch(gemm_f32_tcgen05_kernel, dim3((N + TF_BM - 1) / TF_BM, (M + a.m_tile - 1) / a.m_tile, a.parts), dim3(TF_THREADS), smem, stream, xm, wm, a);
    if (a.parts > 1) pico_launch(gemm_f32_sum_kernel, dim3((unsigned)(((size_t)M * N / 4 + 255) / 256)), dim3(256), 0, stream, (const float*)scratch, out, a);
    return pico_launch_status();
}
