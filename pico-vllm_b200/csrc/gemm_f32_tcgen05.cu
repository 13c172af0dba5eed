// float32 products for more than a handful of tokens on the 5th-generation tensor cores: y[t, n] = sum_k x[t, k] w[n, k], float32 in and
// out, no less exact than float32 multiply-adds.  Each operand is two numbers of tf32's eleven digits, x = h + l (l is what h leaves, to
// below half a unit of float32's last place), and h h + l h + h l are three tcgen05.mma.kind::tf32 (l l is below that unit, too).  The
// tensor cores cut a sum off where float32 rounds it, so the large products' sums leave them after 64 terms and are added in float32; the
// small ones' sums, 2^-12 of those, stay to the end.
//
// What bounds it: the CUDA cores have 74 TFLOP/s for float32, and the library's product reaches 32 (340 x 2,048 x 1,536, K last: 68 us) and
// less for few rows; three tf32 products have 366.  A tile is 128 rows of w (the instruction's M) x up to 128 tokens (its N), and K is cut
// into as many parts as fill the chip; the parts are added by a second kernel in a fixed order.  Per block: one warp copies (TMA, 128-byte
// swizzle, 32 k at a time), eight warps split what came - h in place of the copy, l beside it - and drain the accumulators, one thread
// multiplies.  Stages of 64 KB, three of them: one is copied, one split, one multiplied.
//
// An infinity has no two parts (nor have numbers above 2^114, whose splitting overflows), so where a sum is no number it is computed again
// with float32 multiply-adds: infinities and NaN are what they would be there.
//
// Waits are bounded as in gemm_tcgen05_pair.cu (pico_tf_status).
#include "common.cuh"
#include <cuda.h>

#define TF_BM 128              // rows of w
#define TF_BN 128              // tokens at most
#define TF_BK 32               // k of a stage (128 bytes)
#define TF_STAGES 3
#define TF_HALF ((TF_BM + TF_BN) * TF_BK * 4)       // the copies of a stage: w, then x; behind them their small parts
#define TF_WORKERS 8
#define TF_THREADS (64 + 32 * TF_WORKERS)
#define TF_GROUP 2             // stages whose large products share a sum
#define TF_WAIT_LIMIT (1 << 16)

__device__ int g_tf_status = 0;        // 0 = fine; 1 = a wait ran out

PICO_API int pico_tf_status(int* out) { return (int)cudaMemcpyFromSymbol(out, g_tf_status, sizeof(int), 0, cudaMemcpyDeviceToHost); }

struct TfArgs {
    const float *x, *w;        // [M, K] (rows ldx apart), [N, K]
    float* out;                // [M, N], or [parts, M, N]
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
// K-major rows of 128 bytes in the 128-byte swizzle; eight k (32 bytes) an instruction
__device__ __forceinline__ uint64_t tf_desc(uint32_t tile, int k8) {
    return (uint64_t)(((tile + k8 * 32) >> 4) & 0x3fff) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
__device__ __forceinline__ void tf_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t add) {
    const uint32_t zero = 0;
    asm volatile(
        "{\n.reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n}\n"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(add), "r"(zero) : "memory");
}
__device__ __forceinline__ void tf_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(tf_u32(bar)) : "memory");
}
__device__ __forceinline__ void tf_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}
// Dekker's splitting, each operation rounded by itself: h has eleven digits of x, and x - h is exact
__device__ __forceinline__ void tf_split(float x, float& h, float& l) {
    const float c = __fmul_rn(8193.f, x);
    h = __fsub_rn(c, __fsub_rn(c, x));
    l = __fsub_rn(x, h);
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
    __shared__ uint64_t full[TF_STAGES], split[TF_STAGES], empty[TF_STAGES], sum_full[2], sum_empty[2], done;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * TF_BM, t0 = blockIdx.y * p.m_tile;
    const int nkb = (p.K + TF_BK - 1) / TF_BK, kb0 = (int)((long long)nkb * blockIdx.z / p.parts), nk = (int)((long long)nkb * (blockIdx.z + 1) / p.parts) - kb0;
    if (threadIdx.x == 0) {
        for (int s = 0; s < TF_STAGES; ++s) {
            tf_init(full + s, 1);
            tf_init(split + s, TF_WORKERS);
            tf_init(empty + s, 1);
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
    const uint32_t tmem = tmem_slot, tmem_small = tmem + 2 * TF_BN;      // two sums of large products, one of small ones
    pdl_wait();
    if (warp == 0) {
        if (lane == 0) {
            const uint32_t bytes = (TF_BM + p.m_tile) * TF_BK * 4;
            int kb = 0;
            for (; kb < nk; ++kb) {
                const int s = kb % TF_STAGES;
                if (kb >= TF_STAGES && !tf_wait(empty + s, ((kb / TF_STAGES) - 1) & 1, &abort_s)) break;
                unsigned char* dst = smem + s * 2 * TF_HALF;
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
            // float32 sums, tf32 operands, both K-major, N = m_tile, M = 128
            const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(p.m_tile >> 3) << 17) | ((uint32_t)(TF_BM >> 4) << 24);
            for (int kb = 0; kb < nk; ++kb) {
                const int s = kb % TF_STAGES, group = kb / TF_GROUP, buf = group & 1, within = kb % TF_GROUP;
                if (within == 0 && group >= 2 && !tf_wait(sum_empty + buf, ((group >> 1) - 1) & 1, &abort_s)) break;
                if (!tf_wait(split + s, (kb / TF_STAGES) & 1, &abort_s)) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t wh = tf_u32(smem + s * 2 * TF_HALF), xh = wh + TF_BM * TF_BK * 4, wl = wh + TF_HALF, xl = xh + TF_HALF;
#pragma unroll
                for (int k8 = 0; k8 < TF_BK / 8; ++k8) {
                    tf_mma(tmem + buf * TF_BN, tf_desc(wh, k8), tf_desc(xh, k8), idesc, (within | k8) ? 1u : 0u);
                    tf_mma(tmem_small, tf_desc(wl, k8), tf_desc(xh, k8), idesc, (kb | k8) ? 1u : 0u);
                    tf_mma(tmem_small, tf_desc(wh, k8), tf_desc(xl, k8), idesc, 1u);
                }
                tf_commit(empty + s);
                if (within == TF_GROUP - 1 || kb == nk - 1) tf_commit(sum_full + buf);
            }
            // products that nobody waits for any more, after an error, end before the tensor memory is given back
            volatile int never = 0;
            tf_commit(&done);
            tf_wait(&done, 0, &never);
        }
    } else {
        // a worker drains tensor-memory lanes 32 (warp % 4) .. (rows of w) at half of the tokens
        const int worker = warp - 2, tid = worker * 32 + lane, half = worker >> 2;
        const uint32_t lanes = (uint32_t)(warp & 3) << 21;
        const bool any = half * 64 < p.m_tile;
        float sum[64];
#pragma unroll
        for (int i = 0; i < 64; ++i) sum[i] = 0.f;
        auto add = [&](uint32_t col) {
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                if (any) {
                    uint32_t r[32];
                    tf_ld32(col + lanes + half * 64 + c * 32, r);
#pragma unroll
                    for (int i = 0; i < 32; ++i) sum[c * 32 + i] += __uint_as_float(r[i]);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        };
        const int groups = (nk + TF_GROUP - 1) / TF_GROUP, pieces = (TF_BM + p.m_tile) * (TF_BK / 4);
        int drained = 0;
        bool ok = true;
        auto drain = [&]() {
            ok = tf_wait(sum_full + (drained & 1), (drained >> 1) & 1, &abort_s);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) return;
            add(tmem + (drained & 1) * TF_BN);
            if (lane == 0) tf_arrive(sum_empty + (drained & 1));
            ++drained;
        };
        for (int kb = 0; ok && kb < nk; ++kb) {
            const int s = kb % TF_STAGES;
            ok = tf_wait(full + s, (kb / TF_STAGES) & 1, &abort_s);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            unsigned char* at = smem + s * 2 * TF_HALF;
#pragma unroll 4
            for (int i = tid; i < pieces; i += 32 * TF_WORKERS) {
                float4* src = reinterpret_cast<float4*>(at) + i;
                const float4 v = *src;
                float4 h, l;
                tf_split(v.x, h.x, l.x);
                tf_split(v.y, h.y, l.y);
                tf_split(v.z, h.z, l.z);
                tf_split(v.w, h.w, l.w);
                *src = h;
                *reinterpret_cast<float4*>(at + TF_HALF + i * 16) = l;
            }
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) tf_arrive(split + s);
            // the sums of the group before the last one are long done
            if (kb % TF_GROUP == TF_GROUP - 1 && kb / TF_GROUP > drained) drain();
        }
        while (ok && drained < groups) drain();
        if (ok) {
            add(tmem_small);                   // (complete with the last group's)
            const int n = n0 + (warp & 3) * 32 + lane;
            if (n < p.N) {
                float* out = p.out + (size_t)blockIdx.z * p.M * p.N + n;
#pragma unroll
                for (int i = 0; i < 64; ++i) {
                    const int m = half * 64 + i, t = t0 + m;
                    if (m < p.m_tile && t < p.M) out[(size_t)t * p.N] = p.parts > 1 ? sum[i] : tf_number(p, sum[i], t, n);
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

// out = the sum of the parts, one after the other
__global__ void __launch_bounds__(256)
gemm_f32_sum_kernel(const float* __restrict__ parts, float* __restrict__ out, const TfArgs p) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t all = (size_t)p.M * p.N, i = ((size_t)blockIdx.x * 256 + threadIdx.x) * 4;
    if (i >= all) return;
    float4 v = *reinterpret_cast<const float4*>(parts + i);
#pragma unroll 8
    for (int z = 1; z < p.parts; ++z) {
        const float4 a = *reinterpret_cast<const float4*>(parts + z * all + i);
        v.x += a.x;
        v.y += a.y;
        v.z += a.z;
        v.w += a.w;
    }
    const int t = (int)(i / p.N), n = (int)(i % p.N);          // N is a multiple of four
    v.x = tf_number(p, v.x, t, n);
    v.y = tf_number(p, v.y, t, n + 1);
    v.z = tf_number(p, v.z, t, n + 2);
    v.w = tf_number(p, v.w, t, n + 3);
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

// out [M, N] = x w^T; x [M, K] with rows ldx apart, w [N, K]; K, N, ldx multiples of 4, addresses of 16 bytes.  scratch: parts * M * N floats
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
    const size_t smem = (size_t)TF_STAGES * 2 * TF_HALF + 1024;
    cudaFuncSetAttribute(gemm_f32_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    pico_launch(gemm_f32_tcgen05_kernel, dim3((N + TF_BM - 1) / TF_BM, (M + a.m_tile - 1) / a.m_tile, a.parts), dim3(TF_THREADS), smem, stream, xm, wm, a);
    if (a.parts > 1) pico_launch(gemm_f32_sum_kernel, dim3((unsigned)(((size_t)M * N / 4 + 255) / 256)), dim3(256), 0, stream, (const float*)scratch, out, a);
    return pico_launch_status();
}
