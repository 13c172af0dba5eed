// Paged causal attention with grouped heads, for any head size that is a multiple of 16 up to
// 640, float32 or bfloat16 storage, float32 arithmetic with a running max and sum.  A block takes the rows of a run of tokens
// for one key/value head and one split of the key range (see paged_attention_tiled_kernel) and either writes the output
// or, with more than one split, a partial (max, sum, unnormalised output) that a second kernel combines.  This is the
// kernel of the 32-bit path and the fallback of the bfloat16 path.
//
// Restated from the reference: query head j uses key/value head j / g
// (pico_vllm/kernels/attention.py:31,139); scores scaled by hd^-1/2 (attention.py:92,231);
// key n is visible to the query at position p iff n <= p (attention.py:193-198); running
// max/sum softmax in float32 (attention.py:67-82, 189-213); pages found through the block table
// (attention.py:47-52, 172-176).  The window rule (only the last W keys) is the meaning of the
// architecture's sliding_window key; the reference has none.  Unlike the reference's prefill
// kernel, p is not rounded to the cache type before p.v, and a key beyond a query never enters its row.
#include "common.cuh"
#include <type_traits>

#define ATT_MAX_HD 640         // widest head
#define ATT_WHOLE (-1.0f)      // as a part's denominator: the row is finished
#define ATT_NOALLOC_MAX_HD 256 // ... that the entry point without allocation takes

// One key/value head's tile: what a block works on.  A tile is up to RT rows, a row being (token, query head of the
// group); its tokens are a run of neighbours in the batch that belong to one request at consecutive positions, so every
// key between the first row's first and the last row's last is seen by some row of the run.  The block of the run's first
// token (inside an aligned group of `bq` tokens) does the run, the blocks of the others leave at once: the kernel needs no
// list of the segments, and single tokens of a mixed batch get blocks of their own.
//   RT = 32: four warps of 8 rows each share the tiles of KT keys (long prompts: a key is read once for 32 rows);
//   RT =  8: four warps share the 8 rows and take every fourth tile of keys, their sums are added at the end (single
//            tokens and short prompts, where blocks are few and a row's chain of keys sets the time).
// With part_keys > 0 every run, a portion's too, goes in parts of at least so many keys, up to n_splits; a run that stays whole is written by
// its own block and left alone by the combining kernel.
// Keys and values come in by cp.async into buffers of their own (values land while the scores are computed, the next keys
// while the values are multiplied); scores: a lane has 2 rows x KT / 8 keys; output: a lane has 8 rows x 4 NJ dimensions,
// probabilities pass through shared memory.  All arithmetic is float32 on the CUDA cores: with enough rows those bound it
// (6 shared-memory wavefronts stand against 16 packed multiply-adds a lane in both products); with few, the latency of a
// warp's chain of instructions (one warp a scheduler, about 5 clocks an instruction).
// Measured (float32, 12 query on 2 key/value heads of 128, pages of 16; the form before: a block a token, a key a lane):
// 333 tokens from the start beside 7 single ones at 500: 58 us (524); 700 tokens: 148 (975); 2,048: 571 (6,156, now
// 23 TFLOP/s); 8 single tokens at 777 keys in one part: 72 (652), in 8 parts: 25 (113).
template <typename T> __device__ __forceinline__ void tile_load16(float* dst, const T* src);
template <> __device__ __forceinline__ void tile_load16<float>(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src));
}
template <> __device__ __forceinline__ void tile_load16<bf16>(float* dst, const bf16* src) {
    const uint4 raw = *reinterpret_cast<const uint4*>(src);
    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw);
    const float2 a = __bfloat1622float2(p[0]), b = __bfloat1622float2(p[1]), c = __bfloat1622float2(p[2]), d = __bfloat1622float2(p[3]);
    reinterpret_cast<float4*>(dst)[0] = make_float4(a.x, a.y, b.x, b.y);
    reinterpret_cast<float4*>(dst)[1] = make_float4(c.x, c.y, d.x, d.y);
}

// two float32 fused multiply-adds in one instruction (each rounded as fmaf rounds)
__device__ __forceinline__ void fma2(float2& d, float2 a, float2 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;\n"
        : "+l"(reinterpret_cast<unsigned long long&>(d))
        : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)));
}

// What the sums of a part (its maximum m and denominator l) are multiplied with when parts are put together under the maximum M.
// A part without keys has m = -inf and l = 0 and counts for nothing; with scores that are all no numbers m is -inf too (a
// maximum passes them over), but l is none, and so is the row that the part belongs to.
__device__ __forceinline__ float part_factor(float m, float l, float M) { return m == -INFINITY ? l : expf(m - M); }

struct TileArgs {
    int q_row_stride, table_stride, T, nh, nkv, hd, page_size, window, n_splits, chunk, bq, row_chunks, part_keys;
    float scale, softcap;
    const int *tok_seg, *positions, *block_table;
    const float *slopes, *sinks, *rates;
    float *part_o, *part_ml;
};

__host__ __device__ constexpr int tile_keys(int nj, int rt) { return rt == 8 ? (nj == 5 ? 8 : 16) : (nj == 1 ? 32 : nj == 2 ? 16 : 8); }

// Whether the parts of a run are neighbours in the grid, at work and in L2 together, or all first parts come before the second ones: single
// tokens in parts lose by the former (64 of 12 / 2 heads of 96, 777 keys in two parts 84.7 us, side by side 86.7; of 128, 300 keys 28.6 / 29.5).
__host__ __device__ constexpr bool tile_side_by_side(int rt, int part_keys) { return rt == 32 || part_keys > 0; }

template <typename T, int NJ, int RT>
__global__ void __launch_bounds__(128) paged_attention_tiled_kernel(const T* __restrict__ q, const T* __restrict__ k_pages,
                                                                    const T* __restrict__ v_pages, T* __restrict__ out, const TileArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int KT = tile_keys(NJ, RT), KL = KT / 8, VEC = 16 / (int)sizeof(T);
    constexpr bool SHARED = RT == 32;                      // the four warps share the key tiles
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // the tokens late in a prompt, which see the most keys, first
    const bool side = tile_side_by_side(RT, a.part_keys);
    const int sp = side ? (int)(blockIdx.x % a.n_splits) : blockIdx.z, chunk_at = side ? (int)(blockIdx.x / a.n_splits) : blockIdx.x;
    const int t0 = a.T - 1 - chunk_at / a.row_chunks, kh = blockIdx.y, rc = chunk_at % a.row_chunks;
    const int g = a.nh / a.nkv, hd = a.hd, ld = hd + 4;
    const int seg = a.tok_seg[t0], pos0 = a.positions[t0];
    const int in_group = t0 % a.bq;
    if (in_group != 0 && a.tok_seg[t0 - 1] == seg && a.positions[t0 - 1] + 1 == pos0) return;
    const bool mine = lane == 0 || (in_group + lane < a.bq && t0 + lane < a.T && a.tok_seg[min(t0 + lane, a.T - 1)] == seg &&
                                    a.positions[min(t0 + lane, a.T - 1)] == pos0 + lane);
    const unsigned in_run = __ballot_sync(0xffffffffu, mine);
    const int nq = in_run == 0xffffffffu ? 32 : __ffs(~in_run) - 1;
    const int row0 = rc * RT, nrows = min(nq * g - row0, RT);
    if (nrows <= 0) return;

    extern __shared__ __align__(16) float tile_smem[];
    float* q_s = tile_smem;                                // [RT][ld]
    float* p_s = q_s + RT * ld + warp * (KT + 1) * 8;      // this warp's probabilities [KT][8], then the rows' corrections [8]
    int2* lim = reinterpret_cast<int2*>(q_s + RT * ld + 4 * (KT + 1) * 8);      // [RT]: the keys lo .. hi - 1 a row sees
    float* kv = reinterpret_cast<float*>(lim + RT);
    float* k_s = kv + (SHARED ? 0 : warp * 2 * KT * ld);   // [KT][ld]
    float* v_s = k_s + KT * ld;                            // [KT][ld]

    auto sees = [&](int r) {                               // the keys lo .. hi - 1 that row r sees
        const int pos = pos0 + (row0 + r) / g, hi = pos + 1;
        int lo = (a.window > 0 && hi > a.window) ? hi - a.window : 0;
        if (a.chunk > 0 && pos >= 0) lo = max(lo, pos / a.chunk * a.chunk);
        return r < nrows ? make_int2(lo, hi) : make_int2(0, 0);
    };
    // the run's keys [lo, hi), and this split's part of them in whole tiles counted from lo
    const int lo = sees(0).x, hi = sees(nrows - 1).y;
    // a run with few keys is cut into fewer parts than n_splits, and one that stays whole is finished here
    const int parts = a.part_keys > 0 ? max(1, min(a.n_splits, (hi - lo) / a.part_keys)) : a.n_splits;
    if (sp >= parts) return;
    const bool whole = parts == 1;
    const int tiles = (hi - lo + KT - 1) / KT, per = (tiles + parts - 1) / parts;
    const int begin = lo + sp * per * KT, end = min(begin + per * KT, hi);
    const int step = SHARED ? KT : 4 * KT, first = SHARED ? begin : begin + warp * KT;
    const int* table = a.block_table + (size_t)seg * a.table_stride;

    auto load = [&](float* dst, const T* pages, int n0) {
        const int kn = n0 + min(lane, KT - 1);
        unsigned row = 0;                                  // row of a key in the pages' [pages x heads x page_size, hd]
        if (kn < end) row = ((unsigned)table[kn / a.page_size] * a.nkv + kh) * a.page_size + kn % a.page_size;
#pragma unroll 4
        for (int key = SHARED ? warp : 0; key < KT; key += SHARED ? 4 : 1) {
            const T* src = pages + (long long)__shfl_sync(0xffffffffu, row, key) * hd;
            const bool ok = n0 + key < end;
#pragma unroll
            for (int j = 0; j < (NJ * 4 + VEC - 1) / VEC; ++j) {
                const int c = (lane + 32 * j) * VEC;
                if (c >= hd) break;
                float* d = dst + key * ld + c;
                if (ok) tile_load16<T>(d, src + c);
                else
#pragma unroll
                    for (int e = 0; e < VEC; e += 4) *reinterpret_cast<float4*>(d + e) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    auto meet = [&]() {
        if (SHARED) __syncthreads(); else __syncwarp();
    };

    if (first < end) {
        load(k_s, k_pages, first);
        load(v_s, v_pages, first);
    }
    if (threadIdx.x < RT) lim[threadIdx.x] = sees(threadIdx.x);
    for (int r = warp; r < RT; r += 4) {
        const int tok = t0 + (row0 + r) / g, h = kh * g + (row0 + r) % g;
        for (int d = lane; d < hd; d += 32)
            q_s[r * ld + d] = r < nrows ? to_f32(q[(size_t)tok * a.q_row_stride + (size_t)h * hd + d]) * a.scale : 0.f;
    }
    __syncthreads();

    const int rbase = SHARED ? warp * 8 : 0;               // this warp's 8 rows of the tile
    const int tx = lane & 7, ty = lane >> 3;               // scores: rows rbase + 2 ty, + 1; keys tx, tx + 8, ...
    const int2 lim0 = lim[rbase + 2 * ty], lim1 = lim[rbase + 2 * ty + 1];
    const int h0 = kh * g + (row0 + rbase + 2 * ty) % g, h1 = kh * g + (row0 + rbase + 2 * ty + 1) % g;
    const float slope0 = a.slopes ? a.slopes[h0] : 0.f, slope1 = a.slopes ? a.slopes[h1] : 0.f;
    const float rate0 = a.rates ? a.rates[h0] : 0.f, rate1 = a.rates ? a.rates[h1] : 0.f;
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
    float2 o[8][NJ][2];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int j = 0; j < NJ; ++j) o[r][j][0] = o[r][j][1] = make_float2(0.f, 0.f);
    // keys that every row of this warp sees: tiles inside need no mask
    int all_lo = 0, all_hi = 0x7fffffff;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        all_lo = max(all_lo, lim[rbase + r].x);
        if (rbase + r < nrows) all_hi = min(all_hi, lim[rbase + r].y);
    }
    const bool busy = rbase < nrows;                       // warps without rows only help to load

    for (int n0 = first; n0 < end; n0 += step) {
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        meet();
        const bool inside = n0 >= all_lo && n0 + KT <= all_hi;
        if (busy) {
            float s[2][KL];
            float2 s2[2][KL][2];                           // sums over the dimensions 0, 1 | 2, 3 mod 4
#pragma unroll
            for (int i = 0; i < KL; ++i) s2[0][i][0] = s2[0][i][1] = s2[1][i][0] = s2[1][i][1] = make_float2(0.f, 0.f);
            const float* q0 = q_s + (rbase + 2 * ty) * ld;
            const float* kk = k_s + tx * ld;
#pragma unroll 4
            for (int d = 0; d < hd; d += 4) {
                const float4 a0 = *reinterpret_cast<const float4*>(q0 + d), a1 = *reinterpret_cast<const float4*>(q0 + ld + d);
#pragma unroll
                for (int i = 0; i < KL; ++i) {
                    const float4 b = *reinterpret_cast<const float4*>(kk + i * 8 * ld + d);
                    fma2(s2[0][i][0], make_float2(a0.x, a0.y), make_float2(b.x, b.y));
                    fma2(s2[1][i][0], make_float2(a1.x, a1.y), make_float2(b.x, b.y));
                    fma2(s2[0][i][1], make_float2(a0.z, a0.w), make_float2(b.z, b.w));
                    fma2(s2[1][i][1], make_float2(a1.z, a1.w), make_float2(b.z, b.w));
                }
            }
#pragma unroll
            for (int i = 0; i < KL; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e) s[e][i] = (s2[e][i][0].x + s2[e][i][0].y) + (s2[e][i][1].x + s2[e][i][1].y);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int2 lm = e ? lim1 : lim0;
                float mx = -INFINITY;
#pragma unroll
                for (int i = 0; i < KL; ++i) {
                    const int n = n0 + tx + 8 * i;
                    float v = s[e][i];
                    if (a.softcap > 0.f) v = a.softcap * tanhf(v / a.softcap);      // bounded by +-softcap before the softmax
                    if (a.slopes) {     // a distance bias: slope * distance, or with a rate slope * ln(1 + rate * distance), comes off
                        const float dist = (float)(lm.y - 1 - n);
                        v -= (e ? slope1 : slope0) * (a.rates ? log1pf((e ? rate1 : rate0) * dist) : dist);
                    }
                    s[e][i] = n >= lm.x && n < lm.y && n < end ? v : -INFINITY;
                    mx = fmaxf(mx, s[e][i]);
                }
#pragma unroll
                for (int x = 1; x < 8; x <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
                const float m_new = fmaxf(m[e], mx);
                const float corr = m[e] == -INFINITY ? 0.f : expf(m[e] - m_new);
                float sum = 0.f;
#pragma unroll
                for (int i = 0; i < KL; ++i) {
                    const int n = n0 + tx + 8 * i;
                    const float p = n >= lm.x && n < lm.y && n < end ? expf(s[e][i] - m_new) : 0.f;
                    p_s[(tx + 8 * i) * 8 + 2 * ty + e] = p;
                    sum += p;
                }
#pragma unroll
                for (int x = 1; x < 8; x <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
                l[e] = l[e] * corr + sum;
                m[e] = m_new;
                if (tx == 0) p_s[KT * 8 + 2 * ty + e] = corr;
            }
        }
        meet();                                            // the keys have been read, the probabilities are there
        if (n0 + step < end) load(k_s, k_pages, n0 + step);
        else asm volatile("cp.async.commit_group;\n" ::);
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        meet();
        if (busy) {
            float c[8];
            *reinterpret_cast<float4*>(c) = *reinterpret_cast<const float4*>(p_s + KT * 8);
            *reinterpret_cast<float4*>(c + 4) = *reinterpret_cast<const float4*>(p_s + KT * 8 + 4);
#pragma unroll
            for (int r = 0; r < 8; ++r)
#pragma unroll
                for (int j = 0; j < NJ; ++j)
#pragma unroll
                    for (int e = 0; e < 2; ++e) o[r][j][e] = make_float2(o[r][j][e].x * c[r], o[r][j][e].y * c[r]);
            auto add_values = [&](auto masked) {
#pragma unroll 4
                for (int key = 0; key < KT; ++key) {
                    float p[8];
                    *reinterpret_cast<float4*>(p) = *reinterpret_cast<const float4*>(p_s + key * 8);
                    *reinterpret_cast<float4*>(p + 4) = *reinterpret_cast<const float4*>(p_s + key * 8 + 4);
#pragma unroll
                    for (int j = 0; j < NJ; ++j) {
                        const int d = lane * 4 + 128 * j;
                        if (d >= hd) break;
                        const float4 v = *reinterpret_cast<const float4*>(v_s + key * ld + d);
#pragma unroll
                        for (int r = 0; r < 8; ++r) {
                            // (a value that is not a number must not reach rows that do not see it: 0 * inf)
                            if (decltype(masked)::value && !(n0 + key >= lim[rbase + r].x && n0 + key < lim[rbase + r].y)) continue;
                            fma2(o[r][j][0], make_float2(p[r], p[r]), make_float2(v.x, v.y));
                            fma2(o[r][j][1], make_float2(p[r], p[r]), make_float2(v.z, v.w));
                        }
                    }
                }
            };
            if (inside) add_values(std::false_type());
            else add_values(std::true_type());
        }
        meet();                                            // the values have been read
        if (n0 + step < end) load(v_s, v_pages, n0 + step);
        else asm volatile("cp.async.commit_group;\n" ::);
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");

    // the warps' results to shared memory, [parts][RT][ld] sums and [parts][RT] (max, denominator), then to memory
    __syncthreads();
    constexpr int PARTS = SHARED ? 1 : 4;
    float* po_s = kv;
    float2* ml_s = reinterpret_cast<float2*>(po_s + PARTS * RT * ld);
    const int part = SHARED ? 0 : warp;
    if (tx == 0) {
        ml_s[part * RT + rbase + 2 * ty] = make_float2(m[0], l[0]);
        ml_s[part * RT + rbase + 2 * ty + 1] = make_float2(m[1], l[1]);
    }
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const int d = lane * 4 + 128 * j;
            if (d < hd)
                *reinterpret_cast<float4*>(po_s + (size_t)(part * RT + rbase + r) * ld + d) = make_float4(o[r][j][0].x, o[r][j][0].y, o[r][j][1].x, o[r][j][1].y);
        }
    __syncthreads();
    for (int r = warp; r < nrows; r += 4) {
        const int tok = t0 + (row0 + r) / g, h = kh * g + (row0 + r) % g;
        float M = -INFINITY;
#pragma unroll
        for (int w = 0; w < PARTS; ++w) M = fmaxf(M, ml_s[w * RT + r].x);
        // one more key of score sinks[h] with no value: it only adds to the denominator
        const bool sink = a.sinks && whole;
        if (sink) M = fmaxf(M, a.sinks[h]);
        float f[PARTS], L = sink ? expf(a.sinks[h] - M) : 0.f;
#pragma unroll
        for (int w = 0; w < PARTS; ++w) {
            const float2 ml = ml_s[w * RT + r];
            f[w] = part_factor(ml.x, ml.y, M);
            L += ml.y * f[w];
        }
        const float inv = whole ? (L == 0.f ? 0.f : 1.0f / L) : 1.0f;
        const size_t slot = ((size_t)tok * a.nh + h) * a.n_splits + sp;
        for (int d = lane; d < hd; d += 32) {
            float v = 0.f;
#pragma unroll
            for (int w = 0; w < PARTS; ++w) v = fmaf(po_s[(size_t)(w * RT + r) * ld + d], f[w], v);
            if (whole) out[((size_t)tok * a.nh + h) * hd + d] = from_f32<T>(v * inv);
            else a.part_o[slot * hd + d] = v;
        }
        if (a.n_splits > 1) {          // the row's first part also says what parts there are not (the scratch may begin at any float)
            if (lane == 0) {
                a.part_ml[slot * 2] = whole ? 0.f : M;
                a.part_ml[slot * 2 + 1] = whole ? ATT_WHOLE : L;
            }
            if (sp == 0)
                for (int i = parts + lane; i < a.n_splits; i += 32) {
                    a.part_ml[(slot + i) * 2] = -INFINITY;
                    a.part_ml[(slot + i) * 2 + 1] = 0.f;
                }
        }
    }
}

template <typename T, int NJ, int RT>
static void tile_launch(const T* q, const T* k, const T* v, T* out, TileArgs a, cudaStream_t stream) {
    constexpr int KT = tile_keys(NJ, RT);
    const int g = a.nh / a.nkv, ld = a.hd + 4;
    a.bq = RT / g > 1 ? RT / g : 1;
    a.row_chunks = (a.bq * g + RT - 1) / RT;
    const size_t fixed = ((size_t)RT * ld + 4 * (KT + 1) * 8 + 2 * RT) * sizeof(float);
    const size_t ring = (size_t)(RT == 32 ? 1 : 4) * 2 * KT * ld * sizeof(float);
    const size_t merge = (size_t)(RT == 32 ? 1 : 4) * RT * (ld + 2) * sizeof(float);
    const size_t smem = fixed + (ring > merge ? ring : merge);
    cudaFuncSetAttribute(paged_attention_tiled_kernel<T, NJ, RT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const bool side = tile_side_by_side(RT, a.part_keys);
    pico_launch((paged_attention_tiled_kernel<T, NJ, RT>), dim3((unsigned)a.T * a.row_chunks * (side ? a.n_splits : 1), a.nkv, side ? 1 : a.n_splits), dim3(128), smem, stream, q, k, v,
                out, a);
}

template <typename T>
static void tile_dispatch(const T* q, const T* k, const T* v, T* out, const TileArgs& a, cudaStream_t stream) {
    // 32 rows a block once that makes two blocks a multiprocessor even if every run were full; fewer rows, with the warps
    // side by side over the keys, below.  At the line (1,000 tokens of 12 / 2 heads of 128: 400 blocks of 32 rows) 270 us with
    // 32 rows; 8 rows take 148 us for 700 tokens, which grows to about 300 for 1,000.
    const int g = a.nh / a.nkv, bq = 32 / g > 1 ? 32 / g : 1;
    const bool tall = (long long)(a.T / bq) * a.nkv * (a.part_keys > 0 ? 1 : a.n_splits) >= 2 * pico_num_sms();
    if (a.hd <= 128) {
        if (tall) tile_launch<T, 1, 32>(q, k, v, out, a, stream); else tile_launch<T, 1, 8>(q, k, v, out, a, stream);
    } else if (a.hd <= 256) {
        if (tall) tile_launch<T, 2, 32>(q, k, v, out, a, stream); else tile_launch<T, 2, 8>(q, k, v, out, a, stream);
    } else {
        if (tall) tile_launch<T, 5, 32>(q, k, v, out, a, stream); else tile_launch<T, 5, 8>(q, k, v, out, a, stream);
    }
}

// out[t, h, :] = sum_i o_i exp(m_i - M) / sum_i l_i exp(m_i - M) over the splits i.  RUNS: a row may be finished already, or have fewer parts than
// n_splits, whose places hold anything; asked for each part in front of its loads that costs every call (attention and this kernel, one token of 12 / 2 heads of
// 128 after 2,000 keys in eight parts: 32.4 us, 29.2 without).
template <typename T, bool RUNS>
__global__ void attention_combine_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                         T* __restrict__ out, int hd, int n_splits, const float* __restrict__ sinks,
                                         int nh) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t th = blockIdx.x;  // t * nh + h
    const float* ml = part_ml + th * n_splits * 2;
    if (RUNS && ml[1] == ATT_WHOLE) return;
    float M = sinks ? sinks[th % nh] : -INFINITY;
    for (int i = 0; i < n_splits; ++i) M = fmaxf(M, ml[2 * i]);
    float L = sinks ? expf(sinks[th % nh] - M) : 0.f;
    for (int i = 0; i < n_splits; ++i) L += ml[2 * i + 1] * part_factor(ml[2 * i], ml[2 * i + 1], M);
    const float inv = L == 0.f ? 0.f : 1.0f / L;
    for (int d = threadIdx.x; d < hd; d += blockDim.x) {
        float acc = 0.f;
        for (int i = 0; i < n_splits; ++i) {
            const float o = part_o[(th * n_splits + i) * hd + d], m = ml[2 * i], l = ml[2 * i + 1];
            acc += (RUNS && m == -INFINITY && l == 0.f ? 0.f : o) * part_factor(m, l, M);
        }
        out[th * hd + d] = from_f32<T>(acc * inv);
    }
}

// q: rows of q_row_stride elements, head h at column h*hd.  out: [T, nh*hd].
// part_o: [T*nh*n_splits*hd] floats and part_ml: [T*nh*n_splits*2] floats of scratch, needed
// only when n_splits > 1.  part_keys > 0: a run of rows is cut into so many parts only that each has that many keys.  block_table: [segments, table_stride] page numbers.
PICO_API int pico_paged_attention_generic(const void* q, int q_row_stride, const void* k_pages,
                                          const void* v_pages, void* out, float* part_o, float* part_ml,
                                          const int* tok_seg, const int* positions, const int* block_table,
                                          int table_stride, int T, int nh, int nkv, int hd, int page_size,
                                          int window, float scale, int n_splits, float softcap, int act_dtype,
                                          const float* slopes, int chunk, const float* sinks, const float* rates, int part_keys,
                                          cudaStream_t stream) {
    if (T <= 0) return 0;
    if (hd % 16 != 0 || hd < 16 || hd > ATT_MAX_HD || (rates && !slopes)) return PICO_ERR_SIZE;
    if (nkv <= 0 || nh % nkv != 0 || n_splits < 1 || n_splits > 65535 || nkv > 65535) return PICO_ERR_SIZE;
    if (n_splits > 1 && (!part_o || !part_ml)) return PICO_ERR_SIZE;
    // (blocks along x: a row's chunks of 8 rows at most, times the parts)
    if (chunk < 0 || part_keys < 0 || (long long)T * ((nh / nkv + 7) / 8) * n_splits > 0x7fffffffLL) return PICO_ERR_SIZE;
    const TileArgs a = {q_row_stride, table_stride, T, nh, nkv, hd, page_size, window, n_splits, chunk, 1, 1, part_keys, scale, softcap,
                        tok_seg, positions, block_table, slopes, sinks, rates, part_o, part_ml};
    if (act_dtype == PICO_F32) {
        if ((q_row_stride % 4) != 0) return PICO_ERR_ALIGN;
        tile_dispatch<float>((const float*)q, (const float*)k_pages, (const float*)v_pages, (float*)out, a, stream);
        if (n_splits > 1)
            pico_launch((part_keys > 0 ? attention_combine_kernel<float, true> : attention_combine_kernel<float, false>), dim3(T * nh), dim3(64), 0, stream, part_o, part_ml, (float*)out, hd, n_splits, sinks, nh);
    } else if (act_dtype == PICO_BF16) {
        tile_dispatch<bf16>((const bf16*)q, (const bf16*)k_pages, (const bf16*)v_pages, (bf16*)out, a, stream);
        if (n_splits > 1)
            pico_launch((part_keys > 0 ? attention_combine_kernel<bf16, true> : attention_combine_kernel<bf16, false>), dim3(T * nh), dim3(64), 0, stream, part_o, part_ml, (bf16*)out, hd, n_splits, sinks, nh);
    } else
        return PICO_ERR_DTYPE;
    return pico_launch_status();
}

// ---------------------------------------------------------------------------------------------
// The entry point that allocates nothing (declared and documented in pico_noalloc.h; it has no
// counterpart in the reference).  Its scratch is this file-scope device array.  In host code the
// name g_noalloc_scratch is only a stand-in for the symbol, not a device address: the address
// the kernels get comes from cudaGetSymbolAddress, looked up once per device below.
#include "pico_noalloc.h"
#include <stdio.h>

#define PICO_ERR_SCRATCH (-5)
#define PICO_ERR_SYMBOL (-6)
#define PICO_NOALLOC_MAX_DEVICES 64

static __device__ __align__(256) float g_noalloc_scratch[PICO_NOALLOC_SCRATCH_FLOATS];
static float* g_noalloc_scratch_ptr[PICO_NOALLOC_MAX_DEVICES];   // device address, per device; 0 = not looked up

static int noalloc_fail(int code, char* err, int err_len, const char* msg) {
    if (err && err_len > 0) snprintf(err, (size_t)err_len, "pico_paged_attention_noalloc: %s", msg);
    return code;
}

PICO_API int pico_paged_attention_noalloc(const void* q, int q_row_stride, const void* k_pages,
                                          const void* v_pages, void* out, const int* tok_seg,
                                          const int* positions, const int* block_table, int table_stride,
                                          int T, int nh, int nkv, int hd, int page_size, int window, float scale,
                                          int n_splits, int act_dtype, cudaStream_t stream, char* err,
                                          int err_len) {
    if (err && err_len > 0) err[0] = 0;
    if (T <= 0) return 0;
    // the same limits as pico_paged_attention_generic, checked first so that the product below cannot wrap
    if (nh <= 0 || nkv <= 0 || nkv > 65535 || nh % nkv != 0 || hd % 16 != 0 || hd < 16 || hd > ATT_NOALLOC_MAX_HD ||
        n_splits < 1 || n_splits > 65535)
        return noalloc_fail(PICO_ERR_SIZE, err, err_len, "a size the attention kernels do not take");
    // one part per token needs no scratch at all: the kernel writes its result straight to out
    const long long need = n_splits == 1 ? 0 : (long long)T * nh * n_splits * (hd + 2);
    if (need > (long long)PICO_NOALLOC_SCRATCH_FLOATS) {
        char msg[200];
        snprintf(msg, sizeof msg,
                 "T*nh*n_splits*(hd+2) = %lld float32 of scratch wanted, the built-in array holds %d "
                 "(use fewer splits or tokens, or pico_paged_attention_generic with your own buffer)",
                 need, (int)PICO_NOALLOC_SCRATCH_FLOATS);
        return noalloc_fail(PICO_ERR_SCRATCH, err, err_len, msg);
    }
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= PICO_NOALLOC_MAX_DEVICES)
        return noalloc_fail(PICO_ERR_SYMBOL, err, err_len, "cannot tell the current device");
    if (!g_noalloc_scratch_ptr[dev]) {
        // set-up, once per device, with that device current
        float* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress((void**)&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            char msg[160];
            snprintf(msg, sizeof msg, "cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
            return noalloc_fail(PICO_ERR_SYMBOL, err, err_len, msg);
        }
        g_noalloc_scratch_ptr[dev] = p;
    }
    float* part_o = g_noalloc_scratch_ptr[dev];
    float* part_ml = part_o + (size_t)T * nh * n_splits * hd;
    const int rc = pico_paged_attention_generic(q, q_row_stride, k_pages, v_pages, out, part_o, part_ml, tok_seg,
                                                positions, block_table, table_stride, T, nh, nkv, hd, page_size,
                                                window, scale, n_splits, 0.f, act_dtype, nullptr, 0, nullptr, nullptr, 0, stream);
    if (rc == PICO_ERR_SIZE) return noalloc_fail(rc, err, err_len, "a size the attention kernels do not take");
    if (rc == PICO_ERR_DTYPE) return noalloc_fail(rc, err, err_len, "act_dtype must be 0 (float32) or 1 (bfloat16)");
    if (rc == PICO_ERR_ALIGN) return noalloc_fail(rc, err, err_len, "q_row_stride must be a multiple of 4 for float32");
    if (rc != 0) return noalloc_fail(rc, err, err_len, "kernel launch failed");
    return 0;
}
