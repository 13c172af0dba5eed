// Next-token choice from float32 logits: argmax (temperature 0), temperature sampling, and nucleus
// (top-p) sampling, by inverse CDF with one uniform number per row that the host supplies.
//
// Restated from the reference: temperature 0 means argmax (pico_vllm/sampler.py:3-8,62-63);
// otherwise probabilities are softmax(logits / temperature) (sampler.py:16); top-p keeps, in
// descending order of probability, every token whose higher-ranked tokens hold less than top_p
// of the mass, and renormalises (sampler.py:26-33); top_p >= 1 turns it off (sampler.py:64).
// The reference draws with torch.multinomial from torch's global generator; here the draw is the
// first token, in vocabulary order, at which the running sum of kept probabilities passes
// uniform * kept mass, so a row's result depends only on its logits, parameters and uniform.
//
// A row (600 KB for a vocabulary of 150 k entries) belongs to one cluster of eight blocks: each reads an eighth of it once, keeps
// it in shared memory through all the passes, and what the blocks have to tell one another goes through distributed shared memory.
// Short rows belong to one block, rows of more than 155,648 entries to sixteen (see sample_shape).
// Masses are summed as 32.32 fixed-point integers (weight = exp((x - max) / T) <= 1), so that sums do not depend on the order in
// which blocks and threads add: the choice is reproducible.
//   1. maximum and its first index (greedy rows end here);
//   2. the kept set without sorting: token i is kept iff the mass of tokens with a larger weight is
//      < top_p * total.  The smallest kept weight is found by its bit pattern, 11 + 11 + 10 bits at a
//      time: a histogram of mass per value of the next bits among the weights that share the bits
//      found so far, then the lowest bin whose mass above is still below the limit (equal weights
//      are kept or dropped together);
//   3. kept mass per block, the block and then the token at which the running sum passes the target.
// A pass that is a kernel of its own, over the row in L2, with the blocks' results in device memory, costs 10 to 25 us at 64 rows
// of 152,064 whatever it computes; the whole choice with top-p took 214 us as five of them (175 without top-p) and 75 (30) as this one; 37 rows run
// at a time.  1, 8, 32 rows: 35, 71, 132 us, now 28, 30, 45.
// Sixteen blocks keep rows of up to 778,240 entries; longer ones are read again in every pass (1,000,000 entries with top-p, 1 / 8 / 32
// rows: 97 / 131 / 319 us; as five kernels with up to 64 parts a row 75 / 187 / 679: single rows of such a length are slower).
#include "common.cuh"

#define SAMPLE_THREADS 512
#define SAMPLE_BINS 2048
#define SAMPLE_FLUSH 65532       // elements whose masses' halves fit into 32-bit sums
#define SAMPLE_KEEP_ALONE 48640  // ... with a multiprocessor to itself
#define SAMPLE_KEEP 19456        // elements of a block's part that shared memory keeps (two blocks on a multiprocessor)

typedef unsigned long long u64;

__device__ __forceinline__ float sample_weight(float x, float mx, float inv_t) { return expf((x - mx) * inv_t); }
__device__ __forceinline__ u64 sample_fixed(float w) { return __float2ull_rz(w * 4294967296.0f); }

// sums and exclusive prefix sums of 64-bit integers over the block, in thread order; scratch: 33 entries
__device__ __forceinline__ u64 block_excl_scan_u64(u64 v, u64* scratch, u64* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nwarps = blockDim.x >> 5;
    u64 inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u64 n = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += n;
    }
    __syncthreads();
    if (lane == 31) scratch[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const u64 w = lane < nwarps ? scratch[lane] : 0ull;
        u64 winc = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u64 n = __shfl_up_sync(0xffffffffu, winc, o);
            if (lane >= o) winc += n;
        }
        scratch[lane] = winc - w;
        if (lane == 31) scratch[32] = winc;
    }
    __syncthreads();
    const u64 res = scratch[warp] + inc - v;
    *total = scratch[32];
    return res;
}
__device__ __forceinline__ int block_min_int(int v, int* scratch) {       // scratch: 33 ints
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        int c = threadIdx.x < (blockDim.x >> 5) ? scratch[threadIdx.x] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) c = min(c, __shfl_xor_sync(0xffffffffu, c, o));
        if (threadIdx.x == 0) scratch[32] = c;
    }
    __syncthreads();
    return scratch[32];
}

// what every block of the cluster has written to another's shared memory is there afterwards
__device__ __forceinline__ void sample_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ uint32_t sample_at(const void* mine, int block) {      // the same place in another block's shared memory
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(mine)), "r"(block));
    return r;
}
__device__ __forceinline__ void sample_put(const u64* mine, int block, u64 v) {
    asm volatile("st.shared::cluster.u64 [%0], %1;\n" ::"r"(sample_at(mine, block)), "l"(v) : "memory");
}
__device__ __forceinline__ u64 sample_get(const u64* mine, int block) {
    u64 v;
    asm volatile("ld.shared::cluster.u64 %0, [%1];\n" : "=l"(v) : "r"(sample_at(mine, block)) : "memory");
    return v;
}

// Grid (BLOCKS, rows) in clusters of BLOCKS.  Block b takes elements [b * per, (b + 1) * per) of the row, per a multiple of 4.  KEEP: they stay in
// shared memory (as weights from pass 2 on); vec: the row starts on 16 bytes and V is a multiple of 4.
template <bool KEEP, int BLOCKS>
__global__ void __launch_bounds__(SAMPLE_THREADS)
sample_row_kernel(const float* __restrict__ logits, int row_stride, int V, const float* __restrict__ temperature,
                  const float* __restrict__ top_p, const float* __restrict__ uniform, int* __restrict__ out, int per, bool vec) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) unsigned char sample_smem[];
    u64* hist = reinterpret_cast<u64*>(sample_smem);                  // [BINS]: this block's masses
    unsigned* halves = reinterpret_cast<unsigned*>(hist + SAMPLE_BINS);       // [BINS] lower 16 bits, [BINS] upper: while they are summed
    u64* all = reinterpret_cast<u64*>(halves);                        // [BINS]: the row's masses, when `halves` is done with
    float* kept = reinterpret_cast<float*>(all + SAMPLE_BINS);        // KEEP: [per]
    __shared__ float scratch[33];
    __shared__ int iscratch[33];
    __shared__ u64 scratch64[33];
    __shared__ u64 told[BLOCKS], told_kept[BLOCKS];     // what the blocks say: maximum and index; kept mass
    __shared__ u64 s_above;
    const int r = blockIdx.y, rank = blockIdx.x, tid = threadIdx.x;
    sample_cluster_sync();              // every block of the cluster runs before another writes to it
    pdl_wait();
    const float* x = logits + (size_t)r * row_stride;
    const int p0 = min(V, rank * per), n = min(V, p0 + per) - p0;
    x += p0;

    // ---- 1: the maximum and its first index; the elements into shared memory
    float best = -INFINITY;
    int best_i = 0x7fffffff;
    // f(element, place) over a, a + step, .. below b; a row that is read again: eight loads under way
    auto walk = [&](int a, int b, int step, auto f) {
        if (KEEP) {
#pragma unroll 4
            for (int i = a; i < b; i += step) f(kept[i], i);
        } else {
            for (int i = a; i < b; i += 8 * step) {
                float v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (i + u * step < b) v[u] = x[i + u * step];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (i + u * step < b) f(v[u], i + u * step);
            }
        }
    };
    auto see = [&](float v, int i) {
        if (v > best) { best = v; best_i = i; }
    };
    if (vec) {
        constexpr int STEP = SAMPLE_THREADS * 4;
        for (int i0 = tid * 4; i0 < n; i0 += 4 * STEP) {              // four loads of 16 bytes under way
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (i0 + u * STEP < n) v[u] = *reinterpret_cast<const float4*>(x + i0 + u * STEP);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = i0 + u * STEP;
                if (i < n) {
                    if (KEEP) *reinterpret_cast<float4*>(kept + i) = v[u];
                    see(v[u].x, p0 + i);
                    see(v[u].y, p0 + i + 1);
                    see(v[u].z, p0 + i + 2);
                    see(v[u].w, p0 + i + 3);
                }
            }
        }
    } else {
#pragma unroll 4
        for (int i = tid; i < n; i += SAMPLE_THREADS) {
            const float v = x[i];
            if (KEEP) kept[i] = v;
            see(v, p0 + i);
        }
    }
    {
        const float pm = block_max(best, scratch);
        const int pc = block_min_int(best == pm ? best_i : 0x7fffffff, iscratch);
        if (tid < BLOCKS) sample_put(told + rank, tid, ((u64)__float_as_uint(pm) << 32) | (unsigned)pc);
    }
    sample_cluster_sync();
    float mx = -INFINITY;
    int arg = 0x7fffffff;
#pragma unroll
    for (int b = 0; b < BLOCKS; ++b) {                         // in the row's order: the first index of the maximum stays the first
        const float m = __uint_as_float((unsigned)(told[b] >> 32));
        const int i = (int)(unsigned)told[b];
        if (m > mx || (m == mx && i < arg)) { mx = m; arg = i; }
    }
    const float temp = temperature ? temperature[r] : 0.f;
    if (!(temp > 0.f) || arg == 0x7fffffff) {                         // greedy, or a row without a finite maximum
        if (rank == 0 && tid == 0) out[r] = arg == 0x7fffffff ? 0 : arg;
        return;
    }
    const float inv_t = 1.0f / temp;
    const float tp = top_p ? top_p[r] : 1.f;

    // ---- 2: the smallest kept weight
    unsigned thresh = 0u, prefix = 0u;
    bool weights = false;                                             // `kept` holds weights
    if (tp < 1.f) {
        u64 limit = 0ull, above = 0ull;
        for (int level = 0; level < 3; ++level) {
            const int bins = level == 2 ? 1024 : SAMPLE_BINS;
            for (int f0 = 0; f0 < n || f0 == 0; f0 += SAMPLE_FLUSH) {
                for (int b = tid; b < 2 * SAMPLE_BINS; b += SAMPLE_THREADS) halves[b] = 0u;
                __syncthreads();
                const int f1 = min(n, f0 + SAMPLE_FLUSH);
                walk(f0 + tid, f1, SAMPLE_THREADS, [&](float v, int i) {
                    float w = v;
                    if (!KEEP || level == 0) {
                        w = sample_weight(v, mx, inv_t);
                        if (KEEP) kept[i] = w;
                    }
                    const unsigned pat = __float_as_uint(w);
                    const u64 fx = sample_fixed(w);
                    if (fx == 0ull || (level == 1 && (pat >> 21) != prefix) || (level == 2 && (pat >> 10) != prefix)) return;
                    const unsigned bin = level == 0 ? pat >> 21 : level == 1 ? (pat >> 10) & 0x7ffu : pat & 0x3ffu;
                    // (32-bit adds: 64-bit ones in shared memory are loops)
                    atomicAdd(halves + bin, (unsigned)fx & 0xffffu);
                    atomicAdd(halves + SAMPLE_BINS + bin, (unsigned)(fx >> 16));
                });
                __syncthreads();
                for (int b = tid; b < SAMPLE_BINS; b += SAMPLE_THREADS) {
                    const u64 m = (u64)halves[b] + ((u64)halves[SAMPLE_BINS + b] << 16);
                    hist[b] = f0 == 0 ? m : hist[b] + m;
                }
                __syncthreads();
            }
            weights = KEEP;
            sample_cluster_sync();                                    // every block's masses are there, every block's `halves` free
            for (int i = tid; i < SAMPLE_BINS / BLOCKS; i += SAMPLE_THREADS) {      // a block adds up its share of the bins and tells all
                const int b = rank * (SAMPLE_BINS / BLOCKS) + i;
                u64 sum = 0ull;
#pragma unroll
                for (int o = 0; o < BLOCKS; ++o) sum += sample_get(hist + b, o);
#pragma unroll
                for (int o = 0; o < BLOCKS; ++o) sample_put(all + b, o, sum);
            }
            sample_cluster_sync();
            // the lowest bin whose mass above (in higher bins, and above the bits found before) is below the limit: thread t has
            // four bins, descending, so that a prefix sum is the mass above
            const int top = bins - 1 - 4 * tid;
            u64 h[4], mine = 0ull, total;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                h[e] = top - e >= 0 ? all[top - e] : 0ull;
                mine += h[e];
            }
            u64 before = above + block_excl_scan_u64(mine, scratch64, &total);
            if (level == 0) limit = (u64)((double)tp * (double)total);
            int cand = 0x7fffffff;
            u64 cand_above = 0ull;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (top - e >= 0 && before < limit) {
                    cand = top - e;
                    cand_above = before;
                }
                before += h[e];
            }
            const int bin = block_min_int(cand, iscratch);
            if (bin == 0x7fffffff) {                                  // a limit of zero: only the largest weight (1.0) is kept
                thresh = __float_as_uint(1.0f);
                break;
            }
            if (cand == bin) s_above = cand_above;
            __syncthreads();
            above = s_above;
            prefix = level == 0 ? (unsigned)bin : level == 1 ? (prefix << 11) | (unsigned)bin : (prefix << 10) | (unsigned)bin;
            thresh = prefix;
            __syncthreads();                                          // `all` has been read, as has s_above
        }
    }

    // ---- 3: kept mass.  Of a row in shared memory a thread takes a run of neighbours (an odd number: distinct banks), so that the scan is in the
    // row's order; of others the whole block reads side by side
    const int run = ((n + SAMPLE_THREADS - 1) / SAMPLE_THREADS) | 1;
    const int c0 = KEEP ? min(n, tid * run) : tid, c1 = KEEP ? min(n, c0 + run) : n, step = KEEP ? 1 : SAMPLE_THREADS;
    auto kept_mass = [&](float v) {
        const float w = weights ? v : sample_weight(v, mx, inv_t);
        return __float_as_uint(w) >= thresh ? sample_fixed(w) : 0ull;
    };
    u64 mine = 0ull, part;
    walk(c0, c1, step, [&](float v, int) { mine += kept_mass(v); });
    u64 before = block_excl_scan_u64(mine, scratch64, &part);
    if (tid < BLOCKS) sample_put(told_kept + rank, tid, part);
    sample_cluster_sync();
    u64 mass = 0ull, start = 0ull;
#pragma unroll
    for (int b = 0; b < BLOCKS; ++b) {
        if (b < rank) start += told_kept[b];
        mass += told_kept[b];
    }
    const u64 target = (u64)((double)uniform[r] * (double)mass);
    int winner = -1;                    // the last block that is not empty and starts at or below the target
    u64 at = 0ull;
#pragma unroll
    for (int b = 0; b < BLOCKS; ++b) {
        if (told_kept[b] > 0ull && at <= target) winner = b;
        at += told_kept[b];
    }
    if (winner < 0) {                   // nothing was kept (cannot happen with a finite maximum)
        if (rank == 0 && tid == 0) out[r] = arg;
        return;
    }
    if (rank != winner) return;
    if (KEEP) {
        before += start;
        const int who = -block_min_int((mine > 0ull && before <= target) ? -tid : 1, iscratch);
        if (tid == who) {
            int pick = -1, last = -1;
            for (int i = c0; i < c1; ++i) {
                const u64 fx = kept_mass(kept[i]);
                if (fx == 0ull) continue;
                before += fx;
                last = p0 + i;
                if (before > target) { pick = p0 + i; break; }
            }
            out[r] = pick >= 0 ? pick : (last >= 0 ? last : arg);
        }
    } else {
        // the part that is not empty and starts at or below the target, the last such one: a sixteenth for each warp, then a sixteenth of
        // that, until an element is left for each thread
        constexpr int WARPS = SAMPLE_THREADS / 32;
        const int lane = tid & 31, warp = tid >> 5;
        int lo = 0, hi = n;
        u64 upto = start;                                             // mass before lo
        while (hi - lo > SAMPLE_THREADS) {
            const int each = (hi - lo + WARPS - 1) / WARPS, w0 = min(hi, lo + warp * each), w1 = min(hi, w0 + each);
            u64 sum = 0ull;
            walk(w0 + lane, w1, 32, [&](float v, int) { sum += kept_mass(v); });
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            if (lane == 0) scratch64[warp] = sum;
            __syncthreads();
            u64 at = upto;
            int who = 0;
            for (int w = 0; w < WARPS; ++w) {
                if (scratch64[w] > 0ull && at <= target) {
                    who = w;
                    upto = at;
                }
                at += scratch64[w];
            }
            lo = min(hi, lo + who * each);
            hi = min(hi, lo + each);
            __syncthreads();                                          // the sums have been read
        }
        mine = lo + tid < hi ? kept_mass(x[lo + tid]) : 0ull;
        before = upto + block_excl_scan_u64(mine, scratch64, &part);
        const int who = -block_min_int((mine > 0ull && before <= target) ? -tid : 1, iscratch);
        if (tid == 0) out[r] = who >= 0 ? p0 + lo + who : arg;
    }
}

static size_t sample_bytes(int per) { return 2 * SAMPLE_BINS * sizeof(u64) + (size_t)per * sizeof(float); }

// Can clusters of sixteen run here with that much shared memory?
template <bool KEEP>
static bool sample_sixteen(size_t smem) {
    if (cudaFuncSetAttribute(sample_row_kernel<KEEP, 16>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaFuncSetAttribute(sample_row_kernel<KEEP, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(SAMPLE_THREADS);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 16;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, sample_row_kernel<KEEP, 16>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return n > 0;
}

struct SampleShape { int blocks; bool keep; };      // blocks of a row, and whether they keep it
// One block for rows of up to 4,096 entries, and while more rows wait than run at once also for those that one block keeps: what the
// passes cost beside the entries, clearing and adding up 2,048 bins and the clusters' barriers, is per block (us with top-p, in 1 / 8 blocks:
// rows of 2,000: 1 row 11 / 15, 64 rows 11 / 44, 256 18 / 132; of 16,384: 1 row 21 / 16, 64 21 / 46).  Eight up to what eight of them keep, two on a multiprocessor.  Beyond, sixteen
// where the device runs such clusters, which keep what they can with a multiprocessor to each (262,144 entries, 1 / 64 rows: 29 / 165 us, in eight that keep nothing
// 72 / 185).  Greedy rows are read once: nothing is kept there.
static SampleShape sample_shape(int R, int V, bool drawn) {
    if (V <= 4096 || (R > pico_num_sms() / 4 && V <= SAMPLE_KEEP)) return {1, true};
    if (V <= 8 * SAMPLE_KEEP) return {8, true};
    static const bool sixteen_keep = sample_sixteen<true>(sample_bytes(SAMPLE_KEEP_ALONE)), sixteen = sample_sixteen<false>(sample_bytes(0));
    if (V <= 16 * SAMPLE_KEEP_ALONE) return drawn && sixteen_keep ? SampleShape{16, true} : SampleShape{8, false};
    return {sixteen ? 16 : 8, false};
}

// logits: [R, row_stride] float32, the first V columns are used.  temperature, top_p, uniform:
// [R] float32 (temperature/top_p may be null: greedy / no nucleus).  out: [R] int32.
PICO_API int pico_sample(const float* logits, int row_stride, int R, int V, const float* temperature,
                         const float* top_p, const float* uniform, int* out, cudaStream_t stream) {
    if (R <= 0) return 0;
    if (V <= 0) return PICO_ERR_SIZE;
    if (temperature && !uniform) return PICO_ERR_SIZE;
    const SampleShape shape = sample_shape(R, V, temperature != nullptr);
    const int per = ((V + shape.blocks - 1) / shape.blocks + 3) / 4 * 4;
    const size_t smem = sample_bytes(shape.keep ? per : 0);
    const bool vec = V % 4 == 0 && row_stride % 4 == 0 && ((uintptr_t)logits & 15) == 0;
    for (int r0 = 0; r0 < R; r0 += 65535) {
        const int rows = R - r0 < 65535 ? R - r0 : 65535;
        const float* lg = logits + (size_t)r0 * row_stride;
        const float *t = temperature ? temperature + r0 : nullptr, *tp = top_p ? top_p + r0 : nullptr, *u = uniform ? uniform + r0 : nullptr;
#define SAMPLE_LAUNCH(K, B)                                                                                                      \
    do {                                                                                                                         \
        cudaFuncSetAttribute(sample_row_kernel<K, B>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);                   \
        pico_launch_cluster((sample_row_kernel<K, B>), dim3(B, rows), dim3(SAMPLE_THREADS), smem, stream, B, lg, row_stride, V, t, tp, u, \
                            out + r0, per, vec);                                                                                 \
    } while (0)
        if (shape.blocks == 1) SAMPLE_LAUNCH(true, 1);
        else if (shape.blocks == 8 && shape.keep) SAMPLE_LAUNCH(true, 8);
        else if (shape.blocks == 8) SAMPLE_LAUNCH(false, 8);
        else if (shape.keep) SAMPLE_LAUNCH(true, 16);
        else SAMPLE_LAUNCH(false, 16);
#undef SAMPLE_LAUNCH
    }
    return pico_launch_status();
}
