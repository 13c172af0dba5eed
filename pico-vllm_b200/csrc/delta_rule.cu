// The gated delta rule: a matrix memory per head and request whose rows decay and whose write is corrected by what the
// memory already holds under the key,
//
//   S <- diag(a_t) S ;   u = beta_t (v_t - S^T k_t) ;   S <- S + k_t u^T ;   o_t = S^T q_t          (S: [d, dv], float32)
//
// token by token, the read seeing the write; the decay a_t is one number per row of S, or one for the whole of it (PER_HEAD).
// With the decayed memory S' = diag(a_t) S both sums over rows are taken in one
// pass,  r1 = S'^T k_t  and  r2 = S'^T q_t :  u = beta_t (v_t - r1),  o_t = r2 + u (k_t . q_t),  so a token costs one pass
// over the registers, one reduction and one update.
//
// delta_prepare_kernel makes the float32 inputs of the recurrence from the projections: q and k as unit vectors per head
// (q times d^-1/2), beta = sigmoid, the decay a = exp(-exp(A_log) softplus(z + bias)) per head and row (or per head), and k . q.
// gated_delta_rule_kernel is the recurrence: the columns of S evolve independently of each other, so a block takes
// 16 columns of one head of one segment, eight or sixteen lanes a column with the rows dealt out among them in
// registers; the state is stored transposed [slot, head, dv, d].  A token's q, k and decay pass through shared
// memory, DR_TOK tokens at a time, the next ones' loads in flight (cp.async) while these are walked.  A segment of one token is a decode step; a
// portion of a prompt goes on from the state the portion before left.
//
// Everything here is float32 whatever the activation type; only the projections read are not.
#include "common.cuh"

#define DR_TOK 8

__device__ __forceinline__ float dr_sigmoid(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float dr_softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }

// Grid (tokens, 1 + H): block y = 0 makes the unit vectors and k . q of all query/key heads (a warp a head), block y = h + 1
// the decays and beta of head h (PER_HEAD: block y = 0 makes those too, a thread a head, and there are no others).  xc float32 [T, >= q_off.. ] holds the convolved q and k (G heads of d each); proj
// (activation type) holds one beta logit per head at b_off; dt [T, H * d] (PER_HEAD: [T, H]; activation type) the
// decay's argument before its bias.  prep float32 [T, P] with P = 2 G d + H d + H + G:  q | k | a | beta | k . q.
// PER_HEAD: P = 2 G d + 4 H + 8 G:  q | k | four numbers a head: a, beta, two of no use | eight numbers a query/key head: q_t . k_(t-j) for
// j = 0 .. 3, k_t . k_(t-j) for j = 1 .. 3 (with `back`; else the first alone), one of no use; k_(t-j) is the row j before - of
// use where that is the same request's token.
template <typename TA, bool PER_HEAD>
__global__ void __launch_bounds__(128)
delta_prepare_kernel(const float* __restrict__ xc, int xc_stride, int q_off, int k_off, const TA* __restrict__ proj,
                     int proj_stride, int b_off, const TA* __restrict__ dt, int dt_stride, const float* __restrict__ dt_bias,
                     const float* __restrict__ a_log, float* __restrict__ prep, int P, int H, int G, int d, float q_scale,
                     float unit_eps, int back, int vec) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t t = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    float* out = prep + t * P;
    if (PER_HEAD) {
        for (int h = threadIdx.x; h < H; h += blockDim.x) {
            const float z = to_f32(dt[t * dt_stride + h]) + (dt_bias ? dt_bias[h] : 0.f);
            out[2 * G * d + 4 * h] = expf(-expf(a_log[h]) * dr_softplus(z));
            out[2 * G * d + 4 * h + 1] = dr_sigmoid(to_f32(proj[t * proj_stride + b_off + h]));
        }
    } else if (blockIdx.y > 0) {
        const int h = blockIdx.y - 1;
        const float rate = expf(a_log[h]);
        for (int i = threadIdx.x; i < d; i += blockDim.x) {
            const float z = to_f32(dt[t * dt_stride + h * d + i]) + (dt_bias ? dt_bias[h * d + i] : 0.f);
            out[2 * G * d + h * d + i] = expf(-rate * dr_softplus(z));
        }
        if (threadIdx.x == 0) out[2 * G * d + H * d + h] = dr_sigmoid(to_f32(proj[t * proj_stride + b_off + h]));
        return;
    }
    const float* row = xc + t * xc_stride;
    if (PER_HEAD && vec) {
        // four numbers a lane, each read once (2,048 tokens of 6 heads of 128: 14 us, 18 in two passes a number a load)
        for (int g = warp; g < G; g += nw) {
            const int i = lane * 4;
            const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
            float4 a = zero, b = zero, c[3] = {zero, zero, zero};
            if (i < d) {
                a = *reinterpret_cast<const float4*>(row + q_off + g * d + i);
                b = *reinterpret_cast<const float4*>(row + k_off + g * d + i);
                if (back) {
#pragma unroll
                    for (int j = 0; j < 3; ++j)
                        if (t > j) c[j] = *reinterpret_cast<const float4*>(row - (size_t)(j + 1) * xc_stride + k_off + g * d + i);
                }
            }
            auto dot = [](float4 x, float4 y) { return fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, x.x * y.x))); };
            float s[12] = {dot(a, a), dot(b, b), dot(a, b), dot(c[0], c[0]), dot(c[1], c[1]), dot(c[2], c[2]),
                           dot(a, c[0]), dot(a, c[1]), dot(a, c[2]), dot(b, c[0]), dot(b, c[1]), dot(b, c[2])};
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
                for (int x = 0; x < 12; ++x)
                    if (x < 3 || back) s[x] += __shfl_xor_sync(0xffffffffu, s[x], o);
            }
            const float iq = q_scale / sqrtf(s[0] + unit_eps), ik = 1.0f / sqrtf(s[1] + unit_eps);
            if (i < d) {
                *reinterpret_cast<float4*>(out + g * d + i) = make_float4(a.x * iq, a.y * iq, a.z * iq, a.w * iq);
                *reinterpret_cast<float4*>(out + G * d + g * d + i) = make_float4(b.x * ik, b.y * ik, b.z * ik, b.w * ik);
            }
            if (lane == 0) {
                float* dots = out + 2 * G * d + 4 * H + 8 * g;
                dots[0] = iq == 0.f || ik == 0.f ? 0.f : s[2] * iq * ik;       // (rows whose squares overflow are nought, not inf * 0)
                if (back) {
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        const float in = 1.0f / sqrtf(s[3 + j] + unit_eps);
                        dots[1 + j] = s[6 + j] * iq * in;
                        dots[4 + j] = s[9 + j] * ik * in;
                    }
                }
            }
        }
        return;
    }
    for (int g = warp; g < G; g += nw) {
        float sq = 0.f, sk = 0.f;
        for (int i = lane; i < d; i += 32) {
            const float a = row[q_off + g * d + i], b = row[k_off + g * d + i];
            sq += a * a;
            sk += b * b;
        }
        sq = warp_sum(sq);
        sk = warp_sum(sk);
        const float iq = q_scale / sqrtf(sq + unit_eps), ik = 1.0f / sqrtf(sk + unit_eps);
        float kq = 0.f;
        for (int i = lane; i < d; i += 32) {
            const float a = row[q_off + g * d + i] * iq, b = row[k_off + g * d + i] * ik;
            out[g * d + i] = a;
            out[G * d + g * d + i] = b;
            kq += a * b;
        }
        kq = warp_sum(kq);
        float* dots = out + 2 * G * d + (PER_HEAD ? 4 * H + 8 * g : H * d + H + g);
        if (lane == 0) dots[0] = kq;
        if (PER_HEAD && back) {
            float n[3] = {0.f, 0.f, 0.f}, dq[3] = {0.f, 0.f, 0.f}, dk[3] = {0.f, 0.f, 0.f};
            for (int i = lane; i < d; i += 32) {
                const float a = row[q_off + g * d + i], b = row[k_off + g * d + i];
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    if (t > j) {
                        const float c = (row - (size_t)(j + 1) * xc_stride)[k_off + g * d + i];
                        n[j] = fmaf(c, c, n[j]);
                        dq[j] = fmaf(a, c, dq[j]);
                        dk[j] = fmaf(b, c, dk[j]);
                    }
            }
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                n[j] = warp_sum(n[j]);
                dq[j] = warp_sum(dq[j]);
                dk[j] = warp_sum(dk[j]);
            }
            if (lane == 0) {
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const float in = 1.0f / sqrtf(n[j] + unit_eps);
                    dots[1 + j] = dq[j] * iq * in;
                    dots[4 + j] = dk[j] * ik * in;
                }
            }
        }
    }
}

PICO_API int pico_delta_prepare(const float* xc, int xc_stride, int q_off, int k_off, const void* proj, int proj_stride,
                                int b_off, const void* dt, int dt_stride, const float* dt_bias, const float* a_log,
                                float* prep, int T, int H, int G, int d, float q_scale, float unit_eps, int per_head,
                                int back, int dtype, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (H < 1 || G < 1 || H % G || d < 1 || H + 1 > 65535) return PICO_ERR_SIZE;
    const int P = 2 * G * d + (per_head ? 4 * H + 8 * G : H * d + H + G);
    const dim3 grid(T, per_head ? 1 : 1 + H);
    const int vec = d % 4 == 0 && d <= 128 && xc_stride % 4 == 0 && q_off % 4 == 0 && k_off % 4 == 0 && (((uintptr_t)xc | (uintptr_t)prep) & 15) == 0;
#define DP_LAUNCH(TA, PH)                                                                                                   \
    pico_launch((delta_prepare_kernel<TA, PH>), grid, dim3(128), 0, stream, xc, xc_stride, q_off, k_off, (const TA*)proj,   \
                proj_stride, b_off, (const TA*)dt, dt_stride, dt_bias, a_log, prep, P, H, G, d, q_scale, unit_eps, back, vec)
    if (dtype == PICO_F32) { if (per_head) DP_LAUNCH(float, true); else DP_LAUNCH(float, false); }
    else if (dtype == PICO_BF16) { if (per_head) DP_LAUNCH(bf16, true); else DP_LAUNCH(bf16, false); }
    else
#undef DP_LAUNCH
        return PICO_ERR_DTYPE;
    return pico_launch_status();
}

__device__ __forceinline__ void dr_cp4(float* dst, const float* src) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(src) : "memory");
}
__device__ __forceinline__ void dr_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void dr_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// prep: the rows delta_prepare_kernel wrote (q at 0, k at G d, a at 2 G d, beta and k . q after them); v float32 rows with
// head h's values at h * dv; state float32 [slots, H, dv, d]; out float32 [T, H * dv].  Grid (column tiles, H, segments).
// A column is held by LPC lanes of a warp; lane l of a column holds the rows 4 l .. 4 l + 3, 4 LPC + 4 l .., ... (RPL of
// them), so a sum over rows is RPL multiply-adds in a lane (four chains side by side) and log2(LPC) exchanges among the lanes: the
// token-to-token chain - decay, two sums, write - is what sets this kernel's time, since tokens cannot run side by side.
// PER_HEAD: the decay is one number a token; it rides behind k . q instead of d numbers of their own.
template <int RPL, int LPC, bool PER_HEAD>      // rows a lane, lanes a column (8 or 16): a block holds 16 columns in 16 * LPC threads
__global__ void __launch_bounds__(16 * LPC)
gated_delta_rule_kernel(const float* __restrict__ prep, int P, const float* __restrict__ v, int v_stride,
                        float* __restrict__ state, const int* __restrict__ seg_slots, const int* __restrict__ cu_q,
                        const int* __restrict__ positions, float* __restrict__ out, int out_stride, int H, int G, int d,
                        int dv) {
    // The kernel that follows is released at the end, not here: its blocks, resident and waiting beside this kernel's
    // few warps, made the token loop 2.7 times slower (2.0 instead of 0.76 ms for 2,048 tokens).
    pdl_wait();
    extern __shared__ __align__(16) float dsm[];
    constexpr int dp = RPL * LPC;
    constexpr int NC = 16, CPW = 32 / LPC, NTH = 16 * LPC;
    // two buffers of DR_TOK tokens: q [dp], k [dp], a [dp] (not PER_HEAD), v [NC], beta, kq, a (PER_HEAD), and what keeps a
    // token 16-byte aligned
    constexpr int VAT = (PER_HEAD ? 2 : 3) * dp, tok_floats = VAT + NC + 4, NSC = PER_HEAD ? 3 : 2;
    const int seg = blockIdx.z, h = blockIdx.y, col_base = blockIdx.x * NC;
    const int t_begin = cu_q[seg], t_end = cu_q[seg + 1];
    if (t_end <= t_begin || positions[t_begin] < 0) return;      // an empty or a padding segment
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = lane % LPC, cw = lane / LPC;                  // row lane and column of the warp
    const int col = col_base + warp * CPW + cw;
    const int hq = h / (H / G);
    float* st = state + ((size_t)seg_slots[seg] * H + h) * (size_t)dv * d;
    float S[RPL];
#pragma unroll
    for (int r = 0; r < RPL; ++r) {
        const int i = 4 * sub + 4 * LPC * (r >> 2) + (r & 3);  // four neighbouring rows at a time: one 16-byte load a token
        S[r] = (i < d && col < dv) ? st[(size_t)col * d + i] : 0.f;
    }
    const int q_at = hq * d, k_at = G * d + hq * d, a_at = 2 * G * d + (PER_HEAD ? 4 * h : h * d),
              b_at = PER_HEAD ? a_at + 1 : 2 * G * d + H * d + h, kq_at = 2 * G * d + (PER_HEAD ? 4 * H + 8 * hq : H * d + H + hq);
    auto fetch = [&](int t0, int nt, float* buf) {
        for (int idx = threadIdx.x; idx < nt * dp; idx += NTH) {
            const int tt = idx / dp, i = idx - tt * dp;
            float* dst = buf + tt * tok_floats;
            if (i < d) {
                const float* src = prep + (size_t)(t0 + tt) * P;
                dr_cp4(dst + i, src + q_at + i);
                dr_cp4(dst + dp + i, src + k_at + i);
                if (!PER_HEAD) dr_cp4(dst + 2 * dp + i, src + a_at + i);
            } else {
                dst[i] = 0.f;
                dst[dp + i] = 0.f;
                if (!PER_HEAD) dst[2 * dp + i] = 1.f;
            }
        }
        for (int idx = threadIdx.x; idx < nt * (NC + NSC); idx += NTH) {
            const int tt = idx / (NC + NSC), c = idx - tt * (NC + NSC);
            float* dst = buf + tt * tok_floats + VAT;
            const float* src = prep + (size_t)(t0 + tt) * P;
            if (c < NC) {
                if (col_base + c < dv) dr_cp4(dst + c, v + (size_t)(t0 + tt) * v_stride + (size_t)h * dv + col_base + c);
                else dst[c] = 0.f;
            } else if (c == NC) dr_cp4(dst + c, src + b_at);
            else dr_cp4(dst + c, src + (PER_HEAD && c == NC + 2 ? a_at : kq_at));
        }
        dr_commit();
    };
    float* buf0 = dsm;
    float* buf1 = dsm + DR_TOK * tok_floats;
    fetch(t_begin, min(DR_TOK, t_end - t_begin), buf0);
    int turn = 0;
    for (int t0 = t_begin; t0 < t_end; t0 += DR_TOK, turn ^= 1) {
        const int nt = min(DR_TOK, t_end - t0);
        dr_wait_all();
        __syncthreads();                    // these tokens are in; everyone is done with the other buffer
        if (t0 + DR_TOK < t_end) fetch(t0 + DR_TOK, min(DR_TOK, t_end - t0 - DR_TOK), turn ? buf0 : buf1);
        const float* buf = turn ? buf1 : buf0;
        float4 nq[RPL / 4], nk[RPL / 4], na[PER_HEAD ? 1 : RPL / 4];      // the next token's rows, asked for a token ahead
        auto rows_of = [&](int tt) {
            const float* tk = buf + tt * tok_floats + 4 * sub;
#pragma unroll
            for (int j = 0; j < RPL / 4; ++j) {
                nq[j] = *reinterpret_cast<const float4*>(tk + 4 * LPC * j);
                nk[j] = *reinterpret_cast<const float4*>(tk + dp + 4 * LPC * j);
                if (!PER_HEAD) na[j] = *reinterpret_cast<const float4*>(tk + 2 * dp + 4 * LPC * j);
            }
        };
        rows_of(0);
        for (int tt = 0; tt < nt; ++tt) {
            const float* tk = buf + tt * tok_floats;
            float p1[4] = {0.f, 0.f, 0.f, 0.f}, p2[4] = {0.f, 0.f, 0.f, 0.f};
            float kr[RPL];
            const float ah = PER_HEAD ? tk[VAT + NC + 2] : 1.0f;
#pragma unroll
            for (int j = 0; j < RPL / 4; ++j) {
                const float4 a4 = PER_HEAD ? make_float4(ah, ah, ah, ah) : na[PER_HEAD ? 0 : j];
                const float qv[4] = {nq[j].x, nq[j].y, nq[j].z, nq[j].w}, kv[4] = {nk[j].x, nk[j].y, nk[j].z, nk[j].w},
                            av[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int r = 4 * j + e;
                    const float s = S[r] * av[e];
                    kr[r] = kv[e];
                    S[r] = s;
                    p1[e] = fmaf(s, kv[e], p1[e]);
                    p2[e] = fmaf(s, qv[e], p2[e]);
                }
            }
            if (tt + 1 < nt) rows_of(tt + 1);
            float r1 = (p1[0] + p1[1]) + (p1[2] + p1[3]), r2 = (p2[0] + p2[1]) + (p2[2] + p2[3]);
#pragma unroll
            for (int o = LPC / 2; o > 0; o >>= 1) {
                r1 += __shfl_xor_sync(0xffffffffu, r1, o);
                r2 += __shfl_xor_sync(0xffffffffu, r2, o);
            }
            const float u = tk[VAT + NC] * (tk[VAT + warp * CPW + cw] - r1);
#pragma unroll
            for (int r = 0; r < RPL; ++r) S[r] = fmaf(kr[r], u, S[r]);
            if (sub == 0 && col < dv)
                out[(size_t)(t0 + tt) * out_stride + (size_t)h * dv + col] = fmaf(u, tk[VAT + NC + 1], r2);
        }
    }
    pdl_launch_dependents();
#pragma unroll
    for (int r = 0; r < RPL; ++r) {
        const int i = 4 * sub + 4 * LPC * (r >> 2) + (r & 3);
        if (i < d && col < dv) st[(size_t)col * d + i] = S[r];
    }
}

// ------------------------------------------------------------------------------------------ four tokens at a time
// With one decay a head (g_t) the memory needs to be touched only once for four tokens.  For a block of tokens 1 .. 4 that
// starts from the memory S, with r_i = S^T k_i, p_i = S^T q_i (eight sums over rows in one pass and one reduction),
// D_ij = g_(j+1) ... g_i and G_i = g_1 ... g_i:
//
//   u_i = beta_i (v_i - G_i r_i - sum_(j < i) D_ij (k_i . k_j) u_j)         o_i = G_i p_i + sum_(j <= i) D_ij (q_i . k_j) u_j
//   S  <- G_4 S + sum_j D_4j k_j u_j
//
// the same recurrence with the sums in another order; the products of decays are taken as products (none is above one, nothing is
// divided).  The dot products come from delta_prepare_kernel, the coefficients of a block from sixteen threads of this one.
// Tokens beyond the segment's end are blanks (k = q = v = 0, beta = 0, g = 1).  A block holds 16 columns as above; a lane holds the
// same rows of CPL columns (what it reads of q and k serves both) and multiplies two rows at a time (fma.rn.f32x2).
#define DB_TOK 32          // tokens fetched at a time
#define DB_COEF 48         // floats of coefficients a block of four tokens: B [4][4], E [4][4], beta G [4], beta [4], G [4], W [4]

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 db_fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 db_mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 db_pair(float lo, float hi) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float2 db_split(f32x2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;\n" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}

__device__ __forceinline__ void dr_cp16(float* dst, const float* src) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(src) : "memory");
}

// RPL rows and CPL columns a lane, LPC lanes a column (at least 8 * CPL).  vec: d, dv, both row strides and all addresses are
// multiples of 16 bytes.  (Measured for 2,048 tokens of twelve heads with d = dv = 128: 285 us with two columns a lane, 303 us with
// one, 357 us when the next block's rows are asked for while the sums are exchanged; 692 us with a pass for every token.)
template <int RPL, int LPC, int CPL>
__global__ void __launch_bounds__(16 * LPC / CPL)
gated_delta_block_kernel(const float* __restrict__ prep, int P, const float* __restrict__ v, int v_stride,
                         float* __restrict__ state, const int* __restrict__ seg_slots, const int* __restrict__ cu_q,
                         const int* __restrict__ positions, float* __restrict__ out, int out_stride, int H, int G, int d,
                         int dv, int vec, int below) {
    pdl_wait();                         // the kernel that follows is released at the end (see above)
    extern __shared__ __align__(16) float dsm[];
    constexpr int dp = RPL * LPC, NC = 16, NTH = NC / CPL * LPC, NV = 8 * CPL, VL = LPC / NV;      // VL: lanes that share a sum
    static_assert(VL >= 1, "a lane ends with one sum");
    constexpr int VAT = 2 * dp, SAT = VAT + NC, tok_floats = SAT + 12;      // q [dp], k [dp], v [NC], a, beta, -, -, eight dot products
    const int seg = blockIdx.z, h = blockIdx.y, col_base = blockIdx.x * NC;
    const int t_begin = cu_q[seg], t_end = cu_q[seg + 1];
    if (t_end <= t_begin || t_end - t_begin >= below || positions[t_begin] < 0) return;      // an empty, a long or a padding segment
    const int sub = threadIdx.x % LPC, lcol = threadIdx.x / LPC * CPL, lane0 = (threadIdx.x & 31) - sub;
    const int hq = h / (H / G);
    float* st = state + ((size_t)seg_slots[seg] * H + h) * (size_t)dv * d;
    f32x2 S[CPL][RPL / 2];
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
        const int col = col_base + lcol + c;
#pragma unroll
        for (int r = 0; r < RPL; r += 2) {
            const int i = 4 * sub + 4 * LPC * (r >> 2) + (r & 3);
            S[c][r / 2] = db_pair(col < dv && i < d ? st[(size_t)col * d + i] : 0.f, col < dv && i + 1 < d ? st[(size_t)col * d + i + 1] : 0.f);
        }
    }
    const int q_at = hq * d, k_at = G * d + hq * d, a_at = 2 * G * d + 4 * h, dot_at = 2 * G * d + 4 * H + 8 * hq;
    auto fetch = [&](int t0, float* buf) {
        const int nt = min(DB_TOK, t_end - t0), nt4 = (nt + 3) & ~3;         // whole blocks of four, blanks at the end
        if (vec) {
            constexpr int DQ = dp / 4;
            const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int idx = threadIdx.x; idx < nt4 * DQ; idx += NTH) {
                const int tt = idx / DQ, i = (idx - tt * DQ) * 4;
                float* dst = buf + tt * tok_floats + i;
                if (i < d && tt < nt) {
                    const float* src = prep + (size_t)(t0 + tt) * P + i;
                    dr_cp16(dst, src + q_at);
                    dr_cp16(dst + dp, src + k_at);
                } else {
                    *reinterpret_cast<float4*>(dst) = zero;
                    *reinterpret_cast<float4*>(dst + dp) = zero;
                }
            }
            for (int idx = threadIdx.x; idx < nt4 * 8; idx += NTH) {         // four vectors of v, one of a and beta, two of dot products
                const int tt = idx >> 3, c = idx & 7;
                float* dst = buf + tt * tok_floats + VAT + 4 * c;
                const float* src = prep + (size_t)(t0 + tt) * P;
                if (c < 4) {
                    if (tt < nt && col_base + 4 * c < dv) dr_cp16(dst, v + (size_t)(t0 + tt) * v_stride + (size_t)h * dv + col_base + 4 * c);
                    else *reinterpret_cast<float4*>(dst) = zero;
                } else if (c < 7) {
                    if (tt < nt) dr_cp16(dst, c == 4 ? src + a_at : src + dot_at + 4 * (c - 5));
                    else *reinterpret_cast<float4*>(dst) = make_float4(c == 4 ? 1.f : 0.f, 0.f, 0.f, 0.f);
                }
            }
        } else {
            for (int idx = threadIdx.x; idx < nt4 * dp; idx += NTH) {
                const int tt = idx / dp, i = idx - tt * dp;
                float* dst = buf + tt * tok_floats + i;
                if (i < d && tt < nt) {
                    const float* src = prep + (size_t)(t0 + tt) * P + i;
                    dr_cp4(dst, src + q_at);
                    dr_cp4(dst + dp, src + k_at);
                } else {
                    dst[0] = 0.f;
                    dst[dp] = 0.f;
                }
            }
            for (int idx = threadIdx.x; idx < nt4 * (NC + 12); idx += NTH) {
                const int tt = idx / (NC + 12), c = idx - tt * (NC + 12);
                float* dst = buf + tt * tok_floats + VAT + c;
                const float* src = prep + (size_t)(t0 + tt) * P;
                if (c < NC) {
                    if (tt < nt && col_base + c < dv) dr_cp4(dst, v + (size_t)(t0 + tt) * v_stride + (size_t)h * dv + col_base + c);
                    else *dst = 0.f;
                } else if (tt < nt) dr_cp4(dst, c < NC + 4 ? src + a_at + c - NC : src + dot_at + c - NC - 4);
                else *dst = c == NC ? 1.f : 0.f;
            }
        }
        dr_commit();
    };
    float* buf0 = dsm;
    float* buf1 = dsm + DB_TOK * tok_floats;
    float* coef = dsm + 2 * DB_TOK * tok_floats;
    fetch(t_begin, buf0);
    // which of the block's outputs this lane writes, if any: sum number sub / VL is p_(oi + 1) of column lcol + oc
    const int val = sub / VL, oc = val >> 3, oi = val & 3, ocol = col_base + lcol + oc;
    const bool writes = (val & 4) != 0 && sub % VL == 0 && ocol < dv;
    float* op = out + (size_t)(t_begin + oi) * out_stride + (size_t)h * dv + ocol;
    int turn = 0;
    for (int t0 = t_begin; t0 < t_end; t0 += DB_TOK, turn ^= 1) {
        const int nt = min(DB_TOK, t_end - t0), nb = (nt + 3) >> 2;
        dr_wait_all();
        __syncthreads();                    // these tokens are in; everyone is done with the other buffer and the coefficients
        if (t0 + DB_TOK < t_end) fetch(t0 + DB_TOK, turn ? buf0 : buf1);
        const float* buf = turn ? buf1 : buf0;
        for (int idx = threadIdx.x; idx < 16 * nb; idx += NTH) {             // a thread per pair (i, j) of a block's tokens
            const int b = idx >> 4, i = (idx >> 2) & 3, j = idx & 3;
            const float* tk = buf + 4 * b * tok_floats + SAT;
            const float* ti = tk + i * tok_floats;
            float* c = coef + b * DB_COEF;
            float D = 1.f, W = 1.f, Gi = 1.f;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const float g = tk[m * tok_floats];
                if (m > j && m <= i) D *= g;
                if (m > j) W *= g;
                if (m <= i) Gi *= g;
            }
            c[4 * i + j] = j < i ? ti[1] * D * ti[7 + i - j] : 0.f;          // ti[8 ..]: k_i . k_(i-1), ...
            c[16 + 4 * i + j] = j <= i ? D * ti[4 + i - j] : 0.f;            // ti[4 ..]: q_i . k_i, q_i . k_(i-1), ...
            if (i == 0) c[44 + j] = W;
            if (j == 0) {
                c[32 + i] = ti[1] * Gi;
                c[36 + i] = ti[1];
                c[40 + i] = Gi;
            }
        }
        __syncthreads();
#pragma unroll 2
        for (int b = 0; b < nb; ++b, op += (size_t)4 * out_stride) {
            const float* tk = buf + 4 * b * tok_floats;
            const float* c = coef + b * DB_COEF;
            ulonglong2 kr[4][RPL / 4], qr[4][RPL / 4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int r = 0; r < RPL / 4; ++r) {
                    const float* at = tk + i * tok_floats + 4 * sub + 4 * LPC * r;
                    qr[i][r] = *reinterpret_cast<const ulonglong2*>(at);
                    kr[i][r] = *reinterpret_cast<const ulonglong2*>(at + dp);
                }
            float s[NV];
#pragma unroll
            for (int cc = 0; cc < CPL; ++cc)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    f32x2 ar = db_mul2(S[cc][0], kr[i][0].x), ap = db_mul2(S[cc][0], qr[i][0].x);
                    ar = db_fma2(S[cc][1], kr[i][0].y, ar);
                    ap = db_fma2(S[cc][1], qr[i][0].y, ap);
#pragma unroll
                    for (int r = 1; r < RPL / 4; ++r) {
                        ar = db_fma2(S[cc][2 * r], kr[i][r].x, ar);
                        ap = db_fma2(S[cc][2 * r], qr[i][r].x, ap);
                        ar = db_fma2(S[cc][2 * r + 1], kr[i][r].y, ar);
                        ap = db_fma2(S[cc][2 * r + 1], qr[i][r].y, ap);
                    }
                    const float2 fr = db_split(ar), fp = db_split(ap);
                    s[8 * cc + i] = fr.x + fr.y;
                    s[8 * cc + 4 + i] = fp.x + fp.y;
                }
            // on their way while the sums are exchanged: the block's values and coefficients
            float vv[4][CPL];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int cc = 0; cc < CPL; ++cc) vv[i][cc] = tk[i * tok_floats + VAT + lcol + cc];
            const float4 bG = *reinterpret_cast<const float4*>(c + 32), be = *reinterpret_cast<const float4*>(c + 36),
                         W = *reinterpret_cast<const float4*>(c + 44), B1 = *reinterpret_cast<const float4*>(c + 4),
                         B2 = *reinterpret_cast<const float4*>(c + 8), B3 = *reinterpret_cast<const float4*>(c + 12),
                         E = *reinterpret_cast<const float4*>(c + 16 + 4 * oi);
            const float Gn = c[43], Go = c[40 + oi];
            // the sums over the column's lanes: each exchange halves the number of sums a lane still carries
#pragma unroll
            for (int w = NV / 2; w > 0; w >>= 1) {
                const bool up = (sub & (w * VL)) != 0;
#pragma unroll
                for (int i = 0; i < w; ++i) {
                    const float send = up ? s[i] : s[i + w], keep = up ? s[i + w] : s[i];
                    s[i] = keep + __shfl_xor_sync(0xffffffffu, send, w * VL);
                }
            }
#pragma unroll
            for (int o = VL / 2; o > 0; o >>= 1) s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
            const float bg[4] = {bG.x, bG.y, bG.z, bG.w}, bb[4] = {be.x, be.y, be.z, be.w};
            float u[CPL][4];
#pragma unroll
            for (int cc = 0; cc < CPL; ++cc) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    u[cc][i] = fmaf(-bg[i], __shfl_sync(0xffffffffu, s[0], lane0 + (8 * cc + i) * VL), bb[i] * vv[i][cc]);
                u[cc][1] = fmaf(-B1.x, u[cc][0], u[cc][1]);
                u[cc][2] = fmaf(-B2.y, u[cc][1], fmaf(-B2.x, u[cc][0], u[cc][2]));
                u[cc][3] = fmaf(-B3.z, u[cc][2], fmaf(-B3.y, u[cc][1], fmaf(-B3.x, u[cc][0], u[cc][3])));
            }
            const float wt[4] = {W.x, W.y, W.z, W.w};
            const f32x2 G2 = db_pair(Gn, Gn);
#pragma unroll
            for (int cc = 0; cc < CPL; ++cc) {
#pragma unroll
                for (int r = 0; r < RPL / 2; ++r) S[cc][r] = db_mul2(S[cc][r], G2);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float w1 = wt[i] * u[cc][i];
                    const f32x2 w2 = db_pair(w1, w1);
#pragma unroll
                    for (int r = 0; r < RPL / 4; ++r) {
                        S[cc][2 * r] = db_fma2(kr[i][r].x, w2, S[cc][2 * r]);
                        S[cc][2 * r + 1] = db_fma2(kr[i][r].y, w2, S[cc][2 * r + 1]);
                    }
                }
            }
            if (writes && t0 + 4 * b + oi < t_end) {
                float uo[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) uo[i] = CPL == 2 && oc ? u[CPL - 1][i] : u[0][i];
                *op = fmaf(E.w, uo[3], fmaf(E.z, uo[2], fmaf(E.y, uo[1], fmaf(E.x, uo[0], Go * s[0]))));
            }
        }
    }
    pdl_launch_dependents();
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
        const int col = col_base + lcol + c;
#pragma unroll
        for (int r = 0; r < RPL; r += 2) {
            const int i = 4 * sub + 4 * LPC * (r >> 2) + (r & 3);
            const float2 f = db_split(S[c][r / 2]);
            if (col < dv && i < d) st[(size_t)col * d + i] = f.x;
            if (col < dv && i + 1 < d) st[(size_t)col * d + i + 1] = f.y;
        }
    }
}

// ------------------------------------------------------------------------------------------ thirty-two tokens at a time
// The same recurrence for a whole chunk of C = 32 tokens, as products of small matrices (the chunked form of the delta rule:
// Yang, Wang, Zhang, Shen, Kim, "Parallelizing Linear Transformers with the Delta Rule over Sequence Length", with the decays of
// Yang, Kautz, Hatamizadeh, "Gated Delta Networks").  With D_ij = g_(j+1) ... g_i, G_i = g_1 ... g_i, rows k_i, q_i, v_i:
//
//   L_ij = beta_i D_ij (k_i . k_j) for j < i        M = (I + L)^-1 diag(beta)        E_ij = D_ij (q_i . k_j) for j <= i
//   U = M V - (M diag(G) K) S        S' = G_C S + K^T diag(D_Cj) U        O = diag(G) Q S + E U
//
// Only U and S' depend on the chunk before, so the work is in three kernels: M V, M diag(G) K and E for all chunks side by side;
// the chain from chunk to chunk, two products, which leaves U and every chunk's S behind; O for all chunks side by side.  All
// float32; decays are products of decays (none is above one, nothing is divided), the inverse comes from forward substitution.
// Tokens beyond a segment's end are blanks (k = q = v = 0, beta = 0, g = 1).
// The chain is bound by the instructions that its warps issue one after the other, over len / 32 dependent steps of the longest segment:
// hence the two products only (with all four in the chain 170 us for the tokens below), 16 columns a block, and four more warps that
// fetch (the loads' addresses were a quarter of the instructions).
// A layer with projections, twelve heads with d = dv = 128, 2,048 tokens in segments of 341, 682 and 1,025 / of 682 and 1,366 / in one / 1,361 in
// one: 235 / 273 / 267 / 193 us; with both products on the CUDA cores, S and all operands from shared memory, 265 / 311 / 307 / 215.
// With two tf32 numbers for a factor, which leave out a unit of its last place, 234 / 273 / 261 / 191; root mean square of S's error against
// float64, relative, without decay 3.60e-7, now 3.54e-7, on the CUDA cores 3.57e-7 (keys of one place 1.135e-7 / 1.129e-7 / 1.129e-7).
// Eight warps that multiply (one block a multiprocessor) were 5 to 20 us slower; both products on the tensor cores left S
// off by 1.1e-7 instead of 0.7e-7 where decays are strong.  The outputs in the chain's fetching warps, without a kernel of their own, lengthened
// the chain by half.
#define DC_C 32
#define DC_D 128                               // rows of S, keys padded with zeros
#define DC_LD (DC_D + 4)                       // rows that lanes read side by side, 16 bytes each
#define DC_NC 16                               // columns of S a block of the chain
#define DC_OC 128                              // columns of O a block
#define DC_COEF (DC_C * DC_D + DC_C * DC_C + 2 * DC_C)      // floats a chunk and head: M diag(G) K, E by columns, G, D_Cj

#define DC_LEAST 64                            // tokens of a segment that goes in chunks; shorter ones are pico_gated_delta_rule's

__device__ __forceinline__ int dc_chunks_of(const int* __restrict__ cu_q, int S, int seg) {
    const int len = seg < S ? cu_q[seg + 1] - cu_q[seg] : 0;
    return len >= DC_LEAST ? (len + DC_C - 1) / DC_C : 0;
}
// Which chunk of which segment number c is, found by every warp for itself; false when there are not that many, or it is padding.
__device__ __forceinline__ bool dc_find(const int* __restrict__ cu_q, const int* __restrict__ positions, int S, int c, int& t0, int& n) {
    const int lane = threadIdx.x & 31;
    for (int first = 0; first < S; first += 32) {
        const int mine = dc_chunks_of(cu_q, S, first + lane);
        int upto = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += up;
        }
        const unsigned after = __ballot_sync(0xffffffffu, c < upto);
        if (after) {
            const int l = __ffs(after) - 1, at = c - __shfl_sync(0xffffffffu, upto - mine, l), begin = cu_q[first + l];
            t0 = begin + at * DC_C;
            n = min(DC_C, cu_q[first + l + 1] - t0);
            return positions[begin] >= 0;
        }
        c -= __shfl_sync(0xffffffffu, upto, 31);
    }
    return false;
}

// Grid (chunks at most, G): block (c, g) takes the heads of query/key head g.  u0 float32 [T, H * dv]: M V.
template <bool THREE>
__global__ void __launch_bounds__(256, THREE ? 3 : 2)
delta_chunk_prepare_kernel(const float* __restrict__ prep, int P, const float* __restrict__ v, int v_stride, const int* __restrict__ cu_q,
                           const int* __restrict__ positions, int S, float* __restrict__ coef, float* __restrict__ u0, int H, int G,
                           int d, int dv, bool keep_v) {
    // (the chain's blocks, released here, would settle where the first of these end, two long segments on one multiprocessor and none on others:
    // they are released at the end; a layer of 2,048 tokens in three segments, 12 / 16 heads: 257 / 333 us, 269 / 346 the other way)
    pdl_wait();
    int t0, n;
    if (!dc_find(cu_q, positions, S, blockIdx.x, t0, n)) return;
    extern __shared__ __align__(16) float dsm[];
    float* k_s = dsm;                          // [C][LD]
    float* q_s = k_s + DC_C * DC_LD;
    const int heads = H / G, slots = min(heads, 8), vw = heads * dv;
    const int v_floats = keep_v ? DC_C * vw : 0;                              // the heads' values [C][heads * dv]
    float* kk = q_s + (THREE ? max(DC_C * DC_LD, v_floats) : DC_C * DC_LD);   // [C][C + 1]: k_i . k_j
    float* qk = kk + DC_C * (DC_C + 1);        // q_i . k_j
    float* l_s = qk + DC_C * (DC_C + 1);       // a head's L [C][C], then M by columns; one for each of the warps that take heads
    float* g_s = l_s + slots * DC_C * DC_C;    // [slots][C]: G
    float* v_s = THREE ? q_s : g_s + slots * DC_C;         // THREE: in the place of the queries, once they are done with
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = blockIdx.y;
    auto fetch_v = [&]() {                     // the heads' values, side by side in a row, on their way while M is made
        for (int idx = threadIdx.x; idx < DC_C * (vw / 4); idx += 256) {
            const int j = idx / (vw / 4), c = idx % (vw / 4) * 4;
            if (j < n) dr_cp16(v_s + j * vw + c, v + (size_t)(t0 + j) * v_stride + (size_t)g * vw + c);
            else *reinterpret_cast<float4*>(v_s + j * vw + c) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        dr_commit();
    };
    if (!THREE && keep_v) fetch_v();
    for (int idx = threadIdx.x; idx < DC_C * (DC_D / 4); idx += 256) {
        const int i = idx / (DC_D / 4), c = idx % (DC_D / 4) * 4;
        float4 k4 = make_float4(0.f, 0.f, 0.f, 0.f), q4 = k4;
        if (i < n && c < d) {
            const float* row = prep + (size_t)(t0 + i) * P + g * d + c;
            q4 = *reinterpret_cast<const float4*>(row);
            k4 = *reinterpret_cast<const float4*>(row + G * d);
        }
        *reinterpret_cast<float4*>(k_s + i * DC_LD + c) = k4;
        *reinterpret_cast<float4*>(q_s + i * DC_LD + c) = q4;
    }
    __syncthreads();
    {   // lane: token j; a warp: tokens i = 4 warp .. + 3 of both products, over even and odd places
        f32x2 sk[4], sq[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) sk[i] = sq[i] = db_pair(0.f, 0.f);
#pragma unroll 4
        for (int c = 0; c < DC_D; c += 4) {
            const ulonglong2 kj = *reinterpret_cast<const ulonglong2*>(k_s + lane * DC_LD + c);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const ulonglong2 ki = *reinterpret_cast<const ulonglong2*>(k_s + (4 * warp + i) * DC_LD + c);
                const ulonglong2 qi = *reinterpret_cast<const ulonglong2*>(q_s + (4 * warp + i) * DC_LD + c);
                sk[i] = db_fma2(ki.y, kj.y, db_fma2(ki.x, kj.x, sk[i]));
                sq[i] = db_fma2(qi.y, kj.y, db_fma2(qi.x, kj.x, sq[i]));
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 a = db_split(sk[i]), b = db_split(sq[i]);
            kk[(4 * warp + i) * (DC_C + 1) + lane] = a.x + a.y;
            qk[(4 * warp + i) * (DC_C + 1) + lane] = b.x + b.y;
        }
    }
    __syncthreads();
    if (THREE && keep_v) fetch_v();
    for (int h0 = 0; h0 < heads; h0 += 8) {    // eight heads at a time, a warp each
        if (h0 + warp < heads) {
            const int h = g * heads + h0 + warp;
            float* L = l_s + warp * DC_C * DC_C;
            // lane i: decay and beta of token i
            float a = 1.f, beta = 0.f;
            if (lane < n) {
                const float2 ab = *reinterpret_cast<const float2*>(prep + (size_t)(t0 + lane) * P + 2 * G * d + 4 * h);
                a = ab.x;
                beta = ab.y;
            }
            float* out = coef + ((size_t)blockIdx.x * H + h) * DC_COEF + DC_C * DC_D;
            // lane j: column j of L (to shared memory) and of E
            float D = 1.f, Gi = 1.f, E[DC_C];
#pragma unroll
            for (int i = 0; i < DC_C; ++i) {
                const float ai = __shfl_sync(0xffffffffu, a, i), bi = __shfl_sync(0xffffffffu, beta, i);
                if (i > lane) D *= ai;
                if (i <= lane) Gi *= ai;
                L[i * DC_C + lane] = i > lane ? bi * D * kk[i * (DC_C + 1) + lane] : 0.f;
                E[i] = i >= lane ? D * qk[i * (DC_C + 1) + lane] : 0.f;
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < DC_C; i += 4)
                *reinterpret_cast<float4*>(out + lane * DC_C + i) = make_float4(E[i], E[i + 1], E[i + 2], E[i + 3]);
            out[DC_C * DC_C + lane] = Gi;
            out[DC_C * DC_C + DC_C + lane] = D;
            g_s[warp * DC_C + lane] = Gi;
            // lane j: column j of (I + L)^-1, row after row
            float X[DC_C];
#pragma unroll
            for (int i = 0; i < DC_C; ++i) X[i] = 0.f;
#pragma unroll
            for (int i = 0; i < DC_C; ++i) {
                float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
                for (int l = 0; l < i; l += 4) {           // (a row of L is nought from its own place on)
                    const float4 m = *reinterpret_cast<const float4*>(L + i * DC_C + l);
                    s0 = fmaf(m.x, X[l], s0);
                    s1 = fmaf(m.y, X[l + 1], s1);
                    s2 = fmaf(m.z, X[l + 2], s2);
                    s3 = fmaf(m.w, X[l + 3], s3);
                }
                X[i] = (i == lane ? 1.f : 0.f) - ((s0 + s1) + (s2 + s3));
            }
            __syncwarp();                                  // L has been read: M by columns takes its place
#pragma unroll
            for (int i = 0; i < DC_C; i += 4)
                *reinterpret_cast<float4*>(L + lane * DC_C + i) = make_float4(X[i] * beta, X[i + 1] * beta, X[i + 2] * beta, X[i + 3] * beta);
        }
        dr_wait_all();
        __syncthreads();
        // M diag(G) K and M V, the heads one after the other: a thread has four columns and eight tokens i
        const int cg = DC_D / 4 + (dv + 3) / 4;
        for (int hh = 0; hh < 8 && h0 + hh < heads; ++hh) {
            const int h = g * heads + h0 + hh;
            const float* M = l_s + hh * DC_C * DC_C;
            float* mgk = coef + ((size_t)blockIdx.x * H + h) * DC_COEF;
            for (int idx = threadIdx.x; idx < 4 * cg; idx += 256) {
                const int c = idx % cg * 4, i0 = idx / cg * 8;
                const bool of_k = c < DC_D;
                float acc[8][4];
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
                const float* vc = v + (size_t)t0 * v_stride + (size_t)h * dv + (of_k ? 0 : c - DC_D);
                auto row_of = [&](int j) {
                    if (of_k) {
                        const float4 k4 = *reinterpret_cast<const float4*>(k_s + j * DC_LD + c);
                        const float gj = g_s[hh * DC_C + j];
                        return make_float4(gj * k4.x, gj * k4.y, gj * k4.z, gj * k4.w);
                    }
                    if (keep_v) return *reinterpret_cast<const float4*>(v_s + j * vw + (h0 + hh) * dv + c - DC_D);
                    return j < n ? *reinterpret_cast<const float4*>(vc + (size_t)j * v_stride) : make_float4(0.f, 0.f, 0.f, 0.f);
                };
                // M is nought above its diagonal, and those places are left out, not multiplied with: a token that holds no
                // number must not reach the tokens before it (0 * inf)
#pragma unroll 4
                for (int j = 0; j < i0; ++j) {
                    const float4 b = row_of(j);
                    float m[8];
                    *reinterpret_cast<float4*>(m) = *reinterpret_cast<const float4*>(M + j * DC_C + i0);
                    *reinterpret_cast<float4*>(m + 4) = *reinterpret_cast<const float4*>(M + j * DC_C + i0 + 4);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        acc[i][0] = fmaf(m[i], b.x, acc[i][0]);
                        acc[i][1] = fmaf(m[i], b.y, acc[i][1]);
                        acc[i][2] = fmaf(m[i], b.z, acc[i][2]);
                        acc[i][3] = fmaf(m[i], b.w, acc[i][3]);
                    }
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float4 b = row_of(i0 + j);
#pragma unroll
                    for (int i = j; i < 8; ++i) {
                        const float m = M[(i0 + j) * DC_C + i0 + i];
                        acc[i][0] = fmaf(m, b.x, acc[i][0]);
                        acc[i][1] = fmaf(m, b.y, acc[i][1]);
                        acc[i][2] = fmaf(m, b.z, acc[i][2]);
                        acc[i][3] = fmaf(m, b.w, acc[i][3]);
                    }
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 r = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
                    if (of_k) *reinterpret_cast<float4*>(mgk + (i0 + i) * DC_D + c) = r;
                    else if (i0 + i < n) *reinterpret_cast<float4*>(u0 + (size_t)(t0 + i0 + i) * H * dv + (size_t)h * dv + c - DC_D) = r;
                }
            }
        }
        __syncthreads();
    }
}

__device__ __forceinline__ void dc_mma(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// c += a b over sixteen places with both in their three parts (pico_split3), in eight products of the nine: the one of the two smallest parts is
// below 2^-30 of a b.  The tensor cores cut sums off where float32 rounds them: the large parts' products leave them after one instruction.
// The others' sums, below 2^-6 of those, are kept in two, as an instruction that adds into the registers of the one before waits 20 clocks for it.
__device__ __forceinline__ void dc_mma8(float (&c)[3][4], const uint32_t (&a)[3][4], const float2& b0, const float2& b1) {
    uint32_t b[3][2];
    pico_split3(b0.x, b0.y, b[0][0], b[1][0], b[2][0]);
    pico_split3(b1.x, b1.y, b[0][1], b[1][1], b[2][1]);
    float big[4] = {};
    dc_mma(big, a[0], b[0]);
    dc_mma(c[1], a[1], b[2]);
    dc_mma(c[2], a[2], b[1]);
    dc_mma(c[1], a[0], b[2]);
    dc_mma(c[2], a[2], b[0]);
    dc_mma(c[1], a[1], b[1]);
    dc_mma(c[2], a[1], b[0]);
    dc_mma(c[1], a[0], b[1]);
#pragma unroll
    for (int e = 0; e < 4; ++e) c[0][e] += big[e];
}
__device__ __forceinline__ void dc_sum3(float (&c)[4], const float (&p)[3][4]) {
#pragma unroll
    for (int e = 0; e < 4; ++e) c[e] = p[0][e] + (p[1][e] + p[2][e]);
}
// The numbers that a lane holds of two neighbouring results of products, rows r and r + 8 at places 2 j and 2 j + 1 of each, as the rows' operand of a
// product over those sixteen places.
__device__ __forceinline__ void dc_rows(const float (&c)[4], const float (&d)[4], uint32_t (&a)[3][4]) {
    pico_split3(c[0], c[1], a[0][0], a[1][0], a[2][0]);
    pico_split3(c[2], c[3], a[0][1], a[1][1], a[2][1]);
    pico_split3(d[0], d[1], a[0][2], a[1][2], a[2][2]);
    pico_split3(d[2], d[3], a[0][3], a[1][3], a[2][3]);
}
__device__ __forceinline__ bool dc_no_number(const float (&c)[4][4]) {
    bool no = false;
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) no |= c[t][e] != c[t][e];
    return __any_sync(0xffffffffu, no);
}

// The chain.  Grid (column tiles, H, segments), four warps and four that fetch.  A warp keeps 32 rows of the block's 16 columns of S in
// registers, as the tensor cores take an operand: with columns as the 16 rows of an instruction, (M diag(G) K) S is over the warp's own rows
// of S, which never goes through shared memory.  The warps' four parts are added through shared memory, each warp makes U for eight tokens,
// and all of them their own rows of S', in float32 on the CUDA cores.  u: M V on the way in, U on the way out; s0 float32 [chunks, H, dv
// rounded up to 4, 128]: S before each chunk, by columns.
// The product with S is eight products of bfloat16 parts that leave nothing of a factor out, sixteen terms at a time.  Where a result is no number,
// plain float32 products decide what it is (the parts of an infinity are no infinity's parts).
#define DC_LDM (DC_D + 8)                      // rows of M diag(G) K: eight read side by side, 8 bytes a lane
#define DC_LDT (DC_D + 4)                      // rows of K: pairs of rows, 4 bytes a lane
#define DC_LDU (DC_NC + 4)
#define DC_WARPS 4                             // warps that multiply; four more fetch
#define DC_ROWS (DC_D / DC_WARPS)              // rows of S a warp
__global__ void __launch_bounds__(32 * (DC_WARPS + 4), 2)
delta_chunk_kernel(const float* __restrict__ prep, int P, float* __restrict__ state, const int* __restrict__ seg_slots,
                   const int* __restrict__ cu_q, const int* __restrict__ positions, const float* __restrict__ coef, float* __restrict__ u,
                   float* __restrict__ s0, int H, int G, int d, int dv) {
    pdl_wait();                         // the kernel that follows is released at the end (see above)
    extern __shared__ __align__(16) float dsm[];
    constexpr int MG = DC_C * DC_LDT, GD = MG + DC_C * DC_LDM, UV = GD + 2 * DC_C, BUF = UV + DC_C * DC_LDU;   // a chunk: K, M diag(G) K, G, D_Cj, M V
    const int seg = blockIdx.z, h = blockIdx.y, col_base = blockIdx.x * DC_NC;
    const int t_begin = cu_q[seg], t_end = cu_q[seg + 1];
    if (t_end - t_begin < DC_LEAST || positions[t_begin] < 0) return;      // a short or a padding segment
    float* parts = dsm + 2 * BUF;              // [warp][4 tiles of tokens][lane][4]
    float* w_s = parts + DC_WARPS * 512;                 // diag(D_Cj) U [C][8][4]: columns c, c, c + 8, c + 8 (the pairs that two rows at a time want)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, hq = h / (H / G);
    int chunk = 0;
    for (int s = lane; s < seg; s += 32) chunk += dc_chunks_of(cu_q, seg, s);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) chunk += __shfl_xor_sync(0xffffffffu, chunk, o);
    auto fetch = [&](int t0, int ch, float* buf) {
        const int n = min(DC_C, t_end - t0);
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        const float* cf = coef + ((size_t)ch * H + h) * DC_COEF;
        const int tid = threadIdx.x - 32 * DC_WARPS;
#pragma unroll
        for (int idx = tid; idx < DC_C * (DC_D / 4); idx += 128) {
            const int i = idx / (DC_D / 4), c = idx % (DC_D / 4) * 4;
            float* dst = buf + i * DC_LDT + c;
            if (i < n && c < d) dr_cp16(dst, prep + (size_t)(t0 + i) * P + G * d + hq * d + c);
            else *reinterpret_cast<float4*>(dst) = zero;
            dr_cp16(buf + MG + i * DC_LDM + c, cf + i * DC_D + c);
        }
        if (tid < 2 * DC_C / 4) dr_cp16(buf + GD + 4 * tid, cf + DC_C * DC_D + DC_C * DC_C + 4 * tid);
        {
            const int i = tid / (DC_NC / 4), c = tid % (DC_NC / 4) * 4;
            float* dst = buf + UV + i * DC_LDU + c;
            if (i < n && col_base + c < dv) dr_cp16(dst, u + (size_t)(t0 + i) * H * dv + (size_t)h * dv + col_base + c);
            else *reinterpret_cast<float4*>(dst) = zero;
        }
        dr_commit();
    };
    if (warp >= DC_WARPS) {
        // the warps that fetch: a chunk ahead of the others
        int turn = 0;
        fetch(t_begin, chunk, dsm);
        for (int t0 = t_begin; t0 < t_end; t0 += DC_C, turn ^= 1, ++chunk) {
            dr_wait_all();
            __syncthreads();                   // the chunk is in, everyone is done with the other buffer
            if (t0 + DC_C < t_end) fetch(t0 + DC_C, chunk + 1, dsm + (turn ? 0 : BUF));
        }
        return;
    }
    float* st = state + ((size_t)seg_slots[seg] * H + h) * (size_t)dv * d;
    const int r = lane >> 2, j = lane & 3, row0 = DC_ROWS * warp + 2 * j;       // this lane: columns r and r + 8, rows row0 + 8 nt and the next
    float S[DC_ROWS / 8][4];
#pragma unroll
    for (int nt = 0; nt < DC_ROWS / 8; ++nt)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int col = col_base + r + 8 * c;
            float2 x = make_float2(0.f, 0.f);
            if (col < dv && row0 + 8 * nt < d) x = *reinterpret_cast<const float2*>(st + (size_t)col * d + row0 + 8 * nt);
            S[nt][2 * c] = x.x;
            S[nt][2 * c + 1] = x.y;
        }
    int turn = 0;
    for (int t0 = t_begin; t0 < t_end; t0 += DC_C, turn ^= 1, ++chunk) {
        __syncthreads();                       // the chunk is in, everyone is done with the other buffer
        const float* buf = dsm + (turn ? BUF : 0);
        const float *k_s = buf + row0, *m_s = buf + MG + row0, *Gd = buf + GD, *Wd = Gd + DC_C, *u_s = buf + UV;
        // S before this chunk, for the outputs
        float* s_out = s0 + (((size_t)chunk * H + h) * ((dv + 3) / 4 * 4) + col_base + r) * DC_D + row0;
#pragma unroll
        for (int nt = 0; nt < DC_ROWS / 8; ++nt)
#pragma unroll
            for (int c = 0; c < 2; ++c)
                if (col_base + r + 8 * c < dv) *reinterpret_cast<float2*>(s_out + c * 8 * DC_D + 8 * nt) = make_float2(S[nt][2 * c], S[nt][2 * c + 1]);
        float x[4][4], x3[4][3][4] = {};       // [tile of tokens]: columns r, r + 8, tokens 8 tt + 2 j and the next
#pragma unroll
        for (int nt = 0; nt < DC_ROWS / 8; nt += 2) {
            uint32_t a[3][4];
            dc_rows(S[nt], S[nt + 1], a);
#pragma unroll
            for (int tt = 0; tt < 4; ++tt) {
                const float* b = m_s + (8 * tt + r) * DC_LDM + 8 * nt;
                dc_mma8(x3[tt], a, *reinterpret_cast<const float2*>(b), *reinterpret_cast<const float2*>(b + 8));
            }
        }
#pragma unroll
        for (int tt = 0; tt < 4; ++tt) dc_sum3(x[tt], x3[tt]);
        if (dc_no_number(x)) {
#pragma unroll
            for (int t = 0; t < DC_C; ++t) {
                float p0 = 0.f, p1 = 0.f;
#pragma unroll
                for (int nt = 0; nt < DC_ROWS / 8; ++nt) {
                    const float2 b = *reinterpret_cast<const float2*>(m_s + t * DC_LDM + 8 * nt);
                    p0 = fmaf(S[nt][1], b.y, fmaf(S[nt][0], b.x, p0));
                    p1 = fmaf(S[nt][3], b.y, fmaf(S[nt][2], b.x, p1));
                }
#pragma unroll
                for (int o = 1; o < 4; o <<= 1) {
                    p0 += __shfl_xor_sync(0xffffffffu, p0, o);
                    p1 += __shfl_xor_sync(0xffffffffu, p1, o);
                }
                if (j == (t & 7) >> 1) {
                    if (x[t >> 3][t & 1] != x[t >> 3][t & 1]) x[t >> 3][t & 1] = p0;
                    if (x[t >> 3][2 + (t & 1)] != x[t >> 3][2 + (t & 1)]) x[t >> 3][2 + (t & 1)] = p1;
                }
            }
        }
        float* mine = parts + lane * 4;
#pragma unroll
        for (int tt = 0; tt < 4; ++tt) *reinterpret_cast<float4*>(mine + (warp * 4 + tt) * 128) = make_float4(x[tt][0], x[tt][1], x[tt][2], x[tt][3]);
        asm volatile("bar.sync 1, %0;\n" ::"n"(32 * DC_WARPS) : "memory");
        static_assert(DC_WARPS == DC_C / 8, "a warp makes U and diag(D_Cj) U of eight tokens");
        {
            float4 a[DC_WARPS];
#pragma unroll
            for (int p = 0; p < DC_WARPS; ++p) a[p] = *reinterpret_cast<const float4*>(mine + (p * 4 + warp) * 128);
#pragma unroll
            for (int o = DC_WARPS / 2; o > 0; o >>= 1)
#pragma unroll
                for (int p = 0; p < o; ++p) a[p] = make_float4(a[p].x + a[p + o].x, a[p].y + a[p + o].y, a[p].z + a[p + o].z, a[p].w + a[p + o].w);
            const float* mv = u_s + (8 * warp + 2 * j) * DC_LDU + r;
            const float2 wj = *reinterpret_cast<const float2*>(Wd + 8 * warp + 2 * j);
            const float u0 = mv[0] - a[0].x, u1 = mv[DC_LDU] - a[0].y, u2 = mv[8] - a[0].z, u3 = mv[DC_LDU + 8] - a[0].w;
            float* wo = w_s + ((8 * warp + 2 * j) * 8 + r) * 4;
            *reinterpret_cast<float4*>(wo) = make_float4(wj.x * u0, wj.x * u0, wj.x * u2, wj.x * u2);
            *reinterpret_cast<float4*>(wo + 32) = make_float4(wj.y * u1, wj.y * u1, wj.y * u3, wj.y * u3);
            const int i = t0 + 8 * warp + 2 * j;
            float* uo = u + (size_t)i * H * dv + (size_t)h * dv + col_base + r;
            const bool c0 = col_base + r < dv, c1 = col_base + r + 8 < dv;
            if (i < t_end && c0) uo[0] = u0;
            if (i + 1 < t_end && c0) uo[(size_t)H * dv] = u1;
            if (i < t_end && c1) uo[8] = u2;
            if (i + 1 < t_end && c1) uo[(size_t)H * dv + 8] = u3;
        }
        asm volatile("bar.sync 1, %0;\n" ::"n"(32 * DC_WARPS) : "memory");
        const float gc = Gd[DC_C - 1];
        const f32x2 g2 = db_pair(gc, gc);
        f32x2 s2[DC_ROWS / 8][2];
#pragma unroll
        for (int nt = 0; nt < DC_ROWS / 8; ++nt)
#pragma unroll
            for (int c = 0; c < 2; ++c) s2[nt][c] = db_mul2(db_pair(S[nt][2 * c], S[nt][2 * c + 1]), g2);
#pragma unroll
        for (int t = 0; t < DC_C; ++t) {
            const ulonglong2 w2 = *reinterpret_cast<const ulonglong2*>(w_s + (t * 8 + r) * 4);
#pragma unroll
            for (int nt = 0; nt < DC_ROWS / 8; ++nt) {
                const f32x2 k = *reinterpret_cast<const f32x2*>(k_s + t * DC_LDT + 8 * nt);
                s2[nt][0] = db_fma2(k, w2.x, s2[nt][0]);
                s2[nt][1] = db_fma2(k, w2.y, s2[nt][1]);
            }
        }
#pragma unroll
        for (int nt = 0; nt < DC_ROWS / 8; ++nt)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const float2 f = db_split(s2[nt][c]);
                S[nt][2 * c] = f.x;
                S[nt][2 * c + 1] = f.y;
            }
    }
    pdl_launch_dependents();
#pragma unroll
    for (int nt = 0; nt < DC_ROWS / 8; ++nt)
#pragma unroll
        for (int c = 0; c < 2; ++c)
            if (col_base + r + 8 * c < dv && row0 + 8 * nt < d)
                *reinterpret_cast<float2*>(st + (size_t)(col_base + r + 8 * c) * d + row0 + 8 * nt) = make_float2(S[nt][2 * c], S[nt][2 * c + 1]);
}

// The outputs.  Grid (chunks at most, H, tiles of 128 columns): O = diag(G) Q S + E U; a thread has tokens 8 ty .. + 7 and columns tx, tx +
// 32, ..
__global__ void __launch_bounds__(128)
delta_chunk_out_kernel(const float* __restrict__ prep, int P, const int* __restrict__ cu_q, const int* __restrict__ positions, int S,
                       const float* __restrict__ coef, const float* __restrict__ u, const float* __restrict__ s0, float* __restrict__ out,
                       int out_stride, int H, int G, int d, int dv) {
    pdl_launch_dependents();
    pdl_wait();
    int t0, n;
    if (!dc_find(cu_q, positions, S, blockIdx.x, t0, n)) return;
    extern __shared__ __align__(16) float dsm[];
    float* s_s = dsm;                          // [OC][LD]: S by columns
    float* q_s = s_s + DC_OC * DC_LD;          // [C][LD]: Q
    float* u_s = q_s + DC_C * DC_LD;           // [C][OC]
    float* e_s = u_s + DC_C * DC_OC;           // [C][C]: E by columns, then G
    const int h = blockIdx.y, hq = h / (H / G), col_base = blockIdx.z * DC_OC, cols = min(DC_OC, dv - col_base);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float* sc = s0 + (((size_t)blockIdx.x * H + h) * ((dv + 3) / 4 * 4) + col_base) * DC_D;
    const float* cf = coef + ((size_t)blockIdx.x * H + h) * DC_COEF + DC_C * DC_D;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int idx = threadIdx.x; idx < DC_OC * (DC_D / 4); idx += 128) {
        const int c = idx / (DC_D / 4), i = idx % (DC_D / 4) * 4;
        float* dst = s_s + c * DC_LD + i;
        if (c < cols) dr_cp16(dst, sc + (size_t)c * DC_D + i);
        else *reinterpret_cast<float4*>(dst) = zero;
    }
    for (int idx = threadIdx.x; idx < DC_C * (DC_D / 4); idx += 128) {
        const int i = idx / (DC_D / 4), c = idx % (DC_D / 4) * 4;
        float* dst = q_s + i * DC_LD + c;
        if (i < n && c < d) dr_cp16(dst, prep + (size_t)(t0 + i) * P + hq * d + c);
        else *reinterpret_cast<float4*>(dst) = zero;
        dst = u_s + i * DC_OC + c;
        if (i < n && c < cols) dr_cp16(dst, u + (size_t)(t0 + i) * H * dv + (size_t)h * dv + col_base + c);
        else *reinterpret_cast<float4*>(dst) = zero;
    }
    for (int idx = threadIdx.x; idx < (DC_C * DC_C + DC_C) / 4; idx += 128) dr_cp16(e_s + 4 * idx, cf + 4 * idx);
    dr_commit();
    dr_wait_all();
    __syncthreads();
    // warp: tokens 8 warp .. + 7, lane: columns lane, lane + 32, ..
    f32x2 acc[8][4];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[r][e] = db_pair(0.f, 0.f);
    const float* row = q_s + 8 * warp * DC_LD;
    const float* col = s_s + lane * DC_LD;
#pragma unroll 2
    for (int c = 0; c < DC_D; c += 4) {
        ulonglong2 b[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) b[e] = *reinterpret_cast<const ulonglong2*>(col + 32 * e * DC_LD + c);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(row + r * DC_LD + c);
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[r][e] = db_fma2(a.y, b[e].y, db_fma2(a.x, b[e].x, acc[r][e]));
        }
    }
    float o[8][4];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const float gi = e_s[DC_C * DC_C + 8 * warp + r];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = db_split(acc[r][e]);
            o[r][e] = gi * (f.x + f.y);
        }
    }
    // E is nought beyond a token's own place, and those places are left out (as above)
    auto add_u = [&](int j, auto from) {
        float ev[8], uv[4];
        *reinterpret_cast<float4*>(ev) = *reinterpret_cast<const float4*>(e_s + j * DC_C + 8 * warp);
        *reinterpret_cast<float4*>(ev + 4) = *reinterpret_cast<const float4*>(e_s + j * DC_C + 8 * warp + 4);
#pragma unroll
        for (int e = 0; e < 4; ++e) uv[e] = u_s[j * DC_OC + lane + 32 * e];
#pragma unroll
        for (int r = 0; r < 8; ++r)
            if (r >= from)
#pragma unroll
                for (int e = 0; e < 4; ++e) o[r][e] = fmaf(ev[r], uv[e], o[r][e]);
    };
    for (int j = 0; j < 8 * warp; ++j) add_u(j, 0);
#pragma unroll
    for (int j = 0; j < 8; ++j) add_u(8 * warp + j, j);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int i = 8 * warp + r;
        if (i >= n) break;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int c = lane + 32 * e;
            if (c < cols) out[(size_t)(t0 + i) * out_stride + (size_t)h * dv + col_base + c] = o[r][e];
        }
    }
}

// Floats of scratch that pico_gated_delta_chunks needs for T tokens in S segments: coefficients, U, S before every chunk.
static long long dc_chunks(int T, int S) { return (long long)T / DC_C + (S < T / DC_LEAST ? S : T / DC_LEAST) + 1; }
PICO_API long long pico_gated_delta_chunk_floats(int T, int S, int H, int dv) {
    return dc_chunks(T, S) * H * (DC_COEF + (long long)((dv + 3) / 4 * 4) * DC_D) + (long long)T * H * dv;
}

// The recurrence with one decay a head in chunks for the segments of DC_LEAST tokens and more; T: tokens of all segments.  d up to 128; d, dv, the strides multiples of 4, all
// addresses of 16 bytes: anything else is refused.
PICO_API int pico_gated_delta_chunks(const float* prep, const float* v, int v_stride, float* state, const int* seg_slots,
                                     const int* cu_q, const int* positions, float* out, int out_stride, int T, int S, int H, int G,
                                     int d, int dv, float* scratch, cudaStream_t stream) {
    if (S <= 0 || T <= 0) return 0;
    if (H < 1 || G < 1 || H % G || d < 4 || d > DC_D || dv < 4) return PICO_ERR_SIZE;
    if (d % 4 || dv % 4 || v_stride % 4 || out_stride % 4 || (((uintptr_t)prep | (uintptr_t)v | (uintptr_t)state | (uintptr_t)out | (uintptr_t)scratch) & 15))
        return PICO_ERR_ALIGN;
    if (S > 65535 || H > 65535 || (dv + DC_OC - 1) / DC_OC > 65535 || dc_chunks(T, S) > 0x7fffffffLL) return PICO_ERR_SIZE;
    const int P = 2 * G * d + 4 * H + 8 * G, chunks = (int)dc_chunks(T, S);
    float* coef = scratch;
    float* s0 = coef + (size_t)chunks * H * DC_COEF;
    float* u = s0 + (size_t)chunks * H * ((dv + 3) / 4 * 4) * DC_D;
    const int slots = H / G < 8 ? H / G : 8;
    const bool keep_v = (size_t)DC_C * (H / G) * dv * sizeof(float) <= 32 * 1024;
    // Two blocks a multiprocessor; three, with fewer registers (80 a thread, 44 bytes of them stored and 56 loaded again) and the values in the place of the
    // queries, where that saves a round of them.  The blocks that have a chunk are counted as if every segment's last chunk were half full; the grid
    // has up to one a segment more, which leave at once: 2 % more blocks were enough for a round that there was not (8 key heads, 1,100 tokens in three
    // segments, 288 at work and 304 in the grid: a layer 189 us, three a multiprocessor 197).  us of a layer, two / three, by the grid: 6 key heads, 324
    // blocks 209 / 202, 408 247 / 236, 432 252 / 242, 624 357 / 349, 870 549 / 542; 8 key heads, 368 243 / 231, 672 404 / 395, 912 539 / 529.
    const long long two = 2LL * pico_num_sms(), three = 3LL * pico_num_sms();
    const long long blocks = (long long)G * (2 * (T / DC_C) + (S < T / DC_LEAST ? S : T / DC_LEAST)) / 2;
    const long long v_floats = keep_v ? (long long)DC_C * (H / G) * dv : 0, q_floats = DC_C * DC_LD;
    const long long other = DC_C * DC_LD + 2 * DC_C * (DC_C + 1) + slots * (DC_C * DC_C + DC_C), shared = other + (v_floats > q_floats ? v_floats : q_floats);
    const bool crowded = keep_v && 3 * (shared * (long long)sizeof(float) + 1024) <= 228 * 1024 &&
                         (blocks + three - 1) / three < (blocks + two - 1) / two;
    const size_t sm1 = (size_t)(crowded ? shared : other + q_floats + v_floats) * sizeof(float);
    auto prepare = crowded ? delta_chunk_prepare_kernel<true> : delta_chunk_prepare_kernel<false>;
    cudaFuncSetAttribute(prepare, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm1);
    pico_launch(prepare, dim3(chunks, G), dim3(256), sm1, stream, prep, P, v, v_stride, cu_q, positions, S, coef, u, H, G, d, dv, keep_v);
    const dim3 grid((dv + DC_NC - 1) / DC_NC, H, S);
    size_t sm2 = (size_t)(2 * (DC_C * DC_LDT + DC_C * DC_LDM + 2 * DC_C + DC_C * DC_LDU) + DC_WARPS * 512 + DC_C * 32) * sizeof(float);
    // (one block a multiprocessor where there are enough of them: see pico_gated_delta_rule)
    if ((long long)grid.x * grid.y * grid.z <= pico_num_sms() && sm2 < 116 * 1024) sm2 = 116 * 1024;
    cudaFuncSetAttribute(delta_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm2);
    pico_launch(delta_chunk_kernel, grid, dim3(32 * (DC_WARPS + 4)), sm2, stream, prep, P, state, seg_slots, cu_q, positions, (const float*)coef, u, s0, H, G, d, dv);
    const size_t sm3 = (size_t)(DC_OC * DC_LD + DC_C * DC_LD + DC_C * DC_OC + DC_C * DC_C + DC_C) * sizeof(float);
    cudaFuncSetAttribute(delta_chunk_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm3);
    pico_launch(delta_chunk_out_kernel, dim3(chunks, H, (dv + DC_OC - 1) / DC_OC), dim3(128), sm3, stream, prep, P, cu_q, positions, S,
                (const float*)coef, (const float*)u, (const float*)s0, out, out_stride, H, G, d, dv);
    return pico_launch_status();
}

// below > 0 (with blocked): only the segments of fewer tokens.
PICO_API int pico_gated_delta_rule(const float* prep, const float* v, int v_stride, float* state, const int* seg_slots,
                                   const int* cu_q, const int* positions, float* out, int out_stride, int S, int H, int G,
                                   int d, int dv, int per_head, int blocked, int below, cudaStream_t stream) {
    if (S <= 0) return 0;
    if (H < 1 || G < 1 || H % G || d < 1 || d > 256 || dv < 1 || (below > 0 && !(per_head && blocked))) return PICO_ERR_SIZE;
    const int P = 2 * G * d + (per_head ? 4 * H + 8 * G : H * d + H + G);
    const dim3 grid((dv + 15) / 16, H, S);
    if (grid.z > 65535 || grid.y > 65535) return PICO_ERR_SIZE;
    // A grid that fits on the device one block to a multiprocessor asks for more shared memory than half of one, so that
    // no two blocks share a multiprocessor: released early behind a kernel that is still draining, the blocks of a
    // 2,048-token prompt landed four to a multiprocessor on the first ones that had room and took 1.5 ms instead of 0.8.
    const bool alone = (long long)grid.x * grid.y * grid.z <= pico_num_sms();
#define DR_LAUNCH_AS(N, L, PH)                                                                                              \
    do {                                                                                                                    \
        size_t smem = (size_t)2 * DR_TOK * ((PH ? 2 : 3) * N * L + 16 + 4) * sizeof(float);                                 \
        if (alone && smem < 116 * 1024) smem = 116 * 1024;                                                                  \
        if (smem > 48 * 1024)                                                                                               \
            cudaFuncSetAttribute(gated_delta_rule_kernel<N, L, PH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);  \
        pico_launch((gated_delta_rule_kernel<N, L, PH>), grid, dim3(16 * L), smem, stream, prep, P, v, v_stride, state,     \
                    seg_slots, cu_q, positions, out, out_stride, H, G, d, dv);                                              \
    } while (0)
#define DR_LAUNCH(N, L)                                                                                                     \
    do {                                                                                                                    \
        if (per_head) DR_LAUNCH_AS(N, L, true);                                                                             \
        else DR_LAUNCH_AS(N, L, false);                                                                                     \
    } while (0)
#define DB_LAUNCH(N, L, C)                                                                                             \
    do {                                                                                                                    \
        size_t smem = (size_t)(2 * DB_TOK * (2 * N * L + 16 + 12) + DB_TOK / 4 * DB_COEF) * sizeof(float);                  \
        if (alone && smem < 116 * 1024) smem = 116 * 1024;                                                                  \
        if (smem > 48 * 1024)                                                                                               \
            cudaFuncSetAttribute(gated_delta_block_kernel<N, L, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
        pico_launch((gated_delta_block_kernel<N, L, C>), grid, dim3(16 * L / C), smem, stream, prep, P, v, v_stride, state, \
                    seg_slots, cu_q, positions, out, out_stride, H, G, d, dv, vec, below > 0 ? below : 0x7fffffff);                                         \
    } while (0)
    if (per_head && blocked) {
        const int vec = d % 4 == 0 && dv % 4 == 0 && v_stride % 4 == 0 && (((uintptr_t)prep | (uintptr_t)v) & 15) == 0;
        if (d <= 32) DB_LAUNCH(4, 8, 1);
        else if (d <= 64) DB_LAUNCH(4, 16, 2);
        else if (d <= 128) DB_LAUNCH(8, 16, 2);
        else DB_LAUNCH(16, 16, 2);
        return pico_launch_status();
    }
#undef DB_LAUNCH
    // keys of up to 32: eight lanes a column (four warps a block); longer keys: sixteen (eight warps), so that a
    // multiprocessor's four schedulers each have two warps to choose from
    if (d <= 32) DR_LAUNCH(4, 8);
    else if (d <= 64) DR_LAUNCH(4, 16);
    else if (d <= 128) DR_LAUNCH(8, 16);
    else DR_LAUNCH(16, 16);
#undef DR_LAUNCH
#undef DR_LAUNCH_AS
    return pico_launch_status();
}
