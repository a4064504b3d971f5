// A recurrent mixer that corrects its state by the error of its own prediction (the gated delta rule), with a
// decay per head and key channel (or one per head: `decay_per_head`, the raw decay inputs are then rows of
// [heads] and dt_bias has one entry a head; g_t[i] is the same for every key channel i):
//
//   S_t   = diag(g_t) S_(t-1)                         S: [key channel, value channel] per head, 32-bit, starts at 0
//   u_t   = beta_t (v_t - S_t^T k_t)
//   S_t  += k_t u_t^T
//   o_t   = S_t^T q_t                                  (the read-out sees the token's own write)
//         = (diag(g_t) S_(t-1))^T q_t + u_t (k_t . q_t)      the form the kernel uses: both sums over key channels in one walk
//
// with q and k made unit vectors per head on the way in (x / sqrt(sum x^2 + unit_eps), q also times q_scale),
// beta_t = sigmoid(raw beta) and g_t[i] = exp(-exp(A_log_h) * softplus(a_t[i] + dt_bias[i])).  Everything behind
// the projections is 32-bit.  The state lives in the request's state slot and is carried from step to step; a
// fresh request starts from zeros.  Steps of few tokens walk a sequence token by token; bfloat16 prompts are taken a chunk
// of tokens at a time, whose sums are formed in another order, as right.
//
// One block per (sequence, head, share of the value columns).  Value column j is held by PARTS neighbouring
// threads, each with NP / PARTS key channels of column j in registers; the two sums over key channels of a
// token (the prediction and the read-out) are joined over those threads by shuffles.  For keys of 128 and more a
// thread holds the same key channels of two neighbouring columns: what it reads of the staged q, k and g serves
// both, and a head needs half the blocks.
#include "chunk_scan.cuh"
#include "common.cuh"

namespace ff {

__device__ __forceinline__ float dr_softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }

struct DeltaArgs {
    const void* q; int q_stride, q_off;          // rows of [groups, N]
    const void* k; int k_stride, k_off;
    const void* v; int v_stride, v_off;          // rows of [heads, V]
    const void* beta; int beta_stride, beta_off; // raw, rows of [heads]
    const float* a; int a_stride, a_off;         // raw decay inputs, rows of [heads, N], 32-bit
    const float* dt_bias;                        // [heads * N]
    const float* a_log;                          // [heads]
    int heads_per_group;
    float q_scale, unit_eps;
    int decay_per_head;                          // 1: `a` rows of [heads], dt_bias [heads]
};

constexpr int DR_CHUNK = 8;
constexpr int DR_AHEAD = 2;     // elements of a chunk's inputs a thread may hold for the chunk to come
constexpr int DR_MAX_THREADS = 512;

struct DeltaPlan { int NP, PARTS, VJ, vsplit, Vb, threads; };
static inline bool delta_plan(int N, int V, DeltaPlan* p) {
    if (N <= 0 || N > 256 || V <= 0 || V > 256) return false;
    p->NP = N <= 16 ? 16 : (N <= 32 ? 32 : (N <= 64 ? 64 : (N <= 128 ? 128 : 256)));
    p->PARTS = p->NP >= 128 ? 16 : (p->NP >= 32 ? 8 : 4);
    p->VJ = p->NP >= 128 ? 2 : 1;              // value columns a thread: long keys share their staged q, k, g over two
    const int max_cols = DR_MAX_THREADS / p->PARTS * p->VJ;
    p->vsplit = (V + max_cols - 1) / max_cols;
    p->Vb = (V + p->vsplit - 1) / p->vsplit;
    p->threads = (((p->Vb + p->VJ - 1) / p->VJ * p->PARTS + 31) / 32) * 32;
    return true;
}

// SOME: sequences of max_len tokens and more go by chunks (else every sequence is this kernel's).
template <typename T, int NP, int PARTS, int VJ, bool SOME>
__global__ void __launch_bounds__(DR_MAX_THREADS) delta_rule_scan_kernel(
    DeltaArgs A, float* __restrict__ state, size_t state_stride, int state_off, const int* __restrict__ cu_q,
    const int* __restrict__ state_slots, const int* __restrict__ seq_fresh, float* __restrict__ o /*[T, heads*V]*/,
    int heads, int N, int V, int Vb, int max_len) {
    pdl_prologue();
    constexpr int KP = NP / PARTS;
    constexpr int CH = NP >= 256 ? DR_CHUNK : 2 * DR_CHUNK;     // tokens staged at a time (shared memory bounds the longest keys)
    constexpr int AH = NP >= 256 ? DR_AHEAD : 2 * DR_AHEAD;
    static_assert(KP % 4 == 0, "a thread reads its key channels four at a time");
    __shared__ __align__(16) float s_q[CH][NP], s_k[CH][NP], s_g[CH][NP];
    __shared__ float s_v[CH][128];
    __shared__ float s_b[CH], s_kq[CH];
    const int s = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, nthr = blockDim.x;
    const int lane = tid & 31, warp = tid >> 5, nwarps = nthr >> 5;
    const int jl = tid / PARTS, part = tid % PARTS;
    const int j0 = blockIdx.z * Vb;                       // the block's first column; the thread's are j0 + jl * VJ + x
    const int t0 = cu_q[s], t1s = cu_q[s + 1];
    const bool mine = !SOME || t1s - t0 < max_len;                 // a sequence that goes by chunks is empty here (as in ssm.cu)
    const int t1 = mine ? t1s : t0;
    bool live[VJ];
#pragma unroll
    for (int x = 0; x < VJ; ++x) live[x] = jl * VJ + x < Vb && j0 + jl * VJ + x < V;
    const bool fresh = seq_fresh[s] != 0;
    // a head's state lies in the slot as [V][NP], whatever kernel wrote it
    float* S_g = state + (size_t)state_slots[s] * state_stride + state_off + (size_t)h * V * NP;
    const bool vec = ((uintptr_t)S_g & 15) == 0;
    float S[VJ][KP];
#pragma unroll
    for (int x = 0; x < VJ; ++x) {
#pragma unroll
        for (int i = 0; i < KP; i += 4) {
            // thread `part` holds key channels 4 PARTS m + 4 part + e (m = i / 4, e < 4)
            const float* p = S_g + (size_t)(j0 + jl * VJ + x) * NP + i * PARTS + part * 4;
            float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!fresh && live[x]) r = vec ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
            S[x][i] = r.x; S[x][i + 1] = r.y; S[x][i + 2] = r.z; S[x][i + 3] = r.w;
        }
    }
    const int group = h / A.heads_per_group;
    const T* qp = pdl_fresh((const T*)A.q) + A.q_off + (size_t)group * N;
    const T* kp = pdl_fresh((const T*)A.k) + A.k_off + (size_t)group * N;
    const T* vp = pdl_fresh((const T*)A.v) + A.v_off + (size_t)h * V + j0;
    const T* bp = pdl_fresh((const T*)A.beta) + A.beta_off + h;
    const int an = A.decay_per_head ? 0 : 1;            // 0: every key channel reads the head's one decay input
    const float* ap = pdl_fresh(A.a) + A.a_off + (A.decay_per_head ? (size_t)h : (size_t)h * N);
    const float* dtb = A.dt_bias + (A.decay_per_head ? (size_t)h : (size_t)h * N);
    const int cols = min(Vb, V - j0);
    const float rate = expf(A.a_log[h]);
    // Where a chunk's inputs are at most AH elements a thread, the next chunk's are asked for (into registers)
    // before the current chunk's tokens are walked, so that their way from memory passes under the recurrence.
    const bool ahead = CH * NP <= AH * nthr && CH * cols <= AH * nthr;
    T nq[AH], nk[AH], nv[AH], nb = from_float<T>(0.f);
    float na[AH];
    auto ask = [&](int c0) {
        const int n = min(CH, t1 - c0);
#pragma unroll
        for (int r = 0; r < AH; ++r) {
            const int idx = tid + r * nthr, c = idx / NP, i = idx - c * NP;
            const bool in = idx < CH * NP && c < n && i < N;
            nq[r] = in ? qp[(size_t)(c0 + c) * A.q_stride + i] : from_float<T>(0.f);
            nk[r] = in ? kp[(size_t)(c0 + c) * A.k_stride + i] : from_float<T>(0.f);
            na[r] = in ? ap[(size_t)(c0 + c) * A.a_stride + i * an] : 0.f;
            const int cv = idx / cols, jj = idx - cv * cols;
            nv[r] = (idx < CH * cols && cv < n) ? vp[(size_t)(c0 + cv) * A.v_stride + jj] : from_float<T>(0.f);
        }
        nb = tid < n ? bp[(size_t)(c0 + tid) * A.beta_stride] : from_float<T>(0.f);
    };
    if (ahead && t0 < t1) ask(t0);
    for (int c0 = t0; c0 < t1; c0 += CH) {
        const int n = min(CH, t1 - c0);
        __syncthreads();
        // staging: the chunk's q, k (raw), decays, v and beta in 32-bit
        if (ahead) {
#pragma unroll
            for (int r = 0; r < AH; ++r) {
                const int idx = tid + r * nthr, c = idx / NP, i = idx - c * NP;
                if (idx < CH * NP) {
                    const bool in = c < n && i < N;
                    s_q[c][i] = to_float(nq[r]);
                    s_k[c][i] = to_float(nk[r]);
                    s_g[c][i] = in ? expf(-rate * dr_softplus(na[r] + dtb[i * an])) : 0.f;
                }
                if (idx < CH * cols) s_v[idx / cols][idx % cols] = to_float(nv[r]);
            }
            if (tid < CH) s_b[tid] = tid < n ? 1.0f / (1.0f + expf(-to_float(nb))) : 0.f;
            if (c0 + CH < t1) ask(c0 + CH);
        } else {
        for (int idx = tid; idx < CH * NP; idx += nthr) {
            const int c = idx / NP, i = idx - c * NP;
            float qv = 0.f, kv = 0.f, gv = 0.f;
            if (c < n && i < N) {
                qv = to_float(qp[(size_t)(c0 + c) * A.q_stride + i]);
                kv = to_float(kp[(size_t)(c0 + c) * A.k_stride + i]);
                gv = expf(-rate * dr_softplus(ap[(size_t)(c0 + c) * A.a_stride + i * an] + dtb[i * an]));
            }
            s_q[c][i] = qv;
            s_k[c][i] = kv;
            s_g[c][i] = gv;
        }
        for (int idx = tid; idx < CH * cols; idx += nthr) {
            const int c = idx / cols, jj = idx - c * cols;
            s_v[c][jj] = c < n ? to_float(vp[(size_t)(c0 + c) * A.v_stride + jj]) : 0.f;
        }
        if (tid < CH)
            s_b[tid] = tid < n ? 1.0f / (1.0f + expf(-to_float(bp[(size_t)(c0 + tid) * A.beta_stride]))) : 0.f;
        }
        __syncthreads();
        // unit vectors: a warp per token
        for (int c = warp; c < n; c += nwarps) {
            float sq = 0.f, sk = 0.f, kq = 0.f;
            for (int i = lane; i < NP; i += 32) {
                sq += s_q[c][i] * s_q[c][i];
                sk += s_k[c][i] * s_k[c][i];
                kq += s_q[c][i] * s_k[c][i];
            }
            sq = warp_sum(sq);
            sk = warp_sum(sk);
            kq = warp_sum(kq);
            const float fq = A.q_scale / sqrtf(sq + A.unit_eps), fk = 1.0f / sqrtf(sk + A.unit_eps);
            for (int i = lane; i < NP; i += 32) { s_q[c][i] *= fq; s_k[c][i] *= fk; }
            if (lane == 0) s_kq[c] = kq * fq * fk;
        }
        __syncthreads();
#pragma unroll 1
        for (int c = 0; c < n; ++c) {
            float vj[VJ];
#pragma unroll
            for (int x = 0; x < VJ; ++x) vj[x] = live[x] ? s_v[c][jl * VJ + x] : 0.f;
            const float beta = s_b[c];
            // one walk over the decayed state gives both sums over key channels: the prediction S^T k and the
            // read-out of the state before the write, S^T q; the write k u^T then adds u (k . q) to the read-out
            float d[VJ][4], a[VJ][4];
#pragma unroll
            for (int x = 0; x < VJ; ++x) {
#pragma unroll
                for (int e = 0; e < 4; ++e) { d[x][e] = 0.f; a[x][e] = 0.f; }
            }
#pragma unroll
            for (int i = 0; i < KP; i += 4) {
                // thread `part` holds key channels 4 PARTS m + 4 part + e (m = i / 4, e < 4)
                const int at = i * PARTS + part * 4;
                const float4 g4 = *reinterpret_cast<const float4*>(&s_g[c][at]);
                const float4 k4 = *reinterpret_cast<const float4*>(&s_k[c][at]);
                const float4 q4 = *reinterpret_cast<const float4*>(&s_q[c][at]);
#pragma unroll
                for (int x = 0; x < VJ; ++x) {
                    S[x][i]     *= g4.x;  d[x][0] += k4.x * S[x][i];      a[x][0] += q4.x * S[x][i];
                    S[x][i + 1] *= g4.y;  d[x][1] += k4.y * S[x][i + 1];  a[x][1] += q4.y * S[x][i + 1];
                    S[x][i + 2] *= g4.z;  d[x][2] += k4.z * S[x][i + 2];  a[x][2] += q4.z * S[x][i + 2];
                    S[x][i + 3] *= g4.w;  d[x][3] += k4.w * S[x][i + 3];  a[x][3] += q4.w * S[x][i + 3];
                }
            }
            float dot[VJ], acc[VJ];
#pragma unroll
            for (int x = 0; x < VJ; ++x) {
                dot[x] = (d[x][0] + d[x][1]) + (d[x][2] + d[x][3]);
                acc[x] = (a[x][0] + a[x][1]) + (a[x][2] + a[x][3]);
            }
#pragma unroll
            for (int off = 1; off < PARTS; off <<= 1) {
#pragma unroll
                for (int x = 0; x < VJ; ++x) {
                    dot[x] += __shfl_xor_sync(0xffffffffu, dot[x], off);
                    acc[x] += __shfl_xor_sync(0xffffffffu, acc[x], off);
                }
            }
            float u[VJ];
#pragma unroll
            for (int x = 0; x < VJ; ++x) {
                u[x] = beta * (vj[x] - dot[x]);
                acc[x] += u[x] * s_kq[c];
            }
#pragma unroll
            for (int i = 0; i < KP; i += 4) {
                const int at = i * PARTS + part * 4;
                const float4 k4 = *reinterpret_cast<const float4*>(&s_k[c][at]);
#pragma unroll
                for (int x = 0; x < VJ; ++x) {
                    S[x][i]     += k4.x * u[x];
                    S[x][i + 1] += k4.y * u[x];
                    S[x][i + 2] += k4.z * u[x];
                    S[x][i + 3] += k4.w * u[x];
                }
            }
            if (part == 0) {
#pragma unroll
                for (int x = 0; x < VJ; ++x)
                    if (live[x]) o[(size_t)(c0 + c) * heads * V + (size_t)h * V + j0 + jl * VJ + x] = acc[x];
            }
        }
    }
#pragma unroll
    for (int x = 0; x < VJ; ++x) {
#pragma unroll
        for (int i = 0; i < KP; i += 4) {
            float* p = S_g + (size_t)(j0 + jl * VJ + x) * NP + i * PARTS + part * 4;
            if (!live[x] || !mine) continue;
            if (vec) *reinterpret_cast<float4*>(p) = make_float4(S[x][i], S[x][i + 1], S[x][i + 2], S[x][i + 3]);
            else { p[0] = S[x][i]; p[1] = S[x][i + 1]; p[2] = S[x][i + 2]; p[3] = S[x][i + 3]; }
        }
    }
}

// Prompts in bfloat16, sixteen tokens at a time (chunk_scan.cuh): the first kernel, a block per (CF_WARPS warps of records, head).  It
// makes q and k unit vectors, forms the decays, the products of pairs of tokens, and the inverse of the unit lower triangle by
// forward substitution, a column a lane.
template <int NK>
__global__ void __launch_bounds__(32 * CF_WARPS, 5) delta_prepare_kernel(DeltaArgs A, ChunkRecord<NK, true>* __restrict__ recs,
                                                                      const int* __restrict__ cu_q, int n_seqs, int n_records, int min_len, int heads) {
    pdl_prologue();
    __shared__ __align__(16) ChunkForm<NK, true> form[cf_records<NK>()];
    constexpr int WR = cf_warps_a_record<NK>();
    const int h = blockIdx.y, group = h / A.heads_per_group, lane = threadIdx.x & 31, warp = threadIdx.x / 32 % WR, c0 = warp * 64, c = c0 + 2 * lane;
    const int r = blockIdx.x * cf_records<NK>() + threadIdx.x / (32 * WR);
    if (r >= n_records) return;
    int s, chunk, t0, left;
    chunk_of_record(cu_q, n_seqs, r, min_len, s, chunk, t0, left);
    if (chunk < 0) return;
    ChunkForm<NK, true>& sh = form[threadIdx.x / (32 * WR)];
    const bf16* qp = pdl_fresh((const bf16*)A.q) + A.q_off + (size_t)group * NK + c0 + (size_t)t0 * A.q_stride;
    const bf16* kp = pdl_fresh((const bf16*)A.k) + A.k_off + (size_t)group * NK + c0 + (size_t)t0 * A.k_stride;
    const float* ap = pdl_fresh(A.a) + A.a_off + (size_t)t0 * A.a_stride + (A.decay_per_head ? h : h * NK + c0);
    const float rate = expf(A.a_log[h]);
    auto& rows = sh.rows[warp];
    if (A.decay_per_head) {                                 // a lane a token, the same for every channel
        cf_fetch<false>(rows, qp, A.q_stride, kp, A.k_stride, ap, A.a_stride, left);
        float g = 1.f;
        if (lane < CS_C && lane < left) g = expf(-rate * dr_softplus(ap[(size_t)lane * A.a_stride] + A.dt_bias[h]));
#pragma unroll
        for (int t = 0; t < CS_C; ++t) {
            const float a = __shfl_sync(0xffffffffu, g, t);
            rows.a[t][lane] = make_float2(a, a);
        }
    } else {
        cf_fetch<true>(rows, qp, A.q_stride, kp, A.k_stride, ap, A.a_stride, left);
        const float bx = A.dt_bias[h * NK + c], by = A.dt_bias[h * NK + c + 1];
#pragma unroll 2
        for (int t = 0; t < CS_C; ++t) {
            float2& a = rows.a[t][lane];
            a = t < left ? make_float2(expf(-rate * dr_softplus(a.x + bx)), expf(-rate * dr_softplus(a.y + by))) : make_float2(1.f, 1.f);
        }
    }
    if (warp == 0 && lane < CS_C) {
        const bf16* bp = pdl_fresh((const bf16*)A.beta) + A.beta_off + h;
        sh.beta[lane] = lane < left ? 1.0f / (1.0f + expf(-to_float(bp[(size_t)(t0 + lane) * A.beta_stride]))) : 0.f;
    }
    // the tokens' lengths: 32 sums over the record's channels, a lane each (q's 16, then k's)
    {
        float x[CS_C];
        const bool other = lane & 16;
#pragma unroll
        for (int t = 0; t < CS_C; ++t) {
            const uint32_t qv = rows.q[t][lane], kv = rows.k[t][lane];
            const float q0 = cm_lo(qv), q1 = cm_hi(qv), k0 = cm_lo(kv), k1 = cm_hi(kv);
            const float qq = q0 * q0 + q1 * q1, kk = k0 * k0 + k1 * k1, away = other ? qq : kk;
            x[t] = (other ? kk : qq) + __shfl_xor_sync(0xffffffffu, away, 16);
        }
        const float mine = cf_join<16, 16>(x);
        sh.sums[warp][(lane & 16) + cf_kept<16>(lane)] = mine;
        cf_sync<NK>();
        if (warp == 0) {
            float sum = sh.sums[0][lane];
            if constexpr (WR == 2) sum += sh.sums[1][lane];
            // rows behind the sequence's end stay zero, also where unit_eps is
            const float f = (lane & 15) < left ? ((lane & 16) ? 1.0f : A.q_scale) / sqrtf(sum + A.unit_eps) : 0.f;
            reinterpret_cast<float*>(sh.unit)[(lane & 15) * 2 + (lane >> 4)] = f;
        }
        cf_sync<NK>();
    }
    ChunkRecord<NK, true>* rec = recs + (size_t)r * heads + h;
    chunk_form<NK, true, false>(rec, sh, warp, 0ull, [&](int t, f32x2& q, f32x2& k, f32x2& a) {
        const float2 f = sh.unit[t];
        q = f2_mul(cf_pair(rows.q[t][lane]), f2_pack(f.x, f.x));
        k = f2_mul(cf_pair(rows.k[t][lane]), f2_pack(f.y, f.y));
        a = *reinterpret_cast<const f32x2*>(&rows.a[t][lane]);
    });
    cf_sync<NK>();
    chunk_emit<NK, WR>(rec->P[0], sh.P);
    if (warp == 0) {
        float x[CS_C];
#pragma unroll
        for (int t = 0; t < CS_C; ++t) {
            const float b = sh.beta[t];
            float y = t == lane ? b : 0.f;
#pragma unroll
            for (int u = 0; u < t; ++u) {
                float m = sh.M[0][t][u];
                if constexpr (WR == 2) m += sh.M[1][t][u];
                y -= b * m * x[u];
            }
            x[t] = y;
        }
        __syncwarp();                                       // everything has been read
        if (lane < CS_C) {
#pragma unroll
            for (int t = 0; t < CS_C; ++t) sh.M[0][t][lane] = x[t];
        }
    }
    cf_sync<NK>();
    chunk_emit<NK, 1>(rec->TB[0], sh.M);
}

// y[t, h*V + i] = o[t, h*V + i] / sqrt(mean_i o[t, h, :]^2 + eps) * w[i] * act(gate[t, gate_off + h*V + i]):
// a norm over each head's values with one weight row for all heads, then a gate, act = sigmoid (gate_act 0) or
// SiLU (gate_act 1).  One warp per (token, head).
template <typename T, typename TG>
__global__ void head_norm_gate_kernel(const float* o, const TG* gate, int gate_stride, int gate_off,
                                      const float* __restrict__ w, float eps, T* __restrict__ y, int rows, int heads, int V,
                                      int gate_act) {
    pdl_prologue();
    o = pdl_fresh(o);
    gate = pdl_fresh(gate);
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= rows) return;
    const int t = row / heads, h = row - t * heads;
    const float* orow = o + (size_t)row * V;
    const TG* grow = gate + (size_t)t * gate_stride + gate_off + (size_t)h * V;
    float ss = 0.f;
    for (int i = lane; i < V; i += 32) ss += orow[i] * orow[i];
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)V + eps);
    for (int i = lane; i < V; i += 32) {
        const float g = to_float(grow[i]), sg = 1.0f / (1.0f + expf(-g));
        y[(size_t)row * V + i] = from_float<T>(orow[i] * inv * w[i] * (gate_act ? g * sg : sg));
    }
}

// The same for heads of 64 or 128 values on 16 bytes: V / 4 lanes a head, four values each, read once: 36 -> 21 us for the two
// portions of three prompts of 1501 tokens and less, 16 heads of 128.
template <typename T, typename TG, int LANES>
__global__ void __launch_bounds__(256) head_norm_gate_vec_kernel(const float* o, const TG* gate, int gate_stride, int gate_off,
                                                                 const float* __restrict__ w, float eps, T* __restrict__ y, int rows, int heads,
                                                                 int gate_act) {
    pdl_prologue();
    o = pdl_fresh(o);
    gate = pdl_fresh(gate);
    constexpr int V = 4 * LANES;
    const int row = (blockIdx.x * 256 + threadIdx.x) / LANES, i = threadIdx.x % LANES * 4;
    const bool live = row < rows;
    const int t = live ? row / heads : 0, h = live ? row - t * heads : 0;
    struct alignas(4 * sizeof(TG)) FourG { TG v[4]; };
    struct alignas(4 * sizeof(T)) Four { T v[4]; };
    float4 ov = make_float4(0.f, 0.f, 0.f, 0.f);
    FourG gv;
    if (live) {
        ov = *reinterpret_cast<const float4*>(o + (size_t)row * V + i);
        gv = *reinterpret_cast<const FourG*>(gate + (size_t)t * gate_stride + gate_off + (size_t)h * V + i);
    }
    float ss = (ov.x * ov.x + ov.y * ov.y) + (ov.z * ov.z + ov.w * ov.w);
#pragma unroll
    for (int off = LANES / 2; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
    if (!live) return;
    const float inv = 1.0f / sqrtf(ss / (float)V + eps);
    const float4 w4 = *reinterpret_cast<const float4*>(w + i);
    const float v[4] = {ov.x, ov.y, ov.z, ov.w}, wv[4] = {w4.x, w4.y, w4.z, w4.w};
    Four out;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float g = to_float(gv.v[e]), sg = 1.0f / (1.0f + expf(-g));
        out.v[e] = from_float<T>(v[e] * inv * wv[e] * (gate_act ? g * sg : sg));
    }
    *reinterpret_cast<Four*>(y + (size_t)row * V + i) = out;
}

}  // namespace ff

using namespace ff;

// floats of a request's state for `heads` heads of key size N and value size V (-1: sizes not supported)
FF_EXPORT long long ff_delta_state_floats(int heads, int N, int V) {
    DeltaPlan p;
    if (!delta_plan(N, V, &p)) return -1;
    return (long long)heads * V * p.NP;
}

// Tokens from which a sequence goes by chunks.  us for n sequences of L tokens, chunks / token by token, 8 heads of 128 x 128:
//   L     n = 1         4             8             16            32
//   16    11.9 / 12.4   14.2 / 12.6   16.1 / 12.7   21.0 / 24.3   32.3 / 47.4
//   24    13.0 / 18.7   16.1 / 19.0   19.1 / 19.0   27.3 / 37.1   50.7 / 73.0
//   64    17.3 / 43.5   19.7 / 43.7   24.8 / 43.8   45.9 / 86.4   89.8 / 172
constexpr int DELTA_CHUNK_MIN = 24;
FF_EXPORT int ff_delta_chunk_min() { return DELTA_CHUNK_MIN; }

// Bytes of scratch memory that a step of T tokens can use (0: none; without it the token-by-token kernel runs).  `bits`: the matrices'
// addresses, row strides and first columns in bytes, or'ed (row_bits).
FF_EXPORT long long ff_delta_scratch_bytes(int dtype, int T, int n_seqs, int heads, int N, int V, int bits) {
    if (dtype != 1 || (bits & 15) || T < DELTA_CHUNK_MIN || n_seqs <= 0 || (N != 64 && N != 128) || V <= 0 || V > 256 || V % 8) return 0;
    return chunk_records(T, n_seqs) * heads * (long long)(N == 64 ? sizeof(ChunkRecord<64, true>) : sizeof(ChunkRecord<128, true>));
}

static unsigned delta_bits(const DeltaArgs& A) {
    return row_bits(A.q, A.q_stride, A.q_off, 2) | row_bits(A.k, A.k_stride, A.k_off, 2) | row_bits(A.v, A.v_stride, A.v_off, 2) |
           (A.decay_per_head ? 0u : row_bits(A.a, A.a_stride, A.a_off, 4));
}

template <int NK>
static int delta_chunk_launch(const DeltaArgs& A, const ChunkScanArgs& B, int T, int n_seqs, int live, void* scratch, cudaStream_t stream) {
    const int n_records = (int)chunk_records(T, n_seqs);
    FF_ALL_SHARED(delta_prepare_kernel<NK>);
    FF_LAUNCH(delta_prepare_kernel<NK>, cf_grid<NK>(n_records, B.heads), 32 * CF_WARPS, 0, stream, A, (ChunkRecord<NK, true>*)scratch, B.cu_q,
              n_seqs, n_records, B.min_len, B.heads);
    return chunk_scan_launch<NK, true>(B, n_seqs, live, stream);
}

template <typename T>
static int delta_launch(const DeltaArgs& A, float* state, long long state_stride, int state_off, const int* cu_q,
                        const int* state_slots, const int* seq_fresh, float* o, int n_seqs, int heads, int N, int V,
                        int max_len, cudaStream_t stream) {
    DeltaPlan p;
    if (!delta_plan(N, V, &p)) return FF_ERR_UNSUPPORTED;
    if (p.Vb > 128) return FF_ERR_UNSUPPORTED;
    dim3 grid(n_seqs, heads, p.vsplit);
#define FF_DELTA_ONE(NP, PARTS, VJ, SOME)                                                                          \
    FF_LAUNCH((delta_rule_scan_kernel<T, NP, PARTS, VJ, SOME>), grid, p.threads, 0, stream, A, state, (size_t)state_stride, \
              state_off, cu_q, state_slots, seq_fresh, o, heads, N, V, p.Vb, max_len)
#define FF_DELTA(NP, PARTS, VJ)                                                                                    \
    do {                                                                                                           \
        constexpr bool SOME = sizeof(T) == 2 && (NP == 64 || NP == 128);        /* no other size goes by chunks */  \
        if (SOME && max_len != 0x7fffffff) FF_DELTA_ONE(NP, PARTS, VJ, SOME);                                      \
        else FF_DELTA_ONE(NP, PARTS, VJ, false);                                                                   \
    } while (0)
    switch (p.NP) {
        case 16: FF_DELTA(16, 4, 1); break;
        case 32: FF_DELTA(32, 8, 1); break;
        case 64: FF_DELTA(64, 8, 1); break;
        case 128: FF_DELTA(128, 16, 2); break;
        case 256: FF_DELTA(256, 16, 2); break;
        default: return FF_ERR_UNSUPPORTED;
    }
#undef FF_DELTA
#undef FF_DELTA_ONE
    FF_LAUNCH_CHECK();
    return 0;
}

// `n_long`: how many of the sequences have ff_delta_chunk_min tokens or more (-1: not known).  `launched`: how many kernels the call put
// on the stream (1: token by token, 2: by chunks, 3: some sequences so and some so).
FF_EXPORT int ff_delta_rule_scan(const void* q, int q_stride, int q_off, const void* k, int k_stride, int k_off,
                                 const void* v, int v_stride, int v_off, const void* beta, int beta_stride, int beta_off,
                                 int dtype, const float* a, int a_stride, int a_off, const float* dt_bias,
                                 const float* a_log, int decay_per_head, int heads_per_group, float q_scale, float unit_eps, float* state,
                                 long long state_stride, int state_off, const int* cu_q, const int* state_slots,
                                 const int* seq_fresh, float* o, int T, int n_seqs, int heads, int N, int V,
                                 int n_long, void* scratch, long long scratch_bytes, int* launched, cudaStream_t stream) {
    *launched = 0;
    if (T <= 0 || n_seqs <= 0) return 0;
    if (heads_per_group <= 0 || heads % heads_per_group) return FF_ERR_BAD_ARG;
    DeltaArgs A{q, q_stride, q_off, k, k_stride, k_off, v, v_stride, v_off, beta, beta_stride, beta_off,
                a, a_stride, a_off, dt_bias, a_log, heads_per_group, q_scale, unit_eps, decay_per_head ? 1 : 0};
    const long long need = ff_delta_scratch_bytes(dtype, T, n_seqs, heads, N, V, (int)delta_bits(A));
    const ChunkRoute R = chunk_route(need > 0 && scratch && scratch_bytes >= need, n_long, n_seqs, DELTA_CHUNK_MIN);
    *launched = R.kernels();
    if (R.walk) {
        int rc = FF_ERR_BAD_ARG;
        if (dtype == 0)
            rc = delta_launch<float>(A, state, state_stride, state_off, cu_q, state_slots, seq_fresh, o, n_seqs, heads, N, V, R.max_walk, stream);
        else if (dtype == 1)
            rc = delta_launch<bf16>(A, state, state_stride, state_off, cu_q, state_slots, seq_fresh, o, n_seqs, heads, N, V, R.max_walk, stream);
        if (rc) return rc;
    }
    if (!R.chunks) return 0;
    const ChunkScanArgs B{scratch, (const bf16*)v, v_stride, v_off, state, state_stride, state_off, V * N, cu_q, state_slots, seq_fresh, o, heads, V, DELTA_CHUNK_MIN};
    return N == 64 ? delta_chunk_launch<64>(A, B, T, n_seqs, R.live, scratch, stream) : delta_chunk_launch<128>(A, B, T, n_seqs, R.live, scratch, stream);
}

// gate_dtype: 32-bit, or the type of y
FF_EXPORT int ff_head_norm_gate(const float* o, const void* gate, int gate_dtype, int gate_stride, int gate_off, const float* w, float eps,
                                void* y, int dtype, int T, int heads, int V, int gate_act, cudaStream_t stream) {
    const int rows = T * heads;
    if (rows <= 0) return 0;
    const int warps = 4;
    const unsigned blocks = (unsigned)((rows + warps - 1) / warps);
    const int es = dtype == 0 ? 4 : 2, eg = gate_dtype == 0 ? 4 : 2;
    if ((V == 64 || V == 128) && (((uintptr_t)o | (uintptr_t)w) & 15) == 0 && ((uintptr_t)y & (4 * es - 1)) == 0 &&
        ((uintptr_t)gate & (4 * eg - 1)) == 0 && gate_stride % 4 == 0 && gate_off % 4 == 0) {
        const unsigned n = (unsigned)(((long long)rows * (V / 4) + 255) / 256);
#define FF_HEAD_NORM(TT, TG)                                                                                                     \
        do {                                                                                                                     \
            if (V == 64) FF_LAUNCH((head_norm_gate_vec_kernel<TT, TG, 16>), n, 256, 0, stream, o, (const TG*)gate, gate_stride, gate_off, w, eps, (TT*)y, rows, heads, gate_act); \
            else FF_LAUNCH((head_norm_gate_vec_kernel<TT, TG, 32>), n, 256, 0, stream, o, (const TG*)gate, gate_stride, gate_off, w, eps, (TT*)y, rows, heads, gate_act); \
        } while (0)
        if (dtype == 0 && gate_dtype == 0) FF_HEAD_NORM(float, float);
        else if (dtype == 1 && gate_dtype == 0) FF_HEAD_NORM(bf16, float);
        else if (dtype == 1 && gate_dtype == 1) FF_HEAD_NORM(bf16, bf16);
        else return FF_ERR_BAD_ARG;
#undef FF_HEAD_NORM
        FF_LAUNCH_CHECK();
        return 0;
    }
    if (dtype == 0 && gate_dtype == 0)
        FF_LAUNCH((head_norm_gate_kernel<float, float>), blocks, warps * 32, 0, stream, o, (const float*)gate, gate_stride,
                  gate_off, w, eps, (float*)y, rows, heads, V, gate_act);
    else if (dtype == 1 && gate_dtype == 0)
        FF_LAUNCH((head_norm_gate_kernel<bf16, float>), blocks, warps * 32, 0, stream, o, (const float*)gate, gate_stride,
                  gate_off, w, eps, (bf16*)y, rows, heads, V, gate_act);
    else if (dtype == 1 && gate_dtype == 1)
        FF_LAUNCH((head_norm_gate_kernel<bf16, bf16>), blocks, warps * 32, 0, stream, o, (const bf16*)gate, gate_stride,
                  gate_off, w, eps, (bf16*)y, rows, heads, V, gate_act);
    else return FF_ERR_BAD_ARG;
    FF_LAUNCH_CHECK();
    return 0;
}
