// A recurrent mixer with a matrix state per head and a per-channel, data-dependent decay
// (RWKV-style time mixing):
//
//   mix_s[t] = x[t] + (x[t-1] - x[t]) * mu_s            s in {r, k, v, g, w};  x[-1] = 0
//   o[t]     = (S + diag(u) k[t] v[t]^T)^T r[t]         per head, S: [key channel, value channel]
//   S       <- diag(w[t]) S + k[t] v[t]^T               w[t] = exp(-exp(d[t] + w0))
//   y[t]     = o[t] / rms(o[t]) * norm * silu(g[t])     rms over a head's channels
//
// The state (S and the last x of the sequence) lives in 32-bit in the request's state slot and
// is carried from step to step; a fresh request starts from zeros.  Everything that enters the
// recurrence is 32-bit: decays, the bonus u, S, the sums.  Steps of few tokens walk a sequence token by token; bfloat16
// prompts are taken a chunk of tokens at a time, whose sums are formed in another order, as right.
#include "chunk_scan.cuh"
#include "common.cuh"
#include "scan_wide.cuh"

namespace ff {

// One block per token: the five mixes.  The token in front is x[t-1] inside a portion and the
// state's saved row at its head (zeros for a fresh request).
template <typename T>
__global__ void wkv_shift_mix_kernel(const T* __restrict__ x, const float* __restrict__ mu /*[5,W]*/,
                                     const float* __restrict__ state, size_t state_stride, int prev_off,
                                     const int* __restrict__ token_seq, const int* __restrict__ cu_q,
                                     const int* __restrict__ state_slots, const int* __restrict__ seq_fresh,
                                     T* __restrict__ mixes /*[5,T,W]*/, int Ttot, int W) {
    pdl_prologue();
    const int t = blockIdx.x;
    const int s = token_seq[t];
    const bool first = t == cu_q[s];
    const bool fresh = seq_fresh[s] != 0;
    const float* prev_state = state + (size_t)state_slots[s] * state_stride + prev_off;
    const T* xr = x + (size_t)t * W;
    const T* xp = x + (size_t)(t - 1) * W;
    for (int i = threadIdx.x; i < W; i += blockDim.x) {
        const float cur = to_float(xr[i]);
        const float prev = first ? (fresh ? 0.f : prev_state[i]) : to_float(xp[i]);
        const float d = prev - cur;
#pragma unroll
        for (int m = 0; m < 5; ++m)
            mixes[((size_t)m * Ttot + t) * W + i] = from_float<T>(cur + d * mu[(size_t)m * W + i]);
    }
}

// The same for widths in steps of 8 on 16 bytes: eight channels a thread, whose five weights stay in registers over
// MIX_TOKENS tokens (with one channel a thread the loads and stores are two bytes each): 52 -> 22.5 us on 4900 rows of 2048, whose bytes take 19.
constexpr int MIX_TOKENS = 4;
template <typename T>
__global__ void __launch_bounds__(128) wkv_shift_mix_vec_kernel(const T* x, const float* __restrict__ mu /*[5,W]*/, const float* state,
                                                                size_t state_stride, int prev_off, const int* __restrict__ token_seq,
                                                                const int* __restrict__ cu_q, const int* __restrict__ state_slots,
                                                                const int* __restrict__ seq_fresh, T* __restrict__ mixes /*[5,T,W]*/, int Ttot, int W,
                                                                int tokens) {
    pdl_prologue();
    x = pdl_fresh(x);
    state = pdl_fresh(state);
    struct alignas(16) Pack { T v[16 / sizeof(T)]; };
    constexpr int PER = 16 / (int)sizeof(T), PACKS = 8 / PER;
    const int i = (blockIdx.y * 128 + threadIdx.x) * 8;
    if (i >= W) return;
    const int tile0 = blockIdx.x * tokens, tile1 = min(Ttot, tile0 + tokens);
    auto row = [&](int t, float v[8]) {
#pragma unroll
        for (int p = 0; p < PACKS; ++p) {
            const Pack r = *reinterpret_cast<const Pack*>(x + (size_t)t * W + i + p * PER);
#pragma unroll
            for (int e = 0; e < PER; ++e) v[p * PER + e] = to_float(r.v[e]);
        }
    };
    float m[5][8], prev[8], cur[8];
#pragma unroll
    for (int s = 0; s < 5; ++s) {
        *reinterpret_cast<float4*>(m[s]) = *reinterpret_cast<const float4*>(mu + (size_t)s * W + i);
        *reinterpret_cast<float4*>(m[s] + 4) = *reinterpret_cast<const float4*>(mu + (size_t)s * W + i + 4);
    }
    if (tile0 > 0) row(tile0 - 1, prev);
    for (int t = tile0; t < tile1; ++t) {
        const int s = token_seq[t];
        row(t, cur);
        if (t == cu_q[s]) {
            const float* saved = state + (size_t)state_slots[s] * state_stride + prev_off + i;
            const bool fresh = seq_fresh[s] != 0;
#pragma unroll
            for (int e = 0; e < 8; ++e) prev[e] = fresh ? 0.f : saved[e];
        }
#pragma unroll
        for (int k = 0; k < 5; ++k) {
#pragma unroll
            for (int p = 0; p < PACKS; ++p) {
                Pack r;
#pragma unroll
                for (int e = 0; e < PER; ++e) {
                    const int c = p * PER + e;
                    r.v[e] = from_float<T>(cur[c] + (prev[c] - cur[c]) * m[k][c]);
                }
                *reinterpret_cast<Pack*>(mixes + ((size_t)k * Ttot + t) * W + i + p * PER) = r;
            }
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) prev[e] = cur[e];
    }
}

// tanh of a 32-bit matrix, into the type of the product that follows
template <typename TO>
__global__ void tanh_cast_kernel(const float* __restrict__ in, TO* __restrict__ out, size_t total) {
    pdl_prologue();
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < total) out[idx] = from_float<TO>(tanhf(in[idx]));
}

// One block per (sequence, head, VB value channels), token by token (scan_wide.cuh): a thread holds four columns of S and
// reads r, k and w of its key channels once for all four.  A chunk's r, k, v and decays are staged in 32-bit in one of two
// buffers, asked for before the chunk in front is walked.  The bonus term's sum p = sum_i r_i u_i k_i is formed on the way, a
// thread's share of it from the u of its own key channels.
//   o_j = sum_i r_i S_ij + p v_j;   S_ij <- w_i S_ij + k_i v_j
// Against one column a thread 518 -> 185 us for a sequence of 999 tokens, 16 heads of 64.
template <typename T, int DIM>
__global__ void __launch_bounds__(WS_THREADS) wkv_scan_kernel(
    const T* __restrict__ rkvg_ /*[4,T,HD]*/, const float* __restrict__ dlog_ /*[T,HD]*/,
    const float* __restrict__ w0, const float* __restrict__ u, float* __restrict__ state, size_t state_stride,
    int prev_off, const T* __restrict__ x_, int W, const int* __restrict__ cu_q,
    const int* __restrict__ state_slots, const int* __restrict__ seq_fresh, float* __restrict__ o /*[T,HD]*/,
    int Ttot, int heads, int dim, int max_len) {
    pdl_prologue();
    using WS = WideState<DIM>;
    constexpr int CH = WS::CH, VB = WS::VB < DIM ? WS::VB : DIM, PQ = CH * DIM / WS_THREADS, PV = CH * VB / WS_THREADS;
    static_assert(CH * DIM % WS_THREADS == 0 && CH * VB % WS_THREADS == 0 && WS_THREADS % DIM == 0, "a thread stages one channel of the same number of tokens");
    __shared__ __align__(16) float s_r[2][CH][DIM], s_k[2][CH][DIM], s_w[2][CH][DIM];
    __shared__ __align__(16) f32x2 s_v[2][CH][VB];             // each value twice
    const int s = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, j0 = blockIdx.z * VB;
    const int t0 = cu_q[s], t1s = cu_q[s + 1];
    const bool mine = t1s - t0 < max_len;                      // a sequence that goes by chunks is empty here (as in ssm.cu)
    const int t1 = mine ? t1s : t0;
    const int HD = heads * dim;
    float* st = state + (size_t)state_slots[s] * state_stride;
    float* S_g = st + (size_t)h * DIM * DIM;
    const bool holds = tid < WS::PARTS * (VB / WS_COLS);       // heads of 32: more threads than columns
    WS w;
    w.place(tid);
    w.load(S_g, j0, holds ? dim : 0, seq_fresh[s] != 0);
    f32x2 ub[WS::KP / 2];
#pragma unroll
    for (int m = 0; m < WS::KP / 2; ++m) {
        const int i = (m >> 1) * 4 * WS::PARTS + w.part * 4 + (m & 1) * 2;
        ub[m] = f2_pack(i < dim ? u[h * dim + i] : 0.f, i + 1 < dim ? u[h * dim + i + 1] : 0.f);
    }
    const T* r_in = pdl_fresh(rkvg_) + (size_t)h * dim;
    const T* k_in = r_in + (size_t)Ttot * HD;
    const T* v_in = k_in + (size_t)Ttot * HD + j0;
    const float* d_in = pdl_fresh(dlog_) + (size_t)h * dim;
    const int ch = tid % DIM;                                  // the thread's channel of every token it stages
    const float w0c = ch < dim ? w0[h * dim + ch] : 0.f;
    T rn[PQ], kn[PQ], vn[PV];
    float dn[PQ];
    auto fetch = [&](int c0) {
        const int n = min(CH, t1 - c0);
#pragma unroll
        for (int p = 0; p < PQ; ++p) {
            const int c = (tid + p * WS_THREADS) / DIM;
            const bool in = c < n && ch < dim;
            const size_t at = in ? (size_t)(c0 + c) * HD + ch : 0;
            rn[p] = in ? r_in[at] : from_float<T>(0.f);
            kn[p] = in ? k_in[at] : from_float<T>(0.f);
            dn[p] = in ? d_in[at] : 0.f;
        }
#pragma unroll
        for (int p = 0; p < PV; ++p) {
            const int idx = tid + p * WS_THREADS, c = idx / VB, jj = idx % VB;
            vn[p] = (c < n && j0 + jj < dim) ? v_in[(size_t)(c0 + c) * HD + jj] : from_float<T>(0.f);
        }
    };
    auto stage = [&](int b) {
#pragma unroll
        for (int p = 0; p < PQ; ++p) {
            const int idx = tid + p * WS_THREADS;
            (&s_r[b][0][0])[idx] = to_float(rn[p]);
            (&s_k[b][0][0])[idx] = to_float(kn[p]);
            (&s_w[b][0][0])[idx] = expf(-expf(dn[p] + w0c));
        }
#pragma unroll
        for (int p = 0; p < PV; ++p) (&s_v[b][0][0])[tid + p * WS_THREADS] = f2_pack(to_float(vn[p]), to_float(vn[p]));
    };
    const int vj = holds ? w.jl * WS_COLS : 0, first = w.first();
    float* oh = o + (size_t)h * dim + j0;
    if (t0 < t1) {
        fetch(t0);
        stage(0);
    }
    __syncthreads();
    int b = 0;
    for (int c0 = t0; c0 < t1; c0 += CH, b ^= 1) {
        const int n = min(CH, t1 - c0);
        if (c0 + CH < t1) fetch(c0 + CH);
        auto token = [&](int c, float* part) {
            f32x2 v[WS_COLS];
            WS::values(&s_v[b][c][vj], v);
            w.template token<true, true>(s_r[b][c], s_k[b][c], s_w[b][c], 1.f, v, part);
            f32x2 p2 = 0ull;
#pragma unroll
            for (int m = 0; m < WS::KP / 4; ++m) {
                const int at = m * 4 * WS::PARTS + w.part * 4;
                const ulonglong2 r2 = *reinterpret_cast<const ulonglong2*>(&s_r[b][c][at]);
                const ulonglong2 k2 = *reinterpret_cast<const ulonglong2*>(&s_k[b][c][at]);
                p2 = f2_fma(f2_mul(r2.x, ub[2 * m]), k2.x, p2);
                p2 = f2_fma(f2_mul(r2.y, ub[2 * m + 1]), k2.y, p2);
            }
            const float p = f2_sum(p2);
#pragma unroll
            for (int x = 0; x < WS_COLS; ++x) part[x] += p * f2_low(v[x]);
        };
        if (n == CH) {
            float part[CH * WS_COLS];
#pragma unroll
            for (int c = 0; c < CH; ++c) token(c, part + c * WS_COLS);
            w.reduce_chunk(part);
#pragma unroll
            for (int r = 0; r < WS::OUTS; ++r) {
                const int at = first + r, jj = w.jl * WS_COLS + at % WS_COLS;
                if (holds && j0 + jj < dim) oh[(size_t)(c0 + at / WS_COLS) * HD + jj] = part[r];
            }
        } else {
            for (int c = 0; c < n; ++c) {
                float part[WS_COLS];
                token(c, part);
                const float y = w.reduce(part);
                const int jj = w.jl * WS_COLS + w.col();
                if (holds && w.part < 4 && j0 + jj < dim) oh[(size_t)(c0 + c) * HD + jj] = y;
            }
        }
        if (c0 + CH < t1) stage(b ^ 1);
        __syncthreads();
    }
    if (mine) w.store(S_g, j0, holds ? dim : 0);
    // the sequence's last input row, for the first token of its next step
    if (h == 0 && blockIdx.z == 0 && t1 > t0) {
        const T* last = pdl_fresh(x_) + (size_t)(t1 - 1) * W;
        for (int i = tid; i < W; i += WS_THREADS) st[prev_off + i] = to_float(last[i]);
    }
}

// Prompts in bfloat16, sixteen tokens at a time (chunk_scan.cuh): the first kernel, a block per (CF_WARPS warps of records, head).
// The read-out sees the state in front of the token's own decay and write; the bonus term is the diagonal of P.
template <int NK>
__global__ void __launch_bounds__(32 * CF_WARPS) wkv_prepare_kernel(const bf16* rkvg, const float* dlog, const float* __restrict__ w0,
                                                                    const float* __restrict__ u, ChunkRecord<NK, false>* __restrict__ recs,
                                                                    float* __restrict__ state, size_t state_stride, int prev_off, const bf16* x, int W,
                                                                    const int* __restrict__ cu_q, const int* __restrict__ state_slots, int n_seqs,
                                                                    int n_records, int min_len, int Ttot, int heads) {
    pdl_prologue();
    __shared__ __align__(16) ChunkForm<NK, false> form[cf_records<NK>()];
    constexpr int WR = cf_warps_a_record<NK>();
    const int h = blockIdx.y, HD = heads * NK, lane = threadIdx.x & 31, warp = threadIdx.x / 32 % WR;
    const int r = blockIdx.x * cf_records<NK>() + threadIdx.x / (32 * WR);
    if (r >= n_records) return;
    int s, chunk, t0, left;
    chunk_of_record(cu_q, n_seqs, r, min_len, s, chunk, t0, left);
    if (chunk < 0) return;
    const int c = h * NK + warp * 64 + 2 * lane;
    const bf16* rp = pdl_fresh(rkvg) + (size_t)t0 * HD + c;
    const bf16* kp = rp + (size_t)Ttot * HD;
    const float* dp = pdl_fresh(dlog) + (size_t)t0 * HD + c;
    uint32_t rv[CS_C], kv[CS_C];
    float2 dv[CS_C];
#pragma unroll
    for (int t = 0; t < CS_C; ++t) {
        const bool in = t < left;
        rv[t] = in ? *reinterpret_cast<const uint32_t*>(rp + (size_t)t * HD) : 0u;
        kv[t] = in ? *reinterpret_cast<const uint32_t*>(kp + (size_t)t * HD) : 0u;
        dv[t] = in ? *reinterpret_cast<const float2*>(dp + (size_t)t * HD) : make_float2(0.f, 0.f);
    }
    const float w0x = w0[c], w0y = w0[c + 1];
    ChunkForm<NK, false>& sh = form[threadIdx.x / (32 * WR)];
    ChunkRecord<NK, false>* rec = recs + (size_t)r * heads + h;
    chunk_form<NK, false, true>(rec, sh, warp, f2_pack(u[c], u[c + 1]), [&](int t, f32x2& q, f32x2& k, f32x2& a) {
        q = cf_pair(rv[t]);
        k = cf_pair(kv[t]);
        a = t < left ? f2_pack(expf(-expf(dv[t].x + w0x)), expf(-expf(dv[t].y + w0y))) : f2_pack(1.f, 1.f);
    });
    cf_sync<NK>();
    chunk_emit<NK, WR>(rec->P[0], sh.P);
    // the sequence's last input row, for the first token of its next step
    if (h == 0 && left <= CS_C) {
        const bf16* last = pdl_fresh(x) + (size_t)(t0 + left - 1) * W;
        float* prev = state + (size_t)state_slots[s] * state_stride + prev_off;
        for (int i = threadIdx.x % (32 * WR); i < W; i += 32 * WR) prev[i] = to_float(last[i]);
    }
}

// One warp per (token, head): y = o / rms(o) * norm * silu(g)
template <typename T>
__global__ void wkv_out_kernel(const float* __restrict__ o, const T* __restrict__ g, const float* __restrict__ norm,
                               float eps, T* __restrict__ y, int Ttot, int heads, int dim) {
    pdl_prologue();
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= Ttot * heads) return;
    const int t = warp / heads, h = warp - t * heads;
    const size_t base = (size_t)t * heads * dim + (size_t)h * dim;
    float ss = 0.f;
    for (int i = lane; i < dim; i += 32) { const float v = o[base + i]; ss += v * v; }
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)dim + eps);
    for (int i = lane; i < dim; i += 32) {
        const float gv = to_float(g[base + i]);
        y[base + i] = from_float<T>(o[base + i] * inv * norm[h * dim + i] * (gv / (1.0f + expf(-gv))));
    }
}

// The same for heads of 64 or 128 on 16 bytes: dim / 4 lanes a head, four values each, read once: 44 -> 18.5 us on 4900 rows of 2048.
template <typename T, int LANES>
__global__ void __launch_bounds__(256) wkv_out_vec_kernel(const float* o, const T* g, const float* __restrict__ norm, float eps,
                                                          T* __restrict__ y, int Ttot, int heads) {
    pdl_prologue();
    o = pdl_fresh(o);
    g = pdl_fresh(g);
    constexpr int D = 4 * LANES;
    const int row = (blockIdx.x * 256 + threadIdx.x) / LANES, i = threadIdx.x % LANES * 4;
    const bool live = row < Ttot * heads;
    struct alignas(4 * sizeof(T)) Four { T v[4]; };
    float4 ov = make_float4(0.f, 0.f, 0.f, 0.f);
    Four gv;
    if (live) {
        ov = *reinterpret_cast<const float4*>(o + (size_t)row * D + i);
        gv = *reinterpret_cast<const Four*>(g + (size_t)row * D + i);
    }
    float ss = (ov.x * ov.x + ov.y * ov.y) + (ov.z * ov.z + ov.w * ov.w);
#pragma unroll
    for (int off = LANES / 2; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
    if (!live) return;
    const float inv = 1.0f / sqrtf(ss / (float)D + eps);
    const float4 w4 = *reinterpret_cast<const float4*>(norm + (row % heads) * D + i);
    const float v[4] = {ov.x, ov.y, ov.z, ov.w}, wv[4] = {w4.x, w4.y, w4.z, w4.w};
    Four out;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float z = to_float(gv.v[e]);
        out.v[e] = from_float<T>(v[e] * inv * wv[e] * (z / (1.0f + expf(-z))));
    }
    *reinterpret_cast<Four*>(y + (size_t)row * D + i) = out;
}

}  // namespace ff

using namespace ff;

FF_EXPORT int ff_wkv_shift_mix(const void* x, int dtype, const float* mu, const float* state, long long state_stride,
                               int prev_off, const int* token_seq, const int* cu_q, const int* state_slots,
                               const int* seq_fresh, void* mixes, int T, int W, cudaStream_t stream) {
    if (T <= 0) return 0;
    const int threads = W >= 1024 ? 256 : 128;
    if (W % 8 == 0 && (((uintptr_t)x | (uintptr_t)mu | (uintptr_t)mixes) & 15) == 0 && (dtype == 0 || dtype == 1)) {
        const int tokens = T >= 1024 ? MIX_TOKENS : 1;           // few tokens: a thread a token, so that they still fill the GPU
        const dim3 grid((T + tokens - 1) / tokens, (W / 8 + 127) / 128);
        if (dtype == 0)
            FF_LAUNCH((wkv_shift_mix_vec_kernel<float>), grid, 128, 0, stream, (const float*)x, mu, state, (size_t)state_stride, prev_off,
                      token_seq, cu_q, state_slots, seq_fresh, (float*)mixes, T, W, tokens);
        else
            FF_LAUNCH((wkv_shift_mix_vec_kernel<bf16>), grid, 128, 0, stream, (const bf16*)x, mu, state, (size_t)state_stride, prev_off,
                      token_seq, cu_q, state_slots, seq_fresh, (bf16*)mixes, T, W, tokens);
        FF_LAUNCH_CHECK();
        return 0;
    }
    if (dtype == 0)
        FF_LAUNCH((wkv_shift_mix_kernel<float>), T, threads, 0, stream, (const float*)x, mu, state, (size_t)state_stride,
                  prev_off, token_seq, cu_q, state_slots, seq_fresh, (float*)mixes, T, W);
    else if (dtype == 1)
        FF_LAUNCH((wkv_shift_mix_kernel<bf16>), T, threads, 0, stream, (const bf16*)x, mu, state, (size_t)state_stride,
                  prev_off, token_seq, cu_q, state_slots, seq_fresh, (bf16*)mixes, T, W);
    else return FF_ERR_BAD_ARG;
    FF_LAUNCH_CHECK();
    return 0;
}

FF_EXPORT int ff_tanh_cast(const float* in, void* out, int out_dtype, long long total, cudaStream_t stream) {
    if (total <= 0) return 0;
    const unsigned blocks = (unsigned)((total + 255) / 256);
    if (out_dtype == 0) FF_LAUNCH((tanh_cast_kernel<float>), blocks, 256, 0, stream, in, (float*)out, (size_t)total);
    else if (out_dtype == 1) FF_LAUNCH((tanh_cast_kernel<bf16>), blocks, 256, 0, stream, in, (bf16*)out, (size_t)total);
    else return FF_ERR_BAD_ARG;
    FF_LAUNCH_CHECK();
    return 0;
}

template <typename T>
static int wkv_scan_launch(const void* rkvg, const float* dlog, const float* w0, const float* u, float* state,
                           long long state_stride, int prev_off, const void* x, int W, const int* cu_q,
                           const int* state_slots, const int* seq_fresh, float* o, int Ttot, int n_seqs, int heads,
                           int dim, int max_len, cudaStream_t stream) {
#define FF_WKV(D)                                                                                                  \
    FF_LAUNCH((wkv_scan_kernel<T, D>), dim3(n_seqs, heads, (dim + min(D, WideState<D>::VB) - 1) / min(D, WideState<D>::VB)), WS_THREADS, 0, stream, \
              (const T*)rkvg, dlog, w0, u, state, (size_t)state_stride, prev_off, (const T*)x, W, cu_q, state_slots, seq_fresh, o, Ttot, heads, dim, max_len)
    if (dim <= 32) FF_WKV(32);
    else if (dim <= 64) FF_WKV(64);
    else if (dim <= 128) FF_WKV(128);
    else return FF_ERR_UNSUPPORTED;
#undef FF_WKV
    FF_LAUNCH_CHECK();
    return 0;
}

// the head size the recurrence kernel is instantiated for (its state keeps that many squared floats a head)
FF_EXPORT int ff_wkv_state_dim(int dim) { return dim <= 32 ? 32 : (dim <= 64 ? 64 : (dim <= 128 ? 128 : -1)); }

// Tokens from which a sequence goes by chunks.  us for n sequences of L tokens, chunks / token by token, 32 heads of 64:
//   L     n = 1         4             8             16            32
//   48    9.5 / 10.1    13.4 / 14.9   18.9 / 19.6   32.0 / 26.3   58.7 / 43.2
//   64    10.9 / 12.8   14.4 / 19.1   22.4 / 25.3   39.4 / 34.3   77.5 / 56.8
//   256   20.2 / 45.3   38.2 / 70.2   72.3 / 94.4   134 / 130     246 / 217
// (two of 48: 11.7 / 10.2).  With 512 heads and more in flight the walk keeps the GPU busy by itself and chunks are up to a quarter slower; the rule
// does not look at that, since it would make a request's numbers depend on how many others there are.
constexpr int WKV_CHUNK_MIN = 64;
FF_EXPORT int ff_wkv_chunk_min() { return WKV_CHUNK_MIN; }

// Bytes of scratch memory that a step of T tokens can use (0: none; without it the token-by-token kernel runs).  `bits`: the addresses of
// rkvg and dlog, or'ed.
FF_EXPORT long long ff_wkv_scratch_bytes(int dtype, int T, int n_seqs, int heads, int dim, int bits) {
    if (dtype != 1 || (bits & 15) || T < WKV_CHUNK_MIN || n_seqs <= 0 || (dim != 64 && dim != 128)) return 0;
    return chunk_records(T, n_seqs) * heads * (long long)(dim == 64 ? sizeof(ChunkRecord<64, false>) : sizeof(ChunkRecord<128, false>));
}

template <int D>
static int wkv_chunk_launch(const bf16* rkvg, const float* dlog, const float* w0, const float* u, int prev_off, const bf16* x, int W,
                            const ChunkScanArgs& B, int Ttot, int n_seqs, int live, void* scratch, cudaStream_t stream) {
    const int n_records = (int)chunk_records(Ttot, n_seqs);
    FF_LAUNCH(wkv_prepare_kernel<D>, cf_grid<D>(n_records, B.heads), 32 * CF_WARPS, 0, stream, rkvg, dlog, w0, u,
              (ChunkRecord<D, false>*)scratch, B.state, (size_t)B.state_stride, prev_off, x, W, B.cu_q, B.state_slots, n_seqs, n_records,
              B.min_len, Ttot, B.heads);
    return chunk_scan_launch<D, false>(B, n_seqs, live, stream);
}

// `n_long`: how many of the sequences have ff_wkv_chunk_min tokens or more (-1: not known).  `launched`: how many kernels the call put
// on the stream (1: token by token, 2: by chunks, 3: some sequences so and some so).
FF_EXPORT int ff_wkv_scan(const void* rkvg, int dtype, const float* dlog, const float* w0, const float* u, float* state,
                          long long state_stride, int prev_off, const void* x, int W, const int* cu_q,
                          const int* state_slots, const int* seq_fresh, float* o, int Ttot, int n_seqs, int heads,
                          int dim, int n_long, void* scratch, long long scratch_bytes, int* launched, cudaStream_t stream) {
    *launched = 0;
    if (Ttot <= 0 || n_seqs <= 0) return 0;
    const long long need = ff_wkv_scratch_bytes(dtype, Ttot, n_seqs, heads, dim, (int)(row_bits(rkvg, 0, 0, 2) | row_bits(dlog, 0, 0, 4)));
    const ChunkRoute R = chunk_route(need > 0 && scratch && scratch_bytes >= need, n_long, n_seqs, WKV_CHUNK_MIN);
    *launched = R.kernels();
    if (R.walk) {
        int rc = FF_ERR_BAD_ARG;
        if (dtype == 0)
            rc = wkv_scan_launch<float>(rkvg, dlog, w0, u, state, state_stride, prev_off, x, W, cu_q, state_slots,
                                        seq_fresh, o, Ttot, n_seqs, heads, dim, R.max_walk, stream);
        else if (dtype == 1)
            rc = wkv_scan_launch<bf16>(rkvg, dlog, w0, u, state, state_stride, prev_off, x, W, cu_q, state_slots,
                                       seq_fresh, o, Ttot, n_seqs, heads, dim, R.max_walk, stream);
        if (rc) return rc;
    }
    if (!R.chunks) return 0;
    const bf16* in = (const bf16*)rkvg;
    const int HD = heads * dim;
    const ChunkScanArgs B{scratch, in + (size_t)2 * Ttot * HD, HD, 0, state, state_stride, 0, dim * dim, cu_q, state_slots, seq_fresh, o, heads, dim, WKV_CHUNK_MIN};
    if (dim == 64) return wkv_chunk_launch<64>(in, dlog, w0, u, prev_off, (const bf16*)x, W, B, Ttot, n_seqs, R.live, scratch, stream);
    return wkv_chunk_launch<128>(in, dlog, w0, u, prev_off, (const bf16*)x, W, B, Ttot, n_seqs, R.live, scratch, stream);
}

FF_EXPORT int ff_wkv_out(const float* o, const void* g, int dtype, const float* norm, float eps, void* y, int T,
                         int heads, int dim, cudaStream_t stream) {
    if (T <= 0) return 0;
    const long long warps = (long long)T * heads;
    const unsigned blocks = (unsigned)((warps + 3) / 4);
    const int es = dtype == 0 ? 4 : 2;
    if ((dim == 64 || dim == 128) && (dtype == 0 || dtype == 1) && (((uintptr_t)o | (uintptr_t)norm) & 15) == 0 &&
        (((uintptr_t)g | (uintptr_t)y) & (4 * es - 1)) == 0) {
        const unsigned n = (unsigned)((warps * (dim / 4) + 255) / 256);
#define FF_WKV_OUT(TT, L) FF_LAUNCH((wkv_out_vec_kernel<TT, L>), n, 256, 0, stream, o, (const TT*)g, norm, eps, (TT*)y, T, heads)
        if (dtype == 0) { if (dim == 64) FF_WKV_OUT(float, 16); else FF_WKV_OUT(float, 32); }
        else { if (dim == 64) FF_WKV_OUT(bf16, 16); else FF_WKV_OUT(bf16, 32); }
#undef FF_WKV_OUT
        FF_LAUNCH_CHECK();
        return 0;
    }
    if (dtype == 0)
        FF_LAUNCH((wkv_out_kernel<float>), blocks, 128, 0, stream, o, (const float*)g, norm, eps, (float*)y, T, heads, dim);
    else if (dtype == 1)
        FF_LAUNCH((wkv_out_kernel<bf16>), blocks, 128, 0, stream, o, (const bf16*)g, norm, eps, (bf16*)y, T, heads, dim);
    else return FF_ERR_BAD_ARG;
    FF_LAUNCH_CHECK();
    return 0;
}
