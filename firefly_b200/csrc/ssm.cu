// Recurrent mixers whose state decays by one scalar per head and token, or by one number per key channel:
//
//   S_t = a_t S_(t-1) + b_t k_t v_t^T        S: [key channel, value channel] per head, 32-bit, starts at 0
//   o_t = S_t^T q_t  (+ D v_t)
//
// Three kinds use it.  A state-space mixer (Mamba-2 style): k = B_t and q = C_t (shared by the heads of a
// group), v = x_t, step = softplus(raw_t + bias), a_t = exp(-exp(A_log) step), b_t = step, with a skip
// term D x_t; its inputs x, B, C come out of a short causal convolution per channel with SiLU
// (`causal_conv_silu_kernel`), whose last taps-1 inputs are part of the request's state.  And linear
// attention with a constant decay per head: a = decay_h, b = 1, q, k, v = SiLU of three projections.  And gated
// linear attention: a_t = diag(alpha_t) with alpha from a low-rank projection (`low_rank_decay_kernel`), b = 1.
//
// The state lives in the request's state slot in 32-bit and is carried from step to step; a fresh request
// starts from zeros.  Decays, steps, S and every sum are 32-bit.  Steps of few tokens walk a sequence token by token;
// bfloat16 prompts are taken a chunk of tokens at a time, whose sums are formed in another order, as right.
#include "chunk_scan.cuh"
#include "common.cuh"
#include "scan_wide.cuh"

namespace ff {

__device__ __forceinline__ float silu_f(float z) { return z / (1.0f + expf(-z)); }
// The same for results that are rounded to 16 bits, by CUDA's fast division (2 units in the last place of 32 bits; 0 where e^-z is
// beyond 2^126, the true result being below 2^-119): 4 of 33 million rounded results differ more than with a true reciprocal.
__device__ __forceinline__ float silu_fast(float z) { return __fdividef(z, 1.0f + expf(-z)); }
__device__ __forceinline__ float softplus_f(float z) { return z > 20.f ? z : log1pf(expf(z)); }

// ----------------------------------------------------------------------------- convolution --
// out[t, c] = act(bias[c] + sum_j w[c, j] * in[t - (taps-1) + j, c]) (+ in[t, c]); inputs in front of the portion
// come from the state slot (`conv_off`: [(taps-1), C] floats, oldest first; zeros for a fresh request).
// `flags`: CONV_SILU the activation is SiLU (else none), CONV_ADD_INPUT the token's own input is added to the
// result (a filter whose output is x + conv(x)).  `bias` may be null.  The output type TO may differ from the
// input's (32-bit rows in, rows of the engine's type out).
// A thread takes VEC neighbouring channels (one 16-byte load where the layout allows it, else one channel)
// and walks `tile` tokens with the last taps-1 inputs in registers, so every input of a long step is read once
// (steps of few tokens get a thread a token, so that they still fill the GPU).
constexpr int CONV_MAX_TAPS = 16;
constexpr int CONV_SILU = 1, CONV_ADD_INPUT = 2;
constexpr int CONV_AHEAD = 4;
constexpr int CONV_BLOCKS = 6, CONV_BLOCKS_ONE = 4;           // blocks an SM, several channels a thread or one

// TAPS > 0: the number of taps is known when the kernel is built (the window stays in registers); 0: any number
// up to CONV_MAX_TAPS.
template <typename T, typename TO, int VEC, int TAPS>
__global__ void __launch_bounds__(128, VEC > 1 ? CONV_BLOCKS : CONV_BLOCKS_ONE) causal_conv_silu_kernel(const T* in, int in_stride, int in_off,
                                        const float* __restrict__ w /*[C,taps]*/, const float* __restrict__ bias,
                                        const float* state, size_t state_stride, int conv_off,
                                        const int* __restrict__ token_seq, const int* __restrict__ cu_q,
                                        const int* __restrict__ state_slots, const int* __restrict__ seq_fresh,
                                        TO* __restrict__ out /*[T,C]*/, int Ttot, int C, int taps_rt, int tile,
                                        int flags) {
    pdl_prologue();
    in = pdl_fresh(in);
    state = pdl_fresh(state);
    constexpr int MT = TAPS ? TAPS : CONV_MAX_TAPS;
    const int taps = TAPS ? TAPS : taps_rt;
    const int c0 = (blockIdx.y * blockDim.x + threadIdx.x) * VEC;
    if (c0 >= C) return;
    const int tile0 = blockIdx.x * tile, tile1 = min(Ttot, tile0 + tile);
    float win[MT > 1 ? MT - 1 : 1][VEC];          // the inputs of the taps-1 tokens in front, oldest first
    float wt[MT][VEC], bs[VEC];
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
        bs[e] = bias ? bias[c0 + e] : 0.f;
        if constexpr (TAPS == 4 && VEC > 1) {         // a channel's four weights in one load (the launcher has seen to the alignment)
            const float4 w4 = *reinterpret_cast<const float4*>(w + (size_t)(c0 + e) * 4);
            wt[0][e] = w4.x; wt[1][e] = w4.y; wt[2][e] = w4.z; wt[3][e] = w4.w;
        } else {
#pragma unroll
            for (int j = 0; j < MT; ++j) wt[j][e] = j < taps ? w[(size_t)(c0 + e) * taps + j] : 0.f;
        }
    }
    struct alignas(VEC * sizeof(T)) Raw { T v[VEC]; };
    auto ask = [&](int tt) { return *reinterpret_cast<const Raw*>(in + (size_t)tt * in_stride + in_off + c0); };      // the inputs of token tt (a row of this step)
    auto load_row = [&](int tt, float* dst) {
        const Raw raw = ask(tt);
#pragma unroll
        for (int e = 0; e < VEC; ++e) dst[e] = to_float(raw.v[e]);
    };
    // the window in front of token t of sequence s: rows of this step where they exist, else the saved rows
    auto fill_window = [&](int t, int s) {
        const int t0 = cu_q[s];
        const bool fresh = seq_fresh[s] != 0;
        const float* st = state + (size_t)state_slots[s] * state_stride + conv_off;
#pragma unroll
        for (int j = 0; j < MT - 1; ++j) {
            if (j < taps - 1) {
                const int tt = t - (taps - 1) + j;
                if (tt >= t0) load_row(tt, win[j]);
                else {
                    const int r = (taps - 1) + (tt - t0);       // row of the saved inputs: 0 oldest
#pragma unroll
                    for (int e = 0; e < VEC; ++e) win[j][e] = fresh ? 0.f : st[(size_t)r * C + c0 + e];
                }
            }
        }
    };
    // The rows and sequences of CONV_AHEAD tokens are asked for together, while the CONV_AHEAD in front of them are worked on: with one at
    // a time the walk waits for memory at every token.  Four channels a thread leave an SM the warps that hide the rest.  8192 tokens
    // of 4096 channels, whose bytes take 21 us: a token at a time 118, four at a time with nothing asked for ahead and eight channels a thread 55, now 50.
    int s_prev = -1;
    float rows[CONV_AHEAD][VEC];
    Raw next[CONV_AHEAD];
    int seqs[CONV_AHEAD], next_seqs[CONV_AHEAD];
    auto ask_ahead = [&](int t) {
#pragma unroll
        for (int a = 0; a < CONV_AHEAD; ++a)
            if (t + a < tile1) {
                next_seqs[a] = token_seq[t + a];
                next[a] = ask(t + a);
            }
    };
    ask_ahead(tile0);
    for (int tb = tile0; tb < tile1; tb += CONV_AHEAD) {
#pragma unroll
      for (int a = 0; a < CONV_AHEAD; ++a) {
        seqs[a] = next_seqs[a];
#pragma unroll
        for (int e = 0; e < VEC; ++e) rows[a][e] = to_float(next[a].v[e]);
      }
      ask_ahead(tb + CONV_AHEAD);
      auto finish = [&](int t, float (&acc)[VEC], const float (&cur)[VEC]) {
        if (flags & CONV_SILU) {
#pragma unroll
            for (int e = 0; e < VEC; ++e) acc[e] = sizeof(TO) == 4 ? silu_f(acc[e]) : silu_fast(acc[e]);
        }
        if (flags & CONV_ADD_INPUT) {
#pragma unroll
            for (int e = 0; e < VEC; ++e) acc[e] += cur[e];
        }
        TO* dst = out + (size_t)t * C + c0;
        if constexpr (VEC == 1) dst[0] = from_float<TO>(acc[0]);
        else {
            struct alignas(VEC * sizeof(TO)) Pack { TO v[VEC]; };
            Pack raw;
#pragma unroll
            for (int e = 0; e < VEC; ++e) raw.v[e] = from_float<TO>(acc[e]);
            *reinterpret_cast<Pack*>(dst) = raw;
        }
      };
      if constexpr (TAPS > 0) {
        // all of them in the sequence the window belongs to: the inputs stand where they were read, nothing slides
        if (tb + CONV_AHEAD <= tile1 && seqs[0] == s_prev && seqs[CONV_AHEAD - 1] == s_prev) {
#pragma unroll
          for (int a = 0; a < CONV_AHEAD; ++a) {
            float acc[VEC];
#pragma unroll
            for (int e = 0; e < VEC; ++e) acc[e] = bs[e];
#pragma unroll
            for (int j = 0; j < MT; ++j) {
              const int from = a - (MT - 1) + j;            // row of this batch, or (negative) of the window
              const float (&x)[VEC] = from >= 0 ? rows[from >= 0 ? from : 0] : win[from < 0 ? MT - 1 + from : 0];
              if constexpr (VEC % 2 == 0) {                 // two channels an instruction
#pragma unroll
                for (int e = 0; e < VEC; e += 2) {
                  const f32x2 r = f2_fma(f2_pack(wt[j][e], wt[j][e + 1]), f2_pack(x[e], x[e + 1]), f2_pack(acc[e], acc[e + 1]));
                  acc[e] = f2_low(r);
                  acc[e + 1] = f2_high(r);
                }
              } else acc[0] += wt[j][0] * x[0];
            }
            finish(tb + a, acc, rows[a]);
          }
#pragma unroll
          for (int j = 0; j < MT - 1; ++j) {
#pragma unroll
            for (int e = 0; e < VEC; ++e) win[j][e] = rows[CONV_AHEAD - (MT - 1) + j][e];
          }
          continue;
        }
      }
#pragma unroll
      for (int a = 0; a < CONV_AHEAD; ++a) {
        const int t = tb + a, s = seqs[a];
        if (t >= tile1) break;
        if (t == tile0 || s != s_prev) fill_window(t, s);
        s_prev = s;
        float cur[VEC], acc[VEC];
#pragma unroll
        for (int e = 0; e < VEC; ++e) { cur[e] = rows[a][e]; acc[e] = bs[e]; }
#pragma unroll
        for (int j = 0; j < MT - 1; ++j)
            if (j < taps - 1) {
#pragma unroll
                for (int e = 0; e < VEC; ++e) acc[e] += wt[j][e] * win[j][e];
            }
#pragma unroll
        for (int j = 0; j < MT; ++j)
            if (j == taps - 1) {
#pragma unroll
                for (int e = 0; e < VEC; ++e) acc[e] += wt[j][e] * cur[e];
            }
        finish(t, acc, cur);
        // slide: the oldest row leaves, the current one comes in
#pragma unroll
        for (int j = 0; j < MT - 1; ++j) {
            if (j < taps - 2) {
#pragma unroll
                for (int e = 0; e < VEC; ++e) win[j][e] = win[j + 1][e];
            } else if (j == taps - 2) {
#pragma unroll
                for (int e = 0; e < VEC; ++e) win[j][e] = cur[e];
            }
        }
      }
    }
}

// The last taps-1 inputs of every sequence, for its next step.  One thread per (sequence, channel) reads what
// it needs of the old rows before it writes.
template <typename T>
__global__ void conv_state_update_kernel(const T* in, int in_stride, int in_off, float* __restrict__ state,
                                         size_t state_stride, int conv_off, const int* __restrict__ cu_q,
                                         const int* __restrict__ state_slots, const int* __restrict__ seq_fresh,
                                         int C, int taps) {
    pdl_prologue();
    in = pdl_fresh(in);
    constexpr int MAX_KEEP = 15;
    const int s = blockIdx.x;
    const int t0 = cu_q[s], t1 = cu_q[s + 1];
    const int keep = taps - 1, n = t1 - t0;
    if (n <= 0) return;
    const bool fresh = seq_fresh[s] != 0;
    float* st = state + (size_t)state_slots[s] * state_stride + conv_off;
    for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < C; c += gridDim.y * blockDim.x) {
        float nv[MAX_KEEP];
#pragma unroll
        for (int r = 0; r < MAX_KEEP; ++r) {
            if (r < keep) {
                const int tt = t1 - keep + r;
                if (tt >= t0) nv[r] = to_float(in[(size_t)tt * in_stride + in_off + c]);
                else nv[r] = fresh ? 0.f : st[(size_t)(keep + (tt - t0)) * C + c];
            }
        }
#pragma unroll
        for (int r = 0; r < MAX_KEEP; ++r)
            if (r < keep) st[(size_t)r * C + c] = nv[r];
    }
}

// ----------------------------------------------------------------------------- the recurrence --
struct ScanArgs {
    const void* q; int q_stride, q_off;          // [T, ...] key-sized rows per group: q_off + group * N + i
    const void* k; int k_stride, k_off;
    const void* v; int v_stride, v_off;          // value rows per head: v_off + h * V + j
    int heads_per_group;                         // heads that share one q/k row (1: a row per head)
    int act;                                     // 1: q, k, v pass SiLU as they are read
    const float* decay;                          // [heads] constant a (mode 0)
    const void* step; int step_stride, step_off; // mode 1: raw step per (token, head)
    const float* step_bias; const float* a_log; const float* skip;   // [heads] each (mode 1; skip may be null)
    int mode;
    // mode 2: the decays themselves, one per key channel, [T, ...] rows of heads * N floats
    const float* channel_decay; int cd_stride, cd_off;
    float q_scale;                               // q is multiplied by this as it is read (behind the activation)
};

// One block per (sequence, head, VB value columns), token by token (scan_wide.cuh).  A chunk's q, k, v and decays are staged in
// 32-bit in one of two buffers; the next chunk's are asked for before the current one is walked and staged behind it, so
// a chunk has one barrier.  CD: mode 2, a decay per key channel (staged beside q and k).
// This is the kernel for steps of few tokens, for 32-bit inputs, for constant decays, for inputs that pass SiLU (both factors of every product
// would have to be split, and on sums that lean to one side, as those of SiLU's do, the tensor cores' cut-off leaves 8e-7 where
// this one leaves 1e-7) and for sizes that the chunked ones do not take.  Against one column a thread: 758 -> 279 us
// for three sequences of 1501, 1000 and 700 tokens with 16 heads of 64 x 128, 1256 -> 745 us for 4 x 2048 tokens, SiLU, 8 heads
// of 128 x 128.
// SOME: sequences of max_len tokens and more go by chunks (else every sequence is this kernel's).
template <typename T, int NP, bool CD, bool SOME>
__global__ void __launch_bounds__(WS_THREADS) scalar_decay_scan_kernel(
    ScanArgs A, float* __restrict__ state, size_t state_stride, int state_off, const int* __restrict__ cu_q,
    const int* __restrict__ state_slots, const int* __restrict__ seq_fresh, float* __restrict__ o /*[T, heads*V]*/,
    int heads, int N, int V, int max_len) {
    pdl_prologue();
    using WS = WideState<NP>;
    constexpr int CH = WS::CH, VB = WS::VB, PQ = CH * NP / WS_THREADS, PV = (CH * VB + WS_THREADS - 1) / WS_THREADS;
    static_assert(CH * NP % WS_THREADS == 0, "a thread stages the same number of elements");
    __shared__ __align__(16) float s_q[2][CH][NP], s_k[2][CH][NP], s_cd[CD ? 2 : 1][CD ? CH : 1][CD ? NP : 4];
    __shared__ __align__(16) f32x2 s_v[2][CH][VB];        // each value twice
    __shared__ float s_a[2][CH], s_d[2][CH];
    const int s = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
    const int j0 = blockIdx.z * VB;
    const int t0 = cu_q[s], t1s = cu_q[s + 1];
    // a sequence that goes by chunks is empty here: a return would put the lengths' way from memory in front of the state's (3.2 -> 3.4 us
    // for eight single tokens of 16 heads of 64 x 128)
    const bool mine = !SOME || t1s - t0 < max_len;
    const int t1 = mine ? t1s : t0;
    WS w;
    w.place(tid);
    float* S_g = state + (size_t)state_slots[s] * state_stride + state_off + (size_t)h * V * NP;
    w.load(S_g, j0, V, seq_fresh[s] != 0);
    const int group = h / A.heads_per_group;
    const T* qp = pdl_fresh((const T*)A.q) + A.q_off + (size_t)group * N;
    const T* kp = pdl_fresh((const T*)A.k) + A.k_off + (size_t)group * N;
    const T* vp = pdl_fresh((const T*)A.v) + A.v_off + (size_t)h * V + j0;
    const T* stepp = pdl_fresh((const T*)A.step);
    const float* cdp = CD ? pdl_fresh(A.channel_decay) + A.cd_off + (size_t)h * N : nullptr;
    const int cols = min(VB, V - j0);
    float a_const = 1.f, rate = 0.f, sbias = 0.f, skip = 0.f;
    if (A.mode == 0) a_const = A.decay[h];
    else if (!CD) { rate = expf(A.a_log[h]); sbias = A.step_bias[h]; skip = A.skip ? A.skip[h] : 0.f; }
    // element u of a thread is flat index tid + u * threads of the chunk's [CH][NP] or [CH][VB]
    T rq[PQ], rk[PQ], rv[PV], rstep = from_float<T>(0.f);
    float rcd[CD ? PQ : 1];
    auto fetch = [&](int c0) {
        const int n = min(CH, t1 - c0);
#pragma unroll
        for (int u = 0; u < PQ; ++u) {
            const int idx = tid + u * WS_THREADS, c = idx / NP, i = idx % NP;
            const bool ok = c < n && i < N;
            rq[u] = ok ? qp[(size_t)(c0 + c) * A.q_stride + i] : from_float<T>(0.f);
            rk[u] = ok ? kp[(size_t)(c0 + c) * A.k_stride + i] : from_float<T>(0.f);
            if constexpr (CD) rcd[u] = ok ? cdp[(size_t)(c0 + c) * A.cd_stride + i] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < PV; ++u) {
            const int idx = tid + u * WS_THREADS, c = idx / VB, jj = idx % VB;
            rv[u] = (idx < CH * VB && c < n && jj < cols) ? vp[(size_t)(c0 + c) * A.v_stride + jj] : from_float<T>(0.f);
        }
        if (A.mode == 1 && tid < n) rstep = stepp[(size_t)(c0 + tid) * A.step_stride + A.step_off + h];
    };
    auto stage = [&](int b, int n) {
#pragma unroll
        for (int u = 0; u < PQ; ++u) {
            const int idx = tid + u * WS_THREADS;
            const float qv = to_float(rq[u]), kv = to_float(rk[u]);
            (&s_q[b][0][0])[idx] = (A.act ? silu_f(qv) : qv) * A.q_scale;
            (&s_k[b][0][0])[idx] = A.act ? silu_f(kv) : kv;
            if constexpr (CD) (&s_cd[b][0][0])[idx] = rcd[u];
        }
#pragma unroll
        for (int u = 0; u < PV; ++u) {
            const float raw = to_float(rv[u]), vv = A.act ? silu_f(raw) : raw;
            if (CH * VB % WS_THREADS == 0 || tid + u * WS_THREADS < CH * VB) (&s_v[b][0][0])[tid + u * WS_THREADS] = f2_pack(vv, vv);
        }
        if (!CD && tid < CH) {
            float a = a_const, d = 1.f;
            if (A.mode == 1 && tid < n) {
                d = softplus_f(to_float(rstep) + sbias);
                a = expf(-rate * d);
            }
            s_a[b][tid] = a;
            s_d[b][tid] = d;
        }
    };
    const int first = w.first();
    const bool owns = w.part < CH * WS_COLS;             // with more threads a column than sums the rest hold copies
    float* oh = o + (size_t)h * V + j0;
    if (t0 < t1) {
        fetch(t0);
        stage(0, min(CH, t1 - t0));
    }
    __syncthreads();
    int b = 0;
    for (int c0 = t0; c0 < t1; c0 += CH, b ^= 1) {
        const int n = min(CH, t1 - c0);
        if (c0 + CH < t1) fetch(c0 + CH);
        auto token = [&](int c, float* part) {
            f32x2 v[WS_COLS];
            WS::values(&s_v[b][c][w.jl * WS_COLS], v);
            if (!CD && A.mode == 1) {
                const f32x2 d = f2_pack(s_d[b][c], s_d[b][c]);
#pragma unroll
                for (int x = 0; x < WS_COLS; ++x) v[x] = f2_mul(v[x], d);
            }
            w.template token<CD, false>(s_q[b][c], s_k[b][c], CD ? s_cd[b][c] : nullptr, CD ? 1.f : s_a[b][c], v, part);
        };
        if (n == CH) {
            float part[CH * WS_COLS];
#pragma unroll
            for (int c = 0; c < CH; ++c) token(c, part + c * WS_COLS);
            w.reduce_chunk(part);
#pragma unroll
            for (int r = 0; r < WS::OUTS; ++r) {
                const int at = first + r, c = at / WS_COLS, jj = w.jl * WS_COLS + at % WS_COLS;
                if (owns && j0 + jj < V)
                    oh[(size_t)(c0 + c) * heads * V + jj] = skip != 0.f ? part[r] + skip * f2_low(s_v[b][c][jj]) : part[r];
            }
        } else {
            for (int c = 0; c < n; ++c) {
                float part[WS_COLS];
                token(c, part);
                const float y = w.reduce(part);
                const int jj = w.jl * WS_COLS + w.col();
                if (w.part < 4 && j0 + jj < V)
                    oh[(size_t)(c0 + c) * heads * V + jj] = skip != 0.f ? y + skip * f2_low(s_v[b][c][jj]) : y;
            }
        }
        if (c0 + CH < t1) stage(b ^ 1, min(CH, t1 - c0 - CH));
        __syncthreads();
    }
    if (mine) w.store(S_g, j0, V);
}

// ------------------------------------------------------------------- the recurrence, a chunk of tokens at a time --
// Mode 1 over prompts, bfloat16 inputs that are read as they are.  With L_t the sum of the logarithms of the decays up
// to token t of a chunk and S the state in front of it:
//
//   P_ts = (q_t . k_s) exp(L_t - L_s) b_s   for s <= t
//   o_t  = exp(L_t) S^T q_t + sum_s P_ts v_s
//   S   <- exp(L_end) S + sum_s exp(L_end - L_s) b_s k_s v_s^T
//
// Every exponent is a difference that is never positive, formed from sums held in twice 32 bits, so it is as right as the
// product of the decays it stands for.  The four sums over key channels or tokens run on the tensor cores in 32-bit
// out of bfloat16 products (chunk_mma.cuh); S never leaves the registers.
// P, the decays' sums and what follows from them do not hold S: a first kernel forms them for all chunks of the step at once and
// leaves them as records in scratch memory.  The second one walks a sequence's chunks: one block per (sequence, head, VB = 16 W
// value columns), whose warps hold S^T as the accumulators of mma.sync; the same registers are, split, the left operand of
// S^T q, so the state goes nowhere between the products.
// Measured on 4 x 2048 tokens, 32 heads of 128 x 64: token by token with one column a thread 1552 us; the two kernels 33 + 143.
constexpr int SC_C = 32;                                  // tokens a chunk
// Tokens from which a sequence goes by chunks.  us for n sequences of L tokens, chunks / token by token, 32 heads of 128 x 64 (in one
// group or in eight the same):
//   L     n = 1         4             8             16            32
//   24    9.5 / 7.9     11.6 / 11.6   16.5 / 17.1   25.7 / 26.7   42.9 / 48.8
//   32    9.7 / 9.9     12.2 / 14.6   16.9 / 21.8   26.1 / 34.4   44.3 / 63.1
//   64    11.6 / 17.9   14.9 / 26.9   22.4 / 41.1   37.3 / 65.2   63.8 / 121
// and for a decay per key channel, 16 heads of 64 x 128:
//   32    7.3 / 7.3     11.7 / 9.9    14.3 / 12.7   19.6 / 17.9   28.6 / 28.6
//   48    8.3 / 10.1    13.8 / 13.8   16.5 / 17.9   23.5 / 25.5   39.5 / 41.1
//   64    8.8 / 12.8    14.8 / 17.5   18.3 / 23.3   26.5 / 33.3   47.5 / 53.7
constexpr int SCAN_CHUNK_MIN = 32;
constexpr int CHANNEL_CHUNK_MIN = 48;
constexpr int SC_PP = SC_C + 8;
constexpr long long SCAN_PREPARE_BLOCKS = 12 * 148;         // blocks of the first kernel that are on the GPU together

struct ScanRecord {
    bf16 P[3][SC_C * SC_PP];
    float e[SC_C], w[SC_C], end[4];                       // exp(L_t), exp(L_end - L_s) b_s, exp(L_end)
};
static_assert(sizeof(ScanRecord) % 16 == 0, "a record is copied in 16-byte pieces");

// The first kernel: a block per (chunk, group of heads that share q and k, share of the group's heads).  Three of its warps multiply q
// with k once for them; then four heads at a time, a warp a head sums up the decays and each tile of the product is scaled for each
// head.  Four heads take 4 us whatever else runs, so a group's heads go to as many blocks as still fit the GPU together, each with the
// product of its own (SCAN_PREPARE_BLOCKS).  Both kernels, us a call, 64 heads of 64 x 64 in one group, all heads of a group in one
// block / now: one prompt of 64 tokens 64.0 / 18.6, eight of 256 106 / 58.8; 32 heads of 128 x 64: 35.8 / 23.7 and 71.8 / 53.4.
template <int NK>
__global__ void __launch_bounds__(128) scalar_decay_prepare_kernel(ScanArgs A, ScanRecord* __restrict__ recs, const int* __restrict__ cu_q,
                                                                   int n_seqs, int min_len, int heads, int heads_a_block) {
    pdl_prologue();
    constexpr int QP = NK + 8;
    __shared__ __align__(16) bf16 sq[SC_C * QP], sk[SC_C * QP];
    __shared__ float lh[4][SC_C], ll[4][SC_C], sb[4][SC_C];
    int s, chunk, row0, left;
    chunk_of_record<SC_C>(cu_q, n_seqs, blockIdx.x, min_len, s, chunk, row0, left);
    if (chunk < 0) return;
    const int group = blockIdx.y, n = min(SC_C, left);
    const int hb0 = blockIdx.z * heads_a_block, hb1 = min(A.heads_per_group, hb0 + heads_a_block);       // heads of the group
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c2 = (lane & 3) * 2;
    const int row_a = (lane & 7) + ((lane >> 3) & 1) * 8, col_a = (lane >> 4) * 8;
    const int row_b = (lane & 7) + (lane >> 4) * 8, col_b = ((lane >> 3) & 1) * 8;
    const bf16* qp = pdl_fresh((const bf16*)A.q) + A.q_off + (size_t)group * NK;
    const bf16* kp = pdl_fresh((const bf16*)A.k) + A.k_off + (size_t)group * NK;
    const bf16* stepp = pdl_fresh((const bf16*)A.step) + A.step_off;
    for (int idx = threadIdx.x; idx < SC_C * (NK / 8); idx += 128) {
        const int r = idx / (NK / 8), c = (idx % (NK / 8)) * 8;
        const bool in = r < n;
        cm_copy16(sq + r * QP + c, qp + (size_t)(row0 + (in ? r : 0)) * A.q_stride + c, in);
        cm_copy16(sk + r * QP + c, kp + (size_t)(row0 + (in ? r : 0)) * A.k_stride + c, in);
    }
    cm_copy_commit();
    // P's tiles: rows (tokens) 16 mt.., columns (keys) 16 nh..; keys behind the tokens are not formed
    const int mt = warp >> 1, nh = warp & 1;
    float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    for (int h0 = hb0; h0 < hb1; h0 += 4) {
        if (h0 + warp < hb1) {                            // the decays of a head, one token a lane
            const int h = group * A.heads_per_group + h0 + warp;
            ScanRecord* rec = recs + (size_t)blockIdx.x * heads + h;
            const bool in = lane < n;
            const float rate = expf(A.a_log[h]);
            const float dt = in ? softplus_f(to_float(stepp[(size_t)(row0 + lane) * A.step_stride + h]) + A.step_bias[h]) : 0.f;
            // at most e^-200 a token: 0 in 32 bits, and the sums stay exact enough to be subtracted from one another
            double L = in ? (double)(-rate * dt < -200.f ? -200.f : -rate * dt) : 0.0;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const double up = __shfl_up_sync(0xffffffffu, L, off);
                if (lane >= off) L += up;
            }
            const double Lend = __shfl_sync(0xffffffffu, L, 31);
            const float hi = (float)L;
            lh[warp][lane] = hi;
            ll[warp][lane] = (float)(L - (double)hi);
            sb[warp][lane] = dt;
            rec->e[lane] = expf(hi) * A.q_scale;
            rec->w[lane] = dt * expf((float)(Lend - L));
            if (lane == 0) rec->end[0] = expf((float)Lend);
        }
        if (h0 == hb0) {
            cm_copy_wait<0>();
            __syncthreads();
            if (nh <= mt) {
#pragma unroll
                for (int kk = 0; kk < NK / 16; ++kk) {
                    uint32_t a[1][4], b[1][4];
                    cm_ldsm4(a[0], sq + (mt * 16 + row_a) * QP + kk * 16 + col_a);
                    cm_ldsm4(b[0], sk + (nh * 16 + row_b) * QP + kk * 16 + col_b);
                    cm_mma_rows(acc, acc, a, b);
                }
            }
        } else __syncthreads();
        if (nh <= mt) {
            for (int hw = 0; hw < min(4, hb1 - h0); ++hw) {
                const int h = group * A.heads_per_group + h0 + hw;
                bf16* Pd = recs[(size_t)blockIdx.x * heads + h].P[0];
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const int t = mt * 16 + g + r * 8, u = nh * 16 + nt * 8 + c2;
                        float x[2];
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int us = u + e;
                            float d = 0.f;
                            if (us <= t) d = expf((lh[hw][t] - lh[hw][us]) + (ll[hw][t] - ll[hw][us])) * sb[hw][us];
                            // a key behind the token counts nothing, whatever its product is
                            x[e] = us <= t ? acc[nt][r * 2 + e] * (d * A.q_scale) : 0.f;
                        }
                        uint32_t p0, p1, p2;
                        cm_split3(x[0], x[1], p0, p1, p2);
                        uint32_t* dst = reinterpret_cast<uint32_t*>(Pd + t * SC_PP + u);
                        dst[0] = p0;
                        dst[SC_C * SC_PP / 2] = p1;
                        dst[SC_C * SC_PP] = p2;
                    }
                }
            }
        }
        __syncthreads();
    }
}

template <int NK, int W>
struct ScanChunkSmem {
    static constexpr int QP = NK + 8, VP = 16 * W + 8;    // row pitches: 16-byte pieces of 8 rows lie in different banks
    struct Stage { ScanRecord rec; bf16 q[SC_C * QP], k[SC_C * QP], v[SC_C * VP]; };
    Stage stage[3];                                       // walked, there, on its way
    float xch[2][2 * W][8][32];
};

// The second kernel; two warps hold the keys' halves of 16 value columns and exchange their shares of S^T q, each for the tokens (16
// of 32) that the other goes on with, as in chunk_scan.cuh.
template <int NK, int W>
__global__ void __launch_bounds__(64 * W + CS_LOADERS) scalar_decay_chunk_kernel(
    ScanArgs A, const ScanRecord* recs_, float* __restrict__ state, size_t state_stride, int state_off, const int* __restrict__ cu_q,
    const int* __restrict__ state_slots, const int* __restrict__ seq_fresh, float* __restrict__ o /*[T, heads*V]*/,
    int heads, int V, int min_len) {
    pdl_prologue();
    using SM = ScanChunkSmem<NK, W>;
    constexpr int QP = SM::QP, VP = SM::VP, PP = SC_PP, NT = NK / 16, VB = 16 * W;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SM& sm = *reinterpret_cast<SM*>(smem_raw);
    const int s = blockIdx.x, h = blockIdx.y, j0 = blockIdx.z * VB;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t0 = cu_q[s], len = cu_q[s + 1] - t0, chunks = (len + SC_C - 1) / SC_C;
    if (len < min_len) return;
    if (warp >= 2 * W) {
        // ---- the warps that load
        const int pt = threadIdx.x - 64 * W, group = h / A.heads_per_group;
        const ScanRecord* recs = pdl_fresh(recs_) + (size_t)chunk_first_record<SC_C>(t0, s) * heads + h;
        const bf16* qp = pdl_fresh((const bf16*)A.q) + A.q_off + (size_t)group * NK;
        const bf16* kp = pdl_fresh((const bf16*)A.k) + A.k_off + (size_t)group * NK;
        const bf16* vp = pdl_fresh((const bf16*)A.v) + A.v_off + (size_t)h * V + j0;
        auto load = [&](int i) {                          // ask for chunk i's record and q, k, v (zeros behind the sequence's end)
            if (i < chunks) {
                typename SM::Stage& st = sm.stage[i % 3];
                const int n = len - i * SC_C;
                const size_t row0 = (size_t)(t0 + i * SC_C);
                const unsigned char* src = reinterpret_cast<const unsigned char*>(recs + (size_t)i * heads);
#pragma unroll 8
                for (int p = pt; p < (int)(sizeof(ScanRecord) / 16); p += CS_LOADERS)
                    cm_copy16(reinterpret_cast<unsigned char*>(&st.rec) + p * 16, src + p * 16, true);
#pragma unroll 4
                for (int idx = pt; idx < SC_C * (NK / 8); idx += CS_LOADERS) {
                    const int r = idx / (NK / 8), c = (idx % (NK / 8)) * 8;
                    const bool in = r < n;
                    const size_t row = in ? row0 + r : (size_t)t0;
                    cm_copy16(st.q + r * QP + c, qp + row * A.q_stride + c, in);
                    cm_copy16(st.k + r * QP + c, kp + row * A.k_stride + c, in);
                }
                for (int idx = pt; idx < SC_C * (VB / 8); idx += CS_LOADERS) {
                    const int r = idx / (VB / 8), c = (idx % (VB / 8)) * 8;
                    const bool in = r < n && j0 + c < V;
                    cm_copy16(st.v + r * VP + c, vp + (in ? (row0 + r) * A.v_stride + c : 0), in);
                }
            }
            cm_copy_commit();
        };
        load(0);
        load(1);
        for (int i = 0; i < chunks; ++i) {
            cm_copy_wait<1>();
            __syncthreads();                              // chunk i is there, and everybody is done with chunk i - 1
            load(i + 2);
        }
        cm_copy_wait<0>();
        return;
    }
    // ---- the warps that hold S^T
    const int tile = warp % W, half = warp / W, other = tile + (1 - half) * W, k0 = half * (NK / 2);
    const int g = lane >> 2, c2 = (lane & 3) * 2;
    // where ldmatrix finds the four 8 x 8 tiles of a lane's row: the second one 8 rows down and the third 8 columns on (a),
    // or the second 8 columns on and the third 8 rows down (b)
    const int row_a = (lane & 7) + ((lane >> 3) & 1) * 8, col_a = (lane >> 4) * 8;
    const int row_b = (lane & 7) + (lane >> 4) * 8, col_b = ((lane >> 3) & 1) * 8;
    float* S_g = state + (size_t)state_slots[s] * state_stride + state_off + (size_t)h * V * NK + k0;      // [V][NK]
    const bool fresh = seq_fresh[s] != 0;
    const int jr[2] = {j0 + tile * 16 + g, j0 + tile * 16 + g + 8};
    float S[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
            S[nt][e] = (fresh || jr[e >> 1] >= V) ? 0.f : S_g[(size_t)jr[e >> 1] * NK + nt * 8 + c2 + (e & 1)];
    }
    const int ld = heads * V, t_own = half * 16 + c2;
    float* op = o + (size_t)(t0 + t_own) * ld + (size_t)h * V + jr[0];
    const bool all_cols = j0 + VB <= V;
    const float skip = A.skip ? A.skip[h] : 0.f;
    for (int i = 0; i < chunks; ++i) {
        __syncthreads();
        const typename SM::Stage& st = sm.stage[i % 3];
        const int n = min(SC_C, len - i * SC_C);
        float acc[4][4], low[4][4];                       // o^T, and the sum of its small terms
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[nt][e] = low[nt][e] = 0.f;
        }
        // S^T q
#pragma unroll
        for (int kk = 0; kk < NK / 32; ++kk) {
            uint32_t a[3][4], r[1][4];
            cm_split3(S[2 * kk][0], S[2 * kk][1], a[0][0], a[1][0], a[2][0]);
            cm_split3(S[2 * kk][2], S[2 * kk][3], a[0][1], a[1][1], a[2][1]);
            cm_split3(S[2 * kk + 1][0], S[2 * kk + 1][1], a[0][2], a[1][2], a[2][2]);
            cm_split3(S[2 * kk + 1][2], S[2 * kk + 1][3], a[0][3], a[1][3], a[2][3]);
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                cm_ldsm4(r[0], st.q + (t * 16 + row_b) * QP + k0 + kk * 16 + col_b);
                cm_mma_rows(&acc[2 * t], &low[2 * t], a, r);
            }
        }
        float own[2][4], own_low[2][4];                   // the own sixteen tokens
        {
            float (*mine)[32] = sm.xch[i & 1][warp];
            const float (*theirs)[32] = sm.xch[i & 1][other];
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) cm_add(acc[nt], low[nt]);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
                for (int e = 0; e < 4; ++e) mine[nt * 4 + e][lane] = half ? acc[nt][e] : acc[2 + nt][e];
            }
            cm_barrier(1 + tile, 64);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    own[nt][e] = (half ? acc[2 + nt][e] : acc[nt][e]) + theirs[nt * 4 + e][lane];
                    own_low[nt][e] = 0.f;
                }
                cm_scale(own[nt], *reinterpret_cast<const f32x2*>(&st.rec.e[nt * 8 + t_own]));
            }
        }
        // the chunk's values, V^T: 16 value columns x 32 tokens
        uint32_t va[2][1][4];
        bool odd = false;
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            cm_ldsm4t(va[b][0], st.v + (b * 16 + row_b) * VP + tile * 16 + col_b);
#pragma unroll
            for (int r = 0; r < 4; ++r) odd |= cm_not_finite(va[b][0][r]);
        }
        if (!__any_sync(0xffffffffu, odd)) {
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                if (b <= half) {                          // tokens of the first half do not see keys of the second
                    uint32_t r[3][4];
#pragma unroll
                    for (int p = 0; p < 3; ++p) cm_ldsm4(r[p], st.rec.P[p] + (half * 16 + row_b) * PP + b * 16 + col_b);
                    cm_mma_rows(own, own_low, va[b], r);
                }
            }
        } else {
            // a value that is not finite must not reach the tokens in front of it through a product with zero
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int t = nt * 8 + t_own + (e & 1), col = tile * 16 + g + (e >> 1) * 8;
                    for (int u = 0; u <= t; ++u) {
                        float pv = 0.f;
                        for (int p = 2; p >= 0; --p) pv += to_float(st.rec.P[p][t * PP + u]);
                        own[nt][e] += pv * to_float(st.v[u * VP + col]);
                    }
                }
            }
        }
        // the skip term: V^T lies in the registers of a left operand as an accumulator does
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            float* d = &own[r >> 1][(r & 1) * 2];
            const float* l = &own_low[r >> 1][(r & 1) * 2];
            const uint32_t v = half ? va[1][0][r] : va[0][0][r];
            d[0] = d[0] + l[0];
            d[1] = d[1] + l[1];
            if (skip != 0.f) { d[0] += skip * cm_lo(v); d[1] += skip * cm_hi(v); }
        }
        if (n == SC_C && all_cols) {
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
                for (int e = 0; e < 4; ++e) op[(size_t)(nt * 8 + (e & 1)) * ld + (e >> 1) * 8] = own[nt][e];
            }
        } else {
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (nt * 8 + t_own + (e & 1) < n && jr[e >> 1] < V) op[(size_t)(nt * 8 + (e & 1)) * ld + (e >> 1) * 8] = own[nt][e];
            }
        }
        op += (size_t)SC_C * ld;
        // S <- end S + sum_s (w_s v_s) k_s
        const float end = st.rec.end[0];
        uint32_t wa[2][3][4];
#pragma unroll
        for (int b = 0; b < 2; ++b) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float2 w2 = *reinterpret_cast<const float2*>(&st.rec.w[b * 16 + (r >> 1) * 8 + c2]);
                cm_split3(cm_lo(va[b][0][r]) * w2.x, cm_hi(va[b][0][r]) * w2.y, wa[b][0][r], wa[b][1][r], wa[b][2][r]);
            }
        }
#pragma unroll
        for (int m = 0; m < NK / 32; ++m) {
            float sl[2][4];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                cm_scale(S[2 * m + nt], f2_pack(end, end));
#pragma unroll
                for (int e = 0; e < 4; ++e) sl[nt][e] = 0.f;
            }
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                uint32_t r[1][4];
                cm_ldsm4t(r[0], st.k + (b * 16 + row_a) * QP + k0 + m * 16 + col_a);
                cm_mma_rows(&S[2 * m], sl, wa[b], r);
            }
            cm_add(S[2 * m], sl[0]);
            cm_add(S[2 * m + 1], sl[1]);
        }
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (jr[e >> 1] < V) S_g[(size_t)jr[e >> 1] * NK + nt * 8 + c2 + (e & 1)] = S[nt][e];
    }
}

// Mode 2 over bfloat16 prompts: sixteen tokens at a time (chunk_scan.cuh).  This is the first kernel: a block per (CF_WARPS warps of
// records, head).
template <int NK>
__global__ void __launch_bounds__(32 * CF_WARPS) channel_decay_prepare_kernel(ScanArgs A, ChunkRecord<NK, false>* __restrict__ recs,
                                                                              const int* __restrict__ cu_q, int n_seqs, int n_records, int min_len,
                                                                              int heads) {
    pdl_prologue();
    __shared__ __align__(16) ChunkForm<NK, false> form[cf_records<NK>()];
    constexpr int WR = cf_warps_a_record<NK>();
    const int h = blockIdx.y, group = h / A.heads_per_group, warp = threadIdx.x / 32 % WR, c = warp * 64 + 2 * (threadIdx.x & 31);
    const int r = blockIdx.x * cf_records<NK>() + threadIdx.x / (32 * WR);
    if (r >= n_records) return;
    int s, chunk, t0, left;
    chunk_of_record(cu_q, n_seqs, r, min_len, s, chunk, t0, left);
    if (chunk < 0) return;
    const bf16* qp = pdl_fresh((const bf16*)A.q) + A.q_off + (size_t)group * NK + c + (size_t)t0 * A.q_stride;
    const bf16* kp = pdl_fresh((const bf16*)A.k) + A.k_off + (size_t)group * NK + c + (size_t)t0 * A.k_stride;
    const float* ap = pdl_fresh(A.channel_decay) + A.cd_off + (size_t)h * NK + c + (size_t)t0 * A.cd_stride;
    uint32_t qv[CS_C], kv[CS_C];
    float2 av[CS_C];
#pragma unroll
    for (int t = 0; t < CS_C; ++t) {
        const bool in = t < left;
        qv[t] = in ? *reinterpret_cast<const uint32_t*>(qp + (size_t)t * A.q_stride) : 0u;
        kv[t] = in ? *reinterpret_cast<const uint32_t*>(kp + (size_t)t * A.k_stride) : 0u;
        av[t] = in ? *reinterpret_cast<const float2*>(ap + (size_t)t * A.cd_stride) : make_float2(1.f, 1.f);
    }
    ChunkForm<NK, false>& sh = form[threadIdx.x / (32 * WR)];
    ChunkRecord<NK, false>* rec = recs + (size_t)r * heads + h;
    const f32x2 scale = f2_pack(A.q_scale, A.q_scale);
    chunk_form<NK, false, false>(rec, sh, warp, 0ull, [&](int t, f32x2& q, f32x2& k, f32x2& a) {
        q = f2_mul(cf_pair(qv[t]), scale);
        k = cf_pair(kv[t]);
        a = f2_pack(av[t].x, av[t].y);
    });
    cf_sync<NK>();
    chunk_emit<NK, WR>(rec->P[0], sh.P);
}

// ------------------------------------------------------------------- decays from a low-rank projection --
// alpha[t, c] = sigmoid(z)^(1 / tau), z = sum_r low[t, r] * w[c, r] + bias[c], all in 32-bit: exp(-softplus(-z) / tau).
// A thread keeps one channel's row of w in registers (up to LRD_R of it at a time) and walks a tile of tokens, LRD_U of
// them at once, whose low rows stand in shared memory, two tokens side by side for the instructions that take two sums.
// Bound by instructions, of which one sum at a time made a third more, and by weights that were asked for two bytes at a
// time.  4140 tokens of 1024 channels 21.2 us, now 14.2; 1000 tokens 7.9, now 5.0.
constexpr int LRD_TOK = 32, LRD_U = 4, LRD_THREADS = 128, LRD_R = 16;

template <typename T>
__global__ void __launch_bounds__(LRD_THREADS) low_rank_decay_kernel(const T* low, int low_stride, int low_off,
                                                                     const T* __restrict__ w, const float* __restrict__ bias,
                                                                     float inv_tau, float* __restrict__ alpha, int Ttot, int C,
                                                                     int R, int tile, int w_pieces /*16 bytes of w at a time*/) {
    extern __shared__ __align__(16) float s_low[];            // [tile / 2][Rp][2], rows filled up to Rp = a multiple of LRD_R with zeros
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int Rp = (R + LRD_R - 1) / LRD_R * LRD_R;
    const int t0 = blockIdx.x * tile, n = min(tile, Ttot - t0);
    const int c = blockIdx.y * LRD_THREADS + threadIdx.x;
    const T* wr = w + (size_t)min(c, C - 1) * R;
    const float b = bias[min(c, C - 1)];
    float wv[LRD_R];
    auto weights = [&](int r0) {
        constexpr int N = 16 / (int)sizeof(T);
        struct alignas(16) Piece { T v[N]; };
        if (w_pieces) {
#pragma unroll
            for (int r = 0; r < LRD_R; r += N) {
                const bool in = r0 + r < R;
                const Piece p = *reinterpret_cast<const Piece*>(wr + (in ? r0 + r : 0));
#pragma unroll
                for (int k = 0; k < N; ++k) wv[r + k] = in ? to_float(p.v[k]) : 0.f;
            }
        } else {
#pragma unroll
            for (int r = 0; r < LRD_R; ++r) wv[r] = r0 + r < R ? to_float(wr[r0 + r]) : 0.f;
        }
    };
    weights(0);                                               // weights do not depend on the kernel in front
    asm volatile("griddepcontrol.wait;" ::: "memory");
    low = pdl_fresh(low);
    for (int idx = threadIdx.x; idx < tile * Rp; idx += LRD_THREADS) {
        const int u = idx / Rp, r = idx - u * Rp;
        s_low[((u >> 1) * Rp + r) * 2 + (u & 1)] = (u < n && r < R) ? to_float(low[(size_t)(t0 + u) * low_stride + low_off + r]) : 0.f;
    }
    __syncthreads();
    if (c >= C) return;
    float* to = alpha + (size_t)t0 * C + c;
    for (int u0 = 0; u0 < n; u0 += LRD_U, to += (size_t)LRD_U * C) {
        f32x2 acc[LRD_U / 2];
#pragma unroll
        for (int u = 0; u < LRD_U / 2; ++u) acc[u] = f2_pack(0.f, 0.f);
        for (int r0 = 0; r0 < Rp; r0 += LRD_R) {
            if (Rp > LRD_R) weights(r0);
#pragma unroll
            for (int u = 0; u < LRD_U / 2; ++u) {
                const float4* l = reinterpret_cast<const float4*>(s_low + ((size_t)(u0 / 2 + u) * Rp + r0) * 2);
#pragma unroll
                for (int r = 0; r < LRD_R; r += 2) {
                    const float4 l4 = l[r / 2];                // channel r of both tokens, then r + 1
                    acc[u] = f2_fma(f2_pack(wv[r], wv[r]), f2_pack(l4.x, l4.y), acc[u]);
                    acc[u] = f2_fma(f2_pack(wv[r + 1], wv[r + 1]), f2_pack(l4.z, l4.w), acc[u]);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < LRD_U; ++u)
            if (u0 + u < n) {
                const float z = (u & 1 ? f2_high(acc[u / 2]) : f2_low(acc[u / 2])) + b;
                // softplus(-z) = -ln sigmoid(z), right to about 1e-7 absolutely, which is a relative 1e-7 / tau of alpha: the decays of
                // thousands of tokens are multiplied, so not with the fast exponential and logarithm (4e-7)
                const float sp = fmaxf(-z, 0.f) + logf(1.0f + expf(-fabsf(z)));
                to[(size_t)u * C] = expf(-sp * inv_tau);
            }
    }
}

// ----------------------------------------------------------------------------- gate and norm --
// One block per (token, part).  order 0: y = rms(o * silu(z)) * w  (the gate in front of the norm, norm over
// each of `parts` equal parts);  order 1: y = rms(o) * w * sigmoid(z)  (the gate behind it).
template <typename T>
__global__ void gated_rms_norm_kernel(const float* o, const T* z, int z_stride, int z_off,
                                      const float* __restrict__ w, float eps, T* __restrict__ y, int width, int parts,
                                      int order) {
    pdl_prologue();
    o = pdl_fresh(o);
    z = pdl_fresh(z);
    __shared__ float scratch[32];
    const int t = blockIdx.x, g = blockIdx.y;
    const int per = width / parts;
    const float* orow = o + (size_t)t * width + (size_t)g * per;
    const T* zrow = z + (size_t)t * z_stride + z_off + (size_t)g * per;
    float ss = 0.f;
    for (int i = threadIdx.x; i < per; i += blockDim.x) {
        float v = orow[i];
        if (order == 0) v *= silu_f(to_float(zrow[i]));
        ss += v * v;
    }
    ss = block_sum(ss, scratch);
    const float inv = 1.0f / sqrtf(ss / (float)per + eps);
    T* yrow = y + (size_t)t * width + (size_t)g * per;
    for (int i = threadIdx.x; i < per; i += blockDim.x) {
        const float zv = to_float(zrow[i]);
        float v = orow[i];
        if (order == 0) v = v * silu_f(zv) * inv * w[g * per + i];
        else v = v * inv * w[g * per + i] / (1.0f + expf(-zv));
        yrow[i] = from_float<T>(v);
    }
}

// The same where a part is 128 to 4096 values in steps of 128 and everything lies on 16 bytes: TP threads a part (whole warps), each with
// its values in registers between the sum and the writes, four at a time (the kernel above reads everything twice and has a
// block of its own for every 256 values): 90 -> 31 us on 8192 rows of 2048 values in 8 parts, whose bytes take 20.
template <typename T, int TP, int MAXV>
__global__ void __launch_bounds__(256) gated_rms_norm_vec_kernel(const float* o, const T* z, int z_stride, int z_off, const float* __restrict__ w,
                                                                 float eps, T* __restrict__ y, int rows, int width, int parts, int order) {
    pdl_prologue();
    o = pdl_fresh(o);
    z = pdl_fresh(z);
    __shared__ float scratch[8];
    const int per = width / parts, lane = threadIdx.x % TP;
    const long long item = (long long)blockIdx.x * (256 / TP) + threadIdx.x / TP;       // row * parts + part
    const bool live = item < (long long)rows * parts;
    const int t = live ? (int)(item / parts) : 0, g = live ? (int)(item % parts) : 0;
    const float* orow = o + (size_t)t * width + (size_t)g * per;
    const T* zrow = z + (size_t)t * z_stride + z_off + (size_t)g * per;
    struct alignas(4 * sizeof(T)) Four { T v[4]; };
    float4 ov[MAXV];
    Four zv[MAXV];
#pragma unroll
    for (int m = 0; m < MAXV; ++m) {
        const int i = (m * TP + lane) * 4;
        if (i < per) {
            ov[m] = *reinterpret_cast<const float4*>(orow + i);
            zv[m] = *reinterpret_cast<const Four*>(zrow + i);
        }
    }
    float ss = 0.f;
#pragma unroll
    for (int m = 0; m < MAXV; ++m) {
        if ((m * TP + lane) * 4 < per) {
            if (order == 0) {
                ov[m].x *= silu_f(to_float(zv[m].v[0]));
                ov[m].y *= silu_f(to_float(zv[m].v[1]));
                ov[m].z *= silu_f(to_float(zv[m].v[2]));
                ov[m].w *= silu_f(to_float(zv[m].v[3]));
            }
            ss += (ov[m].x * ov[m].x + ov[m].y * ov[m].y) + (ov[m].z * ov[m].z + ov[m].w * ov[m].w);
        }
    }
    ss = warp_sum(ss);
    if constexpr (TP > 32) {                             // the block is one part: 256 threads
        if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = ss;
        __syncthreads();
        ss = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) ss += scratch[i];
    }
    if (!live) return;
    const float inv = 1.0f / sqrtf(ss / (float)per + eps);
    T* yrow = y + (size_t)t * width + (size_t)g * per;
#pragma unroll
    for (int m = 0; m < MAXV; ++m) {
        const int i = (m * TP + lane) * 4;
        if (i < per) {
            const float4 w4 = *reinterpret_cast<const float4*>(w + g * per + i);
            const float wv[4] = {w4.x, w4.y, w4.z, w4.w}, v[4] = {ov[m].x, ov[m].y, ov[m].z, ov[m].w};
            Four out;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float r = v[e] * inv * wv[e];
                out.v[e] = from_float<T>(order == 0 ? r : r / (1.0f + expf(-to_float(zv[m].v[e]))));
            }
            *reinterpret_cast<Four*>(yrow + i) = out;
        }
    }
}

}  // namespace ff

using namespace ff;

template <typename T, typename TO>
static int conv_launch(const void* in, int in_stride, int in_off, const float* w, const float* bias, float* state,
                       long long state_stride, int conv_off, const int* token_seq, const int* cu_q, const int* state_slots,
                       const int* seq_fresh, void* out, int T_, int n_seqs, int C, int taps, int flags,
                       cudaStream_t stream) {
    constexpr int V = 16 / (int)sizeof(T), PER = 4;
    const bool vec = taps >= 2 && taps <= 4 && C % V == 0 && in_off % V == 0 && in_stride % V == 0 &&
                     (((uintptr_t)in | (uintptr_t)out | (uintptr_t)w) & 15) == 0;
    const int per = vec ? PER : 1;
    const int lanes = (C + per - 1) / per;
    const int threads = lanes >= 128 ? 128 : ((lanes + 31) / 32) * 32;
    // A thread's weights are read once for its tile of tokens; few tokens get small tiles, so that they still fill the GPU.  Longer steps get the
    // tile (up to 48) with which the blocks fill the GPU's places a whole number of times: at 32 whatever the rest, 8192 tokens of 2048 channels
    // were 1.15 rounds of blocks, 31 us (now 28), and of 4096 channels 2.3, 51 us (now 50, of instructions); 2048 tokens of 4096 channels at 4 21 us (now 17).
    const int cols = (lanes + threads - 1) / threads;
    int tile = 1;
    if (T_ >= 512) {
        int dev = 0, sms = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return (int)e;
        const int places = max(1, sms * (vec ? CONV_BLOCKS : CONV_BLOCKS_ONE) / cols), rounds = (T_ + places * 48 - 1) / (places * 48);
        tile = ((T_ + places * rounds - 1) / (places * rounds) + CONV_AHEAD - 1) / CONV_AHEAD * CONV_AHEAD;
    }
    dim3 grid((T_ + tile - 1) / tile, cols);
#define FF_CONV(VV, TT)                                                                                              \
    FF_LAUNCH((causal_conv_silu_kernel<T, TO, VV, TT>), grid, threads, 0, stream, (const T*)in, in_stride, in_off, w, bias, \
              (const float*)state, (size_t)state_stride, conv_off, token_seq, cu_q, state_slots, seq_fresh, (TO*)out, T_, C, taps, \
              tile, flags)
    if (vec) {
        switch (taps) {
            case 2: FF_CONV(PER, 2); break;
            case 3: FF_CONV(PER, 3); break;
            case 4: FF_CONV(PER, 4); break;
            default: return FF_ERR_BAD_ARG;      // not reached: `vec` holds only for 2 to 4 taps
        }
    } else {
        switch (taps) {
            case 2: FF_CONV(1, 2); break;
            case 3: FF_CONV(1, 3); break;
            case 4: FF_CONV(1, 4); break;
            default: FF_CONV(1, 0); break;
        }
    }
#undef FF_CONV
    if (taps > 1) {
        const int cy = min(64, (C + 255) / 256);
        FF_LAUNCH((conv_state_update_kernel<T>), dim3(n_seqs, cy), 256, 0, stream, (const T*)in, in_stride, in_off, state,
                  (size_t)state_stride, conv_off, cu_q, state_slots, seq_fresh, C, taps);
    }
    FF_LAUNCH_CHECK();
    return 0;
}

// `out_dtype`: the type of `out` (the input's, or the engine's type for 32-bit input rows).
FF_EXPORT int ff_causal_conv(const void* in, int dtype, int in_stride, int in_off, const float* w, const float* bias,
                             float* state, long long state_stride, int conv_off, const int* token_seq,
                             const int* cu_q, const int* state_slots, const int* seq_fresh, void* out, int out_dtype,
                             int T, int n_seqs, int C, int taps, int flags, cudaStream_t stream) {
    if (T <= 0 || C <= 0) return 0;
    if (taps < 1 || taps > CONV_MAX_TAPS) return FF_ERR_UNSUPPORTED;
#define FF_CONV_TYPES(TI, TOUT)                                                                                          \
    return conv_launch<TI, TOUT>(in, in_stride, in_off, w, bias, state, state_stride, conv_off, token_seq, cu_q, state_slots, \
                                 seq_fresh, out, T, n_seqs, C, taps, flags, stream)
    if (dtype == 0 && out_dtype == 0) FF_CONV_TYPES(float, float);
    if (dtype == 1 && out_dtype == 1) FF_CONV_TYPES(bf16, bf16);
    if (dtype == 0 && out_dtype == 1) FF_CONV_TYPES(float, bf16);
#undef FF_CONV_TYPES
    return FF_ERR_BAD_ARG;
}

FF_EXPORT int ff_causal_conv_silu(const void* in, int dtype, int in_stride, int in_off, const float* w, const float* bias,
                                  float* state, long long state_stride, int conv_off, const int* token_seq,
                                  const int* cu_q, const int* state_slots, const int* seq_fresh, void* out, int T,
                                  int n_seqs, int C, int taps, cudaStream_t stream) {
    return ff_causal_conv(in, dtype, in_stride, in_off, w, bias, state, state_stride, conv_off, token_seq, cu_q, state_slots,
                          seq_fresh, out, dtype, T, n_seqs, C, taps, CONV_SILU, stream);
}

// Only the second half of the convolution: the last taps-1 rows of `in` of every sequence go into its state
// slot, for a part that convolves inside a kernel of its own.
FF_EXPORT int ff_conv_state_update(const void* in, int dtype, int in_stride, int in_off, float* state, long long state_stride,
                                   int conv_off, const int* cu_q, const int* state_slots, const int* seq_fresh, int n_seqs,
                                   int C, int taps, cudaStream_t stream) {
    if (n_seqs <= 0 || C <= 0 || taps <= 1) return 0;
    if (taps > CONV_MAX_TAPS) return FF_ERR_UNSUPPORTED;
    const int cy = min(64, (C + 255) / 256);
    if (dtype == 0)
        FF_LAUNCH((conv_state_update_kernel<float>), dim3(n_seqs, cy), 256, 0, stream, (const float*)in, in_stride, in_off, state,
                  (size_t)state_stride, conv_off, cu_q, state_slots, seq_fresh, C, taps);
    else if (dtype == 1)
        FF_LAUNCH((conv_state_update_kernel<bf16>), dim3(n_seqs, cy), 256, 0, stream, (const bf16*)in, in_stride, in_off, state,
                  (size_t)state_stride, conv_off, cu_q, state_slots, seq_fresh, C, taps);
    else return FF_ERR_BAD_ARG;
    FF_LAUNCH_CHECK();
    return 0;
}

// floats of a request's state for `heads` heads of key size N and value size V (-1: sizes not supported)
FF_EXPORT long long ff_scan_state_floats(int heads, int N, int V) {
    const int NP = ws_key_size(N);
    if (!NP || V <= 0 || V > 256) return -1;
    return (long long)heads * V * NP;
}

// Whether a step's prompts can go a chunk at a time: bfloat16, sizes that the tiles take and layouts that 16-byte copies take.  One decay
// per head and token (its inputs read as they are), or one per key channel.
static bool scalar_chunk_sizes(int mode, int act, int T, int N, int V) {
    return mode == 1 && !act && T >= SCAN_CHUNK_MIN && (N == 64 || N == 128) && V % 8 == 0;
}
static bool channel_chunk_sizes(int mode, int act, int T, int N, int V) {
    return mode == 2 && !act && T >= CHANNEL_CHUNK_MIN && (N == 64 || N == 128) && V % 8 == 0;
}
FF_EXPORT int ff_scan_chunk_min(int mode) { return mode == 2 ? CHANNEL_CHUNK_MIN : SCAN_CHUNK_MIN; }
static unsigned scan_bits(const ScanArgs& A) {
    return row_bits(A.q, A.q_stride, A.q_off, 2) | row_bits(A.k, A.k_stride, A.k_off, 2) | row_bits(A.v, A.v_stride, A.v_off, 2) |
           (A.mode == 2 ? row_bits(A.channel_decay, A.cd_stride, A.cd_off, 4) : 0u);
}

// Bytes of scratch memory that a step of T tokens can use (0: none; without it the token-by-token kernel runs).  `bits`: the matrices'
// addresses, row strides and first columns in bytes, or'ed (row_bits).
FF_EXPORT long long ff_scan_scratch_bytes(int dtype, int mode, int act, int T, int n_seqs, int heads, int heads_per_group, int N, int V, int bits) {
    if (dtype != 1 || T <= 0 || n_seqs <= 0 || heads <= 0 || heads_per_group <= 0 || heads % heads_per_group || V <= 0 || V > 256 || (bits & 15)) return 0;
    if (scalar_chunk_sizes(mode, act, T, N, V)) return chunk_records<SC_C>(T, n_seqs) * heads * (long long)sizeof(ScanRecord);
    if (!channel_chunk_sizes(mode, act, T, N, V)) return 0;
    return chunk_records(T, n_seqs) * heads * (long long)(N == 64 ? sizeof(ChunkRecord<64, false>) : sizeof(ChunkRecord<128, false>));
}

template <int NK>
static int scan_chunk_launch(const ScanArgs& A, float* state, long long state_stride, int state_off, const int* cu_q, const int* state_slots,
                             const int* seq_fresh, float* o, int T, int n_seqs, int live, int heads, int V, void* scratch, cudaStream_t stream) {
    ScanRecord* recs = (ScanRecord*)scratch;
    const long long records = chunk_records<SC_C>(T, n_seqs), groups = heads / A.heads_per_group, quads = (A.heads_per_group + 3) / 4;
    const long long quads_a_block = std::max(1ll, std::min(quads, (records * groups * quads + SCAN_PREPARE_BLOCKS - 1) / SCAN_PREPARE_BLOCKS));
    FF_LAUNCH(scalar_decay_prepare_kernel<NK>, dim3((unsigned)records, (unsigned)groups, (unsigned)((quads + quads_a_block - 1) / quads_a_block)), 128, 0,
              stream, A, recs, cu_q, n_seqs, SCAN_CHUNK_MIN, heads, (int)quads_a_block * 4);
#define FF_SCAN_CHUNK(W)                                                                                                \
    do {                                                                                                                \
        const dim3 grid(n_seqs, heads, (V + 16 * W - 1) / (16 * W));                                                    \
        const size_t smem = chunk_even_smem(sizeof(ScanChunkSmem<NK, W>), (long long)live * grid.y * grid.z);           \
        FF_SMEM_LIMIT((scalar_decay_chunk_kernel<NK, W>), 227 * 1024);                                                  \
        FF_LAUNCH((scalar_decay_chunk_kernel<NK, W>), grid, 64 * W + CS_LOADERS, smem, stream,                          \
                  A, recs, state, (size_t)state_stride, state_off, cu_q, state_slots, seq_fresh, o, heads, V, SCAN_CHUNK_MIN); \
    } while (0)
    // 64 value columns a block if that gives most SMs a block, else 32
    if ((long long)live * heads * ((V + 63) / 64) >= 100) FF_SCAN_CHUNK(4);
    else FF_SCAN_CHUNK(2);
#undef FF_SCAN_CHUNK
    FF_LAUNCH_CHECK();
    return 0;
}

template <int NK>
static int channel_chunk_launch(const ScanArgs& A, const ChunkScanArgs& B, int T, int n_seqs, int live, void* scratch, cudaStream_t stream) {
    const int n_records = (int)chunk_records(T, n_seqs);
    FF_LAUNCH(channel_decay_prepare_kernel<NK>, cf_grid<NK>(n_records, B.heads), 32 * CF_WARPS, 0, stream, A, (ChunkRecord<NK, false>*)scratch, B.cu_q,
              n_seqs, n_records, B.min_len, B.heads);
    return chunk_scan_launch<NK, false>(B, n_seqs, live, stream);
}

template <typename T>
static int scan_launch(const ScanArgs& A, float* state, long long state_stride, int state_off, const int* cu_q,
                       const int* state_slots, const int* seq_fresh, float* o, int T_tot, int n_seqs, int heads, int N, int V,
                       int n_long, void* scratch, long long scratch_bytes, int* launched, cudaStream_t stream) {
    if (!ws_key_size(N) || V <= 0 || V > 256) return FF_ERR_UNSUPPORTED;
    const long long need = sizeof(T) == 2 ? ff_scan_scratch_bytes(1, A.mode, A.act, T_tot, n_seqs, heads, A.heads_per_group, N, V, (int)scan_bits(A)) : 0;
    const ChunkRoute R = chunk_route(need > 0 && scratch && scratch_bytes >= need, n_long, n_seqs, ff_scan_chunk_min(A.mode));
    *launched = R.kernels();
#define FF_SCAN_ONE(NP, CD, SOME)                                                                                       \
    FF_LAUNCH((scalar_decay_scan_kernel<T, NP, CD, SOME>), dim3(n_seqs, heads, (V + WideState<NP>::VB - 1) / WideState<NP>::VB), \
              WS_THREADS, 0, stream, A, state, (size_t)state_stride, state_off, cu_q, state_slots, seq_fresh, o, heads, N, V, R.max_walk)
#define FF_SCAN(NP)                                                                                                     \
    do {                                                                                                                \
        if (sizeof(T) == 2 && (NP == 64 || NP == 128) && R.chunks) {                                                    \
            constexpr bool SOME = sizeof(T) == 2 && (NP == 64 || NP == 128);    /* no other size goes by chunks */       \
            if (A.mode == 2) FF_SCAN_ONE(NP, true, SOME);                                                               \
            else FF_SCAN_ONE(NP, false, SOME);                                                                          \
        } else if (A.mode == 2) FF_SCAN_ONE(NP, true, false);                                                           \
        else FF_SCAN_ONE(NP, false, false);                                                                             \
    } while (0)
    if (R.walk) {
        switch (ws_key_size(N)) {
            case 16: FF_SCAN(16); break;
            case 32: FF_SCAN(32); break;
            case 64: FF_SCAN(64); break;
            case 128: FF_SCAN(128); break;
            default: FF_SCAN(256); break;
        }
        FF_LAUNCH_CHECK();
    }
#undef FF_SCAN
#undef FF_SCAN_ONE
    if (!R.chunks) return 0;
    if (A.mode == 1) {
        if (N == 64) return scan_chunk_launch<64>(A, state, state_stride, state_off, cu_q, state_slots, seq_fresh, o, T_tot, n_seqs, R.live, heads, V, scratch, stream);
        return scan_chunk_launch<128>(A, state, state_stride, state_off, cu_q, state_slots, seq_fresh, o, T_tot, n_seqs, R.live, heads, V, scratch, stream);
    }
    const ChunkScanArgs B{scratch, (const bf16*)A.v, A.v_stride, A.v_off, state, state_stride, state_off, V * N, cu_q, state_slots, seq_fresh, o, heads, V, CHANNEL_CHUNK_MIN};
    return N == 64 ? channel_chunk_launch<64>(A, B, T_tot, n_seqs, R.live, scratch, stream) : channel_chunk_launch<128>(A, B, T_tot, n_seqs, R.live, scratch, stream);
}

// `n_long`: how many of the sequences have ff_scan_chunk_min tokens or more (-1: not known).  `launched`: how many kernels the call put
// on the stream (1: token by token, 2: by chunks, 3: some sequences so and some so).
FF_EXPORT int ff_scalar_decay_scan(const void* q, int q_stride, int q_off, const void* k, int k_stride, int k_off,
                                   const void* v, int v_stride, int v_off, int dtype, int heads_per_group, int act,
                                   int mode, const float* decay, const void* step, int step_stride, int step_off,
                                   const float* step_bias, const float* a_log, const float* skip,
                                   const float* channel_decay, int cd_stride, int cd_off, float q_scale, float* state,
                                   long long state_stride, int state_off, const int* cu_q, const int* state_slots,
                                   const int* seq_fresh, float* o, int T, int n_seqs, int heads, int N, int V,
                                   int n_long, void* scratch, long long scratch_bytes, int* launched, cudaStream_t stream) {
    *launched = 0;
    if (T <= 0 || n_seqs <= 0) return 0;
    if (heads_per_group <= 0 || mode < 0 || mode > 2 || (mode == 2 && !channel_decay)) return FF_ERR_BAD_ARG;
    ScanArgs A{q, q_stride, q_off, k, k_stride, k_off, v, v_stride, v_off, heads_per_group, act, decay,
               step, step_stride, step_off, step_bias, a_log, skip, mode, channel_decay, cd_stride, cd_off, q_scale};
    if (dtype == 0)
        return scan_launch<float>(A, state, state_stride, state_off, cu_q, state_slots, seq_fresh, o, T, n_seqs, heads, N, V, n_long, scratch, scratch_bytes, launched, stream);
    if (dtype == 1)
        return scan_launch<bf16>(A, state, state_stride, state_off, cu_q, state_slots, seq_fresh, o, T, n_seqs, heads, N, V, n_long, scratch, scratch_bytes, launched, stream);
    return FF_ERR_BAD_ARG;
}

FF_EXPORT int ff_low_rank_decay(const void* low, int dtype, int low_stride, int low_off, const void* w, const float* bias,
                                float tau, float* alpha, int T, int C, int R, cudaStream_t stream) {
    if (T <= 0 || C <= 0) return 0;
    if (R <= 0 || !(tau > 0.f)) return FF_ERR_BAD_ARG;
    const int Rp = (R + LRD_R - 1) / LRD_R * LRD_R;
    const int cols = (C + LRD_THREADS - 1) / LRD_THREADS;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return (int)e;
    // as many tokens a block (up to LRD_TOK) as leave every SM eight blocks: a block's weights cost as much as four tokens
    const int tiles = max(1, sms * 8 / cols);
    int tile = min(LRD_TOK, ((T + tiles - 1) / tiles + LRD_U - 1) / LRD_U * LRD_U);
    while (tile > LRD_U && (size_t)Rp * tile * sizeof(float) > 48 * 1024) tile = max(LRD_U, tile / 2 / LRD_U * LRD_U);
    const size_t smem = (size_t)Rp * tile * sizeof(float);
    if (smem > 48 * 1024) return FF_ERR_UNSUPPORTED;
    dim3 grid((T + tile - 1) / tile, cols);
    auto w_pieces = [&](int n) { return ((uintptr_t)w & 15) == 0 && R % n == 0 ? 1 : 0; };
    if (dtype == 0)
        FF_LAUNCH((low_rank_decay_kernel<float>), grid, LRD_THREADS, smem, stream, (const float*)low, low_stride, low_off,
                  (const float*)w, bias, 1.0f / tau, alpha, T, C, R, tile, w_pieces(4));
    else if (dtype == 1)
        FF_LAUNCH((low_rank_decay_kernel<bf16>), grid, LRD_THREADS, smem, stream, (const bf16*)low, low_stride, low_off,
                  (const bf16*)w, bias, 1.0f / tau, alpha, T, C, R, tile, w_pieces(8));
    else return FF_ERR_BAD_ARG;
    FF_LAUNCH_CHECK();
    return 0;
}

FF_EXPORT int ff_gated_rms_norm(const float* o, const void* z, int dtype, int z_stride, int z_off, const float* w,
                                float eps, void* y, int T, int width, int parts, int order, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (parts <= 0 || width % parts || (order != 0 && order != 1)) return FF_ERR_BAD_ARG;
    const int per = width / parts;
    const int threads = per >= 1024 ? 256 : (per >= 256 ? 128 : 64);
    const int es = dtype == 0 ? 4 : 2;
    if (per % 128 == 0 && per <= 4096 && (((uintptr_t)o | (uintptr_t)w) & 15) == 0 && (((uintptr_t)z | (uintptr_t)y) & (4 * es - 1)) == 0 &&
        z_stride % 4 == 0 && z_off % 4 == 0) {
        const bool one_warp = per <= 1024;
        const long long items = (long long)T * parts;
        const unsigned blocks = (unsigned)(one_warp ? (items + 7) / 8 : items);
#define FF_GATED_NORM(TT, TP, MV) \
        FF_LAUNCH((gated_rms_norm_vec_kernel<TT, TP, MV>), blocks, 256, 0, stream, o, (const TT*)z, z_stride, z_off, w, eps, (TT*)y, T, width, parts, order)
#define FF_GATED_NORM_SIZE(TT)                                  \
        do {                                                    \
            if (!one_warp) FF_GATED_NORM(TT, 256, 4);           \
            else if (per <= 256) FF_GATED_NORM(TT, 32, 2);      \
            else if (per <= 512) FF_GATED_NORM(TT, 32, 4);      \
            else FF_GATED_NORM(TT, 32, 8);                      \
        } while (0)
        if (dtype == 0) FF_GATED_NORM_SIZE(float);
        else if (dtype == 1) FF_GATED_NORM_SIZE(bf16);
        else return FF_ERR_BAD_ARG;
#undef FF_GATED_NORM_SIZE
#undef FF_GATED_NORM
        FF_LAUNCH_CHECK();
        return 0;
    }
    if (dtype == 0)
        FF_LAUNCH((gated_rms_norm_kernel<float>), dim3(T, parts), threads, 0, stream, o, (const float*)z, z_stride, z_off, w, eps,
                  (float*)y, width, parts, order);
    else if (dtype == 1)
        FF_LAUNCH((gated_rms_norm_kernel<bf16>), dim3(T, parts), threads, 0, stream, o, (const bf16*)z, z_stride, z_off, w, eps,
                  (bf16*)y, width, parts, order);
    else return FF_ERR_BAD_ARG;
    FF_LAUNCH_CHECK();
    return 0;
}
