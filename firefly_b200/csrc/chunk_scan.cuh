// Recurrences with a decay per key channel, and the delta rule, sixteen tokens at a time (bfloat16 prompts).
//
// With E_t the product of a channel's decays up to token t of a chunk, F_s that of the ones behind s, G that of all
// sixteen, and S the state in front of the chunk:
//
//   o_t = sum_n (q E)_t S + sum_(s <= t) P_ts v_s,    P_ts = sum_n q_t k_s prod(decays of s+1 .. t)
//   S  <- G S + sum_s (k F)_s v_s^T
//
// and for the delta rule, whose writes are u instead of v,  U = T diag(beta) (V - (k E) S),  T the inverse of the unit lower
// triangle 1 + beta_t sum_n k_t k_s prod(...).  None of q E, k E, k F, P, T, G holds the state, so a first kernel forms them for
// all chunks of the step at once (every factor a product of decays, never one divided by another, so no decay is too strong
// for it) and leaves them as records in scratch memory, split in bfloat16 parts (chunk_mma.cuh).  The second kernel walks a
// sequence's records: what is left to do one chunk after the other is a few dozen tensor-core products.
#pragma once

#include "chunk_mma.cuh"

namespace ff {

constexpr int CS_C = 16;                                    // tokens a chunk
// Records a block of the first kernel forms, one behind the other (the next one's inputs are on their way while it forms one): up
// to four while that leaves every SM eight blocks, else one, so that short steps do not leave SMs idle.
static inline int chunk_records_a_block(long long records_and_heads) { return records_and_heads >= 4 * 8 * 148 ? 4 : 1; }

template <int NK, bool DELTA>
struct ChunkRecord {
    static constexpr int QP = NK + 8, PP = CS_C + 8;        // row pitches: 16-byte pieces of eight rows lie in different banks
    bf16 qe[3][CS_C * QP];                                  // q E (the decays in front of the token for a read-out in front of the write)
    bf16 kf[3][CS_C * QP];                                  // k F
    bf16 P[3][CS_C * PP];
    float G[NK];
    bf16 ke[DELTA ? 3 : 1][DELTA ? CS_C * QP : 8];          // k E
    bf16 TB[DELTA ? 3 : 1][DELTA ? CS_C * PP : 8];          // T diag(beta)
};

// With chunks of C tokens, a sequence that starts at token t0 of the step and is number s has its records from here on; at
// most T / C + n in all.
template <int C = CS_C> __host__ __device__ __forceinline__ int chunk_first_record(int t0, int s) { return t0 / C + s; }
template <int C = CS_C> static inline long long chunk_records(int T, int n_seqs) { return T / C + n_seqs; }

// What 16-byte copies of rows ask for: the low four bits of this, or'ed over the matrices, are zero.
static inline unsigned row_bits(const void* p, long long stride, long long off, int element) {
    return (unsigned)((uintptr_t)p | (unsigned long long)(stride * element) | (unsigned long long)(off * element));
}

// Which sequences of a step go by chunks: those of at least `chunk_min` tokens, whoever else is in the step, so that a request's numbers
// do not depend on its company.  `n_long`: how many they are (-1: not known); the other sequences go token by token.
struct ChunkRoute {
    bool chunks, walk;                                      // which kernels have anything to do
    int live;                                               // sequences that go by chunks, for the size of blocks
    int max_walk;                                           // the token-by-token kernel leaves sequences of this length and longer alone
    int kernels() const { return 2 * chunks + walk; }
};
static inline ChunkRoute chunk_route(bool possible, int n_long, int n_seqs, int chunk_min) {
    const bool chunks = possible && n_long != 0;
    return {chunks, !chunks || n_long != n_seqs, n_long > 0 ? n_long : n_seqs, chunks ? chunk_min : 0x7fffffff};
}

// The sequence and chunk of record r (chunk -1: none); all lanes of a warp ask together.
template <int C = CS_C>
__device__ __forceinline__ void chunk_of_record(const int* cu_q, int n_seqs, int r, int min_len, int& s, int& chunk) {
    const int lane = threadIdx.x & 31;
    s = -1;
    for (int s0 = 0; s0 < n_seqs; s0 += 32) {
        const bool mine = s0 + lane < n_seqs && chunk_first_record<C>(cu_q[s0 + lane], s0 + lane) <= r;
        const unsigned m = __ballot_sync(0xffffffffu, mine);
        if (m) s = s0 + 31 - __clz(m);
        if (m != 0xffffffffu) break;
    }
    chunk = -1;
    if (s >= 0) {
        const int i = r - chunk_first_record<C>(cu_q[s], s);
        const int len = cu_q[s + 1] - cu_q[s];
        if (len >= min_len && i * C < len) chunk = i;
    }
}

// ---------------------------------------------------------------------------------- the first kernel's parts --
// sq, sk, sa: the chunk's q, k and decays in shared memory, [16][NK] 32-bit; rows behind the sequence's end have q = k = 0 and
// decay 1.  2 NK threads.

// A thread's eight neighbouring elements of a chunk: row tid / (NK / 8), columns 8 (tid % (NK / 8)) ..
__device__ __forceinline__ void chunk_unpack(const uint4& v, float x[8]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { x[2 * i] = cm_lo(w[i]); x[2 * i + 1] = cm_hi(w[i]); }
}
__device__ __forceinline__ void chunk_stage8(float* to, const float x[8]) {
    *reinterpret_cast<float4*>(to) = make_float4(x[0], x[1], x[2], x[3]);
    *reinterpret_cast<float4*>(to + 4) = make_float4(x[4], x[5], x[6], x[7]);
}

// The chunk's two halves of eight tokens, each row scaled to the border between them: a pair of tokens on either side of it
// needs no more than the product of these rows.
template <int NK, bool DELTA>
struct ChunkHalves {
    static constexpr int HP = NK + 4;                       // row pitch: 16-byte pieces of eight rows lie in different banks
    float q[CS_C / 2][HP], k[CS_C / 2][HP];                 // tokens 8..: q times the decays of 8 ..; tokens ..7: k times the ones behind it up to 7
    float k_late[DELTA ? CS_C / 2 : 1][DELTA ? HP : 4];     // tokens 8..: k as q
};

// q E, k F, k E and G, and the halves.  Thread (pair of channels, side, half of the tokens).  BEFORE: E without the token's own decay.
template <int NK, bool DELTA, bool BEFORE>
__device__ __forceinline__ void chunk_scaled_rows(ChunkRecord<NK, DELTA>* rec, ChunkHalves<NK, DELTA>& hs, const float* sq, const float* sk, const float* sa) {
    using R = ChunkRecord<NK, DELTA>;
    constexpr int H = CS_C / 2, PW = R::QP / 2, PART = CS_C * PW;
    const int n = 2 * (threadIdx.x % (NK / 2)), side = threadIdx.x / (NK / 2) & 1, half = threadIdx.x / NK;
    auto decay = [&](int t) { return *reinterpret_cast<const float2*>(sa + t * NK + n); };
    auto put = [&](bf16* to, int t, float x, float y) {
        uint32_t* dst = reinterpret_cast<uint32_t*>(to) + t * PW + n / 2;
        cm_split3(x, y, dst[0], dst[PART], dst[2 * PART]);
    };
    float2 base = make_float2(1.f, 1.f), e = base;          // the decays of the half that lies between, and those within the own half
    if (side == 0) {                                        // products from the chunk's start
        if (half) {
#pragma unroll
            for (int t = 0; t < H; ++t) { const float2 a = decay(t); base.x *= a.x; base.y *= a.y; }
        }
#pragma unroll
        for (int i = 0; i < H; ++i) {
            const int t = half * H + i;
            const float2 a = decay(t), q = *reinterpret_cast<const float2*>(sq + t * NK + n);
            const float2 out = e;
            e.x *= a.x;
            e.y *= a.y;
            const float2 r = BEFORE ? make_float2(q.x * out.x, q.y * out.y) : make_float2(q.x * e.x, q.y * e.y);
            put(rec->qe[0], t, r.x * base.x, r.y * base.y);
            if (half) *reinterpret_cast<float2*>(&hs.q[i][n]) = r;
            if constexpr (DELTA) {
                const float2 k = *reinterpret_cast<const float2*>(sk + t * NK + n);
                put(rec->ke[0], t, k.x * e.x * base.x, k.y * e.y * base.y);
                if (half) *reinterpret_cast<float2*>(&hs.k_late[i][n]) = make_float2(k.x * e.x, k.y * e.y);
            }
        }
        if (half) *reinterpret_cast<float2*>(&rec->G[n]) = make_float2(e.x * base.x, e.y * base.y);
    } else {                                                // products to the chunk's end
        if (!half) {
#pragma unroll
            for (int t = CS_C - 1; t >= H; --t) { const float2 a = decay(t); base.x *= a.x; base.y *= a.y; }
        }
#pragma unroll
        for (int i = H - 1; i >= 0; --i) {
            const int t = half * H + i;
            const float2 a = decay(t), k = *reinterpret_cast<const float2*>(sk + t * NK + n);
            const float2 r = make_float2(k.x * e.x, k.y * e.y);
            put(rec->kf[0], t, r.x * base.x, r.y * base.y);
            if (!half) *reinterpret_cast<float2*>(&hs.k[i][n]) = r;
            e.x *= a.x;
            e.y *= a.y;
        }
    }
}

// Pairs of tokens of one half: sum_n q_t[n] k_s[n] prod(decays of s+1 .. t) for s <= t (BEFORE: .. t-1, and sum_n q_t[n] k_s[n] u[n]
// for s = t), zero else; with DELTA also the same of k_t.  Thread (s, eight channels) walks the half's tokens; the channels'
// shares are joined over NK / 8 neighbouring threads, which ends with one token each: put(t, s, of q, of k).
template <int NK, bool DELTA, bool BEFORE, typename Put>
__device__ __forceinline__ void chunk_near_pairs(const float* sq, const float* sk, const float* sa, const float* u, Put put) {
    constexpr int L = NK / 8, H = CS_C / 2;
    const int part = threadIdx.x % L, s = threadIdx.x / L, t0 = s & H, ls = s & (H - 1), n = part * 8;
    float d[8], x[H], y[DELTA ? H : 1] = {};
    auto row8 = [&](const float* m, int t, float v[8]) {
        *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(m + t * NK + n);
        *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(m + t * NK + n + 4);
    };
    row8(sk, s, d);
#pragma unroll
    for (int i = 0; i < H; ++i) {
        float q[8], a[8], k[8], p0 = 0.f, p1 = 0.f, r0 = 0.f, r1 = 0.f;
        row8(sq, t0 + i, q);
        row8(sa, t0 + i, a);
        if constexpr (DELTA) row8(sk, t0 + i, k);
#pragma unroll
        for (int c = 0; c < 8; c += 2) {
            if (!BEFORE) { d[c] *= i > ls ? a[c] : 1.f; d[c + 1] *= i > ls ? a[c + 1] : 1.f; }
            if constexpr (BEFORE) {
                p0 += q[c] * (i == ls ? d[c] * u[n + c] : d[c]);
                p1 += q[c + 1] * (i == ls ? d[c + 1] * u[n + c + 1] : d[c + 1]);
            } else {
                p0 += q[c] * d[c];
                p1 += q[c + 1] * d[c + 1];
            }
            if constexpr (DELTA) { r0 += k[c] * d[c]; r1 += k[c + 1] * d[c + 1]; }
            if (BEFORE) { d[c] *= i > ls ? a[c] : 1.f; d[c + 1] *= i > ls ? a[c + 1] : 1.f; }
        }
        x[i] = i >= ls ? p0 + p1 : 0.f;
        if constexpr (DELTA) y[i] = r0 + r1;
    }
    int t = t0, off = 1;
#pragma unroll
    for (int m = H / 2; m >= 1; m >>= 1) {                  // every step halves the tokens a thread still adds up
        const bool up = part & off;
#pragma unroll
        for (int i = 0; i < m; ++i) {
            const float away = up ? x[i] : x[i + m];
            x[i] = (up ? x[i + m] : x[i]) + __shfl_xor_sync(0xffffffffu, away, off);
            if constexpr (DELTA) {
                const float away_y = up ? y[i] : y[i + m];
                y[i] = (up ? y[i + m] : y[i]) + __shfl_xor_sync(0xffffffffu, away_y, off);
            }
        }
        if (up) t += m;
        off <<= 1;
    }
#pragma unroll
    for (; off < L; off <<= 1) {
        x[0] += __shfl_xor_sync(0xffffffffu, x[0], off);
        if constexpr (DELTA) y[0] += __shfl_xor_sync(0xffffffffu, y[0], off);
    }
    if (part < H) put(t, s, x[0], DELTA ? y[0] : 0.f);
}

// Pairs across the border: token 8 + i and token s, a thread 32 channels of one pair.
template <int NK, bool DELTA, typename Put>
__device__ __forceinline__ void chunk_far_pairs(const ChunkHalves<NK, DELTA>& hs, Put put) {
    constexpr int L = NK / 32, H = CS_C / 2;
    const int part = threadIdx.x % L, s = threadIdx.x / L % H, i = threadIdx.x / (L * H);
    float p0 = 0.f, p1 = 0.f, r0 = 0.f, r1 = 0.f;
#pragma unroll
    for (int c = 0; c < 32; c += 4) {
        const int n = c * L + part * 4;                     // neighbouring threads read neighbouring pieces
        const float4 k = *reinterpret_cast<const float4*>(&hs.k[s][n]), q = *reinterpret_cast<const float4*>(&hs.q[i][n]);
        p0 += q.x * k.x + q.y * k.y;
        p1 += q.z * k.z + q.w * k.w;
        if constexpr (DELTA) {
            const float4 kl = *reinterpret_cast<const float4*>(&hs.k_late[i][n]);
            r0 += kl.x * k.x + kl.y * k.y;
            r1 += kl.z * k.z + kl.w * k.w;
        }
    }
    float x = p0 + p1, y = r0 + r1;
#pragma unroll
    for (int off = 1; off < L; off <<= 1) {
        x += __shfl_xor_sync(0xffffffffu, x, off);
        if constexpr (DELTA) y += __shfl_xor_sync(0xffffffffu, y, off);
    }
    if (part == 0) put(H + i, s, x, y);
}

// one number of a [16][16] matrix of a record, split
__device__ __forceinline__ void chunk_put(bf16* to, int t, int s, float x) {
    uint32_t p0, p1, p2;
    cm_split3(x, 0.f, p0, p1, p2);
    constexpr int pitch = CS_C + 8, part = CS_C * pitch;
    const int at = t * pitch + s;
    reinterpret_cast<uint16_t*>(to)[at] = (uint16_t)p0;
    reinterpret_cast<uint16_t*>(to)[at + part] = (uint16_t)p1;
    reinterpret_cast<uint16_t*>(to)[at + 2 * part] = (uint16_t)p2;
}
// the same of a pair across the border, with the zero on the other side of the diagonal
__device__ __forceinline__ void chunk_put_far(bf16* to, int t, int s, float x) {
    chunk_put(to, t, s, x);
    chunk_put(to, t - CS_C / 2, s + CS_C / 2, 0.f);
}

// ---------------------------------------------------------------------------------- the second kernel --
struct ChunkScanArgs {
    const void* records;                                    // [chunk_records][heads] ChunkRecord
    const bf16* v; long long v_stride; int v_off;           // value rows per head: v_off + h * V + j
    float* state; long long state_stride; int state_off, head_floats;      // a head's state: [V][NK] floats
    const int* cu_q; const int* state_slots; const int* seq_fresh;
    float* o; int heads, V;                                 // [T, heads * V]
    int min_len;                                            // shorter sequences are not this kernel's
};

constexpr int CS_STAGES = 3;
constexpr int CS_LOADERS = 64;                              // threads that bring in records and values

// acc^T += x^T M^T for a lower triangle M (three bfloat16 parts) without the entries above the diagonal, a warp's 16 columns
// x 16 tokens at a time; x and acc as accumulators of mma.sync lie.  The slow way, for numbers that are not finite.
__device__ __forceinline__ void chunk_lower(float (*tmp)[CS_C + 1], const float x[2][4], const bf16* M, float acc[2][4], int lane) {
    const int g = lane >> 2, c2 = (lane & 3) * 2;
    __syncwarp();
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) tmp[g + (e >> 1) * 8][nt * 8 + c2 + (e & 1)] = x[nt][e];
    __syncwarp();
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int t = nt * 8 + c2 + (e & 1), j = g + (e >> 1) * 8, part = CS_C * (CS_C + 8);
            float r = 0.f;
            for (int s = 0; s <= t; ++s) {
                const bf16* m = M + t * (CS_C + 8) + s;
                r += (to_float(m[0]) + to_float(m[part]) + to_float(m[2 * part])) * tmp[j][s];
            }
            acc[nt][e] += r;
        }
    __syncwarp();
}

template <int NK, int W, bool DELTA>
struct ChunkScanSmem {
    struct Stage { ChunkRecord<NK, DELTA> rec; bf16 v[CS_C * (16 * W + 8)]; };
    Stage stage[CS_STAGES];
    float xch[2][2 * W][DELTA ? 12 : 4][32];
    float slow[2 * W][16][CS_C + 1];
};

// One block per (sequence, head, 16 W value columns).  Two warps hold S^T of 16 value columns, half of the keys each, as the
// accumulators of mma.sync; the same registers are, split, the left operand of S^T (q E), so the state goes nowhere between the
// products.  The two exchange their shares of S^T (q E) and S^T (k E); what follows of the read-out each does for eight of the
// tokens.  Two more warps bring in records and values by 16-byte copies, two chunks ahead; one barrier a chunk.
// (With all keys in one warp, which also did its own loads, a chunk took half as long again: 135 against 90 us for three
// sequences of 1501, 1000 and 700 tokens with 16 heads of 64 x 128, 384 against 232 us for the delta rule on 4 x 2048 tokens.)
template <int NK, int W, bool DELTA>
__global__ void __launch_bounds__(64 * W + CS_LOADERS) chunk_scan_kernel(ChunkScanArgs A) {
    pdl_prologue();
    using R = ChunkRecord<NK, DELTA>;
    using SM = ChunkScanSmem<NK, W, DELTA>;
    constexpr int QP = R::QP, PP = R::PP, VB = 16 * W, VP = VB + 8, NT = NK / 16;
    static_assert(sizeof(R) % 16 == 0, "a record is copied in 16-byte pieces");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SM& sm = *reinterpret_cast<SM*>(smem_raw);
    const int s = blockIdx.x, h = blockIdx.y, j0 = blockIdx.z * VB, V = A.V;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t0 = A.cu_q[s], len = A.cu_q[s + 1] - t0, chunks = (len + CS_C - 1) / CS_C;
    if (len < A.min_len) return;
    if (warp >= 2 * W) {
        // ---- the warps that load
        const int pt = threadIdx.x - 64 * W;
        const unsigned char* src = reinterpret_cast<const unsigned char*>(pdl_fresh((const R*)A.records) + (size_t)chunk_first_record(t0, s) * A.heads + h);
        const bf16* vp = pdl_fresh(A.v) + A.v_off + (size_t)h * V + j0;
        auto load = [&](int i) {
            if (i < chunks) {
                typename SM::Stage& st = sm.stage[i % CS_STAGES];
                unsigned char* dst = reinterpret_cast<unsigned char*>(&st.rec);
                const unsigned char* from = src + (size_t)i * A.heads * sizeof(R);
#pragma unroll 8
                for (int p = pt; p < (int)(sizeof(R) / 16); p += CS_LOADERS) cm_copy16(dst + p * 16, from + p * 16, true);
                for (int p = pt; p < CS_C * (VB / 8); p += CS_LOADERS) {
                    const int r = p / (VB / 8), c = p % (VB / 8) * 8;
                    const bool in = i * CS_C + r < len && j0 + c < V;
                    cm_copy16(st.v + r * VP + c, vp + (in ? (t0 + i * CS_C + r) * A.v_stride + c : 0), in);
                }
            }
            cm_copy_commit();
        };
        load(0);
        load(1);
        for (int i = 0; i < chunks; ++i) {
            cm_copy_wait<1>();
            __syncthreads();                                // chunk i is there, and everybody is done with chunk i - 1
            load(i + 2);
        }
        cm_copy_wait<0>();
        return;
    }
    // ---- the warps that hold S^T
    const int tile = warp % W, half = warp / W, other = tile + (1 - half) * W, k0 = half * (NK / 2);
    const int g = lane >> 2, c2 = (lane & 3) * 2;
    // rows and columns of ldmatrix: the second 8 x 8 tile 8 rows down and the third 8 columns on (a), or the other way round (b)
    const int row_a = (lane & 7) + ((lane >> 3) & 1) * 8, col_a = (lane >> 4) * 8;
    const int row_b = (lane & 7) + (lane >> 4) * 8, col_b = ((lane >> 3) & 1) * 8;
    float* S_g = A.state + (size_t)A.state_slots[s] * A.state_stride + A.state_off + (size_t)h * A.head_floats + k0;
    const bool fresh = A.seq_fresh[s] != 0;
    const int jr[2] = {j0 + tile * 16 + g, j0 + tile * 16 + g + 8};
    float S[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
            S[nt][e] = (fresh || jr[e >> 1] >= V) ? 0.f : S_g[(size_t)jr[e >> 1] * NK + nt * 8 + c2 + (e & 1)];
    }
    const int ld = A.heads * V, t_own = half * 8 + c2;      // the first of the lane's two tokens of a chunk
    float* op = A.o + (size_t)(t0 + t_own) * ld + (size_t)h * V + jr[0];
    const bool all_cols = j0 + VB <= V;
    for (int i = 0; i < chunks; ++i) {
        __syncthreads();
        const typename SM::Stage& st = sm.stage[i % CS_STAGES];
        const R& rec = st.rec;
        float acc[2][4], low[2][4], pred[2][4], plow[2][4];        // o^T and the sum of its small terms; S^T (k E) and the same
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[nt][e] = low[nt][e] = pred[nt][e] = plow[nt][e] = 0.f;
        }
#pragma unroll
        for (int kk = 0; kk < NK / 32; ++kk) {
            uint32_t a[3][4], r[3][4];
            cm_split3(S[2 * kk][0], S[2 * kk][1], a[0][0], a[1][0], a[2][0]);
            cm_split3(S[2 * kk][2], S[2 * kk][3], a[0][1], a[1][1], a[2][1]);
            cm_split3(S[2 * kk + 1][0], S[2 * kk + 1][1], a[0][2], a[1][2], a[2][2]);
            cm_split3(S[2 * kk + 1][2], S[2 * kk + 1][3], a[0][3], a[1][3], a[2][3]);
#pragma unroll
            for (int p = 0; p < 3; ++p) cm_ldsm4(r[p], rec.qe[p] + row_b * QP + k0 + kk * 16 + col_b);
            cm_mma_rows(acc, low, a, r);
            if constexpr (DELTA) {
#pragma unroll
                for (int p = 0; p < 3; ++p) cm_ldsm4(r[p], rec.ke[p] + row_b * QP + k0 + kk * 16 + col_b);
                cm_mma_rows(pred, plow, a, r);
            }
        }
        // the two warps of these columns exchange their shares: of the other's tokens, and all of S^T (k E)
        float own[4], own_low[4];
        {
            float (*mine)[32] = sm.xch[i & 1][warp];
            const float (*theirs)[32] = sm.xch[i & 1][other];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                mine[e][lane] = half ? acc[0][e] + low[0][e] : acc[1][e] + low[1][e];
                if constexpr (DELTA) {
                    pred[0][e] += plow[0][e];
                    pred[1][e] += plow[1][e];
                    mine[4 + e][lane] = pred[0][e];
                    mine[8 + e][lane] = pred[1][e];
                }
            }
            cm_barrier(1 + tile, 64);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                own[e] = (half ? acc[1][e] + low[1][e] : acc[0][e] + low[0][e]) + theirs[e][lane];
                own_low[e] = 0.f;
                if constexpr (DELTA) {
                    pred[0][e] += theirs[4 + e][lane];
                    pred[1][e] += theirs[8 + e][lane];
                }
            }
        }
        // what is written: V^T, 16 value columns x 16 tokens, as a left operand; and the own tokens' rows of P as a right one
        uint32_t va[DELTA ? 3 : 1][4], pb[3][2];
        cm_ldsm4t(va[0], st.v + row_b * VP + tile * 16 + col_b);
        {
            uint32_t r[4];
            cm_ldsm4(r, rec.P[lane >> 4] + (half * 8 + (lane & 7)) * PP + col_b);
            pb[0][0] = r[0]; pb[0][1] = r[1]; pb[1][0] = r[2]; pb[1][1] = r[3];
            cm_ldsm4(r, rec.P[2] + (half * 8 + (lane & 7)) * PP + col_b);
            pb[2][0] = r[0]; pb[2][1] = r[1];
        }
        bool odd = false;
        float x[2][4];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const uint32_t pair = va[0][nt * 2 + (e >> 1)];
                x[nt][e] = (e & 1) ? cm_hi(pair) : cm_lo(pair);
                if constexpr (DELTA) x[nt][e] -= pred[nt][e];
                odd |= !(fabsf(x[nt][e]) <= 3.4028235e38f);
            }
        }
        odd = __any_sync(0xffffffffu, odd);
        if constexpr (DELTA) {
            float u[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}}, ul[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
            if (!odd) {
                uint32_t xa[3][4], r[3][4];
#pragma unroll
                for (int q = 0; q < 4; ++q) cm_split3(x[q >> 1][(q & 1) * 2], x[q >> 1][(q & 1) * 2 + 1], xa[0][q], xa[1][q], xa[2][q]);
#pragma unroll
                for (int p = 0; p < 3; ++p) cm_ldsm4(r[p], rec.TB[p] + row_b * PP + col_b);
                cm_mma_rows(u, ul, xa, r);
                cm_add(u[0], ul[0]);
                cm_add(u[1], ul[1]);
            } else {
                // a number that is not finite must not reach the tokens in front of it through a product with zero
                chunk_lower(sm.slow[warp], x, rec.TB[0], u, lane);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                x[q >> 1][(q & 1) * 2] = u[q >> 1][(q & 1) * 2];
                x[q >> 1][(q & 1) * 2 + 1] = u[q >> 1][(q & 1) * 2 + 1];
                cm_split3(x[q >> 1][(q & 1) * 2], x[q >> 1][(q & 1) * 2 + 1], va[0][q], va[1][q], va[2][q]);
            }
            // nor must a write that became one here (a beta that is none, an overflow)
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
                for (int e = 0; e < 4; ++e) odd |= !(fabsf(x[nt][e]) <= 3.4028235e38f);
            }
            odd = __any_sync(0xffffffffu, odd);
        }
        if (!odd) cm_mma_parts<DELTA ? 3 : 1, 3>(own, own_low, va, pb);
        else {
            float y[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
            chunk_lower(sm.slow[warp], x, rec.P[0], y, lane);
#pragma unroll
            for (int e = 0; e < 4; ++e) own[e] += half ? y[1][e] : y[0][e];
        }
        cm_add(own, own_low);
        if (all_cols && (i + 1) * CS_C <= len) {
#pragma unroll
            for (int e = 0; e < 4; ++e) op[(size_t)(e & 1) * ld + (e >> 1) * 8] = own[e];
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (i * CS_C + t_own + (e & 1) < len && jr[e >> 1] < V) op[(size_t)(e & 1) * ld + (e >> 1) * 8] = own[e];
        }
        op += (size_t)CS_C * ld;
        // S <- G S + sum_s (k F)_s v_s^T
#pragma unroll
        for (int m = 0; m < NK / 32; ++m) {
            uint32_t r[3][4];
#pragma unroll
            for (int p = 0; p < 3; ++p) cm_ldsm4t(r[p], rec.kf[p] + row_a * QP + k0 + m * 16 + col_a);
            float sl[2][4];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                const float2 G2 = *reinterpret_cast<const float2*>(&rec.G[k0 + m * 16 + nt * 8 + c2]);
#pragma unroll
                for (int e = 0; e < 4; ++e) { S[2 * m + nt][e] *= (e & 1) ? G2.y : G2.x; sl[nt][e] = 0.f; }
            }
            cm_mma_rows(&S[2 * m], sl, va, r);
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

// Shared memory to ask for so that no SM takes more blocks than an even spread gives it: the blocks run for long, and those
// that start while the kernel in front still holds part of the SMs would otherwise crowd the rest.
static inline size_t chunk_even_smem(size_t need, long long blocks) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) return need;
    constexpr size_t sm_all = 228 * 1024, most = 227 * 1024, own = 1024;      // an SM's, a block's largest, and what a block takes for itself
    const size_t per_sm = (size_t)((blocks + sms - 1) / sms), share = sm_all / (per_sm + 1);
    if (share < own) return need;
    const size_t even = (share - own) / 16 * 16 + 16;       // just too much for one block more
    return need > even ? need : (even > most ? most : even);
}

template <int NK, int W, bool DELTA>
static int chunk_scan_one(const ChunkScanArgs& A, int n_seqs, int live, cudaStream_t stream) {
    const dim3 grid(n_seqs, A.heads, (A.V + 16 * W - 1) / (16 * W));
    const size_t smem = chunk_even_smem(sizeof(ChunkScanSmem<NK, W, DELTA>), (long long)live * grid.y * grid.z);
    FF_SMEM_LIMIT((chunk_scan_kernel<NK, W, DELTA>), 227 * 1024);
    FF_LAUNCH((chunk_scan_kernel<NK, W, DELTA>), grid, 64 * W + CS_LOADERS, smem, stream, A);
    FF_LAUNCH_CHECK();
    return 0;
}

// Value columns of a block, in sixteens: four warp pairs share a record where that still gives most SMs a block, else two.
template <int NK, bool DELTA>
static int chunk_scan_launch(const ChunkScanArgs& A, int n_seqs, int live, cudaStream_t stream) {
    if ((long long)live * A.heads * ((A.V + 63) / 64) >= 90) return chunk_scan_one<NK, 4, DELTA>(A, n_seqs, live, stream);
    return chunk_scan_one<NK, 2, DELTA>(A, n_seqs, live, stream);
}

}  // namespace ff
