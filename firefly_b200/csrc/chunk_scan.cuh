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

#include <type_traits>

namespace ff {

constexpr int CS_C = 16;                                    // tokens a chunk
// A record: rows side by side, so that whole sectors are written (with the pitch that shared memory wants,
// which made rows straddle them, the first kernels took 67 us instead of 46, 40 instead of 31 and 102 instead of 82).
template <int NK, bool DELTA>
struct ChunkRecord {
    bf16 qe[3][CS_C * NK];                                  // q E (the decays in front of the token for a read-out in front of the write)
    bf16 kf[3][CS_C * NK];                                  // k F
    bf16 P[3][CS_C * CS_C];
    float G[NK];
    bf16 ke[DELTA ? 3 : 1][DELTA ? CS_C * NK : 8];          // k E
    bf16 TB[DELTA ? 3 : 1][DELTA ? CS_C * CS_C : 8];        // T diag(beta)
};
// The same as the walk has it in shared memory.
template <int NK, bool DELTA>
struct ChunkRows {
    static constexpr int QP = NK + 8, PP = CS_C + 8;        // row pitches: 16-byte pieces of eight rows lie in different banks
    bf16 qe[3][CS_C * QP], kf[3][CS_C * QP], P[3][CS_C * PP];
    float G[NK];
    bf16 ke[DELTA ? 3 : 1][DELTA ? CS_C * QP : 8], TB[DELTA ? 3 : 1][DELTA ? CS_C * PP : 8];
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

// The sequence and chunk of record r (chunk -1: none), the chunk's first token and how many the sequence has from there on; all lanes of
// a warp ask together, and the sequence's borders come from the lanes that have read them.
template <int C = CS_C>
__device__ __forceinline__ void chunk_of_record(const int* cu_q, int n_seqs, int r, int min_len, int& s, int& chunk, int& row0, int& left) {
    const int lane = threadIdx.x & 31;
    int begin = 0, end = 0;
    s = -1;
    for (int s0 = 0; s0 < n_seqs; s0 += 32) {
        const int i = min(s0 + lane, n_seqs - 1), at = cu_q[i], next = cu_q[i + 1];
        const unsigned m = __ballot_sync(0xffffffffu, s0 + lane < n_seqs && chunk_first_record<C>(at, s0 + lane) <= r);
        if (m) {
            const int l = 31 - __clz(m);
            s = s0 + l;
            begin = __shfl_sync(0xffffffffu, at, l);
            end = __shfl_sync(0xffffffffu, next, l);
        }
        if (m != 0xffffffffu) break;
    }
    chunk = -1;
    row0 = left = 0;
    if (s >= 0) {
        const int i = r - chunk_first_record<C>(begin, s);
        if (end - begin >= min_len && i * C < end - begin) {
            chunk = i;
            row0 = begin + i * C;
            left = end - row0;
        }
    }
}

// ---------------------------------------------------------------------------------- the first kernel's parts --
// A warp forms 64 key channels of a record, two a lane, all sixteen tokens: NK / 64 warps a record, CF_WARPS warps a block.  Token
// after token in registers: d_s, k of an earlier token times the decays since, is all that P needs of it, and k F in the end; a row
// of P is the lanes' shares of q_t d_s, joined by shuffles that halve the sums a lane still adds up.
// Formed out of rows in shared memory with a thread a token and eight channels, the same rows were read once for every token in front:
// 90 % of the shared-memory pipe.  What bounds it now are some 2400 instructions a warp (delta rule: 5900, the decays' logarithms
// and exponentials among them) and the 16 to 20 warps an SM that their registers leave to hide waits with.
// us, before / now: wkv, 4900 tokens of 32 heads of 64 74.4 / 46, channel decays, 3000 tokens of 16 heads of 64 46.1 / 31, delta rule, 8192 tokens of 8
// heads of 128 136 / 82.  (The delta rule with its rows in registers, as the other two have them, took a tenth longer; the other two with
// theirs in shared memory are no faster and keep the second kernel's blocks off the SMs until they end: 12 us longer for wkv.)
constexpr int CF_WARPS = 4;
template <int NK> constexpr int cf_warps_a_record() { return NK / 64; }
template <int NK> constexpr int cf_records() { return CF_WARPS / cf_warps_a_record<NK>(); }
template <int NK> static inline dim3 cf_grid(int n_records, int heads) { return dim3((unsigned)((n_records + cf_records<NK>() - 1) / cf_records<NK>()), (unsigned)heads); }

template <int NK, bool DELTA>
struct ChunkForm {                                          // of one record
    static constexpr int PITCH = CS_C + 4;
    struct Rows { uint32_t q[DELTA ? CS_C : 1][32], k[DELTA ? CS_C : 1][32]; float2 a[DELTA ? CS_C : 1][32]; };       // a warp's 64 channels, two a lane
    Rows rows[DELTA ? cf_warps_a_record<NK>() : 1];
    float P[cf_warps_a_record<NK>()][CS_C][PITCH];          // each warp's share of q_t d_s, s <= t
    float M[DELTA ? cf_warps_a_record<NK>() : 1][DELTA ? CS_C : 1][PITCH];         // and of k_t d_s, s < t; then T diag(beta)
    float sums[DELTA ? cf_warps_a_record<NK>() : 1][32];    // of q^2 and k^2 of the tokens
    float2 unit[DELTA ? CS_C : 1];                          // what q and k are multiplied by
    float beta[DELTA ? CS_C : 1];
};
// all warps of the thread's record
template <int NK> __device__ __forceinline__ void cf_sync() {
    if constexpr (NK == 64) __syncwarp();
    else cm_barrier(1 + threadIdx.x / (NK / 2), NK / 2);
}

__device__ __forceinline__ f32x2 cf_pair(uint32_t p) { return f2_pack(cm_lo(p), cm_hi(p)); }

// Asks for a warp's rows of q and k (bfloat16) and, with DECAYS, of what the decays are made of (32-bit): the `left` first of sixteen
// tokens, zeros behind them.  q, k, a: the warp's first channel of the chunk's first token; rows on 16 bytes.
template <bool DECAYS, typename Rows>
__device__ __forceinline__ void cf_fetch(Rows& to, const bf16* q, size_t q_stride, const bf16* k, size_t k_stride, const float* a, size_t a_stride, int left) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = i * 4 + (lane >> 3), c = lane & 7;
        const bool in = t < left;
        cm_copy16(&to.q[t][c * 4], q + (in ? t * q_stride + c * 8 : 0), in);
        cm_copy16(&to.k[t][c * 4], k + (in ? t * k_stride + c * 8 : 0), in);
    }
    if (DECAYS) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int t = i * 2 + (lane >> 4), c = lane & 15;
            const bool in = t < left;
            cm_copy16(&to.a[t][c * 2], a + (in ? t * a_stride + c * 4 : 0), in);
        }
    }
    cm_copy_commit();
    cm_copy_wait<0>();
    __syncwarp();
}

// v[0 .. V) summed over groups of LANES lanes; a lane keeps the sum cf_kept<V>(lane).
template <int V, int LANES>
__device__ __forceinline__ float cf_join(float (&v)[CS_C]) {
    const int lane = threadIdx.x & 31;
    int off = 1;
#pragma unroll
    for (int m = V / 2; m >= 1; m >>= 1) {
        const bool up = lane & off;
#pragma unroll
        for (int i = 0; i < m; ++i) {
            const float away = up ? v[i] : v[i + m];
            v[i] = (up ? v[i + m] : v[i]) + __shfl_xor_sync(0xffffffffu, away, off);
        }
        off <<= 1;
    }
#pragma unroll
    for (; off < LANES; off <<= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
    return v[0];
}
template <int V> __device__ __forceinline__ int cf_kept(int lane) {
    int i = 0, m = V / 2;
#pragma unroll
    for (int off = 1; off < V; off <<= 1, m >>= 1) i += (lane & off) ? m : 0;
    return i;
}

// The lane's two channels (of the warp's 64) of q E, k E, k F and G into the record, and the shares of P (and M) into sh.  token(t): q, k
// and the decays of the lane's channels.  BEFORE: the read-out sees the state in front of the token's own decay and write, and its
// own write by u.
template <int NK, bool DELTA, bool BEFORE, typename Token>
__device__ __forceinline__ void chunk_form(ChunkRecord<NK, DELTA>* rec, ChunkForm<NK, DELTA>& sh, int warp, f32x2 u, Token token) {
    constexpr int PW = NK / 2, PART = CS_C * PW;
    const int lane = threadIdx.x & 31, col = warp * 32 + lane;
    auto put = [&](bf16* to, int t, f32x2 v) {
        uint32_t* dst = reinterpret_cast<uint32_t*>(to) + t * PW + col;
        cm_split3(f2_low(v), f2_high(v), dst[0], dst[PART], dst[2 * PART]);
    };
    f32x2 d[CS_C], E = f2_pack(1.f, 1.f), q, k, a, q_next, k_next, a_next;
    token(0, q_next, k_next, a_next);
#pragma unroll
    for (int t = 0; t < CS_C; ++t) {
        q = q_next;
        k = k_next;
        a = a_next;
        if (t + 1 < CS_C) token(t + 1, q_next, k_next, a_next);        // in front of the writes of sums below, which the compiler must not pass
        if (!BEFORE) {
            E = f2_mul(E, a);
#pragma unroll
            for (int s = 0; s < t; ++s) d[s] = f2_mul(d[s], a);
            d[t] = k;
        }
        put(rec->qe[0], t, f2_mul(q, E));
        if constexpr (DELTA) put(rec->ke[0], t, f2_mul(k, E));
        float x[CS_C], y[CS_C];
#pragma unroll
        for (int s = 0; s < CS_C; ++s) {
            x[s] = s < t || (!BEFORE && s == t) ? f2_sum(f2_mul(q, d[s])) : 0.f;
            if constexpr (DELTA) y[s] = s < t ? f2_sum(f2_mul(k, d[s])) : 0.f;
        }
        if constexpr (BEFORE) x[t] = f2_sum(f2_mul(f2_mul(q, u), k));
        if constexpr (DELTA) {                              // half of the lanes go on with the sums of q, half with those of k
            const bool other = lane & 16;
#pragma unroll
            for (int s = 0; s <= t; ++s) {
                const float away = other ? x[s] : y[s];
                x[s] = (other ? y[s] : x[s]) + __shfl_xor_sync(0xffffffffu, away, 16);
            }
        }
        constexpr int L = DELTA ? 16 : 32;
        float sum;
        int at;
        if (t == 0) { sum = cf_join<1, L>(x); at = cf_kept<1>(lane); }
        else if (t < 2) { sum = cf_join<2, L>(x); at = cf_kept<2>(lane); }
        else if (t < 4) { sum = cf_join<4, L>(x); at = cf_kept<4>(lane); }
        else if (t < 8) { sum = cf_join<8, L>(x); at = cf_kept<8>(lane); }
        else { sum = cf_join<16, L>(x); at = cf_kept<16>(lane); }
        if constexpr (DELTA) {
            if (lane & 16) sh.M[warp][t][at] = sum;
            else sh.P[warp][t][at] = sum;
        } else sh.P[warp][t][at] = sum;
        if constexpr (BEFORE) {
            E = f2_mul(E, a);
#pragma unroll
            for (int s = 0; s < t; ++s) d[s] = f2_mul(d[s], a);
            d[t] = k;
        }
    }
#pragma unroll
    for (int t = 0; t < CS_C; ++t) put(rec->kf[0], t, d[t]);
    *reinterpret_cast<float2*>(&rec->G[2 * col]) = make_float2(f2_low(E), f2_high(E));
}

// A lower triangle of 16 x 16 (the sum of N shares) into its place in a record, split, with zeros above the diagonal; the record's threads.
template <int NK, int N, int PITCH>
__device__ __forceinline__ void chunk_emit(bf16* to, const float (*m)[CS_C][PITCH]) {
    constexpr int PW = CS_C / 2, PART = CS_C * PW, THREADS = NK / 2;
#pragma unroll
    for (int i = 0; i < CS_C * CS_C / 2 / THREADS; ++i) {
        const int idx = threadIdx.x % THREADS + i * THREADS, t = idx / (CS_C / 2), s = idx % (CS_C / 2) * 2;
        float2 x = *reinterpret_cast<const float2*>(&m[0][t][s]);
        if constexpr (N == 2) {
            const float2 y = *reinterpret_cast<const float2*>(&m[1][t][s]);
            x.x += y.x;
            x.y += y.y;
        }
        uint32_t* dst = reinterpret_cast<uint32_t*>(to) + t * PW + s / 2;
        cm_split3(s <= t ? x.x : 0.f, s + 1 <= t ? x.y : 0.f, dst[0], dst[PART], dst[2 * PART]);
    }
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
    struct Stage { ChunkRows<NK, DELTA> rec; bf16 v[CS_C * (16 * W + 8)]; };
    Stage stage[CS_STAGES];
    float xch[2][2 * W][DELTA ? 12 : 4][32];
    float slow[2 * W][16][CS_C + 1];
};

// One block per (sequence, head, 16 W value columns).  Two warps hold S^T of 16 value columns, half of the keys each, as the
// accumulators of mma.sync; the same registers are, split, the left operand of S^T (q E), so the state goes nowhere between the
// products.  The two exchange their shares of S^T (q E) and S^T (k E); what follows of the read-out each does for eight of the
// tokens.  Two more warps bring in records and values by 16-byte copies, two chunks ahead; one barrier a chunk.
// (With all keys in one warp, which also did its own loads, a chunk took half as long again: 135 against 90 us for three
// sequences of 1501, 1000 and 700 tokens with 16 heads of 64 x 128, 384 against 232 us for the delta rule on 4 x 2048 tokens.  With a
// quarter of the keys in a warp and twice the warps: 139 against 107 and 242 against 216.  With the read-out of a chunk ended behind
// the next one's barrier, so that only G S + (k F)^T v runs from chunk to chunk: 112 against 107, and as long for scalar decays.  What bounds a
// chunk is neither that chain nor the tensor cores (half of their time) nor the copies (a stage more or two: the same) but two warps a
// scheduler, which wait for their own instructions half of the time.)
template <int NK, int W, bool DELTA>
__global__ void __launch_bounds__(64 * W + CS_LOADERS) chunk_scan_kernel(ChunkScanArgs A) {
    pdl_prologue();
    using R = ChunkRows<NK, DELTA>;
    using Record = ChunkRecord<NK, DELTA>;
    using SM = ChunkScanSmem<NK, W, DELTA>;
    constexpr int QP = R::QP, PP = R::PP, VB = 16 * W, VP = VB + 8, NT = NK / 16;
    static_assert(sizeof(Record) % 16 == 0 && sizeof(R) % 16 == 0, "a record is copied in 16-byte pieces");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SM& sm = *reinterpret_cast<SM*>(smem_raw);
    const int s = blockIdx.x, h = blockIdx.y, j0 = blockIdx.z * VB, V = A.V;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t0 = A.cu_q[s], len = A.cu_q[s + 1] - t0, chunks = (len + CS_C - 1) / CS_C;
    if (len < A.min_len) return;
    if (warp >= 2 * W) {
        // ---- the warps that load
        const int pt = threadIdx.x - 64 * W;
        const Record* recs = pdl_fresh((const Record*)A.records) + (size_t)chunk_first_record(t0, s) * A.heads + h;
        // rows of N pieces of 16 bytes, which lie `pitch` numbers apart in shared memory
        auto copy_rows = [&](auto n, bf16* to, int pitch, const bf16* from, int rows) {
            constexpr int N = decltype(n)::value;
#pragma unroll 8
            for (int p = pt; p < rows * N; p += CS_LOADERS) cm_copy16(to + p / N * pitch + p % N * 8, from + p * 8, true);
        };
        using Row = std::integral_constant<int, NK / 8>;
        using Pair = std::integral_constant<int, CS_C / 8>;
        const bf16* vp = pdl_fresh(A.v) + A.v_off + (size_t)h * V + j0;
        auto load = [&](int i) {
            if (i < chunks) {
                typename SM::Stage& st = sm.stage[i % CS_STAGES];
                const Record* from = recs + (size_t)i * A.heads;
                copy_rows(Row(), st.rec.qe[0], QP, from->qe[0], 3 * CS_C);
                copy_rows(Row(), st.rec.kf[0], QP, from->kf[0], 3 * CS_C);
                copy_rows(Pair(), st.rec.P[0], PP, from->P[0], 3 * CS_C);
                if (pt < NK / 4) cm_copy16(st.rec.G + pt * 4, from->G + pt * 4, true);
                if constexpr (DELTA) {
                    copy_rows(Row(), st.rec.ke[0], QP, from->ke[0], 3 * CS_C);
                    copy_rows(Pair(), st.rec.TB[0], PP, from->TB[0], 3 * CS_C);
                }
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
            for (int nt = 0; nt < 2; ++nt) {
                cm_add(acc[nt], low[nt]);
                if constexpr (DELTA) cm_add(pred[nt], plow[nt]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                mine[e][lane] = half ? acc[0][e] : acc[1][e];
                if constexpr (DELTA) {
                    mine[4 + e][lane] = pred[0][e];
                    mine[8 + e][lane] = pred[1][e];
                }
            }
            cm_barrier(1 + tile, 64);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                own[e] = (half ? acc[1][e] : acc[0][e]) + theirs[e][lane];
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
                cm_scale(S[2 * m + nt], *reinterpret_cast<const f32x2*>(&rec.G[k0 + m * 16 + nt * 8 + c2]));
#pragma unroll
                for (int e = 0; e < 4; ++e) sl[nt][e] = 0.f;
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
