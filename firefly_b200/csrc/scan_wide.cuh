// The inner part of the recurrences that walk a sequence token by token: a head's state S [key channel, value channel] in
// registers, four neighbouring value columns and NP / PARTS key channels of each a thread.
//
// What bounds such a walk is the arithmetic pipe and what feeds it: an element of S costs three operations a token
// (k v, the decayed sum, the read-out), so a thread's operands from shared memory (q, k and the decays of its key
// channels) must serve several columns.  Four columns a thread read a quarter of what one column a thread read, and two
// key channels at a time go through one packed 32-bit instruction.  Blocks are four warps, one for every quarter of an
// SM, however many columns that makes; a head's columns go to as many blocks as they need.
//
// The state lies in the slot as [heads][V][NP], whatever kernel wrote it.
#pragma once

#include "common.cuh"

namespace ff {

using f32x2 = unsigned long long;      // two 32-bit numbers, the first in the low half

__device__ __forceinline__ f32x2 f2_fma(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 f2_add(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 f2_mul(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 f2_pack(float lo, float hi) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float f2_low(f32x2 a) { return __uint_as_float((unsigned)a); }
__device__ __forceinline__ float f2_high(f32x2 a) { return __uint_as_float((unsigned)(a >> 32)); }
__device__ __forceinline__ float f2_sum(f32x2 a) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a));
    return lo + hi;
}

constexpr int WS_THREADS = 128;
constexpr int WS_COLS = 4;             // value columns a thread

// the key size a recurrence is instantiated for (0: not supported)
static inline __host__ __device__ int ws_key_size(int N) {
    return N <= 0 || N > 256 ? 0 : (N <= 16 ? 16 : (N <= 32 ? 32 : (N <= 64 ? 64 : (N <= 128 ? 128 : 256))));
}

template <int NP>
struct WideState {
    static constexpr int PARTS = NP <= 32 ? 4 : NP / 8;        // threads that share a value column
    static constexpr int KP = NP / PARTS;                      // key channels a thread holds of each of its columns
    static constexpr int VB = WS_THREADS / PARTS * WS_COLS;    // value columns a block
    static constexpr int CH = NP <= 128 ? 8 : 4;               // tokens staged at a time
    f32x2 S[WS_COLS][KP / 2];
    int part, jl;                                              // thread `part` of the columns 4 jl ..: key channels 4 PARTS m + 4 part + e

    __device__ __forceinline__ void place(int tid) { part = tid % PARTS; jl = tid / PARTS; }

    // `head`: the head's [V][NP] floats in the slot
    __device__ __forceinline__ void load(const float* head, int j0, int V, bool fresh) {
        const bool vec = ((uintptr_t)head & 15) == 0;
#pragma unroll
        for (int x = 0; x < WS_COLS; ++x) {
            const int j = j0 + jl * WS_COLS + x;
#pragma unroll
            for (int m = 0; m < KP / 4; ++m) {
                float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
                if (!fresh && j < V) {
                    const float* p = head + (size_t)j * NP + m * 4 * PARTS + part * 4;
                    if (vec) r = *reinterpret_cast<const float4*>(p);
                    else r = make_float4(p[0], p[1], p[2], p[3]);
                }
                S[x][2 * m] = f2_pack(r.x, r.y);
                S[x][2 * m + 1] = f2_pack(r.z, r.w);
            }
        }
    }
    __device__ __forceinline__ void store(float* head, int j0, int V) const {
        const bool vec = ((uintptr_t)head & 15) == 0;
#pragma unroll
        for (int x = 0; x < WS_COLS; ++x) {
            const int j = j0 + jl * WS_COLS + x;
#pragma unroll
            for (int m = 0; m < KP / 4; ++m) {
                if (j < V) {
                    float* p = head + (size_t)j * NP + m * 4 * PARTS + part * 4;
                    float4 r;
                    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(S[x][2 * m]));
                    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.z), "=f"(r.w) : "l"(S[x][2 * m + 1]));
                    if (vec) *reinterpret_cast<float4*>(p) = r;
                    else { p[0] = r.x; p[1] = r.y; p[2] = r.z; p[3] = r.w; }
                }
            }
        }
    }

    // One token: S <- d S + k v^T and the thread's share of S^T q, of the state behind the write (or in front of decay
    // and write with BEFORE).  q, k, d: the staged rows; with CD false the decay is `a` for every key channel.  `v`: the
    // thread's values, each twice, as they are staged.
    template <bool CD, bool BEFORE>
    __device__ __forceinline__ void token(const float* q, const float* k, const float* d, float a, const f32x2 v[WS_COLS],
                                          float out[WS_COLS]) {
        f32x2 acc[WS_COLS];
        const f32x2 aa = CD ? 0ull : f2_pack(a, a);
#pragma unroll
        for (int m = 0; m < KP / 4; ++m) {
            const int at = m * 4 * PARTS + part * 4;
            const ulonglong2 q2 = *reinterpret_cast<const ulonglong2*>(q + at);
            const ulonglong2 k2 = *reinterpret_cast<const ulonglong2*>(k + at);
            ulonglong2 d2 = make_ulonglong2(aa, aa);
            if constexpr (CD) d2 = *reinterpret_cast<const ulonglong2*>(d + at);
#pragma unroll
            for (int x = 0; x < WS_COLS; ++x) {
                f32x2& s0 = S[x][2 * m];
                f32x2& s1 = S[x][2 * m + 1];
                if constexpr (BEFORE) {
                    acc[x] = m == 0 ? f2_mul(q2.x, s0) : f2_fma(q2.x, s0, acc[x]);
                    acc[x] = f2_fma(q2.y, s1, acc[x]);
                }
                s0 = f2_fma(d2.x, s0, f2_mul(k2.x, v[x]));
                s1 = f2_fma(d2.y, s1, f2_mul(k2.y, v[x]));
                if constexpr (!BEFORE) {
                    acc[x] = m == 0 ? f2_mul(q2.x, s0) : f2_fma(q2.x, s0, acc[x]);
                    acc[x] = f2_fma(q2.y, s1, acc[x]);
                }
            }
        }
#pragma unroll
        for (int x = 0; x < WS_COLS; ++x) out[x] = f2_sum(acc[x]);
    }
    // the thread's four values of a token, staged twice each
    static __device__ __forceinline__ void values(const f32x2* row, f32x2 v[WS_COLS]) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(row), b = *reinterpret_cast<const ulonglong2*>(row + 2);
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    }

    // The sum over a column's threads of their shares; thread `part` returns that of column `col()` (threads part and
    // part + 4 the same one).
    __device__ __forceinline__ float reduce(const float x[WS_COLS]) const {
        const bool b0 = part & 1, b1 = part & 2;
        float r0 = b0 ? x[2] : x[0], r1 = b0 ? x[3] : x[1];
        r0 += __shfl_xor_sync(0xffffffffu, b0 ? x[0] : x[2], 1);
        r1 += __shfl_xor_sync(0xffffffffu, b0 ? x[1] : x[3], 1);
        float y = b1 ? r1 : r0;
        y += __shfl_xor_sync(0xffffffffu, b1 ? r0 : r1, 2);
#pragma unroll
        for (int off = 4; off < PARTS; off <<= 1) y += __shfl_xor_sync(0xffffffffu, y, off);
        return y;
    }
    __device__ __forceinline__ int col() const { return ((part & 1) << 1) | ((part >> 1) & 1); }

    // The same for a whole chunk, shares x[4 token + column]: every step halves what a thread still adds up, so the
    // exchanges are few, do not wait for one another, and every thread ends with OUTS of the sums in x[0..]: those
    // of `first()` and the following ones in the same count.
    static constexpr int OUTS = CH * WS_COLS / PARTS > 1 ? CH * WS_COLS / PARTS : 1;
    __device__ __forceinline__ void reduce_chunk(float x[CH * WS_COLS]) const {
        int off = 1;
#pragma unroll
        for (int m = CH * WS_COLS / 2; m >= 1; m >>= 1) {
            if (off < PARTS) {
                const bool up = part & off;
#pragma unroll
                for (int i = 0; i < m; ++i) {
                    const float away = up ? x[i] : x[i + m];
                    x[i] = (up ? x[i + m] : x[i]) + __shfl_xor_sync(0xffffffffu, away, off);
                }
                off <<= 1;
            }
        }
#pragma unroll
        for (; off < PARTS; off <<= 1) x[0] += __shfl_xor_sync(0xffffffffu, x[0], off);
    }
    __device__ __forceinline__ int first() const {
        int at = 0, off = 1;
#pragma unroll
        for (int m = CH * WS_COLS / 2; m >= 1; m >>= 1) {
            if (off < PARTS) {
                if (part & off) at += m;
                off <<= 1;
            }
        }
        return at;
    }
};

}  // namespace ff
