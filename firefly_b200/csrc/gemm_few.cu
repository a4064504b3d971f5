// out[t, n] = sum_k x[t, k] * W[n, k] for steps of one to eight tokens.
//
// Such a product is the time to stream W, and in a small model not even that: its few microseconds are a chain of a launch, the
// fetch of the activations, the sum and the way to the next kernel.  The tcgen05 product (gemm_tcgen05.cu) has a tensor-memory
// allocation, mbarriers, a cluster of K ranges with two cluster barriers and sums out of other blocks' shared memory on that
// chain.  Here a block of NW warps holds 16 rows of W over all of K and nothing outside it is waited for: a lane copies 16
// bytes of a row at a time into shared memory, all of them before the kernel in front has ended, and reads back what it copied
// itself as the left operand of mma.sync m16n8k16 (which eight of k a register pair stands for is the same for W and x, so the order
// within a row need not be undone); the tokens are the eight columns of the right one, and the warps' shares of a sum meet once in
// shared memory.  The rows wait in shared memory because registers would keep the next product's blocks off the SM until this one's have
// gone: chains of one product of the 0.6B shape for one token (q|k|v, o, gate|up, down; before: gemm_tcgen05.cu) take 5.4 / 5.3 / 6.5 / 5.9
// -> 2.9 / 2.2 / 3.8 / 2.6 us, with the rows in registers 3.6 / 2.7 / 4.3 / 3.7; its decode step of 28 layers 938 -> 657 us, 836 in registers.
//
// The epilogues and the RMSNorm folded in on both sides are those of gemm_tcgen05.cu; a sum of squares stands for the rows of a block.
// A product behind it that gemm_tcgen05.cu takes adds eight times as many of them, one thread a token: o here or there with gate|up there, us a pair, one
// token: 2048 x 2048 with 12288 x 2048 17.9 / 18.8, 2560 x 2560 with 19456 x 2560 23.6 / 25.7, of the 2.8 that o alone is faster.  (32 of them asked
// for at once there instead of eight gave 16.8 of these 17.9, but cost every other product behind a norm 0.1 to 0.7.)
#include "chunk_mma.cuh"

#include <algorithm>

namespace ff {

enum FewEpilogue { FEW_BF16 = 0, FEW_F32 = 1, FEW_RESIDUAL_ADD = 2, FEW_SWIGLU = 3, FEW_RELU2 = 4 };
constexpr int FEW_TOKENS = 8, FEW_K = 32;                    // tokens at most; k of a step: 16 bytes of a row in each of four lanes
constexpr int FEW_ROWS = 16;                                 // rows of W a block takes
constexpr int FEW_PITCH = FEW_ROWS + 4;                      // of the shares of a sum: four tokens' eight rows lie in different banks
constexpr int FEW_SQ = 4;                                    // sums of squares a lane asks for at once: those of 128 blocks
constexpr int FEW_AHEAD = 4;                                 // steps of x a lane asks for at once
constexpr int FEW_MAX_K = 3584;                              // a block's rows take 112 KB at most

struct FewArgs {
    const bf16* x; const bf16* w; void* out;
    int ldo, T, N, K, epilogue;
    bf16* xw_out; const float* xw_w; float* ssq_out;         // norm folded in, producing side
    const float* ssq_in; int ssq_parts, norm_dim; float norm_eps;      // consuming side
};

// what the kernel in front wrote: only the L2 cache has it for certain
__device__ __forceinline__ uint4 few_rows(const bf16* p) {
    uint4 v;
    asm volatile("ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}

constexpr int FEW_THREADS_SM = 1024;                         // threads an SM that its registers are shared out for

template <int NW>
__global__ void __launch_bounds__(32 * NW, FEW_THREADS_SM / (32 * NW)) gemm_few_kernel(const FewArgs a) {
    constexpr int RP = FEW_PITCH;
    extern __shared__ __align__(16) uint4 w_rows[];           // [step of the warp][row half][thread]
    __shared__ float part[NW][FEW_TOKENS][RP];
    __shared__ float s_inv[FEW_TOKENS];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
    const int n0 = blockIdx.x * FEW_ROWS, steps = a.K / FEW_K, mine = (steps - warp + NW - 1) / NW;      // steps of this warp: warp, warp + NW, ...
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        // gate and up rows alternate in sixteens: a block takes eight of the ones and the same eight of the others
        const int row = a.epilogue == FEW_SWIGLU ? (n0 & ~31) + r * 16 + (n0 & 16) / 2 + g : n0 + r * 8 + g;
        const bf16* wp = a.w + (size_t)min(row, a.N - 1) * a.K + warp * FEW_K + c * 8;
#pragma unroll 4
        for (int i = 0; i < mine; ++i) cm_copy16(w_rows + (i * 2 + r) * 32 * NW + threadIdx.x, wp + (size_t)i * NW * FEW_K, true);
    }
    cm_copy_commit();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const bool live = g < a.T;
    const bf16* xp = a.x + (size_t)(live ? g : 0) * a.K + warp * FEW_K + c * 8;
    uint4 xv[FEW_AHEAD];
#pragma unroll
    for (int d = 0; d < FEW_AHEAD; ++d) {
        xv[d] = make_uint4(0, 0, 0, 0);
        if (d < mine && live) xv[d] = few_rows(xp + (size_t)d * NW * FEW_K);
    }
    // what the epilogue needs of this thread's output is on its way while the products run
    const int row = threadIdx.x % FEW_ROWS, tok = threadIdx.x / FEW_ROWS, n = n0 + row;
    const bool owns = tok < a.T && n < a.N;                   // 32 NW >= 8 * 16 threads
    float res = 0.f, wn = 0.f;
    if (a.epilogue == FEW_RESIDUAL_ADD && owns) {
        res = __ldcg(reinterpret_cast<const float*>(a.out) + (size_t)tok * a.ldo + n);
        if (a.xw_out) wn = __ldg(a.xw_w + n);
    }
    float sq_part[FEW_SQ];                                    // a warp a token: its sums of squares, all on their way at once
#pragma unroll
    for (int j = 0; j < FEW_SQ; ++j) {
        const int p = lane + 32 * j;
        sq_part[j] = a.ssq_in && warp < a.T && p < a.ssq_parts ? __ldcg(a.ssq_in + (size_t)p * a.T + warp) : 0.f;
    }
    float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};      // the even and the odd sixteens of k
    cm_copy_wait<0>();                                        // a lane reads what it copied itself: nobody else is waited for
    for (int i0 = 0; i0 < mine; i0 += FEW_AHEAD) {
#pragma unroll
        for (int d = 0; d < FEW_AHEAD; ++d) {
            const int i = i0 + d;
            if (i >= mine) break;
            const uint4 lo = w_rows[i * 2 * 32 * NW + threadIdx.x], hi = w_rows[(i * 2 + 1) * 32 * NW + threadIdx.x];
            const uint32_t a0[4] = {lo.x, hi.x, lo.y, hi.y}, a1[4] = {lo.z, hi.z, lo.w, hi.w};
            const uint32_t b0[2] = {xv[d].x, xv[d].y}, b1[2] = {xv[d].z, xv[d].w};
            cm_mma(acc[0], a0, b0);
            cm_mma(acc[1], a1, b1);
            if (i + FEW_AHEAD < mine && live) xv[d] = few_rows(xp + (size_t)(i + FEW_AHEAD) * NW * FEW_K);
        }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) part[warp][2 * c + (e & 1)][(e >> 1) * 8 + g] = acc[0][e] + acc[1][e];
    if (a.ssq_in && warp < a.T) {                             // in a fixed order
        float ss = 0.f;
#pragma unroll
        for (int j = 0; j < FEW_SQ; ++j) ss += sq_part[j];
        for (int p = lane + 32 * FEW_SQ; p < a.ssq_parts; p += 32) ss += __ldcg(a.ssq_in + (size_t)p * a.T + warp);
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
        if (lane == 0) s_inv[warp] = 1.0f / sqrtf(ss / (float)a.norm_dim + a.norm_eps);
    }
    __syncthreads();
    if (tok >= FEW_TOKENS) return;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < NW; ++w) v += part[w][tok][row];      // in the warps' order
    if (a.ssq_in && tok < a.T) v *= s_inv[tok];
    if (a.epilogue == FEW_SWIGLU) {
        // the first half of a block's rows are gate rows, the second the up rows of the same columns
        const float up = __shfl_xor_sync(0xffffffffu, v, FEW_ROWS / 2);
        const int col = n0 / 2 + row;
        if (owns && row < FEW_ROWS / 2) reinterpret_cast<bf16*>(a.out)[(size_t)tok * a.ldo + col] = __float2bfloat16_rn(v / (1.0f + expf(-v)) * up);
    } else if (a.epilogue == FEW_RESIDUAL_ADD) {
        const float r = res + v;
        if (owns) reinterpret_cast<float*>(a.out)[(size_t)tok * a.ldo + n] = r;
        if (a.xw_out) {
            if (owns) a.xw_out[(size_t)tok * a.N + n] = __float2bfloat16_rn(r * wn);
            float sq = owns ? r * r : 0.f;
#pragma unroll
            for (int off = FEW_ROWS / 2; off >= 1; off >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, off);
            if (row == 0 && tok < a.T) a.ssq_out[(size_t)blockIdx.x * a.T + tok] = sq;
        }
    } else if (owns) {
        const size_t o = (size_t)tok * a.ldo + n;
        if (a.epilogue == FEW_F32) reinterpret_cast<float*>(a.out)[o] = v;
        else {
            const float p = a.epilogue == FEW_RELU2 ? fmaxf(v, 0.f) * fmaxf(v, 0.f) : v;
            reinterpret_cast<bf16*>(a.out)[o] = __float2bfloat16_rn(p);
        }
    }
}

static int few_blocks(int N) { return (N + FEW_ROWS - 1) / FEW_ROWS; }
template <int NW> static size_t few_rows_bytes(int K) { return (size_t)((K / FEW_K + NW - 1) / NW) * 2 * 32 * NW * 16; }
// blocks that an SM holds: its 228 KB, of which every block takes 1 KB besides its rows and its static part
template <int NW> static int few_blocks_per_sm(int K) {
    const size_t block = few_rows_bytes<NW>(K) + (size_t)NW * FEW_TOKENS * FEW_PITCH * sizeof(float) + FEW_TOKENS * sizeof(float) + 1024;
    return (int)std::min<size_t>(228 * 1024 / block, FEW_THREADS_SM / (32 * NW));
}

template <int NW>
static int few_launch(const FewArgs& a, cudaStream_t stream) {
    static_assert(32 * NW >= FEW_TOKENS * FEW_ROWS && NW >= FEW_TOKENS, "a thread an output, a warp a token's sum of squares");
    FF_SMEM_LIMIT(gemm_few_kernel<NW>, FEW_ROWS * FEW_MAX_K * 2);
    FF_LAUNCH(gemm_few_kernel<NW>, few_blocks(a.N), 32 * NW, few_rows_bytes<NW>(a.K), stream, a);
    FF_LAUNCH_CHECK();
    return 0;
}

}  // namespace ff

using namespace ff;

FF_EXPORT int ff_gemm_few_rows() { return FEW_ROWS; }

// Whether a product takes this kernel on a GPU of so many SMs: where all its blocks are there at once.  Then it is 1.2 to 1.6 times as fast as
// gemm_tcgen05.cu (alone, 1 and 8 tokens, K of 1792 to 3584).  A second round of blocks has nothing under way while it copies its rows, 2.5 us: us here / there, 8
// tokens: K = 2560, N = 4736 (one round) 6.1 / 8.3, 5008 9.1 / 8.6, 7104 (a round and a half) 10.0 / 10.9; K = 3328 7.8 / 9.5, 12.0 / 9.9, 13.1 / 12.9; K = 3584, of which
// an SM holds one block, 2368 4.9 / 7.1, 3072 8.5 / 8.1, 5120 13.6 / 10.4.  It pays where the rows are short (K = 2304, N = 5008 8.0 / 8.3; 2048, 9232 10.3 / 10.6)
// or the second round is half full.  Every block reads all of x: with a second eight of tokens the wide products took longer than there
// (16 tokens: q|k|v 5.5 there / 6.3, gate|up 7.1 / 6.9), and a step with only the narrow ones here (o 5.4 / 4.0, down 6.1 / 4.6) 10 % longer.
FF_EXPORT int ff_gemm_few_usable(int T, int N, int K, int sms) {
    if (T > FEW_TOKENS || K <= 0 || K % FEW_K || K > FEW_MAX_K) return 0;
    const int blocks = few_blocks(N);
    if (blocks <= sms) return 1;                               // 16 warps a block, one an SM
    const int places = sms * few_blocks_per_sm<8>(K);
    if (blocks <= places) return 1;
    return blocks <= 4 * sms && (K <= 2304 || (K <= 3072 && 2 * blocks >= 3 * places));
}

// x: bfloat16 [T, K], T <= 8; w: bfloat16 [N, K]; K a multiple of 32 up to FEW_MAX_K; both on 16 bytes.  Epilogues, norm folded in: as
// ff_gemm_tc, with ssq_out [ceil(N / FEW_ROWS), T].
FF_EXPORT int ff_gemm_few(const void* x, const void* w, void* out, int ldo, int T, int N, int K, int epilogue, void* xw_out, const float* xw_w,
                          float* ssq_out, const float* ssq_in, int ssq_parts, int norm_dim, float norm_eps, cudaStream_t stream) {
    if (xw_out && (epilogue != FEW_RESIDUAL_ADD || !xw_w || !ssq_out)) return FF_ERR_BAD_ARG;
    if (ssq_in && (ssq_parts <= 0 || norm_dim <= 0)) return FF_ERR_BAD_ARG;
    if (T <= 0 || N <= 0) return 0;
    if (T > FEW_TOKENS || K <= 0 || K > FEW_MAX_K || K % FEW_K || epilogue < 0 || epilogue > FEW_RELU2 || (((uintptr_t)x | (uintptr_t)w) & 15))
        return FF_ERR_BAD_ARG;
    if (epilogue == FEW_SWIGLU && N % 32) return FF_ERR_UNSUPPORTED;
    const FewArgs a{(const bf16*)x, (const bf16*)w, out, ldo, T, N, K, epilogue, (bf16*)xw_out, xw_w, ssq_out, ssq_in, ssq_parts, norm_dim, norm_eps};
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return (int)e;
    // with a block an SM and fewer, more warps share its rows
    return few_blocks(N) <= sms ? few_launch<16>(a, stream) : few_launch<8>(a, stream);
}
