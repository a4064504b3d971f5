// The grouped products of routed experts on the fifth-generation tensor cores.
//
// A block takes one tile of 128 rows of one expert (the plan's row tiles, see moe.cu) and BC rows of the expert's
// matrices.  The rows are the M operand of tcgen05.mma and the matrices' rows its N operand; the accumulator
// [128 rows][BC] is in tensor memory.  For the first product the rows are tokens' activations picked by `src_tok`: four
// at a time by TMA gather, one gather a lane (a tile with fewer rows asks for that many only: what lies in shared memory
// beyond them only makes accumulator rows that nobody reads).  The experts' matrices are stacked, so that a box of
// weight rows is a plain 2D tile of one tall matrix.  With gate and up a tile's first half is gate rows and its second
// half the same rows of up: the pair of a column is in one thread's accumulator row, and the epilogue applies the
// activation there.  Two blocks share an SM, one's epilogue under the other's main loop.
//
// A result is a dot product over K in a fixed order, whatever shares its tile.  Every wait on an mbarrier is bounded:
// after about a second the kernel records an error code, lets its copies land, frees its tensor memory and returns.
#include "tcgen05.cuh"
#include "moe.cuh"

namespace ff {

constexpr int GM = GROUPED_TC_ROWS;   // rows of a row tile (MMA M)
constexpr int GROUPED_THREADS = 192;  // a warp for the loads, one for the MMAs, four for the epilogue

template <int BC> struct GroupedCfg {
    static constexpr int A_BYTES = GM * BK * 2;
    static constexpr int B_BYTES = BC * BK * 2;
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int STAGES = (108 * 1024) / STAGE_BYTES;          // two blocks an SM
    static constexpr size_t SMEM = (size_t)STAGES * STAGE_BYTES + 1024 /* alignment slack */ + 256 /* barriers */;
};

struct GroupedArgs {
    const int* src_tok;
    const int* seg;
    const int* tile_expert;
    const int* tile_row0;
    const int* n_tiles;
    const float* row_w;
    void* out;
    int N, K;
    float limit;
    int act;
    int* status;
};

__device__ __forceinline__ void tma_gather4(bool issue, uint32_t dst, const CUtensorMap* map, int x, const int (&r)[4], uint32_t bar) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %8, 0;\n\t"
                 "@q cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes "
                 "[%0], [%1, {%3, %4, %5, %6, %7}], [%2];\n\t}"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"((uint32_t)issue) : "memory");
}

template <int KIND, int BC>
__global__ void __launch_bounds__(GROUPED_THREADS)
moe_grouped_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b0,
                      const __grid_constant__ CUtensorMap map_b1, const GroupedArgs a) {
    using Cfg = GroupedCfg<BC>;
    constexpr int STAGES = Cfg::STAGES;
    constexpr bool GATHER = KIND != MOE_DOWN;
    constexpr int COLS = KIND == MOE_GATEUP ? BC / 2 : BC;             // output columns of a block
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(tiles + (size_t)STAGES * Cfg::STAGE_BYTES);
    // bars[0..S) full, bars[S..2S) empty, bars[2S] accumulator ready
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const bool issue = lane == 0;

    // the plan comes from the kernel in front: nothing can be asked for before it is there
    grid_dependency_wait();
    const int* seg = pdl_fresh(a.seg);
    if ((int)blockIdx.y >= *pdl_fresh(a.n_tiles)) return;
    const int e = pdl_fresh(a.tile_expert)[blockIdx.y], row0 = pdl_fresh(a.tile_row0)[blockIdx.y];
    const int rows = min(GM, seg[e + 1] - row0);
    const int n0 = blockIdx.x * COLS;
    const int n_iters = (a.K + BK - 1) / BK;

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int i = 0; i < 2 * STAGES + 1; ++i) mbar_init(smem_addr(&bars[i]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_addr(&s_tmem_base)), "r"((uint32_t)BC) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = s_tmem_base;
    volatile int* abort_flag = &s_abort;
    // only now: a kernel that starts early must not take tensor memory that this block still waits for
    grid_launch_dependents();

    if (warp == 0) {
        // ------------------------------------------------ producer: TMA loads --
        int src[4];
        const int groups = (rows + 3) >> 2;                            // gathers of four rows that the tile needs
        if (GATHER) {
            const int* st = pdl_fresh(a.src_tok);
#pragma unroll
            for (int j = 0; j < 4; ++j) src[j] = st[row0 + min(4 * lane + j, rows - 1)];
        }
        const uint32_t bytes = Cfg::B_BYTES + (GATHER ? (uint32_t)groups * 4 * BK * 2 : (uint32_t)Cfg::A_BYTES);
        int issued = 0;
        for (int it = 0; it < n_iters; ++it) {
            const int s = it % STAGES;
            if (it >= STAGES &&
                !__all_sync(0xffffffffu, mbar_wait(smem_addr(&bars[STAGES + s]), ((it / STAGES) & 1) ^ 1, a.status, abort_flag, 111)))
                break;
            const uint32_t full = smem_addr(&bars[s]);
            const uint32_t sa = smem_addr(tiles + (size_t)s * Cfg::STAGE_BYTES), sb = sa + Cfg::A_BYTES;
            mbar_expect_tx(issue, full, bytes);
            __syncwarp();
            if (KIND == MOE_GATEUP) {
                tma_load_2d(issue, sb, &map_b0, it * BK, e * a.N + n0, full);
                tma_load_2d(issue, sb + Cfg::B_BYTES / 2, &map_b1, it * BK, e * a.N + n0, full);
            } else {
                tma_load_2d(issue, sb, &map_b0, it * BK, e * a.N + n0, full);
            }
            if (GATHER) tma_gather4(lane < groups, sa + lane * 4 * BK * 2, &map_a, it * BK, src, full);
            else tma_load_2d(issue, sa, &map_a, it * BK, row0, full);
            issued = it + 1;
        }
        if (*abort_flag) {
            // let the copies that are still in flight land before the block's memory goes away
            for (int it = max(0, issued - STAGES); it < issued; ++it) {
                const unsigned long long start = clock64();
                while (!mbar_try_wait(smem_addr(&bars[it % STAGES]), (it / STAGES) & 1))
                    if (clock64() - start > WAIT_LIMIT_CYCLES) break;
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------ MMA issuer ----------
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BC >> 3) << 17) | ((uint32_t)(GM >> 4) << 24);
        for (int it = 0; it < n_iters; ++it) {
            const int s = it % STAGES;
            if (!__all_sync(0xffffffffu, mbar_wait(smem_addr(&bars[s]), (it / STAGES) & 1, a.status, abort_flag, 112))) break;
            tc_fence_after();
            const uint32_t sa = smem_addr(tiles + (size_t)s * Cfg::STAGE_BYTES), sb = sa + Cfg::A_BYTES;
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k)
                tc_mma_bf16(issue, tmem_base, smem_desc_sw128(sa + k * UMMA_K * 2), smem_desc_sw128(sb + k * UMMA_K * 2), idesc,
                            (it > 0 || k > 0) ? 1u : 0u);
            tc_commit(issue, smem_addr(&bars[STAGES + s]));            // stage free when these MMAs have read it
            __syncwarp();
        }
        tc_commit(issue, smem_addr(&bars[2 * STAGES]));                // accumulator complete
    } else {
        // ------------------------------------------------ epilogue: one accumulator row a thread --
        const int quad = warp & 3;                                     // this warp's 32 lanes of tensor memory
        const int r = quad * 32 + lane;
        const bool live = r < rows;
        const float wr = KIND != MOE_DOWN && a.row_w && live ? pdl_fresh(a.row_w)[row0 + r] : 1.0f;
        const bool ok = __all_sync(0xffffffffu, mbar_wait(smem_addr(&bars[2 * STAGES]), 0, a.status, abort_flag, 113)) && !*abort_flag;
        tc_fence_after();
        const uint32_t acc = tmem_base + ((uint32_t)(quad * 32) << 16);
        const int cols = min(COLS, a.N - n0);
        if (__all_sync(0xffffffffu, ok) && quad * 32 < rows) {          // the same for the whole warp: the loads are warp-wide
            const bool vec = (a.N & (KIND == MOE_DOWN ? 3 : 7)) == 0;  // 16-byte stores stay aligned
#pragma unroll 1
            for (int c0 = 0; c0 < cols; c0 += 16) {
                float v[16];
                tc_ld16(acc + c0, v);
                if constexpr (KIND == MOE_GATEUP) {
                    float u[16];
                    tc_ld16(acc + BC / 2 + c0, u);
                    if (a.act == 1) {                                  // one branch for all: a branch a value would keep them from overlapping
#pragma unroll
                        for (int i = 0; i < 16; ++i) v[i] = clamped_glu_fast(v[i] * wr, u[i] * wr, a.limit, 1);
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; ++i) v[i] = clamped_glu_fast(v[i] * wr, u[i] * wr, a.limit, 0);
                    }
                } else if constexpr (KIND == MOE_UP) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] = relu2(v[i] * wr);
                }
                if (!live) continue;
                const size_t o = (size_t)(row0 + r) * a.N + n0 + c0;
                if constexpr (KIND == MOE_DOWN) {
                    float* dst = (float*)a.out + o;
                    if (vec && c0 + 16 <= cols) {
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            reinterpret_cast<float4*>(dst)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            if (c0 + i < cols) dst[i] = v[i];
                    }
                } else {
                    bf16* dst = (bf16*)a.out + o;
                    if (vec && c0 + 16 <= cols) {
                        uint32_t w[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            __nv_bfloat162 p = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
                            w[i] = *reinterpret_cast<uint32_t*>(&p);
                        }
                        reinterpret_cast<uint4*>(dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
                        reinterpret_cast<uint4*>(dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            if (c0 + i < cols) dst[i] = __float2bfloat16_rn(v[i]);
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)BC) : "memory");
    }
}

template <int KIND, int BC>
static int grouped_launch(const CUtensorMap& ma, const CUtensorMap& mb0, const CUtensorMap& mb1, const GroupedArgs& a, int max_tiles,
                          cudaStream_t stream) {
    constexpr int COLS = KIND == MOE_GATEUP ? BC / 2 : BC;
    FF_SMEM_LIMIT((moe_grouped_tc_kernel<KIND, BC>), GroupedCfg<BC>::SMEM);
    dim3 grid((a.N + COLS - 1) / COLS, max_tiles);
    FF_LAUNCH((moe_grouped_tc_kernel<KIND, BC>), grid, GROUPED_THREADS, GroupedCfg<BC>::SMEM, stream, ma, mb0, mb1, a);
    FF_LAUNCH_CHECK();
    return 0;
}

// ------------------------------------------------------------------------------ pairs of SMs that stay --
// The same products where they fill the GPU: one pair of blocks (tcgen05 cta_group::2) per pair of SMs walks over tiles of 256
// rows of one expert x 256 matrix rows (8192 tokens, 4 of 16 experts of 512 x 1024: gate|up 120.7 -> 77.1 us with the gather, down 77.8 -> 47.9;
// the one-block kernel with its activation behind one branch 99.6).  What bounded the kernel above at these sizes: an SM's own 128 x 256 tile reads 96 bytes
// from L2 for every clock that its MMAs take, two stages of 48 KB are all that two blocks an SM have room for, a TMA gather of
// four rows keeps the copy engine for 60 clocks and more, twice what the MMAs of its rows take, and a thread's 16-byte stores of its own row
// reach the L2 as half sectors.  Here each block of a pair loads its 128 rows and half of the matrix rows (64 bytes a clock), six
// stages ahead, from rows that moe_gather_kernel has put side by side; two accumulators in tensor memory let a tile's epilogue run
// under the next tile's main loop; and a warp's 32 rows leave through shared memory, 128 bytes of each at a time, as TMA stores.
// (Rows picked by cp.async and a proxy fence for every stage took 1.2 us a stage where the MMAs take 0.3.)
constexpr int GP_EPI = 8;                                              // epilogue warps: two for every 32 rows, each half of the columns
constexpr int GP_THREADS = 64 + 32 * GP_EPI;
constexpr int GP_ROWS = 256, GP_BC = 256, GP_STAGES = 6, GP_STAGE_BYTES = 2 * GM * BK * 2, GP_BOX = 32 * 128, GP_STAGING = GP_EPI * GP_BOX;
constexpr size_t GP_SMEM = (size_t)GP_STAGES * GP_STAGE_BYTES + GP_STAGING + 1024 /* alignment slack */ + 256 /* barriers */;

// The tiles of 256 rows, expert after expert; every role of a block walks the list by itself.
struct GroupWalk {
    const int* seg;
    int E, e, base, lo, hi;
    __device__ __forceinline__ void begin(const int* s, int experts) { seg = s; E = experts; e = 0; base = 0; lo = s[0]; hi = s[1]; }
    __device__ __forceinline__ bool find(int m) {                      // m never decreases; false: behind the last tile
        for (;;) {
            const int n = (hi - lo + GP_ROWS - 1) / GP_ROWS;
            if (m < base + n) return true;
            base += n;
            if (++e >= E) return false;
            lo = hi;
            hi = seg[e + 1];
        }
    }
    __device__ __forceinline__ int row0(int m) const { return lo + (m - base) * GP_ROWS; }
};

__device__ __forceinline__ void gp_store_2d(const CUtensorMap* map, uint32_t src, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map), "r"(src), "r"(x), "r"(y) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void gp_arrive_leader(uint32_t bar) {
    uint32_t peer;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(peer) : "r"(bar));
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(peer) : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16(float x, float y) {
    __nv_bfloat162 p = __floats2bfloat162_rn(x, y);
    return *reinterpret_cast<uint32_t*>(&p);
}

template <int KIND>
__global__ void __launch_bounds__(GP_THREADS)
moe_grouped_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b0,
                        const __grid_constant__ CUtensorMap map_b1, const __grid_constant__ CUtensorMap map_out, const GroupedArgs a, const int E) {
    constexpr int COLS = KIND == MOE_GATEUP ? GP_BC / 2 : GP_BC;       // output columns of a tile
    constexpr int BOX_COLS = KIND == MOE_DOWN ? 32 : 64;               // of 128 bytes of an output row
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* staging = tiles + (size_t)GP_STAGES * GP_STAGE_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(staging + GP_STAGING);
    // [0..S) full (the first block's), [S..2S) empty, [2S..2S+2) accumulator ready, [2S+2..2S+4) accumulator free (the first block's)
    constexpr int FULL = 0, EMPTY = GP_STAGES, READY = 2 * GP_STAGES, FREE = READY + 2;
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const bool issue = lane == 0;
    const int half = blockIdx.x & 1;                                   // the cluster is (2, 1, 1)
    const int pairs = gridDim.x >> 1, NT = (a.N + COLS - 1) / COLS;
    const int n_iters = (a.K + BK - 1) / BK;

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int i = 0; i < FREE; ++i) mbar_init(smem_addr(&bars[i]), 1);
        for (int i = FREE; i < FREE + 2; ++i) mbar_init(smem_addr(&bars[i]), 2 * GP_EPI);  // the epilogue warps of both blocks
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_addr(&s_tmem_base)), "r"((uint32_t)(2 * GP_BC)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                                                // the other block's barriers are there
    tc_fence_after();
    const uint32_t tmem_base = s_tmem_base;
    volatile int* abort_flag = &s_abort;
    grid_launch_dependents();
    // the plan and the rows come from the kernels in front
    grid_dependency_wait();
    GroupWalk walk;
    walk.begin(pdl_fresh(a.seg), E);

    if (warp == 0) {
        // ------------------------------------------------ producer: TMA loads --
        const CUtensorMap* mb = KIND == MOE_GATEUP && half ? &map_b1 : &map_b0;
        int g = 0;                                                     // stages asked for
        bool ok = true;
        for (int i = blockIdx.x >> 1; ok; i += pairs) {
            const int m = i / NT, n0 = (i - m * NT) * COLS;
            if (!walk.find(m)) break;
            const int row0 = walk.row0(m) + half * GM;
            const int y = walk.e * a.N + n0 + (KIND == MOE_GATEUP ? 0 : half * GM);
            for (int it = 0; it < n_iters; ++it, ++g) {
                const int s = g % GP_STAGES;
                if (g >= GP_STAGES &&
                    !__all_sync(0xffffffffu, mbar_wait(smem_addr(&bars[EMPTY + s]), ((g / GP_STAGES) & 1) ^ 1, a.status, abort_flag, 111))) {
                    ok = false;
                    break;
                }
                const uint32_t full = smem_addr(&bars[FULL + s]), sa = smem_addr(tiles + (size_t)s * GP_STAGE_BYTES);
                if (half == 0) mbar_expect_tx(issue, full, 2 * GP_STAGE_BYTES);            // both blocks' bytes
                __syncwarp();
                tma_load_2d_pair(issue, sa, &map_a, it * BK, row0, full);
                tma_load_2d_pair(issue, sa + GM * BK * 2, mb, it * BK, y, full);
            }
        }
        // the last stages' releases, which come from the first block's MMAs, have arrived before this block goes
        for (int it = max(0, g - GP_STAGES); ok && it < g; ++it)
            ok = __all_sync(0xffffffffu, mbar_wait(smem_addr(&bars[EMPTY + it % GP_STAGES]), (it / GP_STAGES) & 1, a.status, abort_flag, 111));
        if (half == 0 && *abort_flag) {
            // let the copies that are still in flight land before the blocks' memory goes away
            const unsigned long long start = clock64();
            for (int it = max(0, g - GP_STAGES); it < g; ++it) {
                while (!mbar_try_wait(smem_addr(&bars[FULL + it % GP_STAGES]), (it / GP_STAGES) & 1))
                    if (clock64() - start > WAIT_LIMIT_CYCLES) break;
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------ MMA issuer: the first block's ----------
        if (half == 0) {
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(GP_BC >> 3) << 17) | ((uint32_t)(GP_ROWS >> 4) << 24);
            int g = 0, t = 0;
            bool ok = true;
            for (int i = blockIdx.x >> 1; ok; i += pairs, ++t) {
                if (!walk.find(i / NT)) break;
                const int buf = t & 1;
                if (t >= 2 && !__all_sync(0xffffffffu, mbar_wait(smem_addr(&bars[FREE + buf]), ((t >> 1) & 1) ^ 1, a.status, abort_flag, 112))) break;
                tc_fence_after();
                for (int it = 0; it < n_iters; ++it, ++g) {
                    const int s = g % GP_STAGES;
                    ok = __all_sync(0xffffffffu, mbar_wait(smem_addr(&bars[FULL + s]), (g / GP_STAGES) & 1, a.status, abort_flag, 112));
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t sa = smem_addr(tiles + (size_t)s * GP_STAGE_BYTES), sb = sa + GM * BK * 2;
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k)
                        tc_mma_bf16_pair(issue, tmem_base + buf * GP_BC, smem_desc_sw128(sa + k * UMMA_K * 2), smem_desc_sw128(sb + k * UMMA_K * 2), idesc,
                               (it > 0 || k > 0) ? 1u : 0u);
                    tc_commit_pair(issue, smem_addr(&bars[EMPTY + s]), 3);     // the stage is free in both blocks
                    __syncwarp();
                }
                if (ok) tc_commit_pair(issue, smem_addr(&bars[READY + buf]), 3);
            }
        }
    } else {
        // ------------------------------------------------ epilogue: one accumulator row a thread --
        const int quad = warp & 3, part = (warp - 2) >> 2;             // this warp's 32 lanes of tensor memory, and which half of the columns
        unsigned char* box = staging + (warp - 2) * GP_BOX;            // 32 rows x 128 bytes on their way out; the other warp's fills meanwhile
        const uint32_t lane_base = tmem_base + ((uint32_t)(quad * 32) << 16);
        // 16 bytes of this thread's row, where the 128-byte swizzle has them (eight rows' pieces lie in different banks)
        auto stage16 = [&](int chunk, uint4 v) {
            *reinterpret_cast<uint4*>(box + lane * 128 + ((chunk ^ (lane & 7)) << 4)) = v;
        };
        // the box has to be free: the store that took it last has read it
        auto box_free = [&]() {
            if (issue) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            __syncwarp();
        };
        // the warp's box goes to rows row0 .., columns c ..; where the expert ends among the rows (or a wait ran out) row by row
        auto leave = [&](int row0, int rows, int c) {
            if (rows >= 32) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (issue) gp_store_2d(&map_out, smem_addr(box), c, row0);
            } else {
                __syncwarp();
                const int w_row = lane >> 3, w_chunk = lane & 7, col = c + w_chunk * (BOX_COLS / 8);      // eight lanes a row's 128 bytes
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int r = j * 4 + w_row;
                    const uint4 v = *reinterpret_cast<const uint4*>(box + r * 128 + ((w_chunk ^ (r & 7)) << 4));
                    if (r < rows && col < a.N) {
                        const size_t at = (size_t)(row0 + r) * a.N + col;
                        if constexpr (KIND == MOE_DOWN) *reinterpret_cast<uint4*>((float*)a.out + at) = v;
                        else *reinterpret_cast<uint4*>((bf16*)a.out + at) = v;
                    }
                }
                __syncwarp();
            }
        };
        int t = 0;
        for (int i = blockIdx.x >> 1;; i += pairs, ++t) {
            const int m = i / NT, n0 = (i - m * NT) * COLS, buf = t & 1;
            if (!walk.find(m)) break;
            const int row0 = walk.row0(m) + half * GM + quad * 32;
            const int rows = walk.hi - row0;                           // of this warp: <= 0 where the expert ends in front of it
            const float wr = KIND != MOE_DOWN && a.row_w && lane < rows ? pdl_fresh(a.row_w)[row0 + lane] : 1.0f;
            if (!__all_sync(0xffffffffu, mbar_wait(smem_addr(&bars[READY + buf]), (t >> 1) & 1, a.status, abort_flag, 113))) break;
            tc_fence_after();
            const uint32_t acc = lane_base + buf * GP_BC;
            if (rows > 0) {
                const int cols = min(COLS, a.N - n0);
#pragma unroll 1
                for (int c0 = part * (COLS / 2); c0 < min(cols, (part + 1) * (COLS / 2)); c0 += BOX_COLS) {
                    if constexpr (KIND == MOE_DOWN) {
                        float v[32];
                        tc_ld32(acc + c0, v);
                        box_free();
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            stage16(j, make_uint4(__float_as_uint(v[4 * j]), __float_as_uint(v[4 * j + 1]), __float_as_uint(v[4 * j + 2]), __float_as_uint(v[4 * j + 3])));
                    } else {
                        box_free();
#pragma unroll
                        for (int c1 = 0; c1 < BOX_COLS; c1 += 32) {
                            float v[32];
                            tc_ld32(acc + c0 + c1, v);
                            if constexpr (KIND == MOE_GATEUP) {
                                float u[32];
                                tc_ld32(acc + GP_BC / 2 + c0 + c1, u);
                                // one branch for all: a branch a value would keep them from overlapping
                                if (a.act == 1) {
#pragma unroll
                                    for (int x = 0; x < 32; ++x) v[x] = clamped_glu_fast(v[x] * wr, u[x] * wr, a.limit, 1);
                                } else {
#pragma unroll
                                    for (int x = 0; x < 32; ++x) v[x] = clamped_glu_fast(v[x] * wr, u[x] * wr, a.limit, 0);
                                }
                            } else {
#pragma unroll
                                for (int x = 0; x < 32; ++x) v[x] = relu2(v[x] * wr);
                            }
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                stage16((c1 >> 3) + j, make_uint4(pack_bf16(v[8 * j], v[8 * j + 1]), pack_bf16(v[8 * j + 2], v[8 * j + 3]),
                                                                  pack_bf16(v[8 * j + 4], v[8 * j + 5]), pack_bf16(v[8 * j + 6], v[8 * j + 7])));
                        }
                    }
                    leave(row0, rows, n0 + c0);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (issue) gp_arrive_leader(smem_addr(&bars[FREE + buf]));
        }
        if (issue) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");       // the stores have left this block's memory and are there
    }
    // the pair's tensor memory is freed together, and its first block's barriers serve both
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)(2 * GP_BC)) : "memory");
    }
}

template <int KIND>
static int grouped_pair_launch(const CUtensorMap& ma, const CUtensorMap& mb0, const CUtensorMap& mb1, const CUtensorMap& mo, const GroupedArgs& a,
                               int E, int max_tiles, cudaStream_t stream) {
    constexpr int COLS = KIND == MOE_GATEUP ? GP_BC / 2 : GP_BC;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return (int)e;
    FF_SMEM_LIMIT(moe_grouped_pair_kernel<KIND>, GP_SMEM);
    const long long items = (long long)max_tiles * ((a.N + COLS - 1) / COLS);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (unsigned)(items < sms / 2 ? items : sms / 2));
    cfg.blockDim = dim3(GP_THREADS);
    cfg.dynamicSmemBytes = GP_SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim.x = 2;
    attrs[0].val.clusterDim.y = attrs[0].val.clusterDim.z = 1;
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = g_ff_pdl ? 2 : 1;
    return (int)cudaLaunchKernelEx(&cfg, moe_grouped_pair_kernel<KIND>, ma, mb0, mb1, mo, a, E);
}

// The tokens' rows in the order of the plan, a warp a row of `pieces` 16-byte pieces.
__global__ void __launch_bounds__(256) moe_gather_kernel(const uint4* x, const int* src_tok, const int* n_rows /* the plan's: seg[E] */, uint4* rows,
                                                         int room, int pieces) {
    pdl_prologue();
    const int r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (r >= min(room, *pdl_fresh(n_rows))) return;
    const uint4* from = pdl_fresh(x) + (size_t)pdl_fresh(src_tok)[r] * pieces;
    uint4* to = rows + (size_t)r * pieces;
    for (int i = lane; i < pieces; i += 128) {
        uint4 v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (i + 32 * j < pieces) v[j] = from[i + 32 * j];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (i + 32 * j < pieces) to[i + 32 * j] = v[j];
    }
}

}  // namespace ff

using namespace ff;

// a: bfloat16 [a_rows, K] (kind MOE_DOWN: the sorted rows themselves; else the tokens' rows, picked by src_tok).
// b0, b1: bfloat16 [E, N, K].  The plan's row tiles have 128 rows.  wide: 256 weight rows a block instead of 128.
// n_rows: of `out`, at least the plan's.  gathered (may be null): room for as many rows of K values; with it pairs of SMs multiply 256 rows with 256 weight rows at a time (N a
// multiple of 8; kind MOE_DOWN: any pointer but null, nothing is gathered).  launched: kernels put on the stream.
FF_EXPORT int ff_moe_grouped_tc(const void* a, int a_rows, const int* src_tok, const void* b0, const void* b1, int E, int kind,
                                const int* seg, const int* tile_expert, const int* tile_row0, const int* n_tiles,
                                const float* row_w, void* out, int max_tiles, int N, int K, float limit, int act, int wide,
                                void* gathered, int n_rows, int* status, int* launched, cudaStream_t stream) {
    *launched = 0;
    if (max_tiles <= 0) return 0;
    if (kind < MOE_DOWN || kind > MOE_UP || (kind == MOE_GATEUP && !b1) || !status || a_rows <= 0 || E <= 0 || N <= 0 || K <= 0 || K % 8)
        return FF_ERR_BAD_ARG;
    if ((((uintptr_t)a | (uintptr_t)b0 | (uintptr_t)b1 | (uintptr_t)out | (uintptr_t)gathered) & 15) != 0 || (long long)E * N >= (1ll << 31) || max_tiles > 65535)
        return FF_ERR_BAD_ARG;
    if (gathered && (N % 8 || n_rows <= 0)) return FF_ERR_BAD_ARG;
    const bool down = kind == MOE_DOWN;
    if (gathered && !down) {
        FF_LAUNCH(moe_gather_kernel, (n_rows + 7) / 8, 256, 0, stream, (const uint4*)a, src_tok, seg + E, (uint4*)gathered, n_rows, K / 8);
        FF_LAUNCH_CHECK();
        ++*launched;
        a = gathered;
        a_rows = n_rows;
    }
    const int bc = wide ? 256 : 128, box = gathered ? GM : kind == MOE_GATEUP ? bc / 2 : bc;
    CUtensorMap ma, mb0, mb1, mo;
    int rc = make_map(a, a_rows, K, down || gathered ? GM : 1, &ma);       // a gather's box is one row high
    if (rc) return rc;
    rc = make_map(b0, E * N, K, box, &mb0);
    if (rc) return rc;
    mb1 = mb0;
    if (kind == MOE_GATEUP && (rc = make_map(b1, E * N, K, box, &mb1))) return rc;
    if (gathered && (rc = make_map(out, n_rows, N, 32, &mo, down ? 4 : 2))) return rc;
    GroupedArgs g{src_tok, seg, tile_expert, tile_row0, n_tiles, row_w, out, N, K, limit, act, status};
    ++*launched;
#define FF_GROUPED(KIND) return gathered ? grouped_pair_launch<KIND>(ma, mb0, mb1, mo, g, E, max_tiles, stream) \
                              : wide ? grouped_launch<KIND, 256>(ma, mb0, mb1, g, max_tiles, stream) \
                                     : grouped_launch<KIND, 128>(ma, mb0, mb1, g, max_tiles, stream)
    if (kind == MOE_GATEUP) FF_GROUPED(MOE_GATEUP);
    if (kind == MOE_UP) FF_GROUPED(MOE_UP);
    FF_GROUPED(MOE_DOWN);
#undef FF_GROUPED
}
