// Matmul for middling and large row counts (large decode batches, prompts; matmul.cu has the rule):
// out_j[rows, N_j] = act(a[rows, K] x W_j[K, N_j] + bias_j), bfloat16, for up to four weights W_j that share the activation, in packed
// bfloat8_b / bfloat4_b tiles; rows, K and N multiples of 32.
//
// "Swap-AB", as in the decode kernels: the MMA's M dimension (128 TMEM lanes) runs over weight columns, its N dimension over up
// to 256 activation rows, and a block owns 128 columns x one chunk of rows, so that a weight is expanded once per chunk (the
// decode kernel does it for every 32 or 64 rows and fetches the activations in tensor-map boxes 32 bytes wide). A packed tile
// crosses shared memory once and the expanded weights go registers -> tensor memory -> MMA (expand_tmem.cuh).
//   * warps 0..7 expand, two teams of four (a warp can only touch the 32 TMEM lanes of its quadrant), each taking two of the four
//     K blocks of a group;
//   * warps 8..15 run the epilogue;
//   * warp 16 streams the packed tiles with one tensor-map copy per group, warps 17..20 copy the activations (16-byte cp.async
//     straight into the MMA's 32-byte-swizzled K-major layout; no re-layout pass), warp 21 issues the MMAs.
// Two rings: packed tiles in shared memory; activations there and expanded weights in the tensor memory that the fp32
// accumulator of up to 128 x 256 leaves, group by group under one pair of barriers.
// Blocks walk their tiles persistently. Where tiles are few, clusters of up to 8 blocks share a tile's K range and add their
// partial sums out of each other's shared memory, in block order: no scratch, the same bits every time. The tiles left after the
// last whole round go to a second launch in that form.
//
// What bounds it, from builds with parts left out, ns per K block of a block that owns its tile (148 tiles, 64 / 128 / 192 / 256 rows):
// everything 163 / 172 / 193 / 258 (bfloat4_b 160 / 172 / 190 / 281); the parts alone: weight copies 145 (bfloat4_b 48), expansion 117
// to 145, activation copies 112 to 146, MMAs 66 / 75 / 111 / 144, bare barriers 45 to 52. With two (256 rows) or three groups in flight
// they overlap only in part; no pipe is busy for more than half the time (tensor pipe 51 % at 256 rows). Groups of one or two K
// blocks were slower. Before, as one to three launches of the decode and prefill kernels, and now, microseconds a launch from a
// graph: 128 x 4096 x 14336 bfloat4_b 46.2 / 26.2, 352 x 4544 x 4672 48.2 / 21.0, 512 x 4096 x 4096 74.8 / 21.9, 512 x 1024 x 1024
// 25.8 / 8.6, 256 x 8192 x 8192 71.6 / 39.8, 64 x 4096 x 1024 14.2 / 8.0, 1536 x 4096 x 14336 210 / 159.
// Every mbarrier wait is bounded; a wait that runs out raises a status word instead of hanging. No such wait begins while it
// depends on the previous kernel (which may itself wait for other GPUs for seconds): the role waits for that kernel first.
#include "decode_common.cuh"
#include "expand_tmem.cuh"

namespace ttb {
unsigned barrier_limit_kcycles();
namespace {

using namespace ptx;

constexpr int BN = 128;      // weight columns per tile (MMA M, TMEM lanes)
constexpr int BK = 32;       // K per stage: one row of four packed tiles
constexpr int kGroup = 4;    // stages per barrier round trip
constexpr int kTeams = 2, kExpandWarps = 4 * kTeams, kEpiWarps = 8, kLoaderWarps = 4;
constexpr int kEpiWarp0 = kExpandWarps, kProducerWarp = kEpiWarp0 + kEpiWarps, kLoaderWarp0 = kProducerWarp + 1, kMmaWarp = kLoaderWarp0 + kLoaderWarps;
constexpr int kThreads = 32 * (kMmaWarp + 1);
constexpr int kAColsPerStage = BK / 2;               // TMEM columns of one expanded stage
constexpr uint32_t kX_SBO = 256;
constexpr int kStageRows = 32;                       // rows of a finished tile that pass through shared memory together

// BR: activation rows per chunk at most (MMA N), 192 or 256.
template <int FMT, int BR>
struct Layout {
    static constexpr int kRing = BR == 192 ? 3 : 2;      // groups in flight: activations in shared and expanded weights in tensor memory
    static constexpr int kXStageBytes = BR * BK * 2;     // activations of a K block: two 16-column halves of BR 32-byte rows
    static constexpr int kACol0 = BR;                    // the accumulator takes the first BR columns of tensor memory
    static_assert(BR + kRing * kGroup * kAColsPerStage <= 512, "tensor memory budget");
    static constexpr int kTile = FMT == TTB_BFLOAT8_B ? kBfp8TileBytes : kBfp4TileBytes;
    static constexpr int kPStageBytes = 4 * kTile;
    static constexpr int kPRing = FMT == TTB_BFLOAT8_B ? 3 : 6;   // groups of packed tiles
    static constexpr int x = 0;
    static constexpr int out = x + kRing * kGroup * kXStageBytes;    // [kStageRows][BN] fp32
    static constexpr int pk = out + kStageRows * BN * 4;
    static constexpr int bars = pk + kPRing * kGroup * kPStageBytes;
    // full, empty [kRing]; full_p, empty_p [kPRing]; acc_full, acc_empty
    static constexpr int nbars = 2 * kRing + 2 * kPRing + 2;
    static constexpr int misc = bars + 8 * nbars;
    static constexpr int total = misc + 16 + 1024;
    static_assert(total <= 232448, "shared memory budget");
    static_assert(kGroup * kPStageBytes % 128 == 0, "tensor-map copies land on 128-byte boundaries");
    static_assert(kRing * kGroup * kXStageBytes >= BR * BN * 4, "the partial sums of a shared tile take the activations' place");
};

struct alignas(64) Args {
    // up to four weights that share the activation; their column tiles form one list, weight j's from tstart[j]
    CUtensorMap wmap[TTB_MAX_GROUP];   // packed weights as [K blocks][tiles per row][tile as 8-byte words], box of kGroup x 4 tiles
    const uint16_t *bias[TTB_MAX_GROUP];
    void *out[TTB_MAX_GROUP];
    int64_t N[TTB_MAX_GROUP];
    int weights, tstart[TTB_MAX_GROUP + 1];
    const uint16_t *a;
    int64_t rows, K;
    int Kt;                 // K blocks
    int chunks, chunk_rows; // row chunks and rows of each (the last may have fewer)
    int tile0, tiles;       // this launch's tiles: tile0 .. tile0 + tiles - 1; row chunks vary fastest
    int split;              // blocks (= cluster size) that share a tile's K range
    int act, a_row_major, out_row_major;
    unsigned wait_limit;   // of every barrier wait, in 1024 SM clocks
    int *status;
};

__device__ __forceinline__ long long wait_clocks(const Args &p) { return (long long)p.wait_limit << 10; }

// Four neighbouring columns n .. n + 3 of one row: bias, activation, store.
template <int ACT>
__device__ __forceinline__ void finish4(const Args &p, int w, int64_t row, int64_t n, float4 v, float4 b) {
    v.x = apply_activation_t<ACT>(v.x + b.x); v.y = apply_activation_t<ACT>(v.y + b.y);
    v.z = apply_activation_t<ACT>(v.z + b.z); v.w = apply_activation_t<ACT>(v.w + b.w);
    const int64_t off = p.out_row_major ? row * p.N[w] + n : tiled_offset(row, n, p.N[w] >> 5);
    *reinterpret_cast<uint2 *>(reinterpret_cast<uint16_t *>(p.out[w]) + off) =
        make_uint2((uint32_t)f32_to_bf16_bits(v.x) | ((uint32_t)f32_to_bf16_bits(v.y) << 16),
                   (uint32_t)f32_to_bf16_bits(v.z) | ((uint32_t)f32_to_bf16_bits(v.w) << 16));
}
__device__ __forceinline__ float4 bias4(const Args &p, int w, int64_t n) {
    if (!p.bias[w] || n >= p.N[w]) return make_float4(0.f, 0.f, 0.f, 0.f);
    return make_float4(bias_at(p.bias[w], n), bias_at(p.bias[w], n + 1), bias_at(p.bias[w], n + 2), bias_at(p.bias[w], n + 3));
}
// Rows r0, r0 + step, ... < r1 of a [rows][BN] fp32 slab in shared memory: a warp's lanes take four columns each.
template <int ACT>
__device__ __forceinline__ void finish_rows(const Args &p, int w, uint32_t slab, int r0, int r1, int step, int64_t row_base, int64_t n, int blocks, const float4 b) {
    if (n >= p.N[w]) return;
    for (int r = r0; r < r1; r += step) {
        const uint32_t at = slab + (uint32_t)(r * BN * 4) + (uint32_t)((threadIdx.x & 31) * 16);
        float4 v;
        if (blocks == 1) {
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
        } else {
            v = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int c = 0; c < blocks; ++c) {
                const float4 x = ld_cluster_f32x4(at, (uint32_t)c);
                v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
            }
        }
        finish4<ACT>(p, w, row_base + r, n, v, b);
    }
}

// A bounded wait whose barrier may depend on the previous kernel: that one's time is not to count. (What is free at once is free
// without it; the wait for it returns at once ever after.)
__device__ __forceinline__ bool mbar_wait_behind(uint32_t bar, uint32_t parity, volatile int *abort_flag, int *status, int code, long long limit) {
    if (mbar_try_wait(bar, parity)) return true;
    grid_dep_wait();
    return mbar_wait(bar, parity, abort_flag, status, code, limit);
}

template <int FMT, int BR>
__global__ void __launch_bounds__(kThreads, 1) matmul_rows_kernel(const __grid_constant__ Args p) {
    using L = Layout<FMT, BR>;
    constexpr int kPRing = L::kPRing, kRing = L::kRing, kXStageBytes = L::kXStageBytes, kACol0 = L::kACol0;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t sbase = smem_u32(smem);
    const uint32_t bar0 = sbase + L::bars;
    auto full = [&](int s) { return bar0 + 8u * s; };                  // the group's activations have landed and its weights are expanded
    auto empty = [&](int s) { return bar0 + 8u * (kRing + s); };       // its MMAs are complete
    auto full_p = [&](int s) { return bar0 + 8u * (2 * kRing + s); };
    auto empty_p = [&](int s) { return bar0 + 8u * (2 * kRing + kPRing + s); };
    const uint32_t acc_full = bar0 + 8u * (2 * kRing + 2 * kPRing), acc_empty = acc_full + 8u;
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(smem + L::misc);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + L::misc + 4);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kRing; ++s) {
            mbar_init(full(s), 32 * kLoaderWarps + kExpandWarps);   // every loader lane, once its copies have landed; every expand warp
            mbar_init(empty(s), 1);                                 // the commit of the MMAs that read the group
        }
        for (int s = 0; s < kPRing; ++s) {
            mbar_init(full_p(s), 1);                   // the producer, with its byte count
            mbar_init(empty_p(s), kExpandWarps);
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, kEpiWarps);
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == kMmaWarp) {
        tmem_alloc(sbase + L::misc, 512);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    // The next kernel on the stream may start while this grid drains; before grid_dep_wait() a role reads packed weights only.
    grid_dep_launch();

    // this block's K blocks of every tile it works on
    const int rank = p.split > 1 ? (int)cluster_rank() : 0;
    const int kb0 = (int)((int64_t)p.Kt * rank / p.split), kb1 = (int)((int64_t)p.Kt * (rank + 1) / p.split);
    const int first = (int)blockIdx.x / p.split, step = (int)gridDim.x / p.split;
    auto chunk_of = [&](int t) { return (p.tile0 + t) % p.chunks; };
    auto column_tile_of = [&](int t, int &w) {   // the weight, and the column tile inside it
        const int c = (p.tile0 + t) / p.chunks;
        w = 0;
#pragma unroll
        for (int j = 1; j < TTB_MAX_GROUP; ++j)
            if (j < p.weights && c >= p.tstart[j]) w = j;
        return c - p.tstart[w];
    };
    auto rows_of = [&](int chunk) { return (int)min((int64_t)p.chunk_rows, p.rows - (int64_t)chunk * p.chunk_rows); };

    if (warp < kExpandWarps) {
        // ---------------- expand warps: packed codes -> bf16 in tensor memory ----------------
        const int team = warp >> 2, quad = warp & 3;
        const uint32_t ld_off = expand_ld_offset<FMT>(lane);
        const int sh0 = 2 * (lane & 3);
        const uint32_t pk_quad = sbase + L::pk + quad * L::kTile;
        const uint32_t a_quad = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)kACol0;
        int gs = 0, ps = 0;
        uint32_t ph = 0, pph = 0;
        bool ok = true;
        for (int t = first; ok && t < p.tiles; t += step) {
            for (int kb = kb0; kb < kb1; kb += kGroup) {
                if (!__all_sync(0xffffffffu, mbar_wait(full_p(ps), pph, abort_flag, p.status, 51, wait_clocks(p)) && mbar_wait_behind(empty(gs), ph ^ 1u, abort_flag, p.status, 52, wait_clocks(p)))) {
                    ok = false;
                    break;
                }
                const int count = min(kGroup / kTeams, kb1 - kb - team * (kGroup / kTeams));
                if (count > 0) {
                    const int j = team * (kGroup / kTeams);
                    tc_fence_after_sync();
                    expand_tiles<FMT>(pk_quad + (uint32_t)((ps * kGroup + j) * L::kPStageBytes), L::kPStageBytes,
                                            a_quad + (uint32_t)((gs * kGroup + j) * kAColsPerStage), kAColsPerStage, count, ld_off, sh0, lane);
                    tmem_st_wait();
                    tc_fence_before_sync();
                }
                __syncwarp();
                if (lane == 0) {   // (also for K blocks that a short last group lacks)
                    mbar_arrive(full(gs));
                    mbar_arrive(empty_p(ps));
                }
                if (++gs == kRing) { gs = 0; ph ^= 1u; }
                if (++ps == kPRing) { ps = 0; pph ^= 1u; }
            }
        }
    } else if (warp == kProducerWarp) {
        // ---------------- packed weight tiles -> shared memory ----------------
        const bool leader = elect_one();
        int s = 0, ahead = kPRing + kRing;
        uint32_t ph = 0;
        bool ok = true;
        for (int t = first; ok && t < p.tiles; t += step) {
            int w;
            const int nt = column_tile_of(t, w);
            for (int kb = kb0; kb < kb1; kb += kGroup) {
                if (ahead-- == 0) grid_dep_wait();   // (the expand warps have emptied kRing groups by then; the next one follows an MMA)
                if (!__all_sync(0xffffffffu, mbar_wait(empty_p(s), ph ^ 1u, abort_flag, p.status, 53, wait_clocks(p)))) { ok = false; break; }
                if (leader) {
                    // (always a whole box: what lies beyond the weight reads as zeros, a surplus K block is not expanded)
                    mbar_arrive_expect_tx(full_p(s), kGroup * L::kPStageBytes);
                    tma_load_3d_plain(sbase + L::pk + s * kGroup * L::kPStageBytes, &p.wmap[w], 0, nt * 4, kb, full_p(s));
                }
                if (++s == kPRing) { s = 0; ph ^= 1u; }
            }
        }
    } else if (warp >= kLoaderWarp0 && warp < kLoaderWarp0 + kLoaderWarps) {
        // ---------------- activations -> shared memory: a 16x16 face per warp instruction ----------------
        grid_dep_wait();
        const int lw = warp - kLoaderWarp0;
        const uint32_t face_dst = face_chunk_sw32(lane);
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int t = first; ok && t < p.tiles; t += step) {
            const int chunk = chunk_of(t), ntr = rows_of(chunk) / 32;
            // this lane's chunk of the first face of tile row lw, and the distances to the lower and right faces and to the next K
            // block and tile row
            const uint16_t *src;
            int64_t down, right, next_k, next_row;
            if (p.a_row_major) {
                src = p.a + ((int64_t)chunk * p.chunk_rows + lw * 32 + (lane >> 1)) * p.K + (int64_t)kb0 * BK + (lane & 1) * 8;
                down = 16 * p.K; right = 16; next_k = BK; next_row = kLoaderWarps * 32 * p.K;
            } else {
                src = p.a + ((int64_t)(chunk * (p.chunk_rows / 32) + lw) * p.Kt + kb0) * 1024 + lane * 8;
                down = 512; right = 256; next_k = 1024; next_row = (int64_t)kLoaderWarps * p.Kt * 1024;
            }
            for (int kb = kb0; kb < kb1; kb += kGroup) {
                if (!__all_sync(0xffffffffu, mbar_wait(empty(s), ph ^ 1u, abort_flag, p.status, 54, wait_clocks(p)))) { ok = false; break; }
                uint32_t d0 = sbase + L::x + s * kGroup * kXStageBytes + lw * 1024 + face_dst;
                for (int j = 0; j < min(kGroup, kb1 - kb); ++j, src += next_k, d0 += kXStageBytes) {
                    const uint16_t *f = src;
                    uint32_t d = d0;
#pragma unroll 4
                    for (int tr = lw; tr < ntr; tr += kLoaderWarps, f += next_row, d += kLoaderWarps * 1024) {
                        cp_async16(d, f);
                        cp_async16(d + 512, f + down);
                        cp_async16((d + kXStageBytes / 2) ^ expand_b_swap<FMT>, f + right);
                        cp_async16((d + kXStageBytes / 2 + 512) ^ expand_b_swap<FMT>, f + down + right);
                    }
                }
                cp_async_arrive(full(s));
                if (++s == kRing) { s = 0; ph ^= 1u; }
            }
        }
        cp_async_wait_all();   // nothing of this warp's is in flight at the teardown
    } else if (warp == kMmaWarp) {
        // ---------------- MMA issuer: A (weights) from tensor memory, B (activations) from shared memory ----------------
        grid_dep_wait();   // (the activations come after it: no bounded wait is to count the previous kernel's time)
        const bool leader = elect_one();
        const uint64_t x_desc0 = smem_desc_sw32(sbase + L::x, kX_SBO);
        const uint32_t x_lo0 = (uint32_t)x_desc0, x_hi = (uint32_t)(x_desc0 >> 32);
        auto mk = [](uint32_t lo, uint32_t hi) { return ((uint64_t)hi << 32) | lo; };
        int gs = 0, n = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int t = first; ok && t < p.tiles; t += step, ++n) {
            if (!__all_sync(0xffffffffu, mbar_wait(acc_empty, (uint32_t)((n & 1) ^ 1), abort_flag, p.status, 55, wait_clocks(p)))) { ok = false; break; }
            tc_fence_after_sync();
            const uint32_t idesc = instr_desc_bf16_f32(BN, 0, /*a_mn_major=*/false, /*b_mn_major=*/false) | ((uint32_t)(rows_of(chunk_of(t)) >> 3) << 17);
            for (int kb = kb0; kb < kb1; kb += kGroup) {
                if (!__all_sync(0xffffffffu, mbar_wait(full(gs), ph, abort_flag, p.status, 56, wait_clocks(p)))) { ok = false; break; }
                fence_proxy_async_smem();   // the activations came through the generic proxy
                tc_fence_after_sync();
                const uint32_t a_col = tmem_base + (uint32_t)(kACol0 + gs * kGroup * kAColsPerStage);
                const uint32_t x_lo = x_lo0 + (uint32_t)((gs * kGroup * kXStageBytes) >> 4);
                auto issue = [&](int j) {
                    mma_bf16_ts(tmem_base, a_col + (uint32_t)(j * kAColsPerStage), mk(x_lo + (uint32_t)((j * kXStageBytes) >> 4), x_hi), idesc, kb > kb0 || j > 0);
                    mma_bf16_ts(tmem_base, a_col + (uint32_t)(j * kAColsPerStage + 8), mk(x_lo + (uint32_t)((j * kXStageBytes + kXStageBytes / 2) >> 4), x_hi), idesc, true);
                };
                if (leader) {
                    if (kb + kGroup <= kb1) {   // straight line: a branch between two MMAs costs more than issuing one
#pragma unroll
                        for (int j = 0; j < kGroup; ++j) issue(j);
                    } else {
                        for (int j = 0; j < kb1 - kb; ++j) issue(j);
                    }
                    mma_commit(empty(gs));
                }
                if (++gs == kRing) { gs = 0; ph ^= 1u; }
            }
            if (ok && leader) mma_commit(acc_full);
        }
    } else {
        // ---------------- epilogue warps: TMEM lanes 32 * (warp % 4) .., alternate groups of 16 rows ----------------
        grid_dep_wait();
        const int ew = warp - kEpiWarp0, quad = warp & 3, half = ew >> 2;
        const int col = quad * 32 + expand_column_of_lane<FMT>(lane);   // the weight column this thread's TMEM lane holds
        const uint32_t t_lane = tmem_base + ((uint32_t)(quad * 32) << 16);
        const uint32_t slab = sbase + (p.split > 1 ? L::x : L::out);
        int n = 0;
        bool ok = true;
        for (int t = first; ok && t < p.tiles; t += step, ++n) {
            const int chunk = chunk_of(t), nrows = rows_of(chunk);
            int w;
            const int64_t row_base = (int64_t)chunk * p.chunk_rows, col0 = (int64_t)column_tile_of(t, w) * BN + lane * 4;
            // (the eight warps meet at named barriers below: they go on together or not at all)
            int good = mbar_wait(acc_full, (uint32_t)(n & 1), abort_flag, p.status, 57, wait_clocks(p)) ? 1 : 0;
            asm volatile(
                "{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %0, 0;\n\tbarrier.cta.red.and.pred q, 1, %1, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
                : "+r"(good)
                : "n"(32 * kEpiWarps)
                : "memory");
            if (!good) { ok = false; break; }
            tc_fence_after_sync();
            const float4 b = bias4(p, w, col0);
            for (int r0 = 0; r0 < nrows; r0 += kStageRows) {
                uint32_t v[16];
                tmem_ld16(t_lane + (uint32_t)(r0 + half * 16), v);
                tmem_ld_wait();
                const uint32_t at = slab + (uint32_t)((((p.split > 1 ? r0 : 0) + half * 16) * BN + col) * 4);
#pragma unroll
                for (int j = 0; j < 16; ++j) asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + (uint32_t)(j * BN * 4)), "r"(v[j]) : "memory");
                if (r0 + kStageRows >= nrows) {
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(acc_empty);   // the next tile's MMAs may overwrite the accumulator
                }
                if (p.split == 1) {
                    asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpiWarps) : "memory");
                    TTB_DISPATCH_ACT(p.act, finish_rows<ACT>(p, w, slab, ew, kStageRows, kEpiWarps, row_base + r0, col0, 1, b));
                    asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpiWarps) : "memory");
                }
            }
        }
    }

    if (p.split > 1) {
        // one tile per cluster: the blocks add each other's partial sums in block order, each for its share of the rows
        __syncwarp();
        cluster_sync();
        if (*abort_flag == 0) {
            const int chunk = chunk_of(first), nrows = rows_of(chunk);
            int w;
            const int64_t col0 = (int64_t)column_tile_of(first, w) * BN + lane * 4;
            const float4 b = bias4(p, w, col0);
            TTB_DISPATCH_ACT(p.act, finish_rows<ACT>(p, w, sbase + L::x, nrows * rank / p.split + warp, nrows * (rank + 1) / p.split, kThreads / 32,
                                                     (int64_t)chunk * p.chunk_rows, col0, p.split, b));
        }
        __syncwarp();
        cluster_sync();   // nobody leaves while another block may still read its shared memory
    }

    // ---------------- teardown ----------------
    tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag) {
        // A wait ran out: give copies and MMAs still in flight a bounded time to land before the block's shared memory and
        // tensor memory are released.
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == kMmaWarp) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 512);
    }
}

struct Device {
    Once once;
    int sms, clusters[9];    // multiprocessors; clusters of 2..8 blocks that run at the same time
};

template <int FMT, int BR>
int32_t configure(Device &d, int dev) {
    constexpr int smem = Layout<FMT, BR>::total;
    TTB_CUDA_TRY(cudaFuncSetAttribute(matmul_rows_kernel<FMT, BR>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    int sms = 0;
    TTB_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    for (int c = 2; c <= 8; ++c) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(sms / c * c));
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)c;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        TTB_CUDA_TRY(cudaOccupancyMaxActiveClusters(&n, matmul_rows_kernel<FMT, BR>, &cfg));
        d.clusters[c] = n;
    }
    d.sms = sms;
    return TTB_OK;
}

template <int FMT, int BR>
int32_t launch_tiles(Args &p, int tile0, int tiles, int split, int sms, bool overlap, cudaStream_t stream) {
    p.tile0 = tile0; p.tiles = tiles; p.split = split;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(split > 1 ? tiles * split : tiles < sms ? tiles : sms));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = Layout<FMT, BR>::total;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (overlap) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (split > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = (unsigned)split;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    TTB_CUDA_TRY(cudaLaunchKernelEx(&cfg, matmul_rows_kernel<FMT, BR>, p));
    TTB_LAUNCH_CHECK("matmul_rows");
    return TTB_OK;
}

// All tiles: whole rounds by one block per tile, what is left over (or all, where tiles are few) by clusters that share tiles.
template <int FMT, int BR>
int32_t launch_all(Args &p, int tiles, int split, int sms, bool overlap, cudaStream_t stream) {
    const int whole = tiles / sms * sms, rest = tiles - whole;
    if (whole == 0) return launch_tiles<FMT, BR>(p, 0, tiles, split, sms, overlap, stream);
    if (rest == 0 || split == 1) return launch_tiles<FMT, BR>(p, 0, tiles, 1, sms, overlap, stream);
    if (int32_t rc = launch_tiles<FMT, BR>(p, 0, whole, 1, sms, overlap, stream)) return rc;
    return launch_tiles<FMT, BR>(p, whole, rest, split, sms, overlap, stream);
}

template <int FMT>
int32_t launch_fmt(Args &p, bool overlap, cudaStream_t stream) {
    static Device devices[64];
    int dev = 0;
    TTB_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(TTB_E_UNSUPPORTED, "ttb_matmul: device index %d is out of range", dev);
    Device &d = devices[dev];
    if (int32_t rc = d.once.run([&] {
            const int32_t c = configure<FMT, 192>(d, dev);
            return c ? c : configure<FMT, 256>(d, dev);
        }))
        return rc;
    // Blocks that share a tile: as many as run at the same time, each with at least eight K blocks (the exchange of the partial
    // sums costs about that much).
    auto split_for = [&](int n) {
        int c = 8;
        while (c > 1 && (n > d.clusters[c] || p.Kt < 8 * c)) --c;
        return c;
    };
    // Row chunks: as few as possible, or up to twice as many where that fills the last round of blocks better. A K block takes
    // about 125 ns + 0.48 ns per row of the chunk, the exchange of partial sums 1 us + 16 ns per row, a further launch 1 us (fitted
    // to timings of 64 to 256 rows: 256 x 2048 x 2048 as one chunk 13.0 us, as two 10.8; 512 x 4096 x 4096 as two 24.0, as four 27.7).
    const int tile_rows = (int)(p.rows / 32), least = (tile_rows + 7) / 8, nt = p.tstart[p.weights];
    double best = 1e30;
    int split = 1;
    for (int c = least; c <= 2 * least && c <= tile_rows; ++c) {
        const int per = (tile_rows + c - 1) / c, chunks = (tile_rows + per - 1) / per;
        const int64_t t = (int64_t)chunks * nt, rest = t % d.sms;
        const int s = rest ? split_for((int)rest) : 1;
        const double kb = 125.0 + 0.48 * 32 * per;
        const double exchange = s > 1 ? 1000.0 + 16.0 * 32 * per : 0.0;
        const double cost = (double)(t / d.sms) * p.Kt * kb + (rest ? (p.Kt + s - 1) / s * kb + exchange + (s > 1 && t > d.sms ? 1000.0 : 0.0) : 0.0);
        if (cost < best) {
            best = cost;
            split = s;
            p.chunks = chunks;
            p.chunk_rows = per * 32;
        }
    }
    const int tiles = p.chunks * nt;
    // (192 rows leave room for a third group in flight)
    return p.chunk_rows <= 192 ? launch_all<FMT, 192>(p, tiles, split, d.sms, overlap, stream) : launch_all<FMT, 256>(p, tiles, split, d.sms, overlap, stream);
}
}  // namespace

// `count` matmuls with bfloat16 results that share the activation, in one or two launches, whatever the row and column counts.
int32_t launch_matmul_rows(const void *a, int count, const void *const *w, int w_dtype, const void *const *bias, void *const *out, int64_t rows,
                           int64_t K, const int64_t *N, int act, int flags, int *status, cudaStream_t stream) {
    Args p = {};
    p.a = (const uint16_t *)a;
    p.rows = rows; p.K = K; p.Kt = (int)(K / BK);
    p.act = act;
    p.a_row_major = (flags & TTB_MM_A_ROW_MAJOR) != 0;
    p.out_row_major = (flags & TTB_MM_OUT_ROW_MAJOR) != 0;
    p.status = status;
    p.wait_limit = barrier_limit_kcycles();
    p.weights = count;
    int64_t tiles = 0;
    for (int j = 0; j < count; ++j) {
        p.bias[j] = (const uint16_t *)(bias ? bias[j] : nullptr);
        p.out[j] = out[j];
        p.N[j] = N[j];
        p.tstart[j] = (int)tiles;
        tiles += (N[j] + BN - 1) / BN;
        if (rows / 32 * tiles > INT32_MAX / 8) return fail(TTB_E_UNSUPPORTED, "ttb_matmul: too many output tiles");
        if (int32_t rc = make_weight_map((const uint8_t *)w[j], K, N[j], w_dtype, kGroup, p.wmap[j])) return rc;
    }
    p.tstart[count] = (int)tiles;
    const bool overlap = (flags & TTB_MM_WEIGHTS_RESIDENT) != 0;
    return w_dtype == TTB_BFLOAT8_B ? launch_fmt<TTB_BFLOAT8_B>(p, overlap, stream) : launch_fmt<TTB_BFLOAT4_B>(p, overlap, stream);
}

}  // namespace ttb
