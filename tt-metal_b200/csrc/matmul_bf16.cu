// Matmul with bfloat16 weights on the tensor cores: out[b, rows, N] = act(a[b, rows, K] x W[b, K, N] + bias), b = 1 for a
// weight shared by every row (linear) or one [K, N] matrix per batch entry (attention scores and the like). All sizes are
// multiples of 32.
//
// One persistent block per SM works through [128 rows] x [128 columns] output tiles, walking K in stages of 64:
//   * four producer warps move the operands with 16-byte cp.async. A 16x16 face (512 contiguous bytes of a tiled tensor, 16
//     rows of 32 bytes) is one warp instruction and stays one 512-byte piece in shared memory: rows of 32 bytes in which the
//     halves of rows 4..7 of every eight change places are the MMA's 32-byte-swizzled operand layout, K-major for the
//     activation and N-major for the weight. Whole lines from memory, no bank conflicts, no re-layout pass. (A tensor map
//     delivers the same layout, but in boxes 32 bytes wide, at 10 to 13 bytes per clock and SM; lanes that take the 16-byte
//     halves of a row apart, for the layout without swizzle, got 12.)
//   * one warp issues tcgen05.mma (128 x 128 x 16);
//   * eight warps keep the tile's sums in registers: every `chunk` stages the MMAs change over to the other of two tensor
//     memory accumulators and these warps add the finished one to their fp32 sums, rounding to nearest. The tensor cores cut
//     off what an addition shifts out, an error that grows with the number of additions in a row. fp32 results change over
//     every stage and come out closer to 64 bits than a chain of fp32 fused multiply-adds (2-norm at K = 512 / 2048 / 28672:
//     8.2e-8 / 1.0e-7 / 2.8e-7 against 1.6e-7 / 3.9e-7 / 2.1e-6); for bfloat16 results every fourth stage is enough (2.3e-7 to
//     2.7e-7 before their rounding of 1.7e-3) and takes 5 to 20 % less time.
//     Finished sums leave while the next tile's MMAs run.
// Few tiles (less than half a wave): clusters of 2, 4 or 8 blocks share a tile's K range and add their partial sums out of
// each other's shared memory, in block order, each finishing its share of the columns - no scratch, no zeroing, same bits
// every time.
//
// What bounds it: small calls, the fixed 5 us of a launch that loads, multiplies and stores one stage. Large ones, the copies: a
// stage of 32 KB takes 399 ns (tensor pipe 34 % busy), 361 without its MMAs, 273 without its copies, 146 by the MMAs alone; with fp32
// results 482, of which the accumulator that changes over every stage takes 447. Before (CUDA cores, 32 x 32 tiles) a ttnn call
// on 1024 x 1024 x 1024 took 120.9 us and one on 32 x [512 x 128 x 512] 118.8 us; now 9.4 and 9.9 us.
// Every mbarrier wait is bounded; a wait that runs out raises a status word instead of hanging.
#include "epilogue.cuh"
#include "sm100_ptx.cuh"

namespace ttb {
unsigned barrier_limit_kcycles();
namespace {

using namespace ptx;

constexpr int BM = 128, BN = 128;      // output tile (MMA M, N)
constexpr int BK = 64;                 // K per stage: two 32-wide tiles
constexpr int kStages = 6;
constexpr int kProducerWarps = 4, kEpiWarps = 8;   // warps 0..7 epilogue (TMEM lane quadrant = warp % 4), 8..11 producers, 12 MMA issuer
constexpr int kMmaWarp = kEpiWarps + kProducerWarps;
constexpr int kThreads = 32 * (kMmaWarp + 1);
constexpr int kOperandBytes = 128 * BK * 2;        // one operand of one stage
constexpr int kStageBytes = 2 * kOperandBytes;
constexpr int kSlabBytes = 128 * 32;               // one operand of one MMA (K = 16): eight faces
constexpr uint32_t kSBO = 256;                     // swizzle atoms of eight 32-byte rows: M groups of A, K groups of B
constexpr uint32_t kBGroup = 512;                  // B: next 16 columns
constexpr int kBars = kStages * kStageBytes;
constexpr int kMisc = kBars + 8 * (2 * kStages + 4);
constexpr int kSmemBytes = kMisc + 16 + 1024;
static_assert(kSmemBytes <= 232448, "shared memory budget");
static_assert(kStages * kStageBytes >= BM * BN * 4, "the partial sums of a shared tile reuse the ring");
constexpr int kTmemCols = 2 * BN;

struct Args {
    const uint16_t *a, *w, *bias;
    void *out;
    int64_t rows, K, N;                    // rows of one batch entry
    int64_t a_bstride, w_bstride, out_bstride;   // elements between batch entries
    int mt, nt;                            // output tiles per batch entry
    int tiles, split;                      // all output tiles; blocks (= cluster size) that share a tile's K range
    int nstages;                           // stages of the whole K range
    int chunk;                             // stages per accumulator
    int act, out_dtype, a_row_major, out_row_major, out_aligned32;
    unsigned wait_limit;   // of every barrier wait, in 1024 SM clocks
    int *status;
};

__device__ __forceinline__ long long wait_clocks(const Args &p) { return (long long)p.wait_limit << 10; }

// 32 bytes, in one store where the tensor allows it (the entry points ask for 16-byte alignment): a bfloat16 face row, so
// that a warp's store covers whole 512-byte faces.
__device__ __forceinline__ void store_32b(void *dst, const uint32_t (&v)[8], bool aligned32) {
    if (aligned32) {
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                     "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                     : "memory");
    } else {
        reinterpret_cast<uint4 *>(dst)[0] = make_uint4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<uint4 *>(dst)[1] = make_uint4(v[4], v[5], v[6], v[7]);
    }
}

// 16 columns from n0 of one row: bias, activation, store. (Coordinates in 32 bits: 64 took the kernel from 4 bytes of register
// spills to 148 and a 1024 x 1024 x 1024 launch from 9.3 us to 9.9.)
template <int ACT>
__device__ __forceinline__ void finish16(const Args &p, int batch, int row, int n0, float *v) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        if (p.bias) v[j] += bias_at(p.bias, n0 + j);
        v[j] = apply_activation_t<ACT>(v[j]);
    }
    const int64_t off = batch * p.out_bstride + (p.out_row_major ? row * p.N + n0 : tiled_offset(row, n0, p.N >> 5));
    uint32_t h[8];
    if (p.out_dtype == TTB_FLOAT32) {
        float *o = reinterpret_cast<float *>(p.out) + off;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
#pragma unroll
            for (int j = 0; j < 8; ++j) h[j] = __float_as_uint(v[8 * q + j]);
            store_32b(o + 8 * q, h, p.out_aligned32);
        }
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) h[j] = (uint32_t)f32_to_bf16_bits(v[2 * j]) | ((uint32_t)f32_to_bf16_bits(v[2 * j + 1]) << 16);
        store_32b(reinterpret_cast<uint16_t *>(p.out) + off, h, p.out_aligned32);
    }
}

// One thread's half row of a tile.
template <int ACT>
__device__ __forceinline__ void finish_half(const Args &p, int batch, int row, int n0, float (&sum)[BN / 2]) {
#pragma unroll
    for (int q = 0; q < BN / 2; q += 16)
        if (n0 + q < p.N) {
            finish16<ACT>(p, batch, row, n0 + q, sum + q);
            asm volatile("" ::: "memory");   // (keeps the compiler from fetching all groups' bias values at once, which spills)
        }
}

__global__ void __launch_bounds__(kThreads, 1) matmul_bf16_kernel(const __grid_constant__ Args p) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t sbase = smem_u32(smem);
    const uint32_t bar0 = sbase + kBars;
    auto full = [&](int s) { return bar0 + 8u * s; };
    auto empty = [&](int s) { return bar0 + 8u * (kStages + s); };
    auto acc_full = [&](int b) { return bar0 + 8u * (2 * kStages + b); };
    auto acc_empty = [&](int b) { return bar0 + 8u * (2 * kStages + 2 + b); };
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(smem + kMisc);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + kMisc + 4);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(full(s), 32 * kProducerWarps);
            mbar_init(empty(s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(acc_full(b), 1);
            mbar_init(acc_empty(b), kEpiWarps);
        }
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == kMmaWarp) {
        tmem_alloc(sbase + kMisc, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    // The launch overlaps the previous kernel's tail (programmatic dependency); nothing above touches global memory, and every
    // role waits for that kernel first: the roles that do touch it, and the issuer because its bounded waits are not to count
    // the time of a kernel that waits for other GPUs.
    grid_dep_launch();

    // this block's share of a tile's K range, in stages (the same for every tile); a split gives every block at least one
    const int rank = p.split > 1 ? (int)cluster_rank() : 0;
    const int first_tile = (int)blockIdx.x / p.split, tile_step = (int)gridDim.x / p.split;
    const int st0 = (int)((int64_t)p.nstages * rank / p.split), st1 = (int)((int64_t)p.nstages * (rank + 1) / p.split);
    const int Kt = (int)(p.K >> 5), Ntt = (int)(p.N >> 5);
    const int mtiles32 = (int)(p.rows >> 5);
    auto locate = [&](int tile, int &b, int &m, int &n) {   // row blocks vary fastest: neighbours share a weight column block
        m = tile % p.mt;
        const int r = tile / p.mt;
        n = r % p.nt;
        b = r / p.nt;
    };

    if (warp >= kEpiWarps && warp < kMmaWarp) {
        // ---------------- producers ----------------
        grid_dep_wait();
        const int pw = warp - kEpiWarps;
        const int fr = lane >> 1, fh = lane & 1;   // inside a face: lane l takes 16-byte chunk l
        const uint32_t face_dst = face_chunk_sw32(lane);
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int tile = first_tile; ok && tile < p.tiles; tile += tile_step) {
            int b, m, n;
            locate(tile, b, m, n);
            const uint16_t *const ab = p.a + b * p.a_bstride, *const wb = p.w + b * p.w_bstride;
            for (int st = st0; st < st1; ++st) {
                if (!__all_sync(0xffffffffu, mbar_wait(empty(s), ph ^ 1, abort_flag, p.status, 41, wait_clocks(p)))) { ok = false; break; }
                const uint32_t dst = sbase + s * kStageBytes;
                // eight tiles per operand: this warp takes tile row (column) pw of each of the stage's two K tiles
#pragma unroll
                for (int kl = 0; kl < 2; ++kl) {
                    const int kt = st * 2 + kl;
                    if (kt < Kt) {
                        const int tr = m * 4 + pw, tc = n * 4 + pw;
                        if (tr < mtiles32) {
                            // face f: rows 16 * (f / 2) .., K 16 * (f % 2) ..
                            const uint32_t d = dst + (uint32_t)(kl * 2 * kSlabBytes + pw * 1024) + face_dst;
                            if (p.a_row_major) {
                                const uint16_t *src = ab + ((int64_t)tr * 32 + fr) * p.K + kt * 32 + fh * 8;
#pragma unroll
                                for (int f = 0; f < 4; ++f) cp_async16(d + (f & 1) * kSlabBytes + (f >> 1) * 512, src + (f >> 1) * 16 * p.K + (f & 1) * 16);
                            } else {
                                const uint16_t *src = ab + ((int64_t)tr * Kt + kt) * 1024 + lane * 8;
#pragma unroll
                                for (int f = 0; f < 4; ++f) cp_async16(d + (f & 1) * kSlabBytes + (f >> 1) * 512, src + f * 256);
                            }
                        }
                        if (tc < Ntt) {
                            // face f: K 16 * (f / 2) .., columns 16 * (f % 2) ..
                            const uint16_t *src = wb + ((int64_t)kt * Ntt + tc) * 1024 + lane * 8;
                            const uint32_t d = dst + kOperandBytes + (uint32_t)(kl * 2 * kSlabBytes + pw * 2 * kBGroup) + face_dst;
#pragma unroll
                            for (int f = 0; f < 4; ++f) cp_async16(d + (f >> 1) * kSlabBytes + (f & 1) * kBGroup, src + f * 256);
                        }
                    }
                }
                cp_async_arrive(full(s));   // every producer thread's copies of the stage, whenever they land
                if (++s == kStages) { s = 0; ph ^= 1; }
            }
        }
        cp_async_wait_all();   // (also after a wait that ran out: nothing is left in flight)
    } else if (warp == kMmaWarp) {
        // ---------------- MMA issuer (warp-uniform, one elected lane issues) ----------------
        grid_dep_wait();
        const bool leader = elect_one();
        constexpr uint32_t idesc = instr_desc_bf16_f32(BM, BN, /*a_mn_major=*/false, /*b_mn_major=*/true);
        const uint64_t a_desc0 = smem_desc_sw32(sbase, kSBO), b_desc0 = smem_desc_sw32_mn(sbase + kOperandBytes, kBGroup, kSBO);
        auto mk = [](uint64_t desc, uint32_t bytes) { return (desc & ~0xffffffffull) | ((uint32_t)desc + (bytes >> 4)); };
        int s = 0, c = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int tile = first_tile; ok && tile < p.tiles; tile += tile_step) {
            for (int st = st0; ok && st < st1; st += p.chunk, ++c) {
                const int buf = c & 1;
                if (!__all_sync(0xffffffffu, mbar_wait(acc_empty(buf), (uint32_t)(((c >> 1) & 1) ^ 1), abort_flag, p.status, 42, wait_clocks(p)))) { ok = false; break; }
                const int end = min(st1, st + p.chunk);
                for (int i = st; i < end; ++i) {
                    if (!__all_sync(0xffffffffu, mbar_wait(full(s), ph, abort_flag, p.status, 43, wait_clocks(p)))) { ok = false; break; }
                    // The copies are generic-proxy writes; ordering them here, before the MMAs read them, and not in the producers
                    // keeps the producers' later copies flowing (a fence there waits for those too: 31 B per clock).
                    fence_proxy_async_smem();
                    tc_fence_after_sync();
                    const uint32_t off = (uint32_t)(s * kStageBytes);
                    if (leader) {
#pragma unroll
                        for (int k16 = 0; k16 < BK / 16; ++k16)   // (the last stage may hold one K tile only)
                            if (k16 < 2 || i * 2 + 1 < Kt)
                                mma_bf16_ss(tmem_base + (uint32_t)(buf * BN), mk(a_desc0, off + k16 * kSlabBytes), mk(b_desc0, off + k16 * kSlabBytes), idesc,
                                            i > st || k16 > 0);
                        mma_commit(empty(s));
                    }
                    if (++s == kStages) { s = 0; ph ^= 1; }
                }
                if (ok && leader) mma_commit(acc_full(buf));
            }
        }
    } else {
        // ---------------- epilogue warps: TMEM lanes (rows) 32 * (warp % 4) .., column half warp / 4 ----------------
        grid_dep_wait();
        const int quad = warp & 3, half = warp >> 2;
        const uint32_t t_lane = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(half * (BN / 2));
        int c = 0;
        bool ok = true;
        for (int tile = first_tile; ok && tile < p.tiles; tile += tile_step) {
            int b, m, n;
            locate(tile, b, m, n);
            float sum[BN / 2];
#pragma unroll
            for (int j = 0; j < BN / 2; ++j) sum[j] = 0.0f;
            for (int st = st0; st < st1; st += p.chunk, ++c) {
                const int buf = c & 1;
                if (!__all_sync(0xffffffffu, mbar_wait(acc_full(buf), (uint32_t)((c >> 1) & 1), abort_flag, p.status, 44, wait_clocks(p)))) { ok = false; break; }
                tc_fence_after_sync();
#pragma unroll
                for (int q = 0; q < BN / 2; q += 32) {
                    uint32_t r0[16], r1[16];
                    tmem_ld16(t_lane + (uint32_t)(buf * BN + q), r0);
                    tmem_ld16(t_lane + (uint32_t)(buf * BN + q + 16), r1);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        sum[q + j] += __uint_as_float(r0[j]);
                        sum[q + 16 + j] += __uint_as_float(r1[j]);
                    }
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty(buf));
            }
            if (!ok) break;
            const int row = m * BM + quad * 32 + lane;
            const int col = n * BN + half * (BN / 2);
            if (p.split == 1) {
                if (row < p.rows) TTB_DISPATCH_ACT(p.act, finish_half<ACT>(p, b, row, col, sum));
            } else {
                // [column / 4][row] float4 in the ring's place: every copy of this block has landed and every MMA has read it
                float4 *part = reinterpret_cast<float4 *>(smem);
#pragma unroll
                for (int q = 0; q < BN / 2; q += 4)
                    part[(half * (BN / 2) + q) / 4 * BM + quad * 32 + lane] = make_float4(sum[q], sum[q + 1], sum[q + 2], sum[q + 3]);
            }
        }
    }

    if (p.split > 1) {
        // one tile per cluster: the blocks add each other's partial sums in block order, each for its share of the columns
        __syncwarp();
        cluster_sync();
        if (warp < kEpiWarps && *abort_flag == 0) {
            const int quad = warp & 3, half = warp >> 2;
            int b, m, n;
            locate(first_tile, b, m, n);
            const int row = m * BM + quad * 32 + lane;
            const int units = BN / 16 / p.split;   // columns in groups of 16
            if (row < p.rows)
                for (int u = half; u < units; u += 2) {
                    const int col = (rank * units + u) * 16;
                    if (n * BN + col >= p.N) break;
                    float v[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = 0.0f;
                    for (int r = 0; r < p.split; ++r) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const float4 x = ld_cluster_f32x4(sbase + (uint32_t)(((col / 4 + j) * BM + quad * 32 + lane) * 16), (uint32_t)r);
                            v[4 * j] += x.x; v[4 * j + 1] += x.y; v[4 * j + 2] += x.z; v[4 * j + 3] += x.w;
                        }
                    }
                    TTB_DISPATCH_ACT(p.act, finish16<ACT>(p, b, row, n * BN + col, v));
                }
        }
        __syncwarp();
        cluster_sync();   // nobody leaves while another block may still read its shared memory
    }

    // ---------------- teardown ----------------
    tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag) {
        // A wait ran out: give MMAs still in flight a bounded time to finish before the block's memory is released.
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == kMmaWarp) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

}  // namespace

// a [batch, rows, K], w [batch, K, N] (batch > 1) or [K, N]; every size a multiple of 32.
int32_t launch_matmul_bf16(const void *a, const void *w, const void *bias, void *out, int out_dtype, int64_t batch, int64_t rows, int64_t K,
                           int64_t N, int act, int flags, int *status, cudaStream_t stream) {
    Args p;
    p.a = (const uint16_t *)a; p.w = (const uint16_t *)w; p.bias = (const uint16_t *)bias; p.out = out;
    p.rows = rows; p.K = K; p.N = N;
    p.a_bstride = rows * K; p.w_bstride = K * N; p.out_bstride = rows * N;
    p.act = act; p.out_dtype = out_dtype;
    p.a_row_major = (flags & TTB_MM_A_ROW_MAJOR) != 0;
    p.out_row_major = (flags & TTB_MM_OUT_ROW_MAJOR) != 0;
    p.out_aligned32 = (reinterpret_cast<uintptr_t>(out) & 31) == 0;
    p.status = status;
    p.wait_limit = barrier_limit_kcycles();
    const int64_t mt = (rows + BM - 1) / BM, nt = (N + BN - 1) / BN, tiles = mt * nt * batch;
    if (tiles > INT32_MAX / 8 || K / 32 > INT32_MAX || rows > INT32_MAX - BM || N > INT32_MAX - BN) return fail(TTB_E_UNSUPPORTED, "ttb_matmul: too many output tiles");
    p.mt = (int)mt; p.nt = (int)nt; p.tiles = (int)tiles;
    p.nstages = (int)((K + BK - 1) / BK);
    p.chunk = out_dtype == TTB_FLOAT32 ? 1 : 4;
    int dev = 0;
    TTB_CUDA_TRY(cudaGetDevice(&dev));
    static struct {
        Once once;
        int sms, clusters[9];   // multiprocessors; clusters of 2, 4 and 8 blocks that run at the same time
    } devices[64];
    if (dev < 0 || dev >= 64) return fail(TTB_E_UNSUPPORTED, "ttb_matmul: device index %d is out of range", dev);
    auto &d = devices[dev];
    if (int32_t rc = d.once.run([&]() -> int32_t {
            TTB_CUDA_TRY(cudaFuncSetAttribute(matmul_bf16_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
            TTB_CUDA_TRY(cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev));
            for (int c = 2; c <= 8; c *= 2) {
                cudaLaunchConfig_t q = {};
                q.gridDim = dim3((unsigned)(d.sms / c * c));
                q.blockDim = dim3(kThreads);
                q.dynamicSmemBytes = kSmemBytes;
                cudaLaunchAttribute ca[1];
                ca[0].id = cudaLaunchAttributeClusterDimension;
                ca[0].val.clusterDim.x = (unsigned)c;
                ca[0].val.clusterDim.y = ca[0].val.clusterDim.z = 1;
                q.attrs = ca;
                q.numAttrs = 1;
                TTB_CUDA_TRY(cudaOccupancyMaxActiveClusters(&d.clusters[c], matmul_bf16_kernel, &q));
            }
            return TTB_OK;
        }))
        return rc;
    // Clusters share a tile while all of them run at the same time and each block keeps at least four stages (the exchange of
    // partial sums costs about as much as two).
    p.split = 1;
    while (p.split < 8 && tiles <= d.clusters[p.split * 2] && p.nstages / (p.split * 2) >= 4) p.split *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(p.split > 1 ? tiles * p.split : tiles < d.sms ? tiles : d.sms));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)p.split;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p.split > 1 ? 2 : 1;
    TTB_CUDA_TRY(cudaLaunchKernelEx(&cfg, matmul_bf16_kernel, p));
    TTB_LAUNCH_CHECK("matmul_bf16");
    return TTB_OK;
}

}  // namespace ttb
