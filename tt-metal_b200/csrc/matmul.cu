// C-ABI entry points for matmul / linear and the all-gather layout helper: argument validation and
// kernel selection. Tensor-core kernels take the shapes their tiling covers (block-float weights) or any shape
// (bfloat16 weights); everything else goes to the shape-generic CUDA-core kernel, which computes the same function.
#include "common.cuh"

namespace ttb {
int32_t launch_matmul_generic(const void *a, const void *w, int w_dtype, const void *bias, void *out, int out_dtype,
                              int64_t rows, int64_t K, int64_t N, int act, int flags, cudaStream_t stream);
int32_t launch_bmm_generic(const void *a, const void *w, int w_dtype, void *out, int out_dtype, int64_t batch, int64_t M, int64_t K,
                           int64_t N, cudaStream_t stream);
int32_t launch_matmul_bf16(const void *a, const void *w, const void *bias, void *out, int out_dtype, int64_t batch, int64_t rows, int64_t K,
                           int64_t N, int act, int flags, int *status, cudaStream_t stream);
bool decode_supported(int w_dtype, int64_t rows, int64_t K, int64_t N);
bool decode_is_faster(int64_t rows, int64_t K, int64_t tiles, bool ragged);
int stream_blocks();
int64_t decode_workspace_bytes(int64_t rows, int64_t K, int64_t N, bool smem_operand);
int32_t launch_matmul_decode(const void *a, const void *w, int w_dtype, const void *bias, void *out, int out_dtype,
                             int64_t rows, int64_t K, int64_t N, int act, int flags, void *workspace,
                             int64_t workspace_bytes, bool counters_are_zero, bool compact, cudaStream_t stream,
                             const ttb_peer_gather *gather, const ttb_peer_wait_t *wait);
int32_t read_and_clear_status(cudaStream_t stream);
int32_t status_word_address(int **out);
bool prefill_supported(int w_dtype, int64_t rows, int64_t K, int64_t N);
int64_t prefill_workspace_bytes(int64_t rows, int64_t K);
int32_t launch_matmul_prefill(const void *a, const void *w, int w_dtype, const void *bias, void *out, int out_dtype, int64_t rows,
                              int64_t K, int64_t N, int act, int flags, void *workspace, int64_t workspace_bytes, int *status,
                              cudaStream_t stream);
int32_t launch_matmul_rows(const void *a, int count, const void *const *w, int w_dtype, const void *const *bias, void *const *out, int64_t rows,
                           int64_t K, const int64_t *N, int act, int flags, int *status, cudaStream_t stream);

namespace {

__global__ void gather_interleave_kernel(const uint4 *__restrict__ src, uint4 *__restrict__ dst, int ranks, int64_t rows,
                                         int64_t vec_per_rank_row) {
    // dst[r][g][v] = src[g][r][v], 16-byte vectors
    const int64_t total = (int64_t)ranks * rows * vec_per_rank_row;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = i % vec_per_rank_row;
        const int64_t g = (i / vec_per_rank_row) % ranks;
        const int64_t r = i / (vec_per_rank_row * ranks);
        dst[i] = __ldg(src + (g * rows + r) * vec_per_rank_row + v);
    }
}

int32_t validate(const void *a, int a_dtype, const void *w, int w_dtype, void *out, int out_dtype, int64_t batch, int64_t M,
                 int64_t K, int64_t N, int act) {
    if (!a || !w || !out) return fail(TTB_E_INVALID, "ttb_matmul: null tensor pointer");
    if (a_dtype != TTB_BFLOAT16) return fail(TTB_E_UNSUPPORTED, "ttb_matmul: activations must be bfloat16");
    if (w_dtype != TTB_BFLOAT8_B && w_dtype != TTB_BFLOAT4_B && w_dtype != TTB_BFLOAT16)
        return fail(TTB_E_UNSUPPORTED, "ttb_matmul: weights must be bfloat8_b, bfloat4_b or bfloat16");
    if (out_dtype != TTB_BFLOAT16 && out_dtype != TTB_FLOAT32)
        return fail(TTB_E_UNSUPPORTED, "ttb_matmul: output must be bfloat16 or float32");
    if (batch <= 0 || M <= 0 || K <= 0 || N <= 0 || M % 32 || K % 32 || N % 32)
        return fail(TTB_E_INVALID, "ttb_matmul: batch, M, K, N must be positive and M, K, N multiples of 32 (got %lld, %lld, %lld, %lld)",
                    (long long)batch, (long long)M, (long long)K, (long long)N);
    if (act < TTB_ACT_NONE || act > TTB_ACT_SILU) return fail(TTB_E_INVALID, "ttb_matmul: unknown activation %d", act);
    if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out)) & 15)
        return fail(TTB_E_INVALID, "ttb_matmul: tensors must be 16-byte aligned");
    return TTB_OK;
}

// bfloat16 weights: the tensor-core kernel, except for
//  * fp32 results of fewer than 128 products, where its additions (which cut off low bits) come out further from 64 bits than a
//    chain of fused multiply-adds (2-norm at K = 64: 6.5e-8 against 5.1e-8; at 128: 7.1e-8 against 7.3e-8, and the longer the
//    further ahead);
//  * 32 products of small results, where its start-up or, with many small batch entries, a 128 x 128 tile for each costs more
//    than the CUDA cores' 32 x 32 tiles (us, CUDA cores / tensor cores: 128 x 32 x 512 2.8 / 3.6, 512 x 32 x 512 3.4 / 3.9, 1000 x [32 x
//    32 x 32] 7.1 / 10.6, but 1024 x 32 x 1024 7.0 / 4.0, 32 x [128 x 32 x 128] 5.1 / 4.1), and 64 products of many batch entries of one
//    tile (4000 x [32 x 64 x 32] 32.5 / 35.2, 1000 10.4 / 10.8, but 500 7.1 / 7.0).
bool bf16_on_tensor_cores(int out_dtype, int64_t batch, int64_t rows, int64_t K, int64_t N) {
    const int64_t small = batch * (rows / 32) * (N / 32), large = batch * ((rows + 127) / 128) * ((N + 127) / 128);
    if (K == 32 && small < 300 + large) return false;
    if (K == 64 && small == large && large >= 1000) return false;
    return out_dtype == TTB_BFLOAT16 || K >= 128;
}

// bfloat16 results that the prefill kernel computes faster than the one of matmul_rows.cu: whole 256 x 256 blocks whose last round
// over the multiprocessors is nearly full (anything broken favours the finer tiles there: us, prefill / rows kernel, 1.5 rounds 512 x
// 1024 x 28416 55.5 / 45.1, blocks of 128 rows or columns 640 x 1024 x 14336 63 / 39, 512 x 1024 x 14208 41 / 28), and
//  * a short K range, where a round's fixed part counts: 1.0 round 1024 x 256 x 9472 18.2 / 20.2, 1024 x 1024 x 9472 30.3 / 31.3, 1.7
//    rounds 1024 x 512 x 16384 40.9 / 44.7, 3.0 rounds 1024 x 768 x 28416 72.9 / 76.5, but 1024 x 2048 x 9472 45.3 / 44.5; at K = 512
//    from four rounds on with any last one: 4.5 rounds 1536 x 512 x 28672 97.8 / 100.8, 6.05 rounds 2048 x 512 x 28672 129.4 / 133.5,
//    but 3.5 rounds 2048 x 512 x 16384 78.3 / 74.1;
//  * a long one, where the chip runs into its power limit and the kernel that moves less data gains: bfloat8_b 2.0 rounds 1024 x 8192 x
//    18944 265.5 / 274.8, 3.0 rounds 1024 x 6144 x 28416 303.6 / 312.3, 0.9 rounds 1024 x 28672 x 8192 432.8 / 450.5, bfloat4_b 4.0
//    rounds 2048 x 12288 x 18944 810.7 / 844.0, 6.0 rounds 2048 x 8192 x 28416 772.8 / 806.4, but bfloat8_b 0.9 rounds 2048 x 8192 x 4096 141.2 / 131.1, 1.7 rounds 2048 x 8192 x 8192
//    275 / 248, bfloat4_b 2.0 rounds 1024 x 8192 x 18944 281 / 259; with many rounds a small remainder costs little: 6.05 rounds
//    2048 x 8192 x 28672 860 / 853 to 890, but 2048 x 4096 x 28672 526 / 479.
bool prefill_is_faster(int w_dtype, int64_t rows, int64_t K, int64_t N) {
    if (rows % 256 || N % 256) return false;
    const int64_t sms = stream_blocks(), blocks = rows / 256 * (N / 256), last = (blocks - 1) % sms + 1;
    const bool full = last * 16 >= sms * 15;
    if (K <= 1024) return last * 10 >= sms * 7 || (K <= 512 && blocks >= 4 * sms);
    if (w_dtype == TTB_BFLOAT4_B) return full && (K >= 12288 || (K >= 8192 && blocks > 5 * sms));
    if (K >= 8192) return full || (K >= 12288 && last * 20 >= sms * 17) || (blocks >= 5 * sms && last * 4 < sms);
    return full && K >= 6144 && blocks > 2 * sms;
}

// bfloat16 results that the kernel of matmul_rows.cu takes, whole and whatever the column count (fp32 results keep the row ranges
// below, whose shorter chains of additions bring them closer to 64 bits). Three lines, with both sides measured (us):
//  * 96 rows and more, except where the decode kernel is faster (decode_is_faster): 96 x 4096 x 4096 16.0 there, 12.0 here; 128 x
//    4096 x 14336 bfloat4_b 46.2 / 28.4; above 256 rows, two launches and more there, always: 288 rows and up 0.28 to 0.78 of it;
//  * 64 rows while its 128-column tiles number at most half the SMs and their K range can be shared: 64 x 8192 x 8192 34.2 /
//    27.1, 64 x 4096 x 1024 14.2 / 8.0, 64 x 8192 x 9472 (74 tiles) 34.1 / 28.1, but 64 x 8192 x 9600 (75 tiles) 34.0 / 46.0; up to a K
//    at which that is so for any column count (64 x 20480 x 512 15.8 / 17.0);
//  * where the prefill kernel applies, except for the shapes that it keeps.
bool rows_kernel_can(int w_dtype, int out_dtype, int flags) {
    // (under TTB_MM_DETERMINISTIC a call gives the bytes of the same stage of a sequence, which the decode kernel computes)
    return w_dtype != TTB_BFLOAT16 && out_dtype == TTB_BFLOAT16 && !(flags & (TTB_MM_FORCE_GENERIC | TTB_MM_DECODE_SMEM_OPERAND | TTB_MM_DETERMINISTIC));
}
bool rows_kernel_takes(int w_dtype, int out_dtype, int64_t rows, int64_t K, int64_t N, int flags) {
    if (!rows_kernel_can(w_dtype, out_dtype, flags)) return false;
    if (rows == 64) return (N + 127) / 128 * 2 <= stream_blocks() && K <= 8192;
    if (rows < 96) return false;
    if (rows <= 256) return !(decode_supported(w_dtype, rows, K, N) && decode_is_faster(rows, K, (N + 127) / 128, N % 128 != 0));
    return !(prefill_supported(w_dtype, rows, K, N) && prefill_is_faster(w_dtype, rows, K, N));
}

// Row ranges of one matmul and the tensor-core kernel that takes each: the decode kernels serve up to 256 rows, the prefill
// kernel multiples of 128 from 512 up (column counts that are multiples of 128). Row counts in between run as two decode
// launches (256 rows + the rest); a ragged count above 512 as the prefill kernel on the whole 128-row blocks plus a decode
// launch on the last 32 to 96 rows; and what the prefill kernel cannot take at all (a last column tile of fewer than 128
// columns) as decode launches over ranges of 256 rows, up to kMaxRowChunks of them. (Rows are
// contiguous in both layouts - a tile row of a tiled tensor is 32 whole rows - so a range is just an offset.)
struct RowChunk {
    int64_t row0, rows;
    bool prefill;
};
constexpr int kMaxRowChunks = 16;
int plan_rows(int w_dtype, int64_t rows, int64_t K, int64_t N, RowChunk (&out)[kMaxRowChunks]) {
    if (decode_supported(w_dtype, rows, K, N)) {
        out[0] = {0, rows, false};
        return 1;
    }
    if (prefill_supported(w_dtype, rows, K, N)) {
        out[0] = {0, rows, true};
        return 1;
    }
    if (rows > 256 && rows < 512 && decode_supported(w_dtype, 256, K, N) && decode_supported(w_dtype, rows - 256, K, N)) {
        out[0] = {0, 256, false};
        out[1] = {256, rows - 256, false};
        return 2;
    }
    const int64_t whole = rows / 128 * 128;
    if (rows > 512 && rows != whole && prefill_supported(w_dtype, whole, K, N) && decode_supported(w_dtype, rows - whole, K, N)) {
        out[0] = {0, whole, true};
        out[1] = {whole, rows - whole, false};
        return 2;
    }
    const int64_t last = rows % 256;
    if (rows >= 512 && rows <= 256 * kMaxRowChunks && decode_supported(w_dtype, 256, K, N) && (last == 0 || decode_supported(w_dtype, last, K, N))) {
        int n = 0;
        for (int64_t r0 = 0; r0 < rows; r0 += 256) out[n++] = {r0, rows - r0 < 256 ? rows - r0 : 256, false};
        return n;
    }
    return 0;
}

// The kernel of a call whose arguments are valid.
int kernel_of(int w_dtype, int out_dtype, int64_t rows, int64_t K, int64_t N, int flags) {
    if (flags & TTB_MM_FORCE_GENERIC) return TTB_KERNEL_GENERIC;
    if (w_dtype == TTB_BFLOAT16) return bf16_on_tensor_cores(out_dtype, 1, rows, K, N) && rows / 32 <= 65535 ? TTB_KERNEL_BF16 : TTB_KERNEL_GENERIC;
    if (rows_kernel_takes(w_dtype, out_dtype, rows, K, N, flags)) return TTB_KERNEL_ROWS;
    RowChunk chunks[kMaxRowChunks];
    return plan_rows(w_dtype, rows, K, N, chunks) ? TTB_KERNEL_RANGES : TTB_KERNEL_GENERIC;
}

}  // namespace
}  // namespace ttb

using namespace ttb;

extern "C" {

int64_t ttb_matmul_workspace_bytes(int32_t w_dtype, int64_t batch, int64_t M, int64_t K, int64_t N, int32_t flags) {
    const int64_t rows = batch * M;
    if (flags & TTB_MM_FORCE_GENERIC) return 0;
    RowChunk chunks[kMaxRowChunks];
    const int n = plan_rows(w_dtype, rows, K, N, chunks);
    int64_t bytes = 0;
    for (int i = 0; i < n; ++i) {
        const int64_t b = chunks[i].prefill ? prefill_workspace_bytes(chunks[i].rows, K) : decode_workspace_bytes(chunks[i].rows, K, N, (flags & TTB_MM_DECODE_SMEM_OPERAND) != 0);
        bytes = b > bytes ? b : bytes;
    }
    return bytes;
}

int32_t ttb_matmul_kernel(int32_t w_dtype, int32_t out_dtype, int64_t batch, int64_t M, int64_t K, int64_t N, int32_t flags) {
    const void *const any = reinterpret_cast<const void *>(uintptr_t(256));   // (no tensors: their checks pass)
    if (int32_t rc = validate(any, TTB_BFLOAT16, any, w_dtype, const_cast<void *>(any), out_dtype, batch, M, K, N, TTB_ACT_NONE)) return rc;
    return kernel_of(w_dtype, out_dtype, batch * M, K, N, flags);
}

/* The row ranges of TTB_KERNEL_RANGES: out[0] = launches (0: the decode and prefill kernels do not take the shape), then per launch
 * its rows and 1 for the prefill kernel, 0 for a decode kernel - for as many launches as `out` has room for (at least two). */
int32_t ttb_matmul_plan(int32_t w_dtype, int64_t batch, int64_t M, int64_t K, int64_t N, int32_t flags, int64_t *out, int32_t out_len) {
    if (!out || out_len < 5) return fail(TTB_E_INVALID, "ttb_matmul_plan: needs room for 5 values");
    RowChunk chunks[kMaxRowChunks];
    const int n = (flags & TTB_MM_FORCE_GENERIC) ? 0 : plan_rows(w_dtype, batch * M, K, N, chunks);
    out[0] = n;
    for (int i = 0; 2 + 2 * i < out_len && i < kMaxRowChunks; ++i) {
        out[1 + 2 * i] = i < n ? chunks[i].rows : 0;
        out[2 + 2 * i] = i < n && chunks[i].prefill ? 1 : 0;
    }
    return TTB_OK;
}

int32_t ttb_matmul(const void *a, int32_t a_dtype, const void *w, int32_t w_dtype, const void *bias, void *out,
                   int32_t out_dtype, int64_t batch, int64_t M, int64_t K, int64_t N, int32_t act, int32_t flags,
                   void *workspace, int64_t workspace_bytes, void *stream) {
    if (int32_t rc = validate(a, a_dtype, w, w_dtype, out, out_dtype, batch, M, K, N, act)) return rc;
    const int64_t rows = batch * M;  // tiled [batch, M, K] with M % 32 == 0 is the same buffer as tiled [batch*M, K]
    auto s = (cudaStream_t)stream;
    int kernel = kernel_of(w_dtype, out_dtype, rows, K, N, flags);
    // (a call that brings no scratch still gets the kernel that needs none)
    if (kernel == TTB_KERNEL_RANGES && rows >= 96 && rows_kernel_can(w_dtype, out_dtype, flags) &&
        !workspace_serves(workspace, workspace_bytes, ttb_matmul_workspace_bytes(w_dtype, batch, M, K, N, flags)))
        kernel = TTB_KERNEL_ROWS;
    if (kernel == TTB_KERNEL_GENERIC) return launch_matmul_generic(a, w, w_dtype, bias, out, out_dtype, rows, K, N, act, flags, s);
    int *status = nullptr;
    if (kernel != TTB_KERNEL_RANGES) {
        if (int32_t rc = status_word_address(&status)) return rc;
        if (kernel == TTB_KERNEL_BF16) return launch_matmul_bf16(a, w, bias, out, out_dtype, 1, rows, K, N, act, flags, status, s);
        return launch_matmul_rows(a, 1, &w, w_dtype, &bias, &out, rows, K, &N, act, flags, status, s);
    }
    RowChunk chunks[kMaxRowChunks];
    const int n = plan_rows(w_dtype, rows, K, N, chunks);
    const int64_t out_elem = out_dtype == TTB_FLOAT32 ? 4 : 2;
    for (int i = 0; i < n; ++i) {
        const void *ai = static_cast<const uint8_t *>(a) + chunks[i].row0 * K * 2;
        void *oi = static_cast<uint8_t *>(out) + chunks[i].row0 * N * out_elem;
        int32_t rc;
        if (chunks[i].prefill) {
            if ((rc = status_word_address(&status))) return rc;
            rc = launch_matmul_prefill(ai, w, w_dtype, bias, oi, out_dtype, chunks[i].rows, K, N, act, flags, workspace, workspace_bytes, status, s);
        } else {
            rc = launch_matmul_decode(ai, w, w_dtype, bias, oi, out_dtype, chunks[i].rows, K, N, act, flags, workspace, workspace_bytes,
                                      (flags & TTB_MM_WORKSPACE_ZEROED) != 0, /*compact=*/false, s, nullptr, nullptr);
        }
        if (rc) return rc;
    }
    return TTB_OK;
}

int32_t ttb_bmm(const void *a, int32_t a_dtype, const void *w, int32_t w_dtype, void *out, int32_t out_dtype, int64_t batch, int64_t M,
                int64_t K, int64_t N, void *stream) {
    if (int32_t rc = validate(a, a_dtype, w, w_dtype, out, out_dtype, batch, M, K, N, TTB_ACT_NONE)) return rc;
    if (w_dtype == TTB_BFLOAT16 && bf16_on_tensor_cores(out_dtype, batch, M, K, N) && M / 32 <= 65535 && batch <= 65535) {
        int *status = nullptr;
        if (int32_t rc = status_word_address(&status)) return rc;
        return launch_matmul_bf16(a, w, nullptr, out, out_dtype, batch, M, K, N, TTB_ACT_NONE, 0, status, (cudaStream_t)stream);
    }
    return launch_bmm_generic(a, w, w_dtype, out, out_dtype, batch, M, K, N, (cudaStream_t)stream);
}

int32_t ttb_check_status(void *stream) { return read_and_clear_status((cudaStream_t)stream); }

int32_t ttb_gather_interleave(const void *src, void *dst, int32_t elem, int32_t ranks, int64_t rows, int64_t cols_per_rank,
                              void *stream) {
    if (!src || !dst) return fail(TTB_E_INVALID, "ttb_gather_interleave: null pointer");
    if (ranks <= 0 || rows <= 0 || cols_per_rank <= 0 || elem <= 0) return fail(TTB_E_INVALID, "ttb_gather_interleave: bad sizes");
    const int64_t row_bytes = cols_per_rank * elem;
    if (row_bytes % 16 || ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15))
        return fail(TTB_E_INVALID, "ttb_gather_interleave: per-rank rows must be a multiple of 16 bytes and pointers 16-byte aligned");
    const int64_t total = (int64_t)ranks * rows * (row_bytes / 16);
    const int blocks = (int)((total + 255) / 256 < 148 * 8 ? (total + 255) / 256 : 148 * 8);
    gather_interleave_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>((const uint4 *)src, (uint4 *)dst, ranks, rows, row_bytes / 16);
    TTB_LAUNCH_CHECK("gather_interleave");
    return TTB_OK;
}

}  // extern "C"
