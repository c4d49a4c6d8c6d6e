// tl_internal.h -- types shared by the C-ABI layer (tl_api.cpp) and the kernel launchers (*.cu).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/tensilelite.h"

namespace tl {

// ---- error reporting ------------------------------------------------------------------------------
void set_error(const std::string& msg);
tl_status fail(tl_status st, const std::string& msg);
tl_status cuda_fail(cudaError_t e, const char* what);
#define TL_CUDA_TRY(call)                                  \
    do {                                                   \
        cudaError_t e_ = (call);                           \
        if (e_ != cudaSuccess) return ::tl::cuda_fail(e_, #call); \
    } while (0)

// ceil(log2 k)
inline int log2_ceil(int64_t k)
{
    int l = 0;
    while ((int64_t(1) << l) < k) ++l;
    return l;
}

inline int dtype_bytes(int dt)
{
    switch (dt) {
    case TL_DTYPE_FP32: return 4;
    case TL_DTYPE_FP16: return 2;
    case TL_DTYPE_BF16: return 2;
    case TL_DTYPE_FP8_E4M3: return 1;
    default: return 0;
    }
}

// ---- tcgen05 GEMM launch description ----------------------------------------------------------------
constexpr int kTcMaxStages = 8;
constexpr int kTcTileN = 128;          // tcgen05 M extent: problem n rows on TMEM lanes
constexpr int kTcRowBytes = 128;       // one swizzle row: depth_u * element size
constexpr int kTcEpiStageBytes = 4 * 32 * 128;   // output staging of 4 epilogue warps
constexpr size_t kTcMaxSmem = 227 * 1024;        // dynamic shared memory a CTA may ask for
// kernel variants: plain accumulation, promoted accumulation, promoted products of shared pieces
constexpr int kModePlain = 0, kModePromo = 1, kModePieces = 2;
// warp 0 TMA, warp 1 MMA, then eight, four or sixteen epilogue warps
constexpr int tc_threads(int mode) { return mode == kModePromo ? 192 : (mode == kModePieces ? 576 : 320); }
// The fp32-split products run with shared pieces (kModePieces) on a promoted CTA pair of 128-column tiles,
// the default solution's: two of them side by side, each piece of A and B loaded once per k-block instead
// of once per product (bf16x3 needs 2 loads for 3 products, bf16x6 3 for 6) and 256-column MMAs, 1536 / 3072
// clocks per k-block against 2 x 1035 / 2070.  Only where the 128-column tiles are more than one wave of
// pairs: below that the wide tile leaves pairs idle (512 x 4096 x 1024: bf16x3 41 us against 36).  Not for an
// explicit split-k, which asks for the tile as it stands.  The ring has kTcSharedStages slots whatever depth
// the solution names: its depth is for the 24 KB stages of single products, and says nothing about which
// loads to make.
constexpr int kTcSharedStages = 6;
inline bool tc_shared_pieces(int pieces, int cg, int bm, int promote_k, int split_k, int64_t M, int64_t N, int64_t batch,
                             int sm_count)
{
    const int64_t tiles = ((M + 127) / 128) * ((N + 255) / 256) * batch;
    return pieces > 1 && cg == 2 && bm == 128 && promote_k > 0 && split_k == 1 && M > 128 && 2 * tiles > sm_count;
}

// Magnitudes of the two operands of a split-precision product, gathered by the split pass: the bits of
// the largest |x| and the complement of the bits of the smallest nonzero |x| (0: none), of A then of B.
struct SplitRange {
    uint32_t max_a, inv_min_a, max_b, inv_min_b;
};
// Whether three bf16 pieces stand for these operands as exactly as fp32 does in a sum of 2^klog2
// products: everything finite and still so when rounded to bf16 (from 0x7f7f8000 on a finite value rounds
// to infinity), no piece below bf16's normal range, no product of pieces (down to 2^-16 of its operands'
// product) below fp32's, and no sum beyond its largest value.
#ifdef __CUDACC__
__host__ __device__
#endif
inline bool split_range_ok(const SplitRange& r, int klog2)
{
    if (r.max_a >= 0x7f7f8000u || r.max_b >= 0x7f7f8000u) return false;
    const int ea = static_cast<int>(r.max_a >> 23), eb = static_cast<int>(r.max_b >> 23);
    const int ma = r.inv_min_a ? static_cast<int>((~r.inv_min_a) >> 23) : 127;
    const int mb = r.inv_min_b ? static_cast<int>((~r.inv_min_b) >> 23) : 127;
    return ea + eb - 254 + 2 + klog2 <= 126 && ma >= 27 && mb >= 27 && ma + mb - 254 >= -100;
}

// One operand's TMA view: K-major (rows x k, k contiguous) or MN-major (k rows of contiguous rows).
struct TcOperand {
    const void* ptr;
    int64_t rows;      // n (opN = problem B) or m (opM = problem A)
    int64_t ld;        // elements
    int64_t batch_stride;
    int mn_major;      // 1: rows contiguous in memory
};

// Per-problem table entry for the grouped kernel (device memory; CUtensorMap members fix the alignment).
struct TcGroupEntry {   // aligned like CUtensorMap
    CUtensorMap tmN;   // problem B view
    CUtensorMap tmM;   // problem A view
    void* D;
    const void* C;
    int64_t ldd, ldc;
    int32_t M, N, K;
    int32_t tiles_m, tiles_n;
    float alpha, beta;
    int32_t vec;         // D and C consist of whole aligned 16-byte vectors
};

struct TcLaunch {
    // operands
    int in_dtype;            // FP16 / BF16 / FP8_E4M3 (BF16 for the fp32 split paths)
    int out_dtype;
    int out_trunc;
    TcOperand opN[3], opM[3];  // operand pieces: [0] the operand (or its bf16 head), [1..2] residuals
    int pieces;              // 1 plain, 2 = bf16x3 (3 products), 3 = bf16x6 (6 products)
    int64_t M, N, K, batch;
    void* D;
    const void* C;
    int64_t ldd, ldc, stride_d, stride_c;
    float alpha, beta;
    // solution
    int bm;                  // tile along m (tcgen05 N): 64..256
    int stages;
    int split_k;
    int raster;
    int ctas;
    int promote_k;           // k elements per TMEM accumulation chain of the A0*B0 product (0: whole k)
    int cg;                  // 1: one CTA per 128-row tile; 2: a CTA pair per 256-row tile
    // runtime
    int* err;
    uint64_t timeout_ns;
    float* workspace;        // split-k partials
    size_t workspace_bytes;
    int* counters;           // split-k arrival counters (zeroed, self-resetting)
    size_t counters_len;
    int tail_split;          // 0 auto, 1 off, S: k splits of the last partial wave's tiles
    int sm_count;
    // fused epilogue: D = act(alpha*acc + beta*C + bias[m]); max |D| into *epi_amax
    const void* epi_bias;
    float* epi_amax;
    float epi_dscale;        // fp8 outputs: multiplied in before the E4M3 rounding
    int epi_bias_dtype;
    int epi_act;
    int epi_on;
    int debug_flags;         // tl_gemm_solution.debug_flags (TL_DEBUG_SKIP_LOADS)
    unsigned long long* trace;   // device timeline (tl_set_trace) or null
    int64_t trace_bytes;
    int out_t;               // D and C hold the transpose of this launch's output (NN run as TT)
    const SplitRange* range; // split products: run only if split_range_ok (device memory), or null
    int shared_gpu;          // launches like this one may run beside it on other streams: no CTA relies on another's
                             // start (the counters are this launch's own, zeroed)
};

// How the splits of a tile are summed: 0 by the last one to arrive, 1 by all of them, a share each, once all have
// arrived, 2 the same without relying on it.  All of a launch's split units have to be resident at
// once for 1: where launches on other streams may hold part of the SMs, two of them, each partly resident,
// would wait until the limit for CTAs that cannot start.
inline int tc_par_reduce(int64_t split_units, int64_t bal_kb, int64_t workers, int shared_gpu)
{
    return split_units > 0 && bal_kb == 0 && split_units <= workers ? (shared_gpu ? 2 : 1) : 0;
}

// Dynamic shared memory of one CTA staging bm_cta m-rows per stage (bm / 2 for a CTA pair).
size_t tc_smem_bytes(int bm_cta, int stages);
// Whether the columns (of `rows` elements) of D, and of C where there is one, are whole aligned 16-byte
// vectors.
bool tc_vec_output(int out_dtype, int64_t rows, const void* D, int64_t ldd, const void* C, int64_t ldc, int64_t batch,
                   int64_t stride_d, int64_t stride_c);
// Persistent workers (CTAs, or co-resident clusters of `cl` CTAs) a tensor-core launch gets.
int tc_workers(int in_dtype, int out_dtype, int cl, int bm, int stages, int sm_count);
tl_status tc_gemm_launch(const TcLaunch& L, cudaStream_t stream, int64_t* launches);
// Checks a tcgen05 GEMM and fills its launch description without allocating anything; the caller
// provides err, workspace and counters (sizes reported in ws_bytes / counter_count).
tl_status plan_tc_noalloc(int device, int sm_count, size_t smem_optin, const tl_gemm_problem* prob,
                          const tl_gemm_solution* sol, void* D, const void* C, const void* A, const void* B,
                          TcLaunch* L, size_t* ws_bytes, size_t* counter_count);

// Grouped: build per-problem entries (host) and launch over a device table.
struct TcGroupLaunch {
    int in_dtype, out_dtype, out_trunc;
    int n_mn_major, m_mn_major;
    const TcGroupEntry* d_entries;   // device
    const int4* d_units;             // device, one entry per work unit: {problem, tile row, tile column, k-blocks}
    int count;
    int64_t total_tiles;
    int bm, stages, ctas;
    int cg;                          // 1 or 2 (CTA pair)
    int* err;
    uint64_t timeout_ns;
    int sm_count;
};
tl_status tc_encode_operand(CUtensorMap* tm, int in_dtype, const TcOperand& op, int64_t K, int64_t batch,
                            int box_rows);
tl_status tc_grouped_launch(const TcGroupLaunch& G, cudaStream_t stream, int64_t* launches);

// ---- SIMT GEMM -----------------------------------------------------------------------------------
struct SimtLaunch {
    int a_dtype, out_dtype, out_trunc;
    int trans_a, trans_b;
    int64_t M, N, K, batch;
    const void* A; const void* B; const void* C; void* D;
    int64_t lda, ldb, ldc, ldd, sa, sb, sc, sd;
    float alpha, beta;   // alpha already multiplied by fp8 scales
    const SplitRange* unless = nullptr;   // run only if split_range_ok fails (device memory), or null
};
tl_status simt_gemm_launch(const SimtLaunch& L, cudaStream_t stream, int64_t* launches);

// ---- auxiliary kernels ------------------------------------------------------------------------------
// x = p0 + p1 (+ p2): each piece the bf16 rounding (RNE) of what the previous pieces leave; p2 may be null.
// The pieces have their own leading dimension and batch stride.  One launch per matrix.
struct SplitOperand {
    const float* src;
    int64_t rows, cols, ld, batch, batch_stride;
    uint16_t* p[3];
    int64_t pld, p_batch_stride;
};
// `range`, if given, receives the operands' magnitudes (zeroed by the caller).
tl_status aux_split_bf16(const SplitOperand* ops, int count, int pieces, SplitRange* range, cudaStream_t s,
                         int64_t* launches);
// 16-bit matrices copied to columns that start on 128-byte lines (pld a multiple of 64 elements; the
// elements between rows and the next multiple of eight are zeroed).  One launch for all of them.
struct PadOperand {
    const uint16_t* src;
    int64_t rows, cols, ld, batch, batch_stride;
    uint16_t* dst;
    int64_t pld, p_batch_stride;
};
tl_status aux_pad16(const PadOperand* ops, int count, cudaStream_t s, int64_t* launches);
// Eight 16-bit elements that start on an even address, as four words: half(i) reads element i, word(i) elements
// i and i + 1 (4-byte aligned).  `odd`: the first starts in the middle of a word.  Nothing outside the eight
// is read.
template <class Half, class Word>
#ifdef __CUDACC__
__device__ __forceinline__
#else
inline
#endif
void load_eight16(bool odd, Half half, Word word, uint32_t (&v)[4])
{
    if (!odd) {
        for (int e = 0; e < 4; ++e) v[e] = word(2 * e);
        return;
    }
    const uint32_t first = half(0), w0 = word(1), w1 = word(3), w2 = word(5), last = half(7);
    v[0] = first | (w0 << 16);
    v[1] = (w0 >> 16) | (w1 << 16);
    v[2] = (w1 >> 16) | (w2 << 16);
    v[3] = (w2 >> 16) | (last << 16);
}
// The way back: rows x cols of `dst` (pld, p_batch_stride) to `src`'s place; the gaps stay as they are.
tl_status aux_unpad16(const PadOperand& op, cudaStream_t s, int64_t* launches);
// Per-tensor E4M3 quantisation: *amax_dev = max |x|, dst = e4m3(x * 448 / amax), *scale_out_dev = amax / 448.
tl_status aux_quantize_e4m3(int src_dtype, const void* src, int64_t n, float* amax_dev, uint8_t* dst,
                            float* scale_out_dev, cudaStream_t s, int64_t* launches);
tl_status aux_error_norms(int dtype_d, const void* D, int64_t ldd, const double* R, const double* W, int64_t ldr,
                          int64_t m, int64_t n, double* out_dev, cudaStream_t s, int64_t* launches);
tl_status aux_fill_pattern(int dtype, void* dst, int64_t count, float code, cudaStream_t s, int64_t* launches);
tl_status aux_scale_c(int out_dtype, int out_trunc, void* D, int64_t ldd, int64_t sd, const void* C, int64_t ldc,
                      int64_t sc, int64_t M, int64_t N, int64_t batch, float beta, cudaStream_t s,
                      int64_t* launches);

}  // namespace tl
