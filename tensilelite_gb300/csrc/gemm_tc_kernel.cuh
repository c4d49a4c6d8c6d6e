// The tcgen05 GEMM kernel template and its launch templates, shared by the translation unit with the
// host code (gemm_tc.cu) and the instance units the build generates (one per operand kind, cluster
// size and epilogue variant, compiled in parallel).  See gemm_tc.cu for the design notes.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <type_traits>
#include "ptx.cuh"
#include "tl_internal.h"

namespace tl {
namespace tc {


struct TcKernelParams {
    CUtensorMap tmN[3], tmM[3];   // split-precision pieces 0..2 (piece 0 = the operand itself)
    int vec;                      // D (and C, with beta) consist of whole aligned 16-byte vectors: whole
                                  // tiles leave through shared memory in full lines
    int epi_bufs;                 // output staging in units of kTcEpiStageBytes (1 or 2)
    // fused epilogue (kernels instantiated with EPI): D = act(alpha*acc + beta*C + bias[m]), and
    // max |D| into *epi_amax
    const void* epi_bias;
    float* epi_amax;
    float epi_dscale;             // fp8 outputs: values are multiplied by this before the E4M3 rounding
    int epi_bias_dtype;
    int epi_act;
    int epi_on;
    int par_reduce;               // every split unit runs in the first round: the splits of a tile
                                  // wait for each other and reduce one share of it each; 2: beside other
                                  // launches (split_finish)
    unsigned long long hand_over_ns;      // par_reduce 2: how long a split waits for the others
    const TcGroupEntry* group;
    const int4* group_units;       // per work unit: {problem, tile row, tile column, k-blocks}
    void* D;
    const void* C;
    int64_t ldd, ldc, stride_d, stride_c;
    int M, N, K, batch;
    float alpha, beta;
    int bm, stages, split_k, raster;
    int tile_rows;                // n rows per tile: 128 (one CTA) or 256 (CTA pair)
    int nterms;                   // stages per k-block: 1, the 3 / 6 products of the fp32 split, or its 2 / 3
                                  // pieces (kModePieces)
    uint8_t term_n[8], term_m[8]; // piece of B / of A in each stage (the last is piece 0 of both)
    int pieces_mode;              // kModePieces
    int promote_kb;               // >0: the A0*B0 product restarts its TMEM chain every promote_kb
                                  // k-blocks; the epilogue adds each chain into fp32 registers
    int promote_half;             // two A0*B0 chains per k-block (16-bit pieces, promote_kb 1)
    int small_chains;             // kModePieces: the small products' accumulator starts anew every so many chains
    int tiles_m, tiles_n;
    int narrow;                   // work units, tiles and split k-block products fit 32 bits, no balanced split
    int64_t total_work;
    int64_t split_units;          // work units below this are k-slices of the first split_tiles tiles
    int64_t split_tiles;          // tiles split along k; the rest are whole
    int tail_split;               // k slices of each split tile (balanced: the workspace slab stride)
    // balanced split (bal_kb > 0): the split tiles' bal_kb k-blocks are cut into bal_workers equal
    // contiguous ranges, one per worker; unit w < 2 * bal_stride is piece w / bal_stride (a range
    // spans at most two tiles) of worker w % bal_stride
    int64_t bal_kb;
    int bal_workers;
    int bal_stride;
    int num_kb;
    uint32_t idesc;
    uint32_t n_lbo, m_lbo, n_kstep, m_kstep;
    int n_mn_major, m_mn_major;
    int out_trunc;
    float* ws;
    int* counters;
    int* err;
    unsigned long long timeout_ns;
    int debug_skip_loads;         // TL_DEBUG_SKIP_LOADS: the producer issues no copies (timeout-path test)
    unsigned long long* trace;    // device timeline, TL_TRACE_SLOTS words per CTA, or null
    const SplitRange* range;      // promoted kernels: run only if split_range_ok(*range, range_klog2), or null
    int range_klog2;
    int out_t;                    // D and C are the transpose of the kernel's output: element (m, n)
                                  // at n + m * ld (an NN problem run as its transposed TT product)
};

// Timeline stamp of event `slot` for this CTA (tl_set_trace): the SM cycle counter.
__device__ __forceinline__ void trace_mark(const TcKernelParams& p, int slot)
{
    if (p.trace != nullptr) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%clock64;" : "=l"(t) :: "memory");
        p.trace[static_cast<size_t>(blockIdx.x) * TL_TRACE_SLOTS + slot] = t;
    }
}
__device__ __forceinline__ void trace_put(const TcKernelParams& p, int slot, unsigned long long v)
{
    if (p.trace != nullptr) p.trace[static_cast<size_t>(blockIdx.x) * TL_TRACE_SLOTS + slot] = v;
}
__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t) :: "memory");
    return t;
}

struct TileJob {
    const void* tmN;
    const void* tmM;
    int vec;                      // D and C in 16-byte vectors (TcKernelParams::vec)
    void* D;
    const void* C;
    int64_t ldd, ldc;
    int M, N;
    float alpha, beta;
    int b, n0, m0;
    int kb0, kb1;
    int split, nsplit;            // this unit's k split and the tile's number of splits
    int out_t;                    // transposed output (TcKernelParams::out_t)
    int64_t slot;                 // split tiles: index of the tile's workspace slabs and counter
};

// Grouped launches: the unit-table entry of work unit w (a zero entry past the end or without a group).
template <bool GROUP>
__device__ __forceinline__ int4 load_unit(const TcKernelParams& p, int64_t w)
{
    if (!GROUP || w >= p.total_work) return make_int4(0, 0, 0, 0);
    return __ldg(p.group_units + w);
}

// Where a work unit lies: tile and its coordinates, its k split and k-blocks.
struct UnitPos {
    int64_t tile;
    int b, in, jm, kb0, kb1, split, nsplit;
};

// The decode of balanced-split units and of launches beyond 32 bits, out of line: 64-bit divisions
// take hundreds of instructions, and inlined at every use they made the kernel 200 KB of code, whose
// fetches stalled every role (ncu: 8 of 10 cycles between a warp's instructions).
static __device__ __noinline__ void unit_pos_wide(const TcKernelParams& p, int64_t w, UnitPos& u)
{
    if (p.bal_kb > 0 && w < 2 * static_cast<int64_t>(p.bal_stride)) {
        // balanced split: worker `wk` owns k-blocks [s0, s1) of the split tiles laid end to end;
        // piece 0 is the part in its first tile, piece 1 the rest (possibly empty)
        const int64_t wk = w % p.bal_stride, piece = w / p.bal_stride;
        const int64_t R = p.bal_kb, Wb = p.bal_workers, nkb = p.num_kb;
        int64_t a = 0, e = 0;
        if (wk < Wb) {
            const int64_t s0 = wk * R / Wb, s1 = (wk + 1) * R / Wb;
            const int64_t cut = min(s1, (s0 / nkb + 1) * nkb);
            a = piece == 0 ? s0 : cut;
            e = piece == 0 ? cut : s1;
        }
        if (a >= e) {
            u.tile = 0;                    // empty unit: every role skips it
            u.kb0 = u.kb1 = 0;
            u.split = 0;
            u.nsplit = 1;
        } else {
            u.tile = a / nkb;
            u.kb0 = static_cast<int>(a - u.tile * nkb);
            u.kb1 = static_cast<int>(e - u.tile * nkb);
            // the workers covering this tile: the one holding its first and its last k-block
            const int64_t first = ((u.tile * nkb + 1) * Wb - 1) / R;
            const int64_t last = (((u.tile + 1) * nkb) * Wb - 1) / R;
            u.nsplit = static_cast<int>(last - first + 1);
            u.split = static_cast<int>(wk - first);
        }
    } else if (w < p.split_units) {
        u.nsplit = p.tail_split;
        u.tile = w / p.tail_split;
        u.split = static_cast<int>(w % p.tail_split);
        u.kb0 = static_cast<int>((static_cast<int64_t>(u.split) * p.num_kb) / u.nsplit);
        u.kb1 = static_cast<int>((static_cast<int64_t>(u.split + 1) * p.num_kb) / u.nsplit);
    } else {
        u.tile = p.split_tiles + (w - p.split_units);
        u.split = 0;
        u.nsplit = 1;
        u.kb0 = 0;
        u.kb1 = p.num_kb;
    }
    const int64_t tpb = static_cast<int64_t>(p.tiles_m) * p.tiles_n;
    u.b = static_cast<int>(u.tile / tpb);
    const int64_t t = u.tile % tpb;
    if (p.raster > 0) {
        const int64_t group_tiles = static_cast<int64_t>(p.raster) * p.tiles_m;
        const int64_t g = t / group_tiles;
        const int first_n = static_cast<int>(g * p.raster);
        const int gsize = min(p.raster, p.tiles_n - first_n);
        const int64_t r = t % group_tiles;
        u.in = first_n + static_cast<int>(r % gsize);
        u.jm = static_cast<int>(r / gsize);
    } else {
        u.in = static_cast<int>(t / p.tiles_m);
        u.jm = static_cast<int>(t % p.tiles_m);
    }
}

// Every index fits 32 bits (host-checked) and no balanced split: 32-bit divisions only, on the path
// between the launch and the first load.
__device__ __forceinline__ void unit_pos_narrow(const TcKernelParams& p, uint32_t w, UnitPos& u)
{
    const uint32_t nkb = static_cast<uint32_t>(p.num_kb);
    uint32_t tile;
    if (w < static_cast<uint32_t>(p.split_units)) {
        // split tiles come first, so the last arriver's reduction overlaps later whole tiles
        const uint32_t ts = static_cast<uint32_t>(p.tail_split);
        tile = w / ts;
        const uint32_t split = w - tile * ts;
        u.split = static_cast<int>(split);
        u.nsplit = static_cast<int>(ts);
        u.kb0 = static_cast<int>((split * nkb) / ts);
        u.kb1 = static_cast<int>(((split + 1) * nkb) / ts);
    } else {
        tile = static_cast<uint32_t>(p.split_tiles) + (w - static_cast<uint32_t>(p.split_units));
        u.split = 0;
        u.nsplit = 1;
        u.kb0 = 0;
        u.kb1 = p.num_kb;
    }
    u.tile = tile;
    uint32_t t = tile;
    u.b = 0;
    if (p.batch > 1) {
        const uint32_t tpb = static_cast<uint32_t>(p.tiles_m) * static_cast<uint32_t>(p.tiles_n);
        const uint32_t ub = tile / tpb;
        u.b = static_cast<int>(ub);
        t = tile - ub * tpb;
    }
    if (p.raster > 0) {
        const uint32_t group_tiles = static_cast<uint32_t>(p.raster) * static_cast<uint32_t>(p.tiles_m);
        const uint32_t g = t / group_tiles;
        const int first_n = static_cast<int>(g * static_cast<uint32_t>(p.raster));
        const uint32_t gsize = static_cast<uint32_t>(min(p.raster, p.tiles_n - first_n));
        const uint32_t r = t - g * group_tiles;
        const uint32_t rq = r / gsize;
        u.in = first_n + static_cast<int>(r - rq * gsize);
        u.jm = static_cast<int>(rq);
    } else {
        const uint32_t q = t / static_cast<uint32_t>(p.tiles_m);
        u.in = static_cast<int>(q);
        u.jm = static_cast<int>(t - q * static_cast<uint32_t>(p.tiles_m));
    }
}

// Without a group the problem's fields stay in the kernel parameters (constant memory): only the
// unit's position is computed.
template <bool GROUP>
__device__ __forceinline__ void get_job(const TcKernelParams& p, int64_t w, const int4& u, TileJob& j)
{
    if constexpr (!GROUP) {
        UnitPos pos;
        if (p.narrow) unit_pos_narrow(p, static_cast<uint32_t>(w), pos);
        else unit_pos_wide(p, w, pos);
        j.tmN = &p.tmN[0];
        j.tmM = &p.tmM[0];
        j.vec = p.vec;
        j.D = static_cast<char*>(p.D);
        j.C = p.C;
        j.ldd = p.ldd;
        j.ldc = p.ldc;
        j.M = p.M;
        j.N = p.N;
        j.alpha = p.alpha;
        j.beta = p.beta;
        j.b = pos.b;
        j.n0 = pos.in * p.tile_rows;
        j.m0 = pos.jm * p.bm;
        j.kb0 = pos.kb0;
        j.kb1 = pos.kb1;
        j.split = pos.split;
        j.nsplit = pos.nsplit;
        j.out_t = p.out_t;
        j.slot = pos.tile;             // split tiles are 0 .. split_tiles-1
    } else {
        // grouped: the unit's problem and tile come from the plan's unit table (loaded ahead by
        // the caller); only the epilogue reads the problem's entry
        const TcGroupEntry& e = p.group[u.x];
        j.tmN = &e.tmN;
        j.tmM = &e.tmM;
        j.vec = e.vec;
        j.D = e.D;
        j.C = e.C;
        j.ldd = e.ldd;
        j.ldc = e.ldc;
        j.M = e.M;
        j.N = e.N;
        j.alpha = e.alpha;
        j.beta = e.beta;
        j.b = 0;
        j.n0 = u.y * p.tile_rows;
        j.m0 = u.z * p.bm;
        j.kb0 = 0;
        j.kb1 = u.w;
        j.split = 0;
        j.nsplit = 1;
        j.out_t = 0;
        j.slot = 0;
    }
}

// Whether a promoted launch runs at all: its operands' magnitudes, known once the split pass before it has
// completed, are within what the pieces can stand for.
template <int MODE>
__device__ __forceinline__ bool launch_live(const TcKernelParams& p)
{
    if constexpr (MODE == kModePlain) return true;
    else return p.range == nullptr || split_range_ok(*p.range, p.range_klog2);
}

__device__ __forceinline__ void record_error(const TcKernelParams& p, volatile int* abort_flag, int code)
{
    *abort_flag = 1;
    atomicOr(p.err, code);
}

// ---- output conversion ------------------------------------------------------------------------------
template <typename TD> struct Out;
template <> struct Out<float> {
    __device__ static __forceinline__ float load(const void* base, int64_t idx)
    { return __ldg(static_cast<const float*>(base) + idx); }
    __device__ static __forceinline__ void store(void* base, int64_t idx, float v, int)
    { static_cast<float*>(base)[idx] = v; }
    static constexpr int kBytes = 4;
};
template <> struct Out<__half> {
    __device__ static __forceinline__ float load(const void* base, int64_t idx)
    { return __half2float(static_cast<const __half*>(base)[idx]); }
    __device__ static __forceinline__ void store(void* base, int64_t idx, float v, int)
    { static_cast<__half*>(base)[idx] = __float2half_rn(v); }
    static constexpr int kBytes = 2;
};
template <> struct Out<__nv_bfloat16> {
    __device__ static __forceinline__ float load(const void* base, int64_t idx)
    { return __bfloat162float(static_cast<const __nv_bfloat16*>(base)[idx]); }
    __device__ static __forceinline__ void store(void* base, int64_t idx, float v, int trunc)
    {
        if (trunc) static_cast<uint16_t*>(base)[idx] = static_cast<uint16_t>(__float_as_uint(v) >> 16);
        else static_cast<__nv_bfloat16*>(base)[idx] = __float2bfloat16_rn(v);
    }
    static constexpr int kBytes = 2;
};

// E4M3 outputs (fused-epilogue kernels; beta must be 0): round to nearest even, saturating to +-448.
template <> struct Out<__nv_fp8_e4m3> {
    __device__ static __forceinline__ float load(const void* base, int64_t idx)
    {
        return __half2float(__half(__nv_cvt_fp8_to_halfraw(static_cast<const __nv_fp8_storage_t*>(base)[idx], __NV_E4M3)));
    }
    __device__ static __forceinline__ void store(void* base, int64_t idx, float v, int)
    { static_cast<__nv_fp8_storage_t*>(base)[idx] = __nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3); }
    static constexpr int kBytes = 1;
};

// Four values as four E4M3 bytes in one word (first value in the low byte).
__device__ __forceinline__ uint32_t pack4_e4m3(float a, float b, float c, float d)
{
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
    const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3);
    return (lo & 0xffffu) | (hi << 16);
}

// The quantisation scale of fp8 outputs (applied after the epilogue function and the amax).
template <typename TD>
__device__ __forceinline__ float out_scale(const TcKernelParams& p, float o)
{
    if constexpr (sizeof(TD) == 1) return o * p.epi_dscale;
    else return o;
}

__device__ __forceinline__ uint32_t pack2(float a, float b, int is_half, int trunc)
{
    if (is_half) {
        __half2 h = __floats2half2_rn(a, b);
        return *reinterpret_cast<uint32_t*>(&h);
    }
    if (trunc) return (__float_as_uint(a) >> 16) | (__float_as_uint(b) & 0xffff0000u);
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}

__device__ __forceinline__ void unpack2(uint32_t w, int is_half, float& a, float& b)
{
    if (is_half) {
        __half2 h = *reinterpret_cast<__half2*>(&w);
        float2 f = __half22float2(h);
        a = f.x;
        b = f.y;
    } else {
        a = __uint_as_float(w << 16);
        b = __uint_as_float(w & 0xffff0000u);
    }
}

// Ragged edges, unaligned matrices and transposed outputs, element by element and out of line (the
// unrolled code of each use took more instruction memory than everything else).
template <typename TD>
__device__ __noinline__ void load_elements(const void* base, int64_t idx, int64_t step, int count, float* out)
{
#pragma unroll 4
    for (int i = 0; i < count; ++i) out[i] = Out<TD>::load(base, idx + i * step);
}
template <typename TD>
__device__ __noinline__ void store_elements(void* base, int64_t idx, int64_t step, int count, const float* v, float scale,
                                            int trunc)
{
#pragma unroll 4
    for (int i = 0; i < count; ++i) Out<TD>::store(base, idx + i * step, sizeof(TD) == 1 ? v[i] * scale : v[i], trunc);
}

// The bias of rows m .. m+W-1 (rows past M: 0), every load in flight at once.
template <int W>
__device__ __forceinline__ void load_bias(const TcKernelParams& p, int M, int m, float (&b)[W])
{
    const int es = p.epi_bias_dtype == TL_DTYPE_FP32 ? 4 : 2;
    const char* src = static_cast<const char*>(p.epi_bias) + static_cast<int64_t>(m) * es;
    if ((W % 8 == 0 || es == 4) && m + W <= M && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
        if (es == 4) {
#pragma unroll
            for (int q = 0; q < W / 4; ++q) {
                const float4 f = __ldg(reinterpret_cast<const float4*>(src) + q);
                b[4 * q] = f.x;
                b[4 * q + 1] = f.y;
                b[4 * q + 2] = f.z;
                b[4 * q + 3] = f.w;
            }
        } else {
            const int is_half = p.epi_bias_dtype == TL_DTYPE_FP16 ? 1 : 0;
#pragma unroll
            for (int q = 0; q < W / 8; ++q) {
                const uint4 w = __ldg(reinterpret_cast<const uint4*>(src) + q);
                unpack2(w.x, is_half, b[8 * q], b[8 * q + 1]);
                unpack2(w.y, is_half, b[8 * q + 2], b[8 * q + 3]);
                unpack2(w.z, is_half, b[8 * q + 4], b[8 * q + 5]);
                unpack2(w.w, is_half, b[8 * q + 6], b[8 * q + 7]);
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < W; ++i) {
            b[i] = 0.f;
            if (m + i < M) {
                if (es == 4) b[i] = __ldg(reinterpret_cast<const float*>(src) + i);
                else if (p.epi_bias_dtype == TL_DTYPE_FP16) b[i] = __half2float(reinterpret_cast<const __half*>(src)[i]);
                else b[i] = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(src)[i]);
            }
        }
    }
}

// The bias of rows m, m + 32, ... (one per lane of a warp and chunk; rows past M: 0).
template <int N>
__device__ __forceinline__ void lane_bias(const TcKernelParams& p, int M, int m, float (&b)[N])
{
#pragma unroll
    for (int t = 0; t < N; ++t) {
        const int r = m + 32 * t;
        b[t] = 0.f;
        if (p.epi_bias != nullptr && r < M) {
            if (p.epi_bias_dtype == TL_DTYPE_FP32) b[t] = __ldg(static_cast<const float*>(p.epi_bias) + r);
            else if (p.epi_bias_dtype == TL_DTYPE_FP16) b[t] = __half2float(static_cast<const __half*>(p.epi_bias)[r]);
            else b[t] = __bfloat162float(static_cast<const __nv_bfloat16*>(p.epi_bias)[r]);
        }
    }
}

// Fused epilogue of W output values at rows m..: + bias b, activation (1 relu, 2 gelu with the tanh
// approximation, 3 silu), and this thread's running max |value| over the stored ones (`row_ok`: the
// column n is stored).  The tests on the kind sit outside the element loops, the bias comes in
// registers, and the activation's code is there once: a launch that does not follow another at once
// fetches its instructions anew, ~500 clocks per 128 bytes of straight-line code, and with a bias load, three
// type tests and both activations unrolled over 32 elements the two chunks of a 32-row linear layer
// took 23000 clocks (11 us).  gelu(x) = x (1 + tanh u) / 2 = x / (1 + exp(-2u)): the form of silu,
// without the cancellation of 1 + tanh at negative x.
// FULL, for fp32 outputs: the quotient without an overflow and corrected by its residual, as a correctly
// rounded division's last step is (Markstein 1990).  The quick quotient is half a unit in the last place
// worse (silu of N(0, 1) products, relative 2-norm 5.3e-8 against 4.2e-8), which narrower outputs round
// away; there it saves 7 % of a 4096 x 1024 x 4096 layer.  A plain division's slow path costs the 32-row layer 10 us.
template <int W, bool FULL>
__device__ __forceinline__ void epi_apply(const TcKernelParams& p, int M, int m, bool row_ok, const float (&b)[W],
                                          float (&o)[W], float& amax)
{
    if (p.epi_bias != nullptr) {
#pragma unroll
        for (int i = 0; i < W; ++i) o[i] += b[i];
    }
    if (p.epi_act == 1) {
#pragma unroll
        for (int i = 0; i < W; ++i) o[i] = fmaxf(o[i], 0.0f);
    } else if (p.epi_act >= 2) {
        const bool gelu = p.epi_act == 2;
        // two elements at a time, the values rotated through the registers: one copy of the code
#pragma unroll 1
        for (int i = 0; i < W; i += 2) {
            float r[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float x = o[e];
                const float t = gelu ? 1.5957691216057308f * fmaf(0.044715f * x * x, x, x) : x;
                if constexpr (FULL) {
                    const float z = expf(-fabsf(t)), y = 1.0f + z, num = t < 0.0f ? x * z : x;
                    const float inv = __fdividef(1.0f, y), q = num * inv;
                    r[e] = fabsf(q) < __int_as_float(0x7f800000) ? fmaf(fmaf(-q, y, num), inv, q) : q;
                } else {
                    r[e] = __fdividef(x, 1.0f + expf(-t));   // 2 ulp; an infinite divisor gives 0 without a slow path
                }
            }
#pragma unroll
            for (int k = 0; k < W - 2; ++k) o[k] = o[k + 2];
            o[W - 2] = r[0];
            o[W - 1] = r[1];
        }
    }
    if (p.epi_amax != nullptr) {
#pragma unroll
        for (int i = 0; i < W; ++i)
            if (row_ok && m + i < M) amax = fmaxf(amax, fabsf(o[i]));
    }
}

// C for one chunk of W outputs, loaded ahead of its use (the epilogue keeps the next chunk's loads in
// flight while it finishes the current one).  16-bit outputs occupy cw[0..W/2-1] as packed pairs.
template <typename TD, int W>
__device__ __forceinline__ void load_c_chunk(const TileJob& j, int64_t base_c, int m, uint32_t (&cw)[W])
{
    if constexpr (sizeof(TD) == 1) return;        // fp8 outputs take beta == 0: no C
    if (!(j.beta != 0.0f && j.C != nullptr) || m >= j.M) return;
    const char* cptr = static_cast<const char*>(j.C) + (base_c + m) * Out<TD>::kBytes;
    if (!j.out_t && m + W <= j.M && (reinterpret_cast<uintptr_t>(cptr) & 15) == 0) {
        constexpr int nvec = W * static_cast<int>(sizeof(TD)) / 16;
#pragma unroll
        for (int q = 0; q < nvec; ++q) {
            const uint4 w = __ldg(reinterpret_cast<const uint4*>(cptr) + q);
            cw[4 * q] = w.x;
            cw[4 * q + 1] = w.y;
            cw[4 * q + 2] = w.z;
            cw[4 * q + 3] = w.w;
        }
    } else {
        float c[W];
        load_elements<TD>(j.C, base_c + m * (j.out_t ? j.ldc : 1), j.out_t ? j.ldc : 1, min(W, j.M - m), c);
#pragma unroll
        for (int i = 0; i < W; ++i) {
            if constexpr (sizeof(TD) == 4) {
                cw[i] = __float_as_uint(c[i]);
            } else {
                // repack as the vector path does: element i in the low (even) / high (odd) half
                const uint32_t bits = std::is_same<TD, __half>::value
                                          ? static_cast<uint32_t>(__half_as_ushort(__float2half_rn(c[i])))
                                          : (__float_as_uint(c[i]) >> 16);
                if (i & 1) cw[i >> 1] |= bits << 16;
                else cw[i >> 1] = bits;
            }
        }
    }
}

// alpha*acc + beta*C for W outputs (C in registers from load_c_chunk), then the fused epilogue when
// EPI.  Rows past N and columns past M are computed but never stored: they stay out of the amax.
template <typename TD, bool EPI, int W>
__device__ __forceinline__ void finish_values(const TcKernelParams& p, float& amax, const TileJob& j, int m, bool row_ok,
                                              const uint32_t (&cw)[W], const float (&bias)[W], float (&o)[W])
{
    if constexpr (sizeof(TD) != 1) {
        if (j.beta != 0.0f && j.C != nullptr) {
#pragma unroll
            for (int i = 0; i < W; ++i) {
                float c;
                if constexpr (sizeof(TD) == 4) {
                    c = __uint_as_float(cw[i]);
                } else {
                    float lo, hi;
                    unpack2(cw[i >> 1], std::is_same<TD, __half>::value ? 1 : 0, lo, hi);
                    c = (i & 1) ? hi : lo;
                }
                o[i] = fmaf(j.alpha, o[i], j.beta * c);
            }
        } else {
#pragma unroll
            for (int i = 0; i < W; ++i) o[i] *= j.alpha;
        }
    } else {
#pragma unroll
        for (int i = 0; i < W; ++i) o[i] *= j.alpha;      // no C: fp8 outputs take beta == 0
    }
    if constexpr (EPI) epi_apply<W, sizeof(TD) == 4>(p, j.M, m, row_ok, bias, o, amax);
}

// W finished values as the output's bytes: W words for fp32, W/2 for 16-bit types, W/4 for fp8.
template <typename TD, int W>
__device__ __forceinline__ void pack_values(const TcKernelParams& p, const float (&o)[W], uint32_t* out)
{
    if constexpr (sizeof(TD) == 4) {
#pragma unroll
        for (int i = 0; i < W; ++i) out[i] = __float_as_uint(o[i]);
    } else if constexpr (sizeof(TD) == 1) {
#pragma unroll
        for (int q = 0; q < W / 4; ++q)
            out[q] = pack4_e4m3(out_scale<TD>(p, o[4 * q]), out_scale<TD>(p, o[4 * q + 1]), out_scale<TD>(p, o[4 * q + 2]),
                                out_scale<TD>(p, o[4 * q + 3]));
    } else {
        constexpr int is_half = std::is_same<TD, __half>::value ? 1 : 0;
        if (!is_half && p.out_trunc) {
#pragma unroll
            for (int h = 0; h < W / 2; ++h) out[h] = pack2(o[2 * h], o[2 * h + 1], 0, 1);
        } else {
#pragma unroll
            for (int h = 0; h < W / 2; ++h) out[h] = pack2(o[2 * h], o[2 * h + 1], is_half, 0);
        }
    }
}

// Finish a chunk of W consecutive outputs m.. of row n with C already in registers (load_c_chunk):
// v = alpha*acc + beta*C, the fused epilogue when EPI, convert, store (16-byte vectors, or element
// by element at ragged edges, unaligned D and for a transposed output, where element m + i lies at
// (m + i) * ld and a warp's 32 rows make one coalesced access per element).
template <typename TD, bool EPI, int W>
__device__ __forceinline__ void store_chunk_pre(const TcKernelParams& p, float& amax, const TileJob& j,
                                                int64_t base_d, int m, float (&o)[W], const uint32_t (&cw)[W])
{
    float bias[W];
    if constexpr (EPI) {
        if (p.epi_bias != nullptr) load_bias<W>(p, j.M, m, bias);
    }
    finish_values<TD, EPI, W>(p, amax, j, m, true, cw, bias, o);
    char* dptr = static_cast<char*>(j.D) + (base_d + m) * Out<TD>::kBytes;
    if (!j.out_t && m + W <= j.M && (reinterpret_cast<uintptr_t>(dptr) & 15) == 0) {
        constexpr int words = W * static_cast<int>(sizeof(TD)) / 4;
        uint32_t w[words];
        pack_values<TD, W>(p, o, w);
#pragma unroll
        for (int q = 0; q < words / 4; ++q)
            reinterpret_cast<uint4*>(dptr)[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
    } else {
        float v[W];
#pragma unroll
        for (int i = 0; i < W; ++i) v[i] = o[i];
        const int64_t step = j.out_t ? j.ldd : 1;
        store_elements<TD>(j.D, base_d + m * step, step, min(W, j.M - m), v, p.epi_dscale, p.out_trunc);
    }
}

// The same with C read here: all of the chunk's C before any of its D is written (D may be C itself).
template <typename TD, bool EPI, int W>
__device__ __forceinline__ void store_chunk(const TcKernelParams& p, float& amax, const TileJob& j, int64_t base_c,
                                           int64_t base_d, int m, float (&acc)[W])
{
    uint32_t cw[W];
    load_c_chunk<TD, W>(j, base_c, m, cw);
    store_chunk_pre<TD, EPI, W>(p, amax, j, base_d, m, acc, cw);
}

// A warp's access to 32 rows x 128 bytes of C or D, whole lines at a time: in step i lane L holds
// 16-byte unit L % 8 of row 4 i + L / 8 (eight lanes to a row's 128 bytes).  In shared memory unit u of
// row r sits at u ^ (r & 7).  Rows past `rows` and units past M are neither read nor written (M is a
// whole number of units).
template <typename TD>
struct LineAccess {
    static constexpr int EPU = 16 / static_cast<int>(sizeof(TD));
    int u, r0, rows, M;
    __device__ __forceinline__ LineAccess(int lane, int rows_, int M_) : u(lane & 7), r0(lane >> 3), rows(rows_), M(M_) {}
    __device__ __forceinline__ uint32_t at(int i) const
    {
        const int r = 4 * i + r0;
        return static_cast<uint32_t>(r * 128 + ((u ^ (r & 7)) * 16));
    }
    // `base`: element (m = 0, first row); `ld`: elements between rows
    __device__ __forceinline__ void load(const void* C, int64_t base, int64_t ld, int m, uint4 (&v)[8]) const
    {
        const int col = m + u * EPU;
        const TD* src = static_cast<const TD*>(C) + base + static_cast<int64_t>(r0) * ld + col;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            v[i] = (4 * i + r0 < rows && col < M) ? __ldg(reinterpret_cast<const uint4*>(src + static_cast<int64_t>(4 * i) * ld))
                                                  : make_uint4(0, 0, 0, 0);
    }
    __device__ __forceinline__ void stage(uint32_t buf, const uint4 (&v)[8]) const
    {
#pragma unroll
        for (int i = 0; i < 8; ++i) ptx::st_shared_v4(buf + at(i), v[i].x, v[i].y, v[i].z, v[i].w);
    }
    __device__ __forceinline__ void store(void* D, int64_t base, int64_t ld, int m, uint32_t buf) const
    {
        const int col = m + u * EPU;
        TD* dst = static_cast<TD*>(D) + base + static_cast<int64_t>(r0) * ld + col;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint4 v = ptx::ld_shared_v4(buf + at(i));
            if (4 * i + r0 < rows && col < M) *reinterpret_cast<uint4*>(dst + static_cast<int64_t>(4 * i) * ld) = v;
        }
    }
};

// Hand a drained TMEM buffer back to the MMA issuer: one arrival per epilogue warp, on the leader
// CTA's barrier (a remote arrival when this CTA is the peer of a pair).
template <int CG>
__device__ __forceinline__ void release_tmem(uint64_t* bar, int lane)
{
    ptx::tc_fence_before();
    __syncwarp();
    if (lane == 0) {
        // the accumulator belongs to the pair's leader (the even rank of the pair)
        if constexpr (CG == 2) ptx::mbar_arrive_cluster(ptx::mapa_shared(ptx::smem_u32(bar), ptx::cluster_ctarank() & ~1u));
        else ptx::mbar_arrive(bar);
    }
}

// Bounded wait until *ctr >= target (acquire at GPU scope); false once limit_ns has passed.
__device__ __forceinline__ bool wait_counter_ge(const int* ctr, int target, uint64_t limit_ns)
{
    const uint64_t t0 = ptx::globaltimer();
    while (true) {
        int v;
        asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
        if (v >= target) return true;
        if (ptx::globaltimer() - t0 > limit_ns) return false;
        __nanosleep(64);
    }
}

// A split has arrived and is not its tile's last: the chunks that it reduces itself, `own` once every split has
// arrived, none if it has no share or leaves it to the last one after limit_ns.
__device__ __forceinline__ int hand_over(int* ctr, int nsplit, int own, uint64_t limit_ns)
{
    if (!own) return 0;
    const uint64_t t0 = ptx::globaltimer();
    while (true) {
        int v;
        asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
        if ((v & 0xff) >= nsplit) return own;
        if (ptx::globaltimer() - t0 > limit_ns) {
            if (atomicCAS(ctr, v, v | (own << 8)) == v) return 0;
            continue;                               // another split came or left: look again
        }
        __nanosleep(64);
    }
}

// Split-k completion, run by the epilogue warps after this split parked its partial tile in the
// workspace (layout [32-column chunk][column][row], so every warp access is one 128-byte line; the
// TMEM buffer is free again).  The partials are summed in split order, so the result does not depend on
// which CTA finishes when, and the epilogue runs on the sums.  A warp of each TMEM quarter takes W of
// a chunk's 32 columns.
//   p.par_reduce   every split unit of the launch is resident at once (all in the first round of the
//                  persistent schedule): each split waits until the tile's other splits have parked
//                  theirs, then reduces its share of the tile -- chunks split, split + nsplit, ...
//                  The tile counter counts arrivals up to nsplit, then finished shares up to
//                  2 * nsplit, when the last one resets it for the next launch.
//   par_reduce 2   the same where launches on other streams may hold part of the SMs, so that a tile's other
//                  splits may be unable to start until this CTA leaves: a split waits hand_over_ns at most, then
//                  leaves its share to the last one to arrive.  The counter's low byte counts arrivals and the
//                  next holds the chunks left; it is not reset (such a launch has zeroed counters of its own).
//   otherwise      the last split to arrive (tile counter) reduces the whole tile and resets it.
// Every thread passes the same named barriers whether or not it has work, so a warp that gave up on
// a wait cannot strand the others.
// BESIDE: kernels that par_reduce 2 may be asked of (the promoted ones; the others' code stays as short as it was).
template <typename TD, bool EPI, int NH, bool BESIDE>
__device__ __forceinline__ void split_finish(const TcKernelParams& p, float& amax, const TileJob& j, bool& ok, int et,
                                             int lane, int half, int row, bool row_ok, int64_t base_c, int64_t base_d,
                                             volatile int* last_flag, volatile int* abort_flag, bool c_staged,
                                             uint32_t c_row)
{
    constexpr int W = 32 / NH;                      // columns of a chunk per warp
    const bool beside = BESIDE && p.par_reduce == 2;
    const bool par = p.par_reduce != 0 && !beside;
    __threadfence();
    ptx::named_sync<NH * 128>();
    if (et == 0) {
        int go = 0;                                 // beside: the chunks that this split reduces, a bit each
        if (ok) {
            int* const ctr = p.counters + j.slot;
            const int before = atomicAdd(ctr, 1);
            if (par) {
                go = wait_counter_ge(ctr, j.nsplit, p.timeout_ns) ? 1 : 0;
                if (!go) record_error(p, abort_flag, 16);
            } else if (beside) {
                int own = 0;
                for (int c = j.split; c < p.bm / 32; c += j.nsplit) own |= 1 << c;
                go = (before & 0xff) == j.nsplit - 1 ? own | (before >> 8) : hand_over(ctr, j.nsplit, own, p.hand_over_ns);
            } else {
                go = before == j.nsplit - 1 ? 1 : 0;
            }
        }
        *last_flag = go;
    }
    ptx::named_sync<NH * 128>();
    const int go = *last_flag;
    if (go) {
        __threadfence();
        const int chunks = p.bm / 32, step = par ? j.nsplit : 1;
        const size_t slab_elems = static_cast<size_t>(kTcTileN) * p.bm;
        const float* base = p.ws + static_cast<size_t>(j.slot) * p.tail_split * slab_elems +
                            static_cast<size_t>(half) * W * kTcTileN + row;
        for (int c = par ? j.split : 0; c < chunks; c += step) {
            if (beside && !((go >> c) & 1)) continue;
            const int m = j.m0 + c * 32 + half * W;
            // two splits' partials at a time are in flight together (the reduction is
            // latency-bound), summed in split order
            float v[W];
#pragma unroll
            for (int i = 0; i < W; ++i) v[i] = 0.f;
            const float* sa = base + static_cast<size_t>(c) * 32 * kTcTileN;
            for (int s = 0; s < j.nsplit; s += 2, sa += 2 * slab_elems) {
                float a[W], b[W];
                const bool two = s + 1 < j.nsplit;
#pragma unroll
                for (int i = 0; i < W; ++i) {
                    a[i] = __ldcg(sa + i * kTcTileN);
                    b[i] = two ? __ldcg(sa + slab_elems + i * kTcTileN) : 0.f;
                }
#pragma unroll
                for (int i = 0; i < W; ++i) v[i] += a[i];
                if (two) {
#pragma unroll
                    for (int i = 0; i < W; ++i) v[i] += b[i];
                }
            }
            if (row_ok && m < j.M) {
                uint32_t cw[W];
                if (c == j.split && c_staged) {
                    // this chunk's C row was copied into shared memory while the tile accumulated
                    // (16-byte unit u at u ^ (lane & 7))
                    ptx::cp_async_wait0();
                    constexpr int NU = W * static_cast<int>(sizeof(TD)) / 16;
#pragma unroll
                    for (int u = 0; u < NU; ++u) {
                        const uint4 w4 = ptx::ld_shared_v4(c_row + static_cast<uint32_t>((u ^ (lane & 7)) * 16));
                        cw[4 * u] = w4.x;
                        cw[4 * u + 1] = w4.y;
                        cw[4 * u + 2] = w4.z;
                        cw[4 * u + 3] = w4.w;
                    }
                } else {
                    load_c_chunk<TD, W>(j, base_c, m, cw);
                }
                store_chunk_pre<TD, EPI, W>(p, amax, j, base_d, m, v, cw);
            }
        }
    } else if (par) {
        ok = false;
    }
    if (c_staged) ptx::cp_async_wait0();   // the staging buffer is free again (also on the error path)
    ptx::named_sync<NH * 128>();           // last_flag is reused by the next tile
    if (et == 0 && go && !beside) {
        if (!par) p.counters[j.slot] = 0;  // ready for the next launch
        // counts this split out of the tile: the last one resets the counter for the next launch.
        // No fence: the counter only orders the splits' waits (same-address atomics), and the next
        // launch's use of the workspace is ordered by the kernel boundary.
        else if (atomicAdd(p.counters + j.slot, 1) == 2 * j.nsplit - 1) atomicExch(p.counters + j.slot, 0);
    }
}

// MODE
//   kModePromo   promoted accumulation (promote_k > 0): four epilogue warps hold 128 running sums per
//                thread.
//   kModePieces  promoted accumulation of the split-precision products, each piece of an operand staged
//                once per k-block for all the products that use it; 256-column tiles, sixteen epilogue
//                warps with 64 running sums per thread.  The A0*B0 chain and the small products have one
//                accumulator each.  With all products in one accumulator and two of those alternating,
//                every product but a chain's first dropped the bits of a sum at full magnitude (bf16x6
//                8192^3, largest error over largest value 5.3e-7).
//   kModePlain   the others: eight epilogue warps, two per quarter of the TMEM lanes,
// which take alternate column groups of a tile (half the drain time of a CTA's last tile, and of every
// tile whose k is too short to hide it).  GROUP: the work units and problems come from a plan's tables.
template <int KIND, typename TD, int CL, bool EPI, int MODE, bool GROUP>
__global__ void __launch_bounds__(tc_threads(MODE), 1) tc_gemm_kernel(const __grid_constant__ TcKernelParams p)
{
    // CL CTAs per cluster.  CL == 2: a CTA pair on two SMs works on one 256-row tile.  Each CTA
    // stages its own 128 rows of the n-side operand and its half of the m-side operand; the leader
    // (even rank) issues the pair MMAs, whose accumulator rows 0-127 live in the leader's TMEM and
    // 128-255 in the peer's.  The leader arms its full barriers with both CTAs' bytes and both CTAs'
    // TMA completions land on them; MMA completions are multicast to both CTAs, and both epilogues
    // release the leader's TMEM buffers with remote arrivals.
    // CL == 4: two such pairs on adjacent 256-row tiles with the same m range.  CTA r of one pair
    // needs the same m-side rows as CTA r of the other, so each loads half of them and multicasts
    // it to both (half the m-side L2 traffic); a ring slot is refilled only after both pairs' MMAs
    // have released it (each slot's empty barrier expects one commit from each pair's leader).
    constexpr int CG = CL >= 2 ? 2 : 1;         // CTAs per MMA (cta_group)
    constexpr int MC = CL / CG;                 // pairs sharing the m-side operand
    constexpr bool PROMO = MODE == kModePromo, PIECES = MODE == kModePieces;
    constexpr int NH = PROMO ? 1 : (PIECES ? 4 : 2);      // epilogue warps per TMEM lane quarter
    constexpr int EW0 = 2;                      // first epilogue warp
    if (threadIdx.x == 0 && p.trace != nullptr) {
        trace_mark(p, TL_TRACE_ENTRY);
        trace_put(p, TL_TRACE_ENTRY_NS, global_ns());
        unsigned int smid;
        asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
        trace_put(p, TL_TRACE_SMID, smid);
    }
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t bmc = static_cast<uint32_t>(p.bm) / CG;            // m-side rows staged by this CTA
    const uint32_t tileN_bytes = kTcTileN * kTcRowBytes;
    const uint32_t stage_bytes = tileN_bytes + bmc * kTcRowBytes;
    // output staging: per epilogue warp 32 rows x 128 bytes (C in, D out), 1024-byte aligned
    uint8_t* epi_stage = smem + static_cast<size_t>(p.stages) * stage_bytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(epi_stage + static_cast<size_t>(p.epi_bufs) * kTcEpiStageBytes);
    uint64_t* empty = full + kTcMaxStages;
    uint64_t* tfull = empty + kTcMaxStages;     // main accumulator buffers (per tile, or per chain)
    uint64_t* tempty = tfull + 2;
    uint64_t* sfull = tempty + 2;               // small-term accumulators (promotion with split terms)
    uint64_t* sempty = sfull + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sempty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* last_flag = abort_flag + 1;

    const uint32_t ring_a = ptx::smem_u32(smem), full_a = ptx::smem_u32(full), empty_a = ptx::smem_u32(empty);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = (CL > 1) ? ptx::cluster_ctarank() : 0u;
    const uint32_t pair_rank = rank & 1u;       // position within the CTA pair
    const uint32_t pair_base = rank & ~1u;      // the pair's leader
    const bool leader = (pair_rank == 0);
    const int64_t unit0 = (CL > 1) ? static_cast<int64_t>(ptx::cluster_id_x()) : static_cast<int64_t>(blockIdx.x);
    const int64_t units = (CL > 1) ? static_cast<int64_t>(ptx::ncluster_x()) : static_cast<int64_t>(gridDim.x);
    const bool sep_small = MODE != kModePlain && p.nterms > 1;
    // TMEM columns: main accumulator x2 (+ small-term accumulator x2 when they are kept apart); with 256
    // columns one of each
    const uint32_t need_cols = static_cast<uint32_t>(p.bm) * (sep_small && !PIECES ? 4u : 2u);
    const uint32_t tmem_cols = need_cols <= 128 ? 128u : (need_cols <= 256 ? 256u : 512u);
    const uint32_t epi_arrivals = 4u * NH * CG;     // one per epilogue warp of each CTA

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            ptx::mbar_init(&full[s], 1);
            ptx::mbar_init(&empty[s], MC);
        }
        for (int a = 0; a < 2; ++a) {
            ptx::mbar_init(&tfull[a], 1);
            ptx::mbar_init(&tempty[a], epi_arrivals);
            ptx::mbar_init(&sfull[a], 1);
            ptx::mbar_init(&sempty[a], epi_arrivals);
        }
        *abort_flag = 0;
        *last_flag = 0;
        ptx::fence_mbar_init();
        ptx::fence_proxy_async_smem();
    }
    if (warp == 1) {
        if constexpr (CG == 2) {
            ptx::tmem_alloc_pair(tmem_slot, tmem_cols);
            ptx::tmem_relinquish_pair();
        } else {
            ptx::tmem_alloc(tmem_slot, tmem_cols);
            ptx::tmem_relinquish();
        }
    }
    if (!GROUP && warp == 0 && lane == 0) {
        for (int v = 0; v < p.nterms; ++v) {
            ptx::prefetch_tmap(&p.tmN[p.term_n[v]]);
            ptx::prefetch_tmap(&p.tmM[p.term_m[v]]);
        }
    }
    ptx::tc_fence_before();
    __syncthreads();
    if constexpr (CL > 1) ptx::cluster_sync();     // peer barriers initialised before any remote arrive
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (threadIdx.x == 0) trace_mark(p, TL_TRACE_SETUP);
    // Launched as a programmatic dependent: everything above (barrier set-up, TMEM allocation,
    // descriptor prefetch) may have run while the previous kernel in the stream was finishing.
    // Every role that touches global memory first decodes its first work unit (from the kernel
    // parameters and, for a group, the plan's tables, which no kernel writes), then waits for that
    // grid to complete (its writes visible); the producer then lets the next dependent grid start
    // its own set-up as soon as SMs free up.  Decoding after the wait put ~2000 clocks, most of it
    // instruction fetch, between the previous grid's end and the first copy.
    const int nvirt = p.nterms;
    const uint64_t tlim = p.timeout_ns;

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer (each CTA)
        // One flat loop over (k-block, product) per tile, run by one lane: a wait on a completed barrier
        // costs it 36 clocks (130 when 32 lanes ask), and everything that does not change from one
        // k-block to the next (shared-memory and barrier addresses, the peer's barrier, the tensor
        // maps of a single product) is formed outside the loop.  With the warp in step, a k-block
        // cost this loop 465-570 clocks and the MMA issuer's 455-525 whatever the tile, more than the
        // 256 clocks of a 128-column k-block's MMAs.
        if (ptx::elect_one())
        {
            uint32_t phase = 0;
            constexpr int W = kTcRowBytes / (KIND == 0 ? 2 : 1);   // elements per 128-byte row
            constexpr uint32_t kChunk = W * kTcRowBytes;           // bytes of one MN-major box
            const bool skip = p.debug_skip_loads != 0;
            // the barrier that counts this CTA's bytes: its own, or the pair leader's
            const uint32_t full_off = (CG == 2) ? ptx::mapa_shared(full_a, pair_base) - empty_a : full_a - empty_a;
            const int nchunk = static_cast<int>(bmc) / W;          // MN-major m-side boxes
            const uint32_t bar_end = empty_a + 8u * static_cast<uint32_t>(p.stages);
            uint32_t bar = empty_a;                // empty barrier and slot of the current stage
            uint32_t sN = ring_a;
            bool ok = true;
            // one stage: wait for its slot, arm its full barrier, issue its copies
            auto fill = [&](auto n_mn, auto m_mn, const void* mapN, const void* mapM, int k0, int n0, int m0, int b) {
                if (!ptx::mbar_wait(bar, phase ^ 1u, tlim)) {
                    record_error(p, abort_flag, 1);
                    return false;
                }
                // the timeout-path test issues nothing: the full barriers never complete, the
                // MMA and epilogue waits run out, and no copy is left in flight
                if (!skip) {
                    const uint32_t sM = sN + tileN_bytes;
                    const uint32_t fb = bar + full_off;
                    if constexpr (CG == 2) {
                        // the leader arms its full barrier with both CTAs' bytes; the peer's loads
                        // only complete transactions on it (they cannot run a phase ahead: the
                        // peer refills a slot only after the leader's MMAs released it)
                        if (leader) ptx::mbar_arrive_expect_tx(bar + (full_a - empty_a), 2u * stage_bytes);
                        if constexpr (!decltype(n_mn)::value) {
                            ptx::tma_load_3d_pair(sN, mapN, fb, k0, n0, b);
                        } else {
#pragma unroll
                            for (int c = 0; c < kTcTileN / W; ++c)
                                ptx::tma_load_3d_pair(sN + c * kChunk, mapN, fb, n0 + c * W, k0, b);
                        }
                        if constexpr (MC == 2) {
                            // this CTA's half of the m rows shared with CTA pair_rank of the other
                            // pair; the copy lands in both and is counted on each pair's leader
                            const int half = static_cast<int>(rank >> 1);
                            const uint16_t mask = static_cast<uint16_t>((1u << pair_rank) | (1u << (pair_rank + 2)));
                            if constexpr (!decltype(m_mn)::value)
                                ptx::tma_load_3d_pair_mc(sM + half * (bmc / 2) * kTcRowBytes, mapM, fb, mask, k0,
                                                         m0 + half * static_cast<int>(bmc / 2), b);
                            else
                                ptx::tma_load_3d_pair_mc(sM + half * kChunk, mapM, fb, mask, m0 + half * W, k0, b);
                        } else if constexpr (!decltype(m_mn)::value) {
                            ptx::tma_load_3d_pair(sM, mapM, fb, k0, m0, b);
                        } else {
#pragma unroll
                            for (int c = 0; c < 2; ++c)      // 64 or 128 m rows per CTA: at most two boxes
                                if (c < nchunk) ptx::tma_load_3d_pair(sM + c * kChunk, mapM, fb, m0 + c * W, k0, b);
                        }
                    } else {
                        ptx::mbar_arrive_expect_tx(fb, stage_bytes);
                        if constexpr (!decltype(n_mn)::value) {
                            ptx::tma_load_3d(sN, mapN, fb, k0, n0, b);
                        } else {
#pragma unroll
                            for (int c = 0; c < kTcTileN / W; ++c)
                                ptx::tma_load_3d(sN + c * kChunk, mapN, fb, n0 + c * W, k0, b);
                        }
                        if constexpr (!decltype(m_mn)::value) {
                            ptx::tma_load_3d(sM, mapM, fb, k0, m0, b);
                        } else {
#pragma unroll
                            for (int c = 0; c < 4; ++c)      // at most four boxes
                                if (c < nchunk) ptx::tma_load_3d(sM + c * kChunk, mapM, fb, m0 + c * W, k0, b);
                        }
                    }
                }
                bar += 8u;
                sN += stage_bytes;
                if (bar == bar_end) {
                    bar = empty_a;
                    sN = ring_a;
                    phase ^= 1u;
                }
                return true;
            };
            // a tile's stages; the layouts are compile-time inside
            auto produce = [&](auto n_mn, auto m_mn, const TileJob& j, int n0, int m0) {
                int k0 = j.kb0 * W;
                if (nvirt == 1) {
                    for (int i = j.kb1 - j.kb0; i > 0; --i) {
                        if (!(ok = fill(n_mn, m_mn, j.tmN, j.tmM, k0, n0, m0, j.b))) break;
                        k0 += W;
                    }
                } else {
                    // split-precision products, smallest first (term table set by the host)
                    int v = 0;
                    for (int i = (j.kb1 - j.kb0) * nvirt; i > 0; --i) {
                        if (!(ok = fill(n_mn, m_mn, &p.tmN[p.term_n[v]], &p.tmM[p.term_m[v]], k0, n0, m0, j.b))) break;
                        if (++v == nvirt) {
                            v = 0;
                            k0 += W;
                        }
                    }
                }
            };
            using Yes = std::true_type;
            using No = std::false_type;
            int64_t w = unit0;                         // < total_work: the grid is never larger
            int4 u = load_unit<GROUP>(p, w);
            int4 u_next = load_unit<GROUP>(p, w + units);     // in flight during this tile
            bool first = true;
#pragma unroll 1
            while (true) {
                TileJob j;
                get_job<GROUP>(p, w, u, j);
                const int n0 = j.n0 + static_cast<int>(rank) * kTcTileN;
                const int m0 = j.m0 + static_cast<int>(pair_rank * bmc);
                // timeline stamps stay outside the k-block loops (a branch there slows the issue)
                if (first) {
                    ptx::grid_dep_wait();
                    ptx::grid_dep_launch_dependents();
                    if (!launch_live<MODE>(p)) break;
                    trace_mark(p, TL_TRACE_DEP);
                    trace_mark(p, TL_TRACE_LOAD_FIRST);
                }
                if (p.n_mn_major) {
                    if (p.m_mn_major) produce(Yes{}, Yes{}, j, n0, m0);
                    else produce(Yes{}, No{}, j, n0, m0);
                } else {
                    if (p.m_mn_major) produce(No{}, Yes{}, j, n0, m0);
                    else produce(No{}, No{}, j, n0, m0);
                }
                if (first) trace_mark(p, TL_TRACE_LOAD_LAST);
                first = false;
                w += units;
                if (!ok || w >= p.total_work) break;
                u = u_next;
                u_next = load_unit<GROUP>(p, w + units);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer (leader CTA)
        // Without promotion a tile's whole k range accumulates in one TMEM buffer (two buffers
        // alternate between tiles).  With promotion the A0*B0 product restarts its accumulation
        // every promote_kb k-blocks in the alternate buffer (the epilogue drains each chain into
        // fp32 registers), and the small split-precision products accumulate for the whole tile in
        // a separate pair of buffers.  One flat loop per tile over (k-block, product), run by one
        // lane (see the producer).
        if (leader && ptx::elect_one()) {
            uint32_t phase = 0, mbuf = 0, mph = 0, sbuf = 0, sph = 0;
            const uint16_t pair_mask = static_cast<uint16_t>(0x3u << pair_base);
            const uint32_t idesc = p.idesc;
            const uint32_t n_kstep = p.n_kstep >> 4, m_kstep = p.m_kstep >> 4;
            const uint32_t bmu = static_cast<uint32_t>(p.bm);
            // the current slot: its full barrier and the low word of its n-side descriptor (the m-side
            // word is a constant further, the high word a constant)
            constexpr uint32_t dhi = ptx::sdesc_hi(1024);
            const uint32_t dN0 = ptx::sdesc_lo(ring_a, p.n_lbo);
            const uint32_t dNM = ptx::sdesc_lo(ring_a + tileN_bytes, p.m_lbo) - dN0;
            const uint32_t dstep = stage_bytes >> 4;
            const uint32_t bar_end = full_a + 8u * static_cast<uint32_t>(p.stages);
            uint32_t dN = dN0, bar = full_a;
            // a stage's bytes have arrived
            auto arrived = [&] {
                if (!ptx::mbar_wait(bar, phase, tlim)) {
                    record_error(p, abort_flag, 4);
                    return false;
                }
                ptx::tc_fence_after();
                return true;
            };
            // its slot is released when the MMAs issued so far complete
            auto release = [&] {
                // both pairs' ring slots are released (MC == 2: every CTA of the cluster)
                if constexpr (CG == 2) ptx::mma_commit_pair(bar + (empty_a - full_a), MC == 2 ? 0xF : 0x3);
                else ptx::mma_commit(bar + (empty_a - full_a));
                bar += 8u;
                dN += dstep;
                if (bar == bar_end) {
                    bar = full_a;
                    dN = dN0;
                    phase ^= 1u;
                }
            };
            // one stage into `d_tmem`
            auto consume = [&](uint32_t d_tmem, uint32_t accumulate) {
                if (!arrived()) return false;
                ptx::mma_kblock<KIND, CG>(d_tmem, dN, dN + dNM, dhi, idesc, accumulate, n_kstep, m_kstep);
                release();
                return true;
            };
            // hand the main accumulator's chain to the epilogue and continue in the other buffer
            auto next_chain = [&] {
                if constexpr (CG == 2) ptx::mma_commit_pair(ptx::smem_u32(&tfull[mbuf]), pair_mask);
                else ptx::mma_commit(ptx::smem_u32(&tfull[mbuf]));
                mbuf ^= 1u;
                if (mbuf == 0) mph ^= 1u;
                if (!ptx::mbar_wait(&tempty[mbuf], mph ^ 1u, tlim)) {
                    record_error(p, abort_flag, 2);
                    return false;
                }
                ptx::tc_fence_after();
                return true;
            };
            bool ok = true;
            // (touches no global memory but the error word and the timeline)
            if (p.trace != nullptr || (MODE != kModePlain && p.range != nullptr)) ptx::grid_dep_wait();
            ok = launch_live<MODE>(p);
            int4 u_next = load_unit<GROUP>(p, unit0);
            for (int64_t w = unit0; w < p.total_work && ok; w += units) {
                const int4 u = u_next;
                u_next = load_unit<GROUP>(p, w + units);      // in flight during this tile
                TileJob j;
                get_job<GROUP>(p, w, u, j);
                const int nkb = j.kb1 - j.kb0;
                if (nkb <= 0) continue;                 // an empty unit of a balanced split
                if (sep_small && !PIECES) {
                    if (!ptx::mbar_wait(&sempty[sbuf], sph ^ 1u, tlim)) {
                        record_error(p, abort_flag, 2);
                        break;
                    }
                    ptx::tc_fence_after();
                }
                if (!PIECES && !ptx::mbar_wait(&tempty[mbuf], mph ^ 1u, tlim)) {
                    record_error(p, abort_flag, 2);
                    break;
                }
                ptx::tc_fence_after();
                if (p.trace != nullptr && w == unit0) {
                    // timeline: the first stage's arrival, waited for here (the loop's own wait on
                    // it then passes at once) so that the k-block loop carries no stamp
                    ptx::mbar_wait(bar, phase, tlim);
                    trace_mark(p, TL_TRACE_MMA_FIRST);
                }
                if constexpr (PIECES) {
                    // A k-block's pieces arrive smallest first in nvirt consecutive slots; every product
                    // of them is formed from there and a slot is released by its last product.  The small
                    // products share one accumulator, which starts anew every small_chains chains, the
                    // A0*B0 products another that starts anew every promote_kb k-blocks.  There is one of
                    // each: a chain is drained while the next k-block's small products run, the small sums
                    // while the last A0*B0 of the chain that they end with does.
                    const uint32_t d_small = tmem_base + bmu;
                    uint32_t small_acc = 0, main_acc = 0;
                    int in_chain = 0, chains = 0;
                    for (int kb = 0; kb < nkb; ++kb) {
                        const bool last = kb == nkb - 1;
                        const bool chain_ends = in_chain + 1 == p.promote_kb || last;
                        const bool small_ends = last || (chain_ends && chains + 1 == p.small_chains);
                        uint32_t sl[3], dn[3];
#pragma unroll
                        for (int v = 0; v < 3; ++v) {
                            if (v < nvirt) {
                                if (ok && !ptx::mbar_wait(bar, phase, tlim)) {
                                    record_error(p, abort_flag, 4);
                                    ok = false;
                                }
                                sl[v] = bar + (empty_a - full_a);
                                dn[v] = dN;
                                bar += 8u;
                                dN += dstep;
                                if (bar == bar_end) {
                                    bar = full_a;
                                    dN = dN0;
                                    phase ^= 1u;
                                }
                            }
                        }
                        if (!ok) break;
                        ptx::tc_fence_after();
                        const uint32_t d0 = nvirt == 3 ? dn[2] : dn[1];          // dn: pieces (2,) 1, 0
                        auto mma = [&](uint32_t n, uint32_t m) {
                            ptx::mma_kblock<KIND, CG>(d_small, n, m + dNM, dhi, idesc, small_acc, n_kstep, m_kstep);
                            small_acc = 1;
                        };
                        if (small_acc == 0 && !ptx::mbar_wait(&sempty[0], sph ^ 1u, tlim)) {
                            record_error(p, abort_flag, 2);
                            ok = false;
                            break;
                        }
                        ptx::tc_fence_after();
                        if (nvirt == 3) {
                            mma(dn[2], dn[0]);
                            mma(dn[1], dn[1]);
                            mma(dn[0], dn[2]);
                            ptx::mma_commit_pair(sl[0], 0x3);
                            mma(dn[2], dn[1]);
                            mma(dn[1], dn[2]);
                            ptx::mma_commit_pair(sl[1], 0x3);
                        } else {
                            mma(dn[1], dn[0]);
                            mma(dn[0], dn[1]);
                            ptx::mma_commit_pair(sl[0], 0x3);
                        }
                        if (small_ends) {
                            ptx::mma_commit_pair(ptx::smem_u32(&sfull[0]), pair_mask);
                            sph ^= 1u;
                            small_acc = 0;
                        }
                        if (in_chain == 0) {
                            if (!ptx::mbar_wait(&tempty[0], mph ^ 1u, tlim)) {
                                record_error(p, abort_flag, 2);
                                ok = false;
                                break;
                            }
                            ptx::tc_fence_after();
                            main_acc = 0;
                        }
                        ptx::mma_kblock<KIND, CG>(tmem_base, d0, d0 + dNM, dhi, idesc, main_acc, n_kstep, m_kstep);
                        main_acc = 1;
                        ++in_chain;
                        if (chain_ends) {
                            ptx::mma_commit_pair(ptx::smem_u32(&tfull[0]), pair_mask);
                            mph ^= 1u;
                            in_chain = 0;
                            ++chains;
                        }
                        if (small_ends) chains = 0;
                        ptx::mma_commit_pair(nvirt == 3 ? sl[2] : sl[1], 0x3);
                    }
                } else if constexpr (!PROMO) {
                    // every product of the tile into one accumulator
                    const uint32_t d_tmem = tmem_base + mbuf * bmu;
                    uint32_t accumulate = 0;
                    for (int i = nkb * nvirt; i > 0; --i) {
                        if (!(ok = consume(d_tmem, accumulate))) break;
                        accumulate = 1;
                    }
                } else {
                    uint32_t main_acc = 0, small_acc = 0;
                    int in_chain = 0;
                    for (int kb = 0; kb < nkb && ok; ++kb) {
                        if (in_chain == p.promote_kb) {
                            // (a tile's last chain is handed over after the loop)
                            if (!(ok = next_chain())) break;
                            in_chain = 0;
                            main_acc = 0;
                        }
                        for (int v = 0; v < nvirt - 1 && ok; ++v) {
                            ok = consume(tmem_base + (2u + sbuf) * bmu, small_acc);
                            small_acc = 1;
                        }
                        if constexpr (KIND == 0) {
                            if (ok && p.promote_half) {
                                if (!(ok = arrived())) break;
                                for (uint32_t i = 0; i < 4u; ++i) {
                                    if (i == 2u && !(ok = next_chain())) break;
                                    ptx::mma_k16<CG>(tmem_base + mbuf * bmu, dN + i * n_kstep, dN + dNM + i * m_kstep, dhi, idesc,
                                                     i & 1u);
                                }
                                if (!ok) break;
                                release();
                                ++in_chain;
                                continue;
                            }
                        }
                        if (ok) ok = consume(tmem_base + mbuf * bmu, main_acc);
                        main_acc = 1;
                        ++in_chain;
                    }
                }
                if (!ok) break;
                if constexpr (PIECES) {              // handed over in the loop; one buffer of each kind
                    if (w == unit0) trace_mark(p, TL_TRACE_MMA_LAST);
                    continue;
                }
                if constexpr (CG == 2) ptx::mma_commit_pair(ptx::smem_u32(&tfull[mbuf]), pair_mask);
                else ptx::mma_commit(ptx::smem_u32(&tfull[mbuf]));
                if (sep_small) {
                    if constexpr (CG == 2) ptx::mma_commit_pair(ptx::smem_u32(&sfull[sbuf]), pair_mask);
                    else ptx::mma_commit(ptx::smem_u32(&sfull[sbuf]));
                }
                if (w == unit0) trace_mark(p, TL_TRACE_MMA_LAST);
                mbuf ^= 1u;
                if (mbuf == 0) mph ^= 1u;
                if (sep_small) {
                    sbuf ^= 1u;
                    if (sbuf == 0) sph ^= 1u;
                }
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ epilogue (4 * NH warps, each CTA)
        // All of them run the same loop and, in split-k mode, the same named barriers: after a
        // timed-out wait a warp keeps the control flow and only skips the work, so no warp can be
        // left waiting at bar.sync 1 for one that gave up.
        const int quarter = warp & 3;             // TMEM lanes 32*quarter .. +31
        const int row = quarter * 32 + lane;      // tile row = problem n offset within this CTA
        const int half = (warp - EW0) >> 2;         // which of the quarter's NH warps
        const int et = threadIdx.x - 32 * EW0;    // 0 .. 128 * NH - 1
        // staging: 4 KB per warp; where shared memory holds only 16 KB of it, the second warp of a quarter
        // takes no part in staged stores.  The promotion kernels stage nothing.
        const int nst = MODE == kModePlain ? min(NH, p.epi_bufs) : 1;      // staging warps per quarter
        const uint32_t my_stage_a = ptx::smem_u32(epi_stage) + static_cast<uint32_t>(min(half, nst - 1) * 4 + quarter) * 4096u;
        const uint32_t lane_off = static_cast<uint32_t>(quarter * 32) << 16;
        uint32_t mbuf = 0, mph = 0, sbuf = 0, sph = 0;
        const int chunks = p.bm / 32;
        bool ok = true;
        float amax = 0.0f;                        // fused epilogue: this thread's max |output|
        unsigned long long units_done = 0;
#pragma unroll 1
        for (int64_t w = unit0; w < p.total_work; w += units) {
            // the epilogue trails the MMAs: no need to load the unit ahead
            TileJob j;
            get_job<GROUP>(p, w, load_unit<GROUP>(p, w), j);
            if (w == unit0) {
                ptx::grid_dep_wait();
                if (!launch_live<MODE>(p)) break;
            }
            if (j.kb1 <= j.kb0) continue;             // an empty unit of a balanced split
            ++units_done;
            const bool tr = (et == 0 && w == unit0);  // timeline stamps: the first tile, one thread
            j.n0 += static_cast<int>(rank) * kTcTileN;
            j.slot = j.slot * CL + rank;              // split-k slabs and counters per CTA
            const int n = j.n0 + row;
            const bool row_ok = n < j.N;
            // this thread's row n of the output: a contiguous run of m, or with a transposed output
            // one element of each of the columns m (stride ld)
            const int64_t base_d = static_cast<int64_t>(j.b) * p.stride_d + static_cast<int64_t>(n) * (j.out_t ? 1 : j.ldd);
            const int64_t base_c = static_cast<int64_t>(j.b) * p.stride_c + static_cast<int64_t>(n) * (j.out_t ? 1 : j.ldc);
            if (ok && row_ok && !j.out_t && j.beta != 0.0f && j.C != nullptr && (j.nsplit == 1 || j.split == j.nsplit - 1)) {
                // C does not depend on the accumulator: start pulling this row's segment into L2
                // while the tile is still accumulating
                const char* cp = static_cast<const char*>(j.C) + (base_c + j.m0) * static_cast<int64_t>(sizeof(TD));
                const int cbytes = (min(p.bm, j.M - j.m0)) * static_cast<int>(sizeof(TD));
                for (int off = 128 * half; off < cbytes; off += 128 * NH)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(cp + off));
            }
            if constexpr (MODE != kModePlain) {
                // ---- promotion: sum the chains (and the separate small terms) in fp32 registers: all 128
                // columns of the tile, or this warp's 64 of 256
                constexpr int RC = PROMO ? 128 : 64;                  // columns of this thread
                constexpr int QW = PROMO ? 16 : 8, NQ = RC / QW;
                const int col0 = PROMO ? 0 : RC * half;
                float run[RC];
#pragma unroll
                for (int i = 0; i < RC; ++i) run[i] = 0.f;
                const int nkb = j.kb1 - j.kb0;
                const int nchain = PROMO && p.promote_half ? 2 * nkb : (nkb + p.promote_kb - 1) / p.promote_kb;
                // the small terms: after the chains, or (one buffer of each kind) before the chain that they end
                // with, the last one and every small_chains'th
                int left = nchain, chains = 0;
                bool sm = PIECES && (left == 1 || p.small_chains == 1);
                while (left > 0 || sm) {
                    uint64_t* const full_bar = sm ? &sfull[sbuf] : &tfull[mbuf];
                    bool got = ok && ptx::mbar_wait(full_bar, sm ? sph : mph, tlim);
                    got = __all_sync(0xffffffffu, got);
                    if (ok && !got) {
                        if (lane == 0) record_error(p, abort_flag, 8);
                        ok = false;
                    }
                    if (ok) {
                        ptx::tc_fence_after();
                        const uint32_t buf = sm ? (PIECES ? 1u : 2u + sbuf) : mbuf;
                        const uint32_t tb = tmem_base + lane_off + buf * static_cast<uint32_t>(p.bm) + static_cast<uint32_t>(col0);
#pragma unroll
                        for (int q = 0; q < NQ; ++q) {
                            float r[QW];
                            __syncwarp();
                            ptx::tmem_ld<QW>(tb + q * QW, r);
#pragma unroll
                            for (int i = 0; i < QW; ++i) run[q * QW + i] += r[i];
                        }
                        release_tmem<CG>(sm ? &sempty[sbuf] : &tempty[mbuf], lane);
                    }
                    if (sm) {
                        if (!PIECES) sbuf ^= 1u;
                        if (sbuf == 0) sph ^= 1u;
                        sm = false;
                        chains = -1;
                    } else {
                        if (!PIECES) mbuf ^= 1u;
                        if (mbuf == 0) mph ^= 1u;
                        --left;
                        ++chains;
                        sm = PIECES ? left == 1 || (left > 0 && chains + 1 == p.small_chains) : sep_small && left == 0;
                    }
                }
                if (tr) trace_mark(p, TL_TRACE_ACC_READY);
                // With 96 registers of which 64 hold sums, the unit is decoded again here instead of
                // being held through the loop above (`w` is laundered so that it is): kept, its fields
                // lived in local memory, which no L1 is left for, and parking a tile took 30000 clocks.
                if constexpr (PIECES) {
                    int64_t w2 = w;
                    asm volatile("" : "+l"(w2));
                    get_job<GROUP>(p, w2, make_int4(0, 0, 0, 0), j);
                    j.n0 += static_cast<int>(rank) * kTcTileN;
                    j.slot = j.slot * CL + rank;
                }
                const int n2 = j.n0 + row;
                const bool row_ok2 = n2 < j.N;
                const int64_t d2 = static_cast<int64_t>(j.b) * p.stride_d + static_cast<int64_t>(n2) * (j.out_t ? 1 : j.ldd);
                const int64_t c2 = static_cast<int64_t>(j.b) * p.stride_c + static_cast<int64_t>(n2) * (j.out_t ? 1 : j.ldc);
                // QW columns at a time, the sums rotated through the registers: one copy of the code (and
                // no C loads hoisted into registers the sums occupy)
                if (j.nsplit == 1) {
                    if constexpr (PIECES) {
                        // 16 columns at a time through 2 KB of staging per warp (32 rows x 64 bytes, unit u of
                        // row r at u ^ (r / 2 % 4)): written by row as they are, read and finished in
                        // 64-byte runs, so that few registers are needed beside the sums and the stores
                        // cover whole sectors (a lane's own 16-byte stores along its row took 48000
                        // clocks a tile)
                        constexpr int SW = 16;
                        const uint32_t st = ptx::smem_u32(epi_stage) + static_cast<uint32_t>(warp - EW0) * 2048u;
                        const uint32_t sr = st + static_cast<uint32_t>(lane * 64);
                        const bool use_c = j.beta != 0.0f && j.C != nullptr;
                        const int nr = j.n0 + quarter * 32 + (lane >> 2);
#pragma unroll 1
                        for (int q = 0; q < RC / SW && ok; ++q) {
#pragma unroll
                            for (int u = 0; u < 4; ++u)
                                ptx::st_shared_v4(sr + static_cast<uint32_t>((u ^ ((lane >> 1) & 3)) * 16),
                                                  __float_as_uint(run[4 * u]), __float_as_uint(run[4 * u + 1]),
                                                  __float_as_uint(run[4 * u + 2]), __float_as_uint(run[4 * u + 3]));
#pragma unroll
                            for (int i = 0; i < RC - SW; ++i) run[i] = run[i + SW];
                            __syncwarp();
                            const int m = j.m0 + col0 + q * SW + 4 * (lane & 3);
#pragma unroll 1
                            for (int it = 0; it < 4; ++it) {
                                const int r = it * 8 + (lane >> 2), n = nr + it * 8;
                                const uint4 w = ptx::ld_shared_v4(st + static_cast<uint32_t>(r * 64 + (((lane & 3) ^ ((r >> 1) & 3)) * 16)));
                                if (n < j.N && m < j.M) {
                                    float o[4] = {__uint_as_float(w.x), __uint_as_float(w.y), __uint_as_float(w.z), __uint_as_float(w.w)};
                                    uint32_t cw[4];
                                    float bias[4];
                                    const int left = j.M - m;
                                    float* d = static_cast<float*>(j.D) + static_cast<int64_t>(j.b) * p.stride_d +
                                               static_cast<int64_t>(n) * j.ldd + m;
                                    if (use_c) {
                                        const float* c = static_cast<const float*>(j.C) + static_cast<int64_t>(j.b) * p.stride_c +
                                                         static_cast<int64_t>(n) * j.ldc + m;
                                        if (j.vec) {
                                            const uint4 c4 = __ldg(reinterpret_cast<const uint4*>(c));
                                            cw[0] = c4.x; cw[1] = c4.y; cw[2] = c4.z; cw[3] = c4.w;
                                        } else {
#pragma unroll
                                            for (int e = 0; e < 4; ++e) cw[e] = e < left ? __float_as_uint(c[e]) : 0u;
                                        }
                                    }
                                    if constexpr (EPI) {
                                        if (p.epi_bias != nullptr) load_bias<4>(p, j.M, m, bias);
                                    }
                                    finish_values<TD, EPI, 4>(p, amax, j, m, true, cw, bias, o);
                                    if (j.vec) {
                                        *reinterpret_cast<float4*>(d) = make_float4(o[0], o[1], o[2], o[3]);
                                    } else {
#pragma unroll
                                        for (int e = 0; e < 4; ++e)
                                            if (e < left) d[e] = o[e];
                                    }
                                }
                            }
                            __syncwarp();
                        }
                    } else {
#pragma unroll 1
                        for (int q = 0; q < NQ; ++q) {
                            const int m = j.m0 + col0 + q * QW;
                            float v[QW];
#pragma unroll
                            for (int i = 0; i < QW; ++i) v[i] = run[i];
#pragma unroll
                            for (int i = 0; i < RC - QW; ++i) run[i] = run[i + QW];
                            if (ok && row_ok2 && m < j.M) store_chunk<TD, EPI, QW>(p, amax, j, c2, d2, m, v);
                        }
                    }
                    if (tr) trace_mark(p, TL_TRACE_STORED);
                } else {
                    float* dst = p.ws + (static_cast<size_t>(j.slot) * p.tail_split + j.split) *
                                            (static_cast<size_t>(kTcTileN) * p.bm) +
                                 static_cast<size_t>(col0) * kTcTileN + row;
                    if (ok) {
#pragma unroll
                        for (int i = 0; i < RC; ++i) __stcg(dst + i * kTcTileN, run[i]);
                    }
                    if (tr) trace_mark(p, TL_TRACE_STORED);
                    split_finish<TD, EPI, NH, true>(p, amax, j, ok, et, lane, half, row, row_ok2, c2, d2, last_flag, abort_flag,
                                              false, 0u);
                    if (tr) trace_mark(p, TL_TRACE_REDUCED);
                }
            } else {
            // ---- one TMEM accumulator per tile
            // parallel split-k: this split finishes 32-column chunk `split` of the tile.  Its C does
            // not depend on the accumulator: each thread copies its row of it into the warp's
            // output staging buffer (free in this mode) while the tile accumulates.
            bool c_staged = false;
            const uint32_t c_row = my_stage_a + static_cast<uint32_t>(lane) * 128u;
            if constexpr (sizeof(TD) >= 2) {
                constexpr int WC = 32 / NH;           // this warp's columns of the chunk
                const int mc = j.m0 + j.split * 32 + half * WC;
                if (p.par_reduce && half < nst && !j.out_t && j.nsplit > 1 && j.beta != 0.0f && j.C != nullptr &&
                    j.split * 32 < p.bm) {
                    const char* cptr = static_cast<const char*>(j.C) + (base_c + mc) * static_cast<int64_t>(sizeof(TD));
                    if (row_ok && mc + WC <= j.M && (reinterpret_cast<uintptr_t>(cptr) & 15) == 0) {
                        constexpr int NU = WC * static_cast<int>(sizeof(TD)) / 16;
#pragma unroll
                        for (int u = 0; u < NU; ++u)
                            ptx::cp_async16(c_row + static_cast<uint32_t>((u ^ (lane & 7)) * 16), cptr + 16 * u);
                        c_staged = true;
                    }
                    ptx::cp_async_commit();
                }
            }
            // whole tiles with 16-byte accessible D and C leave through this warp's staging buffer, a
            // group of CPS 32-column chunks (128 bytes of output per row) at a time.  C comes in
            // through it too, whole lines at a time like the stores; the first group's C is in flight
            // before the accumulator is ready (D may be C itself: a group's C is read before any of
            // its columns is stored).  A 192-column tile of one-byte outputs ends in half a group: two of
            // its four chunks.
            constexpr int CPS = static_cast<int>(4 / sizeof(TD));
            const int nrow0 = j.n0 + quarter * 32;
            const bool staged = j.vec && j.nsplit == 1 && !j.out_t && chunks >= CPS;
            const bool use_c = j.beta != 0.0f && j.C != nullptr;
            const int groups = half < nst ? (chunks + CPS - 1) / CPS : 0;
            constexpr int WQ = EPI && sizeof(TD) != 1 ? 8 : 16;      // columns finished at a time
            LineAccess<TD> la(lane, j.N - nrow0, sizeof(TD) == 1 ? min(j.M, j.m0 + p.bm) : j.M);
            uint4 cl[8];
            float bl[CPS];
            if constexpr (EPI) {
                if (staged && half < groups) lane_bias<CPS>(p, j.M, j.m0 + half * CPS * 32 + lane, bl);
            }
            if constexpr (sizeof(TD) >= 2) {
                if (staged && use_c && half < groups)
                    la.load(j.C, static_cast<int64_t>(j.b) * p.stride_c + static_cast<int64_t>(nrow0) * j.ldc, j.ldc,
                            j.m0 + half * CPS * 32, cl);
            }
            const uint32_t tbase = tmem_base + lane_off + mbuf * static_cast<uint32_t>(p.bm);
            bool got = ok && ptx::mbar_wait(&tfull[mbuf], mph, tlim);
            got = __all_sync(0xffffffffu, got);
            if (ok && !got) {
                if (lane == 0) record_error(p, abort_flag, 8);
                ok = false;
            }
            if (ok) ptx::tc_fence_after();
            if (tr) trace_mark(p, TL_TRACE_ACC_READY);
            if constexpr (sizeof(TD) >= 2 && !EPI) {
                if (j.out_t && j.nsplit == 1 && j.vec) {
                    // transposed output (beta == 0): a warp's 32 rows are 32 consecutive elements of D's
                    // columns, so each 32-column chunk is staged [column][row] and written in runs of
                    // a column's 64 (16-bit) or 128 bytes
                    constexpr int COLB = 32 * static_cast<int>(sizeof(TD));      // bytes per column
                    constexpr int UPC = COLB / 16, EPU = 16 / static_cast<int>(sizeof(TD));
                    const int u = lane % UPC, col0 = lane / UPC;
                    const bool in_n = nrow0 + u * EPU < j.N;      // N (D's rows here) is whole units
                    if (half >= nst && ok) release_tmem<CG>(&tempty[mbuf], lane);
                    for (int c = half; c < chunks && half < nst && ok; c += nst) {
                        const int m = j.m0 + c * 32;
                        uint32_t r[32];
                        __syncwarp();
                        ptx::tmem_ld32(tbase + c * 32, r);
                        if (c + nst >= chunks) release_tmem<CG>(&tempty[mbuf], lane);
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            const uint32_t a = my_stage_a + static_cast<uint32_t>((i * 32 + lane) * static_cast<int>(sizeof(TD)));
                            const float o = j.alpha * __uint_as_float(r[i]);
                            if constexpr (sizeof(TD) == 4) {
                                ptx::st_shared_u32(a, __float_as_uint(o));
                            } else {
                                uint16_t ob;
                                if constexpr (std::is_same<TD, __half>::value) ob = __half_as_ushort(__float2half_rn(o));
                                else ob = p.out_trunc ? static_cast<uint16_t>(__float_as_uint(o) >> 16)
                                                      : __bfloat16_as_ushort(__float2bfloat16_rn(o));
                                ptx::st_shared_u16(a, ob);
                            }
                        }
                        __syncwarp();
#pragma unroll
                        for (int it = 0; it < UPC; ++it) {
                            const int col = it * (32 / UPC) + col0;
                            const uint4 v = ptx::ld_shared_v4(my_stage_a + static_cast<uint32_t>(col * COLB + u * 16));
                            if (m + col < j.M && in_n)
                                *reinterpret_cast<uint4*>(static_cast<TD*>(j.D) + static_cast<int64_t>(j.b) * p.stride_d +
                                                          static_cast<int64_t>(m + col) * j.ldd + nrow0 + u * EPU) = v;
                        }
                    }
                    if (tr) trace_mark(p, TL_TRACE_STORED);
                    mbuf ^= 1u;
                    if (mbuf == 0) mph ^= 1u;
                    continue;
                }
            }
            if (staged) {
                // 16-byte unit u of row r sits at u ^ (r & 7): rows are written and lines read without
                // bank conflicts.  The columns are finished WQ at a time in a loop that is not unrolled: a
                // tile passes through this code a few times only, and straight-line code for 64 columns
                // ran at the rate of instruction fetch (~580 clocks per 32 columns).
                constexpr int GC = CPS * 32;                     // columns of a group
                constexpr int UPQ = WQ * static_cast<int>(sizeof(TD)) / 16;
                constexpr int CWN = WQ * static_cast<int>(sizeof(TD)) / 4;
                const bool warp_ok = nrow0 < j.N;                // this warp has rows to store
                if (half >= groups && ok) release_tmem<CG>(&tempty[mbuf], lane);
                const uint32_t rowaddr = my_stage_a + static_cast<uint32_t>(lane) * 128u;
                for (int g = half; g < groups && ok; g += nst) {
                    const int m = j.m0 + g * GC;
                    const uint32_t tcol = tbase + static_cast<uint32_t>(g * GC);
                    if (!warp_ok) {
                        if (g + nst >= groups) release_tmem<CG>(&tempty[mbuf], lane);
                        continue;
                    }
                    float bcur[CPS];
                    if constexpr (EPI) {
#pragma unroll
                        for (int t = 0; t < CPS; ++t) bcur[t] = bl[t];
                        if (g + nst < groups) lane_bias<CPS>(p, j.M, m + nst * GC + lane, bl);
                    }
                    if constexpr (sizeof(TD) >= 2) {
                        if (use_c) {
                            la.stage(my_stage_a, cl);
                            __syncwarp();
                            if (g + nst < groups)
                                la.load(j.C, static_cast<int64_t>(j.b) * p.stride_c + static_cast<int64_t>(nrow0) * j.ldc,
                                        j.ldc, m + nst * GC, cl);
                        }
                    }
                    __syncwarp();        // tcgen05.ld is for the whole warp; the loads above are not
                    // only a group of one-byte outputs can be partial (every tile is whole pairs of chunks)
                    const int nq = sizeof(TD) == 1 ? min(GC, p.bm - g * GC) / WQ : GC / WQ;
#pragma unroll 1
                    for (int q = 0; q < nq; ++q) {
                        float o[WQ];
                        ptx::tmem_ld<WQ>(tcol + static_cast<uint32_t>(q * WQ), o);
                        if (q == nq - 1 && g + nst >= groups) release_tmem<CG>(&tempty[mbuf], lane);
                        const uint32_t u0 = static_cast<uint32_t>(q * UPQ);
                        const uint32_t sw = static_cast<uint32_t>(lane & 7);
                        uint32_t cw[WQ];
                        if (use_c) {
#pragma unroll
                            for (int uu = 0; uu < UPQ; ++uu) {
                                const uint4 v = ptx::ld_shared_v4(rowaddr + ((u0 + uu) ^ sw) * 16u);
                                cw[4 * uu] = v.x;
                                cw[4 * uu + 1] = v.y;
                                cw[4 * uu + 2] = v.z;
                                cw[4 * uu + 3] = v.w;
                            }
                        }
                        float bias[WQ];
                        if constexpr (EPI) {
                            float bsel = bcur[0];
#pragma unroll
                            for (int t = 1; t < CPS; ++t) bsel = q * WQ >= 32 * t ? bcur[t] : bsel;
#pragma unroll
                            for (int i = 0; i < WQ; ++i) bias[i] = __shfl_sync(0xffffffffu, bsel, (q * WQ + i) & 31);
                        }
                        finish_values<TD, EPI, WQ>(p, amax, j, m + q * WQ, row_ok, cw, bias, o);
                        uint32_t w[CWN];
                        pack_values<TD, WQ>(p, o, w);
#pragma unroll
                        for (int uu = 0; uu < UPQ; ++uu)
                            ptx::st_shared_v4(rowaddr + ((u0 + uu) ^ sw) * 16u, w[4 * uu], w[4 * uu + 1], w[4 * uu + 2],
                                              w[4 * uu + 3]);
                    }
                    __syncwarp();
                    la.store(j.D, static_cast<int64_t>(j.b) * p.stride_d + static_cast<int64_t>(nrow0) * j.ldd, j.ldd, m,
                             my_stage_a);
                    __syncwarp();
                }
                if (tr) trace_mark(p, TL_TRACE_STORED);
            } else if (j.nsplit == 1) {
                // D or C not made of whole 16-byte vectors (and fp8 tiles narrower than a line)
                for (int c = half; c < chunks && ok; c += NH) {       // at least two chunks: one per warp
                    const int m = j.m0 + c * 32;
                    uint32_t r[32];
                    __syncwarp();
                    ptx::tmem_ld32(tbase + c * 32, r);
                    if (c + NH >= chunks) release_tmem<CG>(&tempty[mbuf], lane);
                    if (row_ok && m < j.M) {
                        float v[32];
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
                        store_chunk<TD, EPI, 32>(p, amax, j, base_c, base_d, m, v);
                    }
                }
                if (tr) trace_mark(p, TL_TRACE_STORED);
            } else {
                // split-k: park this split's partial tile, layout [chunk][column][row] (coalesced)
                float* slab = p.ws + (static_cast<size_t>(j.slot) * p.tail_split + j.split) *
                                         (static_cast<size_t>(kTcTileN) * p.bm);
                for (int c = half; c < chunks && ok; c += NH) {
                    uint32_t r[32];
                    __syncwarp();
                    ptx::tmem_ld32(tbase + c * 32, r);
                    float* dst = slab + static_cast<size_t>(c) * 32 * kTcTileN + row;
#pragma unroll
                    for (int i = 0; i < 32; ++i) __stcg(dst + i * kTcTileN, __uint_as_float(r[i]));
                }
                if (tr) trace_mark(p, TL_TRACE_STORED);
                if (ok) release_tmem<CG>(&tempty[mbuf], lane);
                split_finish<TD, EPI, NH, false>(p, amax, j, ok, et, lane, half, row, row_ok, base_c, base_d, last_flag,
                                          abort_flag, c_staged, c_row);
                if (tr) trace_mark(p, TL_TRACE_REDUCED);
            }
            mbuf ^= 1u;
            if (mbuf == 0) mph ^= 1u;
            }
        }
        if (et == 0) {
            trace_mark(p, TL_TRACE_EPI_END);
            trace_put(p, TL_TRACE_TILES, units_done);
        }
        if constexpr (EPI) {
            if (p.epi_amax != nullptr) {
                // max |output| of the warp, then one atomic per warp (non-negative floats order as ints)
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
                if (lane == 0) atomicMax(reinterpret_cast<int*>(p.epi_amax), __float_as_int(amax));
            }
        }
    }

    ptx::tc_fence_before();
    __syncthreads();
    if constexpr (CL > 1) ptx::cluster_sync();     // no remote arrival, multicast or pair MMA still targets us
    if (warp == 1) {
        ptx::tc_fence_after();
        if constexpr (CG == 2) ptx::tmem_dealloc_pair(tmem_base, tmem_cols);
        else ptx::tmem_dealloc(tmem_base, tmem_cols);
        if (lane == 0 && p.trace != nullptr) {
            trace_mark(p, TL_TRACE_EXIT);
            trace_put(p, TL_TRACE_EXIT_NS, global_ns());
        }
    }
}

// ---- host side ------------------------------------------------------------------------------------
// ---- launch (templates; instantiated in the generated instance units) ---------------------------
bool pdl_enabled();

template <int KIND, typename TD, int CL, bool EPI, int MODE, bool GROUP>
tl_status launch_kernel(const TcKernelParams& kp, int grid, size_t smem, cudaStream_t stream)
{
    auto kern = tc_gemm_kernel<KIND, TD, CL, EPI, MODE, GROUP>;
    static std::once_flag once;
    static cudaError_t attr_err = cudaSuccess;
    std::call_once(once, [&] {
        attr_err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kTcMaxSmem));
    });
    if (attr_err != cudaSuccess) return cuda_fail(attr_err, "cudaFuncSetAttribute(tc_gemm_kernel)");
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(static_cast<unsigned>(grid), 1, 1);
    cfg.blockDim = dim3(tc_threads(MODE), 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (pdl_enabled()) {
        // programmatic dependent launch: this grid's prologue may overlap the previous kernel's tail
        // (the kernel waits for the previous grid before its first global-memory access)
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    if constexpr (CL > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = CL;
        attr[na].val.clusterDim.y = 1;
        attr[na].val.clusterDim.z = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, kp);
    if (e != cudaSuccess) return cuda_fail(e, CL > 1 ? "cudaLaunchKernelEx(tc_gemm_kernel, cluster launch)"
                                                     : "cudaLaunchKernelEx(tc_gemm_kernel)");
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "tc_gemm_kernel launch");
    return TL_SUCCESS;
}

// Number of clusters of CL CTAs that can be resident at once with this shared-memory size (cached).
template <int KIND, typename TD, int CL>
int max_clusters(size_t smem)
{
    static std::mutex mu;
    static std::map<size_t, int> cache;
    std::lock_guard<std::mutex> g(mu);
    auto it = cache.find(smem);
    if (it != cache.end()) return it->second;
    auto kern = tc_gemm_kernel<KIND, TD, CL, false, kModePlain, false>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kTcMaxSmem));
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(CL, 1, 1);
    cfg.blockDim = dim3(tc_threads(kModePlain), 1, 1);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CL;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
        cudaGetLastError();
        n = 0;
    }
    cache[smem] = n;
    return n;
}

}  // namespace tc
}  // namespace tl
