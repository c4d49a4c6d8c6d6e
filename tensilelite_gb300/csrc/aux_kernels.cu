// aux_kernels.cu -- the memory-bound helpers around the GEMM:
//   split_bf16       fp32 -> 2 or 3 bf16 pieces for the FP32-accurate bf16x3 / bf16x6 products
//   amax / quant     per-tensor amax and E4M3 quantisation (scale = 448 / amax)
//   error_norms      FP64 reduction of max|d - r|, max|r| and the componentwise ratio
//   fill_pattern     the reference's deterministic InitRealData codes, on the device
//   scale_c          D = beta * C (the k == 0 GEMM)
// All are grid-stride kernels over 16-byte vectors where the layout allows; grids are multiples of
// the SM count.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include "tl_internal.h"

namespace tl {
namespace tc {
bool pdl_enabled();   // programmatic dependent launch switch, shared with the tensor-core kernel
}
namespace {

int grid_for(int64_t n, int per_thread, int threads)
{
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 132;
    }
    int64_t want = (n + static_cast<int64_t>(per_thread) * threads - 1) / (static_cast<int64_t>(per_thread) * threads);
    const int64_t cap = static_cast<int64_t>(sms) * 8;
    if (want > cap) want = cap;
    if (want < 1) want = 1;
    return static_cast<int>(want);
}

__device__ __forceinline__ float load_as_float(int dtype, const void* p, int64_t i)
{
    switch (dtype) {
    case TL_DTYPE_FP32: return static_cast<const float*>(p)[i];
    case TL_DTYPE_FP16: return __half2float(static_cast<const __half*>(p)[i]);
    case TL_DTYPE_BF16: return __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]);
    case TL_DTYPE_FP8_E4M3: return static_cast<float>(static_cast<const __nv_fp8_e4m3*>(p)[i]);
    default: return 0.f;
    }
}

__device__ __forceinline__ void store_from_float(int dtype, int trunc, void* p, int64_t i, float v)
{
    switch (dtype) {
    case TL_DTYPE_FP32: static_cast<float*>(p)[i] = v; break;
    case TL_DTYPE_FP16: static_cast<__half*>(p)[i] = __float2half_rn(v); break;
    case TL_DTYPE_BF16:
        if (trunc) static_cast<uint16_t*>(p)[i] = static_cast<uint16_t>(__float_as_uint(v) >> 16);
        else static_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v);
        break;
    case TL_DTYPE_FP8_E4M3:
        static_cast<uint8_t*>(p)[i] = static_cast<uint8_t>(__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3));
        break;
    default: break;
    }
}

// ---- split-precision pieces -------------------------------------------------------------------------
// p0 = bf16(x), p1 = bf16(x - p0), p2 = bf16(x - p0 - p1); every subtraction is exact in fp32 (the
// residual of a rounding is representable), so x = p0 + p1 + p2 + O(2^-24 |x|).
template <int NP>
__device__ __forceinline__ void split_pieces(float x, uint16_t (&o)[3])
{
    float r = x;
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        const __nv_bfloat16 b = __float2bfloat16_rn(r);
        o[i] = __bfloat16_as_ushort(b);
        r = r - __bfloat162float(b);
    }
}

// Bound by HBM: 4 bytes read and 2 NP written per element.  Four consecutive elements of a column per
// thread and step, by flat index, so that neither few long columns nor many short ones leave threads
// idle.  The operands of a GEMM are split by two launches that overlap: the second is a programmatic
// dependent of the first and waits for it only before it ends (so what depends on the second
// has both).  RANGE: the operand's magnitudes go to args.range, one pair of atomics per block.
struct SplitArgs {
    SplitOperand op;
    uint32_t* range;
};
template <int NP, bool RANGE>
__global__ void __launch_bounds__(256) split_kernel(const __grid_constant__ SplitArgs args)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    uint32_t most = 0, least = 0xffffffffu;                  // bits of the largest and smallest nonzero |x|
    auto seen = [&](float x) {
        if constexpr (RANGE) {
            const uint32_t u = __float_as_uint(x) & 0x7fffffffu;
            most = max(most, u);
            least = min(least, u - 1u);                       // zero wraps to the largest value
        }
    };
    const SplitOperand& o = args.op;
    const int64_t g = (o.rows + 3) / 4;                       // groups of four per column
    const int64_t total = g * o.cols * o.batch;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    // without gaps in either layout the groups follow each other
    const bool flat = o.rows % 4 == 0 && o.ld == o.rows && o.pld == o.rows &&
                      (o.batch == 1 || (o.batch_stride == o.rows * o.cols && o.p_batch_stride == o.batch_stride));
    const bool small = total < (int64_t(1) << 31);
    bool vec = (reinterpret_cast<uintptr_t>(o.src) & 15) == 0 && (o.cols == 1 || (o.ld % 4 == 0 && o.pld % 4 == 0)) &&
               (o.batch == 1 || (o.batch_stride % 4 == 0 && o.p_batch_stride % 4 == 0));
#pragma unroll
    for (int i = 0; i < NP; ++i) vec = vec && (reinterpret_cast<uintptr_t>(o.p[i]) & 7) == 0;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total; i += stride) {
        int64_t src, dst;
        int left = 4;
        if (flat) {
            src = dst = 4 * i;
        } else {
            int64_t col, r, b = 0;
            if (small) {
                col = static_cast<uint32_t>(i) / static_cast<uint32_t>(g);
            } else {
                col = i / g;
            }
            r = 4 * (i - col * g);
            if (o.batch > 1) {
                b = col / o.cols;
                col -= b * o.cols;
            }
            src = b * o.batch_stride + col * o.ld + r;
            dst = b * o.p_batch_stride + col * o.pld + r;
            left = static_cast<int>(o.rows - r < 4 ? o.rows - r : 4);
        }
        if (vec && left == 4) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(o.src + src));
            seen(v.x);
            seen(v.y);
            seen(v.z);
            seen(v.w);
            uint16_t q[4][3];
            split_pieces<NP>(v.x, q[0]);
            split_pieces<NP>(v.y, q[1]);
            split_pieces<NP>(v.z, q[2]);
            split_pieces<NP>(v.w, q[3]);
#pragma unroll
            for (int pc = 0; pc < NP; ++pc)
                *reinterpret_cast<uint2*>(o.p[pc] + dst) = make_uint2(q[0][pc] | (uint32_t(q[1][pc]) << 16),
                                                                     q[2][pc] | (uint32_t(q[3][pc]) << 16));
        } else {
            for (int t = 0; t < left; ++t) {
                uint16_t q[3];
                const float x = o.src[src + t];
                seen(x);
                split_pieces<NP>(x, q);
#pragma unroll
                for (int pc = 0; pc < NP; ++pc) o.p[pc][dst + t] = q[pc];
            }
        }
    }
    if constexpr (RANGE) {
        __shared__ uint32_t sm[2][8];
        most = __reduce_max_sync(0xffffffffu, most);
        least = __reduce_min_sync(0xffffffffu, least);
        if ((threadIdx.x & 31) == 0) {
            sm[0][threadIdx.x >> 5] = most;
            sm[1][threadIdx.x >> 5] = least;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
#pragma unroll
            for (int w = 1; w < 8; ++w) {
                most = max(most, sm[0][w]);
                least = min(least, sm[1][w]);
            }
            atomicMax(args.range, most);
            if (least != 0xffffffffu) atomicMax(args.range + 1, ~(least + 1u));
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// ---- fp8 ----------------------------------------------------------------------------------------------
// Both passes are bound by memory (the second reads the source from L2 where it fits): 16-byte loads,
// enough of them in flight per SM to cover HBM's latency, and 16-byte stores of 16 quantised elements.
// The three launches are chained as programmatic dependents: a pass starts while the one before it
// drains, and waits for it before it touches what that one writes.  bf16 4096 x 4096: 28.9 us with one
// element per thread and step, of which 7.4 us are the bytes at HBM rate.
template <typename T> struct Vec;      // one 16-byte vector of T as floats
template <> struct Vec<float> {
    static constexpr int N = 4;
    __device__ static __forceinline__ void unpack(const uint4& w, float* f)
    {
        f[0] = __uint_as_float(w.x);
        f[1] = __uint_as_float(w.y);
        f[2] = __uint_as_float(w.z);
        f[3] = __uint_as_float(w.w);
    }
};
template <> struct Vec<__half> {
    static constexpr int N = 8;
    __device__ static __forceinline__ void unpack(const uint4& w, float* f)
    {
        const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 p = __half22float2(*reinterpret_cast<const __half2*>(&u[i]));
            f[2 * i] = p.x;
            f[2 * i + 1] = p.y;
        }
    }
};
template <> struct Vec<__nv_bfloat16> {
    static constexpr int N = 8;
    __device__ static __forceinline__ void unpack(const uint4& w, float* f)
    {
        const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            f[2 * i] = __uint_as_float(u[i] << 16);
            f[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
        }
    }
};
__device__ __forceinline__ float widen(float v) { return v; }
__device__ __forceinline__ float widen(__half v) { return __half2float(v); }
__device__ __forceinline__ float widen(__nv_bfloat16 v) { return __bfloat162float(v); }

// Two blocks of 512 threads per SM with eight 16-byte loads in flight each: 128 KB per SM, and the whole
// grid is resident (four blocks per SM with four loads each left a tail of single loads in a second wave:
// bf16 4096 x 4096 16.9 us on the device against 14.2, fp32 2^24 27.2 against 24.1).
constexpr int kQuantThreads = 512, kQuantBlocks = 2, kQuantFly = 8;

// Elements before the first 16-byte boundary of p.
template <typename T>
__device__ __forceinline__ int64_t head_of(const T* p, int64_t n)
{
    const int64_t h = static_cast<int64_t>(((16 - (reinterpret_cast<uintptr_t>(p) & 15)) & 15) / sizeof(T));
    return h < n ? h : n;
}

__global__ void zero_kernel(float* p)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    *p = 0.f;
}

template <typename T>
__global__ void __launch_bounds__(kQuantThreads, kQuantBlocks) amax_kernel(const T* __restrict__ src, int64_t n, float* amax)
{
    constexpr int N = Vec<T>::N, U = kQuantFly;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    float m = 0.f;
    const int64_t tid = blockIdx.x * static_cast<int64_t>(kQuantThreads) + threadIdx.x;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * kQuantThreads;
    const int64_t head = head_of(src, n), nv = (n - head) / N;
    const uint4* v = reinterpret_cast<const uint4*>(src + head);
    for (int64_t i = tid; i < nv; i += U * stride) {
        uint4 w[U];
#pragma unroll
        for (int u = 0; u < U; ++u) w[u] = i + u * stride < nv ? __ldg(v + i + u * stride) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float f[N];
            Vec<T>::unpack(w[u], f);
#pragma unroll
            for (int k = 0; k < N; ++k) m = fmaxf(m, fabsf(f[k]));
        }
    }
    if (tid < head) m = fmaxf(m, fabsf(widen(src[tid])));
    for (int64_t e = head + nv * N + tid; e < n; e += stride) m = fmaxf(m, fabsf(widen(src[e])));
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ float sm[kQuantThreads / 32];
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < kQuantThreads / 32 ? sm[threadIdx.x] : 0.f;
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        asm volatile("griddepcontrol.wait;" ::: "memory");       // *amax has been zeroed
        if (threadIdx.x == 0) atomicMax(reinterpret_cast<unsigned int*>(amax), __float_as_uint(m));
    }
}

template <typename T>
__global__ void __launch_bounds__(kQuantThreads, kQuantBlocks) quant_kernel(const T* __restrict__ src, int64_t n,
                                                                            const float* __restrict__ amax, uint8_t* dst,
                                                                            float* scale_out)
{
    constexpr int L = static_cast<int>(sizeof(T));            // 16-byte loads per 16 elements
    constexpr int U = kQuantFly / L;                          // 16-element items in flight
    const int64_t tid = blockIdx.x * static_cast<int64_t>(kQuantThreads) + threadIdx.x;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * kQuantThreads;
    const int64_t head = head_of(src, n);
    // whole 16-element items where source and destination are aligned together, else element by element
    const int64_t ni = (reinterpret_cast<uintptr_t>(dst + head) & 15) == 0 ? (n - head) / 16 : 0;
    const uint4* v = reinterpret_cast<const uint4*>(src + head);
    uint4* d = reinterpret_cast<uint4*>(dst + head);
    uint4 w[U][L];
    const auto load = [&](int64_t i) {
#pragma unroll
        for (int t = 0; t < U; ++t)
            if (i + t * stride < ni) {
#pragma unroll
                for (int u = 0; u < L; ++u) w[t][u] = __ldg(v + (i + t * stride) * L + u);
            }
    };
    // the source does not depend on the amax pass: the first items are loaded while that pass ends
    load(tid);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const float a = *reinterpret_cast<const volatile float*>(amax);
    const float s = a > 0.f ? 448.0f / a : 1.0f;
    if (blockIdx.x == 0 && threadIdx.x == 0 && scale_out) *scale_out = a > 0.f ? a / 448.0f : 1.0f;
    auto pack = [&](const uint4* w) {
        uint32_t q[4];
        float f[16];
#pragma unroll
        for (int u = 0; u < L; ++u) Vec<T>::unpack(w[u], f + u * Vec<T>::N);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * k] * s, f[4 * k + 1] * s), __NV_SATFINITE, __NV_E4M3);
            const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * k + 2] * s, f[4 * k + 3] * s), __NV_SATFINITE, __NV_E4M3);
            q[k] = (lo & 0xffffu) | (hi << 16);
        }
        return make_uint4(q[0], q[1], q[2], q[3]);
    };
    for (int64_t i = tid; i < ni; i += U * stride) {
        if (i != tid) load(i);
#pragma unroll
        for (int t = 0; t < U; ++t)
            if (i + t * stride < ni) d[i + t * stride] = pack(w[t]);
    }
    if (tid < head) dst[tid] = static_cast<uint8_t>(__nv_cvt_float_to_fp8(widen(src[tid]) * s, __NV_SATFINITE, __NV_E4M3));
    for (int64_t e = head + ni * 16 + tid; e < n; e += stride)
        dst[e] = static_cast<uint8_t>(__nv_cvt_float_to_fp8(widen(src[e]) * s, __NV_SATFINITE, __NV_E4M3));
}

// ---- error norms ------------------------------------------------------------------------------------
__device__ __forceinline__ void atomic_max_nonneg(double* p, double v)
{
    atomicMax(reinterpret_cast<unsigned long long*>(p), static_cast<unsigned long long>(__double_as_longlong(v)));
}

__global__ void norms_kernel(int dtype, const void* __restrict__ D, int64_t ldd, const double* __restrict__ R,
                             const double* __restrict__ W, int64_t ldr, int64_t m, int64_t n, double* out)
{
    double md = 0.0, mr = 0.0, mc = 0.0;
    const int64_t total = m * n;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; e < total; e += stride) {
        const int64_t i = e % m, j = e / m;
        const double d = static_cast<double>(load_as_float(dtype, D, i + j * ldd));
        const double r = R[i + j * ldr];
        const double diff = fabs(d - r);
        md = fmax(md, diff);
        mr = fmax(mr, fabs(r));
        if (W) {
            const double w = W[i + j * ldr];
            if (w > 0.0) mc = fmax(mc, diff / w);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        md = fmax(md, __shfl_xor_sync(0xffffffffu, md, o));
        mr = fmax(mr, __shfl_xor_sync(0xffffffffu, mr, o));
        mc = fmax(mc, __shfl_xor_sync(0xffffffffu, mc, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomic_max_nonneg(out + 0, md);
        atomic_max_nonneg(out + 1, mr);
        atomic_max_nonneg(out + 2, mc);
    }
}

// ---- patterns ------------------------------------------------------------------------------------
// InitRealData codes (ff_gpu_src/ff_gpu.cpp:110-148) that depend on the flat index only.
__global__ void fill_kernel(int dtype, void* dst, int64_t count, float code)
{
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < count; i += stride) {
        const uint32_t idx = static_cast<uint32_t>(i);
        float v;
        if (code == 0.5f || code == 0.0f) v = 0.f;
        else if (code == 1.0f) v = 1.0f;
        else if (code == 2.0f) v = static_cast<float>(idx);
        else if (code == 2.1f) v = 0.01f * static_cast<float>(idx % 1137u);
        else if (code == 2.3f) v = 0.1f * static_cast<float>(idx % 17u);
        else if (code == 2.4f) v = static_cast<float>(idx % 7u);
        else if (code == -1.0f) v = -1.0f;
        else if (code == -2.0f) v = -static_cast<float>(idx);
        else if (code == -2.1f) v = -0.01f * static_cast<float>(idx % 1137u);
        else if (code == -2.3f) v = -0.1f * static_cast<float>(idx % 17u);
        else if (code == -2.4f) v = -static_cast<float>(idx % 11u);
        else v = code;
        if (dtype == TL_DTYPE_FP8_E4M3)
            static_cast<uint8_t*>(dst)[i] = static_cast<uint8_t>(__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3));
        else
            store_from_float(dtype, 0, dst, i, v);
    }
}

__global__ void scale_c_kernel(int dtype, int trunc, void* D, int64_t ldd, int64_t sd, const void* C, int64_t ldc,
                               int64_t sc, int64_t M, int64_t N, int64_t batch, float beta)
{
    const int64_t total = M * N * batch;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; e < total; e += stride) {
        const int64_t i = e % M, j = (e / M) % N, b = e / (M * N);
        float v = 0.f;
        if (beta != 0.f && C) v = beta * load_as_float(dtype, C, b * sc + i + j * ldc);
        store_from_float(dtype, trunc, D, b * sd + i + j * ldd, v);
    }
}

tl_status check_launch(const char* what, int64_t* launches)
{
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, what);
    if (launches) ++*launches;
    return TL_SUCCESS;
}

}  // namespace

// Launch as a programmatic dependent of the kernel before it in the stream.
template <typename... KArgs, typename... Args>
static cudaError_t launch_dependent(void (*kern)(KArgs...), int grid, int threads, cudaStream_t s, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(grid), 1, 1);
    cfg.blockDim = dim3(static_cast<unsigned>(threads), 1, 1);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    if (tc::pdl_enabled()) {
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

// ---- padded copies --------------------------------------------------------------------------------
// Bound by memory: 2 B read and 2 B written per element.  The source's columns start on any even
// address, so a lane reads the aligned words that lie whole in its eight elements and a half word at either
// end, shifts them into place if they start in the middle of a word, and writes one 16-byte vector.  A warp takes 256 rows of a column
// at a time: one index division per warp and 512 bytes.
struct PadArgs {
    PadOperand op[3];
    int64_t chunks[3], tasks[3];          // 256-row chunks per column; chunks of the operand (0: not there)
};

__global__ void __launch_bounds__(256) pad_kernel(const __grid_constant__ PadArgs args)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x / 32);
    const int64_t total = args.tasks[0] + args.tasks[1] + args.tasks[2];
    for (int64_t t = static_cast<int64_t>(blockIdx.x) * (blockDim.x / 32) + threadIdx.x / 32; t < total; t += warps) {
        int w = 0;
        int64_t i = t;
        while (i >= args.tasks[w]) i -= args.tasks[w++];
        const PadOperand& o = args.op[w];
        int64_t col, b = 0;
        if (i < (int64_t(1) << 31)) col = static_cast<uint32_t>(i) / static_cast<uint32_t>(args.chunks[w]);
        else col = i / args.chunks[w];
        const int64_t r = (i - col * args.chunks[w]) * 256 + lane * 8;
        if (o.batch > 1) {
            b = col / o.cols;
            col -= b * o.cols;
        }
        if (r >= o.rows) continue;
        const uint16_t* src = o.src + b * o.batch_stride + col * o.ld + r;
        uint32_t v[4];
        if (o.rows - r >= 8) {
            load_eight16((reinterpret_cast<uintptr_t>(src) & 2) != 0, [&](int e) { return static_cast<uint32_t>(__ldg(src + e)); },
                         [&](int e) { return __ldg(reinterpret_cast<const uint32_t*>(src + e)); }, v);
        } else {
            const int left = static_cast<int>(o.rows - r);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const uint32_t lo = 2 * e < left ? src[2 * e] : 0u;
                const uint32_t hi = 2 * e + 1 < left ? src[2 * e + 1] : 0u;
                v[e] = lo | (hi << 16);
            }
        }
        *reinterpret_cast<uint4*>(o.dst + b * o.p_batch_stride + col * o.pld + r) = make_uint4(v[0], v[1], v[2], v[3]);
    }
}

// The way back: an aligned 16-byte load per lane, stored to any even address as the words that lie whole
// in the lane's eight elements and a half word at either end.
__global__ void __launch_bounds__(256) unpad_kernel(const __grid_constant__ PadArgs args)
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int lane = threadIdx.x & 31;
    const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x / 32);
    const PadOperand& o = args.op[0];
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * (blockDim.x / 32) + threadIdx.x / 32; i < args.tasks[0]; i += warps) {
        int64_t col, b = 0;
        if (i < (int64_t(1) << 31)) col = static_cast<uint32_t>(i) / static_cast<uint32_t>(args.chunks[0]);
        else col = i / args.chunks[0];
        const int64_t r = (i - col * args.chunks[0]) * 256 + lane * 8;
        if (o.batch > 1) {
            b = col / o.cols;
            col -= b * o.cols;
        }
        if (r >= o.rows) continue;
        const uint4 v = __ldcg(reinterpret_cast<const uint4*>(o.dst + b * o.p_batch_stride + col * o.pld + r));
        const uint32_t q[4] = {v.x, v.y, v.z, v.w};
        uint16_t* out = const_cast<uint16_t*>(o.src) + b * o.batch_stride + col * o.ld + r;
        if (o.rows - r >= 8) {
            if ((reinterpret_cast<uintptr_t>(out) & 2) == 0) {
#pragma unroll
                for (int e = 0; e < 4; ++e) reinterpret_cast<uint32_t*>(out)[e] = q[e];
            } else {
                out[0] = static_cast<uint16_t>(q[0]);
#pragma unroll
                for (int e = 0; e < 3; ++e) reinterpret_cast<uint32_t*>(out + 1)[e] = __funnelshift_r(q[e], q[e + 1], 16);
                out[7] = static_cast<uint16_t>(q[3] >> 16);
            }
        } else {
            const int left = static_cast<int>(o.rows - r);
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (e < left) out[e] = static_cast<uint16_t>(e & 1 ? q[e / 2] >> 16 : q[e / 2]);
        }
    }
}

tl_status aux_split_bf16(const SplitOperand* ops, int count, int pieces, SplitRange* range, cudaStream_t s,
                         int64_t* launches)
{
    bool first = true;
    for (int i = 0; i < count; ++i) {
        const int64_t total = ops[i].rows * ops[i].cols * ops[i].batch;
        if (total == 0) continue;
        const SplitArgs args = {ops[i], range ? reinterpret_cast<uint32_t*>(range) + 2 * i : nullptr};
        const int grid = grid_for(total, 8, 256);
        void (*kern)(SplitArgs) = pieces == 3 ? (range ? split_kernel<3, true> : split_kernel<3, false>) : split_kernel<2, false>;
        if (first) {
            // an ordinary launch: it starts after whatever wrote the operands, or still reads the pieces
            kern<<<grid, 256, 0, s>>>(args);
            const tl_status st = check_launch("split_kernel", launches);
            if (st != TL_SUCCESS) return st;
        } else {
            const cudaError_t e = launch_dependent(kern, grid, 256, s, args);
            if (e != cudaSuccess) return cuda_fail(e, "split_kernel");
            if (launches) ++*launches;
        }
        first = false;
    }
    return TL_SUCCESS;
}

tl_status aux_pad16(const PadOperand* ops, int count, cudaStream_t s, int64_t* launches)
{
    PadArgs args;
    memset(&args, 0, sizeof(args));
    for (int i = 0; i < count; ++i) {
        args.op[i] = ops[i];
        args.chunks[i] = (ops[i].rows + 255) / 256;
        args.tasks[i] = args.chunks[i] * ops[i].cols * ops[i].batch;
    }
    const int64_t total = args.tasks[0] + args.tasks[1] + args.tasks[2];
    if (total == 0) return TL_SUCCESS;
    pad_kernel<<<grid_for(total * 32, 1, 256), 256, 0, s>>>(args);
    return check_launch("pad_kernel", launches);
}

tl_status aux_unpad16(const PadOperand& op, cudaStream_t s, int64_t* launches)
{
    PadArgs args;
    memset(&args, 0, sizeof(args));
    args.op[0] = op;
    args.chunks[0] = (op.rows + 255) / 256;
    args.tasks[0] = args.chunks[0] * op.cols * op.batch;
    const cudaError_t e = launch_dependent(unpad_kernel, grid_for(args.tasks[0] * 32, 1, 256), 256, s, args);
    if (e != cudaSuccess) return cuda_fail(e, "unpad_kernel");
    if (launches) ++*launches;
    return TL_SUCCESS;
}

// Blocks of a quantisation pass over `bytes` of source: at most the resident grid, whose threads stay a
// batch each in step.  A source that L2 does not hold for the second pass is streamed from DRAM twice, and
// there four waves of shorter blocks keep more of it in flight (fp32 2^25 elements 53 -> 49 us; bf16 2^24,
// which L2 holds, would go 14.2 -> 19.6).
static int quant_grid(int64_t bytes, int64_t n, int per_thread)
{
    const int resident = grid_for(INT64_MAX / 2, 1, kQuantThreads) / 8 * kQuantBlocks;
    const int64_t most = bytes >= (int64_t(128) << 20) ? 4 * resident : resident;
    const int64_t want = (n + static_cast<int64_t>(per_thread) * kQuantThreads - 1) / (static_cast<int64_t>(per_thread) * kQuantThreads);
    return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(want, most)));
}

template <typename T>
static tl_status quantize(const T* src, int64_t n, float* amax_dev, uint8_t* dst, float* scale_out, cudaStream_t s,
                          int64_t* launches)
{
    // the zeroing is an ordinary launch: it starts after whatever wrote the source has finished
    zero_kernel<<<1, 1, 0, s>>>(amax_dev);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "zero_kernel");
    if (n > 0) {
        e = launch_dependent(amax_kernel<T>, quant_grid(n * sizeof(T), n, 4 * Vec<T>::N), kQuantThreads, s, src, n, amax_dev);
        if (e != cudaSuccess) return cuda_fail(e, "amax_kernel");
        if (launches) ++*launches;
    }
    e = launch_dependent(quant_kernel<T>, quant_grid(n * sizeof(T), n, 16), kQuantThreads, s, src, n,
                         static_cast<const float*>(amax_dev), dst, scale_out);
    if (e != cudaSuccess) return cuda_fail(e, "quant_kernel");
    if (launches) ++*launches;
    return TL_SUCCESS;
}

tl_status aux_quantize_e4m3(int src_dtype, const void* src, int64_t n, float* amax_dev, uint8_t* dst,
                            float* scale_out_dev, cudaStream_t s, int64_t* launches)
{
    switch (src_dtype) {
    case TL_DTYPE_FP32: return quantize(static_cast<const float*>(src), n, amax_dev, dst, scale_out_dev, s, launches);
    case TL_DTYPE_FP16: return quantize(static_cast<const __half*>(src), n, amax_dev, dst, scale_out_dev, s, launches);
    case TL_DTYPE_BF16: return quantize(static_cast<const __nv_bfloat16*>(src), n, amax_dev, dst, scale_out_dev, s, launches);
    default: return fail(TL_ERR_UNSUPPORTED, "quantize: source must be fp32, fp16 or bf16");
    }
}

tl_status aux_error_norms(int dtype_d, const void* D, int64_t ldd, const double* R, const double* W, int64_t ldr,
                          int64_t m, int64_t n, double* out_dev, cudaStream_t s, int64_t* launches)
{
    TL_CUDA_TRY(cudaMemsetAsync(out_dev, 0, 3 * sizeof(double), s));
    if (m * n == 0) return TL_SUCCESS;
    norms_kernel<<<grid_for(m * n, 8, 256), 256, 0, s>>>(dtype_d, D, ldd, R, W, ldr, m, n, out_dev);
    return check_launch("norms_kernel", launches);
}

tl_status aux_fill_pattern(int dtype, void* dst, int64_t count, float code, cudaStream_t s, int64_t* launches)
{
    if (count == 0) return TL_SUCCESS;
    fill_kernel<<<grid_for(count, 8, 256), 256, 0, s>>>(dtype, dst, count, code);
    return check_launch("fill_kernel", launches);
}

tl_status aux_scale_c(int out_dtype, int out_trunc, void* D, int64_t ldd, int64_t sd, const void* C, int64_t ldc,
                      int64_t sc, int64_t M, int64_t N, int64_t batch, float beta, cudaStream_t s,
                      int64_t* launches)
{
    const int64_t total = M * N * batch;
    if (total == 0) return TL_SUCCESS;
    scale_c_kernel<<<grid_for(total, 8, 256), 256, 0, s>>>(out_dtype, out_trunc, D, ldd, sd, C, ldc, sc, M, N, batch,
                                                           beta);
    return check_launch("scale_c_kernel", launches);
}

}  // namespace tl
