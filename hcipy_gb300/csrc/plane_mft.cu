// Tensor-core form of the plain-precision matrix Fourier transform: the cut phase matrices of a plan, the kernels
// that cut fields into planes, and the two GEMMs of a transform (plane_gemm.cuh describes the arithmetic).
//
// A transform out = alpha L . in . R (in K1 x K2, R K2 x C, L R x K1) runs as
//   1. rows of in, times the source weights along them -> planes (K2 long)
//   2. T^T[c][k1] = sum_k2 in[k1, k2] R[k2, c]          (GEMM over K2, written transposed)
//   3. rows of T^T, times the source weights along them -> planes (K1 long)
//   4. out[r][c] = alpha sum_k1 T^T[c][k1] L[r, k1]     (GEMM over K1, written transposed, with the epilogue)
// for every direction, the fields of a batch stacked along the rows of both GEMMs.
//
// The planes keep their bits below a row's maximum, so what varies along the sum belongs into one operand: the weights of
// a non-uniform source grid multiply the field before it is cut, and the constants are phases of modulus 1.  With the
// weights in the constants, weights over 9 decades (a logarithmic axis) against a field that falls as they rise lost
// all but 12 bits of complex64 and 28 of complex128.
#include "plane_mft.cuh"
#include "plane_gemm.cuh"

#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>

namespace hx {
using namespace pg;
namespace {

// ---- cutting values into planes -----------------------------------------------------------------------------

// Floating planes: power of two s with |x| / s <= 2^15 for every |x| <= mx.  The fp16 value h of x / s then leaves room for a
// second one of the same weight, x / s - h, whose 11 bits are normal down to 2^-18 of the row's maximum.  s and 1 / s are
// normal floats, and a row below 2^-111 keeps every bit of its subnormal values.
__device__ __forceinline__ float plane_scale(float mx) {
    if (!(mx > 0.0f)) return 1.0f;
    int e = 128;  // infinities: the planes then hold infinities and NaNs
    if (isfinite(mx)) frexpf(mx, &e);
    return ldexpf(1.0f, max(e, -111) - 15);
}

// Digits: exponent E with |x| <= 2^E for every |x| whose bit pattern is at most mx.
__device__ __forceinline__ int plane_exponent(unsigned long long mx) {
    const int e = (int)(mx >> 52);
    if (e == 0x7ff) return NAN_EXP;
    if (mx == 0) return 0;
    return max(e - 1023 + ((mx & 0xfffffffffffffull) != 0), -1022);
}

// The same for a float's.
__device__ __forceinline__ int plane_exponent(unsigned int mx) {
    const int e = (int)(mx >> 23);
    if (e == 0xff) return NAN_EXP;
    if (mx == 0) return 0;
    if (e == 0) return 32 - __clz((int)mx) - 149;
    return e - 127 + ((mx & 0x7fffffu) != 0);
}

// x 2^(55 - E) rounded to an integer (|x| <= 2^E).
__device__ __forceinline__ long long to_fixed(double x, int E) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    int e = (int)((b >> 52) & 0x7ff);
    unsigned long long m = b & 0xfffffffffffffull;
    if (e) m |= 0x10000000000000ull;
    else e = 1;
    const int sh = e - 1020 - E;  // m 2^(e - 1075) 2^(55 - E)
    unsigned long long q;
    if (sh >= 0) q = m << sh;
    else if (sh < -53) q = 0;
    else q = (m + (1ull << (-sh - 1))) >> -sh;
    return (b >> 63) ? -(long long)q : (long long)q;
}

// The planes of four consecutive real values: out[p] holds them as four halves.
__device__ __forceinline__ void cut4(C64Floats, const float* x, float inv, uint2* out) {
    __half2 h[2], l[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const float a = x[2 * q] * inv, b = x[2 * q + 1] * inv;
        h[q] = __floats2half2_rn(a, b);
        const float2 f = __half22float2(h[q]);
        l[q] = __floats2half2_rn(a - f.x, b - f.y);
    }
    out[0] = make_uint2(*reinterpret_cast<uint32_t*>(&h[0]), *reinterpret_cast<uint32_t*>(&h[1]));
    out[1] = make_uint2(*reinterpret_cast<uint32_t*>(&l[0]), *reinterpret_cast<uint32_t*>(&l[1]));
}

// v = x 2^(26 - E) (in two exact steps, since 2^(26 - E) itself may be out of range) is 2^9 h and a rest of 256 at most: h, an
// integer of 18 bits, makes digits 0 and 1 (with 256 added to each, its bits 9 up and 0-8), the rest is digit 2, rounded
// to the 11 bits of an fp16 value.
__device__ __forceinline__ void cut4(C64Digits, const float* x, int E, uint2* out) {
    const int k = E == NAN_EXP ? 0 : 26 - E, k1 = min(k, 120);
    const float f1 = __int_as_float((k1 + 127) << 23), f2 = __int_as_float((k - k1 + 127) << 23);
    uint32_t q[4];
    float r[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float v = E == NAN_EXP ? 0.0f : x[j] * f1 * f2;
        const int h = __float2int_rn(v * 0x1p-9f);
        q[j] = (uint32_t)h + 0x20100u;
        r[j] = fmaf((float)h, -512.0f, v);
    }
    const __half2 bias = __halves2half2(__ushort_as_half(0x6500), __ushort_as_half(0x6500));  // 1024 + 256
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        uint32_t w[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint32_t a = p == 0 ? q[2 * i] >> 9 : q[2 * i] & 0x1ff;
            const uint32_t b = p == 0 ? q[2 * i + 1] >> 9 : q[2 * i + 1] & 0x1ff;
            const uint32_t u = 0x64006400u + (a | (b << 16));  // the halves 1024 + digit + 256
            const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&u), bias);
            w[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
        out[p] = make_uint2(w[0], w[1]);
    }
    const __half2 l0 = __floats2half2_rn(r[0], r[1]), l1 = __floats2half2_rn(r[2], r[3]);
    out[2] = make_uint2(*reinterpret_cast<const uint32_t*>(&l0), *reinterpret_cast<const uint32_t*>(&l1));
}

__device__ __forceinline__ void cut4(C128Digits, const double* x, int E, uint2* out) {
    unsigned long long q[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)  // each digit + 128: bytes 0-5 are planes 6-1, what is left of byte 6 up plane 0
        q[j] = (unsigned long long)(E == NAN_EXP ? 0ll : to_fixed(x[j], E)) + 0x0080808080808080ull;
    const __half2 bias = __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480));  // 1024 + 128
#pragma unroll
    for (int p = 0; p < 7; ++p) {
        uint32_t w[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const uint32_t a = p == 0 ? (uint32_t)(q[2 * k] >> 48) & 0x1ff : (uint32_t)(q[2 * k] >> (48 - 8 * p)) & 0xff;
            const uint32_t b =
                p == 0 ? (uint32_t)(q[2 * k + 1] >> 48) & 0x1ff : (uint32_t)(q[2 * k + 1] >> (48 - 8 * p)) & 0xff;
            const uint32_t u = 0x64006400u + (a | (b << 16));  // the halves 1024 + digit + 128
            const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&u), bias);
            w[k] = *reinterpret_cast<const uint32_t*>(&h);
        }
        out[p] = make_uint2(w[0], w[1]);
    }
}

template <typename T> struct MaxBits;
template <> struct MaxBits<float> {
    using V = unsigned int;
    __device__ static V of(float x) { return __float_as_uint(x) & 0x7fffffffu; }
};
template <> struct MaxBits<double> {
    using V = unsigned long long;
    __device__ static V of(double x) { return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull; }
};

// The scale of a row from the bit pattern of its maximum, and what cut4 takes of it.
__device__ __forceinline__ float row_scale(C64Floats, unsigned int m) {
    return plane_scale(__uint_as_float(min(m, 0x7f800000u)));
}
template <typename F, typename V> __device__ __forceinline__ int row_scale(F, V m) { return plane_exponent(m); }
__device__ __forceinline__ float cut_factor(float s) { return 1.0f / s; }
__device__ __forceinline__ int cut_factor(int e) { return e; }

template <typename V> __device__ __forceinline__ V block_max(V m, V* red) {
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    m = red[0];
    for (int i = 1; i < (int)(blockDim.x >> 5); ++i) m = max(m, red[i]);
    return m;
}

// Four consecutive complex values from a row of K (16-byte loads where the address allows them), zeros past K.
__device__ __forceinline__ void load4(const float2* p, int k0, int K, float* re, float* im) {
    if (k0 + 4 <= K && (reinterpret_cast<uintptr_t>(p + k0) & 15) == 0) {
        const float4 a = reinterpret_cast<const float4*>(p + k0)[0], b = reinterpret_cast<const float4*>(p + k0)[1];
        re[0] = a.x, im[0] = a.y, re[1] = a.z, im[1] = a.w, re[2] = b.x, im[2] = b.y, re[3] = b.z, im[3] = b.w;
        return;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 v = k0 + j < K ? p[k0 + j] : make_float2(0.0f, 0.0f);
        re[j] = v.x, im[j] = v.y;
    }
}
__device__ __forceinline__ void load4(const double2* p, int k0, int K, double* re, double* im) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const double2 v = k0 + j < K ? p[k0 + j] : make_double2(0.0, 0.0);
        re[j] = v.x, im[j] = v.y;
    }
}

// One CTA per row of K complex values: the row's scale, and its planes [Re | Im], each Kp long with zeros past K.
// Four values per thread and step, kept in registers between the maximum and the cut up to G steps (a longer row is
// read twice), so the pass is bound by the bytes it moves: 8 B in and 12 B (8 B) out per complex64 value, 16 and 28 B per
// complex128 value.  W: value k of a row is multiplied by wk[k].
template <typename F, int G, bool W>
__global__ void __launch_bounds__(256) plane_rows_kernel(const typename cplx<typename Shape<F>::T>::type* __restrict__ in,
                                                         long long ld, int K, int Kp,
                                                         const typename Shape<F>::T* __restrict__ wk,
                                                         __half* __restrict__ planes, long long plane_stride,
                                                         int kpitch,
                                                         typename Shape<F>::Scale* __restrict__ scale_out) {
    using T = typename Shape<F>::T;
    using MB = MaxBits<T>;
    constexpr int NP = Shape<F>::NP;
    __shared__ typename MB::V red[8];
    auto load = [&](const typename cplx<T>::type* p, int k0, T* a, T* b) {
        load4(p, k0, K, a, b);
        if constexpr (W) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const T w = k0 + j < K ? __ldg(&wk[k0 + j]) : T(0);
                a[j] *= w;
                b[j] *= w;
            }
        }
    };
    const long long m = blockIdx.x;
    const typename cplx<T>::type* row = in + m * ld;
    const int step = 4 * blockDim.x;
    T re[G][4], im[G][4];
    typename MB::V mx = 0;
#pragma unroll
    for (int g = 0; g < G; ++g) {
        load(row, 4 * threadIdx.x + g * step, re[g], im[g]);
#pragma unroll
        for (int j = 0; j < 4; ++j) mx = max(mx, max(MB::of(re[g][j]), MB::of(im[g][j])));
    }
    for (int k0 = 4 * threadIdx.x + G * step; k0 < K; k0 += step) {
        T a[4], b[4];
        load(row, k0, a, b);
#pragma unroll
        for (int j = 0; j < 4; ++j) mx = max(mx, max(MB::of(a[j]), MB::of(b[j])));
    }
    const auto s = row_scale(F(), block_max(mx, red));
    if (threadIdx.x == 0) scale_out[m] = s;
    const auto f = cut_factor(s);
    auto put = [&](int k0, const T* a, const T* b) {
        uint2 cr[NP], ci[NP];
        cut4(F(), a, f, cr);
        cut4(F(), b, f, ci);
        __half* dst = planes + m * kpitch + k0;
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            *reinterpret_cast<uint2*>(dst + p * plane_stride) = cr[p];
            *reinterpret_cast<uint2*>(dst + p * plane_stride + Kp) = ci[p];
        }
    };
#pragma unroll
    for (int g = 0; g < G; ++g) {
        const int k0 = 4 * threadIdx.x + g * step;
        if (k0 < Kp) put(k0, re[g], im[g]);
    }
    for (int k0 = 4 * threadIdx.x + G * step; k0 < Kp; k0 += step) {
        T a[4], b[4];
        load(row, k0, a, b);
        put(k0, a, b);
    }
}

// One CTA per column n of a constant operand V[n][k] = wn[n] exp(sign i a[n] b[k]), evaluated in float64 as the phase
// matrices of the CUDA-core form are: the rows [Re | -Im] and [Im | Re] of its embedding.
template <typename F>
__global__ void __launch_bounds__(256) plane_const_kernel(int K, int Kp, const double* __restrict__ a,
                                                          const double* __restrict__ b, double sign,
                                                          const double* __restrict__ wn, __half* __restrict__ planes,
                                                          long long plane_stride, int kpitch,
                                                          typename Shape<F>::Scale* __restrict__ scale_out) {
    using T = typename Shape<F>::T;
    using MB = MaxBits<T>;
    constexpr int NP = Shape<F>::NP;
    const int n = blockIdx.x;
    const double w = wn ? wn[n] : 1.0;
    const auto s = row_scale(F(), MB::of((T)w));  // both parts are at most |w|
    if (threadIdx.x == 0) scale_out[n] = s;
    const auto f = cut_factor(s);
    const long long r_re = (long long)(n >> 3) * 16 + (n & 7), r_im = r_re + 8;
    for (int k0 = 4 * threadIdx.x; k0 < Kp; k0 += 4 * blockDim.x) {
        T re[4], im[4], ni[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = k0 + j;
            double sn = 0.0, co = 0.0;
            if (k < K) {
                sincos(a[n] * b[k], &sn, &co);
                co *= w;
                sn *= w * sign;
            }
            re[j] = (T)co;
            im[j] = (T)sn;
            ni[j] = -im[j];
        }
        uint2 cr[NP], ci[NP], cn[NP];
        cut4(F(), re, f, cr);
        cut4(F(), im, f, ci);
        cut4(F(), ni, f, cn);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            __half* pl = planes + p * plane_stride;
            *reinterpret_cast<uint2*>(pl + r_re * kpitch + k0) = cr[p];
            *reinterpret_cast<uint2*>(pl + r_re * kpitch + Kp + k0) = cn[p];
            *reinterpret_cast<uint2*>(pl + r_im * kpitch + k0) = ci[p];
            *reinterpret_cast<uint2*>(pl + r_im * kpitch + Kp + k0) = cr[p];
        }
    }
}

// Weights of a source axis in the fields' type.
template <typename T> __global__ void plane_weights_kernel(int K, const double* __restrict__ w, T* __restrict__ out) {
    for (int k = threadIdx.x; k < K; k += blockDim.x) out[k] = (T)w[k];
}

// ---- host side ----------------------------------------------------------------------------------------------

inline long long round_up(long long x, long long m) { return (x + m - 1) / m * m; }

PFN_cuTensorMapEncodeTiled_v12000 get_encode() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, []() {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

// An operand in planes: NP planes of rows x kpitch halves, one scale per complex row or column.
struct PlaneMat {
    __half* planes = nullptr;
    void* scale = nullptr;
    long long rows = 0;
    int K = 0, Kp = 0, kpitch = 0;
    int n = 0;  // complex columns of a constant operand
    bool digits = true;
    CUtensorMap map;  // of a constant operand, encoded once
    long long plane_stride() const { return rows * kpitch; }
};

struct Carver {
    uint8_t* base;
    size_t off = 0;
    explicit Carver(void* b) : base((uint8_t*)b) {}
    void* take(size_t bytes) {
        off = (off + 255) / 256 * 256;
        void* p = base ? base + off : nullptr;
        off += bytes;
        return p;
    }
};

// The form of complex64 operands.  Floating planes take half the products of digits, but what their truncated sums lose adds up
// along a chain of transforms, beside the CUDA cores' error, which grows with the sums.  Gradients in FP32 through a Lyot
// coronagraph and an image (512^2 and 256^2 points, six transforms of two products) are off by, in 1e-7:
//   pupil                  all digits   as below   second products   all floating   CUDA cores
//   512^2                     0.8         2.9           3.0              4.0           3.5
//   256^2                     0.9         2.8           4.0              5.3           3.5
//   400^2                     1.1         2.6           3.0              3.5           2.6
//   700^2                     0.9         2.9                            3.8           3.3
//   1024^2                    1.2                                        3.7           4.6
//   (the step, 64 of 512^2)  4.7 ms       4.5           4.2              3.8            13
// Images of Lyot coronagraphs (511^2 to 700^2 pupils) are off by 1.0-5.9, 5.0-6.8, 5.5-6.6, 7.6-10 and 14-24, and a pass over
// four 700^2 fields takes 326, 313, 285, 255 and 1022 us.  The plain form is to be as near as the CUDA cores everywhere, at
// the least time (nearer still is what the split form is for): up to 960 points a side digits in both products of the forward
// direction and in the second of the others, floating planes beyond.  Short sums take digits always: a sum of few partial
// sums has no mean loss to take back (see Sums<C64Floats>), and its GEMM is not bound by its products.
inline bool takes_digits(int K, int longest, int direction, bool second) {
    return K <= 128 || (longest <= 960 && (second || direction == HX_FORWARD));
}

// fn with the form as a value of its type.
template <typename T, typename Fn> auto with_form(bool digits, Fn&& fn) {
    if constexpr (sizeof(T) == 8) return fn(C128Digits());
    else return digits ? fn(C64Digits()) : fn(C64Floats());
}

template <typename F> void carve_mat(Carver& c, PlaneMat& m, long long rows, long long scales, int K) {
    m.K = K;
    m.Kp = (int)round_up(K, 32);
    m.kpitch = 2 * m.Kp;
    m.rows = rows;
    m.planes = (__half*)c.take(sizeof(__half) * Shape<F>::NP * (size_t)rows * m.kpitch);
    m.scale = c.take(sizeof(typename Shape<F>::Scale) * (size_t)scales);
}

template <typename F> int encode_map(CUtensorMap* map, const PlaneMat& m, int box_rows) {
    auto enc = get_encode();
    if (!enc) {
        set_error("cuTensorMapEncodeTiled is not available from the driver");
        return HX_ERR_UNSUPPORTED;
    }
    cuuint64_t dims[3] = {(cuuint64_t)m.kpitch, (cuuint64_t)m.rows, (cuuint64_t)Shape<F>::NP};
    cuuint64_t strides[2] = {(cuuint64_t)m.kpitch * 2, (cuuint64_t)m.rows * m.kpitch * 2};
    cuuint32_t box[3] = {(cuuint32_t)Shape<F>::BK, (cuuint32_t)box_rows, (cuuint32_t)Shape<F>::NP};
    cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, m.planes, dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE,
                           Layout<F>::ROW_BYTES == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed (%d) for %lld rows x %d", (int)r, m.rows, m.kpitch);
        return HX_ERR_CUDA;
    }
    return HX_OK;
}

template <typename F>
int launch_rows(const void* in, long long rows, int K, const void* wk, const PlaneMat& m, cudaStream_t st) {
    using T = typename Shape<F>::T;
    using Cx = typename cplx<T>::type;
    using Sc = typename Shape<F>::Scale;
    const int threads = std::min<int>(256, (int)round_up((m.Kp + 3) / 4, 32));
    const int steps = (m.Kp + 4 * threads - 1) / (4 * threads);
    const unsigned grid = (unsigned)rows;
    auto run = [&](auto g, auto weighted) {
        plane_rows_kernel<F, decltype(g)::value, decltype(weighted)::value><<<grid, threads, 0, st>>>(
            (const Cx*)in, K, K, m.Kp, (const T*)wk, m.planes, m.plane_stride(), m.kpitch, (Sc*)m.scale);
    };
    if (wk) run(std::integral_constant<int, 1>(), std::true_type());
    else if (steps == 1) run(std::integral_constant<int, 1>(), std::false_type());
    else if (steps == 2) run(std::integral_constant<int, 2>(), std::false_type());
    else run(std::integral_constant<int, 4>(), std::false_type());
    return launch_status("plane_rows_kernel");
}

// Whether clusters of ks CTAs of the GEMM can be resident on this device.
template <typename F> bool cluster_ok(int ks) {
    static int cache[64][9];  // per device: 0 unknown, 1 yes, 2 no
    static const bool off = [] {  // HX_NO_CLUSTERS=1: no K split (tests of that path)
        const char* e = getenv("HX_NO_CLUSTERS");
        return e && e[0] == '1';
    }();
    int dev = 0;
    if (off || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    if (!cache[dev][ks]) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)ks);
        cfg.blockDim = dim3(Layout<F>::THREADS);
        cfg.dynamicSmemBytes = Layout<F>::SMEM;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)ks;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        const bool ok = cudaFuncSetAttribute(plane_gemm_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             Layout<F>::SMEM) == cudaSuccess &&
                        cudaOccupancyMaxActiveClusters(&n, plane_gemm_kernel<F>, &cfg) == cudaSuccess && n > 0;
        cudaGetLastError();
        cache[dev][ks] = ok ? 1 : 2;
    }
    return cache[dev][ks] == 1;
}

// CTAs along K per tile: enough to occupy the SMs, each with at least 256 terms of K' (128 in complex128), below which the
// exchange costs more than the shorter chain saves.
template <typename F> int k_split(long long tiles, int ktiles, bool throughput) {
    if (throughput) return 1;
    const int parts = (ktiles + Shape<F>::CT - 1) / Shape<F>::CT;
    constexpr int least = std::is_same<F, C64Floats>::value ? 4 : 1;
    for (int ks : {8, 4, 2})
        if (tiles * ks <= num_sms() && parts / ks >= least && cluster_ok<F>(ks)) return ks;
    return 1;
}

template <typename F> int launch_gemm(PlaneArgs<F>& g, const PlaneMat& a, const PlaneMat& b, bool throughput,
                                      double cmacs, cudaStream_t st) {
    using LY = Layout<F>;
    HX_TRY(encode_map<F>(&g.tmap_a, a, BM));
    g.tmap_b = b.map;
    static bool configured[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        HX_TRY(cuda_status(cudaFuncSetAttribute(plane_gemm_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                LY::SMEM),
                           "cudaFuncSetAttribute(plane_gemm_kernel)"));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    g.M = (int)a.rows;
    g.N = b.n;
    g.alpha_kind = g.alpha.y == 0 ? (g.alpha.x == 1 ? 0 : 1) : g.alpha.x == 0 ? 2 : 3;
    g.row_scale = (const typename Shape<F>::Scale*)a.scale;
    g.col_scale = (const typename Shape<F>::Scale*)b.scale;
    g.ktiles = a.kpitch / Shape<F>::BK;
    g.stall = fault_injected("wait");
    g.wait_limit = g.stall ? 10000000ull : WAIT_LIMIT;
    g.n_tiles = (int)ceil_div(b.n, LY::TN);
    const unsigned m_tiles = ceil_div(a.rows, BM);
    g.ksplit = k_split<F>((long long)m_tiles * g.n_tiles, g.ktiles, throughput);
    TraceScope trace(HX_TRACE_SIMT_GEMM, cmacs, st);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(g.n_tiles * g.ksplit), m_tiles);
    cfg.blockDim = dim3(Layout<F>::THREADS);
    cfg.dynamicSmemBytes = LY::SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)g.ksplit;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g.ksplit > 1 ? 1 : 0;
    HX_TRY(cuda_status(cudaLaunchKernelEx(&cfg, plane_gemm_kernel<F>, g), "plane_gemm_kernel"));
    return launch_status("plane_gemm_kernel");
}

}  // namespace

struct PlaneMft {
    int dtype, nx, ny, nu, nv;
    void* mem = nullptr;
    PlaneMat rgt[3], lft[3];  // by direction: the operand along x (R) and the one along y (L)
    void* wk2[3] = {};        // weights along the rows of the field (K2 of them) and of T^T (K1), or nullptr
    void* wk1[3] = {};
    int* status = nullptr;
};

namespace {

// The source plane (K1 x K2) and the destination plane (R x C) of a direction.
struct Dims {
    int K1, K2, R, C, direction;
    int longest() const { return std::max(std::max(K1, K2), std::max(R, C)); }
    bool digits(bool second) const { return takes_digits(second ? K1 : K2, longest(), direction, second); }
};
Dims dims_of(const PlaneMft* p, int direction) {
    if (direction == HX_FORWARD) return {p->ny, p->nx, p->nv, p->nu, direction};
    return {p->nv, p->nu, p->ny, p->nx, direction};
}

// Fields per pass: the scratch of a pass stays within 4 GB.
template <typename T> struct Pass {
    PlaneMat s1, s2;
    void* t = nullptr;
    void* parts = nullptr;  // partial sums of a K split
    size_t bytes = 0;
    int fields = 1;
};

template <typename T> size_t carve_pass(void* ws, const Dims& d, int fields, Pass<T>* out) {
    Carver c((void*)(((uintptr_t)ws + 255) / 256 * 256));  // TMA wants 16 bytes; a caller's scratch may start anywhere
    Pass<T> q;
    const long long r1 = (long long)fields * d.K1, r2 = (long long)fields * d.C;
    auto mat = [&](PlaneMat& m, long long rows, int K, bool digits) {
        m.digits = digits;
        with_form<T>(m.digits, [&](auto f) { carve_mat<decltype(f)>(c, m, rows, rows, K); });
    };
    mat(q.s1, r1, d.K2, d.digits(false));
    q.t = c.take(2 * sizeof(T) * (size_t)r2 * d.K1);
    mat(q.s2, r2, d.K1, d.digits(true));
    auto part_bytes = [&](const PlaneMat& a, int N) {
        return with_form<T>(a.digits, [&](auto f) {
            using F = decltype(f);
            const long long tiles = (long long)ceil_div(a.rows, BM) * ceil_div(N, Layout<F>::TN);
            const int ks = k_split<F>(tiles, a.kpitch / Shape<F>::BK, false);
            return ks > 1 ? (size_t)tiles * ks * Layout<F>::TN * 2 * BM * sizeof(typename Shape<F>::Acc) : (size_t)0;
        });
    };
    q.parts = c.take(std::max(part_bytes(q.s1, d.C), part_bytes(q.s2, d.R)));
    q.bytes = c.off + 255;
    q.fields = fields;
    if (out) *out = q;
    return q.bytes;
}

template <typename T> int fields_per_pass(const Dims& d, int batch) {
    const size_t one = carve_pass<T>(nullptr, d, 1, nullptr);
    // rows of either GEMM: grid y takes 65535 tiles
    const long long rows = 65535ll * BM / std::max(d.K1, d.C);
    return (int)std::max<long long>(1, std::min<long long>({batch, rows, (long long)(((size_t)4 << 30) / one)}));
}

// Where the tensor-core form is the faster one, transforms that the one-launch form takes aside: its four launches take 33
// to 45 us however small.  On the CUDA cores a pair of GEMMs takes 0.075 us for each term of its two sums (one after
// the other: 384^2 -> 192^2 60 us, 700^2 -> 100^2 103 us, 1001 x 501 -> 33^2 109 us in complex64), or what its products
// take where they are many and the sums short (700^2 <- 100^2, 5.6e7 products, 31 us).  complex128 there waits for the
// float64 pipe: 50^2 -> 50^2 (2.5e5 products) 123 us against 42, 16 fields of 64^2 -> 32^2 141 against 45.
template <typename T> bool takes(const Dims& d, int batch) {
    if (std::min(std::min(d.K1, d.K2), std::min(d.R, d.C)) < 16) return false;
    const double cmacs = (double)batch * ((double)d.K1 * d.K2 * d.C + (double)d.R * d.K1 * d.C);
    return sizeof(T) == 4 ? cmacs >= 6e7 || d.K1 + d.K2 >= 600 : cmacs >= 1e5;
}

template <typename T> int make_const(PlaneMat& m, int N, const double* a, const double* b, double sign,
                                     const double* wn, cudaStream_t st) {
    m.n = N;
    if (fault_injected("operand_map")) return HX_ERR_INJECTED;
    return with_form<T>(m.digits, [&](auto f) {
        using F = decltype(f);
        HX_TRY(encode_map<F>(&m.map, m, Shape<F>::BN));
        plane_const_kernel<F><<<(unsigned)N, 256, 0, st>>>(m.K, m.Kp, a, b, sign, wn, m.planes, m.plane_stride(), m.kpitch,
                                                           (typename Shape<F>::Scale*)m.scale);
        return launch_status("plane_const_kernel");
    });
}

template <typename T>
int create_t(PlaneMft* p, const double* x, const double* y, const double* u, const double* v, const double* wx,
             const double* wy, const double* wu, const double* wv, cudaStream_t st) {
    const bool own_adjoint = wx || wy || wu || wv;
    auto layout = [&](Carver& c) {
        for (int d = 0; d < (own_adjoint ? 3 : 2); ++d) {
            const Dims q = dims_of(p, d);
            auto mat = [&](PlaneMat& m, int columns, int K, bool digits) {
                m.digits = digits;
                with_form<T>(m.digits, [&](auto f) { carve_mat<decltype(f)>(c, m, 2 * round_up(columns, 8), columns, K); });
            };
            mat(p->rgt[d], q.C, q.K2, q.digits(false));
            mat(p->lft[d], q.R, q.K1, q.digits(true));
        }
        auto weights = [&](const double* w, int n) { return w ? c.take(sizeof(T) * (size_t)n) : nullptr; };
        p->wk2[HX_FORWARD] = weights(wx, p->nx);
        p->wk1[HX_FORWARD] = weights(wy, p->ny);
        p->wk2[HX_BACKWARD] = weights(wu, p->nu);
        p->wk1[HX_BACKWARD] = weights(wv, p->nv);
        p->status = (int*)c.take(sizeof(int));
    };
    Carver count(nullptr);
    layout(count);
    const cudaError_t mem = fault_injected("operand_memory") ? cudaErrorMemoryAllocation : cudaMalloc(&p->mem, count.off);
    if (mem == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        return HX_ERR_ALLOC;
    }
    HX_TRY(cuda_status(mem, "cudaMalloc(plane MFT plan)"));
    HX_TRY(cuda_status(cudaMemsetAsync(p->mem, 0, count.off, st), "memset plane MFT plan"));
    Carver c(p->mem);
    layout(c);
    HX_TRY(make_const<T>(p->rgt[HX_FORWARD], p->nu, u, x, -1.0, nullptr, st));
    HX_TRY(make_const<T>(p->lft[HX_FORWARD], p->nv, v, y, -1.0, nullptr, st));
    HX_TRY(make_const<T>(p->rgt[HX_BACKWARD], p->nx, x, u, +1.0, nullptr, st));
    HX_TRY(make_const<T>(p->lft[HX_BACKWARD], p->ny, y, v, +1.0, nullptr, st));
    auto weights = [&](void* out, int n, const double* w) {
        if (!out) return (int)HX_OK;
        plane_weights_kernel<T><<<1, 256, 0, st>>>(n, w, (T*)out);
        return launch_status("plane_weights_kernel");
    };
    HX_TRY(weights(p->wk2[HX_FORWARD], p->nx, wx));
    HX_TRY(weights(p->wk1[HX_FORWARD], p->ny, wy));
    HX_TRY(weights(p->wk2[HX_BACKWARD], p->nu, wu));
    HX_TRY(weights(p->wk1[HX_BACKWARD], p->nv, wv));
    if (own_adjoint) {
        HX_TRY(make_const<T>(p->rgt[HX_ADJOINT], p->nx, x, u, +1.0, wx, st));
        HX_TRY(make_const<T>(p->lft[HX_ADJOINT], p->ny, y, v, +1.0, wy, st));
    } else {
        p->rgt[HX_ADJOINT] = p->rgt[HX_BACKWARD];
        p->lft[HX_ADJOINT] = p->lft[HX_BACKWARD];
    }
    return HX_OK;
}

template <typename T>
int execute_t(const PlaneMft* p, int direction, int batch, const void* in, void* out, double are, double aim,
              int epilogue, const void* mask, const void* src, bool throughput, void* ws, cudaStream_t st) {
    using Cx = typename cplx<T>::type;
    const Dims d = dims_of(p, direction);
    const int per = fields_per_pass<T>(d, batch);
    // Fields that grow are taken from the last on: a result written over its own input (out == in) then lies past the inputs
    // of the passes still to come; fields that shrink lie before them.
    const bool grow = (long long)d.R * d.C > (long long)d.K1 * d.K2;
    const int passes = (batch + per - 1) / per;
    for (int i = 0; i < passes; ++i) {
        const int b0 = (grow ? passes - 1 - i : i) * per, nb = std::min(per, batch - b0);
        Pass<T> q;
        carve_pass<T>(ws, d, nb, &q);
        const long long oplane = (long long)d.R * d.C;
        // cut the rows of `from`, then multiply them with a constant
        auto product = [&](const void* from, long long rows, const void* wk, const PlaneMat& a, const PlaneMat& b,
                           double cmacs, auto&& set) {
            return with_form<T>(a.digits, [&](auto f) {
                using F = decltype(f);
                HX_TRY(launch_rows<F>(from, rows, a.K, wk, a, st));
                PlaneArgs<F> g;
                memset(&g, 0, sizeof(g));
                g.parts = (typename Shape<F>::Acc*)q.parts;
                g.status = p->status;
                set(g);
                return launch_gemm<F>(g, a, b, throughput, cmacs, st);
            });
        };
        HX_TRY(product((const Cx*)in + (long long)b0 * d.K1 * d.K2, (long long)nb * d.K1, p->wk2[direction], q.s1,
                       p->rgt[direction], (double)nb * d.K1 * d.K2 * d.C, [&](auto& g) {
                           g.rows_per_field = d.K1;
                           g.ldo = d.K1;
                           g.out_z = (long long)d.C * d.K1;
                           g.out = (Cx*)q.t;
                           g.alpha = make_c<T>(T(1), T(0));
                           g.epi = HX_EPI_NONE;
                       }));
        HX_TRY(product(q.t, (long long)nb * d.C, p->wk1[direction], q.s2, p->lft[direction],
                       (double)nb * d.R * d.K1 * d.C, [&](auto& g) {
                           g.rows_per_field = d.C;
                           g.ldo = d.C;
                           g.out_z = oplane;
                           g.out = (Cx*)out + b0 * oplane;
                           g.alpha = make_c<T>((T)are, (T)aim);
                           g.epi = epilogue;
                           g.mask = (const Cx*)mask;
                           g.src = src ? (const Cx*)src + b0 * oplane : nullptr;
                       }));
    }
    return HX_OK;
}

}  // namespace

bool plane_mft_fits(int nx, int ny, int nu, int nv, int dtype, bool weighted) {
    if (std::max(std::max(nx, ny), std::max(nu, nv)) > 8192) return false;
    if (std::min(std::min(nx, ny), std::min(nu, nv)) < 16) return false;
    // The operands of the two directions, and of the adjoint where weights make it a third: at most 8 GB, 3% of the memory
    // (complex64 transforms between uniform grids of 8192^2 points take 6.4).
    const double bytes = 8.0 * (dtype == HX_C64 ? Shape<C64Digits>::NP : Shape<C128Digits>::NP) * (weighted ? 3.0 : 2.0) *
                         ((double)nx * nu + (double)ny * nv);
    return bytes <= 8e9;
}

int plane_mft_create(int dtype, int nx, int ny, int nu, int nv, const double* x, const double* y, const double* u,
                     const double* v, const double* wx, const double* wy, const double* wu, const double* wv,
                     cudaStream_t st, PlaneMft** out) {
    *out = nullptr;
    PlaneMft* p = new PlaneMft();
    p->dtype = dtype;
    p->nx = nx, p->ny = ny, p->nu = nu, p->nv = nv;
    const int rc = dtype == HX_C64 ? create_t<float>(p, x, y, u, v, wx, wy, wu, wv, st)
                                   : create_t<double>(p, x, y, u, v, wx, wy, wu, wv, st);
    if (rc != HX_OK) {
        plane_mft_destroy(p);
        return rc == HX_ERR_ALLOC ? (int)HX_OK : rc;  // no room for the cut operands: the plan runs on the CUDA cores
    }
    *out = p;
    return HX_OK;
}

void plane_mft_destroy(PlaneMft* p) {
    if (!p) return;
    cudaFree(p->mem);
    delete p;
}

size_t plane_mft_workspace_bytes(const PlaneMft* p, int direction, int batch) {
    if (!p || batch <= 0) return 0;
    const Dims d = dims_of(p, direction);
    if (p->dtype == HX_C64)
        return takes<float>(d, batch) ? carve_pass<float>(nullptr, d, fields_per_pass<float>(d, batch), nullptr) : 0;
    return takes<double>(d, batch) ? carve_pass<double>(nullptr, d, fields_per_pass<double>(d, batch), nullptr) : 0;
}

int plane_mft_execute(const PlaneMft* p, int direction, int batch, const void* in, void* out, double are, double aim,
                      int epilogue, const void* mask, const void* src, bool throughput, void* ws, cudaStream_t st) {
    if (p->dtype == HX_C64)
        return execute_t<float>(p, direction, batch, in, out, are, aim, epilogue, mask, src, throughput, ws, st);
    return execute_t<double>(p, direction, batch, in, out, are, aim, epilogue, mask, src, throughput, ws, st);
}

int plane_mft_status(const PlaneMft* p, int reset) {
    if (!p || !p->status) return HX_OK;
    int h = 0;
    HX_TRY(cuda_status(cudaMemcpy(&h, p->status, sizeof(int), cudaMemcpyDeviceToHost), "read plane MFT status"));
    if (reset && h != 0) cudaMemset(p->status, 0, sizeof(int));
    if (h != 0) set_error("a bounded wait in the tensor-core MFT gave up");
    return h;
}

}  // namespace hx
