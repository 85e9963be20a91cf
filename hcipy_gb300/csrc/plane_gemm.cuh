// Tensor-core GEMM of the plain-precision matrix Fourier transform (complex64 and complex128 plans) on tcgen05.
//
// out^T = alpha B . A^T for a field A (M x K, complex, one transform row per A row) and a plan constant B (N x K,
// one row per output column): D[m, n] = sum_k A[m, k] B[n, k] is written as out[n][m], so that the 32 lanes of a
// warp (consecutive m) store consecutive addresses straight from the accumulators, and so that the second GEMM of a
// transform reads the first one's result by contiguous rows.
//
// Operands.  Every row of A and of B is scaled by a power of two and cut into fp16 planes, in one of three forms (plane_mft.cu
// says which a complex64 operand takes):
//   C64Digits : x = 2^E sum_i d_i 2^(-8 - 9 i) with |x| <= 2^E, two whole digits of base 512, d_i in [-256, 256], and the rest
//               as an fp16 value: exact for |x| >= 2^(E - 6), to 2^-30 of 2^E below; the six products d_i d_j with
//               i + j <= 2 go to three accumulators, one per level i + j;
//   C64Floats : x = s (h + l), h and l the fp16 roundings of x / s and of x / s - h, which keeps 22 bits of every element;
//               the products h l, l h and h h go to one FP32 accumulator, the small ones first;
//   C128Digits: x = 2^E sum_i d_i 2^(-7 - 8 i), seven digits of base 256, d_i in [-128, 128], to 2^-56 of 2^E; the 28
//               products with i + j <= 6 go to seven accumulators.
// A holds [Ar | Ai] per row (K' = 2K), B holds the complex embedding in blocks of 8 complex columns: the 8 real
// columns [Br | -Bi], then the 8 imaginary ones [Bi | Br].
//
// Sums.  The tensor cores truncate an FP32 sum that no longer fits 24 bits (a sum of 4096 positive products comes out
// 2.5e-5 low, of 64 products 1.5e-7 low: measured against float64), so no accumulator runs long:
//   C64Digits : 256 terms of K': level 0 is at most 256 * 2^16 = 2^24, hence exact, and is added to 32-bit integers (2^30
//               over the longest K' of 16384).  Levels 1 and 2 weigh 2^-9 and 2^-18 of it: what they lose below 24 bits is
//               below 2^-32 of the terms' size.  They are added in FP32, and the sum is rounded once, at the end;
//   C64Floats : 32 terms of K', then the accumulator is added to FP32 registers in round-to-nearest, in blocks of 16
//               partial sums.  Such a sum is truncated after its first 16 terms and at the end, by half an ulp on
//               average: 2^-24 / (2 ln 2) = 4.3e-8 of a value with mantissas spread over their logarithm, and half of
//               that for the first truncation, 6.4e-8 together (6.5e-8 measured).  A factor so close to 1 on every
//               GEMM adds up along a chain of transforms, so it is taken back on average (Sums<C64Floats>::add);
//   C128Digits: 128 terms: every level is below 7 * 128 * 2^14 < 2^24, hence exact, and is added to 64-bit integers
//               (levels 0-3 in one, 4-6 in another), exact over any K the plans take.
// The error of a transform in digits is that of its operands (above), of the dropped products (of digits 1 and 2 in complex64:
// 2^-26 of the two scales at most, 2.5e-9 in the mean square) and one rounding of each sum: 3.5-7e-8 in complex64, for fields
// whose brightest pixel is 1e3 to 1e7 times the others 1.0-5.2e-7 (96 to 960 terms; CUDA cores 3.5e-7 to 1.7e-6).  In
// floating planes it is 1.1-2.0e-7, where the CUDA cores' sums of as many terms are 5e-7 to 1.6e-6 off.
//
// Pipeline.  One CTA per 128 rows x BN real columns (BN = 128 for complex64, 64 for complex128, whose seven levels
// take 448 of the 512 TMEM columns): warp 0 issues TMA boxes of all planes of a K step, warp 1 the MMAs, the others
// drain.  Each accumulator has its own pair of barriers, so level l of the next partial sum starts as soon as level l of
// this one is drained, in the order in which the next step's MMAs reach them; floating planes have four sets of their one
// accumulator, two partial sums of a stage in each half.
// With few tiles the CTAs of a thread-block cluster split K and add their partial sums in rank order, each CTA
// finishing a slice of the columns.  The sums travel through L2 under the cluster's barrier: through distributed shared
// memory they moved at 7 to 13 bytes per clock and SM.
// Measured against the GEMMs on the CUDA cores: a complex128 lens of 512^2 points to 256^2 1060 -> 73 us (float64 pipe), a
// complex64 Lyot pass over four fields of 1024^2 points 1700 -> 333 us in floating planes, 434 us in digits (FP32 pipe).
// complex64 is bound by shared memory, which moves 128 bytes a clock: per 16 K' the MMAs of digits read 40 KB in 384 clocks
// while the loads write 24 KB, those of floating planes 24 and 16 KB in 192 (1270 clocks per 64 K' measured).  complex128
// is bound by the epilogue (10 of 38 thousand clocks are MMAs where K is split eight ways).
// All waits are bounded (2 s): a wait that runs out records HX_ERR_TIMEOUT in the plan's status word, and the CTA, with the
// others of its cluster, writes NaN instead of sums that are not complete, so that no result looks like one.
#pragma once

#include "hx_common.cuh"
#include "tc_ptx.cuh"

#include <cuda_fp16.h>

namespace hx {
namespace pg {

constexpr int BM = 128;            // rows of A per tile (TMEM lanes)
constexpr uint64_t WAIT_LIMIT = 2000000000ull;  // ns
constexpr int NAN_EXP = -(1 << 28);  // exponent of a row that holds an infinity or a NaN

// The three forms of an operand.
struct C64Digits {};   // complex64, three digits
struct C64Floats {};   // complex64, two floating planes
struct C128Digits {};  // complex128, seven digits

// Element type (T), planes (NP), levels (LV), real columns per tile (BN), K' per stage (BK), accumulator sets (SETS), stages
// per partial sum (CT) and partial sums per stage (PPS), pipeline stages (ST), epilogue threads (EPI: floating planes drain
// often and little, digits seldom and much, and their conversions want warps).
template <typename F> struct Shape;
template <> struct Shape<C64Digits> {
    using T = float;
    static constexpr int NP = 3, LV = 3, BN = 128, BK = 32, SETS = 1, CT = 8, PPS = 1, ST = 4, EPI = 512;
    struct __align__(8) Acc {
        int hi;    // value = hi 2^-16 + lo 2^-34 (times the scales)
        float lo;
    };
    using Scale = int;  // exponent of the power-of-two scale
    static __device__ Scale poison() { return NAN_EXP; }
};
template <> struct Shape<C64Floats> {
    using T = float;
    static constexpr int NP = 2, LV = 1, BN = 128, BK = 64, SETS = 4, CT = 1, PPS = 2, ST = 3, EPI = 256;
    using Acc = float;
    using Scale = float;
    static __device__ Scale poison() { return __int_as_float(0x7fc00000); }
};
template <> struct Shape<C128Digits> {
    using T = double;
    static constexpr int NP = 7, LV = 7, BN = 64, BK = 32, SETS = 1, CT = 4, PPS = 1, ST = 2, EPI = 512;
    struct __align__(16) Acc {
        long long hi, lo;  // value = hi 2^-38 + lo 2^-62 (times the scales)
    };
    using Scale = int;
    static __device__ Scale poison() { return NAN_EXP; }
};

template <typename F> struct Layout {
    using S = Shape<F>;
    static constexpr int ROW_BYTES = S::BK * 2;  // 128 (128-byte swizzle) or 64 (64-byte swizzle)
    static constexpr int A_PLANE = BM * ROW_BYTES;
    static constexpr int B_PLANE = S::BN * ROW_BYTES;
    static constexpr int STAGE = S::NP * (A_PLANE + B_PLANE);
    static constexpr int PIPE = S::ST * STAGE;
    static constexpr int SMEM = PIPE + 1024 + 1024;  // alignment slack; barriers, flags, column scales
    static constexpr int TN = S::BN / 2;            // complex columns per tile
    static constexpr int THREADS = S::EPI + 64;     // TMA warp, MMA warp, epilogue warps
    static constexpr int COLS = S::BN / (S::EPI / BM);  // real columns per epilogue thread
    static constexpr int LD = COLS < 32 ? COLS : 32;    // columns per TMEM load
    static constexpr int NACC = S::SETS * S::LV;
    static constexpr int TMEM_COLS = 512;
    static_assert(NACC * S::BN <= TMEM_COLS, "the accumulators must fit TMEM");
    static_assert(BM * S::BN * (int)sizeof(typename S::Acc) <= PIPE, "partial sums must fit the pipeline buffers");
    static_assert(SMEM <= 227 * 1024, "shared memory per CTA");
};

template <typename F>
struct PlaneArgs {
    using Cx = typename cplx<typename Shape<F>::T>::type;
    CUtensorMap tmap_a;
    CUtensorMap tmap_b;
    int ktiles;             // K' / BK
    int ksplit;             // CTAs along K per tile (the size of the cluster)
    int n_tiles;
    int M, N;               // rows of A, complex columns
    const typename Shape<F>::Scale* row_scale;
    const typename Shape<F>::Scale* col_scale;
    int rows_per_field;     // row m is row m % rows_per_field of field m / rows_per_field
    long long ldo, out_z;   // element (m, n): out[field * out_z + n * ldo + row of the field]
    Cx* out;
    Cx alpha;
    int alpha_kind;         // 0: 1, 1: real, 2: imaginary, 3: complex (told apart on the host, not on the float64 pipe)
    int epi;                // HX_EPI_*
    const Cx* mask;         // one field, indexed n * ldo + row
    const Cx* src;          // indexed like out
    typename Shape<F>::Acc* parts;  // scratch of a K split: one tile's sums per CTA
    int* status;
    uint64_t wait_limit;    // ns (WAIT_LIMIT)
    int stall;              // test of the waits: the first CTA along K loads nothing, so that its waits run out
};

// Words of the shared-memory descriptor of a K-major operand whose rows are ROW_BYTES wide and swizzled over that
// width: the low word holds the start address in units of 16 bytes, the high word the distance of the 8-row groups,
// the descriptor version and the swizzle mode.
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr) { return ((saddr & 0x3FFFF) >> 4) | (1u << 16); }
template <int ROW_BYTES> constexpr uint32_t desc_hi() {
    static_assert(ROW_BYTES == 128 || ROW_BYTES == 64, "128- or 64-byte swizzle");
    return ((8 * ROW_BYTES) >> 4) | (1u << 14) | ((ROW_BYTES == 128 ? 2u : 4u) << 29);
}

template <int N> __device__ __forceinline__ void tmem_ld(uint32_t taddr, float* v);
template <> __device__ __forceinline__ void tmem_ld<16>(uint32_t taddr, float* v) { ptx::tmem_ld_16(taddr, v); }
template <> __device__ __forceinline__ void tmem_ld<32>(uint32_t taddr, float* v) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,"
        "%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// (hi 2^24 + lo) 2^e rounded to float64 (|hi| < 2^53, |lo| < 2^48), with integer operations (the float64 pipe issues
// about 1.6 operations per clock and SM) and without branches, so that the conversions of several columns overlap:
// the sum's magnitude is normalised to a leading one at bit 63, rounded to 53 bits and given its exponent.  An exponent
// out of float64's normal range sets `rare`; the caller then takes scaled_value.
__device__ __forceinline__ double fixed_to_double(long long hi, long long lo, int e, bool& rare) {
    const long long up = hi + (lo >> 24);            // units of 2^24, below 2^54
    const unsigned int low = (unsigned int)lo << 8;  // the 24 bits below, left-aligned in 32
    const unsigned int sign = (unsigned int)(up >> 63);
    const unsigned long long mag = (unsigned long long)(up ^ (up >> 63)) + (low == 0 ? (sign & 1) : 0);
    const unsigned int x2 = (unsigned int)(mag >> 32), x1 = (unsigned int)mag, x0 = low == 0 ? 0 : (low ^ sign) + (sign & 1);
    // the leading non-zero word of x2 x1 x0 (x2 x1 in units of 2^24) and the two below it
    const bool two = x2 != 0, one = x1 != 0;
    const unsigned int y2 = two ? x2 : one ? x1 : x0, y1 = two ? x1 : one ? x0 : 0, y0 = two ? x0 : 0;
    const int lz = __clz((int)y2);
    const unsigned long long m =
        ((unsigned long long)__funnelshift_l(y1, y2, lz) << 32 | __funnelshift_l(y0, y1, lz)) + 0x400;
    // the exponent of the leading one, one more where the rounding carried out of the top
    const int be = (two ? 63 : one ? 31 : -1) - lz + 24 + e + 1023 + (int)(m < 0x400);
    rare |= y2 != 0 && (be < 1 || be > 2046);
    const unsigned int fh = (unsigned int)(m >> 43) & 0xfffffu, fl = (unsigned int)(m >> 11);
    const unsigned int top = fh | ((unsigned int)be << 20) | (sign & 0x80000000u);
    return __hiloint2double(y2 == 0 ? 0 : (int)top, y2 == 0 ? 0 : (int)fl);
}
__device__ __noinline__ double scaled_value(long long hi, long long lo, int e) {
    return scalbn(fma((double)hi, 0x1p24, (double)lo), e);
}

// (hi 2^18 + lo) 2^e with one rounding to 24 bits (and, where the result is subnormal, one more).
__device__ __forceinline__ float fixed_to_float(int hi, float lo, int e) {
    const float f = (float)hi;
    const float v = fmaf(f, 0x1p18f, fmaf((float)(hi - (int)f), 0x1p18f, lo));
    const int c = min(max(e, -252), 254), h = c >> 1;  // past these v 2^e is 0 or infinite either way
    return v * __int_as_float((h + 127) << 23) * __int_as_float((c - h + 127) << 23);
}

__device__ __forceinline__ float acc_value(const Shape<C64Digits>::Acc& a, int re, int ce, bool& rare) {
    rare |= re == NAN_EXP || ce == NAN_EXP;
    return fixed_to_float(a.hi, a.lo, re + ce - 34);
}
__device__ __forceinline__ double acc_value(const Shape<C128Digits>::Acc& a, int re, int ce, bool& rare) {
    rare |= re == NAN_EXP || ce == NAN_EXP;
    return fixed_to_double(a.hi, a.lo, re + ce - 62, rare);
}
__device__ __forceinline__ float acc_rare(const Shape<C64Digits>::Acc& a, int re, int ce) {
    if (re == NAN_EXP || ce == NAN_EXP) return __int_as_float(0x7fc00000);
    return fixed_to_float(a.hi, a.lo, re + ce - 34);
}
__device__ __forceinline__ double acc_rare(const Shape<C128Digits>::Acc& a, int re, int ce) {
    if (re == NAN_EXP || ce == NAN_EXP) return __longlong_as_double(0x7ff8000000000000ll);
    return scaled_value(a.hi, a.lo, re + ce - 62);
}

__device__ __forceinline__ float acc_value(const float& a, float rs, float cs, bool&) { return a * cs * rs; }
__device__ __forceinline__ float acc_rare(const float& a, float rs, float cs) { return a * cs * rs; }

__device__ __forceinline__ void acc_add(float& a, const float& b) { a += b; }
template <typename A> __device__ __forceinline__ void acc_add(A& a, const A& b) {
    a.hi += b.hi;
    a.lo += b.lo;
}

// Partial sums of the other CTAs of a K split travel through L2.
__device__ __forceinline__ void put_part(float* p, float v) { __stcg(p, v); }
__device__ __forceinline__ float get_part(const float* p) { return __ldcg(p); }
__device__ __forceinline__ void put_part(Shape<C64Digits>::Acc* p, const Shape<C64Digits>::Acc& v) {
    __stcg(reinterpret_cast<int2*>(p), make_int2(v.hi, __float_as_int(v.lo)));
}
__device__ __forceinline__ void put_part(Shape<C128Digits>::Acc* p, const Shape<C128Digits>::Acc& v) {
    __stcg(reinterpret_cast<longlong2*>(p), make_longlong2(v.hi, v.lo));
}
__device__ __forceinline__ Shape<C64Digits>::Acc get_part(const Shape<C64Digits>::Acc* p) {
    const int2 v = __ldcg(reinterpret_cast<const int2*>(p));
    return {v.x, __int_as_float(v.y)};
}
__device__ __forceinline__ Shape<C128Digits>::Acc get_part(const Shape<C128Digits>::Acc* p) {
    const longlong2 v = __ldcg(reinterpret_cast<const longlong2*>(p));
    return {v.x, v.y};
}

// Running sums of one thread's columns.
template <typename F> struct Sums;
template <> struct Sums<C64Digits> {
    static constexpr int COLS = Layout<C64Digits>::COLS;
    Shape<C64Digits>::Acc a[COLS];
    __device__ __forceinline__ void start(int, int) {
#pragma unroll
        for (int j = 0; j < COLS; ++j) a[j] = {0, 0.0f};
    }
    // level 0 in units of its own, levels 1 and 2 (2^9 and 1) in units of level 2
    template <int L> __device__ __forceinline__ void add(int j0, const float* v) {
#pragma unroll
        for (int j = 0; j < Layout<C64Digits>::LD; ++j) {
            if (L == 0) a[j0 + j].hi += __float2int_rn(v[j]);
            else if (L == 1) a[j0 + j].lo = fmaf(v[j], 512.0f, a[j0 + j].lo);
            else a[j0 + j].lo += v[j];
        }
    }
    __device__ __forceinline__ void end_partial(bool) {}
    __device__ __forceinline__ const Shape<C64Digits>::Acc& get(int j) const { return a[j]; }
};
template <> struct Sums<C64Floats> {
    static constexpr int COLS = Layout<C64Floats>::COLS;
    float tot[COLS], blk[COLS];
    int n = 0, q, half;
    __device__ __forceinline__ void start(int half_, int first) {
        half = half_;
        q = first % half_;
#pragma unroll
        for (int j = 0; j < COLS; ++j) tot[j] = blk[j] = 0.0f;
    }
    // Every second partial sum times 1 + 2^-23, in the one rounding of the addition: 6.0e-8 of the 6.4e-8 that truncated sums
    // lose on average.  Counted from the start of either half of K', so that real and imaginary fields fare alike.  A sum
    // of one or few terms (a field of few pixels) may have lost nothing; its transform is then up to 2^-23 too large per GEMM,
    // 1.0-2.2e-7 in all where the CUDA cores are 0.4-0.6e-7 off.
    template <int L> __device__ __forceinline__ void add(int j0, const float* v) {
        const float w = (q & 1) ? 1.0f : 1.0f + 0x1p-23f;
#pragma unroll
        for (int j = 0; j < Layout<C64Floats>::LD; ++j) blk[j0 + j] = fmaf(v[j], w, blk[j0 + j]);
    }
    __device__ __forceinline__ void end_partial(bool last) {
        if (++q == half) q = 0;
        if ((++n & 15) != 0 && !last) return;
#pragma unroll
        for (int j = 0; j < COLS; ++j) {
            tot[j] += blk[j];
            blk[j] = 0.0f;
        }
    }
    __device__ __forceinline__ float get(int j) const { return tot[j]; }
};
template <> struct Sums<C128Digits> {
    static constexpr int COLS = Layout<C128Digits>::COLS;
    Shape<C128Digits>::Acc a[COLS];
    __device__ __forceinline__ void start(int, int) {
#pragma unroll
        for (int j = 0; j < COLS; ++j) a[j] = {0, 0};
    }
    // integer level sums: levels 0-3 weigh 2^24, 2^16, 2^8, 1 in hi, levels 4-6 weigh 2^16, 2^8, 1 in lo
    template <int L> __device__ __forceinline__ void add(int j0, const float* v) {
        constexpr int W = L < 4 ? 1 << (8 * (3 - L)) : 1 << (8 * (6 - L));
#pragma unroll
        for (int j = 0; j < Layout<C128Digits>::LD; ++j) {
            const long long p = (long long)__float2int_rn(v[j]) * W;
            if (L < 4) a[j0 + j].hi += p;
            else a[j0 + j].lo += p;
        }
    }
    __device__ __forceinline__ void end_partial(bool) {}
    __device__ __forceinline__ const Shape<C128Digits>::Acc& get(int j) const { return a[j]; }
};

// f with the compile-time numbers 0 .. N - 1.
template <int N, typename F> __device__ __forceinline__ void each_level(F&& f) {
    if constexpr (N > 0) {
        each_level<N - 1>(f);
        f(std::integral_constant<int, N - 1>());
    }
}

// The finished columns of a tile: all of them, or with a K split over KS CTAs the ks-th of KS slices of its complex
// columns, the CTA's own partial sums from shared memory and the others' from `others` (L2), added in rank order.
// Lanes along the rows, so that the reads and the stores are contiguous; U columns at a time, their loads ahead of
// their arithmetic.
template <typename F, int KS>
__device__ __forceinline__ void finish_columns(const PlaneArgs<F>& g, const typename Shape<F>::Acc* part_s,
                                               const typename Shape<F>::Acc* others,
                                               const typename Shape<F>::Scale* s_cs, typename Shape<F>::Scale rs,
                                               int m0, int n_tile, int ks, int et) {
    using T = typename Shape<F>::T;
    using Cx = typename cplx<T>::type;
    using Acc = typename Shape<F>::Acc;
    constexpr int TN = Layout<F>::TN, STEP = Shape<F>::EPI / BM, TNS = TN / KS;
    constexpr int UMAX = sizeof(Acc) == 4 || (sizeof(Acc) == 8 && KS < 4) ? 4 : 2, U = TNS / STEP < UMAX ? TNS / STEP : UMAX;
    static_assert(TNS % (STEP * U) == 0, "whole batches");
    constexpr int PART = TN * 2 * BM;  // one CTA's partial sums
    const int r = et & (BM - 1), m = m0 + r;
    const bool mok = m < g.M;
    const int z = mok ? m / g.rows_per_field : 0, y = mok ? m - z * g.rows_per_field : 0;
    const Cx al = g.alpha;
    const int kind = g.alpha_kind;
    const Cx* mask = g.epi != HX_EPI_NONE ? g.mask : nullptr;
#pragma unroll 1
    for (int c = ks * TNS + et / BM; c < (ks + 1) * TNS; c += U * STEP) {
        Acc re[U], im[U], xr[U][KS], xi[U][KS];
        Cx e[U], mk[U], v[U];
        bool rare = false;
        long long o[U];
        bool ok[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int at = (c + u * STEP) * 2 * BM + r;
            if constexpr (KS > 1) {
#pragma unroll
                for (int sp = 0; sp < KS; ++sp) {
                    if (sp == ks) continue;
                    xr[u][sp] = get_part(others + sp * PART + at);
                    xi[u][sp] = get_part(others + sp * PART + at + BM);
                }
            }
            const int n = n_tile * TN + c + u * STEP;
            const long long mo = (long long)n * g.ldo + y;
            ok[u] = mok && n < g.N;
            o[u] = (long long)z * g.out_z + mo;
            if (ok[u] && g.epi == HX_EPI_BABINET) e[u] = g.src[o[u]];
            if (ok[u] && mask) mk[u] = mask[mo];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int at = (c + u * STEP) * 2 * BM + r;
            re[u] = part_s[at];
            im[u] = part_s[at + BM];
            if constexpr (KS > 1) {
                const Acc own_r = re[u], own_i = im[u];
#pragma unroll
                for (int sp = 0; sp < KS; ++sp) {
                    const Acc a = sp == ks ? own_r : xr[u][sp], b = sp == ks ? own_i : xi[u][sp];
                    if (sp == 0) {
                        re[u] = a;
                        im[u] = b;
                    } else {
                        acc_add(re[u], a);
                        acc_add(im[u], b);
                    }
                }
            }
            const auto cs = s_cs[c + u * STEP];
            v[u] = make_c<T>(acc_value(re[u], rs, cs, rare), acc_value(im[u], rs, cs, rare));
        }
        if (rare) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const auto cs = s_cs[c + u * STEP];
                v[u] = make_c<T>(acc_rare(re[u], rs, cs), acc_rare(im[u], rs, cs));
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            Cx w = v[u];
            if (kind == 1) w = make_c<T>(al.x * w.x, al.x * w.y);
            else if (kind == 2) w = make_c<T>(-al.y * w.y, al.y * w.x);
            else if (kind == 3) w = cmul(al, w);
            if (g.epi == HX_EPI_BABINET) {
                w.x = e[u].x - w.x;
                w.y = e[u].y - w.y;
            }
            if (mask) w = cmul(w, mk[u]);
            if (ok[u]) g.out[o[u]] = w;
        }
    }
}

template <typename F>
__global__ void __launch_bounds__(Layout<F>::THREADS, 1) plane_gemm_kernel(const __grid_constant__ PlaneArgs<F> g) {
    using S = Shape<F>;
    using LY = Layout<F>;
    using Acc = typename S::Acc;
    extern __shared__ __align__(1024) uint8_t pg_smem[];
    const uint32_t raw = ptx::smem_addr(pg_smem);
    uint8_t* smem = pg_smem + ((1024 - (raw & 1023)) & 1023);
    uint8_t* extra = smem + LY::PIPE;
    // full[ST], empty[ST], ready[NACC], drained[NACC], done
    uint64_t* bars = reinterpret_cast<uint64_t*>(extra);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(extra + 256);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(extra + 260);
    typename S::Scale* s_cs = reinterpret_cast<typename S::Scale*>(extra + 512);  // scales of the tile's columns
    static_assert(LY::TN * sizeof(typename S::Scale) <= 512, "column scales");
    auto bar_full = [&](int s) { return ptx::smem_addr(&bars[s]); };
    auto bar_empty = [&](int s) { return ptx::smem_addr(&bars[S::ST + s]); };
    auto bar_ready = [&](int a) { return ptx::smem_addr(&bars[2 * S::ST + a]); };
    auto bar_drained = [&](int a) { return ptx::smem_addr(&bars[2 * S::ST + LY::NACC + a]); };
    const uint32_t bar_done = ptx::smem_addr(&bars[2 * S::ST + 2 * LY::NACC]);
    static_assert((2 * S::ST + 2 * LY::NACC + 1) * 8 <= 256, "barriers");

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // warp-uniform
    const int KS = g.ksplit;
    const int n_tile = blockIdx.x / KS, ks = blockIdx.x % KS;
    const int m0 = blockIdx.y * BM;
    // K split on whole partial sums
    const int parts = (g.ktiles + S::CT - 1) / S::CT;
    const int kt0 = (int)((long long)parts * ks / KS) * S::CT;
    const int kt1 = min(g.ktiles, (int)((long long)parts * (ks + 1) / KS) * S::CT);
    const int nkt = kt1 - kt0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S::ST; ++s) {
            ptx::mbar_init(bar_full(s), 1);
            ptx::mbar_init(bar_empty(s), 1);
        }
        for (int a = 0; a < LY::NACC; ++a) {
            ptx::mbar_init(bar_ready(a), 1);
            ptx::mbar_init(bar_drained(a), S::EPI / 32);
        }
        ptx::mbar_init(bar_done, 1);
        *abort_flag = 0;
        ptx::fence_mbar_init();
        ptx::fence_cluster();  // the flag, before the cluster barrier's first phase
        ptx::prefetch_tensormap(&g.tmap_a);
        ptx::prefetch_tensormap(&g.tmap_b);
    }
    // what the epilogue needs from global memory, loaded ahead of the main loop
    typename S::Scale rs = 0;
    if (warp >= 2) {
        const int t = threadIdx.x - 64;
        const int m = m0 + (t & (BM - 1)), n = n_tile * LY::TN + t;
        if (m < g.M) rs = g.row_scale[m];
        if (t < LY::TN) s_cs[t] = n < g.N ? g.col_scale[n] : typename S::Scale(0);
    }
    if (warp == 1) {
        ptx::tmem_alloc(ptx::smem_addr(tmem_slot), LY::TMEM_COLS);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    if (KS > 1) ptx::cluster_arrive_relaxed();  // waited for before a CTA writes another's flag: that has started by then
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    const uint32_t smem_a = ptx::smem_addr(smem);
    auto give_up = [&] {
        *abort_flag = 1;
        if (g.status) atomicExch(g.status, HX_ERR_TIMEOUT);
    };

    if (warp == 0) {
        if (lane == 0) {
            int last_use[S::ST];
            for (int s = 0; s < S::ST; ++s) last_use[s] = -1;
            const int loads = g.stall && ks == 0 ? 0 : nkt;
            for (int i = 0; i < loads; ++i) {
                if (*abort_flag) break;
                const int s = i % S::ST, u = i / S::ST;
                if (u > 0 && !ptx::mbar_wait_bounded(bar_empty(s), (u - 1) & 1, g.wait_limit)) {
                    give_up();
                    break;
                }
                uint8_t* sa = smem + s * LY::STAGE;
                uint8_t* sb = sa + S::NP * LY::A_PLANE;
                ptx::mbar_arrive_expect_tx(bar_full(s), LY::STAGE);
                ptx::tma_load_3d(ptx::smem_addr(sa), &g.tmap_a, (kt0 + i) * S::BK, m0, 0, bar_full(s));
                ptx::tma_load_3d(ptx::smem_addr(sb), &g.tmap_b, (kt0 + i) * S::BK, n_tile * S::BN, 0, bar_full(s));
                last_use[s] = u;
            }
            // No copy may land in shared memory after this CTA leaves the pipeline.
            for (int s = 0; s < S::ST; ++s)
                if (last_use[s] >= 0 && !ptx::mbar_wait_bounded(bar_full(s), last_use[s] & 1, g.wait_limit)) give_up();
        }
    } else if (warp == 1) {
        // the whole warp runs this branch (see ptx::elect_one)
        const bool leader = ptx::elect_one();
        bool ok = true;
        for (int i = 0; i < nkt && ok; ++i) {
            const int s = i % S::ST, u = i / S::ST;
            const int part = i / S::CT * S::PPS, use = part / S::SETS;  // a stage's partial sums are of one use
            const int set = part % S::SETS;
            const bool first = i % S::CT == 0, last = i % S::CT == S::CT - 1 || i == nkt - 1;
            ok = __all_sync(0xffffffffu, ptx::mbar_wait_bounded(bar_full(s), u & 1, g.wait_limit));
            if (!ok) break;
            ptx::tc_fence_after();
            const uint32_t a0 = desc_lo(smem_a + s * LY::STAGE);
            const uint32_t b0 = a0 + (S::NP * LY::A_PLANE >> 4);
            const uint32_t d0 = tmem + set * (S::LV * S::BN);
            constexpr uint32_t hi = desc_hi<LY::ROW_BYTES>();
            auto drained = [&](int l) {  // the accumulator's previous partial sum must have been read
                if (ok)
                    ok = __all_sync(0xffffffffu, ptx::mbar_wait_bounded(bar_drained(set * S::LV + l), (use - 1) & 1,
                                                                        g.wait_limit));
                ptx::tc_fence_after();
            };
            // planes pb .. pb + count - 1 of B, which follow one another as the levels do in TMEM
            auto mma = [&](auto count, int pa, int pb, int l, int kk, bool start) {
                constexpr uint32_t idesc = ptx::umma_idesc_f16(BM, S::BN * decltype(count)::value);
                if (leader)
                    ptx::umma_f16_lo(d0 + l * S::BN, a0 + ((pa * LY::A_PLANE + kk * 32) >> 4),
                                     b0 + ((pb * LY::B_PLANE + kk * 32) >> 4), hi, idesc, start);
            };
            using one = std::integral_constant<int, 1>;
            if constexpr (S::LV == 1) {
                // one accumulator: the small products h l and l h first, while the sum is small and is truncated little
                static_assert(S::CT == 1 && S::SETS % S::PPS == 0, "whole partial sums per stage");
                constexpr int KH = S::BK / 16 / S::PPS;
#pragma unroll
                for (int h = 0; h < S::PPS; ++h) {
                    if (use > 0) drained(h);
#pragma unroll
                    for (int kk = h * KH; kk < (h + 1) * KH; ++kk) {
                        mma(one{}, 0, 1, h, kk, kk == h * KH);
                        mma(one{}, 1, 0, h, kk, false);
                    }
#pragma unroll
                    for (int kk = h * KH; kk < (h + 1) * KH; ++kk) mma(one{}, 0, 0, h, kk, false);
                    if (leader) ptx::umma_commit(bar_ready(set + h));
                }
            } else {
                // The first step of a partial sum takes a level at a time, as the accumulators are read out.  The others
                // take a plane of A at a time, against as many planes of B in one MMA as 256 columns hold: an MMA of 64
                // columns reads 4 KB of A and 2 KB of B in its 32 clocks, more than shared memory gives beside the
                // loads.  complex128: 10 MMAs and 96 KB per 16 K' instead of 28 and 168 KB, complex64: 4 and 40 KB instead
                // of 6 and 48 KB.  Exact sums may be taken in any order.
                constexpr int G = 256 / S::BN;
                auto row = [&](auto plane, int kk) {
                    constexpr int P = decltype(plane)::value, CNT = S::LV - P;
                    mma(std::integral_constant<int, (CNT < G ? CNT : G)>{}, P, 0, P, kk, false);
                    if constexpr (CNT > G) mma(std::integral_constant<int, CNT - G>{}, P, G, P + G, kk, false);
                };
                static_assert(S::LV <= 2 * G, "two MMAs at most for each plane of A");
#pragma unroll
                for (int kk = 0; kk < S::BK / 16; ++kk) {
                    const bool end = kk == S::BK / 16 - 1 && last;
                    if (kk == 0 && first) {
#pragma unroll
                        for (int l = 0; l < S::LV; ++l) {
                            if (use > 0) drained(l);
#pragma unroll
                            for (int p = 0; p <= l; ++p) mma(one{}, p, l - p, l, kk, p == 0);
                            if (end && leader) ptx::umma_commit(bar_ready(set * S::LV + l));
                        }
                    } else {
                        auto plane = [&](auto p) {  // with it the level of its own index has all its products
                            row(p, kk);
                            if (end && leader) ptx::umma_commit(bar_ready(set * S::LV + decltype(p)::value));
                        };
                        each_level<S::LV>(plane);
                    }
                }
            }
            if (leader) ptx::umma_commit(bar_empty(s));
        }
        // TMEM and the pipeline buffers are released only after every MMA issued above
        if (leader) ptx::umma_commit(bar_done);
        ok = __all_sync(0xffffffffu, ptx::mbar_wait_bounded(bar_done, 0, g.wait_limit)) && ok;
        if (!ok && leader) give_up();
    }
    // ---- warps 2 and up: two or four per TMEM lane quarter, each a slice of the columns ---------------------------------
    const bool epi = warp >= 2;
    const int et = threadIdx.x - 64;
    const int row = (warp & 3) * 32 + lane;
    const int slice = (warp - 2) >> 2;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    constexpr int COLS = LY::COLS;
    Acc* part_s = reinterpret_cast<Acc*>(smem);  // [complex column][re, im][row]
    // of a K split: the partial sums of the tile's CTAs, [CTA][complex column][re, im][row]
    Acc* others = g.parts + ((long long)blockIdx.y * g.n_tiles + n_tile) * KS * (LY::TN * 2 * BM);
    if (epi) {
        Sums<F> sums;
        sums.start(g.ktiles * S::PPS / 2, kt0 * S::PPS);  // partial sums per half of K', and the first one's index
        bool live = true;
        const int nparts = (nkt + S::CT - 1) / S::CT * S::PPS;
#pragma unroll 1
        for (int p = 0; p < nparts; ++p) {
            const int set = p % S::SETS, ph = (p / S::SETS) & 1;
            auto level = [&](auto lc) {
                constexpr int l = decltype(lc)::value;
                const int a = set * S::LV + l;
                if (live && !ptx::mbar_wait_bounded(bar_ready(a), ph, g.wait_limit)) give_up();
                // warp-uniform: the TMEM loads are .sync.aligned
                live = __shfl_sync(0xffffffffu, (int)(live && *abort_flag == 0), 0) != 0;
                if (!live) return;
                ptx::tc_fence_after();
#pragma unroll
                for (int j0 = 0; j0 < COLS; j0 += LY::LD) {
                    float v[LY::LD];
                    tmem_ld<LY::LD>(tmem + lane_base + a * S::BN + slice * COLS + j0, v);
                    sums.template add<l>(j0, v);
                }
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(bar_drained(a));
            };
            each_level<S::LV>(level);
            if (!live) break;
            sums.end_partial(p == nparts - 1);
        }
        // every warp has seen the last accumulators, so this CTA's copies and MMAs are complete
        ptx::named_barrier(1, S::EPI);
        if (live) {
            constexpr int LOG_TN = LY::TN == 64 ? 6 : 5;
            static_assert(1 << LOG_TN == LY::TN, "complex columns per tile");
            Acc* mine = others + (long long)ks * LY::TN * 2 * BM;
#pragma unroll
            for (int j = 0; j < COLS; ++j) {
                const int c = slice * COLS + j;  // real column of the tile
                const int cc = (c >> 4) * 8 + (c & 7);
                const int at = (cc * 2 + ((c >> 3) & 1)) * BM + row;
                if ((cc * KS) >> LOG_TN == ks) part_s[at] = sums.get(j);
                else put_part(mine + at, sums.get(j));
            }
        }
    }
    if (KS > 1) {
        __syncwarp();
        ptx::cluster_wait();
        if (epi && et < KS && *abort_flag) {  // what this CTA lacks is missing from every slice of the columns
            ptx::fence_cluster();
            ptx::st_cluster_u32(ptx::map_shared_rank(ptx::smem_addr(const_cast<int*>(abort_flag)), et), 1);
        }
        __syncwarp();
        ptx::cluster_sync();  // every CTA's partial sums are written (release and acquire cover L2 too)
    }
    if (epi) {
        if (KS == 1) ptx::named_barrier(1, S::EPI);
        if (*abort_flag) rs = S::poison();  // sums that are not complete: every result of theirs is NaN
        if (KS == 1) finish_columns<F, 1>(g, part_s, others, s_cs, rs, m0, n_tile, 0, et);
        else if (KS == 2) finish_columns<F, 2>(g, part_s, others, s_cs, rs, m0, n_tile, ks, et);
        else if (KS == 4) finish_columns<F, 4>(g, part_s, others, s_cs, rs, m0, n_tile, ks, et);
        else finish_columns<F, 8>(g, part_s, others, s_cs, rs, m0, n_tile, ks, et);
    }
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem, LY::TMEM_COLS);
    }
}

}  // namespace pg
}  // namespace hx
