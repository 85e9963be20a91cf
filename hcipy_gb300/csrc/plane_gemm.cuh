// Tensor-core GEMM of the plain-precision matrix Fourier transform (complex64 and complex128 plans) on tcgen05.
//
// out^T = alpha B . A^T for a field A (M x K, complex, one transform row per A row) and a plan constant B (N x K,
// one row per output column): D[m, n] = sum_k A[m, k] B[n, k] is written as out[n][m], so that the 32 lanes of a
// warp (consecutive m) store consecutive addresses straight from the accumulators, and so that the second GEMM of a
// transform reads the first one's result by contiguous rows.
//
// Operands.  Every row of A and of B is scaled by a power of two and cut into fp16 planes:
//   complex64 : two planes, x = s (h + l), h and l the fp16 roundings of x / s and of x / s - h, which keeps 22 bits
//               of every element; the products h l, l h and h h go to one FP32 accumulator, the small ones first.
//   complex128: seven planes of balanced base-256 digits, x = s sum_i d_i 2^(-7 - 8 i) with d_i in [-128, 128],
//               55 bits below the row maximum; the 28 products d_i d_j with i + j <= 6 go to seven accumulators, one
//               per level i + j.
// A holds [Ar | Ai] per row (K' = 2K), B holds the complex embedding in blocks of 8 complex columns: the 8 real
// columns [Br | -Bi], then the 8 imaginary ones [Bi | Br].
//
// Sums.  The tensor cores truncate an FP32 sum that no longer fits 24 bits (a sum of 4096 positive
// products comes out 2.5e-5 low, of 64 products 1.5e-7 low: measured against float64), so no accumulator runs long:
//   complex64 : 32 terms of K' (6.5e-8 low), then the accumulator is added to FP32 registers in round-to-nearest, in
//               blocks of 16 partial sums;
//   complex128: 128 terms: every level is then an integer below 7 * 128 * 2^14 < 2^24, hence exact, and is added to
//               64-bit integers (levels 0-3 in one, 4-6 in another), exact over any K the plans take.
// The error of a complex128 transform is that of its operands (2^-56 of a row maximum) and of the dropped products
// (below 2^-56 of the two scales), both under the rounding of a float64 product.
//
// Pipeline.  One CTA per 128 rows x BN real columns (BN = 128 for complex64, 64 for complex128, whose seven levels
// take 448 of the 512 TMEM columns): warp 0 issues TMA boxes of all planes of a K step, warp 1 the MMAs, warps 2-9
// drain.  Each accumulator has its own pair of barriers, so level l of the next partial sum starts as soon as level
// l of this one is drained: complex64 alternates two sets of accumulators, complex128 drains its levels in the order
// in which the next step's MMAs reach them.
// With few tiles the CTAs of a thread-block cluster split K and add their partial sums, in rank order, through
// distributed shared memory, each CTA finishing a slice of the columns.
// All waits are bounded (2 s): a wait that runs out records HX_ERR_TIMEOUT in the plan's status word.
#pragma once

#include "hx_common.cuh"
#include "tc_ptx.cuh"

#include <cuda_fp16.h>

namespace hx {
namespace pg {

constexpr int BM = 128;            // rows of A per tile (TMEM lanes)
constexpr int NUM_THREADS = 320;   // TMA warp, MMA warp, 8 epilogue warps
constexpr int EPI_THREADS = 256;
constexpr uint64_t WAIT_LIMIT = 2000000000ull;
constexpr int NAN_EXP = -(1 << 28);  // row exponent of a row that holds an infinity or a NaN (complex128)

// Planes (NP), accumulators (LV), real columns per tile (BN), K' per stage (BK), accumulator sets (SETS), stages per
// partial sum (CT) and partial sums per stage (PPS), pipeline stages (ST).
template <typename T> struct Shape;
template <> struct Shape<float> {
    static constexpr int NP = 2, LV = 1, BN = 128, BK = 64, SETS = 4, CT = 1, PPS = 2, ST = 3;
    using Acc = float;
    using Scale = float;
};
template <> struct Shape<double> {
    static constexpr int NP = 7, LV = 7, BN = 64, BK = 32, SETS = 1, CT = 4, PPS = 1, ST = 2;
    struct __align__(16) Acc {
        long long hi, lo;  // value = hi 2^-38 + lo 2^-62 (times the scales)
    };
    using Scale = int;  // exponent of the power-of-two scale
};

template <typename T> struct Layout {
    using S = Shape<T>;
    static constexpr int ROW_BYTES = S::BK * 2;  // 128 (128-byte swizzle) or 64 (64-byte swizzle)
    static constexpr int A_PLANE = BM * ROW_BYTES;
    static constexpr int B_PLANE = S::BN * ROW_BYTES;
    static constexpr int STAGE = S::NP * (A_PLANE + B_PLANE);
    static constexpr int PIPE = S::ST * STAGE;
    static constexpr int SMEM = PIPE + 1024 + 1024;  // alignment slack; barriers, flags, column scales
    static constexpr int TN = S::BN / 2;            // complex columns per tile
    static constexpr int NACC = S::SETS * S::LV;
    static constexpr int TMEM_COLS = 512;
    static_assert(NACC * S::BN <= TMEM_COLS, "the accumulators must fit TMEM");
    static_assert(BM * S::BN * (int)sizeof(typename S::Acc) <= PIPE, "partial sums must fit the pipeline buffers");
    static_assert(SMEM <= 227 * 1024, "shared memory per CTA");
};

template <typename T>
struct PlaneArgs {
    using Cx = typename cplx<T>::type;
    CUtensorMap tmap_a;
    CUtensorMap tmap_b;
    int ktiles;             // K' / BK
    int ksplit;             // CTAs along K per tile (the size of the cluster)
    int n_tiles;
    int M, N;               // rows of A, complex columns
    const typename Shape<T>::Scale* row_scale;
    const typename Shape<T>::Scale* col_scale;
    int rows_per_field;     // row m is row m % rows_per_field of field m / rows_per_field
    long long ldo, out_z;   // element (m, n): out[field * out_z + n * ldo + row of the field]
    Cx* out;
    Cx alpha;
    int epi;                // HX_EPI_*
    const Cx* mask;         // one field, indexed n * ldo + row
    const Cx* src;          // indexed like out
    int* status;
};

// Words of the shared-memory descriptor of a K-major operand whose rows are ROW_BYTES wide and swizzled over that
// width: the low word holds the start address in units of 16 bytes, the high word the distance of the 8-row groups,
// the descriptor version and the swizzle mode.
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr) { return ((saddr & 0x3FFFF) >> 4) | (1u << 16); }
template <int ROW_BYTES> constexpr uint32_t desc_hi() {
    static_assert(ROW_BYTES == 128 || ROW_BYTES == 64, "128- or 64-byte swizzle");
    return ((8 * ROW_BYTES) >> 4) | (1u << 14) | ((ROW_BYTES == 128 ? 2u : 4u) << 29);
}

__device__ __forceinline__ void tmem_ld_32(uint32_t taddr, float* v) {
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

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// (hi 2^24 + lo) 2^e rounded to float64 with integer operations (the float64 pipe issues two operations per clock
// and SM): normalise to 64 bits, round to 53, place the exponent.
__device__ __forceinline__ double fixed_to_double(long long hi, long long lo, int e) {
    long long h = hi + (lo >> 24);
    unsigned int l = (unsigned int)lo & 0xffffffu;
    const bool neg = h < 0;
    if (neg) {
        h = l ? ~h : -h;
        l = (0x1000000u - l) & 0xffffffu;
    }
    unsigned long long x = (unsigned long long)h;
    int sh;
    if (x == 0) {
        if (l == 0) return 0.0;
        sh = __clz((int)l) + 32;
        x = (unsigned long long)l << sh;
    } else {
        const int lz = __clzll((long long)x);  // h is below 2^54
        x = (x << lz) | (lz >= 24 ? (unsigned long long)l << (lz - 24) : (unsigned long long)(l >> (24 - lz)));
        sh = lz - 24;
    }
    // the value is x 2^(e - sh) with the leading one of x at bit 63
    const int be = e - sh + 63 + 1023;
    const unsigned long long mant = (x >> 11) + ((x >> 10) & 1);  // 2^52 .. 2^53
    if (be <= 0 || be >= 2046) {
        // subnormal results and overflow: scale in two exact or correctly flushed steps
        const double v = scalbn((double)mant, e - sh + 11);
        return neg ? -v : v;
    }
    const unsigned long long bits = ((unsigned long long)(be - 1) << 52) + mant;  // a carry moves the exponent
    return __longlong_as_double((long long)(bits | (neg ? 0x8000000000000000ull : 0)));
}

__device__ __forceinline__ float acc_value(const float& a, float rs, float cs) { return a * cs * rs; }
__device__ __forceinline__ double acc_value(const Shape<double>::Acc& a, int re, int ce) {
    if (re == NAN_EXP || ce == NAN_EXP) return __longlong_as_double(0x7ff8000000000000ll);
    return fixed_to_double(a.hi, a.lo, re + ce - 62);
}

__device__ __forceinline__ void acc_add(float& a, const float& b) { a += b; }
__device__ __forceinline__ void acc_add(Shape<double>::Acc& a, const Shape<double>::Acc& b) {
    a.hi += b.hi;
    a.lo += b.lo;
}

__device__ __forceinline__ void st_cluster(uint32_t addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(uint32_t addr, const Shape<double>::Acc& v) {
    asm volatile("st.shared::cluster.v2.b64 [%0], {%1, %2};" ::"r"(addr), "l"(v.hi), "l"(v.lo) : "memory");
}

// Running sums of one thread's columns.
template <typename T> struct Sums;
template <> struct Sums<float> {
    static constexpr int COLS = Shape<float>::BN / 2;
    float tot[COLS], blk[COLS];
    int n = 0;
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int j = 0; j < COLS; ++j) tot[j] = blk[j] = 0.0f;
    }
    template <int L> __device__ __forceinline__ void add(int j0, const float* v) {
#pragma unroll
        for (int j = 0; j < 32; ++j) blk[j0 + j] += v[j];
    }
    __device__ __forceinline__ void end_partial(bool last) {
        if ((++n & 15) != 0 && !last) return;
#pragma unroll
        for (int j = 0; j < COLS; ++j) {
            tot[j] += blk[j];
            blk[j] = 0.0f;
        }
    }
    __device__ __forceinline__ float get(int j) const { return tot[j]; }
};
template <> struct Sums<double> {
    static constexpr int COLS = Shape<double>::BN / 2;
    Shape<double>::Acc a[COLS];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int j = 0; j < COLS; ++j) a[j] = {0, 0};
    }
    // integer level sums: levels 0-3 weigh 2^24, 2^16, 2^8, 1 in hi, levels 4-6 weigh 2^16, 2^8, 1 in lo
    template <int L> __device__ __forceinline__ void add(int j0, const float* v) {
        constexpr int W = L < 4 ? 1 << (8 * (3 - L)) : 1 << (8 * (6 - L));
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            const long long p = (long long)__float2int_rn(v[j]) * W;
            if (L < 4) a[j0 + j].hi += p;
            else a[j0 + j].lo += p;
        }
    }
    __device__ __forceinline__ void end_partial(bool) {}
    __device__ __forceinline__ const Shape<double>::Acc& get(int j) const { return a[j]; }
};

template <typename T>
__global__ void __launch_bounds__(NUM_THREADS, 1) plane_gemm_kernel(const __grid_constant__ PlaneArgs<T> g) {
    using S = Shape<T>;
    using LY = Layout<T>;
    using Cx = typename cplx<T>::type;
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
            ptx::mbar_init(bar_drained(a), EPI_THREADS / 32);
        }
        ptx::mbar_init(bar_done, 1);
        *abort_flag = 0;
        ptx::fence_mbar_init();
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
            for (int i = 0; i < nkt; ++i) {
                if (*abort_flag) break;
                const int s = i % S::ST, u = i / S::ST;
                if (u > 0 && !ptx::mbar_wait_bounded(bar_empty(s), (u - 1) & 1, WAIT_LIMIT)) {
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
                if (last_use[s] >= 0 && !ptx::mbar_wait_bounded(bar_full(s), last_use[s] & 1, WAIT_LIMIT)) give_up();
        }
    } else if (warp == 1) {
        // the whole warp runs this branch (see ptx::elect_one)
        constexpr uint32_t idesc = ptx::umma_idesc_f16(BM, S::BN);
        const bool leader = ptx::elect_one();
        bool ok = true;
        for (int i = 0; i < nkt && ok; ++i) {
            const int s = i % S::ST, u = i / S::ST;
            const int part = i / S::CT * S::PPS, use = part / S::SETS;  // a stage's partial sums are of one use
            const int set = part % S::SETS;
            const bool first = i % S::CT == 0, last = i % S::CT == S::CT - 1 || i == nkt - 1;
            ok = __all_sync(0xffffffffu, ptx::mbar_wait_bounded(bar_full(s), u & 1, WAIT_LIMIT));
            if (!ok) break;
            ptx::tc_fence_after();
            const uint32_t a0 = desc_lo(smem_a + s * LY::STAGE);
            const uint32_t b0 = a0 + (S::NP * LY::A_PLANE >> 4);
            const uint32_t d0 = tmem + set * (S::LV * S::BN);
            constexpr uint32_t hi = desc_hi<LY::ROW_BYTES>();
            auto drained = [&](int l) {  // the accumulator's previous partial sum must have been read
                if (ok)
                    ok = __all_sync(0xffffffffu, ptx::mbar_wait_bounded(bar_drained(set * S::LV + l), (use - 1) & 1,
                                                                        WAIT_LIMIT));
                ptx::tc_fence_after();
            };
            auto mma = [&](int pa, int pb, int l, int kk, bool start) {
                if (leader)
                    ptx::umma_f16_lo(d0 + l * S::BN, a0 + ((pa * LY::A_PLANE + kk * 32) >> 4),
                                     b0 + ((pb * LY::B_PLANE + kk * 32) >> 4), hi, idesc, start);
            };
            if constexpr (S::LV == 1) {
                // one accumulator: the small products h l and l h first, while the sum is small and is truncated little
                static_assert(S::CT == 1 && S::SETS % S::PPS == 0, "whole partial sums per stage");
                constexpr int KH = S::BK / 16 / S::PPS;
#pragma unroll
                for (int h = 0; h < S::PPS; ++h) {
                    if (use > 0) drained(h);
#pragma unroll
                    for (int kk = h * KH; kk < (h + 1) * KH; ++kk) {
                        mma(0, 1, h, kk, kk == h * KH);
                        mma(1, 0, h, kk, false);
                    }
#pragma unroll
                    for (int kk = h * KH; kk < (h + 1) * KH; ++kk) mma(0, 0, h, kk, false);
                    if (leader) ptx::umma_commit(bar_ready(set + h));
                }
            } else {
#pragma unroll
                for (int kk = 0; kk < S::BK / 16; ++kk) {
#pragma unroll
                    for (int l = 0; l < S::LV; ++l) {
                        if (kk == 0 && first && use > 0) drained(l);
#pragma unroll
                        for (int p = 0; p <= l; ++p) mma(p, l - p, l, kk, first && kk == 0 && p == 0);
                        if (kk == S::BK / 16 - 1 && last && leader) ptx::umma_commit(bar_ready(set * S::LV + l));
                    }
                }
            }
            if (leader) ptx::umma_commit(bar_empty(s));
        }
        // TMEM and the pipeline buffers are released only after every MMA issued above
        if (leader) ptx::umma_commit(bar_done);
        ok = __all_sync(0xffffffffu, ptx::mbar_wait_bounded(bar_done, 0, WAIT_LIMIT)) && ok;
        if (!ok && leader) give_up();
    }
    // ---- warps 2..9: two per TMEM lane quarter, each one half of the columns ------------------------------------
    const bool epi = warp >= 2;
    const int et = threadIdx.x - 64;
    const int row = (warp & 3) * 32 + lane;
    const int half = (warp - 2) >> 2;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    constexpr int COLS = S::BN / 2;
    const int Sx = KS, TNS = LY::TN / Sx;
    Acc* part_s = reinterpret_cast<Acc*>(smem);  // [split][complex column of the slice][re, im][row]
    if (epi) {
        Sums<T> sums;
        sums.clear();
        bool live = true;
        const int nparts = (nkt + S::CT - 1) / S::CT * S::PPS;
#pragma unroll 1
        for (int p = 0; p < nparts; ++p) {
            const int set = p % S::SETS, ph = (p / S::SETS) & 1;
            auto level = [&](auto lc) {
                constexpr int l = decltype(lc)::value;
                const int a = set * S::LV + l;
                if (live && !ptx::mbar_wait_bounded(bar_ready(a), ph, WAIT_LIMIT)) give_up();
                // warp-uniform: the TMEM loads are .sync.aligned
                live = __shfl_sync(0xffffffffu, (int)(live && *abort_flag == 0), 0) != 0;
                if (!live) return;
                ptx::tc_fence_after();
#pragma unroll
                for (int j0 = 0; j0 < COLS; j0 += 32) {
                    float v[32];
                    tmem_ld_32(tmem + lane_base + a * S::BN + half * COLS + j0, v);
                    sums.template add<l>(j0, v);
                }
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_drained(a));
            };
            level(std::integral_constant<int, 0>());
            if constexpr (S::LV > 1) {
                level(std::integral_constant<int, 1>());
                level(std::integral_constant<int, 2>());
                level(std::integral_constant<int, 3>());
                level(std::integral_constant<int, 4>());
                level(std::integral_constant<int, 5>());
                level(std::integral_constant<int, 6>());
            }
            if (!live) break;
            sums.end_partial(p == nparts - 1);
        }
        if (Sx > 1) {
            __syncwarp();
            ptx::cluster_sync();  // every CTA's copies and MMAs are complete: the pipeline buffers are free
        } else {
            ptx::named_barrier(1, EPI_THREADS);
        }
        if (live) {
#pragma unroll
            for (int j = 0; j < COLS; ++j) {
                const int c = half * COLS + j;                    // real column of the tile
                const int cc = (c >> 4) * 8 + (c & 7), ri = (c >> 3) & 1;
                const int owner = cc / TNS, ccl = cc - owner * TNS;
                Acc* dst = part_s + ((ks * TNS + ccl) * 2 + ri) * BM + row;
                if (owner == ks) *dst = sums.get(j);
                else st_cluster(ptx::map_shared_rank(ptx::smem_addr(dst), (uint32_t)owner), sums.get(j));
            }
        }
    } else if (Sx > 1) {
        __syncwarp();
        ptx::cluster_sync();
    }
    if (Sx > 1) {
        __syncwarp();
        ptx::cluster_sync();  // every partial sum is in place
    }
    if (epi) {
        if (Sx == 1) ptx::named_barrier(1, EPI_THREADS);
        const int r = et & (BM - 1), m = m0 + r;
        if (m < g.M && *abort_flag == 0) {
            const int z = m / g.rows_per_field, y = m - z * g.rows_per_field;
            const int n0 = n_tile * LY::TN + ks * TNS;
            const Cx al = g.alpha;
            const bool imag_alpha = al.x == T(0), real_alpha = al.y == T(0);
            const Cx* mask = g.epi != HX_EPI_NONE ? g.mask : nullptr;
            const int step = EPI_THREADS / BM;
#pragma unroll(sizeof(T) == 4 ? 8 : 4)
            for (int cc = et / BM; cc < TNS; cc += step) {
                const int n = n0 + cc;
                if (n >= g.N) break;
                const long long o = (long long)z * g.out_z + (long long)n * g.ldo + y;
                const long long mo = (long long)n * g.ldo + y;
                Acc re = part_s[(cc * 2) * BM + r], im = part_s[(cc * 2 + 1) * BM + r];
                for (int sp = 1; sp < Sx; ++sp) {
                    acc_add(re, part_s[((sp * TNS + cc) * 2) * BM + r]);
                    acc_add(im, part_s[((sp * TNS + cc) * 2 + 1) * BM + r]);
                }
                const auto cs = s_cs[ks * TNS + cc];
                Cx v = make_c<T>(acc_value(re, rs, cs), acc_value(im, rs, cs));
                if (real_alpha) v = al.x == T(1) ? v : make_c<T>(al.x * v.x, al.x * v.y);
                else if (imag_alpha) v = make_c<T>(-al.y * v.y, al.y * v.x);
                else v = cmul(al, v);
                if (g.epi == HX_EPI_BABINET) {
                    const Cx e = g.src[o];
                    v.x = e.x - v.x;
                    v.y = e.y - v.y;
                }
                if (mask) v = cmul(v, mask[mo]);
                g.out[o] = v;
            }
        }
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
