// The split-operand tcgen05 GEMM for more output tiles than SMs: one persistent CTA per SM, whose epilogue of one tile
// runs beside the main loop of the next.
//
// split_gemm_kernel gives every tile its own CTA, and since one CTA fills an SM's shared memory and TMEM, nothing runs
// while a tile is finished: of the 62 thousand clocks of a 128 x 64 complex tile over 512 points 35 were MMAs, the rest
// the set-up, reading TMEM into shared memory (4) and finishing rows from there (8-15, the stores among them).  Here
// the sixteen epilogue warps take the combined levels of a tile into registers (32 columns of one TMEM lane per thread),
// hand TMEM back at once, and scale, mask and store from the registers while the MMAs of the next tile run; loads run
// ahead across tiles.  The arithmetic of an element is that of split_gemm_kernel, in the same order: the same bits.
//
// The stores go out in pieces of 16 bytes, so the output rows must be aligned to that (stream_fits); others keep
// split_gemm_kernel, whose warps store element by element along a row.
//
// What it measured: GEMMs of 64 stacked fields, 512^2 points to 512^2, complex64-to-float-float 395 -> 298 us, and with
// complex128 results from 256 points 319 -> 199 us; a gradient step through a Lyot coronagraph over 64 fields of 512^2
// points 5955 -> 4947 us.  A tile of 16 K steps of 64 takes 37 to 41 thousand clocks, 33 of them MMAs: what is left is the
// 2 thousand in which the levels are read (TMEM holds one tile's) and loads that the stores delay.
// On the way there: the loads alone take 23 thousand clocks a tile, so neither they nor L2 bound the loop; the epilogue
// did, through instructions (see `scale` and store_rows), and through stores that touched 32 lines each.
#include "split_gemm.cuh"

namespace hx {
namespace sg {

namespace {

constexpr int SBN = 128;  // columns of B' per tile
// Stages of 32 K' (STREAM_BK, rows of 64 bytes): four of 48 KB ride out delayed loads better than two of 96 KB with
// rows of 128 bytes (complex128 results 194 against 205 us; float-float the same within 2%).
constexpr int ROW_BYTES = 2 * STREAM_BK;
constexpr int STAGE_A = NSLICE * BM * ROW_BYTES, STAGE = STAGE_A + NSLICE * SBN * ROW_BYTES;
constexpr int STAGES = 196608 / STAGE;
constexpr int SMEM = STAGES * STAGE + 2048;  // alignment slack; barriers and flags
constexpr int TMEM_COLS = 4 * SBN;

// Transposes 4 x 4 blocks of W words over the four lanes of a group: lane a's block s becomes lane s's block a.
template <int W> __device__ __forceinline__ void transpose4(uint32_t (&d)[4][W], int lane) {
#pragma unroll
    for (int bit = 1; bit < 4; bit <<= 1) {
        const bool high = lane & bit;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            if (b & bit) continue;
#pragma unroll
            for (int w = 0; w < W; ++w) {
                const uint32_t got = __shfl_xor_sync(0xffffffffu, high ? d[b][w] : d[b | bit][w], bit);
                if (high) d[b][w] = got;
                else d[b | bit][w] = got;
            }
        }
    }
}

// Stores the 16 columns of each lane's row (re, im; columns n0 ..), element (row, n0) at off.  A lane's own row would
// make every 16-byte store of a warp touch 32 lines; after a transposition four lanes store 64 bytes of one row, 8
// lines to a store.  rows: how many of the four rows from this lane group's first are valid; ldo: distance of rows.
template <int OUT>
__device__ __forceinline__ void store_rows(const FieldIO& f, long long off, long long ldo, int rows, int cols, int lane,
                                           ff* re, ff* im) {
    const int a = lane & 3;
    auto put = [&](void* base, auto size_c, int first, const uint32_t (&d)[4][4]) {  // 16 bytes = 16 / size columns
        constexpr int size = decltype(size_c)::value, per = 16 / size;
        const int n = first + a * per;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            if (s >= rows || n >= cols) continue;
            uint8_t* p = static_cast<uint8_t*>(base) + (off + s * ldo + n) * size;
            if (n + per <= cols) {
                *reinterpret_cast<uint4*>(p) = make_uint4(d[s][0], d[s][1], d[s][2], d[s][3]);
            } else {
#pragma unroll
                for (int w = 0; w < 4; ++w)
                    if (n + w / (size / 4) < cols) reinterpret_cast<uint32_t*>(p)[w] = d[s][w];
            }
        }
    };
    uint32_t d[4][4];
    if constexpr (OUT == FMT_FF) {
        float* planes[4] = {f.re_hi, f.re_lo, f.im_hi, f.im_lo};
#pragma unroll
        for (int p = 0; p < 4; ++p) {
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                const ff v = p < 2 ? re[k] : im[k];
                d[k >> 2][k & 3] = __float_as_uint(p & 1 ? v.lo : v.hi);
            }
            transpose4<4>(d, lane);
            put(planes[p], std::integral_constant<int, 4>{}, 0, d);
        }
    } else if constexpr (OUT == FMT_C128) {
        // A real loop that turns the columns through the same registers: unrolled, its conversions came to more
        // instructions than the cache holds beside the rest.
#pragma unroll 1
        for (int c = 0; c < 16; c += 4) {
            bool rare = false;
            auto set = [&](int k, double x, double y) {
                d[k][0] = (uint32_t)__double2loint(x), d[k][1] = (uint32_t)__double2hiint(x);
                d[k][2] = (uint32_t)__double2loint(y), d[k][3] = (uint32_t)__double2hiint(y);
            };
#pragma unroll
            for (int k = 0; k < 4; ++k) set(k, ff_to_double_fast(re[k], rare), ff_to_double_fast(im[k], rare));
            if (__builtin_expect(rare, 0)) {
#pragma unroll
                for (int k = 0; k < 4; ++k) set(k, ff_to_double_rare(re[k]), ff_to_double_rare(im[k]));
            }
            __syncwarp();
            transpose4<4>(d, lane);
            put(f.c128_out, std::integral_constant<int, 16>{}, c, d);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const ff r0 = re[k], i0 = im[k];
#pragma unroll
                for (int q = k; q < 12; q += 4) re[q] = re[q + 4], im[q] = im[q + 4];
                re[12 + k] = r0, im[12 + k] = i0;
            }
        }
    } else {
#pragma unroll
        for (int c = 0; c < 16; c += 8) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                d[k >> 1][2 * (k & 1)] = __float_as_uint(__fadd_rn(re[c + k].hi, re[c + k].lo));
                d[k >> 1][2 * (k & 1) + 1] = __float_as_uint(__fadd_rn(im[c + k].hi, im[c + k].lo));
            }
            transpose4<4>(d, lane);
            put(f.c64_out, std::integral_constant<int, 8>{}, c, d);
        }
    }
}

// Maxima over the 16 rows of each half warp of 16 columns: lane l (of a half) gets column l's.  15 exchanges, where a
// reduction for each column would take as many steps and 16 atomics.
__device__ __forceinline__ float column_max(float (&mag)[16], int lane) {
#pragma unroll
    for (int half = 8; half > 0; half >>= 1) {
        const bool high = lane & half;
#pragma unroll
        for (int k = 0; k < half; ++k) {
            const float got = __shfl_xor_sync(0xffffffffu, high ? mag[k] : mag[k + half], half);
            mag[k] = fmaxf(high ? mag[k + half] : mag[k], got);
        }
    }
    return mag[0];
}

// Every CTA loads both operands of its tiles itself, mostly from L2.
template <int OUT, int EMB>
__global__ void __launch_bounds__(NUM_THREADS, 1)
    split_stream_kernel(const __grid_constant__ GemmArgs g, int m_tiles, int tiles) {
    constexpr int TM = EMB ? 128 : 64;
    constexpr int TN = EMB ? SBN / 2 : SBN;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t raw_addr = ptx::smem_addr(smem_raw);
    uint8_t* smem = smem_raw + ((1024 - (raw_addr & 1023)) & 1023);
    uint8_t* extra = smem + STAGES * STAGE;
    uint64_t* bars = reinterpret_cast<uint64_t*>(extra);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(extra + 128);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(extra + 132);
    auto bar_full = [&](int s) { return ptx::smem_addr(&bars[s]); };
    auto bar_empty = [&](int s) { return ptx::smem_addr(&bars[STAGES + s]); };
    const uint32_t bar_accum = ptx::smem_addr(&bars[2 * STAGES]);      // a tile's MMAs are complete
    const uint32_t bar_drained = ptx::smem_addr(&bars[2 * STAGES + 1]);  // its levels are in registers
    const uint32_t bar_done = ptx::smem_addr(&bars[2 * STAGES + 2]);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            ptx::mbar_init(bar_full(s), 1);
            ptx::mbar_init(bar_empty(s), 1);
        }
        ptx::mbar_init(bar_accum, 1);
        ptx::mbar_init(bar_drained, EPI_WARPS);
        ptx::mbar_init(bar_done, 1);
        *abort_flag = 0;
        ptx::fence_mbar_init();
    }
    if (warp == 1) {
        ptx::tmem_alloc(ptx::smem_addr(tmem_slot), TMEM_COLS);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    const uint32_t smem_base = ptx::smem_addr(smem);
    const int nkt = g.ktiles;
    const int tile0 = blockIdx.x, step = gridDim.x;
    auto place = [&](int t, int& n_tile, int& m_tile, int& z) {
        n_tile = t % g.n_tiles;
        m_tile = t / g.n_tiles % m_tiles;
        z = t / g.n_tiles / m_tiles;
    };

    if (warp == 0) {
        if (lane == 0) {
            int last_use[STAGES];
            for (int s = 0; s < STAGES; ++s) last_use[s] = -1;
            int it = 0;
            for (int t = tile0; t < tiles && !*abort_flag; t += step) {
                int n_tile, m_tile, z;
                place(t, n_tile, m_tile, z);
                const int a_row0 = m_tile * BM + z * g.a_rows_per_z;
                const int b_row0 = n_tile * SBN + z * g.b_rows_per_z;
                for (int i = 0; i < nkt; ++i, ++it) {
                    if (*abort_flag) break;
                    const int s = it % STAGES, u = it / STAGES;
                    if (u > 0 && !ptx::mbar_wait_bounded(bar_empty(s), (u - 1) & 1, WAIT_LIMIT)) {
                        raise_status(g.status, abort_flag);
                        break;
                    }
                    uint8_t* sa = smem + s * STAGE;
                    uint8_t* sb = sa + STAGE_A;
                    ptx::mbar_arrive_expect_tx(bar_full(s), STAGE);
                    ptx::tma_load_3d(ptx::smem_addr(sa), &g.tmap_a, i * STREAM_BK, a_row0, 0, bar_full(s));
                    ptx::tma_load_3d(ptx::smem_addr(sb), &g.tmap_b, i * STREAM_BK, b_row0, 0, bar_full(s));
                    last_use[s] = u;
                }
            }
            // No copy may land in shared memory after this CTA exits.
            for (int s = 0; s < STAGES; ++s)
                if (last_use[s] >= 0 && !ptx::mbar_wait_bounded(bar_full(s), last_use[s] & 1, WAIT_LIMIT))
                    raise_status(g.status, abort_flag);
        }
        __syncwarp();
    } else if (warp == 1) {
        const bool leader = ptx::elect_one();
        bool ok = true;
        int it = 0, j = 0;
        for (int t = tile0; t < tiles && ok; t += step, ++j) {
            if (j > 0) ok = __all_sync(0xffffffffu, ptx::mbar_wait_bounded(bar_drained, (j - 1) & 1, WAIT_LIMIT));
            ptx::tc_fence_after();
            for (int i = 0; i < nkt && ok; ++i, ++it) {
                const int s = it % STAGES, u = it / STAGES;
                ok = __all_sync(0xffffffffu, ptx::mbar_wait_bounded(bar_full(s), u & 1, WAIT_LIMIT));
                if (!ok) break;
                ptx::tc_fence_after();
                slice_products<SBN, ROW_BYTES>(tmem, smem_base + s * STAGE, i == 0, leader);
                if (leader) ptx::umma_commit(bar_empty(s));
            }
            if (!ok && leader) raise_status(g.status, abort_flag);
            if (leader) ptx::umma_commit(bar_accum);
        }
        // TMEM and the pipeline buffers are released only after every MMA issued above.
        if (leader) ptx::umma_commit(bar_done);
        if (!__all_sync(0xffffffffu, ptx::mbar_wait_bounded(bar_done, 0, WAIT_LIMIT)) && leader)
            raise_status(g.status, abort_flag);
    } else {
        const int quarter = warp & 3;      // TMEM lane quarter this warp may access
        const int slot = (warp - 2) >> 2;  // its 32 of the 128 TMEM columns of a level
        const uint32_t base = tmem + ((uint32_t)(quarter * 32) << 16) + slot * 32;
        const int upper = lane >> 4;
        const cff alpha = {{g.alpha[0], g.alpha[1]}, {g.alpha[2], g.alpha[3]}};
        const bool real_alpha = g.alpha[2] == 0.0f && g.alpha[3] == 0.0f;
        const bool imag_alpha = g.alpha[0] == 0.0f && g.alpha[1] == 0.0f;
        const bool unit_alpha = real_alpha && g.alpha[0] == 1.0f && g.alpha[1] == 0.0f;
        const float2* mask = g.epi == HX_EPI_MUL ? g.mask : nullptr;
        const bool mask_pairs = g.N % 2 == 0 && (reinterpret_cast<uintptr_t>(mask) & 15) == 0;
        int j = 0;
        for (int t = tile0; t < tiles; t += step, ++j) {
            int n_tile, m_tile, z;
            place(t, n_tile, m_tile, z);
            // this thread's row and its 16 columns
            const int m = m_tile * TM + (EMB ? quarter * 32 + lane : quarter * 16 + (lane & 15));
            const int n0 = n_tile * TN + (EMB ? slot * 16 : slot * 32 + upper * 16);
            const bool row_ok = m < g.M;
            const float rsc = row_ok ? __ldg(&g.row_scale[z * g.row_scale_z + m]) : 0.0f;
            const float2* mrow = mask && row_ok ? mask + (long long)(m % g.rows_per_field) * g.N : nullptr;
            const float* csc = g.col_scale + z * g.col_scale_z;

            if (!ptx::mbar_wait_bounded(bar_accum, j & 1, WAIT_LIMIT)) raise_status(g.status, abort_flag);
            ptx::tc_fence_after();
            // Warp-uniform decision: the TMEM loads below are .sync.aligned.
            if (!__shfl_sync(0xffffffffu, (int)(*abort_flag == 0), 0)) break;
            ff v[32];
#pragma unroll
            for (int h = 0; h < 32; h += 8) {
                float v0[8], v1[8], v2[8], v3[8];
                ptx::tmem_ld_8x4(base + h, SBN, v0, v1, v2, v3);
#pragma unroll
                for (int q = 0; q < 8; ++q) v[h + q] = combine_levels(v0[q], v1[q], v2[q], v3[q]);
            }
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(bar_drained);

            if (!EMB) {
                // The lower half of the warp holds 16 rows of Re, the upper half the same rows of Im: swap half of the
                // columns, so that each thread has Re (v[0..15]) and Im (v[16..31]) of 16 columns.
#pragma unroll
                for (int q = 0; q < 16; ++q) {
                    const ff give = upper ? v[q] : v[16 + q];
                    const ff got = {__shfl_xor_sync(0xffffffffu, give.hi, 16), __shfl_xor_sync(0xffffffffu, give.lo, 16)};
                    if (upper) v[q] = got;
                    else v[16 + q] = got;
                }
            }
            // v[re(k)], v[im(k)]: column k of this thread's row
            auto at_re = [](int k) { return EMB ? (k >> 3) * 16 + (k & 7) : k; };
            auto at_im = [](int k) { return EMB ? (k >> 3) * 16 + (k & 7) + 8 : 16 + k; };
            // `scale` is unrolled for each kind of factor on its own, so that a launch runs through the code of one: with the
            // kinds told apart in every column, waiting for instructions took most of the epilogue's time.
            ff re[16], im[16];
            auto scale = [&](auto times_alpha) {
#pragma unroll
                for (int k = 0; k < 16; ++k) {
                    const float sc = row_ok && n0 + k < g.N ? rsc * __ldg(&csc[n0 + k]) : 0.0f;  // powers of two: exact
                    const ff a = v[at_re(k)], b = v[at_im(k)];
                    const cff x = times_alpha(cff{{a.hi * sc, a.lo * sc}, {b.hi * sc, b.lo * sc}});
                    re[k] = x.re, im[k] = x.im;
                }
            };
            if (unit_alpha) scale([](cff x) { return x; });
            else if (real_alpha) scale([&](cff x) { return cff{ff_mul(x.re, alpha.re), ff_mul(x.im, alpha.re)}; });
            else if (imag_alpha) scale([&](cff x) { return cff{ff_neg(ff_mul(x.im, alpha.im)), ff_mul(x.re, alpha.im)}; });
            else scale([&](cff x) { return cff_mul(x, alpha); });
            if (mask) {
#pragma unroll
                for (int k = 0; k < 16; k += 2) {
                    float2 mk[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
                    if (mask_pairs && row_ok && n0 + k + 1 < g.N) {
                        const float4 w = __ldg(reinterpret_cast<const float4*>(mrow + n0 + k));
                        mk[0] = make_float2(w.x, w.y), mk[1] = make_float2(w.z, w.w);
                    } else if (row_ok) {
#pragma unroll
                        for (int q = 0; q < 2; ++q)
                            if (n0 + k + q < g.N) mk[q] = __ldg(&mrow[n0 + k + q]);
                    }
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const cff x = {re[k + q], im[k + q]};
                        const cff y = mk[q].y == 0.0f ? cff{ff_mulf(x.re, mk[q].x), ff_mulf(x.im, mk[q].x)}
                                                      : cff_mul_c64(x, mk[q]);
                        re[k + q] = y.re, im[k + q] = y.im;
                    }
                }
            }
            const int first = m - (lane & 3);  // row of the first lane of the group of four
            store_rows<OUT>(g.out, z * g.out_z + (long long)first * g.ldo + n0, g.ldo, g.M - first, g.N - n0, lane, re, im);
            if (!g.colmax && !g.rowmax) continue;
            float mag[16];
            float rmax = 0.0f;
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                const bool ok = row_ok && n0 + k < g.N;
                mag[k] = ok ? fmaxf(0.0f, fmaxf(fabsf(re[k].hi), fabsf(im[k].hi))) : 0.0f;  // NaN passed over
                rmax = fmaxf(rmax, mag[k]);
            }
            if (g.colmax) {
                const int field = row_ok && g.colmax_rows_per_field > 0 ? m / g.colmax_rows_per_field : 0;
                const int field0 = __shfl_sync(0xffffffffu, field, 0);
                unsigned int* cm = g.colmax + z * g.colmax_z;
                if (__all_sync(0xffffffffu, !row_ok || field == field0)) {
                    float mx = column_max(mag, lane);
                    if (EMB) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                    if (mx > 0.0f && (!EMB || !upper))
                        atomicMax(&cm[field0 * g.colmax_field_stride + n0 + (lane & 15)], __float_as_uint(mx));
                } else {
#pragma unroll
                    for (int k = 0; k < 16; ++k)
                        if (mag[k] > 0.0f) atomicMax(&cm[field * g.colmax_field_stride + n0 + k], __float_as_uint(mag[k]));
                }
            }
            if (g.rowmax) {
                if (!EMB) rmax = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, 16));
                if (row_ok && rmax > 0.0f && (EMB || !upper))
                    atomicMax(&g.rowmax[z * g.rowmax_z + m], __float_as_uint(rmax));
            }
        }
    }
    ptx::tc_fence_before();
    __syncwarp();
    __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem, TMEM_COLS);
    }
}

template <int OUT, int EMB> int launch(const GemmArgs& g, int m_tiles, int tiles, int ctas, cudaStream_t st) {
    static bool configured[64];
    auto kern = split_stream_kernel<OUT, EMB>;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        HX_TRY(cuda_status(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM),
                           "cudaFuncSetAttribute(split_stream_kernel)"));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    kern<<<(unsigned)ctas, NUM_THREADS, SMEM, st>>>(g, m_tiles, tiles);
    return launch_status("split_stream_kernel");
}

template <int OUT> int launch_emb(const GemmArgs& g, int m_tiles, int tiles, int ctas, cudaStream_t st) {
    return g.emb ? launch<OUT, 1>(g, m_tiles, tiles, ctas, st) : launch<OUT, 0>(g, m_tiles, tiles, ctas, st);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

bool stream_fits(const GemmArgs& g) {
    if (g.ksplit != 1 || (g.epi != HX_EPI_NONE && g.epi != HX_EPI_MUL)) return false;
    switch (output_fmt(g.out)) {
        case FMT_FF:
            return g.ldo % 4 == 0 && g.out_z % 4 == 0 && aligned16(g.out.re_hi) && aligned16(g.out.re_lo) &&
                   aligned16(g.out.im_hi) && aligned16(g.out.im_lo);
        case FMT_C128: return true;
        default: return g.ldo % 2 == 0 && g.out_z % 2 == 0 && aligned16(g.out.c64_out);
    }
}

int launch_stream(const GemmArgs& g, int m_tiles, int tiles, int ctas, cudaStream_t st) {
    switch (output_fmt(g.out)) {
        case FMT_FF: return launch_emb<FMT_FF>(g, m_tiles, tiles, ctas, st);
        case FMT_C128: return launch_emb<FMT_C128>(g, m_tiles, tiles, ctas, st);
        default: return launch_emb<FMT_C64>(g, m_tiles, tiles, ctas, st);
    }
}

}  // namespace sg
}  // namespace hx
