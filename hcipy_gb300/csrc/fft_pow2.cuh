// Register-resident FFT of complex64 lines whose length is a power of two from 256 to 4096 points.
//
// The same transform as fft_line_kernel (zero-padding and index shift on load, phase factors, index shift and
// crop on store; see fft_line.cuh for the index maps), specialised at compile time for one length N:
//   N = 4096: three radix-16 stages;  N = 256: two;  N = 512 / 1024 / 2048: two radix-16 stages and a last
//   radix-2 / 4 / 8 stage.
// Each thread owns one 16-point butterfly per stage (N/16 threads per line).  The first stage reads its 16
// inputs straight from global memory (only the valid ones; padding is never loaded), and the last stage writes
// its outputs, which are then in natural order, straight to global memory, so a 4096-point line makes two round
// trips through shared memory and the index arithmetic is shifts and masks of compile-time constants.  Stockham
// stage with radix R after sub-transforms of length Ns: butterfly j (k = j mod Ns) reads x[j + r N/R], multiplies
// by W^(r k) with W = exp(-+2 pi i / (Ns R)), and writes (j / Ns) Ns R + k + r Ns.  Shared memory holds one
// padding element per 16, so the stride-16 writes of the first stage hit distinct banks.
//
// CONV (the column pass of the Fourier filter): a forward transform, the product with the transfer function and the
// inverse transform in one launch.  Thread t holds the spectrum at t + r N/16, which are the inputs of its own first
// inverse butterfly, so the spectrum never leaves the registers.
//
// The kernel is bound by instruction issue (1912 instructions a thread for the 16 points of a 4096-point line in a form
// with 64-bit index products, general shared-memory indices and a complex scale, 56% issued), so: offsets into shared
// memory are compile-time constants from one base, every global access is one 32 x 32-bit product from a line pointer,
// complex additions are packed (two FP32 additions per instruction), and the lines of a CTA synchronise on their own
// where a line's threads are whole warps.  1435 instructions now, 62% issued: the padded FFT of 1024^2 points to 4096^2
// 160 -> 94 us (1024 columns 27, then 4096 rows 65), the filter's column pass over 2048 points 121 -> 36 us.
#pragma once

#include "fft_line.cuh"

namespace hx {

template <int N> struct Pow2Shape {
    static_assert(N == 256 || N == 512 || N == 1024 || N == 2048 || N == 4096, "supported lengths");
    static constexpr int T = N / 16;                  // threads per line
    static constexpr int RL = N == 4096 ? 1 : N / 256;  // radix of the last stage (1: none)
    // Threads per CTA: 512, two CTAs per SM; 1024 for strided lines of 4096 points, so that a CTA reads and writes
    // segments of four lines (32 bytes, a sector) and not of two.
    template <bool LF> __host__ __device__ static constexpr int threads() { return LF && N == 4096 ? 1024 : 512; }
    // Lines per CTA where there are enough.
    template <bool LF> __host__ __device__ static constexpr int lines() { return threads<LF>() / T; }
    // Shared-memory elements per line.  In a column pass a half warp's 16 accesses of 8 bytes are to 16 / lines() points
    // of lines() lines, which the extra elements spread over the banks.
    template <bool LF> __host__ __device__ static constexpr int pitch() {
        return N + N / 16 + (LF ? (lines<LF>() < 16 ? 16 / lines<LF>() : 1) : 0);
    }
};

// ---- packed FP32 ------------------------------------------------------------------------------------------------

__device__ __forceinline__ float2 p2_add(float2 a, float2 b) {
    float2 r;
    asm("add.rn.f32x2 %0, %1, %2;"
        : "=l"(reinterpret_cast<unsigned long long&>(r))
        : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
    return r;
}
__device__ __forceinline__ float2 p2_sub(float2 a, float2 b) {
    // a - b as fma(b, -1, a), which rounds once like the subtraction
    float2 r;
    const unsigned long long m1 = 0xbf800000bf800000ull;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(reinterpret_cast<unsigned long long&>(r))
        : "l"(reinterpret_cast<unsigned long long&>(b)), "l"(m1), "l"(reinterpret_cast<unsigned long long&>(a)));
    return r;
}

// 4-point DFT in place over v[i0 + st k] (W = exp(SIGN 2 pi i / 4)).
template <int SIGN> __device__ __forceinline__ void p2_dft4(float2* v, int i0, int st) {
    const float2 a = v[i0], b = v[i0 + st], c = v[i0 + 2 * st], d = v[i0 + 3 * st];
    const float2 t0 = p2_add(a, c), t1 = p2_sub(a, c), t2 = p2_add(b, d), t3 = p2_sub(b, d);
    v[i0] = p2_add(t0, t2);
    v[i0 + 2 * st] = p2_sub(t0, t2);
    if (SIGN < 0) {
        v[i0 + st] = make_float2(t1.x + t3.y, t1.y - t3.x);
        v[i0 + 3 * st] = make_float2(t1.x - t3.y, t1.y + t3.x);
    } else {
        v[i0 + st] = make_float2(t1.x - t3.y, t1.y + t3.x);
        v[i0 + 3 * st] = make_float2(t1.x + t3.y, t1.y - t3.x);
    }
}

// 16-point DFT as 4 x 4, in slot order: X[k1 + 4 k2] in v[4 k1 + k2] (p2_out).
template <int SIGN> __device__ __forceinline__ void p2_dft16(float2* v) {
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) p2_dft4<SIGN>(v, n2, 4);
    v[5] = w16<float, SIGN, 1>(v[5]);
    v[9] = w16<float, SIGN, 2>(v[9]);
    v[13] = w16<float, SIGN, 3>(v[13]);
    v[6] = w16<float, SIGN, 2>(v[6]);
    v[10] = w16<float, SIGN, 4>(v[10]);
    v[14] = w16<float, SIGN, 6>(v[14]);
    v[7] = w16<float, SIGN, 3>(v[7]);
    v[11] = w16<float, SIGN, 6>(v[11]);
    v[15] = w16<float, SIGN, 9>(v[15]);
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) p2_dft4<SIGN>(v, 4 * k1, 1);
}
__host__ __device__ constexpr int p2_out(int r) { return (r >> 2) + 4 * (r & 3); }

// ---- stages -----------------------------------------------------------------------------------------------------

// Stage twiddle tables of an N-point line (built at plan time, see make_stage_tables): for the radix-16 stages
// NS = 16 and 256, four rows of NS entries, exp(-2 pi i p k / (16 NS)) for p = 1, 2, 4, 8, so that the threads of a
// warp (consecutive k) read consecutive entries.  Offset of the stage's rows in the table:
template <int NS> __host__ __device__ constexpr int p2_tw_offset() { return NS == 16 ? 0 : 4 * 16; }
constexpr int kP2TwEntries = 4 * 16 + 4 * 256;

// v[r] *= W^(r k) for the 16 points of a radix-16 butterfly, W = exp(-+2 pi i / (16 NS)), from the stage's four
// table rows (W^k, W^2k, W^4k, W^8k) and products at most three deep.
template <int SIGN, int NS>
__device__ __forceinline__ void p2_twiddle16(float2* v, int k, const float2* __restrict__ tws) {
    const float2* t = tws + p2_tw_offset<NS>() + k;
    float2 w1 = __ldg(t), w2 = __ldg(t + NS), w4 = __ldg(t + 2 * NS), w8 = __ldg(t + 3 * NS);
    if (SIGN > 0) {
        w1.y = -w1.y;
        w2.y = -w2.y;
        w4.y = -w4.y;
        w8.y = -w8.y;
    }
    float2 wl[8];
    wl[1] = w1;
    wl[2] = w2;
    wl[3] = c_mul(w2, w1);
    wl[4] = w4;
    wl[5] = c_mul(w4, w1);
    wl[6] = c_mul(w4, w2);
    wl[7] = c_mul(w4, wl[3]);
    v[8] = c_mul(v[8], w8);
#pragma unroll
    for (int r = 1; r < 8; ++r) {
        v[r] = c_mul(v[r], wl[r]);
        v[8 + r] = c_mul(v[8 + r], c_mul(w8, wl[r]));
    }
}

// Shared-memory element x of a line lies at x + x / 16; the accesses of a stage are one base plus constants.
// Inputs of butterfly t: x = t + r N/16.
template <int N> __device__ __forceinline__ void p2_read16(const float2* buf, int t, float2* v) {
    const float2* p = buf + t + (t >> 4);
#pragma unroll
    for (int r = 0; r < 16; ++r) v[r] = p[r * (N / 16 + N / 256)];
}
// Outputs of stage NS = 1 (x = 16 t + m) and NS = 16 (x = 256 (t / 16) + t % 16 + 16 m), from slot order.
template <int NS> __device__ __forceinline__ void p2_write16(float2* buf, int t, const float2* v) {
    float2* p = NS == 1 ? buf + 17 * t : buf + 272 * (t >> 4) + (t & 15);
#pragma unroll
    for (int r = 0; r < 16; ++r) p[p2_out(r) * (NS == 1 ? 1 : 17)] = v[r];
}

// The lines of a CTA in step: a line's threads alone where they are whole warps of one line.
template <int T, bool LF> __device__ __forceinline__ void p2_sync(int line) {
    if constexpr (LF) __syncthreads();
    else if constexpr (T == 32) __syncwarp();
    else if constexpr (T >= 64) asm volatile("bar.sync %0, %1;" ::"r"(line + 1), "r"(T) : "memory");
    else __syncthreads();
}

// Transform of the 16 values v[r] = x[t + r N/16] of a line; on return v[p2_slot<N>(s)] = X[t + s N/16].
template <int N, int SIGN, bool LF>
__device__ __forceinline__ void p2_transform(float2* v, float2* buf, int t, int line, const float2* __restrict__ tw,
                                             const float2* __restrict__ tws) {
    constexpr int T = N / 16;
    p2_dft16<SIGN>(v);
    p2_write16<1>(buf, t, v);
    p2_sync<T, LF>(line);
    p2_read16<N>(buf, t, v);
    p2_twiddle16<SIGN, 16>(v, t & 15, tws);
    p2_dft16<SIGN>(v);
    if constexpr (N > 256) {
        p2_sync<T, LF>(line);
        p2_write16<16>(buf, t, v);
        p2_sync<T, LF>(line);
        if constexpr (N == 4096) {
            p2_read16<N>(buf, t, v);
            p2_twiddle16<SIGN, 256>(v, t, tws);
            p2_dft16<SIGN>(v);
        } else {
            // last stage, radix RL after 256-point sub-transforms: butterflies b = t + i T (i < 16 / RL), inputs
            // b + 256 r, twiddles W_N^(r b), outputs b + 256 r = t + (i + 16 / RL r) T
            constexpr int RL = Pow2Shape<N>::RL, NB = 16 / RL;
            const float2* p = buf + t + (t >> 4);
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                float2 u[RL];
#pragma unroll
                for (int r = 0; r < RL; ++r) {
                    // element t + i T + 256 r: t / 16 carries into the padding only with T a multiple of 16
                    u[r] = p[(i * T + 256 * r) + ((i * T + 256 * r) >> 4)];
                    if (r > 0) {
                        float2 w = __ldg(&tw[r * (t + i * T)]);
                        if (SIGN > 0) w.y = -w.y;
                        u[r] = c_mul(u[r], w);
                    }
                }
                Dft<float, RL, SIGN>::run(u);
#pragma unroll
                for (int r = 0; r < RL; ++r) v[i + NB * r] = u[r];
            }
        }
    }
}
// Register of X[t + s N/16] after p2_transform.
template <int N> __host__ __device__ constexpr int p2_slot(int s) {
    return (N == 256 || N == 4096) ? p2_out(s) : s;  // p2_out is its own inverse
}

// grid: x = blocks of lines_per_cta lines, y = batch; blockDim = lines_per_cta * N / 16.  LF: lines adjacent in
// memory (a column pass), so consecutive threads take consecutive lines and the global accesses coalesce across
// lines; else consecutive threads take consecutive points of one line.  CONV: SIGN is that of the first transform.
template <int N, int SIGN, bool LF, bool CONV>
__global__ void __launch_bounds__(Pow2Shape<N>::template threads<LF>(), 1024 / Pow2Shape<N>::template threads<LF>())
    fft_pow2_kernel(const __grid_constant__ LineArgs<float> a) {
    constexpr int T = Pow2Shape<N>::T;
    extern __shared__ __align__(16) float2 p2_smem[];
    const int lpc = a.lines_per_cta;
    const int line = LF ? (int)threadIdx.x & (lpc - 1) : (int)threadIdx.x / T;
    const int t = LF ? (int)threadIdx.x >> (31 - __clz(lpc)) : (int)threadIdx.x % T;
    const long long l = (long long)blockIdx.x * lpc + line;
    const bool lok = l < a.nlines;
    float2* buf = p2_smem + line * Pow2Shape<N>::template pitch<LF>();
    const float2* in = a.in + a.in_bs * blockIdx.y + l * a.in_ls;
    float2* out = a.out + a.out_bs * blockIdx.y + l * a.out_ls;
    const int in_es = LF ? (int)a.in_es : 1, out_es = LF ? (int)a.out_es : 1;

    // ---- inputs x[t + r T], taken from position (t + r T + load_add - in_offset) mod N of the input line -----------
    const int lshift = (a.load_add - a.in_offset) & (N - 1);
    float2 v[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const int p = (t + r * T + lshift) & (N - 1);
        v[r] = make_float2(0.0f, 0.0f);
        if (lok && p < a.in_count) v[r] = in[(long long)p * in_es];
    }
    if (a.pre) {
        const float2* pre = a.pre + l * a.pre_ls;
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const int p = (t + r * T + lshift) & (N - 1);
            if (lok && p < a.in_count) v[r] = c_mul(v[r], pre[p]);
        }
    }
    p2_transform<N, SIGN, LF>(v, buf, t, line, a.tw, a.tws);
    if constexpr (CONV) {
        const int mid_es = (int)a.mid_es;
        const float2* mid = a.mid + l * a.mid_ls + (long long)t * mid_es;
        const float cs = a.mid_conj ? -1.0f : 1.0f;
        float2 u[16];
#pragma unroll
        for (int s = 0; s < 16; ++s) {
            float2 m = make_float2(0.0f, 0.0f);
            if (lok) m = __ldg(mid + (long long)(s * T) * mid_es);
            m.y *= cs;
            u[s] = c_mul(v[p2_slot<N>(s)], m);
        }
        p2_sync<T, LF>(line);  // the last reads of the first transform
        p2_transform<N, -SIGN, LF>(u, buf, t, line, a.tw, a.tws);
#pragma unroll
        for (int s = 0; s < 16; ++s) v[s] = u[s];
    }

    // ---- output (t + s T - out_offset - store_add) mod N of the output line is X[t + s T] ---------------------------
    const int sshift = (-(a.out_offset + a.store_add)) & (N - 1);
    if (a.scale.y != 0.0f) {
#pragma unroll
        for (int s = 0; s < 16; ++s) v[s] = c_mul(v[s], a.scale);
    } else if (a.scale.x != 1.0f) {
#pragma unroll
        for (int s = 0; s < 16; ++s) v[s] = make_float2(v[s].x * a.scale.x, v[s].y * a.scale.x);
    }
    if (a.post) {
        const float2* post = a.post + l * a.post_ls;
        const int post_es = (int)a.post_es;
#pragma unroll
        for (int s = 0; s < 16; ++s) {
            const int kk = (t + s * T + sshift) & (N - 1);
            if (lok && kk < a.out_count) v[p2_slot<N>(s)] = c_mul(v[p2_slot<N>(s)], post[(long long)kk * post_es]);
        }
    }
#pragma unroll
    for (int s = 0; s < 16; ++s) {
        const int kk = (t + s * T + sshift) & (N - 1);
        if (lok && kk < a.out_count) out[(long long)kk * out_es] = v[p2_slot<N>(s)];
    }
}

}  // namespace hx
