// fdk.cu -- the ramp filter of filtered backprojection (FDK), for the FDK-weighted VI
// backprojector (vi_device.cuh, FDK = true).
//
// The filter follows the reference's ramp_filter_TOMO8.m (Matlab/Tomo8): a ramp |k| over an
// oversampled length M = oversampling * nu, normalised to 1, times a centred Hann window of
// round(M * cutoff) points (made even), taken back to the spatial domain; the taps of lags
// -round(nu/2) .. round(nu/2) - 1 (those the Matlab code keeps after its 2 nu-point
// circular convolution) are applied to every detector row, zero outside the row, and the
// result divided by 2 du. The taps are computed once per (nu, oversampling, cutoff) on the
// host in double; the convolution runs in FP32.
#include <cmath>
#include <vector>

#include "tomo_kernels.cuh"

namespace tomo {

// Spatial taps of ramp_filter_TOMO8 for rows of nu pixels, scaled by 1 / (2 du). Returns
// half = round(nu / 2) and taps[l] for lag l - half, l in [0, 2 half).
int ramp_taps(int nu, int oversampling, double cutoff, double du, std::vector<float>& taps) {
    const long M = (long)oversampling * nu;
    // window: hann(Nr) (symmetric), Nr = round(M cutoff) made even, centred in M points,
    // then fftshift (even M: a shift by M/2)
    long nr = (long)std::floor(M * cutoff + 0.5);
    if (nr % 2) --nr;
    std::vector<double> win(M, 0.0), g(M);
    const long off = (M - nr) / 2;
    for (long n = 0; n < nr; ++n)
        win[off + n] = nr > 1 ? 0.5 * (1.0 - std::cos(2.0 * M_PI * n / (double)(nr - 1))) : 1.0;
    for (long k = 0; k < M; ++k) {
        const double ramp = (double)(k <= M / 2 ? k : M - k) / (double)(M / 2);  // |k| in FFT order, max 1
        g[k] = ramp * win[(k + M / 2) % M];
    }
    std::vector<double> cs(M);
    for (long k = 0; k < M; ++k) cs[k] = std::cos(2.0 * M_PI * (double)k / (double)M);
    const int half = (int)std::floor(nu / 2.0 + 0.5);
    const int lo = (int)std::floor(3.0 * nu / 2.0 + 0.5) - 2 * nu;  // most negative kept lag
    taps.assign(2 * half, 0.f);
    for (int l = 0; l < 2 * half; ++l) {
        const int lag = l - half;
        if (lag < lo) continue;
        // real part of the inverse DFT at n = lag mod M
        const long n = lag >= 0 ? lag : M + lag;
        double s = 0.0;
        for (long k = 0, kn = 0; k < M; ++k, kn = (kn + n) % M) s += g[k] * cs[kn];
        taps[l] = (float)(s / (double)M / (2.0 * du));
    }
    return half;
}

// Each output is the sum over l ascending of taps[l] row[i - (l - half)]. A warp filters 32
// rows (one per lane) for 32 consecutive outputs: the tap of (output k, pixel j) depends on
// k - j only, so the 32 taps in use are the same for all lanes and slide by one per pixel; a
// pixel costs one shared-memory read of its own, one of the next tap and 32 FMAs, which is
// what bounds it (one thread per output read two words per FMA). Pixels run in descending j in
// segments of 32; taps outside [0, 2 half) are skipped, not multiplied by zero, so a pixel
// only reaches the outputs within its lags whatever its value. 256^3, 256 views: the filter
// and the FDK backprojection together 4.62 -> 4.09 ms.
constexpr int RAMP_WARPS = 4;  // 128 outputs per block
template <typename Ti>
__global__ void __launch_bounds__(32 * RAMP_WARPS) ramp_filter_kernel(const Ti* __restrict__ in, float* __restrict__ out,
                                                                     const float* __restrict__ taps, int half, int nu,
                                                                     long rows) {
    __shared__ float px[32][33];                     // [pixel of the segment][row]
    __shared__ float tp[32 * RAMP_WARPS + 32];       // taps of (k - j) for the block's outputs
    __shared__ float tile[RAMP_WARPS][32][33];       // [output][row]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ib = blockIdx.y * (32 * RAMP_WARPS), i0 = ib + warp * 32;
    const long r0 = (long)blockIdx.x * 32;
    const int nr = (int)min(32l, rows - r0);
    const int ilast = min(nu, ib + 32 * RAMP_WARPS) - 1;
    const int jlo = max(0, ib - half + 1), jhi = min(nu - 1, ilast + half);
    float acc[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) acc[k] = 0.f;
    for (int je = jhi; je >= jlo; je -= 32) {
        const int js = je - 31;  // pixels below jlo are not used
        __syncthreads();
        for (int r = warp; r < 32; r += RAMP_WARPS) {
            const int j = js + lane;
            px[lane][r] = r < nr && j >= jlo ? ldp(in + (r0 + r) * nu + j) : 0.f;
        }
        const int lb = ib - je + half;  // lag index of (output ib, pixel je)
        for (int t = threadIdx.x; t < 32 * RAMP_WARPS + 32; t += 32 * RAMP_WARPS)
            tp[t] = lb + t >= 0 && lb + t < 2 * half ? __ldg(taps + lb + t) : 0.f;
        __syncthreads();
        const int l0 = i0 - je + half;  // lag index of (output i0, pixel je)
        const float* w = tp + warp * 32;
        if (js >= jlo && l0 >= 0 && l0 + 62 < 2 * half) {
            float win[32];
#pragma unroll
            for (int k = 0; k < 32; ++k) win[k] = w[k];
#pragma unroll
            for (int s = 0; s < 32; ++s) {
                const float x = px[31 - s][lane];
#pragma unroll
                for (int k = 0; k < 32; ++k) acc[k] = fmaf(win[(k + s) & 31], x, acc[k]);
                if (s < 31) win[s] = w[32 + s];
            }
        } else {
            for (int s = 0; s < 32 && je - s >= jlo; ++s) {
                const float x = px[31 - s][lane];
#pragma unroll
                for (int k = 0; k < 32; ++k)
                    if ((unsigned)(l0 + s + k) < (unsigned)(2 * half)) acc[k] = fmaf(w[s + k], x, acc[k]);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 32; ++k) tile[warp][k][lane] = acc[k];
    __syncwarp();
    if (i0 + lane < nu)
        for (int r = 0; r < nr; ++r) out[(r0 + r) * nu + i0 + lane] = tile[warp][lane][r];
}

// The same sums in the same order, one block per detector row: it loads the row before it writes,
// so the output may be the input, and a thread has one output, so few rows still spread over the
// chip where the tiles above wait for one another's pixels.
template <typename Ti>
__global__ void ramp_row_kernel(const Ti* in, float* out, const float* __restrict__ taps, int half, int nu) {
    extern __shared__ float sm[];
    float *row = sm, *tp = sm + nu;  // the row's pixels, the 2 half taps
    const long r = blockIdx.x;
    for (int i = threadIdx.x; i < nu; i += blockDim.x) row[i] = ldp(in + r * nu + i);
    for (int i = threadIdx.x; i < 2 * half; i += blockDim.x) tp[i] = taps[i];
    __syncthreads();
    for (int i = threadIdx.x; i < nu; i += blockDim.x) {
        float acc = 0.f;
        const int l0 = max(0, i - nu + 1 + half), l1 = min(2 * half, i + half + 1);
        for (int l = l0; l < l1; ++l) acc = fmaf(tp[l], row[i - (l - half)], acc);
        out[r * nu + i] = acc;
    }
}

cudaError_t launch_ramp_filter(const void* in, tomo_dtype idt, float* out, const float* taps, int half, int nu, int nv,
                               int np, cudaStream_t st) {
    const long rows = (long)nv * np;
    const size_t smem = (size_t)(nu + 2 * half) * sizeof(float);
    const uintptr_t i0 = (uintptr_t)in, i1 = i0 + (size_t)rows * nu * dtype_size(idt), o0 = (uintptr_t)out;
    const bool overlap = i0 < o0 + (size_t)rows * nu * sizeof(float) && o0 < i1;
    // Row by row / in tiles, us: 64 pixels x 4096 rows 10.2 / 13.5, 128 x 4096 18.6 / 22.8, 128 x 8192
    // 33.0 / 28.9, 256 x 64 8.9 / 28.9, 256 x 2048 28.9 / 29.0, 256 x 65536 796 / 373, 512 x 512
    // 31 / 41, 512 x 1024 52 / 41, 1024 x 128 33 / 64, 1024 x 512 110 / 64, 2048 x 1 115 / 98.
    const bool few = nu <= 1536 && (nu < 64 ? rows <= 6144 : (double)rows * nu * nu <= (nu < 256 ? 1.2e8 : 1.8e8));
    if (overlap || few) {
        switch (idt) {
            case TOMO_F32: ramp_row_kernel<<<(unsigned)rows, 256, smem, st>>>((const float*)in, out, taps, half, nu); break;
            case TOMO_BF16:
                ramp_row_kernel<<<(unsigned)rows, 256, smem, st>>>((const __nv_bfloat16*)in, out, taps, half, nu);
                break;
            case TOMO_F16: ramp_row_kernel<<<(unsigned)rows, 256, smem, st>>>((const __half*)in, out, taps, half, nu); break;
        }
        return cudaGetLastError();
    }
    const dim3 grid((unsigned)((rows + 31) / 32), (nu + 32 * RAMP_WARPS - 1) / (32 * RAMP_WARPS)), block(32 * RAMP_WARPS);
    switch (idt) {
        case TOMO_F32: ramp_filter_kernel<<<grid, block, 0, st>>>((const float*)in, out, taps, half, nu, rows); break;
        case TOMO_BF16: ramp_filter_kernel<<<grid, block, 0, st>>>((const __nv_bfloat16*)in, out, taps, half, nu, rows); break;
        case TOMO_F16: ramp_filter_kernel<<<grid, block, 0, st>>>((const __half*)in, out, taps, half, nu, rows); break;
    }
    return cudaGetLastError();
}

}  // namespace tomo
