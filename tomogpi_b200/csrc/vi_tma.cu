// vi_tma.cu -- VI backprojector with each view's detector window staged in shared memory by
// the Tensor Memory Accelerator (TMA), single GPU.
//
// What the default tuning and the "tma" form run, for VI, its UM variant and the FDK weights.
// The block is the VI tile of vi_device.cuh (32 x 8 voxel columns, NS = 16, 8 or 4 slices per
// thread: eight consumer warps) plus one producer warp. For every view the producer bounds the
// detector window the tile's voxels can touch -- the projections of the tile's corner columns
// at its first and last slice; u and v are monotone in x, y and z over the tile, so the
// corners give the extremes -- and copies that box of the FP32 sinogram [P][nv][pitch] into
// one of three shared-memory stages with one cp.async.bulk.tensor (into this CTA only; the tensor
// map covers this GPU's own buffer). Texels off the detector come back as zeros (the TMA's
// out-of-bounds fill), which is the texture border of the reference (a sample there adds 0,
// as skipping it does). mbarriers hand the stages over: `full` (the copy's bytes landed),
// `empty` (the eight consumer warps are done with it). Consumers run the same arithmetic as
// vi_tile (backprojection3D_kernel_16reg.cuh:401-453: u, A, v by repeated addition, the
// three lerps, FP32 sums in view order) with the four texels of a sample read from shared
// memory; a view whose window exceeds the box reads that view's texels from global memory
// instead. Same texels, same operations, bit-identical to vi_tile.
//
// Measured (B200): 512^3, 512 views 44.1 ms (51.6 before the window checks moved from every
// thread to the producer, the texture's 0.5 offsets went and the reads took byte addresses;
// the padded form 72.3); 256^3 2.81 ms (padded 4.85); filter and FDK backprojection together 4.62 ms
// (padded 9.99: the weights take a reciprocal square root now, in place of an IEEE division and
// root per sample); 64^3, 60 views 35 us (padded, 64 blocks of 16 slices: 148).
//
// Every wait is bounded (one second by the global timer): a wait that gives up sets
// ERR_TIMEOUT in the context's error word and the block stops; the producer first waits
// (bounded) for the copies it issued.
#include <cuda.h>

#include <climits>
#include <mutex>

#include "tma_pipe.cuh"
#include "vi_device.cuh"

namespace tomo {

// Box rows of 80 floats: a row pitch of 16 banks modulo 32, so a warp's footprints on two
// adjacent rows fall on different banks. Rows: what NS slices and the tile's spread of
// magnification need at the usual cone angles (taller windows read global memory).
constexpr int VT_BOX_U = 80, VT_STAGES = 3;
constexpr int vt_box_v(int ns) { return ns == 16 ? 40 : ns == 8 ? 30 : 24; }
constexpr int VT_CONSUMERS = VI_BX * VI_BY;  // 256

// The detector box of view p for the tile (x0..x1, y0..y1, z0..z1): origin (u0, v0) with u0 a
// multiple of 4 (the copy's row starts on 16 bytes); false when the window exceeds the box.
// u and v are monotone in x, y and z over the tile, so its corners bound every footprint; one
// texel more on each side covers the rounding here and that of the consumers' row chain (at
// most 16 additions of values below 16384: under 0.01).
__device__ __forceinline__ bool vt_window(const DevGeom& g, int p, int x0, int x1, int y0, int y1, int z0, int z1,
                                          int box_v, int& u0, int& v0) {
    const float4 cv = __ldg(g.vi + p);
    float umin = 3.0e38f, umax = -3.0e38f, vmin = 3.0e38f, vmax = -3.0e38f;
    const float zl = (float)z0 - g.zc, zh = (float)z1 - g.zc;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const float xn = (float)((c & 1) ? x1 : x0) - g.xc, yn = (float)((c & 2) ? y1 : y0) - g.yc;
        const float w = cv.z * xn + cv.w * yn + g.fod;
        if (!(w > 0.f)) return false;
        const float a0 = 1.0f / w;
        const float ub = (cv.x * xn + cv.y * yn) * a0 + g.uc;
        const float A = a0 * g.inv_gamma_f;
        umin = fminf(umin, ub);
        umax = fmaxf(umax, ub);
        vmin = fminf(vmin, fminf(A * zl, A * zh) + g.vc);
        vmax = fmaxf(vmax, fmaxf(A * zl, A * zh) + g.vc);
    }
    const float ulo = floorf(umin) - 1.f, uhi = floorf(umax) + 2.f, vlo = floorf(vmin) - 1.f, vhi = floorf(vmax) + 2.f;
    if (!(ulo > -16384.f && uhi < 16384.f && vlo > -16384.f && vhi < 16384.f)) return false;
    u0 = (int)ulo;
    u0 -= ((u0 % 4) + 4) % 4;  // round down to a multiple of 4
    v0 = (int)vlo;
    return (int)uhi - u0 < VT_BOX_U && (int)vhi - v0 < box_v;
}

// What bounds it: at 512^3 the shared-memory reads (four words per voxel and view, 128 B a
// clock and SM) and instruction issue, both near three quarters busy. NS slices per thread:
// 16 amortise the per-column work best; 8 and 4 (the remaining slices of a 16-slice chunk
// are other blocks, which repeat the chunk's row additions up to their first slice) spread a
// small volume over the SMs (launch_vi_back_tma has the rule).
template <int UM, int NS, typename Tv, bool FDK>
__global__ void __launch_bounds__(VT_CONSUMERS + 32, FDK ? 3 : 4)
    vi_back_tma_kernel(DevGeom g, const __grid_constant__ CUtensorMap map, const float* __restrict__ sino, long pitch,
                       Tv* __restrict__ vol, float scale, unsigned* err, int stall) {
    constexpr int BOX_V = vt_box_v(NS);
    __shared__ __align__(128) float win[VT_STAGES][BOX_V * VT_BOX_U];
    __shared__ __align__(8) unsigned long long full[VT_STAGES], empty[VT_STAGES];
    // per stage: the byte address of texel (0, 0) in biased floors, and whether it is staged
    __shared__ uint2 org[VT_STAGES];
    const int tid = threadIdx.x, lane = tid & 31;
    const int x0 = blockIdx.x * VI_BX, y0 = blockIdx.y * VI_BY, z0 = blockIdx.z * NS;
    if (tid == 0) {
        for (int s = 0; s < VT_STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], VT_CONSUMERS / 32);  // one arrival per consumer warp
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (tid >= VT_CONSUMERS) {  // producer warp: each lane bounds one of 32 views, lane 0 issues the copies
        if (stall) return;      // tests only: no copy, so every wait runs out
        const int x1 = min(x0 + VI_BX, g.nx) - 1, y1 = min(y0 + VI_BY, g.ny) - 1, z1 = z0 + NS - 1;
        int issued = 0, s = 0, k = 0;
        bool alive = true;
        for (int pb = 0; pb < g.np && alive; pb += 32) {
            int u0 = 0, v0 = 0;
            const bool ok = pb + lane < g.np && vt_window(g, pb + lane, x0, x1, y0, y1, z0, z1, BOX_V, u0, v0);
            const unsigned staged = __ballot_sync(0xffffffffu, ok);
            for (int j = 0; j < min(32, g.np - pb); ++j) {
                const int uj = __shfl_sync(0xffffffffu, u0, j), vj = __shfl_sync(0xffffffffu, v0, j);
                if (k > 0 && !mbar_wait(&empty[s], (k - 1) & 1)) {
                    if (lane == 0) atomicOr(err, ERR_TIMEOUT);
                    alive = false;  // the consumers' waits run out as well
                    break;
                }
                if (lane == 0) {
                    if (staged >> j & 1) {
                        org[s] = make_uint2(smem_addr(win[s]) - (unsigned)(VI_FLOOR_KBITS + uj) * 4u -
                                                (unsigned)(VI_FLOOR_KBITS + vj) * (VT_BOX_U * 4u),
                                            1u);
                        mbar_arrive_tx(&full[s], BOX_V * VT_BOX_U * 4);
                        tma_load_3d(win[s], &map, uj, vj, pb + j, &full[s]);
                    } else {
                        org[s] = make_uint2(0u, 0u);
                        mbar_arrive(&full[s]);
                    }
                }
                __syncwarp();
                ++issued;
                if (++s == VT_STAGES) {
                    s = 0;
                    ++k;
                }
            }
        }
        // the copies in flight land before the block may exit
        for (int p = max(0, issued - VT_STAGES); p < issued; ++p)
            if (!mbar_wait(&full[p % VT_STAGES], (p / VT_STAGES) & 1) && lane == 0) atomicOr(err, ERR_TIMEOUT);
        return;
    }

    // a warp covers 8 x by 4 y columns (not 32 x 1): its footprints span about a third of the
    // detector columns a 32-wide row of voxels does, so its shared-memory reads need fewer
    // wavefronts
    const int warp = tid >> 5;
    const int x = x0 + (warp & 3) * 8 + (lane & 7), y = y0 + (warp >> 2) * 4 + (lane >> 3);
    const bool live = x < g.nx && y < g.ny;
    const float xn = fsub((float)min(x, g.nx - 1), g.xc);
    const float yn = fsub((float)min(y, g.ny - 1), g.yc);
    const float2 K = make_float2(VI_FLOOR_K, VI_FLOOR_K), MK = make_float2(-VI_FLOOR_K, -VI_FLOOR_K);
    const float2 M1 = make_float2(-1.0f, -1.0f);
    const int skip = z0 & 15;  // slices of the 16-slice chunk before the thread's first
    const float zp = fsub((float)(z0 - skip), g.zc);
    float2 acc[NS / 2];
#pragma unroll
    for (int k = 0; k < NS / 2; ++k) acc[k] = make_float2(0.f, 0.f);

    int s = 0;
    unsigned parity = 0;
    for (int p = 0; p < g.np; ++p) {
        const float4 cv = __ldg(g.vi + p);
        float A = frcp(fadd(fadd(fmul(cv.z, xn), fmul(cv.w, yn)), g.fod));                 // :401
        const float up = fmul(fadd(fmul(cv.x, xn), fmul(cv.y, yn)), A);                  // u' (:403)
        const float ub = fadd(up, g.uc);
        A = (p + g.p0 == 0 && !FDK) ? __double2float_rn(dmul(g.inv_gamma_d, (double)A))  // :404
                                    : fmul(g.inv_gamma_f, A);                           // :464
        const float mu = __fadd_rd(ub, VI_FLOOR_K);  // floor(u) + K
        const float a = fsub(ub, fsub(mu, VI_FLOOR_K));
        const unsigned iu = (unsigned)__float_as_int(mu);
        const float2 aa = make_float2(a, a);
        float vp = fmul(A, zp);                                                          // v' (:75)
        float vn = fadd(vp, g.vc);                                                       // :405
        if (!UM && NS < 16)
            for (int k = 0; k < skip; ++k) {  // the rows of the chunk's earlier slices (:410)
                vn = fadd(vn, A);
                if (FDK) vp = fadd(vp, A);
            }
        float fnum = 0.f, q0 = 0.f;
        if (FDK) {  // alphaC (FDD/du) / denum^2 and betaC + u'^2 (FDK3D_kernel_16reg.cuh:77-84)
            const float denum = fadd(fadd(fmul(fmul(xn, __ldg(g.alpha + p)), g.dx), fmul(fmul(yn, __ldg(g.beta + p)), g.dx)),
                                     g.fod);
            fnum = fdiv(fmul(g.fdk_alpha, g.fdd_du), fmul(denum, denum));
            q0 = fmaf(up, up, g.fdk_beta);
        }
        if (!mbar_wait(&full[s], parity)) {
            atomicOr(err, ERR_TIMEOUT);
            break;
        }
        const uint2 o = org[s];
        // the slices in pairs; fetch(mx, my) returns the texel pairs (t00, t10, t01, t11) of the
        // two slices whose row floors + FLOOR_K have the bit patterns mx, my
        auto run = [&](auto fetch) {
#pragma unroll
            for (int k = 0; k < NS; k += 2) {
                float2 vb;
                if (UM) {
                    const float k0 = (float)(k + (NS < 16 ? skip : 0));
                    vb = __fadd2_rn(make_float2(vn, vn), make_float2(fmul(k0, A), fmul(k0 + 1.0f, A)));
                } else {
                    vb.x = vn;
                    vn = fadd(vn, A);
                    vb.y = vn;
                    vn = fadd(vn, A);
                }
                const float2 m = __fadd2_rd(vb, K);
                const float2 f = __fadd2_rn(m, MK);
                const float2 b = __ffma2_rn(f, M1, vb);
                float2 t00, t10, t01, t11;
                fetch((unsigned)__float_as_int(m.x), (unsigned)__float_as_int(m.y), t00, t10, t01, t11);
                const float2 t = vi_bilerp2(t00, t10, t01, t11, aa, b);
                if (FDK) {
                    float2 vk;
                    vk.x = vp;
                    vp = fadd(vp, A);
                    vk.y = vp;
                    vp = fadd(vp, A);
                    const float2 q = __ffma2_rn(vk, vk, make_float2(q0, q0));
                    acc[k >> 1] = __ffma2_rn(make_float2(fmul(fnum, rsqrtf(q.x)), fmul(fnum, rsqrtf(q.y))), t, acc[k >> 1]);
                } else {
                    acc[k >> 1] = __fadd2_rn(acc[k >> 1], t);
                }
            }
        };
        if (o.y) {
            const unsigned rb = o.x + iu * 4u;
            run([&](unsigned mx, unsigned my, float2& t00, float2& t10, float2& t01, float2& t11) {
                const unsigned i0 = rb + mx * (VT_BOX_U * 4u), i1 = rb + my * (VT_BOX_U * 4u);
                t00 = make_float2(lds_f32<0>(i0), lds_f32<0>(i1));
                t10 = make_float2(lds_f32<4>(i0), lds_f32<4>(i1));
                t01 = make_float2(lds_f32<VT_BOX_U * 4>(i0), lds_f32<VT_BOX_U * 4>(i1));
                t11 = make_float2(lds_f32<VT_BOX_U * 4 + 4>(i0), lds_f32<VT_BOX_U * 4 + 4>(i1));
            });
        } else if (ub > -1.f && ub < (float)g.nu) {  // from global memory, zero off the detector
            const int ui = (int)iu - VI_FLOOR_KBITS;
            const float* sg = sino + (p * (long)g.nv) * pitch + ui;  // column ui of view p
            const bool c0 = ui >= 0, c1 = ui + 1 < g.nu;
            run([&](unsigned mx, unsigned my, float2& t00, float2& t10, float2& t01, float2& t11) {
                const int r0 = (int)mx - VI_FLOOR_KBITS, r1 = (int)my - VI_FLOOR_KBITS;
                const bool a0r = r0 >= 0 && r0 < g.nv, a1r = r0 + 1 >= 0 && r0 + 1 < g.nv;
                const bool b0r = r1 >= 0 && r1 < g.nv, b1r = r1 + 1 >= 0 && r1 + 1 < g.nv;
                const float* q0 = sg + (long)r0 * pitch;
                const float* q1 = sg + (long)r1 * pitch;
                t00 = make_float2(c0 && a0r ? __ldg(q0) : 0.f, c0 && b0r ? __ldg(q1) : 0.f);
                t10 = make_float2(c1 && a0r ? __ldg(q0 + 1) : 0.f, c1 && b0r ? __ldg(q1 + 1) : 0.f);
                t01 = make_float2(c0 && a1r ? __ldg(q0 + pitch) : 0.f, c0 && b1r ? __ldg(q1 + pitch) : 0.f);
                t11 = make_float2(c1 && a1r ? __ldg(q0 + pitch + 1) : 0.f, c1 && b1r ? __ldg(q1 + pitch + 1) : 0.f);
            });
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
        if (++s == VT_STAGES) {
            s = 0;
            parity ^= 1u;
        }
    }
    if (!live) return;
    const long plane = (long)g.nx * g.ny;
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        const int z = z0 + k;
        const float r = (k & 1) ? acc[k >> 1].y : acc[k >> 1].x;
        if (z < g.nz) vol[z * plane + (long)y * g.nx + x] = cvt<Tv>(FDK ? fmul(r, scale) : fmul(fmul(r, g.dx), scale));
    }
}

// ---------------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------------
EncodeTiledFn tma_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
        cudaGetLastError();
    });
    return fn;
}

namespace {

// Slices per thread. A thread's fixed work per view is about that of four slices, so 16 are
// fastest wherever their blocks fill the chip; below that, more and smaller blocks win
// (64^3, 60 views: 64 blocks of 16 slices, 256 of 4).
int vt_slices(const DevGeom& g) {
    const long cols = (long)((g.nx + VI_BX - 1) / VI_BX) * ((g.ny + VI_BY - 1) / VI_BY);
    if (cols * ((g.nz + 15) / 16) >= 148 * 4) return 16;
    return cols * ((g.nz + 7) / 8) >= 148 * 4 ? 8 : 4;
}

struct TmaCall {
    const DevGeom& g;
    const CUtensorMap& map;
    const float* sino;
    long pitch;
    void* vol;
    float scale;
    unsigned* err;
    cudaStream_t st;
    int stall;
};

template <int UM, int NS, typename Tv, bool FDK>
cudaError_t launch_tma_k(const TmaCall& c) {
    const DevGeom& g = c.g;
    const dim3 block(VT_CONSUMERS + 32), grid((g.nx + VI_BX - 1) / VI_BX, (g.ny + VI_BY - 1) / VI_BY, (g.nz + NS - 1) / NS);
    vi_back_tma_kernel<UM, NS, Tv, FDK><<<grid, block, 0, c.st>>>(g, c.map, c.sino, c.pitch, (Tv*)c.vol, c.scale, c.err,
                                                                  c.stall);
    return cudaGetLastError();
}

template <int UM, typename Tv, bool FDK>
cudaError_t launch_tma_n(const TmaCall& c, int ns) {
    return ns == 16 ? launch_tma_k<UM, 16, Tv, FDK>(c) : ns == 8 ? launch_tma_k<UM, 8, Tv, FDK>(c) : launch_tma_k<UM, 4, Tv, FDK>(c);
}

template <typename Tv>
cudaError_t launch_tma_v(const TmaCall& c, int kind, int ns) {
    return kind == 2 ? launch_tma_n<0, Tv, true>(c, ns) : kind == 1 ? launch_tma_n<1, Tv, false>(c, ns)
                                                                   : launch_tma_n<0, Tv, false>(c, ns);
}

// A sinogram of any type into FP32 rows of `pitch` words (a multiple of 4).
template <typename T>
__global__ void sino_rows_kernel(const T* __restrict__ in, float* __restrict__ out, int nu, long rows, int pitch) {
    const long total = rows * nu;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
        const long r = i / nu;
        out[r * pitch + (i - r * nu)] = ldp(in + i);
    }
}

}  // namespace

cudaError_t launch_sino_rows(const void* in, tomo_dtype idt, float* out, int nu, int nv, int np, int pitch, cudaStream_t st) {
    const long rows = (long)nv * np, n = rows * nu;
    const int b = (int)(n + 255 < 148L * 32 * 256 ? (n + 255) / 256 : 148L * 32);
    switch (idt) {
        case TOMO_F32: sino_rows_kernel<<<b, 256, 0, st>>>((const float*)in, out, nu, rows, pitch); break;
        case TOMO_BF16: sino_rows_kernel<<<b, 256, 0, st>>>((const __nv_bfloat16*)in, out, nu, rows, pitch); break;
        case TOMO_F16: sino_rows_kernel<<<b, 256, 0, st>>>((const __half*)in, out, nu, rows, pitch); break;
    }
    return cudaGetLastError();
}

bool vi_tma_supported(const void* sino, long pitch) {
    return tma_encode_fn() != nullptr && pitch % 4 == 0 && ((uintptr_t)sino & 15) == 0;
}

cudaError_t launch_vi_back_tma(int kind, const DevGeom& g, const float* sino, long pitch, void* vol, tomo_dtype vdt,
                               float scale, unsigned* err, cudaStream_t st, int stall) {
    if (!vi_tma_supported(sino, pitch)) return cudaErrorNotSupported;
    const int ns = vt_slices(g);
    CUtensorMap map;
    const cuuint64_t dims[3] = {(cuuint64_t)g.nu, (cuuint64_t)g.nv, (cuuint64_t)g.np};
    const cuuint64_t strides[2] = {(cuuint64_t)pitch * 4, (cuuint64_t)pitch * g.nv * 4};
    const cuuint32_t box[3] = {VT_BOX_U, (cuuint32_t)vt_box_v(ns), 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    if (tma_encode_fn()(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(sino), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorInvalidValue;
    const TmaCall c{g, map, sino, pitch, vol, scale, err, st, stall};
    switch (vdt) {
        case TOMO_F32: return launch_tma_v<float>(c, kind, ns);
        case TOMO_BF16: return launch_tma_v<__nv_bfloat16>(c, kind, ns);
        case TOMO_F16: return launch_tma_v<__half>(c, kind, ns);
    }
    return cudaErrorInvalidValue;
}

}  // namespace tomo
