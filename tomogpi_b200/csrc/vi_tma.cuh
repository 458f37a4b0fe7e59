// vi_tma.cuh -- device code of the TMA-staged VI backprojector (see vi_tma.cu), shared by the
// single-job kernel and the batched persistent kernel (batch.cu).
#pragma once

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

// The tensor map of a sinogram [P][nv][pitch] for NS slices per thread.
bool vi_tma_encode(const float* sino, int nu, int nv, int np, long pitch, int ns, CUtensorMap* map);

// Shared memory of a block.
template <int NS>
struct VtShared {
    __align__(128) float win[VT_STAGES][vt_box_v(NS) * VT_BOX_U];
    unsigned long long full[VT_STAGES], empty[VT_STAGES];
    // per stage: the byte address of texel (0, 0) in biased floors, and whether it is staged
    uint2 org[VT_STAGES];
};

// The stage a thread comes to next, carried from tile to tile.
struct VtTurn {
    int s = 0;
    unsigned phase = 0;
    __device__ __forceinline__ void next() {
        if (++s == VT_STAGES) {
            s = 0;
            phase ^= 1u;
        }
    }
};

// Once per block, before the first tile; a __syncthreads() follows.
template <int NS>
__device__ __forceinline__ void vt_init(VtShared<NS>& sh) {
    if (threadIdx.x == 0) {
        for (int s = 0; s < VT_STAGES; ++s) {
            mbar_init(&sh.full[s], 1);
            mbar_init(&sh.empty[s], VT_CONSUMERS / 32);  // one arrival per consumer warp
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
}

// What bounds it: at 512^3 the shared-memory reads (four words per voxel and view, 128 B a
// clock and SM) and instruction issue, both near three quarters busy. NS slices per thread:
// 16 amortise the per-column work best; 8 and 4 (the remaining slices of a 16-slice chunk
// are other blocks, which repeat the chunk's row additions up to their first slice) spread a
// small volume over the SMs (launch_vi_back_tma has the rule).
// All VT_CONSUMERS + 32 threads call it; false: a wait ran out (ERR_TIMEOUT is set), the block
// must stop.
template <int UM, int NS, typename Tv, bool FDK>
__device__ __forceinline__ bool vi_tma_tile(const DevGeom& g, const CUtensorMap* map, const float* __restrict__ sino,
                                            long pitch, Tv* __restrict__ vol, float scale, unsigned* err, int stall,
                                            VtShared<NS>& sh, VtTurn& turn, int xt, int yt, int zt) {
    constexpr int BOX_V = vt_box_v(NS);
    const int tid = threadIdx.x, lane = tid & 31;
    const int x0 = xt * VI_BX, y0 = yt * VI_BY, z0 = zt * NS;
    if (tid >= VT_CONSUMERS) {  // producer warp: each lane bounds one of 32 views, lane 0 issues the copies
        if (stall) return true;  // tests only: no copy, so every consumer wait runs out
        const int x1 = min(x0 + VI_BX, g.nx) - 1, y1 = min(y0 + VI_BY, g.ny) - 1, z1 = z0 + NS - 1;
        int issued = 0;
        bool alive = true;
        const VtTurn first = turn;
        for (int pb = 0; pb < g.np && alive; pb += 32) {
            int u0 = 0, v0 = 0;
            const bool ok = pb + lane < g.np && vt_window(g, pb + lane, x0, x1, y0, y1, z0, z1, BOX_V, u0, v0);
            const unsigned staged = __ballot_sync(0xffffffffu, ok);
            for (int j = 0; j < min(32, g.np - pb); ++j) {
                const int uj = __shfl_sync(0xffffffffu, u0, j), vj = __shfl_sync(0xffffffffu, v0, j);
                const int s = turn.s;
                if (!mbar_wait_warp(&sh.empty[s], turn.phase ^ 1u)) {  // a fresh barrier counts as emptied
                    if (lane == 0) atomicOr(err, ERR_TIMEOUT);
                    alive = false;  // the consumers' waits run out as well
                    break;
                }
                if (lane == 0) {
                    if (staged >> j & 1) {
                        sh.org[s] = make_uint2(smem_addr(sh.win[s]) - (unsigned)(VI_FLOOR_KBITS + uj) * 4u -
                                                   (unsigned)(VI_FLOOR_KBITS + vj) * (VT_BOX_U * 4u),
                                               1u);
                        mbar_arrive_tx(&sh.full[s], BOX_V * VT_BOX_U * 4);
                        tma_load_3d(sh.win[s], map, uj, vj, pb + j, &sh.full[s]);
                    } else {
                        sh.org[s] = make_uint2(0u, 0u);
                        mbar_arrive(&sh.full[s]);
                    }
                }
                __syncwarp();
                ++issued;
                turn.next();
            }
        }
        // the copies in flight land before the block may exit
        VtTurn q = first;
        for (int p = 0; p < issued; ++p, q.next())
            if (p >= issued - VT_STAGES && !mbar_wait_warp(&sh.full[q.s], q.phase)) {
                if (lane == 0) atomicOr(err, ERR_TIMEOUT);
                alive = false;
            }
        return alive;
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

    bool alive = true;
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
        float vn = fadd(fmul(A, zp), g.vc);                                              // v' (:75), v (:405)
        if (!UM && NS < 16)
            for (int k = 0; k < skip; ++k) {  // the rows of the chunk's earlier slices (:410)
                vn = fadd(vn, A);
            }
        const float2 fdk = FDK ? fdk_column(g, xn, yn, up, p) : make_float2(0.f, 0.f);
        if (!mbar_wait_warp(&sh.full[turn.s], turn.phase)) {
            if (lane == 0) atomicOr(err, ERR_TIMEOUT);
            alive = false;
            break;
        }
        const uint2 o = sh.org[turn.s];
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
                if (FDK) {  // fdk_weight of the two slices
                    const float2 vk = __fadd2_rn(vb, make_float2(-g.vc, -g.vc));
                    const float2 q = __ffma2_rn(vk, vk, make_float2(fdk.y, fdk.y));
                    const float2 w = __fmul2_rn(make_float2(fdk.x, fdk.x), make_float2(vi_rsqrt(q.x), vi_rsqrt(q.y)));
                    acc[k >> 1] = __ffma2_rn(w, t, acc[k >> 1]);
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
        if (lane == 0) mbar_arrive(&sh.empty[turn.s]);
        turn.next();
    }
    if (!live) return alive;
    const long plane = (long)g.nx * g.ny;
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        const int z = z0 + k;
        const float r = (k & 1) ? acc[k >> 1].y : acc[k >> 1].x;
        if (z < g.nz) vol[z * plane + (long)y * g.nx + x] = cvt<Tv>(FDK ? fmul(r, scale) : fmul(fmul(r, g.dx), scale));
    }
    return alive;
}

}  // namespace tomo
