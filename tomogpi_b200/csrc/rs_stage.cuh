// rs_stage.cuh -- device code of the STAGE form of the regular-sampling projector: the part
// of the volume that a block's rays cross is brought into shared memory by the Tensor
// Memory Accelerator (TMA), a few planes at a time, while the rays march through it.
//
// What bounds the other layouts is the L1TEX unit: a texture gather returns 32 B a clock and
// SM, so each of a TEX sample's two gathers (one for 16-bit slice pairs) takes it 16 clocks
// per warp, whatever the cache hit rate. Shared memory returns 128 B a clock: an FP32
// sample's eight 32-bit reads take 14.7 clocks per warp with their bank conflicts (the 32
// lanes' texels lie in a patch of about 40 words, so two lanes of some bank usually differ).
// Neighbouring rays share texels: about 3 words are copied in per sample. FP32, 256^3, 256
// views: TEX 13.7 ms, HYBRID 8.4, STAGE 7.18, with the shared-memory reads at 87% of their
// rate; 512^3: TEX 218 ms, HYBRID 133, STAGE 109. 16-bit volumes read four words of slice pairs
// per sample and are bound by issue (60 instructions per sample at 85%), no faster than the
// texture alone; together they are (RSG_SHARE16).
//
// A block is one detector tile of one view (256 rays) plus a producer warp. The rays march
// across the planes of the axis (x or y) that the tile's central ray runs along. The volume
// exists in two copies, [z][y][x] and [z][x][y], so that the other in-plane axis t is
// contiguous in either. The producer cuts the march into chunks of C planes: it bounds the
// (t, z) window of the tile's four corner rays over the chunk (t and z are linear in the
// march coordinate and monotone in u and v, so the corners give the extremes), takes the
// largest C whose C + 2 planes of the window fit a stage, and issues one
// cp.async.bulk.tensor per plane (no multicast; this GPU's own buffer; texels off the volume
// come back as the copy's zero fill, which is the reference's texture border). The window's
// width W is one of a few values that put the four rows (z) of a warp's 8 u x 4 v rays on
// different banks (256^3: {24, 40, 56, 72, 88} takes 1.5% longer, {36, 44, 52, 68, 84} 7%). The rays of a block stay within a
// chunk of each other, so a plane is staged once per block.
//
// A ray's samples are the repeated additions and the arithmetic of rs_device.cuh whatever
// the chunking: bit-identical to the other layouts. A ray is staged when its line lies
// between the corner rays at both of its ends (then it does at every plane: all lines go
// through the source) and it runs along the march axis; the windows are padded by what its
// repeated additions can drift, so every footprint of a staged ray lies in its chunk's
// window (tests/test_rs_stage_window.py checks this in FP32). Other rays, and chunks whose
// window fits no stage, read global memory with bounds tests.
#pragma once

#include <climits>

#include "rs_device.cuh"
#include "tma_pipe.cuh"

namespace tomo {

constexpr int RSG_THREADS = 256 + 32;  // consumers (one ray each), producer warp
constexpr int RSG_STAGES = 2;
// Words of a stage: four blocks of two 27 KB stages per SM (256^3, 256 views, blocks x words
// against 4 x 6912: 2 x 12288 12% longer, 3 x 8192 1%, 5 x 5440 5%, 6 x 4608 19%: more blocks
// hide the waits at chunk ends, shorter chunks stage their two shared planes more often).
constexpr int RSG_CAP = 6912, RSG_MIN_BLOCKS = 4;
// Sixteenths of the blocks that gather from the packed texture instead (16-bit volumes): the
// gathers are bound by the texture's return path, staged samples by instruction issue, so
// blocks of both kinds on an SM overlap. 384^3, 384 views, BF16: all gathered 34.7 ms, 12
// sixteenths 31.6, 10 31.0, 8 31.3, none 34.6. FP32 volumes take none (2 sixteenths would gain
// 1.5% for a texture beside the copies).
constexpr int RSG_SHARE16 = 10;
constexpr int RSG_CMAX = 30;            // planes of a chunk + 2 <= 32 lanes of the producer
constexpr int RSG_WIDTHS = 5, RSG_HEIGHTS = 8;
__host__ __device__ __forceinline__ int rsg_width(int i) { return i < 2 ? 24 + 16 * i : 20 + 16 * i; }  // 24, 40, 52, 68, 84
__host__ __device__ __forceinline__ int rsg_height(int j) { return j < 5 ? 8 + 2 * j : j < 7 ? 4 * j : 32; }  // 8..16, 20, 24, 32

// Slices of a copy: FP32 one word per voxel, slices 0 .. nz - 1; 16-bit storage one word per
// slice pair (k, k + 1), low and high half, k = -1 .. nz - 1.
template <typename Tv>
__host__ __device__ __forceinline__ int rsg_slices(int nz) { return sizeof(Tv) == 4 ? nz : nz + 1; }

// The copies' tensor maps, a kernel parameter (10 KB): maps in device memory would need a
// proxy fence per block, since a freed copy's maps may have been at the same address.
struct RsStageMaps {
    CUtensorMap m[2][RSG_WIDTHS][RSG_HEIGHTS];  // [axis: 0 = y-march, 1 = x-march]
};

struct RsStageSrc {              // what the kernel reads beside them
    const unsigned* rows;        // the [z][y][x] copy
    int px;                      // its row pitch in words
    unsigned long long tex;      // the packed texture (16-bit volumes)
    int share;                   // sixteenths of the blocks that gather from it (RSG_SHARE16)
};

struct __align__(16) RsChunk {
    unsigned bias;               // byte address of texel (0, 0, 0) in biased floors, modulo 2^32
    unsigned pp;                 // bytes of a plane in the stage
    float edge;                  // the chunk's samples lie below it (march up) or from it on (march down)
    int w_last;                  // window width (0: not staged), + RSG_LAST for the block's last chunk
};
constexpr int RSG_LAST = 1 << 16;

struct RsStageShared {
    unsigned long long full[RSG_STAGES], empty[RSG_STAGES];
    RsChunk chunk[RSG_STAGES];
    int lo, hi;                  // plane floors of the block's samples
    float st[2], sz[2];          // range of the corner rays' slopes: t and z per plane
    int along;                   // the corner rays run along the march axis
};
constexpr int RSG_HEADER = 512;  // bytes before the stages
static_assert(sizeof(RsStageShared) <= RSG_HEADER, "the stages start after the header");
constexpr int RSG_SMEM = RSG_HEADER + RSG_STAGES * RSG_CAP * 4;

// Once per block, before the first tile; a __syncthreads() follows.
__device__ __forceinline__ void rsg_init(RsStageShared* sh) {
    if (threadIdx.x == 0) {
        for (int s = 0; s < RSG_STAGES; ++s) {
            mbar_init(&sh->full[s], 1);
            mbar_init(&sh->empty[s], 8);  // one arrival per consumer warp
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
}

// The texels of a sample whose (m, t, z) is at address a, pp = bytes of a plane: the slices
// lo and up in tld4 order, (i, j+1), (i+1, j+1), (i+1, j), (i, j).
template <typename Tv, int W, bool XM>
__device__ __forceinline__ void rsg_texels(unsigned a, unsigned pp, float4& lo, float4& up) {
    const unsigned b = a + pp;
    if constexpr (sizeof(Tv) == 4) {
        lo.w = lds_f32<0>(a);
        up.w = lds_f32<W * 4>(a);
        const float lt = lds_f32<4>(a), ut = lds_f32<W * 4 + 4>(a);
        const float lm = lds_f32<0>(b), um = lds_f32<W * 4>(b);
        lo.y = lds_f32<4>(b);
        up.y = lds_f32<W * 4 + 4>(b);
        lo.x = XM ? lt : lm;  // t is y for an x-march
        lo.z = XM ? lm : lt;
        up.x = XM ? ut : um;
        up.z = XM ? um : ut;
    } else {
        auto word = [](float f) { return __float_as_uint(f); };
        unpack_pair(word(lds_f32<0>(a)), lo.w, up.w, (Tv*)nullptr);
        const unsigned wt = word(lds_f32<4>(a)), wm = word(lds_f32<0>(b));
        unpack_pair(word(lds_f32<4>(b)), lo.y, up.y, (Tv*)nullptr);
        unpack_pair(XM ? wt : wm, lo.x, up.x, (Tv*)nullptr);
        unpack_pair(XM ? wm : wt, lo.z, up.z, (Tv*)nullptr);
    }
}

// One sample from global memory (the [z][y][x] copy), zero outside the volume.
template <typename Tv>
__device__ __forceinline__ float rsg_global(const RsStageSrc& sv, int nx, int ny, int nz, const RsSample& s) {
    if (!rs_inside(s, (float)nx, (float)ny, (float)nz)) return 0.f;
    const int i = s.ix - FLOOR_KBITS, j = s.iy - FLOOR_KBITS, k = s.iz - FLOOR_KBITS;
    auto word = [&](int x, int y, int z) {
        return x >= 0 && y >= 0 && z >= 0 && x < nx && y < ny && z < rsg_slices<Tv>(nz)
                   ? __ldg(sv.rows + ((long)z * ny + y) * sv.px + x)
                   : 0u;
    };
    float4 lo, up;
    if constexpr (sizeof(Tv) == 4) {
        auto texel = [&](int x, int y, int z) { return __uint_as_float(word(x, y, z)); };
        lo = make_float4(texel(i, j + 1, k), texel(i + 1, j + 1, k), texel(i + 1, j, k), texel(i, j, k));
        up = make_float4(texel(i, j + 1, k + 1), texel(i + 1, j + 1, k + 1), texel(i + 1, j, k + 1), texel(i, j, k + 1));
    } else {
        unpack_pair(word(i, j + 1, k + 1), lo.x, up.x, (Tv*)nullptr);
        unpack_pair(word(i + 1, j + 1, k + 1), lo.y, up.y, (Tv*)nullptr);
        unpack_pair(word(i + 1, j, k + 1), lo.z, up.z, (Tv*)nullptr);
        unpack_pair(word(i, j, k + 1), lo.w, up.w, (Tv*)nullptr);
    }
    return trilerp(lo, up, s);
}

// The source in voxel coordinates along and across the march: the rays are the lines
// t = ts + (m - ms) slope_t, z = zc + (m - ms) slope_z.
__device__ __forceinline__ float2 rsg_source(const DevGeom& g, bool xm, float al, float be) {
    const float inv_dx = 1.0f / g.dx;
    const float xs = g.xc - g.fod * al * inv_dx, ys = g.yc - g.fod * be * inv_dx;
    return xm ? make_float2(xs, ys) : make_float2(ys, xs);
}

// What a ray's repeated additions (at most 3 nmax of them, each within half an ulp of a value
// below nmax + 2) can drift off its line, plus 0.1.
__device__ __forceinline__ float rsg_pad(const DevGeom& g) {
    const float m = (float)max(max(g.nx, g.ny), g.nz) + 2.0f;
    return 0.1f + 3.0f * m * m * 2.98023224e-8f;
}

// The slopes of the tile's corner rays (one thread).
__device__ __forceinline__ void rsg_corners(const DevGeom& g, RsStageShared* sh, bool xm, bool upward, float al, float be,
                                            int u0, int u1, int v0, int v1) {
    float st[2], sz[4];
    bool along = true;
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        const float uu = ((float)(a ? u1 : u0) - g.uc) * g.du;
        const float dxr = al * g.fdd - uu * be, dyr = be * g.fdd + uu * al;
        const float dm = xm ? dxr : dyr;
        along &= (upward ? dm : -dm) > 0.25f * g.fdd;
        st[a] = (xm ? dyr : dxr) / dm;
        sz[2 * a] = ((float)v0 - g.vc) * g.dv / dm;
        sz[2 * a + 1] = ((float)v1 - g.vc) * g.dv / dm;
    }
    sh->st[0] = fminf(st[0], st[1]);
    sh->st[1] = fmaxf(st[0], st[1]);
    sh->sz[0] = fminf(fminf(sz[0], sz[1]), fminf(sz[2], sz[3]));
    sh->sz[1] = fmaxf(fmaxf(sz[0], sz[1]), fmaxf(sz[2], sz[3]));
    sh->along = along;
}

// The producer warp: chunks from plane floor `lo` to `hi` (marching up) or from `hi` down.
template <typename Tv>
__device__ __forceinline__ void rsg_produce(const DevGeom& g, const RsStageMaps& maps, float* stages, RsStageShared* sh,
                                            unsigned& turn, bool xm, bool upward, float2 src, int lo, int hi,
                                            unsigned* err, int stall) {
    if (stall) return;  // tests only: no copy, so every consumer wait runs out
    const int lane = threadIdx.x & 31;
    const float st0 = sh->st[0], st1 = sh->st[1], sz0 = sh->sz[0], sz1 = sh->sz[1], pad = rsg_pad(g);
    const bool along = sh->along;
    int cur = upward ? lo : hi;
    const unsigned first = turn;
    while (upward ? cur <= hi : cur >= lo) {
        const int left = upward ? hi - cur + 1 : cur - lo + 1;
        // lane c tries a chunk of c + 1 planes
        const int C = min(lane + 1, left);
        const int ma = upward ? cur : cur - C + 1;
        const float e0 = (float)ma - 0.15f - src.x, e1 = (float)(ma + C) + 0.15f - src.x;
        const float tl = floorf(src.y + fminf(fminf(e0 * st0, e1 * st0), fminf(e0 * st1, e1 * st1)) - pad);
        const float th = floorf(src.y + fmaxf(fmaxf(e0 * st0, e1 * st0), fmaxf(e0 * st1, e1 * st1)) + pad);
        const float zl = floorf(g.zc + fminf(fminf(e0 * sz0, e1 * sz0), fminf(e0 * sz1, e1 * sz1)) - pad);
        const float zh = floorf(g.zc + fmaxf(fmaxf(e0 * sz0, e1 * sz0), fmaxf(e0 * sz1, e1 * sz1)) + pad);
        const bool sane = along && fabsf(tl) < 1.0e6f && fabsf(th) < 1.0e6f && fabsf(zl) < 1.0e6f && fabsf(zh) < 1.0e6f;
        const int t0 = sane ? (int)tl & ~3 : 0;  // the copy's rows start on 16 bytes
        const int z0 = sane ? (int)zl : 0;
        const int wn = sane ? (int)th + 2 - t0 : 1 << 20;
        const int hn = sane ? (int)zh + (sizeof(Tv) == 4 ? 2 : 1) - z0 : 1 << 20;
        int wi = 0, hj = 0;
        while (wi < RSG_WIDTHS && rsg_width(wi) < wn) ++wi;
        while (hj < RSG_HEIGHTS && rsg_height(hj) < hn) ++hj;
        const int wh = rsg_width(wi) * rsg_height(hj), pp = (wh + 31) & ~31;  // planes start on 128 bytes
        const bool fits = wi < RSG_WIDTHS && hj < RSG_HEIGHTS && lane < RSG_CMAX && lane < left && (C + 2) * pp <= RSG_CAP;
        const unsigned ok = __ballot_sync(0xffffffffu, fits);
        const int s = turn % RSG_STAGES;
        const unsigned k = turn / RSG_STAGES;
        if (k > 0 && !mbar_wait_warp(&sh->empty[s], (k - 1) & 1)) {
            if (lane == 0) atomicOr(err, ERR_TIMEOUT);
            break;  // the consumers' waits run out as well
        }
        const int best = ok ? 31 - __clz(ok) : min(8, left) - 1;  // not staged: eight planes from global memory
        const int n = best + 1;
        const int mb = upward ? cur : cur - n + 1, plane0 = upward ? mb - 1 : mb;
        const int bt = __shfl_sync(0xffffffffu, t0, best), bz = __shfl_sync(0xffffffffu, z0, best);
        const int bw = __shfl_sync(0xffffffffu, wi, best), bh = __shfl_sync(0xffffffffu, hj, best);
        const int bpp = __shfl_sync(0xffffffffu, pp, best), words = __shfl_sync(0xffffffffu, wh, best);
        cur += upward ? n : -n;
        if (lane == 0) {
            const int w = ok ? rsg_width(bw) : 0;
            RsChunk ch;
            ch.pp = (unsigned)bpp * 4u;
            ch.bias = smem_addr(stages + s * RSG_CAP) -
                      ((unsigned)(plane0 + FLOOR_KBITS) * ch.pp + (unsigned)(bz + FLOOR_KBITS) * (unsigned)(w * 4) +
                       (unsigned)(bt + FLOOR_KBITS) * 4u);
            ch.edge = (float)(upward ? mb + n : mb);
            ch.w_last = w + ((upward ? cur <= hi : cur >= lo) ? 0 : RSG_LAST);
            sh->chunk[s] = ch;
            if (ok) mbar_arrive_tx(&sh->full[s], (unsigned)((n + 2) * words) * 4u);
            else mbar_arrive(&sh->full[s]);
        }
        __syncwarp();
        if (ok && lane < n + 2)
            tma_load_3d(stages + s * RSG_CAP + lane * bpp, &maps.m[xm][bw][bh], bt, bz + (sizeof(Tv) == 4 ? 0 : 1),
                        plane0 + lane, &sh->full[s]);
        ++turn;
    }
    // the copies in flight land before the block may exit
    for (unsigned q = turn - first < RSG_STAGES ? first : turn - RSG_STAGES; q != turn; ++q)
        if (!mbar_wait_warp(&sh->full[q % RSG_STAGES], (q / RSG_STAGES) & 1) && lane == 0) atomicOr(err, ERR_TIMEOUT);
}

// One tile of view p (as rs_tile; all RSG_THREADS threads call it). turn: the block's count
// of chunks, carried from tile to tile.
template <int MODE, typename Tv, typename To, int EPI, typename Tr = To>
__device__ __forceinline__ void rs_stage_tile(const DevGeom& g, const RsStageMaps& maps, const RsStageSrc& sv,
                                              unsigned char* smem, unsigned& turn, const OutView<To>& out, const OutView<Tr>& real,
                                              double* __restrict__ norm, int p, int ut, int vt, unsigned* err, int stall) {
    RsStageShared* sh = reinterpret_cast<RsStageShared*>(smem);
    float* stages = reinterpret_cast<float*>(smem + RSG_HEADER);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float al = __ldg(g.alpha + p), be = __ldg(g.beta + p);
    const int u0 = ut << g.rs_tlog, u1 = min(u0 + rs_tile_u(g), g.nu) - 1;
    const int v0 = vt * rs_tile_v(g), v1 = min(v0 + rs_tile_v(g), g.nv) - 1;
    // the axis and the sense in which the tile's central ray runs
    const float cu = (0.5f * (float)(u0 + u1) - g.uc) * g.du;
    const float cx = al * g.fdd - cu * be, cy = be * g.fdd + cu * al;
    const bool xm = fabsf(cx) >= fabsf(cy), upward = (xm ? cx : cy) > 0.f;
    if (threadIdx.x == RSG_THREADS - 32) {
        sh->lo = INT_MAX;
        sh->hi = INT_MIN;
        rsg_corners(g, sh, xm, upward, al, be, u0, u1, v0, v1);
    }
    __syncthreads();
    const float2 src = rsg_source(g, xm, al, be);
    const int wl = g.rs_wlog, wu = 1 << wl, wpr = 1 << (g.rs_tlog - wl);
    const int u = u0 + (warp & (wpr - 1)) * wu + (lane & (wu - 1));
    const int v = v0 + (warp >> (g.rs_tlog - wl)) * (32 >> wl) + (lane >> wl);
    const bool active = warp < 8 && u < g.nu && v < g.nv;
    RsRay r;
    r.n = 0;
    float inv_s = 0.f;  // steps per plane; 0: not staged
    if (warp < 8) {
        int lo = INT_MAX, hi = INT_MIN;
        if (active) {
            const bool hit = MODE == 0 ? rs_ray_box(g, u, v, al, be, r) : rs_ray_um(g, u, v, al, be, r);
            if (!hit) r.n = 0;
            if (r.n) {
                const float len = (float)(r.n - 1), top = (float)(xm ? g.nx : g.ny);
                const float sm = xm ? r.sx : r.sy, m0 = xm ? r.A : r.B, m1 = fmaf(len, sm, m0);
                const float t0 = xm ? r.B : r.A, t1 = fmaf(len, xm ? r.sy : r.sx, t0), z1 = fmaf(len, r.sz, r.C);
                // the line between the corner rays (+- 0.05) at both ends
                auto between = [&](float e, float t, float z) {
                    const float a = e * sh->st[0], b = e * sh->st[1], c = e * sh->sz[0], d = e * sh->sz[1];
                    return t >= src.y + fminf(a, b) - 0.05f && t <= src.y + fmaxf(a, b) + 0.05f &&
                           z >= g.zc + fminf(c, d) - 0.05f && z <= g.zc + fmaxf(c, d) + 0.05f;
                };
                if (sh->along && (upward ? sm : -sm) > 0.25f && fminf(m0, m1) >= -1.5f && fmaxf(m0, m1) <= top + 0.5f &&
                    between(m0 - src.x, t0, r.C) && between(m1 - src.x, t1, z1)) {
                    inv_s = 1.0f / fabsf(sm);
                    lo = (int)floorf(fminf(m0, m1) - 0.15f);
                    hi = (int)floorf(fmaxf(m0, m1) + 0.15f);
                }
            }
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if (lane == 0 && lo <= hi) {
            atomicMin(&sh->lo, lo);
            atomicMax(&sh->hi, hi);
        }
    }
    __syncthreads();
    const int lo = sh->lo, hi = sh->hi;
    float acc = 0.f;
    if (warp >= 8) {
        rsg_produce<Tv>(g, maps, stages, sh, turn, xm, upward, src, lo, hi, err, stall);
    } else {
        const float dx = g.dx;
        const float2 SXY = make_float2(r.sx, r.sy);
        float2 AB = make_float2(r.A, r.B);
        float C = r.C;
        int rem = (int)r.n;
        auto march = [&](int cnt, auto sample) {
            for (; cnt > 0; --cnt) {
                const RsSample sp = rs_sample(AB, C);
                acc = fadd(acc, fmul(dx, sample(sp)));  // :292
                AB = __fadd2_rn(AB, SXY);              // :295-297
                C = fadd(C, r.sz);
            }
        };
        auto global = [&](const RsSample& sp) { return rsg_global<Tv>(sv, g.nx, g.ny, g.nz, sp); };
        auto chunks = [&](auto axis) {
            constexpr bool XM = decltype(axis)::value;
            for (bool more = lo <= hi; more;) {
                const int s = turn % RSG_STAGES;
                if (!mbar_wait_warp(&sh->full[s], (turn / RSG_STAGES) & 1)) {
                    if (lane == 0) atomicOr(err, ERR_TIMEOUT);
                    break;
                }
                const RsChunk ch = sh->chunk[s];
                // samples before the chunk's edge; one within 0.1 of it waits for the next chunk,
                // whose planes start one earlier
                const float m = XM ? AB.x : AB.y;
                const float dist = (upward ? ch.edge - m : m - ch.edge) - 0.1f;
                const int cnt = dist > 0.f && inv_s > 0.f ? min(rem, (int)(dist * inv_s) + 1) : 0;
                rem -= cnt;
                auto staged = [&](auto width) {
                    constexpr int W = decltype(width)::value;
                    march(cnt, [&](const RsSample& sp) {
                        const unsigned a = (unsigned)(XM ? sp.ix : sp.iy) * ch.pp +
                                           ((unsigned)sp.iz * (W * 4u) + ((unsigned)(XM ? sp.iy : sp.ix) * 4u + ch.bias));
                        float4 lo, up;
                        rsg_texels<Tv, W, XM>(a, ch.pp, lo, up);
                        return trilerp(lo, up, sp);
                    });
                };
                switch (ch.w_last & (RSG_LAST - 1)) {
                    case 24: staged(std::integral_constant<int, 24>{}); break;
                    case 40: staged(std::integral_constant<int, 40>{}); break;
                    case 52: staged(std::integral_constant<int, 52>{}); break;
                    case 68: staged(std::integral_constant<int, 68>{}); break;
                    case 84: staged(std::integral_constant<int, 84>{}); break;
                    default: march(cnt, global); break;
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh->empty[s]);
                ++turn;
                more = !(ch.w_last & RSG_LAST);
            }
        };
        if (xm) chunks(std::true_type{});
        else chunks(std::false_type{});
        march(rem, global);  // rays that are not staged
    }
    epilogue<EPI, To, Tr>(active, acc, u, v, p, out, real, norm);
}

}  // namespace tomo
