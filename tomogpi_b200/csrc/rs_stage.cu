// rs_stage.cu -- the STAGE form of the regular-sampling projector (rs_stage.cuh): the
// kernel, the two volume copies that it reads and their tensor maps.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <mutex>
#include <new>

#include "rs_stage.cuh"

namespace tomo {

template <int MODE, typename Tv, typename To, int EPI, typename Tr>
__global__ void __launch_bounds__(RSG_THREADS, RSG_MIN_BLOCKS)
    rs_stage_kernel(DevGeom g, const __grid_constant__ RsStageMaps maps, RsStageSrc sv, OutView<To> out, OutView<Tr> real,
                    double* __restrict__ norm, unsigned* err, int stall) {
    extern __shared__ __align__(1024) unsigned char smem[];
    // blockIdx.z: the v-tiles of the views whose rays run along x, then those of the others, so
    // that the resident blocks read one of the two copies
    const int tv = rs_tiles_v(g);
    const bool other = (int)blockIdx.z >= tv;
    const int i = blockIdx.x, n = other ? g.np - g.view_cols : g.view_cols;
    if (i >= n) {  // uniform over the block: no view here (its norm partial is 0)
        if (EPI == EPI_NORM && threadIdx.x == 0) norm[linear_block()] = 0.0;
        return;
    }
    const int p = __ldg(g.view_order + (other ? g.view_cols + i : i)), vt = blockIdx.z - (other ? tv : 0);
    if (sizeof(Tv) == 2 && (int)((i * 7u + blockIdx.y * 5u + vt * 3u) & 15u) < sv.share) {
        rs_tile<MODE, RS_LAYOUT_TEX, Tv, To, EPI, Tr>(g, nullptr, sv.tex, out, real, norm, p, blockIdx.y, vt);
        return;
    }
    rsg_init(reinterpret_cast<RsStageShared*>(smem));
    unsigned turn = 0;
    rs_stage_tile<MODE, Tv, To, EPI, Tr>(g, maps, sv, smem, turn, out, real, norm, p, blockIdx.y, vt, err, stall);
}

// The two copies of a volume [z][y][x] of type Ti: a block reads a 32 x 32 tile of a slice
// (16-bit copies: of two slices) and writes it along x and, through shared memory, along y.
template <typename Ti, typename Tv>
__global__ void __launch_bounds__(256) rs_stage_fill_kernel(const Ti* __restrict__ in, unsigned* __restrict__ rows,
                                                            unsigned* __restrict__ cols, int nx, int ny, int nz, int px,
                                                            int py, const unsigned* amax) {
    __shared__ unsigned tile[32][33];
    const float sc = fp16_scale(amax);
    const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32, z = blockIdx.z;
    const long plane = (long)nx * ny;
    for (int r = threadIdx.y; r < 32; r += 8) {
        const int x = x0 + threadIdx.x, y = y0 + r;
        if (x >= nx || y >= ny) continue;
        const long xy = (long)y * nx + x;
        unsigned w;
        if constexpr (sizeof(Tv) == 4) {
            w = __float_as_uint(in[z * plane + xy]);
        } else {  // slices z - 1 (low half) and z
            const Tv a = cvt<Tv>(z > 0 ? ldp(in + ((z - 1) * plane + xy)) * sc : 0.f);
            const Tv b = cvt<Tv>(z < nz ? ldp(in + (z * plane + xy)) * sc : 0.f);
            w = (unsigned)*reinterpret_cast<const unsigned short*>(&a) |
                ((unsigned)*reinterpret_cast<const unsigned short*>(&b) << 16);
        }
        rows[((long)z * ny + y) * px + x] = w;
        tile[r][threadIdx.x] = w;
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += 8) {
        const int x = x0 + r, y = y0 + threadIdx.x;
        if (x < nx && y < ny) cols[((long)z * nx + x) * py + y] = tile[threadIdx.x][r];
    }
}

static int stage_slices(tomo_dtype dt, int nz) { return dt == TOMO_F32 ? nz : nz + 1; }
static int pitch4(int n) { return (n + 3) & ~3; }

// What the producer would stage (rsg_produce) for a few tiles, planes and directions of the
// geometry: 27 tiles x 6 planes, about 10 us, once per geometry and launch shape.
RsStageFit rs_stage_fit(const DevGeom& g, tomo_dtype dt) {
    RsStageFit f;
    if (!tma_encode_fn() || !g.view_order || std::max({g.nx, g.ny, g.nz}) > 4096) return f;
    // a tile's window at the volume's centre, worst over the view angles: a stage holds four of its
    // planes or more
    const double su = g.du * g.fod / (g.fdd * g.dx), sv = g.dv * g.fod / (g.fdd * g.dx);
    const double w0 = 1.42 * su * rs_tile_u(g) * 1.2 + 12.0, h0 = sv * rs_tile_v(g) * 1.2 + 6.0;
    f.fits = w0 <= 84.0 && h0 <= 32.0 && w0 * h0 * 4.0 <= RSG_CAP;
    if (!f.fits) return f;
    const int tu = rs_tile_u(g), tv = rs_tile_v(g), nut = rs_tiles_u(g), nvt = rs_tiles_v(g);
    const double edge = dt == TOMO_F32 ? 2.5 : 1.5;  // rows beside a window's span: FP32 slices / slice pairs
    const double fod = g.fod / g.dx, fdd = g.fdd / g.dx, du = g.du / g.dx, dv = g.dv / g.dx;
    double samples = 0, words = 0, missed = 0, length = 0;
    int tiles = 0;
    for (int d = 0; d < (g.nx == g.ny ? 3 : 6); ++d) {  // three directions of the first octant, and across it
        const double phi = d < 3 ? 0.1 + 0.3 * d : M_PI / 2 - 0.1 - 0.3 * (d - 3), al = std::cos(phi), be = std::sin(phi);
        for (int i = 0; i < 9; ++i) {
            const int ut = (2 * (i % 3) + 1) * nut / 6, vt = (2 * (i / 3) + 1) * nvt / 6;
            const int u0 = ut * tu, u1 = std::min(u0 + tu, g.nu) - 1, v0 = vt * tv, v1 = std::min(v0 + tv, g.nv) - 1;
            // the axis that the tile's central ray runs along
            const double um = 0.5 * (u0 + u1), cm = (um - g.uc) * du;
            const bool xm = std::fabs(al * fdd - cm * be) >= std::fabs(be * fdd + cm * al);
            const double nm = xm ? g.nx : g.ny, nt = xm ? g.ny : g.nx;
            const double ms = (xm ? g.xc : g.yc) - fod * (xm ? al : be), ts = (xm ? g.yc : g.xc) - fod * (xm ? be : al);
            // a ray's steps along and across it for detector column u
            auto along = [&](double u) { const double c = (u - g.uc) * du; return xm ? al * fdd - c * be : be * fdd + c * al; };
            auto across = [&](double u) { const double c = (u - g.uc) * du; return xm ? be * fdd + c * al : al * fdd - c * be; };
            const double m = along(um), t = across(um), z = (0.5 * (v0 + v1) - g.vc) * dv;
            double lo = 0, hi = nm - 1;  // planes that the central ray crosses inside the volume
            const double c[2] = {ts, g.zc}, s[2] = {t / m, z / m}, n[2] = {nt - 1, (double)g.nz - 1};
            for (int k = 0; k < 2; ++k) {
                const double p0 = (0 - c[k]) / s[k], p1 = (n[k] - c[k]) / s[k];
                if (std::fabs(s[k]) < 1e-9) continue;
                lo = std::max(lo, ms + std::min(p0, p1));
                hi = std::min(hi, ms + std::max(p0, p1));
            }
            if (!(hi - lo >= 1)) continue;
            const double a0 = along(u0), a1 = along(u1);
            const double steps = (hi - lo + 1) * std::sqrt(m * m + t * t + z * z) / std::fabs(m);
            const double here = steps * (u1 - u0 + 1) * (v1 - v0 + 1);
            samples += here;
            length += steps;
            ++tiles;
            if (!(std::min(a0, a1) > 0.25 * fdd || std::max(a0, a1) < -0.25 * fdd)) {
                missed += here;
                continue;
            }
            const double st[2] = {across(u0) / a0, across(u1) / a1};
            double zl = 1e30, zh = -1e30;
            for (int k = 0; k < 4; ++k) {
                const double q = ((k & 1 ? v1 : v0) - g.vc) * dv / (k & 2 ? a1 : a0);
                zl = std::min(zl, q);
                zh = std::max(zh, q);
            }
            const double sl[2] = {std::min(st[0], st[1]), zl}, sh[2] = {std::max(st[0], st[1]), zh};
            for (int k = 0; k < 6; ++k) {
                const double p = std::floor(lo + k * (hi - lo) / 5.0), weight = (k % 5 ? 0.2 : 0.1);
                double best = 0;
                for (int C = 1; C <= RSG_CMAX && C <= hi - lo + 1; ++C) {
                    const double e0 = p - 0.5 * (C - 1) - 0.15 - ms, e1 = p + 0.5 * (C + 1) + 0.15 - ms;
                    double span[2];
                    for (int q = 0; q < 2; ++q)
                        span[q] = std::max({e0 * sl[q], e0 * sh[q], e1 * sl[q], e1 * sh[q]}) -
                                  std::min({e0 * sl[q], e0 * sh[q], e1 * sl[q], e1 * sh[q]}) + 0.2;
                    int wi = 0, hj = 0;
                    while (wi < RSG_WIDTHS && rsg_width(wi) < span[0] + 3.5) ++wi;
                    while (hj < RSG_HEIGHTS && rsg_height(hj) < span[1] + edge) ++hj;
                    const int wh = rsg_width(wi) * rsg_height(hj);
                    if (wi == RSG_WIDTHS || hj == RSG_HEIGHTS || (C + 2) * ((wh + 31) & ~31) > RSG_CAP) break;
                    best = (C + 2.0) * wh / C;  // words per plane
                }
                if (best > 0) words += weight * best * (hi - lo + 1);
                else missed += weight * here;
            }
        }
    }
    if (!tiles) return f;
    f.words = words / samples;
    f.missed = missed / samples;
    f.length = length / tiles;
    f.hit = tiles / (g.nx == g.ny ? 27.0 : 54.0);
    return f;
}

// Whether staging is the faster. A projection's time over that of the texture's gathers was
// measured for 600 FP32 and 170 16-bit geometries (16^3 .. 288^3, 8 .. 300 views, pixels of
// 0.12 .. 1.3 voxels at the centre, sources from 0.75 to 5 volume widths away, flat and deep
// volumes) and fits: staged words per sample, the share of the samples whose window fits no stage
// and that read global memory, and the wait for a block's first chunks over its rays' length,
// which shows more where few rays cross the volume. None of them is staged at a loss. E.g. FP32 160^3: 0.46 (0.25 voxels a pixel), 0.57
// (1.0), 0.76 (1.3), 1.33 (1.3, source 0.75 widths away); 33 x 33 x 500: 2.6. 16-bit volumes,
// which also pay a second fill: 0.89 (200^3, 60 views, 0.5 voxels), 0.98 (1.0), 1.11 (1.2);
// 128^3 1.04 (64 views), 0.99 (128); below 128^3 1.02 to 1.4 from 0.5 voxels on; 300 x 300 x 30
// (2400 blocks) 1.03.
bool rs_stage_pays(const RsStageFit& f, const DevGeom& g, tomo_dtype dt) {
    if (!f.fits) return false;
    const double vox = (double)g.nx * g.ny * g.nz, rays = (double)g.np * g.nu * g.nv;
    if (dt == TOMO_F32) {
        const double full = f.hit * rays / 256;  // blocks' worth of rays through the volume
        const double warp = g.rs_wlog == 3 ? 0.0 : g.rs_wlog == 4 ? 0.07 : 0.17;  // wider warps: more bank conflicts
        return 0.33 + 0.101 * f.words + 5.7 * f.missed + (6.2 + 2.4 * std::min(3.0, 900 / full)) / f.length + warp < 0.885;
    }
    const double blocks = (double)g.np * rs_tiles_u(g) * rs_tiles_v(g);  // 256 blocks / rays: partial tiles
    return vox >= 2097152.0 && blocks >= 3000 &&
           0.453 + 0.0523 * f.words + 5.5 * f.missed + 3.68 * vox / (rays * f.length) + 11.2 / f.length +
                   0.281 * 256 * blocks / rays < 0.985;
}

// Copies of up to 64 MiB come from a pool of their device that keeps as much of what is freed, so
// that small jobs, one context after another, do not pay the driver's allocation each time (a
// context's first FP32 projection, 64^3, 60 views: 110 us, 420 with cudaMalloc). Larger ones
// are cudaMalloc's: at 384^3 2.5 ms from the pool, 0.4. Pool memory is allocated and released
// on a stream of the pool's on which nothing else runs.
constexpr size_t POOL_KEEP = 64u << 20;
struct StagePool {
    std::mutex mu;
    cudaMemPool_t pool = nullptr;
    cudaStream_t st = nullptr;
};
static StagePool* stage_pool(int dev) {
    static StagePool pools[64];
    return dev >= 0 && dev < 64 ? &pools[dev] : nullptr;
}
static cudaError_t pool_alloc(void** p, size_t bytes, int dev) {
    StagePool* sp = stage_pool(dev);
    if (!sp) return cudaErrorMemoryAllocation;
    {
        std::lock_guard<std::mutex> lock(sp->mu);
        cudaError_t e = cudaSuccess;
        if (!sp->st) e = cudaStreamCreateWithFlags(&sp->st, cudaStreamNonBlocking);
        if (e == cudaSuccess && !sp->pool) {
            cudaMemPoolProps pp{};
            pp.allocType = cudaMemAllocationTypePinned;
            pp.location.type = cudaMemLocationTypeDevice;
            pp.location.id = dev;
            unsigned long long keep = POOL_KEEP;
            e = cudaMemPoolCreate(&sp->pool, &pp);
            if (e == cudaSuccess) e = cudaMemPoolSetAttribute(sp->pool, cudaMemPoolAttrReleaseThreshold, &keep);
        }
        if (e != cudaSuccess) return e;
    }
    const cudaError_t e = cudaMallocFromPoolAsync(p, bytes, sp->pool, sp->st);
    return e == cudaSuccess ? cudaStreamSynchronize(sp->st) : e;  // usable from any stream
}

void rs_stage_trim(int dev) {
    StagePool* sp = stage_pool(dev);
    if (!sp) return;
    std::lock_guard<std::mutex> lock(sp->mu);
    if (sp->pool) cudaMemPoolTrimTo(sp->pool, 0);
}

cudaError_t rs_stage_create(int nx, int ny, int nz, tomo_dtype dt, RsStage* t) {
    *t = RsStage();
    const int nzr = stage_slices(dt, nz);
    const int px = pitch4(nx), py = pitch4(ny);
    // one allocation: rows, then cols from a 256-byte boundary
    const size_t rb = ((size_t)nzr * ny * px * 4 + 255) & ~(size_t)255, cb = (size_t)nzr * nx * py * 4;
    char* base = nullptr;
    cudaError_t e = cudaGetDevice(&t->device);
    t->pooled = rb + cb <= POOL_KEEP;
    if (e == cudaSuccess) e = t->pooled ? pool_alloc((void**)&base, rb + cb, t->device) : cudaMalloc((void**)&base, rb + cb);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return e;
    }
    t->rows = base;
    t->cols = base + rb;
    t->maps = new (std::nothrow) RsStageMaps;
    if (!t->maps) e = cudaErrorMemoryAllocation;
    for (int o = 0; o < 2 && e == cudaSuccess; ++o) {
        // dimensions (t, z, m): rows [z][y][x] march along y, cols [z][x][y] along x
        void* p = o ? t->cols : t->rows;
        const cuuint64_t nt = o ? ny : nx, nm = o ? nx : ny, pitch = o ? py : px;
        const cuuint64_t dims[3] = {nt, (cuuint64_t)nzr, nm};
        const cuuint64_t strides[2] = {nm * pitch * 4, pitch * 4};
        const cuuint32_t estr[3] = {1, 1, 1};
        for (int i = 0; i < RSG_WIDTHS && e == cudaSuccess; ++i)
            for (int j = 0; j < RSG_HEIGHTS && e == cudaSuccess; ++j) {
                const cuuint32_t box[3] = {(cuuint32_t)rsg_width(i), (cuuint32_t)rsg_height(j), 1};
                if (tma_encode_fn()(&t->maps->m[o][i][j], CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, p, dims,
                                    strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                    CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                    e = cudaErrorInvalidValue;
            }
    }
    if (e != cudaSuccess) {
        rs_stage_destroy(t);
        cudaGetLastError();
        return e;
    }
    t->dt = dt;
    t->px = px;
    t->py = py;
    return cudaSuccess;
}

void rs_stage_destroy(RsStage* t) {
    if (t->rows && t->pooled) {
        // the launches that read the copies may be on any stream; where they cannot be waited for
        // (another thread captures) the memory is not reused
        if (cudaDeviceSynchronize() == cudaSuccess) {
            cudaFreeAsync(t->rows, stage_pool(t->device)->st);
            cudaStreamSynchronize(stage_pool(t->device)->st);
        }
    } else {
        cudaFree(t->rows);  // the one allocation
    }
    delete t->maps;
    *t = RsStage();
}

cudaError_t rs_stage_fill(const void* vol, tomo_dtype vdt, int nx, int ny, int nz, const RsStage& t, cudaStream_t st,
                          const unsigned* amax) {
    const dim3 block(32, 8), grid((nx + 31) / 32, (ny + 31) / 32, stage_slices(t.dt, nz));
#define TOMO_FILL(TI, TV)                                                                                          \
    {                                                                                                              \
        rs_stage_fill_kernel<TI, TV><<<grid, block, 0, st>>>((const TI*)vol, (unsigned*)t.rows, (unsigned*)t.cols, \
                                                             nx, ny, nz, t.px, t.py, amax);                        \
        return cudaGetLastError();                                                                                 \
    }
    if (vdt == TOMO_F32 && t.dt == TOMO_F32) TOMO_FILL(float, float)
    if (vdt == TOMO_F32 && t.dt == TOMO_BF16) TOMO_FILL(float, __nv_bfloat16)
    if (vdt == TOMO_F32 && t.dt == TOMO_F16) TOMO_FILL(float, __half)
    if (vdt == TOMO_BF16 && t.dt == TOMO_BF16) TOMO_FILL(__nv_bfloat16, __nv_bfloat16)
    if (vdt == TOMO_F16 && t.dt == TOMO_F16) TOMO_FILL(__half, __half)
#undef TOMO_FILL
    return cudaErrorInvalidValue;
}

static dim3 stage_grid(const DevGeom& g) {
    return dim3(std::max(g.view_cols, g.np - g.view_cols), rs_tiles_u(g), 2 * rs_tiles_v(g));
}

size_t rs_stage_grid_blocks(const DevGeom& g) {
    const dim3 d = stage_grid(g);
    return (size_t)d.x * d.y * d.z;
}

template <int MODE, int EPI, typename Tv, typename To, typename Tr>
static cudaError_t launch_stage_k(const DevGeom& g, const RsStage& t, unsigned long long tex, const OutView<void>& out, const OutView<void>& real,
                                  double* norm, unsigned* err, cudaStream_t st, int stall) {
    auto k = rs_stage_kernel<MODE, Tv, To, EPI, Tr>;
    static std::atomic<unsigned long long> ready{0};  // devices on which the kernel may use its shared memory
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess && !(ready.load() >> (dev & 63) & 1)) {
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, RSG_SMEM);
        if (e == cudaSuccess && dev < 64) ready.fetch_or(1ull << dev);
    }
    if (e != cudaSuccess) return e;
    const RsStageSrc sv{(const unsigned*)t.rows, t.px, tex, sizeof(Tv) == 4 ? 0 : RSG_SHARE16};
    k<<<stage_grid(g), RSG_THREADS, RSG_SMEM, st>>>(g, *t.maps, sv, out.as<To>(), real.as<Tr>(), norm, err, stall);
    return cudaGetLastError();
}

template <int MODE, typename Tv>
static cudaError_t launch_stage_e(int epi, const DevGeom& g, const RsStage& t, unsigned long long tex, const OutView<void>& out, tomo_dtype odt,
                                  const OutView<void>& real, tomo_dtype rdt, double* norm, unsigned* err, cudaStream_t st, int stall) {
    using B = __nv_bfloat16;
    if (epi == EPI_STORE) {
        switch (odt) {
            case TOMO_F32: return launch_stage_k<MODE, EPI_STORE, Tv, float, float>(g, t, tex, out, real, norm, err, st, stall);
            case TOMO_BF16: return launch_stage_k<MODE, EPI_STORE, Tv, B, B>(g, t, tex, out, real, norm, err, st, stall);
            case TOMO_F16: return launch_stage_k<MODE, EPI_STORE, Tv, __half, __half>(g, t, tex, out, real, norm, err, st, stall);
        }
    } else if (epi == EPI_RESIDUAL) {
        switch (rdt) {
            case TOMO_F32: return launch_stage_k<MODE, EPI_RESIDUAL, Tv, float, float>(g, t, tex, out, real, norm, err, st, stall);
            case TOMO_BF16: return launch_stage_k<MODE, EPI_RESIDUAL, Tv, float, B>(g, t, tex, out, real, norm, err, st, stall);
            case TOMO_F16: return launch_stage_k<MODE, EPI_RESIDUAL, Tv, float, __half>(g, t, tex, out, real, norm, err, st, stall);
        }
    } else if (epi == EPI_NORM) {
        return launch_stage_k<MODE, EPI_NORM, Tv, float, float>(g, t, tex, out, real, norm, err, st, stall);
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_rs_stage(int mode, int epi, const DevGeom& g, const RsStage& t, unsigned long long tex, const OutView<void>& out,
                            tomo_dtype odt, const OutView<void>& real, tomo_dtype rdt, double* norm, unsigned* err,
                            cudaStream_t st, int stall) {
#define TOMO_STAGE(TV)                                                                          \
    return mode == 0 ? launch_stage_e<0, TV>(epi, g, t, tex, out, odt, real, rdt, norm, err, st, stall)     \
                     : launch_stage_e<1, TV>(epi, g, t, tex, out, odt, real, rdt, norm, err, st, stall);
    switch (t.dt) {
        case TOMO_F32: TOMO_STAGE(float)
        case TOMO_BF16: TOMO_STAGE(__nv_bfloat16)
        case TOMO_F16: TOMO_STAGE(__half)
    }
#undef TOMO_STAGE
    return cudaErrorInvalidValue;
}

}  // namespace tomo
