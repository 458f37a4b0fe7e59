// rs_stage.cu -- the STAGE form of the regular-sampling projector (rs_stage.cuh): the
// kernel, the two volume copies that it reads and their tensor maps.
#include <algorithm>
#include <atomic>
#include <vector>

#include "rs_stage.cuh"

namespace tomo {

template <int MODE, typename To, int EPI, typename Tr>
__global__ void __launch_bounds__(RSG_THREADS, RSG_MIN_BLOCKS)
    rs_stage_kernel(DevGeom g, RsStageSrc sv, OutView<To> out, OutView<Tr> real, double* __restrict__ norm, unsigned* err) {
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
    rsg_init(reinterpret_cast<RsStageShared*>(smem));
    unsigned turn = 0;
    rs_stage_tile<MODE, To, EPI, Tr>(g, sv, smem, turn, out, real, norm, __ldg(g.view_order + (other ? g.view_cols + i : i)),
                                         blockIdx.y, blockIdx.z - (other ? tv : 0), err);
}

// The two copies of a volume [z][y][x]: a block reads a 32 x 32 tile of a slice and writes it
// along x and, through shared memory, along y.
__global__ void __launch_bounds__(256) rs_stage_fill_kernel(const float* __restrict__ in, float* __restrict__ rows,
                                                            float* __restrict__ cols, int nx, int ny, int px, int py) {
    __shared__ float tile[32][33];
    const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32, z = blockIdx.z;
    for (int r = threadIdx.y; r < 32; r += 8) {
        const int x = x0 + threadIdx.x, y = y0 + r;
        if (x >= nx || y >= ny) continue;
        const float v = in[((long)z * ny + y) * nx + x];
        rows[((long)z * ny + y) * px + x] = v;
        tile[r][threadIdx.x] = v;
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += 8) {
        const int x = x0 + r, y = y0 + threadIdx.x;
        if (x < nx && y < ny) cols[((long)z * nx + x) * py + y] = tile[threadIdx.x][r];
    }
}

static int pitch4(int n) { return (n + 3) & ~3; }

bool rs_stage_supported(const DevGeom& g) {
    if (!tma_encode_fn() || !g.view_order || std::max({g.nx, g.ny, g.nz}) > 4096) return false;
    // A tile's window at the volume's centre, worst over the view angles: a stage has to hold
    // four of its planes or more (at spacings of several voxels per pixel a staged word
    // serves less than one sample, and the gathers of the texture are faster).
    const float su = g.du * g.fod / (g.fdd * g.dx), sv = g.dv * g.fod / (g.fdd * g.dx);
    const float w = 1.42f * su * (float)rs_tile_u(g) * 1.2f + 12.0f, h = sv * (float)rs_tile_v(g) * 1.2f + 6.0f;
    return w <= 88.0f && h <= 32.0f && w * h * 4.0f <= (float)RSG_CAP;
}

cudaError_t rs_stage_create(int nx, int ny, int nz, RsStage* t) {
    *t = RsStage();
    const int px = pitch4(nx), py = pitch4(ny);
    // one allocation: rows, then cols, then the maps, each from a 256-byte boundary
    auto up = [](size_t n) { return (n + 255) & ~(size_t)255; };
    const size_t rb = up((size_t)nz * ny * px * 4), cb = up((size_t)nz * nx * py * 4);
    char* base = nullptr;
    cudaError_t e = cudaMalloc((void**)&base, rb + cb + 2 * RSG_WIDTHS * RSG_HEIGHTS * sizeof(CUtensorMap));
    if (e != cudaSuccess) {
        cudaGetLastError();
        return e;
    }
    t->rows = base;
    t->cols = base + rb;
    t->maps = base + rb + cb;
    std::vector<CUtensorMap> m(2 * RSG_WIDTHS * RSG_HEIGHTS);
    for (int o = 0; o < 2 && e == cudaSuccess; ++o) {
        // dimensions (t, z, m): rows [z][y][x] march along y, cols [z][x][y] along x
        void* p = o ? t->cols : t->rows;
        const cuuint64_t nt = o ? ny : nx, nm = o ? nx : ny, pitch = o ? py : px;
        const cuuint64_t dims[3] = {nt, (cuuint64_t)nz, nm};
        const cuuint64_t strides[2] = {nm * pitch * 4, pitch * 4};
        const cuuint32_t estr[3] = {1, 1, 1};
        for (int i = 0; i < RSG_WIDTHS && e == cudaSuccess; ++i)
            for (int j = 0; j < RSG_HEIGHTS && e == cudaSuccess; ++j) {
                const cuuint32_t box[3] = {(cuuint32_t)rsg_width(i), (cuuint32_t)rsg_height(j), 1};
                if (tma_encode_fn()(&m[(o * RSG_WIDTHS + i) * RSG_HEIGHTS + j], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, p, dims,
                                    strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                    CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                    e = cudaErrorInvalidValue;
            }
    }
    if (e == cudaSuccess)
        e = cudaMemcpy(t->maps, m.data(), m.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        rs_stage_destroy(t);
        cudaGetLastError();
        return e;
    }
    t->px = px;
    t->py = py;
    return cudaSuccess;
}

void rs_stage_destroy(RsStage* t) {
    cudaFree(t->rows);  // the one allocation
    *t = RsStage();
}

cudaError_t rs_stage_fill(const float* vol, int nx, int ny, int nz, const RsStage& t, cudaStream_t st) {
    const dim3 block(32, 8), grid((nx + 31) / 32, (ny + 31) / 32, nz);
    rs_stage_fill_kernel<<<grid, block, 0, st>>>(vol, (float*)t.rows, (float*)t.cols, nx, ny, t.px, t.py);
    return cudaGetLastError();
}

template <int MODE, int EPI, typename To, typename Tr>
static cudaError_t launch_stage_k(const DevGeom& g, const RsStage& t, const OutView<void>& out, const OutView<void>& real,
                                  double* norm, unsigned* err, cudaStream_t st) {
    auto k = rs_stage_kernel<MODE, To, EPI, Tr>;
    static std::atomic<unsigned long long> ready{0};  // devices on which the kernel may use its shared memory
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess && !(ready.load() >> (dev & 63) & 1)) {
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, RSG_SMEM);
        if (e == cudaSuccess && dev < 64) ready.fetch_or(1ull << dev);
    }
    if (e != cudaSuccess) return e;
    const dim3 grid(std::max(g.view_cols, g.np - g.view_cols), rs_tiles_u(g), 2 * rs_tiles_v(g));
    const RsStageSrc sv{(const CUtensorMap*)t.maps, (const float*)t.rows, t.px};
    k<<<grid, RSG_THREADS, RSG_SMEM, st>>>(g, sv, out.as<To>(), real.as<Tr>(), norm, err);
    return cudaGetLastError();
}

template <int MODE>
static cudaError_t launch_stage_e(int epi, const DevGeom& g, const RsStage& t, const OutView<void>& out, tomo_dtype odt,
                                  const OutView<void>& real, tomo_dtype rdt, double* norm, unsigned* err, cudaStream_t st) {
    using B = __nv_bfloat16;
    if (epi == EPI_STORE) {
        switch (odt) {
            case TOMO_F32: return launch_stage_k<MODE, EPI_STORE, float, float>(g, t, out, real, norm, err, st);
            case TOMO_BF16: return launch_stage_k<MODE, EPI_STORE, B, B>(g, t, out, real, norm, err, st);
            case TOMO_F16: return launch_stage_k<MODE, EPI_STORE, __half, __half>(g, t, out, real, norm, err, st);
        }
    } else if (epi == EPI_RESIDUAL) {
        switch (rdt) {
            case TOMO_F32: return launch_stage_k<MODE, EPI_RESIDUAL, float, float>(g, t, out, real, norm, err, st);
            case TOMO_BF16: return launch_stage_k<MODE, EPI_RESIDUAL, float, B>(g, t, out, real, norm, err, st);
            case TOMO_F16: return launch_stage_k<MODE, EPI_RESIDUAL, float, __half>(g, t, out, real, norm, err, st);
        }
    } else if (epi == EPI_NORM) {
        return launch_stage_k<MODE, EPI_NORM, float, float>(g, t, out, real, norm, err, st);
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_rs_stage(int mode, int epi, const DevGeom& g, const RsStage& t, const OutView<void>& out,
                            tomo_dtype odt, const OutView<void>& real, tomo_dtype rdt, double* norm, unsigned* err,
                            cudaStream_t st) {
    return mode == 0 ? launch_stage_e<0>(epi, g, t, out, odt, real, rdt, norm, err, st)
                     : launch_stage_e<1>(epi, g, t, out, odt, real, rdt, norm, err, st);
}

}  // namespace tomo
