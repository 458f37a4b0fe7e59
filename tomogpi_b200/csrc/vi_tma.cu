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
// Measured (B200): 512^3, 512 views 43.6 ms (51.6 before the window checks moved from every
// thread to the producer, the texture's 0.5 offsets went and the reads took byte addresses;
// the padded form 72.3); 256^3 2.80 ms (padded 4.85); filter and FDK backprojection together 3.80 ms
// (padded 9.99: the weights take one reciprocal square root now, in place of an IEEE division and
// root per sample); 64^3, 60 views 37 us (padded, 64 blocks of 16 slices: 148).
//
// Every wait is bounded (one second by the global timer): a wait that gives up sets
// ERR_TIMEOUT in the context's error word and the block stops; the producer first waits
// (bounded) for the copies it issued.
#include <cuda.h>

#include <mutex>

#include "vi_tma.cuh"

namespace tomo {

template <int UM, int NS, typename Tv, bool FDK>
__global__ void __launch_bounds__(VT_CONSUMERS + 32, 4)
    vi_back_tma_kernel(DevGeom g, const __grid_constant__ CUtensorMap map, const float* __restrict__ sino, long pitch,
                       Tv* __restrict__ vol, float scale, unsigned* err, int stall) {
    __shared__ VtShared<NS> sh;
    vt_init(sh);
    __syncthreads();
    VtTurn turn;
    vi_tma_tile<UM, NS, Tv, FDK>(g, &map, sino, pitch, vol, scale, err, stall, sh, turn, blockIdx.x, blockIdx.y, blockIdx.z);
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

bool vi_tma_encode(const float* sino, int nu, int nv, int np, long pitch, int ns, CUtensorMap* map) {
    const cuuint64_t dims[3] = {(cuuint64_t)nu, (cuuint64_t)nv, (cuuint64_t)np};
    const cuuint64_t strides[2] = {(cuuint64_t)pitch * 4, (cuuint64_t)pitch * nv * 4};
    const cuuint32_t box[3] = {VT_BOX_U, (cuuint32_t)vt_box_v(ns), 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    return tma_encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(sino), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

cudaError_t launch_vi_back_tma(int kind, const DevGeom& g, const float* sino, long pitch, void* vol, tomo_dtype vdt,
                               float scale, unsigned* err, cudaStream_t st, int stall) {
    if (!vi_tma_supported(sino, pitch)) return cudaErrorNotSupported;
    const int ns = vt_slices(g);
    CUtensorMap map;
    if (!vi_tma_encode(sino, g.nu, g.nv, g.np, pitch, ns, &map)) return cudaErrorInvalidValue;
    const TmaCall c{g, map, sino, pitch, vol, scale, err, st, stall};
    switch (vdt) {
        case TOMO_F32: return launch_tma_v<float>(c, kind, ns);
        case TOMO_BF16: return launch_tma_v<__nv_bfloat16>(c, kind, ns);
        case TOMO_F16: return launch_tma_v<__half>(c, kind, ns);
    }
    return cudaErrorInvalidValue;
}

}  // namespace tomo
