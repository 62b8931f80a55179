// k_map64.cu -- batched persistent kernel instantiations, plain FP64 (compiled with --fmad=false, the reference's rounding).
#include "batch_kernels.cuh"

namespace erlbm {

namespace {

// The Taylor-Green map's lattice has 256 fluid nodes, the obstacle map's 232.  Bounded to 256 threads, two CTAs an SM
// leave 128 registers a thread; with 288, nine warps a CTA, they leave 96 and the exact D3Q19 collision stores 728 bytes
// of spills instead of 468.  600 obstacle runs of 1000 steps when the bound came in: 117.2 -> 112 ms with the fixed-point
// sums of the collision, 113.8 without them (76.7 now; without 113).
constexpr int MAP_THREADS = 256;

template <int Q, int NPT, int MAXT = BatchBounds<NPT, 8>::MAXT>
cudaError_t go(const BatchGeo &g, const BatchRun *runs, int n_runs, int *counter, BatchResult *res, const double *aos,
               int grid, int block, size_t smem, int dbl, cudaStream_t s)
{
    auto k = k_batch<PrecExact64, Q, NPT, MAXT>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<grid, block, smem, s>>>(g, runs, n_runs, counter, res, aos, dbl);
    return cudaGetLastError();
}

template <int Q, int NPT, int MAXT = BatchBounds<NPT, 8>::MAXT>
int occ(int block, size_t smem)
{
    auto k = k_batch<PrecExact64, Q, NPT, MAXT>;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, block, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

}  // namespace

int launch_batch_fp64(int q, int npt, const BatchGeo &g, const BatchRun *runs, int n_runs, int *counter,
                      BatchResult *res, const double *aos, int grid, int block, size_t smem, int dbl,
                      cudaStream_t s)
{
    cudaError_t e;
    if (q == 19 && npt == 1 && block <= MAP_THREADS)
        e = go<19, 1, MAP_THREADS>(g, runs, n_runs, counter, res, aos, grid, block, smem, dbl, s);
    else if (q == 19 && npt == 1) e = go<19, 1>(g, runs, n_runs, counter, res, aos, grid, block, smem, dbl, s);
    else if (q == 19 && npt == 2) e = go<19, 2>(g, runs, n_runs, counter, res, aos, grid, block, smem, dbl, s);
    else if (q == 9 && npt == 1) e = go<9, 1>(g, runs, n_runs, counter, res, aos, grid, block, smem, dbl, s);
    else if (q == 9 && npt == 2) e = go<9, 2>(g, runs, n_runs, counter, res, aos, grid, block, smem, dbl, s);
    else if (q == 9 && npt == 4) e = go<9, 4>(g, runs, n_runs, counter, res, aos, grid, block, smem, dbl, s);
    else return -1;
    return e == cudaSuccess ? 0 : -3;
}

int batch_occupancy_fp64(int q, int npt, int block, size_t smem)
{
    if (q == 19 && npt == 1) return block <= MAP_THREADS ? occ<19, 1, MAP_THREADS>(block, smem) : occ<19, 1>(block, smem);
    if (q == 19 && npt == 2) return occ<19, 2>(block, smem);
    if (q == 9 && npt == 1) return occ<9, 1>(block, smem);
    if (q == 9 && npt == 2) return occ<9, 2>(block, smem);
    if (q == 9 && npt == 4) return occ<9, 4>(block, smem);
    return 0;
}


int launch_slot_server_fp64(const SlotRing &ring, int max_nb, int grid, int block, size_t smem, int dbl,
                            cudaStream_t s)
{
    auto k = k_slot_server<PrecExact64, 19, 1>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return -3;
    // every resident loop asks for the largest shared-memory carveout: an SM runs CTAs of kernels with
    // one carveout at a time, so loops with different ones would keep each other off the SMs
    e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return -3;
    k<<<grid, block, smem, s>>>(ring, max_nb, dbl);
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

int slot_server_occupancy_fp64(int block, size_t smem)
{
    auto k = k_slot_server<PrecExact64, 19, 1>;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) !=
            cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, block, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

}  // namespace erlbm
