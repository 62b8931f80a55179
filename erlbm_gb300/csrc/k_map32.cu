// k_map32.cu -- batched persistent kernel instantiations, FP32-shifted.
#include "batch_kernels.cuh"

namespace erlbm {

namespace {

template <int Q, int NPT>
cudaError_t go(const BatchGeo &g, const BatchRun *runs, int n_runs, int *counter, BatchResult *res, const double *aos,
               int grid, int block, size_t smem, int dbl, cudaStream_t s)
{
    auto k = k_batch<PrecShifted32, Q, NPT>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<grid, block, smem, s>>>(g, runs, n_runs, counter, res, aos, dbl);
    return cudaGetLastError();
}

template <int Q, int NPT>
int occ(int block, size_t smem)
{
    auto k = k_batch<PrecShifted32, Q, NPT>;
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

// Taylor-Green map runs, whose D3Q19 lattice of one layer is mirror symmetric in z from its initial state on
// (shifted::collide19_mirror): 14 populations a node instead of 19.  A thread owns the nodes tid and tid + H of the
// 2 H-node lattice, y and y + ny / 2, as float2 lanes: the neighbours of such a pair are a pair again, with the
// halves swapped where y wraps in the half lattice, so a population of both nodes is one 8-byte shared-memory access.
// The CTA of H threads and its energy sum are k_batch's (two nodes a thread), and so are the results' bits.
// k_batch issued some 300 instructions an update (39 memory accesses) and waited on its barriers with 14 warps an SM;
// packed arithmetic does not raise the FP32 rate, but it halves the instructions, which leaves issue slots to the
// shared-memory accesses.  2500 points, both operators, up to 3000 steps: 31.1 -> 13.1 ms.  Four CTAs of 128 threads
// an SM (128 registers); five and six are slower (13.7, 14.0).
template <int H>
__global__ void __launch_bounds__(H, H <= 128 ? 512 / H : 1)
    k_batch_mirror(BatchGeo g, const BatchRun *__restrict__ runs, int n_runs, int *__restrict__ counter,
                   BatchResult *__restrict__ res)
{
    constexpr int S = shifted::MIRROR19;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *buf = reinterpret_cast<float2 *>(smem_raw);                // two buffers of S x H
    double *red = reinterpret_cast<double *>(buf + 2 * S * H);         // H + 1
    __shared__ int s_run;
    const int tid = threadIdx.x, nx = g.nx, hy = g.ny / 2;
    const int x = tid % nx, y = tid / nx;
    // slots of the neighbours x - cx, y - cy; the halves change places where y wraps
    const int xm = wrap1(x - 1, nx), xp = wrap1(x + 1, nx), ym = wrap1(y - 1, hy) * nx, yp = wrap1(y + 1, hy) * nx;
    const bool lo = y == 0, hi = y == hy - 1;
    const bool warp_lo = __any_sync(0xffffffffu, lo), warp_hi = __any_sync(0xffffffffu, hi);
    for (;;) {
        __syncthreads();
        if (tid == 0) s_run = atomicAdd(counter, 1);
        __syncthreads();
        const int ri = s_run;
        if (ri >= n_runs) break;
        const BatchRun &r = runs[ri];
        const int op = r.op, n_steps = r.n_steps;
        const shifted::CoefMirror k = shifted::make_coef_mirror(r.k);
        float2 f[S];
        {
            float a[19], b[19];
            tg_map_init<PrecShifted32, 19>(a, x, y, r.u0, g);
            tg_map_init<PrecShifted32, 19>(b, x, y + hy, r.u0, g);
#pragma unroll
            for (int s = 0; s < S; s++) f[s] = make_float2(a[shifted::mirror19_dir(s)], b[shifted::mirror19_dir(s)]);
        }
        auto energy = [&] {
            float a[19], b[19];
#pragma unroll
            for (int s = 0; s < S; s++) {
                a[shifted::mirror19_dir(s)] = f[s].x;
                b[shifted::mirror19_dir(s)] = f[s].y;
            }
            a[6] = a[5], a[13] = a[11], a[14] = a[12], a[17] = a[15], a[18] = a[16];
            b[6] = b[5], b[13] = b[11], b[14] = b[12], b[17] = b[15], b[18] = b[16];
            double e = 0.0;
            e += PrecShifted32::energy<19>(a);
            e += PrecShifted32::energy<19>(b);
            return block_sum<false>(e, red, 2 * H, -1);
        };
        double E0 = 0.0, E = 0.0, margin = 0.0;
        int label = 0, decided = n_steps, status = 0;
        if (g.energy_every > 0) E = E0 = energy();
        int until_check = g.energy_every;
        float2 *cur = buf, *nxt = buf + S * H;
        for (int step = 0; step < n_steps; step++, until_check--) {
            if (step > 0) {
#pragma unroll
                for (int s = 0; s < S; s++) {
                    const int i = shifted::mirror19_dir(s), cx = Lat<19>::cx(i), cy = Lat<19>::cy(i);
                    const int xs = cx == 1 ? xm : (cx == -1 ? xp : x);
                    f[s] = cur[s * H + (cy == 1 ? xs + ym : (cy == -1 ? xs + yp : xs + y * nx))];
                }
                if (warp_lo) {
#pragma unroll
                    for (int s = 0; s < S; s++)
                        if (Lat<19>::cy(shifted::mirror19_dir(s)) == 1 && lo) f[s] = make_float2(f[s].y, f[s].x);
                }
                if (warp_hi) {
#pragma unroll
                    for (int s = 0; s < S; s++)
                        if (Lat<19>::cy(shifted::mirror19_dir(s)) == -1 && hi) f[s] = make_float2(f[s].y, f[s].x);
                }
            }
            if (g.energy_every > 0 && until_check == 0) {  // step > 0 && step % energy_every == 0
                until_check = g.energy_every;
                E = energy();
                const double lim = g.energy_factor * E0;
                margin = fmax(margin, isfinite(E) ? E / lim : INFINITY);
                if (E > lim || !isfinite(E)) {
                    label = 1;
                    decided = step;
                    status = 4;
                    break;
                }
            }
            if (op == OP_BGK)
                shifted::collide19_mirror<OP_BGK>(f, k);
            else
                shifted::collide19_mirror<OP_EXTREG>(f, k);  // RLBM: the same operations with its coefficients
#pragma unroll
            for (int s = 0; s < S; s++) nxt[s * H + tid] = f[s];
            float2 *t = cur;
            cur = nxt;
            nxt = t;
            __syncthreads();
        }
        if (tid == 0) {
            BatchResult o;
            o.label = label;
            o.decided_step = decided;
            o.steps_done = decided;
            o.status = status;
            o.margin = margin;
            o.energy = E;
            res[r.out] = o;
        }
    }
}

size_t mirror_smem(int h) { return (size_t)2 * shifted::MIRROR19 * h * sizeof(float2) + (h + 1) * sizeof(double); }

template <class F>
int mirror_kernel(int h, F &&f)
{
    switch (h) {
    case 32: return f(k_batch_mirror<32>);
    case 128: return f(k_batch_mirror<128>);
    case 288: return f(k_batch_mirror<288>);
    case 512: return f(k_batch_mirror<512>);
    default: return -1;
    }
}

}  // namespace

int launch_batch_fp32(int q, int npt, const BatchGeo &g, const BatchRun *runs, int n_runs, int *counter,
                      BatchResult *res, const double *aos, int grid, int block, size_t smem, int dbl,
                      cudaStream_t s)
{
    cudaError_t e;
    if (q == 19 && npt == 1) e = go<19, 1>(g, runs, n_runs, counter, res, aos, grid, block, smem, dbl, s);
    else if (q == 19 && npt == 2) e = go<19, 2>(g, runs, n_runs, counter, res, aos, grid, block, smem, dbl, s);
    else if (q == 9 && npt == 1) e = go<9, 1>(g, runs, n_runs, counter, res, aos, grid, block, smem, dbl, s);
    else if (q == 9 && npt == 2) e = go<9, 2>(g, runs, n_runs, counter, res, aos, grid, block, smem, dbl, s);
    else if (q == 9 && npt == 4) e = go<9, 4>(g, runs, n_runs, counter, res, aos, grid, block, smem, dbl, s);
    else if (q == 19 && npt == 4) e = go<19, 4>(g, runs, n_runs, counter, res, aos, grid, block, smem, dbl, s);
    else if (q == 9 && npt == 8) e = go<9, 8>(g, runs, n_runs, counter, res, aos, grid, block, smem, dbl, s);
    else return -1;
    return e == cudaSuccess ? 0 : -3;
}

// Lattices that k_batch_mirror takes: periodic one-layer D3Q19 runs from the Taylor-Green map's initial state, half
// the nodes (whole rows) being the threads of k_batch's CTA.
bool batch_mirror_ok(int prec, int q, const BatchGeo &g)
{
    const int h = g.nb / 2;
    return prec == 1 && q == 19 && g.init == INIT_TG_MAP && !g.solid && g.inlet_x < 0 && g.outlet_x < 0 &&
           !g.density_check && g.ny % 2 == 0 && (h == 32 || h == 128 || h == 288 || h == 512);
}

int batch_mirror_shape(const BatchGeo &g, int slots, int sms, int n_runs, LaunchShape *out)
{
    const int h = g.nb / 2;
    const size_t smem = mirror_smem(h);
    return mirror_kernel(h, [&](auto k) {
        int occ = 0;
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, h, smem) != cudaSuccess || occ < 1) {
            cudaGetLastError();
            return -1;
        }
        const int per_sm = slots > 0 && slots < occ ? slots : occ;
        out->npt = 2;
        out->block = h;
        out->smem = smem;
        out->dbl = 1;
        out->grid = n_runs < per_sm * sms ? n_runs : per_sm * sms;
        if (out->grid < 1) out->grid = 1;
        return 0;
    });
}

int launch_batch_mirror(const BatchGeo &g, const BatchRun *runs, int n_runs, int *counter, BatchResult *res,
                        const LaunchShape &sh, cudaStream_t s)
{
    return mirror_kernel(sh.block, [&](auto k) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh.smem);
        if (e != cudaSuccess) return -3;
        k<<<sh.grid, sh.block, sh.smem, s>>>(g, runs, n_runs, counter, res);
        return cudaGetLastError() == cudaSuccess ? 0 : -3;
    });
}

int batch_occupancy_fp32(int q, int npt, int block, size_t smem)
{
    if (q == 19 && npt == 1) return occ<19, 1>(block, smem);
    if (q == 19 && npt == 2) return occ<19, 2>(block, smem);
    if (q == 19 && npt == 4) return occ<19, 4>(block, smem);
    if (q == 9 && npt == 1) return occ<9, 1>(block, smem);
    if (q == 9 && npt == 2) return occ<9, 2>(block, smem);
    if (q == 9 && npt == 4) return occ<9, 4>(block, smem);
    if (q == 9 && npt == 8) return occ<9, 8>(block, smem);
    return 0;
}

int batch_occupancy_fp64(int q, int npt, int block, size_t smem);

int batch_occupancy(int prec, int q, int npt, int block, size_t smem)
{
    return prec == 0 ? batch_occupancy_fp64(q, npt, block, smem) : batch_occupancy_fp32(q, npt, block, smem);
}

size_t batch_smem(int prec, int q, int nb, int block, int dbl)
{
    if (prec == 0)
        return q == 9 ? batch_smem_bytes<PrecExact64, 9>(nb, block, dbl)
                      : batch_smem_bytes<PrecExact64, 19>(nb, block, dbl);
    return q == 9 ? batch_smem_bytes<PrecShifted32, 9>(nb, block, dbl)
                  : batch_smem_bytes<PrecShifted32, 19>(nb, block, dbl);
}


int launch_slot_server_fp32(const SlotRing &ring, int max_nb, int grid, int block, size_t smem, int dbl,
                            cudaStream_t s)
{
    auto k = k_slot_server<PrecShifted32, 19, 1>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return -3;
    // every resident loop asks for the largest shared-memory carveout: an SM runs CTAs of kernels with
    // one carveout at a time, so loops with different ones would keep each other off the SMs
    e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return -3;
    k<<<grid, block, smem, s>>>(ring, max_nb, dbl);
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

int slot_server_occupancy_fp32(int block, size_t smem)
{
    auto k = k_slot_server<PrecShifted32, 19, 1>;
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
