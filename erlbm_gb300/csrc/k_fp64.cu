// k_fp64.cu -- plain FP64 kernels.  This translation unit is compiled with --fmad=false so that
// every multiply and add is rounded on its own, as in the reference's GCC -std=c++17 build.
#include "lattice_kernels.cuh"
#include "quad_fp64.cuh"

namespace erlbm {

// From this size on every scheduler has two warps or more, and the fixed-point sums of the collision cost less than
// the FP64 operations they replace; below, a warp waits for its own integer chains.  us per step without and with, one
// lane a node: D3Q19 16^3 14.4 / 18.5, 24^3 15.4 / 18.5, 32^3 23.7 / 22.6, 64^3 135.7 / 114.9; D2Q9 160^2 10.3 / 10.3,
// 200^2 16.3 / 13.4, 512^2 65.7 / 49.2.
constexpr long long FIXED_MIN_NODES = 32768;

namespace {

// k_step with four lanes a node (quad_fp64.cuh).
constexpr int QUAD_BLOCK = 64;

template <int Q, int OP>
__global__ void __launch_bounds__(QUAD_BLOCK) k_step_quad(const double *src, double *__restrict__ dst, Geo g,
                                                          BCp bc, Relax R, StepArgs a)
{
    after_previous();
    if (a.stop_on_flag && a.status != nullptr) {  // as k_step
        const int ds = __shfl_sync(0xffffffffu, *(volatile int *)&a.status->decided_step, 0);
        if (ds < a.step_index) return;
    }
    uint32_t known = 0;
    if (a.check_density) known = (uint32_t)(*(volatile unsigned long long *)&a.status->max_abs_rho_bits >> 32);
    const unsigned thread = blockIdx.x * QUAD_BLOCK + threadIdx.x;
    const long long node = thread >> 2;
    const quad::Team t{(int)(threadIdx.x & 3), (int)(threadIdx.x & 28)};
    bool active = node < g.nbox;
    if (active && g.solid != nullptr && g.solid[node]) active = false;
    double f[Q], out[2 * quad::SLOTS<Q>];
    if (active) {
        int x, y, z;
        node_xyz(g, node, x, y, z);
        state_after_planes<PrecExact64, Q>(src, g, bc, a.mode, x, y, z, node, f);
    } else {  // lanes without a node take part in the warp's shuffles
#pragma unroll
        for (int i = 0; i < Q; i++) f[i] = Lat<Q>::w(i);
    }
    const uint32_t hint = quad::collide<Q, OP>(f, t, R, out);
    if (active) {
#pragma unroll
        for (int k = 0; k < 2 * quad::SLOTS<Q>; k++) {
            const int i = quad::population<Q>(t.sub, k / 2, k % 2);
            if (i >= 0) dst[(long long)i * g.plane + node] = out[k];
        }
    }
    if (!a.check_density) return;
    const bool check = active && !exact::density_below(hint, known);
    if (!__any_sync(0xffffffffu, check)) return;
    double p[Q];
#pragma unroll
    for (int i = 0; i < Q; i++) p[i] = quad::gathered<Q>(out, t, i);
    const double rho = exact::node_density<Q>(p);
    unsigned long long rho_bits = 0;
    int flag = 0;
    if (check && !isfinite(rho)) {
        flag = 2;
    } else if (check) {
        rho_bits = (unsigned long long)__double_as_longlong(fabs(rho));
        if (fabs(rho) > a.density_limit) flag = 1;
    }
    report_density(a.status, a.step_index, rho_bits, flag);
}

// Four lanes a node up to this size.  4864 nodes give each of the 608 schedulers one such warp; beyond, a second warp
// shares the FP64 pipe, and the 13.6 warp instructions a node (8 for one lane a node) decide.  us per step with one
// lane and with four: D2Q9 32^2 6.3 / 4.4, 64^2 6.3 / 4.5, 90^2 6.3 / 6.4, 112^2 6.8 / 8.6; D3Q19 10^3 12.6 / 6.7, 16^3
// 12.3 / 7.1, 20^3 12.3 / 10.4, 22^3 13.2 / 14.4; 82 x 48 D3Q19 with planes and solids 12.3 / 7.1.
template <int Q>
constexpr long long QUAD_MAX_NODES = Q == 9 ? 7296 : 9728;

template <int Q, int OP>
int launch_quad(const Geo &g, const BCp &bc, const Relax &R, const StepArgs &a, const double *src, double *dst,
                cudaStream_t s)
{
    launch_step_kernel<k_step_quad<Q, OP>, QUAD_BLOCK>(blocks_for(4 * g.nbox, QUAD_BLOCK), s, src, dst, g, bc, R, a);
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace

int launch_step_fp64(int q, int op, const Geo &g, const BCp &bc, const Relax &R, const StepArgs &a, const double *src,
                     double *dst, cudaStream_t s)
{
    if ((q == 9 && g.nbox <= QUAD_MAX_NODES<9>) || (q == 19 && g.nbox <= QUAD_MAX_NODES<19>)) {
        if (op == OP_BGK) return (q == 9 ? launch_quad<9, OP_BGK> : launch_quad<19, OP_BGK>)(g, bc, R, a, src, dst, s);
        if (op == OP_REG) return (q == 9 ? launch_quad<9, OP_REG> : launch_quad<19, OP_REG>)(g, bc, R, a, src, dst, s);
        if (op == OP_EXTREG)
            return (q == 9 ? launch_quad<9, OP_EXTREG> : launch_quad<19, OP_EXTREG>)(g, bc, R, a, src, dst, s);
    }
    if (g.nbox < FIXED_MIN_NODES) return step_any<PrecExact64Small>(q, op, g, bc, R, a, src, dst, s);
    return step_any<PrecExact64>(q, op, g, bc, R, a, src, dst, s);
}

int launch_stream_only_fp64(int q, const Geo &g, const double *src, double *dst, cudaStream_t s)
{
    return stream_only_any<PrecExact64>(q, g, src, dst, s);
}

int launch_aos_to_soa_fp64(int q, const Geo &g, long long n, const int *nof, const double *aos, double *soa,
                           cudaStream_t s)
{
    return aos_to_soa_any<PrecExact64>(q, g, n, nof, aos, soa, s);
}

int launch_soa_to_aos_fp64(int q, const Geo &g, long long n, const int *nof, const double *soa, double *aos,
                           cudaStream_t s)
{
    return soa_to_aos_any<PrecExact64>(q, g, n, nof, soa, aos, s);
}

int launch_node_fields_fp64(int q, const Geo &g, long long n, const int *nof, const double *buf, double *e,
                            double *rho, double *u, cudaStream_t s)
{
    return node_fields_any<PrecExact64>(q, g, n, nof, buf, e, rho, u, s);
}

int launch_box_field_fp64(int q, const Geo &g, const double *buf, int field, double *out, cudaStream_t s)
{
    return box_field_any<PrecExact64>(q, g, buf, field, out, s);
}

// ------------------------------------------------------------------------------------------------
// Reductions (FP64; deterministic)
// ------------------------------------------------------------------------------------------------

namespace {

// Serial sum in index order: the reference's kinectic_energy loop (Other_functions.cpp:100-115), rounded
// after every add as that loop is, by one block.  One thread's chain of adds costs a load and an add
// latency per element (4096 elements: 170 us).  While the sum s stays in one binade [2^e, 2^(e+1)), with unit
// u = 2^(e-52), adding x >= 0 rounds to s + u rint(x / u): what each element adds is an integer multiple of u
// that does not depend on s, except at a tie.  So a chunk of SER_CHUNK elements is rounded in parallel and summed
// exactly in 64-bit integers by a scan, up to the first element that takes s out of its binade, ties, or
// is not a non-negative finite number; that element is added by a plain FP64 add, and the chunk goes on
// behind it.  A sum of n similar terms leaves its binade log2(n) times and ties ln(n) times, which is what the
// passes over a chunk are spent on.  A chunk with more than SER_STOPS such elements (ties on equal inputs) is
// finished by a plain loop.  us of erlbm_kinetic_energy, launches and read-back (some 40) included, with one thread /
// a warp / four warps / eight: 4096 nodes 214 / 66 / 55 / 60, 16384 781 / 129 / 80 / 79, 65536 3059 / 361 / 153 / 129.
constexpr int SER_WARPS = 4;
constexpr int SER_THREADS = 32 * SER_WARPS;
constexpr int SER_PER_LANE = 8;
constexpr int SER_CHUNK = SER_THREADS * SER_PER_LANE;
constexpr int SER_STOPS = 34;
// Up to this length the plain loop is as fast: the first terms leave the sum's binade one after the other, a pass over
// the chunk each.  us of erlbm_kinetic_energy by the loop and by passes: FP64 16 nodes 22 / 30, 144 30 / 45, 256 32 / 48,
// 484 43 / 56, 576 56 / 56; FP32 484 43 / 43, 784 58 / 44.
constexpr int SER_PLAIN = 512;

__global__ void __launch_bounds__(SER_THREADS) k_sum_serial(const double *__restrict__ x, long long n, double *out)
{
    constexpr unsigned long long HIDDEN = 1ull << 52, MANT = HIDDEN - 1;
    // each pass uses the other set, so that a set is written again only after two barriers
    __shared__ unsigned long long warp_sum[2][SER_WARPS], stop_sum[2][SER_WARPS];
    __shared__ double stop_x[2][SER_WARPS];
    __shared__ int stop_at[2][SER_WARPS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double s = 0.0;  // the same in every thread
    if (n <= SER_PLAIN) {
        if (tid != 0) return;
        for (long long i = 0; i < n; i++) s = s + x[i];
        *out = s;
        return;
    }
    double v[SER_PER_LANE], nx[SER_PER_LANE];
    auto load = [&](long long base, double w[SER_PER_LANE]) {
#pragma unroll
        for (int j = 0; j < SER_PER_LANE; j++) {
            const long long i = base + tid * SER_PER_LANE + j;
            w[j] = i < n ? x[i] : 0.0;  // adding +0 changes nothing
        }
    };
    load(0, nx);
    int set = 0;
    for (long long base = 0; base < n; base += SER_CHUNK) {
#pragma unroll
        for (int j = 0; j < SER_PER_LANE; j++) v[j] = nx[j];
        load(base + SER_CHUNK, nx);
        int done = 0;  // elements of the chunk already in s
        for (int stops = 0;; stops++, set ^= 1) {
            const unsigned long long sb = (unsigned long long)__double_as_longlong(s);
            const int se = (int)(sb >> 52);  // 0 for s = 0, > 2046 for a negative, infinite or NaN sum
            const bool in_binade = se >= 1 && se <= 2046;
            if (stops == SER_STOPS || (se > 2046 && done == 0)) {
                const int m = (int)(n - base < SER_CHUNK ? n - base : SER_CHUNK);
                for (int i = done; i < m; i++) s = s + x[base + i];
                break;
            }
            const unsigned long long S = in_binade ? (sb & MANT) | HIDDEN : 0ull;
            // each element in units of u: q, and whether it has to be added on its own
            unsigned long long q[SER_PER_LANE], sum = 0;
            unsigned own = 0;
#pragma unroll
            for (int j = 0; j < SER_PER_LANE; j++) {
                const bool todo = tid * SER_PER_LANE + j >= done;
                const unsigned long long b = (unsigned long long)__double_as_longlong(v[j]);
                const int xe = (int)(b >> 52);
                const int sh = se - xe;
                q[j] = 0;
                if (todo && b != 0) {
                    if (!in_binade || xe < 1 || sh < 0) {
                        own |= 1u << j;  // no binade yet, subnormal, larger than s, negative or non-finite
                    } else if (sh <= 53) {
                        const unsigned long long m = (b & MANT) | HIDDEN;
                        const unsigned long long half = sh ? 1ull << (sh - 1) : 0ull;
                        const unsigned long long rem = sh ? m & ((1ull << sh) - 1) : 0ull;
                        q[j] = (m >> sh) + (rem > half ? 1ull : 0ull);
                        if (sh && rem == half) own |= 1u << j;
                    }
                }
                sum += q[j];
            }
            // a thread whose elements alone leave the binade stops there, so what it hands on may be cut short:
            // SER_THREADS times 4 HIDDEN fit 64 bits
            sum = sum < 4 * HIDDEN ? sum : 4 * HIDDEN;
            unsigned long long incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            if (lane == 31) warp_sum[set][warp] = incl;
            __syncthreads();
            unsigned long long before = 0, total = S;
#pragma unroll
            for (int w = 0; w < SER_WARPS; w++) {
                const unsigned long long t = warp_sum[set][w];
                before += w < warp ? t : 0ull;
                total += t;
            }
            // the thread's first element that cannot be taken, with the sum before it
            unsigned long long acc = S + before + (incl - sum), at = 0;
            int stop = SER_PER_LANE;
#pragma unroll
            for (int j = 0; j < SER_PER_LANE; j++) {
                if (stop == SER_PER_LANE && (((own >> j) & 1u) || acc + q[j] >= 2 * HIDDEN)) {
                    stop = j;
                    at = acc;
                }
                acc += q[j];
            }
            const unsigned who = __ballot_sync(0xffffffffu, stop < SER_PER_LANE);
            if (lane == (who ? __ffs(who) - 1 : 0)) {
                double mine = 0.0;
#pragma unroll
                for (int j = 0; j < SER_PER_LANE; j++)
                    if (j == stop) mine = v[j];
                stop_at[set][warp] = who ? tid * SER_PER_LANE + stop : -1;
                stop_sum[set][warp] = at;
                stop_x[set][warp] = mine;
            }
            __syncthreads();
            int first = SER_WARPS;
#pragma unroll
            for (int w = SER_WARPS - 1; w >= 0; w--)
                if (stop_at[set][w] >= 0) first = w;
            if (first == SER_WARPS) {
                if (in_binade) s = __longlong_as_double((long long)((total & MANT) | ((unsigned long long)se << 52)));
                set ^= 1;
                break;
            }
            if (in_binade)
                s = __longlong_as_double((long long)((stop_sum[set][first] & MANT) | ((unsigned long long)se << 52)));
            s = s + stop_x[set][first];
            done = stop_at[set][first] + 1;
        }
    }
    if (tid == 0) *out = s;
}

constexpr int RB = 256;   // threads per reduction block
constexpr int RG = 1024;  // reduction blocks (fixed, so the tree shape does not depend on the GPU)

__global__ void __launch_bounds__(RB) k_sum_partial(const double *__restrict__ x, long long n, double *part)
{
    __shared__ double sh[RB];
    double s = 0;
    for (long long i = (long long)blockIdx.x * RB + threadIdx.x; i < n; i += (long long)RG * RB) s += x[i];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = RB / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

__global__ void __launch_bounds__(RB) k_sum_final(const double *__restrict__ part, double *out)
{
    __shared__ double sh[RB];
    double s = 0;
    for (int i = threadIdx.x; i < RG; i += RB) s += part[i];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = RB / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = sh[0];
}

__global__ void __launch_bounds__(RB) k_maxabs_partial(const double *__restrict__ x, long long n, double *part)
{
    __shared__ double sm[RB];
    __shared__ int snf[RB];
    double m = 0;
    int nf = 0;
    for (long long i = (long long)blockIdx.x * RB + threadIdx.x; i < n; i += (long long)RG * RB) {
        const double v = x[i];
        if (!isfinite(v))
            nf = 1;
        else
            m = fmax(m, fabs(v));
    }
    sm[threadIdx.x] = m;
    snf[threadIdx.x] = nf;
    __syncthreads();
    for (int o = RB / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            sm[threadIdx.x] = fmax(sm[threadIdx.x], sm[threadIdx.x + o]);
            snf[threadIdx.x] |= snf[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = sm[0];
        part[2 * blockIdx.x + 1] = snf[0] ? 1.0 : 0.0;
    }
}

__global__ void __launch_bounds__(RB) k_maxabs_final(const double *__restrict__ part, double *out)
{
    __shared__ double sm[RB], sf[RB];
    double m = 0, nf = 0;
    for (int i = threadIdx.x; i < RG; i += RB) {
        m = fmax(m, part[2 * i]);
        nf = fmax(nf, part[2 * i + 1]);
    }
    sm[threadIdx.x] = m;
    sf[threadIdx.x] = nf;
    __syncthreads();
    for (int o = RB / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            sm[threadIdx.x] = fmax(sm[threadIdx.x], sm[threadIdx.x + o]);
            sf[threadIdx.x] = fmax(sf[threadIdx.x], sf[threadIdx.x + o]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[0] = sm[0];
        out[1] = sf[0];
    }
}

}  // namespace

int launch_sum(const double *x, long long n, long long serial_limit, double *scratch, double *out, cudaStream_t s)
{
    if (n <= serial_limit) {
        k_sum_serial<<<1, SER_THREADS, 0, s>>>(x, n, out);
    } else {
        k_sum_partial<<<RG, RB, 0, s>>>(x, n, scratch);
        k_sum_final<<<1, RB, 0, s>>>(scratch, out);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

int launch_maxabs(const double *x, long long n, double *scratch, double *out, cudaStream_t s)
{
    k_maxabs_partial<<<RG, RB, 0, s>>>(x, n, scratch);
    k_maxabs_final<<<1, RB, 0, s>>>(scratch, out);
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
}


// Initial fields on the device (lattice_kernels.cuh): kind 1 = D2Q9 Taylor-Green program init,
// 4 = D3Q19 3-D Taylor-Green equilibrium, 0 = rest equilibrium.
int launch_init_fp64(int kind, int q, const Geo &g, double *buf, const double *tab, double u0, double tau, double k,
                     double rho, cudaStream_t s)
{
    return init_any<PrecExact64>(kind, q, g, buf, tab, u0, tau, k, rho, s);
}

}  // namespace erlbm

// ------------------------------------------------------------------------------------------------
// FP64 add / multiply issue rate (the roofline of the exact path, which issues them unfused)
// ------------------------------------------------------------------------------------------------

namespace erlbm {
namespace {

constexpr int RATE_CHAINS = 8;

// Eight independent multiply-then-add chains per thread; with --fmad=false each is one DMUL and one
// DADD.  The values stay bounded (x -> a x + b with a < 1); the final test keeps the work alive.
__global__ void __launch_bounds__(256) k_fp64_rate(double *out, int iters, double a, double b)
{
    double x[RATE_CHAINS];
#pragma unroll
    for (int k = 0; k < RATE_CHAINS; k++) x[k] = 1.0 + 1e-9 * (double)(threadIdx.x + 37 * k);
    for (int i = 0; i < iters; i++) {
#pragma unroll
        for (int k = 0; k < RATE_CHAINS; k++) x[k] = x[k] * a + b;
    }
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < RATE_CHAINS; k++) s = s + x[k];
    if (s == -1.0 && out) out[blockIdx.x] = s;  // never true: every x stays near 1
}

}  // namespace

// FP64 operations (each DADD and DMUL counted once, per thread) per second over one full wave of
// resident CTAs, timed with events on a private stream after one warm-up launch.
int measure_fp64_rate(double *ops_per_s)
{
    int dev = 0, sms = 0, occ = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_fp64_rate, 256, 0);
    if (e != cudaSuccess) return -3;
    if (occ < 1) occ = 1;
    const int grid = sms * occ, iters = 4096;
    cudaStream_t s = nullptr;
    cudaEvent_t a = nullptr, b = nullptr;
    int rc = -3;
    if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) == cudaSuccess && cudaEventCreate(&a) == cudaSuccess &&
        cudaEventCreate(&b) == cudaSuccess) {
        k_fp64_rate<<<grid, 256, 0, s>>>(nullptr, iters / 8, 0.999999, 1e-6);
        cudaEventRecord(a, s);
        k_fp64_rate<<<grid, 256, 0, s>>>(nullptr, iters, 0.999999, 1e-6);
        cudaEventRecord(b, s);
        float ms = 0.f;
        if (cudaEventSynchronize(b) == cudaSuccess && cudaEventElapsedTime(&ms, a, b) == cudaSuccess && ms > 0.f) {
            *ops_per_s = (double)grid * 256.0 * iters * RATE_CHAINS * 2.0 / (ms * 1e-3);
            rc = 0;
        }
    }
    if (a) cudaEventDestroy(a);
    if (b) cudaEventDestroy(b);
    if (s) cudaStreamDestroy(s);
    return rc == 0 && cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace erlbm
