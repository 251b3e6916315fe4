// Quantum-jump helpers of the Monte Carlo stepper (C ABI emusv_qubit_densities,
// emusv_apply_1q): the single-qubit reduced density matrices of a state, whose traces with
// L^dag L give the jump weights of every (qubit, operator) pair (emu_sv/algebra.py:4-25,
// expect_batch), and a 2x2 operator applied to one qubit in place (algebra.py:28-37).
#include "hpsi_kernel.cuh"
#include "profile.cuh"

namespace emusv {

constexpr int RHO_THREADS = 256;

// part[4 p + c][block]: sums over the pairs (x0, x1 = x0 | 2^p) of |psi_x0|^2, |psi_x1|^2 and
// psi_x1 conj(psi_x0) (re, im).  Blocks with blockIdx.y = g take the bits 3g..3g+2: a thread
// reads the 8 amplitudes that differ in them, so the state is read once for three bits (from
// the L2 after the first) and all groups run together.  Bound by those reads and the launch:
// n = 19 complex128 31 us before (one bit after the other, each reading the whole state).
constexpr int RHO_G = 3;
template <typename R>
__global__ void __launch_bounds__(RHO_THREADS) k_qubit_rho(const void *psi_, int n, double *part) {
    typedef typename cvec<R>::T C;
    const C *psi = reinterpret_cast<const C *>(psi_);
    constexpr int NA = 1 << RHO_G, NV = 4 * RHO_G;
    __shared__ double red[(RHO_THREADS / 32) * NV];
    const int b0 = RHO_G * blockIdx.y, m = n - b0 < RHO_G ? n - b0 : RHO_G, na = 1 << m;
    const i64 count = i64(1) << (n - m), lowmask = (i64(1) << b0) - 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double acc[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) acc[k] = 0.0;
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (i64)gridDim.x * blockDim.x) {
        const i64 x0 = ((i >> b0) << (b0 + m)) | (i & lowmask);
        C v[NA];
#pragma unroll
        for (int a = 0; a < NA; ++a) v[a] = a < na ? psi[x0 | ((i64)a << b0)] : cmake<C>(0.0, 0.0);
#pragma unroll
        for (int q = 0; q < RHO_G; ++q)
#pragma unroll
            for (int a = 0; a < NA; ++a) {
                if ((a >> q) & 1) continue;
                const double ar = double(v[a].x), ai = double(v[a].y);
                const double br = double(v[a | (1 << q)].x), bi = double(v[a | (1 << q)].y);
                acc[4 * q] += ar * ar + ai * ai;
                acc[4 * q + 1] += br * br + bi * bi;
                acc[4 * q + 2] += br * ar + bi * ai;  // b conj(a)
                acc[4 * q + 3] += bi * ar - br * ai;
            }
    }
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        acc[k] = warp_sum(acc[k]);
        if (lane == 0) red[warp * NV + k] = acc[k];
    }
    __syncthreads();
    if (threadIdx.x < 4 * m) {
        double t = 0.0;
        for (int w = 0; w < RHO_THREADS / 32; ++w) t += red[w * NV + threadIdx.x];
        part[((i64)4 * b0 + threadIdx.x) * gridDim.x + blockIdx.x] = t;
    }
}

// rho[i] (qubit i = bit n-1-i): 2x2 complex row-major, 8 doubles: [00, 01, 10, 11].  One
// block per qubit, one warp per sum.
__global__ void __launch_bounds__(128) k_finish_rho(const double *part, int nb, int n, double *rho) {
    const int i = blockIdx.x, p = n - 1 - i, k = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double v = 0.0;
#pragma unroll 4
    for (int b = lane; b < nb; b += 32) v += part[((i64)4 * p + k) * nb + b];
    v = warp_sum(v);
    if (lane) return;
    double *o = rho + 8 * i;
    if (k == 0) {
        o[0] = v;  // rho_00
        o[1] = 0.0;
    } else if (k == 1) {
        o[6] = v;  // rho_11
        o[7] = 0.0;
    } else if (k == 2) {
        o[2] = v;  // rho_01 = sum psi_0 conj(psi_1) = conj(rho_10)
        o[4] = v;  // rho_10 = sum psi_1 conj(psi_0)
    } else {
        o[3] = -v;
        o[5] = v;
    }
}

template <typename R>
__global__ void __launch_bounds__(BLOCK)
k_apply_1q(void *psi_, int n, int p, double o00r, double o00i, double o01r, double o01i, double o10r,
           double o10i, double o11r, double o11i) {
    typedef typename cvec<R>::T C;
    C *psi = reinterpret_cast<C *>(psi_);
    const i64 half = i64(1) << (n - 1);
    const i64 lowmask = (i64(1) << p) - 1;
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < half; i += (i64)gridDim.x * blockDim.x) {
        const i64 x0 = ((i >> p) << (p + 1)) | (i & lowmask), x1 = x0 | (i64(1) << p);
        const C a = psi[x0], b = psi[x1];
        const double ar = double(a.x), ai = double(a.y), br = double(b.x), bi = double(b.y);
        psi[x0] = cmake<C>(o00r * ar - o00i * ai + o01r * br - o01i * bi,
                           o00r * ai + o00i * ar + o01r * bi + o01i * br);
        psi[x1] = cmake<C>(o10r * ar - o10i * ai + o11r * br - o11i * bi,
                           o10r * ai + o10i * ar + o11r * bi + o11i * br);
    }
}

// Blocks per group of bits: eight amplitudes a thread, at most four blocks per SM over all
// groups.
static int rho_grid(int n) {
    const i64 count = n > RHO_G ? i64(1) << (n - RHO_G) : 1;
    const int groups = (n + RHO_G - 1) / RHO_G;
    const i64 g = (count + RHO_THREADS - 1) / RHO_THREADS, cap = ((i64)sm_count() * 4 + groups - 1) / groups;
    return (int)(g < cap ? g : cap);
}

}  // namespace emusv

using namespace emusv;

extern "C" {

size_t emusv_qubit_densities_scratch_bytes(int nqubits) {
    if (nqubits < 1 || nqubits > EMUSV_MAX_QUBITS) return 0;
    return sizeof(double) * (size_t)sm_count() * 4 * MAXQ * 4 + 256;
}

int emusv_qubit_densities(int nqubits, int dtype, const void *psi, double *rho_dev, void *scratch,
                          size_t scratch_bytes, void *stream) {
    if (nqubits < 1 || nqubits > EMUSV_MAX_QUBITS || !psi || !rho_dev || !scratch ||
        (dtype != EMUSV_C128 && dtype != EMUSV_C64) ||
        scratch_bytes < emusv_qubit_densities_scratch_bytes(nqubits))
        return EMUSV_BAD_ARGUMENT;
    cudaStream_t s = as_stream(stream);
    double *partials = reinterpret_cast<double *>(scratch);
    const int g = rho_grid(nqubits);
    {
        ProfScope ps_(PROF_OBS, s);
        const dim3 grid(g, (nqubits + RHO_G - 1) / RHO_G);
        if (dtype == EMUSV_C128) k_qubit_rho<double><<<grid, RHO_THREADS, 0, s>>>(psi, nqubits, partials);
        else k_qubit_rho<float><<<grid, RHO_THREADS, 0, s>>>(psi, nqubits, partials);
        k_finish_rho<<<nqubits, 128, 0, s>>>(partials, g, nqubits, rho_dev);
    }
    EMUSV_CHECK_LAUNCH();
    return EMUSV_OK;
}

int emusv_apply_1q(int nqubits, int dtype, void *psi, int qubit, const double *op, void *stream) {
    if (nqubits < 1 || nqubits > EMUSV_MAX_QUBITS || !psi || !op || qubit < 0 || qubit >= nqubits ||
        (dtype != EMUSV_C128 && dtype != EMUSV_C64))
        return EMUSV_BAD_ARGUMENT;
    for (int k = 0; k < 8; ++k)
        if (!isfinite(op[k])) return EMUSV_BAD_ARGUMENT;
    cudaStream_t s = as_stream(stream);
    const int p = nqubits - 1 - qubit;
    const i64 half = i64(1) << (nqubits - 1);
    i64 g = (half + BLOCK - 1) / BLOCK;
    if (g > (i64)sm_count() * 8) g = (i64)sm_count() * 8;
    {
        ProfScope ps_(PROF_OBS, s);
        if (dtype == EMUSV_C128)
            k_apply_1q<double><<<(int)g, BLOCK, 0, s>>>(psi, nqubits, p, op[0], op[1], op[2], op[3],
                                                         op[4], op[5], op[6], op[7]);
        else
            k_apply_1q<float><<<(int)g, BLOCK, 0, s>>>(psi, nqubits, p, op[0], op[1], op[2], op[3],
                                                        op[4], op[5], op[6], op[7]);
    }
    EMUSV_CHECK_LAUNCH();
    return EMUSV_OK;
}

}  // extern "C"
