// C ABI: Hamiltonian diagonal, fused H*psi, energy moments, occupations, correlations.
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "hpsi_kernel.cuh"
#include "pairsums.cuh"
#include "profile.cuh"

namespace emusv {

bool make_params(int n, const double *omegas, const double *deltas, const double *phis,
                 const double *interaction, HamParams *P) {
    if (n < 1 || n > EMUSV_MAX_QUBITS || !omegas || !deltas || !phis || !interaction || !P)
        return false;
    memset(P, 0, sizeof(*P));
    P->n = n;
    int real = 1;
    for (int i = 0; i < n; ++i) {
        const int p = n - 1 - i;  // qubit i is bit n-1-i
        const double h = 0.5 * omegas[i];  // hamiltonian.py:52
        const double c = cos(phis[i]), s = sin(phis[i]);
        if (phis[i] != 0.0) real = 0;      // hamiltonian.py:61
        P->up_re[p] = h * c;               // Omega/2 e^{i phi} (hamiltonian.py:62-64)
        P->up_im[p] = h * s;
        P->dn_re[p] = h * c;               // its conjugate
        P->dn_im[p] = -h * s;
        P->field[p] = -deltas[i];
        if (!isfinite(omegas[i]) || !isfinite(deltas[i]) || !isfinite(phis[i])) return false;
    }
    if (real) {
        for (int p = 0; p < n; ++p) P->up_im[p] = P->dn_im[p] = 0.0;
    }
    P->real_coef = real;
    for (int i = 0; i < n; ++i)
        for (int j = i + 1; j < n; ++j) {
            const double u = interaction[i * n + j];  // upper triangle only
            if (!isfinite(u)) return false;
            const int p = n - 1 - i, q = n - 1 - j;
            P->U[p * MAXQ + q] = u;
            P->U[q * MAXQ + p] = u;
        }
    return true;
}

bool add_noise(const double *noise, HamParams *P) {
    if (!noise) return true;
    for (int k = 0; k < 8; ++k)
        if (!isfinite(noise[k])) return false;
    // noise[a][b] at (2a + b) * 2 (re) and + 1 (im)
    const double n00r = noise[0], n00i = noise[1], n01r = noise[2], n01i = noise[3];
    const double n10r = noise[4], n10i = noise[5], n11r = noise[6], n11i = noise[7];
    for (int p = 0; p < P->n; ++p) {
        P->up_re[p] += n10r;  // |1><0| (hamiltonian.py:66)
        P->up_im[p] += n10i;
        P->dn_re[p] += n01r;  // |0><1| (hamiltonian.py:67)
        P->dn_im[p] += n01i;
        P->field[p] += n11r - n00r;  // diagonal noise per excitation (hamiltonian.py:147-151)
    }
    P->real_coef = 0;
    P->noisy = 1;
    P->dc_re = P->n * n00r;
    P->dc_im = P->n * n00i;
    P->dg_im = n11i - n00i;
    return true;
}

int sm_count() {
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (!cached[dev]) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0)
            v = 148;
        cached[dev] = v;
    }
    return cached[dev];
}

int stream_status(cudaError_t e) { return e == cudaSuccess ? EMUSV_OK : EMUSV_CUDA_ERROR; }

// Library-wide device word for errors of calls without a status word of their own.
__device__ int g_device_error = 0;

int *device_error_word() {
    int *p = nullptr;
    if (cudaGetSymbolAddress((void **)&p, g_device_error) != cudaSuccess) return nullptr;
    return p;
}

int hpsi_tile_bits(int n) {
    int b = n - 8;
    if (b > 11) b = 11;
    if (b < 6) b = 6;
    if (b > n) b = n;
    return b;
}

template <typename R, bool REALC, int MODE>
static int launch_one(const HamParams &P, HpsiArgs A, int max_grid, cudaStream_t s, int *grid_out) {
    typedef typename cvec<R>::T C;
    const int b = A.tile_bits;
    const size_t smem = hpsi_smem<C>(b).total;
    auto kern = k_hpsi<R, REALC, MODE>;
    EMUSV_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    EMUSV_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, BLOCK, smem));
    if (per_sm < 1) per_sm = 1;
    const i64 ntiles = i64(1) << (P.n - b);
    i64 grid = (i64)sm_count() * per_sm;
    if (grid > ntiles) grid = ntiles;
    if (max_grid > 0 && grid > max_grid) grid = max_grid;
    {
        ProfScope ps_(PROF_HPSI, s);
        kern<<<(int)grid, BLOCK, smem, s>>>(P, A);
    }
    EMUSV_CHECK_LAUNCH();
    if (grid_out) *grid_out = (int)grid;
    return EMUSV_OK;
}

int pass_min_qubits(int dtype);
int launch_hpsi_passes(int dtype, const HamParams &H, const HpsiArgs &A, cudaStream_t s);

// EMUSV_HPSI_SINGLE_PASS=1 selects the single-pass tile kernel for every size (A/B checks).
static bool single_pass_forced() {
    static int v = -1;
    if (v < 0) {
        const char *e = getenv("EMUSV_HPSI_SINGLE_PASS");
        v = (e && e[0] == '1') ? 1 : 0;
    }
    return v == 1;
}

bool lz_applies(int dtype, int n);
int lz_moments(int dtype, const HamParams &H, const void *psi, void *part, double *partials,
               double *part_h, unsigned *cnt, int *err, cudaStream_t s, int *grid_out);
// Dispatch on dtype / real coefficients / mode.  Registers of at least one pass-L tile
// use the two-pass kernels for H*psi; the single-pass kernel serves small registers, the
// energy reductions and the diagonal.
int launch_hpsi(int dtype, int mode, const HamParams &P, HpsiArgs A, int max_grid,
                cudaStream_t s, int *grid_out) {
    if (mode == HP_STORE && (dtype == EMUSV_C64 || dtype == EMUSV_C128) &&
        P.n >= pass_min_qubits(dtype) && !single_pass_forced())
        return launch_hpsi_passes(dtype, P, A, s);
#define EMUSV_DISPATCH(R, M)                                                           \
    return P.real_coef ? launch_one<R, true, M>(P, A, max_grid, s, grid_out)           \
                       : launch_one<R, false, M>(P, A, max_grid, s, grid_out)
    if (dtype == EMUSV_C128) {
        switch (mode) {
        case HP_STORE: EMUSV_DISPATCH(double, HP_STORE);
        case HP_ENERGY: EMUSV_DISPATCH(double, HP_ENERGY);
        case HP_DIAG: return launch_one<double, true, HP_DIAG>(P, A, max_grid, s, grid_out);
        }
    } else if (dtype == EMUSV_C64) {
        switch (mode) {
        case HP_STORE: EMUSV_DISPATCH(float, HP_STORE);
        case HP_ENERGY: EMUSV_DISPATCH(float, HP_ENERGY);
        case HP_DIAG: return launch_one<float, true, HP_DIAG>(P, A, max_grid, s, grid_out);
        }
    }
#undef EMUSV_DISPATCH
    return EMUSV_BAD_ARGUMENT;
}

// Largest grid any streaming kernel of this library launches (bounds partial buffers).
int max_grid_blocks() { return sm_count() * 8; }

// ---------------------------------------------------------------- reduction kernels
// Sum partials[nblocks][NRED] into out[NRED] (one block, fixed order).
__global__ void k_sum_partials(const double *partials, int nblocks, double *out) {
    __shared__ double scratch[(BLOCK / 32) * NRED];
    double v[NRED];
    sum_partials<NRED>(partials, nblocks, NRED, v, scratch);
    if (threadIdx.x == 0)
        for (int k = 0; k < NRED; ++k) out[k] = v[k];
}

// |psi_x|^2 as the weight of the pair sums (occupations and correlations).
template <typename R> struct PsiWeight {
    const typename cvec<R>::T *psi;
    __device__ __forceinline__ void operator()(i64 x, double (&w)[1]) const {
        const typename cvec<R>::T a = psi[x];
        w[0] = double(a.x) * double(a.x) + double(a.y) * double(a.y);
    }
};

template <bool PAIRS>
static int launch_psi_sums(int dtype, const void *psi, int n, double *part, double *out, cudaStream_t s) {
    ProfScope ps_(PROF_OBS, s);
    if (dtype == EMUSV_C128)
        return launch_pair_sums<1, PAIRS>(PsiWeight<double>{reinterpret_cast<const double2 *>(psi)}, n, part, out,
                                          true, s);
    return launch_pair_sums<1, PAIRS>(PsiWeight<float>{reinterpret_cast<const float2 *>(psi)}, n, part, out, true, s);
}

}  // namespace emusv

using namespace emusv;

extern "C" {

int emusv_build_arch(void) { return 100; }

int emusv_device_error(void *stream) {
    int *p = device_error_word();
    if (!p) return EMUSV_CUDA_ERROR;
    int h = 0;
    cudaStream_t s = as_stream(stream);
    EMUSV_CHECK(cudaMemcpyAsync(&h, p, sizeof(int), cudaMemcpyDeviceToHost, s));
    EMUSV_CHECK(cudaStreamSynchronize(s));
    if (h) EMUSV_CHECK(cudaMemsetAsync(p, 0, sizeof(int), s));
    return h;
}

const char *emusv_status_string(int status) {
    switch (status) {
    case EMUSV_OK: return "ok";
    case EMUSV_NOT_CONVERGED: return "Krylov iteration did not converge within max_krylov_dim";
    case EMUSV_NONFINITE: return "non-finite value in a reduction";
    case EMUSV_BAD_ARGUMENT: return "bad argument";
    case EMUSV_WORKSPACE_TOO_SMALL: return "workspace too small";
    case EMUSV_CUDA_ERROR: return "CUDA runtime error";
    case EMUSV_TIMEOUT: return "device-side wait timed out";
    default: return "unknown status";
    }
}

// Scratch of the observables: FP64 partial sums, and for the moments of H on registers
// wider than one pass-L tile (emusv_expect through the streaming passes) one vector of
// the register's size for the flips of the high bits.
static size_t scratch_head_bytes(int n) {
    const size_t per = (size_t)MAXQ * MAXQ > NRED ? (size_t)MAXQ * MAXQ : NRED;
    size_t d = (size_t)max_grid_blocks() * per + 64;
    if (d < ps_partials(n, 1)) d = ps_partials(n, 1);
    return (sizeof(double) * d + 255) / 256 * 256;
}
static bool expect_by_passes(int dtype, int n) {
    return !single_pass_forced() && lz_applies(dtype, n);
}

size_t emusv_scratch_bytes(int nqubits, int dtype) {
    if (nqubits < 1 || nqubits > EMUSV_MAX_QUBITS) return 0;
    size_t b = scratch_head_bytes(nqubits);
    if (expect_by_passes(dtype, nqubits)) b += (size_t(1) << nqubits) * (dtype == EMUSV_C128 ? 16 : 8);
    return b;
}

int emusv_hamiltonian_diag(int nqubits, const double *deltas, const double *interaction,
                           double *diag_out, void *stream) {
    HamParams P;
    static const double zeros[EMUSV_MAX_QUBITS] = {0};
    if (!diag_out || !make_params(nqubits, zeros, deltas, zeros, interaction, &P))
        return EMUSV_BAD_ARGUMENT;
    HpsiArgs A = {};
    A.out = diag_out;
    A.tile_bits = hpsi_tile_bits(nqubits);
    A.su = 1.0;
    return launch_hpsi(EMUSV_C128, HP_DIAG, P, A, 0, as_stream(stream), nullptr);
}

int emusv_hpsi(int nqubits, int dtype, const double *omegas, const double *deltas,
               const double *phis, const double *interaction, const void *psi, void *out,
               void *stream) {
    HamParams P;
    if (!psi || !out || psi == out || !make_params(nqubits, omegas, deltas, phis, interaction, &P))
        return EMUSV_BAD_ARGUMENT;
    HpsiArgs A = {};
    A.u = psi;
    A.su = 1.0;
    A.out = out;
    A.part_buf = out;  // the two-pass kernels keep their partial sums in place
    A.err = device_error_word();
    A.tile_bits = hpsi_tile_bits(nqubits);
    return launch_hpsi(dtype, HP_STORE, P, A, 0, as_stream(stream), nullptr);
}

// H psi with the noise term (2x2 complex matrix on every qubit, 8 doubles row-major).
int emusv_hpsi_noisy(int nqubits, int dtype, const double *omegas, const double *deltas,
                     const double *phis, const double *interaction, const double *noise,
                     const void *psi, void *out, void *stream) {
    HamParams P;
    if (!psi || !out || psi == out || !noise ||
        !make_params(nqubits, omegas, deltas, phis, interaction, &P) || !add_noise(noise, &P))
        return EMUSV_BAD_ARGUMENT;
    HpsiArgs A = {};
    A.u = psi;
    A.su = 1.0;
    A.out = out;
    A.part_buf = out;
    A.err = device_error_word();
    A.tile_bits = hpsi_tile_bits(nqubits);
    return launch_hpsi(dtype, HP_STORE, P, A, 0, as_stream(stream), nullptr);
}

// result_dev[0..1] = <psi|H|psi> (re, im), result_dev[2] = ||H psi||^2.
int emusv_expect(int nqubits, int dtype, const double *omegas, const double *deltas,
                 const double *phis, const double *interaction, const void *psi,
                 double *result_dev, void *scratch, size_t scratch_bytes, void *stream) {
    HamParams P;
    if (!psi || !result_dev || !scratch || scratch_bytes < emusv_scratch_bytes(nqubits, dtype) ||
        !make_params(nqubits, omegas, deltas, phis, interaction, &P))
        return EMUSV_BAD_ARGUMENT;
    cudaStream_t s = as_stream(stream);
    double *partials = reinterpret_cast<double *>(scratch);
    double *sums = partials + (size_t)max_grid_blocks() * NRED;
    int grid = 0, st;
    if (expect_by_passes(dtype, nqubits) && !P.noisy) {
        // streaming passes: X_high psi into the scratch vector, then H psi per tile
        if (reinterpret_cast<uintptr_t>(psi) & 15) return EMUSV_BAD_ARGUMENT;
        unsigned char *vec = reinterpret_cast<unsigned char *>(scratch) + scratch_head_bytes(nqubits);
        double *part_h = sums + 64;  // the pass H kernels' partials (not used here)
        unsigned *cnt = reinterpret_cast<unsigned *>(part_h + (size_t)max_grid_blocks() * NRED);
        st = lz_moments(dtype, P, psi, vec, partials, part_h, cnt, device_error_word(), s, &grid);
        if (st) return st;
    } else {
        HpsiArgs A = {};
        A.u = psi;
        A.su = 1.0;
        A.partials = partials;
        A.tile_bits = hpsi_tile_bits(nqubits);
        st = launch_hpsi(dtype, HP_ENERGY, P, A, max_grid_blocks(), s, &grid);
        if (st) return st;
    }
    {
        ProfScope ps_(PROF_SMALL, s);
        k_sum_partials<<<1, BLOCK, 0, s>>>(partials, grid, sums);
    }
    EMUSV_CHECK_LAUNCH();
    // result layout: [<v,Hv> re, im, ||Hv||^2]
    EMUSV_CHECK(cudaMemcpyAsync(result_dev, sums + 1, 2 * sizeof(double), cudaMemcpyDeviceToDevice, s));
    EMUSV_CHECK(cudaMemcpyAsync(result_dev + 2, sums, sizeof(double), cudaMemcpyDeviceToDevice, s));
    return EMUSV_OK;
}

int emusv_occupation(int nqubits, int dtype, const void *psi, double *occ_dev, void *scratch,
                     size_t scratch_bytes, void *stream) {
    if (!psi || !occ_dev || !scratch || nqubits < 1 || nqubits > EMUSV_MAX_QUBITS ||
        scratch_bytes < emusv_scratch_bytes(nqubits, dtype) || (dtype != EMUSV_C128 && dtype != EMUSV_C64))
        return EMUSV_BAD_ARGUMENT;
    cudaStream_t s = as_stream(stream);
    return launch_psi_sums<false>(dtype, psi, nqubits, reinterpret_cast<double *>(scratch), occ_dev, s);
}

int emusv_correlation(int nqubits, int dtype, const void *psi, double *corr_dev, void *scratch,
                      size_t scratch_bytes, void *stream) {
    if (!psi || !corr_dev || !scratch || nqubits < 1 || nqubits > EMUSV_MAX_QUBITS ||
        scratch_bytes < emusv_scratch_bytes(nqubits, dtype) || (dtype != EMUSV_C128 && dtype != EMUSV_C64))
        return EMUSV_BAD_ARGUMENT;
    cudaStream_t s = as_stream(stream);
    return launch_psi_sums<true>(dtype, psi, nqubits, reinterpret_cast<double *>(scratch), corr_dev, s);
}

}  // extern "C"
