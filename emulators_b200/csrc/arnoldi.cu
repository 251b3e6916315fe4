// Arnoldi exponential step for the non-Hermitian Hamiltonian with the noise term (C ABI
// emusv_arnoldi_step): exp(-i dt H) psi with H = H_Rydberg - 0.5i sum_j L_j^dag L_j, the
// Krylov path of the Monte Carlo stepper (emu_sv/time_evolution/implementations.py:148-166,
// krylov_exp.py:23-106 with is_hermitian=False).
//
// Per iteration j (basis vectors stored unnormalised with FP64 scales, as in krylov.cu):
//   1. w = (H - sigma) v~_j by the streaming H*psi kernels (noise diagonal fused into pass
//      L; sigma = the previous step's energy, as in the Lanczos step: same basis, T minus
//      sigma on its diagonal, added back in every exponential);
//   2. two Gram-Schmidt passes with the second round of v~_j lagged into them (see
//      k_arn_lagdots below): the same Hessenberg matrix and basis as the reference's
//      modified Gram-Schmidt (krylov_exp.py:54-58) in exact arithmetic, every vector
//      orthogonalised twice, in two streaming passes instead of 2(j+1) dependent dot/axpy
//      pairs;
//   3. k_arn_decide (one CTA, FP64): ||w'||, the happy-breakdown test (krylov_exp.py:
//   63-71) at every iteration, and from the host's hint on the exponential of the extended
//   Hessenberg matrix and the Expokit error estimate (krylov_exp.py:76-86); when the first
//   tested iteration already converges, the untested earlier ones are tested in order.
// The small exponentials: exp(A) e_0 of the dense extended Hessenberg matrix by s
// substeps of a 34-term Taylor series with ||A/s||_1 <= 4 (truncation below 1e-19 per
// substep), matrix-vector products split over 2-8 threads per row.
#include <string.h>

#include "krylov_internal.cuh"
#include "profile.cuh"

namespace emusv {

int launch_hpsi(int dtype, int mode, const HamParams &P, HpsiArgs A, int max_grid,
                cudaStream_t s, int *grid_out);
int hpsi_tile_bits(int n);
int arnoldi_run(const HamParams &P, const LindbladJumps *J, int dtype, double dt, const void *psi_in,
                void *psi_out, double exp_tolerance, double norm_tolerance, int max_krylov_dim,
                int krylov_dim_hint, void *workspace, size_t workspace_bytes,
                emusv_krylov_info *info, void *stream);

constexpr int ARN_KMAX = 100;                  // largest Arnoldi max_krylov_dim
constexpr int ARN_M = ARN_KMAX + 2;            // largest extended matrix
constexpr int ARN_KA = ARN_KMAX + 1;           // finalised basis vectors at most
// Partial sums of a pass, value-major ([value][block]): per group of ARN_KB basis vectors 32
// values, (k - group start) * 4 + c with c = 0, 1: z_k = <v_k, w> (re, im), 2, 3: s_k =
// <v_k, vt>; then a = <vt, w> (re, im), ||w||^2, ||vt||^2 (pass A) and pass B's norm.
constexpr int ARN_KB = 8;
constexpr int ARN_GROUPS = (ARN_KA + ARN_KB - 1) / ARN_KB;
constexpr int ARN_A0 = 32 * ARN_GROUPS, ARN_NORM = ARN_A0 + 4;
constexpr int ARN_PS = ARN_A0 + 5;
constexpr int ORTHO_THREADS = 256;
constexpr int DECIDE_THREADS = 512;
constexpr int STAGE_THREADS = 1024;

struct ArnState {
    double2 T[ARN_M * ARN_M];  // Hessenberg matrix of H - sigma (row-major [r][c]), basis v_k
    double2 cw1[ARN_M];        // pass B: w' = cw w - ct vt - sum cw1_l v_l
    double2 cvj[ARN_M];        //         v_j = cv vt - sum cvj_l v_l
    double2 ct;
    double cw, cv;
};

// The orthogonalisation is classical Gram-Schmidt with its second round lagged by one
// iteration (the low-synchronisation "DCGS2" form): iteration j receives w = (H - sigma) vt
// for the not yet reorthogonalised vt = v~_j, and
//   pass A (k_arn_lagdots): one pass over w, vt and the final v_0..v_{j-1}: z = V^H w,
//     s = V^H vt, <vt, w>, ||w||^2, ||vt||^2;
//   k_arn_lagstage: v_j = (vt - V s) / alpha (alpha^2 = ||vt||^2 - |s|^2) corrects the
//     previous Hessenberg column (T[:, j-1] += beta s, T[j][j-1] = beta alpha), H v_j =
//     (w - V_j T s) / alpha by the Arnoldi relation, h = V_j^H H v_j from z, s and T;
//   pass B (k_arn_lagupdate): w' = H v_j - V_j h and the corrected v_j in one pass (both
//     combinations of w, vt and V), ||w'||^2.
// Two streaming passes per iteration; every basis vector but the newest is orthogonalised
// twice, as in classical Gram-Schmidt with reorthogonalisation.
//
// Pass A is the basis read once (nk + 2 vectors).  A block takes chunks of E amplitudes a
// thread; per group of ARN_KB vectors a thread adds its 32 products and the warp reduces all
// 32 values at once by a transposing butterfly (31 FP64 shuffles instead of 5 for each value:
// one value at a time, the shuffles took as long as the loads -- 140 us a pass against 70 us
// for pass B at 2^20 complex128 amplitudes and 24 vectors), lane l ending with value l, which
// it adds to the warp's row in shared memory.  Blocks with blockIdx.y = g take every
// gridDim.y-th group: on registers with fewer chunks than the GPU has blocks, the groups are
// what fills it.
__device__ __forceinline__ double warp_transpose_sum(double (&v)[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) {
        const bool up = (lane & m) != 0;
#pragma unroll
        for (int i = 0; i < m; ++i) {
            const double send = up ? v[i] : v[i + m], keep = up ? v[i + m] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
        }
    }
    return v[0];  // value `lane`, summed over the warp
}

constexpr int LAG_E = 4;  // amplitudes per thread and chunk
// Blocks of pass A per SM.  Its 16 to 32 loads and 32 sums a thread take 202 registers: complex128
// (half the amplitudes in flight) streams at one block an SM.  Complex64 does the same arithmetic
// on half the bytes, conversions besides, and one block's eight warps do not cover it: 2^22
// amplitudes, 18 iterations 420 us a pass with one block and 176 with two on 128 registers (2^20
// 107 and 52; 208 and 67 with one value at a time).
template <typename R> constexpr int LAG_BLOCKS = sizeof(R) == 8 ? 1 : 2;
template <typename R>
__global__ void __launch_bounds__(ORTHO_THREADS, LAG_BLOCKS<R>)
k_arn_lagdots(const KState *ks, int j, const void *v0_, const unsigned char *basis, i64 D,
              const void *w_, double *part) {
    typedef typename cvec<R>::T C;
    if (ks->status != KS_RUNNING) return;
    constexpr int NW = ORTHO_THREADS / 32, E = LAG_E, KB = ARN_KB;
    constexpr int EL = sizeof(R) == 8 ? 2 : 4;  // amplitudes whose loads are in flight: 256 bytes a thread
    __shared__ double acc[NW][ARN_GROUPS][32];
    __shared__ double sa[NW][4];
    const bool has_vt = j >= 1;
    const int nk = has_vt ? j : 1, ngroups = (nk + KB - 1) / KB;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g0 = blockIdx.y, gs = gridDim.y;
    for (int g = g0; g < ngroups; g += gs) acc[warp][g][lane] = 0.0;
    const double st = has_vt ? ks->scale[j] : 0.0;
    const C *v0 = reinterpret_cast<const C *>(v0_);
    const C *bs = reinterpret_cast<const C *>(basis);
    const C *w = reinterpret_cast<const C *>(w_);
    const C *vt = has_vt ? bs + (i64)j * D : nullptr;
    double nw = 0.0, nv = 0.0, ar = 0.0, ai = 0.0;
    const i64 CH = (i64)ORTHO_THREADS * E;
    for (i64 c0 = (i64)blockIdx.x * CH; c0 < D; c0 += (i64)gridDim.x * CH) {
        double wr[E], wi[E], tr[E], ti[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const i64 x = c0 + tid + (i64)e * ORTHO_THREADS;
            wr[e] = wi[e] = tr[e] = ti[e] = 0.0;
            if (x < D) {
                const C a = w[x];
                wr[e] = double(a.x);
                wi[e] = double(a.y);
                if (has_vt) {
                    const C b = vt[x];
                    tr[e] = st * double(b.x);
                    ti[e] = st * double(b.y);
                }
            }
            if (g0 == 0) {
                nw += wr[e] * wr[e] + wi[e] * wi[e];
                nv += tr[e] * tr[e] + ti[e] * ti[e];
                ar += tr[e] * wr[e] + ti[e] * wi[e];
                ai += tr[e] * wi[e] - ti[e] * wr[e];
            }
        }
        for (int g = g0; g < ngroups; g += gs) {
            double v[4 * KB];
#pragma unroll
            for (int i = 0; i < 4 * KB; ++i) v[i] = 0.0;
#pragma unroll
            for (int h = 0; h < E; h += EL) {
                C a[KB][EL];
#pragma unroll
                for (int kb = 0; kb < KB; ++kb) {
                    const int k = g * KB + kb;
                    const C *vk = k == 0 ? v0 : bs + (i64)k * D;
#pragma unroll
                    for (int e = 0; e < EL; ++e) {
                        const i64 x = c0 + tid + (i64)(h + e) * ORTHO_THREADS;
                        a[kb][e] = (k < nk && x < D) ? vk[x] : cmake<C>(0.0, 0.0);
                    }
                }
#pragma unroll
                for (int kb = 0; kb < KB; ++kb)
#pragma unroll
                    for (int e = 0; e < EL; ++e) {
                        const double px = double(a[kb][e].x), py = double(a[kb][e].y);
                        v[4 * kb] += px * wr[h + e] + py * wi[h + e];
                        v[4 * kb + 1] += px * wi[h + e] - py * wr[h + e];
                        v[4 * kb + 2] += px * tr[h + e] + py * ti[h + e];
                        v[4 * kb + 3] += px * ti[h + e] - py * tr[h + e];
                    }
            }
            acc[warp][g][lane] += warp_transpose_sum(v);
        }
    }
    if (g0 == 0) {
        nw = warp_sum(nw);
        nv = warp_sum(nv);
        ar = warp_sum(ar);
        ai = warp_sum(ai);
        if (lane == 0) {
            sa[warp][0] = ar;
            sa[warp][1] = ai;
            sa[warp][2] = nw;
            sa[warp][3] = nv;
        }
    }
    __syncthreads();
    const size_t nb = gridDim.x;
    for (int g = g0 + gs * warp; g < ngroups; g += gs * NW) {  // one warp per group, lane = value
        const int k = g * KB + (lane >> 2);
        double t = 0.0;
#pragma unroll
        for (int u = 0; u < NW; ++u) t += acc[u][g][lane];
        if (k < nk) part[(size_t)(32 * g + lane) * nb + blockIdx.x] = ks->scale[k] * t;
    }
    if (g0 == 0 && tid < 4) {
        double t = 0.0;
        for (int u = 0; u < NW; ++u) t += sa[u][tid];
        part[(size_t)(ARN_A0 + tid) * nb + blockIdx.x] = t;
    }
}

// Pass B: w' = cw w - ct vt - sum cw1_l v_l (in place over w) and, for j >= 1, the
// corrected v_j = cv vt - sum cvj_l v_l (in place over vt, stored with scale 1); ||w'||^2.
// REVERSE: the chunks run from the last to the first, pass A's from the first to the last, so each
// pass begins on the part of the basis that the other left in the L2 (for a basis larger than that).
template <typename R, bool REVERSE, int E = 4, int KB = 4>
__global__ void __launch_bounds__(ORTHO_THREADS)
k_arn_lagupdate(const KState *ks, const ArnState *as, int j, const void *v0_, unsigned char *basis,
                i64 D, void *w_, double *part) {
    typedef typename cvec<R>::T C;
    if (ks->status != KS_RUNNING) return;
    constexpr int NW = ORTHO_THREADS / 32;
    __shared__ double2 c1[ARN_M], c2[ARN_M];
    __shared__ double snorm[NW];
    const bool has_vt = j >= 1;
    const int nk = has_vt ? j : 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int k = tid; k < nk; k += ORTHO_THREADS) {
        const double sk = ks->scale[k];
        c1[k] = make_double2(as->cw1[k].x * sk, as->cw1[k].y * sk);
        c2[k] = make_double2(as->cvj[k].x * sk, as->cvj[k].y * sk);
    }
    const double st = has_vt ? ks->scale[j] : 0.0;
    const double cw = as->cw, cv = as->cv * st;
    const double2 ct = make_double2(as->ct.x * st, as->ct.y * st);
    __syncthreads();
    const C *v0 = reinterpret_cast<const C *>(v0_);
    C *bs = reinterpret_cast<C *>(basis);
    C *w = reinterpret_cast<C *>(w_);
    C *vt = has_vt ? bs + (i64)j * D : nullptr;
    auto vk = [&](int k) -> const C * { return k == 0 ? v0 : bs + (i64)k * D; };
    double nacc = 0.0;
    const i64 CH = (i64)ORTHO_THREADS * E, nch = (D + CH - 1) / CH;
    for (i64 ch = blockIdx.x; ch < nch; ch += gridDim.x) {
        const i64 c0 = (REVERSE ? nch - 1 - ch : ch) * CH;
        double ur[E], ui[E], qr[E], qi[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const i64 x = c0 + tid + (i64)e * ORTHO_THREADS;
            ur[e] = ui[e] = qr[e] = qi[e] = 0.0;
            if (x < D) {
                const C a = w[x];
                ur[e] = cw * double(a.x);
                ui[e] = cw * double(a.y);
                if (has_vt) {
                    const C b = vt[x];
                    const double bx = double(b.x), by = double(b.y);
                    ur[e] -= ct.x * bx - ct.y * by;
                    ui[e] -= ct.x * by + ct.y * bx;
                    qr[e] = cv * bx;
                    qi[e] = cv * by;
                }
            }
        }
        int k = 0;
        for (; k < nk; k += KB) {
            C a[KB][E];
#pragma unroll
            for (int kb = 0; kb < KB; ++kb)
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const i64 x = c0 + tid + (i64)e * ORTHO_THREADS;
                    a[kb][e] = (k + kb < nk && x < D) ? vk(k + kb)[x] : cmake<C>(0.0, 0.0);
                }
#pragma unroll
            for (int kb = 0; kb < KB; ++kb) {
                if (k + kb >= nk) break;
                const double2 p1 = c1[k + kb], p2 = c2[k + kb];
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const double px = double(a[kb][e].x), py = double(a[kb][e].y);
                    ur[e] -= p1.x * px - p1.y * py;
                    ui[e] -= p1.x * py + p1.y * px;
                    qr[e] -= p2.x * px - p2.y * py;
                    qi[e] -= p2.x * py + p2.y * px;
                }
            }
        }
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const i64 x = c0 + tid + (i64)e * ORTHO_THREADS;
            if (x < D) {
                const C o = cmake<C>(ur[e], ui[e]);
                w[x] = o;
                nacc += double(o.x) * double(o.x) + double(o.y) * double(o.y);
                if (has_vt) vt[x] = cmake<C>(qr[e], qi[e]);
            }
        }
    }
    nacc = warp_sum(nacc);
    if (lane == 0) snorm[warp] = nacc;
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
        for (int u = 0; u < NW; ++u) t += snorm[u];
        part[(size_t)ARN_NORM * gridDim.x + blockIdx.x] = t;
    }
}

// Sum of value i of a pass over its nb blocks by one warp (lanes stride over the blocks,
// then a fixed shuffle tree: deterministic).  Result in every lane.
__device__ __forceinline__ double arn_sum_warp(const double *part, int nb, int i) {
    double t = 0.0;
#pragma unroll 4
    for (int b = threadIdx.x & 31; b < nb; b += 32) t += part[(size_t)i * nb + b];
    return warp_sum(t);
}

__device__ __forceinline__ double2 cmulc(double2 a, double2 b) {  // conj(a) b
    return make_double2(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}

// After pass A of iteration j: the lagged correction of v_j and of column j-1, column j of
// T, ||H v_j|| (krylov_exp.py:52), and pass B's coefficients (see the pass comments).  One
// block, latency-bound: one warp per partial sum and per row of T s, every sum over k by the
// lanes of a warp (2^20 amplitudes, 47 iterations: 50 us a stage before, with one thread
// walking T and the sums).
__global__ void __launch_bounds__(STAGE_THREADS)
k_arn_lagstage(KState *ks, ArnState *as, int j, const double *part, int nb) {
    if (ks->status != KS_RUNNING) return;
    __shared__ double2 zs[ARN_M], ss[ARN_M], hs[ARN_M], cc[ARN_M];
    __shared__ double sa[4];
    __shared__ double salpha;
    __shared__ int bad;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NWD = STAGE_THREADS / 32;
    const bool has_vt = j >= 1;
    const int nk = has_vt ? j : 1;
    if (tid == 0) bad = 0;
    for (int i = warp; i < 4 * nk + 4; i += NWD) {  // value 4 k + c, then the four of vt and w
        const double v = arn_sum_warp(part, nb, i < 4 * nk ? i : ARN_A0 + i - 4 * nk);
        if (lane) continue;
        if (i >= 4 * nk) {
            sa[i - 4 * nk] = v;
        } else if (i & 2) {
            (&ss[i >> 2].x)[i & 1] = has_vt ? v : 0.0;
        } else {
            (&zs[i >> 2].x)[i & 1] = v;
        }
    }
    __syncthreads();
    const double beta = has_vt ? ks->r[j - 1] : 0.0;
    if (warp == 0) {
        double alpha = 1.0;
        if (has_vt) {
            double s2 = 0.0;
            for (int k = lane; k < nk; k += 32) s2 += ss[k].x * ss[k].x + ss[k].y * ss[k].y;
            s2 = warp_sum(s2);
            const double a2 = sa[3] - s2;  // ||vt||^2 - |V^H vt|^2
            alpha = a2 > 0.0 ? sqrt(a2) : 0.0;
        }
        if (lane == 0) {
            if (!(alpha > 0.0) || !isfinite(alpha)) bad = 1;
            salpha = alpha;
        }
    } else if (has_vt) {  // column j-1: w'_{j-1} = beta (alpha v_j + V s)
        for (int l = tid - 32; l < j; l += STAGE_THREADS - 32) {
            double2 &t = as->T[l * ARN_M + (j - 1)];
            t.x += beta * ss[l].x;
            t.y += beta * ss[l].y;
        }
    }
    __syncthreads();
    const double alpha = salpha;
    if (has_vt && tid == 0) {
        as->T[j * ARN_M + (j - 1)] = make_double2(beta * alpha, 0.0);
        ks->r[j - 1] = beta * alpha;
    }
    if (has_vt && warp == 0) {  // <v_j, w> = (<vt, w> - s^H z) / alpha
        double2 p = make_double2(0.0, 0.0);
        for (int k = lane; k < nk; k += 32) {
            const double2 q = cmulc(ss[k], zs[k]);
            p.x += q.x;
            p.y += q.y;
        }
        p.x = warp_sum(p.x);
        p.y = warp_sum(p.y);
        if (lane == 0) zs[j] = make_double2((sa[0] - p.x) / alpha, (sa[1] - p.y) / alpha);
    }
    __syncthreads();
    // (T s)_l for l <= j over the columns k < j (Hessenberg rows: k >= l - 1), a warp per row
    for (int l = warp; l <= j; l += NWD) {
        double2 acc = make_double2(0.0, 0.0);
        if (has_vt)
            for (int k = (l > 0 ? l - 1 : 0) + lane; k < j; k += 32) {
                const double2 t = as->T[l * ARN_M + k], q = ss[k];
                acc.x += t.x * q.x - t.y * q.y;
                acc.y += t.x * q.y + t.y * q.x;
            }
        acc.x = warp_sum(acc.x);
        acc.y = warp_sum(acc.y);
        if (lane == 0) {
            hs[l] = acc;
            // h_l = (z_l - (T s)_l) / alpha
            const double2 h = make_double2((zs[l].x - acc.x) / alpha, (zs[l].y - acc.y) / alpha);
            if (!isfinite(h.x) || !isfinite(h.y)) bad = 1;
            cc[l] = make_double2(acc.x + alpha * h.x, acc.y + alpha * h.y);
            if (l == j) ks->a_re[j] = h.x;  // Re <v_j, (H - sigma) v_j>
            as->T[l * ARN_M + j] = h;
        }
    }
    __syncthreads();
    // pass B: w' = (w - V_j c) / alpha with v_j = (vt - V s) / alpha substituted
    for (int l = tid; l < nk; l += STAGE_THREADS) {
        const double2 sl = ss[l], cj = has_vt ? cc[j] : make_double2(0.0, 0.0);
        const double2 p = make_double2((cj.x * sl.x - cj.y * sl.y) / alpha, (cj.x * sl.y + cj.y * sl.x) / alpha);
        as->cw1[l] = has_vt ? make_double2((cc[l].x - p.x) / alpha, (cc[l].y - p.y) / alpha) : cc[l];
        as->cvj[l] = make_double2(sl.x / alpha, sl.y / alpha);
    }
    if (warp == NWD - 1) {
        // ||(H - sigma) v_j||^2 = ||w - V_j (T s)||^2 / alpha^2, then ||H v_j||
        double n2 = 0.0;
        for (int l = lane; l <= (has_vt ? j : 0); l += 32) {
            const double2 p = cmulc(hs[l], zs[l]);
            n2 += -2.0 * p.x + hs[l].x * hs[l].x + hs[l].y * hs[l].y;
        }
        n2 = (sa[2] + warp_sum(n2)) / (alpha * alpha);
        if (lane == 0) {
            as->cw = 1.0 / alpha;
            as->cv = 1.0 / alpha;
            as->ct = has_vt ? make_double2(cc[j].x / (alpha * alpha), cc[j].y / (alpha * alpha))
                            : make_double2(0.0, 0.0);
            const double sg = ks->shift;
            ks->hn[j] = sqrt(fmax(0.0, n2 + 2.0 * sg * ks->a_re[j] + sg * sg));
            if (bad || !isfinite(n2)) {
                ks->status = KS_NONFINITE;
                ks->iters = j + 1;
            }
        }
    }
}

// y = exp(A) e_0 for the M x M matrix A in shared memory (column-major A[c*M + r]).
// s substeps of sum_{k<=34} (A/s)^k / k! with ||A/s||_1 <= 4: truncation below
// 4^35/35! ~ 1e-19 relative per substep, terms at most 4^4/4! ~ 11 times the result (about
// one digit of cancellation).  Returns false when the norm is not finite or would need
// more than 2^20 substeps.  All threads of the block.
// A serial chain of 34 s matrix-vector products: TPR threads share a row, each with its NC
// entries in registers, and the terms alternate between two vectors in shared memory, one
// barrier a product.
template <int TPR, int NC>
__device__ __forceinline__ void arn_taylor(const double2 *A, int M, int s, double2 *y, double2 *t, double2 *tn) {
    const int tid = threadIdx.x, r = tid / TPR, q = tid % TPR;
    double2 a[NC];
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        const int c = q + i * TPR;
        a[i] = (r < M && c < M) ? A[c * M + r] : make_double2(0.0, 0.0);
    }
    double2 yr = make_double2(r == 0 ? 1.0 : 0.0, 0.0);  // y[r] in every thread of the row
    const double is = 1.0 / (double)s;
    for (int step = 0; step < s; ++step) {
        if (q == 0 && r < M) t[r] = yr;
        __syncthreads();
        for (int k = 1; k <= 34; ++k) {
            double2 acc = make_double2(0.0, 0.0);
#pragma unroll
            for (int i = 0; i < NC; ++i) {
                const int c = q + i * TPR;
                const double2 v = c < M ? t[c] : make_double2(0.0, 0.0);
                acc.x += a[i].x * v.x - a[i].y * v.y;
                acc.y += a[i].x * v.y + a[i].y * v.x;
            }
#pragma unroll
            for (int o = TPR >> 1; o > 0; o >>= 1) {  // TPR lanes of one warp
                acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
                acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
            }
            const double f = is / (double)k;
            acc.x *= f;
            acc.y *= f;
            yr.x += acc.x;
            yr.y += acc.y;
            if (q == 0 && r < M) tn[r] = acc;
            __syncthreads();
            double2 *tmp = t;
            t = tn;
            tn = tmp;
        }
    }
    if (q == 0 && r < M) y[r] = yr;
    __syncthreads();
}

__device__ bool arn_expm_col0(const double2 *A, int M, double2 *y, double2 *t, double2 *tn,
                              double *red) {
    const int tid = threadIdx.x;
    // ||A||_1: column sums
    double cs = 0.0;
    if (tid < M)
        for (int r = 0; r < M; ++r) cs += hypot(A[tid * M + r].x, A[tid * M + r].y);
    red[tid] = cs;
    __syncthreads();
    for (int o = DECIDE_THREADS / 2; o > 0; o >>= 1) {
        if (tid < o) red[tid] = fmax(red[tid], red[tid + o]);
        __syncthreads();
    }
    const double nrm = red[0];
    __syncthreads();
    if (!isfinite(nrm) || nrm > 4.0 * 1048576.0) return false;
    const int s = nrm > 4.0 ? (int)ceil(nrm / 4.0) : 1;
    static_assert(DECIDE_THREADS == 512 && ARN_M <= 128, "threads per row below");
    if (M <= 32) arn_taylor<16, 2>(A, M, s, y, t, tn);
    else if (M <= 64) arn_taylor<8, 8>(A, M, s, y, t, tn);
    else arn_taylor<4, (ARN_M + 3) / 4>(A, M, s, y, t, tn);
    return true;
}

// Extended matrix of iteration jj (krylov_exp.py:77-78) in my basis: A = -i dt T[:jj+2,
// :jj+1] plus A[jj+2][jj+1] = 1 (M = jj + 3); happy: A = -i dt T[:jj+1, :jj+1] (M = jj + 1).
__device__ void arn_build(const ArnState *as, int jj, double dt, double sigma, bool happy, double2 *A,
                          int *Mo) {
    const int M = happy ? jj + 1 : jj + 3;
    for (int i = threadIdx.x; i < M * M; i += DECIDE_THREADS) {
        const int c = i / M, r = i % M;
        double2 v = make_double2(0.0, 0.0);
        if (c <= jj && r <= c + 1 && r <= (happy ? jj : jj + 1)) {  // Hessenberg entries
            double2 h = as->T[r * ARN_M + c];
            if (r == c) h.x += sigma;  // T of H itself
            v = make_double2(dt * h.y, -dt * h.x);  // -i dt h
        }
        if (!happy && c == jj + 1 && r == jj + 2) v = make_double2(1.0, 0.0);
        A[i] = v;
    }
    *Mo = M;
    __syncthreads();
}

// Error estimate of iteration jj (krylov_exp.py:81-84); writes c[0..jj+1].  The estimate
// is NaN when both terms are zero (0 * 0 / 0, as in the reference, where NaN fails the
// convergence test); *fail is set when the exponential itself failed.
__device__ double arn_eval(KState *ks, const ArnState *as, int jj, double dt, double2 *A, double2 *y,
                           double2 *t, double2 *tn, double *red, bool *fail) {
    int M;
    arn_build(as, jj, dt, ks->shift, false, A, &M);
    if (!arn_expm_col0(A, M, y, t, tn, red)) {
        *fail = true;
        return nan("");
    }
    for (int k = threadIdx.x; k <= jj + 1; k += DECIDE_THREADS) {
        ks->c_re[k] = y[k].x;
        ks->c_im[k] = y[k].y;
    }
    const double err1 = hypot(y[jj + 1].x, y[jj + 1].y);
    const double err2 = hypot(y[jj + 2].x, y[jj + 2].y) * (fabs(dt) * ks->hn[jj]);
    __syncthreads();
    return err1 < err2 ? err1 : (err1 * err2 / (err1 - err2));
}

// y = exp(A) e_0 for a caller's dense complex M x M matrix (row-major, complex128, in
// global memory): one block, the Arnoldi decision's Taylor routine; *status = 0, or
// EMUSV_NONFINITE when the matrix norm is not finite or too large for the substeps.
__global__ void __launch_bounds__(DECIDE_THREADS)
k_dense_expm_col(int M, const double2 *a_rowmajor, double2 *x, int *status) {
    extern __shared__ __align__(16) unsigned char arn_smem[];
    double2 *A = reinterpret_cast<double2 *>(arn_smem);
    double2 *y = A + M * M;
    double2 *t = y + M;
    double2 *tn = t + M;
    double *red = reinterpret_cast<double *>(tn + M);  // [DECIDE_THREADS]
    for (int i = threadIdx.x; i < M * M; i += DECIDE_THREADS) {
        const int r = i / M, c = i % M;
        A[c * M + r] = a_rowmajor[i];
    }
    __syncthreads();
    const bool ok = arn_expm_col0(A, M, y, t, tn, red);
    for (int k = threadIdx.x; k < M; k += DECIDE_THREADS)
        x[k] = ok ? y[k] : make_double2(nan(""), nan(""));
    if (threadIdx.x == 0) *status = ok ? EMUSV_OK : EMUSV_NONFINITE;
}

__global__ void __launch_bounds__(DECIDE_THREADS)
k_arn_decide(KState *ks, ArnState *as, int j, const double *part, int nb, double dt, double exp_tol,
             double norm_tol, int poll, int first_poll, int maxdim) {
    if (ks->status != KS_RUNNING) return;
    extern __shared__ __align__(16) unsigned char arn_smem[];
    const int Mmax = maxdim + 2;
    double2 *A = reinterpret_cast<double2 *>(arn_smem);
    double2 *y = A + Mmax * Mmax;
    double2 *t = y + Mmax;
    double2 *tn = t + Mmax;
    double *red = reinterpret_cast<double *>(tn + Mmax);  // [DECIDE_THREADS]
    const int tid = threadIdx.x;
    if (ks->kerr) {  // a streaming kernel gave up on a bounded wait
        if (tid == 0) {
            ks->status = KS_TIMEOUT;
            ks->iters = j + 1;
        }
        return;
    }
    __shared__ double n2s;
    if (tid < 32) {
        const double v = arn_sum_warp(part, nb, ARN_NORM);
        if (tid == 0) n2s = v;
    }
    __syncthreads();
    const double r = sqrt(n2s);
    if (!isfinite(r)) {
        if (tid == 0) {
            ks->status = KS_NONFINITE;
            ks->iters = j + 1;
        }
        return;
    }
    if (tid == 0) {
        as->T[(j + 1) * ARN_M + j] = make_double2(r, 0.0);  // krylov_exp.py:61 (until corrected)
        ks->r[j] = r;
        ks->scale[j + 1] = 1.0 / r;
        if (j >= 1) ks->scale[j] = 1.0;  // pass B stored the corrected v_j normalised
    }
    __syncthreads();
    if (fabs(dt) * r < norm_tol) {  // happy breakdown (krylov_exp.py:63-71)
        int M;
        arn_build(as, j, dt, ks->shift, true, A, &M);
        const bool ok = arn_expm_col0(A, M, y, t, tn, red);
        for (int k = tid; k < M; k += DECIDE_THREADS) {
            ks->c_re[k] = y[k].x;
            ks->c_im[k] = y[k].y;
        }
        if (tid == 0) {
            ks->nvec = j + 1;
            ks->iters = j + 1;
            ks->status = ok ? KS_HAPPY : KS_NONFINITE;
        }
        return;
    }
    if (!poll) return;
    bool fail = false;
    double err = arn_eval(ks, as, j, dt, A, y, t, tn, red, &fail);
    int jc = j;
    // the first test also looks at the untested iterations, in order, when this one
    // converges or its estimate is NaN (both error terms underflowed: an earlier
    // iteration may have converged already)
    if ((err < exp_tol || err != err) && first_poll && j > 0 && !fail) {
        for (int jj = 0; jj < j; ++jj) {
            const double e = arn_eval(ks, as, jj, dt, A, y, t, tn, red, &fail);
            if (e < exp_tol) {
                err = e;
                jc = jj;
                break;
            }
        }
        if (jc == j) err = arn_eval(ks, as, j, dt, A, y, t, tn, red, &fail);
    }
    if (tid == 0) {
        ks->err = err;
        ks->nvec = jc + 2;
        ks->iters = jc + 1;
        if (fail)
            ks->status = KS_NONFINITE;
        else if (err < exp_tol)
            ks->status = KS_CONVERGED;
        else if (j + 1 >= maxdim)
            ks->status = KS_MAXDIM;
    }
}

static size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

static size_t arn_header_bytes() {
    return align_up(sizeof(KState), 256) + align_up(sizeof(ArnState), 256) +
           align_up(sizeof(double) * (size_t)sm_count() * 8 * ARN_PS, 256) +
           align_up(sizeof(double) * (size_t)sm_count() * 8 * NRED, 256);
}

static size_t decide_smem(int maxdim) {
    const size_t M = (size_t)maxdim + 2;
    return sizeof(double2) * (M * M + 3 * M) + sizeof(double) * DECIDE_THREADS;
}

// Grid of the Gram-Schmidt passes: never more blocks than chunks; *grid_out receives the
// number of blocks in x (the partial sums per value).  Pass A is a persistent grid (LAG_BLOCKS an
// SM); where that leaves SMs idle, the groups of basis vectors are spread over blocks in y.  Pass B
// runs backwards once the vectors of an iteration are more than the L2 holds (126 MB): 2^20
// complex128 amplitudes, 21 iterations 32.1 us a pass against 35.8 forwards; on a basis inside the
// L2 forwards is the faster one (2^18: 8.4 against 9.1, complex64 10.0 against 11.2).
constexpr i64 LAG_L2_BYTES = i64(100) << 20;
template <typename R>
static int launch_lagged(int pass, const KState *ks, const ArnState *as, int j, const void *v0,
                         unsigned char *basis, i64 D, void *w, double *part, cudaStream_t s,
                         int *grid_out) {
    constexpr int E = LAG_E;
    const i64 chunks = (D + (i64)ORTHO_THREADS * E - 1) / ((i64)ORTHO_THREADS * E);
    const i64 resident = (i64)sm_count() * LAG_BLOCKS<R>;
    i64 grid = pass == 0 ? resident : (i64)krylov_stream_grid(D);
    if (grid > chunks) grid = chunks;
    *grid_out = (int)grid;
    ProfScope ps_(PROF_ORTH, s);
    if (pass == 0) {
        const int groups = ((j >= 1 ? j : 1) + ARN_KB - 1) / ARN_KB;
        int gy = (int)(resident / grid);
        if (gy > groups) gy = groups;
        k_arn_lagdots<R><<<dim3((unsigned)grid, gy), ORTHO_THREADS, 0, s>>>(ks, j, v0, basis, D, w, part);
    } else {
        const bool reverse = (i64)(j + 2) * D * (i64)sizeof(typename cvec<R>::T) > LAG_L2_BYTES;
        auto *kern = reverse ? k_arn_lagupdate<R, true, E> : k_arn_lagupdate<R, false, E>;
        kern<<<(int)grid, ORTHO_THREADS, 0, s>>>(ks, as, j, v0, basis, D, w, part);
    }
    EMUSV_CHECK_LAUNCH();
    return EMUSV_OK;
}

}  // namespace emusv

using namespace emusv;

extern "C" {

static size_t dense_expm_smem(int m) {
    return sizeof(double2) * ((size_t)m * m + 3 * (size_t)m) + sizeof(double) * DECIDE_THREADS;
}

size_t emusv_dense_expm_scratch_bytes(int m) {
    if (m < 1 || m > ARN_M) return 0;
    return align_up(sizeof(double2) * (size_t)m * m, 256) + align_up(sizeof(double2) * m, 256) + 256;
}

int emusv_dense_expm_col(int m, const double *a, double *x_dev, void *scratch, size_t scratch_bytes,
                         void *stream) {
    if (m < 1 || m > ARN_M || !a || !x_dev || !scratch || scratch_bytes < emusv_dense_expm_scratch_bytes(m))
        return EMUSV_BAD_ARGUMENT;
    cudaStream_t s = as_stream(stream);
    unsigned char *p = reinterpret_cast<unsigned char *>(scratch);
    double2 *A = reinterpret_cast<double2 *>(p);
    int *status = reinterpret_cast<int *>(p + align_up(sizeof(double2) * (size_t)m * m, 256) +
                                          align_up(sizeof(double2) * m, 256));
    EMUSV_CHECK(cudaMemcpyAsync(A, a, sizeof(double2) * (size_t)m * m, cudaMemcpyHostToDevice, s));
    const size_t smem = dense_expm_smem(m);
    EMUSV_CHECK(cudaFuncSetAttribute(k_dense_expm_col, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    {
        ProfScope ps_(PROF_SMALL, s);
        k_dense_expm_col<<<1, DECIDE_THREADS, smem, s>>>(m, A, reinterpret_cast<double2 *>(x_dev), status);
    }
    EMUSV_CHECK_LAUNCH();
    int h = 0;
    EMUSV_CHECK(cudaMemcpyAsync(&h, status, sizeof(int), cudaMemcpyDeviceToHost, s));
    EMUSV_CHECK(cudaStreamSynchronize(s));  // the host matrix may be reused once this returns
    return h;
}

size_t emusv_arnoldi_workspace_bytes(int nqubits, int dtype, int basis_capacity) {
    if (nqubits < 1 || nqubits > EMUSV_MAX_QUBITS || basis_capacity < 0 ||
        (dtype != EMUSV_C128 && dtype != EMUSV_C64))
        return 0;
    const size_t es = dtype == EMUSV_C128 ? 16 : 8;
    return arn_header_bytes() + (size_t)(basis_capacity + 1) * (size_t(1) << nqubits) * es;
}

int emusv_arnoldi_step(int nqubits, int dtype, double dt, const double *omegas, const double *deltas,
                       const double *phis, const double *interaction, const double *noise,
                       const void *psi_in, void *psi_out, double exp_tolerance, double norm_tolerance,
                       int max_krylov_dim, int krylov_dim_hint, void *workspace,
                       size_t workspace_bytes, emusv_krylov_info *info, void *stream) {
    HamParams P;
    if (!make_params(nqubits, omegas, deltas, phis, interaction, &P) || !add_noise(noise, &P))
        return EMUSV_BAD_ARGUMENT;
    return arnoldi_run(P, nullptr, dtype, dt, psi_in, psi_out, exp_tolerance, norm_tolerance,
                       max_krylov_dim, krylov_dim_hint, workspace, workspace_bytes, info, stream);
}

}  // extern "C"

namespace emusv {

// The Arnoldi step for the operator of P (nqubits = P.n bits), plus, when J is given, the
// Lindblad jump term i sum_q K_q added to every product (lindblad.cu).
int arnoldi_run(const HamParams &P, const LindbladJumps *J, int dtype, double dt, const void *psi_in,
                void *psi_out, double exp_tolerance, double norm_tolerance, int max_krylov_dim,
                int krylov_dim_hint, void *workspace, size_t workspace_bytes,
                emusv_krylov_info *info, void *stream) {
    const int nqubits = P.n;
    if (!psi_in || !psi_out || !workspace || (dtype != EMUSV_C128 && dtype != EMUSV_C64) ||
        max_krylov_dim < 1 || max_krylov_dim > ARN_KMAX || !isfinite(dt))
        return EMUSV_BAD_ARGUMENT;
    if ((reinterpret_cast<uintptr_t>(workspace) & 255) || (reinterpret_cast<uintptr_t>(psi_in) & 15) ||
        (reinterpret_cast<uintptr_t>(psi_out) & 15))
        return EMUSV_BAD_ARGUMENT;
    if (workspace_bytes < arn_header_bytes()) return EMUSV_WORKSPACE_TOO_SMALL;
    cudaStream_t s = as_stream(stream);
    const i64 D = i64(1) << nqubits;
    const size_t es = dtype == EMUSV_C128 ? 16 : 8;
    unsigned char *p = reinterpret_cast<unsigned char *>(workspace);
    KState *ks = reinterpret_cast<KState *>(p);
    p += align_up(sizeof(KState), 256);
    ArnState *as = reinterpret_cast<ArnState *>(p);
    p += align_up(sizeof(ArnState), 256);
    double *part = reinterpret_cast<double *>(p);
    p += align_up(sizeof(double) * (size_t)sm_count() * 8 * ARN_PS, 256);
    double *part_n = reinterpret_cast<double *>(p);
    p += align_up(sizeof(double) * (size_t)sm_count() * 8 * NRED, 256);
    unsigned char *basis = p;  // slot 0: partial sums of the multi-pass H*psi; slots 1..
    const int capacity = (int)((workspace_bytes - arn_header_bytes()) / (D * es)) - 1;
    if (capacity < 1) return EMUSV_WORKSPACE_TOO_SMALL;
    auto stored = [&](int k) -> const void * {
        return k == 0 ? psi_in : (const void *)(basis + (size_t)k * D * es);
    };
    const size_t dsmem = decide_smem(max_krylov_dim);
    EMUSV_CHECK(cudaFuncSetAttribute(k_arn_decide, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dsmem));
    int st = krylov_begin(dtype, psi_in, D, ks, part_n, true, s);
    if (st) return st;

    int status = KS_RUNNING;
    bool polled = false;
    for (int j = 0; j < max_krylov_dim; ++j) {
        if (j + 1 > capacity) {
            if ((st = read_status(ks, s, &status))) return st;
            if (status == KS_RUNNING) return EMUSV_WORKSPACE_TOO_SMALL;
            break;
        }
        void *w = const_cast<void *>(stored(j + 1));
        HpsiArgs A = {};
        A.u = stored(j);
        A.su_dev = &ks->scale[j];
        A.out = w;
        A.tile_bits = hpsi_tile_bits(nqubits);
        A.gate = &ks->status;
        A.err = &ks->kerr;
        A.part_buf = basis;
        A.eshift = &ks->shift;
        if ((st = launch_hpsi(dtype, HP_STORE, P, A, 0, s, nullptr))) return st;
        if (J && (st = launch_lindblad_jumps(dtype, *J, stored(j), &ks->scale[j], w, &ks->status, s)))
            return st;
        int og = 0;
        for (int pass = 0; pass < 2; ++pass) {
            st = dtype == EMUSV_C128
                     ? launch_lagged<double>(pass, ks, as, j, psi_in, basis, D, w, part, s, &og)
                     : launch_lagged<float>(pass, ks, as, j, psi_in, basis, D, w, part, s, &og);
            if (st) return st;
            if (pass == 0) {
                ProfScope ps_(PROF_SMALL, s);
                k_arn_lagstage<<<1, STAGE_THREADS, 0, s>>>(ks, as, j, part, og);
                EMUSV_CHECK_LAUNCH();
            }
        }
        const bool poll = (j + 1 >= krylov_dim_hint) || (j + 1 >= max_krylov_dim);
        {
            ProfScope ps_(PROF_SMALL, s);
            k_arn_decide<<<1, DECIDE_THREADS, dsmem, s>>>(ks, as, j, part, og, dt, exp_tolerance,
                                                          norm_tolerance, poll ? 1 : 0,
                                                          (poll && !polled) ? 1 : 0, max_krylov_dim);
            EMUSV_CHECK_LAUNCH();
        }
        if (poll) {
            polled = true;
            if ((st = read_status(ks, s, &status))) return st;
            if (status != KS_RUNNING) break;
        }
    }
    if (status == KS_RUNNING)
        if ((st = read_status(ks, s, &status))) return st;
    if (status == KS_TIMEOUT) {
        if (info) memset(info, 0, sizeof(*info));
        return EMUSV_TIMEOUT;
    }
    if (status == KS_NONFINITE || status == KS_RUNNING) {
        if (info) memset(info, 0, sizeof(*info));
        return EMUSV_NONFINITE;
    }
    if ((st = krylov_combine(dtype, ks, psi_in, basis, D, psi_out, part_n, s))) return st;
    if (info) {
        KHead h;
        if ((st = read_heads(&ks, 1, s, &h))) return st;
        fill_info(h, h.iters > 0 ? h.iters - 1 : 0, info);  // every vector but the first
    }
    return status == KS_MAXDIM ? EMUSV_NOT_CONVERGED : EMUSV_OK;
}

}  // namespace emusv
