// Single-launch Lanczos runs (see persist.cuh).
#include <atomic>
#include <chrono>

#include "persist_device.cuh"
#include "profile.cuh"

namespace emusv {

// ------------------------------------------------------------------ the run
// Cluster jobs: ND deciding warps follow the CT compute threads of every CTA.  Grid jobs (ND =
// 0): one more CTA decides, so that the compute threads keep 128 registers each.
template <typename R, bool REALC, int NA, int CT, int ND, bool CL>
__global__ void __launch_bounds__(CT + 32 * ND, 1) k_lanczos_persist(const __grid_constant__ PArgs A) {
    typedef typename cvec<R>::T C;
    constexpr int LB = CT == 256 ? 8 : 9;  // thread bits
    constexpr int RB = NA == 1 ? 0 : NA == 2 ? 1 : NA == 4 ? 2 : NA == 8 ? 3 : 4;
    constexpr int GB = CL ? PCL_BITS : PMAXG_BITS;  // CTA bits at most
    constexpr int CA = NA < (sizeof(R) == 8 ? 2 : 4) ? NA : (sizeof(R) == 8 ? 2 : 4);  // amplitudes at a time
    extern __shared__ __align__(16) unsigned char psm[];
    __shared__ PShared<CT> sh;
    const int S = NA * CT;                  // slots of the arrays below (at least 2^tb)
    C *us = reinterpret_cast<C *>(psm);     // this CTA's part of v_j (unscaled)
    C *vps = us + S;                        // cluster jobs: its part of v_{j-1}
    double *dg = reinterpret_cast<double *>(CL ? vps + S : us + S);  // diagonal minus sigma
    const int G = 1 << A.gbits;
    // grid jobs: the compute CTAs of all jobs, then one cluster whose CTA k decides job k
    const bool decides = !CL && (int)blockIdx.x >= A.njobs << A.gbits;
    const int r = blockIdx.x & (G - 1);
    const int jb = decides ? (r < A.njobs ? r : 0) : blockIdx.x >> A.gbits;
    const PJob &J = A.job[jb];
    const HamParams &P = A.P;
    const int n = P.n, tb = A.tbits, nlow = tb < LB ? tb : LB;
    const int tid = threadIdx.x;
    KState *ks = J.ks;
    PExchange *X = J.x;
    if (tid == 0) {
        sh.ready = 0;
        sh.done = 0;
        sh.dead = 0;
        sh.lost = 0;
        mbar_init_count(&sh.bar, CL ? 3 * G : 3 << PGC_BITS);
        // sigma from the previous finished run (read before anyone overwrites the state)
        double sg = 0.0;
        if (J.energy_shift && (ks->status == KS_CONVERGED || ks->status == KS_HAPPY) && ks->iters > 0) {
            sg = ks->shift + ks->a_re[0];
            if (!isfinite(sg) || fabs(sg) > 1e12) sg = 0.0;
        }
        sh.sigma = sg;
    }
    for (int k = tid; k < n; k += blockDim.x) {
        sh.up_re[k] = P.up_re[k];
        sh.up_im[k] = P.up_im[k];
        sh.field[k] = P.field[k];
    }
    for (int k = tid; k < n * MAXQ; k += blockDim.x) sh.U[k] = P.U[k];
    for (int k = tid; k < KMAX; k += blockDim.x) sh.result[k] = 0;
    __syncthreads();
    cl_sync_all();  // mbarriers and flags are set before a sibling touches them
    const PRun run = {ks, X, A.epoch, A.gbits, A.limit, A.maxdim, A.dt, A.exp_tol, A.wait};
    if constexpr (CL) {
        if (tid >= CT) {
            p_decider<CT, CL>(run, sh, r + (((tid - CT) >> 5) << A.gbits), ND << A.gbits);
            cl_sync_all();
            return;
        }
    } else if (decides) {
        if (r < A.njobs) {
            if (tid < 32) p_collect<CT>(run, sh);
            else p_decider<CT, CL>(run, sh, (tid >> 5) - 1, CT / 32 - 1);
        }
        cl_sync_all();
        return;
    }
    const i64 D = i64(1) << n, base = (i64)r << tb;
    const bool on = tid < (1 << nlow);  // fewer amplitudes than threads on the smallest registers
    const double sigma = sh.sigma;
    const C zero = cmake<C>(0.0, 0.0);
    const C *u0 = reinterpret_cast<const C *>(J.v0) + base;
    C *bs = reinterpret_cast<C *>(J.basis) + base;  // slot k at bs + k * D
    double acc[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const int l = tid + a * CT;
        const C v = on ? u0[l] : zero;
        us[l] = v;
        if (CL) vps[l] = zero;
        acc[0] += double(v.x) * double(v.x) + double(v.y) * double(v.y);
    }
    {  // diagonal: thread and CTA bits, then the register bits with their crosses
        const unsigned x = (unsigned)base + tid;
        double e = -sigma, f[RB > 0 ? RB : 1];
#pragma unroll
        for (int k = 0; k < RB; ++k) f[k] = sh.field[LB + k];
        for (unsigned m = x; m; m &= m - 1) {
            const int p = __ffs(m) - 1;
            const double *Up = sh.U + p * MAXQ;
            e += sh.field[p];
            for (unsigned q = m & (m - 1); q; q &= q - 1) e += Up[__ffs(q) - 1];
#pragma unroll
            for (int k = 0; k < RB; ++k) f[k] += Up[LB + k];
        }
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            double t = e;
#pragma unroll
            for (int k = 0; k < RB; ++k)
                if ((a >> k) & 1) {
                    t += f[k];
#pragma unroll
                    for (int k2 = k + 1; k2 < RB; ++k2)
                        if ((a >> k2) & 1) t += sh.U[(LB + k) * MAXQ + LB + k2];
                }
            dg[tid + a * CT] = t;
        }
    }
    uint32_t parity = 0;
    bool stop = false;
    // failure-path test: this CTA's sums stay out, so its siblings' waits for them run out, and in
    // its end its own wait for the verdict
    const bool mute = A.withhold && jb == 0 && r == G - 1;
    // every CTA has read the previous state once this exchange is complete
    bool ok = mute || p_exchange<CT, CL, 1, false>(sh, acc, X, A.epoch, r, A.gbits, parity, false, &stop, A.wait);
    const double s0 = sqrt(acc[0]);  // krylov_exp.py:43
    const bool fine = isfinite(s0) && s0 > 0.0;
    double sj = 1.0 / s0, sp = 0.0, b = 0.0, vvr = 0.0, vvi = 0.0;
    if (tid == 0) {
        sh.scale[0] = sj;
        if (r == 0) {
            ks->s0 = s0;
            ks->shift = sigma;
            ks->outnorm2 = 0.0;
            ks->kerr = 0;
            ks->status = KS_RUNNING;
            if (!CL) {
                rec_put(&X->start[0], sigma, A.epoch);
                rec_put(&X->start[1], sj, A.epoch);
            }
        }
        if (!fine && !mute) {  // decided as iteration 0
            sh.ar[0] = sh.ai[0] = sh.r[0] = sh.hn2[0] = 0.0;
            sh.scale[1] = 0.0;
            sh.flag[0] = KD_NONFINITE;
            __threadfence_block();
            sh.ready = 1;
        }
    }
    const unsigned long long e0 = A.epoch + 1;
    if (!CL && !fine && !mute && r == 0 && tid < 5) rec_put(&X->iter[0][tid], tid == 4 ? (double)KD_NONFINITE : 0.0, e0);
    for (int j = 0; fine && ok && !mute && !stop && j < A.limit; ++j) {
        // grid jobs: CTA 0 looks whether the run is decided, meanwhile
        PRec vd;
        vd.e = 0;
        if (!CL && r == 0 && tid == CT - 1) vd = rec_get(&X->verdict);
        const C *uj = j == 0 ? reinterpret_cast<const C *>(J.v0) : reinterpret_cast<const C *>(J.basis) + (i64)j * D;
        // ---------------- A: h = (H - sigma) v_j
        double hr[NA], hi[NA];
        acc[0] = acc[1] = acc[2] = 0.0;
#pragma unroll
        for (int a0 = 0; a0 < NA; a0 += CA) {
            // the CTA bits: partners in the other CTAs' parts, in flight during the rest
            C q[GB][CA];
#pragma unroll
            for (int k = 0; k < GB; ++k) {
                if (k >= A.gbits) {
#pragma unroll
                    for (int a = 0; a < CA; ++a) q[k][a] = zero;
                    continue;
                }
                if constexpr (CL) {
                    const uint32_t pa = cl_addr(us, (uint32_t)(r ^ (1 << k))) + (uint32_t)((tid + a0 * CT) * sizeof(C));
#pragma unroll
                    for (int a = 0; a < CA; ++a) q[k][a] = cl_ld(pa + (uint32_t)(a * CT * sizeof(C)), zero);
                } else {
                    const C *pp = uj + (base ^ (i64(1) << (tb + k))) + tid + a0 * CT;
#pragma unroll
                    for (int a = 0; a < CA; ++a) q[k][a] = __ldcg(pp + a * CT);
                }
            }
            R ar[CA], ai[CA];
#pragma unroll
            for (int a = 0; a < CA; ++a) ar[a] = ai[a] = R(0);
            auto flip = [&](int a, R cr, R ci, const C &w) {
                if (REALC) {
                    ar[a] = fmar(cr, w.x, ar[a]);
                    ai[a] = fmar(cr, w.y, ai[a]);
                } else {
                    ar[a] = fmar(cr, w.x, fmar(-ci, w.y, ar[a]));
                    ai[a] = fmar(cr, w.y, fmar(ci, w.x, ai[a]));
                }
            };
            // thread and register bits: partners in shared memory
#pragma unroll
            for (int k = 0; k < LB; ++k) {
                if (k >= nlow) break;
                const R cr = R(sh.up_re[k]);
                R ci = REALC ? R(0) : R(sh.up_im[k]);
                if (!((tid >> k) & 1)) ci = -ci;
#pragma unroll
                for (int a = 0; a < CA; ++a) flip(a, cr, ci, us[(tid ^ (1 << k)) + (a0 + a) * CT]);
            }
#pragma unroll
            for (int k = 0; k < RB; ++k) {
                const R cr = R(sh.up_re[LB + k]), ci = REALC ? R(0) : R(sh.up_im[LB + k]);
#pragma unroll
                for (int a = 0; a < CA; ++a)
                    flip(a, cr, ((a0 + a) >> k) & 1 ? ci : -ci, us[tid + ((a0 + a) ^ (1 << k)) * CT]);
            }
#pragma unroll
            for (int k = 0; k < GB; ++k) {
                if (k >= A.gbits) break;
                const R cr = R(sh.up_re[tb + k]);
                R ci = REALC ? R(0) : R(sh.up_im[tb + k]);
                if (!((r >> k) & 1)) ci = -ci;
#pragma unroll
                for (int a = 0; a < CA; ++a) flip(a, cr, ci, q[k][a]);
            }
#pragma unroll
            for (int a = 0; a < CA; ++a) {
                const C v = us[tid + (a0 + a) * CT];
                const double d = dg[tid + (a0 + a) * CT], vx = double(v.x), vy = double(v.y);
                const double x = on ? sj * (double(ar[a]) + d * vx) : 0.0;
                const double y = on ? sj * (double(ai[a]) + d * vy) : 0.0;
                hr[a0 + a] = x;
                hi[a0 + a] = y;
                acc[0] += vx * x + vy * y;
                acc[1] += vx * y - vy * x;
                acc[2] += x * x + y * y;
            }
        }
        acc[0] *= sj;
        acc[1] *= sj;
        constexpr bool PRE = !CL && NA <= 4;  // v_{j-1} loaded ahead of the exchange
        const C *up = j == 1 ? u0 : bs + (i64)(j - 1) * D;
        C vp[PRE ? NA : 1];
        if (PRE) {
#pragma unroll
            for (int a = 0; a < NA; ++a) vp[a] = j > 0 ? __ldcg(up + tid + a * CT) : zero;
        }
        bool dummy;
        ok = p_exchange<CT, CL, 0, false>(sh, acc, X, e0 + 2 * j, r, A.gbits, parity, false, &dummy, A.wait);
        if (!ok) break;
        // ---------------- B: w = h - a v_j - b v_{j-1}
        const double are = acc[0] - b * vvr, aim = acc[1] - b * vvi;
        const double car = are * sj, cai = aim * sj, cb = b * sp;
        const double hn2 = acc[2] + 2.0 * sigma * acc[0] + sigma * sigma;
        acc[0] = acc[1] = acc[2] = 0.0;
        C *w = bs + (i64)(j + 1) * D;
        constexpr int BA = NA < 4 ? NA : 4;
#pragma unroll
        for (int a0 = 0; a0 < NA; a0 += BA) {
            C p[BA];
#pragma unroll
            for (int a = 0; a < BA; ++a) {
                if (CL) p[a] = vps[tid + (a0 + a) * CT];
                else if (PRE) p[a] = vp[PRE ? a0 + a : 0];
                else p[a] = j > 0 ? __ldcg(up + tid + (a0 + a) * CT) : zero;
            }
#pragma unroll
            for (int a = 0; a < BA; ++a) {
                const int l = tid + (a0 + a) * CT;
                const C v = us[l];
                const double vx = double(v.x), vy = double(v.y);
                const double wr = hr[a0 + a] - (car * vx - cai * vy) - cb * double(p[a].x);
                const double wi = hi[a0 + a] - (car * vy + cai * vx) - cb * double(p[a].y);
                const C o = on ? cmake<C>(wr, wi) : zero;
                if (on) w[l] = o;
                us[l] = o;  // phase A's readers are past the exchange
                if (CL) vps[l] = v;
                const double ox = double(o.x), oy = double(o.y);
                acc[0] += ox * ox + oy * oy;
                acc[1] += vx * ox + vy * oy;  // <v_j, w>
                acc[2] += vx * oy - vy * ox;
            }
        }
        acc[1] *= sj;
        acc[2] *= sj;
        if (!CL && r == 0 && tid == CT - 1 && vd.e == A.epoch) sh.done = (int)vd.v + 1;
        ok = p_exchange<CT, CL, 1, true>(sh, acc, X, e0 + 2 * j + 1, r, A.gbits, parity,
                                         r == 0 && tid == 0 && sh.done, &stop, A.wait);
        if (!ok) break;
        const double rj = sqrt(acc[0]), inv = 1.0 / rj;
        int flag = KD_OK;
        if (!isfinite(rj) || !isfinite(hn2) || !isfinite(are) || !isfinite(aim)) flag = KD_NONFINITE;
        else if (fabs(A.dt) * rj < A.norm_tol) flag = KD_HAPPY;
        if (!CL && r == 0 && tid < 5)
            rec_put(&X->iter[j][tid],
                    tid == 0 ? are : tid == 1 ? aim : tid == 2 ? rj : tid == 3 ? hn2 : (double)flag, e0 + j);
        if (tid == 0) {
            sh.scale[j + 1] = inv;
            if (CL) {
                sh.ar[j] = are;
                sh.ai[j] = aim;
                sh.r[j] = rj;
                sh.hn2[j] = hn2;
                sh.flag[j] = flag;
                __threadfence_block();
                sh.ready = j + 1;
            }
        }
        sp = sj;
        sj = inv;
        b = rj;
        vvr = acc[1] * inv;  // <v_{j+1}, v_j> = conj(<v_j, w>) / ||w||
        vvi = -acc[2] * inv;
        if (flag != KD_OK) break;
    }
    // ---------------- the verdict and the combination out = s0 sum_k c_k v_k
    if (tid == 0) {
        const long long t0 = clock64();
        while (ok && !p_decided<CT, CL>(sh, X, A.epoch))
            if (clock64() - t0 > A.wait) ok = false;
        sh.verdict = ok ? sh.done : 0;  // not decided: a deciding warp gave up
        if (!sh.verdict) {
            sh.dead = 1;
            atomicExch(&ks->kerr, (int)EMUSV_TIMEOUT);
        }
        __threadfence();
    }
    compute_sync<CT>();
    const int st = sh.verdict - 1;
    if (J.out && (st == KS_CONVERGED || st == KS_HAPPY || st == KS_MAXDIM)) {
        const int nv = __ldcg(&ks->nvec);
        for (int k = tid; k < nv; k += CT) {
            const double f = s0 * sh.scale[k];
            sh.coef[k] = make_double2(f * __ldcg(&ks->c_re[k]), f * __ldcg(&ks->c_im[k]));
        }
        compute_sync<CT>();
        acc[0] = acc[1] = acc[2] = 0.0;
        C *out = reinterpret_cast<C *>(J.out) + base;
        constexpr int OA = NA < 4 ? NA : 4, KU = 16 / OA;  // 16 loads in flight
#pragma unroll
        for (int a0 = 0; a0 < NA; a0 += OA) {
            if (!on) break;
            double re[OA], im[OA];
#pragma unroll
            for (int a = 0; a < OA; ++a) {
                const C v = u0[tid + (a0 + a) * CT];
                re[a] = sh.coef[0].x * double(v.x) - sh.coef[0].y * double(v.y);
                im[a] = sh.coef[0].x * double(v.y) + sh.coef[0].y * double(v.x);
            }
            for (int k = 1; k < nv; k += KU) {
                C q[KU][OA];
#pragma unroll
                for (int u = 0; u < KU; ++u)
#pragma unroll
                    for (int a = 0; a < OA; ++a)
                        q[u][a] = k + u < nv ? __ldcs(bs + (i64)(k + u) * D + tid + (a0 + a) * CT) : zero;
#pragma unroll
                for (int u = 0; u < KU; ++u) {
                    if (k + u >= nv) break;
                    const double2 c = sh.coef[k + u];
#pragma unroll
                    for (int a = 0; a < OA; ++a) {
                        re[a] += c.x * double(q[u][a].x) - c.y * double(q[u][a].y);
                        im[a] += c.x * double(q[u][a].y) + c.y * double(q[u][a].x);
                    }
                }
            }
#pragma unroll
            for (int a = 0; a < OA; ++a) {
                const C o = cmake<C>(re[a], im[a]);
                out[tid + (a0 + a) * CT] = o;
                acc[0] += double(o.x) * double(o.x) + double(o.y) * double(o.y);
            }
        }
        ok = p_exchange<CT, CL, 0, false>(sh, acc, X, A.epoch + 4 * KMAX - 1, r, A.gbits, parity, false, &stop,
                                           A.wait);
        if (r == 0 && tid == 0) {
            ks->outnorm2 = acc[0];
            if (!ok) atomicExch(&ks->kerr, (int)EMUSV_TIMEOUT);
        }
    }
    cl_sync_all();  // no CTA leaves while a sibling may still read its shared memory
}

// ------------------------------------------------------------------ host side
struct PShape {
    bool cluster;
    int gbits, tbits, na_bits;
};
// Cluster jobs hold v_j, v_{j-1} and the diagonal in shared memory; 256 compute threads and
// four deciding warps.  Grid jobs read v_{j-1} from the basis; 512 compute threads, a deciding
// CTA.
constexpr int CCT = 256, CND = 4, GCT = 512;
static size_t persist_smem(const PShape &s, int dtype) {
    const int lb = s.cluster ? 8 : 9;
    const size_t es = dtype == EMUSV_C128 ? 16 : 8, slots = size_t(1) << (s.tbits > lb ? s.tbits : lb);
    return slots * (es * (s.cluster ? 2 : 1) + sizeof(double));
}
// One CTA up to 11 qubits (11 qubits on four CTAs: 76 us a step of 16 iterations, on one 82 with
// three SMs left to others); clusters to 15 (16 qubits on a cluster of 16: 14.6 us an
// iteration, on the grid 10: the partners' amplitudes come through distributed shared memory
// at about 18 bytes a clock); the grid to 20, where v_j and the diagonal still fit (20 qubits
// complex128: 1340 us against 1909 for the streaming passes).
static PShape persist_shape(int n, int njobs) {
    PShape s;
    s.cluster = n <= 15;
    if (s.cluster) s.gbits = n <= 11 ? 0 : (n == 12 ? 3 : PCL_BITS);
    else s.gbits = njobs == 2 ? PMAXG_BITS - 1 : PMAXG_BITS;  // side by side on half the CTAs each
    s.tbits = n - s.gbits;
    const int lb = s.cluster ? 8 : 9;
    s.na_bits = s.tbits > lb ? s.tbits - lb : 0;
    return s;
}

template <typename R, bool REALC, int NA>
static void *pick_na(bool cluster) {
    if constexpr (NA < 16) {  // a cluster job's CTA has at most 2^11 amplitudes
        if (cluster) return reinterpret_cast<void *>(k_lanczos_persist<R, REALC, NA, CCT, CND, true>);
    }
    return reinterpret_cast<void *>(k_lanczos_persist<R, REALC, NA, GCT, 0, false>);
}
template <typename R, bool REALC>
static void *pick(const PShape &s) {
    switch (s.na_bits) {
    case 0: return pick_na<R, REALC, 1>(s.cluster);
    case 1: return pick_na<R, REALC, 2>(s.cluster);
    case 2: return pick_na<R, REALC, 4>(s.cluster);
    case 3: return pick_na<R, REALC, 8>(s.cluster);
    default: return pick_na<R, REALC, 16>(s.cluster);
    }
}
static void *pick(const PShape &s, int dtype, bool realc) {
    return dtype == EMUSV_C128 ? (realc ? pick<double, true>(s) : pick<double, false>(s))
                               : (realc ? pick<float, true>(s) : pick<float, false>(s));
}
static cudaError_t set_attributes(void *kern, const PShape &s, size_t smem) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess || !s.cluster || s.gbits <= 3) return e;
    return cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}
static void fill_config(cudaLaunchConfig_t *cfg, cudaLaunchAttribute (&attr)[2], const PShape &s, int njobs,
                        size_t smem) {
    *cfg = {};
    cfg->gridDim = dim3((njobs << s.gbits) + (s.cluster ? 0 : 1 << PGC_BITS));
    cfg->blockDim = dim3(s.cluster ? CCT + 32 * CND : GCT);
    cfg->dynamicSmemBytes = smem;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1u << (s.cluster ? s.gbits : PGC_BITS);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeCooperative;  // grid jobs wait for one another's CTAs:
    attr[1].val.cooperative = 1;                  // all resident at once
    cfg->attrs = attr;
    cfg->numAttrs = s.cluster ? 1 : 2;
}
// Does the current device hold a launch of this shape: the cluster of a cluster job (up to 16 CTAs
// in one cluster's reach, which a partition of a GPU may not have), every cluster of a grid job at
// once?  The launched kernel with its own shared memory is what is asked about, once per device.
static bool shape_fits(const PShape &s, int n, int dtype, bool realc, int njobs) {
    const size_t smem = persist_smem(s, dtype);
    if (n > PMAXN || s.na_bits > 4 || smem > 200 * 1024) return false;
    if (s.cluster && s.gbits == 0) return true;
    static std::atomic<signed char> known[64][2][2][2][PMAXN + 1];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    std::atomic<signed char> &k = known[dev][dtype == EMUSV_C128][realc][njobs - 1][n];
    if (!k.load()) {
        void *kern = pick(s, dtype, realc);
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[2];
        fill_config(&cfg, attr, s, njobs, smem);
        cfg.numAttrs = 1;  // the cluster's size
        int clusters = 0;
        if (set_attributes(kern, s, smem) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess) {
            cudaGetLastError();
            clusters = 0;
        }
        k.store(clusters >= (s.cluster ? 1 : (njobs << s.gbits >> PGC_BITS) + 1) ? 1 : 2);
    }
    return k.load() == 1;
}

// Test switch of the calling thread (emusv_krylov_set_streaming).
static thread_local int tl_streaming = 0;
void persist_set_streaming(int on) { tl_streaming = on ? 1 : 0; }

bool lz_applies(int dtype, int n);
// A register that no launch of this kind holds takes the streaming passes (lanczos_run), which run
// from 12 qubits on; up to 11 a run is one CTA.
bool persist_applies(const HamParams &P, int dtype) {
    if (P.n < 1 || (dtype != EMUSV_C128 && dtype != EMUSV_C64)) return false;
    if (tl_streaming && lz_applies(dtype, P.n)) return false;
    return shape_fits(persist_shape(P.n, 1), P.n, dtype, P.real_coef != 0, 1);
}
size_t persist_exchange_bytes() { return (sizeof(PExchange) + 255) / 256 * 256; }

// Failure-path test switch of the calling thread (emusv_krylov_set_wait_test).
static thread_local long long tl_wait = PWAIT_LIMIT;
static thread_local int tl_withhold = 0;
void persist_set_wait_test(long long wait_cycles, int withhold) {
    tl_wait = wait_cycles > 0 ? wait_cycles : PWAIT_LIMIT;
    tl_withhold = withhold ? 1 : 0;
}

// Epochs of a launch: 4 KMAX consecutive values that no other launch uses.
static unsigned long long next_epoch() {
    static std::atomic<unsigned long long> next{
        ((unsigned long long)std::chrono::steady_clock::now().time_since_epoch().count() << 10) & ~(1ull << 63)};
    return next.fetch_add(4 * KMAX) & ~(1ull << 63);
}

int persist_launch(const HamParams &P, int dtype, double dt, const PJob *jobs, int njobs, int capacity,
                   double exp_tol, double norm_tol, int maxdim, cudaStream_t s) {
    PShape sh = persist_shape(P.n, njobs);
    int together = njobs;
    const bool realc = P.real_coef != 0;
    if (njobs > 1 && !shape_fits(sh, P.n, dtype, realc, njobs)) {  // in turn
        sh = persist_shape(P.n, 1);
        together = 1;
    }
    PArgs A;
    A.P = P;
    A.njobs = together;
    A.gbits = sh.gbits;
    A.tbits = sh.tbits;
    A.limit = maxdim < capacity ? maxdim : capacity;
    A.maxdim = maxdim;
    A.dt = dt;
    A.exp_tol = exp_tol;
    A.norm_tol = norm_tol;
    A.wait = tl_wait;
    A.withhold = tl_withhold;
    const size_t smem = persist_smem(sh, dtype);
    void *kern = pick(sh, dtype, realc);
    EMUSV_CHECK(set_attributes(kern, sh, smem));
    for (int j0 = 0; j0 < njobs; j0 += together) {
        for (int j = 0; j < together; ++j) A.job[j] = jobs[j0 + j];
        A.epoch = next_epoch();
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[2];
        fill_config(&cfg, attr, sh, together, smem);
        cfg.stream = s;
        void *args[] = {(void *)&A};
        ProfScope ps_(PROF_HPSI, s);
        EMUSV_CHECK(cudaLaunchKernelExC(&cfg, kern, args));
    }
    return EMUSV_OK;
}

}  // namespace emusv
