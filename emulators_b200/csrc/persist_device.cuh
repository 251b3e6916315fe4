// Device code of the runs that stay on chip: the exchange of sums between a job's CTAs and the
// convergence decisions (see persist.cuh) of the single steps (persist.cu), and the records of
// value and epoch, which the batches' gangs (batch.cu) use too.
#pragma once

#include "persist.cuh"
#include "tridiag_real.cuh"

namespace emusv {

// ------------------------------------------------------------------ records in global memory
__device__ __forceinline__ void rec_put(PRec *r, double v, unsigned long long e) {
    asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}"
                 ::"l"(r), "l"(__double_as_longlong(v)), "l"(e) : "memory");
}
template <bool ACQUIRE = false>
__device__ __forceinline__ PRec rec_get(const PRec *r) {
    long long v;
    unsigned long long e;
    if (ACQUIRE)
        asm volatile("{\n .reg .b128 t;\n ld.acquire.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
                     : "=l"(v), "=l"(e) : "l"(r) : "memory");
    else
        asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
                     : "=l"(v), "=l"(e) : "l"(r) : "memory");
    PRec o;
    o.v = __longlong_as_double(v);
    o.e = e;
    return o;
}
constexpr unsigned long long PSTOP = 1ull << 63;  // epoch flag: the run was decided

// Waits until the record carries the epoch; false on a timeout.
template <bool ACQUIRE = false>
__device__ __forceinline__ bool rec_wait(const PRec *r, unsigned long long e, PRec *o, long long limit) {
    *o = rec_get<ACQUIRE>(r);
    if ((o->e & ~PSTOP) == e) return true;
    const long long t0 = clock64();
    for (unsigned i = 1;; ++i) {
        *o = rec_get<ACQUIRE>(r);
        if ((o->e & ~PSTOP) == e) return true;
        if ((i & 255u) == 0 && clock64() - t0 > limit) return false;
    }
}

// ------------------------------------------------------------------ cluster helpers
__device__ __forceinline__ uint32_t sm_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t cl_addr(const void *p, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(sm_addr(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ float2 cl_ld(uint32_t a, float2) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ double2 cl_ld(uint32_t a, double2) {
    double2 v;
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void cl_st(uint32_t a, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void cl_st_rel(uint32_t a, int v) {
    asm volatile("st.release.cluster.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ int cl_ld_acq(uint32_t a) {
    int v;
    asm volatile("ld.acquire.cluster.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void mbar_init_count(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\nfence.mbarrier_init.release.cluster;"
                 ::"r"(sm_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void cl_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool cl_wait(uint64_t *bar, uint32_t parity, long long limit) {
    const long long t0 = clock64();
    for (unsigned i = 1;; ++i) {
        uint32_t ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
                     " selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(ok) : "r"(sm_addr(bar)), "r"(parity) : "memory");
        if (ok) return true;
        if ((i & 255u) == 0 && clock64() - t0 > limit) return false;
    }
}
__device__ __forceinline__ void cl_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// ------------------------------------------------------------------ shared state of a CTA
template <int CT> struct PShared {
    double red[2][CT / 32][3];      // the warps' sums, alternating between exchanges
    double xs[2][3][1 << PCL_BITS]; // the cluster's CTAs' sums of phases A and B
    double part[3];                 // the job's sums of the last exchange
    double up_re[MAXQ], up_im[MAXQ], field[MAXQ];
    double U[MAXQ * MAXQ];
    // the run's scalars, every CTA's own copy
    double ar[KMAX], ai[KMAX], r[KMAX], hn2[KMAX], scale[KMAX + 2];
    double2 coef[KMAX + 2];
    int flag[KMAX];
    int result[KMAX];               // iteration j: 1 goes on, 2 ends the run (in CTA 0 of a
                                    // cluster job, in the deciding CTA of a grid job)
    uint64_t bar;
    volatile int ready;             // iterations whose scalars are here
    volatile int done;              // the run's status + 1 once it is decided
    volatile int dead;              // a wait of this CTA ran out
    int lost;                       // a wait for the job's sums ran out (set by the warps that wait,
                                    // read by the compute warps after the exchange's barrier)
    int verdict;                    // `done` as the compute warps act on it, 0 after a timeout
    int fin[2];
    double sigma;
};

template <int CT> __device__ __forceinline__ void compute_sync() {  // the compute warps only
    asm volatile("bar.sync 1, %0;" ::"n"(CT) : "memory");
}

// The sums of v[0..2] over the job's compute threads, in every thread, in a fixed order; a
// barrier of the job (ordering global stores before it for grid jobs when PUBLISH).  PH 0:
// phase A, 1: phase B.  *stop: CTA 0's flag.  False, in every thread of the CTA alike, on a timeout.
template <int CT, bool CL, int PH, bool PUBLISH>
__device__ __forceinline__ bool p_exchange(PShared<CT> &sh, double (&v)[3], PExchange *X, unsigned long long e, int r,
                                           int gbits, uint32_t &parity, bool stop_in, bool *stop, long long wait) {
    constexpr int NW = CT / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, G = 1 << gbits;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int k = 0; k < 3; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    }
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) sh.red[PH][warp][k] = v[k];
    }
    if (gbits == 0 && threadIdx.x == 0) sh.fin[PH] = stop_in;
    compute_sync<CT>();
    auto block_total = [&](int k) {
        double t[NW];
#pragma unroll
        for (int w = 0; w < NW; ++w) t[w] = sh.red[PH][w][k];
#pragma unroll
        for (int o = NW / 2; o > 0; o >>= 1)
#pragma unroll
            for (int w = 0; w < o; ++w) t[w] += t[w + o];
        return t[0];
    };
    if (gbits == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) v[k] = block_total(k);
        *stop = sh.fin[PH] != 0;
        return true;
    }
    if constexpr (CL) {
        // every CTA receives every CTA's sums (and CTA 0's flag), then the phase completes; one warp
        // per sum waits for it
        const int fin = __shfl_sync(0xffffffffu, (int)stop_in, 0);
        if (warp < 3) {
            if (lane < G) {
                cl_st(cl_addr(&sh.xs[PH][warp][r], lane), block_total(warp));
                if (warp == 0 && r == 0)
                    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cl_addr(&sh.fin[PH], lane)), "r"(fin)
                                 : "memory");
                cl_arrive(cl_addr(&sh.bar, lane));
            }
            if (!cl_wait(&sh.bar, parity, wait)) sh.lost = 1;
            double t = 0.0;
            for (int g = 0; g < G; g += 2) t += sh.xs[PH][warp][g] + sh.xs[PH][warp][g + 1];
            if (lane == 0) sh.part[warp] = t;
        }
    } else {
        // clusters of PGC CTAs first: their sums meet in the cluster's first CTA, which writes
        // the cluster's records; every CTA reads all clusters' records, one a lane
        constexpr int PGC = 1 << PGC_BITS;
        static_assert((PMAXG >> PGC_BITS) <= 32, "a warp reads the records of one sum");
        PRec(*recs)[PMAXG >> PGC_BITS] = PH == 0 ? X->a : X->b;
        if (warp < 3) {
            if (lane == 0) {
                cl_st(cl_addr(&sh.xs[PH][warp][r & (PGC - 1)], 0), block_total(warp));
                cl_arrive(cl_addr(&sh.bar, 0));
            }
            bool ok = true;
            if ((r & (PGC - 1)) == 0 && lane == 0) {
                ok = cl_wait(&sh.bar, parity, wait);
                double t = 0.0;
#pragma unroll
                for (int g = 0; g < PGC; ++g) t += sh.xs[PH][warp][g];
                if (PUBLISH) __threadfence();  // the cluster's stores before its record
                if (ok) rec_put(&recs[warp][r >> PGC_BITS], t, e | (stop_in ? PSTOP : 0ull));
            }
            __syncwarp();
            double t = 0.0;
            if (lane < (G >> PGC_BITS)) {
                PRec o;
                ok = rec_wait<PUBLISH>(&recs[warp][lane], e, &o, wait) && ok;
                t = o.v;
                if (warp == 0 && lane == 0) sh.fin[PH] = (o.e & PSTOP) != 0;
            }
            t = warp_sum(t);
            if (lane == 0) sh.part[warp] = t;
            if (!ok) sh.lost = 1;
        }
    }
    parity ^= 1u;
    compute_sync<CT>();
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] = sh.part[k];
    *stop = sh.fin[PH] != 0;
    return sh.lost == 0;
}

// ------------------------------------------------------------------ decisions
// What the deciding warps need of a run.
struct PRun {
    KState *ks;
    PExchange *x;               // grid jobs
    unsigned long long epoch;
    int gbits, limit, maxdim;   // see PArgs
    double dt, exp_tol;
    long long wait;             // clock cycles a wait lasts at most
};

// Is the run decided?  (cluster jobs: every CTA's `done`; grid jobs: the verdict record)
template <int CT, bool CL>
__device__ __forceinline__ bool p_decided(PShared<CT> &sh, const PExchange *X, unsigned long long epoch) {
    if (sh.done || sh.dead) return true;
    if constexpr (!CL) {
        const PRec v = rec_get(&X->verdict);
        if (v.e == epoch) {
            sh.done = (int)v.v + 1;
            return true;
        }
    }
    return false;
}

// Announces the run's status to the job's CTAs (one lane; the state's arrays are written).
template <int CT, bool CL>
__device__ __forceinline__ void p_announce(PShared<CT> &sh, PExchange *X, unsigned long long epoch, int G, int status) {
    __threadfence();
    if constexpr (CL) {
        for (int g = 0; g < G; ++g) cl_st_rel(cl_addr((const void *)&sh.done, g), status + 1);
    } else {
        rec_put(&X->verdict, (double)status, epoch);
        sh.done = status + 1;
    }
}

// Conclusion of iteration j (krylov_exp.py:63-96) by one warp; NE: the smallest register
// layout that holds the extended matrix's rows.
template <int NE, int CT, bool CL>
__device__ __noinline__ void p_conclude(const PRun &A, PShared<CT> &sh, int j) {
    const int lane = threadIdx.x & 31, G = 1 << A.gbits;
    KState *ks = A.ks;
    const int m = j + 1, flag = sh.flag[j];
    const bool ext = flag == KD_OK;
    double2 y[NE];
    double err = 0.0;
    if (flag != KD_NONFINITE) {
        double d[NE], l[NE], u[NE];  // rows of T (b_{k+1} = r_k), the extension rows
#pragma unroll
        for (int e = 0; e < NE; ++e) {
            const int k = lane * NE + e;
            d[e] = k < m ? sh.ar[k] + sh.sigma : 0.0;  // a_k of H (the run uses H - sigma)
            l[e] = k > 0 && k < m ? sh.r[k - 1] : 0.0;
            u[e] = k + 1 < m ? sh.r[k] : 0.0;
        }
        if (ext) extend_rows<NE>(m, sh.r[j], A.dt, l);
        cheb_expm_real<NE>(d, l, u, -1, 0.0, 0, A.dt, ext ? m + 2 : m, y, &sh.done);
        if (__any_sync(0xffffffffu, sh.done)) return;
        if (ext) err = expokit_error<NE>(y, m, A.dt, sqrt(fmax(0.0, sh.hn2[j])));
    }
    int st = KS_RUNNING, nvec = j + 2;
    if (flag == KD_NONFINITE) {
        st = KS_NONFINITE;
    } else if (flag == KD_HAPPY) {
        st = KS_HAPPY;
        nvec = m;
    } else if (err < A.exp_tol) {
        st = KS_CONVERGED;
    } else if (j + 1 >= A.maxdim) {
        st = KS_MAXDIM;
    }
    const bool ends = st != KS_RUNNING || j + 1 >= A.limit;
    if (lane == 0) {
        if constexpr (CL) cl_st_rel(cl_addr(&sh.result[j], 0), ends ? 2 : 1);
        else *(volatile int *)&sh.result[j] = ends ? 2 : 1;
    }
    if (!ends) return;
    // every earlier iteration must be known to go on
    const long long t0 = clock64();
    for (int k = lane; k < j; k += 32) {
        for (;;) {
            int res;
            if constexpr (CL) res = cl_ld_acq(cl_addr(&sh.result[k], 0));
            else res = *(volatile int *)&sh.result[k];
            if (res == 2) st = -1;  // an earlier iteration ended the run
            if (res) break;
            if (p_decided<CT, CL>(sh, A.x, A.epoch) || clock64() - t0 > A.wait) {
                st = -1;
                break;
            }
        }
        if (st < 0) break;
    }
    if (!__all_sync(0xffffffffu, st >= 0)) return;
    // the run ends here (KS_RUNNING: the basis has no room for another vector)
    if (st != KS_NONFINITE) {
#pragma unroll
        for (int e = 0; e < NE; ++e) {
            const int k = lane * NE + e;
            if (k < nvec) {  // c[m] = x1 multiplies v_{j+1} (krylov_exp.py:88-90)
                ks->c_re[k] = y[e].x;
                ks->c_im[k] = y[e].y;
            }
        }
    }
    for (int k = lane; k <= j; k += 32) {  // the run's scalars, as the adjoint reads them
        const double b = k > 0 ? sh.r[k - 1] : 0.0;
        ks->a_re[k] = sh.ar[k];
        ks->a_im[k] = sh.ai[k];
        ks->b_re[k] = b;
        ks->b_im[k] = 0.0;
        ks->r[k] = sh.r[k];
        ks->hn[k] = sqrt(fmax(0.0, sh.hn2[k]));
    }
    for (int k = lane; k <= j + 1; k += 32) ks->scale[k] = sh.scale[k];
    __syncwarp();
    if (lane == 0) {
        ks->status = st;
        ks->iters = j + 1;
        ks->nvec = nvec;
        ks->err = err;
        p_announce<CT, CL>(sh, A.x, A.epoch, G, st);
    }
    __syncwarp();
}

// The deciding CTA of a grid job: its first warp brings the iterations' scalars from CTA 0's
// records into shared memory.
template <int CT>
__device__ void p_collect(const PRun &A, PShared<CT> &sh) {
    const int lane = threadIdx.x & 31;
    const unsigned long long e0 = A.epoch + 1;
    for (int j = -1; j < A.limit; ++j) {
        PRec q;
        q.v = 0.0;
        bool got = true;
        if (lane < (j < 0 ? 2 : 5)) {
            const PRec *rec = j < 0 ? &A.x->start[lane] : &A.x->iter[j][lane];
            const unsigned long long e = j < 0 ? A.epoch : e0 + j;
            const long long t0 = clock64();
            for (;;) {
                q = rec_get(rec);
                if (q.e == e) break;
                if (sh.done || sh.dead || clock64() - t0 > A.wait) {
                    got = false;
                    break;
                }
            }
        }
        if (!__all_sync(0xffffffffu, got)) {
            if (lane == 0 && !sh.done) {  // a wait ran out
                sh.dead = 1;
                atomicExch(&A.ks->kerr, (int)EMUSV_TIMEOUT);
            }
            return;
        }
        if (j < 0) {
            if (lane == 0) sh.sigma = q.v;
            if (lane == 1) sh.scale[0] = q.v;
        } else {
            if (lane == 0) sh.ar[j] = q.v;
            if (lane == 1) sh.ai[j] = q.v;
            if (lane == 2) {
                sh.r[j] = q.v;
                sh.scale[j + 1] = 1.0 / q.v;
            }
            if (lane == 3) sh.hn2[j] = q.v;
            if (lane == 4) sh.flag[j] = (int)q.v;
        }
        __syncwarp();
        __threadfence_block();
        if (lane == 0) sh.ready = j + 1;
        __syncwarp();
    }
}

// The deciding warps of a CTA: iterations q, q + Q, ... of the job's Q deciding warps.
template <int CT, bool CL>
__device__ void p_decider(const PRun &A, PShared<CT> &sh, int q, int Q) {
    const int lane = threadIdx.x & 31;
    for (int j = q; j < A.limit; j += Q) {
        int go = 1;
        if (lane == 0) {
            const long long t0 = clock64();
            while (sh.ready <= j) {
                if (p_decided<CT, CL>(sh, A.x, A.epoch)) {
                    go = 0;
                    break;
                }
                if (clock64() - t0 > A.wait) {
                    sh.dead = 1;
                    go = 0;
                    break;
                }
                __nanosleep(40);
            }
        }
        if (!__shfl_sync(0xffffffffu, go, 0)) return;
        __threadfence_block();
        const int M = j + 3;
        if (M <= 32) p_conclude<1, CT, CL>(A, sh, j);
        else if (M <= 64) p_conclude<2, CT, CL>(A, sh, j);
        else if (M <= 96) p_conclude<3, CT, CL>(A, sh, j);
        else p_conclude<(KMAX + 2 + 31) / 32, CT, CL>(A, sh, j);
    }
}

}  // namespace emusv
