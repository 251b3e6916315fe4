// Exponentials of the small tridiagonal matrices in real arithmetic: the decisions of the
// single-launch runs (persist_device.cuh) and the adjoint's block exponentials.
#pragma once

#include "krylov_device.cuh"

namespace emusv {

template <int NE>
__device__ __forceinline__ double reg_pick(const double (&v)[NE], int k) {  // entry k, in every lane
    const int owner = k / NE, e = k - owner * NE;
    double r = v[0];
#pragma unroll
    for (int q = 1; q < NE; ++q)
        if (q == e) r = v[q];
    return __shfl_sync(0xffffffffu, r, owner);
}

// One warp, y = exp(-i dt T) e_col for a real M x M matrix T that is tridiagonal up to one
// coupling entry T[0][cpl] = cplv (cpl < 0: none) and whose eigenvalues lie inside its
// Gershgorin interval [c - R, c + R]; rows in the lanes (d diagonal, l below, u above, zero
// outside the matrix).  With X = (T - c)/R and z = |dt| R
//   exp(-i dt T) = e^{-i dt c} [J_0(z) + 2 sum_{k>=1} (-i sgn dt)^k J_k(z) T_k(X)],
// summed by Clenshaw's recurrence from the top term down while Miller's backward recurrence
// produces the Bessel values in the same order (normalised at the end by J_0 + 2 sum J_2k =
// 1).  T is real, so the real and the imaginary part (the even and the odd terms) are two
// independent real recurrences: a serial chain of two shuffles and three fused operations a
// term.  z + 10 z^(1/3) + 12 terms leave a tail below 1e-17 up to z = 300, 3e-17 at 1000 and 1.4e-16
// at 3000 (a basis of at most 127 vectors converges for z of about a hundred); Miller's recurrence
// starts eight terms above.  Kept real for the chain's length, which is what a single step waits for at its
// end: a step of 10 qubits takes 196 us with it and 235 with the complex rows of cheb_expm (the
// rounding-level imaginary part of the diagonal in them, 1.1 z + 40 terms), which stay where a
// decision is hidden behind other registers or a long iteration.  dt = 0: e_col.
// `abandon`: when given and set, the result is no longer wanted and y is left undefined
// (looked at every eighth term).
template <int NE>
static __device__ void cheb_expm_real(const double (&d)[NE], const double (&l)[NE], const double (&u)[NE], int cpl,
                                 double cplv, int col, double dt, int M, double2 (&y)[NE],
                                 const volatile int *abandon = nullptr) {
    const int lane = threadIdx.x & 31;
    if (dt == 0.0) {  // (a coupling entry of 1/dt is left out: what it leads to is multiplied by dt)
#pragma unroll
        for (int e = 0; e < NE; ++e) y[e] = make_double2(lane * NE + e == col ? 1.0 : 0.0, 0.0);
        return;
    }
    double lo = 1e300, hi = -1e300;
#pragma unroll
    for (int e = 0; e < NE; ++e) {
        const int k = lane * NE + e;
        if (k < M) {
            double rad = fabs(l[e]) + fabs(u[e]);
            if (cpl >= 0 && k == 0) rad += fabs(cplv);
            lo = fmin(lo, d[e] - rad);
            hi = fmax(hi, d[e] + rad);
        }
    }
    lo = -warp_max(-lo);
    hi = warp_max(hi);
    const double c = 0.5 * (lo + hi);
    // radius at least 1/|dt| (z >= 1): keeps X bounded when T's own spread is tiny, and
    // Miller's recurrence (factors 2k/z) far from overflow
    const double R = fmax(0.5 * (hi - lo), 1.0 / fabs(dt));
    const double z = fabs(dt) * R, iR = 1.0 / R;
    double xd[NE], xl[NE], xu[NE];
#pragma unroll
    for (int e = 0; e < NE; ++e) {
        xd[e] = lane * NE + e < M ? (d[e] - c) * iR : 0.0;
        xl[e] = l[e] * iR;
        xu[e] = u[e] * iR;
    }
    const double xc = cplv * iR;
    const bool first = lane == 0, last = lane == 31;
    auto xmul = [&](const double (&v)[NE], double (&out)[NE]) {  // X v
        double prev = __shfl_up_sync(0xffffffffu, v[NE - 1], 1);
        double next = __shfl_down_sync(0xffffffffu, v[0], 1);
        if (first) prev = 0.0;
        if (last) next = 0.0;
        const double cp = cpl >= 0 ? reg_pick(v, cpl) : 0.0;
#pragma unroll
        for (int e = 0; e < NE; ++e) {
            double o = fma(xl[e], e > 0 ? v[e - 1] : prev, fma(xd[e], v[e], xu[e] * (e < NE - 1 ? v[e + 1] : next)));
            if (cpl >= 0 && first && e == 0) o = fma(xc, cp, o);
            out[e] = o;
        }
    };
    const int N = (int)ceil(z + 10.0 * cbrt(z)) + 12;  // terms kept
    const int K = N + 8;                               // Miller's start
    const double twoz = 2.0 / z, sgn = dt >= 0.0 ? 1.0 : -1.0;
    double r1[NE], r2[NE], i1[NE], i2[NE];  // b_{k+1}, b_{k+2}: real and imaginary parts
#pragma unroll
    for (int e = 0; e < NE; ++e) r1[e] = r2[e] = i1[e] = i2[e] = 0.0;
    double jk1 = 0.0, jk = 1e-280, S = 0.0;  // J~_{k+1}, J~_k, normalisation sum
    double kd = K;                           // k
    for (int k = K; k >= 1; --k, kd -= 1.0) {
        // the whole warp or none of it: another warp may set the word between two lanes' loads
        if (abandon && (k & 7) == 0 && __any_sync(0xffffffffu, *abandon)) return;
        if ((k & 1) == 0) S += 2.0 * jk;
        if (k <= N) {  // b_k = 2 (-i sgn)^k J~_k e_col + 2 X b_{k+1} - b_{k+2}
            double xr[NE], xi[NE];
            xmul(r1, xr);
            xmul(i1, xi);
            const double ck = (k & 2) ? -2.0 * jk : 2.0 * jk;  // (-i)^k = 1, -i, -1, i
            const double cr = (k & 1) ? 0.0 : ck, ci = (k & 1) ? -sgn * ck : 0.0;
#pragma unroll
            for (int e = 0; e < NE; ++e) {
                const bool at = lane * NE + e == col;
                const double nr = fma(2.0, xr[e], (at ? cr : 0.0) - r2[e]);
                const double ni = fma(2.0, xi[e], (at ? ci : 0.0) - i2[e]);
                r2[e] = r1[e];
                r1[e] = nr;
                i2[e] = i1[e];
                i1[e] = ni;
            }
        }
        // J~_{k-1} = (2k / z) J~_k - J~_{k+1}
        const double jm = (twoz * kd) * jk - jk1;
        jk1 = jk;
        jk = jm;
        if (fabs(jk) > 1e250) {  // rescale everything linear in the J~
            const double g = 1e-250;
            jk *= g;
            jk1 *= g;
            S *= g;
#pragma unroll
            for (int e = 0; e < NE; ++e) {
                r1[e] *= g;
                r2[e] *= g;
                i1[e] *= g;
                i2[e] *= g;
            }
        }
    }
    // now jk = J~_0, b1 = b_1, b2 = b_2:  sum = J~_0 e_col + X b_1 - b_2
    S += jk;
    double xr[NE], xi[NE], es, ec;
    xmul(r1, xr);
    xmul(i1, xi);
    sincos(-dt * c, &es, &ec);
    const double inv = 1.0 / S;
#pragma unroll
    for (int e = 0; e < NE; ++e) {
        const double vr = (xr[e] - r2[e] + (lane * NE + e == col ? jk : 0.0)) * inv, vi = (xi[e] - i2[e]) * inv;
        y[e] = make_double2(ec * vr - es * vi, ec * vi + es * vr);
    }
}

// The two extension rows of the matrix [[A, 0, 0], [l e_jj^T, 0, 0], [0, 1, 0]] (A = -i dt T of
// size m, l = -i dt r): in units of T, the entry r and -- the last component taken times -i,
// which leaves its modulus -- the real entry 1/dt.
template <int NE>
__device__ __forceinline__ void extend_rows(int m, double r, double dt, double (&l)[NE]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int e = 0; e < NE; ++e) {
        const int k = lane * NE + e;
        if (k == m) l[e] = r;
        if (k == m + 1) l[e] = 1.0 / dt;
    }
}

// The Expokit error estimate (krylov_exp.py:81-84) from the extension entries y[m], y[m + 1].
template <int NE>
__device__ __forceinline__ double expokit_error(const double2 (&y)[NE], int m, double dt, double hn) {
    const double2 x1 = reg_pick(y, m), x2 = reg_pick(y, m + 1);
    const double err1 = hypot(x1.x, x1.y);
    const double err2 = hypot(x2.x, x2.y) * (fabs(dt) * hn);
    return err1 < err2 ? err1 : (err1 * err2 / (err1 - err2));
}

}  // namespace emusv
