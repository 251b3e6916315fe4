// Pair sums over bit positions: S_PQ = sum_x w(x) x_P x_Q (P <= Q, S_PP the single sums) of
// real or complex weights w over the 2^n bitstrings, in one pass over the weights.
//
// An index is split into [chunk bits | H loop bits | 8 thread bits]: a block takes a chunk of
// 2^(8+H) consecutive weights, thread t the weights whose low 8 bits are t.  Only the loop
// bits vary within a thread, so it accumulates the total, one sum per loop bit and one per
// pair of loop bits in registers (about 6 FP64 additions a weight); the thread bits are
// constant per thread and enter once per chunk, when the block reduces its 256 threads'
// sums under bit masks; the chunk bits are constant per block and enter once per launch,
// when k_pair_finish adds the chunks' sums (one warp per pair, chunk-contiguous rows).
// Bound by reading the weights: n = 22 complex128 (64 MB) 1832 + 153 us before (a shuffle and
// n predicated additions per weight and row, one block adding all partial rows).
#pragma once

#include "common.cuh"

namespace emusv {

constexpr int PS_TB = 8;               // thread bits (256 threads)
constexpr int PS_MAXH = 6;             // loop bits at most
constexpr int PS_T0 = 1 + PS_TB + PS_TB * (PS_TB - 1) / 2;  // sums of the plain totals: 37

// Loop bits for n qubits: none until 2^9 chunks exist (a few blocks per SM), then up to
// PS_MAXH, which spreads the block reduction over 64 weights per thread.
__host__ __device__ inline int ps_loop_bits(int n) {
    const int h = n - PS_TB - 9;
    return h < 0 ? 0 : (h > PS_MAXH ? PS_MAXH : h);
}
__host__ __device__ inline int ps_values(int H) { return PS_T0 + 9 * H + H * (H - 1) / 2; }
__host__ inline i64 ps_chunks(int n) {
    const int b = n - PS_TB - ps_loop_bits(n);
    return b > 0 ? i64(1) << b : 1;
}
// doubles of partial sums: [value][component][chunk]
__host__ inline size_t ps_partials(int n, int nc) {
    return (size_t)ps_values(ps_loop_bits(n)) * nc * (size_t)ps_chunks(n);
}

// Index of pair a < b among m items.
__host__ __device__ inline int ps_pair(int a, int b, int m) { return a * (2 * m - a - 1) / 2 + (b - a - 1); }

// Value index and chunk mask of the pair of bit positions P <= Q.
__device__ inline int ps_locate(int P, int Q, int H, i64 *mask) {
    *mask = 0;
    const int lim = PS_TB + H;
    if (Q >= lim) *mask |= i64(1) << (Q - lim);
    if (P >= lim) *mask |= i64(1) << (P - lim);
    const bool qin = Q < lim, pin = P < lim;
    if (!pin) return 0;
    if (!qin || P == Q)  // one bit inside the chunk
        return P < PS_TB ? 1 + P : PS_T0 + 9 * (P - PS_TB);
    if (Q < PS_TB) return 9 + ps_pair(P, Q, PS_TB);
    if (P < PS_TB) return PS_T0 + 9 * (Q - PS_TB) + 1 + P;
    return PS_T0 + 9 * H + ps_pair(P - PS_TB, Q - PS_TB, H);
}

// Partial sums of every chunk.  F: device functor, w = f(x) fills NC doubles (x < 2^n).
// PAIRS false: only the totals and the single sums.
template <int NC, int H, bool PAIRS, typename F>
__global__ void __launch_bounds__(1 << PS_TB) k_pair_sums(const F f, int n, i64 nchunks, double *part) {
    constexpr int NT = 1 << PS_TB, NWP = NT / 32;
    constexpr int HI = H < 3 ? H : 3, NI = 1 << HI, HO = H - HI, NO = 1 << HO;
    constexpr int NHH = H * (H - 1) / 2;
    __shared__ double rows[(1 + H) * NC][NT];
    __shared__ double hhw[NHH * NC > 0 ? NHH * NC : 1][NWP];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const i64 D = i64(1) << n;
    for (i64 c = blockIdx.x; c < nchunks; c += gridDim.x) {
        double R[NC], S[H > 0 ? H : 1][NC], HH[NHH > 0 ? NHH : 1][NC];
#pragma unroll
        for (int k = 0; k < NC; ++k) {
            R[k] = 0.0;
#pragma unroll
            for (int q = 0; q < H; ++q) S[q][k] = 0.0;
#pragma unroll
            for (int q = 0; q < NHH; ++q) HH[q][k] = 0.0;
        }
        const i64 x0 = (c << (PS_TB + H)) + tid;
#pragma unroll(HO > 0 ? 2 : 1)
        for (int ko = 0; ko < NO; ++ko) {
            double w[NI][NC];
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const i64 x = x0 + ((i64)(ko * NI + i) << PS_TB);
                if (x < D) {
                    f(x, w[i]);
                } else {
#pragma unroll
                    for (int k = 0; k < NC; ++k) w[i][k] = 0.0;
                }
            }
#pragma unroll
            for (int k = 0; k < NC; ++k) {
                double r = 0.0, g[HI > 0 ? HI : 1], gp[3] = {0.0, 0.0, 0.0};
#pragma unroll
                for (int q = 0; q < HI; ++q) g[q] = 0.0;
#pragma unroll
                for (int i = 0; i < NI; ++i) {
                    r += w[i][k];
#pragma unroll
                    for (int q = 0; q < HI; ++q)
                        if ((i >> q) & 1) g[q] += w[i][k];
                    if (PAIRS && HI == 2 && i == 3) gp[0] += w[i][k];
                    if (PAIRS && HI == 3) {
                        if ((i & 3) == 3) gp[0] += w[i][k];
                        if ((i & 5) == 5) gp[1] += w[i][k];
                        if ((i & 6) == 6) gp[2] += w[i][k];
                    }
                }
                R[k] += r;
#pragma unroll
                for (int q = 0; q < HI; ++q) S[q][k] += g[q];
                if (PAIRS) {
#pragma unroll
                    for (int a = 0; a < HI; ++a)
#pragma unroll
                        for (int b = a + 1; b < HI; ++b) HH[ps_pair(a, b, H)][k] += gp[ps_pair(a, b, HI)];
                }
#pragma unroll
                for (int q = 0; q < HO; ++q) {  // outer loop bits: uniform in the block
                    if (!((ko >> q) & 1)) continue;
                    S[HI + q][k] += r;
                    if (PAIRS) {
#pragma unroll
                        for (int a = 0; a < HI; ++a) HH[ps_pair(a, HI + q, H)][k] += g[a];
#pragma unroll
                        for (int b = q + 1; b < HO; ++b)
                            if ((ko >> b) & 1) HH[ps_pair(HI + q, HI + b, H)][k] += r;
                    }
                }
            }
        }
        __syncthreads();  // the previous chunk's reduction is finished
#pragma unroll
        for (int k = 0; k < NC; ++k) {
            rows[k][tid] = R[k];
#pragma unroll
            for (int q = 0; q < H; ++q) rows[(1 + q) * NC + k][tid] = S[q][k];
            if (PAIRS) {
#pragma unroll
                for (int q = 0; q < NHH; ++q) {
                    const double v = warp_sum(HH[q][k]);
                    if (lane == 0) hhw[q * NC + k][warp] = v;
                }
            }
        }
        __syncthreads();
        // masked sums over the 256 threads, one warp per value
        for (int o = warp; o < (PS_T0 + 9 * H) * NC; o += NWP) {
            const int v = o / NC, k = o - v * NC;
            int row = 0, mask = 0;
            if (v < PS_T0) {
                if (v >= 9) {
                    if (!PAIRS) continue;
                    int r = v - 9, a = 0;
                    while (r >= PS_TB - 1 - a) r -= PS_TB - 1 - a++;
                    mask = (1 << a) | (1 << (a + 1 + r));
                } else if (v >= 1) {
                    mask = 1 << (v - 1);
                }
            } else {
                const int q = (v - PS_T0) / 9, m = (v - PS_T0) - 9 * q;
                if (!PAIRS && m) continue;
                row = 1 + q;
                mask = m ? 1 << (m - 1) : 0;
            }
            const double *p = rows[row * NC + k];
            double s = 0.0;
#pragma unroll
            for (int i = 0; i < NWP; ++i) {
                const int t = i * 32 + lane;
                const double x = p[t];
                s += (t & mask) == mask ? x : 0.0;
            }
            s = warp_sum(s);
            if (lane == 0) part[((size_t)v * NC + k) * nchunks + c] = s;
        }
        if (PAIRS && tid < NHH * NC) {
            double s = 0.0;
#pragma unroll
            for (int u = 0; u < NWP; ++u) s += hhw[tid][u];
            part[((size_t)(PS_T0 + 9 * H) * NC + tid) * nchunks + c] = s;
        }
    }
}

// out[P*n + Q] (component-interleaved) for every P <= Q (PAIRS) or P == Q, by bit position;
// one warp each, the chunks' rows read coalesced.  by_qubit: out[i*n + j] and out[j*n + i]
// by qubit (bit n-1-i) instead, or out[i] without PAIRS.
template <int NC, bool PAIRS>
__global__ void __launch_bounds__(128) k_pair_finish(const double *part, int n, int H, i64 nchunks, int by_qubit,
                                                     double *out) {
    const int lane = threadIdx.x & 31;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int P = w, Q = w;
    if (PAIRS) {
        P = 0;
        int r = w;
        while (P < n && r >= n - P) r -= n - P++;
        Q = P + r;
    }
    if (P >= n) return;
    i64 mask;
    const int v = ps_locate(P, Q, H, &mask);
#pragma unroll
    for (int k = 0; k < NC; ++k) {
        const double *p = part + ((size_t)v * NC + k) * nchunks;
        double s = 0.0;
#pragma unroll 8
        for (i64 c = lane; c < nchunks; c += 32) {
            const double x = p[c];
            s += (c & mask) == mask ? x : 0.0;
        }
        s = warp_sum(s);
        if (lane == 0) {
            if (!by_qubit) {
                out[((size_t)P * n + Q) * NC + k] = s;
            } else if (PAIRS) {
                const int i = n - 1 - P, j = n - 1 - Q;
                out[((size_t)i * n + j) * NC + k] = s;
                out[((size_t)j * n + i) * NC + k] = s;
            } else {
                out[(size_t)(n - 1 - P) * NC + k] = s;
            }
        }
    }
}

template <int NC, bool PAIRS, typename F>
inline int launch_pair_sums(const F &f, int n, double *part, double *out, bool by_qubit, cudaStream_t s) {
    const int H = ps_loop_bits(n);
    const i64 nchunks = ps_chunks(n), cap = (i64)sm_count() * 16;
    const int grid = (int)(nchunks < cap ? nchunks : cap);
    switch (H) {
    case 0: k_pair_sums<NC, 0, PAIRS><<<grid, 1 << PS_TB, 0, s>>>(f, n, nchunks, part); break;
    case 1: k_pair_sums<NC, 1, PAIRS><<<grid, 1 << PS_TB, 0, s>>>(f, n, nchunks, part); break;
    case 2: k_pair_sums<NC, 2, PAIRS><<<grid, 1 << PS_TB, 0, s>>>(f, n, nchunks, part); break;
    case 3: k_pair_sums<NC, 3, PAIRS><<<grid, 1 << PS_TB, 0, s>>>(f, n, nchunks, part); break;
    case 4: k_pair_sums<NC, 4, PAIRS><<<grid, 1 << PS_TB, 0, s>>>(f, n, nchunks, part); break;
    case 5: k_pair_sums<NC, 5, PAIRS><<<grid, 1 << PS_TB, 0, s>>>(f, n, nchunks, part); break;
    default: k_pair_sums<NC, PS_MAXH, PAIRS><<<grid, 1 << PS_TB, 0, s>>>(f, n, nchunks, part); break;
    }
    EMUSV_CHECK_LAUNCH();
    const int warps = PAIRS ? n * (n + 1) / 2 : n;
    k_pair_finish<NC, PAIRS><<<(warps + 3) / 4, 128, 0, s>>>(part, n, H, nchunks, by_qubit ? 1 : 0, out);
    EMUSV_CHECK_LAUNCH();
    return EMUSV_OK;
}

}  // namespace emusv
