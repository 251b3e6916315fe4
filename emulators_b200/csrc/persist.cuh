// One Lanczos run (and the time step built on it) in ONE launch, for registers whose vectors
// fit the shared memory of the GPU: norm, iterations, convergence decisions, combination.
//
// A job (one register) is run by G = 2^gbits CTAs.  A CTA owns 2^tb consecutive amplitudes of
// every vector; its part of v_j and the diagonal of H stay in shared memory, a thread owns the
// same NA amplitudes throughout, and the basis is written to the workspace as the iteration
// goes.  Per iteration:
//   A  h = (H - sigma) v_j: flips of the low bits from shared memory, of the CTA bits from the
//      other CTAs' parts; sums <v_j, h>, ||h||^2;
//   B  w = h - a_j v_j - b_j v_{j-1}, stored as u_{j+1}; sums ||w||^2, <v_j, w>.
// Each of the two ends in an exchange of the CTAs' sums, which is also the job's barrier.
//   Up to 16 CTAs the job is one thread-block cluster: partners are read and sums exchanged
//   through distributed shared memory, the barrier is an mbarrier in every CTA that all CTAs
//   arrive on (about 1 us an exchange).
//   Beyond, the clusters (of four CTAs) of a cooperative launch exchange through the L2: a
//   cluster writes every sum as a 16-byte record (value, epoch) and every CTA reads the records
//   of all clusters until each carries the phase's epoch, so one round trip both synchronises
//   and delivers; partners are read from the stored vector.
//
// The decisions (krylov_exp.py:60-96: happy breakdown, exponential of the extended tridiagonal
// matrix, Expokit estimate) are taken by extra warps (of every CTA of a cluster job, of one
// more CTA of a grid job), one iteration each, while the compute warps go on: an iteration of
// a small register takes a few us, a decision about ten.  An iteration that ends the run does so
// once every earlier one is known not to, so the run stops at the first iteration that converges,
// where the reference stops; the iterations computed meanwhile are left unused.
//
// Bound by latencies: per iteration two exchanges and the flips.  Measured on B200 (us per further
// iteration of the kernel, complex128 unless said; in brackets the us an iteration took as several
// kernels): 12 qubits 4.3 (47), 14 6.2, 15 complex64 7.0 (50), 16 9.9, 18 14.7, 20 38 (60).  In one
// CTA the decisions bound it, whose work grows with the basis and which four warps share: 10 qubits
// 79 us for 14 iterations, 142 for 28, 400 for 54 (40 us each as kernels).  An exchange takes 0.4 us in one CTA, 1.5-1.8 in
// a cluster, 3.1-3.8 through the L2 with 32 clusters of four (4.9-6.4 when 128 CTAs read each
// other's records); one warp a sum waits and hands it on (with all eight warps waiting 12 qubits
// took 4.5 us an iteration, 14 6.5, 18 15.4).
//
// Every wait is bounded (PArgs::wait): on a timeout the CTA records EMUSV_TIMEOUT in the run's state
// and the job's CTAs return.  Whether a wait ran out is decided by the warps that wait and handed
// to the CTA through a barrier, so its threads always leave together.
#pragma once

#include "krylov_device.cuh"

namespace emusv {

constexpr int PMAXN = 20;          // qubits of a run at most
constexpr int PMAXG_BITS = 7;      // CTAs per job: at most 128
constexpr int PMAXG = 1 << PMAXG_BITS;
constexpr int PCL_BITS = 4;        // CTAs of a cluster job: at most 16
constexpr int PGC_BITS = 2;        // CTAs per cluster of a grid job: 4 (33 such clusters fit the GPU)
constexpr long long PWAIT_LIMIT = 4000000000LL;  // SM clock cycles a wait lasts at most (about 2 s)

struct __align__(16) PRec {  // written and read as one 16-byte access
    double v;
    unsigned long long e;
};
// Exchange area of one job (in the workspace header; needs no initial value: an epoch is
// used by one launch only).
struct PExchange {
    PRec a[3][PMAXG >> PGC_BITS];  // phase A: <v,h> re, im, ||h||^2
    PRec b[3][PMAXG >> PGC_BITS];  // phase B: ||w||^2, <v_j, w> re, im (and the input norm)
    PRec iter[KMAX][5];      // iteration j: a_re, a_im, r, ||H v_j||^2, outcome flag
    PRec start[2];           // sigma, the input's scale
    PRec verdict;            // v = the run's status once decided
};

// One run: v0 -> basis (ks, slots 1..) and, when out is given, the combination.
struct PJob {
    const void *v0;
    void *out;
    KState *ks;
    PExchange *x;
    unsigned char *basis;    // slot k at k * 2^n amplitudes
    int energy_shift;
};
struct PArgs {
    HamParams P;
    PJob job[2];
    int njobs, gbits, tbits; // log2 of the job's CTAs and of the amplitudes per CTA
    int limit, maxdim;       // iterations computed at most (basis slots), max_krylov_dim
    double dt, exp_tol, norm_tol;
    unsigned long long epoch;  // the launch's first epoch
    long long wait;            // clock cycles a wait lasts at most
    int withhold;              // failure-path test: the last CTA of job 0 sends no sums
};

// Host side (persist.cu).
bool persist_applies(const HamParams &P, int dtype);  // on the current device
size_t persist_exchange_bytes();
void persist_set_wait_test(long long wait_cycles, int withhold);
void persist_set_streaming(int on);
// Runs 1 or 2 jobs of the same operator; the caller reads their states afterwards.
int persist_launch(const HamParams &P, int dtype, double dt, const PJob *jobs, int njobs, int capacity,
                   double exp_tol, double norm_tol, int maxdim, cudaStream_t s);

}  // namespace emusv
