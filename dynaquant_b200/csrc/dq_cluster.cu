// dq_cluster.cu — one launch per step for ensembles that fit on the chip.
//
// Trajectories do not exchange anything, so a thread-block cluster can carry a
// few of them through a whole step by itself: noise, the m Lanczos iterations,
// the exponential, the combination, the norms.  The grid-wide form of
// dq_batched.cu runs 2 m + 4 launches for the same step, and on a small system
// each is bound by its launch, its dependent scalar loads and its grid-wide
// reduction (ticket, partials through L2), not by the data: 12 us per
// iteration for a 1 MB slab, 20 us for 2 to 4 MB.
//
// A cluster owns TC trajectories, each of its CTAs a contiguous range of rows.
// Shared memory holds, for the whole step, the CTA's window of r_j (its own
// rows and the bandwidth on either side), r_{j-1} (then w in its place), the
// diagonal and, where they fit, the coupling records: the gathers of an
// iteration touch nothing else.  r_{j+1} also goes to its global slab, for the
// combination.  alpha_j and beta_j are sums over the cluster: every CTA stores
// its part into every CTA's shared memory (DSMEM), and after one hardware
// cluster barrier (0.2 to 0.3 us) every CTA adds the parts in rank order, so
// all hold the same bits and no scalar takes a trip through global memory.
// After the second barrier the window's margins are read from the
// neighbours' shared memory.  A one-CTA cluster needs none of this.
//
// What bounds it: at 2 couplings per row the latency of an iteration's two
// reductions; at 28 per row the gathers' shared-memory wavefronts.
#include <algorithm>
#include <cmath>

#include "dq_batched.cuh"
#include "dq_rng.cuh"
#include "dq_tma.cuh"

namespace dq {

constexpr int kClThreads = 512;
constexpr int kClWarps = kClThreads / 32;
constexpr int kClMaxCtas = 16;            // CTAs per cluster (above 8: not portable, sm_100 allows 16)
// dynamic shared memory of one CTA (one CTA per SM: 128 registers a thread)
constexpr size_t kClSmemMax = 224 * 1024;

// margins above this are read through L2 instead of the neighbours' shared memory
constexpr size_t kClWideMargin = 32 * 1024;

enum { kClNoise = 1, kClFinish = 2 };

struct ClusterArgs {
    int n, B, TC, rpc, bw, m, flags, bil, chunks;
    int rec_smem;             // bytes of coupling records kept in shared memory (0: read through L1)
    const int* bptr;
    const int* bcol;
    const void* bcoef;
    void* slabs;
    size_t slab;              // complex values per slab
    void* diag;
    BatchedScalars S;
    int noise, ns, traj0, step;   // step: kPlain
    double subdt, sqrt_subdt;
    uint64_t seed;
    const double* sigma;
    const double* invtau;
    const double* coeff;
    const double* eps;
    double* deps;
    const double* zzD;
    const int* zz_start;
    int norm_mode, m_min;
    double tau_im, tol;
    double* erracc;
    const cd* bra;
    // one trajectory through the drop-in step (kPlain): the state comes from psi_in as it is (q_1) and
    // goes to psi_out normalised; the sums of the record may be null
    const cd* psi_in;
    cd* psi_out;
    double* pops_row;
    cd* corr_pt;
    PlainScalars* ps;
    PlainGrid* grid;          // kDropInGrid: the partial sums and the barrier
    // Taylor-Krylov step (kTaylor): psi_in and psi_out are the ensemble's states, the matrix above is the
    // step's Hamiltonian, the Lanczos iterations run on B; per trajectory <bra|psi> and sum |psi|^4
    int tk_p;
    const int* b_ptr;
    const int* b_col;
    const double* b_val;
    const double* b_diag;
    cd tk_coef[kMaxL];        // tau^k / k!
    double* tk_obs;           // [3][B]
    int smem;                 // dynamic shared memory of a CTA
    unsigned char* scratch;   // the dense exponential's matrices where shared memory is too small for them
    size_t scratch_stride;    // of one CTA that takes trajectories
};

// Shared memory of a CTA: reductions, the chunk's scalars, the vectors, the records.
struct ClLayout {
    size_t ex, red, al, y, par, be, sc, acc, win, prev, d, rec, total;
};

static __host__ __device__ inline ClLayout cl_layout(int n, int CS, int TC, int m, int rpc, int bw, size_t rsz,
                                                     size_t rec, bool taylor = false) {
    ClLayout L;
    size_t p = 0;
    L.ex = p; p += sizeof(double2) * 2 * CS * TC;
    L.red = p; p += sizeof(double2) * 2 * kClWarps * TC;
    L.al = p; p += sizeof(double2) * (m + 2) * TC;
    L.y = p; p += sizeof(double2) * m * TC;
    L.par = p; p += sizeof(double2) * 3 * TC;
    L.be = p; p += sizeof(double) * (m + 2) * TC;
    L.sc = p; p += sizeof(double) * (m + 2) * TC;
    p = (p + 127) & ~(size_t)127;
    const size_t row = (size_t)TC * 2 * rsz;
    L.acc = p; p += taylor ? rpc * row : 0;   // the Taylor sum of the own rows
    p = (p + 15) & ~(size_t)15;
    // from here on the dense exponential may take the place of everything
    const size_t wide = rpc + 2 * (size_t)bw;   // never more than the rows there are (bw may be n)
    L.win = p; p += (CS > 1 ? (wide < (size_t)n ? wide : (size_t)(n > rpc ? n : rpc)) : rpc) * row;
    L.prev = p; p += rpc * row;
    L.d = p; p += rpc * row / 2;
    p = (p + 15) & ~(size_t)15;
    L.rec = p; p += rec;
    L.total = (p + 15) & ~(size_t)15;
    return L;
}

// What a launch carries through its step.
// (kAdaptive: an ensemble with the adaptive dimension, whose checks stay out of the other kernels' registers)
enum { kEnsemble = 0, kDropIn = 1, kTaylor = 2, kDropInGrid = 3, kAdaptive = 4 };

// The layout of one of a launch's CTAs.
template <typename Real, int kMode>
__device__ __forceinline__ ClLayout cl_shape(const ClusterArgs& A, int CS) {
    return cl_layout(A.n, kMode == kDropInGrid ? 2 : CS, A.TC, A.m, A.rpc, A.bw, sizeof(Real), A.rec_smem,
                     kMode == kTaylor);
}

// Bytes of the block and group starts in front of the records of nb row blocks, `per` to a group.
static __host__ __device__ inline size_t cl_rec_head(size_t nb, int per) {
    return ((nb + (nb + per - 1) / per + 2) * 4 + 15) / 16 * 16;
}

__device__ __forceinline__ unsigned cl_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cl_size() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cl_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// p in the shared memory of CTA `rank` of the cluster
__device__ __forceinline__ void cl_store(double2* p, unsigned rank, double2 v) {
    unsigned a = (unsigned)__cvta_generic_to_shared(p), ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(ra), "d"(v.x), "d"(v.y) : "memory");
}

// 16 or 8 bytes of `p` in the shared memory of CTA `rank`
template <typename T>
__device__ __forceinline__ T cl_load(const T* p, unsigned rank) {
    unsigned a = (unsigned)__cvta_generic_to_shared(p), ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
    T v;
    if constexpr (sizeof(T) == 16) {
        unsigned* u = reinterpret_cast<unsigned*>(&v);
        asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]) : "r"(ra) : "memory");
    } else {
        unsigned* u = reinterpret_cast<unsigned*>(&v);
        asm volatile("ld.shared::cluster.v2.u32 {%0, %1}, [%2];" : "=r"(u[0]), "=r"(u[1]) : "r"(ra) : "memory");
    }
    return v;
}

// Trajectory b's error estimate of the step.
template <bool kPlain>
__device__ __forceinline__ void cl_estimate(const ClusterArgs& A, int b, double est) {
    if (kPlain) {
        A.ps->err = est;
        if (A.erracc) *A.erracc += est;
    } else {
        A.erracc[b] += est;
    }
}

// The dense exponential of a cluster's trajectories (absolute site energies or
// long steps).  CTA `rank` takes trajectories rank, rank + CS, ... and works on
// up to kMaxTeams of them at once, each by its own part of the CTA with its
// matrices (6 L^2 complex) in the shared memory of the window, the diagonal and
// the records.  An LU of this size is a chain of small steps with a barrier
// each, 30 to 60 us for m = 12 to 20 whatever the threads, so trajectories side
// by side are what counts: one CTA that took all of them in a row, its matrices
// in global memory, spent 1.08 ms of a step of 1.43 ms (4,731 sites x 100,
// eight to a cluster of nine CTAs), and 1.6 ms of 2.0 ms at 132 x 4,096, 32 to
// a CTA.

// Teams for nt trajectories with matrices of L rows in `room` bytes (0: not even one fits).
static __host__ __device__ inline int cl_dense_teams(size_t room, int L, int nt) {
    if (pade_mats_bytes(L) > room) return 0;
    int teams = 1;
    while (teams < kMaxTeams && teams < nt && 2 * (size_t)teams * pade_mats_bytes(L) <= room) teams *= 2;
    return teams;
}
// Shared memory from the window on that holds all teams of a CTA, in all at most `room`.
static __host__ inline size_t cl_dense_bytes(size_t room, int L, int nt) {
    return cl_dense_teams(room, L, nt) * pade_mats_bytes(L);
}

// One team's view of that work: its trajectories t = first, first + step, ...
// < nt of the chunk.
struct ClDense {
    const double2* al;        // [j][t]
    const double* be;
    const double* sc;
    const double2* nav;       // [t].x: ||H q_{m+1}||
    int TC, c0, nt, first, step;
    WarpsTeam team;
    unsigned char* mats;
};

// matrices of at most L rows
template <typename Real, int kMode>
__device__ __forceinline__ ClDense cl_dense(const ClusterArgs& A, unsigned char* smem, int chunk, int rank, int CS,
                                            int L) {
    const ClLayout Y = cl_shape<Real, kMode>(A, CS);
    ClDense D;
    D.al = reinterpret_cast<const double2*>(smem + Y.al);
    D.be = reinterpret_cast<const double*>(smem + Y.be);
    D.sc = reinterpret_cast<const double*>(smem + Y.sc);
    D.nav = reinterpret_cast<const double2*>(smem + Y.par) + 2 * A.TC;
    D.TC = A.TC;
    D.c0 = chunk * A.TC;
    D.nt = min(A.TC, A.B - D.c0);
    int teams = cl_dense_teams(A.smem - Y.win, L, (D.nt + CS - 1) / CS);
    D.mats = smem + Y.win;
    if (teams == 0) {
        teams = 1;
        D.mats = A.scratch + ((size_t)chunk * min(CS, A.TC) + min(rank, A.TC - 1)) * A.scratch_stride;
    }
    D.team = WarpsTeam{(int)threadIdx.x / (kClThreads / teams), kClThreads / teams};
    D.mats += D.team.id() * pade_mats_bytes(L);
    D.first = rank + D.team.id() * CS;
    D.step = CS * teams;
    return D;
}

// exp(tau Tbar) of trajectory t, dimension m with p rows of augmentation
__device__ __forceinline__ int cl_dense_one(const ClusterArgs& A, const ClDense& D, int t, int m, int p, cd** E) {
    const int L = m + p;
    cd* M = reinterpret_cast<cd*>(D.mats);
    for (int e = D.team.rank(); e < L * L; e += D.team.size()) {
        const int i = e / L, j = e - i * L;
        cd v = cmk(0.0, 0.0);
        if (i < m && j < m) {
            if (i == j) v = cmk(D.al[(i + 1) * D.TC + t].x, D.al[(i + 1) * D.TC + t].y);
            else if (j == i + 1) v = cmk(D.be[(i + 1) * D.TC + t], 0.0);
            else if (i == j + 1) v = cmk(D.be[(j + 1) * D.TC + t], 0.0);
        } else if ((i == 0 && j == m) || (i >= m && j == i + 1)) {
            v = cmk(1.0, 0.0);
        }
        M[e] = cmul(cmk(0.0, A.tau_im), v);
    }
    D.team.sync();
    return pade_exp_team(D.team, L, A.norm_mode, D.mats, E);
}

// The combine weights of the CTA's marked trajectories (mtr = -m), zero from
// their dimension to mmax, through global memory, and their error estimates.
// Taylor-Krylov: the last column's times ||A^p psi|| = 1 / sc_1.
template <typename Real, int kMode>
__device__ __noinline__ void cl_dense_weights(const ClusterArgs& A, unsigned char* smem, const int* mtr, int chunk,
                                              int rank, int CS, int mmax) {
    constexpr bool kTk = kMode == kTaylor, kPlain = kMode == kDropIn || kMode == kDropInGrid;
    const int p = kTk ? A.tk_p : 2;
    const ClDense D = cl_dense<Real, kMode>(A, smem, chunk, rank, CS, mmax + p);
    double* yt = kPlain ? reinterpret_cast<double*>(A.ps->yt) : A.S.yt;   // [j][trajectory]
    for (int t = D.first; t < D.nt; t += D.step) {
        if (mtr[t] >= 0) continue;   // uniform over the team
        const int m = -mtr[t], L = m + p, b = D.c0 + t;
        cd* E = nullptr;
        const int s = cl_dense_one(A, D, t, m, p, &E);
        for (int j = D.team.rank(); j < mmax; j += D.team.size()) {
            cd v = cmk(0.0, 0.0);
            if (j < m && s >= 0) {
                v = E[j * L + (kTk ? L - 1 : 0)];
                if (kTk) v = cscale(v, 1.0 / D.sc[D.TC + t]);
                v = cscale(v, D.sc[(j + 1) * D.TC + t]);
            }
            double* y = yt + 2 * ((size_t)(j + 1) * A.B + b);
            y[0] = v.x;
            y[1] = v.y;
        }
        if (D.team.rank() == 0) {
            if (s < 0) {
                atomicCAS(A.S.status, 0, s == -1 ? DQ_ERR_SCALING : DQ_ERR_SINGULAR);
            } else {
                const double bm = D.be[m * D.TC + t];
                const cd e1 = E[(m - 1) * L + m], e2 = E[(m - 1) * L + m + 1];
                // with the adaptive dimension only err1 (||H q_{m+1}|| belongs to the largest m)
                const double est = kMode == kAdaptive ? fmax(fabs(bm) * sqrt(cabs2(e1)), 1.110223e-16)
                                                      : expokit_error(bm, D.nav[t].x, e1, e2);
                if (kTk) A.tk_obs[b] = est;   // completed with the norm
                else cl_estimate<kPlain>(A, b, est);
            }
            if (kMode == kAdaptive) A.S.mtraj[b] = m;
        }
        D.team.sync();
    }
}

// One CTA's view of its cluster's sums.
template <int TPT, bool kLocal>
struct ClSum {
    double2* ex;    // [2][CS][TC]
    double2* red;   // [2][warps][TC]
    int TC, CS;
    unsigned rank;
    int pt, pd;     // threadIdx.x % TC, threadIdx.x / TC

    __device__ __forceinline__ void sync() const {
        if constexpr (kLocal) __syncthreads();
        else cl_sync();
    }
    // this CTA's part of sum `buf` into every CTA's ex[buf]; the caller syncs.
    // kPair: y is summed too.
    template <bool kPair>
    __device__ __forceinline__ void part(int buf, const double (&x)[TPT], const double (&y)[TPT]) const {
        const int TL = TC / TPT, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        double a[TPT], b[TPT];
#pragma unroll
        for (int t = 0; t < TPT; ++t) {
            a[t] = x[t];
            b[t] = kPair ? y[t] : 0.0;
        }
        for (int o = TL; o < 32; o <<= 1) {
#pragma unroll
            for (int t = 0; t < TPT; ++t) {
                a[t] += __shfl_xor_sync(0xffffffffu, a[t], o);
                if (kPair) b[t] += __shfl_xor_sync(0xffffffffu, b[t], o);
            }
        }
        if (lane < TL) {
#pragma unroll
            for (int t = 0; t < TPT; ++t) red[(buf * kClWarps + warp) * TC + lane * TPT + t] = make_double2(a[t], b[t]);
        }
        __syncthreads();
        for (int dst = pd; dst < CS; dst += kClThreads / TC) {
            const int t = pt;
            double2 v[kClWarps];
#pragma unroll
            for (int w = 0; w < kClWarps; ++w) v[w] = red[(buf * kClWarps + w) * TC + t];
#pragma unroll
            for (int h = kClWarps / 2; h > 0; h >>= 1)
#pragma unroll
                for (int w = 0; w < h; ++w) {
                    v[w].x += v[w + h].x;
                    if (kPair) v[w].y += v[w + h].y;
                }
            double2* p = ex + ((size_t)buf * CS + rank) * TC + t;
            if constexpr (kLocal) *p = v[0];
            else cl_store(p, dst, v[0]);
        }
    }
    // the whole sum of trajectory t (after the sync), in rank order
    __device__ __forceinline__ double2 get(int buf, int t) const {
        double2 s = ex[(size_t)buf * CS * TC + t];
        if constexpr (!kLocal) {
#pragma unroll 4
            for (int r = 1; r < CS; ++r) {
                const double2 v = ex[((size_t)buf * CS + r) * TC + t];
                s.x += v.x;
                s.y += v.y;
            }
        }
        return s;
    }
};

// Budget of the grid barrier's wait in SM cycles, as dq_debug_set_wait_cycles
// sets it for the device: negative values make a CTA wait that many cycles for
// a count that never comes.
__device__ long long g_cl_wait_cycles = kWaitCycles;

// The same over the whole grid (one trajectory, a cooperative launch).  A CTA
// writes its part, fences it with its slab rows and counts itself in; one
// thread of each CTA waits for the count, then all CTAs add the parts in rank
// order.  The parts are double-buffered by the barrier's parity: a CTA writes
// a buffer again only after a barrier that all readers of its old contents
// have passed.  (Parts as tagged words polled by a thread per rank, without a
// count, took 3700 to 12,500 cycles with 63 CTAs: the polls crowd the words.)
// The wait is bounded: a CTA that gives up records DQ_ERR_TIMEOUT and stops
// waiting for the rest of the launch (its results are void, its accesses stay
// in bounds), so every CTA ends; it still counts itself in at every barrier
// and out at the end, where the last one clears the counts.
struct ClGridSum {
    double2* ex;    // [2]: the totals
    double2* red;   // [2][warps]
    PlainGrid* g;
    int* status;
    int* dead;      // shared: this CTA gave up
    int G;
    unsigned rank;
    unsigned seq;   // barriers passed
    int pending;
    long long budget;

    template <bool kPair>
    __device__ __forceinline__ void part(int buf, const double (&x)[1], const double (&y)[1]) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const double a = warp_sum(x[0]), b = kPair ? warp_sum(y[0]) : 0.0;
        if (lane == 0) red[buf * kClWarps + warp] = make_double2(a, b);
        pending |= 1 << buf;
    }
    __device__ __forceinline__ void sync() {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const unsigned par = seq & 1;
        __syncthreads();
        if (threadIdx.x < 32) {
            // a warp: lane w + 16 buf holds a warp's part of sum buf
            static_assert(kClWarps == 16, "a half warp per sum");
            double2 v = red[lane];
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) {
                v.x += __shfl_down_sync(0xffffffffu, v.x, o, 16);
                v.y += __shfl_down_sync(0xffffffffu, v.y, o, 16);
            }
            if ((lane & 15) == 0 && ((pending >> (lane >> 4)) & 1)) __stcg(&g->part[par][lane >> 4][rank], v);
            __syncwarp();
            if (lane == 0) {
                __threadfence();   // the CTA's stores (ordered by the barriers before this) before the count
                atomicAdd(&g->count, 1u);
                const unsigned want = (seq + 1) * (unsigned)G;
                const long long t0 = clock64();
                while (*dead == 0) {
                    unsigned c;
                    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(&g->count) : "memory");
                    if (c >= want && budget > 0) break;
                    if (clock64() - t0 > llabs(budget)) {
                        *dead = 1;
                        atomicCAS(status, 0, DQ_ERR_TIMEOUT);
                    }
                }
                __threadfence();
            }
        }
        __syncthreads();
        for (int buf = 0; buf < 2; ++buf) {
            if (!((pending >> buf) & 1)) continue;
            double2 s = make_double2(0.0, 0.0);
            if ((int)threadIdx.x < G) s = __ldcg(&g->part[par][buf][threadIdx.x]);
            s.x = warp_sum(s.x);
            s.y = warp_sum(s.y);
            if (lane == 0) red[buf * kClWarps + warp] = s;
        }
        __syncthreads();
        if (threadIdx.x < 2 && ((pending >> threadIdx.x) & 1)) {
            double2 s = red[threadIdx.x * kClWarps];
            for (int w = 1; w < kPlainGridMax / 32; ++w) {
                const double2 v = red[threadIdx.x * kClWarps + w];
                s.x += v.x;
                s.y += v.y;
            }
            ex[threadIdx.x] = s;
        }
        __syncthreads();
        pending = 0;
        ++seq;
    }
    __device__ __forceinline__ double2 get(int buf, int) const { return ex[buf]; }
    // the last CTA to leave clears the count for the next launch
    __device__ __forceinline__ void leave() {
        if (threadIdx.x == 0 && atomicAdd(&g->left, 1u) == (unsigned)G - 1) {
            g->count = 0;
            g->left = 0;
            __threadfence();
        }
    }
};
static_assert(kPlainGridMax <= kClThreads && kPlainGridMax / 32 <= kClWarps, "a thread per rank");

__device__ __forceinline__ unsigned sm_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ float4 lds_f4(unsigned a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ double2 lds_d2(unsigned a) {
    double2 v;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a));
    return v;
}

// The power of two at or below |s| (0 for 0), as a float, and 1 over it.
__device__ __forceinline__ float cl_pow2(double s) {
    if (s == 0.0) return 0.f;
    return ldexpf(1.f, max(-120, min(120, ilogb(s))));
}
__device__ __forceinline__ double cl_pow2_inv(double s) { return ldexp(1.0, -max(-120, min(120, ilogb(s)))); }

// Where a thread's coupling records are.  In global memory (lg < 0) the
// records of a block are contiguous from bptr[k]; in shared memory those of
// the 2^lg = 32 / TL blocks a warp works on are interleaved entry by entry, so
// the warp's loads of one entry are one contiguous run instead of one
// bank-conflicting piece per block.
struct ClRecs {
    const int* bptr;     // starts of the own blocks
    const int* col;      // FP64 form: columns
    const void* rec;     // packed records, or FP64 coefficients
    unsigned scol, srec; // the same in shared memory
    const int* goff;     // first entry of each interleaved group of 2^lg blocks
    int lg;
};

// The records of a CTA's nbo row blocks from kb0 on, copied to `area` where its
// `room` bytes hold them; all threads of the CTA, which sync before they use them.
template <typename Real, int R>
__device__ __forceinline__ ClRecs cl_load_records(unsigned char* area, size_t room, int kb0, int nbo, int TL,
                                                  const int* gptr, const int* gcol, const void* gcoef) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
            ClRecs Q = ClRecs{gptr + kb0, gcol, gcoef, 0u, 0u, nullptr, -1};
            // block starts, group starts (a group is as long as its longest block), columns (FP64), coefficients
            const int lg = __ffs(32 / TL) - 1, per = 1 << lg, ng = (nbo + per - 1) >> lg;
            const size_t head = cl_rec_head(nbo, per);
            if (head > room) return Q;
            int* sb = reinterpret_cast<int*>(area);
            int* sg = sb + nbo + 1;
            for (int k = threadIdx.x; k <= nbo; k += kClThreads) sb[k] = __ldg(gptr + kb0 + k);
            __syncthreads();
            for (int g = warp; g < ng; g += kClWarps) {
                const int k = (g << lg) + lane;
                int len = lane < per && k < nbo ? sb[k + 1] - sb[k] : 0;
                len = __reduce_max_sync(0xffffffffu, len);
                if (lane == 0) sg[g + 1] = len;
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                sg[0] = 0;
                for (int g = 0; g < ng; ++g) sg[g + 1] += sg[g];
            }
            __syncthreads();
            const size_t slots = (size_t)sg[ng] << lg;
            const size_t cols = sizeof(Real) == 8 ? (slots * 4 + 15) / 16 * 16 : 0;
            unsigned char* q = area + head + cols;
            Q.bptr = sb;
            if (head + cols + slots * (sizeof(Real) == 8 ? R * 8 : 16) <= room) {
                int* scol = reinterpret_cast<int*>(area + head);
                // a warp per block, a lane per entry
                for (int k = warp; k < nbo; k += kClWarps) {
                    const int p0 = sb[k], ne = sb[k + 1] - p0, g = sg[k >> lg], i = k & (per - 1);
                    for (int e = lane; e < ne; e += 32) {
                        if constexpr (sizeof(Real) == 4) {
                            reinterpret_cast<float4*>(q)[(g + e) * per + i] =
                                __ldg(reinterpret_cast<const float4*>(gcoef) + p0 + e);
                        } else {
                            const Real* gr = reinterpret_cast<const Real*>(gcoef) + (size_t)(p0 + e) * R;
                            scol[(g + e) * per + i] = __ldg(gcol + p0 + e);
                            if constexpr (R == 1) {
                                reinterpret_cast<Real*>(q)[(g + e) * per + i] = __ldg(gr);
                            } else {
    #pragma unroll
                                for (int h = 0; h < R / 2; ++h)
                                    reinterpret_cast<double2*>(q)[((g + e) * (R / 2) + h) * per + i] =
                                        __ldg(reinterpret_cast<const double2*>(gr) + h);
                            }
                        }
                    }
                }
                Q.scol = sm_addr(scol);
                Q.srec = sm_addr(q);
                Q.goff = sg;
                Q.lg = lg;
            }
    return Q;
}

// Four coupling entries of one row block: column and R coefficients each.
template <typename Real, int R>
struct ClRec {
    int c[4];
    Real cf[4][R];
    __device__ __forceinline__ void put(int u, float4 r) {
        c[u] = __float_as_int(r.x);
        cf[u][0] = r.y;
        if constexpr (R > 1) cf[u][R > 1 ? 1 : 0] = r.z;
        if constexpr (R > 2) cf[u][R > 2 ? 2 : 0] = r.w;
    }
    // entries [e, e + 4) of a block of `len` entries; `off` is the block's
    // first slot (kShared: byte offset of its 16-byte records)
    template <bool kShared>
    __device__ __forceinline__ void load(const ClRecs& Q, int off, int e, int len) {
        if constexpr (sizeof(Real) == 4) {
            // packed records {col, c0, c1, c2}, a multiple of 4 per block
            if constexpr (kShared) {
                const unsigned a = Q.srec + off + (e << (Q.lg + 4));
#pragma unroll
                for (int u = 0; u < 4; ++u) put(u, lds_f4(a + (u << (Q.lg + 4))));
            } else {
                const float4* r4 = reinterpret_cast<const float4*>(Q.rec) + off + e;
#pragma unroll
                for (int u = 0; u < 4; ++u) put(u, __ldg(r4 + u));
            }
        } else {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int p = min(e + u, len - 1);
                if constexpr (kShared) {
                    // columns [slot], coefficients by pairs in planes of 2^lg (R = 1: singles)
                    const int g = off >> Q.lg, i = off & ((1 << Q.lg) - 1), slot = ((g + p) << Q.lg) + i;
                    asm volatile("ld.shared.s32 %0, [%1];" : "=r"(c[u]) : "r"(Q.scol + 4 * slot));
                    if constexpr (R == 1) {
                        asm volatile("ld.shared.f64 %0, [%1];" : "=d"(cf[u][0]) : "r"(Q.srec + 8 * slot));
                    } else {
#pragma unroll
                        for (int h = 0; h < R / 2; ++h) {
                            const double2 v = lds_d2(Q.srec + 16 * ((((g + p) * (R / 2) + h) << Q.lg) + i));
                            cf[u][2 * h] = v.x;
                            cf[u][2 * h + 1] = v.y;
                        }
                    }
                } else {
                    c[u] = __ldg(Q.col + off + p);
                    const Real* cb = reinterpret_cast<const Real*>(Q.rec) + (size_t)(off + p) * R;
#pragma unroll
                    for (int i = 0; i < R; ++i) cf[u][i] = __ldg(cb + i);
                }
                if (e + u >= len)
#pragma unroll
                    for (int i = 0; i < R; ++i) cf[u][i] = Real(0);
            }
        }
    }
};

// acc += the couplings of one row block times the window's rows (`win`: shared
// address of this thread's trajectories of global row 0, `row` bytes a row);
// the next four entries load while the current four gather.
template <typename Real, int TPT, int R, bool kShared>
__device__ __forceinline__ void cl_gather(const ClRecs& Q, int off, int len, unsigned win, int row,
                                          CV<Real, TPT> (&acc)[R]) {
    ClRec<Real, R> A;
    A.template load<kShared>(Q, off, 0, len);
    for (int e = 0;; e += 4) {
        const bool more = e + 4 < len;
        ClRec<Real, R> N;
        if (more) N.template load<kShared>(Q, off, e + 4, len);
        CV<Real, TPT> y[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const unsigned a = win + A.c[u] * row;
            if constexpr (TPT == 2) {
                const float4 v = lds_f4(a);
                y[u].v[0] = v.x;
                y[u].v[1] = v.y;
                y[u].v[2 * TPT - 2] = v.z;
                y[u].v[2 * TPT - 1] = v.w;
            } else {
                const double2 v = lds_d2(a);
                y[u].v[0] = (Real)v.x;
                y[u].v[1] = (Real)v.y;
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int i = 0; i < R; ++i) cfma<Real, TPT>(acc[i], A.cf[u][i], y[u]);
        if (!more) break;
        A = N;
    }
}

// Brings back what the dense exponential overwrote after iteration j: the
// records, the window of r_{j+1} with its margins, r_j and the diagonal, all of
// which are in global memory too.
template <typename Real, int TPT, int R>
__device__ __forceinline__ void cl_restore(const ClusterArgs& A, unsigned char* smem, int chunk, int rank, int CS, int j) {
    using T = typename VL<Real, TPT>::T;
    const ClLayout Y = cl_shape<Real, kAdaptive>(A, CS);
    const int TC = A.TC, TL = TC / TPT, B = A.B, n = A.n, tl = threadIdx.x % TL, RL = kClThreads / TL;
    const int c0 = chunk * TC, r0 = min(rank * A.rpc, n), nrow = min(n - r0, A.rpc);
    const int bw = CS == 1 ? 0 : A.bw, hlo = min(bw, r0), hhi = min(bw, n - (r0 + nrow));
    cl_load_records<Real, R>(smem + Y.rec, (size_t)A.rec_smem, r0 / R, (nrow + R - 1) / R, TL, A.bptr, A.bcol, A.bcoef);
    if (c0 + tl * TPT < B) {
        const int tca = min(TC, B - c0);
        const Real* slabs = reinterpret_cast<const Real*>(A.slabs);
        // this thread's trajectories on site g of slab q: [chunk][site][trajectory of the chunk], slab 1 plain
        auto at = [&](int q, int g) {
            const size_t x = q == 1 ? (size_t)g * B + c0 : (size_t)c0 * n + (size_t)g * tca;
            return __ldcg(reinterpret_cast<const T*>(slabs + 2 * (A.slab * q + x)) + tl);
        };
        T* win = reinterpret_cast<T*>(smem + Y.win);
        T* prev = reinterpret_cast<T*>(smem + Y.prev);
        Real* dsm = reinterpret_cast<Real*>(smem + Y.d);
        const Real* dg = reinterpret_cast<const Real*>(A.diag);
        for (int h = threadIdx.x / TL; h < hlo + nrow + hhi; h += RL) {
            const int row = h - hlo, g = r0 + row;
            win[(size_t)h * TL + tl] = at(j + 1, g);
            if (row < 0 || row >= nrow) continue;
            prev[(size_t)row * TL + tl] = at(j, g);
#pragma unroll
            for (int t = 0; t < TPT; ++t) dsm[(size_t)row * TC + tl * TPT + t] = dg[(size_t)g * B + c0 + tl * TPT + t];
        }
    }
    __syncthreads();
}

// A CTA's words shared by its threads: a chunk's choices of the adaptive
// dimension (elsewhere marks of the trajectories whose exponential is dense),
// whether there are any, and whether it gave up waiting.
struct ClWords {
    int mtr[kMaxTC];
    int flag, dead;
};

// The adaptive dimension's check after iteration j: EXPOKIT's first term of the
// nt trajectories' undecided ones, a warp each.  Returns, to every thread of the
// CTA, whether some need the dense form (the CTA syncs before the next call).
__device__ __forceinline__ bool cl_series_check(const ClusterArgs& A, const double2* al, const double* be, ClWords& W,
                                                int nt, int j) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) W.flag = 0;
    __syncthreads();
    bool dense = false;
    for (int t = warp; t < nt; t += kClWarps) {
        if (W.mtr[t]) continue;
        const int q = (min(lane, j - 1) + 1) * A.TC + t;
        cd y, f1, f2;
        int s;
        const bool ok = series_exp_tbar(j, cmk(al[q].x, al[q].y), be[q], A.tau_im, A.norm_mode, y, f1, f2, s);
        if (ok && s >= 0 && lane == j - 1 && fabs(be[q]) * sqrt(cabs2(f1)) <= A.tol) W.mtr[t] = j;
        dense = dense || !ok;
    }
    if (dense && lane == 0) atomicOr(&W.flag, 1);
    __syncthreads();
    return W.flag != 0;
}

// The whole check, dense forms included; every CTA of the cluster decides
// alike.  Returns whether all trajectories of the chunk have chosen.
template <typename Real, int TPT, int R>
__device__ __noinline__ bool cl_check(const ClusterArgs& A, unsigned char* smem, ClWords& W, int chunk, int rank,
                                      int CS, int j) {
    int* mtr = W.mtr;
    const ClLayout Y = cl_shape<Real, kAdaptive>(A, CS);
    const double2* al = reinterpret_cast<const double2*>(smem + Y.al);
    const double* be = reinterpret_cast<const double*>(smem + Y.be);
    const int TC = A.TC, c0 = chunk * TC, nt = min(TC, A.B - c0);
    auto sync = [&]() {
        if (CS == 1) __syncthreads();
        else cl_sync();
    };
    const bool dense = cl_series_check(A, al, be, W, nt, j);
    if (dense) {
        // each CTA its own trajectories, the choices, made before or now, through global memory
        sync();   // the neighbours have their margins from this CTA's window
        const ClDense D = cl_dense<Real, kAdaptive>(A, smem, chunk, rank, CS, j + 2);
        for (int t = D.first; t < D.nt; t += D.step) {
            int choice = mtr[t];
            if (choice == 0) {
                cd* E = nullptr;
                const int s = cl_dense_one(A, D, t, j, 2, &E);
                if (s >= 0 && fabs(D.be[j * D.TC + t]) * sqrt(cabs2(E[(j - 1) * (j + 2) + j])) <= A.tol) choice = j;
                D.team.sync();
            }
            if (D.team.rank() == 0) A.S.mtraj[c0 + t] = choice;
        }
        sync();
        if ((int)threadIdx.x < nt) mtr[threadIdx.x] = A.S.mtraj[c0 + threadIdx.x];
        sync();   // the choices may be written again only after all have read them
    }
    bool done = true;
    for (int t = 0; t < nt; ++t) done = done && mtr[t] != 0;
    if (dense && !done) cl_restore<Real, TPT, R>(A, smem, chunk, rank, CS, j);
    return done;
}

// A launch's whole work.  An ensemble with the adaptive dimension whose check
// needs the dense exponential leaves at that iteration (its number is
// returned, else 0) and comes back in here as kResume from it.  The two are
// copies of the code because the loop has few registers to spare: with the
// dense check's call in it a step takes 8 to 13 % longer (600 sites x 1024 FP64:
// 329 us, 301 without), with the second copy out of line 4 %.
template <typename Real, int TPT, int R, bool kLocal, int kMode, bool kResume>
__device__ __forceinline__ int cl_step(const ClusterArgs& A, unsigned char* smem, ClWords& W, int resume) {
    constexpr bool kGrid = kMode == kDropInGrid, kPlain = kMode == kDropIn || kGrid, kTk = kMode == kTaylor;
    constexpr bool adaptive = kMode == kAdaptive, kEns = kMode == kEnsemble || adaptive;
    using T = typename VL<Real, TPT>::T;
    int* mtr = W.mtr;
    int& flag = W.flag;
    const int TC = A.TC, TL = TC / TPT, B = A.B, n = A.n;
    const int CS = kLocal ? 1 : kGrid ? (int)gridDim.x : (int)cl_size();
    const unsigned rank = kLocal ? 0u : kGrid ? blockIdx.x : cl_rank();
    const int bw = kLocal ? 0 : A.bw;
    const ClLayout Y = cl_shape<Real, kMode>(A, CS);
    double2* al = reinterpret_cast<double2*>(smem + Y.al);     // [j][t]
    double2* yts = reinterpret_cast<double2*>(smem + Y.y);     // [j - 1][t]
    // [0][t] the update's coefficients, [1][t] (sc_j, the factor of r_{j-1}), [2][t] complex64: Im alpha's low part
    double2* par = reinterpret_cast<double2*>(smem + Y.par);
    double* be = reinterpret_cast<double*>(smem + Y.be);
    double* scs = reinterpret_cast<double*>(smem + Y.sc);
    const int rowr = TC * 2;                                   // Reals of one row
    Real* win = reinterpret_cast<Real*>(smem + Y.win);
    Real* prev = reinterpret_cast<Real*>(smem + Y.prev);
    Real* dsm = reinterpret_cast<Real*>(smem + Y.d);
    auto make_sum = [&]() {
        double2* ex = reinterpret_cast<double2*>(smem + Y.ex);
        double2* red = reinterpret_cast<double2*>(smem + Y.red);
        if constexpr (kGrid) return ClGridSum{ex, red, A.grid, A.S.status, &W.dead, CS, rank, 0u, 0, g_cl_wait_cycles};
        else return ClSum<TPT, kLocal>{ex, red, TC, CS, rank, (int)threadIdx.x % TC, (int)threadIdx.x / TC};
    };
    auto sum = make_sum();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tl = threadIdx.x % TL, rl = threadIdx.x / TL, RL = kClThreads / TL;
    const int chunk = kGrid ? 0 : blockIdx.x / CS, c0 = chunk * TC;
    const int b0 = c0 + tl * TPT;
    const bool act = b0 < B;                 // lanes past the last trajectory only keep the barriers
    const int bb = act ? b0 : 0;
    const int r0 = min((int)rank * A.rpc, n), nrow = min(n - r0, A.rpc);
    const int nbk = act ? (nrow + R - 1) / R : 0;
    const int hlo = kLocal ? 0 : min(bw, r0);
    Real* cur = win + (size_t)hlo * rowr;                      // the own rows of the window
    const int hhi = kLocal ? 0 : min(bw, n - (r0 + nrow));
    Real* slabs = reinterpret_cast<Real*>(A.slabs);
    auto slab = [&](int j) { return slabs + 2 * A.slab * j; };
    const Real* first = kPlain || kTk ? reinterpret_cast<const Real*>(A.psi_in) : slab(1);
    // own row `row` (within the CTA) of this thread's trajectories
    auto loc = [&](int row) { return (size_t)row * TC + tl * TPT; };
    auto glo = [&](int row) { return (size_t)(r0 + row) * B + bb; };

    // slab j >= 2: [chunk][site][trajectory of the chunk], so a CTA's rows are one contiguous run
    const int tca = min(TC, B - c0);
    auto basis = [&](int j, int row) {
        return slab(j) + 2 * ((size_t)c0 * n + (size_t)(r0 + row) * tca + (act ? tl * TPT : 0));
    };

    // ---- the coupling records of the own row blocks --------------------------
    const int kb0 = r0 / R, nbo = (nrow + R - 1) / R;
    ClRecs Q;
    auto load_records = [&](const int* gptr, const int* gcol, const void* gcoef) {
        Q = cl_load_records<Real, R>(smem + Y.rec, (size_t)A.rec_smem, kb0, nbo, TL, gptr, gcol, gcoef);
    };
    load_records(A.bptr, A.bcol, A.bcoef);

    // ---- r_1 = psi over the window, the diagonal (noise of this step, or as it is)
    if (!kResume && act) {
        const int step = kEns ? *A.S.step : A.step;
        const double* D = A.noise == DQ_NOISE_ZZ && (A.flags & kClNoise)
                              ? A.zzD + (size_t)(step - *A.zz_start) * n * B : nullptr;
        Real* dg = reinterpret_cast<Real*>(A.diag);
        for (int row = rl - hlo; row < nrow + hhi; row += RL) {
            const size_t x = ((ptrdiff_t)r0 + row) * B + bb;
            stv<Real, TPT>(cur + (ptrdiff_t)row * rowr, tl * TPT, ldv<Real, TPT, false>(first, x));
            if (row < 0 || row >= nrow) continue;
            const size_t l = loc(row);
            if (!(A.flags & kClNoise)) {
#pragma unroll
                for (int t = 0; t < TPT; ++t) dsm[l + t] = dg[x + t];
                continue;
            }
            const int site = r0 + row;
            double v[TPT];
            if (A.noise == DQ_NOISE_OU) {
                if constexpr (TPT == 2) {
                    double u0 = A.deps[x], u1 = A.deps[x + 1];
                    ou_update_pair(u0, u1, A.invtau[site], A.coeff[site], A.subdt, A.sqrt_subdt, A.ns, A.seed,
                                   (A.traj0 + bb) >> 1, step, site);
                    A.deps[x] = u0;
                    A.deps[x + 1] = u1;
                    v[0] = __dadd_rn(u0, A.eps[x]);
                    v[TPT - 1] = __dadd_rn(u1, A.eps[x + 1]);
                } else {
                    const double u = ou_update(A.deps[x], A.invtau[site], A.coeff[site], A.subdt, A.sqrt_subdt, A.ns,
                                               A.seed, A.traj0 + bb, step, site);
                    A.deps[x] = u;
                    v[0] = __dadd_rn(u, A.eps[x]);
                }
            } else {
#pragma unroll
                for (int t = 0; t < TPT; ++t) {
                    if (A.noise == DQ_NOISE_GAUSS)
                        v[t] = __dadd_rn(__dmul_rn(normal(A.seed, P_GAUSS, A.traj0 + bb + t, step, site, 0),
                                                   A.sigma[site]), A.eps[x + t]);
                    else if (A.noise == DQ_NOISE_ZZ)
                        v[t] = __dadd_rn(D[x + t], A.eps[x + t]);
                    else
                        v[t] = A.eps[x + t];
                }
            }
#pragma unroll
            for (int t = 0; t < TPT; ++t) {
                dg[x + t] = (Real)v[t];
                dsm[l + t] = (Real)v[t];
            }
        }
    }
    if (!kResume && threadIdx.x < TC) {
        const double s1 = kPlain || kTk ? 1.0 : c0 + (int)threadIdx.x < B ? A.S.sc[(size_t)B + c0 + threadIdx.x] : 0.0;
        scs[TC + threadIdx.x] = s1;
        par[TC + threadIdx.x] = make_double2(s1, 0.0);
        mtr[threadIdx.x] = 0;
    }
    if constexpr (kGrid) {
        if (threadIdx.x == 0) W.dead = 0;
        __syncthreads();
    } else {
        sum.sync();   // every CTA of the cluster runs; the window is in place
    }

    const int rowb = rowr * (int)sizeof(Real);
    const unsigned wcol = sm_addr(cur) - (unsigned)(r0 * rowb) + tl * TPT * 2 * (int)sizeof(Real);   // global row 0
    // H_off r_j of block k
    auto product = [&](int k, CV<Real, TPT> (&acc)[R]) {
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int v = 0; v < 2 * TPT; ++v) acc[i].v[v] = 0;
        const int p0 = Q.bptr[k], len = Q.bptr[k + 1] - p0;
        if (len <= 0) return;
        if (Q.lg < 0) {
            cl_gather<Real, TPT, R, false>(Q, p0, len, wcol, rowb, acc);
        } else {
            const int slot = (Q.goff[k >> Q.lg] << Q.lg) + (k & ((1 << Q.lg) - 1));
            cl_gather<Real, TPT, R, true>(Q, sizeof(Real) == 4 ? slot << 4 : slot, len, wcol, rowb, acc);
        }
    };
    // The window's margins of r_j (j >= 2): the neighbours' rows from their shared memory, or, when
    // the margins are wide, from the slab that the barrier has just published (a window of all 5,278
    // rows in 11 CTAs: a step of 12 iterations took 232 us by DSMEM, 199 us this way)
    const bool wide = kGrid || (size_t)(hlo + hhi) * rowr * sizeof(Real) > kClWideMargin;
    auto margins = [&](int j) {
        if constexpr (!kLocal) {
            const int nh = act ? hlo + hhi : 0;
            const T* src = reinterpret_cast<const T*>(slab(j) + 2 * ((size_t)c0 * n + (act ? tl * TPT : 0)));
            const int stride = tca / TPT;
            for (int h0 = rl; h0 < nh; h0 += 4 * RL) {
                T v[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int h = h0 + q * RL;
                    if (h >= nh) break;
                    const int g = r0 + (h < hlo ? h - hlo : nrow + h - hlo);
                    if (wide) {
                        v[q] = __ldcg(src + (size_t)g * stride);
                    } else if constexpr (!kGrid) {
                        const int own = g / A.rpc;
                        // the owner's own rows start after its lower margin
                        const int at = min(bw, own * A.rpc) + g - own * A.rpc;
                        v[q] = cl_load(reinterpret_cast<const T*>(win + (size_t)at * rowr) + tl, own);
                    }
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int h = h0 + q * RL;
                    if (h >= nh) break;
                    const int row = h < hlo ? h - hlo : nrow + h - hlo;
                    reinterpret_cast<T*>(cur + (ptrdiff_t)row * rowr)[tl] = v[q];
                }
            }
        }
    };

    // the last warp's lanes take the sums' scalars: the margins' loads start with the first warps
    const int last = warp == kClWarps - 1 ? lane : kMaxTC;
    if constexpr (kTk) {
        // the Taylor sum over k < p of tau^k / k! A^k psi, and r_1 = A^p psi with its norm
        Real* tsum = reinterpret_cast<Real*>(smem + Y.acc);
        for (int k = rl; k < nbk; k += RL) stv<Real, TPT>(tsum, loc(k), ldv<Real, TPT, false>(cur, loc(k)));
        double b2[TPT];
        for (int q = 1; q <= A.tk_p; ++q) {
            for (int k = rl; k < nbk; k += RL) {
                CV<Real, TPT> acc[R];
                product(k, acc);
                const size_t l = loc(k);
                const CV<Real, TPT> x = ldv<Real, TPT, false>(cur, l);
#pragma unroll
                for (int v = 0; v < 2 * TPT; ++v) acc[0].v[v] = fma(dsm[l + v / 2], x.v[v], acc[0].v[v]);
                stv<Real, TPT>(prev, l, acc[0]);
            }
            sum.sync();   // the neighbours have read these rows into their margins
            const cd c = q < A.tk_p ? A.tk_coef[q] : cmk(0.0, 0.0);
            b2[0] = 0.0;
            for (int k = rl; k < nbk; k += RL) {
                const size_t l = loc(k);
                const CV<Real, TPT> y = ldv<Real, TPT, false>(prev, l);
                stv<Real, TPT>(cur, l, y);
                stv<Real, TPT>(basis(1, k), 0, y);
                if (q < A.tk_p) {
                    CV<Real, TPT> a = ldv<Real, TPT, false>(tsum, l);
                    a.v[0] += c.x * y.v[0] - c.y * y.v[1];
                    a.v[1] += c.x * y.v[1] + c.y * y.v[0];
                    stv<Real, TPT>(tsum, l, a);
                } else {
                    b2[0] += (double)y.v[0] * y.v[0] + (double)y.v[1] * y.v[1];
                }
            }
            if (q == A.tk_p) sum.template part<false>(1, b2, b2);
            sum.sync();
            margins(1);
            if (q == A.tk_p) {
                for (int t = last; t < TC; t += 32) {
                    const double nb = sqrt(sum.get(1, t).x);
                    if ((!(nb > 0.0) || !isfinite(nb)) && c0 + t < B && rank == 0) atomicCAS(A.S.status, 0, DQ_ERR_NAN);
                    const double s1 = 1.0 / nb;
                    scs[TC + t] = s1;
                    par[TC + t] = make_double2(s1, 0.0);
                }
                // the Lanczos iterations run on B
                for (int k = rl; k < nbk; k += RL)
#pragma unroll
                    for (int t = 0; t < TPT; ++t) dsm[loc(k) + t] = (Real)A.b_diag[r0 + k];
                load_records(A.b_ptr, A.b_col, A.b_val);
            }
            __syncthreads();
        }
    }
    int jl = A.m;   // iterations done
    int j0 = 1;
    if constexpr (kResume) {
        // the check that the first pass left at
        j0 = resume + 1;
        if (cl_check<Real, TPT, R>(A, smem, W, chunk, (int)rank, CS, resume)) {
            jl = resume;
            j0 = A.m + 1;
        }
    }
    for (int j = j0; j <= A.m; ++j) {
        // u = H r_j - (beta_{j-1} sc_{j-1} / sc_j) r_{j-1} over r_{j-1} (w = sc_j u); alpha_j
        double x2[TPT], y2[TPT], sc[TPT];
        Real fm[TPT];
#pragma unroll
        for (int t = 0; t < TPT; ++t) {
            const double2 p = par[TC + tl * TPT + t];
            sc[t] = p.x;
            fm[t] = (Real)p.y;
            x2[t] = y2[t] = 0.0;
        }
        for (int k = rl; k < nbk; k += RL) {
            CV<Real, TPT> acc[R];
            product(k, acc);
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int row = k * R + i;
                if (row >= nrow) break;
                const size_t l = loc(row);
                const CV<Real, TPT> x = ldv<Real, TPT, false>(cur, l);
                CV<Real, TPT> o = x;
                if (j > 1) o = ldv<Real, TPT, false>(prev, l);
#pragma unroll
                for (int t = 0; t < TPT; ++t) {
                    const Real dv = dsm[l + t];
                    Real ur = acc[i].v[2 * t], ui = acc[i].v[2 * t + 1];
                    if constexpr (!kEns) {
                        // the reference's order: alpha_j from H q_j alone (the unconjugated dot of
                        // complex states does not make q_j orthogonal to q_{j-1})
                        ur = fma(dv, x.v[2 * t], ur);
                        ui = fma(dv, x.v[2 * t + 1], ui);
                        o.v[2 * t] = fma(-fm[t], o.v[2 * t], ur);
                        o.v[2 * t + 1] = fma(-fm[t], o.v[2 * t + 1], ui);
                    } else {
                        ur = fma(dv, x.v[2 * t], fma(-fm[t], o.v[2 * t], ur));
                        ui = fma(dv, x.v[2 * t + 1], fma(-fm[t], o.v[2 * t + 1], ui));
                        o.v[2 * t] = ur;
                        o.v[2 * t + 1] = ui;
                    }
                    // the bilinear dot takes q_j itself, the Hermitian one its conjugate
                    const double xr = x.v[2 * t], xi = A.bil ? -x.v[2 * t + 1] : x.v[2 * t + 1], dr = ur, di = ui;
                    x2[t] += xr * dr + xi * di;
                    y2[t] += xr * di - xi * dr;
                }
                stv<Real, TPT>(prev, l, o);
            }
        }
        sum.template part<true>(0, x2, y2);
        sum.sync();
        for (int t = last; t < TC; t += 32) {
            const double2 a = sum.get(0, t);
            const double s = scs[j * TC + t], ar = a.x * s * s, ai = a.y * s * s;
            al[j * TC + t] = make_double2(ar, ai);
            if constexpr (sizeof(Real) == 4) {
                const float p2 = cl_pow2(s), h = (float)ar, g = (float)ai;
                *reinterpret_cast<float4*>(par + t) = make_float4(p2, -p2 * h, -p2 * (float)(ar - h), p2 * g);
                par[2 * TC + t].x = p2 * (float)(ai - g);
            } else {
                par[t] = make_double2(ar * s, ai * s);
            }
        }
        __syncthreads();
        // r_{j+1} over r_j, r_j over r_{j-1}; beta_j.  complex128: r_{j+1} = sc_j (u - alpha_j r_j).
        // complex64: the scale is the power of two below sc_j and alpha a pair of floats, so that
        // fma(-alpha_lo, r, fma(-alpha_hi, r, u)) is within an ulp of the exact difference without
        // a conversion to FP64 (16 a clock and SM: eight of them a value bound this pass)
        double2 aj[TPT];
        float4 af[TPT];
        float aq[TPT];
#pragma unroll
        for (int t = 0; t < TPT; ++t) {
            if constexpr (sizeof(Real) == 4) {
                af[t] = *reinterpret_cast<const float4*>(par + tl * TPT + t);
                aq[t] = (float)par[2 * TC + tl * TPT + t].x;
            } else {
                aj[t] = par[tl * TPT + t];
            }
            x2[t] = 0.0;
        }
        Real* out = basis(j + 1, 0);
        for (int k = rl; k < nbk; k += RL)
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int row = k * R + i;
                if (row >= nrow) break;
                const size_t l = loc(row);
                const CV<Real, TPT> x = ldv<Real, TPT, false>(cur, l);
                CV<Real, TPT> o = ldv<Real, TPT, false>(prev, l);
#pragma unroll
                for (int t = 0; t < TPT; ++t) {
                    if constexpr (sizeof(Real) == 4) {
                        const float xr = x.v[2 * t], xi = x.v[2 * t + 1];
                        float2 v = make_float2(af[t].x * o.v[2 * t], af[t].x * o.v[2 * t + 1]);   // exact
                        v = __ffma2_rn(make_float2(af[t].y, af[t].y), make_float2(xr, xi), v);
                        v = __ffma2_rn(make_float2(af[t].z, af[t].z), make_float2(xr, xi), v);
                        v = __ffma2_rn(make_float2(af[t].w, -af[t].w), make_float2(xi, xr), v);
                        if (A.bil) v = __ffma2_rn(make_float2(aq[t], -aq[t]), make_float2(xi, xr), v);
                        o.v[2 * t] = v.x;
                        o.v[2 * t + 1] = v.y;
                    } else {
                        const double xr = x.v[2 * t], xi = x.v[2 * t + 1];
                        o.v[2 * t] = (Real)(sc[t] * (double)o.v[2 * t] - (aj[t].x * xr - aj[t].y * xi));
                        o.v[2 * t + 1] = (Real)(sc[t] * (double)o.v[2 * t + 1] - (aj[t].x * xi + aj[t].y * xr));
                    }
                    const double rr = o.v[2 * t], ri = o.v[2 * t + 1];
                    x2[t] += rr * rr + ri * ri;
                }
                stv<Real, TPT>(prev, l, x);
                stv<Real, TPT>(cur, l, o);
                stv<Real, TPT>(out + (size_t)row * tca * 2, 0, o);
            }
        sum.template part<false>(1, x2, y2);
        sum.sync();
        for (int t = last; t < TC; t += 32) {
            const double b2 = sum.get(1, t).x;
            // 1 / ||r_{j+1}|| and ||r_{j+1}||; sqrt only where the reciprocal has no value
            double s1 = rsqrt(b2), nr = b2 * s1;
            if (!(b2 > 1e-290) || !(b2 < 1e290)) {
                nr = sqrt(b2);
                s1 = nr > 0.0 ? 1.0 / nr : 0.0;
            }
            // beta_j = ||H q_j - ..|| = sc_j ||r_{j+1}|| / scale (complex128: scale = sc_j)
            const double scj = scs[j * TC + t];
            double bt = nr;
            if constexpr (sizeof(Real) == 4) bt = scj != 0.0 ? nr * (scj * cl_pow2_inv(scj)) : 0.0;
            if (!isfinite(bt) && c0 + t < B && rank == 0) atomicCAS(A.S.status, 0, DQ_ERR_NAN);
            // lucky breakdown: invariant Krylov space, continue with q_{j+1} = 0
            const double bp = j > 1 ? be[(j - 1) * TC + t] : 0.0;
            const double2 a = al[j * TC + t];
            if (bt <= 2.0 * kBreakdownRel * (fabs(a.x) + fabs(a.y) + bp) &&
                bt <= kBreakdownRel * (sqrt(a.x * a.x + a.y * a.y) + bp)) {
                bt = 0.0;
                s1 = 0.0;
            }
            be[j * TC + t] = bt;
            scs[(j + 1) * TC + t] = s1;
            // beta_j sc_j / sc_{j+1}
            par[TC + t] = make_double2(s1, bt * scj * (s1 > 0.0 ? nr : 0.0));
        }
        margins(j + 1);
        __syncthreads();
        if (adaptive && j >= A.m_min && j < A.m && (j - A.m_min) % kMCheckStride == 0) {
            bool done;
            if constexpr (kResume) {
                done = cl_check<Real, TPT, R>(A, smem, W, chunk, (int)rank, CS, j);
            } else {
                const int nt = min(TC, B - c0);
                if (cl_series_check(A, al, be, W, nt, j)) {
                    __syncthreads();   // all have read the flag
                    return j;
                }
                static_assert(kMaxTC <= 64, "two trajectories a lane");
                done = __all_sync(0xffffffffu, (lane >= nt || mtr[lane] != 0) && (lane + 32 >= nt || mtr[lane + 32] != 0));
            }
            if (done) {
                jl = j;
                break;
            }
        }
    }
    // ---- the recurrence's scalars (the adjoint and the getters read them) ----
    __syncthreads();
    if (kEns && rank == 0) {
        for (int e = threadIdx.x; e < jl * TC; e += kClThreads) {
            const int j = 1 + e / TC, t = e % TC;
            if (c0 + t >= B) continue;
            const size_t k = (size_t)j * B + c0 + t;
            A.S.alpha[2 * k] = al[j * TC + t].x;
            A.S.alpha[2 * k + 1] = al[j * TC + t].y;
            A.S.beta[k] = be[j * TC + t];
            A.S.sc[k + B] = scs[(j + 1) * TC + t];
        }
    }
    if (!(A.flags & kClFinish)) {
        // the neighbours may still read this CTA's rows of the last window
        if constexpr (!kLocal && !kGrid) cl_sync();
        return 0;
    }
    // ---- ||H q_{m+1}|| ---------------------------------------------------------
    double nav = 0.0;   // set where it is used, per trajectory
    if (!adaptive) {
        double x2[TPT];
#pragma unroll
        for (int t = 0; t < TPT; ++t) x2[t] = 0.0;
        for (int k = rl; k < nbk; k += RL) {
            CV<Real, TPT> acc[R];
            product(k, acc);
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int row = k * R + i;
                if (row >= nrow) break;
                const size_t l = loc(row);
                const CV<Real, TPT> x = ldv<Real, TPT, false>(cur, l);
#pragma unroll
                for (int t = 0; t < TPT; ++t) {
                    const Real dv = dsm[l + t];
                    const double ur = fma(dv, x.v[2 * t], acc[i].v[2 * t]);
                    const double ui = fma(dv, x.v[2 * t + 1], acc[i].v[2 * t + 1]);
                    x2[t] += ur * ur + ui * ui;
                }
            }
        }
        sum.template part<false>(0, x2, x2);
        sum.sync();
    }
    // ---- exp(tau Tbar) e_1: one warp per trajectory, in every CTA -------------
    if (threadIdx.x == 0) flag = 0;
    __syncthreads();
    auto estimate = [&](int m, int t, cd e1, cd e2) {
        const double bmm = be[m * TC + t];
        // with the adaptive dimension only err1 (||H q_{m+1}|| belongs to the largest m)
        return adaptive ? fmax(fabs(bmm) * sqrt(cabs2(e1)), 1.110223e-16) : expokit_error(bmm, nav, e1, e2);
    };
    int mmax = adaptive ? 0 : A.m;
    for (int t = 0; t < TC && c0 + t < B; ++t)
        if (adaptive) mmax = max(mmax, mtr[t] ? mtr[t] : A.m);
    __syncthreads();   // before a warp below marks its trajectory
    for (int t = warp; t < TC; t += kClWarps) {
        if (c0 + t >= B) continue;
        const int m = adaptive && mtr[t] ? mtr[t] : A.m;
        const int q = (min(lane, m - 1) + 1) * TC + t;
        cd y, f1, f2;
        int s = 0;
        bool ok;
        if constexpr (kTk) {
            // the weights are the last column's, times ||A^p psi|| = 1 / sc_1
            ok = series_exp_tk(m, A.tk_p, cmk(al[q].x, al[q].y), be[q], A.tau_im, A.norm_mode, y, f1, f2);
            y = cscale(y, 1.0 / scs[TC + t]);
        } else {
            ok = series_exp_tbar(m, cmk(al[q].x, al[q].y), be[q], A.tau_im, A.norm_mode, y, f1, f2, s);
        }
        if (!ok) {
            if (lane == 0) atomicOr(&flag, 1);
            if (lane == 0) mtr[t] = -m;   // dense below
            continue;
        }
        if (lane < mmax) {
            const cd v = lane < m ? cscale(y, scs[(lane + 1) * TC + t]) : cmk(0.0, 0.0);
            yts[lane * TC + t] = make_double2(v.x, v.y);
        }
        if (!adaptive) nav = sqrt(sum.get(0, t).x) * scs[(A.m + 1) * TC + t];
        if (rank == 0 && lane == m - 1) {
            if (s < 0) atomicCAS(A.S.status, 0, DQ_ERR_SCALING);
            else if constexpr (kTk) A.tk_obs[c0 + t] = estimate(m, t, f1, f2);   // completed with the norm below
            else cl_estimate<kPlain>(A, c0 + t, estimate(m, t, f1, f2));
        }
        if (adaptive && rank == 0 && lane == 0) A.S.mtraj[c0 + t] = m;
    }
    __syncthreads();
    if (flag) {
        if constexpr (adaptive) sum.sync();   // as in the check
        else if (threadIdx.x < TC)
            par[2 * TC + threadIdx.x].x = sqrt(sum.get(0, threadIdx.x).x) * scs[(A.m + 1) * TC + threadIdx.x];
        __syncthreads();
        cl_dense_weights<Real, kMode>(A, smem, mtr, chunk, (int)rank, CS, mmax);
        sum.sync();
        for (int e = threadIdx.x; e < mmax * TC; e += kClThreads) {
            const int j = e / TC, t = e % TC;
            if (c0 + t >= B || mtr[t] >= 0) continue;
            const size_t k = (size_t)(j + 1) * B + c0 + t;
            const double* yt = kPlain ? reinterpret_cast<const double*>(A.ps->yt) : A.S.yt;
            yts[e] = make_double2(yt[2 * k], yt[2 * k + 1]);
        }
        __syncthreads();
    }
    // ---- psi = sum_j yt_j r_j over slab 1, its norm, <bra|psi> -----------------
    double nn[TPT], cr[TPT], ci[TPT], q4[TPT];
#pragma unroll
    for (int t = 0; t < TPT; ++t) nn[t] = cr[t] = ci[t] = q4[t] = 0.0;
    for (int k = rl; k < nbk; k += RL)
        for (int row = k * R; row < min(nrow, k * R + R); ++row) {
            const size_t x = glo(row);
            double pr[TPT], pi[TPT];
#pragma unroll
            for (int t = 0; t < TPT; ++t) pr[t] = pi[t] = 0.0;
            for (int j0 = 1; j0 <= mmax; j0 += 8) {
                CV<Real, TPT> v[8];
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (j0 + q <= mmax)
                        v[q] = j0 + q == 1 && !kTk ? ldv<Real, TPT, false>(first, x)
                                           : ldv<Real, TPT, false>(basis(j0 + q, row), 0);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    if (j0 + q > mmax) break;
#pragma unroll
                    for (int t = 0; t < TPT; ++t) {
                        const double2 yv = yts[(j0 + q - 1) * TC + tl * TPT + t];
                        pr[t] += yv.x * v[q].v[2 * t] - yv.y * v[q].v[2 * t + 1];
                        pi[t] += yv.x * v[q].v[2 * t + 1] + yv.y * v[q].v[2 * t];
                    }
                }
            }
            if constexpr (kTk) {
                const CV<Real, TPT> a = ldv<Real, TPT, false>(reinterpret_cast<const Real*>(smem + Y.acc), loc(row));
                pr[0] += a.v[0];
                pi[0] += a.v[1];
            }
            const cd p0 = !kPlain || A.corr_pt ? A.bra[r0 + row] : cmk(0.0, 0.0);
            CV<Real, TPT> o;
#pragma unroll
            for (int t = 0; t < TPT; ++t) {
                o.v[2 * t] = (Real)pr[t];
                o.v[2 * t + 1] = (Real)pi[t];
                const double vr = o.v[2 * t], vi = o.v[2 * t + 1];
                nn[t] += vr * vr + vi * vi;
                cr[t] += p0.x * vr + p0.y * vi;   // conj(bra) * psi
                ci[t] += p0.x * vi - p0.y * vr;
                if (kTk) q4[t] += (vr * vr + vi * vi) * (vr * vr + vi * vi);
            }
            if (kPlain || kTk) stv<Real, TPT>(prev, loc(row), o);   // its norm is not known yet
            else stv<Real, TPT>(slab(1), x, o);
        }
    // ex[0] still holds ||H q_{m+1}||, which slower CTAs may be reading
    if constexpr (kGrid) __syncthreads();
    else sum.sync();
    sum.template part<true>(0, cr, ci);
    sum.template part<kTk>(1, nn, q4);
    sum.sync();
    if constexpr (kTk) {
        if (act) {
            const double inv = 1.0 / sqrt(sum.get(1, tl).x);
            for (int k = rl; k < nbk; k += RL) {
                const CV<Real, TPT> v = ldv<Real, TPT, false>(prev, loc(k));
                A.psi_out[glo(k)] = cmk(v.v[0] * inv, v.v[1] * inv);
            }
        }
        if (rank == 0 && threadIdx.x < TC && c0 + (int)threadIdx.x < B) {
            const int t = threadIdx.x, b = c0 + t;
            const double2 n2 = sum.get(1, t), c = sum.get(0, t);
            const double nrm = sqrt(n2.x), inv = 1.0 / nrm;
            if (!(nrm > 0.0) || !isfinite(nrm)) atomicCAS(A.S.status, 0, DQ_ERR_NAN);
            // taylorKrylovClass.cu:417-434: the B part's estimate plus |1 - norm|
            double est = A.tk_obs[b] + fabs(1.0 - nrm);
            if (est < 1.110223e-16) est = 1.110223e-16;
            A.erracc[b] += est;
            A.tk_obs[b] = c.x * inv;
            A.tk_obs[B + b] = c.y * inv;
            A.tk_obs[2 * B + b] = n2.y * (inv * inv) * (inv * inv);
        }
    } else if constexpr (kPlain) {
        const double n2 = sum.get(1, 0).x, nrm = sqrt(n2), inv = 1. / nrm;
        for (int k = rl; k < nbk; k += RL)
            for (int row = k * R; row < min(nrow, k * R + R); ++row) {
                const CV<Real, TPT> v = ldv<Real, TPT, false>(prev, loc(row));
                const cd o = cmk(v.v[0] * inv, v.v[1] * inv);
                A.psi_out[r0 + row] = o;
                if (A.pops_row) A.pops_row[r0 + row] += cabs2(o);
            }
        if (rank == 0 && threadIdx.x == 0) {
            A.ps->norm = nrm;
            A.ps->invnorm = inv;
            if (!(nrm > 0.0) || !isfinite(nrm)) atomicCAS(&A.ps->status, 0, DQ_ERR_NAN);
            if (A.corr_pt) {
                const double2 c = sum.get(0, 0);
                A.corr_pt->x += c.x * inv;
                A.corr_pt->y += c.y * inv;
            }
        }
        if constexpr (kGrid) sum.leave();
    } else if (rank == 0) {
        double* cs = reinterpret_cast<double*>(sum.red);   // free again: the chunk's correlation terms
        if (threadIdx.x < TC) {
            const int t = threadIdx.x, b = c0 + t;
            double sr = 0.0, si = 0.0;
            if (b < B) {
                const double n2 = sum.get(1, t).x;
                const double2 c = sum.get(0, t);
                const double s1 = 1.0 / sqrt(n2);
                A.S.norm2[b] = n2;
                A.S.sc[(size_t)B + b] = s1;   // next step's q_1 = psi / ||psi||
                if (!(n2 > 0.0) || !isfinite(n2)) atomicCAS(A.S.status, 0, DQ_ERR_NAN);
                sr = c.x * s1;
                si = c.y * s1;
            }
            cs[2 * t] = sr;
            cs[2 * t + 1] = si;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double sr = 0.0, si = 0.0;
            for (int t = 0; t < TC; ++t) {
                sr += cs[2 * t];
                si += cs[2 * t + 1];
            }
            double* cp = A.S.corr + ((size_t)(*A.S.step + 1) * A.chunks + chunk) * 2;
            cp[0] = sr;
            cp[1] = si;
        }
    }
    return 0;
}

template <typename Real, int TPT, int R, bool kLocal, int kMode = kEnsemble>
__global__ void __launch_bounds__(kClThreads, 1) k_cluster_step(const __grid_constant__ ClusterArgs A) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ ClWords W;
    const int left = cl_step<Real, TPT, R, kLocal, kMode, false>(A, smem, W, 0);
    if constexpr (kMode == kAdaptive)
        if (left) cl_step<Real, TPT, R, kLocal, kAdaptive, true>(A, smem, W, left);
}

// ---------------------------------------------------------------------------
using ClKernel = void (*)(const ClusterArgs);

template <typename Real, int TPT, int R>
static ClKernel cl_pick(bool local, bool adaptive) {
    if (adaptive) return local ? k_cluster_step<Real, TPT, R, true, kAdaptive> : k_cluster_step<Real, TPT, R, false, kAdaptive>;
    return local ? k_cluster_step<Real, TPT, R, true> : k_cluster_step<Real, TPT, R, false>;
}

static ClKernel cl_kernel(bool mixed, int tpt, int R, bool local, bool adaptive) {
    if (mixed && tpt != 2) return nullptr;
    switch (R) {
        case 1: return mixed ? cl_pick<float, 2, 1>(local, adaptive) : cl_pick<double, 1, 1>(local, adaptive);
        case 2: return mixed ? cl_pick<float, 2, 2>(local, adaptive) : cl_pick<double, 1, 2>(local, adaptive);
        case 3: return mixed ? cl_pick<float, 2, 3>(local, adaptive) : nullptr;
        case 4: return mixed ? nullptr : cl_pick<double, 1, 4>(local, adaptive);
        default: return nullptr;
    }
}

static const ::BlockFmt& cl_fmt(const BatchedState* bs, int R) {
    return bs->fmt[R == 1 ? 0 : R == 2 ? 1 : R == 3 ? 2 : 3];
}

static int cl_rows(int n, int CS, int R) {
    const int rpc = (n + CS - 1) / CS;
    return (rpc + R - 1) / R * R;
}

static cudaLaunchConfig_t cl_config(int chunks, int CS, size_t smem, cudaStream_t st, cudaLaunchAttribute* at) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(chunks * CS);
    cfg.blockDim = dim3(kClThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = CS;
    at->val.clusterDim.y = 1;
    at->val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

// Bytes of the largest CTA's coupling records (block starts, columns, coefficients).
static size_t cl_rec_bytes(const ::BlockFmt& f, bool mixed, int rpc, int R, int TL) {
    const size_t per = 32 / TL, nb = rpc / R, slots = (nb + per - 1) / per * per * (size_t)f.max_block;
    const size_t head = cl_rec_head(nb, (int)per);
    if (mixed) return head + slots * 16;
    return head + (slots * 4 + 15) / 16 * 16 + slots * R * sizeof(double);
}

// Clusters of this shape that the device holds at once (0: it cannot run);
// *smem its dynamic shared memory, *rec the part that holds the records (0
// when they do not fit).
static int cluster_resident(dq_ctx* c, int tc, int tpt, int CS, int R, const ::BlockFmt& f, size_t* smem, size_t* rec) {
    const BatchedState* bs = c->bat;
    const int n = c->n, m = c->cfg.m;
    if (CS < 1 || CS > kClMaxCtas) return 0;
    if (tc < tpt || tc > kMaxTC || tc % tpt || ((tc / tpt) & (tc / tpt - 1)) || tc / tpt > 32) return 0;
    ClKernel k = cl_kernel(bs->mixed, tpt, R, CS == 1, bs->s.mtraj != nullptr);
    if (!k) return 0;
    const size_t rsz = bs->mixed ? sizeof(float) : sizeof(double);
    const int rpc = cl_rows(n, CS, R);
    size_t rb = cl_rec_bytes(f, bs->mixed, rpc, R, tc / tpt);
    size_t sm = cl_layout(n, CS, tc, m, rpc, c->bw, rsz, rb).total;
    if (sm > kClSmemMax) {
        rb = 0;
        sm = cl_layout(n, CS, tc, m, rpc, c->bw, rsz, 0).total;
    }
    if (sm > kClSmemMax) return 0;
    // the dense exponential's matrices, in the place of the window and what follows it
    const size_t win = cl_layout(n, CS, tc, m, rpc, c->bw, rsz, 0).win;
    sm = std::max(sm, win + cl_dense_bytes(kClSmemMax - win, m + 2, (std::min(tc, bs->B) + CS - 1) / CS));
    int found = 0;
    auto prepare = [&](ClKernel f) {
        return raise_smem_limit(f, (int)kClSmemMax) == cudaSuccess &&
               (CS <= 8 || cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess);
    };
    // the iterations alone never check: they run the other kernel
    if (prepare(k) && prepare(cl_kernel(bs->mixed, tpt, R, CS == 1, false))) {
        cudaLaunchAttribute at;
        const cudaLaunchConfig_t cfg = cl_config(1, CS, sm, nullptr, &at);
        if (cudaOccupancyMaxActiveClusters(&found, k, &cfg) != cudaSuccess) found = 0;
    }
    cudaGetLastError();
    *smem = sm;
    *rec = rb;
    return found;
}

// The shape with the least estimated SM cycles of one Lanczos iteration over
// CTAs per cluster and trajectories per chunk (R rows per block, its blocks
// built), and the estimate for the choice between this form and the grid-wide
// ones.  An iteration is a fixed part (two reductions with their barriers, the
// margins' round trip), the shared-memory wavefronts of the gathers and records
// (records read through L1: a wavefront each) and the elementwise part; times
// the waves of clusters that the device needs.  Measured against it on a B200
// (us per iteration): 4096 sites x 128, 8 couplings per row, 4 CTAs x 4
// trajectories 8.0 (model 8.1); 4731 x 100, 28 couplings, 9 x 8 13.8 (13.0).
// It orders shapes; those within 10 % change places with the matrix.
//
// complex64: 1.1 to 1.7 times the model over 80 ensembles (700 to 15,000 sites,
// 2 to 78 couplings, 16 to 320 trajectories), much like the grid-wide estimate
// (0.6 to 1.2), so the two are compared as they are.  complex128: 1.3 to 3
// times, most where a thread has many rows of few couplings (a row's chain of
// FP64 operations is not hidden), so the choice takes an estimate fitted to 80
// such ensembles (within 27 %, standard deviation 10 %): a base, 3.8 cycles a
// row of a thread (4.8 with one trajectory a chunk), 0.26 a gathered value,
// 1.6 a record.
double cluster_plan(dq_ctx* c, int R, int* tc_out, int* cs_out) {
    const BatchedState* bs = c->bat;
    const ::BlockFmt& f = cl_fmt(bs, R);
    const int n = c->n, B = bs->B, tpt = bs->mixed ? 2 : 1;
    const double len = (double)f.nunion / std::max(1, f.nb), csz = bs->mixed ? 8.0 : 16.0;
    double best = 1e30, est = 1e30;
    for (int CS = 1; CS <= kClMaxCtas; ++CS) {
        const int rpc = cl_rows(n, CS, R);
        if (CS > 1 && (size_t)rpc * (CS - 1) >= (size_t)n) continue;   // a CTA without rows
        for (int tc = tpt; tc <= 32 && tc < 2 * B; tc *= 2) {
            const int chunks = (B + tc - 1) / tc, TL = tc / tpt;
            // threads with a block to do set the pace when there are fewer than the CTA has
            const double nbk = rpc / R, rounds = std::ceil(nbk * TL / kClThreads) * kClThreads / (nbk * TL);
            const double gather = nbk * len * tc * csz / 128.0 * 1.3;
            const double elem = (double)rpc * tc * (bs->mixed ? 1.2 : 0.8) * std::min(rounds, 1.5);
            auto cycles = [&](bool in_smem) {
                return 5500.0 + 60.0 * CS + 1.6 * (gather + nbk * len * (in_smem ? 0.125 * (bs->mixed ? 1 : R) : 0.8)) +
                       elem;
            };
            if (cycles(true) >= best) continue;
            size_t smem = 0, rec = 0;
            const int fit = cluster_resident(c, tc, tpt, CS, R, f, &smem, &rec);
            if (fit < 1) continue;
            const int waves = (chunks + fit - 1) / fit;
            const double t = waves * cycles(rec > 0);
            if (t < best) {
                best = t;
                est = bs->mixed ? t
                                : waves * (4400.0 + (tc == 1 ? 4.84 : 3.83) * R * kClThreads * std::ceil(nbk * TL / kClThreads) +
                                           0.262 * nbk * len * tc + 1.58 * nbk * len);
                *tc_out = tc;
                *cs_out = CS;
            }
        }
    }
    return est;
}

// One cluster launch: the whole step (flags kClNoise | kClFinish), or the
// Lanczos iterations of a given slab 1 and diagonal alone (flags 0), all m of
// them whether or not the ensemble chooses its dimension.
cudaError_t cluster_launch(dq_ctx* c, bool whole_step, const ZZBlockRef& zz) {
    BatchedState* bs = c->bat;
    const ::BlockFmt& f = cl_fmt(bs, bs->R);
    ClusterArgs a = {};
    a.n = c->n;
    a.B = bs->B;
    a.TC = bs->TC;
    a.rpc = bs->rpc;
    a.bw = c->bw;
    a.rec_smem = (int)bs->cl_rec;
    a.m = c->cfg.m;
    a.flags = whole_step ? kClNoise | kClFinish : 0;
    a.bil = c->cfg.dot_mode == DQ_DOT_BILINEAR;
    a.chunks = bs->chunks;
    a.bptr = f.bptr;
    a.bcol = f.bcol;
    a.bcoef = f.bcoef;
    a.slabs = bs->slabs;
    a.slab = (size_t)c->n * bs->B;
    a.diag = bs->diag;
    a.S = bs->s;
    a.noise = c->cfg.noise_model;
    a.ns = c->cfg.ka_substeps > 0 ? c->cfg.ka_substeps : 1;
    a.traj0 = c->traj0;
    a.subdt = c->cfg.dt / (double)a.ns;
    a.sqrt_subdt = sqrt(a.subdt);
    a.seed = c->cfg.seed;
    a.sigma = c->d_sigma;
    a.invtau = c->d_invtau;
    a.coeff = c->d_coeff;
    a.eps = bs->eps;
    a.deps = bs->deps;
    a.zzD = zz.D;
    a.zz_start = zz.start;
    a.norm_mode = c->cfg.norm_mode;
    a.m_min = c->cfg.m_min;
    a.tol = c->cfg.m_tol > 0 ? c->cfg.m_tol : 1e-7;
    a.tau_im = c->tau_im;
    a.erracc = c->d_erracc;
    a.bra = corr_bra(c);
    a.scratch = static_cast<unsigned char*>(bs->cl_scratch);
    a.scratch_stride = pade_mats_bytes(c->cfg.m + 2);
    a.smem = (int)bs->win_smem;
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = cl_config(bs->chunks, bs->ctas_per_sm, bs->win_smem, c->stream, &at);
    const bool adaptive = whole_step && bs->s.mtraj != nullptr;
    return cudaLaunchKernelEx(&cfg, cl_kernel(bs->mixed, bs->TPT, bs->R, bs->ctas_per_sm == 1, adaptive), a);
}

// Shapes `bs` for the cluster form (its coupling blocks of R rows exist).
dq_status cluster_set(dq_ctx* c, int tc, int tpt, int CS, int R) {
    BatchedState* bs = c->bat;
    size_t smem = 0, rec = 0;
    if (cluster_resident(c, tc, tpt, CS, R, cl_fmt(bs, R), &smem, &rec) < 1) return DQ_ERR_ARG;
    const int chunks = (bs->B + tc - 1) / tc;
    const size_t win = cl_layout(c->n, CS, tc, c->cfg.m, cl_rows(c->n, CS, R), c->bw,
                                 bs->mixed ? sizeof(float) : sizeof(double), 0).win;
    const size_t mats = pade_mats_bytes(c->cfg.m + 2), need = win + mats <= smem ? 0 : mats * chunks * std::min(CS, tc);
    if (need > bs->cl_scratch_bytes) {
        cudaFree(bs->cl_scratch);
        bs->cl_scratch = nullptr;
        bs->cl_scratch_bytes = 0;
        dq_status st = check_cuda(c, cudaMalloc(&bs->cl_scratch, need), "cluster scratch");
        if (st) {
            cudaGetLastError();   // the caller may go on with another form
            return st;
        }
        bs->cl_scratch_bytes = need;
    }
    bs->TC = tc;
    bs->TPT = tpt;
    bs->chunks = chunks;
    bs->ctas_per_sm = CS;
    bs->R = R;
    bs->rpc = cl_rows(c->n, CS, R);
    bs->gx = bs->gxs = CS;
    bs->win_smem = smem;
    bs->cl_rec = rec;
    bs->staged = kStagedCluster;
    bs->groups = 1;
    return DQ_OK;
}

// ---- the drop-in step ------------------------------------------------------
// A single trajectory: rows of the off-diagonal CSR as they are (R = 1), a
// thread each, the records in shared memory where a CTA's turn out to fit (the
// kernel looks).  `bw` is the matrix bandwidth, or n where only the device
// knows the columns (then every CTA's window is the whole vector); `z` the
// couplings of a row, 0 when unknown; `fit` what the device can hold of it at
// once (a launch beyond that would be refused, or wait for itself).  ctas = 0:
// no shape fits, the step takes several launches.
// Estimated cycles of an iteration: rounds of rows by the CTA's threads, the
// wavefronts of the records and gathers (7 per 32 entries), the barriers.
PlainCluster plain_cluster_plan(int n, int m, int bw, double z, const PlainFit& fit) {
    PlainCluster best;
    double t_best = 1e30;
    for (int CS = 1; CS <= std::min(kClMaxCtas, fit.cluster); ++CS) {
        const int rpc = cl_rows(n, CS, 1);
        if (CS > 1 && ((size_t)rpc * (CS - 1) >= (size_t)n || rpc < 32)) continue;
        const size_t fixed = cl_layout(n, CS, 1, m, rpc, bw, sizeof(double), 0).total;
        if (fixed + 4096 > kClSmemMax) continue;
        const size_t room = (kClSmemMax - fixed) / 16 * 16 - 16;
        const double zz = z > 0.0 ? z : 8.0;
        if (rpc * (zz * 1.15 + 2.0) * 12.0 > (double)room) continue;
        // unknown rows may be long: as many CTAs as there are rows for, so that their records fit
        const double t = z > 0.0 ? std::ceil((double)rpc / kClThreads) * (400.0 + 75.0 * z) + 0.25 * rpc * z +
                                       (CS > 1 ? 700.0 + 60.0 * CS : 0.0)
                                 : std::abs(rpc - 128.0);
        if (t < t_best) {
            t_best = t;
            best.ctas = CS;
            best.rpc = rpc;
            best.smem = fixed + room;
            best.rec = room;
        }
    }
    // Larger systems: a cooperative grid, of as few CTAs as hold the records and give every row a
    // thread (fewer have a cheaper barrier, and steps of other streams run beside them).  Its two
    // barriers take about 4500 of an iteration's 14,800 cycles each (30,000 sites with 28 couplings,
    // m = 20: 184 us a step as 2 m + 5 launches, 91 us this way, three states in turn)
    if (z > 0.0) {
        for (int G = kClMaxCtas + 1; G <= std::min(fit.grid, kPlainGridMax); ++G) {
            const int rpc = cl_rows(n, G, 1);
            if (rpc > kClThreads) continue;
            const size_t fixed = cl_layout(n, 2, 1, m, rpc, bw, sizeof(double), 0).total;
            if (fixed + 4096 > kClSmemMax || rpc * (z * 1.15 + 2.0) * 12.0 > (double)(kClSmemMax - fixed - 4096)) continue;
            const double t = 400.0 + 75.0 * z + 0.25 * rpc * z + 6500.0;
            if (t < t_best) {
                best.ctas = (n + rpc - 1) / rpc;
                best.rpc = rpc;
                best.rec = (kClSmemMax - fixed) / 16 * 16 - 16;
                best.smem = fixed + best.rec;
            }
            break;
        }
    }
    return best;
}

// After plain_cluster_attributes, for the current device.
PlainFit plain_cluster_fit() {
    PlainFit f;
    int dev = 0, sms = 0, per = 0;
    for (int CS = kClMaxCtas; CS >= 1 && f.cluster == 0; --CS) {
        cudaLaunchAttribute at;
        const cudaLaunchConfig_t cfg = cl_config(1, CS, kClSmemMax, nullptr, &at);
        int found = 0;
        const void* k = CS == 1 ? (const void*)k_cluster_step<double, 1, 1, true, kDropIn>
                                : (const void*)k_cluster_step<double, 1, 1, false, kDropIn>;
        if (cudaOccupancyMaxActiveClusters(&found, k, &cfg) == cudaSuccess && found > 0) f.cluster = CS;
    }
    if (cudaGetDevice(&dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_cluster_step<double, 1, 1, false, kDropInGrid>, kClThreads,
                                                      kClSmemMax) == cudaSuccess)
        f.grid = sms * per;
    cudaGetLastError();   // a query that was refused leaves its part at 0
    return f;
}

cudaError_t cluster_set_wait_cycles(long long cycles) {
    return cudaMemcpyToSymbol(g_cl_wait_cycles, &cycles, sizeof(cycles));
}

cudaError_t plain_cluster_attributes() {
    cudaError_t e = raise_smem_limit(k_cluster_step<double, 1, 1, true, kDropIn>, (int)kClSmemMax);
    if (e == cudaSuccess) e = raise_smem_limit(k_cluster_step<double, 1, 1, false, kDropIn>, (int)kClSmemMax);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_cluster_step<double, 1, 1, false, kDropIn>,
                                 cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = raise_smem_limit(k_cluster_step<double, 1, 1, false, kDropInGrid>, (int)kClSmemMax);
    return e;
}

cudaError_t plain_cluster_launch(const PlainCluster& P, const PlainStep& q, cudaStream_t st) {
    ClusterArgs a = {};
    a.n = q.n;
    a.B = 1;
    a.TC = 1;
    a.rpc = P.rpc;
    a.bw = q.bw;
    a.m = q.m;
    a.flags = kClFinish | (q.draw ? kClNoise : 0);
    a.bil = q.dot_mode == DQ_DOT_BILINEAR;
    a.chunks = 1;
    a.rec_smem = (int)P.rec;
    a.bptr = q.rowptr;
    a.bcol = q.col;
    a.bcoef = q.val;
    a.slabs = q.Q;
    a.slab = (size_t)q.n;
    a.diag = q.diag;
    a.S.status = &q.ps->status;
    a.noise = q.noise;
    a.ns = q.ns;
    a.traj0 = q.traj;
    a.step = q.step;
    a.subdt = q.subdt;
    a.sqrt_subdt = sqrt(q.subdt);
    a.seed = q.seed;
    a.sigma = q.sigma;
    a.invtau = q.invtau;
    a.coeff = q.coeff;
    a.eps = q.eps;
    a.deps = q.deps;
    a.norm_mode = q.norm_mode;
    a.tau_im = q.tau_im;
    a.erracc = q.erracc;
    a.bra = q.bra;
    a.psi_in = q.psi_in;
    a.psi_out = q.psi_out;
    a.pops_row = q.pops_row;
    a.corr_pt = q.corr_pt;
    a.ps = q.ps;
    a.grid = q.grid;
    a.smem = (int)P.smem;   // always room for the dense exponential: one trajectory's scalars take 3 KB
    cudaLaunchAttribute at;
    cudaLaunchConfig_t cfg = cl_config(1, P.ctas, P.smem, st, &at);
    if (P.ctas > kClMaxCtas) {
        // every CTA resident at once: they wait for one another
        at.id = cudaLaunchAttributeCooperative;
        at.val.cooperative = 1;
        return cudaLaunchKernelEx(&cfg, k_cluster_step<double, 1, 1, false, kDropInGrid>, a);
    }
    return cudaLaunchKernelEx(&cfg, P.ctas == 1 ? k_cluster_step<double, 1, 1, true, kDropIn>
                                                : k_cluster_step<double, 1, 1, false, kDropIn>, a);
}

// ---- Taylor-Krylov steps of an ensemble --------------------------------------
// The shape of n sites on CS CTAs with tc trajectories (false: it does not fit):
// rows per CTA, shared memory, the part of it left for the records.  The kernel
// decides whether a CTA's records fit there; where not even their block starts
// do, none is asked for and all is read through L1.
bool taylor_cluster_shape(int n, int CS, int tc, int mb, int bw, TaylorCluster* P) {
    const int rpc = cl_rows(n, CS, 1);
    if (CS > 1 && (size_t)rpc * (CS - 1) >= (size_t)n) return false;
    const size_t fixed = cl_layout(n, CS, tc, mb, rpc, bw, sizeof(double), 0, true).total;
    if (fixed + 4096 > kClSmemMax) return false;
    const size_t room = (kClSmemMax - fixed) / 16 * 16 - 16;
    P->ctas = CS;
    P->tc = tc;
    P->rpc = rpc;
    P->rec = cl_rec_head(rpc, 32 / tc) <= room ? room : 0;
    P->smem = fixed + P->rec;
    return true;
}

size_t taylor_cluster_head(const TaylorCluster& P) { return cl_rec_head(P.rpc, 32 / P.tc); }

// CTAs and trajectories of a cluster for n sites x B trajectories, z couplings
// per row of the larger matrix and bandwidth bw, by cluster_plan's estimate;
// ctas = 0: nothing fits.
TaylorCluster taylor_cluster_plan(int n, int B, int mb, int p, int bw, double z) {
    TaylorCluster best;
    double t_best = 1e30;
    ClKernel local = k_cluster_step<double, 1, 1, true, kTaylor>, wide = k_cluster_step<double, 1, 1, false, kTaylor>;
    if (raise_smem_limit(local, (int)kClSmemMax) != cudaSuccess || raise_smem_limit(wide, (int)kClSmemMax) != cudaSuccess ||
        cudaFuncSetAttribute(wide, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return best;
    }
    for (int CS = 1; CS <= kClMaxCtas; ++CS) {
        int fit = 0;   // one CTA per SM whatever its shared memory: resident clusters depend on CS alone
        for (int tc = 1; tc <= 32 && tc < 2 * B; tc *= 2) {
            TaylorCluster P;
            if (!taylor_cluster_shape(n, CS, tc, mb, bw, &P)) continue;
            const int rpc = P.rpc;
            const bool in_smem = rpc * (z * 1.15 + 2.0) * 12.0 <= (double)P.rec;
            P.chunks = (B + tc - 1) / tc;
            const double cycles = 5500.0 + 60.0 * CS +
                                  1.6 * (rpc * z * tc * 16.0 / 128.0 * 1.3 + rpc * z * (in_smem ? 0.125 : 1.6)) +
                                  0.8 * rpc * tc;
            if (cycles >= t_best) continue;
            if (!fit) {
                cudaLaunchAttribute at;
                const cudaLaunchConfig_t cfg = cl_config(1, CS, kClSmemMax, nullptr, &at);
                if (cudaOccupancyMaxActiveClusters(&fit, CS == 1 ? local : wide, &cfg) != cudaSuccess || fit < 1) {
                    cudaGetLastError();
                    fit = -1;
                }
            }
            if (fit < 1) continue;
            const double t = cycles * ((P.chunks + fit - 1) / fit);
            if (t < t_best) {
                t_best = t;
                best = P;
            }
        }
    }
    if (best.ctas) {
        // the dense exponential's matrices: in the place of the window and what follows it, or in global memory
        const size_t win = cl_layout(n, best.ctas, best.tc, mb, best.rpc, bw, sizeof(double), 0, true).win;
        const size_t mats = pade_mats_bytes(mb + p);
        if (win + mats <= kClSmemMax) best.smem = std::max(best.smem, win + mats);
        else best.scratch = mats * best.chunks * std::min(best.ctas, best.tc);
    }
    return best;
}

cudaError_t taylor_cluster_launch(const TaylorCluster& P, const TaylorStep& q, cudaStream_t st) {
    ClusterArgs a = {};
    a.n = q.n;
    a.B = q.B;
    a.TC = P.tc;
    a.rpc = P.rpc;
    a.bw = q.bw;
    a.m = q.mb;
    a.flags = kClFinish | kClNoise;
    a.bil = q.dot_mode == DQ_DOT_BILINEAR;
    a.chunks = P.chunks;
    a.rec_smem = (int)P.rec;
    a.bptr = q.rowptr;
    a.bcol = q.col;
    a.bcoef = q.val;
    a.slabs = q.Q;
    a.slab = (size_t)q.n * q.B;
    a.diag = q.diag;
    a.S.status = q.status;
    a.S.yt = q.yt;
    a.noise = q.noise;
    a.ns = q.ns;
    a.traj0 = q.traj0;
    a.step = q.step;
    a.subdt = q.subdt;
    a.sqrt_subdt = sqrt(q.subdt);
    a.seed = q.seed;
    a.sigma = q.sigma;
    a.invtau = q.invtau;
    a.coeff = q.coeff;
    a.eps = q.eps;
    a.deps = q.deps;
    if (q.noise == DQ_NOISE_ZZ) a.flags = kClFinish;   // the diagonal is drawn by a launch of its own
    a.norm_mode = q.norm_mode;
    a.tau_im = q.tau_im;
    a.erracc = q.erracc;
    a.bra = q.bra;
    a.psi_in = q.psi;
    a.psi_out = q.psi;
    a.tk_p = q.p;
    a.b_ptr = q.b_rowptr;
    a.b_col = q.b_col;
    a.b_val = q.b_val;
    a.b_diag = q.b_diag;
    for (int k = 0; k < q.p; ++k) a.tk_coef[k] = q.coef[k];
    a.tk_obs = q.obs;
    a.smem = (int)P.smem;
    a.scratch = q.scratch;
    a.scratch_stride = pade_mats_bytes(q.mb + q.p);
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = cl_config(P.chunks, P.ctas, P.smem, st, &at);
    return cudaLaunchKernelEx(&cfg, P.ctas == 1 ? k_cluster_step<double, 1, 1, true, kTaylor>
                                                : k_cluster_step<double, 1, 1, false, kTaylor>, a);
}

}  // namespace dq
