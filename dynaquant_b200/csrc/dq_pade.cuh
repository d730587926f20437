// dq_pade.cuh — exp(tau * Tbar) of the augmented Lanczos matrix for one
// trajectory, computed by one CTA in shared memory in FP64.
//
// Reference: padeClass.cu:206-487 (Padé(6,6) odd/even form, Zgemm/Zgeam +
// CULA Zgesv), padeClass.cu:585-706 (scaling by the row-sum infinity norm and
// repeated squaring), gpuLanczosHelper.cu:14-60 (augmented Tbar, EXPOKIT
// Theorem 1), padeClass.cu:750-782 (EXPOKIT Algorithm 3.2 error estimate).
// Here the whole chain runs in one CTA: the (m+2)^2 matrices live in shared
// memory, the quotient is solved by our own LU with partial pivoting, and
// nothing returns to the host.
#pragma once
#include "dq_common.cuh"

namespace dq {

constexpr int kMaxM = 32;            // Krylov dimension limit
constexpr int kMaxL = kMaxM + 2;     // augmented size
// beta_j <= kBreakdownRel * (|alpha_j| + beta_{j-1}) is treated as an exact
// (lucky) Lanczos breakdown: beta_j = 0 and q_{j+1} = 0 from there on.
constexpr double kBreakdownRel = 1e-12;

// Padé(6,6) coefficients c_k = c_{k-1} (p+1-k)/((2p+1-k) k), p = 6
// (padeClass.cu:161-168), evaluated in the same order on the host.
struct PadeCoeffs { double c[7]; };

__host__ __device__ inline PadeCoeffs pade_coeffs() {
    PadeCoeffs P;
    P.c[0] = 1.0;
    for (int k = 1; k <= 6; ++k) {
        double fk = (double)k;
        P.c[k] = P.c[k - 1] * (6.0 + 1. - fk) / ((2 * 6.0 + 1. - fk) * fk);
    }
    return P;
}

// The threads that work on one matrix: a CTA, or one of up to kMaxTeams parts
// of a CTA (whole warps, `size` threads each) with a named barrier of its own,
// so that a CTA can take several matrices at once.
constexpr int kMaxTeams = 8;
struct CtaTeam {
    __device__ __forceinline__ int id() const { return 0; }
    __device__ __forceinline__ int rank() const { return threadIdx.x; }
    __device__ __forceinline__ int size() const { return blockDim.x; }
    __device__ __forceinline__ void sync() const { __syncthreads(); }
};
struct WarpsTeam {
    int id_, size_;
    __device__ __forceinline__ int id() const { return id_; }
    __device__ __forceinline__ int rank() const { return threadIdx.x - id_ * size_; }
    __device__ __forceinline__ int size() const { return size_; }
    __device__ __forceinline__ void sync() const {
        asm volatile("barrier.sync %0, %1;" ::"r"(id_ + 1), "r"(size_) : "memory");
    }
};

__host__ __device__ inline size_t pade_mats_bytes(int L) { return sizeof(cd) * 6 * (size_t)L * L; }
__host__ __device__ inline size_t pade_smem_bytes(int L) { return pade_mats_bytes(L) + 64 * sizeof(double); }

// C = A * B (L x L row-major, shared memory), all threads of the team.
template <class Team>
__device__ __forceinline__ void sm_matmul(const Team& T, int L, const cd* A, const cd* B, cd* C) {
    for (int e = T.rank(); e < L * L; e += T.size()) {
        int i = e / L, j = e - i * L;
        cd s = cmk(0, 0);
        for (int k = 0; k < L; ++k) s = cadd(s, cmul(A[i * L + k], B[k * L + j]));
        C[e] = s;
    }
    T.sync();
}

struct PadeOut {
    int s;          // squarings (or -1 when s would reach 50, or -2 singular)
    cd e_m1_m;      // E(m-1, m)
    cd e_m1_mp1;    // E(m-1, m+1)
};

// E = exp(A) for the L x L complex matrix A held in the first L*L entries of
// smem_raw (6 L^2 complex values): Padé(6,6) in the odd/even form with scaling
// by the row-sum infinity norm (norm_mode 0: |Re|-only sums as
// padeClass.cu:585-706; 1: complex modulus) and repeated squaring.  Returns the number of squarings s (or -1 when s would reach 50,
// -2 for a singular quotient) and sets *E_out to the result (A itself or the
// second buffer).  All threads of the team call it and all return s; the team
// syncs before its next call.
template <class Team>
__device__ __forceinline__ int pade_exp_team(const Team& T, int L, int norm_mode, unsigned char* smem_raw, cd** E_out) {
    const int LL = L * L;
    cd* A = reinterpret_cast<cd*>(smem_raw);
    cd* A2 = A + LL;
    cd* A4 = A2 + LL;
    cd* A6 = A4 + LL;
    cd* U = A6 + LL;
    cd* D = U + LL;
    __shared__ int sh[kMaxTeams][3];
    int& s_sh = sh[T.id()][0];
    int& piv_sh = sh[T.id()][1];
    int& fail_sh = sh[T.id()][2];
    const int rank = T.rank(), size = T.size();

    const PadeCoeffs P = pade_coeffs();
    if (rank == 0) fail_sh = 0;
    T.sync();

    // scaling: s = number of halvings until the row-sum norm is <= 0.5
    if (rank < 32) {
        double mx = 0.0;
        for (int i = rank; i < L; i += 32) {
            double rs = 0.0;
            for (int j = 0; j < L; ++j) {
                cd a = A[i * L + j];
                rs += norm_mode == 0 ? fabs(a.x) : sqrt(cabs2(a));
            }
            mx = fmax(mx, rs);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (rank == 0) {
            int s = 0;
            double nrm = mx;
            while (nrm > 0.5 && s < 60) { nrm *= 0.5; s++; }
            s_sh = s;
        }
    }
    T.sync();
    const int s = s_sh;
    *E_out = A;
    if (s >= 50) return -1;
    if (s > 0) {
        double sc = ldexp(1.0, -s);
        for (int e = rank; e < LL; e += size) A[e] = cscale(A[e], sc);
        T.sync();
    }
    sm_matmul(T, L, A, A, A2);
    sm_matmul(T, L, A2, A2, A4);
    sm_matmul(T, L, A2, A4, A6);
    // odd part U = A (c1 I + c3 A^2 + c5 A^4); the bracket goes to D first
    for (int e = rank; e < LL; e += size) {
        int i = e / L, j = e - i * L;
        cd t = cadd(cscale(A2[e], P.c[3]), cscale(A4[e], P.c[5]));
        if (i == j) t.x += P.c[1];
        D[e] = t;
    }
    T.sync();
    sm_matmul(T, L, A, D, U);
    // even part V = c0 I + c2 A^2 + c4 A^4 + c6 A^6; D = V - U
    for (int e = rank; e < LL; e += size) {
        int i = e / L, j = e - i * L;
        cd t = cadd(cadd(cscale(A2[e], P.c[2]), cscale(A4[e], P.c[4])), cscale(A6[e], P.c[6]));
        if (i == j) t.x += P.c[0];
        D[e] = csub(t, U[e]);
    }
    T.sync();

    // LU with partial pivoting: D X = U, X overwrites U (stands in for
    // culaDeviceZgesv, padeClass.cu:715-745)
    for (int k = 0; k < L; ++k) {
        if (rank < 32) {
            double best = -1.0;
            int bi = k;
            for (int i = k + rank; i < L; i += 32) {
                double v = cabs2(D[i * L + k]);
                if (v > best) { best = v; bi = i; }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                double ob = __shfl_xor_sync(0xffffffffu, best, o);
                int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
            }
            if (rank == 0) {
                piv_sh = bi;
                if (best == 0.0) fail_sh = 1;
            }
        }
        T.sync();
        if (fail_sh) break;
        const int p = piv_sh;
        if (p != k) {
            for (int j = rank; j < L; j += size) {
                cd t = D[k * L + j]; D[k * L + j] = D[p * L + j]; D[p * L + j] = t;
                t = U[k * L + j]; U[k * L + j] = U[p * L + j]; U[p * L + j] = t;
            }
            T.sync();
        }
        const cd inv = cdiv(cmk(1.0, 0.0), D[k * L + k]);
        // multipliers into column k below the pivot
        for (int i = k + 1 + rank; i < L; i += size) D[i * L + k] = cmul(D[i * L + k], inv);
        T.sync();
        const int rows = L - k - 1;
        for (int e = rank; e < rows * L; e += size) {
            int i = k + 1 + e / L, j = e % L;
            cd f = D[i * L + k];
            if (j > k) D[i * L + j] = csub(D[i * L + j], cmul(f, D[k * L + j]));
            U[i * L + j] = csub(U[i * L + j], cmul(f, U[k * L + j]));
        }
        T.sync();
    }
    if (fail_sh) return -2;
    for (int k = L - 1; k >= 0; --k) {
        const cd inv = cdiv(cmk(1.0, 0.0), D[k * L + k]);
        for (int j = rank; j < L; j += size) {
            cd acc = U[k * L + j];
            for (int c = k + 1; c < L; ++c) acc = csub(acc, cmul(D[k * L + c], U[c * L + j]));
            U[k * L + j] = cmul(acc, inv);
        }
        T.sync();
    }
    // E = I + 2X
    cd* E = A;
    for (int e = rank; e < LL; e += size) {
        int i = e / L, j = e - i * L;
        cd t = cscale(U[e], 2.0);
        if (i == j) t.x += 1.0;
        E[e] = t;
    }
    T.sync();
    cd* Tmp = A2;
    for (int k = 0; k < s; ++k) {
        sm_matmul(T, L, E, E, Tmp);
        cd* sw = E; E = Tmp; Tmp = sw;
    }
    *E_out = E;
    return s;
}

__device__ inline int pade_exp_sm(int L, int norm_mode, unsigned char* smem_raw, cd** E_out) {
    return pade_exp_team(CtaTeam{}, L, norm_mode, smem_raw, E_out);
}

// Computes E = exp(tau * Tbar) for Tbar built from alpha[1..m], beta[1..m]
// (complex, shared or global), writes y[j] = E(j, 0) for j = 0..m-1 when
// y != nullptr.  norm_mode 0: reference |Re|-only row sums; 1: |.|.
// Returns in every thread.
__device__ inline PadeOut pade_exp_tbar(int m, const cd* alpha, const cd* beta, cd tau, int norm_mode,
                                        cd* y, unsigned char* smem_raw) {
    const int L = m + 2;
    const int LL = L * L;
    cd* A = reinterpret_cast<cd*>(smem_raw);
    // tau * Tbar (gpuLanczosHelper.cu:14-60, padeClass.cu:240-246)
    for (int e = threadIdx.x; e < LL; e += blockDim.x) {
        int i = e / L, j = e - i * L;
        cd t = cmk(0, 0);
        if (i < m && j < m) {
            if (i == j) t = alpha[i + 1];
            else if (j == i + 1) t = beta[i + 1];
            else if (i == j + 1) t = beta[j + 1];
        } else {
            if (i == 0 && j == m) t = cmk(1.0, 0.0);
            else if (i >= m && j >= m && i == j - 1) t = cmk(1.0, 0.0);
        }
        A[e] = cmul(tau, t);
    }
    __syncthreads();
    cd* E = nullptr;
    PadeOut out;
    out.s = pade_exp_sm(L, norm_mode, smem_raw, &E);
    if (out.s < 0) {
        out.e_m1_m = cmk(0, 0);
        out.e_m1_mp1 = cmk(0, 0);
        return out;
    }
    if (y) for (int j = threadIdx.x; j < m; j += blockDim.x) y[j] = E[j * L];
    out.e_m1_m = E[(m - 1) * L + m];
    out.e_m1_mp1 = E[(m - 1) * L + m + 1];
    __syncthreads();
    return out;
}

// ---------------------------------------------------------------------------
// The columns of exp(tau Tbar) that a step uses, by one warp.
//
// A step needs E e_0 (the combine weights) and E(m-1, m), E(m-1, m+1) (the
// error estimate) only.  With A = tau T (m x m, tridiagonal) the augmented
// columns are E e_{m+q-1} = tau^q sum_k A^k e_0 / (k+q)!, q >= 1, so one
// sequence t_k = A^k e_0 / k! gives all of them, and lane i of a warp holds
// row i: two neighbour shuffles and ten FP64 operations per term, no shared
// memory and no barrier.  The matrix is scaled by the dense form's own rule
// (row-sum norm <= 1/2 after s halvings), where the series reaches 1e-19 in
// about 16 terms; with s > 0 the scaled exponential is applied 2^s times.
// The dense Padé(6,6) above (LU of a (m+2)^2 matrix by one CTA, a serial chain
// of about 6 L barriers) stays for what the series does not cover: more than
// kSeriesMaxS halvings, and the |Re|-only norm on a matrix of complex norm
// above 1/2, whose quotient the reference takes unscaled.
// Measured on a B200 (kernel time): one trajectory, m = 16, 41 us dense and
// 4.4 us this way; 256 trajectories, m = 20, 61 and 8.4 us (a CTA each).
// ---------------------------------------------------------------------------
constexpr int kSeriesMaxS = 4;
constexpr int kSeriesTerms = 24;   // never reached at a norm <= 1/2 (16 terms); bounds the loops

// 1/k
__device__ __constant__ static const double kInvK[kSeriesTerms + 3] = {
    0.0,      1.0,      1.0 / 2,  1.0 / 3,  1.0 / 4,  1.0 / 5,  1.0 / 6,  1.0 / 7,  1.0 / 8,
    1.0 / 9,  1.0 / 10, 1.0 / 11, 1.0 / 12, 1.0 / 13, 1.0 / 14, 1.0 / 15, 1.0 / 16, 1.0 / 17,
    1.0 / 18, 1.0 / 19, 1.0 / 20, 1.0 / 21, 1.0 / 22, 1.0 / 23, 1.0 / 24, 1.0 / 25, 1.0 / 26};

// The dense form's halvings of one norm.
__device__ __forceinline__ int halvings(double nrm) {
    int s = 0;
    while (nrm > 0.5 && s < 60) { nrm *= 0.5; s++; }
    return s;
}

// A warp's tridiagonal matrix: lane i holds row i of A = tau T, its diagonal
// and the imaginary parts of its (purely imaginary) couplings to rows i - 1
// and i + 1; lanes >= m hold zeros.
struct WarpTri {
    cd a;
    double bl, br;
    // A v
    __device__ __forceinline__ cd mul(cd v) const {
        const double px = __shfl_down_sync(0xffffffffu, v.x, 1), py = __shfl_down_sync(0xffffffffu, v.y, 1);
        const double mx = __shfl_up_sync(0xffffffffu, v.x, 1), my = __shfl_up_sync(0xffffffffu, v.y, 1);
        return cmk(a.x * v.x - a.y * v.y - (br * py + bl * my), a.x * v.y + a.y * v.x + (br * px + bl * mx));
    }
};

// alpha, beta of rows 0..m-1 as the warp's lanes hold them (lane i: alpha_{i+1}
// and beta_{i+1}); lanes >= m pass anything.
__device__ __forceinline__ WarpTri warp_tri(int m, cd alpha, double beta, double tau_im) {
    const int lane = threadIdx.x & 31;
    WarpTri t;
    t.a = lane < m ? cmk(-tau_im * alpha.y, tau_im * alpha.x) : cmk(0.0, 0.0);
    t.br = lane < m - 1 ? tau_im * beta : 0.0;
    const double up = __shfl_up_sync(0xffffffffu, t.br, 1);
    t.bl = lane > 0 && lane < m ? up : 0.0;
    return t;
}

// Row-sum infinity norms of the augmented matrix (the ones of its extra
// columns scaled by tau, too): |Re|-only and complex.
__device__ __forceinline__ void warp_tri_norms(const WarpTri& t, double tau_im, double& re, double& cn) {
    const int lane = threadIdx.x & 31;
    const double one = fabs(tau_im);
    re = fabs(t.a.x);
    cn = fmax(sqrt(cabs2(t.a)) + fabs(t.bl) + fabs(t.br) + (lane == 0 ? one : 0.0), one);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        re = fmax(re, __shfl_xor_sync(0xffffffffu, re, o));
        cn = fmax(cn, __shfl_xor_sync(0xffffffffu, cn, o));
    }
}

// Rows of E e_0 (y), E e_m (f1) and E e_{m+1} (f2) in their lanes.  Returns
// false where the dense form has to be used; s is its number of halvings, -1
// when that would reach 50 (then nothing is computed).  Called by all 32
// lanes; every lane returns the same.
__device__ __forceinline__ bool series_exp_tbar(int m, cd alpha, double beta, double tau_im, int norm_mode, cd& y,
                                                cd& f1, cd& f2, int& s) {
    const int lane = threadIdx.x & 31;
    WarpTri t = warp_tri(m, alpha, beta, tau_im);
    double re, cn;
    warp_tri_norms(t, tau_im, re, cn);
    s = halvings(norm_mode == 0 ? re : cn);
    y = f1 = f2 = cmk(0.0, 0.0);
    if (s >= 50) {
        s = -1;
        return true;
    }
    if (s > kSeriesMaxS || (norm_mode == 0 && cn > 0.5)) return false;
    const double h = ldexp(1.0, -s);
    t.a = cscale(t.a, h);
    t.bl *= h;
    t.br *= h;
    cn *= h;
    // t_k = A^k e_0 / k!: the sums of t_k, t_k / (k+1) and t_k / ((k+1)(k+2))
    cd v = cmk(lane == 0 ? 1.0 : 0.0, 0.0);
    y = v;
    f1 = v;
    f2 = cscale(v, 0.5);
    double bound = 1.0;
    for (int k = 1; k <= kSeriesTerms && bound > 1e-19; ++k) {
        v = cscale(t.mul(v), kInvK[k]);
        bound *= cn * kInvK[k];
        y = cadd(y, v);
        const cd u = cscale(v, kInvK[k + 1]);
        f1 = cadd(f1, u);
        f2 = cadd(f2, cscale(u, kInvK[k + 2]));
    }
    // times tau h and (tau h)^2 = -(tau_im h)^2
    const double th = tau_im * h;
    f1 = cmk(-th * f1.y, th * f1.x);
    f2 = cscale(f2, -th * th);
    if (s == 0) return true;
    // the other 2^s - 1 steps of length h: (x; c; 1) -> (exp(hA) x + c g1 + g2; c + tau h; 1)
    const cd g1 = f1, g2 = f2;
    double c = th;   // the (m, m+1) entry so far, times -i
    for (int r = 1; r < (1 << s); ++r) {
        cd vy = y, v1 = f1, v2 = f2;
        double bd = 1.0;
        for (int k = 1; k <= kSeriesTerms && bd > 1e-19; ++k) {
            vy = cscale(t.mul(vy), kInvK[k]);
            v1 = cscale(t.mul(v1), kInvK[k]);
            v2 = cscale(t.mul(v2), kInvK[k]);
            bd *= cn * kInvK[k];
            y = cadd(y, vy);
            f1 = cadd(f1, v1);
            f2 = cadd(f2, v2);
        }
        f1 = cadd(f1, g1);
        f2 = cadd(f2, cadd(cmk(-c * g1.y, c * g1.x), g2));
        c += th;
    }
    return true;
}

// Taylor-Krylov's augmented matrix (ones at (0, mb) and (mb+k, mb+k+1), k < p
// - 1): rows of its last column (fp), of column mb (f1) and of column mb + 1
// (f2).  Returns false where the dense form has to be used (any halving).
__device__ __forceinline__ bool series_exp_tk(int mb, int p, cd alpha, double beta, double tau_im, int norm_mode,
                                              cd& fp, cd& f1, cd& f2) {
    const int lane = threadIdx.x & 31;
    const WarpTri t = warp_tri(mb, alpha, beta, tau_im);
    double re, cn;
    warp_tri_norms(t, tau_im, re, cn);
    fp = f1 = f2 = cmk(0.0, 0.0);
    if (!(cn <= 0.5) || !(re <= 0.5)) return false;
    // c_k = k! / (k + p)!; fp's terms are t_k c_k
    double c = 1.0;
    for (int q = 2; q <= p; ++q) c /= q;
    cd v = cmk(lane == 0 ? 1.0 : 0.0, 0.0);
    fp = cscale(v, c);
    f1 = v;
    f2 = cscale(v, 0.5);
    double bound = 1.0;
    for (int k = 1; k <= kSeriesTerms && bound > 1e-19; ++k) {
        v = cscale(t.mul(v), kInvK[k]);
        bound *= cn * kInvK[k];
        c *= (double)k / (double)(k + p);
        fp = cadd(fp, cscale(v, c));
        const cd u = cscale(v, kInvK[k + 1]);
        f1 = cadd(f1, u);
        f2 = cadd(f2, cscale(u, kInvK[k + 2]));
    }
    cd tp = cmk(1.0, 0.0);
    for (int q = 0; q < p; ++q) tp = cmk(-tau_im * tp.y, tau_im * tp.x);
    fp = cmul(fp, tp);
    f1 = cmk(-tau_im * f1.y, tau_im * f1.x);
    f2 = cscale(f2, -tau_im * tau_im);
    return true;
}

// EXPOKIT Algorithm 3.2 as padeClass.cu:750-782 with the floor of
// systemClass.cu:2075-2077.
__device__ __forceinline__ double expokit_error(double beta_m, double norm_av, cd e_m1_m, cd e_m1_mp1) {
    double hm = fabs(beta_m);
    double err1 = hm * sqrt(cabs2(e_m1_m));
    double err2 = hm * norm_av * sqrt(cabs2(e_m1_mp1));
    double est = (err1 > err2) ? err2 / (1 - err2 / err1) : err1;
    if (est < 1.110223e-16) est = 1.110223e-16;
    return est;
}

}  // namespace dq
