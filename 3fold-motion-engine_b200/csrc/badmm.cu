// Batched proximal ADMM for many small contact problems, with its adjoint: the reference's
// BatchProxADMMGPU (src/motion_engine/ncp/ncp_batch_gpu.py:918-1313, "NB").
//
// The reference runs every step as a separate kernel over the whole batch (133 launches per
// ADMM iteration, ~35 000 graph nodes per step and gradient).  Here one launch runs everything
// and ONE LANE OWNS ONE CONTACT: a problem of nc contacts takes 1, 2, 4 or 8 lanes (the power of
// two that holds nc), a warp 32 / that many problems.  The arithmetic is float64:
//  * set-up (NB:974-1000): b = J v_free, M^-1 J^T (k_mj) and the Delassus matrix G = J M^-1 J^T
//    (k_gdense), the warp's problems one after the other; G's spectrum by cyclic Jacobi in the
//    reference's row-cyclic order (k_jacobi; see spectrum()), the diagonal blocks and their
//    largest eigenvalue (k_gd3, f_eigmax), eta and the per-contact step (k_eta), the bilateral
//    regime test by a Cholesky solve (k_bilat), rho (k_rho), the block-Jacobi preconditioner
//    (k_pjac);
//  * the product G x + (eta + rho) x (NB:326-388) from G's rows, which a lane keeps in registers
//    (3 rows of 3 nc): the lanes of a problem pass x through shared memory, everything else of a
//    contact (its 3x3 preconditioner, cone projection, multiplier) is the lane's own, and a dot
//    product is a 3-term sum and a butterfly over the problem's lanes;
//  * ADMM (NB:466-543, 1075-1099): x-step by block-Jacobi preconditioned CG warm-started from
//    the last x, z = proj_K(x + gamma / rho), gamma += rho (x - z), and every `refresh_every`
//    iterations u = G z + b, the slip speeds, the natural residual and the convergence mask (a
//    converged problem freezes x, z and gamma);
//  * the gradient (NB:556-808, 1145-1206): the active set (open / stick / slip with its
//    projector Z and diagonal D), the Schur preconditioner, and grad_affine -- the de Saxce
//    sigma map is affine, sigma -> a + B sigma: a from the direction with sigma = 0, B's columns
//    from unit sigmas, one (I - B) sigma = a elimination and the response at that sigma, each a
//    CG solve of the fixed-branch system -- for the direction db = dt J M^-1 e_j (and v+'s
//    response) and for mu at each problem's first slip contact.  B does not depend on the
//    direction where the CG converges, so both directions share its columns (grad_affine()), and
//    the solves run two at a time.
//
// What bounds it: the CG recurrence's dependent chain (exchange, 3 nc-term row sums, two dot
// products, one division).  The time per CG step hardly depends on how many problems share a
// warp, so the split puts as many there as there are contacts to own lanes, and leaves the
// problem's matrix on chip.
//
// Measured on a B200 (200 iterations of 8 CG steps and both gradients; before: a warp per problem,
// the products matrix-free), B problems of 4 contacts and 18 coordinates: B = 64 5.8 -> 1.24 ms,
// B = 4096 20.8 -> 1.31 ms (forward alone 11.7 -> 1.00), B = 16384 112 -> 3.1 ms; at B = 4096, 1
// contact 10.2 -> 0.91 ms, 8 contacts 81.9 -> 5.3 ms.  Difference from a float64 restatement with
// direct solves, on the batch of 4096: 1.2e-14 of the worst output's norm (before: 3.3e-13).
#include <math_constants.h>

#include "b2c_common.cuh"

namespace b2c {
namespace badmm {

constexpr double kTiny = 1.0e-300;
constexpr unsigned kAll = 0xffffffffu;

// the shapes of an instantiation: C contacts a problem
template <int C>
struct Dim {
    static constexpr int M = 3 * C;                               // rows
    static constexpr int L = C <= 1 ? 1 : C <= 2 ? 2 : C <= 4 ? 4 : 8;  // lanes of a problem
    static constexpr int PW = 32 / L;                             // problems of a warp
    static constexpr int XS = 2 * (((M + 1) / 2) | 1);            // exchange stride: an odd number of 16-byte words
    static constexpr int GS = (M * M) | 1;                        // stride of a problem's matrix
    static constexpr int CS = 2 * (M / 2 + 1);                    // rotations of a Jacobi stage
    static constexpr int R = C <= 5 ? 2 : 1;                      // gradient solves run side by side
    static constexpr int kVec = 3 * M + 9 * C + C * C + 6 * C;    // per problem: b, MJ column, work, Z, B, sigma
};

__host__ __device__ constexpr int odd(int n) { return n | 1; }

// staging of one problem while G is formed: J and M^-1 J^T (M rows) and M^-1 (nv rows), rows padded
template <int C>
__host__ __device__ inline size_t stage_doubles(int nv)
{
    return (size_t)(2 * Dim<C>::M + nv) * odd(nv);
}
template <int C>
__host__ __device__ inline size_t work_doubles(int nv)
{
    const size_t a = (size_t)Dim<C>::PW * Dim<C>::GS, b = stage_doubles<C>(nv);
    return (a > b ? a : b) + 1;
}
template <int C>
inline size_t smem_bytes(int nv)
{
    using D = Dim<C>;
    return 8 * (2 * (size_t)D::PW * D::XS * D::R + (size_t)D::PW * (D::GS + D::CS + D::kVec) + work_doubles<C>(nv));
}

// f_proj (NB:113-126); icm = 1 / (1 + mu^2)
__device__ __forceinline__ void proj3(const double z[3], double mu, double icm, double out[3])
{
    const double zn = z[0], zt = sqrt(fma(z[1], z[1], z[2] * z[2]));
    if (zt <= mu * zn) {
        out[0] = z[0];
        out[1] = z[1];
        out[2] = z[2];
    } else if (mu * zt <= -zn) {
        out[0] = out[1] = out[2] = 0.0;
    } else {
        const double s = fma(mu, zt, zn) * icm;
        const double f = mu * s / zt;
        out[0] = s;
        out[1] = f * z[1];
        out[2] = f * z[2];
    }
}

// 3x3 inverse (adjugate over determinant; zero when singular)
__device__ inline void inv3(const double a[9], double o[9])
{
    const double c00 = a[4] * a[8] - a[5] * a[7], c01 = a[2] * a[7] - a[1] * a[8], c02 = a[1] * a[5] - a[2] * a[4];
    const double c10 = a[5] * a[6] - a[3] * a[8], c11 = a[0] * a[8] - a[2] * a[6], c12 = a[2] * a[3] - a[0] * a[5];
    const double c20 = a[3] * a[7] - a[4] * a[6], c21 = a[1] * a[6] - a[0] * a[7], c22 = a[0] * a[4] - a[1] * a[3];
    const double det = a[0] * c00 + a[1] * c10 + a[2] * c20;
    const double adj[9] = {c00, c01, c02, c10, c11, c12, c20, c21, c22};
#pragma unroll
    for (int i = 0; i < 9; ++i) o[i] = det != 0.0 ? adj[i] / det : 0.0;
}

// f_eigmax (NB:130-146): largest eigenvalue of a symmetric 3x3 block, closed form
__device__ inline double eigmax3(const double A[9])
{
    const double p1 = A[1] * A[1] + A[2] * A[2] + A[5] * A[5];
    const double q = (A[0] + A[4] + A[8]) / 3.0;
    double out = fmax(A[0], fmax(A[4], A[8]));
    if (p1 > 0.0) {
        const double p2 = (A[0] - q) * (A[0] - q) + (A[4] - q) * (A[4] - q) + (A[8] - q) * (A[8] - q) + 2.0 * p1;
        const double p = sqrt(p2 / 6.0);
        if (p > 1.0e-300) {
            double Bm[9];
#pragma unroll
            for (int i = 0; i < 9; ++i) Bm[i] = (A[i] - ((i % 4) == 0 ? q : 0.0)) / p;
            const double det = Bm[0] * (Bm[4] * Bm[8] - Bm[5] * Bm[7]) - Bm[1] * (Bm[3] * Bm[8] - Bm[5] * Bm[6]) +
                               Bm[2] * (Bm[3] * Bm[7] - Bm[4] * Bm[6]);
            const double r = fmin(1.0, fmax(-1.0, det / 2.0));
            out = q + 2.0 * p * cos(acos(r) / 3.0);
        }
    }
    return out;
}

// one warp's view of its shared memory; g is the problem (lane group) of this lane
template <int C>
struct Env {
    using D = Dim<C>;
    int ln, g, c;       // lane, problem within the warp, contact
    bool on;            // this lane owns a contact (c < C)
    int turn;           // which exchange buffer is next
    double *xch;        // two buffers of PW x XS x R
    double *G, *A;      // the problem's G; scratch of the same shape (the spectrum, the Cholesky factor)
    double *cs;         // the stage's rotations
    double *bb, *mjc, *bw, *Z, *Bm, *a, *sg;  // b, (M^-1 J^T) column, work, projectors, B, a (2 x C), sigma (2 x C)
    double *stage;      // the whole warp's staging area (A's storage)
};

template <int C>
__device__ inline Env<C> carve(double *p, int nv)
{
    using D = Dim<C>;
    Env<C> E;
    E.ln = (int)(threadIdx.x & 31);
    E.g = E.ln / D::L;
    E.c = E.ln % D::L;
    E.on = E.c < C;
    E.turn = 0;
    E.xch = p;
    p += 2 * D::PW * D::XS * D::R;
    E.stage = p;
    E.A = p + (size_t)E.g * D::GS;
    p += work_doubles<C>(nv);
    E.G = p + (size_t)E.g * D::GS;
    p += (size_t)D::PW * D::GS;
    E.cs = p + (size_t)E.g * D::CS;
    p += (size_t)D::PW * D::CS;
    p += (size_t)E.g * D::kVec;
    E.bb = p;
    E.mjc = p + D::M;
    E.bw = p + 2 * D::M;
    E.Z = p + 3 * D::M;
    E.Bm = E.Z + 9 * C;
    E.a = E.Bm + C * C;
    E.sg = E.a + 3 * C;
    return E;
}

// sum over the problem's lanes: a butterfly, the same bits on every lane (IEEE addition commutes)
template <int L>
__device__ __forceinline__ double gsum(double s)
{
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) s = s + __shfl_xor_sync(kAll, s, o);
    return s;
}
__device__ __forceinline__ double dot3(const double a[3], const double b[3])
{
    return fma(a[2], b[2], fma(a[1], b[1], a[0] * b[0]));
}

// y[k] = rows x for N vectors at once: the lanes pass their three entries through shared memory
// (two buffers in turn, so one __syncwarp an exchange: a lane writes a buffer again only after
// the barrier that follows its last reads of it) and each forms its contact's three rows in two
// interleaved sums a row
template <int C, int N>
__device__ __forceinline__ void rows_times(Env<C> &E, const double (&g)[3][3 * C], const double (&x)[N][3],
                                           double (&y)[N][3])
{
    using D = Dim<C>;
    constexpr int NS = D::PW * D::XS;  // from one vector of the exchange to the next
    double *buf = E.xch + (size_t)E.turn * D::R * NS + E.g * D::XS;
    E.turn ^= 1;
    if (E.on) {
#pragma unroll
        for (int n = 0; n < N; ++n)
#pragma unroll
            for (int k = 0; k < 3; ++k) buf[n * NS + 3 * E.c + k] = x[n][k];
    }
    __syncwarp();
#pragma unroll
    for (int n = 0; n < N; ++n) {
        double s0[3], s1[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) s0[k] = s1[k] = 0.0;
        const double2 *q = reinterpret_cast<const double2 *>(buf + n * NS);
#pragma unroll
        for (int j = 0; j < D::M / 2; ++j) {
            const double2 v = q[j];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                s0[k] = fma(g[k][2 * j], v.x, s0[k]);
                s1[k] = fma(g[k][2 * j + 1], v.y, s1[k]);
            }
        }
        if (D::M & 1) {
            const double v = buf[n * NS + D::M - 1];
#pragma unroll
            for (int k = 0; k < 3; ++k) s0[k] = fma(g[k][D::M - 1], v, s0[k]);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) y[n][k] = s0[k] + s1[k];
    }
}

__device__ __forceinline__ void apply3(const double P[9], const double r[3], double z[3])
{
#pragma unroll
    for (int k = 0; k < 3; ++k) z[k] = fma(P[3 * k + 2], r[2], fma(P[3 * k + 1], r[1], P[3 * k] * r[0]));
}

// _pcg (NB:1048-1073) on N right-hand sides at once: the operator is rows + diag(d), the
// preconditioner the lane's 3x3 block P; x is updated where `upd`.  beta = s3 / s0 by the
// reciprocal of s0, which is formed beside the product instead of after the dot product; below
// 1e-290, where the reciprocal would overflow, by the quotient itself.
template <int C, int N>
__device__ __forceinline__ void pcg(Env<C> &E, const double (&g)[3][3 * C], const double (&d)[3], const double P[9],
                                    const double (&rhs)[N][3], double (&x)[N][3], int n_it, bool zero, bool upd)
{
    using D = Dim<C>;
    double r[N][3], p[N][3], Ap[N][3], s0[N];
    if (zero) {
#pragma unroll
        for (int n = 0; n < N; ++n)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                x[n][k] = 0.0;
                r[n][k] = rhs[n][k];
            }
    } else {
        rows_times<C, N>(E, g, x, Ap);
#pragma unroll
        for (int n = 0; n < N; ++n)
#pragma unroll
            for (int k = 0; k < 3; ++k) r[n][k] = rhs[n][k] - fma(d[k], x[n][k], Ap[n][k]);
    }
#pragma unroll
    for (int n = 0; n < N; ++n) {
        apply3(P, r[n], p[n]);
        s0[n] = gsum<D::L>(dot3(r[n], p[n]));
    }
    for (int it = 0; it < n_it; ++it) {
        rows_times<C, N>(E, g, p, Ap);
        double s1[N], i0[N];
#pragma unroll
        for (int n = 0; n < N; ++n) {
            i0[n] = 1.0 / s0[n];
#pragma unroll
            for (int k = 0; k < 3; ++k) Ap[n][k] = fma(d[k], p[n][k], Ap[n][k]);
            s1[n] = gsum<D::L>(dot3(p[n], Ap[n]));
        }
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const double s2 = (s1[n] > 0.0 || s1[n] < 0.0) ? s0[n] / s1[n] : 0.0;
            double z[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                if (upd) x[n][k] = fma(s2, p[n][k], x[n][k]);
                r[n][k] = fma(-s2, Ap[n][k], r[n][k]);
            }
            apply3(P, r[n], z);
            const double s3 = gsum<D::L>(dot3(r[n], z));
            double s4 = s3 * i0[n];
            if (!(fabs(s0[n]) > 1e-290)) s4 = (s0[n] > 0.0 || s0[n] < 0.0) ? s3 / s0[n] : 0.0;
#pragma unroll
            for (int k = 0; k < 3; ++k) p[n][k] = fma(s4, p[n][k], z[k]);
            s0[n] = s3;
        }
    }
}

// G's eigenvalues into the diagonal of E.A (k_jacobi): `sweeps` cyclic Jacobi sweeps in the
// row-cyclic pair order (0,1), (0,2), ..., (M-2, M-1).  Rotations on disjoint pairs commute, and
// in that order the pair (p, q) of sweep s only waits for pairs of smaller p + q + s M: stage t
// therefore runs every pair with p + q = t (mod M) at once, two sweeps overlapping, and M stages
// do a sweep's work where the pairs one by one are M (M - 1) / 2 steps.  A stage is a rotation
// per pair (spread over the problem's lanes), then the 2x2 blocks of the pairs' rows and columns,
// each one lane's.  A problem is done when a whole sweep met none of its off-diagonal entries
// above 1e-17 of its diagonal's geometric mean: its eigenvalues are then known to a rounding.  It
// takes no rotation from there on, because two nearly equal diagonal entries still turn by a large
// angle and can move by that rounding, and a problem's result must not depend on how long its
// neighbours in the warp go on.
template <int C>
__device__ void spectrum(Env<C> &E, int sweeps)
{
    using D = Dim<C>;
    constexpr int M = D::M;
    double *A = E.A, *cs = E.cs;
    bool big = false, done = false;
    for (int t = 1; t <= sweeps * M + M - 3; ++t) {
        const int r = t % M, s = t / M;
        const int n1 = r / 2 + 1, K = n1 + (r + M) / 2 - r;  // pairs with p + q = r, and with p + q = r + M
        for (int k = E.c; k < K && !done; k += D::L) {
            const int p = k < n1 ? k : r + 1 + (k - n1), q = k < n1 ? r - p : r + M - p;
            const int sw = k < n1 ? s : s - 1;
            double c = 1.0, sn = 0.0;
            if (p != q && sw >= 0 && sw < sweeps) {
                const double apq = A[p * M + q], app = A[p * M + p], aqq = A[q * M + q];
                if (apq > kTiny || apq < -kTiny) {
                    if (apq * apq > 1e-34 * fabs(app * aqq)) big = true;
                    const double th = (aqq - app) / (2.0 * apq);
                    double tt = 1.0 / (fabs(th) + sqrt(fma(th, th, 1.0)));
                    if (th < 0.0) tt = -tt;
                    c = 1.0 / sqrt(fma(tt, tt, 1.0));
                    sn = tt * c;
                }
            }
            cs[2 * k] = c;
            cs[2 * k + 1] = sn;
        }
        __syncwarp();
        for (int P = 0; P < K && !done; ++P) {
            const int p = P < n1 ? P : r + 1 + (P - n1), q = P < n1 ? r - p : r + M - p;
            const double cp = cs[2 * P], sp = cs[2 * P + 1];
            for (int Q = E.c; Q < K; Q += D::L) {
                const int u = Q < n1 ? Q : r + 1 + (Q - n1), v = Q < n1 ? r - u : r + M - u;
                const double cq = cs[2 * Q], sq = cs[2 * Q + 1];
                const double b00 = A[p * M + u], b01 = A[p * M + v], b10 = A[q * M + u], b11 = A[q * M + v];
                const double e00 = cq * b00 - sq * b01, e01 = sq * b00 + cq * b01;
                const double e10 = cq * b10 - sq * b11, e11 = sq * b10 + cq * b11;
                A[p * M + u] = cp * e00 - sp * e10;
                if (u != v) A[p * M + v] = cp * e01 - sp * e11;
                if (p != q) {
                    A[q * M + u] = sp * e00 + cp * e10;
                    if (u != v) A[q * M + v] = sp * e01 + cp * e11;
                }
            }
        }
        __syncwarp();
        if (t % M == 0) {  // stages t - M + 1 .. t met every pair once (from the second window on)
            const unsigned met = __ballot_sync(kAll, big) >> (E.g * D::L) & ((1u << D::L) - 1u);
            done = done || (met == 0 && t >= 2 * M);
            if (__all_sync(kAll, done)) break;
            big = false;
        }
    }
}

// does the bilateral solution -G^-1 b leave a cone (k_bilat: Cholesky of G with floored pivots)?
// The problem's lanes share the factor's rows; the two substitutions are each lane's own.
template <int C>
__device__ bool leaves_cone(Env<C> &E, double mu)
{
    using D = Dim<C>;
    constexpr int M = D::M;
    double *A = E.A;
    for (int i = E.c; i < M * M; i += D::L) A[i] = E.G[i];
    __syncwarp();
    for (int k = 0; k < M; ++k) {
        double d = A[k * M + k];
        for (int j = 0; j < k; ++j) d = fma(-A[k * M + j], A[k * M + j], d);
        if (d < kTiny) d = kTiny;
        d = sqrt(d);
        for (int i = k + 1 + E.c; i < M; i += D::L) {
            double s = A[i * M + k];
            for (int j = 0; j < k; ++j) s = fma(-A[i * M + j], A[k * M + j], s);
            A[i * M + k] = s / d;
        }
        __syncwarp();
        if (E.c == 0) A[k * M + k] = d;
        __syncwarp();
    }
    if (E.c == 0) {
        for (int i = 0; i < M; ++i) {
            double s = -E.bb[i];
            for (int j = 0; j < i; ++j) s = fma(-A[i * M + j], E.bw[j], s);
            E.bw[i] = s / A[i * M + i];
        }
        for (int i = M - 1; i >= 0; --i) {
            double s = E.bw[i];
            for (int j = i + 1; j < M; ++j) s = fma(-A[j * M + i], E.bw[j], s);
            E.bw[i] = s / A[i * M + i];
        }
    }
    __syncwarp();
    bool bind = false;
    if (E.on) {
        const double *w = E.bw + 3 * E.c;
        const double lt = sqrt(w[1] * w[1] + w[2] * w[2]);
        bind = w[0] <= 0.0 || lt > mu * w[0];
    }
    const unsigned all = __ballot_sync(kAll, bind);
    const unsigned mine = (D::L == 32 ? kAll : ((1u << D::L) - 1u)) << (E.g * D::L);
    __syncwarp();
    return (all & mine) != 0;
}

// b, G and the column jdir of M^-1 J^T of the warp's problems, one problem after the other with
// the whole warp (NB:974-1000)
template <int C>
__device__ void form(Env<C> &E, const b2c_admm &P, int e0, int jdir)
{
    using D = Dim<C>;
    constexpr int M = D::M;
    const int nv = P.nv, S = odd(nv), ln = E.ln;
    double *J = E.stage, *MJ = J + (size_t)M * S, *Mi = MJ + (size_t)M * S;
    for (int q = 0; q < D::PW; ++q) {
        const int e = min(e0 + q, P.n_env - 1);
        const double *Jg = P.J + (size_t)e * M * nv, *Mg = P.Minv + (size_t)e * nv * nv, *vg = P.v_free + (size_t)e * nv;
        double *G = E.G + (q - E.g) * D::GS, *bb = E.bb + (q - E.g) * D::kVec;
        for (int i = ln; i < M * nv; i += 32) J[(i / nv) * S + i % nv] = Jg[i];
        for (int i = ln; i < nv * nv; i += 32) Mi[(i / nv) * S + i % nv] = Mg[i];
        __syncwarp();
        for (int i = ln; i < M; i += 32) {
            double s = 0.0;
            for (int k = 0; k < nv; ++k) s = fma(J[i * S + k], vg[k], s);
            bb[i] = P.b_in ? P.b_in[(size_t)e * M + i] : s;
        }
        for (int i = ln; i < M * nv; i += 32) {
            const int row = i / nv, k = i - row * nv;
            double s = 0.0;
            for (int l = 0; l < nv; ++l) s = fma(Mi[k * S + l], J[row * S + l], s);
            MJ[row * S + k] = s;
        }
        __syncwarp();
        for (int i = ln; i < M * M; i += 32) {
            const int row = i / M, col = i - row * M;
            double s = 0.0;
            for (int k = 0; k < nv; ++k) s = fma(J[row * S + k], MJ[col * S + k], s);
            G[i] = s;
        }
        for (int i = ln; i < M; i += 32) bb[M + i] = MJ[i * S + jdir];
        __syncwarp();
    }
}

// out[e] = base + M^-1 J^T x of the warp's problems (base: v_free, or dt M^-1 e_jdir), x (M a
// problem) in E.bw
template <int C>
__device__ void respond(Env<C> &E, const b2c_admm &P, int e0, double *out, bool free_v, int jdir, double dt)
{
    using D = Dim<C>;
    constexpr int M = D::M;
    const int nv = P.nv, ln = E.ln;
    double *y = E.stage;
    __syncwarp();
    for (int q = 0; q < D::PW; ++q) {
        const int e = e0 + q;
        if (e >= P.n_env) break;
        const double *Jg = P.J + (size_t)e * M * nv, *Mg = P.Minv + (size_t)e * nv * nv;
        const double *x = E.bw + (q - E.g) * D::kVec;
        if (ln < nv) {
            double s = 0.0;
            for (int i = 0; i < M; ++i) s = fma(Jg[(size_t)i * nv + ln], x[i], s);
            y[ln] = s;
        }
        __syncwarp();
        if (ln < nv) {
            double s = 0.0;
            for (int l = 0; l < nv; ++l) s = fma(Mg[(size_t)ln * nv + l], y[l], s);
            out[(size_t)e * nv + ln] = s + (free_v ? P.v_free[(size_t)e * nv + ln] : dt * Mg[(size_t)ln * nv + jdir]);
        }
        __syncwarp();
    }
}

// the fixed-branch gradient's per-contact quantities (k_active, NB:546-627)
struct Branch {
    int lab;          // 0 open, 1 stick, 2 slip
    double Z[9], D[3], h1, h2;
    double Ps[9];     // (Z^T (Gd + eta I) Z + diag D)^-1
};

template <int C>
__device__ Branch branch_of(Env<C> &E, const double lam[3], const double u[3], double mu, double eta,
                            double tol_lam, double tol_rel)
{
    using D = Dim<C>;
    Branch b;
    double lsc = E.on ? fmax(fabs(lam[0]), fmax(fabs(lam[1]), fabs(lam[2]))) : 0.0;
#pragma unroll
    for (int o = D::L / 2; o > 0; o >>= 1) lsc = fmax(lsc, __shfl_xor_sync(kAll, lsc, o));
    lsc = fmax(lsc, 1.0e-30);
#pragma unroll
    for (int i = 0; i < 9; ++i) b.Z[i] = 0.0;
    b.D[0] = b.D[1] = b.D[2] = 0.0;
    b.h1 = b.h2 = 0.0;
    const double lt = sqrt(lam[1] * lam[1] + lam[2] * lam[2]);
    if (!E.on || lam[0] <= tol_lam + tol_rel * lsc) {
        b.lab = 0;
        b.D[0] = b.D[1] = b.D[2] = 1.0;
    } else if (lt >= mu * lam[0] * (1.0 - tol_rel) - tol_lam) {
        b.lab = 2;
        double nw = sqrt(u[1] * u[1] + u[2] * u[2]);
        if (nw < 1.0e-300) nw = 1.0e-300;
        b.h1 = u[1] / nw;
        b.h2 = u[2] / nw;
        b.Z[0] = 1.0;
        b.Z[3] = -mu * b.h1;
        b.Z[6] = -mu * b.h2;
        b.Z[4] = -b.h2;
        b.Z[7] = b.h1;
        b.D[1] = nw / fmax(mu * lam[0], 1.0e-300);
        b.D[2] = 1.0;
    } else {
        b.lab = 1;
        b.Z[0] = b.Z[4] = b.Z[8] = 1.0;
    }
    double Q[9], T[9], S[9];
#pragma unroll
    for (int i = 0; i < 9; ++i)
        Q[i] = E.on ? E.G[(3 * E.c + i / 3) * D::M + 3 * E.c + i % 3] + ((i % 4) == 0 ? eta : 0.0) : 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < 3; ++k) s = fma(b.Z[3 * k + i], Q[3 * k + j], s);
            T[3 * i + j] = s;
        }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            double s = i == j ? b.D[i] : 0.0;
#pragma unroll
            for (int k = 0; k < 3; ++k) s = fma(T[3 * i + k], b.Z[3 * k + j], s);
            S[3 * i + j] = s;
        }
    inv3(S, b.Ps);
    return b;
}

// the lane's three rows of Z^T (G + eta I) Z (NB:1040-1043 formed once instead of applied thrice)
template <int C>
__device__ __forceinline__ void schur_rows(Env<C> &E, const Branch &b, double eta, double (&S)[3][3 * C])
{
    using D = Dim<C>;
    constexpr int M = D::M;
    if (E.on)
        for (int i = 0; i < 9; ++i) E.Z[9 * E.c + i] = b.Z[i];
    __syncwarp();
#pragma unroll
    for (int c = 0; c < C; ++c) {
        double T[3][3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                double s = 0.0;
                if (E.on)
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                        s = fma(b.Z[3 * k + i],
                                E.G[(3 * E.c + k) * M + 3 * c + j] + (c == E.c && k == j ? eta : 0.0), s);
                T[i][j] = s;
            }
        const double *Z = E.Z + 9 * c;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j)
                S[i][3 * c + j] = fma(T[i][2], Z[6 + j], fma(T[i][1], Z[3 + j], T[i][0] * Z[j]));
    }
    __syncwarp();
}

// y[n] = (G + eta) x[n], G from shared memory (a few times a gradient)
template <int C, int N>
__device__ __forceinline__ void g_times(Env<C> &E, double eta, const double (&x)[N][3], double (&y)[N][3])
{
    using D = Dim<C>;
    constexpr int NS = D::PW * D::XS;
    double *buf = E.xch + (size_t)E.turn * D::R * NS + E.g * D::XS;
    E.turn ^= 1;
    if (E.on)
#pragma unroll
        for (int n = 0; n < N; ++n)
#pragma unroll
            for (int k = 0; k < 3; ++k) buf[n * NS + 3 * E.c + k] = x[n][k];
    __syncwarp();
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            double s = 0.0;
            if (E.on)
                for (int j = 0; j < D::M; ++j) s = fma(E.G[(3 * E.c + k) * D::M + j], buf[n * NS + j], s);
            y[n][k] = fma(eta, x[n][k], s);
        }
}

// Z^T v
__device__ __forceinline__ void zt3(const Branch &b, const double v[3], double o[3])
{
#pragma unroll
    for (int j = 0; j < 3; ++j) o[j] = fma(b.Z[6 + j], v[2], fma(b.Z[3 + j], v[1], b.Z[j] * v[0]));
}

// N right-hand sides through the fixed-branch system: dlam = Z y + pinh, and the slip speed's
// rate sigo = w . ((G + eta) dlam + db)_t on a slip contact (_grad_once, NB:1162-1170)
template <int C, int N>
__device__ __forceinline__ void branch_solve(Env<C> &E, const Branch &b, const double (&S)[3][3 * C], double eta,
                                             const double (&rhs)[N][3], const double (&pinh)[N][3],
                                             const double (&db)[N][3], int cg, double (&dl)[N][3], double (&sigo)[N])
{
    double y[N][3], t[N][3];
    pcg<C, N>(E, S, b.D, b.Ps, rhs, y, cg, true, true);
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            dl[n][k] = fma(b.Z[3 * k + 2], y[n][2], fma(b.Z[3 * k + 1], y[n][1], b.Z[3 * k] * y[n][0])) + pinh[n][k];
    g_times<C, N>(E, eta, dl, t);
#pragma unroll
    for (int n = 0; n < N; ++n)
        sigo[n] = b.lab == 2 ? fma(b.h1, t[n][1] + db[n][1], b.h2 * (t[n][2] + db[n][2])) : 0.0;
}

// (I - B) sigma = a over the n slip contacts: Gauss with partial pivoting, one lane (k_solvesig);
// W (n x n) and r (n) are overwritten
__device__ inline void eliminate(double *W, int ld, double *r, double *sig, int n)
{
    for (int k = 0; k < n; ++k) {
        int piv = k;
        double big = fabs(W[k * ld + k]);
        for (int i = k + 1; i < n; ++i) {
            const double v = fabs(W[i * ld + k]);
            if (v > big) {
                big = v;
                piv = i;
            }
        }
        if (piv != k) {
            for (int j = 0; j < n; ++j) {
                const double t = W[k * ld + j];
                W[k * ld + j] = W[piv * ld + j];
                W[piv * ld + j] = t;
            }
            const double t = r[k];
            r[k] = r[piv];
            r[piv] = t;
        }
        const double d = W[k * ld + k];
        if (d > kTiny || d < -kTiny)
            for (int i = k + 1; i < n; ++i) {
                const double f = W[i * ld + k] / d;
                for (int j = k; j < n; ++j) W[i * ld + j] = fma(-f, W[k * ld + j], W[i * ld + j]);
                r[i] = fma(-f, r[k], r[i]);
            }
    }
    for (int i = n - 1; i >= 0; --i) {
        double s = r[i];
        for (int j = i + 1; j < n; ++j) s = fma(-W[i * ld + j], sig[j], s);
        const double d = W[i * ld + i];
        sig[i] = (d > kTiny || d < -kTiny) ? s / d : 0.0;
    }
}

// grad_affine (NB:1172-1186) for N directions (pinh, db): dlam.  n_calls - 2 columns of B at most
// (the rest are zero, as the reference's loop leaves them).
//
// The reference takes a column of B as the slip speeds' rate with a unit sigma less that without.
// A solved system is linear, so the column is as well the rate for the unit sigma alone, which
// every direction shares.  A conjugate gradient that has not converged is not linear in its
// right-hand side (4 steps at 4 contacts: 0.05 of the gradient), so the short
// cut is taken from twice the system's rows on (own_columns), where the two forms have agreed to
// rounding since M steps (batches of 1 to 8 contacts, 6 to 32 coordinates, 2e-13 of the gradient);
// below, each direction has columns of its own, as the reference forms them.
template <int C>
__host__ __device__ constexpr bool own_columns(int cg)
{
    return cg < 2 * Dim<C>::M;
}

template <int C, int N>
__device__ void grad_affine(Env<C> &E, const Branch &b, const double (&S)[3][3 * C], double mu, double eta,
                            const double (&pinh)[N][3], const double (&db)[N][3], int n_calls, int cg,
                            double (&dl)[N][3])
{
    using D = Dim<C>;
    double t[N][3], base[N][3], rhs[N][3], so[N];
    g_times<C, N>(E, eta, pinh, t);
#pragma unroll
    for (int n = 0; n < N; ++n) {
#pragma unroll
        for (int k = 0; k < 3; ++k) t[n][k] = t[n][k] + db[n][k];
        zt3(b, t[n], base[n]);
#pragma unroll
        for (int k = 0; k < 3; ++k) base[n][k] = -base[n][k];
    }
    branch_solve<C, N>(E, b, S, eta, base, pinh, db, cg, dl, so);
    // the rank of this lane's contact among the problem's slip contacts, and their number
    const unsigned slips = (__ballot_sync(kAll, b.lab == 2) >> (E.g * D::L)) & ((1u << D::L) - 1u);
    const int rank = __popc(slips & ((1u << E.c) - 1u)), ns = __popc(slips);
    if (b.lab == 2)
#pragma unroll
        for (int n = 0; n < N; ++n) E.a[n * C + rank] = so[n];
    // B's columns: the response of the slip speeds to a unit sigma (one direction: maybe its own)
    const bool own = N == 1 && own_columns<C>(cg);
    int most = ns;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(kAll, most, o));
    const int K = n_calls - 2;
    for (int i = E.c; i < C * C; i += D::L) E.Bm[i] = 0.0;
    __syncwarp();
    for (int j = 0; j < K && j < most; j += D::R) {
        double ur[D::R][3], up[D::R][3], ub[D::R][3], ud[D::R][3], us[D::R];
#pragma unroll
        for (int n = 0; n < D::R; ++n)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                up[n][k] = own ? pinh[0][k] : 0.0;
                ub[n][k] = own ? db[0][k] : 0.0;
                ur[n][k] = (own ? base[0][k] : 0.0) - (k == 0 && b.lab == 2 && rank == j + n ? mu : 0.0);
            }
        branch_solve<C, D::R>(E, b, S, eta, ur, up, ub, cg, ud, us);
        if (b.lab == 2)
#pragma unroll
            for (int n = 0; n < D::R; ++n)
                if (j + n < ns && j + n < K) E.Bm[rank * C + j + n] = own ? us[n] - so[0] : us[n];
    }
    __syncwarp();
    if (E.c == 0) {
        double *W = E.A;  // C x C
#pragma unroll
        for (int n = 0; n < N; ++n) {
            for (int i = 0; i < ns; ++i)
                for (int j = 0; j < ns; ++j) W[i * C + j] = (i == j ? 1.0 : 0.0) - E.Bm[i * C + j];
            eliminate(W, C, E.a + n * C, E.sg + n * C, ns);
        }
    }
    __syncwarp();
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            rhs[n][k] = k == 0 && b.lab == 2 ? fma(-mu, E.sg[n * C + rank], base[n][k]) : base[n][k];
    __syncwarp();
    branch_solve<C, N>(E, b, S, eta, rhs, pinh, db, cg, dl, so);
}

template <int C>
__global__ void __launch_bounds__(32, C <= 5 ? 8 : 4) k_admm(b2c_admm P, b2c_admm_params prm)
{
    using D = Dim<C>;
    constexpr int M = D::M;
    extern __shared__ __align__(16) double s_env[];
    const int e0 = blockIdx.x * D::PW;
    Env<C> E = carve<C>(s_env, P.nv);
    const int e = min(e0 + E.g, P.n_env - 1);
    const bool live = E.on && e0 + E.g < P.n_env;  // this lane writes its contact's results
    const bool forward = (prm.flags & B2C_ADMM_FORWARD) != 0;
    form<C>(E, P, e0, prm.jdir);
    const double mu = E.on ? P.mu[(size_t)e * C + E.c] : 0.0, icm = 1.0 / (1.0 + mu * mu);
    double g[3][M], bb[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        bb[k] = E.on ? E.bb[3 * E.c + k] : 0.0;
#pragma unroll
        for (int j = 0; j < M; ++j) g[k][j] = E.on ? E.G[(3 * E.c + k) * M + j] : 0.0;
    }
    // the diagonal block's largest eigenvalue, eta, the residual's step (k_gd3, k_eta)
    double W[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) W[i] = E.on ? E.G[(3 * E.c + i / 3) * M + 3 * E.c + i % 3] : 0.0;
    const double gn = eigmax3(W), eta = prm.alpha_eta * gn, gs = gn + eta;
    const double rhoc = gs > 0.0 ? 1.0 / gs : 1.0;
    double x[1][3] = {{0.0, 0.0, 0.0}}, zv[1][3] = {{0.0, 0.0, 0.0}}, gam[3] = {0.0, 0.0, 0.0}, u[3] = {0.0, 0.0, 0.0};
    if (forward) {
        // rho (k_rho): sqrt(lmin+ lmax) | lmin+ | lmax | the regime's choice | given
        double rho;
        if (prm.rho_mode == B2C_ADMM_RHO_GIVEN) {
            rho = P.rho[e];
        } else {
            for (int i = E.c; i < M * M; i += D::L) E.A[i] = E.G[i];
            __syncwarp();
            spectrum<C>(E, prm.jacobi_sweeps);
            double mx = -1.0e300;
            for (int i = 0; i < M; ++i) mx = fmax(mx, E.A[i * M + i]);
            const double thr = 1e-12 * mx;
            double mn = mx;
            for (int i = 0; i < M; ++i) {
                const double v = E.A[i * M + i];
                if (v > thr && v < mn) mn = v;
            }
            __syncwarp();
            rho = sqrt(mn * mx);
            if (prm.rho_mode == B2C_ADMM_RHO_LMIN) rho = mn;
            if (prm.rho_mode == B2C_ADMM_RHO_LMAX) rho = mx;
            if (prm.rho_mode == B2C_ADMM_RHO_REGIME) rho = leaves_cone<C>(E, mu) ? mx : mn;
        }
        const double irho = 1.0 / rho;
        // block-Jacobi preconditioner (k_pjac)
        double Pj[9], d[3];
        const double sh = eta + rho;
#pragma unroll
        for (int i = 0; i < 9; ++i) W[i] = W[i] + ((i % 4) == 0 ? sh : 0.0);
        inv3(W, Pj);
        if (!E.on)
#pragma unroll
            for (int i = 0; i < 9; ++i) Pj[i] = 0.0;
        d[0] = d[1] = d[2] = sh;
        double sl = 0.0, resm = CUDART_NAN;
        bool run = true;
        for (int it = 0; it < prm.n_iter; ++it) {
            // one iteration (NB:1075-1082)
            double rhs[1][3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const double q = k == 0 ? fma(mu, sl, bb[0]) : bb[k];
                rhs[0][k] = -fma(-rho, zv[0][k], q + gam[k]);
            }
            pcg<C, 1>(E, g, d, Pj, rhs, x, prm.cg_iters, false, run);
            double v[3], zn[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) v[k] = fma(gam[k], irho, x[0][k]);
            proj3(v, mu, icm, zn);
            if (run) {
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    zv[0][k] = zn[k];
                    gam[k] = fma(rho, x[0][k] - zn[k], gam[k]);
                }
            }
            const int kk = prm.chunk > 0 ? it % prm.chunk : it;
            if (prm.refresh_every > 0 && (kk + 1) % prm.refresh_every == 0) {
                // the Cadoux refresh, the natural residual and the mask (NB:1084-1092, 498-543)
                double y[1][3];
                rows_times<C, 1>(E, g, zv, y);
#pragma unroll
                for (int k = 0; k < 3; ++k) u[k] = fma(eta, zv[0][k], y[0][k]) + bb[k];
                sl = sqrt(fma(u[1], u[1], u[2] * u[2]));
                double q[3], pr[3];
                q[0] = fma(-rhoc, prm.desax ? fma(mu, sl, u[0]) : u[0], zv[0][0]);
                q[1] = fma(-rhoc, u[1], zv[0][1]);
                q[2] = fma(-rhoc, u[2], zv[0][2]);
                proj3(q, mu, icm, pr);
                double m = fmax(fabs(zv[0][0] - pr[0]), fmax(fabs(zv[0][1] - pr[1]), fabs(zv[0][2] - pr[2])));
                // NaN-propagating maximum (k_resmax): fmax drops a NaN, so it is carried beside it
                double bad = (zv[0][0] - pr[0]) + (zv[0][1] - pr[1]) + (zv[0][2] - pr[2]);
                if (!E.on) m = bad = 0.0;
                bad = bad != bad ? 1.0 : 0.0;
#pragma unroll
                for (int o = D::L / 2; o > 0; o >>= 1) {
                    m = fmax(m, __shfl_xor_sync(kAll, m, o));
                    bad = fmax(bad, __shfl_xor_sync(kAll, bad, o));
                }
                resm = bad > 0.0 ? CUDART_NAN : m;
                if (resm < prm.tol) run = false;
                if (!__any_sync(kAll, run)) break;  // every problem of the warp is frozen: nothing moves any more
            }
        }
        if (E.on) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                E.bw[3 * E.c + k] = zv[0][k];
                if (live) {
                    P.lam[(size_t)e * M + 3 * E.c + k] = zv[0][k];
                    P.u[(size_t)e * M + 3 * E.c + k] = u[k];
                }
            }
        }
        if (live && E.c == 0) {
            if (P.res) P.res[e] = resm;
            if (P.mask) P.mask[e] = run ? 1 : 0;
            if (P.rho) P.rho[e] = rho;
        }
        respond<C>(E, P, e0, P.v_plus, true, 0, 0.0);  // v+ = v_free + M^-1 J^T lam (NB:1057-1062)
    } else if (E.on) {
        // the impulses and velocities are given (the gradient of an outside solve)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            zv[0][k] = P.lam[(size_t)e * M + 3 * E.c + k];
            u[k] = P.u[(size_t)e * M + 3 * E.c + k];
        }
    }
    if (!(prm.flags & (B2C_ADMM_GRADIENT | B2C_ADMM_GRAD_GIVEN))) return;
    const bool given = (prm.flags & B2C_ADMM_GRAD_GIVEN) != 0;
    const Branch b = branch_of<C>(E, zv[0], u, mu, eta, 1e-10, 1e-6);
    schur_rows<C>(E, b, eta, g);  // from here g holds the rows of Z^T (G + eta I) Z
    const int n_calls = prm.n_calls > 0 ? prm.n_calls : C + 2;
    const unsigned slips = (__ballot_sync(kAll, b.lab == 2) >> (E.g * D::L)) & ((1u << D::L) - 1u);
    // the directions: b (given, or dt J M^-1 e_jdir), and mu at the first slip contact (k_pmu)
    double dbt[3], pm[3] = {0.0, 0.0, 0.0}, lt[3] = {0.0, 0.0, 0.0}, lm[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int k = 0; k < 3; ++k)
        dbt[k] = !E.on ? 0.0 : given ? P.dbv_in[(size_t)e * M + 3 * E.c + k] : prm.dt * E.mjc[3 * E.c + k];
    if (b.lab == 2 && (slips & ((1u << E.c) - 1u)) == 0) {
        pm[1] = -zv[0][0] * b.h1;
        pm[2] = -zv[0][0] * b.h2;
    }
    const int dirs = !given && prm.do_mu ? 2 : 1;
    int done = 0;
    if constexpr (D::R == 2) {
        if (dirs == 2 && !own_columns<C>(prm.grad_cg)) {
            double pin[2][3], db[2][3], dl[2][3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                pin[0][k] = db[1][k] = 0.0;
                db[0][k] = dbt[k];
                pin[1][k] = pm[k];
            }
            grad_affine<C, 2>(E, b, g, mu, eta, pin, db, n_calls, prm.grad_cg, dl);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                lt[k] = dl[0][k];
                lm[k] = dl[1][k];
            }
            done = 2;
        }
    }
#pragma unroll 1
    for (int n = done; n < dirs; ++n) {
        double pin[1][3], db[1][3], dl[1][3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            pin[0][k] = n == 0 ? 0.0 : pm[k];
            db[0][k] = n == 0 ? dbt[k] : 0.0;
        }
        grad_affine<C, 1>(E, b, g, mu, eta, pin, db, n_calls, prm.grad_cg, dl);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if (n == 0) lt[k] = dl[0][k];
            else lm[k] = dl[0][k];
        }
    }
    if (E.on)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            E.bw[3 * E.c + k] = lt[k];
            if (live) {
                P.dlam_tau[(size_t)e * M + 3 * E.c + k] = lt[k];
                if (!given) P.dlam_mu[(size_t)e * M + 3 * E.c + k] = lm[k];
            }
        }
    if (live) {
        P.labels[(size_t)e * C + E.c] = b.lab;
        if (E.c == 0) P.nslip[e] = __popc(slips);
    }
    if (!given) respond<C>(E, P, e0, P.dv_tau, false, prm.jdir, prm.dt);
}

template <int C>
static void launch(const b2c_admm &a, const b2c_admm_params &p, cudaStream_t st)
{
    const size_t smem = smem_bytes<C>(a.nv);
    // above the 48 KB a launch may have by default; the opt-in is the device's, so for every launch
    cudaFuncSetAttribute(k_admm<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
    const int per = Dim<C>::PW;
    k_admm<C><<<(a.n_env + per - 1) / per, 32, smem, st>>>(a, p);
}

}  // namespace badmm
}  // namespace b2c

extern "C" int64_t b2c_admm_smem_bytes(int32_t nc, int32_t nv)
{
    if (nc < 1 || nc > B2C_ADMM_MAX_CONTACTS || nv < 1 || nv > B2C_ADMM_MAX_DOFS) return -1;
    using namespace b2c::badmm;
    size_t n = 0;
    switch (nc) {
#define B2C_ADMM_CASE(k)        \
    case k:                     \
        n = smem_bytes<k>(nv);  \
        break;
        B2C_ADMM_CASE(1)
        B2C_ADMM_CASE(2)
        B2C_ADMM_CASE(3)
        B2C_ADMM_CASE(4)
        B2C_ADMM_CASE(5)
        B2C_ADMM_CASE(6)
        B2C_ADMM_CASE(7)
        B2C_ADMM_CASE(8)
#undef B2C_ADMM_CASE
    }
    return (int64_t)n;
}

extern "C" int32_t b2c_admm_solve(const b2c_admm *a, const b2c_admm_params *p, b2c_stream st)
{
    using namespace b2c;
    if (!a || !p) {
        set_error("b2c_admm_solve: null argument");
        return B2C_EARG;
    }
    if (a->n_env < 0 || a->nc < 1 || a->nc > B2C_ADMM_MAX_CONTACTS || a->nv < 1 || a->nv > B2C_ADMM_MAX_DOFS) {
        set_error("b2c_admm_solve: n_env %d, nc %d (1..%d), nv %d (1..%d) out of range", a->n_env, a->nc,
                  B2C_ADMM_MAX_CONTACTS, a->nv, B2C_ADMM_MAX_DOFS);
        return B2C_EARG;
    }
    const bool fwd = (p->flags & B2C_ADMM_FORWARD) != 0, grad = (p->flags & B2C_ADMM_GRADIENT) != 0,
               given = (p->flags & B2C_ADMM_GRAD_GIVEN) != 0;
    if (fwd == given || (grad && given) || p->jdir < 0 || p->jdir >= a->nv || p->n_iter < 0 || p->cg_iters < 0 ||
        p->grad_cg < 0 || p->n_calls > a->nc + 2 || p->rho_mode < 0 || p->rho_mode > B2C_ADMM_RHO_GIVEN) {
        set_error("b2c_admm_solve: bad parameters (flags %d: exactly one of FORWARD and GRAD_GIVEN; jdir %d)", p->flags,
                  p->jdir);
        return B2C_EARG;
    }
    if (!a->J || !a->Minv || !a->v_free || !a->mu || !a->lam || !a->u ||
        (fwd && !a->v_plus) || ((grad || given) && (!a->dlam_tau || !a->labels || !a->nslip)) ||
        (grad && (!a->dv_tau || !a->dlam_mu)) || (given && !a->dbv_in) ||
        (p->rho_mode == B2C_ADMM_RHO_GIVEN && !a->rho)) {
        set_error("b2c_admm_solve: a required array is NULL");
        return B2C_EARG;
    }
    if (a->n_env == 0) return B2C_OK;
    switch (a->nc) {
#define B2C_ADMM_CASE(n)                              \
    case n:                                           \
        badmm::launch<n>(*a, *p, stream_of(st));      \
        break;
        B2C_ADMM_CASE(1)
        B2C_ADMM_CASE(2)
        B2C_ADMM_CASE(3)
        B2C_ADMM_CASE(4)
        B2C_ADMM_CASE(5)
        B2C_ADMM_CASE(6)
        B2C_ADMM_CASE(7)
        B2C_ADMM_CASE(8)
#undef B2C_ADMM_CASE
    }
    return check_launch("admm");
}
