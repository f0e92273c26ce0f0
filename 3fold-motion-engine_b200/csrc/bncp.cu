// Batched exact-cone NCP in Delassus form with its implicit sensitivity (the reference's
// batched adjoint, src/motion_engine/ncp/ncp_batch_gpu.py:918-1313, and the CPU
// implicit-function response of src/motion_engine/ncp/ncp_ref.py:786-959).
//
// Every environment e holds a small contact problem: G_e (n x n, n = 3 n_c <= 48), b_e, mu_e.
// In the solve one lane owns one contact, a problem the power of two of lanes that holds its
// contacts (see k_solve); in the adjoint one warp owns one environment, its matrices in shared
// memory:
//
//   solve     projected Gauss-Seidel over the contacts, lambda_c <- proj_K(lambda_c - rho_c
//             (u_c + Gamma(u_c))), u = G lambda + b, rho_c = 1 / lambda_max(G_cc) (the sweep of
//             ncp_gpu.py:485-568 on the Delassus operator), until the natural residual
//             max_c |lambda_c - proj_K(...)| is below tol (checked every `check` sweeps; the
//             convergence mask of the batched solver) or max_iters;
//   adjoint   the contacts labelled open / stick / slip from lambda (ncp_ref.classify,
//             :251-274), the fixed-branch residual Jacobian A and the parameter maps Bmu, Bb
//             (ncp_ref._active_system, :786-842), LU with partial pivoting, then either the full
//             responses X = -A^-1 [Bmu Bb] (ncp_ref.sensitivity) or the vector-Jacobian product
//             y = A^-T g, dL/db = -Bb^T y, dL/dmu = -Bmu^T y.  A pivot below 1e-12 max|A| marks
//             the branch singular and, like a branch boundary, returns NaN (the reference's
//             guarded_response without a selection).
//
// Sums run in a fixed order that padding with empty contacts does not change, so results are
// bit-identical run to run and whatever a batch is padded to.
#include <type_traits>

#include "b2c_common.cuh"

namespace b2c {
namespace bncp {

constexpr int kMaxN = 48;  // 3 x 16 contacts

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ double eigmax3(const double W[3][3])
{
    const double c2 = W[0][0] + W[1][1] + W[2][2];
    const double c1 = (W[0][0] * W[1][1] - W[0][1] * W[1][0]) + (W[0][0] * W[2][2] - W[0][2] * W[2][0]) +
                      (W[1][1] * W[2][2] - W[1][2] * W[2][1]);
    const double c0 = W[0][0] * (W[1][1] * W[2][2] - W[1][2] * W[2][1]) -
                      W[0][1] * (W[1][0] * W[2][2] - W[1][2] * W[2][0]) +
                      W[0][2] * (W[1][0] * W[2][1] - W[1][1] * W[2][0]);
    double x = 0.0;
    for (int i = 0; i < 3; ++i) {
        const double r = W[i][i] + fabs(W[i][(i + 1) % 3]) + fabs(W[i][(i + 2) % 3]);
        if (r > x) x = r;
    }
    if (!(x > 0.0)) return 0.0;
    for (int it = 0; it < 100; ++it) {
        const double p = ((x - c2) * x + c1) * x - c0;
        const double dp = (3.0 * x - 2.0 * c2) * x + c1;
        if (!(dp > 0.0)) break;
        const double xn = x - p / dp;
        if (!(xn < x)) break;
        x = xn;
    }
    return x;
}

// u_r = b_r + sum_j G[r][j] lam[j] for the warp, every lane returns it
__device__ __forceinline__ double row_u(const double *G, const double *lam, const double *b, int n, int r, int lane)
{
    double s = 0.0;
    for (int j = lane; j < n; j += 32) s += G[r * n + j] * lam[j];
    return warp_sum(s) + b[r];
}

// One contact's update: the projection onto K_mu of lambda - rho (u + Gamma(u)), den = 1 + mu^2
// and iden its reciprocal.  The slip speed |u_t| and the tangential length |z_t| do not wait for
// each other; |z_t| and its reciprocal come from one reciprocal square root, and each quotient by
// a known reciprocal takes one correction by its remainder (q + (a - q b) / b), as |z_t| does, so
// that all three are as good as the rounded operations they stand for.
__device__ __forceinline__ void update(const double u[3], const double lo[3], double mu, double rho, double den,
                                       double iden, double out[3])
{
    const double z1 = lo[1] - rho * u[1], z2 = lo[2] - rho * u[2];
    const double zz = fma(z1, z1, z2 * z2), rz = rsqrt(zz);
    double zt = zz * rz;
    zt = zz > 0.0 ? fma(fma(-zt, zt, zz), 0.5 * rz, zt) : 0.0;
    const double zn = lo[0] - rho * fma(mu, sqrt(fma(u[1], u[1], u[2] * u[2])), u[0]);
    const double num = fma(mu, zt, zn);
    double s = num * iden;
    s = fma(fma(-s, den, num), iden, s);
    const double ms = mu * s;
    double f = ms * rz;
    f = fma(fma(-f, zt, ms), rz, f);
    const bool inside = zt <= mu * zn, below = mu * zt <= -zn;
    out[0] = inside ? zn : below ? 0.0 : s;
    out[1] = inside ? z1 : below ? 0.0 : f * z1;
    out[2] = inside ? z2 : below ? 0.0 : f * z2;
}

// Lanes of a problem of at most C contacts: the power of two that holds them.
template <int C>
struct Lanes {
    static constexpr int L = C <= 1 ? 1 : C <= 2 ? 2 : C <= 4 ? 4 : C <= 8 ? 8 : 16;
    static constexpr int PW = 32 / L;      // problems of a warp
    static constexpr int M = 3 * C;
    static constexpr bool kRegs = C <= 8;  // G's rows and lambda in registers, else in shared memory
    static constexpr int S = M | 1;        // row stride in shared memory
};

// Projected Gauss-Seidel, one lane a contact.  A lane keeps its contact's three rows of G and all
// of its problem's lambda in registers (3 x 3C + 3C float64; above 8 contacts in shared memory).
// Contact c's turn: every lane sums its own rows, of which only lane c's count, lane c's updated
// impulse goes to the others by shuffle.  Row c is summed from contact c on around to contact
// c - 1, so only its last three terms wait for the update before it and the rest of the row is
// summed beside that update's square roots.  What bounds it is that chain -- three multiply-adds,
// a square root, the projection, a shuffle -- times the sweeps of a batch's slowest problems, so
// the split puts as many problems in a warp as have lanes to own their contacts.
//
// Measured on a B200 to a residual of 1e-6 (before: a warp a problem, a butterfly per row), B
// problems: 4 contacts B = 64 1.42 -> 0.31 ms, B = 4096 4.34 -> 0.87 ms, B = 16384 5.5 -> 1.0 ms
// (the slowest problem's 940 sweeps); at B = 4096, 1 contact 107 -> 28 us, 8 contacts 20.0 ->
// 4.9 ms.  Error of lambda against 80-bit arithmetic, same sweeps: 1 contact 1.2e-16 -> 1.1e-16 of
// its norm, 4 contacts 2.5e-16 -> 2.2e-16.
//
// Above 8 contacts the rows come from shared memory, whose bandwidth bounds a full SM, so a
// problem's rows have its batch's length, only the lane whose turn it is reads its own, and a warp
// stops at its own problems' contacts.  100 sweeps of 4 096 problems, us, a warp a problem before:
// 9 contacts 1 502 -> 1 006, 12 3 346 -> 1 990, 16 6 136 -> 4 515, 1 to 16 at random 3 990 -> 4 150;
// padded, 1 contact each in a batch of 8: 192 -> 125.
template <int C>
__global__ void __launch_bounds__(32) k_solve(int n_env, int n_max, const int *__restrict__ ncs,
                                              const double *__restrict__ G, const double *__restrict__ b,
                                              const double *__restrict__ mu, double *__restrict__ lam_io,
                                              double *__restrict__ res_out, int *__restrict__ iters_out,
                                              int max_iters, double tol, int check)
{
    using D = Lanes<C>;
    constexpr int M = D::M, R = D::kRegs ? M : 1, U = D::kRegs ? C : 1;
    extern __shared__ double sm[];
    const int lane = (int)(threadIdx.x & 31), pg = lane / D::L, me = lane % D::L;
    const int e = (int)blockIdx.x * D::PW + pg, ec = e < n_env ? e : n_env - 1;
    const int ncm = n_max / 3, nc = min(ncs[ec], ncm);
    const bool own = me < nc;
    const double *Ge = G + (size_t)ec * n_max * n_max;
    double *Gs = sm + (size_t)pg * (M * D::S + M), *xs = Gs + M * D::S;  // kRegs: not used
    // the most contacts of a problem of the warp: above 8 its turns and rows end there; up to 8, where
    // it is a third of C or less (a batch of padded problems), there are only so many turns.  A
    // reduction, not shuffles: the branches on it are then known to be the same for the whole warp.
    const int cm = __reduce_max_sync(0xffffffffu, nc);
    double g[3][R], x[R], bb[3] = {0.0, 0.0, 0.0}, rho = 0.0, m = 0.0;
    if (D::kRegs) {
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int j = 0; j < R; ++j)
                g[k][j] = own && j < 3 * nc ? Ge[(size_t)(3 * me + k) * n_max + j] : 0.0;
#pragma unroll
        for (int j = 0; j < R; ++j) x[j] = j < 3 * nc ? lam_io[(size_t)ec * n_max + j] : 0.0;
    } else {
        for (int k = 0; k < 3; ++k)
            for (int j = 0; j < M; ++j)
                if (me < C) Gs[(3 * me + k) * D::S + j] = own && j < 3 * nc ? Ge[(size_t)(3 * me + k) * n_max + j] : 0.0;
        for (int k = 0; k < 3; ++k)
            if (me < C) xs[3 * me + k] = own ? lam_io[(size_t)ec * n_max + 3 * me + k] : 0.0;
        __syncwarp();
    }
    if (own) {
        m = mu[(size_t)ec * ncm + me];
        double W[3][3];
        for (int i = 0; i < 3; ++i) {
            bb[i] = b[(size_t)ec * n_max + 3 * me + i];
            for (int j = 0; j < 3; ++j) W[i][j] = Ge[(size_t)(3 * me + i) * n_max + 3 * me + j];
        }
        const double lm = eigmax3(W);
        rho = lm > 1e-300 ? 1.0 / lm : 0.0;
    }
    const double den = 1.0 + m * m, iden = 1.0 / den;
    // the lane's rows times lambda plus b, from contact `first` on
    auto rows = [&](int first, double u[3]) {
#pragma unroll
        for (int k = 0; k < 3; ++k) u[k] = bb[k];
        if (D::kRegs) {
#pragma unroll
            for (int q = 0; q < U; ++q) {
                const int j = 3 * ((first + q) % C);
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    u[k] = fma(g[k][j + 2], x[j + 2], fma(g[k][j + 1], x[j + 1], fma(g[k][j], x[j], u[k])));
            }
        } else {
            const double *r0 = Gs + 3 * (me < C ? me : 0) * D::S;
            auto part = [&](int from, int to) {
#pragma unroll 4
                for (int c = from; c < to; ++c) {
                    const int j = 3 * c;
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const double *r = r0 + k * D::S;
                        u[k] = fma(r[j + 2], xs[j + 2], fma(r[j + 1], xs[j + 1], fma(r[j], xs[j], u[k])));
                    }
                }
            };
            if (cm == C) {  // the bound known when compiled: 1.3 times as fast at 16 contacts
#pragma unroll
                for (int q = 0; q < C; ++q) {
                    const int c = first + q < C ? first + q : first + q - C, j = 3 * c;
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const double *r = r0 + k * D::S;
                        u[k] = fma(r[j + 2], xs[j + 2], fma(r[j + 1], xs[j + 1], fma(r[j], xs[j], u[k])));
                    }
                }
            } else {
                part(first, cm);
                part(0, first);
            }
        }
    };
    // max over the problem's contacts of |lambda_c - its update| (fmax drops a NaN)
    auto residual = [&]() -> double {
        double u[3], out[3], lo[3] = {0.0, 0.0, 0.0};
        rows(0, u);
        if (D::kRegs) {
#pragma unroll
            for (int j = 0; j < U; ++j)
                if (j == me) {
#pragma unroll
                    for (int k = 0; k < 3; ++k) lo[k] = x[3 * j + k];
                }
        } else {
            for (int k = 0; k < 3; ++k) lo[k] = me < C ? xs[3 * me + k] : 0.0;
        }
        update(u, lo, m, rho, den, iden, out);
        double r = own ? fmax(fmax(fmax(0.0, fabs(lo[0] - out[0])), fabs(lo[1] - out[1])), fabs(lo[2] - out[2])) : 0.0;
#pragma unroll
        for (int o = D::L / 2; o > 0; o >>= 1) r = fmax(r, __shfl_xor_sync(0xffffffffu, r, o));
        return r;
    };
    bool run = e < n_env;
    double res = 0.0;
    int iters = max_iters;
    // the sweeps, over T turns (in shared memory cm)
    auto sweeps = [&](auto turns) {
        constexpr int T = decltype(turns)::value;
        for (int it = 0; it < max_iters; ++it) {
            if (check > 0 && it % check == 0) {
                const double r = residual();
                if (run) {
                    res = r;
                    if (r < tol) {
                        run = false;
                        iters = it;
                    }
                }
                if (!__any_sync(0xffffffffu, run)) break;
            }
#pragma unroll U
            for (int c = 0; c < (D::kRegs ? T : cm); ++c) {
                double u[3], out[3], lo[3];
                if (D::kRegs || me == c) {  // in shared memory the other lanes' rows would only cost its bandwidth
                    rows(c, u);
#pragma unroll
                    for (int k = 0; k < 3; ++k) lo[k] = D::kRegs ? x[(3 * c + k) % R] : xs[3 * c + k];
                    update(u, lo, m, rho, den, iden, out);
                }
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const double v = __shfl_sync(0xffffffffu, out[k], c, D::L);
                    if (run && c < nc) {
                        if (D::kRegs) x[(3 * c + k) % R] = v;
                        else if (me == 0) xs[3 * c + k] = v;
                    }
                }
                if (!D::kRegs) __syncwarp();
            }
        }
    };
    if (D::kRegs && 3 * cm <= C) sweeps(std::integral_constant<int, C / 3>{});
    else sweeps(std::integral_constant<int, C>{});
    if (__any_sync(0xffffffffu, run)) {  // the residual of the final iterate
        const double r = residual();
        if (run) res = r;
    }
    if (e >= n_env) return;
    if (D::kRegs) {
#pragma unroll
        for (int j = 0; j < R; ++j)
            if (j < n_max && j % D::L == me) lam_io[(size_t)e * n_max + j] = j < 3 * nc ? x[j] : 0.0;
    } else {
        for (int j = me; j < n_max; j += D::L) lam_io[(size_t)e * n_max + j] = j < 3 * nc ? xs[j] : 0.0;
    }
    if (me == 0) {
        res_out[e] = res;
        iters_out[e] = iters;
    }
}

// Fixed-branch system of one environment into shared memory: A (n x n), Bmu (n x nc), Bb (n x n).
// Returns the status bits (2 = a branch boundary); labels written per contact.
__device__ int assemble(const double *Gs, const double *bs, const double *lam, const double *mus, int n, int nc,
                        double *A, double *Bmu, double *Bb, int *labels, int lane)
{
    __shared__ double s_u[kMaxN];
    for (int r = 0; r < n; ++r) {
        const double u = row_u(Gs, lam, bs, n, r, lane);
        if (lane == 0) s_u[r] = u;
    }
    for (int i = lane; i < n * n; i += 32) {
        A[i] = 0.0;
        Bb[i] = 0.0;
    }
    for (int i = lane; i < n * nc; i += 32) Bmu[i] = 0.0;
    __syncwarp();
    int status = 0;
    if (lane == 0) {
        double scale = 0.0;
        for (int i = 0; i < n; ++i) scale = fmax(scale, fabs(lam[i]));
        scale = fmax(scale, 1e-30);
        for (int c = 0; c < nc; ++c) {
            const int i = 3 * c;
            const double ln = lam[i], lt = sqrt(lam[i + 1] * lam[i + 1] + lam[i + 2] * lam[i + 2]);
            const double m = mus[c];
            int lab;
            if (ln <= 1e-10 + 1e-6 * scale) lab = 0;
            else if (lt >= m * ln * (1.0 - 1e-6) - 1e-10) lab = 2;
            else lab = 1;
            labels[c] = lab;
            if (lab == 0) {
                for (int k = 0; k < 3; ++k) A[(i + k) * n + i + k] = 1.0;
                if (fabs(s_u[i]) < 1e-9) status |= 2;
            } else if (lab == 1) {
                for (int k = 0; k < 3; ++k) {
                    for (int j = 0; j < n; ++j) A[(i + k) * n + j] = Gs[(i + k) * n + j];
                    Bb[(i + k) * n + i + k] = 1.0;
                }
            } else {
                for (int j = 0; j < n; ++j) A[i * n + j] = Gs[i * n + j];
                Bb[i * n + i] = 1.0;
                const double s0 = s_u[i + 1], s1 = s_u[i + 2];
                double ns = sqrt(s0 * s0 + s1 * s1);
                if (ns < 1e-14) {
                    status |= 2;
                    ns = 1e-14;
                }
                const double h0 = s0 / ns, h1 = s1 / ns;
                const double P[2][2] = {{(1.0 - h0 * h0) / ns, (-h0 * h1) / ns}, {(-h1 * h0) / ns, (1.0 - h1 * h1) / ns}};
                const double ml = m * ln;
                for (int a = 0; a < 2; ++a) {
                    for (int j = 0; j < n; ++j)
                        A[(i + 1 + a) * n + j] = ml * (P[a][0] * Gs[(i + 1) * n + j] + P[a][1] * Gs[(i + 2) * n + j]);
                    A[(i + 1 + a) * n + i] += m * (a == 0 ? h0 : h1);
                    A[(i + 1 + a) * n + i + 1 + a] += 1.0;
                    Bb[(i + 1 + a) * n + i + 1] = ml * P[a][0];
                    Bb[(i + 1 + a) * n + i + 2] = ml * P[a][1];
                    Bmu[(i + 1 + a) * nc + c] = ln * (a == 0 ? h0 : h1);
                }
            }
            const double sc = fmax(fabs(ln), 1e-12);
            if (lab == 1 && fabs(lt - m * ln) < 1e-7 * m * sc) status |= 2;
            if (lab != 0 && ln < 1e-9) status |= 2;
        }
    }
    __syncwarp();
    return __shfl_sync(0xffffffffu, status, 0);
}

// In-place LU with partial pivoting of A (n x n); piv[k] = row swapped with k.  Returns 1 when a
// pivot is below 1e-12 max|A| (the branch is numerically singular).
__device__ int lu(double *A, int *piv, int n, int lane)
{
    double amax = 0.0;
    for (int i = lane; i < n * n; i += 32) amax = fmax(amax, fabs(A[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    for (int k = 0; k < n; ++k) {
        // pivot: the largest |A[r][k]|, r >= k (lowest row on ties)
        double best = -1.0;
        int br = k;
        for (int r = k + lane; r < n; r += 32) {
            const double v = fabs(A[r * n + k]);
            if (v > best) {
                best = v;
                br = r;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int orr = __shfl_xor_sync(0xffffffffu, br, o);
            if (ov > best || (ov == best && orr < br)) {
                best = ov;
                br = orr;
            }
        }
        if (!(best > 1e-12 * amax)) return 1;
        if (lane == 0) piv[k] = br;
        if (br != k)
            for (int j = lane; j < n; j += 32) {
                const double t = A[k * n + j];
                A[k * n + j] = A[br * n + j];
                A[br * n + j] = t;
            }
        __syncwarp();
        const double d = A[k * n + k];
        for (int r = k + 1 + lane; r < n; r += 32) A[r * n + k] /= d;
        __syncwarp();
        for (int idx = lane; idx < (n - k - 1) * (n - k - 1); idx += 32) {
            const int r = k + 1 + idx / (n - k - 1), j = k + 1 + idx % (n - k - 1);
            A[r * n + j] -= A[r * n + k] * A[k * n + j];
        }
        __syncwarp();
    }
    return 0;
}

// X (n x m, row-major) <- A^-1 X with the factors of lu()
__device__ void lu_solve(const double *A, const int *piv, int n, double *X, int m, int lane)
{
    for (int k = 0; k < n; ++k) {
        const int p = piv[k];
        if (p != k)
            for (int j = lane; j < m; j += 32) {
                const double t = X[k * m + j];
                X[k * m + j] = X[p * m + j];
                X[p * m + j] = t;
            }
    }
    __syncwarp();
    for (int j = lane; j < m; j += 32) {
        for (int r = 1; r < n; ++r) {
            double s = X[r * m + j];
            for (int k = 0; k < r; ++k) s -= A[r * n + k] * X[k * m + j];
            X[r * m + j] = s;
        }
        for (int r = n - 1; r >= 0; --r) {
            double s = X[r * m + j];
            for (int k = r + 1; k < n; ++k) s -= A[r * n + k] * X[k * m + j];
            X[r * m + j] = s / A[r * n + r];
        }
    }
    __syncwarp();
}

// y <- A^-T y with the factors of lu() (A = P^T L U, so A^T y = g is U^T L^T P y = g)
__device__ void lu_solve_t(const double *A, const int *piv, int n, double *y, int lane)
{
    if (lane == 0) {
        for (int r = 0; r < n; ++r) {  // U^T z = g
            double s = y[r];
            for (int k = 0; k < r; ++k) s -= A[k * n + r] * y[k];
            y[r] = s / A[r * n + r];
        }
        for (int r = n - 1; r >= 0; --r) {  // L^T w = z (unit diagonal)
            double s = y[r];
            for (int k = r + 1; k < n; ++k) s -= A[k * n + r] * y[k];
            y[r] = s;
        }
        for (int k = n - 1; k >= 0; --k) {  // y = P^T w: undo the swaps in reverse
            const int p = piv[k];
            if (p != k) {
                const double t = y[k];
                y[k] = y[p];
                y[p] = t;
            }
        }
    }
    __syncwarp();
}

// A warp's matrices are sized by the batch's largest problem, C contacts: at 4 contacts 4.2 KB, so 32
// warps fit an SM where the 64 KB of a 16-contact problem let three (4096 problems: 285 -> 56 us).
// C is a template parameter because the matrices' places are then known when the kernel is
// compiled (a place worked out from n_max cost a batch of 16 problems 3 to 4 %, 8 contacts
// 71.8 -> 74.9 us).
template <int C>
constexpr size_t adjoint_smem()
{
    return sizeof(double) * (27 * C * C + 3 * C * C + 9 * C + C);
}

// mode 0: full responses dlam/dmu (n x nc) and dlam/db (n x n); mode 1: vector-Jacobian product
template <int C>
__global__ void __launch_bounds__(32) k_adjoint(int n_env, int n_max, const int *__restrict__ ncs,
                                                const double *__restrict__ G, const double *__restrict__ b,
                                                const double *__restrict__ mu, const double *__restrict__ lam_in,
                                                int *__restrict__ labels_out, int *__restrict__ status_out, int mode,
                                                double *__restrict__ dmu, double *__restrict__ db,
                                                const double *__restrict__ glam, double *__restrict__ gb,
                                                double *__restrict__ gmu)
{
    extern __shared__ double sm[];
    const int e = blockIdx.x, lane = threadIdx.x;
    if (e >= n_env) return;
    const int nc = ncs[e], n = 3 * nc, ncm = n_max / 3;
    constexpr int N = 3 * C;
    double *Gs = sm, *A = Gs + N * N, *Bb = A + N * N, *Bmu = Bb + N * N;
    double *bs = Bmu + N * C, *lam = bs + N, *mus = lam + N, *y = mus + C;
    __shared__ int piv[kMaxN];
    __shared__ int labels[kMaxN / 3];
    const double *Ge = G + (size_t)e * n_max * n_max;
    for (int i = lane; i < n * n; i += 32) Gs[i] = Ge[(i / n) * n_max + (i % n)];
    for (int i = lane; i < n; i += 32) {
        bs[i] = b[(size_t)e * n_max + i];
        lam[i] = lam_in[(size_t)e * n_max + i];
    }
    for (int c = lane; c < nc; c += 32) mus[c] = mu[(size_t)e * ncm + c];
    __syncwarp();
    int status = assemble(Gs, bs, lam, mus, n, nc, A, Bmu, Bb, labels, lane);
    if (lu(A, piv, n, lane)) status |= 1;
    for (int c = lane; c < ncm; c += 32) labels_out[(size_t)e * ncm + c] = c < nc ? labels[c] : 0;
    if (lane == 0) status_out[e] = status;
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    if (mode == 0) {
        // X = -A^-1 [Bmu | Bb], columns solved together in Bb-sized chunks
        double *X = Bb;  // n x n, Bb's own storage (Bb is not needed after the copy below)
        if (!status) {
            // Bmu columns first, into y-sized scratch one column at a time
            for (int c = 0; c < nc; ++c) {
                for (int r = lane; r < n; r += 32) y[r] = -Bmu[r * nc + c];
                __syncwarp();
                lu_solve(A, piv, n, y, 1, lane);
                for (int r = lane; r < n; r += 32) dmu[((size_t)e * n_max + r) * ncm + c] = y[r];
                __syncwarp();
            }
            for (int i = lane; i < n * n; i += 32) X[i] = -X[i];
            __syncwarp();
            lu_solve(A, piv, n, X, n, lane);
        }
        for (int i = lane; i < n_max * n_max; i += 32) {
            const int r = i / n_max, j = i % n_max;
            db[(size_t)e * n_max * n_max + i] = (r < n && j < n) ? (status ? nan : X[r * n + j]) : 0.0;
        }
        for (int i = lane; i < n_max * ncm; i += 32) {
            const int r = i / ncm, c = i % ncm;
            if (status || r >= n || c >= nc)
                dmu[(size_t)e * n_max * ncm + i] = (r < n && c < nc) ? nan : 0.0;
        }
    } else {
        for (int r = lane; r < n; r += 32) y[r] = glam[(size_t)e * n_max + r];
        __syncwarp();
        if (!status) lu_solve_t(A, piv, n, y, lane);
        // dL/db = -Bb^T y, dL/dmu = -Bmu^T y
        for (int j = lane; j < n_max; j += 32) {
            double s = 0.0;
            if (j < n)
                for (int r = 0; r < n; ++r) s -= Bb[r * n + j] * y[r];
            gb[(size_t)e * n_max + j] = j < n ? (status ? nan : s) : 0.0;
        }
        for (int c = lane; c < ncm; c += 32) {
            double s = 0.0;
            if (c < nc)
                for (int r = 0; r < n; ++r) s -= Bmu[r * nc + c] * y[r];
            gmu[(size_t)e * ncm + c] = c < nc ? (status ? nan : s) : 0.0;
        }
    }
}

template <int C>
int32_t solve(const b2c_bncp *p, int max_iters, double tol, int check, cudaStream_t st)
{
    using D = Lanes<C>;
    const size_t smem = D::kRegs ? 0 : sizeof(double) * D::PW * (size_t)(D::M * D::S + D::M);
    k_solve<C><<<(p->n_env + D::PW - 1) / D::PW, 32, smem, st>>>(p->n_env, p->n_max, p->nc, p->G, p->b, p->mu, p->lam,
                                                                  p->res, p->iters, max_iters, tol, check);
    return check_launch("bncp_solve");
}

template <int C>
int32_t adjoint(const b2c_bncp *p, int mode, double *dmu, double *db, const double *glam, double *gb, double *gmu,
                cudaStream_t st)
{
    // the opt-in above 48 KB is the device's, so for every launch
    cudaFuncSetAttribute(k_adjoint<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)adjoint_smem<C>());
    k_adjoint<C><<<p->n_env, 32, adjoint_smem<C>(), st>>>(p->n_env, p->n_max, p->nc, p->G, p->b, p->mu, p->lam,
                                                          p->labels, p->status, mode, dmu, db, glam, gb, gmu);
    return check_launch("bncp_adjoint");
}

}  // namespace bncp
}  // namespace b2c

static bool bncp_ok(const b2c_bncp *p)
{
    return p && p->n_env >= 0 && p->n_max >= 3 && p->n_max % 3 == 0 && p->n_max <= b2c::bncp::kMaxN && p->nc &&
           p->G && p->b && p->mu && p->lam && p->res && p->iters && p->labels && p->status;
}

extern "C" int32_t b2c_bncp_max_rows(void) { return b2c::bncp::kMaxN; }

extern "C" int32_t b2c_bncp_solve(const b2c_bncp *p, int32_t max_iters, double tol, int32_t check, b2c_stream s)
{
    if (!bncp_ok(p) || max_iters < 0) {
        b2c::set_error("b2c_bncp_solve: bad argument (n_max must be a multiple of 3, at most %d)", b2c::bncp::kMaxN);
        return B2C_EARG;
    }
    if (p->n_env == 0) return B2C_OK;
    const cudaStream_t st = b2c::stream_of(s);
    switch (p->n_max / 3) {
        case 1: return b2c::bncp::solve<1>(p, max_iters, tol, check, st);
        case 2: return b2c::bncp::solve<2>(p, max_iters, tol, check, st);
        case 3: return b2c::bncp::solve<3>(p, max_iters, tol, check, st);
        case 4: return b2c::bncp::solve<4>(p, max_iters, tol, check, st);
        case 5: return b2c::bncp::solve<5>(p, max_iters, tol, check, st);
        case 6: return b2c::bncp::solve<6>(p, max_iters, tol, check, st);
        case 7: return b2c::bncp::solve<7>(p, max_iters, tol, check, st);
        case 8: return b2c::bncp::solve<8>(p, max_iters, tol, check, st);
        case 9: return b2c::bncp::solve<9>(p, max_iters, tol, check, st);
        case 10: return b2c::bncp::solve<10>(p, max_iters, tol, check, st);
        case 11: return b2c::bncp::solve<11>(p, max_iters, tol, check, st);
        case 12: return b2c::bncp::solve<12>(p, max_iters, tol, check, st);
        case 13: return b2c::bncp::solve<13>(p, max_iters, tol, check, st);
        case 14: return b2c::bncp::solve<14>(p, max_iters, tol, check, st);
        case 15: return b2c::bncp::solve<15>(p, max_iters, tol, check, st);
        default: return b2c::bncp::solve<16>(p, max_iters, tol, check, st);
    }
}

static int32_t bncp_adjoint(const b2c_bncp *p, int mode, double *dmu, double *db, const double *glam, double *gb,
                            double *gmu, b2c_stream s)
{
    if (p->n_env == 0) return B2C_OK;
    const cudaStream_t st = b2c::stream_of(s);
    switch (p->n_max / 3) {
#define B2C_BNCP_CASE(c) \
    case c: return b2c::bncp::adjoint<c>(p, mode, dmu, db, glam, gb, gmu, st);
        B2C_BNCP_CASE(1)
        B2C_BNCP_CASE(2)
        B2C_BNCP_CASE(3)
        B2C_BNCP_CASE(4)
        B2C_BNCP_CASE(5)
        B2C_BNCP_CASE(6)
        B2C_BNCP_CASE(7)
        B2C_BNCP_CASE(8)
        B2C_BNCP_CASE(9)
        B2C_BNCP_CASE(10)
        B2C_BNCP_CASE(11)
        B2C_BNCP_CASE(12)
        B2C_BNCP_CASE(13)
        B2C_BNCP_CASE(14)
        B2C_BNCP_CASE(15)
#undef B2C_BNCP_CASE
        default: return b2c::bncp::adjoint<16>(p, mode, dmu, db, glam, gb, gmu, st);
    }
}

extern "C" int32_t b2c_bncp_sensitivity(const b2c_bncp *p, double *dlam_dmu, double *dlam_db, b2c_stream s)
{
    if (!bncp_ok(p) || !dlam_dmu || !dlam_db) {
        b2c::set_error("b2c_bncp_sensitivity: bad argument");
        return B2C_EARG;
    }
    return bncp_adjoint(p, 0, dlam_dmu, dlam_db, nullptr, nullptr, nullptr, s);
}

extern "C" int32_t b2c_bncp_vjp(const b2c_bncp *p, const double *glam, double *gb, double *gmu, b2c_stream s)
{
    if (!bncp_ok(p) || !glam || !gb || !gmu) {
        b2c::set_error("b2c_bncp_vjp: bad argument");
        return B2C_EARG;
    }
    return bncp_adjoint(p, 1, nullptr, nullptr, glam, gb, gmu, s);
}
