// Exact-cone NCP solve: the coloured projected Gauss-Seidel of the reference's NCPSolverGPU
// (src/motion_engine/ncp/ncp_gpu.py:361-1063) on per-contact 3x6 Jacobian blocks, in float32 or
// float64.
//
//   setup     rho_c = 1 / lambda_max(Ja Minv_a Ja^T + Jb Minv_b Jb^T) (k_rho, :441-459; the
//             largest eigenvalue by Newton's method on the characteristic polynomial from the
//             Gershgorin bound, in float64), acc = sum_c round(1e10 Minv J_c^T lambda_c) of the
//             warm start (k_scatter, :468-483), v = v_free + acc / 1e10 (k_apply, :570-581);
//   colour    Jones-Plassmann over the contacts, claims on dynamic bodies only (k_claim /
//             k_win, :682-722), priority a bijective 64-bit hash of the canonical key
//             (body_a, body_b, feature) (:656-664), so the colouring is a pure function of the
//             contact set and not of its order; cached while pairs, features and masses stay
//             the same (k_cache_cmp, :736-765);
//   sweeps    per colour, per contact: u = bias + Ja v_a + Jb v_b, the de Saxce term, the
//             soft-step branch, lambda <- proj_K(z) (k_sweep, :485-568); acc swaps the contact's
//             old rounded contribution for the new one (f_swap, :425-438) and the velocity of
//             the contact's dynamic bodies is rebuilt from acc at once (k_apply_c, :583-599: a
//             colour holds each dynamic body at most once, so the thread that owns the contact
//             owns those bodies for the phase).  All colours of all iterations run in ONE
//             persistent launch with a barrier between colours (one CTA, a cluster, a grid);
//   residual  max_c |lambda_c - proj_K(z_c)| of the same map (k_resid, :601-649).
//
// Every sum runs in index order with separately rounded operations (the library is built
// with -fmad=false), so the oracle's C restatement reproduces the results bit for bit.
#include <cooperative_groups.h>

#include "b2c_barrier.cuh"
#include "b2c_common.cuh"

namespace cg = cooperative_groups;

namespace b2c {
namespace ncp {

constexpr double kScale = 1.0e10;
constexpr int kColorThreads = 1024;
constexpr int kClusterMax = 16;
constexpr int kMaxColors = 1024;  // the reference's _NCOLMAX

enum Stat { kNColors = 0, kCacheValid = 1, kCachedC = 2, kCacheHit = 3, kHits = 4, kMisses = 5, kRounds = 6,
            kError = 7 };
enum ErrBit { kErrColorOverflow = 1, kErrColorTimeout = 2, kErrBarrier = 4 };

__device__ __forceinline__ float rsq(float x) { return sqrtf(x); }
__device__ __forceinline__ double rsq(double x) { return sqrt(x); }
__device__ __forceinline__ float rab(float x) { return fabsf(x); }
__device__ __forceinline__ double rab(double x) { return fabs(x); }

// splitmix64's output function: a bijection of 64-bit integers
__device__ __forceinline__ unsigned long long mix64(unsigned long long z)
{
    z ^= z >> 30;
    z *= 0xbf58476d1ce4e5b9ULL;
    z ^= z >> 27;
    z *= 0x94d049bb133111ebULL;
    z ^= z >> 31;
    return z;
}

// largest eigenvalue of a symmetric positive semi-definite 3x3: Newton's method on the
// characteristic polynomial p(x) = x^3 - c2 x^2 + c1 x - c0 from the Gershgorin bound; the
// iterates decrease monotonically to the largest root
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

template <typename T>
__device__ void add_jmjt(T W[3][3], const T *__restrict__ J, const T *__restrict__ M)
{
    T Tm[3][6];
    for (int i = 0; i < 3; ++i)
        for (int l = 0; l < 6; ++l) {
            T s = J[i * 6 + 0] * M[0 * 6 + l];
            for (int k = 1; k < 6; ++k) s = s + J[i * 6 + k] * M[k * 6 + l];
            Tm[i][l] = s;
        }
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
            T s = Tm[i][0] * J[j * 6 + 0];
            for (int l = 1; l < 6; ++l) s = s + Tm[i][l] * J[j * 6 + l];
            W[i][j] = W[i][j] + s;
        }
}

template <typename T>
__global__ void k_rho(int nc, const T *__restrict__ Ja, const T *__restrict__ Jb, const T *__restrict__ Minv,
                      const int *__restrict__ pa, const int *__restrict__ pb, T *__restrict__ rho)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nc) return;
    T W[3][3] = {{T(0), T(0), T(0)}, {T(0), T(0), T(0)}, {T(0), T(0), T(0)}};
    if (pa[c] >= 0) add_jmjt(W, Ja + 18 * (size_t)c, Minv + 36 * (size_t)pa[c]);
    if (pb[c] >= 0) add_jmjt(W, Jb + 18 * (size_t)c, Minv + 36 * (size_t)pb[c]);
    double Wd[3][3];
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) Wd[i][j] = (double)W[i][j];
    const double lm = eigmax3(Wd);
    rho[c] = lm > 1e-14 ? (T)(1.0 / lm) : T(0);
}

template <typename T>
__global__ void k_dyn(int nb, const T *__restrict__ Minv, int *__restrict__ dyn)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nb) return;
    int d = 0;
    for (int k = 0; k < 36; ++k) d |= Minv[36 * (size_t)i + k] != T(0);
    dyn[i] = d;
}

// d = Minv (J^T l)
template <typename T>
__device__ __forceinline__ void minv_jt(const T *__restrict__ J, const T *__restrict__ M, const T l[3], T d[6])
{
    T t[6];
    for (int j = 0; j < 6; ++j) {
        T s = J[0 * 6 + j] * l[0];
        s = s + J[1 * 6 + j] * l[1];
        s = s + J[2 * 6 + j] * l[2];
        t[j] = s;
    }
    for (int k = 0; k < 6; ++k) {
        T s = M[k * 6 + 0] * t[0];
        for (int j = 1; j < 6; ++j) s = s + M[k * 6 + j] * t[j];
        d[k] = s;
    }
}

template <typename T>
__device__ __forceinline__ long long quant(T x)
{
    return llround((double)x * kScale);
}

template <typename T>
__global__ void k_scatter(int nc, const T *__restrict__ Ja, const T *__restrict__ Jb, const T *__restrict__ Minv,
                          const int *__restrict__ pa, const int *__restrict__ pb, const T *__restrict__ lam,
                          long long *__restrict__ acc)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nc) return;
    const T l[3] = {lam[3 * (size_t)c], lam[3 * (size_t)c + 1], lam[3 * (size_t)c + 2]};
    for (int side = 0; side < 2; ++side) {
        const int b = side == 0 ? pa[c] : pb[c];
        if (b < 0) continue;
        T d[6];
        minv_jt((side == 0 ? Ja : Jb) + 18 * (size_t)c, Minv + 36 * (size_t)b, l, d);
        for (int k = 0; k < 6; ++k)
            atomicAdd(reinterpret_cast<unsigned long long *>(acc + 6 * (size_t)b + k), (unsigned long long)quant(d[k]));
    }
}

template <typename T>
__global__ void k_apply(int nb, const T *__restrict__ vfree, const long long *__restrict__ acc, T *__restrict__ v)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 6 * nb) return;
    v[i] = vfree[i] + (T)((double)acc[i] / kScale);
}

// u = bias + Ja v_a + Jb v_b (v read through L2: other CTAs of the sweep write it)
template <typename T>
__device__ __forceinline__ void contact_u(int c, const T *__restrict__ Ja, const T *__restrict__ Jb, int a, int b,
                                          const T *__restrict__ bias, const T *v, T u[3])
{
    T va[6], vb[6];
    if (a >= 0)
        for (int j = 0; j < 6; ++j) va[j] = __ldcg(v + 6 * (size_t)a + j);
    if (b >= 0)
        for (int j = 0; j < 6; ++j) vb[j] = __ldcg(v + 6 * (size_t)b + j);
    for (int i = 0; i < 3; ++i) {
        T ui = bias[3 * (size_t)c + i];
        if (a >= 0) {
            const T *J = Ja + 18 * (size_t)c + 6 * i;
            T s = J[0] * va[0];
            for (int j = 1; j < 6; ++j) s = s + J[j] * va[j];
            ui = ui + s;
        }
        if (b >= 0) {
            const T *J = Jb + 18 * (size_t)c + 6 * i;
            T s = J[0] * vb[0];
            for (int j = 1; j < 6; ++j) s = s + J[j] * vb[j];
            ui = ui + s;
        }
        u[i] = ui;
    }
}

struct Soft {
    int on, use_bias;
    double p[5];  // bias_rate, mass_scale, impulse_scale, inv_h, contact_speed
};

// the argument of the projection (k_sweep's two branches)
template <typename T>
__device__ __forceinline__ void contact_z(const T u[3], const T lo[3], T mu, T rho, int desaxce, const Soft &sf, T sp,
                                          T z[3])
{
    if (sf.on) {
        T vb = T(0), ms = T(1), isc = T(0);
        if (sp > T(0)) {
            vb = sp * (T)sf.p[3];
        } else if (sf.use_bias) {
            const T t = (T)sf.p[1] * (T)sf.p[0] * sp;
            vb = t > -(T)sf.p[4] ? t : -(T)sf.p[4];
            ms = (T)sf.p[1];
            isc = (T)sf.p[2];
        }
        T rn = u[0];
        if (desaxce) rn = rn + mu * rsq(u[1] * u[1] + u[2] * u[2]);
        z[0] = (T(1) - isc) * lo[0] - rho * (ms * rn + vb);
        z[1] = lo[1] - rho * u[1];
        z[2] = lo[2] - rho * u[2];
    } else {
        T s0 = u[0];
        if (desaxce) s0 = u[0] + mu * rsq(u[1] * u[1] + u[2] * u[2]);
        z[0] = lo[0] - rho * s0;
        z[1] = lo[1] - rho * u[1];
        z[2] = lo[2] - rho * u[2];
    }
}

// exact projection onto K_mu (f_proj, :382-397)
template <typename T>
__device__ __forceinline__ void proj(const T z[3], T mu, T out[3])
{
    const T zn = z[0], zt = rsq(z[1] * z[1] + z[2] * z[2]);
    if (zt <= mu * zn) {
        out[0] = z[0];
        out[1] = z[1];
        out[2] = z[2];
    } else if (mu * zt <= -zn) {
        out[0] = out[1] = out[2] = T(0);
    } else {
        const T s = (zn + mu * zt) / (T(1) + mu * mu);
        const T f = mu * s / zt;
        out[0] = s;
        out[1] = f * z[1];
        out[2] = f * z[2];
    }
}

enum Kind { kBlock = 0, kCluster = 1, kGrid = 2 };

// What a phase costs is its barrier (0.1 us in one CTA, 0.5 in a cluster, 1.3 over every SM), the
// contact's chain (~1.3 us) and how many contacts a group has to take one after the other, so the
// form is the smallest launch that has a group for each contact of an average colour.  Measured
// on a B200 (us per colour phase, float64; one CTA / cluster of 16 / grid of 148): 12 contacts a
// colour 1.5 / 2.0 / 3.2, 22 2.4 / 2.0 / 3.2, 85 7.3 / 2.1 / 3.2, 300 24 / 2.3 / 3.3, 350 - / 2.5 / 3.4,
// 380 - / 3.6 / 3.4, 400 - / 4.6 / 3.4, 5 000 - / 31 / 4.4; float32 (640 groups in the cluster), 600 - /
// 2.7 / 2.9, 635 - / 3.6 / 2.9, 700 - / 4.4 / 2.9.  The wider of the colours are over the average, so
// the line is a thirty-second below the cluster's groups.
struct Form {
    int asked;            // 0 auto: the launched kernels choose by the colouring; else the form is given
    int narrow;           // contacts a colour, on average, below which one CTA runs the sweeps ...
    int narrow_contacts;  // ... of at most this many contacts
    int wide;             // contacts a colour, on average, from which the grid runs
    int many;             // from which the form's kernel with more groups a CTA runs (0: it has none)
    __device__ __forceinline__ bool here(int kind, bool of_many, int nc, int ncol) const
    {
        const long long n = nc;
        if (asked == 0) {
            const bool one = nc <= narrow_contacts && n < (long long)narrow * ncol;
            if (kind != (one ? kBlock : ncol > 0 && n >= (long long)wide * ncol ? kGrid : kCluster)) return false;
        }
        return of_many == (many > 0 && n >= (long long)many * ncol);
    }
};

template <typename T>
struct SweepArgs {
    Form form;
    int smem_bodies;  // one CTA: the bodies whose state it holds in shared memory (0: none)
    int nc;
    const T *Ja, *Jb, *Minv, *vfree, *mu, *bias, *sep, *rho;
    const int *pa, *pb, *order, *cstart, *ccount, *dyn;
    T *lam, *v;
    long long *acc;
    double *trace;  // null, or (iters, nc, kTraceWords): what each contact's update of each sweep started from
    int *stats;
    unsigned int *bar;
    long long timeout_ns;
    int iters, desaxce;
    Soft soft;
};


// A recorded update, written by the sweeps: the contact's impulse before it [0, 3), the
// velocities of its bodies a, b [3, 9), [9, 15) (zero where there is no body), the impulse
// change dl [18, 21), the projection's argument z [33, 36) and the contact velocity u [36, 39);
// the reverse sweep adds the update's adjoints: ub [15, 18) and the adjoints of both bodies'
// velocities after the update [21, 27), [27, 33).
constexpr int kTraceWords = 39;

// The barrier between colours, split into an arrive and a wait.  The grid form (a cooperative
// launch, every CTA co-resident) is the arrival-counter barrier of b2c_barrier.cuh over a.bar[0]
// (cleared by the host before the launch); `epoch` counts the grid barriers of this launch.  Its
// wait is bounded by a.timeout_ns, after which it sets kErrBarrier and every CTA leaves the sweep.
template <int kKind, typename A>
__device__ __forceinline__ void phase_arrive(const A &a, unsigned int &epoch)
{
    if (kKind == kCluster) {
        cluster_arrive();
    } else if (kKind == kGrid) {
        ++epoch;
        grid_arrive(a.bar);
    }
}
template <int kKind, typename A>
__device__ __forceinline__ bool phase_wait(const A &a, unsigned int epoch)
{
    if (kKind == kBlock) {
        __syncthreads();
        return true;
    }
    if (kKind == kCluster) {
        asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory");
        return true;
    }
    return grid_wait(a.bar, epoch, a.timeout_ns, a.stats + kError, kErrBarrier);
}

// a / b correctly rounded from y = RN(1 / b), without a division: each correction q + (a - q b) y
// takes the quotient's error to its square, the first to within an ulp and the second to the
// rounded quotient (Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", 1990: with y the rounded reciprocal and q within an ulp, RN(q + r y) = RN(a / b)).
// The caller keeps a and b away from the ends of the exponent range, where the remainder would
// not be exact.
__device__ __forceinline__ double quotient(double a, double b, double y)
{
    double q = a * y;
    q = fma(fma(-q, b, a), y, q);
    return fma(fma(-q, b, a), y, q);
}
__device__ __forceinline__ float quotient(float a, float b, float y)
{
    float q = a * y;
    q = fmaf(fmaf(-q, b, a), y, q);
    return fmaf(fmaf(-q, b, a), y, q);
}
__device__ __forceinline__ bool in_range(double x) { return fabs(x) > 1e-140 && fabs(x) < 1e140; }
__device__ __forceinline__ bool in_range(float x) { return fabsf(x) > 1e-12f && fabsf(x) < 1e12f; }
// an int64 sum over the fixed-point scale (a whole number: no exponent near the ends)
__device__ __forceinline__ double unscale(long long s) { return quotient((double)s, kScale, 1.0 / kScale); }

// One contact update of k_sweep (:485-568): u = bias + Ja v_a + Jb v_b (contact_u's sums), the
// projection of contact_z's argument, then for each dynamic body the swap of the contact's
// rounded contribution Minv J^T lambda in the int64 accumulator (f_swap, :425-438) and the
// body's velocity rebuilt from it (k_apply_c, :583-599).  It runs on a group of kGroup = 16
// lanes, so that one contact's dependent chain is short: lanes 0..5 form the six 6-term sums of
// u (row i = lane % 3 of side lane / 3); every lane then has u, z and the projection (the same
// bits in each); lanes 0..11 each own one velocity component k of one side: entry k of J^T
// lambda, row k of Minv times the side's six entries, the accumulator swap and the velocity
// rebuild.  Every sum runs in the same order as a one-thread update would.
//
// What bounds a colour phase is that chain behind the barrier, so only what depends on the
// other contacts of the sweep is in it -- the bodies' velocities and accumulators, both loaded
// at once -- and everything else (SweepPre: the indices, the blocks' and Minv's rows, the
// impulse the contact holds and its rounded contribution, the reciprocal of 1 + mu^2) is loaded
// before the barrier's wait.  The two square roots do not wait for each other and
// run as one instruction sequence on alternate lanes; the two divisions by known numbers
// (1 + mu^2, the fixed-point scale) are multiply-adds (quotient()).  Of the 2.7 us of a phase of a
// 16-CTA cluster (240 contacts) the barrier and the stores it waits for take 0.9, the chain 1.3 and
// the fixed words, when they are loaded inside the phase, 0.5.
//
// Measured on a B200 against every load behind the barrier, true divisions and one CTA up to
// 16 384 contacts: us per colour phase of 300 contacts 18.6 -> 2.3 (float32 15.1 -> 2.1), of 5 000
// 5.9 -> 4.4; 16 sweeps of 1, 4, 24 and 48 stacks of boxes (488, 1 946, 11 668 and 23 250 contacts)
// 1 598 -> 990, 3 166 -> 1 530, 13 040 -> 1 945 and 4 219 -> 2 670 us.  Staging the blocks in shared
// memory with cp.async (1.16 -> 1.27 ms for 60 float32 sweeps of 600 bodies) and the bodies' state
// in the cluster's distributed shared memory (2.70 -> 2.96 us a phase) were both slower.
constexpr int kGroup = 16;
constexpr unsigned kWarp = 0xffffffffu;

template <typename T>
__device__ __forceinline__ T group_get(T x, int src)
{
    return __shfl_sync(kWarp, x, src, kGroup);
}

// One contact's task: the contact, its bodies, and bits: 1, 2 the body is dynamic, 4 the group
// has this contact (a group beyond its colour goes along with its warp on the colour's first).
struct Task {
    int c, pa, pb, bits;
};

// The tasks of a CTA's groups, every colour's first round, in shared memory: a contact keeps its
// group in every sweep, so the three dependent loads that lead to its words (order, bodies,
// dynamic flags) are paid once a launch and not behind every barrier, whose acquire empties L1.
// Colours beyond the table, and later rounds of a colour wider than the launch, take the loads.
constexpr int kTableBytes = 96 * 1024;
extern __shared__ int4 s_tasks[];

struct TaskTable {
    const int *pa, *pb, *order, *dyn;
    const int *start, *count;  // shared copies of the colour offsets and sizes
    int per, colors;           // groups of the CTA; colours in the table

    __device__ __forceinline__ Task load(int ci, int t) const
    {
        const bool on = t < count[ci];
        Task k;
        k.c = order[start[ci] + (on ? t : 0)];
        k.pa = pa[k.c];
        k.pb = pb[k.c];
        k.bits = (k.pa >= 0 && dyn[k.pa] ? 1 : 0) | (k.pb >= 0 && dyn[k.pb] ? 2 : 0) | (on ? 4 : 0);
        return k;
    }
    // task t of colour ci, the CTA's group lg; first: of the group's first round
    __device__ __forceinline__ Task get(int ci, int t, int lg, bool first) const
    {
        if (!first || ci >= colors) return load(ci, t);
        const int4 w = s_tasks[ci * per + lg];
        return Task{w.x, w.y, w.z, w.w};
    }
};

// every thread of the CTA calls it
template <typename A>
__device__ __forceinline__ TaskTable task_table(const A &a, int ncol, int *s_start, int *s_count)
{
    for (int c = threadIdx.x; c < ncol; c += blockDim.x) {
        s_start[c] = a.cstart[c];
        s_count[c] = a.ccount[c];
    }
    __syncthreads();
    TaskTable tt{a.pa, a.pb, a.order, a.dyn, s_start, s_count, (int)blockDim.x / 16, 0};
    tt.colors = min(ncol, kTableBytes / (16 * tt.per));
    for (int i = threadIdx.x; i < tt.colors * tt.per; i += blockDim.x) {
        const int ci = i / tt.per, lg = i - ci * tt.per;
        const Task k = tt.load(ci, lg * (int)gridDim.x + (int)blockIdx.x);
        s_tasks[i] = make_int4(k.c, k.pa, k.pb, k.bits);
    }
    __syncthreads();
    return tt;
}

// what a contact's update needs besides its bodies' velocities and accumulators
template <typename T>
struct SweepPre {
    Task k;
    bool dyn;          // this lane's component belongs to a dynamic body
    T Jr[6];           // lanes 0..5: row lane % 3 of side lane / 3
    T Jc[3], Mr[6];    // lanes 0..11: column k of the side's block, row k of its body's Minv
    T lo[3], bias, mu, rho, vf, rden;  // bias: lanes 0..2; rden = 1 / (1 + mu^2)
    long long qold;    // the rounded contribution of `lo` to this lane's component
};

// row k of Minv (J^T l) on lane (side, k), minv_jt's order: every lane forms its entry of J^T l
// and reads its side's six
template <typename T>
__device__ __forceinline__ T component(const SweepPre<T> &q, const T l3[3], int l)
{
    T t = q.Jc[0] * l3[0];
    t = t + q.Jc[1] * l3[1];
    t = t + q.Jc[2] * l3[2];
    const int base = l < 6 ? 0 : 6;
    T d = q.Mr[0] * group_get(t, base);
#pragma unroll
    for (int j = 1; j < 6; ++j) d = d + q.Mr[j] * group_get(t, base + j);
    return d;
}

// the loads of a contact's words ...
template <typename T>
__device__ __forceinline__ void sweep_load(const SweepArgs<T> &a, const Task &task, int l, SweepPre<T> &q)
{
    q.k = task;
    const int c = task.c;
    const int side = l / 6, k = l - 6 * side, b = side == 0 ? task.pa : task.pb;
#pragma unroll
    for (int j = 0; j < 6; ++j) q.Jr[j] = T(0);
    if (l < 6) {
        const T *J = (l < 3 ? a.Ja : a.Jb) + 18 * (size_t)c + 6 * (l % 3);
#pragma unroll
        for (int j = 0; j < 6; ++j) q.Jr[j] = J[j];
    }
    q.dyn = side < 2 && (task.bits & (side == 0 ? 1 : 2)) != 0;
    q.vf = T(0);
#pragma unroll
    for (int j = 0; j < 3; ++j) q.Jc[j] = T(0);
#pragma unroll
    for (int j = 0; j < 6; ++j) q.Mr[j] = T(0);
    if (q.dyn) {
        const T *J = (side == 0 ? a.Ja : a.Jb) + 18 * (size_t)c + k, *M = a.Minv + 36 * (size_t)b + 6 * k;
#pragma unroll
        for (int j = 0; j < 3; ++j) q.Jc[j] = J[6 * j];
#pragma unroll
        for (int j = 0; j < 6; ++j) q.Mr[j] = M[j];
        q.vf = a.vfree[6 * (size_t)b + k];
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) q.lo[j] = a.lam[3 * (size_t)c + j];
    q.bias = l < 3 ? a.bias[3 * (size_t)c + l] : T(0);
    q.mu = a.mu[c];
    q.rho = a.rho[c];
}
// ... and what is computed from them alone, while the other CTAs arrive
template <typename T>
__device__ __forceinline__ void sweep_finish(int l, SweepPre<T> &q)
{
    q.rden = T(1) / (T(1) + q.mu * q.mu);
    q.qold = quant(component(q, q.lo, l));
}

// Body velocities and accumulators: through L2 where other SMs write them; where one CTA runs
// the whole sweep, ordinary accesses, to the CTA's own shared copy when it fits (State).
template <int kKind, typename U>
__device__ __forceinline__ U shared_load(const U *p)
{
    return kKind == kBlock ? *p : __ldcg(p);
}
template <int kKind, typename U>
__device__ __forceinline__ void shared_store(U *p, U x)
{
    if (kKind == kBlock) *p = x;
    else __stcg(p, x);
}

template <typename T>
struct State {
    T *v;
    long long *acc;
};

template <typename T, int kKind>
__device__ __forceinline__ void sweep_contact_group(const SweepArgs<T> &a, const State<T> &S, const SweepPre<T> &q,
                                                    int it, int l)
{
    const int side = l / 6, k = l - 6 * side, pa = q.k.pa, pb = q.k.pb, bk = side == 0 ? pa : pb;
    // what the other contacts of the sweep have changed: the velocities and the accumulators
    T vs[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
    const int bu = l < 3 ? pa : pb;
    if (l < 6 && bu >= 0) {
#pragma unroll
        for (int j = 0; j < 6; ++j) vs[j] = shared_load<kKind>(S.v + 6 * (size_t)bu + j);
    }
    long long sacc = 0;
    if (q.dyn) sacc = shared_load<kKind>(S.acc + 6 * (size_t)bk + k);
    T part = q.Jr[0] * vs[0];
#pragma unroll
    for (int j = 1; j < 6; ++j) part = part + q.Jr[j] * vs[j];
    // lane i < 3: u_i, then every lane the three
    const T sb = group_get(part, 3 + l % 3);
    T ui = q.bias;
    if (pa >= 0) ui = ui + part;
    if (pb >= 0) ui = ui + sb;
    const T u[3] = {group_get(ui, 0), group_get(ui, 1), group_get(ui, 2)};
    // contact_z and proj: the tangential part of z does not depend on the slip speed, so the odd
    // lanes take |z_t|, the even ones |u_t|
    T z[3], zn[3];
    z[1] = q.lo[1] - q.rho * u[1];
    z[2] = q.lo[2] - q.rho * u[2];
    const bool odd = (l & 1) != 0;
    const T x1 = odd ? z[1] : u[1], x2 = odd ? z[2] : u[2];
    const T root = rsq(x1 * x1 + x2 * x2), other = __shfl_xor_sync(kWarp, root, 1, kGroup);
    const T ut = odd ? other : root, zt = odd ? root : other;
    if (a.soft.on) {
        const T sep = a.sep ? a.sep[q.k.c] : T(0);
        T vb = T(0), ms = T(1), isc = T(0);
        if (sep > T(0)) {
            vb = sep * (T)a.soft.p[3];
        } else if (a.soft.use_bias) {
            const T t = (T)a.soft.p[1] * (T)a.soft.p[0] * sep;
            vb = t > -(T)a.soft.p[4] ? t : -(T)a.soft.p[4];
            ms = (T)a.soft.p[1];
            isc = (T)a.soft.p[2];
        }
        T rn = u[0];
        if (a.desaxce) rn = rn + q.mu * ut;
        z[0] = (T(1) - isc) * q.lo[0] - q.rho * (ms * rn + vb);
    } else {
        T s0 = u[0];
        if (a.desaxce) s0 = u[0] + q.mu * ut;
        z[0] = q.lo[0] - q.rho * s0;
    }
    if (zt <= q.mu * z[0]) {
        zn[0] = z[0];
        zn[1] = z[1];
        zn[2] = z[2];
    } else if (q.mu * zt <= -z[0]) {
        zn[0] = zn[1] = zn[2] = T(0);
    } else {
        const T num = z[0] + q.mu * zt, den = T(1) + q.mu * q.mu;
        const T s = in_range(num) && in_range(den) ? quotient(num, den, q.rden) : num / den;
        const T f = q.mu * s / zt;
        zn[0] = s;
        zn[1] = f * z[1];
        zn[2] = f * z[2];
    }
    const T d = component(q, zn, l);
    if (!(q.k.bits & 4)) return;
    const size_t c = (size_t)q.k.c;
    if (q.dyn) {
        sacc = sacc + (quant(d) - q.qold);
        shared_store<kKind>(S.acc + 6 * (size_t)bk + k, sacc);
        shared_store<kKind>(S.v + 6 * (size_t)bk + k, q.vf + (T)unscale(sacc));
    }
    if (l < 3) a.lam[3 * c + l] = l == 0 ? zn[0] : l == 1 ? zn[1] : zn[2];
    if (a.trace) {
        double *t = a.trace + kTraceWords * ((size_t)it * a.nc + c);
        if (l == 0)
            for (int i = 0; i < 3; ++i) {
                t[i] = (double)q.lo[i];
                t[18 + i] = (double)zn[i] - (double)q.lo[i];
                t[33 + i] = (double)z[i];
                t[36 + i] = (double)u[i];
            }
        if (l == 0 || l == 3)
            for (int i = 0; i < 6; ++i) t[(l == 0 ? 3 : 9) + i] = (double)vs[i];
    }
}

// A group loads its next task's fixed words while it computes the one before it (kAhead), which
// takes a second SweepPre of registers and so a smaller CTA.  The grid instead has more groups, one
// for each contact of the widest colours, and loads between its barrier's arrive and wait, which
// are apart as long as the loads take.
template <int kKind>
constexpr bool kAhead = kKind != kGrid;
template <typename T, int kKind>
constexpr int sweep_threads()
{
    return kAhead<kKind> ? (sizeof(T) == 4 ? 640 : 384) : sizeof(T) == 4 ? 1024 : 640;
}

template <typename T, int kKind>
__global__ void __launch_bounds__(sweep_threads<T, kKind>()) k_sweeps(SweepArgs<T> a)
{
    const int ncol = a.stats[kNColors];
    if (ncol == 0 || !a.form.here(kKind, false, a.nc, ncol)) return;  // uniform over the launch
    __shared__ int s_start[kMaxColors], s_count[kMaxColors];
    const TaskTable tt = task_table(a, ncol, s_start, s_count);
    State<T> S{a.v, a.acc};
    if (kKind == kBlock && a.smem_bodies) {  // behind the task table
        S.acc = reinterpret_cast<long long *>(s_tasks + tt.colors * tt.per);
        S.v = reinterpret_cast<T *>(S.acc + 6 * (size_t)a.smem_bodies);
        for (int i = threadIdx.x; i < 6 * a.smem_bodies; i += blockDim.x) {
            S.acc[i] = a.acc[i];
            S.v[i] = a.v[i];
        }
        __syncthreads();
    }
    // Task slot: one group of kGroup lanes per contact; group g = (group in CTA) x CTAs + CTA,
    // so consecutive contacts of a colour land on different CTAs and a colour narrower than
    // the launch is spread over every SM of it.  A contact keeps its group in every sweep (so
    // its impulse is written and read by the same lanes).
    const int nb = gridDim.x, groups = nb * tt.per;
    const int lg = (int)threadIdx.x / kGroup, g = lg * nb + (int)blockIdx.x, l = (int)threadIdx.x % kGroup;
    const int g0 = (lg & ~1) * nb + (int)blockIdx.x;  // the warp's first group
    // One loop over the group's tasks, phase after phase.  A task's fixed words are loaded while the
    // group's task before it is computed, so that their trip to L2 is on no phase's path, and
    // worked up while the other CTAs arrive at the barrier.  A contact is always its group's own,
    // so the impulse among them is final, unless the task before is the same contact (one colour).
    SweepPre<T> pre = {}, next = {};
    unsigned int epoch = 0;
    int it = 0, ci = 0, cnt = s_count[0], t = g, t0 = g0;
    bool have = t0 < cnt;
    if (have) {
        sweep_load(a, tt.get(0, t, lg, true), l, pre);
        sweep_finish(l, pre);
    }
    for (;;) {
        const bool now = have;
        const int at = it;
        if (!kAhead<kKind> && now) sweep_contact_group<T, kKind>(a, S, pre, at, l);
        t += groups;
        t0 += groups;
        const bool more = t0 < cnt;
        if (!more) {
            t = g;
            t0 = g0;
            if (++ci == ncol) {
                ci = 0;
                ++it;
            }
            cnt = s_count[ci];
        }
        have = it < a.iters && t0 < cnt;
        if (kAhead<kKind>) {
            if (have) sweep_load(a, tt.get(ci, t, lg, !more), l, next);
            if (now) sweep_contact_group<T, kKind>(a, S, pre, at, l);
        }
        __syncwarp();
        if (!more) phase_arrive<kKind>(a, epoch);
        if (have) {
            if (!kAhead<kKind>) {
                sweep_load(a, tt.get(ci, t, lg, !more), l, pre);
            } else {
                if (next.k.c == pre.k.c) {
#pragma unroll
                    for (int j = 0; j < 3; ++j) next.lo[j] = a.lam[3 * (size_t)next.k.c + j];
                }
                pre = next;
            }
            sweep_finish(l, pre);
        }
        if (!more) {
            if (!phase_wait<kKind>(a, epoch)) return;
            if (it == a.iters) break;
        }
    }
    if (kKind == kBlock && a.smem_bodies)
        for (int i = threadIdx.x; i < 6 * a.smem_bodies; i += blockDim.x) {
            a.acc[i] = S.acc[i];
            a.v[i] = S.v[i];
        }
}

// The same update for a launch whose CTAs take several contacts each in every phase: there the time
// is how many groups of a CTA are in flight, not one contact's chain, so everything is loaded where
// it is used, which needs 64 registers a thread and lets a CTA have 64 groups (k_sweeps: 24 to 40,
// float32 grid 64).  From kManyRounds rounds on, on average, this one runs: a launch of few CTAs that
// was asked for, and the grid on scenes of 100 000 contacts.  Measured on a B200 (12 sweeps of 8
// colours, us; k_sweeps / this one): one CTA, float64, 30 contacts a colour 267 / 298, 75 628 / 554,
// 200 1 635 / 1 250, 1 250 10 497 / 7 058; a cluster of 8, 500 707 / 726, 1 250 1 629 / 1 312; a grid of
// 16, 1 250 943 / 1 005, 2 500 1 529 / 1 359; a grid of 148, 25 000 2 047 / 1 524; float32, one CTA, 75
// 457 / 468, 200 1 054 / 905, a cluster of 2, 200 679 / 734, 500 1 473 / 1 430.
template <typename T>
__device__ __forceinline__ T group_get(T x, int src, unsigned mask)
{
    return __shfl_sync(mask, x, src, kGroup);
}

template <typename T, int kKind>
__device__ __forceinline__ void sweep_contact_many(const SweepArgs<T> &a, int c, int it, int l, unsigned mask)
{
    const int pa = a.pa[c], pb = a.pb[c];
    const T lo[3] = {a.lam[3 * (size_t)c], a.lam[3 * (size_t)c + 1], a.lam[3 * (size_t)c + 2]};
    // the six partial sums of u
    T part = T(0), vs[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
    if (l < 6) {
        const int i = l % 3, side = l / 3, b = side == 0 ? pa : pb;
        if (b >= 0) {
            for (int j = 0; j < 6; ++j) vs[j] = shared_load<kKind>(a.v + 6 * (size_t)b + j);
            const T *J = (side == 0 ? a.Ja : a.Jb) + 18 * (size_t)c + 6 * i;
            T sacc = J[0] * vs[0];
            for (int j = 1; j < 6; ++j) sacc = sacc + J[j] * vs[j];
            part = sacc;
        }
    }
    T u[3];
    for (int i = 0; i < 3; ++i) {
        const T sa = group_get(part, i, mask), sb = group_get(part, 3 + i, mask);
        T ui = a.bias[3 * (size_t)c + i];
        if (pa >= 0) ui = ui + sa;
        if (pb >= 0) ui = ui + sb;
        u[i] = ui;
    }
    T z[3], zn[3];
    contact_z(u, lo, a.mu[c], a.rho[c], a.desaxce, a.soft, a.sep ? a.sep[c] : T(0), z);
    proj(z, a.mu[c], zn);
    if (a.trace) {
        double *t = a.trace + kTraceWords * ((size_t)it * a.nc + c);
        if (l == 0)
            for (int k = 0; k < 3; ++k) {
                t[k] = (double)lo[k];
                t[18 + k] = (double)zn[k] - (double)lo[k];
                t[33 + k] = (double)z[k];
                t[36 + k] = (double)u[k];
            }
        if (l == 0 || l == 3)
            for (int k = 0; k < 6; ++k) t[(l == 0 ? 3 : 9) + k] = (double)vs[k];
    }
    if (l < 3) a.lam[3 * (size_t)c + l] = l == 0 ? zn[0] : l == 1 ? zn[1] : zn[2];
    if (l >= 12) return;
    const int side = l / 6, k = l % 6, b = side == 0 ? pa : pb;
    if (b < 0 || !a.dyn[b]) return;
    const T *J = (side == 0 ? a.Ja : a.Jb) + 18 * (size_t)c;
    const T *M = a.Minv + 36 * (size_t)b + 6 * k;
    // row k of Minv (J^T l), minv_jt's order, for the new and the old impulse
    T dn = T(0), dold = T(0);
    for (int j = 0; j < 6; ++j) {
        T tn = J[j] * zn[0];
        tn = tn + J[6 + j] * zn[1];
        tn = tn + J[12 + j] * zn[2];
        T to = J[j] * lo[0];
        to = to + J[6 + j] * lo[1];
        to = to + J[12 + j] * lo[2];
        if (j == 0) {
            dn = M[0] * tn;
            dold = M[0] * to;
        } else {
            dn = dn + M[j] * tn;
            dold = dold + M[j] * to;
        }
    }
    long long *p = a.acc + 6 * (size_t)b + k;
    const long long sacc = shared_load<kKind>(p) + (quant(dn) - quant(dold));
    shared_store<kKind>(p, sacc);
    shared_store<kKind>(a.v + 6 * (size_t)b + k, a.vfree[6 * (size_t)b + k] + (T)unscale(sacc));
}

constexpr int kManyThreads = 1024;
// rounds, in halves, from which k_sweeps_many runs (0: never)
template <typename T, int kKind>
constexpr int kManyRounds = sizeof(T) == 8 ? 5 : kKind == kGrid ? 0 : 9;

template <typename T, int kKind>
__global__ void __launch_bounds__(kManyThreads) k_sweeps_many(SweepArgs<T> a)
{
    const int ncol = a.stats[kNColors];
    if (ncol == 0 || !a.form.here(kKind, true, a.nc, ncol)) return;  // uniform over the launch
    const int nb = gridDim.x, groups = nb * (kManyThreads / kGroup);
    const int g = ((int)threadIdx.x / kGroup) * nb + (int)blockIdx.x, l = (int)threadIdx.x % kGroup;
    const unsigned mask = 0xFFFFu << (((int)threadIdx.x & 31) & ~(kGroup - 1));
    unsigned int epoch = 0;
    for (int it = 0; it < a.iters; ++it)
        for (int ci = 0; ci < ncol; ++ci) {
            const int s0 = a.cstart[ci], cnt = a.ccount[ci];
            for (int t = g; t < cnt; t += groups) sweep_contact_many<T, kKind>(a, a.order[s0 + t], it, l, mask);
            // in a cluster a warp's writes go out while others still compute: every warp's own release
            if (kKind == kCluster) asm volatile("barrier.cluster.arrive.release;\n" ::: "memory");
            else phase_arrive<kKind>(a, epoch);
            if (!phase_wait<kKind>(a, epoch)) return;
        }
}

template <typename T>
__global__ void k_resid(SweepArgs<T> a, T *__restrict__ res, T *__restrict__ uout,
                        unsigned long long *__restrict__ res_max)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= a.nc) return;
    T u[3], z[3], zn[3];
    const T lo[3] = {a.lam[3 * (size_t)c], a.lam[3 * (size_t)c + 1], a.lam[3 * (size_t)c + 2]};
    contact_u(c, a.Ja, a.Jb, a.pa[c], a.pb[c], a.bias, a.v, u);
    contact_z(u, lo, a.mu[c], a.rho[c], a.desaxce, a.soft, a.sep ? a.sep[c] : T(0), z);
    proj(z, a.mu[c], zn);
    T m = T(0);
    for (int i = 0; i < 3; ++i) {
        const T d = rab(lo[i] - zn[i]);
        if (d > m) m = d;
    }
    res[c] = m;
    uout[3 * (size_t)c] = u[0];
    uout[3 * (size_t)c + 1] = u[1];
    uout[3 * (size_t)c + 2] = u[2];
    // non-negative reals order like their bit patterns
    atomicMax(res_max, (unsigned long long)__double_as_longlong((double)m));
}

// ---------------------------------------------------------------------------------------------
// host drivers
// ---------------------------------------------------------------------------------------------
template <typename T>
SweepArgs<T> sweep_args(const b2c_ncp_scene *sc, b2c_ncp_state *st, const b2c_ncp_params *p, int iters)
{
    SweepArgs<T> a;
    a.nc = sc->n_c;
    a.Ja = (const T *)sc->Ja;
    a.Jb = (const T *)sc->Jb;
    a.Minv = (const T *)sc->Minv;
    a.vfree = (const T *)sc->v_free;
    a.mu = (const T *)sc->mu;
    a.bias = (const T *)sc->bias;
    a.sep = (const T *)sc->sep;
    a.rho = (const T *)st->rho;
    a.pa = sc->pa;
    a.pb = sc->pb;
    a.order = st->order;
    a.cstart = st->cstart;
    a.ccount = st->ccount;
    a.dyn = st->dyn;
    a.lam = (T *)st->lam;
    a.v = (T *)st->v;
    a.acc = reinterpret_cast<long long *>(st->acc);
    a.trace = nullptr;
    a.stats = st->stats;
    a.bar = st->barrier;
    a.timeout_ns = (p && p->barrier_timeout_ns > 0) ? p->barrier_timeout_ns : 1000000000LL;  // default 1 s
    a.iters = iters;
    a.desaxce = p ? p->desaxce : 1;
    a.soft.on = p ? p->soft : 0;
    a.soft.use_bias = p ? p->use_bias : 1;
    for (int k = 0; k < 5; ++k) a.soft.p[k] = p ? p->softp[k] : 0.0;
    return a;
}

template <typename T>
int setup(const b2c_ncp_scene *sc, b2c_ncp_state *st, int warm, cudaStream_t s)
{
    const int nc = sc->n_c, nb = sc->n_b;
    if (nc > 0)
        k_rho<T><<<blocks_for(nc), kThreads, 0, s>>>(nc, (const T *)sc->Ja, (const T *)sc->Jb, (const T *)sc->Minv,
                                                     sc->pa, sc->pb, (T *)st->rho);
    if (nb > 0) k_dyn<T><<<blocks_for(nb), kThreads, 0, s>>>(nb, (const T *)sc->Minv, st->dyn);
    cudaMemsetAsync(st->acc, 0, sizeof(int64_t) * 6 * (size_t)nb, s);
    if (!warm) cudaMemsetAsync(st->lam, 0, sizeof(T) * 3 * (size_t)nc, s);
    else if (nc > 0)
        k_scatter<T><<<blocks_for(nc), kThreads, 0, s>>>(nc, (const T *)sc->Ja, (const T *)sc->Jb,
                                                         (const T *)sc->Minv, sc->pa, sc->pb, (const T *)st->lam,
                                                         reinterpret_cast<long long *>(st->acc));
    if (nb > 0)
        k_apply<T><<<blocks_for(6 * (long long)nb), kThreads, 0, s>>>(
            nb, (const T *)sc->v_free, reinterpret_cast<const long long *>(st->acc), (T *)st->v);
    return check_launch("ncp_setup");
}

// Colouring behind the cache (Jones-Plassmann over the contacts): a contact takes colour r when it
// holds the smallest key at each of its dynamic bodies among the contacts still uncoloured.  A
// round is two phases: every uncoloured contact claims its bodies (atomicMin of its key), then
// each looks whether it holds them all.  A contact that does takes its bodies' claims back at
// once: whoever still reads one sees a key or a cleared claim, neither his own, and has lost
// either way; and a claim left standing belongs to a contact that is still uncoloured, so it is
// a lower bound that the next round's claims complete.  So nothing is cleared between rounds.
// A thread keeps its contacts' keys and bodies in registers (kColorHold of them; more are read
// again each round), so a round is the two barriers and one trip to the claims each, and that is
// what bounds it: ~60 rounds for a stack of boxes, whatever the number of contacts.  Which
// launch runs it is the price of its barrier against the contacts a thread walks: one CTA up to
// two contacts a thread, a cluster up to the same, above it every SM.  Measured on a B200 (float64,
// us; one CTA / cluster / grid; before: one CTA up to 16 384 contacts and a grid with three
// barriers a round above) -- stacks of 1 946 contacts 112 / 125 / 175 (before 154), 3 912 176 /
// 136 / 189 (231), 11 668 611 / 151 / 205 (588), 23 250 1 355 / 207 / 220 (476), 61 941 4 270 / 321 /
// 258 (522); two-colour lattices of 10 000 contacts 36 (104), of 40 000 58 (93).
constexpr int kColorHold = 4;
constexpr int kColorGridThreads = 512;

template <int kKind>
constexpr int color_threads()
{
    return kKind == kGrid ? kColorGridThreads : kColorThreads;
}

template <typename T, int kKind>
__global__ void __launch_bounds__(color_threads<kKind>())
    k_color(int nc, int nb, const int *__restrict__ pa, const int *__restrict__ pb, const int *__restrict__ feat,
            const T *__restrict__ Minv, const int *__restrict__ dyn, b2c_ncp_state st, int use_cache, int max_colors,
            long long timeout_ns)
{
    __shared__ int s_raised, s_seen, s_scan[kMaxColors];
    const int tid = threadIdx.x, gid = blockIdx.x * blockDim.x + tid, nth = gridDim.x * blockDim.x;
    const bool lead = gid == 0;
    int *S = st.stats;
    T *cm = reinterpret_cast<T *>(st.cache_minv);
    unsigned long long *claim = reinterpret_cast<unsigned long long *>(st.claim);
    unsigned int epoch = 0;
    auto sync = [&]() -> bool {
        if (kKind == kBlock) {
            __syncthreads();
            return true;
        }
        if (kKind == kCluster) {
            cg::this_cluster().sync();
            return true;
        }
        ++epoch;
        grid_arrive(st.barrier);
        return grid_wait(st.barrier, epoch, timeout_ns, S + kError, kErrBarrier);
    };
    // a barrier that tells whether any thread of the launch raised `flag`; ok: the barrier held.
    // The count of CTAs that raised one only grows; nobody raises again before all have read it,
    // since a barrier of the next phase lies between.
    int seen = 0;
    if (kKind == kCluster) {
        if (tid == 0) s_raised = 0;
        cg::this_cluster().sync();
    }
    auto any = [&](bool flag, bool &ok) -> bool {
        const int mine = __syncthreads_or(flag);
        ok = true;
        if (kKind == kBlock) return mine != 0;
        if (kKind == kCluster) {
            int *raised = cg::this_cluster().map_shared_rank(&s_raised, 0);
            if (tid == 0 && mine) atomicAdd(raised, 1);
            cg::this_cluster().sync();
            if (tid == 0) s_seen = *(volatile int *)raised;
            __syncthreads();
        } else {
            if (tid == 0 && mine) atomicAdd(st.barrier + 8, 1u);
            ok = sync();
            if (tid == 0) s_seen = (int)__ldcg(st.barrier + 8);
            __syncthreads();
        }
        const int now = s_seen;
        const bool r = now != seen;
        seen = now;
        return r;
    };
    bool ok;
    if (use_cache && S[kCacheValid] == 1 && S[kCachedC] == nc) {
        bool mism = false;
        for (int c = gid; c < nc; c += nth)
            mism |= (pa[c] != st.cache_pa[c]) | (pb[c] != st.cache_pb[c]) | (feat[c] != st.cache_feat[c]);
        // the translational block (1/m I) and the dynamic flag (k_cache_cmp, :750-765)
        for (int i = gid; i < nb; i += nth)
            mism |= (Minv[36 * (size_t)i] != cm[4 * (size_t)i]) | (Minv[36 * (size_t)i + 7] != cm[4 * (size_t)i + 1]) |
                    (Minv[36 * (size_t)i + 14] != cm[4 * (size_t)i + 2]) | ((T)dyn[i] != cm[4 * (size_t)i + 3]);
        const bool miss = any(mism, ok);
        if (!ok) return;
        if (!miss) {
            if (lead) {
                S[kCacheHit] = 1;
                S[kHits] += 1;
            }
            // no CTA leaves while another may still read the cluster's counter
            if (kKind == kCluster) cg::this_cluster().sync();
            return;
        }
    }
    // a contact's key and its dynamic bodies (-1: none); alive: not coloured yet
    struct Held {
        unsigned long long key;
        int a, b;
    };
    auto held = [&](int c) -> Held {
        Held h;
        const int A = pa[c], B = pb[c];
        h.key = mix64(((unsigned long long)(A + 1) * (unsigned long long)(nb + 1) + (unsigned long long)(B + 1)) *
                          1048576ull +
                      (unsigned long long)(unsigned)feat[c]);
        h.a = A >= 0 && dyn[A] ? A : -1;
        h.b = B >= 0 && dyn[B] ? B : -1;
        return h;
    };
    auto put = [&](const Held &h) {
        if (h.a >= 0) atomicMin(claim + h.a, h.key);
        if (h.b >= 0) atomicMin(claim + h.b, h.key);
    };
    // does the contact hold its bodies' claims; then it gives them back
    auto wins = [&](const Held &h) -> bool {
        const bool w = (h.a < 0 || __ldcg(claim + h.a) == h.key) && (h.b < 0 || __ldcg(claim + h.b) == h.key);
        if (w) {
            if (h.a >= 0) __stcg(claim + h.a, ~0ull);
            if (h.b >= 0) __stcg(claim + h.b, ~0ull);
        }
        return w;
    };
    Held mine[kColorHold];
    unsigned alive = 0;
#pragma unroll
    for (int q = 0; q < kColorHold; ++q) {
        const int c = gid + q * nth;
        if (c < nc) {
            mine[q] = held(c);
            alive |= 1u << q;
        }
    }
    for (int c = gid + kColorHold * nth; c < nc; c += nth) st.col[c] = -1;
    for (int i = gid; i < nb; i += nth) claim[i] = ~0ull;
    if (!sync()) return;
    int r = 0;
    bool done = nc == 0;
    for (; !done && r <= nc && r < max_colors; ++r) {
#pragma unroll
        for (int q = 0; q < kColorHold; ++q)
            if (alive >> q & 1) put(mine[q]);
        for (int c = gid + kColorHold * nth; c < nc; c += nth)
            if (st.col[c] < 0) put(held(c));
        if (!sync()) return;
        bool left = false;
#pragma unroll
        for (int q = 0; q < kColorHold; ++q)
            if (alive >> q & 1) {
                if (wins(mine[q])) {
                    st.col[gid + q * nth] = r;
                    alive &= ~(1u << q);
                } else {
                    left = true;
                }
            }
        for (int c = gid + kColorHold * nth; c < nc; c += nth)
            if (st.col[c] < 0) {
                if (wins(held(c))) st.col[c] = r;
                else left = true;
            }
        done = !any(left, ok);
        if (!ok) return;
    }
    const int ncol = done ? (nc > 0 ? r : 0) : r;
    if (!done || ncol > max_colors || ncol > kMaxColors) {
        if (lead) {
            S[kError] |= done ? kErrColorOverflow : kErrColorTimeout;
            S[kNColors] = 0;
            S[kCacheValid] = 0;
            S[kRounds] = r;
        }
        if (kKind == kCluster) cg::this_cluster().sync();
        return;
    }
    // counts per colour, their exclusive scan (the first CTA), then the scatter with the counts as
    // cursors (they end where they started)
    for (int k = gid; k < ncol; k += nth) st.ccount[k] = 0;
    if (!sync()) return;
    for (int c = gid; c < nc; c += nth) atomicAdd(st.ccount + st.col[c], 1);
    if (!sync()) return;
    if (blockIdx.x == 0) {
        for (int k = tid; k < ncol; k += blockDim.x) s_scan[k] = __ldcg(st.ccount + k);
        __syncthreads();
        if (tid == 0) {
            int acc = 0;
            for (int k = 0; k < ncol; ++k) {
                const int n = s_scan[k];
                s_scan[k] = acc;
                acc += n;
            }
        }
        __syncthreads();
        for (int k = tid; k < ncol; k += blockDim.x) {
            st.cstart[k] = s_scan[k];
            st.ccount[k] = 0;
        }
    }
    if (!sync()) return;
    for (int c = gid; c < nc; c += nth) {
        const int k = st.col[c];
        st.order[__ldcg(st.cstart + k) + atomicAdd(st.ccount + k, 1)] = c;
    }
    if (use_cache) {
        for (int c = gid; c < nc; c += nth) {
            st.cache_pa[c] = pa[c];
            st.cache_pb[c] = pb[c];
            st.cache_feat[c] = feat[c];
        }
        for (int i = gid; i < nb; i += nth) {
            cm[4 * (size_t)i] = Minv[36 * (size_t)i];
            cm[4 * (size_t)i + 1] = Minv[36 * (size_t)i + 7];
            cm[4 * (size_t)i + 2] = Minv[36 * (size_t)i + 14];
            cm[4 * (size_t)i + 3] = (T)dyn[i];
        }
    }
    if (lead) {
        S[kNColors] = ncol;
        S[kRounds] = r;
        S[kCacheHit] = 0;
        S[kCacheValid] = use_cache ? 1 : 0;
        S[kCachedC] = nc;
        S[kMisses] += 1;
    }
}

constexpr size_t kStateBytes = 96 * 1024;  // the body state a single sweep CTA holds: 1000 bodies in float64

bool allow_smem(const void *fn, size_t bytes)
{
    const bool ok = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess;
    if (!ok) cudaGetLastError();
    return ok;
}

// the largest power-of-two cluster (at most kClusterMax) of a kernel that the device holds at once
int cluster_size_of(const void *fn, int threads, size_t smem)
{
    if (smem > 0) allow_smem(fn, smem);
    cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kClusterMax);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    int cs = 0;
    if (cudaOccupancyMaxPotentialClusterSize(&cs, fn, &cfg) != cudaSuccess) {
        cudaGetLastError();
        cs = 1;
    }
    int p2 = 1;
    for (int c = 1; c <= std::min(cs, kClusterMax); c *= 2) p2 = c;
    return p2;
}

// CTAs of a kernel the device holds at once (SMs x resident CTAs per SM)
int grid_blocks_of(const void *fn, int threads, size_t smem)
{
    int dev = 0, sms = 0, per = 0;
    if (smem > 0) allow_smem(fn, smem);
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, threads, smem);
    return std::min(kBarrierMaxCTAs, std::max(1, sms * per));
}

// of the sweep kernels, cached per type
template <typename T>
int cluster_size()
{
    static const int n =
        cluster_size_of((const void *)k_sweeps<T, kCluster>, sweep_threads<T, kCluster>(), kTableBytes);
    return n;
}
template <typename T>
int grid_blocks()
{
    static const int n = grid_blocks_of((const void *)k_sweeps<T, kGrid>, sweep_threads<T, kGrid>(), kTableBytes);
    return n;
}

// One CTA, a cluster or a cooperative grid of a kernel.  What a launch opts in to (its shared memory
// above 48 KB, a cluster above eight CTAs) is the device's, not the process's, so it is set for
// every launch, and to the kernel's most, so that two threads do not undo each other's.
int launch_kind(const void *fn, void **args, int kind, int ctas, int threads, size_t smem, const char *what,
                cudaStream_t s)
{
    if (smem > 0) allow_smem(fn, kTableBytes + (kind == kBlock ? kStateBytes : 0));
    if (kind == kCluster) cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    if (kind == kGrid) {
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
    } else {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = ctas;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = kind == kBlock ? 0 : 1;
    const cudaError_t e = cudaLaunchKernelExC(&cfg, fn, args);
    if (e != cudaSuccess) {
        set_error("%s: launch of %d CTAs (%s): %s", what, ctas,
                  kind == kGrid ? "cooperative" : kind == kCluster ? "cluster" : "one", cudaGetErrorString(e));
        return B2C_ECUDA;
    }
    return check_launch(what);
}

template <typename T>
int color(const b2c_ncp_scene *sc, b2c_ncp_state *st, const b2c_ncp_params *p, cudaStream_t s)
{
    const int maxc = std::min(st->max_colors, kMaxColors);
    static const int clusters = cluster_size_of((const void *)k_color<T, kCluster>, kColorThreads, 0);
    static const int grid = std::min(kSMs, grid_blocks_of((const void *)k_color<T, kGrid>, kColorGridThreads, 0));
    int kind = p->solve_blocks > 1 ? kGrid : p->solve_blocks == 1 ? kBlock : kCluster;
    if (p->solve_blocks == 0)
        kind = sc->n_c <= 2 * kColorThreads ? kBlock : sc->n_c <= 2 * clusters * kColorThreads ? kCluster : kGrid;
    if (kind == kCluster && clusters < 2) kind = kGrid;
    if (kind == kGrid && grid < 2) kind = kBlock;
    const int ctas = kind == kGrid ? grid : kind == kCluster ? clusters : 1;
    const void *fn = kind == kGrid ? (const void *)k_color<T, kGrid>
                     : kind == kCluster ? (const void *)k_color<T, kCluster> : (const void *)k_color<T, kBlock>;
    if (kind == kGrid) cudaMemsetAsync(st->barrier, 0, sizeof(uint32_t) * kBarrierWords, s);
    int nc = sc->n_c, nb = sc->n_b, cache = p->color_cache, mc = maxc;
    const T *Minv = (const T *)sc->Minv;
    long long tmo = p->barrier_timeout_ns > 0 ? p->barrier_timeout_ns : 1000000000LL;
    b2c_ncp_state state = *st;
    void *args[] = {&nc, &nb, (void *)&sc->pa, (void *)&sc->pb, (void *)&sc->feature, &Minv, &st->dyn, &state, &cache,
                    &mc, &tmo};
    return launch_kind(fn, args, kind, ctas, kind == kGrid ? kColorGridThreads : kColorThreads, 0, "ncp_color", s);
}

// A phase kernel: its three forms (one CTA, a cluster, a cooperative grid), their threads and shared
// memory, the most CTAs of the cluster and the grid that the device holds at once, where the
// automatic form changes (Form), and the kernels for many rounds of contacts a phase (NULL: none)
// with the rounds, in halves, from which they run
struct PhaseKernel {
    const void *fn[3];
    int threads[3];
    size_t smem;
    int cluster_max, grid_max;
    int narrow, narrow_contacts, wide;
    const void *many[3];
    int many_rounds[3];
};

// Runs a phase kernel in the form asked for (b2c_ncp_params.solve_blocks: 1 one CTA, n > 1 a
// cooperative grid, -n a cluster) or, for 0, in the one that suits the scene.  block_extra: shared
// memory of the one CTA behind its task table.
template <typename A>
int run_phases(A &a, int asked, const PhaseKernel &k, size_t block_extra, const char *what, cudaStream_t s)
{
    const int nc = a.nc;
    a.form = Form{asked, k.narrow, k.narrow_contacts, k.wide, 0};
    // a form's kernel and, where a colour can be wide enough, its kernel for many rounds: the
    // colouring lets one of the two run (automatic: only the grid, the others change form before)
    auto launch = [&](int kind, int ctas) {
        const bool has_many = k.many[kind] && (a.form.asked != 0 || kind == kGrid);
        a.form.many = has_many ? std::max(1, ctas * (k.threads[kind] / kGroup) * k.many_rounds[kind] / 2) : 0;
        void *args[] = {&a};
        if (kind == kGrid) cudaMemsetAsync(a.bar, 0, sizeof(uint32_t), s);  // the arrival count restarts every launch
        const int rc = launch_kind(k.fn[kind], args, kind, ctas, k.threads[kind],
                                   k.smem + (kind == kBlock ? block_extra : 0), what, s);
        if (rc != B2C_OK || !has_many || nc < a.form.many) return rc;
        return launch_kind(k.many[kind], args, kind, ctas, kManyThreads, 0, what, s);
    };
    if (asked > 1 && std::min(asked, k.grid_max) > 1) return launch(kGrid, std::min(asked, k.grid_max));
    if (asked < 0 && std::min(-asked, k.cluster_max) >= 2) return launch(kCluster, std::min(-asked, k.cluster_max));
    if (asked != 0 || k.cluster_max < 2) {  // one CTA, asked for or all there is; without clusters the grid
        const bool grid = asked == 0 && k.grid_max > 1 && nc > k.narrow_contacts;
        a.form.asked = grid ? k.grid_max : 1;
        return grid ? launch(kGrid, k.grid_max) : launch(kBlock, 1);
    }
    // auto: every form that some colouring of nc contacts wants is launched, and the colouring that
    // the device found lets one of them run (Form::here; the others return at once)
    if (k.grid_max < 2) a.form.wide = nc + 1;
    int rc = B2C_OK;
    if (nc <= k.narrow_contacts) rc = launch(kBlock, 1);
    if (rc == B2C_OK && nc >= k.narrow) rc = launch(kCluster, k.cluster_max);
    if (rc == B2C_OK && nc >= a.form.wide) rc = launch(kGrid, k.grid_max);
    return rc;
}

template <typename T>
int sweeps(const b2c_ncp_scene *sc, b2c_ncp_state *st, const b2c_ncp_params *p, int iters, cudaStream_t s,
           double *trace = nullptr)
{
    if (iters <= 0 || sc->n_c == 0) return B2C_OK;
    SweepArgs<T> a = sweep_args<T>(sc, st, p, iters);
    a.trace = trace;
    const size_t state = 6 * (sizeof(T) + 8) * (size_t)sc->n_b;
    a.smem_bodies = state <= kStateBytes ? sc->n_b : 0;
    static const PhaseKernel k = {
        {(const void *)k_sweeps<T, kBlock>, (const void *)k_sweeps<T, kCluster>, (const void *)k_sweeps<T, kGrid>},
        {sweep_threads<T, kBlock>(), sweep_threads<T, kCluster>(), sweep_threads<T, kGrid>()},
        kTableBytes,
        std::min(cluster_size<T>(), cluster_size_of((const void *)k_sweeps_many<T, kCluster>, kManyThreads, 0)),
        std::min(grid_blocks<T>(), grid_blocks_of((const void *)k_sweeps_many<T, kGrid>, kManyThreads, 0)),
        16, 2048, cluster_size<T>() * (sweep_threads<T, kCluster>() / kGroup) * 31 / 32,
        {(const void *)k_sweeps_many<T, kBlock>, (const void *)k_sweeps_many<T, kCluster>,
         kManyRounds<T, kGrid> ? (const void *)k_sweeps_many<T, kGrid> : nullptr},
        {kManyRounds<T, kBlock>, kManyRounds<T, kCluster>, kManyRounds<T, kGrid>}};
    return run_phases(a, p->solve_blocks, k, a.smem_bodies ? state : 0, "ncp_sweeps", s);
}

template <typename T>
int residual(const b2c_ncp_scene *sc, b2c_ncp_state *st, const b2c_ncp_params *p, cudaStream_t s)
{
    cudaMemsetAsync(st->res_max, 0, sizeof(uint64_t), s);
    if (sc->n_c == 0) return check_launch("ncp_residual");
    const SweepArgs<T> a = sweep_args<T>(sc, st, p, 0);
    k_resid<T><<<blocks_for(sc->n_c), kThreads, 0, s>>>(a, (T *)st->res, (T *)st->u,
                                                         reinterpret_cast<unsigned long long *>(st->res_max));
    return check_launch("ncp_residual");
}

// ---------------------------------------------------------------------------------------------
// The adjoint of the sweeps at a fixed point (float64): the implicit-function derivative of the
// converged impulses, as the reverse of `iters` sweeps evaluated at the final iterate.
//
// A forward sweep maps lambda -> Phi(lambda; b, mu) with b = J v_free + bias; at its fixed point
// lambda* the implicit function theorem gives d lambda* = (I - dPhi/dlambda)^-1 dPhi/d(b, mu).
// Its transpose applied to an adjoint g is the limit of the reverse sweeps: starting from g,
// each reverse sweep (colours in reverse order, each contact the transposed derivative of its
// update at lambda*) pushes the adjoint back through one sweep and hands the free velocity, the
// bias and the friction their share; `iters` reverse sweeps sum the first `iters` terms of that
// Neumann series, the same truncation as `iters` forward sweeps from a warm start.
//
// One contact update (forward, in colour order, v the current body velocities):
//   u = J v + bias,  z = lambda - rho (u + (mu |u_t|, 0, 0)),  lambda' = proj_K(z),
//   v += Minv J^T (lambda' - lambda).
// Its reverse, given the adjoints gl of lambda' and Vb of v after it:
//   g  = gl + J Minv Vb;  (zb, mub) = the transposed derivative of proj_K at z applied to g;
//   gl <- zb - J Minv Vb;  ub = -rho (zb + mu zb_n u_t / |u_t| on the tangential rows);
//   Vb += J^T ub;  bias_b += ub;  mu_b += mub - rho |u_t| zb_n.
// After the last (first) colour, the adjoint of v at the sweep's start goes to v_free (v =
// v_free + Minv J^T lambda) and, through J Minv, back onto every gl; Vb restarts at zero.
// Within a colour no two contacts share a dynamic body, so every write is the owner's; the
// adjoint of kinematic and static bodies is not kept (their velocity is prescribed).
// ---------------------------------------------------------------------------------------------
struct AdjArgs {
    Form form;
    int nc, nb, iters, desaxce;
    const double *Ja, *Jb, *Minv, *mu, *rho, *lam, *u;
    double *trace;  // null: every reverse sweep at the final iterate (lam, u); else the recorded sweeps
    const int *pa, *pb, *order, *cstart, *ccount, *dyn;
    double *gl, *vb, *vfree_b, *bias_b, *mu_b;
    double *Ja_b, *Jb_b, *Minv_b, *rho_b;  // the recorded form's adjoints of the blocks and step sizes
    int *stats;
    unsigned int *bar;
    long long timeout_ns;
};

// J_side (3x6) Minv_b (6x6) x, x = Vb of body b (6): out[3] += J (Minv x)
__device__ __forceinline__ void add_j_minv(const double *J, const double *M, const double *x, double out[3])
{
    double t[6];
    for (int k = 0; k < 6; ++k) {
        double s = 0.0;
        for (int j = 0; j < 6; ++j) s += M[k * 6 + j] * x[j];
        t[k] = s;
    }
    for (int r = 0; r < 3; ++r) {
        double s = 0.0;
        for (int k = 0; k < 6; ++k) s += J[r * 6 + k] * t[k];
        out[r] += s;
    }
}

// The de Saxce term mu |u_t| has a kink at u_t = 0, where a sticking contact sits: its slip
// speed there is the rounding of the fixed-point velocity sums (1e-10 m/s), whose direction says
// nothing.  Below this speed the adjoints take the term's derivative in u_t as zero (the stick
// rows of the implicit-function system, ncp_ref.py:_active_system, carry no such term either).
constexpr double kStickSpeed = 1e-8;

// transposed derivative of proj_K (the branches of proj) at z, applied to g: zb, and mub
__device__ __forceinline__ void proj_adjoint(const double z[3], double mu, const double g[3], double zb[3],
                                             double &mub)
{
    const double zn = z[0], zt = sqrt(z[1] * z[1] + z[2] * z[2]);
    if (zt <= mu * zn) {
        zb[0] = g[0];
        zb[1] = g[1];
        zb[2] = g[2];
        return;
    }
    if (mu * zt <= -zn) {
        zb[0] = zb[1] = zb[2] = 0.0;
        return;
    }
    // s = (zn + mu zt) / (1 + mu^2), f = mu s / zt, out = (s, f z1, f z2)
    const double den = 1.0 + mu * mu, iden = 1.0 / den, izt = 1.0 / zt;
    const double sv = (zn + mu * zt) * iden;
    const double f = mu * sv * izt;
    const double t1 = z[1] * izt, t2 = z[2] * izt;
    const double ds_dzn = iden;
    const double ds_dt1 = mu * t1 * iden, ds_dt2 = mu * t2 * iden;
    const double ds_dmu = (zt * den - 2.0 * mu * (zn + mu * zt)) * iden * iden;
    const double df_dzn = mu * ds_dzn * izt;
    const double df_dt1 = (mu * ds_dt1 - mu * sv * t1 * izt) * izt;
    const double df_dt2 = (mu * ds_dt2 - mu * sv * t2 * izt) * izt;
    const double df_dmu = (sv + mu * ds_dmu) * izt;
    const double gz = g[1] * z[1] + g[2] * z[2];
    zb[0] = g[0] * ds_dzn + gz * df_dzn;
    zb[1] = g[0] * ds_dt1 + f * g[1] + gz * df_dt1;
    zb[2] = g[0] * ds_dt2 + f * g[2] + gz * df_dt2;
    mub += g[0] * ds_dmu + gz * df_dmu;
}

__device__ void adj_contact(const AdjArgs &a, int c)
{
    const int A = a.pa[c], B = a.pb[c];
    const bool dA = A >= 0 && a.dyn[A], dB = B >= 0 && a.dyn[B];
    double vA[6], vBb[6];
    double jm[3] = {0.0, 0.0, 0.0};
    if (dA) {
        for (int k = 0; k < 6; ++k) vA[k] = __ldcg(a.vb + 6 * (size_t)A + k);
        add_j_minv(a.Ja + 18 * (size_t)c, a.Minv + 36 * (size_t)A, vA, jm);
    }
    if (dB) {
        for (int k = 0; k < 6; ++k) vBb[k] = __ldcg(a.vb + 6 * (size_t)B + k);
        add_j_minv(a.Jb + 18 * (size_t)c, a.Minv + 36 * (size_t)B, vBb, jm);
    }
    double g[3], z[3], u[3], lo[3];
    const double mu = a.mu[c], rho = a.rho[c];
    for (int k = 0; k < 3; ++k) {
        g[k] = a.gl[3 * (size_t)c + k] + jm[k];
        u[k] = a.u[3 * (size_t)c + k];
        lo[k] = a.lam[3 * (size_t)c + k];
    }
    const double ut = sqrt(u[1] * u[1] + u[2] * u[2]);
    const double s0 = a.desaxce ? u[0] + mu * ut : u[0];
    z[0] = lo[0] - rho * s0;
    z[1] = lo[1] - rho * u[1];
    z[2] = lo[2] - rho * u[2];
    double zb[3], mub = 0.0;
    proj_adjoint(z, mu, g, zb, mub);
    double ub[3];
    ub[0] = -rho * zb[0];
    ub[1] = -rho * zb[1];
    ub[2] = -rho * zb[2];
    if (a.desaxce) {
        mub += -rho * ut * zb[0];
        if (ut > kStickSpeed) {
            ub[1] += -rho * mu * (u[1] / ut) * zb[0];
            ub[2] += -rho * mu * (u[2] / ut) * zb[0];
        }
    }
    for (int k = 0; k < 3; ++k) {
        a.gl[3 * (size_t)c + k] = zb[k] - jm[k];
        a.bias_b[3 * (size_t)c + k] += ub[k];
    }
    a.mu_b[c] += mub;
    for (int side = 0; side < 2; ++side) {
        if (!(side == 0 ? dA : dB)) continue;
        const int b = side == 0 ? A : B;
        const double *J = (side == 0 ? a.Ja : a.Jb) + 18 * (size_t)c;
        const double *cur = side == 0 ? vA : vBb;
        for (int k = 0; k < 6; ++k)
            __stcg(a.vb + 6 * (size_t)b + k, cur[k] + ((J[k] * ub[0] + J[6 + k] * ub[1]) + J[12 + k] * ub[2]));
    }
}

// The reverse of one recorded update of contact c in sweep `it` (sweep_contact_group):
//   u = bias + Ja va + Jb vb,  z = lo - rho (u_n + mu |u_t| (de Saxce), u_t),  l = proj(z),
//   v_a += Minv_a Ja^T (l - lo),  v_b likewise,
// with z and u read back from the record.  On entry gl[c] is the adjoint of l and vb the
// adjoint of the velocities after the update; on exit gl[c] is the adjoint of lo and vb that of
// the velocities before it, and bias_b, mu_b, rho_b hold the update's share.  Only vb and gl
// are on the path to the next update; what the blocks' and Minv's adjoints need (ub, the impulse
// change dl, the velocity adjoints) goes back into the trace for adj_start_group.
// It runs on a group of kGroup lanes (the forward's layout): lanes 0..5 the six sums of u,
// lanes 0..11 one velocity component k of one side each (its vbar, row k of Minv vbar, its
// share of J Minv vbar -- summed over the lanes by a fixed butterfly -- and its vbar update),
// every lane the projection and its adjoint.
//
// The projection's derivative depends on the record alone, so it is formed, with every other
// word that the other contacts of the sweep do not change (AdjPre), before the barrier's wait;
// behind the barrier are the bodies' vbar, two small products, three butterflies and the update.
// Measured on a B200 with the whole update behind the barrier before: forward and backward over a
// four-step rollout of 24 stacks of boxes (11 668 contacts) 524 -> 75 ms, of 4 stacks 55 ms.
struct AdjPre {
    Task k;
    int b;                      // this lane's body
    bool mine;                  // lane (side, k) of a dynamic body
    double *tr;
    double Jc[3], Mr[6];        // column k of the side's block, row k of Minv
    double gl[3], mu, rho, s0, u1, u2, q;  // q = -rho mu / |u_t| of the de Saxce term (0 where it has none)
    double ds[3], df[3], f, zn, z1, z2;    // the projection's derivative: zb = g0 ds + (g_t . z_t) df + f g_t
    double dsm, dfm, mut;              // and in mu: mub = g0 dsm + (g_t . z_t) dfm + mut zb0
    double old;                 // the running sum this lane adds to: bias_b (lanes 0..2), mu_b (3), rho_b (4)
};

__device__ __forceinline__ double *adj_sum(const AdjArgs &a, size_t c, int l)
{
    return l < 3 ? a.bias_b + 3 * c + l : l == 3 ? a.mu_b + c : a.rho_b + c;
}

// what the contact's own updates change
__device__ __forceinline__ void adj_own(const AdjArgs &a, int l, AdjPre &q)
{
    const size_t c = (size_t)q.k.c;
#pragma unroll
    for (int r = 0; r < 3; ++r) q.gl[r] = a.gl[3 * c + r];
    q.old = l < 5 ? *adj_sum(a, c, l) : 0.0;
}

__device__ __forceinline__ void adj_load(const AdjArgs &a, const Task &task, int it, int l, AdjPre &q)
{
    const int c = task.c;
    q.k = task;
    q.tr = a.trace + kTraceWords * ((size_t)it * a.nc + c);
    const int side = l / 6, k = l - 6 * side;
    q.b = side == 0 ? task.pa : task.pb;
    q.mine = side < 2 && (task.bits & (side == 0 ? 1 : 2)) != 0;
#pragma unroll
    for (int r = 0; r < 3; ++r) q.Jc[r] = 0.0;
#pragma unroll
    for (int j = 0; j < 6; ++j) q.Mr[j] = 0.0;
    if (q.mine) {
        const double *J = (side == 0 ? a.Ja : a.Jb) + 18 * (size_t)c + k, *M = a.Minv + 36 * (size_t)q.b + 6 * k;
#pragma unroll
        for (int r = 0; r < 3; ++r) q.Jc[r] = J[6 * r];
#pragma unroll
        for (int j = 0; j < 6; ++j) q.Mr[j] = M[j];
    }
    q.zn = q.tr[33];
    q.z1 = q.tr[34];
    q.z2 = q.tr[35];
    q.s0 = q.tr[36];
    q.u1 = q.tr[37];
    q.u2 = q.tr[38];
    q.mu = a.mu[c];
    q.rho = a.rho[c];
    adj_own(a, l, q);
}

__device__ __forceinline__ void adj_finish(const AdjArgs &a, int l, AdjPre &q)
{
    const double mu = q.mu, zn = q.zn, z1 = q.z1, z2 = q.z2;
    // |u_t| on the even lanes, |z_t| on the odd ones
    const bool odd = (l & 1) != 0;
    const double x1 = odd ? z1 : q.u1, x2 = odd ? z2 : q.u2;
    const double root = sqrt(x1 * x1 + x2 * x2), other = __shfl_xor_sync(kWarp, root, 1, kGroup);
    const double ut = odd ? other : root, zt = odd ? root : other;
    if (a.desaxce) q.s0 = q.s0 + mu * ut;
    q.q = a.desaxce && ut > kStickSpeed ? -q.rho * mu / ut : 0.0;
    q.mut = a.desaxce ? -q.rho * ut : 0.0;
    // proj's branches (proj_adjoint): inside the cone zb = g, below it 0, else the side's derivative
    const bool inside = zt <= mu * zn, below = mu * zt <= -zn;
    q.ds[0] = q.f = inside ? 1.0 : 0.0;
    q.ds[1] = q.ds[2] = q.df[0] = q.df[1] = q.df[2] = q.dsm = q.dfm = 0.0;
    if (!inside && !below) {
        const double den = 1.0 + mu * mu, iden = 1.0 / den, izt = 1.0 / zt;
        const double sv = (zn + mu * zt) * iden;
        const double t1 = z1 * izt, t2 = z2 * izt;
        q.f = mu * sv * izt;
        q.ds[0] = iden;
        q.ds[1] = mu * t1 * iden;
        q.ds[2] = mu * t2 * iden;
        q.dsm = (zt * den - 2.0 * mu * (zn + mu * zt)) * iden * iden;
        q.df[0] = mu * iden * izt;
        q.df[1] = (mu * q.ds[1] - mu * sv * t1 * izt) * izt;
        q.df[2] = (mu * q.ds[2] - mu * sv * t2 * izt) * izt;
        q.dfm = (sv + mu * q.dsm) * izt;
    }
}

template <int kKind>
__device__ __forceinline__ void adj_contact_group(const AdjArgs &a, const AdjPre &q, int l)
{
    const int side = l / 6, k = l - 6 * side;
    double *vb = a.vb + 6 * (size_t)(q.mine ? q.b : 0) + k;
    const double w = q.mine ? shared_load<kKind>(vb) : 0.0;
    // row k of Minv vbar for this lane's side, then J Minv vbar summed over the lanes
    const int base = l < 6 ? 0 : 6;
    double mk = 0.0;
#pragma unroll
    for (int j = 0; j < 6; ++j) mk += q.Mr[j] * group_get(w, base + j);
    double jm[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        double x = q.Jc[r] * mk;
#pragma unroll
        for (int off = kGroup / 2; off > 0; off >>= 1) x += __shfl_xor_sync(kWarp, x, off, kGroup);
        jm[r] = x;
    }
    const double g0 = q.gl[0] + jm[0], g1 = q.gl[1] + jm[1], g2 = q.gl[2] + jm[2];
    const double gz = g1 * q.z1 + g2 * q.z2;
    const double zb0 = g0 * q.ds[0] + gz * q.df[0];
    const double zb1 = g0 * q.ds[1] + q.f * g1 + gz * q.df[1];
    const double zb2 = g0 * q.ds[2] + q.f * g2 + gz * q.df[2];
    const double ub0 = -q.rho * zb0, ub1 = -q.rho * zb1 + q.q * q.u1 * zb0, ub2 = -q.rho * zb2 + q.q * q.u2 * zb0;
    if (!(q.k.bits & 4)) return;
    if (q.mine) shared_store<kKind>(vb, w + ((q.Jc[0] * ub0 + q.Jc[1] * ub1) + q.Jc[2] * ub2));
    if (l < 12) q.tr[21 + 6 * side + k] = w;  // zero where the side has no dynamic body
    const size_t c = (size_t)q.k.c;
    if (l < 3) {
        const double ub = l == 0 ? ub0 : l == 1 ? ub1 : ub2;
        q.tr[15 + l] = ub;
        a.gl[3 * c + l] = (l == 0 ? zb0 : l == 1 ? zb1 : zb2) - (l == 0 ? jm[0] : l == 1 ? jm[1] : jm[2]);
        *adj_sum(a, c, l) = q.old + ub;
    } else if (l == 3) {
        *adj_sum(a, c, l) = q.old + (g0 * q.dsm + gz * q.dfm + q.mut * zb0);
    } else if (l == 4) {
        *adj_sum(a, c, l) = q.old - (zb0 * q.s0 + zb1 * q.u1 + zb2 * q.u2);
    }
}

// unit eigenvector of the largest eigenvalue lm of a symmetric 3x3 W, from the largest cross
// product of two rows of W - lm I; false when that eigenvalue is not simple (no derivative)
__device__ bool eigvec_max3(const double W[3][3], double lm, double e[3])
{
    double R[3][3];
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) R[i][j] = W[i][j] - (i == j ? lm : 0.0);
    double best = 0.0;
    for (int p = 0; p < 3; ++p) {
        const double *x = R[p], *y = R[(p + 1) % 3];
        const double cr[3] = {x[1] * y[2] - x[2] * y[1], x[2] * y[0] - x[0] * y[2], x[0] * y[1] - x[1] * y[0]};
        const double nn = cr[0] * cr[0] + cr[1] * cr[1] + cr[2] * cr[2];
        if (nn > best) {
            best = nn;
            for (int k = 0; k < 3; ++k) e[k] = cr[k];
        }
    }
    if (!(best > 1e-20 * lm * lm * lm * lm)) return false;
    const double inv = 1.0 / sqrt(best);
    for (int k = 0; k < 3; ++k) e[k] *= inv;
    return true;
}

// The derivative of rho_c = 1 / lambda_max(W_c) takes the projector P onto the eigenspace of
// the largest eigenvalue lm, divided by its dimension k: d lm = tr(P dW) / k.  For a simple
// eigenvalue (k = 1) that is the derivative; for a repeated one -- every corner contact of a
// cube on the ground, whose inertia is isotropic, has lm twice -- lm is not differentiable and
// tr(P dW) / k, the derivative of the mean of the k top eigenvalues, is what a central
// difference measures.  Eigenvalues within 1e-6 lm of lm count as repeated.
__device__ void top_projector(const double W[3][3], double lm, double P[3][3])
{
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) P[i][j] = 0.0;
    const double c2 = W[0][0] + W[1][1] + W[2][2];
    const double c1 = (W[0][0] * W[1][1] - W[0][1] * W[1][0]) + (W[0][0] * W[2][2] - W[0][2] * W[2][0]) +
                      (W[1][1] * W[2][2] - W[1][2] * W[2][1]);
    const double sm = c2 - lm, pr = c1 - lm * sm;  // the other two: sum and product
    const double disc = sqrt(fmax(sm * sm - 4.0 * pr, 0.0));
    const double l2 = 0.5 * (sm + disc), l3 = 0.5 * (sm - disc);
    const double tol = 1e-6 * lm;
    if (lm - l3 <= tol) {
        for (int i = 0; i < 3; ++i) P[i][i] = 1.0 / 3.0;
        return;
    }
    if (lm - l2 <= tol) {  // W - lm I ~ (l3 - lm) e3 e3^T: its largest row is along e3
        int best = 0;
        double bn = -1.0;
        for (int r = 0; r < 3; ++r) {
            double nn = 0.0;
            for (int k = 0; k < 3; ++k) {
                const double x = W[r][k] - (r == k ? lm : 0.0);
                nn += x * x;
            }
            if (nn > bn) {
                bn = nn;
                best = r;
            }
        }
        double e3[3];
        const double inv = 1.0 / sqrt(bn);
        for (int k = 0; k < 3; ++k) e3[k] = (W[best][k] - (best == k ? lm : 0.0)) * inv;
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) P[i][j] = 0.5 * ((i == j ? 1.0 : 0.0) - e3[i] * e3[j]);
        return;
    }
    double e[3];
    if (!eigvec_max3(W, lm, e)) return;
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) P[i][j] = e[i] * e[j];
}

// Wbar of contact c (below), symmetric: its six words in w
__device__ __noinline__ void adj_step_size(const AdjArgs &a, int c, double w[6])
{
    const int A = a.pa[c], B = a.pb[c];
    const double rho = a.rho[c], rb = a.rho_b[c];
#pragma unroll
    for (int i = 0; i < 6; ++i) w[i] = 0.0;
    if (rb == 0.0 || !(rho > 0.0)) return;
    double W[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    if (A >= 0) add_jmjt(W, a.Ja + 18 * (size_t)c, a.Minv + 36 * (size_t)A);
    if (B >= 0) add_jmjt(W, a.Jb + 18 * (size_t)c, a.Minv + 36 * (size_t)B);
    double P[3][3];
    top_projector(W, eigmax3(W), P);
    const double lmb = -rho * rho * rb;  // rho = 1 / lambda_max
#pragma unroll
    for (int i = 0, n = 0; i < 3; ++i)
#pragma unroll
        for (int j = i; j < 3; ++j) w[n++] = lmb * P[i][j];
}

// After the reverse sweeps, per contact (colour by colour, so that each dynamic body belongs to
// one contact at a time): the blocks' and Minv's adjoints summed over the recorded updates --
// ub (x) v (through u) and dl (x) Minv vbar (through the velocity change) for the blocks,
// vbar (x) J^T dl for Minv -- and the start of the sweeps, v = v_free + Minv sum_c J_c^T lo_c
// (setup, lo the warm start) and rho_c = 1 / lambda_max(W_c), W_c = sum_sides J Minv J^T
// (k_rho): gl[c] += J Minv vbar (the warm start's adjoint), lo (x) Minv vbar and vbar (x) J^T lo,
// and rho_b through Wbar = -rho^2 rho_b P / k (top_projector).  A group of kGroup lanes per
// contact: lane (side, k), k < 6, owns column k of its side's block adjoint (3 entries) and of
// its body's Minv adjoint (6 entries) and walks the sweeps for them.
// Wbar is the longest part of it, a Newton iteration, and needs no order: it comes from shared
// memory (`wb`), where the threads of the CTA formed those of its tasks of all colours at once.
// (What a reverse sweep costs besides its sweeps, on a B200: 640 -> 520 us for 24 stacks of boxes.)
template <int kKind>
__device__ void adj_start_group(const AdjArgs &a, int c, int l, unsigned mask, const double *wb)
{
    const int A = a.pa[c], B = a.pb[c];
    const double *tr0 = a.trace + kTraceWords * (size_t)c;  // sweep 0
    const double lo[3] = {tr0[0], tr0[1], tr0[2]};
    double w6[6];
    if (wb) {
#pragma unroll
        for (int i = 0; i < 6; ++i) w6[i] = wb[i];
    } else {
        adj_step_size(a, c, w6);
    }
    const double Wb[3][3] = {{w6[0], w6[1], w6[2]}, {w6[1], w6[3], w6[4]}, {w6[2], w6[4], w6[5]}};
    const int side = l / 6, k = l % 6, b = side == 0 ? A : B;
    const bool on = l < 12 && b >= 0, d = on && a.dyn[b] != 0;
    double jm[3] = {0.0, 0.0, 0.0};
    if (on) {
        const double *M = a.Minv + 36 * (size_t)b, *J = (side == 0 ? a.Ja : a.Jb) + 18 * (size_t)c;
        const int vo = side == 0 ? 3 : 9, wo = side == 0 ? 21 : 27;
        double Jc[3] = {0.0, 0.0, 0.0}, Mc[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll 4
        for (int it = 0; it < a.iters; ++it) {
            const double *tr = a.trace + kTraceWords * ((size_t)it * a.nc + c);
            const double ub[3] = {tr[15], tr[16], tr[17]}, vk = tr[vo + k];
            const double dl[3] = {tr[18], tr[19], tr[20]};
            double w[6], mk = 0.0;
            for (int j = 0; j < 6; ++j) {
                w[j] = tr[wo + j];
                mk += M[6 * k + j] * w[j];
            }
            for (int r = 0; r < 3; ++r) Jc[r] += ub[r] * vk;
            if (!d) continue;
            for (int r = 0; r < 3; ++r) Jc[r] += dl[r] * mk;
            const double jt = (J[k] * dl[0] + J[6 + k] * dl[1]) + J[12 + k] * dl[2];
            for (int i = 0; i < 6; ++i) Mc[i] += w[i] * jt;
        }
        double *Jbar = (side == 0 ? a.Ja_b : a.Jb_b) + 18 * (size_t)c;
        if (d) {
            // the start: vbar of the sweeps' initial velocities
            double w0[6], m0 = 0.0;
            for (int j = 0; j < 6; ++j) {
                w0[j] = shared_load<kKind>(a.vb + 6 * (size_t)b + j);
                m0 += M[6 * k + j] * w0[j];
            }
            const double jt0 = (J[k] * lo[0] + J[6 + k] * lo[1]) + J[12 + k] * lo[2];
            for (int r = 0; r < 3; ++r) jm[r] = J[6 * r + k] * m0;
            // WJ = Wbar J (3x6); Jbar += 2 Wbar J Minv, Minv_bar += J^T Wbar J (column k)
            double WJ[3][6];
            for (int r = 0; r < 3; ++r)
                for (int j = 0; j < 6; ++j) WJ[r][j] = (Wb[r][0] * J[j] + Wb[r][1] * J[6 + j]) + Wb[r][2] * J[12 + j];
            for (int r = 0; r < 3; ++r) {
                double sacc = 0.0;
                for (int j = 0; j < 6; ++j) sacc += WJ[r][j] * M[j * 6 + k];
                Jbar[6 * r + k] += Jc[r] + lo[r] * m0 + 2.0 * sacc;
            }
            double *Mb = a.Minv_b + 36 * (size_t)b;
            for (int i = 0; i < 6; ++i) {
                const double jwj = (J[i] * WJ[0][k] + J[6 + i] * WJ[1][k]) + J[12 + i] * WJ[2][k];
                shared_store<kKind>(Mb + 6 * i + k, shared_load<kKind>(Mb + 6 * i + k) + (Mc[i] + w0[i] * jt0 + jwj));
            }
        } else {
            for (int r = 0; r < 3; ++r) Jbar[6 * r + k] += Jc[r];
        }
    }
    for (int r = 0; r < 3; ++r) {
        double x = jm[r];
        for (int off = kGroup / 2; off > 0; off >>= 1) x += __shfl_xor_sync(mask, x, off, kGroup);
        if (l == 0) a.gl[3 * (size_t)c + r] += x;
    }
}

template <int kKind>
__device__ __forceinline__ bool adj_barrier(const AdjArgs &a, unsigned int &epoch)
{
    phase_arrive<kKind>(a, epoch);
    return phase_wait<kKind>(a, epoch);
}

template <int kKind>
constexpr int adj_threads()
{
    return kAhead<kKind> ? 384 : 512;
}

template <int kKind>
__global__ void __launch_bounds__(adj_threads<kKind>()) k_adj_sweeps(AdjArgs a)
{
    const int ncol = a.stats[kNColors];
    if (!a.form.here(kKind, false, a.nc, ncol)) return;  // uniform over the launch
    const int nb = gridDim.x, nth = gridDim.x * blockDim.x;
    const int tid = ((((int)threadIdx.x >> 5) * nb + (int)blockIdx.x) << 5) | ((int)threadIdx.x & 31);
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned int epoch = 0;
    if (a.trace) {
        // the recorded sweeps in reverse (a group of kGroup lanes per contact, the forward's
        // task layout), then their start; vb carries through
        __shared__ int s_start[kMaxColors], s_count[kMaxColors];
        const TaskTable tt = task_table(a, ncol, s_start, s_count);
        const int groups = nb * tt.per;
        const int lg = (int)threadIdx.x / kGroup, g = lg * nb + (int)blockIdx.x, l = (int)threadIdx.x % kGroup;
        const int g0 = (lg & ~1) * nb + (int)blockIdx.x;  // the warp's first group
        const unsigned mask = 0xFFFFu << (((int)threadIdx.x & 31) & ~(kGroup - 1));
        AdjPre pre = {}, next = {};
        int it = a.iters - 1, ci = ncol - 1, cnt = ncol > 0 ? s_count[ncol - 1] : 0, t = g, t0 = g0;
        bool have = t0 < cnt;
        if (have) {
            adj_load(a, tt.get(ci, t, lg, true), it, l, pre);
            adj_finish(a, l, pre);
        }
        while (it >= 0 && ncol > 0) {
            const bool now = have;
            if (!kAhead<kKind> && now) adj_contact_group<kKind>(a, pre, l);
            t += groups;
            t0 += groups;
            const bool more = t0 < cnt;
            if (!more) {
                t = g;
                t0 = g0;
                if (--ci < 0) {
                    ci = ncol - 1;
                    --it;
                }
                cnt = s_count[ci];
            }
            have = it >= 0 && t0 < cnt;
            if (kAhead<kKind>) {
                if (have) adj_load(a, tt.get(ci, t, lg, !more), it, l, next);
                if (now) adj_contact_group<kKind>(a, pre, l);
            }
            __syncwarp();
            if (!more) phase_arrive<kKind>(a, epoch);
            if (have) {
                if (!kAhead<kKind>) {
                    adj_load(a, tt.get(ci, t, lg, !more), it, l, pre);
                } else {
                    if (next.k.c == pre.k.c) adj_own(a, l, next);
                    pre = next;
                }
                adj_finish(a, l, pre);
            }
            if (!more && !phase_wait<kKind>(a, epoch)) return;
        }
        // the task table is done with: its memory takes Wbar of the groups' first rounds
        double *wbar = reinterpret_cast<double *>(s_tasks);
        const int held = min(ncol, kTableBytes / (48 * tt.per));
        __syncthreads();
        for (int i = threadIdx.x; i < held * tt.per; i += blockDim.x) {
            const int ci = i / tt.per, first = (i - ci * tt.per) * nb + (int)blockIdx.x;
            if (first < s_count[ci]) adj_step_size(a, a.order[s_start[ci] + first], wbar + 6 * i);
        }
        __syncthreads();
        for (int ci = 0; ci < ncol; ++ci) {
            const int s0 = a.cstart[ci], cnt = a.ccount[ci];
            for (int t = g; t < cnt; t += groups)
                adj_start_group<kKind>(a, a.order[s0 + t], l, mask,
                                       t == g && ci < held ? wbar + 6 * (ci * tt.per + lg) : nullptr);
            if (!adj_barrier<kKind>(a, epoch)) return;
        }
        for (int i = gid; i < 6 * a.nb; i += nth) {
            a.vfree_b[i] += __ldcg(a.vb + i);
            __stcg(a.vb + i, 0.0);
        }
        return;
    }
    for (int it = 0; it < a.iters; ++it) {
        for (int ci = ncol - 1; ci >= 0; --ci) {
            const int s0 = a.cstart[ci], cnt = a.ccount[ci];
            for (int t = tid; t < cnt; t += nth) adj_contact(a, a.order[s0 + t]);
            if (!adj_barrier<kKind>(a, epoch)) return;
        }
        // the sweep's start: v = v_free + Minv J^T lambda
        for (int c = gid; c < a.nc; c += nth) {
            const int A = a.pa[c], B = a.pb[c];
            double jm[3] = {0.0, 0.0, 0.0}, x[6];
            if (A >= 0 && a.dyn[A]) {
                for (int k = 0; k < 6; ++k) x[k] = __ldcg(a.vb + 6 * (size_t)A + k);
                add_j_minv(a.Ja + 18 * (size_t)c, a.Minv + 36 * (size_t)A, x, jm);
            }
            if (B >= 0 && a.dyn[B]) {
                for (int k = 0; k < 6; ++k) x[k] = __ldcg(a.vb + 6 * (size_t)B + k);
                add_j_minv(a.Jb + 18 * (size_t)c, a.Minv + 36 * (size_t)B, x, jm);
            }
            for (int k = 0; k < 3; ++k) a.gl[3 * (size_t)c + k] += jm[k];
        }
        if (!adj_barrier<kKind>(a, epoch)) return;
        for (int i = gid; i < 6 * a.nb; i += nth) {
            a.vfree_b[i] += __ldcg(a.vb + i);
            __stcg(a.vb + i, 0.0);
        }
        if (!adj_barrier<kKind>(a, epoch)) return;
    }
}

int adjoint_sweeps(const b2c_ncp_scene *sc, b2c_ncp_state *st, const b2c_ncp_params *p, int iters,
                   double *trace, double *gl, double *vb, double *vfree_b, double *bias_b, double *mu_b,
                   double *Ja_b, double *Jb_b, double *Minv_b, cudaStream_t s)
{
    if (iters <= 0 || sc->n_c == 0) return B2C_OK;
    AdjArgs a;
    a.nc = sc->n_c;
    a.nb = sc->n_b;
    a.iters = iters;
    a.desaxce = p->desaxce;
    a.Ja = (const double *)sc->Ja;
    a.Jb = (const double *)sc->Jb;
    a.Minv = (const double *)sc->Minv;
    a.mu = (const double *)sc->mu;
    a.rho = (const double *)st->rho;
    a.lam = (const double *)st->lam;
    a.u = (const double *)st->u;
    a.trace = trace;
    a.Ja_b = Ja_b;
    a.Jb_b = Jb_b;
    a.Minv_b = Minv_b;
    a.rho_b = (double *)st->res;
    a.pa = sc->pa;
    a.pb = sc->pb;
    a.order = st->order;
    a.cstart = st->cstart;
    a.ccount = st->ccount;
    a.dyn = st->dyn;
    a.gl = gl;
    a.vb = vb;
    a.vfree_b = vfree_b;
    a.bias_b = bias_b;
    a.mu_b = mu_b;
    a.stats = st->stats;
    a.bar = st->barrier;
    a.timeout_ns = p->barrier_timeout_ns > 0 ? p->barrier_timeout_ns : 1000000000LL;
    cudaMemsetAsync(vb, 0, sizeof(double) * 6 * (size_t)sc->n_b, s);
    if (trace) cudaMemsetAsync(st->res, 0, sizeof(double) * (size_t)sc->n_c, s);
    // the recorded sweeps (a group of lanes per contact, the task table in shared memory) and the
    // sweeps at the final iterate (a thread per contact, the blocks through L1, from which a task table
    // would take 96 KB: 80 contacts a colour in one CTA 781 us with it, 599 without).  A thread a
    // contact makes one CTA the best form up to more contacts.  us for 20 reverse sweeps of 8 colours,
    // one CTA / cluster / grid: 75 contacts a colour 982 / 1 113 / 1 362, 100 1 206 / 1 189 / 1 407, 125
    // 1 343 / 1 178 / 1 436, 500 4 380 / 1 212 / 1 515, 1 000 - / 1 410 / 1 517, 1 250 - / 1 578 / 1 534.
    auto phase_kernel = [](bool recorded) {
        const size_t smem = recorded ? kTableBytes : 0;
        const int clusters = cluster_size_of((const void *)k_adj_sweeps<kCluster>, adj_threads<kCluster>(), smem);
        return PhaseKernel{
            {(const void *)k_adj_sweeps<kBlock>, (const void *)k_adj_sweeps<kCluster>, (const void *)k_adj_sweeps<kGrid>},
            {adj_threads<kBlock>(), adj_threads<kCluster>(), adj_threads<kGrid>()}, smem, clusters,
            grid_blocks_of((const void *)k_adj_sweeps<kGrid>, adj_threads<kGrid>(), smem),
            recorded ? 16 : 100, recorded ? 2048 : 16384,
            recorded ? clusters * (adj_threads<kCluster>() / kGroup) : 1200, {}, {}};
    };
    static const PhaseKernel recorded = phase_kernel(true), implicit = phase_kernel(false);
    PhaseKernel k = trace ? recorded : implicit;
    int asked = p->solve_blocks;
    if (!trace && asked < 0) {  // a cluster was asked for: that one, or one CTA below it
        k.cluster_max = std::min(-asked, k.cluster_max);
        k.grid_max = 1;
        asked = 0;
    }
    return run_phases(a, asked, k, 0, "ncp_adjoint", s);
}

}  // namespace ncp
}  // namespace b2c

static bool ncp_scene_ok(const b2c_ncp_scene *sc, const b2c_ncp_state *st)
{
    return sc && st && (sc->dtype == 4 || sc->dtype == 8) && sc->n_c >= 0 && sc->n_b >= 0 &&
           sc->n_c <= st->max_contacts && sc->n_b <= st->n_bodies && sc->Ja && sc->Jb && sc->Minv && sc->v_free &&
           sc->mu && sc->bias && sc->pa && sc->pb && sc->feature && st->rho && st->lam && st->v && st->acc &&
           st->res && st->u && st->col && st->order && st->cstart && st->ccount && st->claim && st->dyn &&
           st->cache_pa && st->cache_pb && st->cache_feat && st->cache_minv && st->stats && st->res_max &&
           st->barrier && st->max_colors >= 1;
}

extern "C" int32_t b2c_ncp_setup(const b2c_ncp_scene *sc, b2c_ncp_state *st, int32_t warm, b2c_stream s)
{
    if (!ncp_scene_ok(sc, st)) {
        b2c::set_error("b2c_ncp_setup: bad argument");
        return B2C_EARG;
    }
    return sc->dtype == 4 ? b2c::ncp::setup<float>(sc, st, warm, b2c::stream_of(s))
                          : b2c::ncp::setup<double>(sc, st, warm, b2c::stream_of(s));
}

extern "C" int32_t b2c_ncp_color(const b2c_ncp_scene *sc, b2c_ncp_state *st, const b2c_ncp_params *p, b2c_stream s)
{
    if (!ncp_scene_ok(sc, st) || !p) {
        b2c::set_error("b2c_ncp_color: bad argument");
        return B2C_EARG;
    }
    return sc->dtype == 4 ? b2c::ncp::color<float>(sc, st, p, b2c::stream_of(s))
                          : b2c::ncp::color<double>(sc, st, p, b2c::stream_of(s));
}

extern "C" int32_t b2c_ncp_sweeps(const b2c_ncp_scene *sc, b2c_ncp_state *st, const b2c_ncp_params *p,
                                  int32_t iters, b2c_stream s)
{
    if (!ncp_scene_ok(sc, st) || !p || iters < 0) {
        b2c::set_error("b2c_ncp_sweeps: bad argument");
        return B2C_EARG;
    }
    return sc->dtype == 4 ? b2c::ncp::sweeps<float>(sc, st, p, iters, b2c::stream_of(s))
                          : b2c::ncp::sweeps<double>(sc, st, p, iters, b2c::stream_of(s));
}

extern "C" int32_t b2c_ncp_residual(const b2c_ncp_scene *sc, b2c_ncp_state *st, const b2c_ncp_params *p,
                                    b2c_stream s)
{
    if (!ncp_scene_ok(sc, st) || !p) {
        b2c::set_error("b2c_ncp_residual: bad argument");
        return B2C_EARG;
    }
    return sc->dtype == 4 ? b2c::ncp::residual<float>(sc, st, p, b2c::stream_of(s))
                          : b2c::ncp::residual<double>(sc, st, p, b2c::stream_of(s));
}

extern "C" int32_t b2c_ncp_adjoint(const b2c_ncp_scene *sc, b2c_ncp_state *st, const b2c_ncp_params *p,
                                   int32_t iters, double *lam_bar, double *v_bar, double *vfree_bar, double *bias_bar,
                                   double *mu_bar, b2c_stream s)
{
    if (!ncp_scene_ok(sc, st) || !p || sc->dtype != 8 || iters < 0 || !v_bar || !vfree_bar || p->soft ||
        (sc->n_c > 0 && (!lam_bar || !bias_bar || !mu_bar))) {
        b2c::set_error("b2c_ncp_adjoint: bad argument (float64 scenes only)");
        return B2C_EARG;
    }
    return b2c::ncp::adjoint_sweeps(sc, st, p, iters, nullptr, lam_bar, v_bar, vfree_bar, bias_bar, mu_bar, nullptr,
                                    nullptr, nullptr, b2c::stream_of(s));
}

extern "C" int32_t b2c_ncp_trace_words(void) { return b2c::ncp::kTraceWords; }

extern "C" int32_t b2c_ncp_sweeps_record(const b2c_ncp_scene *sc, b2c_ncp_state *st, const b2c_ncp_params *p,
                                         int32_t iters, double *trace, int64_t trace_len, b2c_stream s)
{
    if (!ncp_scene_ok(sc, st) || !p || sc->dtype != 8 || iters < 0 ||
        (sc->n_c > 0 && iters > 0 && (!trace || trace_len < b2c::ncp::kTraceWords * (int64_t)iters * sc->n_c))) {
        b2c::set_error("b2c_ncp_sweeps_record: bad argument (float64 scenes; trace of b2c_ncp_trace_words() * iters * n_c doubles)");
        return B2C_EARG;
    }
    return b2c::ncp::sweeps<double>(sc, st, p, iters, b2c::stream_of(s), trace);
}

extern "C" int32_t b2c_ncp_adjoint_unrolled(const b2c_ncp_scene *sc, b2c_ncp_state *st, const b2c_ncp_params *p,
                                            int32_t iters, double *trace, int64_t trace_len, double *lam_bar,
                                            double *v_bar, double *vfree_bar, double *bias_bar, double *mu_bar,
                                            double *Ja_bar, double *Jb_bar, double *Minv_bar, b2c_stream s)
{
    if (!ncp_scene_ok(sc, st) || !p || sc->dtype != 8 || iters < 0 || !v_bar || !vfree_bar || p->soft ||
        (sc->n_c > 0 && (!lam_bar || !bias_bar || !mu_bar || !Ja_bar || !Jb_bar || !Minv_bar)) ||
        (sc->n_c > 0 && iters > 0 && (!trace || trace_len < b2c::ncp::kTraceWords * (int64_t)iters * sc->n_c))) {
        b2c::set_error("b2c_ncp_adjoint_unrolled: bad argument (float64 hard-contact scenes; the trace of "
                       "b2c_ncp_sweeps_record)");
        return B2C_EARG;
    }
    return b2c::ncp::adjoint_sweeps(sc, st, p, iters, trace, lam_bar, v_bar, vfree_bar, bias_bar, mu_bar, Ja_bar,
                                    Jb_bar, Minv_bar, b2c::stream_of(s));
}
