// Batched, level-synchronous AMG-PCG for the Poisson projection.
//
// A program may hold many independent instances (a batch); each one keeps its
// own Krylov scalars and convergence test, so its result does not depend on the
// other instances it shares the launches with.  Every kernel covers all
// instances of one multigrid level at once: rows are concatenated instance by
// instance per level, and a table of blocks (Blk) maps each CTA to a row range
// of exactly one instance.  That gives
//   - full-device launches even when single instances are small, and
//   - per-instance reductions without atomics on data: each CTA writes its
//     partial sums, the last CTA of an instance to arrive adds the instance's
//     partials in block order (the same order on every run) and updates the
//     instance's scalars.
// Converged instances are skipped block by block.
//
// One CG iteration (hig-flow-step.c:48-131 solves the same system with PETSc's
// KSP; the operator here is the reduced, negated SPD form built on the host):
//   V-cycle  down: x = w D^-1 b, r = b - A x, b_next = R r     (per level)
//            coarsest: x = inv b per instance (dense)
//            up:   x += P e, out = x + w D^-1 (b - A x)         (per level)
//   z        finest post-smoothing writes z, r.z -> beta
//   dir      p = z + beta p_old, q = A p, p.q -> alpha
//   update   x += alpha p, r -= alpha q, r.r -> convergence
// Precision: the CG recurrences and the finest operator are always FP64; the
// mixed form runs the V-cycle (a preconditioner only needs a few digits) on
// FP32 copies of the hierarchy, halving its bytes.
//
// The iterations of a step run inside a CUDA graph as a conditional WHILE node;
// the last CTA of the second update kernel of each loop body sets the condition
// (any instance still active and the body cap not reached), so a whole time
// step is one graph launch with no host round trip.
#pragma once

#include <cstdint>

constexpr int kMaxLevels = 16;       // multigrid levels including the finest
// mixed form: inner FP32 sweeps per solve, each to eta times the FP64 residual
// it starts from (FP32 CG reaches about 1e-6 of its start), at most
// kInnerMaxit iterations
constexpr int kMaxSweeps = 4;
constexpr double kInnerEta = 1e-5;
constexpr int kInnerMaxit = 60;
constexpr int kMaxCoarse = 128;      // rows of the coarsest level (dense inverse)
constexpr int kCoarseCap = 1024;     // largest coarsest level accepted (stalled coarsening)

// Every level-synchronous kernel gives each thread kRPT rows of its block
// (rows row0 + threadIdx.x + q * kBlock): their independent load chains
// overlap, and a block's fixed costs (descriptor, reduction) are shared.
constexpr int kRPT = 4;
constexpr int kBlockRows = kBlock * kRPT;

// Programmatic dependent launch: the kernels of the CG loop body are launched
// with programmatic stream serialization, so a kernel's grid is scheduled
// while its predecessor's last blocks finish.  Each waits here, before its
// first access to device memory, until the predecessor grid has completed
// and its writes are visible (a no-op for a plain launch).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// rows [row0, row0 + cnt) of instance inst at one level (cnt <= kBlockRows);
// first/nblk: the instance's block range in the same table (for reductions).
// On the finest level pad0 <= 0 <= pad1 are the lowest and highest column
// offsets the block's rows reach (its halo).
struct Blk {
    int32_t row0, cnt, inst, first, nblk, pad0, pad1, pad2;
};

// A finest-level kernel that applies the operator to a vector it derives per
// row (p = z + beta p_old) stages that vector over the block's rows and halo in
// shared memory when the span fits: each value is then loaded and formed once
// per block instead of once per referencing row.
constexpr int kStageRows = kBlockRows + 1024;

// Krylov state of one instance
struct IScal {
    double rz, alpha, beta, rr, bb, tol2;
    int32_t iters, status, done, tail0;  // tail0: the whole V-cycle is the tail (s = 0)
    uint32_t counter, pad;
    int64_t total_iters;
    // mixed form (FP32 inner CG inside FP64 refinement): the inner sweep's
    // target, sweeps done, inner iterations of the step's earlier sweeps, and
    // fin = the FP64 residual met the target (or the solve failed)
    double tol2in;
    int32_t outer, iters_prev, fin;
    // under step limits: the instance's first failed step's status (sticky;
    // the instance is frozen from that step on)
    int32_t failed;
};

// loop control and error record of the whole case
struct Ctl {
    int32_t active;       // instances not converged in the running step
    int32_t bodies;       // loop bodies run in the running step
    uint32_t gcount;      // blocks arrived at the last update kernel of a body
    int32_t maxbodies;
    int32_t err_status, err_inst;
    int64_t err_step;
    int64_t step;         // steps completed
    int64_t total_bodies;
    int32_t hist, pad;    // earlier solutions the initial guess can use (0..2)
};

// The finest operator as row templates: row i applies the template described
// by rd[i] = (first entry << kTLenBits) | entry count, whose entries are
// (column offset toff[k], value tval[k]).  On a uniform grid a handful of
// templates per instance cover every row, so a row costs one 4-byte word
// instead of its CSR columns and values (and one dependent load less than a
// template index would).
constexpr int kTLenBits = 7;   // rows of up to 127 entries (AMR interface rows reach 75), 2^25 entries

template <typename T>
struct TRows {
    const uint32_t *rd;
    const int32_t *toff;
    const T *tval;
};

// sum over row i of val_k * f(i + off_k), in the row's entry order
template <typename T, typename Fn>
__device__ __forceinline__ T trow(const TRows<T> &A, int i, Fn f)
{
    const uint32_t d = __ldg(A.rd + i);
    const int k0 = (int)(d >> kTLenBits), e = k0 + (int)(d & ((1u << kTLenBits) - 1));
    T s = T(0);
    for (int k = k0; k < e; k++) s += __ldg(A.tval + k) * f(i + __ldg(A.toff + k));
    return s;
}

// Rows of a transfer operator (prolongation or restriction) as templates
// anchored at a per-row column: rb[i] = (descriptor as in TRows, anchor), the
// entries' columns are anchor + toff[k].  Smoothed aggregation on a uniform
// grid repeats a few tens of row patterns per level, so a row costs 8 bytes
// instead of 8 per entry.
template <typename T>
struct BRows {
    const uint2 *rb;
    const int32_t *toff;
    const T *tval;
};

// trow with the row's descriptor already loaded (kernels load the descriptors
// of all their rows up front, as independent loads)
template <typename T, typename Fn>
__device__ __forceinline__ T trow_d(const TRows<T> &A, uint32_t d, int i, Fn f)
{
    const int k0 = (int)(d >> kTLenBits), e = k0 + (int)(d & ((1u << kTLenBits) - 1));
    T s = T(0);
    for (int k = k0; k < e; k++) s += __ldg(A.tval + k) * f(i + __ldg(A.toff + k));
    return s;
}

template <typename T, typename Fn>
__device__ __forceinline__ T brow(const BRows<T> &A, int i, Fn f)
{
    const uint2 d = __ldg(A.rb + i);
    const int k0 = (int)(d.x >> kTLenBits), e = k0 + (int)(d.x & ((1u << kTLenBits) - 1));
    const int a = (int)d.y;
    T s = T(0);
    for (int k = k0; k < e; k++) s += __ldg(A.tval + k) * f(a + __ldg(A.toff + k));
    return s;
}


// The level-synchronous kernels read the operator and the transfers of a
// level as templates (At, Pt, Rt) when the level has them; the per-instance
// tails read the CSR form (the same entries in the same order, so both give
// the same sums).
template <typename T>
struct VLev {
    int n;
    const int32_t *Ap, *Ac;   // CSR on the coarse levels (the finest level has At only)
    const T *Av, *dinv;
    TRows<T> At;
    const int32_t *Pp, *Pc;   // rows: this level, columns: next level
    const T *Pv;
    const int32_t *Rp, *Rc;   // rows: next level, columns: this level
    const T *Rv;
    BRows<T> Pt, Rt;
    T *b, *x, *r, *out;       // b unused on the finest level (the CG residual is)
    const Blk *sblk, *ablk;   // smoothed instances' rows / all rows of the level
    int nsblk, nablk;
};

// The small levels of one instance, from the first level with at most
// kTailRows rows (s) down to its coarsest (clev, dense inverse), run by one
// CTA: phases separated by __syncthreads instead of kernel launches.
// 256 rows: a tail phase is then at most one row per thread, so the tail's
// dependent load chains stay short; larger levels run level-synchronously
// (measured on the batched cavities: taking levels of up to 2048 rows into
// the tail saves four launches per CG iteration but doubles the tail's time,
// 2.74 against 2.68 ms of Poisson iterations per step; run by an 8-CTA
// cluster per instance with a fence and a cluster barrier between phases,
// the tail took 43 against 20 us and the step 15 % longer)
constexpr int kTailRows = 256;
constexpr int kTailThreads = 512;

template <typename T>
struct TailInst {
    const T *inv;             // row-major cn x cn, cn = nrow[clev]
    int32_t inst, s, clev, pad;
    int32_t row0[kMaxLevels], nrow[kMaxLevels];   // the instance's rows on each level
};

struct PcgFine {
    int n;
    TRows<double> A;
    const double *dinv, *apin, *brhs;
    const int32_t *ipin;      // per instance: pinned global row or -1
    const hf_params *ipar;
    double *p, *dp;           // unknown: dp (incremental projection) or p
    double *xprev, *xprev2;   // the unknown of the steps before (initial-guess extrapolation)
    double *xw;               // the one-launch solve's initial guess (k_pcg_init), null otherwise
    const int32_t *cinst;     // cell -> instance
    double *r, *z, *q;
    double *partials;
    IScal *S;
    Ctl *ctl;
    const Blk *blk;
    int nblk, ninst;
    int projtype_all;         // the projection type of every instance, or -1
    double rtol, atol;
    int maxit;
    // mixed form: the inner solve of A e = r in FP32 (operator, vectors and
    // V-cycle), e applied to the FP64 unknown and r updated in FP64 after
    // each sweep (k_ir_correct); r32 is null in the plain form
    TRows<float> A32;
    float *r32, *z32, *q32, *e32;
    // per-instance step limits (DevProg::ilim): a frozen instance (0 steps
    // left) takes no part in the step's solve; null when no limits are set
    int64_t *ilim;
    double eta;               // inner sweep target: ||r_in|| <= eta ||r|| (or the outer target)
    int inner_maxit;          // iterations per inner sweep
};

// The smoothing sweeps use each level's dinv array already scaled by the
// level's damped-Jacobi weight (omega_l D^-1, per instance; hf_amg.cuh).

namespace pcg {

template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double (*sh)[kBlock / 32])
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; k++) {
        double x = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) sh[k][wid] = x;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; k++) {
        double x = threadIdx.x < kBlock / 32 ? sh[k][threadIdx.x] : 0.0;
        if (wid == 0) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        }
        v[k] = x;   // valid in thread 0
    }
    __syncthreads();
}

// Per-instance sums: true in every thread of the instance's last block, with
// tot[] the instance totals (partials added in block order).
template <int NV>
__device__ bool inst_sum(double (&v)[NV], const Blk &B, double *partials, IScal *S, double (&tot)[NV])
{
    __shared__ double sh[NV][kBlock / 32];
    __shared__ bool last;
    block_sum<NV>(v, sh);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < NV; k++) partials[(size_t)blockIdx.x * NV + k] = v[k];
        __threadfence();
        const unsigned t = atomicAdd(&S[B.inst].counter, 1u);
        last = (t == (unsigned)B.nblk - 1);
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double acc[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) acc[k] = 0.0;
    for (int b = threadIdx.x; b < B.nblk; b += kBlock) {
#pragma unroll
        for (int k = 0; k < NV; k++) acc[k] += ((volatile double *)partials)[(size_t)(B.first + b) * NV + k];
    }
    block_sum<NV>(acc, sh);
    __shared__ double bc[NV];
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < NV; k++) bc[k] = acc[k];
        S[B.inst].counter = 0;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; k++) tot[k] = bc[k];
    return true;
}

// block descriptor and the instance's done flag, shared by the block
// (split: grid blocks per table entry)
__device__ __forceinline__ bool load_blk(const Blk *tab, const IScal *S, Blk &B, int split = 1)
{
    __shared__ Blk sb;
    __shared__ int sd;
    if (threadIdx.x == 0) {
        sb = tab[blockIdx.x / split];
        sd = ((volatile const IScal *)S)[sb.inst].done;
    }
    __syncthreads();
    B = sb;
    return sd != 0;
}

__device__ __forceinline__ void finish_instance(IScal &s, Ctl *ctl)
{
    s.done = 1;
    atomicSub(&ctl->active, 1);
}

// The rows of one thread in a level-synchronous kernel: row q is
// row0 + threadIdx.x + q * kBlock, present for q < nrow.
struct RowSet {
    int row[kRPT];
    int nrow;
};

__device__ __forceinline__ RowSet rowset(const Blk &B)
{
    RowSet R;
    const int left = B.cnt - (int)threadIdx.x;
    R.nrow = left <= 0 ? 0 : min(kRPT, (left + kBlock - 1) / kBlock);
#pragma unroll
    for (int q = 0; q < kRPT; q++) R.row[q] = B.row0 + (int)threadIdx.x + q * kBlock;
    return R;
}

// The row descriptors of a thread's rows (row0 + threadIdx.x + q * kBlock),
// loaded together before any row is evaluated; absent rows (or no table) get 0
template <typename D>
__device__ __forceinline__ void row_descs(const D *tab, const Blk &B, D (&d)[kRPT])
{
#pragma unroll
    for (int q = 0; q < kRPT; q++) {
        const int t = (int)threadIdx.x + q * kBlock;
        d[q] = tab && t < B.cnt ? __ldg(tab + B.row0 + t) : D{};
    }
}

// Row sums of a thread's rows, entry k of every row before entry k + 1: the
// rows' gathers are independent loads in flight together, and each row still
// adds its entries in its own order (the sums equal trow's / brow's).  Faster
// than one row after the other on the prolongation and the finest
// post-smoothing; slower on the long restriction rows and on the kernels with
// two gathers per entry, which keep the per-row loop.
template <typename T, typename Fn>
__device__ __forceinline__ void rows_lockstep(const T *__restrict__ tval, const int32_t *__restrict__ toff,
                                              const uint32_t (&d)[kRPT], const int (&a)[kRPT], T (&s)[kRPT], Fn f)
{
    int k0[kRPT], len[kRPT], maxlen = 0;
#pragma unroll
    for (int q = 0; q < kRPT; q++) {
        k0[q] = (int)(d[q] >> kTLenBits);
        len[q] = (int)(d[q] & ((1u << kTLenBits) - 1));
        maxlen = max(maxlen, len[q]);
        s[q] = T(0);
    }
    for (int k = 0; k < maxlen; k++) {
#pragma unroll
        for (int q = 0; q < kRPT; q++)
            if (k < len[q]) s[q] += __ldg(tval + k0[q] + k) * f(a[q] + __ldg(toff + k0[q] + k));
    }
}

template <typename T, typename Fn>
__device__ __forceinline__ void trows(const TRows<T> &A, const RowSet &R, T (&s)[kRPT], Fn f)
{
    uint32_t d[kRPT];
#pragma unroll
    for (int q = 0; q < kRPT; q++) d[q] = q < R.nrow ? __ldg(A.rd + R.row[q]) : 0u;
    rows_lockstep(A.tval, A.toff, d, R.row, s, f);
}

template <typename T, typename Fn>
__device__ __forceinline__ void brows(const BRows<T> &A, const RowSet &R, T (&s)[kRPT], Fn f)
{
    uint32_t d[kRPT];
    int a[kRPT];
#pragma unroll
    for (int q = 0; q < kRPT; q++) {
        const uint2 v = q < R.nrow ? __ldg(A.rb + R.row[q]) : make_uint2(0u, 0u);
        d[q] = v.x;
        a[q] = (int)v.y;
    }
    rows_lockstep(A.tval, A.toff, d, a, s, f);
}

// CSR row sums (the per-instance tails' levels, and levels without templates)
template <typename T, typename Fn>
__device__ __forceinline__ void csr_rows(const int32_t *__restrict__ ptr, const int32_t *__restrict__ col,
                                         const T *__restrict__ val, const RowSet &R, T (&s)[kRPT], Fn f)
{
#pragma unroll
    for (int q = 0; q < kRPT; q++) {
        s[q] = T(0);
        if (q < R.nrow)
            for (int k = ptr[R.row[q]]; k < ptr[R.row[q] + 1]; k++) s[q] += val[k] * f(col[k]);
    }
}

}  // namespace pcg

// Initial guess of the step's solve: extrapolation in time of the unknown from
// the solutions of the steps before (x_n is the previous step's solution, the
// reference's own initial guess, solver-petsc.c:386-399): quadratic,
// x0 = 3 x_n - 3 x_{n-1} + x_{n-2}, once two earlier solutions are known,
// linear, 2 x_n - x_{n-1}, with one, x_n with none (Ctl::hist counts them;
// a restart clears it).  The solution is the same to the solve's tolerance;
// the extrapolated start is closer to it, so fewer iterations are needed.
__device__ __forceinline__ double extrapolated(int hist, double xn, double x1, double x2)
{
    return hist >= 2 ? 3.0 * xn - 3.0 * x1 + x2 : hist == 1 ? 2.0 * xn - x1 : xn;
}

// divergence right-hand side of every instance and the first residual
// (higflow_pressure, hig-flow-step.c:58-120, with the instance's own dt and pin).
// EXT: the initial guess too, formed at every entry's column from the unknown
// and its history, and written to xw (the one-launch solve shifts the history:
// a launch of its own for that, k_pcg_extrapolate, costs 6 us of a step)
template <int D, bool EXT>
__global__ void __launch_bounds__(kBlock) k_pcg_init(DevProg P, DevFields F, PcgFine G)
{
    // (the one-launch solve loads its tables meanwhile)
    if (EXT) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    Blk B;
    pcg::load_blk(G.blk, G.S, B);   // a new solve: the done flags are reset here
    // a frozen instance keeps done (and fin) from its last solve
    if (G.ilim && G.ilim[B.inst] == 0) return;
    const hf_params &par = G.ipar[B.inst];
    const bool incr = par.projtype == HF_INCREMENTAL;
    const double *x = incr ? G.dp : G.p;
    const int pin = G.ipin[B.inst];
    const double pinv = pin >= 0 ? (incr ? P.ipinv[B.inst] - F.p[pin] : P.ipinv[B.inst]) : 0.0;
    const int n = P.ncell;
    const int hist = EXT ? __ldg(&G.ctl->hist) : 0;
    auto guess = [&](int j) { return EXT ? extrapolated(hist, x[j], G.xprev[j], G.xprev2[j]) : x[j]; };
    double part[2] = {0.0, 0.0};   // r.r, b.b
#pragma unroll
    for (int q = 0; q < kRPT; q++) {
        const int t = threadIdx.x + q * kBlock;
        if (t >= B.cnt) break;
        const int cc = B.row0 + t;
        double borig;
        if (cc == pin) {
            borig = pinv;
        } else {
            const double *cd = P.delta + (size_t)__ldg(P.cdelta + cc) * D;
            double sumdudx = 0.0;
#pragma unroll
            for (int dim = 0; dim < D; dim++) {
                const double ustarl = hf::query(P.rows, __ldg(P.dslots + (size_t)HF_P_UL(dim) * n + cc), F.us[dim]);
                const double ustarr = hf::query(P.rows, __ldg(P.dslots + (size_t)HF_P_UR(dim) * n + cc), F.us[dim]);
                sumdudx += (ustarr - ustarl) / (2.0 * 0.5 * cd[dim]);
            }
            borig = sumdudx / par.dt + G.brhs[cc];
        }
        const double bred = cc == pin ? pinv : -(borig - G.apin[cc] * pinv);
        const double ax = trow(G.A, cc, guess);
        if (EXT) G.xw[cc] = guess(cc);
        const double r = bred - ax;
        G.r[cc] = r;
        if (G.r32) {
            G.r32[cc] = (float)r;
            G.e32[cc] = 0.f;
        }
        part[0] += r * r;
        part[1] += borig * borig;
    }
    double tot[2];
    if (pcg::inst_sum<2>(part, B, G.partials, G.S, tot) && threadIdx.x == 0) {
        IScal &s = G.S[B.inst];
        s.rr = tot[0];
        s.bb = tot[1];
        const double t = fmax(G.rtol * sqrt(tot[1]), G.atol);
        s.tol2 = t * t;
        // the inner sweep aims at the outer target, or eta of where it starts
        s.tol2in = G.r32 ? fmax(s.tol2, G.eta * G.eta * tot[0]) : s.tol2;
        s.outer = 0;
        s.iters_prev = 0;
        s.fin = 0;
        s.beta = 0.0;
        s.iters = 0;
        s.status = 0;
        s.done = !(tot[0] > s.tol2);
        if (!isfinite(tot[0]) || !isfinite(tot[1])) { s.status = HF_ERR_NAN; s.done = 1; }
        if (!s.done) atomicAdd(&G.ctl->active, 1);
    }
}

// x = w D^-1 b ; r = b - A x on the smoothed rows of one level
template <typename T, bool FINE, typename R = double>
__global__ void __launch_bounds__(kBlock) k_vc_down(VLev<T> L, const R *__restrict__ r0, const IScal *S)
{
    pdl_wait();
    Blk B;
    if (pcg::load_blk(L.sblk, S, B)) return;
    // (the finest level's descriptors up front: faster there, slower on the
    // coarse levels)
    uint32_t d[kRPT];
    if (FINE) pcg::row_descs(L.At.rd, B, d);
#pragma unroll
    for (int q = 0; q < kRPT; q++) {
        const int t = threadIdx.x + q * kBlock;
        if (t >= B.cnt) break;
        const int i = B.row0 + t;
        const T bi = FINE ? T(r0[i]) : L.b[i];
        T s = T(0);
        if (FINE) {
            s = trow_d(L.At, d[q], i, [&](int j) { return __ldg(L.dinv + j) * T(__ldg(r0 + j)); });
        } else if (L.At.rd) {
            s = trow(L.At, i, [&](int j) { return L.dinv[j] * L.b[j]; });
        } else {
            for (int k = L.Ap[i]; k < L.Ap[i + 1]; k++) {
                const int j = L.Ac[k];
                s += L.Av[k] * (L.dinv[j] * L.b[j]);
            }
        }
        L.x[i] = L.dinv[i] * bi;
        L.r[i] = bi - s;
    }
}

// b_next = R r on every row of the next level
template <typename T>
__global__ void __launch_bounds__(kBlock) k_vc_restrict(VLev<T> L, VLev<T> Ln, const IScal *S)
{
    pdl_wait();
    Blk B;
    if (pcg::load_blk(Ln.ablk, S, B)) return;
#pragma unroll
    for (int q = 0; q < kRPT; q++) {
        const int t = threadIdx.x + q * kBlock;
        if (t >= B.cnt) break;
        const int i = B.row0 + t;
        T s = T(0);
        if (L.Rt.rb) s = brow(L.Rt, i, [&](int j) { return L.r[j]; });
        else
            for (int k = L.Rp[i]; k < L.Rp[i + 1]; k++) s += L.Rv[k] * L.r[L.Rc[k]];
        Ln.b[i] = s;
    }
}

// The V-cycle of one instance from its tail level s down to its coarsest level
// and back, one CTA per instance (H: the level table in device memory; levels
// are copied to shared memory one at a time, a dynamic index into the kernel
// parameters would spill them).  Level s's b is the regular restriction's
// output (or the CG residual when s is the finest level); level s's out is the
// correction the regular prolongation reads.  Same arithmetic as the
// level-synchronous kernels; the dense solve splits each row over a warp.
template <typename T, typename R = double>
__global__ void __launch_bounds__(kTailThreads) k_vc_tail(const VLev<T> *H, const TailInst<T> *TI,
                                                        const R *__restrict__ r0, const IScal *S)
{
    pdl_wait();
    __shared__ TailInst<T> ti;
    __shared__ VLev<T> L, Ln;
    __shared__ int done;
    __shared__ T sb[kCoarseCap];
    if (threadIdx.x == 0) {
        ti = TI[blockIdx.x];
        done = ((volatile const IScal *)S)[ti.inst].done;
    }
    __syncthreads();
    if (done) return;
    const int tid = threadIdx.x;
    // down: x = w D^-1 b, r = b - A x, b_next = R r
    for (int l = ti.s; l < ti.clev; l++) {
        if (tid == 0) {
            L = H[l];
            Ln = H[l + 1];
        }
        __syncthreads();
        const int a = ti.row0[l], e = a + ti.nrow[l];
        for (int i = a + tid; i < e; i += kTailThreads) {
            T bi, s = T(0);
            if (l == 0) {
                bi = T(r0[i]);
                s = trow(L.At, i, [&](int j) { return __ldg(L.dinv + j) * T(__ldg(r0 + j)); });
            } else {
                bi = L.b[i];
                for (int k = L.Ap[i]; k < L.Ap[i + 1]; k++) {
                    const int j = L.Ac[k];
                    s += L.Av[k] * (L.dinv[j] * L.b[j]);
                }
            }
            L.x[i] = L.dinv[i] * bi;
            L.r[i] = bi - s;
        }
        __syncthreads();
        const int an = ti.row0[l + 1], en = an + ti.nrow[l + 1];
        for (int i = an + tid; i < en; i += kTailThreads) {
            T s = T(0);
            for (int k = L.Rp[i]; k < L.Rp[i + 1]; k++) s += L.Rv[k] * L.r[L.Rc[k]];
            Ln.b[i] = s;
        }
        __syncthreads();
    }
    // coarsest: out = inv b, one warp per row, lanes over the row
    {
        if (tid == 0) L = H[ti.clev];
        __syncthreads();
        const int a = ti.row0[ti.clev], cn = ti.nrow[ti.clev];
        for (int i = tid; i < cn; i += kTailThreads) sb[i] = ti.clev == 0 ? T(r0[a + i]) : L.b[a + i];
        __syncthreads();
        const int lane = tid & 31, warp = tid >> 5;
        for (int i = warp; i < cn; i += kTailThreads / 32) {
            const T *row = ti.inv + (size_t)i * cn;
            T s = T(0);
            for (int k = lane; k < cn; k += 32) s += row[k] * sb[k];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) L.out[a + i] = s;
        }
        __syncthreads();
    }
    // up: x += P e, out = x + w D^-1 (b - A x)
    for (int l = ti.clev - 1; l >= ti.s; l--) {
        if (tid == 0) {
            L = H[l];
            Ln = H[l + 1];
        }
        __syncthreads();
        const int a = ti.row0[l], e = a + ti.nrow[l];
        for (int i = a + tid; i < e; i += kTailThreads) {
            T s = T(0);
            for (int k = L.Pp[i]; k < L.Pp[i + 1]; k++) s += L.Pv[k] * Ln.out[L.Pc[k]];
            L.x[i] += s;
        }
        __syncthreads();
        for (int i = a + tid; i < e; i += kTailThreads) {
            T bi, s;
            if (l == 0) {
                bi = T(r0[i]);
                s = trow(L.At, i, [&](int j) { return L.x[j]; });
            } else {
                bi = L.b[i];
                s = T(0);
                for (int k = L.Ap[i]; k < L.Ap[i + 1]; k++) s += L.Av[k] * L.x[L.Ac[k]];
            }
            L.out[i] = L.x[i] + L.dinv[i] * (bi - s);
        }
        __syncthreads();
    }
}

// x += P e on the smoothed rows (e: the next level's correction)
template <typename T>
__global__ void __launch_bounds__(kBlock) k_vc_prolong(VLev<T> L, const T *__restrict__ e, const IScal *S)
{
    pdl_wait();
    Blk B;
    if (pcg::load_blk(L.sblk, S, B)) return;
    const pcg::RowSet R = pcg::rowset(B);
    T s[kRPT];
    if (L.Pt.rb) pcg::brows(L.Pt, R, s, [&](int j) { return e[j]; });
    else pcg::csr_rows(L.Pp, L.Pc, L.Pv, R, s, [&](int j) { return e[j]; });
#pragma unroll
    for (int q = 0; q < kRPT; q++)
        if (q < R.nrow) L.x[R.row[q]] += s[q];
}

// out = x + w D^-1 (b - A x) on the smoothed rows of a coarse level
template <typename T>
__global__ void __launch_bounds__(kBlock) k_vc_post(VLev<T> L, const IScal *S)
{
    pdl_wait();
    Blk B;
    if (pcg::load_blk(L.sblk, S, B)) return;
#pragma unroll
    for (int q = 0; q < kRPT; q++) {
        const int t = threadIdx.x + q * kBlock;
        if (t >= B.cnt) break;
        const int i = B.row0 + t;
        T s = T(0);
        if (L.At.rd) s = trow(L.At, i, [&](int j) { return L.x[j]; });
        else
            for (int k = L.Ap[i]; k < L.Ap[i + 1]; k++) s += L.Av[k] * L.x[L.Ac[k]];
        L.out[i] = L.x[i] + L.dinv[i] * (L.b[i] - s);
    }
}

// ---------------------------------------------------------------------------
// the folded V-cycle (hf_solve.cuh states its operators): one kernel per level
// down, b_{l+1} = Rt b_l, and one up, out_l = Mt b_l + Pt out_{l+1}, in place of
// smoothing, residual, transfer and smoothing again.  A level's At, Pt, Rt and
// CSR arrays then hold Mt, Pt and Rt (the finest level's At: Mt).  What bounds
// the loop on one large instance is the number of its launches: 9 instead of 20
// per iteration on 512 x 512 cells
// ---------------------------------------------------------------------------
// b_next = Rt b on every row of the next level (src: the level's b, the CG
// residual on the finest)
constexpr int kFoldSplit = 4;
template <typename T, typename R = T>
__global__ void __launch_bounds__(kBlock) k_vf_down(VLev<T> L, VLev<T> Ln, const R *src, const IScal *S)
{
    pdl_wait();
    Blk B;
    if (pcg::load_blk(Ln.ablk, S, B, kFoldSplit)) return;
    // four threads per row: the rows are long (27 entries in 2D, 70 in 3D) and
    // few; kFoldSplit grid blocks share a block's rows, so that a thread sums one
    // row of a level of one row per thread
    const int g = threadIdx.x >> 2, lane = threadIdx.x & 3;
    const int per = (B.cnt + kFoldSplit - 1) / kFoldSplit, lo = (int)(blockIdx.x % kFoldSplit) * per, hi = min(B.cnt, lo + per);
    for (int b = lo; b < hi; b += kBlock / 4) {
        const int t = b + g;
        T s = T(0);
        if (t < hi) {
            const int i = B.row0 + t;
            if (L.Rt.rb) {
                const uint2 d = __ldg(L.Rt.rb + i);
                const int k0 = (int)(d.x >> kTLenBits), e = k0 + (int)(d.x & ((1u << kTLenBits) - 1)), a = (int)d.y;
#pragma unroll 8
                for (int k = k0 + lane; k < e; k += 4) s += __ldg(L.Rt.tval + k) * T(src[a + __ldg(L.Rt.toff + k)]);
            } else {
                const int e = L.Rp[i + 1];
#pragma unroll 8
                for (int k = L.Rp[i] + lane; k < e; k += 4) s += __ldg(L.Rv + k) * T(src[__ldg(L.Rc + k)]);
            }
        }
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        if (t < hi && lane == 0) Ln.b[B.row0 + t] = s;
    }
}

// Mt b + Pt e on a thread's rows
template <typename T, typename Fn>
__device__ __forceinline__ void folded_up(const VLev<T> &L, const pcg::RowSet &R, const T *e, T (&s)[kRPT], Fn b)
{
    // (unrolled by eight, so that the loads of several entries are in flight: as
    // many as the 32 registers a thread that ptxas takes here can hold, fewer than
    // eight in FP64, where k_vf_z spills 36 bytes)
#pragma unroll
    for (int q = 0; q < kRPT; q++) {
        s[q] = T(0);
        if (q >= R.nrow) continue;
        const int i = R.row[q];
        T u = T(0), v = T(0);
        if (L.At.rd) {
            const uint32_t d = __ldg(L.At.rd + i);
            const int k0 = (int)(d >> kTLenBits), n = (int)(d & ((1u << kTLenBits) - 1));
#pragma unroll 8
            for (int k = 0; k < n; k++) u += __ldg(L.At.tval + k0 + k) * b(i + __ldg(L.At.toff + k0 + k));
        } else {
            const int n = L.Ap[i + 1];
#pragma unroll 8
            for (int k = L.Ap[i]; k < n; k++) u += __ldg(L.Av + k) * b(__ldg(L.Ac + k));
        }
        if (L.Pt.rb) {
            const uint2 d = __ldg(L.Pt.rb + i);
            const int k0 = (int)(d.x >> kTLenBits), n = (int)(d.x & ((1u << kTLenBits) - 1)), a = (int)d.y;
#pragma unroll 8
            for (int k = 0; k < n; k++) v += __ldg(L.Pt.tval + k0 + k) * e[a + __ldg(L.Pt.toff + k0 + k)];
        } else {
            const int n = L.Pp[i + 1];
#pragma unroll 8
            for (int k = L.Pp[i]; k < n; k++) v += __ldg(L.Pv + k) * e[__ldg(L.Pc + k)];
        }
        s[q] = u + v;
    }
}

// out = Mt b + Pt e on the smoothed rows of a coarse level
template <typename T>
__global__ void __launch_bounds__(kBlock) k_vf_up(VLev<T> L, const T *e, const IScal *S)
{
    pdl_wait();
    Blk B;
    if (pcg::load_blk(L.sblk, S, B)) return;
    const pcg::RowSet R = pcg::rowset(B);
    T s[kRPT];
    folded_up(L, R, e, s, [&](int j) { return L.b[j]; });
#pragma unroll
    for (int q = 0; q < kRPT; q++)
        if (q < R.nrow) L.out[R.row[q]] = s[q];
}

// z = Mt r + Pt e on the finest level (or the tail's output), r.z -> beta per
// instance; r, z: the plain form's vectors or the mixed form's FP32 ones
template <typename T>
__global__ void __launch_bounds__(kBlock) k_vf_z(PcgFine G, VLev<T> L0, const T *e, const T *r, T *z)
{
    pdl_wait();
    Blk B;
    if (pcg::load_blk(G.blk, G.S, B)) return;
    const bool tail0 = G.S[B.inst].tail0;
    const pcg::RowSet R = pcg::rowset(B);
    T s[kRPT];
    if (!tail0) folded_up(L0, R, e, s, [&](int j) { return r[j]; });
    double part[1] = {0.0};
#pragma unroll
    for (int q = 0; q < kRPT; q++) {
        if (q >= R.nrow) break;
        const int i = R.row[q];
        const T zi = tail0 ? L0.out[i] : s[q];
        z[i] = zi;
        part[0] += (double)r[i] * (double)zi;
    }
    double tot[1];
    if (pcg::inst_sum<1>(part, B, G.partials, G.S, tot) && threadIdx.x == 0) {
        IScal &s = G.S[B.inst];
        s.beta = s.iters == 0 ? 0.0 : tot[0] / s.rz;
        s.rz = tot[0];
        if (!isfinite(tot[0])) { s.status = HF_ERR_NAN; pcg::finish_instance(s, G.ctl); }
    }
}

// the small levels of one instance, down and up, one CTA (as k_vc_tail): eight
// threads per row down, one up
constexpr int kFoldTailRows = 1024;
constexpr int kFoldTailThreads = 1024;
template <typename T>
__global__ void __launch_bounds__(kFoldTailThreads) k_vf_tail(const VLev<T> *H, const TailInst<T> *TI, const T *r0, const IScal *S)
{
    pdl_wait();
    __shared__ TailInst<T> ti;
    __shared__ VLev<T> L, Ln;
    __shared__ int done;
    __shared__ T sb[kCoarseCap];
    if (threadIdx.x == 0) {
        ti = TI[blockIdx.x];
        done = ((volatile const IScal *)S)[ti.inst].done;
    }
    __syncthreads();
    if (done) return;
    const int tid = threadIdx.x;
    for (int l = ti.s; l < ti.clev; l++) {
        if (tid == 0) {
            L = H[l];
            Ln = H[l + 1];
        }
        __syncthreads();
        const T *b = l == 0 ? r0 : L.b;
        const int a = ti.row0[l + 1], n = ti.nrow[l + 1], lane = tid & 7;
        for (int t = tid >> 3; t - (tid >> 3) < n; t += kFoldTailThreads / 8) {
            T s = T(0);
            if (t < n)
            {
                const int e = L.Rp[a + t + 1];
#pragma unroll 8
                for (int k = L.Rp[a + t] + lane; k < e; k += 8) s += __ldg(L.Rv + k) * b[__ldg(L.Rc + k)];
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (t < n && lane == 0) Ln.b[a + t] = s;
        }
        __syncthreads();
    }
    // coarsest: out = inv b, one warp per row, lanes over the row
    {
        if (tid == 0) L = H[ti.clev];
        __syncthreads();
        const int a = ti.row0[ti.clev], cn = ti.nrow[ti.clev];
        for (int i = tid; i < cn; i += kFoldTailThreads) sb[i] = ti.clev == 0 ? r0[a + i] : L.b[a + i];
        __syncthreads();
        const int lane = tid & 31, warp = tid >> 5;
        for (int i = warp; i < cn; i += kFoldTailThreads / 32) {
            const T *row = ti.inv + (size_t)i * cn;
            T s = T(0);
            for (int k = lane; k < cn; k += 32) s += row[k] * sb[k];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) L.out[a + i] = s;
        }
        __syncthreads();
    }
    for (int l = ti.clev - 1; l >= ti.s; l--) {
        if (tid == 0) {
            L = H[l];
            Ln = H[l + 1];
        }
        __syncthreads();
        const T *b = l == 0 ? r0 : L.b;
        const int a = ti.row0[l], e = a + ti.nrow[l];
        for (int i = a + tid; i < e; i += kFoldTailThreads) {
            T s = T(0);
            if (l == 0) {
                s = trow(L.At, i, [&](int j) { return b[j]; });
            } else {
                const int n = L.Ap[i + 1];
#pragma unroll 8
                for (int k = L.Ap[i]; k < n; k++) s += __ldg(L.Av + k) * b[__ldg(L.Ac + k)];
            }
            const int n = L.Pp[i + 1];
#pragma unroll 8
            for (int k = L.Pp[i]; k < n; k++) s += __ldg(L.Pv + k) * Ln.out[__ldg(L.Pc + k)];
            L.out[i] = s;
        }
        __syncthreads();
    }
}

// z on the finest level (post-smoothing, the tail's output, or D^-1 r), then
// r.z -> beta per instance
template <typename T, bool JACOBI>
__global__ void __launch_bounds__(kBlock) k_pcg_z(PcgFine G, VLev<T> L0)
{
    pdl_wait();
    Blk B;
    if (pcg::load_blk(G.blk, G.S, B)) return;
    const bool tail0 = G.S[B.inst].tail0;
    const pcg::RowSet R = pcg::rowset(B);
    T s[kRPT];
    if (!JACOBI && !tail0) pcg::trows(L0.At, R, s, [&](int j) { return L0.x[j]; });
    double part[1] = {0.0};
#pragma unroll
    for (int q = 0; q < kRPT; q++) {
        if (q >= R.nrow) break;
        const int i = R.row[q];
        const double ri = G.r[i];
        double z;
        if (JACOBI) {
            z = G.dinv[i] * ri;
        } else if (tail0) {
            z = double(L0.out[i]);
        } else {
            z = double(L0.x[i] + L0.dinv[i] * (T(ri) - s[q]));
        }
        G.z[i] = z;
        part[0] += ri * z;
    }
    double tot[1];
    if (pcg::inst_sum<1>(part, B, G.partials, G.S, tot) && threadIdx.x == 0) {
        IScal &s = G.S[B.inst];
        s.beta = s.iters == 0 ? 0.0 : tot[0] / s.rz;
        s.rz = tot[0];
        if (!isfinite(tot[0])) { s.status = HF_ERR_NAN; pcg::finish_instance(s, G.ctl); }
    }
}

// w = M^-1 v on the BiCGStab path (a non-symmetric Poisson operator: AMR
// interfaces): after the V-cycle on v, the finest level's post-smoothing
// (k_pcg_z's arithmetic, without its reduction)
__global__ void __launch_bounds__(kBlock) k_bi_amg_post(PcgFine G, VLev<double> L0, const double *__restrict__ v,
                                                     double *__restrict__ w)
{
    pdl_wait();
    Blk B;
    if (pcg::load_blk(G.blk, G.S, B)) return;
    const bool tail0 = G.S[B.inst].tail0;
    const pcg::RowSet R = pcg::rowset(B);
    double s[kRPT];
    if (!tail0) pcg::trows(L0.At, R, s, [&](int j) { return L0.x[j]; });
#pragma unroll
    for (int q = 0; q < kRPT; q++) {
        if (q >= R.nrow) break;
        const int i = R.row[q];
        w[i] = tail0 ? L0.out[i] : L0.x[i] + L0.dinv[i] * (v[i] - s[q]);
    }
}

// p_new = z + beta p_old ; q = A p_new ; alpha = r.z / p.q
__global__ void __launch_bounds__(kBlock) k_pcg_dir(PcgFine G, const double *__restrict__ po, double *__restrict__ pn)
{
    pdl_wait();
    Blk B;
    if (pcg::load_blk(G.blk, G.S, B)) return;
    const IScal &sc = G.S[B.inst];
    const bool first = sc.iters == 0;
    const double beta = sc.beta;
    uint32_t d[kRPT];
    pcg::row_descs(G.A.rd, B, d);
    __shared__ double sp[kStageRows];
    const int s0 = B.row0 + B.pad0, ns = B.cnt + B.pad1 - B.pad0;
    const bool staged = ns <= kStageRows;
    if (staged) {
        for (int j = threadIdx.x; j < ns; j += kBlock) sp[j] = first ? G.z[s0 + j] : G.z[s0 + j] + beta * po[s0 + j];
        __syncthreads();
    }
    double part[1] = {0.0};
#pragma unroll
    for (int q = 0; q < kRPT; q++) {
        const int t = threadIdx.x + q * kBlock;
        if (t >= B.cnt) break;
        const int i = B.row0 + t;
        double qi, p;
        if (staged) {
            qi = trow_d(G.A, d[q], i, [&](int j) { return sp[j - s0]; });
            p = sp[i - s0];
        } else if (first) {
            qi = trow_d(G.A, d[q], i, [&](int j) { return G.z[j]; });
            p = G.z[i];
        } else {
            qi = trow_d(G.A, d[q], i, [&](int j) { return G.z[j] + beta * po[j]; });
            p = G.z[i] + beta * po[i];
        }
        pn[i] = p;
        G.q[i] = qi;
        part[0] += p * qi;
    }
    double tot[1];
    if (pcg::inst_sum<1>(part, B, G.partials, G.S, tot) && threadIdx.x == 0) {
        IScal &s = G.S[B.inst];
        if (!(tot[0] > 0.0) || !isfinite(tot[0])) {
            // p.q <= 0: the recurrence has reached rounding level.  Accept when
            // the residual is within 100x of the target, else report it.
            s.status = !isfinite(tot[0]) ? HF_ERR_NAN : (s.rr <= 1e4 * s.tol2 ? 0 : HF_ERR_NOT_CONVERGED);
            pcg::finish_instance(s, G.ctl);
        } else {
            s.alpha = s.rz / tot[0];
        }
    }
}

// x += alpha p ; r -= alpha q ; convergence on ||r||.  set_cond != 0: the last
// block of the grid counts the loop body and (set_cond == 1, inside the step
// graph) sets the loop condition for the next body; with eager launches the
// host reads the count and the active instances instead.
__global__ void __launch_bounds__(kBlock) k_pcg_update(PcgFine G, const double *__restrict__ pn,
                                                       cudaGraphConditionalHandle cond, int set_cond)
{
    pdl_wait();
    Blk B;
    const bool skip = pcg::load_blk(G.blk, G.S, B);
    if (!skip) {
        const int pt = G.projtype_all >= 0 ? G.projtype_all : G.ipar[B.inst].projtype;
        double *x = pt == HF_INCREMENTAL ? G.dp : G.p;
        const double alpha = G.S[B.inst].alpha;
        const pcg::RowSet R = pcg::rowset(B);
        double xv[kRPT], pv[kRPT], rv[kRPT], qv[kRPT];
#pragma unroll
        for (int q = 0; q < kRPT; q++) {
            if (q < R.nrow) {
                const int i = R.row[q];
                xv[q] = x[i];
                pv[q] = pn[i];
                rv[q] = G.r[i];
                qv[q] = G.q[i];
            }
        }
        double part[1] = {0.0};
#pragma unroll
        for (int q = 0; q < kRPT; q++) {
            if (q >= R.nrow) break;
            const int i = R.row[q];
            x[i] = xv[q] + alpha * pv[q];
            const double r = rv[q] - alpha * qv[q];
            G.r[i] = r;
            part[0] += r * r;
        }
        double tot[1];
        if (pcg::inst_sum<1>(part, B, G.partials, G.S, tot) && threadIdx.x == 0) {
            IScal &s = G.S[B.inst];
            s.rr = tot[0];
            s.iters += 1;
            if (!isfinite(tot[0])) { s.status = HF_ERR_NAN; pcg::finish_instance(s, G.ctl); }
            else if (!(tot[0] > s.tol2)) pcg::finish_instance(s, G.ctl);
            else if (s.iters >= G.maxit) { s.status = HF_ERR_NOT_CONVERGED; pcg::finish_instance(s, G.ctl); }
        }
    }
    if (!set_cond) return;
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned t = atomicAdd(&G.ctl->gcount, 1u);
        if (t == gridDim.x - 1) {
            __threadfence();
            Ctl &c = *G.ctl;
            c.gcount = 0;
            c.bodies += 1;
            const int active = ((volatile Ctl *)G.ctl)->active;
            if (set_cond == 1) cudaGraphSetConditional(cond, (active > 0 && c.bodies < c.maxbodies) ? 1u : 0u);
        }
    }
}

// the level-synchronous loop's initial guess
__global__ void __launch_bounds__(kBlock) k_pcg_extrapolate(PcgFine G)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= G.n) return;
    // (the instance lookup only when the instances differ in projection
    // type: it would delay every load behind two dependent ones)
    if (G.ilim && G.ilim[__ldg(G.cinst + i)] == 0) return;
    const int pt = G.projtype_all >= 0 ? G.projtype_all : __ldg(&G.ipar[__ldg(G.cinst + i)].projtype);
    double *x = pt == HF_INCREMENTAL ? G.dp : G.p;
    const double xn = x[i], x1 = G.xprev[i], x2 = G.xprev2[i];
    // (a plain load: the history count was written by an earlier kernel)
    const int hist = __ldg(&G.ctl->hist);
    G.xprev2[i] = x1;
    G.xprev[i] = xn;
    x[i] = extrapolated(hist, xn, x1, x2);
}

// restart the time history: the next extrapolation starts from the unknown's
// current value (after the host has written the pressure or its increment)
__global__ void __launch_bounds__(kBlock) k_pcg_restart(PcgFine G)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= G.n) return;
    const int pt = G.projtype_all >= 0 ? G.projtype_all : __ldg(&G.ipar[__ldg(G.cinst + i)].projtype);
    G.xprev[i] = (pt == HF_INCREMENTAL ? G.dp : G.p)[i];
    if (i == 0) G.ctl->hist = 0;
}

// end of a step: per-instance totals, the first failure, loop counters reset.
// One block runs it, the last of the step's last kernel (k_final)
__device__ __forceinline__ void step_end(const PcgFine &G)
{
    Ctl *c = G.ctl;
    for (int i = threadIdx.x; i < G.ninst; i += kBlock) {
        IScal &s = G.S[i];
        if (G.ilim) {
            if (G.ilim[i] == 0) continue;   // frozen during this step
            if (G.ilim[i] > 0) G.ilim[i] -= 1;
        }
        // stopped by the body cap (or, mixed, by the sweep cap): not converged
        if (G.r32 ? !s.fin : !s.done) {
            if (s.status == 0) s.status = HF_ERR_NOT_CONVERGED;
            s.done = 1;
            s.fin = 1;
        }
        s.total_iters += s.iters + s.iters_prev;
        if (s.status && G.ilim) {
            // a batch under step limits goes on without the failed instance
            G.ilim[i] = 0;
            if (!s.failed) s.failed = s.status;
        }
        if (s.status && atomicCAS(&c->err_status, 0, s.status) == 0) {
            c->err_inst = i;
            c->err_step = c->step;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        c->total_bodies += c->bodies;
        c->step += 1;
        if (c->hist < 2) c->hist += 1;
        c->active = 0;
        c->bodies = 0;
    }
}

// ---------------------------------------------------------------------------
// mixed form: FP32 inner CG on A e = r, FP64 refinement
// ---------------------------------------------------------------------------
// Each sweep runs the CG recurrences of the plain form in FP32 (vectors r32,
// z32, q32, directions, e32; the finest operator's FP32 templates; the FP32
// V-cycle) from e = 0 until ||r32|| <= max(eta ||r||, outer target) or the
// sweep's iteration cap (measured on the batched cavities: aiming at the outer
// target itself, one correction still meets the FP64 test at nearly every
// step, with 7.6 CG iterations per instance-step in the first steps and 3.8
// later, against 8.0 and 4.1 when aiming at half of it; a second sweep runs
// when it does not); then k_ir_correct adds e to the FP64 unknown and
// updates the FP64 residual r -= A e with the FP64 operator, which decides
// convergence against the plain form's test.  Dot products of FP32 vectors
// are accumulated in FP64.

// z32 from the V-cycle (finest post-smoothing or the tail's output), r.z
__global__ void __launch_bounds__(kBlock) k_pcg_z32(PcgFine G, VLev<float> L0)
{
    pdl_wait();
    Blk B;
    if (pcg::load_blk(G.blk, G.S, B)) return;
    const bool tail0 = G.S[B.inst].tail0;
    const pcg::RowSet R = pcg::rowset(B);
    float s[kRPT];
    if (!tail0) pcg::trows(L0.At, R, s, [&](int j) { return L0.x[j]; });
    double part[1] = {0.0};
#pragma unroll
    for (int q = 0; q < kRPT; q++) {
        if (q >= R.nrow) break;
        const int i = R.row[q];
        const float ri = G.r32[i];
        const float z = tail0 ? L0.out[i] : L0.x[i] + L0.dinv[i] * (ri - s[q]);
        G.z32[i] = z;
        part[0] += (double)ri * (double)z;
    }
    double tot[1];
    if (pcg::inst_sum<1>(part, B, G.partials, G.S, tot) && threadIdx.x == 0) {
        IScal &s = G.S[B.inst];
        s.beta = s.iters == 0 ? 0.0 : tot[0] / s.rz;
        s.rz = tot[0];
        if (!isfinite(tot[0])) { s.status = HF_ERR_NAN; pcg::finish_instance(s, G.ctl); }
    }
}

// p = z + beta p_old ; q = A32 p ; alpha = r.z / p.q  (FP32 vectors)
__global__ void __launch_bounds__(kBlock) k_pcg_dir32(PcgFine G, const float *__restrict__ po, float *__restrict__ pn)
{
    pdl_wait();
    Blk B;
    if (pcg::load_blk(G.blk, G.S, B)) return;
    const IScal &sc = G.S[B.inst];
    const bool first = sc.iters == 0;
    const float beta = (float)sc.beta;
    uint32_t d[kRPT];
    pcg::row_descs(G.A32.rd, B, d);
    __shared__ float sp[kStageRows];
    const int s0 = B.row0 + B.pad0, ns = B.cnt + B.pad1 - B.pad0;
    const bool staged = ns <= kStageRows;
    if (staged) {
        for (int j = threadIdx.x; j < ns; j += kBlock) sp[j] = first ? G.z32[s0 + j] : G.z32[s0 + j] + beta * po[s0 + j];
        __syncthreads();
    }
    double part[1] = {0.0};
#pragma unroll
    for (int q = 0; q < kRPT; q++) {
        const int t = threadIdx.x + q * kBlock;
        if (t >= B.cnt) break;
        const int i = B.row0 + t;
        float qi, p;
        if (staged) {
            qi = trow_d(G.A32, d[q], i, [&](int j) { return sp[j - s0]; });
            p = sp[i - s0];
        } else if (first) {
            qi = trow_d(G.A32, d[q], i, [&](int j) { return G.z32[j]; });
            p = G.z32[i];
        } else {
            qi = trow_d(G.A32, d[q], i, [&](int j) { return G.z32[j] + beta * po[j]; });
            p = G.z32[i] + beta * po[i];
        }
        pn[i] = p;
        G.q32[i] = qi;
        part[0] += (double)p * (double)qi;
    }
    double tot[1];
    if (pcg::inst_sum<1>(part, B, G.partials, G.S, tot) && threadIdx.x == 0) {
        IScal &s = G.S[B.inst];
        if (!isfinite(tot[0])) {
            s.status = HF_ERR_NAN;
            pcg::finish_instance(s, G.ctl);
        } else if (!(tot[0] > 0.0)) {
            // p.q <= 0: the FP32 recurrence is at its rounding level; the sweep
            // ends and the FP64 correction decides
            pcg::finish_instance(s, G.ctl);
        } else {
            s.alpha = s.rz / tot[0];
        }
    }
}

// e += alpha p ; r32 -= alpha q ; the sweep ends at its target or cap.  The
// first update of a sweep overwrites e (e = alpha p): e is not cleared between
// sweeps.  set_cond as in k_pcg_update.
__global__ void __launch_bounds__(kBlock) k_pcg_update32(PcgFine G, const float *__restrict__ pn,
                                                         cudaGraphConditionalHandle cond, int set_cond)
{
    pdl_wait();
    Blk B;
    const bool skip = pcg::load_blk(G.blk, G.S, B);
    if (!skip) {
        const IScal &sc = G.S[B.inst];
        const float alpha = (float)sc.alpha;
        const bool first = sc.iters == 0;
        const pcg::RowSet R = pcg::rowset(B);
        double part[1] = {0.0};
#pragma unroll
        for (int q = 0; q < kRPT; q++) {
            if (q >= R.nrow) break;
            const int i = R.row[q];
            const float pv = pn[i], qv = G.q32[i];
            G.e32[i] = (first ? 0.f : G.e32[i]) + alpha * pv;
            const float r = G.r32[i] - alpha * qv;
            G.r32[i] = r;
            part[0] += (double)r * (double)r;
        }
        double tot[1];
        if (pcg::inst_sum<1>(part, B, G.partials, G.S, tot) && threadIdx.x == 0) {
            IScal &s = G.S[B.inst];
            s.iters += 1;
            if (!isfinite(tot[0])) { s.status = HF_ERR_NAN; pcg::finish_instance(s, G.ctl); }
            else if (!(tot[0] > s.tol2in) || s.iters >= G.inner_maxit || s.iters + s.iters_prev >= G.maxit)
                pcg::finish_instance(s, G.ctl);
        }
    }
    if (!set_cond) return;
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned t = atomicAdd(&G.ctl->gcount, 1u);
        if (t == gridDim.x - 1) {
            __threadfence();
            Ctl &c = *G.ctl;
            c.gcount = 0;
            c.bodies += 1;
            const int active = ((volatile Ctl *)G.ctl)->active;
            if (set_cond == 1) cudaGraphSetConditional(cond, (active > 0 && c.bodies < c.maxbodies) ? 1u : 0u);
        }
    }
}

// The FP64 refinement step after an inner sweep, on every instance not yet
// finished: x += e, r -= A e (FP64 operator, FP64 arithmetic on the FP32 e),
// ||r|| against the plain form's target; an instance above it starts another
// sweep (last == 0) or is reported not converged (last != 0).  The last block
// of the grid sets the next sweep's loop condition (set_next == 1) or leaves
// the count for the host (eager launches).
__global__ void __launch_bounds__(kBlock) k_ir_correct(PcgFine G, cudaGraphConditionalHandle next, int set_next,
                                                       int last)
{
    __shared__ Blk sb;
    __shared__ int sfin, sstat;
    if (threadIdx.x == 0) {
        sb = G.blk[blockIdx.x];
        const volatile IScal &v = ((volatile IScal *)G.S)[sb.inst];
        sfin = v.fin;
        sstat = v.status;
    }
    __syncthreads();
    const Blk B = sb;
    if (!sfin) {
        const int pt = G.projtype_all >= 0 ? G.projtype_all : G.ipar[B.inst].projtype;
        double *x = pt == HF_INCREMENTAL ? G.dp : G.p;
        const bool apply = sstat == 0;
        double part[1] = {0.0};
        uint32_t d[kRPT];
        pcg::row_descs(G.A.rd, B, d);
#pragma unroll
        for (int q = 0; q < kRPT; q++) {
            const int t = threadIdx.x + q * kBlock;
            if (t >= B.cnt) break;
            const int i = B.row0 + t;
            double r = G.r[i];
            if (apply) {
                x[i] += (double)G.e32[i];
                r -= trow_d(G.A, d[q], i, [&](int j) { return (double)G.e32[j]; });
                G.r[i] = r;
                G.r32[i] = (float)r;
            }
            part[0] += r * r;
        }
        double tot[1];
        if (pcg::inst_sum<1>(part, B, G.partials, G.S, tot) && threadIdx.x == 0) {
            IScal &s = G.S[B.inst];
            s.rr = tot[0];
            if (s.status != 0) {
                s.fin = 1;
            } else if (!isfinite(tot[0])) {
                s.status = HF_ERR_NAN;
                s.fin = 1;
            } else if (!(tot[0] > s.tol2)) {
                s.fin = 1;
            } else if (last || s.iters + s.iters_prev >= G.maxit) {
                s.status = HF_ERR_NOT_CONVERGED;
                s.fin = 1;
            } else {
                s.outer += 1;
                s.iters_prev += s.iters;
                s.iters = 0;
                s.beta = 0.0;
                s.tol2in = fmax(s.tol2, G.eta * G.eta * tot[0]);
                s.done = 0;
                atomicAdd(&G.ctl->active, 1);
            }
        }
    }
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned t = atomicAdd(&G.ctl->gcount, 1u);
        if (t == gridDim.x - 1) {
            __threadfence();
            Ctl &c = *G.ctl;
            c.gcount = 0;
            const int active = ((volatile Ctl *)G.ctl)->active;
            if (set_next) cudaGraphSetConditional(next, active > 0 ? 1u : 0u);
        }
    }
}
