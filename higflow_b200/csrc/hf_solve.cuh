// The Poisson solve of a step as one launch: every instance's whole AMG-PCG
// iteration (hf_pcg.cuh states the recurrences) runs inside one thread-block
// cluster, from the first V-cycle to the converged unknown.
//
// What bounds it: at the sizes of single cases and of the batches' instances
// (10^3 to 10^5 rows) a CG iteration of level-synchronous launches is a chain of
// 8 to 20 dependent kernels of 4 to 5 us each.  Here the phases are separated by
// the hardware's cluster barrier instead, and there are fewer of them:
//  - the V-cycle's smoothing is folded into its transfers when the case is
//    created, so each level takes one phase down and one up:
//      b_{l+1} = Rt b_l,  Rt = R (I - A w D^-1)   (pre-smoothing, residual, R)
//      out_l = Mt b_l + Pt out_{l+1},  Mt = 2 w D^-1 - w D^-1 A w D^-1,
//      Pt = (I - w D^-1 A) P                      (prolongation, post-smoothing)
//    (the same V-cycle in exact arithmetic);
//  - the small levels (kSolveTail rows and below) run in every CTA of the
//    cluster for itself, so they need block barriers only;
//  - q = A p is carried as q = A z + beta q, so p has no neighbour reads;
//  - each dot product's partial sums travel with the barrier that follows it.
// And a phase is short: a CTA owns a contiguous range of every level's rows and
// holds the vectors over that range and the columns its rows reach (its halo)
// in shared memory.  The owner of a value stores it to its own copy and to the
// halo copies of the CTAs that read it (distributed shared memory), so every
// gather is a local shared-memory load.  The operators are row templates (a few
// hundred entries per level on a uniform grid) in shared memory too.  What does
// not fit stays in global memory (L2) behind the same indexing.
//
// Partial sums are added in a fixed order: the same results on every run.
#pragma once

#include <cstdint>

constexpr int kSolveThreads = 1024;
constexpr int kSolveWarps = kSolveThreads / 32;
constexpr int kSolveTail = 1024;             // largest level run by every CTA for itself
constexpr int kSolveSmem = 206 * 1024;       // dynamic shared memory
constexpr int kSolveLenBits = 10;            // rows of up to 1023 entries, 2^22 entries per operator
constexpr int kSolveMaxCluster = 16;
constexpr int kSolveVecs = 2 * kMaxLevels;   // vectors with halos: r, z, then b and out of the levels between
constexpr uint32_t kSolveGlobal = 0xffffffffu;   // "not in shared memory"

// one operator entry: column offset from the row's anchor, value
template <typename T>
struct SEnt;
template <>
struct __align__(8) SEnt<float> {
    int32_t off;
    float v;
};
template <>
struct __align__(16) SEnt<double> {
    double v;
    int32_t off, pad;
};

// an array of the instance's tables: its place in global memory and, when it
// is copied to shared memory, there (byte offsets)
struct STab {
    uint32_t g, s, bytes;
};

// one level of one instance (every level but the coarsest).  Row descriptors
// are (first entry << kSolveLenBits) | entry count.
struct SLevel {
    int32_t n;                // rows
    int32_t lanes_r, lanes_u; // threads per row of the way down (a row of the next level) / up
    // row descriptors down (uint2: row, anchor) and up (uint4: Mt row, Pt row,
    // Pt anchor): global arrays; of the levels above the tail every CTA copies
    // its own rows to shared memory, of the tail all rows
    uint32_t row_r, row_u;    // first descriptor in SInst::rows_r / rows_u
    uint32_t srow_r, srow_u;  // their place in shared memory (bytes) or kSolveGlobal
    STab r, m, p;             // operator tables
    uint32_t vb, vo;          // vectors b and out: T elements into shared memory (kSolveGlobal: into gvec)
    uint32_t gb, go;          // ... into SInst::gvec (levels above the tail)
};

template <typename T>
struct SInst {
    int32_t inst, row0, n, s, clev, nc;      // s: first tail level; nc: rows of the coarsest
    uint32_t vr, vz, vp, vq, vx;             // finest vectors in shared memory (bytes; vx: x, or e in the mixed form)
    uint32_t cvec;                           // the coarsest level's vectors (T elements into shared memory)
    STab a, a64, inv;                        // finest operator (T, FP64), dense inverse
    const char *tables;
    const uint2 *rows_r;
    const uint4 *rows_u;
    T *gvec;
    // [kSolveVecs][cluster]: rows [x, y) each rank holds of a vector, and the
    // ranks [z, w] that hold some of its own rows
    const int4 *rng;
    SLevel L[kMaxLevels];
};

template <typename T>
struct SolveArgs {
    const SInst<T> *I;
    T *r, *z, *p, *q, *e;                    // finest vectors in global memory (e: mixed form only)
    int first;                               // first instance of this launch in I
};

namespace solve {

namespace cg = ::cooperative_groups;

__device__ __forceinline__ float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_(double a, double b, double c) { return __fma_rn(a, b, c); }

// a row's entries k0, k0 + step, ... (two per turn: the host pads rows to an
// even number of turns) times f
template <typename T>
__device__ __forceinline__ T row_part(const SEnt<T> *tab, uint32_t d, int lane, int lanes, const T *f)
{
    const SEnt<T> *t = tab + (d >> kSolveLenBits) + lane;
    int len = (int)(d & ((1u << kSolveLenBits) - 1));
    T s = T(0), u = T(0);
#pragma unroll 2
    for (; len > 0; len -= 2 * lanes) {
        const SEnt<T> e0 = t[0], e1 = t[lanes];
        t += 2 * lanes;
        s = fma_(e0.v, f[e0.off], s);
        u = fma_(e1.v, f[e1.off], u);
    }
    return s + u;
}

// a row of exactly K entries (shorter rows are padded)
template <int K, typename T>
__device__ __forceinline__ T row_fixed(const SEnt<T> *tab, uint32_t d, const T *f)
{
    const SEnt<T> *t = tab + (d >> kSolveLenBits);
    T s = T(0), u = T(0);
#pragma unroll
    for (int k = 0; k < K; k++) {
        const SEnt<T> e = t[k];
        T &a = k & 1 ? u : s;
        a = fma_(e.v, f[e.off], a);
    }
    return s + u;
}

// a row of the finest operator: K entries, or any even number (K = 0)
template <int K, typename T>
__device__ __forceinline__ T fine_row(const SEnt<T> *tab, uint32_t d, const T *f)
{
    return K > 0 ? row_fixed<K>(tab, d, f) : row_part(tab, d, 0, 1, f);
}

template <typename T>
__device__ __forceinline__ T lanes_sum(T s, int lanes)
{
    for (int o = lanes >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

struct Team {
    int rank, size;
    double (*slot)[kSolveMaxCluster][kSolveWarps];   // [2][rank][warp] partial sums, double buffered
    int par;
};

__device__ __forceinline__ void team_sync(const Team &t)
{
    if (t.size > 1) cg::this_cluster().sync();
    else __syncthreads();
}

// sum over the cluster, the same value in every thread; a team barrier: what
// was written before it is visible to every thread of the cluster after it
__device__ __forceinline__ double team_sum(Team &t, double v)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    t.par ^= 1;
    double *mine = &t.slot[t.par][t.rank][wid];
    if (t.size > 1) {
        if (lane < t.size) *cg::this_cluster().map_shared_rank(mine, lane) = v;
    } else if (lane == 0) {
        *mine = v;
    }
    team_sync(t);
    // (the slots of warps that do not exist stay zero)
    double s = 0.0;
    for (int k = 0; k < t.size; k++) s += t.slot[t.par][k][lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// rows [lo, hi) of rank k of a level of n rows
__host__ __device__ __forceinline__ void rank_rows(int k, int size, int n, int &lo, int &hi)
{
    const int ch = (n + size - 1) / size;
    lo = k * ch < n ? k * ch : n;
    hi = lo + ch < n ? lo + ch : n;
}

// A vector by global row index: at[i] for the rows this CTA holds.  put()
// stores an own row's value, to the other holders' copies too: rows in
// [own_lo, own_hi) have none.
template <typename T>
struct Vec {
    T *at;
    T *sh;              // this CTA's copy (null: global memory)
    const int4 *rng;    // per rank
    int rank, klo, khi, own_lo, own_hi;
    __device__ __forceinline__ void put(int i, T v) const
    {
        at[i] = v;
        if (i < own_lo || i >= own_hi) put_far(i, v);
    }
    __device__ __forceinline__ void put_far(int i, T v) const
    {
        for (int k = klo; k <= khi; k++) {
            const int4 g = rng[k];
            if (k != rank && i >= g.x && i < g.y) cg::this_cluster().map_shared_rank(sh, k)[i - g.x] = v;
        }
    }
};

// what a CTA needs of a level, resolved once per solve
template <typename T>
struct Plan {
    const SEnt<T> *tr, *tm, *tp;
    const uint2 *rr;          // by row
    const uint4 *ru;
    Vec<T> b, o;              // by row (the tail's: shared, no halo)
    int rlo, rhi, ulo, uhi;   // own rows of the way down (the next level's) and up
    int lr, lu;               // log2 of the threads per row
};

// the own rows of the operator down to the next level: put(row, value, lane)
// by every lane of the row
template <typename T, typename Put>
__device__ __forceinline__ void down(const Plan<T> &P, const T *b, Put put)
{
    const int lr = P.lr, hi = P.rhi, step = blockDim.x >> lr, lane = threadIdx.x & ((1 << lr) - 1);
    const SEnt<T> *tab = P.tr;
    const uint2 *rows = P.rr;
    for (int base = P.rlo; base < hi; base += step) {
        const int i = base + (threadIdx.x >> lr);
        const uint2 d = i < hi ? rows[i] : make_uint2(0u, 0u);
        const T s = lanes_sum(row_part(tab, d.x, lane, 1 << lr, b + (int)d.y), 1 << lr);
        if (i < hi) put(i, s, lane);
    }
}

// out_l = Mt b_l + Pt e on the own rows
template <typename T, typename Put>
__device__ __forceinline__ void up(const Plan<T> &P, const T *b, const T *e, Put put)
{
    const int lu = P.lu, hi = P.uhi, step = blockDim.x >> lu, lane = threadIdx.x & ((1 << lu) - 1);
    const SEnt<T> *tm = P.tm, *tp = P.tp;
    const uint4 *rows = P.ru;
    for (int base = P.ulo; base < hi; base += step) {
        const int i = base + (threadIdx.x >> lu);
        const uint4 d = i < hi ? rows[i] : make_uint4(0u, 0u, 0u, 0u);
        T s = row_part(tm, d.x, lane, 1 << lu, b + i);
        s += row_part(tp, d.y, lane, 1 << lu, e + (int)d.z);
        s = lanes_sum(s, 1 << lu);
        if (i < hi && lane == 0) put(i, s);
    }
}

}  // namespace solve

// K: entries of the finest operator's rows (5: 2D, 7: 3D uniform grids), 0: any
template <typename T, bool MIX, int K>
__global__ void __launch_bounds__(kSolveThreads, 1) k_solve(PcgFine G, SolveArgs<T> A)
{
    extern __shared__ __align__(16) char dyn[];
    __shared__ SInst<T> I;
    __shared__ solve::Plan<T> plan[kMaxLevels];
    __shared__ double slot[2][kSolveMaxCluster][kSolveWarps];
    __shared__ int4 rng[kSolveVecs][kSolveMaxCluster];
    namespace cg = ::cooperative_groups;
    const int tid = threadIdx.x, nt = blockDim.x;
    solve::Team t;
    t.rank = (int)cg::this_cluster().block_rank();
    t.size = (int)cg::this_cluster().num_blocks();
    t.slot = slot;
    t.par = 0;
    {
        const uint32_t *src = reinterpret_cast<const uint32_t *>(A.I + A.first + blockIdx.x / t.size);
        for (int k = tid; k < (int)(sizeof(SInst<T>) / 4); k += nt) reinterpret_cast<uint32_t *>(&I)[k] = src[k];
        for (int k = tid; k < 2 * kSolveMaxCluster * kSolveWarps; k += nt) (&slot[0][0][0])[k] = 0.0;
    }
    __syncthreads();
    IScal &S = G.S[I.inst];
    // (read by every CTA before its first team barrier, written after the last)
    const bool idle = ((volatile const IScal &)S).done != 0;
    if (idle) {
        if (tid == 0 && t.rank == 0) S.fin = 1;
        return;
    }
    const double tol2 = S.tol2;
    double tol2in = S.tol2in, rr = S.rr;
    int status = 0, iters = 0, iters_prev = 0, outer = 0;
    const int n = I.n, s0 = I.s, clev = I.clev;
    for (int k = tid; k < kSolveVecs * t.size; k += nt) rng[k / t.size][k % t.size] = I.rng[k];
    __syncthreads();

    // ---- shared memory: tables, row descriptors, vectors
    auto copy16 = [&](uint32_t to, const void *from, uint32_t bytes) {
        for (uint32_t k = tid; k < bytes / 16; k += nt)
            reinterpret_cast<uint4 *>(dyn + to)[k] = __ldg(reinterpret_cast<const uint4 *>(from) + k);
    };
    auto load_tab = [&](const STab &b) { if (b.s != kSolveGlobal) copy16(b.s, I.tables + b.g, b.bytes); };
    auto table = [&](const STab &b) -> const char * { return b.s != kSolveGlobal ? dyn + b.s : I.tables + b.g; };
    auto ents = [&](const STab &b) { return reinterpret_cast<const SEnt<T> *>(table(b)); };
    load_tab(I.a);
    load_tab(I.inv);
    if (MIX) load_tab(I.a64);
    T *tail = reinterpret_cast<T *>(dyn);
    auto vec = [&](int id, T *sh, T *global, int lo, int hi) {
        solve::Vec<T> v;
        const int4 g = rng[id][t.rank];
        v.sh = sh;
        v.at = sh ? sh - g.x : global;
        v.rng = rng[id];
        v.rank = t.rank;
        v.klo = g.z;
        v.khi = g.w;
        v.own_lo = lo;
        v.own_hi = hi;
        if (sh && t.size > 1) {
            // rows that some other rank holds too: below own_lo, from own_hi
            for (int k = g.z; k < t.rank; k++) v.own_lo = max(v.own_lo, min(hi, rng[id][k].y));
            for (int k = t.rank + 1; k <= g.w; k++) v.own_hi = min(v.own_hi, max(lo, rng[id][k].x));
        }
        return v;
    };
    int lo, hi;
    solve::rank_rows(t.rank, t.size, n, lo, hi);
    auto log2i = [](int v) { return 31 - __clz(v); };
    for (int l = 0; l < max(1, clev); l++) {
        const SLevel &L = I.L[l];
        load_tab(L.r);
        load_tab(L.m);
        load_tab(L.p);
        // row descriptors: of the own rows (above the tail), or all
        const int nr = l + 1 < clev ? I.L[l + 1].n : clev > 0 ? I.nc : 0;
        int a = 0, h = nr, ua = 0, uh = L.n;
        if (l < s0 || clev == 0) {
            solve::rank_rows(t.rank, t.size, nr, a, h);
            solve::rank_rows(t.rank, t.size, L.n, ua, uh);
        }
        if (L.srow_u != kSolveGlobal)
            for (int i = ua + tid; i < uh; i += nt)
                reinterpret_cast<uint4 *>(dyn + L.srow_u)[i - ua] = __ldg(I.rows_u + L.row_u + i);
        if (L.srow_r != kSolveGlobal)
            for (int i = a + tid; i < h; i += nt)
                reinterpret_cast<uint2 *>(dyn + L.srow_r)[i - a] = __ldg(I.rows_r + L.row_r + i);
        if (tid == 0) {
            solve::Plan<T> &P = plan[l];
            P.tr = ents(L.r);
            P.tm = ents(L.m);
            P.tp = ents(L.p);
            P.rr = L.srow_r != kSolveGlobal ? reinterpret_cast<const uint2 *>(dyn + L.srow_r) - a : I.rows_r + L.row_r;
            P.ru = L.srow_u != kSolveGlobal ? reinterpret_cast<const uint4 *>(dyn + L.srow_u) - ua : I.rows_u + L.row_u;
            P.rlo = a;
            P.rhi = h;
            P.ulo = ua;
            P.uhi = uh;
            P.lr = log2i(L.lanes_r);
            P.lu = log2i(L.lanes_u);
            if (l == 0) {
                P.b = vec(0, I.vr == kSolveGlobal ? nullptr : reinterpret_cast<T *>(dyn + I.vr), A.r + I.row0, ua, uh);
                P.o = vec(1, I.vz == kSolveGlobal ? nullptr : reinterpret_cast<T *>(dyn + I.vz), A.z + I.row0, ua, uh);
            } else if (l < s0) {
                P.b = vec(2 * l, L.vb == kSolveGlobal ? nullptr : tail + L.vb, I.gvec + L.gb, ua, uh);
                P.o = vec(2 * l + 1, L.vo == kSolveGlobal ? nullptr : tail + L.vo, I.gvec + L.go, ua, uh);
            } else {
                P.b.at = tail + L.vb;
                P.o.at = tail + L.vo;
            }
        }
    }
    __syncthreads();
    const solve::Plan<T> &P0 = plan[0];
    const solve::Vec<T> r = P0.b, z = P0.o;
    // own rows only
    auto priv = [&](uint32_t off, T *global) { return off == kSolveGlobal ? global : reinterpret_cast<T *>(dyn + off) - lo; };
    T *p = priv(I.vp, A.p + I.row0), *q = priv(I.vq, A.q + I.row0);
    T *e = MIX ? priv(I.vx, A.e + I.row0) : nullptr;
    const int pt = G.projtype_all >= 0 ? G.projtype_all : G.ipar[I.inst].projtype;
    double *xg = (pt == HF_INCREMENTAL ? G.dp : G.p) + I.row0;
    double *x = !MIX && I.vx != kSolveGlobal ? reinterpret_cast<double *>(dyn + I.vx) - lo : xg;
    if (x != xg)
        for (int i = lo + tid; i < hi; i += nt) x[i] = xg[i];
    if (I.vr != kSolveGlobal) {
        const int4 g = rng[0][t.rank];
        for (int i = g.x + tid; i < g.y; i += nt) r.at[i] = A.r[I.row0 + i];
    }
    const SEnt<T> *tabA = ents(I.a), *tabM = P0.tm;
    const uint4 *rows0 = P0.ru;
    // every CTA of the cluster has started (its shared memory may be written)
    solve::team_sync(t);

    // the dense solve of the coarsest level
    const T *inv = reinterpret_cast<const T *>(table(I.inv));
    T *cb = tail + I.cvec, *co = cb + I.nc;
    auto dense = [&]() {
        const int nc = I.nc;
        int lg = 5;
        while (lg > 0 && (nc << lg) > nt) lg--;
        const int lanes = 1 << lg, lane = tid & (lanes - 1), step = nt >> lg;
        for (int base = 0; base < nc; base += step) {
            const int i = base + (tid >> lg);
            T s = T(0);
            if (i < nc) {
                const T *row = inv + (size_t)i * nc;
#pragma unroll 4
                for (int k = lane; k < nc; k += lanes) s = solve::fma_(row[k], cb[k], s);
            }
            s = solve::lanes_sum(s, lanes);
            if (i < nc && lane == 0) co[i] = s;
        }
        __syncthreads();
    };

    // z = V-cycle of r; returns this thread's part of r.z (the team has not
    // yet met on z)
    auto vcycle = [&]() -> double {
        double part = 0.0;
        if (clev == 0) {
            // the finest level is the coarsest: one CTA
            for (int i = tid; i < n; i += nt) cb[i] = r.at[i];
            __syncthreads();
            dense();
            for (int i = lo + tid; i < hi; i += nt) {
                z.put(i, co[i]);
                part += (double)r.at[i] * (double)co[i];
            }
            return part;
        }
        // down the distributed levels
        for (int l = 0; l < s0; l++) {
            const solve::Plan<T> &P = plan[l];
            if (l + 1 == s0) {
                // the tail's rows: to every CTA
                T *nb = l + 1 == clev ? cb : plan[l + 1].b.at;
                solve::down(P, (const T *)P.b.at, [&](int i, T v, int lane) {
                    if (t.size > 1) {
                        for (int k = lane; k < t.size; k += 1 << P.lr) cg::this_cluster().map_shared_rank(nb, k)[i] = v;
                    } else if (lane == 0) {
                        nb[i] = v;
                    }
                });
            } else {
                const solve::Vec<T> &nb = plan[l + 1].b;
                solve::down(P, (const T *)P.b.at, [&](int i, T v, int lane) { if (lane == 0) nb.put(i, v); });
            }
            solve::team_sync(t);
        }
        // the tail, every CTA for itself
        for (int l = s0; l < clev; l++) {
            const solve::Plan<T> &P = plan[l];
            T *nb = l + 1 == clev ? cb : plan[l + 1].b.at;
            solve::down(P, (const T *)P.b.at, [&](int i, T v, int lane) { if (lane == 0) nb[i] = v; });
            __syncthreads();
        }
        dense();
        const T *ev = co;
        for (int l = clev - 1; l >= s0; l--) {
            const solve::Plan<T> &P = plan[l];
            T *ol = P.o.at;
            solve::up(P, (const T *)P.b.at, ev, [&](int i, T v) { ol[i] = v; });
            __syncthreads();
            ev = ol;
        }
        // up the distributed levels
        for (int l = s0 - 1; l > 0; l--) {
            const solve::Plan<T> &P = plan[l];
            solve::up(P, (const T *)P.b.at, ev, [&](int i, T v) { P.o.put(i, v); });
            solve::team_sync(t);
            ev = P.o.at;
        }
        const SEnt<T> *tp = P0.tp;
        for (int i = lo + tid; i < hi; i += nt) {
            const uint4 d = rows0[i];
            const T v = solve::fine_row<K>(tabM, d.x, (const T *)(r.at + i)) + solve::row_part(tp, d.y, 0, 1, ev + (int)d.z);
            z.put(i, v);
            part += (double)r.at[i] * (double)v;
        }
        return part;
    };

    for (int sweep = 0;; sweep++) {
        double rz = 0.0;
        iters = 0;
        bool inner = true;
        while (inner) {
            double tot = solve::team_sum(t, vcycle());
            const bool first = iters == 0;
            const T beta = first ? T(0) : T(tot / rz);
            rz = tot;
            if (!isfinite(tot)) {
                status = HF_ERR_NAN;
                break;
            }
            // p = z + beta p, q = A z + beta q
            double part = 0.0;
            for (int i = lo + tid; i < hi; i += nt) {
                const T w = solve::fine_row<K>(tabA, rows0[i].x, (const T *)(z.at + i));
                const T zi = z.at[i];
                const T pi = first ? zi : solve::fma_(beta, p[i], zi);
                const T qi = first ? w : solve::fma_(beta, q[i], w);
                p[i] = pi;
                q[i] = qi;
                part += (double)pi * (double)qi;
            }
            tot = solve::team_sum(t, part);
            if (!isfinite(tot)) {
                status = HF_ERR_NAN;
                break;
            }
            if (!(tot > 0.0)) {
                // p.q <= 0: the recurrence has reached rounding level.  Plain:
                // accept when the residual is within 100x of the target, else
                // report it; mixed: the sweep ends and the FP64 correction decides
                if (!MIX) status = rr <= 1e4 * tol2 ? 0 : HF_ERR_NOT_CONVERGED;
                break;
            }
            const double alpha = rz / tot;
            const T al = (T)alpha;
            part = 0.0;
            for (int i = lo + tid; i < hi; i += nt) {
                const T pi = p[i];
                const T ri = solve::fma_(-al, q[i], r.at[i]);
                r.put(i, ri);
                part += (double)ri * (double)ri;
                if (MIX) e[i] = first ? al * pi : solve::fma_(al, pi, e[i]);
                else x[i] = __fma_rn(alpha, (double)pi, x[i]);
            }
            tot = solve::team_sum(t, part);
            iters++;
            if (!MIX) rr = tot;
            if (!isfinite(tot)) {
                status = HF_ERR_NAN;
                inner = false;
            } else if (!(tot > (MIX ? tol2in : tol2))) {
                inner = false;
            } else if (MIX ? (iters >= G.inner_maxit || iters + iters_prev >= G.maxit) : iters >= G.maxit) {
                if (!MIX) status = HF_ERR_NOT_CONVERGED;
                inner = false;
            }
        }
        if (!MIX) break;
        // the FP64 refinement step (k_ir_correct): x += e, r -= A e, ||r||
        // against the plain form's target; e takes z's place, with its halo
        double *r64 = G.r + I.row0;
        const SEnt<double> *tab64 = reinterpret_cast<const SEnt<double> *>(table(I.a64));
        // (a sweep that ended before its first update has no correction)
        const bool apply = status == 0 && iters > 0;
        if (apply) {
            for (int i = lo + tid; i < hi; i += nt) z.put(i, e[i]);
            solve::team_sync(t);
        }
        double part = 0.0;
        for (int i = lo + tid; i < hi; i += nt) {
            double ri = r64[i];
            if (apply) {
                const uint32_t d = rows0[i].x;
                const SEnt<double> *te = tab64 + (d >> kSolveLenBits);
                const int len = (int)(d & ((1u << kSolveLenBits) - 1));
                double ax = 0.0;
                for (int k = 0; k < len; k++) {
                    const SEnt<double> a = te[k];
                    ax += a.v * (double)z.at[i + a.off];
                }
                x[i] += (double)e[i];
                ri -= ax;
                r64[i] = ri;
                r.put(i, (T)ri);
            }
            part += ri * ri;
        }
        rr = solve::team_sum(t, part);
        if (status != 0) break;
        if (!isfinite(rr)) {
            status = HF_ERR_NAN;
            break;
        }
        if (!(rr > tol2)) break;
        if (sweep == kMaxSweeps - 1 || iters + iters_prev >= G.maxit) {
            status = HF_ERR_NOT_CONVERGED;
            break;
        }
        outer++;
        iters_prev += iters;
        tol2in = fmax(tol2, G.eta * G.eta * rr);
    }
    if (x != xg)
        for (int i = lo + tid; i < hi; i += nt) xg[i] = x[i];
    if (tid == 0 && t.rank == 0) {
        S.rr = rr;
        S.iters = iters;
        S.iters_prev = iters_prev;
        S.outer = outer;
        S.tol2in = tol2in;
        S.status = status;
        S.done = 1;
        S.fin = 1;
    }
    // no CTA leaves while another may still write to its shared memory
    solve::team_sync(t);
}

// ---------------------------------------------------------------------------
// host: the folded operators of one instance as row templates
// ---------------------------------------------------------------------------
namespace solve {

// rows as templates: entries (offset from the anchor, value), deduplicated by
// content; several value sets of one pattern share the descriptor.  Rows are
// padded with zero entries to a multiple of `pad` (to `fixed` entries each when
// that is set).
struct Tables {
    int pad = 1, fixed = 0;
    std::vector<uint32_t> desc;
    std::vector<int32_t> off;
    std::vector<double> v, v2;
    std::unordered_map<std::string, uint32_t> seen;
    std::string key;
    bool ok = true;
    uint32_t row(const int *col, const double *val, const double *val2, int len, int anchor)
    {
        key.clear();
        for (int k = 0; k < len; k++) {
            const int32_t o = col[k] - anchor;
            key.append((const char *)&o, sizeof o);
            key.append((const char *)&val[k], sizeof(double));
            if (val2) key.append((const char *)&val2[k], sizeof(double));
        }
        auto it = seen.find(key);
        if (it != seen.end()) return it->second;
        const int full = fixed ? fixed : (len + pad - 1) / pad * pad;
        if (full < len || full >= (1 << kSolveLenBits) || off.size() + full >= ((size_t)1 << (32 - kSolveLenBits))) {
            ok = false;
            return 0;
        }
        const uint32_t d = ((uint32_t)off.size() << kSolveLenBits) | (uint32_t)full;
        seen.emplace(key, d);
        for (int k = 0; k < len; k++) {
            off.push_back(col[k] - anchor);
            v.push_back(val[k]);
            if (val2) v2.push_back(val2[k]);
        }
        for (int k = len; k < full; k++) {
            off.push_back(len ? col[len - 1] - anchor : 0);
            v.push_back(0.0);
            if (val2) v2.push_back(0.0);
        }
        return d;
    }
};

struct HostSolve {
    bool ok = false;
    int s = 0, clev = 0, nc = 0, cluster = 1, fine = 0;   // fine: k_solve's K
    std::vector<int4> rng;      // [kSolveVecs][cluster], see SInst::rng
    int held[kSolveVecs] = {};  // most rows a rank holds of the vector
    struct Level {
        int n = 0, lanes_r = 1, lanes_u = 1;
        std::vector<uint2> rows_r;
        std::vector<uint4> rows_u;
        std::vector<int32_t> off_r, off_m, off_p;
        std::vector<double> v_r, v_m, v_p, v_a;   // v_a: the finest operator on off_m's pattern
    };
    std::vector<Level> L;
};

inline int lanes_for(double avg)
{
    int l = 1;
    while (l < 32 && avg > 12.0 * l) l *= 2;
    return l;
}

// CTAs of an instance's cluster: about kSolveRows rows each while the case's
// instances leave SMs idle (a phase then takes one row per thread or less and
// the barriers dominate), up to 4096 when they fill the device anyway.
// Measured, Poisson solve per step: 4,096 rows alone (FP64) 218 / 232 / 269 /
// 311 / 383 us at 256 / 512 / 1024 / 2048 / 4096 rows a CTA; 32 instances with
// 515,000 rows (mixed) 1785 / 1540 / 1354 / 1310 us at 512 / 1024 / 2048 / 4096.
constexpr int kSolveRows = 512;
inline int cluster_size(int n, long total)
{
    int rows = kSolveRows;
    while (rows < 4096 && total > 148l * rows) rows *= 2;
    int c = 1;
    while (c < kSolveMaxCluster && (long)c * rows < n) c *= 2;
    return c;
}

// the rows of every vector that each rank holds: its own and the columns its
// rows reach
inline void ranges(HostSolve &S)
{
    const int C = S.cluster;
    S.rng.assign((size_t)kSolveVecs * C, make_int4(0, 0, 0, 0));
    auto rows = [&](int l) { return l < (int)S.L.size() ? S.L[l].n : S.nc; };
    auto grow = [](int4 &g, int lo, int hi) {
        g.x = std::min(g.x, lo);
        g.y = std::max(g.y, hi);
    };
    auto reach = [&](int4 &g, const std::vector<int32_t> &off, uint32_t d, int anchor) {
        for (uint32_t k = d >> kSolveLenBits, e = k + (d & ((1u << kSolveLenBits) - 1)); k < e; k++)
            grow(g, anchor + off[k], anchor + off[k] + 1);
    };
    const int levels = std::max(1, S.s);   // levels with distributed vectors
    for (int l = 0; l < levels; l++) {
        const HostSolve::Level &L = S.L[l];
        for (int k = 0; k < C; k++) {
            int lo, hi, a, h;
            rank_rows(k, C, L.n, lo, hi);
            // b of the level (the residual on the finest): Mt and Rt rows
            int4 &b = S.rng[(size_t)(2 * l) * C + k];
            b = make_int4(lo, hi, k, k);
            for (int i = lo; i < hi; i++) reach(b, L.off_m, L.rows_u[i].x, i);
            if (l < S.clev) {
                rank_rows(k, C, rows(l + 1), a, h);
                for (int i = a; i < h; i++) reach(b, L.off_r, L.rows_r[i].x, (int)L.rows_r[i].y);
            }
            // z on the finest level: A rows (Mt's pattern); out of a level
            // between: the Pt rows of the level above
            int4 &o = S.rng[(size_t)(2 * l + 1) * C + k];
            o = make_int4(lo, hi, k, k);
            if (l == 0) {
                for (int i = lo; i < hi; i++) reach(o, L.off_m, L.rows_u[i].x, i);
            } else {
                const HostSolve::Level &F = S.L[l - 1];
                rank_rows(k, C, F.n, a, h);
                for (int i = a; i < h; i++) reach(o, F.off_p, F.rows_u[i].y, (int)F.rows_u[i].z);
            }
        }
    }
    for (int v = 0; v < 2 * levels; v++)
        for (int k = 0; k < C; k++) {
            int4 &g = S.rng[(size_t)v * C + k];
            S.held[v] = std::max(S.held[v], g.y - g.x);
            int lo, hi;
            rank_rows(k, C, S.L[v / 2].n, lo, hi);
            for (int j = 0; j < C; j++) {
                const int4 &f = S.rng[(size_t)v * C + j];
                if (f.x < hi && f.y > lo) {
                    g.z = std::min(g.z, j);
                    g.w = std::max(g.w, j);
                }
            }
        }
}

inline HostSolve build(const std::vector<hf::HostLevel> &H, long total)
{
    HostSolve S;
    S.clev = (int)H.size() - 1;
    S.nc = H.back().A.n;
    S.s = S.clev == 0 ? 0 : 1;
    while (S.s < S.clev && H[S.s].A.n > kSolveTail) S.s++;
    if (S.nc > kCoarseCap || S.clev >= kMaxLevels) return S;
    size_t tail = 2 * S.nc;   // the tail's vectors always live in shared memory
    for (int l = std::max(1, S.s); l < S.clev; l++) tail += 2 * H[l].A.n;
    if (tail * sizeof(double) > kSolveSmem / 2) return S;
    S.cluster = S.clev == 0 ? 1 : cluster_size(H[0].A.n, total);
    S.L.resize(std::max(1, S.clev));
    for (int l = 0; l < (int)S.L.size(); l++) {
        const hf::HostLevel &h = H[l];
        HostSolve::Level &o = S.L[l];
        const int n = h.A.n;
        o.n = n;
        o.rows_u.resize(n);
        std::vector<double> d(n);
        for (int i = 0; i < n; i++) d[i] = h.omega * h.dinv[i];
        Tables tm, tp, tr;
        o.lanes_r = l < S.clev ? lanes_for((double)h.R.ptr[h.R.n] / std::max(1, h.R.n) * 1.9) : 1;
        o.lanes_u = l == 0 ? 1 : lanes_for((double)h.A.ptr[n] / n * 0.75);
        tr.pad = 2 * o.lanes_r;
        tm.pad = tp.pad = 2 * o.lanes_u;
        if (l == 0) {
            int most = 0;
            for (int i = 0; i < n; i++) most = std::max(most, h.A.ptr[i + 1] - h.A.ptr[i]);
            S.fine = tm.fixed = most <= 5 ? 5 : most <= 7 ? 7 : 0;
        }
        std::vector<double> mv;
        for (int i = 0; i < n; i++) {
            const int a = h.A.ptr[i], len = h.A.ptr[i + 1] - a;
            mv.resize(len);
            for (int k = 0; k < len; k++) {
                const int j = h.A.col[a + k];
                mv[k] = (j == i ? 2.0 * d[i] : 0.0) - d[i] * h.A.val[a + k] * d[j];
            }
            const uint32_t ds = tm.row(&h.A.col[a], mv.data(), l == 0 ? &h.A.val[a] : nullptr, len, i);
            o.rows_u[i] = make_uint4(ds, 0u, 0u, 0u);
        }
        o.off_m = std::move(tm.off);
        o.v_m = std::move(tm.v);
        o.v_a = std::move(tm.v2);
        if (!tm.ok) return S;
        if (l >= S.clev) {   // the finest level is the coarsest: its operator only
            ranges(S);
            S.ok = true;
            return S;
        }
        // Pt = P - w D^-1 A P
        hf::HostCSR AP = hf::csr_multiply(h.A, h.P);
        std::vector<int> col;
        std::vector<double> val, acc(std::max(h.P.m, n), 0.0);
        for (int i = 0; i < n; i++) {
            for (int k = h.P.ptr[i]; k < h.P.ptr[i + 1]; k++) acc[h.P.col[k]] = h.P.val[k];
            col.clear();
            val.clear();
            for (int k = AP.ptr[i]; k < AP.ptr[i + 1]; k++) {
                const double v = acc[AP.col[k]] - d[i] * AP.val[k];
                if (v != 0.0) {
                    col.push_back(AP.col[k]);
                    val.push_back(v);
                }
            }
            for (int k = h.P.ptr[i]; k < h.P.ptr[i + 1]; k++) acc[h.P.col[k]] = 0.0;
            const int anchor = col.empty() ? 0 : col[0];
            o.rows_u[i].y = tp.row(col.data(), val.data(), nullptr, (int)col.size(), anchor);
            o.rows_u[i].z = (uint32_t)anchor;
        }
        o.off_p = std::move(tp.off);
        o.v_p = std::move(tp.v);
        // Rt = R - R A w D^-1
        hf::HostCSR RA = hf::csr_multiply(h.R, h.A);
        const int nn = h.R.n;
        o.rows_r.resize(nn);
        for (int i = 0; i < nn; i++) {
            for (int k = h.R.ptr[i]; k < h.R.ptr[i + 1]; k++) acc[h.R.col[k]] = h.R.val[k];
            col.clear();
            val.clear();
            for (int k = RA.ptr[i]; k < RA.ptr[i + 1]; k++) {
                const double v = acc[RA.col[k]] - RA.val[k] * d[RA.col[k]];
                if (v != 0.0) {
                    col.push_back(RA.col[k]);
                    val.push_back(v);
                }
            }
            for (int k = h.R.ptr[i]; k < h.R.ptr[i + 1]; k++) acc[h.R.col[k]] = 0.0;
            const int anchor = col.empty() ? 0 : col[0];
            o.rows_r[i] = make_uint2(tr.row(col.data(), val.data(), nullptr, (int)col.size(), anchor), (uint32_t)anchor);
        }
        o.off_r = std::move(tr.off);
        o.v_r = std::move(tr.v);
        if (!tp.ok || !tr.ok) return S;
    }
    ranges(S);
    S.ok = true;
    return S;
}

}  // namespace solve
