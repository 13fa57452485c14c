// The Poisson solve of a step as one launch: every instance's whole AMG-PCG
// iteration (hf_pcg.cuh states the recurrences) runs inside one thread-block
// cluster, from the first V-cycle to the converged unknown.
//
// What bounds it: at the sizes of single cases and of the batches' instances
// (10^3 to 10^5 rows) a CG iteration of level-synchronous launches is a chain of
// 8 to 20 dependent kernels of 4 to 5 us each.  Here the phases are separated by
// the hardware's cluster barrier instead (400 to 600 cycles), and there are few
// of them, two per level and three for the finest:
//  - the V-cycle's smoothing is folded into its transfers when the case is
//    created, so each level takes one phase down and one up:
//      b_{l+1} = Rt b_l,  Rt = R (I - A w D^-1)   (pre-smoothing, residual, R)
//      out_l = Mt b_l + Pt out_{l+1},  Mt = 2 w D^-1 - w D^-1 A w D^-1,
//      Pt = (I - w D^-1 A) P                      (prolongation, post-smoothing)
//    (the same V-cycle in exact arithmetic); the coarsest levels are one dense
//    operator with its rows shared out over the CTAs where it is small, else
//    the dense solve runs in every CTA for itself;
//  - q = A p is carried as q = A z + beta q, so p has no neighbour reads, and r
//    is updated over a CTA's halo as well as its own rows from the halo of q, so
//    the update and the first phase down need no barrier between them;
//  - each dot product's partial sums travel with the barrier that follows it.
// A phase is short because nothing in it leaves the SM: a CTA owns a contiguous
// range of every level's rows and holds the vectors over that range and the
// columns its rows reach (its halo) in shared memory.  The owner of a value
// stores it to its own copy and to the halo copies of the CTAs that read it
// (distributed shared memory), so every gather is a local shared-memory load.
// The operators lie in shared memory too, as far as they fit: the finest level's
// as row templates (a few hundred entries on a uniform grid, read by most of a
// warp at once), the coarse levels' as the CTA's own rows in slices of 32
// threads (rows there rarely share a template: 32 threads reading 32 templates
// conflict on the banks), with columns as 16-bit shared-memory element indices.
//
// Partial sums are added in a fixed order: the same results on every run.
#pragma once

#include <cstdint>

constexpr int kSolveThreads = 1024;          // most threads of a CTA
constexpr int kSolveWarps = kSolveThreads / 32;
constexpr int kSolveSmem = 213 * 1024;       // dynamic shared memory (227 KB less the static part)
constexpr int kSolveLenBits = 10;            // template rows of up to 1023 entries, 2^22 entries per operator
constexpr int kSolveMaxCluster = 16;
constexpr int kSolveVecs = 2 * kMaxLevels;   // vectors with halos: r (and q), z, then b and out of the levels between
constexpr uint32_t kSolveGlobal = 0xffffffffu;   // "not in shared memory"

// one entry of the finest operator's rows: column offset from the row (SInst::a
// and m: in bytes of T, a64: in rows), value
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

// an array of the instance's (or rank's) tables: byte offset in global memory
// and, when it is copied to shared memory, there
struct STab {
    uint32_t g, s, bytes;
};

// An operator's rows of one rank as slices: slice k holds 32 >> lg rows, 1 << lg
// threads each; the entries of its 32 threads lie side by side, turn by turn
// (turns ptr[k] to ptr[k + 1]).  t: ptr (padded to 16 bytes), the values, the
// columns (16-bit element indices into shared memory).  Padding is value 0 at
// element 0, which k_solve sets to a number first.
struct SOp {
    STab t;
    int32_t row0, rows, lg, nsl;
    uint32_t val, idx;        // byte offsets of the values and columns in t
};

// what one rank of an instance's cluster reads
struct SRank {
    SOp down[kMaxLevels];     // Rt of level l (rows: the next level's)
    SOp up[kMaxLevels];       // Mt and Pt of level l > 0 together; the finest level: Pt
    SOp coarse;               // the coarsest levels' operator (SInst::dist)
    STab desc0;               // finest level's own rows: uint2 {Pt template row, Pt anchor (element index) << 16 | Mt/A template}
    STab desc_r;              // template form of the first way down: uint2 {Rt template row, anchor (element index)}
};

template <typename T>
struct SInst {
    int32_t inst, row0, n, clev, nc;         // clev: the coarsest level; nc: its rows
    int32_t ndown, ncb;                      // operators down; rows the last of them writes (cvec; nc results follow)
    int32_t dist;                            // 0: dense inverse in every CTA; 1: SRank::coarse, rows shared out
    int32_t tpl_p, tpl_r, lg_r;              // the finest Pt / Rt as templates; threads per Rt row (log2)
    uint32_t vr, vq, vz, vp, vx;             // finest vectors in shared memory (bytes; vx: x, or e in the mixed form)
    uint32_t vb[kMaxLevels], vo[kMaxLevels]; // vectors of the levels between (bytes)
    uint32_t cvec;                           // the coarsest level's vectors (bytes)
    STab a, m, a64, inv;                     // finest operator (T), Mt, finest operator (FP64), dense inverse
    STab tpv, tpo, trv, tro;                 // template entries of Pt / Rt: values, 16-bit column offsets
    int32_t lvl[kMaxLevels];                 // rows of the levels
    const char *tables;
    const char *rank_tables;                 // the ranks' tables (SRank offsets are into these)
    const SRank *ranks;
    // [kSolveVecs][cluster]: rows [x, y) each rank holds of a vector, and the
    // ranks [z, w] that hold some of its own rows
    const int4 *rng;
};

template <typename T>
struct SolveArgs {
    const SInst<T> *I;
    const T *r;                              // the first residual
    T *p, *e;                                // where p and e do not fit (e: mixed form only)
    int first;                               // first instance of this launch in I
};

namespace solve {

__device__ __forceinline__ float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_(double a, double b, double c) { return __fma_rn(a, b, c); }

// Shared memory is addressed by 32-bit byte offsets into the kernel's dynamic
// part (dyn): the loads are then plain shared-memory loads with 32-bit address
// arithmetic, where pointers kept in a struct would be generic 64-bit ones (the
// phases are chains of a few hundred instructions a warp, so these count).
extern __shared__ __align__(16) char dyn[];
template <typename T>
__device__ __forceinline__ T &at(uint32_t off)
{
    return *reinterpret_cast<T *>(dyn + off);
}

// the address of a shared variable in another CTA of the cluster, and a store to it
__device__ __forceinline__ uint32_t peer(uint32_t local, int rank)
{
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
    return a;
}
__device__ __forceinline__ uint32_t address(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void store_peer(uint32_t a, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void store_peer(uint32_t a, float v)
{
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

// a template row's entries lane, lane + lanes, ... (two per turn: the host pads
// rows to a whole number of turns) times f; val, off: byte offsets of the tables
template <typename T>
__device__ __forceinline__ T row_part(uint32_t val, uint32_t off, uint32_t d, int lane, int lanes, uint32_t f)
{
    const uint32_t k0 = (d >> kSolveLenBits) + lane;
    val += k0 * (uint32_t)sizeof(T);
    off += k0 * 2u;
    int len = (int)(d & ((1u << kSolveLenBits) - 1));
    T s = T(0), u = T(0);
#pragma unroll 2
    for (; len > 0; len -= 2 * lanes) {
        const int o0 = at<int16_t>(off), o1 = at<int16_t>(off + 2u * lanes);
        s = fma_(at<T>(val), at<T>(f + o0 * (int)sizeof(T)), s);
        u = fma_(at<T>(val + (uint32_t)sizeof(T) * lanes), at<T>(f + o1 * (int)sizeof(T)), u);
        val += 2u * (uint32_t)sizeof(T) * lanes;
        off += 4u * lanes;
    }
    return s + u;
}

// a row of exactly K entries (shorter rows are padded); k: entries, K = 0.
// t: byte offset of the entries, f: of the row's own element
template <int K, typename T>
__device__ __forceinline__ T row_fixed(uint32_t t, int k, uint32_t f)
{
    T s = T(0), u = T(0);
    if (K > 0) {
        SEnt<T> e[K > 0 ? K : 1];
#pragma unroll
        for (int j = 0; j < K; j++) e[j] = at<SEnt<T>>(t + j * (uint32_t)sizeof(SEnt<T>));
#pragma unroll
        for (int j = 0; j < K; j++) {
            T &a = j & 1 ? u : s;
            a = fma_(e[j].v, at<T>(f + e[j].off), a);
        }
    } else {
#pragma unroll 4
        for (int j = 0; j < k; j++) {
            const SEnt<T> e = at<SEnt<T>>(t + j * (uint32_t)sizeof(SEnt<T>));
            s = fma_(e.v, at<T>(f + e.off), s);
        }
    }
    return s + u;
}

template <typename T>
__device__ __forceinline__ T lanes_sum(T s, int lanes)
{
    for (int o = lanes >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

struct Team {
    int rank, size, par;
    double (*slot)[kSolveMaxCluster];   // [2][rank] partial sums, double buffered
    double *warp;                       // per-warp partial sums (zero beyond the block's warps)
};

// every thread of the cluster; what was written before is visible after
__device__ __forceinline__ void team_sync(const Team &t)
{
    if (t.size > 1) {
        __syncwarp();   // (.aligned: whole warps arrive)
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
}

// sum over the cluster, the same value in every thread; a team barrier
__device__ __forceinline__ double team_sum(Team &t, double v)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) t.warp[wid] = v;
    __syncthreads();
    t.par ^= 1;
    double *mine = &t.slot[t.par][t.rank];
    if (wid == 0) {
        v = t.warp[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (t.size > 1) {
            if (lane < t.size) store_peer(peer(address(mine), lane), v);
        } else if (lane == 0) {
            *mine = v;
        }
    }
    team_sync(t);
    const double2 *s2 = reinterpret_cast<const double2 *>(t.slot[t.par]);
    double s = 0.0, u = 0.0;
    for (int k = 0; 2 * k < t.size; k++) {
        const double2 w = s2[k];
        s += w.x;
        u += w.y;   // (zero beyond the cluster)
    }
    return s + u;
}

// rows [lo, hi) of rank k of a level of n rows
__host__ __device__ __forceinline__ void rank_rows(int k, int size, int n, int &lo, int &hi)
{
    const int ch = (n + size - 1) / size;
    lo = k * ch < n ? k * ch : n;
    hi = lo + ch < n ? lo + ch : n;
}

// A vector over the rows this CTA holds: row i at byte offset base + i *
// sizeof(T).  put() stores an own row's value, to the other holders' copies too:
// rows in [own_lo, own_hi) have none.
template <typename T>
struct Vec {
    uint32_t base;
    uint32_t sh;        // shared address of this CTA's copy
    const int4 *rng;    // per rank
    int rank, klo, khi, own_lo, own_hi;
    __device__ __forceinline__ uint32_t row(int i) const { return base + (uint32_t)i * (uint32_t)sizeof(T); }
    __device__ __forceinline__ T get(int i) const { return solve::at<T>(row(i)); }
    __device__ __forceinline__ void put(int i, T v) const
    {
        solve::at<T>(row(i)) = v;
        if (i >= own_lo && i < own_hi) return;
        for (int k = klo; k <= khi; k++) {
            const int2 g = *reinterpret_cast<const int2 *>(rng + k);
            if (k != rank && i >= g.x && i < g.y) store_peer(peer(sh + (uint32_t)(i - g.x) * (uint32_t)sizeof(T), k), v);
        }
    }
};

// a rank's operator, resolved once per solve: in shared memory (byte offsets) or
// global (g)
struct Op {
    const char *g;
    uint32_t ptr, val, idx;
    int row0, rows, lg, nsl;
};

// this thread's part of slice k
template <typename T>
__device__ __forceinline__ T slice_part(const Op &P, int k)
{
    const int lane = threadIdx.x & 31;
    T s = T(0);
    if (!P.g) {
        const uint32_t a = at<uint32_t>(P.ptr + 4u * k);
        int len = (int)(at<uint32_t>(P.ptr + 4u * k + 4u) - a);
        uint32_t val = P.val + (a * 32u + lane) * (uint32_t)sizeof(T), idx = P.idx + (a * 32u + lane) * 2u;
#pragma unroll 4
        for (; len > 0; len--, val += 32u * (uint32_t)sizeof(T), idx += 64u)
            s = fma_(at<T>(val), at<T>(at<uint16_t>(idx) * (uint32_t)sizeof(T)), s);
        return s;
    }
    const uint32_t *ptr = reinterpret_cast<const uint32_t *>(P.g + P.ptr);
    const uint32_t a = __ldg(ptr + k);
    int len = (int)(__ldg(ptr + k + 1) - a);
    const T *val = reinterpret_cast<const T *>(P.g + P.val) + a * 32 + lane;
    const uint16_t *idx = reinterpret_cast<const uint16_t *>(P.g + P.idx) + a * 32 + lane;
#pragma unroll 8
    for (; len > 0; len--, val += 32, idx += 32) s = fma_(__ldg(val), at<T>(__ldg(idx) * (uint32_t)sizeof(T)), s);
    return s;
}

// every own row of the operator: put(row, value, lane) by every lane of the row
template <typename T, typename Put>
__device__ __forceinline__ void apply(const Op &O, Put put)
{
    const Op P = O;
    const int warps = blockDim.x >> 5, lane = threadIdx.x & 31;
    for (int k = threadIdx.x >> 5; k < P.nsl; k += warps) {
        const T s = lanes_sum(slice_part<T>(P, k), 1 << P.lg);
        const int i = (k << (5 - P.lg)) + (lane >> P.lg);
        if (i < P.rows) put(P.row0 + i, s, lane & ((1 << P.lg) - 1));
    }
}

}  // namespace solve

// K: entries of the finest operator's rows (5: 2D, 7: 3D uniform grids), 0: see
// kf.  NT: most threads of a CTA; 512 leave a thread 128 registers instead of 64
// (Poisson solve per step: 1,089 rows 131 -> 126 us, 4,913 rows in 3D 183 -> 177)
template <typename T, bool MIX, int K, int NT>
__global__ void __launch_bounds__(NT, 1) k_solve(PcgFine G, SolveArgs<T> A, int kf)
{
    using solve::at;
    __shared__ SInst<T> I;
    __shared__ SRank Rk;
    __shared__ solve::Op od[kMaxLevels], ou[kMaxLevels], ocoarse;
    __shared__ solve::Vec<T> vb[kMaxLevels], vo[kMaxLevels];
    __shared__ __align__(16) double slot[2][kSolveMaxCluster];
    __shared__ double warp_sums[kSolveWarps];
    __shared__ int4 rng[kSolveVecs][kSolveMaxCluster];
    const int tid = threadIdx.x, nt = blockDim.x;
    constexpr uint32_t kT = (uint32_t)sizeof(T), kE = (uint32_t)sizeof(SEnt<T>);
    solve::Team t;
    t.rank = (int)cooperative_groups::this_cluster().block_rank();
    t.size = (int)cooperative_groups::this_cluster().num_blocks();
    t.slot = slot;
    t.warp = warp_sums;
    t.par = 0;
    auto copy4 = [&](void *to, const void *from, int bytes) {
        for (int k = tid; k < bytes / 4; k += nt) static_cast<uint32_t *>(to)[k] = static_cast<const uint32_t *>(from)[k];
    };
    copy4(&I, A.I + A.first + blockIdx.x / t.size, sizeof I);
    if (tid < 2 * kSolveMaxCluster) (&slot[0][0])[tid] = 0.0;
    if (tid < kSolveWarps) warp_sums[tid] = 0.0;
    __syncthreads();
    const int n = I.n, clev = I.clev;
    for (int k = tid; k < kSolveVecs * t.size; k += nt) rng[k / t.size][k % t.size] = I.rng[k];
    copy4(&Rk, I.ranks + t.rank, sizeof Rk);
    __syncthreads();

    // ---- shared memory: operators, descriptors, vectors
    const char *rt = I.rank_tables;
    auto load = [&](const STab &b, const char *from) {
        if (b.s == kSolveGlobal) return;
        for (uint32_t k = tid; k < b.bytes / 16; k += nt)
            at<uint4>(b.s + 16 * k) = __ldg(reinterpret_cast<const uint4 *>(from + b.g) + k);
    };
    load(I.a, I.tables);
    load(I.m, I.tables);
    load(I.inv, I.tables);
    load(I.tpv, I.tables);
    load(I.tpo, I.tables);
    load(I.trv, I.tables);
    load(I.tro, I.tables);
    load(Rk.desc0, rt);
    load(Rk.desc_r, rt);
    for (int l = 0; l < clev; l++) {
        load(Rk.down[l].t, rt);
        load(Rk.up[l].t, rt);
    }
    if (I.dist) load(Rk.coarse.t, rt);
    auto vec = [&](int id, uint32_t off, int rows) {
        solve::Vec<T> v;
        const int4 g = rng[id][t.rank];
        int lo, hi;
        solve::rank_rows(t.rank, t.size, rows, lo, hi);
        v.base = off - (uint32_t)g.x * kT;
        v.sh = solve::address(solve::dyn + off);
        v.rng = rng[id];
        v.rank = t.rank;
        v.klo = g.z;
        v.khi = g.w;
        // rows that some other rank holds too: below own_lo, from own_hi
        v.own_lo = lo;
        v.own_hi = hi;
        for (int k = g.z; k < t.rank; k++) v.own_lo = max(v.own_lo, min(hi, rng[id][k].y));
        for (int k = t.rank + 1; k <= g.w; k++) v.own_hi = min(v.own_hi, max(lo, rng[id][k].x));
        return v;
    };
    auto resolve = [&](const SOp &o) {
        const uint32_t b = o.t.s != kSolveGlobal ? o.t.s : 0u;
        return solve::Op{o.t.s != kSolveGlobal ? nullptr : rt + o.t.g, b, b + o.val, b + o.idx, o.row0, o.rows, o.lg, o.nsl};
    };
    if (tid == 0) ocoarse = resolve(Rk.coarse);
    if (tid < clev) {
        od[tid] = resolve(Rk.down[tid]);
        ou[tid] = resolve(Rk.up[tid]);
        if (tid > 0) {
            vb[tid] = vec(2 * tid, I.vb[tid], I.lvl[tid]);
            vo[tid] = vec(2 * tid + 1, I.vo[tid], I.lvl[tid]);
        }
    }
    int lo, hi;
    solve::rank_rows(t.rank, t.size, n, lo, hi);
    const solve::Vec<T> r = vec(0, I.vr, n), q = vec(0, I.vq, n), z = vec(1, I.vz, n);
    const int xlo = rng[0][t.rank].x, xhi = rng[0][t.rank].y;   // rows held of r and q
    // own rows only
    const bool ps = I.vp != kSolveGlobal, xs = I.vx != kSolveGlobal;
    T *pg = A.p + I.row0, *eg = MIX ? A.e + I.row0 : nullptr;
    const uint32_t pb = I.vp - (uint32_t)lo * kT, xb = I.vx - (uint32_t)lo * (MIX ? kT : 8u);
    const int pt = G.projtype_all >= 0 ? G.projtype_all : G.ipar[I.inst].projtype;
    double *xg = (pt == HF_INCREMENTAL ? G.dp : G.p) + I.row0;
    // Everything so far was the case's constant data, and overlaps k_pcg_init;
    // from here on its results are read
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (G.ilim && G.ilim[I.inst] == 0) return;   // frozen: nothing changes
    IScal &S = G.S[I.inst];
    // (read by every CTA before its first team barrier, written after the last)
    const bool idle = ((volatile const IScal &)S).done != 0;
    // the unknown's history, and its initial guess in place
    for (int i = lo + tid; i < hi; i += nt) {
        const int j = I.row0 + i;
        const double w = G.xw[j];
        G.xprev2[j] = G.xprev[j];
        G.xprev[j] = xg[i];
        if (!MIX && xs && !idle) at<double>(xb + 8u * i) = w;
        else xg[i] = w;
    }
    if (idle) {
        if (tid == 0 && t.rank == 0) S.fin = 1;
        return;
    }
    const double tol2 = S.tol2;
    double tol2in = S.tol2in, rr = S.rr;
    int status = 0, iters = 0, iters_prev = 0, outer = 0;
    for (int i = xlo + tid; i < xhi; i += nt) at<T>(r.row(i)) = A.r[I.row0 + i];
    const uint32_t tabA = I.a.s, tabM = I.m.s, desc = Rk.desc0.s - 8u * (uint32_t)lo;
    const int kk = K > 0 ? K : kf;
    const uint32_t cb = I.cvec, co = cb + (uint32_t)I.ncb * kT, cb_sh = solve::address(solve::dyn + cb),
                   co_sh = solve::address(solve::dyn + co);
    const int ndown = I.ndown;
    const bool dist = I.dist != 0;
    // the first way down in template form: own rows
    int ra, rh;
    solve::rank_rows(t.rank, t.size, ndown == 1 ? I.ncb : ndown > 1 ? I.lvl[1] : 0, ra, rh);
    const uint32_t desc_r = Rk.desc_r.s - 8u * (uint32_t)ra;
    const bool tpl_p = I.tpl_p != 0, tpl_r = I.tpl_r != 0;
    const uint32_t tpv = I.tpv.s, tpo = I.tpo.s, trv = I.trv.s, tro = I.tro.s;
    const int lg_r = I.lg_r;
    int lg_d = 5;   // threads per row of the dense solve (log2)
    while (lg_d > 0 && (I.nc << lg_d) > nt) lg_d--;
    // (a slice's padding multiplies element 0 of shared memory, the first of cvec,
    // by zero: it has to be a number before the first way down)
    if (tid == 0) at<T>(cb) = T(0);
    // every CTA of the cluster has started (its shared memory may be written)
    solve::team_sync(t);

    // the dense solve of the coarsest level, every CTA for itself
    auto dense = [&]() {
        const int nc = I.nc, lanes = 1 << lg_d, lane = tid & (lanes - 1), step = nt >> lg_d;
        const uint32_t is = I.inv.s;
        for (int b = 0; b < nc; b += step) {
            const int i = b + (tid >> lg_d);
            T s = T(0);
            if (i < nc) {
                if (is != kSolveGlobal) {
                    const uint32_t row = is + (uint32_t)(i * nc) * kT;
#pragma unroll 4
                    for (int k = lane; k < nc; k += lanes) s = solve::fma_(at<T>(row + k * kT), at<T>(cb + k * kT), s);
                } else {
                    const T *row = reinterpret_cast<const T *>(I.tables + I.inv.g) + (size_t)i * nc;
#pragma unroll 4
                    for (int k = lane; k < nc; k += lanes) s = solve::fma_(__ldg(row + k), at<T>(cb + k * kT), s);
                }
            }
            s = solve::lanes_sum(s, lanes);
            if (i < nc && lane == 0) at<T>(co + i * kT) = s;
        }
        __syncthreads();
    };
    // rows of the coarsest vectors: to every CTA
    auto to_all = [&](uint32_t sh, uint32_t own, int i, T v, int lane, int lanes) {
        if (t.size > 1) {
            for (int k = lane; k < t.size; k += lanes) solve::store_peer(solve::peer(sh + i * kT, k), v);
        } else if (lane == 0) {
            at<T>(own + i * kT) = v;
        }
    };
    // the way down from level l: b_{l+1} = Rt b_l
    auto down = [&](int l) {
        const bool last = l + 1 == ndown;
        const solve::Vec<T> nb = vb[last ? l : l + 1];
        const int lg = od[l].lg;
        solve::apply<T>(od[l], [&](int i, T v, int lane) {
            if (last) to_all(cb_sh, cb, i, v, lane, 1 << lg);
            else if (lane == 0) nb.put(i, v);
        });
    };
    auto first_down = [&]() {
        if (clev == 0) {
            // the finest level is the coarsest: one CTA
            for (int i = tid; i < n; i += nt) at<T>(cb + i * kT) = r.get(i);
            return;
        }
        if (!tpl_r) {
            down(0);
            return;
        }
        const bool last = ndown == 1;
        const solve::Vec<T> nb = vb[1];
        const int lanes = 1 << lg_r, lane = tid & (lanes - 1), step = nt >> lg_r;
        for (int b = ra; b < rh; b += step) {
            const int i = b + (tid >> lg_r);
            const uint2 d = i < rh ? at<uint2>(desc_r + 8u * i) : make_uint2(0u, 0u);
            const T s = solve::lanes_sum(solve::row_part<T>(trv, tro, d.x, lane, lanes, d.y * kT), lanes);
            if (i < rh) {
                if (last) to_all(cb_sh, cb, i, s, lane, lanes);
                else if (lane == 0) nb.put(i, s);
            }
        }
    };
    // the V-cycle's rest: z, and this thread's part of r.z (the team has met on
    // b_1, and has not yet on z)
    auto vcycle = [&]() -> double {
        double part = 0.0;
        for (int l = 1; l < ndown; l++) {
            down(l);
            solve::team_sync(t);
        }
        if (dist) {
            const int lg = ocoarse.lg;
            solve::apply<T>(ocoarse, [&](int i, T v, int lane) { to_all(co_sh, co, i, v, lane, 1 << lg); });
            solve::team_sync(t);
        } else {
            dense();
        }
        for (int l = clev - 1; l > 0; l--) {
            const solve::Vec<T> ol = vo[l];
            solve::apply<T>(ou[l], [&](int i, T v, int lane) { if (lane == 0) ol.put(i, v); });
            solve::team_sync(t);
        }
        if (clev == 0) {
            for (int i = lo + tid; i < hi; i += nt) {
                const T v = at<T>(co + i * kT);
                z.put(i, v);
                part += (double)r.get(i) * (double)v;
            }
        } else if (tpl_p) {
            for (int i = lo + tid; i < hi; i += nt) {
                const uint2 d = at<uint2>(desc + 8u * i);
                const T v = solve::row_fixed<K, T>(tabM + (d.y & 0xffffu) * kk * kE, kk, r.row(i)) +
                            solve::row_part<T>(tpv, tpo, d.x, 0, 1, (d.y >> 16) * kT);
                z.put(i, v);
                part += (double)r.get(i) * (double)v;
            }
        } else {
            const solve::Op P = ou[0];
            for (int k = tid >> 5; k < P.nsl; k += nt >> 5) {
                const int i = lo + 32 * k + (tid & 31);
                T v = solve::slice_part<T>(P, k);
                if (i < hi) {
                    v += solve::row_fixed<K, T>(tabM + (at<uint2>(desc + 8u * i).y & 0xffffu) * kk * kE, kk, r.row(i));
                    z.put(i, v);
                    part += (double)r.get(i) * (double)v;
                }
            }
        }
        return part;
    };

    for (int sweep = 0;; sweep++) {
        double rz = 0.0, part = 0.0;
        iters = 0;
        while (true) {
            first_down();
            if (iters == 0) {
                solve::team_sync(t);
            } else {
                // ||r|| of the last update
                const double tot = solve::team_sum(t, part);
                if (!MIX) rr = tot;
                if (!isfinite(tot)) {
                    status = HF_ERR_NAN;
                    break;
                }
                if (!(tot > (MIX ? tol2in : tol2))) break;
                if (MIX ? (iters >= G.inner_maxit || iters + iters_prev >= G.maxit) : iters >= G.maxit) {
                    if (!MIX) status = HF_ERR_NOT_CONVERGED;
                    break;
                }
            }
            double tot = solve::team_sum(t, vcycle());
            const bool first = iters == 0;
            const T beta = first ? T(0) : T(tot / rz);
            rz = tot;
            if (!isfinite(tot)) {
                status = HF_ERR_NAN;
                break;
            }
            // p = z + beta p, q = A z + beta q
            part = 0.0;
            for (int i = lo + tid; i < hi; i += nt) {
                const T w = solve::row_fixed<K, T>(tabA + (at<uint2>(desc + 8u * i).y & 0xffffu) * kk * kE, kk, z.row(i));
                T pi = z.get(i), qi = w;
                if (!first) {
                    pi = solve::fma_(beta, ps ? at<T>(pb + i * kT) : pg[i], pi);
                    qi = solve::fma_(beta, q.get(i), w);
                }
                if (ps) at<T>(pb + i * kT) = pi;
                else pg[i] = pi;
                q.put(i, qi);
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
            for (int i = xlo + tid; i < xhi; i += nt) {
                const T ri = solve::fma_(-al, q.get(i), r.get(i));
                at<T>(r.row(i)) = ri;
                if (i < lo || i >= hi) continue;   // the halo
                const T pi = ps ? at<T>(pb + i * kT) : pg[i];
                part += (double)ri * (double)ri;
                if (MIX) {
                    T v = al * pi;
                    if (!first) v = solve::fma_(al, pi, xs ? at<T>(xb + i * kT) : eg[i]);
                    if (xs) at<T>(xb + i * kT) = v;
                    else eg[i] = v;
                } else if (xs) {
                    at<double>(xb + 8u * i) = __fma_rn(alpha, (double)pi, at<double>(xb + 8u * i));
                } else {
                    xg[i] = __fma_rn(alpha, (double)pi, xg[i]);
                }
            }
            iters++;
            __syncthreads();
        }
        if (!MIX) break;
        // the FP64 refinement step (k_ir_correct): x += e, r -= A e, ||r||
        // against the plain form's target; e takes z's place, with its halo
        double *r64 = G.r + I.row0;
        const SEnt<double> *tab64 = reinterpret_cast<const SEnt<double> *>(I.tables + I.a64.g);
        // (a sweep that ended before its first update has no correction)
        const bool apply = status == 0 && iters > 0;
        if (apply) {
            for (int i = lo + tid; i < hi; i += nt) z.put(i, xs ? at<T>(xb + i * kT) : eg[i]);
            solve::team_sync(t);
        }
        part = 0.0;
        for (int i = lo + tid; i < hi; i += nt) {
            double ri = r64[i];
            if (apply) {
                const SEnt<double> *te = tab64 + (at<uint2>(desc + 8u * i).y & 0xffffu) * kk;
                double ax = 0.0;
                for (int k = 0; k < kk; k++) ax += __ldg(&te[k].v) * (double)z.get(i + __ldg(&te[k].off));
                xg[i] += (double)z.get(i);
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
    if (!MIX && xs)
        for (int i = lo + tid; i < hi; i += nt) xg[i] = at<double>(xb + 8u * i);
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
// host: the folded operators of one instance
// ---------------------------------------------------------------------------
namespace solve {

// rows as templates: entries (offset from the anchor, value), deduplicated by
// content; several value sets of one pattern share the descriptor.  Rows are
// padded with zero entries to a multiple of `pad` (to `fixed` entries each when
// that is set).
struct Tables {
    int pad = 1, fixed = 0;
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
        for (int k = 0; k < full; k++) {
            off.push_back(k < len ? col[k] - anchor : len ? col[len - 1] - anchor : 0);
            v.push_back(k < len ? val[k] : 0.0);
            if (val2) v2.push_back(k < len ? val2[k] : 0.0);
        }
        return d;
    }
};

// sparse rows of one folded operator
struct Csr {
    std::vector<int> ptr{0}, col;
    std::vector<double> val;
    void add(int c, double v)
    {
        if (v == 0.0) return;
        col.push_back(c);
        val.push_back(v);
    }
    void end_row() { ptr.push_back((int)col.size()); }
    int rows() const { return (int)ptr.size() - 1; }
};

// row i of A as row rpos[i], its columns c as cpos[c] (empty: unchanged), sorted
inline Csr permuted(const Csr &A, const std::vector<int> &rpos, const std::vector<int> &cpos)
{
    const int n = A.rows();
    std::vector<int> at(n);
    for (int i = 0; i < n; i++) at[rpos.empty() ? i : rpos[i]] = i;
    Csr B;
    B.col.reserve(A.col.size());
    B.val.reserve(A.val.size());
    std::vector<std::pair<int, double>> row;
    for (int j = 0; j < n; j++) {
        row.clear();
        for (int k = A.ptr[at[j]]; k < A.ptr[at[j] + 1]; k++)
            row.emplace_back(cpos.empty() ? A.col[k] : cpos[A.col[k]], A.val[k]);
        std::sort(row.begin(), row.end(), [](const auto &a, const auto &b) { return a.first < b.first; });
        for (const auto &e : row) {
            B.col.push_back(e.first);
            B.val.push_back(e.second);
        }
        B.end_row();
    }
    return B;
}

// the folded operators of one level (m only where wanted)
inline void fold(const hf::HostLevel &h, Csr *m, Csr &p, Csr &r)
{
    const int n = h.A.n;
    std::vector<double> d(n);
    for (int i = 0; i < n; i++) d[i] = h.omega * h.dinv[i];
    if (m)
        for (int i = 0; i < n; i++) {
            for (int k = h.A.ptr[i]; k < h.A.ptr[i + 1]; k++) {
                const int j = h.A.col[k];
                m->add(j, (j == i ? 2.0 * d[i] : 0.0) - d[i] * h.A.val[k] * d[j]);
            }
            m->end_row();
        }
    if (h.P.ptr.empty()) return;   // the coarsest level
    // Pt = P - w D^-1 A P
    hf::HostCSR AP = hf::csr_multiply(h.A, h.P);
    std::vector<double> acc(std::max(h.P.m, n), 0.0);
    for (int i = 0; i < n; i++) {
        for (int k = h.P.ptr[i]; k < h.P.ptr[i + 1]; k++) acc[h.P.col[k]] = h.P.val[k];
        for (int k = AP.ptr[i]; k < AP.ptr[i + 1]; k++) p.add(AP.col[k], acc[AP.col[k]] - d[i] * AP.val[k]);
        for (int k = h.P.ptr[i]; k < h.P.ptr[i + 1]; k++) acc[h.P.col[k]] = 0.0;
        p.end_row();
    }
    // Rt = R - R A w D^-1
    hf::HostCSR RA = hf::csr_multiply(h.R, h.A);
    for (int i = 0; i < h.R.n; i++) {
        for (int k = h.R.ptr[i]; k < h.R.ptr[i + 1]; k++) acc[h.R.col[k]] = h.R.val[k];
        for (int k = RA.ptr[i]; k < RA.ptr[i + 1]; k++) r.add(RA.col[k], acc[RA.col[k]] - RA.val[k] * d[RA.col[k]]);
        for (int k = h.R.ptr[i]; k < h.R.ptr[i + 1]; k++) acc[h.R.col[k]] = 0.0;
        r.end_row();
    }
}

struct HostSolve {
    bool ok = false;
    int clev = 0, nc = 0, cluster = 1, threads = 256, fine = 0;   // fine: entries of the finest operator's rows
    std::vector<int4> rng;      // [kSolveVecs][cluster], see SInst::rng
    int held[kSolveVecs] = {};  // most rows a rank holds of the vector
    struct Level {
        int n = 0;
        Csr m, p, r;            // Mt (levels above 0), Pt, Rt
    };
    std::vector<Level> L;
    std::vector<int> cpos;      // the coarsest level's rows: their places here (empty: unchanged)
    // The coarsest levels as one dense operator, its rows shared out over the
    // ranks (row-major, nc x ncb); empty: the coarsest level's inverse in every
    // CTA.  g false: the whole V-cycle from level clev's b to its out, Mt + Pt
    // inverse Rt of that level and the one below it; g true: inverse Rt, from
    // level clev - 1's b to the coarsest level's out.
    std::vector<double> coarse;
    bool g = false;
    int ndown = 0, ncb = 0;
    // finest level: A and Mt as templates of `fine` entries, per row the template
    std::vector<uint32_t> tpl;
    std::vector<int32_t> off;
    std::vector<double> va, vm;
};

// CTAs of an instance's cluster: about kSolveRows rows each while the case's
// instances leave SMs idle (a phase then takes one row per thread or less and
// its latency counts), up to 4096 when they fill the device anyway.  Measured,
// Poisson solve per step: 4,096 rows alone (FP64) 135 / 137 / 181 us at
// 256 / 512 / 1024 rows a CTA, 4,913 rows in 3D 184 / 183 / 240.
// 128 cavities of 2.06 M rows in all, whole step: 2.65 ms, 3.75 at 512 rows
// whatever the batch.  The sums' grouping, so the last bits, follow the batch.
constexpr int kSolveRows = 512;
inline int cluster_size(int n, long total, int sms)
{
    int rows = kSolveRows;
    while (rows < 4096 && total > (long)sms * rows) rows *= 2;
    int c = 1;
    while (c < kSolveMaxCluster && (long)c * rows < n) c *= 2;
    return c;
}

// Threads of a CTA with `own` rows of the finest level: the fewest turns a full
// block needs, and no more warps than these turns take (every warp pays a
// phase's fixed instructions); of 512 threads up to kSolveSmall rows, where the
// registers are worth more than the threads.  The instances of a batch share
// three sizes, so that few launches cover them.
constexpr int kSolveSmall = 1536;
inline int block_threads(int own, bool batch)
{
    if (batch) return own <= 256 ? 256 : own <= 512 ? 512 : kSolveThreads;
    const int most = own <= kSolveSmall ? 512 : kSolveThreads, turns = (own + most - 1) / most;
    return std::min(most, std::max(128, ((own + turns - 1) / turns + 31) / 32 * 32));
}

// the rows of every vector that each rank holds: its own and the columns its
// rows reach
inline void ranges(HostSolve &S)
{
    const int C = S.cluster;
    S.rng.assign((size_t)kSolveVecs * C, make_int4(0, 0, 0, 0));
    auto rows = [&](int l) { return l < (int)S.L.size() ? S.L[l].n : S.nc; };
    auto grow = [](int4 &g, int c) {
        g.x = std::min(g.x, c);
        g.y = std::max(g.y, c + 1);
    };
    auto reach = [&](int4 &g, const Csr &A, int lo, int hi) {
        for (int k = A.ptr[lo]; k < A.ptr[hi]; k++) grow(g, A.col[k]);
    };
    auto reach_fine = [&](int4 &g, int lo, int hi) {
        for (int i = lo; i < hi; i++)
            for (int k = 0; k < S.fine; k++) grow(g, i + S.off[(size_t)S.tpl[i] * S.fine + k]);
    };
    const int levels = std::max(1, S.clev);   // levels with distributed vectors
    auto whole = [&](int l) { return S.g && l == S.clev - 1; };   // b: the coarse operator's input, held by all
    for (int l = 0; l < levels; l++) {
        const HostSolve::Level &L = S.L[l];
        for (int k = 0; k < C; k++) {
            int lo, hi, a, h;
            rank_rows(k, C, L.n, lo, hi);
            // b of the level (the residual on the finest): Mt and Rt rows
            int4 &b = S.rng[(size_t)(2 * l) * C + k];
            b = make_int4(lo, hi, k, k);
            if (l == 0) reach_fine(b, lo, hi);
            else reach(b, L.m, lo, hi);
            if (whole(l)) {
                b.x = 0;
                b.y = L.n;
            } else if (l < S.clev) {
                rank_rows(k, C, rows(l + 1), a, h);
                reach(b, L.r, a, h);
            }
            // z on the finest level: A rows; out of a level between: the Pt
            // rows of the level above
            int4 &o = S.rng[(size_t)(2 * l + 1) * C + k];
            o = make_int4(lo, hi, k, k);
            if (l == 0) {
                reach_fine(o, lo, hi);
            } else {
                const HostSolve::Level &F = S.L[l - 1];
                rank_rows(k, C, F.n, a, h);
                reach(o, F.p, a, h);
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

// The coarsest levels as one dense operator where a rank's rows of it are small:
// one phase and no replicated dense solve, in place of two to three phases.  The
// square form up to half of kSolveCoarse bytes (beyond that it displaces finer
// operators from shared memory: 129 x 129 FP64 228 us a step with it, 214 with
// inverse Rt alone), inverse Rt up to kSolveCoarse.
constexpr size_t kSolveCoarse = 76 * 1024;
inline void coarse_operator(HostSolve &S, const std::vector<double> &inverse)
{
    const int last = S.clev - 1, n = S.L[last].n, nc = S.nc, C = S.cluster;
    const HostSolve::Level &L = S.L[last];
    auto bytes = [&](int rows) { return (size_t)((rows + C - 1) / C) * n * 10; };
    if (bytes(nc) > kSolveCoarse) return;
    // G = inverse Rt (rows and columns in this file's order)
    std::vector<int> old(nc);
    for (int i = 0; i < nc; i++) old[S.cpos.empty() ? i : S.cpos[i]] = i;
    std::vector<double> G((size_t)nc * n, 0.0);
    for (int i = 0; i < nc; i++)
        for (int j = 0; j < nc; j++) {
            const double v = inverse[(size_t)old[i] * nc + old[j]];
            for (int k = L.r.ptr[j]; k < L.r.ptr[j + 1]; k++) G[(size_t)i * n + L.r.col[k]] += v * L.r.val[k];
        }
    if (bytes(n) > kSolveCoarse / 2) {
        S.g = true;
        S.coarse = std::move(G);
        S.ndown = last;
        S.ncb = n;
        return;
    }
    // Mt + Pt G
    S.coarse.assign((size_t)n * n, 0.0);
    for (int i = 0; i < n; i++) {
        double *row = S.coarse.data() + (size_t)i * n;
        for (int k = L.m.ptr[i]; k < L.m.ptr[i + 1]; k++) row[L.m.col[k]] += L.m.val[k];
        for (int k = L.p.ptr[i]; k < L.p.ptr[i + 1]; k++) {
            const double *g = G.data() + (size_t)L.p.col[k] * n;
            for (int j = 0; j < n; j++) row[j] += L.p.val[k] * g[j];
        }
    }
    S.clev = S.ndown = last;
    S.nc = S.ncb = n;
    S.L.resize(last);
    S.cpos.clear();
}

inline HostSolve build(const std::vector<hf::HostLevel> &H, const std::vector<double> &inverse, long total, int sms)
{
    HostSolve S;
    S.clev = (int)H.size() - 1;
    S.nc = H.back().A.n;
    if (S.nc > kCoarseCap || S.clev >= kMaxLevels) return S;
    S.cluster = S.clev == 0 ? 1 : cluster_size(H[0].A.n, total, sms);
    S.threads = block_threads((H[0].A.n + S.cluster - 1) / S.cluster, total > H[0].A.n);
    S.L.resize(std::max(1, S.clev));
    for (int l = 0; l < (int)S.L.size(); l++) {
        const hf::HostLevel &h = H[l];
        HostSolve::Level &o = S.L[l];
        const int n = h.A.n;
        o.n = n;
        if (l == 0) {
            int most = 1;
            for (int i = 0; i < n; i++) most = std::max(most, h.A.ptr[i + 1] - h.A.ptr[i]);
            Tables tm;
            S.fine = tm.fixed = most <= 5 ? 5 : most <= 7 ? 7 : most;
            S.tpl.resize(n);
            std::vector<double> mv;
            for (int i = 0; i < n; i++) {
                const int a = h.A.ptr[i], len = h.A.ptr[i + 1] - a;
                const double di = h.omega * h.dinv[i];
                mv.resize(len);
                for (int k = 0; k < len; k++) {
                    const int j = h.A.col[a + k];
                    mv[k] = (j == i ? 2.0 * di : 0.0) - di * h.A.val[a + k] * (h.omega * h.dinv[j]);
                }
                S.tpl[i] = (tm.row(&h.A.col[a], mv.data(), &h.A.val[a], len, i) >> kSolveLenBits) / S.fine;
                if (S.tpl[i] > 0xffffu) tm.ok = false;
                if (!tm.ok) return S;
            }
            S.off = std::move(tm.off);
            S.vm = std::move(tm.v);
            S.va = std::move(tm.v2);
        }
        if (l >= S.clev) break;   // the finest level is the coarsest
        fold(h, l > 0 ? &o.m : nullptr, o.p, o.r);
    }
    // Rows of the coarse levels in the order of the fine rows they stand for:
    // aggregation numbers leftover rows (the pinned cell, corners) last, and a
    // rank that owned them would hold most of every vector.
    std::vector<int> fine_pos;
    for (int l = 0; l < S.clev; l++) {
        const hf::HostLevel &h = H[l];
        const int nn = h.R.n;
        std::vector<std::pair<double, int>> key(nn);
        double run = 0.0, span = 0.0;
        for (int pass = 0; pass < 2; pass++)
            for (int i = 0; i < nn; i++) {
                double sum = 0.0, lo = h.A.n, hi = 0.0;
                const int a = h.R.ptr[i], e = h.R.ptr[i + 1];
                for (int k = a; k < e; k++) {
                    const double c = l == 0 ? h.R.col[k] : fine_pos[h.R.col[k]];
                    sum += c;
                    lo = std::min(lo, c);
                    hi = std::max(hi, c);
                }
                if (pass == 0) {
                    span = std::max(span, hi - lo);
                    continue;
                }
                // rows that follow their predecessors keep their order (and the
                // regular numbering that makes rows share templates); a row far
                // behind them goes to its place
                const double mean = e > a ? sum / (e - a) : 0.0;
                const bool in_order = mean + span >= run;
                if (in_order) run = std::max(run, mean);
                key[i] = {in_order ? run : mean, i};
            }
        std::sort(key.begin(), key.end());
        std::vector<int> pos(nn);
        for (int i = 0; i < nn; i++) pos[key[i].second] = i;
        HostSolve::Level &o = S.L[l];
        o.r = permuted(o.r, pos, fine_pos);
        o.p = permuted(o.p, fine_pos, pos);
        if (l + 1 < S.clev) S.L[l + 1].m = permuted(S.L[l + 1].m, pos, pos);
        else S.cpos = pos;
        fine_pos = std::move(pos);
    }
    S.ndown = S.clev;
    S.ncb = S.nc;
    if (S.clev > 1) coarse_operator(S, inverse);
    ranges(S);
    S.ok = true;
    return S;
}

// Rows beyond which an instance fits no cluster: r, q, z and the row descriptors
// always lie in shared memory (with halos, coarse levels and operators beside
// them 73,000 rows of a square fit in FP64 and 130,000 in FP32, of these 109,000
// and 174,000)
template <typename T>
constexpr int most_rows()
{
    return kSolveMaxCluster * (kSolveSmem / (3 * (int)sizeof(T) + (int)sizeof(uint2)));
}

// the instance's tables and its shared-memory layout
template <typename T>
struct Packed {
    SInst<T> inst;
    std::vector<SRank> ranks;
    std::vector<char> tables, rank_tables;
    size_t smem = 0;
    bool ok = false;
};

template <typename T>
Packed<T> pack(const HostSolve &S, const std::vector<double> &inverse, bool mixed)
{
    Packed<T> K;
    SInst<T> &o = K.inst;
    memset(&o, 0, sizeof o);
    const int C = S.cluster, nt = S.threads;
    o.n = S.L[0].n;
    o.clev = S.clev;
    o.nc = S.nc;
    o.ndown = S.ndown;
    o.ncb = S.ncb;
    o.dist = !S.coarse.empty();
    for (int l = 0; l < (int)S.L.size(); l++) o.lvl[l] = S.L[l].n;
    size_t at = 0;
    auto round = [](size_t b) { return (b + 15) & ~size_t(15); };
    auto take = [&](size_t bytes) -> uint32_t {
        if (at + round(bytes) > (size_t)kSolveSmem) return kSolveGlobal;
        const uint32_t r = (uint32_t)at;
        at += round(bytes);
        return r;
    };
    // the vectors that are gathered from or exchanged always live in shared
    // memory, at element indices of 16 bits
    o.cvec = take(sizeof(T) * (S.ncb + S.nc));
    o.vr = take(sizeof(T) * S.held[0]);
    o.vz = take(sizeof(T) * S.held[1]);
    for (int l = 1; l < S.clev; l++) {
        o.vb[l] = S.g && l == S.clev - 1 ? o.cvec : take(sizeof(T) * S.held[2 * l]);
        o.vo[l] = take(sizeof(T) * S.held[2 * l + 1]);
        if (o.vb[l] == kSolveGlobal || o.vo[l] == kSolveGlobal) return K;
    }
    if (o.cvec == kSolveGlobal || o.vr == kSolveGlobal || o.vz == kSolveGlobal || at / sizeof(T) > 0xffff) return K;
    o.vq = take(sizeof(T) * S.held[0]);
    if (o.vq == kSolveGlobal) return K;
    const int own = (o.n + C - 1) / C;
    auto blob = [&](std::vector<char> &to, const void *data, size_t bytes) {
        const uint32_t g = (uint32_t)to.size();
        to.insert(to.end(), (const char *)data, (const char *)data + bytes);
        to.resize(round(to.size()), 0);
        return g;
    };
    auto part = [&](const void *data, size_t bytes) {
        STab t;
        t.bytes = (uint32_t)round(bytes);
        t.s = take(bytes);
        t.g = blob(K.tables, data, bytes);
        return t;
    };
    auto vals = [](const std::vector<double> &v) { return std::vector<T>(v.begin(), v.end()); };
    auto ents = [&](const std::vector<double> &v) {
        std::vector<SEnt<T>> e(v.size());
        memset((void *)e.data(), 0, e.size() * sizeof(SEnt<T>));
        for (size_t k = 0; k < e.size(); k++) {
            e[k].off = S.off[k] * (int)sizeof(T);
            e[k].v = (T)v[k];
        }
        return part(e.data(), e.size() * sizeof(SEnt<T>));
    };
    K.ranks.resize(C);
    memset((void *)K.ranks.data(), 0, C * sizeof(SRank));
    o.a = ents(S.va);
    o.m = ents(S.vm);
    if (o.a.s == kSolveGlobal || o.m.s == kSolveGlobal) return K;
    // element index of row i of a vector in rank k's shared memory
    auto elem = [&](uint32_t off, int vec, int k, int i) {
        return (uint32_t)(off / sizeof(T)) + (uint32_t)(i - S.rng[(size_t)vec * C + k].x);
    };
    // one operator's rows of every rank in slices; f adds row i's entries
    using Row = std::vector<std::pair<uint16_t, T>>;
    auto slices = [&](int rows, int lg_max, auto f, auto of) {
        size_t most = 0;
        std::vector<std::vector<char>> data(C);
        double entries = 0;
        std::vector<std::vector<Row>> R(C);
        for (int k = 0; k < C; k++) {
            int a, h;
            rank_rows(k, C, rows, a, h);
            R[k].resize(h - a);
            for (int i = a; i < h; i++) {
                f(k, i, R[k][i - a]);
                entries += (double)R[k][i - a].size();
            }
        }
        const int m = (rows + C - 1) / C;
        const double avg = entries / std::max(1, rows);
        // threads per row: while the block has idle threads and a thread keeps
        // a few entries
        int lg = 0;
        while (lg < lg_max && ((long)m << (lg + 1)) <= nt && avg > 3.0 * (1 << (lg + 1))) lg++;
        for (int k = 0; k < C; k++) {
            int a, h;
            rank_rows(k, C, rows, a, h);
            SOp &op = of(K.ranks[k]);
            op.row0 = a;
            op.rows = h - a;
            op.lg = lg;
            const int per = 32 >> lg, lanes = 1 << lg;
            op.nsl = (op.rows + per - 1) / per;
            std::vector<uint32_t> ptr(1, 0);
            std::vector<T> val;
            std::vector<uint16_t> idx;
            for (int s = 0; s < op.nsl; s++) {
                int turns = 0;
                for (int j = 0; j < per && s * per + j < op.rows; j++)
                    turns = std::max(turns, ((int)R[k][s * per + j].size() + lanes - 1) / lanes);
                const size_t b = val.size();
                val.resize(b + (size_t)turns * 32, T(0));
                idx.resize(b + (size_t)turns * 32, 0);
                for (int j = 0; j < per && s * per + j < op.rows; j++) {
                    const Row &row = R[k][s * per + j];
                    for (size_t q = 0; q < row.size(); q++) {
                        const size_t w = b + (q / lanes) * 32 + j * lanes + q % lanes;
                        idx[w] = row[q].first;
                        val[w] = row[q].second;
                    }
                }
                ptr.push_back((uint32_t)(val.size() / 32));
            }
            std::vector<char> &c = data[k];
            auto push = [&](const void *p, size_t bytes) {
                const uint32_t w = (uint32_t)c.size();
                c.insert(c.end(), (const char *)p, (const char *)p + bytes);
                c.resize(round(c.size()), 0);
                return w;
            };
            push(ptr.data(), ptr.size() * 4);
            op.val = push(val.data(), val.size() * sizeof(T));
            op.idx = push(idx.data(), idx.size() * 2);
            most = std::max(most, c.size());
        }
        const uint32_t s = take(most);
        for (int k = 0; k < C; k++) {
            SOp &op = of(K.ranks[k]);
            op.t.s = s;
            op.t.bytes = (uint32_t)data[k].size();
            op.t.g = blob(K.rank_tables, data[k].data(), data[k].size());
        }
    };
    auto add = [](Row &row, const Csr &A, int i, auto index) {
        for (int q = A.ptr[i]; q < A.ptr[i + 1]; q++) row.emplace_back((uint16_t)index(A.col[q]), (T)A.val[q]);
    };
    // level l's out (the coarsest level's: co)
    auto out_elem = [&](int l, int k, int i) {
        return l == S.clev ? (uint32_t)(o.cvec / sizeof(T)) + S.ncb + i : elem(o.vo[l], 2 * l + 1, k, i);
    };
    auto b_elem = [&](int l, int k, int i) { return l == 0 ? elem(o.vr, 0, k, i) : elem(o.vb[l], 2 * l, k, i); };
    // the finest level's Pt and Rt as templates, where that form is the smaller
    Tables tp, tr;
    std::vector<uint32_t> dp(o.n, 0), dr;
    int lg_r = 0;
    if (S.clev > 0) {
        const HostSolve::Level &L = S.L[0];
        tp.pad = 2;
        for (int i = 0; i < o.n; i++) {
            const int a = L.p.ptr[i], len = L.p.ptr[i + 1] - a;
            dp[i] = tp.row(L.p.col.data() + a, L.p.val.data() + a, nullptr, len, len ? L.p.col[a] : 0);
        }
        const int nr = L.r.rows(), m = (nr + C - 1) / C;
        while (lg_r < 5 && ((long)m << (lg_r + 1)) <= nt && L.r.col.size() > 3.0 * nr * (1 << (lg_r + 1))) lg_r++;
        tr.pad = 2 << lg_r;
        dr.resize(nr);
        for (int i = 0; i < nr; i++) {
            const int a = L.r.ptr[i], len = L.r.ptr[i + 1] - a;
            dr[i] = tr.row(L.r.col.data() + a, L.r.val.data() + a, nullptr, len, len ? L.r.col[a] : 0);
        }
        auto short_off = [](const Tables &t) {
            for (int32_t v : t.off)
                if (v < -32768 || v > 32767) return false;
            return t.ok;
        };
        const size_t eb = sizeof(T) + 2;
        // (with the row descriptors, and only where they fit beside the rest)
        const size_t room = kSolveSmem - std::min<size_t>(kSolveSmem, at + sizeof(uint2) * own + sizeof(uint2) * m + 64);
        const size_t bp = tp.off.size() * eb, br = tr.off.size() * eb;
        o.tpl_r = short_off(tr) && br + 64 < room && br < L.r.col.size() / C * eb / 2;
        o.tpl_p = short_off(tp) && bp + 64 < room - (o.tpl_r ? br : 0) && bp < L.p.col.size() / C * eb;
    }
    o.lg_r = lg_r;
    {
        // the finest level's own rows
        std::vector<std::vector<uint2>> d(C);
        for (int k = 0; k < C; k++) {
            int lo, hi;
            rank_rows(k, C, o.n, lo, hi);
            for (int i = lo; i < hi; i++) {
                uint32_t anchor = 0;
                if (S.clev > 0 && S.L[0].p.ptr[i + 1] > S.L[0].p.ptr[i]) anchor = out_elem(1, k, S.L[0].p.col[S.L[0].p.ptr[i]]);
                d[k].push_back(make_uint2(o.tpl_p ? dp[i] : 0u, anchor << 16 | S.tpl[i]));
            }
        }
        const uint32_t s = take(sizeof(uint2) * own);
        if (s == kSolveGlobal) return K;
        for (int k = 0; k < C; k++) {
            STab &t = K.ranks[k].desc0;
            t.s = s;
            t.bytes = (uint32_t)round(sizeof(uint2) * d[k].size());
            t.g = blob(K.rank_tables, d[k].data(), sizeof(uint2) * d[k].size());
        }
    }
    auto tables16 = [&](const Tables &t, STab &v, STab &f) {
        std::vector<T> tv = vals(t.v);
        std::vector<int16_t> to(t.off.begin(), t.off.end());
        v = part(tv.data(), tv.size() * sizeof(T));
        f = part(to.data(), to.size() * 2);
    };
    if (S.clev > 0) {
        const HostSolve::Level &L = S.L[0];
        if (o.tpl_r) {
            tables16(tr, o.trv, o.tro);
            std::vector<std::vector<uint2>> d(C);
            size_t most = 0;
            for (int k = 0; k < C; k++) {
                int a, h;
                rank_rows(k, C, L.r.rows(), a, h);
                for (int i = a; i < h; i++)
                    d[k].push_back(make_uint2(dr[i], L.r.ptr[i + 1] > L.r.ptr[i] ? b_elem(0, k, L.r.col[L.r.ptr[i]]) : 0u));
                most = std::max(most, d[k].size());
            }
            const uint32_t s = take(sizeof(uint2) * most);
            if (s == kSolveGlobal || o.trv.s == kSolveGlobal || o.tro.s == kSolveGlobal) return K;
            for (int k = 0; k < C; k++) {
                STab &t = K.ranks[k].desc_r;
                t.s = s;
                t.bytes = (uint32_t)round(sizeof(uint2) * d[k].size());
                t.g = blob(K.rank_tables, d[k].data(), sizeof(uint2) * d[k].size());
            }
        }
        if (o.tpl_p) {
            tables16(tp, o.tpv, o.tpo);
            if (o.tpv.s == kSolveGlobal || o.tpo.s == kSolveGlobal) return K;
        }
    }
    o.vp = take(sizeof(T) * own);
    o.vx = take((mixed ? sizeof(T) : sizeof(double)) * own);
    for (int l = S.clev - 1; l > 0; l--) {
        const HostSolve::Level &L = S.L[l];
        slices(L.n, 5, [&](int k, int i, Row &row) {
            add(row, L.m, i, [&](int c) { return b_elem(l, k, c); });
            add(row, L.p, i, [&](int c) { return out_elem(l + 1, k, c); });
        }, [l](SRank &r) -> SOp & { return r.up[l]; });
        if (l < S.ndown)
            slices(L.r.rows(), 5, [&](int k, int i, Row &row) { add(row, L.r, i, [&](int c) { return b_elem(l, k, c); }); },
                   [l](SRank &r) -> SOp & { return r.down[l]; });
    }
    if (o.dist) {
        slices(S.nc, 5, [&](int, int i, Row &row) {
            for (int j = 0; j < S.ncb; j++)
                row.emplace_back((uint16_t)(o.cvec / sizeof(T) + j), (T)S.coarse[(size_t)i * S.ncb + j]);
        }, [](SRank &r) -> SOp & { return r.coarse; });
    } else {
        std::vector<T> d(inverse.size());
        for (int i = 0; i < S.nc; i++)
            for (int j = 0; j < S.nc; j++)
                d[(size_t)(S.cpos.empty() ? i : S.cpos[i]) * S.nc + (S.cpos.empty() ? j : S.cpos[j])] =
                    (T)inverse[(size_t)i * S.nc + j];
        o.inv = part(d.data(), d.size() * sizeof(T));
    }
    if (S.clev > 0) {
        const HostSolve::Level &L = S.L[0];
        if (!o.tpl_r)
            slices(L.r.rows(), 5, [&](int k, int i, Row &row) { add(row, L.r, i, [&](int c) { return b_elem(0, k, c); }); },
                   [](SRank &r) -> SOp & { return r.down[0]; });
        if (!o.tpl_p)
            slices(L.n, 0, [&](int k, int i, Row &row) { add(row, L.p, i, [&](int c) { return out_elem(1, k, c); }); },
                   [](SRank &r) -> SOp & { return r.up[0]; });
    }
    if (mixed) {
        std::vector<SEnt<double>> e(S.off.size());
        for (size_t q = 0; q < e.size(); q++) e[q] = SEnt<double>{S.va[q], S.off[q], 0};
        o.a64.g = blob(K.tables, e.data(), e.size() * sizeof(SEnt<double>));
        o.a64.s = kSolveGlobal;
    }
    K.smem = at;
    K.ok = K.tables.size() < 0xffffffffu && K.rank_tables.size() < 0xffffffffu;
    return K;
}

}  // namespace solve
