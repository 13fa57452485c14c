// The semi-implicit velocity systems as one launch: the BiCGStab iteration of
// k_slv_init, k_bi_p, k_bi_spmv, k_bi_s and k_bi_update, one thread-block
// cluster per direction, from the initial guess to the converged velocity.
//
// What bounds it: launched one by one an iteration is five kernels of about 5 us
// on systems of 10^3 to 10^4 rows, queued in chunks that run past convergence
// and end in a host read; here the five phases are separated by cluster
// barriers.  Every rank keeps its rows' vectors, matrix rows and the halos of the
// two gathered vectors in shared memory.
//
// The arithmetic is that of the separate kernels to the last bit, sums included:
// partial sums cover the same 256 rows in the same order and are added in the
// same order.  (BiCGStab turns last-bit differences into differences of the size
// of its tolerance; a step's pressure follows them.)
#pragma once

#include <cstdint>

constexpr int kBiThreads = 1024;
constexpr int kBiSmem = 200 * 1024;          // dynamic shared memory
constexpr int kBiMaxCluster = 16;
constexpr int kBiMaxBlocks = 256;            // blocks of kBlock rows of one system

struct BiSys {
    int n, m;                 // rows; blocks of kBlock rows per rank
    int k;                    // most entries of a row
    int in_smem;              // the matrix is copied to shared memory
    uint32_t ext;             // rows a rank holds of a gathered vector (most)
    uint32_t rank_bytes;      // matrix bytes of a rank
    // per rank: lengths (uint8, m * kBlock), values (k x m * kBlock, entry by
    // entry), columns (uint16 indices into the rank's gathered rows)
    const char *mat;
    const int4 *rng;          // per rank: rows held [x, y), ranks [z, w] that hold some of its own
    const double *dinv, *b, *x0;
    double *x;
    Scal *sc;
};
struct BiArgs {
    BiSys s[3];
    double rtol, atol;
    int maxit;
};

namespace bicg {

extern __shared__ __align__(16) char dyn[];
__device__ __forceinline__ double &at(uint32_t off) { return *reinterpret_cast<double *>(dyn + off); }

struct Team {
    int rank, size, m, nvb;
    double (*wsum)[8];                      // [2 * m]: the warps' sums of the own blocks
    double (*blk)[2][kBiMaxBlocks];         // [2][value][block], double buffered
    double (*fin)[8];                       // [value]: sums of 32 blocks
    int par;
};

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

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;   // in lane 0
}
// the order in which block_sum adds eight warps' sums
__device__ __forceinline__ double add8(const double *x)
{
    return ((x[0] + x[4]) + (x[2] + x[6])) + ((x[1] + x[5]) + (x[3] + x[7]));
}

// one value per row in (the warps' sums of block j: wsum[2 j + v]), the grid's
// sums out, as grid_sum adds them: block by block in add8's order, the blocks'
// sums 32 at a time, these in add8's order.  A team barrier.
template <int NV>
__device__ __forceinline__ void team_sum(Team &t, double (&tot)[NV])
{
    const int tid = threadIdx.x, lane = tid & 31;
    __syncthreads();
    t.par ^= 1;
    const int mine = min(t.m, t.nvb - t.rank * t.m);
    for (int k = tid; k < mine * t.size * NV; k += blockDim.x) {
        const int to = k % t.size, j = k / t.size % mine, v = k / t.size / mine;
        const double s = add8(t.wsum[2 * j + v]);
        double *p = &t.blk[t.par][v][t.rank * t.m + j];
        if (t.size > 1) *cooperative_groups::this_cluster().map_shared_rank(p, to) = s;
        else *p = s;
    }
    team_sync(t);
    // a warp per value and 32 blocks (the sums of blocks that do not exist stay
    // zero)
    const int parts = (t.nvb + 31) / 32;
    for (int k = tid >> 5; k < NV * parts; k += blockDim.x >> 5) {
        const int v = k / parts, q = k % parts;
        const double s = warp_sum(32 * q + lane < t.nvb ? t.blk[t.par][v][32 * q + lane] : 0.0);
        if (lane == 0) t.fin[v][q] = s;
    }
    __syncthreads();
#pragma unroll
    for (int v = 0; v < NV; v++) tot[v] = add8(t.fin[v]);
}

}  // namespace bicg

// (64 registers a thread at 1,024 threads; ptxas spills 16 bytes beyond them)
__global__ void __launch_bounds__(kBiThreads, 1) k_bi_solve(const BiArgs *args)
{
    using bicg::at;
    __shared__ BiSys Y;
    __shared__ double wsum[2 * kBiMaxBlocks / 4][8];
    __shared__ double blk[2][2][kBiMaxBlocks];
    __shared__ double fin[2][8];
    __shared__ int4 rng[kBiMaxCluster];
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31;
    bicg::Team t;
    t.rank = (int)cooperative_groups::this_cluster().block_rank();
    t.size = (int)cooperative_groups::this_cluster().num_blocks();
    {
        const uint32_t *src = reinterpret_cast<const uint32_t *>(&args->s[blockIdx.x / t.size]);
        for (int k = tid; k < (int)(sizeof(BiSys) / 4); k += nt) reinterpret_cast<uint32_t *>(&Y)[k] = src[k];
    }
    __syncthreads();
    const int n = Y.n, rows = Y.m * kBlock;
    t.m = Y.m;
    t.nvb = (n + kBlock - 1) / kBlock;
    t.wsum = wsum;
    t.blk = blk;
    t.fin = fin;
    if (tid < 16) (&fin[0][0])[tid] = 0.0;
    t.par = 0;
    if (tid < t.size) rng[tid] = Y.rng[tid];
    const int lo = min(n, t.rank * rows), own = min(n, lo + rows) - lo;
    // shared memory: own rows of x, r, rh, p, v, s, t, dinv; ph and sh over the
    // rows held; the matrix
    const uint32_t vb = 8u * (uint32_t)rows;
    const uint32_t ox = 0, orr = vb, orh = 2 * vb, op = 3 * vb, ov = 4 * vb, os = 5 * vb, ot = 6 * vb, od = 7 * vb;
    const uint32_t oph = 8 * vb, osh = oph + 8u * Y.ext, om = osh + 8u * Y.ext;
    const char *mat = Y.mat + (size_t)t.rank * Y.rank_bytes;
    if (Y.in_smem) {
        for (uint32_t k = tid; k < Y.rank_bytes / 16; k += nt)
            *reinterpret_cast<uint4 *>(bicg::dyn + om + 16 * k) = __ldg(reinterpret_cast<const uint4 *>(mat) + k);
        mat = bicg::dyn + om;
    }
    __syncthreads();
    const int xlo = rng[t.rank].x, klo = rng[t.rank].z, khi = rng[t.rank].w;
    const uint8_t *len = reinterpret_cast<const uint8_t *>(mat);
    const double *val = reinterpret_cast<const double *>(mat + rows);
    const uint16_t *idx = reinterpret_cast<const uint16_t *>(mat + rows + 8 * (size_t)Y.k * rows);
    // an own row's value into a gathered vector, every holder's copy
    auto put = [&](uint32_t base, int li, double v) {
        const int i = lo + li;
        at(base + 8u * (uint32_t)(i - xlo)) = v;
        for (int k = klo; k <= khi; k++) {
            if (k == t.rank) continue;
            const int4 g = rng[k];
            if (i >= g.x && i < g.y)
                *cooperative_groups::this_cluster().map_shared_rank(&at(base + 8u * (uint32_t)(i - g.x)), k) = v;
        }
    };
    auto spmv = [&](uint32_t base, int li) {
        double acc = 0.0;
        const int e = len[li];
        for (int k = 0; k < e; k++) acc += val[(size_t)k * rows + li] * at(base + 8u * idx[(size_t)k * rows + li]);
        return acc;
    };
    // f(li) for every own row, by whole warps; the warps' sums of what it
    // returns go to wsum
    auto each = [&](auto nv, auto f) {
        constexpr int NV = decltype(nv)::value;
        for (int b = tid & ~31; b < rows; b += nt) {
            double part[2] = {0.0, 0.0};
            if (b + lane < own) f(b + lane, part);
#pragma unroll
            for (int v = 0; v < NV; v++) {
                const double s = bicg::warp_sum(part[v]);
                if (lane == 0) wsum[2 * (b / kBlock) + v][(b >> 5) & 7] = s;
            }
        }
    };
    using None = std::integral_constant<int, 0>;
    using One = std::integral_constant<int, 1>;
    using Two = std::integral_constant<int, 2>;

    for (int li = tid; li < own; li += nt) {
        at(ox + 8 * li) = Y.x0[lo + li];
        at(od + 8 * li) = Y.dinv[lo + li];
    }
    bicg::team_sync(t);   // every CTA has started (its shared memory may be written)
    double tol2 = 0.0, rr = 0.0, bb = 0.0, rho = 1.0, alpha = 1.0, omega = 1.0, rho1 = 0.0, beta = 0.0;
    int status = 0, iters = 0;
    for (int restarts = 0;; restarts++) {
        // k_slv_init: r = b - A x
        for (int li = tid; li < own; li += nt) put(oph, li, at(ox + 8 * li));
        bicg::team_sync(t);
        each(Two{}, [&](int li, double (&part)[2]) {
            const double b = Y.b[lo + li], r = b - spmv(oph, li);
            at(orr + 8 * li) = r;
            at(orh + 8 * li) = r;
            at(op + 8 * li) = 0.0;
            at(ov + 8 * li) = 0.0;
            part[0] = r * r;
            part[1] = b * b;
        });
        double two[2];
        bicg::team_sum<2>(t, two);
        rr = two[0];
        if (restarts == 0) {
            bb = two[1];
            const double tol = fmax(args->rtol * sqrt(two[1]), args->atol);
            tol2 = tol * tol;
        }
        rho = alpha = omega = 1.0;
        rho1 = two[0];
        beta = 0.0;
        status = 0;
        bool done = !(two[0] > tol2);
        if (!finite(two[0])) {
            status = HF_ERR_NAN;
            done = true;
        }
        while (!done) {
            each(None{}, [&](int li, double (&)[2]) {
                const double p = at(orr + 8 * li) + beta * (at(op + 8 * li) - omega * at(ov + 8 * li));
                at(op + 8 * li) = p;
                put(oph, li, at(od + 8 * li) * p);
            });
            bicg::team_sync(t);
            each(One{}, [&](int li, double (&part)[2]) {
                const double acc = spmv(oph, li);
                at(ov + 8 * li) = acc;
                part[0] = at(orh + 8 * li) * acc;
            });
            double one[1];
            bicg::team_sum<1>(t, one);
            if (one[0] == 0.0 || !finite(one[0])) {
                status = finite(one[0]) ? 1 : HF_ERR_NAN;
                break;
            }
            alpha = rho1 / one[0];
            each(None{}, [&](int li, double (&)[2]) {
                const double s = at(orr + 8 * li) - alpha * at(ov + 8 * li);
                at(os + 8 * li) = s;
                put(osh, li, at(od + 8 * li) * s);
            });
            bicg::team_sync(t);
            each(Two{}, [&](int li, double (&part)[2]) {
                const double acc = spmv(osh, li);
                at(ot + 8 * li) = acc;
                part[0] = acc * at(os + 8 * li);
                part[1] = acc * acc;
            });
            bicg::team_sum<2>(t, two);
            omega = two[1] > 0.0 ? two[0] / two[1] : 0.0;
            if (!finite(omega)) {
                status = HF_ERR_NAN;
                break;
            }
            each(Two{}, [&](int li, double (&part)[2]) {
                const uint32_t g = 8u * (uint32_t)(lo + li - xlo);
                at(ox + 8 * li) += alpha * at(oph + g) + omega * at(osh + g);
                const double r = at(os + 8 * li) - omega * at(ot + 8 * li);
                at(orr + 8 * li) = r;
                part[0] = r * r;
                part[1] = at(orh + 8 * li) * r;
            });
            bicg::team_sum<2>(t, two);
            rr = two[0];
            rho = rho1;
            rho1 = two[1];
            iters++;
            if (!finite(two[0])) {
                status = HF_ERR_NAN;
                done = true;
            } else if (!(two[0] > tol2)) {
                done = true;
            } else if (iters >= args->maxit) {
                status = HF_ERR_NOT_CONVERGED;
                done = true;
            } else if (rho1 == 0.0 || omega == 0.0) {   // breakdown: restart
                status = 1;
                done = true;
            } else {
                beta = (rho1 / rho) * (alpha / omega);
            }
        }
        if (!(status == 1 && restarts < 50)) break;   // breakdown: restart from x
    }
    for (int li = tid; li < own; li += nt) Y.x[lo + li] = at(ox + 8 * li);
    if (tid == 0 && t.rank == 0) {
        Scal &s = *Y.sc;
        s.rr = rr;
        s.bb = bb;
        s.tol2 = tol2;
        s.iters = iters;
        s.status = status;
        s.done = 1;
    }
    bicg::team_sync(t);   // no CTA leaves while another may still write to its shared memory
}

// host: one system's rows for the ranks of a cluster; empty where it does not fit
namespace bicg {

struct Packed {
    bool ok = false;
    int cluster = 1, m = 1, k = 0, in_smem = 0, threads = kBiThreads;
    uint32_t ext = 0, rank_bytes = 0;
    size_t smem = 0;
    std::vector<char> mat;
    std::vector<int4> rng;
};

// cluster: the same for every system of a launch
inline int cluster_size(int n)
{
    int c = 1;
    while (c < kBiMaxCluster && (long)c * 512 < n) c *= 2;
    return c;
}

inline Packed pack(const std::vector<int32_t> &ptr, const std::vector<int32_t> &col, const std::vector<double> &val, int C)
{
    Packed P;
    const int n = (int)ptr.size() - 1, nvb = (n + kBlock - 1) / kBlock;
    P.cluster = C;
    P.m = (nvb + C - 1) / C;
    if (nvb > kBiMaxBlocks || P.m > kBiMaxBlocks / 4) return P;
    const int rows = P.m * kBlock;
    P.threads = std::min(kBiThreads, rows);
    for (int i = 0; i < n; i++) P.k = std::max(P.k, ptr[i + 1] - ptr[i]);
    if (P.k > 255) return P;
    P.rng.resize(C);
    for (int r = 0; r < C; r++) {
        const int lo = std::min(n, r * rows), hi = std::min(n, lo + rows);
        int4 g = make_int4(lo, hi, r, r);
        for (int k = ptr[lo]; k < ptr[hi]; k++) {
            g.x = std::min(g.x, col[k]);
            g.y = std::max(g.y, col[k] + 1);
        }
        P.rng[r] = g;
        P.ext = std::max(P.ext, (uint32_t)(g.y - g.x));
    }
    if (P.ext > 0xffffu) return P;
    for (int r = 0; r < C; r++) {
        const int lo = std::min(n, r * rows), hi = std::min(n, lo + rows);
        for (int j = 0; j < C; j++)
            if (P.rng[j].x < hi && P.rng[j].y > lo) {
                P.rng[r].z = std::min(P.rng[r].z, j);
                P.rng[r].w = std::max(P.rng[r].w, j);
            }
    }
    P.rank_bytes = (uint32_t)(((size_t)rows * (1 + 10 * (size_t)P.k) + 15) & ~size_t(15));
    const size_t vecs = 8 * (8 * (size_t)rows + 2 * (size_t)P.ext);
    if (vecs > (size_t)kBiSmem) return P;
    P.in_smem = vecs + P.rank_bytes <= (size_t)kBiSmem;
    P.smem = vecs + (P.in_smem ? P.rank_bytes : 0);
    P.mat.assign((size_t)P.rank_bytes * C, 0);
    for (int i = 0; i < n; i++) {
        const int r = i / rows, li = i % rows;
        char *b = P.mat.data() + (size_t)r * P.rank_bytes;
        b[li] = (char)(ptr[i + 1] - ptr[i]);
        double *v = reinterpret_cast<double *>(b + rows);
        uint16_t *x = reinterpret_cast<uint16_t *>(b + rows + 8 * (size_t)P.k * rows);
        for (int k = 0; k < ptr[i + 1] - ptr[i]; k++) {
            v[(size_t)k * rows + li] = val[ptr[i] + k];
            x[(size_t)k * rows + li] = (uint16_t)(col[ptr[i] + k] - P.rng[r].x);
        }
    }
    P.ok = true;
    return P;
}

}  // namespace bicg
