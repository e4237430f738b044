// many.cu -- Linear_EQS::CG and ::BiCGStab (FEM/equation_class.cpp:1129-1187,
// 1287-1420) with many iterations per launch.
//
// The kernels of krylov.cu run one step of an iteration each.  A launch here
// runs whole iterations instead: a block owns a contiguous share of the
// rows, keeps its part of the vectors in shared memory as far as they fit,
// and publishes only the vector the products of other blocks read.  What it saves per iteration: three to five launches
// with their gaps and the last-block sums behind them, and the vector
// traffic through L2.  What stays is the FP64 pipe (a warp's instruction
// takes 17.7 cycles of its SM): one FMA a stored entry and the 6 (CG) or 14
// (BiCGStab) operations a row of the vectors, and the waits.
//
// Every iteration waits where its data demands it: CG after the product (p .
// s), after the update (r . r, r . z) and before the next product (p
// published); BiCGStab after p_h, v, s_h, t and r.  A wait is one counter in
// global memory (1.3 us for 152 blocks), or the hardware barrier where the
// grid is one cluster (about 0.7 us with the published vector).  The
// arithmetic per entry and row is that of krylov.cu; the sums are grouped
// by thread and block of this launch, in a fixed order.
#include <algorithm>
#include <cfloat>

#include <cuda.h>

#include "krylov.cuh"

namespace ogs {

namespace {

constexpr int kManyMaxSmem = 208 * 1024;
// The same where a row's columns lie anywhere (no few diagonals): loads from
// as many places need L1 to be under way at the same time, and the vectors in
// shared memory take it away.  us per BiCGStab iteration with 208 / 140 / 64
// KB and of the graph: hexes of 531k rows in random order 313 / 155 / 145 / 166,
// in runs of eight 148 / 99 / 100 / 118; tets of 754k rows 242 / 132 / 131 / 145
constexpr int kManyScatteredSmem = 140 * 1024;
constexpr int64_t kManyClusterWork = 155 * 1000, kManySharedWork = 600 * 1000;
// FP64 operations of an iteration up to which a half and a third of the SMs are
// as fast as all of them, where a thread has one row; the solves of several
// threads then run beside each other.  us per iteration of one thread's and of
// eight threads' solves, all SMs / here / single-step graphs: CG quads 11.8k rows 9.5,
// 8.7 / 9.5, 3.0 / 17.1, 3.2; hexes 9.3k 10.2, 9.3 / 10.3, 4.7 / 19.9, 3.6; BiCGStab tets
// 16.3k 19.4, 17.9 / 19.2, 9.1 / 35.2, 6.7.  Half of the SMs for hexes of 16k rows
// (540,000 operations) would cost the one thread 4%
constexpr int64_t kManyPartWork[4] = {0, 0, 340 * 1000, 200 * 1000};
// Rows per SM above which the graph's kernels, with more warps to hide the
// memory behind, are as fast: by method, and for rows whose entries come in
// nines (quads, hexes) and others (tets: the last of their 15 entries go
// three at a time).  us per iteration, here / graph, of million rows:
//   CG       quads 2.56 101/112, 3.24 141/135, 5.5 287/215; hexes 2.8 206/214, 3.7 321/273;
//            tets 0.75 54/57, 1.03 71/70, 2.0 127/113
//   BiCGStab quads 1.57 150/167, 1.96 207/208, 2.56 273/263; hexes 2.25 384/396, 2.8 482/478;
//            tets 1.37 175/180, 2.0 293/257
constexpr int kManyRowsCg = 17000, kManyRowsBi = 12500, kManyOddRowsCg = 5500, kManyOddRowsBi = 9200;

// v into `slot` of block `rank` of the cluster (distributed shared memory)
__device__ __forceinline__ void cluster_store(double* slot, unsigned rank, double v)
{
    const unsigned a = (unsigned)__cvta_generic_to_shared(slot);
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(r), "d"(v) : "memory");
}

__device__ __forceinline__ void many_cluster_sync()
{
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Row product with nine entries' loads in flight; x changes during the
// launch (coherent loads), the matrix does not.  STREAM: the matrix is
// larger than what stays in L2 (evict-first loads).
template <bool STREAM>
__device__ __forceinline__ double many_row(const SellView<double>& A, const double* x, int row)
{
    const int s = row >> 5;
    const int b0 = __ldg(A.slice_ptr + s), b1 = __ldg(A.slice_ptr + s + 1);
    const int w = (b1 - b0) >> 5;
    const int beg = b0 + (row & 31);
    constexpr int U = 9;
    double acc = 0.0;
    int j = 0;
    for (; j + U <= w; j += U)
    {
        double m[U], xv[U];
        int c[U];
#pragma unroll
        for (int q = 0; q < U; q++)
        {
            const int k = beg + ((j + q) << 5);
            c[q] = STREAM ? __ldcs(A.col + k) : __ldg(A.col + k);
            m[q] = STREAM ? __ldcs(A.val + k) : __ldg(A.val + k);
        }
#pragma unroll
        for (int q = 0; q < U; q++) xv[q] = OGS_IN(c[q], A.n, kOobSpmvCol) ? x[c[q]] : 0.0;
#pragma unroll
        for (int q = 0; q < U; q++) acc += m[q] * xv[q];
    }
#pragma unroll 3
    for (; j < w; j++)
    {
        const int k = beg + (j << 5);
        const int c = STREAM ? __ldcs(A.col + k) : __ldg(A.col + k);
        if (OGS_IN(c, A.n, kOobSpmvCol)) acc += (STREAM ? __ldcs(A.val + k) : __ldg(A.val + k)) * x[c];
    }
    return acc;
}

// The waits of one launch.  Thread 0 of warp k < NV arrives and waits for
// value k; ok falls to false in every thread of the block once a wait of it
// gave up.
template <int NT, bool CLUSTER>
struct ManySync
{
    KState* st;
    unsigned arrived = 0;  // arrivals that complete the last barrier
    unsigned seq = 0;      // sums so far
    double (*red)[NT];
    double (*parts)[2][16];  // CLUSTER: every block's partial sums, written by their blocks
    double* tot;
    int* fail;
    int used;  // threads that have rows
    const unsigned* limit;  // polls of one wait (in shared memory)

    // The launch's start: this block's shared memory is set up, and every
    // block of the cluster has started.  Until then its shared memory may not
    // be there, and a block without rows reaches its first remote store
    // within a microsecond
    __device__ __forceinline__ void enter()
    {
        if (CLUSTER) many_cluster_sync();
        else __syncthreads();
    }
    // Sums of v[0 .. NV) over the grid, in every thread.  Each value is
    // added by one warp: the block's values, then the blocks' partial sums
    // (FP64 adds of whole blocks would take the pipe from all warps)
    template <int NV>
    __device__ __forceinline__ bool sum(const double (&v)[NV], double (&out)[NV])
    {
        const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
#pragma unroll
        for (int k = 0; k < NV; k++) red[k][tid] = v[k];
        __syncthreads();
        arrived += NV * gridDim.x;
        // two buffers in turn: a block writes the next sum's partials while a
        // slower one still reads this sum's
        const int par = seq++ & 1;
        double* part = st->part[2 + par] + wid * kMaxBlocks;
        if (NT > 256)
        {
            // 256 values a warp first
            if (wid < NV * (NT / 256))
            {
                const int k = wid % NV, g = wid / NV * 256;
                double q = red[k][g + lane];
#pragma unroll
                for (int t = 32; t < 256; t += 32) q += red[k][g + lane + t];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
                __syncwarp();
                if (lane == 0) red[k][g] = q;
            }
            __syncthreads();
        }
        if (wid < NV)
        {
            double q = red[wid][NT > 256 ? 0 : lane];
            if (NT > 256)
            {
#pragma unroll
                for (int t = 256; t < NT; t += 256) q += red[wid][t];
            }
            else
            {
#pragma unroll
                for (int t = 32; t < NT; t += 32)
                    if (t < used) q += red[wid][lane + t];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
            }
            if (CLUSTER)
            {
                if (lane < 16) cluster_store(&parts[par][wid][blockIdx.x], lane, q);
            }
            else if (lane == 0)
            {
                __stcg(part + blockIdx.x, q);
                asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&st->bar_count) : "memory");
                if (!grid_wait(st, arrived, limit)) *fail = 1;
            }
            __syncwarp();
        }
        if (CLUSTER) many_cluster_sync();
        if (wid < NV)
        {
            double q;
            if (CLUSTER)
            {
                q = parts[par][wid][lane & 15];
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
            }
            else
                q = half_warp_partials(part, gridDim.x, lane & 15);
            if (lane == 0) tot[wid] = q;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < NV; k++) out[k] = tot[k];
        return *fail == 0;
    }
    // all blocks' writes before, visible after
    __device__ __forceinline__ bool publish()
    {
        if (CLUSTER)
        {
            many_cluster_sync();
            return true;
        }
        __syncthreads();
        arrived += gridDim.x;
        if (threadIdx.x == 0)
        {
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&st->bar_count) : "memory");
            if (!grid_wait(st, arrived, limit)) *fail = 1;
        }
        __syncthreads();
        return *fail == 0;
    }
    // the launch's end; false: a wait gave up
    __device__ __forceinline__ void leave()
    {
        // no block's shared memory may go while others write to it
        if (CLUSTER) many_cluster_sync();
        if (threadIdx.x != 0) return;
        if (*fail)
        {
            st->bar_err = 1;
            st->status = OGS_CUDA_ERROR;
            st->done = 1;
        }
        else if (!CLUSTER)
            grid_leave(st);
    }
};

// |r| / |b| < tol from r . r: compared as squares on their bits, except
// near the limits of double's range
struct ManyGoal
{
    double tol, bnorm, goal2;
    bool plain;
    __device__ explicit ManyGoal(const KState* st) : tol(st->tol), bnorm(st->bnorm)
    {
        const double g = tol * bnorm;
        goal2 = g * g;
        plain = goal2 > 1e-280 && goal2 < 1e280;
    }
    __device__ __forceinline__ bool reached(double rr) const
    {
        return plain ? less_bits(rr, goal2) : sqrt(rr) / bnorm < tol;
    }
};

}  // namespace

// The block's part of a vector: the next `per` doubles of shared memory when
// bit `bit` of lay is set (copied from global memory where it has a value
// yet), else the rows in global memory
__device__ __forceinline__ double* many_part(double*& next, int per, int lay, int bit, double* global)
{
    if (!(lay >> bit & 1)) return global;
    double* p = next;
    next += per;
    return p;
}

// The vectors in the order in which they get shared memory: CG s, r, p, x,
// dinv; BiCGStab s, t, r, v, p, r0, dinv
constexpr int kCgVecs = 5, kBiVecs = 7;

template <int PC, int NT, bool CLUSTER, bool STREAM>
__global__ void __launch_bounds__(NT, 1) k_cg_many(SolveArgs a, int per, int lay, int iters)
{
    extern __shared__ double many_smem[];
    __shared__ double red[2][NT], parts[2][2][16], tot[2], s_sc[2];
    __shared__ int s_fail, s_stop;
    __shared__ unsigned s_limit;
    KState* st = a.st;
    if (st->done) return;  // uniform: nothing writes it before every block has passed a wait
    const int n = a.A.n, tid = threadIdx.x;
    const int row0 = blockIdx.x * per, cnt = max(0, min(per, n - row0));
    double* next = many_smem;
    double* ss = many_part(next, per, lay, 0, a.v.s + row0);
    double* sr = many_part(next, per, lay, 1, a.v.r + row0);
    double* sp = many_part(next, per, lay, 2, a.v.p + row0);
    double* X = many_part(next, per, lay, 3, a.v.x + row0);
    double* D = many_part(next, per, lay, 4, a.v.dinv + row0);
    if (tid == 0)
    {
        s_fail = 0;
        s_limit = st->spin_limit ? st->spin_limit : kGridSpins;
    }
    for (int k = tid; k < cnt; k += NT)
    {
        if (lay & 2) sr[k] = a.v.r[row0 + k];
        if (lay & 4) sp[k] = a.v.p[row0 + k];
        if (lay & 8) X[k] = a.v.x[row0 + k];
        if (lay & 16) D[k] = a.v.dinv[row0 + k];
    }
    ManySync<NT, CLUSTER> sync{st, 0, 0, red, parts, tot, &s_fail, min(per, NT), &s_limit};
    sync.enter();
    // scalars of thread 0
    const int it0 = st->iter, max_iter = st->max_iter;
    int it = it0, stop = -1;
    double rz = it0 == st->base_iter ? st->rz_base : st->rz_hist[it0 & 1], inv_rz = 1.0 / rz, rr = 0.0;
    const ManyGoal goal(st);
    bool ok = true;
    for (int t = 0; t < iters; t++)
    {
        double ps[1] = {0.0}, v[2] = {0.0, 0.0}, g[2];
        for (int k = tid; k < cnt; k += NT)
        {
            const double s = many_row<STREAM>(a.A, a.v.p, row0 + k);
            ss[k] = s;
            ps[0] += sp[k] * s;
        }
        double q[1];
        if (!(ok = sync.sum(ps, q))) break;
        if (tid == 0) s_sc[0] = rz / q[0];
        __syncthreads();
        const double alpha = s_sc[0];
        for (int k = tid; k < cnt; k += NT)
        {
            const double r = sr[k] - alpha * ss[k];
            const double z = PC == 1 ? r * D[k] : r;
            sr[k] = r;
            ss[k] = z;
            v[0] += r * r;
            v[1] += PC == 1 ? z * r : r * r;
        }
        if (!(ok = sync.sum(v, g))) break;
        if (tid == 0)
        {
            it += 1;
            rr = g[0];
            stop = !finite_bits(rr) ? OGS_NONFINITE : goal.reached(rr) ? OGS_OK : it >= max_iter ? OGS_NOT_CONVERGED : -1;
            s_stop = stop;
            s_sc[1] = rz > 1e-290 ? g[1] * inv_rz : g[1] / rz;  // (1 / rz formed off this path)
            rz = g[1];
        }
        __syncthreads();
        const double beta = s_sc[1];
        const bool last = s_stop >= 0;
        for (int k = tid; k < cnt; k += NT)
        {
            const double p = sp[k];
            X[k] += alpha * p;
            const double pn = ss[k] + beta * p;
            if (lay & 4) sp[k] = pn;
            if (!last) a.v.p[row0 + k] = pn;
        }
        if (last) break;
        if (tid == 0) inv_rz = 1.0 / rz;
        if (!(ok = sync.publish())) break;
    }
    for (int k = tid; k < cnt; k += NT)
    {
        if (lay & 2) a.v.r[row0 + k] = sr[k];
        if (lay & 8) a.v.x[row0 + k] = X[k];
    }
    sync.leave();
    if (!ok || blockIdx.x != 0 || tid != 0) return;
    st->iter = it;
    st->rz_hist[it & 1] = rz;
    if (it > it0) st->error = sqrt(rr) / st->bnorm;
    if (stop >= 0)
    {
        st->status = stop;
        st->done = 1;
    }
}

template <int PC, int NT, bool CLUSTER, bool STREAM>
__global__ void __launch_bounds__(NT, 1) k_bi_many(SolveArgs a, int per, int lay, int iters)
{
    extern __shared__ double many_smem[];
    __shared__ double red[2][NT], parts[2][2][16], tot[2], s_sc[3];
    __shared__ int s_fail, s_stop;
    __shared__ unsigned s_limit;
    KState* st = a.st;
    if (st->done) return;
    const int n = a.A.n, tid = threadIdx.x;
    const int row0 = blockIdx.x * per, cnt = max(0, min(per, n - row0));
    double* next = many_smem;
    double* ss = many_part(next, per, lay, 0, a.v.s + row0);
    double* stt = many_part(next, per, lay, 1, a.v.t + row0);
    double* sr = many_part(next, per, lay, 2, a.v.r + row0);
    double* sv = many_part(next, per, lay, 3, a.v.v + row0);
    double* sp = many_part(next, per, lay, 4, a.v.p + row0);
    double* s0 = many_part(next, per, lay, 5, a.v.r0 + row0);
    double* D = many_part(next, per, lay, 6, a.v.dinv + row0);
    if (tid == 0)
    {
        s_fail = 0;
        s_limit = st->spin_limit ? st->spin_limit : kGridSpins;
    }
    for (int k = tid; k < cnt; k += NT)
    {
        if (lay & 4) sr[k] = a.v.r[row0 + k];
        if (lay & 8) sv[k] = a.v.v[row0 + k];
        if (lay & 16) sp[k] = a.v.p[row0 + k];
        if (lay & 32) s0[k] = a.v.r0[row0 + k];
        if (lay & 64) D[k] = a.v.dinv[row0 + k];
    }
    ManySync<NT, CLUSTER> sync{st, 0, 0, red, parts, tot, &s_fail, min(per, NT), &s_limit};
    sync.enter();
    const int max_iter = st->max_iter;
    int it = st->iter, stop = -1, finish = 0;
    double alpha = st->alpha, omega = st->omega, beta = st->beta, rho0 = st->rho0, rho1 = st->rho1, nrm = -1.0;
    const ManyGoal goal(st);
    bool ok = true;
    for (int t = 0; t < iters; t++)
    {
        // p = r (first) or r + beta (p - omega v) ; p_h = M^-1 p
        const bool first = it == 1;
        for (int k = tid; k < cnt; k += NT)
        {
            const double p = first ? sr[k] : sr[k] + beta * (sp[k] - omega * sv[k]);
            sp[k] = p;
            a.v.ph[row0 + k] = PC == 1 ? p * D[k] : p;
        }
        if (!(ok = sync.publish())) break;
        double d1[1] = {0.0}, o1[1], d2[2] = {0.0, 0.0}, o2[2], n1[1] = {0.0};
        for (int k = tid; k < cnt; k += NT)
        {
            const double v = many_row<STREAM>(a.A, a.v.ph, row0 + k);
            sv[k] = v;
            d1[0] += s0[k] * v;
        }
        if (!(ok = sync.sum(d1, o1))) break;
        if (tid == 0) s_sc[0] = rho1 / o1[0];
        __syncthreads();
        alpha = s_sc[0];
        for (int k = tid; k < cnt; k += NT)
        {
            const double s = sr[k] - alpha * sv[k];
            ss[k] = s;
            a.v.sh[row0 + k] = PC == 1 ? s * D[k] : s;
            n1[0] += s * s;
        }
        // the sum's wait also publishes s_h
        if (!(ok = sync.sum(n1, o1))) break;
        nrm = o1[0];
        if (!finite_bits(nrm)) { stop = OGS_NONFINITE; break; }
        if (goal.reached(nrm)) { stop = OGS_OK; finish = 1; break; }
        for (int k = tid; k < cnt; k += NT)
        {
            const double v = many_row<STREAM>(a.A, a.v.sh, row0 + k);
            stt[k] = v;
            d2[0] += v * v;
            d2[1] += v * ss[k];
        }
        if (!(ok = sync.sum(d2, o2))) break;
        if (tid == 0) s_sc[1] = o2[0] > DBL_MIN ? o2[1] / o2[0] : 1.0;
        __syncthreads();
        omega = s_sc[1];
        d2[0] = d2[1] = 0.0;
        for (int k = tid; k < cnt; k += NT)
        {
            const double s = ss[k];
            a.v.x[row0 + k] += alpha * a.v.ph[row0 + k] + omega * a.v.sh[row0 + k];
            const double r = s - omega * stt[k];
            sr[k] = r;
            d2[0] += r * r;
            d2[1] += s0[k] * r;
        }
        if (!(ok = sync.sum(d2, o2))) break;
        nrm = o2[0];
        rho0 = rho1;
        // the tests in the order of Linear_EQS::BiCGStab, alike in every thread
        if (!finite_bits(nrm)) { stop = OGS_NONFINITE; break; }
        if (goal.reached(nrm)) { stop = OGS_OK; break; }
        if (less_bits(fabs(omega), DBL_MIN)) { stop = OGS_BREAKDOWN; break; }
        if (it >= max_iter) { stop = OGS_NOT_CONVERGED; break; }
        rho1 = o2[1];
        if (less_bits(fabs(rho1), DBL_MIN)) { stop = OGS_BREAKDOWN; break; }
        if (tid == 0) s_sc[2] = (rho1 / rho0) * (alpha / omega);
        __syncthreads();
        beta = s_sc[2];
        it += 1;
    }
    for (int k = tid; k < cnt; k += NT)
    {
        if (lay & 4) a.v.r[row0 + k] = sr[k];
        if (lay & 8) a.v.v[row0 + k] = sv[k];
        if (lay & 16) a.v.p[row0 + k] = sp[k];
    }
    sync.leave();
    if (!ok || blockIdx.x != 0 || tid != 0) return;
    st->iter = it;
    st->alpha = alpha;
    st->omega = omega;
    st->beta = beta;
    st->rho0 = rho0;
    st->rho1 = rho1;
    if (nrm >= 0.0 || nrm != nrm) st->error = sqrt(nrm) / st->bnorm;
    if (finish) st->finish_s = 1;
    if (stop >= 0)
    {
        st->status = stop;
        st->done = 1;
    }
}

// ------------------------------------------------------------------
// plan and launch
// ------------------------------------------------------------------
using ManyKernel = void (*)(SolveArgs, int, int, int);

template <int PC, int NT, bool CL>
static const void* many_kernel(int kind, bool stream)
{
    ManyKernel k = kind == SK_CG ? k_cg_many<PC, NT, CL, false> : k_bi_many<PC, NT, CL, false>;
    if constexpr (!CL)  // a cluster's systems are far smaller than L2
        if (stream) k = kind == SK_CG ? k_cg_many<PC, NT, CL, true> : k_bi_many<PC, NT, CL, true>;
    return (const void*)k;
}

constexpr int kManyWide = 512;

// A stream made in a green context has part of the SMs, which neither the
// device's SM count nor the occupancy queries tell
static bool has_all_sms(cudaStream_t s)
{
    using GetGreenCtx = CUresult (*)(CUstream, CUgreenCtx*);
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion("cuStreamGetGreenCtx", &f, 12040, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess || !f)
    {
        cudaGetLastError();
        return true;  // no green contexts in this CUDA version
    }
    CUgreenCtx g = nullptr;
    return ((GetGreenCtx)f)(s, &g) != CUDA_SUCCESS || !g;
}

bool resident_together(const void* kernel, int grid, int threads, size_t smem, bool cluster, cudaStream_t s)
{
    if (!has_all_sms(s)) return false;
    int dev = 0, sms = 0, blocks = 0, mps = 0;
    if (cluster)
    {
        cudaLaunchConfig_t lc = {};
        lc.gridDim = dim3(grid);
        lc.blockDim = dim3(threads);
        lc.dynamicSmemBytes = smem;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = grid;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        lc.attrs = at;
        lc.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&blocks, kernel, &lc) == cudaSuccess) return blocks > 0;
    }
    else if (cudaGetDevice(&dev) == cudaSuccess &&
             cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
             cudaDeviceGetAttribute(&mps, cudaDevAttrMpsEnabled, dev) == cudaSuccess &&
             cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kernel, threads, smem) == cudaSuccess)
        // under MPS the grids of other processes, whose order this one does not
        // know (CooperativeOrder), run on the same SMs
        return !mps && grid <= (int64_t)blocks * sms;
    cudaGetLastError();
    return false;
}

// The launch of many FP64 iterations for a system of n rows and `slots`
// stored entries, or none (kernel NULL): ILU(0), more rows than kManyRows..
// allows, or a stream whose SMs do not hold its blocks.  Vectors that do not fit
// the shared memories stay in global memory.  One cluster of 16 SMs while its FP64 work is short
// against the waits of a grid (us per iteration, cluster / grid / graph: CG 4.1k
// hex rows 7.7 / 9.6 / 18.9, 10.2k quad rows 8.1 / 8.8 / 16.3, 19.9k 11.5 / 9.1, 9.3k hex
// rows 12.4 / 9.7; BiCGStab 4.1k hex rows 14.8 / 18.0 / 38.6, 10.2k quad rows
// 16.2 / 16.2 / 31.7, 19.9k 22.5 / 16.5); it leaves 136 SMs to other threads' solves.
// shared: beside other solves only clusters (16.7k hex rows 18.8 / - / 19.9,
// on a tenth of the SMs).
ManyPlan many_plan(int n, int64_t slots, int kind, int precond, bool shared, bool scattered, cudaStream_t s)
{
    ManyPlan p;
    if (precond != OGS_PRECOND_NONE && precond != OGS_PRECOND_JACOBI) return p;
    int dev = 0, sms = 152, coop = 0, maxsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    cudaDeviceGetAttribute(&maxsm, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const size_t cap = std::min(kManyMaxSmem, maxsm - 20 * 1024);
    const bool stream = slots * 12 > (int64_t)96 << 20;
    const size_t hold = scattered ? std::min(cap, (size_t)kManyScatteredSmem) : cap;
    auto shape = [&](int blocks) {
        p.per = ((n + blocks - 1) / blocks + 31) & ~31;  // whole SELL slices
        p.grid = (n + p.per - 1) / p.per;
        const int vecs = (kind == SK_CG ? kCgVecs : kBiVecs) - (precond == OGS_PRECOND_JACOBI ? 0 : 1);
        const int fit = std::min<int64_t>(vecs, (int64_t)(hold / (sizeof(double) * p.per)));
        p.lay = (1 << fit) - 1;
        p.smem = sizeof(double) * p.per * fit;
    };
    const bool jac = precond == OGS_PRECOND_JACOBI;
    const int64_t work = slots + 6 * (int64_t)n;  // FP64 operations of an iteration
    const bool nines = (slots + n / 2) / n % 9 == 0;  // entries of most rows
    const int rows_per_sm = kind == SK_CG ? (nines ? kManyRowsCg : kManyOddRowsCg) : nines ? kManyRowsBi : kManyOddRowsBi;
    if (work <= (shared ? kManySharedWork : kManyClusterWork))
    {
        shape(16);
        p.cluster = true;
        p.grid = 16;  // blocks without rows still meet the barriers
        p.threads = 256;
        p.kernel = jac ? many_kernel<1, 256, true>(kind, false) : many_kernel<0, 256, true>(kind, false);
        cudaFuncSetAttribute(p.kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
    else if (!shared && coop && n <= (int64_t)sms * rows_per_sm)
    {
        int blocks = std::min(sms, n / 64);
        for (int k = 3; k >= 2; k--)
            if (blocks > sms / k && work <= kManyPartWork[k] && n <= sms / k * 256)
            {
                blocks = sms / k;
                break;
            }
        shape(std::max(1, blocks));
        p.threads = p.per > 512 ? kManyWide : 256;
        if (p.threads == 256)
            p.kernel = jac ? many_kernel<1, 256, false>(kind, stream) : many_kernel<0, 256, false>(kind, stream);
        else
            p.kernel = jac ? many_kernel<1, kManyWide, false>(kind, stream) : many_kernel<0, kManyWide, false>(kind, stream);
    }
    // the attribute is the function's, for every thread's launches: always
    // the same value
    if (p.kernel && cudaFuncSetAttribute(p.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap) != cudaSuccess)
    {
        cudaGetLastError();
        p.kernel = nullptr;
    }
    if (p.kernel && !resident_together(p.kernel, p.grid, p.threads, p.smem, p.cluster, s)) p.kernel = nullptr;
    return p;
}

cudaError_t launch_many(const SolveArgs& a, const ManyPlan& p, int iters, cudaStream_t s)
{
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(p.grid);
    lc.blockDim = dim3(p.threads);
    lc.dynamicSmemBytes = p.smem;
    lc.stream = s;
    cudaLaunchAttribute at[1];
    if (p.cluster)
    {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = p.grid;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    }
    else
    {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    }
    lc.attrs = at;
    lc.numAttrs = 1;
    int per = p.per, lay = p.lay;
    void* args[] = {const_cast<SolveArgs*>(&a), &per, &lay, &iters};
    auto go = [&]() { return cudaLaunchKernelExC(&lc, p.kernel, args); };
    return p.cluster ? go() : launch_cooperative_in_order(s, p.grid, go);
}

}  // namespace ogs

unsigned long long ogs_oob_many() { return ogs::oob_take(); }
