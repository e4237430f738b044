// batch_box.cuh -- Monte-Carlo batch: one realisation at a time on a group of
// blocks, its FP32 CG held on the SMs (included by batch.cu).
//
// The tile form of the batch (k_batch) walks one step of every realisation
// at a time, so each step streams the operator and the vectors of the whole
// batch from HBM (116 B a row) and waits for the whole grid.  Here a
// realisation runs to its end on as many blocks as hold it: the box is cut
// into bricks of whole x lines, a brick's vectors and cell coefficients live
// in its block's shared memory (about 32 B a node with the halo), and the FP32
// product is formed from one coefficient a cell instead of 14 stored values
// a row.  Per iteration only the bricks' faces go through L2 and the group
// waits twice; 304 blocks (two per SM, one waiting while the other works)
// run several realisations side by side.
//
// The iteration is CG preconditioned with the FP32 Jacobi inverse d, written
// on u = d r (a block needs no r): w = A u, gamma = sum u^2 / d, delta =
// sum w u, s = d w + beta s, p = u + beta p, x += alpha p, u -= alpha s.
//
// The product.  On a box of spacing h the Laplace matrix of a cell with
// coefficient k is k times K (x) M (x) M + M (x) K (x) M + M (x) M (x) K,
// K = [[1, -1], [-1, 1]] / h, M = [[2, 1], [1, 2]] h / 6.  For a node and
// the neighbour on one side, K gives c - n and M gives 2 c + n; so per plane
// z and side (sx, sy) three sums serve all cells that touch the plane:
//   KM = 2 k0 + k1, MK = m0 - m1, MM = 2 m0 + m1   (0: own line, 1: line sy)
// and a cell contributes k cz (Q(own plane) + R(its other plane)) with
// P = cx / cz KM + cy / cz MK, Q = 2 P + MM, R = P - MM.  Both sides sx go
// through one packed FP32 instruction (the kernel is bound by instruction
// issue), marching up z with the last plane's sums in registers.  Constant
// vectors map to zero exactly.
//
// The FP64 residual replacements use the stored upper half of the operator
// (U64), as the tile form does.
//
// Measured (solve at 1e-11; tile form tuned / here): one box of 24^3 4.1 / 0.9
// ms, 64^3 11.1 / 3.7, 96^3 31 / 7.8; 64 of 24^3 20.7 / 2.4; 24 boxes of 28^3
// to 95^3 202 / 73.  On full blocks an iteration takes 13 us: of 27,000
// cycles with two blocks on the SM the product has 6,000 to 9,000, the sums
// (mostly waiting for the slowest brick) 6,000 to 10,000, the updates 4,600,
// the halo 4,000.
#pragma once

namespace ogs {

constexpr int kBoxThreads = 256;
constexpr int kBoxSmem = 111 * 1024;  // two blocks per SM

struct BoxReal
{
    int by, bz, qy, need;  // lines per brick (y, z), bricks along y, bricks
    int member0;           // first entry of its block list / partial sums
};

// scheduling of realisations on blocks
struct BoxCtl
{
    int lock, n_free, taken;  // blocks waiting for work; realisations of several blocks given out
    int first;                // realisations before it (in `order`) are all given out
    int single;               // next realisation of one block (in `order`, beyond n_multi)
    int beat;                 // grows as long as some realisation iterates
};

struct BoxArgs
{
    const BReal* real;
    const BoxReal* box;
    const int* order;     // realisations by falling size
    int n_real, n_multi;  // the first n_multi of `order` take several blocks
    const double* ek;
    double *U64, *b, *x64, *r64;
    float* u32;           // u of the bricks' faces
    double* part;         // [bricks][2][4]
    unsigned* count;      // [n_real] barrier counters
    int* given;           // [n_real]
    int* mail;            // [n_blocks] 0 waiting, -1 leave, else 1 + realisation << 10 | rank
    int* free_list;       // [n_blocks]
    int* members;         // [bricks] block of each rank
    BoxCtl* sched;
    BCtl* ctl;
    int* real_done;
    ogs_batch_stats* out;
    double tol, delta;
    int max_iter;
    const double* kloc;
    double cz;            // hx hy / (36 hz) times time_unit_factor: in the cell coefficients
    float fx, fy;         // cx / cz, cy / cz
};

constexpr unsigned kBarSpins = 1u << 22;
constexpr int kBeatIters = 64;  // iterations from one beat to the next

struct BoxGroup
{
    unsigned* count;
    unsigned target;  // arrivals that complete the last barrier
    int nb, rank;
    double* part;  // this realisation's partial sums
    unsigned seq;
    const unsigned* limit;  // polls of one wait, in shared memory (see grid_wait)
};

__device__ __forceinline__ void box_arrive(BoxGroup& G)
{
    G.target += G.nb;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(G.count) : "memory");
}

__device__ __forceinline__ bool box_wait(const BoxArgs& a, const BoxGroup& G)
{
    unsigned spins = 0;
    while ((int)(ld_acquire(G.count) - G.target) < 0)
        if (++spins > kBarSpins || ((spins & 255u) == 0 && ld_volatile(&a.ctl->err)) ||
            ((spins == 4u || (spins & 255u) == 0) && spins >= *(const volatile unsigned*)G.limit))
        {
            atomicExch(&a.ctl->err, 1);
            return false;
        }
    return true;
}

// Group sums of NV values per thread, in every thread of every block: added
// in T within a warp, in FP64 from the warps on, in rank order.  The wait is
// also the group's barrier.  false: a wait gave up.
template <int NV, typename T>
__device__ __forceinline__ bool box_sum(const BoxArgs& a, BoxGroup& G, const T (&v)[NV], double (&out)[NV],
                                        double (*s_warp)[8], double* s_tot, int* s_fail)
{
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    T w[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) w[k] = v[k];
    warp_allsum<NV, T>(w);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; k++) s_warp[k][wid] = (double)w[k];
    __syncthreads();
    double* part = G.part + (G.seq & 1) * (size_t)G.nb * 4;
    G.seq++;
    const unsigned target = G.target + G.nb;
    if (wid == 0)
    {
        // eight lanes a value, two buffers of partial sums in turn
        const int k = lane >> 3;
        double q = k < NV ? s_warp[k < NV ? k : 0][lane & 7] : 0.0;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
        if (k < NV && (lane & 7) == 0) __stcg(part + (size_t)k * G.nb + G.rank, q);
        __syncwarp();
        if (lane == 0) box_arrive(G);
    }
    G.target = target;
    if (wid == 0)
    {
        // one thread polls: a poll per value and block cost 6% of the iteration
        if (lane == 0 && !box_wait(a, G)) *s_fail = 1;
        __syncwarp();
        constexpr int K = 5;
        double q[NV];
#pragma unroll
        for (int k = 0; k < NV; k++) q[k] = 0.0;
        for (int b0 = 0; b0 < G.nb; b0 += 32 * K)
        {
            double w[NV][K];
#pragma unroll
            for (int j = 0; j < K; j++)
            {
                const int b = b0 + 32 * j + lane;
#pragma unroll
                for (int k = 0; k < NV; k++) w[k][j] = b < G.nb ? __ldcg(part + (size_t)k * G.nb + b) : 0.0;
            }
#pragma unroll
            for (int j = 0; j < K; j++)
#pragma unroll
                for (int k = 0; k < NV; k++) q[k] += w[k][j];
        }
        warp_allsum<NV, double>(q);
        if (lane == 0)
#pragma unroll
            for (int k = 0; k < NV; k++) s_tot[k] = q[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; k++) out[k] = s_tot[k];
    return *s_fail == 0;
}

__device__ __forceinline__ bool box_barrier(const BoxArgs& a, BoxGroup& G, int* s_fail)
{
    __syncthreads();
    if (threadIdx.x == 0)
    {
        box_arrive(G);
        if (!box_wait(a, G)) *s_fail = 1;
    }
    else
        G.target += G.nb;
    __syncthreads();
    return *s_fail == 0;
}

// packed FP32 pairs
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float a, float b)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float sum2(f32x2 v)
{
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return a + b;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// One plane's sums at a node, both sides sx a pair, by side sy: lines y - 1,
// y, y + 1 around x (p: the value at x - 1 of line y - 1).  c: u at the node
__device__ __forceinline__ void box_plane(const float* p, int lx, f32x2 fx, f32x2 fy, f32x2 (&Q)[2], f32x2 (&R)[2],
                                          float& c)
{
    const f32x2 two = pack2(2.f, 2.f), neg = pack2(-1.f, -1.f);
    f32x2 k[3], m[3];
#pragma unroll
    for (int l = 0; l < 3; l++)
    {
        const f32x2 ab = pack2(p[l * lx], p[l * lx + 2]);
        const float v = p[l * lx + 1];
        const f32x2 cc = pack2(v, v);
        if (l == 1) c = v;
        k[l] = fma2(ab, neg, cc);
        m[l] = fma2(cc, two, ab);
    }
#pragma unroll
    for (int sy = 0; sy < 2; sy++)
    {
        const int o = 2 * sy;
        const f32x2 KM = fma2(k[1], two, k[o]), MK = fma2(m[o], neg, m[1]), MM = fma2(m[1], two, m[o]);
        const f32x2 P = fma2(KM, fx, mul2(MK, fy));
        Q[sy] = fma2(P, two, MM);
        R[sy] = fma2(MM, neg, P);
    }
}

// u of the neighbouring bricks' faces into the halo (lines outside the box
// stay zero)
__device__ __forceinline__ void box_halo(const float* u32, float* su, const BReal& R, int y0, int z0, int by, int bz,
                                         int LX, int LY)
{
    constexpr int NT = kBoxThreads, K = 8;
    const int nx = R.nx, total = (2 * LY + 2 * bz) * nx;
    const unsigned magic = 0xffffffffu / (unsigned)nx + 1u;  // e / nx: exact while e nx < 2^32
    for (int e0 = threadIdx.x; e0 < total; e0 += K * NT)
    {
        float v[K];
        int at[K];
#pragma unroll
        for (int k = 0; k < K; k++)
        {
            const int e = e0 + k * NT;
            at[k] = -1;
            if (e < total)
            {
                const int h = __umulhi((unsigned)e, magic), x = e - h * nx;
                int yy, zz;
                if (h < LY) { zz = 0; yy = h; }
                else if (h < 2 * LY) { zz = bz + 1; yy = h - LY; }
                else { zz = 1 + (h - 2 * LY) / 2; yy = (h - 2 * LY) & 1 ? by + 1 : 0; }
                const int gy = y0 + yy - 1, gz = z0 + zz - 1;
                if (gy >= 0 && gy < R.ny && gz >= 0 && gz < R.nz)
                {
                    at[k] = (zz * LY + yy) * LX + x + 1;
                    v[k] = __ldcg(u32 + x + nx * (gy + R.ny * gz));
                }
            }
        }
#pragma unroll
        for (int k = 0; k < K; k++)
            if (at[k] >= 0) su[at[k]] = v[k];
    }
}

// FP64 row of the upper half of the operator applied to x64, which changes
// during the launch (as row64, without the FP32 correction)
__device__ __forceinline__ double row64_x(const double* U, int nx, int nxy, int n, int i, const double* x64)
{
    double acc = U[i] * x64[i];
#pragma unroll
    for (int d = 1; d < 14; d++)
    {
        const int o = up_offset(d, nx, nxy);
        const double* Ud = U + (size_t)d * n;
        if (i + o < n) acc += Ud[i] * x64[i + o];
        if (i - o >= 0) acc += Ud[i - o] * x64[i - o];
    }
    return acc;
}

// The realisation of the block's mail on its group; rank 0 writes the
// statistics.  false: a wait gave up.
__device__ bool box_realisation(const BoxArgs& a, int ri, int rank, float* sm)
{
    constexpr int NT = kBoxThreads;
    __shared__ double s_warp[4][8], s_tot[4];
    __shared__ float s_ab[2];
    __shared__ int s_fail, s_stop;
    __shared__ unsigned s_limit;
    const BReal R = a.real[ri];
    const BoxReal B = a.box[ri];
    const int tid = threadIdx.x;
    const int nx = R.nx, nxy = R.nx * R.ny;
    const int y0 = rank % B.qy * B.by, z0 = rank / B.qy * B.bz;
    const int by = min(B.by, R.ny - y0), bz = min(B.bz, R.nz - z0);
    const int ncol = nx * by, nodes = ncol * bz;
    const int LX = nx + 2, LY = by + 2, KX = nx + 1, KY = by + 1;
    // shared memory: u with its halo, cell coefficients, d w, p, s, x, d
    float* su = sm;
    float* sk = su + LX * LY * (bz + 2);
    float* sw = sk + KX * KY * (bz + 1);
    float *sp = sw + nodes, *ss = sp + nodes, *sx = ss + nodes, *sd = sx + nodes;
    const double* ek = a.ek + R.elem0;
    double* U = a.U64 + 14 * R.row0;
    double *b = a.b + R.row0, *x64 = a.x64 + R.row0, *r64 = a.r64 + R.row0;
    float* u32 = a.u32 + R.row0;
    BoxGroup G{a.count + ri, 0u, B.need, rank, a.part + (size_t)B.member0 * 8, 0u, &s_limit};
    if (tid == 0)
    {
        s_fail = 0;
        s_limit = a.ctl->spin_limit ? a.ctl->spin_limit : kBarSpins;
    }
    for (int i = tid; i < LX * LY * (bz + 2); i += NT) su[i] = 0.f;
    for (int i = tid; i < KX * KY * (bz + 1); i += NT)
    {
        // the cell below node (x, y, z) of the brick, 0 outside the box
        const int l = i / KX, cx = i - l * KX - 1, lz = l / KY, cy = y0 + l - lz * KY - 1, cz = z0 + lz - 1;
        const bool in = cx >= 0 && cx < nx - 1 && cy >= 0 && cy < R.ny - 1 && cz >= 0 && cz < R.nz - 1;
        sk[i] = in ? (float)(a.cz * __ldg(ek + cx + (int64_t)(nx - 1) * (cy + (int64_t)(R.ny - 1) * cz))) : 0.f;
    }
    for (int q = tid; q < nodes; q += NT)
    {
        const int l = q / nx, x = q - l * nx, lz = l / by, y = y0 + l - lz * by, z = z0 + lz;
        const int i = x + nx * y + nxy * z;
        double diag;
        assemble_row(a.kloc, R, ek, i, x, y, z, U, (float*)nullptr, b, x64, diag);
        // the Jacobi inverse; 0 drops the Dirichlet rows and columns
        sd[q] = x == 0 || x == nx - 1 ? 0.f : (float)(fabs(diag) < DBL_MIN ? 1.0 : 1.0 / diag);
        sp[q] = 0.f;
        ss[q] = 0.f;
        sx[q] = 0.f;
    }
    // solver scalars, alike in every block (thread 0 of the FP32 iterations)
    double bnorm = 1.0, scale = 1.0, gam = 0.0, eta = 0.0, gam1 = 0.0, eta1 = 0.0, error = 0.0;
    int iter = 0, status = OGS_NOT_CONVERGED, refinements = 0;
    const f32x2 fx = pack2(a.fx, a.fx), fy = pack2(a.fy, a.fy);
    bool first = true;
    for (;;)
    {
        // FP64 residual replacement: x64 += x / scale ; r64 = b - A x64
        if (!first)
        {
            const double inv = 1.0 / scale;
            for (int q = tid; q < nodes; q += NT)
            {
                const int l = q / nx, x = q - l * nx, lz = l / by;
                const int i = x + nx * (y0 + l - lz * by) + nxy * (z0 + lz);
                x64[i] += (double)sx[q] * inv;
                sx[q] = 0.f;
            }
        }
        if (!box_barrier(a, G, &s_fail)) return false;
        double v[3] = {0.0, 0.0, 0.0}, g[3];
        for (int q = tid; q < nodes; q += NT)
        {
            const int l = q / nx, x = q - l * nx, lz = l / by;
            const int i = x + nx * (y0 + l - lz * by) + nxy * (z0 + lz);
            const double bi = b[i], r = bi - row64_x(U, nx, nxy, R.n, i, x64);
            r64[i] = r;
            v[0] += r * r;
            v[1] += r * r * (double)sd[q];
            if (first) v[2] += bi * bi;
        }
        if (!box_sum<3, double>(a, G, v, g, s_warp, s_tot, &s_fail)) return false;
        bool done = false;
        if (first)
        {
            // Linear_EQS::CheckNormRHS of a fresh system (bNorm = 1.0)
            bnorm = sqrt(g[2]);
            if (!isfinite(bnorm)) { status = OGS_NONFINITE; error = bnorm; done = true; }
            else if (bnorm / 1.0 < a.tol) { status = OGS_OK; error = bnorm; done = true; }
            else if (bnorm < DBL_MIN) { status = OGS_OK; error = 0.0; done = true; }
        }
        if (!done)
        {
            error = sqrt(g[0]) / bnorm;
            refinements++;
            if (!isfinite(error)) { status = OGS_NONFINITE; done = true; }
            else if (error < a.tol) { status = OGS_OK; done = true; }
            else if (iter >= a.max_iter) { status = OGS_NOT_CONVERGED; done = true; }
        }
        if (done) break;
        // (a negative definite operator has negative d and products; the same
        // iteration on it needs their size only)
        const double rc = sqrt(fabs(g[1]));
        const double ns = rc > DBL_MIN ? 1.0 / rc : 1.0;
        const double ratio = first ? 1.0 : ns / scale;
        scale = ns;
        for (int c = tid; c < ncol; c += NT)
        {
            const int y = c / nx, x = c - y * nx;
            for (int z = 0; z < bz; z++)
            {
                const int q = z * ncol + c, i = x + nx * (y0 + y) + nxy * (z0 + z);
                const float u = (float)(r64[i] * ns) * sd[q];
                sp[q] *= (float)ratio;
                ss[q] *= (float)ratio;
                su[((z + 1) * LY + y + 1) * LX + x + 1] = u;
                if (y == 0 || y == by - 1 || z == 0 || z == bz - 1) u32[i] = u;
            }
        }
        // the iteration that asked for the replacement is redone
        if (!first)
        {
            iter -= 1;
            const double r2 = ratio * ratio;
            gam = gam1 * r2;
            eta = eta1 * r2;
        }
        const int base = iter;
        double inv_gam = first ? 0.0 : 1.0 / gam, drop2 = 0.0;
        const double eu = a.tol / error, est2 = eu * eu, dl2 = a.delta * a.delta;
        first = false;
        if (!box_barrier(a, G, &s_fail)) return false;
        box_halo(u32, su, R, y0, z0, by, bz, LX, LY);
        __syncthreads();
        int nonfinite = 0;
        double rho = 0.0;
        for (;;)
        {
            // S: w = A u ; u . u / d, w . u
            float d2[2] = {0.f, 0.f};
            for (int c = tid; c < ncol; c += NT)
            {
                const int y = c / nx, x = c - y * nx;
                const float* pu = su + y * LX + x;
                const float* pk = sk + y * KX + x;
                const int zu = LX * LY, zk = KX * KY;
                f32x2 Rm[2], Q0[2], R0[2], Q1[2], R1[2], al[2], ah[2];
                float u0, u1;
                box_plane(pu, LX, fx, fy, Q1, Rm, u1);
                box_plane(pu + zu, LX, fx, fy, Q0, R0, u0);
                pu += 2 * zu;
#pragma unroll
                for (int sy = 0; sy < 2; sy++) al[sy] = pack2(pk[sy * KX], pk[sy * KX + 1]);
                int q = c;
#pragma unroll 3
                for (int z = 0; z < bz; z++, q += ncol)
                {
                    box_plane(pu, LX, fx, fy, Q1, R1, u1);
                    pu += zu;
                    pk += zk;
                    f32x2 acc = 0ull;
#pragma unroll
                    for (int sy = 0; sy < 2; sy++)
                    {
                        ah[sy] = pack2(pk[sy * KX], pk[sy * KX + 1]);
                        acc = fma2(al[sy], add2(Q0[sy], Rm[sy]), acc);
                        acc = fma2(ah[sy], add2(Q0[sy], R1[sy]), acc);
                        al[sy] = ah[sy];
                        Rm[sy] = R0[sy];
                        R0[sy] = R1[sy];
                        Q0[sy] = Q1[sy];
                    }
                    const float w = sum2(acc), d = sd[q];
                    sw[q] = w * d;
                    if (d != 0.f) d2[0] += __fdividef(u0 * u0, d);
                    d2[1] += w * u0;
                    u0 = u1;
                }
            }
            double g2[2];
            if (!box_sum<2, float>(a, G, d2, g2, s_warp, s_tot, &s_fail)) return false;
            if (tid == 0)
            {
                rho = g2[0];
                const int it = iter + 1;
                const bool one = it == 1, fresh = it == base + 1;
                const double beta = one ? 0.0 : rho * inv_gam;
                gam1 = gam;
                eta1 = eta;
                eta = one ? g2[1] : g2[1] - beta * beta * eta;
                const float alpha = quotient_f32(rho, eta);
                s_ab[0] = alpha;
                s_ab[1] = (float)beta;
                const double size = fabs(rho);
                if (fresh) drop2 = dl2 * size;
                const bool due = less_bits(size, est2) || less_bits(size, drop2) || it > a.max_iter;
                nonfinite = !finite_bits(rho) || !finite_bits(eta) || !isfinite(alpha);
                gam = rho;
                s_stop = nonfinite ? 2 : !fresh && due ? 1 : 0;
            }
            iter += 1;
            if (rank == 0 && tid == 0 && iter % kBeatIters == 0) atomicAdd(&a.sched->beat, 1);
            __syncthreads();
            if (s_stop) break;
            // V: p = u + beta p ; s = d w + beta s ; u -= alpha s, its faces published
            const float fa = s_ab[0], fb = s_ab[1];
            for (int c = tid; c < ncol; c += NT)
            {
                const int y = c / nx, x = c - y * nx;
                const bool edge = y == 0 || y == by - 1;
                float* pu = su + (LY + y + 1) * LX + x + 1;
                float* gu = u32 + x + nx * (y0 + y) + (int64_t)nxy * z0;
                int q = c;
#pragma unroll 4
                for (int z = 0; z < bz; z++, q += ncol, pu += LX * LY, gu += nxy)
                {
                    const float u0 = *pu, s = sw[q] + fb * ss[q], u = u0 - fa * s;
                    ss[q] = s;
                    sp[q] = u0 + fb * sp[q];
                    *pu = u;
                    if (edge || z == 0 || z == bz - 1) *gu = u;
                }
            }
            __syncthreads();
            if (tid == 0) box_arrive(G);
            else G.target += G.nb;
            // x += alpha p, while the group arrives
#pragma unroll 4
            for (int q = tid; q < nodes; q += NT) sx[q] += fa * sp[q];
            if (tid == 0)
            {
                inv_gam = 1.0 / gam;
                if (!box_wait(a, G)) s_fail = 1;
            }
            __syncthreads();
            if (s_fail) return false;
            box_halo(u32, su, R, y0, z0, by, bz, LX, LY);
            __syncthreads();
        }
        if (s_stop == 2)
        {
            status = OGS_NONFINITE;
            if (tid == 0) error = sqrt(fabs(rho));
            // x64 as of the last replacement, as the tile form leaves it
            break;
        }
        __syncthreads();  // s_stop is read before the next cycle writes it
    }
    if (rank == 0 && tid == 0)
    {
        ogs_batch_stats o;
        o.iterations = iter;
        o.status = status;
        o.refinements = refinements;
        o.pad0 = 0;
        o.rel_residual = error;
        o.finish_ms = (double)(global_ns() - *(volatile unsigned long long*)&a.ctl->t0) * 1e-6;
        a.out[ri] = o;
        a.real_done[ri] = 1;
    }
    return true;
}

// The next realisation of one block as mail, for a block that has just done
// one, while none of several blocks is open (those are given out under the
// lock, largest first): -1 when there is none left, 0 when the lock decides.
// Without this the lock was taken for each of 10,000 boxes of 4^3: 47 ms, 35 with
// the tile form, 9 so.
__device__ __forceinline__ int box_next_single(const BoxArgs& a)
{
    BoxCtl* c = a.sched;
    if (ld_volatile(&c->taken) < a.n_multi) return 0;
    const int o = ld_volatile(&c->single) < a.n_real ? atomicAdd(&c->single, 1) : a.n_real;
    if (o >= a.n_real) return -1;
    const int r = a.order[o];
    a.members[a.box[r].member0] = blockIdx.x;
    return 1 + (r << 10);
}

// Gives waiting blocks to the realisations not yet given out, largest first,
// smaller ones where the next does not fit; blocks that no realisation is
// left for are sent home.  One warp, lock held.
__device__ void box_dispatch(const BoxArgs& a)
{
    BoxCtl* c = a.sched;
    const int lane = threadIdx.x & 31;
    int n_free = ld_volatile(&c->n_free), taken = ld_volatile(&c->taken), first = ld_volatile(&c->first);
    for (int o0 = first; o0 < a.n_multi && n_free > 0; o0 += 32)
    {
        const int o = o0 + lane;
        const int r = o < a.n_multi ? a.order[o] : -1;
        const bool open = r >= 0 && !ld_volatile(a.given + r);
        const int need = open ? a.box[r].need : 0x7fffffff;
        for (;;)
        {
            const unsigned fits = __ballot_sync(0xffffffffu, need <= n_free && open && !ld_volatile(a.given + (r < 0 ? 0 : r)));
            if (!fits) break;
            const int src = __ffs(fits) - 1;
            const int rr = __shfl_sync(0xffffffffu, r, src), nn = __shfl_sync(0xffffffffu, need, src);
            for (int k = lane; k < nn; k += 32)
            {
                const int blk = *(volatile int*)(a.free_list + n_free - 1 - k);
                a.members[a.box[rr].member0 + k] = blk;
                st_release((unsigned*)(a.mail + blk), (unsigned)(1 + (rr << 10 | k)));
            }
            if (lane == 0) *(volatile int*)(a.given + rr) = 1;
            n_free -= nn;
            taken += 1;
            __syncwarp();
        }
    }
    // one block each for the others
    int single = ld_volatile(&c->single);
    if (n_free > 0 && single < a.n_real)
    {
        if (lane == 0) single = atomicAdd(&c->single, n_free);
        single = __shfl_sync(0xffffffffu, single, 0);
        const int n = min(n_free, max(0, a.n_real - single));
        for (int k = lane; k < n; k += 32)
        {
            const int r = a.order[single + k], blk = *(volatile int*)(a.free_list + n_free - 1 - k);
            a.members[a.box[r].member0] = blk;
            st_release((unsigned*)(a.mail + blk), (unsigned)(1 + (r << 10)));
        }
        single += n;
        n_free -= n;
        __syncwarp();
    }
    if (taken == a.n_multi && single >= a.n_real)
    {
        for (int k = lane; k < n_free; k += 32) st_release((unsigned*)(a.mail + *(volatile int*)(a.free_list + k)), (unsigned)-1);
        n_free = 0;
    }
    // realisations given out at the front need no second look
    while (first < a.n_multi && ld_volatile(a.given + a.order[first])) first++;
    if (lane == 0)
    {
        *(volatile int*)&c->n_free = n_free;
        *(volatile int*)&c->taken = taken;
        *(volatile int*)&c->first = first;
        atomicAdd(&c->beat, 1);
    }
}

__global__ void __launch_bounds__(kBoxThreads, 2) k_batch_box(BoxArgs a)
{
    extern __shared__ float box_smem[];
    __shared__ int s_mail;
    if (blockIdx.x == 0 && threadIdx.x == 0) a.ctl->t0 = global_ns();
    int have = 0;  // the next realisation is known already
    for (;;)
    {
        if (!have && threadIdx.x == 0)
        {
            // a block without work waits as long as the others make progress:
            // the limit is of polls without a beat (each group's own waits
            // are bounded, so beats end when something is wrong)
            const unsigned limit = a.ctl->spin_limit ? a.ctl->spin_limit : kSpinLimit;
            unsigned spins = 0;
            int m, beat = ld_volatile(&a.sched->beat);
            while ((m = (int)ld_acquire((const unsigned*)(a.mail + blockIdx.x))) == 0)
            {
                bool stop = ld_volatile(&a.ctl->err) != 0;
                if (++spins > limit)
                {
                    const int now = ld_volatile(&a.sched->beat);
                    stop = stop || now == beat;
                    beat = now;
                    spins = 0;
                }
                if (stop)
                {
                    atomicExch(&a.ctl->err, 1);
                    m = -1;
                    break;
                }
                __nanosleep(200);
            }
            if (m > 0) a.mail[blockIdx.x] = 0;
            s_mail = m;
        }
        __syncthreads();
        const int m = s_mail;
        if (m < 0) return;
        const int ri = (m - 1) >> 10, rank = (m - 1) & 1023;
        if (!box_realisation(a, ri, rank, box_smem)) return;
        __syncthreads();
        have = 0;
        if (a.box[ri].need == 1)
        {
            if (threadIdx.x == 0) s_mail = box_next_single(a);
            __syncthreads();
            have = s_mail;
            if (have < 0) return;
            if (have > 0) continue;
        }
        // the group's first block hands all of its blocks back
        if (rank == 0 && threadIdx.x < 32)
        {
            const BoxReal B = a.box[ri];
            unsigned spins = 0;
            bool got = false;
            while (!got && spins < kSpinLimit)
            {
                if (threadIdx.x == 0) got = atomicCAS(&a.sched->lock, 0, 1) == 0;
                got = __shfl_sync(0xffffffffu, got, 0);
                if (!got) __nanosleep(100);
                spins++;
            }
            if (!got)
                atomicExch(&a.ctl->err, 1);
            else
            {
                __threadfence();
                const int nf = ld_volatile(&a.sched->n_free);
                for (int k = threadIdx.x; k < B.need; k += 32)
                    *(volatile int*)(a.free_list + nf + k) = *(volatile int*)(a.members + B.member0 + k);
                __syncwarp();
                if (threadIdx.x == 0) *(volatile int*)&a.sched->n_free = nf + B.need;
                __syncwarp();
                __threadfence();
                box_dispatch(a);
                __threadfence();
                __syncwarp();
                if (threadIdx.x == 0) atomicExch(&a.sched->lock, 0);
            }
        }
        __syncthreads();
    }
}

}  // namespace ogs
