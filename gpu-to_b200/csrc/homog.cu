// Periodic homogenization of a voxel unit cell: the six unit-strain load
// cases solved together as six right-hand sides, and the effective 6x6
// elasticity tensor.  No counterpart in the reference (its Homogenization
// directory solves a self-weight problem, Homogenization/QNC/QNC_V1_mod1m.m:
// 180-199); the method is the reference's MGCG (mgcg1.cu:184-651) carried to
// a periodic grid:
//
//  * grid: n_x x n_y x n_z elements = nodes, node / element (i, j, k) at
//    (n_z n_y) i + n_y k + j (y fastest, the reference's order); element
//    (i, j, k) has the corners (i + x_a, j + y_a, k + z_a) mod n in the
//    reference's local order.  Node 0 is held (its three dofs) to remove the
//    rigid translations, the periodic operator's only null space;
//  * vectors: nine planes of load-case pairs, plane 3 d + p holding component
//    d of cases 2p and 2p + 1 as one float2 / double2 per node, so that a warp
//    along y reads and writes whole 128-byte lines in every kernel (with the
//    six cases of a dof adjacent, a warp's loads were 72 or 144 bytes apart
//    and the sweeps were bound by L1 wavefronts);
//  * load case r (Voigt xx, yy, zz, yz, xz, xy; engineering shears): the
//    fluctuation chi_r solves K chi_r = -sum_e CX_e Ke u0_r, u0_r the affine
//    field of unit strain r at an element's local corners;
//  * operator: a node-centred gather over the 27 neighbours; the 3x3 block
//    of each neighbour, sum over the shared elements of CX_e Ke(a, b), is
//    formed once per node and applied to all six load cases;
//  * preconditioner: an FP32 V-cycle (damped Jacobi, the reference's
//    nswp / omega / pre-relaxation; trilinear periodic transfers) on
//    re-discretised coarse levels (CX_l = 2 mean of the eight children, as
//    the reference's mgcg9 builds them, Homogenization/QNC/mgcg9.cu:753-781),
//    and a dense Cholesky solve on the coarsest grid;
//  * outer iteration: flexible PCG (Polak-Ribiere beta) in FP64, one
//    recurrence per load case, a load case frozen (alpha = 0) once it meets
//    the tolerance; one CUDA graph launch per iteration of all six;
//  * C_rs = (1 / n_el) sum_e CX_e (u0_r + chi_r)_e' Ke (u0_s + chi_s)_e.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "gputo_internal.h"

namespace gputo {

namespace {

constexpr int NR = 6;                  // load cases
constexpr int kHBlocks = 1184;         // CTAs of the reduction kernels (8 per SM)

__constant__ double cPKe64[576];
__constant__ float cPKe32[576];
__constant__ double cPG[24 * NR];      // Ke u0_r, [24][6]
__constant__ double cPU0[NR * 24];     // u0_r at the local corners, [6][24]

struct PGrid {
    int nx, ny, nz;
    __host__ __device__ long long nnod() const { return (long long)nx * ny * nz; }
    __host__ __device__ long long ndof() const { return 3 * nnod(); }
    __host__ __device__ long long node(int i, int j, int k) const
    {
        return ((long long)nz * ny) * i + (long long)ny * k + j;
    }
};

__host__ __device__ constexpr int corner_of(int x, int y, int z) { return 4 * z + (y ? (x ? 2 : 3) : (x ? 1 : 0)); }

__device__ __forceinline__ int wrap(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

template <typename T> __device__ __forceinline__ T pke(int idx);
template <> __device__ __forceinline__ double pke<double>(int idx) { return cPKe64[idx]; }
template <> __device__ __forceinline__ float pke<float>(int idx) { return cPKe32[idx]; }

enum PMode { P_APPLY = 0, P_DEFECT = 1, P_JACOBI = 2, P_PRE = 3 };

template <typename T> struct Pair;
template <> struct Pair<float> {
    using V = float2;
};
template <> struct Pair<double> {
    using V = double2;
};
__device__ __forceinline__ float2 pfma(float b, float2 v, float2 a) { return __ffma2_rn(make_float2(b, b), v, a); }
__device__ __forceinline__ double2 pfma(double b, double2 v, double2 a)
{
    return make_double2(fma(b, v.x, a.x), fma(b, v.y, a.y));
}
__device__ __forceinline__ float2 pscale(float b, float2 v) { return make_float2(b * v.x, b * v.y); }
__device__ __forceinline__ double2 pscale(double b, double2 v) { return make_double2(b * v.x, b * v.y); }

// One operator sweep over all six load cases, thread per NX nodes along x.
// Modes as the fine sweeps: K u (with the per-case p'q partials), f - K u,
// damped Jacobi z = u + omega (f - K u) / diag, and the pre-relaxation that
// starts from u = prerelax f / diag.  Node 0's dofs are held at zero residual.
//
// Per node 576 FMAs form the 27 blocks and 1458 apply them to the six cases
// (as 729 paired FP32 instructions): 118 us of FMA pipe at 128^3 in FP32 and
// 237 us in FP64, above the 70 and 93 us of HBM traffic.  The 27 x 9
// neighbour pairs come through L1, coalesced along y; a CTA covers 32 (y) x 8
// (z) columns so that most of them hit (the apply takes 256 consecutive nodes,
// the order of its p'q sums).  In FP32 a thread takes two nodes on large
// grids, which share two of their three neighbour planes (18 instead of 27
// plane reads per node).  The neighbours' loads are kept three at a time:
// left to itself the compiler hoists them all and spills.
// Measured at 128^3: FP32 Jacobi sweep 232 us (FMA pipe 54 % active; 727 us
// with the cases of a dof adjacent, bound by L1 wavefronts), FP64 apply 402 us
// (1272 us); the same bits.  One node per thread at three CTAs per SM gave the
// same time as two nodes at two CTAs, two nodes at three CTAs spilled (6 %
// slower per solve), and keeping the node's own values in registers for the
// epilogue cost the FP64 apply its second CTA (4 % slower per solve).
template <typename T, int MODE, int NX>
__global__ void __launch_bounds__(256, 2)
psweep_kernel(PGrid g, int ty, int ntj, int nt, const T *__restrict__ CX, const T *__restrict__ u_, const T *__restrict__ f_,
              const T *__restrict__ rdiag, T *__restrict__ out_, T omega, T prerelax, double *__restrict__ partial,
              const int *__restrict__ done)
{
    if (done && *done) return;
    using V = typename Pair<T>::V;
    const V *__restrict__ u = reinterpret_cast<const V *>(u_);
    const V *__restrict__ f = reinterpret_cast<const V *>(f_);
    V *__restrict__ out = reinterpret_cast<V *>(out_);
    const int nn = (int)g.nnod();
    const size_t N = (size_t)nn;
    int i0, j, k;
    bool mine;
    if (MODE == P_APPLY) {   // 256 consecutive nodes: the p'q partials sum in node order
        const int n = (int)(blockIdx.x * 256 + threadIdx.x), t = n / g.ny;
        j = n - t * g.ny;
        i0 = t / g.nz;
        k = t - i0 * g.nz;
        mine = n < nn;
    } else {
        const int tz = 256 / ty;
        const int bi = (int)(blockIdx.x / (unsigned)nt), bt = (int)blockIdx.x - bi * nt;   // x step, (y, z) tile
        const int tk = bt / ntj, tj = bt - tk * ntj;
        const int lk = (int)threadIdx.x / ty;
        j = tj * ty + ((int)threadIdx.x - lk * ty);
        k = tk * tz + lk;
        i0 = bi * NX;
        mine = j < g.ny && lk < tz && k < g.nz;
    }
    V dsum[3];
#pragma unroll
    for (int p = 0; p < 3; ++p) dsum[p].x = dsum[p].y = T(0);
    if (mine) {
        const int ps = g.nz * g.ny;
        const int yj[3] = {wrap(j - 1, g.ny), j, wrap(j + 1, g.ny)};
        const int zk[3] = {wrap(k - 1, g.nz) * g.ny, k * g.ny, wrap(k + 1, g.nz) * g.ny};
        int xi[NX + 2];   // planes i0 - 1 .. i0 + NX
        xi[0] = wrap(i0 - 1, g.nx) * ps;
#pragma unroll
        for (int q = 1; q < NX + 2; ++q) {
            int v = i0 + q - 1;
            v = v >= g.nx ? v - g.nx : v;
            xi[q] = v * ps;
        }
        // the elements around the nodes: element (i0 - 1 + ex, j - 1 + ey, k - 1 + ez)
        T cxe[NX + 1][2][2];
#pragma unroll
        for (int ex = 0; ex < NX + 1; ++ex)
#pragma unroll
            for (int ey = 0; ey < 2; ++ey)
#pragma unroll
                for (int ez = 0; ez < 2; ++ez) cxe[ex][ey][ez] = CX[xi[ex] + zk[ez] + yj[ey]];
        V acc[NX][9];   // [3 d + p]
#pragma unroll
        for (int m = 0; m < NX; ++m)
#pragma unroll
            for (int q = 0; q < 9; ++q) acc[m][q].x = acc[m][q].y = T(0);
#pragma unroll
        for (int px = 0; px < NX + 2; ++px)
#pragma unroll
            for (int dy = -1; dy <= 1; ++dy) {
                asm volatile("" ::: "memory");   // keep the loads of three neighbours in flight, not of all
#pragma unroll
                for (int dz = -1; dz <= 1; ++dz) {
                    const int nb = xi[px] + zk[dz + 1] + yj[dy + 1];
                    V v[9];
#pragma unroll
                    for (int b = 0; b < 3; ++b) {
                        if (MODE == P_PRE) {
                            const T s = prerelax * rdiag[3 * (size_t)nb + b];
#pragma unroll
                            for (int p = 0; p < 3; ++p) v[3 * b + p] = pscale(s, f[(3 * b + p) * N + nb]);
                        } else {
#pragma unroll
                            for (int p = 0; p < 3; ++p) v[3 * b + p] = u[(3 * b + p) * N + nb];
                        }
                    }
#pragma unroll
                    for (int m = 0; m < NX; ++m) {
                        const int dx = px - 1 - m;   // offset from node i0 + m
                        if (dx < -1 || dx > 1) continue;
                        // 3x3 block between the node and neighbour (dx, dy, dz)
                        T B[3][3];
#pragma unroll
                        for (int a = 0; a < 3; ++a)
#pragma unroll
                            for (int b = 0; b < 3; ++b) B[a][b] = T(0);
#pragma unroll
                        for (int ex = 0; ex < 2; ++ex)
#pragma unroll
                            for (int ey = 0; ey < 2; ++ey)
#pragma unroll
                                for (int ez = 0; ez < 2; ++ez) {
                                    const int bx = dx + 1 - ex, by = dy + 1 - ey, bz = dz + 1 - ez;
                                    if (bx < 0 || bx > 1 || by < 0 || by > 1 || bz < 0 || bz > 1) continue;
                                    const int ca = corner_of(1 - ex, 1 - ey, 1 - ez), cb = corner_of(bx, by, bz);
                                    const T c = cxe[m + ex][ey][ez];
#pragma unroll
                                    for (int a = 0; a < 3; ++a)
#pragma unroll
                                        for (int b = 0; b < 3; ++b)
                                            B[a][b] = fma(c, pke<T>((3 * ca + a) * 24 + 3 * cb + b), B[a][b]);
                                }
#pragma unroll
                        for (int a = 0; a < 3; ++a)
#pragma unroll
                            for (int b = 0; b < 3; ++b)
#pragma unroll
                                for (int p = 0; p < 3; ++p)
                                    acc[m][3 * a + p] = pfma(B[a][b], v[3 * b + p], acc[m][3 * a + p]);
                    }
                }
            }
#pragma unroll
        for (int m = 0; m < NX; ++m) {
            if (i0 + m >= g.nx) break;
            const int n = (i0 + m) * ps + k * g.ny + j;
            const bool held = n == 0;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const T rd = (MODE == P_JACOBI || MODE == P_PRE) ? rdiag[3 * (size_t)n + d] : T(0);
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    const size_t at = (3 * d + p) * N + n;
                    const V ku = acc[m][3 * d + p];
                    // the node's own value, read again (L1): keeping it cost registers that a second CTA needs
                    const V uu = MODE == P_PRE ? pscale(prerelax * rd, f[at]) : u[at];
                    V o;
                    if (MODE == P_APPLY) {
                        o.x = held ? T(0) : ku.x;
                        o.y = held ? T(0) : ku.y;
                        dsum[p].x = fma(uu.x, o.x, dsum[p].x);
                        dsum[p].y = fma(uu.y, o.y, dsum[p].y);
                    } else {
                        const V fv = f[at];
                        o.x = held ? T(0) : fv.x - ku.x;
                        o.y = held ? T(0) : fv.y - ku.y;
                        if (MODE != P_DEFECT) {
                            o.x = fma(omega * o.x, rd, uu.x);
                            o.y = fma(omega * o.y, rd, uu.y);
                        }
                    }
                    out[at] = o;
                }
            }
        }
    }
    if (MODE == P_APPLY && partial) {   // partial[CTA][case]
        __shared__ double red[8][NR];
        double ds[NR];
#pragma unroll
        for (int p = 0; p < 3; ++p) ds[2 * p] = (double)dsum[p].x, ds[2 * p + 1] = (double)dsum[p].y;
#pragma unroll
        for (int r = 0; r < NR; ++r)
            for (int o = 16; o > 0; o >>= 1) ds[r] += __shfl_xor_sync(0xffffffffu, ds[r], o);
        if ((threadIdx.x & 31) == 0)
#pragma unroll
            for (int r = 0; r < NR; ++r) red[threadIdx.x >> 5][r] = ds[r];
        __syncthreads();
        if (threadIdx.x < NR) {
            double s = 0.0;
            for (int w = 0; w < 8; ++w) s += red[w][threadIdx.x];
            partial[(size_t)blockIdx.x * NR + threadIdx.x] = s;
        }
    }
}

// 1/diag of K per dof (the same for all six cases); 0 on node 0.
__global__ void pdiag_kernel(PGrid g, const double *__restrict__ CX, double *__restrict__ rdiag)
{
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= g.nnod()) return;
    const int j = (int)(n % g.ny);
    const long long t = n / g.ny;
    const int k = (int)(t % g.nz), i = (int)(t / g.nz);
    double dg[3] = {0.0, 0.0, 0.0};
    for (int ex = 0; ex < 2; ++ex)
        for (int ey = 0; ey < 2; ++ey)
            for (int ez = 0; ez < 2; ++ez) {
                const double c = CX[g.node(wrap(i - 1 + ex, g.nx), wrap(j - 1 + ey, g.ny), wrap(k - 1 + ez, g.nz))];
                const int ca = corner_of(1 - ex, 1 - ey, 1 - ez);
                for (int d = 0; d < 3; ++d) dg[d] += c * cPKe64[(3 * ca + d) * 24 + 3 * ca + d];
            }
    for (int d = 0; d < 3; ++d) rdiag[3 * n + d] = n == 0 ? 0.0 : 1.0 / dg[d];
}

// Coarse element scales: CX_c = 2 mean of the eight children (mgcg9.cu:753-781).
__global__ void pcoarse_cx_kernel(PGrid gc, const double *__restrict__ CXf, double *__restrict__ CXc)
{
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= gc.nnod()) return;
    const PGrid gf{2 * gc.nx, 2 * gc.ny, 2 * gc.nz};
    const int j = (int)(e % gc.ny);
    const long long t = e / gc.ny;
    const int k = (int)(t % gc.nz), i = (int)(t / gc.nz);
    double s = 0.0;
    for (int a = 0; a < 2; ++a)
        for (int c = 0; c < 2; ++c)
            for (int b = 0; b < 2; ++b) s += CXf[gf.node(2 * i + a, 2 * j + b, 2 * k + c)];
    CXc[e] = 0.25 * s;
}

// Full-weighting restriction (the transpose of the trilinear prolongation):
// coarse node (I, J, K) gathers fine nodes (2I + dx, ...) with weights
// 1, 1/2 per direction; node 0 gets zero.  Thread per coarse node and
// component (blockIdx.y), the three load-case pairs of that component.
__global__ void __launch_bounds__(256)
prestrict_kernel(PGrid gc, const float *__restrict__ rf, float *__restrict__ fc, const int *done)
{
    if (done && *done) return;
    const int n = (int)(blockIdx.x * blockDim.x + threadIdx.x), nc = (int)gc.nnod();
    if (n >= nc) return;
    const PGrid gf{2 * gc.nx, 2 * gc.ny, 2 * gc.nz};
    const size_t Nf = (size_t)gf.nnod();
    const float2 *src = reinterpret_cast<const float2 *>(rf) + 3 * blockIdx.y * Nf;
    const int J = n % gc.ny, t = n / gc.ny, K = t % gc.nz, I = t / gc.nz;
    float2 acc[3];
#pragma unroll
    for (int p = 0; p < 3; ++p) acc[p] = make_float2(0.f, 0.f);
#pragma unroll
    for (int dx = -1; dx <= 1; ++dx)
#pragma unroll
        for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
            for (int dy = -1; dy <= 1; ++dy) {
                const float w = (dx ? 0.5f : 1.f) * (dy ? 0.5f : 1.f) * (dz ? 0.5f : 1.f);
                const size_t fn = (size_t)gf.node(wrap(2 * I + dx, gf.nx), wrap(2 * J + dy, gf.ny),
                                                  wrap(2 * K + dz, gf.nz));
#pragma unroll
                for (int p = 0; p < 3; ++p) acc[p] = pfma(w, src[p * Nf + fn], acc[p]);
            }
    float2 *dst = reinterpret_cast<float2 *>(fc) + 3 * blockIdx.y * (size_t)nc + n;
#pragma unroll
    for (int p = 0; p < 3; ++p) dst[p * (size_t)nc] = n == 0 ? make_float2(0.f, 0.f) : acc[p];
}

// u_f += P u_c (trilinear, periodic); node 0 stays zero.  Thread per fine
// node and component (blockIdx.y).
__global__ void __launch_bounds__(256)
pprolong_kernel(PGrid gf, const float *__restrict__ uc, float *__restrict__ uf, const int *done)
{
    if (done && *done) return;
    const int n = (int)(blockIdx.x * blockDim.x + threadIdx.x), nf = (int)gf.nnod();
    if (n >= nf) return;
    const PGrid gc{gf.nx / 2, gf.ny / 2, gf.nz / 2};
    const size_t Nc = (size_t)gc.nnod();
    const float2 *src = reinterpret_cast<const float2 *>(uc) + 3 * blockIdx.y * Nc;
    float2 *dst = reinterpret_cast<float2 *>(uf) + 3 * blockIdx.y * (size_t)nf + n;
    const int j = n % gf.ny, t = n / gf.ny, k = t % gf.nz, i = t / gf.nz;
    float2 old[3];
#pragma unroll
    for (int p = 0; p < 3; ++p) old[p] = dst[p * (size_t)nf];
    const int ix[2] = {i >> 1, (i & 1) ? wrap((i >> 1) + 1, gc.nx) : (i >> 1)};
    const int iy[2] = {j >> 1, (j & 1) ? wrap((j >> 1) + 1, gc.ny) : (j >> 1)};
    const int iz[2] = {k >> 1, (k & 1) ? wrap((k >> 1) + 1, gc.nz) : (k >> 1)};
    const int mx = (i & 1) ? 2 : 1, my = (j & 1) ? 2 : 1, mz = (k & 1) ? 2 : 1;
    const float w = 1.f / (float)(mx * my * mz);
    float2 acc[3];
#pragma unroll
    for (int p = 0; p < 3; ++p) acc[p] = make_float2(0.f, 0.f);
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                if (a >= mx || c >= mz || b >= my) continue;
                const size_t q = (size_t)gc.node(ix[a], iy[b], iz[c]);
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    const float2 v = src[p * Nc + q];
                    acc[p].x += v.x;
                    acc[p].y += v.y;
                }
            }
#pragma unroll
    for (int p = 0; p < 3; ++p) dst[p * (size_t)nf] = n == 0 ? make_float2(0.f, 0.f) : pfma(w, acc[p], old[p]);
}

// Dense coarsest matrix (row per thread, no atomics); node 0's rows and
// columns become the identity.
__global__ void pdense_kernel(PGrid g, const double *__restrict__ CX, double *__restrict__ A)
{
    const int nd = (int)g.ndof();
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= nd) return;
    double *Ar = A + (long long)row * nd;
    for (int c = 0; c < nd; ++c) Ar[c] = 0.0;
    const int n = row / 3, d = row - 3 * n;
    if (n == 0) {
        Ar[row] = 1.0;
        return;
    }
    const int j = n % g.ny, t = n / g.ny, k = t % g.nz, i = t / g.nz;
    for (int ex = 0; ex < 2; ++ex)
        for (int ey = 0; ey < 2; ++ey)
            for (int ez = 0; ez < 2; ++ez) {
                const int ei = wrap(i - 1 + ex, g.nx), ej = wrap(j - 1 + ey, g.ny), ek = wrap(k - 1 + ez, g.nz);
                const double c = CX[g.node(ei, ej, ek)];
                const int ca = corner_of(1 - ex, 1 - ey, 1 - ez);
                for (int cb = 0; cb < 8; ++cb) {
                    const int bx = local_x(cb), by = local_y(cb), bz = local_z(cb);
                    const long long nb = g.node(wrap(ei + bx, g.nx), wrap(ej + by, g.ny), wrap(ek + bz, g.nz));
                    if (nb == 0) continue;
                    for (int b = 0; b < 3; ++b) Ar[3 * nb + b] += c * cPKe64[(3 * ca + d) * 24 + 3 * cb + b];
                }
            }
}

// Index of dof c = 3 n + d, load case r, in the pair planes of a grid of N nodes.
__device__ __forceinline__ long long pidx(int c, int r, int N)
{
    const int n = c / 3, d = c - 3 * n;
    return 2 * ((long long)(3 * d + (r >> 1)) * N + n) + (r & 1);
}

// y = M x on the coarsest grid for the six cases (warp per row; lower: the
// lower triangle of M, else the upper).  The FP32 side is in pair planes, the
// FP64 intermediate as [dof][case].
template <typename Tin, typename Tout>
__global__ void pgemv6_kernel(int n, const double *__restrict__ M, const Tin *__restrict__ x, Tout *__restrict__ y,
                              int lower, const int *done)
{
    if (done && *done) return;
    const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (row >= n) return;
    const int lo = lower ? 0 : row, hi = lower ? row + 1 : n;
    const double *mr = M + (long long)row * n;
    double s[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) s[r] = 0.0;
    for (int c = lo + lane; c < hi; c += 32) {
        const double m = mr[c];
#pragma unroll
        for (int r = 0; r < NR; ++r)
            s[r] = fma(m, (double)x[sizeof(Tin) == 4 ? pidx(c, r, n / 3) : (long long)c * NR + r], s[r]);
    }
#pragma unroll
    for (int r = 0; r < NR; ++r)
        for (int o = 16; o > 0; o >>= 1) s[r] += __shfl_xor_sync(0xffffffffu, s[r], o);
    if (lane < NR) {
        double v = s[0];
#pragma unroll
        for (int r = 1; r < NR; ++r)
            if (lane == r) v = s[r];
        y[sizeof(Tout) == 4 ? pidx(row, lane, n / 3) : (long long)row * NR + lane] = (Tout)v;
    }
}

// The right-hand sides f[dof][r] = -sum_e CX_e (Ke u0_r)[local dof].
__global__ void pload_kernel(PGrid g, const double *__restrict__ CX, double *__restrict__ F)
{
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= g.nnod()) return;
    const int j = (int)(n % g.ny);
    const long long t = n / g.ny;
    const int k = (int)(t % g.nz), i = (int)(t / g.nz);
    double f[3][NR] = {};
    for (int ex = 0; ex < 2; ++ex)
        for (int ey = 0; ey < 2; ++ey)
            for (int ez = 0; ez < 2; ++ez) {
                const double c = CX[g.node(wrap(i - 1 + ex, g.nx), wrap(j - 1 + ey, g.ny), wrap(k - 1 + ez, g.nz))];
                const int ca = corner_of(1 - ex, 1 - ey, 1 - ez);
                for (int d = 0; d < 3; ++d)
                    for (int r = 0; r < NR; ++r) f[d][r] -= c * cPG[(3 * ca + d) * NR + r];
            }
    const size_t N = (size_t)g.nnod();
    for (int d = 0; d < 3; ++d)
        for (int p = 0; p < 3; ++p)
            reinterpret_cast<double2 *>(F)[(3 * d + p) * N + n] =
                n == 0 ? make_double2(0.0, 0.0) : make_double2(f[d][2 * p], f[d][2 * p + 1]);
}

// ---- PCG over the six cases (FP64) ----------------------------------------

struct HScal {
    double res0[NR], rho[NR], alpha[NR], beta[NR], relres[NR], rr[NR];
    int done_r[NR], nit[NR];
    double tol;
    int iter, maxit, done, status;
    int pending;   // the last iteration's U += alpha P is still to be applied
};

// Per-CTA sums of K values -> partial[CTA][K].
template <int K>
__device__ __forceinline__ void block_partials(double (&v)[K], double *partial)
{
    __shared__ double red[8][K];
#pragma unroll
    for (int q = 0; q < K; ++q)
        for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int q = 0; q < K; ++q) red[threadIdx.x >> 5][q] = v[q];
    __syncthreads();
    if (threadIdx.x < K) {
        double s = 0.0;
        for (int w = 0; w < 8; ++w) s += red[w][threadIdx.x];
        partial[blockIdx.x * K + threadIdx.x] = s;
    }
}

// The vector kernels: a thread takes dofs c = 3 n + d a grid stride apart, all
// six cases of each (the order of the sums), so a warp reads 11 consecutive
// nodes of three planes per pair.  All are bound by HBM: at 128^3 pupdate 203
// us for 1.06 GB, pdot2 98 us for 0.60 GB, ppupdate 220 us for 1.51 GB (with
// the cases adjacent, 48 bytes between a warp's lanes, and U updated here:
// 589, 95 and 269 us).

// U = 0, R = F, float(R), |F_r|^2 partials.
__global__ void __launch_bounds__(256) pinit_kernel(size_t N, const double2 *__restrict__ F, double2 *__restrict__ U,
                                                    double2 *__restrict__ R, float2 *__restrict__ Rf,
                                                    double *__restrict__ partial)
{
    double s[NR] = {};
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < 3 * N; c += (size_t)gridDim.x * blockDim.x) {
        const size_t n = c / 3, d = c - 3 * n;
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            const size_t q = (3 * d + p) * N + n;
            const double2 f = F[q];
            U[q] = make_double2(0.0, 0.0);
            R[q] = f;
            Rf[q] = make_float2((float)f.x, (float)f.y);
            s[2 * p] = fma(f.x, f.x, s[2 * p]);
            s[2 * p + 1] = fma(f.y, f.y, s[2 * p + 1]);
        }
    }
    block_partials<NR>(s, partial);
}

// R -= alpha Q, float(R), |R_r|^2 partials.  U += alpha P waits for
// ppupdate_kernel, which reads P anyway.
__global__ void __launch_bounds__(256) pupdate_kernel(size_t N, double2 *__restrict__ R,
                                                      const double2 *__restrict__ Q, float2 *__restrict__ Rf,
                                                      const HScal *__restrict__ sc, double *__restrict__ partial)
{
    if (sc->done) return;
    double al[NR], s[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        al[r] = sc->alpha[r];
        s[r] = 0.0;
    }
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < 3 * N; c += (size_t)gridDim.x * blockDim.x) {
        const size_t n = c / 3, d = c - 3 * n;
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            const size_t q = (3 * d + p) * N + n;
            const double2 r = R[q], a = Q[q];
            const double2 v = make_double2(fma(-al[2 * p], a.x, r.x), fma(-al[2 * p + 1], a.y, r.y));
            R[q] = v;
            Rf[q] = make_float2((float)v.x, (float)v.y);
            s[2 * p] = fma(v.x, v.x, s[2 * p]);
            s[2 * p + 1] = fma(v.y, v.y, s[2 * p + 1]);
        }
    }
    block_partials<NR>(s, partial);
}

// r'z and r'z_old per case.
__global__ void __launch_bounds__(256) pdot2_kernel(size_t N, const double2 *__restrict__ R,
                                                    const float2 *__restrict__ Z, const float2 *__restrict__ Zo,
                                                    double *__restrict__ partial, const HScal *__restrict__ sc)
{
    if (sc && sc->done) return;
    double s[2 * NR] = {};
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < 3 * N; c += (size_t)gridDim.x * blockDim.x) {
        const size_t n = c / 3, d = c - 3 * n;
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            const size_t q = (3 * d + p) * N + n;
            const double2 r = R[q];
            const float2 z = Z[q];
            s[2 * p] = fma(r.x, (double)z.x, s[2 * p]);
            s[2 * p + 1] = fma(r.y, (double)z.y, s[2 * p + 1]);
            if (Zo) {
                const float2 o = Zo[q];
                s[NR + 2 * p] = fma(r.x, (double)o.x, s[NR + 2 * p]);
                s[NR + 2 * p + 1] = fma(r.y, (double)o.y, s[NR + 2 * p + 1]);
            }
        }
    }
    block_partials<2 * NR>(s, partial);
}

// U += alpha P, P = z + beta P, z_old = z (first: P = z and z_old = z alone).
// Once done, only a pending U update.  blockIdx.y = load-case pair.
__global__ void __launch_bounds__(256) ppupdate_kernel(size_t N, const float2 *__restrict__ Z, double2 *__restrict__ P,
                                                       double2 *__restrict__ U, float2 *__restrict__ Zo,
                                                       const HScal *__restrict__ sc, int first)
{
    const bool done = sc->done != 0, up = !first && sc->pending != 0;
    if (!first && !up) return;
    const int p = blockIdx.y;
    const double bx = first ? 0.0 : sc->beta[2 * p], by = first ? 0.0 : sc->beta[2 * p + 1];
    const double ax = up ? sc->alpha[2 * p] : 0.0, ay = up ? sc->alpha[2 * p + 1] : 0.0;
    for (size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x; n < N; n += (size_t)gridDim.x * blockDim.x)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const size_t q = (3 * d + p) * N + n;
            const double2 pv = P[q];
            if (up) {
                const double2 u = U[q];
                U[q] = make_double2(fma(ax, pv.x, u.x), fma(ay, pv.y, u.y));
            }
            if (done && !first) continue;
            const float2 z = Z[q];
            P[q] = first ? make_double2((double)z.x, (double)z.y)
                         : make_double2(fma(bx, pv.x, (double)z.x), fma(by, pv.y, (double)z.y));
            Zo[q] = z;
        }
}

// The fluctuations from the pair planes to the caller's [3 node + d][case].
__global__ void __launch_bounds__(256) pchi_kernel(size_t N, const double2 *__restrict__ U, double *__restrict__ chi)
{
    __shared__ double t[256 * 19];   // odd row length: no bank conflicts
    const size_t n0 = (size_t)blockIdx.x * 256, n = n0 + threadIdx.x;
    if (n < N)
#pragma unroll
        for (int q = 0; q < 9; ++q) {   // plane 3 d + p -> row entry 6 d + 2 p
            const double2 v = U[q * N + n];
            t[threadIdx.x * 19 + 2 * q] = v.x;
            t[threadIdx.x * 19 + 2 * q + 1] = v.y;
        }
    __syncthreads();
    const int cnt = (int)min((size_t)256, N - n0) * 18;
    for (int q = threadIdx.x; q < cnt; q += 256) chi[n0 * 18 + q] = t[(q / 18) * 19 + q % 18];
}

enum PFinish { PF_INIT = 0, PF_RHO0 = 1, PF_ALPHA = 2, PF_END = 3 };

constexpr int kFinThreads = 1024;
constexpr int kFinChunk = 3072;   // partials staged in shared memory at a time (24 KB), a multiple of 2 NR

// tot[q] = sum over CTAs b, in order, of partial[b][K].  The sum of a row is
// one serial chain of additions (its order is part of the result), so the
// partials are staged in shared memory by the whole CTA and thread q runs the
// chain from there, eight loads ahead: 60 us over the apply's 8192 partials
// (bound by the chain of additions), where one thread per row reading global
// memory took 400 us.
template <int K>
__device__ __forceinline__ void row_sums(int nb, const double *__restrict__ partial, double *st, double *tot)
{
    double s = 0.0;
    const long long n = (long long)nb * K;
    for (long long c0 = 0; c0 < n; c0 += kFinChunk) {
        const int m = (int)min((long long)kFinChunk, n - c0);
        __syncthreads();
        for (int q = threadIdx.x; q < m; q += kFinThreads) st[q] = partial[c0 + q];
        __syncthreads();
        if (threadIdx.x < K) {
            const int rows = m / K;
            int b = 0;
            for (; b + 8 <= rows; b += 8) {
                double v[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] = st[(b + e) * K + threadIdx.x];
#pragma unroll
                for (int e = 0; e < 8; ++e) s += v[e];
            }
            for (; b < rows; ++b) s += st[b * K + threadIdx.x];
        }
    }
    if (threadIdx.x < K) tot[threadIdx.x] = s;
}

// Sums the CTA partials and moves the scalars (one CTA).  INIT: res0; RHO0:
// rho; ALPHA: alpha = rho / p'q (0 for finished cases); END (partials: r'z,
// r'z_old; rr from the update): beta, relres, convergence per case,
// iteration count.
template <int WHICH>
__global__ void __launch_bounds__(kFinThreads) pfinish_kernel(int nb, const double *__restrict__ partial,
                                                              const double *__restrict__ partial_rr, HScal *sc)
{
    if (WHICH >= PF_ALPHA && sc->done) {
        if (WHICH == PF_ALPHA && threadIdx.x == 0) sc->pending = 0;
        return;
    }
    // pdot2 writes 2 NR rows (INIT: pinit, ALPHA: the apply, NR each)
    constexpr int K = (WHICH == PF_END || WHICH == PF_RHO0) ? 2 * NR : NR;
    __shared__ double st[kFinChunk], tot[2 * NR], tot_rr[NR];
    row_sums<K>(nb, partial, st, tot);
    if (WHICH == PF_END) row_sums<NR>(nb, partial_rr, st, tot_rr);
    __syncthreads();
    if (threadIdx.x != 0) return;
    if (WHICH == PF_INIT) {
        for (int r = 0; r < NR; ++r) {
            sc->res0[r] = sqrt(tot[r]);
            sc->relres[r] = 1.0;
            sc->nit[r] = sc->maxit;
            sc->done_r[r] = 0;
            if (!isfinite(sc->res0[r])) {
                sc->status = GPUTO_ERR_BREAKDOWN;
                sc->done_r[r] = 1;
            } else if (!(sc->res0[r] > 0.0)) {   // F_r = 0: chi_r = 0
                sc->done_r[r] = 1;
                sc->relres[r] = 0.0;
                sc->nit[r] = 0;
            }
        }
        int all = 1;
        for (int r = 0; r < NR; ++r) all &= sc->done_r[r];
        sc->done = all || sc->status || sc->maxit <= 0;
        sc->iter = 0;
    } else if (WHICH == PF_RHO0) {
        for (int r = 0; r < NR; ++r) sc->rho[r] = tot[r];
    } else if (WHICH == PF_ALPHA) {
        sc->pending = 0;
        for (int r = 0; r < NR; ++r) {
            const double a = sc->rho[r] / tot[r];
            if (sc->done_r[r]) {
                sc->alpha[r] = 0.0;
            } else if (!(tot[r] > 0.0) || !isfinite(a)) {
                sc->alpha[r] = 0.0;
                sc->status = GPUTO_ERR_BREAKDOWN;
                sc->done = 1;
            } else {
                sc->alpha[r] = a;
            }
        }
    } else {
        const int it = sc->iter;
        int all = 1;
        for (int r = 0; r < NR; ++r) {
            if (!sc->done_r[r]) {
                const double rz = tot[r], rzo = tot[NR + r];
                sc->beta[r] = (rz - rzo) / sc->rho[r];
                sc->rho[r] = rz;
                sc->rr[r] = tot_rr[r];
                sc->relres[r] = sqrt(tot_rr[r]) / sc->res0[r];
                if (!isfinite(sc->relres[r]) || !isfinite(sc->beta[r])) {
                    sc->status = GPUTO_ERR_BREAKDOWN;
                    sc->done_r[r] = 1;
                    sc->nit[r] = it;
                } else if (sc->relres[r] < sc->tol) {
                    sc->done_r[r] = 1;
                    sc->nit[r] = it;
                }
            } else {
                sc->beta[r] = 0.0;
            }
            all &= sc->done_r[r];
        }
        sc->pending = 1;
        sc->iter = it + 1;
        if (all || sc->status || it + 1 >= sc->maxit) sc->done = 1;
    }
}

// C_rs partials: per element W_r = u0_r + chi_r (24 values), C_rs += CX_e
// W_r' Ke W_s; the 21 upper-triangle entries per block.
__global__ void __launch_bounds__(256) pceff_kernel(PGrid g, const double *__restrict__ CX,
                                                    const double *__restrict__ U, double *__restrict__ partial)
{
    const long long N = g.nnod();
    double c[21] = {};
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < g.nnod();
         e += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(e % g.ny);
        const long long t = e / g.ny;
        const int k = (int)(t % g.nz), i = (int)(t / g.nz);
        long long nodes[8];
#pragma unroll
        for (int a = 0; a < 8; ++a)
            nodes[a] = g.node(wrap(i + local_x(a), g.nx), wrap(j + local_y(a), g.ny), wrap(k + local_z(a), g.nz));
        const double cx = CX[e];
        int q = 0;
#pragma unroll 1
        for (int r = 0; r < NR; ++r) {
            double w[24], kw[24];
#pragma unroll
            for (int a = 0; a < 8; ++a)
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    w[3 * a + d] = cPU0[r * 24 + 3 * a + d] + U[2 * ((3 * d + (r >> 1)) * N + nodes[a]) + (r & 1)];
#pragma unroll
            for (int m = 0; m < 24; ++m) {
                double s = 0.0;
#pragma unroll
                for (int p = 0; p < 24; ++p) s = fma(cPKe64[m * 24 + p], w[p], s);
                kw[m] = s;
            }
#pragma unroll 1
            for (int s2 = r; s2 < NR; ++s2, ++q) {
                double dot = 0.0;
#pragma unroll
                for (int a = 0; a < 8; ++a)
#pragma unroll
                    for (int d = 0; d < 3; ++d)
                        dot = fma(cPU0[s2 * 24 + 3 * a + d] + U[2 * ((3 * d + (s2 >> 1)) * N + nodes[a]) + (s2 & 1)],
                                  kw[3 * a + d], dot);
                // q indexes the upper triangle in row order
#pragma unroll
                for (int z = 0; z < 21; ++z)
                    if (z == q) c[z] = fma(cx, dot, c[z]);
            }
        }
    }
    block_partials<21>(c, partial);
}

inline unsigned nblk(long long n, int bs = 256) { return (unsigned)((n + bs - 1) / bs); }

}  // namespace

// ---------------------------------------------------------------------------

struct Homog {
    int nl = 0, device = 0, nc = 0;
    PGrid g[kMaxLevels]{};
    gputo_options opt{};
    cudaStream_t own_stream = nullptr;
    std::vector<void *> owned;
    size_t bytes = 0;
    // FP64 outer vectors (pair planes)
    double *F = nullptr, *U = nullptr, *R = nullptr, *P = nullptr, *Q = nullptr;
    float *Rf = nullptr, *Zold = nullptr;
    // per level: element scales (FP64 natural, FP32), 1/diag (FP64, FP32), FP32 buffers (pair planes)
    double *CXd[kMaxLevels]{}, *rdd[kMaxLevels]{};
    float *CXf[kMaxLevels]{}, *rdf[kMaxLevels]{};
    float *u0[kMaxLevels]{}, *u1[kMaxLevels]{}, *fl[kMaxLevels]{}, *rl[kMaxLevels]{};
    // coarsest
    double *A = nullptr, *Linv = nullptr, *LinvT = nullptr, *ctmp = nullptr;
    int *info = nullptr;
    HScal *sc = nullptr, *h_sc = nullptr;
    double *part = nullptr, *part_rr = nullptr, *part_c = nullptr;
    int nb_red = 0, nb_apply = 0;   // CTAs of the vector kernels and of the operator apply
    cudaGraphExec_t graph = nullptr;
    cudaStream_t graph_stream = nullptr;

    ~Homog()
    {
        if (own_stream) cudaStreamSynchronize(own_stream);
        if (graph) cudaGraphExecDestroy(graph);
        for (void *p : owned) cudaFree(p);
        if (h_sc) cudaFreeHost(h_sc);
        if (own_stream) cudaStreamDestroy(own_stream);
    }

    template <typename T>
    int alloc(T **p, long long count)
    {
        const size_t b = sizeof(T) * (size_t)std::max(count, 1LL);
        cudaError_t e = cudaMalloc((void **)p, b);
        if (e != cudaSuccess) {
            cudaGetLastError();
            *p = nullptr;
            set_error("cudaMalloc of " + std::to_string(b) + " bytes failed: " + cudaGetErrorString(e));
            return e == cudaErrorMemoryAllocation ? GPUTO_ERR_OOM : GPUTO_ERR_CUDA;
        }
        owned.push_back(*p);
        bytes += b;
        GPUTO_CUDA(cudaMemsetAsync(*p, 0, b, own_stream));
        return GPUTO_OK;
    }

    int create(int nx, int ny, int nz, int nl_, const gputo_options *o)
    {
        if (o) opt = *o;
        else gputo_default_options(&opt);
        if (nl_ < 1 || nl_ > kMaxLevels || nx < 2 || ny < 2 || nz < 2) {
            set_error("periodic cell sizes must be >= 2 and 1 <= nl <= 12");
            return GPUTO_ERR_ARG;
        }
        const int m = 1 << (nl_ - 1);
        if (nx % m || ny % m || nz % m || nx / m < 2 || ny / m < 2 || nz / m < 2) {
            set_error("nx, ny, nz must be divisible by 2^(nl-1), with at least 2 coarsest elements per direction");
            return GPUTO_ERR_ARG;
        }
        if (opt.nswp < 1 || !(opt.omega > 0) || opt.check_every < 1) {
            set_error("homogenization needs nswp >= 1, omega > 0 and check_every >= 1");
            return GPUTO_ERR_ARG;
        }
        nl = nl_;
        for (int l = 0; l < nl; ++l) g[l] = PGrid{nx >> l, ny >> l, nz >> l};
        nc = (int)g[nl - 1].ndof();
        if (nc > opt.max_coarse_dofs) {
            set_error("coarsest grid has " + std::to_string(nc) + " dofs, above max_coarse_dofs=" +
                      std::to_string(opt.max_coarse_dofs) + "; use more levels");
            return GPUTO_ERR_ARG;
        }
        GPUTO_CUDA(cudaGetDevice(&device));
        GPUTO_CUDA(cudaStreamCreateWithFlags(&own_stream, cudaStreamNonBlocking));
        const long long nv = g[0].ndof() * NR;
        int s = GPUTO_OK;
        if (!s) s = alloc(&F, nv);
        if (!s) s = alloc(&U, nv);
        if (!s) s = alloc(&R, nv);
        if (!s) s = alloc(&P, nv);
        if (!s) s = alloc(&Q, nv);
        if (!s) s = alloc(&Rf, nv);
        if (!s) s = alloc(&Zold, nv);
        for (int l = 0; l < nl && !s; ++l) {
            const long long nvl = g[l].ndof() * NR;
            s = alloc(&CXd[l], g[l].nnod());
            if (!s) s = alloc(&CXf[l], g[l].nnod());
            if (!s) s = alloc(&rdd[l], g[l].ndof());
            if (!s) s = alloc(&rdf[l], g[l].ndof());
            if (!s) s = alloc(&u0[l], nvl);
            if (!s) s = alloc(&u1[l], nvl);
            if (!s && l > 0) s = alloc(&fl[l], nvl);
            if (!s) s = alloc(&rl[l], nvl);
        }
        if (!s) s = alloc(&A, (long long)nc * nc);
        if (!s) s = alloc(&Linv, (long long)nc * nc);
        if (!s) s = alloc(&LinvT, (long long)nc * nc);
        if (!s) s = alloc(&ctmp, (long long)nc * NR);
        if (!s) s = alloc(&info, 4);
        if (!s) s = alloc(&sc, 1);
        nb_red = (int)std::min<long long>(kHBlocks, std::max(1LL, (g[0].ndof() + 255) / 256));
        nb_apply = (int)nblk(g[0].nnod());
        if (!s) s = alloc(&part, (long long)std::max(nb_apply, nb_red) * 2 * NR);
        if (!s) s = alloc(&part_rr, (long long)nb_red * NR);
        if (!s) s = alloc(&part_c, (long long)nb_red * 21);
        if (s) return s;
        GPUTO_CUDA(cudaMallocHost((void **)&h_sc, sizeof(HScal)));
        GPUTO_CUDA(cudaStreamSynchronize(own_stream));
        return GPUTO_OK;
    }

    int upload_ke(const double *Ke, cudaStream_t st)
    {
        for (int m = 0; m < 576; ++m)
            if (!std::isfinite(Ke[m])) {
                set_error("Ke0 has a non-finite entry");
                return GPUTO_ERR_ARG;
            }
        float kf[576];
        for (int m = 0; m < 576; ++m) kf[m] = (float)Ke[m];
        // u0_r at the local corners and G = Ke u0
        double u0h[NR * 24] = {}, gh[24 * NR] = {};
        for (int a = 0; a < 8; ++a) {
            const double x = local_x(a), y = local_y(a), z = local_z(a);
            const double f[NR][3] = {{x, 0, 0}, {0, y, 0}, {0, 0, z}, {0, z / 2, y / 2}, {z / 2, 0, x / 2},
                                     {y / 2, x / 2, 0}};
            for (int r = 0; r < NR; ++r)
                for (int d = 0; d < 3; ++d) u0h[r * 24 + 3 * a + d] = f[r][d];
        }
        for (int m = 0; m < 24; ++m)
            for (int r = 0; r < NR; ++r) {
                double sum = 0.0;
                for (int p = 0; p < 24; ++p) sum += Ke[m * 24 + p] * u0h[r * 24 + p];
                gh[m * NR + r] = sum;
            }
        GPUTO_CUDA(cudaMemcpyToSymbolAsync(cPKe64, Ke, sizeof(double) * 576, 0, cudaMemcpyHostToDevice, st));
        GPUTO_CUDA(cudaMemcpyToSymbolAsync(cPKe32, kf, sizeof(kf), 0, cudaMemcpyHostToDevice, st));
        GPUTO_CUDA(cudaMemcpyToSymbolAsync(cPU0, u0h, sizeof(u0h), 0, cudaMemcpyHostToDevice, st));
        GPUTO_CUDA(cudaMemcpyToSymbolAsync(cPG, gh, sizeof(gh), 0, cudaMemcpyHostToDevice, st));
        GPUTO_CUDA(cudaStreamSynchronize(st));   // the host arrays are on the stack
        return GPUTO_OK;
    }

    // Hierarchy for CX (device, natural order, FP64).
    int setup(const double *CX, cudaStream_t st)
    {
        GPUTO_CUDA(cudaMemcpyAsync(CXd[0], CX, sizeof(double) * g[0].nnod(), cudaMemcpyDeviceToDevice, st));
        for (int l = 1; l < nl; ++l)
            pcoarse_cx_kernel<<<nblk(g[l].nnod()), 256, 0, st>>>(g[l], CXd[l - 1], CXd[l]);
        for (int l = 0; l < nl; ++l) {
            pdiag_kernel<<<nblk(g[l].nnod()), 256, 0, st>>>(g[l], CXd[l], rdd[l]);
            launch_cast_f32(g[l].nnod(), CXd[l], CXf[l], st);
            launch_cast_f32(g[l].ndof(), rdd[l], rdf[l], st);
        }
        pdense_kernel<<<nblk(nc), 256, 0, st>>>(g[nl - 1], CXd[nl - 1], A);
        launch_cholesky(nc, A, info, st);
        launch_tri_inverse(nc, A, Linv, LinvT, st);
        pload_kernel<<<nblk(g[0].nnod()), 256, 0, st>>>(g[0], CXd[0], F);
        count_launches(4 * nl + 4);
        int h_info = 0;
        GPUTO_CUDA(cudaMemcpyAsync(&h_info, info, sizeof(int), cudaMemcpyDeviceToHost, st));
        GPUTO_CUDA(cudaStreamSynchronize(st));
        GPUTO_CUDA(cudaGetLastError());
        if (h_info) {
            set_error("coarsest periodic matrix is not positive definite (pivot " + std::to_string(h_info) + ")");
            return GPUTO_ERR_NOT_SPD;
        }
        return GPUTO_OK;
    }

    // Tiles of a sweep: 32 (y) x 8 (z) node columns per CTA, or the whole
    // (shorter) y row by 256 / ny, and nx planes per thread.
    struct SweepGrid {
        unsigned grid;
        int ty, ntj, nt;
    };
    static SweepGrid sweep_grid(const PGrid &q, int nxt)
    {
        const int ty = std::min(q.ny, 32), tz = 256 / ty;
        const int ntj = (q.ny + ty - 1) / ty, ntk = (q.nz + tz - 1) / tz;
        return SweepGrid{(unsigned)(ntj * ntk) * (unsigned)((q.nx + nxt - 1) / nxt), ty, ntj, ntj * ntk};
    }

    // Two nodes per thread halve the CTAs and the plane reads: from about one
    // wave of CTAs on (2 x 148 of 512 nodes).  Below that the sweeps are bound
    // by latency (7-8 us) and more CTAs are worth more.
    template <int MODE>
    void sweep(int l, const float *u, const float *f, float *out, const int *done, cudaStream_t st)
    {
        const float om = (float)opt.omega, pr = (float)opt.prerelax;
        if (g[l].nnod() >= 2LL * 148 * 512) {
            const SweepGrid s = sweep_grid(g[l], 2);
            psweep_kernel<float, MODE, 2>
                <<<s.grid, 256, 0, st>>>(g[l], s.ty, s.ntj, s.nt, CXf[l], u, f, rdf[l], out, om, pr, nullptr, done);
        } else {
            const SweepGrid s = sweep_grid(g[l], 1);
            psweep_kernel<float, MODE, 1>
                <<<s.grid, 256, 0, st>>>(g[l], s.ty, s.ntj, s.nt, CXf[l], u, f, rdf[l], out, om, pr, nullptr, done);
        }
        count_launches(1);
    }

    // z = M r on all six cases (FP32), the solver's V-cycle schedule.
    void vcycle(const float *r0, float *z0, const int *done, cudaStream_t st)
    {
        const int ns = opt.nswp;
        auto buf = [&](int l, int which) -> float * {
            if (l == 0) return which ? z0 : u0[0];
            return which ? u1[l] : u0[l];
        };
        for (int l = 0; l < nl; ++l) {
            const float *f = l == 0 ? r0 : fl[l];
            if (l > 0) {
                prestrict_kernel<<<dim3(nblk(g[l].nnod()), 3), 256, 0, st>>>(g[l], rl[l - 1], fl[l], done);
                count_launches(1);
            }
            if (l < nl - 1) {
                for (int s = 0; s < ns; ++s) {
                    if (s == 0) sweep<P_PRE>(l, nullptr, f, buf(l, 0), done, st);
                    else sweep<P_JACOBI>(l, buf(l, (s - 1) & 1), f, buf(l, s & 1), done, st);
                }
                sweep<P_DEFECT>(l, buf(l, (ns - 1) & 1), f, rl[l], done, st);
            } else {
                const unsigned nbw = (unsigned)((nc * 32 + 255) / 256);
                pgemv6_kernel<float, double><<<nbw, 256, 0, st>>>(nc, Linv, f, ctmp, 1, done);
                pgemv6_kernel<double, float><<<nbw, 256, 0, st>>>(nc, LinvT, ctmp, buf(l, 1), 0, done);
                count_launches(2);
            }
        }
        for (int l = nl - 2; l >= 0; --l) {
            const float *f = l == 0 ? r0 : fl[l];
            int cur = (ns - 1) & 1;
            pprolong_kernel<<<dim3(nblk(g[l].nnod()), 3), 256, 0, st>>>(g[l], buf(l + 1, 1), buf(l, cur), done);
            count_launches(1);
            // starting from buffer (ns - 1) & 1, ns sweeps end in buffer 1
            for (int s = 0; s < ns; ++s) {
                sweep<P_JACOBI>(l, buf(l, cur), f, buf(l, cur ^ 1), done, st);
                cur ^= 1;
            }
        }
    }

    // One flexible PCG iteration of all six cases.
    void iteration(cudaStream_t st)
    {
        const size_t N = (size_t)g[0].nnod();
        const int *done = &sc->done;
        const dim3 gp((unsigned)(nb_red + 2) / 3, 3);
        psweep_kernel<double, P_APPLY, 1><<<nb_apply, 256, 0, st>>>(g[0], 0, 0, 0, CXd[0], P, nullptr, nullptr, Q, 1.0,
                                                                    0.0, part, done);
        pfinish_kernel<PF_ALPHA><<<1, kFinThreads, 0, st>>>(nb_apply, part, nullptr, sc);
        pupdate_kernel<<<nb_red, 256, 0, st>>>(N, (double2 *)R, (const double2 *)Q, (float2 *)Rf, sc, part_rr);
        vcycle(Rf, u1[0], done, st);
        pdot2_kernel<<<nb_red, 256, 0, st>>>(N, (const double2 *)R, (const float2 *)u1[0], (const float2 *)Zold, part, sc);
        pfinish_kernel<PF_END><<<1, kFinThreads, 0, st>>>(nb_red, part, part_rr, sc);
        ppupdate_kernel<<<gp, 256, 0, st>>>(N, (const float2 *)u1[0], (double2 *)P, (double2 *)U, (float2 *)Zold, sc, 0);
        count_launches(7);
    }

    int run_graph(int batch, cudaStream_t st)
    {
        if (!graph || graph_stream != st) {
            if (graph) cudaGraphExecDestroy(graph);
            graph = nullptr;
            cudaGraph_t gr;
            GPUTO_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
            iteration(st);
            GPUTO_CUDA(cudaStreamEndCapture(st, &gr));
            cudaError_t e = cudaGraphInstantiate(&graph, gr, 0);
            cudaGraphDestroy(gr);
            GPUTO_CUDA(e);
            graph_stream = st;
        }
        for (int b = 0; b < batch; ++b) GPUTO_CUDA(cudaGraphLaunch(graph, st));
        return GPUTO_OK;
    }

    int solve(double tol, int maxit, double *Ceff, double *relres, int *nit, cudaStream_t st)
    {
        if (maxit < 0 || !(tol >= 0)) {
            set_error("maxit must be >= 0 and tol >= 0");
            return GPUTO_ERR_ARG;
        }
        const size_t N = (size_t)g[0].nnod();
        const dim3 gp((unsigned)(nb_red + 2) / 3, 3);
        HScal z{};
        z.tol = tol;
        z.maxit = maxit;
        GPUTO_CUDA(cudaMemcpyAsync(sc, &z, sizeof(HScal), cudaMemcpyHostToDevice, st));
        pinit_kernel<<<nb_red, 256, 0, st>>>(N, (const double2 *)F, (double2 *)U, (double2 *)R, (float2 *)Rf, part);
        pfinish_kernel<PF_INIT><<<1, kFinThreads, 0, st>>>(nb_red, part, nullptr, sc);
        vcycle(Rf, u1[0], &sc->done, st);
        pdot2_kernel<<<nb_red, 256, 0, st>>>(N, (const double2 *)R, (const float2 *)u1[0], nullptr, part, nullptr);
        pfinish_kernel<PF_RHO0><<<1, kFinThreads, 0, st>>>(nb_red, part, nullptr, sc);
        ppupdate_kernel<<<gp, 256, 0, st>>>(N, (const float2 *)u1[0], (double2 *)P, (double2 *)U, (float2 *)Zold, sc, 1);
        count_launches(5);
        GPUTO_CUDA(cudaStreamSynchronize(st));   // the host struct z is on the stack
        int it = 0;
        for (;;) {
            GPUTO_CUDA(cudaMemcpyAsync(h_sc, sc, sizeof(HScal), cudaMemcpyDeviceToHost, st));
            GPUTO_CUDA(cudaStreamSynchronize(st));
            if (h_sc->done || it >= maxit) break;
            const int batch = std::min(opt.check_every, maxit - it);
            if (opt.use_graph) {
                int s = run_graph(batch, st);
                if (s) return s;
            } else {
                for (int b = 0; b < batch; ++b) iteration(st);
            }
            it += batch;
        }
        GPUTO_CUDA(cudaGetLastError());
        for (int r = 0; r < NR; ++r) {
            if (relres) relres[r] = h_sc->relres[r];
            if (nit) nit[r] = h_sc->done_r[r] ? h_sc->nit[r] : h_sc->iter;
        }
        if (h_sc->status) {
            set_error("homogenization PCG breakdown (non-finite loads or p'q <= 0)");
            return h_sc->status;
        }
        if (Ceff) {
            const unsigned nbc = (unsigned)std::min<long long>(kHBlocks, (long long)nblk(g[0].nnod()));
            pceff_kernel<<<nbc, 256, 0, st>>>(g[0], CXd[0], U, part_c);
            count_launches(1);
            std::vector<double> hp((size_t)nbc * 21);
            GPUTO_CUDA(cudaMemcpyAsync(hp.data(), part_c, sizeof(double) * hp.size(), cudaMemcpyDeviceToHost, st));
            GPUTO_CUDA(cudaStreamSynchronize(st));
            double c[21] = {};
            for (unsigned b = 0; b < nbc; ++b)
                for (int q = 0; q < 21; ++q) c[q] += hp[(size_t)b * 21 + q];
            const double inv = 1.0 / (double)g[0].nnod();
            int q = 0;
            for (int r = 0; r < NR; ++r)
                for (int s2 = r; s2 < NR; ++s2, ++q) Ceff[r * NR + s2] = Ceff[s2 * NR + r] = c[q] * inv;
        }
        return GPUTO_OK;
    }
};

}  // namespace gputo

struct gputo_homog {
    gputo::Homog h;
};

extern "C" {

int gputo_homog_create(gputo_homog **out, int nx, int ny, int nz, int nl, const gputo_options *opt)
{
    if (!out) return GPUTO_ERR_ARG;
    *out = nullptr;
    int dev = 0, major = 0, n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) {
        cudaGetLastError();
        gputo::set_error("no CUDA device is visible");
        return GPUTO_ERR_NO_DEVICE;
    }
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
    if (major != 10) {
        gputo::set_error("gputo is built for sm_100a (B200)");
        return GPUTO_ERR_NO_DEVICE;
    }
    auto *h = new gputo_homog();
    const int st = h->h.create(nx, ny, nz, nl, opt);
    if (st) {
        delete h;
        return st;
    }
    *out = h;
    return GPUTO_OK;
}

void gputo_homog_destroy(gputo_homog *h) { delete h; }

size_t gputo_homog_device_bytes(const gputo_homog *h) { return h ? h->h.bytes : 0; }

int gputo_homog_solve_dev(gputo_homog *hh, const double *Ke0, const double *CX, double tol, int maxit,
                          double *Ceff, double *relres, int *nit, double *chi, void *stream)
{
    if (!hh || !Ke0 || !CX) return GPUTO_ERR_ARG;
    gputo::Homog &h = hh->h;
    cudaStream_t st = stream ? (cudaStream_t)stream : h.own_stream;
    int s = h.upload_ke(Ke0, st);
    if (!s) s = h.setup(CX, st);
    if (!s) s = h.solve(tol, maxit, Ceff, relres, nit, st);
    if (!s && chi) {
        const size_t N = (size_t)h.g[0].nnod();
        gputo::pchi_kernel<<<(unsigned)((N + 255) / 256), 256, 0, st>>>(N, (const double2 *)h.U, chi);
        gputo::count_launches(1);
        GPUTO_CUDA(cudaStreamSynchronize(st));
        GPUTO_CUDA(cudaGetLastError());
    }
    return s;
}

}  // extern "C"
