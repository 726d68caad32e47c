// Design-loop steps that the MATLAB driver runs around the solve
// (Cantilever/TOP3D125MGCGCUDA/top3D125modCuda.m:95-96,109,139-141,163).
#include "gputo_internal.h"
#include "hadamard.h"

#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

namespace gputo {

// Element matrix for the energy kernel.  Constant memory is per translation
// unit without relocatable device code, so this file keeps its own copy,
// written by upload_fine_ke() together with the solver's.  When Ke has the
// cube element's Hadamard pattern, its eight constants (per device) select
// the Hadamard-basis energy pass.
__constant__ double cKeD[576];
static HadamardKe g_design_hk[64];
static std::mutex g_design_hk_mu;   // writers (upload) and readers (launch) on other threads

int upload_design_ke(const double *Ke_host, cudaStream_t st)
{
    int dev = 0;
    GPUTO_CUDA(cudaGetDevice(&dev));
    HadamardKe hk;
    (void)hadamard_ke(Ke_host, &hk);   // sets ok = false without the pattern
    {
        std::lock_guard<std::mutex> lock(g_design_hk_mu);
        g_design_hk[dev < 64 ? dev : 63] = hk;
    }
    GPUTO_CUDA(cudaMemcpyToSymbolAsync(cKeD, Ke_host, sizeof(double) * 576, 0,
                                       cudaMemcpyHostToDevice, st));
    return GPUTO_OK;
}

constexpr int kMaxFilterRadius = 6;           // stencil up to 13^3
constexpr int kFilterW = 2 * kMaxFilterRadius + 1;
__constant__ double cFilterH[kFilterW * kFilterW * kFilterW];

// The CTAs' compliance partials, summed by the last CTA to finish with all its
// threads, in a fixed order.
__device__ __forceinline__ void sum_compliance(double csum, double *partial, unsigned *ticket, double *compliance)
{
    __shared__ double red[8];
    __shared__ bool is_last;
    for (int o = 16; o > 0; o >>= 1) csum += __shfl_xor_sync(0xffffffffu, csum, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = csum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += red[w];
        partial[blockIdx.x] = v;
        __threadfence();
        is_last = (atomicAdd(ticket, 1u) == gridDim.x - 1);
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    double v = 0.0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x) v += __ldcg(partial + b);
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        v = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += red[w];
        *compliance = v;
        *ticket = 0;
    }
}

// ce_e = u_e^T Ke u_e, dc_e = dsK_e ce_e, and sum_e CX_e ce_e, dense 24x24
// product with Ke from constant memory (1152 FLOP), thread per element: any Ke
// without the cube element's Hadamard pattern.  U is in the solver frame: the
// driver's U(cMat) gather (top3D125modCuda.m:39-41,139) lists element nodes in
// an order mirrored in y, which matches the y-negated U the MEX hands back, so
// both give the same ce.
__global__ void __launch_bounds__(256)
element_energy_kernel(Grid g, const double *__restrict__ U, const double *__restrict__ CX,
                      const double *__restrict__ dsK, double *__restrict__ ce,
                      double *__restrict__ dc, double *__restrict__ partial, unsigned *ticket,
                      double *compliance)
{
    const long long nel = g.nel();
    double csum = 0.0;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < nel;
         e += (long long)gridDim.x * blockDim.x) {
        const long long t = e / g.ny;
        const int j = (int)(e - t * g.ny);
        const int i = (int)(t / g.nz);
        const int k = (int)(t - (long long)i * g.nz);
        double s = 0.0, ue[24];
#pragma unroll
        for (int a = 0; a < 8; ++a) {
            const long long n = g.node(i + local_x(a), j + local_y(a), k + local_z(a));
#pragma unroll
            for (int d = 0; d < 3; ++d) ue[3 * a + d] = U[3 * n + d];
        }
#pragma unroll 4
        for (int m = 0; m < 24; ++m) {
            double tm = 0.0;
#pragma unroll
            for (int q = 0; q < 24; ++q) tm = fma(cKeD[m * 24 + q], ue[q], tm);
            s = fma(ue[m], tm, s);
        }
        if (ce) ce[e] = s;
        if (dc) dc[e] = dsK[e] * s;
        if (CX) csum = fma(CX[e], s, csum);
    }
    if (compliance) sum_compliance(csum, partial, ticket, compliance);
}

__device__ __forceinline__ void cp_async8(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// The same for the cube element's Ke, as (T u_e)' (S / 64) (T u_e) in the
// element's Hadamard basis.  A CTA takes 32 (y) x 4 (z) element columns and
// marches along x: node planes come by cp.async (8 bytes: rows start anywhere)
// into a ring of four, two ahead of the one in use, and each face is
// transformed once for the two elements that share it (about 116 FP64
// operations per element).  Work items are (tile, x chunk) pairs, so any grid
// runs on as many CTAs as there are partial slots.  57 bytes and 116 FP64
// operations per element bound it (36 and 27 us at 256 x 128 x 128); it is
// held by latency at the 16 warps per SM its registers allow.  Per call at 256
// x 128 x 128 78 us, on 193 x 97 x 95 (a last y tile of one column) 67 us, on
// 114 x 82 x 50 31 us; 148, 92 and 62 us with a thread per element gathering
// its 24 corner values and a one-thread sum of the CTAs' partials.  Tiles of 8
// rows took 82, 67 and 33 us.
// Thin grids have tiles of their own (FIXED = false, energy_tile()).
constexpr int kEnY = 32, kEnZ = 4, kEnT = kEnY * kEnZ, kEnRing = 4;

template <bool FIXED>
__global__ void __launch_bounds__(kEnT, 512 / kEnT)
element_energy_march_kernel(Grid g, HC<double> hc, int ty_, int tz_, int xc, int ntj, int ntk, long long nitems,
                            const double *__restrict__ U, const double *__restrict__ CX,
                            const double *__restrict__ dsK, double *__restrict__ ce, double *__restrict__ dc,
                            double *__restrict__ partial, unsigned *ticket, double *compliance)
{
    // values of a plane tile: 3 (ty + 1) (tz + 1) is largest at 1 x kEnT columns
    constexpr int kMax = FIXED ? 3 * (kEnY + 1) * (kEnZ + 1) : 3 * 2 * (kEnT + 1), kPos = (kMax + kEnT - 1) / kEnT;
    __shared__ double ring[kEnRing][kMax];
    const int ty = FIXED ? kEnY : ty_, tz = FIXED ? kEnZ : tz_, row = 3 * (ty + 1), plane = row * (tz + 1);
    const int tid = threadIdx.x, w = tid / ty, l = tid - w * ty;
    const long long ps = 3LL * (g.ny + 1) * (g.nz + 1);   // values per node plane
    double csum = 0.0;
    for (long long item = blockIdx.x; item < nitems; item += gridDim.x) {
        const long long tile = item % ((long long)ntj * ntk);
        const int i0 = (int)(item / ((long long)ntj * ntk)) * xc, i1 = min(i0 + xc, g.nx);
        const int j0 = (int)(tile % ntj) * ty, k0 = (int)(tile / ntj) * tz;
        const int np = i1 - i0 + 1;
        long long off[kPos];   // this thread's values of a plane tile, clamped to the grid
#pragma unroll
        for (int q = 0; q < kPos; ++q) {
            const int p = tid + kEnT * q, kk = p / row, c = p - kk * row;
            const int v = min(3 * j0 + c, 3 * g.ny + 2);
            off[q] = (long long)min(k0 + kk, g.nz) * (3 * (g.ny + 1)) + v;
        }
        auto fetch = [&](int t) {
            if (t < np) {
                const double *src = U + (i0 + t) * ps;
                double *dst = ring[t % kEnRing];
#pragma unroll
                for (int q = 0; q < kPos; ++q)
                    if (tid + kEnT * q < plane) cp_async8(dst + tid + kEnT * q, src + off[q]);
            }
            cp_async_commit();
        };
        const int j = j0 + l, k = k0 + w;
        const bool mine = j < g.ny && k < g.nz && (FIXED || w < tz);
        const long long es = (long long)g.ny * g.nz;
        long long e = (long long)i0 * es + (long long)k * g.ny + j;   // element in front of plane t
        __syncthreads();   // the ring is free
#pragma unroll
        for (int t = 0; t < kEnRing - 1; ++t) fetch(t);
        auto face = [&](int t, double (&F)[HF]) {
            cp_async_wait<kEnRing - 2>();
            __syncthreads();   // plane t has landed for everyone; slot (t - 1) is free
            fetch(t + kEnRing - 1);
            const double *P = ring[t % kEnRing] + (FIXED ? w : min(w, tz - 1)) * row + 3 * l;
#pragma unroll
            for (int cy = 0; cy < 2; ++cy)
#pragma unroll
                for (int cz = 0; cz < 2; ++cz)
#pragma unroll
                    for (int d = 0; d < 3; ++d) F[(2 * cy + cz) * 4 + d] = P[cz * row + 3 * cy + d];
            face_h(F);
        };
        auto element = [&](const double (&Fp)[HF], const double (&Fn)[HF], double cx, double ds) {
            if (mine) {
                const double s = element_energy_h(Fp, Fn, hc);
                if (ce) ce[e] = s;
                if (dc) dc[e] = ds * s;
                csum = fma(cx, s, csum);
            }
            e += es;
        };
        double Fa[HF], Fb[HF];
        // the scales of the element after the next face, a step ahead
        double cx = mine && CX ? CX[e] : 0.0, ds = mine && dc ? dsK[e] : 0.0, cn = 0.0, dn = 0.0;
        auto ahead = [&](int t) {
            if (mine && t + 1 < np) {
                if (CX) cn = CX[e + es];
                if (dc) dn = dsK[e + es];
            }
        };
        face(0, Fa);
        for (int t = 1; t < np; t += 2) {   // two planes a trip: no face is copied
            ahead(t);
            face(t, Fb);
            element(Fa, Fb, cx, ds);
            if (t + 1 < np) {
                cx = cn, ds = dn;
                ahead(t + 1);
                face(t + 1, Fa);
                element(Fb, Fa, cx, ds);
                cx = cn, ds = dn;
            }
        }
        cp_async_wait<0>();   // the empty trailing groups
    }
    if (compliance) sum_compliance(csum, partial, ticket, compliance);
}

// Planes per x chunk of a marching kernel: tiles x chunks CTAs run in waves of
// 'slots', and a CTA takes its planes and 'extra' more (halo planes, filling
// the ring), so the chunk count with the smallest waves x (planes + extra):
// one full wave on large grids, a plane or two per CTA where latency counts
// (the radius-2 filter of 64 x 32 x 32 elements 26.5 -> 18.5 us per call).
static int chunk_planes(int nx, long long tiles, long long slots, int extra)
{
    int best = nx;
    long long cost = -1;
    for (int c = 1; c <= nx && c <= 512; ++c) {
        const int xc = (nx + c - 1) / c;
        const long long n = (nx + xc - 1) / xc, t = ((tiles * n + slots - 1) / slots) * (xc + extra);
        if (cost < 0 || t < cost) {
            cost = t;
            best = xc;
        }
    }
    return best;
}

// Columns of a CTA of the energy pass.  Up to 16 elements along y, or two along
// z, 32 x 4 columns would lie outside the grid for the most part, so a CTA
// takes all of that direction and what its threads allow of the other.
static void energy_tile(const Grid &g, int &ty, int &tz)
{
    ty = kEnY, tz = kEnZ;
    if (g.ny <= 16) {
        ty = g.ny;
        tz = std::min(kEnT / ty, g.nz);
    } else if (g.nz <= 2) {
        tz = g.nz;
        ty = std::min(kEnT / tz, g.ny);
    }
}

// One partial slot per CTA: kEnergyCtas of them, or nblocks for the dense
// kernel.  The plan's CTAs are the launch's: with the dense kernel's count of
// 256-thread CTAs as their limit a CTA ran many short chunks, each filling the
// ring anew (allocation-free call on 9 x 2 x 300 elements 255 us, now 39; 64 x
// 32 x 32 55 and 35; 40 and 42 with a thread per element).
void launch_element_energy_blocks(const Grid &g, const double *U, const double *CX,
                                  const double *dsK, double *ce, double *dc, double *partial,
                                  unsigned *ticket, double *compliance, int nblocks,
                                  cudaStream_t st)
{
    int dev = 0;
    cudaGetDevice(&dev);
    HadamardKe hk;
    {
        std::lock_guard<std::mutex> lock(g_design_hk_mu);
        hk = g_design_hk[dev < 64 ? dev : 63];
    }
    if (hk.ok) {
        int ty, tz;
        energy_tile(g, ty, tz);
        const int ntj = (g.ny + ty - 1) / ty, ntk = (g.nz + tz - 1) / tz;
        const long long tiles = (long long)ntj * ntk;
        const int xc = chunk_planes(g.nx, tiles, (512 / kEnT) * 148, 5);
        const long long items = tiles * ((g.nx + xc - 1) / xc);
        auto *kernel = ty == kEnY && tz == kEnZ ? element_energy_march_kernel<true> : element_energy_march_kernel<false>;
        kernel<<<(unsigned)std::min<long long>(items, kEnergyCtas), kEnT, 0, st>>>(
            g, make_hc<double>(hk), ty, tz, xc, ntj, ntk, items, U, CX, dsK, ce, dc, partial, ticket, compliance);
    } else {
        element_energy_kernel<<<(unsigned)nblocks, 256, 0, st>>>(g, U, CX, dsK, ce, dc, partial, ticket, compliance);
    }
    count_launches(1);
}

void launch_element_energy(const Grid &g, const double *U, const double *CX, const double *dsK,
                           double *ce, double *dc, double *partial, unsigned *ticket,
                           double *compliance, cudaStream_t st)
{
    long long nb = (g.nel() + 255) / 256;
    if (nb > kEnergyCtas) nb = kEnergyCtas;
    if (nb < 1) nb = 1;
    launch_element_energy_blocks(g, U, CX, dsK, ce, dc, partial, ticket, compliance, (int)nb, st);
}

// MATLAB 'symmetric' padding: mirror including the edge sample.
__device__ __forceinline__ int mirror_index(int i, int n)
{
    while (i < 0 || i >= n) {
        if (i < 0) i = -1 - i;
        if (i >= n) i = 2 * n - 1 - i;
    }
    return i;
}

// out = correlate(in ./ div, h) [/ sum h], elements in (y fastest) order
// (imfilter(..., 'symmetric'), top3D125modCuda.m:109,140-141).
//
// Shared-memory tiled: a CTA owns an output tile of 32 (y, one per lane) x 8
// (z, one per warp) element columns and marches along x through a chunk of
// planes.  Each input plane of the tile plus its R-wide halo, mirrored at the
// grid faces, is loaded from global memory once (the quotient in ./ div is
// taken at load time) into a ring of 2R + 2 plane slots; the loads of the
// plane FPF steps ahead are in flight while the current output plane is
// computed from shared memory, with one barrier per plane (the slot being
// filled is never one being read).  The weights are in constant memory and
// the same for every lane (broadcast).  The sum runs in the order x offset,
// z offset, y offset, as a direct 3-D correlation would.
constexpr int kFTY = 32, kFTZ = 8, kFPF = 2;

template <int R> struct FiltTile {
    static constexpr int W = 2 * R + 1;
    static constexpr int TYH = kFTY + 2 * R, TZH = kFTZ + 2 * R;
    static constexpr int PLANE = TYH * TZH;
    static constexpr int NPOS = (PLANE + 255) / 256;   // halo-tile positions per thread
    static constexpr int SLOTS = 2 * R + 2;
    static constexpr size_t bytes = sizeof(double) * SLOTS * PLANE;
};

template <int R>
__global__ void __launch_bounds__(256)
filter_kernel(Grid g, const double *__restrict__ in, const double *__restrict__ div,
              double *__restrict__ out, double scale, int xc)
{
    using FT = FiltTile<R>;
    constexpr int W = FT::W;
    extern __shared__ double fs[];   // [SLOTS][PLANE]
    const int tid = threadIdx.x, ly = tid & 31, lz = tid >> 5;
    const int j0 = blockIdx.x * kFTY, k0 = blockIdx.y * kFTZ;
    const int x0 = blockIdx.z * xc, x1 = min(x0 + xc, g.nx);
    const long long ps = (long long)g.ny * g.nz;   // elements per x plane
    // this thread's positions in a halo tile: offset inside an x plane (-1: none)
    long long off[FT::NPOS];
#pragma unroll
    for (int q = 0; q < FT::NPOS; ++q) {
        const int p = tid + 256 * q;
        off[q] = -1;
        if (p < FT::PLANE) {
            const int zz = p / FT::TYH, yy = p - zz * FT::TYH;
            off[q] = (long long)mirror_index(k0 + zz - R, g.nz) * g.ny + mirror_index(j0 + yy - R, g.ny);
        }
    }
    auto fetch = [&](int px, double (&v)[FT::NPOS]) {
        const long long base = (long long)mirror_index(px, g.nx) * ps;
#pragma unroll
        for (int q = 0; q < FT::NPOS; ++q)
            if (off[q] >= 0) {
                const long long s = base + off[q];
                v[q] = div ? in[s] / div[s] : in[s];
            }
    };
    auto put = [&](int px, const double (&v)[FT::NPOS]) {
        double *P = fs + ((px - x0 + R) % FT::SLOTS) * FT::PLANE;
#pragma unroll
        for (int q = 0; q < FT::NPOS; ++q)
            if (off[q] >= 0) P[tid + 256 * q] = v[q];
    };
    // planes x0 - R .. x0 + R - 1 before the first output plane
    for (int px = x0 - R; px < x0 + R; ++px) {
        double v[FT::NPOS];
        fetch(px, v);
        put(px, v);
    }
    double pre[kFPF][FT::NPOS];
#pragma unroll
    for (int d = 0; d < kFPF; ++d)
        if (x0 + d < x1) fetch(x0 + R + d, pre[d]);
    const int j = j0 + ly, k = k0 + lz;
    const bool mine = j < g.ny && k < g.nz;
    for (int i0 = x0; i0 < x1; i0 += kFPF)
#pragma unroll
    for (int pf = 0; pf < kFPF; ++pf) {   // register sets by constant index
        const int i = i0 + pf;
        if (i >= x1) break;               // the same for the whole CTA
        put(i + R, pre[pf]);
        __syncthreads();
        if (i + kFPF < x1) fetch(i + R + kFPF, pre[pf]);   // in flight while plane i is computed
        if (mine) {
            double acc = 0.0;
#pragma unroll
            for (int a = -R; a <= R; ++a) {
                const double *P = fs + ((i + a - x0 + R) % FT::SLOTS) * FT::PLANE;
#pragma unroll
                for (int c = -R; c <= R; ++c) {
                    const double *row = P + (lz + R + c) * FT::TYH + ly + R;
#pragma unroll
                    for (int b = -R; b <= R; ++b)
                        acc = fma(cFilterH[((a + R) * W + (b + R)) * W + (c + R)], row[b], acc);
                }
            }
            out[(long long)i * ps + (long long)k * g.ny + j] = acc * scale;
        }
    }
}

// The correlation for R = 2 and 3, decomposed by x plane and by distance: the
// weight of a tap depends on its offsets' magnitudes alone, so plane q
// contributes P_a(q) = sum over the classes (m, n), 0 <= m <= n <= R, of
// h[a][m][n] (the sum of the plane's values at offsets (+-m, +-n) and (+-n,
// +-m)) to the outputs at planes q - a and q + a.  A thread has ZR output rows
// along z of one y: it reads its (ZR + 2R) x (2R + 1) window of the plane once,
// folds each row to its R + 1 values |dy| = 0..R, and forms the class sums of
// its rows from those.  It keeps the 2R + 1 outputs of each row that are still
// open in registers (a ring indexed at compile time: the march is unrolled by
// 2R + 1).  At R = 2 that is 36 FP64 operations and 10-15 shared loads per
// output and plane, against 80 and 25 without the classes and the row reuse.
// Output i sums P_R(i - R), ..., P_0(i), ..., P_R(i + R) in plane order.
// Planes arrive by cp.async into a ring of kFPS shared-memory slots (input,
// and the divisor when given), kFPS - 1 planes ahead of the one in use, one
// barrier per plane (a second one with a divisor, whose quotients are taken in
// place once per plane).  At 256 x 128 x 128 per call: R = 2 with a divisor 57
// us (84 us with all 25 taps read and multiplied), without 42 us (73), R = 3 90
// and 69 us (177 and 165); at 64 x 32 x 32 18.5 and 22 us (27 and 52).
constexpr int kFPS = 4;

template <int R, int ZR> struct FiltClass {
    static constexpr int TYH = kFTY + 2 * R, TZH = 8 * ZR + 2 * R;
    static constexpr int PLANE = TYH * TZH;
    static constexpr int NPOS = (PLANE + 255) / 256;
    static constexpr size_t bytes(bool div) { return sizeof(double) * (div ? 2 : 1) * kFPS * PLANE; }
};

template <int R, int ZR, bool DIV>
__global__ void __launch_bounds__(256, 2)
filter_class_kernel(Grid g, const double *__restrict__ in, const double *__restrict__ div,
                    double *__restrict__ out, double scale, int xc)
{
    using FT = FiltClass<R, ZR>;
    constexpr int W = 2 * R + 1;
    extern __shared__ double fs[];   // [kFPS][PLANE] input planes, then (DIV) [kFPS][PLANE] divisor planes
    double *fd = fs + kFPS * FT::PLANE;
    const int tid = threadIdx.x, ly = tid & 31, lg = tid >> 5;
    const int j0 = blockIdx.x * kFTY, k0 = blockIdx.y * (8 * ZR);
    const int x0 = blockIdx.z * xc, x1 = min(x0 + xc, g.nx);
    const long long ps = (long long)g.ny * g.nz;
    int off[FT::NPOS];   // offsets in an x plane (the launcher keeps planes of 2^31 elements away)
#pragma unroll
    for (int q = 0; q < FT::NPOS; ++q) {
        const int p = tid + 256 * q;
        off[q] = -1;
        if (p < FT::PLANE) {
            const int zz = p / FT::TYH, yy = p - zz * FT::TYH;
            off[q] = mirror_index(k0 + zz - R, g.nz) * g.ny + mirror_index(j0 + yy - R, g.ny);
        }
    }
    const int T = x1 - x0 + 2 * R;   // planes x0 - R .. x1 + R - 1
    auto fetch = [&](int t) {
        if (t < T) {
            const long long base = (long long)mirror_index(x0 - R + t, g.nx) * ps;
            const int sl = (t % kFPS) * FT::PLANE;
#pragma unroll
            for (int q = 0; q < FT::NPOS; ++q)
                if (off[q] >= 0) {
                    cp_async8(fs + sl + tid + 256 * q, in + base + off[q]);
                    if (DIV) cp_async8(fd + sl + tid + 256 * q, div + base + off[q]);
                }
        }
        cp_async_commit();
    };
    const int j = j0 + ly, kr = k0 + ZR * lg;   // output column; first of the thread's rows
    const bool jok = j < g.ny;
    double acc[W][ZR];
#pragma unroll
    for (int s = 0; s < W; ++s)
#pragma unroll
        for (int r = 0; r < ZR; ++r) acc[s][r] = 0.0;
#pragma unroll
    for (int t = 0; t < kFPS - 1; ++t) fetch(t);
    for (int t0 = 0; t0 < T; t0 += W)
#pragma unroll
    for (int u = 0; u < W; ++u) {
        const int t = t0 + u;
        if (t >= T) break;                 // the same for the whole CTA
        const int q = x0 - R + t;          // this plane
        cp_async_wait<kFPS - 2>();         // this thread's copies of plane t have landed
        __syncthreads();                   // everyone's have; slot (t - 1) mod kFPS is free
        fetch(t + kFPS - 1);
        double *P = fs + (t % kFPS) * FT::PLANE;
        if (DIV) {
            const double *D = fd + (t % kFPS) * FT::PLANE;
#pragma unroll
            for (int v = 0; v < FT::NPOS; ++v)
                if (off[v] >= 0) P[tid + 256 * v] = P[tid + 256 * v] / D[tid + 256 * v];
            __syncthreads();
        }
        // row folds: e[row][m] = sum of the values at |dy| = m
        double e[ZR + 2 * R][R + 1];
#pragma unroll
        for (int z = 0; z < ZR + 2 * R; ++z) {
            const double *row = P + (ZR * lg + z) * FT::TYH + ly + R;
            e[z][0] = row[0];
#pragma unroll
            for (int m = 1; m <= R; ++m) e[z][m] = row[-m] + row[m];
        }
#pragma unroll
        for (int r = 0; r < ZR; ++r) {
            double pa[R + 1];
#pragma unroll
            for (int a = 0; a <= R; ++a) pa[a] = 0.0;
#pragma unroll
            for (int m = 0; m <= R; ++m)
#pragma unroll
                for (int n = m; n <= R; ++n) {
                    // rows +-m with |dy| = n and, for m < n, rows +-n with |dy| = m
                    double c = m ? e[r + R - m][n] + e[r + R + m][n] : e[r + R][n];
                    if (m < n) c += e[r + R - n][m] + e[r + R + n][m];
#pragma unroll
                    for (int a = 0; a <= R; ++a) pa[a] = fma(cFilterH[((a + R) * W + (m + R)) * W + (n + R)], c, pa[a]);
                }
            // output q + a (a = -R..R) sits in slot (u + a + R) mod W
#pragma unroll
            for (int a = -R; a <= R; ++a) acc[(u + a + R) % W][r] += pa[a < 0 ? -a : a];
        }
        // output q - R is complete
        const int i = q - R;
#pragma unroll
        for (int r = 0; r < ZR; ++r) {
            if (i >= x0 && jok && kr + r < g.nz)
                out[(long long)i * ps + (long long)(kr + r) * g.ny + j] = acc[u][r] * scale;
            acc[u][r] = 0.0;
        }
    }
    cp_async_wait<0>();   // the empty trailing groups
}

// Radius 1 with four output rows along z per thread, tiles of 32 (y) x 32 (z)
// outputs: a thread reads its 6 x 3 window of each plane once for its four
// outputs, 4.5 shared loads per output instead of 9 (the 32 x 8 tiles above
// are bound by shared-memory bandwidth in FP64).  The same ring and the same
// plane sums as filter_class_kernel with the four weights of radius 1.
constexpr int kF1Y = 32, kF1Z = 32;

template <bool DIV>
__global__ void __launch_bounds__(256)
filter_r1_kernel(Grid g, const double *__restrict__ in, const double *__restrict__ div,
                 double *__restrict__ out, double scale, int xc)
{
    constexpr int TYH = kF1Y + 2, TZH = kF1Z + 2, PLANE = TYH * TZH, NPOS = (PLANE + 255) / 256;
    extern __shared__ double fs[];   // [kFPS][PLANE] input planes, then (DIV) [kFPS][PLANE] divisor planes
    double *fd = fs + kFPS * PLANE;
    const int tid = threadIdx.x, ly = tid & 31, lg = tid >> 5;
    const int j0 = blockIdx.x * kF1Y, k0 = blockIdx.y * kF1Z;
    const int x0 = blockIdx.z * xc, x1 = min(x0 + xc, g.nx);
    const long long ps = (long long)g.ny * g.nz;
    long long off[NPOS];
#pragma unroll
    for (int q = 0; q < NPOS; ++q) {
        const int p = tid + 256 * q;
        off[q] = -1;
        if (p < PLANE) {
            const int zz = p / TYH, yy = p - zz * TYH;
            off[q] = (long long)mirror_index(k0 + zz - 1, g.nz) * g.ny + mirror_index(j0 + yy - 1, g.ny);
        }
    }
    const int T = x1 - x0 + 2;   // planes x0 - 1 .. x1
    auto fetch = [&](int t) {
        if (t < T) {
            const long long base = (long long)mirror_index(x0 - 1 + t, g.nx) * ps;
            const int sl = (t % kFPS) * PLANE;
#pragma unroll
            for (int q = 0; q < NPOS; ++q)
                if (off[q] >= 0) {
                    cp_async8(fs + sl + tid + 256 * q, in + base + off[q]);
                    if (DIV) cp_async8(fd + sl + tid + 256 * q, div + base + off[q]);
                }
        }
        cp_async_commit();
    };
    const int j = j0 + ly, kr = k0 + 4 * lg;   // output column; first of the thread's four rows
    const bool jok = j < g.ny;
    const double w0 = cFilterH[13], w1 = cFilterH[12], w2 = cFilterH[9], w3 = cFilterH[0];
    double acc[3][4];
#pragma unroll
    for (int s = 0; s < 3; ++s)
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[s][r] = 0.0;
#pragma unroll
    for (int t = 0; t < kFPS - 1; ++t) fetch(t);
    for (int t0 = 0; t0 < T; t0 += 6)
#pragma unroll
    for (int u = 0; u < 6; ++u) {
        const int t = t0 + u;
        if (t >= T) break;   // the same for the whole CTA
        const int q = x0 - 1 + t;
        cp_async_wait<kFPS - 2>();
        __syncthreads();
        fetch(t + kFPS - 1);
        double *P = fs + (t % kFPS) * PLANE;
        if (DIV) {   // in / divisor, in place, once per plane
            const double *D = fd + (t % kFPS) * PLANE;
#pragma unroll
            for (int v = 0; v < NPOS; ++v)
                if (off[v] >= 0) P[tid + 256 * v] = P[tid + 256 * v] / D[tid + 256 * v];
            __syncthreads();
        }
        double v[6][3];
#pragma unroll
        for (int r = 0; r < 6; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) v[r][c] = P[(4 * lg + r) * TYH + ly + c];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const double s0 = v[r + 1][1];
            const double s1 = (v[r + 1][0] + v[r + 1][2]) + (v[r][1] + v[r + 2][1]);
            const double s2 = (v[r][0] + v[r][2]) + (v[r + 2][0] + v[r + 2][2]);
            const double p0 = fma(w2, s2, fma(w1, s1, w0 * s0));
            const double p1 = fma(w3, s2, fma(w2, s1, w1 * s0));
            // output q + a (a = -1, 0, 1) sits in slot (u + a + 1) mod 3
            acc[u % 3][r] += p1;
            acc[(u + 1) % 3][r] += p0;
            acc[(u + 2) % 3][r] += p1;
        }
        // output q - 1 is complete
        const int i = q - 1, sl = u % 3;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            if (i >= x0 && jok && kr + r < g.nz) out[(long long)i * ps + (long long)(kr + r) * g.ny + j] = acc[sl][r] * scale;
            acc[sl][r] = 0.0;
        }
    }
    cp_async_wait<0>();   // the empty trailing groups
}

template <int R>
int filter_launch(const Grid &g, const double *in, const double *div, double *out, double scale,
                  cudaStream_t st)
{
    using FT = FiltTile<R>;
    if (FT::bytes > 48 * 1024) {
        static std::once_flag once[64];
        int dev = 0;
        GPUTO_CUDA(cudaGetDevice(&dev));
        cudaError_t e = cudaSuccess;
        std::call_once(once[dev < 64 ? dev : 63], [&]() {
            e = cudaFuncSetAttribute(filter_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)FT::bytes);
        });
        GPUTO_CUDA(e);
    }
    if constexpr (R == 1) {
        constexpr size_t plane = sizeof(double) * (kF1Y + 2) * (kF1Z + 2);
        const size_t smem = (div ? 2 : 1) * kFPS * plane;
        if (div) {
            static std::once_flag once[64];
            int dev = 0;
            GPUTO_CUDA(cudaGetDevice(&dev));
            cudaError_t e = cudaSuccess;
            std::call_once(once[dev < 64 ? dev : 63], [&]() {
                e = cudaFuncSetAttribute(filter_r1_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(2 * kFPS * plane));
            });
            GPUTO_CUDA(e);
        }
        const unsigned ty = (unsigned)((g.ny + kF1Y - 1) / kF1Y), tz = (unsigned)((g.nz + kF1Z - 1) / kF1Z);
        const long long tiles = (long long)ty * tz;
        // x chunks for about 592 CTAs (4 per SM, one wave), at least 6 planes
        // each (a chunk reads two more than it writes); where those leave SMs
        // without a CTA the call is bound by latency, and chunks are as short as
        // give every SM one (64 x 32 x 32: 22.9 -> 18.1 us per call)
        const long long want = std::max(1LL, (592 + tiles - 1) / tiles);
        long long xl = std::max(6LL, ((long long)g.nx + want - 1) / want);
        if (tiles * ((g.nx + xl - 1) / xl) < 148) xl = std::max(1LL, (g.nx * tiles + 147) / 148);
        const int xc = (int)std::min<long long>(xl, g.nx);
        const unsigned tx = (unsigned)((g.nx + xc - 1) / xc);
        if (div)
            filter_r1_kernel<true><<<dim3(ty, tz, tx), 256, smem, st>>>(g, in, div, out, scale, xc);
        else
            filter_r1_kernel<false><<<dim3(ty, tz, tx), 256, smem, st>>>(g, in, div, out, scale, xc);
        count_launches(1);
        return GPUTO_OK;
    }
    const unsigned ty = (unsigned)((g.ny + kFTY - 1) / kFTY), tz = (unsigned)((g.nz + kFTZ - 1) / kFTZ);
    // x chunks: about 1184 CTAs (8 per SM) in all, at least 16 planes each
    const long long tiles = (long long)ty * tz;
    const long long want = std::max(1LL, (1184 + tiles - 1) / tiles);
    int xc = (int)std::max(16LL, ((long long)g.nx + want - 1) / want);
    if (xc > g.nx) xc = g.nx;
    const unsigned tx = (unsigned)((g.nx + xc - 1) / xc);
    filter_kernel<R><<<dim3(ty, tz, tx), 256, FT::bytes, st>>>(g, in, div, out, scale, xc);
    count_launches(1);
    return GPUTO_OK;
}

// R = 2 and 3: ZR output rows per thread.
template <int R, int ZR, bool DIV>
int filter_class_launch(const Grid &g, const double *in, const double *div, double *out, double scale, cudaStream_t st)
{
    using FT = FiltClass<R, ZR>;
    static std::once_flag once[64];
    int dev = 0;
    GPUTO_CUDA(cudaGetDevice(&dev));
    cudaError_t e = cudaSuccess;
    std::call_once(once[dev < 64 ? dev : 63], [&]() {
        e = cudaFuncSetAttribute(filter_class_kernel<R, ZR, DIV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)FT::bytes(DIV));
    });
    GPUTO_CUDA(e);
    const unsigned ty = (unsigned)((g.ny + kFTY - 1) / kFTY), tz = (unsigned)((g.nz + 8 * ZR - 1) / (8 * ZR));
    const long long tiles = (long long)ty * tz;
    const int xc = chunk_planes(g.nx, tiles, 2 * 148, 2 * R + 3);
    const unsigned tx = (unsigned)((g.nx + xc - 1) / xc);
    filter_class_kernel<R, ZR, DIV><<<dim3(ty, tz, tx), 256, FT::bytes(DIV), st>>>(g, in, div, out, scale, xc);
    count_launches(1);
    return GPUTO_OK;
}

int launch_filter(const Grid &g, const double *in, const double *div, double *out, double rmin,
                  int normalize, cudaStream_t st)
{
    const int R = (int)std::ceil(rmin) - 1;
    if (R < 0 || R > kMaxFilterRadius) return GPUTO_ERR_ARG;
    const int W = 2 * R + 1;
    std::vector<double> h((size_t)W * W * W);
    double hs = 0.0;
    for (int a = -R; a <= R; ++a)
        for (int b = -R; b <= R; ++b)
            for (int c = -R; c <= R; ++c) {
                const double v = rmin - std::sqrt((double)(a * a + b * b + c * c));
                const double w = v > 0 ? v : 0.0;
                h[((a + R) * W + (b + R)) * W + (c + R)] = w;
                hs += w;
            }
    static double last_rmin[64];
    static bool have[64] = {};
    int dev = 0;
    GPUTO_CUDA(cudaGetDevice(&dev));
    const int slot = dev < 64 ? dev : 63;
    if (!have[slot] || rmin != last_rmin[slot] || dev >= 64) {   // constant memory is per device
        GPUTO_CUDA(cudaMemcpyToSymbolAsync(cFilterH, h.data(), sizeof(double) * h.size(), 0,
                                           cudaMemcpyHostToDevice, st));
        GPUTO_CUDA(cudaStreamSynchronize(st));
        last_rmin[slot] = rmin;
        have[slot] = true;
    }
    const double scale = normalize ? 1.0 / hs : 1.0;
    const bool small_plane = (long long)g.ny * g.nz < (1LL << 31);   // the class kernels' plane offsets are 32-bit
    switch (R) {
    case 0: return filter_launch<0>(g, in, div, out, scale, st);
    case 1: return filter_launch<1>(g, in, div, out, scale, st);
    case 2:
        if (!small_plane) return filter_launch<2>(g, in, div, out, scale, st);
        // four rows per thread make a tile 32 rows high: fewer where z is shorter
        // than that.  With a divisor, 4 / 1 or 2 rows and, in brackets, all taps
        // read: 1000 x 1000 x 8 262 / 136 us (145), 700 x 700 x 16 142 / 102 (146).
        // Radius 3 has tiles of 16 rows (1000 x 1000 x 4 258 us, 293 with all taps).
        if (g.nz <= 8) return div ? filter_class_launch<2, 1, true>(g, in, div, out, scale, st)
                                  : filter_class_launch<2, 1, false>(g, in, div, out, scale, st);
        if (g.nz <= 16) return div ? filter_class_launch<2, 2, true>(g, in, div, out, scale, st)
                                   : filter_class_launch<2, 2, false>(g, in, div, out, scale, st);
        return div ? filter_class_launch<2, 4, true>(g, in, div, out, scale, st)
                   : filter_class_launch<2, 4, false>(g, in, div, out, scale, st);
    case 3:
        if (!small_plane) return filter_launch<3>(g, in, div, out, scale, st);
        return div ? filter_class_launch<3, 2, true>(g, in, div, out, scale, st)
                   : filter_class_launch<3, 2, false>(g, in, div, out, scale, st);
    case 4: return filter_launch<4>(g, in, div, out, scale, st);
    case 5: return filter_launch<5>(g, in, div, out, scale, st);
    default: return filter_launch<6>(g, in, div, out, scale, st);
    }
}

}  // namespace gputo

namespace gputo {

// SIMP stiffness and its derivative (top3D125modCuda.m:124,130):
//   CX = Emin + x^p (E0 - Emin),   dsK = -p (E0 - Emin) x^(p-1)
__global__ void simp_kernel(long long n, const double *__restrict__ x, double penal, double E0,
                            double Emin, double *__restrict__ CX, double *__restrict__ dsK)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const double xi = x[i];
        const double xp1 = pow(xi, penal - 1.0);
        CX[i] = Emin + xp1 * xi * (E0 - Emin);
        if (dsK) dsK[i] = -penal * (E0 - Emin) * xp1;
    }
}

void launch_simp(long long n, const double *x, double penal, double E0, double Emin, double *CX,
                 double *dsK, cudaStream_t st)
{
    long long nb = (n + 255) / 256;
    if (nb > 4736) nb = 4736;
    simp_kernel<<<(unsigned)nb, 256, 0, st>>>(n, x, penal, E0, Emin, CX, dsK);
    count_launches(1);
}

// ---------------------------------------------------------------------------
// The OC update and the projection threshold are each one cooperative launch
// that loops on the device: every iteration sums over the design, the CTAs
// meet at a grid barrier, and every CTA then adds all CTAs' partials in the
// same order and takes the same decision, so one barrier per iteration is
// enough.  The passes re-read 67 MB (OC) or 33 MB (threshold) at the bench
// grid, which stay in the 126 MB L2.  (One launch per step, queued up to the
// limit of 60-64 steps, with a one-thread sum of up to 1184 partials per step,
// took 0.82 ms for the OC update and 0.78 ms for the projection of 4.19M
// elements; 0.17 and 0.14 ms now.  Bound by FP64 latency: two elements in
// flight per thread, and two CTAs of 512 threads per SM, 20-25 % faster than
// one.)
// ---------------------------------------------------------------------------
constexpr int kLoopThreads = 512;
constexpr int kLoopPerSm = 2;

struct LoopSync {
    unsigned arrived, left, failed;   // zero between launches
};

// How long a grid barrier waits before it gives up (2 s but in tests), and
// whether the last CTA leaves out its first arrival (test hook).
struct LoopWait {
    uint32_t wait_ns;
    int skip;
};

static LoopWait loop_wait()
{
    const SweepFaultHook h = sweep_fault_hook();
    return LoopWait{h.wait_ns, h.skip_stage >= 0};
}

// All CTAs of the launch have arrived (round: 1, 2, ... in every CTA alike).
// False when the wait gave up.
__device__ __forceinline__ bool grid_barrier(LoopSync *sync, unsigned round, LoopWait lw)
{
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (!lw.skip || round > 1 || blockIdx.x != gridDim.x - 1) atomicAdd(&sync->arrived, 1u);
        const unsigned want = round * gridDim.x;
        unsigned seen;
        uint64_t t0 = 0;
        ok = 1;
        for (unsigned it = 0;; ++it) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&sync->arrived) : "memory");
            if (seen >= want) break;
            if ((it & 63u) == 0) {
                uint64_t t;
                asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
                if (t0 == 0) t0 = t;
                else if (t - t0 > lw.wait_ns) {
                    ok = 0;
                    break;
                }
            }
        }
        __threadfence();
    }
    __syncthreads();
    return ok != 0;
}

// The last CTA to leave makes the counters ready for the next launch, and
// turns the result into a failure when any CTA's barrier gave up.
__device__ __forceinline__ void grid_leave(LoopSync *sync, bool ok, int *done)
{
    __syncthreads();
    if (threadIdx.x != 0) return;
    if (!ok) atomicExch(&sync->failed, 1u);
    __threadfence();
    if (atomicAdd(&sync->left, 1u) == gridDim.x - 1) {
        __threadfence();
        if (atomicExch(&sync->failed, 0u)) *(volatile int *)done = 2;
        sync->arrived = 0;
        sync->left = 0;
    }
}

// CTA sums of K values -> partial[q][CTA].
template <int K>
__device__ __forceinline__ void loop_partials(double (&v)[K], double *partial)
{
    __shared__ double red[K][kLoopThreads / 32];
#pragma unroll
    for (int q = 0; q < K; ++q) {
        for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
        if ((threadIdx.x & 31) == 0) red[q][threadIdx.x >> 5] = v[q];
    }
    __syncthreads();
    if (threadIdx.x < K) {
        double s = 0.0;
        for (int w = 0; w < kLoopThreads / 32; ++w) s += red[threadIdx.x][w];
        partial[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = s;
    }
}

// tot[q] = sum over CTAs of partial[q][CTA], a warp per quantity.
template <int K>
__device__ __forceinline__ void loop_totals(const double *partial, double *tot)
{
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (w < K) {
        double s = 0.0;
        for (unsigned b = lane; b < gridDim.x; b += 32) s += __ldcg(partial + (size_t)w * gridDim.x + b);
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) tot[w] = s;
    }
    __syncthreads();
}

// OC update with bisection on the Lagrange multiplier
// (top3D125modCuda.m:143-151).  An iteration sums the candidate designs of the
// next kOcDepth bisection steps at once: the 2^kOcDepth - 1 multipliers that
// those steps could try, whichever way they go, formed with the same
// arithmetic as one step after the other.  The candidates' sums use ocP (1 /
// lmid); the design written at the end divides, as the MATLAB line does.  As
// in the MATLAB loop it is the design of the last multiplier tried.
struct OcState {
    double l1, l2, lmid;
    int steps, done;   // done: 1 finished, 2 a grid barrier gave up
};

constexpr int kOcDepth = 2;   // measured at the bench grid: 1, 2, 3 steps a pass 215, 186, 216 us per update
constexpr int kOcCand = (1 << kOcDepth) - 1;

__device__ __forceinline__ double oc_candidate(double x, double ocp, double lmid, double move)
{
    // max(max(min(min(ocP/lmid, xU), 1), xL), 0)
    const double xU = x + move, xL = x - move;
    double v = ocp / lmid;
    v = fmin(v, xU);
    v = fmin(v, 1.0);
    v = fmax(v, xL);
    return fmax(v, 0.0);
}

__global__ void __launch_bounds__(kLoopThreads, kLoopPerSm)
oc_update_kernel(long long n, const double *__restrict__ x, const double *dc, const double *dv0, double *ocp,
                 double move, double volfrac, double *xnew, double *partial, LoopSync *sync, LoopWait lw, int max_steps,
                 OcState *state)
{
    __shared__ double tot[kOcCand];
    const long long i0 = (long long)blockIdx.x * kLoopThreads + threadIdx.x, st = (long long)gridDim.x * kLoopThreads;
    unsigned round = 0;
    bool ok = true;
    double l1 = 0.0, l2, lmid;
    int steps = 0;
    bool done;
    {
        double s[1] = {0.0};
        for (long long i = i0; i < n; i += st) {
            const double v = x[i] * sqrt(-dc[i] / dv0[i]);
            ocp[i] = v;
            s[0] += v;
        }
        loop_partials<1>(s, partial);
        ok = grid_barrier(sync, ++round, lw);
        loop_totals<1>(partial, tot);
        l2 = (tot[0] / (double)n) / volfrac;
        lmid = 0.5 * (l1 + l2);
        done = !((l2 - l1) / (l2 + l1) > 1e-4);
    }
    while (ok && !done && steps < max_steps) {
        // node m of the step tree tries mid[m]; 2 m + 1 follows when l2 moves
        // there, 2 m + 2 when l1 does
        double lo[kOcCand], hi[kOcCand], mid[kOcCand], inv[kOcCand], s[kOcCand];
        lo[0] = l1;
        hi[0] = l2;
#pragma unroll
        for (int m = 0; m < kOcCand; ++m) {
            if (m > 0) {
                const int up = (m - 1) / 2;
                lo[m] = (m & 1) ? lo[up] : mid[up];
                hi[m] = (m & 1) ? mid[up] : hi[up];
            }
            mid[m] = 0.5 * (lo[m] + hi[m]);
            inv[m] = 1.0 / mid[m];
            s[m] = 0.0;
        }
        for (long long i = i0; i < n; i += 2 * st) {   // two elements in flight per thread
            const long long j = i + st;
            const double xi = x[i], oi = ocp[i], xj = j < n ? x[j] : 0.0, oj = j < n ? ocp[j] : 0.0;
            const double top = fmin(xi + move, 1.0), bot = fmax(xi - move, 0.0);
            const double top2 = j < n ? fmin(xj + move, 1.0) : 0.0, bot2 = j < n ? fmax(xj - move, 0.0) : 0.0;
#pragma unroll
            for (int m = 0; m < kOcCand; ++m) {
                s[m] += fmax(fmin(oi * inv[m], top), bot);
                s[m] += fmax(fmin(oj * inv[m], top2), bot2);
            }
        }
        double *part = partial + (size_t)(round & 1) * kOcCand * gridDim.x;   // the slowest CTA may still read the last
        loop_partials<kOcCand>(s, part);
        ok = grid_barrier(sync, ++round, lw);
        loop_totals<kOcCand>(part, tot);
        int m = 0;
#pragma unroll
        for (int k = 0; k < kOcDepth; ++k) {
            if (done || steps >= max_steps) break;
            lmid = 0.5 * (l1 + l2);
            if (tot[m] / (double)n > volfrac) {
                l1 = lmid;
                m = 2 * m + 2;
            } else {
                l2 = lmid;
                m = 2 * m + 1;
            }
            ++steps;
            done = !((l2 - l1) / (l2 + l1) > 1e-4);
        }
    }
    if (ok)
        for (long long i = i0; i < n; i += st)   // x itself when the loop never ran (bracket already tight)
            xnew[i] = steps > 0 ? oc_candidate(x[i], ocp[i], lmid, move) : x[i];
    if (blockIdx.x == 0 && threadIdx.x == 0) *state = OcState{l1, l2, lmid, steps, 1};
    grid_leave(sync, ok, &state->done);
}

int oc_state_bytes() { return (int)sizeof(OcState); }

// ---------------------------------------------------------------------------
// Heaviside projection with the volume-preserving threshold
// (top3D125modCuda.m:60-64 prj/deta/dprj, :111-119 the eta Newton loop):
//   while |mean(prj(xTilde, eta, beta)) - volfrac| > 1e-6:
//       eta -= f / mean(deta(xTilde, eta, beta))
//   xPhys = prj(xTilde, eta, beta),  dprj(xTilde, eta, beta) for the chain rule
// ---------------------------------------------------------------------------
struct ProjState {
    double eta;
    int steps, done;   // done: 1 converged, 0 not within the steps, 2 a grid barrier gave up
};

__device__ __forceinline__ double prj_v(double v, double eta, double beta)
{
    return (tanh(beta * eta) + tanh(beta * (v - eta))) / (tanh(beta * eta) + tanh(beta * (1.0 - eta)));
}

__device__ __forceinline__ double deta_v(double v, double eta, double beta)
{
    const double c = cosh(beta * (v - eta));
    return -beta / sinh(beta) / (c * c) * sinh(v * beta) * sinh((1.0 - v) * beta);
}

__device__ __forceinline__ double dprj_v(double v, double eta, double beta)
{
    const double t = tanh(beta * (v - eta));
    return beta * (1.0 - t * t) / (tanh(beta * eta) + tanh(beta * (1.0 - eta)));
}

// The Newton sums need, per element, t = tanh(beta (v - eta)) and deta, which
// is -beta / sinh(beta) times sech^2 times sinh(v beta) sinh((1 - v) beta).
// Both come from one value per element that does not change between the steps
// (kept in ex), with one division instead of a tanh, a cosh and two sinh:
//  * beta < 2: from V = tanh(beta v), with H = tanh(beta eta), D = tanh(beta)
//    and u = 1 - V H,
//      t = (V - H) / u,  deta = -(beta / D) (1 - H^2) V (D - V) / u^2;
//  * beta from 2 to 300: from E = exp(2 beta v), with a = E exp(-2 beta eta)
//    and q = 1 / (a + 1),
//      t = (a - 1) q,
//      sech^2 sinh sinh = 2 q^2 (a cosh(beta) - (a E exp(-beta) + exp(beta - 2 beta eta)) / 2).
// As beta goes to zero a - 1 loses the bits of t that V - H keeps, and as V and
// H go to one u loses those that a keeps.  The error that each leaves in eta,
// against 80 bits and over that of the direct formulas, is 0.9 to 1.1 for the
// first form from 0.02 to 1.9, and for the second 1.2 at 2, 1.2 to 1.5 (below
// one ulp of eta) from 4 to 300, but 1.5 at 1, 2.4 at 0.5 and 26 at 0.02.
// Other betas, and elements out of the range in which a form is good, take the
// direct formulas.  The design itself is projected with tanh.

// exp(x y) with the rounding of the product made up for: at large exponents it
// is many times that of exp.
__device__ __forceinline__ double exp_product(double x, double y)
{
    const double p = x * y, e = exp(p);
    return fma(e, fma(x, y, -p), e);
}

enum ProjForm { PROJ_TANH, PROJ_EXP, PROJ_DIRECT };

template <int FORM>
__global__ void __launch_bounds__(kLoopThreads, kLoopPerSm)
projection_kernel(long long n, const double *__restrict__ xt, double beta, double volfrac, double eta, double *ex,
                  double *partial, LoopSync *sync, LoopWait lw, int max_steps, ProjState *state, double *__restrict__ xphys,
                  double *__restrict__ dprj)
{
    __shared__ double tot[2];
    const long long i0 = (long long)blockIdx.x * kLoopThreads + threadIdx.x, st = (long long)gridDim.x * kLoopThreads;
    unsigned round = 0;
    bool ok = true, done = false;
    int steps = 0;
    for (int k = 0; k < max_steps && ok && !done; ++k) {
        const double t0 = tanh(beta * eta), den = t0 + tanh(beta * (1.0 - eta));
        const double t1 = FORM == PROJ_TANH ? tanh(beta) : 0.0, c = FORM == PROJ_EXP ? exp_product(-2.0 * beta, eta) : 0.0;
        const double eb = exp(beta), emb = exp(-beta), ch = 0.5 * (eb + emb);
        const double half_ceb = 0.5 * c * eb, half_emb = 0.5 * emb;
        const double kd = FORM == PROJ_TANH ? -(beta / t1) * (1.0 - t0 * t0) : -2.0 * beta / sinh(beta);
        double s[2] = {0.0, 0.0};   // sums of tanh(beta (v - eta)) and of deta
        auto add = [&](long long i, double E) {
            const double a = FORM == PROJ_TANH ? fma(-E, t0, 1.0) : E * c;   // u of the first form
            if (FORM == PROJ_TANH && a > 0.01 && fabs(E) < 1.0) {
                const double q = 1.0 / a;
                s[0] = fma(E - t0, q, s[0]);
                s[1] = fma(kd * (q * q), E * (t1 - E), s[1]);
            } else if (FORM == PROJ_EXP && E > 1e-150 && E < 1e150 && a < 1e150) {
                const double q = 1.0 / (a + 1.0);
                s[0] = fma(a - 1.0, q, s[0]);
                s[1] = fma(kd * (q * q), fma(a, ch, -fma(a * E, half_emb, half_ceb)), s[1]);
            } else {
                s[0] += tanh(beta * (xt[i] - eta));
                s[1] += deta_v(xt[i], eta, beta);
            }
        };
        auto once = [&](double v) {
            return FORM == PROJ_TANH ? tanh(beta * v) : FORM == PROJ_EXP ? exp_product(2.0 * beta, v) : 0.0;
        };
        // two elements in flight per thread
        for (long long i = i0; i < n; i += 2 * st) {
            const long long j = i + st;
            const bool two = j < n;
            double E, F = 0.0;
            if (k == 0) {
                const double u = xt[i], v = two ? xt[j] : 0.0;
                E = once(u);
                F = once(v);
                ex[i] = E;
                if (two) ex[j] = F;
            } else {
                E = ex[i];
                if (two) F = ex[j];
            }
            add(i, E);
            if (two) add(j, F);
        }
        double *part = partial + (size_t)(round & 1) * 2 * gridDim.x;
        loop_partials<2>(s, part);
        ok = grid_barrier(sync, ++round, lw);
        loop_totals<2>(part, tot);
        const double f = (t0 + tot[0] / (double)n) / den - volfrac;   // mean(prj) - volfrac
        if (fabs(f) > 1e-6) {
            eta = eta - f / (tot[1] / (double)n);
            ++steps;
        } else {
            done = true;
        }
        __syncthreads();   // tot is rewritten by the next step
    }
    if (ok) {
        for (long long i = i0; i < n; i += st) {
            xphys[i] = prj_v(xt[i], eta, beta);
            if (dprj) dprj[i] = dprj_v(xt[i], eta, beta);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *state = ProjState{eta, steps, done ? 1 : 0};
    grid_leave(sync, ok, &state->done);
}

int proj_state_bytes() { return (int)sizeof(ProjState); }

// CTAs of a looping launch: at most two per SM, at least four elements per
// thread, and never more than fit the device at once (the cooperative launch
// refuses that).
static int loop_blocks(long long n)
{
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long want = (n + 4 * kLoopThreads - 1) / (4 * kLoopThreads);
    return (int)std::max(1LL, std::min<long long>({want, (long long)kLoopPerSm * sms, kLoopMaxBlocks}));
}

int launch_heaviside(long long n, const double *xt, double volfrac, double beta, double eta0, double *xphys,
                     double *dprj, double *ex, double *partial, void *sync, void *state, int max_steps,
                     cudaStream_t st)
{
    ProjState *ps = (ProjState *)state;
    LoopSync *ls = (LoopSync *)sync;
    LoopWait lw = loop_wait();
    void *args[] = {&n, &xt, &beta, &volfrac, &eta0, &ex, &partial, &ls, &lw, &max_steps, &ps, &xphys, &dprj};
    const void *kernel = beta < 2.0      ? (const void *)projection_kernel<PROJ_TANH>
                         : beta <= 300.0 ? (const void *)projection_kernel<PROJ_EXP>
                                         : (const void *)projection_kernel<PROJ_DIRECT>;
    GPUTO_CUDA(cudaLaunchCooperativeKernel(kernel, dim3((unsigned)loop_blocks(n)),
                                           dim3(kLoopThreads), args, 0, st));
    count_launches(1);
    return GPUTO_OK;
}

__global__ void mul_kernel(long long n, const double *__restrict__ a, const double *__restrict__ b,
                           double *__restrict__ out)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        out[i] = a[i] * b[i];
}

void launch_mul(long long n, const double *a, const double *b, double *out, cudaStream_t st)
{
    long long nb = (n + 255) / 256;
    if (nb > 4096) nb = 4096;
    mul_kernel<<<(unsigned)nb, 256, 0, st>>>(n, a, b, out);
    count_launches(1);
}

int launch_oc_update(long long n, const double *x, const double *dc, const double *dv0, double volfrac, double move,
                     double *ocp, double *xnew, double *partial, void *sync, void *state, int max_steps,
                     cudaStream_t st)
{
    OcState *os = (OcState *)state;
    LoopSync *ls = (LoopSync *)sync;
    LoopWait lw = loop_wait();
    void *args[] = {&n, &x, &dc, &dv0, &ocp, &move, &volfrac, &xnew, &partial, &ls, &lw, &max_steps, &os};
    GPUTO_CUDA(cudaLaunchCooperativeKernel((const void *)oc_update_kernel, dim3((unsigned)loop_blocks(n)),
                                           dim3(kLoopThreads), args, 0, st));
    count_launches(1);
    return GPUTO_OK;
}

}  // namespace gputo
