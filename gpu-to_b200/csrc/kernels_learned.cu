// The learned coarse-grid correction network: forward, backward and Adam
// kernels, written for this project (the reference has no learned part).
//
// Network (level-2 node grid, channels-first [C][X][Z][Y], Y fastest as in
// the solver's node order): three 3x3x3 convolutions 4 -> 16 -> 32 -> 64 with
// bias and ReLU, zero padding, then a 1x1x1 convolution 64 -> 3.  Weights are
// kept in FP32 for training and used rounded to BF16; activations and sums are
// FP32.  Flat parameter layout per layer: w[co][ci][tap] then b[co], tap =
// 9 (dx+1) + 3 (dz+1) + (dy+1).
//
// The 16 -> 32 and 32 -> 64 convolutions and their data gradients are implicit
// GEMMs on the 5th-generation tensor cores (conv_tc_kernel); so are their
// weight gradients (wgrad_tc_kernel); the first layer and the 1x1x1 head run on
// the CUDA cores.
//
// Activations and gradients between the layers are stored as "split rows":
//  * a grid node is row r = guard + ((s (X + 1) + x) (Z + 1) + z) (Y + 1) + y;
//    one zero row after each y line, one zero line after each z plane, one
//    zero plane after each sample and `guard` zero rows in front and behind
//    stand in for the zero padding, so every tap of every node is a fixed row
//    offset and needs no test;
//  * each FP32 value is the exact sum of three BF16 parts (hi, mid, lo: the 24
//    significand bits, split by truncation), kept in planes
//    [part][channel / 8][row][8]: 16 bytes per row, the K-major operand rows
//    of the tensor cores, which a bulk copy brings in as they are and whose
//    shift by a row is a shift of the operand's address by 16 bytes.
// Products of the parts with the BF16 weights are exact in FP32, so three
// BF16 MMAs give the FP32 convolution up to the order of its sums.  Weight
// gradients are reduced in a fixed order, so training is deterministic.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "gputo_internal.h"
#include "tma.h"

namespace gputo {

namespace {

__host__ __device__ constexpr int net_ch(int l) { return l == 0 ? 4 : l == 1 ? 16 : l == 2 ? 32 : l == 3 ? 64 : 3; }
__host__ __device__ constexpr int net_k(int l) { return l == 3 ? 1 : 3; }

__device__ __forceinline__ float bf16r(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

constexpr int kRows = 128;                       // rows of one tile (TMEM lanes)
constexpr uint32_t kNetWaitNs = 2000000000u;     // bounded waits give up after 2 s

// Eight FP32 values -> their three BF16 parts, eight per 16-byte row entry
// (the same truncating split as kernels_tc.cu's).
__device__ __forceinline__ void split8(const float (&v)[8], uint4 (&o)[3])
{
    uint32_t w[3][4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uint32_t a[3], b[3];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const float x = v[2 * q + e];
            const uint32_t b0 = __float_as_uint(x);
            // an infinity stays one: its remainder would be a NaN
            const float r1 = (b0 & 0x7F800000u) == 0x7F800000u ? 0.f : x - __uint_as_float(b0 & 0xFFFF0000u);
            const uint32_t b1 = __float_as_uint(r1);
            const float r2 = r1 - __uint_as_float(b1 & 0xFFFF0000u);
            uint32_t *t = e ? b : a;
            t[0] = b0;
            t[1] = b1;
            t[2] = __float_as_uint(r2);
        }
#pragma unroll
        for (int p = 0; p < 3; ++p) w[p][q] = __byte_perm(a[p], b[p], 0x7632);
    }
#pragma unroll
    for (int p = 0; p < 3; ++p) o[p] = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
}

__device__ __forceinline__ void add_part(float (&v)[8], const uint4 &u)
{
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        v[2 * q] += __uint_as_float(w[q] << 16);
        v[2 * q + 1] += __uint_as_float(w[q] & 0xFFFF0000u);
    }
}

// Geometry of the split rows of S samples.
struct RowGeo {
    int X, Z, Y, S;
    int py, pz;            // row offsets of dz = 1 and dx = 1
    long long rows;        // S (X + 1) (Z + 1) (Y + 1)
    long long guard, R;    // zero rows in front; rows of a plane (a whole number of tiles, guards included)
    int ntiles;
};

RowGeo row_geo(const NetDims &d, int S)
{
    RowGeo q;
    q.X = d.X, q.Z = d.Z, q.Y = d.Y, q.S = S;
    q.py = d.Y + 1;
    q.pz = (d.Z + 1) * (d.Y + 1);
    q.rows = (long long)S * (d.X + 1) * q.pz;
    q.guard = ((long long)q.pz + q.py + 1 + 7) / 8 * 8;
    q.ntiles = (int)((q.rows + kRows - 1) / kRows);
    q.R = 2 * q.guard + (long long)q.ntiles * kRows;
    return q;
}

// Row r (without the guard) -> sample, node; false on padding rows.  In 32
// bits: 2^31 rows of the first layer alone (96 bytes each) would be 206 GB.
__device__ __forceinline__ bool row_node(const RowGeo &q, long long r, int &s, int &x, int &z, int &y)
{
    const uint32_t r32 = (uint32_t)r, line = r32 / (uint32_t)q.py, plane = line / (uint32_t)(q.Z + 1);
    y = (int)(r32 - line * q.py);
    z = (int)(line - plane * (q.Z + 1));
    s = (int)(plane / (uint32_t)(q.X + 1));
    x = (int)(plane - (uint32_t)s * (q.X + 1));
    return s < q.S && x < q.X && z < q.Z && y < q.Y;
}

// Zeroes the guard rows of up to five sets of planes.
struct GuardSets {
    uint4 *p[5];
    int planes[5];
};

__global__ void __launch_bounds__(256) zero_guards_kernel(GuardSets g, RowGeo q)
{
    uint4 *p = g.p[blockIdx.y];
    const long long n = 2 * q.guard * g.planes[blockIdx.y];
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
        const long long pl = i / (2 * q.guard), k = i - pl * 2 * q.guard;
        p[pl * q.R + (k < q.guard ? k : q.R - 2 * q.guard + k)] = make_uint4(0u, 0u, 0u, 0u);
    }
}

// The BF16 weight operands of the four tensor-core convolutions, as the
// shared-memory image [tap][K / 8][N][8] that a CTA copies whole:
//   forward l: K = ci, N = co; data gradient l: K = co, N = ci, tap mirrored.
constexpr int kImg2 = 27 * 16 * 32, kImg3 = 27 * 32 * 64;   // elements

__global__ void __launch_bounds__(256)
pack_weights_kernel(const float *__restrict__ w2, const float *__restrict__ w3, __nv_bfloat16 *__restrict__ img)
{
    int i = blockIdx.x * 256 + threadIdx.x;   // images: forward 2, forward 3, data 3, data 2
    if (i >= 2 * (kImg2 + kImg3)) return;
    const int out = i;
    int l = 2, back = 0;
    if (i >= kImg2) {
        i -= kImg2;
        l = 3;
        if (i >= kImg3) {
            i -= kImg3;
            back = 1;
            if (i >= kImg3) {
                i -= kImg3;
                l = 2;
            }
        }
    }
    const int ci_n = l == 2 ? 16 : 32, co_n = l == 2 ? 32 : 64;
    const int K = back ? co_n : ci_n, N = back ? ci_n : co_n;
    const int e = i & 7, n = (i >> 3) % N, rest = (i >> 3) / N, kc = rest % (K / 8), t = rest / (K / 8);
    const int k = 8 * kc + e;
    const int co = back ? k : n, ci = back ? n : k, tap = back ? 26 - t : t;
    const float *w = l == 2 ? w2 : w3;
    img[out] = __float2bfloat16_rn(w[(co * ci_n + ci) * 27 + tap]);
}

// Layer 1 (4 -> 16): the 108 taps from the caller's dense input, weights
// broadcast from shared memory, output pairs on paired FP32 instructions;
// writes the split rows of its 16 channels (zeros on padding).  4 x 27 x 16
// FMAs per node are too few channels for the tensor cores.  A thread takes
// kC1R rows a CTA width apart, which share each weight read: with one row the
// kernel was bound by those reads (94 us at 129 x 65 x 65, 66 with two); four
// rows take too many registers and leave too few warps (72 us).  The taps are
// summed in blocks of nine: a chain of 108 roundings was half of the network's
// error, and an activation whose sum is within that error of zero changes sign
// and with it a term of the gradients.  For 10 us more the training gradients'
// error against 64 bits falls from 8.7e-7 to 3.2e-7 (geometric mean over twelve
// sets of eight 33^3 samples; 1.6e-6 as FP32 FMA chains throughout).
constexpr int kC1R = 2;

__global__ void __launch_bounds__(128)
conv1_kernel(const float *__restrict__ xin, const float *__restrict__ w, const float *__restrict__ b,
             uint4 *__restrict__ out, RowGeo q)
{
    __shared__ __align__(16) float ws[4 * 27 * 16];
    __shared__ float bs[16];
    for (int i = threadIdx.x; i < 4 * 27 * 16; i += 128) {
        const int c = i & 15, t = i >> 4;   // t = ci 27 + tap
        ws[i] = bf16r(w[c * 108 + t]);
    }
    if (threadIdx.x < 16) bs[threadIdx.x] = b[threadIdx.x];
    __syncthreads();
    const long long r0 = (long long)blockIdx.x * (128 * kC1R) + threadIdx.x, nr = (long long)q.ntiles * kRows;
    const int N = q.X * q.Z * q.Y;
    const float *xs[kC1R];
    unsigned ok[kC1R];   // bits 0-8: the (dx, dz) line is inside, 9 and 10: y - 1 and y + 1 are; 0 on padding
    float2 acc[kC1R][8];
#pragma unroll
    for (int k = 0; k < kC1R; ++k) {
        int s, x, z, y;
        const bool in = row_node(q, r0 + 128 * k, s, x, z, y);
        xs[k] = in ? xin + (size_t)s * 4 * N + ((size_t)x * q.Z + z) * q.Y + y : xin;
        ok[k] = 0;
        if (in) {
#pragma unroll
            for (int g = 0; g < 9; ++g)
                if ((unsigned)(x + g / 3 - 1) < (unsigned)q.X && (unsigned)(z + g % 3 - 1) < (unsigned)q.Z) ok[k] |= 1u << g;
            ok[k] |= (y > 0 ? 1u << 9 : 0u) | (y < q.Y - 1 ? 1u << 10 : 0u);
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[k][c] = make_float2(bs[2 * c], bs[2 * c + 1]);
    }
#pragma unroll 1
    for (int ci = 0; ci < 4; ++ci)
#pragma unroll 1
        for (int dx = 0; dx < 3; ++dx) {
            float v[kC1R][9];
#pragma unroll
            for (int k = 0; k < kC1R; ++k)
#pragma unroll
                for (int dz = 0; dz < 3; ++dz) {
                    const bool in = (ok[k] >> (3 * dx + dz)) & 1u;
                    const float *p = xs[k] + (size_t)ci * N + (ptrdiff_t)((dx - 1) * q.Z + dz - 1) * q.Y;
                    v[k][3 * dz] = in && (ok[k] & (1u << 9)) ? p[-1] : 0.f;
                    v[k][3 * dz + 1] = in ? p[0] : 0.f;
                    v[k][3 * dz + 2] = in && (ok[k] & (1u << 10)) ? p[1] : 0.f;
                }
            const float4 *wr = reinterpret_cast<const float4 *>(ws + (ci * 27 + 9 * dx) * 16);
            float2 blk[kC1R][8];   // sums of nine taps
#pragma unroll
            for (int k = 0; k < kC1R; ++k)
#pragma unroll
                for (int c = 0; c < 8; ++c) blk[k][c] = make_float2(0.f, 0.f);
#pragma unroll
            for (int t = 0; t < 9; ++t)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float4 m = wr[4 * t + c];
#pragma unroll
                    for (int k = 0; k < kC1R; ++k) {
                        const float2 vv = make_float2(v[k][t], v[k][t]);
                        blk[k][2 * c] = __ffma2_rn(make_float2(m.x, m.y), vv, blk[k][2 * c]);
                        blk[k][2 * c + 1] = __ffma2_rn(make_float2(m.z, m.w), vv, blk[k][2 * c + 1]);
                    }
                }
#pragma unroll
            for (int k = 0; k < kC1R; ++k)
#pragma unroll
                for (int c = 0; c < 8; ++c) acc[k][c] = __fadd2_rn(acc[k][c], blk[k][c]);
        }
#pragma unroll
    for (int k = 0; k < kC1R; ++k) {
        const long long r = r0 + 128 * k;
        if (r >= nr) break;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            float v[8];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                v[2 * e] = ok[k] ? fmaxf(acc[k][4 * c + e].x, 0.f) : 0.f;
                v[2 * e + 1] = ok[k] ? fmaxf(acc[k][4 * c + e].y, 0.f) : 0.f;
            }
            uint4 o[3];
            split8(v, o);
#pragma unroll
            for (int p = 0; p < 3; ++p) out[(size_t)(p * 2 + c) * q.R + q.guard + r] = o[p];
        }
    }
}

// What conv_tc_kernel does with a finished row of N sums.
enum ConvEpi {
    EPI_RELU = 0,   // + bias, ReLU -> split rows
    EPI_HEAD = 1,   // + bias, ReLU (stored in FP32 when training), then the 64 -> 3 head -> dense output
    EPI_MASK = 2    // data gradient: zero where the layer's activation is -> split rows
};

struct ConvArgs {
    const uint4 *a;          // input split rows, 3 K / 8 planes
    const uint4 *img;        // weight operand image
    const float *bias;
    uint4 *out;              // split rows, 3 N / 8 planes
    const uint4 *mask;       // EPI_MASK: the activation's split rows (its hi planes decide)
    const float *w4, *b4;    // EPI_HEAD
    float *y, *act;          // EPI_HEAD: dense output [S][3][n]; FP32 rows [N / 8][rows of the tiles][8] or null
    int *err;                // set when a bounded wait gives up
};

// One convolution as an implicit GEMM: D[row][N] = sum over 27 taps, K input
// channels and 3 parts.  Per tile of 128 rows and (dx, dz) pair ("segment"),
// 130 rows of every plane are brought in by bulk copies; the three dy taps are
// the same rows shifted by one, i.e. operand addresses 16 bytes apart.
//
// Warp 4's first thread issues the copies, warp 5's first thread the MMAs,
// warps 0-3 add the segment sums from TMEM (double-buffered) into FP32
// registers and run the epilogue.  The tensor core's adds truncate, which
// shrinks every sum a little, and gradients add that up over all nodes.  So a
// segment has four accumulators, the hi parts of each dy and the mid and lo
// parts of all: products of hi parts and weights have 16 bits, few of which
// are lost in the K / 16 adds of a chain, and the four sums are added with
// rounding.  With one accumulator per segment the output is low by 1.2e-7 and
// small grids' gradients are off by 4.3e-7; now 3e-8 and 1.5e-7, no more than
// with FP32 FMA chains (outputs 2.7e-7 against 6.3e-7, relative to the norm),
// for 10 % of the forward pass.
//
// Persistent, weights resident (110 KB for 32 x 64).  Copies, MMAs and drains
// overlap but share the shared memory and TMEM ports, and none of them alone
// is the bound: a forward pass at 129 x 65 x 65 takes 465 us, 384 with a third
// of the MMAs, 399 without drains and epilogue, 303 without both, which is the
// nine reads of the activations (978 MB at about 6.5 TB/s).  Measured at 129 x 65 x 65: 32 -> 64
// with the head 280 us (0.8 PFLOP/s of BF16 MMAs; 3167 + 50 us as direct FP32
// convolutions on the CUDA cores), 16 -> 32 115 us (733 us); data gradients of
// eight 33^3 samples 232 and 91 us (2988 and 784 us).
template <int CK, int CN> struct ConvCfg {
    static constexpr int C8 = CK / 8;
    static constexpr int RS = kRows + 2;                    // rows of a segment
    static constexpr int STAGE = 3 * C8 * RS * 16;          // bytes
    static constexpr int BBYTES = 27 * CK * CN * 2;
    // three stages let two CTAs of 32 -> 16 share an SM (91 us; 132 us with four)
    static constexpr int NST = CK == 64 ? 2 : CN == 16 ? 3 : 4;
    static constexpr int COLS = 8 * CN;                     // TMEM columns (a power of two): 2 x 4 accumulators
    static constexpr int BARS = BBYTES + NST * STAGE;
    static constexpr size_t SMEM = BARS + 8 * (2 * NST + 5) + 16 + 200 * 4;
    static_assert(BBYTES % 128 == 0 && STAGE % 16 == 0 && BARS % 16 == 0, "bulk copies need 16-byte alignment");
    static_assert(SMEM <= 227 * 1024, "shared memory of one CTA");
};

__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tc_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// K-major BF16 operand without swizzle: 8 rows x 16 bytes contiguous, the
// next 8 rows 128 bytes on (SBO), the next 8 channels lbo bytes on (LBO).
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr, uint32_t lbo, uint32_t sbo = 128)
{
    return ((uint64_t)(addr >> 4) & 0x3FFFull) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46);
}

__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
        : "memory");
}

__device__ __forceinline__ void tc_load16(uint32_t addr, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr)
        : "memory");
}

// The registers of earlier TMEM loads may be read from here on (they pass
// through, so that no use moves ahead of the wait).
__device__ __forceinline__ void tc_wait_loads(uint32_t (&r)[16])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
}

template <int CK, int CN, int EPI>
__global__ void __launch_bounds__(192) conv_tc_kernel(ConvArgs A, RowGeo q)
{
    using C = ConvCfg<CK, CN>;
    extern __shared__ __align__(128) unsigned char sm[];
    unsigned char *sB = sm, *sA = sm + C::BBYTES;
    uint64_t *full = reinterpret_cast<uint64_t *>(sm + C::BARS), *empty = full + C::NST, *tfull = empty + C::NST,
             *tempty = tfull + 2, *bbar = tempty + 2;
    uint32_t *tbase = reinterpret_cast<uint32_t *>(bbar + 1);
    float *hw = reinterpret_cast<float *>(tbase + 4);   // head weights [64][3] and bias
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tbase)),
                     "r"(C::COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 128) {
        for (int s = 0; s < C::NST; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&tfull[s], 1);
            mbar_init(&tempty[s], 128);
        }
        mbar_init(bbar, 1);
        fence_barrier_init();
    }
    if (EPI == EPI_HEAD)
        for (int i = tid; i < 195; i += 192) hw[i] = i < 192 ? bf16r(A.w4[(i % 3) * 64 + i / 3]) : A.b4[i - 192];
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tbase;
    bool bad = false;
    auto wait = [&](uint64_t *b, uint32_t parity) {
        if (!bad && !mbar_wait_for(b, parity, kNetWaitNs)) {
            bad = true;
            if (A.err) *(volatile int *)A.err = GPUTO_ERR_TIMEOUT;
        }
    };
    if (warp == 4) {
        if (lane == 0) {
            mbar_arrive_expect_tx(bbar, C::BBYTES);
            bulk_load(sB, A.img, C::BBYTES, bbar);
            int it = 0, issued = 0;
            for (int tile = blockIdx.x; tile < q.ntiles && !bad; tile += gridDim.x)
                for (int seg = 0; seg < 9; ++seg, ++it) {
                    const int s = it % C::NST;
                    if (it >= C::NST) wait(&empty[s], (uint32_t)((it / C::NST - 1) & 1));
                    if (bad) break;
                    const long long row =
                        q.guard + (long long)tile * kRows + (long long)(seg / 3 - 1) * q.pz + (seg % 3 - 1) * q.py - 1;
                    mbar_arrive_expect_tx(&full[s], C::STAGE);
                    unsigned char *dst = sA + s * C::STAGE;
                    for (int pl = 0; pl < 3 * C::C8; ++pl)
                        bulk_load(dst + pl * (C::RS * 16), A.a + pl * q.R + row, C::RS * 16, &full[s]);
                    ++issued;
                }
            // copies in flight land before the CTA leaves (they already have unless a wait gave up)
            if (bad) {
                mbar_wait_for(bbar, 0, kNetWaitNs);
                for (int k = issued > C::NST ? issued - C::NST : 0; k < issued; ++k)
                    mbar_wait_for(&full[k % C::NST], (uint32_t)((k / C::NST) & 1), kNetWaitNs);
            }
        }
    } else if (warp == 5) {
        if (lane == 0) {
            constexpr uint32_t idesc =
                (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(CN >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);
            const uint32_t b0 = smem_u32(sB), a0 = smem_u32(sA);
            wait(bbar, 0);
            const int mine = 9 * ((q.ntiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x);
            int it = 0;
            for (int tile = blockIdx.x; tile < q.ntiles && !bad; tile += gridDim.x)
                for (int seg = 0; seg < 9; ++seg, ++it) {
                    const int s = it % C::NST, tb = it & 1;
                    wait(&full[s], (uint32_t)((it / C::NST) & 1));
                    if (it >= 2) wait(&tempty[tb], (uint32_t)((it / 2 - 1) & 1));
                    if (bad) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t d = tmem + (uint32_t)(tb * 4 * CN);
#pragma unroll
                    for (int part = 2; part >= 0; --part)
#pragma unroll
                        for (int dy = 0; dy < 3; ++dy)
#pragma unroll
                            for (int ks = 0; ks < CK / 16; ++ks) {
                                const uint64_t da = tc_desc(
                                    a0 + s * C::STAGE + ((part * C::C8 + 2 * ks) * C::RS + dy) * 16, C::RS * 16);
                                const uint64_t db =
                                    tc_desc(b0 + ((3 * seg + dy) * C::C8 + 2 * ks) * CN * 16, CN * 16);
                                const bool first = ks == 0 && (part == 0 || (part == 2 && dy == 0));
                                tc_mma(d + (part ? 3 : dy) * CN, da, db, idesc, first ? 0u : 1u);
                            }
                    // only where the producer waits for it: no arrival is left under way at the end
                    if (it + C::NST < mine) tc_commit(&empty[s]);
                    tc_commit(&tfull[tb]);
                }
            // MMAs in flight end before TMEM is freed
            if (bad && it > 0) mbar_wait_for(&tfull[(it - 1) & 1], (uint32_t)(((it - 1) / 2) & 1), kNetWaitNs);
        }
    } else {
        const uint32_t lane_off = (uint32_t)(warp * 32) << 16;
        int it = 0;
        for (int tile = blockIdx.x; tile < q.ntiles && !bad; tile += gridDim.x) {
            float acc[CN];
#pragma unroll
            for (int c = 0; c < CN; ++c) acc[c] = 0.f;
            for (int seg = 0; seg < 9; ++seg, ++it) {
                const int tb = it & 1;
                wait(&tfull[tb], (uint32_t)((it / 2) & 1));
                if (__any_sync(0xffffffffu, bad)) {   // the TMEM loads are warp-wide
                    bad = true;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int c0 = 0; c0 < CN; c0 += 16) {
                    uint32_t r[4][16];
#pragma unroll
                    for (int p = 0; p < 4; ++p) tc_load16(tmem + lane_off + (uint32_t)((4 * tb + p) * CN + c0), r[p]);
#pragma unroll
                    for (int p = 0; p < 4; ++p) tc_wait_loads(r[p]);
#pragma unroll
                    for (int c = 0; c < 16; ++c)
                        acc[c0 + c] += (__uint_as_float(r[0][c]) + __uint_as_float(r[1][c])) +
                                       (__uint_as_float(r[2][c]) + __uint_as_float(r[3][c]));
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&tempty[tb])) : "memory");
            }
            if (bad) break;
            const long long r = (long long)tile * kRows + warp * 32 + lane;
            int s, x, z, y;
            const bool in = row_node(q, r, s, x, z, y);
            if (EPI == EPI_HEAD) {
                float o3[3] = {hw[192], hw[193], hw[194]};
#pragma unroll
                for (int c = 0; c < CN; ++c) {
                    acc[c] = in ? fmaxf(acc[c] + A.bias[c], 0.f) : 0.f;
#pragma unroll
                    for (int o = 0; o < 3; ++o) o3[o] = fmaf(hw[3 * c + o], acc[c], o3[o]);
                }
                if (in) {
                    const long long n = (long long)q.X * q.Z * q.Y, at = ((long long)x * q.Z + z) * q.Y + y;
#pragma unroll
                    for (int o = 0; o < 3; ++o) A.y[(3LL * s + o) * n + at] = o3[o];
                }
                if (A.act) {
                    float4 *dst = reinterpret_cast<float4 *>(A.act);
                    const size_t nr = (size_t)q.ntiles * kRows;
#pragma unroll
                    for (int c = 0; c < CN / 8; ++c)
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            dst[2 * (c * nr + r) + h] = make_float4(acc[8 * c + 4 * h], acc[8 * c + 4 * h + 1],
                                                                    acc[8 * c + 4 * h + 2], acc[8 * c + 4 * h + 3]);
                }
            } else {
#pragma unroll
                for (int c = 0; c < CN / 8; ++c) {
                    float v[8];
                    if (EPI == EPI_RELU) {
#pragma unroll
                        for (int e = 0; e < 8; ++e) v[e] = in ? fmaxf(acc[8 * c + e] + A.bias[8 * c + e], 0.f) : 0.f;
                    } else {
                        const uint4 m = A.mask[(size_t)c * q.R + q.guard + r];
                        const uint32_t mw[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            v[e] = in && ((e & 1) ? (mw[e >> 1] >> 16) : (mw[e >> 1] & 0xFFFFu)) ? acc[8 * c + e] : 0.f;
                    }
                    uint4 o[3];
                    split8(v, o);
#pragma unroll
                    for (int p = 0; p < 3; ++p) A.out[(size_t)(p * (CN / 8) + c) * q.R + q.guard + r] = o[p];
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::COLS) : "memory");
}

// Backward through the head and layer 3's ReLU: from the output gradient gy
// (dense [S][3][n]) and the FP32 activations, the split rows of layer 3's
// gradient, g3 = [act > 0] w4' gy, and the CTA's partial sums of the head's
// weight and bias gradients, part[CTA][195] (co 64 + ci, then co).
constexpr int kHeadPart = 195;

__global__ void __launch_bounds__(256)
head_backward_kernel(const float *__restrict__ gy, const float *__restrict__ act, const float *__restrict__ w4,
                     uint4 *__restrict__ g3, float *__restrict__ part, RowGeo q)
{
    __shared__ float as[kRows][65], gs[kRows][4], hw[192];
    const int tid = threadIdx.x;
    if (tid < 192) hw[tid] = bf16r(w4[tid]);
    const long long n = (long long)q.X * q.Z * q.Y;
    const size_t nr = (size_t)q.ntiles * kRows;
    float sum = 0.f;
    for (int tile = blockIdx.x; tile < q.ntiles; tile += gridDim.x) {
        __syncthreads();
        if (tid < kRows) {
            int s, x, z, y;
            const bool in = row_node(q, (long long)tile * kRows + tid, s, x, z, y);
            const long long at = ((long long)x * q.Z + z) * q.Y + y;
#pragma unroll
            for (int o = 0; o < 3; ++o) gs[tid][o] = in ? gy[(3LL * s + o) * n + at] : 0.f;
        }
        __syncthreads();
        for (int i = tid; i < 8 * kRows; i += 256) {   // (chunk, row)
            const int c = i / kRows, rr = i - c * kRows;
            const size_t r = (size_t)tile * kRows + rr;
            const float4 *src = reinterpret_cast<const float4 *>(act) + 2 * (c * nr + r);
            const float4 lo = src[0], hi = src[1];
            const float a[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                as[rr][8 * c + e] = a[e];
                float g = hw[8 * c + e] * gs[rr][0];
                g = fmaf(hw[64 + 8 * c + e], gs[rr][1], g);
                g = fmaf(hw[128 + 8 * c + e], gs[rr][2], g);
                v[e] = a[e] > 0.f ? g : 0.f;
            }
            uint4 o[3];
            split8(v, o);
#pragma unroll
            for (int p = 0; p < 3; ++p) g3[(size_t)(p * 8 + c) * q.R + q.guard + r] = o[p];
        }
        __syncthreads();
        if (tid < 192) {
            const int co = tid >> 6, ci = tid & 63;
#pragma unroll 8
            for (int rr = 0; rr < kRows; ++rr) sum = fmaf(gs[rr][co], as[rr][ci], sum);
        } else if (tid < kHeadPart) {
            for (int rr = 0; rr < kRows; ++rr) sum += gs[rr][tid - 192];
        }
    }
    if (tid < kHeadPart) part[(size_t)blockIdx.x * kHeadPart + tid] = sum;
}

// Weight gradients gw[co][ci][tap] = sum over rows of g[row][co]
// x[row + offset(tap)][ci] and bias gradients of layers 2 and 3, as GEMMs over
// the rows: A = g' (M = output channels), B = x (N = input channels), both
// M- / N-major, straight from the split rows.  A tap's shift by dy is again an
// operand address 16 bytes on.  A CTA takes a range of 128-row tiles and SEG
// of the nine (dx, dz) pairs, i.e. 3 SEG taps with a TMEM accumulator each.
//
// Both operands have three parts.  16 x 32: M holds all parts of g (96 of 128
// lanes), N all parts of x: the nine products in one MMA.  32 x 64: M = 128
// is (hi, mid) of g against all of x, and a second MMA adds (mid, lo) x hi to
// the columns of x's lo part, where its upper half, lo x hi, belongs; its
// lower half is the mid x hi that the first one left in the upper lanes of x's
// hi columns, which are not read.  Left out are lo x mid and lo x lo, below
// 2^-23 of a product.  A plane of ones in front of the last pair's rows gives
// the bias gradients: the first group of CTAs takes its last tap 16 columns
// wider, 8 of ones in front and 8 behind that are not read.
//
// Every kWgChunk tiles (256 rows) the accumulators are added into FP32
// registers, so that the tensor core's truncating adds stay 16 long (with 32
// the relative error against 64 bits is 1.3 times as large, for 1 % of the time);
// a tap is drained while the others' MMAs run.  Per CTA the sums over a range go to
// part[range and lane group][tap][ci][co], added in order by sum_parts_kernel.
//
// Bound by the MMAs: the tensor unit is 71 % busy, at 38 % of its BF16 rate,
// with 4 KB of A to read for 32 to 96 columns.  A CTA keeps only three (nine) taps, since 512 columns
// hold no more of them for 32 x 64 and the copies of g would grow.  Eight 33^3
// samples: 368 and 178 us for layers 3 and 2; 892 and 290 us as FP32 FMAs on
// the CUDA cores (53 % of their rate), 7.0 ms with a CTA per (co, ci) pair.
constexpr int kWgChunk = 2;   // tiles per accumulation in TMEM

template <int CO, int CI> struct WgCfg {
    static constexpr int GP = 3 * CO / 8, XP = 3 * CI / 8;   // planes
    static constexpr int SEG = CO == 64 ? 1 : 3, T = 3 * SEG, GROUPS = 9 / SEG;
    static constexpr int SUBS = CO == 64 ? 2 : 3;            // lane groups with sums of their own
    static constexpr int XR = kRows + 2;
    static constexpr int GBYTES = GP * kRows * 16, SEGBYTES = XP * XR * 16, ONES = XR * 16;
    static constexpr int STAGE = GBYTES + SEG * SEGBYTES + ONES, COPIED = GBYTES + SEG * SEGBYTES;
    static constexpr int NST = 3;
    static constexpr int N = 3 * CI;
    static constexpr int COLS = 512;
    static constexpr int BIAS2 = T * N + 32;                 // columns of lo's bias sums (32 x 64)
    static constexpr int BARS = NST * STAGE;
    // the unused last 8 columns of the widened operand read up to a plane past the last stage
    static constexpr size_t SMEM = BARS + XR * 16 + 16;
    static_assert(8 * (2 * NST + 2 * T + 1) + 8 <= XR * 16, "barriers");
    static_assert(BIAS2 + 16 <= COLS && N % 16 == 0, "accumulators");
    static_assert(CO == 64 || GBYTES + 4 * kRows * 16 <= STAGE, "A's unused planes lie within the stage");
    static_assert(STAGE % 16 == 0 && BARS % 16 == 0 && SMEM <= 227 * 1024, "shared memory of one CTA");
    // the rows of pair s within a stage; the plane of ones is in front of the last
    __host__ __device__ static constexpr int xoff(int s) { return GBYTES + s * SEGBYTES + (s == SEG - 1 ? ONES : 0); }
    __host__ __device__ static constexpr int dcol(int t) { return t * N + (t == T - 1 ? 16 : 0); }
};

template <int CO, int CI>
__global__ void __launch_bounds__(192)
wgrad_tc_kernel(const uint4 *__restrict__ g, const uint4 *__restrict__ x, float *__restrict__ part,
                float *__restrict__ bpart, RowGeo q, int tiles_per, int *err)
{
    using C = WgCfg<CO, CI>;
    constexpr int T = C::T;
    extern __shared__ __align__(128) unsigned char sm[];
    uint64_t *full = reinterpret_cast<uint64_t *>(sm + C::BARS), *empty = full + C::NST, *tfull = empty + C::NST,
             *tempty = tfull + T, *fin = tempty + T;
    uint32_t *tbase = reinterpret_cast<uint32_t *>(fin + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tbase)),
                     "r"(C::COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 128) {
        for (int s = 0; s < C::NST; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int t = 0; t < T; ++t) {
            mbar_init(&tfull[t], 1);
            mbar_init(&tempty[t], 128);
        }
        mbar_init(fin, 1);
        fence_barrier_init();
    }
    for (int i = tid; i < C::NST * (C::ONES / 16); i += 192) {
        const int s = i / (C::ONES / 16), k = i - s * (C::ONES / 16);
        reinterpret_cast<uint4 *>(sm + s * C::STAGE + C::xoff(C::SEG - 1) - C::ONES)[k] =
            make_uint4(0x3F803F80u, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tbase;
    const int grp = (int)blockIdx.y;
    const bool bias = grp == 0;
    const int t0 = (int)blockIdx.x * tiles_per, nt = min(tiles_per, q.ntiles - t0);
    bool bad = false;
    auto wait = [&](uint64_t *b, uint32_t parity) {
        if (!bad && !mbar_wait_for(b, parity, kNetWaitNs)) {
            bad = true;
            if (err) *(volatile int *)err = GPUTO_ERR_TIMEOUT;
        }
    };
    if (warp == 4) {
        int it = 0;
        for (; it < nt; ++it) {
            const int s = it % C::NST;
            if (it >= C::NST) wait(&empty[s], (uint32_t)((it / C::NST - 1) & 1));
            if (__any_sync(0xffffffffu, bad)) {
                bad = true;
                break;
            }
            if (lane == 0) mbar_arrive_expect_tx(&full[s], C::COPIED);
            __syncwarp();
            unsigned char *dst = sm + s * C::STAGE;
            const long long row = q.guard + (long long)(t0 + it) * kRows;
            for (int pl = lane; pl < C::GP + C::SEG * C::XP; pl += 32) {
                if (pl < C::GP) {
                    bulk_load(dst + pl * (kRows * 16), g + pl * q.R + row, kRows * 16, &full[s]);
                } else {
                    const int sg = (pl - C::GP) / C::XP, xp = (pl - C::GP) % C::XP, pair = grp * C::SEG + sg;
                    bulk_load(dst + C::xoff(sg) + xp * (C::XR * 16),
                              x + xp * q.R + row + (long long)(pair / 3 - 1) * q.pz + (pair % 3 - 1) * q.py - 1,
                              C::XR * 16, &full[s]);
                }
            }
        }
        // copies in flight land before the CTA leaves (they already have unless a wait gave up)
        if (bad)
            for (int k = it > C::NST ? it - C::NST : 0; k < it; ++k)
                mbar_wait_for(&full[k % C::NST], (uint32_t)((k / C::NST) & 1), kNetWaitNs);
    } else if (warp == 5) {
        if (lane == 0) {
            // M = 128, both operands transposed
            constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((128u >> 4) << 24);
            auto width = [](int n) { return (uint32_t)(n >> 3) << 17; };
            const uint32_t s0 = smem_u32(sm);
            bool issued = false;
            for (int it = 0; it < nt && !bad; ++it) {
                const int s = it % C::NST, ch = it / kWgChunk;
                const bool first = it % kWgChunk == 0, last = it % kWgChunk == kWgChunk - 1 || it == nt - 1;
                wait(&full[s], (uint32_t)((it / C::NST) & 1));
                if (bad) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t ga = s0 + s * C::STAGE;
#pragma unroll
                for (int t = 0; t < T; ++t) {
                    if (first && ch > 0) {
                        wait(&tempty[t], (uint32_t)((ch - 1) & 1));
                        if (bad) break;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    }
                    const bool ones = t == T - 1 && bias;
                    const uint32_t xa = ga + C::xoff(t / 3) + (t % 3) * 16 - (ones ? C::ONES : 0);
                    const uint32_t d = tmem + C::dcol(t) - (ones ? 8 : 0);
                    const uint32_t id = idesc | (ones ? width(C::N + 16) : width(C::N));
#pragma unroll
                    for (int ks = 0; ks < kRows / 16; ++ks) {
                        const uint32_t acc = first && ks == 0 ? 0u : 1u;
                        const uint64_t da = tc_desc(ga + ks * 256, 128, kRows * 16);
                        tc_mma(d, da, tc_desc(xa + ks * 256, 128, C::XR * 16), id, acc);
                        if (CO == 64) {
                            const uint64_t d2 = tc_desc(ga + (CO / 8) * kRows * 16 + ks * 256, 128, kRows * 16);
                            tc_mma(tmem + C::dcol(t) + 2 * CI, d2,
                                   tc_desc(ga + C::xoff(t / 3) + (t % 3) * 16 + ks * 256, 128, C::XR * 16),
                                   idesc | width(CI), 1u);
                            if (ones)
                                tc_mma(tmem + C::BIAS2, d2, tc_desc(xa + ks * 256, 128, C::XR * 16),
                                       idesc | width(16), acc);
                        }
                    }
                    issued = true;
                    if (last) tc_commit(&tfull[t]);
                }
                // only where the producer waits for it, as in conv_tc_kernel
                if (!bad && it + C::NST < nt) tc_commit(&empty[s]);
            }
            // MMAs in flight end before TMEM is freed
            if (bad && issued) {
                tc_commit(fin);
                mbar_wait_for(fin, 0, kNetWaitNs);
            }
        }
    } else {
        const uint32_t base = tmem + ((uint32_t)(warp * 32) << 16);
        const bool upper = CO == 64 && warp >= 2;
        float acc[T][CI], bacc = 0.f;
#pragma unroll
        for (int t = 0; t < T; ++t)
#pragma unroll
            for (int c = 0; c < CI; ++c) acc[t][c] = 0.f;
        const int nch = (nt + kWgChunk - 1) / kWgChunk;
        for (int ch = 0; ch < nch && !bad; ++ch) {
#pragma unroll
            for (int t = 0; t < T; ++t) {
                wait(&tfull[t], (uint32_t)(ch & 1));
                if (__any_sync(0xffffffffu, bad)) {   // the TMEM loads are warp-wide
                    bad = true;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int c0 = 0; c0 < CI; c0 += 16) {
                    uint32_t hi[16], mid[16], lo[16];
                    tc_load16(base + C::dcol(t) + 2 * CI + c0, lo);
                    tc_load16(base + C::dcol(t) + CI + c0, mid);
                    tc_load16(base + C::dcol(t) + c0, hi);
                    tc_wait_loads(lo);
                    tc_wait_loads(mid);
                    tc_wait_loads(hi);
#pragma unroll
                    for (int c = 0; c < 16; ++c) {
                        float s = __uint_as_float(lo[c]) + __uint_as_float(mid[c]);
                        if (!upper) s += __uint_as_float(hi[c]);
                        acc[t][c0 + c] += s;
                    }
                }
                if (t == T - 1 && bias) {
                    uint32_t o[16];
                    tc_load16(base + C::dcol(T - 1) - 8, o);
                    tc_wait_loads(o);
                    bacc += __uint_as_float(o[0]);
                    if (upper) {
                        tc_load16(base + C::BIAS2, o);
                        tc_wait_loads(o);
                        bacc += __uint_as_float(o[0]);
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&tempty[t])) : "memory");
            }
        }
        const int sub = tid / CO, co = tid % CO;
        if (!bad && sub < C::SUBS) {
            const size_t k = (size_t)blockIdx.x * C::SUBS + sub;
            float *dst = part + (k * 27 + 3 * C::SEG * grp) * (CI * CO) + co;
#pragma unroll
            for (int t = 0; t < T; ++t)
#pragma unroll
                for (int c = 0; c < CI; ++c) dst[(t * CI + c) * CO] = acc[t][c];
            if (bias) bpart[k * CO + co] = bacc;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::COLS) : "memory");
}

// The same sums of layer 1, whose 4 channels are too few for the tensor cores,
// one CTA per (row range, dx).  A thread keeps two output channels x the 9
// (dz, dy) taps of one input channel in registers: per row it reads its two
// gradients (the same for a warp) and three new input values (the dy taps
// slide along the row), for 18 FMAs as paired instructions.  The CTAs' sums go
// to part[range][(co 4 + ci) 27 + tap].  Bound by the staging's latency: with
// the index arithmetic of every channel of its own and in 64 bits, eight 33^3
// samples took 158 us, now 70 us; tiles of 96 or 30 rows 5 and 15 us more.
constexpr int kWg1Rows = 48;   // rows staged at a time

__global__ void __launch_bounds__(32)
wgrad1_kernel(const uint4 *__restrict__ g, const float *__restrict__ xd, float *__restrict__ part,
              float *__restrict__ bpart, RowGeo q, int tiles_per)
{
    constexpr int CO = 16, CI = 4, GP = CO + 4;
    __shared__ __align__(16) float gs[kWg1Rows][GP];
    __shared__ __align__(16) float xs[3][kWg1Rows + 2][CI + 4];
    const int tid = threadIdx.x, ci = tid % CI, cg = tid / CI;
    const int dx = (int)blockIdx.y - 1;
    const long long ntile = (q.rows + kWg1Rows - 1) / kWg1Rows, n = (long long)q.X * q.Z * q.Y;
    const long long t0 = (long long)blockIdx.x * tiles_per, t1 = min(t0 + tiles_per, ntile);
    float2 acc[9], bsum = make_float2(0.f, 0.f);
#pragma unroll
    for (int t = 0; t < 9; ++t) acc[t] = make_float2(0.f, 0.f);
    for (long long tile = t0; tile < t1; ++tile) {
        const long long r0 = tile * kWg1Rows;
        __syncthreads();
        for (int i = tid; i < kWg1Rows * (CO / 8); i += 32) {
            const int c = i / kWg1Rows, rr = i - c * kWg1Rows;
            float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (r0 + rr < q.rows)
#pragma unroll
                for (int p = 2; p >= 0; --p) add_part(v, g[(size_t)(p * (CO / 8) + c) * q.R + q.guard + r0 + rr]);
            float4 *d = reinterpret_cast<float4 *>(&gs[rr][8 * c]);
            d[0] = make_float4(v[0], v[1], v[2], v[3]);
            d[1] = make_float4(v[4], v[5], v[6], v[7]);
        }
#pragma unroll
        for (int k = 0; k < (3 * (kWg1Rows + 2) + 31) / 32; ++k) {
            const int i = tid + 32 * k, dz = i / (kWg1Rows + 2), rr = i - dz * (kWg1Rows + 2);
            if (dz > 2) break;
            const long long r = r0 + rr - 1 + (long long)dx * q.pz + (dz - 1) * q.py;
            int s, x, z, y;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r >= 0 && row_node(q, r, s, x, z, y)) {
                const float *p = xd + 4LL * s * n + ((long long)x * q.Z + z) * q.Y + y;
                v = make_float4(p[0], p[n], p[2 * n], p[3 * n]);
            }
            *reinterpret_cast<float4 *>(xs[dz][rr]) = v;
        }
        __syncthreads();
        float xw[3][3];   // [dz][row mod 3]
#pragma unroll
        for (int dz = 0; dz < 3; ++dz) {
            xw[dz][0] = xs[dz][0][ci];
            xw[dz][1] = xs[dz][1][ci];
        }
#pragma unroll 1
        for (int rb = 0; rb < kWg1Rows; rb += 3)
#pragma unroll
            for (int u = 0; u < 3; ++u) {
                const int rr = rb + u;
                const float2 gv = *reinterpret_cast<const float2 *>(&gs[rr][2 * cg]);
#pragma unroll
                for (int dz = 0; dz < 3; ++dz) xw[dz][(u + 2) % 3] = xs[dz][rr + 2][ci];
                if (dx == -1) bsum = __fadd2_rn(bsum, gv);
#pragma unroll
                for (int dz = 0; dz < 3; ++dz)
#pragma unroll
                    for (int dy = 0; dy < 3; ++dy) {
                        const float v = xw[dz][(u + dy) % 3];
                        acc[3 * dz + dy] = __ffma2_rn(gv, make_float2(v, v), acc[3 * dz + dy]);
                    }
            }
    }
    float *dst = part + (size_t)blockIdx.x * (CO * CI * 27) + 9 * blockIdx.y;
#pragma unroll
    for (int t = 0; t < 9; ++t) {
        dst[(2 * cg * CI + ci) * 27 + t] = acc[t].x;
        dst[((2 * cg + 1) * CI + ci) * 27 + t] = acc[t].y;
    }
    if (dx == -1 && ci == 0) {
        bpart[(size_t)blockIdx.x * CO + 2 * cg] = bsum.x;
        bpart[(size_t)blockIdx.x * CO + 2 * cg + 1] = bsum.y;
    }
}

// grads[i] += sum over ranges of part[range][i]: a CTA takes 32 entries, its
// eight warps every eighth range, and the warps' sums are added in order.
// With co > 0 the parts are in the order [tap][ci][co] of wgrad_tc_kernel.
__global__ void __launch_bounds__(256)
sum_parts_kernel(const float *__restrict__ part, int n, int ranges, float *__restrict__ grads, int co = 0, int ci = 0)
{
    __shared__ float red[8][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (i < n)
#pragma unroll 8
        for (int b = w; b < ranges; b += 8) s += part[(size_t)b * n + i];
    red[w][lane] = s;
    __syncthreads();
    if (w == 0 && i < n) {
        s = red[0][lane];
        for (int k = 1; k < 8; ++k) s += red[k][lane];
        grads[co ? ((i % co) * ci + i / co % ci) * 27 + i / (co * ci) : i] += s;
    }
}

// Masked mean square error: partial sums per CTA (blockIdx.y = sample), then
// a single-CTA finish (a warp per sample, lanes in order of the CTAs) that
// adds the losses and writes the gradients' scales; fixed order.
__global__ void __launch_bounds__(256)
mse_partial_kernel(const float *__restrict__ y, const float *__restrict__ t, const float *__restrict__ m, long long n,
                   double *__restrict__ part)
{
    const long long o = (long long)blockIdx.y * n;
    double s = 0.0, c = 0.0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double r = (double)y[o + i] - (double)t[o + i];
        s += (double)m[o + i] * r * r;
        c += (double)m[o + i];
    }
    __shared__ double rs[8], rc[8];
    for (int w = 16; w > 0; w >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, w);
        c += __shfl_xor_sync(0xffffffffu, c, w);
    }
    if ((threadIdx.x & 31) == 0) rs[threadIdx.x >> 5] = s, rc[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int w = 0; w < 8; ++w) a += rs[w], b += rc[w];
        double *p = part + 2 * ((size_t)blockIdx.y * gridDim.x + blockIdx.x);
        p[0] = a;
        p[1] = b;
    }
}

__global__ void __launch_bounds__(1024)
mse_finish_kernel(const double *__restrict__ part, int nb, int samples, double *__restrict__ loss_acc,
                  float *__restrict__ gscale)
{
    __shared__ double ls[32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int s0 = 0; s0 < samples; s0 += 32) {
        const int s = s0 + warp;
        double a = 0.0, b = 0.0;
        if (s < samples)
            for (int k = lane; k < nb; k += 32) {
                a += part[2 * ((size_t)s * nb + k)];
                b += part[2 * ((size_t)s * nb + k) + 1];
            }
        for (int w = 16; w > 0; w >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, w);
            b += __shfl_xor_sync(0xffffffffu, b, w);
        }
        const double den = b > 1.0 ? b : 1.0;
        if (lane == 0) {
            ls[warp] = s < samples ? a / den : 0.0;
            if (s < samples) gscale[s] = (float)(2.0 / den);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double l = *loss_acc;
            for (int w = 0; w < 32; ++w) l += ls[w];
            *loss_acc = l;
        }
        __syncthreads();
    }
}

__global__ void mse_grad_kernel(const float *__restrict__ y, const float *__restrict__ t, const float *__restrict__ m,
                                long long n, const float *__restrict__ gscale, float *__restrict__ g)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long o = (long long)blockIdx.y * n + i;
    if (i < n) g[o] = gscale[blockIdx.y] * m[o] * (y[o] - t[o]);
}

__global__ void adam_kernel(float *__restrict__ p, float *__restrict__ g, float *__restrict__ m1, float *__restrict__ m2,
                            long long n, float lr, float gscale, float bc1, float bc2)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i] * gscale;
    const float a = 0.9f * m1[i] + 0.1f * gi;
    const float v = 0.999f * m2[i] + 0.001f * gi * gi;
    m1[i] = a;
    m2[i] = v;
    p[i] -= lr * (a / bc1) / (sqrtf(v / bc2) + 1e-8f);
    g[i] = 0.f;
}

// Persistent grids: CTAs per SM by shared memory (1 for K N >= 2048, else 2).
template <int CK, int CN, int EPI>
void launch_conv(const ConvArgs &a, const RowGeo &q, int sms, cudaStream_t st)
{
    using C = ConvCfg<CK, CN>;
    const int per = C::SMEM <= 113 * 1024 ? 2 : 1;
    conv_tc_kernel<CK, CN, EPI><<<std::min(q.ntiles, per * sms), 192, C::SMEM, st>>>(a, q);
    count_launches(1);
}

// Partial sums of the weight gradients: layer 1 in up to 784 row ranges (a CTA
// of one warp per range and dx; with 98 most of the chip idles, 848 us on
// eight 33^3 samples), layers 2 and 3 in as many as give every SM one CTA.
constexpr int kWg1Ranges = 784, kWgMaxCtas = 296;
constexpr int kWgMaxWeights = std::max({kWg1Ranges * 16 * 4 * 27, kWgMaxCtas / 3 * 3 * 32 * 16 * 27, kWgMaxCtas / 9 * 2 * 64 * 32 * 27});
constexpr int kWgMaxBias = std::max({kWg1Ranges * 16, kWgMaxCtas / 3 * 3 * 32, kWgMaxCtas / 9 * 2 * 64});

void launch_wgrad1(const uint4 *g, const float *x, float *part, float *bpart, float *gw, float *gb, const RowGeo &q,
                   cudaStream_t st)
{
    const long long ntile = (q.rows + kWg1Rows - 1) / kWg1Rows;
    const int per = (int)((ntile + kWg1Ranges - 1) / kWg1Ranges), ranges = (int)((ntile + per - 1) / per);
    wgrad1_kernel<<<dim3((unsigned)ranges, 3), 32, 0, st>>>(g, x, part, bpart, q, per);
    constexpr int n = 16 * 4 * 27;
    sum_parts_kernel<<<(n + 31) / 32, 256, 0, st>>>(part, n, ranges, gw);
    sum_parts_kernel<<<1, 256, 0, st>>>(bpart, 16, ranges, gb);
    count_launches(3);
}

template <int CO, int CI>
void launch_wgrad(const uint4 *g, const uint4 *x, float *part, float *bpart, float *gw, float *gb, const RowGeo &q,
                  int sms, int *err, cudaStream_t st)
{
    using C = WgCfg<CO, CI>;
    const int most = std::max(1, std::min(sms, kWgMaxCtas) / C::GROUPS);
    const int per = (q.ntiles + most - 1) / most, ranges = (q.ntiles + per - 1) / per;
    wgrad_tc_kernel<CO, CI><<<dim3((unsigned)ranges, C::GROUPS), 192, C::SMEM, st>>>(g, x, part, bpart, q, per, err);
    constexpr int n = CO * CI * 27;
    sum_parts_kernel<<<(n + 31) / 32, 256, 0, st>>>(part, n, ranges * C::SUBS, gw, CO, CI);
    sum_parts_kernel<<<(CO + 31) / 32, 256, 0, st>>>(bpart, CO, ranges * C::SUBS, gb);
    count_launches(3);
}

}  // namespace

// ---------------------------------------------------------------------------
// Net: parameters, Adam state and work buffers on one device
// ---------------------------------------------------------------------------

long long Net::num_params()
{
    long long s = 0;
    for (int l = 0; l < 4; ++l) s += (long long)net_ch(l + 1) * net_ch(l) * net_k(l) * net_k(l) * net_k(l) + net_ch(l + 1);
    return s;
}

long long Net::param_offset(int l, bool bias)
{
    long long o = 0;
    for (int q = 0; q < l; ++q) o += (long long)net_ch(q + 1) * net_ch(q) * net_k(q) * net_k(q) * net_k(q) + net_ch(q + 1);
    if (bias) o += (long long)net_ch(l + 1) * net_ch(l) * net_k(l) * net_k(l) * net_k(l);
    return o;
}

Net::~Net()
{
    for (void *p : owned) cudaFree(p);
    if (h_err) cudaFreeHost(h_err);
}

int Net::create(unsigned long long seed)
{
    GPUTO_CUDA(cudaGetDevice(&device));
    GPUTO_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    const long long np = num_params();
    for (float **p : {&params, &grads, &m1, &m2}) {
        GPUTO_CUDA(cudaMalloc(p, sizeof(float) * np));
        owned.push_back(*p);
        GPUTO_CUDA(cudaMemset(*p, 0, sizeof(float) * np));
    }
    // part: kNetPart doubles of reduction scratch, the summed loss, a gradient scale per sample of a group
    GPUTO_CUDA(cudaMalloc(&part, sizeof(double) * (kNetPart + 1) + sizeof(float) * kNetGroup));
    owned.push_back(part);
    loss_acc = part + kNetPart;
    gscale = reinterpret_cast<float *>(loss_acc + 1);
    GPUTO_CUDA(cudaMalloc(&img, 2 * 2 * (size_t)(kImg2 + kImg3)));
    owned.push_back(img);
    // where a kernel's bounded wait reports that it gave up: read by the host after a synchronisation
    GPUTO_CUDA(cudaHostAlloc((void **)&h_err, sizeof(int), cudaHostAllocMapped));
    *h_err = 0;
    GPUTO_CUDA(cudaHostGetDevicePointer((void **)&d_err, h_err, 0));
    // He-normal initial weights (last layer scaled by 0.1), zero biases;
    // a fixed generator so that a seed reproduces the network
    std::vector<float> h((size_t)np, 0.f);
    unsigned long long s = seed * 6364136223846793005ULL + 1442695040888963407ULL;
    auto uni = [&]() {
        s = s * 6364136223846793005ULL + 1442695040888963407ULL;
        return ((s >> 11) + 0.5) * (1.0 / 9007199254740992.0);
    };
    for (int l = 0; l < 4; ++l) {
        const long long nw = (long long)net_ch(l + 1) * net_ch(l) * net_k(l) * net_k(l) * net_k(l);
        const double std = std::sqrt(2.0 / ((double)net_ch(l) * net_k(l) * net_k(l) * net_k(l))) * (l == 3 ? 0.1 : 1.0);
        const long long o = param_offset(l, false);
        for (long long i = 0; i < nw; ++i) {
            const double u1 = uni(), u2 = uni();
            h[(size_t)(o + i)] = (float)(std * std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2));
        }
    }
    GPUTO_CUDA(cudaMemcpy(params, h.data(), sizeof(float) * np, cudaMemcpyHostToDevice));
    return GPUTO_OK;
}

// Work buffers for S samples of a grid at once (train: also the backward
// pass's).  They only grow; a buffer that is outgrown stays allocated until
// the network goes, since a solver's captured graph may still use it.
int Net::reserve(const NetDims &d, int S, bool train)
{
    const RowGeo q = row_geo(d, S);
    auto grow = [&](auto **p, size_t &cap, size_t bytes) -> int {
        if (bytes <= cap) return GPUTO_OK;
        void *v = nullptr;
        GPUTO_CUDA(cudaMalloc(&v, bytes));
        owned.push_back(v);
        *p = reinterpret_cast<std::remove_reference_t<decltype(*p)>>(v);
        cap = bytes;
        return GPUTO_OK;
    };
    const size_t plane = 16 * (size_t)q.R, dense = sizeof(float) * 3 * (size_t)d.n() * S;
    int s = grow(&rows1, cap[0], 6 * plane);
    if (!s) s = grow(&rows2, cap[1], 12 * plane);
    if (!s) s = grow(&y, cap[2], dense);
    if (train) {
        if (!s) s = grow(&gy, cap[3], dense);
        if (!s) s = grow(&act3, cap[4], sizeof(float) * 64 * (size_t)q.ntiles * kRows);
        if (!s) s = grow(&g3, cap[5], 24 * plane);
        if (!s) s = grow(&g2, cap[6], 12 * plane);
        if (!s) s = grow(&g1, cap[7], 6 * plane);
        if (!s) s = grow(&wpart, cap[8], sizeof(float) * ((size_t)kWgMaxWeights + kWgMaxBias +
                                                          (size_t)4 * sms * kHeadPart));
    }
    return s;
}

int Net::group(const NetDims &d, int ns) const
{
    const long long per = row_geo(d, 1).rows;
    return (int)std::max(1LL, std::min<long long>({(long long)ns, (long long)kNetGroup, (1LL << 20) / per}));
}

int init_net_kernels()
{
    static bool done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && done[dev]) return GPUTO_OK;
    auto set = [](auto *k, size_t b) {
        return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b);
    };
    GPUTO_CUDA(set(conv_tc_kernel<16, 32, EPI_RELU>, ConvCfg<16, 32>::SMEM));
    GPUTO_CUDA(set(conv_tc_kernel<32, 64, EPI_HEAD>, ConvCfg<32, 64>::SMEM));
    GPUTO_CUDA(set(conv_tc_kernel<64, 32, EPI_MASK>, ConvCfg<64, 32>::SMEM));
    GPUTO_CUDA(set(conv_tc_kernel<32, 16, EPI_MASK>, ConvCfg<32, 16>::SMEM));
    GPUTO_CUDA(set(wgrad_tc_kernel<64, 32>, WgCfg<64, 32>::SMEM));
    GPUTO_CUDA(set(wgrad_tc_kernel<32, 16>, WgCfg<32, 16>::SMEM));
    if (dev < 64) done[dev] = true;
    return GPUTO_OK;
}

int Net::check()
{
    if (!*(volatile int *)h_err) return GPUTO_OK;
    const int e = *(volatile int *)h_err;
    *(volatile int *)h_err = 0;
    set_error("a bounded wait of the network's convolution gave up");
    return e;
}

int Net::forward(const float *x, const NetDims &d, int S, float *yout, bool train, cudaStream_t st)
{
    int s = reserve(d, S, train);
    if (s) return s;
    const RowGeo q = row_geo(d, S);
    const float *p = params;
    GuardSets gs{{rows1, rows2, g3, g2, nullptr}, {6, 12, 24, 12, 0}};
    zero_guards_kernel<<<dim3(64, train ? 4 : 2), 256, 0, st>>>(gs, q);
    pack_weights_kernel<<<(2 * (kImg2 + kImg3) + 255) / 256, 256, 0, st>>>(p + param_offset(1, false),
                                                                          p + param_offset(2, false),
                                                                          (__nv_bfloat16 *)img);
    conv1_kernel<<<(q.ntiles + kC1R - 1) / kC1R, 128, 0, st>>>(x, p + param_offset(0, false), p + param_offset(0, true), rows1, q);
    count_launches(3);
    const uint4 *im = reinterpret_cast<const uint4 *>(img);
    ConvArgs a{};
    a.err = d_err;
    a.a = rows1;
    a.img = im;
    a.bias = p + param_offset(1, true);
    a.out = rows2;
    launch_conv<16, 32, EPI_RELU>(a, q, sms, st);
    a.a = rows2;
    a.img = im + kImg2 / 8;
    a.bias = p + param_offset(2, true);
    a.w4 = p + param_offset(3, false);
    a.b4 = p + param_offset(3, true);
    a.y = yout ? yout : y;
    a.act = train ? act3 : nullptr;
    launch_conv<32, 64, EPI_HEAD>(a, q, sms, st);
    return GPUTO_OK;
}

// Losses of S samples (x, target t, mask m) added to loss_acc, gradients
// added to grads.
int Net::accumulate(const float *x, const float *t, const float *m, const NetDims &d, int S, cudaStream_t st)
{
    int s = forward(x, d, S, nullptr, true, st);
    if (s) return s;
    const long long n3 = 3 * d.n();
    const int nb = (int)std::max(1LL, std::min<long long>(kNetPart / 2 / S, (n3 + 255) / 256));
    mse_partial_kernel<<<dim3((unsigned)nb, (unsigned)S), 256, 0, st>>>(y, t, m, n3, part);
    mse_finish_kernel<<<1, 1024, 0, st>>>(part, nb, S, loss_acc, gscale);
    mse_grad_kernel<<<dim3((unsigned)((n3 + 255) / 256), (unsigned)S), 256, 0, st>>>(y, t, m, n3, gscale, gy);
    count_launches(3);
    return backward_from(x, d, S, st);
}

int Net::adam(float lr, int nsamples, cudaStream_t st)
{
    ++step;
    const float bc1 = 1.f - std::pow(0.9f, (float)step), bc2 = 1.f - std::pow(0.999f, (float)step);
    const long long np = num_params();
    adam_kernel<<<(unsigned)((np + 255) / 256), 256, 0, st>>>(params, grads, m1, m2, np, lr,
                                                             1.f / (float)std::max(nsamples, 1), bc1, bc2);
    count_launches(1);
    return GPUTO_OK;
}

// The backward pass of the last training forward from the output gradient in
// gy; adds to grads.
int Net::backward_from(const float *x, const NetDims &d, int S, cudaStream_t st)
{
    const RowGeo q = row_geo(d, S);
    const float *p = params;
    float *bpart = wpart + kWgMaxWeights, *hpart = bpart + kWgMaxBias;
    // four CTAs fit an SM and wait on memory: 67 us with two, 48 with four (eight 33^3 samples)
    const int hb = std::min(q.ntiles, 4 * sms);
    head_backward_kernel<<<hb, 256, 0, st>>>(gy, act3, p + param_offset(3, false), g3, hpart, q);
    // the head's 192 weights and 3 biases are adjacent in grads
    sum_parts_kernel<<<(kHeadPart + 31) / 32, 256, 0, st>>>(hpart, kHeadPart, hb, grads + param_offset(3, false));
    count_launches(2);
    const uint4 *im = reinterpret_cast<const uint4 *>(img);
    ConvArgs a{};
    a.err = d_err;
    a.a = g3;
    a.img = im + (kImg2 + kImg3) / 8;
    a.mask = rows2;
    a.out = g2;
    launch_conv<64, 32, EPI_MASK>(a, q, sms, st);
    a.a = g2;
    a.img = im + (kImg2 + 2 * kImg3) / 8;
    a.mask = rows1;
    a.out = g1;
    launch_conv<32, 16, EPI_MASK>(a, q, sms, st);
    auto gw = [&](int l) { return grads + param_offset(l, false); };
    auto gb = [&](int l) { return grads + param_offset(l, true); };
    launch_wgrad<64, 32>(g3, rows2, wpart, bpart, gw(2), gb(2), q, sms, d_err, st);
    launch_wgrad<32, 16>(g2, rows1, wpart, bpart, gw(1), gb(1), q, sms, d_err, st);
    launch_wgrad1(g1, x, wpart, bpart, gw(0), gb(0), q, st);
    return GPUTO_OK;
}

// ---------------------------------------------------------------------------
// level-2 features and the correction's way back to the fine grid
// ---------------------------------------------------------------------------

// Density feature at a level-2 node: mean element scale of the adjacent
// level-2 elements (each the mean of its fine elements), (log10 + 9) / 9.
__global__ void net_density_kernel(Grid g2, Grid gf, const double *__restrict__ CXf, float *__restrict__ dens2)
{
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= g2.nnod()) return;
    const int j = (int)(n % (g2.ny + 1));
    const long long r = n / (g2.ny + 1);
    const int k = (int)(r % (g2.nz + 1)), i = (int)(r / (g2.nz + 1));
    const int fx = gf.nx / g2.nx, fy = gf.ny / g2.ny, fz = gf.nz / g2.nz;
    double s = 0.0;
    int cnt = 0;
    for (int ex = i - 1; ex <= i; ++ex)
        for (int ez = k - 1; ez <= k; ++ez)
            for (int ey = j - 1; ey <= j; ++ey) {
                if (ex < 0 || ex >= g2.nx || ez < 0 || ez >= g2.nz || ey < 0 || ey >= g2.ny) continue;
                double c = 0.0;
                for (int a = 0; a < fx; ++a)
                    for (int b = 0; b < fz; ++b)
                        for (int q = 0; q < fy; ++q) c += CXf[gf.elem(ex * fx + a, ey * fy + q, ez * fz + b)];
                s += c / (fx * fy * fz);
                ++cnt;
            }
    const double m = cnt ? s / cnt : 1e-9;
    dens2[n] = (float)((log10(fmax(m, 1e-9)) + 9.0) / 9.0);
}

void launch_net_density(const Grid &g2, const Grid &gf, const double *CXf, float *dens2, cudaStream_t st)
{
    net_density_kernel<<<(unsigned)((g2.nnod() + 255) / 256), 256, 0, st>>>(g2, gf, CXf, dens2);
    count_launches(1);
}

// The network works in Jacobi-scaled units, in which the level-2 operator
// has a unit diagonal: input r~ = D^-1/2 r, output e~ with e = D^-1/2 e~,
// both divided by s = RMS of r~ (free dofs; fixed dofs have r = 0).  That
// keeps the stiffness contrast of SIMP designs (1e9 here) out of the values
// the network sees.

// s = RMS of D^-1/2 r2 (one CTA, fixed order)
__global__ void __launch_bounds__(1024) net_rms_kernel(Lay L2, const float *__restrict__ r2,
                                                     const float *__restrict__ diag2, float *__restrict__ s,
                                                     const int *__restrict__ done)
{
    if (done && *done) return;
    const Grid &g = L2.g;
    const long long nn = g.nnod();
    double acc = 0.0;
    for (long long n = threadIdx.x; n < nn; n += blockDim.x) {
        const int j = (int)(n % (g.ny + 1));
        const long long r = n / (g.ny + 1);
        const int k = (int)(r % (g.nz + 1)), i = (int)(r / (g.nz + 1));
        const long long b = L2.at(i, j, k);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double dv = diag2[b + d];
            if (dv > 0.0) acc += (double)r2[b + d] * r2[b + d] / dv;
        }
    }
    __shared__ double red[32];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
        const double rms = sqrt(t / (3.0 * (double)nn));
        *s = rms > 0.0 ? (float)rms : 1.f;
    }
}

__global__ void net_features_kernel(Lay L2, const float *__restrict__ r2, const float *__restrict__ diag2,
                                    const float *__restrict__ dens2, float *__restrict__ x, float *__restrict__ dsq,
                                    const float *__restrict__ s, const int *__restrict__ done)
{
    if (done && *done) return;
    const Grid &g = L2.g;
    const long long nn = g.nnod();
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nn) return;
    const int j = (int)(n % (g.ny + 1));
    const long long r = n / (g.ny + 1);
    const int k = (int)(r % (g.nz + 1)), i = (int)(r / (g.nz + 1));
    const float inv = 1.f / *s;
    const long long b = L2.at(i, j, k);
    x[n] = dens2[n];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float dv = diag2[b + d];
        const float sq = dv > 0.f ? sqrtf(dv) : 1.f;
        x[(1 + d) * nn + n] = r2[b + d] / sq * inv;
        if (dsq) dsq[d * nn + n] = sq;
    }
}

void launch_net_features(const Lay &L2, const float *r2, const float *diag2, const float *dens2, float *x,
                         float *dsq, float *s, const int *done, cudaStream_t st)
{
    net_rms_kernel<<<1, 1024, 0, st>>>(L2, r2, diag2, s, done);
    net_features_kernel<<<(unsigned)((L2.g.nnod() + 255) / 256), 256, 0, st>>>(L2, r2, diag2, dens2, x, dsq, s,
                                                                               done);
    count_launches(2);
}

// e2 = s D^-1/2 y at the free dofs of level 2, 0 at fixed dofs
__global__ void net_output_kernel(Lay L2, const float *__restrict__ y, const float *__restrict__ diag2,
                                  const float *__restrict__ s, const uint8_t *__restrict__ mask2,
                                  float *__restrict__ e2, const int *__restrict__ done)
{
    if (done && *done) return;
    const Grid &g = L2.g;
    const long long nn = g.nnod();
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nn) return;
    const int j = (int)(n % (g.ny + 1));
    const long long r = n / (g.ny + 1);
    const int k = (int)(r % (g.nz + 1)), i = (int)(r / (g.nz + 1));
    const unsigned m = mask2[n];
    const float sc = *s;
    const long long b = L2.at(i, j, k);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float dv = diag2[b + d];
        e2[b + d] = ((m >> d) & 1u) || !(dv > 0.f) ? 0.f : sc * y[d * nn + n] / sqrtf(dv);
    }
}

void launch_net_output(const Lay &L2, const float *y, const float *diag2, const float *s, const uint8_t *mask2,
                       float *e2, const int *done, cudaStream_t st)
{
    net_output_kernel<<<(unsigned)((L2.g.nnod() + 255) / 256), 256, 0, st>>>(L2, y, diag2, s, mask2, e2, done);
    count_launches(1);
}

__global__ void add_f2d_kernel(long long n, const float *__restrict__ e, double *__restrict__ z,
                               const int *__restrict__ done)
{
    if (done && *done) return;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) z[i] += (double)e[i];
}

void launch_add_f2d(long long n, const float *e, double *z, const int *done, cudaStream_t st)
{
    add_f2d_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, e, z, done);
    count_launches(1);
}

// Loss mask of the level-2 dofs: 1 free, 0 fixed, channels-first [3][n]
__global__ void net_mask_kernel(Grid g2, const uint8_t *__restrict__ mask2, float *__restrict__ m)
{
    const long long nn = g2.nnod();
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nn) return;
    const unsigned b = mask2[n];
#pragma unroll
    for (int d = 0; d < 3; ++d) m[d * nn + n] = ((b >> d) & 1u) ? 0.f : 1.f;
}

void launch_net_mask(const Grid &g2, const uint8_t *mask2, float *m, cudaStream_t st)
{
    net_mask_kernel<<<(unsigned)((g2.nnod() + 255) / 256), 256, 0, st>>>(g2, mask2, m);
    count_launches(1);
}

// Values of a fine dense vector (the reference's layout) at the level-2
// nodes (fine node (fx i, fy j, fz k)), channels-first [3][n]
__global__ void level2_inject_kernel(Grid g2, Grid gf, const double *__restrict__ v, float *__restrict__ out)
{
    const long long nn = g2.nnod();
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nn) return;
    const int j = (int)(n % (g2.ny + 1));
    const long long r = n / (g2.ny + 1);
    const int k = (int)(r % (g2.nz + 1)), i = (int)(r / (g2.nz + 1));
    const long long nf = gf.node(i * (gf.nx / g2.nx), j * (gf.ny / g2.ny), k * (gf.nz / g2.nz));
#pragma unroll
    for (int d = 0; d < 3; ++d) out[d * nn + n] = (float)v[3 * nf + d];
}

void launch_level2_inject(const Grid &g2, const Grid &gf, const double *v, float *out, cudaStream_t st)
{
    level2_inject_kernel<<<(unsigned)((g2.nnod() + 255) / 256), 256, 0, st>>>(g2, gf, v, out);
    count_launches(1);
}

// ---------------------------------------------------------------------------
// energy loss of the correction (level-2 operator A2 in the scaled units)
// ---------------------------------------------------------------------------
//
// With the correction c = s D^-1/2 y added after the V-cycle, the energy of
// the remaining error is, up to a constant, c'A2 c - 2 c'g2 with
// g2 = P'(r - A z) the twice-restricted post-V-cycle residual and A2 = P'AP
// the Galerkin level-2 operator.  Divided by s^2 this is
//   L = y'A~y - 2 y'g~,   A~ = D^-1/2 A2 D^-1/2,  g~ = D^-1/2 g2 / s,
// with gradient 2 (A~y - g~).  L(0) = 0: any learned correction lowers it.

// w = D^-1/2 y in the padded level-2 layout (0 at fixed dofs)
__global__ void net_to_padded_kernel(Lay L2, const float *__restrict__ y, const float *__restrict__ diag2,
                                     const uint8_t *__restrict__ mask2, float *__restrict__ w)
{
    const Grid &g = L2.g;
    const long long nn = g.nnod();
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nn) return;
    const int j = (int)(n % (g.ny + 1));
    const long long r = n / (g.ny + 1);
    const int k = (int)(r % (g.nz + 1)), i = (int)(r / (g.nz + 1));
    const unsigned m = mask2[n];
    const long long b = L2.at(i, j, k);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float dv = diag2[b + d];
        w[b + d] = ((m >> d) & 1u) || !(dv > 0.f) ? 0.f : y[d * nn + n] / sqrtf(dv);
    }
}

// gy = 2 (D^-1/2 q - g~), partial sums of y'(D^-1/2 q) - 2 y'g~ per CTA
__global__ void __launch_bounds__(256)
net_energy_kernel(Lay L2, const float *__restrict__ y, const float *__restrict__ q, const float *__restrict__ diag2,
                  const float *__restrict__ gt, const uint8_t *__restrict__ mask2, float *__restrict__ gy,
                  double *__restrict__ part)
{
    const Grid &g = L2.g;
    const long long nn = g.nnod();
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double acc = 0.0;
    if (n < nn) {
        const int j = (int)(n % (g.ny + 1));
        const long long r = n / (g.ny + 1);
        const int k = (int)(r % (g.nz + 1)), i = (int)(r / (g.nz + 1));
        const unsigned m = mask2[n];
        const long long b = L2.at(i, j, k);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const float dv = diag2[b + d];
            const bool free_dof = !((m >> d) & 1u) && dv > 0.f;
            const float aq = free_dof ? q[b + d] / sqrtf(dv) : 0.f;
            const float gv = free_dof ? gt[d * nn + n] : 0.f;
            const float yv = free_dof ? y[d * nn + n] : 0.f;
            gy[d * nn + n] = 2.f * (aq - gv);
            acc += (double)yv * aq - 2.0 * (double)yv * gv;
        }
    }
    __shared__ double red[8];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < 8; ++w) s += red[w];
        part[blockIdx.x] = s;
    }
}

__global__ void net_energy_finish_kernel(const double *__restrict__ part, int nb, double *__restrict__ loss_acc)
{
    if (threadIdx.x != 0) return;
    double s = 0.0;
    for (int q = 0; q < nb; ++q) s += part[q];
    *loss_acc += s;
}

void launch_net_to_padded(const Lay &L2, const float *y, const float *diag2, const uint8_t *mask2, float *w,
                          cudaStream_t st)
{
    net_to_padded_kernel<<<(unsigned)((L2.g.nnod() + 255) / 256), 256, 0, st>>>(L2, y, diag2, mask2, w);
    count_launches(1);
}

int launch_net_energy(const Lay &L2, const float *y, const float *q, const float *diag2, const float *gt,
                      const uint8_t *mask2, float *gy, double *part, int part_cap, double *loss_acc, cudaStream_t st)
{
    const int nb = (int)((L2.g.nnod() + 255) / 256);
    if (nb > part_cap) {
        set_error("level-2 grid too large for the network loss scratch");
        return GPUTO_ERR_ARG;
    }
    net_energy_kernel<<<nb, 256, 0, st>>>(L2, y, q, diag2, gt, mask2, gy, part);
    net_energy_finish_kernel<<<1, 32, 0, st>>>(part, nb, loss_acc);
    count_launches(2);
    return GPUTO_OK;
}

// g~ = D^-1/2 v2 / s at the level-2 nodes, channels-first (0 at fixed dofs),
// for a padded level-2 vector v2
__global__ void net_energy_rhs_kernel(Lay L2, const float *__restrict__ v2, const float *__restrict__ diag2,
                                      const uint8_t *__restrict__ mask2, float scale, float *__restrict__ gt)
{
    const Grid &g = L2.g;
    const long long nn = g.nnod();
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nn) return;
    const int j = (int)(n % (g.ny + 1));
    const long long r = n / (g.ny + 1);
    const int k = (int)(r % (g.nz + 1)), i = (int)(r / (g.nz + 1));
    const unsigned m = mask2[n];
    const long long b = L2.at(i, j, k);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float dv = diag2[b + d];
        gt[d * nn + n] = ((m >> d) & 1u) || !(dv > 0.f) ? 0.f : v2[b + d] / sqrtf(dv) / scale;
    }
}

void launch_net_energy_rhs(const Lay &L2, const float *v2, const float *diag2, const uint8_t *mask2, float scale,
                           float *gt, cudaStream_t st)
{
    net_energy_rhs_kernel<<<(unsigned)((L2.g.nnod() + 255) / 256), 256, 0, st>>>(L2, v2, diag2, mask2, scale, gt);
    count_launches(1);
}

}  // namespace gputo
