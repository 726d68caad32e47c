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
// Inference and training run different kernels:
//  * inference (Net::forward): the 16 -> 32 and 32 -> 64 convolutions are
//    implicit GEMMs on the 5th-generation tensor cores (conv_tc_kernel), the
//    first layer and the 1x1x1 head run on the CUDA cores;
//  * training (Net::accumulate, Net::backward_from): direct FP32 convolutions,
//    forward and backward, each sum one chain of FMAs in a fixed order.  An
//    Adam step divides the gradient by its own size and the weights are rounded
//    to BF16, so a training amplifies the last bit of a sum: after five steps
//    two roundings of the same sums give gradients 1e-4 to 3e-3 apart
//    (measured).  A training repeats only where the order of its sums does not
//    change, so that order is part of the result.
//
// Inference stores the activations between the layers as "split rows":
//  * a grid node is row r = guard + (x (Z + 1) + z) (Y + 1) + y;
//    one zero row after each y line, one zero line after each z plane, one
//    zero plane at the end and `guard` zero rows in front and behind
//    stand in for the zero padding, so every tap of every node is a fixed row
//    offset and needs no test;
//  * each FP32 value is the exact sum of three BF16 parts (hi, mid, lo: the 24
//    significand bits, split by truncation), kept in planes
//    [part][channel / 8][row][8]: 16 bytes per row, the K-major operand rows
//    of the tensor cores, which a bulk copy brings in as they are and whose
//    shift by a row is a shift of the operand's address by 16 bytes.
// Products of the parts with the BF16 weights are exact in FP32, so three
// BF16 MMAs give the FP32 convolution up to the order of its sums.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <functional>
#include <mutex>
#include <vector>

#include "gputo_internal.h"
#include "tma.h"

namespace gputo {

namespace {

__host__ __device__ constexpr int net_ch(int l) { return l == 0 ? 4 : l == 1 ? 16 : l == 2 ? 32 : l == 3 ? 64 : 3; }
__host__ __device__ constexpr int net_k(int l) { return l == 3 ? 1 : 3; }

__device__ __forceinline__ float bf16r(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

constexpr int kRows = 128;                       // rows of one tile (TMEM lanes)

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

// Geometry of the split rows.
struct RowGeo {
    int X, Z, Y;
    int py, pz;            // row offsets of dz = 1 and dx = 1
    long long rows;        // (X + 1) (Z + 1) (Y + 1)
    long long guard, R;    // zero rows in front; rows of a plane (a whole number of tiles, guards included)
    int ntiles;
};

RowGeo row_geo(const NetDims &d)
{
    RowGeo q;
    q.X = d.X, q.Z = d.Z, q.Y = d.Y;
    q.py = d.Y + 1;
    q.pz = (d.Z + 1) * (d.Y + 1);
    q.rows = (long long)(d.X + 1) * q.pz;
    q.guard = ((long long)q.pz + q.py + 1 + 7) / 8 * 8;
    q.ntiles = (int)((q.rows + kRows - 1) / kRows);
    q.R = 2 * q.guard + (long long)q.ntiles * kRows;
    return q;
}

// Row r (without the guard) -> node; false on padding rows.  In 32 bits: 2^31
// rows of the first layer alone (96 bytes each) would be 206 GB.
__device__ __forceinline__ bool row_node(const RowGeo &q, long long r, int &x, int &z, int &y)
{
    const uint32_t r32 = (uint32_t)r, line = r32 / (uint32_t)q.py;
    x = (int)(line / (uint32_t)(q.Z + 1));
    z = (int)(line - (uint32_t)x * (q.Z + 1));
    y = (int)(r32 - line * q.py);
    return x < q.X && z < q.Z && y < q.Y;
}

// Zeroes the guard rows of two sets of planes.
struct GuardSets {
    uint4 *p[2];
    int planes[2];
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

// The BF16 weight operands of the two tensor-core convolutions, as the
// shared-memory image [tap][ci / 8][co][8] that a CTA copies whole.
constexpr int kImg2 = 27 * 16 * 32, kImg3 = 27 * 32 * 64;   // elements

__global__ void __launch_bounds__(256)
pack_weights_kernel(const float *__restrict__ w2, const float *__restrict__ w3, __nv_bfloat16 *__restrict__ img)
{
    const int out = blockIdx.x * 256 + threadIdx.x;
    if (out >= kImg2 + kImg3) return;
    const bool second = out >= kImg2;
    const int i = second ? out - kImg2 : out, ci_n = second ? 32 : 16, co_n = second ? 64 : 32;
    const int e = i & 7, co = (i >> 3) % co_n, rest = (i >> 3) / co_n, ci = 8 * (rest % (ci_n / 8)) + e,
              tap = rest / (ci_n / 8);
    img[out] = __float2bfloat16_rn((second ? w3 : w2)[(co * ci_n + ci) * 27 + tap]);
}

// Layer 1 (4 -> 16): the 108 taps from the caller's dense input, weights
// broadcast from shared memory, output pairs on paired FP32 instructions;
// writes the split rows of its 16 channels (zeros on padding).  4 x 27 x 16
// FMAs per node are too few channels for the tensor cores.  A thread takes
// kC1R rows a CTA width apart, which share each weight read: with one row the
// kernel was bound by those reads (94 us at 129 x 65 x 65, 66 with two); four
// rows take too many registers and leave too few warps (72 us).  The taps are
// summed in blocks of nine: a chain of 108 roundings was half of the network's
// error, for 10 us more.
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
        int x, z, y;
        const bool in = row_node(q, r0 + 128 * k, x, z, y);
        xs[k] = in ? xin + ((size_t)x * q.Z + z) * q.Y + y : xin;
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
    EPI_HEAD = 1    // + bias, ReLU, then the 64 -> 3 head -> dense output
};

struct ConvArgs {
    const uint4 *a;          // input split rows, 3 K / 8 planes
    const uint4 *img;        // weight operand image
    const float *bias;
    uint4 *out;              // EPI_RELU: split rows, 3 N / 8 planes
    const float *w4, *b4;    // EPI_HEAD
    float *y;                // EPI_HEAD: dense output [3][n]
    int *err;                // set when a bounded wait gives up
    uint32_t wait_ns;        // how long that takes
    int skip_stage;          // ring stage whose copies are left unissued (test hook; -1: none)
};

// One convolution as an implicit GEMM: D[row][N] = sum over 27 taps, K input
// channels and 3 parts.  Per tile of 128 rows and (dx, dz) pair ("segment"),
// 130 rows of every plane are brought in by bulk copies; the three dy taps are
// the same rows shifted by one, i.e. operand addresses 16 bytes apart.
//
// Warp 4's first thread issues the copies, warp 5's first thread the MMAs,
// warps 0-3 add the segment sums from TMEM (double-buffered) into FP32
// registers and run the epilogue.  The tensor core's adds truncate, which
// shrinks every sum a little.  So a segment has four accumulators, the hi parts
// of each dy and the mid and lo parts of all: products of hi parts and weights
// have 16 bits, few of which are lost in the K / 16 adds of a chain, and the
// four sums are added with rounding.  With one accumulator per segment the
// output is low by 1.2e-7; now by 3e-8, and its error against 64 bits is 1.6e-7
// of the norm (4.1e-7 with FP32 FMA chains), for 10 % of the forward pass.
//
// Persistent, weights resident (110 KB for 32 x 64).  Copies, MMAs and drains
// overlap but share the shared memory and TMEM ports, and none of them alone
// is the bound: a forward pass at 129 x 65 x 65 takes 465 us, 384 with a third
// of the MMAs, 399 without drains and epilogue, 303 without both.  Of those 303
// about 76 are the first layer, the rest the nine reads of the activations
// (0.49 GB for 16 -> 32 and 0.98 GB for 32 -> 64).  Measured at 129 x 65 x 65:
// 32 -> 64 with the head 270 us (0.8 PFLOP/s of BF16 MMAs; 3167 + 50 us as
// direct FP32 convolutions on the CUDA cores), 16 -> 32 112 us (733 us).
template <int CK, int CN> struct ConvCfg {
    static constexpr int C8 = CK / 8;
    static constexpr int RS = kRows + 2;                    // rows of a segment
    static constexpr int STAGE = 3 * C8 * RS * 16;          // bytes
    static constexpr int BBYTES = 27 * CK * CN * 2;
    static constexpr int NST = 4;                           // stages
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
        if (!bad && !mbar_wait_for(b, parity, A.wait_ns)) {
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
                    if (s != A.skip_stage)
                        for (int pl = 0; pl < 3 * C::C8; ++pl)
                            bulk_load(dst + pl * (C::RS * 16), A.a + pl * q.R + row, C::RS * 16, &full[s]);
                    ++issued;
                }
            // copies in flight land before the CTA leaves, whichever warp's wait gave up
            mbar_wait_for(bbar, 0, A.wait_ns);
            for (int k = issued > C::NST ? issued - C::NST : 0; k < issued; ++k)
                mbar_wait_for(&full[k % C::NST], (uint32_t)((k / C::NST) & 1), A.wait_ns);
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
            // MMAs in flight end before TMEM is freed, whichever warp's wait gave up
            if (it > 0) mbar_wait_for(&tfull[(it - 1) & 1], (uint32_t)(((it - 1) / 2) & 1), A.wait_ns);
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
            int x, z, y;
            const bool in = row_node(q, r, x, z, y);
            if (EPI == EPI_HEAD) {
                float o3[3] = {hw[192], hw[193], hw[194]};
#pragma unroll
                for (int c = 0; c < CN; ++c) {
                    acc[c] = fmaxf(acc[c] + A.bias[c], 0.f);
#pragma unroll
                    for (int o = 0; o < 3; ++o) o3[o] = fmaf(hw[3 * c + o], acc[c], o3[o]);
                }
                if (in) {
                    const long long n = (long long)q.X * q.Z * q.Y, at = ((long long)x * q.Z + z) * q.Y + y;
#pragma unroll
                    for (int o = 0; o < 3; ++o) A.y[o * n + at] = o3[o];
                }
            } else {
#pragma unroll
                for (int c = 0; c < CN / 8; ++c) {
                    float v[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[e] = in ? fmaxf(acc[8 * c + e] + A.bias[8 * c + e], 0.f) : 0.f;
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

// ---------------------------------------------------------------------------
// Training: direct FP32 convolutions.  One thread per node computes a chunk of
// output channels, the chunk's weights sit in shared memory and every thread of
// a warp reads the same weight at the same time (broadcast), the input reads
// are coalesced along Y.  Weight gradients are reduced per (co, ci) pair by
// one CTA in a fixed order, so training is deterministic.  Bound by FP32 FMAs
// and, in the weight gradients, by their index arithmetic: eight 33^3 samples
// take 15.7 ms, of which the weight gradients 8.6, the data gradients 3.8 and
// the forward passes 2.4 ms.  (On the tensor cores a step took 1.4 ms, but its
// sums differ in their last bits, and with them every later step.)
// ---------------------------------------------------------------------------
constexpr int kNetThreads = 128;

// Offset of tap t of a 3x3x3 stencil, and whether it stays inside the grid.
__device__ __forceinline__ bool tap_in(int t, int xi, int zi, int yi, const NetDims &d, long long &off)
{
    const int dx = t / 9 - 1, dz = (t / 3) % 3 - 1, dy = t % 3 - 1;
    off = ((long long)dx * d.Z + dz) * d.Y + dy;
    return (unsigned)(xi + dx) < (unsigned)d.X && (unsigned)(zi + dz) < (unsigned)d.Z && (unsigned)(yi + dy) < (unsigned)d.Y;
}

template <int CIN, int COT, int K, bool RELU>
__global__ void __launch_bounds__(kNetThreads)
conv_fwd_kernel(const float *__restrict__ x, const float *__restrict__ w, const float *__restrict__ b,
                float *__restrict__ y, NetDims d, int cout)
{
    constexpr int K3 = K * K * K;
    extern __shared__ float ws[];   // [CIN][K3][COT], BF16-rounded
    const int co0 = blockIdx.y * COT;
    for (int idx = threadIdx.x; idx < CIN * K3 * COT; idx += blockDim.x) {
        const int c = idx % COT, rest = idx / COT, t = rest % K3, ci = rest / K3;
        const int co = co0 + c;
        ws[idx] = co < cout ? bf16r(w[((long long)co * CIN + ci) * K3 + t]) : 0.f;
    }
    __syncthreads();
    const long long N = d.n();
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N) return;
    const int yi = (int)(n % d.Y);
    const long long r = n / d.Y;
    const int zi = (int)(r % d.Z), xi = (int)(r / d.Z);
    float acc[COT];
#pragma unroll
    for (int c = 0; c < COT; ++c) acc[c] = co0 + c < cout ? b[co0 + c] : 0.f;
    for (int ci = 0; ci < CIN; ++ci) {
        const float *xc = x + (long long)ci * N;
#pragma unroll
        for (int t = 0; t < K3; ++t) {
            long long off = 0;
            const bool in = K == 1 ? true : tap_in(t, xi, zi, yi, d, off);
            const float v = in ? xc[n + off] : 0.f;
            const float *wr = ws + (ci * K3 + t) * COT;
#pragma unroll
            for (int c = 0; c < COT; ++c) acc[c] = fmaf(wr[c], v, acc[c]);
        }
    }
#pragma unroll
    for (int c = 0; c < COT; ++c)
        if (co0 + c < cout) y[(long long)(co0 + c) * N + n] = RELU ? fmaxf(acc[c], 0.f) : acc[c];
}

// gx[ci](n) = sum_co sum_tap w[co][ci][tap] g[co](n - offset(tap))
template <int COUT, int CIT, int K>
__global__ void __launch_bounds__(kNetThreads)
conv_bwd_data_kernel(const float *__restrict__ g, const float *__restrict__ w, float *__restrict__ gx, NetDims d,
                     int cin)
{
    constexpr int K3 = K * K * K;
    extern __shared__ float ws[];   // [COUT][K3][CIT]
    const int ci0 = blockIdx.y * CIT;
    for (int idx = threadIdx.x; idx < COUT * K3 * CIT; idx += blockDim.x) {
        const int c = idx % CIT, rest = idx / CIT, t = rest % K3, co = rest / K3;
        const int ci = ci0 + c;
        ws[idx] = ci < cin ? bf16r(w[((long long)co * cin + ci) * K3 + t]) : 0.f;
    }
    __syncthreads();
    const long long N = d.n();
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N) return;
    const int yi = (int)(n % d.Y);
    const long long r = n / d.Y;
    const int zi = (int)(r % d.Z), xi = (int)(r / d.Z);
    float acc[CIT];
#pragma unroll
    for (int c = 0; c < CIT; ++c) acc[c] = 0.f;
    for (int co = 0; co < COUT; ++co) {
        const float *gc = g + (long long)co * N;
#pragma unroll
        for (int t = 0; t < K3; ++t) {
            long long off = 0;
            // output node n - offset(t): the mirrored tap of n
            const bool in = K == 1 ? true : tap_in(K3 - 1 - t, xi, zi, yi, d, off);
            const float v = in ? gc[n + off] : 0.f;
            const float *wr = ws + (co * K3 + t) * CIT;
#pragma unroll
            for (int c = 0; c < CIT; ++c) acc[c] = fmaf(wr[c], v, acc[c]);
        }
    }
#pragma unroll
    for (int c = 0; c < CIT; ++c)
        if (ci0 + c < cin) gx[(long long)(ci0 + c) * N + n] = acc[c];
}

// gw[co][ci][tap] += sum_n g[co](n) x[ci](n + offset(tap)): one CTA per (co, ci)
template <int K>
__global__ void __launch_bounds__(256)
conv_bwd_weight_kernel(const float *__restrict__ g, const float *__restrict__ x, float *__restrict__ gw, NetDims d,
                       int cin)
{
    constexpr int K3 = K * K * K;
    const int co = blockIdx.x / cin, ci = blockIdx.x % cin;
    const long long N = d.n();
    const float *gc = g + (long long)co * N, *xc = x + (long long)ci * N;
    float acc[K3];
#pragma unroll
    for (int t = 0; t < K3; ++t) acc[t] = 0.f;
    for (long long n = threadIdx.x; n < N; n += blockDim.x) {
        const float gv = gc[n];
        if (gv == 0.f) continue;
        const int yi = (int)(n % d.Y);
        const long long r = n / d.Y;
        const int zi = (int)(r % d.Z), xi = (int)(r / d.Z);
#pragma unroll
        for (int t = 0; t < K3; ++t) {
            long long off = 0;
            const bool in = K == 1 ? true : tap_in(t, xi, zi, yi, d, off);
            if (in) acc[t] = fmaf(gv, xc[n + off], acc[t]);
        }
    }
    __shared__ float red[8][K3];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int t = 0; t < K3; ++t) {
        float v = acc[t];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) red[wid][t] = v;
    }
    __syncthreads();
    if (threadIdx.x < K3) {
        float s = 0.f;
        for (int q = 0; q < 8; ++q) s += red[q][threadIdx.x];
        gw[((long long)co * cin + ci) * K3 + threadIdx.x] += s;
    }
}

// gb[co] += sum_n g[co](n)
__global__ void __launch_bounds__(256) bias_grad_kernel(const float *__restrict__ g, float *__restrict__ gb, NetDims d)
{
    const long long N = d.n();
    const float *gc = g + (long long)blockIdx.x * N;
    float v = 0.f;
    for (long long n = threadIdx.x; n < N; n += blockDim.x) v += gc[n];
    __shared__ float red[8];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        float s = 0.f;
        for (int q = 0; q < 8; ++q) s += red[q];
        gb[blockIdx.x] += s;
    }
}

// g <- g where the layer's ReLU output is positive, else 0
__global__ void relu_mask_kernel(float *__restrict__ g, const float *__restrict__ y, long long n)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && !(y[i] > 0.f)) g[i] = 0.f;
}

// Masked mean square error of one sample: partial sums per CTA, then a
// single-CTA finish that also writes the gradient scale; fixed order.
__global__ void __launch_bounds__(256)
mse_partial_kernel(const float *__restrict__ y, const float *__restrict__ t, const float *__restrict__ m, long long n,
                   double *__restrict__ part)
{
    double s = 0.0, c = 0.0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double r = (double)y[i] - (double)t[i];
        s += (double)m[i] * r * r;
        c += (double)m[i];
    }
    __shared__ double rs[8], rc[8];
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        c += __shfl_xor_sync(0xffffffffu, c, o);
    }
    if ((threadIdx.x & 31) == 0) rs[threadIdx.x >> 5] = s, rc[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int q = 0; q < 8; ++q) a += rs[q], b += rc[q];
        part[2 * blockIdx.x] = a;
        part[2 * blockIdx.x + 1] = b;
    }
}

__global__ void mse_finish_kernel(const double *__restrict__ part, int nb, double *__restrict__ loss_acc,
                                  float *__restrict__ gscale)
{
    if (threadIdx.x != 0) return;
    double a = 0.0, b = 0.0;
    for (int q = 0; q < nb; ++q) a += part[2 * q], b += part[2 * q + 1];
    const double den = b > 1.0 ? b : 1.0;
    *loss_acc += a / den;
    *gscale = (float)(2.0 / den);
}

__global__ void mse_grad_kernel(const float *__restrict__ y, const float *__restrict__ t, const float *__restrict__ m,
                                long long n, const float *__restrict__ gscale, float *__restrict__ g)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) g[i] = *gscale * m[i] * (y[i] - t[i]);
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

// Persistent grids: CTAs per SM by shared memory (two of 16 -> 32, one of 32 -> 64).
template <int CK, int CN, int EPI>
void launch_conv(const ConvArgs &a, const RowGeo &q, int sms, cudaStream_t st)
{
    using C = ConvCfg<CK, CN>;
    const int per = C::SMEM <= 113 * 1024 ? 2 : 1;
    conv_tc_kernel<CK, CN, EPI><<<std::min(q.ntiles, per * sms), 192, C::SMEM, st>>>(a, q);
    count_launches(1);
}

template <int CIN, int COT, int K, bool RELU>
void launch_fwd(const float *x, const float *w, const float *b, float *y, const NetDims &d, int cout, cudaStream_t st)
{
    constexpr int K3 = K * K * K;
    const size_t smem = sizeof(float) * CIN * K3 * COT;
    const dim3 grid((unsigned)((d.n() + kNetThreads - 1) / kNetThreads), (unsigned)((cout + COT - 1) / COT));
    conv_fwd_kernel<CIN, COT, K, RELU><<<grid, kNetThreads, smem, st>>>(x, w, b, y, d, cout);
    count_launches(1);
}

template <int COUT, int CIT, int K>
void launch_bwd_data(const float *g, const float *w, float *gx, const NetDims &d, int cin, cudaStream_t st)
{
    constexpr int K3 = K * K * K;
    const size_t smem = sizeof(float) * COUT * K3 * CIT;
    const dim3 grid((unsigned)((d.n() + kNetThreads - 1) / kNetThreads), (unsigned)((cin + CIT - 1) / CIT));
    conv_bwd_data_kernel<COUT, CIT, K><<<grid, kNetThreads, smem, st>>>(g, w, gx, d, cin);
    count_launches(1);
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
    for (int l = 1; l <= 4; ++l) cudaFree(act[l]);
    cudaFree(gA);
    cudaFree(gB);
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
    GPUTO_CUDA(cudaMalloc(&part, sizeof(double) * (kNetPart + 1) + sizeof(float)));
    owned.push_back(part);
    loss_acc = part + kNetPart;   // part: kNetPart doubles of reduction scratch
    gscale = reinterpret_cast<float *>(loss_acc + 1);
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

// Mapped host flags for the bounded waits.  Allocating mapped memory takes 1 to
// 3 ms, more than the rest of a small network's first pass, so one page serves
// the process: a slot per NetWork, given back with it, and memory of its own
// for those that find no slot.
namespace {
struct FlagPage {
    static constexpr int kSlots = 1024;
    std::mutex mu;
    int *page = nullptr;
    std::vector<int *> free;

    int *take()
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!page) {
            if (cudaHostAlloc((void **)&page, kSlots * sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable) !=
                cudaSuccess) {
                page = nullptr;
                return nullptr;
            }
            for (int i = kSlots; i-- > 0;) free.push_back(page + i);
        }
        int *f = nullptr;
        if (!free.empty()) {
            f = free.back();
            free.pop_back();
        } else if (cudaHostAlloc((void **)&f, sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
            return nullptr;
        }
        *f = 0;
        return f;
    }
    void give_back(int *f)
    {
        std::lock_guard<std::mutex> lock(mu);
        if (std::less_equal<int *>()(page, f) && std::less<int *>()(f, page + kSlots)) free.push_back(f);
        else cudaFreeHost(f);
    }
};

FlagPage &flag_page()
{
    static FlagPage *p = new FlagPage;   // outlives every network
    return *p;
}
}  // namespace

void NetWork::release()
{
    cudaFree(img);   // waits for kernels that may still write the flag
    if (h_err) flag_page().give_back(h_err);
    img = nullptr;
    rows1 = rows2 = nullptr;
    h_err = d_err = nullptr;
    cap_rows = 0;
}

int NetWork::reserve(const NetDims &d)
{
    if (!h_err) {
        // where a kernel's bounded wait reports that it gave up: read by the host after a synchronisation
        h_err = flag_page().take();
        if (!h_err) GPUTO_CUDA(cudaErrorMemoryAllocation);
        GPUTO_CUDA(cudaHostGetDevicePointer((void **)&d_err, h_err, 0));
    }
    const long long rows = row_geo(d).R;
    if (rows <= cap_rows) return GPUTO_OK;
    cudaFree(img);
    img = nullptr;
    rows1 = rows2 = nullptr;
    cap_rows = 0;
    constexpr size_t wbytes = 2 * (size_t)(kImg2 + kImg3);
    static_assert(wbytes % 256 == 0, "the rows behind it start as aligned as the allocation");
    GPUTO_CUDA(cudaMalloc(&img, wbytes + 16 * 18 * (size_t)rows));
    rows1 = reinterpret_cast<uint4 *>((char *)img + wbytes);
    rows2 = rows1 + 6 * rows;
    cap_rows = rows;
    return GPUTO_OK;
}

int Net::reserve_train(long long n)
{
    if (n <= cap_n) return GPUTO_OK;
    for (int l = 1; l <= 4; ++l) cudaFree(act[l]), act[l] = nullptr;
    cudaFree(gA), cudaFree(gB);
    gA = gB = nullptr;
    cap_n = 0;
    for (int l = 1; l <= 4; ++l) GPUTO_CUDA(cudaMalloc(&act[l], sizeof(float) * net_ch(l) * n));
    GPUTO_CUDA(cudaMalloc(&gA, sizeof(float) * 64 * n));
    GPUTO_CUDA(cudaMalloc(&gB, sizeof(float) * 64 * n));
    cap_n = n;
    return GPUTO_OK;
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
    GPUTO_CUDA(set(conv_fwd_kernel<32, 16, 3, true>, 32 * 27 * 16 * 4));
    GPUTO_CUDA(set(conv_bwd_data_kernel<64, 16, 3>, 64 * 27 * 16 * 4));
    GPUTO_CUDA(set(conv_bwd_data_kernel<32, 16, 3>, 32 * 27 * 16 * 4));
    if (dev < 64) done[dev] = true;
    return GPUTO_OK;
}

int NetWork::check()
{
    if (!h_err || !*(volatile int *)h_err) return GPUTO_OK;
    const int e = *(volatile int *)h_err;
    *(volatile int *)h_err = 0;
    set_error("a bounded wait of the network's convolution gave up");
    return e;
}

int Net::forward(NetWork &w, const float *x, const NetDims &d, float *y, cudaStream_t st) const
{
    const RowGeo q = row_geo(d);
    if (q.R > w.cap_rows) return GPUTO_ERR_ARG;
    const float *p = params;
    GuardSets gs{{w.rows1, w.rows2}, {6, 12}};
    zero_guards_kernel<<<dim3(64, 2), 256, 0, st>>>(gs, q);
    pack_weights_kernel<<<(kImg2 + kImg3 + 255) / 256, 256, 0, st>>>(p + param_offset(1, false), p + param_offset(2, false),
                                                                    (__nv_bfloat16 *)w.img);
    conv1_kernel<<<(q.ntiles + kC1R - 1) / kC1R, 128, 0, st>>>(x, p + param_offset(0, false), p + param_offset(0, true),
                                                               w.rows1, q);
    count_launches(3);
    const uint4 *im = reinterpret_cast<const uint4 *>(w.img);
    ConvArgs a{};
    a.err = w.d_err;
    const SweepFaultHook hook = sweep_fault_hook();
    a.wait_ns = hook.wait_ns;
    a.skip_stage = hook.skip_stage;
    a.a = w.rows1;
    a.img = im;
    a.bias = p + param_offset(1, true);
    a.out = w.rows2;
    launch_conv<16, 32, EPI_RELU>(a, q, sms, st);
    a.a = w.rows2;
    a.img = im + kImg2 / 8;
    a.bias = p + param_offset(2, true);
    a.out = nullptr;
    a.w4 = p + param_offset(3, false);
    a.b4 = p + param_offset(3, true);
    a.y = y;
    launch_conv<32, 64, EPI_HEAD>(a, q, sms, st);
    return GPUTO_OK;
}

int Net::train_forward(const float *x, const NetDims &d, cudaStream_t st)
{
    int s = reserve_train(d.n());
    if (s) return s;
    act[0] = const_cast<float *>(x);
    const float *p = params;
    launch_fwd<4, 16, 3, true>(x, p + param_offset(0, false), p + param_offset(0, true), act[1], d, 16, st);
    launch_fwd<16, 16, 3, true>(act[1], p + param_offset(1, false), p + param_offset(1, true), act[2], d, 32, st);
    launch_fwd<32, 16, 3, true>(act[2], p + param_offset(2, false), p + param_offset(2, true), act[3], d, 64, st);
    launch_fwd<64, 3, 1, false>(act[3], p + param_offset(3, false), p + param_offset(3, true), act[4], d, 3, st);
    return GPUTO_OK;
}

// Loss of one sample (x, target t, mask m) added to loss_acc, gradients
// added to grads.
int Net::accumulate(const float *x, const float *t, const float *m, const NetDims &d, cudaStream_t st)
{
    int s = train_forward(x, d, st);
    if (s) return s;
    const long long N = d.n(), n3 = 3 * N;
    const int nb = (int)std::min<long long>(kNetPart / 2, (n3 + 255) / 256);
    mse_partial_kernel<<<nb, 256, 0, st>>>(act[4], t, m, n3, part);
    mse_finish_kernel<<<1, 32, 0, st>>>(part, nb, loss_acc, gscale);
    mse_grad_kernel<<<(unsigned)((n3 + 255) / 256), 256, 0, st>>>(act[4], t, m, n3, gscale, gA);
    count_launches(3);
    return backward_from(d, st);
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

// Backward pass of the last training forward from the output gradient in gA; adds to grads.
int Net::backward_from(const NetDims &d, cudaStream_t st)
{
    const long long N = d.n();
    float *g = gA, *gn = gB;
    for (int l = 3; l >= 0; --l) {
        const int cin = net_ch(l), cout = net_ch(l + 1);
        float *gw = grads + param_offset(l, false), *gb = grads + param_offset(l, true);
        if (l < 3) {
            relu_mask_kernel<<<(unsigned)((cout * N + 255) / 256), 256, 0, st>>>(g, act[l + 1], cout * N);
            count_launches(1);
        }
        if (net_k(l) == 3)
            conv_bwd_weight_kernel<3><<<cout * cin, 256, 0, st>>>(g, act[l], gw, d, cin);
        else
            conv_bwd_weight_kernel<1><<<cout * cin, 256, 0, st>>>(g, act[l], gw, d, cin);
        bias_grad_kernel<<<cout, 256, 0, st>>>(g, gb, d);
        count_launches(2);
        if (l == 0) break;
        const float *w = params + param_offset(l, false);
        switch (l) {
        case 3: launch_bwd_data<3, 16, 1>(g, w, gn, d, 64, st); break;
        case 2: launch_bwd_data<64, 16, 3>(g, w, gn, d, 32, st); break;
        default: launch_bwd_data<32, 16, 3>(g, w, gn, d, 16, st); break;
        }
        std::swap(g, gn);
    }
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
