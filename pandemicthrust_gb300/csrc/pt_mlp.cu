// pt_mlp.cu - the surrogate's multilayer perceptron: BF16 weights and activations,
// FP32 accumulation, FP32 master weights and Adam, all in hand-written kernels.
//
// Layers l = 0..L-1 map width[l] -> width[l+1]; hidden layers apply GELU, the last
// is linear.  Parameters live in one FP32 array, layer by layer: W_l (width[l+1] x
// width[l], row-major) then b_l (width[l+1]); a BF16 copy of every weight feeds the
// tensor cores.  The library owns all device memory; callers pass host arrays.
//
// Training GEMMs are small (a minibatch of a few hundred rows by 256) and need
// transposed operands, so they run on the warp-level tensor-core instruction mma.sync
// (k_gemm below).  Inference over large batches runs every layer on tcgen05.mma.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <numeric>
#include <random>
#include <string>
#include <vector>

#include "pandemic_gb300.h"
#include "pt_mapped.h"

namespace {

typedef __nv_bfloat16 bf16;

// The activation: GELU in its tanh form (Hendrycks and Gimpel, arXiv:1606.08415),
// 0.5 z (1 + tanh(u)), u = sqrt(2/pi) (z + 0.044715 z^3), with the hardware tanh
// (tanh.approx.f32).  Training and inference evaluate the same expression.
constexpr float kGeluC0 = 0.7978845608028654f;               // sqrt(2 / pi)
constexpr float kGeluC1 = 0.7978845608028654f * 0.044715f;   // sqrt(2 / pi) * 0.044715

__device__ __forceinline__ float tanh_approx(float x)
{
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// rounded step by step as the tcgen05 epilogue's paired form (gelu_bf16x2):
// w = c0 + c1 z^2, t = tanh(w z), h = z / 2, h + h t
__device__ __forceinline__ float gelu(float z)
{
    const float w = __fmaf_rn(__fmul_rn(z, z), kGeluC1, kGeluC0);
    const float t = tanh_approx(__fmul_rn(w, z));
    const float h = __fmul_rn(0.5f, z);
    return __fmaf_rn(h, t, h);
}

__device__ __forceinline__ float gelu_grad(float z)
{
    // d/dz [0.5 z (1 + t)] = 0.5 (1 + t) + 0.5 z (1 - t^2) du/dz, du/dz = c0 + 3 c1 z^2
    const float z2 = z * z;
    const float t = tanh_approx(z * (kGeluC0 + kGeluC1 * z2));
    return 0.5f * (1.f + t) + 0.5f * z * (1.f - t * t) * (kGeluC0 + 3.f * kGeluC1 * z2);
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---------------------------------------------------------------- training GEMMs
// A training step is a chain of small GEMMs (a batch of a few hundred rows by a few
// hundred columns, a microsecond of work each), so what counts is how many launches
// the chain has, how long one takes from its first load to its last store, and that
// every SM has a part.  Hence: 32 x 32 output tiles (128 blocks for 512 x 256), the
// whole reduction of 256 in flight at once (four cp.async stages of 64), operands read
// by ldmatrix in either order, everything elementwise in the epilogues (bias, GELU and
// its derivative, the loss, Adam; their inputs are read before the products start), and
// independent GEMMs of a step in one launch.  A step of the 11-4x256-222 network at
// batch 512 is 10 launches instead of 23 and takes 82 us on a GB300 instead of 640
// (100 with programmatic dependent launches: the next launch's blocks get in the way).
//
// Products run on mma.sync m16n8k16 (BF16 in, FP32 accumulate), the reduction in
// ascending steps of 16 into one accumulator, whatever the tiling.
constexpr int kGemmThreads = 128, kGemmTile = 32, kGemmK = 64, kGemmStages = 4;
constexpr int kGemmPitchK = (kGemmK + 8) * 2, kGemmPitchN = (kGemmTile + 8) * 2;   // bytes; odd multiples of 16
constexpr int kGemmOperand = kGemmK * kGemmPitchN;   // one stage of one operand in either order (>= 32 x pitch K)
static_assert(kGemmTile * kGemmPitchK <= kGemmOperand, "a stage holds an operand tile in both orders");
constexpr int kGemmSmem = kGemmStages * 2 * kGemmOperand;
constexpr int kBiasCols = 16, kBiasRows = 512;   // a bias block: columns, rows staged at once
static_assert(kBiasCols * kBiasRows * 4 <= kGemmSmem, "the bias sums stage their rows in the same shared memory");

// Adam's state of a layer's parameters, for the updates in the epilogues.
struct AdamArgs {
    float *w, *m, *v;   // FP32 parameters and moments, all layers
    float lr, c1, c2;   // c1, c2: the bias corrections of the step
};

// Adam (Kingma and Ba, 2015) for parameter i with gradient gr and its values before the
// step (w, m, v): stores the new ones, returns the new parameter.
__device__ __forceinline__ float adam_step(const AdamArgs &a, long long i, float gr, float w, float m, float v)
{
    constexpr float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float mi = b1 * m + (1.f - b1) * gr;
    const float vi = b2 * v + (1.f - b2) * gr * gr;
    a.m[i] = mi;
    a.v[i] = vi;
    const float wi = w - a.lr * (mi / a.c1) / (sqrtf(vi / a.c2) + eps);
    a.w[i] = wi;
    return wi;
}

enum GemmKind {
    kOpNone = 0,
    kOpForward,   // z = H W^T + b; Z = z, next H = act(z) (BF16)
    kOpOutput,    // z = H W^T + b; Z = z
    kOpLoss,      // z = H W^T + b; dz = 2 (z - y) / (rows x columns), the loss summed
    kOpBackward,  // dz' = (dZ W) GELU'(Z')
    kOpWeights,   // g = dZ^T H: the gradient, or Adam's update with it
    kOpBias       // g = column sums of dZ: likewise
};

// One GEMM (or bias sum) of a launch.  A, B: BF16, row strides lda / ldb multiples of 16,
// columns from the true width to the stride zero.
struct GemmOp {
    int kind, blocks;     // thread blocks of the op
    int M, N, R;          // output rows and columns, terms of the reduction
    const bf16 *A, *B;
    int lda, ldb;
    int Brows;            // rows of B in memory (weights: padded with zero rows)
    const float *bias;
    float *Z;             // forward: pre-activations out; backward: those of the layer before, in
    int ldz;
    bf16 *H;              // forward: next activations, row stride ldh
    int ldh;
    float *dZf;           // dz in FP32 (row stride ldd) and BF16
    bf16 *dZb;
    int ldd;
    const float *Y;       // loss: targets, rows by `rows` (nullptr: in order)
    const int *rows;
    float *loss;
    long long param;      // weights / bias: index of the first parameter
    float *grad;          // the gradient array, or nullptr: update the parameters
    bf16 *wpk;            // padded BF16 weights (row stride ldw) refreshed by the update
    int ldw;
};

constexpr int kMaxOps = 16;
struct GemmLaunch {
    GemmOp op[kMaxOps];
    AdamArgs adam;
};

__device__ __forceinline__ void mma_bf16(float d[4], const uint32_t a[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <bool TRANS>
__device__ __forceinline__ void ldmatrix4(uint32_t r[4], uint32_t addr)
{
    if (TRANS)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
    else
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

// 16 bytes to shared memory, or zeros
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool valid)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

// A stage of an operand.  KMAJOR: rows mn0 .. mn0 + 31 of the matrix, columns k0 .. k0 + 63
// (the reduction runs along rows); else rows k0 .. k0 + 63, columns mn0 .. mn0 + 31.  Rows from
// `rows` on and columns from `ld` on read as zeros.
template <bool KMAJOR>
__device__ __forceinline__ void load_operand(uint32_t dst, const bf16 *src, int ld, int rows, int mn0, int k0)
{
    constexpr int kChunks = (KMAJOR ? kGemmK : kGemmTile) / 8;   // 16-byte pieces of a row
#pragma unroll
    for (int i = 0; i < kGemmTile * kGemmK / 8 / kGemmThreads; i++) {
        const int e = (int)threadIdx.x + i * kGemmThreads, r = e / kChunks, c = (e % kChunks) * 8;
        const int row = (KMAJOR ? mn0 : k0) + r, col = (KMAJOR ? k0 : mn0) + c;
        const bool ok = row < rows && col < ld;
        cp_async16(dst + r * (KMAJOR ? kGemmPitchK : kGemmPitchN) + c * 2, ok ? src + (long long)row * ld + col : src, ok);
    }
}

// acc(i, j) of the block's 32 x 32 tile at (bm, bn); warp w has rows 16 (w / 2), columns
// 16 (w % 2) of it: acc[0] columns 0-7, acc[1] columns 8-15.
template <bool A_KMAJOR, bool B_KMAJOR>
__device__ __forceinline__ void gemm_tile(const GemmOp &g, int a_rows, int b_rows, int bm, int bn, uint32_t smem,
                                          float acc[2][4])
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = (warp >> 1) * 16, wn = (warp & 1) * 16;
    const int steps = (g.R + 15) / 16, chunks = (g.R + kGemmK - 1) / kGemmK;
#pragma unroll
    for (int q = 0; q < 4; q++) acc[0][q] = acc[1][q] = 0.f;
    auto load = [&](int c) {
        const uint32_t d = smem + (c % kGemmStages) * 2 * kGemmOperand;
        load_operand<A_KMAJOR>(d, g.A, g.lda, a_rows, bm, c * kGemmK);
        load_operand<B_KMAJOR>(d + kGemmOperand, g.B, g.ldb, b_rows, bn, c * kGemmK);
    };
    // one commit group a chunk (empty past the end), so the waits below count alike
#pragma unroll
    for (int c = 0; c < kGemmStages - 1; c++) {
        if (c < chunks) load(c);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const int l7 = lane & 7, l8 = (lane >> 3) & 1, l16 = lane >> 4;
    for (int c = 0; c < chunks; c++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kGemmStages - 2) : "memory");
        __syncthreads();   // chunk c has landed for every thread, and chunk c - 1 is used up
        if (c + kGemmStages - 1 < chunks) load(c + kGemmStages - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const uint32_t sa = smem + (c % kGemmStages) * 2 * kGemmOperand, sb = sa + kGemmOperand;
        const int n = min(kGemmK / 16, steps - c * (kGemmK / 16));
#pragma unroll
        for (int k = 0; k < kGemmK / 16; k++) {
            if (k < n) {
                uint32_t a[4], b[4];
                if (A_KMAJOR) ldmatrix4<false>(a, sa + (wm + l7 + 8 * l8) * kGemmPitchK + (16 * k + 8 * l16) * 2);
                else ldmatrix4<true>(a, sa + (16 * k + l7 + 8 * l16) * kGemmPitchN + (wm + 8 * l8) * 2);
                if (B_KMAJOR) ldmatrix4<false>(b, sb + (wn + l7 + 8 * l16) * kGemmPitchK + (16 * k + 8 * l8) * 2);
                else ldmatrix4<true>(b, sb + (16 * k + l7 + 8 * l8) * kGemmPitchN + (wn + 8 * l16) * 2);
                mma_bf16(acc[0], a, b[0], b[1]);
                mma_bf16(acc[1], a, b[2], b[3]);
            }
        }
    }
}

// Column sums of dZ in row order: the block's rows staged in shared memory, then one
// thread a column adds them.
__device__ __forceinline__ void bias_block(const GemmOp &g, const AdamArgs &adam, int block, float *stage)
{
    const int j0 = block * kBiasCols, t = threadIdx.x;
    const bool mine = t < kBiasCols && j0 + t < g.N;
    const long long p = g.param + j0 + t;
    float s = 0.f, w = 0.f, mm = 0.f, v = 0.f;
    if (mine && !g.grad) {
        w = adam.w[p];
        mm = adam.m[p];
        v = adam.v[p];
    }
    for (int i0 = 0; i0 < g.M; i0 += kBiasRows) {
        const int rows = min(kBiasRows, g.M - i0);
        for (int e = t; e < rows * (kBiasCols / 4); e += kGemmThreads) {
            const int r = e / (kBiasCols / 4), c = e % (kBiasCols / 4) * 4;
            cp_async16(smem_u32(stage + r * kBiasCols + c), g.dZf + (long long)(i0 + r) * g.ldd + j0 + c, true);
        }
        asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (t < kBiasCols) {
#pragma unroll 32
            for (int r = 0; r < rows; r++) s += stage[r * kBiasCols + t];
        }
        __syncthreads();
    }
    if (mine) {
        if (g.grad) g.grad[p] = s;
        else adam_step(adam, p, s, w, mm, v);
    }
}

__global__ void __launch_bounds__(kGemmThreads) k_gemm(const __grid_constant__ GemmLaunch l)
{
    __shared__ __align__(16) uint8_t smem[kGemmSmem];
    int block = blockIdx.x, o = 0;
    while (block >= l.op[o].blocks) block -= l.op[o++].blocks;
    const GemmOp &g = l.op[o];
    if (g.kind == kOpBias) {
        bias_block(g, l.adam, block, reinterpret_cast<float *>(smem));
        return;
    }
    const int nb = (g.N + kGemmTile - 1) / kGemmTile;
    const int bm = block / nb * kGemmTile, bn = block % nb * kGemmTile;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i0 = bm + (warp >> 1) * 16 + (lane >> 2), j0 = bn + (warp & 1) * 16 + 2 * (lane & 3);
    // what the epilogue reads of its eight outputs, on its way while the products run
    // (output e: row i0 + 8 ((e / 2) % 2), column j0 + 8 (e / 4) + e % 2)
    float x0[8], x1[8], x2[8];
#pragma unroll
    for (int e = 0; e < 8; e++) {
        const int i = i0 + 8 * ((e >> 1) & 1), j = j0 + 8 * (e >> 2) + (e & 1);
        x0[e] = x1[e] = x2[e] = 0.f;
        if (i >= g.M || j >= g.N) continue;
        if (g.kind == kOpBackward) {
            x0[e] = g.Z[(long long)i * g.ldz + j];
        } else if (g.kind == kOpWeights) {
            if (!g.grad) {
                const long long p = g.param + (long long)i * g.N + j;
                x0[e] = l.adam.w[p];
                x1[e] = l.adam.m[p];
                x2[e] = l.adam.v[p];
            }
        } else {
            x0[e] = g.bias[j];
            if (g.kind == kOpLoss) x1[e] = g.Y[(g.rows ? (long long)g.rows[i] : i) * g.N + j];
        }
    }
    float acc[2][4];
    if (g.kind == kOpWeights) gemm_tile<false, false>(g, g.R, g.R, bm, bn, smem_u32(smem), acc);
    else if (g.kind == kOpBackward) gemm_tile<true, false>(g, g.M, g.Brows, bm, bn, smem_u32(smem), acc);
    else gemm_tile<true, true>(g, g.M, g.Brows, bm, bn, smem_u32(smem), acc);
    const float scale = 2.f / (float)((long long)g.M * g.N);
    float part = 0.f;
#pragma unroll
    for (int e = 0; e < 8; e++) {
        const int i = i0 + 8 * ((e >> 1) & 1), j = j0 + 8 * (e >> 2) + (e & 1);
        if (i >= g.M || j >= g.N) continue;
        const float v = acc[e >> 2][e & 3];
        if (g.kind == kOpForward) {
            const float z = v + x0[e];
            g.Z[(long long)i * g.ldz + j] = z;
            g.H[(long long)i * g.ldh + j] = __float2bfloat16(gelu(z));
        } else if (g.kind == kOpOutput) {
            g.Z[(long long)i * g.ldz + j] = v + x0[e];
        } else if (g.kind == kOpLoss) {
            const float d = v + x0[e] - x1[e];
            part += d * d;
            g.dZf[(long long)i * g.ldd + j] = scale * d;
            g.dZb[(long long)i * g.ldd + j] = __float2bfloat16(scale * d);
        } else if (g.kind == kOpBackward) {
            const float dz = v * gelu_grad(x0[e]);
            g.dZf[(long long)i * g.ldd + j] = dz;
            g.dZb[(long long)i * g.ldd + j] = __float2bfloat16(dz);
        } else {
            const long long p = g.param + (long long)i * g.N + j;
            if (g.grad) g.grad[p] = v;
            else g.wpk[(long long)i * g.ldw + j] = __float2bfloat16(adam_step(l.adam, p, v, x0[e], x1[e], x2[e]));
        }
    }
    if (g.kind == kOpLoss) {
#pragma unroll
        for (int o2 = 16; o2 > 0; o2 >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o2);
        if (lane == 0) atomicAdd(g.loss, part / (float)((long long)g.M * g.N));
    }
}

// ---------------------------------------------------------------- tcgen05 inference
// Forward layers for inference on the fifth-generation tensor cores.  One persistent
// CTA per SM, in three roles:
//   warp 0 (one lane), the producer: loads the layer's weights (Np x Kp BF16, at most
//     256 x 256 = 128 KB) once, then streams 128-row tiles of the input through a ring
//     of kUmmaStages shared-memory stages (up to 128 K columns each) with TMA
//     (cp.async.bulk.tensor), each stage completing on its `full` mbarrier;
//   warp 1 (one lane), the MMA issuer: per tile it waits for a free accumulator (two
//     128 x 256 FP32 accumulators in tensor memory, all 512 columns), then per stage
//     waits for `full`, issues tcgen05.mma (kind::f16, K = 16 each) and commits the
//     stage back to the producer (`empty`); the tile's last commit goes to the
//     epilogue (`acc_full`);
//   the epilogue warps: read the accumulator with tcgen05.ld.32x32b (warp w reads
//     lanes, i.e. tile rows, 32 (w % 4) .. + 31), add the bias, apply GELU, store,
//     and release the accumulator (`acc_empty`).
// So the fill of tile i + 1, its MMAs and the epilogue of tile i overlap.  Every wait
// is bounded: one that gives up sets the error word and a shared flag that ends every
// role's loop; the MMA issuer then waits (bounded) for its last MMAs and the producer
// for its last copies before the tensor memory is freed.
//
// Shared-memory operand layouts (K-major), each written by TMA boxes as they land:
//  * 128-byte swizzle, when K is a multiple of 64: a box is 64 columns (128 bytes) x R
//    rows, row r at byte 128 r of its block with its eight 16-byte pieces permuted by
//    r % 8 (the TMA's SWIZZLE_128B); blocks of 64 columns follow each other at 128 R
//    bytes.  Descriptor: stride byte offset 1024 (eight rows), swizzle mode 128-byte;
//    the MMA over K columns [16 s, 16 s + 16) starts at block s / 4, byte 32 (s % 4).
//  * no swizzle, otherwise: a box is 8 columns (16 bytes) x R rows, so the 8-row x
//    16-byte core matrix (row group g, K group c) sits at byte (c R / 8 + g) * 128.
//    The K-direction core stride (leading byte offset) is 16 R bytes, the row-group
//    stride (stride byte offset) 128 bytes; the MMA over K columns [16 s, 16 s + 16)
//    starts at byte 32 R s.
// Wide boxes matter: a 16-byte box row is one request that moves a 32-byte sector.
constexpr int kUmmaM = 128;                    // rows per tile (the MMA's M)
constexpr int kUmmaStages = 3;                 // input stages in the ring
constexpr int kUmmaKS = 128;                   // K columns per stage at most
constexpr int kUmmaMaxN = 256, kUmmaMaxK = 256;
constexpr int kUmmaStageBytes = kUmmaM * kUmmaKS * 2;
constexpr int kUmmaBarBytes = 1024, kUmmaBiasBytes = 4 * kUmmaMaxN;
constexpr int kUmmaSmem = kUmmaBarBytes + kUmmaBiasBytes + kUmmaMaxN * kUmmaMaxK * 2 + kUmmaStages * kUmmaStageBytes;
constexpr int kUmmaEpiWarps = 8;               // epilogue warps: two per lane quarter
constexpr long long kUmmaSpin = 1ll << 22;     // polls of an mbarrier before a wait gives up
static_assert(kUmmaSmem <= 227 * 1024, "the tcgen05 layer needs more shared memory than a CTA has");

// two FP32 lanes in one 64-bit register, for the paired FP32 instructions (f32x2)
__device__ __forceinline__ uint64_t f2(float lo, float hi)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}

__device__ __forceinline__ void f2_split(uint64_t x, float &lo, float &hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(x));
}

__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// BF16 pair, lo in the low half (round to nearest even)
__device__ __forceinline__ uint32_t bf16x2(float lo, float hi)
{
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}

// GELU (the tanh form above) of a pair of pre-activations, packed to BF16: four
// paired FP32 instructions and two tanh per pair
__device__ __forceinline__ uint32_t gelu_bf16x2(uint64_t z)
{
    const uint64_t w = f2_fma(f2_mul(z, z), f2(kGeluC1, kGeluC1), f2(kGeluC0, kGeluC0));   // c0 + c1 z^2
    float u0, u1;
    f2_split(f2_mul(w, z), u0, u1);
    const uint64_t h = f2_mul(z, f2(0.5f, 0.5f));
    float r0, r1;
    f2_split(f2_fma(h, f2(tanh_approx(u0), tanh_approx(u1)), h), r0, r1);   // h (1 + t)
    return bf16x2(r0, r1);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Waits for the phase of the given parity to complete; false when it gives up after
// kUmmaSpin polls or when another role has raised `fail` (if given).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, const volatile int *fail)
{
    for (long long i = 0; i < kUmmaSpin; i++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if (fail && (i & 63) == 63 && *fail) return false;
    }
    return false;
}

// (error: host memory, read after the stream has been synchronised)
__device__ __forceinline__ void umma_fail(volatile int *fail, int *error)
{
    *fail = 1;
    *(volatile int *)error = 1;
    __threadfence_system();
}

// TMA: the box at element coordinates (x, y) of the map into shared memory at dst,
// completing on the mbarrier
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// One lane of the (whole) warp.  The MMA warps run their loops with every lane and issue
// under this for a few instructions at a time: the compiler then knows that one thread
// issues.  Under a plain lane == 0 an MMA takes 140 issue cycles and a commit 410,
// whatever the MMA's size; this way a 128 x 256 x 16 MMA with a commit every second one
// takes the 128 it needs.
__device__ __forceinline__ bool elect_one()
{
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e != 0;
}

// A plain bulk copy of `bytes` (a multiple of 16, both ends 16-byte aligned).
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void umma_bf16(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, bool accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(ad), "l"(bd), "r"(idesc), "r"((uint32_t)accumulate));
}

// the mbarrier completes when every tcgen05.mma this thread issued before has completed
__device__ __forceinline__ void umma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// tcgen05 shared-memory matrix descriptor: start >> 4 (bits 0-13), leading byte offset
// >> 4 (16-29), stride byte offset >> 4 (32-45), the fixed 0b001 (46-48), base offset 0
// (49-51, the operands are 1024-byte aligned), the swizzle mode (61-63: 0 none,
// 2 128-byte, 4 64-byte).
constexpr uint32_t kSwizzleNone = 0, kSwizzle128B = 2, kSwizzle64B = 4;
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo, uint32_t swizzle)
{
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46) | ((uint64_t)swizzle << 61);
}

// Instruction descriptor of kind::f16: FP32 accumulator (bits 4-5 = 1), BF16 A and B
// (bits 7-9, 10-12 = 1), both K-major (bits 15, 16 = 0), N >> 3 (17-22), M >> 4 (24-28).
__host__ __device__ constexpr uint32_t umma_idesc(int M, int N)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// tcgen05.ld of 32 consecutive accumulator columns of the warp's 32 lanes (one row a
// thread).  The registers are written asynchronously: read them only after
// tmem_ld_wait on the same array.
__device__ __forceinline__ void tmem_ld32_issue(uint32_t taddr, uint32_t v[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
        "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
          "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
          "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
}

// Waits for the warp's tcgen05.ld; the array is an operand so that no use of it is
// moved above the wait.
__device__ __forceinline__ void tmem_ld_wait(uint32_t v[32])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                   "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]),
                   "+r"(v[15]), "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]),
                   "+r"(v[22]), "+r"(v[23]), "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]),
                   "+r"(v[29]), "+r"(v[30]), "+r"(v[31])
                 :
                 : "memory");
}

// 16 columns, complete on return.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t v[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];\n\ttcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}

// The epilogue of one 32-column chunk of a tile row (v: its accumulator values): bias,
// GELU and BF16 stores for hidden layers (H), the accumulating FP32 stores for the last.
__device__ __forceinline__ void epilogue_chunk(const uint32_t v[32], int c0, long long row, const float *s_bias,
                                               int N, int gelu, bf16 *H, long long ldh, float *Y, long long ldy,
                                               float scale, int first, int vec)
{
    if (H) {
        const float4 *bq = reinterpret_cast<const float4 *>(s_bias + c0);
        uint32_t packed[16];
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
            const float4 bb = bq[j / 4];
            const uint64_t z01 = f2_add(f2(__uint_as_float(v[j]), __uint_as_float(v[j + 1])), f2(bb.x, bb.y));
            const uint64_t z23 = f2_add(f2(__uint_as_float(v[j + 2]), __uint_as_float(v[j + 3])), f2(bb.z, bb.w));
            if (gelu) {
                packed[j / 2] = gelu_bf16x2(z01);
                packed[j / 2 + 1] = gelu_bf16x2(z23);
            } else {
                float a0, a1, a2, a3;
                f2_split(z01, a0, a1);
                f2_split(z23, a2, a3);
                packed[j / 2] = bf16x2(a0, a1);
                packed[j / 2 + 1] = bf16x2(a2, a3);
            }
        }
        // N is a multiple of 32 for hidden layers: two 32-byte stores, whole sectors
        bf16 *dst = H + row * ldh + c0;
#pragma unroll
        for (int k = 0; k < 2; k++)
            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst + 16 * k),
                         "r"(packed[8 * k]), "r"(packed[8 * k + 1]), "r"(packed[8 * k + 2]), "r"(packed[8 * k + 3]),
                         "r"(packed[8 * k + 4]), "r"(packed[8 * k + 5]), "r"(packed[8 * k + 6]),
                         "r"(packed[8 * k + 7])
                         : "memory");
        return;
    }
    float *dst = Y + row * ldy + c0;
    if (vec) {
        // the four 32-byte runs of the accumulator are loaded together
        float o[32];
        if (!first)
#pragma unroll
            for (int k = 0; k < 4; k++)
                asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                             : "=f"(o[8 * k]), "=f"(o[8 * k + 1]), "=f"(o[8 * k + 2]), "=f"(o[8 * k + 3]),
                               "=f"(o[8 * k + 4]), "=f"(o[8 * k + 5]), "=f"(o[8 * k + 6]), "=f"(o[8 * k + 7])
                             : "l"(dst + 8 * k));
#pragma unroll
        for (int i = 0; i < 32; i++) {
            const float z = __uint_as_float(v[i]) + s_bias[c0 + i];
            o[i] = first ? scale * z : fmaf(scale, z, o[i]);
        }
#pragma unroll
        for (int k = 0; k < 4; k++)
            asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst + 8 * k),
                         "f"(o[8 * k]), "f"(o[8 * k + 1]), "f"(o[8 * k + 2]), "f"(o[8 * k + 3]), "f"(o[8 * k + 4]),
                         "f"(o[8 * k + 5]), "f"(o[8 * k + 6]), "f"(o[8 * k + 7])
                         : "memory");
    } else {
#pragma unroll
        for (int j = 0; j < 32; j++) {
            const int c = c0 + j;
            if (c < N) {
                const float z = __uint_as_float(v[j]) + s_bias[c];
                dst[j] = first ? scale * z : fmaf(scale, z, dst[j]);
            }
        }
    }
}

// One layer: out = act(A W^T + bias) over M rows, EPI epilogue warps.  tmA: the input
// (M x Kp BF16), box bw x kUmmaM; tmW: the weights (Np x Kp BF16, zero rows past N),
// box bw x Np; bw = 64 with the 128-byte swizzle (sw, Kp a multiple of 64), else 8.
// Kp a multiple of 16, Np of 16, both <= 256.  Hidden layers (H set) store
// BF16 activations (row stride ldh, N a multiple of 32).  The last layer (Y set)
// accumulates its FP32 outputs z: Y = scale z (first) or Y + scale z, row stride ldy;
// with `vec` (ldy a multiple of 32, Y 32-byte aligned) in whole 32-byte sectors,
// columns from N to the next multiple of 32 included (padding).  error: set when a
// wait gives up.
template <int EPI>
__global__ void __launch_bounds__(32 * (2 + EPI), 1)
    k_umma_layer(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, int M, int Kp,
                 int Np, int N, int sw, const float *bias, int gelu, bf16 *H, long long ldh, float *Y, long long ldy,
                 float scale, int first, int vec, int *error)
{
    static_assert(EPI % 4 == 0, "each of the four lane quarters needs the same number of epilogue warps");
    extern __shared__ __align__(1024) uint8_t smem[];
    // barrier page: full[S], empty[S], acc_full[2], acc_empty[2], weights, drain;
    // then the tensor-memory address and the failure flag
    const uint32_t b_full = smem_u32(smem), b_empty = b_full + 8 * kUmmaStages, b_accf = b_empty + 8 * kUmmaStages,
                   b_acce = b_accf + 16, b_w = b_acce + 16, b_drain = b_w + 8;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + 256);
    volatile int *fail = reinterpret_cast<volatile int *>(smem + 320);
    float *s_bias = reinterpret_cast<float *>(smem + kUmmaBarBytes);
    uint8_t *sW = smem + kUmmaBarBytes + kUmmaBiasBytes;
    const uint32_t sW_u = smem_u32(sW), sA_u = sW_u + kUmmaMaxN * kUmmaMaxK * 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 32) {
        for (int i = 0; i < kUmmaStages; i++) {
            mbar_init(b_full + 8 * i, 1);
            mbar_init(b_empty + 8 * i, 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(b_accf + 8 * i, 1);
            mbar_init(b_acce + 8 * i, EPI);
        }
        mbar_init(b_w, 1);
        mbar_init(b_drain, 1);
        *fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    for (int c = threadIdx.x; c < kUmmaMaxN; c += blockDim.x) s_bias[c] = c < N ? bias[c] : 0.f;
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = *tmem_slot;
    const int tiles = (M + kUmmaM - 1) / kUmmaM;
    const int bw = sw ? 64 : 8;   // K columns per TMA box
    // K columns per stage: all of K up to kUmmaKS, else about half, in whole boxes and MMA steps
    const int KS = Kp <= kUmmaKS ? Kp : (sw ? 64 * ((Kp / 64 + 1) / 2) : 16 * ((Kp / 16 + 1) / 2));
    const int nks = (Kp + KS - 1) / KS;                              // stages per tile: 1 or 2
    if (warp == 0) {
        if (lane == 0) {
            // producer
            mbar_expect_tx(b_w, (uint32_t)(Np * Kp * 2));
            for (int c = 0; c < Kp / bw; c++) tma_load_2d(sW_u + c * Np * bw * 2, &tmW, bw * c, 0, b_w);
            bool ok = true;
            int it = 0;   // stage fills issued
            for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x)
                for (int ks = 0; ks < nks; ks++) {
                    const int s = it % kUmmaStages, use = it / kUmmaStages;
                    if (use > 0 && !mbar_wait(b_empty + 8 * s, (use - 1) & 1, fail)) {
                        ok = false;
                        break;
                    }
                    const int k0 = ks * KS, kc = min(KS, Kp - k0);
                    const uint32_t dst = sA_u + s * kUmmaStageBytes;
                    mbar_expect_tx(b_full + 8 * s, (uint32_t)(kUmmaM * kc * 2));
                    for (int c = 0; c < kc / bw; c++)
                        tma_load_2d(dst + c * kUmmaM * bw * 2, &tmA, k0 + bw * c, t * kUmmaM, b_full + 8 * s);
                    it++;
                }
            if (!ok) umma_fail(fail, error);
            // every copy lands before the CTA ends: the last fill of each stage, the weights
            for (int s = 0; s < kUmmaStages; s++) {
                const int uses = it / kUmmaStages + (s < it % kUmmaStages ? 1 : 0);
                if (uses > 0) mbar_wait(b_full + 8 * s, (uses - 1) & 1, nullptr);
            }
            mbar_wait(b_w, 0, nullptr);
        }
        __syncwarp();
    } else if (warp == 1) {
        // MMA issuer (every lane; elect_one issues)
        bool ok = __all_sync(0xffffffffu, mbar_wait(b_w, 0, fail));   // (the lanes decide together)
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t idesc = umma_idesc(kUmmaM, Np);
        int it = 0, tc = 0;
        for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x, tc++) {
            const int b = tc & 1, use = tc >> 1;
            ok = __all_sync(0xffffffffu, use == 0 || mbar_wait(b_acce + 8 * b, (use - 1) & 1, fail));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint32_t d = tmem + 256u * b;
            for (int ks = 0; ks < nks; ks++, it++) {
                const int s = it % kUmmaStages, u = it / kUmmaStages;
                ok = __all_sync(0xffffffffu, mbar_wait(b_full + 8 * s, u & 1, fail));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;");
                const int k0 = ks * KS, kc = min(KS, Kp - k0);
                const uint32_t a0 = sA_u + s * kUmmaStageBytes;
                if (elect_one()) {
                    for (int j = 0; j < kc / 16; j++) {
                        const int g = k0 / 16 + j;   // the MMA step within K
                        uint64_t ad, wd;
                        if (sw) {
                            ad = umma_desc(a0 + (j >> 2) * kUmmaM * 128 + 32 * (j & 3), 16, 1024, kSwizzle128B);
                            wd = umma_desc(sW_u + (g >> 2) * Np * 128 + 32 * (g & 3), 16, 1024, kSwizzle128B);
                        } else {
                            ad = umma_desc(a0 + j * 32 * kUmmaM, 16 * kUmmaM, 128, kSwizzleNone);
                            wd = umma_desc(sW_u + g * 32 * Np, 16 * Np, 128, kSwizzleNone);
                        }
                        umma_bf16(d, ad, wd, idesc, (ks | j) != 0);
                    }
                    umma_commit(b_empty + 8 * s);   // the stage is free once these MMAs complete
                    if (ks == nks - 1) umma_commit(b_accf + 8 * b);
                }
                __syncwarp();
            }
        }
        if (!ok && lane == 0) umma_fail(fail, error);
        // every MMA issued completes before the tensor memory is freed
        if (elect_one()) umma_commit(b_drain);
        __syncwarp();
        mbar_wait(b_drain, 0, nullptr);
        __syncwarp();
    } else {
        // epilogue: lanes (tile rows) 32 q .. 32 q + 31, 32-column chunks part, part + EPI / 4, ...
        const int q = warp & 3, part = (warp - 2) >> 2;
        constexpr int parts = EPI / 4;
        int tc = 0;
        for (int t = blockIdx.x; t < tiles; t += gridDim.x, tc++) {
            const int b = tc & 1, use = tc >> 1;
            if (!__all_sync(0xffffffffu, mbar_wait(b_accf + 8 * b, use & 1, fail))) {
                if (lane == 0) umma_fail(fail, error);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;");
            const int row = t * kUmmaM + 32 * q + lane;
            const uint32_t tb = tmem + ((uint32_t)(32 * q) << 16) + 256u * b;
            for (int c0 = 32 * part; c0 < Np; c0 += 32 * parts) {
                uint32_t v[32];
                __syncwarp();   // tcgen05.ld and its wait are warp-collective
                tmem_ld32_issue(tb + c0, v);
                tmem_ld_wait(v);
                if (row < M) epilogue_chunk(v, c0, row, s_bias, N, gelu, H, ldh, Y, ldy, scale, first, vec);
            }
            // the accumulator is free for the tile after next
            asm volatile("tcgen05.fence::before_thread_sync;");
            __syncwarp();
            if (lane == 0) mbar_arrive(b_acce + 8 * b);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

// ---------------------------------------------------------------- training chain
// The forward pass, the loss and the data gradients of a batch in one launch: a row
// needs nothing of another row until the parameters' gradients are summed.  Sixteen rows
// are one m16 tile, and a cluster of four CTAs takes them through all layers, each CTA
// 64 of a layer's columns (8 a warp): a batch of 512 fills 128 SMs, and an SM reads a
// quarter of the weights.  The activations (then the dZ) of the rows lie in every CTA's
// shared memory, twice: a step's epilogue sends its columns to all four CTAs with
// st.async, whose bytes complete the mbarrier that the next step waits for.  A CTA with no
// columns in a layer (they all lie past its padded width) sends 16 bytes instead, which no
// product reads.  So whoever has a step's rows complete knows that every CTA has the rows of
// the step before and that every warp has read them, and nothing else guards the two copies
// and their barriers, nor the ring of the CTA's weights (forward: its 64 rows of
// W; back: its 64 columns; loaded two steps ahead).  What the parameter gradients
// read (activations, dZ) goes to global memory on the side, and so does Z, which the
// thread that wrote it reads again on the way back.
//
// Bound by the chain itself: per step 16 dependent MMAs, an epilogue and the way to the
// other CTAs.  With the parameter gradients of all layers in a second launch, a step of
// the 11-4x256-222 network at batch 512 takes 34 us on a GB300, 17 of them here; layer by
// layer it was ten launches, 82 us.  (With cluster barriers and without the four loader
// warps 42: a barrier's release waits 0.5 us for what was stored, and queueing a step's
// weights takes as long.)  Products, their order and the epilogues are k_gemm's, and so
// are the results.  Every wait is bounded.
constexpr int kChainCtas = 4, kChainRows = 16, kChainThreads = 256, kChainLoaders = 128, kChainStages = 3, kChainLayers = 8;
constexpr int kChainWidth = 256, kChainCols = kChainWidth / kChainCtas;
constexpr int kChainPitchK = (kChainWidth + 8) * 2, kChainPitchN = (kChainCols + 8) * 2;   // bytes; odd multiples of 16
constexpr int kChainStage = kChainWidth * kChainPitchN, kChainAct = kChainRows * kChainPitchK;
static_assert(kChainCols * kChainPitchK <= kChainStage, "a stage holds a CTA's part of a layer in both orders");
static_assert(kChainThreads / 32 * 8 == kChainCols, "eight columns a warp");
static_assert(2 * kChainLayers <= kMaxOps, "the parameter gradients of all layers are one launch");
constexpr int kChainBars = 8 * 2;   // each copy of the rows is complete
constexpr int kChainSmem = 2 * kChainAct + kChainStages * kChainStage + kChainBars;
static_assert(kChainSmem <= 227 * 1024, "the chain needs more shared memory than a CTA has");

struct ChainLayer {
    const bf16 *w;        // ldn x ldk, zero outside N x (the layer before's N)
    const float *bias;
    float *Z, *dZf;       // row stride ldn
    bf16 *H, *dZb;        // the layer's activations and dZ, row stride ldn
    int N, ldn, ldk;
    int bytes;            // of the rows' ldn columns and of the tokens of the CTAs that have none of them
};

struct ChainArgs {
    ChainLayer layer[kChainLayers];
    int L, B;
    const bf16 *x;        // inputs, row stride layer[0].ldk
    const float *Y;       // targets, rows by `rows` (nullptr: in order)
    const int *rows;
    float *loss;
    int *error;
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

// Queues loader t's share of CTA q's part of step c's weights: c < L the rows of layer c, then layers L - 1 to 1
// column by column.  (As bulk copies of a row each, 64 or 256 a step, a training step took
// 70 us: the copy engine takes them one after another.)
__device__ __forceinline__ void chain_load(const ChainArgs &a, int c, int q, uint32_t dst, int t)
{
    const bool fwd = c < a.L;
    const ChainLayer &w = a.layer[fwd ? c : 2 * a.L - 1 - c];
    const int first = q * kChainCols;
    if (fwd) {   // a row a warp
        const int k = t % 32 * 8, rows = k < w.ldk ? min(kChainCols, w.ldn - first) : 0;
#pragma unroll
        for (int i = 0; i < kChainCols * 32 / kChainLoaders; i++) {
            const int r = t / 32 + i * (kChainLoaders / 32);
            if (r < rows) cp_async16(dst + r * kChainPitchK + k * 2, w.w + (first + r) * w.ldk + k, true);
        }
    } else {     // four rows a warp
        const int k = t % (kChainCols / 8) * 8, rows = first + k < w.ldk ? w.ldn : 0;
#pragma unroll
        for (int i = 0; i < kChainWidth * (kChainCols / 8) / kChainLoaders; i++) {
            const int r = t / (kChainCols / 8) + i * (kChainLoaders * 8 / kChainCols);
            if (r < rows) cp_async16(dst + r * kChainPitchN + k * 2, w.w + r * w.ldk + first + k, true);
        }
    }
}

// 16 bytes to shared address dst of CTA `cta`, counted by its barrier at bar.
constexpr int kChainToken = 16;
__device__ __forceinline__ void chain_send(uint32_t dst, uint32_t bar, int cta, const uint32_t v[4])
{
    asm volatile("{\n\t.reg .b32 ra, rb;\n\tmapa.shared::cluster.u32 ra, %0, %2;\n\t"
                 "mapa.shared::cluster.u32 rb, %1, %2;\n\t"
                 "st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [ra], {%3, %4, %5, %6}, [rb];\n\t}"
                 ::"r"(dst), "r"(bar), "r"(cta), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3])
                 : "memory");
}

__global__ void __cluster_dims__(kChainCtas, 1, 1) __launch_bounds__(kChainThreads + kChainLoaders, 1)
    k_chain(const __grid_constant__ ChainArgs a)
{
    extern __shared__ __align__(16) uint8_t chain_smem[];
    __shared__ int s_fail;
    const uint32_t s_act = smem_u32(chain_smem), s_w = s_act + 2 * kChainAct;
    const uint32_t b_act = s_w + kChainStages * kChainStage;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q = (int)blockIdx.x % kChainCtas, r0 = (int)blockIdx.x / kChainCtas * kChainRows;
    const int steps = 2 * a.L - 1;
    const int ldx = a.layer[0].ldk;
    if (threadIdx.x == 0) {
        mbar_init(b_act, 1);
        mbar_init(b_act + 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_fail = 0;
    }
    if (threadIdx.x >= kChainThreads) {
        // the loaders: step 0's rows and weights, then a step's weights two steps ahead
        const int t = threadIdx.x - kChainThreads;
        cluster_arrive();
        for (int e = t; e < kChainRows * (ldx / 8); e += kChainLoaders) {
            const int r = e / (ldx / 8), k = e % (ldx / 8) * 8;
            const bool in = r0 + r < a.B;
            cp_async16(s_act + r * kChainPitchK + k * 2, in ? a.x + (long long)(r0 + r) * ldx + k : a.x, in);
        }
        chain_load(a, 0, q, s_w, t);
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (steps > 1) chain_load(a, 1, q, s_w + kChainStage, t);
        asm volatile("cp.async.commit_group;" ::: "memory");
        cluster_wait();
        for (int c = 0; c < steps; c++) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kChainStages - 2) : "memory");
            if (!__syncthreads_and(1)) break;   // step c's weights have landed; step c - 1's are used up
            if (c + kChainStages - 1 < steps)
                chain_load(a, c + kChainStages - 1, q, s_w + (c + kChainStages - 1) % kChainStages * kChainStage, t);
            asm volatile("cp.async.commit_group;" ::: "memory");   // (empty past the end, so the waits count alike)
            // a CTA with no columns in this step's outputs says to each that it has come here
            const int ldn = a.layer[c < a.L ? c : 2 * a.L - 2 - c].ldn;
            if (q * kChainCols >= ldn && t < kChainCtas && c + 1 < steps) {
                const uint32_t none[4] = {0u, 0u, 0u, 0u};
                chain_send(s_act + ((c + 1) & 1) * kChainAct + q * kChainCols * 2, b_act + 8 * ((c + 1) & 1), t, none);
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
        cluster_wait();
        return;
    }
    const int l7 = lane & 7, l8 = (lane >> 3) & 1, l16 = lane >> 4;
    const int row = lane >> 2, j = q * kChainCols + 8 * warp + 2 * (lane & 3);   // outputs (row + 8h, j + 0..1)
    const float count = (float)((long long)a.B * a.layer[a.L - 1].N), scale = 2.f / count;
    // what step c's epilogue reads, loaded while the step before runs: biases (forward) or
    // Z (back), and the targets (outside the rows and columns: the last ones', not used)
    const int i0 = min(r0 + row, a.B - 1), i1 = min(r0 + row + 8, a.B - 1);
    float x0[4], x1[4], y0[4], y1[4];
    auto fetch = [&](int c) {
        if (c < a.L) {
            const ChainLayer &o = a.layer[c];
            const int j0 = min(j, o.N - 1), j1 = min(j + 1, o.N - 1);
            y0[0] = y0[2] = o.bias[j0];
            y0[1] = y0[3] = o.bias[j1];
            if (c == a.L - 1) {
                const float *const t0 = a.Y + (long long)(a.rows ? a.rows[i0] : i0) * o.N;
                const float *const t1 = a.Y + (long long)(a.rows ? a.rows[i1] : i1) * o.N;
                y1[0] = t0[j0];
                y1[1] = t0[j1];
                y1[2] = t1[j0];
                y1[3] = t1[j1];
            }
        } else {
            const ChainLayer &o = a.layer[2 * a.L - 2 - c];
            const int jj = min(j, o.ldn - 2);   // (even, and so is the stride)
            const float2 z0 = *reinterpret_cast<const float2 *>(o.Z + (long long)i0 * o.ldn + jj);
            const float2 z1 = *reinterpret_cast<const float2 *>(o.Z + (long long)i1 * o.ldn + jj);
            y0[0] = z0.x;
            y0[1] = z0.y;
            y0[2] = z1.x;
            y0[3] = z1.y;
        }
    };
    cluster_arrive();   // every CTA of the cluster is here before one sends to it
    fetch(0);
    cluster_wait();
    float part = 0.f;
    bool ok = true;
    int c = 0;
    for (; c < steps; c++) {
        const bool fwd = c < a.L, last = c == a.L - 1;
        const ChainLayer &w = a.layer[fwd ? c : 2 * a.L - 1 - c], &o = fwd ? w : a.layer[2 * a.L - 2 - c];   // o: the outputs'
        const bool active = j - 2 * (lane & 3) < o.ldn;   // (of the whole warp)
        const uint32_t sa = s_act + (c & 1) * kChainAct, sw = s_w + (c % kChainStages) * kChainStage;
        const uint32_t next_act = b_act + 8 * ((c + 1) & 1);
        if (threadIdx.x == 0 && c + 1 < steps) mbar_expect_tx(next_act, o.bytes);
        ok = c == 0 || mbar_wait(b_act + 8 * (c & 1), ((c - 1) >> 1) & 1, &s_fail);
        ok = __syncthreads_and(ok);   // (step c's weights have landed for every thread)
        if (!ok) break;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            x0[e] = y0[e];
            x1[e] = y1[e];
        }
        if (c + 1 < steps) fetch(c + 1);
        float f[4];
        bf16 b[4];
        if (active) {
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
            const int n = (fwd ? w.ldk : w.ldn) / 16;
            const uint32_t pa = sa + (l7 + 8 * l8) * kChainPitchK + 16 * l16;
            // B of two steps: four 8 x 8 matrices along the reduction
            const uint32_t pb = fwd ? sw + (8 * warp + l7) * kChainPitchK + 16 * (l8 + 2 * l16)
                                    : sw + (l7 + 8 * (l8 + 2 * l16)) * kChainPitchN + 16 * warp;
            // all fragments first (those past n lie in the buffers and are not used)
            constexpr int kSteps = kChainWidth / 16;
            uint32_t fa[kSteps][4], fb[kSteps / 2][4];
#pragma unroll
            for (int k = 0; k < kSteps; k += 2) {
                if (fwd) ldmatrix4<false>(fb[k / 2], pb + 32 * k);
                else ldmatrix4<true>(fb[k / 2], pb + 16 * k * kChainPitchN);
                ldmatrix4<false>(fa[k], pa + 32 * k);
                ldmatrix4<false>(fa[k + 1], pa + 32 * (k + 1));
            }
#pragma unroll
            for (int k = 0; k < kSteps; k++)
                if (k < n) mma_bf16(acc, fa[k], fb[k / 2][2 * (k & 1)], fb[k / 2][2 * (k & 1) + 1]);
            // (output e: row + 8 (e / 2), column j + e % 2)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                if (fwd && !last) {
                    f[e] = acc[e] + x0[e];
                    b[e] = __float2bfloat16(gelu(f[e]));
                } else if (last) {
                    const float d = r0 + row + 8 * (e >> 1) < a.B && j + (e & 1) < o.N ? acc[e] + x0[e] - x1[e] : 0.f;
                    part += d * d;
                    f[e] = scale * d;
                    b[e] = __float2bfloat16(f[e]);
                } else {
                    f[e] = acc[e] * gelu_grad(x0[e]);
                    b[e] = __float2bfloat16(f[e]);
                }
                if (j + (e & 1) >= o.N) b[e] = __float2bfloat16(0.f);
            }
            if (c + 1 < steps) {
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    // a quad has a row's eight columns: its lane r sends them to CTA r
                    const __nv_bfloat162 pair(b[2 * h], b[2 * h + 1]);
                    const uint32_t word = *reinterpret_cast<const uint32_t *>(&pair);
                    uint32_t v[4];
#pragma unroll
                    for (int r = 0; r < 4; r++) v[r] = __shfl_sync(0xffffffffu, word, (lane & ~3) + r);
                    chain_send(s_act + ((c + 1) & 1) * kChainAct + (row + 8 * h) * kChainPitchK +
                                   (q * kChainCols + 8 * warp) * 2, next_act, lane & 3, v);
                }
            }
        }
        if (active) {
            float *const out = fwd && !last ? o.Z : o.dZf;
            bf16 *const outb = fwd && !last ? o.H : o.dZb;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int i = r0 + row + 8 * h;
                const long long at = (long long)i * o.ldn + j;
                if (i < a.B && j + 1 < o.N) {
                    *reinterpret_cast<float2 *>(out + at) = make_float2(f[2 * h], f[2 * h + 1]);
                    *reinterpret_cast<__nv_bfloat162 *>(outb + at) = __nv_bfloat162(b[2 * h], b[2 * h + 1]);
                } else if (i < a.B && j < o.N) {
                    out[at] = f[2 * h];
                    outb[at] = b[2 * h];
                }
            }
        }
    }
    if (!ok && threadIdx.x == 0) umma_fail(&s_fail, a.error);
    // no CTA leaves while another may still send to it
    asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
    cluster_wait();
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) part += __shfl_xor_sync(0xffffffffu, part, s);
    if (lane == 0 && part != 0.f) atomicAdd(a.loss, part / count);
}

// ---------------------------------------------------------------- fused hidden layers
// All hidden layers of one or more networks of a shape, activations kept on chip.  A
// layer-by-layer launch writes and reads 0.5 KB of activations per row and layer, which
// bounds it by DRAM (50 us a layer of 262,144 rows against 40 for the copies alone); here
// a row's activations leave the SM once, after the last hidden layer.  A persistent CTA
// takes items (a network and a tile of 128 rows) two at a time, X and Y, each with its
// activations in shared memory (64 KB, the MMA's A operand) and a 128 x 256 FP32
// accumulator in tensor memory, and works through X's layer 0, Y's layer 0, X's layer 1
// and so on: a layer's MMAs need the whole epilogue before it, so Y's MMAs run beside X's
// epilogue and the other way round.
//   warp 0      producer: an item's inputs and, for each step (a layer of X or Y), the layer's
//               weight slices of 32 K columns (16 KB) from L2 through a ring of kNetStages
//   warp 1      MMA issuer
//   warps 2-17  epilogue: bias, GELU, the next layer's activations (to shared memory in
//               the operand layout; the last layer's to global memory)
// Barriers: full / empty per stage; per item slot (X, Y) x: the inputs have landed, acc: the
// layer's MMAs are done, a: its epilogue is (activations stored, accumulator drained), free:
// the item's last MMAs are done.  The producer waits for `free`, one phase an item, before an
// item's inputs go into a slot.  (acc has a phase a layer: a wait by parity on it is only
// right for one who has seen the phase before, and at 64 hidden columns the ring holds more
// slices than an item has.)
// Every wait is bounded, as in k_umma_layer.  The order of the MMAs into an accumulator is
// that of k_umma_layer, and so are the results, bit for bit.  262,144 rows through 11-256-
// 256-256-222 take 764 us with it, 607 of them here, against 1,031 layer by layer (GB300);
// 32 rows 65 us instead of 220.  No unit is near its limit (tensor pipe 29% busy, issue
// 42%, shared-memory banks 13%; with half of each weight slice copied 752 us, so L2 is not
// it): a slice's two MMAs take 500 to 650 cycles beside the other item's epilogue, 256 alone.
constexpr int kNetStages = 6, kNetK = 32, kNetStageBytes = kUmmaMaxN * kNetK * 2, kNetTileBytes = kUmmaM * kUmmaMaxK * 2;
constexpr int kNetBarBytes = 1024;
constexpr int kNetSmem = kNetBarBytes + 2 * kNetTileBytes + kNetStages * kNetStageBytes;
constexpr int kNetEpiWarps = 16, kNetThreads = 32 * (2 + kNetEpiWarps);
constexpr int kNetMaxMembers = 8;
static_assert(kNetSmem <= 227 * 1024, "the fused layers need more shared memory than a CTA has");

struct NetShape {
    int M, kp0, hid, layers, members;   // rows, padded inputs, hidden width, hidden layers, networks
    int sw0;                            // the input layer's operands are swizzled (kp0 a multiple of 64)
    int slots;                          // items a CTA takes at a time: 1 or 2
    const bf16 *w0, *w;                 // the networks' weight slices (PackArgs)
    const float *bias;                  // members x layers x hid
    bf16 *out[kNetMaxMembers];          // each network's last hidden activations, M x hid
    int *error;
};

__global__ void __launch_bounds__(kNetThreads, 1)
    k_umma_hidden(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ NetShape n)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t b_full = smem_u32(smem), b_empty = b_full + 8 * kNetStages, b_x = b_empty + 8 * kNetStages,
                   b_acc = b_x + 16, b_a = b_acc + 16, b_free = b_a + 16, b_drain = b_free + 16;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + 512);
    volatile int *fail = reinterpret_cast<volatile int *>(smem + 576);
    const uint32_t sA_u = smem_u32(smem + kNetBarBytes), sW_u = sA_u + 2 * kNetTileBytes;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 32) {
        for (int i = 0; i < kNetStages; i++) {
            mbar_init(b_full + 8 * i, 1);
            mbar_init(b_empty + 8 * i, 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(b_x + 8 * i, 1);
            mbar_init(b_acc + 8 * i, 1);
            mbar_init(b_a + 8 * i, kNetEpiWarps);
            mbar_init(b_free + 8 * i, 1);
        }
        mbar_init(b_drain, 1);
        *fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = *tmem_slot;
    const int items = (n.M + kUmmaM - 1) / kUmmaM * n.members;   // item i: row tile i / members of network i % members
    const int step = (int)gridDim.x * n.slots;
    if (warp == 0) {
        if (lane == 0) {
            bool ok = true;
            int it = 0, seen[2] = {0, 0};   // stage fills; items of each slot
            for (int i0 = blockIdx.x * n.slots; ok && i0 < items; i0 += step) {
                const int here = min(n.slots, items - i0);
                for (int l = 0; ok && l < n.layers; l++)
                    for (int t = 0; ok && t < here; t++) {
                        const int m = (i0 + t) % n.members;
                        if (l == 0) {
                            // the slot's buffer is free once its last item's last MMAs have read it
                            if (seen[t] > 0 && !mbar_wait(b_free + 8 * t, (seen[t] - 1) & 1, fail)) {
                                ok = false;
                                break;
                            }
                            seen[t]++;
                            const int bw = n.sw0 ? 64 : 8, row = (i0 + t) / n.members * kUmmaM;
                            mbar_expect_tx(b_x + 8 * t, (uint32_t)(kUmmaM * n.kp0 * 2));
                            for (int c = 0; c < n.kp0 / bw; c++)
                                tma_load_2d(sA_u + t * kNetTileBytes + c * kUmmaM * bw * 2, &tmX, bw * c, row, b_x + 8 * t);
                        }
                        // the layer's slices lie in memory as they do in a stage
                        const int K = l == 0 ? n.kp0 : n.hid;
                        const bf16 *src = l == 0 ? n.w0 + (size_t)m * n.kp0 * n.hid
                                                 : n.w + (size_t)(m * (n.layers - 1) + l - 1) * n.hid * n.hid;
                        for (int k0 = 0; k0 < K; k0 += kNetK, it++) {
                            const int st = it % kNetStages, use = it / kNetStages;
                            if (use > 0 && !mbar_wait(b_empty + 8 * st, (use - 1) & 1, fail)) {
                                ok = false;
                                break;
                            }
                            const uint32_t bytes = (uint32_t)(min(kNetK, K - k0) * n.hid * 2);
                            mbar_expect_tx(b_full + 8 * st, bytes);
                            bulk_load(sW_u + st * kNetStageBytes, src + (size_t)k0 * n.hid, bytes, b_full + 8 * st);
                        }
                    }
            }
            if (!ok) umma_fail(fail, n.error);
            // every copy lands before the CTA ends: the last fill of each stage, the last inputs
            for (int st = 0; st < kNetStages; st++) {
                const int uses = it / kNetStages + (st < it % kNetStages ? 1 : 0);
                if (uses > 0) mbar_wait(b_full + 8 * st, (uses - 1) & 1, nullptr);
            }
            for (int t = 0; t < 2; t++)
                if (seen[t] > 0) mbar_wait(b_x + 8 * t, (seen[t] - 1) & 1, nullptr);
        }
        __syncwarp();
    } else if (warp == 1) {
        // (every lane; elect_one issues)
        bool ok = true;
        const uint32_t idesc = umma_idesc(kUmmaM, n.hid);
        int it = 0, seen[2] = {0, 0}, done[2] = {0, 0};   // stages; items and layers of each slot
        for (int i0 = blockIdx.x * n.slots; ok && i0 < items; i0 += step) {
            const int here = min(n.slots, items - i0);
            for (int l = 0; ok && l < n.layers; l++)
                for (int t = 0; ok && t < here; t++) {
                    // the layer's activations (or inputs), and a drained accumulator
                    ok = __all_sync(0xffffffffu, (done[t] == 0 || mbar_wait(b_a + 8 * t, (done[t] - 1) & 1, fail)) &&
                                                     (l > 0 || mbar_wait(b_x + 8 * t, seen[t] & 1, fail)));
                    if (!ok) break;
                    done[t]++;
                    if (l == 0) seen[t]++;
                    const int K = l == 0 ? n.kp0 : n.hid;
                    const uint32_t a0 = sA_u + t * kNetTileBytes, d = tmem + 256u * t;
                    for (int k0 = 0; k0 < K; k0 += kNetK, it++) {
                        const int st = it % kNetStages;
                        ok = __all_sync(0xffffffffu, mbar_wait(b_full + 8 * st, (it / kNetStages) & 1, fail));
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;");
                        const uint32_t w0 = sW_u + st * kNetStageBytes;
                        if (elect_one()) {
#pragma unroll
                            for (int j = 0; j < kNetK / 16; j++) {
                                if (k0 + 16 * j >= K) break;
                                const int g = k0 / 16 + j;   // the MMA step within K
                                uint64_t ad, wd;
                                if (l > 0 || n.sw0) {
                                    ad = umma_desc(a0 + (g >> 2) * kUmmaM * 128 + 32 * (g & 3), 16, 1024, kSwizzle128B);
                                    wd = umma_desc(w0 + 32 * j, 16, 512, kSwizzle64B);
                                } else {
                                    ad = umma_desc(a0 + g * 32 * kUmmaM, 16 * kUmmaM, 128, kSwizzleNone);
                                    wd = umma_desc(w0 + j * 32 * n.hid, 16 * n.hid, 128, kSwizzleNone);
                                }
                                umma_bf16(d, ad, wd, idesc, g != 0);
                            }
                            umma_commit(b_empty + 8 * st);   // the stage is free once these MMAs complete
                            if (k0 + kNetK >= K) {
                                umma_commit(b_acc + 8 * t);
                                if (l + 1 == n.layers) umma_commit(b_free + 8 * t);
                            }
                        }
                        __syncwarp();
                    }
                }
        }
        if (!ok && lane == 0) umma_fail(fail, n.error);
        // every MMA issued completes before the tensor memory is freed
        if (elect_one()) umma_commit(b_drain);
        __syncwarp();
        mbar_wait(b_drain, 0, nullptr);
        __syncwarp();
    } else {
        // epilogue: rows 32 q .. 32 q + 31, columns c0 .. c0 + cw - 1
        const int part = (warp - 2) >> 2, q = warp & 3;
        const int cw = n.hid / 4, c0 = part * cw;   // 16 to 64, a multiple of 16
        const int r = 32 * q + lane;
        int done[2] = {0, 0};
        bool ok = true;
        for (int i0 = blockIdx.x * n.slots; ok && i0 < items; i0 += step) {
            const int here = min(n.slots, items - i0);
            for (int l = 0; ok && l < n.layers; l++)
                for (int t = 0; t < here; t++) {
                    const int m = (i0 + t) % n.members, row = (i0 + t) / n.members * kUmmaM + r;
                    const float *bias = n.bias + (size_t)(m * n.layers + l) * n.hid + c0;
                    const bool last = l + 1 == n.layers;
                    const uint32_t tb = tmem + 256u * t + ((uint32_t)(32 * q) << 16) + c0;
                    const uint32_t arow = sA_u + t * kNetTileBytes + r * 128;
                    if (!__all_sync(0xffffffffu, mbar_wait(b_acc + 8 * t, done[t] & 1, fail))) {
                        ok = false;
                        break;
                    }
                    done[t]++;
                    asm volatile("tcgen05.fence::after_thread_sync;");
                    for (int c = 0; c < cw; c += 16) {
                        float4 bb[4];
#pragma unroll
                        for (int j = 0; j < 4; j++) bb[j] = __ldg(reinterpret_cast<const float4 *>(bias + c) + j);
                        uint32_t v[16];
                        __syncwarp();   // tcgen05.ld and its wait are warp-collective
                        tmem_ld16(tb + (uint32_t)c, v);
                        uint32_t p[8];
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            const uint32_t *w = v + 4 * j;
                            p[2 * j] = gelu_bf16x2(f2_add(f2(__uint_as_float(w[0]), __uint_as_float(w[1])), f2(bb[j].x, bb[j].y)));
                            p[2 * j + 1] =
                                gelu_bf16x2(f2_add(f2(__uint_as_float(w[2]), __uint_as_float(w[3])), f2(bb[j].z, bb[j].w)));
                        }
                        const int k0 = c0 + c;
                        if (!last) {
                            // two 16-byte pieces of the row, where the 128-byte swizzle has them
                            const uint32_t blk = arow + (uint32_t)(k0 >> 6) * (kUmmaM * 128);
#pragma unroll
                            for (int k = 0; k < 2; k++) {
                                const uint32_t a = blk + (uint32_t)(((((k0 & 63) >> 3) + k) ^ (r & 7)) << 4);
                                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(p[4 * k]),
                                             "r"(p[4 * k + 1]), "r"(p[4 * k + 2]), "r"(p[4 * k + 3]) : "memory");
                            }
                        } else if (row < n.M) {
                            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(
                                             n.out[m] + (size_t)row * n.hid + k0),
                                         "r"(p[0]), "r"(p[1]), "r"(p[2]), "r"(p[3]), "r"(p[4]), "r"(p[5]), "r"(p[6]),
                                         "r"(p[7])
                                         : "memory");
                        }
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;");
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(b_a + 8 * t);
                }
        }
        if (!ok && lane == 0) umma_fail(fail, n.error);
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

// The members' weights side by side: for the mean layer wc (np x members * hid: member
// m's last weights in columns [m hid, (m + 1) hid)) and the summed last biases; for
// k_umma_hidden (w0 set) the input layers' weights w0 (members x kp0 hid), the later hidden
// ones' w (members x (layers - 1) x hid hid) and their biases (members x layers x hid).  The
// hidden weights lie in slices of 32 K columns, each in the operand layout of its stage, so
// a slice is one bulk copy of 16 KB: with the 64-byte swizzle row n has 64 bytes, its four 16-byte
// pieces permuted by n / 2 % 4; without (input widths that are no multiple of 64) groups of
// eight columns follow each other, 16 bytes a row.
struct PackArgs {
    const bf16 *wpk[kNetMaxMembers][16];
    const float *bias[kNetMaxMembers][16];
    int members, layers, kp0, hid, np, nout;
    bf16 *w0, *w, *wc;
    float *hbias, *bsum;
};

__global__ void k_pack_members(const __grid_constant__ PackArgs a)
{
    const long long stride = (long long)gridDim.x * blockDim.x, first = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long n0 = (long long)a.hid * a.kp0, nh = (long long)a.hid * a.hid, nc = (long long)a.np * a.hid;
    if (a.w0) {
        // element i of a layer with K columns: its row r and column c
        auto place = [&](int i, int K, bool swizzled) {
            const int s = i / (kNetK * a.hid), e = i % (kNetK * a.hid);   // slice, element of it
            const int kc = min(kNetK, K - kNetK * s);
            int r, c;
            if (swizzled) {
                r = e / kNetK;
                c = ((e % kNetK / 8) ^ (r >> 1 & 3)) * 8 + e % 8;
            } else {
                r = e / 8 % a.hid;
                c = e / (8 * a.hid) * 8 + e % 8;
            }
            return (long long)r * K + kNetK * s + min(c, kc - 1);
        };
        const bool sw0 = a.kp0 % 64 == 0;
        for (long long i = first; i < n0 * a.members; i += stride)
            a.w0[i] = a.wpk[i / n0][0][place((int)(i % n0), a.kp0, sw0)];
        for (long long i = first; i < nh * a.members * (a.layers - 1); i += stride) {
            const int k = (int)(i / nh);
            a.w[i] = a.wpk[k / (a.layers - 1)][1 + k % (a.layers - 1)][place((int)(i % nh), a.hid, true)];
        }
        for (long long i = first; i < (long long)a.hid * a.layers * a.members; i += stride) {
            const int k = (int)(i / a.hid);
            a.hbias[i] = a.bias[k / a.layers][k % a.layers][i % a.hid];
        }
    }
    for (long long i = first; i < nc * a.members; i += stride) {
        const long long r = i / ((long long)a.hid * a.members);
        const int c = (int)(i % ((long long)a.hid * a.members));
        a.wc[i] = a.wpk[c / a.hid][a.layers][r * a.hid + c % a.hid];
    }
    for (long long i = first; i < a.nout; i += stride) {
        float s = 0.f;
        for (int m = 0; m < a.members; m++) s += a.bias[m][a.layers][i];
        a.bsum[i] = s;
    }
}

// ---------------------------------------------------------------- ensemble mean layer
// The members' last layers in one GEMM: y = inv * (sum_m W_m h_m + sum_m b_m), the
// mean of the members' outputs (one member: its outputs).  The members' last hidden
// activations h_m (M x Kh BF16 each) are one operand concatenated along K, their weights
// W_m (Np x Kh) side by side in Wc (Np x members * Kh), so the tensor cores sum over
// members in the accumulator and the outputs are written once, to their rows of N
// columns: a warp turns its 32 x 32 piece in shared memory, so that each store is 128
// consecutive bytes.  (Written to padded rows and compacted by a second kernel, 262,144 x
// 222 outputs cost 70 us more.)  Wc is too large for shared memory, so every stage of
// the ring carries a 64-column slice of both operands (128-byte swizzled boxes); the
// roles, accumulators and waits are those of k_umma_layer.
constexpr int kMeanStages = 4, kMeanEpiWarps = 8;
constexpr int kMeanAStage = kUmmaM * 64 * 2;        // 16 KB
constexpr int kMeanWStage = kUmmaMaxN * 64 * 2;     // 32 KB
constexpr int kMeanTurn = 32 * 32 * 4;              // a warp's piece
constexpr int kMeanSmem = kUmmaBarBytes + kUmmaBiasBytes + kMeanStages * (kMeanAStage + kMeanWStage) +
                          kMeanEpiWarps * kMeanTurn;
static_assert(kMeanSmem <= 227 * 1024, "the ensemble layer needs more shared memory than a CTA has");

struct MeanMaps {
    CUtensorMap a[kNetMaxMembers];   // member m's hidden activations, box 64 x kUmmaM, 128-byte swizzle
};

__global__ void __launch_bounds__(32 * (2 + kMeanEpiWarps), 1)
    k_umma_mean_layer(const __grid_constant__ MeanMaps maps, const __grid_constant__ CUtensorMap tmW, int M, int Kh,
                      int members, int Np, int N, const float *bias_sum, float inv, float *Y, int *error)
{
    constexpr int EPI = kMeanEpiWarps;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t b_full = smem_u32(smem), b_empty = b_full + 8 * kMeanStages, b_accf = b_empty + 8 * kMeanStages,
                   b_acce = b_accf + 16, b_drain = b_acce + 16;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + 256);
    volatile int *fail = reinterpret_cast<volatile int *>(smem + 320);
    float *s_bias = reinterpret_cast<float *>(smem + kUmmaBarBytes);
    const uint32_t sA_u = smem_u32(smem + kUmmaBarBytes + kUmmaBiasBytes);   // stage s: A at +s*(A+W), W after it
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 32) {
        for (int i = 0; i < kMeanStages; i++) {
            mbar_init(b_full + 8 * i, 1);
            mbar_init(b_empty + 8 * i, 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(b_accf + 8 * i, 1);
            mbar_init(b_acce + 8 * i, EPI);
        }
        mbar_init(b_drain, 1);
        *fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    for (int c = threadIdx.x; c < kUmmaMaxN; c += blockDim.x) s_bias[c] = c < N ? bias_sum[c] : 0.f;
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = *tmem_slot;
    const int tiles = (M + kUmmaM - 1) / kUmmaM;
    const int per = Kh / 64, nks = per * members;   // 64-column slices per member, per tile
    const uint32_t stage_bytes = kMeanAStage + kMeanWStage;
    if (warp == 0) {
        if (lane == 0) {
            // producer: per stage, the slice of one member's activations and of the weights
            bool ok = true;
            int it = 0;
            for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x)
                for (int j = 0; j < nks; j++) {
                    const int s = it % kMeanStages, use = it / kMeanStages;
                    if (use > 0 && !mbar_wait(b_empty + 8 * s, (use - 1) & 1, fail)) {
                        ok = false;
                        break;
                    }
                    const uint32_t a = sA_u + s * stage_bytes;
                    mbar_expect_tx(b_full + 8 * s, (uint32_t)(kUmmaM * 128 + Np * 128));
                    tma_load_2d(a, &maps.a[j / per], 64 * (j % per), t * kUmmaM, b_full + 8 * s);
                    tma_load_2d(a + kMeanAStage, &tmW, 64 * j, 0, b_full + 8 * s);
                    it++;
                }
            if (!ok) umma_fail(fail, error);
            for (int s = 0; s < kMeanStages; s++) {
                const int uses = it / kMeanStages + (s < it % kMeanStages ? 1 : 0);
                if (uses > 0) mbar_wait(b_full + 8 * s, (uses - 1) & 1, nullptr);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // MMA issuer (every lane; elect_one issues): 4 MMAs (K = 16) per 64-column slice
        bool ok = true;
        const uint32_t idesc = umma_idesc(kUmmaM, Np);
        int it = 0, tc = 0;
        for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x, tc++) {
            const int b = tc & 1, use = tc >> 1;
            ok = __all_sync(0xffffffffu, use == 0 || mbar_wait(b_acce + 8 * b, (use - 1) & 1, fail));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint32_t d = tmem + 256u * b;
            for (int j = 0; j < nks; j++, it++) {
                const int s = it % kMeanStages, u = it / kMeanStages;
                ok = __all_sync(0xffffffffu, mbar_wait(b_full + 8 * s, u & 1, fail));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;");
                const uint32_t a = sA_u + s * stage_bytes, w = a + kMeanAStage;
                if (elect_one()) {
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        umma_bf16(d, umma_desc(a + 32 * q, 16, 1024, kSwizzle128B),
                                  umma_desc(w + 32 * q, 16, 1024, kSwizzle128B), idesc, (j | q) != 0);
                    umma_commit(b_empty + 8 * s);
                    if (j == nks - 1) umma_commit(b_accf + 8 * b);
                }
                __syncwarp();
            }
        }
        if (!ok && lane == 0) umma_fail(fail, error);
        if (elect_one()) umma_commit(b_drain);
        __syncwarp();
        mbar_wait(b_drain, 0, nullptr);
        __syncwarp();
    } else {
        // epilogue: y = inv * (acc + sum of the biases), written once
        const int q = warp & 3, part = (warp - 2) >> 2;
        constexpr int parts = EPI / 4;
        float *const turn = reinterpret_cast<float *>(smem + kUmmaBarBytes + kUmmaBiasBytes +
                                                      kMeanStages * (kMeanAStage + kMeanWStage) + (warp - 2) * kMeanTurn);
        int tc = 0;
        for (int t = blockIdx.x; t < tiles; t += gridDim.x, tc++) {
            const int b = tc & 1, use = tc >> 1;
            if (!__all_sync(0xffffffffu, mbar_wait(b_accf + 8 * b, use & 1, fail))) {
                if (lane == 0) umma_fail(fail, error);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;");
            const int row0 = t * kUmmaM + 32 * q;
            const uint32_t tb = tmem + ((uint32_t)(32 * q) << 16) + 256u * b;
            for (int c0 = 32 * part; c0 < Np; c0 += 32 * parts) {
                uint32_t v[32];
                __syncwarp();   // (also: the last piece has been written)
                tmem_ld32_issue(tb + c0, v);
                tmem_ld_wait(v);
                // element (row l, column j) of the piece at word 32 l + (j ^ l): no bank conflicts either way
#pragma unroll
                for (int j = 0; j < 32; j++)
                    turn[32 * lane + (j ^ lane)] = inv * (__uint_as_float(v[j]) + s_bias[c0 + j]);
                __syncwarp();
                if (c0 + lane < N) {
                    float *y = Y + (long long)row0 * N + c0 + lane;
#pragma unroll 8
                    for (int i = 0; i < 32; i++)
                        if (row0 + i < M) y[(long long)i * N] = turn[32 * i + (lane ^ i)];
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;");
            __syncwarp();
            if (lane == 0) mbar_arrive(b_acce + 8 * b);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

// FP32 rows x cols (from src, contiguous rows) -> BF16 at dst, row stride ld (round to
// nearest even); the rest of a row is left as it is.
__global__ void k_weights_bf16(const float *src, int rows, int cols, bf16 *dst, int ld)
{
    const long long n = (long long)rows * cols;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i / cols * ld + i % cols] = __float2bfloat16(src[i]);
}

// The tcgen05 path's input: rows x din FP32 -> rows x kp BF16 (round to nearest even,
// zero columns past din), one 16-byte group of eight columns per thread.
__global__ void k_input_bf16(const float *x, int rows, int din, bf16 *dst, int kp)
{
    const int groups = kp / 8;
    const long long n = (long long)rows * groups;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const long long r = i / groups;
        const int c0 = (int)(i % groups) * 8;
        const float *xr = x + r * din;
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int c = c0 + 2 * k;
            w[k] = bf16x2(c < din ? xr[c] : 0.f, c + 1 < din ? xr[c + 1] : 0.f);
        }
        *reinterpret_cast<uint4 *>(dst + r * kp + c0) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// rows x cols FP32 from src (row stride lds) to dst (contiguous rows), a warp per row
__global__ void k_compact_rows(const float *src, long long lds, float *dst, int rows, int cols)
{
    const int lane = threadIdx.x & 31, wpb = blockDim.x / 32;
    const long long warps = (long long)gridDim.x * wpb;
    for (long long r = (long long)blockIdx.x * wpb + (threadIdx.x >> 5); r < rows; r += warps) {
        const float *s = src + r * lds;
        float *d = dst + r * cols;
        for (int c = lane; c < cols; c += 32) d[c] = s[c];
    }
}

// rows of x in the order idx (nullptr: as they are) -> BF16 rows of stride ld, zeros
// past din
__global__ void k_gather(const float *X, const int *idx, int B, int din, bf16 *Hb, int ld)
{
    const long long n = (long long)B * ld;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int row = (int)(i / ld), c = (int)(i % ld);
        Hb[i] = __float2bfloat16(c < din ? X[(long long)(idx ? idx[row] : row) * din + c] : 0.f);
    }
}

// acc = scale z (first) or acc + scale z over rows x cols (row strides lda, ldz), the
// arithmetic of the tcgen05 layer's accumulating epilogue
__global__ void k_accumulate(float *acc, long long lda, const float *z, int ldz, int rows, int cols, float scale, int first)
{
    const long long n = (long long)rows * cols;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        float *a = acc + (i / cols) * lda + i % cols;
        const float v = z[i / cols * ldz + i % cols];
        *a = first ? scale * v : fmaf(scale, v, *a);
    }
}

thread_local std::string g_mlp_create_error;

}  // namespace

struct pt_mlp {
    int L = 0;
    std::vector<int> width;
    std::vector<long long> woff, boff;   // offsets of W_l and b_l in the parameter arrays
    long long nparam = 0;
    int max_batch = 0;
    cudaStream_t stream = nullptr;
    // device
    float *w = nullptr, *m = nullptr, *v = nullptr, *grad = nullptr;
    std::vector<int> ld;        // width[l] to a multiple of 16: the row stride of H, Z and dZ
    std::vector<bf16 *> wpk;    // BF16 weights of each layer, ld[l + 1] x ld[l], zero outside width[l + 1] x width[l]
    std::vector<bf16 *> H;      // H[0] = input batch, H[l+1] = layer l output (BF16)
    std::vector<float *> Z;     // Z[l] = layer l pre-activation (FP32)
    std::vector<float *> dZf;   // dZ[l] (FP32)
    std::vector<bf16 *> dZb;    // dZ[l] (BF16)
    float *loss = nullptr;              // of each step of an epoch (loss_cap)
    int loss_cap = 0;
    float *X = nullptr, *Y = nullptr;   // data set
    bf16 *Xe = nullptr;                 // its inputs in the epoch's order, BF16, row stride ld[0]
    int *perm = nullptr;
    int n = 0;
    long long step = 0;
    std::string err;
    std::vector<void *> allocs;
    uint64_t version = 0;       // of the weights: another number after every change, in any network
    // tcgen05 inference: the padded input batch and a wait error word (host memory the
    // device writes)
    int use_umma = 1;
    bool chain_ready = false;   // training: k_chain may be launched
    bf16 *h0p = nullptr;
    ptm::Mapped err_word;
    int *umma_err = nullptr;    // err_word's
    // inference input (FP32 rows copied from the host), and the accumulator of last layers
    // that run one by one (rows padded to a multiple of 32), max_batch rows each
    float *xin = nullptr;
    float *zout = nullptr;
    int ldz = 0;
    // the members' weights side by side (held by an ensemble's first network), the
    // versions they were packed from and the capacity in members
    PackArgs pack{};
    bool pack_always = false;   // a call of this network has been captured
    std::vector<uint64_t> packed;
    int pack_cap = 0;
};

static std::atomic<uint64_t> g_weights_version{0};

static pt_status mfail(pt_mlp *m, pt_status st, const std::string &msg)
{
    if (m) m->err = msg;
    else g_mlp_create_error = msg;
    return st;
}

#define MCK(expr, where)                                                                                       \
    do {                                                                                                       \
        cudaError_t _e = (expr);                                                                               \
        if (_e != cudaSuccess) {                                                                               \
            cudaGetLastError(); /* reported here; the next launch would report it again */                     \
            return mfail(m, _e == cudaErrorMemoryAllocation ? PT_ERR_OOM : PT_ERR_CUDA,                        \
                         std::string(where) + ": " + cudaGetErrorString(_e));                                  \
        }                                                                                                      \
    } while (0)

template <typename T>
static cudaError_t dalloc(pt_mlp *m, T **p, size_t count)
{
    cudaError_t e = cudaMalloc((void **)p, std::max<size_t>(count, 1) * sizeof(T));
    if (e == cudaSuccess) m->allocs.push_back(*p);
    return e;
}

// One launch of up to kMaxOps independent GEMMs.
static cudaError_t gemm(pt_mlp *m, GemmLaunch &l, int ops)
{
    unsigned blocks = 0;
    for (int o = 0; o < ops; o++) {
        GemmOp &g = l.op[o];
        g.blocks = g.kind == kOpBias ? (g.N + kBiasCols - 1) / kBiasCols
                                     : ((g.M + kGemmTile - 1) / kGemmTile) * ((g.N + kGemmTile - 1) / kGemmTile);
        blocks += (unsigned)g.blocks;
    }
    if (blocks == 0) return cudaSuccess;
    k_gemm<<<blocks, kGemmThreads, 0, m->stream>>>(l);
    return cudaGetLastError();
}

// forward pass over the B rows at h0 (BF16, row stride ld[0]).  With Y, the last layer forms
// the loss (added to *loss) and its gradient dZ against the targets, rows by `rows`;
// without, it leaves its outputs in Z.
static cudaError_t forward(pt_mlp *m, int B, const bf16 *h0, const float *Y = nullptr, const int *rows = nullptr,
                           float *loss = nullptr)
{
    for (int l = 0; l < m->L; l++) {
        const bool last = l + 1 == m->L;
        GemmLaunch gl = {};
        GemmOp &g = gl.op[0];
        g.kind = !last ? kOpForward : (Y ? kOpLoss : kOpOutput);
        g.A = l == 0 ? h0 : m->H[l];
        g.lda = m->ld[l];
        g.B = m->wpk[l];   // B(r, j) = W_l[j][r]
        g.ldb = m->ld[l];
        g.Brows = m->ld[l + 1];
        g.M = B;
        g.N = m->width[l + 1];
        g.R = m->width[l];
        g.bias = m->w + m->boff[l];
        g.Z = m->Z[l];
        g.ldz = m->ld[l + 1];
        g.H = m->H[l + 1];
        g.ldh = m->ld[l + 1];
        g.dZf = m->dZf[l];
        g.dZb = m->dZb[l];
        g.ldd = m->ld[l + 1];
        g.Y = Y;
        g.rows = rows;
        g.loss = loss;
        cudaError_t e = gemm(m, gl, 1);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// gradients of every parameter for the B rows at h0 whose forward pass has run: into
// `grad`, or (nullptr) straight into Adam's update.  Layer l's weights are updated one
// launch after the last product that reads them.  With `chained` every dZ is there
// already, and all parameters are one launch.
static cudaError_t backward(pt_mlp *m, int B, const bf16 *h0, float *grad, const AdamArgs &adam, bool chained)
{
    auto weights = [&](GemmOp &g, int l) {   // dW_l[j][k] = sum_i dZ_l[i][j] H_l[i][k]
        g = GemmOp{};
        g.kind = kOpWeights;
        g.A = m->dZb[l];
        g.lda = m->ld[l + 1];
        g.B = l == 0 ? h0 : m->H[l];
        g.ldb = m->ld[l];
        g.M = m->width[l + 1];
        g.N = m->width[l];
        g.R = B;
        g.param = m->woff[l];
        g.grad = grad;
        g.wpk = m->wpk[l];
        g.ldw = m->ld[l];
    };
    auto bias = [&](GemmOp &g, int l) {      // db_l[j] = sum_i dZ_l[i][j]
        g = GemmOp{};
        g.kind = kOpBias;
        g.M = B;
        g.N = m->width[l + 1];
        g.dZf = m->dZf[l];
        g.ldd = m->ld[l + 1];
        g.param = m->boff[l];
        g.grad = grad;
    };
    GemmLaunch gl = {};
    gl.adam = adam;
    const int last = m->L - 1;
    for (int l = chained ? 0 : last; l >= 1; l--) {
        // dZ_{l-1}[i][k] = (sum_j dZ_l[i][j] W_l[j][k]) GELU'(Z_{l-1}[i][k])
        GemmOp &g = gl.op[0];
        g = GemmOp{};
        g.kind = kOpBackward;
        g.A = m->dZb[l];
        g.lda = m->ld[l + 1];
        g.B = m->wpk[l];
        g.ldb = m->ld[l];
        g.Brows = m->ld[l + 1];
        g.M = B;
        g.N = m->width[l];
        g.R = m->width[l + 1];
        g.Z = m->Z[l - 1];
        g.ldz = m->ld[l];
        g.dZf = m->dZf[l - 1];
        g.dZb = m->dZb[l - 1];
        g.ldd = m->ld[l];
        int ops = 1;
        if (l < last) {
            weights(gl.op[ops++], l + 1);
            bias(gl.op[ops++], l + 1);
        }
        cudaError_t e = gemm(m, gl, ops);
        if (e != cudaSuccess) return e;
    }
    int ops = 0;
    for (int l = chained ? last : std::min(1, last); l >= 0; l--) {
        weights(gl.op[ops++], l);
        bias(gl.op[ops++], l);
    }
    return gemm(m, gl, ops);
}

// Whether a network trains by k_chain: its layers and their widths fit one cluster.
static bool chain_fits(const pt_mlp *m)
{
    bool ok = m->L <= kChainLayers;
    for (int ld : m->ld) ok = ok && ld <= kChainWidth;
    return ok;
}

// The word that a device wait writes when it gives up (host memory the device writes).
static cudaError_t error_word(pt_mlp *m)
{
    if (m->umma_err) return cudaSuccess;
    const cudaError_t e = ptm::mapped_take(sizeof(int), &m->err_word);
    if (e != cudaSuccess) return e;
    m->umma_err = (int *)m->err_word.ptr;
    *m->umma_err = 0;
    return cudaSuccess;
}

static cudaError_t chain(pt_mlp *m, int B, const bf16 *h0, const float *Y, const int *rows, float *loss)
{
    if (!m->chain_ready) {   // (a kernel's attributes are those of the network's device)
        cudaError_t e = cudaFuncSetAttribute(k_chain, cudaFuncAttributeMaxDynamicSharedMemorySize, kChainSmem);
        if (e == cudaSuccess) e = error_word(m);
        if (e != cudaSuccess) return e;
        m->chain_ready = true;
    }
    ChainArgs a = {};
    a.error = m->umma_err;
    a.L = m->L;
    a.B = B;
    a.x = h0;
    a.Y = Y;
    a.rows = rows;
    a.loss = loss;
    for (int l = 0; l < m->L; l++) {
        ChainLayer &c = a.layer[l];
        c.w = m->wpk[l];
        c.bias = m->w + m->boff[l];
        c.Z = m->Z[l];
        c.dZf = m->dZf[l];
        c.H = m->H[l + 1];
        c.dZb = m->dZb[l];
        c.N = m->width[l + 1];
        c.ldn = m->ld[l + 1];
        c.ldk = m->ld[l];
        c.bytes = kChainRows * c.ldn * 2 + kChainToken * (kChainCtas - (c.ldn + kChainCols - 1) / kChainCols);
    }
    k_chain<<<(B + kChainRows - 1) / kChainRows * kChainCtas, kChainThreads + kChainLoaders, kChainSmem, m->stream>>>(a);
    return cudaGetLastError();
}

// The loss (added to *loss) of the B rows at h0 against the targets Y, rows by `rows`, and
// the gradients of every parameter: into `grad`, or (nullptr) into Adam's update.
static cudaError_t training_pass(pt_mlp *m, int B, const bf16 *h0, const float *Y, const int *rows, float *loss,
                                 float *grad, const AdamArgs &adam)
{
    const bool chained = chain_fits(m);
    const cudaError_t e = chained ? chain(m, B, h0, Y, rows, loss) : forward(m, B, h0, Y, rows, loss);
    return e == cudaSuccess ? backward(m, B, h0, grad, adam, chained) : e;
}

static int grid_for(long long n) { return (int)std::min<long long>((n + 255) / 256, 4096); }

static int pad16(int x) { return (x + 15) / 16 * 16; }

// the BF16 weights from the FP32 parameters
static cudaError_t refresh_weights(pt_mlp *m)
{
    for (int l = 0; l < m->L; l++)
        k_weights_bf16<<<grid_for((long long)m->width[l + 1] * m->width[l]), 256, 0, m->stream>>>(
            m->w + m->woff[l], m->width[l + 1], m->width[l], m->wpk[l], m->ld[l]);
    return cudaGetLastError();
}

// The tcgen05 path takes every layer whose padded sizes fit the kernel: inputs and
// outputs at most 256 wide, hidden widths a multiple of 32.
static bool umma_fits(const pt_mlp *m)
{
    for (int l = 0; l < m->L; l++) {
        const int din = m->width[l], dout = m->width[l + 1];
        if (pad16(din) > kUmmaMaxK || pad16(dout) > kUmmaMaxN) return false;
        if (l > 0 && din % 16 != 0) return false;           // read in place from H[l]
        if (l + 1 < m->L && dout % 32 != 0) return false;  // whole 64-byte output runs
    }
    return true;
}

static int sm_count_mlp()
{
    static const int n = [] {
        int dev = 0, v = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        return v > 0 ? v : 1;
    }();
    return n;
}

// The driver's tensor-map encoder, through the runtime's entry-point query (no link
// against the driver library).
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled()
{
    static const EncodeTiledFn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return (EncodeTiledFn) nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// A map over a rows x cols BF16 matrix (row stride ld elements, a multiple of 8) whose
// box is box_rows rows by box_cols columns: 64 with the 128-byte swizzle, 8 without (cols a
// multiple of box_cols): the TMA boxes of a tcgen05 operand in the kernels' two
// shared-memory layouts.  Rows past `rows` read as zeros.
static bool operand_map(CUtensorMap *map, const bf16 *base, int rows, int cols, long long ld, int box_rows, int box_cols)
{
    const EncodeTiledFn fn = encode_tiled();
    if (!fn || ld % 8 != 0 || cols % box_cols != 0) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1u, 1u};
    const CUtensorMapSwizzle swizzle = box_cols == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE;
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16 *>(base), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static int pad32(int x) { return (x + 31) / 32 * 32; }

// The padded accumulator of a network, kept between calls.
static cudaError_t ensure_zout(pt_mlp *m)
{
    if (m->zout) return cudaSuccess;
    m->ldz = pad32(m->width[m->L]);
    return dalloc(m, &m->zout, (size_t)m->max_batch * m->ldz);
}

// The tcgen05 path's per-network state: the padded input buffer and the wait error word.
static cudaError_t umma_prepare(pt_mlp *m)
{
    if (m->h0p) return cudaSuccess;
    cudaError_t e = error_word(m);
    if (e != cudaSuccess) return e;
    // once a network: a kernel's attributes are those of its device
    e = cudaFuncSetAttribute(k_umma_layer<kUmmaEpiWarps>, cudaFuncAttributeMaxDynamicSharedMemorySize, kUmmaSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_umma_mean_layer, cudaFuncAttributeMaxDynamicSharedMemorySize, kMeanSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_umma_hidden, cudaFuncAttributeMaxDynamicSharedMemorySize, kNetSmem);
    if (e != cudaSuccess) return e;
    return dalloc(m, &m->h0p, (size_t)m->max_batch * m->ld[0]);
}

// forward pass for inference over B rows of x (device, B x width[0] FP32), its outputs
// z accumulated into y (row stride ldy): y = scale z when `first`, else y + scale z.
// tcgen05 layers when the shapes fit (hidden H[l] receive the activations, the last
// layer accumulates in its epilogue), else forward() and k_accumulate.  *x0 caches the
// zero-padded BF16 copy of x that the tcgen05 layers read: the first network of an
// ensemble makes it (into its h0p), the others reuse it.
// With hidden_only, the tcgen05 path stops after the last hidden layer (H[L-1] holds
// its activations) and y is not written.
static cudaError_t forward_infer(pt_mlp *m, int B, const float *x, const bf16 **x0, float *y, long long ldy,
                                 float scale, bool first, bool hidden_only = false)
{
    if (!m->use_umma || !umma_fits(m)) {
        if (B == 0) return cudaSuccess;
        k_gather<<<grid_for((long long)B * m->ld[0]), 256, 0, m->stream>>>(x, nullptr, B, m->width[0], m->H[0], m->ld[0]);
        cudaError_t e = forward(m, B, m->H[0]);
        if (e != cudaSuccess) return e;
        const long long total = (long long)B * m->width[m->L];
        k_accumulate<<<(int)std::min<long long>((total + 255) / 256, 4096), 256, 0, m->stream>>>(
            y, ldy, m->Z[m->L - 1], m->ld[m->L], B, m->width[m->L], scale, first ? 1 : 0);
        return cudaGetLastError();
    }
    cudaError_t e = umma_prepare(m);
    if (e != cudaSuccess) return e;
    if (!*x0) {
        k_input_bf16<<<grid_for((long long)B * m->ld[0] / 8), 256, 0, m->stream>>>(x, B, m->width[0], m->h0p,
                                                                                    m->ld[0]);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        *x0 = m->h0p;
    }
    const int tiles = (B + kUmmaM - 1) / kUmmaM;
    for (int l = 0; l < (hidden_only ? m->L - 1 : m->L); l++) {
        const int Kp = m->ld[l], Np = m->ld[l + 1];
        const bool last = l + 1 == m->L;
        // one CTA per SM: the full shared-memory request keeps a second one off the SM,
        // so the 512 tensor-memory columns a CTA allocates are always free
        const int grid = std::max(1, std::min(tiles, sm_count_mlp()));
        const bf16 *A = l == 0 ? *x0 : m->H[l];
        const long long lda = m->ld[l];
        const bool sw = Kp % 64 == 0;   // the 128-byte swizzled layout: whole 128-byte box rows
        CUtensorMap ma, mw;
        if (!operand_map(&ma, A, B, Kp, lda, kUmmaM, sw ? 64 : 8) ||
            !operand_map(&mw, m->wpk[l], Np, Kp, Kp, Np, sw ? 64 : 8))
            return cudaErrorNotSupported;
        const int N = m->width[l + 1];
        const float *bias = m->w + m->boff[l];
        bf16 *Hn = last ? nullptr : m->H[l + 1];
        float *Yn = last ? y : nullptr;
        // whole-sector accumulation: 32-column runs fit the row and start 32-byte aligned
        const int vec = last && ldy % 32 == 0 && ldy >= pad32(N) && reinterpret_cast<uintptr_t>(y) % 32 == 0;
        k_umma_layer<kUmmaEpiWarps><<<grid, 32 * (2 + kUmmaEpiWarps), kUmmaSmem, m->stream>>>(
            ma, mw, B, Kp, Np, N, sw ? 1 : 0, bias, last ? 0 : 1, Hn, N, Yn, ldy, scale, first ? 1 : 0, vec,
            m->umma_err);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// Whether the networks' hidden layers run fused (k_umma_hidden): all on the tcgen05 path,
// at least one hidden layer, every one as wide, 64 to 256 in steps of 64.
static bool net_fits(pt_mlp *const *members, int count)
{
    const pt_mlp *m = members[0];
    if (count > kNetMaxMembers || m->L < 2 || m->L > 15) return false;
    const int hid = m->width[1];
    if (hid % 64 != 0) return false;
    for (int l = 2; l < m->L; l++)
        if (m->width[l] != hid) return false;
    for (int j = 0; j < count; j++)
        if (!members[j]->use_umma || !umma_fits(members[j])) return false;
    return true;
}

// Whether an ensemble runs its last layers as one GEMM (k_umma_mean_layer): up to
// kNetMaxMembers members, all on the tcgen05 path, the last layer's input a multiple of
// 64 wide and its output at most kUmmaMaxN.  A single network does when its hidden layers
// are fused: that saves the pass that compacts padded outputs.
static bool mean_layer_fits(pt_mlp *const *members, int count)
{
    if (net_fits(members, count)) return true;
    if (count < 2 || count > kNetMaxMembers) return false;
    for (int j = 0; j < count; j++)
        if (!members[j]->use_umma || !umma_fits(members[j])) return false;
    const pt_mlp *m = members[0];
    return m->L >= 2 && m->L <= 15 && m->width[m->L - 1] % 64 == 0;
}

// The members' weights side by side in the first one's buffers, packed again when any of
// them has changed (versions are never used twice, so equal versions are equal weights).
// A captured call packs whenever its graph runs, so that it has the weights of that time;
// from then on every call does, for a replay may have left another ensemble's there.
static cudaError_t pack_members(pt_mlp *const *members, int count, bool hidden, cudaStream_t s)
{
    pt_mlp *m = members[0];
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (!m->pack_always) {
        const cudaError_t q = cudaStreamIsCapturing(s, &capture);
        if (q != cudaSuccess) return q;
        m->pack_always = capture != cudaStreamCaptureStatusNone;
        if (m->pack_always) m->packed.clear();
    }
    std::vector<uint64_t> v(1, hidden ? 1 : 0);
    for (int j = 0; j < count; j++) v.push_back(members[j]->version);
    if (v == m->packed) return cudaSuccess;
    m->packed.clear();
    PackArgs &a = m->pack;
    const int L = m->L;
    a.members = count;
    a.layers = L - 1;
    a.kp0 = m->ld[0];
    a.hid = m->width[L - 1];
    a.np = m->ld[L];
    a.nout = m->width[L];
    cudaError_t e = cudaSuccess;
    if (m->pack_cap < count) {   // (smaller buffers are freed with the network)
        m->pack_cap = 0;
        const size_t c = (size_t)count;
        e = dalloc(m, &a.wc, c * a.np * a.hid);
        if (e == cudaSuccess) e = dalloc(m, &a.bsum, kUmmaMaxN);
        if (e == cudaSuccess) e = dalloc(m, &a.w0, c * a.hid * a.kp0);
        if (e == cudaSuccess) e = dalloc(m, &a.w, c * std::max(1, a.layers - 1) * a.hid * a.hid);
        if (e == cudaSuccess) e = dalloc(m, &a.hbias, c * a.layers * a.hid);
        if (e != cudaSuccess) return e;
        m->pack_cap = count;
    }
    for (int j = 0; j < count; j++)
        for (int l = 0; l < L; l++) {
            a.wpk[j][l] = members[j]->wpk[l];
            a.bias[j][l] = members[j]->w + members[j]->boff[l];
        }
    PackArgs args = a;
    if (!hidden) args.w0 = nullptr;
    k_pack_members<<<2 * sm_count_mlp(), 256, 0, s>>>(args);
    e = cudaGetLastError();
    if (e == cudaSuccess && !m->pack_always) m->packed = v;
    return e;
}

// Every member's hidden layers over the B rows of x, fused: H[L-1] of each holds its last
// activations.
static cudaError_t hidden_fused(pt_mlp *const *members, int count, int B, const float *x, cudaStream_t s)
{
    pt_mlp *m = members[0];
    cudaError_t e = umma_prepare(m);
    if (e != cudaSuccess) return e;
    const int kp0 = m->ld[0], hid = m->width[1], layers = m->L - 1;
    k_input_bf16<<<grid_for((long long)B * kp0 / 8), 256, 0, s>>>(x, B, m->width[0], m->h0p, kp0);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    NetShape n = {};
    n.M = B;
    n.kp0 = kp0;
    n.hid = hid;
    n.layers = layers;
    n.members = count;
    n.sw0 = kp0 % 64 == 0;
    n.bias = m->pack.hbias;
    for (int j = 0; j < count; j++) n.out[j] = members[j]->H[m->L - 1];
    n.error = m->umma_err;
    n.w0 = m->pack.w0;
    n.w = m->pack.w;
    CUtensorMap mx;
    if (!operand_map(&mx, m->h0p, B, kp0, kp0, kUmmaM, n.sw0 ? 64 : 8)) return cudaErrorNotSupported;
    // two items a CTA once every SM has one
    const int items = (B + kUmmaM - 1) / kUmmaM * count;
    n.slots = items > sm_count_mlp() ? 2 : 1;
    const int grid = std::min((items + n.slots - 1) / n.slots, sm_count_mlp());
    k_umma_hidden<<<grid, kNetThreads, kNetSmem, s>>>(mx, n);
    return cudaGetLastError();
}

// The mean of the members' last layers over B rows into y (contiguous rows), after every
// member's hidden layers have run (H[L-1] of each holds its activations).
static cudaError_t mean_layer(pt_mlp *const *members, int count, int B, float *y, cudaStream_t s)
{
    pt_mlp *m = members[0];
    const int L = m->L, kh = m->width[L - 1], N = m->width[L], np = m->ld[L];
    MeanMaps maps;
    memset(&maps, 0, sizeof(maps));
    for (int j = 0; j < count; j++)
        if (!operand_map(&maps.a[j], members[j]->H[L - 1], B, kh, kh, kUmmaM, 64)) return cudaErrorNotSupported;
    CUtensorMap mw;
    if (!operand_map(&mw, m->pack.wc, np, kh * count, (long long)kh * count, np, 64)) return cudaErrorNotSupported;
    const int tiles = (B + kUmmaM - 1) / kUmmaM;
    const int grid = std::max(1, std::min(tiles, sm_count_mlp()));
    k_umma_mean_layer<<<grid, 32 * (2 + kMeanEpiWarps), kMeanSmem, s>>>(maps, mw, B, kh, count, np, N, m->pack.bsum,
                                                                        1.0f / (float)count, y, m->umma_err);
    return cudaGetLastError();
}

// One chunk of B rows of x (device) through every member, their mean to the contiguous
// rows of `out`: the members' hidden layers (fused where they fit), then one mean layer
// when it fits, else each member's last layer accumulating in its epilogue.
static cudaError_t ensemble_chunk(pt_mlp *const *members, int count, int B, const float *x, float *out, cudaStream_t s)
{
    if (B == 0) return cudaSuccess;
    pt_mlp *m = members[0];
    const bool net = net_fits(members, count), mean = mean_layer_fits(members, count);
    cudaError_t e = mean ? pack_members(members, count, net, s) : ensure_zout(m);
    if (e == cudaSuccess && net) e = hidden_fused(members, count, B, x, s);
    const bf16 *x0 = nullptr;
    for (int j = 0; j < count && e == cudaSuccess && !net; j++) {
        pt_mlp *q = members[j];
        const cudaStream_t own = q->stream;
        q->stream = s;
        e = forward_infer(q, B, x, &x0, m->zout, m->ldz, 1.0f / (float)count, j == 0, mean);
        q->stream = own;
    }
    if (e != cudaSuccess) return e;
    if (mean) return mean_layer(members, count, B, out, s);
    k_compact_rows<<<std::min((B + 7) / 8, 8192), 256, 0, s>>>(m->zout, m->ldz, out, B, m->width[m->L]);
    return cudaGetLastError();
}

// A device wait of a kernel here that gave up: reported once, then cleared.  The
// stream has been synchronised.
static pt_status umma_check(pt_mlp *m)
{
    if (!m->umma_err || *(volatile int *)m->umma_err == 0) return PT_OK;
    *(volatile int *)m->umma_err = 0;
    return mfail(m, PT_ERR_TIMEOUT, "a device-side wait gave up");
}

// The checks of an ensemble call; the rows its networks take at a time.
static pt_status ensemble_check(pt_mlp *const *members, int count, int *chunk)
{
    pt_mlp *m = members[0];
    if (!m) return PT_ERR_ARG;
    *chunk = m->max_batch;
    for (int j = 0; j < count; j++) {
        pt_mlp *q = members[j];
        if (!q) return PT_ERR_ARG;
        if (q->L != m->L) return mfail(m, PT_ERR_ARG, "ensemble members differ in depth");
        for (int l = 0; l <= m->L; l++)
            if (q->width[l] != m->width[l]) return mfail(m, PT_ERR_ARG, "ensemble members differ in widths");
        *chunk = std::min(*chunk, q->max_batch);
    }
    // every member runs on the first member's stream: finish what is queued on its own
    for (int j = 1; j < count; j++)
        if (members[j]->stream != m->stream)
            MCK(cudaStreamSynchronize(members[j]->stream), "ensemble member stream");
    return PT_OK;
}

extern "C" {

pt_status pt_mlp_create(int layers, const int *widths, int max_batch, uint64_t seed, void *cuda_stream, pt_mlp **out)
{
    if (!widths || !out || layers < 1 || layers > 16 || max_batch < 1 || max_batch > (1 << 20))
        return mfail(nullptr, PT_ERR_ARG, "layers must be 1..16 and max_batch 1..2^20");
    for (int l = 0; l <= layers; l++)
        if (widths[l] < 1 || widths[l] > 4096) return mfail(nullptr, PT_ERR_ARG, "widths must be 1..4096");
    *out = nullptr;
    pt_mlp *m = new pt_mlp();
    m->L = layers;
    m->width.assign(widths, widths + layers + 1);
    m->max_batch = max_batch;
    m->stream = (cudaStream_t)cuda_stream;
    for (int l = 0; l <= layers; l++) m->ld.push_back(pad16(widths[l]));
    for (int l = 0; l < layers; l++) {
        m->woff.push_back(m->nparam);
        m->nparam += (long long)widths[l + 1] * widths[l];
        m->boff.push_back(m->nparam);
        m->nparam += widths[l + 1];
    }
    auto bad = [&](cudaError_t e, const char *what) {
        if (e == cudaSuccess) return false;
        mfail(nullptr, e == cudaErrorMemoryAllocation ? PT_ERR_OOM : PT_ERR_CUDA,
              std::string(what) + ": " + cudaGetErrorString(e));
        pt_mlp_destroy(m);
        return true;
    };
    const size_t P = (size_t)m->nparam;
    if (bad(dalloc(m, &m->w, P), "parameters") || bad(dalloc(m, &m->m, P), "adam m") ||
        bad(dalloc(m, &m->v, P), "adam v") || bad(dalloc(m, &m->grad, P), "gradients") ||
        bad(dalloc(m, &m->loss, 1), "loss"))
        return PT_ERR_CUDA;
    m->loss_cap = 1;
    // The BF16 buffers' padding columns (and the weights' padding rows) stay zero: they
    // are cleared here and never written.  A buffer without any is left as it is (clearing
    // the 1.3 GB of a 262,144-row network takes 200 us).
    m->wpk.resize(layers);
    m->H.resize(layers + 1);
    m->Z.resize(layers);
    m->dZf.resize(layers);
    m->dZb.resize(layers);
    auto zeroed = [&](bf16 **p, size_t n, const char *what, bool padded = true) {
        return bad(dalloc(m, p, n), what) ||
               (padded && bad(cudaMemsetAsync(*p, 0, n * sizeof(bf16), m->stream), what));
    };
    auto padded = [&](int l) { return m->ld[l] != widths[l]; };
    for (int l = 0; l <= layers; l++)
        if (zeroed(&m->H[l], (size_t)max_batch * m->ld[l], "activations", padded(l))) return PT_ERR_CUDA;
    for (int l = 0; l < layers; l++) {
        const size_t n = (size_t)max_batch * m->ld[l + 1];
        if (bad(dalloc(m, &m->Z[l], n), "pre-activations") || bad(dalloc(m, &m->dZf[l], n), "gradients") ||
            zeroed(&m->dZb[l], n, "gradients", padded(l + 1)) ||
            zeroed(&m->wpk[l], (size_t)m->ld[l + 1] * m->ld[l], "bf16 weights"))
            return PT_ERR_CUDA;
    }
    // He-uniform weights (bound sqrt(6 / fan_in)), zero biases, from a seeded generator
    std::vector<float> init(P, 0.f);
    std::mt19937_64 rng(seed);
    for (int l = 0; l < layers; l++) {
        const float bound = std::sqrt(6.f / (float)widths[l]);
        std::uniform_real_distribution<float> U(-bound, bound);
        for (long long i = 0; i < (long long)widths[l + 1] * widths[l]; i++) init[m->woff[l] + i] = U(rng);
    }
    *out = m;
    return pt_mlp_set_params(m, init.data());
}

pt_status pt_mlp_param_count(const pt_mlp *m, int64_t *count)
{
    if (!m || !count) return PT_ERR_ARG;
    *count = m->nparam;
    return PT_OK;
}

pt_status pt_mlp_set_params(pt_mlp *m, const float *params)
{
    if (!m || !params) return PT_ERR_ARG;
    const size_t bytes = (size_t)m->nparam * sizeof(float);
    MCK(cudaMemcpyAsync(m->w, params, bytes, cudaMemcpyHostToDevice, m->stream), "parameters");
    MCK(cudaMemsetAsync(m->m, 0, bytes, m->stream), "adam m");
    MCK(cudaMemsetAsync(m->v, 0, bytes, m->stream), "adam v");
    MCK(refresh_weights(m), "bf16 weights");
    MCK(cudaStreamSynchronize(m->stream), "sync");
    m->step = 0;
    m->version = ++g_weights_version;
    return PT_OK;
}

pt_status pt_mlp_get_params(pt_mlp *m, float *params)
{
    if (!m || !params) return PT_ERR_ARG;
    MCK(cudaMemcpyAsync(params, m->w, (size_t)m->nparam * sizeof(float), cudaMemcpyDeviceToHost, m->stream), "copy");
    MCK(cudaStreamSynchronize(m->stream), "sync");
    return PT_OK;
}

pt_status pt_mlp_set_data(pt_mlp *m, const float *X, const float *Y, int n)
{
    if (!m || !X || !Y || n < 1) return PT_ERR_ARG;
    for (void *p : {(void *)m->X, (void *)m->Y, (void *)m->Xe, (void *)m->perm}) {
        if (!p) continue;
        cudaFree(p);
        m->allocs.erase(std::remove(m->allocs.begin(), m->allocs.end(), p), m->allocs.end());
    }
    m->X = m->Y = nullptr;
    m->Xe = nullptr;
    m->perm = nullptr;
    const int din = m->width[0], dout = m->width[m->L];
    MCK(dalloc(m, &m->X, (size_t)n * din), "data");
    MCK(dalloc(m, &m->Y, (size_t)n * dout), "data");
    MCK(dalloc(m, &m->Xe, (size_t)n * m->ld[0]), "data");
    MCK(dalloc(m, &m->perm, (size_t)n), "data");
    MCK(cudaMemcpyAsync(m->X, X, (size_t)n * din * sizeof(float), cudaMemcpyHostToDevice, m->stream), "data");
    MCK(cudaMemcpyAsync(m->Y, Y, (size_t)n * dout * sizeof(float), cudaMemcpyHostToDevice, m->stream), "data");
    MCK(cudaStreamSynchronize(m->stream), "sync");
    m->n = n;
    return PT_OK;
}

pt_status pt_mlp_train(pt_mlp *m, int epochs, int batch, float lr, uint64_t shuffle_seed, float *epoch_loss)
{
    if (!m || epochs < 1 || batch < 1 || batch > m->max_batch || !(lr > 0.f)) return PT_ERR_ARG;
    if (!m->X) return mfail(m, PT_ERR_STATE, "pt_mlp_train before pt_mlp_set_data");
    m->version = ++g_weights_version;
    const int din = m->width[0], steps = (m->n + batch - 1) / batch;
    if (steps > m->loss_cap) {
        float *p = nullptr;
        MCK(dalloc(m, &p, (size_t)steps), "losses");
        m->loss = p;   // (the smaller one is freed with the network)
        m->loss_cap = steps;
    }
    std::vector<int> perm(m->n);
    std::mt19937_64 rng(shuffle_seed);
    for (int ep = 0; ep < epochs; ep++) {
        std::iota(perm.begin(), perm.end(), 0);
        std::shuffle(perm.begin(), perm.end(), rng);
        MCK(cudaMemcpyAsync(m->perm, perm.data(), perm.size() * sizeof(int), cudaMemcpyHostToDevice, m->stream),
            "permutation");
        // the epoch's inputs in its order, and a loss word a step
        k_gather<<<grid_for((long long)m->n * m->ld[0]), 256, 0, m->stream>>>(m->X, m->perm, m->n, din, m->Xe, m->ld[0]);
        MCK(cudaGetLastError(), "gather");
        MCK(cudaMemsetAsync(m->loss, 0, (size_t)steps * sizeof(float), m->stream), "losses");
        for (int s = 0; s < steps; s++) {
            const int s0 = s * batch, B = std::min(batch, m->n - s0);
            const bf16 *h0 = m->Xe + (size_t)s0 * m->ld[0];
            m->step++;
            AdamArgs a;
            a.w = m->w;
            a.m = m->m;
            a.v = m->v;
            a.lr = lr;
            a.c1 = 1.f - std::pow(0.9f, (float)m->step);
            a.c2 = 1.f - std::pow(0.999f, (float)m->step);
            MCK(training_pass(m, B, h0, m->Y, m->perm + s0, m->loss + s, nullptr, a), "training step");
        }
    }
    // the last epoch's losses
    std::vector<float> l(steps);
    MCK(cudaMemcpyAsync(l.data(), m->loss, (size_t)steps * sizeof(float), cudaMemcpyDeviceToHost, m->stream), "losses");
    MCK(cudaStreamSynchronize(m->stream), "sync");
    const pt_status waits = umma_check(m);
    if (waits != PT_OK) return waits;
    double sum = 0.0;
    for (int s = 0; s < steps; s++) sum += l[s] * std::min(batch, m->n - s * batch);
    if (epoch_loss) *epoch_loss = (float)(sum / m->n);
    return PT_OK;
}

pt_status pt_mlp_gradients(pt_mlp *m, const float *X, const float *Y, int n, float *grads, float *loss)
{
    if (!m || !X || !Y || !grads || n < 1 || n > m->max_batch) return PT_ERR_ARG;
    const int din = m->width[0], dout = m->width[m->L];
    float *dX = nullptr, *dY = nullptr;
    MCK(cudaMalloc(&dX, (size_t)n * din * sizeof(float)), "batch");
    cudaError_t e = cudaMalloc(&dY, (size_t)n * dout * sizeof(float));
    if (e == cudaSuccess) e = cudaMemcpyAsync(dX, X, (size_t)n * din * sizeof(float), cudaMemcpyHostToDevice, m->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dY, Y, (size_t)n * dout * sizeof(float), cudaMemcpyHostToDevice, m->stream);
    if (e == cudaSuccess) {
        k_gather<<<grid_for((long long)n * m->ld[0]), 256, 0, m->stream>>>(dX, nullptr, n, din, m->H[0], m->ld[0]);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemsetAsync(m->loss, 0, sizeof(float), m->stream);
    if (e == cudaSuccess) e = training_pass(m, n, m->H[0], dY, nullptr, m->loss, m->grad, AdamArgs{});
    float l = 0.f;
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(grads, m->grad, (size_t)m->nparam * sizeof(float), cudaMemcpyDeviceToHost, m->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&l, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
    cudaFree(dX);
    cudaFree(dY);
    MCK(e, "gradients");
    if (loss) *loss = l;
    return umma_check(m);
}

pt_status pt_mlp_predict(pt_mlp *m, const float *X, int n, float *Y)
{
    if (!m || !X || !Y || n < 0) return PT_ERR_ARG;
    return pt_mlp_predict_ensemble(&m, 1, X, n, Y);
}

pt_status pt_mlp_set_tcgen05(pt_mlp *m, int enabled)
{
    if (!m) return PT_ERR_ARG;
    m->use_umma = enabled ? 1 : 0;
    return PT_OK;
}

pt_status pt_mlp_predict_ensemble(pt_mlp *const *members, int count, const float *X, int n, float *Y)
{
    if (!members || count < 1 || !X || !Y || n < 0) return PT_ERR_ARG;
    int chunk = 0;
    pt_status st = ensemble_check(members, count, &chunk);
    if (st != PT_OK) return st;
    pt_mlp *m = members[0];
    const int din = m->width[0], dout = m->width[m->L];
    const cudaStream_t s = m->stream;
    if (!m->xin) MCK(dalloc(m, &m->xin, (size_t)m->max_batch * din), "inference input");
    float *dX = m->xin, *dY = m->Z[m->L - 1];   // chunk <= m->max_batch rows
    cudaError_t e = cudaSuccess;
    for (int s0 = 0; s0 < n && e == cudaSuccess; s0 += chunk) {
        const int B = std::min(chunk, n - s0);
        e = cudaMemcpyAsync(dX, X + (size_t)s0 * din, (size_t)B * din * sizeof(float), cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) e = ensemble_chunk(members, count, B, dX, dY, s);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(Y + (size_t)s0 * dout, dY, (size_t)B * dout * sizeof(float), cudaMemcpyDeviceToHost, s);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    MCK(e, "predict");
    for (int j = 0; j < count && st == PT_OK; j++) st = umma_check(members[j]);
    return st;
}

pt_status pt_mlp_predict_ensemble_device(pt_mlp *const *members, int count, const float *X, int n, float *Y)
{
    if (!members || count < 1 || !X || !Y || n < 0) return PT_ERR_ARG;
    int chunk = 0;
    pt_status st = ensemble_check(members, count, &chunk);
    if (st != PT_OK) return st;
    pt_mlp *m = members[0];
    const int din = m->width[0], dout = m->width[m->L];
    for (int s0 = 0; s0 < n; s0 += chunk) {
        const int B = std::min(chunk, n - s0);
        MCK(ensemble_chunk(members, count, B, X + (size_t)s0 * din, Y + (size_t)s0 * dout, m->stream),
            "ensemble predict (device)");
    }
    return PT_OK;
}

void pt_mlp_destroy(pt_mlp *m)
{
    if (!m) return;
    // (not the device, which is forbidden while any stream is being captured)
    bool idle = cudaStreamSynchronize(m->stream) == cudaSuccess;
    for (void *p : m->allocs) idle = cudaFree(p) == cudaSuccess && idle;   // (waits for other streams' use, too)
    ptm::mapped_give(m->err_word, idle);
    delete m;
}

const char *pt_mlp_last_error(const pt_mlp *m) { return m ? m->err.c_str() : g_mlp_create_error.c_str(); }

}  // extern "C"
