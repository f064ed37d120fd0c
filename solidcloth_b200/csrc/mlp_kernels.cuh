// mlp_kernels.cuh — the learned warm start: a per-particle MLP
// 12 -> 64 -> 64 -> 64 -> 3 (GELU) that predicts the Gauss-Seidel correction of a
// substep from 1-ring features, so that plain iterations start closer to the
// solution. It has no counterpart in the reference; the plain iterations still
// run after it, and the residual target decides when a substep is done.
//
// Every contraction runs on the fifth-generation tensor cores (tc05.cuh): tiles
// of 128 particles (rows) per CTA, BF16 operands staged in shared memory, FP32
// accumulators in tensor memory, one thread issuing tcgen05.mma and the CTA
// waiting on an mbarrier that tcgen05.commit arrives on; the eight warps read
// 32 rows by 32 columns each back with tcgen05.ld for the bias / GELU epilogue,
// which writes the next layer's BF16 operand tile.
//
// What bounds it: the GELU's tanhf (192 a row, about 30 instructions each, against
// 2 x 9,200 multiply-adds that the tensor cores do in passing) and the chain of
// layers of a tile. Eight warps instead of four a tile halve the epilogue of every
// layer; the weights of layers 2 to 4 are staged, eight at a time, behind layer 1's
// product. The training pass keeps the GELU's derivative from the forward epilogue
// in shared memory instead of taking tanhf again. 65,536 rows: forward 31 ->
// 25 us, gradients and Adam 175 -> 115 us (61 with the GELU form and the vector
// reductions below). Training runs the same forward, then the
// backward on the tensor cores too: dH = dZ W (K-major operands, transposed
// weights in shared memory) and dW = dZ^T H (the activation tiles read
// MN-major, summed over the CTA's tiles in tensor memory before one atomic
// pass). Adam updates the FP32 master weights. Included by step_kernels.cu (the
// features use the collider queries defined there).
#pragma once
#include <cuda_bf16.h>
#include "tc05.cuh"

namespace sc {

constexpr int ML_IN = 12, ML_H = 64, ML_OUT = 3;
// FP32 parameter vector: W[out][in] row-major per layer, then the biases
constexpr int ML_W1 = 0, ML_B1 = ML_W1 + ML_H * ML_IN;
constexpr int ML_W2 = ML_B1 + ML_H, ML_B2 = ML_W2 + ML_H * ML_H;
constexpr int ML_W3 = ML_B2 + ML_H, ML_B3 = ML_W3 + ML_H * ML_H;
constexpr int ML_W4 = ML_B3 + ML_H, ML_B4 = ML_W4 + ML_OUT * ML_H;
constexpr int ML_NPARAM = ML_B4 + ML_OUT;     // 9347
constexpr int ML_NNORM = 2 * ML_IN + ML_OUT;  // feature mean, feature 1/std, output scale
constexpr int ML_ROWS = 128;                  // rows (particles / samples) per tile = MMA M
constexpr int ML_THREADS = 256;               // row threadIdx.x & 127, columns 32 (threadIdx.x >> 7) onwards

// instruction descriptors: M = 128 rows, N = 64 hidden units or 16 (padded outputs
// / padded inputs); forward and dH operands K-major, weight-gradient operands MN-major
constexpr uint32_t IDESC_N64 = umma_idesc(128, 64, 0, 0);
constexpr uint32_t IDESC_N16 = umma_idesc(128, 16, 0, 0);
constexpr uint32_t IDESC_GRAD_N64 = umma_idesc(128, 64, 1, 1);
constexpr uint32_t IDESC_GRAD_N16 = umma_idesc(128, 16, 1, 1);

// BF16 weights in core layout: forward operands W[out][in] (layer 1 inputs padded
// to 16, layer 4 outputs padded to 16) and, for training, the transposes
// W^T[in][out] of layers 2-4 (layer 4's outputs padded to 16)
struct __align__(128) MlpTcWeights
{
    unsigned char w1[64 * 16 * 2];
    unsigned char w2[64 * 64 * 2];
    unsigned char w3[64 * 64 * 2];
    unsigned char w4[16 * 64 * 2];
    float b1[ML_H], b2[ML_H], b3[ML_H], b4[16];
    float mean[ML_IN], istd[ML_IN], oscale[ML_OUT];
};
struct __align__(128) MlpTcTrans
{
    unsigned char w2t[64 * 64 * 2];
    unsigned char w3t[64 * 64 * 2];
    unsigned char w4t[64 * 16 * 2];
};

__device__ __forceinline__ void put_bf16(unsigned char* tile, int r, int k, int K, float v)
{
    *reinterpret_cast<__nv_bfloat16*>(tile + core_off(r, k, K)) = __float2bfloat16_rn(v);
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);   // .x = lo (lower 16 bits)
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ void put_chunk8(unsigned char* tile, int r, int k, int K, const float* x)
{
    uint4 q;
    q.x = pack_bf16(x[0], x[1]); q.y = pack_bf16(x[2], x[3]); q.z = pack_bf16(x[4], x[5]); q.w = pack_bf16(x[6], x[7]);
    *reinterpret_cast<uint4*>(tile + core_off(r, k, K)) = q;
}
// eight consecutive floats; the caller's vector may start at any float
__device__ __forceinline__ void ld8(const float* p, float* x)
{
    if ((reinterpret_cast<unsigned long long>(p) & 15ull) == 0ull)
    {
        const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
    }
    else
        for (int k = 0; k < 8; k++) x[k] = __ldg(p + k);
}

// what layer 1 needs, and the rest: 64 x 64 matrices in chunks of eight along a row
__device__ __forceinline__ void mlp_tc_load_first(MlpTcWeights& s, const float* prm, const float* norm)
{
    for (int k = threadIdx.x; k < 64 * 16; k += blockDim.x)
    {
        const int o = k / 16, i = k % 16;
        put_bf16(s.w1, o, i, 16, i < ML_IN ? prm[ML_W1 + o * ML_IN + i] : 0.f);
    }
    if (threadIdx.x < ML_IN) { s.mean[threadIdx.x] = norm[threadIdx.x]; s.istd[threadIdx.x] = norm[ML_IN + threadIdx.x]; }
    if (threadIdx.x < ML_OUT) s.oscale[threadIdx.x] = norm[2 * ML_IN + threadIdx.x];
}

__device__ __forceinline__ void mlp_tc_load_rest(MlpTcWeights& s, MlpTcTrans* t, const float* prm)
{
#pragma unroll
    for (int k = threadIdx.x; k < 512; k += ML_THREADS)
    {
        const int o = k >> 3, i = (k & 7) * 8;
        float a[8], b[8];
        ld8(prm + ML_W2 + o * 64 + i, a);
        ld8(prm + ML_W3 + o * 64 + i, b);
        put_chunk8(s.w2, o, i, 64, a);
        put_chunk8(s.w3, o, i, 64, b);
    }
    if (t)
#pragma unroll
        for (int k = threadIdx.x; k < 512; k += ML_THREADS)
        {
            // the transposes: eight outputs of one input (neighbouring threads: neighbouring inputs)
            const int i = k & 63, o = (k >> 6) * 8;
            float a[8], b[8];
            for (int j = 0; j < 8; j++) { a[j] = __ldg(prm + ML_W2 + (o + j) * 64 + i); b[j] = __ldg(prm + ML_W3 + (o + j) * 64 + i); }
            put_chunk8(t->w2t, i, o, 64, a);
            put_chunk8(t->w3t, i, o, 64, b);
        }
    for (int k = threadIdx.x; k < 16 * 64; k += blockDim.x)
    {
        const int o = k / 64, i = k % 64;
        const float w = o < ML_OUT ? prm[ML_W4 + o * ML_H + i] : 0.f;
        put_bf16(s.w4, o, i, 64, w);
        if (t) put_bf16(t->w4t, i, o, 16, w);
    }
    for (int k = threadIdx.x; k < ML_H; k += blockDim.x)
    {
        s.b1[k] = prm[ML_B1 + k]; s.b2[k] = prm[ML_B2 + k]; s.b3[k] = prm[ML_B3 + k];
    }
    if (threadIdx.x < 16) s.b4[threadIdx.x] = threadIdx.x < ML_OUT ? prm[ML_B4 + threadIdx.x] : 0.f;
}

// GELU, tanh form (inference). The form below was measured here too: 24.6 -> 22.5 us at
// 65,536 rows, but it moves last bits, which the BF16 rounding of the next layer's
// operand turns into one part in 256 here and there.
__device__ __forceinline__ float gelu(float x)
{
    const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
    return 0.5f * x * (1.f + tanhf(u));
}
// The value and the derivative (training): 0.5 x (1 + tanh u) = x / (1 + exp(-2 u)).
// With e = exp(-2 |u|) and the logistic tail q = e / (1 + e) it is x - x q for x >= 0 and
// x q below: one exponential and one reciprocal of the special-function unit (about 2 ulp
// each) in the place of tanhf's two branches of some 30 instructions. The unit's error
// reaches the result only through |x| q <= 0.17, and neither 1 + tanh for negative x nor
// 1 - tanh^2 cancels: over [-9, 9] the largest errors against 64 bits are 2.4e-7 (value)
// and 1.8e-7 (derivative) where the tanhf form has 4.3e-7 and 5.6e-7. 65,536 rows,
// gradients and Adam, with add_columns below: 113 -> 61 us.
__device__ __forceinline__ float gelu_and_grad(float x, float& grad)
{
    const float x2 = x * x;
    // -2 |u| log2(e): the constants are -2 log2(e) sqrt(2/pi) and 0.044715 times that
    const float k = fabsf(x) * __fmaf_rn(-0.10294324f, x2, -2.3022082f);
    float e, r;
    asm("ex2.approx.f32 %0, %1;" : "=f"(e) : "f"(k));
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(1.f + e));
    const float q = e * r;
    // s + x s (1 - s) (2 u)', where s and 1 - s are q and r
    grad = __fmaf_rn(x * q * r, __fmaf_rn(0.21406445f, x2, 1.5957691f), x >= 0.f ? 1.f - q : q);
    // the bound keeps +inf: 0 times it would be NaN
    return x >= 0.f ? __fmaf_rn(-fminf(x, 3e38f), q, x) : x * q;
}

// this thread's row of a 16-column operand tile (K = 16) from 16 floats
__device__ __forceinline__ void put_row16(unsigned char* tile, int r, const float* x)
{
    uint4 q0, q1;
    q0.x = pack_bf16(x[0], x[1]); q0.y = pack_bf16(x[2], x[3]); q0.z = pack_bf16(x[4], x[5]); q0.w = pack_bf16(x[6], x[7]);
    q1.x = pack_bf16(x[8], x[9]); q1.y = pack_bf16(x[10], x[11]); q1.z = pack_bf16(x[12], x[13]); q1.w = pack_bf16(x[14], x[15]);
    *reinterpret_cast<uint4*>(tile + core_off(r, 0, 16)) = q0;
    *reinterpret_cast<uint4*>(tile + core_off(r, 8, 16)) = q1;
}

// 32 accumulator columns of this thread's row (tensor memory at taddr) plus bias,
// through GELU, into columns [c0, c0 + 32) of row r of a K-column operand tile;
// GRAD: the derivatives to grad, [column][row]
template <bool GRAD>
__device__ __forceinline__ void epilogue_gelu32(uint32_t taddr, const float* bias, unsigned char* tile, int r, int c0, int K, float* grad)
{
    uint32_t v[32];
    tc_ld32(taddr, v);
    tc_wait_ld();
#pragma unroll
    for (int c = 0; c < 4; c++)
    {
        float h[8];
#pragma unroll
        for (int j = 0; j < 8; j++)
        {
            const int col = c0 + 8 * c + j;
            const float x = __uint_as_float(v[8 * c + j]) + bias[col];
            if constexpr (GRAD) { float g; h[j] = gelu_and_grad(x, g); grad[col * ML_ROWS + r] = g; }
            else h[j] = gelu(x);
        }
        put_chunk8(tile, r, c0 + 8 * c, K, h);
    }
}

// Shared state of a CTA driving the tensor cores: the mbarrier the commits arrive
// on, its next parity, and the tensor-memory base.
struct TcCtx
{
    uint32_t mbar, phase, tmem;
    bool ok;
    __device__ __forceinline__ bool wait()
    {
        const bool done = mbar_wait(mbar, phase);
        phase ^= 1u;
        tc_fence_after();
        return __syncthreads_and(done) != 0;   // every thread takes the same path
    }
};

// Forward of the CTA's 128-row tile whose normalised inputs (BF16, K = 16) are
// already in x: hidden layers into tensor-memory columns zcol[0..2] (pre-
// activations, no bias), their GELU outputs as operand tiles h[0..2] (each may be
// the same buffer when they need not survive), outputs into column ycol; GRAD:
// the three layers' GELU derivatives into grad. `behind` runs between layer 1's
// issue and its wait. Returns false if a wait gave up.
template <bool GRAD, class F>
__device__ __forceinline__ bool mlp_tc_forward(TcCtx& t, const MlpTcWeights& s, unsigned char* x, unsigned char* const* h,
                                               const uint32_t* zcol, uint32_t ycol, float* grad, F&& behind)
{
    const int r = threadIdx.x & (ML_ROWS - 1), c0 = 32 * (threadIdx.x >> 7);
    const uint32_t lanes = tmem_lane_base(t.tmem);
    tc_sync_for_mma();
    if (threadIdx.x == 0)
    {
        umma_bf16(t.tmem + zcol[0], desc_kmajor(smem_addr(x), 16), desc_kmajor(smem_addr(s.w1), 16), IDESC_N64, 0);
        umma_commit(t.mbar);
    }
    behind();
    if (!t.wait()) return false;
    const float* bias[3] = {s.b1, s.b2, s.b3};
    const unsigned char* w[3] = {s.w2, s.w3, s.w4};
#pragma unroll
    for (int l = 0; l < 3; l++)
    {
        epilogue_gelu32<GRAD>(lanes + zcol[l] + c0, bias[l], h[l], r, c0, 64, GRAD ? grad + l * ML_H * ML_ROWS : nullptr);
        tc_sync_for_mma();
        if (threadIdx.x == 0)
        {
            const uint32_t dst = l < 2 ? zcol[l + 1] : ycol;
            for (int ks = 0; ks < 4; ks++)
                umma_bf16(t.tmem + dst, desc_kmajor(smem_addr(h[l]) + 256 * ks, 64), desc_kmajor(smem_addr(w[l]) + 256 * ks, 64),
                          l < 2 ? IDESC_N64 : IDESC_N16, ks > 0);
            umma_commit(t.mbar);
        }
        if (!t.wait()) return false;
    }
    return true;
}

// the outputs (before the output scale) of this thread's row
__device__ __forceinline__ void mlp_tc_outputs(const TcCtx& t, const MlpTcWeights& s, uint32_t ycol, float* y)
{
    uint32_t v[16];
    tc_ld16(tmem_lane_base(t.tmem) + ycol, v);
    tc_wait_ld();
    for (int k = 0; k < ML_OUT; k++) y[k] = __uint_as_float(v[k]) + s.b4[k];
}

// CTA set-up of the inference kernels: weights, mbarrier, 128 tensor-memory columns
struct __align__(128) MlpTcInferSmem
{
    MlpTcWeights w;
    unsigned char x[ML_ROWS * 16 * 2];
    unsigned char h[ML_ROWS * 64 * 2];
    unsigned long long mbar;
    uint32_t tmemSlot;
};

__device__ __forceinline__ TcCtx mlp_tc_begin(MlpTcInferSmem& s, uint32_t cols)
{
    TcCtx t;
    if (threadIdx.x == 0) mbar_init(smem_addr(&s.mbar), 1);
    t.tmem = tmem_alloc(&s.tmemSlot, cols);    // includes a CTA barrier
    t.mbar = smem_addr(&s.mbar);
    t.phase = 0;
    t.ok = true;
    return t;
}

// ------------------------------------------------------------- features
// The 12 inputs of particle i after the substep's prediction: predicted minus
// previous position (3), velocity (3), mean strain of its incident edges (1),
// collision-mesh normal (3), signed distance to its first sphere / SDF collider
// (1, clamped to +-1 m), and — the twelfth, chosen here — the previous
// substep's solver correction along that normal (1): corrections are coherent
// in time, and the normal component carries the contact response.
__device__ __forceinline__ void ml_features(const DevCloth& c, const Buffers& b, int i, float* f)
{
    const float4 p = c.pos[i], q = c.prev[i], v = c.vel[i];
    f[0] = p.x - q.x; f[1] = p.y - q.y; f[2] = p.z - q.z;
    f[3] = v.x; f[4] = v.y; f[5] = v.z;
    float strain = 0.f;
    const int r0 = c.eRingStart[i], r1 = c.eRingStart[i + 1];
    for (int k = r0; k < r1; k++)
    {
        const int e = c.eRing[k];
        const int4 ed = c.edge[e];
        const int j = ed.x == i ? ed.y : ed.x;
        const float4 pj = c.pos[j];
        const float dx = p.x - pj.x, dy = p.y - pj.y, dz = p.z - pj.z;
        strain += sqrtf(dx * dx + dy * dy + dz * dz) / c.edgeRest[e] - 1.f;
    }
    f[6] = r1 > r0 ? strain / (float)(r1 - r0) : 0.f;
    const float4 n = c.prevN[i];
    f[7] = n.x; f[8] = n.y; f[9] = n.z;
    float dist = 1.f;
    const int2 cr = colliders_of(c, b, i);
    for (int ci = cr.x; ci < cr.x + cr.y; ci++)
    {
        const VColl& g = b.vcoll[ci];
        if (g.type != 3 && g.type != 7) continue;
        V3 cp, nn; int fe;
        dist = query_point(g, mk(p.x, p.y, p.z), cp, nn, fe);
        break;
    }
    f[10] = fminf(1.f, fmaxf(-1.f, dist));
    f[11] = c.lastCorr[i];
}

struct MlpArgs
{
    const float* prm;    // ML_NPARAM FP32 master weights
    const float* norm;   // ML_NNORM
};

// warm start: features -> MLP -> position correction, tiles of 128 particles
// (one per thread), CTAs persistent over the tiles; pinned particles are left
// alone. A wait that gives up sets ST_TC_TIMEOUT and ends the CTA's work.
__global__ void __launch_bounds__(ML_THREADS, 4) k_mlp_warm(DevCloth c, Buffers b, MlpArgs ml)
{
    __shared__ MlpTcInferSmem s;
    mlp_tc_load_first(s.w, ml.prm, ml.norm);
    TcCtx t = mlp_tc_begin(s, 128);
    unsigned char* hs[3] = {s.h, s.h, s.h};
    const uint32_t zc[3] = {0, 64, 0};
    const int tiles = (c.N + ML_ROWS - 1) / ML_ROWS;
    bool loaded = false;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x)
    {
        const int i = tile * ML_ROWS + (int)(threadIdx.x & (ML_ROWS - 1));
        if (threadIdx.x < ML_ROWS)
        {
            float f[16];
            if (i < c.N) ml_features(c, b, i, f);
#pragma unroll
            for (int k = 0; k < 16; k++) f[k] = (i < c.N && k < ML_IN) ? (f[k] - s.w.mean[k]) * s.w.istd[k] : 0.f;
            put_row16(s.x, threadIdx.x, f);
        }
        if (!mlp_tc_forward<false>(t, s.w, s.x, hs, zc, 64, nullptr, [&] { if (!loaded) mlp_tc_load_rest(s.w, nullptr, ml.prm); loaded = true; }))
        {
            if (threadIdx.x == 0) atomicOr(c.status, ST_TC_TIMEOUT);
            break;
        }
        if (threadIdx.x < ML_ROWS)
        {
            float y[ML_OUT];
            mlp_tc_outputs(t, s.w, 64, y);
            if (i < c.N)
            {
                float4 p = c.pos[i];
                if (p.w > 0.f)
                {
                    p.x += y[0] * s.w.oscale[0];
                    p.y += y[1] * s.w.oscale[1];
                    p.z += y[2] * s.w.oscale[2];
                    c.pos[i] = p;
                }
            }
        }
    }
    tmem_free(t.tmem, 128);
}

// the predicted positions, and (sample recording) every particle's raw features
__global__ void k_mlp_features(DevCloth c, Buffers b, float* feat)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.N) return;
    if (feat)
    {
        float f[ML_IN];
        ml_features(c, b, i, f);
        for (int k = 0; k < ML_IN; k++) feat[(size_t)i * ML_IN + k] = f[k];
    }
    c.xpred[i] = c.pos[i];
}

// the substep's correction (solved minus predicted positions): its normal
// component for the next substep's features, and (sample recording) the target
__global__ void k_mlp_targets(DevCloth c, float* target)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.N) return;
    const float4 p = c.pos[i], q = c.xpred[i], n = c.prevN[i];
    const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
    c.lastCorr[i] = dx * n.x + dy * n.y + dz * n.z;
    if (target) { target[3 * (size_t)i] = dx; target[3 * (size_t)i + 1] = dy; target[3 * (size_t)i + 2] = dz; }
}

// one raw feature row; the caller's array may start at any float
__device__ __forceinline__ void ld_row12(const float* p, float* f)
{
    if ((reinterpret_cast<unsigned long long>(p) & 15ull) == 0ull)
    {
        const float4* q = reinterpret_cast<const float4*>(p);
        const float4 a = __ldg(q), b = __ldg(q + 1), d = __ldg(q + 2);
        f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
        f[8] = d.x; f[9] = d.y; f[10] = d.z; f[11] = d.w;
    }
    else
        for (int k = 0; k < ML_IN; k++) f[k] = __ldg(p + k);
}

// this tile's normalised inputs into x (rows past S: zero)
__device__ __forceinline__ void put_inputs(const MlpTcWeights& w, unsigned char* x, const float* X, int row, int S)
{
    float f[16];
    if (row < S) ld_row12(X + (size_t)row * ML_IN, f);
#pragma unroll
    for (int k = 0; k < 16; k++) f[k] = (row < S && k < ML_IN) ? (f[k] - w.mean[k]) * w.istd[k] : 0.f;
    put_row16(x, threadIdx.x, f);
}

// forward over raw feature rows (S x 12) -> outputs (S x 3, output scale applied)
__global__ void __launch_bounds__(ML_THREADS, 4) k_mlp_forward(const float* X, int S, MlpArgs ml, float* Y, int* status)
{
    __shared__ MlpTcInferSmem s;
    mlp_tc_load_first(s.w, ml.prm, ml.norm);
    TcCtx t = mlp_tc_begin(s, 128);
    unsigned char* hs[3] = {s.h, s.h, s.h};
    const uint32_t zc[3] = {0, 64, 0};
    const int tiles = (S + ML_ROWS - 1) / ML_ROWS;
    bool loaded = false;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x)
    {
        const int r = tile * ML_ROWS + (int)(threadIdx.x & (ML_ROWS - 1));
        if (threadIdx.x < ML_ROWS) put_inputs(s.w, s.x, X, r, S);
        if (!mlp_tc_forward<false>(t, s.w, s.x, hs, zc, 64, nullptr, [&] { if (!loaded) mlp_tc_load_rest(s.w, nullptr, ml.prm); loaded = true; }))
        {
            if (threadIdx.x == 0 && status) atomicOr(status, 1);
            break;
        }
        if (threadIdx.x < ML_ROWS)
        {
            float y[ML_OUT];
            mlp_tc_outputs(t, s.w, 64, y);
            if (r < S)
                for (int k = 0; k < ML_OUT; k++) Y[(size_t)r * ML_OUT + k] = y[k] * s.w.oscale[k];
        }
    }
    tmem_free(t.tmem, 128);
}

// ------------------------------------------------------------ training
// Sum over a warp of 32 per-lane values: a butterfly in which each step halves the
// columns a lane keeps, so that lane l ends with the sum of column l (31 shuffles
// instead of 32 x 5).
__device__ __forceinline__ float warp_colsum32(const float (&v)[32])
{
    const int lane = threadIdx.x & 31;
    float a[16];
#pragma unroll
    for (int j = 0; j < 16; j++)
    {
        const bool hi = lane & 16;
        a[j] = (hi ? v[j + 16] : v[j]) + __shfl_xor_sync(0xffffffffu, hi ? v[j] : v[j + 16], 16);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
    {
        const bool hi = lane & o;
#pragma unroll
        for (int j = 0; j < 8; j++)
            if (j < o)
            {
                const float keep = hi ? a[j + o] : a[j], send = hi ? a[j] : a[j + o];
                a[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
    }
    return a[0];
}

// dZ = dH * gelu'(Z + b) for 32 columns from c0 of this thread's row: dH from tensor
// memory, the derivatives kept by the forward epilogue; dZ as BF16 into row r of the
// 128-column tile d, and its column sums over the warp into bsum (lane l: column c0 + l)
__device__ __forceinline__ void epilogue_dz(uint32_t lanes, uint32_t dhCol, const float* grad, unsigned char* d, int r, int c0, float& bsum)
{
    float dz[32];
    uint32_t vh[32];
    tc_ld32(lanes + dhCol + c0, vh);
    tc_wait_ld();
#pragma unroll
    for (int j = 0; j < 32; j++) dz[j] = __uint_as_float(vh[j]) * grad[(c0 + j) * ML_ROWS + r];
#pragma unroll
    for (int c = 0; c < 4; c++) put_chunk8(d, r, c0 + 8 * c, 128, dz + 8 * c);
    bsum += warp_colsum32(dz);
}

// N accumulator columns added to consecutive floats: four to a reduction where the
// caller's array allows it. A row of a gradient lies 256 bytes from the next lane's, so
// that each lane's word is a memory transaction of its own.
template <int N>
__device__ __forceinline__ void add_columns(float* g, const uint32_t* v)
{
    if ((reinterpret_cast<unsigned long long>(g) & 15ull) == 0ull)
    {
#pragma unroll
        for (int j = 0; j < N; j += 4)
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" :: "l"(g + j), "f"(__uint_as_float(v[j])),
                         "f"(__uint_as_float(v[j + 1])), "f"(__uint_as_float(v[j + 2])), "f"(__uint_as_float(v[j + 3])) : "memory");
    }
    else
#pragma unroll
        for (int j = 0; j < N; j++) atomicAdd(g + j, __uint_as_float(v[j]));
}

// Tensor-memory columns of the training kernel (512 allocated)
constexpr uint32_t TM_Z1 = 0, TM_Z2 = 64, TM_Z3 = 128, TM_Y = 192, TM_DH = 208;
constexpr uint32_t TM_DW4 = 272, TM_DW3 = 336, TM_DW2 = 400, TM_DW1 = 464;

struct __align__(128) MlpTcTrainSmem
{
    MlpTcWeights w;
    MlpTcTrans t;
    unsigned char x[ML_ROWS * 16 * 2];
    unsigned char h1[ML_ROWS * 64 * 2], h2[ML_ROWS * 64 * 2], h3[ML_ROWS * 64 * 2];
    // dY / dZ tile, 128 columns: 0..63 in use, 64..127 zero (the padded rows of
    // the M = 128 weight-gradient products)
    unsigned char d[ML_ROWS * 128 * 2];
    float grad[3 * ML_H * ML_ROWS];       // GELU derivatives of the three hidden layers, [layer][column][row]
    unsigned long long mbar;
    uint32_t tmemSlot;
};

// Gradients of the mean squared error between the network's output and
// target / output scale (mean over S x 3 elements), accumulated into grad[] and
// loss[0] (both zeroed by the caller). CTAs are persistent over 128-row tiles;
// the weight gradients of all their tiles are summed in tensor memory and added
// to grad[] once per CTA. A wait that gives up sets *status (if given).
__global__ void __launch_bounds__(ML_THREADS) k_mlp_grad(const float* X, const float* T, int S, MlpArgs ml, float* grad,
                                                         float* loss, int* status)
{
    extern __shared__ __align__(1024) unsigned char dyn[];
    MlpTcTrainSmem& s = *reinterpret_cast<MlpTcTrainSmem*>(dyn);
    mlp_tc_load_first(s.w, ml.prm, ml.norm);
    for (int k = threadIdx.x; k < ML_ROWS * 128 * 2 / 16; k += blockDim.x)
        reinterpret_cast<uint4*>(s.d)[k] = make_uint4(0u, 0u, 0u, 0u);
    TcCtx t;
    if (threadIdx.x == 0) mbar_init(smem_addr(&s.mbar), 1);
    t.tmem = tmem_alloc(&s.tmemSlot, 512);
    t.mbar = smem_addr(&s.mbar);
    t.phase = 0;
    const int r = threadIdx.x & (ML_ROWS - 1), lane = threadIdx.x & 31, half = threadIdx.x >> 7, c0 = 32 * half;
    const uint32_t lanes = tmem_lane_base(t.tmem);
    const float inv = 1.f / (float)(S * ML_OUT);
    float db[3] = {0.f, 0.f, 0.f};
    float db4[ML_OUT] = {0.f, 0.f, 0.f}, lsum = 0.f;
    unsigned char* hs[3] = {s.h1, s.h2, s.h3};
    const uint32_t zc[3] = {TM_Z1, TM_Z2, TM_Z3};
    const int tiles = (S + ML_ROWS - 1) / ML_ROWS;
    bool first = true, ok = true;
    for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x)
    {
        const int row = tile * ML_ROWS + r;
        const bool live = row < S;
        if (half == 0) put_inputs(s.w, s.x, X, row, S);
        if (!(ok = mlp_tc_forward<true>(t, s.w, s.x, hs, zc, TM_Y, s.grad, [&] { if (first) mlp_tc_load_rest(s.w, &s.t, ml.prm); }))) break;
        // output layer: dL/dy (zero for rows past S) into dY columns 0..2
        uint4 q0 = make_uint4(0u, 0u, 0u, 0u);
        if (half == 0)
        {
            float y[ML_OUT], dy[ML_OUT] = {0.f, 0.f, 0.f};
            mlp_tc_outputs(t, s.w, TM_Y, y);
            for (int k = 0; k < ML_OUT; k++)
                if (live)
                {
                    const float e = y[k] - T[(size_t)row * ML_OUT + k] / s.w.oscale[k];
                    lsum += e * e * inv;
                    dy[k] = 2.f * e * inv;
                }
            for (int k = 0; k < ML_OUT; k++)
            {
                float v = dy[k];
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                db4[k] += v;
            }
            q0.x = pack_bf16(dy[0], dy[1]); q0.y = pack_bf16(dy[2], 0.f);
        }
        for (int c = 0; c < 4; c++)
            *reinterpret_cast<uint4*>(s.d + core_off(r, c0 + 8 * c, 128)) = c == 0 ? q0 : make_uint4(0u, 0u, 0u, 0u);
        // dH3 = dY W4 (K = 16) and dW4 += dY^T H3 (sum over the tile's rows)
        tc_sync_for_mma();
        if (threadIdx.x == 0)
        {
            umma_bf16(t.tmem + TM_DH, desc_kmajor(smem_addr(s.d), 128), desc_kmajor(smem_addr(s.t.w4t), 16), IDESC_N64, 0);
            for (int ks = 0; ks < ML_ROWS / 16; ks++)
                umma_bf16(t.tmem + TM_DW4, desc_mnmajor(smem_addr(s.d) + ks * 2 * 2048, 128),
                          desc_mnmajor(smem_addr(s.h3) + ks * 2 * 1024, 64), IDESC_GRAD_N64, (!first || ks > 0) ? 1u : 0u);
            umma_commit(t.mbar);
        }
        if (!(ok = t.wait())) break;
        // hidden layers 3, 2, 1: dZ, then dH of the layer below and dW += dZ^T H
        const unsigned char* wt[3] = {nullptr, s.t.w2t, s.t.w3t};
        const uint32_t dwc[3] = {TM_DW1, TM_DW2, TM_DW3};
#pragma unroll
        for (int l = 2; l >= 0; l--)
        {
            if (!ok) break;
            epilogue_dz(lanes, TM_DH, s.grad + l * ML_H * ML_ROWS, s.d, r, c0, db[l]);
            tc_sync_for_mma();
            if (threadIdx.x == 0)
            {
                if (l > 0)
                    for (int ks = 0; ks < 4; ks++)
                        umma_bf16(t.tmem + TM_DH, desc_kmajor(smem_addr(s.d) + 256 * ks, 128),
                                  desc_kmajor(smem_addr(wt[l]) + 256 * ks, 64), IDESC_N64, ks > 0);
                const unsigned char* hb = l > 0 ? hs[l - 1] : s.x;
                const int hk = l > 0 ? 64 : 16;
                for (int ks = 0; ks < ML_ROWS / 16; ks++)
                    umma_bf16(t.tmem + dwc[l], desc_mnmajor(smem_addr(s.d) + ks * 2 * 2048, 128),
                              desc_mnmajor(smem_addr(hb) + ks * 2 * hk * 16, hk), l > 0 ? IDESC_GRAD_N64 : IDESC_GRAD_N16,
                              (!first || ks > 0) ? 1u : 0u);
                umma_commit(t.mbar);
            }
            ok = t.wait();
        }
        first = false;
    }
    if (!ok && threadIdx.x == 0 && status) atomicOr(status, 1);
    // this CTA's sums: weight gradients (rows 0..63 = output units), bias gradients
    // (lane l: unit c0 + l), loss. Tensor-memory loads are warp-collective: every warp
    // loads its half of the columns, the warps holding rows 0..63 add them.
    if (ok && !first)
    {
        const bool mine = r < 64;
        uint32_t v[32];
        tc_ld32(lanes + TM_DW3 + c0, v);
        tc_wait_ld();
        if (mine) add_columns<32>(&grad[ML_W3 + r * ML_H + c0], v);
        tc_ld32(lanes + TM_DW2 + c0, v);
        tc_wait_ld();
        if (mine) add_columns<32>(&grad[ML_W2 + r * ML_H + c0], v);
        tc_ld32(lanes + TM_DW4 + c0, v);
        tc_wait_ld();
        if (r < ML_OUT) add_columns<32>(&grad[ML_W4 + r * ML_H + c0], v);
        if (half == 0)
        {
            uint32_t v16[16];
            tc_ld16(lanes + TM_DW1, v16);
            tc_wait_ld();
            if (mine) add_columns<ML_IN>(&grad[ML_W1 + r * ML_IN], v16);
        }
        atomicAdd(&grad[ML_B1 + c0 + lane], db[0]);
        atomicAdd(&grad[ML_B2 + c0 + lane], db[1]);
        atomicAdd(&grad[ML_B3 + c0 + lane], db[2]);
        if (half == 0)
        {
            if (lane == 0)
                for (int k = 0; k < ML_OUT; k++) atomicAdd(&grad[ML_B4 + k], db4[k]);
            for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
            if (lane == 0) atomicAdd(loss, lsum);
        }
    }
    tmem_free(t.tmem, 512);
}

// Adam (Kingma & Ba 2015) on the FP32 master weights; m and v follow the parameters
__global__ void k_adam(float* prm, const float* grad, float* m, float* v, int step, float lr, float b1, float b2, float eps)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= ML_NPARAM) return;
    const float g = grad[k];
    const float mk = b1 * m[k] + (1.f - b1) * g;
    const float vk = b2 * v[k] + (1.f - b2) * g * g;
    m[k] = mk; v[k] = vk;
    const float mh = mk / (1.f - powf(b1, (float)step)), vh = vk / (1.f - powf(b2, (float)step));
    prm[k] -= lr * mh / (sqrtf(vh) + eps);
}

} // namespace sc
