// Learned thin absorbing boundary: stencil gather, the boundary MLP's training kernels
// (forward, backward, Adam), its inference kernels and the boundary fix-up of the Yee updates.
//
// The boundary model: on every face with the learned layer, each column (one cell of the face's
// plane) reads the six field components on a 3 x 3 tangential patch two cells deep, scales
// them by their RMS r (Maxwell's equations are linear, so scaling the fields by a scales the
// answer by a: dividing by r makes the network's job amplitude-free), and a 108 -> 64 -> 64 -> 6
// MLP with GELU returns the fields of the ghost cell just outside the face, times r. The grid's
// own edges wrap; the fix-up replaces, in the updates of the outermost cells, the wrapped
// neighbour by the ghost (H ghosts outside side-0 faces for the E update, E ghosts outside
// side-1 faces for the H update), which is what a wave leaving the grid needs from the CPML
// layers that the learned layer replaces.
//
// Training runs in float32 on the CUDA cores: blocks of 32 samples for the per-sample passes and a
// split reduction over samples for the weight gradients (deterministic: fixed partition, fixed
// folding order). Inference uses bfloat16 weights on
// the tensor cores (mma.sync, float32 accumulation) or float32 weights on the CUDA cores.
#include <cuda_bf16.h>

#include "lbc.h"
#include "yee_common.cuh"

namespace fdtd {

namespace {

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }

__device__ __forceinline__ float gelu_d(float x)
{
    return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

__device__ __forceinline__ uint32_t clampu(int v, uint32_t n) { return (uint32_t)(v < 0 ? 0 : (v >= (int)n ? (int)n - 1 : v)); }

// cell coordinates of column (u, v) of face f at depth d with tangential offset (du, dv)
__device__ __forceinline__ uint64_t cell_of(const LGrid &g, const LFace &f, uint32_t u, uint32_t v, int d,
                                            int du, int dv)
{
    const int a = f.axis, ua = a == 0 ? 1 : 0, va = a == 2 ? 1 : 2;
    uint32_t c[3];
    c[a] = f.side ? g.s[a] - 1u - (uint32_t)d : (uint32_t)d;
    c[ua] = clampu((int)u + du, g.s[ua]);
    c[va] = clampu((int)v + dv, g.s[va]);
    return ((uint64_t)c[0] * g.s[1] + c[1]) * g.s[2] + c[2];
}

__device__ __forceinline__ bool in_window(const LGrid &g, int fi, uint32_t u, uint32_t v)
{
    return u >= g.win[fi][0] && u < g.win[fi][1] && v >= g.win[fi][2] && v < g.win[fi][3];
}

__device__ __forceinline__ int face_of(const LGrid &g, uint32_t col)
{
    int f = 0;
    while (f + 1 < g.nface && col >= g.face[f + 1].col0) ++f;
    return f;
}

// the 108 stencil values of a column; returns their RMS
__device__ __forceinline__ float gather(const LGrid &g, const LFace &f, uint32_t u, uint32_t v, const float *E,
                                        const float *H, float *x)
{
    float ss = 0.f;
    int k = 0;
#pragma unroll
    for (int d = 0; d < 2; ++d)
#pragma unroll
        for (int du = -1; du <= 1; ++du)
#pragma unroll
            for (int dv = -1; dv <= 1; ++dv) {
                const uint64_t i = cell_of(g, f, u, v, d, du, dv);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const float e = E[c * g.N + i], h = H[c * g.N + i];
                    x[k + c] = e;
                    x[k + 3 + c] = h;
                    ss += e * e + h * h;
                }
                k += 6;
            }
    return sqrtf(ss * (1.0f / LBC_IN));
}

// ---- stencil gather: normalised inputs, their scale, the depth-0 centre values -----------------
__global__ void k_lbc_gather(const LGrid g, const float *E, const float *H, float *X, float *R, float *C)
{
    const uint32_t col = blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= g.ncol) return;
    const LFace &f = g.face[face_of(g, col)];
    const uint32_t c = col - f.col0;
    const uint32_t u = f.u0 + c / f.nv, v = f.v0 + c % f.nv;
    float x[LBC_IN];
    const float r = gather(g, f, u, v, E, H, x);
    const float inv = r > 0.f ? 1.0f / r : 0.f;
    if (X)
        for (int k = 0; k < LBC_IN; ++k) X[(uint64_t)col * LBC_IN + k] = x[k] * inv;
    if (R) R[col] = r;
    if (C) {
        // depth 0, du = dv = 0: stencil entry ((0 * 3 + 1) * 3 + 1) * 6
        for (int k = 0; k < LBC_OUT; ++k) C[(uint64_t)col * LBC_OUT + k] = x[24 + k];
    }
}

// ---- training kernels (float32) -----------------------------------------------------------------
// A batch of 4096 samples is 0.23 GFLOP and 9 MB: a few microseconds of the chip's float32 units, so
// what costs time is how much of the chip works and how long the serial chain of a block is. One
// thread per sample (32 blocks of 128 threads, 2.4% of the chip's threads) took 61 us forward and 46
// us backward, and the weight gradients (16 blocks) 265 us. Now a block has 32 samples and 128
// threads, each 4 samples x 4 units (16 independent sums; every value read from shared memory is
// used four times), and the weight gradients are split by input row as well as by sample. The order of
// every sum is the one of the per-sample form, so outputs and gradients are the same bits.
constexpr int TR_ROWS = 32;      // samples of a block
constexpr int TR_T = 128;        // threads: 8 row groups (4 samples each) x 16 unit lanes (4 units each)
constexpr int TR_LD = LBC_HID + 4;   // row pitch of hidden values and of W2: the rows that the lanes of
                                     // a warp read at once lie in different banks
// the parameters in shared memory: as in the vector, W2's rows TR_LD apart
constexpr int SW_W2 = LBC_W2, SW_B2 = SW_W2 + LBC_HID * TR_LD, SW_W3 = SW_B2 + LBC_HID, SW_B3 = SW_W3 + LBC_HID * LBC_OUT;
constexpr int SW_N = (SW_B3 + LBC_OUT + 3) / 4 * 4;
constexpr size_t ROWS_SMEM = (size_t)(SW_N + TR_ROWS * (LBC_IN + TR_LD)) * sizeof(float);
static_assert(LBC_W2 % 4 == 0 && LBC_IN % 4 == 0 && TR_LD % 4 == 0, "16-byte rows in shared memory");

// asynchronous 4-byte copy to shared memory (any float pointer is aligned for it); 0 when !in
__device__ __forceinline__ void copy4(float *dst, const float *src, bool in)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int n = in ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// acc[4 samples][4 units] += in[sample][k] w[k][unit], k ascending; the thread's units are u, u + 16, ...
template <int K, int PITCH, int WPITCH>
__device__ __forceinline__ void dense(float (&acc)[4][4], const float *in, const float *w, int u)
{
#pragma unroll 3
    for (int k = 0; k < K; k += 4) {
        float x[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) *reinterpret_cast<float4 *>(x[i]) = *reinterpret_cast<const float4 *>(in + i * PITCH + k);
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float wj = w[(k + q) * WPITCH + u + 16 * j];
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[i][j] += x[i][q] * wj;
            }
    }
}

// acc[4 samples][4 units] += d[sample][k] w2[unit][k], k ascending (both TR_LD pitch)
__device__ __forceinline__ void back_dense(float (&acc)[4][4], const float *d, const float *w2, int u)
{
#pragma unroll 2
    for (int k = 0; k < LBC_HID; k += 4) {
        float4 x[4], v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const float4 *>(d + i * TR_LD + k);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = *reinterpret_cast<const float4 *>(w2 + (u + 16 * j) * TR_LD + k);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                acc[i][j] += x[i].x * v[j].x;
                acc[i][j] += x[i].y * v[j].y;
                acc[i][j] += x[i].z * v[j].z;
                acc[i][j] += x[i].w * v[j].w;
            }
    }
}

// The forward pass of 32 samples. GRAD: and the gradient of the loss with respect to every layer's
// pre-activations (DY, D2, D1), which stay in registers on the way, with the block's share of the loss:
// loss = scale * sum over the batch and the outputs of w_o (Y - T)^2 (scale = 1 / (B * 6) for the mean,
// w_o = 1 without wout). 4096 samples: 10.8 us forward, and 22 us for the backward pass as a launch of
// its own, which waits for the activations and the weights again.
struct RowsK {
    const float *P, *X;
    int B;
    float *Y, *A1, *A2, *H1, *H2;                            // Y, A1, A2: without GRAD
    const float *T, *wout;                                   // from here on: GRAD
    float scale;
    float *DY, *D2, *D1, *loss;                              // loss: one partial sum per block
};

template <bool GRAD>
__global__ void __launch_bounds__(TR_T) k_mlp_rows(const __grid_constant__ RowsK g)
{
    extern __shared__ __align__(16) float mlp_smem[];
    float *const w = mlp_smem;
    float *const xs = w + SW_N;                              // [TR_ROWS][LBC_IN]; then D2 [TR_ROWS][TR_LD]
    float *const hs = xs + TR_ROWS * LBC_IN;                 // [TR_ROWS][TR_LD]
    __shared__ float dy[TR_ROWS * LBC_OUT];
    __shared__ float part[TR_T / 32];
    const float *const P = g.P;
    const int t = threadIdx.x, u = t & 15, s0 = (t >> 4) * 4;
    const int r0 = blockIdx.x * TR_ROWS, nr = min(TR_ROWS, g.B - r0);
    grid_dependency_sync();
    // the first layer's operands first: the other layers' weights arrive behind its arithmetic
    for (int i = t; i < TR_ROWS * LBC_IN; i += TR_T) {
        const bool in = i < nr * LBC_IN;
        copy4(xs + i, g.X + (uint64_t)r0 * LBC_IN + (in ? i : 0), in);
    }
    for (int i = t; i < LBC_W2; i += TR_T) copy4(w + i, P + i, true);
    copy_commit();
    for (int i = t; i < LBC_HID * LBC_HID; i += TR_T) copy4(w + SW_W2 + i / LBC_HID * TR_LD + i % LBC_HID, P + LBC_W2 + i, true);
    for (int i = t; i < LBC_NPARAM - LBC_B2; i += TR_T) copy4(w + SW_B2 + i, P + LBC_B2 + i, true);
    copy_commit();
    copy_wait<1>();
    __syncthreads();
    float acc[4][4], a1[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = w[LBC_B1 + u + 16 * j];
    dense<LBC_IN, LBC_IN, LBC_HID>(acc, xs + s0 * LBC_IN, w + LBC_W1, u);
    // a layer's outputs: to the arrays and, activated, to shared memory for the next layer
    const auto put = [&](float *A, float *Hh) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float hj = gelu(acc[i][j]);
                hs[(s0 + i) * TR_LD + u + 16 * j] = hj;
                if (s0 + i < nr) {
                    const uint64_t o = (uint64_t)(r0 + s0 + i) * LBC_HID + u + 16 * j;
                    if (!GRAD) A[o] = acc[i][j];
                    Hh[o] = hj;
                }
            }
    };
    put(g.A1, g.H1);
    copy_wait<0>();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            a1[i][j] = acc[i][j];
            acc[i][j] = w[SW_B2 + u + 16 * j];
        }
    dense<LBC_HID, TR_LD, TR_LD>(acc, hs + s0 * TR_LD, w + SW_W2, u);
    __syncthreads();                                         // every thread has read the first layer's values
    put(g.A2, g.H2);
    __syncthreads();
    float ls = 0.f;
    for (int e = t; e < TR_ROWS * LBC_OUT; e += TR_T) {
        const int r = e / LBC_OUT, o = e - r * LBC_OUT;
        const bool in = r < nr;
        float y = w[SW_B3 + o];
#pragma unroll 8
        for (int k = 0; k < LBC_HID; ++k) y += hs[r * TR_LD + k] * w[SW_W3 + k * LBC_OUT + o];
        const uint64_t ge = (uint64_t)r0 * LBC_OUT + e;
        if (!GRAD && in) g.Y[ge] = y;
        if (GRAD) {
            float v = 0.f;
            if (in) {
                const float wo = g.wout ? g.wout[o] : 1.0f, d = y - g.T[ge];
                v = 2.0f * g.scale * wo * d;
                g.DY[ge] = v;
                ls += d * d * wo;
            }
            dy[e] = v;
        }
    }
    if (!GRAD) return;
#pragma unroll
    for (int m = 16; m; m >>= 1) ls += __shfl_xor_sync(0xffffffffu, ls, m);
    if (!(t & 31)) part[t >> 5] = ls;
    __syncthreads();
    if (!t) g.loss[blockIdx.x] = (part[0] + part[1]) + (part[2] + part[3]);
    static_assert(TR_T == 128, "four warps");
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = s0 + i, c = u + 16 * j;
            float s = 0.f;
#pragma unroll
            for (int o = 0; o < LBC_OUT; ++o) s += dy[r * LBC_OUT + o] * w[SW_W3 + c * LBC_OUT + o];
            const float v = s * gelu_d(acc[i][j]);
            if (r < nr) g.D2[(uint64_t)(r0 + r) * LBC_HID + c] = v;
            xs[r * TR_LD + c] = v;
            acc[i][j] = 0.f;
        }
    __syncthreads();
    back_dense(acc, xs + s0 * TR_LD, w + SW_W2, u);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (s0 + i < nr) g.D1[(uint64_t)(r0 + s0 + i) * LBC_HID + u + 16 * j] = acc[i][j] * gelu_d(a1[i][j]);
}

// ---- training: backward through the activations of a forward pass made earlier --------------------
__global__ void __launch_bounds__(TR_T) k_mlp_bwd_rows(const float *P, const float *Y, const float *T,
                                                       const float *wout, int B, float scale, const float *A1,
                                                       const float *A2, float *DY, float *D2, float *D1)
{
    __shared__ __align__(16) float w2[LBC_HID * TR_LD];
    __shared__ float w3[LBC_HID * LBC_OUT];
    __shared__ float dy[TR_ROWS * LBC_OUT];
    __shared__ __align__(16) float d2[TR_ROWS * TR_LD];
    const int t = threadIdx.x, u = t & 15, s0 = (t >> 4) * 4;
    const int r0 = blockIdx.x * TR_ROWS, nr = min(TR_ROWS, B - r0);
    grid_dependency_sync();
    for (int i = t; i < LBC_HID * LBC_OUT; i += TR_T) copy4(w3 + i, P + LBC_W3 + i, true);
    copy_commit();
    for (int i = t; i < LBC_HID * LBC_HID; i += TR_T) copy4(w2 + i / LBC_HID * TR_LD + i % LBC_HID, P + LBC_W2 + i, true);
    copy_commit();
    // all of the thread's activations at once: loaded where they are used, they cost 16 latencies
    float a1[4][4], a2[4][4], acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint64_t g = (uint64_t)(r0 + min(s0 + i, nr - 1)) * LBC_HID + u + 16 * j;
            a1[i][j] = A1[g];
            a2[i][j] = A2[g];
            acc[i][j] = 0.f;
        }
    for (int e = t; e < TR_ROWS * LBC_OUT; e += TR_T) {
        float v = 0.f;
        if (e < nr * LBC_OUT) {
            const uint64_t g = (uint64_t)r0 * LBC_OUT + e;
            const float wo = wout ? wout[e % LBC_OUT] : 1.0f;
            v = 2.0f * scale * wo * (Y[g] - T[g]);
            DY[g] = v;
        }
        dy[e] = v;
    }
    copy_wait<1>();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = s0 + i, c = u + 16 * j;
            float s = 0.f;
#pragma unroll
            for (int o = 0; o < LBC_OUT; ++o) s += dy[r * LBC_OUT + o] * w3[c * LBC_OUT + o];
            const float v = s * gelu_d(a2[i][j]);
            if (r < nr) D2[(uint64_t)(r0 + r) * LBC_HID + c] = v;
            d2[r * TR_LD + c] = v;
        }
    copy_wait<0>();
    __syncthreads();
    back_dense(acc, d2 + s0 * TR_LD, w2, u);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (s0 + i < nr) D1[(uint64_t)(r0 + s0 + i) * LBC_HID + u + 16 * j] = acc[i][j] * gelu_d(a1[i][j]);
}

// ---- training: weight gradients dW[k][n] = sum_r In[r][k] D[r][n], bias row k = K ------------
// A block sums WG_RPB rows (blockIdx.y) of a tile of WG_KT input rows x NT columns into
// partial[blockIdx.y][(K + 1) * N]; the fold kernel then adds the partials in block order (same
// partition, same order: deterministic). All rows of the tile are requested at once and summed as
// the groups arrive. The layers of the network are tiles of one launch (17 tiles x 16 row blocks for
// 4096 samples), two blocks an SM by shared memory.
constexpr int WG_RPB = 256;      // rows of a block: one float32 chain
constexpr int WG_KT = 16;
constexpr int WG_T = 128;
constexpr int WG_GROUPS = 4;     // groups of rows waited for one after another
constexpr size_t WG_SMEM = (size_t)WG_RPB * (WG_KT + 64) * sizeof(float);

struct WLayer {
    const float *in, *d;         // [rows][K], [rows][N]
    int K, N;
    int tile0;                   // first tile (blockIdx.x); tiles run over n within k
    uint32_t part;               // offset of (k, n) = (0, 0) within a block's partials
};
struct WLayers {
    WLayer l[3];
    int n;
    uint32_t stride;             // partials of a row block
};

// TN columns per thread, NT / TN lanes of columns, TK input rows per thread
template <int NT, int TN>
__device__ __forceinline__ void outer_tile(const WLayer &l, int tile, uint32_t stride, int rows, float *sh, float *partial)
{
    constexpr int LANES = NT / TN, TK = WG_KT / (WG_T / LANES), GR = WG_RPB / WG_GROUPS;
    static_assert(TK >= 1 && TN <= 4, "tile layout");
    const int K = l.K, N = l.N, ntn = (N + NT - 1) / NT;
    const int k0 = tile / ntn * WG_KT, n0 = tile % ntn * NT;
    const int t = threadIdx.x;
    const int r0 = blockIdx.y * WG_RPB, nr = min(WG_RPB, rows - r0);
    float *const si = sh, *const sd = sh + WG_RPB * WG_KT;
    grid_dependency_sync();
#pragma unroll 1
    for (int g = 0; g < WG_GROUPS; ++g) {
        for (int i = t; i < GR * WG_KT; i += WG_T) {
            const int r = g * GR + i / WG_KT, k = k0 + i % WG_KT;
            if (k == K) si[r * WG_KT + i % WG_KT] = r < nr ? 1.f : 0.f;      // the bias row
            else {
                const bool in = r < nr && k < K;
                copy4(si + r * WG_KT + i % WG_KT, l.in + (in ? (uint64_t)(r0 + r) * K + k : 0), in);
            }
        }
        for (int i = t; i < GR * NT; i += WG_T) {
            const int r = g * GR + i / NT, n = n0 + i % NT;
            const bool in = r < nr && n < N;
            copy4(sd + r * NT + i % NT, l.d + (in ? (uint64_t)(r0 + r) * N + n : 0), in);
        }
        copy_commit();
    }
    const int nl = (t % LANES) * TN, kl = (t / LANES) * TK;
    float acc[TK][TN];
#pragma unroll
    for (int q = 0; q < TK; ++q)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[q][j] = 0.f;
    const auto sum = [&](int g) {
        __syncthreads();
#pragma unroll 8
        for (int r = g * GR; r < (g + 1) * GR; ++r) {
            float d[TN], x[TK];
            if (TN == 4) *reinterpret_cast<float4 *>(d) = *reinterpret_cast<const float4 *>(sd + r * NT + nl);
            else
#pragma unroll
                for (int j = 0; j < TN; ++j) d[j] = sd[r * NT + nl + j];
#pragma unroll
            for (int q = 0; q < TK; ++q) x[q] = si[r * WG_KT + kl + q];
#pragma unroll
            for (int q = 0; q < TK; ++q)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[q][j] += x[q] * d[j];
        }
    };
    static_assert(WG_GROUPS == 4, "one wait per group");
    copy_wait<3>(); sum(0);
    copy_wait<2>(); sum(1);
    copy_wait<1>(); sum(2);
    copy_wait<0>(); sum(3);
#pragma unroll
    for (int q = 0; q < TK; ++q)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int k = k0 + kl + q, n = n0 + nl + j;
            if (k <= K && n < N) partial[(uint64_t)blockIdx.y * stride + l.part + (uint32_t)k * N + n] = acc[q][j];
        }
}

// narrow layers (N <= 8): one column a thread
__device__ __host__ __forceinline__ int wg_nt(int N) { return N <= 8 ? 8 : 64; }

__global__ void __launch_bounds__(WG_T) k_mlp_wgrad(const __grid_constant__ WLayers L, int rows, float *partial)
{
    extern __shared__ __align__(16) float wg_smem[];
    int i = 0;
    while (i + 1 < L.n && (int)blockIdx.x >= L.l[i + 1].tile0) ++i;
    const WLayer &l = L.l[i];
    const int tile = (int)blockIdx.x - l.tile0;
    if (wg_nt(l.N) == 8) outer_tile<8, 1>(l, tile, L.stride, rows, wg_smem, partial);
    else outer_tile<64, 4>(l, tile, L.stride, rows, wg_smem, partial);
}

// out[i] = the partials of entry i, row blocks in order; the last block, if there is a loss: the mean
// of the nl blocks' losses' sum over count values
constexpr int FOLD_T = 128;

__global__ void __launch_bounds__(FOLD_T) k_mlp_wgrad_fold(const float *partial, int G, uint32_t n, float *out,
                                                           const float *lpart, int nl, float count, float *loss)
{
    grid_dependency_sync();
    if (loss && blockIdx.x == gridDim.x - 1) {
        __shared__ float part[FOLD_T / 32];
        float s = 0.f;
        for (int b = threadIdx.x; b < nl; b += FOLD_T) s += lpart[b];
#pragma unroll
        for (int m = 16; m; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
        if (!(threadIdx.x & 31)) part[threadIdx.x >> 5] = s;
        __syncthreads();
        if (!threadIdx.x) *loss = ((part[0] + part[1]) + (part[2] + part[3])) / count;
        return;
    }
    const uint32_t e = blockIdx.x * FOLD_T + threadIdx.x;
    if (e >= n) return;
    float s = 0.f;
#pragma unroll 16
    for (int b = 0; b < G; ++b) s += partial[(uint64_t)b * n + e];
    out[e] = s;
}

// ---- Adam (Kingma & Ba 2015) with bias correction ---------------------------------------------
__global__ void k_adam(float *P, const float *G, float *M, float *V, int n, float lr, float b1, float b2,
                       float eps, float c1, float c2)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    grid_dependency_sync();
    const float g = G[i];
    const float m = b1 * M[i] + (1.f - b1) * g;
    const float v = b2 * V[i] + (1.f - b2) * g * g;
    M[i] = m;
    V[i] = v;
    P[i] -= lr * (m / c1) / (sqrtf(v / c2) + eps);
}

// ---- inference ---------------------------------------------------------------------------------
// A boundary step: every face's columns predict their ghosts from E^n, H^{n+1/2}, as
// r * MLP(stencil / r) + memory * (the previous step's ghost): H^{n+1/2} outside side-0 faces,
// E^{n+1} outside side-1 faces; the E update; the E fix-up; sources; the H update; the H fix-up
// (k_lbc_fix). With memory = (1 - c dt) / (1 + c dt) the form contains Mur's first-order
// absorbing condition written for the ghost (the rest of Mur's update is linear in the stencil).
constexpr int T_APPLY = 128;

// Dynamic shared memory of the float32 inference kernel: the parameters, then one column of 64
// hidden activations per thread, stored k-major (hs[k * T + t]) so that the runtime loops over
// k read them without bank conflicts and every register array keeps compile-time indices (a
// hidden vector indexed by the runtime k would live in local memory).
constexpr size_t MLP32_SMEM = ((size_t)LBC_NPARAM + (size_t)LBC_HID * 128) * sizeof(float);

// float32 weights [6 faces][LBC_NPARAM] on the CUDA cores (the checker of the bfloat16 kernel)
static_assert(T_APPLY == 128, "MLP32_SMEM holds 128 hidden columns");

__global__ void __launch_bounds__(T_APPLY) k_lbc_predict32(const LGrid g, int side, float memory, const float *W,
                                                           const float *E, const float *H, float *pred)
{
    extern __shared__ float mlp_smem[];
    float *const w = mlp_smem;
    float *const hs = mlp_smem + LBC_NPARAM + threadIdx.x;   // hs[k * T_APPLY]: this thread's column
    // blockIdx.y: face; its columns: blockIdx.x * T_APPLY + threadIdx.x
    const int fi = blockIdx.y;
    const LFace &f = g.face[fi];
    if (side >= 0 && f.side != side) return;                 // block-uniform
    const float *Wf = W + (uint64_t)(f.axis * 2 + f.side) * LBC_NPARAM;
    for (int i = threadIdx.x; i < LBC_NPARAM; i += blockDim.x) w[i] = Wf[i];
    __syncthreads();
    const uint32_t c = blockIdx.x * T_APPLY + threadIdx.x;
    if (c >= f.ncol) return;
    const uint32_t u = f.u0 + c / f.nv, v = f.v0 + c % f.nv;
    float *out = pred + (uint64_t)(f.col0 + c) * LBC_OUT;
    if (!in_window(g, fi, u, v)) {
#pragma unroll
        for (int o = 0; o < LBC_OUT; ++o) out[o] = memory * out[o];
        return;
    }
    // layer 1 is linear in the inputs: accumulate W1^T x on the raw stencil while summing its
    // squares, then scale by 1/r (the normalisation) and add the bias
    float a[LBC_HID];
#pragma unroll
    for (int j = 0; j < LBC_HID; ++j) a[j] = 0.f;
    float ss = 0.f;
    // the 18 stencil cells as a runtime loop (unrolling them with the 64-wide inner products
    // multiplies the code and the compile time for a kernel that only checks the others)
#pragma unroll 1
    for (int d = 0; d < 2; ++d)
#pragma unroll 1
        for (int du = -1; du <= 1; ++du)
#pragma unroll 1
            for (int dv = -1; dv <= 1; ++dv) {
                const uint64_t i = cell_of(g, f, u, v, d, du, dv);
                const int k0 = ((d * 3 + (du + 1)) * 3 + (dv + 1)) * 6;
#pragma unroll
                for (int q = 0; q < 6; ++q) {
                    const float xv = q < 3 ? E[q * g.N + i] : H[(q - 3) * g.N + i];
                    ss += xv * xv;
#pragma unroll
                    for (int j = 0; j < LBC_HID; ++j) a[j] += xv * w[LBC_W1 + (k0 + q) * LBC_HID + j];
                }
            }
    const float r = sqrtf(ss * (1.0f / LBC_IN));
    if (!(r > 0.f)) {
#pragma unroll
        for (int o = 0; o < LBC_OUT; ++o) out[o] = memory * out[o];
        return;
    }
    const float inv = 1.0f / r;
#pragma unroll
    for (int j = 0; j < LBC_HID; ++j) a[j] = w[LBC_B1 + j] + a[j] * inv;
#pragma unroll
    for (int j = 0; j < LBC_HID; ++j) hs[j * T_APPLY] = gelu(a[j]);
#pragma unroll
    for (int j = 0; j < LBC_HID; ++j) a[j] = w[LBC_B2 + j];
    for (int k = 0; k < LBC_HID; ++k) {
        const float hk = hs[k * T_APPLY];
#pragma unroll
        for (int j = 0; j < LBC_HID; ++j) a[j] += hk * w[LBC_W2 + k * LBC_HID + j];
    }
#pragma unroll
    for (int j = 0; j < LBC_HID; ++j) hs[j * T_APPLY] = gelu(a[j]);
    float y[LBC_OUT];
#pragma unroll
    for (int o = 0; o < LBC_OUT; ++o) y[o] = w[LBC_B3 + o];
    for (int k = 0; k < LBC_HID; ++k) {
        const float hk = hs[k * T_APPLY];
#pragma unroll
        for (int o = 0; o < LBC_OUT; ++o) y[o] += hk * w[LBC_W3 + k * LBC_OUT + o];
    }
#pragma unroll
    for (int o = 0; o < LBC_OUT; ++o) out[o] = y[o] * r + memory * out[o];
}

// ---- stencil tiles staged per warp (the linear and the tensor-core inference) ------------------
// A warp's job: a tile of MMA_TU x 16 columns of one face (MMA_TU rows along u, 16 columns along
// v). The cells its stencils read, (MMA_TU + 2) x 18 positions x 2 depths x 6 components, are
// staged once in shared memory, plane (component q, depth d) by plane with a stride of
// MMA_PL floats (MMA_PL = 16 mod 32, so the two depths a lane pair reads fall in different
// banks), before the columns are evaluated 16 at a time. The loads follow the memory order:
// along z (v) on x and y faces, over the depth pair z = 0, 1 (or s - 1, s - 2) first on z faces.
constexpr int MMA_TU = 4;
constexpr int MMA_SU = MMA_TU + 2, MMA_SV = 16 + 2;
constexpr int MMA_PL = 112;
static_assert(MMA_SU * MMA_SV <= MMA_PL && MMA_PL % 32 == 16, "stage plane layout");
constexpr int MMA_STAGE = 12 * MMA_PL;                                   // floats per warp

// Stage the cells of the tile whose first (face-local) column is (cu0, cv0) into st.
__device__ __forceinline__ void stage_tile(const LGrid &g, const LFace &f, uint32_t cu0, uint32_t cv0,
                                           const float *E, const float *H, float *st, int lane)
{
        // stage: cells (u0 + cu0 - 1 + su, v0 + cv0 - 1 + sv), clamped to the grid like cell_of.
        // Per (component, su) row of the stage a lane loads the pairs (sv, d) number lane and
        // lane + 32 of 36, ordered (sv, d) on z faces (the depth pair is contiguous in memory)
        // and (d, sv) on x and y faces (v = z is contiguous).
        const int a = f.axis, ua = a == 0 ? 1 : 0, va = a == 2 ? 1 : 2;
        const uint64_t syz = (uint64_t)g.s[1] * g.s[2];
        const uint64_t sd = a == 0 ? syz : a == 1 ? (uint64_t)g.s[2] : 1u;     // strides of the depth,
        const uint64_t sua = ua == 0 ? syz : (uint64_t)g.s[2];                 // u and v axes
        const uint64_t sva = va == 1 ? (uint64_t)g.s[2] : 1u;
        uint64_t off[2];
        int soff[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int e = lane + 32 * h < 2 * MMA_SV ? lane + 32 * h : 0;
            const int d = a == 2 ? (e & 1) : e / MMA_SV;
            const int sv = a == 2 ? (e >> 1) : e % MMA_SV;
            const uint32_t cd = f.side ? g.s[a] - 1u - (uint32_t)d : (uint32_t)d;
            const uint32_t cv = clampu((int)(f.v0 + cv0) - 1 + sv, g.s[va]);
            off[h] = cd * sd + cv * sva;
            soff[h] = d * MMA_PL + sv;
        }
        const bool second = lane + 32 < 2 * MMA_SV;
#pragma unroll 1
        for (int su = 0; su < MMA_SU; ++su) {
            const uint64_t ou = clampu((int)(f.u0 + cu0) - 1 + su, g.s[ua]) * sua;
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                const float *src = q < 3 ? E + q * g.N : H + (q - 3) * g.N;
                float *dst = st + q * 2 * MMA_PL + su * MMA_SV;
                dst[soff[0]] = src[ou + off[0]];
                if (second) dst[soff[1]] = src[ou + off[1]];
            }
        }
}

constexpr int MMA_WARPS = 4;                      // warps of a block of the staged kernels

// an exactly linear layer (LBC_LINEAR), weights [6][IN + 1][OUT] float32 in shared memory: a
// warp stages a tile of 4 x 16 columns (stage_tile) and each lane forms the 108 x 6 products of
// two of them (column lane % 16 of the tile's rows lane / 16 and lane / 16 + 2), in the order
// of the stencil
__global__ void __launch_bounds__(MMA_WARPS * 32) k_lbc_predict_lin(const LGrid g, int side, float memory,
                                                                    const float *W, const float *E,
                                                                    const float *H, float *pred)
{
    __shared__ float w[(LBC_IN + 1) * LBC_OUT];
    __shared__ float stage[MMA_WARPS][MMA_STAGE];
    const LFace &f = g.face[blockIdx.y];
    if (side >= 0 && f.side != side) return;                 // block-uniform
    const float *Wf = W + (uint64_t)(f.axis * 2 + f.side) * (LBC_IN + 1) * LBC_OUT;
    for (int i = threadIdx.x; i < (LBC_IN + 1) * LBC_OUT; i += blockDim.x) w[i] = Wf[i];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t ntv = (f.nv + 15u) / 16u, ntu = (f.nu + MMA_TU - 1u) / MMA_TU;
    const uint32_t job = blockIdx.x * MMA_WARPS + warp;
    if (job >= ntu * ntv) return;                            // warp-uniform; no block barrier below
    const uint32_t cu0 = (job / ntv) * MMA_TU, cv0 = (job % ntv) * 16u;
    float *st = stage[warp];
    stage_tile(g, f, cu0, cv0, E, H, st, lane);
    __syncwarp();
    const int jv = lane & 15;
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        const int tr = (lane >> 4) + 2 * h;
        const uint32_t cu = cu0 + (uint32_t)tr, cv = cv0 + (uint32_t)jv;
        if (cu >= f.nu || cv >= f.nv) continue;
        const uint32_t c = cu * f.nv + cv;
        float *out = pred + (uint64_t)(f.col0 + c) * LBC_OUT;
        if (!in_window(g, blockIdx.y, f.u0 + cu, f.v0 + cv)) {
#pragma unroll
            for (int o = 0; o < LBC_OUT; ++o) out[o] = memory * out[o];
            continue;
        }
        float acc[LBC_OUT];
#pragma unroll
        for (int o = 0; o < LBC_OUT; ++o) acc[o] = 0.f;
        float ss = 0.f;
#pragma unroll
        for (int d = 0; d < 2; ++d)
#pragma unroll
            for (int du = -1; du <= 1; ++du)
#pragma unroll
                for (int dv = -1; dv <= 1; ++dv) {
                    const int k0 = ((d * 3 + (du + 1)) * 3 + (dv + 1)) * 6;
                    const float *sp = st + d * MMA_PL + (tr + 1 + du) * MMA_SV + (jv + 1 + dv);
#pragma unroll
                    for (int q = 0; q < 6; ++q) {
                        const float xv = sp[q * 2 * MMA_PL];
                        ss += xv * xv;
#pragma unroll
                        for (int o = 0; o < LBC_OUT; ++o) acc[o] += xv * w[(k0 + q) * LBC_OUT + o];
                    }
                }
        const float r = sqrtf(ss * (1.0f / LBC_IN));
#pragma unroll
        for (int o = 0; o < LBC_OUT; ++o) out[o] = acc[o] + r * w[LBC_IN * LBC_OUT + o] + memory * out[o];
    }
}

// ---- bfloat16 tensor-core inference (mma.sync m16n8k16, float32 accumulation) ------------------
// Weights are packed once per face into the B-fragment order of mma.m16n8k16 (PTX ISA, "Matrix
// fragments for mma.m16n8k16"): for k-step ks and n-tile nt, lane (g = lane / 4, t = lane % 4)
// holds B[16 ks + 2t + {0, 1}][8 nt + g] in word 0 and B[16 ks + 2t + 8 + {0, 1}][8 nt + g] in
// word 1, the lower k in the low half. Layer 1's K = 108 is padded to 112 with zero rows,
// layer 3's N = 6 to 8 with zero columns. Biases stay float32.
constexpr int PK_W1 = 0;                          // [7][8][32][2] words
constexpr int PK_W2 = PK_W1 + 7 * 8 * 64;         // [4][8][32][2]
constexpr int PK_W3 = PK_W2 + 4 * 8 * 64;         // [4][1][32][2]
constexpr int PK_B1 = PK_W3 + 4 * 64;             // float [64]
constexpr int PK_B2 = PK_B1 + LBC_HID;            // float [64]
constexpr int PK_B3 = PK_B2 + LBC_HID;            // float [8]
static_assert(PK_B3 + 8 == LBC_PACK_WORDS, "packed layout size");

// two floats rounded to bfloat16 in one conversion (lo in the low half)
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
    const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&p);
}

// x = hi + lo with hi = bf16(x), lo = bf16(x - hi): about 16 significant bits in two bf16 parts
__device__ __forceinline__ void split_bf16(float x0, float x1, uint32_t &hi, uint32_t &lo)
{
    hi = pack_bf16(x0, x1);
    const float h0 = __uint_as_float(hi << 16), h1 = __uint_as_float(hi & 0xffff0000u);
    lo = pack_bf16(x0 - h0, x1 - h1);
}

// GELU of the tensor-core inference: erf by Abramowitz & Stegun, Handbook of Mathematical
// Functions, formula 7.1.26 (Hastings' rational approximation, |error| <= 1.5e-7 for all x),
// with the exponential and reciprocal on the special-function unit; well inside the bfloat16
// (and split-bfloat16) precision of the layer inputs it feeds. Training and the float32 checker
// use erff.
__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float ex2_approx(float x)
{
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// PTX: the reciprocal and 2^x by rcp.approx / ex2.approx and the last step as one fma;
// otherwise the __fdividef / __expf intrinsics. Same approximation either way; each form
// measured faster in one of the two kernels (bf16x2: PTX, bf16: intrinsics).
template <bool PTX>
__device__ __forceinline__ float gelu_mma(float x)
{
    const float z = x * 0.70710678118654752f;                 // x / sqrt(2)
    const float az = fabsf(z);
    const float den = fmaf(0.3275911f, az, 1.0f);
    const float t = PTX ? rcp_approx(den) : __fdividef(1.0f, den);
    const float poly = t * fmaf(t, fmaf(t, fmaf(t, fmaf(t, 1.061405429f, -1.453152027f), 1.421413741f),
                                        -0.284496736f), 0.254829592f);
    if (PTX) {
        // exp(-z^2) = 2^(-z^2 log2(e))
        const float e = copysignf(fmaf(-poly, ex2_approx((az * az) * -1.4426950408889634f), 1.0f), z);
        const float h = 0.5f * x;
        return fmaf(h, e, h);                                 // x (1 + erf(z)) / 2
    }
    const float e = copysignf(1.0f - poly * __expf(-az * az), z);
    return 0.5f * x * (1.0f + e);
}

__device__ __forceinline__ void mma_bf16(float c[4], const uint32_t a[4], uint32_t b0, uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__global__ void k_lbc_pack(const float *P, uint32_t *out)
{
    const int face = blockIdx.y;
    const float *w = P + (uint64_t)face * LBC_NPARAM;
    uint32_t *o = out + (uint64_t)face * LBC_PACK_WORDS;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < LBC_PACK_WORDS; e += gridDim.x * blockDim.x) {
        uint32_t word;
        if (e >= PK_B1) {
            const int j = e - PK_B1;
            const float b = j < LBC_HID ? w[LBC_B1 + j] : j < 2 * LBC_HID ? w[LBC_B2 + j - LBC_HID]
                                                         : (j - 2 * LBC_HID < LBC_OUT ? w[LBC_B3 + j - 2 * LBC_HID] : 0.f);
            word = __float_as_uint(b);
        } else {
            int base, K, N, nt_count, off;
            if (e < PK_W2) { off = e - PK_W1; base = LBC_W1; K = LBC_IN; N = LBC_HID; nt_count = 8; }
            else if (e < PK_W3) { off = e - PK_W2; base = LBC_W2; K = LBC_HID; N = LBC_HID; nt_count = 8; }
            else { off = e - PK_W3; base = LBC_W3; K = LBC_HID; N = LBC_OUT; nt_count = 1; }
            const int reg = off & 1, lane = (off >> 1) & 31, nt = (off >> 6) % nt_count, ks = (off >> 6) / nt_count;
            const int g = lane >> 2, t = lane & 3;
            const int k = 16 * ks + 2 * t + 8 * reg, n = 8 * nt + g;
            const float v0 = (k < K && n < N) ? w[base + k * N + n] : 0.f;
            const float v1 = (k + 1 < K && n < N) ? w[base + (k + 1) * N + n] : 0.f;
            word = pack_bf16(v0, v1);
        }
        o[e] = word;
    }
}

// GELU of a layer's accumulators, re-cut into the A fragments of the next layer: n-tiles 2 ks and
// 2 ks + 1 of a 16 x 64 output are the k-step ks A fragment (rows g / g + 8, cols 2t / 2t + 8).
template <bool SPLIT>
__device__ __forceinline__ void act_to_a(const float acc[8][4], uint32_t ah[4][4], uint32_t al[4][4])
{
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const float *c = acc[2 * ks + half];
            const float g0 = gelu_mma<SPLIT>(c[0]), g1 = gelu_mma<SPLIT>(c[1]);
            const float g2 = gelu_mma<SPLIT>(c[2]), g3 = gelu_mma<SPLIT>(c[3]);
            if (SPLIT) {
                split_bf16(g0, g1, ah[ks][2 * half], al[ks][2 * half]);
                split_bf16(g2, g3, ah[ks][2 * half + 1], al[ks][2 * half + 1]);
            } else {
                ah[ks][2 * half] = pack_bf16(g0, g1);
                ah[ks][2 * half + 1] = pack_bf16(g2, g3);
            }
        }
}


// A block holds its face's packed weights in shared memory and gives each warp a tile of MW_TU x 16
// columns, whose stencil cells the warp stages as component pairs (two neighbouring inputs of the
// network), plane (pair, depth) by plane. A lane then reads the A fragments of layer 1 straight from
// the stage: inputs 2 m and 2 m + 1, m = 8 ks + tq (+ 4), of the columns gq and gq + 8.
//
// What bounds it: latency. One step's ghosts of a 203x177x61 grid are 118 k columns, 2.7 GFLOP: a few
// microseconds of the tensor units and 15 of instruction issue. With the weights read through L1 (64%
// hits beside the stages), inputs normalised into a second shared array, 4-row tiles (two uneven waves
// of blocks, half of them empty) it took 55 us, now 36 (1-row tiles 38, 4-row 42; 8 warps a block 40).
constexpr int MW_TU = 2, MW_WARPS = 4, MW_SU = MW_TU + 2, MW_SV = 18;
// words of a plane; the three pairs' planes of a depth start 12 or 24 banks apart, so that the four inputs
// that the lanes of a column read at once fall in different banks
constexpr int mw_plane(int n)
{
    return (2 * n) % 32 == 24 || (2 * n) % 32 == 12 ? n : mw_plane(n + 2);
}
constexpr int MW_PL = mw_plane(MW_SU * MW_SV * 2);
constexpr int MW_STAGE = 6 * MW_PL;                                       // words per warp
constexpr size_t MW_SMEM = (size_t)(LBC_PACK_WORDS + MW_WARPS * MW_STAGE) * 4;
static_assert(LBC_PACK_WORDS % 4 == 0 && MW_PL % 2 == 0, "16-byte weights, 8-byte pairs");

struct MFirst {
    uint32_t block[7];                                                    // first block of each face
};

// the cells of the tile whose first (face-local) column is (cu0, cv0), clamped to the grid like cell_of;
// lanes take the positions (sv, d) in memory order, as in stage_tile
__device__ __forceinline__ void stage_pairs(const LGrid &g, const LFace &f, uint32_t cu0, uint32_t cv0, const float *E,
                                            const float *H, float *st, int lane)
{
    const int a = f.axis, ua = a == 0 ? 1 : 0, va = a == 2 ? 1 : 2;
    const uint32_t syz = g.s[1] * g.s[2];
    const uint32_t sd = a == 0 ? syz : a == 1 ? g.s[2] : 1u, sua = ua == 0 ? syz : g.s[2], sva = va == 1 ? g.s[2] : 1u;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int e = lane + 32 * h;
        if (e >= 2 * MW_SV) break;
        const int d = a == 2 ? (e & 1) : e / MW_SV, sv = a == 2 ? (e >> 1) : e % MW_SV;
        const uint32_t cd = f.side ? g.s[a] - 1u - (uint32_t)d : (uint32_t)d;
        const uint32_t off = cd * sd + clampu((int)(f.v0 + cv0) - 1 + sv, g.s[va]) * sva;
        float *const dst = st + d * MW_PL + sv * 2;
        float v[MW_SU][6];
#pragma unroll
        for (int su = 0; su < MW_SU; ++su) {
            const uint32_t i = off + clampu((int)(f.u0 + cu0) - 1 + su, g.s[ua]) * sua;
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                v[su][q] = E[q * g.N + i];
                v[su][3 + q] = H[q * g.N + i];
            }
        }
#pragma unroll
        for (int su = 0; su < MW_SU; ++su)
#pragma unroll
            for (int qp = 0; qp < 3; ++qp)
                *reinterpret_cast<float2 *>(dst + qp * 2 * MW_PL + su * MW_SV * 2) = make_float2(v[su][2 * qp], v[su][2 * qp + 1]);
    }
}

template <bool SPLIT>
__global__ void __launch_bounds__(MW_WARPS * 32, 4) k_lbc_predict_mma(const __grid_constant__ LGrid g, const __grid_constant__ MFirst first,
                                                                      float memory, const uint32_t *Wp, const float *E,
                                                                      const float *H, float *pred)
{
    extern __shared__ __align__(16) uint32_t smem_w[];
    int fi = 0;
    while (blockIdx.x >= first.block[fi + 1]) ++fi;
    const LFace &f = g.face[fi];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gq = lane >> 2, tq = lane & 3;
    float *const st = reinterpret_cast<float *>(smem_w + LBC_PACK_WORDS) + warp * MW_STAGE;
    grid_dependency_sync();
    {
        const uint32_t *src = Wp + (uint64_t)(f.axis * 2 + f.side) * LBC_PACK_WORDS;
        const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem_w);
        for (int i = threadIdx.x; i < LBC_PACK_WORDS / 4; i += MW_WARPS * 32)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16 * i), "l"(src + 4 * i) : "memory");
        copy_commit();
    }
    const uint32_t ntv = (f.nv + 15u) / 16u, ntu = (f.nu + MW_TU - 1u) / MW_TU;
    const uint32_t job = (blockIdx.x - first.block[fi]) * MW_WARPS + warp;
    const bool work = job < ntu * ntv;                                    // warp-uniform
    const uint32_t tu = job / ntv, tv = job - tu * ntv;
    const uint32_t cu0 = tu * MW_TU, cv0 = tv * 16u;                      // first column of the tile (face-local)
    if (work) stage_pairs(g, f, cu0, cv0, E, H, st, lane);
    copy_wait<0>();
    __syncthreads();
    if (!work) return;
    const float *const wb = reinterpret_cast<const float *>(smem_w);
    const uint2 *const w1 = reinterpret_cast<const uint2 *>(smem_w + PK_W1);
    const uint2 *const w2 = reinterpret_cast<const uint2 *>(smem_w + PK_W2);
    const uint2 *const w3 = reinterpret_cast<const uint2 *>(smem_w + PK_W3);
#pragma unroll 1
    for (int tr = 0; tr < MW_TU; ++tr) {
        const uint32_t cu = cu0 + (uint32_t)tr;
        if (cu >= f.nu) break;                                            // warp-uniform
        // RMS of column lane / 2, each lane of the pair one depth, in the order of the stencil
        float rl;
        {
            const int row = lane >> 1;
            const float *const sp = st + (lane & 1) * MW_PL + (tr * MW_SV + row) * 2;
            float ss = 0.f;
#pragma unroll
            for (int du = 0; du < 3; ++du)
#pragma unroll
                for (int dv = 0; dv < 3; ++dv)
#pragma unroll
                    for (int qp = 0; qp < 3; ++qp) {
                        const float2 v = *reinterpret_cast<const float2 *>(sp + qp * 2 * MW_PL + (du * MW_SV + dv) * 2);
                        ss += v.x * v.x;
                        ss += v.y * v.y;
                    }
            ss += __shfl_xor_sync(0xffffffffu, ss, 1);
            // columns outside the window: r = 0, no network term
            const uint32_t cv = cv0 + (uint32_t)row;
            rl = cv < f.nv && in_window(g, fi, f.u0 + cu, f.v0 + cv) ? sqrtf(ss * (1.0f / LBC_IN)) : 0.f;
        }
        // rows (columns of the face) gq and gq + 8
        float r[2], inv[2];
#pragma unroll
        for (int hr = 0; hr < 2; ++hr) {
            r[hr] = __shfl_sync(0xffffffffu, rl, 2 * (gq + 8 * hr));
            inv[hr] = r[hr] > 0.f ? 1.0f / r[hr] : 0.f;
        }
        // layer 1: [16 x 112] x [112 x 64]
        float acc[8][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const float b0 = wb[PK_B1 + 8 * nt + 2 * tq], b1 = wb[PK_B1 + 8 * nt + 2 * tq + 1];
            acc[nt][0] = b0; acc[nt][1] = b1; acc[nt][2] = b0; acc[nt][3] = b1;
        }
#pragma unroll
        for (int ks = 0; ks < 7; ++ks) {
            uint32_t ah[4], al[4];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int m = 8 * ks + 4 * h + tq;
                const int pos = m / 3, qp = m - 3 * pos, d = pos / 9, du = (pos - 9 * d) / 3, dv = pos - 9 * d - 3 * du;
                const float *const sp = st + (qp * 2 + d) * MW_PL + ((tr + du) * MW_SV + gq + dv) * 2;
#pragma unroll
                for (int hr = 0; hr < 2; ++hr) {
                    float2 v = make_float2(0.f, 0.f);                     // K padding 108..111
                    if (8 * ks + 4 * h + 3 < 54 || m < 54) v = *reinterpret_cast<const float2 *>(sp + 16 * hr);
                    v.x *= inv[hr];
                    v.y *= inv[hr];
                    if (SPLIT) split_bf16(v.x, v.y, ah[2 * h + hr], al[2 * h + hr]);
                    else ah[2 * h + hr] = pack_bf16(v.x, v.y);
                }
            }
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                const uint2 b = w1[(ks * 8 + nt) * 32 + lane];
                mma_bf16(acc[nt], ah, b.x, b.y);
                if (SPLIT) mma_bf16(acc[nt], al, b.x, b.y);
            }
        }
        uint32_t ah2[4][4], al2[4][4];
        act_to_a<SPLIT>(acc, ah2, al2);
        // layer 2: [16 x 64] x [64 x 64]
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const float b0 = wb[PK_B2 + 8 * nt + 2 * tq], b1 = wb[PK_B2 + 8 * nt + 2 * tq + 1];
            acc[nt][0] = b0; acc[nt][1] = b1; acc[nt][2] = b0; acc[nt][3] = b1;
        }
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                const uint2 b = w2[(ks * 8 + nt) * 32 + lane];
                mma_bf16(acc[nt], ah2[ks], b.x, b.y);
                if (SPLIT) mma_bf16(acc[nt], al2[ks], b.x, b.y);
            }
        act_to_a<SPLIT>(acc, ah2, al2);
        // layer 3: [16 x 64] x [64 x 8]
        float y[4];
        {
            const float b0 = wb[PK_B3 + 2 * tq], b1 = wb[PK_B3 + 2 * tq + 1];
            y[0] = b0; y[1] = b1; y[2] = b0; y[3] = b1;
        }
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
            const uint2 b = w3[ks * 32 + lane];
            mma_bf16(y, ah2[ks], b.x, b.y);
            if (SPLIT) mma_bf16(y, al2[ks], b.x, b.y);
        }
        // rows gq and gq + 8, output components 2 tq and 2 tq + 1 (< 6)
        if (tq < 3) {
#pragma unroll
            for (int hr = 0; hr < 2; ++hr) {
                const uint32_t cv = cv0 + (uint32_t)(gq + 8 * hr);
                if (cv < f.nv) {
                    float *out = pred + (uint64_t)(f.col0 + cu * f.nv + cv) * LBC_OUT + 2 * tq;
                    out[0] = (r[hr] > 0.f ? y[2 * hr] * r[hr] : 0.f) + memory * out[0];
                    out[1] = (r[hr] > 0.f ? y[2 * hr + 1] * r[hr] : 0.f) + memory * out[1];
                }
            }
        }
    }
}

// Levi-Civita sign of distinct (q, a, p): +1 for the cyclic orders of (0, 1, 2)
__device__ __forceinline__ float lc(int q, int a) { return ((a - q + 3) % 3) == 1 ? 1.f : -1.f; }

__device__ __forceinline__ int own_of(const LGrid &g, uint32_t col)
{
    int f = 0;
    while (f + 1 < g.nface && col >= g.own[f + 1].col0) ++f;
    return f;
}

// One thread per outer cell: every learned face of the side (E fix-up: side 0, H fix-up: side 1) through
// the cell adds its term, faces in order. A cell lies on at most one such face per axis, so what its
// terms need is requested at once (8.7 us a fix-up of a 203x177x61 grid when each face's values were
// loaded after the one before, and the field after them).
struct FixFaces {
    uint32_t col0[3], nv[3];                                 // per axis: the face's first column and row length
    int32_t on[3];
};

template <bool EFIX>
__global__ void __launch_bounds__(128) k_lbc_fix(const __grid_constant__ LGrid g, const __grid_constant__ FixFaces ff,
                                                 const float *pred, float *P, const float *Q, const float *coef, float dt)
{
    const uint32_t col = blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= g.nown) return;
    const LFace &o = g.own[own_of(g, col)];
    const uint32_t k = col - o.col0;
    const uint32_t cu = o.u0 + k / o.nv, cv = o.v0 + k % o.nv, cw = o.side ? g.s[o.axis] - 1u : 0u;
    const uint32_t c[3] = {o.axis == 0 ? cw : cu, o.axis == 0 ? cu : o.axis == 1 ? cw : cv, o.axis == 2 ? cw : cv};
    const uint64_t st[3] = {(uint64_t)g.s[1] * g.s[2], g.s[2], 1};
    const uint64_t i = c[0] * st[0] + c[1] * st[1] + c[2];
    bool on[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) on[a] = ff.on[a] && c[a] == (EFIX ? 0u : g.s[a] - 1u);
    if (!(on[0] || on[1] || on[2])) return;
    grid_dependency_sync();
    float ghost[3][3], wrapped[3][3], co[3], p[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        co[q] = coef ? coef[q * g.N + i] : dt;
        p[q] = P[q * g.N + i];
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (!on[a]) continue;
        const float *gp = pred + ((uint64_t)ff.col0[a] + (uint64_t)c[a == 0 ? 1 : 0] * ff.nv[a] + c[a == 2 ? 1 : 2]) * LBC_OUT;
        // the wrapped neighbour: index s_a - 1 (side 0) or 0 (side 1) along a
        const uint64_t j = EFIX ? i + (uint64_t)(g.s[a] - 1u) * st[a] : i - (uint64_t)(g.s[a] - 1u) * st[a];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            if (q == a) continue;
            ghost[a][q] = gp[(EFIX ? 3 : 0) + q];
            wrapped[a][q] = Q[q * g.N + j];
        }
    }
    float d[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int q = 0; q < 3; ++q)
            if (q != a && on[a]) d[q] -= lc(q, a) * (ghost[a][3 - a - q] - wrapped[a][3 - a - q]);
#pragma unroll
    for (int q = 0; q < 3; ++q)
        if (d[q] != 0.f) P[q * g.N + i] = p[q] + co[q] * d[q];
}

}  // namespace

// the column grids of the faces in face_mask (bit 2a + side): whole planes, and owned cells
LGrid lbc_grid(const uint32_t s[3], int face_mask)
{
    LGrid g;
    g.s[0] = s[0];
    g.s[1] = s[1];
    g.s[2] = s[2];
    g.N = (uint64_t)s[0] * s[1] * s[2];
    g.mask = face_mask;
    g.nface = 0;
    g.ncol = 0;
    g.nown = 0;
    bool owned[3][2] = {{false, false}, {false, false}, {false, false}};
    for (int a = 0; a < 3; ++a)
        for (int side = 0; side < 2; ++side) {
            if (!(face_mask & (1 << (2 * a + side)))) continue;
            const int ua = a == 0 ? 1 : 0, va = a == 2 ? 1 : 2;
            LFace f;
            f.axis = a;
            f.side = side;
            f.u0 = 0;
            f.v0 = 0;
            f.nu = s[ua];
            f.nv = s[va];
            f.ncol = f.nu * f.nv;
            f.col0 = g.ncol;
            g.ncol += f.ncol;
            // owned: skip the cells of an earlier face's plane (lower axes own the edges)
            LFace o = f;
            uint32_t u0 = 0, u1 = s[ua], v0 = 0, v1 = s[va];
            if (owned[ua][0]) u0 = 1;
            if (owned[ua][1] && u1 > 0) u1 -= 1;
            if (owned[va][0]) v0 = 1;
            if (owned[va][1] && v1 > 0) v1 -= 1;
            o.u0 = u0;
            o.v0 = v0;
            o.nu = u1 > u0 ? u1 - u0 : 0;
            o.nv = v1 > v0 ? v1 - v0 : 0;
            o.ncol = o.nu * o.nv;
            o.col0 = g.nown;
            g.nown += o.ncol;
            g.face[g.nface] = f;
            g.own[g.nface] = o;
            g.win[g.nface][0] = 0;
            g.win[g.nface][1] = s[ua];
            g.win[g.nface][2] = 0;
            g.win[g.nface][3] = s[va];
            ++g.nface;
            owned[a][side] = true;
        }
    return g;
}

LGrid lbc_grid_window(const uint32_t s[3], int face_mask, const uint32_t lo[3], const uint32_t hi[3])
{
    LGrid g = lbc_grid(s, face_mask);
    for (int i = 0; i < g.nface; ++i) {
        const int a = g.face[i].axis, ua = a == 0 ? 1 : 0, va = a == 2 ? 1 : 2;
        g.win[i][0] = lo[ua] < s[ua] ? lo[ua] : s[ua];
        g.win[i][1] = hi[ua] < s[ua] ? s[ua] - hi[ua] : 0;
        g.win[i][2] = lo[va] < s[va] ? lo[va] : s[va];
        g.win[i][3] = hi[va] < s[va] ? s[va] - hi[va] : 0;
    }
    return g;
}

cudaError_t launch_lbc_gather(const LGrid &g, const float *E, const float *H, float *X, float *R, float *C,
                              cudaStream_t st)
{
    if (!g.ncol) return cudaSuccess;
    k_lbc_gather<<<(g.ncol + 127) / 128, 128, 0, st>>>(g, E, H, X, R, C);
    return cudaGetLastError();
}

// The shared-memory opt-in above 48 KB is a per-device function attribute: set it once per device
// and kernel slot (setting it twice from two threads is harmless).
enum : int { SMEM_MLP_FWD = 0, SMEM_PREDICT32 = 1, SMEM_MMA = 2, SMEM_MMA_SPLIT = 3, SMEM_WGRAD = 4, SMEM_MLP_GRAD = 5, SMEM_SLOTS = 6 };

static cudaError_t smem_opt_in(const void *fn, int slot, size_t bytes)
{
    constexpr int MAX_DEV = 64;
    static bool set[MAX_DEV][SMEM_SLOTS] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < MAX_DEV && set[dev][slot]) return cudaSuccess;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < MAX_DEV) set[dev][slot] = true;
    return cudaSuccess;
}

cudaError_t launch_mlp_fwd(const float *P, const float *X, int B, float *Y, float *A1, float *A2, float *H1,
                           float *H2, cudaStream_t st)
{
    if (B <= 0) return cudaSuccess;
    const cudaError_t e = smem_opt_in((const void *)k_mlp_rows<false>, SMEM_MLP_FWD, ROWS_SMEM);
    if (e != cudaSuccess) return e;
    const RowsK k = {P, X, B, Y, A1, A2, H1, H2, nullptr, nullptr, 0.f, nullptr, nullptr, nullptr, nullptr};
    k_mlp_rows<false><<<(B + TR_ROWS - 1) / TR_ROWS, TR_T, ROWS_SMEM, st>>>(k);
    return cudaGetLastError();
}

// the tiles of the layers, one launch, then the fold into out (their (K + 1) * N entries in order);
// with loss, the fold also takes the mean of rows * LBC_OUT values from lpart, one sum per TR_ROWS rows
static cudaError_t launch_wgrad(WLayers L, int rows, float *ws, float *out, const float *lpart, float *loss, cudaStream_t st)
{
    cudaError_t e = smem_opt_in((const void *)k_mlp_wgrad, SMEM_WGRAD, WG_SMEM);
    if (e != cudaSuccess) return e;
    int tiles = 0;
    uint32_t n = 0;
    for (int i = 0; i < L.n; ++i) {
        WLayer &l = L.l[i];
        l.tile0 = tiles;
        l.part = n;
        tiles += (l.K + WG_KT) / WG_KT * ((l.N + wg_nt(l.N) - 1) / wg_nt(l.N));
        n += (uint32_t)(l.K + 1) * l.N;
    }
    L.stride = n;
    // row blocks beyond the y extent of a grid: further launches, partials side by side
    const int G = (rows + WG_RPB - 1) / WG_RPB;
    for (int g = 0; g < G; g += 65535) {
        const int m = G - g < 65535 ? G - g : 65535, r0 = g * WG_RPB;
        WLayers Lg = L;
        for (int i = 0; i < L.n; ++i) {
            Lg.l[i].in += (size_t)r0 * L.l[i].K;
            Lg.l[i].d += (size_t)r0 * L.l[i].N;
        }
        e = launch_dependent_smem(k_mlp_wgrad, dim3(tiles, m, 1), WG_T, WG_SMEM, st, true, Lg, rows - r0, ws + (size_t)g * n);
        if (e != cudaSuccess) return e;
    }
    return launch_dependent_smem(k_mlp_wgrad_fold, dim3((n + FOLD_T - 1) / FOLD_T + (loss ? 1 : 0), 1, 1), FOLD_T, 0, st, true,
                                 (const float *)ws, G, n, out, lpart, (rows + TR_ROWS - 1) / TR_ROWS, (float)rows * LBC_OUT, loss);
}

// the weight gradients of the network's layers from their inputs and pre-activation gradients
static cudaError_t launch_layers(const float *X, const float *H1, const float *H2, const float *D1, const float *D2,
                                 const float *DY, int B, float *part, float *grad, const float *lpart, float *loss,
                                 cudaStream_t st)
{
    // the gradient's layout is the parameters': each layer's weights, then its bias row
    static_assert(LBC_W1 == 0 && LBC_B1 == LBC_IN * LBC_HID && LBC_W2 == LBC_B1 + LBC_HID &&
                      LBC_B2 == LBC_W2 + LBC_HID * LBC_HID && LBC_W3 == LBC_B2 + LBC_HID &&
                      LBC_B3 == LBC_W3 + LBC_HID * LBC_OUT && LBC_NPARAM == LBC_B3 + LBC_OUT, "parameter layout");
    const WLayers L = {{{X, D1, LBC_IN, LBC_HID, 0, 0}, {H1, D2, LBC_HID, LBC_HID, 0, 0}, {H2, DY, LBC_HID, LBC_OUT, 0, 0}},
                       3, 0};
    return launch_wgrad(L, B, part, grad, lpart, loss, st);
}

// workspace floats needed by launch_mlp_bwd for a batch of B
size_t mlp_bwd_workspace(int B)
{
    const size_t G = ((size_t)B + WG_RPB - 1) / WG_RPB;
    return (size_t)B * (LBC_OUT + 2 * LBC_HID) + G * LBC_NPARAM;
}

cudaError_t launch_mlp_bwd(const float *P, const float *X, const float *Y, const float *T, const float *wout,
                           int B, const float *A1, const float *A2, const float *H1, const float *H2,
                           float *grad, float *ws, cudaStream_t st)
{
    if (B <= 0) return cudaSuccess;
    float *DY = ws, *D2 = DY + (size_t)B * LBC_OUT, *D1 = D2 + (size_t)B * LBC_HID;
    float *part = D1 + (size_t)B * LBC_HID;
    k_mlp_bwd_rows<<<(B + TR_ROWS - 1) / TR_ROWS, TR_T, 0, st>>>(P, Y, T, wout, B, 1.0f / ((float)B * LBC_OUT),
                                                                 A1, A2, DY, D2, D1);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_layers(X, H1, H2, D1, D2, DY, B, part, grad, nullptr, nullptr, st);
}

size_t mlp_grad_workspace(int B)
{
    return mlp_bwd_workspace(B) + (size_t)B * 2 * LBC_HID + ((size_t)B + TR_ROWS - 1) / TR_ROWS;
}

cudaError_t launch_mlp_grad(const float *P, const float *X, const float *T, const float *wout, int B, float *grad,
                            float *loss, float *ws, cudaStream_t st)
{
    if (B <= 0) return cudaSuccess;
    cudaError_t e = smem_opt_in((const void *)k_mlp_rows<true>, SMEM_MLP_GRAD, ROWS_SMEM);
    if (e != cudaSuccess) return e;
    const size_t nh = (size_t)B * LBC_HID;
    float *DY = ws, *D2 = DY + (size_t)B * LBC_OUT, *D1 = D2 + nh, *H1 = D1 + nh, *H2 = H1 + nh, *lpart = H2 + nh;
    const int blocks = (B + TR_ROWS - 1) / TR_ROWS;
    const RowsK k = {P, X, B, nullptr, nullptr, nullptr, H1, H2, T, wout, 1.0f / ((float)B * LBC_OUT), DY, D2, D1, lpart};
    // the launches of a training step depend on each other: each is set up while the one before drains
    if ((e = launch_dependent_smem(k_mlp_rows<true>, dim3(blocks, 1, 1), TR_T, ROWS_SMEM, st, true, k)) != cudaSuccess) return e;
    return launch_layers(X, H1, H2, D1, D2, DY, B, lpart + blocks, grad, lpart, loss, st);
}

// out[(K + 1) x N]: A^T B (rows k < K) and the column sums of B (row K), A [rows][K], B [rows][N];
// ws: ceil(rows / 256) * (K + 1) * N floats
size_t gram_workspace(int rows, int K, int N) { return ((size_t)rows + WG_RPB - 1) / WG_RPB * (size_t)(K + 1) * N; }

cudaError_t launch_gram(const float *A, int rows, int K, const float *B, int N, float *out, float *ws,
                        cudaStream_t st)
{
    if (rows <= 0) return cudaSuccess;
    const WLayers L = {{{A, B, K, N, 0, 0}}, 1, 0};
    return launch_wgrad(L, rows, ws, out, nullptr, nullptr, st);
}

cudaError_t launch_adam(float *P, const float *G, float *M, float *V, int n, float lr, float b1, float b2,
                        float eps, int step, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    return launch_dependent_smem(k_adam, dim3((n + 255) / 256, 1, 1), 256, 0, st, true, P, G, M, V, n, lr, b1, b2, eps, c1, c2);
}

cudaError_t launch_lbc_pack(const float *P, uint32_t *out, cudaStream_t st)
{
    k_lbc_pack<<<dim3((LBC_PACK_WORDS + 255) / 256, 6, 1), 256, 0, st>>>(P, out);
    return cudaGetLastError();
}

cudaError_t launch_lbc_predict(const LGrid &g, int side, int precision, float memory, const void *W, const float *E,
                               const float *H, float *pred, cudaStream_t st, bool pdl)
{
    if (!g.ncol) return cudaSuccess;
    uint32_t maxc = 0;
    for (int f = 0; f < g.nface; ++f) maxc = g.face[f].ncol > maxc ? g.face[f].ncol : maxc;
    if (precision == LBC_F32 || precision == LBC_LINEAR) {
        const dim3 gi((maxc + T_APPLY - 1) / T_APPLY, (unsigned)g.nface, 1);
        uint32_t maxj = 0;
        for (int f = 0; f < g.nface; ++f) {
            const uint32_t nj = ((g.face[f].nu + MMA_TU - 1) / MMA_TU) * ((g.face[f].nv + 15) / 16);
            maxj = nj > maxj ? nj : maxj;
        }
        if (precision == LBC_F32) {
            const cudaError_t e = smem_opt_in((const void *)k_lbc_predict32, SMEM_PREDICT32, MLP32_SMEM);
            if (e != cudaSuccess) return e;
            k_lbc_predict32<<<gi, T_APPLY, MLP32_SMEM, st>>>(g, side, memory, (const float *)W, E, H, pred);
        } else {
            const dim3 gl((maxj + MMA_WARPS - 1) / MMA_WARPS, (unsigned)g.nface, 1);
            k_lbc_predict_lin<<<gl, MMA_WARPS * 32, 0, st>>>(g, side, memory, (const float *)W, E, H, pred);
        }
        return cudaGetLastError();
    }
    const int split = precision == LBC_BF16X2 ? 1 : 0;
    const cudaError_t e = split ? smem_opt_in((const void *)k_lbc_predict_mma<true>, SMEM_MMA_SPLIT, MW_SMEM)
                                : smem_opt_in((const void *)k_lbc_predict_mma<false>, SMEM_MMA, MW_SMEM);
    if (e != cudaSuccess) return e;
    // the blocks of every face that is asked for, side by side
    MFirst first;
    uint32_t blocks = 0;
    for (int f = 0; f < 7; ++f) {
        first.block[f] = blocks;
        if (f < g.nface && (side < 0 || g.face[f].side == side))
            blocks += ((g.face[f].nu + MW_TU - 1) / MW_TU * ((g.face[f].nv + 15) / 16) + MW_WARPS - 1) / MW_WARPS;
    }
    if (!blocks) return cudaSuccess;
    return launch_dependent_smem(split ? k_lbc_predict_mma<true> : k_lbc_predict_mma<false>, dim3(blocks, 1, 1),
                                 (unsigned)MW_WARPS * 32u, MW_SMEM, st, pdl, g, first, memory, (const uint32_t *)W, E, H, pred);
}

cudaError_t launch_lbc_fix(const LGrid &g, int fields, const float *pred, float *E, float *H, const float *ce,
                           const float *cm, float dt, cudaStream_t st, bool pdl)
{
    if (!g.nown) return cudaSuccess;
    const bool e = fields == LBC_FIX_E;
    FixFaces ff = {};
    for (int f = 0; f < g.nface; ++f) {
        const LFace &lf = g.face[f];
        if (lf.side != (e ? 0 : 1)) continue;
        ff.on[lf.axis] = 1;
        ff.col0[lf.axis] = lf.col0;
        ff.nv[lf.axis] = lf.nv;
    }
    // nothing to do; and a launch without a thread that waits for the kernel before it could end first
    if (!ff.on[0] && !ff.on[1] && !ff.on[2]) return cudaSuccess;
    const dim3 grid((g.nown + 127) / 128, 1, 1);
    return e ? launch_dependent_smem(k_lbc_fix<true>, grid, 128u, 0, st, pdl, g, ff, pred, E, (const float *)H, ce, dt)
             : launch_dependent_smem(k_lbc_fix<false>, grid, 128u, 0, st, pdl, g, ff, pred, H, (const float *)E, cm, dt);
}

}  // namespace fdtd
