// ib_mlp.cu -- training kernels of the drag-decay MLP (FP32) and its exact training targets.
//
// The network (16 inputs, 3 x 64 ReLU, 1 linear output; parameter layout IB_MLP_OFF_* in
// imogen_b200.h) is trained on the GPU with these kernels.  A CTA is two groups of 256 threads that
// share the weights in shared memory; each group walks tiles of 64 samples: forward pass with every
// activation in shared memory, back-propagation of the mean squared error, gradients summed over the
// group's tiles in registers.  A CTA writes one gradient to its own row of a workspace and a second
// kernel sums the rows in a fixed order (so the gradient is deterministic); an Adam kernel updates
// the FP32 master parameters.  Inference in the drag step runs the same network in BF16 on the
// tensor cores (ib_drag_learned.cu).
//
// What bounds a step is FP32 FMA issue (27 kMAC a sample: 47 us for 65536 samples at 74 TFLOP/s) as
// long as the operands do not have to come from shared memory one by one: a thread forms 4 x 4
// outputs of a layer from one float4 of each operand per k, with packed f32x2 FMAs.  Activations are
// kept transposed, [unit][sample] with rows of 68 floats, and a thread's four units are 16 apart: 16-byte
// accesses are then free of bank conflicts in all three contractions (over inputs, units and samples).
// The weights' columns are permuted to match when they are loaded.
#include "ib_drag.cuh"
#include "ib_internal.cuh"

namespace ib {

constexpr int MT = 64;    // samples per tile
constexpr int MG = 256;   // threads per group
constexpr int LD = 68;    // floats between units of the activation arrays
constexpr int H = IB_MLP_HID, IN = IB_MLP_IN;

struct alignas(16) MlpGroup {
    float X[IN][LD], H1[H][LD], H2[H][LD], H3[H][LD];
    float yp[4][MT], dy[MT];
};
// Forward weights [input][unit], backward weights [unit][input]; the fast index holds unit (input)
// c + 16 i at 4 c + i
struct alignas(16) MlpSmem {
    float W1f[IN][H], W2f[H][H], W3f[H][H], W2b[H][H], W3b[H][H];
    float b1[H], b2[H], b3[H], w4[H];
    MlpGroup g[2];
};

__device__ __forceinline__ int mlp_perm(int j) { return 4 * (j & 15) + (j >> 4); }

__device__ void mlp_load_params(MlpSmem &s, const float *__restrict__ p, bool backward)
{
    for (int i = threadIdx.x; i < H * IN; i += blockDim.x) s.W1f[i % IN][mlp_perm(i / IN)] = p[IB_MLP_OFF_W1 + i];
    for (int i = threadIdx.x; i < H * H; i += blockDim.x) {
        const int j = i / H, k = i % H;
        const float w2 = p[IB_MLP_OFF_W2 + i], w3 = p[IB_MLP_OFF_W3 + i];
        s.W2f[k][mlp_perm(j)] = w2;
        s.W3f[k][mlp_perm(j)] = w3;
        if (backward) {
            s.W2b[j][mlp_perm(k)] = w2;
            s.W3b[j][mlp_perm(k)] = w3;
        }
    }
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        s.b1[i] = p[IB_MLP_OFF_B1 + i];
        s.b2[i] = p[IB_MLP_OFF_B2 + i];
        s.b3[i] = p[IB_MLP_OFF_B3 + i];
        s.w4[i] = p[IB_MLP_OFF_W4 + i];
    }
}

__device__ __forceinline__ void group_sync(int grp) { asm volatile("bar.sync %0, 256;" ::"r"(grp + 1) : "memory"); }

// two FP32 lanes at once (packed f32x2 arithmetic of sm_100)
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c)
{
    unsigned long long x = *reinterpret_cast<unsigned long long *>(&a), y = *reinterpret_cast<unsigned long long *>(&b),
                       z = *reinterpret_cast<unsigned long long *>(&c);
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(z) : "l"(x), "l"(y));
    return *reinterpret_cast<float2 *>(&z);
}

// acc[i] = samples 4 rg .. 4 rg + 3 of unit cg + 16 i: += sum over k < K of A[k][sample] B[k][unit]
template <int K>
__device__ __forceinline__ void mlp_layer(const float (*A)[LD], const float (*B)[H], int cg, int rg, float2 (&acc)[4][2])
{
#pragma unroll 8
    for (int k = 0; k < K; k++) {
        const float4 a = *reinterpret_cast<const float4 *>(&A[k][4 * rg]);
        const float4 b = *reinterpret_cast<const float4 *>(&B[k][4 * cg]);
        const float2 a0 = make_float2(a.x, a.y), a1 = make_float2(a.z, a.w);
        const float w[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float2 ww = make_float2(w[i], w[i]);
            acc[i][0] = ffma2(a0, ww, acc[i][0]);
            acc[i][1] = ffma2(a1, ww, acc[i][1]);
        }
    }
}

// out = relu(A B + b), zero for samples past `rows`
template <int K>
__device__ __forceinline__ void mlp_dense_relu(const float (*A)[LD], const float (*B)[H], const float *b, float (*out)[LD],
                                               int rows, int cg, int rg)
{
    float2 acc[4][2];
#pragma unroll
    for (int i = 0; i < 4; i++) acc[i][0] = acc[i][1] = make_float2(b[cg + 16 * i], b[cg + 16 * i]);
    mlp_layer<K>(A, B, cg, rg, acc);
    const int r = 4 * rg;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float4 o;
        o.x = (r < rows && acc[i][0].x > 0.f) ? acc[i][0].x : 0.f;
        o.y = (r + 1 < rows && acc[i][0].y > 0.f) ? acc[i][0].y : 0.f;
        o.z = (r + 2 < rows && acc[i][1].x > 0.f) ? acc[i][1].x : 0.f;
        o.w = (r + 3 < rows && acc[i][1].y > 0.f) ? acc[i][1].y : 0.f;
        *reinterpret_cast<float4 *>(&out[cg + 16 * i][r]) = o;
    }
}

// back through a ReLU layer, in place: A[k][sample] becomes (sum over j of G[j][sample] W[j][k]) where
// A > 0, else 0
__device__ __forceinline__ void mlp_dense_back(const float (*G)[LD], const float (*W)[H], float (*A)[LD], int cg, int rg)
{
    float2 acc[4][2];
#pragma unroll
    for (int i = 0; i < 4; i++) acc[i][0] = acc[i][1] = make_float2(0.f, 0.f);
    mlp_layer<H>(G, W, cg, rg, acc);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float4 *cell = reinterpret_cast<float4 *>(&A[cg + 16 * i][4 * rg]);
        float4 o = *cell;
        o.x = (o.x > 0.f) ? acc[i][0].x : 0.f;
        o.y = (o.y > 0.f) ? acc[i][0].y : 0.f;
        o.z = (o.z > 0.f) ? acc[i][1].x : 0.f;
        o.w = (o.w > 0.f) ? acc[i][1].y : 0.f;
        *cell = o;
    }
}

// gw[i][m] += sum over the tile's samples of G[jg + 16 i][sample] A[kg + 16 m][sample]
template <int NK>
__device__ __forceinline__ void mlp_dense_grad(const float (*G)[LD], const float (*A)[LD], int jg, int kg, float (&gw)[4][NK])
{
    float2 acc[4][NK];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int m = 0; m < NK; m++) acc[i][m] = make_float2(0.f, 0.f);
#pragma unroll 2
    for (int r = 0; r < MT; r += 4) {
        float4 g[4], a[NK];
#pragma unroll
        for (int i = 0; i < 4; i++) g[i] = *reinterpret_cast<const float4 *>(&G[jg + 16 * i][r]);
#pragma unroll
        for (int m = 0; m < NK; m++) a[m] = *reinterpret_cast<const float4 *>(&A[kg + 16 * m][r]);
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int m = 0; m < NK; m++) {
                acc[i][m] = ffma2(make_float2(g[i].x, g[i].y), make_float2(a[m].x, a[m].y), acc[i][m]);
                acc[i][m] = ffma2(make_float2(g[i].z, g[i].w), make_float2(a[m].z, a[m].w), acc[i][m]);
            }
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int m = 0; m < NK; m++) gw[i][m] += acc[i][m].x + acc[i][m].y;
}

// sum over a quarter (16 samples) of row j of A, times w if given
__device__ __forceinline__ float mlp_row_sum(const float (*A)[LD], int j, int quarter, const float *w)
{
    float acc = 0.f;
#pragma unroll
    for (int r = 16 * quarter; r < 16 * quarter + 16; r += 4) {
        const float4 v = *reinterpret_cast<const float4 *>(&A[j][r]);
        if (w) {
            const float4 d = *reinterpret_cast<const float4 *>(&w[r]);
            acc = fmaf(v.x, d.x, acc);
            acc = fmaf(v.y, d.y, acc);
            acc = fmaf(v.z, d.z, acc);
            acc = fmaf(v.w, d.w, acc);
        } else {
            acc += (v.x + v.y) + (v.z + v.w);
        }
    }
    return acc;
}

// Forward pass of one tile by one group; leaves the output of sample t in the returned value of thread
// t < MT (others 0).
__device__ __forceinline__ float mlp_tile_forward(const MlpSmem &s, MlpGroup &g, const float *__restrict__ x, int64_t base,
                                                  int rows, float b4, int grp, int t)
{
    const int cg = t & 15, rg = t >> 4;
    {
        const int r = t >> 2, k = 4 * (t & 3);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows) {
            const float *src = x + (base + r) * IN + k;  // the caller's buffer: any 4-byte alignment
            v = make_float4(src[0], src[1], src[2], src[3]);
        }
        g.X[k][r] = v.x;
        g.X[k + 1][r] = v.y;
        g.X[k + 2][r] = v.z;
        g.X[k + 3][r] = v.w;
    }
    group_sync(grp);
    mlp_dense_relu<IN>(g.X, s.W1f, s.b1, g.H1, rows, cg, rg);
    group_sync(grp);
    mlp_dense_relu<H>(g.H1, s.W2f, s.b2, g.H2, rows, cg, rg);
    group_sync(grp);
    mlp_dense_relu<H>(g.H2, s.W3f, s.b3, g.H3, rows, cg, rg);
    group_sync(grp);
    {  // y = b4 + w4 . H3: a quarter of the units per thread
        const int r = t & 63, q = t >> 6;
        float acc = 0.f;
#pragma unroll
        for (int j = 16 * q; j < 16 * q + 16; j++) acc = fmaf(g.H3[j][r], s.w4[j], acc);
        g.yp[q][r] = acc;
    }
    group_sync(grp);
    return (t < MT) ? ((g.yp[0][t] + g.yp[1][t]) + (g.yp[2][t] + g.yp[3][t])) + b4 : 0.f;
}

__global__ void __launch_bounds__(2 * MG) mlp_forward_kernel(const float *__restrict__ p, const float *__restrict__ x,
                                                             int64_t n, float *__restrict__ y)
{
    extern __shared__ __align__(16) unsigned char mlp_smem_raw[];
    MlpSmem &s = *reinterpret_cast<MlpSmem *>(mlp_smem_raw);
    mlp_load_params(s, p, false);
    const float b4 = p[IB_MLP_OFF_B4];
    __syncthreads();
    const int grp = threadIdx.x / MG, t = threadIdx.x % MG;
    const int64_t ntiles = (n + MT - 1) / MT;
    for (int64_t tile = blockIdx.x + (int64_t)grp * gridDim.x; tile < ntiles; tile += 2 * (int64_t)gridDim.x) {
        const int64_t base = tile * MT;
        const int rows = (int)((n - base < (int64_t)MT) ? (n - base) : (int64_t)MT);
        const float v = mlp_tile_forward(s, s.g[grp], x, base, rows, b4, grp, t);
        if (t < rows) y[base + t] = v;
    }
}

// Gradient of the summed loss over this CTA's tiles into partial[blockIdx.x][*], its summed squared
// error into partial[blockIdx.x][IB_MLP_NPARAM].
__global__ void __launch_bounds__(2 * MG) mlp_grad_kernel(const float *__restrict__ p, const float *__restrict__ x,
                                                          const float *__restrict__ target, int64_t n,
                                                          float *__restrict__ partial, int64_t stride)
{
    extern __shared__ __align__(16) unsigned char mlp_smem_raw[];
    MlpSmem &s = *reinterpret_cast<MlpSmem *>(mlp_smem_raw);
    mlp_load_params(s, p, true);
    const float b4 = p[IB_MLP_OFF_B4];
    __syncthreads();
    const int grp = threadIdx.x / MG, t = threadIdx.x % MG;
    MlpGroup &g = s.g[grp];
    const int cg = t & 15, rg = t >> 4;        // layers: units cg + 16 i, samples 4 rg ..
    const int bj = t >> 2, bq = t & 3;         // row sums: unit, quarter of the samples
    const int64_t ntiles = (n + MT - 1) / MT;
    const float inv_n = 1.0f / (float)n;
    // this thread's share of the gradient: units rg + 16 i, inputs cg + 16 m; unit bj's quarter sums
    float gw3[4][4], gw2[4][4], gw1[4][1], gb3 = 0.f, gb2 = 0.f, gb1 = 0.f, gw4 = 0.f, gb4 = 0.f, loss = 0.f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
#pragma unroll
        for (int m = 0; m < 4; m++) gw3[i][m] = gw2[i][m] = 0.f;
        gw1[i][0] = 0.f;
    }
    for (int64_t tile = blockIdx.x + (int64_t)grp * gridDim.x; tile < ntiles; tile += 2 * (int64_t)gridDim.x) {
        const int64_t base = tile * MT;
        const int rows = (int)((n - base < (int64_t)MT) ? (n - base) : (int64_t)MT);
        const float tv = (t < rows) ? target[base + t] : 0.f;
        const float y = mlp_tile_forward(s, g, x, base, rows, b4, grp, t);
        if (t < MT) {
            const float e = (t < rows) ? y - tv : 0.f;
            const float d = 2.f * e * inv_n;
            g.dy[t] = d;
            gb4 += d;
            loss = fmaf(e, e, loss);
        }
        group_sync(grp);
        // output layer: dw4[j] = sum_r dy[r] H3[r][j]; then H3 becomes its own gradient dy w4 (H3 > 0)
        gw4 += mlp_row_sum(g.H3, bj, bq, g.dy);
        __syncwarp();  // a row of H3 is read by the four threads of one warp that rewrite it
        {
            const float w = s.w4[bj];
#pragma unroll
            for (int r = 16 * bq; r < 16 * bq + 16; r += 4) {
                float4 *cell = reinterpret_cast<float4 *>(&g.H3[bj][r]);
                const float4 d = *reinterpret_cast<const float4 *>(&g.dy[r]);
                float4 v = *cell;
                v.x = (v.x > 0.f) ? d.x * w : 0.f;
                v.y = (v.y > 0.f) ? d.y * w : 0.f;
                v.z = (v.z > 0.f) ? d.z * w : 0.f;
                v.w = (v.w > 0.f) ? d.w * w : 0.f;
                *cell = v;
            }
        }
        group_sync(grp);
        mlp_dense_grad<4>(g.H3, g.H2, rg, cg, gw3);
        gb3 += mlp_row_sum(g.H3, bj, bq, nullptr);
        group_sync(grp);
        mlp_dense_back(g.H3, s.W3b, g.H2, cg, rg);
        group_sync(grp);
        mlp_dense_grad<4>(g.H2, g.H1, rg, cg, gw2);
        gb2 += mlp_row_sum(g.H2, bj, bq, nullptr);
        group_sync(grp);
        mlp_dense_back(g.H2, s.W2b, g.H1, cg, rg);
        group_sync(grp);
        mlp_dense_grad<1>(g.H1, g.X, rg, cg, gw1);
        gb1 += mlp_row_sum(g.H1, bj, bq, nullptr);
        group_sync(grp);  // the next tile rewrites X and H1
    }
    // the quarters of a row sum sit in four neighbouring lanes; gb4 and loss in 64 threads
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
        gb3 += __shfl_xor_sync(0xffffffffu, gb3, o);
        gb2 += __shfl_xor_sync(0xffffffffu, gb2, o);
        gb1 += __shfl_xor_sync(0xffffffffu, gb1, o);
        gw4 += __shfl_xor_sync(0xffffffffu, gw4, o);
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        gb4 += __shfl_xor_sync(0xffffffffu, gb4, o);
        loss += __shfl_xor_sync(0xffffffffu, loss, o);
    }
    // the second group hands its sums over in shared memory (the activations are done with), the first
    // adds them to its own
    __syncthreads();
    float *sum = &s.g[0].X[0][0];  // parameter order, then the loss, then the two warps' parts of gb4 and loss
    static_assert(sizeof(MlpGroup) >= (IB_MLP_NPARAM + 8) * sizeof(float), "room for one gradient");
    auto each = [&](auto f) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
#pragma unroll
            for (int m = 0; m < 4; m++) {
                f(IB_MLP_OFF_W3 + (rg + 16 * i) * H + cg + 16 * m, gw3[i][m]);
                f(IB_MLP_OFF_W2 + (rg + 16 * i) * H + cg + 16 * m, gw2[i][m]);
            }
            f(IB_MLP_OFF_W1 + (rg + 16 * i) * IN + cg, gw1[i][0]);
        }
        if (bq == 0) {
            f(IB_MLP_OFF_B3 + bj, gb3);
            f(IB_MLP_OFF_B2 + bj, gb2);
            f(IB_MLP_OFF_B1 + bj, gb1);
            f(IB_MLP_OFF_W4 + bj, gw4);
        }
    };
    if (grp == 1) {
        each([&](int i, float v) { sum[i] = v; });
        if (t == 0 || t == 32) {
            sum[IB_MLP_NPARAM + t / 32] = gb4;
            sum[IB_MLP_NPARAM + 2 + t / 32] = loss;
        }
    } else if (t == 32) {
        sum[IB_MLP_NPARAM + 4] = gb4;
        sum[IB_MLP_NPARAM + 5] = loss;
    }
    __syncthreads();
    if (grp == 0) {
        float *gp = partial + blockIdx.x * stride;
        each([&](int i, float v) { gp[i] = v + sum[i]; });
        if (t == 0) {
            const float *e = sum + IB_MLP_NPARAM;
            gp[IB_MLP_OFF_B4] = (gb4 + e[4]) + (e[0] + e[1]);
            gp[IB_MLP_NPARAM] = (loss + e[5]) + (e[2] + e[3]);
        }
    }
}

// grad[i] = sum over rows of partial[row][i], four interleaved sums per parameter (so that enough loads
// are in flight) added in a fixed order; loss = the rows' summed squared errors / n
__global__ void __launch_bounds__(256) mlp_reduce_kernel(const float *__restrict__ partial, int nrows, int64_t stride,
                                                         float *__restrict__ grad, float *__restrict__ loss, float inv_n)
{
    __shared__ float part[4][64];
    const int c = threadIdx.x & 63, q = threadIdx.x >> 6;
    const int i = blockIdx.x * 64 + c;
    float acc = 0.f;
    if (i <= IB_MLP_NPARAM) {
#pragma unroll 8
        for (int t = q; t < nrows; t += 4) acc += partial[t * stride + i];
    }
    part[q][c] = acc;
    __syncthreads();
    if (q == 0 && i <= IB_MLP_NPARAM) {
        const float v = (part[0][c] + part[1][c]) + (part[2][c] + part[3][c]);
        if (i < IB_MLP_NPARAM) grad[i] = v;
        else if (loss) *loss = v * inv_n;
    }
}

__global__ void mlp_adam_kernel(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                                float *__restrict__ v, int64_t n, float lr, float b1, float b2, float eps, float c1,
                                float c2)
{
    for (int64_t i = threadIdx.x + (int64_t)blockIdx.x * blockDim.x; i < n; i += (int64_t)blockDim.x * gridDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

// Exact LogTrap2 decay exponent s = t k_eff for raw features (rho_g, rho_d, |dv|, u, dt)
__global__ void drag_decay_kernel(const double *__restrict__ f, int64_t n, DragParams d, double *__restrict__ s)
{
    for (int64_t i = threadIdx.x + (int64_t)blockIdx.x * blockDim.x; i < n; i += (int64_t)blockDim.x * gridDim.x) {
        const double g0 = f[5 * i], d0 = f[5 * i + 1], t0 = f[5 * i + 2], t1 = f[5 * i + 3], t = f[5 * i + 4];
        s[i] = t * logtrap_keff<2>(d, g0, d0, t0, t1, t);
    }
}

static int mlp_smem_attr(const void *fn)
{
    static SmemOptIn forward, grad;
    return opt_in(fn == (const void *)mlp_forward_kernel ? forward : grad, fn, sizeof(MlpSmem));
}

}  // namespace ib

using namespace ib;

extern "C" int64_t ib_mlpWorkspaceFloats(int64_t n)
{
    if (n < 1) return 0;
    const int64_t stride = ((int64_t)IB_MLP_NPARAM + 1 + 7) / 8 * 8;
    return ((n + MT - 1) / MT) * stride;
}

extern "C" int ib_mlpLossGrad(const float *params, const float *x, const float *target, int64_t n, float *grad,
                              float *loss_out, float *partial, void *stream)
{
    if (!params || !x || !target || !grad || !partial) return IB_ERROR_NULL_POINTER;
    if (n < 1) return IB_ERROR_INVALID_ARGS;
    cudaStream_t st = (cudaStream_t)stream;
    int rc;
    if ((rc = mlp_smem_attr((const void *)mlp_grad_kernel))) return rc;
    const int64_t ntiles = (n + MT - 1) / MT;
    const int64_t stride = ((int64_t)IB_MLP_NPARAM + 1 + 7) / 8 * 8;
    const int grid = (int)std::min<int64_t>(ntiles, (int64_t)num_sms());
    mlp_grad_kernel<<<grid, 2 * MG, sizeof(MlpSmem), st>>>(params, x, target, n, partial, stride);
    if ((rc = check_launch())) return rc;
    mlp_reduce_kernel<<<(IB_MLP_NPARAM + 1 + 63) / 64, 256, 0, st>>>(partial, grid, stride, grad, loss_out,
                                                                    1.0f / (float)n);
    return check_launch();
}

extern "C" int ib_mlpForward(const float *params, const float *x, int64_t n, float *y, void *stream)
{
    if (!params || !x || !y) return IB_ERROR_NULL_POINTER;
    if (n < 1) return IB_ERROR_INVALID_ARGS;
    int rc;
    if ((rc = mlp_smem_attr((const void *)mlp_forward_kernel))) return rc;
    const int64_t ntiles = (n + MT - 1) / MT;
    const int grid = (int)std::min<int64_t>(ntiles, (int64_t)num_sms());
    mlp_forward_kernel<<<grid, 2 * MG, sizeof(MlpSmem), (cudaStream_t)stream>>>(params, x, n, y);
    return check_launch();
}

extern "C" int ib_mlpAdam(float *params, const float *grad, float *m, float *v, int64_t nparam, float lr, float beta1,
                          float beta2, float eps, int step, void *stream)
{
    if (!params || !grad || !m || !v) return IB_ERROR_NULL_POINTER;
    if (nparam < 1 || step < 1) return IB_ERROR_INVALID_ARGS;
    const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
    mlp_adam_kernel<<<(unsigned)std::min<int64_t>((nparam + 255) / 256, 1024), 256, 0, (cudaStream_t)stream>>>(
        params, grad, m, v, nparam, lr, beta1, beta2, eps, c1, c2);
    return check_launch();
}

extern "C" int ib_dragDecayExact(const double *features, int64_t n, const ib_thermo *tg, const ib_thermo *td,
                                 double *s_out, void *stream)
{
    if (!features || !tg || !td || !s_out) return IB_ERROR_NULL_POINTER;
    if (n < 1) return IB_ERROR_INVALID_ARGS;
    const DragParams d = drag_constants(tg, td);
    const int nb = (int)std::min<int64_t>((n + 255) / 256, (int64_t)16 * num_sms());
    drag_decay_kernel<<<nb, 256, 0, (cudaStream_t)stream>>>(features, n, d, s_out);
    return check_launch();
}
