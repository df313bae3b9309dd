// The tuner's learned cost model: a 3-layer FP32 MLP (D -> 128 -> 128 -> 1,
// ReLU), trained with hand-written forward, backward and Adam kernels.
//
// Parameters are one packed FP32 vector: W1[H][D], b1[H], W2[H][H], b2[H],
// W3[H], b3.  Training minimises the mean squared error of the predicted
// log-time.  Every sum runs in a fixed order (no atomics), so a training run
// on a GPU is deterministic; the backward pass is checked against a
// float64 numpy restatement (oracle/mlp_ref.py).
//
// The matrices are small (H = 128, D = 24), so these are FP32 CUDA-core tiles:
// the model costs microseconds next to the loops it ranks.
#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "../../../include/dvmh_gb.h"
#include "../../../include/dvmh_gb_kernels.h"
#include "devinfo.cuh"

namespace {

constexpr int D = DVMHGB_TUNE_NF, H = 128;
constexpr long OFF_W1 = 0, OFF_B1 = OFF_W1 + (long)H * D, OFF_W2 = OFF_B1 + H, OFF_B2 = OFF_W2 + (long)H * H,
               OFF_W3 = OFF_B2 + H, OFF_B3 = OFF_W3 + H, NPARAM = OFF_B3 + 1;
// ---- forward and backward in one launch, the weight gradients as one partial per CTA
//
// A CTA of 512 threads owns a contiguous range of rows and walks it in tiles of 40.  Both forms of W2 (by
// rows for the input gradients, by columns for the forward pass), W1 by columns and the tile's activations stay
// in shared memory, so a pass over the rows reads X and y once and writes nothing but the CTA's partial gradient,
// which it accumulates in registers over its tiles; kGradFold adds the partials in a fixed order.
//
// What bounds it: shared-memory reads of the weights, then FP32 issue.  A batch of 4096 rows is 0.46 GFLOP, 6 us at
// the FP32 rate.  One launch per layer and direction (13 launches) took 791 us of GPU time, 723 of it in the weight
// gradients: 16 CTAs, each a serial pass over all rows.  Row ranges per CTA give every SM a share of that
// contraction.  A warp multiplies 5 rows by 64 columns (2 a lane): 13 shared-memory cycles per 10 of FMAs, against
// 24 per 8 for 2 rows by 128 columns; 40 rows a tile is one tile per CTA where the partials allow 38.6 rows a CTA.
// Loss, gradient and Adam step on 4096 rows, back to back: 830 us before, 62 with 2 rows by 128 columns, 40 with 5
// by 64, 37 since the fold and Adam are launched while the kernel before them runs.
constexpr int MT = 512;       // threads of a CTA: 16 warps, warps 2g and 2g + 1 on rows 5g .. 5g + 4 of a tile
constexpr int WR = 5, MR = 8 * WR;
constexpr int XP = D + 2;     // row stride of the staged features
constexpr int HP = H + 4;     // row stride of the transposed weights (their stores are 4-way conflicts, not 32-way)
constexpr int MLP_SMEM_FWD = (D * HP + H * HP + MR * XP + MR * H + 2 * MR) * 4;
constexpr int MLP_SMEM = MLP_SMEM_FWD + (H * H + 2 * MR * H + 64) * 4;
static_assert(MT == 2 * 32 * (MR / WR) && H == 2 * 64 && MLP_SMEM <= 227 * 1024, "warp pairs cover the tile");
static_assert(D % 4 == 0 && XP % 2 == 0 && (D * HP) % 4 == 0 && (MR * XP) % 4 == 0, "vector accesses stay aligned");

// acc[r][c] = sum_k In[r][k] * Wt[k][c], k = 0 .. K - 1 in order (In: the warp's first row, row stride IP; Wt: the
// lane's first column, row stride WP)
template <int K, int IP, int WP>
__device__ __forceinline__ void rowsBy2(const float *In, const float *Wt, float acc[WR][2]) {
#pragma unroll 4
    for (int k = 0; k < K; k += 2) {
        const float2 w0 = *reinterpret_cast<const float2 *>(Wt + k * WP);
        const float2 w1 = *reinterpret_cast<const float2 *>(Wt + (k + 1) * WP);
#pragma unroll
        for (int r = 0; r < WR; r++) {
            const float2 x = *reinterpret_cast<const float2 *>(In + r * IP + k);
            acc[r][0] = fmaf(x.x, w0.x, acc[r][0]);
            acc[r][1] = fmaf(x.x, w0.y, acc[r][1]);
            acc[r][0] = fmaf(x.y, w1.x, acc[r][0]);
            acc[r][1] = fmaf(x.y, w1.y, acc[r][1]);
        }
    }
}

// one value per column and row group, summed over the CTA's 8 row groups in order, to out[0 .. H - 1]
__device__ __forceinline__ void columnsOut(float *sm, const float v[2], int group, int col, float *out) {
    __syncthreads();
    *reinterpret_cast<float2 *>(sm + group * H + col) = make_float2(v[0], v[1]);
    __syncthreads();
    if (threadIdx.x < H) {
        float s = 0;
        for (int w = 0; w < MR / WR; w++) s += sm[w * H + threadIdx.x];
        out[threadIdx.x] = s;
    }
}

// Rows [blockIdx.x * per, +per) of n: pred (when not null), and with GRAD the gradient of the mean squared error
// over these rows, out[blockIdx.x * pitch + p] for parameter p, the rows' sum of squared errors after them
// (to *lossOut / n instead when the launch is one CTA: out is then the gradient itself).
template <bool GRAD>
__global__ void __launch_bounds__(MT, 1)
    kMlp(const float *__restrict__ P, const float *__restrict__ X, const float *__restrict__ y, long n, long per,
         float *pred, float *out, long pitch, float *lossOut) {
    extern __shared__ __align__(16) float sm[];
    float *W1t = sm, *W2t = W1t + D * HP, *Xs = W2t + H * HP, *H1 = Xs + MR * XP, *ps = H1 + MR * H;
    gbdev::nextMayLaunch();
    float *W2 = ps + 2 * MR, *Z2 = W2 + H * H, *Z1 = Z2 + MR * H, *es = Z1 + MR * H;
    const int tid = threadIdx.x, lane = tid & 31, group = tid >> 6, half = (tid >> 5) & 1;
    const int row0 = WR * group, col0 = 64 * half + 2 * lane;
    for (int q = tid; q < D * H; q += MT) W1t[(q % D) * HP + q / D] = P[OFF_W1 + q];
    for (int q = tid; q < H * H; q += MT) {
        const float w = P[OFF_W2 + q];
        W2t[(q % H) * HP + q / H] = w;
        if (GRAD) W2[q] = w;
    }
    float b1[2], b2[2], w3[2];
#pragma unroll
    for (int c = 0; c < 2; c++) {
        b1[c] = P[OFF_B1 + col0 + c];
        b2[c] = P[OFF_B2 + col0 + c];
        w3[c] = P[OFF_W3 + col0 + c];
    }
    const float b3 = P[OFF_B3];
    // gradient shares: W2's 4 x 8 block (rows 4 (tid / 16) .., columns 4 (tid % 16) .. and those + 64), W1's 1 x 6
    float g2[4][8] = {}, g1[6] = {}, gw3[2] = {}, gb2[2] = {}, gb1[2] = {}, gb3 = 0, loss = 0;
    const int o2 = 4 * (tid >> 4), i2 = 4 * (tid & 15), o1 = tid >> 2, i1 = 6 * (tid & 3);
    const long ra = blockIdx.x * per, rb = ra + per < n ? ra + per : n;
    for (long r0 = ra; r0 < rb; r0 += MR) {
        __syncthreads();  // the last tile's readers are done (first tile: the weights are in place after the next one)
        for (int q = tid; q < MR * D; q += MT) {
            const int r = q / D, c = q - r * D;
            Xs[r * XP + c] = r0 + r < rb ? X[(r0 + r) * D + c] : 0.0f;
        }
        __syncthreads();
        float h1[WR][2] = {}, h2[WR][2] = {};
        rowsBy2<D, XP, HP>(Xs + row0 * XP, W1t + col0, h1);
#pragma unroll
        for (int r = 0; r < WR; r++) {
            const bool in = r0 + row0 + r < rb;
#pragma unroll
            for (int c = 0; c < 2; c++) h1[r][c] = in ? fmaxf(h1[r][c] + b1[c], 0.0f) : 0.0f;
            *reinterpret_cast<float2 *>(H1 + (row0 + r) * H + col0) = make_float2(h1[r][0], h1[r][1]);
        }
        __syncthreads();
        rowsBy2<H, H, HP>(H1 + row0 * H, W2t + col0, h2);
#pragma unroll
        for (int r = 0; r < WR; r++) {
            const bool in = r0 + row0 + r < rb;
#pragma unroll
            for (int c = 0; c < 2; c++) h2[r][c] = in ? fmaxf(h2[r][c] + b2[c], 0.0f) : 0.0f;
            float p = fmaf(h2[r][1], w3[1], h2[r][0] * w3[0]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
            if (lane == 0) ps[half * MR + row0 + r] = p;
        }
        __syncthreads();
        if (pred && tid < MR && r0 + tid < rb) pred[r0 + tid] = (ps[tid] + ps[MR + tid]) + b3;
        if (!GRAD) continue;
#pragma unroll
        for (int r = 0; r < WR; r++) {
            const long row = r0 + row0 + r;
            const float e = row < rb ? ((ps[row0 + r] + ps[MR + row0 + r]) + b3) - y[row] : 0.0f;
            const float d = 2.0f * e / (float)n;
            loss += e * e;
            gb3 += d;
            float z[2];  // dZ2 = d W3 where H2 > 0
#pragma unroll
            for (int c = 0; c < 2; c++) {
                gw3[c] = fmaf(d, h2[r][c], gw3[c]);
                z[c] = h2[r][c] <= 0.0f ? 0.0f : d * w3[c];
                gb2[c] += z[c];
            }
            *reinterpret_cast<float2 *>(Z2 + (row0 + r) * H + col0) = make_float2(z[0], z[1]);
        }
        __syncthreads();
        float z1[WR][2] = {};  // dZ1 = (dZ2 . W2) where H1 > 0
        rowsBy2<H, H, H>(Z2 + row0 * H, W2 + col0, z1);
#pragma unroll
        for (int r = 0; r < WR; r++) {
#pragma unroll
            for (int c = 0; c < 2; c++) {
                if (h1[r][c] <= 0.0f) z1[r][c] = 0.0f;
                gb1[c] += z1[r][c];
            }
            *reinterpret_cast<float2 *>(Z1 + (row0 + r) * H + col0) = make_float2(z1[r][0], z1[r][1]);
        }
        __syncthreads();
        // weight gradients: the tile's rows in order
#pragma unroll 4
        for (int r = 0; r < MR; r++) {
            const float4 zo = *reinterpret_cast<const float4 *>(Z2 + r * H + o2);
            const float4 ha = *reinterpret_cast<const float4 *>(H1 + r * H + i2);
            const float4 hb = *reinterpret_cast<const float4 *>(H1 + r * H + 64 + i2);
            const float zv[4] = {zo.x, zo.y, zo.z, zo.w}, hv[8] = {ha.x, ha.y, ha.z, ha.w, hb.x, hb.y, hb.z, hb.w};
#pragma unroll
            for (int o = 0; o < 4; o++)
#pragma unroll
                for (int i = 0; i < 8; i++) g2[o][i] = fmaf(zv[o], hv[i], g2[o][i]);
            const float zr = Z1[r * H + o1];
#pragma unroll
            for (int i = 0; i < 6; i += 2) {
                const float2 x = *reinterpret_cast<const float2 *>(Xs + r * XP + i1 + i);
                g1[i] = fmaf(zr, x.x, g1[i]);
                g1[i + 1] = fmaf(zr, x.y, g1[i + 1]);
            }
        }
    }
    if (!GRAD) return;
    float *g = out + blockIdx.x * pitch;
#pragma unroll
    for (int o = 0; o < 4; o++)
#pragma unroll
        for (int i = 0; i < 8; i++) g[OFF_W2 + (long)(o2 + o) * H + (i < 4 ? i2 + i : 60 + i2 + i)] = g2[o][i];
#pragma unroll
    for (int i = 0; i < 6; i++) g[OFF_W1 + (long)o1 * D + i1 + i] = g1[i];
    float *red = H1;  // 8 row groups x 128 columns
    columnsOut(red, gw3, group, col0, g + OFF_W3);
    columnsOut(red, gb2, group, col0, g + OFF_B2);
    columnsOut(red, gb1, group, col0, g + OFF_B1);
    if ((tid & 63) == 0) {  // every thread of a row group holds the same two sums
        es[group] = gb3;
        es[32 + group] = loss;
    }
    __syncthreads();
    if (tid == 0) {
        float s = 0, l = 0;
        for (int w = 0; w < MR / WR; w++) s += es[w], l += es[32 + w];
        g[OFF_B3] = s;
        if (gridDim.x > 1)
            g[NPARAM] = l;
        else if (lossOut)
            *lossOut = l / (float)n;
    }
}

// grad[p] = sum over the CTAs' partials, 8 interleaved chains of CTAs per parameter and then those in order
__global__ void __launch_bounds__(256) kGradFold(const float *__restrict__ part, int ctas, long pitch, long n,
                                                 float *grad, float *loss) {
    __shared__ float sh[8][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const long p = blockIdx.x * 32L + tx;
    float s = 0;
    gbdev::nextMayLaunch();
    gbdev::waitForKernelBefore();
    if (p <= NPARAM) {
#pragma unroll 4
        for (int c = ty; c < ctas; c += 8) s += part[c * pitch + p];
    }
    sh[ty][tx] = s;
    __syncthreads();
    if (ty == 0 && p <= NPARAM) {
        for (int q = 1; q < 8; q++) s += sh[q][tx];
        if (p < NPARAM)
            grad[p] = s;
        else if (loss)
            *loss = s / (float)n;
    }
}

// Rows per CTA, at least a tile: a CTA loads 76 KB of weights (140 KB in shared memory) whatever its rows.
long rowsPerCta(long n, long ctas) {
    const long per = (n + ctas - 1) / ctas;
    return per < MR ? MR : per;
}

template <bool GRAD>
bool mlpShared() {  // raised once per device
    static std::atomic<int> occ[gbdev::MAX_DEVICES];
    return gbdev::residentCtas(occ, kMlp<GRAD>, MT, GRAD ? MLP_SMEM : MLP_SMEM_FWD) >= 1;
}

__global__ void kAdam(float *p, const float *g, float *m, float *v, long cnt, float lr, float b1, float b2, float eps,
                      float c1, float c2) {
    gbdev::waitForKernelBefore();
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < cnt; i += (long)gridDim.x * blockDim.x) {
        float mi = b1 * m[i] + (1 - b1) * g[i];
        float vi = b2 * v[i] + (1 - b2) * g[i] * g[i];
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

// He-style uniform initialisation from a counter-based hash (splitmix64)
__global__ void kInit(float *p, unsigned long long seed) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < NPARAM; i += (long)gridDim.x * blockDim.x) {
        unsigned long long z = seed + (unsigned long long)(i + 1) * 0x9E3779B97F4A7C15ull;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        float u = (float)(z >> 40) * (1.0f / 16777216.0f) * 2.0f - 1.0f;
        float scale = i < OFF_B1 ? sqrtf(6.0f / D) : (i < OFF_W2 ? 0.0f : (i < OFF_B2 ? sqrtf(6.0f / H)
                      : (i < OFF_W3 ? 0.0f : (i < OFF_B3 ? sqrtf(3.0f / H) : 0.0f))));
        p[i] = u * scale;
    }
}

}  // namespace

extern "C" {

long dvmhgb_mlp_nparams(void) { return NPARAM; }

// work floats for n rows (the gradient's partials take what of it they need)
long dvmhgb_mlp_work_floats(long n) { return 4 * n * H + 2 * n + 1024; }

int dvmhgb_mlp_init(float *params, unsigned long long seed, void *stream) {
    if (!params) return -1;
    kInit<<<64, 256, 0, (cudaStream_t)stream>>>(params, seed);
    dvmhgb_count_launches(1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int dvmhgb_mlp_forward(const float *P, const float *X, long n, float *pred, float *work, void *stream) {
    if (!P || !X || !pred || !work || n < 1 || !mlpShared<false>()) return -1;
    const long per = rowsPerCta(n, gbdev::smCount());
    kMlp<false><<<(unsigned)((n + per - 1) / per), MT, MLP_SMEM_FWD, (cudaStream_t)stream>>>(P, X, nullptr, n, per, pred,
                                                                                            nullptr, 0, nullptr);
    dvmhgb_count_launches(1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// gradient of the mean squared error of the prediction w.r.t. every parameter
int dvmhgb_mlp_loss_grad(const float *P, const float *X, const float *y, long n, float *grad, float *loss,
                         float *work, void *stream) {
    if (!P || !X || !y || !grad || !work || n < 1 || !mlpShared<true>()) return -1;
    cudaStream_t s = (cudaStream_t)stream;
    // one CTA per SM, as many as `work` holds partials for (38.6 rows' worth of it each); a single CTA writes grad
    const long pitch = NPARAM + 1, room = dvmhgb_mlp_work_floats(n) / pitch;
    const long ctas = room < 1 ? 1 : (room < gbdev::smCount() ? room : gbdev::smCount());
    const long per = rowsPerCta(n, ctas), grid = (n + per - 1) / per;
    kMlp<true><<<(unsigned)grid, MT, MLP_SMEM, s>>>(P, X, y, n, per, nullptr, grid > 1 ? work : grad, pitch, loss);
    if (grid > 1 && gbdev::launchAfter(kGradFold, (unsigned)((pitch + 31) / 32), 256, s, work, (int)grid, pitch, n, grad,
                                       loss) != cudaSuccess)
        return -1;
    dvmhgb_count_launches(grid > 1 ? 2 : 1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int dvmhgb_mlp_adam(float *P, const float *grad, float *m, float *v, long step, float lr, void *stream) {
    if (!P || !grad || !m || !v || step < 1) return -1;
    const float b1 = 0.9f, b2 = 0.999f;
    float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
    if (gbdev::launchAfter(kAdam, 64, 256, (cudaStream_t)stream, P, grad, m, v, NPARAM, lr, b1, b2, 1e-8f, c1, c2) !=
        cudaSuccess)
        return -1;
    dvmhgb_count_launches(1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// Minibatch Adam on the GPU: X[n][D], y[n] host arrays (rows in the order given,
// batches taken in order every epoch).  Returns 0; params (NPARAM floats) and
// losses (one per epoch: loss of the last batch) written to host memory.
int dvmhgb_mlp_train(const float *X, const float *y, long n, int epochs, long batch, float lr,
                     unsigned long long seed, float *params, float *losses) {
    if (!X || !y || !params || n < 1 || epochs < 1 || batch < 1) return -1;
    cudaStream_t s = nullptr;
    float *dX, *dY, *dP, *dG, *dM, *dV, *work, *dLoss;
    if (batch > n) batch = n;
    size_t ok = 0;
    ok |= cudaMalloc(&dX, sizeof(float) * n * D);
    ok |= cudaMalloc(&dY, sizeof(float) * n);
    ok |= cudaMalloc(&dP, sizeof(float) * NPARAM);
    ok |= cudaMalloc(&dG, sizeof(float) * NPARAM);
    ok |= cudaMalloc(&dM, sizeof(float) * NPARAM);
    ok |= cudaMalloc(&dV, sizeof(float) * NPARAM);
    ok |= cudaMalloc(&work, sizeof(float) * dvmhgb_mlp_work_floats(batch));
    ok |= cudaMalloc(&dLoss, sizeof(float));
    if (ok) return -1;
    cudaMemcpy(dX, X, sizeof(float) * n * D, cudaMemcpyHostToDevice);
    cudaMemcpy(dY, y, sizeof(float) * n, cudaMemcpyHostToDevice);
    cudaMemset(dM, 0, sizeof(float) * NPARAM);
    cudaMemset(dV, 0, sizeof(float) * NPARAM);
    dvmhgb_mlp_init(dP, seed, s);
    long step = 0;
    for (int ep = 0; ep < epochs; ep++) {
        for (long b0 = 0; b0 < n; b0 += batch) {
            long nb = (b0 + batch <= n) ? batch : n - b0;
            dvmhgb_mlp_loss_grad(dP, dX + b0 * D, dY + b0, nb, dG, dLoss, work, s);
            dvmhgb_mlp_adam(dP, dG, dM, dV, ++step, lr, s);
        }
        if (losses) cudaMemcpy(&losses[ep], dLoss, sizeof(float), cudaMemcpyDeviceToHost);
    }
    cudaMemcpy(params, dP, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost);
    cudaError_t e = cudaGetLastError();
    cudaFree(dX);
    cudaFree(dY);
    cudaFree(dP);
    cudaFree(dG);
    cudaFree(dM);
    cudaFree(dV);
    cudaFree(work);
    cudaFree(dLoss);
    return e == cudaSuccess ? 0 : -1;
}

}  // extern "C"
