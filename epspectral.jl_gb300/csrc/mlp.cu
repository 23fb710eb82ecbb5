// mlp.cu -- the learned warm start: a small multilayer perceptron, its training and its inference,
// on the GPU with hand-written kernels.
//
// Network: L fully connected layers d_0 -> d_1 -> ... -> d_L, SiLU between layers, linear output.
// Weights W_l [d_{l+1}][d_l] (row-major) are kept in FP32 (the optimiser's master copy) and used in
// BF16 by the products (BF16 weights, FP32 accumulation); biases FP32. The loss is the mean squared
// error over the batch and the outputs; the optimiser is Adam. Every product of the training, of
// the gradient and of the prediction runs on the tensor cores (tc_gemm_launch: tcgen05, TMA, TMEM)
// with the FP32 activations and gradients split into three BF16 parts (~2^-24 relative, as FP32:
// three products against the BF16 weights, six between two such operands), every reduction in fixed
// order, so a training run is bitwise reproducible. The scGD0 hook's inference (forward_tc) splits
// the activations into two parts.
#include "common.cuh"
#include "tc_gemm.cuh"
#include "warmstart.cuh"

#include <cuda_bf16.h>

#include <cmath>
#include <memory>

namespace epsp {

// C[m scm + n scn] = Σ_z P[z][m][n], z ascending.
__global__ void partial_sum_kernel(const float* __restrict__ P, int M, int N, int nz, float* __restrict__ C, long scm,
                                   long scn) {
  const long k = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= long(M) * N) return;
  float acc = 0.f;
  for (int z = 0; z < nz; ++z) acc += P[long(z) * M * N + k];
  C[(k / N) * scm + (k % N) * scn] = acc;
}

__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + expf(-x)); }

// One pass over a [rows][cols] matrix in 32 x 32 tiles. The value v(m, j) is, by MODE:
//   kEmitCopy    src[m ld_src + j];
//   kEmitBiasAct z = Σ_s part[s pstride + j + cols m] + bias[j] (a product's split-K slabs, summed in
//                order), written to Zout[m cols + j] when given, then v = SiLU(z) if act, else z;
//   kEmitActBack Σ_s part[s pstride + j + cols m] times SiLU'(Zin[m cols + j]);
//   kEmitGather  src[idx[m] ld_src + j], idx = B.perm + *B.cur B.batch (the minibatch's rows);
//   kEmitLoss    inv_nd2 (z - Y[idx[m] cols + j]), z as in kEmitBiasAct (linear, written to Zout): the loss gradient.
// v goes to out32[m cols + j] (FP32) and, as three BF16 parts, to rp[p rpart + m ldr + j] (rows)
// and tp[p tpart + j ldt + m] (transposed, through shared memory; columns m in [rows, ldt) get
// zeros, so that the padded K of a product over the rows adds nothing). Grid (cols / 32, M / 32)
// with M = ldt when tp is given, else rows; 32 x 8 threads.
enum { kEmitCopy = 0, kEmitBiasAct = 1, kEmitActBack = 2, kEmitGather = 3, kEmitLoss = 4 };
// A training step's minibatch: its rows are perm[*cur batch ..], its targets Y.
struct Batch {
  const int64_t* perm = nullptr;
  const int* cur = nullptr;
  long batch = 0;
  const float* Y = nullptr;
  float inv_nd2 = 0.f;
};
template <int MODE>
__global__ void __launch_bounds__(256)
    emit_kernel(int rows, int cols, const float* __restrict__ src, long ld_src, const float* __restrict__ part, int splits,
                long pstride, const float* __restrict__ bias, bool act, const float* __restrict__ Zin,
                float* __restrict__ Zout, float* __restrict__ out32, __nv_bfloat16* __restrict__ rp, long ldr, long rpart,
                __nv_bfloat16* __restrict__ tp, long ldt, long tpart, const Batch B = Batch()) {
  __shared__ float tile[32][33];
  const int64_t* idx = nullptr;
  if constexpr (MODE == kEmitGather || MODE == kEmitLoss) idx = B.perm + *B.cur * B.batch;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int j0 = blockIdx.x * 32, m0 = blockIdx.y * 32;
  const int j = j0 + tx;
  // the slabs of the thread's four elements, each in ascending order, all loads of a slab and several slabs in flight
  float sum[4] = {0.f, 0.f, 0.f, 0.f};
  if constexpr (MODE == kEmitBiasAct || MODE == kEmitActBack || MODE == kEmitLoss) {
    const float* q[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) q[r] = part + min(j, cols - 1) + long(cols) * min(m0 + ty + 8 * r, rows - 1);
    int sp = 0;
    for (; sp + 4 <= splits; sp += 4) {
      float x[4][4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int r = 0; r < 4; ++r) x[u][r] = q[r][(sp + u) * pstride];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int r = 0; r < 4; ++r) sum[r] += x[u][r];
    }
    for (; sp < splits; ++sp)
#pragma unroll
      for (int r = 0; r < 4; ++r) sum[r] += q[r][sp * pstride];
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int ml = ty + 8 * r, m = m0 + ml;
    float v = 0.f;
    if (m < rows && j < cols) {
      if constexpr (MODE == kEmitCopy) {
        v = src[long(m) * ld_src + j];
      } else if constexpr (MODE == kEmitGather) {
        v = src[idx[m] * ld_src + j];
      } else {
        const float acc = sum[r];
        if constexpr (MODE == kEmitBiasAct) {
          const float z = acc + bias[j];
          if (Zout) Zout[long(m) * cols + j] = z;
          v = act ? z * sigmoidf_(z) : z;
        } else if constexpr (MODE == kEmitLoss) {
          const float z = acc + bias[j];
          Zout[long(m) * cols + j] = z;
          const float e = z - B.Y[idx[m] * cols + j];
          v = B.inv_nd2 * e;
        } else {
          const float z = Zin[long(m) * cols + j], sg = sigmoidf_(z);
          v = acc * (sg * (1.f + z * (1.f - sg)));
        }
      }
      if (out32) out32[long(m) * cols + j] = v;
      if (rp) {
        __nv_bfloat16 q[3];
        split_bf16_n(v, 3, q);
#pragma unroll
        for (int p = 0; p < 3; ++p) rp[p * rpart + long(m) * ldr + j] = q[p];
      }
    }
    tile[ml][tx] = v;
  }
  if (!tp) return;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int jl = ty + 8 * r, jj = j0 + jl, m = m0 + tx;
    if (jj >= cols || m >= ldt) continue;
    __nv_bfloat16 q[3];
    split_bf16_n(tile[tx][jl], 3, q);  // zero for m >= rows
#pragma unroll
    for (int p = 0; p < 3; ++p) tp[p * tpart + long(jj) * ldt + m] = q[p];
  }
}

// db[j] = Σ_m dZ[m][j] in ascending m.
__global__ void bias_grad_kernel(const float* __restrict__ dZ, long n, int d, float* __restrict__ db) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= d) return;
  float s = 0.f;
  for (long m = 0; m < n; ++m) s += dZ[m * d + j];
  db[j] = s;
}

// dY = 2 (P - Y) / (n d) and per-row sums of squared errors; one block per row, fixed order.
__global__ void __launch_bounds__(256) mse_kernel(const float* __restrict__ P, const float* __restrict__ Y, int d,
                                                  float inv_nd2, float* __restrict__ dY, float* __restrict__ row_loss) {
  __shared__ float sh[256];
  const long m = blockIdx.x;
  float s = 0.f;
  for (int j = threadIdx.x; j < d; j += 256) {
    const float e = P[m * d + j] - Y[m * d + j];
    s += e * e;
    dY[m * d + j] = inv_nd2 * e;
  }
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if (threadIdx.x < st) sh[threadIdx.x] += sh[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) row_loss[m] = sh[0];
}

// out[slot] = Σ_k x[k] (one block, fixed order, FP64 accumulation).
__global__ void sum_kernel(const float* __restrict__ x, long n, double* __restrict__ out, int slot) {
  __shared__ double sh[256];
  double s = 0;
  for (long k = threadIdx.x; k < n; k += 256) s += x[k];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if (threadIdx.x < st) sh[threadIdx.x] += sh[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[slot] = sh[0];
}

// A training step's row losses (mse_kernel's, the targets gathered), and their sum into out[*cur], after which the
// cursor and Adam's step count move on: every reader of this step's cursor has run, Adam reads the new count.
__global__ void __launch_bounds__(256) row_loss_kernel(const float* __restrict__ P, int d, const Batch B,
                                                       float* __restrict__ row_loss) {
  __shared__ float sh[256];
  const long m = blockIdx.x;
  const float* Y = B.Y + B.perm[*B.cur * B.batch + m] * d;
  float s = 0.f;
  for (int j = threadIdx.x; j < d; j += 256) {
    const float e = P[m * d + j] - Y[j];
    s += e * e;
  }
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if (threadIdx.x < st) sh[threadIdx.x] += sh[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) row_loss[m] = sh[0];
}
__global__ void loss_step_kernel(const float* __restrict__ x, long n, double* __restrict__ out, int* cur, int* step) {
  __shared__ double sh[256];
  double s = 0;
  for (long k = threadIdx.x; k < n; k += 256) s += x[k];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if (threadIdx.x < st) sh[threadIdx.x] += sh[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[*cur] = sh[0];
    *cur += 1;
    *step += 1;
  }
}

// BF16 copies of the weight element k = o d_in + i of W [d_out][d_in]: wbf[k], the tensor-core
// products' rows wp[o ldp + i] and the transposed rows wt[i ldt + o].
__device__ __forceinline__ void store_wbf(long k, float w, int din, __nv_bfloat16* __restrict__ wbf,
                                          __nv_bfloat16* __restrict__ wp, long ldp, __nv_bfloat16* __restrict__ wt,
                                          long ldt) {
  const __nv_bfloat16 h = __float2bfloat16_rn(w);
  wbf[k] = h;
  const long o = k / din, i = k % din;
  wp[o * ldp + i] = h;
  wt[i * ldt + o] = h;
}

// Adam step *t on every layer's weights in one launch, tiles of 32 x 32, the gradient summed from its product's
// split-K slabs (element k = o d_in + i of slab z at z pstride + k, z ascending) as it is read; writes the BF16 copies
// the products use, the transposed one through shared memory. (One launch a block of parameters with separate
// slab sums took 12 launches a step and wrote the transposed weights 2 bytes at a time.)
struct AdamLayer {
  float *w, *m1, *m2;
  const float* slab;
  long pstride, ldp, ldt;
  __nv_bfloat16 *wbf, *wp, *wt;
  int splits, din, dout, tile0;  // the layer's first tile
};
struct AdamAll {
  AdamLayer l[16];
  int L;
  float lr, b1, b2, eps;
  const int* t;
};
// One parameter: the new moments stored, the new value returned.
__device__ __forceinline__ float adam_one(float w, float gk, float* m1, float* m2, float lr, float b1, float b2, float eps,
                                          float c1, float c2) {
  const float a = b1 * *m1 + (1.f - b1) * gk;
  const float v = b2 * *m2 + (1.f - b2) * gk * gk;
  *m1 = a;
  *m2 = v;
  return w - lr * (a / c1) / (sqrtf(v / c2) + eps);
}
__global__ void __launch_bounds__(256) adam_weights_kernel(const __grid_constant__ AdamAll A) {
  __shared__ __nv_bfloat16 tile[32][33];
  __shared__ float sc[2];
  int l = 0;
  while (l + 1 < A.L && int(blockIdx.x) >= A.l[l + 1].tile0) ++l;
  const AdamLayer& y = A.l[l];
  const int tx = threadIdx.x % 32, ty = threadIdx.x / 32;
  if (threadIdx.x == 0) {
    sc[0] = 1.f - powf(A.b1, float(*A.t));
    sc[1] = 1.f - powf(A.b2, float(*A.t));
  }
  const int ti = (y.din + 31) / 32, tl = int(blockIdx.x) - y.tile0;
  const int i0 = (tl % ti) * 32, o0 = (tl / ti) * 32;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int o = o0 + ty + 8 * r, i = i0 + tx;
    if (o >= y.dout || i >= y.din) continue;
    const long k = long(o) * y.din + i;
    float g = 0.f;
#pragma unroll 4
    for (int z = 0; z < y.splits; ++z) g += y.slab[z * y.pstride + k];
    const float wn = adam_one(y.w[k], g, y.m1 + k, y.m2 + k, A.lr, A.b1, A.b2, A.eps, sc[0], sc[1]);
    y.w[k] = wn;
    const __nv_bfloat16 h = __float2bfloat16_rn(wn);
    y.wbf[k] = h;
    y.wp[o * y.ldp + i] = h;
    tile[ty + 8 * r][tx] = h;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = i0 + ty + 8 * r, o = o0 + tx;
    if (o < y.dout && i < y.din) y.wt[i * y.ldt + o] = tile[tx][ty + 8 * r];
  }
}
// The biases of every layer: db[j] = Σ_m dZ[m][j] in ascending m (32 loads in flight), then their Adam step.
struct BiasLayer {
  const float* dz;
  float *b, *m1, *m2;
  int d, col0;
};
struct BiasAll {
  BiasLayer l[16];
  int L, cols;
  long n;
  float lr, b1, b2, eps;
  const int* t;
};
__global__ void __launch_bounds__(32) adam_bias_kernel(const __grid_constant__ BiasAll A) {
  const int c = blockIdx.x * 32 + threadIdx.x;
  if (c >= A.cols) return;
  int l = 0;
  while (l + 1 < A.L && c >= A.l[l + 1].col0) ++l;
  const BiasLayer& y = A.l[l];
  const int j = c - y.col0;
  float s = 0.f;
#pragma unroll 32
  for (long m = 0; m < A.n; ++m) s += y.dz[m * y.d + j];
  const float c1 = 1.f - powf(A.b1, float(*A.t)), c2 = 1.f - powf(A.b2, float(*A.t));
  y.b[j] = adam_one(y.b[j], s, y.m1 + j, y.m2 + j, A.lr, A.b1, A.b2, A.eps, c1, c2);
}

__global__ void to_bf16_kernel(const float* __restrict__ w, long n, int din, __nv_bfloat16* __restrict__ wbf,
                               __nv_bfloat16* __restrict__ wp, long ldp, __nv_bfloat16* __restrict__ wt, long ldt) {
  long k = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k < n) store_wbf(k, w[k], din, wbf, wp, ldp, wt, ldt);
}

struct Mlp {
  Ctx* ctx = nullptr;
  int L = 0;
  std::vector<int> dims;
  std::vector<DBuf<float>> W, b, gW, gb, mW, vW, mb, vb;
  std::vector<DBuf<__nv_bfloat16>> Wbf;
  std::vector<DBuf<float>> Z, X;  // per layer, sized for the largest batch
  DBuf<float> dA, dB, loss_rows, Yb;
  DBuf<int> d_err;                // the tensor-core products' bounded-wait flag
  DBuf<double> loss_sum;
  DBuf<int> d_step;  // Adam's step counter, and the training epoch's next minibatch
  long cap = 0;      // rows the activation buffers hold
  DBuf<float> dataX, dataY;
  DBuf<int64_t> perm;  // the epoch's row order
  long ndata = 0;
  DBuf<float> x_mean, x_std, y_mean;  // feature standardisation for the in-iteration hook
  float y_scale = 1.f;
  bool scaled = false;
  long wgen = 0;  // bumped whenever the weights change (set_params, train)
  double train_ms = 0;  // device milliseconds of the last training's epochs
  // Tensor-core inference: weights as the B operand [d_{l+1}][d_l padded to 8] (hi = the BF16
  // weights, lo = 0), activations as the A operand (BF16 hi/lo of the FP32 values) [cap][d_l
  // padded], split-K partials; rebuilt when wgen or the row capacity changes.
  struct Infer {
    long wgen = -1, cap = 0;
    std::vector<int> dpad, bn;
    std::vector<DBuf<__nv_bfloat16>> Wh, Wl, Ah, Al;
    std::vector<TcOperand> opA, opB;
    DBuf<float> part;
  } inf;
  // Tensor-core training and prediction (three BF16 parts per operand, FP32 accumulation). Layer l
  // (d_l -> d_{l+1}), batches of up to cap rows, rows padded to ldT = cap rounded up to 8:
  //   forward   Z_l^T = W_l X_l^T     A = W_l  [d_{l+1}][dp_l]  B = Xs_l  [cap][dp_l]      K = d_l
  //   gradient  gW_l^T = X_l^T dZ_l   A = XT_l [d_l][ldT]       B = dZT_l [d_{l+1}][ldT]   K = rows
  //   backward  dX_l^T = W_l^T dZ_l^T A = WT_l [d_l][dp_{l+1}]  B = dZs_l [cap][dp_{l+1}]  K = d_{l+1}
  // (dp_l = d_l padded to 8: 16-byte rows); the activation and gradient buffers hold their three
  // parts one after the other.
  struct Train {
    long cap = 0, ldT = 0;
    std::vector<int> dp;
    std::vector<DBuf<__nv_bfloat16>> Wp, WT, Xs, XT, dZs, dZT;
    std::vector<TcOperand> opW, opWT, opXs, opXT, opdZs, opdZT;
    DBuf<float> part;
    // a training step's FP32 dZ and gradient slabs of every layer, and the stream that runs beside the backward chain
    std::vector<DBuf<float>> dz, slab;
    struct Side {
      cudaStream_t s = nullptr;
      cudaEvent_t fork = nullptr, join = nullptr;
      ~Side() {
        if (fork) cudaEventDestroy(fork);
        if (join) cudaEventDestroy(join);
        if (s) cudaStreamDestroy(s);
      }
    } side;
  } tr;
};

// X[i][j] = (feature j of state i - x_mean[j]) / x_std[j]: Re Σ(ω_j), Im Σ(ω_j), T, μ, scale, ε_i - μ.
__global__ void features_kernel(const double2* __restrict__ S, int nw, int ni, const double* __restrict__ eps_i, double T,
                                double mu, double scale, const float* __restrict__ xm, const float* __restrict__ xs,
                                float* __restrict__ X) {
  const int d0 = 2 * nw + 4;
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (j >= d0) return;
  double v;
  if (j < nw)
    v = S[long(i) * nw + j].x;
  else if (j < 2 * nw)
    v = S[long(i) * nw + j - nw].y;
  else if (j == 2 * nw)
    v = T;
  else if (j == 2 * nw + 1)
    v = mu;
  else if (j == 2 * nw + 2)
    v = scale;
  else
    v = eps_i[i] - mu;
  X[long(i) * d0 + j] = (float(v) - xm[j]) / xs[j];
}

// Σ(ω_j, i) += (Y[i][j] y_scale + y_mean[j]) + i (Y[i][nω + j] y_scale + y_mean[nω + j]).
__global__ void correct_kernel(double2* __restrict__ S, int nw, const float* __restrict__ Y, float ys,
                               const float* __restrict__ ym) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (j >= nw) return;
  const float* y = Y + long(i) * 2 * nw;
  double2 v = S[long(i) * nw + j];
  v.x += double(y[j] * ys + ym[j]);
  v.y += double(y[nw + j] * ys + ym[nw + j]);
  S[long(i) * nw + j] = v;
}

// An operand of ns = 3 parts (three consecutive [rows][ld] BF16 blocks) or, for the weights, of one; boxes of
// box_rows rows.
static TcOperand operand_parts(const __nv_bfloat16* parts, int ns, long rows, long cols, long ld, int box_rows) {
  TcOperand op;
  op.ns = ns;
  for (int p = 0; p < ns; ++p) {
    const __nv_bfloat16* base = parts + long(p) * rows * ld;
    op.m[p] = make_tmap_bf16(base, rows, cols, ld, box_rows);
    op.base[p] = base;
  }
  op.rows = rows;
  op.cols = cols;
  op.ld = ld;
  return op;
}

// The BF16 weight rows of the products and their operands (fixed sizes; built once per network).
static void train_weights_init(Mlp* P) {
  Mlp::Train& T = P->tr;
  const int L = P->L;
  T.dp.resize(size_t(L + 1));
  for (int l = 0; l <= L; ++l) T.dp[size_t(l)] = (P->dims[size_t(l)] + 7) / 8 * 8;
  T.Wp.resize(size_t(L));
  T.WT.resize(size_t(L));
  for (int l = 0; l < L; ++l) {
    const long din = P->dims[size_t(l)], dout = P->dims[size_t(l + 1)];
    T.Wp[size_t(l)].alloc(P->ctx, size_t(dout * T.dp[size_t(l)]));
    T.WT[size_t(l)].alloc(P->ctx, size_t(din * T.dp[size_t(l + 1)]));
    T.Wp[size_t(l)].zero(P->ctx->stream);  // the padding columns stay zero
    T.WT[size_t(l)].zero(P->ctx->stream);
  }
  T.opW.resize(size_t(L));
  T.opWT.resize(size_t(L));
  for (int l = 0; l < L; ++l) {
    const long din = P->dims[size_t(l)], dout = P->dims[size_t(l + 1)];
    T.opW[size_t(l)] = operand_parts(T.Wp[size_t(l)].p, 1, dout, din, T.dp[size_t(l)], kTcBM);
    T.opWT[size_t(l)] = operand_parts(T.WT[size_t(l)].p, 1, din, dout, T.dp[size_t(l + 1)], kTcBM);
  }
}

static void ensure_cap(Mlp* P, long n) {
  if (n <= P->cap) return;
  Ctx* ctx = P->ctx;
  const int L = P->L;
  int dmax = 0;
  for (int d : P->dims) dmax = std::max(dmax, d);
  P->Z.resize(size_t(L));
  P->X.resize(size_t(L + 1));
  for (int l = 0; l <= L; ++l) P->X[size_t(l)].alloc(ctx, size_t(n) * size_t(P->dims[size_t(l)]));
  for (int l = 0; l < L; ++l) P->Z[size_t(l)].alloc(ctx, size_t(n) * size_t(P->dims[size_t(l + 1)]));
  P->dA.alloc(ctx, size_t(n) * size_t(dmax));
  P->dB.alloc(ctx, size_t(n) * size_t(dmax));
  P->loss_rows.alloc(ctx, size_t(n));
  P->Yb.alloc(ctx, size_t(n) * size_t(P->dims.back()));
  // the tensor-core operands of the activations and gradients, and the products' split-K slabs:
  // a product of t tiles takes at most ceil(SMs / t) splits, so splits x M x N stays below
  // (SMs + t) tiles of 128 x 128
  Mlp::Train& T = P->tr;
  T.cap = n;
  T.ldT = (n + 7) / 8 * 8;
  for (auto* v : {&T.Xs, &T.XT, &T.dZs, &T.dZT}) v->resize(size_t(L));
  for (auto* v : {&T.dz, &T.slab}) v->resize(size_t(L));
  for (auto* v : {&T.opXs, &T.opXT, &T.opdZs, &T.opdZT}) v->resize(size_t(L));
  const long sm = ctx->sm_count;
  auto tiles = [](long M, long N) { return ((M + 127) / 128) * ((N + 127) / 128); };
  long part = 0;
  for (int l = 0; l < L; ++l) {
    const long din = P->dims[size_t(l)], dout = P->dims[size_t(l + 1)];
    const long dpi = T.dp[size_t(l)], dpo = T.dp[size_t(l + 1)];
    T.Xs[size_t(l)].alloc(ctx, size_t(3 * n * dpi));
    T.XT[size_t(l)].alloc(ctx, size_t(3 * din * T.ldT));
    T.dZs[size_t(l)].alloc(ctx, size_t(3 * n * dpo));
    T.dZT[size_t(l)].alloc(ctx, size_t(3 * dout * T.ldT));
    T.opXs[size_t(l)] = operand_parts(T.Xs[size_t(l)].p, 3, n, din, dpi, 128);
    T.opXT[size_t(l)] = operand_parts(T.XT[size_t(l)].p, 3, din, T.ldT, T.ldT, kTcBM);
    T.opdZs[size_t(l)] = operand_parts(T.dZs[size_t(l)].p, 3, n, dout, dpo, 128);
    T.opdZT[size_t(l)] = operand_parts(T.dZT[size_t(l)].p, 3, dout, T.ldT, T.ldT, 128);
    T.dz[size_t(l)].alloc(ctx, size_t(n * dout));
    const long tw = tiles(din, dout);
    T.slab[size_t(l)].alloc(ctx, size_t(std::min<long>(16, (sm + tw - 1) / tw) * din * dout));
    for (const long t : {tiles(dout, n), tiles(din, dout), tiles(din, n)}) part = std::max(part, (sm + t) * 128 * 128);
  }
  T.part.alloc(ctx, size_t(part));
  P->cap = n;
}

// One three-part product into the split-K slabs `out` (T.part by default; out[s][m + ld_out n]); returns the splits.
static int mlp_product(Mlp* P, const TcOperand& A, const TcOperand& B, int M, int N, int K, long ld_out,
                       DBuf<float>* out = nullptr) {
  if (!out) out = &P->tr.part;
  int bn = 0, sp = 0;
  tc_gemm_shape(P->ctx, M, N, K, 16, 3, &bn, &sp);
  if (bn != 128) fail(EPSP_EINVAL, "three-part products run with tiles of 128 columns");
  if (size_t(sp) * size_t(M) * size_t(N) > out->n) fail(EPSP_EINVAL, "split-K slabs exceed their buffer");
  return tc_gemm_launch(P->ctx, A, B, M, N, K, out->p, ld_out, long(M) * N, 16, P->d_err.p, "mlp");
}

static dim3 emit_grid(long cols, long rows) { return dim3(unsigned((cols + 31) / 32), unsigned((rows + 31) / 32)); }

// Forward over the n rows in P->X[0] on the tensor cores; output in P->X[L]. With `train` the
// transposed activations (the gradient products' operands) and the pre-activations Z are kept.
static void forward_train(Mlp* P, long n, bool train) {
  Ctx* ctx = P->ctx;
  cudaStream_t s = ctx->stream;
  Mlp::Train& T = P->tr;
  const dim3 blk(32, 8);
  const int d0 = P->dims[0];
  emit_kernel<kEmitCopy><<<emit_grid(d0, train ? T.ldT : n), blk, 0, s>>>(
      int(n), d0, P->X[0].p, d0, nullptr, 0, 0, nullptr, false, nullptr, nullptr, nullptr, T.Xs[0].p, T.dp[0],
      long(T.cap) * T.dp[0], train ? T.XT[0].p : nullptr, T.ldT, long(d0) * T.ldT);
  EPSP_LAUNCHED(ctx);
  for (int l = 0; l < P->L; ++l) {
    const int din = P->dims[size_t(l)], dout = P->dims[size_t(l + 1)];
    const bool last = l + 1 == P->L;
    const int sp = mlp_product(P, T.opW[size_t(l)], T.opXs[size_t(l)], dout, int(n), din, dout);
    const bool tpose = train && !last;
    emit_kernel<kEmitBiasAct><<<emit_grid(dout, tpose ? T.ldT : n), blk, 0, s>>>(
        int(n), dout, nullptr, 0, T.part.p, sp, long(dout) * n, P->b[size_t(l)].p, !last, nullptr,
        (train && !last) ? P->Z[size_t(l)].p : nullptr, last ? P->X[size_t(P->L)].p : nullptr,
        last ? nullptr : T.Xs[size_t(l + 1)].p, last ? 0 : T.dp[size_t(l + 1)], last ? 0 : long(T.cap) * T.dp[size_t(l + 1)],
        tpose ? T.XT[size_t(l + 1)].p : nullptr, T.ldT, long(dout) * T.ldT);
    EPSP_LAUNCHED(ctx);
  }
}

// Gradients of the mean squared error of the batch in P->X[0], P->Yb (n rows, normalised by
// n_total rows) into gW, gb; the batch's sum of squared errors goes to P->loss_sum[slot]. Needs the
// forward with `train`.
static void backward(Mlp* P, long n, long n_total, int slot) {
  Ctx* ctx = P->ctx;
  cudaStream_t s = ctx->stream;
  Mlp::Train& T = P->tr;
  const dim3 blk(32, 8);
  const int L = P->L, dl = P->dims.back();
  mse_kernel<<<unsigned(n), 256, 0, s>>>(P->X[size_t(L)].p, P->Yb.p, dl, 2.f / (float(n_total) * float(dl)), P->dA.p,
                                         P->loss_rows.p);
  EPSP_LAUNCHED(ctx);
  sum_kernel<<<1, 256, 0, s>>>(P->loss_rows.p, n, P->loss_sum.p, slot);
  EPSP_LAUNCHED(ctx);
  // dZ of the last layer (linear output) as the products' operands
  emit_kernel<kEmitCopy><<<emit_grid(dl, T.ldT), blk, 0, s>>>(
      int(n), dl, P->dA.p, dl, nullptr, 0, 0, nullptr, false, nullptr, nullptr, nullptr, T.dZs[size_t(L - 1)].p,
      T.dp[size_t(L)], long(T.cap) * T.dp[size_t(L)], T.dZT[size_t(L - 1)].p, T.ldT, long(dl) * T.ldT);
  EPSP_LAUNCHED(ctx);
  float* dZ = P->dA.p;  // FP32 dZ of layer l, [n][d_{l+1}]
  float* other = P->dB.p;
  for (int l = L - 1; l >= 0; --l) {
    const int din = P->dims[size_t(l)], dout = P->dims[size_t(l + 1)];
    // gW[o][i] = Σ_m dZ[m][o] X[m][i]: the product's slab element (i, o) at i + din o
    const int sg = mlp_product(P, T.opXT[size_t(l)], T.opdZT[size_t(l)], din, dout, int(n), din);
    partial_sum_kernel<<<div_up(size_t(dout) * size_t(din), 256), 256, 0, s>>>(T.part.p, dout, din, sg,
                                                                               P->gW[size_t(l)].p, din, 1);
    EPSP_LAUNCHED(ctx);
    bias_grad_kernel<<<div_up(size_t(dout), 128), 128, 0, s>>>(dZ, n, dout, P->gb[size_t(l)].p);
    EPSP_LAUNCHED(ctx);
    if (l > 0) {
      // dX[m][i] = Σ_o dZ[m][o] W[o][i] (slab element (i, m) at i + din m), through SiLU of layer l - 1
      const int sx = mlp_product(P, T.opWT[size_t(l)], T.opdZs[size_t(l)], din, int(n), dout, din);
      emit_kernel<kEmitActBack><<<emit_grid(din, T.ldT), blk, 0, s>>>(
          int(n), din, nullptr, 0, T.part.p, sx, long(din) * n, nullptr, false, P->Z[size_t(l - 1)].p, nullptr, other,
          T.dZs[size_t(l - 1)].p, T.dp[size_t(l)], long(T.cap) * T.dp[size_t(l)], T.dZT[size_t(l - 1)].p, T.ldT,
          long(din) * T.ldT);
      EPSP_LAUNCHED(ctx);
      std::swap(dZ, other);
    }
  }
}

// Reports (and clears) a bounded wait that ran out in the network's tensor-core products.
static void check_mlp_err(Mlp* P) {
  int e = 0;
  P->d_err.download(&e, 1, P->ctx->stream);
  EPSP_CUDA(cudaStreamSynchronize(P->ctx->stream));
  if (e) {
    P->d_err.zero(P->ctx->stream);
    fail(EPSP_EDEVICE_TIMEOUT, "a tensor-core GEMM wait ran out in the warm-start network (bounded device wait)");
  }
}

// ---- tensor-core inference (the scGD0 hook on the tensor-core path) ----

// out[r][c] = in[r][c] for c < cols, 0 for cols <= c < ldo (BF16 rows padded to 16 bytes).
__global__ void pad_rows_bf16_kernel(const __nv_bfloat16* __restrict__ in, long rows, int cols, int ldo,
                                     __nv_bfloat16* __restrict__ out) {
  const long k = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= rows * ldo) return;
  const long r = k / ldo;
  const int c = int(k % ldo);
  out[k] = c < cols ? in[r * cols + c] : __float2bfloat16_rn(0.f);
}

// A operand of the first product: X [n][d] FP32 rows split into BF16 hi/lo rows of ldo.
__global__ void split_rows_mlp_kernel(const float* __restrict__ X, int n, int d, int ldo, __nv_bfloat16* __restrict__ oh,
                                      __nv_bfloat16* __restrict__ ol) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (j >= d || i >= n) return;
  const float x = X[long(i) * d + j];
  const __nv_bfloat16 h = __float2bfloat16_rn(x);
  oh[long(i) * ldo + j] = h;
  ol[long(i) * ldo + j] = __float2bfloat16_rn(x - __bfloat162float(h));
}

// z = Σ_s part[s][m + n j] + b[j] (the product's column-major FP32 splits, in order); SiLU when act;
// into the next product's A operand (BF16 hi/lo rows of ldo) or, for the last layer, X [n][dout].
__global__ void bias_act_split_kernel(const float* __restrict__ part, int splits, long stride, int n, int dout,
                                      const float* __restrict__ b, bool act, __nv_bfloat16* __restrict__ oh,
                                      __nv_bfloat16* __restrict__ ol, int ldo, float* __restrict__ X) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
  if (m >= n) return;
  float z = 0.f;
  for (int p = 0; p < splits; ++p) z += part[stride * p + m + long(n) * j];
  z += b[j];
  const float x = act ? z * sigmoidf_(z) : z;
  if (oh) {
    const __nv_bfloat16 h = __float2bfloat16_rn(x);
    oh[long(m) * ldo + j] = h;
    ol[long(m) * ldo + j] = __float2bfloat16_rn(x - __bfloat162float(h));
  } else {
    X[long(m) * dout + j] = x;
  }
}

static void infer_reserve(Mlp* P, long n) {
  Mlp::Infer& I = P->inf;
  Ctx* ctx = P->ctx;
  cudaStream_t s = ctx->stream;
  const bool grow = n > I.cap;
  if (I.wgen == P->wgen && !grow) return;
  const int L = P->L;
  if (I.dpad.empty()) {
    I.dpad.resize(size_t(L));
    I.bn.resize(size_t(L));
    I.Wh.resize(size_t(L));
    I.Wl.resize(size_t(L));
    I.Ah.resize(size_t(L));
    I.Al.resize(size_t(L));
    I.opA.resize(size_t(L));
    I.opB.resize(size_t(L));
    for (int l = 0; l < L; ++l) {
      const int din = P->dims[size_t(l)], dout = P->dims[size_t(l + 1)];
      I.dpad[size_t(l)] = (din + 7) / 8 * 8;
      int bn, sp;
      tc_gemm_shape(ctx, 1, dout, din, 16, 2, &bn, &sp);  // the tile width depends on N only
      I.bn[size_t(l)] = bn;
      I.Wh[size_t(l)].alloc(ctx, size_t(dout) * size_t(I.dpad[size_t(l)]));
      I.Wl[size_t(l)].alloc(ctx, size_t(dout) * size_t(I.dpad[size_t(l)]));
      I.Wl[size_t(l)].zero(s);  // the weights are exact in BF16: no low part
      I.opB[size_t(l)].ns = 2;
      I.opB[size_t(l)].m[0] = make_tmap_bf16(I.Wh[size_t(l)].p, dout, din, I.dpad[size_t(l)], bn);
      I.opB[size_t(l)].m[1] = make_tmap_bf16(I.Wl[size_t(l)].p, dout, din, I.dpad[size_t(l)], bn);
    }
  }
  if (I.wgen != P->wgen) {
    for (int l = 0; l < L; ++l) {
      const int din = P->dims[size_t(l)], dout = P->dims[size_t(l + 1)], dp = I.dpad[size_t(l)];
      pad_rows_bf16_kernel<<<div_up(size_t(dout) * size_t(dp), 256), 256, 0, s>>>(P->Wbf[size_t(l)].p, dout, din, dp,
                                                                                 I.Wh[size_t(l)].p);
      EPSP_LAUNCHED(ctx);
    }
    I.wgen = P->wgen;
  }
  if (grow) {
    size_t part = 0;
    for (int l = 0; l < L; ++l) {
      const int din = P->dims[size_t(l)], dout = P->dims[size_t(l + 1)], dp = I.dpad[size_t(l)];
      I.Ah[size_t(l)].alloc(ctx, size_t(n) * size_t(dp));
      I.Al[size_t(l)].alloc(ctx, size_t(n) * size_t(dp));
      I.Ah[size_t(l)].zero(s);  // the padding columns stay zero
      I.Al[size_t(l)].zero(s);
      I.opA[size_t(l)].ns = 2;
      I.opA[size_t(l)].m[0] = make_tmap_bf16(I.Ah[size_t(l)].p, n, din, dp, kTcBM);
      I.opA[size_t(l)].m[1] = make_tmap_bf16(I.Al[size_t(l)].p, n, din, dp, kTcBM);
      int bn, sp;
      tc_gemm_shape(ctx, int(n), dout, dp, 16, 2, &bn, &sp);
      part = std::max(part, size_t(sp) * size_t(n) * size_t(dout));
    }
    I.part.alloc(ctx, part);
    I.cap = n;
  }
}

// Forward over the rows in P->X[0] (n rows) on the tensor cores: each product A x W^T with A the
// FP32 activations as BF16 hi + lo (three products, the weights' lo part is zero: FP32-accurate
// activations times the BF16 weights, as the SIMT forward), FP32 accumulation; output in P->X[L].
// Bounded waits report to d_err.
static void forward_tc(Mlp* P, long n, int* d_err) {
  Ctx* ctx = P->ctx;
  cudaStream_t s = ctx->stream;
  infer_reserve(P, n);
  Mlp::Infer& I = P->inf;
  const int d0 = P->dims[0];
  split_rows_mlp_kernel<<<dim3(div_up(size_t(d0), 256), unsigned(n)), 256, 0, s>>>(P->X[0].p, int(n), d0, I.dpad[0],
                                                                                 I.Ah[0].p, I.Al[0].p);
  EPSP_LAUNCHED(ctx);
  for (int l = 0; l < P->L; ++l) {
    const int dout = P->dims[size_t(l + 1)], dp = I.dpad[size_t(l)];
    const int sp = tc_gemm_launch(ctx, I.opA[size_t(l)], I.opB[size_t(l)], int(n), dout, dp, I.part.p, n, n * long(dout),
                                  16, d_err, "mlp");
    const bool last = l + 1 == P->L;
    bias_act_split_kernel<<<dim3(div_up(size_t(n), 128), unsigned(dout)), 128, 0, s>>>(
        I.part.p, sp, n * long(dout), int(n), dout, P->b[size_t(l)].p, !last, last ? nullptr : I.Ah[size_t(l + 1)].p,
        last ? nullptr : I.Al[size_t(l + 1)].p, last ? 0 : I.dpad[size_t(l + 1)], P->X[size_t(P->L)].p);
    EPSP_LAUNCHED(ctx);
  }
}

// One training step on the minibatch of n rows at the cursor (B; the data set's inputs dataX): forward, backward, Adam.
// The gradient products, the losses and the biases run on the side stream beside the backward chain, of which each
// layer is one product and one epilogue: for four layers 17 launches in a row and 6 beside them, where the step was 41
// in a row. Bound by the latency of those 17 (256 rows are 16 to 152 tiles of work). Measured with widths 2506, 256, 256,
// 256, 2502: 238 -> 145 us a step of 256 rows, bitwise the same parameters.
static void train_step(Mlp* P, long n, const Batch& B, float lr) {
  Ctx* ctx = P->ctx;
  cudaStream_t s = ctx->stream;
  Mlp::Train& T = P->tr;
  auto& sd = T.side;
  if (!sd.s) {
    EPSP_CUDA(cudaStreamCreateWithFlags(&sd.s, cudaStreamNonBlocking));
    EPSP_CUDA(cudaEventCreateWithFlags(&sd.fork, cudaEventDisableTiming));
    EPSP_CUDA(cudaEventCreateWithFlags(&sd.join, cudaEventDisableTiming));
  }
  struct OnSide {  // launches through ctx go to the side stream while it lives, after what the main stream holds
    Ctx* c;
    cudaStream_t main;
    OnSide(Ctx* c_, Mlp::Train::Side& d) : c(c_), main(c_->stream) {
      EPSP_CUDA(cudaEventRecord(d.fork, main));
      EPSP_CUDA(cudaStreamWaitEvent(d.s, d.fork, 0));
      c->stream = d.s;
    }
    ~OnSide() { c->stream = main; }
  };
  const dim3 blk(32, 8);
  const int L = P->L, d0 = P->dims[0], dl = P->dims.back();
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  emit_kernel<kEmitGather><<<emit_grid(d0, T.ldT), blk, 0, s>>>(
      int(n), d0, P->dataX.p, d0, nullptr, 0, 0, nullptr, false, nullptr, nullptr, nullptr, T.Xs[0].p, T.dp[0],
      long(T.cap) * T.dp[0], T.XT[0].p, T.ldT, long(d0) * T.ldT, B);
  EPSP_LAUNCHED(ctx);
  for (int l = 0; l < L; ++l) {
    const int din = P->dims[size_t(l)], dout = P->dims[size_t(l + 1)];
    const int sp = mlp_product(P, T.opW[size_t(l)], T.opXs[size_t(l)], dout, int(n), din, dout);
    if (l + 1 < L)
      emit_kernel<kEmitBiasAct><<<emit_grid(dout, T.ldT), blk, 0, s>>>(
          int(n), dout, nullptr, 0, T.part.p, sp, long(dout) * n, P->b[size_t(l)].p, true, nullptr, P->Z[size_t(l)].p,
          nullptr, T.Xs[size_t(l + 1)].p, T.dp[size_t(l + 1)], long(T.cap) * T.dp[size_t(l + 1)], T.XT[size_t(l + 1)].p,
          T.ldT, long(dout) * T.ldT);
    else  // the output and dZ of the last layer
      emit_kernel<kEmitLoss><<<emit_grid(dout, T.ldT), blk, 0, s>>>(
          int(n), dout, nullptr, 0, T.part.p, sp, long(dout) * n, P->b[size_t(l)].p, false, nullptr, P->X[size_t(L)].p,
          T.dz[size_t(l)].p, T.dZs[size_t(l)].p, T.dp[size_t(L)], long(T.cap) * T.dp[size_t(L)], T.dZT[size_t(l)].p, T.ldT,
          long(dl) * T.ldT, B);
    EPSP_LAUNCHED(ctx);
  }
  AdamAll aw{};
  BiasAll ab{};
  aw.L = ab.L = L;
  aw.lr = ab.lr = lr;
  aw.b1 = ab.b1 = b1;
  aw.b2 = ab.b2 = b2;
  aw.eps = ab.eps = eps;
  aw.t = ab.t = P->d_step.p;
  ab.n = n;
  // gW[o][i] = Σ_m dZ[m][o] X[m][i]: the product's slab element (i, o) at i + din o
  auto weight_gradient = [&](int l) {
    const int din = P->dims[size_t(l)], dout = P->dims[size_t(l + 1)];
    aw.l[l].splits = mlp_product(P, T.opXT[size_t(l)], T.opdZT[size_t(l)], din, dout, int(n), din, &T.slab[size_t(l)]);
  };
  {
    OnSide on(ctx, sd);
    row_loss_kernel<<<unsigned(n), 256, 0, sd.s>>>(P->X[size_t(L)].p, dl, B, P->loss_rows.p);
    EPSP_LAUNCHED(ctx);
    loss_step_kernel<<<1, 256, 0, sd.s>>>(P->loss_rows.p, n, P->loss_sum.p, P->d_step.p + 1, P->d_step.p);
    EPSP_LAUNCHED(ctx);
    if (L > 1) weight_gradient(L - 1);
  }
  for (int l = L - 1; l >= 1; --l) {
    // dX[m][i] = Σ_o dZ[m][o] W[o][i] (slab element (i, m) at i + din m), through SiLU of layer l - 1
    const int din = P->dims[size_t(l)], dout = P->dims[size_t(l + 1)];
    const int sx = mlp_product(P, T.opWT[size_t(l)], T.opdZs[size_t(l)], din, int(n), dout, din);
    emit_kernel<kEmitActBack><<<emit_grid(din, T.ldT), blk, 0, s>>>(
        int(n), din, nullptr, 0, T.part.p, sx, long(din) * n, nullptr, false, P->Z[size_t(l - 1)].p, nullptr,
        T.dz[size_t(l - 1)].p, T.dZs[size_t(l - 1)].p, T.dp[size_t(l)], long(T.cap) * T.dp[size_t(l)],
        T.dZT[size_t(l - 1)].p, T.ldT, long(din) * T.ldT);
    EPSP_LAUNCHED(ctx);
    if (l > 1) {
      OnSide on(ctx, sd);
      weight_gradient(l - 1);
    }
  }
  {
    OnSide on(ctx, sd);
    for (int l = 0, c = 0; l < L; c += P->dims[size_t(++l)])
      ab.l[l] = BiasLayer{T.dz[size_t(l)].p, P->b[size_t(l)].p, P->mb[size_t(l)].p, P->vb[size_t(l)].p, P->dims[size_t(l + 1)],
                          c};
    ab.cols = ab.l[L - 1].col0 + dl;
    adam_bias_kernel<<<div_up(size_t(ab.cols), 32), 32, 0, sd.s>>>(ab);
    EPSP_LAUNCHED(ctx);
    EPSP_CUDA(cudaEventRecord(sd.join, sd.s));
  }
  weight_gradient(0);
  EPSP_CUDA(cudaStreamWaitEvent(s, sd.join, 0));
  int tiles = 0;
  for (int l = 0; l < L; ++l) {
    const int din = P->dims[size_t(l)], dout = P->dims[size_t(l + 1)];
    aw.l[l] = AdamLayer{P->W[size_t(l)].p, P->mW[size_t(l)].p, P->vW[size_t(l)].p, T.slab[size_t(l)].p, long(din) * dout,
                        T.dp[size_t(l)], T.dp[size_t(l + 1)], P->Wbf[size_t(l)].p, T.Wp[size_t(l)].p, T.WT[size_t(l)].p,
                        aw.l[l].splits, din, dout, tiles};
    tiles += ((din + 31) / 32) * ((dout + 31) / 32);
  }
  adam_weights_kernel<<<unsigned(tiles), 256, 0, s>>>(aw);
  EPSP_LAUNCHED(ctx);
}

static long nparams(const Mlp* P) {
  long t = 0;
  for (int l = 0; l < P->L; ++l) t += long(P->dims[size_t(l)]) * P->dims[size_t(l + 1)] + P->dims[size_t(l + 1)];
  return t;
}

}  // namespace epsp

using namespace epsp;

struct epsp_warmstart {
  Mlp m;
};

namespace epsp {

void warmstart_correct(epsp_warmstart* w, Ctx* ctx, double2* S_T, long nw, long ni, const double* d_eps_i, double T,
                       double mu, double scale, int* tc_err) {
  Mlp& P = w->m;
  if (P.ctx != ctx) fail(EPSP_EINVAL, "the warm-start network belongs to another context");
  if (P.dims[0] != 2 * nw + 4 || P.dims.back() != 2 * nw)
    fail(EPSP_EINVAL, "the warm-start network's widths do not match 2 nω + 4 inputs and 2 nω outputs (nω = " +
                          std::to_string(nw) + ")");
  if (!P.scaled) fail(EPSP_EINVAL, "the warm-start network has no feature scaling (epsp_warmstart_set_scaling)");
  cudaStream_t s = ctx->stream;
  ensure_cap(&P, ni);
  features_kernel<<<dim3(div_up(size_t(2 * nw + 4), 256), unsigned(ni)), 256, 0, s>>>(
      S_T, int(nw), int(ni), d_eps_i, T, mu, scale, P.x_mean.p, P.x_std.p, P.X[0].p);
  EPSP_LAUNCHED(ctx);
  if (tc_err) {
    forward_tc(&P, ni, tc_err);
  } else {
    forward_train(&P, ni, false);
    check_mlp_err(&P);
  }
  correct_kernel<<<dim3(div_up(size_t(nw), 256), unsigned(ni)), 256, 0, s>>>(S_T, int(nw), P.X[size_t(P.L)].p, P.y_scale,
                                                                            P.y_mean.p);
  EPSP_LAUNCHED(ctx);
}

}  // namespace epsp

template <class F>
static epsp_status wguard(Ctx* c, F&& f) {
  try {
    EPSP_CUDA(cudaSetDevice(c->device));
    f();
    c->last_error.clear();
    return EPSP_OK;
  } catch (const Error& e) {
    c->last_error = e.msg;
    return epsp_status(e.code);
  } catch (const std::bad_alloc&) {
    c->last_error = "host allocation failed";
    return EPSP_ENOMEM;
  }
}

extern "C" {

epsp_status epsp_warmstart_create(epsp_ctx* ctx, int32_t nlayers, const int32_t* dims, epsp_warmstart** out) {
  if (!ctx || !out || !dims || nlayers < 1 || nlayers > 16) return EPSP_EINVAL;
  *out = nullptr;
  return wguard(&ctx->c, [&] {
    for (int l = 0; l <= nlayers; ++l)
      if (dims[l] < 1 || dims[l] > (1 << 20)) fail(EPSP_EINVAL, "layer widths must be in [1, 2^20]");
    auto* w = new epsp_warmstart;
    std::unique_ptr<epsp_warmstart> guard(w);
    Mlp& P = w->m;
    P.ctx = &ctx->c;
    P.L = nlayers;
    P.dims.assign(dims, dims + nlayers + 1);
    P.W.resize(size_t(nlayers));
    P.b.resize(size_t(nlayers));
    P.gW.resize(size_t(nlayers));
    P.gb.resize(size_t(nlayers));
    P.mW.resize(size_t(nlayers));
    P.vW.resize(size_t(nlayers));
    P.mb.resize(size_t(nlayers));
    P.vb.resize(size_t(nlayers));
    P.Wbf.resize(size_t(nlayers));
    for (int l = 0; l < nlayers; ++l) {
      const size_t nw = size_t(dims[l]) * size_t(dims[l + 1]), nb = size_t(dims[l + 1]);
      for (auto* v : {&P.W[size_t(l)], &P.gW[size_t(l)], &P.mW[size_t(l)], &P.vW[size_t(l)]}) v->alloc(P.ctx, nw);
      for (auto* v : {&P.b[size_t(l)], &P.gb[size_t(l)], &P.mb[size_t(l)], &P.vb[size_t(l)]}) v->alloc(P.ctx, nb);
      P.Wbf[size_t(l)].alloc(P.ctx, nw);
      for (auto* v : {&P.W[size_t(l)], &P.mW[size_t(l)], &P.vW[size_t(l)], &P.b[size_t(l)], &P.mb[size_t(l)], &P.vb[size_t(l)]})
        v->zero(P.ctx->stream);
    }
    P.loss_sum.alloc(P.ctx, 1);
    P.d_step.alloc(P.ctx, 2);
    P.d_step.zero(P.ctx->stream);
    P.d_err.alloc(P.ctx, 1);
    P.d_err.zero(P.ctx->stream);
    train_weights_init(&P);
    EPSP_CUDA(cudaStreamSynchronize(P.ctx->stream));
    *out = guard.release();
  });
}

void epsp_warmstart_destroy(epsp_warmstart* w) {
  if (!w) return;
  cudaSetDevice(w->m.ctx->device);
  delete w;
}

int64_t epsp_warmstart_nparams(const epsp_warmstart* w) { return w ? nparams(&w->m) : 0; }

/* Device milliseconds of the epochs of the last epsp_warmstart_train (CUDA events around each
 * epoch's graph replays; the uploads and the capture are not included). */
double epsp_warmstart_train_ms(const epsp_warmstart* w) { return w ? w->m.train_ms : 0.0; }

/* Parameters as one flat FP32 vector: for each layer, W [d_{l+1}][d_l] then b [d_{l+1}]. Setting
 * them resets the optimiser state. */
epsp_status epsp_warmstart_set_params(epsp_warmstart* w, const float* params) {
  if (!w || !params) return EPSP_EINVAL;
  Mlp& P = w->m;
  return wguard(P.ctx, [&] {
    cudaStream_t s = P.ctx->stream;
    long off = 0;
    for (int l = 0; l < P.L; ++l) {
      const long nw = long(P.dims[size_t(l)]) * P.dims[size_t(l + 1)], nb = P.dims[size_t(l + 1)];
      P.W[size_t(l)].upload(params + off, size_t(nw), s);
      off += nw;
      P.b[size_t(l)].upload(params + off, size_t(nb), s);
      off += nb;
      to_bf16_kernel<<<div_up(size_t(nw), 256), 256, 0, s>>>(P.W[size_t(l)].p, nw, P.dims[size_t(l)], P.Wbf[size_t(l)].p,
                                                             P.tr.Wp[size_t(l)].p, P.tr.dp[size_t(l)],
                                                             P.tr.WT[size_t(l)].p, P.tr.dp[size_t(l + 1)]);
      EPSP_LAUNCHED(P.ctx);
      P.mW[size_t(l)].zero(s);
      P.vW[size_t(l)].zero(s);
      P.mb[size_t(l)].zero(s);
      P.vb[size_t(l)].zero(s);
    }
    P.d_step.zero(s);
    ++P.wgen;
    EPSP_CUDA(cudaStreamSynchronize(s));
  });
}

epsp_status epsp_warmstart_get_params(epsp_warmstart* w, float* params) {
  if (!w || !params) return EPSP_EINVAL;
  Mlp& P = w->m;
  return wguard(P.ctx, [&] {
    cudaStream_t s = P.ctx->stream;
    long off = 0;
    for (int l = 0; l < P.L; ++l) {
      const long nw = long(P.dims[size_t(l)]) * P.dims[size_t(l + 1)], nb = P.dims[size_t(l + 1)];
      P.W[size_t(l)].download(params + off, size_t(nw), s);
      off += nw;
      P.b[size_t(l)].download(params + off, size_t(nb), s);
      off += nb;
    }
    EPSP_CUDA(cudaStreamSynchronize(s));
  });
}

/* Standardisation used when the network corrects Σ inside the scGD0 iteration: inputs
 * (x - x_mean) / x_std, outputs y * y_scale + y_mean. */
epsp_status epsp_warmstart_set_scaling(epsp_warmstart* w, const float* x_mean, const float* x_std, const float* y_mean,
                                       float y_scale) {
  if (!w || !x_mean || !x_std || !y_mean || !(y_scale > 0.f) || !std::isfinite(y_scale)) return EPSP_EINVAL;
  Mlp& P = w->m;
  return wguard(P.ctx, [&] {
    const int d0 = P.dims[0], dl = P.dims.back();
    for (int j = 0; j < d0; ++j)
      if (!(x_std[j] > 0.f) || !std::isfinite(x_std[j]) || !std::isfinite(x_mean[j]))
        fail(EPSP_EINVAL, "x_std must be positive and x_mean finite");
    for (int j = 0; j < dl; ++j)
      if (!std::isfinite(y_mean[j])) fail(EPSP_EINVAL, "y_mean must be finite");
    cudaStream_t s = P.ctx->stream;
    P.x_mean.alloc(P.ctx, size_t(d0));
    P.x_std.alloc(P.ctx, size_t(d0));
    P.y_mean.alloc(P.ctx, size_t(dl));
    P.x_mean.upload(x_mean, size_t(d0), s);
    P.x_std.upload(x_std, size_t(d0), s);
    P.y_mean.upload(y_mean, size_t(dl), s);
    P.y_scale = y_scale;
    P.scaled = true;
    EPSP_CUDA(cudaStreamSynchronize(s));
  });
}

/* Inference: Y [n][d_L] from X [n][d_0] (host arrays, row-major). */
epsp_status epsp_warmstart_predict(epsp_warmstart* w, const float* X, int64_t n, float* Y) {
  if (!w || !X || !Y || n < 1) return EPSP_EINVAL;
  Mlp& P = w->m;
  return wguard(P.ctx, [&] {
    cudaStream_t s = P.ctx->stream;
    const long chunk = 8192;
    ensure_cap(&P, std::min<long>(n, chunk));
    for (long r0 = 0; r0 < n; r0 += chunk) {
      const long nb = std::min(chunk, n - r0);
      P.X[0].upload(X + r0 * P.dims[0], size_t(nb * P.dims[0]), s);
      forward_train(&P, nb, false);
      P.X[size_t(P.L)].download(Y + r0 * P.dims.back(), size_t(nb * P.dims.back()), s);
    }
    check_mlp_err(&P);
  });
}

/* Loss (mean squared error) and its gradient with respect to every parameter (flat, as
 * epsp_warmstart_set_params) for the batch (X [n][d_0], Y [n][d_L]); no parameter update. */
epsp_status epsp_warmstart_grad(epsp_warmstart* w, const float* X, const float* Y, int64_t n, double* loss, float* grad) {
  if (!w || !X || !Y || n < 1 || !grad) return EPSP_EINVAL;
  Mlp& P = w->m;
  return wguard(P.ctx, [&] {
    cudaStream_t s = P.ctx->stream;
    ensure_cap(&P, n);
    P.X[0].upload(X, size_t(n * P.dims[0]), s);
    P.Yb.upload(Y, size_t(n * P.dims.back()), s);
    forward_train(&P, n, true);
    backward(&P, n, n, 0);
    long off = 0;
    for (int l = 0; l < P.L; ++l) {
      const long nw = long(P.dims[size_t(l)]) * P.dims[size_t(l + 1)], nb = P.dims[size_t(l + 1)];
      P.gW[size_t(l)].download(grad + off, size_t(nw), s);
      off += nw;
      P.gb[size_t(l)].download(grad + off, size_t(nb), s);
      off += nb;
    }
    double ls = 0;
    P.loss_sum.download(&ls, 1, s);
    check_mlp_err(&P);
    if (loss) *loss = ls / (double(n) * P.dims.back());
  });
}

/* Training: the set (X [n][d_0], Y [n][d_L]) is uploaded once; `epochs` passes of Adam (learning
 * rate lr) over minibatches of `batch` rows in the order perm (n indices per epoch, epochs x n in
 * total, or NULL for the identity); each minibatch's loss is its own mean. loss_history [epochs]
 * receives each epoch's mean loss over the set. */
epsp_status epsp_warmstart_train(epsp_warmstart* w, const float* X, const float* Y, int64_t n, int32_t epochs,
                                 int32_t batch, float lr, const int64_t* perm, double* loss_history) {
  if (!w || !X || !Y || n < 1 || epochs < 1 || batch < 1 || !(lr > 0.f)) return EPSP_EINVAL;
  Mlp& P = w->m;
  return wguard(P.ctx, [&] {
    cudaStream_t s = P.ctx->stream;
    const int d0 = P.dims[0], dl = P.dims.back();
    if (perm)
      for (long k = 0; k < long(epochs) * n; ++k)
        if (perm[k] < 0 || perm[k] >= n) fail(EPSP_EINVAL, "perm holds an index outside [0, n)");
    const long nbat = (n + batch - 1) / batch, rows = std::min<long>(n, batch);
    ensure(P.dataX, P.ctx, size_t(n) * size_t(d0));
    ensure(P.dataY, P.ctx, size_t(n) * size_t(dl));
    P.dataX.upload(X, size_t(n) * size_t(d0), s);
    P.dataY.upload(Y, size_t(n) * size_t(dl), s);
    ensure(P.perm, P.ctx, size_t(n));
    ensure(P.loss_sum, P.ctx, size_t(nbat));
    ensure_cap(&P, rows);
    std::vector<int64_t> ident;
    if (!perm) {
      ident.resize(size_t(n));
      for (long k = 0; k < n; ++k) ident[size_t(k)] = k;
    }
    std::vector<double> bl(static_cast<size_t>(nbat));
    // A step's launches are captured once in a CUDA graph and replayed for every full minibatch (its rows, loss slot and
    // step count come from the device); the first step and a last, smaller minibatch are launched one by one (the first
    // launches set the kernels' attributes).
    auto step = [&](long nb) { train_step(&P, nb, Batch{P.perm.p, P.d_step.p + 1, batch, P.dataY.p, 2.f / (float(nb) * float(dl))}, lr); };
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    struct GraphGuard {
      cudaGraph_t* g;
      cudaGraphExec_t* e;
      ~GraphGuard() {
        if (*e) cudaGraphExecDestroy(*e);
        if (*g) cudaGraphDestroy(*g);
      }
    } gguard{&graph, &exec};
    int64_t per_step = 0;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    struct EventGuard {
      cudaEvent_t* e;
      ~EventGuard() {
        for (int k = 0; k < 2; ++k)
          if (e[k]) cudaEventDestroy(e[k]);
      }
    } eguard{ev};
    for (auto& e : ev) EPSP_CUDA(cudaEventCreate(&e));
    P.train_ms = 0;
    for (int e = 0; e < epochs; ++e) {
      P.perm.upload(perm ? perm + long(e) * n : ident.data(), size_t(n), s);
      EPSP_CUDA(cudaMemsetAsync(P.d_step.p + 1, 0, sizeof(int), s));  // the epoch's first minibatch
      EPSP_CUDA(cudaEventRecord(ev[0], s));
      for (long bi = 0; bi < nbat; ++bi) {
        const long nb = std::min<long>(batch, n - bi * batch);
        if ((e == 0 && bi == 0) || nb < rows) {
          step(nb);
          continue;
        }
        if (!exec) {
          const int64_t l0 = P.ctx->launches;
          EPSP_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
          try {
            step(nb);
          } catch (...) {
            cudaStreamEndCapture(s, &graph);
            throw;
          }
          EPSP_CUDA(cudaStreamEndCapture(s, &graph));
          EPSP_CUDA(cudaGraphInstantiate(&exec, graph, 0));
          per_step = P.ctx->launches - l0;
          P.ctx->launches = l0;
        }
        EPSP_CUDA(cudaGraphLaunch(exec, s));
        P.ctx->launches += per_step;
      }
      EPSP_CUDA(cudaEventRecord(ev[1], s));
      P.loss_sum.download(bl.data(), size_t(nbat), s);
      check_mlp_err(&P);
      float ms = 0;
      EPSP_CUDA(cudaEventElapsedTime(&ms, ev[0], ev[1]));
      P.train_ms += double(ms);
      double tot = 0;
      for (double v : bl) tot += v;
      if (loss_history) loss_history[e] = tot / (double(n) * dl);
    }
    // a data set of up to 256 MiB keeps its memory for the next call
    if ((P.dataX.n + P.dataY.n) * sizeof(float) > (size_t(256) << 20)) {
      P.dataX.release();
      P.dataY.release();
    }
    ++P.wgen;
  });
}

}  // extern "C"
