// Training kernels of the learned transport closure: forward, backward and
// Adam for the 4-layer MLP (n_in -> H -> H -> H -> n_out, SiLU) with the
// inference kernel's rounding points (quantisation-aware training): every
// weight is rounded to BF16 (round to nearest even) in the forward pass and
// the rounding is passed through unchanged in the backward pass
// (straight-through); the network inputs are BF16 (hi, lo) pairs as the
// kernel forms them; the hidden activations stay FP32 (the inference kernel
// carries them as BF16 hi/lo pairs, ~16 significant bits); accumulation,
// biases and the master weights are FP32.  Loss: mean over the batch and the outputs of
// ((o - y) scale_o)^2, i.e. the squared error of the log properties.
//
// Parameters are one FP32 buffer in the order W1 [H][n_in], b1 [H],
// W2 [H][H], b2, W3 [H][H], b3, W4 [n_out][H], b4 [n_out].  All arrays are
// device memory owned by the caller; the workspace size comes from
// cc_mlp_workspace_bytes.  Every sum runs in a fixed order (per-CTA partial
// sums reduced in CTA order), so a gradient is reproducible bit for bit.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <string>

#include "../../include/cc_b200.h"

void ccb_set_last_error(const std::string &msg);  // api.cu

namespace {

constexpr int kRows = 32;     // batch rows per CTA
constexpr int kThreads = 256;
constexpr int kMaxWidth = 64; // widest layer (n_in, H, n_out <= 64)
static_assert(kThreads / 32 * 4 == kRows && kThreads / 32 * 8 == kMaxWidth, "a warp holds 4 rows or 8 outputs");

__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ float sigm(float z) { return 1.0f / (1.0f + expf(-z)); }

// Shared memory of k_mlp_grad: activations and gradients in rows of
// kMaxWidth, weights both transposed (forward) and as they are (backward, the
// layers above the first).  The transposed rows are padded by two, so that
// filling them column by column meets two-way bank conflicts at most.
constexpr int kLdT = kMaxWidth + 2;
struct GradSmem {
  float wt[4][kMaxWidth * kLdT];          // r(W)^T: [i][o]
  float w[3][kMaxWidth * kMaxWidth];      // r(W) of layers 1..3: [o][i]
  float a[4][kRows * kMaxWidth];          // inputs of the layers
  float dsilu[3][kRows * kMaxWidth];      // silu'(Z) of the hidden layers
  float g[2][kRows * kMaxWidth];          // dL/dZ, this layer's and the next one's
  float bias[4][kMaxWidth];
  float red[kThreads];
};
static_assert(sizeof(GradSmem) <= 227 * 1024, "one CTA's shared memory");

// acc[r][c] = start[c] + sum over k < K of A[row + r][k] M[k][col + c], the
// sum in the order of k; A in rows of kMaxWidth, zero beyond K up to the next
// multiple of 4, and M's rows zero there too.
__device__ __forceinline__ void tile_product(const float *A, const float *M, int ld, int K, int row, int col,
                                             float (&acc)[4][2]) {
  for (int k = 0; k < K; k += 4) {
    float4 x[4];
    float2 m[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) x[r] = *reinterpret_cast<const float4 *>(A + (row + r) * kMaxWidth + k);
#pragma unroll
    for (int q = 0; q < 4; ++q) m[q] = *reinterpret_cast<const float2 *>(M + (k + q) * ld + col);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float xs[4] = {x[r].x, x[r].y, x[r].z, x[r].w};
#pragma unroll
      for (int q = 0; q < 4; ++q)
        acc[r][0] = fmaf(xs[q], m[q].x, acc[r][0]), acc[r][1] = fmaf(xs[q], m[q].y, acc[r][1]);
    }
  }
}

struct Shape {
  int n_in, H, n_out, B, n_cta;
  int off_w[4], off_b[4], n_params;
  int width_in[4], width_out[4];
};

// Forward, loss and backward of kRows batch rows: Z = A r(W)^T + b, H =
// silu(Z); G = 2 (o - y) s^2 / (B n_out) and the rows' sum of ((o - y) s)^2;
// dZ_prev = (G r(W)) silu'(Z_prev); the rows' weight and bias gradients
// sum_r G[r][o] A[r][i] and sum_r G[r][o].  CTA 0 writes its gradient to
// grad, CTA c > 0 to part[c - 1]; k_grad_reduce adds them in CTA order.
//
// Each warp holds 4 rows x 64 columns (two columns a thread): per 4 steps of
// k, 4 two-value and 4 broadcast four-value shared loads serve 32
// multiply-adds, free of bank conflicts.  Everything between the batch and
// the gradient stays in the CTA's shared memory (192,512 bytes, one CTA per SM).
// At 4096 rows one gradient and Adam step went from 313 us in 20 launches
// (dense kernels with 32-way conflicts, every layer through memory) to 50 us
// in 3; sums run in the order of the separate kernels: equal bit for bit.
__global__ void __launch_bounds__(kThreads, 1)
    k_mlp_grad(const Shape s, const float *__restrict__ params, const float *__restrict__ x,
               const float *__restrict__ y, const float *__restrict__ scale, float *__restrict__ grad,
               float *__restrict__ part, float *__restrict__ loss_part) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  GradSmem &S = *reinterpret_cast<GradSmem *>(smem_raw);
  const int tid = threadIdx.x, r0 = blockIdx.x * kRows;
  const int row = 4 * (tid / 32), col = 2 * (tid % 32);
  {  // zero the padding that tile_product multiplies
    float4 *z = reinterpret_cast<float4 *>(smem_raw);
    for (int e = tid; e < (int)(sizeof(GradSmem) / 16); e += kThreads) z[e] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    const int wi = s.width_in[l], wo = s.width_out[l];
    const float *W = params + s.off_w[l];
    for (int e = tid; e < wo * wi; e += kThreads) {
      const float v = bf16r(W[e]);
      const int o = e / wi, i = e % wi;
      S.wt[l][i * kLdT + o] = v;
      if (l > 0) S.w[l - 1][o * kMaxWidth + i] = v;
    }
    if (tid < wo) S.bias[l][tid] = params[s.off_b[l] + tid];
  }
  for (int e = tid; e < kRows * s.n_in; e += kThreads) {
    const int r = e / s.n_in;
    if (r0 + r < s.B) S.a[0][r * kMaxWidth + e % s.n_in] = x[(size_t)r0 * s.n_in + e];
  }
  __syncthreads();
#pragma unroll 1
  for (int l = 0; l < 4; ++l) {
    const int wo = s.width_out[l];
    if (col < wo) {
      float acc[4][2];
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[r][0] = S.bias[l][col], acc[r][1] = S.bias[l][col + 1 < wo ? col + 1 : col];
      tile_product(S.a[l], S.wt[l], kLdT, s.width_in[l], row, col, acc);
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          if (col + c >= wo || r0 + row + r >= s.B) continue;
          const float z = acc[r][c];
          const int q = (row + r) * kMaxWidth + col + c;
          if (l < 3) {
            const float sg = sigm(z);
            S.a[l + 1][q] = z * sg;
            S.dsilu[l][q] = sg * (1.0f + z * (1.0f - sg));
          } else {
            S.g[0][q] = z;  // the outputs, replaced by their gradient below
          }
        }
    }
    __syncthreads();
  }
  {
    const float inv = 1.0f / ((float)s.B * (float)s.n_out);
    float acc = 0.0f;
    for (int e = tid; e < kRows * s.n_out; e += kThreads) {
      const int r = e / s.n_out, o = e % s.n_out;
      if (r0 + r >= s.B) continue;
      float &g = S.g[0][r * kMaxWidth + o];
      const float err = (g - y[(size_t)(r0 + r) * s.n_out + o]) * scale[o];
      acc = fmaf(err, err, acc);
      g = 2.0f * err * scale[o] * inv;
    }
    S.red[tid] = acc;
    __syncthreads();
    for (int h = kThreads / 2; h > 0; h >>= 1) {
      if (tid < h) S.red[tid] += S.red[tid + h];
      __syncthreads();
    }
    if (tid == 0) loss_part[blockIdx.x] = S.red[0];
  }
  float *out = blockIdx.x == 0 ? grad : part + (size_t)(blockIdx.x - 1) * s.n_params;
#pragma unroll 1
  for (int l = 3; l >= 0; --l) {
    const float *g = S.g[(3 - l) & 1];
    float *g_next = S.g[(4 - l) & 1];
    const int wi = s.width_in[l], wo = s.width_out[l];
    // weight gradients: 8 outputs o x 2 inputs i a thread
    const int o0 = 8 * (tid / 32);
    if (col < wi && o0 < wo) {
      float acc[8][2];
#pragma unroll
      for (int o = 0; o < 8; ++o) acc[o][0] = acc[o][1] = 0.0f;
#pragma unroll 4
      for (int r = 0; r < kRows; ++r) {
        const float2 v = *reinterpret_cast<const float2 *>(S.a[l] + r * kMaxWidth + col);
        const float4 ga = *reinterpret_cast<const float4 *>(g + r * kMaxWidth + o0);
        const float4 gb = *reinterpret_cast<const float4 *>(g + r * kMaxWidth + o0 + 4);
        const float gs[8] = {ga.x, ga.y, ga.z, ga.w, gb.x, gb.y, gb.z, gb.w};
#pragma unroll
        for (int o = 0; o < 8; ++o) acc[o][0] = fmaf(gs[o], v.x, acc[o][0]), acc[o][1] = fmaf(gs[o], v.y, acc[o][1]);
      }
#pragma unroll
      for (int o = 0; o < 8; ++o)
        if (o0 + o < wo) {
          float *w = out + s.off_w[l] + (o0 + o) * wi + col;
          w[0] = acc[o][0];
          if (col + 1 < wi) w[1] = acc[o][1];
        }
    }
    if (tid < wo) {
      float acc = 0.0f;
      for (int r = 0; r < kRows; ++r) acc += g[r * kMaxWidth + tid];
      out[s.off_b[l] + tid] = acc;
    }
    if (l > 0) {
      if (col < wi) {
        float acc[4][2];
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = 0.0f;
        tile_product(g, S.w[l - 1], kMaxWidth, wo, row, col, acc);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int q = (row + r) * kMaxWidth + col + c;
            g_next[q] = col + c < wi ? acc[r][c] * S.dsilu[l - 1][q] : 0.0f;
          }
      } else {  // columns of a wider layer's gradient that this buffer held
#pragma unroll
        for (int r = 0; r < 4; ++r) g_next[(row + r) * kMaxWidth + col] = g_next[(row + r) * kMaxWidth + col + 1] = 0.0f;
      }
      __syncthreads();
    }
  }
}

// grad[e] += the partial gradients of CTAs 1.. in order; the last CTA adds
// up the loss.
__global__ void __launch_bounds__(64) k_grad_reduce(float *__restrict__ grad, const float *__restrict__ part,
                                                    int n_parts, int n, const float *__restrict__ loss_part,
                                                    float inv_count, float *__restrict__ loss) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < n) {
    float acc = grad[e];
#pragma unroll 16
    for (int p = 0; p < n_parts; ++p) acc += part[(size_t)p * n + e];
    grad[e] = acc;
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
    float acc = 0.0f;
#pragma unroll 16
    for (int p = 0; p <= n_parts; ++p) acc += loss_part[p];
    *loss = acc * inv_count;
  }
}

// Adam (Kingma & Ba 2015) with bias correction, no weight decay.
__global__ void k_adam(int64_t n, float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                       float *__restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const float gi = g[e];
  const float mi = b1 * m[e] + (1.0f - b1) * gi;
  const float vi = b2 * v[e] + (1.0f - b2) * gi * gi;
  m[e] = mi, v[e] = vi;
  p[e] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

Shape shape_of(int n_in, int H, int n_out, int B) {
  Shape s{};
  s.n_in = n_in, s.H = H, s.n_out = n_out, s.B = B, s.n_cta = (B + kRows - 1) / kRows;
  const int wi[4] = {n_in, H, H, H}, wo[4] = {H, H, H, n_out};
  int o = 0;
  for (int l = 0; l < 4; ++l) {
    s.width_in[l] = wi[l], s.width_out[l] = wo[l];
    s.off_w[l] = o, o += wo[l] * wi[l];
    s.off_b[l] = o, o += wo[l];
  }
  s.n_params = o;
  return s;
}

// Workspace (floats): the partial gradients of CTAs 1.. (n_params each), then
// the CTAs' loss partials.  The size keeps room for every layer's rows (more
// than the partials need at every shape), so that callers' buffers of earlier
// sizes stay valid.
int64_t work_floats(const Shape &s) {
  return (int64_t)s.B * (3 * s.H + s.n_out) + (int64_t)3 * s.B * s.H + 2LL * s.B * kMaxWidth +
         (int64_t)s.n_cta * kMaxWidth * kMaxWidth + (int64_t)s.n_cta * kMaxWidth + s.n_cta;
}

int fail(int code, const std::string &msg) {
  ccb_set_last_error(msg);
  return code;
}

int check_shape(int n_in, int H, int n_out, int B) {
  if (n_in < 1 || H < 1 || n_out < 1 || n_in > kMaxWidth || H > kMaxWidth || n_out > kMaxWidth)
    return fail(CC_ERR_ARG, "cc_mlp: layer widths must lie in [1, 64]");
  if (B < 1) return fail(CC_ERR_ARG, "cc_mlp: batch must be positive");
  return CC_OK;
}

}  // namespace

extern "C" int64_t cc_mlp_param_count(int n_in, int hidden, int n_out) {
  if (check_shape(n_in, hidden, n_out, 1)) return -1;
  return shape_of(n_in, hidden, n_out, 1).n_params;
}

extern "C" int64_t cc_mlp_workspace_bytes(int n_in, int hidden, int n_out, int batch) {
  if (check_shape(n_in, hidden, n_out, batch)) return -1;
  return work_floats(shape_of(n_in, hidden, n_out, batch)) * (int64_t)sizeof(float);
}

extern "C" int cc_mlp_grad(int n_in, int hidden, int n_out, int batch, const float *params, const float *x,
                           const float *y, const float *out_scale, float *grad, float *loss, void *workspace,
                           void *stream) {
  if (int r = check_shape(n_in, hidden, n_out, batch)) return r;
  if (!params || !x || !y || !out_scale || !grad || !loss || !workspace)
    return fail(CC_ERR_ARG, "cc_mlp_grad: null pointer");
  const Shape s = shape_of(n_in, hidden, n_out, batch);
  float *part = static_cast<float *>(workspace), *loss_part = part + (int64_t)(s.n_cta - 1) * s.n_params;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // above the default limit of dynamic shared memory; an attribute of the
  // kernel on the current device, cheap to set on every call
  cudaError_t attr = cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(GradSmem));
  if (attr != cudaSuccess) return fail(CC_ERR_CUDA, std::string("cc_mlp_grad: ") + cudaGetErrorString(attr));
  k_mlp_grad<<<s.n_cta, kThreads, sizeof(GradSmem), st>>>(s, params, x, y, out_scale, grad, part, loss_part);
  k_grad_reduce<<<(s.n_params + 63) / 64, 64, 0, st>>>(grad, part, s.n_cta - 1, s.n_params, loss_part,
                                                       1.0f / ((float)s.B * (float)s.n_out), loss);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(CC_ERR_CUDA, std::string("cc_mlp_grad: ") + cudaGetErrorString(e));
  return CC_OK;
}

extern "C" int cc_mlp_adam(int64_t n, float *params, const float *grad, float *m, float *v, float lr, float beta1,
                           float beta2, float eps, int step, void *stream) {
  if (n < 1 || step < 1 || !params || !grad || !m || !v) return fail(CC_ERR_ARG, "cc_mlp_adam: bad arguments");
  const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
  k_adam<<<(unsigned)((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(n, params, grad, m, v, lr, beta1,
                                                                                   beta2, eps, c1, c2);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(CC_ERR_CUDA, std::string("cc_mlp_adam: ") + cudaGetErrorString(e));
  return CC_OK;
}
