// One optimiser step of the surrogate MLP in a dozen launches: forward, mean-squared error, backward
// and Adam, enqueued by one call (pgb_mlp_train_step).
//
// The step at its batch of 8192 (4 x 256) is 11 GFLOP, about 10 us of tensor time; what it took
// (1.32 ms) went into some fifty launches, the host work between them, and kernels that left the
// chip idle: a weight gradient of 4 CTAs walking the whole batch, bias gradients of 8 CTAs, and a
// transpose before each product. Here
//  * products read their operands as they lie (ldmatrix with or without .trans), so nothing is
//    transposed; forward and input gradients keep the accumulation order of gemm_nt_kernel (mlp.cu),
//    k in steps of 16 in one FP32 accumulator, so activations and gradients keep their bits;
//  * GELU, its derivative, the loss and the bias-gradient column sums are epilogues;
//  * the weight gradients of all layers are one launch, split along the batch so that about two CTAs
//    per SM work, and Adam adds the splits (in order: deterministic) as it reads them.
// Measured (batch 8192, 4 x 256): 1312 -> 170 us a step; batch 256: 370 -> 90 us (host calls).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "mlp_common.cuh"
#include "reactor_registry.cuh"

namespace pgb_mlp {

constexpr int TM = 128, TN = 128, TK = 32, STAGES = 4;
constexpr int LD_K = TK + 8;    // operand tile [row][k]: 40 bf16 = 80 B rows
constexpr int LD_MN = TM + 8;   // operand tile [k][row]: 136 bf16 = 272 B rows
constexpr int kMaxLayers = 16;

enum Epilogue : int { FORWARD = 0, LOSS = 1, INPUT_GRAD = 2, PARTIAL = 3 };

struct StepEpi {
  const float* bias;        // FORWARD, LOSS
  float* pre;               // FORWARD: pre-activation out; INPUT_GRAD: in
  bf16* out;                // activation, or dZ
  float* bias_part;         // LOSS, INPUT_GRAD: [row tile][ldo] column sums of dZ
  const float* target;      // LOSS
  float* loss;
  float scale;
  int ldo, n_valid;
  float* part;              // PARTIAL: C of this split
};

// Bytes of one stage of an operand whose tile is [row][k] (KMAJOR) or [k][row].
template <bool KMAJOR>
__host__ __device__ constexpr int tile_bytes() {
  return 2 * (KMAJOR ? TM * LD_K : TK * LD_MN);
}

// Loads a 128 x 32 operand tile (rows r0.., k k0..) of a matrix stored [row][k] (KMAJOR) or [k][row].
template <bool KMAJOR>
__device__ __forceinline__ void load_tile(bf16* s, const bf16* __restrict__ g, int ld, int r0, int rows, int k0) {
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const int idx = threadIdx.x + c * 256;
    if constexpr (KMAJOR) {
      const int row = idx >> 2, ch = idx & 3;
      cp_async16(s + row * LD_K + ch * 8, g + (size_t)min(r0 + row, rows - 1) * ld + k0 + ch * 8, r0 + row < rows);
    } else {
      const int k = idx >> 4, ch = idx & 15;
      const bool ok = r0 + ch * 8 < rows;
      cp_async16(s + k * LD_MN + ch * 8, g + (size_t)(k0 + k) * ld + (ok ? r0 + ch * 8 : 0), ok);
    }
  }
}

// C tile (m0, n0) of A (M x K) and B (N x K) over k in [k0, k1), 8 warps as 4 x 2 of 32 x 64.
template <bool AK, bool BK_, int EPI>
__device__ __forceinline__ void step_tile(unsigned char* smem, const bf16* __restrict__ A, int lda, int M, int m0,
                                          const bf16* __restrict__ B, int ldb, int N, int n0, int k0, int k1,
                                          const StepEpi& e) {
  constexpr int TA = tile_bytes<AK>(), TB = tile_bytes<BK_>();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp >> 1, wn = warp & 1;
  float acc[2][8][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[i][j][r] = 0.f;
  auto sa = [&](int st) { return reinterpret_cast<bf16*>(smem + st * (TA + TB)); };
  auto sb = [&](int st) { return reinterpret_cast<bf16*>(smem + st * (TA + TB) + TA); };
  const int nk = (k1 - k0) / TK;
  auto load = [&](int kt) {
    if (kt < nk) {
      load_tile<AK>(sa(kt % STAGES), A, lda, m0, M, k0 + kt * TK);
      load_tile<BK_>(sb(kt % STAGES), B, ldb, n0, N, k0 + kt * TK);
    }
    cp_async_commit();
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) load(s);
  for (int kt = 0; kt < nk; ++kt) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    load(kt + STAGES - 1);
    const bf16* a_s = sa(kt % STAGES);
    const bf16* b_s = sb(kt % STAGES);
#pragma unroll
    for (int kk = 0; kk < TK; kk += 16) {
      unsigned a[2][4], b[8][2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = wm * 32 + i * 16;
        if constexpr (AK)
          ldmatrix_x4(a[i][0], a[i][1], a[i][2], a[i][3], a_s + (r + (lane & 15)) * LD_K + kk + (lane >> 4) * 8);
        else
          ldmatrix_x4_trans(a[i][0], a[i][1], a[i][2], a[i][3],
                            a_s + (kk + (lane & 7) + (lane >> 4) * 8) * LD_MN + r + ((lane >> 3) & 1) * 8);
      }
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        const int r = wn * 64 + j * 8;
        if constexpr (BK_)
          ldmatrix_x4(b[j][0], b[j][1], b[j + 1][0], b[j + 1][1],
                      b_s + (r + (lane & 7) + ((lane >> 4) << 3)) * LD_K + kk + ((lane >> 3) & 1) * 8);
        else
          ldmatrix_x4_trans(b[j][0], b[j][1], b[j + 1][0], b[j + 1][1],
                            b_s + (kk + (lane & 7) + ((lane >> 3) & 1) * 8) * LD_MN + r + (lane >> 4) * 8);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) mma_bf16(acc[i][j], a[i], b[j]);
    }
  }
  cp_async_wait<0>();
  __syncthreads();  // the column sums below reuse the tiles' memory

  float col[8][2];
  float sq = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) col[j][0] = col[j][1] = 0.f;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int m = m0 + wm * 32 + i * 16 + (lane >> 2) + h * 8;
        const int n = n0 + wn * 64 + j * 8 + (lane & 3) * 2;
        if (m >= M || n >= N) continue;  // N is even
        float v[2] = {acc[i][j][h * 2], acc[i][j][h * 2 + 1]};
        const size_t at = (size_t)m * e.ldo + n;
        if constexpr (EPI == PARTIAL) {
          *reinterpret_cast<float2*>(e.part + at) = make_float2(v[0], v[1]);
        } else {
          if constexpr (EPI == FORWARD) {
            v[0] += e.bias[n];
            v[1] += e.bias[n + 1];
            *reinterpret_cast<float2*>(e.pre + at) = make_float2(v[0], v[1]);
            v[0] = gelu(v[0]);
            v[1] = gelu(v[1]);
          } else if constexpr (EPI == LOSS) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              const float y = v[c] + e.bias[n + c];
              v[c] = 0.f;
              if (n + c < e.n_valid) {
                const float d = y - e.target[at + c];
                sq += d * d;
                v[c] = e.scale * d;
              }
            }
          } else {
            const float2 p = *reinterpret_cast<const float2*>(e.pre + at);
            v[0] *= gelu_grad(p.x);
            v[1] *= gelu_grad(p.y);
          }
          if constexpr (EPI != FORWARD) {
            col[j][0] += v[0];
            col[j][1] += v[1];
          }
          *reinterpret_cast<__nv_bfloat162*>(e.out + at) = __nv_bfloat162(__float2bfloat16(v[0]), __float2bfloat16(v[1]));
        }
      }
  if constexpr (EPI == LOSS || EPI == INPUT_GRAD) {
    // column sums of the tile: over a warp's 32 rows by shuffles, then over the four warp rows
    float* cs = reinterpret_cast<float*>(smem);  // [4][TN]
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) col[j][c] += __shfl_xor_sync(0xffffffffu, col[j][c], o);
        if (lane < 4) cs[wm * TN + wn * 64 + j * 8 + lane * 2 + c] = col[j][c];
      }
    __syncthreads();
    if (tid < TN && n0 + tid < N)
      e.bias_part[(size_t)(m0 / TM) * e.ldo + n0 + tid] = cs[tid] + cs[TN + tid] + cs[2 * TN + tid] + cs[3 * TN + tid];
  }
  if constexpr (EPI == LOSS) {
#pragma unroll
    for (int o = 16; o; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if (lane == 0 && sq != 0.f) atomicAdd(e.loss, sq);
  }
}

template <bool BK_, int EPI>
__global__ void __launch_bounds__(256, 2) step_gemm_kernel(const bf16* __restrict__ A, int lda, int M,
                                                           const bf16* __restrict__ B, int ldb, int N, int K, StepEpi e) {
  extern __shared__ __align__(16) unsigned char step_smem[];
  step_tile<true, BK_, EPI>(step_smem, A, lda, M, blockIdx.y * TM, B, ldb, N, blockIdx.x * TN, 0, K, e);
}

// Weight gradients of all layers: layer l's dW (N x Kw) = dZ^T act over the batch, its tiles and the
// batch's splits dealt to the grid.
struct WGradLayer {
  const bf16 *dz, *act;
  int N, Kw, lda, tiles_k, first_tile;  // first_tile: of this layer in the tile order
  float* part;                          // [split][N][Kw]
};
struct WGradParams {
  WGradLayer l[kMaxLayers];
  int nlayer, ntile, batch, chunk;  // chunk: batch rows of one split
};

__global__ void __launch_bounds__(256, 2) wgrad_kernel(const __grid_constant__ WGradParams p) {
  extern __shared__ __align__(16) unsigned char step_smem[];
  const int split = blockIdx.x / p.ntile;
  int t = blockIdx.x % p.ntile, li = 0;
  while (li + 1 < p.nlayer && p.l[li + 1].first_tile <= t) ++li;
  const WGradLayer& L = p.l[li];
  t -= L.first_tile;
  StepEpi e{};
  e.ldo = L.Kw;
  e.part = L.part + (size_t)split * L.N * L.Kw;
  step_tile<false, false, PARTIAL>(step_smem, L.dz, L.N, L.N, (t / L.tiles_k) * TM, L.act, L.lda, L.Kw,
                                   (t % L.tiles_k) * TN, split * p.chunk, min(p.batch, (split + 1) * p.chunk), e);
}

// Adam over all parameters; a gradient is the sum of its partials in order.
struct AdamTensor {
  float *p, *m, *v;
  const float* part;
  int n, npart, stride;  // partial s at part + s * stride
  bf16* out;             // BF16 copy, or null
  int cols, ldo, dup;    // out row stride; dup: second copy at column dup (0: none)
  int first_block;
};
struct AdamParams {
  AdamTensor t[2 * kMaxLayers];
  int nt;
  float lr, b1, b2, eps, bc1, bc2;
};

__global__ void __launch_bounds__(256) adam_step_kernel(const __grid_constant__ AdamParams P) {
  int k = 0;
  while (k + 1 < P.nt && P.t[k + 1].first_block <= (int)blockIdx.x) ++k;
  const AdamTensor& t = P.t[k];
  const int i = (blockIdx.x - t.first_block) * 256 + threadIdx.x;
  if (i >= t.n) return;
  float g = 0.f;
#pragma unroll 8
  for (int s = 0; s < t.npart; ++s) g += t.part[(size_t)s * t.stride + i];
  const float m = P.b1 * t.m[i] + (1.f - P.b1) * g;
  const float v = P.b2 * t.v[i] + (1.f - P.b2) * g * g;
  t.m[i] = m;
  t.v[i] = v;
  const float w = t.p[i] - P.lr * (m / P.bc1) / (sqrtf(v / P.bc2) + P.eps);
  t.p[i] = w;
  if (t.out) {
    const size_t at = (size_t)(i / t.cols) * t.ldo + i % t.cols;
    t.out[at] = __float2bfloat16(w);
    if (t.dup) t.out[at + t.dup] = __float2bfloat16(w);
  }
}

}  // namespace pgb_mlp

using namespace pgb_host;
using namespace pgb_mlp;

namespace {

constexpr int kStepSmem = STAGES * 2 * 2 * TM * LD_K;  // the larger of the layouts
static_assert(tile_bytes<true>() >= tile_bytes<false>() && 4 * TN * 4 <= kStepSmem, "stage memory");

size_t align16(size_t n) { return (n + 255) / 256 * 256; }

// Workspace of a step: activations, pre-activations and dZ of the layers, gradient partials.
struct Layout {
  size_t act[kMaxLayers], pre[kMaxLayers], dz[kMaxLayers], wpart[kMaxLayers], bpart[kMaxLayers], total;
  int split, chunk, ntile, mtiles;
};

int weight_cols(const pgb_mlp_step& s, int l) { return l == 0 && s.k_half > 0 ? s.k_half : s.dims[l]; }

Layout layout_of(const pgb_mlp_step& s) {
  Layout y;
  size_t o = 0;
  auto take = [&](size_t n) { const size_t at = o; o += align16(n); return at; };
  y.ntile = 0;
  for (int l = 0; l < s.nlayer; ++l)
    y.ntile += ((s.dims[l + 1] + TM - 1) / TM) * ((weight_cols(s, l) + TN - 1) / TN);
  // about two CTAs per SM of a GB300, each with at least two k steps of the batch
  const int want = std::max(1, 304 / y.ntile), most = std::max(1, s.batch / (2 * TK));
  const int split = std::min(want, most);
  y.chunk = ((s.batch / TK + split - 1) / split) * TK;
  y.split = (s.batch + y.chunk - 1) / y.chunk;
  y.mtiles = (s.batch + TM - 1) / TM;
  for (int l = 0; l < s.nlayer; ++l) {
    const size_t n = (size_t)s.batch * s.dims[l + 1];
    y.act[l] = l + 1 < s.nlayer ? take(n * 2) : 0;
    y.pre[l] = l + 1 < s.nlayer ? take(n * 4) : 0;
    y.dz[l] = take(n * 2);
    y.wpart[l] = take((size_t)y.split * s.dims[l + 1] * weight_cols(s, l) * 4);
    y.bpart[l] = take((size_t)y.mtiles * s.dims[l + 1] * 4);
  }
  y.total = o;
  return y;
}

int check_step(const pgb_mlp_step* s) {
  if (!s) return set_err("mlp_train_step: null argument");
  if (s->nlayer < 1 || s->nlayer > kMaxLayers) return set_err("mlp_train_step: 1 to %d layers", kMaxLayers);
  if (s->batch <= 0 || s->batch % TK || s->ldx % 8)
    return set_err("mlp_train_step: need batch > 0, batch %% 32 == 0, ldx a multiple of 8");
  for (int l = 0; l <= s->nlayer; ++l)
    if (s->dims[l] <= 0 || s->dims[l] % 32) return set_err("mlp_train_step: layer sizes must be multiples of 32");
  if (s->k_half < 0 || s->k_half % 16 || 2 * s->k_half > s->dims[0])
    return set_err("mlp_train_step: k_half must be a multiple of 16 with 2 k_half <= dims[0]");
  if (s->n_out < 1 || s->n_out > s->dims[s->nlayer]) return set_err("mlp_train_step: bad n_out");
  if (s->step < 1) return set_err("adam: step must be >= 1");
  return 0;
}

}  // namespace

extern "C" {

long long pgb_mlp_train_workspace(const pgb_mlp_step* s) {
  if (check_step(s)) return -1;
  return (long long)layout_of(*s).total;
}

int pgb_mlp_train_step(const pgb_mlp_step* sp, void* workspace, void* stream) {
  if (check_step(sp)) return -1;
  const pgb_mlp_step& s = *sp;
  if (!s.X || !s.T || !s.loss || !workspace) return set_err("mlp_train_step: null argument");
  for (int l = 0; l < s.nlayer; ++l)
    if (!s.W[l] || !s.b[l] || !s.Wb[l] || !s.mW[l] || !s.vW[l] || !s.mb[l] || !s.vb[l])
      return set_err("mlp_train_step: null parameter of layer %d", l);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const Layout y = layout_of(s);
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  const int L = s.nlayer, B = s.batch, last = L - 1;
  auto act = [&](int l) { return l < 0 ? static_cast<const bf16*>(s.X) : reinterpret_cast<bf16*>(ws + y.act[l]); };
  auto ld = [&](int l) { return l < 0 ? s.ldx : s.dims[l + 1]; };  // of act(l)
  auto fp = [&](size_t at) { return reinterpret_cast<float*>(ws + at); };
  auto dz = [&](int l) { return reinterpret_cast<bf16*>(ws + y.dz[l]); };
  auto wb = [&](int l) { return static_cast<const bf16*>(s.Wb[l]); };
  auto grid = [&](int n) { return dim3((n + TN - 1) / TN, y.mtiles); };
  PGB_CUDA(cudaFuncSetAttribute(step_gemm_kernel<true, FORWARD>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStepSmem));
  PGB_CUDA(cudaFuncSetAttribute(step_gemm_kernel<true, LOSS>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStepSmem));
  PGB_CUDA(cudaFuncSetAttribute(step_gemm_kernel<false, INPUT_GRAD>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStepSmem));
  PGB_CUDA(cudaFuncSetAttribute(wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStepSmem));
  PGB_CUDA(cudaMemsetAsync(s.loss, 0, sizeof(float), st));
  for (int l = 0; l < L; ++l) {
    StepEpi e{};
    e.bias = s.b[l];
    e.ldo = s.dims[l + 1];
    if (l < last) {
      e.pre = fp(y.pre[l]);
      e.out = reinterpret_cast<bf16*>(ws + y.act[l]);
      step_gemm_kernel<true, FORWARD><<<grid(e.ldo), 256, kStepSmem, st>>>(act(l - 1), ld(l - 1), B, wb(l), s.dims[l],
                                                                          e.ldo, s.dims[l], e);
    } else {
      e.out = dz(l);
      e.bias_part = fp(y.bpart[l]);
      e.target = s.T;
      e.loss = s.loss;
      e.scale = 2.f / ((float)B * (float)s.n_out);
      e.n_valid = s.n_out;
      step_gemm_kernel<true, LOSS><<<grid(e.ldo), 256, kStepSmem, st>>>(act(l - 1), ld(l - 1), B, wb(l), s.dims[l],
                                                                       e.ldo, s.dims[l], e);
    }
    PGB_CUDA(cudaGetLastError());
  }
  for (int l = last; l > 0; --l) {  // dZ of layer l - 1 = (dZ_l W_l) GELU'(pre)
    StepEpi e{};
    e.ldo = s.dims[l];
    e.pre = fp(y.pre[l - 1]);
    e.out = dz(l - 1);
    e.bias_part = fp(y.bpart[l - 1]);
    step_gemm_kernel<false, INPUT_GRAD><<<grid(e.ldo), 256, kStepSmem, st>>>(dz(l), s.dims[l + 1], B, wb(l), s.dims[l],
                                                                            e.ldo, s.dims[l + 1], e);
    PGB_CUDA(cudaGetLastError());
  }
  WGradParams w;
  w.nlayer = L;
  w.ntile = y.ntile;
  w.batch = B;
  w.chunk = y.chunk;
  int first = 0;
  for (int l = 0; l < L; ++l) {
    WGradLayer& g = w.l[l];
    g.dz = dz(l);
    g.act = act(l - 1);
    g.lda = ld(l - 1);
    g.N = s.dims[l + 1];
    g.Kw = weight_cols(s, l);
    g.tiles_k = (g.Kw + TN - 1) / TN;
    g.first_tile = first;
    g.part = fp(y.wpart[l]);
    first += ((g.N + TM - 1) / TM) * g.tiles_k;
  }
  wgrad_kernel<<<y.ntile * y.split, 256, kStepSmem, st>>>(w);
  PGB_CUDA(cudaGetLastError());
  AdamParams a;
  a.nt = 0;
  a.lr = s.lr; a.b1 = s.b1; a.b2 = s.b2; a.eps = s.eps;
  a.bc1 = 1.f - powf(s.b1, (float)s.step);
  a.bc2 = 1.f - powf(s.b2, (float)s.step);
  int blocks = 0;
  auto add = [&](float* p, float* m, float* v, const float* part, int n, int npart, int stride, void* out, int cols,
                 int ldo, int dup) {
    AdamTensor& t = a.t[a.nt++];
    t.p = p; t.m = m; t.v = v; t.part = part;
    t.n = n; t.npart = npart; t.stride = stride;
    t.out = static_cast<bf16*>(out); t.cols = cols; t.ldo = ldo; t.dup = dup;
    t.first_block = blocks;
    blocks += (n + 255) / 256;
  };
  for (int l = 0; l < L; ++l) {
    const int n = s.dims[l + 1], kw = weight_cols(s, l);
    const bool split_in = l == 0 && s.k_half > 0;
    add(s.W[l], s.mW[l], s.vW[l], fp(y.wpart[l]), n * kw, y.split, n * kw, s.Wb[l], kw, s.dims[l], split_in ? kw : 0);
    add(s.b[l], s.mb[l], s.vb[l], fp(y.bpart[l]), n, y.mtiles, n, nullptr, 1, 1, 0);
  }
  adam_step_kernel<<<blocks, 256, 0, st>>>(a);
  PGB_CUDA(cudaGetLastError());
  return 0;
}

}  // extern "C"
