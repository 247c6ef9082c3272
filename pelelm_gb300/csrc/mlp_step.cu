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
//  * GELU, its derivative and the loss are epilogues;
//  * the gradients of all layers are one launch (grad_kernel), all parameters' Adam another, one block
//    of which adds the loss's partials in FP64.
// Measured (4 x 256): batch 8192 1310 -> 216 us a step, of it 62 us grad_kernel (the batch split over
// more CTAs: 167 us, with other bits).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "mlp_common.cuh"
#include "reactor_registry.cuh"

namespace pgb_mlp {

constexpr int TM = 128, TN = 128, TK = 32, STAGES = 4;
constexpr int LD_K = TK + 8;    // operand tile [row][k]: 40 bf16 = 80 B rows
constexpr int LD_MN = TM + 8;   // operand tile [k][row]: 136 bf16 = 272 B rows
constexpr int kMaxLayers = 16;

enum Epilogue : int { FORWARD = 0, LOSS = 1, INPUT_GRAD = 2 };

struct StepEpi {
  const float* bias;        // FORWARD, LOSS
  float* pre;               // FORWARD: pre-activation out; INPUT_GRAD: in, then the FP32 dZ; LOSS: FP32 dZ
  bf16* out;                // activation, or dZ
  const float* target;      // LOSS
  float* loss_part;         // LOSS: [row tile][column tile][8] sums of the tile's warps
  float scale;
  int ldo, n_valid;
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

// C tile of A (M x K, [row][k]) and B (N x K, [row][k] or [k][row]), 8 warps as 4 x 2 of 32 x 64.
template <bool BK_, int EPI>
__global__ void __launch_bounds__(256, 2) step_gemm_kernel(const bf16* __restrict__ A, int lda, int M,
                                                           const bf16* __restrict__ B, int ldb, int N, int K, StepEpi e) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
  constexpr int TA = tile_bytes<true>(), TB = tile_bytes<BK_>();
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
  const int nk = K / TK;
  auto load = [&](int kt) {
    if (kt < nk) {
      load_tile<true>(sa(kt % STAGES), A, lda, m0, M, kt * TK);
      load_tile<BK_>(sb(kt % STAGES), B, ldb, n0, N, kt * TK);
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
        ldmatrix_x4(a[i][0], a[i][1], a[i][2], a[i][3], a_s + (r + (lane & 15)) * LD_K + kk + (lane >> 4) * 8);
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

  float sq = 0.f;
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
        if constexpr (EPI != FORWARD) *reinterpret_cast<float2*>(e.pre + at) = make_float2(v[0], v[1]);
        *reinterpret_cast<__nv_bfloat162*>(e.out + at) = __nv_bfloat162(__float2bfloat16(v[0]), __float2bfloat16(v[1]));
      }
  if constexpr (EPI == LOSS) {
#pragma unroll
    for (int o = 16; o; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if (lane == 0) e.loss_part[((m0 / TM) * ((N + TN - 1) / TN) + n0 / TN) * 8 + warp] = sq;
  }
}

// Gradients of all layers in one launch: dW (N x Kw) = dZ^T act over the batch by tiles of 32 x 64,
// and db, the column sums of the FP32 dZ, 16 columns a block.
//
// Each entry of dW is one FP32 accumulator that walks the batch in steps of 16, and each column of
// db eight chains (row mod 8) added in order: the orders of gemm_nt_kernel and bias_grad_kernel (mlp.cu),
// so both keep their bits. Adam's first steps divide a gradient by its own size, so another order
// shows in the parameters (measured with the batch split: 5e-5 of a bias vector).
// What bounds it is a stage's turn-round: a tile walks the batch in 128 stages of 64 rows at 1,100 cycles each
// (batch 8192, four layers of 256: 62 us; 174 CTAs, issue slots of a busy SM 26 % used), and of these the four
// dependent products of an accumulator are some 130; the rest is the wait for the copies, the block's barrier, and
// each thread's three copies and eight fragment loads. The tiles are the long part (a step without them takes
// 156 us, without the column sums 212, with both 214). Tiles of 64 x 64 with four, eight or sixteen products a
// scheduler in flight and of 32 x 64 with four or eight all took 62 to 71 us (seven stages or ten in flight); the
// small tile reaches most SMs at narrow layers too. A stage's fragments are read while the products of the one
// before run. The batch split over two CTAs per SM took 20 us, but gave other sums.
constexpr int GN = 32, GT = 64, GB = 64, GSTAGES = 7, LD_N = GN + 8, LD_G = GT + 8, GTHREADS = 256;
constexpr int kGradSmem = GSTAGES * GB * (LD_N + LD_G) * 2;
constexpr int kBiasCols = 16, kBiasRows = 256, kBiasStages = 6;
static_assert(kBiasStages * kBiasRows * kBiasCols * 4 <= kGradSmem, "stage memory");

struct GradLayer {
  const bf16 *dz, *act;
  const float* dzf;
  int N, Kw, lda, tiles_k, first_tile, first_bias;  // first block of this layer's tiles, of its columns
  float *dW, *db;
};
struct GradParams {
  GradLayer l[kMaxLayers];
  int nlayer, nbias, batch;  // nbias: blocks of column sums, which come first
};

__device__ __forceinline__ void bias_columns(const GradLayer& L, int n0, int batch, float* smem) {
  __shared__ float chain[8][kBiasCols];
  const int tid = threadIdx.x, c = tid % kBiasCols, y = tid / kBiasCols;
  const int nst = (batch + kBiasRows - 1) / kBiasRows;
  auto load = [&](int st) {
    if (st < nst) {
#pragma unroll
      for (int k = 0; k < kBiasRows * 4 / GTHREADS; ++k) {
        const int row = (tid >> 2) + GTHREADS / 4 * k, m = st * kBiasRows + row, ch = (tid & 3) * 4;
        cp_async16(smem + ((st % kBiasStages) * kBiasRows + row) * kBiasCols + ch,
                   L.dzf + (size_t)min(m, batch - 1) * L.N + n0 + ch, m < batch);
      }
    }
    cp_async_commit();
  };
  for (int st = 0; st < kBiasStages - 1; ++st) load(st);
  float acc = 0.f;
  for (int st = 0; st < nst; ++st) {
    cp_async_wait<kBiasStages - 2>();
    __syncthreads();
    load(st + kBiasStages - 1);
    if (y < 8) {
      const float* p = smem + ((st % kBiasStages) * kBiasRows + y) * kBiasCols + c;
      const int n = min(kBiasRows, batch - st * kBiasRows) / 8;  // a multiple of 4
      for (int u = 0; u < n; u += 4) {
        float v[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) v[w] = p[(u + w) * 8 * kBiasCols];
#pragma unroll
        for (int w = 0; w < 4; ++w) acc += v[w];
      }
    }
  }
  cp_async_wait<0>();
  if (y < 8) chain[y][c] = acc;
  __syncthreads();
  if (y == 0) {
    float t = 0.f;
    for (int k = 0; k < 8; ++k) t += chain[k][c];
    L.db[n0 + c] = t;
  }
}

__global__ void __launch_bounds__(GTHREADS, 2) grad_kernel(const __grid_constant__ GradParams p) {
  extern __shared__ __align__(16) unsigned char smem[];
  int li = 0;
  if ((int)blockIdx.x < p.nbias) {
    while (li + 1 < p.nlayer && p.l[li + 1].first_bias <= (int)blockIdx.x) ++li;
    bias_columns(p.l[li], (blockIdx.x - p.l[li].first_bias) * kBiasCols, p.batch, reinterpret_cast<float*>(smem));
    return;
  }
  int t = blockIdx.x - p.nbias;
  while (li + 1 < p.nlayer && p.l[li + 1].first_tile <= t) ++li;
  const GradLayer& L = p.l[li];
  t -= L.first_tile;
  const int n0 = t / L.tiles_k * GN, k0 = t % L.tiles_k * GT;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wn = (warp >> 2) * 16, wk = (warp & 3) * 16;
  const int nst = (p.batch + GB - 1) / GB;
  // this thread's share of each stage: rows past the batch and columns past the matrix are zeros
  const int rz = tid >> 2, cz = (tid & 3) * 8, rx = tid >> 3, cx = (tid & 7) * 8;
  const bool ik = k0 + cx < L.Kw;
  const bf16* gz = L.dz + (size_t)rz * L.N + n0 + cz;  // N is a multiple of 32
  const bf16* gx = L.act + (size_t)rx * L.lda + (ik ? k0 + cx : 0);
  const size_t step_z = (size_t)GB * L.N, half_x = (size_t)(GB / 2) * L.lda;
  bf16* const s0 = reinterpret_cast<bf16*>(smem);
  constexpr int SLOT = GB * (LD_N + LD_G);
  int left = p.batch, wslot = 0, rslot = 0;  // left: rows of the batch from the next stage on
  auto load = [&]() {
    bf16* z = s0 + wslot * SLOT + rz * LD_N + cz;
    bf16* x = s0 + wslot * SLOT + GB * LD_N + rx * LD_G + cx;
    cp_async16(z, rz < left ? gz : L.dz, rz < left);
    cp_async16(x, rx < left ? gx : L.act, ik && rx < left);
    cp_async16(x + GB / 2 * LD_G, rx + GB / 2 < left ? gx + half_x : L.act, ik && rx + GB / 2 < left);
    gz += step_z;
    gx += 2 * half_x;
    left -= GB;
    wslot = wslot + 1 < GSTAGES ? wslot + 1 : 0;
    cp_async_commit();
  };
  struct Fragments {
    unsigned a[GB / 16][4], b[GB / 16][2][2];
  };
  float acc[2][4];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int r = 0; r < 4; ++r) acc[j][r] = 0.f;
  const bf16* const fa = s0 + ((lane & 7) + (lane >> 4) * 8) * LD_N + wn + ((lane >> 3) & 1) * 8;
  const bf16* const fb = s0 + GB * LD_N + ((lane & 7) + ((lane >> 3) & 1) * 8) * LD_G + wk + (lane >> 4) * 8;
  auto fetch = [&](Fragments& f) {
    cp_async_wait<GSTAGES - 2>();
    __syncthreads();
    load();
    const int at = rslot * SLOT;
    rslot = rslot + 1 < GSTAGES ? rslot + 1 : 0;
#pragma unroll
    for (int q = 0; q < GB / 16; ++q) {
      ldmatrix_x4_trans(f.a[q][0], f.a[q][1], f.a[q][2], f.a[q][3], fa + at + 16 * q * LD_N);
      ldmatrix_x4_trans(f.b[q][0][0], f.b[q][0][1], f.b[q][1][0], f.b[q][1][1], fb + at + 16 * q * LD_G);
    }
  };
  auto products = [&](const Fragments& f) {
#pragma unroll
    for (int q = 0; q < GB / 16; ++q)
#pragma unroll
      for (int j = 0; j < 2; ++j) mma_bf16(acc[j], f.a[q], f.b[q][j]);
  };
  for (int st = 0; st < GSTAGES - 1; ++st) load();
  Fragments f0, f1;
  fetch(f0);
#pragma unroll 1
  for (int st = 0; st < nst; st += 2) {
    if (st + 1 < nst) fetch(f1);
    products(f0);
    if (st + 1 >= nst) break;
    if (st + 2 < nst) fetch(f0);
    products(f1);
  }
  cp_async_wait<0>();
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int n = n0 + wn + (lane >> 2) + h * 8, k = k0 + wk + j * 8 + (lane & 3) * 2;
      if (k < L.Kw)
        *reinterpret_cast<float2*>(L.dW + (size_t)n * L.Kw + k) = make_float2(acc[j][h * 2], acc[j][h * 2 + 1]);
    }
}

// Adam over all parameters.
struct AdamTensor {
  float *p, *m, *v;
  const float* grad;
  int n;
  bf16* out;             // BF16 copy, or null
  int cols, ldo, dup;    // out row stride; dup: second copy at column dup (0: none)
  int first_block;
};
struct AdamParams {
  AdamTensor t[2 * kMaxLayers];
  int nt;
  float* loss;             // the last block adds the loss's partials, in order
  const float* loss_part;
  int nloss;
  float lr, b1, b2, eps, bc1, bc2;
};

__global__ void __launch_bounds__(256) adam_step_kernel(const __grid_constant__ AdamParams P) {
  if (blockIdx.x == gridDim.x - 1) {
    __shared__ double warp_part[8];
    double sum = 0.0;
    for (int i = threadIdx.x; i < P.nloss; i += 256) sum += (double)P.loss_part[i];
#pragma unroll
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31) == 0) warp_part[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < 8; ++w) sum += warp_part[w];
      *P.loss = (float)sum;
    }
    return;
  }
  int k = 0;
  while (k + 1 < P.nt && P.t[k + 1].first_block <= (int)blockIdx.x) ++k;
  const AdamTensor& t = P.t[k];
  const int i = (blockIdx.x - t.first_block) * 256 + threadIdx.x;
  if (i >= t.n) return;
  const float g = t.grad[i];
  const float m = P.b1 * t.m[i] + (1.f - P.b1) * g;
  const float v = __fmaf_rn(__fmul_rn(1.f - P.b2, g), g, __fmul_rn(P.b2, t.v[i]));
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
static_assert(tile_bytes<true>() >= tile_bytes<false>(), "stage memory");

size_t align16(size_t n) { return (n + 255) / 256 * 256; }

// Workspace of a step: activations, pre-activations (then FP32 dZ) and dZ of the layers, gradients.
struct Layout {
  size_t act[kMaxLayers], pre[kMaxLayers], dz[kMaxLayers], dw[kMaxLayers], db[kMaxLayers], loss, total;
  int mtiles;
};

int weight_cols(const pgb_mlp_step& s, int l) { return l == 0 && s.k_half > 0 ? s.k_half : s.dims[l]; }

Layout layout_of(const pgb_mlp_step& s) {
  Layout y;
  size_t o = 0;
  auto take = [&](size_t n) { const size_t at = o; o += align16(n); return at; };
  y.mtiles = (s.batch + TM - 1) / TM;
  for (int l = 0; l < s.nlayer; ++l) {
    const size_t n = (size_t)s.batch * s.dims[l + 1];
    y.act[l] = l + 1 < s.nlayer ? take(n * 2) : 0;
    y.pre[l] = take(n * 4);
    y.dz[l] = take(n * 2);
    y.dw[l] = take((size_t)s.dims[l + 1] * weight_cols(s, l) * 4);
    y.db[l] = take((size_t)s.dims[l + 1] * 4);
  }
  y.loss = take((size_t)y.mtiles * ((s.dims[s.nlayer] + TN - 1) / TN) * 8 * 4);
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
  PGB_CUDA(cudaFuncSetAttribute(grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGradSmem));
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
      e.pre = fp(y.pre[l]);
      e.target = s.T;
      e.loss_part = fp(y.loss);
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
    step_gemm_kernel<false, INPUT_GRAD><<<grid(e.ldo), 256, kStepSmem, st>>>(dz(l), s.dims[l + 1], B, wb(l), s.dims[l],
                                                                            e.ldo, s.dims[l + 1], e);
    PGB_CUDA(cudaGetLastError());
  }
  GradParams w;
  w.nlayer = L;
  w.batch = B;
  int tiles = 0;
  w.nbias = 0;
  for (int l = 0; l < L; ++l) {
    GradLayer& g = w.l[l];
    g.dz = dz(l);
    g.act = act(l - 1);
    g.dzf = fp(y.pre[l]);
    g.lda = ld(l - 1);
    g.N = s.dims[l + 1];
    g.Kw = weight_cols(s, l);
    g.tiles_k = (g.Kw + GT - 1) / GT;
    g.first_tile = tiles;
    g.first_bias = w.nbias;
    g.dW = fp(y.dw[l]);
    g.db = fp(y.db[l]);
    tiles += g.N / GN * g.tiles_k;
    w.nbias += g.N / kBiasCols;
  }
  grad_kernel<<<w.nbias + tiles, GTHREADS, kGradSmem, st>>>(w);
  PGB_CUDA(cudaGetLastError());
  AdamParams a;
  a.nt = 0;
  a.lr = s.lr; a.b1 = s.b1; a.b2 = s.b2; a.eps = s.eps;
  a.bc1 = 1.f - powf(s.b1, (float)s.step);
  a.bc2 = 1.f - powf(s.b2, (float)s.step);
  int blocks = 0;
  auto add = [&](float* p, float* m, float* v, const float* grad, int n, void* out, int cols, int ldo,
                 int dup) {
    AdamTensor& t = a.t[a.nt++];
    t.p = p; t.m = m; t.v = v; t.grad = grad;
    t.n = n;
    t.out = static_cast<bf16*>(out); t.cols = cols; t.ldo = ldo; t.dup = dup;
    t.first_block = blocks;
    blocks += (n + 255) / 256;
  };
  for (int l = 0; l < L; ++l) {
    const int n = s.dims[l + 1], kw = weight_cols(s, l);
    const bool split_in = l == 0 && s.k_half > 0;
    add(s.W[l], s.mW[l], s.vW[l], fp(y.dw[l]), n * kw, s.Wb[l], kw, s.dims[l], split_in ? kw : 0);
    add(s.b[l], s.mb[l], s.vb[l], fp(y.db[l]), n, nullptr, 1, 1, 0);
  }
  a.loss = s.loss;
  a.loss_part = fp(y.loss);
  a.nloss = y.mtiles * ((s.dims[L] + TN - 1) / TN) * 8;
  adam_step_kernel<<<blocks + 1, 256, 0, st>>>(a);
  PGB_CUDA(cudaGetLastError());
  return 0;
}

}  // extern "C"
