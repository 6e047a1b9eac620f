// fvs_mlp.cu — the learned warm start: a small MLP trained and evaluated on
// the GPU with the library's own kernels.
//
// Network: n_in -> width (GELU) -> ... -> width (GELU) -> n_out, `depth`
// hidden layers.  Weights are kept in FP32 (Adam master copy) and rounded to
// BF16 for every GEMM; activations enter the GEMMs in BF16; every GEMM
// accumulates in FP32 on the tensor cores: tcgen05.mma with the accumulator in
// tensor memory (fvs_tcgemm.cuh, the default engine), or the warp-level
// mma.sync m16n8k16 kernel below (kept as the comparison engine).
// Training: minibatch Adam on the mean squared error.
//
// With tcgen05 a training step is a gather, one GEMM per layer forward (the last
// one with the loss and its gradient as epilogue), one per layer backward (GELU'
// as epilogue), one launch for all weight and bias gradients and one that adds
// their partial sums and applies Adam: 2 (depth + 1) + 2 launches.
//
// GEMM convention: C[m][n] = sum_k A(m,k) B(n,k) (+ bias[n]); each operand is
// either K-major (row m at A + m*lda) or stored transposed (element (m,k) at
// A + k*lda + m), which covers the forward pass (X W^T), the input gradient
// (dZ W) and the weight gradient (dZ^T X) without explicit transposes.
//
// The reference has no learned component; this is the third "AI-systems
// pattern" laid over the drop-in FP64 path, which stays unchanged.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <memory>
#include <new>
#include <random>
#include <string>
#include <vector>

#include "../../include/fvs2d.h"
#include "fvs_internal.hpp"
#include "fvs_tcgemm.cuh"

namespace {

thread_local std::string g_mlp_error;

typedef __nv_bfloat16 bf16;

constexpr int BM = 128, BN = 128, BK = 32, KPAD = 8;  // smem rows padded to avoid bank conflicts
constexpr int GEMM_THREADS = 256;                       // 8 warps: 4 along M x 2 along N, 32x64 each

enum Epilogue : int { EPI_F32 = 0, EPI_BIAS_F32 = 1, EPI_BIAS_GELU = 2 };

__device__ __forceinline__ void mma_bf16(float* d, const uint32_t* a, const uint32_t* b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
  return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

// tile loader: operand element (row r, col k) of a [rows x K] view into smem
// s[r][k]; out-of-range elements read as zero
template <bool KMAJOR>
__device__ __forceinline__ void load_tile(bf16 (*s)[BK + KPAD], const bf16* g, int ld, int row0, int rows, int k0, int K,
                                          int ntile_rows) {
  const int t = threadIdx.x;
  if (KMAJOR) {
    // 8 contiguous k per load
    for (int i = t; i < ntile_rows * (BK / 8); i += GEMM_THREADS) {
      const int r = i / (BK / 8), kk = (i % (BK / 8)) * 8;
      const int gr = row0 + r, gk = k0 + kk;
#pragma unroll
      for (int j = 0; j < 8; j++)
        s[r][kk + j] = (gr < rows && gk + j < K) ? g[(size_t)gr * ld + gk + j] : __float2bfloat16(0.f);
    }
  } else {
    // element (r, k) at g + k*ld + r: contiguous along r
    for (int i = t; i < ntile_rows * BK; i += GEMM_THREADS) {
      const int kk = i / ntile_rows, r = i % ntile_rows;
      const int gr = row0 + r, gk = k0 + kk;
      s[r][kk] = (gr < rows && gk < K) ? g[(size_t)gk * ld + gr] : __float2bfloat16(0.f);
    }
  }
}

template <bool A_KM, bool B_KM>
__global__ void __launch_bounds__(GEMM_THREADS) k_gemm(const bf16* __restrict__ A, int lda, const bf16* __restrict__ B,
                                                       int ldb, int M, int N, int K, int epi,
                                                       const float* __restrict__ bias, float* __restrict__ C, int ldc,
                                                       bf16* __restrict__ Cact, int ldact) {
  __shared__ __align__(16) bf16 sA[BM][BK + KPAD];
  __shared__ __align__(16) bf16 sB[BN][BK + KPAD];
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wm = (warp & 3) * 32, wn = (warp >> 2) * 64;
  const int g = lane >> 2, tq = lane & 3;
  float acc[2][8][4];
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 8; j++)
#pragma unroll
      for (int q = 0; q < 4; q++) acc[i][j][q] = 0.f;
  for (int k0 = 0; k0 < K; k0 += BK) {
    load_tile<A_KM>(sA, A, lda, m0, M, k0, K, BM);
    load_tile<B_KM>(sB, B, ldb, n0, N, k0, K, BN);
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; kk += 16) {
      uint32_t af[2][4], bfr[8][2];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const int r = wm + 16 * i + g;
        af[i][0] = *reinterpret_cast<const uint32_t*>(&sA[r][kk + 2 * tq]);
        af[i][1] = *reinterpret_cast<const uint32_t*>(&sA[r + 8][kk + 2 * tq]);
        af[i][2] = *reinterpret_cast<const uint32_t*>(&sA[r][kk + 8 + 2 * tq]);
        af[i][3] = *reinterpret_cast<const uint32_t*>(&sA[r + 8][kk + 8 + 2 * tq]);
      }
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const int c = wn + 8 * j + g;
        bfr[j][0] = *reinterpret_cast<const uint32_t*>(&sB[c][kk + 2 * tq]);
        bfr[j][1] = *reinterpret_cast<const uint32_t*>(&sB[c][kk + 8 + 2 * tq]);
      }
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) mma_bf16(acc[i][j], af[i], bfr[j]);
    }
    __syncthreads();
  }
  // epilogue
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 8; j++)
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int m = m0 + wm + 16 * i + g + (q >= 2 ? 8 : 0);
        const int n = n0 + wn + 8 * j + 2 * tq + (q & 1);
        if (m >= M || n >= N) continue;
        float z = acc[i][j][q];
        if (epi != EPI_F32 && bias) z += bias[n];
        if (C) C[(size_t)m * ldc + n] = z;
        if (epi == EPI_BIAS_GELU && Cact) Cact[(size_t)m * ldact + n] = __float2bfloat16(gelu(z));
      }
}

__global__ void k_f32_to_bf16(const float* __restrict__ x, bf16* __restrict__ y, size_t n) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i < n) y[i] = __float2bfloat16(x[i]);
}

// rows of the dataset selected by idx (null: all), padded to ld columns, as BF16
__global__ void k_gather_rows(const float* __restrict__ x, int ncol, const int* __restrict__ idx, int n, bf16* __restrict__ out,
                              int ld) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * ld) return;
  const int r = i / ld, c = i % ld;
  out[i] = __float2bfloat16(c < ncol ? x[(size_t)(idx ? idx[r] : r) * ncol + c] : 0.f);
}

// the first nout columns of Y
__global__ void k_columns(const float* __restrict__ Y, int ldy, int n, int nout, float* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n * nout) out[i] = Y[(size_t)(i / nout) * ldy + i % nout];
}

// dY = 2 (Y - T[idx]) / (n * nout) as BF16 (ld = ldg), squared error summed into loss
__global__ void k_mse(const float* __restrict__ Y, int ldy, const float* __restrict__ T, const int* __restrict__ idx, int n,
                      int nout, bf16* __restrict__ dY, int ldg, float* __restrict__ loss_acc) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  float e2 = 0.f;
  if (i < n * ldg) {
    const int r = i / ldg, c = i % ldg;
    float d = 0.f;
    if (c < nout) {
      d = Y[(size_t)r * ldy + c] - T[(size_t)(idx ? idx[r] : r) * nout + c];
      e2 = d * d;
    }
    dY[i] = __float2bfloat16(2.f * d / float(n * nout));
  }
  for (int o = 16; o > 0; o >>= 1) e2 += __shfl_down_sync(0xffffffffu, e2, o);
  if ((threadIdx.x & 31) == 0 && e2 != 0.f) atomicAdd(loss_acc, e2);
}

// dZ = dA * gelu'(Z) as BF16
__global__ void k_gelu_back(const float* __restrict__ dA, const float* __restrict__ Z, bf16* __restrict__ dZ, size_t n) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i < n) dZ[i] = __float2bfloat16(dA[i] * gelu_grad(Z[i]));
}

// bias gradient: column sums of a [n x cols] BF16 matrix (ld).  A block of
// 32 x 32 threads takes 32 columns: each thread row sums every 32nd matrix
// row, then the 32 partial sums of a column are added in a fixed order
// (deterministic).
__global__ void __launch_bounds__(1024) k_colsum(const bf16* __restrict__ g, int n, int cols, int ld,
                                                 float* __restrict__ out) {
  __shared__ float part[32][33];
  const int c = blockIdx.x * 32 + threadIdx.x;
  float s = 0.f;
  if (c < cols)
    for (int r = threadIdx.y; r < n; r += 32) s += __bfloat162float(g[(size_t)r * ld + c]);
  part[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && c < cols) {
    float t = 0.f;
    for (int k = 0; k < 32; k++) t += part[k][threadIdx.x];
    out[c] = t;
  }
}

__global__ void k_adam(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v, size_t n,
                       float lr, float b1, float b2, float eps, float bc1, float bc2) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  w[i] -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
}

inline unsigned nblk(size_t n, int b = 256) { return (unsigned)((n + b - 1) / b); }
inline int pad16(int x) { return (x + 15) / 16 * 16; }

}  // namespace

struct fvs_mlp {
  int n_in = 0, width = 0, depth = 0, n_out = 0;
  int in_pad = 0, out_pad = 0;
  int nl = 0;                        // GEMM layers = depth + 1
  std::vector<int> din, dout;        // padded layer dimensions
  std::vector<size_t> woff, boff;    // offsets into the FP32 parameter vector
  size_t nparam = 0;
  std::string err;
  cudaStream_t stream = nullptr;
  float* w = nullptr;                // FP32 master parameters (padded layout)
  float* g = nullptr;                // gradients
  float* am = nullptr;               // Adam moments
  float* av = nullptr;
  bf16* wb = nullptr;                // BF16 copy of the weights
  // workspaces, grown to the largest call so far and kept until the handle goes
  template <typename V>
  struct Buf {
    V* p = nullptr;
    size_t cap = 0;
    bool grow(size_t n) {
      if (n <= cap) return true;
      if (p) cudaFree(p);
      p = nullptr;
      cap = 0;
      if (cudaMalloc(&p, sizeof(V) * n) != cudaSuccess) {
        cudaGetLastError();  // reported to the caller as FVS_ERR_NOMEM
        p = nullptr;
        return false;
      }
      cap = n;
      return true;
    }
    Buf() = default;
    Buf(const Buf&) = delete;
    Buf& operator=(const Buf&) = delete;
    Buf(Buf&& o) noexcept : p(o.p), cap(o.cap) { o.p = nullptr; o.cap = 0; }
    ~Buf() { if (p) cudaFree(p); }
  };
  std::vector<Buf<bf16>> act;        // act[l]: input of layer l, [rows][din[l]]
  std::vector<Buf<float>> pre;       // pre[l]: layer output before GELU, [rows][dout[l]] (training)
  std::vector<Buf<bf16>> dz;         // dz[l]: loss gradient of pre[l] (training)
  Buf<float> part;                   // partial sums of the parameter gradients
  Buf<float> da;                     // mma.sync engine: gradient of a layer's input
  Buf<float> out;                    // mma.sync engine: last layer's output; prediction rows
  Buf<float> data_x, data_y;         // the call's rows on the device
  Buf<int> data_idx;
  float* loss = nullptr;
  int* gemm_err = nullptr;           // set by a tcgen05 GEMM whose bounded wait expired
  int engine = 0;                    // 0: tcgen05, 1: mma.sync
  int step = 0;
  int nsm = fvs::sm_count();             // multiprocessors of the device
  std::vector<void*> owned;

  ~fvs_mlp() {
    if (stream) cudaStreamSynchronize(stream);
    for (void* p : owned) cudaFree(p);
    if (stream) cudaStreamDestroy(stream);
  }
  int fail(int code, const std::string& m) {
    err = m;
    return code;
  }
  template <typename V>
  V* dalloc(size_t n) {
    void* p = nullptr;
    if (cudaMalloc(&p, sizeof(V) * std::max<size_t>(n, 1)) != cudaSuccess) return nullptr;
    owned.push_back(p);
    if (cudaMemsetAsync(p, 0, sizeof(V) * std::max<size_t>(n, 1), stream) != cudaSuccess) return nullptr;
    return static_cast<V*>(p);
  }
  // layer buffers for `rows` rows; train: those of the backward pass too
  bool ensure_rows(size_t rows, bool train) {
    act.resize(nl);
    pre.resize(nl);
    dz.resize(nl);
    const size_t maxd = (size_t)std::max(*std::max_element(din.begin(), din.end()), *std::max_element(dout.begin(), dout.end()));
    bool ok = true;
    for (int l = 0; l < nl && ok; l++) {
      ok = act[l].grow(rows * din[l]);
      if (ok && train) ok = dz[l].grow(rows * dout[l]);
      if (ok && (engine == 1 || (train && l < nl - 1))) ok = pre[l].grow(rows * dout[l]);
    }
    if (ok && engine == 1 && train) ok = da.grow(rows * maxd);
    return ok;
  }
};

namespace {

// launch in stream order, the kernel's set-up beside its predecessor's tail
// (each waits for it with griddepcontrol.wait before it reads or writes)
template <typename... KArgs, typename... Args>
void launch_tc(void (*kern)(KArgs...), dim3 grid, int threads, size_t smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, args...);
}

template <bool A_KM, bool B_KM, int OUT, int STAGES, int BN>
void gemm_tc_launch(fvs_mlp* m, const tc::GemmArgs& a) {
  const dim3 grid((unsigned)((a.N + BN - 1) / BN), (unsigned)((a.M + tc::BM - 1) / tc::BM));
  launch_tc(tc::k_gemm_tc<A_KM, B_KM, OUT, STAGES, BN>, grid, tc::THREADS, tc::smem_bytes(STAGES, BN), m->stream, a, m->gemm_err);
}

// With more tiles than two per SM the epilogues of some CTAs run beside the
// loads of others, and CTAs with two stages, four to an SM, beat two with four
// (65,536 x 256 x 256 with GELU: 68 / 79 us before the swizzle); below that a
// CTA has only its own blocks in flight.  A hidden layer whose tiles of 128
// columns are still that many reads A half as often with them (prediction of
// 240,000 rows, 256 wide: 686 us, 718 with 64 columns; 112 wide: 365 / 361, so
// not below a whole tile).
constexpr bool wide_tiles(int out) { return out == tc::OUT_GELU; }
template <bool A_KM, bool B_KM, int OUT>
void gemm_tc(fvs_mlp* m, const tc::GemmArgs& a) {
  const long long rows = (a.M + tc::BM - 1) / tc::BM;
  if constexpr (wide_tiles(OUT)) {
    if (a.N >= 128 && rows * ((a.N + 127) / 128) > 2 * m->nsm) return gemm_tc_launch<A_KM, B_KM, OUT, 2, 128>(m, a);
  }
  if (rows * ((a.N + 63) / 64) > 2 * m->nsm) gemm_tc_launch<A_KM, B_KM, OUT, 2, 64>(m, a);
  else gemm_tc_launch<A_KM, B_KM, OUT, 4, 64>(m, a);
}

template <bool A_KM, bool B_KM>
void gemm_mma(fvs_mlp* m, const bf16* A, int lda, const bf16* B, int ldb, int M, int N, int K, int epi,
              const float* bias, float* C, int ldc, bf16* Cact, int ldact) {
  dim3 grid((unsigned)((N + BN - 1) / BN), (unsigned)((M + BM - 1) / BM));
  k_gemm<A_KM, B_KM><<<grid, GEMM_THREADS, 0, m->stream>>>(A, lda, B, ldb, M, N, K, epi, bias, C, ldc, Cact, ldact);
}

// dynamic shared memory of the tcgen05 GEMMs
template <class Kernel>
bool tc_smem(Kernel k, int stages, int bn) {
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, tc::smem_bytes(stages, bn)) == cudaSuccess;
}
template <bool A_KM, bool B_KM, int OUT>
bool tc_smem_all() {
  if constexpr (wide_tiles(OUT)) {
    if (!tc_smem(tc::k_gemm_tc<A_KM, B_KM, OUT, 2, 128>, 2, 128)) return false;
  }
  return tc_smem(tc::k_gemm_tc<A_KM, B_KM, OUT, 2, 64>, 2, 64) && tc_smem(tc::k_gemm_tc<A_KM, B_KM, OUT, 4, 64>, 4, 64);
}
bool tc_gemm_setup() {
  return tc_smem_all<true, true, tc::OUT_GELU>() && tc_smem_all<true, true, tc::OUT_PRED>() &&
         tc_smem_all<true, true, tc::OUT_MSE>() && tc_smem_all<true, false, tc::OUT_DGELU>() &&
         tc_smem(tc::k_grads, 2, tc::GRAD_BN);
}

void refresh_bf16(fvs_mlp* m) { k_f32_to_bf16<<<nblk(m->nparam), 256, 0, m->stream>>>(m->w, m->wb, m->nparam); }

// Forward over n rows already in act[0].  Training (y given): the loss
// gradient of the last layer into dz, the squared errors against rows idx of
// y (null: the first n) added to loss, the hidden layers' pre-activations
// kept.  Otherwise the output's n_out columns into pred.
void forward(fvs_mlp* m, int n, const float* y, const int* idx, float* pred) {
  const int last = m->nl - 1;
  for (int l = 0; l <= last; l++) {
    const int di = m->din[l], dn = m->dout[l];
    const bf16* W = m->wb + m->woff[l];
    const float* bias = m->w + m->boff[l];
    if (m->engine == 1) {
      gemm_mma<true, true>(m, m->act[l].p, di, W, di, n, dn, di, l == last ? EPI_BIAS_F32 : EPI_BIAS_GELU, bias,
                           m->pre[l].p, dn, l == last ? nullptr : m->act[l + 1].p, dn);
      continue;
    }
    tc::GemmArgs a = {};
    a.A = m->act[l].p; a.lda = di;
    a.B = W; a.ldb = di;
    a.M = n; a.N = dn; a.K = di;
    a.bias = bias;
    if (l < last) {
      a.C = y ? m->pre[l].p : nullptr;
      a.H = m->act[l + 1].p;
      gemm_tc<true, true, tc::OUT_GELU>(m, a);
    } else if (y) {
      a.H = m->dz[l].p;
      a.T = y; a.idx = idx; a.nt = m->n_out; a.loss = m->loss;
      gemm_tc<true, true, tc::OUT_MSE>(m, a);
    } else {
      a.C = pred; a.nt = m->n_out;
      gemm_tc<true, true, tc::OUT_PRED>(m, a);
    }
  }
  if (m->engine != 1) return;
  if (y)
    k_mse<<<nblk((size_t)n * m->out_pad), 256, 0, m->stream>>>(m->pre[last].p, m->out_pad, y, idx, n, m->n_out,
                                                              m->dz[last].p, m->out_pad, m->loss);
  else
    k_columns<<<nblk((size_t)n * m->n_out), 256, 0, m->stream>>>(m->pre[last].p, m->out_pad, n, m->n_out, pred);
}

// The runs of K blocks that the parameter gradients are summed in (tc::k_grads).
// A layer's runs are as many as make GRAD_TILES tiles of 128 x 128: their number
// fixes the order of the FP32 sums, and with it the training's trajectory (runs
// five times longer, added in the same order, moved a weight by 5e-5 of the
// weights' norm after 32 steps, through BF16 roundings that fell the other way).
// So it is a constant, near the number of SMs but not bound to the device's.
// A CTA takes as many consecutive runs as leave the launch in one wave of four
// CTAs per SM.
constexpr int GRAD_TILES = 148;
bool grad_plan(fvs_mlp* m, int rows, tc::GradPlan& p) {
  p = tc::GradPlan();
  p.nl = m->nl;
  p.rows = rows;
  const int nk = (rows + tc::BK - 1) / tc::BK;
  size_t off = 0;
  long long tile_runs = 0;
  for (int l = 0; l < m->nl; l++) {
    tc::GradLayer& g = p.l[l];
    g.dZ = m->dz[l].p; g.X = m->act[l].p;
    g.din = m->din[l]; g.dout = m->dout[l];
    g.tiles_n = (g.din + tc::GRAD_BN - 1) / tc::GRAD_BN;
    g.tiles = g.tiles_n * ((g.dout + tc::BM - 1) / tc::BM);
    const int square = ((g.din + 127) / 128) * ((g.dout + 127) / 128);
    g.per = nk;
    if (square < 64 && nk >= 4) {
      const int want = std::max(1, GRAD_TILES / square);
      g.per = std::max(1, (nk + want - 1) / want);
    }
    g.nsplit = (nk + g.per - 1) / g.per;
    tile_runs += (long long)g.tiles * g.nsplit;
    g.w0 = m->woff[l]; g.b0 = m->boff[l];
    g.part = off;
    off += (size_t)g.nsplit * g.din * g.dout + (size_t)g.dout;
  }
  int bias_ctas = 0;
  for (int l = 0; l < m->nl; l++) bias_ctas += (m->dout[l] + tc::BIAS_COLS - 1) / tc::BIAS_COLS;
  const int room = std::max(2 * m->nsm, 4 * m->nsm - bias_ctas);
  p.runs = (int)std::max<long long>(1, (tile_runs + room - 1) / room);
  for (int l = 0; l < m->nl; l++) {
    tc::GradLayer& g = p.l[l];
    g.cta0 = p.gemm_ctas;
    p.gemm_ctas += g.tiles * ((g.nsplit + p.runs - 1) / p.runs);
  }
  p.ctas = p.gemm_ctas;
  for (int l = 0; l < m->nl; l++) {
    p.l[l].bias0 = p.ctas;
    p.ctas += (m->dout[l] + tc::BIAS_COLS - 1) / tc::BIAS_COLS;
  }
  return m->part.grow(off);
}

// Backward from dz of the last layer: the other layers' dz, then the
// parameter gradients: into g, or (adam) straight into Adam's step.
bool backward(fvs_mlp* m, int n, const tc::AdamArgs* adam) {
  for (int l = m->nl - 1; l >= 0; l--) {
    const int di = m->din[l], dn = m->dout[l];
    if (m->engine == 1) {
      // dW_l[n][k] = sum_m dZ[m][n] act_l[m][k]
      gemm_mma<false, false>(m, m->dz[l].p, dn, m->act[l].p, di, dn, di, n, EPI_F32, nullptr, m->g + m->woff[l], di, nullptr, 0);
      k_colsum<<<(dn + 31) / 32, dim3(32, 32), 0, m->stream>>>(m->dz[l].p, n, dn, dn, m->g + m->boff[l]);
    }
    if (l == 0) break;
    // dA_l[m][k] = sum_n dZ[m][n] W_l[n][k]; dZ_{l-1} = dA * gelu'(pre_{l-1})
    if (m->engine == 1) {
      gemm_mma<true, false>(m, m->dz[l].p, dn, m->wb + m->woff[l], di, n, di, dn, EPI_F32, nullptr, m->da.p, di, nullptr, 0);
      k_gelu_back<<<nblk((size_t)n * di), 256, 0, m->stream>>>(m->da.p, m->pre[l - 1].p, m->dz[l - 1].p, (size_t)n * di);
    } else {
      tc::GemmArgs a = {};
      a.A = m->dz[l].p; a.lda = dn;
      a.B = m->wb + m->woff[l]; a.ldb = di;
      a.M = n; a.N = di; a.K = dn;
      a.Z = m->pre[l - 1].p;
      a.H = m->dz[l - 1].p;
      gemm_tc<true, false, tc::OUT_DGELU>(m, a);
    }
  }
  if (m->engine == 1) {
    if (adam) {
      k_adam<<<nblk(m->nparam), 256, 0, m->stream>>>(m->w, m->g, m->am, m->av, m->nparam, adam->lr, adam->b1, adam->b2,
                                                     adam->eps, adam->bc1, adam->bc2);
      refresh_bf16(m);
    }
    return true;
  }
  tc::GradPlan p;
  if (!grad_plan(m, n, p)) return false;
  launch_tc(tc::k_grads, dim3((unsigned)p.ctas), tc::THREADS, tc::smem_bytes(2, tc::GRAD_BN), m->stream, p,
            m->part.p, m->gemm_err);
  if (adam)
    launch_tc(tc::k_finish_grads<true>, dim3(nblk(m->nparam)), 256, 0, m->stream, p, (const float*)m->part.p, m->nparam,
              m->g, m->w, m->am, m->av, m->wb, *adam);
  else
    launch_tc(tc::k_finish_grads<false>, dim3(nblk(m->nparam)), 256, 0, m->stream, p, (const float*)m->part.p, m->nparam,
              m->g, m->w, m->am, m->av, m->wb, tc::AdamArgs());
  return true;
}

// the call's launches and copies are complete when it returns, with or without an error
int check(fvs_mlp* m, const char* where) {
  cudaError_t e = cudaGetLastError();
  const cudaError_t es = cudaStreamSynchronize(m->stream);
  if (e == cudaSuccess) e = es;
  if (e != cudaSuccess) return m->fail(FVS_ERR_CUDA, std::string(where) + ": " + cudaGetErrorString(e));
  int flag = 0;
  e = cudaMemcpy(&flag, m->gemm_err, sizeof flag, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return m->fail(FVS_ERR_CUDA, std::string(where) + ": " + cudaGetErrorString(e));
  if (flag) return m->fail(FVS_ERR_TIMEOUT, std::string(where) + ": a tensor-core GEMM wait ran out of its budget");
  return FVS_OK;
}

// an allocation of a call that has copies from the caller's arrays in flight failed
int fail_in_flight(fvs_mlp* m, const char* what) {
  cudaStreamSynchronize(m->stream);
  return m->fail(FVS_ERR_NOMEM, what);
}

}  // namespace

extern "C" {

int fvs_mlp_create(int32_t n_in, int32_t width, int32_t depth, int32_t n_out, uint64_t seed, fvs_mlp** out) {
  if (!out) return FVS_ERR_INVALID;
  *out = nullptr;
  if (n_in <= 0 || n_in > 64 || width <= 0 || width > 1024 || width % 16 || depth < 1 || depth > 16 || n_out <= 0 ||
      n_out > 64) {
    g_mlp_error = "MLP sizes: 1 <= n_in, n_out <= 64; width a multiple of 16 up to 1024; 1 <= depth <= 16";
    return FVS_ERR_INVALID;
  }
  std::unique_ptr<fvs_mlp> m(new fvs_mlp());
  m->n_in = n_in; m->width = width; m->depth = depth; m->n_out = n_out;
  m->in_pad = pad16(n_in);
  m->out_pad = pad16(n_out);
  m->nl = depth + 1;
  for (int l = 0; l < m->nl; l++) {
    m->din.push_back(l == 0 ? m->in_pad : width);
    m->dout.push_back(l == m->nl - 1 ? m->out_pad : width);
  }
  size_t off = 0;
  for (int l = 0; l < m->nl; l++) {
    m->woff.push_back(off);
    off += (size_t)m->din[l] * m->dout[l];
    m->boff.push_back(off);
    off += m->dout[l];
  }
  m->nparam = off;
  if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess) {
    g_mlp_error = "cudaStreamCreate failed";
    return FVS_ERR_CUDA;
  }
  if (!tc_gemm_setup()) {
    g_mlp_error = "tensor-core GEMM setup (dynamic shared memory) failed";
    return FVS_ERR_CUDA;
  }
  m->w = m->dalloc<float>(off);
  m->g = m->dalloc<float>(off);
  m->am = m->dalloc<float>(off);
  m->av = m->dalloc<float>(off);
  m->wb = m->dalloc<bf16>(off);
  m->loss = m->dalloc<float>(4);
  m->gemm_err = m->dalloc<int>(4);
  if (!m->w || !m->g || !m->am || !m->av || !m->wb || !m->loss || !m->gemm_err) {
    g_mlp_error = "MLP device allocation failed";
    return FVS_ERR_NOMEM;
  }
  // He-style init (seeded), zero biases; padded rows/columns stay zero
  std::vector<float> h(off, 0.f);
  std::mt19937_64 rng(seed);
  for (int l = 0; l < m->nl; l++) {
    const int fan_in = l == 0 ? n_in : width, rows = l == m->nl - 1 ? n_out : width;
    std::normal_distribution<float> nd(0.f, std::sqrt(2.f / fan_in));
    for (int r = 0; r < rows; r++)
      for (int k = 0; k < fan_in; k++) h[m->woff[l] + (size_t)r * m->din[l] + k] = nd(rng);
  }
  cudaMemcpyAsync(m->w, h.data(), 4 * off, cudaMemcpyHostToDevice, m->stream);
  refresh_bf16(m.get());
  if (check(m.get(), "MLP init")) {
    g_mlp_error = m->err;
    return FVS_ERR_CUDA;
  }
  *out = m.release();
  return FVS_OK;
}

void fvs_mlp_destroy(fvs_mlp* m) { delete m; }

const char* fvs_mlp_last_error(const fvs_mlp* m) { return m ? m->err.c_str() : g_mlp_error.c_str(); }

// number of parameters in the unpadded layout: per layer W[out][in], b[out]
int fvs_mlp_num_params(const fvs_mlp* m, int64_t* n) {
  if (!m || !n) return FVS_ERR_INVALID;
  int64_t s = 0;
  for (int l = 0; l < m->nl; l++) {
    const int i = l == 0 ? m->n_in : m->width, o = l == m->nl - 1 ? m->n_out : m->width;
    s += (int64_t)i * o + o;
  }
  *n = s;
  return FVS_OK;
}

int fvs_mlp_set_engine(fvs_mlp* m, int32_t engine) {
  if (!m || engine < 0 || engine > 1) return FVS_ERR_INVALID;
  m->engine = engine;
  return FVS_OK;
}

static int copy_params(fvs_mlp* m, float* host, const float* in, int64_t n, bool get, const float* dev_src) {
  int64_t need = 0;
  fvs_mlp_num_params(m, &need);
  if (n < need) return m->fail(FVS_ERR_INVALID, "parameter buffer too small");
  std::vector<float> pad(m->nparam, 0.f);
  if (get && cudaMemcpy(pad.data(), dev_src, 4 * m->nparam, cudaMemcpyDeviceToHost) != cudaSuccess)
    return m->fail(FVS_ERR_CUDA, "parameter download");
  int64_t p = 0;
  for (int l = 0; l < m->nl; l++) {
    const int i = l == 0 ? m->n_in : m->width, o = l == m->nl - 1 ? m->n_out : m->width;
    for (int r = 0; r < o; r++)
      for (int k = 0; k < i; k++, p++) {
        float& dst = pad[m->woff[l] + (size_t)r * m->din[l] + k];
        if (get) host[p] = dst; else dst = in[p];
      }
    for (int r = 0; r < o; r++, p++) {
      float& dst = pad[m->boff[l] + r];
      if (get) host[p] = dst; else dst = in[p];
    }
  }
  if (!get) {
    // (check() waits for the copy)
    cudaMemcpyAsync(m->w, pad.data(), 4 * m->nparam, cudaMemcpyHostToDevice, m->stream);
    cudaMemsetAsync(m->am, 0, 4 * m->nparam, m->stream);
    cudaMemsetAsync(m->av, 0, 4 * m->nparam, m->stream);
    m->step = 0;
    refresh_bf16(m);
    return check(m, "set_params");
  }
  return FVS_OK;
}

int fvs_mlp_get_params(fvs_mlp* m, float* dst, int64_t n) {
  if (!m || !dst) return FVS_ERR_INVALID;
  return copy_params(m, dst, nullptr, n, true, m->w);
}

int fvs_mlp_set_params(fvs_mlp* m, const float* src, int64_t n) {
  if (!m || !src) return FVS_ERR_INVALID;
  return copy_params(m, nullptr, src, n, false, nullptr);
}

// loss and parameter gradients of one batch (no update), for checking
int fvs_mlp_loss_grad(fvs_mlp* m, const float* x, const float* y, int32_t n, float* loss, float* grads) {
  if (!m || !x || !y || n <= 0) return FVS_ERR_INVALID;
  if (!m->ensure_rows(n, true)) return m->fail(FVS_ERR_NOMEM, "activation allocation");
  if (!m->data_x.grow((size_t)n * m->n_in) || !m->data_y.grow((size_t)n * m->n_out))
    return m->fail(FVS_ERR_NOMEM, "batch allocation");
  cudaMemcpyAsync(m->data_x.p, x, 4 * (size_t)n * m->n_in, cudaMemcpyHostToDevice, m->stream);
  cudaMemcpyAsync(m->data_y.p, y, 4 * (size_t)n * m->n_out, cudaMemcpyHostToDevice, m->stream);
  cudaMemsetAsync(m->loss, 0, 4, m->stream);
  if (m->engine == 1) cudaMemsetAsync(m->g, 0, 4 * m->nparam, m->stream);
  k_gather_rows<<<nblk((size_t)n * m->in_pad), 256, 0, m->stream>>>(m->data_x.p, m->n_in, nullptr, n, m->act[0].p, m->in_pad);
  forward(m, n, m->data_y.p, nullptr, nullptr);
  if (!backward(m, n, nullptr)) return fail_in_flight(m, "gradient workspace");
  int rc = check(m, "loss_grad");
  if (rc) return rc;
  float l = 0.f;
  cudaMemcpy(&l, m->loss, 4, cudaMemcpyDeviceToHost);
  if (loss) *loss = l / float(n * m->n_out);
  if (grads) {
    int64_t np = 0;
    fvs_mlp_num_params(m, &np);
    rc = copy_params(m, grads, nullptr, np, true, m->g);
  }
  return rc;
}

// minibatch Adam; loss_per_epoch[epochs] (mean squared error of the epoch)
int fvs_mlp_train(fvs_mlp* m, const float* x, const float* y, int64_t n, int32_t batch, int32_t epochs, float lr,
                  uint64_t seed, float* loss_per_epoch) {
  if (!m || !x || !y || n <= 0 || batch <= 0 || epochs <= 0 || n > (int64_t)1 << 31) return FVS_ERR_INVALID;
  batch = (int)std::min<int64_t>(batch, n);
  if (!m->ensure_rows(batch, true)) return m->fail(FVS_ERR_NOMEM, "activation allocation");
  if (!m->data_x.grow((size_t)n * m->n_in) || !m->data_y.grow((size_t)n * m->n_out) || !m->data_idx.grow((size_t)n))
    return m->fail(FVS_ERR_NOMEM, "dataset allocation");
  // Orders of the even and of the odd epochs: one is written while the copy of
  // the other may still be in flight (an asynchronous copy from pageable memory
  // may read it after the call has returned); check() ends every epoch.
  std::vector<int> order[2];
  try {
    order[0].resize((size_t)n);
    if (epochs > 1) order[1].resize((size_t)n);
  } catch (const std::bad_alloc&) {
    return m->fail(FVS_ERR_NOMEM, "sample order");
  }
  cudaMemcpyAsync(m->data_x.p, x, 4 * (size_t)n * m->n_in, cudaMemcpyHostToDevice, m->stream);
  cudaMemcpyAsync(m->data_y.p, y, 4 * (size_t)n * m->n_out, cudaMemcpyHostToDevice, m->stream);
  std::mt19937_64 rng(seed);
  auto shuffle = [&](std::vector<int>& idx) {
    for (int64_t i = 0; i < n; i++) idx[i] = (int)i;
    std::shuffle(idx.begin(), idx.end(), rng);
  };
  shuffle(order[0]);
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  for (int ep = 0; ep < epochs; ep++) {
    cudaMemcpyAsync(m->data_idx.p, order[ep & 1].data(), 4 * (size_t)n, cudaMemcpyHostToDevice, m->stream);
    cudaMemsetAsync(m->loss, 0, 4, m->stream);
    for (int64_t s0 = 0; s0 + batch <= n; s0 += batch) {
      const int* bi = m->data_idx.p + s0;
      k_gather_rows<<<nblk((size_t)batch * m->in_pad), 256, 0, m->stream>>>(m->data_x.p, m->n_in, bi, batch, m->act[0].p,
                                                                            m->in_pad);
      forward(m, batch, m->data_y.p, bi, nullptr);
      m->step++;
      const tc::AdamArgs ad = {lr, b1, b2, eps, 1.f - std::pow(b1, (float)m->step), 1.f - std::pow(b2, (float)m->step)};
      if (!backward(m, batch, &ad)) return fail_in_flight(m, "gradient workspace");
    }
    if (ep + 1 < epochs) shuffle(order[(ep + 1) & 1]);  // the next epoch's order, beside this epoch's steps
    int rc = check(m, "train");
    if (rc) return rc;
    if (loss_per_epoch) {
      float l = 0.f;
      cudaMemcpy(&l, m->loss, 4, cudaMemcpyDeviceToHost);
      loss_per_epoch[ep] = l / float((n / batch) * batch * m->n_out);
    }
  }
  return FVS_OK;
}

int fvs_mlp_predict(fvs_mlp* m, const float* x, int64_t n, float* y) {
  if (!m || !x || !y || n <= 0) return FVS_ERR_INVALID;
  const int chunk = (int)std::min<int64_t>(n, 65536);
  if (!m->ensure_rows(chunk, false)) return m->fail(FVS_ERR_NOMEM, "activation allocation");
  if (!m->data_x.grow((size_t)chunk * m->n_in) || !m->out.grow((size_t)chunk * m->n_out))
    return m->fail(FVS_ERR_NOMEM, "batch allocation");
  for (int64_t s0 = 0; s0 < n; s0 += chunk) {
    const int c = (int)std::min<int64_t>(chunk, n - s0);
    cudaMemcpyAsync(m->data_x.p, x + s0 * m->n_in, 4 * (size_t)c * m->n_in, cudaMemcpyHostToDevice, m->stream);
    k_gather_rows<<<nblk((size_t)c * m->in_pad), 256, 0, m->stream>>>(m->data_x.p, m->n_in, nullptr, c, m->act[0].p, m->in_pad);
    forward(m, c, nullptr, nullptr, m->out.p);
    cudaMemcpyAsync(y + s0 * m->n_out, m->out.p, 4 * (size_t)c * m->n_out, cudaMemcpyDeviceToHost, m->stream);
  }
  return check(m, "predict");
}

}  // extern "C"
