// fvs_tcgemm.cuh — BF16 GEMM on the 5th-generation tensor cores (tcgen05),
// FP32 accumulation in tensor memory:  C[m][n] = sum_k A(m,k) B(n,k).
//
// Operands are K-major (row m at A + m*lda) or MN-major (element (m,k) at A +
// k*lda + m), as in the mma.sync GEMM of fvs_mlp.cu.  Leading dimensions and
// the contiguous extents are multiples of 16 elements and the bases 16-byte
// aligned (the padded layers of fvs_mlp.cu), so every 16-byte chunk lies
// wholly inside or outside its matrix.
//
// CTA tile 128 x 64 or 128 x 128, K in blocks of 64 over two or four shared-
// memory stages (49, 65 or 97 KB).  256 threads (8 warps):
//   - all threads bring the next blocks in with 16-byte cp.async, one or three
//     blocks ahead, straight into the tensor core's canonical layouts with the
//     128-byte swizzle (stage_block); chunks outside the matrix are zero-filled;
//   - thread 0 issues the MMAs (tcgen05.mma.cta_group::1.kind::f16, M 128,
//     N 64 or 128, K 16) and commits them to the stage's mbarrier, which frees it;
//   - warp w reads the accumulator rows of tensor-memory lanes 32 (w % 4)..,
//     32 columns from 32 (w / 4), of the wider tile also 64 further on
//     (tcgen05.ld): a thread holds 32 consecutive columns of one row, applies
//     the epilogue and stores 32-byte vectors.
// The MLP's layers are 256 wide: with tiles of 128 x 128, two K stages filled
// between barriers and one warpgroup, a 4096 x 256 x 256 layer ran on 64 CTAs
// in 48 us, most of it waiting on loads and in the epilogue of 128 outputs a
// thread; 128 CTAs of 32 outputs a thread take 7.7 us (10.3 before the swizzle).
// Every mbarrier wait is bounded (clock64 budget).  On expiry the kernel sets
// *err, skips the remaining K blocks and the epilogue, waits for the MMAs it
// already issued (bounded, up to 9 budgets in all), frees its tensor memory
// and returns.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace tc {

typedef __nv_bfloat16 bf16;

constexpr int BM = 128, BK = 64, THREADS = 256;
constexpr int A_BYTES = BM * BK * 2;  // one stage of A: 16 KB; of B: 8 KB per 64 columns
constexpr int smem_bytes(int stages, int bn) { return stages * (A_BYTES + bn * BK * 2) + 1024; }
constexpr long long WAIT_BUDGET = 4000000000ll;              // clock cycles (~2 s at 2 GHz)

// Shared-memory matrix descriptors: start address >> 4 (bits 0-13), leading
// byte offset >> 4 (bits 16-29), stride byte offset >> 4 (bits 32-45),
// descriptor version 1 (bits 46-47), 128-byte swizzle (mode 2 in bits 61-63).
// Both majors keep atoms of 8 lines of 128 bytes, the 16-byte chunk c of line l
// at c ^ l:
//  K-major: a line is 64 K of a row; groups of 8 rows 1024 bytes apart (stride
//  offset), a 16-wide K step 32 bytes on.
//  MN-major: a line is 64 rows of one k; groups of 8 k 1024 bytes apart (stride
//  offset), blocks of 64 rows 8192 bytes apart (leading offset), a 16-wide K
//  step 2048 bytes on.
template <bool KMAJOR>
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(KMAJOR ? 1 : 8192 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// Instruction descriptor of kind::f16: D FP32 (bits 4-5 = 1), A BF16 (bits 7-9
// = 1), B BF16 (bits 10-12 = 1), no negation, bit 15 / 16: A / B MN-major,
// N >> 3 (bits 17-22), M >> 4 (bits 24-28).
template <bool A_KM, bool B_KM, int BN>
__host__ __device__ constexpr uint32_t idesc() {
  return (1u << 4) | (1u << 7) | (1u << 10) | (A_KM ? 0u : 1u << 15) | (B_KM ? 0u : 1u << 16) |
         ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  while (true) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if (clock64() - t0 > WAIT_BUDGET) return false;
  }
}

// cp.async of 16 bytes; bytes = 0 fills with zeros and reads nothing
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// One operand's block of R rows (M or N) x 64 K into shared memory, laid out as
// its descriptor says, in copies of 16 bytes: K-major, 8 consecutive k of a row;
// MN-major, 8 consecutive rows of one k.  A warp's copies are four lines of 128
// contiguous bytes, and the swizzle spreads them over all banks.  (Without the
// swizzle a line was 64 bytes: a layer of 65,536 rows and 256 outputs took
// 60.5 us against 36.2, all weight gradients of a batch of 4,096 23.3 against
// 17.3.)
template <bool KMAJOR, int R>
__device__ __forceinline__ void stage_block(uint32_t s, const bf16* g, int ld, int row0, int rows, int k0, int K) {
#pragma unroll
  for (int q = 0; q < R * 8 / THREADS; q++) {
    const int i = q * THREADS + (int)threadIdx.x, c = i & 7, l = i >> 3;
    // line l: row l (K-major), or k l % 64 of the block l / 64 of 64 rows
    const int r = KMAJOR ? l : ((l >> 6) << 6) + (c << 3), k = KMAJOR ? c << 3 : l & 63;
    const bool in = row0 + r < rows && k0 + k < K;
    const bf16* src = KMAJOR ? g + (size_t)(row0 + r) * ld + (k0 + k) : g + (size_t)(k0 + k) * ld + (row0 + r);
    cp_async16(s + l * 128 + ((c ^ (l & 7)) << 4), in ? src : g, in ? 16u : 0u);
  }
}

__device__ __forceinline__ float gelu_tc(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad_tc(float z) {
  return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

// What becomes of the accumulator:
//  OUT_RAW   C = acc (a split-K partial)
//  OUT_PRED  C = acc + bias, the first nt columns only (ld nt)
//  OUT_GELU  z = acc + bias; C = z (where C is given), H = BF16(GELU(z))
//  OUT_MSE   z = acc + bias against the targets T[idx[m]][0..nt) (idx null: T[m]): H = BF16(2 (z - T) / (rows nt)),
//            the squared errors added to *loss
//  OUT_DGELU H = BF16(acc * GELU'(Z))
enum Out : int { OUT_RAW = 0, OUT_PRED = 1, OUT_GELU = 2, OUT_MSE = 3, OUT_DGELU = 4 };

struct GemmArgs {
  const bf16* A;
  const bf16* B;
  int lda, ldb, M, N, K;
  const float* bias;
  float* C;        // ld N (rows of N columns)
  bf16* H;         // ld N
  const float* Z;  // ld N
  const float* T;
  const int* idx;
  int nt;
  float* loss;
};

// 32-byte accesses (a thread's columns are one row's, so a warp's access
// touches 32 rows: the wider it is, the fewer passes it takes)
__device__ __forceinline__ void ld8(const float* p, float* v) {
  asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
               : "l"(p));
}
__device__ __forceinline__ void st8(float* p, const float* v) {
  asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]),
               "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}

// `ncol` (a multiple of 16, at most 32) of a thread's 32 columns; rows and
// columns start at multiples of 32 bytes
__device__ __forceinline__ void store_f32(float* p, const float* v, int ncol) {
#pragma unroll
  for (int j = 0; j < 4; j++)
    if (8 * j < ncol) st8(p + 8 * j, v + 8 * j);
}
__device__ __forceinline__ void store_bf16(bf16* p, const float* v, int ncol) {
#pragma unroll
  for (int j = 0; j < 2; j++)
    if (16 * j < ncol) {
      uint32_t h[8];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const __nv_bfloat162 q = __floats2bfloat162_rn(v[16 * j + 2 * i], v[16 * j + 2 * i + 1]);
        h[i] = *reinterpret_cast<const uint32_t*>(&q);
      }
      asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"l"(p + 16 * j), "r"(h[0]), "r"(h[1]), "r"(h[2]),
                   "r"(h[3]), "r"(h[4]), "r"(h[5]), "r"(h[6]), "r"(h[7])
                   : "memory");
    }
}

// One 128 x BN output tile at (m0, n0) over the K blocks [kb0, kb0 + nk).
// OUT_RAW sums each run of `per` blocks by itself: the accumulators of the
// runs lie in two halves of the CTA's tensor memory in turn, so a run's partial
// goes out (to C, C + run, ...) beside the next one's MMAs.
template <bool A_KM, bool B_KM, int OUT, int STAGES, int BN>
__device__ __forceinline__ void gemm_tile(const GemmArgs& a, int m0, int n0, int kb0, int nk, int per, size_t run,
                                          int* err) {
  constexpr int B_BYTES = BN * BK * 2;
  constexpr uint32_t TMEM_COLS = OUT == OUT_RAW ? 2 * BN : BN;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(8) uint64_t mbar[STAGES];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_ok;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t sbase = (smem_u32(smem) + 1023u) & ~1023u;  // the swizzle works on address bits

  if (tid == 0) {
#pragma unroll
    for (int s = 0; s < STAGES; s++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&mbar[s])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    s_ok = 1;
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = tmem_slot;
  // set up so far beside the tail of the kernel before; its results from here
  asm volatile("griddepcontrol.wait;" ::: "memory");

  auto load = [&](int kb) {  // one commit group per call, empty past the last block
    if (kb < nk) {
      const uint32_t s = sbase + (uint32_t)(kb % STAGES) * (A_BYTES + B_BYTES);
      stage_block<A_KM, BM>(s, a.A, a.lda, m0, a.M, (kb0 + kb) * BK, a.K);
      stage_block<B_KM, BN>(s + A_BYTES, a.B, a.ldb, n0, a.N, (kb0 + kb) * BK, a.K);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
#pragma unroll
  for (int kb = 0; kb < STAGES - 1; kb++) load(kb);
  // the accumulator of this warp's 32 rows and 32 columns
  const int c0 = (warp >> 2) * 32;  // and 64 columns further on for wider tiles
  auto read_acc = [&](uint32_t acc, int c0, uint32_t* u) {
    const uint32_t taddr = acc + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0;
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]),
          "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15]),
          "=r"(u[16]), "=r"(u[17]), "=r"(u[18]), "=r"(u[19]), "=r"(u[20]), "=r"(u[21]), "=r"(u[22]), "=r"(u[23]),
          "=r"(u[24]), "=r"(u[25]), "=r"(u[26]), "=r"(u[27]), "=r"(u[28]), "=r"(u[29]), "=r"(u[30]), "=r"(u[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
  };
  const int m = m0 + (warp & 3) * 32 + lane;
  // the partial of run r, once its MMAs are complete
  auto store_run = [&](int r) {
    uint32_t u[32];
    read_acc(tmem + (uint32_t)(r & 1) * BN, c0, u);
    const int n = n0 + c0, ncol = min(32, a.N - n);
    if (m < a.M && ncol > 0)
      store_f32(a.C + (size_t)r * run + (size_t)m * a.N + n, reinterpret_cast<const float*>(u), ncol);
  };
  int issued = -1;  // last K block whose MMAs thread 0 committed
  for (int kb = 0; kb < nk; kb++) {
    // block kb has arrived (all but the newest STAGES - 2 groups)
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const uint32_t a0 = sbase + (uint32_t)(kb % STAGES) * (A_BYTES + B_BYTES), b0 = a0 + A_BYTES;
      const int steps = min(BK / 16, (a.K - (kb0 + kb) * BK + 15) / 16);
      for (int kk = 0; kk < steps; kk++) {
        const uint64_t ad = smem_desc<A_KM>(a0 + kk * (A_KM ? 32 : 2048)), bd = smem_desc<B_KM>(b0 + kk * (B_KM ? 32 : 2048));
        const uint32_t acc = ((OUT == OUT_RAW ? kb % per > 0 : kb > 0) || kk > 0) ? 1u : 0u;
        const uint32_t dst = OUT == OUT_RAW ? tmem + (uint32_t)((kb / per) & 1) * BN : tmem;
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(dst),
            "l"(ad), "l"(bd), "r"(idesc<A_KM, B_KM, BN>()), "r"(acc)
            : "memory");
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                       smem_u32(&mbar[kb % STAGES]))
                   : "memory");
      issued = kb;
    }
    // block kb + STAGES - 1 goes where block kb - 1 was: wait for that block's MMAs;
    // a run's partial goes out after the next run's first block was issued
    const bool run_done = OUT == OUT_RAW && kb > 0 && kb % per == 0;
    if ((kb + STAGES - 1 < nk || run_done) && kb > 0) {
      if (tid == 0 && !mbar_wait(smem_u32(&mbar[(kb - 1) % STAGES]), (uint32_t)(((kb - 1) / STAGES) & 1))) s_ok = 0;
      __syncthreads();
      if (!s_ok) break;
    }
    load(kb + STAGES - 1);
    if (OUT == OUT_RAW && run_done) {
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      store_run(kb / per - 1);
      // (the accumulator is written again one run later, after further block barriers)
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    }
  }
  // the successor may be scheduled beside the epilogue (it waits for this
  // grid's results)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // No copy may land in shared memory after the CTA has exited (an early
  // break leaves groups in flight)
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  // Every MMA this CTA issued must be complete before its tensor memory is
  // read or freed, and before the CTA exits (the MMAs read the operand
  // stages in shared memory).  The commit of the last issued block tracks
  // all earlier MMAs of thread 0, so one wait on it covers them all; this
  // wait also runs after an earlier wait ran out (s_ok == 0, loop left
  // early).  The MMAs' operands are staged and nothing else gates them, so
  // the tensor core completes them; only a GPU stalled for the whole budget
  // makes the wait expire.  Then it is repeated with 8 times the budget, and
  // the CTA frees its tensor memory only after that: freeing it earlier could
  // let a later CTA's accumulator receive these MMAs' writes.
  if (tid == 0 && issued >= 0) {
    const uint32_t fb = smem_u32(&mbar[issued % STAGES]), fp = (uint32_t)((issued / STAGES) & 1);
    if (!mbar_wait(fb, fp)) {
      s_ok = 0;
      for (int r = 0; r < 8 && !mbar_wait(fb, fp); r++) {
      }
    }
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  if (s_ok && OUT == OUT_RAW) {
    if (nk > 0) store_run((nk - 1) / per);
  } else if (s_ok) {
    float e2 = 0.f;
#pragma unroll 1
    for (int cc = c0; cc < BN; cc += 64) {
      uint32_t u[32];
      read_acc(tmem, cc, u);
      const int n = n0 + cc;
      const int ncol = min(32, a.N - n);  // a multiple of 16; <= 0: columns past the matrix
      float v[32];
#pragma unroll
      for (int j = 0; j < 32; j++) v[j] = __uint_as_float(u[j]);
      if (m < a.M && ncol > 0) {
        const size_t at = (size_t)m * a.N + n;
        if (OUT == OUT_PRED || OUT == OUT_GELU || OUT == OUT_MSE) {
#pragma unroll
          for (int j = 0; j < 32; j++)
            if (j < ncol) v[j] += a.bias[n + j];
        }
        if (OUT == OUT_GELU && a.C) store_f32(a.C + at, v, ncol);
        if (OUT == OUT_PRED) {
#pragma unroll
          for (int j = 0; j < 32; j++)
            if (n + j < a.nt) a.C[(size_t)m * a.nt + n + j] = v[j];
        }
        if (OUT == OUT_GELU) {
#pragma unroll
          for (int j = 0; j < 32; j++) v[j] = gelu_tc(v[j]);
          store_bf16(a.H + at, v, ncol);
        }
        if (OUT == OUT_MSE) {
          const float* t = a.T + (size_t)(a.idx ? a.idx[m] : m) * a.nt;
#pragma unroll
          for (int j = 0; j < 32; j++) {
            float d = 0.f;
            if (n + j < a.nt) {
              d = v[j] - t[n + j];
              e2 += d * d;
            }
            v[j] = 2.f * d / float(a.M * a.nt);
          }
          store_bf16(a.H + at, v, ncol);
        }
        if (OUT == OUT_DGELU) {
          float z[32];
#pragma unroll
          for (int j = 0; j < 32; j++) z[j] = 0.f;
#pragma unroll
          for (int j = 0; j < 4; j++)
            if (8 * j < ncol) ld8(a.Z + at + 8 * j, z + 8 * j);
#pragma unroll
          for (int j = 0; j < 32; j++) v[j] = v[j] * gelu_grad_tc(z[j]);
          store_bf16(a.H + at, v, ncol);
        }
      }
    }
    if (OUT == OUT_MSE) {
      for (int o = 16; o > 0; o >>= 1) e2 += __shfl_down_sync(0xffffffffu, e2, o);
      if (lane == 0 && e2 != 0.f) atomicAdd(a.loss, e2);
    }
  } else if (tid == 0) {
    atomicExch(err, 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

// one GEMM: a CTA per 128 x BN tile (x along N)
template <bool A_KM, bool B_KM, int OUT, int STAGES, int BN>
__global__ void __launch_bounds__(THREADS, BN == 128 ? 3 : STAGES == 2 ? (OUT == OUT_DGELU ? 3 : 4) : 2)
    k_gemm_tc(const GemmArgs a, int* __restrict__ err) {
  gemm_tile<A_KM, B_KM, OUT, STAGES, BN>(a, (int)blockIdx.y * BM, (int)blockIdx.x * BN, 0, (a.K + BK - 1) / BK, 1, 0, err);
}

// All weight gradients of a network, dW_l[n][k] = sum_m dZ_l[m][n] X_l[m][k],
// and bias gradients, db_l[n] = sum_m dZ_l[m][n], in one launch.  K is the
// batch: a layer's K blocks are summed in runs of `per`, and the runs' partial
// sums added in order by k_finish_grads (deterministic).  A CTA takes `runs`
// consecutive runs of one 128 x 64 tile; a bias CTA 32 columns of one layer's
// dZ, each column in 32 interleaved row sums added in order.
constexpr int MAX_LAYERS = 17, BIAS_COLS = 32, GRAD_BN = 64;
struct GradLayer {
  const bf16* dZ;  // [rows][dout]
  const bf16* X;   // [rows][din]
  int din, dout;
  int tiles_n, tiles;  // tiles along din, and in all
  int per, nsplit;     // K blocks of a run, runs
  int cta0, bias0;     // first CTA of the layer's tiles, and of its bias columns
  size_t part;         // offset of its partial sums: [nsplit][dout][din], then db[dout]
  size_t w0, b0;       // its weights and biases in the parameter vector
};
struct GradPlan {
  int nl, rows, runs;
  int gemm_ctas, ctas;
  GradLayer l[MAX_LAYERS];
};

__global__ void __launch_bounds__(THREADS, 4) k_grads(const GradPlan p, float* __restrict__ part, int* __restrict__ err) {
  const int b = (int)blockIdx.x;
  if (b < p.gemm_ctas) {
    int l = 0;
    while (l + 1 < p.nl && b >= p.l[l + 1].cta0) l++;
    const GradLayer& g = p.l[l];
    const int i = b - g.cta0, tile = i % g.tiles, z = i / g.tiles * p.runs;
    GemmArgs a = {};
    a.A = g.dZ; a.lda = g.dout; a.M = g.dout;
    a.B = g.X; a.ldb = g.din; a.N = g.din;
    a.K = p.rows;
    const size_t run = (size_t)g.dout * g.din;
    a.C = part + g.part + (size_t)z * run;
    const int nk = (p.rows + BK - 1) / BK, kb0 = z * g.per;
    gemm_tile<false, false, OUT_RAW, 2, GRAD_BN>(a, tile / g.tiles_n * BM, tile % g.tiles_n * GRAD_BN, kb0,
                                     max(0, min(nk - kb0, p.runs * g.per)), g.per, run, err);
    return;
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  int l = 0;
  while (l + 1 < p.nl && b >= p.l[l + 1].bias0) l++;
  const GradLayer& g = p.l[l];
  extern __shared__ __align__(128) uint8_t smem[];
  float(*sh)[BIAS_COLS] = reinterpret_cast<float(*)[BIAS_COLS]>(smem);  // [32][32]
  const int col0 = (b - g.bias0) * BIAS_COLS, c = col0 + 4 * ((int)threadIdx.x & 7), ty = (int)threadIdx.x >> 3;
  float s[4] = {0.f, 0.f, 0.f, 0.f};
  if (c < g.dout) {
#pragma unroll 16
    for (int r = ty; r < p.rows; r += 32) {
      const uint2 q = *reinterpret_cast<const uint2*>(g.dZ + (size_t)r * g.dout + c);
      const bf16* h = reinterpret_cast<const bf16*>(&q);
#pragma unroll
      for (int j = 0; j < 4; j++) s[j] += __bfloat162float(h[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < 4; j++) sh[ty][c - col0 + j] = s[j];
  __syncthreads();
  const int o = col0 + (int)threadIdx.x;
  if (threadIdx.x < BIAS_COLS && o < g.dout) {
    float t = 0.f;
    for (int q = 0; q < 32; q++) t += sh[q][threadIdx.x];
    part[g.part + (size_t)g.nsplit * g.dout * g.din + o] = t;
  }
}

// Adam's constants of a step (bc1, bc2: bias corrections 1 - beta^step)
struct AdamArgs {
  float lr, b1, b2, eps, bc1, bc2;
};

// Gradient of every parameter from its partial sums, added in order; with
// ADAM also the update of the moments, the FP32 parameters and their BF16 copy.
template <bool ADAM>
__global__ void __launch_bounds__(256) k_finish_grads(const GradPlan p, const float* __restrict__ part, size_t n,
                                                      float* __restrict__ grad, float* __restrict__ w,
                                                      float* __restrict__ am, float* __restrict__ av,
                                                      bf16* __restrict__ wb, AdamArgs ad) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int l = 0;
  while (l + 1 < p.nl && i >= p.l[l + 1].w0) l++;
  const GradLayer& g = p.l[l];
  const size_t nw = (size_t)g.dout * g.din;
  float gi = 0.f;
  if (i < g.b0) {
    const float* s = part + g.part + (i - g.w0);
#pragma unroll 16
    for (int z = 0; z < g.nsplit; z++) gi += s[z * nw];
  } else {
    gi = part[g.part + (size_t)g.nsplit * nw + (i - g.b0)];
  }
  if (!ADAM) {
    grad[i] = gi;
    return;
  }
  const float mi = ad.b1 * am[i] + (1.f - ad.b1) * gi;
  const float vi = ad.b2 * av[i] + (1.f - ad.b2) * gi * gi;
  am[i] = mi;
  av[i] = vi;
  const float wi = w[i] - ad.lr * (mi / ad.bc1) / (sqrtf(vi / ad.bc2) + ad.eps);
  w[i] = wi;
  wb[i] = __float2bfloat16(wi);
}

}  // namespace tc
