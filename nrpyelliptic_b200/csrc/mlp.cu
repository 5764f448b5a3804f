// Learned initial guess: a small MLP (puncture parameters -> POD coefficients
// of uu) trained and evaluated on the GPU with BF16 matrix products on the
// fifth-generation tensor cores (tcgen05.mma, FP32 accumulators in tensor
// memory), FP32 master weights and Adam; plus the POD reconstruction of the
// guess.
//
// Every matrix product of the network -- forward Z = H W, backward
// dH = dZ W^T and dW = H^T dZ -- runs in one kernel, k_gemm_tc.  Operands are
// rounded to BF16 once, by the kernel that produces them, and stored in both
// orientations, so that every product reads both operands with the summed
// index contiguous: 16-byte asynchronous copies go straight into the tensor
// cores' shared-memory layout.  What follows a product elementwise (bias, tanh,
// the loss and its derivative, the tanh derivative) runs in its epilogue, and
// the products and column sums of one backward layer share a launch: a
// minibatch is 12 launches.
#include <cuda_bf16.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <vector>

#include "common.cuh"

namespace nrpyell {

namespace {

// ------------------------------------------------------------------ GEMM
// C[M x N] = A[M x K] B[K x N] with A(m,k) = A[m*lda + k] and B(k,n) =
// B[n*ldb + k] in BF16 (leading dimensions a multiple of 64, zero beyond K up
// to the next multiple of 16), FP32 accumulation.
//
// One CTA of 512 threads computes a 128 x 32 tile of C on the fifth-
// generation tensor cores: 64-deep K chunks of both operands are copied by
// cp.async into a ring of eight shared-memory stages in the tensor cores'
// no-swizzle K-major layout (8 x 8 core matrices of 128 contiguous bytes; a
// 16-byte copy is one of their rows), all stages in flight at once; one thread
// issues tcgen05.mma.cta_group::1.kind::f16 (M = 128, N = 32, K = 16) with the
// FP32 accumulator in tensor memory, tcgen05.commit signals the stage's
// mbarrier when its products are done (a stage is refilled after that), and
// each warp reads 32 rows x 8 columns of the accumulator back with tcgen05.ld
// for the epilogue.  A launch of the training step takes 11 us on average (a
// minibatch of 256 rows at 13-4x512-256: 1110 us with FP32 operands read and
// rounded chunk by chunk in 38 launches, 140 us here), bound by the latency of
// its serial chain (copies, one barrier per chunk, epilogue): with 128 threads,
// one warp per scheduler, it took 15 us.
constexpr int TC_M = 128, TC_N = 32, TC_KC = 64;      // CTA tile and K chunk
constexpr int TC_STAGES = 8;
constexpr int TC_THREADS = 512;
constexpr int TC_COLS = TC_N / (TC_THREADS / 128);    // columns a thread takes in the epilogue
// A stage: per group of 8 rows the eight core matrices of the chunk, 144 bytes
// apart: the eight pieces of a row then fall on different banks, so that eight
// lanes can copy a whole 128-byte row.
constexpr int TC_LBO = 144, TC_SBO = 8 * TC_LBO;
constexpr int TC_B_OFF = TC_M / 8 * TC_SBO;           // B tile behind the A tile of a stage
constexpr int TC_STAGE = (TC_M + TC_N) / 8 * TC_SBO;  // bytes of a stage
constexpr int TC_SMEM = TC_STAGES * TC_STAGE;         // dynamic shared memory per CTA
constexpr int TC_TMEM_COLS = 32;                      // tensor-memory columns
constexpr long long kTcWaitLimit = 1ll << 22;         // bounded mbarrier wait (iterations)

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat16 l = __float2bfloat16_rn(lo), h = __float2bfloat16_rn(hi);
  return (uint32_t)__bfloat16_as_ushort(l) | ((uint32_t)__bfloat16_as_ushort(h) << 16);
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor of a no-swizzle K-major operand: start
// address, leading-dimension byte offset (between core matrices adjacent in
// K), stride-dimension byte offset (between core matrices adjacent in M/N),
// descriptor version 1, layout type 0 (no swizzle).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: FP32 accumulator (bits 4-5 = 1), BF16 A
// and B (bits 7-9, 10-12 = 1), both K-major (bits 15, 16 = 0), N >> 3 at bit
// 17, M >> 4 at bit 24.
constexpr uint32_t kTcIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TC_N >> 3) << 17) |
                              ((uint32_t)(TC_M >> 4) << 24);

__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
  for (long long it = 0; it < kTcWaitLimit; it++) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

using bf16 = __nv_bfloat16;

// What a product's epilogue does with C.
enum Epilogue {
  EPI_TANH,    // h = tanh(C + bias): FP32, and BF16 in both orientations
  EPI_OUT,     // y = C + bias (FP32)
  EPI_LOSS,    // d = y - target, dZ = 2 d scale (FP32, BF16 both ways) and the sum of d^2
  EPI_GRAD,    // C (FP32)
  EPI_BACK     // dZ = C (1 - h^2) (FP32, BF16 both ways)
};

struct Product {
  int M, N, K, epi;
  const bf16 *A, *B;
  int lda, ldb;
  float* out;         // [M x N] FP32 (EPI_LOSS: dZ)
  bf16* row;          // [M x ld_row] BF16 copy
  bf16* col;          // [N x ld_col] BF16 transposed copy
  int ld_row, ld_col;
  const float* bias;
  const float* h;     // EPI_BACK: [M x N]; EPI_LOSS: targets
  float scale;
  double* loss;
  int tiles_n, tiles; // 32-column tiles per row of tiles, tiles in all
};

// The products of one launch and the column sums that go with them: blocks 0 ..
// of the first product's tiles, then the second's, then column sums (one
// thread per column, rows summed in order).
struct GemmArgs {
  Product p[2];
  const float* cs_in;
  float* cs_out;
  int cs_rows, cs_cols;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}

// K chunk k0 of both operands into stage memory `st`: eight lanes copy one row's
// 128 bytes.  Rows past M or N are left as they are: they only enter results
// that are dropped.
__device__ __forceinline__ void load_chunk(const Product& P, int m0, int n0, int k0, uint32_t st) {
  constexpr int RP = TC_THREADS / 8;  // rows per pass
  const int kk = threadIdx.x & 7, r = threadIdx.x >> 3;
  const uint32_t dst = st + kk * TC_LBO + (r >> 3) * TC_SBO + (r & 7) * 16;
  const int rows = min(TC_M, P.M - m0), cols = min(TC_N, P.N - n0);
  const bf16* a = P.A + (long long)(m0 + r) * P.lda + k0 + kk * 8;
#pragma unroll
  for (int i = 0; i < TC_M / RP; i++, a += RP * P.lda)
    if (i * RP + r < rows) cp_async16(dst + i * (RP / 8) * TC_SBO, a);
  if (r < cols) cp_async16(dst + TC_B_OFF, P.B + (long long)(n0 + r) * P.ldb + k0 + kk * 8);
}
static_assert(TC_THREADS / 8 >= TC_N && TC_M % (TC_THREADS / 8) == 0, "rows of a pass");

__global__ void __launch_bounds__(TC_THREADS) k_gemm_tc(const __grid_constant__ GemmArgs g, int* err) {
  extern __shared__ __align__(1024) unsigned char tc_smem[];
  __shared__ __align__(8) unsigned long long mbar[TC_STAGES];
  __shared__ uint32_t tmem_base;
  __shared__ int failed;
  __shared__ double lsum[TC_THREADS / 32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  int b = blockIdx.x;
  if (b >= g.p[0].tiles + g.p[1].tiles) {
    const int n = (b - g.p[0].tiles - g.p[1].tiles) * 128 + tid;
    if (tid < 128 && n < g.cs_cols) {
      float s = 0.f;
#pragma unroll 16
      for (int r = 0; r < g.cs_rows; r++) s += g.cs_in[(long long)r * g.cs_cols + n];
      g.cs_out[n] = s;
    }
    return;
  }
  const bool second = b >= g.p[0].tiles;
  if (second) b -= g.p[0].tiles;
  const Product& P = g.p[second ? 1 : 0];
  const int m0 = b / P.tiles_n * TC_M, n0 = b % P.tiles_n * TC_N;
  const uint32_t sm = smem_addr(tc_smem);
  const int nchunks = (P.K + TC_KC - 1) / TC_KC;
  // every stage's copies in flight before anything else
  for (int c = 0; c < TC_STAGES; c++) {
    if (c < nchunks) load_chunk(P, m0, n0, c * TC_KC, sm + c * TC_STAGE);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(&tmem_base)),
                 "n"(TC_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (tid == 0) {
    for (int c = 0; c < TC_STAGES; c++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_addr(&mbar[c])) : "memory");
    failed = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = tmem_base;
  for (int c = 0; c < nchunks; c++) {
    const int s = c % TC_STAGES;
    asm volatile("cp.async.wait_group %0;\n" ::"n"(TC_STAGES - 1) : "memory");  // this thread's copies of chunk c
    // make the copies visible to the tensor cores
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      const uint32_t as = sm + s * TC_STAGE, bs = as + TC_B_OFF;
      const int steps = min(TC_KC, P.K - c * TC_KC);
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      for (int k = 0; k < steps; k += 16) {
        // K sub-block: core-matrix columns k/8 and k/8 + 1
        const uint64_t ad = smem_desc(as + (k >> 3) * TC_LBO, TC_LBO, TC_SBO);
        const uint64_t bd = smem_desc(bs + (k >> 3) * TC_LBO, TC_LBO, TC_SBO);
        const uint32_t acc = (c > 0 || k > 0) ? 1u : 0u;
        asm volatile(
            "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
            "l"(ad), "l"(bd), "r"(kTcIdesc), "r"(acc)
            : "memory");
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                       smem_addr(&mbar[s]))
                   : "memory");
    }
    // refill the stage once its products are done
    if (c + TC_STAGES < nchunks) {
      if (!mbar_wait(smem_addr(&mbar[s]), (uint32_t)((c / TC_STAGES) & 1))) failed = 1;
      __syncthreads();
      if (failed) break;
      load_chunk(P, m0, n0, (c + TC_STAGES) * TC_KC, sm + s * TC_STAGE);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  // the last chunk's products (they complete in order)
  const uint32_t last_bar = smem_addr(&mbar[(nchunks - 1) % TC_STAGES]);
  const uint32_t last_parity = (uint32_t)(((nchunks - 1) / TC_STAGES) & 1);
  __syncthreads();
  bool ok = !failed;
  if (ok) ok = mbar_wait(last_bar, last_parity);
  ok = __syncthreads_and(ok);
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  double l = 0.0;
  if (ok) {
    // warp w reads accumulator rows 32 (w % 4) .. (tensor-memory lanes a warp
    // can reach), columns 8 (w / 4) ..
    const int m = m0 + 32 * (warp & 3) + lane, nc = n0 + TC_COLS * (warp >> 2), N = P.N;
    const uint32_t taddr = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + TC_COLS * (warp >> 2);
    static_assert(TC_COLS == 8, "tcgen05.ld of 8 columns");
    uint32_t v[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
    const bool live = m < P.M;
    const int mpad = (P.M + 15) / 16 * 16;   // transposed copies are zero up to here
    const int cols = live ? min(N - nc, 8) : 0;  // columns of this thread that count (may be negative)
    const long long at = (long long)m * N + nc;
    float f[8];
#pragma unroll
    for (int j = 0; j < 8; j++) f[j] = __uint_as_float(v[j]);
    if (P.epi <= EPI_LOSS) {
#pragma unroll
      for (int j = 0; j < 8; j++)
        if (j < cols) f[j] += P.bias[nc + j];
    }
    if (P.epi == EPI_TANH) {
#pragma unroll
      for (int j = 0; j < 8; j++) f[j] = tanhf(f[j]);
    } else if (P.epi == EPI_LOSS) {
#pragma unroll
      for (int j = 0; j < 8; j++)
        if (j < cols) {
          const float d = f[j] - P.h[at + j];
          f[j] = 2.f * d * P.scale;
          l += (double)d * d;
        }
    } else if (P.epi == EPI_BACK) {
#pragma unroll
      for (int j = 0; j < 8; j++)
        if (j < cols) {
          const float h = P.h[at + j];
          f[j] *= 1.f - h * h;
        }
    }
    if (cols == 8 && (N & 3) == 0 && (reinterpret_cast<size_t>(P.out) & 15) == 0) {
      float4* o = reinterpret_cast<float4*>(P.out + at);
      o[0] = make_float4(f[0], f[1], f[2], f[3]);
      o[1] = make_float4(f[4], f[5], f[6], f[7]);
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++)
        if (j < cols) P.out[at + j] = f[j];
    }
    // a row is zero from N to the next multiple of 16: the product that reads it
    // sums up to there, and the same memory may have held longer rows (zero
    // weights would not cancel infinities or NaNs of an earlier pass)
    if (P.row && live && nc < (N + 15) / 16 * 16) {
#pragma unroll
      for (int j = 0; j < 8; j++)
        if (j >= cols) f[j] = 0.f;
      *reinterpret_cast<uint4*>(P.row + (long long)m * P.ld_row + nc) =
          make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
    }
    if (P.col && m < mpad) {
      bf16* o = P.col + (long long)nc * P.ld_col + m;
#pragma unroll
      for (int j = 0; j < 8; j++, o += P.ld_col)
        if (nc + j < N) *o = __float2bfloat16_rn(live ? f[j] : 0.f);
    }
    if (P.epi == EPI_LOSS) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
      if (lane == 0) lsum[warp] = l;
    }
  } else {
    // a wait gave up: record it, let the products in flight finish (again
    // bounded) before the tensor memory is released
    if (tid == 0) atomicExch(err, 1);
    mbar_wait(last_bar, last_parity);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (ok && P.epi == EPI_LOSS && tid == 0) {
    double t = 0.0;
    for (int w = 0; w < TC_THREADS / 32; w++) t += lsum[w];
    atomicAdd(P.loss, t);
  }
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "n"(TC_TMEM_COLS) : "memory");
  }
}

int* g_tc_err = nullptr;  // set by k_gemm_tc when a bounded wait gave up

void launch_products(GemmArgs& g) {
  static unsigned long long opted = 0;
  int dev = 0;
  NRPYELL_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !(opted >> dev & 1ull)) {
    NRPYELL_CUDA(cudaFuncSetAttribute(k_gemm_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM));
    opted |= 1ull << dev;
  }
  if (!g_tc_err) {
    NRPYELL_CUDA(dev_alloc(&g_tc_err, sizeof(int)));
    NRPYELL_CUDA(cudaMemsetAsync(g_tc_err, 0, sizeof(int), stream()));
  }
  int blocks = (g.cs_cols + 127) / 128;
  for (Product& p : g.p) {
    p.tiles = 0;
    if (p.M <= 0) continue;  // one product only
    if (p.N <= 0 || p.K <= 0) {
      NRPYELL_FAIL("k_gemm_tc: empty matrix product");
      return;
    }
    p.tiles_n = (p.N + TC_N - 1) / TC_N;
    p.tiles = p.tiles_n * ((p.M + TC_M - 1) / TC_M);
    blocks += p.tiles;
  }
  NRPYELL_LAUNCH_PDL(k_gemm_tc, blocks, TC_THREADS, TC_SMEM, g, g_tc_err);
}

// Reports (once) a bounded wait of the tensor-core GEMM that gave up.
bool gemm_ok() {
  if (!g_tc_err) return true;
  int e = 0;
  NRPYELL_CUDA(cudaMemcpy(&e, g_tc_err, sizeof(int), cudaMemcpyDeviceToHost));
  if (e) {
    NRPYELL_CUDA(cudaMemsetAsync(g_tc_err, 0, sizeof(int), stream()));
    NRPYELL_FAIL("k_gemm_tc: a bounded wait for the tensor-core products gave up");
    return false;
  }
  return status_ok();
}

// ------------------------------------------------------ elementwise pieces
// Rows of x (and of t) selected by idx (nullptr: all in order): x in BF16 in
// both orientations, t copied.  Transposed columns past `rows` are zero up to
// the next multiple of 16.
__global__ void k_minibatch(const float* __restrict__ x, const float* __restrict__ t, const int* __restrict__ idx,
                            int rows, int nx, int nt, bf16* __restrict__ row, int ld_row, bf16* __restrict__ col,
                            int ld_col, float* __restrict__ tb) {
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  const int rpad = (rows + 15) / 16 * 16;
  const long long na = (long long)rpad * nx, n = na + (long long)rows * nt;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    if (i < na) {
      const int r = (int)(i / nx), c = (int)(i % nx);
      const bf16 v = __float2bfloat16_rn(r < rows ? x[(long long)(idx ? idx[r] : r) * nx + c] : 0.f);
      if (r < rows) row[(long long)r * ld_row + c] = v;
      if (col) col[(long long)c * ld_col + r] = v;
    } else {
      const long long k = i - na;
      const int r = (int)(k / nt), c = (int)(k % nt);
      tb[k] = t[(long long)(idx ? idx[r] : r) * nt + c];
    }
  }
}

// One layer's parameters: W [in x out] row-major at woff, b at boff, and the
// BF16 copies of W (row) and its transpose (col).
struct LayerRef {
  int in, out, ld_row, ld_col, tile0;  // tile0: first block of the layer
  long long woff, boff;
  bf16 *row, *col;
};
constexpr int kMaxLayers = 64;
struct AdamArgs {
  LayerRef layer[kMaxLayers];
  int layers;
  float *p, *m, *v;
  const float* g;
  float lr, b1, b2, eps, c1, c2;
};

// Adam on the FP32 master parameters (ADAM), and the BF16 copies of the
// weights.  A block takes a 32 x 32 tile of a layer's W (or 1024 entries of
// its b), so that both copies are written along their rows.
template <bool ADAM>
__global__ void __launch_bounds__(256) k_adam(const __grid_constant__ AdamArgs a) {
  __shared__ float tile[32][33];
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  int l = 0;
  while (l + 1 < a.layers && (int)blockIdx.x >= a.layer[l + 1].tile0) l++;
  const LayerRef& L = a.layer[l];
  const int tn = (L.out + 31) / 32, tk = (L.in + 31) / 32, b = (int)blockIdx.x - L.tile0;
  auto update = [&](long long i) -> float {
    float p = a.p[i];
    if (ADAM) {
      const float g = a.g[i];
      // roundings spelled out: training must not depend on how the compiler
      // fuses these
      const float mi = __fmaf_rn(1.f - a.b1, g, __fmul_rn(a.b1, a.m[i]));
      const float vi = __fmaf_rn(__fmul_rn(1.f - a.b2, g), g, __fmul_rn(a.b2, a.v[i]));
      a.m[i] = mi;
      a.v[i] = vi;
      p -= a.lr * (mi / a.c1) / (sqrtf(vi / a.c2) + a.eps);
      a.p[i] = p;
    }
    return p;
  };
  if (b >= tn * tk) {
    if (ADAM)
      for (int n = (b - tn * tk) * 1024 + threadIdx.x; n < min(L.out, (b - tn * tk + 1) * 1024); n += 256)
        update(L.boff + n);
    return;
  }
  const int k0 = b / tn * 32, n0 = b % tn * 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
  for (int r = ty; r < 32; r += 8) {
    const int k = k0 + r, n = n0 + tx;
    if (k < L.in && n < L.out) {
      const float p = update(L.woff + (long long)k * L.out + n);
      tile[r][tx] = p;
      L.row[(long long)k * L.ld_row + n] = __float2bfloat16_rn(p);
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = ty; r < 32; r += 8) {
    const int n = n0 + r, k = k0 + tx;
    if (k < L.in && n < L.out) L.col[(long long)n * L.ld_col + k] = __float2bfloat16_rn(tile[tx][r]);
  }
}

unsigned blocks_for(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

}  // namespace

// ------------------------------------------------------------------- MLP

struct Mlp {
  int n_in, width, depth, n_out, batch_max;
  // layer l: dims[l] -> dims[l+1]; W_l [in x out] row-major, then b_l
  std::vector<int> dims;
  std::vector<long long> woff, boff;  // offsets into the parameter vector
  long long n_params = 0;
  float *p = nullptr, *grad = nullptr, *m = nullptr, *v = nullptr;
  std::vector<float*> h;   // output of layer l [batch_max x dims[l+1]]
  float* t = nullptr;      // minibatch targets
  float* dz[2] = {nullptr, nullptr};  // dZ of two consecutive layers [batch_max x widest]
  // BF16 operands, leading dimensions a multiple of 64 and zero padding up to the
  // next multiple of 16 (the epilogue writes it: dZ's memory serves layers of
  // several lengths):
  // hb[l] the input of layer l [batch_max x dims[l]] and its transpose, wb[l]
  // W_l and its transpose, db / dbt dZ of two consecutive layers
  std::vector<bf16*> hb, hbt, wb, wbt;
  bf16 *db[2] = {nullptr, nullptr}, *dbt[2] = {nullptr, nullptr};
  int ld_batch = 0;
  unsigned char* bf = nullptr;  // their memory
  double* loss = nullptr;
  int* idx = nullptr;      // an epoch's row order
  int idx_cap = 0;
  long long step = 0;
};

static int ld64(int n) { return (n + 63) / 64 * 64; }

// Adam (grad given; one step at learning rate lr) or only the BF16 copies of
// the weights.
static void launch_weights(Mlp* q, const float* grad, float lr) {
  AdamArgs a;
  memset(&a, 0, sizeof(a));
  const int L = (int)q->dims.size() - 1;
  const float b1 = 0.9f, b2 = 0.999f;
  a.p = q->p;
  a.m = q->m;
  a.v = q->v;
  a.g = grad;
  a.lr = lr;
  a.b1 = b1;
  a.b2 = b2;
  a.eps = 1e-8f;
  if (grad) {
    q->step++;
    a.c1 = 1.f - powf(b1, (float)q->step);
    a.c2 = 1.f - powf(b2, (float)q->step);
  }
  for (int l0 = 0; l0 < L; l0 += kMaxLayers) {
    a.layers = L - l0 < kMaxLayers ? L - l0 : kMaxLayers;
    int blocks = 0;
    for (int k = 0; k < a.layers; k++) {
      const int l = l0 + k, in = q->dims[l], out = q->dims[l + 1];
      a.layer[k] = {in, out, ld64(out), ld64(in), blocks, q->woff[l], q->boff[l], q->wb[l], q->wbt[l]};
      blocks += ((in + 31) / 32) * ((out + 31) / 32) + (out + 1023) / 1024;
    }
    if (grad)
      NRPYELL_LAUNCH_PDL(k_adam<true>, blocks, 256, 0, a);
    else
      NRPYELL_LAUNCH_PDL(k_adam<false>, blocks, 256, 0, a);
  }
}

static Mlp* mlp_new(int n_in, int width, int depth, int n_out, int batch_max, unsigned seed) {
  Mlp* q = new Mlp();
  q->n_in = n_in;
  q->width = width;
  q->depth = depth;
  q->n_out = n_out;
  q->batch_max = batch_max;
  q->dims.push_back(n_in);
  for (int i = 0; i < depth; i++) q->dims.push_back(width);
  q->dims.push_back(n_out);
  const int L = (int)q->dims.size() - 1;
  for (int l = 0; l < L; l++) {
    q->woff.push_back(q->n_params);
    q->n_params += (long long)q->dims[l] * q->dims[l + 1];
    q->boff.push_back(q->n_params);
    q->n_params += q->dims[l + 1];
  }
  // Glorot-uniform weights from a fixed 64-bit LCG, zero biases
  std::vector<float> host(q->n_params, 0.f);
  unsigned long long s = 0x9E3779B97F4A7C15ull ^ seed;
  for (int l = 0; l < L; l++) {
    const float a = sqrtf(6.f / (q->dims[l] + q->dims[l + 1]));
    for (long long i = 0; i < (long long)q->dims[l] * q->dims[l + 1]; i++) {
      s = s * 6364136223846793005ull + 1442695040888963407ull;
      const float u = (float)((s >> 11) * (1.0 / 9007199254740992.0));
      host[q->woff[l] + i] = a * (2.f * u - 1.f);
    }
  }
  const size_t pb = sizeof(float) * q->n_params;
  NRPYELL_CUDA(dev_alloc(&q->p, pb));
  NRPYELL_CUDA(dev_alloc(&q->grad, pb));
  NRPYELL_CUDA(dev_alloc(&q->m, pb));
  NRPYELL_CUDA(dev_alloc(&q->v, pb));
  NRPYELL_CUDA(cudaMemcpyAsync(q->p, host.data(), pb, cudaMemcpyHostToDevice, stream()));
  NRPYELL_CUDA(cudaMemsetAsync(q->m, 0, pb, stream()));
  NRPYELL_CUDA(cudaMemsetAsync(q->v, 0, pb, stream()));
  int wmax = n_out > width ? n_out : width;
  if (n_in > wmax) wmax = n_in;
  q->ld_batch = ld64(batch_max);
  std::vector<size_t> at;
  size_t total = 0;
  auto want = [&](size_t n) {
    at.push_back(total);
    total += (n * sizeof(bf16) + 255) / 256 * 256;
  };
  for (int l = 0; l < L; l++) {
    want((size_t)batch_max * ld64(q->dims[l]));
    want((size_t)q->dims[l] * q->ld_batch);
    want((size_t)q->dims[l] * ld64(q->dims[l + 1]));
    want((size_t)q->dims[l + 1] * ld64(q->dims[l]));
  }
  for (int k = 0; k < 2; k++) {
    want((size_t)batch_max * ld64(wmax));
    want((size_t)wmax * q->ld_batch);
  }
  NRPYELL_CUDA(dev_alloc(&q->bf, total));
  if (!status_ok()) return q;
  NRPYELL_CUDA(cudaMemsetAsync(q->bf, 0, total, stream()));
  size_t k = 0;
  for (int l = 0; l < L; l++) {
    q->hb.push_back((bf16*)(q->bf + at[k++]));
    q->hbt.push_back((bf16*)(q->bf + at[k++]));
    q->wb.push_back((bf16*)(q->bf + at[k++]));
    q->wbt.push_back((bf16*)(q->bf + at[k++]));
  }
  for (int i = 0; i < 2; i++) {
    q->db[i] = (bf16*)(q->bf + at[k++]);
    q->dbt[i] = (bf16*)(q->bf + at[k++]);
  }
  for (int l = 0; l < L; l++) {
    float* b = nullptr;
    NRPYELL_CUDA(dev_alloc(&b, sizeof(float) * (size_t)batch_max * q->dims[l + 1]));
    q->h.push_back(b);
  }
  NRPYELL_CUDA(dev_alloc(&q->t, sizeof(float) * (size_t)batch_max * n_out));
  for (float*& b : q->dz) NRPYELL_CUDA(dev_alloc(&b, sizeof(float) * (size_t)batch_max * wmax));
  NRPYELL_CUDA(dev_alloc(&q->loss, sizeof(double)));
  if (!status_ok()) return q;
  launch_weights(q, nullptr, 0.f);
  NRPYELL_CUDA(cudaStreamSynchronize(stream()));
  return q;
}

static void mlp_free(Mlp* q) {
  if (!q) return;
  cudaStreamSynchronize(stream());
  cudaFree(q->p);
  cudaFree(q->grad);
  cudaFree(q->m);
  cudaFree(q->v);
  for (float* b : q->h) cudaFree(b);
  cudaFree(q->t);
  cudaFree(q->dz[0]);
  cudaFree(q->dz[1]);
  cudaFree(q->bf);
  cudaFree(q->loss);
  cudaFree(q->idx);
  delete q;
}

// Minibatch inputs (rows of x by idx, or the first `rows`) into the BF16
// operand of the first layer; targets into q->t when t is given.
static void mlp_inputs(Mlp* q, const float* x, const float* t, const int* idx, int rows) {
  const long long n = (long long)((rows + 15) / 16 * 16) * q->n_in + (t ? (long long)rows * q->n_out : 0);
  const unsigned blocks = blocks_for(n, 256) < 592 ? blocks_for(n, 256) : 592;
  NRPYELL_LAUNCH_PDL(k_minibatch, blocks, 256, 0, x, t, idx, rows, q->n_in, t ? q->n_out : 0, q->hb[0],
                     ld64(q->n_in), q->hbt[0], q->ld_batch, q->t);
}

// Forward pass of the `rows` inputs set by mlp_inputs; output in q->h.back().
// With `train` the last layer also evaluates the loss against q->t (added to
// *q->loss) and dZ.
static void mlp_forward(Mlp* q, int rows, bool train) {
  const int L = (int)q->dims.size() - 1;
  for (int l = 0; l < L; l++) {
    const bool last = l == L - 1;
    GemmArgs g;
    memset(&g, 0, sizeof(g));
    Product& p = g.p[0];
    p.M = rows;
    p.N = q->dims[l + 1];
    p.K = q->dims[l];
    p.epi = !last ? EPI_TANH : train ? EPI_LOSS : EPI_OUT;
    p.A = q->hb[l];
    p.lda = ld64(q->dims[l]);
    p.B = q->wbt[l];
    p.ldb = ld64(q->dims[l]);
    p.bias = q->p + q->boff[l];
    p.out = q->h[l];
    p.ld_row = ld64(q->dims[l + 1]);
    p.ld_col = q->ld_batch;
    if (!last) {
      p.row = q->hb[l + 1];
      p.col = q->hbt[l + 1];
    } else if (train) {
      p.out = q->dz[0];
      p.h = q->t;
      p.row = q->db[0];
      p.col = q->dbt[0];
      p.scale = 1.f / (float)((long long)rows * q->n_out);
      p.loss = q->loss;
    }
    launch_products(g);
  }
}

// Gradient of the mean squared error into q->grad after mlp_forward(train):
// layer l's dW = H^T dZ and db, and layer l-1's dZ, in one launch.
static void mlp_backward(Mlp* q, int rows) {
  const int L = (int)q->dims.size() - 1;
  for (int l = L - 1; l >= 0; l--) {
    const int K = q->dims[l], N = q->dims[l + 1], cur = (L - 1 - l) & 1;
    GemmArgs g;
    memset(&g, 0, sizeof(g));
    Product& w = g.p[0];
    w.M = K;
    w.N = N;
    w.K = rows;
    w.epi = EPI_GRAD;
    w.A = q->hbt[l];
    w.lda = q->ld_batch;
    w.B = q->dbt[cur];
    w.ldb = q->ld_batch;
    w.out = q->grad + q->woff[l];
    g.cs_in = q->dz[cur];
    g.cs_out = q->grad + q->boff[l];
    g.cs_rows = rows;
    g.cs_cols = N;
    if (l > 0) {
      Product& p = g.p[1];
      p.M = rows;
      p.N = K;
      p.K = N;
      p.epi = EPI_BACK;
      p.A = q->db[cur];
      p.lda = ld64(N);
      p.B = q->wb[l];
      p.ldb = ld64(N);
      p.out = q->dz[1 - cur];
      p.h = q->h[l - 1];
      p.row = q->db[1 - cur];
      p.col = q->dbt[1 - cur];
      p.ld_row = ld64(K);
      p.ld_col = q->ld_batch;
    }
    launch_products(g);
  }
}

// ------------------------------------------------------------ POD guess
// y[0..Ntot) = mean + sum_k c[k] basis[k][.] (uu), y[Ntot..2 Ntot) = eta uu (vv),
// V consecutive points per thread.  The basis is read once (507 MB at 256
// modes on 128x128x16, which takes 89 us, 5.7 TB/s): the memory's rate bounds it,
// so a thread streams two points of 16 modes at a time.
template <int V>
__global__ void __launch_bounds__(256) k_pod_guess(const float* __restrict__ mean, const float* __restrict__ basis,
                                                   int K, long long ntot, const float* __restrict__ c, double eta,
                                                   double* y) {
  constexpr int U = 16;
  extern __shared__ float cs[];
  for (int k = threadIdx.x; k < K; k += blockDim.x) cs[k] = c[k];
  __syncthreads();
  const long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * V;
  if (i >= ntot) return;
  double u[V];
#pragma unroll
  for (int v = 0; v < V; v++) u[v] = (double)mean[i + v];
  const float* b = basis + i;
  int k = 0;
  for (; k + U <= K; k += U) {
    float w[U][V];
#pragma unroll
    for (int j = 0; j < U; j++) {
      if constexpr (V == 2) {
        const float2 t = __ldcs(reinterpret_cast<const float2*>(b + (k + j) * ntot));
        w[j][0] = t.x;
        w[j][1] = t.y;
      } else {
        w[j][0] = __ldcs(b + (k + j) * ntot);
      }
    }
#pragma unroll
    for (int j = 0; j < U; j++)
#pragma unroll
      for (int v = 0; v < V; v++) u[v] += (double)cs[k + j] * (double)w[j][v];
  }
  for (; k < K; k++)
#pragma unroll
    for (int v = 0; v < V; v++) u[v] += (double)cs[k] * (double)b[k * ntot + v];
#pragma unroll
  for (int v = 0; v < V; v++) {
    y[i + v] = u[v];
    y[ntot + i + v] = eta * u[v];
  }
}

}  // namespace nrpyell

using namespace nrpyell;

extern "C" {

void* nrpyell_mlp_create(int n_in, int width, int depth, int n_out, int batch_max, unsigned seed) {
  if (n_in <= 0 || width <= 0 || depth < 0 || n_out <= 0 || batch_max <= 0) {
    NRPYELL_FAIL("nrpyell_mlp_create: sizes must be positive");
    return nullptr;
  }
  Mlp* q = mlp_new(n_in, width, depth, n_out, batch_max, seed);
  if (!status_ok()) {
    mlp_free(q);
    return nullptr;
  }
  return q;
}

void nrpyell_mlp_destroy(void* mlp) { mlp_free((Mlp*)mlp); }

long long nrpyell_mlp_num_params(void* mlp) { return mlp ? ((Mlp*)mlp)->n_params : 0; }

int nrpyell_mlp_get_params(void* mlp, float* host) {
  Mlp* q = (Mlp*)mlp;
  NRPYELL_CUDA(cudaMemcpyAsync(host, q->p, sizeof(float) * q->n_params, cudaMemcpyDeviceToHost, stream()));
  NRPYELL_CUDA(cudaStreamSynchronize(stream()));
  return status_ok() ? 0 : -1;
}
int nrpyell_mlp_set_params(void* mlp, const float* host) {
  Mlp* q = (Mlp*)mlp;
  NRPYELL_CUDA(cudaMemcpyAsync(q->p, host, sizeof(float) * q->n_params, cudaMemcpyHostToDevice, stream()));
  launch_weights(q, nullptr, 0.f);
  NRPYELL_CUDA(cudaStreamSynchronize(stream()));
  return status_ok() ? 0 : -1;
}

int nrpyell_mlp_predict(void* mlp, const float* x, int n, float* y) {
  Mlp* q = (Mlp*)mlp;
  for (int r0 = 0; r0 < n; r0 += q->batch_max) {
    const int rows = (n - r0 < q->batch_max) ? n - r0 : q->batch_max;
    mlp_inputs(q, x + (long long)r0 * q->n_in, nullptr, nullptr, rows);
    mlp_forward(q, rows, false);
    NRPYELL_CUDA(cudaMemcpyAsync(y + (long long)r0 * q->n_out, q->h.back(), sizeof(float) * rows * q->n_out,
                                 cudaMemcpyDeviceToDevice, stream()));
  }
  NRPYELL_CUDA(cudaStreamSynchronize(stream()));
  return gemm_ok() ? 0 : -1;
}

double nrpyell_mlp_loss_grad(void* mlp, const float* x, const float* t, int rows, float* grad_host) {
  Mlp* q = (Mlp*)mlp;
  if (rows > q->batch_max || rows <= 0) {
    NRPYELL_FAIL("nrpyell_mlp_loss_grad: need 0 < rows <= batch_max");
    return NAN;
  }
  NRPYELL_CUDA(cudaMemsetAsync(q->loss, 0, sizeof(double), stream()));
  mlp_inputs(q, x, t, nullptr, rows);
  mlp_forward(q, rows, true);
  mlp_backward(q, rows);
  double loss = NAN;
  NRPYELL_CUDA(cudaMemcpyAsync(&loss, q->loss, sizeof(double), cudaMemcpyDeviceToHost, stream()));
  if (grad_host)
    NRPYELL_CUDA(cudaMemcpyAsync(grad_host, q->grad, sizeof(float) * q->n_params, cudaMemcpyDeviceToHost, stream()));
  NRPYELL_CUDA(cudaStreamSynchronize(stream()));
  if (!gemm_ok()) return NAN;
  return loss / ((double)rows * q->n_out);
}

double nrpyell_mlp_train(void* mlp, const float* x, const float* t, int n, int batch, int epochs, float lr,
                         unsigned seed, double* loss_history) {
  Mlp* q = (Mlp*)mlp;
  if (batch > q->batch_max || batch <= 0 || n < batch || epochs < 1) {
    NRPYELL_FAIL("nrpyell_mlp_train: need 0 < batch <= batch_max, batch <= n and epochs >= 1");
    return NAN;
  }
  if (n > q->idx_cap) {
    NRPYELL_CUDA(cudaStreamSynchronize(stream()));
    cudaFree(q->idx);
    q->idx = nullptr;
    q->idx_cap = 0;
    NRPYELL_CUDA(dev_alloc(&q->idx, sizeof(int) * n));
    if (!status_ok()) return NAN;
    q->idx_cap = n;
  }
  // perm is shuffled while the previous epoch runs; the copy to the GPU reads
  // `order`, which changes only after a wait for the epoch that it belongs to (an
  // asynchronous copy may read pageable memory at any time until then)
  std::vector<int> perm(n), order(n);
  for (int i = 0; i < n; i++) perm[i] = i;
  unsigned long long s = 0xD1B54A32D192ED03ull ^ seed;
  const int per_epoch = n / batch;
  const long long total = (long long)per_epoch * epochs;
  long long it = 0;
  double last = NAN;
  for (int e = 0; e < epochs && status_ok(); e++) {
    for (int i = n - 1; i > 0; i--) {  // Fisher-Yates
      s = s * 6364136223846793005ull + 1442695040888963407ull;
      const int j = (int)((s >> 33) % (unsigned long long)(i + 1));
      const int tmp = perm[i];
      perm[i] = perm[j];
      perm[j] = tmp;
    }
    double sum = 0.0;
    if (e > 0) {  // the previous epoch's loss
      NRPYELL_CUDA(cudaMemcpyAsync(&sum, q->loss, sizeof(double), cudaMemcpyDeviceToHost, stream()));
      NRPYELL_CUDA(cudaStreamSynchronize(stream()));
      if (!gemm_ok()) return NAN;
      last = sum / ((double)per_epoch * batch * q->n_out);
      if (loss_history) loss_history[e - 1] = last;
    }
    NRPYELL_CUDA(cudaMemsetAsync(q->loss, 0, sizeof(double), stream()));
    order = perm;
    NRPYELL_CUDA(cudaMemcpyAsync(q->idx, order.data(), sizeof(int) * n, cudaMemcpyHostToDevice, stream()));
    for (int b = 0; b < per_epoch; b++, it++) {
      mlp_inputs(q, x, t, q->idx + (long long)b * batch, batch);
      mlp_forward(q, batch, true);
      mlp_backward(q, batch);
      const float lr_t = lr * (0.01f + 0.99f * 0.5f * (1.f + cosf(3.14159265f * (float)it / (float)total)));
      launch_weights(q, q->grad, lr_t);
    }
  }
  double sum = 0.0;
  NRPYELL_CUDA(cudaMemcpyAsync(&sum, q->loss, sizeof(double), cudaMemcpyDeviceToHost, stream()));
  NRPYELL_CUDA(cudaStreamSynchronize(stream()));
  if (!gemm_ok()) return NAN;
  last = sum / ((double)per_epoch * batch * q->n_out);
  if (loss_history) loss_history[epochs - 1] = last;
  return last;
}

int nrpyell_pod_guess(const float* mean, const float* basis, int K, long long ntot, const float* c, double eta,
                      double* y_n) {
  if (K <= 0 || K > 4096 || ntot <= 0) {
    NRPYELL_FAIL("nrpyell_pod_guess: need 0 < K <= 4096 and ntot > 0");
    return -1;
  }
  // pairs of points where every mode's row starts on an 8-byte boundary
  if (ntot % 2 == 0 && reinterpret_cast<size_t>(basis) % 8 == 0)
    NRPYELL_LAUNCH(k_pod_guess<2>, blocks_for(ntot / 2, 256), 256, sizeof(float) * K, mean, basis, K, ntot, c, eta, y_n);
  else
    NRPYELL_LAUNCH(k_pod_guess<1>, blocks_for(ntot, 256), 256, sizeof(float) * K, mean, basis, K, ntot, c, eta, y_n);
  NRPYELL_CUDA(cudaStreamSynchronize(stream()));
  return status_ok() ? 0 : -1;
}

}  // extern "C"
