// Training kernels of the learned face flux (the network of flux_mlp.cuh), two
// launches per step: k_fwd_bwd runs the forward and the backward pass of
// 128-row tiles on the 5th-generation tensor cores and leaves each CTA's sums
// of the gradients, k_update adds them up and takes the Adam step.  Every
// product rounds its operands to BF16 and accumulates in FP32 (tensor memory);
// biases, activations before rounding, the loss and its derivatives are FP32.
//
// Included by fvm_kernels.cu.
#pragma once

namespace mlpt {

using mlp::kmajor_off;
using mlp::NH;
using mlp::NIN;
using mlp::NOUT;
using mlp::NOUTP;
using mlp::NPARAM;

constexpr int TM = 128;  // rows of a tile
constexpr int P_W1 = 0, P_B1 = P_W1 + NH * NIN, P_W2 = P_B1 + NH, P_B2 = P_W2 + NH * NH, P_W3 = P_B2 + NH,
              P_B3 = P_W3 + NH * NH, P_W4 = P_B3 + NH, P_B4 = P_W4 + NOUT * NH;  // parameters, in their order
constexpr int PART = NPARAM + 4;  // a CTA's sums: gradients, loss, padding

// The BF16 weight operands (K-major, no swizzle) in global memory: those of the
// forward products (rows: outputs, K: inputs) and their transposes for the
// backward ones (rows: inputs, K: outputs; the eight outputs of layer 4 padded
// to 16).
constexpr int I_W1 = 0, I_W4 = I_W1 + NH * NIN * 2, I_W4T = I_W4 + NOUTP * NH * 2, I_W2 = I_W4T + NH * NOUTP * 2,
              I_W3 = I_W2 + NH * NH * 2, I_W3T = I_W3 + NH * NH * 2, I_W2T = I_W3T + NH * NH * 2,
              I_BYTES = I_W2T + NH * NH * 2;

// Shared memory of k_fwd_bwd.  S_A: the forward products' activations, then
// the backward products' dZ [row][n].  S_T: A1, A2, A3 transposed [n][row], the
// operands of the weight gradients; dZ transposed takes A3's place once the
// layer 4 gradient has read it.  S_WA holds W2, then W3^T; S_WB W3, then W2^T.
constexpr int BIG = NH * NH * 2, SMALL = NH * 16 * 2;
constexpr int S_W1 = 0, S_W4 = S_W1 + SMALL, S_W4T = S_W4 + SMALL, S_X = S_W4T + SMALL, S_XT = S_X + SMALL,
              S_GT = S_XT + SMALL, S_WA = S_GT + SMALL, S_WB = S_WA + BIG, S_A = S_WB + BIG, S_T = S_A + BIG,
              S_BIAS = S_T + 3 * BIG, S_COL = S_BIAS + (3 * NH + 16) * 4, S_BAR = S_COL + 4 * 4,
              S_BYTES = S_BAR + 16;
static_assert(I_W4 == S_W4 && I_W4T == S_W4T && S_X % 1024 == 0 && S_WA % 1024 == 0 && S_BAR % 8 == 0, "layout");
static_assert(S_BYTES <= 227 * 1024, "shared memory");
constexpr int THREADS = 256;

__device__ __forceinline__ float gelu_grad(float x) {
  const float c = 0.7978845608028654f;
  const float t = mlp::tanh_hw(c * (x + 0.044715f * x * x * x));
  return 0.5f * (1.0f + t) + 0.5f * x * (1.0f - t * t) * c * (1.0f + 3.0f * 0.044715f * x * x);
}

__host__ __device__ __forceinline__ unsigned long long mix64(unsigned long long x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// Copies `bytes` (a multiple of 16 times THREADS) of a weight operand into
// shared memory without waiting (cp.async; wait_copies).
__device__ __forceinline__ void copy_async(unsigned char *dst, const unsigned char *src, int bytes) {
  for (int i = 16 * threadIdx.x; i < bytes; i += 16 * THREADS)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(mlp::smem_u32(dst + i)), "l"(src + i) : "memory");
}
__device__ __forceinline__ void wait_copies() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// D[128 x N] (tensor-memory columns at d) = A[128 x K] B[N x K]^T, added to D
// with acc, both operands K-major in shared memory; one thread.
__device__ __forceinline__ void product(uint32_t d, uint32_t a, uint32_t b, int N, int K, bool acc = false) {
  const uint32_t lbo_b = (uint32_t)(N / 8) * 128, idesc = mlp::instr_desc(TM, N);
  constexpr uint32_t LBO_A = (TM / 8) * 128, SBO = 128;
#pragma unroll 1
  for (int k = 0; k < K / 16; k++)
    mlp::mma_f16kind(d, mlp::smem_desc(a + 2 * k * LBO_A, LBO_A, SBO), mlp::smem_desc(b + 2 * k * lbo_b, lbo_b, SBO),
                     idesc, acc || k > 0);
}

// Eight BF16 values of row r, columns c .. c + 7 of a [128 x 128] operand, and
// the same transposed.  Two lanes hold neighbouring rows, so they exchange
// halves and each stores pairs (rows r and r ^ 1) of every second column.
// keep: all bits set, or zero for a row past the batch, which is zero in every
// operand: what the network makes of such a row's zero inputs may overflow
// where no row of the batch does, and 0 times that is not 0.  (Masks on the
// packed pairs cost nothing to speak of; a select per value took a step of
// 8,192 rows from 86 to 94 us.)
__device__ __forceinline__ void store_both(unsigned char *A, unsigned char *T, int r, int c, const float *v,
                                           uint32_t keep) {
  uint32_t w[4];
#pragma unroll
  for (int k = 0; k < 4; k++) w[k] = mlp::pack_bf16(v[2 * k], v[2 * k + 1]) & keep;
  if (A) *reinterpret_cast<uint4 *>(A + kmajor_off(r, c, TM)) = make_uint4(w[0], w[1], w[2], w[3]);
  const int odd = r & 1;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint32_t o = __shfl_xor_sync(0xffffffffu, w[k], 1);
    const uint32_t pair = odd ? __byte_perm(o, w[k], 0x7632) : __byte_perm(w[k], o, 0x5410);
    *reinterpret_cast<uint32_t *>(T + kmajor_off(c + 2 * k + odd, r & ~1, NH)) = pair;
  }
}

// 32 or 8 columns of this warp's lane quarter, written.
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float *v) {
  uint32_t r[32];
#pragma unroll
  for (int k = 0; k < 32; k++) r[k] = __float_as_uint(v[k]);
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};\n\t"
      "tcgen05.wait::st.sync.aligned;" ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const float *v) {
  uint32_t r[8];
#pragma unroll
  for (int k = 0; k < 8; k++) r[k] = __float_as_uint(v[k]);
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};\n\t"
      "tcgen05.wait::st.sync.aligned;" ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(taddr)
      : "memory");
}

// Forward and backward pass of a batch.  CTA z takes rows [z per, (z + 1) per),
// 128 at a time, row r being pair r of (X, T), or with pairs drawn (draw != 0)
// the pair a counter-based hash of (seed, step, r) names.  part[z]: its sums of
// the weight gradients, in parameter order, and of the loss; dz: dZ1, dZ2, dZ3
// (each four blocks of 32 columns, rows x 32) and dL/dY (rows x 8), which
// k_update sums into the bias gradients.  256 threads: warp w takes rows 32 (w % 4) .. + 31 and columns
// 64 (w / 4) .. + 63 of every accumulator; thread 0 issues the products.  The
// pre-activations Z1, Z2, Z3 stay in tensor memory (384 columns) from the
// forward to the backward pass and every operand in shared memory; a weight
// gradient of more than 128 rows goes on from its partial sum, put back into
// the last 128 columns.  Training amplifies round-off (after 40 steps 1e-7 is
// 1e-4), so the order of every sum is fixed: by the 16 rows of a product
// within a CTA's rows, by CTA, and for the bias gradients by row.
// A step of 8,192 rows takes 43 us here and 44 in k_update; as separate
// products, elementwise passes and column sums it was 32 launches and 1.25 ms.
// err bit 4: an mbarrier wait gave up.
static __global__ void __launch_bounds__(THREADS, 1) k_fwd_bwd(int rows, int per, long long n, const float *__restrict__ X,
                                                               const float *__restrict__ T, int draw,
                                                               unsigned long long seed, int step,
                                                               const float *__restrict__ P,
                                                               const unsigned char *__restrict__ img,
                                                               const float *__restrict__ wt, float *__restrict__ part,
                                                               float *__restrict__ dz, int *__restrict__ err) {
  extern __shared__ __align__(1024) unsigned char sm[];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, q = warp & 3, h = warp >> 2, r = 32 * q + lane;
  uint64_t *bar = reinterpret_cast<uint64_t *>(sm + S_BAR);
  uint32_t *tslot = reinterpret_cast<uint32_t *>(sm + S_BAR + 8);
  float *bias = reinterpret_cast<float *>(sm + S_BIAS), *col = reinterpret_cast<float *>(sm + S_COL);
  float *out = part + (size_t)blockIdx.x * PART;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(mlp::smem_u32(tslot)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (t == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mlp::smem_u32(bar)), "r"(1));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  copy_async(sm + S_W1, img + I_W1, 3 * SMALL);
  for (int i = t; i < NH; i += THREADS) {
    bias[i] = P[P_B1 + i];
    bias[NH + i] = P[P_B2 + i];
    bias[2 * NH + i] = P[P_B3 + i];
    if (i < NOUT) bias[3 * NH + i] = P[P_B4 + i];
  }
  for (int i = t; i < SMALL / 4; i += THREADS) reinterpret_cast<uint32_t *>(sm + S_GT)[i] = 0;  // outputs 8 .. 15
  mlp::fence_before();
  __syncthreads();
  mlp::fence_after();
  const uint32_t tm = *tslot, lanes = (uint32_t)(32 * q) << 16, s0 = mlp::smem_u32(sm), bar_a = mlp::smem_u32(bar);
  const uint32_t Z1 = tm, Z2 = tm + NH, Z3 = tm + 2 * NH, ZT = tm + 3 * NH;
  uint32_t parity = 0;
  bool ok = true;
  // a barrier before the products (operands written, accumulators read), the
  // products by one thread, and the wait for them
  auto products = [&](auto &&issue) {
    mlp::fence_async_smem();
    mlp::fence_before();
    __syncthreads();
    if (t == 0) {
      mlp::fence_after();
      issue();
      mlp::mma_commit(bar_a);
    }
    ok = __syncthreads_and(warp == 0 ? mlp::bar_wait(bar_a, parity) : true);
    parity ^= 1;
    mlp::fence_after();
    return ok;
  };
  // hidden layer L (1 .. 3): activations of the accumulator z
  auto forward = [&](uint32_t z, int L, uint32_t keep) {
#pragma unroll 1
    for (int c = 64 * h; c < 64 * h + 64; c += 32) {
      float v[32];
      mlp::tmem_ld32(z + lanes + (uint32_t)c, v);
#pragma unroll
      for (int j = 0; j < 32; j++) v[j] = mlp::gelu(v[j] + bias[(L - 1) * NH + c + j]);
#pragma unroll
      for (int j = 0; j < 32; j += 8) store_both(sm + S_A, sm + S_T + (L - 1) * BIG, r, c + j, v + j, keep);
    }
  };
  // layer L's dZ of row `row` (if it is in the batch) from dA (accumulator d)
  // and Z, also as an operand and transposed
  auto backward = [&](uint32_t d, uint32_t z, int L, bool rows_too, int row, int end) {
    float *o = dz + ((size_t)(L - 1) * NH * rows + (size_t)row * 32);
#pragma unroll 1
    for (int c = 64 * h; c < 64 * h + 64; c += 32) {
      float v[32], g[32];
      mlp::tmem_ld32(z + lanes + (uint32_t)c, g);
#pragma unroll
      for (int j = 0; j < 32; j++) g[j] = gelu_grad(g[j] + bias[(L - 1) * NH + c + j]);
      mlp::tmem_ld32(d + lanes + (uint32_t)c, v);
#pragma unroll
      for (int j = 0; j < 32; j++) v[j] *= g[j];
#pragma unroll
      for (int j = 0; j < 32; j += 8)
        store_both(rows_too ? sm + S_A : nullptr, sm + S_T + 2 * BIG, r, c + j, v + j, row < end ? ~0u : 0u);
      if (row < end) {
#pragma unroll
        for (int j = 0; j < 32; j += 4)
          *reinterpret_cast<float4 *>(o + (size_t)c * rows + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
      }
    }
  };
  // a 128 x 128 weight gradient (rows: outputs): its partial sum put back into
  // the accumulator, and the sum with this tile's rows stored
  auto take_weights = [&](uint32_t d, int p) {
#pragma unroll 1
    for (int c = 64 * h; c < 64 * h + 64; c += 32) {
      float v[32];
      const float4 *o = reinterpret_cast<const float4 *>(out + p + r * NH + c);
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const float4 w = o[j];
        v[4 * j] = w.x; v[4 * j + 1] = w.y; v[4 * j + 2] = w.z; v[4 * j + 3] = w.w;
      }
      tmem_st32(d + lanes + (uint32_t)c, v);
    }
  };
  auto put_weights = [&](uint32_t d, int p) {
#pragma unroll 1
    for (int c = 64 * h; c < 64 * h + 64; c += 32) {
      float v[32];
      mlp::tmem_ld32(d + lanes + (uint32_t)c, v);
      float4 *o = reinterpret_cast<float4 *>(out + p + r * NH + c);
#pragma unroll
      for (int j = 0; j < 8; j++) o[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    }
  };
  // the same for the 16-column gradients of layers 1 and 4 (column k of row r at
  // out[p + r rs + k ks], cols of them)
  auto take_narrow = [&](uint32_t d, int p, int rs, int ks, int cols) {
    if (h != 0) return;
    for (int c = 0; c < cols; c += 8) {
      float v[8];
#pragma unroll
      for (int k = 0; k < 8; k++) v[k] = out[p + r * rs + (c + k) * ks];
      tmem_st8(d + lanes + (uint32_t)c, v);
    }
  };
  auto put_narrow = [&](uint32_t d, int p, int rs, int ks, int cols) {
    if (h != 0) return;
    for (int c = 0; c < cols; c += 8) {
      float v[8];
      mlp::tmem_ld8(d + lanes + (uint32_t)c, v);
#pragma unroll
      for (int k = 0; k < 8; k++) out[p + r * rs + (c + k) * ks] = v[k];
    }
  };
  float loss = 0.0f;  // of this thread's rows
  const int begin = blockIdx.x * per, end = min(rows, begin + per);
#pragma unroll 1
  for (int base = begin; base < end && ok; base += TM) {
    const bool more = base > begin;  // the gradients go on from their partial sums
    copy_async(sm + S_WA, img + I_W2, BIG);
    copy_async(sm + S_WB, img + I_W3, BIG);
    // rows past the CTA's: zero inputs, and zero derivatives below
    const int row = base + r;
    const long long src =
        draw ? (long long)(mix64(seed ^ ((unsigned long long)step << 32) ^ (unsigned long long)row) %
                           (unsigned long long)n)
             : row;
    if (h == 0) {
      float x[NIN];
#pragma unroll
      for (int k = 0; k < NIN; k += 4) {
        const float4 v = row < end ? *reinterpret_cast<const float4 *>(X + src * NIN + k) : make_float4(0, 0, 0, 0);
        x[k] = v.x; x[k + 1] = v.y; x[k + 2] = v.z; x[k + 3] = v.w;
      }
      uint32_t w[8];
#pragma unroll
      for (int k = 0; k < 8; k++) w[k] = mlp::pack_bf16(x[2 * k], x[2 * k + 1]);
      *reinterpret_cast<uint4 *>(sm + S_X + kmajor_off(r, 0, TM)) = make_uint4(w[0], w[1], w[2], w[3]);
      *reinterpret_cast<uint4 *>(sm + S_X + kmajor_off(r, 8, TM)) = make_uint4(w[4], w[5], w[6], w[7]);
#pragma unroll
      for (int k = 0; k < NIN; k++)
        *reinterpret_cast<uint16_t *>(sm + S_XT + kmajor_off(k, r, NIN)) = (uint16_t)(w[k / 2] >> (16 * (k & 1)));
    }
    wait_copies();
    if (!products([&] { product(Z1, s0 + S_X, s0 + S_W1, NH, NIN); })) break;
    forward(Z1, 1, row < end ? ~0u : 0u);
    if (!products([&] { product(Z2, s0 + S_A, s0 + S_WA, NH, NH); })) break;
    copy_async(sm + S_WA, img + I_W3T, BIG);  // W2 has been read
    forward(Z2, 2, row < end ? ~0u : 0u);
    if (!products([&] { product(Z3, s0 + S_A, s0 + S_WB, NH, NH); })) break;
    copy_async(sm + S_WB, img + I_W2T, BIG);  // W3 has been read
    forward(Z3, 3, row < end ? ~0u : 0u);
    if (!products([&] { product(ZT, s0 + S_A, s0 + S_W4, NOUTP, NH); })) break;
    // output layer: Y = Z + b; G = dL/dY of L = mean w (Y - T)^2
    if (h == 0) {
      float y[8], g[8];
      mlp::tmem_ld8(ZT + lanes, y);
      const float s = 1.0f / (float)((long long)rows * NOUT);
#pragma unroll
      for (int k = 0; k < NOUT; k++) {
        const float e = row < end ? y[k] + bias[3 * NH + k] - T[src * NOUT + k] : 0.0f;
        g[k] = 2.0f * wt[k] * e * s;
        loss += wt[k] * e * e * s;
      }
      uint32_t w[4];
#pragma unroll
      for (int k = 0; k < 4; k++) w[k] = mlp::pack_bf16(g[2 * k], g[2 * k + 1]);
      *reinterpret_cast<uint4 *>(sm + S_X + kmajor_off(r, 0, TM)) = make_uint4(w[0], w[1], w[2], w[3]);
      *reinterpret_cast<uint4 *>(sm + S_X + kmajor_off(r, 8, TM)) = make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int k = 0; k < NOUT; k++)
        *reinterpret_cast<uint16_t *>(sm + S_GT + kmajor_off(k, r, NOUTP)) = (uint16_t)(w[k / 2] >> (16 * (k & 1)));
      if (row < end) {
        float4 *o = reinterpret_cast<float4 *>(dz + (size_t)3 * rows * NH + (size_t)row * NOUT);
        o[0] = make_float4(g[0], g[1], g[2], g[3]);
        o[1] = make_float4(g[4], g[5], g[6], g[7]);
      }
    }
    // gW4^T (rows: inputs of layer 4) = A3^T G
    if (more) take_narrow(ZT, P_W4, 1, NH, NOUT);
    if (!products([&] { product(ZT, s0 + S_T + 2 * BIG, s0 + S_GT, NOUTP, TM, more); })) break;
    put_narrow(ZT, P_W4, 1, NH, NOUT);
    if (!products([&] { product(ZT, s0 + S_X, s0 + S_W4T, NH, NOUTP); })) break;  // dA3 = G W4
    backward(ZT, Z3, 3, true, row, end);
    if (more) {
      mlp::fence_before();
      __syncthreads();  // dA3 has been read
      mlp::fence_after();
      take_weights(ZT, P_W3);
    }
    wait_copies();  // W3^T and W2^T
    if (!products([&] {
          product(ZT, s0 + S_T + 2 * BIG, s0 + S_T + BIG, NH, TM, more);  // gW3 = dZ3^T A2
          product(Z3, s0 + S_A, s0 + S_WA, NH, NH);                       // dA2 = dZ3 W3
        }))
      break;
    put_weights(ZT, P_W3);
    backward(Z3, Z2, 2, true, row, end);
    if (more) take_weights(ZT, P_W2);
    if (!products([&] {
          product(ZT, s0 + S_T + 2 * BIG, s0 + S_T, NH, TM, more);  // gW2 = dZ2^T A1
          product(Z3, s0 + S_A, s0 + S_WB, NH, NH);                 // dA1 = dZ2 W2
        }))
      break;
    put_weights(ZT, P_W2);
    backward(Z3, Z1, 1, false, row, end);
    if (more) {
      mlp::fence_before();
      __syncthreads();  // gW2 has been read
      mlp::fence_after();
      take_narrow(ZT, P_W1, NIN, 1, NIN);
    }
    if (!products([&] { product(ZT, s0 + S_T + 2 * BIG, s0 + S_XT, NIN, TM, more); })) break;  // gW1 = dZ1^T X
    put_narrow(ZT, P_W1, NIN, 1, NIN);
    mlp::fence_before();
    __syncthreads();  // accumulators and operands are read before the next tile's
    mlp::fence_after();
  }
  if (h == 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
    if (lane == 0) col[q] = loss;
  }
  __syncthreads();
  if (t == 0) out[NPARAM] = (col[0] + col[1]) + (col[2] + col[3]);
  if (!ok) {
    if (t == 0) atomicOr(err, 4);
    // products may still be in flight: wait (bounded) before the tensor memory
    // is released
    mlp::bar_wait(bar_a, parity ^ 1);
    wait_copies();
  }
  mlp::fence_before();
  __syncthreads();
  if (warp == 0) {
    mlp::fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm), "r"(512));
  }
}

// Parameter i's BF16 value where k_fwd_bwd's operands hold it.
__device__ __forceinline__ void put_operand(unsigned char *img, int i, float p) {
  const __nv_bfloat16 v = __float2bfloat16_rn(p);
  auto at = [&](int base, int row, int k, int rows) {
    *reinterpret_cast<__nv_bfloat16 *>(img + base + kmajor_off(row, k, rows)) = v;
  };
  if (i < P_B1) {
    at(I_W1, (i - P_W1) / NIN, (i - P_W1) % NIN, NH);
  } else if (i >= P_W2 && i < P_B2) {
    const int o = (i - P_W2) / NH, k = (i - P_W2) % NH;
    at(I_W2, o, k, NH);
    at(I_W2T, k, o, NH);
  } else if (i >= P_W3 && i < P_B3) {
    const int o = (i - P_W3) / NH, k = (i - P_W3) % NH;
    at(I_W3, o, k, NH);
    at(I_W3T, k, o, NH);
  } else if (i >= P_W4 && i < P_B4) {
    const int o = (i - P_W4) / NH, k = (i - P_W4) % NH;
    at(I_W4, o, k, NOUTP);
    at(I_W4T, k, o, NH);
  }
}
static __global__ void k_operands(const float *__restrict__ p, unsigned char *__restrict__ img) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < NPARAM) put_operand(img, i, p[i]);
}

// The gradient and (m not null) the Adam step with the weight operands of the
// next.  The first BBLOCKS blocks sum the bias gradients over the rows of dz,
// 32 columns (one warp) or layer 4's eight each, a column per thread and in row
// order: a chain of dependent adds (four cycles each, 17 us for 8,192 rows),
// fed by bulk copies of CROWS rows CSTAGES - 1 stages ahead.  (A layer's 128
// columns in one block wait for its SM's 4 MB: 82 us against 44.)  The others add the
// CTAs' sums of the weight gradients in their order, and the loss.  err bit 4:
// a copy's wait gave up.
constexpr int UTHREADS = 128, BBLOCKS = 13, CROWS = 128, CSTAGES = 4, U_BYTES = CSTAGES * CROWS * 32 * 4;
constexpr int UBLOCKS = BBLOCKS + (NPARAM + 1 + UTHREADS - 1) / UTHREADS;
// The sum of column `lane` of src (rows x COLS), by one warp.
template <int COLS>
__device__ __forceinline__ float column_sum(int rows, const float *__restrict__ src, float *ring, uint64_t *bars,
                                            int lane, int *err) {
  const int stages = (rows + CROWS - 1) / CROWS;
  if (lane == 0) {
    for (int b = 0; b < CSTAGES; b++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mlp::smem_u32(bars + b)), "r"(1));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncwarp();
  auto fetch = [&](int s) {  // by one thread
    if (s >= stages) return;
    const int bytes = min(CROWS, rows - s * CROWS) * COLS * 4;  // a multiple of 32
    const uint32_t bar = mlp::smem_u32(bars + s % CSTAGES);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     mlp::smem_u32(ring + (s % CSTAGES) * CROWS * COLS)),
                 "l"(src + (size_t)s * CROWS * COLS), "r"(bytes), "r"(bar)
                 : "memory");
  };
  if (lane == 0)
    for (int s = 0; s < CSTAGES - 1; s++) fetch(s);
  float g = 0.0f;
  bool ok = true;
  for (int s = 0; s < stages && ok; s++) {
    ok = mlp::bar_wait(mlp::smem_u32(bars + s % CSTAGES), (uint32_t)(s / CSTAGES & 1));
    ok = __all_sync(0xffffffffu, ok);  // and every lane is done with the stage before
    if (lane == 0 && ok) fetch(s + CSTAGES - 1);
    if (ok && lane < COLS) {
      const float *at = ring + (s % CSTAGES) * CROWS * COLS + lane;
      const int cnt = min(CROWS, rows - s * CROWS);
      int k = 0;
      for (; k + 16 <= cnt; k += 16) {
        float x[16];
#pragma unroll
        for (int j = 0; j < 16; j++) x[j] = at[(k + j) * COLS];
#pragma unroll
        for (int j = 0; j < 16; j++) g += x[j];
      }
      for (; k < cnt; k++) g += at[k * COLS];
    }
  }
  if (!ok) {  // the copies in flight write this block's memory: wait (bounded) for them
    if (lane == 0) atomicOr(err, 4);
    for (int b = 0; b < CSTAGES; b++)
      for (int par = 0; par < 2; par++) mlp::bar_wait(mlp::smem_u32(bars + b), (uint32_t)par);
  }
  return g;
}
static __global__ void __launch_bounds__(UTHREADS) k_update(int rows, int ncta, const float *__restrict__ part,
                                                            const float *__restrict__ dz, float *__restrict__ grad,
                                                            float *__restrict__ loss, float *__restrict__ p,
                                                            float *__restrict__ m, float *__restrict__ v,
                                                            unsigned char *__restrict__ img, int *__restrict__ err,
                                                            float lr, float b1, float b2, float eps, float c1,
                                                            float c2) {
  extern __shared__ __align__(128) float ring[];
  __shared__ __align__(8) uint64_t bars[CSTAGES];
  const int t = threadIdx.x;
  int i;
  float g = 0.0f;
  if (blockIdx.x < BBLOCKS) {
    if (t >= 32) return;
    const float *src = dz + (size_t)blockIdx.x * 32 * rows;
    if (blockIdx.x == BBLOCKS - 1) {
      g = column_sum<NOUT>(rows, src, ring, bars, t, err);
      if (t >= NOUT) return;
      i = P_B4 + t;
    } else {
      g = column_sum<32>(rows, src, ring, bars, t, err);
      const int L = blockIdx.x / 4;
      i = (L == 0 ? P_B1 : L == 1 ? P_B2 : P_B3) + 32 * (blockIdx.x % 4) + t;
    }
  } else {
    i = (blockIdx.x - BBLOCKS) * UTHREADS + t;
    if (i > NPARAM || (i >= P_B1 && i < P_W2) || (i >= P_B2 && i < P_W3) || (i >= P_B3 && i < P_W4) ||
        (i >= P_B4 && i < NPARAM))
      return;
#pragma unroll 8
    for (int z = 0; z < ncta; z++) g += part[(size_t)z * PART + i];
    if (i == NPARAM) {
      *loss = g;
      return;
    }
  }
  if (grad) grad[i] = g;
  if (!m) return;
  const float mi = b1 * m[i] + (1.0f - b1) * g;
  const float vi = b2 * v[i] + (1.0f - b2) * g * g;
  m[i] = mi;
  v[i] = vi;
  const float w = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  p[i] = w;
  put_operand(img, i, w);
}

}  // namespace mlpt
