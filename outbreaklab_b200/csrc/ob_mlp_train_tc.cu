// ob_mlp_train_tc.cu — training of the microphysics surrogate on the 5th-generation tensor cores (sm_100a):
// BF16 operands, FP32 accumulation in TMEM, the elementwise work fused into the GEMM epilogues, every batch
// reduction in a fixed order (a seed fixes the trained network).
//
// One training step on a batch of B samples (B a multiple of 128) is three launches:
//   k_mlp_step   a CTA takes 128 samples through the whole network and back. It holds every weight image in shared memory
//                (164 KB, TMA-loaded, K-major with a 128-byte swizzle), one activation tile (the A operand of the next
//                tcgen05.mma, M = 128, K = 16 per instruction) and the three hidden layers' products, then their GELU', in
//                TMEM (3 x 128 columns; the fourth 128 serve the output and the backward products), so that nothing but
//                the operands of the weight gradients goes to memory: the samples drawn and normalised in place, then
//                forward, layers 1-3   Z = H W^T; + bias, GELU -> H (bf16)
//                forward, layer 4      Y = H3 W4^T; + bias, the loss of the 8 scheme tendencies (FP64 partial per tile)
//                                      and dY = 2 (Y - T) / (B * 8)
//                backward, layers 3-1  dH = dZ W (W transposed, kept as its own bf16 image); dZ = dH * GELU'(Z)
//                with X, H, dY and dZ written feature-major;
//   k_mlp_wgrad  weight gradients dW = dZ^T [H, 1]: M = 128 output features (10 for layer 4, zero-padded), N = the input
//                features plus a row of ones (so the last column is the bias gradient), K = the batch, split over CTAs
//                into partial slices;
//   k_grad_adam  the slices added in split order, Adam on the fp32 master parameters and their bf16 images both ways; the
//                loss partials in tile order.
// What bounds a step is the instructions of GELU and its derivative (27 us of k_mlp_step; 38 us with two threads per sample
// and the derivative worked out again on the way back) and the latency of the seven layers in turn: 124 -> 48 us a step at
// a batch of 16384 against a launch per layer (15 launches), which wrote and read activations, GELU' (fp32) and targets
// in between. Each launch sets itself up under the tail of the one before (56 -> 48 us).
// Every mbarrier wait is bounded (ob_tc.cuh): a timed-out wait sets a bit in the error word the host checks.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "../../include/ob.h"
#include "ob_mlp.cuh"
#include "ob_tc.cuh"

namespace ob {
void set_error(const char* fmt, ...);

namespace mlp {

constexpr int GBM = 128, GBK = 64;   // samples per tile, K per 128-byte swizzled row
constexpr int NHX = NH + 16;   // feature-major activations: 128 features, a row of ones, 15 zero rows (N = 144)
constexpr int NXX = 16;        // feature-major inputs: 12 features, a row of ones, 3 zero rows
constexpr int KPAD = 64;       // K of the first layer's and of dY's images, padded to one swizzled row
constexpr int WSPLIT_MAX = 16; // batch splits of a weight-gradient GEMM

// shared memory of k_mlp_step: the weight images, the activation tile, barriers
constexpr int S_W1 = 0, S_W2 = S_W1 + NH * 128, S_W3 = S_W2 + 2 * NH * 128, S_W4 = S_W3 + 2 * NH * 128, S_W4T = S_W4 + 2 * 16 * 128,
              S_W3T = S_W4T + NH * 128, S_W2T = S_W3T + 2 * NH * 128, S_ACT = S_W2T + 2 * NH * 128, S_BAR = S_ACT + 2 * GBM * 128,
              STEP_SMEM = S_BAR + 1024 /*align*/ + 256;
constexpr int STEP_THREADS = 544;   // four threads per sample, and a warp for TMA and MMA
// k_mlp_wgrad: a ring of stages of 128 output features and 80 input features by 64 samples
constexpr int WN = 80, WA_BYTES = GBM * GBK * 2, WSTAGE = WA_BYTES + WN * GBK * 2, WSTAGES = 8, WSMEM = WSTAGES * WSTAGE + 1024 + 256,
              WTHREADS = 192;

struct StepMaps {
  CUtensorMap f[4];   // W1, W2, W3, W4 (forward images)
  CUtensorMap b[3];   // W2^T, W3^T, W4^T
};
struct StepArgs {
  const float* pairs;
  unsigned npairs, step, seed;
  int draw;                  // samples drawn by a hash of (step, sample); else in order
  long B;                    // batch
  Norm nm;
  const float* w;            // fp32 parameters (the biases)
  __nv_bfloat16* Xt;         // feature-major [NXX][B]
  __nv_bfloat16* Ht[3];      // [NHX][B]
  __nv_bfloat16* dYt;        // [128][B]
  __nv_bfloat16* dZt[3];     // [128][B]
  double* lossp;             // per-tile loss partial (sum of squares)
  float inv;                 // 2 / (B * NLOSS)
};

// one weight-gradient GEMM of the grouped launch: A = dZ^T (or dY^T) [128][B], B = [H, 1]^T [N][B]
struct WgradSet {
  CUtensorMap a[4];
  CUtensorMap b[4];
  int N[4];
  float* part[4];            // [split][128][N]
};

__device__ __forceinline__ void tmem_ld16x(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// 32 columns of fp32 to TMEM, one row (lane) per thread
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float (&v)[32]) {
  uint32_t r[32];
#pragma unroll
  for (int i = 0; i < 32; i++) r[i] = __float_as_uint(v[i]);
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};" ::"r"(r[0]),
      "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]),
      "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
      "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// byte offset of 8 consecutive bf16 of a K-major tile in the 128-byte swizzled layout (64-column blocks of `rows` rows)
__device__ __forceinline__ uint32_t swz(int row, int col, int rows) {
  return uint32_t((col >> 6) * rows * 128 + row * 128 + ((((col & 63) >> 3) ^ (row & 7)) << 4));
}
__device__ __forceinline__ void act8(uint8_t* act, int row, int col, const float* v) {
  __align__(16) __nv_bfloat16 h[8];
#pragma unroll
  for (int e = 0; e < 8; e++) h[e] = __float2bfloat16_rn(v[e]);
  *reinterpret_cast<uint4*>(act + swz(row, col, GBM)) = *reinterpret_cast<const uint4*>(h);
}
// 32 features of a sample (one lane each) as bf16: into the activation tile (if any), and feature-major: two neighbouring
// lanes exchange, so that each stores its own features of both samples as one word
__device__ __forceinline__ void put_features(uint8_t* act, __nv_bfloat16* t_out, long B, int row, int c0, long s, int lane, const float* v) {
  uint32_t h[16];
#pragma unroll
  for (int e = 0; e < 16; e++) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
    h[e] = *reinterpret_cast<const uint32_t*>(&p);
  }
  if (act) {
#pragma unroll
    for (int e = 0; e < 16; e += 4) *reinterpret_cast<uint4*>(act + swz(row, c0 + 2 * e, GBM)) = make_uint4(h[e], h[e + 1], h[e + 2], h[e + 3]);
  }
  const bool odd = lane & 1;
  uint32_t* o = reinterpret_cast<uint32_t*>(t_out + long(c0 + (odd ? 1 : 0)) * B + (s & ~1l));
#pragma unroll
  for (int e = 0; e < 16; e++) {   // even lanes keep feature 2 e, odd lanes 2 e + 1
    const uint32_t other = __shfl_xor_sync(0xffffffffu, h[e], 1);
    *o = odd ? __byte_perm(other, h[e], 0x7632) : __byte_perm(h[e], other, 0x5410);
    o += B;   // two features on: 2 B bf16
  }
}
// D[128 x N] = A[128 x K] W[N x K]^T, K in steps of 16 in ascending order; the commit arrives at bar
__device__ __forceinline__ void issue_layer(uint32_t acc, uint32_t a, uint32_t w, int wrows, int K, int N, uint64_t* bar) {
  const uint32_t idesc = tc::idesc_bf16_f32(GBM, N);
  for (int k = 0; k < K; k += 16) {
    const uint32_t ao = uint32_t((k >> 6) * GBM * 128 + ((k & 63) >> 3) * 16), wo = uint32_t((k >> 6) * wrows * 128 + ((k & 63) >> 3) * 16);
    tc::mma_bf16(acc, tc::desc_k_sw128(a + ao), tc::desc_k_sw128(w + wo), idesc, k > 0 ? 1u : 0u);
  }
  tc::mma_commit(bar);
}

__global__ void __launch_bounds__(STEP_THREADS, 1) k_mlp_step(const __grid_constant__ StepMaps M, const __grid_constant__ StepArgs P,
                                                              unsigned int* err) {
  extern __shared__ uint8_t smraw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smraw) + 1023) & ~uintptr_t(1023));
  __shared__ double lred[4];
  uint64_t* wbar = reinterpret_cast<uint64_t*>(sm + S_BAR);   // the weight images have arrived
  uint64_t* bar = wbar + 1;                                   // the phase's product is complete
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool ctl = warp == 16;
  uint8_t* act = sm + S_ACT;
  if (tid == 0) {
    tc::mbar_init(wbar, 1);
    tc::mbar_init(bar, 1);
    tc::fence_mbar_init();
  }
  if (ctl) {
    tc::tmem_alloc(tslot, 512);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tslot, sa = tc::smem_u32(act);
  const int row = tid & 127, quarter = tid >> 7;   // of the sample threads: the sample, and its 32 of a layer's 128 features
  const long s = long(blockIdx.x) * GBM + row;
  float T[NLOSS];   // targets (threads of the first quarter)
  if (ctl && lane == 0) {
    tc::grid_wait();   // the images are the previous step's
    tc::mbar_expect_tx(wbar, uint32_t(S_ACT));
    tc::tma_load_2d(sm + S_W1, &M.f[0], wbar, 0, 0);
    for (int h = 0; h < 2; h++) {
      tc::tma_load_2d(sm + S_W2 + h * NH * 128, &M.f[1], wbar, h * GBK, 0);
      tc::tma_load_2d(sm + S_W3 + h * NH * 128, &M.f[2], wbar, h * GBK, 0);
      tc::tma_load_2d(sm + S_W4 + h * 16 * 128, &M.f[3], wbar, h * GBK, 0);
      tc::tma_load_2d(sm + S_W3T + h * NH * 128, &M.b[1], wbar, h * GBK, 0);
      tc::tma_load_2d(sm + S_W2T + h * NH * 128, &M.b[0], wbar, h * GBK, 0);
    }
    tc::tma_load_2d(sm + S_W4T, &M.b[2], wbar, 0, 0);
  } else if (quarter < 2) {
    // a sample: drawn by a hash of (step, sample) reduced to [0, npairs) (the same draw as the fp32 trainer's), its inputs
    // normalised to bf16 (8 of the 16 columns of K in each of two threads; 12 features, zeros past them)
    unsigned idx = unsigned(s);
    if (P.draw) {
      unsigned h = unsigned(s) * 0x9E3779B1u ^ (P.step * 0x85EBCA77u + P.seed);
      h ^= h >> 16; h *= 0x7FEB352Du; h ^= h >> 15; h *= 0x846CA68Bu; h ^= h >> 16;
      idx = unsigned((uint64_t(h) * P.npairs) >> 32);
    }
    const float* p = P.pairs + size_t(idx) * PAIR;
    __align__(16) __nv_bfloat16 x8[8];   // (the previous step has been done with Xt since before its last kernel began)
    if (quarter == 0) {
#pragma unroll
      for (int i = 0; i < 8; i++) x8[i] = __float2bfloat16_rn((feature(i, p[i]) - P.nm.in_mean[i]) * P.nm.in_scale[i]);
#pragma unroll
      for (int i = 0; i < 8; i++) P.Xt[size_t(i) * P.B + s] = x8[i];
#pragma unroll
      for (int j = 0; j < NLOSS; j++) T[j] = P.nm.out_scale[j] > 0.f ? p[NIN + j] / P.nm.out_scale[j] : 0.f;
    } else {
#pragma unroll
      for (int i = 8; i < 16; i++)
        x8[i - 8] = __float2bfloat16_rn(i < NIN ? (feature(i, p[i]) - P.nm.in_mean[i]) * P.nm.in_scale[i] : 0.f);
#pragma unroll
      for (int i = 8; i < NIN; i++) P.Xt[size_t(i) * P.B + s] = x8[i - 8];
    }
    *reinterpret_cast<uint4*>(act + swz(row, quarter * 8, GBM)) = *reinterpret_cast<const uint4*>(x8);
  }
  tc::grid_wait();
  tc::grid_release();
  // the phases: the control warp multiplies the activation tile, the sample threads turn the product into the next tile
  const uint32_t trow = tmem + (uint32_t((warp & 3) * 32) << 16), D = 3 * NH;   // TMEM columns: Z1, Z2, Z3, D
  const int c0 = quarter * 32;
  bool ok = true;
  for (int ph = 0; ph < 7; ph++) {
    if (!ctl) tc::fence_proxy_async_smem();
    tc::tc_fence_before();
    __syncthreads();
    if (ctl) {
      if (lane == 0) {
        if (ph == 0) ok = tc::mbar_wait(wbar, 0, err, 1u);   // without weights no product is begun
        tc::tc_fence_after();
        const uint32_t sw = tc::smem_u32(sm);
        if (ok) switch (ph) {   // the first layer has 12 inputs, dY 10 outputs: one step of K (the rest of their images is zero)
          case 0: issue_layer(tmem, sa, sw + S_W1, NH, 16, NH, bar); break;
          case 1: issue_layer(tmem + NH, sa, sw + S_W2, NH, NH, NH, bar); break;
          case 2: issue_layer(tmem + 2 * NH, sa, sw + S_W3, NH, NH, NH, bar); break;
          case 3: issue_layer(tmem + D, sa, sw + S_W4, 16, NH, 16, bar); break;
          case 4: issue_layer(tmem + D, sa, sw + S_W4T, NH, 16, NH, bar); break;
          case 5: issue_layer(tmem + D, sa, sw + S_W3T, NH, NH, NH, bar); break;
          default: issue_layer(tmem + D, sa, sw + S_W2T, NH, NH, NH, bar); break;
        }
      }
      __syncwarp();
      continue;
    }
    if (ok) ok = tc::mbar_wait_warp(bar, uint32_t(ph & 1), err, 4u);
    tc::tc_fence_after();
    if (ph < 3) {   // hidden layer: bias, GELU; its derivative takes Z's place in TMEM for the way back
      const float* bias = P.w + (ph == 0 ? OB1 : ph == 1 ? OB2 : OB3) + c0;
      float v[32], gp[32];
      tc::tmem_ld32(trow + uint32_t(ph * NH + c0), v);
#pragma unroll
      for (int e = 0; e < 32; e++) {
        const float z = v[e] + tc::ld_late(bias + e);
        v[e] = gelu(z);
        gp[e] = gelu_grad(z);
      }
      tmem_st32(trow + uint32_t(ph * NH + c0), gp);
      if (ok) put_features(act, P.Ht[ph], P.B, row, c0, s, lane, v);
    } else if (ph == 3) {   // N = 16 columns, 10 outputs, the first NLOSS in the loss
      if (quarter == 0) {
        float y[16];
        tmem_ld16x(trow + D, y);
        double l = 0.0;
        if (ok) {
          float dy[16];
#pragma unroll
          for (int e = 0; e < 16; e++) {
            float d = 0.f;
            if (e < NLOSS) d = y[e] + tc::ld_late(P.w + OB4 + e) - T[e < NLOSS ? e : 0];
            l += double(d) * d;
            dy[e] = P.inv * d;
          }
          act8(act, row, 0, dy);
          act8(act, row, 8, dy + 8);
#pragma unroll
          for (int e = 0; e < 16; e++) P.dYt[long(e) * P.B + s] = __float2bfloat16_rn(dy[e]);
        }
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if (lane == 0) lred[warp] = l;
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (tid == 0) P.lossp[blockIdx.x] = lred[0] + lred[1] + lred[2] + lred[3];
      }
    } else {   // backward: dZ = dH * GELU'(Z) of layer 6 - ph
      const int l = 6 - ph;
      float v[32], gp[32];
      tc::tmem_ld32(trow + uint32_t(D + c0), v);
      tc::tmem_ld32(trow + uint32_t(l * NH + c0), gp);
#pragma unroll
      for (int e = 0; e < 32; e++) v[e] *= gp[e];
      if (ok) put_features(l > 0 ? act : nullptr, P.dZt[l], P.B, row, c0, s, lane, v);
    }
  }
  // every product is complete once the sample threads have waited for the last one; where a wait ran out, what is in flight gets
  // that long again before its memory is given up
  if (ctl && lane == 0) tc::mbar_wait(ok ? bar : wbar, 0, err, ok ? 4u : 1u);
  tc::tc_fence_before();
  __syncthreads();
  if (ctl) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem, 512);
  }
}

// the four weight gradients at once: blockIdx.y = problem, blockIdx.x = batch split (ktiles stages of 64 samples),
// blockIdx.z = input features 0..79 or 64..143 (each output element sums the same products in the same order as in one
// tile of 144; the overlap is written once)
__global__ void __launch_bounds__(WTHREADS, 1) k_mlp_wgrad(const __grid_constant__ WgradSet S, int ktiles, unsigned int* err) {
  extern __shared__ uint8_t smraw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smraw) + 1023) & ~uintptr_t(1023));
  const int p = blockIdx.y, z = blockIdx.x, NT = S.N[p], n0 = int(blockIdx.z) * 64, N = NT < WN ? NT : WN;
  if (n0 >= NT) return;
  uint64_t* full = reinterpret_cast<uint64_t*>(sm + WSTAGES * WSTAGE);
  uint64_t* empty = full + WSTAGES;
  uint64_t* accf = empty + WSTAGES;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(accf + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < WSTAGES; s++) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    tc::mbar_init(accf, 1);
    tc::fence_mbar_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(tslot, 128);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tslot;
  tc::grid_wait();
  tc::grid_release();
  const int kel0 = z * ktiles * GBK;
  bool ok = true;
  if (warp == 0 && lane == 0) {
    const uint32_t bytes = uint32_t(WA_BYTES + N * GBK * 2);
    for (int t = 0; t < ktiles; t++) {
      const int s = t % WSTAGES;
      if (!tc::mbar_wait(&empty[s], (uint32_t(t / WSTAGES) & 1u) ^ 1u, err, 1u)) break;
      tc::mbar_expect_tx(&full[s], bytes);
      tc::tma_load_2d(sm + s * WSTAGE, &S.a[p], &full[s], kel0 + t * GBK, 0);
      tc::tma_load_2d(sm + s * WSTAGE + WA_BYTES, &S.b[p], &full[s], kel0 + t * GBK, n0);
    }
  } else if (warp == 1 && lane == 0) {
    const uint32_t idesc = tc::idesc_bf16_f32(GBM, N);
    for (int t = 0; t < ktiles; t++) {
      const int s = t % WSTAGES;
      if (!tc::mbar_wait(&full[s], uint32_t(t / WSTAGES) & 1u, err, 2u)) break;
      tc::tc_fence_after();
      const uint32_t a = tc::smem_u32(sm + s * WSTAGE), b = a + WA_BYTES;
#pragma unroll
      for (int kk = 0; kk < GBK / 16; kk++)
        tc::mma_bf16(tmem, tc::desc_k_sw128(a + kk * 32), tc::desc_k_sw128(b + kk * 32), idesc, (t > 0 || kk > 0) ? 1u : 0u);
      tc::mma_commit(&empty[s]);
    }
    tc::mma_commit(accf);
  }
  if (warp >= 2) {
    ok = tc::mbar_wait_warp(accf, 0, err, 4u);
    tc::tc_fence_after();
    const int q = warp & 3, row = q * 32 + lane;
    const uint32_t trow = tmem + (uint32_t(q * 32) << 16);
    float* out = S.part[p] + (long(z) * GBM + row) * NT + n0;
#pragma unroll 1
    for (int c0 = n0 ? WN - 64 : 0; c0 < N; c0 += 16) {
      float v[16];
      tmem_ld16x(trow + uint32_t(c0), v);
      if (!ok) continue;
#pragma unroll
      for (int e = 0; e < 16; e += 4) *reinterpret_cast<float4*>(out + c0 + e) = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem, 128);
  }
}

// bf16 images of the weights, both ways: W1i [128][64], W2i / W3i [128][128], W4i [16][128] (forward, K-major over
// the inputs) and W2T / W3T [128][128], W4T [128][64] (backward, K-major over the outputs); padding stays zero
struct Images {
  __nv_bfloat16 *w1, *w2, *w3, *w4, *w2t, *w3t, *w4t;
};
__device__ __forceinline__ void put_image(const Images& im, int t, float w) {
  const __nv_bfloat16 b = __float2bfloat16_rn(w);
  if (t < OB1) { const int j = t / NIN, i = t - j * NIN; im.w1[j * KPAD + i] = b; }
  else if (t >= OW2 && t < OB2) { const int j = (t - OW2) / NH, i = (t - OW2) % NH; im.w2[j * NH + i] = b; im.w2t[i * NH + j] = b; }
  else if (t >= OW3 && t < OB3) { const int j = (t - OW3) / NH, i = (t - OW3) % NH; im.w3[j * NH + i] = b; im.w3t[i * NH + j] = b; }
  else if (t >= OW4 && t < OB4) { const int j = (t - OW4) / NH, i = (t - OW4) % NH; im.w4[j * NH + i] = b; im.w4t[i * KPAD + j] = b; }
}
__global__ void k_images(const float* __restrict__ w, Images im) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < NPARAM) put_image(im, t, w[t]);
}
struct Adam {
  float *w, *m, *v;   // null w: the gradient alone
  float lr, b1, b2, eps, c1, c2;
};
struct Parts {
  const float* p[4];   // the partial slices of the four layers
  int nsplit;
};
// gradient of parameter t = sum over the splits, in split order, of its element of the partial slices; then its Adam
// step. The last block adds the loss: += (the per-tile partials, summed in tile order) / (B * NLOSS)
__global__ void __launch_bounds__(256) k_grad_adam(Parts S, float* __restrict__ g, Adam A, Images im, const double* __restrict__ lossp,
                                                   int tiles, long B, double* __restrict__ loss) {
  tc::grid_wait();
  tc::grid_release();
  if (blockIdx.x == gridDim.x - 1) {
    if (threadIdx.x == 0) {
      double l = 0.0;
#pragma unroll 16
      for (int i = 0; i < tiles; i++) l += lossp[i];
      *loss += l / double(B * NLOSS);
    }
    return;
  }
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= NPARAM) return;
  const float* part;
  int N, j, n;
  if (t < OB1) { part = S.p[0]; N = NXX; j = t / NIN; n = t - j * NIN; }
  else if (t < OW2) { part = S.p[0]; N = NXX; j = t - OB1; n = NIN; }
  else if (t < OB2) { part = S.p[1]; N = NHX; j = (t - OW2) / NH; n = (t - OW2) % NH; }
  else if (t < OW3) { part = S.p[1]; N = NHX; j = t - OB2; n = NH; }
  else if (t < OB3) { part = S.p[2]; N = NHX; j = (t - OW3) / NH; n = (t - OW3) % NH; }
  else if (t < OW4) { part = S.p[2]; N = NHX; j = t - OB3; n = NH; }
  else if (t < OB4) { part = S.p[3]; N = NHX; j = (t - OW4) / NH; n = (t - OW4) % NH; }
  else { part = S.p[3]; N = NHX; j = t - OB4; n = NH; }
  float gi = 0.f;
#pragma unroll 16
  for (int z = 0; z < S.nsplit; z++) gi += tc::ld_late(part + (long(z) * GBM + j) * N + n);
  g[t] = gi;
  if (!A.w) return;
  const float mi = A.b1 * A.m[t] + (1.f - A.b1) * gi, vi = A.b2 * A.v[t] + (1.f - A.b2) * gi * gi;
  A.m[t] = mi;
  A.v[t] = vi;
  const float wi = A.w[t] - A.lr * (mi / A.c1) / (sqrtf(vi / A.c2) + A.eps);
  A.w[t] = wi;
  put_image(im, t, wi);
}
__global__ void k_fill_bf16(__nv_bfloat16* p, long n, float v) {
  for (long i = blockIdx.x * long(blockDim.x) + threadIdx.x; i < n; i += long(gridDim.x) * blockDim.x) p[i] = __float2bfloat16_rn(v);
}

}  // namespace mlp

// ---------------------------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------------------------
namespace {
typedef CUresult (*PFN_encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
PFN_encode encoder() {
  static PFN_encode fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_encode>(p);
  }
  return fn;
}
// K-major bf16 operand [rows][cols] (pitch cols), box 64 columns x box_rows, 128-byte swizzle
bool kmap(CUtensorMap* m, const void* base, long rows, long cols, int box_rows) {
  PFN_encode enc = encoder();
  if (!enc) return false;
  cuuint64_t dims[2] = {cuuint64_t(cols), cuuint64_t(rows)};
  cuuint64_t strides[1] = {cuuint64_t(cols * 2)};
  cuuint32_t box[2] = {cuuint32_t(mlp::GBK), cuuint32_t(box_rows)};
  cuuint32_t es[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
}  // namespace

struct MlpTcTrainer {
  long B = 0;     // batch the buffers and maps are made for
  __nv_bfloat16 *Xt = nullptr, *Ht[3] = {}, *dYt = nullptr, *dZt[3] = {};
  __nv_bfloat16* img = nullptr;
  mlp::Images im{};
  float* part[4] = {};
  double* lossp = nullptr;
  unsigned int* err = nullptr;
  int nsplit = 1, wktiles = 1;
  mlp::StepMaps M{};
  mlp::WgradSet W{};
};

namespace mlp {
namespace {
int ok_or(bool ok, const char* what) {
  if (ok) return OB_OK;
  set_error("mlp tensor-core training: %s", what);
  return OB_ERR_DEVICE;
}
void free_all(MlpTcTrainer* t) {
  std::vector<void*> ps = {t->Xt, t->dYt, t->img, t->lossp, t->err};
  for (int l = 0; l < 3; l++) { ps.push_back(t->Ht[l]); ps.push_back(t->dZt[l]); }
  for (int p = 0; p < 4; p++) ps.push_back(t->part[p]);
  for (void* p : ps)
    if (p) cudaFree(p);
  *t = MlpTcTrainer();
}
}  // namespace

// buffers and tensor maps for batches of B samples (B a multiple of 128)
int tc_train_prepare(MlpTcTrainer* t, long B, const float* d_w, cudaStream_t s) {
  if (B % GBM != 0 || B < GBM) { set_error("mlp tensor-core training: the batch must be a positive multiple of 128"); return OB_ERR_INVALID; }
  if (B == t->B) return OB_OK;
  free_all(t);
  bool ok = true;
  auto al = [&](void** p, size_t bytes) { ok = ok && cudaMalloc(p, bytes) == cudaSuccess && cudaMemsetAsync(*p, 0, bytes, s) == cudaSuccess; };
  const size_t b = size_t(B);
  al((void**)&t->Xt, NXX * b * 2);
  al((void**)&t->dYt, GBM * b * 2);
  for (int l = 0; l < 3; l++) {
    al((void**)&t->Ht[l], NHX * b * 2);
    al((void**)&t->dZt[l], GBM * b * 2);
  }
  const size_t img = size_t(NH) * KPAD + 2 * NH * NH + 16 * NH + 2 * NH * NH + NH * KPAD;
  al((void**)&t->img, img * 2);
  al((void**)&t->lossp, (b / GBM) * 8);
  al((void**)&t->err, 16);
  // weight gradients: at most WSPLIT_MAX batch splits of whole 64-sample stages
  const int kt = int(B / GBK);
  t->nsplit = 1;
  for (int d = WSPLIT_MAX; d >= 1; d--)
    if (kt % d == 0) { t->nsplit = d; break; }
  t->wktiles = kt / t->nsplit;
  for (int p = 0; p < 4; p++) al((void**)&t->part[p], size_t(t->nsplit) * GBM * NHX * 4);
  if (!ok) { free_all(t); set_error("mlp tensor-core training: out of device memory"); return OB_ERR_OOM; }
  t->B = B;
  __nv_bfloat16* q = t->img;
  t->im.w1 = q; q += NH * KPAD;
  t->im.w2 = q; q += NH * NH;
  t->im.w3 = q; q += NH * NH;
  t->im.w4 = q; q += 16 * NH;
  t->im.w2t = q; q += NH * NH;
  t->im.w3t = q; q += NH * NH;
  t->im.w4t = q;
  // the rows of ones that make the weight-gradient GEMMs return the bias gradients
  k_fill_bf16<<<64, 256, 0, s>>>(t->Xt + size_t(NIN) * b, long(b), 1.f);
  for (int l = 0; l < 3; l++) k_fill_bf16<<<64, 256, 0, s>>>(t->Ht[l] + size_t(NH) * b, long(b), 1.f);
  k_images<<<(NPARAM + 255) / 256, 256, 0, s>>>(d_w, t->im);
  // the images as B operands: forward W1 .. W4, backward W2^T, W3^T, W4^T
  ok = kmap(&t->M.f[0], t->im.w1, NH, KPAD, NH) && kmap(&t->M.f[1], t->im.w2, NH, NH, NH) && kmap(&t->M.f[2], t->im.w3, NH, NH, NH) &&
       kmap(&t->M.f[3], t->im.w4, 16, NH, 16) && kmap(&t->M.b[0], t->im.w2t, NH, NH, NH) && kmap(&t->M.b[1], t->im.w3t, NH, NH, NH) &&
       kmap(&t->M.b[2], t->im.w4t, NH, KPAD, NH);
  // weight gradients: A = dZ^T / dY^T [128][B], B = [H, 1]^T / [X, 1]^T [N][B]
  ok = ok && kmap(&t->W.a[0], t->dZt[0], GBM, B, GBM) && kmap(&t->W.b[0], t->Xt, NXX, B, NXX);
  ok = ok && kmap(&t->W.a[1], t->dZt[1], GBM, B, GBM) && kmap(&t->W.b[1], t->Ht[0], NHX, B, WN);
  ok = ok && kmap(&t->W.a[2], t->dZt[2], GBM, B, GBM) && kmap(&t->W.b[2], t->Ht[1], NHX, B, WN);
  ok = ok && kmap(&t->W.a[3], t->dYt, GBM, B, GBM) && kmap(&t->W.b[3], t->Ht[2], NHX, B, WN);
  t->W.N[0] = NXX; t->W.N[1] = t->W.N[2] = t->W.N[3] = NHX;
  for (int p = 0; p < 4; p++) t->W.part[p] = t->part[p];
  cudaFuncSetAttribute(k_mlp_step, cudaFuncAttributeMaxDynamicSharedMemorySize, STEP_SMEM);
  cudaFuncSetAttribute(k_mlp_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, WSMEM);
  return ok_or(ok, "tensor map encoding failed");
}

// one step on t->B samples at the parameters w: the gradient into g, the loss added into *loss, then Adam (A.w not null)
static void tc_step(MlpTcTrainer* t, const float* w, float* g, const float* pairs, const Norm& nm, bool draw, unsigned npairs, unsigned step,
                    unsigned seed, const Adam& A, double* loss, cudaStream_t s) {
  const long B = t->B;
  const int tiles = int(B / GBM);
  StepArgs P{};
  P.pairs = pairs;
  P.npairs = npairs;
  P.step = step;
  P.seed = seed;
  P.draw = draw ? 1 : 0;
  P.B = B;
  P.nm = nm;
  P.w = w;
  P.Xt = t->Xt;
  P.dYt = t->dYt;
  for (int l = 0; l < 3; l++) {
    P.Ht[l] = t->Ht[l];
    P.dZt[l] = t->dZt[l];
  }
  P.lossp = t->lossp;
  P.inv = 2.f / float(B * NLOSS);
  // each kernel sets itself up (and draws its samples) under the tail of the one before
  tc::launch_early(true, k_mlp_step, tiles, STEP_THREADS, STEP_SMEM, s, t->M, P, t->err);
  tc::launch_early(true, k_mlp_wgrad, dim3(t->nsplit, 4, 2), WTHREADS, WSMEM, s, t->W, t->wktiles, t->err);
  const Parts S{{t->part[0], t->part[1], t->part[2], t->part[3]}, t->nsplit};
  tc::launch_early(true, k_grad_adam, (NPARAM + 255) / 256 + 1, 256, 0, s, S, g, A, t->im, t->lossp, tiles, B, loss);
}

// ---- entry points for ob_mlp.cu (the network's handle owns one trainer) ----
MlpTcTrainer* tc_trainer_new() { return new MlpTcTrainer(); }
void tc_trainer_delete(MlpTcTrainer* t) {
  if (!t) return;
  free_all(t);
  delete t;
}

static int tc_check_err(MlpTcTrainer* t, cudaStream_t s) {
  unsigned h = 0;
  if (cudaMemcpyAsync(&h, t->err, 4, cudaMemcpyDeviceToHost, s) != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess) {
    set_error("mlp tensor-core training: %s", cudaGetErrorString(cudaGetLastError()));
    return OB_ERR_DEVICE;
  }
  if (h) {
    cudaMemsetAsync(t->err, 0, 4, s);
    set_error("mlp tensor-core training: a pipeline wait timed out (code %u)", h);
    return OB_ERR_TIMEOUT;
  }
  return OB_OK;
}

// `steps` Adam steps on random batches of `batch` recorded pairs; the loss of every step is added into *d_loss
int tc_train_run(MlpTcTrainer* t, float* w, float* g, float* m, float* v, int& adam_t, const float* pairs, unsigned npairs,
                 const Norm& nm, int batch, int steps, float lr, unsigned seed, double* d_loss, cudaStream_t s) {
  int rc = tc_train_prepare(t, batch, w, s);
  if (rc != OB_OK) return rc;
  k_images<<<(NPARAM + 255) / 256, 256, 0, s>>>(w, t->im);   // the parameters may have been set since the last run
  const float b1 = 0.9f, b2 = 0.999f;
  for (int st = 0; st < steps; st++) {
    const unsigned step = unsigned(adam_t);
    adam_t++;
    const float c1 = 1.f - std::pow(b1, float(adam_t)), c2 = 1.f - std::pow(b2, float(adam_t));
    tc_step(t, w, g, pairs, nm, true, npairs, step, seed, Adam{w, m, v, lr, b1, b2, 1e-8f, c1, c2}, d_loss, s);
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("mlp tensor-core training launch: %s", cudaGetErrorString(e));
    return OB_ERR_DEVICE;
  }
  return tc_check_err(t, s);
}

// loss (added into *d_loss) and gradient g of `count` pairs in order (count a multiple of 128), at the parameters w
int tc_grad_run(MlpTcTrainer* t, const float* w, float* g, const float* pairs, int count, const Norm& nm, double* d_loss,
                cudaStream_t s) {
  int rc = tc_train_prepare(t, count, w, s);
  if (rc != OB_OK) return rc;
  k_images<<<(NPARAM + 255) / 256, 256, 0, s>>>(w, t->im);
  tc_step(t, w, g, pairs, nm, false, 0, 0, 0, Adam{}, d_loss, s);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("mlp tensor-core gradient launch: %s", cudaGetErrorString(e));
    return OB_ERR_DEVICE;
  }
  return tc_check_err(t, s);
}

}  // namespace mlp
}  // namespace ob
