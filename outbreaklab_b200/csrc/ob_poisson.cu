// ob_poisson.cu — exact anelastic pressure solve on the padded grid (solver.js:1-165), sm_100a.
//
//   rho_c(z) lap_h(phi) + d/dz(rho_w(z) d phi/dz) = rhs,  phi = 0 beyond the lateral faces, Neumann at ground / lid.
//
// Orthonormal DST-II in x and y (four dense transforms), one tridiagonal per horizontal mode (l, m) in z.
//   precision 0: fp32 SIMT transforms (tiled GEMM, fp32 FMA) — the reference's own precision;
//   precision 1: bf16x3 tensor-core transforms (ob_dst_tc.cu) with fp32 accumulation; 2: plus a bf16x3
//   refinement sweep on the FP64-accumulated residual; 3: that sweep in plain bf16.
// The tridiagonals: fp32 Thomas with the column in shared memory for every mode except the lowest
// 2 x 2 modes, which are near-singular (Neumann in z, shift ~ -(pi/L)^2) and run in FP64.
#include <cstdio>
#include <cmath>
#include <cstdint>
#include <vector>

#include "ob_poisson.cuh"

namespace ob {

// ---------------------------------------------------------------------------------------------------------------
// fp32 transforms as SIMT GEMMs: C(r, c) = sum_q R(r, q) B(q, c), one fmaf chain per output with q ascending, so no
// tile shape or split changes a bit of the result.
//
// What bounds it is the fp32 pipe next to shared-memory reads, which deliver 128 bytes per clock and SM whether or not
// lanes share an address: a thread that owns r x c outputs reads 4 (r + c) bytes per r c FMAs. 8 x 8 outputs per thread
// would need all of it, 16 x 4 more (measured: shared memory 86 % busy, 390 us per transform at 464 x 464 x 60), 16 x 8
// needs three quarters: 288 us there (under ncu; the fp32 pipe 67-74 % busy, shared memory 60 %), against 546 us for
// 64 x 64 tiles with 4 x 4 outputs per thread; a whole solve 2.08 -> 1.06 ms. The rows a thread owns are read as float4,
// which are the register pairs of the packed fma.rn.f32x2 (two fmaf in one instruction, each rounded as fmaf is, and
// half the issue slots), the columns as float2. Tiles: BR = 32 GR rows (the output's contiguous dimension) x BC = 16 CPT
// columns by 4 warps that share all the rows and own 4 CPT columns each; the side that spans the DST matrix is 96 or
// 128 wide, whichever pads its extent less (656 = 6.8 x 96, but 5.1 x 128). A ring of GST stages of GBK q-values is
// filled by 4-byte cp.async (zero beyond the edges), which transposes into [q][row] on the way and asks nothing of the
// alignment of the caller's pointers or of odd row lengths.
// ---------------------------------------------------------------------------------------------------------------
constexpr int GBK = 16, GST = 4, GTH = 128;
__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool in) {
  const uint32_t d = uint32_t(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(in ? 4 : 0) : "memory");
}
// acc.{x,y} += a.{x,y} * b, each as fmaf
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
template <int GR, int CPT>
constexpr int gemm_smem_bytes() { return GST * GBK * (32 * GR + 4 + 16 * CPT + 4) * 4; }

// XT: x-transform. Rows = outputs l of the matrix Mx[l][q], columns = field rows (j, k): B(q, c) = src[q + K c],
//     C[l + nx c].
// otherwise y-transform. Rows = (k, i) of the field: R(r, q) = src[i + nx q + pl k]; columns = outputs m of the matrix
//     My[m][q], C[i + nx m + pl k].
template <bool XT, int GR, int CPT>
__global__ void __launch_bounds__(GTH, GR == 2 ? 4 : 2)
    k_gemm_f32(int M, int N, int K, const float* __restrict__ mat, const float* __restrict__ src, float* __restrict__ C, int nx, long pl, int mtiles) {
  static_assert(XT || GTH % (32 * GR) == 0, "the y-transform loads one field row per thread");
  constexpr int BR = 32 * GR, BC = 16 * CPT, LR = BR + 4, LC = BC + 4, STG = GBK * (LR + LC), YQ = GTH / BR;
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lx = lane & 7, ly = lane >> 3;
  // the matrix's tiles vary fastest, so that blocks running together share a field tile through L2
  const int bm = int(blockIdx.x % unsigned(mtiles)), bf = int(blockIdx.x / unsigned(mtiles));
  const int r0 = (XT ? bm : bf) * BR, c0 = (XT ? bf : bm) * BC;
  // this thread's cp.async lines: K-contiguous operands take (q = tid & 15, 8 lines per pass); the y-transform's field
  // rows take row tid % BR, YQ q-values per pass
  const int kq = tid & 15, kl = tid >> 4;
  const float* rbase;   // rows operand
  bool rin = true;
  if (XT) {
    rbase = mat + long(r0 + kl) * K + kq;
  } else {
    const int r = r0 + tid % BR;
    rin = r < M;
    const int k = r / nx, i = r - k * nx;
    rbase = src + (rin ? long(k) * pl + i : 0);
  }
  const float* cbase = (XT ? src : mat) + long(c0 + kl) * K + kq;
  auto load = [&](int kt) {
    float* s = sm + (kt % GST) * STG;
    const int q0 = kt * GBK;
    const bool qin = q0 + kq < K;
    if (XT) {
#pragma unroll
      for (int p = 0; p < BR / 8; p++) {
        const bool in = r0 + kl + 8 * p < M && qin;
        cp_async4(s + kq * LR + kl + 8 * p, in ? rbase + long(8 * p) * K + q0 : mat, in);
      }
    } else {
#pragma unroll
      for (int p = 0; p < GBK; p += YQ) {
        const int q = YQ == 1 ? p : p + tid / BR;
        const bool in = rin && q0 + q < K;
        cp_async4(s + q * LR + tid % BR, in ? rbase + long(q0 + q) * nx : src, in);
      }
    }
    float* sc = s + GBK * LR;
#pragma unroll
    for (int p = 0; p < BC / 8; p++) {
      const bool in = c0 + kl + 8 * p < N && qin;
      cp_async4(sc + kq * LC + kl + 8 * p, in ? cbase + long(8 * p) * K + q0 : mat, in);
    }
  };
  uint64_t acc[2 * GR][CPT];
#pragma unroll
  for (int a = 0; a < 2 * GR; a++)
#pragma unroll
    for (int c = 0; c < CPT; c++) acc[a][c] = 0ull;
  const int nk = (K + GBK - 1) / GBK;
#pragma unroll
  for (int t = 0; t < GST - 1; t++) {
    if (t < nk) load(t);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int kt = 0; kt < nk; kt++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(GST - 2) : "memory");
    __syncthreads();   // stage kt has arrived for every thread, and every thread is done with the stage refilled below
    if (kt + GST - 1 < nk) load(kt + GST - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* s = sm + (kt % GST) * STG;
    const float* rs = s + lx * 4;
    const float* cs = s + GBK * LR + warp * 4 * CPT + ly * 2;   // columns 8 h + 2 ly + {0, 1} of the warp's
#pragma unroll
    for (int kk = 0; kk < GBK; kk++) {
      ulonglong2 a[GR];
#pragma unroll
      for (int g = 0; g < GR; g++) a[g] = *reinterpret_cast<const ulonglong2*>(rs + kk * LR + 32 * g);
#pragma unroll
      for (int h = 0; h < CPT / 2; h++) {
        const float2 b = *reinterpret_cast<const float2*>(cs + kk * LC + 8 * h);
        uint64_t bx, by;
        asm("mov.b64 %0, {%1, %1};" : "=l"(bx) : "f"(b.x));
        asm("mov.b64 %0, {%1, %1};" : "=l"(by) : "f"(b.y));
#pragma unroll
        for (int g = 0; g < GR; g++) {
          fma2(acc[2 * g][2 * h], a[g].x, bx);
          fma2(acc[2 * g + 1][2 * h], a[g].y, bx);
          fma2(acc[2 * g][2 * h + 1], a[g].x, by);
          fma2(acc[2 * g + 1][2 * h + 1], a[g].y, by);
        }
      }
    }
  }
#pragma unroll
  for (int c = 0; c < CPT; c++) {
    const int col = c0 + warp * 4 * CPT + 8 * (c >> 1) + 2 * ly + (c & 1);
    if (col >= N) continue;
#pragma unroll
    for (int g = 0; g < GR; g++) {
      const int r = r0 + 32 * g + lx * 4;
      float v[4];
      asm("mov.b64 {%0, %1}, %2;" : "=f"(v[0]), "=f"(v[1]) : "l"(acc[2 * g][c]));
      asm("mov.b64 {%0, %1}, %2;" : "=f"(v[2]), "=f"(v[3]) : "l"(acc[2 * g + 1][c]));
      // four consecutive rows, which are consecutive outputs but where a plane of the y-transform ends
      float* o = XT ? C + long(col) * nx + r : C + long(r / nx) * pl + long(col) * nx + r % nx;
      if (r + 3 < M && (reinterpret_cast<uintptr_t>(o) & 15) == 0 && (XT || r % nx + 3 < nx)) {
        *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; e++)
          if (r + e < M) (XT ? C + long(col) * nx : C + long((r + e) / nx) * pl + long(col) * nx)[XT ? r + e : (r + e) % nx] = v[e];
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------
// tridiagonal solves per mode (solver.js:70-103); zop = (lo, up, diag, rho_c) per level
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ bool low_mode(int l, int m) { return l < 2 && m < 2; }

// One thread per mode, 64 modes in l per block. The column stays in shared memory between the sweeps (c' and d of every
// level, 512 nz bytes per block), so T2 is read once and written once, and a batch of levels is loaded ahead of the
// recurrence, whose two IEEE divisions per level are the rest of the time. The lowest 2 x 2 modes run in FP64 in their
// own threads of the same launch, their columns in cpd. 464 x 464 x 60: 61 us against 69 us for a kernel that kept c' and
// the column in global memory plus 47 us for the lowest modes in a launch of their own.
// 440 levels (220 KB) is what shared memory holds; there one block of two warps is all an SM has, and whether that still
// pays depends on the grid: whole solves at 440 levels against 441, which take k_tri_f32_any, 289 and 521 us at 64 x 64, 441 and
// 765 at 128 x 128, 1.86 and 1.97 ms at 240 x 240, but 9.7 and 8.3 at 464 x 464.
constexpr int kTriThreads = 64, kTriBatch = 16, kTriSmemLevels = 440;
__global__ void __launch_bounds__(kTriThreads) k_tri_f32(int nx, int ny, int nz, const float* __restrict__ lam,
                                                         const float4* __restrict__ zop, float* __restrict__ hat,
                                                         double* __restrict__ cpd) {
  extern __shared__ float tsm[];
  const int l = blockIdx.x * kTriThreads + threadIdx.x, m = blockIdx.y;
  if (l >= nx) return;
  const long sxy = long(nx) * ny;
  float* h = hat + l + long(nx) * m;
  float hv[kTriBatch], hn[kTriBatch];   // the batch being swept, the next one in flight
  auto fetch = [&](float (&to)[kTriBatch], int k0) {
#pragma unroll
    for (int u = 0; u < kTriBatch; u++) to[u] = k0 + u < nz ? h[sxy * (k0 + u)] : 0.f;
  };
  auto advance = [&](int k0) {
#pragma unroll
    for (int u = 0; u < kTriBatch; u++) hv[u] = hn[u];
    fetch(hn, k0 + kTriBatch);
  };
  fetch(hn, 0);
  if (low_mode(l, m)) {
    const double shift = double(lam[l]) + double(lam[nx + m]);
    double* cp = cpd + (m * 2 + l) * nz;
    double* dd = cpd + 4 * nz + (m * 2 + l) * nz;
    double cprev = 0.0, dprev = 0.0;
    for (int k0 = 0; k0 < nz; k0 += kTriBatch) {
      advance(k0);
#pragma unroll
      for (int u = 0; u < kTriBatch; u++) {
        if (k0 + u >= nz) break;
        const float4 o = __ldg(zop + k0 + u);
        const double den = double(o.z) + shift * double(o.w) - double(o.x) * cprev;
        cprev = double(o.y) / den;
        dprev = (double(hv[u]) - double(o.x) * dprev) / den;
        cp[k0 + u] = cprev;
        dd[k0 + u] = dprev;
      }
    }
    double above = dprev;
    h[sxy * (nz - 1)] = float(above);
#pragma unroll 8
    for (int k = nz - 2; k >= 0; k--) {
      above = dd[k] - cp[k] * above;
      h[sxy * k] = float(above);
    }
    return;
  }
  const float shift = __ldg(lam + l) + __ldg(lam + nx + m);
  float* cp = tsm + threadIdx.x;
  float* d = cp + nz * kTriThreads;
  float cprev = 0.f, dprev = 0.f;
  for (int k0 = 0; k0 < nz; k0 += kTriBatch) {
    advance(k0);
#pragma unroll
    for (int u = 0; u < kTriBatch; u++) {
      if (k0 + u >= nz) break;
      const float4 o = __ldg(zop + k0 + u);
      const float den = o.z + shift * o.w - o.x * cprev;
      cprev = o.y / den;
      dprev = (hv[u] - o.x * dprev) / den;
      cp[(k0 + u) * kTriThreads] = cprev;
      d[(k0 + u) * kTriThreads] = dprev;
    }
  }
  float above = dprev;
  h[sxy * (nz - 1)] = above;
#pragma unroll 4
  for (int k = nz - 2; k >= 0; k--) {
    above = d[k * kTriThreads] - cp[k * kTriThreads] * above;
    h[sxy * k] = above;
  }
}
// columns too long for shared memory: forward-sweep coefficients in a global scratch column
__global__ void k_tri_f32_any(int nx, int ny, int nz, const float* __restrict__ lam, const float4* __restrict__ zop,
                              float* __restrict__ hat, float* __restrict__ cpbuf) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x, m = blockIdx.y;
  if (l >= nx || low_mode(l, m)) return;
  const float shift = __ldg(lam + l) + __ldg(lam + nx + m);
  const long sxy = long(nx) * ny;
  float* h = hat + l + long(nx) * m;
  float* cp = cpbuf + l + long(nx) * m;
  float cprev = 0.f, dprev = 0.f;
  for (int k = 0; k < nz; k++) {
    const float4 o = __ldg(zop + k);
    const float den = o.z + shift * o.w - o.x * cprev;
    cprev = o.y / den;
    dprev = (h[sxy * k] - o.x * dprev) / den;
    cp[sxy * k] = cprev;
    h[sxy * k] = dprev;
  }
  float above = dprev;
  for (int k = nz - 2; k >= 0; k--) {
    above = h[sxy * k] - cp[sxy * k] * above;
    h[sxy * k] = above;
  }
}
// their lowest 2 x 2 modes in FP64 (one warp)
__global__ void k_tri_f64_low(int nx, int ny, int nz, const float* __restrict__ lam, const float4* __restrict__ zop,
                              float* __restrict__ hat, double* __restrict__ cpbuf) {
  const int t = threadIdx.x;
  const int l = t & 1, m = t >> 1;
  if (t >= 4 || l >= nx || m >= ny) return;
  const double shift = double(lam[l]) + double(lam[nx + m]);
  const long sxy = long(nx) * ny;
  float* h = hat + l + long(nx) * m;
  double* cp = cpbuf + t * nz;
  double* dd = cpbuf + 4 * nz + t * nz;
  double cprev = 0.0, dprev = 0.0;
  for (int k = 0; k < nz; k++) {
    const float4 o = zop[k];
    const double den = double(o.z) + shift * double(o.w) - double(o.x) * cprev;
    cprev = double(o.y) / den;
    dprev = (double(h[sxy * k]) - double(o.x) * dprev) / den;
    cp[k] = cprev;
    dd[k] = dprev;
  }
  double above = dprev;
  h[sxy * (nz - 1)] = float(above);
  for (int k = nz - 2; k >= 0; k--) {
    above = dd[k] - cp[k] * above;
    h[sxy * k] = float(above);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// plan
// ---------------------------------------------------------------------------------------------------------------
static int ck(cudaError_t e, const char* what) {
  if (e != cudaSuccess) {
    set_error("%s: %s", what, cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? OB_ERR_OOM : OB_ERR_DEVICE;
  }
  return OB_OK;
}

int PoissonPlan::create(int nx_, int ny_, int nz_, double dx_, double dz_, int precision_) {
  nx = nx_; ny = ny_; nz = nz_; dx = dx_; dz = dz_; precision = precision_;
  if (nx < 2 || ny < 2 || nz < 2 || nz > 4096) { set_error("poisson: bad size %d x %d x %d", nx, ny, nz); return OB_ERR_INVALID; }
  const size_t n = size_t(nx) * ny * nz;
  // DST-II matrices (solver.js:115-125), computed in f64 and stored f32 as the reference does
  std::vector<float> M(2 * size_t(nx) * nx + 2 * size_t(ny) * ny);
  auto dst = [&](int N, float* q, float* qi) {
    for (int i = 0; i < N; i++)
      for (int l = 0; l < N; l++) {
        const double c = std::sqrt((l == N - 1 ? 1.0 : 2.0) / N);
        const double v = c * std::sin(M_PI * (l + 1) * (i + 0.5) / N);
        q[size_t(i) * N + l] = float(v);
        qi[size_t(l) * N + i] = float(v);
      }
  };
  ofs_qix = 0;
  ofs_qx = size_t(nx) * nx;
  ofs_qiy = 2 * size_t(nx) * nx;
  ofs_qy = 2 * size_t(nx) * nx + size_t(ny) * ny;
  dst(nx, M.data() + ofs_qx, M.data() + ofs_qix);
  dst(ny, M.data() + ofs_qy, M.data() + ofs_qiy);
  std::vector<float> lamh(nx + ny);
  for (int l = 0; l < nx; l++) lamh[l] = float(-4.0 / (dx * dx) * std::pow(std::sin(M_PI * (l + 1) / (2.0 * nx)), 2));
  for (int m = 0; m < ny; m++) lamh[nx + m] = float(-4.0 / (dx * dx) * std::pow(std::sin(M_PI * (m + 1) / (2.0 * ny)), 2));
  int rc;
  if ((rc = ck(cudaMalloc(&mats, M.size() * sizeof(float)), "poisson mats"))) return rc;
  if ((rc = ck(cudaMalloc(&lam, lamh.size() * sizeof(float)), "poisson eig"))) return rc;
  if ((rc = ck(cudaMalloc(&zop, size_t(nz) * sizeof(float4)), "poisson zop"))) return rc;
  if (precision == 0) {   // the tensor-core precisions hold their fields in the buffers of tc_create
    if ((rc = fp32_prepare())) return rc;
    if ((rc = ck(cudaMalloc(&tmp, n * sizeof(float)), "poisson tmp"))) return rc;
    if ((rc = ck(cudaMalloc(&hat, n * sizeof(float)), "poisson hat"))) return rc;
    if ((rc = ck(cudaMalloc(&cpd, size_t(8) * nz * sizeof(double)), "poisson low-mode scratch"))) return rc;
    if (nz > kTriSmemLevels) {
      if ((rc = ck(cudaMalloc(&cpf, n * sizeof(float)), "poisson tri scratch"))) return rc;
    }
  }
  if ((rc = ck(cudaMemcpy(mats, M.data(), M.size() * sizeof(float), cudaMemcpyHostToDevice), "poisson upload"))) return rc;
  if ((rc = ck(cudaMemcpy(lam, lamh.data(), lamh.size() * sizeof(float), cudaMemcpyHostToDevice), "poisson upload"))) return rc;
  std::vector<float> rc1(nz, 1.f), rw1(nz + 1, 1.f);
  if ((rc = set_density(rc1.data(), rw1.data()))) return rc;
  if (precision >= 1) {
    if ((rc = tc_create())) return rc;
  }
  return OB_OK;
}

int PoissonPlan::set_density(const float* rhoC, const float* rhoW) {  // solver.js:139-146
  std::vector<float4> zo(nz);
  const double a = 1.0 / (dz * dz);
  for (int k = 0; k < nz; k++) {
    const double lo = k > 0 ? double(rhoW[k]) * a : 0.0, up = k < nz - 1 ? double(rhoW[k + 1]) * a : 0.0;
    zo[k] = make_float4(float(lo), float(up), float(-(lo + up)), rhoC[k]);
  }
  const int rc = ck(cudaMemcpy(zop, zo.data(), zo.size() * sizeof(float4), cudaMemcpyHostToDevice), "poisson setDensity");
  if (rc != OB_OK || !tc) return rc;
  return tc_factor_low();
}

void PoissonPlan::destroy() {
  tc_destroy();
  for (void* p : {(void*)mats, (void*)lam, (void*)zop, (void*)tmp, (void*)hat, (void*)cpf, (void*)cpd})
    if (p) cudaFree(p);
  mats = lam = tmp = hat = cpf = nullptr;
  zop = nullptr;
  cpd = nullptr;
}

// the width of the tiles that span n outputs of a DST matrix: 96 where that pads n less than 128 does
static bool narrow_tiles(int n) { return (n + 95) / 96 * 96 < (n + 127) / 128 * 128; }
// Tiles of 64 x 64 with 8 x 4 outputs per thread, where the wide ones would leave a third of the 148 SMs without a block: a
// block's time is then all there is, and a quarter of the outputs take a quarter of it. Whole solves, wide -> small: 128 x
// 128 x 28 (28 wide tiles) 103 -> 53 us, 64 x 64 x 56 (28) 74 -> 53, 64 x 300 x 28 (66 and 42) 122 -> 64, 192 x 192 x 28 (84)
// 108 -> 84, 224 x 224 x 28 (98) 144 -> 125; from there on the wide tiles' fewer reads of shared memory tell: 256 x 256 x
// 28 (112) 159 -> 167, 464 x 464 x 60 (1090) 1165 -> 1428.
constexpr int kFewTiles = 98;
static bool small_tiles(int n, int rows) {
  const int t = narrow_tiles(n) ? 96 : 128;
  return long((n + t - 1) / t) * ((rows + 127) / 128) <= kFewTiles;
}
template <bool XT, int GR, int CPT>
static void launch_gemm(int M, int N, int K, const float* mat, const float* src, float* dst, int nx, long pl, cudaStream_t s) {
  const int rt = (M + 32 * GR - 1) / (32 * GR), ct = (N + 16 * CPT - 1) / (16 * CPT);
  k_gemm_f32<XT, GR, CPT><<<unsigned(rt) * unsigned(ct), GTH, gemm_smem_bytes<GR, CPT>(), s>>>(M, N, K, mat, src, dst, nx, pl, XT ? rt : ct);
}
// a function's attributes belong to the device that is current
int fp32_prepare() {
  const auto smem = [](auto* k, int bytes) { return ck(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes), "poisson fp32 kernels"); };
  int rc = smem(k_gemm_f32<true, 4, 8>, gemm_smem_bytes<4, 8>());
  if (rc == OB_OK) rc = smem(k_gemm_f32<true, 3, 8>, gemm_smem_bytes<3, 8>());
  if (rc == OB_OK) rc = smem(k_gemm_f32<false, 4, 8>, gemm_smem_bytes<4, 8>());
  if (rc == OB_OK) rc = smem(k_gemm_f32<false, 4, 6>, gemm_smem_bytes<4, 6>());
  if (rc == OB_OK) rc = smem(k_tri_f32, kTriSmemLevels * kTriThreads * 8);
  return rc;
}
// x-transform (solver.js mode 0): dst(l, col) = sum_i M(l, i) src(i, col), col = j + ny k
void PoissonPlan::gemm_x(const float* Mx, const float* src, float* dst, cudaStream_t s) const {
  if (small_tiles(nx, ny * nz)) launch_gemm<true, 2, 4>(nx, ny * nz, nx, Mx, src, dst, nx, 0, s);
  else if (narrow_tiles(nx)) launch_gemm<true, 3, 8>(nx, ny * nz, nx, Mx, src, dst, nx, 0, s);
  else launch_gemm<true, 4, 8>(nx, ny * nz, nx, Mx, src, dst, nx, 0, s);
}
// y-transform (mode 1), per plane k: dst(i, m) = sum_j src(i, j) M(m, j)
void PoissonPlan::gemm_y(const float* My, const float* src, float* dst, cudaStream_t s) const {
  const long pl = long(nx) * ny;
  if (small_tiles(ny, nx * nz)) launch_gemm<false, 2, 4>(nx * nz, ny, ny, My, src, dst, nx, pl, s);
  else if (narrow_tiles(ny)) launch_gemm<false, 4, 6>(nx * nz, ny, ny, My, src, dst, nx, pl, s);
  else launch_gemm<false, 4, 8>(nx * nz, ny, ny, My, src, dst, nx, pl, s);
}
void PoissonPlan::tri(float* h, cudaStream_t s) const {
  if (nz <= kTriSmemLevels) {
    k_tri_f32<<<dim3((nx + kTriThreads - 1) / kTriThreads, ny), kTriThreads, size_t(nz) * kTriThreads * 8, s>>>(nx, ny, nz, lam, zop, h, cpd);
    return;
  }
  k_tri_f32_any<<<dim3((nx + 127) / 128, ny, 1), 128, 0, s>>>(nx, ny, nz, lam, zop, h, cpf);
  k_tri_f64_low<<<1, 32, 0, s>>>(nx, ny, nz, lam, zop, h, cpd);
}

int PoissonPlan::solve(const float* rhs, float* phi, cudaStream_t s) {
  if (precision >= 1) return tc_solve(rhs, phi, s);
  gemm_x(mats + ofs_qix, rhs, tmp, s);
  gemm_y(mats + ofs_qiy, tmp, hat, s);
  tri(hat, s);
  gemm_y(mats + ofs_qy, hat, tmp, s);
  gemm_x(mats + ofs_qx, tmp, phi, s);
  return ck(cudaGetLastError(), "poisson solve launch");
}

}  // namespace ob
