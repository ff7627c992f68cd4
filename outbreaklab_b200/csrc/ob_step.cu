// ob_step.cu — the storm-model step kernels for sm_100a (one kernel per pass of model.js:1457-1472).
//
// Each kernel restates one WGSL pass of the reference (citations per kernel) over the structure-of-arrays layout of
// ob_common.cuh: one thread per texel, x fastest within a warp so that every stencil row is a coalesced 128-byte
// read, neighbours served from L1/L2. Semi-Lagrangian sampling is a software trilinear filter in fp32 (exact
// weights; WebGPU's hardware filter uses low-precision fixed-point weights, which are not reproduced).
#include <algorithm>
#include <vector>

#include "ob_common.cuh"
#include "ob_micro.cuh"
#include "ob_tc.cuh"
#include "ob_step.cuh"

namespace ob {

// reads of what the pass just before has written (ldo, gather8)
using tc::ld_late;
__device__ __forceinline__ float ldo_late(const float* f, unsigned b) { return ld_late(reinterpret_cast<const float*>(reinterpret_cast<const char*>(f) + b)); }
__device__ __forceinline__ float gather8_late(const float* f, const Corners& t) {
  return lerp8(t, ldo_late(f, t.a), ldo_late(f, t.b), ldo_late(f, t.c), ldo_late(f, t.d), ldo_late(f, t.e), ldo_late(f, t.h), ldo_late(f, t.k),
               ldo_late(f, t.l));
}

// members of the grouped launches (ensemble steps), uploaded by group_upload_members. A grouped launch's grid is
// (x-y blocks of all members, 1, levels): the members share nz, and blockIdx.x indexes a map that gives each x-y
// block its member and its block coordinates (one 8-byte load per thread, the same for the whole block).
__constant__ MemberC c_members[kMaxMembers];
#define OB_GROUP_RESOLVE                                                               \
  const uint2 gm__ = __ldg(map + blockIdx.x);                                         \
  const int mem = int(gm__.x), gbx = int(gm__.y & 0xffffu), gby = int(gm__.y >> 16u), \
            gbz = int(blockIdx.z);

// block coordinates: blockIdx for a launch over one model, or the (member, block) a grouped launch resolved
#define OB_BLOCKS_DIRECT const int BX = blockIdx.x, BY = blockIdx.y, BZ = blockIdx.z;
#define OB_TEXEL_LOOP_BEGIN(XMAX, YMAX, ZMAX)             \
  const int ci = BX * blockDim.x + threadIdx.x;           \
  const int cj = BY * blockDim.y + threadIdx.y;           \
  const int ck = BZ;                                      \
  if (ci > (XMAX) || cj > (YMAX) || ck > (ZMAX)) return;

// ---------------------------------------------------------------------------------------------------------------
// target state (model.js:121-134)
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ float tprof(float z, float H) { return 1.f - sstep(0.7f * H, 1.15f * H, z); }
__device__ __forceinline__ float4 l2d(const float4* __restrict__ m, const Grid& g, int i, int j) {
  return __ldg(m + clampi(j, 0, g.ny - 1) * g.nx + clampi(i, 0, g.nx - 1));
}
__device__ __forceinline__ float tgtTh(const float* B, const Grid& g, float dz, float4 A, int k) {
  float z = (float(k) + 0.5f) * dz;
  return bsA(B, g.nz, k).x + A.x / bsB(B, g.nz, k).x * tprof(z, A.y);
}
__device__ __forceinline__ float tgtQv(const float* B, const Grid& g, float dz, float4 A, int k) {
  float z = (float(k) + 0.5f) * dz;
  return bsA(B, g.nz, k).y * (1.f - A.z * tprof(z, A.w));
}
// with no boundary air masses (LSF over zero boundaries gives lsfA = (0, 100, 0, 100), lsfB = (0, 0, 100, 0) and
// phi_t = +-0), every target expression below reduces exactly to the base state: x + 0 * t == x, qv0 * (1 - 0 * t)
// == qv0, and +-0 differences of phi_t change nothing. The BND = false instantiations skip those loads.
template <bool BND>
__device__ __forceinline__ float tgtUb(const Fields& F, const Grid& g, float dz, int i, int j, int k);
template <bool BND>
__device__ __forceinline__ float tgtVb(const Fields& F, const Grid& g, float dz, int i, int j, int k);
__device__ __forceinline__ float tgtU(const Fields& F, const Grid& g, float dz, int i, int j, int k) {
  float z = (float(k) + 0.5f) * dz;
  float4 a = l2d(F.lsfB, g, i - 1, j), b = l2d(F.lsfB, g, i, j);
  return bsB(F.B, g.nz, k).z + 0.5f * (a.x * tprof(z, a.z) + b.x * tprof(z, b.z));
}
__device__ __forceinline__ float tgtV(const Fields& F, const Grid& g, float dz, int i, int j, int k) {
  float z = (float(k) + 0.5f) * dz;
  float4 a = l2d(F.lsfB, g, i, j - 1), b = l2d(F.lsfB, g, i, j);
  return bsB(F.B, g.nz, k).w + 0.5f * (a.y * tprof(z, a.z) + b.y * tprof(z, b.z));
}

template <>
__device__ __forceinline__ float tgtUb<true>(const Fields& F, const Grid& g, float dz, int i, int j, int k) { return tgtU(F, g, dz, i, j, k); }
template <>
__device__ __forceinline__ float tgtUb<false>(const Fields& F, const Grid& g, float, int, int, int k) { return bsB(F.B, g.nz, k).z; }
template <>
__device__ __forceinline__ float tgtVb<true>(const Fields& F, const Grid& g, float dz, int i, int j, int k) { return tgtV(F, g, dz, i, j, k); }
template <>
__device__ __forceinline__ float tgtVb<false>(const Fields& F, const Grid& g, float, int, int, int k) { return bsB(F.B, g.nz, k).w; }

// ---------------------------------------------------------------------------------------------------------------
// WGSL_M_LSF (model.js:142-244): per column, target anomalies of the boundaries' air masses + hydrostatic phi_t
// ---------------------------------------------------------------------------------------------------------------
__device__ void bpt(const float* bd, int i, float t, float& x, float& y) {
  const float* q = bd + 20 + 4 * i;
  x = q[0] + q[2] * t;
  y = q[1] + q[3] * t;
}
__device__ __forceinline__ void lsf_body(const Grid& g, const Uni& U, const Fields& F, int par, const int BX, const int BY, const int BZ) {
  const int i = BX * blockDim.x + threadIdx.x, j = BY * blockDim.y + threadIdx.y;
  if (i >= g.nx || j >= g.ny) return;
  const float dx = U.dims.w, t = float(__ldg(F.clock));
  const float x = (float(i) + 0.5f) * dx, y = (float(j) + 0.5f) * dx;
  float sT = 0, sH = 0, sQ = 0, sHq = 0, sU = 0, sV = 0, sHw = 0, sw = 0, nud = 0;
  const int nb = int(U.cor.z);
  for (int b = 0; b < nb; b++) {
    const float* bd = F.bnd + b * 148;
    // signed distance to the moving polyline (model.js:157-179)
    const int np = int(bd[0]);
    float best = 1e30f, sg = 1.f, over = 0.f, along = 0.f, s0 = 0.f;
    for (int s = 0; s < np - 1; s++) {
      float ax, ay, ex, ey;
      bpt(bd, s, t, ax, ay);
      bpt(bd, s + 1, t, ex, ey);
      float abx = ex - ax, aby = ey - ay;
      float la = fmaxf(sqrtf(abx * abx + aby * aby), 1.f);
      float t0 = ((x - ax) * abx + (y - ay) * aby) / (la * la);
      float tt = t0;
      if (s > 0) tt = fmaxf(tt, 0.f);
      if (s < np - 2) tt = fminf(tt, 1.f);
      float ddx = x - (ax + tt * abx), ddy = y - (ay + tt * aby);
      float d = sqrtf(ddx * ddx + ddy * ddy);
      if (d < best) {
        best = d;
        sg = (abx * (y - ay) - aby * (x - ax) > 0.f) ? 1.f : -1.f;
        over = (s == 0 ? fmaxf(-t0, 0.f) * la : 0.f) + (s == np - 2 ? fmaxf(t0 - 1.f, 0.f) * la : 0.f);
        along = s0 + tt * la;
      }
      s0 += la;
    }
    const float d = best * sg * bd[15];
    const float w = sstep(-bd[3], bd[3], d) * (1.f - sstep(0.f, 60000.f, over));
    if (w <= 0.f) continue;
    const float vr = bd[16];
    const float fade = 1.f - sstep(30000.f, 90000.f, d);
    // along-front variation (model.js:183-187) and hot spots (model.js:191-206)
    float avv = 0.f;
    if (bd[16] > 0.f) avv = clampf(fbm2(along / bd[18], bd[17] + t / 5400.f, 2) * 1.6f, -1.f, 1.f);
    const float av = vr * avv * fade;
    float lift = 1.f;
    if (vr > 0.f) {
      const float L = bd[18];
      const int sd = int(bd[17] * 1000.f);
      const float ph = t / 4800.f;
      const int e = int(floorf(ph));
      const float fe = sstep(0.f, 1.f, ph - floorf(ph));
      const int k0 = int(floorf(along / L));
      float acc = 0.f;
      for (int k = k0 - 1; k <= k0 + 1; k++)
        for (int q = 0; q < 2; q++) {
          uint32_t h = hash3i(k, e + q, sd);
          float r1 = float(h & 0xffffu) / 65535.f, r2 = float((h >> 16u) & 0xffffu) / 65535.f;
          float z = (along - (float(k) + 0.5f + 0.7f * (r1 - 0.5f)) * L) / (0.17f * L);
          acc += (q == 1 ? fe : 1.f - fe) * (0.35f + 0.65f * r2) * expf(-z * z);
        }
      lift = mixf(1.f, mixf(1.f - 0.85f * vr, 1.f + 1.3f * vr, clampf(acc, 0.f, 1.f)), fade);
    }
    const float Hmin = bd[7] * clampf(lift, 0.15f, 3.f);
    const float H = fminf(fmaxf(bd[6] * fmaxf(d + bd[3], 0.f) * (1.f + 0.4f * av), Hmin), bd[5]);
    sT += w * bd[4] * expf(0.5f * av);
    sQ += w * bd[8];
    sU += w * bd[10] * lift;
    sV += w * bd[11] * lift;
    sH += w * H;
    sHq += w * H * bd[9];
    sHw += w * H * bd[12];
    sw += w;
    nud = fmaxf(nud, bd[13] * sstep(bd[14], bd[14] + 40000.f, d) * (1.f - sstep(0.f, 60000.f, over)));
  }
  const float iw = 1.f / fmaxf(sw, 1e-6f);
  const float4 A = make_float4(clampf(sT, -20.f, 10.f), fmaxf(sH * iw, 100.f), clampf(sQ, 0.f, 0.92f), fmaxf(sHq * iw, 100.f));
  F.lsfA[j * g.nx + i] = A;
  F.lsfB[j * g.nx + i] = make_float4(sU, sV, fmaxf(sHw * iw, 100.f), nud);
  const float dz = U.dzv.x;
  float ph = 0.f, bprev = 0.f;
  for (int k = g.nz - 1; k >= 0; k--) {
    const float z = (float(k) + 0.5f) * dz;
    const float4 a = bsA(F.B, g.nz, k), bb = bsB(F.B, g.nz, k);
    const float dth = A.x / bb.x * tprof(z, A.y);
    const float dqv = -a.y * A.z * tprof(z, A.w);
    const float bt = 9.81f * (dth / a.x + 0.608f * dqv);
    if (k == g.nz - 1) ph = -bt * 0.5f * dz;
    else ph -= 0.5f * (bt + bprev) * dz;
    bprev = bt;
    F.phT[g.at(i, j, k)] = ph;
  }
}
__global__ void k_lsf(Grid g, Uni U, Fields F) { lsf_body(g, U, F, 0, blockIdx.x, blockIdx.y, blockIdx.z); }
__global__ void k_lsf_grp(const uint2* __restrict__ map, int par) {
  OB_GROUP_RESOLVE
  {
    const double t = *c_members[mem].F.clock, t0 = *c_members[mem].lsfT;
    if (!(t - t0 >= 60.0 || t == 0.0)) return;
  }
  lsf_body(c_members[mem].g, c_members[mem].U, c_members[mem].F, par, gbx, gby, gbz);
}

// ---------------------------------------------------------------------------------------------------------------
// WGSL_M_CI (model.js:249-281): strongest active updraft-nudging event per column
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void ci_body(const Grid& g, const Uni& U, const Fields& F, int par, const int BX, const int BY, const int BZ) {
  const int i = BX * blockDim.x + threadIdx.x, j = BY * blockDim.y + threadIdx.y;
  if (i >= g.nx || j >= g.ny) return;
  const float dx = U.dims.w, t = float(__ldg(F.clock));
  const float x = (float(i) + 0.5f) * dx, y = (float(j) + 0.5f) * dx;
  float4 best = make_float4(0.f, 0.f, 1500.f, 1500.f);
  const int ne = int(U.ci.x);
  for (int e = 0; e < ne; e++) {
    const float* E = F.ci + e * 12;
    if (t < E[6] || t > E[7]) continue;
    const float dxv = x - (E[0] + E[8] * (t - E[6])), dyv = y - (E[1] + E[9] * (t - E[6]));
    const float ang = atan2f(dyv, dxv);
    const float wob = 1.f + 0.25f * gnoise2(cosf(ang) * 1.6f + E[10], sinf(ang) * 1.6f + 3.7f * E[10]);
    const float gg = sstep(E[6], E[6] + fmaxf(E[11], 60.f), t);
    const float r = sqrtf(dxv * dxv + dyv * dyv) / (E[3] * wob * (0.35f + 0.65f * gg));
    if (r >= 1.f) continue;
    const float Lx = float(g.nx) * dx, Ly = float(g.ny) * dx;
    const float edge = fminf(fminf(x, Lx - x), fminf(y, Ly - y));
    const float h = sstep(E[6], E[6] + 60.f, t) * (1.f - sstep(E[7] - 180.f, E[7], t)) * sstep(U.sponge.x, U.sponge.x + 10000.f, edge);
    const float wt = E[5] * (0.4f + 0.6f * gg) * cosf(1.5707963f * r);
    if (h * wt > best.x * best.y) best = make_float4(h, wt, E[2], E[4]);
  }
  F.ciMap[j * g.nx + i] = best;
}
__global__ void k_ci(Grid g, Uni U, Fields F) { ci_body(g, U, F, 0, blockIdx.x, blockIdx.y, blockIdx.z); }
__global__ void k_ci_grp(const uint2* __restrict__ map, int par) {
  OB_GROUP_RESOLVE
  if (gbx == 0 && gby == 0 && gbz == 0 && threadIdx.x == 0 && threadIdx.y == 0) {  // after the LSF pass of this step
    const double t = *c_members[mem].F.clock;
    double* t0 = c_members[mem].lsfT;
    if (t - *t0 >= 60.0 || t == 0.0) *t0 = t;
    if (c_members[mem].micro == kMicroSurrogate) {  // this step's surrogate queue and fallback count start empty
      c_members[mem].F.mlp_count[0] = 0u;
      c_members[mem].F.mlp_count[1] = 0u;
    }
  }
  ci_body(c_members[mem].g, c_members[mem].U, c_members[mem].F, par, gbx, gby, gbz);
}

// ---------------------------------------------------------------------------------------------------------------
// WGSL_M_INIT (model.js:284-339), outbreak mode (no vortex)
// ---------------------------------------------------------------------------------------------------------------
__global__ void k_init(Grid g, Uni U, Fields F) {
  OB_BLOCKS_DIRECT
  OB_TEXEL_LOOP_BEGIN(g.nx, g.ny, g.nz)
  const int k = min(ck, g.nz - 1);
  const float dz = U.dzv.x;
  const float4 A = l2d(F.lsfA, g, ci, cj);
  const float z = (float(k) + 0.5f) * dz;
  const float dx = U.dims.w;
  const bool vortex = U.vtx2.z > 0.5f && F.vx;
  float nz0 = sstep(800.f, 1500.f, z);
  // hurricane mode: the noise reaches up through the moist core (model.js:306-309)
  if (U.vtx2.z > 0.5f) {
    const float px = (float(ci) + 0.5f) * dx - U.vtx.x, py = (float(cj) + 0.5f) * dx - U.vtx.y;
    nz0 = sqrtf(px * px + py * py) < U.vtx2.x ? sstep(6000.f, 8000.f, z) : 1.f;
  }
  const float noise = U.misc.z * (rnd3(ci + 17, cj + 3, ck + 5) - 0.5f) * 2.f * (1.f - nz0);
  float th = tgtTh(F.B, g, dz, A, k) + noise;
  float u = (cj < g.ny && ck < g.nz) ? tgtU(F, g, dz, ci, cj, k) : 0.f;
  float v = (ci < g.nx && ck < g.nz) ? tgtV(F, g, dz, ci, cj, k) : 0.f;
  // the vortex table at radius r (model.js:292-297): (tangential wind, theta')
  auto vxAt = [&](float r) {
    const int nr = int(U.vtx.w);
    const float fr = r / U.vtx.z;
    const int i0 = int(floorf(fr));
    if (i0 >= nr - 1) return make_float2(0.f, 0.f);
    const int q = clampi(k, 0, g.nz - 1) * nr + i0;
    const float4 a = __ldg(F.vx + q), b = __ldg(F.vx + q + 1);
    const float t = fr - float(i0);
    return make_float2(a.x * (1.f - t) + b.x * t, a.y * (1.f - t) + b.y * t);
  };
  if (vortex) {  // a warm-core vortex in gradient-wind and hydrostatic balance (model.js:314-325)
    const float pux = float(ci) * dx - U.vtx.x, puy = (float(cj) + 0.5f) * dx - U.vtx.y;
    const float ru = fmaxf(sqrtf(pux * pux + puy * puy), 1.f);
    const float pvx = (float(ci) + 0.5f) * dx - U.vtx.x, pvy = float(cj) * dx - U.vtx.y;
    const float rv = fmaxf(sqrtf(pvx * pvx + pvy * pvy), 1.f);
    const float pcx = (float(ci) + 0.5f) * dx - U.vtx.x, pcy = (float(cj) + 0.5f) * dx - U.vtx.y;
    const float rc = sqrtf(pcx * pcx + pcy * pcy);
    u -= vxAt(ru).x * puy / ru;
    v += vxAt(rv).x * pvx / rv;
    th += vxAt(rc).y;
  }
  const float T = th * bsB(F.B, g.nz, k).x;
  float qv = fminf(tgtQv(F.B, g, dz, A, k), 0.95f * qvsat(T, bsB(F.B, g.nz, k).y, fIce(T)));
  if (vortex) {  // a nearly saturated core at the same density (model.js:328-335)
    const float pcx = (float(ci) + 0.5f) * dx - U.vtx.x, pcy = (float(cj) + 0.5f) * dx - U.vtx.y;
    const float f = (1.f - sstep(0.6f, 1.f, sqrtf(pcx * pcx + pcy * pcy) / U.vtx2.x)) * sstep(500.f, 1500.f, z) *
                    (1.f - sstep(7000.f, 10000.f, z));
    const float q2 = fmaxf(qv, f * U.vtx2.y * qvsat(T, bsB(F.B, g.nz, k).y, fIce(T)));
    const float dqv = q2 - qv;
    qv = q2;
    th -= 0.608f * dqv * bsA(F.B, g.nz, k).x;
  }
  const int o = g.at(ci, cj, ck);
  for (int p = 0; p < 2; p++) {  // both ping-pong slots (reset copies V0 to V1, model.js:1437)
    F.V[p][0][o] = u;
    F.V[p][1][o] = v;
    F.V[p][2][o] = 0.f;
    F.V[p][3][o] = th;
  }
  if (ci < g.nx && cj < g.ny && ck < g.nz) {
    F.Q[0][0][o] = qv;
#pragma unroll
    for (int c = 1; c < 8; c++) F.Q[0][c][o] = 0.f;
  }
}

// ---------------------------------------------------------------------------------------------------------------
// WGSL_M_NUT (model.js:342-389): Smagorinsky-Lilly viscosities with the Richardson correction
// ---------------------------------------------------------------------------------------------------------------
template <bool HUR = false>
__device__ __forceinline__ void nut_body(const Grid& g, const Uni& U, const Fields& F, int par, const int BX, const int BY, const int BZ) {
  OB_TEXEL_LOOP_BEGIN(g.nx - 1, g.ny - 1, g.nz - 1)
  // a cell's +1 neighbours on the staggered box always exist; the -1 ones clamp to the edge
  const unsigned o = 4u * unsigned(g.at(ci, cj, ck)), sy = 4u * unsigned(g.px), sz = 4u * unsigned(g.plane);
  const unsigned xm = ci > 0 ? o - 4u : o, ym = cj > 0 ? o - sy : o, zm = ck > 0 ? o - sz : o;
  const unsigned xp = o + 4u, yp = o + sy, zp = o + sz;
  const float* __restrict__ u = F.V[par][0];
  const float* __restrict__ v = F.V[par][1];
  const float* __restrict__ w = F.V[par][2];
  const float* __restrict__ th = F.V[par][3];
  const float u0m = bsB(F.B, g.nz, ck - 1).z, u00 = bsB(F.B, g.nz, ck).z, u0p = bsB(F.B, g.nz, ck + 1).z;
  const float v0m = bsB(F.B, g.nz, ck - 1).w, v00 = bsB(F.B, g.nz, ck).w, v0p = bsB(F.B, g.nz, ck + 1).w;
  auto uc = [&](unsigned at, float u0) { return 0.5f * (ldo(u, at) + ldo(u + 1, at)) - u0; };
  auto vc = [&](unsigned at, float v0) { return 0.5f * (ldo(v, at) + ldo(v, at + sy)) - v0; };
  auto wc = [&](unsigned at) { return 0.5f * (ldo(w, at) + ldo(w, at + sz)); };
  const float dx = U.dims.w, dz = U.dzv.x;
  // differences times the correctly rounded reciprocals 1/dx, 1/dz (and their exact halves) instead of divisions
  const float idx = U.dzv.y, idz = U.dzv.z, ih2x = 0.5f * idx, ih2z = 0.5f * idz;
  const float dudx = (ldo(u + 1, o) - ldo(u, o)) * idx;
  const float dvdy = (ldo(v, yp) - ldo(v, o)) * idx;
  const float dwdz = (ldo(w, zp) - ldo(w, o)) * idz;
  const float dudy = (uc(yp, u00) - uc(ym, u00)) * ih2x, dudz = (uc(zp, u0p) - uc(zm, u0m)) * ih2z;
  const float dvdx = (vc(xp, v00) - vc(xm, v00)) * ih2x, dvdz = (vc(zp, v0p) - vc(zm, v0m)) * ih2z;
  const float dwdx = (wc(xp) - wc(xm)) * ih2x, dwdy = (wc(yp) - wc(ym)) * ih2x;
  const float s12 = 0.5f * (dudy + dvdx), s13 = 0.5f * (dudz + dwdx), s23 = 0.5f * (dvdz + dwdy);
  const float S2 = 2.f * (dudx * dudx + dvdy * dvdy + dwdz * dwdz) + 4.f * (s12 * s12 + s13 * s13 + s23 * s23);
  const int kz0 = max(ck - 1, 0), kz1 = min(ck + 1, g.nz - 1);
  float N2 = 9.81f / bsA(F.B, g.nz, ck).x * (ldo(th, o + unsigned(kz1 - ck) * sz) - ldo(th, o + unsigned(kz0 - ck) * sz)) / (float(kz1 - kz0) * dz);
  if (U.cor.w > 0.5f && ldo(F.Q[0][1], o) + ldo(F.Q[0][2], o) > 1e-5f) N2 = fminf(N2, 0.f);
  const float dtc = fmaxf(U.step.x, 0.1f);
  // Ri clearly past the critical value: the Richardson factor and both viscosities are exactly zero, as the divisions and
  // roots below would find (a stable, weakly sheared cell; most are). An infinite S2 or a NaN takes the full form. The pass is
  // bound by instruction issue (88 % of slots): with this and the byte offsets 190 -> 150 us at 640 x 640 x 40.
  float nuh = 0.f, nuv = 0.f;
  const float S2c = fmaxf(S2, 1e-10f);
  if (!(N2 > 0.331f * S2c)) {
    const float Ri = N2 / S2c;
    const float fst = sqrtf(fmaxf(0.f, 1.f - Ri / 0.33f));
    const float sS = sqrtf(fmaxf(S2, 0.f));
    const float lh = U.turb.x * dx, lv = 0.18f * dz;
    nuh = fminf(lh * lh * sS * fst, 0.08f * dx * dx / dtc);
    nuv = fminf(lv * lv * sS * fst, 0.15f * dz * dz / dtc);
  }
  sto(F.aux[0], o, nuh);
  if (HUR) {  // hurricane mode: a K-profile boundary layer (model.js:377-386)
    const float zc = (float(ck) + 0.5f) * dz, h = U.hur2.z;
    if (zc < h) {
      const int o0 = g.at(ci, cj, 0);
      const float ua = 0.5f * (__ldg(F.V[par][0] + o0) + __ldg(F.V[par][0] + o0 + 1));
      const float va = 0.5f * (__ldg(F.V[par][1] + o0) + __ldg(F.V[par][1] + o0 + g.px));
      const float u1 = sqrtf(ua * ua + va * va);
      const float ust = sqrtf(cdSfc(U, u1, __ldg(F.sfc + cj * g.nx + ci).x)) * fmaxf(u1, U.hur3.y);
      const float q = 1.f - zc / h;
      nuv = fmaxf(nuv, fminf(0.4f * ust * zc * q * q, 0.15f * dz * dz / dtc));
    }
  }
  sto(F.aux[1], o, nuv);
}
__global__ void __launch_bounds__(128, 16) k_nut(Grid g, Uni U, Fields F) { nut_body(g, U, F, 0, blockIdx.x, blockIdx.y, blockIdx.z); }
__global__ void k_nut_hur(Grid g, Uni U, Fields F) { nut_body<true>(g, U, F, 0, blockIdx.x, blockIdx.y, blockIdx.z); }
__global__ void __launch_bounds__(128, 12) k_nut_grp(const uint2* __restrict__ map, int par) {
  OB_GROUP_RESOLVE
  nut_body(c_members[mem].g, c_members[mem].U, c_members[mem].F, par, gbx, gby, gbz);
}

// ---------------------------------------------------------------------------------------------------------------
// advection of the winds and theta (model.js:391-481)
// ---------------------------------------------------------------------------------------------------------------
struct Loc {
  float vu[3], vv[3], vw[3], vc[3];
};
__device__ __forceinline__ Loc localVel(const Fields& F, const Grid& g, int par, int i, int j, int k) {
  // clamp-to-edge neighbour offsets of the staggered box (bytes), once per texel
  const unsigned o = 4u * unsigned(g.at(i, j, k));
  const unsigned xm = i > 0 ? -4u : 0u, xp = i < g.nx ? 4u : 0u;
  const unsigned px4 = 4u * unsigned(g.px), pl4 = 4u * unsigned(g.plane);
  const unsigned ym = j > 0 ? 0u - px4 : 0u, yp = j < g.ny ? px4 : 0u;
  const unsigned zm = k > 0 ? 0u - pl4 : 0u, zp = k < g.nz ? pl4 : 0u;
  const float* __restrict__ u = F.V[par][0];
  const float* __restrict__ v = F.V[par][1];
  const float* __restrict__ w = F.V[par][2];
  const unsigned oxm = o + xm, oxp = o + xp, oym = o + ym, oyp = o + yp, ozm = o + zm, ozp = o + zp;
  Loc L;
  const float pu = ldo(u, o), pv = ldo(v, o), pw = ldo(w, o);
  const float xpu = ldo(u, oxp), ypv = ldo(v, oyp), zpw = ldo(w, ozp);
  L.vu[0] = pu;
  L.vu[1] = 0.25f * (ldo(v, oxm) + pv + ldo(v, oxm + yp) + ypv);
  L.vu[2] = 0.25f * (ldo(w, oxm) + pw + ldo(w, oxm + zp) + zpw);
  L.vv[0] = 0.25f * (ldo(u, oym) + pu + ldo(u, oym + xp) + xpu);
  L.vv[1] = pv;
  L.vv[2] = 0.25f * (ldo(w, oym) + pw + ldo(w, oym + zp) + zpw);
  L.vw[0] = 0.25f * (ldo(u, ozm) + pu + ldo(u, ozm + xp) + xpu);
  L.vw[1] = 0.25f * (ldo(v, ozm) + pv + ldo(v, ozm + yp) + ypv);
  L.vw[2] = pw;
  L.vc[0] = 0.5f * (pu + xpu);
  L.vc[1] = 0.5f * (pv + ypv);
  L.vc[2] = 0.5f * (pw + zpw);
  return L;
}
// departure (s = 1) or forward (s = -1) point, first-order trace clamped to the box (model.js:428-432)
__device__ __forceinline__ void traceV(const Grid& g, const float k[3], float px, float py, float pz, const float v[3], float s,
                                       float& x, float& y, float& z) {
  x = clampf(px - s * k[0] * v[0], 0.f, float(g.nx));
  y = clampf(py - s * k[1] * v[1], 0.f, float(g.ny));
  z = clampf(pz - s * k[2] * v[2], 0.f, float(g.nz));
}
// channel sample at a point in grid units (texel offsets of u, v, w, theta: model.js:419-422)
__device__ __forceinline__ float sampleVch(const float* f, const Grid& g, int ch, float x, float y, float z) {
  const float ox = ch == 0 ? 0.f : 0.5f, oy = ch == 1 ? 0.f : 0.5f, oz = ch == 2 ? 0.f : 0.5f;
  return trilerpB(f, g, g.nx + 1, g.ny + 1, g.nz + 1, x - ox, y - oy, z - oz);
}

// the same from the scratch that ADVV1 has just written
__device__ __forceinline__ float sampleVt(const Fields& F, const Grid& g, int ch, float x, float y, float z) {
  const float ox = ch == 0 ? 0.f : 0.5f, oy = ch == 1 ? 0.f : 0.5f, oz = ch == 2 ? 0.f : 0.5f;
  return gather8_late(F.Vt[ch], corners(g, g.nx + 1, g.ny + 1, g.nz + 1, x - ox, y - oy, z - oz));
}

// the departure-point sample of a channel, with the min / max of its 8 texels (ADVV2's limiter window: the
// reference's limiter traces the same point, model.js:455-479)
__device__ __forceinline__ void sampleVch_mm(const Fields& F, const Grid& g, int par, int ch, unsigned o, float x, float y, float z) {
  const float ox = ch == 0 ? 0.f : 0.5f, oy = ch == 1 ? 0.f : 0.5f, oz = ch == 2 ? 0.f : 0.5f;
  float lo, hi;
  const float t = trilerpB_mm(F.V[par][ch], g, g.nx + 1, g.ny + 1, g.nz + 1, x - ox, y - oy, z - oz, lo, hi);
  sto(F.Vt[ch], o, t);
  sto(F.Vlo[ch], o, lo);
  sto(F.Vhi[ch], o, hi);
}
__device__ __forceinline__ void advv1_body(const Grid& g, const Uni& U, const Fields& F, int par, const int BX, const int BY, const int BZ) {
  OB_TEXEL_LOOP_BEGIN(g.nx, g.ny, g.nz)
  const Loc L = localVel(F, g, par, ci, cj, ck);
  const float kk[3] = {U.der.x, U.der.x, U.der.y};  // dt/dx, dt/dx, dt/dz
  const float fi = float(ci), fj = float(cj), fk = float(ck);
  const unsigned o = 4u * unsigned(g.at(ci, cj, ck));
  float x, y, z;
  traceV(g, kk, fi, fj + 0.5f, fk + 0.5f, L.vu, 1.f, x, y, z);
  sampleVch_mm(F, g, par, 0, o, x, y, z);
  traceV(g, kk, fi + 0.5f, fj, fk + 0.5f, L.vv, 1.f, x, y, z);
  sampleVch_mm(F, g, par, 1, o, x, y, z);
  traceV(g, kk, fi + 0.5f, fj + 0.5f, fk, L.vw, 1.f, x, y, z);
  sampleVch_mm(F, g, par, 2, o, x, y, z);
  traceV(g, kk, fi + 0.5f, fj + 0.5f, fk + 0.5f, L.vc, 1.f, x, y, z);
  sampleVch_mm(F, g, par, 3, o, x, y, z);
}
__global__ void __launch_bounds__(128, 16) k_advv1(Grid g, Uni U, Fields F) { advv1_body(g, U, F, 0, blockIdx.x, blockIdx.y, blockIdx.z); }
__global__ void k_advv1_grp(const uint2* __restrict__ map, int par) {
  OB_GROUP_RESOLVE
  advv1_body(c_members[mem].g, c_members[mem].U, c_members[mem].F, par, gbx, gby, gbz);
}

__device__ __forceinline__ void advv2_body(const Grid& g, const Uni& U, const Fields& F, int par, const int BX, const int BY, const int BZ) {
  OB_TEXEL_LOOP_BEGIN(g.nx, g.ny, g.nz)
  const Loc L = localVel(F, g, par, ci, cj, ck);
  const float kk[3] = {U.der.x, U.der.x, U.der.y};  // dt/dx, dt/dx, dt/dz
  const float fi = float(ci), fj = float(cj), fk = float(ck);
  const float P[4][3] = {{fi, fj + 0.5f, fk + 0.5f}, {fi + 0.5f, fj, fk + 0.5f}, {fi + 0.5f, fj + 0.5f, fk}, {fi + 0.5f, fj + 0.5f, fk + 0.5f}};
  const float* vel[4] = {L.vu, L.vv, L.vw, L.vc};
  const float cx = L.vc[0] * kk[0], cy = L.vc[1] * kk[1], cz = L.vc[2] * kk[2];
  const float cour = sqrtf(cx * cx + cy * cy + cz * cz);
  const float sm = 0.5f * U.misc.y * clampf(cour / 0.35f, U.dzv.w, 1.f);
  const unsigned o = 4u * unsigned(g.at(ci, cj, ck));
#pragma unroll
  for (int c = 0; c < 4; c++) {
    float x, y, z;
    traceV(g, kk, P[c][0], P[c][1], P[c][2], vel[c], -1.f, x, y, z);
    const float b = sampleVt(F, g, c, x, y, z);
    const float hat = ldo_late(F.Vt[c], o), old = ldo(F.V[par][c], o);
    const float r = hat + sm * (old - b);
    sto(F.V[1 - par][c], o, clampf(r, ldo_late(F.Vlo[c], o), ldo_late(F.Vhi[c], o)));
  }
}
__global__ void __launch_bounds__(128, 12) k_advv2(Grid g, Uni U, Fields F) {
  tc::grid_wait();
  advv2_body(g, U, F, 0, blockIdx.x, blockIdx.y, blockIdx.z);
}
__global__ void __launch_bounds__(128, 10) k_advv2_grp(const uint2* __restrict__ map, int par) {
  OB_GROUP_RESOLVE
  advv2_body(c_members[mem].g, c_members[mem].U, c_members[mem].F, par, gbx, gby, gbz);
}

// ---------------------------------------------------------------------------------------------------------------
// scalar advection with fall speeds (model.js:482-576)
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void cellVel(const Fields& F, const Grid& g, int par, int i, int j, int k, float v[3]) {
  const unsigned o = 4u * unsigned(g.at(i, j, k));
  v[0] = 0.5f * (ldo(F.V[par][0], o) + ldo(F.V[par][0], o + 4u));
  v[1] = 0.5f * (ldo(F.V[par][1], o) + ldo(F.V[par][1], o + 4u * unsigned(g.px)));
  v[2] = 0.5f * (ldo(F.V[par][2], o) + ldo(F.V[par][2], o + 4u * unsigned(g.plane)));
}
__device__ __forceinline__ void traceQ(const Grid& g, const float k[3], const float p[3], const float v[3], float fall, float s,
                                       float& x, float& y, float& z) {
  x = clampf(p[0] - s * k[0] * v[0], 0.5f, float(g.nx) - 0.5f);
  y = clampf(p[1] - s * k[1] * v[1], 0.5f, float(g.ny) - 0.5f);
  z = clampf(p[2] - s * k[2] * (v[2] - fall), 0.5f, float(g.nz) - 0.5f);
}
// A trilinear tap on the cell-centred box: the corners of the 2 x 2 x 2 neighbourhood (clamp-to-edge) and the weights;
// the same footprint is the 8-texel min/max window of the MacCormack limiter (model.js:537-540).
using Tap = Corners;
__device__ __forceinline__ Tap tapQ(const Grid& g, float x, float y, float z) {
  // x, y, z come from traceQ, clamped to [0.5, n - 0.5]: the floor indices lie in [0, n - 1], so only the upper
  // corner needs its clamp-to-edge bound
  const float tx = x - 0.5f, ty = y - 0.5f, tz = z - 0.5f;
  const int i0 = __float2int_rd(tx), j0 = __float2int_rd(ty), k0 = __float2int_rd(tz);
  Tap t;
  t.ax = tx - float(i0);
  t.ay = ty - float(j0);
  t.az = tz - float(k0);
  const unsigned px4 = 4u * unsigned(g.px), pl4 = 4u * unsigned(g.plane);
  const unsigned dx4 = i0 < g.nx - 1 ? 4u : 0u, dy4 = j0 < g.ny - 1 ? px4 : 0u, dz4 = k0 < g.nz - 1 ? pl4 : 0u;
  t.a = 4u * unsigned(i0) + px4 * unsigned(j0) + pl4 * unsigned(k0);
  t.c = t.a + dy4;
  t.e = t.a + dz4;
  t.k = t.c + dz4;
  t.b = t.a + dx4;
  t.d = t.c + dx4;
  t.h = t.e + dx4;
  t.l = t.k + dx4;
  return t;
}
__device__ __forceinline__ float gatherQ(const float* __restrict__ f, const Tap& t) { return gather8(f, t); }
__device__ __forceinline__ float2 minmaxQ(const float* __restrict__ f, const Tap& t) {
  const float a = ldo(f, t.a), b = ldo(f, t.b), c = ldo(f, t.c), d = ldo(f, t.d);
  const float e = ldo(f, t.e), h = ldo(f, t.h), k = ldo(f, t.k), l = ldo(f, t.l);
  return make_float2(min8(a, b, c, d, e, h, k, l), max8(a, b, c, d, e, h, k, l));
}

// Skip of the hydrometeor channels (qc, qi, qr, qs, qg, Nr) and of the spare fourth Q2 channel (which no scheme sets and
// physics only carries) where they are absent. A block (one brick of 32 x 4 x 1 cells) reads a channel only inside the
// footprints of its departure points; if no brick touching that region holds it (the flags below keep one bit per
// channel), the semi-Lagrangian sample, the MacCormack correction, the limiter and the clip all give exactly +0, so the
// block writes zeros (once) instead of gathering. Falling hydrometeors shift a departure point vertically by at most
// dt/dz * fallmax, which widens the region in z. One bit per channel and not one per brick, because most bricks of a
// storm hold some species only (an anvil is ice and snow, a warm shower cloud and rain, the Lin scheme never sets Nr and
// the spare): 640 x 640 x 40 with a storm every 60 km, ADVQ1 396 -> 335 us, ADVQ2 842 -> 631 us.
constexpr unsigned kHydro = 0xfeu;   // bits of the hydrometeor and spare channels, 1..7
// the bits that any thread of a 128-thread block sets, in every thread
__device__ __forceinline__ unsigned block_or(unsigned v) {
  __shared__ unsigned w[4];
  const int t = threadIdx.x + blockDim.x * threadIdx.y;
  v = __reduce_or_sync(0xffffffffu, v);
  if ((t & 31) == 0) w[t >> 5] = v;
  __syncthreads();
  return w[0] | w[1] | w[2] | w[3];
}
struct Region {
  int x0, x1, y0, y1, z0, z1;
};
// the channels (bits 1..7) that the bricks of a box of cells hold, in every thread of the block; the caller has set held
// to 0 and synchronised since
__device__ __forceinline__ unsigned box_channels(const Grid& g, const Fields& F, Region r, const unsigned int* flagsA,
                                                 const unsigned int* flagsB, unsigned& held) {
  const int bx0 = clampi(r.x0, 0, g.nx - 1) / 32, bx1 = clampi(r.x1, 0, g.nx - 1) / 32;
  const int by0 = clampi(r.y0, 0, g.ny - 1) / 4, by1 = clampi(r.y1, 0, g.ny - 1) / 4;
  const int bz0 = clampi(r.z0, 0, g.nz - 1), bz1 = clampi(r.z1, 0, g.nz - 1);
  const int nxb = bx1 - bx0 + 1, nyb = by1 - by0 + 1, nzb = bz1 - bz0 + 1;
  const int count = nxb * nyb * nzb;
  const int tid = threadIdx.x + blockDim.x * threadIdx.y;
  unsigned any = 0;
  for (int t = tid; t < count; t += blockDim.x * blockDim.y) {
    const int bx = bx0 + t % nxb, by = by0 + (t / nxb) % nyb, bz = bz0 + t / (nxb * nyb);
    const int b = bx + F.nbx * (by + F.nby * bz);
    any |= __ldg(flagsA + b);
    if (flagsB) any |= ld_late(flagsB + b);   // those of ADVQ1, just before
  }
  any = __reduce_or_sync(0xffffffffu, any);
  if ((threadIdx.x & 31) == 0 && any) atomicOr(&held, any);
  __syncthreads();
  return held;
}
// the channels that a brick touching the block's region holds, the region spanned by its threads' boxes r
__device__ __forceinline__ unsigned region_channels(const Grid& g, const Fields& F, Region r, const unsigned int* flagsA,
                                                    const unsigned int* flagsB) {
  __shared__ int red[6];
  __shared__ unsigned held;
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    red[0] = red[2] = red[4] = 1 << 30;
    red[1] = red[3] = red[5] = -(1 << 30);
    held = 0u;
  }
  __syncthreads();
  // warp-level min/max, then one shared atomic per warp
  const unsigned m = 0xffffffffu;
  const int a0 = __reduce_min_sync(m, r.x0), a1 = __reduce_max_sync(m, r.x1);
  const int b0 = __reduce_min_sync(m, r.y0), b1 = __reduce_max_sync(m, r.y1);
  const int c0 = __reduce_min_sync(m, r.z0), c1 = __reduce_max_sync(m, r.z1);
  if ((threadIdx.x & 31) == 0) {
    atomicMin(&red[0], a0); atomicMax(&red[1], a1);
    atomicMin(&red[2], b0); atomicMax(&red[3], b1);
    atomicMin(&red[4], c0); atomicMax(&red[5], c1);
  }
  __syncthreads();
  return box_channels(g, F, Region{red[0], red[1], red[2], red[3], red[4], red[5]}, flagsA, flagsB, held);
}

// ---- ADVQ1 (model.js:500-529): semi-Lagrangian step of the 8 scalars, channels grouped by the fall speed of
// their trace (qv, qc, qi, spare [and Nr for Lin] at the air's speed; qr, qs, qg, Nr (Thompson) each their own) ----
__device__ __forceinline__ void advq1_body(const Grid& g, const Uni& U, const Fields& F, int par, const int BX, const int BY, const int BZ) {
  const int ci = BX * blockDim.x + threadIdx.x, cj = BY * blockDim.y + threadIdx.y, ck = BZ;
  const bool in = ci < g.nx && cj < g.ny && ck < g.nz;
  const unsigned o = in ? 4u * unsigned(g.at(ci, cj, ck)) : 0u;
  const float kk[3] = {U.der.x, U.der.x, U.der.y};  // dt/dx, dt/dx, dt/dz
  float v[3] = {0.f, 0.f, 0.f};
  const float p[3] = {float(ci) + 0.5f, float(cj) + 0.5f, float(ck) + 0.5f};
  float x = 0.5f, y = 0.5f, z = 0.5f;
  Region r{ci, ci, cj, cj, ck, ck};
  if (in) {
    cellVel(F, g, par, ci, cj, ck, v);
    traceQ(g, kk, p, v, 0.f, 1.f, x, y, z);
    r.x0 = min(r.x0, int(floorf(x - 0.5f)));
    r.x1 = max(r.x1, int(floorf(x - 0.5f)) + 1);
    r.y0 = min(r.y0, int(floorf(y - 0.5f)));
    r.y1 = max(r.y1, int(floorf(y - 0.5f)) + 1);
    r.z0 = min(r.z0, int(floorf(z - 0.5f)));
    r.z1 = max(r.z1, int(floorf(fminf(z + kk[2] * F.fallmax, float(g.nz) - 0.5f) - 0.5f)) + 1);
  }
  const int brick = BX + F.nbx * (BY + F.nby * BZ);
  const unsigned zeros = F.zeroQt[brick];   // read by every thread before the barriers of the region, written after them
  const unsigned act = region_channels(g, F, r, F.actQ0, nullptr);
  auto has = [&](int c) { return ((act >> c) & 1u) != 0u; };
  if (in) {
    const Tap t0 = tapQ(g, x, y, z);
    sto(F.Qt[0], o, gatherQ(F.Q[0][0], t0));
    if (act) {
      const Fall fl{U.step.z, U.micro2.z > 0.5f};
      if (has(1)) sto(F.Qt[1], o, gatherQ(F.Q[0][1], t0));
      if (has(2)) sto(F.Qt[2], o, gatherQ(F.Q[0][2], t0));
      if (has(7)) sto(F.Qt[7], o, gatherQ(F.Q[0][7], t0));
      if (has(6) && !fl.thm) sto(F.Qt[6], o, gatherQ(F.Q[0][6], t0));
      const float rho = bsA(F.B, g.nz, ck).z;
      if (has(3) || (has(6) && fl.thm)) {
        const float2 fv = fl.vtRain(ldo(F.Q[0][3], o), ldo(F.Q[0][6], o), rho);
        if (has(3)) {
          traceQ(g, kk, p, v, fv.x, 1.f, x, y, z);
          sto(F.Qt[3], o, gatherQ(F.Q[0][3], tapQ(g, x, y, z)));
        }
        if (has(6) && fl.thm) {
          traceQ(g, kk, p, v, fv.y, 1.f, x, y, z);
          sto(F.Qt[6], o, gatherQ(F.Q[0][6], tapQ(g, x, y, z)));
        }
      }
      if (has(4)) {
        traceQ(g, kk, p, v, fl.vtS(ldo(F.Q[0][4], o), rho), 1.f, x, y, z);
        sto(F.Qt[4], o, gatherQ(F.Q[0][4], tapQ(g, x, y, z)));
      }
      if (has(5)) {
        traceQ(g, kk, p, v, fl.vtGrau(ldo(F.Q[0][5], o), rho), 1.f, x, y, z);
        sto(F.Qt[5], o, gatherQ(F.Q[0][5], tapQ(g, x, y, z)));
      }
    }
    const unsigned clear = kHydro & ~act & ~zeros;
    if (clear) {
#pragma unroll
      for (int c = 1; c < 8; c++)
        if ((clear >> c) & 1u) sto(F.Qt[c], o, 0.f);
    }
  }
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    F.actQt[brick] = act;
    F.zeroQt[brick] = kHydro & ~act;
  }
}
__global__ void __launch_bounds__(128, 16) k_advq1(Grid g, Uni U, Fields F) { advq1_body(g, U, F, 0, blockIdx.x, blockIdx.y, blockIdx.z); }
__global__ void __launch_bounds__(128, 12) k_advq1_grp(const uint2* __restrict__ map, int par) {
  OB_GROUP_RESOLVE
  advq1_body(c_members[mem].g, c_members[mem].U, c_members[mem].F, par, gbx, gby, gbz);
}

// ---- ADVQ2 (model.js:530-576): MacCormack correction, limiter on the departure cell's 8 texels, clip >= 0 ----
__device__ __forceinline__ float advq2_channel(const Fields& F, const Grid& g, const float kk[3], const float p[3], const float v[3],
                                               float fall, float sm, float qc_, int c, unsigned o) {
  float x, y, z;
  traceQ(g, kk, p, v, fall, -1.f, x, y, z);
  const float b = gather8_late(F.Qt[c], tapQ(g, x, y, z));
  const float r = ldo_late(F.Qt[c], o) + sm * (qc_ - b);
  traceQ(g, kk, p, v, fall, 1.f, x, y, z);
  const float2 m = minmaxQ(F.Q[0][c], tapQ(g, x, y, z));
  return fmaxf(clampf(r, m.x, m.y), 0.f);
}

__device__ __forceinline__ void advq2_body(const Grid& g, const Uni& U, const Fields& F, int par, const int BX, const int BY, const int BZ) {
  const int ci = BX * blockDim.x + threadIdx.x, cj = BY * blockDim.y + threadIdx.y, ck = BZ;
  const bool in = ci < g.nx && cj < g.ny && ck < g.nz;
  const unsigned o = in ? 4u * unsigned(g.at(ci, cj, ck)) : 0u;
  const float kk[3] = {U.der.x, U.der.x, U.der.y};  // dt/dx, dt/dx, dt/dz
  float v[3] = {0.f, 0.f, 0.f};
  const float p[3] = {float(ci) + 0.5f, float(cj) + 0.5f, float(ck) + 0.5f};
  float xb = 0.5f, yb = 0.5f, zb = 0.5f, xf = 0.5f, yf = 0.5f, zf = 0.5f;
  Region r{ci, ci, cj, cj, ck, ck};
  if (in) {
    cellVel(F, g, par, ci, cj, ck, v);
    traceQ(g, kk, p, v, 0.f, -1.f, xb, yb, zb);
    traceQ(g, kk, p, v, 0.f, 1.f, xf, yf, zf);
    r.x0 = min(r.x0, int(floorf(fminf(xb, xf) - 0.5f)));
    r.x1 = max(r.x1, int(floorf(fmaxf(xb, xf) - 0.5f)) + 1);
    r.y0 = min(r.y0, int(floorf(fminf(yb, yf) - 0.5f)));
    r.y1 = max(r.y1, int(floorf(fmaxf(yb, yf) - 0.5f)) + 1);
    const float dzf = kk[2] * F.fallmax;
    r.z0 = min(r.z0, int(floorf(fmaxf(fminf(zb, zf) - dzf, 0.5f) - 0.5f)));
    r.z1 = max(r.z1, int(floorf(fminf(fmaxf(zb, zf) + dzf, float(g.nz) - 0.5f) - 0.5f)) + 1);
  }
  const int brick = BX + F.nbx * (BY + F.nby * BZ);
  const unsigned zeros = F.zeroQ1[brick];   // read by every thread before the barriers of the region, written after them
  const unsigned act = region_channels(g, F, r, F.actQ0, F.actQt);
  auto has = [&](int c) { return ((act >> c) & 1u) != 0u; };
  if (in) {
    const float cx = v[0] * kk[0], cy = v[1] * kk[1], cz = v[2] * kk[2];
    const float cour = sqrtf(cx * cx + cy * cy + cz * cz);
    const float sm = 0.5f * U.misc.y * clampf(cour / 0.35f, U.dzv.w, 1.f);
    const Fall fl{U.step.z, U.micro2.z > 0.5f};
    {  // the air-speed group: qv always; qc, qi, the spare channel and, in the Lin scheme, Nr where held
      const Tap tb = tapQ(g, xb, yb, zb), tf = tapQ(g, xf, yf, zf);
      auto air = [&](int c) {
        const float b = gather8_late(F.Qt[c], tb);
        const float rr = ldo_late(F.Qt[c], o) + sm * (ldo(F.Q[0][c], o) - b);
        const float2 m = minmaxQ(F.Q[0][c], tf);
        sto(F.Q[1][c], o, fmaxf(clampf(rr, m.x, m.y), 0.f));
      };
      air(0);
      if (act) {
        if (has(1)) air(1);
        if (has(2)) air(2);
        if (has(7)) air(7);
        if (has(6) && !fl.thm) air(6);
      }
    }
    if (act & 0x78u) {
      const float rho = bsA(F.B, g.nz, ck).z;
      if (has(3) || (has(6) && fl.thm)) {
        const float q3 = ldo(F.Q[0][3], o), q6 = ldo(F.Q[0][6], o);
        const float2 fv = fl.vtRain(q3, q6, rho);
        if (has(3)) sto(F.Q[1][3], o, advq2_channel(F, g, kk, p, v, fv.x, sm, q3, 3, o));
        if (has(6) && fl.thm) sto(F.Q[1][6], o, advq2_channel(F, g, kk, p, v, fv.y, sm, q6, 6, o));
      }
      if (has(4)) {
        const float q4 = ldo(F.Q[0][4], o);
        sto(F.Q[1][4], o, advq2_channel(F, g, kk, p, v, fl.vtS(q4, rho), sm, q4, 4, o));
      }
      if (has(5)) {
        const float q5 = ldo(F.Q[0][5], o);
        sto(F.Q[1][5], o, advq2_channel(F, g, kk, p, v, fl.vtGrau(q5, rho), sm, q5, 5, o));
      }
    }
    const unsigned clear = kHydro & ~act & ~zeros;
    if (clear) {
#pragma unroll
      for (int c = 1; c < 8; c++)
        if ((clear >> c) & 1u) sto(F.Q[1][c], o, 0.f);
    }
  }
  if (threadIdx.x == 0 && threadIdx.y == 0) F.zeroQ1[brick] = kHydro & ~act;
}
__global__ void __launch_bounds__(128, 10) k_advq2(Grid g, Uni U, Fields F) {
  tc::grid_wait();
  advq2_body(g, U, F, 0, blockIdx.x, blockIdx.y, blockIdx.z);
}
__global__ void __launch_bounds__(128, 9) k_advq2_grp(const uint2* __restrict__ map, int par) {
  OB_GROUP_RESOLVE
  advq2_body(c_members[mem].g, c_members[mem].U, c_members[mem].F, par, gbx, gby, gbz);
}

// hydrometeor flags of Q slot 0 per brick, from scratch (after a reset or a host upload of Q); the scratch-known-zero
// flags are cleared because the host may have written anywhere
__global__ void __launch_bounds__(128) k_activity(Grid g, Fields F) {
  const int ci = blockIdx.x * blockDim.x + threadIdx.x, cj = blockIdx.y * blockDim.y + threadIdx.y, ck = blockIdx.z;
  unsigned act = 0u;
  if (ci < g.nx && cj < g.ny && ck < g.nz) {
    const int o = g.at(ci, cj, ck);
#pragma unroll
    for (int c = 1; c < 8; c++) act |= F.Q[0][c][o] != 0.f ? 1u << c : 0u;
  }
  act = block_or(act);
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    const int b = blockIdx.x + F.nbx * (blockIdx.y + F.nby * blockIdx.z);
    F.actQ0[b] = act;
    F.actQt[b] = kHydro;
    F.zeroQt[b] = 0u;
    F.zeroQ1[b] = 0u;
  }
}

// ---------------------------------------------------------------------------------------------------------------
// WGSL_M_PHYS (model.js:578-907): forcing stencils + microphysics, outbreak mode
// ---------------------------------------------------------------------------------------------------------------
// lateral sponge of one distance to the nearest side wall, and the top sponge at height z (model.js:611-626)
__device__ __forceinline__ float spongeLat1(const Uni& U, float e) {
  const float d = clampf(1.f - e / U.sponge.x, 0.f, 1.f);
  return d * (0.3f + 0.7f * d) / U.sponge.y;
}
__device__ __forceinline__ float spongeTop(const Uni& U, const Grid& g, float z) {
  const float ztop = float(g.nz) * U.dzv.x;
  if (z < U.sponge.z) return 0.f;
  const float s = sinf(1.5707963f * (z - U.sponge.z) / (ztop - U.sponge.z));
  return s * s / U.sponge.w;
}
// sponge tables (Fields::spz/slx/sly) and the per-level rain-speed density factor sqrt(rho_sfc / rho) (spz[4k+2])
__global__ void k_tables(Grid g, Uni U, const float* B, float* spz, float* slx, float* sly) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const float dx = U.dims.w, dz = U.dzv.x;
  if (t <= g.nz) {
    spz[4 * t + 0] = spongeTop(U, g, (float(t) + 0.5f) * dz);
    spz[4 * t + 1] = spongeTop(U, g, float(t) * dz);
    spz[4 * t + 2] = sqrtf(U.step.z / bsA(B, g.nz, t).z);
    spz[4 * t + 3] = 0.f;
  }
  const float Lx = float(g.nx) * dx, Ly = float(g.ny) * dx;
  if (t <= g.nx) {
    const float xf = float(t) * dx, xc = (float(t) + 0.5f) * dx;
    slx[2 * t] = spongeLat1(U, fminf(xf, Lx - xf));
    slx[2 * t + 1] = spongeLat1(U, fminf(xc, Lx - xc));
  }
  if (t <= g.ny) {
    const float yf = float(t) * dx, yc = (float(t) + 0.5f) * dx;
    sly[2 * t] = spongeLat1(U, fminf(yf, Ly - yf));
    sly[2 * t + 1] = spongeLat1(U, fminf(yc, Ly - yc));
  }
}
__device__ __forceinline__ float bsV(const float* B, int nz, int k, int ch) {
  const int kk = clampi(k, 0, nz - 1);
  if (ch == 0) return bsB(B, nz, kk).z;
  if (ch == 1) return bsB(B, nz, kk).w;
  if (ch == 3) return bsA(B, nz, kk).x;
  return 0.f;
}

// one slot of an append-only list per calling thread: one atomic per warp, slots in lane order
__device__ __forceinline__ unsigned warp_append(unsigned* ctr) {
  const unsigned mask = __activemask();
  const int lane = threadIdx.x & 31, leader = __ffs(mask) - 1;
  unsigned base = 0;
  if (lane == leader) base = atomicAdd(ctr, unsigned(__popc(mask)));
  base = __shfl_sync(mask, base, leader);
  return base + unsigned(__popc(mask & ((1u << lane) - 1u)));
}

// one texel of the physics pass; returns the hydrometeor and spare channels that the cell's new state holds (bits 1..7). MM: microphysics as the
// scheme (kMicroPlain), the scheme plus sampled (state, tendency) pairs (kMicroRecord), or queued for the surrogate
// kernel where it can act (kMicroSurrogate).
// Neighbour reads clamp to the edge of their texture (textureLoad with clamped coordinates, model.js:596-606): the byte
// offsets below are those of the clamped neighbours, for the staggered box [0, n] (V) and the cell box [0, n-1] (Q, aux,
// phi_t), computed once per texel. BND: boundary air masses present (else the target state is the
// base state, see tgtUb).
template <bool BND, int MM, bool HUR = false>
__device__ __forceinline__ unsigned phys_texel(const Grid& g, const Uni& U, const Fields& F, int par, int ci, int cj, int ck, bool dry,
                                               unsigned old) {
  unsigned hyd = 0u;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int o = g.at(ci, cj, ck);
  const unsigned b = unsigned(o) * 4u, sy = unsigned(g.px) * 4u, sz = unsigned(g.plane) * 4u;
  const float* __restrict__ Vu = F.V[1 - par][0];
  const float* __restrict__ Vv = F.V[1 - par][1];
  const float* __restrict__ Vw = F.V[1 - par][2];
  const float* __restrict__ Vth = F.V[1 - par][3];
  const float* __restrict__ A0 = F.aux[0];
  const float* __restrict__ A1 = F.aux[1];
  // staggered box
  const unsigned xm = ci > 0 ? b - 4u : b, xp = ci < nx ? b + 4u : b;
  const unsigned ym = cj > 0 ? b - sy : b, yp = cj < ny ? b + sy : b;
  const unsigned zm = ck > 0 ? b - sz : b, zp = ck < nz ? b + sz : b;
  // cell box: own index and +-1, clamped to [0, n-1]
  const unsigned xc0 = ci < nx ? b : b - 4u, xcp = ci < nx - 1 ? b + 4u : xc0;
  const unsigned yc0 = cj < ny ? b : b - sy, ycp = cj < ny - 1 ? b + sy : yc0;
  auto LP = [&](unsigned at) {
    if (!BND) return 0.f;
    return ldo(F.phT, at);
  };
  const float dx = U.dims.w, dz = U.dzv.x, dt = U.step.x;
  float V[4] = {ldo(Vu, b), ldo(Vv, b), ldo(Vw, b), ldo(Vth, b)};
  float out[4] = {V[0], V[1], V[2], V[3]};
  const float ix2 = U.der.z, iz2 = U.der.w;
  const float fc = U.cor.x;
  const float* __restrict__ Vc[4] = {Vu, Vv, Vw, Vth};
  auto lapH = [&](int ch, float me) { return ldo(Vc[ch], xp) + ldo(Vc[ch], xm) + ldo(Vc[ch], yp) + ldo(Vc[ch], ym) - 4.f * me; };
  auto lapZp = [&](int ch, float me, bool lo, bool hi) {
    const float m0 = me - bsV(F.B, nz, ck, ch);
    const float a = lo ? m0 : ldo(Vc[ch], zm) - bsV(F.B, nz, ck - 1, ch);
    const float b = hi ? m0 : ldo(Vc[ch], zp) - bsV(F.B, nz, ck + 1, ch);
    return a + b - 2.f * m0;
  };
  const float4 spk = __ldg(reinterpret_cast<const float4*>(F.spz) + ck);  // (top sponge centre, face, rain factor, -)
  const float2 slx = __ldg(reinterpret_cast<const float2*>(F.slx) + ci);  // (face, centre)
  const float2 sly = __ldg(reinterpret_cast<const float2*>(F.sly) + cj);
  // u
  if (cj < ny && ck < nz) {
    const float nux = 0.5f * (ldo(A0, xm) + ldo(A0, xc0)) + U.turb.y;
    const float nuy = 0.5f * (ldo(A1, xm) + ldo(A1, xc0)) + U.turb.y;
    float du = nux * lapH(0, V[0]) * ix2 + nuy * lapZp(0, V[0], ck == 0, ck == nz - 1) * iz2;
    const float ut = tgtUb<BND>(F, g, dz, ci, cj, ck);
    const float vbar = 0.25f * (ldo(Vv, xm) + V[1] + ldo(Vv, xm + yp - b) + ldo(Vv, yp));
    const float vtb = 0.5f * (tgtVb<BND>(F, g, dz, ci - 1, cj, ck) + tgtVb<BND>(F, g, dz, ci, cj + 1, ck));
    const float sp = fmaxf(slx.x, sly.y) + spk.x;
    if (BND) {
      const float nw = 0.5f * (l2d(F.lsfB, g, ci - 1, cj).w + l2d(F.lsfB, g, ci, cj).w);
      du += (sp + nw * (1.f / U.cor.y)) * (ut - V[0]);
    } else {
      du += sp * (ut - V[0]);
    }
    du += fc * (vbar - vtb);
    if (BND && ci > 0 && ci < nx) du -= (LP(b) - LP(b - 4u)) / dx;
    if (ck == 0 && U.turb.w > 0.5f) {
      float cd = U.micro.w;
      if (HUR) {  // sea / land drag (model.js:649-652)
        const float land = 0.5f * (__ldg(F.sfc + cj * nx + max(ci - 1, 0)).x + __ldg(F.sfc + min(cj, ny - 1) * nx + min(ci, nx - 1)).x);
        cd = cdSfc(U, sqrtf(V[0] * V[0] + vbar * vbar), land);
      }
      du += cd * (-sqrtf(V[0] * V[0] + vbar * vbar) * V[0] + sqrtf(ut * ut + vtb * vtb) * ut) / dz;
    }
    out[0] = V[0] + dt * du;
  } else out[0] = 0.f;
  // v
  if (ci < nx && ck < nz) {
    const float nux = 0.5f * (ldo(A0, ym) + ldo(A0, yc0)) + U.turb.y;
    const float nuy = 0.5f * (ldo(A1, ym) + ldo(A1, yc0)) + U.turb.y;
    float dv = nux * lapH(1, V[1]) * ix2 + nuy * lapZp(1, V[1], ck == 0, ck == nz - 1) * iz2;
    const float vt = tgtVb<BND>(F, g, dz, ci, cj, ck);
    const float ubar = 0.25f * (ldo(Vu, ym) + V[0] + ldo(Vu, xp + ym - b) + ldo(Vu, xp));
    const float utb = 0.5f * (tgtUb<BND>(F, g, dz, ci, cj - 1, ck) + tgtUb<BND>(F, g, dz, ci + 1, cj, ck));
    const float sp = fmaxf(slx.y, sly.x) + spk.x;
    if (BND) {
      const float nw = 0.5f * (l2d(F.lsfB, g, ci, cj - 1).w + l2d(F.lsfB, g, ci, cj).w);
      dv += (sp + nw * (1.f / U.cor.y)) * (vt - V[1]);
    } else {
      dv += sp * (vt - V[1]);
    }
    dv -= fc * (ubar - utb);
    if (BND && cj > 0 && cj < ny) dv -= (LP(b) - LP(b - sy)) / dx;
    if (ck == 0 && U.turb.w > 0.5f) {
      float cd = U.micro.w;
      if (HUR) {
        const float land = 0.5f * (__ldg(F.sfc + max(cj - 1, 0) * nx + ci).x + __ldg(F.sfc + min(cj, ny - 1) * nx + min(ci, nx - 1)).x);
        cd = cdSfc(U, sqrtf(ubar * ubar + V[1] * V[1]), land);
      }
      dv += cd * (-sqrtf(ubar * ubar + V[1] * V[1]) * V[1] + sqrtf(utb * utb + vt * vt) * vt) / dz;
    }
    out[1] = V[1] + dt * dv;
  } else out[1] = 0.f;
  // w
  if (ci < nx && cj < ny && ck > 0 && ck < nz) {
    const float nux = 0.5f * (ldo(A0, b - sz) + ldo(A0, b)) + U.turb.y;
    const float nuy = 0.5f * (ldo(A1, b - sz) + ldo(A1, b)) + U.turb.y;
    float dw = nux * lapH(2, V[2]) * ix2 + nuy * (ldo(Vw, b - sz) + ldo(Vw, b + sz) - 2.f * V[2]) * iz2;
    auto buoy = [&](int kk, unsigned at) {
      const float4 A = bsA(F.B, nz, kk);
      float h[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
      if (!dry) {
#pragma unroll
        for (int c = 0; c < 5; c++) h[c] = ldo(F.Q[1][1 + c], at);
      }
      return 9.81f * ((ldo(Vth, at) - A.x) / A.x + 0.608f * (ldo(F.Q[1][0], at) - A.y) -
                      (h[0] + h[1] + h[2] + h[3] + h[4]));
    };
    dw += 0.5f * (buoy(ck - 1, b - sz) + buoy(ck, b));
    if (BND) dw -= (LP(b) - LP(b - sz)) / dz;
    dw += (fmaxf(slx.y, sly.y) + spk.y) * (0.f - V[2]);
    const float4 civ = __ldg(F.ciMap + cj * nx + ci);
    if (!HUR && civ.x > 0.f) {  // hurricane mode starts storms as warm bubbles instead (model.js:686-687)
      const float z = float(ck) * dz;
      const float zz = fabsf(z - civ.z) / civ.w;
      if (zz < 1.f) {
        const float cv = cosf(1.5707963f * zz);
        dw += U.misc.w * civ.x * cv * fmaxf(civ.y * cv - V[2], 0.f);
      }
    }
    out[2] = V[2] + dt * dw;
  } else out[2] = 0.f;
  // theta + microphysics at cell centres
  if (ci < nx && cj < ny && ck < nz) {
    const float4 A = bsA(F.B, nz, ck), Bb = bsB(F.B, nz, ck);
    const float4 LAv = BND ? l2d(F.lsfA, g, ci, cj) : make_float4(0.f, 100.f, 0.f, 100.f);
    const float tth = BND ? tgtTh(F.B, g, dz, LAv, ck) : A.x, tqv = BND ? tgtQv(F.B, g, dz, LAv, ck) : A.y;
    const float sl = fmaxf(slx.y, sly.y);
    const float relax = BND ? sl + l2d(F.lsfB, g, ci, cj).w * (1.f / U.cor.y) : sl;
    const float nux = ldo(A0, b) * 3.f + U.turb.y, nuy = ldo(A1, b) * 3.f + U.turb.y;
    float th = V[3] + dt * (nux * lapH(3, V[3]) * ix2 + nuy * lapZp(3, V[3], ck == 0, ck == nz - 1) * iz2 + (relax + spk.x) * (tth - V[3]));
    // hydrometeor and spare channels: exactly +0 throughout a dry block's reach, so not read there (the sums below
    // then see the same +0 operands the loads would have returned)
    float q1[4] = {ldo(F.Q[1][0], b), 0.f, 0.f, 0.f}, q2[4] = {0.f, 0.f, 0.f, 0.f};
    float l1[3] = {0.f, 0.f, 0.f}, l1z[3] = {0.f, 0.f, 0.f};
    if (!dry) {
#pragma unroll
      for (int c = 0; c < 4; c++) {
        if (c) q1[c] = ldo(F.Q[1][c], b);
        q2[c] = ldo(F.Q[1][4 + c], b);
      }
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
      if (c && dry) continue;
      const float* __restrict__ q = F.Q[1][c];
      l1[c] = ldo(q, xcp) + ldo(q, xm) + ldo(q, ycp) + ldo(q, ym) - 4.f * q1[c];
      l1z[c] = (ck == 0 ? q1[c] : ldo(q, zm)) + (ck == nz - 1 ? q1[c] : ldo(q, b + sz)) - 2.f * q1[c];
    }
    const float qvb = (ck == 0 ? A.y : bsA(F.B, nz, ck - 1).y) + (ck == nz - 1 ? A.y : bsA(F.B, nz, ck + 1).y) - 2.f * A.y;
    l1z[0] -= qvb;
#pragma unroll
    for (int c = 0; c < 3; c++) q1[c] = q1[c] + dt * (nux * l1[c] * ix2 + nuy * l1z[c] * iz2);
    q1[0] += dt * relax * (tqv - q1[0]);
    const float xmx = (float(ci) + 0.5f) * dx, xmy = (float(cj) + 0.5f) * dx;
    float envDecay = 0.f;
    if (HUR) {  // the warm sea and the tropical environment (model.js:713-774)
      const float z = (float(ck) + 0.5f) * dz;
      th += dt * clampf((tth - V[3]) / U.hur2.x, -U.hur2.y, U.hur2.y);
      const float4 cs = __ldg(F.ciMap + cj * nx + ci);
      if (cs.x > 0.f) {  // storm starts: a warm, moist bubble through the push's depth
        const float zz = fabsf(z - cs.z) / cs.w;
        if (zz < 1.f) {
          const float f = cs.x * cosf(1.5707963f * zz) * cs.y / 8.f;
          th += dt * 1.2e-3f * f;
          q1[0] += dt * f / 600.f * fmaxf(0.97f * qvsat(V[3] * Bb.x, Bb.y, 0.f) - q1[0], 0.f);
        }
      }
      const float dxh = xmx - U.hur4.x, dyh = xmy - U.hur4.y;
      const float rS = sqrtf(dxh * dxh + dyh * dyh);
      const float wEnv = sstep(U.hur4.w, 1.5f * U.hur4.w, rS) / 3600.f;  // the far field held to the sounding
      th += dt * wEnv * (tth - V[3]);
      q1[0] += dt * wEnv * (tqv - q1[0]);
      envDecay = sstep(U.hur4.w, 1.5f * U.hur4.w, rS) / 1800.f;
      if (z < U.hur2.z) {  // boundary-layer thermals: coherent ~6 km cells living ~15 min
        const int o0 = g.at(ci, cj, 0);
        const float ua = 0.5f * (__ldg(F.V[1 - par][0] + o0) + __ldg(F.V[1 - par][0] + o0 + 1));
        const float va = 0.5f * (__ldg(F.V[1 - par][1] + o0) + __ldg(F.V[1 - par][1] + o0 + g.px));
        const float u1 = sqrtf(ua * ua + va * va);
        const float e = float(__ldg(F.clock)) / 900.f, e0 = floorf(e);
        const float qx = xmx / 6000.f, qy = xmy / 6000.f;
        const float r = 0.5f * mixf(gnoise2(qx + 37.1f * e0, qy + 11.3f * e0), gnoise2(qx + 37.1f * (e0 + 1.f), qy + 11.3f * (e0 + 1.f)),
                                    sstep(0.f, 1.f, e - floorf(e)));
        const float fu = fminf(u1 * u1 / 225.f, 1.f) * (1.f - sstep(20.f, 32.f, u1)) * (1.f - sstep(U.hur4.z, 1.5f * U.hur4.z, rS));
        th += dt * U.hur3.z * 2.f * r * fu * (1.f - z / U.hur2.z);
      }
      if (ck == 0) {  // the sea's sensible and latent heat; dissipative heating
        const float4 sf = __ldg(F.sfc + cj * nx + ci);
        const float land = clampf(sf.x, 0.f, 1.f);
        const float ua = 0.5f * (V[0] + ldo(Vu, b + 4u)), va = 0.5f * (V[1] + ldo(Vv, b + sy));
        const float u1 = sqrtf(ua * ua + va * va);
        const float ch = U.hur.y * U.hur2.w * fmaxf(u1, U.hur3.y) / dz;
        const float ps = fmaxf(U.hur.w + A.z * U.cn.y * __ldg(F.phi + g.pidx(ci, cj, ck)), 50000.f);
        const float ths = sf.y * powf(1.0e5f / ps, 0.2854f);
        th += dt * ch * (1.f - land) * (ths - V[3]);
        if (U.hur5.y > 0.5f) {
          const float cdh = cdSfc(U, u1, land);
          th += dt * cdh * u1 * u1 * u1 / (1005.7f * dz) / Bb.x;
        }
        const float qsS = qvsat(sf.y, ps, 0.f);
        const float qsL = qvsat(V[3] * Bb.x, ps, 0.f);
        q1[0] += dt * ch * ((1.f - land) * (qsS - q1[0]) + land * U.hur.z * fmaxf(qsL - q1[0], 0.f));
      }
    }
#pragma unroll
    for (int c = 0; c < 4; c++) {
      q1[c] = fmaxf(q1[c], 0.f);
      q2[c] = fmaxf(q2[c], 0.f);
    }
    const float pi0 = Bb.x, p0 = Bb.y, rho = A.z;
    float T = th * pi0;
    float qv = q1[0], qc = q1[1], qi = q1[2], qr = q1[3], qs = q2[0], qg = q2[1];
    const bool thm = U.micro2.z > 0.5f;
    MCell mc{T, qv, qc, qi, qr, qs, qg, fmaxf(q2[2], 0.f)};
    bool done = false;
    if (MM == kMicroSurrogate && surrogate_cell(mc)) {
      // surrogate cell: store the state before the microphysics and queue the cell; the surrogate kernel applies
      // the process tendencies, the saturation adjustment, the sponge removal and the clips (a full queue falls
      // through to the scheme here)
      const unsigned slot = warp_append(F.mlp_count);
      if (slot < F.mlp_cap) {
        reinterpret_cast<unsigned*>(F.mlp_buf)[slot] = unsigned(o);
        F.Q[0][0][o] = mc.qv; F.Q[0][1][o] = mc.qc; F.Q[0][2][o] = mc.qi; F.Q[0][3][o] = mc.qr;
        F.Q[0][4][o] = mc.qs; F.Q[0][5][o] = mc.qg; F.Q[0][6][o] = mc.nr; F.Q[0][7][o] = q2[3];
        out[3] = mc.T / pi0;
        hyd = kHydro;
        done = true;
      }
    }
    if (!done) {
      const MCell pre = mc;
      // with every hydrometeor exactly +0 each process rate is zero and the block leaves the cell as it is; the
      // saturation adjustment below still runs (a supersaturated cell condenses)
      if (!dry && (mc.qc > 0.f || mc.qi > 0.f || mc.qr > 0.f || mc.qs > 0.f || mc.qg > 0.f || mc.nr > 0.f))
        micro_processes(U, dt, p0, rho, spk.z, mc);
      if (MM == kMicroRecord && surrogate_cell(pre) &&
          float(hash3i(ci, cj, ck ^ int(__float_as_uint(float(__ldg(F.clock))) * 2654435761u)) >> 8u) * (1.f / 16777216.f) < F.mlp_rate) {
        // one (state, process tendency) pair of the scheme: 12 inputs, 10 tendencies (before the saturation
        // adjustment), the cell's texel offset (as bits), the model time of the step (the two order the pairs
        // canonically: ob_mlp_sort_pairs)
        const unsigned slot = warp_append(F.mlp_count);
        if (slot < F.mlp_cap) {
          float* r = F.mlp_buf + size_t(slot) * 24;
          const float x[12] = {pre.T, p0, rho, pre.qv, pre.qc, pre.qr, pre.qi, pre.qs, pre.qg, pre.nr, q2[3], V[2]};
          const float y[12] = {mc.T - pre.T, mc.qv - pre.qv, mc.qc - pre.qc, mc.qi - pre.qi, mc.qr - pre.qr, mc.qs - pre.qs,
                               mc.qg - pre.qg, mc.nr - pre.nr, 0.f, 0.f, __uint_as_float(unsigned(o)), float(__ldg(F.clock))};
#pragma unroll
          for (int e = 0; e < 12; e++) {
            r[e] = x[e];
            r[12 + e] = y[e];
          }
        }
      }
      sat_adjust(p0, mc);
      T = mc.T; qv = mc.qv; qc = mc.qc; qi = mc.qi; qr = mc.qr; qs = mc.qs; qg = mc.qg;
      float nr = mc.nr;
      th = T / pi0;
      // 1 / (1 + 0) == 1 exactly: no division outside the sponge (and, in hurricane mode, the far-field decay)
      const float keep = HUR ? 1.f / (1.f + 2.f * dt * sl + dt * envDecay) : (sl > 0.f ? 1.f / (1.f + 2.f * dt * sl) : 1.f);
      qc *= keep; qi *= keep; qr *= keep; qs *= keep; qg *= keep; nr *= keep;
      const float nv[8] = {0.f, qc, qi, qr, qs, qg, thm ? nr : q2[2], q2[3]};
      sto(F.Q[0][0], b, fmaxf(qv, 0.f));
      const bool any = qc > 0.f || qi > 0.f || qr > 0.f || qs > 0.f || qg > 0.f || nv[6] > 0.f || nv[7] > 0.f;
      if (any || old) {  // else the channels below are zero here and slot 0 already holds zeros
#pragma unroll
        for (int c = 1; c < 8; c++) {
          if (nv[c] > 0.f) hyd |= 1u << c;
          if (nv[c] > 0.f || ((old >> c) & 1u)) sto(F.Q[0][c], b, c == 7 ? nv[c] : fmaxf(nv[c], 0.f));
        }
      }
      out[3] = th;
    }
  }
  const float s2 = out[0] * out[0] + out[1] * out[1] + out[2] * out[2];
  if (s2 > 0.999f * U.misc.x * U.misc.x) {   // no root for a speed below the cap
    const float sp = sqrtf(s2);
    if (sp > U.misc.x) {
      const float s = U.misc.x / sp;
      out[0] *= s; out[1] *= s; out[2] *= s;
    }
  }
  if (!(out[0] == out[0]) || !(out[1] == out[1]) || !(out[2] == out[2]) || !(out[3] == out[3])) {
    out[0] = bsB(F.B, nz, ck).z; out[1] = bsB(F.B, nz, ck).w; out[2] = 0.f; out[3] = bsA(F.B, nz, ck).x;
    atomicAdd(F.flags, 1u);
  }
#pragma unroll
  for (int c = 0; c < 4; c++) sto(F.V[par][c], b, out[c]);
  return hyd;
}

// The clear-air flags of a physics block (one 32 x 4 brick of cells; blocks past the last brick hold only faces, which
// read and write no scalar), the same for all its threads: dry = Q slot 1 holds no hydrometeor and no nonzero spare in
// the brick and its six face neighbours (ADVQ2 wrote them as zeros), which bound every scalar read of the block; old
// = the hydrometeor and spare channels that the previous physics pass left in slot 0 of the brick (actQ0), so a cell
// whose new value of another channel is zero need not store it again. Hurricane mode's 2-dx filter writes slot 0 between
// physics passes, so there every channel counts as held.
template <bool HUR>
__device__ __forceinline__ void phys_flags(const Grid& g, const Fields& F, int BX, int BY, int ck, bool& dry, unsigned& old) {
  dry = false;
  old = kHydro;
  if (BX >= F.nbx || BY >= F.nby || ck >= g.nz) return;
  const int lane = threadIdx.x & 31;
  unsigned z = kHydro;
  if (lane < 7) {
    const int bx = BX + (lane == 1 ? -1 : lane == 2 ? 1 : 0), by = BY + (lane == 3 ? -1 : lane == 4 ? 1 : 0);
    const int bz = ck + (lane == 5 ? -1 : lane == 6 ? 1 : 0);
    if (bx >= 0 && bx < F.nbx && by >= 0 && by < F.nby && bz >= 0 && bz < g.nz) z = F.zeroQ1[bx + F.nbx * (by + F.nby * bz)];
  }
  dry = __all_sync(0xffffffffu, z == kHydro);
  if (!HUR) old = F.actQ0[BX + F.nbx * (BY + F.nby * ck)];
}

// BND: 1 = boundary air masses present, 0 = none, -1 = decided per launch from the uniforms (U.cor.z)
template <int MM, bool HUR = false, int BND = -1>
__device__ __forceinline__ void phys_body(const Grid& g, const Uni& U, const Fields& F, int par, const int BX, const int BY, const int BZ) {
  const int ci = BX * blockDim.x + threadIdx.x, cj = BY * blockDim.y + threadIdx.y, ck = BZ;
  bool dry;
  unsigned old, hyd = 0u;
  phys_flags<HUR>(g, F, BX, BY, ck, dry, old);
  if (ci <= g.nx && cj <= g.ny && ck <= g.nz)
    hyd = (BND == 1 || (BND < 0 && U.cor.z > 0.5f)) ? phys_texel<BND != 0, MM, HUR>(g, U, F, par, ci, cj, ck, dry, old)
                                                    : phys_texel<false, MM, HUR>(g, U, F, par, ci, cj, ck, dry, old);
  // the channels this block's brick holds, for the next step's scalar advection
  hyd = block_or(hyd);
  if (threadIdx.x == 0 && threadIdx.y == 0 && int(BX) < F.nbx && int(BY) < F.nby && ck < g.nz)
    F.actQ0[BX + F.nbx * (BY + F.nby * ck)] = hyd;
}
// one kernel per microphysics mode and per presence of boundary air masses: with one texel body per kernel, ten
// 128-thread blocks fit on an SM at 48 registers without spilling (the surrogate with boundaries keeps nine), where the
// kernel holding both bodies needed 56 registers at nine blocks; 0.64 -> 0.61 ms at 640 x 640 x 40
template <int MM, int BND>
__global__ void __launch_bounds__(128, (MM == kMicroSurrogate && BND == 1) ? 9 : 10) k_phys(Grid g, Uni U, Fields F) {
  constexpr int par = 0;
  phys_body<MM, false, BND>(g, U, F, par, blockIdx.x, blockIdx.y, blockIdx.z);
}
template <int BND>
__global__ void __launch_bounds__(128) k_phys_hur(Grid g, Uni U, Fields F) {
  phys_body<kMicroPlain, true, BND>(g, U, F, 0, blockIdx.x, blockIdx.y, blockIdx.z);
}
template <int MM>
__global__ void __launch_bounds__(128, 9) k_phys_grp(const uint2* __restrict__ map, int par) {
  OB_GROUP_RESOLVE
  phys_body<MM>(c_members[mem].g, c_members[mem].U, c_members[mem].F, par, gbx, gby, gbz);
}

// ---------------------------------------------------------------------------------------------------------------
// WGSL_M_DIV (model.js:909-925): density-weighted divergence / dt on the padded solve grid
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void div_body(const Grid& g, const Uni& U, const Fields& F, int par, const int BX, const int BY, const int BZ) {
  OB_TEXEL_LOOP_BEGIN(g.nx - 1, g.ny - 1, g.nz - 1)
  const int o = g.at(ci, cj, ck);
  const float* u = F.V[par][0];   // PHYS has just written these
  const float* v = F.V[par][1];
  const float* w = F.V[par][2];
  const float rc = bsA(F.B, g.nz, ck).z;
  const float wt = ck == g.nz - 1 ? 0.f : ld_late(w + o + g.plane);
  const float wb = ck == 0 ? 0.f : ld_late(w + o);
  // the reference divides by dx, dz and dt (model.js:909-925); multiplying by the host's reciprocals (1/dx, 1/dz in
  // dzv, 1/dt in der2) saves three IEEE divisions per cell and moves r by a few ulp
  const float d = rc * (ld_late(u + o + 1) - ld_late(u + o) + ld_late(v + o + g.px) - ld_late(v + o)) * U.dzv.y +
                  (rhoW(F.B, g.nz, ck + 1) * wt - rhoW(F.B, g.nz, ck) * wb) * U.dzv.z;
  const float r = d * U.der2.x;
  if (F.rhs_hi) {  // tensor-core solve: write the split directly in its [z][y][x] layout with pitch rhs_ld
    const long o2 = (long(ck) * g.nyp + (cj + g.pad)) * F.rhs_ld + (ci + g.pad);
    const __nv_bfloat16 h = __float2bfloat16_rn(r);
    F.rhs_hi[o2] = h;
    if (F.rhs_lo) F.rhs_lo[o2] = __float2bfloat16_rn(r - __bfloat162float(h));   // none when no pass reads it
  }
  if (F.rhs) F.rhs[g.pidx(ci, cj, ck)] = r;  // fp32 solve, or the residual of the refined solve
}
__global__ void k_div(Grid g, Uni U, Fields F) {
  tc::grid_wait();
  div_body(g, U, F, 0, blockIdx.x, blockIdx.y, blockIdx.z);
}
__global__ void k_div_grp(const uint2* __restrict__ map, int par) {
  OB_GROUP_RESOLVE
  div_body(c_members[mem].g, c_members[mem].U, c_members[mem].F, par, gbx, gby, gbz);
}

// ---------------------------------------------------------------------------------------------------------------
// WGSL_M_PROJ (model.js:927-946): u -= dt grad(phi), phi from the padded solve
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void proj_body(const Grid& g, const Uni& U, const Fields& F, int par, const int BX, const int BY, const int BZ) {
  OB_TEXEL_LOOP_BEGIN(g.nx, g.ny, g.nz)
  auto P = [&](int a, int b, int c) {   // the solve's last kernel has just written phi
    return ld_late(F.phi + g.pidx(clampi(a, -g.pad, g.nx + g.pad - 1), clampi(b, -g.pad, g.ny + g.pad - 1), clampi(c, 0, g.nz - 1)));
  };
  const int o = g.at(ci, cj, ck);
  const float kx = U.der.x, kz = U.der.y;
  const float pc = P(ci, cj, ck);
  float u = __ldg(F.V[par][0] + o), v = __ldg(F.V[par][1] + o), w = __ldg(F.V[par][2] + o);
  if (cj < g.ny && ck < g.nz) u = u - kx * (pc - P(ci - 1, cj, ck));
  if (ci < g.nx && ck < g.nz) v = v - kx * (pc - P(ci, cj - 1, ck));
  if (ci < g.nx && cj < g.ny && ck > 0 && ck < g.nz) w = w - kz * (pc - P(ci, cj, ck - 1));
  else w = 0.f;
  F.V[1 - par][0][o] = u;
  F.V[1 - par][1][o] = v;
  F.V[1 - par][2][o] = w;
  F.V[1 - par][3][o] = __ldg(F.V[par][3] + o);
}
__global__ void k_proj(Grid g, Uni U, Fields F) {
  tc::grid_wait();
  proj_body(g, U, F, 0, blockIdx.x, blockIdx.y, blockIdx.z);
}
__global__ void k_proj_grp(const uint2* __restrict__ map, int par) {
  OB_GROUP_RESOLVE
  proj_body(c_members[mem].g, c_members[mem].U, c_members[mem].F, par, gbx, gby, gbz);
}

// accumulated surface precipitation (no counterpart in the reference): rho(0) sum_x q_x vt_x at the lowest level
__device__ __forceinline__ void rain_body(const Grid& g, const Uni& U, const Fields& F, int par, const int BX, const int BY, const int BZ) {
  const int i = BX * blockDim.x + threadIdx.x, j = BY * blockDim.y + threadIdx.y;
  if (i >= g.nx || j >= g.ny) return;
  const int o = g.at(i, j, 0);
  const Fall fl{U.step.z, U.micro2.z > 0.5f, U.hur3.w > 0.5f && U.micro2.z <= 0.5f};
  const float rho = bsA(F.B, g.nz, 0).z;
  const float qr = F.Q[0][3][o], qs = F.Q[0][4][o], qg = F.Q[0][5][o];
  const float2 fv = fl.vtRain(qr, F.Q[0][6][o], rho);
  const double flux = double(rho) * (double(qr) * double(fv.x) + double(qs) * double(fl.vtS(qs, rho)) + double(qg) * double(fl.vtGrau(qg, rho)));
  F.rain[j * g.nx + i] += flux * double(U.step.x);
  if (i == 0 && j == 0) *F.clock += double(U.step.x);  // the step's last pass advances the model time
}
__global__ void k_rain(Grid g, Uni U, Fields F) { rain_body(g, U, F, 0, blockIdx.x, blockIdx.y, blockIdx.z); }
__global__ void k_rain_grp(const uint2* __restrict__ map, int par) {
  OB_GROUP_RESOLVE
  rain_body(c_members[mem].g, c_members[mem].U, c_members[mem].F, par, gbx, gby, gbz);
}

// ---------------------------------------------------------------------------------------------------------------
// WGSL_M_MAP (model.js:1028-1100): 16 diagnostics per column
// ---------------------------------------------------------------------------------------------------------------
// A warp takes 32 columns of a row (one brick wide) and W of them share the levels, 4 W at a time; a block of eight has 8 / W
// rows. What needs an order (the updraft-helicity sum upwards, the cloud-top radiance downwards) leaves its terms in
// shared memory for the first of the W to add in that order, so W changes no bit; the maxima need none. Levels whose brick
// holds no precipitation have -30 dBZ and levels without any hydrometeor are transparent (F.actQ0). One thread per column
// (column "1 thread", 2-D blocks) spends its time on the latency of nz levels in turn; but the sums and what follows them
// are left to one warp in W, which tells where there are warps enough without sharing. us:
//                    1 thread   W = 8      4      2      1
//   64 x 64 x 40         36.6    13.6   19.0   29.2   51.5
//   203 x 157 x 16       16.8    14.2   11.7   15.1   22.8
//   260 x 260 x 40       60.6    36.5   36.7   38.2   56.1
//   400 x 380 x 40       97.6    94.1   77.6   76.2   87.7
//   640 x 640 x 40      241     252    213    190    213
//   900 x 900 x 16      174     291    208    173    159
// (lin scheme, a storm every 60 km)
constexpr int kMapWarps = 8;
template <int W>
__global__ void __launch_bounds__(32 * kMapWarps) k_maps(Grid g, Uni U, Fields F, float4* out) {
  constexpr int par = 0, R = kMapWarps / W, LV = 4 * W;
  __shared__ float s_uh[R][LV][32], s_a[R][LV][32], s_t[R][LV][32];
  __shared__ float s_max[2][kMapWarps][32];
  const int row = int(threadIdx.y) / W, warp = int(threadIdx.y) % W, lane = threadIdx.x;
  const int bx = int(blockIdx.x % unsigned(F.nbx)), j = int(blockIdx.x / unsigned(F.nbx)) * R + row;
  const int nx = g.nx, ny = g.ny, nz = g.nz, i = bx * 32 + lane;
  const bool in = i < nx && j < ny;
  const float* const* V = F.V[par];
  auto L = [&](int ch, int a, int b, int c) { return __ldg(V[ch] + g.at(clampi(a, 0, nx), clampi(b, 0, ny), clampi(c, 0, nz))); };
  auto cvel = [&](int a, int b, int c, float v[3]) {
    v[0] = 0.5f * (L(0, a, b, c) + L(0, a + 1, b, c));
    v[1] = 0.5f * (L(1, a, b, c) + L(1, a, b + 1, c));
    v[2] = 0.5f * (L(2, a, b, c) + L(2, a, b, c + 1));
  };
  const Fall fl{U.step.z, U.micro2.z > 0.5f, U.hur3.w > 0.5f && U.micro2.z <= 0.5f};
  auto held = [&](int k) { return __ldg(F.actQ0 + bx + F.nbx * ((j >> 2) + F.nby * k)); };
  auto dbz = [&](int k) {
    if (!(held(k) & 0x38u)) return -30.f;   // no rain, snow or graupel
    const int o = g.at(i, j, k);
    const float rho = bsA(F.B, nz, k).z;
    const float T = __ldg(V[3] + o) * bsB(F.B, nz, k).x;
    const float Zr = fl.zRain(__ldg(F.Q[0][3] + o), __ldg(F.Q[0][6] + o), rho);
    const float Zs = 9.80e8f * powf(fmaxf(rho * __ldg(F.Q[0][4] + o), 0.f), 1.75f) * 0.224f * 4.f;
    const float Zg = fl.zGrau(__ldg(F.Q[0][5] + o), rho, T);
    const float Z = Zr + Zs + Zg;
    return Z > 1e-3f ? 10.f * logf(Z) / 2.302585f : -30.f;
  };
  auto zeta = [&](int k) {
    float a[3], b[3], c[3], d[3];
    cvel(i + 1, j, k, a);
    cvel(i - 1, j, k, b);
    cvel(i, j + 1, k, c);
    cvel(i, j - 1, k, d);
    return (a[1] - b[1] - c[0] + d[0]) / (2.f * U.dims.w);
  };
  const float dz = U.dzv.x;
  float comp = -30.f, wmx = 0.f, uh = 0.f;
  const int k12 = min(int(12000.f / dz), nz - 1);
  for (int k0 = 0; k0 < k12; k0 += LV) {
    const int n = min(LV, k12 - k0);
    for (int t = warp; t < n; t += W) {
      const int k = k0 + t;
      float term = 0.f;
      if (in) {
        const float w = 0.5f * (L(2, i, j, k) + L(2, i, j, k + 1));
        wmx = fmaxf(wmx, w);
        comp = fmaxf(comp, dbz(k));
        const float z = (float(k) + 0.5f) * dz;
        if (z > 2000.f && z < 5000.f && w > 0.f) term = w * fmaxf(zeta(k), 0.f) * dz;
      }
      s_uh[row][t][lane] = term;
    }
    __syncthreads();
    if (warp == 0)
      for (int t = 0; t < n; t++) uh += s_uh[row][t][lane];
    __syncthreads();
  }
  s_max[0][threadIdx.y][lane] = comp;
  s_max[1][threadIdx.y][lane] = wmx;
  // radiance of the column from the top down: opacity and temperature of each level, then the sum in order
  float tr = 1.f, bt = 0.f;
  for (int k0 = nz - 1; k0 >= 0; k0 -= LV) {
    const int n = min(LV, k0 + 1);
    for (int t = warp; t < n; t += W) {
      const int k = k0 - t;
      float a = 0.f, T = 0.f;
      if (in) T = __ldg(V[3] + g.at(i, j, k));
      if (in && (held(k) & 0x3eu)) {
        const int o = g.at(i, j, k);
        const float dtau = (80.f * __ldg(F.Q[0][1] + o) + 60.f * __ldg(F.Q[0][2] + o) + 25.f * __ldg(F.Q[0][4] + o) + 4.f * __ldg(F.Q[0][5] + o) +
                            1.f * __ldg(F.Q[0][3] + o)) * bsA(F.B, nz, k).z * dz;
        a = 1.f - expf(-dtau);
      }
      s_a[row][t][lane] = a;
      s_t[row][t][lane] = T;
    }
    __syncthreads();
    if (warp == 0 && tr >= 1e-3f)
      for (int t = 0; t < n; t++) {
        const float a = s_a[row][t][lane];
        bt += tr * a * s_t[row][t][lane] * bsB(F.B, nz, k0 - t).x;
        tr *= 1.f - a;
        if (tr < 1e-3f) break;
      }
    __syncthreads();
  }
  if (warp != 0 || !in) return;
#pragma unroll
  for (int w = 1; w < W; w++) {
    comp = fmaxf(comp, s_max[0][row * W + w][lane]);
    wmx = fmaxf(wmx, s_max[1][row * W + w][lane]);
  }
  const int k1 = clampi(int(1000.f / dz), 1, nz - 2);
  float v0[3], v1[3];
  cvel(i, j, 0, v0);
  cvel(i, j, k1, v1);
  const float conv = -((L(0, i + 1, j, 0) - L(0, i, j, 0) + L(1, i, j + 1, 0) - L(1, i, j, 0)) / U.dims.w) * 1000.f;
  const int idx = j * nx + i, n2 = nx * ny;
  out[idx] = make_float4(comp, dbz(k1), L(3, i, j, 0) - bsA(F.B, nz, 0).x, zeta(k1));
  out[idx + n2] = make_float4(wmx, uh, conv, sqrtf(v0[0] * v0[0] + v0[1] * v0[1]));
  out[idx + 2 * n2] = make_float4(v0[0], v0[1], v1[0], v1[1]);
  const float sst = F.sfc[idx].y;
  bt += tr * (sst > 200.f ? sst : L(3, i, j, 0) * bsB(F.B, nz, 0).x);
  const float ps = bsA(F.B, nz, 0).z * U.cn.z * __ldg(F.phi + (i + g.pad) + g.nxp * (j + g.pad)) / 100.f;
  const int k5 = clampi(int(5000.f / dz), 1, nz - 2);
  out[idx + 3 * n2] = make_float4(ps, bt, U.hur2.w * sqrtf(v0[0] * v0[0] + v0[1] * v0[1]), zeta(k5));
}

// ---------------------------------------------------------------------------------------------------------------
// layout conversion between the texel float4 layout of the C ABI and the device SoA layout
// ---------------------------------------------------------------------------------------------------------------
__global__ void k_pack(Grid g, Ptr8 src, int nch, int X, int Y, int Z, float* dst) {
  OB_BLOCKS_DIRECT
  OB_TEXEL_LOOP_BEGIN(X - 1, Y - 1, Z - 1)
  const int o = g.at(ci, cj, ck);
  const size_t t = (size_t(ck) * Y + cj) * X + ci;
#pragma unroll
  for (int c = 0; c < 8; c++)
    if (c < nch) dst[t * nch + c] = src.p[c][o];
}
__global__ void k_unpack(Grid g, Ptr8 dst, int nch, int X, int Y, int Z, const float* src) {
  OB_BLOCKS_DIRECT
  OB_TEXEL_LOOP_BEGIN(X - 1, Y - 1, Z - 1)
  const int o = g.at(ci, cj, ck);
  const size_t t = (size_t(ck) * Y + cj) * X + ci;
#pragma unroll
  for (int c = 0; c < 8; c++)
    if (c < nch) dst.p[c][o] = src[t * nch + c];
}

// ---------------------------------------------------------------------------------------------------------------
// hurricane mode: the advection with midpoint trajectories and settling ice, the pressure force carried along the
// trajectories (WGSL_M_PREP) and the 2-dx filter (WGSL_M_FILT), one thread per texel.
// ---------------------------------------------------------------------------------------------------------------
// the winds at a point in grid units, from the true winds (model.js:420-423)
__device__ __forceinline__ void velAt(const Fields& F, const Grid& g, int par, float x, float y, float z, float v[3]) {
  v[0] = sampleVch(F.V[par][0], g, 0, x, y, z);
  v[1] = sampleVch(F.V[par][1], g, 1, x, y, z);
  v[2] = sampleVch(F.V[par][2], g, 2, x, y, z);
}
// departure (s = 1) or forward (s = -1) point: first order, or with the wind at the midpoint when cn.w (model.js:424-433)
__device__ __forceinline__ void traceH(const Uni& U, const Fields& F, const Grid& g, int par, const float k[3], float px, float py,
                                       float pz, const float v[3], float s, float& x, float& y, float& z) {
  if (U.cn.w < 0.5f) {
    traceV(g, k, px, py, pz, v, s, x, y, z);
    return;
  }
  float mx, my, mz, vm[3];
  traceV(g, k, px, py, pz, v, 0.5f * s, mx, my, mz);
  velAt(F, g, par, mx, my, mz, vm);
  traceV(g, k, px, py, pz, vm, s, x, y, z);
}
// the same for a cell centre and something falling at `fall` (model.js:494-499)
__device__ __forceinline__ void traceQH(const Uni& U, const Fields& F, const Grid& g, int par, const float k[3], const float p[3],
                                        const float v[3], float fall, float s, float& x, float& y, float& z) {
  if (U.cn.w < 0.5f) {
    traceQ(g, k, p, v, fall, s, x, y, z);
    return;
  }
  const float mx = clampf(p[0] - 0.5f * s * k[0] * v[0], 0.f, float(g.nx));
  const float my = clampf(p[1] - 0.5f * s * k[1] * v[1], 0.f, float(g.ny));
  const float mz = clampf(p[2] - 0.5f * s * k[2] * (v[2] - fall), 0.f, float(g.nz));
  float vm[3];
  velAt(F, g, par, mx, my, mz, vm);
  traceQ(g, k, p, vm, fall, s, x, y, z);
}

__global__ void k_prep(Grid g, Uni U, Fields F) {
  constexpr int par = 0;
  OB_BLOCKS_DIRECT
  OB_TEXEL_LOOP_BEGIN(g.nx, g.ny, g.nz)
  auto P = [&](int a, int b, int c) {
    return __ldg(F.phi + g.pidx(clampi(a, -g.pad, g.nx + g.pad - 1), clampi(b, -g.pad, g.ny + g.pad - 1), clampi(c, 0, g.nz - 1)));
  };
  const int o = g.at(ci, cj, ck);
  const float f = U.cn.x * U.cn.y;
  const float kx = f * U.step.x / U.dims.w, kz = f * U.step.x / U.dzv.x;
  const float pc = P(ci, cj, ck);
  float u = __ldg(F.V[par][0] + o), v = __ldg(F.V[par][1] + o), w = __ldg(F.V[par][2] + o);
  if (cj < g.ny && ck < g.nz) u = u - kx * (pc - P(ci - 1, cj, ck));
  if (ci < g.nx && ck < g.nz) v = v - kx * (pc - P(ci, cj - 1, ck));
  if (ci < g.nx && cj < g.ny && ck > 0 && ck < g.nz) w = w - kz * (pc - P(ci, cj, ck - 1));
  F.Vp[0][o] = u;
  F.Vp[1][o] = v;
  F.Vp[2][o] = w;
  F.Vp[3][o] = __ldg(F.V[par][3] + o);
}
// the domain's largest |u|, |v| and |w| (as the bits of a float, which order as integers; a NaN counts as infinite) into
// F.vmax, which the host has set to 0: they bound every trajectory of the step
__global__ void __launch_bounds__(256) k_wind_max(Grid g, Fields F) {
  __shared__ unsigned red[3];
  if (threadIdx.x < 3) red[threadIdx.x] = 0u;
  __syncthreads();
  const long rows = long(g.ny + 1) * (g.nz + 1);
  unsigned m[3] = {0u, 0u, 0u};
  for (long r = long(blockIdx.x) * 8 + (threadIdx.x >> 5); r < rows; r += long(gridDim.x) * 8) {   // a warp per row
    const long base = r * g.px;
    for (int i = threadIdx.x & 31; i <= g.nx; i += 32)
#pragma unroll
      for (int c = 0; c < 3; c++) m[c] = max(m[c], __float_as_uint(__ldg(F.V[0][c] + base + i)) & 0x7fffffffu);
  }
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const unsigned w = __reduce_max_sync(0xffffffffu, m[c]);
    if ((threadIdx.x & 31) == 0) atomicMax(&red[c], w);
  }
  __syncthreads();
  if (threadIdx.x < 3) atomicMax(F.vmax + threadIdx.x, red[threadIdx.x]);
}

// 4th-order horizontal hyperdiffusion of V and Q into V[1-par], Q slot 1 (model.js:948-994)
__global__ void k_filt(Grid g, Uni U, Fields F) {
  constexpr int par = 0;
  OB_BLOCKS_DIRECT
  OB_TEXEL_LOOP_BEGIN(g.nx, g.ny, g.nz)
  const float a = U.hur5.z;
  auto bih = [&](const float* __restrict__ f, int X, int Y) {
    auto L = [&](int i, int j) { return __ldg(f + g.at(clampi(i, 0, X), clampi(j, 0, Y), ck)); };
    return 20.f * L(ci, cj) - 8.f * (L(ci + 1, cj) + L(ci - 1, cj) + L(ci, cj + 1) + L(ci, cj - 1)) +
           2.f * (L(ci + 1, cj + 1) + L(ci + 1, cj - 1) + L(ci - 1, cj + 1) + L(ci - 1, cj - 1)) + L(ci + 2, cj) + L(ci - 2, cj) +
           L(ci, cj + 2) + L(ci, cj - 2);
  };
  const int o = g.at(ci, cj, ck);
#pragma unroll
  for (int c = 0; c < 4; c++) {
    float val = __ldg(F.V[par][c] + o) - a * bih(F.V[par][c], g.nx, g.ny);
    if (c == 2 && (ck == 0 || ck >= g.nz)) val = 0.f;  // the lid / ground faces of w stay zero
    F.V[1 - par][c][o] = val;
  }
  if (ci < g.nx && cj < g.ny && ck < g.nz) {
#pragma unroll
    for (int c = 0; c < 8; c++) F.Q[1][c][o] = fmaxf(__ldg(F.Q[0][c] + o) - a * bih(F.Q[0][c], g.nx - 1, g.ny - 1), 0.f);
  }
}

// ADVV1/2 of hurricane mode (model.js:434-481): trajectories from the true winds, values carried from Vp. As in the outbreak
// passes, ADVV1 keeps the limiter's window of its departure sample, so that ADVV2 traces forwards alone (a trajectory
// costs 24 gathers for its midpoint wind): ADVV2 292 -> 145 us at 256 x 224 x 40.
__global__ void k_advv1_hur(Grid g, Uni U, Fields F) {
  constexpr int par = 0;
  OB_BLOCKS_DIRECT
  OB_TEXEL_LOOP_BEGIN(g.nx, g.ny, g.nz)
  const Loc L = localVel(F, g, par, ci, cj, ck);
  const float kk[3] = {U.der.x, U.der.x, U.der.y};
  const float fi = float(ci), fj = float(cj), fk = float(ck);
  const unsigned o = 4u * unsigned(g.at(ci, cj, ck));
  const float P[4][3] = {{fi, fj + 0.5f, fk + 0.5f}, {fi + 0.5f, fj, fk + 0.5f}, {fi + 0.5f, fj + 0.5f, fk}, {fi + 0.5f, fj + 0.5f, fk + 0.5f}};
  const float* vel[4] = {L.vu, L.vv, L.vw, L.vc};
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const float ox = c == 0 ? 0.f : 0.5f, oy = c == 1 ? 0.f : 0.5f, oz = c == 2 ? 0.f : 0.5f;
    float x, y, z, lo, hi;
    traceH(U, F, g, par, kk, P[c][0], P[c][1], P[c][2], vel[c], 1.f, x, y, z);
    const float t = trilerpB_mm(F.Vp[c], g, g.nx + 1, g.ny + 1, g.nz + 1, x - ox, y - oy, z - oz, lo, hi);
    sto(F.Vt[c], o, t);
    sto(F.Vlo[c], o, lo);
    sto(F.Vhi[c], o, hi);
  }
}
__global__ void k_advv2_hur(Grid g, Uni U, Fields F) {
  constexpr int par = 0;
  OB_BLOCKS_DIRECT
  OB_TEXEL_LOOP_BEGIN(g.nx, g.ny, g.nz)
  const Loc L = localVel(F, g, par, ci, cj, ck);
  const float kk[3] = {U.der.x, U.der.x, U.der.y};
  const float fi = float(ci), fj = float(cj), fk = float(ck);
  const float P[4][3] = {{fi, fj + 0.5f, fk + 0.5f}, {fi + 0.5f, fj, fk + 0.5f}, {fi + 0.5f, fj + 0.5f, fk}, {fi + 0.5f, fj + 0.5f, fk + 0.5f}};
  const float* vel[4] = {L.vu, L.vv, L.vw, L.vc};
  const float cx = L.vc[0] * kk[0], cy = L.vc[1] * kk[1], cz = L.vc[2] * kk[2];
  const float cour = sqrtf(cx * cx + cy * cy + cz * cz);
  const float sm = 0.5f * U.misc.y * clampf(cour / 0.35f, U.dzv.w, 1.f);
  const unsigned o = 4u * unsigned(g.at(ci, cj, ck));
#pragma unroll
  for (int c = 0; c < 4; c++) {
    float x, y, z;
    traceH(U, F, g, par, kk, P[c][0], P[c][1], P[c][2], vel[c], -1.f, x, y, z);
    const float b = sampleVch(F.Vt[c], g, c, x, y, z);
    const float hat = ldo(F.Vt[c], o), old = ldo(F.Vp[c], o);
    const float r = hat + sm * (old - b);
    sto(F.V[1 - par][c], o, clampf(r, ldo(F.Vlo[c], o), ldo(F.Vhi[c], o)));
  }
}

// ADVQ1/2 of hurricane mode (model.js:500-576): maritime graupel, settling ice. Channels absent from a block's reach are
// skipped as in the outbreak passes, but the reach comes from the step's largest winds (F.vmax) instead of the block's own
// departure points, which would need every channel's trajectory first: a trajectory's wind is a mean of winds, so it ends
// within dt / dx of that bound (and, downwards and upwards, of it plus the largest fall speed). Channels at the air's
// speed share one trajectory each way. 256 x 224 x 40 with a storm every 60 km: ADVQ1 210 -> 109 us, ADVQ2 589 -> 220 us,
// and PHYS, which finds dry blocks by the same flags, 222 -> 193 us; the winds' maxima take 10 us.
__device__ __forceinline__ unsigned reach_channels(const Grid& g, const Uni& U, const Fields& F, const unsigned int* flagsA,
                                                   const unsigned int* flagsB) {
  __shared__ unsigned held;
  if (threadIdx.x == 0 && threadIdx.y == 0) held = 0u;
  __syncthreads();
  auto cells = [](float d) { return d < 1e6f ? int(ceilf(d * 1.001f + 0.01f)) : 1 << 24; };   // also for a NaN
  const int rx = cells(U.der.x * __uint_as_float(__ldg(F.vmax))), ry = cells(U.der.x * __uint_as_float(__ldg(F.vmax + 1)));
  const int rz = cells(U.der.y * (__uint_as_float(__ldg(F.vmax + 2)) + F.fallmax));
  const int x = blockIdx.x * 32, y = blockIdx.y * 4, z = blockIdx.z;
  return box_channels(g, F, Region{x - rx, x + 32 + rx, y - ry, y + 4 + ry, z - rz, z + 1 + rz}, flagsA, flagsB, held);
}
__global__ void __launch_bounds__(128) k_advq1_hur(Grid g, Uni U, Fields F) {
  constexpr int par = 0;
  const int ci = blockIdx.x * blockDim.x + threadIdx.x, cj = blockIdx.y * blockDim.y + threadIdx.y, ck = blockIdx.z;
  const int brick = blockIdx.x + F.nbx * (blockIdx.y + F.nby * blockIdx.z);
  const unsigned zeros = F.zeroQt[brick];   // read by every thread before the barriers, written after them
  const unsigned act = reach_channels(g, U, F, F.actQ0, nullptr);
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    F.actQt[brick] = act;
    F.zeroQt[brick] = kHydro & ~act;
  }
  if (ci >= g.nx || cj >= g.ny || ck >= g.nz) return;
  auto has = [&](int c) { return ((act >> c) & 1u) != 0u; };
  const unsigned o = 4u * unsigned(g.at(ci, cj, ck));
  const float kk[3] = {U.der.x, U.der.x, U.der.y};
  const float p[3] = {float(ci) + 0.5f, float(cj) + 0.5f, float(ck) + 0.5f};
  float v[3];
  cellVel(F, g, par, ci, cj, ck, v);
  float x, y, z;
  traceQH(U, F, g, par, kk, p, v, 0.f, 1.f, x, y, z);
  const Tap t0 = tapQ(g, x, y, z);
  sto(F.Qt[0], o, gatherQ(F.Q[0][0], t0));
  if (act) {
    const float rho = bsA(F.B, g.nz, ck).z;
    const bool thm = U.micro2.z > 0.5f;
    const Fall fl{U.step.z, thm, U.hur3.w > 0.5f && !thm};
    auto at = [&](float fall, int c) {
      traceQH(U, F, g, par, kk, p, v, fall, 1.f, x, y, z);
      sto(F.Qt[c], o, gatherQ(F.Q[0][c], tapQ(g, x, y, z)));
    };
    if (has(1)) sto(F.Qt[1], o, gatherQ(F.Q[0][1], t0));
    if (has(7)) sto(F.Qt[7], o, gatherQ(F.Q[0][7], t0));
    if (has(6) && !thm) sto(F.Qt[6], o, gatherQ(F.Q[0][6], t0));
    if (has(2)) {
      const float fi = vtI(U, ldo(F.Q[0][2], o), rho);
      if (fi > 0.f) at(fi, 2);
      else sto(F.Qt[2], o, gatherQ(F.Q[0][2], t0));
    }
    if (has(3) || (has(6) && thm)) {
      const float2 fv = fl.vtRain(ldo(F.Q[0][3], o), ldo(F.Q[0][6], o), rho);
      if (has(3)) at(fv.x, 3);
      if (has(6) && thm) at(fv.y, 6);
    }
    if (has(4)) at(fl.vtS(ldo(F.Q[0][4], o), rho), 4);
    if (has(5)) at(fl.vtGrau(ldo(F.Q[0][5], o), rho), 5);
  }
  const unsigned clear = kHydro & ~act & ~zeros;
  if (clear) {
#pragma unroll
    for (int c = 1; c < 8; c++)
      if ((clear >> c) & 1u) sto(F.Qt[c], o, 0.f);
  }
}
__global__ void __launch_bounds__(128) k_advq2_hur(Grid g, Uni U, Fields F) {
  constexpr int par = 0;
  const int ci = blockIdx.x * blockDim.x + threadIdx.x, cj = blockIdx.y * blockDim.y + threadIdx.y, ck = blockIdx.z;
  const int brick = blockIdx.x + F.nbx * (blockIdx.y + F.nby * blockIdx.z);
  const unsigned zeros = F.zeroQ1[brick];
  const unsigned act = reach_channels(g, U, F, F.actQ0, F.actQt);
  if (threadIdx.x == 0 && threadIdx.y == 0) F.zeroQ1[brick] = kHydro & ~act;
  if (ci >= g.nx || cj >= g.ny || ck >= g.nz) return;
  auto has = [&](int c) { return ((act >> c) & 1u) != 0u; };
  const unsigned o = 4u * unsigned(g.at(ci, cj, ck));
  const float kk[3] = {U.der.x, U.der.x, U.der.y};
  const float p[3] = {float(ci) + 0.5f, float(cj) + 0.5f, float(ck) + 0.5f};
  float v[3];
  cellVel(F, g, par, ci, cj, ck, v);
  const float cx = v[0] * kk[0], cy = v[1] * kk[1], cz = v[2] * kk[2];
  const float cour = sqrtf(cx * cx + cy * cy + cz * cz);
  const float sm = 0.5f * U.misc.y * clampf(cour / 0.35f, U.dzv.w, 1.f);
  // channel c from its forward tap in the scratch, limited by the window of its departure tap
  auto put = [&](int c, const Tap& tb, const Tap& tf) {
    const float b = gatherQ(F.Qt[c], tb);
    const float r = ldo(F.Qt[c], o) + sm * (ldo(F.Q[0][c], o) - b);
    const float2 m = minmaxQ(F.Q[0][c], tf);
    sto(F.Q[1][c], o, fmaxf(clampf(r, m.x, m.y), 0.f));
  };
  float x, y, z;
  auto tap = [&](float fall, float s) {
    traceQH(U, F, g, par, kk, p, v, fall, s, x, y, z);
    return tapQ(g, x, y, z);
  };
  const bool thm = U.micro2.z > 0.5f;
  const float rho = bsA(F.B, g.nz, ck).z;
  const float fi = has(2) ? vtI(U, ldo(F.Q[0][2], o), rho) : 0.f;
  {  // at the air's speed
    const Tap tb = tap(0.f, -1.f), tf = tap(0.f, 1.f);
    put(0, tb, tf);
    if (has(1)) put(1, tb, tf);
    if (has(2) && fi == 0.f) put(2, tb, tf);
    if (has(6) && !thm) put(6, tb, tf);
    if (has(7)) put(7, tb, tf);
  }
  if (act & 0x7cu) {
    const Fall fl{U.step.z, thm, U.hur3.w > 0.5f && !thm};
    auto falling = [&](int c, float fall) {
      const Tap tb = tap(fall, -1.f), tf = tap(fall, 1.f);
      put(c, tb, tf);
    };
    if (has(2) && fi != 0.f) falling(2, fi);
    if (has(3) || (has(6) && thm)) {
      const float2 fv = fl.vtRain(ldo(F.Q[0][3], o), ldo(F.Q[0][6], o), rho);
      if (has(3)) falling(3, fv.x);
      if (has(6) && thm) falling(6, fv.y);
    }
    if (has(4)) falling(4, fl.vtS(ldo(F.Q[0][4], o), rho));
    if (has(5)) falling(5, fl.vtGrau(ldo(F.Q[0][5], o), rho));
  }
  const unsigned clear = kHydro & ~act & ~zeros;
  if (clear) {
#pragma unroll
    for (int c = 1; c < 8; c++)
      if ((clear >> c) & 1u) sto(F.Q[1][c], o, 0.f);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------------------------------------------
static inline dim3 grid3(int X, int Y, int Z, dim3 b) { return dim3((X + b.x - 1) / b.x, (Y + b.y - 1) / b.y, Z); }
static const dim3 kB3(32, 4, 1);
// the fields with the wind slot of this parity first: a kernel over one model always reads V[0] and writes V[1] (or the
// other way round), so that its field pointers are launch constants and not picked by an index
static Fields facing(Fields F, int par) {
  if (par)
    for (int c = 0; c < 4; c++) std::swap(F.V[0][c], F.V[1][c]);
  return F;
}
static const dim3 kB2(32, 8, 1);
// A pass whose inputs come from the pass just before it on its stream is launched under that one's tail where a step's
// launches count: with the rain pass and the LSF and CI maps off the main stream, a pass of steps and maps takes 777 -> 734 us at
// 64 x 64 x 40 and 2310 -> 2248 us at 203 x 157 x 40; at 320 x 320 x 56 (5.7e6 cells) there is nothing in it either way.
static bool launches_count(const Grid& g) { return long(g.nx) * g.ny * g.nz <= 1l << 21; }

void launch_lsf(const Grid& g, const Uni& U, const Fields& F, cudaStream_t s) {
  k_lsf<<<grid3(g.nx, g.ny, 1, kB2), kB2, 0, s>>>(g, U, F);
}
void launch_ci(const Grid& g, const Uni& U, const Fields& F, cudaStream_t s) {
  k_ci<<<grid3(g.nx, g.ny, 1, kB2), kB2, 0, s>>>(g, U, F);
}
void launch_init(const Grid& g, const Uni& U, const Fields& F, cudaStream_t s) {
  k_init<<<grid3(g.nx + 1, g.ny + 1, g.nz + 1, kB3), kB3, 0, s>>>(g, U, F);
}
void launch_nut(const Grid& g, const Uni& U, const Fields& F, int par, cudaStream_t s) {
  if (U.hur.x > 0.5f) k_nut_hur<<<grid3(g.nx, g.ny, g.nz, kB3), kB3, 0, s>>>(g, U, facing(F, par));
  else k_nut<<<grid3(g.nx, g.ny, g.nz, kB3), kB3, 0, s>>>(g, U, facing(F, par));
}
void launch_advv(const Grid& g, const Uni& U, const Fields& F, int par, cudaStream_t s) {
  if (U.hur.x > 0.5f && F.Vp[0]) {
    k_advv1_hur<<<grid3(g.nx + 1, g.ny + 1, g.nz + 1, kB3), kB3, 0, s>>>(g, U, facing(F, par));
    k_advv2_hur<<<grid3(g.nx + 1, g.ny + 1, g.nz + 1, kB3), kB3, 0, s>>>(g, U, facing(F, par));
    return;
  }
  k_advv1<<<grid3(g.nx + 1, g.ny + 1, g.nz + 1, kB3), kB3, 0, s>>>(g, U, facing(F, par));
  tc::launch_early(launches_count(g), k_advv2, grid3(g.nx + 1, g.ny + 1, g.nz + 1, kB3), kB3, 0, s, g, U, facing(F, par));
}
void launch_advq(const Grid& g, const Uni& U, const Fields& F, int par, cudaStream_t s) {
  if (U.hur.x > 0.5f) {
    k_advq1_hur<<<grid3(g.nx, g.ny, g.nz, kB3), kB3, 0, s>>>(g, U, facing(F, par));
    k_advq2_hur<<<grid3(g.nx, g.ny, g.nz, kB3), kB3, 0, s>>>(g, U, facing(F, par));
    return;
  }
  k_advq1<<<grid3(g.nx, g.ny, g.nz, kB3), kB3, 0, s>>>(g, U, facing(F, par));
  tc::launch_early(launches_count(g), k_advq2, grid3(g.nx, g.ny, g.nz, kB3), kB3, 0, s, g, U, facing(F, par));
}
void launch_prep(const Grid& g, const Uni& U, const Fields& F, int par, cudaStream_t s) {
  k_prep<<<grid3(g.nx + 1, g.ny + 1, g.nz + 1, kB3), kB3, 0, s>>>(g, U, facing(F, par));
  cudaMemsetAsync(F.vmax, 0, 3 * sizeof(unsigned), s);
  k_wind_max<<<592, 256, 0, s>>>(g, facing(F, par));
}
void launch_filt(const Grid& g, const Uni& U, const Fields& F, int par, cudaStream_t s) {
  k_filt<<<grid3(g.nx + 1, g.ny + 1, g.nz + 1, kB3), kB3, 0, s>>>(g, U, facing(F, par));
}
void launch_activity(const Grid& g, const Fields& F, cudaStream_t s) {
  k_activity<<<grid3(g.nx, g.ny, g.nz, kB3), kB3, 0, s>>>(g, F);
}
void launch_tables(const Grid& g, const Uni& U, const Fields& F, cudaStream_t s) {
  const int n = std::max(g.nz, std::max(g.nx, g.ny)) + 1;
  k_tables<<<(n + 127) / 128, 128, 0, s>>>(g, U, F.B, const_cast<float*>(F.spz), const_cast<float*>(F.slx), const_cast<float*>(F.sly));
}
void launch_phys(const Grid& g, const Uni& U, const Fields& F, int par, cudaStream_t s, int micro_mode) {
  if (U.hur.x > 0.5f) {  // hurricane mode runs the scheme (model.js:578-907 with its hurricane branches)
    if (U.cor.z > 0.5f) k_phys_hur<1><<<grid3(g.nx + 1, g.ny + 1, g.nz + 1, kB3), kB3, 0, s>>>(g, U, facing(F, par));
    else k_phys_hur<0><<<grid3(g.nx + 1, g.ny + 1, g.nz + 1, kB3), kB3, 0, s>>>(g, U, facing(F, par));
    return;
  }
  const dim3 grid = grid3(g.nx + 1, g.ny + 1, g.nz + 1, kB3);
  const bool bnd = U.cor.z > 0.5f;
  if (micro_mode == kMicroRecord) {
    if (bnd) k_phys<kMicroRecord, 1><<<grid, kB3, 0, s>>>(g, U, facing(F, par));
    else k_phys<kMicroRecord, 0><<<grid, kB3, 0, s>>>(g, U, facing(F, par));
  } else if (micro_mode == kMicroSurrogate) {
    if (bnd) k_phys<kMicroSurrogate, 1><<<grid, kB3, 0, s>>>(g, U, facing(F, par));
    else k_phys<kMicroSurrogate, 0><<<grid, kB3, 0, s>>>(g, U, facing(F, par));
  } else {
    if (bnd) k_phys<kMicroPlain, 1><<<grid, kB3, 0, s>>>(g, U, facing(F, par));
    else k_phys<kMicroPlain, 0><<<grid, kB3, 0, s>>>(g, U, facing(F, par));
  }
}
void launch_div(const Grid& g, const Uni& U, const Fields& F, int par, cudaStream_t s) {
  tc::launch_early(launches_count(g), k_div, grid3(g.nx, g.ny, g.nz, kB3), kB3, 0, s, g, U, facing(F, par));
}
void launch_proj(const Grid& g, const Uni& U, const Fields& F, int par, cudaStream_t s) {
  tc::launch_early(launches_count(g), k_proj, grid3(g.nx + 1, g.ny + 1, g.nz + 1, kB3), kB3, 0, s, g, U, facing(F, par));
}
void launch_rain(const Grid& g, const Uni& U, const Fields& F, cudaStream_t s) {
  k_rain<<<grid3(g.nx, g.ny, 1, kB2), kB2, 0, s>>>(g, U, F);
}
void launch_maps(const Grid& g, const Uni& U, const Fields& F, int par, float4* out, cudaStream_t s) {
  // two from where the row blocks of 32 columns number 2560 (260 x 260: 2340, 320 x 320: 3200). Four would gain 2 us at 203 x
  // 157 and 260 x 260 with the fields in L2, but lose 4 at 256 x 224 x 40 without (47 -> 51 us)
  const unsigned rows = unsigned(F.nbx) * unsigned(g.ny);
  const auto launch = [&](auto k, int w) {
    const int r = kMapWarps / w;
    k<<<unsigned(F.nbx) * unsigned((g.ny + r - 1) / r), dim3(32, kMapWarps), 0, s>>>(g, U, facing(F, par), out);
  };
  if (rows <= 2560) launch(k_maps<8>, 8);
  else launch(k_maps<2>, 2);
}

// ---------------------------------------------------------------------------------------------------------------
// tornado candidates of the sub-grid tornado scheme (tornadoCandidates, app.js:1457-1472) on the device maps: on the
// stride-2 lattice 6 cells inside the edges, a point whose 1-km vorticity (map0.w) is at least zmin and whose
// low-level theta' (map0.z) is not below -4.5 K, that has the largest vorticity of its stride-2 5 x 5 window, with a
// window maximum of 2-5 km updraft helicity (map1.y) above 60 m2/s2 and of updraft (map1.x) above 12 m/s. Appends
// (i, j, x, y, zeta, uh, w) per candidate; the host restores the lattice order (j, then i).
// ---------------------------------------------------------------------------------------------------------------
__global__ void k_tor_candidates(const float4* __restrict__ maps, int nx, int ny, float dx, float zmin, float* out, int cap,
                                 unsigned* count) {
  const int i = 6 + 2 * (blockIdx.x * blockDim.x + threadIdx.x), j = 6 + 2 * (blockIdx.y * blockDim.y + threadIdx.y);
  if (i >= nx - 6 || j >= ny - 6) return;
  const float4* m0 = maps;
  const float4* m1 = maps + size_t(nx) * ny;
  const float4 c = __ldg(m0 + j * nx + i);
  const float z1 = c.w;
  if (z1 < zmin || c.z < -4.5f) return;
  bool is_max = true;
  float uh = 0.f, w = 0.f;
  for (int dj = -4; dj <= 4; dj += 2)
    for (int di = -4; di <= 4; di += 2) {
      const int q = (i + di) + nx * (j + dj);
      if ((di || dj) && __ldg(m0 + q).w > z1) is_max = false;
      const float4 b = __ldg(m1 + q);
      uh = fmaxf(uh, b.y);
      w = fmaxf(w, b.x);
    }
  if (!(is_max && uh > 60.f && w > 12.f)) return;
  const unsigned slot = atomicAdd(count, 1u);
  if (slot >= unsigned(cap)) return;
  float* o = out + size_t(slot) * 7;
  o[0] = float(i); o[1] = float(j); o[2] = (float(i) + 0.5f) * dx; o[3] = (float(j) + 0.5f) * dx; o[4] = z1; o[5] = uh; o[6] = w;
}
// ---------------------------------------------------------------------------------------------------------------
// grouped launches (ensemble steps)
// ---------------------------------------------------------------------------------------------------------------
int group_kind(int pass) {
  switch (pass) {
    case kGroupLSF: case kGroupCI: case kGroupRAIN: return kGroup2D;
    case kGroupNUT: case kGroupADVQ1: case kGroupADVQ2: case kGroupDIV: return kGroupCell;
    default: return kGroupStag;
  }
}

dim3 group_default_block(int pass) { return group_kind(pass) == kGroup2D ? kB2 : kB3; }

bool group_block_fixed(int pass) {
  // the scalar advection and the physics pass share the 32 x 4 bricks of the clear-air flags; the 2-D passes are
  // not worth tuning
  return pass == kGroupADVQ1 || pass == kGroupADVQ2 || pass == kGroupPHYS || group_kind(pass) == kGroup2D;
}

int group_map(const Grid* grids, const int* pos, int n, int pass, dim3 block, std::vector<uint2>& map) {
  if (n < 1 || n > kMaxMembers) return -1;
  const int kind = group_kind(pass);
  map.clear();
  int Z = -1;
  for (int i = 0; i < n; i++) {
    const Grid& g = grids[i];
    int X = g.nx, Y = g.ny, z = g.nz;
    if (kind == kGroupStag) { X++; Y++; z++; }
    if (kind == kGroup2D) z = 1;
    if (Z >= 0 && z != Z) return -1;  // the members share nz
    Z = z;
    const int gx = (X + block.x - 1) / block.x, gy = (Y + block.y - 1) / block.y;
    if (gx > 65535 || gy > 65535) return -1;
    for (int by = 0; by < gy; by++)
      for (int bx = 0; bx < gx; bx++) map.push_back(make_uint2(unsigned(pos[i]), unsigned(bx) | (unsigned(by) << 16)));
  }
  return Z;
}

int group_upload_members(const MemberC* d_src, int n, cudaStream_t s) {
  if (n < 1 || n > kMaxMembers) return -1;
  return cudaMemcpyToSymbolAsync(c_members, d_src, sizeof(MemberC) * n, 0, cudaMemcpyDeviceToDevice, s) == cudaSuccess ? 0 : -1;
}

void launch_group(int pass, const uint2* map, int nxy, int Z, dim3 block, int par, cudaStream_t s, int micro_mode) {
  if (nxy < 1 || Z < 1) return;
  const dim3 grid(nxy, 1, Z);
  switch (pass) {
    case kGroupLSF: k_lsf_grp<<<grid, block, 0, s>>>(map, par); break;
    case kGroupCI: k_ci_grp<<<grid, block, 0, s>>>(map, par); break;
    case kGroupNUT: k_nut_grp<<<grid, block, 0, s>>>(map, par); break;
    case kGroupADVV1: k_advv1_grp<<<grid, block, 0, s>>>(map, par); break;
    case kGroupADVV2: k_advv2_grp<<<grid, block, 0, s>>>(map, par); break;
    case kGroupADVQ1: k_advq1_grp<<<grid, block, 0, s>>>(map, par); break;
    case kGroupADVQ2: k_advq2_grp<<<grid, block, 0, s>>>(map, par); break;
    case kGroupPHYS:
      if (micro_mode == kMicroRecord) k_phys_grp<kMicroRecord><<<grid, block, 0, s>>>(map, par);
      else if (micro_mode == kMicroSurrogate) k_phys_grp<kMicroSurrogate><<<grid, block, 0, s>>>(map, par);
      else k_phys_grp<kMicroPlain><<<grid, block, 0, s>>>(map, par);
      break;
    case kGroupDIV: k_div_grp<<<grid, block, 0, s>>>(map, par); break;
    case kGroupPROJ: k_proj_grp<<<grid, block, 0, s>>>(map, par); break;
    case kGroupRAIN: k_rain_grp<<<grid, block, 0, s>>>(map, par); break;
    default: break;
  }
}

void launch_tor_candidates(const Grid& g, float dx, const float4* maps, float zmin, float* out, int cap, unsigned* count, cudaStream_t s) {
  const int ni = (g.nx - 12 + 1) / 2, nj = (g.ny - 12 + 1) / 2;
  if (ni <= 0 || nj <= 0) return;
  k_tor_candidates<<<dim3((ni + 31) / 32, (nj + 7) / 8), dim3(32, 8), 0, s>>>(maps, g.nx, g.ny, dx, zmin, out, cap, count);
}
void launch_pack(const Grid& g, const Ptr8& src, int nch, int X, int Y, int Z, float* dst, cudaStream_t s) {
  k_pack<<<grid3(X, Y, Z, kB3), kB3, 0, s>>>(g, src, nch, X, Y, Z, dst);
}
void launch_unpack(const Grid& g, const Ptr8& dst, int nch, int X, int Y, int Z, const float* src, cudaStream_t s) {
  k_unpack<<<grid3(X, Y, Z, kB3), kB3, 0, s>>>(g, dst, nch, X, Y, Z, src);
}

}  // namespace ob
