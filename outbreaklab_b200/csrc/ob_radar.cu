// ob_radar.cu — virtual WSR-88D gate sampling for sm_100a (radar.js:41-268).
//
// k_radar_scan and k_radar_cut restate WGSL_R_CUT: one thread per gate (the reference packs 4 gates per thread), gates
// of one radial along x so that neighbouring lanes sample neighbouring points of the model (250 m apart) and share L1
// lines. Each gate samples the model three times across the beam (beam filling), turns the hydrometeors into
// reflectivity, radial velocity, spectrum width, ZDR, rho_hv and KDP, and stores one 8-bit Level II code per moment. The
// codes go out as bytes: a warp stores 32 consecutive codes of a radial, which is the reference's little-endian packing
// of 4 codes per u32 word (radar.js:229-240) written as one 32-byte sector.
//
// k_radar_phi restates WGSL_R_PHI: PhiDP is a running fp32 sum of 2 * KDP * dr along each radial, in gate order, so
// each radial stays sequential (a parallel scan would round differently).
//
// The quantisation code() and the PhiDP accumulation use explicitly rounded fp32 operations (no FMA contraction),
// so identical moments give bit-identical codes to the CPU restatement; the geometry and microphysics use CUDA's
// IEEE-accurate math functions and may contract to FMA.
#include <cmath>
#include <cstdint>

#include "ob_common.cuh"
#include "ob_radar.cuh"

namespace ob {

namespace {

struct Smp {
  float zr, zs, zg, vt, u, v, w, T, rho, nu, lr;
  bool inside;
};

__device__ __forceinline__ float db2lin(float d) { return powf(10.f, 0.1f * d); }
__device__ __forceinline__ float sqf(float x) { return x * x; }

// WGSL code(): u32(clamp(round(v * sc + ofs), 2, 255)), round half-to-even
__device__ __forceinline__ uint32_t lcode(float v, float sc, float ofs) {
  const float t = rintf(__fadd_rn(__fmul_rn(v, sc), ofs));
  return uint32_t(fminf(fmaxf(t, 2.f), 255.f));
}

// great-circle destination (bearing a rad, ground distance s m) -> model metres (radar.js:51-64)
__device__ __forceinline__ float2 gatePos(const RadarU& R, float a, float s) {
  const float RE = 6371000.f;
  const float p1 = R.geo.z, l1 = R.geo.w, d = s / RE;
  const float sp2 = sinf(p1) * cosf(d) + cosf(p1) * sinf(d) * cosf(a);
  const float p2 = asinf(clampf(sp2, -1.f, 1.f));
  const float l2 = l1 + atan2f(sinf(a) * sinf(d) * cosf(p1), cosf(d) - sinf(p1) * sp2);
  const float p0 = R.geo.x, dl = l2 - R.geo.y;
  const float cc = clampf(sinf(p0) * sinf(p2) + cosf(p0) * cosf(p2) * cosf(dl), -1.f, 1.f);
  const float c = acosf(cc);
  const float k = c < 1e-6f ? 1.f : c / sinf(c);
  return make_float2(RE * k * cosf(p2) * sinf(dl) - R.mdl2.z, RE * k * (cosf(p0) * sinf(p2) - sinf(p0) * cosf(p2) * cosf(dl)) - R.mdl2.w);
}
// 4/3-earth beam: (height above the antenna, ground distance) at slant range r (radar.js:66-72)
__device__ __forceinline__ float2 beam(const RadarU& R, float r, float el) {
  const float a = R.site.w;
  const float q = r * r + 2.f * r * a * sinf(el);
  const float h = q / (sqrtf(q + a * a) + a);
  return make_float2(h, a * asinf(clampf(r * cosf(el) / (a + h), -1.f, 1.f)));
}

// radar.js:89-139; full = false skips what the outer samples of the beam never use (w, fall speed, nu)
template <bool FULL>
__device__ __forceinline__ Smp sample(const RadarU& R, const Grid& g, const Fields& F, int par, float px, float py, float z) {
  Smp o;
  const float n0 = R.mdl.x, n1 = R.mdl.y, n2 = R.mdl.z, dx = R.mdl.w, dz = R.mdl2.x;
  const float gx = px / dx, gy = py / dx, gz = z / dz;
  o.inside = gx >= 0.f && gy >= 0.f && gz >= 0.f && gx <= n0 && gy <= n1 && gz <= n2 && z >= 0.f;
  const float cx = clampf(gx, 0.f, n0), cy = clampf(gy, 0.f, n1), cz = clampf(gz, 0.f, n2);
  const float qx = cx - 0.5f, qy = cy - 0.5f, qz = cz - 0.5f;
  const bool thm = R.phys.z > 0.5f;
  const float qr = fmaxf(trilerp(F.Q[0][3], g, g.nx, g.ny, g.nz, qx, qy, qz), 0.f);
  const float qs = fmaxf(trilerp(F.Q[0][4], g, g.nx, g.ny, g.nz, qx, qy, qz), 0.f);
  const float qg = fmaxf(trilerp(F.Q[0][5], g, g.nx, g.ny, g.nz, qx, qy, qz), 0.f);
  const int X = g.nx + 1, Y = g.ny + 1, Z = g.nz + 1;
  o.u = trilerp(F.V[par][0], g, X, Y, Z, cx, cy - 0.5f, cz - 0.5f);
  o.v = trilerp(F.V[par][1], g, X, Y, Z, cx - 0.5f, cy, cz - 0.5f);
  o.w = FULL ? trilerp(F.V[par][2], g, X, Y, Z, cx - 0.5f, cy - 0.5f, cz) : 0.f;
  const float th = trilerp(F.V[par][3], g, X, Y, Z, qx, qy, qz);
  const int k = int(clampf(floorf(cz), 0.f, n2 - 1.f));
  const float4 A = bsA(F.B, g.nz, k), B = bsB(F.B, g.nz, k);
  const float rho = A.z, T = th * B.x;
  o.zr = 3.63e9f * powf(rho * qr, 1.75f);
  o.zs = 9.80e8f * powf(rho * qs, 1.75f) * 0.224f * 4.0f;
  o.zg = (T < 273.15f ? 1.2e10f : 4.33e10f) * powf(rho * qg, 1.75f);
  const float sq = sqrtf(R.phys.x / rho);
  float vr = 0.f, vs = 0.f, vg = 0.f;
  if (FULL) {
    vr = fminf(36.34f * powf(fmaxf(0.001f * rho * qr, 0.f), 0.1364f) * sq, 10.f * sq);
    vs = clampf(1.1f * powf(fmaxf(1000.f * rho * qs, 1e-6f), 0.11f), 0.3f, 2.2f) * sq;
    vg = clampf(9.f * powf(fmaxf(1000.f * rho * qg, 1e-6f), 0.42f), 1.f, 55.f) * sq;
    const float rr = qg / 0.009f;
    vg = fminf(vg * (1.f + rr * rr), 65.f);
  }
  // hurricane mode's maritime graupel (radar.js:113)
  if (R.phys2.x > 0.5f && !thm) {
    o.zg = (T < 273.15f ? 1.3e9f : 1.0e10f) * powf(rho * qg, 1.75f);
    if (FULL) vg = clampf(5.f * powf(fmaxf(1000.f * rho * qg, 1e-6f), 0.25f), 1.f, 9.f) * sq;
  }
  o.lr = FULL ? powf(float(3.14159 * 1000.0 * 8e6) / fmaxf(rho * qr, 1e-9f), 0.25f) : 0.f;
  if (thm) {
    const float nr = fmaxf(trilerp(F.Q[0][6], g, g.nx, g.ny, g.nz, qx, qy, qz), 0.f);
    if (qr > 1e-9f) {
      const float l = clampf(powf(float(3.14159 * 1000.0) * fmaxf(nr, 1e-3f) / qr, 0.33333f), 1000.f, 1.0e5f);
      const float nb = qr * l * l * l / 3141.59f;
      o.zr = 720e18f * rho * nb / powf(l, 6.f);
      if (FULL) {
        o.lr = l;
        vr = fminf(3949.f * powf(l, -0.8f), 10.f) * sq;
      }
    } else {
      o.zr = 0.f;
    }
    if (qg > 1e-9f) {
      const float n0g = clampf(200.f / (rho * qg), 1e4f, 3e6f);
      const float l = powf(float(3.14159 * 500.0) * n0g / (rho * qg), 0.25f);
      o.zg = 720e18f * n0g / powf(l, 7.f) * (T < 273.15f ? 0.0666f : 0.24f);
      if (FULL) vg = fminf(2483.f * powf(l, -0.89f), 30.f) * sq;
    } else {
      o.zg = 0.f;
    }
  }
  const float zt = o.zr + o.zs + o.zg;
  o.vt = (FULL && zt > 1e-6f) ? (o.zr * vr + o.zs * vs + o.zg * vg) / zt : 0.f;
  o.T = T;
  o.rho = rho;
  o.nu = FULL ? trilerp(F.aux[0], g, g.nx, g.ny, g.nz, qx, qy, qz) : 0.f;
  return o;
}

struct GateOut {
  uint32_t c[5];  // REF, VEL, SW, ZDR, RHO codes (0 = empty)
  float kdp;      // -1 = empty
  float m[6];     // moments (dBZ, Vr, SW, ZDR, rho_hv, KDP), NaN where empty
};

// radar.js:144-227
__device__ GateOut gate(const RadarU& R, const Grid& g, const Fields& F, int par, const float* __restrict__ tor, int ri, int gi) {
  GateOut G;
#pragma unroll
  for (int i = 0; i < 5; i++) G.c[i] = 0u;
  G.kdp = -1.f;
#pragma unroll
  for (int i = 0; i < 6; i++) G.m[i] = __int_as_float(0x7fc00000);
  const float r = R.gates.z + R.gates.w * float(gi);
  const float el = R.cut.x;
  const float az = (R.cut.y + R.cut.z * float(ri)) * 0.017453293f;
  const float bw = 0.0165f;
  const float2 hc = beam(R, r, el);
  const float2 p = gatePos(R, az, hc.y);
  const float2 p2 = gatePos(R, az, hc.y + 200.f);
  float ex = p2.x - p.x, ey = p2.y - p.y;
  const float en = sqrtf(ex * ex + ey * ey);
  ex /= en;
  ey /= en;
  const float zAnt = R.site.z - R.mdl2.y;
  const float zc = zAnt + hc.x;
  if (zc > R.mdl.z * R.mdl2.x - 200.f) return G;
  const float hl = beam(R, r, el - 0.4f * bw).x + zAnt, hu = beam(R, r, el + 0.4f * bw).x + zAnt;
  const Smp s0 = sample<true>(R, g, F, par, p.x, p.y, fmaxf(zc, 5.f));
  if (!s0.inside) return G;
  const Smp s1 = sample<false>(R, g, F, par, p.x, p.y, fmaxf(hl, 5.f));
  const Smp s2 = sample<false>(R, g, F, par, p.x, p.y, fmaxf(hu, 5.f));
  const float zr = 0.5f * s0.zr + 0.25f * (s1.zr + s2.zr), zs = 0.5f * s0.zs + 0.25f * (s1.zs + s2.zs);
  const float zg = 0.5f * s0.zg + 0.25f * (s1.zg + s2.zg);
  const float zmet = zr + zs + zg;
  // sub-grid tornadoes: beam-smeared Rankine vortex and lofted debris
  float zdeb = 0.f, dvx = 0.f, dvy = 0.f, swt = 0.f;
  const float bwm = 0.5f * r * bw;
  const int ntor = int(R.phys.w);
  for (int q = 0; q < ntor; q++) {
    const float4 A = __ldg(reinterpret_cast<const float4*>(tor) + 2 * q), B = __ldg(reinterpret_cast<const float4*>(tor) + 2 * q + 1);
    const float dxv = p.x - A.x, dyv = p.y - A.y;
    const float rt = sqrtf(dxv * dxv + dyv * dyv);
    const float Re = sqrtf(A.z * A.z + bwm * bwm + 125.f * 125.f);
    if (rt > 8.f * Re) continue;
    const float vmx = A.w * A.z / Re;
    const float vt = vmx * (rt < Re ? rt / Re : Re / fmaxf(rt, 1.f));
    const float ir = fmaxf(rt, 1.f);
    const float etx = -dyv / ir, ety = dxv / ir, erx = dxv / ir, ery = dyv / ir;
    const float fz = 1.f - sstep(1200.f, 3500.f, zc);
    dvx += (vt * etx - 0.25f * vt * erx) * fz;
    dvy += (vt * ety - 0.25f * vt * ery) * fz;
    swt = fmaxf(swt, vmx * 0.4f * expf(-rt * rt / (4.f * Re * Re)) * fz);
    if (B.z > 0.f && zc < B.x) {
      const float rd = fmaxf(1.4f * A.z, 150.f);
      zdeb += db2lin(B.y) * fminf(1.f, rd * rd / (Re * Re)) * expf(-rt * rt / (Re * Re)) * (1.f - sstep(0.55f * B.x, B.x, zc)) * B.z;
    }
  }
  const float ztot = zmet + zdeb;
  if (ztot <= 1e-6f) return G;
  const float dbz = 10.f * logf(ztot) / 2.302585f;
  if (dbz < R.phys.y) return G;
  G.m[0] = dbz;
  G.c[0] = lcode(dbz, 2.f, 66.f);
  if (gi >= int(R.gates.y)) return G;
  const float ce = cosf(el), se = sinf(el);
  const float vtf = s0.vt * zmet / ztot;
  float vr = ((s0.u + dvx) * ex + (s0.v + dvy) * ey) * ce + (s0.w - vtf) * se;
  const float nyq = R.nyq.x;
  vr = vr - 2.f * nyq * floorf((vr + nyq) / (2.f * nyq));
  G.m[1] = vr;
  G.c[1] = lcode(vr, 2.f, 129.f);
  const float vru = (s2.u * ex + s2.v * ey) * ce, vrl = (s1.u * ex + s1.v * ey) * ce;
  const float swv = sqrtf(1.f + sqf(clampf(2.5f * sqrtf(fmaxf(s0.nu, 0.f) / 1000.f), 0.f, 8.f)) + sqf((vru - vrl) / 2.5f) +
                          sqf(0.15f * s0.vt * se) + sqf(swt));
  G.m[2] = fminf(swv, 19.5f);
  G.c[2] = lcode(G.m[2], 2.f, 129.f);
  const float d0 = 3.67f / s0.lr * 1000.f;
  const bool melt = s0.T > 273.15f;
  const float zdrR = clampf(0.2f + 1.15f * (d0 - 0.5f), 0.1f, 4.8f);
  const float zdrS = melt ? 1.3f : 0.3f;
  const float zdrG = melt ? (zg > 3.2e5f ? 0.f : 0.7f) : 0.15f;
  const float zv = zr / db2lin(zdrR) + zs / db2lin(zdrS) + zg / db2lin(zdrG) + zdeb / db2lin(0.2f);
  const float zdr = 10.f * logf(fmaxf(ztot, 1e-9f) / fmaxf(zv, 1e-9f)) / 2.302585f;
  G.m[3] = clampf(zdr, -7.9f, 7.9f);
  G.c[3] = lcode(G.m[3], 16.f, 128.f);
  const float fr = zr / ztot, fs = zs / ztot, fg = zg / ztot, fd = zdeb / ztot;
  float cc = fr * (d0 > 2.5f ? 0.986f : 0.995f) + fs * (melt ? 0.93f : 0.985f) + fg * (melt ? (zg > 3.2e5f ? 0.90f : 0.94f) : 0.985f) +
             fd * 0.55f;
  cc -= 0.24f * fr * fg;
  G.m[4] = clampf(cc, 0.2f, 1.05f);
  G.c[4] = lcode(G.m[4], 300.f, -60.5f);
  G.kdp = powf(0.017f * powf(fmaxf(zr, 0.f), 0.714f) / 44.f, 1.2165f);
  G.m[5] = G.kdp;
  return G;
}

// What the scan of a cut needs of its trigonometry, worked out on the host in 64 bits: the sines of the elevation at the
// beam's three points, its cosine, and the site's up, north and east vectors in the frame (east, north, up) of the
// projection's centre. all: no gate may be left out, because the cut comes within 6 degrees of a pole, where gatePos takes its
// position from an arc sine near 1 and an arc tangent of two small numbers: their rounding moves it by about a metre over the
// cosine of the latitude, which is past the scan's margin within 2 degrees.
struct ScanU {
  float se, sl, su, ce;
  float3 up, north, east;
  bool all;
};
static ScanU scan_uniforms(const RadarU& R) {
  const double p0 = R.geo.x, p1 = R.geo.z, dl = double(R.geo.w) - double(R.geo.y), el = R.cut.x, q = 0.4 * 0.0165;
  auto f3 = [](double x, double y, double z) { return make_float3(float(x), float(y), float(z)); };
  ScanU S;
  S.se = float(std::sin(el));
  S.sl = float(std::sin(el - q));
  S.su = float(std::sin(el + q));
  S.ce = float(std::cos(el));
  S.up = f3(std::cos(p1) * std::sin(dl), std::cos(p0) * std::sin(p1) - std::sin(p0) * std::cos(p1) * std::cos(dl),
            std::sin(p0) * std::sin(p1) + std::cos(p0) * std::cos(p1) * std::cos(dl));
  S.north = f3(-std::sin(p1) * std::sin(dl), std::cos(p0) * std::cos(p1) + std::sin(p0) * std::sin(p1) * std::cos(dl),
               std::sin(p0) * std::cos(p1) - std::cos(p0) * std::sin(p1) * std::cos(dl));
  S.east = f3(std::cos(dl), std::sin(p0) * std::sin(dl), -std::cos(p0) * std::sin(dl));
  S.all = !(std::fabs(p1) + (double(R.gates.z) + double(R.gates.w) * double(R.gates.x)) / 6371000.0 <= 1.466);
  return S;
}
// Whether a gate can come out anything but empty: false only if gate() leaves it empty, whatever its last bits. The
// beam's three points are worked out with vectors and short series (the ground arc d < 0.2, the angle to the centre under
// 0.3: errors below 1e-8, so what is left is fp32 rounding, about a metre on either side), and every bound has a margin
// many times that (25 m in the horizontal, 1 m in the vertical); the texels looked at are all that any point within it
// interpolates. First the hydrometeor flags of the 32 x 4 bricks around (F.actQ0, as fresh as the state: the physics pass
// and every write of the scalars remake them), then the rain, snow and graupel themselves. Out of these alone each
// reflectivity is +0, and with no tornado about there is no debris, so the echo is below any floor.
__device__ __forceinline__ bool may_echo(const RadarU& R, const ScanU& S, const Grid& g, const Fields& F, int ri, int gi) {
  if (S.all) return true;
  const float r = R.gates.z + R.gates.w * float(gi);
  const float az = (R.cut.y + R.cut.z * float(ri)) * 0.017453293f;
  const float dx = R.mdl.w, dz = R.mdl2.x, zAnt = R.site.z - R.mdl2.y, a = R.site.w;
  auto height = [&](float sn) {
    const float q = r * r + 2.f * r * a * sn;
    return q / (sqrtf(q + a * a) + a);
  };
  const float h = height(S.se), zc = zAnt + h;
  if (zc > R.mdl.z * dz - 199.f) return false;
  const float s = a * asinf(clampf(r * S.ce / (a + h), -1.f, 1.f));
  constexpr float RE = 6371000.f;
  const float d = s / RE, d2 = d * d;
  const float sd = d * (1.f - d2 * (1.f / 6.f - d2 * (1.f / 120.f))), cd = 1.f - d2 * (0.5f - d2 * (1.f / 24.f - d2 * (1.f / 720.f)));
  float sa, ca;
  sincosf(az, &sa, &ca);
  const float ux = cd * S.up.x + sd * (ca * S.north.x + sa * S.east.x), uy = cd * S.up.y + sd * (ca * S.north.y + sa * S.east.y);
  const float uz = cd * S.up.z + sd * (ca * S.north.z + sa * S.east.z);
  const float t2 = ux * ux + uy * uy;   // sin^2 of the angle to the centre: angle / sine = asin(t) / t
  float2 p;
  if (d < 0.2f && t2 < 0.09f && uz > 0.f) {
    const float k = 1.f + t2 * (1.f / 6.f + t2 * (3.f / 40.f + t2 * (15.f / 336.f + t2 * (105.f / 3456.f + t2 * (945.f / 42240.f)))));
    p = make_float2(RE * k * ux - R.mdl2.z, RE * k * uy - R.mdl2.w);
  } else {
    p = gatePos(R, az, s);
  }
  const float ex = 25.f / dx + 0.01f, ez = 1.f / dz + 0.001f;
  const float gx = p.x / dx, gy = p.y / dx, gz = fmaxf(zc, 5.f) / dz;
  if (!(gx >= -ex && gy >= -ex && gz >= -ez && gx <= R.mdl.x + ex && gy <= R.mdl.y + ex && gz <= R.mdl.z + ez)) return false;
  if (int(R.phys.w) > 0) return true;
  const float hl = height(S.sl) + zAnt, hu = height(S.su) + zAnt;
  const float zl = fminf(fmaxf(hl, 5.f), fmaxf(zc, 5.f)) / dz, zu = fmaxf(fmaxf(hu, 5.f), fmaxf(zc, 5.f)) / dz;
  const int i0 = clampi(int(floorf(gx - 0.5f - ex)), 0, g.nx - 1), i1 = clampi(int(floorf(gx - 0.5f + ex)) + 1, 0, g.nx - 1);
  const int j0 = clampi(int(floorf(gy - 0.5f - ex)), 0, g.ny - 1), j1 = clampi(int(floorf(gy - 0.5f + ex)) + 1, 0, g.ny - 1);
  const int k0 = clampi(int(floorf(zl - 0.5f - ez)), 0, g.nz - 1), k1 = clampi(int(floorf(zu - 0.5f + ez)) + 1, 0, g.nz - 1);
  unsigned any = 0;
  for (int k = k0; k <= k1; k++)
    for (int by = j0 >> 2; by <= j1 >> 2; by++)
      for (int bx = i0 >> 5; bx <= i1 >> 5; bx++) any |= __ldg(F.actQ0 + bx + F.nbx * (by + F.nby * k));
  if (!any) return false;
  // the corners of a level at once: their 12 loads are in flight together (a middle row or column is rare)
  const bool wide = i1 - i0 > 1 || j1 - j0 > 1;
  for (int k = k0; k <= k1; k++) {
    const int a = g.at(i0, j0, k), b = g.at(i1, j0, k), c = g.at(i0, j1, k), d = g.at(i1, j1, k);
    unsigned bits = 0;
#pragma unroll
    for (int q = 3; q < 6; q++)
      bits |= __float_as_uint(__ldg(F.Q[0][q] + a)) | __float_as_uint(__ldg(F.Q[0][q] + b)) | __float_as_uint(__ldg(F.Q[0][q] + c)) |
              __float_as_uint(__ldg(F.Q[0][q] + d));
    if (wide)
      for (int j = j0; j <= j1; j++)
        for (int i = i0; i <= i1; i++)
#pragma unroll
          for (int q = 3; q < 6; q++) bits |= __float_as_uint(__ldg(F.Q[0][q] + g.at(i, j, k)));
    if (bits) return true;   // a zero of either sign adds nothing, but a -0 here only sends the gate on
  }
  return false;
}

// A cut in two launches. Most gates of a volume see no rain, snow or graupel in any of their three samples, so their
// codes are all 0. k_radar_scan tells these from the others (may_echo, in 32 registers and a third of the instructions)
// and writes them; the rest get kActive in place of their REF code, a code that no gate has (0 is empty, values start at
// 2), and k_radar_cut works out those. Both take one thread per gate, x = gate along the radial, y = radial. The scan is
// bound by its instructions (arithmetic of the position, issue slots 60-70 % busy), the rest by the latency of a warp's
// gathers and powers. VCP 212 over a 256 x 256 x 40 storm field (17 cuts of 936 gates a radial): 2051 us for one launch
// per cut over every gate, now 380 + 601 us; a texel test on gate()'s own trigonometry took 568 us. Codes are compared
// bit for bit, and the compiler's choice of fused multiply-adds moves with the code around them, so gate() and its launch
// stay whole: packing the active gates into full warps changed the last bit of some moments.
constexpr uint8_t kActive = 1;
__global__ void __launch_bounds__(128) k_radar_scan(RadarU R, ScanU S, Grid g, Fields F, uint8_t* __restrict__ out, float* __restrict__ kdp,
                                                    float* __restrict__ mom) {
  const int gi = blockIdx.x * blockDim.x + threadIdx.x, ri = blockIdx.y;
  const int ngR = int(R.gates.x), ngD = int(R.gates.y);
  if (gi >= ngR) return;
  const bool active = may_echo(R, S, g, F, ri, gi);
  const size_t oR = size_t(R.offA.x) * 4 + size_t(ri) * ngR + gi;
  out[oR] = active ? kActive : uint8_t(0);
  if (active) return;
  const uint32_t mask = uint32_t(R.offB.w);
  if (gi < ngD) {
    const size_t o = size_t(ri) * ngD + gi;
    if (mask & 2u) out[size_t(R.offA.y) * 4 + o] = 0;
    if (mask & 4u) out[size_t(R.offA.z) * 4 + o] = 0;
    if (mask & 8u) out[size_t(R.offA.w) * 4 + o] = 0;
    if (mask & 32u) out[size_t(R.offB.y) * 4 + o] = 0;
    kdp[o] = -1.f;
  }
  if (mom) {
    float* mp = mom + (size_t(ri) * ngR + gi) * 6;
#pragma unroll
    for (int c = 0; c < 6; c++) mp[c] = __int_as_float(0x7fc00000);
  }
}
__global__ void __launch_bounds__(128) k_radar_cut(RadarU R, Grid g, Fields F, int par, const float* __restrict__ tor,
                                                   uint8_t* __restrict__ out, float* __restrict__ kdp, float* __restrict__ mom) {
  const int gi = blockIdx.x * blockDim.x + threadIdx.x, ri = blockIdx.y;
  const int ngR = int(R.gates.x), ngD = int(R.gates.y);
  if (gi >= ngR) return;
  if (out[size_t(R.offA.x) * 4 + size_t(ri) * ngR + gi] != kActive) return;
  const GateOut G = gate(R, g, F, par, tor, ri, gi);
  const uint32_t mask = uint32_t(R.offB.w);
  out[size_t(R.offA.x) * 4 + size_t(ri) * ngR + gi] = uint8_t(G.c[0]);
  if (gi < ngD) {
    const size_t o = size_t(ri) * ngD + gi;
    if (mask & 2u) out[size_t(R.offA.y) * 4 + o] = uint8_t(G.c[1]);
    if (mask & 4u) out[size_t(R.offA.z) * 4 + o] = uint8_t(G.c[2]);
    if (mask & 8u) out[size_t(R.offA.w) * 4 + o] = uint8_t(G.c[3]);
    if (mask & 32u) out[size_t(R.offB.y) * 4 + o] = uint8_t(G.c[4]);
    kdp[o] = G.kdp;
  }
  if (mom) {
    float* mp = mom + (size_t(ri) * ngR + gi) * 6;
#pragma unroll
    for (int c = 0; c < 6; c++) mp[c] = G.m[c];
  }
}

// PhiDP (radar.js:243-268): one block per 32 radials. The sum along a radial is a chain of fp32 additions in gate order,
// so the only serial part is kept to just that: in turn i warp 0 (lane = radial) runs the additions of chunk i over
// increments that are already in shared memory, while the other warps turn the KDP of chunk i + 1 (fetched before they
// do anything else) into increments and the sums of chunk i - 1 into codes. What bounds it is the latency of the chain
// and of a turn's loads: 175 -> 18 us per cut of 720 radials x 936 gates against one warp doing all of it for 32
// radials.
constexpr int kPhiChunk = 96, kPhiWarps = 16, kPhiThreads = 32 * kPhiWarps;
constexpr int kPhiSpan = kPhiChunk / 32, kPhiRows = (32 + kPhiWarps - 2) / (kPhiWarps - 1);   // rows per helping warp
__global__ void __launch_bounds__(kPhiThreads) k_radar_phi(RadarU R, const float* __restrict__ kdp, uint8_t* __restrict__ out) {
  constexpr unsigned kEmpty = 0xffffffffu;   // an empty gate (no addition, code 0): a NaN that no sum produces
  __shared__ unsigned buf[3][32][kPhiChunk + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r0 = blockIdx.x * 32;
  const int nrad = int(R.cut.w), ng = int(R.gates.y), ngq = (ng / 4) * 4;
  const float gw = R.gates.w;
  uint8_t* dst = out + size_t(R.offB.x) * 4;
  const int nch = (ngq + kPhiChunk - 1) / kPhiChunk;
  float kd[kPhiRows][kPhiSpan];
  // rows warp - 1, warp - 1 + 15, ... of a chunk: its KDP, its increments, its codes
  auto fetch = [&](int c) {
#pragma unroll
    for (int j = 0; j < kPhiRows; j++)
#pragma unroll
      for (int u = 0; u < kPhiSpan; u++) {
        const int r = warp - 1 + j * (kPhiWarps - 1), gi = c * kPhiChunk + u * 32 + lane;
        kd[j][u] = (r < 32 && r0 + r < nrad && gi < ngq) ? __ldg(kdp + size_t(r0 + r) * ng + gi) : -1.f;
      }
  };
  auto increments = [&](int c) {
#pragma unroll
    for (int j = 0; j < kPhiRows; j++)
#pragma unroll
      for (int u = 0; u < kPhiSpan; u++) {
        const int r = warp - 1 + j * (kPhiWarps - 1);
        const float k = kd[j][u];
        if (r < 32) buf[c % 3][r][u * 32 + lane] = k >= 0.f ? __float_as_uint(__fmul_rn(__fmul_rn(__fmul_rn(2.f, k), gw), 0.001f)) : kEmpty;
      }
  };
  auto encode = [&](int c) {
#pragma unroll
    for (int j = 0; j < kPhiRows; j++)
#pragma unroll
      for (int u = 0; u < kPhiSpan; u++) {
        const int r = warp - 1 + j * (kPhiWarps - 1), gi = c * kPhiChunk + u * 32 + lane;
        if (r >= 32 || r0 + r >= nrad || gi >= ngq) continue;
        const unsigned b = buf[c % 3][r][u * 32 + lane];
        uint8_t code = 0;
        if (b != kEmpty) {
          const float acc = __uint_as_float(b);
          const float ph = __fsub_rn(acc, __fmul_rn(360.f, floorf(__fdiv_rn(acc, 360.f))));
          code = uint8_t(fminf(fmaxf(rintf(__fadd_rn(__fdiv_rn(__fmul_rn(ph, 253.f), 360.f), 2.f)), 2.f), 255.f));
        }
        dst[size_t(r0 + r) * ng + gi] = code;
      }
  };
  if (warp > 0) {
    fetch(0);
    increments(0);
  }
  __syncthreads();
  float acc = R.nyq.w;
  for (int i = 0; i <= nch; i++) {
    if (warp == 0) {
      if (i < nch) {
        unsigned* row = buf[i % 3][lane];
        for (int t0 = 0; t0 < kPhiChunk; t0 += 32) {
          unsigned b[32];
#pragma unroll
          for (int t = 0; t < 32; t++) b[t] = row[t0 + t];
#pragma unroll
          for (int t = 0; t < 32; t++) {
            const float next = __fadd_rn(acc, __uint_as_float(b[t]));
            const bool empty = b[t] == kEmpty;
            acc = empty ? acc : next;
            b[t] = empty ? kEmpty : __float_as_uint(acc);
          }
#pragma unroll
          for (int t = 0; t < 32; t++) row[t0 + t] = b[t];
        }
      }
    } else {
      if (i + 1 < nch) fetch(i + 1);
      if (i > 0) encode(i - 1);
      if (i + 1 < nch) increments(i + 1);
    }
    __syncthreads();
  }
}

}  // namespace

void launch_radar_cut(const RadarU& R, const Grid& g, const Fields& F, int par, const float* tor, uint8_t* out, float* kdp,
                      float* mom, cudaStream_t s) {
  const int ngR = int(R.gates.x), nrad = int(R.cut.w);
  k_radar_scan<<<dim3((ngR + 127) / 128, nrad), 128, 0, s>>>(R, scan_uniforms(R), g, F, out, kdp, mom);
  k_radar_cut<<<dim3((ngR + 127) / 128, nrad), 128, 0, s>>>(R, g, F, par, tor, out, kdp, mom);
  if (uint32_t(R.offB.w) & 16u) k_radar_phi<<<(nrad + 31) / 32, kPhiThreads, 0, s>>>(R, kdp, out);
}

}  // namespace ob
