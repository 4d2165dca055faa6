// Forward projection by exact per-cell summation ("fast" projector).
//
// The reference's ray marcher (ForwardProjectionRayMarcher_TL.cu:130-151,
// ForwardProjectionSlicer.cu:130-151) samples the trilinear interpolant at
// t_j = t_in + j*h', j = 0..J-1, and sums the samples. Within one cell of
// the interpolation lattice the interpolant is a trilinear polynomial of the
// cell-local coordinates, and these are linear in j. So the sum over the
// samples inside a cell has a closed form in the power sums of j. Rays of a
// single-axis series stay in one y plane and take the layer walk (axis_walk:
// one layer of the major axis per step, its samples as weights of two rows of
// voxels; plane_sums the same for a line of rays), rays whose y moves slowly
// a walk like it (tilted_sum);
// other rays walk the cells they cross with a 3-D DDA (cell_sum), loading
// each cell's 8 corners once (4 when it enters through a face shared with
// the previous cell). Either replaces ~5 trilinear evaluations (40 loads)
// per cell with 4-8 loads and a few dozen FLOPs.
//
// The sample positions are the reference's: t is the reference's float
// recurrence t += 0.15*voxelSize, whose step on the float grid of t ~ 1e4 is
// a constant h' inside one binade (a power-of-two interval) of t. Rays whose
// samples leave the binade of t_in, or whose step alternates (a rounding
// tie), fall back to sample-by-sample marching. Sample positions are exact
// affine functions of j here, where the reference rounds each position
// computation: the difference is a ~1e-3 voxel jitter of the sample
// positions (rel-L2 ~1e-5 on projections).
//
// One thread per sub-ray. The 4 sub-rays of a pixel sit in adjacent lanes and
// are combined with warp shuffles.
#include <algorithm>
#include <float.h>

#include "esb_axis.cuh"

namespace esb {

namespace {

using namespace raycore;

// Sum of the trilinear interpolant over samples j = j0 .. J-1 at coordinates
// q + j*dq, by exact cell-wise closed forms.
template <int VT>
__device__ float cell_sum(const Cell<VT>& C, float qx, float qy, float qz, float dqx, float dqy, float dqz, int j0,
                          int J) {
  if (j0 >= J) return 0.0f;
  // position of sample j0
  float px = qpos(qx, j0, dqx), py = qpos(qy, j0, dqy), pz = qpos(qz, j0, dqz);
  float fx = floorf(px), fy = floorf(py), fz = floorf(pz);
  int ix = (int)fx, iy = (int)fy, iz = (int)fz;
  // sample parameter s (in units of j, relative to j0) of the next boundary per axis
  const float inf = FLT_MAX;
  float isx = dqx != 0.f ? 1.0f / fabsf(dqx) : inf;
  float isy = dqy != 0.f ? 1.0f / fabsf(dqy) : inf;
  float isz = dqz != 0.f ? 1.0f / fabsf(dqz) : inf;
  float nxs = dqx > 0.f ? (fx + 1.f - px) * isx : (dqx < 0.f ? (px - fx) * isx : inf);
  float nys = dqy > 0.f ? (fy + 1.f - py) * isy : (dqy < 0.f ? (py - fy) * isy : inf);
  float nzs = dqz > 0.f ? (fz + 1.f - pz) * isz : (dqz < 0.f ? (pz - fz) * isz : inf);
  const int stx = dqx > 0.f ? 1 : -1, sty = dqy > 0.f ? 1 : -1, stz = dqz > 0.f ? 1 : -1;
  float c000 = C.at(ix, iy, iz), c100 = C.at(ix + 1, iy, iz), c010 = C.at(ix, iy + 1, iz),
        c110 = C.at(ix + 1, iy + 1, iz);
  float c001 = C.at(ix, iy, iz + 1), c101 = C.at(ix + 1, iy, iz + 1), c011 = C.at(ix, iy + 1, iz + 1),
        c111 = C.at(ix + 1, iy + 1, iz + 1);
  const int M_total = J - j0;
  int m0 = 0;  // samples consumed so far (relative to j0)
  float acc = 0.0f;
#pragma unroll 1
  for (int guard = 0; guard < 1 << 20; ++guard) {
    // exit of the current cell in s; samples m0 .. m1-1 lie in it
    float sexit = fminf(nxs, fminf(nys, nzs));
    int m1 = (sexit >= (float)M_total) ? M_total : (int)ceilf(sexit);
    if (m1 > M_total) m1 = M_total;
    if (m1 > m0) {
      // local coordinates of sample m0 and per-sample increments
      const float a0 = __fsub_rn(qpos(qx, j0 + m0, dqx), (float)ix);
      const float b0 = __fsub_rn(qpos(qy, j0 + m0, dqy), (float)iy);
      const float e0 = __fsub_rn(qpos(qz, j0 + m0, dqz), (float)iz);
      const float M = (float)(m1 - m0);
      const float S1 = 0.5f * M * (M - 1.f);
      const float S2 = S1 * (2.f * M - 1.f) * (1.f / 3.f);
      const float S3 = S1 * S1;
      const float k1 = c100 - c000, k2 = c010 - c000, k3 = c001 - c000;
      const float k4 = c110 - c100 - c010 + c000, k5 = c101 - c100 - c001 + c000, k6 = c011 - c010 - c001 + c000;
      const float k7 = c111 - c110 - c101 - c011 + c100 + c010 + c001 - c000;
      const float sa = M * a0 + S1 * dqx, sb = M * b0 + S1 * dqy, sc = M * e0 + S1 * dqz;
      const float sab = M * a0 * b0 + S1 * (a0 * dqy + b0 * dqx) + S2 * dqx * dqy;
      const float sac = M * a0 * e0 + S1 * (a0 * dqz + e0 * dqx) + S2 * dqx * dqz;
      const float sbc = M * b0 * e0 + S1 * (b0 * dqz + e0 * dqy) + S2 * dqy * dqz;
      const float sabc = M * a0 * b0 * e0 + S1 * (a0 * b0 * dqz + a0 * e0 * dqy + b0 * e0 * dqx) +
                         S2 * (a0 * dqy * dqz + b0 * dqx * dqz + e0 * dqx * dqy) + S3 * dqx * dqy * dqz;
      acc += c000 * M + k1 * sa + k2 * sb + k3 * sc + k4 * sab + k5 * sac + k6 * sbc + k7 * sabc;
      m0 = m1;
    }
    if (m0 >= M_total) break;
    // step into the next cell through the nearest face, reusing the 4 shared
    // corners; face crossings are recomputed from the fixed start point, so
    // they carry no accumulated rounding
    if (nxs <= nys && nxs <= nzs) {
      ix += stx;
      nxs = stx > 0 ? ((float)(ix + 1) - px) * isx : (px - (float)ix) * isx;
      if (stx > 0) {
        c000 = c100; c010 = c110; c001 = c101; c011 = c111;
        c100 = C.at(ix + 1, iy, iz); c110 = C.at(ix + 1, iy + 1, iz);
        c101 = C.at(ix + 1, iy, iz + 1); c111 = C.at(ix + 1, iy + 1, iz + 1);
      } else {
        c100 = c000; c110 = c010; c101 = c001; c111 = c011;
        c000 = C.at(ix, iy, iz); c010 = C.at(ix, iy + 1, iz);
        c001 = C.at(ix, iy, iz + 1); c011 = C.at(ix, iy + 1, iz + 1);
      }
    } else if (nys <= nzs) {
      iy += sty;
      nys = sty > 0 ? ((float)(iy + 1) - py) * isy : (py - (float)iy) * isy;
      if (sty > 0) {
        c000 = c010; c100 = c110; c001 = c011; c101 = c111;
        c010 = C.at(ix, iy + 1, iz); c110 = C.at(ix + 1, iy + 1, iz);
        c011 = C.at(ix, iy + 1, iz + 1); c111 = C.at(ix + 1, iy + 1, iz + 1);
      } else {
        c010 = c000; c110 = c100; c011 = c001; c111 = c101;
        c000 = C.at(ix, iy, iz); c100 = C.at(ix + 1, iy, iz);
        c001 = C.at(ix, iy, iz + 1); c101 = C.at(ix + 1, iy, iz + 1);
      }
    } else {
      iz += stz;
      nzs = stz > 0 ? ((float)(iz + 1) - pz) * isz : (pz - (float)iz) * isz;
      if (stz > 0) {
        c000 = c001; c100 = c101; c010 = c011; c110 = c111;
        c001 = C.at(ix, iy, iz + 1); c101 = C.at(ix + 1, iy, iz + 1);
        c011 = C.at(ix, iy + 1, iz + 1); c111 = C.at(ix + 1, iy + 1, iz + 1);
      } else {
        c001 = c000; c101 = c100; c011 = c010; c111 = c110;
        c000 = C.at(ix, iy, iz); c100 = C.at(ix + 1, iy, iz);
        c010 = C.at(ix, iy + 1, iz); c110 = C.at(ix + 1, iy + 1, iz);
      }
    }
  }
  return acc;
}

// cell_sum for a ray whose y coordinate stays in one interpolation cell with
// a constant weight b (single-axis tilt about y: n.y is 0 or ~1e-10): the
// trilinear interpolant is a bilinear one in (x, z) of the y-interpolated
// corners.
//
// The walk goes layer by layer along the major axis (z or x, the one with the
// larger per-sample step). A layer holds at most one crossing of the minor
// axis, so every step sums two cells, the second empty when the ray does not
// cross in that layer, and the loop has no data-dependent branches: lanes
// whose rays cross in different layers stay converged. Both axes are
// mirrored so that the walk advances in the + direction of each.
//
// A cell's M samples have local coordinates (a0 + m da, c0 + m dc); with
// their mean (a, c) and the bilinear f = e00 + k1 a + k3 c + k5 a c,
//   sum_m f = M [f(a, c) + k5 da dc (M^2 - 1) / 12].
// Samples are assigned to cells exactly as by the cell-by-cell DDA (the
// sample parameter of each face crossing, rounded up).
template <int VT, bool ZMAJ, class Off>
__device__ float layer_sum_xz(const Cell<VT>& C, float qx, float b, int iy, float qz, float dqx, float dqz, int j0,
                              int J) {
  if (j0 >= J) return 0.0f;
  // major axis m (layers), minor axis n
  const float qm = ZMAJ ? qz : qx, dqm = ZMAJ ? dqz : dqx;
  const float qn = ZMAJ ? qx : qz, dqn = ZMAJ ? dqx : dqz;
  const int sm = dqm < 0.f ? -1 : 1, sn = dqn < 0.f ? -1 : 1;
  const float Mq = sm > 0 ? qm : -qm, dM = fabsf(dqm);
  const float Nq = sn > 0 ? qn : -qn, dN = fabsf(dqn);
  const float fj0 = (float)j0;
  const float pM = __fmaf_rn(fj0, dM, Mq), pN = __fmaf_rn(fj0, dN, Nq);
  float fcm = floorf(pM), fcn = floorf(pN);
  const float inf = FLT_MAX;
  const float isM = 1.0f / dM;  // dM > 0: the ray moves in x-z, and the major step is the larger one
  const float isN = dN > 0.f ? 1.0f / dN : inf;
  float nMs = ((fcm + 1.f) - pM) * isM;
  float nNs = dN > 0.f ? ((fcn + 1.f) - pN) * isN : inf;
  const float g = dN * dM * (1.0f / 12.0f);
  const float jb = fj0 - 0.5f;
  // element offsets of type Off: 32-bit below 2^32 voxels (cheaper address
  // arithmetic), 64-bit above (the launchers choose)
  const Off SM = ZMAJ ? (Off)C.sz : (Off)1, SN = ZMAJ ? (Off)1 : (Off)C.sz;
  const int nMax = ZMAJ ? C.nz - 1 : C.nx - 1, nNax = ZMAJ ? C.nx - 1 : C.nz - 1;
  auto clampM = [&](int i) { return (Off)(i < 0 ? 0 : (i > nMax ? nMax : i)) * SM; };
  auto clampN = [&](int i) { return (Off)(i < 0 ? 0 : (i > nNax ? nNax : i)) * SN; };
  const Off y0 = (Off)(iy < 0 ? 0 : (iy > C.ny - 1 ? C.ny - 1 : iy)) * (Off)C.sy;
  const Off y1 = (Off)(iy + 1 < 0 ? 0 : (iy + 1 > C.ny - 1 ? C.ny - 1 : iy + 1)) * (Off)C.sy;
  const float ib = 1.0f - b;
  auto ey = [&](Off o) {
    return ib * Voxel<VT>::load(C.vol, (long)(o + y0)) + b * Voxel<VT>::load(C.vol, (long)(o + y1));
  };
  // original indices of the current cell's near and far corners per axis
  int inF = sn * (int)fcn + sn;
  int imF = sm * (int)fcm + sm;
  Off on = clampN(inF - sn), of = clampN(inF);
  Off omn = clampM(imF - sm), omf = clampM(imF);
  float enn = ey(on + omn), efn = ey(of + omn);
  const float Mt = (float)(J - j0);
  float fm0 = 0.0f, acc = 0.0f;
  // two layers per iteration give the scheduler independent loads; the
  // 64-bit-offset instances stay at one (registers)
  constexpr int kUnroll = sizeof(Off) == 4 ? 2 : 1;
#pragma unroll kUnroll
  for (int guard = 0; guard < 1 << 20; ++guard) {
    // samples [fm0, fmA) lie in cell (n, m), [fmA, fmL) in cell (n + 1, m)
    const float fmL = nMs >= Mt ? Mt : ceilf(nMs);
    const bool X = nNs <= nMs;
    const float sA = fminf(nNs, nMs);
    const float fmA = fmaxf(sA >= Mt ? Mt : ceilf(sA), fm0);
    const int inF2 = inF + sn;
    const Off o2 = clampN(inF2);
    const float enf = ey(on + omf), eff = ey(of + omf);
    const float e2n = ey(o2 + omn), e2f = ey(o2 + omf);
    {
      const float M = fmA - fm0;
      const float jm = __fmaf_rn(0.5f, fm0 + fmA, jb);
      const float a = __fmaf_rn(jm, dN, Nq) - fcn, c = __fmaf_rn(jm, dM, Mq) - fcm;
      const float k1 = efn - enn, k3 = enf - enn, k5 = (eff - enf) - k1;
      const float f = fmaf(c, fmaf(a, k5, k3), fmaf(a, k1, enn));
      acc = fmaf(M, fmaf(k5, fmaf(M * M, g, -g), f), acc);
    }
    {
      const float M = fmL - fmA;
      const float jm = __fmaf_rn(0.5f, fmA + fmL, jb);
      const float a = __fmaf_rn(jm, dN, Nq) - (fcn + 1.f), c = __fmaf_rn(jm, dM, Mq) - fcm;
      const float k1 = e2n - efn, k3 = eff - efn, k5 = (e2f - eff) - k1;
      const float f = fmaf(c, fmaf(a, k5, k3), fmaf(a, k1, efn));
      acc = fmaf(M, fmaf(k5, fmaf(M * M, g, -g), f), acc);
    }
    fm0 = fmL;
    if (fm0 >= Mt) break;
    // next layer, one minor cell further when this layer crossed
    enn = X ? eff : enf;
    efn = X ? e2f : eff;
    if (X) {
      fcn += 1.f;
      inF = inF2;
      on = of;
      of = o2;
      nNs = ((fcn + 1.f) - pN) * isN;
    }
    fcm += 1.f;
    imF += sm;
    omn = omf;
    omf = clampM(imF);
    nMs = ((fcm + 1.f) - pM) * isM;
  }
  return acc;
}

template <int VT, class Off>
__device__ float cell_sum_xz(const Cell<VT>& C, float qx, float b, int iy, float qz, float dqx, float dqz, int j0,
                             int J) {
  if (fabsf(dqz) >= fabsf(dqx)) return layer_sum_xz<VT, true, Off>(C, qx, b, iy, qz, dqx, dqz, j0, J);
  return layer_sum_xz<VT, false, Off>(C, qx, b, iy, qz, dqx, dqz, j0, J);
}

// cell_sum for a ray whose y moves slowly (a beam declined by up to about 14
// degrees against the tilt axis): the layer walk along the major axis, with
// the y interpolation weight a linear function of the sample.
//
// The walk forms the weights of the voxels (axis_walk): a cell's M samples
// with mean local coordinates (a, c) in x-z and b in y, and steps da, dc, db,
// have with V = (M^2 - 1) / 12 the moments
//   sum ac  = M (a c + da dc V),      sum ba = M (b a + db da V),
//   sum bac = M (b (a c + da dc V) + a db dc V + c db da V),
// so each corner's weight splits into its parts on the y planes of the cell.
// A step ends at the next layer or, rarely, at the next y plane, where the
// far row's weights are applied before the planes change. Against the walk
// from cell to cell a step has no case distinction but that one, and reads 8
// voxels at most where a cell reads 4 to 8 and there are 1.5 cells a layer.
// What bounds it: instruction issue. 256 x 240 x 96 at 0.8 degrees, 12
// projections: 4.2 -> 3.05 ms.
template <int VT>
__device__ __noinline__ float tilted_sum(const Cell<VT>& C, float qx, float qy, float qz, float dqx, float dqy,
                                         float dqz, int j0, int J) {
  if (j0 >= J) return 0.0f;
  const bool zmaj = fabsf(dqz) >= fabsf(dqx);
  const float qm = zmaj ? qz : qx, dqm = zmaj ? dqz : dqx;
  const float qn = zmaj ? qx : qz, dqn = zmaj ? dqx : dqz;
  const int sm = dqm < 0.f ? -1 : 1, sn = dqn < 0.f ? -1 : 1, sy = dqy < 0.f ? -1 : 1;
  const float Mq = sm > 0 ? qm : -qm, Nq = sn > 0 ? qn : -qn, Yq = sy > 0 ? qy : -qy;
  const float dM = fabsf(dqm), dN = fabsf(dqn), dY = fabsf(dqy);
  const float fj0 = (float)j0, jb = fj0 - 0.5f;
  const float pM = __fmaf_rn(fj0, dM, Mq), pN = __fmaf_rn(fj0, dN, Nq), pY = __fmaf_rn(fj0, dY, Yq);
  const float fm = floorf(pM), fn = floorf(pN), fy = floorf(pY);
  const float isM = 1.0f / dM, isN = dN > 0.f ? 1.0f / dN : 0.f, isY = dY > 0.f ? 1.0f / dY : 0.f;
  const float nM0 = ((fm + 1.f) - pM) * isM;
  const float nN0 = dN > 0.f ? ((fn + 1.f) - pN) * isN : FLT_MAX;
  const float nY0 = dY > 0.f ? ((fy + 1.f) - pY) * isY : FLT_MAX;
  const float Mt = (float)(J - j0);
  const float gMN = dM * dN * (1.0f / 12.0f), gMY = dM * dY * (1.0f / 12.0f), gNY = dN * dY * (1.0f / 12.0f);
  const float hM = 0.5f * dM, hN = 0.5f * dN, hY = 0.5f * dY;
  float relM = __fmaf_rn(jb, dM, __fsub_rn(Mq, fm)), relN = __fmaf_rn(jb, dN, __fsub_rn(Nq, fn)),
        relY = __fmaf_rn(jb, dY, __fsub_rn(Yq, fy));
  const int nM = zmaj ? C.nz : C.nx, nN = zmaj ? C.nx : C.nz;
  const long eM = zmaj ? C.sz : 1, eN = zmaj ? 1 : C.sz;
  int im = sm * (int)fm, in = sn * (int)fn, iy = sy * (int)fy;
  long y0 = 0, y1 = 0;
  auto planes = [&]() {
    const int a = iy + sy;
    y0 = (long)(iy < 0 ? 0 : (iy > C.ny - 1 ? C.ny - 1 : iy)) * C.sy;
    y1 = (long)(a < 0 ? 0 : (a > C.ny - 1 ? C.ny - 1 : a)) * C.sy;
  };
  planes();
  float S = 0.f, T = 0.f;
  // weights w and their parts b on the second plane, positions first .. in + 2
  auto row = [&](int mi, float w0, float w1, float w2, float w3, float b0, float b1, float b2, float b3, bool first,
                 bool last) {
    mi = mi < 0 ? 0 : (mi > nM - 1 ? nM - 1 : mi);
    const long r = (long)mi * eM;
    auto at = [&](int n) { return r + (long)(n < 0 ? 0 : (n > nN - 1 ? nN - 1 : n)) * eN; };
    auto add = [&](long o, float w, float b) {
      const float u = Voxel<VT>::load(C.vol, o + y0), v = Voxel<VT>::load(C.vol, o + y1);
      S = fmaf(u, w - b, S);
      T = fmaf(v, b, T);
    };
    if (first) add(at(in - sn), w0, b0);
    add(at(in), w1, b1);
    add(at(in + sn), w2, b2);
    if (last) add(at(in + 2 * sn), w3, b3);
  };
  float k = 0.f, kn = 0.f, ky = 0.f, fm0 = 0.f;
  float g0 = 0.f, g1 = 0.f, g2 = 0.f, e0 = 0.f, e1 = 0.f, e2 = 0.f;  // far weights and their second-plane parts
  bool Xp = false;
#pragma unroll 1
  for (int guard = 0; guard < 1 << 20; ++guard) {
    const float nMs = __fmaf_rn(k, isM, nM0), nNs = __fmaf_rn(kn, isN, nN0), nYs = __fmaf_rn(ky, isY, nY0);
    const bool Y = nYs <= nMs;          // the y plane comes first
    const float end = fminf(nMs, nYs);
    const bool X = nNs <= end;
    const float tL = fminf(end, Mt);
    const float2 f = ceil2(fminf(nNs, tL), tL);
    const float MA = f.x - fm0, MB = f.y - f.x, sA = fm0 + f.x, sB = f.x + f.y;
    // sums of one cell: M, Ma, Mc, ac and the same with b
    struct Moments {
      float w00, w10, w01, w11, b00, b10, b01, b11;
    };
    auto moments = [&](float M, float s, float off) {
      const float a = fmaf(s, hN, relN) - off, c = fmaf(s, hM, relM), b = fmaf(s, hY, relY);
      const float V = fmaf(M, M, -1.f);
      const float ac = fmaf(a, c, gMN * V), ba = gNY * V, bc = gMY * V;  // (the last two: the covariances)
      const float Ma = M * a, Mc = M * c, t = M * ac;
      const float Mb = M * b, Mba = M * fmaf(b, a, ba), Mbc = M * fmaf(b, c, bc);
      const float Mbac = M * fmaf(b, ac, fmaf(a, bc, c * ba));
      Moments m;
      m.w11 = t;
      m.w10 = Ma - t;
      m.w01 = Mc - t;
      m.w00 = (M - Ma) - m.w01;
      m.b11 = Mbac;
      m.b10 = Mba - Mbac;
      m.b01 = Mbc - Mbac;
      m.b00 = (Mb - Mba) - m.b01;
      return m;
    };
    const Moments A = moments(MA, sA, 0.f), B = moments(MB, sB, 1.f);
    row(im, g0, g1 + A.w00, g2 + (A.w10 + B.w00), B.w10, e0, e1 + A.b00, e2 + (A.b10 + B.b00), B.b10, Xp, X);
    const float F1 = A.w11 + B.w01, E1 = A.b11 + B.b01;
    fm0 = f.y;
    const bool done = fm0 >= Mt;
    if (Y || done) {  // the far row, in the planes at hand
      row(im + sm, 0.f, A.w01, F1, B.w11, 0.f, A.b01, E1, B.b11, false, X);
      if (done) break;
      g0 = g1 = g2 = e0 = e1 = e2 = 0.f;
      ky += 1.f;
      relY -= 1.f;
      iy += sy;
      planes();
    } else {
      g0 = X ? A.w01 : 0.f;
      g1 = X ? F1 : A.w01;
      g2 = X ? B.w11 : F1;
      e0 = X ? A.b01 : 0.f;
      e1 = X ? E1 : A.b01;
      e2 = X ? B.b11 : E1;
      k += 1.f;
      relM -= 1.f;
      im += sm;
    }
    if (X) {
      relN -= 1.f;
      kn += 1.f;
      in += sn;
    }
    Xp = X && !Y;
  }
  return S + T;
}

// Sum over the samples of one sub-ray from t0 to tout (first_at_source: the
// slicer's first sample is taken at the ray start, ForwardProjectionSlicer.cu:126-141).
template <int VT, class Off>
__device__ float ray_sum(const KConst& c, const Cell<VT>& C, float3 s, float t0, float tout, bool first_at_source) {
  const float h = c.vs.x * 0.15f;
  float step;
  bool ok;
  int J = progression(t0, tout, h, step, ok);
  if (!(t0 <= tout)) return 0.0f;
  if (!ok) {  // sample-by-sample marching with the reference's float recurrence
    float sum = 0.0f, t = t0;
    bool first = true;
#pragma unroll 1
    while (t <= tout) {
      float3 p = first && first_at_source ? s : ray_point(c, s, t);
      float3 q = interp_coord(c, p);
      sum += trilinear<VT>(C, q.x, q.y, q.z);
      first = false;
      t += h;
    }
    return sum;
  }
  // q(j) = q(t0) + j * dq
  float3 q0 = interp_coord(c, ray_point(c, s, t0));
  const float3 dq = interp_step(c, step);
  const float dqx = dq.x, dqy = dq.y, dqz = dq.z;
  float sum = 0.0f;
  int j0 = 0;
  if (first_at_source) {
    float3 q = interp_coord(c, s);
    sum += trilinear<VT>(C, q.x, q.y, q.z);
    j0 = 1;
  }
  // y stays in one cell and moves by < 1e-5 voxel over the ray: bilinear x-z walk
  const float ylast = qpos(q0.y, J - 1, dqy);
  if (fabsf(dqy) * (float)J < 1e-5f && floorf(q0.y) == floorf(ylast)) {
    const float fy = floorf(q0.y);
    return sum + cell_sum_xz<VT, Off>(C, q0.x, q0.y - fy, (int)fy, q0.z, dqx, dqz, j0, J);
  }
  // y slow against the major axis: layers; else cell by cell
  if (fabsf(dqy) <= 0.25f * fmaxf(fabsf(dqx), fabsf(dqz)))
    return sum + tilted_sum<VT>(C, q0.x, q0.y, q0.z, dqx, dqy, dqz, j0, J);
  return sum + cell_sum<VT>(C, q0.x, q0.y, q0.z, dqx, dqy, dqz, j0, J);
}

// mode 0: march (proj += sum/4, dist = mean chord); mode 1: slicer (proj += sum/4 within [tmin, tmax])
// NW warps per block: NW detector columns x 8 rows; blocks of 128 threads
// fit 6 per SM at the walker's register count (256-thread blocks fit 3); the
// launch shape is picked per problem by the reconstructor's autotuner.
template <int VT, int MODE, class Off, int NW>
__global__ void __launch_bounds__(32 * NW, 24 / NW) k_project_fast(KConst c, const void* __restrict__ vol, float* __restrict__ proj,
                                                      float* __restrict__ dist, size_t pitchE, float tminDef,
                                                      float tmaxDef, int x0, int y0, int x1, int y1) {
  // lanes: 4 sub-rays of a pixel adjacent; a warp spans 8 detector rows (v);
  // the NW warps of a block, NW detector columns (u)
  const int lane = threadIdx.x & 31;
  const int sub = lane & 3;
  const int row = (threadIdx.x >> 2) & 7;
  const int warp = threadIdx.x >> 5;
  const int x = x0 + (int)blockIdx.x * NW + warp;
  const int y = y0 + (int)blockIdx.y * 8 + row;
  const bool active = x < x1 && y < y1;
  Cell<VT> C{vol, (int)c.dim.x, (int)c.dim.y, (int)c.dim.z, (long)c.dim.x, (long)c.dim.x * (long)c.dim.y};
  float sum = 0.0f, gx = 0.0f, gz = 0.0f;
  if (active) {
    const float osx = (sub & 2) ? 0.75f : 0.25f, osy = (sub & 1) ? 0.75f : 0.25f;
    float3 s = ray_src(c, (float)x + osx, (float)y + osy);
    float tin, tout;
    hit(s, c.n, c.bbMin, c.bbMax, tin, tout);
    if (tout - tin > 0.0f) {
      gx = 1.0f;
      gz = tout - tin;
      if (MODE == 1) {
        tin = fmaxf(tin, tminDef);
        tout = fminf(tout, tmaxDef);
      }
      sum = ray_sum<VT, Off>(c, C, s, tin, tout, MODE == 1);
    }
  }
  sum = quad_sum_ordered(sum);
  if (MODE == 0) {
    gx = quad_sum_ordered(gx);
    gz = quad_sum_ordered(gz);
  }
  if (active && sub == 0) {
    const size_t i = (size_t)y * pitchE + x;
    proj[i] += sum * c.vs.x * 0.15f * 0.25f;
    if (MODE == 0) dist[i] = fmaxf(0.0f, gz / gx);
  }
}

// Zero in the slab images that a pixel's rays do not meet (they meet
// [klo, khi]).
__device__ __forceinline__ void clear_slabs(float* img, size_t stride, int count, int klo, int khi) {
  for (int k = 0; k < count; ++k)
    if (k < klo || k > khi) img[(size_t)k * stride] = 0.0f;
}

// All defocus slabs of one projection in one launch: slab k's image gets
// the slicer's integral over [bound[k], bound[k+1]] (ForwardProjectionSlicer.cu:57-220,
// called once per slab by Reconstructor.cpp:515-585). The 4 lanes of a pixel
// walk the union of their slab ranges together so each slab's sum keeps the
// reference's sub-ray order. clear: the pixels that no ray of a slab reaches
// are set to 0 (else the caller clears the images first).
template <int VT, class Off, int NW>
__global__ void __launch_bounds__(32 * NW, 24 / NW) k_slicer_fused(KConst c, const void* __restrict__ vol, float* __restrict__ imgs,
                                                      size_t img_stride, size_t pitchE, SlabTable slabs, int clear, int x0,
                                                      int y0, int x1, int y1) {
  const int lane = threadIdx.x & 31;
  const int sub = lane & 3;
  const int row = (threadIdx.x >> 2) & 7;
  const int warp = threadIdx.x >> 5;
  const int x = x0 + (int)blockIdx.x * NW + warp;
  const int y = y0 + (int)blockIdx.y * 8 + row;
  const bool active = x < x1 && y < y1;
  Cell<VT> C{vol, (int)c.dim.x, (int)c.dim.y, (int)c.dim.z, (long)c.dim.x, (long)c.dim.x * (long)c.dim.y};
  float3 s = make_float3(0.f, 0.f, 0.f);
  float tin = 0.f, tout = -1.f;
  int klo = ESB_MAX_SLABS, khi = -1;
  bool hitray = false;
  if (active) {
    const float osx = (sub & 2) ? 0.75f : 0.25f, osy = (sub & 1) ? 0.75f : 0.25f;
    s = ray_src(c, (float)x + osx, (float)y + osy);
    hit(s, c.n, c.bbMin, c.bbMax, tin, tout);
    hitray = tout - tin > 0.0f;
    if (hitray) {
      for (int k = 0; k < slabs.count; ++k) {
        // slab k has samples when max(tin, b_k) <= min(tout, b_{k+1})
        if (fmaxf(tin, slabs.bound[k]) <= fminf(tout, slabs.bound[k + 1])) {
          klo = min(klo, k);
          khi = max(khi, k);
        }
      }
    }
  }
  for (int o = 1; o <= 2; o <<= 1) {
    klo = min(klo, __shfl_xor_sync(0xffffffffu, klo, o));
    khi = max(khi, __shfl_xor_sync(0xffffffffu, khi, o));
  }
  // the warp walks the union of its pixels' slab ranges (shuffles need all lanes)
  int wlo = klo, whi = khi;
  for (int o = 4; o <= 16; o <<= 1) {
    wlo = min(wlo, __shfl_xor_sync(0xffffffffu, wlo, o));
    whi = max(whi, __shfl_xor_sync(0xffffffffu, whi, o));
  }
  const size_t pix = (size_t)y * pitchE + x;
  for (int k = wlo; k <= whi; ++k) {
    float v = 0.0f;
    if (hitray && k >= klo && k <= khi) {
      const float t0 = fmaxf(tin, slabs.bound[k]);
      const float t1 = fminf(tout, slabs.bound[k + 1]);
      v = ray_sum<VT, Off>(c, C, s, t0, t1, true);
    }
    v = quad_sum_ordered(v);
    if (active && sub == 0 && k >= klo && k <= khi) imgs[(size_t)k * img_stride + pix] = v * c.vs.x * 0.15f * 0.25f;
  }
  if (clear && active && sub == 0) clear_slabs(imgs + pix, img_stride, slabs.count, klo, khi);
}

// ---------------------------------------------------------------------------
// Single-axis series: k_project_axis, k_slicer_axis.
//
// Every ray of a single-axis projection moves in the x-z plane with the same
// direction, so the major axis of the layer walk and the signs of both steps
// are the same for all rays of a launch: they become template parameters
// (ZMAJ, SM, SN), and the host picks the instance from the beam direction.
// The samples and their split into cells are layer_sum_xz's.

// A voxel as loaded (float, or the 16 bits of a half / bfloat16), converted
// to float where it is used.
template <int VT>
struct RawVoxel {
  typedef unsigned short T;
};
template <>
struct RawVoxel<ESB_VOXEL_F32> {
  typedef float T;
};
template <int VT>
__device__ __forceinline__ typename RawVoxel<VT>::T ldraw(const char* p) {
  if constexpr (VT == ESB_VOXEL_F32) return __ldg((const float*)p);
  else return __ldg((const unsigned short*)p);
}
// v = the voxel at p where `on`, else v stays (a predicated load, no branch).
template <int VT>
__device__ __forceinline__ void ldraw_if(typename RawVoxel<VT>::T& v, const char* p, bool on) {
  if constexpr (VT == ESB_VOXEL_F32)
    asm("{.reg .pred q; setp.ne.u32 q, %2, 0; @q ld.global.nc.f32 %0, [%1];}" : "+f"(v) : "l"(p), "r"((unsigned)on));
  else
    asm("{.reg .pred q; setp.ne.u32 q, %2, 0; @q ld.global.nc.u16 %0, [%1];}" : "+h"(v) : "l"(p), "r"((unsigned)on));
}
template <int VT>
__device__ __forceinline__ float cvt(typename RawVoxel<VT>::T r) {
  if constexpr (VT == ESB_VOXEL_F32) return r;
  else if constexpr (VT == ESB_VOXEL_F16) return __half2float(__ushort_as_half(r));
  else return __uint_as_float((unsigned)r << 16);
}

// Sum of the trilinear interpolant over samples j0 .. J-1 of one ray whose y
// interpolation coordinate lies in cell iy with weight b, walked along major
// axis z (ZMAJ) or x with step signs SM (major) and SN (minor). Mq, Nq:
// mirrored major / minor coordinate of sample 0. Off: byte offsets into the
// volume, 32-bit below 4 GiB.
//
// The sum is linear in the voxels, so the walk forms the weight of every
// voxel instead of evaluating the interpolant: the samples of a layer lie in
// at most two cells A = (n, m) and B = (n + 1, m); a cell's M samples with
// mean local coordinates (a, c) give its corners the weights
//   t = M (a c + q) to the far upper one, M a - t, M c - t and
//   M - M a - (M c - t) to the others, q = dN dM (M^2 - 1) / 12.
// A row of voxels gets the far weights of the layer before it and the near
// weights of the layer after it: 4 weights at the minor positions n - 1 ..
// n + 2 of the layer's cell n, the first only after a crossing, the last
// only before one. They are applied to the rows of both y planes with
// separate sums, which are interpolated in y once at the end.
//
// What bounds it: instruction issue and the FMA pipe, with the latency of
// the rows' loads behind them. Additions and products of cells A and B are
// packed pairs, one issue slot for both; fused multiply-adds are not (a
// packed one with three different operands holds the pipe for 3.2 cycles,
// two plain ones for 2.6), the ceilings of the two crossings are a packed
// add that rounds up (no conversion-unit instruction), the outer positions
// are read only by the lanes whose ray needs them, the next row's loads are
// in flight during a layer's arithmetic, and layers whose rows and window
// lie inside the volume and wholly inside the ray take no clamps, no index
// arithmetic and no end test. 64 registers and 32 warps per SM: with 80 and
// 24 warps 974 us where this takes 866.
// 1024 x 1024 x 64 FP32, one projection, against the sums of the interpolant
// per cell that it replaces: in-plane rotation 0.2 degrees, tilts 0 / 24 /
// -40 / -50: 1090 / 1047 / 926 / 1046 -> 866 / 854 / 772 / 922 us.
template <int VT, bool ZMAJ, int SM, int SN, class Off>
__device__ __forceinline__ float axis_walk(const AxisStep& A, const Cell<VT>& C, float Mq, float Nq, float b, int iy,
                                           int j0, int J) {
  typedef typename RawVoxel<VT>::T Raw;
  constexpr int ES = VT == ESB_VOXEL_F32 ? 4 : 2;
  const Off sM = ES * (ZMAJ ? (Off)C.sz : (Off)1), sN = ES * (ZMAJ ? (Off)1 : (Off)C.sz);  // strides in bytes
  const int nM = ZMAJ ? C.nz : C.nx, nN = ZMAJ ? C.nx : C.nz;
  const char* const base = (const char*)C.vol;
  const float fj0 = (float)j0;
  const float pM = __fmaf_rn(fj0, A.dM, Mq), pN = __fmaf_rn(fj0, A.dN, Nq);
  const float fm = floorf(pM), fn = floorf(pN);  // mirrored cell of the first sample
  // sample parameters of the k-th major and the kn-th minor crossing
  const float nM0 = ((fm + 1.f) - pM) * A.isM;
  const float nN0 = A.isN > 0.f ? ((fn + 1.f) - pN) * A.isN : FLT_MAX;
  const float Mt = (float)(J - j0);
  // a cell's mean local coordinate is s * step / 2 + rel, s the sum of its
  // first and past-the-last sample numbers
  const float jb = fj0 - 0.5f;
  float2 relN;
  relN.x = __fmaf_rn(jb, A.dN, __fsub_rn(Nq, fn));
  relN.y = relN.x - 1.f;
  float relM = __fmaf_rn(jb, A.dM, __fsub_rn(Mq, fm));
  const int ny = C.ny;
  const Off yA = (Off)(ES * C.sy) * (Off)(iy < 0 ? 0 : (iy > ny - 1 ? ny - 1 : iy));
  const Off dy = (Off)(ES * C.sy) * (Off)(iy + 1 < 0 ? 0 : (iy + 1 > ny - 1 ? ny - 1 : iy + 1)) - yA;
  // near row of the current layer and its cell
  int im = SM * (int)fm, in0 = SN * (int)fn;
  const int lowN = SN > 0 ? 1 : 2, highN = SN > 0 ? nN - 3 : nN - 2;  // in0 with its window inside
  float k = 0.f, kn = 0.f, fm0 = 0.f;
  float g0 = 0.f, g1 = 0.f, g2 = 0.f;  // far weights of the layer before, at n - 1, n, n + 1
  float S0 = 0.f, T0 = 0.f, S1 = 0.f, T1 = 0.f;  // sums over planes iy and iy + 1
  // layers below kEnd end before the ray's last sample, on rows of the volume
  const float kEnd = fminf(floorf((Mt - nM0) * A.dM), SM > 0 ? (float)(nM - 1) - fm : -fm);
  // one layer: row values v* (plane iy) and w* (plane iy + 1) at n - 1 .. n + 2
  auto layer = [&](bool X, float tA, float tL, Raw va, Raw vb, Raw vc, Raw vd, Raw wa, Raw wb, Raw wc, Raw wd) {
    const float2 f = ceil2(tA, tL);
    // samples [fm0, f.x) lie in cell A, [f.x, f.y) in cell B
    const float2 M = make_float2(f.x - fm0, f.y - f.x), mM = make_float2(fm0 - f.x, f.x - f.y);
    const float sA = fm0 + f.x, sB = f.x + f.y;
    const float2 a = make_float2(fmaf(sA, A.hN, relN.x), fmaf(sB, A.hN, relN.y));
    const float2 c = make_float2(fmaf(sA, A.hM, relM), fmaf(sB, A.hM, relM));
    const float2 MM = __fmul2_rn(M, M), Ma = __fmul2_rn(M, a), Mc = __fmul2_rn(M, c);
    const float2 acq = make_float2(fmaf(a.x, c.x, fmaf(MM.x, A.g, -A.g)), fmaf(a.y, c.y, fmaf(MM.y, A.g, -A.g)));
    const float2 mt = __fmul2_rn(mM, acq);  // - t
    const float2 w10 = __fadd2_rn(Ma, mt), wf = __fadd2_rn(Mc, mt);
    const float2 m00 = __fadd2_rn(__fadd2_rn(Ma, wf), mM);  // minus the near lower weights
    const float i0 = g1 - m00.x, i1 = g2 + (w10.x - m00.y);
    S0 = fmaf(cvt<VT>(vb), i0, S0);
    S1 = fmaf(cvt<VT>(wb), i0, S1);
    T0 = fmaf(cvt<VT>(vc), i1, T0);
    T1 = fmaf(cvt<VT>(wc), i1, T1);
    S0 = fmaf(cvt<VT>(va), g0, S0);
    S1 = fmaf(cvt<VT>(wa), g0, S1);
    T0 = fmaf(cvt<VT>(vd), w10.y, T0);
    T1 = fmaf(cvt<VT>(wd), w10.y, T1);
    const float F1 = wf.y - mt.x;
    g0 = X ? wf.x : 0.f;
    g1 = X ? F1 : wf.x;
    g2 = X ? -mt.y : F1;
    fm0 = f.y;
    if (X) relN = __fadd2_rn(relN, splat(-1.f));
    relM -= 1.f;
  };
  auto clamped = [&](int mi, int n) -> const char* {
    mi = mi < 0 ? 0 : (mi > nM - 1 ? nM - 1 : mi);
    n = n < 0 ? 0 : (n > nN - 1 ? nN - 1 : n);
    return base + (Off)((Off)mi * sM + (Off)n * sN + yA);
  };
  const long step1 = SN > 0 ? (long)sN : -(long)sN;
  Raw va = Raw(0), vb, vc, vd = Raw(0), wa = Raw(0), wb, wc, wd = Raw(0);
  float nMs = 0.f, nNs = 0.f;
  bool X = false, Xp = false;  // a minor crossing in this layer, in the one before
  // row im with its window, clamped; the outer positions 0 where they have no
  // weight (0 times an infinite voxel or NaN is NaN; loads under predicates
  // made small volumes 3 % slower)
  auto fetch = [&]() {
    nMs = __fmaf_rn(k, A.isM, nM0);
    nNs = __fmaf_rn(kn, A.isN, nN0);
    X = nNs <= nMs;
    const char* p = clamped(im, in0 - SN);
    va = ldraw<VT>(p), wa = ldraw<VT>(p + dy);
    p = clamped(im, in0);
    vb = ldraw<VT>(p), wb = ldraw<VT>(p + dy);
    p = clamped(im, in0 + SN);
    vc = ldraw<VT>(p), wc = ldraw<VT>(p + dy);
    p = clamped(im, in0 + 2 * SN);
    vd = ldraw<VT>(p), wd = ldraw<VT>(p + dy);
    if (!Xp) va = wa = Raw(0);
    if (!X) vd = wd = Raw(0);
  };
  // the layer of the row at hand, which may be the ray's last
  auto edge_layer = [&]() {
    const float tL = fminf(nMs, Mt);
    layer(X, fminf(nNs, tL), tL, va, vb, vc, vd, wa, wb, wc, wd);
    im += SM;
    k += 1.f;
    Xp = X;
    if (X) {
      in0 += SN;
      kn += 1.f;
    }
  };
  // Edge layers until every ray of the warp is inside the volume or done:
  // the rays enter the loop over inner layers together.
  const unsigned mask = __activemask();
  fetch();
  for (int guard = 0; guard < 1 << 20; ++guard) {
    const bool in = k < kEnd && (unsigned)im < (unsigned)nM && in0 >= lowN && in0 < highN;
    if (__all_sync(mask, in || fm0 >= Mt)) break;
    if (fm0 < Mt) {
      edge_layer();
      fetch();
    }
  }
  // minor crossings until the window may leave the volume
  const float knEnd = kn + (float)(SN > 0 ? highN - in0 : in0 - lowN);
  if (fm0 < Mt && k < kEnd && kn < knEnd) {
    const float k0 = k, kn0 = kn;
    Off off = (Off)im * sM + (Off)in0 * sN + yA;
#pragma unroll 2
    do {
      k += 1.f;
      off += SM > 0 ? sM : (Off)0 - sM;
      if (X) {
        kn += 1.f;
        off += SN > 0 ? sN : (Off)0 - sN;
      }
      const float nM1 = __fmaf_rn(k, A.isM, nM0), nN1 = __fmaf_rn(kn, A.isN, nN0);
      const bool X1 = nN1 <= nM1;
      // the next row, in flight during this layer's arithmetic
      const char *u = base + off, *r = base + (Off)(off + dy);
      Raw na = va, nd = vd, oa = wa, od = wd;
      const Raw nb = ldraw<VT>(u), ob = ldraw<VT>(r), nc = ldraw<VT>(u + step1), oc = ldraw<VT>(r + step1);
      ldraw_if<VT>(na, u - step1, X);
      ldraw_if<VT>(oa, r - step1, X);
      ldraw_if<VT>(nd, u + 2 * step1, X1);
      ldraw_if<VT>(od, r + 2 * step1, X1);
      layer(X, fminf(nNs, nMs), nMs, va, vb, vc, vd, wa, wb, wc, wd);
      va = na, vb = nb, vc = nc, vd = nd, wa = oa, wb = ob, wc = oc, wd = od;
      nMs = nM1;
      nNs = nN1;
      X = X1;
    } while (k < kEnd && kn < knEnd);
    im += SM * (int)(k - k0);
    in0 += SN * (int)(kn - kn0);
  }
#pragma unroll 1
  for (int guard = 0; guard < 1 << 20 && fm0 < Mt; ++guard) {
    edge_layer();
    fetch();
  }
  {  // the far row of the last layer
    const char *p1 = clamped(im, in0), *p2 = clamped(im, in0 + SN);
    S0 = fmaf(cvt<VT>(ldraw<VT>(p1)), g1, S0);
    S1 = fmaf(cvt<VT>(ldraw<VT>(p1 + dy)), g1, S1);
    T0 = fmaf(cvt<VT>(ldraw<VT>(p2)), g2, T0);
    T1 = fmaf(cvt<VT>(ldraw<VT>(p2 + dy)), g2, T1);
    if (Xp) {
      const char* p0 = clamped(im, in0 - SN);
      S0 = fmaf(cvt<VT>(ldraw<VT>(p0)), g0, S0);
      S1 = fmaf(cvt<VT>(ldraw<VT>(p0 + dy)), g0, S1);
    }
  }
  return fmaf(b, S1 + T1, (1.0f - b) * (S0 + T0));
}

// ray_sum for the few rays that do not fit an axis kernel's instance; a call
// of its own, so that its registers do not weigh on the walk.
template <int VT>
__device__ __noinline__ float other_ray_sum(const KConst* c, const void* vol, float3 s, float t0, float tout,
                                            bool first_at_source) {
  const Cell<VT> C{vol, (int)c->dim.x, (int)c->dim.y, (int)c->dim.z, (long)c->dim.x, (long)c->dim.x * (long)c->dim.y};
  return ray_sum<VT, unsigned long long>(*c, C, s, t0, tout, first_at_source);
}

// First sample of run `seg` of J samples in `segs` runs.
__device__ __forceinline__ int run_start(int J, int seg, int segs) { return (int)((long long)J * seg / segs); }

// A block's warps in groups of `segs` that sum one run of the same rays each:
// adds the group's sums in the runs' order, valid in its first warp.
template <int N>
__device__ __forceinline__ void sum_runs(float (&v)[N], int segs) {
  __shared__ float part[8][N][32];
  if (segs == 1) return;  // uniform
  const int w = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31), seg = w & (segs - 1);
#pragma unroll
  for (int i = 0; i < N; ++i) part[w][i][lane] = v[i];
  __syncthreads();
  if (seg == 0)
    for (int r = 1; r < segs; ++r)
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] += part[w + r][i][lane];
}

// Sum over the samples of one sub-ray from t0 to tout (ray_sum) with the
// axis walk when the ray fits the launch's instance (its y in one cell, its
// step the launch's), else other_ray_sum. With first_at_source the first
// sample is the one at the ray's start, whose value is `source`. seg, segs:
// without first_at_source the samples are cut into `segs` runs, and this is
// the sum over run `seg`.
template <int VT, bool ZMAJ, int SM, int SN, class Off>
__device__ __forceinline__ float axis_ray_sum(const KConst& c, const AxisStep& A, const Cell<VT>& C, float3 s,
                                              float t0, float tout, bool first_at_source, float source, int seg,
                                              int segs) {
  if (!(t0 <= tout)) return 0.0f;
  const float h = c.vs.x * 0.15f;
  float step;
  bool ok;
  const int J = progression(t0, tout, h, step, ok);
  const float3 q0 = interp_coord(c, ray_point(c, s, t0));
  const float dqy = __fmul_rn(__fmul_rn(__fmul_rn(step, c.n.y), c.bbRcp.y), c.dim.y);
  const float ylast = qpos(q0.y, J - 1, dqy);
  const float fy = floorf(q0.y);
  if (!(ok && step == A.step && fabsf(dqy) * (float)J < 1e-5f && fy == floorf(ylast)))
    return seg == 0 ? other_ray_sum<VT>(&c, C.vol, s, t0, tout, first_at_source) : 0.0f;
  const float sum = first_at_source ? source : 0.0f;
  const int j0 = first_at_source ? 1 : run_start(J, seg, segs), j1 = first_at_source ? J : run_start(J, seg + 1, segs);
  if (j0 >= j1) return sum;
  const float qm = ZMAJ ? q0.z : q0.x, qn = ZMAJ ? q0.x : q0.z;
  return sum + axis_walk<VT, ZMAJ, SM, SN, Off>(A, C, SM > 0 ? qm : -qm, SN > 0 ? qn : -qn, q0.y - fy, (int)fy, j0, j1);
}

// Pixel of a thread in the axis kernels: the 4 sub-rays of a pixel in
// adjacent lanes, a warp spans 8 pixels along the detector axis that crosses
// the tilt axis (v, or u when `swap`), so that its rays lie in few y planes;
// the warps of a block step along the other axis, `segs` warps (a power of
// two) for the same pixels.
struct AxisPixel {
  int sub, x, y, seg;
  bool active;
  __device__ __forceinline__ AxisPixel(int swap, int segs, int x0, int y0, int x1, int y1) {
    const int lane = threadIdx.x & 31;
    sub = lane & 3;
    const int along = (int)blockIdx.y * 8 + (lane >> 2);
    const int w = (int)blockIdx.x * (blockDim.x >> 5) + (int)(threadIdx.x >> 5), across = w / segs;
    seg = w - across * segs;
    x = x0 + (swap ? along : across);
    y = y0 + (swap ? across : along);
    active = x < x1 && y < y1;
  }
};

// k_project_fast (march) for single-axis series.
template <int VT, bool ZMAJ, int SM, int SN, class Off>
__global__ void __launch_bounds__(256, 4) k_project_axis(const __grid_constant__ KConst c, const __grid_constant__ AxisStep A,
                                                      const void* __restrict__ vol, float* __restrict__ proj,
                                                      float* __restrict__ dist, size_t pitchE, int swap, int segs,
                                                      int x0, int y0, int x1, int y1) {
  const AxisPixel P(swap, segs, x0, y0, x1, y1);
  Cell<VT> C{vol, (int)c.dim.x, (int)c.dim.y, (int)c.dim.z, (long)c.dim.x, (long)c.dim.x * (long)c.dim.y};
  float sum = 0.0f, gx = 0.0f, gz = 0.0f;
  if (P.active) {
    const float osx = (P.sub & 2) ? 0.75f : 0.25f, osy = (P.sub & 1) ? 0.75f : 0.25f;
    const float3 s = ray_src(c, (float)P.x + osx, (float)P.y + osy);
    float tin, tout;
    hit(s, c.n, c.bbMin, c.bbMax, tin, tout);
    if (tout - tin > 0.0f) {
      gx = 1.0f;
      gz = tout - tin;
      sum = axis_ray_sum<VT, ZMAJ, SM, SN, Off>(c, A, C, s, tin, tout, false, 0.0f, P.seg, segs);
    }
  }
  float runs[1] = {sum};
  sum_runs(runs, segs);
  sum = quad_sum_ordered(runs[0]);
  gx = quad_sum_ordered(gx);
  gz = quad_sum_ordered(gz);
  if (P.active && P.sub == 0 && P.seg == 0) {
    const size_t i = (size_t)P.y * pitchE + P.x;
    proj[i] += sum * c.vs.x * 0.15f * 0.25f;
    dist[i] = fmaxf(0.0f, gz / gx);
  }
}

// The slabs ka .. kb - 1 of wlo .. whi that this block of gridDim.z walks.
__device__ __forceinline__ void slab_part(int wlo, int whi, int& ka, int& kb) {
  const int n = max(whi - wlo + 1, 0), z = (int)blockIdx.z, nz = (int)gridDim.z;
  ka = wlo + n * z / nz;
  kb = wlo + n * (z + 1) / nz;
}

// k_slicer_fused for single-axis series; pixels as k_project_axis. The
// sample at the ray's start, the first of every slab, is formed once.
template <int VT, bool ZMAJ, int SM, int SN, class Off>
__global__ void __launch_bounds__(256, 4) k_slicer_axis(const __grid_constant__ KConst c, const __grid_constant__ AxisStep A,
                                                     const void* __restrict__ vol, float* __restrict__ imgs,
                                                     size_t img_stride, size_t pitchE, SlabTable slabs, int clear,
                                                     int swap, int x0, int y0, int x1, int y1) {
  const AxisPixel P(swap, 1, x0, y0, x1, y1);
  Cell<VT> C{vol, (int)c.dim.x, (int)c.dim.y, (int)c.dim.z, (long)c.dim.x, (long)c.dim.x * (long)c.dim.y};
  float3 s = make_float3(0.f, 0.f, 0.f);
  float tin = 0.f, tout = -1.f, source = 0.f;
  int klo = ESB_MAX_SLABS, khi = -1;
  bool hitray = false;
  if (P.active) {
    const float osx = (P.sub & 2) ? 0.75f : 0.25f, osy = (P.sub & 1) ? 0.75f : 0.25f;
    s = ray_src(c, (float)P.x + osx, (float)P.y + osy);
    hit(s, c.n, c.bbMin, c.bbMax, tin, tout);
    hitray = tout - tin > 0.0f;
    if (hitray) {
      for (int k = 0; k < slabs.count; ++k) {
        // slab k has samples when max(tin, b_k) <= min(tout, b_{k+1})
        if (fmaxf(tin, slabs.bound[k]) <= fminf(tout, slabs.bound[k + 1])) {
          klo = min(klo, k);
          khi = max(khi, k);
        }
      }
      const float3 q = interp_coord(c, s);
      source = trilinear<VT>(C, q.x, q.y, q.z);
    }
  }
  for (int o = 1; o <= 2; o <<= 1) {
    klo = min(klo, __shfl_xor_sync(0xffffffffu, klo, o));
    khi = max(khi, __shfl_xor_sync(0xffffffffu, khi, o));
  }
  // the warp walks the union of its pixels' slab ranges (shuffles need all lanes)
  int wlo = klo, whi = khi;
  for (int o = 4; o <= 16; o <<= 1) {
    wlo = min(wlo, __shfl_xor_sync(0xffffffffu, wlo, o));
    whi = max(whi, __shfl_xor_sync(0xffffffffu, whi, o));
  }
  const size_t pix = (size_t)P.y * pitchE + P.x;
  int ka, kb;
  slab_part(wlo, whi, ka, kb);
  for (int k = ka; k < kb; ++k) {
    float v = 0.0f;
    if (hitray && k >= klo && k <= khi)
      v = axis_ray_sum<VT, ZMAJ, SM, SN, Off>(c, A, C, s, fmaxf(tin, slabs.bound[k]), fminf(tout, slabs.bound[k + 1]),
                                              true, source, 0, 1);
    v = quad_sum_ordered(v);
    if (P.active && P.sub == 0 && k >= klo && k <= khi)
      imgs[(size_t)k * img_stride + pix] = v * c.vs.x * 0.15f * 0.25f;
  }
  if (clear && blockIdx.z == 0 && P.active && P.sub == 0) clear_slabs(imgs + pix, img_stride, slabs.count, klo, khi);
}

// ---------------------------------------------------------------------------
// Series with next to no in-plane rotation: k_project_planes, k_slicer_planes.
//
// The rays of a detector row differ in y, and in x-z by the tilt axis'
// rotation against the detector: half a pixel along u moves a ray by half its
// sine, 0.0026 voxels at 0.3 degrees. A thread walks one line of 2 G sub-rays
// (G pixels along u) with the weights of its middle ray (axis_walk's). A
// layer's weights are bilinear in the ray's offset (e, f) along the minor and
// major axis as long as the samples stay in their cells, so with the weights'
// derivatives the sums of every ray of the line follow from the sums over
// the G + 2 y planes that the rays interpolate between,
//   S + e Se + f Sf + e f Sef,
// formed once per line; only the blend of two planes and the offset are a
// ray's own.
//
// A sample that the offset carries across a cell's face is evaluated on the
// face's other side, off by the distance past the face times the kink there.
// The sum of those errors grows with the offset's power 3/2, the walk's own
// error, from the rounding of a ray's float start point, with the beam's
// inclination. So offsets are bounded by kMaxShear and by a quarter of the
// minor step; beams next to a volume axis, where whole rays would lie on the
// far side of a face, thereby take the walk per ray. Against sums in 64 bits,
// 389 x 421 x 96, lines / walk per ray, beams of 0 to 60 degrees, rotations
// of 0.03 to 0.38: a smooth density with a tenth of noise, ratio at most
// 1.004; white noise, the worst case, at most 1.18 (1.38e-4 / 1.17e-4 at 11
// degrees). Offsets of up to 1/64 at any inclination gave 1.12 and 2.5, and
// 17 and 45 at 0 degrees. Correcting those samples one by one makes lines and
// walk agree to 1e-6, but every lane reads the volume at another layer: 93 ms
// where the walk per ray takes 61.
//
// Per ray and layer that leaves a 2 G-th of the weights, control and loads
// of each plane in place of all of them for two planes. What bounds it: the
// latency of a layer's loads at 12 to 16 warps per SM (issue 65 % busy, FMA
// pipe 41 %); caps of 96 and 80 registers (20 and 24 warps) spill and took
// 33.5 and 44.3 ms where 128 take 33.3. 1024 x 1024 x 256, 16 tilts with 0.3
// degrees jitter, CTF slabs: 61.1 ms with k_slicer_axis -> 39.5 (33.3 where
// offsets may reach 1/64); 256 x 256 x 128, 41 tilts: 7.3 ms with
// k_project_axis -> 3.2 (4 runs). A warp holds 16 detector rows x 2 sub-rows,
// so that its loads of a plane are contiguous. `swap` exchanges u and v (a
// tilt axis across the image).
struct PlaneWalk {
  int sM, sN;          // step signs
  int nM, nN;          // voxels along the major and minor axis
  unsigned dM, dN;     // their strides in bytes
};
constexpr float kMaxShear = 1.0f / 144.0f;  // voxels

// Plane sums over samples j0 .. J-1 of one ray: S[0] of the weights, and with
// SHEAR S[1], S[2] of their derivatives along the mirrored minor and major
// axis and S[3] of the mixed one; yoff: byte offsets of the planes
// (32-bit: the volume is below 4 GiB).
template <int VT, int NP, bool SHEAR>
__device__ __forceinline__ void plane_sums(const AxisStep& A, const PlaneWalk& W, const void* __restrict__ vol,
                                           const unsigned (&yoff)[NP], float Mq, float Nq, int j0, int J,
                                           float (&S)[SHEAR ? 4 : 1][NP]) {
  constexpr int NS = SHEAR ? 4 : 1;
  typedef typename RawVoxel<VT>::T Raw;
  const char* const base = (const char*)vol;
  const float fj0 = (float)j0, jb = fj0 - 0.5f;
  const float pM = __fmaf_rn(fj0, A.dM, Mq), pN = __fmaf_rn(fj0, A.dN, Nq);
  const float fm = floorf(pM), fn = floorf(pN);
  const float nM0 = ((fm + 1.f) - pM) * A.isM;
  const float nN0 = A.isN > 0.f ? ((fn + 1.f) - pN) * A.isN : FLT_MAX;
  const float Mt = (float)(J - j0);
  float relN = __fmaf_rn(jb, A.dN, __fsub_rn(Nq, fn)), relM = __fmaf_rn(jb, A.dM, __fsub_rn(Mq, fm));
  int im = W.sM * (int)fm, in = W.sN * (int)fn;
  float k = 0.f, kn = 0.f, fm0 = 0.f;
  float g[NS][3];  // far weights of the layer before, at n - 1, n, n + 1
  bool Xp = false;
  Raw va[NP], vd[NP];  // the outer positions, kept where a layer does not read them (weight 0)
#pragma unroll
  for (int p = 0; p < NP; ++p) va[p] = vd[p] = Raw(0);
#pragma unroll
  for (int q = 0; q < NS; ++q) {
    g[q][0] = g[q][1] = g[q][2] = 0.f;
#pragma unroll
    for (int p = 0; p < NP; ++p) S[q][p] = 0.f;
  }
  Raw vb[NP], vc[NP];
  auto load_row = [&](bool first, bool last) {
    const unsigned r = (unsigned)min(max(im, 0), W.nM - 1) * W.dM;
    auto col = [&](int n) { return r + (unsigned)min(max(n, 0), W.nN - 1) * W.dN; };
    const unsigned oa = col(in - W.sN), ob = col(in), oc = col(in + W.sN), od = col(in + 2 * W.sN);
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      vb[p] = ldraw<VT>(base + (ob + yoff[p]));
      vc[p] = ldraw<VT>(base + (oc + yoff[p]));
      ldraw_if<VT>(va[p], base + (oa + yoff[p]), first);
      ldraw_if<VT>(vd[p], base + (od + yoff[p]), last);
    }
  };
  auto add_row = [&](const float (&w)[NS][4]) {
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const float a = cvt<VT>(va[p]), b = cvt<VT>(vb[p]), c = cvt<VT>(vc[p]), d = cvt<VT>(vd[p]);
#pragma unroll
      for (int q = 0; q < NS; ++q) {
        S[q][p] = fmaf(b, w[q][1], S[q][p]);
        S[q][p] = fmaf(c, w[q][2], S[q][p]);
        S[q][p] = fmaf(a, w[q][0], S[q][p]);
        S[q][p] = fmaf(d, w[q][3], S[q][p]);
      }
    }
  };
#pragma unroll 1
  for (int guard = 0; guard < 1 << 20; ++guard) {
    const float nMs = __fmaf_rn(k, A.isM, nM0), nNs = __fmaf_rn(kn, A.isN, nN0);
    const bool X = nNs <= nMs;
    load_row(Xp, X);  // in flight during the weights' arithmetic
    const float tL = fminf(nMs, Mt);
    const float2 f = ceil2(fminf(nNs, tL), tL);
    const float MA = f.x - fm0, MB = f.y - f.x;
    const float sA = fm0 + f.x, sB = f.x + f.y;
    const float aA = fmaf(sA, A.hN, relN), aB = fmaf(sB, A.hN, relN - 1.f);
    const float cA = fmaf(sA, A.hM, relM), cB = fmaf(sB, A.hM, relM);
    const float MaA = MA * aA, MaB = MB * aB, McA = MA * cA, McB = MB * cB;
    const float tA = MA * fmaf(aA, cA, fmaf(MA * MA, A.g, -A.g)), tB = MB * fmaf(aB, cB, fmaf(MB * MB, A.g, -A.g));
    float n[NS][3], far[NS][3];  // near and far weights at n, n + 1, n + 2
    const float uA = McA - tA, uB = McB - tB;
    n[0][0] = (MA - MaA) - uA;
    n[0][1] = (MaA - tA) + ((MB - MaB) - uB);
    n[0][2] = MaB - tB;
    far[0][0] = uA;
    far[0][1] = tA + uB;
    far[0][2] = tB;
    if constexpr (SHEAR) {
      const float vA = MA - McA, vB = MB - McB, wA = MA - MaA, wB = MB - MaB;
      n[1][0] = -vA, n[1][1] = vA - vB, n[1][2] = vB;
      far[1][0] = -McA, far[1][1] = McA - McB, far[1][2] = McB;
      n[2][0] = -wA, n[2][1] = -(MaA + wB), n[2][2] = -MaB;
      far[2][0] = wA, far[2][1] = MaA + wB, far[2][2] = MaB;
      n[3][0] = MA, n[3][1] = MB - MA, n[3][2] = -MB;
      far[3][0] = -MA, far[3][1] = MA - MB, far[3][2] = MB;
    }
    float w[NS][4];
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      w[q][0] = g[q][0];
      w[q][1] = g[q][1] + n[q][0];
      w[q][2] = g[q][2] + n[q][1];
      w[q][3] = n[q][2];
    }
    add_row(w);
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      g[q][0] = X ? far[q][0] : 0.f;
      g[q][1] = X ? far[q][1] : far[q][0];
      g[q][2] = X ? far[q][2] : far[q][1];
    }
    fm0 = f.y;
    k += 1.f;
    relM -= 1.f;
    im += W.sM;
    if (X) {
      relN -= 1.f;
      kn += 1.f;
      in += W.sN;
    }
    Xp = X;
    if (fm0 >= Mt) break;
  }
  float w[NS][4];
#pragma unroll
  for (int q = 0; q < NS; ++q) {
    w[q][0] = g[q][0], w[q][1] = g[q][1], w[q][2] = g[q][2];
    w[q][3] = 0.f;
  }
  load_row(Xp, false);
  add_row(w);
}

// One thread's line of 2 G sub-rays (kept in local memory, read a few times
// per walk).
template <int G>
struct PlaneLine {
  static constexpr int N = 2 * G, NP = G + 2;
  float3 s[N];           // starts
  float tin[N], tout[N];
  float b[N], source[N]; // weight of the upper plane, and the sample at the start
  int cell[N];           // lower plane, relative to the line's first
  unsigned in;           // sub-rays that meet the volume
  // x, y: first pixel; the lane's sub-row along v (u with swap)
  template <int VT>
  __device__ __forceinline__ void init(const KConst& c, const void* vol, int x, int y, int swap, bool sources,
                                       unsigned (&yoff)[NP]) {
    in = 0;
    int p0 = 1 << 30;
    const float sub = (threadIdx.x & 1) ? 0.75f : 0.25f;
    const Cell<VT> C{vol, (int)c.dim.x, (int)c.dim.y, (int)c.dim.z, (long)c.dim.x, (long)c.dim.x * (long)c.dim.y};
#pragma unroll 1
    for (int g = 0; g < N; ++g) {
      const float step = (float)(g >> 1) + ((g & 1) ? 0.75f : 0.25f);
      s[g] = swap ? ray_src(c, (float)x + sub, (float)y + step) : ray_src(c, (float)x + step, (float)y + sub);
      hit(s[g], c.n, c.bbMin, c.bbMax, tin[g], tout[g]);
      if (tout[g] - tin[g] > 0.0f) {
        in |= 1u << g;
        if (sources) {
          const float3 q = interp_coord(c, s[g]);
          source[g] = trilinear<VT>(C, q.x, q.y, q.z);
        }
      }
      // y is constant along a ray (PlaneRay checks it)
      const float t = (in >> g & 1u) ? tin[g] : 0.0f;
      const float q = interp_coord(c, ray_point(c, s[g], t)).y;
      const float fy = floorf(q);
      b[g] = q - fy;
      cell[g] = (int)fy;
      p0 = min(p0, cell[g]);
    }
#pragma unroll 1
    for (int g = 0; g < N; ++g) cell[g] -= p0;
    const int ny = (int)c.dim.y, nx = (int)c.dim.x;
    constexpr unsigned ES = VT == ESB_VOXEL_F32 ? 4 : 2;
#pragma unroll
    for (int p = 0; p < NP; ++p) yoff[p] = (unsigned)min(max(p0 + p, 0), ny - 1) * (unsigned)nx * ES;
  }
};

// Samples of one sub-ray over [t0, t1]: their count, the position of the
// first, and whether they can join the line's walk.
struct PlaneRay {
  int J;
  float3 q, dq;
  bool ok;
  __device__ __forceinline__ PlaneRay(const KConst& c, const AxisStep& A, float3 s, float t0, float t1, float b) {
    float step;
    J = progression(t0, t1, c.vs.x * 0.15f, step, ok);
    q = interp_coord(c, ray_point(c, s, t0));
    dq = interp_step(c, step);
    const float fy = floorf(q.y);
    ok = ok && step == A.step && fabsf(dq.y) * (float)J < 1e-5f && fy == floorf(qpos(q.y, J - 1, dq.y)) &&
         fabsf((q.y - fy) - b) < 1e-4f;
  }
};

// Sums v[] of the line's sub-rays, each over its [tin, tout] cut to [lo, hi]
// (0 for those outside). slab: the first sample is the one at the ray's
// start; else run `seg` of `segs` of the samples (axis_ray_sum).
template <int VT, int G, bool SHEAR>
__device__ __forceinline__ void line_sums(const KConst& c, const AxisStep& A, const PlaneWalk& W, int zmaj,
                                          const void* vol, const PlaneLine<G>& L, const unsigned (&yoff)[G + 2],
                                          bool slab, float lo, float hi, int seg, int segs, float* v) {
  constexpr int N = 2 * G, NP = G + 2, NS = SHEAR ? 4 : 1;
  float S[NS][NP];
#pragma unroll
  for (int q = 0; q < NS; ++q)
#pragma unroll
    for (int p = 0; p < NP; ++p) S[q][p] = 0.f;
  // the middle ray
  const float m0 = fmaxf(L.tin[G], lo), m1 = fminf(L.tout[G], hi);
  bool mid = (L.in >> G & 1u) && m0 <= m1;
  float bm = 0.f, bn = 0.f;
  int Jm = 0;
  if (mid) {
    const PlaneRay R(c, A, L.s[G], m0, m1, L.b[G]);
    mid = R.ok;
    Jm = R.J;
    bm = zmaj ? R.q.z : R.q.x;
    bn = zmaj ? R.q.x : R.q.z;
  }
  const int j0 = slab ? 1 : run_start(Jm, seg, segs), j1 = slab ? Jm : run_start(Jm, seg + 1, segs);
  if (mid && j0 < j1)
    plane_sums<VT, NP, SHEAR>(A, W, vol, yoff, W.sM > 0 ? bm : -bm, W.sN > 0 ? bn : -bn, j0, j1, S);
  float P[NS][NP];  // (indexed by a ray's planes: local memory)
#pragma unroll
  for (int q = 0; q < NS; ++q)
#pragma unroll
    for (int p = 0; p < NP; ++p) P[q][p] = S[q][p];
#pragma unroll 1
  for (int g = 0; g < N; ++g) {
    v[g] = 0.f;
    if (!(L.in >> g & 1u)) continue;
    const float t0 = fmaxf(L.tin[g], lo), t1 = fminf(L.tout[g], hi);
    if (!(t0 <= t1)) continue;
    const PlaneRay R(c, A, L.s[g], t0, t1, L.b[g]);
    const float f = ((zmaj ? R.q.z : R.q.x) - bm) * (float)W.sM, e = ((zmaj ? R.q.x : R.q.z) - bn) * (float)W.sN;
    const bool joins = mid && R.ok && L.cell[g] <= G && abs(R.J - Jm) <= 1 &&
                       (SHEAR ? fabsf(e) <= kMaxShear && fabsf(f) <= kMaxShear : e == 0.f && f == 0.f);
    if (!joins) {
      if (seg == 0) v[g] = other_ray_sum<VT>(&c, vol, L.s[g], t0, t1, slab);
      continue;
    }
    float sum[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int p = L.cell[g] + h;
      sum[h] = P[0][p];
      if constexpr (SHEAR) sum[h] = fmaf(e * f, P[3][p], fmaf(e, P[1][p], fmaf(f, P[2][p], sum[h])));
    }
    float r = fmaf(L.b[g], sum[1], (1.0f - L.b[g]) * sum[0]);
    if (R.J != Jm && seg == segs - 1) {  // one sample more or less than the middle ray
      const int j = min(R.J, Jm);
      const Cell<VT> C{vol, (int)c.dim.x, (int)c.dim.y, (int)c.dim.z, (long)c.dim.x, (long)c.dim.x * (long)c.dim.y};
      const float last = trilinear<VT>(C, qpos(R.q.x, j, R.dq.x), qpos(R.q.y, j, R.dq.y), qpos(R.q.z, j, R.dq.z));
      if (j >= (slab ? 1 : 0)) r += R.J > Jm ? last : -last;
    }
    v[g] = slab ? r + L.source[g] : r;
  }
}

// First pixel of the line of G that holds pixel i: lines start at multiples
// of G of the detector, whatever the launched region, so that a pixel is
// summed with the same middle ray in every region.
__host__ __device__ __forceinline__ int line_start(int i, int G) { return i & ~(G - 1); }

// Pixels of a thread: G along u (v with swap) from x, y; a lane pair shares
// them, one sub-row each, and `segs` warps the same. The region's pixels
// among them (`inside`) are written.
template <int G>
struct PlanePixel {
  int x, y, seg, x0, y0, x1, y1;
  bool active;
  __device__ __forceinline__ PlanePixel(int swap, int segs, int x0_, int y0_, int x1_, int y1_)
      : x0(x0_), y0(y0_), x1(x1_), y1(y1_) {
    const int lane = threadIdx.x & 31;
    const int w = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)), across = G * (w / segs);
    seg = w % segs;
    const int along = (int)blockIdx.y * 16 + (lane >> 1);
    x = swap ? x0 + along : line_start(x0, G) + across;
    y = swap ? line_start(y0, G) + across : y0 + along;
    active = x < x1 && y < y1;
  }
  __device__ __forceinline__ bool inside(int px, int py) const { return px >= x0 && py >= y0 && px < x1 && py < y1; }
};

// Sum of pixel i's 4 sub-rays in the reference's order, valid in even lanes.
__device__ __forceinline__ float pixel_sum(const float* v, int i, int swap) {
  const float a = v[2 * i], b = v[2 * i + 1];
  const float c = __shfl_down_sync(0xffffffffu, a, 1), d = __shfl_down_sync(0xffffffffu, b, 1);
  return swap ? __fadd_rn(__fadd_rn(__fadd_rn(a, b), c), d) : __fadd_rn(__fadd_rn(__fadd_rn(a, c), b), d);
}

template <int VT, int G, bool SHEAR>
__global__ void __launch_bounds__(128) k_project_planes(const __grid_constant__ KConst c,
                                                        const __grid_constant__ AxisStep A,
                                                        const __grid_constant__ PlaneWalk W, int zmaj, int swap, int segs,
                                                        const void* __restrict__ vol, float* __restrict__ proj,
                                                        float* __restrict__ dist, size_t pitchE, int x0, int y0,
                                                        int x1, int y1) {
  const PlanePixel<G> P(swap, segs, x0, y0, x1, y1);
  PlaneLine<G> L;
  unsigned yoff[G + 2];
  float v[2 * G];
  L.in = 0;
  if (P.active) {
    L.template init<VT>(c, vol, P.x, P.y, swap, false, yoff);
    line_sums<VT, G, SHEAR>(c, A, W, zmaj, vol, L, yoff, false, -FLT_MAX, FLT_MAX, P.seg, segs, v);
  } else {
#pragma unroll
    for (int g = 0; g < 2 * G; ++g) v[g] = 0.0f;
  }
  sum_runs(v, segs);
#pragma unroll 1
  for (int i = 0; i < G; ++i) {
    float n[2], d[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int g = 2 * i + h;
      const bool in = (L.in >> g & 1u) != 0;
      n[h] = in ? 1.0f : 0.0f;
      d[h] = in ? L.tout[g] - L.tin[g] : 0.0f;
      if (!in) v[g] = 0.0f;
    }
    const float sum = pixel_sum(v, i, swap), gx = pixel_sum(n, 0, swap), gz = pixel_sum(d, 0, swap);
    const int x = P.x + (swap ? 0 : i), y = P.y + (swap ? i : 0);
    if (P.active && P.seg == 0 && !(threadIdx.x & 1) && P.inside(x, y)) {
      const size_t o = (size_t)y * pitchE + x;
      proj[o] += sum * c.vs.x * 0.15f * 0.25f;
      dist[o] = fmaxf(0.0f, gz / gx);
    }
  }
}

template <int VT, int G, bool SHEAR>
__global__ void __launch_bounds__(128) k_slicer_planes(const __grid_constant__ KConst c,
                                                       const __grid_constant__ AxisStep A,
                                                       const __grid_constant__ PlaneWalk W, int zmaj, int swap,
                                                       const void* __restrict__ vol, float* __restrict__ imgs,
                                                       size_t img_stride, size_t pitchE,
                                                       const __grid_constant__ SlabTable slabs, int clear, int x0,
                                                       int y0, int x1, int y1) {
  const PlanePixel<G> P(swap, 1, x0, y0, x1, y1);
  PlaneLine<G> L;
  unsigned yoff[G + 2];
  L.in = 0;
  if (P.active) L.template init<VT>(c, vol, P.x, P.y, swap, true, yoff);
  // slabs met by each pixel's rays, and the union over the warp's
  int klo[G], khi[G], wlo = ESB_MAX_SLABS, whi = -1;
#pragma unroll
  for (int i = 0; i < G; ++i) {
    klo[i] = ESB_MAX_SLABS;
    khi[i] = -1;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (!(L.in >> (2 * i + h) & 1u)) continue;
      const float t0 = L.tin[2 * i + h], t1 = L.tout[2 * i + h];
      for (int k = 0; k < slabs.count; ++k) {
        if (fmaxf(t0, slabs.bound[k]) <= fminf(t1, slabs.bound[k + 1])) {
          klo[i] = min(klo[i], k);
          khi[i] = max(khi[i], k);
        }
      }
    }
    klo[i] = min(klo[i], __shfl_xor_sync(0xffffffffu, klo[i], 1));
    khi[i] = max(khi[i], __shfl_xor_sync(0xffffffffu, khi[i], 1));
    wlo = min(wlo, klo[i]);
    whi = max(whi, khi[i]);
  }
  for (int o = 2; o <= 16; o <<= 1) {
    wlo = min(wlo, __shfl_xor_sync(0xffffffffu, wlo, o));
    whi = max(whi, __shfl_xor_sync(0xffffffffu, whi, o));
  }
  const bool writer = P.active && !(threadIdx.x & 1);
  int ka, kb;
  slab_part(wlo, whi, ka, kb);
  for (int k = ka; k < kb; ++k) {
    float v[2 * G];
    if (L.in) {
      line_sums<VT, G, SHEAR>(c, A, W, zmaj, vol, L, yoff, true, slabs.bound[k], slabs.bound[k + 1], 0, 1, v);
    } else {
#pragma unroll
      for (int g = 0; g < 2 * G; ++g) v[g] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < G; ++i) {
      const float sum = pixel_sum(v, i, swap);
      const int x = P.x + (swap ? 0 : i), y = P.y + (swap ? i : 0);
      if (writer && P.inside(x, y) && k >= klo[i] && k <= khi[i])
        imgs[(size_t)k * img_stride + (size_t)y * pitchE + x] = sum * c.vs.x * 0.15f * 0.25f;
    }
  }
  if (clear && blockIdx.z == 0 && writer) {
#pragma unroll
    for (int i = 0; i < G; ++i) {
      const int x = P.x + (swap ? 0 : i), y = P.y + (swap ? i : 0);
      if (P.inside(x, y)) clear_slabs(imgs + (size_t)y * pitchE + x, img_stride, slabs.count, klo[i], khi[i]);
    }
  }
}

// Parts that each ray is cut into, up to max_parts, for `warps` warps to
// become `full`, the warps that the GPU holds at once: a small launch waits
// for the loads of one layer after the other (64 x 64 x 32: 15.4 us a
// projection with whole rays, 9.6 in 4 runs).
int parts_for(double warps, double full, int max_parts) {
  return std::max(1, std::min(max_parts, (int)(full / warps + 0.5)));
}

// Runs that a ray's samples may be cut into: at least 8 layers in each, a
// power of two up to `most`.
int max_runs(const KConst& c, bool zmaj, int most) {
  int n = 1;
  while (2 * n <= most && 16 * n <= (int)(zmaj ? c.dim.z : c.dim.x)) n *= 2;
  return n;
}

// The plane kernels' launch: G pixels per thread (0: not taken), whether the
// line's rays differ in y only. Chosen by the detector (w x h), not by the
// region of it that is launched: a region's pixels are the whole detector's
// bit for bit.
struct PlaneLaunch {
  int G = 0, shear = 0, swap = 0, zmaj = 0;
  AxisStep A;
  PlaneWalk W;
  // Warps of g pixels per thread that a region of w x h takes.
  double warps(int w, int h, int g) const {
    const int along = swap ? w : h, across = swap ? h : w;
    return (double)((across + g - 1) / g) * ((along + 15) / 16);
  }
  // Parts, runs or slabs, for them to fill the GPU.
  int parts(int w, int h, int max_parts) const { return parts_for(warps(w, h, G), 16.0 * kSMs, max_parts); }
  // runs: how often a ray's samples may be cut into runs
  PlaneLaunch(const KConst& c, int vt, int w, int h, int runs) {
    bool z;
    int sm, sn;
    A = axis_step(c, z, sm, sn);
    if (!axis_projection(c) || !(A.step > 0.0f) || (double)c.dim.x * c.dim.y * c.dim.z >= 1073741824.0) return;
    swap = axis_swap(c);
    zmaj = z ? 1 : 0;
    // voxels that half a pixel along the line moves a ray in x, y, z
    const float au = swap ? c.aniso[1] : c.aniso[0], av = swap ? c.aniso[4] : c.aniso[3];
    const float ex = 0.5f * fabsf(au * c.u.x + av * c.v.x) * c.bbRcp.x * c.dim.x;
    const float ey = 0.5f * fabsf(au * c.u.y + av * c.v.y) * c.bbRcp.y * c.dim.y;
    const float ez = 0.5f * fabsf(au * c.u.z + av * c.v.z) * c.bbRcp.z * c.dim.z;
    shear = ex > 0.f || ez > 0.f ? 1 : 0;
    for (int g = 4; g >= 2 && !G; g -= 2) {
      // the offset of the line's outermost ray, taken at its start or along
      // the ray to the volume's face, against its bounds (above), and the
      // line's planes
      const float offset = (float)g * (ex + ez);
      const bool small = !shear || (offset <= kMaxShear && 4.0f * offset <= A.dN);
      const bool planes = (float)(2 * g - 1) * ey < (float)g - 0.05f;
      // 2 pixels per thread from 2 warps per scheduler on, 4 from 4, runs
      // counted. Measured without runs: 128 warps of 2 pixels 25 us against
      // the axis walk's 15, 2048 warps 113 against 178, 1024 warps of 4
      // pixels 141, and with 4 runs 78. Slabs do not count: they are few
      // layers each, and 1024 warps of 4 pixels with their slabs spread took
      // 105 us where 2048 of 2 pixels take 72.
      const bool enough = warps(w, h, g) * runs >= 4.0 * kSMs * g;
      if (small && planes && enough) G = g;
    }
    const unsigned es = vt == ESB_VOXEL_F32 ? 4 : 2, sz = es * (unsigned)c.dim.x * (unsigned)c.dim.y;
    W.sM = sm;
    W.sN = sn;
    W.nM = (int)(z ? c.dim.z : c.dim.x);
    W.nN = (int)(z ? c.dim.x : c.dim.z);
    W.dM = z ? sz : es;
    W.dN = z ? es : sz;
  }
};

// Runs of a ray's samples in k_project_axis, by the whole detector's warps of
// one pixel across: they, and with them the order of a ray's sum, depend
// neither on the block shape nor on the region.
int axis_runs(const KConst& c, bool zmaj, int pw, int ph) {
  const dim3 warps = axis_grid(axis_swap(c), 1, pw, ph);
  return max_runs(c, zmaj, parts_for((double)warps.x * warps.y, 32.0 * kSMs, 8));
}

// Volumes of 2^32 voxels or more take 64-bit element offsets in the walk.
bool big_volume(const KConst& c) { return (double)c.dim.x * c.dim.y * c.dim.z > 4294967295.0; }

}  // namespace

// Whether nw (warps per block) makes a difference to launch_slicer_fused and
// launch_project_fast (mode 0): not to lines of rays, rays cut into runs and
// volumes with 64-bit offsets.
bool slicer_takes_nw(const KConst& c, int vt, int pw, int ph) {
  return axis_projection(c) ? PlaneLaunch(c, vt, pw, ph, 1).G == 0 : !big_volume(c);
}
bool project_takes_nw(const KConst& c, int vt, int pw, int ph) {
  if (!axis_projection(c)) return !big_volume(c);
  bool zmaj;
  int sm, sn;
  axis_step(c, zmaj, sm, sn);
  return PlaneLaunch(c, vt, pw, ph, max_runs(c, zmaj, 4)).G == 0 && axis_runs(c, zmaj, pw, ph) == 1;
}

// nw: warps per block (2, 4 or 8; 64-bit-offset volumes always take 4).

// One launch of an axis kernel instance per beam orientation.
#define ESB_AXIS_ORIENT(KER, VT, OFF, GRD, BLK, ST, ...)                         \
  do {                                                                          \
    bool zmaj_;                                                                 \
    int sm_, sn_;                                                               \
    const AxisStep A_ = axis_step(c, zmaj_, sm_, sn_);                           \
    const int o_ = (zmaj_ ? 4 : 0) + (sm_ > 0 ? 2 : 0) + (sn_ > 0 ? 1 : 0);     \
    switch (o_) {                                                               \
      case 0: KER<VT, false, -1, -1, OFF><<<GRD, BLK, 0, ST>>>(c, A_, __VA_ARGS__); break;  \
      case 1: KER<VT, false, -1, 1, OFF><<<GRD, BLK, 0, ST>>>(c, A_, __VA_ARGS__); break;   \
      case 2: KER<VT, false, 1, -1, OFF><<<GRD, BLK, 0, ST>>>(c, A_, __VA_ARGS__); break;   \
      case 3: KER<VT, false, 1, 1, OFF><<<GRD, BLK, 0, ST>>>(c, A_, __VA_ARGS__); break;    \
      case 4: KER<VT, true, -1, -1, OFF><<<GRD, BLK, 0, ST>>>(c, A_, __VA_ARGS__); break;   \
      case 5: KER<VT, true, -1, 1, OFF><<<GRD, BLK, 0, ST>>>(c, A_, __VA_ARGS__); break;    \
      case 6: KER<VT, true, 1, -1, OFF><<<GRD, BLK, 0, ST>>>(c, A_, __VA_ARGS__); break;    \
      default: KER<VT, true, 1, 1, OFF><<<GRD, BLK, 0, ST>>>(c, A_, __VA_ARGS__); break;    \
    }                                                                           \
  } while (0)

// A launch of a plane kernel (ESB_PLANES), 4 warps per block.
#define ESB_PLANES_SH(VT, GG)              \
  do {                                     \
    if (L.shear) ESB_PLANES(VT, GG, true); \
    else ESB_PLANES(VT, GG, false);        \
  } while (0)
#define ESB_PLANES_VT(VT)                  \
  do {                                     \
    if (L.G == 4) ESB_PLANES_SH(VT, 4);    \
    else ESB_PLANES_SH(VT, 2);             \
  } while (0)
#define ESB_PLANES_LAUNCH()                                                                          \
  do {                                                                                               \
    const int along = L.swap ? x1 - x0 : y1 - y0;                                                     \
    const int across = L.swap ? y1 - line_start(y0, L.G) : x1 - line_start(x0, L.G);                  \
    const int cols = 4 / segs * L.G; /* across a block of 4 warps */                                  \
    const dim3 blk(128), grd((across + cols - 1) / cols, (along + 15) / 16, slab_parts);              \
    if (vt == ESB_VOXEL_F32) ESB_PLANES_VT(ESB_VOXEL_F32);                                           \
    else if (vt == ESB_VOXEL_F16) ESB_PLANES_VT(ESB_VOXEL_F16);                                      \
    else ESB_PLANES_VT(ESB_VOXEL_BF16);                                                              \
    ESB_COUNT_LAUNCH();                                                                              \
    return cudaGetLastError();                                                                       \
  } while (0)

// Volumes below 4 GiB take 32-bit byte offsets in the axis walk (an address
// is one addition instead of a 64-bit one and its carries).
#define ESB_AXIS_LAUNCH(KER, GRD, BLK, ST, ...)                                                                \
  do {                                                                                                        \
    const double bytes_ = (double)c.dim.x * c.dim.y * c.dim.z * (vt == ESB_VOXEL_F32 ? 4.0 : 2.0);            \
    if (bytes_ < 4294967296.0) {                                                                              \
      if (vt == ESB_VOXEL_F32) ESB_AXIS_ORIENT(KER, ESB_VOXEL_F32, unsigned, GRD, BLK, ST, __VA_ARGS__);      \
      else if (vt == ESB_VOXEL_F16) ESB_AXIS_ORIENT(KER, ESB_VOXEL_F16, unsigned, GRD, BLK, ST, __VA_ARGS__); \
      else ESB_AXIS_ORIENT(KER, ESB_VOXEL_BF16, unsigned, GRD, BLK, ST, __VA_ARGS__);                         \
    } else {                                                                                                  \
      if (vt == ESB_VOXEL_F32) ESB_AXIS_ORIENT(KER, ESB_VOXEL_F32, size_t, GRD, BLK, ST, __VA_ARGS__);        \
      else if (vt == ESB_VOXEL_F16) ESB_AXIS_ORIENT(KER, ESB_VOXEL_F16, size_t, GRD, BLK, ST, __VA_ARGS__);   \
      else ESB_AXIS_ORIENT(KER, ESB_VOXEL_BF16, size_t, GRD, BLK, ST, __VA_ARGS__);                           \
    }                                                                                                         \
  } while (0)

cudaError_t launch_slicer_fused(const KConst& c, const void* vol, int vt, float* imgs, size_t img_stride,
                                size_t pitchE, const SlabTable& slabs, int clear, int pw, int ph, int x0, int y0,
                                int x1, int y1, cudaStream_t st, int nw) {
  if (x1 <= x0 || y1 <= y0 || slabs.count <= 0) return cudaSuccess;
  const PlaneLaunch L(c, vt, pw, ph, 1);
  if (L.G) {
    const int segs = 1, slab_parts = L.parts(x1 - x0, y1 - y0, slabs.count);
#define ESB_PLANES(VT, GG, SH)                                                                                        \
  k_slicer_planes<VT, GG, SH><<<grd, blk, 0, st>>>(c, L.A, L.W, L.zmaj, L.swap, vol, imgs, img_stride, pitchE, \
                                                           slabs, clear, x0, y0, x1, y1)
    ESB_PLANES_LAUNCH();
#undef ESB_PLANES
  }
  if (axis_projection(c)) {  // the axis walk, one sub-ray per thread
    if (nw != 2 && nw != 8) nw = 4;
    const int swap = axis_swap(c);
    dim3 blk(32 * nw), grd = axis_grid(swap, nw, x1 - x0, y1 - y0);
    grd.z = parts_for((double)grd.x * grd.y * nw, 32.0 * kSMs, slabs.count);
    ESB_AXIS_LAUNCH(k_slicer_axis, grd, blk, st, vol, imgs, img_stride, pitchE, slabs, clear, swap, x0, y0, x1, y1);
    ESB_COUNT_LAUNCH();
    return cudaGetLastError();
  }
  const bool big = big_volume(c);
  if (big || (nw != 2 && nw != 8)) nw = 4;
  dim3 blk(32 * nw), grd((x1 - x0 + nw - 1) / nw, (y1 - y0 + 7) / 8);
#define ESB_LAUNCH(VT, OFF, NW) \
  k_slicer_fused<VT, OFF, NW><<<grd, blk, 0, st>>>(c, vol, imgs, img_stride, pitchE, slabs, clear, x0, y0, x1, y1)
#define ESB_LAUNCH_VT(OFF, NW)                                  \
  do {                                                          \
    if (vt == ESB_VOXEL_F32) ESB_LAUNCH(ESB_VOXEL_F32, OFF, NW);   \
    else if (vt == ESB_VOXEL_F16) ESB_LAUNCH(ESB_VOXEL_F16, OFF, NW); \
    else ESB_LAUNCH(ESB_VOXEL_BF16, OFF, NW);                   \
  } while (0)
  if (big) ESB_LAUNCH_VT(unsigned long long, 4);
  else if (nw == 2) ESB_LAUNCH_VT(unsigned, 2);
  else if (nw == 8) ESB_LAUNCH_VT(unsigned, 8);
  else ESB_LAUNCH_VT(unsigned, 4);
#undef ESB_LAUNCH_VT
#undef ESB_LAUNCH
  ESB_COUNT_LAUNCH();
  return cudaGetLastError();
}

cudaError_t launch_project_fast(const KConst& c, const void* vol, int vt, int mode, float* proj, float* dist,
                                size_t pitchE, float tmin, float tmax, int pw, int ph, int x0, int y0, int x1, int y1,
                                cudaStream_t st, int nw) {
  if (x1 <= x0 || y1 <= y0) return cudaSuccess;
  bool zmaj;
  int sm, sn;
  axis_step(c, zmaj, sm, sn);
  const PlaneLaunch L(c, vt, pw, ph, max_runs(c, zmaj, 4));
  if (mode == 0 && L.G) {
    const int segs = max_runs(c, zmaj, L.parts(pw, ph, 4)), slab_parts = 1;
#define ESB_PLANES(VT, GG, SH) \
  k_project_planes<VT, GG, SH><<<grd, blk, 0, st>>>(c, L.A, L.W, L.zmaj, L.swap, segs, vol, proj, dist, pitchE, x0, y0, x1, y1)
    ESB_PLANES_LAUNCH();
#undef ESB_PLANES
  }
  if (mode == 0 && axis_projection(c)) {  // the axis walk, one sub-ray per thread
    if (nw != 2 && nw != 8) nw = 4;
    const int swap = axis_swap(c);
    dim3 grd = axis_grid(swap, nw, x1 - x0, y1 - y0);
    const int segs = axis_runs(c, zmaj, pw, ph);
    if (segs > 1) {
      nw = 8;
      grd = axis_grid(swap, nw / segs, x1 - x0, y1 - y0);
    }
    const dim3 blk(32 * nw);
    ESB_AXIS_LAUNCH(k_project_axis, grd, blk, st, vol, proj, dist, pitchE, swap, segs, x0, y0, x1, y1);
    ESB_COUNT_LAUNCH();
    return cudaGetLastError();
  }
  const bool big = big_volume(c);
  if (big || (nw != 2 && nw != 8)) nw = 4;
  dim3 blk(32 * nw), grd((x1 - x0 + nw - 1) / nw, (y1 - y0 + 7) / 8);
#define ESB_LAUNCH(VT, M, OFF, NW) \
  k_project_fast<VT, M, OFF, NW><<<grd, blk, 0, st>>>(c, vol, proj, dist, pitchE, tmin, tmax, x0, y0, x1, y1)
#define ESB_LAUNCH_VT(M, OFF, NW)                                  \
  do {                                                             \
    if (vt == ESB_VOXEL_F32) ESB_LAUNCH(ESB_VOXEL_F32, M, OFF, NW);   \
    else if (vt == ESB_VOXEL_F16) ESB_LAUNCH(ESB_VOXEL_F16, M, OFF, NW); \
    else ESB_LAUNCH(ESB_VOXEL_BF16, M, OFF, NW);                   \
  } while (0)
#define ESB_LAUNCH_NW(M)                                      \
  do {                                                        \
    if (big) ESB_LAUNCH_VT(M, unsigned long long, 4);          \
    else if (nw == 2) ESB_LAUNCH_VT(M, unsigned, 2);           \
    else if (nw == 8) ESB_LAUNCH_VT(M, unsigned, 8);           \
    else ESB_LAUNCH_VT(M, unsigned, 4);                        \
  } while (0)
  if (mode == 0) ESB_LAUNCH_NW(0);
  else ESB_LAUNCH_NW(1);
#undef ESB_LAUNCH_NW
#undef ESB_LAUNCH_VT
#undef ESB_LAUNCH
  ESB_COUNT_LAUNCH();
  return cudaGetLastError();
}

}  // namespace esb
