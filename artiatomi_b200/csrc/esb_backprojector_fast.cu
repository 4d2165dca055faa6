// Ray-length-normalised back-projection by per-voxel shadows ("fast").
//
// The reference kernel (BackProjectionSquareOS.cu:263-782) bounds the
// 5x1x1-voxel macro cell of a 4-voxel quad on the detector, walks the
// sub-pixel samples of that rectangle (pixel += 1/OS from the rectangle's
// clamped integer corner) and intersects each sample's ray with each of the
// 4 voxels. Most of those tests miss, and each hit is computed from a ray
// origin 1e5 units away, so float rounding is ~1e-2 on a chord of ~1.
//
// This kernel computes the same macro-cell rectangle and walks the same
// sub-pixel recurrence. For each voxel it visits only the samples inside
// that voxel's own shadow, and computes the chord in voxel-local coordinates:
// the sample's ray is c + d + tau*n, with d the sample's in-plane offset from
// the projected voxel centre c. The result is the reference's
// sum(sample*chord)/sum(chord) over the reference's samples, with exact
// rather than noisy chords.
//
// CTF mode: the reference launches the back-projection once per defocus
// slab, each launch re-reading the whole volume, and updates a quad in the
// slab that holds its first corner's depth (:365-369). Here one launch
// covers all slabs of a projection: each quad looks its slab up in the
// table of slab boundaries (the reference's float recurrence
// ray += thickness) and reads that slab's filtered image.
#include <float.h>

#include "esb_bp_core.cuh"

namespace esb {

namespace {

using namespace bpcore;

template <int VT>
__global__ void __launch_bounds__(128) k_bp_fast(KConst k, BpGeom g, void* __restrict__ vol,
                                                 const float* __restrict__ imgs, size_t img_stride, SlabTable slabs,
                                                 int pw, int ph, size_t pitchE, float lambda, int os, float inv,
                                                 float distMin, float distMax, int linear, int transposed,
                                                 const float2* __restrict__ ups, size_t up_stride) {
  const int q = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int y = (int)(blockIdx.y * blockDim.y + threadIdx.y);
  const int z = (int)blockIdx.z;
  const int ny = (int)k.dim.y, nz = (int)k.dim.z;
  if (q >= k.dimXQuarter || y >= ny || z >= nz) return;
  const int x = 4 * q;
  float depth;
  int pbx, pby, pbz, pbw;
  macro_footprint(k, x, y, z, pw, ph, depth, pbx, pby, pbz, pbw);
  const float* img = imgs;
  const float2* up = ups;
  if (slabs.count > 0) {  // fused CTF slabs
    if (!(depth >= slabs.bound[0] && depth < slabs.bound[slabs.count])) return;
    int s = 0;
    while (s + 1 < slabs.count && depth >= slabs.bound[s + 1]) ++s;
    img = imgs + (size_t)s * img_stride;
    if (up) up += (size_t)s * up_stride;
  } else if (!(depth >= distMin && depth < distMax)) {
    return;
  }
  const long base = ((long)z * ny + y) * (long)k.dim.x + x;
  float acc[4], dacc[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    voxel_sums(k, g, img, pw, ph, pitchE, os, inv, linear != 0, transposed != 0, x + i, y, z, pbx, pby, pbz, pbw,
               acc[i], dacc[i], up, ph * os);
  if (VT == ESB_VOXEL_F32 && (((uintptr_t)((float*)vol + base)) & 15) == 0) {
    float4 v = *((float4*)((float*)vol + base));
    if (dacc[0] > 0.f) v.x += lambda * acc[0] / dacc[0];
    if (dacc[1] > 0.f) v.y += lambda * acc[1] / dacc[1];
    if (dacc[2] > 0.f) v.z += lambda * acc[2] / dacc[2];
    if (dacc[3] > 0.f) v.w += lambda * acc[3] / dacc[3];
    *((float4*)((float*)vol + base)) = v;
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (dacc[i] > 0.f) Voxel<VT>::store(vol, base + i, Voxel<VT>::loadrw(vol, base + i) + lambda * acc[i] / dacc[i]);
    }
  }
}

// k_bp_fast for single-axis tilt series (axis_sums), reading the slab images
// directly.
template <int VT>
__global__ void __launch_bounds__(128) k_bp_axis(KConst k, AxisGeom g, void* __restrict__ vol,
                                                 const float* __restrict__ imgs, size_t img_stride, SlabTable slabs,
                                                 int pw, int ph, size_t pitchE, float lambda, int os, float inv,
                                                 float distMin, float distMax, int linear, int transposed, int z0) {
  // plane z0 + blockIdx.z of the geometry, stored at plane blockIdx.z of vol
  // (z0 = 0 but for the autotuner's trial launches on a scratch slab)
  const int q = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int y = (int)(blockIdx.y * blockDim.y + threadIdx.y);
  const int zl = (int)blockIdx.z;
  const int z = z0 + zl;
  const int ny = (int)k.dim.y, nz = (int)k.dim.z;
  if (q >= k.dimXQuarter || y >= ny || z >= nz) return;
  const int x = 4 * q;
  const float depth = macro_depth(k, x, y, z);
  const float* img = imgs;
  if (slabs.count > 0) {
    if (!(depth >= slabs.bound[0] && depth < slabs.bound[slabs.count])) return;
    int s = 0;
    while (s + 1 < slabs.count && depth >= slabs.bound[s + 1]) ++s;
    img += (size_t)s * img_stride;
  } else if (!(depth >= distMin && depth < distMax)) {
    return;
  }
  int pbx, pby, pbz, pbw;
  if (g.clips) {
    float d;
    macro_footprint(k, x, y, z, pw, ph, d, pbx, pby, pbz, pbw);
  } else {
    macro_rect(g, x, y, z, pw, ph, pbx, pby, pbz, pbw);
  }
  const float fos = (float)os;
  const float cy = k.bbMin.y + ((float)y + 0.5f) * k.vs.y, cz = k.bbMin.z + ((float)z + 0.5f) * k.vs.z;
  const float uyz = g.U.y * cy + g.U.z * cz + g.U0, vyz = g.V.y * cy + g.V.z * cz + g.V0;
  const float dwv = inv * g.wv;
  const bool lin = linear != 0, tr = transposed != 0;
  const bool interior = !lin || (pbx >= 1 && pbz >= 1);
  const size_t sx = tr ? (size_t)ph : 1, sy = tr ? 1 : pitchE;
  const long base = ((long)zl * ny + y) * (long)k.dim.x + x;
  float res[4], has[4];
  auto read = [&](int mu, int mv) -> float {
    const float px = ((float)mu + 0.5f) * inv, py = ((float)mv + 0.5f) * inv;
    return interior ? sample_interior(img, sx, sy, px, py, lin) : sample_image(img, pw, ph, pitchE, px, py, lin, tr);
  };
  const bool patch = os == 2 && lin && interior;
  const float cx0 = k.bbMin.x + ((float)x + 0.5f) * k.vs.x;
  const RowAnchor anchor(g, y, g.U.x * cx0 + uyz, g.V.x * cx0 + vyz, fos);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float cx = k.bbMin.x + ((float)(x + i) + 0.5f) * k.vs.x;
    const float uc = g.U.x * cx + uyz, vc = g.V.x * cx + vyz;
    if (!(patch && axis_sums_os2(g, uc, vc, dwv, anchor, pbx * 2, pby * 2 - 1, pbz * 2, pbw * 2 - 1, img, sx, sy, pw,
                                 ph, res[i], has[i])))
      axis_sums(g, uc, vc, fos, inv, dwv, anchor, pbx * os, pby * os - 1, pbz * os, pbw * os - 1, read, res[i],
                has[i]);
  }
  if (VT == ESB_VOXEL_F32 && (((uintptr_t)((float*)vol + base)) & 15) == 0) {
    float4 v = *((float4*)((float*)vol + base));
    if (has[0] > 0.f) v.x += __fdividef(lambda * res[0], has[0]);
    if (has[1] > 0.f) v.y += __fdividef(lambda * res[1], has[1]);
    if (has[2] > 0.f) v.z += __fdividef(lambda * res[2], has[2]);
    if (has[3] > 0.f) v.w += __fdividef(lambda * res[3], has[3]);
    *((float4*)((float*)vol + base)) = v;
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (has[i] > 0.f)
        Voxel<VT>::store(vol, base + i, Voxel<VT>::loadrw(vol, base + i) + __fdividef(lambda * res[i], has[i]));
    }
  }
}

// Threads of a block of (quads x rows): a group of min(blockDim.x, 32)
// threads covers 4 voxels per thread of one volume row (up_voxels).
struct UpThread {
  int lanes, lane, x0, y;
  __device__ __forceinline__ UpThread() {
    lanes = min((int)blockDim.x, 32);
    lane = (int)threadIdx.x & (lanes - 1);
    x0 = 4 * (int)(blockIdx.x * blockDim.x + threadIdx.x - lane);
    y = (int)(blockIdx.y * blockDim.y + threadIdx.y);
  }
};

// k_bp_axis on pre-sampled slab images (k_upsample): one load per sample.
// What bounds it: instruction issue (grid_sums) and the latency of its loads:
// the thread's 4 voxels are read before the sums, and 9 blocks per SM asked
// for. 1024 x 1024 x 256, oversampling 2, 16 tilts: 30.2 ms with each voxel
// read after its sums, 26.2 before them, 25.5 with 36 warps per SM; 32.0 with
// the kernel that this one replaced. Eight planes per block, for the samples
// that neighbouring planes share, were 5 % slower.
template <int VT, int NC>
__global__ void __launch_bounds__(128, 9) k_bp_up(const __grid_constant__ KConst k, const __grid_constant__ AxisGeom a,
                                               const __grid_constant__ UpGeom g, void* __restrict__ vol,
                                               const __grid_constant__ SlabTable slabs, int pw, int ph, float lambda,
                                               int os, float distMin, float distMax, const float2* __restrict__ ups,
                                               size_t up_stride, OddFlag odd, int z0) {
  // plane z0 + blockIdx.z of the geometry, stored at plane blockIdx.z of vol
  // (z0 = 0 but for the autotuner's trial launches on a scratch slab)
  const UpThread t;
  const int z = z0 + (int)blockIdx.z;
  const int ny = (int)k.dim.y;
  const bool active = t.y < ny && z < (int)k.dim.z;
  const long base = ((long)blockIdx.z * ny + t.y) * (long)k.dim.x + t.x0 + t.lane;
  float v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    v[i] = active && t.x0 + t.lane + t.lanes * i < 4 * k.dimXQuarter ? Voxel<VT>::loadrw(vol, base + t.lanes * i) : 0.f;
  up_voxels<NC>(k, a, g, slabs.bound, slabs.count, distMin, distMax, ups, up_stride, odd, pw, ph, os, t.x0, t.lane,
                t.lanes, t.y, z, active, [&](int i, float acc, float dacc) {
                  Voxel<VT>::store(vol, base + t.lanes * i, v[i] + __fdividef(lambda * acc, dacc));
                });
}

// One ordered subset back-projected in one pass over the volume (the
// SIRTCount back-projections of EmSart.cpp:649-673): each quad is read once,
// the updates of the subset's projections are added to it in the order of
// the subset, as the per-projection launches add them, and it is stored once.
// Every projection contributes exactly what k_bp_up adds for it
// (pre-sampled slab images, CTF slab chosen by the first corner's depth).
// FP32 volumes: the result is bit for bit that of the per-projection
// launches. FP16 / BF16 volumes: the sum is rounded to the storage type once
// per subset instead of once per projection.
struct BpSetItem {
  KConst k;
  AxisGeom a;
  UpGeom g;
  const float2* up;  // pre-sampled slab images of this projection
  OddFlag odd;
  int nslab;         // 0: no CTF slabs
  float bound[ESB_BP_SET_MAX_SLABS + 1];
};
struct BpSet {
  int count;
  size_t up_stride;
  BpSetItem p[ESB_BP_SET_MAX];
};

template <int VT, int NC>
__global__ void __launch_bounds__(128, 8) k_bp_axis_set(const __grid_constant__ BpSet set, void* __restrict__ vol,
                                                     int pw, int ph, float lambda, int os) {
  const UpThread t;
  const int z = (int)blockIdx.z;
  const KConst& k0 = set.p[0].k;
  const int ny = (int)k0.dim.y, nx4 = 4 * k0.dimXQuarter;
  const bool active = t.y < ny && z < (int)k0.dim.z;
  const long base = ((long)z * ny + t.y) * (long)k0.dim.x + t.x0 + t.lane;
  float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (active && t.x0 + t.lane + t.lanes * i < nx4) v[i] = Voxel<VT>::loadrw(vol, base + t.lanes * i);
  unsigned touched = 0;
#pragma unroll 1
  for (int j = 0; j < set.count; ++j) {
    const BpSetItem& it = set.p[j];
    up_voxels<NC>(it.k, it.a, it.g, it.bound, it.nslab, -FLT_MAX, FLT_MAX, it.up, set.up_stride, it.odd, pw, ph, os,
              t.x0, t.lane, t.lanes, t.y, z, active, [&](int i, float acc, float dacc) {
                v[i] += __fdividef(lambda * acc, dacc);
                touched |= 1u << i;
              });
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (touched >> i & 1u) Voxel<VT>::store(vol, base + t.lanes * i, v[i]);
}

// The slab images (transposed, [x][y], stride img_stride) sampled at every
// sub-pixel grid point, with the voxel row of the grid point's ray:
// up[s][mu][mv] (up[s][mv][mu] when swapped: UpGeom) = (image s at
// ((mu + 0.5) / os, (mv + 0.5) / os), row as int bits), clamp addressing,
// nearest or bilinear as the back-projection reads it (sample_row;
// meaningful for single-axis projections, which read it). The row depends on
// the grid point and the projection only: it is formed once per grid point
// and stored with the point's value in every slab image. odd: see OddFlag.
__global__ void __launch_bounds__(256) k_upsample(const float* __restrict__ imgs, size_t img_stride, int count, int pw,
                                                  int ph, int os, float inv, int linear, RowGeom rg, int swapped,
                                                  const __grid_constant__ KConst k, float2* __restrict__ up,
                                                  size_t up_stride, OddFlag odd) {
  const int fast = blockIdx.x * blockDim.x + threadIdx.x, slow = blockIdx.y * blockDim.y + threadIdx.y;
  const int nf = (swapped ? pw : ph) * os, ns = (swapped ? ph : pw) * os;
  if (fast >= nf || slow >= ns) return;
  const int mu = swapped ? fast : slow, mv = swapped ? slow : fast;
  const float px = ((float)mu + 0.5f) * inv, py = ((float)mv + 0.5f) * inv;
  // where the sample is read: through the inverse magnification anisotropy
  const float xA = k.anisoInv[0] * px + k.anisoInv[1] * py + k.anisoInv[2];
  const float yA = k.anisoInv[3] * px + k.anisoInv[4] * py + k.anisoInv[5];
  const float row = __int_as_float(sample_row(rg, mu, mv));
  float2* out = up + (size_t)slow * nf + fast;
#pragma unroll 1
  for (int s = 0; s < count; ++s) {
    const float v = sample_image(imgs + (size_t)s * img_stride, pw, ph, (size_t)pw, xA, yA, linear != 0, true);
    odd.see(v);
    out[(size_t)s * up_stride] = make_float2(v, row);
  }
}

}  // namespace

cudaError_t launch_bp_fast_slabs(const KConst& k, void* vol, int vt, const float* imgs, size_t img_stride,
                                 const SlabTable& slabs, int pw, int ph, size_t pitchE, float lambda, int os,
                                 float distMin, float distMax, int linear, cudaStream_t st, int transposed,
                                 const float2* ups, size_t up_stride, OddFlag odd, const BpShape* shape) {
  const int nq = k.dimXQuarter, ny = (int)k.dim.y, nz = (int)k.dim.z;
  if (nq <= 0 || ny <= 0 || nz <= 0) return cudaSuccess;
  const BpGeom g = make_geom(k, os);
  const float inv = 1.0f / (float)os;
  dim3 blk(32, 4, 1), grd((nq + 31) / 32, (ny + 3) / 4, nz);
  if (ups ? axis_beam(k, g) : axis_eligible(k, g)) {
    const AxisGeom a = make_axis_geom(k, g, os);
    int z0 = 0;
    if (shape) {  // block of bx quads x by rows (bx * by <= 128); planes [z0, z0 + nz)
      blk = dim3(shape->bx, shape->by, 1);
      z0 = shape->z0;
      grd = dim3((nq + shape->bx - 1) / shape->bx, (ny + shape->by - 1) / shape->by,
                 shape->nz > 0 ? shape->nz : nz - z0);
    }
    if (ups) {
      const UpGeom u = make_up_geom(k, a, pw, ph, os, up_swapped(a));
#define ESB_AXIS(VT)                                                                                                 \
  do {                                                                                                               \
    if (os == 1)                                                                                                     \
      k_bp_up<VT, 2><<<grd, blk, 0, st>>>(k, a, u, vol, slabs, pw, ph, lambda, os, distMin, distMax, ups, up_stride, odd, z0); \
    else                                                                                                             \
      k_bp_up<VT, 3><<<grd, blk, 0, st>>>(k, a, u, vol, slabs, pw, ph, lambda, os, distMin, distMax, ups, up_stride, odd, z0); \
  } while (0)
      if (vt == ESB_VOXEL_F32) ESB_AXIS(ESB_VOXEL_F32);
      else if (vt == ESB_VOXEL_F16) ESB_AXIS(ESB_VOXEL_F16);
      else ESB_AXIS(ESB_VOXEL_BF16);
#undef ESB_AXIS
    } else {
#define ESB_AXIS(VT)                                                                                              \
  k_bp_axis<VT><<<grd, blk, 0, st>>>(k, a, vol, imgs, img_stride, slabs, pw, ph, pitchE, lambda, os, inv, distMin, \
                                     distMax, linear, transposed, z0)
      if (vt == ESB_VOXEL_F32) ESB_AXIS(ESB_VOXEL_F32);
      else if (vt == ESB_VOXEL_F16) ESB_AXIS(ESB_VOXEL_F16);
      else ESB_AXIS(ESB_VOXEL_BF16);
    }
#undef ESB_AXIS
    ESB_COUNT_LAUNCH();
    return cudaGetLastError();
  }
  switch (vt) {
    case ESB_VOXEL_F32: k_bp_fast<ESB_VOXEL_F32><<<grd, blk, 0, st>>>(k, g, vol, imgs, img_stride, slabs, pw, ph, pitchE, lambda, os, inv, distMin, distMax, linear, transposed, ups, up_stride); ESB_COUNT_LAUNCH(); break;
    case ESB_VOXEL_F16: k_bp_fast<ESB_VOXEL_F16><<<grd, blk, 0, st>>>(k, g, vol, imgs, img_stride, slabs, pw, ph, pitchE, lambda, os, inv, distMin, distMax, linear, transposed, ups, up_stride); ESB_COUNT_LAUNCH(); break;
    default: k_bp_fast<ESB_VOXEL_BF16><<<grd, blk, 0, st>>>(k, g, vol, imgs, img_stride, slabs, pw, ph, pitchE, lambda, os, inv, distMin, distMax, linear, transposed, ups, up_stride); ESB_COUNT_LAUNCH(); break;
  }
  return cudaGetLastError();
}

cudaError_t launch_bp_fast(const KConst& k, void* vol, int vt, const float* img, int pw, int ph, size_t pitchE,
                           float lambda, int os, float distMin, float distMax, int linear, cudaStream_t st) {
  SlabTable none;
  none.count = 0;
  return launch_bp_fast_slabs(k, vol, vt, img, 0, none, pw, ph, pitchE, lambda, os, distMin, distMax, linear, st, 0,
                              nullptr, 0, OddFlag{nullptr, 0}, nullptr);
}

// Whether projection k can join a subset launch (launch_bp_axis_set): the
// single-axis kernel on pre-sampled images, at most ESB_BP_SET_MAX_SLABS
// CTF slabs.
bool bp_set_eligible(const KConst& k, int os, int nslab) {
  const BpGeom g = make_geom(k, os);
  return axis_eligible(k, g) && g.exact_grid && g.aniso_identity && nslab <= ESB_BP_SET_MAX_SLABS;
}

// The back-projections of `count` (<= ESB_BP_SET_MAX) projections of one
// ordered subset in one launch (k_bp_axis_set): ks[j] the constants of
// projection j, ups[j] its pre-sampled slab images (up_stride apart) and odd[j]
// their flag,
// slabs[j] its CTF slabs (count 0: none); all bp_set_eligible, all on the
// same volume geometry. The block shape is shape's (bx, by); its planes are
// the whole volume.
cudaError_t launch_bp_axis_set(const KConst* ks, const float2* const* ups, const OddFlag* odd, const SlabTable* slabs,
                               int count, size_t up_stride, void* vol, int vt, int pw, int ph, float lambda, int os,
                               const BpShape* shape, cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  if (count > ESB_BP_SET_MAX) return cudaErrorInvalidValue;
  const KConst& k0 = ks[0];
  const int nq = k0.dimXQuarter, ny = (int)k0.dim.y, nz = (int)k0.dim.z;
  if (nq <= 0 || ny <= 0 || nz <= 0) return cudaSuccess;
  BpSet set;  // the kernel parameter (copied into the launch)
  set.count = count;
  set.up_stride = up_stride;
  for (int j = 0; j < count; ++j) {
    const BpGeom g = make_geom(ks[j], os);
    if (!(axis_eligible(ks[j], g) && g.exact_grid && g.aniso_identity) || slabs[j].count > ESB_BP_SET_MAX_SLABS ||
        !ups[j])
      return cudaErrorInvalidValue;
    BpSetItem& it = set.p[j];
    it.k = ks[j];
    it.a = make_axis_geom(ks[j], g, os);
    it.g = make_up_geom(ks[j], it.a, pw, ph, os, up_swapped(it.a));
    it.up = ups[j];
    it.odd = odd[j];
    it.nslab = slabs[j].count;
    for (int b = 0; b <= it.nslab; ++b) it.bound[b] = slabs[j].bound[b];
  }
  const int bx = shape ? shape->bx : 32, by = shape ? shape->by : 4;
  const dim3 blk(bx, by, 1), grd((nq + bx - 1) / bx, (ny + by - 1) / by, nz);
#define ESB_SET(VT)                                                                    \
  do {                                                                                 \
    if (os == 1) k_bp_axis_set<VT, 2><<<grd, blk, 0, st>>>(set, vol, pw, ph, lambda, os); \
    else k_bp_axis_set<VT, 3><<<grd, blk, 0, st>>>(set, vol, pw, ph, lambda, os);         \
  } while (0)
  if (vt == ESB_VOXEL_F32) ESB_SET(ESB_VOXEL_F32);
  else if (vt == ESB_VOXEL_F16) ESB_SET(ESB_VOXEL_F16);
  else ESB_SET(ESB_VOXEL_BF16);
#undef ESB_SET
  ESB_COUNT_LAUNCH();
  return cudaGetLastError();
}

// Pre-sampled slab images for k_bp_fast / k_bp_axis (transposed input
// images, up_stride (value, row) pairs per output image of (pw * os) x
// (ph * os)); k gives the geometry of the rows.
cudaError_t launch_upsample(const KConst& k, const float* imgs, size_t img_stride, int count, int pw, int ph, int os,
                            int linear, float2* up, size_t up_stride, OddFlag odd, cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  const BpGeom g = make_geom(k, os);
  const int swapped = axis_beam(k, g) && up_swapped(make_axis_geom(k, g, os)) ? 1 : 0;
  const int nf = (swapped ? pw : ph) * os, ns = (swapped ? ph : pw) * os;
  const dim3 blk(32, 8), grd((nf + 31) / 32, (ns + 7) / 8);
  k_upsample<<<grd, blk, 0, st>>>(imgs, img_stride, count, pw, ph, os, 1.0f / (float)os, linear, make_row_geom(k, os),
                                  swapped, k, up, up_stride, odd);
  ESB_COUNT_LAUNCH();
  return cudaGetLastError();
}

// Whether the back-projection may read pre-sampled images: the sub-pixel
// recurrence is exact (power-of-two oversampling).
bool bp_can_upsample(const KConst& k, int os) { return make_geom(k, os).exact_grid != 0; }

// Whether samples are read where they lie (no magnification anisotropy):
// launch_crop_upsample's case.
bool bp_reads_at_samples(const KConst& k, int os) { return make_geom(k, os).aniso_identity != 0; }

// Whether launch_bp_fast_slabs takes the single-axis kernel (whose launch
// shape BpShape sets), on pre-sampled images (up) or reading directly.
bool bp_uses_axis(const KConst& k, int os, bool up) {
  const BpGeom g = make_geom(k, os);
  return up ? axis_beam(k, g) : axis_eligible(k, g);
}

}  // namespace esb
