// Batched sub-volume weighted back-projection (EmSARTSubVolumes).
//
// The reference reconstructs particles in batches. For every tilt it binds
// each particle's 3-D array to the surface reference and launches the
// back-projection once per particle (Reconstructor.cpp:893-914), and once per
// particle per defocus slab with CTF (:975-1033). At 2000 particles x 61
// tilts that is 122k mostly small launches, most of which cannot fill the
// GPU (a 48^3 box is 216 blocks of 128 quads).
//
// Here one persistent launch processes every particle, of mixed box sizes.
// The work list holds blocks of 512 consecutive voxels of one particle. The
// launch also loops over tilts: each thread keeps its voxels in registers,
// adds the tilts in list order and writes them once. Without CTF the launch
// covers all tilts and reads the tilts' images. With CTF the slab images of
// all tilts do not fit the device (61 tilts x ~25 slabs x 4096^2), so after
// each tilt's CTF chain k_patch_sample evaluates, for every particle, the
// part of the slab images that its voxels read (the slabs its depth range
// meets, the rectangle of its box's shadow with a margin) at every sub-pixel
// grid point, into a patch buffer: by default one tilt's patches, followed
// by a launch for that tilt, or the patches of all tilts (a few GB), followed
// by one launch over all of them. Both give the same boxes bit for bit.
//
// The per-voxel sums are those of the single-volume back-projector on
// pre-sampled images (grid_sums in esb_bp_core.cuh) for projections without
// a y component of the beam. Other geometry takes k_subvol_batch, the general
// chords on the images; particles whose patches do not fit the buffer take the
// single-volume back-projector on the slab images, one launch each.
#include <string.h>

#include <atomic>
#include <cmath>

#include "esb_bp_core.cuh"
#include "esb_subvolume.cuh"

namespace esb {

using namespace bpcore;

namespace {

constexpr int kQuadsPerItem = 128;

struct SubvolWork {
  int particle;
  int quad0;  // first quad of the block within the particle
};

struct SubvolParticle {
  float* box;
  int nqx, ny, nquads;
  int pad;
};

// Kernel constants of one (particle, list position) pair.
struct PairConst {
  KConst k;
  BpGeom g;
  int active;
};

// The same for a call whose pairs all take the single-axis sums: the depth
// and rectangle expressions' constants, the grid geometry, and the row test
// per slow and fast grid step.
struct GridPair {
  KConst k;
  UpGeom g;
  RowGeom r;
  float rs, rf, hby;
  int clips, active;
};

// Any geometry, the general chords.
__global__ void __launch_bounds__(kQuadsPerItem, 5) k_subvol_batch(const SubvolWork* __restrict__ work, int n_work,
                                                                const SubvolParticle* __restrict__ parts,
                                                                const PairConst* __restrict__ pairs, int n_list,
                                                                int t0, int nt, const float* __restrict__ imgs,
                                                                size_t img_stride, SlabTable slabs, int pw, int ph,
                                                                int os, float inv, int linear) {
  for (int w = blockIdx.x; w < n_work; w += gridDim.x) {
    const SubvolWork item = work[w];
    const SubvolParticle P = parts[item.particle];
    const int q = item.quad0 + (int)threadIdx.x;
    if (q >= P.nquads) continue;
    const int qx = q % P.nqx, y = (q / P.nqx) % P.ny, z = q / (P.nqx * P.ny);
    const int x = 4 * qx;
    float4* cell = (float4*)(P.box + ((size_t)z * P.ny + y) * (size_t)(4 * P.nqx) + x);
    float4 v = *cell;
    bool touched = false;
#pragma unroll 1
    for (int t = t0; t < t0 + nt; ++t) {
      const PairConst& pc = pairs[(size_t)item.particle * n_list + t];
      if (!pc.active) continue;
      float depth;
      int pbx, pby, pbz, pbw;
      macro_footprint(pc.k, x, y, z, pw, ph, depth, pbx, pby, pbz, pbw);
      const float* img;
      if (slabs.count > 0) {
        if (!(depth >= slabs.bound[0] && depth < slabs.bound[slabs.count])) continue;
        int s = 0;
        while (s + 1 < slabs.count && depth >= slabs.bound[s + 1]) ++s;
        img = imgs + (size_t)s * img_stride;
      } else {
        if (!(depth >= 0.0f && depth < 9999999999999.0f)) continue;
        img = imgs + (size_t)(t - t0) * img_stride;
      }
      float acc[4], dacc[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        voxel_sums(pc.k, pc.g, img, pw, ph, (size_t)pw, os, inv, linear != 0, true, x + i, y, z, pbx, pby, pbz, pbw,
                   acc[i], dacc[i]);
      // lambda = 1 (weighted back-projection): v += 1 * acc / dacc
      if (dacc[0] > 0.f) v.x += 1.0f * acc[0] / dacc[0];
      if (dacc[1] > 0.f) v.y += 1.0f * acc[1] / dacc[1];
      if (dacc[2] > 0.f) v.z += 1.0f * acc[2] / dacc[2];
      if (dacc[3] > 0.f) v.w += 1.0f * acc[3] / dacc[3];
      touched = true;
    }
    if (touched) *cell = v;
  }
}

// One (particle, list position) pair's patches: ns slab patches of pw x ph
// sub-pixel samples ([mu][mv], ph floats per column), patch sample (i, j) =
// the slab image at grid point (ox + i, oy + j).
struct PatchInfo {
  long long off;  // first float in the patch buffer
  int ox, oy;
  int pw, ph;
  int s0, ns;     // slabs s0 .. s0 + ns - 1 (ns = 0: no quad of the pair in a slab)
};
static_assert(sizeof(PatchInfo) == 32, "PatchInfo layout");

// The patches of list position t: a warp per patch column, threads along it.
// Bound by its writes; 200 particles of three sizes and one tilt 41 us, where
// the boxes' filtered reads cost k_subvol_batch 230 us more a tilt than the
// plain loads that k_subvol_grid is left with.
__global__ void __launch_bounds__(256) k_patch_sample(const PatchInfo* __restrict__ info, int n_particles, int n_list,
                                                      int t, const float* __restrict__ imgs, size_t img_stride,
                                                      int pw, int ph, float inv, float* __restrict__ patches,
                                                      OddFlag odd) {
  const int lane = threadIdx.x & 31, warp = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int nwarps = gridDim.y * (blockDim.x >> 5);
  for (int p = blockIdx.x; p < n_particles; p += gridDim.x) {
    const PatchInfo pi = info[(size_t)p * n_list + t];
    const int cols = pi.ns * pi.pw;
    for (int col = warp; col < cols; col += nwarps) {
      const int sl = col / pi.pw, i = col - sl * pi.pw;
      const float* img = imgs + (size_t)(pi.s0 + sl) * img_stride;
      const float px = ((float)(pi.ox + i) + 0.5f) * inv;
      float* dst = patches + pi.off + (long long)col * pi.ph;
      for (int j = lane; j < pi.ph; j += 32) {
        const float v = sample_image(img, pw, ph, (size_t)pw, px, ((float)(pi.oy + j) + 0.5f) * inv, true, true);
        odd.see(v);
        dst[j] = v;
      }
    }
  }
}

// Values on the grid with the row test made per sample: the offset of the
// sample's ray from the voxel row's centre plane is stepped from the exact
// one of the quad's anchor sample. Nearest reads of an image (shift = log2 of
// the oversampling) or samples of a patch (shift 0).
struct GridSamples {
  typedef float Raw;
  const float* __restrict__ base;  // grid point (0, 0)
  int m0, n0, pitch, shift;        // slow and fast grid index of sample (0, 0)
  float y, rs, rf, hby;
  __device__ __forceinline__ Raw fetch(int r, int j) const {
    return __ldg(base + ((long)((m0 + r) >> shift) * pitch + ((n0 + j) >> shift)));
  }
  __device__ __forceinline__ Raw load(int r, int j, bool take) const {
    float v = 0.f;
    asm("{.reg .pred q; setp.ne.u32 q, %2, 0; @q ld.global.nc.f32 %0, [%1];}"
        : "+f"(v)
        : "l"(base + ((long)((m0 + r) >> shift) * pitch + ((n0 + j) >> shift))), "r"((unsigned)take));
    return v;
  }
  __device__ __forceinline__ bool mine(const Raw&, int r, int j, bool taken) const {
    return taken && fabsf(fmaf((float)j, rf, fmaf((float)r, rs, y))) < hby;
  }
  __device__ __forceinline__ float value(const Raw& t) const { return t; }
};

// Every particle's boxes, list positions [t0, t0 + nt), single-axis pairs.
// Each warp takes 128 consecutive voxels of an item, thread `lane` the
// voxels lane + 32 i (neighbouring threads read neighbouring samples); per
// quad of 4 voxels thread `lane` forms depth, slab, rectangle, grid position
// and row anchor of quad `lane`, and the quad's voxels take them from there.
// Without patches (info NULL) position t reads image imgs + (t - t0) *
// img_stride by nearest texel; with them the pair's patches of the quad's
// slab. Samples outside a planned patch (none, by the plan's margins) are
// counted in *misses and the quad is skipped.
// What bounds it: instruction issue. 200 particles, 9 tilts of 1024^2, CTF: 7.96
// ms with k_subvol_batch, 5.8 here; 60 particles, 41 tilts, no CTF: 7.56 and 5.7.
template <int NC>
__global__ void __launch_bounds__(kQuadsPerItem, 6) k_subvol_grid(
    const SubvolWork* __restrict__ work, int n_work, const SubvolParticle* __restrict__ parts,
    const GridPair* __restrict__ pairs, const PatchInfo* __restrict__ info, const SlabTable* __restrict__ slabs,
    int n_list, int t0, int nt, const float* __restrict__ imgs, size_t img_stride, int pw, int ph, int os, int shift,
    OddFlag odd, unsigned long long* __restrict__ misses) {
  const int lane = threadIdx.x & 31;
  const bool any_odd = odd.set();
  for (int w = blockIdx.x; w < n_work; w += gridDim.x) {
    const SubvolWork item = work[w];
    const SubvolParticle P = parts[item.particle];
    const int q = item.quad0 + (int)threadIdx.x;
    const bool there = q < P.nquads;
    const int qx = q % P.nqx, y = (q / P.nqx) % P.ny, z = q / (P.nqx * P.ny);
    const int x = 4 * qx;
    // voxel i of the thread: voxel lane & 3 of quad (lane + 32 i) / 4 of the warp
    const long vox0 = 4l * (item.quad0 + ((int)threadIdx.x & ~31)) + lane, nvox = 4l * P.nquads;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (vox0 + 32 * i < nvox) v[i] = P.box[vox0 + 32 * i];
    unsigned touched = 0;
    const float cx = (float)(lane & 3);
#pragma unroll 1
    for (int t = t0; t < t0 + nt; ++t) {
      const GridPair& pc = pairs[(size_t)item.particle * n_list + t];
      if (!pc.active) continue;
      const UpGeom& g = pc.g;
      const bool plain = g.fits && !any_odd;
      int slab = -1, is = 0, js = 0, r0 = 0, r1 = 0, r2 = 0, r3 = 0;
      float s0 = 0.f, f0 = 0.f, ya = 0.f;
      PatchInfo pi{0, 0, 0, 0, 0, 0, 0};
      if (info) pi = info[(size_t)item.particle * n_list + t];
      if (there) {
        const float depth = macro_depth(pc.k, x, y, z);
        if (info) {
          const SlabTable& T = slabs[t];
          const int nsl = T.count;
          if (depth >= T.bound[0] && depth < T.bound[nsl]) {
            int b = 0;
            while (b + 1 < nsl && depth >= T.bound[b + 1]) ++b;
            slab = b;
          }
        } else if (depth >= 0.0f && depth < 9999999999999.0f) {
          slab = 0;
        }
        const double ds = g.s0 + x * g.sx + y * g.sy + z * g.sz, df = g.f0 + x * g.fx + y * g.fy + z * g.fz;
        const double fs = floor(ds), ff = floor(df);
        is = (int)fs, js = (int)ff;
        s0 = (float)(ds - fs), f0 = (float)(df - ff);
        ya = row_offset(pc.r, y, is, js);
        if (pc.clips) {
          float d;
          macro_footprint(pc.k, x, y, z, pw, ph, d, r0, r1, r2, r3);
        }
        if (info && slab >= 0) {
          // the quad's samples, cut to the image, lie in the patch
          const float es = 3.f * fabsf(g.dsx) + g.hs + 1.f, ef = 3.f * fabsf(g.dfx) + g.hf + 1.f;
          const float sl = fmaxf((float)is - es, 0.f), sh = fminf((float)is + 1.f + es, (float)g.smax);
          const float fl = fmaxf((float)js - ef, 0.f), fh = fminf((float)js + 1.f + ef, (float)g.fmax);
          if (sl <= sh && fl <= fh &&
              (slab < pi.s0 || slab >= pi.s0 + pi.ns || sl < (float)pi.ox || sh > (float)(pi.ox + pi.pw - 1) ||
               fl < (float)pi.oy || fh > (float)(pi.oy + pi.ph - 1))) {
            atomicAdd(misses, 1ull);
            slab = -1;
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int quad = (lane >> 2) + 8 * i;
        const int sl = __shfl_sync(0xffffffffu, slab, quad);
        const int qs = __shfl_sync(0xffffffffu, is, quad), qf = __shfl_sync(0xffffffffu, js, quad);
        const float ss = __shfl_sync(0xffffffffu, s0, quad), sf = __shfl_sync(0xffffffffu, f0, quad);
        const float yq = __shfl_sync(0xffffffffu, ya, quad);
        float a0 = (float)-qs, a1 = (float)(g.smax - qs), b0 = (float)-qf, b1 = (float)(g.fmax - qf);
        if (pc.clips) {
          a0 = (float)(__shfl_sync(0xffffffffu, r0, quad) * os - qs);
          a1 = (float)(__shfl_sync(0xffffffffu, r1, quad) * os - 1 - qs);
          b0 = (float)(__shfl_sync(0xffffffffu, r2, quad) * os - qf);
          b1 = (float)(__shfl_sync(0xffffffffu, r3, quad) * os - 1 - qf);
        }
        // slab < 0: no such quad, or outside every slab
        const float* base = imgs;
        int pitch = ph;
        if (info) {  // the patch addressed in grid points
          pitch = pi.ph;
          base += pi.off + (long long)(sl - pi.s0) * pi.pw * pi.ph - (long long)pi.ox * pi.ph - pi.oy;
        } else {
          base += (size_t)(t - t0) * img_stride;
        }
        float acc, dacc;
        grid_sums<NC>(g, fmaf(cx, g.dsx, ss), fmaf(cx, g.dfx, sf), a0, a1, b0, b1, sl >= 0, plain,
                      [&](int ds, int dj, float fds, float fdj) {
                        GridSamples r;
                        r.base = base;
                        r.m0 = qs + ds;
                        r.n0 = qf + dj;
                        r.pitch = pitch;
                        r.shift = shift;
                        r.rs = pc.rs;
                        r.rf = pc.rf;
                        r.hby = pc.hby;
                        r.y = fmaf(fdj, pc.rf, fmaf(fds, pc.rs, yq));
                        return r;
                      },
                      acc, dacc);
        // lambda = 1 (weighted back-projection)
        if (dacc > 0.f) {
          v[i] += acc / dacc;
          touched |= 1u << i;
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (touched >> i & 1u) P.box[vox0 + 32 * i] = v[i];
  }
}

size_t align256(size_t n) { return (n + 255) & ~(size_t)255; }

}  // namespace

bool subvol_batchable(int n_particles, float* const* boxes, const KConst* consts, int n_list) {
  for (int p = 0; p < n_particles; ++p) {
    const KConst& k = consts[(size_t)p * n_list];
    if (((uintptr_t)boxes[p] & 15) != 0) return false;
    if ((int)k.dim.x != 4 * k.dimXQuarter) return false;
  }
  return true;
}

// Pinned staging of `bytes`, grown on demand: waits for the copy out of it.
static cudaError_t staging(unsigned char*& host, size_t& cap, cudaEvent_t& copied, size_t bytes) {
  cudaError_t e;
  if (copied && (e = cudaEventSynchronize(copied)) != cudaSuccess) return e;
  if (!copied && (e = cudaEventCreateWithFlags(&copied, cudaEventDisableTiming)) != cudaSuccess) return e;
  if (bytes > cap) {
    cudaFreeHost(host);
    host = nullptr;
    cap = 0;
    if ((e = cudaHostAlloc((void**)&host, bytes, cudaHostAllocDefault)) != cudaSuccess) return e;
    cap = bytes;
  }
  return cudaSuccess;
}

// Device buffer of `bytes`, grown on demand once the stream no longer uses it.
static cudaError_t device_buffer(void*& dev, size_t& cap, size_t bytes, cudaStream_t st) {
  if (bytes <= cap) return cudaSuccess;
  cudaError_t e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return e;
  cudaFree(dev);
  dev = nullptr;
  cap = 0;
  if ((e = cudaMalloc(&dev, bytes)) != cudaSuccess) return e;
  cap = bytes;
  return cudaSuccess;
}

// Whether an allocation failed for want of memory; clears the error.
static bool out_of_memory(cudaError_t e) {
  if (e != cudaErrorMemoryAllocation) return false;
  cudaGetLastError();
  return true;
}

constexpr long kPairsPerThread = 512;  // host threads are worth starting beyond this many pairs

cudaError_t subvol_batch_build(SubvolBatch& b, int n_particles, float* const* boxes, const KConst* consts,
                               const unsigned char* active, int n_list, int pw, int ph, int os, cudaStream_t st) {
  std::vector<SubvolWork> work;
  std::vector<SubvolParticle> parts((size_t)n_particles);
  b.first_work.assign((size_t)n_particles + 1, 0);
  for (int p = 0; p < n_particles; ++p) {
    b.first_work[p] = (int)work.size();
    const KConst& k = consts[(size_t)p * n_list];
    SubvolParticle& P = parts[p];
    P.box = boxes[p];
    P.nqx = k.dimXQuarter;
    P.ny = (int)k.dim.y;
    P.nquads = P.nqx * P.ny * (int)k.dim.z;
    P.pad = 0;
    bool any = false;
    for (int t = 0; t < n_list && !any; ++t) any = !active || active[(size_t)p * n_list + t];
    if (!any) continue;
    for (int q0 = 0; q0 < P.nquads; q0 += kQuadsPerItem) work.push_back(SubvolWork{p, q0});
  }
  b.first_work[n_particles] = (int)work.size();
  const size_t n_pairs = (size_t)n_particles * n_list;
  b.off_parts = align256(work.size() * sizeof(SubvolWork));
  b.off_odd = b.off_parts + align256(parts.size() * sizeof(SubvolParticle));
  b.off_pairs = b.off_odd + align256(sizeof(unsigned));
  const size_t most = b.off_pairs + n_pairs * std::max(sizeof(GridPair), sizeof(PairConst));
  cudaError_t e;
  if ((e = staging(b.host, b.host_cap, b.copied, most)) != cudaSuccess) return e;
  memcpy(b.host, work.data(), work.size() * sizeof(SubvolWork));
  memcpy(b.host + b.off_parts, parts.data(), parts.size() * sizeof(SubvolParticle));
  memset(b.host + b.off_odd, 0, sizeof(unsigned));
  // per-pair constants on the host cores (the tables of 2000 particles x 61
  // tilts are 1.2e5 pairs)
  std::atomic<int> others{0};
  GridPair* gp = (GridPair*)(b.host + b.off_pairs);
  host_parallel_for((long)n_pairs, [&](long i) {
    const BpGeom bg = make_geom(consts[i], os);
    if (!axis_eligible(consts[i], bg)) {
      others.store(1, std::memory_order_relaxed);
      return;
    }
    const AxisGeom a = make_axis_geom(consts[i], bg, os);
    GridPair& q = gp[i];
    q.k = consts[i];
    q.g = make_up_geom(consts[i], a, pw, ph, os, false);  // transposed images: fast axis v
    q.r = a.r;
    q.rs = a.r.u;
    q.rf = a.r.v;
    q.hby = a.hby;
    q.clips = a.clips;
    q.active = !active || active[i];
  }, kPairsPerThread);
  b.all_axis = others.load() == 0 ? 1 : 0;
  if (!b.all_axis) {
    PairConst* pc = (PairConst*)(b.host + b.off_pairs);
    host_parallel_for((long)n_pairs, [&](long i) {
      PairConst& q = pc[i];
      q.k = consts[i];
      q.g = make_geom(consts[i], os);
      q.active = !active || active[i];
    }, kPairsPerThread);
  }
  const size_t bytes = b.off_pairs + n_pairs * (b.all_axis ? sizeof(GridPair) : sizeof(PairConst));
  if ((e = device_buffer(b.dev, b.cap, bytes, st)) != cudaSuccess) return e;
  b.n_work = (int)work.size();
  b.n_list = n_list;
  b.n_particles = n_particles;
  if ((e = cudaMemcpyAsync(b.dev, b.host, bytes, cudaMemcpyHostToDevice, st)) != cudaSuccess) return e;
  return cudaEventRecord(b.copied, st);
}

OddFlag subvol_odd(const SubvolBatch& b) { return OddFlag{(unsigned*)((char*)b.dev + b.off_odd), 1}; }

// Blocks of a persistent grid: every resident block slot of every SM, at
// most one per work item.
static cudaError_t persistent_blocks(const void* kernel, int n_work, unsigned& blocks) {
  int dev = 0, n_sm = 0, per_sm = 0;
  cudaError_t e;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kQuadsPerItem, 0)) != cudaSuccess) return e;
  const long most = (long)n_sm * (per_sm > 0 ? per_sm : 1);
  blocks = (unsigned)std::min<long>(most, n_work);
  return cudaSuccess;
}

cudaError_t subvol_batch_launch(const SubvolBatch& b, int t0, int nt, const float* imgs, size_t img_stride,
                                const SlabTable& slabs, int pw, int ph, int os, int linear, cudaStream_t st) {
  if (b.n_work <= 0 || nt <= 0) return cudaSuccess;
  if (b.all_axis && (slabs.count > 0 || linear)) return cudaErrorInvalidValue;  // patches, or a launch per particle
  unsigned blocks = 0;
  cudaError_t e;
  const char* base = (const char*)b.dev;
  if (b.all_axis) {  // without CTF: nearest texels of the tilts' images
    const auto kernel = os == 1 ? k_subvol_grid<2> : k_subvol_grid<3>;
    if ((e = persistent_blocks((const void*)kernel, b.n_work, blocks)) != cudaSuccess) return e;
    int shift = 0;
    while ((1 << shift) < os) ++shift;
    kernel<<<blocks, kQuadsPerItem, 0, st>>>(
        (const SubvolWork*)base, b.n_work, (const SubvolParticle*)(base + b.off_parts),
        (const GridPair*)(base + b.off_pairs), nullptr, nullptr, b.n_list, t0, nt, imgs, img_stride, pw, ph, os, shift,
        subvol_odd(b), nullptr);
  } else {
    if ((e = persistent_blocks((const void*)k_subvol_batch, b.n_work, blocks)) != cudaSuccess) return e;
    k_subvol_batch<<<blocks, kQuadsPerItem, 0, st>>>(
        (const SubvolWork*)base, b.n_work, (const SubvolParticle*)(base + b.off_parts),
        (const PairConst*)(base + b.off_pairs), b.n_list, t0, nt, imgs, img_stride, slabs, pw, ph, os,
        1.0f / (float)os, linear);
  }
  ESB_COUNT_LAUNCH();
  return cudaGetLastError();
}

cudaError_t subvol_patch_plan(SubvolBatch& b, const SlabTable* slabs, int pw, int ph, int os, bool all_tilts,
                              size_t max_bytes, cudaStream_t st, bool& ok) {
  ok = false;
  if (!b.all_axis || b.n_work <= 0 || b.n_list <= 0) return cudaSuccess;
  const int np = b.n_particles, nl = b.n_list;
  b.off_slabs = align256((size_t)np * nl * sizeof(PatchInfo));
  const size_t bytes = b.off_slabs + (size_t)nl * sizeof(SlabTable);
  cudaError_t e;
  if (!b.miss_host) {
    if ((e = cudaHostAlloc((void**)&b.miss_host, sizeof(*b.miss_host), cudaHostAllocDefault)) != cudaSuccess)
      return out_of_memory(e) ? cudaSuccess : e;
    *b.miss_host = 0;
  }
  if (!b.miss_dev) {
    if ((e = cudaMalloc((void**)&b.miss_dev, sizeof(*b.miss_dev))) != cudaSuccess)
      return out_of_memory(e) ? cudaSuccess : e;
    if ((e = cudaMemsetAsync(b.miss_dev, 0, sizeof(*b.miss_dev), st)) != cudaSuccess) return e;
  }
  if ((e = staging(b.phost, b.phost_cap, b.pcopied, bytes)) != cudaSuccess) return out_of_memory(e) ? cudaSuccess : e;
  if ((e = device_buffer(b.pdev, b.pcap, bytes, st)) != cudaSuccess) return out_of_memory(e) ? cudaSuccess : e;
  const SubvolParticle* parts = (const SubvolParticle*)(b.host + b.off_parts);
  const GridPair* pcs = (const GridPair*)(b.host + b.off_pairs);
  PatchInfo* info = (PatchInfo*)b.phost;
  host_parallel_for((long)np * nl, [&](long i) {
    const int p = (int)(i / nl), t = (int)(i % nl);
    PatchInfo& pi = info[i];
    pi = PatchInfo{0, 0, 0, 1, 1, 0, 0};
    const GridPair& q = pcs[i];
    const SubvolParticle& P = parts[p];
    const SlabTable& T = slabs[t];
    if (!q.active || P.nquads <= 0 || T.count <= 0) return;
    const KConst& k = q.k;
    const int nz = P.nquads / (P.nqx * P.ny);
    // depth range of the quads' first corners (macro_depth), and the shadow
    // of the box (x extended by the last quad's 5-voxel macro cell)
    const double n[3] = {k.n.x, k.n.y, k.n.z};
    const double ndet = -(n[0] * k.det.x + n[1] * k.det.y + n[2] * k.det.z);
    const double bmin[3] = {k.bbMin.x, k.bbMin.y, k.bbMin.z}, vs[3] = {k.vs.x, k.vs.y, k.vs.z};
    const double qlast[3] = {4.0 * (P.nqx - 1), (double)(P.ny - 1), (double)(nz - 1)};
    const double ext[3] = {(double)(4 * P.nqx + 1), (double)P.ny, (double)nz};
    const double U[3] = {k.detMat[0].x, k.detMat[0].y, k.detMat[0].z}, V[3] = {k.detMat[1].x, k.detMat[1].y, k.detMat[1].z};
    double dlo = 1e300, dhi = -1e300, tlo = 1e300, thi = -1e300;
    double umin = 1e300, umax = -1e300, vmin = 1e300, vmax = -1e300;
    for (int c = 0; c < 8; ++c) {
      double tq = ndet, u = k.detMat[0].w, v = k.detMat[1].w;
      for (int j = 0; j < 3; ++j) {
        const int hi = (c >> j) & 1;
        tq += n[j] * (bmin[j] + (hi ? qlast[j] : 0.0) * vs[j]);
        const double pj = bmin[j] + (hi ? ext[j] : 0.0) * vs[j];
        u += U[j] * pj;
        v += V[j] * pj;
      }
      tlo = std::min(tlo, tq), thi = std::max(thi, tq);
      umin = std::min(umin, u), umax = std::max(umax, u);
      vmin = std::min(vmin, v), vmax = std::max(vmax, v);
    }
    if (tlo >= 0.0) dlo = tlo, dhi = thi;
    else if (thi <= 0.0) dlo = -thi, dhi = -tlo;
    else dlo = 0.0, dhi = std::max(-tlo, thi);
    const double eps = 1e-2 + 1e-5 * dhi;
    if (dhi + eps < T.bound[0] || dlo - eps >= T.bound[T.count]) return;  // no quad in a slab
    auto slab_of = [&](double d) {
      int s = 0;
      while (s + 1 < T.count && d >= T.bound[s + 1]) ++s;
      return s;
    };
    const int s0 = slab_of(dlo - eps), s1 = slab_of(dhi + eps);
    // margin around the shadow: a voxel's half shadow, the quad's extent and
    // a step of rounding, in pixels
    const double mu = (3.0 * std::fabs(q.g.dsx) + q.g.hs + 3.0) / os, mv = (3.0 * std::fabs(q.g.dfx) + q.g.hf + 3.0) / os;
    auto clampd = [](double a, int lo, int hi) { return a < lo ? lo : (a > hi ? hi : (int)a); };
    const int bx0 = clampd(std::floor(umin - mu), 0, pw - 1), bx1 = clampd(std::ceil(umax + mu), 0, pw - 1);
    const int by0 = clampd(std::floor(vmin - mv), 0, ph - 1), by1 = clampd(std::ceil(vmax + mv), 0, ph - 1);
    pi.ox = bx0 * os;
    pi.pw = (bx1 - bx0 + 1) * os;
    pi.oy = by0 * os;
    pi.ph = (by1 - by0 + 1) * os;
    pi.s0 = s0;
    pi.ns = s1 - s0 + 1;
  }, kPairsPerThread);
  // offsets: over all pairs, or per list position, the particles in chunks
  // that fit the buffer; the bound is halved until the device has room
  for (size_t max_floats = max_bytes / sizeof(float);;) {
    size_t most = 0;
    b.chunks.clear();
    if (all_tilts) {
      for (long i = 0; i < (long)np * nl; ++i) {
        info[i].off = (long long)most;
        most += (size_t)info[i].ns * info[i].pw * info[i].ph;
      }
      if (most > max_floats) return cudaSuccess;
    } else {
      for (int t = 0; t < nl; ++t) {
        size_t used = 0;
        int first = 0;
        auto cut = [&](int p, bool patches) {  // a chunk up to particle p
          if (p > first) b.chunks.push_back({t, first, p, patches});
          first = p;
          used = 0;
        };
        for (int p = 0; p < np; ++p) {
          PatchInfo& pi = info[(size_t)p * nl + t];
          const size_t n = (size_t)pi.ns * pi.pw * pi.ph;
          if (used + n > max_floats) cut(p, true);
          pi.off = (long long)used;
          if (n > max_floats) {
            cut(p + 1, false);
          } else {
            used += n;
            most = std::max(most, used);
          }
        }
        cut(np, true);
      }
    }
    void* buf = b.patches;
    e = device_buffer(buf, b.patches_cap, std::max<size_t>(most, 1) * sizeof(float), st);
    b.patches = (float*)buf;
    if (e == cudaSuccess) break;
    if (!out_of_memory(e)) return e;
    if (all_tilts || most <= 1) return cudaSuccess;
    max_floats = most / 2;
  }
  memcpy(b.phost + b.off_slabs, slabs, (size_t)nl * sizeof(SlabTable));
  if ((e = cudaMemcpyAsync(b.pdev, b.phost, bytes, cudaMemcpyHostToDevice, st)) != cudaSuccess) return e;
  if ((e = cudaEventRecord(b.pcopied, st)) != cudaSuccess) return e;
  ok = true;
  return cudaSuccess;
}

cudaError_t subvol_patch_sample(const SubvolBatch& b, int t, int p0, int p1, const float* imgs, size_t img_stride,
                                int pw, int ph, int os, cudaStream_t st) {
  if (p1 <= p0) return cudaSuccess;
  // about 2000 blocks, however few the particles
  const unsigned gx = (unsigned)std::min(p1 - p0, kSMs * 8);
  const dim3 grd(gx, std::max(1u, std::min(16u, 2048u / gx)));
  k_patch_sample<<<grd, 256, 0, st>>>((const PatchInfo*)b.pdev + (size_t)p0 * b.n_list, p1 - p0, b.n_list, t, imgs,
                                      img_stride, pw, ph, 1.0f / (float)os, b.patches, subvol_odd(b));
  ESB_COUNT_LAUNCH();
  return cudaGetLastError();
}

cudaError_t subvol_patch_launch(const SubvolBatch& b, int t0, int nt, int p0, int p1, int pw, int ph, int os,
                                cudaStream_t st) {
  const int w0 = b.first_work[p0], n_work = b.first_work[p1] - w0;
  if (n_work <= 0 || nt <= 0) return cudaSuccess;
  unsigned blocks = 0;
  cudaError_t e;
  const auto kernel = os == 1 ? k_subvol_grid<2> : k_subvol_grid<3>;
  if ((e = persistent_blocks((const void*)kernel, n_work, blocks)) != cudaSuccess) return e;
  const char* base = (const char*)b.dev;
  const char* pbase = (const char*)b.pdev;
  kernel<<<blocks, kQuadsPerItem, 0, st>>>(
      (const SubvolWork*)base + w0, n_work, (const SubvolParticle*)(base + b.off_parts),
      (const GridPair*)(base + b.off_pairs), (const PatchInfo*)pbase, (const SlabTable*)(pbase + b.off_slabs),
      b.n_list, t0, nt, b.patches, 0, pw, ph, os, 0, subvol_odd(b), b.miss_dev);
  ESB_COUNT_LAUNCH();
  return cudaGetLastError();
}

cudaError_t subvol_patch_count(const SubvolBatch& b, cudaStream_t st) {
  return cudaMemcpyAsync(b.miss_host, b.miss_dev, sizeof(*b.miss_host), cudaMemcpyDeviceToHost, st);
}

cudaError_t subvol_patch_misses(SubvolBatch& b, cudaStream_t st, unsigned long long& misses) {
  misses = b.miss_host ? *(volatile unsigned long long*)b.miss_host : 0;
  if (!misses) return cudaSuccess;
  *b.miss_host = 0;
  return cudaMemsetAsync(b.miss_dev, 0, sizeof(*b.miss_dev), st);
}

void subvol_batch_free(SubvolBatch& b) {
  cudaFree(b.miss_dev);
  b.miss_dev = nullptr;
  cudaFree(b.pdev);
  b.pdev = nullptr;
  b.pcap = 0;
  cudaFree(b.patches);
  b.patches = nullptr;
  b.patches_cap = 0;
  cudaFree(b.dev);
  b.dev = nullptr;
  b.cap = 0;
  if (b.copied) cudaEventSynchronize(b.copied);
  cudaFreeHost(b.host);
  b.host = nullptr;
  b.host_cap = 0;
  if (b.copied) cudaEventDestroy(b.copied);
  b.copied = nullptr;
  if (b.pcopied) cudaEventSynchronize(b.pcopied);
  cudaFreeHost(b.miss_host);  // (the frees above waited for the last copy to it)
  b.miss_host = nullptr;
  cudaFreeHost(b.phost);
  b.phost = nullptr;
  b.phost_cap = 0;
  if (b.pcopied) cudaEventDestroy(b.pcopied);
  b.pcopied = nullptr;
}

}  // namespace esb
