// Host interface of the batched sub-volume back-projection (esb_subvolume.cu).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <thread>
#include <vector>

#include "esb_device.cuh"

namespace esb {

// f(i) for i in [0, n) on the host cores (chunks of consecutive i per
// thread; serial below `serial_below` items).
template <class F>
void host_parallel_for(long n, F f, long serial_below = 4096) {
  const unsigned hw = std::thread::hardware_concurrency();
  const long nt = std::min<long>(std::max(1u, std::min(hw, 32u)), (n + serial_below - 1) / std::max(serial_below, 1L));
  if (nt <= 1) {
    for (long i = 0; i < n; ++i) f(i);
    return;
  }
  std::vector<std::thread> pool;
  const long chunk = (n + nt - 1) / nt;
  for (long t = 0; t < nt; ++t)
    pool.emplace_back([=, &f]() {
      const long e = std::min(n, (t + 1) * chunk);
      for (long i = t * chunk; i < e; ++i) f(i);
    });
  for (auto& th : pool) th.join();
}

// Device tables of one batched call: the work list (blocks of 128 voxel
// quads of one particle), the particles' boxes and the kernel constants of
// every (particle, list position) pair. Kept by the reconstructor and grown
// on demand, so that repeated calls allocate nothing.
struct SubvolBatch {
  void* dev = nullptr;
  size_t cap = 0;
  unsigned char* host = nullptr;  // pinned staging copy of the tables
  size_t host_cap = 0;
  cudaEvent_t copied = nullptr;   // the last copy of the staging buffer to the device
  size_t off_parts = 0, off_odd = 0, off_pairs = 0;
  int n_work = 0;
  int n_list = 0;
  int n_particles = 0;
  int all_axis = 0;  // every pair takes the single-axis sums
  // CTF patches (subvol_patch_plan): per pair the part of its tilt's slab
  // images that the box's quads read, gathered into one buffer
  void* pdev = nullptr;  // patch table, slab tables
  size_t pcap = 0;
  unsigned char* phost = nullptr;  // pinned staging copy of them
  size_t phost_cap = 0;
  cudaEvent_t pcopied = nullptr;
  size_t off_slabs = 0;
  unsigned long long *miss_dev = nullptr, *miss_host = nullptr;  // miss counter, and its pinned copy
  float* patches = nullptr;
  size_t patches_cap = 0;  // bytes
  struct Chunk {
    int t, p0, p1;  // list position, particles [p0, p1)
    bool patches;   // they fit the buffer; else the caller reads the slab images
  };
  std::vector<Chunk> chunks;     // of a plan per list position
  std::vector<int> first_work;   // first work item of every particle, and their number
};

// True when every box can be updated with aligned float4 accesses (x extent a
// multiple of 4, 16-byte aligned pointer): the batched kernel's layout.
bool subvol_batchable(int n_particles, float* const* boxes, const KConst* consts, int n_list);

// consts/active: [n_particles][n_list] for the list positions of one call;
// active may be NULL (all pairs active).
cudaError_t subvol_batch_build(SubvolBatch& b, int n_particles, float* const* boxes, const KConst* consts,
                               const unsigned char* active, int n_list, int pw, int ph, int os, cudaStream_t st);

// Flag of the call's images, set by the kernels that write them
// (launch_transpose, subvol_patch_sample); cleared by subvol_batch_build.
OddFlag subvol_odd(const SubvolBatch& b);

// Adds list positions [t0, t0 + nt) to every box. Without slabs
// (slabs.count == 0) position t reads image imgs + (t - t0) * img_stride;
// with slabs each quad reads the image of its slab. Images are transposed
// ([x][y]). Where every pair takes the single-axis sums (b.all_axis), slabs
// and the linear filter are refused: those calls read patches.
cudaError_t subvol_batch_launch(const SubvolBatch& b, int t0, int nt, const float* imgs, size_t img_stride,
                                const SlabTable& slabs, int pw, int ph, int os, int linear, cudaStream_t st);

// With CTF: plans, for every (particle, list position) pair, the patch of
// the position's slab images (slabs[t], images transposed, pw x ph) that the
// particle's quads read: the slabs its depth range meets, and the detector
// rectangle of its box's shadow with a margin, at every sub-pixel grid point.
// all_tilts: the patches of all positions in one buffer; else a buffer for
// one position, its particles in chunks (b.chunks) that fit max_bytes, a
// particle whose patches alone exceed them in a chunk without patches. Where
// the device has no room for max_bytes, as much as there is is taken. ok is
// false (nothing planned) when some pair does not take the single-axis sums,
// with all_tilts when the patches do not fit, and when there is no memory for
// the tables.
cudaError_t subvol_patch_plan(SubvolBatch& b, const SlabTable* slabs, int pw, int ph, int os, bool all_tilts,
                              size_t max_bytes, cudaStream_t st, bool& ok);

// Evaluates list position t's slab images at the patches of particles
// [p0, p1).
cudaError_t subvol_patch_sample(const SubvolBatch& b, int t, int p0, int p1, const float* imgs, size_t img_stride,
                                int pw, int ph, int os, cudaStream_t st);

// Adds list positions [t0, t0 + nt) to the boxes of particles [p0, p1) in one
// persistent launch, reading the patches.
cudaError_t subvol_patch_launch(const SubvolBatch& b, int t0, int nt, int p0, int p1, int pw, int ph, int os,
                                cudaStream_t st);

// The quads (per position) whose samples a plan did not cover: they are left
// out, so that nothing is read outside the patches, and counted on the device.
// subvol_patch_count copies the count to pinned memory when the stream gets
// there, subvol_patch_misses returns what has arrived and starts again from 0.
cudaError_t subvol_patch_count(const SubvolBatch& b, cudaStream_t st);
cudaError_t subvol_patch_misses(SubvolBatch& b, cudaStream_t st, unsigned long long& misses);

void subvol_batch_free(SubvolBatch& b);

}  // namespace esb
