// Host-side objects behind the C ABI (include/glamer_b200.h).
#pragma once
#include <cuda_runtime.h>

#include <memory>
#include <string>
#include <vector>

#include "glb_internal.h"

struct glb_particle_rec {
  float x[3];
  float Mass;
  float Size;
  int type;
};
static_assert(sizeof(glb_particle_rec) == 24, "ParticleType<float> is 24 bytes");

namespace glb {

// Error status carried through the C ABI.
struct Status {
  int code = 0;
  std::string msg;
  static Status ok() { return Status(); }
  static Status err(int c, const std::string &m) {
    Status s;
    s.code = c;
    s.msg = m;
    return s;
  }
  bool good() const { return code == 0; }
};

// The largest device allocation this thread may make, 0 for no limit
// (GLB_OPT_ALLOC_LIMIT: for tests of refused allocations).
inline thread_local size_t alloc_limit = 0;
inline bool alloc_refused(size_t bytes) { return alloc_limit && bytes > alloc_limit; }

// Gives back to the device what its scratch pools hold unused.
void trim_scratch_pools();

// Device memory owned by RAII.  An allocation that finds no memory is tried
// again once the scratch pools have given back what they keep.  After a refused allocation the buffer is empty
// and the runtime's last error is cleared (the caller has the status).
template <typename T>
struct DBuf {
  T *p = nullptr;
  size_t n = 0;
  DBuf() = default;
  DBuf(const DBuf &) = delete;
  DBuf &operator=(const DBuf &) = delete;
  ~DBuf() { release(); }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
  }
  cudaError_t alloc(size_t count) {
    release();
    if (count == 0) return cudaSuccess;
    cudaError_t e = try_alloc(count);
    if (e == cudaErrorMemoryAllocation) {
      trim_scratch_pools();
      e = try_alloc(count);
    }
    if (e == cudaSuccess) n = count;
    return e;
  }

 private:
  cudaError_t try_alloc(size_t count) {
    const cudaError_t e = alloc_refused(count * sizeof(T)) ? cudaErrorMemoryAllocation
                                                           : cudaMalloc((void **)&p, count * sizeof(T));
    if (e != cudaSuccess) {
      p = nullptr;
      (void)cudaGetLastError();
    }
    return e;
  }
};

// The pools of this device's scratch memory.  Each keeps what it was at most asked
// for at once, up to kScratchKept, between uses, so that building many trees does
// not map memory for each (a build takes some twenty buffers); what it holds beyond
// that goes back to the device at the next synchronisation.  Shared walks have a
// pool of their own: among the blocks that builds leave behind, their 12 to 113 MB
// in one piece were mapped again by every call (81 rays 1.28 ms for 1.25); and its
// limit holds a dozen calls at once (eight threads, 4,097 rays each: 0.8 ms a call,
// 0.8 to 1.5 with 256 MB).
enum ScratchKind { kBuildScratch, kWalkScratch, kScratchKinds };
constexpr unsigned long long kScratchKept[kScratchKinds] = {256ull << 20, 1024ull << 20};
cudaError_t scratch_pool(cudaMemPool_t *pool, ScratchKind kind);

// Scratch memory from a pool, taken and given back in the order of a stream.
// An arena is one such allocation that later ones carve their buffers from while
// it has room (a small tree's twenty buffers take longer to allocate than to
// fill).
template <typename T>
struct ABuf {
  T *p = nullptr;
  size_t n = 0;
  cudaStream_t s;
  struct Arena *arena;
  ScratchKind kind = kBuildScratch;
  bool carved = false;
  explicit ABuf(cudaStream_t st, Arena *a = nullptr) : s(st), arena(a) {}
  ABuf(cudaStream_t st, ScratchKind k) : s(st), arena(nullptr), kind(k) {}
  ABuf(const ABuf &) = delete;
  ABuf &operator=(const ABuf &) = delete;
  ~ABuf() { release(); }
  void release() {
    if (p && !carved) cudaFreeAsync(p, s);
    p = nullptr;
    n = 0;
    carved = false;
  }
  cudaError_t alloc(size_t count);

 private:
  cudaError_t try_alloc(size_t count);
};
struct Arena {
  ABuf<char> mem;
  size_t used = 0;
  explicit Arena(cudaStream_t st) : mem(st) {}
  char *carve(size_t bytes) {
    const size_t at = (used + 255) / 256 * 256;
    if (!mem.p || at + bytes > mem.n) return nullptr;
    used = at + bytes;
    return mem.p + at;
  }
};
template <typename T>
cudaError_t ABuf<T>::alloc(size_t count) {
  release();
  if (count == 0) return cudaSuccess;
  if (arena)
    if (char *c = arena->carve(count * sizeof(T))) {
      p = reinterpret_cast<T *>(c);
      n = count;
      carved = true;
      return cudaSuccess;
    }
  const cudaError_t e0 = try_alloc(count);
  if (e0 != cudaErrorMemoryAllocation) return e0;
  trim_scratch_pools();
  return try_alloc(count);
}
template <typename T>
cudaError_t ABuf<T>::try_alloc(size_t count) {
  cudaMemPool_t pool;
  cudaError_t e = alloc_refused(count * sizeof(T)) ? cudaErrorMemoryAllocation : scratch_pool(&pool, kind);
  if (e == cudaSuccess) e = cudaMallocFromPoolAsync((void **)&p, count * sizeof(T), pool, s);
  if (e == cudaSuccess) {
    n = count;
  } else {
    p = nullptr;
    (void)cudaGetLastError();
  }
  return e;
}

// TreeQuadParticles built on the device.
struct Tree {
  TreeDev dev{};
  // Every array per node and the exponential's table; the sorted records and their
  // leaf-relative form.  In one allocation each, or in two (`more`) where that is
  // over 1 MB and its halves are not: cudaMalloc carves up to 1 MB out of blocks
  // that it keeps, and maps and unmaps memory for more (35,000 particles, bucket 20:
  // build and destruction 2.19 ms in one piece each, 1.94 in two).
  DBuf<char> node_mem, node_more;
  DBuf<float4> particles, particles_more;
  DBuf<float4> bigs;
  int nnodes = 0;
  size_t nparticles = 0;
  size_t nbranches = 0;            // including empty children (reference count)
  double theta = 0.1;              // opening angle the tree was built with
  std::vector<double> export_rows; // 16 doubles per branch when requested
  float build_ms = 0;
};

// Whether two pieces of these sizes are allocated one by one.
inline bool in_pieces(size_t a, size_t b) {
  constexpr size_t kSmall = (size_t)1 << 20;
  return a + b > kSmall && a <= kSmall && b <= kSmall;
}

struct TreeParams {
  float mass_fixed = -1, size_fixed = -1;
  double inv_area = 0;
  int bucket = 5;
  double theta = 0.1;
  int periodic = 0;
  double inv_screening = 0;
  double max_range = -1;
};

// Builds a tree from host particle records (ParticleType<float>).
Status build_tree(const glb_particle_rec *host_particles, size_t n, const TreeParams &prm,
                  bool want_export, cudaStream_t stream, std::unique_ptr<Tree> &out);

// TreeQuadHalos (include/quadTreeHalos.h:129-515) built on the host: branch
// arrays in preorder, ready for upload.  xp: 2n halo positions (physical
// Mpc), rmax / mass: the haloes' float members.  Returns false with `err` set
// when the positions span no area ("particles in same place.").
struct HaloTreeHost {
  std::vector<HNode> nodes;
  std::vector<int> bigs;
  double period_x = 0, period_y = 0;
};
bool build_halo_tree(const std::vector<double> &xp, const std::vector<float> &rmax, const std::vector<float> &mass,
                     int bucket, double theta, double max_range, HaloTreeHost &out, std::string &err);

// LensHaloParticles::calculate_smoothing on the device: Size of every record
// of d_p (device, n records) written to d_size (device, n floats) as the
// distance to the (nsmooth+1)-th nearest particle, the particle itself
// counted.  ms_out (nullable): [0] sort and bucket boxes, [1] search, in ms.
Status smooth_particles_device(const glb_particle_rec *d_p, size_t n, int nsmooth, float *d_size,
                               cudaStream_t stream, float *ms_out);

// Global options.
extern int g_keep_tree_export;

}  // namespace glb
