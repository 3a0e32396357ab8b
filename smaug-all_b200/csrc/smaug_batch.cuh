// smaug_batch.cuh -- device-side description of a batch: many independent
// simulations (same ndim and precision, any sizes) advanced together, one
// launch per RK stage for all of them.
#pragma once
#include <algorithm>
#include <vector>

#include "smaug_device.cuh"

namespace smaug {

// One simulation of a batch, resident in the batch's device table.
struct BatchInst {
  Geo geo;
  Phys phys;
  const double *bg;  // NB background fields
  double *W[4];      // FP64 path: state and the three RK stage buffers; mixed: W[0] only (load/store)
  float *F[5];       // mixed path: w32, c32, two FP32 stage states, FP32 RK sum
  DevScalars *sc;
  int tiles[3];      // 2-D: tiles per dimension for the batch's current tile shape
  int active;        // slot holds a simulation
};

// Work list entry: simulation slot and tile index within it.
struct WorkItem {
  int inst;
  int tile;    // stage items: the tile's x index; advance items: the first chunk
  int by, bz;  // stage items: the tile's y and z indices; advance items: by chunks
};

// The 3-D stage runs over slabs: inner planes z0 .. z1-1 of one simulation with
// a workspace of their own (smaug_pass3.cuh).  The derived arrays cover the
// planes pz0 .. pz1-1 (the slab +-3, and plane 5 where the left pad reads it),
// the face arrays the planes z0-1 .. z1.
struct Slab3 {
  int inst;
  int z0, z1;
  int pz0, pz1;
  int NP, NV;  // cells per derived array and per face array
  void *P, *V;
};

// Workspace elements per cell: derived arrays (smaug_pass3.cuh: 3 pairs, 2
// four-vectors and the background) and face arrays (2 four-vectors per dim).
constexpr int kDerived3 = 18, kFaces3 = 24;
// Cells per derive item, faces or line segments per faces item, and threads of
// the faces kernel.
constexpr int kDeriveChunk = 1024, kFaceChunk = 512, kFaceSegs = 128;
// Faces a thread takes along y and z.
constexpr int face_seg(bool mixed) { return mixed ? 8 : 4; }
// Workspace limit of one group of slabs.  Slabs bound the memory; small ones that
// stay in L2 between their passes were slower, each pass paying its ramp and tail
// (blast wave 128^3 mixed, ms per step: 512 MB 1.86, 128 MB 2.09, 64 MB 2.33).  A
// slab has at least four planes, its halo being as large as they are, and takes
// what they need (1.3 KB, in FP64 2.6 KB, per cell of a plane) where that is more;
// only under a lower limit, where the device has less to give, do slabs go down to
// one plane.
constexpr size_t kSlabBytes = (size_t)512 << 20;
constexpr size_t kLeastSlabBytes = (size_t)4 << 20;  // the last limit that is tried

// The workspace of a context or a batch: kept from plan to plan, with the limit
// that plans keep to (lowered for good where the memory for more was refused).
struct Workspace3 {
  char *p = nullptr;
  size_t bytes = 0, limit = kSlabBytes;
};

// The work of one 3-D stage: groups of slabs that run one after another
// through the same workspace, each with its items for the three passes
// (WorkItem.inst is the slab; faces: tile = chunk, by = dimension).
struct Plan3 {
  struct Group {
    int item[3], count[3];  // first item and number of items per pass
  };
  std::vector<Slab3> slabs;  // P, V: offsets in the workspace until placed
  std::vector<WorkItem> items;
  std::vector<Group> groups;
  size_t bytes = 0;  // workspace

  // Plan for the simulations and find the workspace: the one in use if a plan
  // within its limit fits it, else a larger one, first beside it, so that a refusal
  // leaves it as it was and the plan is cut to it; at last, without it, smaller
  // ones.  want: what to take rather than the bare need, so that later plans fit
  // (at most the limit; twice the one in use in any case).  alloc(void **, bytes)
  // returns a cudaError_t; release(p) waits for queued work that uses p and
  // frees it.
  template <typename Alloc, typename Release>
  cudaError_t fit(Workspace3 &ws, const std::vector<std::pair<int, Geo>> &sims, const int *t, bool mixed, size_t want,
                  Alloc alloc, Release release) {
    build(sims, t, mixed, ws.limit);
    if (bytes <= ws.bytes) return cudaSuccess;
    cudaError_t e = cudaErrorMemoryAllocation;
    auto refused = [&](size_t n) {
      char *p = nullptr;
      e = alloc((void **)&p, n);
      if (e == cudaSuccess) {
        if (ws.p) release(ws.p);
        ws.p = p;
        ws.bytes = n;
      }
      return e == cudaErrorMemoryAllocation;
    };
    const size_t room = std::max(bytes, std::min(ws.limit, std::max(want, 2 * ws.bytes)));
    if (!refused(room) || (room > bytes && !refused(bytes))) return e;
    if (ws.p) {
      build(sims, t, mixed, ws.bytes);
      if (bytes <= ws.bytes) {
        ws.limit = ws.bytes;
        return cudaSuccess;
      }
      release(ws.p);
      ws.p = nullptr;
      ws.bytes = 0;
    }
    for (size_t limit = ws.limit; limit >= kLeastSlabBytes; limit /= 4) {
      build(sims, t, mixed, limit);
      if (refused(bytes)) continue;
      if (e == cudaSuccess) ws.limit = limit;
      return e;
    }
    return e;
  }

  // sims: (slot, geometry) of every simulation; t: the terms tile; limit: of
  // the workspace.
  void build(const std::vector<std::pair<int, Geo>> &sims, const int *t, bool mixed, size_t limit = kSlabBytes) {
    slabs.clear();
    items.clear();
    groups.clear();
    bytes = 0;
    const size_t es = mixed ? sizeof(float) : sizeof(double);
    struct Cut {
      Slab3 s;
      const Geo *g;
    };
    std::vector<Cut> cur;
    size_t used = 0;
    auto flush = [&] {
      if (cur.empty()) return;
      Group gr{};
      const int s0 = (int)slabs.size();
      for (auto &c : cur) slabs.push_back(c.s);
      for (int pass = 0; pass < 3; ++pass) {
        gr.item[pass] = (int)items.size();
        for (int k = 0; k < (int)cur.size(); ++k) add_items(pass, s0 + k, cur[k].s, *cur[k].g, t, mixed);
        gr.count[pass] = (int)items.size() - gr.item[pass];
      }
      groups.push_back(gr);
      bytes = std::max(bytes, used);
      cur.clear();
      used = 0;
    };
    for (const auto &sim : sims) {
      const Geo &g = sim.second;
      const int inner = g.n[2] - 4;
      const size_t plane = (size_t)g.st[2] * es * (kDerived3 + kFaces3);
      // equal slabs of at least `least` planes, each within the limit where it can be
      const int least = limit < kSlabBytes ? 1 : 4;
      const int most = std::max(least, (int)(limit / plane) - 4);
      const int cuts = std::max(1, std::min((inner + most - 1) / most, inner / least));
      for (int k = 0; k < cuts; ++k) {
        Slab3 s{};
        s.inst = sim.first;
        s.z0 = 2 + (int)((long long)inner * k / cuts);
        s.z1 = 2 + (int)((long long)inner * (k + 1) / cuts);
        s.pz0 = std::max(0, s.z0 - 3);
        s.pz1 = std::min(g.n[2], std::max(s.z1 + 3, 6));
        s.NP = (int)(((s.pz1 - s.pz0) * g.st[2] + 7) & ~7LL);
        s.NV = (int)(((s.z1 - s.z0 + 2) * g.st[2] + 7) & ~7LL);
        const size_t pb = align((size_t)s.NP * kDerived3 * es), vb = align((size_t)s.NV * kFaces3 * es);
        if (used + pb + vb > limit) flush();
        s.P = (void *)used;
        s.V = (void *)(used + pb);
        used += pb + vb;
        cur.push_back({s, &g});
      }
    }
    flush();
  }
  // Turn the offsets into addresses.
  void place(char *base) {
    for (auto &s : slabs) {
      s.P = base + (size_t)s.P;
      s.V = base + (size_t)s.V;
    }
  }

 private:
  static size_t align(size_t x) { return (x + 255) & ~(size_t)255; }
  void add_items(int pass, int slab, const Slab3 &s, const Geo &g, const int *t, bool mixed) {
    const long long nx = g.n[0] - 4, ny = g.n[1] - 4, nz = s.z1 - s.z0;
    auto chunks = [&](long long n, long long per, int by) {
      for (long long c = 0; c < (n + per - 1) / per; ++c) items.push_back({slab, (int)c, by, 0});
    };
    if (pass == 0) {
      chunks((s.pz1 - s.pz0) * g.st[2], kDeriveChunk, 0);
    } else if (pass == 1) {
      const int seg = face_seg(mixed);
      const long long zl = std::min(s.z1, g.n[2] - 3) - std::max(s.z0 - 1, 2) + 1;  // inner planes with x and y faces
      chunks(((nz + 1 + seg - 1) / seg) * nx * ny, kFaceSegs, 2);
      chunks(((g.n[1] - 3 + seg - 1) / seg) * nx * zl, kFaceSegs, 1);
      chunks((g.n[0] - 3) * ny * zl, kFaceChunk, 0);
    } else {
      for (int z = 0; z < (nz + t[2] - 1) / t[2]; ++z)
        for (int y = 0; y < (ny + t[1] - 1) / t[1]; ++y)
          for (int x = 0; x < (nx + t[0] - 1) / t[0]; ++x) items.push_back({slab, x, y, z});
    }
  }
};

// Cells of an advance item (in storage order, from the first inner row of the
// last dim on), and the number of a simulation's advance items.
constexpr int kAdvChunk = 256;
// Blocks per SM the advance kernel's registers are capped for, the fastest of
// 2..5 on a B200 (ms per step at 2, 3, 4, 5: 2-D mixed ensemble of 24 2.44, 2.20,
// 2.15, 2.22; 2-D FP64 ensemble of 12 1.23, 1.21, 1.25, 1.36; blast wave 128^3
// mixed 1.94, 1.86, 1.87, 2.00; 85^3 FP64 1.39, 1.44, 1.49, 1.65).
constexpr int advance_blocks(int D, bool mixed) { return mixed ? (D == 2 ? 4 : 3) : (D == 2 ? 3 : 2); }
inline int advance_items(const Geo &g, int D) {
  return (int)((g.N - 4 * g.st[D - 1] + kAdvChunk - 1) / kAdvChunk);
}

// Tile shapes and, in 2-D, occupancy targets (resident blocks per SM the
// register allocation is made for) the stage kernel is built for; the autotuner
// picks one.  In 3-D one terms kernel takes every shape: the ten variants are
// five shapes (those of the tile kernels that the numbers were given to), and
// min_blocks says nothing.
constexpr int kBatchVariants2 = 11;
constexpr int kBatchVariants3 = 10;
struct BatchVariant {
  int t[3];
  int min_blocks;
};
__host__ __device__ inline BatchVariant batch_variant(int D, int v) {
  if (D == 2) {
    switch (v) {
      case 1: return {{32, 8, 1}, 2};
      case 2: return {{8, 32, 1}, 2};
      case 3: return {{32, 16, 1}, 1};
      case 4: return {{16, 16, 1}, 3};
      case 5: return {{32, 8, 1}, 3};
      case 6: return {{16, 16, 1}, 4};
      case 7: return {{32, 8, 1}, 4};
      case 8: return {{16, 16, 1}, 5};
      case 9: return {{16, 8, 1}, 8};
      case 10: return {{32, 16, 1}, 2};
      default: return {{16, 16, 1}, 2};
    }
  }
  switch (v) {
    case 1: return {{16, 8, 2}, 2};
    case 2: return {{32, 4, 2}, 2};
    case 3: return {{8, 8, 4}, 3};
    case 4: return {{16, 8, 2}, 3};
    case 5: return {{8, 8, 4}, 4};
    case 6: return {{8, 8, 8}, 2};
    case 7: return {{16, 8, 4}, 2};
    case 8: return {{8, 8, 8}, 1};
    case 9: return {{16, 8, 4}, 1};
    default: return {{8, 8, 4}, 2};
  }
}

// Default variant of a single simulation and of an untuned batch (the
// serving loop's), per ndim and precision: in 2-D the fastest of the variants in
// B200 sweeps of RK stage 1 on 96 Orszag-Tang simulations 128^2..768^2 and on
// 48 driven atmosphere slices (the served mix).  In 3-D one terms kernel takes
// every tile shape; 32-wide tiles keep a warp's loads in whole lines (blast wave
// 128^3 mixed, ms per step: 32x4x2 1.86, 16x8x2 1.90, 16x8x4 1.91).  A batch
// and a single-simulation context on the same variant give the same bits.
__host__ __device__ inline int batch_default_variant(int D, bool mixed) {
  if (D == 2) return mixed ? 6 : 0;
  return 2;
}

__host__ __device__ inline void batch_tile_shape(int D, int v, int *t) {
  const BatchVariant b = batch_variant(D, v);
  t[0] = b.t[0];
  t[1] = b.t[1];
  t[2] = b.t[2];
}

// Do the 2-D mixed stage's tiles run one cell per thread (twice the threads of the
// pairs, one kernel for all occupancy targets)?  16x16 tiles, at most two of them
// per SM (us per step of a vortex, one cell / pairs: 12 tiles 50.4 / 63.1, 144
// 54.7 / 64.2, 256 68.2 / 70.5, 400 95.5 / 77.2, 1024 144 / 125).  The batch's list
// has the tiles of all its simulations.
__host__ __device__ inline bool batch_single_cells(int tx, int ty, int tiles, int sms) {
  return tx == 16 && ty == 16 && tiles <= 2 * sms;
}

// The variant that stands for those that launch what variant v does over `tiles`
// tiles: in 3-D the first of its shape, in 2-D mixed, where all 16x16 tiles run one
// cell per thread, the default.
__host__ __device__ inline int batch_alike(int D, bool mixed, int v, int tiles, int sms) {
  const BatchVariant b = batch_variant(D, v);
  if (D == 2) return mixed && batch_single_cells(b.t[0], b.t[1], tiles, sms) ? batch_default_variant(2, true) : v;
  for (int u = 0; u < v; ++u) {
    const BatchVariant a = batch_variant(3, u);
    if (a.t[0] == b.t[0] && a.t[1] == b.t[1] && a.t[2] == b.t[2]) return u;
  }
  return v;
}

}  // namespace smaug

namespace smaug_batchk {
// per (ndim, stencil type) translation units (batch_k{2,3}{f,d}.cu)
void launch_batch_stage_2f(int, const smaug::BatchInst *, const smaug::WorkItem *, int, int, int, cudaStream_t);
void launch_batch_stage_2d(int, const smaug::BatchInst *, const smaug::WorkItem *, int, int, int, cudaStream_t);
void launch_pass3_f(int, const smaug::BatchInst *, const smaug::Slab3 *, const smaug::WorkItem *,
                    const smaug::Plan3 &, int, int, cudaStream_t);
void launch_pass3_d(int, const smaug::BatchInst *, const smaug::Slab3 *, const smaug::WorkItem *,
                    const smaug::Plan3 &, int, int, cudaStream_t);
void launch_batch_advance_2f(const smaug::BatchInst *, const smaug::WorkItem *, int, int, int, cudaStream_t);
void launch_batch_advance_2d(const smaug::BatchInst *, const smaug::WorkItem *, int, int, int, cudaStream_t);
void launch_batch_advance_3f(const smaug::BatchInst *, const smaug::WorkItem *, int, int, int, cudaStream_t);
void launch_batch_advance_3d(const smaug::BatchInst *, const smaug::WorkItem *, int, int, int, cudaStream_t);
int batch_stage_occupancy_2f(int);
int batch_stage_occupancy_2d(int);
int batch_stage_occupancy_3f(int);
int batch_stage_occupancy_3d(int);

// Launch one RK stage (1..4) of a 2-D batch for every work item whose
// simulation takes the current step (work == nullptr: items are the tiles of
// simulation 0).  grid: persistent block count.
inline void launch_batch_stage2(bool mixed, int variant, const smaug::BatchInst *tab, const smaug::WorkItem *work,
                                int nwork, int stage, int grid, cudaStream_t st) {
  (mixed ? launch_batch_stage_2f : launch_batch_stage_2d)(variant, tab, work, nwork, stage, grid, st);
}
// One RK stage of 3-D simulations: the three passes of every group of the
// plan (slabs, items: its lists on the device; resident: blocks of the terms
// pass the device keeps resident).  Returns the number of launches.
inline int launch_pass3(bool mixed, int variant, const smaug::BatchInst *tab, const smaug::Slab3 *slabs,
                        const smaug::WorkItem *items, const smaug::Plan3 &plan, int stage, int resident,
                        cudaStream_t st) {
  (mixed ? launch_pass3_f : launch_pass3_d)(variant, tab, slabs, items, plan, stage, resident, st);
  return 3 * (int)plan.groups.size();
}
// The advance pass of RK stage `stage` (work == nullptr: the n chunks of
// simulation 0).
inline void launch_batch_advance(int D, bool mixed, const smaug::BatchInst *tab, const smaug::WorkItem *work, int n,
                                 int stage, int sms, cudaStream_t st) {
  if (D == 2)
    (mixed ? launch_batch_advance_2f : launch_batch_advance_2d)(tab, work, n, stage, sms, st);
  else
    (mixed ? launch_batch_advance_3f : launch_batch_advance_3d)(tab, work, n, stage, sms, st);
}
// Blocks per SM the stage kernel of (D, mixed, variant) can keep resident.
inline int batch_stage_occupancy(int D, bool mixed, int variant) {
  if (D == 2) return mixed ? batch_stage_occupancy_2f(variant) : batch_stage_occupancy_2d(variant);
  return mixed ? batch_stage_occupancy_3f(variant) : batch_stage_occupancy_3d(variant);
}
}  // namespace smaug_batchk
