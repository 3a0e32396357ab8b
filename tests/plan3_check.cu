// The 3-D plan and its workspace against an allocator with a budget: prints one
// line per check, exits 1 where one fails (compiled and run by test_plan3.py; no GPU).
#include <cstdio>
#include <map>

#include "smaug_batch.cuh"

using namespace smaug;

static Geo grid(int a, int b, int c) {
  Geo g{};
  g.n[0] = a;
  g.n[1] = b;
  g.n[2] = c;
  g.st[0] = 1;
  g.st[1] = a;
  g.st[2] = (long long)a * b;
  g.N = g.st[2] * c;
  return g;
}

static int bad = 0;
static void check(bool ok, const char *what) {
  std::printf("%s %s\n", ok ? "ok  " : "FAIL", what);
  bad += !ok;
}

// Every inner plane in one slab, slabs and groups within the workspace, halos in the grid.
static bool covers(const Plan3 &p, const std::vector<std::pair<int, Geo>> &sims) {
  std::map<int, int> next;
  for (auto &s : sims) next[s.first] = 2;
  for (auto &s : p.slabs) {
    const Geo *g = nullptr;
    for (auto &x : sims)
      if (x.first == s.inst) g = &x.second;
    if (!g || s.z0 != next[s.inst] || s.z1 <= s.z0) return false;
    next[s.inst] = s.z1;
    const int need0 = s.z0 == 2 ? 0 : s.z0 - 3, need1 = std::min(g->n[2], s.z0 == 2 ? std::max(s.z1 + 3, 6) : s.z1 + 3);
    if (s.pz0 > need0 || s.pz1 < need1 || s.pz0 < 0 || s.pz1 > g->n[2]) return false;
    if (s.NP < (s.pz1 - s.pz0) * g->st[2] || s.NV < (s.z1 - s.z0 + 2) * g->st[2]) return false;
  }
  for (auto &x : sims)
    if (next[x.first] != x.second.n[2] - 2) return false;
  return true;
}

struct Device {  // an allocator with a budget
  size_t budget, used = 0;
  std::map<char *, size_t> live;
  int allocs = 0, frees = 0, next = 1;
  cudaError_t alloc(void **p, size_t n) {
    if (used + n > budget) return cudaErrorMemoryAllocation;
    used += n;
    char *q = (char *)(size_t)(next++ * 4096);
    live[q] = n;
    *p = q;
    ++allocs;
    return cudaSuccess;
  }
  void release(char *p) {
    used -= live.at(p);
    live.erase(p);
    ++frees;
  }
};

int main() {
  const int t[3] = {32, 4, 2};
  const size_t MB = (size_t)1 << 20;
  using Sims = std::vector<std::pair<int, Geo>>;
  // thinner slabs under a lower limit, four planes at the usual one
  for (const Geo &g : {grid(516, 516, 36), grid(40, 30, 10), grid(260, 200, 25)})
    for (bool mixed : {true, false})
      for (size_t limit : {kSlabBytes, 64 * MB, 16 * MB, 4 * MB}) {
        Plan3 p;
        const Sims sims = {{0, g}, {3, grid(34, 20, 11)}};
        p.build(sims, t, mixed, limit);
        const size_t es = mixed ? 4 : 8, one = (size_t)g.st[2] * es * (7 * kDerived3 + 3 * kFaces3) + 65536;
        const size_t four = (size_t)g.st[2] * es * (10 * kDerived3 + 6 * kFaces3) + 65536;
        char what[160];
        std::snprintf(what, sizeof what, "%d x %d x %d %s limit %zu MB: %.1f MB in %zu slabs", g.n[0], g.n[1], g.n[2],
                      mixed ? "mixed" : "fp64", limit / MB, p.bytes / 1e6, p.slabs.size());
        check(covers(p, sims) && p.bytes <= std::max(limit, limit < kSlabBytes ? one : four), what);
      }
  auto fit = [&](Device &d, Plan3 &p, Workspace3 &ws, const Sims &sims, size_t want = 0) {
    return p.fit(
        ws, sims, t, true, want, [&](void **q, size_t n) { return d.alloc(q, n); }, [&](char *q) { d.release(q); });
  };
  {  // plenty: a batch that grows allocates few times and ends at the limit
    Device d{4096 * MB};
    Plan3 p;
    Workspace3 ws;
    Sims sims;
    bool ok = true;
    for (int k = 0; k < 40; ++k) {
      sims.push_back({k, grid(68, 68, 68)});
      ok = ok && fit(d, p, ws, sims) == cudaSuccess && covers(p, sims) && p.bytes <= ws.bytes;
    }
    check(ok && ws.bytes <= kSlabBytes && d.allocs <= 6 && d.live.size() == 1, "growing batch, plenty of memory");
  }
  {  // with a first size that fits the rest: one allocation
    Device d{4096 * MB};
    Plan3 p;
    Workspace3 ws;
    Sims sims;
    for (int k = 0; k < 8; ++k) {
      sims.push_back({k, grid(68, 68, 68)});
      fit(d, p, ws, sims, 500 * MB);
    }
    check(d.allocs == 1 && ws.bytes >= 8 * 50 * MB, "growing batch, first size for all");
  }
  {  // the memory goes meanwhile: the workspace in use is kept, nothing is freed, and it is remembered
    Device d{200 * MB};
    Plan3 p;
    Workspace3 ws;
    Sims sims = {{0, grid(68, 68, 68)}};
    bool ok = fit(d, p, ws, sims) == cudaSuccess;
    d.budget = d.used;  // somebody else took the rest
    const char *first = ws.p;
    for (int k = 1; k < 6; ++k) {
      sims.push_back({k, grid(68, 68, 68)});
      ok = ok && fit(d, p, ws, sims) == cudaSuccess && ws.p == first && covers(p, sims) && p.bytes <= ws.bytes;
    }
    check(ok && d.frees == 0 && d.allocs == 1 && ws.limit == ws.bytes && p.groups.size() > 1, "memory gone: workspace kept");
  }
  {  // little from the start: the limit that succeeded is kept, later plans do not try the larger ones again
    Device d{40 * MB};
    Plan3 p;
    Workspace3 ws;
    Sims sims = {{0, grid(132, 132, 132)}};
    bool ok = fit(d, p, ws, sims) == cudaSuccess && covers(p, sims) && ws.limit < kSlabBytes;
    const int a = d.allocs;
    sims.push_back({1, grid(132, 132, 132)});
    ok = ok && fit(d, p, ws, sims) == cudaSuccess && covers(p, sims) && p.bytes <= ws.bytes;
    check(ok && d.allocs == a, "little memory from the start");
  }
  {  // the one in use is too small for the thinnest slab of a new member and there is no room beside it
    Device d{60 * MB};
    Plan3 p;
    Workspace3 ws;
    Sims sims = {{0, grid(60, 60, 60)}};
    bool ok = fit(d, p, ws, sims) == cudaSuccess;
    sims.push_back({1, grid(240, 240, 20)});
    ok = ok && fit(d, p, ws, sims) == cudaSuccess && covers(p, sims) && d.live.size() == 1;
    check(ok && d.frees == 1, "too small: replaced");
  }
  {  // none: an error, and nothing held; with memory again it works
    Device d{1 * MB};
    Plan3 p;
    Workspace3 ws;
    const Sims sims = {{0, grid(132, 132, 132)}};
    bool ok = fit(d, p, ws, sims) == cudaErrorMemoryAllocation && !ws.p && d.live.empty();
    d.budget = 4096 * MB;
    ok = ok && fit(d, p, ws, sims) == cudaSuccess && p.bytes <= ws.bytes;
    check(ok, "no memory: refused, and later taken");
  }
  return bad != 0;
}
