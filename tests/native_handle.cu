// Host program of tests/test_gpu_native_handle.py: checks of a handle that the
// C ABI alone cannot set up.  Linked with the library's own objects, so that both
// share one CUDA runtime.  Usage: native_handle <check>; exits 0 when it holds.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <set>
#include <string>
#include <utility>
#include <vector>

#include <cuda_runtime.h>

#include "../include/sphg.h"
#include "../sph-simulations_gb300/csrc/sphg_internal.cuh"

// A kernel's attributes belong to the device that was current when they were set.
// With one device at hand the program plays two: it keeps, by the device it plays,
// which kernels may use more than 48 KB of shared memory, and refuses the launches
// that the device would refuse (the program is linked with --wrap of the calls it replaces).
static int fake_device = 0;
static int launched = 0;  // kernels of iterations, captured ones included
static std::set<std::pair<int, const void*>> large_memory;
extern "C" cudaError_t __real_cudaFuncSetAttribute(const void* f, cudaFuncAttribute attr, int value);
extern "C" cudaError_t __wrap_cudaFuncSetAttribute(const void* f, cudaFuncAttribute attr, int value) {
  if (attr == cudaFuncAttributeMaxDynamicSharedMemorySize) large_memory.insert({fake_device, f});
  return __real_cudaFuncSetAttribute(f, attr, value);
}
extern "C" cudaError_t __real_cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args);
extern "C" cudaError_t __wrap_cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  ++launched;
  if (c->dynamicSmemBytes > (48u << 10) && !large_memory.count({fake_device, f})) return cudaErrorInvalidValue;
  return __real_cudaLaunchKernelExC(c, f, args);
}
// Allocations that fail on request: the next `refuse_pinned` pinned ones, and device
// ones after the next `allow_device`.
static int refuse_pinned = 0;
extern "C" cudaError_t __real_cudaMallocHost(void** p, size_t bytes);
extern "C" cudaError_t __wrap_cudaMallocHost(void** p, size_t bytes) {
  return refuse_pinned-- > 0 ? cudaErrorMemoryAllocation : __real_cudaMallocHost(p, bytes);
}
static int allow_device = 1 << 30;
extern "C" cudaError_t __real_cudaMalloc(void** p, size_t bytes);
extern "C" cudaError_t __wrap_cudaMalloc(void** p, size_t bytes) {
  return allow_device-- <= 0 ? cudaErrorMemoryAllocation : __real_cudaMalloc(p, bytes);
}

namespace {

int failed(const char* what) {
  std::printf("%s: %s\n", what, sphg_last_error_string());
  return 1;
}

struct State {
  std::vector<double> x, y, vx, vy;
};
State lattice(int nx, int ny) {
  State s;
  for (int i = 0; i < nx * ny; ++i) {
    s.x.push_back((i % nx + 0.5) / nx);
    s.y.push_back((i / nx + 0.5) / ny);
    s.vx.push_back(std::sin(0.1 * i));
    s.vy.push_back(std::cos(0.1 * i));
  }
  return s;
}
sphg_params box(double h) {
  sphg_params p;
  sphg_default_params(&p);
  p.h = h;
  p.dt = 1e-4;
  p.lo[0] = p.lo[1] = 0.0;
  p.hi[0] = p.hi[1] = 1.0;
  return p;
}

// A small handle's iterations, and its state after them.
int small_run(int precision, std::vector<double>& out) {
  const State st = lattice(40, 30);
  const int64_t n = (int64_t)st.x.size();
  const sphg_params p = box(0.04);
  sphg_options o;
  sphg_default_options(&o);
  o.precision = precision;
  sphg_sim* s = nullptr;
  if (sphg_create(&p, &o, n, &s) != SPHG_OK) return failed("create");
  out.assign(4 * n, 0.0);
  const int bad = sphg_upload(s, st.x.data(), st.y.data(), st.vx.data(), st.vy.data(), nullptr) != SPHG_OK ||
                  sphg_preloop(s, nullptr) != SPHG_OK || sphg_step(s, 10, nullptr) != SPHG_OK ||
                  sphg_download(s, &out[0], &out[n], &out[2 * n], &out[3 * n], nullptr, nullptr, nullptr, nullptr,
                                nullptr) != SPHG_OK;
  if (bad) failed("run");
  sphg_destroy(s);
  return bad;
}

// Handles on two devices: the second is played by the wrapped calls.
int devices() {
  for (int precision : {SPHG_PRECISION_PLAIN, SPHG_PRECISION_SPLIT}) {
    std::vector<double> a, b;
    fake_device = 0;
    if (small_run(precision, a)) return 1;
    fake_device = 1;
    if (small_run(precision, b)) return 1;
    if (std::memcmp(a.data(), b.data(), a.size() * sizeof(double))) return failed("another result");
  }
  return 0;
}

struct Lists {
  std::vector<int64_t> offs;
  std::vector<int32_t> idx;
  int64_t total = 0;
  sphg_status count(sphg_sim* s) { return sphg_neighbor_lists(s, nullptr, nullptr, &total, nullptr); }
  sphg_status get(sphg_sim* s, int64_t n) {
    sphg_status st = count(s);
    if (st != SPHG_OK) return st;
    offs.assign(n + 1, -1);
    idx.assign(total, -1);
    return sphg_neighbor_lists(s, offs.data(), idx.data(), &total, nullptr);
  }
};
// A computed state of n = 200 particles: two blocks of the list assembly.
constexpr int64_t kListN = 200;
sphg_sim* list_handle() {
  const State st = lattice(20, 10);
  const sphg_params p = box(0.12);
  sphg_sim* s = nullptr;
  if (sphg_create(&p, nullptr, kListN, &s) != SPHG_OK ||
      sphg_upload(s, st.x.data(), st.y.data(), st.vx.data(), st.vy.data(), nullptr) != SPHG_OK ||
      sphg_preloop(s, nullptr) != SPHG_OK)
    std::exit(failed("handle"));
  return s;
}

// The assembly's blocks take the numbers 1 and 2 instead of 0 and 1 (its words are
// padded to 256 bytes), so their look-back waits for a block that never comes and
// gives up: the export says so, the state and the next export are as they were.
int lookback() {
  sphg_sim* s = list_handle();
  Lists a, b, c;
  if (a.get(s, kListN) != SPHG_OK) return failed("export");
  const uint32_t one = 1;
  if (cudaMemcpy(s->list_ctl, &one, sizeof(one), cudaMemcpyHostToDevice) != cudaSuccess) return failed("copy");
  b.offs.assign(kListN + 1, -1);
  b.idx.assign(a.total, -1);
  if (sphg_neighbor_lists(s, b.offs.data(), b.idx.data(), &b.total, nullptr) != SPHG_TIMEOUT)
    return failed("a wait that gave up is not reported");
  if (c.get(s, kListN) != SPHG_OK) return failed("the next export");
  if (c.offs != a.offs || c.idx != a.idx) return failed("the next export is another");
  std::vector<double> x(kListN);
  if (sphg_download(s, x.data(), nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr) != SPHG_OK)
    return failed("the state after it");
  return sphg_destroy(s);
}

// The first export gets its device buffer but not its pinned one; the second both.
int pinned() {
  sphg_sim* s = list_handle();
  Lists a;
  refuse_pinned = 1;
  if (a.count(s) != SPHG_OOM) return failed("an allocation that failed is not reported");
  refuse_pinned = 0;
  if (a.get(s, kListN) != SPHG_OK) return failed("the export after it");
  if (a.total < kListN || a.offs[kListN] != a.total) return failed("its lists");
  return sphg_destroy(s);
}

// A call for the total needs no room for the entries.
int count_only() {
  sphg_sim* s = list_handle();
  Lists a;
  allow_device = 1;  // the offsets
  if (a.count(s) != SPHG_OK || a.total < kListN) return failed("the total");
  a.idx.assign(a.total, -1);
  if (sphg_neighbor_lists(s, nullptr, a.idx.data(), &a.total, nullptr) != SPHG_OOM)
    return failed("an allocation that failed is not reported");
  allow_device = 1 << 30;
  if (a.get(s, kListN) != SPHG_OK) return failed("the export after it");
  if (a.offs[kListN] != a.total || a.idx[a.total - 1] < 0) return failed("its lists");
  return sphg_destroy(s);
}

// The library's counts of launches against those made: graphs hold what their
// iterations launch when they sort fully.
int launches() {
  for (int n1 : {130, 30})  // graphs; one cluster
    for (int graph : {1, 0})
      for (int resort : {1, 0}) {
        const State st = lattice(n1, n1);
        const sphg_params p = box(1.3 / n1);
        sphg_options o;
        sphg_default_options(&o);
        o.use_graph = graph;
        o.resort = resort;
        sphg_sim* s = nullptr;
        launched = 0;
        if (sphg_create(&p, &o, (int64_t)n1 * n1, &s) != SPHG_OK) return failed("create");
        const int made = launched;
        if (sphg_upload(s, st.x.data(), st.y.data(), st.vx.data(), st.vy.data(), nullptr) != SPHG_OK ||
            sphg_preloop(s, nullptr) != SPHG_OK)
          return failed("run");
        launched = 0;
        int32_t rs[3];
        if (sphg_step(s, 1, nullptr) != SPHG_OK || sphg_get_debug(s, SPHG_DBG_RESORT, rs, nullptr) != SPHG_OK)
          return failed("step");
        const int full = sphg_launches_per_step(s), merged = full - rs[2];
        std::printf("%d %d %d: made %d step %d full %d merged %d\n", n1, graph, resort, made, launched, full, merged);
        if (!graph) {
          if (launched != full || merged != full) return failed("launches without a graph");
        } else if (n1 == 130) {  // two graphs, the second with its header (in the branch too)
          if (made != 2 * full + (resort ? 2 : 1) || merged != (resort ? 3 : full)) return failed("launches of a graph");
        } else if (resort && (launched != 1 || merged != 3)) {  // counted as its graph
          return failed("launches of a cluster");
        }
        sphg_destroy(s);
      }
  return 0;
}

}  // namespace

int main(int argc, char** argv) {
  const std::string check = argc > 1 ? argv[1] : "";
  if (check == "devices") return devices();
  if (check == "lookback") return lookback();
  if (check == "pinned") return pinned();
  if (check == "count_only") return count_only();
  if (check == "launches") return launches();
  std::printf("unknown check\n");
  return 2;
}
