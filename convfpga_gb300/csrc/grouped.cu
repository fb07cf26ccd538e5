// Uneven batches as one CUDA graph of per-size launches.
//
// Jobs of the same cube size run together: each of the seven passes of a convolution
// (filter x, signal x, filter y, signal y, fused z, signal y-inv, signal x-inv) is one
// launch of the TMA-fed pass kernel over every job of that size, in table mode: each job
// brings its own tensor maps and destination base, so the jobs' cubes may sit anywhere.
// The size classes run as parallel branches of one CUDA graph, captured once per
// sequence of job sizes and replayed on every call; tensor maps are re-encoded and
// uploaded only when a job's buffers move. When the plan fuses the x and y passes of
// N = 256 or 128 (L2-staged pass), that class runs filter x+y, signal x+y, fused z and
// inverse y+x instead: three table-mode launches of the fused pass around the z launch. With
// the two-pass transform in the plan, no job of the class in place, and tiles the faster form
// beside the other classes (uneven_grouped), it runs that: filters and signals forward (signals
// through their outputs), middle pass into the spectra's workspace, inverse; such classes run
// in turn.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "engine_internal.h"
#include "passes.cuh"

namespace convgpu {
namespace {

// rows(filter) rows(signal) rows(out) y(spec) y(out) z(out) z(spec), then the fused x+y
// pass's rows maps (N = 256 and 128): filter, signal, out; then the two-pass transform's
// maps of cubes in tile order: spectrum, out
constexpr int kKinds = 12;
// kXyTiles: filters and signals forward in one launch; kXyTilesOrdered: one after the other,
// where a filter lies among the outputs. kWhole: N = 16, one launch.
enum XyForm { kXySeparate = 0, kXyStaged = 1, kXyTiles = 2, kXyTilesOrdered = 3, kWhole = 4 };
static bool tiles(XyForm f) { return f == kXyTiles || f == kXyTilesOrdered; }

struct SizeGroup {
  int n = 0;
  std::vector<int> jobs;
  CUtensorMap *d_maps = nullptr;  // [kind][job in group]
  float2 **d_dsts = nullptr;      // [0][j] spectrum, [1][j] output, [2][j] filter, [3][j] signal
  std::vector<CUtensorMap> h_maps;
  std::vector<float2 *> h_dsts;
  unsigned *d_ctr = nullptr;  // dependency counters of the fused x+y launches
  XyForm xy = kXySeparate;
};

struct GPlan {
  std::vector<int> sizes;
  std::vector<SizeGroup> groups;
  float2 *d_spec = nullptr;
  std::vector<size_t> spec_off;
  std::vector<const void *> ptr_key;  // buffers the uploaded maps describe
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  cudaEvent_t done = nullptr;
  unsigned long long kernels = 0;  // the graph's
  bool launched = false;
  ~GPlan() {
    if (done) cudaEventDestroy(done);
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    for (auto &g : groups) {
      if (g.d_maps) cudaFree(g.d_maps);
      if (g.d_dsts) cudaFree(g.d_dsts);
      if (g.d_ctr) cudaFree(g.d_ctr);
    }
    if (d_spec) cudaFree(d_spec);
  }
};

cudaError_t count_kernels(cudaGraph_t graph, unsigned long long &kernels) {
  size_t n = 0;
  cudaError_t e = cudaGraphGetNodes(graph, nullptr, &n);
  std::vector<cudaGraphNode_t> nodes(n);
  if (e == cudaSuccess) e = cudaGraphGetNodes(graph, nodes.data(), &n);
  for (size_t i = 0; i < n && e == cudaSuccess; ++i) {
    cudaGraphNodeType t;
    if ((e = cudaGraphNodeGetType(nodes[i], &t)) == cudaSuccess) kernels += t == cudaGraphNodeTypeKernel;
  }
  return e;
}

std::mutex g_mu;
// key: job sizes, normalize + 2 * (form of each size, base 5)
std::map<std::pair<std::vector<int>, int>, std::unique_ptr<GPlan>> g_plans;

cudaError_t enqueue_group(const SizeGroup &g, float scale, const float2 *tw512, cudaStream_t s) {
  const int k = (int)g.jobs.size();
  const CUtensorMap *m = g.d_maps;
  float2 *const *spec = g.d_dsts;
  float2 *const *out = g.d_dsts + k;
  cudaError_t e;
  if (g.xy == kWhole) return launch_cube16_table(g.d_dsts + 3 * k, g.d_dsts + 2 * k, out, k, scale, s);
  if (tiles(g.xy)) {
    const int both = g.xy == kXyTiles ? 2 * k : k;  // filters, then signals
    if ((e = launch_tp_fwd_table(g.n, g.d_dsts + 2 * k, m + 10 * k, both, tw512, s)) != cudaSuccess) return e;
    if (both == k && (e = launch_tp_fwd_table(g.n, g.d_dsts + 3 * k, m + 11 * k, k, tw512, s)) != cudaSuccess) return e;
    if ((e = launch_tp_mid_table(g.n, out, spec, spec, k, tw512, s)) != cudaSuccess) return e;
    return launch_tp_inv_table(g.n, m + 10 * k, out, k, scale, tw512, s);
  }
  if (g.xy == kXyStaged) {
    unsigned *st = device_status_address();
    if ((e = launch_xy_l2_table(g.n, m + 7 * k, spec, k, false, 1.f, tw512, st, g.d_ctr, s)) != cudaSuccess)
      return e;
    if ((e = launch_xy_l2_table(g.n, m + 8 * k, out, k, false, 1.f, tw512, st, g.d_ctr, s)) != cudaSuccess)
      return e;
    if ((e = launch_axis_pass_table(g.n, 2, OP_CONV_FZ, m + 5 * k, m + 6 * k, out, k, 1.f, tw512, s)) != cudaSuccess)
      return e;
    return launch_xy_l2_table(g.n, m + 9 * k, out, k, true, scale, tw512, st, g.d_ctr, s);
  }
  if ((e = launch_axis_pass_table(g.n, 0, OP_FWD, m + 0 * k, nullptr, spec, k, 1.f, tw512, s)) != cudaSuccess) return e;
  if ((e = launch_axis_pass_table(g.n, 0, OP_FWD, m + 1 * k, nullptr, out, k, 1.f, tw512, s)) != cudaSuccess) return e;
  if ((e = launch_axis_pass_table(g.n, 1, OP_FWD, m + 3 * k, nullptr, spec, k, 1.f, tw512, s)) != cudaSuccess) return e;
  if ((e = launch_axis_pass_table(g.n, 1, OP_FWD, m + 4 * k, nullptr, out, k, 1.f, tw512, s)) != cudaSuccess) return e;
  if ((e = launch_axis_pass_table(g.n, 2, OP_CONV_FZ, m + 5 * k, m + 6 * k, out, k, 1.f, tw512, s)) != cudaSuccess)
    return e;
  if ((e = launch_axis_pass_table(g.n, 1, OP_INV, m + 4 * k, nullptr, out, k, 1.f, tw512, s)) != cudaSuccess) return e;
  return launch_axis_pass_table(g.n, 0, OP_INV, m + 2 * k, nullptr, out, k, scale, tw512, s);
}

// Form of each size class, and where they stand.
struct Forms {
  XyForm of[6] = {};
  static int index(int n) { return n == 16 ? 0 : (n == 32 ? 1 : (n == 64 ? 2 : (n == 128 ? 3 : (n == 256 ? 4 : 5)))); }
};

cudaError_t build(GPlan &p, bool normalize, const Forms &forms, const float2 *tw512) {
  std::map<int, int> idx;
  for (int j = 0; j < (int)p.sizes.size(); ++j) {
    const int n = p.sizes[j];
    if (!idx.count(n)) {
      idx[n] = (int)p.groups.size();
      p.groups.emplace_back();
      p.groups.back().n = n;
    }
    p.groups[idx[n]].jobs.push_back(j);
  }
  // largest cubes first: their launches are the long ones
  std::sort(p.groups.begin(), p.groups.end(), [](const SizeGroup &a, const SizeGroup &b) { return a.n > b.n; });
  size_t spec = 0;
  p.spec_off.resize(p.sizes.size());
  for (size_t j = 0; j < p.sizes.size(); ++j) {
    p.spec_off[j] = spec;
    spec += (size_t)p.sizes[j] * p.sizes[j] * p.sizes[j];
  }
  cudaError_t e;
  if ((e = allocate((void **)&p.d_spec, spec * sizeof(float2))) != cudaSuccess) return e;
  for (auto &g : p.groups) {
    const size_t k = g.jobs.size();
    g.h_maps.resize(kKinds * k);
    g.h_dsts.resize(4 * k);
    if ((e = cudaMalloc(&g.d_maps, sizeof(CUtensorMap) * kKinds * k)) != cudaSuccess) return e;
    if ((e = cudaMalloc(&g.d_dsts, sizeof(float2 *) * 4 * k)) != cudaSuccess) return e;
    g.xy = forms.of[Forms::index(g.n)];
    if (g.xy == kWhole && (e = prepare_cube16()) != cudaSuccess) return e;
    if (tiles(g.xy) && (e = prepare_tp(g.n)) != cudaSuccess) return e;
    if (g.xy == kXyStaged) {
      if ((e = prepare_xy_l2(g.n)) != cudaSuccess) return e;
      if ((e = cudaMalloc(&g.d_ctr, xy_l2_counter_bytes(g.n, (int)k))) != cudaSuccess) return e;
    }
  }
  if ((e = cudaEventCreateWithFlags(&p.done, cudaEventDisableTiming)) != cudaSuccess) return e;
  for (auto &g : p.groups)
    if ((e = prepare_table_launches(g.n)) != cudaSuccess) return e;
  // Capture: one branch per size class that runs the three-axis passes.
  cudaStream_t cap;
  if ((e = cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking)) != cudaSuccess) return e;
  std::vector<cudaStream_t> br(p.groups.size(), nullptr);
  std::vector<cudaEvent_t> ev(p.groups.size() + 1, nullptr);
  for (auto &b : br)
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&b, cudaStreamNonBlocking);
  for (auto &v : ev)
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    // Classes of the two-pass transform run one after another: a CTA of theirs holds an SM, so
    // two side by side leave each other's CTAs waiting (two cubes of 256^3, four of 128^3, ten
    // of 64^3 and of 32^3: 725 us side by side, 666 in turn). The others, and a class of 32^3,
    // whose launches are short, run beside them, a branch each.
    auto in_turn = [](const SizeGroup &g) { return tiles(g.xy) && g.n > 32; };
    auto scale_of = [&](int n) { return normalize ? (float)(1.0 / ((double)n * n * n)) : 1.0f; };
    cudaEventRecord(ev.back(), cap);
    for (auto &g : p.groups)
      if (in_turn(g) && e == cudaSuccess) e = enqueue_group(g, scale_of(g.n), tw512, cap);
    for (size_t gi = 0; gi < p.groups.size() && e == cudaSuccess; ++gi) {
      if (in_turn(p.groups[gi])) continue;
      cudaStreamWaitEvent(br[gi], ev.back(), 0);
      e = enqueue_group(p.groups[gi], scale_of(p.groups[gi].n), tw512, br[gi]);
      cudaEventRecord(ev[gi], br[gi]);
      cudaStreamWaitEvent(cap, ev[gi], 0);
    }
    cudaError_t e2 = cudaStreamEndCapture(cap, &p.graph);
    if (e == cudaSuccess) e = e2;
  }
  if (e == cudaSuccess) e = cudaGraphInstantiate(&p.exec, p.graph, 0);
  if (e == cudaSuccess) e = count_kernels(p.graph, p.kernels);
  for (auto b : br)
    if (b) cudaStreamDestroy(b);
  for (auto v : ev)
    if (v) cudaEventDestroy(v);
  cudaStreamDestroy(cap);
  return e;
}

}  // namespace

int uneven_grouped(const UnevenJob *jobs, unsigned njobs, const void *d_sig, const void *d_filt, void *d_out,
                   bool normalize, const float2 *tw512, cudaStream_t stream, std::string &err) {
  if (njobs == 0) return 0;
  std::vector<int> sizes(njobs);
  std::vector<const void *> ptrs(3 * njobs);
  for (unsigned j = 0; j < njobs; ++j) {
    sizes[j] = (int)jobs[j].n;
    ptrs[3 * j] = (const float2 *)d_sig + jobs[j].sig_off;
    ptrs[3 * j + 1] = (const float2 *)d_filt + jobs[j].filt_off;
    ptrs[3 * j + 2] = (const float2 *)d_out + jobs[j].out_off;
    for (int q = 0; q < 3; ++q)
      if ((reinterpret_cast<uintptr_t>(ptrs[3 * j + q]) & 15u) != 0) {
        err = "uneven batch: a cube is not 16-byte aligned";
        return -5;  // caller falls back to one job at a time
      }
  }
  std::lock_guard<std::mutex> lk(g_mu);
  // What decides a class's form: its jobs, whether their signals are apart from their outputs,
  // and whether no filter lies among the outputs (by the ranges they span).
  struct Class {
    int jobs = 0;
    bool apart = true;
    uintptr_t flo = ~(uintptr_t)0, fhi = 0, olo = ~(uintptr_t)0, ohi = 0;
    bool filters_apart() const { return fhi <= olo || ohi <= flo; }
  } cls[6];
  for (unsigned j = 0; j < njobs; ++j) {
    Class &c = cls[Forms::index(sizes[j])];
    const uintptr_t bytes = (uintptr_t)sizes[j] * sizes[j] * sizes[j] * sizeof(float2),
                    su = reinterpret_cast<uintptr_t>(ptrs[3 * j]), f = reinterpret_cast<uintptr_t>(ptrs[3 * j + 1]),
                    o = reinterpret_cast<uintptr_t>(ptrs[3 * j + 2]);
    ++c.jobs;
    if (su < o + bytes && o < su + bytes) c.apart = false;
    c.flo = std::min(c.flo, f), c.fhi = std::max(c.fhi, f + bytes);
    c.olo = std::min(c.olo, o), c.ohi = std::max(c.ohi, o + bytes);
  }
  auto of_size = [&](int n) { return cls[Forms::index(n)].jobs; };
  int classes = 0;  // sizes present, 16 aside
  for (int i = 1; i < 6; ++i) classes += cls[i].jobs > 0;
  // Whether tiles are the faster form of a class, given those beside it (the axis passes' CTAs
  // are small and fill in beside other kernels). us, tiles / axis passes, with the autotuned
  // shapes and the default ones: 32^3 alone x16 32.9 / 35.0 and 32.9 / 35.0, x20 38.5 / 39.1 and
  // 37.5 / 37.1, x28 45.3 / 39.3 and 44.7 / 39.2, x50 64.5 / 52.1 and 64.0 / 51.6, x170 149.7 /
  // 150.6 and 148.7 / 148.6, x300 224.8 / 258.4; 64^3 alone x1 22.7 / 28.8, x20 111.5 / 143.1. Beside
  // each other both in tiles / both by axes: 64^3 x2 and 32^3 x1 35 / 40, x2 and x5 47 / 42, x4 and
  // x20 70 / 61, x8 and x40 110 / 96. 64^3 beside 32^3 by axes: x12 and x12 104 / 100, x20 and x20
  // 142 / 157; beside two of 128^3 x8 138 / 144, x12 158 / 170. One cube of 128^3 beside both by
  // axes: 64^3 x4 and 32^3 x5 102 / 92, 32^3 x10 64 / 70, x40 96 / 90.
  const bool few32 = of_size(32) <= 2 && of_size(128) + of_size(256) + of_size(512) == 0;
  const bool tiles64 = classes == 1 || few32 || of_size(64) >= (of_size(32) ? 14 : 8);
  auto in_tiles = [&](int n) {
    if (n == 32) return few32 || (classes == 1 && (of_size(n) <= 20 || of_size(n) >= 170));
    if (n == 64) return tiles64;
    return n != 128 || of_size(n) > 1 || tiles64 || (of_size(64) < 2 && of_size(32) < 32);
  };
  // The L2-staged variant (1) and the two-pass transform (3) have table modes. The latter
  // takes signals through their outputs, so a class with a job in place (or partly so) runs
  // the former, as does every class when tensor maps are switched off; one cube of 128^3
  // runs separate passes, beside others 89 us where the staged pass takes 100.
  auto form = [&](int n) {
    const int v = get_pass_variant(n, kKindXy);
    const Class &c = cls[Forms::index(n)];
    if (v == kXyTwoPass && tma_enabled() && c.apart && in_tiles(n)) return c.filters_apart() ? kXyTiles : kXyTilesOrdered;
    if (n < 128 || (v != 1 && v != kXyTwoPass)) return kXySeparate;
    if (v == kXyTwoPass && n == 128 && c.jobs == 1) return kXySeparate;
    if (v == kXyTwoPass && prepare_xy_l2(n) != cudaSuccess) {  // no memory for its ring
      cudaGetLastError();
      return kXySeparate;
    }
    return kXyStaged;
  };
  Forms forms;
  for (int n : {32, 64, 128, 256})
    if (of_size(n) > 0) forms.of[Forms::index(n)] = form(n);
  // 16^3 jobs run whole, in any order
  forms.of[0] = of_size(16) > 0 && cls[0].filters_apart() ? kWhole : kXySeparate;
  int form_key = 0;
  for (XyForm f : forms.of) form_key = 5 * form_key + f;
  auto key = std::make_pair(sizes, (normalize ? 1 : 0) + 2 * form_key);
  auto it = g_plans.find(key);
  if (it == g_plans.end()) {
    auto p = std::make_unique<GPlan>();
    p->sizes = sizes;
    cudaError_t e = build(*p, normalize, forms, tw512);
    if (e != cudaSuccess) {
      err = std::string("uneven grouped plan: ") + cudaGetErrorString(e);
      cudaGetLastError();
      return e == cudaErrorMemoryAllocation ? -4 : -3;
    }
    it = g_plans.emplace(key, std::move(p)).first;
  }
  GPlan &p = *it->second;
  cudaError_t e = cudaSuccess;
  if (p.ptr_key != ptrs) {
    // The previous replay may still read the maps being replaced.
    if (p.launched) cudaEventSynchronize(p.done);
    for (auto &g : p.groups) {
      const size_t k = g.jobs.size();
      for (size_t v = 0; v < k; ++v) {
        const int j = g.jobs[v];
        const void *sg = ptrs[3 * j], *ft = ptrs[3 * j + 1], *ot = ptrs[3 * j + 2];
        float2 *sp = p.d_spec + p.spec_off[j];
        bool ok = encode_table_map(&g.h_maps[0 * k + v], ft, g.n, 0) && encode_table_map(&g.h_maps[1 * k + v], sg, g.n, 0) &&
                  encode_table_map(&g.h_maps[2 * k + v], ot, g.n, 0) && encode_table_map(&g.h_maps[3 * k + v], sp, g.n, 1) &&
                  encode_table_map(&g.h_maps[4 * k + v], ot, g.n, 1) && encode_table_map(&g.h_maps[5 * k + v], ot, g.n, 2) &&
                  encode_table_map(&g.h_maps[6 * k + v], sp, g.n, 2);
        if (ok && tiles(g.xy))
          ok = tp_encode_tiles(&g.h_maps[10 * k + v], sp, g.n, 1) && tp_encode_tiles(&g.h_maps[11 * k + v], ot, g.n, 1);
        if (ok && g.xy == kXyStaged)
          ok = encode_xy_table_map(&g.h_maps[7 * k + v], ft, g.n) &&
               encode_xy_table_map(&g.h_maps[8 * k + v], sg, g.n) && encode_xy_table_map(&g.h_maps[9 * k + v], ot, g.n);
        if (!ok) {
          err = "uneven batch: tensor map encoding failed";
          return -5;
        }
        g.h_dsts[v] = sp;
        g.h_dsts[k + v] = (float2 *)ot;
        g.h_dsts[2 * k + v] = (float2 *)const_cast<void *>(ft);
        g.h_dsts[3 * k + v] = (float2 *)const_cast<void *>(sg);
      }
      // pageable sources: each call returns once the host data is staged
      e = cudaMemcpyAsync(g.d_maps, g.h_maps.data(), sizeof(CUtensorMap) * g.h_maps.size(), cudaMemcpyHostToDevice,
                          stream);
      if (e == cudaSuccess)
        e = cudaMemcpyAsync(g.d_dsts, g.h_dsts.data(), sizeof(float2 *) * g.h_dsts.size(), cudaMemcpyHostToDevice,
                            stream);
      if (e != cudaSuccess) break;
    }
    if (e == cudaSuccess) p.ptr_key = ptrs;
  }
  if (e == cudaSuccess) e = cudaGraphLaunch(p.exec, stream);
  if (e == cudaSuccess) e = cudaEventRecord(p.done, stream);
  if (e != cudaSuccess) {
    err = std::string("uneven grouped launch: ") + cudaGetErrorString(e);
    return -3;
  }
  p.launched = true;
  count_launches(p.kernels);
  return 0;
}

void release_grouped_plans() {
  std::lock_guard<std::mutex> lk(g_mu);
  g_plans.clear();
}

}  // namespace convgpu
