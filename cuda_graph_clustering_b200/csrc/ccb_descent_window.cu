// Instances and launcher of the windowed descent (ccb_descent_window.cuh).
#include <cuda_runtime.h>

#include "ccb_descent_window.cuh"
#include "ccb_plans.h"

namespace ccb {
namespace {

template <int K, int kCap, bool S, bool kHalf, typename GainT>
cudaError_t Go(const SmallKPlan& p, const DescentArgs<GainT>& a, int grid, cudaStream_t st, bool configure) {
  auto kernel = k_descent_window<K, kCap, S, kHalf, GainT>;
  if (configure) return RaiseDynamicSmem(kernel, p.smem_bytes);
  if (grid > 0) kernel<<<grid, kWindowThreads, p.smem_bytes, st>>>(a);
  return cudaGetLastError();
}

template <int kBound>
cudaError_t ByPlacement(const SmallKPlan& p, const DescentArgs<int16_t>& a, int grid, cudaStream_t st, bool cfg) {
  if (!p.half) return Go<kBound, kWindowCap, false, false>(p, a, grid, st, cfg);
  return p.smem_state ? Go<kBound, kWindowCap, true, true>(p, a, grid, st, cfg)
                      : Go<kBound, kWindowCap, false, true>(p, a, grid, st, cfg);
}

// Members of the wide form's windows: as many as their keys leave registers for, since a refresh passes over twice the
// narrow path's vertices and more.
constexpr int WideCap(int k) { return k <= 4 ? 4 * kWindowCap : k <= 8 ? 2 * kWindowCap : kWindowCap; }

template <int kBound>
cudaError_t Wide(const SmallKPlan& p, const DescentArgs<int32_t>& a, int grid, cudaStream_t st, bool cfg) {
  return Go<kBound, WideCap(kBound), false, false>(p, a, grid, st, cfg);
}

}  // namespace

bool PlanWindow(SmallKPlan& p, int n, int k, bool wide, size_t limit) {
  p.window = true;
  p.k = WindowBound(k);
  p.threads = kWindowThreads;
  p.registers = false;
  p.smem_rows = false;
  const int cap = wide ? WideCap(p.k) : kWindowCap;
  const size_t fixed = 8 * 1024 + (size_t)cap * 4;  // the kernels' static shared memory
  if (limit < fixed) return false;
  limit -= fixed;
  p.half = n <= kWindowHalfMax;
  p.smem_state = p.half && WindowSmem(n, k, true, cap) <= limit;
  p.smem_bytes = WindowSmem(n, k, p.smem_state, cap);
  return p.smem_bytes <= limit;
}

size_t WindowGlobalBytes(int n, int k) { return (size_t)k * WindowLd(n) * 2; }

cudaError_t LaunchDescentWindow(const SmallKPlan& p, const DescentArgs<int16_t>& a, int grid, cudaStream_t st,
                                bool cfg) {
  switch (p.k) {
    case 2: return ByPlacement<2>(p, a, grid, st, cfg);
    case 3: return ByPlacement<3>(p, a, grid, st, cfg);
    case 4: return ByPlacement<4>(p, a, grid, st, cfg);
    case 5: return ByPlacement<5>(p, a, grid, st, cfg);
    case 6: return ByPlacement<6>(p, a, grid, st, cfg);
    case 7: return ByPlacement<7>(p, a, grid, st, cfg);
    case 8: return ByPlacement<8>(p, a, grid, st, cfg);
    case 16: return ByPlacement<16>(p, a, grid, st, cfg);
    case 32: return ByPlacement<32>(p, a, grid, st, cfg);
    case 64: return ByPlacement<64>(p, a, grid, st, cfg);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t LaunchDescentWindowWide(const SmallKPlan& p, const DescentArgs<int32_t>& a, int grid, cudaStream_t st,
                                    bool cfg) {
  switch (p.k) {
    case 2: return Wide<2>(p, a, grid, st, cfg);
    case 3: return Wide<3>(p, a, grid, st, cfg);
    case 4: return Wide<4>(p, a, grid, st, cfg);
    case 5: return Wide<5>(p, a, grid, st, cfg);
    case 6: return Wide<6>(p, a, grid, st, cfg);
    case 7: return Wide<7>(p, a, grid, st, cfg);
    case 8: return Wide<8>(p, a, grid, st, cfg);
    case 16: return Wide<16>(p, a, grid, st, cfg);
    case 32: return Wide<32>(p, a, grid, st, cfg);
    case 64: return Wide<64>(p, a, grid, st, cfg);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace ccb
