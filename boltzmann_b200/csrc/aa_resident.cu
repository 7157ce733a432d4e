// Host side of the resident kernel (aa_resident.cuh): when it applies, its tiles and its launch.
#include "aa_resident.cuh"

#include <algorithm>

#include "aa_launch.cuh"
#include "device_once.h"

namespace lbm {
namespace {

// Steps of one launch at most: a launch of seconds would hold the device's other users up.
constexpr int64_t kResidentSteps = 4000;

struct ResidentPlan {
  ResidentArgs args{};
  size_t smem = 0;
  int threads = 0;
};

// Published slots of a cell: populations, and with a tracer its populations and value.
template <int K, int NT>
constexpr int resident_slots() {
  return D2Q9::Q + (NT == 1 ? D2Q5::Q + 1 : 0);
}

// The tiling for gy x gz CTAs; false when a tile does not fit an SM's shared memory.
template <int K, int NT, int KT>
bool layout(int ny, int nz, int gy, int gz, size_t limit, ResidentPlan& p) {
  const int h = (ny + gy - 1) / gy, w = (nz + gz - 1) / gz;
  if ((h + 4) * (w + 4) > resident_stride<K, NT, KT>()) return false;
  ResidentArgs& d = p.args;
  d.gy = gy;
  d.gz = gz;
  // Over the tiles of one row or column less, too (a thin one has no interior to leave out).
  d.published = std::max(std::max(rim_cells(h, w), rim_cells(h - 1, w)),
                         std::max(rim_cells(h, w - 1), rim_cells(h - 1, w - 1)));
  d.messages = resident_slots<K, NT>() * halo_entries(h, w);
  p.smem = ResidentStage<K, NT, KT>::off_table + (size_t)2 * d.messages * 8;
  // A thread per cell, or per message where those are more.
  const int most = resident_threads<K, NT>();
  p.threads = std::min(most, std::max((h + 2) * (w + 2), std::min(d.messages, 512)));
  p.threads = std::min(most, (p.threads + 31) / 32 * 32);
  return p.smem <= limit;
}

// The tiling with the least work for its busiest CTA, per step: its cells, half of the ring's, and the
// messages of its edges at about a tenth of a cell's instructions each.
template <int K, int NT, int KT>
bool plan_for(lbm_sim& s, int sms, size_t limit, ResidentPlan& best) {
  const int ny = (int)s.counts[0], nz = (int)s.counts[1];
  // Cheap bounds first: a cell of every slot and its flag must fit, and tile arithmetic is 32-bit.
  if (s.n > (int64_t)sms * resident_stride<K, NT, KT>() || s.n >= (1 << 22)) return false;
  if (s.resident_key == NT)  // the search's result for this number of tracers
    return s.resident_gy > 0 && layout<K, NT, KT>(ny, nz, s.resident_gy, s.resident_gz, limit, best);
  // Tiles of some 64 cells at least: smaller ones send more words than they update cells.
  const int ctas = (int)std::min<int64_t>(sms, std::max<int64_t>(1, s.n / 64));
  double least = 0;
  bool found = false;
  for (int gy = 1; gy <= std::min(ny, ctas); ++gy)
    for (int gz = 1; gz <= std::min(nz, ctas / gy); ++gz) {
      const int h = (ny + gy - 1) / gy, w = (nz + gz - 1) / gz;
      const double cost = (double)h * w + 2.5 * (h + w);
      if (found && cost >= least) continue;
      ResidentPlan p;
      if (!layout<K, NT, KT>(ny, nz, gy, gz, limit, p)) continue;
      best = p;
      least = cost;
      found = true;
    }
  s.resident_key = NT;
  s.resident_gy = found ? best.args.gy : 0;
  s.resident_gz = found ? best.args.gz : 0;
  return found;
}

template <bool TRT, int K, int NT, int KT>
cudaError_t run(lbm_sim& s, const ResidentPlan& plan, int64_t steps) {
  using Real = typename Pop<K>::real;
  auto kern = aa_resident_kernel<D2Q9, TRT, K, NT, KT>;
  static DeviceOnce once;
  const cudaError_t setup_err = once([&] {
    int limit = 0;
    cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, s.device);
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
  });
  if (setup_err != cudaSuccess) return setup_err;
  for (int64_t left = steps; left > 0;) {
    const int now = (int)std::min(left, kResidentSteps);
    left -= now;
    const StepArgs<Real> a = make_step_args<Real>(s, left == 0);
    ResidentArgs d = plan.args;
    d.steps = now;
    d.seq = s.mail_seq;
    d.polls = s.spin_limit < 0 ? kResidentPolls
                               : (unsigned)std::min<int64_t>(s.spin_limit, kResidentPolls);
    for (int k = 0; k < 2; ++k) d.mail[k] = static_cast<unsigned long long*>(s.mail[k]);
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(d.gy * d.gz));
    cfg.blockDim = dim3((unsigned)plan.threads);
    cfg.dynamicSmemBytes = plan.smem;
    cfg.stream = s.stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cudaError_t e = cudaLaunchKernelEx(&cfg, kern, a, d)) {
      cudaGetLastError();  // reported here, not by the next launch's check too
      const bool first = left + now == steps;  // nothing enqueued yet
      if (e != cudaErrorCooperativeLaunchTooLarge || !first) return e;
      // Fewer SMs than the device has (a partition): single steps.
      s.resident_gy = 0;
      return cudaErrorNotSupported;
    }
    s.mail_seq += (unsigned)(now / 2);
    s.launches[lbm_sim::kDirectSteps] += now;
    ++s.launches[lbm_sim::kKernels + LBM_KERNEL_RESIDENT];
  }
  return cudaSuccess;
}

template <int K, int NT, int KT>
bool plan_here(lbm_sim& s, ResidentPlan& plan) {
  int sms = 0, smem = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s.device);
  cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, s.device);
  return plan_for<K, NT, KT>(s, sms, (size_t)smem, plan);
}

template <int K, int NT, int KT>
size_t mail_bytes(lbm_sim& s) {
  ResidentPlan plan;
  if (!plan_here<K, NT, KT>(s, plan)) return 0;
  return (size_t)mail_words<typename Pop<K>::type>() * plan.args.gy * plan.args.gz *
         resident_slots<K, NT>() * plan.args.published * 8;
}

// Whether a simulation that is stepped beside others (threads, streams) should still take the resident
// kernel: resident launches whose CTAs do not fit the chip side by side take turns, while the single
// steps of several small domains overlap. us a step and simulation, single steps / resident, in calls
// of 200 steps by a thread each: 128^2 two at once 0.87 / 1.04, three 0.71 / 1.03, eight 0.33 / 1.02;
// 256^2 two 1.16 / 1.33, three 0.92 / 1.31, eight 0.64 / 1.30; 400 x 350 three 1.41 / 1.77; 512 x 500
// four 2.29 / 2.46, eight 2.32 / 2.46; 64^2, of which two fit, four 0.45 / 0.48, eight 0.27 / 0.47. The
// line lies at three turns, below 200,000 cells: a simulation that shares the chip for part of a call
// only is not sent to single steps by that. The results are the same either way.
bool worth_waiting(const lbm_sim& s, const ResidentArgs& d) {
  if (s.n >= 200000) return true;
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s.device);
  return (int64_t)simulations_in_flight(s.device) * d.gy * d.gz <= 2 * (int64_t)sms;
}

template <int K, int NT, int KT>
cudaError_t iterate(lbm_sim& s, int64_t steps) {
  ResidentPlan plan;
  if (s.mail[1] == nullptr || s.mail_tracers != NT || !plan_here<K, NT, KT>(s, plan))
    return cudaErrorNotSupported;
  if (!worth_waiting(s, plan.args)) return cudaErrorNotSupported;
  return s.collision == 1 ? run<true, K, NT, KT>(s, plan, steps)
                          : run<false, K, NT, KT>(s, plan, steps);
}

// fn with the variant of the simulation's storage for nt tracers.
template <class F>
auto with_variant(const lbm_sim& s, int nt, F fn) {
  switch (s.storage) {
    case kF16:
      return nt == 0 ? fn.template operator()<kF16, 0, kF32>()
                     : (s.tracer_storage == kF16 ? fn.template operator()<kF16, 1, kF16>()
                                                 : fn.template operator()<kF16, 1, kF32>());
    case kBF16:
      return nt == 0 ? fn.template operator()<kBF16, 0, kF32>()
                     : (s.tracer_storage == kBF16 ? fn.template operator()<kBF16, 1, kBF16>()
                                                  : fn.template operator()<kBF16, 1, kF32>());
    case kF64:
      return nt == 0 ? fn.template operator()<kF64, 0, kF64>()
                     : fn.template operator()<kF64, 1, kF64>();
    default:
      return nt == 0 ? fn.template operator()<kF32, 0, kF32>()
                     : fn.template operator()<kF32, 1, kF32>();
  }
}

// FP64, whose updates take longest, gains by the kernel on small domains only: 256^2 2.74 us a step, 3.40
// in single steps; 300 x 299 3.7 and 3.6, with a tracer 4.8 and 4.4, 512 x 500 6.7 and 6.4.
bool resident_size(const lbm_sim& s) { return s.storage != kF64 || s.n <= 80000; }

struct MailBytes {
  lbm_sim& s;
  template <int K, int NT, int KT>
  size_t operator()() const {
    return mail_bytes<K, NT, KT>(s);
  }
};
struct Iterate {
  lbm_sim& s;
  int64_t steps;
  template <int K, int NT, int KT>
  cudaError_t operator()() const {
    return iterate<K, NT, KT>(s, steps);
  }
};

}  // namespace

size_t resident_mail_bytes(lbm_sim& s, int tracers) {
  if (s.dim != 2 || s.q != D2Q9::Q || tracers > 1 || !resident_size(s)) return 0;
  return with_variant(s, tracers, MailBytes{s});
}

cudaError_t iterate_resident(lbm_sim& s, int64_t steps) {
  // A launch costs the way of the domain into and out of shared memory (6 us for 64^2, 16 us for
  // 1000 x 501), which some steps have to earn: measured even with single steps at 6 of them for 64^2, 8
  // for 256^2, 12 for 512 x 500, 14 for 700 x 451 in FP16.
  if (s.dim != 2 || s.q != D2Q9::Q || s.kernel_path != 0 || s.tracers.size() > 1 ||
      steps < 6 + s.n / 32768 || !resident_size(s))
    return cudaErrorNotSupported;
  return with_variant(s, (int)s.tracers.size(), Iterate{s, steps});
}

}  // namespace lbm
