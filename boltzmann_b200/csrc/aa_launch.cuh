// Host-side dispatch of the AA kernel family for one fluid lattice. Included by one .cu file per
// lattice so the instantiations compile in parallel.
#pragma once

#include <cudaTypedefs.h>

#include <atomic>
#include <type_traits>

#include "aa_tma.cuh"
#include "aa_step.cuh"
#include "device_once.h"
#include "sim.h"

namespace lbm {

template <class Real>
StepArgs<Real> make_step_args(const lbm_sim& s, bool write_moments) {
  StepArgs<Real> a{};
  a.f = s.f;
  a.rho = static_cast<Real*>(s.rho);
  a.vel = static_cast<Real*>(s.vel);
  a.flags = s.flags;
  if (s.dim == 3) {
    a.nx = (int)s.counts[0];
    a.ny = (int)s.counts[1];
    a.nz = (int)s.counts[2];
  } else {
    a.nx = 1;
    a.ny = (int)s.counts[0];
    a.nz = (int)s.counts[1];
  }
  a.n = s.n;
  a.om_pos = s.om_pos;
  a.om_neg = s.om_neg;
  const int off = 3 - s.dim;
  // Acceleration source, as src/simulation.rs:326-373 leaves it for the fluid kernel: any
  // Boussinesq coupling overwrites the constant acceleration every step, the last one winning.
  if (!s.couplings.empty()) {
    const lbm_sim::Coupling& c = s.couplings.back();
    a.acc_mode = kAccBoussinesq;
    // (g b) / om_pos in the reference (src/lib.cl:72 then 254); b (g / om_pos) here: the same
    // shift up to one rounding of a term of the size of the buoyancy.
    for (int k = 0; k < s.dim; ++k) a.force[off + k] = (Real)c.g[k] / (Real)s.om_pos;
    a.alpha = c.alpha;
    a.c0 = c.c0;
    a.coupled = c.tracer;
    a.coupled_val = static_cast<const Real*>(s.tracers[c.tracer].val);
  } else if (s.has_gravity) {
    a.acc_mode = kAccConstant;
    // acc / om_pos, the division the reference makes per cell (src/lib.cl:254), made once.
    for (int k = 0; k < s.dim; ++k) a.force[off + k] = (Real)s.gravity[k] / (Real)s.om_pos;
  }
  a.ntracers = (int)s.tracers.size();
  for (int t = 0; t < a.ntracers; ++t) {
    a.tr[t].g = s.tracers[t].g;
    a.tr[t].val = static_cast<Real*>(s.tracers[t].val);
    a.tr[t].omega = s.tracers[t].omega;
    a.tr[t].omega_neg = s.tracers[t].omega_neg;
    a.tr[t].trt = s.tracers[t].collision == 1;
  }
  a.write_moments = write_moments ? 1 : 0;
  a.path = s.kernel_path;
  a.omega_field = s.omega_field;
  a.status = s.status;
  a.spin_limit = s.spin_limit < 0 ? kSpinLimit
                                  : (unsigned)(s.spin_limit < (int64_t)kSpinLimit ? s.spin_limit
                                                                                 : kSpinLimit);
  return a;
}

// Ring depth of the TMA kernel: as many stages as fit in ~50 KB per CTA (2-4), so that three or
// four CTAs (24-32 consumer warps) share an SM and each keeps one or more tiles of copies in
// flight while it computes another.
template <class L, int K, int NT, bool EVEN, bool WR, int KT = default_tracer_kind<K>()>
constexpr int tma_stages() {
  constexpr size_t b = TmaStage<L, K, NT, EVEN, WR, KT>::bytes;
  constexpr int s = (int)((50 * 1024) / b);
  return s < 2 ? 2 : (s > 4 ? 4 : s);
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link against libcuda).
inline PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return (PFN_cuTensorMapEncodeTiled_v12000) nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }();
  return fn;
}

template <class T>
constexpr CUtensorMapDataType tensor_map_type() {
  if constexpr (sizeof(T) == 8) return CU_TENSOR_MAP_DATA_TYPE_FLOAT64;
  else if constexpr (sizeof(T) == 4) return CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  else if constexpr (std::is_same_v<T, __half>) return CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  else return CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
}

// A [q slots][n cells] array (slot stride n elements) as a 2D tensor with a box of
// kTmaTile cells by all q slots. False when it cannot be described (the caller then copies row
// segments).
template <class T>
bool encode_slot_map(CUtensorMap* map, const void* base, long long n, int q) {
  auto encode = tensor_map_encoder();
  if (encode == nullptr || n >= (1ll << 31) || q > 256) return false;
  cuuint64_t dims[2] = {(cuuint64_t)n, (cuuint64_t)q};
  cuuint64_t strides[1] = {(cuuint64_t)n * sizeof(T)};
  if (strides[0] % 16 != 0 || (reinterpret_cast<uintptr_t>(base) & 15) != 0) return false;
  cuuint32_t box[2] = {(cuuint32_t)kTmaTile, (cuuint32_t)q};
  cuuint32_t elem[2] = {1, 1};
  return encode(map, tensor_map_type<T>(), 2, const_cast<void*>(base), dims, strides, box, elem,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The population array as a 2D tensor of rows of nz cells, row (slot, x, y), with a box of one
// row of kTmaTile cells (the four-row copies of even steps of one-tile rows).
template <class T>
bool encode_row_map(CUtensorMap* map, const void* base, long long rows, int nz) {
  auto encode = tensor_map_encoder();
  if (encode == nullptr || rows >= (1ll << 31) || nz != kTmaTile) return false;
  cuuint64_t dims[2] = {(cuuint64_t)nz, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)nz * sizeof(T)};
  if (strides[0] % 16 != 0 || (reinterpret_cast<uintptr_t>(base) & 15) != 0) return false;
  cuuint32_t box[2] = {(cuuint32_t)kTmaTile, 1};
  cuuint32_t elem[2] = {1, 1};
  return encode(map, tensor_map_type<T>(), 2, const_cast<void*>(base), dims, strides, box, elem,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <class L, bool TRT, int K, bool EVEN, int NT, bool WR, int KT>
cudaError_t launch_tma(const StepArgs<typename Pop<K>::real>& a, cudaStream_t stream) {
  constexpr int S = tma_stages<L, K, NT, EVEN, WR, KT>();
  constexpr size_t smem = tma_smem_bytes<L, K, NT, EVEN, S, WR, KT>();
  // Two cells a consumer thread with 16-bit populations: D3Q27 BGK without a tracer, on the
  // steps whose results go back through the stage (D3Q27 TRT needs more than the 128 registers
  // three CTAs a SM leave a thread, and spills); D2Q9 BGK / TRT with none or one fused tracer, on
  // every step.
  constexpr bool PAIR = pair_form<L, TRT, K, NT>() && (L::D == 2 || !EVEN || WR);
  constexpr int threads = tma_threads<PAIR>();
  auto kern = aa_tma_kernel<L, TRT, K, EVEN, NT, S, WR, PAIR, KT>;
  static DeviceOnce once;
  static std::atomic<int> occupancy{1};
  const cudaError_t setup_err = once([&] {
    int fit = 1;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kern, threads, smem);
    occupancy = fit < 1 ? 1 : fit;
    return e;
  });
  if (setup_err != cudaSuccess) return setup_err;
  const int per_sm = occupancy;
  int device = 0, sms = 148;
  cudaGetDevice(&device);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  const long long tiles = (long long)a.nx * a.ny * (a.nz / kTmaTile);
  long long grid = (long long)sms * per_sm;
  if (grid > tiles) grid = tiles;
  TmaMaps maps{};
  if constexpr (EVEN && WR) {
    using T = typename Pop<K>::type;
    maps.use = encode_row_map<T>(&maps.f, a.f, (long long)L::Q * a.nx * a.ny, a.nz) ? 1 : 0;
  } else if constexpr (!EVEN) {
    using T = typename Pop<K>::type;
    using Real = typename Pop<K>::real;
    bool ok = encode_slot_map<T>(&maps.f, a.f, a.n, L::Q);
    if constexpr (NT == 1)
      ok = ok && encode_slot_map<typename TracerPop<KT>::type>(&maps.g, a.tr[0].g, a.n,
                                                              TracerLattice<L::D>::type::Q);
    maps.use = ok ? 1 : 0;
  }
  // Not a dependent launch: its steps are long and its CTAs fill the SMs until they end (4096 x 2048
  // with a tracer, 100 steps: 19.69 ms, 19.82 as one).
  kern<<<(unsigned)grid, threads, smem, stream>>>(a, maps);
  return cudaGetLastError();
}

// Whether the TMA-staged kernel is the faster one for rows of whole 256-cell tiles (fused tracers: none
// or one). It keeps more loads in flight per SM with fewer instructions, the direct kernels more warps
// at work: domains that sit in L2, and FP32 or FP64 cells with more arithmetic per byte, are better off
// direct. Rows of one tile, whose even steps return by rows too, suit it best. us a step, direct /
// staged, each the median of some tenths of a second under its own load:
//   D2Q9  FP32         2048x1024 20.2 / 26.3, 1500x2560 47.8 / 52.4, 4096x2048 103 / 112, in a channel
//                      with TRT 109 / 114
//         with tracer  2048x1024 42.2 / 43.3; 4096x2048 159 / 175 in a periodic box, in a channel with
//                      TRT 170.3 / 170.3
//         FP64         2048x512 21.4 / 27.2, 1500x2560 94 / 101, 4096x2048 207 / 211
//         FP16         2048x1024 16.8 / 21.6, 4096x2048 73.4 / 77.4 (TRT 78.3 / 78.0)
//         FP32 tracer  2048x512 12.8 / 15.4, 2048x1024 28.3 / 28.1, 1500x1536 33.6 / 31.2, 8000x768
//                      94.6 / 90.2
//         FP16 tracer  1000x2560 31.5 / 33.1, 1500x2560 52.9 / 50.9, 4096x2048 113 / 111; TRT
//                      1500x1536 29.4 / 30.2, 1000x2560 34.2 / 33.5, 4096x2048 121 / 111
//   D3Q27 FP32 BGK     48x64x256 23.5 / 24.0, 64x64x256 with a relaxation field 43.4 / 41.1, 256^3
//                      617 / 583; 128x100x512 231 / 241
//         FP32 TRT     100x100x256 92.9 / 107, 256^3 612 / 668; with a tracer 120 / 132
//         FP64         100x100x256 182.3 / 182.4, 256^3 1173 / 1170, 24x48x1024 85.0 / 93.7; with a
//                      tracer 224 / 226, 105 / 114
//         FP16 BGK     24x48x256 7.7 / 8.6, 48x64x256 17.4 / 15.9; 48x64x512 35.9 / 38.2, 40x90x512
//                      44.3 / 43.7, 128x100x512 159 / 157
//         FP16 TRT     24x48x256 7.9 / 9.4, 48x64x256 18.4 / 18.1, 256^3 464 / 362; 48x64x512 37.7 /
//                      41.0, 40x90x512 47.6 / 47.3, 128x100x512 175 / 160
//         FP32 tracer  48x64x256 21.2 / 22.3, 64x64x256 30.8 / 30.6, 100x100x256 87.0 / 79.3; 128x100x512
//                      219 / 223; TRT 64x64x256 32.0 / 37.1, 64x90x256 52.6 / 52.2, 128x100x512 226 / 234
//         FP16 tracer  48x64x256 21.9 / 21.8, 64x90x256 48.6 / 42.1; 24x48x1024 34.3 / 38.3, 48x64x512
//                      51.5 / 51.3, 128x100x512 214 / 201; TRT 64x90x256 45.7 / 48.3, 100x100x256 80.7 /
//                      79.2, 128x100x512 201 / 215
// KT: storage kind of the tracer's populations.
template <class L, bool TRT, int K, int NT, int KT>
bool staged_pays(const StepArgs<typename Pop<K>::real>& a) {
  const long long cells = (long long)a.nx * a.ny * a.nz;
  const bool one_tile = a.nz == kTmaTile;
  constexpr bool wide_tracer = KT == kF32;
  if (K == kF64) return false;
  if (L::D == 2) {
    if (K == kF32) return NT != 0 && cells >= 6000000;
    return NT != 0 && cells >= (wide_tracer ? 2000000 : (TRT ? 2500000 : 3000000));
  }
  if (K == kF32) return !TRT && NT == 0 && one_tile && cells >= 700000;
  if (NT == 0) return cells >= (one_tile ? 700000 : 1700000);
  if (wide_tracer) return one_tile && cells >= (TRT ? 1400000 : 1000000);
  return one_tile ? cells >= (TRT ? 2000000 : 750000) : !TRT && cells >= 1400000;
}

// Whether a step of the one-cell direct kernel is launched as a dependent one: with cells of much work
// (FP64, or a run-time number of tracers) not where its grid fills half to three quarters of the chip's
// CTA slots. The next grid's CTAs then find room on some SMs only while this one runs, and the SMs that
// took more of them end last. us a step, dependent / plain: 36^3 FP64 with two tracers 8.6 / 7.1, 1 x 70000
// 5.6 / 4.9, 300 x 200 5.4 / 5.0; 350 x 300 with two tracers 4.5 / 4.0, 62 x 17 x 48 5.0 / 4.6. With less
// work a cell it pays there, too: 400 x 350 2.5 / 2.7, FP16 2.3 / 2.6, 40^3 FP16 3.2 / 3.5.
template <int K, int NT>
bool dependent_pays(long long ctas, long long room) {
  return (K != kF64 && NT >= 0) || 2 * ctas <= room || 4 * ctas >= 3 * room;
}

template <class L, bool TRT, int K, bool EVEN, int NT, int KT = default_tracer_kind<K>()>
cudaError_t launch_one(const StepArgs<typename Pop<K>::real>& a, cudaStream_t stream,
                       int64_t* launches) {
  if constexpr (NT >= 0) {
    const bool fits = a.nz % kTmaTile == 0;
    const bool staged = a.path == 2 || (a.path == 0 && staged_pays<L, TRT, K, NT, KT>(a));
    if (fits && staged) {
      cudaError_t e;
      if (EVEN && a.nz == kTmaTile)
        e = launch_tma<L, TRT, K, EVEN, NT, EVEN, KT>(a, stream);
      else
        e = launch_tma<L, TRT, K, EVEN, NT, false, KT>(a, stream);
      if (e == cudaSuccess) {
        ++launches[lbm_sim::kStagedSteps];
        ++launches[lbm_sim::kKernels + LBM_KERNEL_STAGED];
      }
      return e;
    }
  }
  const DirectArgs d = make_direct_args<L>(a, sizeof(typename Pop<K>::type),
                                           sizeof(typename TracerPop<KT>::type));
  if constexpr (pair_form<L, TRT, K, NT>()) {
    if ((long long)d.cells >= pair_direct_cells<L>()) {
      const unsigned grid = (unsigned)(((long long)d.cells + 2 * kDirectThreads - 1) / (2 * kDirectThreads));
      const cudaError_t e = launch_step_kernel(aa_step2_kernel<L, TRT, K, EVEN, NT, KT>, grid,
                                               kDirectThreads, 0, stream, true, a, d);
      if (e == cudaSuccess) {
        ++launches[lbm_sim::kDirectSteps];
        ++launches[lbm_sim::kKernels + LBM_KERNEL_STEP2];
      }
      return e;
    }
  }
  constexpr int threads = DirectForm<L, K, NT>::threads;
  const unsigned grid = (unsigned)(((long long)d.cells + threads - 1) / threads);
  auto kern = aa_step_kernel<L, TRT, K, EVEN, NT, KT>;
  static DeviceOnce once;
  static std::atomic<long long> room{0};
  const cudaError_t setup_err = once([&] {
    int device = 0, sms = 148, fit = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kern, threads, 0);
    room = (long long)sms * fit;
    return e;
  });
  if (setup_err != cudaSuccess) return setup_err;
  const cudaError_t e = launch_step_kernel(kern, grid, threads, 0, stream,
                                           dependent_pays<K, NT>(grid, room), a, d);
  if (e == cudaSuccess) {
    ++launches[lbm_sim::kDirectSteps];
    ++launches[lbm_sim::kKernels + LBM_KERNEL_STEP];
  }
  return e;
}

template <class L, bool TRT, int K>
cudaError_t launch_typed(const lbm_sim& s, bool even, bool write_moments) {
  using Real = typename Pop<K>::real;
  const StepArgs<Real> a = make_step_args<Real>(s, write_moments);
  // Fused tracers: none, exactly one (loads hoisted with the fluid's), or a runtime count.
  // 16-bit tracer populations (the fluid's own 16-bit kind) take the one-tracer path only.
  const int nt = a.ntracers;
  const bool t16 = s.tracer_storage == K && dev_in<K>();
  if (t16 && nt > 1) return cudaErrorNotSupported;
  if (even) {
    if (nt == 0) return launch_one<L, TRT, K, true, 0>(a, s.stream, s.launches);
    if (nt == 1) {
      if constexpr (dev_in<K>())
        if (t16) return launch_one<L, TRT, K, true, 1, K>(a, s.stream, s.launches);
      return launch_one<L, TRT, K, true, 1>(a, s.stream, s.launches);
    }
    return launch_one<L, TRT, K, true, -1>(a, s.stream, s.launches);
  }
  if (nt == 0) return launch_one<L, TRT, K, false, 0>(a, s.stream, s.launches);
  if (nt == 1) {
    if constexpr (dev_in<K>())
      if (t16) return launch_one<L, TRT, K, false, 1, K>(a, s.stream, s.launches);
    return launch_one<L, TRT, K, false, 1>(a, s.stream, s.launches);
  }
  return launch_one<L, TRT, K, false, -1>(a, s.stream, s.launches);
}

template <class L>
cudaError_t launch_lattice(const lbm_sim& s, bool even, bool write_moments) {
  const bool trt = s.collision == 1;
  switch (s.storage) {
    case kF32:
      return trt ? launch_typed<L, true, kF32>(s, even, write_moments)
                 : launch_typed<L, false, kF32>(s, even, write_moments);
    case kF16:
      return trt ? launch_typed<L, true, kF16>(s, even, write_moments)
                 : launch_typed<L, false, kF16>(s, even, write_moments);
    case kBF16:
      return trt ? launch_typed<L, true, kBF16>(s, even, write_moments)
                 : launch_typed<L, false, kBF16>(s, even, write_moments);
    case kF64:
      return trt ? launch_typed<L, true, kF64>(s, even, write_moments)
                 : launch_typed<L, false, kF64>(s, even, write_moments);
  }
  return cudaErrorInvalidValue;
}

}  // namespace lbm
