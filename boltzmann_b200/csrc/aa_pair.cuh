// Two cells a thread for the TMA-staged kernel with 16-bit populations: consumer thread t
// updates cells t and t + 128 of its 256-cell tile, with every FP32 operation of the cell update
// on Blackwell's packed instructions (lane x: cell t, lane y: cell t + 128). Each lane performs
// exactly the operations of update_cell / moments_packed / collide_packed / tracer_update in the
// same order (the packed instructions round each lane as the scalar one), so the results are
// the bits of the one-cell path; the operation count per cell drops because every operation is
// packed, not only the ones that pair opposite directions.
// Used for D3Q27 BGK without a tracer (results through the stage; +1.4% on the 256^3
// Taylor-Green run, whose kernel is close to its memory time) and for D2Q9 BGK / TRT with none or
// one fused tracer (both parities: results through the stage, or straight to HBM on even steps
// of rows longer than one tile), whose one-cell kernels are issue-bound.
#pragma once

#include "aa_step.cuh"

namespace lbm {

__device__ __forceinline__ float2 over_den2_hi_lo(float2 x, float hi, float lo) {
  return fma2(x, splat(hi), mul2(x, splat(lo)));
}

// c_i . u for both cells, the additions of c_dot in its order.
template <class L>
__device__ __forceinline__ float2 c_dot2(int i, const float2 (&u)[3]) {
  float2 cu = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (comp<L>(i, a) > 0) cu = add2(cu, u[a]);
    if (comp<L>(i, a) < 0) cu = sub2(cu, u[a]);
  }
  return cu;
}

// moments_packed<L, true> for two cells: v holds deviations.
template <class L>
__device__ __forceinline__ void moments2(const float2 (&v)[L::Q], float2& dr, float2 (&m)[3]) {
  constexpr int P = (L::Q - 1) / 2;
  float2 del[P];
  float2 acc_even = make_float2(0.0f, 0.0f), acc_odd = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int p = 0; p + 1 < P; p += 2) {
    const int i = 2 * p + 1, j = 2 * p + 3;
    del[p] = sub2(v[i], v[i + 1]);
    del[p + 1] = sub2(v[j], v[j + 1]);
    acc_even = add2(acc_even, add2(v[i], v[i + 1]));
    acc_odd = add2(acc_odd, add2(v[j], v[j + 1]));
  }
  float2 sig_last = make_float2(0.0f, 0.0f);
  if constexpr (P % 2 == 1) {
    constexpr int i = 2 * (P - 1) + 1;
    del[P - 1] = sub2(v[i], v[i + 1]);
    sig_last = add2(v[i], v[i + 1]);
  }
  dr = add2(add2(add2(v[0], add2(acc_even, acc_odd)), sig_last), splat(weight_defect<L, float>()));
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) m[ax] = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int p = 0; p < P; ++p) {
#pragma unroll
    for (int ax = 3 - L::D; ax < 3; ++ax) {
      if (comp<L>(2 * p + 1, ax) > 0) m[ax] = add2(m[ax], del[p]);
      if (comp<L>(2 * p + 1, ax) < 0) m[ax] = sub2(m[ax], del[p]);
    }
  }
}

// One opposite pair (i, i + 1) of collide_packed<L, TRT, DEV> for two cells.
template <class L, bool TRT, bool DEV>
__device__ __forceinline__ void collide_pair2(float2 (&v)[L::Q], int i, float2 ru, float2 unit,
                                              float2 quad, const float2 (&u)[3], float2 om_pos,
                                              float2 om_neg) {
  const float k = float(L::wk(i));
  const float2 cu = c_dot2<L>(i, u);
  const float2 kr = mul2(splat(k), ru);
  const float2 ku = fma2(splat(k), unit, splat(DEV ? weight_gap<L, float>(i) : 0.0f));
  const float2 X = fma2(mul2(splat(4.5f), cu), cu, quad);
  const float2 A = fma2(kr, X, ku);
  const float2 B = mul2(mul2(kr, splat(3.0f)), cu);
  float2 F = v[i], G = v[i + 1];
  if constexpr (TRT) {
    const float2 S = mul2(splat(0.5f), add2(F, G));
    const float2 D = mul2(splat(0.5f), sub2(F, G));
    const float2 fp = mul2(om_pos, sub2(A, S));
    const float2 fn = mul2(om_neg, sub2(B, D));
    F = add2(F, add2(fp, fn));
    G = add2(G, sub2(fp, fn));
  } else {
    F = fma2(om_pos, sub2(add2(A, B), F), F);
    G = fma2(om_pos, sub2(sub2(A, B), G), G);
  }
  v[i] = F;
  v[i + 1] = G;
}

// collide_packed<L, TRT, DEV> for two cells (r: densities, dr: r - 1; the tracers pass their
// concentration as both).
template <class L, bool TRT, bool DEV>
__device__ __forceinline__ void collide2(float2 (&v)[L::Q], float2 r, float2 dr,
                                         const float2 (&u)[3], float2 uu, float2 om_pos,
                                         float2 om_neg) {
  const float2 ru = over_den2_hi_lo(r, inv_den_hi<L, float>(), inv_den_lo<L, float>());
  const float2 unit =
      DEV ? over_den2_hi_lo(dr, inv_den_hi<L, float>(), inv_den_lo<L, float>()) : ru;
  const float2 quad = mul2(splat(-1.5f), uu);
  {
    const float k0 = float(L::wk(0));
    const float2 e0 = fma2(mul2(splat(k0), ru), quad,
                           fma2(splat(k0), unit, splat(DEV ? weight_gap<L, float>(0) : 0.0f)));
    v[0] = fma2(om_pos, sub2(e0, v[0]), v[0]);
  }
#pragma unroll
  for (int i = 1; i < L::Q; i += 2) collide_pair2<L, TRT, DEV>(v, i, ru, unit, quad, u, om_pos, om_neg);
}

// Where update_cell2 puts its results: into the stage the operands came from, at StageSink's
// positions (slot i of the cell on odd steps, the very position read on even steps); walls
// (skip) leave theirs untouched.
template <class St, int TILE>
struct PairSink {
  unsigned char* st;
  int tid;  // cell A's column; cell B is tid + TILE / 2

  template <class L, class P, bool EVEN>
  __device__ __forceinline__ void fluid(bool skipA, bool skipB, const float2 (&v)[L::Q]) const {
    using T = typename P::type;
    T* base = reinterpret_cast<T*>(st);
#pragma unroll
    for (int i = 0; i < L::Q; ++i) {
      const int cz = comp<L>(i, 2);
      const int pa = stage_pos<St::kWR, EVEN>(St::H, tid, cz);
      const int pb = stage_pos<St::kWR, EVEN>(St::H, tid + TILE / 2, cz);
      const float2 val = EVEN ? v[opp(i)] : v[i];
      if (!skipA) P::store_dev(base + i * St::SEG + pa, val.x, 0.0f);
      if (!skipB) P::store_dev(base + i * St::SEG + pb, val.y, 0.0f);
    }
    if constexpr (EVEN && St::QP > L::Q) {
      // The padding rows of the last four-row group repeat slot Q - 1.
      constexpr int i = L::Q - 1;
      const int pa = stage_pos<St::kWR, EVEN>(St::H, tid, comp<L>(i, 2));
      const int pb = stage_pos<St::kWR, EVEN>(St::H, tid + TILE / 2, comp<L>(i, 2));
      const T wa = base[i * St::SEG + pa], wb = base[i * St::SEG + pb];
#pragma unroll
      for (int rr = L::Q; rr < St::QP; ++rr) {
        base[rr * St::SEG + pa] = wa;
        base[rr * St::SEG + pb] = wb;
      }
    }
  }

  template <class TL, class TP, bool EVEN>
  __device__ __forceinline__ void tracer(bool skipA, bool skipB, const float2 (&v)[TL::Q]) const {
    using TT = typename TP::type;
#pragma unroll
    for (int i = 0; i < TL::Q; ++i) {
      const float2 val = EVEN ? v[opp(i)] : v[i];
      TT* base = reinterpret_cast<TT*>(st + St::off_trc) + i * St::SEGG;
      const int cz = comp<TL>(i, 2);
      if (!skipA) TP::store(base + stage_pos<St::kWR, EVEN>(St::HG, tid, cz), val.x, 0.0f);
      if (!skipB) TP::store(base + stage_pos<St::kWR, EVEN>(St::HG, tid + TILE / 2, cz), val.y, 0.0f);
    }
  }
};

// tracer_update<TL, TP, EVEN, true> for two cells: the concentration, the fixed-value override,
// the packed collision and the AA store. Wall cells (skip) are computed but not stored.
template <class TL, class TP, bool EVEN, class Sink>
__device__ __forceinline__ void tracer_update2(const TracerArgs<float>& tr, long long n,
                                               const CellPos& cA, const CellPos& cB, int flagA,
                                               int flagB, bool wallA, bool wallB,
                                               float2 (&g)[TL::Q], const float2 (&u)[3],
                                               float2 uu, bool keep, const Sink& sink) {
  float2 rt = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int i = 0; i < TL::Q; ++i) rt = add2(rt, g[i]);
  float2 om = splat(tr.omega), om_n = splat(tr.omega_neg);
  const bool tfA = (flagA & 8) != 0, tfB = (flagB & 8) != 0;  // FIXED_SCALAR_VALUE
  if (tfA) {
    om.x = 1.0f;
    om_n.x = 1.0f;
    rt.x = tr.val[cA.cell];
  }
  if (tfB) {
    om.y = 1.0f;
    om_n.y = 1.0f;
    rt.y = tr.val[cB.cell];
  }
  if (tr.trt)
    collide2<TL, true, false>(g, rt, rt, u, uu, om, om_n);
  else
    collide2<TL, false, false>(g, rt, rt, u, uu, om, om);
  sink.template tracer<TL, TP, EVEN>(wallA, wallB, g);
  if (keep) {
    if (!wallA && !tfA) tr.val[cA.cell] = rt.x;
    if (!wallB && !tfB) tr.val[cB.cell] = rt.y;
  }
}

// update_cell<L, TRT, K, EVEN, NT, ..., KT> for two cells whose deviations were loaded into f
// (and, NT == 1, the first tracer's populations into g); cA / cB: the cells' positions (with
// their neighbourhoods when the sink stores to HBM on even steps); flagA / flagB their flags;
// cval: the coupled values.
template <class L, bool TRT, int K, bool EVEN, int NT, int KT, class Sink>
__device__ __forceinline__ void update_cell2(const StepArgs<float>& a, const Sink& sink,
                                             const CellPos& cA, const CellPos& cB, int flagA,
                                             int flagB, float2 (&f)[L::Q],
                                             float2 (&g)[NT == 1 ? TracerLattice<L::D>::type::Q : 1],
                                             float2 cval) {
  using P = Pop<K>;
  using TL = typename TracerLattice<L::D>::type;
  using TP = TracerPop<KT>;
  constexpr int D = L::D;
  static_assert(dev_in<K>(), "two cells a thread: 16-bit storage");
  const bool wallA = (flagA & 1) != 0, wallB = (flagB & 1) != 0;
  if (wallA && wallB) return;
  const unsigned cellA = cA.cell, cellB = cB.cell;

  float2 dr, m[3];
  moments2<L>(f, dr, m);
  float2 r = add2(splat(1.0f), dr);
  const float2 rinv = make_float2(__frcp_rn(r.x), __frcp_rn(r.y));
  float2 u[3];
  u[0] = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int ax = 3 - D; ax < 3; ++ax) u[ax] = mul2(m[ax], rinv);

  float2 om_pos = splat(a.om_pos), om_neg = splat(a.om_neg);
  if (a.omega_field != nullptr)
    om_pos = make_float2(__ldg(a.omega_field + cellA), __ldg(a.omega_field + cellB));
  if (a.acc_mode == kAccConstant) {
#pragma unroll
    for (int ax = 3 - D; ax < 3; ++ax) u[ax] = add2(u[ax], splat(a.force[ax]));
  } else if (a.acc_mode == kAccBoussinesq) {
    const float2 b = mul2(splat(a.alpha), sub2(cval, splat(a.c0)));
#pragma unroll
    for (int ax = 3 - D; ax < 3; ++ax) u[ax] = fma2(b, splat(a.force[ax]), u[ax]);
  }
  const bool fixedA = (flagA & 6) != 0, fixedB = (flagB & 6) != 0;
  if (fixedA) {
    om_pos.x = 1.0f;
    om_neg.x = 1.0f;
    r.x = a.rho[cellA];
    dr.x = r.x - 1.0f;
#pragma unroll
    for (int ax = 3 - D; ax < 3; ++ax) u[ax].x = a.vel[(size_t)cellA * D + ax - (3 - D)];
  }
  if (fixedB) {
    om_pos.y = 1.0f;
    om_neg.y = 1.0f;
    r.y = a.rho[cellB];
    dr.y = r.y - 1.0f;
#pragma unroll
    for (int ax = 3 - D; ax < 3; ++ax) u[ax].y = a.vel[(size_t)cellB * D + ax - (3 - D)];
  }
  float2 uu = mul2(u[3 - D], u[3 - D]);
#pragma unroll
  for (int ax = 4 - D; ax < 3; ++ax) uu = fma2(u[ax], u[ax], uu);

  collide2<L, TRT, true>(f, r, dr, u, uu, om_pos, om_neg);
  sink.template fluid<L, P, EVEN>(wallA, wallB, f);

  if (a.write_moments) {
    if (!wallA && !fixedA) {
      a.rho[cellA] = r.x;
#pragma unroll
      for (int ax = 3 - D; ax < 3; ++ax) a.vel[(size_t)cellA * D + ax - (3 - D)] = u[ax].x;
      if (!isfinite(r.x) || !isfinite(uu.x)) atomicOr(a.status, 1);
    }
    if (!wallB && !fixedB) {
      a.rho[cellB] = r.y;
#pragma unroll
      for (int ax = 3 - D; ax < 3; ++ax) a.vel[(size_t)cellB * D + ax - (3 - D)] = u[ax].y;
      if (!isfinite(r.y) || !isfinite(uu.y)) atomicOr(a.status, 1);
    }
  }

  if constexpr (NT == 1) {
    const bool keep = a.write_moments || (a.acc_mode == kAccBoussinesq && a.coupled == 0);
    tracer_update2<TL, TP, EVEN>(a.tr[0], a.n, cA, cB, flagA, flagB, wallA, wallB, g, u, uu, keep,
                                 sink);
  }
}

// update_cell2's results straight to HBM, like GlobalSink.
template <bool RENEW>
struct GlobalPairSink {
  const SlotTable& table;
  const CellPos &cA, &cB;

  template <class L, class P, bool EVEN>
  __device__ __forceinline__ void fluid(bool skipA, bool skipB, const float2 (&v)[L::Q]) const {
    using T = typename P::type;
    put<L, P, EVEN, true, T>(table.f, skipA, skipB, v);
  }
  template <class TL, class TP, bool EVEN>
  __device__ __forceinline__ void tracer(bool skipA, bool skipB, const float2 (&v)[TL::Q]) const {
    using T = typename TP::type;
    put<TL, TP, EVEN, false, T>(table.g, skipA, skipB, v);
  }

 private:
  template <class L, class P, bool EVEN, bool DEV, class T>
  __device__ __forceinline__ void put(void* const* slots, bool skipA, bool skipB,
                                      const float2 (&v)[L::Q]) const {
    const CellPos eA = RENEW ? renewed<EVEN>(cA) : cA, eB = RENEW ? renewed<EVEN>(cB) : cB;
#pragma unroll
    for (int i = 0; i < L::Q; ++i) {
      T* slot = static_cast<T*>(slots[i]);
      T* pa = slot + (EVEN ? eA.upstream<L>(i) : eA.cell);
      T* pb = slot + (EVEN ? eB.upstream<L>(i) : eB.cell);
      const float2 val = EVEN ? v[opp(i)] : v[i];
      if constexpr (DEV) {
        if (!skipA) P::store_dev(pa, val.x, 0.0f);
        if (!skipB) P::store_dev(pb, val.y, 0.0f);
      } else {
        if (!skipA) P::store(pa, val.x, 0.0f);
        if (!skipB) P::store(pb, val.y, 0.0f);
      }
    }
  }
};

// Whether a simulation's 16-bit kernels update two cells a thread: D3Q27 BGK without a tracer, and
// D2Q9 with none or one. (D3Q27 TRT needs more registers than that leaves a thread, and spills.)
template <class L, bool TRT, int K, int NT>
constexpr bool pair_form() {
  return dev_in<K>() && ((L::Q >= 27 && !TRT && NT == 0) || (L::D == 2 && (NT == 0 || NT == 1)));
}
// Smallest domain (cells) for the direct two-cell kernel: below it its CTAs, half as many, leave SMs short
// of warps. us a step, one cell a thread / two: 450 x 400 2.66 / 2.92, 500 x 451 3.12 / 2.93 (TRT 3.30 /
// 2.92), 2000 x 1001 18.2 / 16.2; with a tracer 3.2 / 3.6, 4.0 / 3.8, 23.8 / 23.2 (between, at 600 x 501
// and 1000 x 501, 4.6 / 4.8 and 6.8 / 7.0); 60 x 60 x 50 5.5 / 5.9, 90 x 90 x 80 15.1 / 15.0, 180 x 150 x
// 100 72.7 / 67.6.
template <class L>
constexpr long long pair_direct_cells() {
  return L::D == 2 ? 200000 : 700000;
}

// The direct kernel with two cells a thread, for 16-bit populations: cells t and t + 128 of the
// CTA's 256 consecutive cells. A 16-bit cell keeps half the bytes of an FP32 one in flight and
// spends as many instructions; two cells on packed instructions mend both. 200^3 BGK 221 -> 194
// us a step, 3000 x 1001 TRT with a 16-bit tracer 41.9 -> 38.6, 2000 x 1000 18.4 -> 16.1. Four CTAs
// an SM for D3Q27 (three 220, five 214), six for D2Q9 (five 42.4, eight 45.0). The next step is let in at
// the start: behind the loads, as in the one-cell kernel, it held the update up (BGK, 128 x 100 x 512
// 159 -> 173, 4096 x 2048 with a 32-bit tracer 127 -> 135).
template <class L, bool TRT, int K, bool EVEN, int NT, int KT>
__global__ void __launch_bounds__(kDirectThreads, L::Q >= 27 ? 4 : 6)
    aa_step2_kernel(const __grid_constant__ StepArgs<float> a,
                    const __grid_constant__ DirectArgs d) {
  using P = Pop<K>;
  using T = typename P::type;
  using TL = typename TracerLattice<L::D>::type;
  using TP = TracerPop<KT>;
  using TT = typename TP::type;

  grid_trigger_next();
  const unsigned first = blockIdx.x * (unsigned)(2 * kDirectThreads) + threadIdx.x;
  CellPos c[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    unsigned cell = first + (unsigned)(k * kDirectThreads);
    if (cell >= d.cells) cell = first < d.cells ? first : 0u;  // a missing cell: see its flag
    const unsigned row = d.by_nz.div(cell);
    const unsigned x = L::D == 2 ? 0u : d.by_ny.div(row);
    c[k] = make_cellpos(a, (int)x, (int)(row - x * (unsigned)a.ny),
                        (int)(cell - row * (unsigned)a.nz), EVEN);
  }
  grid_wait_previous();
  if (first >= d.cells) return;
  const bool hasB = d.cells - first > (unsigned)kDirectThreads;
  const int flagA = a.flags[c[0].cell];
  const int flagB = hasB ? a.flags[c[1].cell] : 1;  // a missing cell acts as a wall
  float2 f[L::Q];
#pragma unroll
  for (int i = 0; i < L::Q; ++i) {
    const T* slot = static_cast<const T*>(d.slots.f[EVEN ? i : opp(i)]);
    f[i] = make_float2(
        P::load_dev(slot + (EVEN ? c[0].template upstream<L>(i) : c[0].cell), 0.0f),
        P::load_dev(slot + (EVEN ? c[1].template upstream<L>(i) : c[1].cell), 0.0f));
  }
  float2 g[NT == 1 ? TL::Q : 1];
  if constexpr (NT == 1) {
#pragma unroll
    for (int i = 0; i < TL::Q; ++i) {
      const TT* slot = static_cast<const TT*>(d.slots.g[EVEN ? i : opp(i)]);
      g[i] = make_float2(
          TP::load(slot + (EVEN ? c[0].template upstream<TL>(i) : c[0].cell), 0.0f),
          TP::load(slot + (EVEN ? c[1].template upstream<TL>(i) : c[1].cell), 0.0f));
    }
  }
  float2 cval = make_float2(0.0f, 0.0f);
  if (a.acc_mode == kAccBoussinesq)
    cval = make_float2(a.coupled_val[c[0].cell], a.coupled_val[c[1].cell]);
  update_cell2<L, TRT, K, EVEN, NT, KT>(a, GlobalPairSink<true>{d.slots, c[0], c[1]}, c[0], c[1], flagA,
                                        flagB, f, g, cval);
}

}  // namespace lbm
