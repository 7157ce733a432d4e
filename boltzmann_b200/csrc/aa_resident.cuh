// A whole iterate call of a 2D domain that fits on the chip, in one launch.
//
// Up to some hundred thousand cells, a step is over in a few microseconds, and most of that is the
// latency from one dependent grid to the next and the way of every population to L2 and back. Here
// each CTA (one per SM, a cooperative launch) keeps a rectangle of the domain in shared memory over
// all steps of the call; only what crosses between rectangles travels, through L2.
//
// The AA layout is kept: slot i of region cell p at [i][p], with a halo of two cells around the tile.
// An even step reads and writes slot i of the cell upstream of c_i, an odd step is local. Before each
// step pair the CTA receives the halo slots that the cells of its tile and of the ring around it read
// in the even step; it updates the ring's cells too (with the bits their owners compute), so the
// slots of its own cells that they write need not travel, and there is one exchange a pair.
//
// A message is one 64-bit word, value and sequence number, written and read with single 64-bit
// accesses at L2: the receiver polls the word itself until it carries the expected number, so an
// exchange costs one store and one load latency, with no fence and no flag behind the data. An
// owner publishes each value once, in one of two sets of words in turn: it comes back to a set two
// pairs later, and by then it has received the pair between from every CTA that reads its words
// (readers and writers are the same neighbours), which each of them sent after it had read the
// earlier set. Sequence numbers go on from launch to launch. Polls are bounded; a CTA that gives up
// sets status bit 1 and leaves, and so, one after the other, do its neighbours.
//
// The cells of a tile that touch no other tile are updated while the messages are under way.
//
// Bound by the instruction stream of the cell update on the larger domains (76% of issue slots at
// 1000 x 501), by the latency of one exchange and two updates a pair on the smallest. us a step,
// single-step launches and this kernel: 64^2 1.57 / 1.00, 256^2 1.98 / 1.33, 300^2 with a tracer
// 2.89 / 1.92, 512 x 500 3.68 / 2.48, 1000 x 501 TRT 6.01 / 4.36, 32 x 2000 1.99 / 1.34, FP16 500^2
// 3.29 / 2.56, FP64 256^2 3.28 / 2.74. (Two exchanges a pair without the ring's redundant cells: 1.75
// for 256^2, 5.61 for 1000 x 501. Slots at a run-time stride: 4.93 for 1000 x 501. At most 512
// threads a CTA: 5.03.)
#pragma once

#include <type_traits>

#include "aa_step.cuh"

namespace lbm {

// Polls of a word before a thread gives up, unless the simulation sets a limit: about a second.
constexpr unsigned kResidentPolls = 1u << 20;

// Threads of a CTA at most: the registers of an SM over what a thread of the variant needs.
template <int K, int NT>
__host__ __device__ constexpr int resident_threads() {
  return K == kF64 ? 512 : (NT == 1 ? 640 : 1024);
}

// Region cells between slots: a compile-time constant, so that a population's shared-memory address
// is the cell's plus an immediate. As many as fit an SM beside the message tables of a square tile.
template <int K, int NT, int KT>
__host__ __device__ constexpr int resident_stride() {
  constexpr int pop = (int)sizeof(typename Pop<K>::type), real = (int)sizeof(typename Pop<K>::real);
  constexpr int trc = (int)sizeof(typename TracerPop<KT>::type);
  constexpr int bytes = 9 * pop + (NT == 1 ? 5 * trc + real : 0) + 1;
  constexpr int slots = NT == 1 ? 15 : 9;
  int side = 16;  // of the region: (side - 4)^2 tile cells, messages of 16 table bytes each
  while ((side + 1) * (side + 1) * bytes + slots * (4 * (side + 1 - 4) + 4) * 16 + 128 <= 227 * 1024)
    ++side;
  return side * side / 16 * 16;
}

struct ResidentArgs {
  int gy, gz;      // tiles along the two axes; CTA = ty * gz + tz
  int steps;       // even
  int published;   // cells a CTA publishes of a slot at most
  int messages;    // table entries for receiving (and for sending) at most
  unsigned seq;    // sequence number of the first pair
  unsigned polls;  // of the words that a thread waits for at a time, before it gives up
  unsigned long long* mail[2];  // two sets of [words][CTAs][slots][published]
};

// Shared-memory layout of a variant (bytes).
template <int K, int NT, int KT>
struct ResidentStage {
  static constexpr int S = resident_stride<K, NT, KT>();
  static constexpr size_t off_g = (size_t)9 * S * sizeof(typename Pop<K>::type);
  static constexpr size_t off_val =
      off_g + (NT == 1 ? (size_t)5 * S * sizeof(typename TracerPop<KT>::type) : 0);
  static constexpr size_t off_flag = off_val + (NT == 1 ? (size_t)S * sizeof(typename Pop<K>::real) : 0);
  static constexpr size_t off_table = off_flag + S;
};

// First row (or column) of tile t of g over n, and the tile of row y. (The products stay below 2^32:
// a resident domain has fewer than 2^22 rows, and tiles are no more than SMs.)
__host__ __device__ __forceinline__ int tile_first(int t, int g, int n) {
  return (int)((unsigned)t * (unsigned)n / (unsigned)g);
}
__host__ __device__ __forceinline__ int tile_of(int y, int g, int n) {
  return (int)(((unsigned)(y + 1) * (unsigned)g - 1) / (unsigned)n);
}
// A coordinate at most one past either end of a periodic axis of n cells.
__device__ __forceinline__ int wrapped(int y, int n) { return y < 0 ? y + n : (y >= n ? y - n : y); }

// One population from global to shared memory: an asynchronous copy where the type allows it (four
// or eight bytes), so that a thread has all of its cells' loads in flight.
template <class T>
__device__ __forceinline__ void fetch_pop(T* dst, const T* src) {
  if constexpr (sizeof(T) >= 4)
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "n"(sizeof(T))
                 : "memory");
  else
    *dst = *src;
}

// Halo cells whose slot with velocity (cy, cz) is read by a cell of the tile or of the ring around
// it: the (h + 2) x (w + 2) rectangle shifted against the velocity, without the tile. Their number
// is the same for every slot; entry k of them.
__host__ __device__ __forceinline__ int halo_entries(int h, int w) { return 2 * (h + w) + 4; }
__host__ __device__ __forceinline__ void halo_cell(int k, int cy, int cz, int h, int w, int& r, int& c) {
  if (k < 2 * (w + 2)) {  // the two rows outside the tile
    const int j = k >= w + 2;
    r = cy == 0 ? (j ? h : -1) : (cy > 0 ? j - 2 : h + j);
    c = k - j * (w + 2) - 1 - cz;
  } else {  // two cells a row beside it
    const int e = k - 2 * (w + 2), j = e & 1;
    r = e >> 1;
    c = cz == 0 ? (j ? w : -1) : (cz > 0 ? j - 2 : w + j);
  }
}

// Cells on the rim of an h x w rectangle, and entry k of them.
__host__ __device__ __forceinline__ int rim_cells(int h, int w) {
  return h <= 2 || w <= 2 ? h * w : 2 * (h + w) - 4;
}
__host__ __device__ __forceinline__ void rim_cell(int k, int h, int w, int& r, int& c) {
  if (h <= 2 || w <= 2) {
    r = k / w;
    c = k - r * w;
  } else if (k < 2 * w) {
    r = k < w ? 0 : h - 1;
    c = k < w ? k : k - w;
  } else {
    r = 1 + ((k - 2 * w) >> 1);
    c = (k - 2 * w) & 1 ? w - 1 : 0;
  }
}

// Cells of the tile whose slot with velocity (cy, cz) is read by a cell that some other tile updates
// too (on the rim, or outside): the tile without its interior shifted against the velocity. As many
// as rim_cells for every slot; entry k of them, and the entry of cell (r, c) that is one of them.
__host__ __device__ __forceinline__ void published_cell(int k, int cy, int cz, int h, int w, int& r,
                                                        int& c) {
  if (h <= 2 || w <= 2) {
    r = k / w;
    c = k - r * w;
  } else if (k < 2 * w) {  // two rows
    const int j = k >= w;
    r = cy == 0 ? (j ? h - 1 : 0) : (cy > 0 ? h - 2 + j : j);
    c = k - j * w;
  } else {  // two cells of every other row
    const int e = k - 2 * w, j = e & 1;
    r = (e >> 1) + 1 - cy;
    c = cz == 0 ? (j ? w - 1 : 0) : (cz > 0 ? w - 2 + j : j);
  }
}
__host__ __device__ __forceinline__ int published_index(int r, int c, int cy, int cz, int h, int w) {
  if (h <= 2 || w <= 2) return r * w + c;
  const int row = cy == 0 ? (r == 0 ? 0 : (r == h - 1 ? 1 : -1))
                          : (cy > 0 ? r - (h - 2) : (r < 2 ? r : -1));
  if (row >= 0) return row * w + c;
  const int col = cz == 0 ? (c == 0 ? 0 : 1) : (cz > 0 ? c - (w - 2) : c);
  return 2 * w + 2 * (r - 1 + cy) + col;
}

__device__ __forceinline__ void mail_put(unsigned long long* p, unsigned v, unsigned seq) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p),
               "l"((unsigned long long)v | ((unsigned long long)seq << 32))
               : "memory");
}
__device__ __forceinline__ unsigned long long mail_peek(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// A stored population as message words: one, or two for FP64.
template <class T>
__host__ __device__ constexpr int mail_words() {
  return sizeof(T) == 8 ? 2 : 1;
}
template <class T>
__device__ __forceinline__ unsigned word_of(const T* p, int k) {
  if constexpr (sizeof(T) == 2)
    return *reinterpret_cast<const unsigned short*>(p);
  else
    return reinterpret_cast<const unsigned*>(p)[k];
}
template <class T>
__device__ __forceinline__ void set_word(T* p, int k, unsigned v) {
  if constexpr (sizeof(T) == 2)
    *reinterpret_cast<unsigned short*>(p) = (unsigned short)v;
  else
    reinterpret_cast<unsigned*>(p)[k] = v;
}

// update_cell's results into the region (see the layout above).
template <int STRIDE, size_t OFF_G>
struct ResidentSink {
  unsigned char* sm;
  int p, rz;  // region index of the cell, region columns

  template <class LL, bool EVEN>
  __device__ __forceinline__ int pos(int i) const {
    return EVEN ? p - comp<LL>(i, 1) * rz - comp<LL>(i, 2) : p;
  }
  template <class LL, class P, bool EVEN, bool DEV>
  __device__ __forceinline__ void fluid(void*, long long, const CellPos&,
                                        const typename P::real (&v)[LL::Q]) const {
    using T = typename P::type;
    using Real = typename P::real;
    T* base = reinterpret_cast<T*>(sm);
#pragma unroll
    for (int i = 0; i < LL::Q; ++i) {
      T* q = base + i * STRIDE + pos<LL, EVEN>(i);
      const Real val = EVEN ? v[opp(i)] : v[i];
      if constexpr (DEV)
        P::store_dev(q, val, weight<LL, Real>(i));
      else
        P::store(q, val, weight<LL, Real>(i));
    }
  }
  template <class TLL, class TP, bool EVEN>
  __device__ __forceinline__ void tracer(void*, long long, const CellPos&,
                                         const typename TP::real (&v)[TLL::Q]) const {
    using TT = typename TP::type;
    TT* base = reinterpret_cast<TT*>(sm + OFF_G);
#pragma unroll
    for (int i = 0; i < TLL::Q; ++i)
      TP::store(base + i * STRIDE + pos<TLL, EVEN>(i), EVEN ? v[opp(i)] : v[i], 0.0f);
  }
};

template <class L, bool TRT, int K, int NT, int KT>
__global__ void __launch_bounds__(resident_threads<K, NT>())
    aa_resident_kernel(const __grid_constant__ StepArgs<typename Pop<K>::real> a,
                       const __grid_constant__ ResidentArgs d) {
  using P = Pop<K>;
  using Real = typename P::real;
  using T = typename P::type;
  using TL = typename TracerLattice<L::D>::type;
  using TP = TracerPop<KT>;
  using TT = typename TP::type;
  constexpr int W = mail_words<T>();
  constexpr int NS = L::Q + (NT == 1 ? TL::Q + 1 : 0);  // published slots: f, g, tracer value
  using St = ResidentStage<K, NT, KT>;
  constexpr int S = St::S;
  using Sink = ResidentSink<S, St::off_g>;
  static_assert(NT == 0 || mail_words<TT>() <= W, "a tracer's words fit the fluid's");

  extern __shared__ __align__(16) unsigned char res_smem[];
  unsigned char* sm = res_smem;
  T* fs = reinterpret_cast<T*>(sm);
  TT* gs = reinterpret_cast<TT*>(sm + St::off_g);
  Real* vals = reinterpret_cast<Real*>(sm + St::off_val);
  unsigned char* flags = sm + St::off_flag;

  const int tid = threadIdx.x, nthreads = blockDim.x;
  const int ty = blockIdx.x / d.gz, tz = blockIdx.x - ty * d.gz;
  const int y0 = tile_first(ty, d.gy, a.ny), z0 = tile_first(tz, d.gz, a.nz);
  const int h = tile_first(ty + 1, d.gy, a.ny) - y0, w = tile_first(tz + 1, d.gz, a.nz) - z0;
  const int rz = w + 4;
  auto region = [&](int r, int c) { return (r + 2) * rz + c + 2; };
  // Byte offset in shared memory of published slot s (0 .. NS - 1) of region cell p, and its size.
  auto slot_at = [&](int s, int p) -> unsigned {
    if (NT == 0 || s < L::Q) return (unsigned)((size_t)(s * S + p) * sizeof(T));
    if (s < L::Q + TL::Q)
      return (unsigned)(St::off_g + (size_t)((s - L::Q) * S + p) * sizeof(TT));
    return (unsigned)(St::off_val + (size_t)p * sizeof(Real));
  };
  auto velocity = [&](int s, int& cy, int& cz) {  // of published slot s (the value: at rest)
    const int i = s < L::Q ? s : (s < L::Q + TL::Q ? s - L::Q : 0);
    cy = comp_rt<L, 1>(i);  // D2Q5's slots are D2Q9's first five
    cz = comp_rt<L, 2>(i);
  };
  // Message tables, {byte offset in shared memory, word}: the published slots of this CTA's cells that
  // another tile (or its ring) reads, and the halo slots this one reads.
  uint2* tx = reinterpret_cast<uint2*>(sm + St::off_table);
  uint2* rx = tx + d.messages;
  const int ntx = NS * rim_cells(h, w), nrx = NS * halo_entries(h, w);
  for (int e = tid; e < ntx; e += nthreads) {
    const int s = e / rim_cells(h, w), k = e - s * rim_cells(h, w);
    int cy, cz, r, c;
    velocity(s, cy, cz);
    published_cell(k, cy, cz, h, w, r, c);
    tx[e] = make_uint2(slot_at(s, region(r, c)), (unsigned)((blockIdx.x * NS + s) * d.published + k));
  }
  for (int e = tid; e < nrx; e += nthreads) {
    const int s = e / halo_entries(h, w), k = e - s * halo_entries(h, w);
    int cy, cz, r, c;
    velocity(s, cy, cz);
    halo_cell(k, cy, cz, h, w, r, c);
    // Up to two past either end: twice, for a domain of a single row or column.
    const int y = wrapped(wrapped(y0 + r, a.ny), a.ny), z = wrapped(wrapped(z0 + c, a.nz), a.nz);
    const int oy = tile_of(y, d.gy, a.ny), oz = tile_of(z, d.gz, a.nz);
    const int fy = tile_first(oy, d.gy, a.ny), fz = tile_first(oz, d.gz, a.nz);
    const int oh = tile_first(oy + 1, d.gy, a.ny) - fy, ow = tile_first(oz + 1, d.gz, a.nz) - fz;
    rx[e] = make_uint2(slot_at(s, region(r, c)),
                       (unsigned)(((oy * d.gz + oz) * NS + s) * d.published +
                                  published_index(y - fy, z - fz, cy, cz, oh, ow)));
  }

  // The tile into the region, and the flags of the tile and its ring (the other halo slots come as
  // messages).
  const FastDiv by_w((unsigned)w), by_ring((unsigned)(w + 2));
  const unsigned n = (unsigned)(h * w), nring = (unsigned)((h + 2) * (w + 2));
  for (unsigned i = tid; i < nring; i += nthreads) {
    const int r = (int)by_ring.div(i), c = (int)i - r * (w + 2);
    const int y = wrapped(y0 + r - 1, a.ny), z = wrapped(z0 + c - 1, a.nz);
    flags[region(r - 1, c - 1)] = a.flags[(unsigned)y * (unsigned)a.nz + (unsigned)z];
  }
#pragma unroll 2
  for (unsigned i = tid; i < n; i += nthreads) {
    const unsigned r = by_w.div(i), c = i - r * w;
    const unsigned cell = (y0 + r) * (unsigned)a.nz + z0 + c;
    const int p = region((int)r, (int)c);
    if constexpr (sizeof(T) >= 4) {
#pragma unroll
      for (int q = 0; q < L::Q; ++q)
        fetch_pop(fs + q * S + p, static_cast<const T*>(a.f) + (size_t)q * a.n + cell);
    } else {  // all loads of a cell before its first store
      T v[L::Q];
#pragma unroll
      for (int q = 0; q < L::Q; ++q) v[q] = static_cast<const T*>(a.f)[(size_t)q * a.n + cell];
#pragma unroll
      for (int q = 0; q < L::Q; ++q) fs[q * S + p] = v[q];
    }
    if constexpr (NT == 1) {
#pragma unroll
      for (int q = 0; q < TL::Q; ++q)
        fetch_pop(gs + q * S + p, static_cast<const TT*>(a.tr[0].g) + (size_t)q * a.n + cell);
      fetch_pop(vals + p, a.tr[0].val + cell);
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();

  auto update = [&](auto even, const StepArgs<Real>& args, int r, int c, unsigned cell) {
    constexpr bool EVEN = decltype(even)::value;
    const int p = region(r, c);
    const Sink sink{sm, p, rz};
    const int flag = flags[p];
    Real f[L::Q];
#pragma unroll
    for (int q = 0; q < L::Q; ++q) {
      const T* src = EVEN ? fs + q * S + sink.template pos<L, true>(q)
                          : fs + opp(q) * S + p;
      if constexpr (dev_in<K>())
        f[q] = P::load_dev(src, weight<L, Real>(q));
      else
        f[q] = P::load(src, weight<L, Real>(q));
    }
    Real g[NT == 1 ? TL::Q : 1];
    Real cval = 0;
    CellPos at;
    at.cell = cell;
    StepArgs<Real> b = args;
    if constexpr (NT == 1) {
#pragma unroll
      for (int q = 0; q < TL::Q; ++q)
        g[q] = TP::load(EVEN ? gs + q * S + sink.template pos<TL, true>(q)
                             : gs + opp(q) * S + p, 0.0f);
      cval = vals[p];
      b.tr[0].val = vals + ((ptrdiff_t)p - (ptrdiff_t)cell);  // tracer_update indexes it by cell
    }
    update_cell<L, TRT, K, EVEN, NT, Sink, KT>(b, at, flag, f, g, cval, a.om_pos, a.om_neg,
                                                       sink);
  };
  using Even = std::integral_constant<bool, true>;
  using Odd = std::integral_constant<bool, false>;
  const int ih = h - 2, iw = w - 2;  // cells that touch no other tile
  // Taken apart above 256 cells, where they hide the messages (200 x 150: 1.24 us a step, 1.33 in
  // one go); below, one pass of few warps is latency itself, and two are twice that.
  const bool apart = ih > 0 && iw > 0 && (h + 2) * (w + 2) > 256;
  const unsigned ni = apart ? (unsigned)(ih * iw) : 0u;
  const FastDiv by_iw((unsigned)(iw > 0 ? iw : 1));
  // The even step's other cells: the tile's rim (or all of it) and the ring around it.
  const int ntile_rim = (int)(n - ni), nouter = apart ? ntile_rim + rim_cells(h + 2, w + 2) : (int)nring;

  StepArgs<Real> now = a;  // only the last step of a call writes moments
  unsigned seq = d.seq;
  const size_t set_words = (size_t)gridDim.x * NS * d.published;
  bool ok = d.polls > 0;
  for (int s = 0; s < d.steps; s += 2, ++seq) {
    unsigned long long* box = d.mail[seq & 1u];
    for (int e = tid; e < ntx; e += nthreads) {
      const uint2 m = tx[e];
      const bool value = NT == 1 && e >= (NS - 1) * rim_cells(h, w);
      const bool tracer = NT == 1 && e >= L::Q * rim_cells(h, w) && !value;
      const unsigned char* src = sm + m.x;
      if (tracer) {
#pragma unroll
        for (int k = 0; k < mail_words<TT>(); ++k)
          mail_put(box + k * set_words + m.y, word_of(reinterpret_cast<const TT*>(src), k), seq);
      } else if (value) {
#pragma unroll
        for (int k = 0; k < mail_words<Real>(); ++k)
          mail_put(box + k * set_words + m.y, word_of(reinterpret_cast<const Real*>(src), k), seq);
      } else {
#pragma unroll
        for (int k = 0; k < W; ++k)
          mail_put(box + k * set_words + m.y, word_of(reinterpret_cast<const T*>(src), k), seq);
      }
    }

    now.write_moments = 0;
    for (unsigned i = tid; i < ni; i += nthreads) {
      const int r = (int)by_iw.div(i) + 1, c = (int)i - (r - 1) * iw + 1;
      update(Even{}, now, r, c, (unsigned)(y0 + r) * (unsigned)a.nz + (unsigned)(z0 + c));
    }

    // Four messages of a thread at a time, polled together.
    constexpr int B = 4;
    for (int e0 = tid; e0 < nrx && ok; e0 += B * nthreads) {
      uint2 m[B];
      unsigned long long v[W][B];
      bool need[B];
#pragma unroll
      for (int j = 0; j < B; ++j) {
        const int e = e0 + j * nthreads;
        need[j] = e < nrx;
        m[j] = need[j] ? rx[e] : make_uint2(0u, 0u);
#pragma unroll
        for (int k = 0; k < W; ++k) v[k][j] = need[j] ? mail_peek(box + k * set_words + m[j].y) : 0ull;
      }
      unsigned polls = 0;
#pragma unroll
      for (int j = 0; j < B; ++j) {
        if (!need[j]) continue;
        const int e = e0 + j * nthreads;
        const bool value = NT == 1 && e >= (NS - 1) * halo_entries(h, w);
        const bool tracer = NT == 1 && e >= L::Q * halo_entries(h, w) && !value;
        const int nk = tracer ? mail_words<TT>() : (value ? mail_words<Real>() : W);
        unsigned char* dst = sm + m[j].x;
#pragma unroll
        for (int k = 0; k < W; ++k) {
          if (k >= nk) break;
          while ((unsigned)(v[k][j] >> 32) != seq) {
            if (++polls > d.polls) {
              ok = false;
              break;
            }
            v[k][j] = mail_peek(box + k * set_words + m[j].y);
          }
          if (tracer)
            set_word(reinterpret_cast<TT*>(dst), k, (unsigned)v[k][j]);
          else if (value)
            set_word(reinterpret_cast<Real*>(dst), k, (unsigned)v[k][j]);
          else
            set_word(reinterpret_cast<T*>(dst), k, (unsigned)v[k][j]);
        }
      }
    }
    if (!__syncthreads_and(ok)) {
      ok = false;
      break;
    }
    for (int i = tid; i < nouter; i += nthreads) {
      int r, c;
      if (!apart) {
        r = (int)by_ring.div((unsigned)i);
        c = i - r * (w + 2) - 1;
        --r;
      } else if (i < ntile_rim) {
        rim_cell(i, h, w, r, c);
      } else {
        rim_cell(i - ntile_rim, h + 2, w + 2, r, c);
        --r;
        --c;
      }
      update(Even{}, now, r, c,
             (unsigned)wrapped(y0 + r, a.ny) * (unsigned)a.nz + (unsigned)wrapped(z0 + c, a.nz));
    }
    __syncthreads();
    now.write_moments = s + 2 < d.steps ? 0 : a.write_moments;
    for (unsigned i = tid; i < n; i += nthreads) {
      const int r = (int)by_w.div(i), c = (int)i - r * w;
      update(Odd{}, now, r, c, (unsigned)(y0 + r) * (unsigned)a.nz + (unsigned)(z0 + c));
    }
    __syncthreads();
  }
  if (!ok) {
    if (tid == 0) atomicOr(a.status, 2);
    return;
  }

  for (unsigned i = tid; i < n; i += nthreads) {
    const unsigned r = by_w.div(i), c = i - r * w;
    const unsigned cell = (y0 + r) * (unsigned)a.nz + z0 + c;
    const int p = region((int)r, (int)c);
#pragma unroll
    for (int q = 0; q < L::Q; ++q) static_cast<T*>(a.f)[(size_t)q * a.n + cell] = fs[q * S + p];
    if constexpr (NT == 1) {
#pragma unroll
      for (int q = 0; q < TL::Q; ++q)
        static_cast<TT*>(a.tr[0].g)[(size_t)q * a.n + cell] = gs[q * S + p];
      a.tr[0].val[cell] = vals[p];
    }
  }
}

}  // namespace lbm
