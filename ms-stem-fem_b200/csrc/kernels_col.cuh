// The column slice pass (also as a slot lane's in FP32; the last slice's stops in
// k-space):
// DFT_x, / s, band limit, propagator, iDFT_x, two adjacent FP32 columns or one
// FP64 column per thread (fft_lines.cuh).  An element is 16 bytes either way,
// so both precisions share the kernels.
//
// What bounds it: a column tile is rows of COLS x 8 (FP64: 16) bytes, and the
// memory system serves about 50 to 65 G requests/s of at most one 128-byte line
// each, whatever part of the line they carry.  An in-place copy of a 1024^2
// batch runs at 2.6-2.9 TB/s with 64-byte rows, 4.9 with 128-byte and 6.0 with
// 256-byte ones (direct loads and stores; TMA tiles of the same width move no
// faster).  So tiles are 128 bytes wide wherever a tile of that width fits an
// SM, and the two kernels differ in how they keep loads in flight beside it:
//
//  * up to 512 points, col_ring_kernel: three tile buffers and two groups of
//    threads that work on different tiles out of step; a tile is transformed
//    in place and leaves by TMA, the third buffer is in flight meanwhile.
//    512^2, 256 probes, FP32: 0.18 ms against 0.22 ms for one 16-column tile
//    of one column per thread behind CTA barriers; 256 points: 0.048 against
//    0.069 ms.  The long-column kernel loses at both (by 10 %).  FP64 tiles of 128
//    and 256 points take three groups and five buffers.
//  * from 1024 points, col_wide_kernel: the tile (128 KB) leaves no room for a
//    second one, so it is read into registers, refilled by TMA at once, and
//    the transforms exchange half a tile (real parts, then imaginary parts)
//    at a time through a 64 KB buffer.  FP32, 1024^2, 256 probes: 0.71 ms
//    against 0.90 ms for two 8-column buffers (64-byte rows); 2048^2, 64
//    probes, 8 columns: 0.87 against 1.25 ms with 4; 4096^2, 16 probes, 4
//    columns: 1.13 ms against 4.4 ms for one column per CTA.  Left: the stores
//    of a tile leave in one burst behind its last stage, which the next tile's
//    first loads wait for.
//
// A batch that does not fill the SMs once pays for the tile copy's latency: up to
// 16 probes at 64^2 10.9 us a launch against 8.9 with direct loads, at 1024 x 64
// 19 against 14.6.
//
// FP64, the same kernels, us a probe: 1024^2 8.45 -> 5.47, 512^2 2.18 -> 1.42 (64
// probes), 256^2 0.45 -> 0.33 (256 probes) against a double-buffered TMA pass of
// half the tile width, 2048^2 67.9 -> 32.7 (16 probes) against a plain strided one.
//
// Every wait is bounded: if a phase does not complete within kSpinLimit polls
// the waiting group records an error in *err and leaves its loop; copies still
// in flight are waited for (bounded again) before the CTA ends.
#pragma once
#include <cuda.h>

#include "async_copy.cuh"
#include "fft_lines.cuh"
#include "kernels.h"

namespace msf {

namespace {

// Product of a thread's column elements with the propagator and the band
// limit: v[m] <- P_x P_y v[m] / s inside the limit (i < lo or i >= hi), else 0
// (slice.cpp:1396-1412).  px(i): the x propagator; a ColumnEdge: what the
// thread's column, or two columns, bring.
template <class V> struct ColumnEdge;
template <> struct ColumnEdge<Pair> {
  int2 lo{}, hi{};
  float4 py{};
  __device__ __forceinline__ void load(const int32_t* mlo, const int32_t* mhi, const void* p,
                                       int j) {
    lo = __ldg(reinterpret_cast<const int2*>(mlo + j));
    hi = __ldg(reinterpret_cast<const int2*>(mhi + j));
    py = __ldg(reinterpret_cast<const float4*>(static_cast<const float2*>(p) + j));
  }
};
template <> struct ColumnEdge<double2> {
  int lo = 0, hi = 0;
  double2 py{};
  __device__ __forceinline__ void load(const int32_t* mlo, const int32_t* mhi, const void* p,
                                       int j) {
    lo = __ldg(mlo + j);
    hi = __ldg(mhi + j);
    py = __ldg(static_cast<const double2*>(p) + j);
  }
};
template <class Sh, class Px>
__device__ __forceinline__ void propagate(Pair (&v)[Sh::E], int t, Px&& px,
                                          const ColumnEdge<Pair>& e, float inv_s) {
  constexpr int E = Sh::E, T = Sh::T;
  const float2 pr = make_float2(e.py.x * inv_s, e.py.z * inv_s);
  const float2 pi = make_float2(e.py.y * inv_s, e.py.w * inv_s);
  sfor<0, E>([&](auto mI) {
    constexpr int m = decltype(mI)::value;
    if constexpr (dead_slot<E>(m)) {
      v[m] = vzero<Pair>();
    } else {
      const int i = t + T * m;
      const float2 p = px(i);
      const float2 qr = f2fma(f2(p.x), pr, f2mul(f2(-p.y), pi));
      const float2 qi = f2fma(f2(p.x), pi, f2mul(f2(p.y), pr));
      Pair r{f2fma(qr, v[m].re, f2mul(f2neg(qi), v[m].im)),
             f2fma(qr, v[m].im, f2mul(qi, v[m].re))};
      if (!(i < e.lo.x || i >= e.hi.x)) r.re.x = r.im.x = 0.f;
      if (!(i < e.lo.y || i >= e.hi.y)) r.re.y = r.im.y = 0.f;
      v[m] = r;
    }
  });
}
template <class Sh, class Px>
__device__ __forceinline__ void propagate(double2 (&v)[Sh::E], int t, Px&& px,
                                          const ColumnEdge<double2>& e, double inv_s) {
  constexpr int E = Sh::E, T = Sh::T;
  sfor<0, E>([&](auto mI) {
    constexpr int m = decltype(mI)::value;
    const int i = t + T * m;
    if (!dead_slot<E>(m) && (i < e.lo || i >= e.hi))
      v[m] = cmul(cmul(px(i), e.py), cscale(v[m], inv_s));
    else
      v[m] = vzero<double2>();
  });
}

// What a probe brings to its column pass: the launch's tables, or (SLOTS) its
// slot's.
struct ColTables {
  const int32_t *lo, *hi;
  const void *px, *py;
  bool idle, stop_in_k;
};
template <bool LAST, bool SLOTS>
__device__ __forceinline__ ColTables col_tables(const PassArgs& a, int b) {
  if constexpr (SLOTS) {
    const SlotPass& s = a.slots[b];
    return ColTables{s.mask_lo, s.mask_hi, s.px, s.py, s.op == SLOT_IDLE, s.last != 0};
  } else {
    return ColTables{a.mask_lo, a.mask_hi, a.px, a.py, false, LAST};
  }
}

// Item -> first column (of the live column groups, when given) and probe.
template <int COLS>
__device__ __forceinline__ int item_column(const PassArgs& a, int item, int& b) {
  const int gi = item / a.nb;
  b = item - gi * a.nb;
  return (a.live_groups ? __ldg(a.live_groups + gi) : gi) * COLS;
}

// columns an element holds, and the 8-byte tensor-map elements of a column
template <class V> __host__ __device__ constexpr int elem_cols() {
  return sizeof(typename LineOf<V>::Real) == 4 ? 2 : 1;
}
template <class V> __host__ __device__ constexpr int col_words() { return 2 / elem_cols<V>(); }

// --------------------------------------------------- up to 512 points ------
constexpr int kRingElems = 8;  // 128-byte tile rows
template <int N> __host__ __device__ constexpr int ring_group() {  // threads of a tile
  return kRingElems * ColShape<N>::T;
}
// 32 elements a thread take 255 registers (256 threads an SM), FP32's 16 take 128
// (512).  FP64's 16 take 168 (384, in three groups): at 128 registers the 256-point
// pass spills 568 / 628 bytes (stores / loads) and takes 0.464 us a probe, at 168 it
// spills 72 / 144 and takes 0.332.  What else spills: FP64 128 points 52 / 84, 512
// points 52 / 100; FP32 128 and 512 points 28 / 52, the slot form of 256 156 / 112.
template <class V, int N> __host__ __device__ constexpr bool ring_three() {
  return elem_cols<V>() == 1 && ColShape<N>::E == 16;
}
template <class V, int N> __host__ __device__ constexpr int ring_groups() {
  return ring_three<V, N>() ? 3 : 2;
}
template <class V, int N> __host__ __device__ constexpr int ring_bufs() {
  return ring_three<V, N>() ? 5 : 3;
}
template <class V, int N> __host__ __device__ constexpr int ring_ctas() {
  constexpr int threads = ColShape<N>::E >= 32 ? 256 : ring_three<V, N>() ? 384 : 512;
  return threads / (ring_group<N>() * ring_groups<V, N>());
}
template <class V, int N> __host__ __device__ constexpr int ring_smem() {
  return ring_bufs<V, N>() * N * kRingElems * 16 + 1024;  // buffers start on 1024 bytes
}

template <class V, int N, bool LAST, bool SLOTS>
__global__ void __launch_bounds__(ring_group<N>() * ring_groups<V, N>(), ring_ctas<V, N>())
col_ring_kernel(const PassArgs a, const __grid_constant__ CUtensorMap tmap, int* err) {
  using Sh = ColShape<N>;
  using Mem = typename LineOf<V>::Mem;
  using C = typename LineOf<V>::C;
  using Real = typename LineOf<V>::Real;
  constexpr int E = Sh::E, T = Sh::T, PC = kRingElems, EC = elem_cols<V>(), COLS = PC * EC;
  constexpr int G = ring_groups<V, N>(), GT = ring_group<N>(), NBUF = ring_bufs<V, N>();
  constexpr int BOX = N < 256 ? N : 256, BUF = N * PC * 16;
  static_assert(T <= 32, "a line's threads share a warp");
  static_assert(NBUF > G, "a buffer is reloaded by its group's next item");
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* bufs = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  __shared__ uint64_t bars[NBUF];
  __shared__ int issued[NBUF];
  __shared__ int flags[G];
  const int g = threadIdx.x / GT, tg = threadIdx.x % GT;
  const int c = tg / T, t = tg % T;  // element column of the tile, thread of the line
  const int items = a.nb * (a.live_groups ? a.n_live_groups : a.ny / COLS);
  const int count = ((int)blockIdx.x < items)
                        ? (items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
  auto load = [&](int k) {  // this CTA's k-th item
    int b;
    const int x = item_column<COLS>(a, blockIdx.x + k * gridDim.x, b);
    unsigned char* dst = bufs + (k % NBUF) * BUF;
    mbar_expect_tx(&bars[k % NBUF], BUF);
#pragma unroll
    for (int q = 0; q < N / BOX; ++q)
      tile_g2s(dst + q * BOX * PC * 16, &tmap, x * col_words<V>(), b * a.nx + q * BOX,
               &bars[k % NBUF]);
    *(volatile int*)&issued[k % NBUF] = k / NBUF + 1;
  };
  // The load of item k has been issued (by the group that freed its buffer)
  // and has landed.  The count comes first: while the buffer's previous item
  // is still on its way, the parity alone would report the one before that.
  auto landed = [&](int k) {
    for (uint32_t it = 0; it < kSpinLimit; ++it)
      if (*(volatile int*)&issued[k % NBUF] > k / NBUF)
        return mbar_wait_bounded(&bars[k % NBUF], (k / NBUF) & 1);
    return false;
  };
  auto line_sync = [] { __syncwarp(); };
  if (threadIdx.x == 0) {
    for (int q = 0; q < NBUF; ++q) {
      mbar_init(&bars[q], 1);
      issued[q] = 0;
    }
    mbar_fence_init();
    for (int k = 0; k < NBUF && k < count; ++k) load(k);
  }
  __syncthreads();
  const GlobalTable<C> tw{static_cast<const C*>(a.tw)};
  const Real inv_s = (Real)a.inv_s;
  int reload = -1;  // item to load once the store of the last one has been read out
  for (int k = g; k < count; k += G) {
    const int w = k % NBUF;
    unsigned char* buf = bufs + w * BUF;
    int b;
    const int j0 = item_column<COLS>(a, blockIdx.x + k * gridDim.x, b), j = j0 + EC * c;
    const ColTables tab = col_tables<LAST, SLOTS>(a, b);
    if (tg == 0) flags[g] = landed(k) ? 1 : 0;
    bar_sync(1 + g, GT);
    if (!flags[g]) {
      if (tg == 0) atomicExch(err, 1);
      break;
    }
    mbar_wait_bounded(&bars[w], (k / NBUF) & 1);  // every thread observes the phase
    // chunk c of row r in the tile as TMA's 128-byte swizzle lays it out
    auto row = [&](int r) { return reinterpret_cast<Mem*>(buf) + r * PC + (c ^ (r & 7)); };
    auto at = [&](int s) { return row(line_slot<Sh>(s)); };
    V v[E];
    if (!tab.idle) {
#pragma unroll
      for (int m = 0; m < E; ++m) get_cols(row(t + T * m), v[m]);
    }
    if (tg == 0 && reload >= 0) {
      bulk_wait_read();
      load(reload);
      reload = -1;
    }
    if (!tab.idle) {
      line_sync();
      fft_lines<Sh, false, false, true>(v, t, tw, at, line_sync);
      ColumnEdge<V> edge;
      edge.load(tab.lo, tab.hi, tab.py, j);
      const C* px = static_cast<const C*>(tab.px);
      propagate<Sh>(v, t, [&](int i) { return __ldg(px + i); }, edge, inv_s);
      line_sync();  // the transform's exchange has been read by all
      if (!tab.stop_in_k) fft_lines<Sh, true, true, false>(v, t, tw, at, line_sync, line_sync);
#pragma unroll
      for (int m = 0; m < E; ++m) put_cols(row(t + T * m), v[m]);
      fence_proxy_async();
    }
    bar_sync(1 + g, GT);
    if (tg == 0) {
      if (!tab.idle) {
#pragma unroll
        for (int q = 0; q < N / BOX; ++q)
          tile_s2g(&tmap, j0 * col_words<V>(), b * a.nx + q * BOX, buf + q * BOX * PC * 16);
        bulk_commit();
      }
      if (k + NBUF < count) reload = k + NBUF;
    }
  }
  if (tg == 0) bulk_wait_all();
  __syncthreads();
  if (threadIdx.x == 0)  // nothing is in flight here unless a wait gave up
    for (int q = 0; q < NBUF; ++q)
      if (issued[q] > 0) mbar_wait_bounded(&bars[q], (issued[q] - 1) & 1);
}

// ---------------------------------------------------- from 1024 points -----
template <int N> __host__ __device__ constexpr int wide_elems() { return 8192 / N; }
constexpr int kWideThreads = 256;  // 8192 elements, 32 a thread
// exchange slots: one of padding every R0, so that the stride-R0 writes of
// neighbouring threads fall on different banks
template <int N> __host__ __device__ constexpr int wide_slots() {
  return N + N / ColShape<N>::radix(0);
}
template <class V, int N> __host__ __device__ constexpr int wide_tw() {  // twiddles
  return ColShape<N>::tw_off(ColShape<N>::S, fused_twiddles<typename LineOf<V>::Real, N>());
}
template <class V, int N> __host__ __device__ constexpr int wide_base() {
  return N * wide_elems<N>() * 16 + wide_slots<N>() * wide_elems<N>() * 8;
}
// which tables fit in shared memory too: the twiddles, then the slice's x
// propagator
template <class V, int N> __host__ __device__ constexpr bool wide_tw_fits() {
  return wide_base<V, N>() + wide_tw<V, N>() * (int)sizeof(typename LineOf<V>::C) <= 226 * 1024;
}
template <class V, int N> __host__ __device__ constexpr bool wide_px_fits() {
  return wide_tw_fits<V, N>() &&
         wide_base<V, N>() + (wide_tw<V, N>() + N) * (int)sizeof(typename LineOf<V>::C) <= 226 * 1024;
}
template <class V, int N> __host__ __device__ constexpr int wide_smem() {
  return wide_base<V, N>() +
         ((wide_tw_fits<V, N>() ? wide_tw<V, N>() : 0) + (wide_px_fits<V, N>() ? N : 0)) *
             (int)sizeof(typename LineOf<V>::C);
}

template <class V, int N, bool LAST, bool SLOTS>
__global__ void __launch_bounds__(kWideThreads, 1)
col_wide_kernel(const PassArgs a, const __grid_constant__ CUtensorMap tmap, int* err) {
  using Sh = ColShape<N>;
  using Mem = typename LineOf<V>::Mem;
  using C = typename LineOf<V>::C;
  using Real = typename LineOf<V>::Real;
  using Half = typename LineOf<V>::Half;
  constexpr int E = Sh::E, T = Sh::T, PC = wide_elems<N>(), EC = elem_cols<V>(), COLS = PC * EC;
  constexpr int BOX = 256, SHIFT = ilog2(Sh::radix(0));
  static_assert(PC * T == kWideThreads);
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  Mem* tile = reinterpret_cast<Mem*>(smem_raw);
  Half* xb = reinterpret_cast<Half*>(smem_raw + N * PC * 16);
  C* tw_s = reinterpret_cast<C*>(smem_raw + wide_base<V, N>());
  C* px_s = tw_s + wide_tw<V, N>();
  __shared__ uint64_t bar;
  __shared__ int flag;
  const int c = threadIdx.x % PC, t = threadIdx.x / PC;
  const int items = a.nb * (a.live_groups ? a.n_live_groups : a.ny / COLS);
  auto load = [&](int item) {
    int b;
    const int x = item_column<COLS>(a, item, b);
    mbar_expect_tx(&bar, N * PC * 16);
#pragma unroll
    for (int q = 0; q < N / BOX; ++q)
      tile_g2s(tile + q * BOX * PC, &tmap, x * col_words<V>(), b * a.nx + q * BOX, &bar);
  };
  auto sync = [] { __syncthreads(); };
  auto xat = [&](int s) { return xb + (s + (s >> SHIFT)) * PC + c; };
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
    if ((int)blockIdx.x < items) load(blockIdx.x);
  }
  // tables that every item reads, in shared memory: the tile and exchange
  // buffers leave too little L1 to keep them (0.748 -> 0.695 ms at 1024^2)
  constexpr bool TW_S = wide_tw_fits<V, N>(), PX_S = !SLOTS && wide_px_fits<V, N>();
  if constexpr (TW_S)
    for (int k = threadIdx.x; k < wide_tw<V, N>(); k += kWideThreads)
      tw_s[k] = static_cast<const C*>(a.tw)[k];
  if constexpr (PX_S)
    for (int k = threadIdx.x; k < N; k += kWideThreads) px_s[k] = static_cast<const C*>(a.px)[k];
  __syncthreads();
  const SharedTable<C> tw{TW_S ? tw_s : static_cast<const C*>(a.tw)};
  const Real inv_s = (Real)a.inv_s;
  uint32_t parity = 0;
  for (int item = blockIdx.x; item < items; item += gridDim.x, parity ^= 1) {
    int b;
    const int j = item_column<COLS>(a, item, b) + EC * c;
    const ColTables tab = col_tables<LAST, SLOTS>(a, b);
    ColumnEdge<V> edge;  // before the tile wait, so that its loads overlap it
    if (!tab.idle) edge.load(tab.lo, tab.hi, tab.py, j);
    if (!cta_wait(&bar, parity, &flag)) {
      if (threadIdx.x == 0) {
        atomicExch(err, 1);
        mbar_wait_bounded(&bar, parity);  // the copy may still be landing
      }
      return;
    }
    auto refill = [&] {  // the tile has been read by all
      if (threadIdx.x == 0 && item + (int)gridDim.x < items) {
        fence_proxy_async();
        load(item + gridDim.x);
      }
    };
    if (tab.idle) {
      __syncthreads();
      refill();
      continue;
    }
    V v[E];
#pragma unroll
    for (int m = 0; m < E; ++m) get_cols(tile + (t + T * m) * PC + c, v[m]);
    // the barrier of the tile wait has ended the exchange buffer's last use
    fft_lines_split<Sh, false, false, true>(v, t, tw, xat, sync, NoHook{}, refill);
    const C* px = static_cast<const C*>(tab.px);
    propagate<Sh>(v, t, [&](int i) { return PX_S ? px_s[i] : __ldg(px + i); }, edge, inv_s);
    if (!tab.stop_in_k)
      fft_lines_split<Sh, true, true, false>(v, t, tw, xat, sync, sync, NoHook{});
    Mem* out = reinterpret_cast<Mem*>(static_cast<C*>(a.psi) + (int64_t)b * a.batch_stride + j);
    const int64_t rs = a.ny / EC;
#pragma unroll
    for (int m = 0; m < E; ++m) put_cols(out + (t + T * m) * rs, v[m]);
  }
}

template <int N> constexpr bool wide() { return N >= 1024; }
template <class V, int N> constexpr int tile_cols() {
  if constexpr (wide<N>()) return wide_elems<N>() * elem_cols<V>();
  else return kRingElems * elem_cols<V>();
}

template <class V, int N, bool LAST, bool SLOTS>
cudaError_t col_launch(const PassArgs& a, const CUtensorMap& map, int* err, cudaStream_t s) {
  static PerDevice configured;
  const int items = a.nb * (a.live_groups ? a.n_live_groups : a.ny / tile_cols<V, N>());
  if (items <= 0) return cudaSuccess;
  if constexpr (wide<N>()) {
    auto k = col_wide_kernel<V, N, LAST, SLOTS>;
    constexpr int smem = wide_smem<V, N>();
    cudaError_t e = smem_limit_once((const void*)k, smem, configured);
    if (e != cudaSuccess) return e;
    k<<<items < sm_count() ? items : sm_count(), kWideThreads, smem, s>>>(a, map, err);
  } else {
    auto k = col_ring_kernel<V, N, LAST, SLOTS>;
    cudaError_t e = smem_limit_once((const void*)k, ring_smem<V, N>(), configured);
    if (e != cudaSuccess) return e;
    const int resident = ring_ctas<V, N>() * sm_count();
    k<<<items < resident ? items : resident, ring_group<N>() * ring_groups<V, N>(), ring_smem<V, N>(), s>>>(
        a, map, err);
  }
  return cudaGetLastError();
}

}  // namespace

#define MSF_COL_LENGTHS(X) X(64) X(128) X(256) X(512) X(1024) X(2048) X(4096)

}  // namespace msf
