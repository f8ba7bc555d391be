// The FP32 column slice pass (COL_SLICE, COL_SLICE_LAST, COL_SLOTS): DFT_x,
// / s, band limit, propagator, iDFT_x, two adjacent columns per thread
// (fft_pair.cuh).
//
// What bounds it: a column tile is rows of COLS x 8 bytes, and the memory
// system serves about 50 to 65 G requests/s of at most one 128-byte line
// each, whatever part of the line they carry.  An in-place copy of a 1024^2
// batch runs at 2.6-2.9 TB/s with 64-byte rows, 4.9 with 128-byte and 6.0 with
// 256-byte ones (direct loads and stores; TMA tiles of the same width move no
// faster).  So tiles are 128 bytes wide wherever a tile of that width fits an
// SM, and the two kernels differ in how they keep loads in flight beside it:
//
//  * up to 512 points, col_ring_kernel: three 16-column buffers and two groups
//    of threads that work on different tiles out of step; a tile is transformed
//    in place and leaves by TMA, the third buffer is in flight meanwhile.
//    512^2, 256 probes: 0.171 ms against 0.217 ms for one 16-column tile of
//    one column per thread behind CTA barriers (4.2 against 3.3 TB/s).  256
//    points: 0.045 ms, against 0.049 ms for the long-column kernel, which also
//    loses at 512 (0.189 ms).
//  * from 1024 points, col_wide_kernel: the tile (128 KB) leaves no room for a
//    second one, so it is read into registers, refilled by TMA at once, and
//    the transforms exchange half a tile (real parts, then imaginary parts)
//    at a time through a 64 KB buffer.  1024^2, 256 probes: 0.695 ms against
//    0.876 ms for two 8-column buffers (64-byte rows); 2048^2, 64 probes,
//    8 columns: 0.845 against 1.246 ms with 4; 4096^2, 16 probes, 4 columns:
//    1.15 ms against 4.3 ms for one column per CTA.  Left: the stores of a
//    tile leave in one burst behind its last stage, which the next tile's
//    first loads wait for.
//
// Every wait is bounded: if a phase does not complete within kSpinLimit polls
// the waiting group records an error in *err and leaves its loop; copies still
// in flight are waited for (bounded again) before the CTA ends.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <cmath>

#include "async_copy.cuh"
#include "fft_pair.cuh"
#include "kernels.h"

namespace msf {

namespace {

// Product of a column pair's elements with the propagator and the band limit:
// v[m] <- P_x P_y v[m] / s inside the limit (i < lo or i >= hi), else 0.
// PY: py / s of the two columns; px(i): the x propagator.
template <class Sh, class Px>
__device__ __forceinline__ void propagate_pair(Pair (&v)[Sh::E], int t, Px&& px, float4 py,
                                               float inv_s, int2 lo, int2 hi) {
  constexpr int E = Sh::E, T = Sh::T;
  const float2 pr = make_float2(py.x * inv_s, py.z * inv_s);
  const float2 pi = make_float2(py.y * inv_s, py.w * inv_s);
  sfor<0, E>([&](auto mI) {
    constexpr int m = decltype(mI)::value;
    if constexpr (dead_slot<E>(m)) {
      v[m] = Pair{f2(0.f), f2(0.f)};
    } else {
      const int i = t + T * m;
      const float2 p = px(i);
      const float2 qr = f2fma(f2(p.x), pr, f2mul(f2(-p.y), pi));
      const float2 qi = f2fma(f2(p.x), pi, f2mul(f2(p.y), pr));
      Pair r{f2fma(qr, v[m].re, f2mul(f2neg(qi), v[m].im)),
             f2fma(qr, v[m].im, f2mul(qi, v[m].re))};
      if (!(i < lo.x || i >= hi.x)) r.re.x = r.im.x = 0.f;
      if (!(i < lo.y || i >= hi.y)) r.re.y = r.im.y = 0.f;
      v[m] = r;
    }
  });
}

// What a probe brings to its column pass: the launch's tables, or (SLOTS) its
// slot's.
struct ColTables {
  const int32_t *lo, *hi;
  const float2 *px, *py;
  bool idle, stop_in_k;
};
template <bool LAST, bool SLOTS>
__device__ __forceinline__ ColTables col_tables(const PassArgs& a, int b) {
  if constexpr (SLOTS) {
    const SlotPass& s = a.slots[b];
    return ColTables{s.mask_lo, s.mask_hi, static_cast<const float2*>(s.px),
                     static_cast<const float2*>(s.py), s.op == SLOT_IDLE, s.last != 0};
  } else {
    return ColTables{a.mask_lo, a.mask_hi, static_cast<const float2*>(a.px),
                     static_cast<const float2*>(a.py), false, LAST};
  }
}

// Item -> first column (of the live column groups, when given) and probe.
template <int COLS>
__device__ __forceinline__ int item_column(const PassArgs& a, int item, int& b) {
  const int gi = item / a.nb;
  b = item - gi * a.nb;
  return (a.live_groups ? __ldg(a.live_groups + gi) : gi) * COLS;
}

// --------------------------------------------------- up to 512 points ------
constexpr int kRingCols = 16, kRingGroups = 2, kRingBufs = 3;
template <int N> __host__ __device__ constexpr int ring_group() {  // threads of a tile
  return kRingCols / 2 * PairShape<N>::T;
}
// 32 values of two columns take 255 registers a thread (256 threads an SM),
// 16 take 128 (512 threads)
template <int N> __host__ __device__ constexpr int ring_ctas() {
  return (PairShape<N>::E >= 32 ? 256 : 512) / (ring_group<N>() * kRingGroups);
}
template <int N> __host__ __device__ constexpr int ring_smem() {
  return kRingBufs * N * kRingCols * 8 + 1024;  // buffers start on 1024 bytes
}

template <int N, bool LAST, bool SLOTS>
__global__ void __launch_bounds__(ring_group<N>() * kRingGroups, ring_ctas<N>())
col_ring_kernel(const PassArgs a, const __grid_constant__ CUtensorMap tmap, int* err) {
  using Sh = PairShape<N>;
  constexpr int E = Sh::E, T = Sh::T, COLS = kRingCols, PC = COLS / 2;
  constexpr int G = kRingGroups, GT = ring_group<N>(), NBUF = kRingBufs;
  constexpr int BOX = N < 256 ? N : 256, BUF = N * COLS * 8;
  static_assert(T <= 32, "a column pair's threads share a warp");
  static_assert(NBUF > G, "a buffer is reloaded by its group's next item");
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* bufs = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  __shared__ uint64_t bars[NBUF];
  __shared__ int issued[NBUF];
  __shared__ int flags[G];
  const int g = threadIdx.x / GT, tg = threadIdx.x % GT;
  const int c = tg / T, t = tg % T;  // column pair of the tile, thread of the pair
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
      tile_g2s(dst + q * BOX * COLS * 8, &tmap, x, b * a.nx + q * BOX, &bars[k % NBUF]);
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
  auto pair_sync = [] { __syncwarp(); };
  if (threadIdx.x == 0) {
    for (int q = 0; q < NBUF; ++q) {
      mbar_init(&bars[q], 1);
      issued[q] = 0;
    }
    mbar_fence_init();
    for (int k = 0; k < NBUF && k < count; ++k) load(k);
  }
  __syncthreads();
  const GlobalTable tw{static_cast<const float2*>(a.tw)};
  const float inv_s = (float)a.inv_s;
  int reload = -1;  // item to load once the store of the last one has been read out
  for (int k = g; k < count; k += G) {
    const int w = k % NBUF;
    unsigned char* buf = bufs + w * BUF;
    int b;
    const int j0 = item_column<COLS>(a, blockIdx.x + k * gridDim.x, b), j = j0 + 2 * c;
    const ColTables tab = col_tables<LAST, SLOTS>(a, b);
    if (tg == 0) flags[g] = landed(k) ? 1 : 0;
    bar_sync(1 + g, GT);
    if (!flags[g]) {
      if (tg == 0) atomicExch(err, 1);
      break;
    }
    mbar_wait_bounded(&bars[w], (k / NBUF) & 1);  // every thread observes the phase
    // chunk c of row r in the tile as TMA's 128-byte swizzle lays it out
    auto at = [&](int r) { return reinterpret_cast<float4*>(buf) + r * PC + (c ^ (r & 7)); };
    Pair v[E];
    if (!tab.idle) {
#pragma unroll
      for (int m = 0; m < E; ++m) {
        const float4 x = *at(t + T * m);
        v[m] = Pair{make_float2(x.x, x.z), make_float2(x.y, x.w)};
      }
    }
    if (tg == 0 && reload >= 0) {
      bulk_wait_read();
      load(reload);
      reload = -1;
    }
    if (!tab.idle) {
      pair_sync();
      fft_pair<Sh, false, false, true>(v, t, tw, at, pair_sync);
      const int2 lo = __ldg(reinterpret_cast<const int2*>(tab.lo + j));
      const int2 hi = __ldg(reinterpret_cast<const int2*>(tab.hi + j));
      const float4 py = __ldg(reinterpret_cast<const float4*>(tab.py + j));
      propagate_pair<Sh>(v, t, [&](int i) { return __ldg(tab.px + i); }, py, inv_s, lo, hi);
      pair_sync();  // the transform's exchange has been read by all
      if (!tab.stop_in_k) fft_pair<Sh, true, true, false>(v, t, tw, at, pair_sync, pair_sync);
#pragma unroll
      for (int m = 0; m < E; ++m)
        *at(t + T * m) = make_float4(v[m].re.x, v[m].im.x, v[m].re.y, v[m].im.y);
      fence_proxy_async();
    }
    bar_sync(1 + g, GT);
    if (tg == 0) {
      if (!tab.idle) {
#pragma unroll
        for (int q = 0; q < N / BOX; ++q)
          tile_s2g(&tmap, j0, b * a.nx + q * BOX, buf + q * BOX * COLS * 8);
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
template <int N> __host__ __device__ constexpr int wide_cols() { return 16384 / N; }
constexpr int kWideThreads = 256;  // 8192 column pair elements, 32 a thread
// exchange slots: one of padding every R0, so that the stride-R0 writes of
// neighbouring threads fall on different banks
template <int N> __host__ __device__ constexpr int wide_slots() {
  return N + N / PairShape<N>::radix(0);
}
template <int N> __host__ __device__ constexpr int wide_tw() {  // twiddles of the length
  return PairShape<N>::tw_off(PairShape<N>::S);
}
// the slice's x propagator fits in shared memory too
template <int N> __host__ __device__ constexpr bool wide_px() { return N <= 2048; }
template <int N> __host__ __device__ constexpr int wide_smem() {
  return N * wide_cols<N>() * 8 + wide_slots<N>() * wide_cols<N>() / 2 * 8 + wide_tw<N>() * 8 +
         (wide_px<N>() ? N * 8 : 0);
}

template <int N, bool LAST, bool SLOTS>
__global__ void __launch_bounds__(kWideThreads, 1)
col_wide_kernel(const PassArgs a, const __grid_constant__ CUtensorMap tmap, int* err) {
  using Sh = PairShape<N>;
  constexpr int E = Sh::E, T = Sh::T, COLS = wide_cols<N>(), PC = COLS / 2;
  constexpr int BOX = 256, SHIFT = ilog2(Sh::radix(0));
  static_assert(PC * T == kWideThreads);
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  float4* tile = reinterpret_cast<float4*>(smem_raw);
  float2* xb = reinterpret_cast<float2*>(smem_raw + N * COLS * 8);
  float2* tw_s = xb + wide_slots<N>() * PC;
  float2* px_s = tw_s + wide_tw<N>();
  __shared__ uint64_t bar;
  __shared__ int flag;
  const int c = threadIdx.x % PC, t = threadIdx.x / PC;
  const int items = a.nb * (a.live_groups ? a.n_live_groups : a.ny / COLS);
  auto load = [&](int item) {
    int b;
    const int x = item_column<COLS>(a, item, b);
    mbar_expect_tx(&bar, N * COLS * 8);
#pragma unroll
    for (int q = 0; q < N / BOX; ++q)
      tile_g2s(tile + q * BOX * PC, &tmap, x, b * a.nx + q * BOX, &bar);
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
  for (int k = threadIdx.x; k < wide_tw<N>(); k += kWideThreads)
    tw_s[k] = static_cast<const float2*>(a.tw)[k];
  if constexpr (!SLOTS && wide_px<N>())
    for (int k = threadIdx.x; k < N; k += kWideThreads)
      px_s[k] = static_cast<const float2*>(a.px)[k];
  __syncthreads();
  const SharedTable tw{tw_s}, px_t{px_s};
  const float inv_s = (float)a.inv_s;
  uint32_t parity = 0;
  for (int item = blockIdx.x; item < items; item += gridDim.x, parity ^= 1) {
    int b;
    const int j = item_column<COLS>(a, item, b) + 2 * c;
    const ColTables tab = col_tables<LAST, SLOTS>(a, b);
    int2 lo{}, hi{};
    float4 py{};
    if (!tab.idle) {  // before the tile wait, so that they overlap it
      lo = __ldg(reinterpret_cast<const int2*>(tab.lo + j));
      hi = __ldg(reinterpret_cast<const int2*>(tab.hi + j));
      py = __ldg(reinterpret_cast<const float4*>(tab.py + j));
    }
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
    Pair v[E];
#pragma unroll
    for (int m = 0; m < E; ++m) {
      const float4 x = tile[(t + T * m) * PC + c];
      v[m] = Pair{make_float2(x.x, x.z), make_float2(x.y, x.w)};
    }
    // the barrier of the tile wait has ended the exchange buffer's last use
    fft_pair_split<Sh, false, false, true>(v, t, tw, xat, sync, NoHook{}, refill);
    propagate_pair<Sh>(
        v, t,
        [&](int i) { return !SLOTS && wide_px<N>() ? px_t(i) : __ldg(tab.px + i); }, py, inv_s,
        lo, hi);
    if (!tab.stop_in_k) fft_pair_split<Sh, true, true, false>(v, t, tw, xat, sync, sync, NoHook{});
    float4* out = reinterpret_cast<float4*>(static_cast<float2*>(a.psi) +
                                            (int64_t)b * a.batch_stride + j);
    const int64_t rs = a.ny / 2;
#pragma unroll
    for (int m = 0; m < E; ++m)
      out[(t + T * m) * rs] = make_float4(v[m].re.x, v[m].im.x, v[m].re.y, v[m].im.y);
  }
}

template <int N> constexpr bool wide() { return N >= 1024; }
template <int N> constexpr int tile_cols() {
  if constexpr (wide<N>()) return wide_cols<N>();
  else return kRingCols;
}

template <int N, bool LAST, bool SLOTS>
cudaError_t col_launch(const PassArgs& a, const CUtensorMap& map, int* err, cudaStream_t s) {
  static PerDevice configured;
  const int items = a.nb * (a.live_groups ? a.n_live_groups : a.ny / tile_cols<N>());
  if (items <= 0) return cudaSuccess;
  if constexpr (wide<N>()) {
    auto k = col_wide_kernel<N, LAST, SLOTS>;
    cudaError_t e = smem_limit_once((const void*)k, wide_smem<N>(), configured);
    if (e != cudaSuccess) return e;
    k<<<items < sm_count() ? items : sm_count(), kWideThreads, wide_smem<N>(), s>>>(a, map, err);
  } else {
    auto k = col_ring_kernel<N, LAST, SLOTS>;
    cudaError_t e = smem_limit_once((const void*)k, ring_smem<N>(), configured);
    if (e != cudaSuccess) return e;
    const int resident = ring_ctas<N>() * sm_count();
    k<<<items < resident ? items : resident, ring_group<N>() * kRingGroups, ring_smem<N>(), s>>>(
        a, map, err);
  }
  return cudaGetLastError();
}

template <int N>
cudaError_t col_ops(const PassArgs& a, bool last, const CUtensorMap& map, int* err,
                    cudaStream_t s) {
  if (a.slots) return col_launch<N, false, true>(a, map, err, s);
  return last ? col_launch<N, true, false>(a, map, err, s)
              : col_launch<N, false, false>(a, map, err, s);
}

template <int N>
void pair_twiddles(std::vector<float>& out) {
  using Sh = PairShape<N>;
  const double two_pi = 6.283185307179586476925286766559;
  for (int s = 1; s < Sh::S; ++s)
    for (int B = 2; B <= Sh::radix(s); B *= 2)
      for (int m = 0; m < (B > 4 ? B / 4 : 1); ++m)
        for (int k = 0; k < Sh::ns(s); ++k) {
          const double x = two_pi * (k + (double)Sh::ns(s) * m) / ((double)Sh::ns(s) * B);
          out.push_back((float)std::cos(x));
          out.push_back((float)-std::sin(x));
        }
}

}  // namespace

#define MSF_PAIR_LENGTHS(X) X(64) X(128) X(256) X(512) X(1024) X(2048) X(4096)

cudaError_t launch_col_pair(const PassArgs& a, bool last, const void* tensor_map, int* err,
                            cudaStream_t s) {
  const CUtensorMap& m = *static_cast<const CUtensorMap*>(tensor_map);
  switch (a.nx) {
#define MSF_CASE(N) case N: return col_ops<N>(a, last, m, err, s);
    MSF_PAIR_LENGTHS(MSF_CASE)
#undef MSF_CASE
  }
  return cudaErrorInvalidValue;
}

int col_pair_tile(int nx) {
  switch (nx) {
#define MSF_CASE(N) case N: return tile_cols<N>();
    MSF_PAIR_LENGTHS(MSF_CASE)
#undef MSF_CASE
  }
  return 0;
}

void fill_pair_twiddles(int n, std::vector<float>& out) {
  out.clear();
  switch (n) {
#define MSF_CASE(N) case N: pair_twiddles<N>(out); break;
    MSF_PAIR_LENGTHS(MSF_CASE)
#undef MSF_CASE
  }
}

// Tensor map over a batch of FP32 planes [nb*nx rows][ny columns] of 8-byte
// complex values: box {tile columns, min(256, nx)} rows, no multicast.  Up to
// 512 points swizzled over the 128-byte tile row, so that eight consecutive
// rows of a column pair lie in eight different 16-byte bank groups; the wide
// tiles are read a whole row at a time and need no swizzle.
cudaError_t encode_pair_map(void* psi, int nb, int nx, int ny, void* map_out) {
  // looked up once per process (a thread-safe static: lanes of the request
  // loop encode maps from their worker thread)
  static const PFN_cuTensorMapEncodeTiled_v12000 encode = [] {
    cudaDriverEntryPointQueryResult q;
    void* fn = nullptr;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
    return (e == cudaSuccess && q == cudaDriverEntryPointSuccess)
               ? reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn)
               : nullptr;
  }();
  if (!encode) return cudaErrorNotSupported;
  const int cols = col_pair_tile(nx);
  if (!cols) return cudaErrorInvalidValue;
  cuuint64_t dims[2] = {(cuuint64_t)ny, (cuuint64_t)nx * (cuuint64_t)nb};
  cuuint64_t strides[1] = {(cuuint64_t)ny * 8};
  cuuint32_t box[2] = {(cuuint32_t)cols, (cuuint32_t)(nx < 256 ? nx : 256)};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = encode(static_cast<CUtensorMap*>(map_out), CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, psi,
                      dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                      nx < 1024 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

}  // namespace msf
