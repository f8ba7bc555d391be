// The FP64 row passes of the slice loop (fft_lines.cuh, one line per T threads):
//   ROW_SLICE         iDFT_y, transmission multiply, DFT_y
//   ROW_SLICE_FIRST   place the shifted probe, transmission multiply, DFT_y
//   ROW_VACUUM        iDFT_y, the wave rounded to FP32 into a table, DFT_y
//   ROW_VACUUM_FIRST  the scaled probe, rounded into the table, DFT_y
//
// What bounds it: at 1024 points the FP64 pipe needs 3.3 us a probe and the live
// columns' bytes 3.4; the rest is load latency at eight warps an SM.  32 elements
// a thread (255 registers, two radix-32 stages and one exchange) still hide it
// better than twelve warps of 16 (three stages): 9.3 against 11.8 us a probe, and
// the transmission row prefetched into L1 during the inverse transform takes
// that to 6.4.  One 16-element line of three stages with a separate twiddle
// product took 12.2.  512 points: 2.57 -> 1.69 us (64 probes), 256: 0.44 -> 0.40,
// 128: 0.122 -> 0.106 (256 probes; the product form of the twiddles, which rounds
// as little as before, fft_lines.cuh: fused they took 0.34 and 0.098).
// From 2048 points 32 elements spill (59 us a probe) and 16 are the better (63.7
// -> 39.8 us; 4096: 362 -> 181).
#include <algorithm>

#include "fft_lines.cuh"
#include "kernels.h"

namespace msf {

namespace {

// lines of a CTA: 64 threads, or one line's
template <int N> constexpr int row64_lines() {
  return RowShape<N>::T >= 64 ? 1 : 64 / RowShape<N>::T;
}
// CTAs an SM the registers must allow: 256 threads at 32 elements and at 4096
// points (255 registers), 384 at 16, 512 at 8
template <int N> constexpr int row64_ctas() {
  constexpr int threads = row64_lines<N>() * RowShape<N>::T;
  constexpr int want = RowShape<N>::E >= 32 || N == 4096 ? 256 : RowShape<N>::E == 16 ? 384 : 512;
  return want / threads > 0 ? want / threads : 1;
}
template <int N> constexpr int row64_stride() {  // exchange slots, one of padding every R0
  return N + N / RowShape<N>::radix(0);
}
template <int N> constexpr int row64_smem() { return row64_lines<N>() * row64_stride<N>() * 16; }

template <int N, int LINES, int CTAS, int OP>
__global__ void __launch_bounds__(LINES * RowShape<N>::T, CTAS) row64_kernel(const PassArgs a) {
  using Sh = RowShape<N>;
  constexpr int E = Sh::E, T = Sh::T, SHIFT = ilog2(Sh::radix(0));
  constexpr int STRIDE = N + N / Sh::radix(0);
  constexpr bool FIRST = OP == ROW_SLICE_FIRST || OP == ROW_VACUUM_FIRST;
  extern __shared__ __align__(16) double2 exchange[];
  const int line = threadIdx.x / T, t = threadIdx.x % T;
  const int b = blockIdx.x, i = blockIdx.y * LINES + line;
  double2* sm = exchange + line * STRIDE;
  double2* row = static_cast<double2*>(a.psi) + (int64_t)b * a.batch_stride + (int64_t)i * N;
  auto at = [sm](int s) { return sm + s + (s >> SHIFT); };
  auto sync = [] {
    if constexpr (T <= 32) __syncwarp();
    else __syncthreads();
  };
  const GlobalTable<double2> tw{static_cast<const double2*>(a.tw)};
  const uint32_t dead = a.row_dead_bits ? __ldg(a.row_dead_bits + t) : 0u;
  double2 v[E];
  if constexpr (FIRST) {
    const double fs = a.first_scale;
    const int sx = OP == ROW_SLICE_FIRST ? a.shifts[2 * b] : 0;
    const int sy = OP == ROW_SLICE_FIRST ? a.shifts[2 * b + 1] : 0;
    const int ix = (i < sx) ? i + a.nx - sx : i - sx;
    const double2* prow = static_cast<const double2*>(a.probe) + (int64_t)ix * N;
#pragma unroll
    for (int m = 0; m < E; ++m) {
      const int y = t + T * m;
      v[m] = cscale(__ldg(prow + ((y < sy) ? y + N - sy : y - sy)), fs);
    }
  } else {
    // columns removed by the band limit are zero (and were not stored)
    const uint32_t skip = (a.row_dead_io & 1) ? dead : 0u;
    sfor<0, E>([&](auto mI) {
      constexpr int m = decltype(mI)::value;
      v[m] = vzero<double2>();
      if constexpr (!dead_slot<E>(m))
        if (!((skip >> m) & 1u)) v[m] = row[t + T * m];
    });
  }
  if constexpr (OP == ROW_SLICE) {
    const char* trow = static_cast<const char*>(a.trans) + (int64_t)i * N * 16;
    for (int l = t; l < N * 16 / 128; l += T)
      asm volatile("prefetch.global.L1 [%0];" ::"l"(trow + 128 * l));
  }
  if constexpr (!FIRST) {
    fft_lines<Sh, true, true, false>(v, t, tw, at, sync);
    sync();  // the exchange has been read by all
  }
  if constexpr (OP == ROW_SLICE || OP == ROW_SLICE_FIRST) {
    // the reference's in-place update order (adfstem.cpp:1929-1949): the new
    // real part feeds the imaginary part
    const double2* trow = static_cast<const double2*>(a.trans) + (int64_t)i * N;
    const double is = a.inv_s;
#pragma unroll
    for (int m = 0; m < E; ++m) {
      if (m % 4 == 0) load_fence();
      const double2 tv = __ldg(trow + t + T * m);
      const double re = (tv.x * v[m].x - tv.y * v[m].y) * is;
      const double im = (tv.x * v[m].y + tv.y * re) * is;
      v[m] = make_double2(re, im);
    }
  } else {
    float2* out = reinterpret_cast<float2*>(a.out32) + (int64_t)i * N;
#pragma unroll
    for (int m = 0; m < E; ++m) out[t + T * m] = make_float2((float)v[m].x, (float)v[m].y);
  }
  fft_lines<Sh, false, false, true>(v, t, tw, at, sync);
  const bool fill = !(a.row_dead_bits && (a.row_dead_io & 2));  // removed columns: store zeros
  sfor<0, E>([&](auto mI) {
    constexpr int m = decltype(mI)::value;
    if (!dead_slot<E>(m) && !((dead >> m) & 1u)) row[t + T * m] = v[m];
    else if (fill) row[t + T * m] = vzero<double2>();
  });
}

template <int N, int OP> cudaError_t row64_launch(const PassArgs& a, cudaStream_t s) {
  constexpr int L = row64_lines<N>();
  static PerDevice configured;
  auto k = row64_kernel<N, L, row64_ctas<N>(), OP>;
  if (cudaError_t e = smem_limit_once((const void*)k, row64_smem<N>(), configured);
      e != cudaSuccess)
    return e;
  if (a.nx % L != 0) return cudaErrorInvalidValue;
  k<<<dim3(a.nb, a.nx / L), L * RowShape<N>::T, row64_smem<N>(), s>>>(a);
  return cudaGetLastError();
}

template <int N> cudaError_t row64_ops(RowOp op, const PassArgs& a, cudaStream_t s) {
  switch (op) {
    case ROW_SLICE: return row64_launch<N, ROW_SLICE>(a, s);
    case ROW_SLICE_FIRST: return row64_launch<N, ROW_SLICE_FIRST>(a, s);
    case ROW_VACUUM: return row64_launch<N, ROW_VACUUM>(a, s);
    case ROW_VACUUM_FIRST: return row64_launch<N, ROW_VACUUM_FIRST>(a, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

#define MSF_ROW_LENGTHS(X) X(64) X(128) X(256) X(512) X(1024) X(2048) X(4096)

cudaError_t launch_row64(RowOp op, const PassArgs& a, cudaStream_t s) {
  switch (a.ny) {
#define MSF_CASE(N) case N: return row64_ops<N>(op, a, s);
    MSF_ROW_LENGTHS(MSF_CASE)
#undef MSF_CASE
  }
  return cudaErrorInvalidValue;
}

int row64_threads(int ny) {
  switch (ny) {
#define MSF_CASE(N) case N: return RowShape<N>::T;
    MSF_ROW_LENGTHS(MSF_CASE)
#undef MSF_CASE
  }
  return 0;
}

void fill_row64_twiddles(int n, std::vector<double>& out) {
  out.clear();
  switch (n) {
#define MSF_CASE(N) case N: line_twiddles<RowShape<N>>(out); break;
    MSF_ROW_LENGTHS(MSF_CASE)
#undef MSF_CASE
  }
}

}  // namespace msf
