// Four-step sphere planes and pencils (split_fft.cuh).
//
// Axis of n = r1 r2 points, x index r2 a + j (a < r1, j < r2), output index
// k + r1 q (k < r1, q < r2):
//   first   per j: r1-point transform over a, times w_n^(j k), stored at slot
//           r2 k + j, the slots it was read from;
//   second  per k: r2-point transform over the slots r2 k + j; slot r2 k + q
//           then holds output k + r1 q.
// One thread runs one short transform; threads of a warp run over lines, so
// twiddles are the same for the warp and shared-memory accesses contiguous.
// The radices are run-time values dispatched to register transforms
// (fft_line_registers), so one kernel serves every length.
//
// Measured (one B200) against radix stages in shared memory, FP64: 97 columns on
// 81^3 (41 rows) planes in 412 -> 226 us, pencils 729 -> 378 us, planes out 691
// -> 239 us; 128 bands on 72^3 density planes (rows and columns) 534 -> 206 us,
// pencils 1005 -> 330 us. The latency of 16 warps an SM (12 in the density's
// pencils) binds all four: of one capture each at 32 columns, issue slots 33-41 %,
// FP64 pipe 21-34 %, shared memory 16-34 %, DRAM 11-21 %, and an issued
// instruction waits 1-3 cycles each on barriers, its operands and loads. In FP32
// the register-resident line kernels of local_hamiltonian.cu stay ahead where they
// exist (70 points, 160 columns: pencils 188 us there, 295 us here; planes 119 and
// 137 us, 137 and 161 us here); lengths without them take these (100 points, 32
// columns: 1185 -> 563 us a pair).
#include <type_traits>

#include "split_fft.cuh"

namespace sdft_b200 {

namespace {

constexpr int kThreads = 256;
constexpr int kDensityThreads = 128;
constexpr int kMaxRadix = 16;

// exp(-2 pi i m / r) of every radix r <= kMaxRadix at [r (r - 1) / 2 + m]: a
// kernel parameter, so each is a constant operand.
template <typename T>
struct RadixTables {
  Cx<T> w[kMaxRadix * (kMaxRadix + 1) / 2];
};

template <typename T>
const RadixTables<T>& radix_tables() {
  static const RadixTables<T> tables = [] {
    RadixTables<T> t;
    for (int r = 1; r <= kMaxRadix; ++r) host_twiddles<T>(r, t.w + r * (r - 1) / 2);
    return t;
  }();
  return tables;
}

// Points a thread reads at once in the sphere's scatter and gather.
constexpr int kPointBatch = 4;

// Resident CTAs per SM the plane kernels are compiled for: in FP32 with the
// short radices four (64 registers), so that a small grid's planes (18 rows x
// 32 columns at 35 points) run in one wave, two otherwise.
template <typename T, int MAXR>
constexpr int plane_blocks() {
  return sizeof(T) == 4 && MAXR <= 10 ? 4 : 2;
}

constexpr bool is_radix(int r) { return (r >= 1 && r <= 10) || r == 12 || r == 14 || r == 15 || r == 16; }

template <typename T, bool INV, int R>
__device__ __forceinline__ void short_transform(Cx<T> (&v)[R], const RadixTables<T>& t) {
  if constexpr (R > 1) fft_line_registers<T, INV, R>(v, t.w + R * (R - 1) / 2);
}

// f(integral_constant<int, r>) for r <= MAXR: kernels compiled for radices up
// to 10 need half the registers of those for 16.
template <int MAXR, typename F>
__device__ __forceinline__ void with_radix(int r, F&& f) {
#define SDFT_RADIX(R)                                                  \
  case R:                                                              \
    if constexpr (R <= MAXR) f(std::integral_constant<int, R>{});      \
    break;
  switch (r) {
    SDFT_RADIX(1)
    SDFT_RADIX(2)
    SDFT_RADIX(3)
    SDFT_RADIX(4)
    SDFT_RADIX(5)
    SDFT_RADIX(6)
    SDFT_RADIX(7)
    SDFT_RADIX(8)
    SDFT_RADIX(9)
    SDFT_RADIX(10)
    SDFT_RADIX(12)
    SDFT_RADIX(14)
    SDFT_RADIX(15)
    SDFT_RADIX(16)
  }
#undef SDFT_RADIX
}

template <typename T, bool INV>
__device__ __forceinline__ Cx<T> twiddled(Cx<T> v, const Cx<T>* tw, int index) {
  return index ? cmul(v, twiddle<T, INV>(tw, index)) : v;
}

// Both steps in place on `count` contiguous lines (stride apart, odd so that
// neighbouring lines fall into different banks); output k + r1 q is left at
// slot r2 k + q. Ends with a CTA barrier.
template <typename T, bool INV, int MAXR>
__device__ __forceinline__ void transform_rows(Cx<T>* rows, int count, int stride, const SplitAxis& a, const Cx<T>* tw,
                                               const RadixTables<T>& tables) {
  with_radix<MAXR>(a.r1, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
    for (int item = threadIdx.x; item < a.r2 * count; item += kThreads) {
      const int j = item / count;
      Cx<T>* line = rows + (item - j * count) * stride + j;
      Cx<T> v[R];
#pragma unroll
      for (int i = 0; i < R; ++i) v[i] = line[a.r2 * i];
      short_transform<T, INV, R>(v, tables);
#pragma unroll
      for (int k = 0; k < R; ++k) line[a.r2 * k] = twiddled<T, INV>(v[k], tw, j * k);
    }
  });
  __syncthreads();
  with_radix<MAXR>(a.r2, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
    for (int item = threadIdx.x; item < a.r1 * count; item += kThreads) {
      const int k = item / count;
      Cx<T>* line = rows + (item - k * count) * stride + R * k;
      Cx<T> v[R];
#pragma unroll
      for (int i = 0; i < R; ++i) v[i] = line[i];
      short_transform<T, INV, R>(v, tables);
#pragma unroll
      for (int q = 0; q < R; ++q) line[q] = v[q];
    }
  });
  __syncthreads();
}

template <typename T>
struct PlaneArgs {
  SplitAxis a1, a2;
  int stride;  // shared-memory row stride, odd
  int slots, krows, tile;
  const int* point_offset;
  const int* point_g;
  const int* point_compact;
  const int* krow;
  const Cx<T>* tw1;
  const Cx<T>* tw2;
};

// Shared memory: both axes' twiddles, the active rows, one tile of columns,
// and the compact position of every i1.
template <typename T>
struct PlaneSmem {
  Cx<T>*tw1, *tw2, *rows, *tile;
  int* kpos;
  __device__ PlaneSmem(unsigned char* raw, const PlaneArgs<T>& a)
      : tw1(reinterpret_cast<Cx<T>*>(raw)),
        tw2(tw1 + a.a1.n),
        rows(tw2 + a.a2.n),
        tile(rows + a.krows * a.stride),
        kpos(reinterpret_cast<int*>(tile + a.a1.n * a.tile)) {}
};
template <typename T>
std::size_t plane_smem(const PlaneArgs<T>& a) {
  return sizeof(Cx<T>) * (a.a1.n + a.a2.n + static_cast<std::size_t>(a.krows) * a.stride +
                          static_cast<std::size_t>(a.a1.n) * a.tile) +
         sizeof(int) * a.a1.n;
}

template <typename T, int MAXR>
__global__ void __launch_bounds__(kThreads, plane_blocks<T, MAXR>()) split_planes_in_kernel(PlaneArgs<T> a,
                                                                      const __grid_constant__ RadixTables<T> tables,
                                                                      const Cx<double>* __restrict__ x, long long ldx,
                                                                      const int* __restrict__ band,
                                                                      Cx<T>* __restrict__ slab,
                                                                      unsigned int* __restrict__ flags) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const PlaneSmem<T> s(smem_raw, a);
  const int slot = blockIdx.x, c = blockIdx.y, tid = threadIdx.x;
  const int n1 = a.a1.n, n2 = a.a2.n;
  for (int i = tid; i < n1; i += kThreads) {
    s.tw1[i] = a.tw1[i];
    s.kpos[i] = -1;
  }
  for (int i = tid; i < n2; i += kThreads) s.tw2[i] = a.tw2[i];
  for (int i = tid; i < a.krows * a.stride; i += kThreads) s.rows[i] = Cx<T>{0, 0};
  __syncthreads();
  for (int i = tid; i < a.krows; i += kThreads) s.kpos[a.krow[i]] = i;
  const Cx<double>* column = x + (band ? static_cast<long long>(band[c]) : c) * ldx;
  bool finite = true;
  const int points_end = a.point_offset[slot + 1];
  for (int first = a.point_offset[slot] + tid; first < points_end; first += kPointBatch * kThreads) {
    int at[kPointBatch], g[kPointBatch];
    Cx<double> v[kPointBatch];
#pragma unroll
    for (int u = 0; u < kPointBatch; ++u) {
      const int p = first + u * kThreads;
      at[u] = p < points_end ? a.point_compact[p] : -1;
      g[u] = p < points_end ? a.point_g[p] : 0;
    }
#pragma unroll
    for (int u = 0; u < kPointBatch; ++u)
      if (at[u] >= 0) v[u] = column[g[u]];
#pragma unroll
    for (int u = 0; u < kPointBatch; ++u)
      if (at[u] >= 0) {
        if (flags) finite = finite && isfinite(v[u].re) && isfinite(v[u].im);
        const int k = at[u] / n2;
        s.rows[k * a.stride + (at[u] - k * n2)] = cconvert<T>(v[u]);
      }
  }
  if (!finite) atomicOr(flags, 1u);
  __syncthreads();
  transform_rows<T, true, MAXR>(s.rows, a.krows, a.stride, a.a2, s.tw2, tables);
  // i1 on tiles of columns, straight to the slab.
  const int j = tid / a.tile, t = tid - j * a.tile;
  Cx<T>* out = slab + (static_cast<long long>(c) * a.slots + slot) * n1 * n2;
  for (int c0 = 0; c0 < n2; c0 += a.tile) {
    const int i2 = c0 + t;
    const bool live = i2 < n2;
    if (live && j < a.a1.r2) {
      const int q = i2 / a.a2.r1, at = a.a2.r2 * (i2 - q * a.a2.r1) + q;  // the row's slot of i2
      with_radix<MAXR>(a.a1.r1, [&](auto radix) {
        constexpr int R = decltype(radix)::value;
        Cx<T> v[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const int k = s.kpos[a.a1.r2 * i + j];
          v[i] = k >= 0 ? s.rows[k * a.stride + at] : Cx<T>{0, 0};
        }
        short_transform<T, true, R>(v, tables);
#pragma unroll
        for (int k = 0; k < R; ++k)
          s.tile[(a.a1.r2 * k + j) * a.tile + t] = twiddled<T, true>(v[k], s.tw1, j * k);
      });
    }
    __syncthreads();
    if (live && j < a.a1.r1)
      with_radix<MAXR>(a.a1.r2, [&](auto radix) {
        constexpr int R = decltype(radix)::value;
        Cx<T> v[R];
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = s.tile[(R * j + i) * a.tile + t];
        short_transform<T, true, R>(v, tables);
#pragma unroll
        for (int q = 0; q < R; ++q) out[static_cast<long long>(j + a.a1.r1 * q) * n2 + i2] = v[q];
      });
    __syncthreads();
  }
}

template <typename T, int MAXR>
__global__ void __launch_bounds__(kThreads, plane_blocks<T, MAXR>()) split_planes_out_kernel(PlaneArgs<T> a,
                                                                       const __grid_constant__ RadixTables<T> tables,
                                                                       const Cx<T>* __restrict__ slab,
                                                                       const Cx<double>* __restrict__ x, long long ldx,
                                                                       const double* __restrict__ kinetic,
                                                                       double count, Cx<double>* __restrict__ y,
                                                                       long long ldy) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const PlaneSmem<T> s(smem_raw, a);
  const int slot = blockIdx.x, c = blockIdx.y, tid = threadIdx.x;
  const int n1 = a.a1.n, n2 = a.a2.n;
  for (int i = tid; i < n1; i += kThreads) {
    s.tw1[i] = a.tw1[i];
    s.kpos[i] = -1;
  }
  for (int i = tid; i < n2; i += kThreads) s.tw2[i] = a.tw2[i];
  __syncthreads();
  for (int i = tid; i < a.krows; i += kThreads) s.kpos[a.krow[i]] = i;
  __syncthreads();
  const int j = tid / a.tile, t = tid - j * a.tile;
  const Cx<T>* in = slab + (static_cast<long long>(c) * a.slots + slot) * n1 * n2;
  for (int c0 = 0; c0 < n2; c0 += a.tile) {
    const int i2 = c0 + t;
    const bool live = i2 < n2;
    if (live && j < a.a1.r2)
      with_radix<MAXR>(a.a1.r1, [&](auto radix) {
        constexpr int R = decltype(radix)::value;
        Cx<T> v[R];
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = in[static_cast<long long>(a.a1.r2 * i + j) * n2 + i2];
        short_transform<T, false, R>(v, tables);
#pragma unroll
        for (int k = 0; k < R; ++k)
          s.tile[(a.a1.r2 * k + j) * a.tile + t] = twiddled<T, false>(v[k], s.tw1, j * k);
      });
    __syncthreads();
    if (live && j < a.a1.r1)
      with_radix<MAXR>(a.a1.r2, [&](auto radix) {
        constexpr int R = decltype(radix)::value;
        Cx<T> v[R];
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = s.tile[(R * j + i) * a.tile + t];
        short_transform<T, false, R>(v, tables);
#pragma unroll
        for (int q = 0; q < R; ++q) {
          const int k = s.kpos[j + a.a1.r1 * q];
          if (k >= 0) s.rows[k * a.stride + i2] = v[q];
        }
      });
    __syncthreads();
  }
  transform_rows<T, false, MAXR>(s.rows, a.krows, a.stride, a.a2, s.tw2, tables);
  const Cx<double>* xc = x + static_cast<long long>(c) * ldx;
  Cx<double>* yc = y + static_cast<long long>(c) * ldy;
  const int points_end = a.point_offset[slot + 1];
  for (int first = a.point_offset[slot] + tid; first < points_end; first += kPointBatch * kThreads) {
    int at[kPointBatch], g[kPointBatch];
    Cx<double> in_g[kPointBatch];
    double kin[kPointBatch];
#pragma unroll
    for (int u = 0; u < kPointBatch; ++u) {
      const int p = first + u * kThreads;
      at[u] = p < points_end ? a.point_compact[p] : -1;
      g[u] = p < points_end ? a.point_g[p] : 0;
    }
#pragma unroll
    for (int u = 0; u < kPointBatch; ++u)
      if (at[u] >= 0) {
        in_g[u] = xc[g[u]];
        kin[u] = kinetic[g[u]];
      }
#pragma unroll
    for (int u = 0; u < kPointBatch; ++u)
      if (at[u] >= 0) {
        const int k = at[u] / n2, i2 = at[u] - k * n2, q = i2 / a.a2.r1;
        const Cx<double> v = cconvert<double>(s.rows[k * a.stride + a.a2.r2 * (i2 - q * a.a2.r1) + q]);
        yc[g[u]] = Cx<double>{kin[u] * in_g[u].re + v.re / count, kin[u] * in_g[u].im + v.im / count};
      }
  }
}

template <typename T>
struct PencilArgs {
  SplitAxis a;
  int slots, tile;
  long long n12;
  const int* slot_row;
  const Cx<T>* tw;
};
template <typename T>
std::size_t pencil_smem(const PencilArgs<T>& a, int buffers) {
  return sizeof(Cx<T>) * (a.a.n + static_cast<std::size_t>(buffers) * a.a.n * a.tile) + sizeof(int) * a.a.n;
}

// The second backward step leaves thread (k, line) the rows k + r1 q, which is
// what the forward transform's first step (r2 points over q) wants: V(r) and
// both short transforms stay in registers.
template <typename T, int MAXR>
__global__ void __launch_bounds__(kThreads, 2) split_pencils_kernel(PencilArgs<T> a,
                                                                    const __grid_constant__ RadixTables<T> tables,
                                                                    const T* __restrict__ potential,
                                                                    Cx<T>* __restrict__ slab) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cx<T>* tw = reinterpret_cast<Cx<T>*>(smem_raw);
  Cx<T>* tile = tw + a.a.n;
  int* slot = reinterpret_cast<int*>(tile + a.a.n * a.tile);
  const int tid = threadIdx.x, j = tid / a.tile, t = tid - j * a.tile, r1 = a.a.r1, r2 = a.a.r2;
  for (int i = tid; i < a.a.n; i += kThreads) {
    tw[i] = a.tw[i];
    slot[i] = -1;
  }
  __syncthreads();
  for (int i = tid; i < a.slots; i += kThreads) slot[a.slot_row[i]] = i;
  __syncthreads();
  const long long kl = static_cast<long long>(blockIdx.x) * a.tile + t;
  const bool live = kl < a.n12;
  Cx<T>* base = slab + static_cast<long long>(blockIdx.y) * a.slots * a.n12 + kl;
  if (live && j < r2)
    with_radix<MAXR>(r1, [&](auto radix) {
      constexpr int R = decltype(radix)::value;
      Cx<T> v[R];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const int s = slot[r2 * i + j];
        v[i] = s >= 0 ? base[s * a.n12] : Cx<T>{0, 0};
      }
      short_transform<T, true, R>(v, tables);
#pragma unroll
      for (int k = 0; k < R; ++k) tile[(r2 * k + j) * a.tile + t] = twiddled<T, true>(v[k], tw, j * k);
    });
  __syncthreads();
  if (live && j < r1)
    with_radix<MAXR>(r2, [&](auto radix) {
      constexpr int R = decltype(radix)::value;
      Cx<T> v[R];
      T pot[R];
#pragma unroll
      for (int q = 0; q < R; ++q) pot[q] = potential[(j + r1 * q) * a.n12 + kl];
#pragma unroll
      for (int i = 0; i < R; ++i) v[i] = tile[(R * j + i) * a.tile + t];
      short_transform<T, true, R>(v, tables);
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = cscale(v[q], pot[q]);
      short_transform<T, false, R>(v, tables);
#pragma unroll
      for (int q = 0; q < R; ++q) tile[(R * j + q) * a.tile + t] = twiddled<T, false>(v[q], tw, j * q);
    });
  __syncthreads();
  if (live && j < r2)
    with_radix<MAXR>(r1, [&](auto radix) {
      constexpr int R = decltype(radix)::value;
      Cx<T> v[R];
#pragma unroll
      for (int k = 0; k < R; ++k) v[k] = tile[(r2 * k + j) * a.tile + t];
      short_transform<T, false, R>(v, tables);
#pragma unroll
      for (int p = 0; p < R; ++p) {
        const int s = slot[j + r2 * p];
        if (s >= 0) base[s * a.n12] = v[p];
      }
    });
}

// Thread (k, line) keeps the density of rows k + r1 q of its line in registers
// over all bands (128 threads a CTA: a 72^3 grid's 371 tiles spread over the SMs); the next band's entries are loaded before the barrier of the
// current one, and two exchange tiles leave one barrier per band.
template <int MAXR>
__global__ void __launch_bounds__(kDensityThreads, 4) split_density_kernel(
    PencilArgs<double> a, const __grid_constant__ RadixTables<double> tables, const Cx<double>* __restrict__ planes,
    const double* __restrict__ weight, int bands, bool accumulate, Cx<double>* __restrict__ grid) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cx<double>* tw = reinterpret_cast<Cx<double>*>(smem_raw);
  Cx<double>* tiles = tw + a.a.n;
  int* slot = reinterpret_cast<int*>(tiles + 2 * a.a.n * a.tile);
  const int tid = threadIdx.x, j = tid / a.tile, t = tid - j * a.tile, r1 = a.a.r1, r2 = a.a.r2;
  for (int i = tid; i < a.a.n; i += kDensityThreads) {
    tw[i] = a.tw[i];
    slot[i] = -1;
  }
  __syncthreads();
  for (int i = tid; i < a.slots; i += kDensityThreads) slot[a.slot_row[i]] = i;
  __syncthreads();
  const long long kl = static_cast<long long>(blockIdx.x) * a.tile + t;
  const bool first = kl < a.n12 && j < r2, second = kl < a.n12 && j < r1;
  const long long band_stride = a.slots * a.n12;
  Cx<double> v[MAXR];
  double sum[MAXR];
  auto load = [&](int b) {
    if (!first || b >= bands) return;
    const Cx<double>* base = planes + b * band_stride + kl;
#pragma unroll
    for (int i = 0; i < MAXR; ++i) {
      const int s = i < r1 ? slot[r2 * i + j] : -1;
      v[i] = s >= 0 ? base[s * a.n12] : Cx<double>{0, 0};
    }
  };
#pragma unroll
  for (int q = 0; q < MAXR; ++q)
    sum[q] = accumulate && second && q < r2 ? grid[(j + r1 * q) * a.n12 + kl].re : 0.0;
  load(0);
  for (int b = 0; b < bands; ++b) {
    Cx<double>* tile = tiles + (b & 1) * a.a.n * a.tile;
    if (first)
      with_radix<MAXR>(r1, [&](auto radix) {
        constexpr int R = decltype(radix)::value;
        Cx<double> u[R];
#pragma unroll
        for (int i = 0; i < R; ++i) u[i] = v[i];
        short_transform<double, true, R>(u, tables);
#pragma unroll
        for (int k = 0; k < R; ++k) tile[(r2 * k + j) * a.tile + t] = twiddled<double, true>(u[k], tw, j * k);
      });
    load(b + 1);
    __syncthreads();
    if (second) {
      const double w = weight[b];
      with_radix<MAXR>(r2, [&](auto radix) {
        constexpr int R = decltype(radix)::value;
        Cx<double> u[R];
#pragma unroll
        for (int i = 0; i < R; ++i) u[i] = tile[(R * j + i) * a.tile + t];
        short_transform<double, true, R>(u, tables);
#pragma unroll
        for (int q = 0; q < R; ++q) sum[q] += w * (u[q].re * u[q].re + u[q].im * u[q].im);
      });
    }
  }
  if (second) {
#pragma unroll
    for (int q = 0; q < MAXR; ++q)
      if (q < r2) grid[(j + r1 * q) * a.n12 + kl] = Cx<double>{sum[q], 0.0};
  }
}

template <typename T>
PlaneArgs<T> plane_args(const SpherePlan& plan, const Cx<T>* tw1, const Cx<T>* tw2) {
  PlaneArgs<T> a{};
  a.a1 = split_axis(plan.n[1]);
  a.a2 = split_axis(plan.n[2]);
  a.stride = plan.n[2] | 1;
  a.slots = plan.slots;
  a.krows = plan.krows;
  if (a.a1.r2) {
    // Equal tiles of at most one short transform per thread.
    const int widest = kThreads / a.a1.r2;
    const int tiles = static_cast<int>(ceil_div(plan.n[2], widest));
    a.tile = static_cast<int>(ceil_div(plan.n[2], tiles));
  }
  a.point_offset = plan.point_offset;
  a.point_g = plan.point_g;
  a.point_compact = plan.point_compact;
  a.krow = plan.krow;
  a.tw1 = tw1;
  a.tw2 = tw2;
  return a;
}

template <typename T>
PencilArgs<T> pencil_args(const SpherePlan& plan, const Cx<T>* tw0, int threads) {
  PencilArgs<T> a{};
  a.a = split_axis(plan.n[0]);
  a.slots = plan.slots;
  a.tile = a.a.r2 ? threads / a.a.r2 : 0;
  a.n12 = static_cast<long long>(plan.n[1]) * plan.n[2];
  a.slot_row = plan.slot_row;
  a.tw = tw0;
  return a;
}

}  // namespace

SplitAxis split_axis(int n) {
  SplitAxis best;
  for (int r1 = 1; r1 * r1 <= n; ++r1)
    if (n % r1 == 0 && is_radix(r1) && n / r1 <= kMaxRadix && is_radix(n / r1)) best = SplitAxis{n, r1, n / r1};
  return best;
}

template <typename T>
bool split_pencils(const SpherePlan& plan, int columns, const T* potential, Cx<T>* slab, const Cx<T>* tw0,
                   cudaStream_t stream) {
  const PencilArgs<T> a = pencil_args(plan, tw0, kThreads);
  if (!a.a.r2) return false;
  const std::size_t smem = pencil_smem(a, 1);
  const dim3 grid(static_cast<unsigned>(ceil_div(static_cast<std::size_t>(a.n12), a.tile)), columns);
  auto go = [&](auto kernel) {
    allow_dynamic_smem(kernel, smem);
    kernel<<<grid, kThreads, smem, stream>>>(a, radix_tables<T>(), potential, slab);
    SDFT_LAUNCH("split_pencils_kernel");
  };
  if (a.a.r2 <= 10) go(split_pencils_kernel<T, 10>);
  else go(split_pencils_kernel<T, 16>);
  return true;
}

template <typename T>
bool split_planes_fit(const SpherePlan& plan) {
  const PlaneArgs<T> a = plane_args<T>(plan, nullptr, nullptr);
  return a.a1.r2 && a.a2.r2 && plane_smem(a) <= kMaxDynamicSmem;
}

template <typename T>
bool split_planes_in(const SpherePlan& plan, const Cx<double>* x, long long ldx, const int* band, int columns,
                     Cx<T>* slab, const Cx<T>* tw1, const Cx<T>* tw2, unsigned int* flags, cudaStream_t stream) {
  const PlaneArgs<T> a = plane_args(plan, tw1, tw2);
  if (!split_planes_fit<T>(plan)) return false;
  auto go = [&](auto kernel) {
    allow_dynamic_smem(kernel, plane_smem(a));
    kernel<<<dim3(a.slots, columns), kThreads, plane_smem(a), stream>>>(a, radix_tables<T>(), x, ldx, band, slab,
                                                                         flags);
    SDFT_LAUNCH("split_planes_in_kernel");
  };
  if (a.a1.r2 <= 10 && a.a2.r2 <= 10) go(split_planes_in_kernel<T, 10>);
  else go(split_planes_in_kernel<T, 16>);
  return true;
}

template <typename T>
bool split_planes_out(const SpherePlan& plan, const Cx<T>* slab, const Cx<double>* x, long long ldx,
                      const double* kinetic, double count, Cx<double>* y, long long ldy, int columns,
                      const Cx<T>* tw1, const Cx<T>* tw2, cudaStream_t stream) {
  const PlaneArgs<T> a = plane_args(plan, tw1, tw2);
  if (!split_planes_fit<T>(plan)) return false;
  auto go = [&](auto kernel) {
    allow_dynamic_smem(kernel, plane_smem(a));
    kernel<<<dim3(a.slots, columns), kThreads, plane_smem(a), stream>>>(a, radix_tables<T>(), slab, x, ldx, kinetic,
                                                                        count, y, ldy);
    SDFT_LAUNCH("split_planes_out_kernel");
  };
  if (a.a1.r2 <= 10 && a.a2.r2 <= 10) go(split_planes_out_kernel<T, 10>);
  else go(split_planes_out_kernel<T, 16>);
  return true;
}

bool split_density_pencils(const SpherePlan& plan, const Cx<double>* planes, const double* weight, int bands,
                           bool accumulate, Cx<double>* grid, const Cx<double>* tw0, cudaStream_t stream) {
  const PencilArgs<double> a = pencil_args(plan, tw0, kDensityThreads);
  if (!a.a.r2) return false;
  const std::size_t smem = pencil_smem(a, 2);
  const unsigned blocks = static_cast<unsigned>(ceil_div(static_cast<std::size_t>(a.n12), a.tile));
  auto go = [&](auto kernel) {
    allow_dynamic_smem(kernel, smem);
    kernel<<<blocks, kDensityThreads, smem, stream>>>(a, radix_tables<double>(), planes, weight, bands, accumulate,
                                                      grid);
    SDFT_LAUNCH("split_density_kernel");
  };
  if (a.a.r2 <= 10) go(split_density_kernel<10>);
  else go(split_density_kernel<16>);
  return true;
}

#define SDFT_SPLIT(T)                                                                                               \
  template bool split_pencils<T>(const SpherePlan&, int, const T*, Cx<T>*, const Cx<T>*, cudaStream_t);             \
  template bool split_planes_fit<T>(const SpherePlan&);                                                             \
  template bool split_planes_in<T>(const SpherePlan&, const Cx<double>*, long long, const int*, int, Cx<T>*,        \
                                   const Cx<T>*, const Cx<T>*, unsigned int*, cudaStream_t);                        \
  template bool split_planes_out<T>(const SpherePlan&, const Cx<T>*, const Cx<double>*, long long, const double*,   \
                                    double, Cx<double>*, long long, int, const Cx<T>*, const Cx<T>*, cudaStream_t);
SDFT_SPLIT(float)
SDFT_SPLIT(double)
#undef SDFT_SPLIT

}  // namespace sdft_b200
