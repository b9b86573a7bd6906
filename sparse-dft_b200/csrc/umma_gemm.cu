// tcgen05 / TMEM / TMA BF16 GEMM for the mixed-precision complex products.
//
// One CTA per SM walks over 128 x BN FP32 tiles of Ahat Bhat^T, each over a
// range of 64-wide K blocks (split-K across tiles). Warp 0 lane 0 streams A and
// B tiles with TMA (128-byte swizzle, no multicast) into a STAGES-deep
// shared-memory ring; warp 1 lane 0 issues tcgen05.mma (M=128, N=BN, K=16 per
// instruction) into one of two tensor-memory accumulators and releases ring
// slots with tcgen05.commit; eight more warps drain the other accumulator with
// tcgen05.ld (warp w may read TMEM lanes 32 (w % 4) and up; two warps share
// each quarter's columns) and write either FP32 split-K partials or the final
// FP64 complex result, while the next tile's products run. Every mbarrier wait
// is bounded; a wait that runs out sets a device error word and the CTA winds
// down (the host turns it into an error).
// Tall products were bound by their FP64 results (and the values they add to),
// not by the tensor cores: with one tile per CTA, four warps reading a chunk's
// prior values only once they came to it and nothing running meanwhile, the
// joint back-projection of 160 columns at 23847 x 512 took 197 us; with the
// epilogue's loads a chunk ahead and beside the next tile's products 113 us
// (245 MB of results and priors, 38 us at copy rate; tensor pipe 55 % active, DRAM
// 32 %). B x of the same block, bound by shared-memory fills, stays at 42-44 us
// (tensor pipe 49 %, DRAM 35 % in a cold launch of 58 us).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <mutex>
#include <string>

#include <map>
#include <tuple>
#include <vector>
#include "umma_gemm.cuh"

namespace sdft_b200 {

namespace {

constexpr int BM = 128, BK = 64;
constexpr int kEpilogueWarps = 8;  // warps 2..9
constexpr int kThreads = 32 * (2 + kEpilogueWarps);
constexpr unsigned long long kWaitLimitNs = 2000000000ULL;  // 2 s per wait

__device__ unsigned int g_umma_error = 0;

__device__ __forceinline__ std::uint32_t smem_u32(const void* p) {
  return static_cast<std::uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(std::uint64_t* bar, std::uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(std::uint64_t* bar, std::uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(std::uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(std::uint64_t* bar, std::uint32_t parity) {
  std::uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: false (and the error word set) when the phase does not
// complete within the limit or another thread already gave up.
__device__ bool mbar_wait(std::uint64_t* bar, std::uint32_t parity) {
  const unsigned long long start = globaltimer();
  for (std::uint32_t spin = 0;; ++spin) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((spin & 255u) == 255u) {
      if (*reinterpret_cast<volatile unsigned int*>(&g_umma_error) != 0u) return false;
      if (globaltimer() - start > kWaitLimitNs) {
        atomicExch(&g_umma_error, 1u);
        return false;
      }
    }
  }
}
// Wait of the wind-down after an error, for work already in flight: the same
// limit, whatever the error word says.
__device__ void mbar_drain(std::uint64_t* bar, std::uint32_t parity) {
  const unsigned long long start = globaltimer();
  while (!mbar_try_wait(bar, parity) && globaltimer() - start <= kWaitLimitNs) {
  }
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int c0, int c1, std::uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<std::uint64_t>(map)), "r"(c0), "r"(c1), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void umma_bf16(std::uint32_t d_tmem, std::uint64_t adesc, std::uint64_t bdesc,
                                          std::uint32_t idesc, std::uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(
          d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void umma_commit(std::uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// K-major, 128-byte swizzle shared-memory matrix descriptor (rows of 128 B,
// 8-row atoms 1024 B apart): start>>4, LBO 1, SBO 64 (x16 B), version 1, SWIZZLE_128B.
__device__ __forceinline__ std::uint64_t smem_desc(std::uint32_t addr) {
  return (static_cast<std::uint64_t>((addr >> 4) & 0x3FFFu)) | (1ULL << 16) | (64ULL << 32) | (1ULL << 46) |
         (2ULL << 61);
}

template <int BN>
__host__ __device__ constexpr std::uint32_t instr_desc() {
  // D=F32 (bits 4-5 = 1), A=B=BF16 (bits 7-9 = 1, 10-12 = 1), K-major both, N>>3 at 17, M>>4 at 24.
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<std::uint32_t>(BN >> 3) << 17) |
         (static_cast<std::uint32_t>(BM >> 4) << 24);
}

template <int BN>
__host__ __device__ constexpr int stages() {
  return BN >= 256 ? 4 : 6;
}

// The tiles of a product: columns fastest, so that the CTAs sharing an A tile
// work on it together and all but the first read it from L2; then rows, then
// shares of K.
struct WorkTile {
  int row, column, split;
};
struct TileGrid {
  int columns, rows;
  long long count;
  __device__ WorkTile at(long long w) const {
    const long long strip = w / columns;
    return {static_cast<int>(strip % rows), static_cast<int>(w % columns), static_cast<int>(strip / rows)};
  }
};

struct EpilogueArgs {
  int m, n2;                   // rows, real columns (2 x complex columns)
  Cx<float>* partial;          // split-K output [split][n2/2][m] or null
  ProductOutput out[2];        // direct outputs (when partial is null)
  int second;                  // first complex column of out[1]
  double alpha;
  bool shared_terms;           // BF16x3 blocks: term 0 in elements 0-31, term 1 in 32-63
};

// PAIR: the product's columns go to two outputs.
template <int BN, bool PAIR>
__global__ void __launch_bounds__(kThreads, 1)
    umma_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                     int k_blocks_total, int k_blocks_per_split, TileGrid tiles, EpilogueArgs ep) {
  constexpr int S = stages<BN>();
  constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE = A_BYTES + B_BYTES;
  constexpr std::uint32_t TMEM_COLS = BN <= 128 ? 256 : 512;  // two accumulators
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<std::uintptr_t>(smem_raw) + 1023) & ~static_cast<std::uintptr_t>(1023));
  std::uint64_t* full = reinterpret_cast<std::uint64_t*>(smem + S * STAGE);
  std::uint64_t* empty = full + S;
  std::uint64_t* acc_full = empty + S;
  std::uint64_t* acc_empty = acc_full + 2;
  std::uint64_t* drained = acc_empty + 2;
  std::uint32_t* tmem_holder = reinterpret_cast<std::uint32_t*>(drained + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], kEpilogueWarps);
    }
    mbar_init(drained, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const std::uint32_t tmem = *tmem_holder;

  int issued = 0;
  if (warp == 0 && lane == 0) {
    // TMA producer
    for (long long w = blockIdx.x; w < tiles.count; w += gridDim.x) {
      const WorkTile t = tiles.at(w);
      const int kb0 = t.split * k_blocks_per_split, kb1 = min(k_blocks_total, kb0 + k_blocks_per_split);
      bool alive = true;
      for (int kb = kb0; kb < kb1 && alive; ++kb) {
        const int s = issued % S;
        alive = issued < S || mbar_wait(&empty[s], ((issued / S) - 1) & 1);
        if (!alive) break;
        mbar_arrive_expect_tx(&full[s], STAGE);
        tma_load_2d(smem + s * STAGE, &map_a, kb * BK, t.row * BM, &full[s]);
        tma_load_2d(smem + s * STAGE + A_BYTES, &map_b, kb * BK, t.column * BN, &full[s]);
        ++issued;
      }
      if (!alive) break;
    }
  } else if (warp == 1 && lane == 0) {
    // tcgen05.mma issuer
    constexpr std::uint32_t idesc = instr_desc<BN>();
    int i = 0, n = 0;
    for (long long w = blockIdx.x; w < tiles.count; w += gridDim.x, ++n) {
      const int kb0 = tiles.at(w).split * k_blocks_per_split, kb1 = min(k_blocks_total, kb0 + k_blocks_per_split);
      const std::uint32_t acc = tmem + (n & 1) * (TMEM_COLS / 2);
      bool alive = n < 2 || mbar_wait(&acc_empty[n & 1], ((n / 2) - 1) & 1);
      tc_fence_after();
      for (int kb = kb0; kb < kb1 && alive; ++kb, ++i) {
        const int s = i % S;
        alive = mbar_wait(&full[s], (i / S) & 1);
        if (!alive) break;
        tc_fence_after();
        const std::uint32_t a_addr = smem_u32(smem + s * STAGE), b_addr = a_addr + A_BYTES;
        if (ep.shared_terms) {
          // Products (0,0), (0,1), (1,0) of the block's terms, two K = 16 steps each (byte offsets in a 128-byte row).
#pragma unroll
          for (int kk = 0; kk < 6; ++kk)
            umma_bf16(acc, smem_desc(a_addr + (kk >= 4 ? 64 : 0) + (kk & 1) * 32),
                      smem_desc(b_addr + (kk == 2 || kk == 3 ? 64 : 0) + (kk & 1) * 32), idesc, kb != kb0 || kk != 0);
        } else {
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk)
            umma_bf16(acc, smem_desc(a_addr + kk * 32), smem_desc(b_addr + kk * 32), idesc, kb != kb0 || kk != 0);
        }
        umma_commit(&empty[s]);
      }
      if (!alive) break;
      umma_commit(&acc_full[n & 1]);
    }
  } else if (warp >= 2) {
    // Epilogue: this warp's quarter of the rows, every second 16-column chunk.
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const int n_complex_total = ep.n2 / 2;
    int n = 0;
    for (long long w = blockIdx.x; w < tiles.count; w += gridDim.x, ++n) {
      const WorkTile t = tiles.at(w);
      const int row = t.row * BM + quarter * 32 + lane, first = t.column * (BN / 2);
      const bool in_rows = row < ep.m;
      // A chunk's prior values (accumulating products) are requested one chunk
      // ahead, the first chunk's before the accumulator is complete.
      auto load_prior = [&](int c0, Cx<double>(&prior)[8]) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int j = first + c0 / 2 + q;
          const bool other = PAIR && j >= ep.second;
          const Cx<double>* from = other ? ep.out[1].prior : ep.out[0].prior;
          const long long at = other ? (j - ep.second) * ep.out[1].ldp : j * ep.out[0].ldp;
          prior[q] = !ep.partial && from && in_rows && c0 < BN && j < n_complex_total ? from[row + at]
                                                                                       : Cx<double>{0.0, 0.0};
        }
      };
      Cx<double> prior[8];
      load_prior(16 * half, prior);
      if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[n & 1], (n / 2) & 1))) break;
      tc_fence_after();
      const std::uint32_t acc = tmem + (n & 1) * (TMEM_COLS / 2) + (static_cast<std::uint32_t>(quarter * 32) << 16);
      for (int c0 = 16 * half; c0 < BN; c0 += 32) {
        std::uint32_t r[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(acc + static_cast<std::uint32_t>(c0)));
        Cx<double> next[8];
        load_prior(c0 + 32, next);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (c0 + 32 >= BN) {  // the accumulator is free once every warp has read its last chunk
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_empty[n & 1]);
        }
        if (in_rows) {
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int j = first + c0 / 2 + q;
            if (j >= n_complex_total) break;
            const float re = __uint_as_float(r[2 * q]), im = __uint_as_float(r[2 * q + 1]);
            if (ep.partial) {
              ep.partial[(static_cast<long long>(t.split) * n_complex_total + j) * ep.m + row] = Cx<float>{re, im};
            } else {
              const bool other = PAIR && j >= ep.second;
              Cx<double>* to = other ? ep.out[1].c : ep.out[0].c;
              const long long at = other ? (j - ep.second) * ep.out[1].ldc : j * ep.out[0].ldc;
              const double scale = other ? ep.out[1].prior_scale : ep.out[0].prior_scale;
              const double vr = ep.alpha * static_cast<double>(re), vi = ep.alpha * static_cast<double>(im);
              to[row + at] = Cx<double>{__dadd_rn(vr, __dmul_rn(scale, prior[q].re)),
                                        __dadd_rn(vi, __dmul_rn(scale, prior[q].im))};
            }
          }
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) prior[q] = next[q];
      }
    }
  }
  __syncwarp();
  // Wind-down: on the error path wait for the TMA copies and the products still in
  // flight (without an error the last epilogue has), then free TMEM.
  if (lane == 0 && warp < 2 && *reinterpret_cast<volatile unsigned int*>(&g_umma_error) != 0u) {
    if (warp == 0) {
      for (int i = max(0, issued - S); i < issued; ++i) mbar_drain(&full[i % S], (i / S) & 1);
    } else {
      umma_commit(drained);
      mbar_drain(drained, 0);
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
}

// alpha * sum_s partial[s] to its output: one thread per (row i = x, column j = y),
// the splits summed in order with two interleaved accumulators.
__global__ void reduce_splits_kernel(int m, int n, int splits, const Cx<float>* __restrict__ partial,
                                     ProductOutput out0, ProductOutput out1, int second, double alpha) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const long long total = static_cast<long long>(m) * n;
  for (int j = blockIdx.y; j < n; j += gridDim.y) {
    const Cx<float>* p = partial + static_cast<long long>(j) * m + i;
    double re0 = 0.0, im0 = 0.0, re1 = 0.0, im1 = 0.0;
    int s = 0;
    for (; s + 1 < splits; s += 2) {
      const Cx<float> a = p[s * total], b = p[(s + 1) * total];
      re0 += a.re;
      im0 += a.im;
      re1 += b.re;
      im1 += b.im;
    }
    if (s < splits) {
      const Cx<float> a = p[s * total];
      re0 += a.re;
      im0 += a.im;
    }
    double re = (re0 + re1) * alpha, im = (im0 + im1) * alpha;
    const ProductOutput& o = j >= second ? out1 : out0;
    const long long column = j >= second ? j - second : j;
    if (o.prior) {
      const Cx<double> v = o.prior[i + column * o.ldp];
      re = __dadd_rn(re, __dmul_rn(o.prior_scale, v.re));
      im = __dadd_rn(im, __dmul_rn(o.prior_scale, v.im));
    }
    o.c[i + column * o.ldc] = Cx<double>{re, im};
  }
}

// ---- packing (FP64 complex -> BF16 split terms) ---------------------------

// Split-term index of BF16x6 product p on the A and B side: (0,0) (0,1) (1,0)
// (0,2) (1,1) (2,0).
__host__ __device__ constexpr int term_a(int p) { return p == 2 || p == 4 ? 1 : p == 5 ? 2 : 0; }
__host__ __device__ constexpr int term_b(int p) { return p == 1 || p == 4 ? 1 : p == 3 ? 2 : 0; }

__device__ __forceinline__ void split3(double x, std::uint16_t t[3]) {
  const __nv_bfloat16 h0 = __double2bfloat16(x);
  const double r1 = x - static_cast<double>(__bfloat162float(h0));
  const __nv_bfloat16 h1 = __double2bfloat16(r1);
  const double r2 = r1 - static_cast<double>(__bfloat162float(h1));
  const __nv_bfloat16 h2 = __double2bfloat16(r2);
  t[0] = __bfloat16_as_ushort(h0);
  t[1] = __bfloat16_as_ushort(h1);
  t[2] = __bfloat16_as_ushort(h2);
}

__device__ __forceinline__ std::uint32_t pair(std::uint16_t lo, std::uint16_t hi) {
  return static_cast<std::uint32_t>(lo) | (static_cast<std::uint32_t>(hi) << 16);
}

// Writes the entries of complex k in an expanded row: terms of (x, y) as pairs.
// BF16x3 rows hold each of the two terms once, BF16x6 rows the six product terms.
template <int P, bool SIDE_B>
__device__ __forceinline__ void write_entry(std::uint16_t* row, long long k, double x, double y, std::uint32_t sign) {
  std::uint16_t u[3], v[3];
  split3(x, u);
  split3(y, v);
  if constexpr (P == 3) {
    auto* d = reinterpret_cast<std::uint32_t*>(row + (k / kSharedBlock) * 64 + (k % kSharedBlock) * 2);
    d[0] = pair(u[0], v[0]) ^ sign;
    d[kSharedBlock] = pair(u[1], v[1]) ^ sign;
  } else {
    auto* d = reinterpret_cast<uint2*>(row + k * 2 * P);  // 24 bytes an entry in 128-byte rows: 8-byte aligned
#pragma unroll
    for (int p = 0; p < P; p += 2) {
      const int t0 = SIDE_B ? term_b(p) : term_a(p), t1 = SIDE_B ? term_b(p + 1) : term_a(p + 1);
      d[p / 2] = make_uint2(pair(u[t0], v[t0]) ^ sign, pair(u[t1], v[t1]) ^ sign);
    }
  }
}
template <int P>
__device__ __forceinline__ void write_a(std::uint16_t* row, long long k, Cx<double> v) {
  write_entry<P, false>(row, k, v.re, v.im, 0u);
}

// Zeros the entries k..end of an expanded row of kexp elements, thread `first` of `count`.
template <int P>
__device__ __forceinline__ void zero_tail(std::uint16_t* row, int k, long long kexp, int first, int count) {
  if constexpr (P == 3) {
    for (long long q = k + first; q < kexp / 64 * kSharedBlock; q += count) {
      auto* d = reinterpret_cast<std::uint32_t*>(row + (q / kSharedBlock) * 64 + (q % kSharedBlock) * 2);
      d[0] = d[kSharedBlock] = 0u;
    }
  } else {
    for (long long q = 2LL * P * k + first; q < kexp; q += count) row[q] = 0;
  }
}

// One row i of A per blockIdx.y; threads stride over k.
template <int P, bool CONJ_T>
__global__ void pack_a_direct_kernel(const Cx<double>* __restrict__ src, long long lds, int rows, int k,
                                     std::uint16_t* __restrict__ out, long long ldo, long long kexp) {
  // CONJ_T: A[i,k] = conj(src[k + i*lds]) (k contiguous in the source).
  // Rows i = blockIdx.y, blockIdx.y + gridDim.y, ... (any row count).
  for (int i = blockIdx.y; i < rows; i += gridDim.y) {
    const Cx<double>* in = src + static_cast<long long>(i) * lds;
    std::uint16_t* row = out + static_cast<long long>(i) * ldo;
    for (int kk = blockIdx.x * blockDim.x + threadIdx.x; kk < k; kk += gridDim.x * blockDim.x) {
      Cx<double> v = in[kk];
      if (CONJ_T) v.im = -v.im;
      write_a<P>(row, kk, v);
    }
    zero_tail<P>(row, k, kexp, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
  }
}

// A[i,k] = src[i + k*lds] (rows contiguous): 32x32 shared-memory transpose.
// kexp > 0: the rows end there, and the last blocks zero what follows entry k.
template <int P>
__global__ void pack_a_transpose_kernel(const Cx<double>* __restrict__ src, long long lds, int rows, int k,
                                        std::uint16_t* __restrict__ out, long long ldo, long long out_k_offset,
                                        long long kexp) {
  __shared__ Cx<double> tile[32][33];
  const int i0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
  for (int r = ty; r < 32; r += 8) {
    const int i = i0 + tx, kk = k0 + r;
    tile[r][tx] = (i < rows && kk < k) ? src[i + static_cast<long long>(kk) * lds] : Cx<double>{0, 0};
  }
  __syncthreads();
  for (int r = ty; r < 32; r += 8) {
    const int i = i0 + r, kk = k0 + tx;
    if (i < rows && kk < k) write_a<P>(out + static_cast<long long>(i) * ldo, out_k_offset + kk, tile[tx][r]);
  }
  if (kexp > 0 && blockIdx.y == gridDim.y - 1)
    for (int r = ty; r < 32 && i0 + r < rows; r += 8)
      zero_tail<P>(out + static_cast<long long>(i0 + r) * ldo, k, kexp, tx, 32);
}

// Source columns j = blockIdx.y, blockIdx.y + gridDim.y, ... (two expanded
// rows each); threads stride over k.
template <int P>
__global__ void pack_b_kernel(const Cx<double>* __restrict__ src, long long ldb, int k, int n,
                              std::uint16_t* __restrict__ out, long long ldo, long long kexp) {
  for (int j = blockIdx.y; j < n; j += gridDim.y) {
    const Cx<double>* in = src + static_cast<long long>(j) * ldb;
    std::uint16_t* row0 = out + (2LL * j) * ldo;
    std::uint16_t* row1 = row0 + ldo;
    for (int kk = blockIdx.x * blockDim.x + threadIdx.x; kk < k; kk += gridDim.x * blockDim.x) {
      const Cx<double> v = in[kk];
      write_entry<P, true>(row0, kk, v.re, v.im, 0x80000000u);  // [Re, -Im] (sign flip is exact)
      write_entry<P, true>(row1, kk, v.im, v.re, 0u);           // [Im, Re]
    }
    zero_tail<P>(row0, k, kexp, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
    zero_tail<P>(row1, k, kexp, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
  }
}

// Largest gridDim.y; kernels that put rows or columns on y stride past it.
constexpr int kMaxGridY = 65535;

// Blocks along a row of `length` entries when `rows` rows run side by side:
// enough CTAs in total for ~16 per SM, at least one per row.
unsigned row_blocks(long long length, int rows) {
  const long long per_row = std::max<long long>(1, (148LL * 16 + rows - 1) / rows);
  return static_cast<unsigned>(std::max<long long>(1, std::min<long long>(per_row, (length + 255) / 256)));
}

// ---- tensor maps -----------------------------------------------------------

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult status;
    SDFT_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &status));
    if (status != cudaDriverEntryPointSuccess || !ptr) throw CudaError("cuTensorMapEncodeTiled is unavailable");
    fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
  });
  return fn;
}

CUtensorMap kmajor_map(const std::uint16_t* base, long long rows, long long kexp, long long ld, int box_rows) {
  if (reinterpret_cast<std::uintptr_t>(base) % 16 != 0 || (ld * 2) % 16 != 0)
    throw InvalidArgument("BF16 operand base and row stride must be 16-byte aligned");
  CUtensorMap map;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(kexp), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld * 2)};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(BK), static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t element_strides[2] = {1, 1};
  const CUresult r = encode_fn()(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<std::uint16_t*>(base), dims,
                                 strides, box, element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                 CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw CudaError("cuTensorMapEncodeTiled failed: " + std::to_string(static_cast<int>(r)));
  return map;
}

template <int BN>
void launch(const std::uint16_t* a, long long lda, const std::uint16_t* b, long long ldb, int m, int n2,
            long long kexp, const EpilogueArgs& ep_in, int splits, int k_blocks, int kpb, cudaStream_t stream) {
  constexpr int S = stages<BN>();
  const std::size_t smem = static_cast<std::size_t>(S) * (BM * BK * 2 + BN * BK * 2) + 1024 + 256;
  const auto kernel = ep_in.second < n2 / 2 && !ep_in.partial ? umma_gemm_kernel<BN, true> : umma_gemm_kernel<BN, false>;
  allow_dynamic_smem(kernel, smem);
  const CUtensorMap map_a = kmajor_map(a, m, kexp, lda, BM);
  const CUtensorMap map_b = kmajor_map(b, n2, kexp, ldb, BN);
  if (ceil_div(m, BM) > 65535) throw InvalidArgument("tensor-core GEMM has more than 65535 row tiles");
  TileGrid tiles{static_cast<int>(ceil_div(n2, BN)), static_cast<int>(ceil_div(m, BM)), 0};
  tiles.count = static_cast<long long>(tiles.columns) * tiles.rows * splits;
  const unsigned grid = static_cast<unsigned>(std::min<long long>(tiles.count, kSmCount));
  kernel<<<grid, kThreads, smem, stream>>>(map_a, map_b, k_blocks, kpb, tiles, ep_in);
  SDFT_LAUNCH("umma_gemm_kernel");
}

}  // namespace

bool umma_available() {
  int device = 0, major = 0;
  if (cudaGetDevice(&device) != cudaSuccess) return false;
  if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device) != cudaSuccess) return false;
  return major == 10;
}

void pack_a(Op aop, const Cx<double>* src, long long lds, int rows, int k, Split split, std::uint16_t* out,
            long long ldo, cudaStream_t stream) {
  const long long kexp = expanded_k(k, split);
  if (aop == Op::C) {
    const dim3 grid(row_blocks(k, rows),
                    static_cast<unsigned>(std::min(rows, kMaxGridY)));
    if (split == Split::BF16x3)
      pack_a_direct_kernel<3, true><<<grid, 256, 0, stream>>>(src, lds, rows, k, out, ldo, kexp);
    else
      pack_a_direct_kernel<6, true><<<grid, 256, 0, stream>>>(src, lds, rows, k, out, ldo, kexp);
    SDFT_LAUNCH("pack_a_direct_kernel");
    return;
  }
  const dim3 grid(static_cast<unsigned>(ceil_div(rows, 32)), static_cast<unsigned>(ceil_div(k, 32)));
  if (split == Split::BF16x3)
    pack_a_transpose_kernel<3><<<grid, dim3(32, 8), 0, stream>>>(src, lds, rows, k, out, ldo, 0, kexp);
  else
    pack_a_transpose_kernel<6><<<grid, dim3(32, 8), 0, stream>>>(src, lds, rows, k, out, ldo, 0, kexp);
  SDFT_LAUNCH("pack_a_transpose_kernel");
}

void pack_a_columns(const Cx<double>* src, long long lds, int rows, int first, int count, Split split,
                    std::uint16_t* out, long long ldo, cudaStream_t stream) {
  if (count <= 0) return;
  const dim3 grid(static_cast<unsigned>(ceil_div(rows, 32)), static_cast<unsigned>(ceil_div(count, 32)));
  const Cx<double>* s = src + static_cast<long long>(first) * lds;
  if (split == Split::BF16x3)
    pack_a_transpose_kernel<3><<<grid, dim3(32, 8), 0, stream>>>(s, lds, rows, count, out, ldo, first, 0);
  else
    pack_a_transpose_kernel<6><<<grid, dim3(32, 8), 0, stream>>>(s, lds, rows, count, out, ldo, first, 0);
  SDFT_LAUNCH("pack_a_transpose_kernel");
}

void pack_b(const Cx<double>* src, long long ldb, int k, int n, Split split, std::uint16_t* out, long long ldo,
            cudaStream_t stream) {
  const long long kexp = expanded_k(k, split);
  const dim3 grid(row_blocks(k, n),
                  static_cast<unsigned>(std::min(n, kMaxGridY)));
  if (split == Split::BF16x3) pack_b_kernel<3><<<grid, 256, 0, stream>>>(src, ldb, k, n, out, ldo, kexp);
  else pack_b_kernel<6><<<grid, 256, 0, stream>>>(src, ldb, k, n, out, ldo, kexp);
  SDFT_LAUNCH("pack_b_kernel");
}

namespace {

// Column tile width of the cost model: the one of 128 / 160 / 256 that pads
// the 2n real columns least (the larger on ties).
int model_width(int n2) {
  int bn = 256;
  long long padded = ceil_div(n2, 256) * 256LL;
  for (int w : {160, 128}) {
    const long long p = ceil_div(n2, w) * static_cast<long long>(w);
    if (p < padded) {
      padded = p;
      bn = w;
    }
  }
  return bn;
}

int max_splits_for(int k_blocks) { return static_cast<int>(std::min<long long>(128, std::max(1, k_blocks / 8))); }

// Split-K count of the cost model for width bn: one CTA per SM is resident
// (the ring takes ~200 KB), so the time goes as waves x K blocks per CTA, plus
// the FP32 partials that a split writes and the reduction reads, counted in K
// blocks' worth of operand traffic spread over the SMs; the smallest split on
// ties, at least 8 K blocks per split.
int model_splits(int m, int n2, int k_blocks, int bn) {
  const long long tiles = static_cast<long long>(ceil_div(m, BM)) * static_cast<long long>(ceil_div(n2, bn));
  const double kblock_bytes = static_cast<double>(BM + bn) * BK * 2;
  double best_cost = -1;
  int splits = 1;
  for (long long s = 1; s <= max_splits_for(k_blocks); ++s) {
    const long long waves = (tiles * s + 147) / 148;
    const double partial = s > 1 ? 2.0 * 4.0 * static_cast<double>(m) * n2 * s / (148.0 * kblock_bytes) : 0.0;
    const double cost = static_cast<double>(waves * ((k_blocks + s - 1) / s)) + partial;
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      splits = static_cast<int>(s);
    }
  }
  return splits;
}

// One product with the given tile width and split count.
void run_config(const std::uint16_t* a, long long lda, const std::uint16_t* b, long long ldb, int m, int n,
                long long kexp, Split split, const ProductOutput out[2], int second, double alpha, int bn, int splits,
                Scratch& workspace, cudaStream_t stream) {
  const int n2 = 2 * n;
  const int k_blocks = static_cast<int>(kexp / BK);
  const int kpb = static_cast<int>(ceil_div(k_blocks, splits));
  splits = static_cast<int>(ceil_div(k_blocks, kpb));
  EpilogueArgs ep{m, n2, nullptr, {out[0], out[1]}, second, alpha, split == Split::BF16x3};
  if (splits > 1)
    ep.partial = static_cast<Cx<float>*>(workspace.reserve(sizeof(Cx<float>) * static_cast<std::size_t>(m) * n * splits));
  if (bn == 256) launch<256>(a, lda, b, ldb, m, n2, kexp, ep, splits, k_blocks, kpb, stream);
  else if (bn == 160) launch<160>(a, lda, b, ldb, m, n2, kexp, ep, splits, k_blocks, kpb, stream);
  else launch<128>(a, lda, b, ldb, m, n2, kexp, ep, splits, k_blocks, kpb, stream);
  if (splits > 1) {
    reduce_splits_kernel<<<dim3(static_cast<unsigned>(ceil_div(m, 256)), static_cast<unsigned>(std::min(n, kMaxGridY))),
                           256, 0, stream>>>(
        m, n, splits, ep.partial, out[0], out[1], second, alpha);
    SDFT_LAUNCH("reduce_splits_kernel");
  }
}

// Tile autotuner. Shapes are grouped into classes (row tiles of 128, real
// column count rounded up to 32, K blocks rounded up to a geometric grid of
// ratio 2^(1/8), so that operators whose plane-wave counts differ by a few
// per cent share their classes); the first product of a class times every
// candidate -- the three column widths, each with the cost model's split
// count and twice it, and no split -- on the caller's
// stream into a scratch output (CUDA events, one untimed run first) and keeps
// the fastest for the class, for the life of the process. Later products of
// the class, on any stream or thread, use that choice, so a given process
// computes every later product of a class with the same tiles and the same
// summation order. SDFT_B200_GEMM_AUTOTUNE=0 uses the cost model alone.
struct ShapeClass {
  int row_tiles, column_units, k_blocks;
  bool share_k;  // whether K may be split
  Split split;
  bool operator<(const ShapeClass& o) const {
    return std::tie(row_tiles, column_units, k_blocks, share_k, split) <
           std::tie(o.row_tiles, o.column_units, o.k_blocks, o.share_k, o.split);
  }
};
struct TileChoice {
  int bn, splits;
  float ms;
};
std::mutex g_tune_mutex;
std::map<ShapeClass, TileChoice> g_tuned;

bool autotune_enabled() {
  static const bool enabled = [] {
    const char* v = std::getenv("SDFT_B200_GEMM_AUTOTUNE");
    if (!v || std::string(v) == "1") return true;
    if (std::string(v) == "0") return false;
    throw InvalidArgument("SDFT_B200_GEMM_AUTOTUNE must be 0 or 1");
  }();
  return enabled;
}

TileChoice tuned_choice(const std::uint16_t* a, long long lda, const std::uint16_t* b, long long ldb, int m, int n,
                        long long kexp, Split split, bool share_k, cudaStream_t stream) {
  const int n2 = 2 * n;
  const int k_blocks = static_cast<int>(kexp / BK);
  int k_class = 1;
  for (int j = 1; k_class < k_blocks; ++j) k_class = static_cast<int>(std::ceil(std::exp2(j / 8.0)));
  const ShapeClass key{static_cast<int>(ceil_div(m, BM)), static_cast<int>(ceil_div(n2, 32)), k_class,
                       share_k, split};
  std::lock_guard<std::mutex> lock(g_tune_mutex);
  auto found = g_tuned.find(key);
  if (found != g_tuned.end()) return found->second;
  std::vector<std::pair<int, int>> candidates;
  for (int bn : {128, 160, 256}) {
    const int s = share_k ? model_splits(m, n2, k_blocks, bn) : 1;
    for (int count : {1, s, share_k ? std::min(max_splits_for(k_blocks), 2 * s) : 1})
      if (std::find(candidates.begin(), candidates.end(), std::make_pair(bn, count)) == candidates.end())
        candidates.emplace_back(bn, count);
  }
  static thread_local Scratch output, partials;
  auto* c = static_cast<Cx<double>*>(output.reserve(sizeof(Cx<double>) * static_cast<std::size_t>(m) * n));
  cudaEvent_t start = nullptr, stop = nullptr;
  SDFT_CUDA(cudaEventCreate(&start));
  SDFT_CUDA(cudaEventCreate(&stop));
  TileChoice best{model_width(n2), 0, -1.0f};
  best.splits = share_k ? model_splits(m, n2, k_blocks, best.bn) : 1;
  const ProductOutput scratch[2] = {product_output(c, m, false), {}};
  try {
    for (const auto& [bn, splits] : candidates) {
      run_config(a, lda, b, ldb, m, n, kexp, split, scratch, n, 1.0, bn, splits, partials, stream);
      SDFT_CUDA(cudaEventRecord(start, stream));
      run_config(a, lda, b, ldb, m, n, kexp, split, scratch, n, 1.0, bn, splits, partials, stream);
      SDFT_CUDA(cudaEventRecord(stop, stream));
      SDFT_CUDA(cudaEventSynchronize(stop));
      float ms = 0;
      SDFT_CUDA(cudaEventElapsedTime(&ms, start, stop));
      if (best.ms < 0 || ms < best.ms) best = TileChoice{bn, splits, ms};
    }
  } catch (...) {
    cudaEventDestroy(start);
    cudaEventDestroy(stop);
    throw;
  }
  cudaEventDestroy(start);
  cudaEventDestroy(stop);
  g_tuned.emplace(key, best);
  return best;
}

}  // namespace

namespace {
void product(const std::uint16_t* a, long long lda, const std::uint16_t* b, long long ldb, int m, int n,
             long long kexp, Split split, const ProductOutput out[2], int second, double alpha, bool share_k,
             Scratch& workspace,
             cudaStream_t stream) {
  if (m <= 0 || n <= 0 || kexp <= 0) return;
  if (kexp % BK != 0) throw InvalidArgument("expanded K must be a multiple of 64");
  int bn, splits;
  if (autotune_enabled()) {
    const TileChoice choice = tuned_choice(a, lda, b, ldb, m, n, kexp, split, share_k, stream);
    bn = choice.bn;
    splits = choice.splits;
  } else {
    bn = model_width(2 * n);
    splits = share_k ? model_splits(m, 2 * n, static_cast<int>(kexp / BK), bn) : 1;
  }
  run_config(a, lda, b, ldb, m, n, kexp, split, out, second, alpha, bn, splits, workspace, stream);
}
}  // namespace

void umma_complex_gemm(const std::uint16_t* a, long long lda, const std::uint16_t* b, long long ldb, int m, int n,
                       long long kexp, Split split, Cx<double>* c, long long ldc, bool add, double alpha,
                       Scratch& workspace,
                       cudaStream_t stream) {
  const ProductOutput out[2] = {product_output(c, ldc, add), {}};
  product(a, lda, b, ldb, m, n, kexp, split, out, n, alpha, true, workspace, stream);
}

std::size_t gemm_tuned_classes(std::size_t capacity, int* rows) {
  std::lock_guard<std::mutex> lock(g_tune_mutex);
  std::size_t i = 0;
  for (const auto& [key, choice] : g_tuned) {
    if (i < capacity && rows) {
      int* r = rows + 5 * i;
      r[0] = key.row_tiles * BM;
      r[1] = key.column_units * 32;
      r[2] = key.k_blocks;
      r[3] = choice.bn;
      r[4] = choice.splits;
    }
    ++i;
  }
  return g_tuned.size();
}

Split search_split() {
  static const Split split = [] {
    const char* v = std::getenv("SDFT_B200_SPLIT");
    if (!v || std::string(v) == "x3") return Split::BF16x3;
    if (std::string(v) == "x6") return Split::BF16x6;
    throw InvalidArgument("SDFT_B200_SPLIT must be x3 or x6");
  }();
  return split;
}

void pack_persistent(Op aop, const Cx<double>* a, long long lda, int rows, int k, Split split, PackedA& out,
                     cudaStream_t stream) {
  release(out);
  out.ld = expanded_k(k, split);
  out.rows = rows;
  out.k = k;
  out.split = split;
  out.stream = stream;
  out.data = static_cast<std::uint16_t*>(
      stream_alloc(sizeof(std::uint16_t) * static_cast<std::size_t>(out.ld) * rows, stream));
  pack_a(aop, a, lda, rows, k, split, out.data, out.ld, stream);
}

void release(PackedA& packed) {
  stream_free(packed.data, packed.stream);
  packed = PackedA{};
}

void gemm_tc(Op aop, int m, int n, int k, const Cx<double>* a, long long lda, const PackedA* packed,
             const Cx<double>* b, long long ldb, Cx<double>* c, long long ldc, bool add, double alpha, Split split,
             TensorCoreWorkspace& ws, cudaStream_t stream) {
  if (m <= 0 || n <= 0 || k <= 0) return;
  const long long kexp = expanded_k(k, split);
  const std::uint16_t* pa;
  long long lda_p;
  if (packed) {
    if (packed->rows != m || packed->k != k || packed->split != split) throw InvalidArgument("packed operand shape mismatch");
    pa = packed->data;
    lda_p = packed->ld;
  } else {
    auto* buf = static_cast<std::uint16_t*>(ws.a.reserve(sizeof(std::uint16_t) * static_cast<std::size_t>(kexp) * m));
    pack_a(aop, a, lda, m, k, split, buf, kexp, stream);
    pa = buf;
    lda_p = kexp;
  }
  auto* pb = static_cast<std::uint16_t*>(ws.b.reserve(sizeof(std::uint16_t) * static_cast<std::size_t>(kexp) * 2 * n));
  pack_b(b, ldb, k, n, split, pb, kexp, stream);
  umma_complex_gemm(pa, lda_p, pb, kexp, m, n, kexp, split, c, ldc, add, alpha, ws.partial, stream);
}

void gemm_tc_packed(const PackedA& packed, int n, const Cx<double>* b, long long ldb, const ProductOutput out[2],
                    int second, TensorCoreWorkspace& ws, cudaStream_t stream) {
  if (packed.rows <= 0 || n <= 0 || packed.k <= 0) return;
  const long long kexp = expanded_k(packed.k, packed.split);
  auto* pb = static_cast<std::uint16_t*>(ws.b.reserve(sizeof(std::uint16_t) * static_cast<std::size_t>(kexp) * 2 * n));
  pack_b(b, ldb, packed.k, n, packed.split, pb, kexp, stream);
  product(packed.data, packed.ld, pb, kexp, packed.rows, n, kexp, packed.split, out, second, 1.0, false, ws.partial, stream);
}

unsigned int umma_error_flag() {
  unsigned int value = 0;
  SDFT_CUDA(cudaMemcpyFromSymbol(&value, g_umma_error, sizeof(value)));
  return value;
}

}  // namespace sdft_b200
