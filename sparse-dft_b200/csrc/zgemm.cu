// FP64 complex products on the FP64 matrix instruction (mma.m8n8k4).
#include <algorithm>

#include "gemm.cuh"

namespace sdft_b200 {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int TM = 8 * kWarps;  // rows of a CTA tile: one 8-row strip per warp
constexpr int KC = 8;           // K entries of a stage
constexpr int kStages = 4;
constexpr int kMaxTiles = 8;    // 8-column tiles per CTA
constexpr int kMaxSplit = 8;    // CTAs of a cluster that share a tile's K

// Shared-memory strides (complex values) that put the 2 rows x 4 K entries of
// a quarter-warp's 16-byte reads into different banks.
constexpr int kRowStride = TM + 2;  // K-major A (op N): entry k * kRowStride + row
constexpr int kKStride = KC + 4;    // row-major A (op C) and B: entry row * kKStride + k

struct ZgemmArgs {
  int m, n, k, k_share;  // K entries of one CTA of a cluster (a multiple of KC)
  const Cx<double>* a;
  const Cx<double>* b;
  ProductOutput out[2];
  int second;  // first column of out[1]
  int row_tiles;
  long long lda, ldb;
  double alpha;
};

template <bool ADJOINT, int NT>
constexpr int stage_entries() {
  return (ADJOINT ? TM * kKStride : KC * kRowStride) + 8 * NT * kKStride;
}
template <bool ADJOINT, int NT>
constexpr std::size_t zgemm_smem() {
  const int stages = kStages * stage_entries<ADJOINT, NT>(), tile = 8 * NT * TM;
  return sizeof(Cx<double>) * (stages > tile ? stages : tile);
}

// 16 bytes to shared memory, zeros where !in (src must be readable memory all the same).
__device__ __forceinline__ void copy_entry(Cx<double>* dst, const Cx<double>* src, bool in) {
  const unsigned to = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(src), "r"(in ? 16 : 0) : "memory");
}

__device__ __forceinline__ void mma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// C tile of TM rows x 8 NT columns = alpha op(A) B (+ C), op = adjoint or none.
// Four real products per complex one, in K order, accumulated in registers;
// stages of KC entries stream through shared memory by cp.async. A warp issues
// 4 NT matrix instructions per K step of 4 for NT + 1 shared-memory reads. At the
// sizes it takes, latency binds it: 160 x 20 x 1000 and 160^3 keep the matrix pipe
// 27 and 23 % active with 72 and 120 CTAs in flight, waiting on the stages'
// barriers, the accumulator chain and the first loads. The CTAs of a cluster (blockIdx.z) take consecutive
// shares of K and add their tiles through distributed shared memory in rank
// order, so a small product spread over K needs no second kernel (cuBLAS's
// shared-K products add one, and a small one leaves most SMs idle: 160 x 20 x
// 1000 10.3 us here and 12.7 there, 64 x 80 x 64 5.4 and 12.5, 160^3 8.5 and
// 10.6; the eight-atom FP64 solve, 1800 such products, 55.5 -> 45.4 ms).
template <bool ADJOINT, int NT>
__global__ void __launch_bounds__(kThreads, 2) zgemm_kernel(const ZgemmArgs g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cx<double>* smem = reinterpret_cast<Cx<double>*>(smem_raw);
  constexpr int A_ENTRIES = ADJOINT ? TM * kKStride : KC * kRowStride, STAGE = stage_entries<ADJOINT, NT>();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, row = lane >> 2, quad = lane & 3;
  // Tiles on one grid axis, rows fastest: any number of rows or columns.
  const int m0 = static_cast<int>(blockIdx.x % g.row_tiles) * TM, n0 = static_cast<int>(blockIdx.x / g.row_tiles) * 8 * NT;
  const int k0 = blockIdx.z * g.k_share, k1 = min(g.k, k0 + g.k_share);
  const int chunks = max(0, (k1 - k0 + KC - 1) / KC);

  auto load = [&](int chunk) {
    Cx<double>* as = smem + (chunk % kStages) * STAGE;
    Cx<double>* bs = as + A_ENTRIES;
    const int kb = k0 + chunk * KC;
#pragma unroll
    for (int u = 0; u < TM * KC / kThreads; ++u) {
      const int i = tid + u * kThreads;
      const int r = ADJOINT ? i / KC : i % TM, kk = ADJOINT ? i % KC : i / TM;
      const bool in = m0 + r < g.m && kb + kk < k1;
      const long long at = ADJOINT ? (kb + kk) + static_cast<long long>(m0 + r) * g.lda
                                   : (m0 + r) + static_cast<long long>(kb + kk) * g.lda;
      copy_entry(as + (ADJOINT ? r * kKStride + kk : kk * kRowStride + r), in ? g.a + at : g.a, in);
    }
#pragma unroll
    for (int u = 0; u < (8 * NT * KC + kThreads - 1) / kThreads; ++u) {
      const int i = tid + u * kThreads, j = i / KC, kk = i % KC;
      if (i < 8 * NT * KC) {
        const bool in = n0 + j < g.n && kb + kk < k1;
        copy_entry(bs + j * kKStride + kk, in ? g.b + (kb + kk) + static_cast<long long>(n0 + j) * g.ldb : g.b, in);
      }
    }
  };

  double re[NT][2] = {}, im[NT][2] = {};
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < chunks) load(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int chunk = 0; chunk < chunks; ++chunk) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();  // the stage has landed, and the one before it has been read by every warp
    if (chunk + kStages - 1 < chunks) load(chunk + kStages - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const Cx<double>* as = smem + (chunk % kStages) * STAGE;
    const Cx<double>* bs = as + A_ENTRIES;
#pragma unroll
    for (int k = 0; k < KC; k += 4) {
      const Cx<double> a = ADJOINT ? as[(warp * 8 + row) * kKStride + k + quad] : as[(k + quad) * kRowStride + warp * 8 + row];
      // C.re += a.re b.re -/+ a.im b.im, C.im += a.re b.im +/- a.im b.re
      const double ai = ADJOINT ? -a.im : a.im;
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const Cx<double> b = bs[(t * 8 + row) * kKStride + k + quad];
        mma(re[t], a.re, b.re);
        mma(im[t], a.re, b.im);
        mma(re[t], -ai, b.im);
        mma(im[t], ai, b.re);
      }
    }
  }

  auto store = [&](int r, int j, Cx<double> v) {
    const int row_c = m0 + r, column = n0 + j;
    if (row_c >= g.m || column >= g.n) return;
    const bool other = column >= g.second;
    const ProductOutput& o = g.out[other ? 1 : 0];
    const long long col = other ? column - g.second : column;
    v = Cx<double>{g.alpha * v.re, g.alpha * v.im};
    if (o.prior) {
      const Cx<double> p = o.prior[row_c + col * o.ldp];
      v.re = __dadd_rn(v.re, __dmul_rn(o.prior_scale, p.re));
      v.im = __dadd_rn(v.im, __dmul_rn(o.prior_scale, p.im));
    }
    o.c[row_c + col * o.ldc] = v;
  };
  if (gridDim.z == 1) {
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int u = 0; u < 2; ++u) store(warp * 8 + row, t * 8 + 2 * quad + u, Cx<double>{re[t][u], im[t][u]});
    return;
  }
  // Shares of K: every CTA leaves its tile in shared memory, then adds up its slice of the cluster's tiles.
  __syncthreads();
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int u = 0; u < 2; ++u) smem[(t * 8 + 2 * quad + u) * TM + warp * 8 + row] = Cx<double>{re[t][u], im[t][u]};
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  const int parts = gridDim.z;
  constexpr int ENTRIES = 8 * NT * TM;
  const unsigned own = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  for (int i = static_cast<int>(blockIdx.z) * kThreads + tid; i < ENTRIES; i += parts * kThreads) {
    Cx<double> sum{0.0, 0.0};
    for (int r = 0; r < parts; ++r) {
      unsigned remote;
      Cx<double> v;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(own), "r"(r));
      asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];"
                   : "=d"(v.re), "=d"(v.im)
                   : "r"(remote + static_cast<unsigned>(sizeof(Cx<double>)) * i)
                   : "memory");
      sum = sum + v;
    }
    store(i % TM, i / TM, sum);
  }
  // No CTA leaves while another may still read its tile.
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <bool ADJOINT, int NT>
void launch(const ZgemmArgs& g, int split, cudaStream_t stream) {
  constexpr std::size_t smem = zgemm_smem<ADJOINT, NT>();
  allow_dynamic_smem(zgemm_kernel<ADJOINT, NT>, smem);
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(static_cast<unsigned>(g.row_tiles * ceil_div(g.n, 8 * NT)), 1, static_cast<unsigned>(split));
  config.blockDim = dim3(kThreads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute cluster{};
  cluster.id = cudaLaunchAttributeClusterDimension;
  cluster.val.clusterDim.x = cluster.val.clusterDim.y = 1;
  cluster.val.clusterDim.z = static_cast<unsigned>(split);
  config.attrs = &cluster;
  config.numAttrs = 1;
  SDFT_CUDA(cudaLaunchKernelEx(&config, zgemm_kernel<ADJOINT, NT>, g));
  SDFT_LAUNCH("zgemm_kernel");
}

template <bool ADJOINT>
void dispatch(const ZgemmArgs& g, int tiles, int split, cudaStream_t stream) {
  switch (tiles) {
    case 1: return launch<ADJOINT, 1>(g, split, stream);
    case 2: return launch<ADJOINT, 2>(g, split, stream);
    case 3: return launch<ADJOINT, 3>(g, split, stream);
    case 4: return launch<ADJOINT, 4>(g, split, stream);
    case 5: return launch<ADJOINT, 5>(g, split, stream);
    case 6: return launch<ADJOINT, 6>(g, split, stream);
    case 7: return launch<ADJOINT, 7>(g, split, stream);
    default: return launch<ADJOINT, 8>(g, split, stream);
  }
}

}  // namespace

void zgemm_device(bool adjoint, int m, int n, int k, const Cx<double>* a, long long lda, const Cx<double>* b,
                  long long ldb, const ProductOutput out[2], int second, double alpha, bool share_k,
                  cudaStream_t stream) {
  // Tile width and K shares of the least estimated time: the SM's pipe takes
  // about 32 NT cycles per K entry of a tile, CTAs run in waves of one per SM
  // (two resident CTAs share the pipe), a CTA costs about 2000 cycles to fill
  // and store and a cluster's sum 1500 more.
  int tiles = 1, split = 1;
  double best = 0.0;
  const long long rows = static_cast<long long>(ceil_div(m, TM)), columns = static_cast<long long>(ceil_div(n, 8));
  for (int t = 1; t <= std::min<long long>(kMaxTiles, columns); ++t)
    for (int s = 1; s <= (share_k ? kMaxSplit : 1); s *= 2) {
      if (s > 1 && k < 32 * s) break;
      const double waves = static_cast<double>(ceil_div(rows * ceil_div(columns, t) * s, kSmCount));
      const double time = waves * (32.0 * t * ceil_div(k, s) + 2000.0) + (s > 1 ? 1500.0 : 0.0);
      if (best == 0.0 || time < best) {
        best = time;
        tiles = t;
        split = s;
      }
    }
  const int share = static_cast<int>(ceil_div(ceil_div(k, split), KC)) * KC;
  const ZgemmArgs g{m, n, k, share, a, b, {out[0], out[1]}, second, static_cast<int>(rows), lda, ldb, alpha};
  if (adjoint) dispatch<true>(g, tiles, split, stream);
  else dispatch<false>(g, tiles, split, stream);
}

}  // namespace sdft_b200
