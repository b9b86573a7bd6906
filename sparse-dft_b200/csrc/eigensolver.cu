// Device eigensolver for the Davidson Rayleigh-Ritz step (lowest `wanted`
// eigenpairs of an m x m Hermitian matrix, m up to kRowsPerThread * kTridiagThreads
// = 1280).
//
// 1. Householder reduction (LAPACK zhetd2, lower, H_j = I - tau v v^H with
//    v[j+1] = 1): tridiagonalize_cluster_kernel for orders up to 256 and for
//    the last 256 rows of larger matrices, in one 16-CTA cluster;
//    tridiagonalize_kernel for the steps before: one cooperative launch, one
//    CTA per SM, columns distributed cyclically and held in shared memory.
//    Its step j needs one grid-wide barrier: every CTA forms w and the next
//    reflector's x redundantly from the published A x and head row, applies
//    the update to its own columns, accumulates the next A x in the same pass,
//    and publishes it with the next head row. Exchange buffers are
//    double-buffered by step parity. The barrier is a counting barrier with a
//    time limit: on expiry an error word is set and every CTA returns.
//    tridiagonalize_columns_kernel: the form of Reduction::Columns.
// 2. bisect_kernel: one warp per wanted eigenvalue, multisection with 64 points
//    (128 for Reduction::Columns) on division-free Sturm counts of the
//    tridiagonal matrix.
// 3. inverse_iteration_kernel: one thread per wanted eigenvalue, factors in
//    shared memory; LU with partial pivoting of T - lambda I, two solves from
//    a start vector of its own; then cluster_orthonormalize_kernel, one CTA
//    per cluster of eigenvalues closer than 1e-9 of the matrix scale, runs
//    CGS2 over the cluster's vectors in eigenvalue order.
// 4. reflector_blocks_kernel: the reflectors in blocks of 64 as
//    I - V T V^H (compact WY); the blocks are applied to the tridiagonal
//    eigenvectors from the last to the first with three cuBLAS ZGEMMs each.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>

#include "dense.cuh"
#include "eigensolver.cuh"

namespace sdft_b200 {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxCpc = 10;
// The tridiagonalisation runs one CTA of kTridiagThreads per SM; each thread
// holds kRowsPerThread rows of the reflector and rank-2 vectors in registers
// (m <= kRowsPerThread * kTridiagThreads). 512 threads with 3 rows each
// measured slower than 256 with 5 (12.1 vs 9.9 ms at m = 1280): the step's
// CTA barriers and reductions grow with the warp count.
constexpr int kTridiagThreads = 256;
constexpr int kTridiagWarps = kTridiagThreads / 32;
constexpr int kRowsPerThread = 5;  // m <= 1280
constexpr int kReflectorBlock = 64;
constexpr int kInvitThreads = 4;
constexpr int kMaxShares = 5;  // CTA shares per lane: grid <= 160
constexpr unsigned long long kWaitNs = 2000000000ULL;
constexpr double kClusterTolerance = 1e-9;


void check_blas(cublasStatus_t status, const char* what) {
  if (status != CUBLAS_STATUS_SUCCESS)
    throw CudaError(std::string("cuBLAS error ") + std::to_string(static_cast<int>(status)) + " in " + what);
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ Cx<double> cconj(Cx<double> a) { return {a.re, -a.im}; }
__device__ __forceinline__ Cx<double> cadd(Cx<double> a, Cx<double> b) { return {a.re + b.re, a.im + b.im}; }
__device__ __forceinline__ Cx<double> csub(Cx<double> a, Cx<double> b) { return {a.re - b.re, a.im - b.im}; }
__device__ __forceinline__ Cx<double> cmulz(Cx<double> a, Cx<double> b) {
  return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
// conj(a) * b
__device__ __forceinline__ Cx<double> cdot1(Cx<double> a, Cx<double> b) {
  return {a.re * b.re + a.im * b.im, a.re * b.im - a.im * b.re};
}

// Counting grid barrier with a time limit. Returns false (and every CTA
// should return) when the limit expired here or the error word is set. Warp
// 0's writes (ordered before thread 0 by its __syncwarp) are released by the
// arrival; the acquire fence after the wait and the CTA barrier order the reads
// that follow.
__device__ bool grid_barrier(unsigned int* arrive, unsigned int* error, unsigned int target, int* ok) {
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrive) : "memory");
    const unsigned long long start = global_ns();
    int good = 1;
    while (true) {
      unsigned int cur;
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(cur) : "l"(arrive) : "memory");
      if (cur >= target) break;
      if (*reinterpret_cast<volatile unsigned int*>(error) != 0u) {
        good = 0;
        break;
      }
      if (global_ns() - start > kWaitNs) {
        atomicOr(error, 1u);
        good = 0;
        break;
      }
    }
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    *ok = good;
  }
  __syncthreads();
  return *ok != 0;
}

struct TridiagArgs {
  Cx<double>* a;
  int m, grid, cpc;
  int rows;  // column stride in shared memory: m rounded up to kTridiagThreads
  int stop;  // reflectors formed here; the cluster kernel takes the trailing matrix
  double* d;
  double* e;
  Cx<double>* tau;
  Cx<double>* reflectors;  // m x m, column j holds v_j in rows j+1..m-1
  Cx<double>* abuf;        // 2 x m: A x
  Cx<double>* hbuf;        // 2 x m: head row
  double* shares;          // 2 x grid: each CTA's part of x^H A x
  unsigned int* arrive;
  unsigned int* error;  // set when a barrier wait runs out; every CTA then returns
};

// Scalars of the reflector that reduces a column with `head` and, below it, a
// part of squared norm xnorm2 (LAPACK zlarfg): H = I - tau v v^H with v = e +
// scale x, and the real off-diagonal beta; tau = scale = 0 where there is
// nothing to reduce. A whole warp calls this: its two reciprocals run on two
// lanes at once.
struct Reflector {
  Cx<double> tau, scale;
  double beta;
};

__device__ __forceinline__ Reflector make_reflector(int lane, Cx<double> head, double xnorm2) {
  const bool trivial = xnorm2 == 0.0 && head.im == 0.0;
  const double beta = -copysign(sqrt(head.re * head.re + head.im * head.im + xnorm2), head.re);
  const double dr = head.re - beta;
  const double inverse = 1.0 / ((lane & 1) ? dr * dr + head.im * head.im : beta);
  const double inv_beta = __shfl_sync(0xffffffffu, inverse, 0), inv_den = __shfl_sync(0xffffffffu, inverse, 1);
  if (trivial) return {{0.0, 0.0}, {0.0, 0.0}, head.re};
  return {{-dr * inv_beta, -head.im * inv_beta}, {dr * inv_den, -head.im * inv_den}, beta};
}

// Sum over the warp of each of N <= 32 values: lane i returns value i, the
// values halving with every exchange.
template <int N>
__device__ __forceinline__ double warp_total(double (&v)[N], int lane) {
  static_assert(N <= 32, "one value per lane");
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int i = 0; i < o; ++i) {
      if (i >= N) continue;
      const bool upper = lane & o;
      const double low = v[i], high = i + o < N ? v[i + o < N ? i + o : 0] : 0.0;
      v[i] = (upper ? high : low) + __shfl_xor_sync(0xffffffffu, upper ? low : high, o);
    }
  }
  return v[0];
}

// The reduction's first `stop` steps, one CTA per SM: column c = cta + G q in
// the CTA's shared memory, rows r = tid + kTridiagThreads k per thread, whose
// entries of v, w and x live in registers. A step is the cluster kernel's below
// (the same vector phase, pass and publication, A x and head rows through
// global memory) with one CTA barrier between the pass's sums and their
// publication, and the grid barrier; the reflector's scalars are formed by the
// last warp while the barrier is waited for, so neither their square root and
// divisions nor a norm reduction lie on the step's chain.
// Bound by that chain: the barrier's release, poll and L2 round trips, and the
// pass over own columns. 5.0 us a step at orders 320 to 640, 5.8 at 1280; with
// p and the next column published instead of A x and the head row (a second
// CTA barrier, and the norm, the square root and the divisions behind the grid
// barrier) 9.3, 7.3 and 8.3 us. Orders 320, 640, 1280 whole: 1.06 -> 0.79,
// 3.25 -> 2.38, 8.91 -> 6.41 ms.
__global__ void __launch_bounds__(kTridiagThreads, 1) tridiagonalize_kernel(TridiagArgs t) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int R = kRowsPerThread, SUMS = 2 * kMaxCpc + 1;
  const int m = t.m, G = t.grid, cpc = t.cpc, LD = t.rows, cta = blockIdx.x, tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  Cx<double>* cols = reinterpret_cast<Cx<double>*>(smem_raw);
  Cx<double>* own = cols + static_cast<long long>(cpc) * LD + 2 * kMaxCpc * warp;  // per warp: w, then v at own columns
  Cx<double>* xown = cols + static_cast<long long>(cpc) * LD + 2 * kMaxCpc * kTridiagWarps;  // [2][kMaxCpc], by step parity
  Cx<double>* pick = xown + 2 * kMaxCpc;  // entry below the head
  Cx<double>* scalars = pick + 1;         // tau, scale
  double* red = reinterpret_cast<double*>(scalars + 2);  // [kTridiagWarps][32]
  __shared__ int ok;

  for (int q = 0; q < cpc; ++q) {
    const int c = cta + q * G;
    for (int r = tid; r < LD; r += kTridiagThreads)
      cols[static_cast<long long>(q) * LD + r] =
          c < m && r < m ? t.a[r + static_cast<long long>(c) * m] : Cx<double>{0.0, 0.0};
  }

  Cx<double> x[R];
  int slot[R];  // own column of the same index as the row, or -1
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const int r = tid + k * kTridiagThreads;
    x[k] = Cx<double>{0.0, 0.0};
    slot[k] = r < m && r >= cta && (r - cta) % G == 0 ? (r - cta) / G : -1;
  }
  int turn = G - 1;  // j mod G: the CTA that stores reflector j
  for (int j = -1; j < t.stop; ++j, turn = turn + 1 == G ? 0 : turn + 1) {
    const int par = j & 1, next = par ^ 1, h = j + 1;
    const bool last = j == t.stop - 1;
    const int first_k = h / kTridiagThreads, last_k = LD / kTridiagThreads;  // rows of a thread that are alive
    const int first_q = last ? (h - cta + G - 1) / G : (h - cta + G) / G;     // own columns c > h (c >= h at the end)
    Cx<double> v[R], w[R];
    double sums[SUMS];
#pragma unroll
    for (int i = 0; i < SUMS; ++i) sums[i] = 0.0;
    {
      const double2* ab = reinterpret_cast<const double2*>(t.abuf + static_cast<long long>(par) * m);
      const double2* hb = reinterpret_cast<const double2*>(t.hbuf + static_cast<long long>(par) * m);
      const double* sb = t.shares + static_cast<long long>(par) * G;
      // All of the step's global reads first (one round of L2 latency).
      const double2 zero2 = make_double2(0.0, 0.0);
      double2 aq[R], hq[R], ah = zero2, hh = zero2, ac = zero2, hc = zero2;
      double part[kMaxShares];
      const int c = cta + lane * G;
      const bool mine = j >= 0 && lane < cpc && c >= h && c < m;
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const int r = tid + k * kTridiagThreads;
        const bool row = j >= 0 && r >= h && r < m;
        aq[k] = row ? __ldcg(ab + r) : zero2;
        hq[k] = row ? __ldcg(hb + r) : zero2;
      }
      if (j >= 0) {
        ah = __ldcg(ab + h);
        hh = __ldcg(hb + h);
      }
      if (mine) {
        ac = __ldcg(ab + c);
        hc = __ldcg(hb + c);
      }
#pragma unroll
      for (int i = 0; i < kMaxShares; ++i) part[i] = j >= 0 && lane + 32 * i < G ? __ldcg(sb + lane + 32 * i) : 0.0;
      Cx<double> tau{0.0, 0.0}, scale{0.0, 0.0}, head_w{0.0, 0.0};
      double alpha = 0.0;
      if (j >= 0) {
        tau = scalars[0];
        scale = scalars[1];
        double xax = 0.0;
#pragma unroll
        for (int i = 0; i < kMaxShares; ++i) xax += part[i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) xax += __shfl_xor_sync(0xffffffffu, xax, o);
        const double vav = fma(scale.re * scale.re + scale.im * scale.im, xax,
                               fma(2.0, scale.re * ah.x - scale.im * ah.y, hh.x));
        alpha = (-0.5 * (tau.re * tau.re + tau.im * tau.im)) * vav;
        head_w = cmulz(tau, cadd(Cx<double>{hh.x, -hh.y}, cmulz(scale, Cx<double>{ah.x, ah.y})));
        head_w.re += alpha;  // v[h] = 1
        head_w.im = -head_w.im;
      }
      // w and v at own columns, for this warp's pass.
      if (lane < cpc) {
        Cx<double> vc{0.0, 0.0}, wc{0.0, 0.0};
        if (mine) {
          vc = c == h ? Cx<double>{1.0, 0.0} : cmulz(scale, xown[par * kMaxCpc + lane]);
          wc = cmulz(tau, cadd(Cx<double>{hc.x, -hc.y}, cmulz(scale, Cx<double>{ac.x, ac.y})));
          wc.re += alpha * vc.re;
          wc.im += alpha * vc.im;
        }
        own[lane] = cconj(wc);
        own[kMaxCpc + lane] = cconj(vc);
      }
      __syncwarp();
      const bool writer = turn == cta;
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const int r = tid + k * kTridiagThreads;
        Cx<double> col{0.0, 0.0};
        v[k] = w[k] = Cx<double>{0.0, 0.0};
        if (r < m && r >= h) {
          if (j < 0) {
            col = t.a[r];
          } else {
            const Cx<double> hr{hq[k].x, -hq[k].y};
            v[k] = r == h ? Cx<double>{1.0, 0.0} : cmulz(x[k], scale);
            w[k] = cmulz(tau, cadd(hr, cmulz(scale, Cx<double>{aq[k].x, aq[k].y})));
            w[k].re += alpha * v[k].re;
            w[k].im += alpha * v[k].im;
            col = csub(hr, cadd(cmulz(v[k], head_w), w[k]));
            if (writer) t.reflectors[r + static_cast<long long>(j) * m] = v[k];
          }
          if (r == h && cta == 0 && !last) t.d[h] = col.re;
          if (r == h + 1) pick[0] = col;
        }
        x[k] = r > h + 1 && r < m ? col : Cx<double>{0.0, 0.0};
        sums[2 * kMaxCpc] += x[k].re * x[k].re + x[k].im * x[k].im;
        if (slot[k] >= 0) xown[next * kMaxCpc + slot[k]] = x[k];
      }
    }

    // Update j on own columns, and the products A x of the next reflector.
    // Finished rows meet zeros of v, w and x; whole finished rows and columns
    // are skipped.
#pragma unroll
    for (int q = 0; q < kMaxCpc; ++q) {
      if (q < first_q || q >= cpc) continue;
      const Cx<double> wc = own[q], vc = own[kMaxCpc + q];
      Cx<double>* a = cols + static_cast<long long>(q) * LD + tid;
      Cx<double> y[R];
#pragma unroll
      for (int k = 0; k < R; ++k)
        if (k >= first_k && k < last_k) y[k] = a[k * kTridiagThreads];
#pragma unroll
      for (int k = 0; k < R; ++k)
        if (k >= first_k && k < last_k) {
          y[k].re = fma(-v[k].re, wc.re, fma(v[k].im, wc.im, fma(-w[k].re, vc.re, fma(w[k].im, vc.im, y[k].re))));
          y[k].im = fma(-v[k].re, wc.im, fma(-v[k].im, wc.re, fma(-w[k].re, vc.im, fma(-w[k].im, vc.re, y[k].im))));
          const Cx<double> p = cdot1(y[k], x[k]);
          sums[2 * q] += p.re;
          sums[2 * q + 1] += p.im;
        }
#pragma unroll
      for (int k = 0; k < R; ++k)
        if (k >= first_k && k < last_k) a[k * kTridiagThreads] = y[k];
    }
    if (last) break;

    const double total = warp_total(sums, lane);
    if (lane < SUMS) red[warp * 32 + lane] = total;
    __syncthreads();
    if (warp == 0) {
      const int c = cta + lane * G;
      double share = 0.0;
      if (lane < cpc && c > h && c < m) {
        Cx<double> ax{0.0, 0.0};
#pragma unroll
        for (int k = 0; k < kTridiagWarps; ++k) ax = cadd(ax, Cx<double>{red[k * 32 + 2 * lane], red[k * 32 + 2 * lane + 1]});
        const Cx<double> xc = xown[next * kMaxCpc + lane];
        t.abuf[static_cast<long long>(next) * m + c] = ax;
        t.hbuf[static_cast<long long>(next) * m + c] = cols[static_cast<long long>(lane) * LD + h + 1];
        share = ax.re * xc.re + ax.im * xc.im;
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) share += __shfl_xor_sync(0xffffffffu, share, o);
      if (lane == 0) t.shares[static_cast<long long>(next) * G + cta] = share;
      __syncwarp();
    } else if (warp == kTridiagWarps - 1) {
      double xnorm2 = lane < kTridiagWarps ? red[lane * 32 + 2 * kMaxCpc] : 0.0;
#pragma unroll
      for (int o = kTridiagWarps / 2; o > 0; o >>= 1) xnorm2 += __shfl_xor_sync(0xffffffffu, xnorm2, o);
      xnorm2 = __shfl_sync(0xffffffffu, xnorm2, 0);
      const Reflector f = make_reflector(lane, pick[0], xnorm2);
      if (lane == 0) {
        scalars[0] = f.tau;
        scalars[1] = f.scale;
        if (cta == 0) {
          t.e[h] = f.beta;
          t.tau[h] = f.tau;
        }
      }
    }
    if (!grid_barrier(t.arrive, t.error, static_cast<unsigned int>(G) * static_cast<unsigned int>(j + 2), &ok)) return;
  }
  __syncthreads();
  // The trailing matrix, every update applied, for the cluster kernel.
  for (int q = 0; q < cpc; ++q) {
    const int c = cta + q * G;
    if (c >= t.stop && c < m)
      for (int r = t.stop + tid; r < m; r += kTridiagThreads)
        t.a[r + static_cast<long long>(c) * m] = cols[static_cast<long long>(q) * LD + r];
  }
}

// Householder reduction of a matrix of order m <= kClusterOrder by one
// cluster of 16 CTAs: column c = rank + 16 q on CTA `rank`, held in registers
// for the whole reduction, every exchange through distributed shared memory.
// The grid kernel above pays a global release, a polled counter and L2 round
// trips per step: about 5 us whatever the order, against 1.25 us at order 64,
// 1.3 at 128 and 1.8 at 256 here (0.5 -> 0.28 ms for order 160 as a whole). The
// step is bound by its serial chain of instructions, not by a pipe or memory.
// It reduces whole matrices up to kClusterOrder and the trailing kClusterOrder
// rows of larger ones; a solve below kClusterOrder needs no cooperative
// launch, so solves on other streams do not queue behind it (its cluster-size
// attribute is still set with each launch).
//
// Reflector j has head row h = j + 1 and v = e_h + scale x, x the part of
// column j below h. Step j starts with x, and A x and row h of the trailing
// matrix (updates < j applied; by symmetry column h) complete in every CTA:
//   vector phase  A v = A e_h + scale A x, w = tau A v + alpha v, column h with
//                 update j applied, and from it the next x;
//   pass          update j and the products A x of the next reflector. A warp's
//                 lanes are 8 columns x 4 rows, a thread's tile RT rows (r = 32 i
//                 + row group) x CT columns (q = 8 k + lane): each v, w, x read
//                 from shared memory serves CT columns. (With the matrix in
//                 shared memory and one column per lane the pass was bound by
//                 shared-memory wavefronts, 20 per row.) Entries of finished
//                 rows and columns meet zeros of v, w and x, and whole tile
//                 rows and columns are skipped once finished;
//   scalars       one more warp forms the next norm, tau and scale meanwhile:
//                 nothing before the next vector phase needs them, so their
//                 square root, reciprocals and sums stay off the step's chain;
//   publish       A x and the head row to every CTA of the cluster (asynchronous
//                 stores that complete an mbarrier there: no cluster barrier and
//                 no flush of the reflector's global stores in a step), and from
//                 one more warp the CTA's share of x^H A x (v^H A v = A_hh +
//                 2 Re(scale (A x)_h) + |scale|^2 x^H A x gives the real
//                 alpha = -|tau|^2 v^H A v / 2).
constexpr int kClusterCtas = 16;    // non-portable cluster size
constexpr int kClusterOrder = 256;  // the largest tile without spills (8 x 2); 10 x 3 for 320 ran at 3.3 us a step
constexpr int kPassWarps = 8;
constexpr int kColumnLanes = 8;     // lanes over columns; the other 4 over rows
constexpr int kRowGroups = kPassWarps * (32 / kColumnLanes);
constexpr int kScalarWarp = kPassWarps, kShareWarp = kPassWarps + 1;
constexpr int kClusterThreads = 32 * (kPassWarps + 2);

struct ClusterArgs {
  const Cx<double>* a;  // m x m, leading dimension ld
  long long ld;
  int m;
  double* d;
  double* e;
  Cx<double>* tau;
  Cx<double>* reflectors;  // column j holds v_j in rows j+1.., leading dimension ld
  unsigned int* error;     // set when an exchange does not complete in time
};

// Position of vector entry c: one pad per 16 entries, so that a CTA's own
// columns (stride 16) fall into different banks.
__host__ __device__ constexpr int padded(int c) { return c + (c >> 4); }

template <int RT, int CT>
constexpr std::size_t cluster_smem() {
  return sizeof(Cx<double>) * (7 * static_cast<std::size_t>(padded(kRowGroups * RT)) +
                               (kPassWarps + 1) * kColumnLanes * CT + 4 + kClusterCtas);
}

__device__ __forceinline__ unsigned cluster_address(const void* local, int rank) {
  unsigned remote;
  const unsigned own = static_cast<unsigned>(__cvta_generic_to_shared(local));
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(own), "r"(rank));
  return remote;
}
// Asynchronous stores to a CTA of the cluster; their bytes count towards the
// phase of the mbarrier at `barrier` in the same CTA.
__device__ __forceinline__ void cluster_store(unsigned address, Cx<double> v, unsigned barrier) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(address),
               "d"(v.re), "d"(v.im), "r"(barrier)
               : "memory");
}
__device__ __forceinline__ void cluster_store(unsigned address, double v, unsigned barrier) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(address), "d"(v),
               "r"(barrier)
               : "memory");
}
// Waits for the phase `parity` of a local mbarrier; false after the time limit.
__device__ __forceinline__ bool exchange_wait(unsigned barrier, unsigned parity) {
  unsigned long long start = 0;
  for (int spins = 0;; ++spins) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(barrier), "r"(parity)
        : "memory");
    if (done) return true;
    if ((spins & 255) == 255) {
      const unsigned long long now = global_ns();
      if (!start) start = now;
      else if (now - start > kWaitNs) return false;
    }
  }
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int RT, int CT>
__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kClusterThreads, 1)
    tridiagonalize_cluster_kernel(ClusterArgs t) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int C = kClusterCtas, CL = kColumnLanes;
  constexpr int L = kRowGroups * RT, PL = padded(L), COLS = CL * CT;
  static_assert(RT % 2 == 0 && kRowGroups % C == 0 && L <= C * COLS && L <= 32 * kPassWarps,
                "every column has a slot, every row a thread of the pass's warps");
  const int m = t.m, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned rank_;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank_));
  const int rank = static_cast<int>(rank_);
  Cx<double>* abuf = reinterpret_cast<Cx<double>*>(smem_raw);  // A x: [2][PL], by step parity
  Cx<double>* hbuf = abuf + 2 * PL;                            // head row: [2][PL]
  Cx<double>* vs = hbuf + 2 * PL;
  Cx<double>* ws = vs + PL;
  Cx<double>* xs = ws + PL;
  Cx<double>* red = xs + PL;                  // [kPassWarps][COLS]
  Cx<double>* heads = red + kPassWarps * COLS;  // head row at own columns
  Cx<double>* pick = heads + COLS;            // entry below the head
  Cx<double>* scalars = pick + 1;             // tau, scale
  double* shares = reinterpret_cast<double*>(scalars + 2);  // x^H A x of each CTA's columns: [2][C]
  unsigned long long* arrived = reinterpret_cast<unsigned long long*>(shares + 2 * C);  // mbarriers, by step parity

  for (int i = tid; i < 7 * PL; i += kClusterThreads) abuf[i] = Cx<double>{0.0, 0.0};
  const int cl = lane % CL, rg = warp * (32 / CL) + lane / CL;
  Cx<double> y[RT][CT];
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int k = 0; k < CT; ++k) {
      const int r = i * kRowGroups + rg, c = rank + C * (cl + CL * k);
      y[i][k] = warp < kPassWarps && r < m && c < m ? t.a[r + static_cast<long long>(c) * t.ld] : Cx<double>{0.0, 0.0};
    }
  // Publish: thread (column pq, part ps) sums partial ps, and stores the sum to CTAs ps and ps + 8.
  const int pq = warp * (32 / kPassWarps) + lane / kPassWarps, ps = lane % kPassWarps;
  const unsigned remote0 = cluster_address(smem_raw, ps), remote1 = cluster_address(smem_raw, ps + kPassWarps);
  const unsigned remote_lane = cluster_address(smem_raw, lane % C);
  auto offset = [&](const void* p) {
    return static_cast<unsigned>(static_cast<const unsigned char*>(p) - smem_raw);
  };
  // A step's exchange is complete when its bytes, the arrival that announces them and the
  // scalars' arrival are in.
  if (tid == 0) {
    for (int i = 0; i < 2; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;" ::"r"(
                       static_cast<unsigned>(__cvta_generic_to_shared(arrived + i)))
                   : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  const unsigned barriers = static_cast<unsigned>(__cvta_generic_to_shared(arrived));
  const int padded_rg = padded(rg);
  const int pairs_end = (m + 2 * kRowGroups - 1) / (2 * kRowGroups), cols_end = (m + C * CL - 1) / (C * CL);
  bool alive = true;
  // No CTA of the cluster writes into one that has not started.
  cluster_barrier();

  Cx<double> x{0.0, 0.0};  // row tid of the current column below its head
  for (int j = -1; j < m - 1; ++j) {
    const int par = j & 1, next = par ^ 1, h = j + 1;
    const bool last = j == m - 2;
    // The exchange of step j - 1 (the u-th use of this parity's barrier, from 0: phase u & 1).
    if (j >= 0 && alive) {
      alive = exchange_wait(barriers + 8 * par, (j >> 1) & 1);
      if (!alive && lane == 0) atomicOr(t.error, 2u);
    }
    if (warp < kPassWarps && (warp + 1) * 32 > j) {  // a warp with live rows (or just finished ones)
      Cx<double> tau{0.0, 0.0}, scale{0.0, 0.0}, head_w{0.0, 0.0};
      double alpha = 0.0;
      const Cx<double>* ab = abuf + par * PL;
      const Cx<double>* hb = hbuf + par * PL;
      if (j >= 0) {
        tau = scalars[0];
        scale = scalars[1];
        double tree[C];
#pragma unroll
        for (int i = 0; i < C; ++i) tree[i] = shares[par * C + i];
#pragma unroll
        for (int o = C / 2; o > 0; o >>= 1)
#pragma unroll
          for (int i = 0; i < o; ++i) tree[i] += tree[i + o];
        const Cx<double> ah = ab[padded(h)], hh = hb[padded(h)];
        const double vav = fma(scale.re * scale.re + scale.im * scale.im, tree[0],
                               fma(2.0, scale.re * ah.re - scale.im * ah.im, hh.re));
        alpha = (-0.5 * (tau.re * tau.re + tau.im * tau.im)) * vav;
        head_w = cmulz(tau, cadd(cconj(hh), cmulz(scale, ah)));
        head_w.re += alpha;  // v[h] = 1
        head_w.im = -head_w.im;
      }
      const int r = tid;
      if (r < m) {
        Cx<double> col{0.0, 0.0}, v{0.0, 0.0}, w{0.0, 0.0};
        if (j < 0) {
          col = t.a[r];
        } else if (r >= h) {
          const Cx<double> hr = cconj(hb[padded(r)]);
          v = r == h ? Cx<double>{1.0, 0.0} : cmulz(x, scale);
          w = cmulz(tau, cadd(hr, cmulz(scale, ab[padded(r)])));
          w.re += alpha * v.re;
          w.im += alpha * v.im;
          col = csub(hr, cadd(cmulz(v, head_w), w));
          if (rank == (j & (C - 1))) t.reflectors[r + static_cast<long long>(j) * t.ld] = v;
        }
        if (r == h && rank == 0) t.d[h] = col.re;
        if (r == h + 1) pick[0] = col;
        x = r > h + 1 ? col : Cx<double>{0.0, 0.0};
        vs[padded(r)] = v;
        ws[padded(r)] = w;
        xs[padded(r)] = x;
      }
    }
    if (last) break;
    __syncthreads();

    if (warp == kScalarWarp) {
      double re2 = 0.0, im2 = 0.0;
#pragma unroll 4
      for (int r = lane; r < L; r += 32) {  // zeros outside the column
        const Cx<double> xr = xs[padded(r)];
        re2 += xr.re * xr.re;
        im2 += xr.im * xr.im;
      }
      double xnorm2 = re2 + im2;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) xnorm2 += __shfl_xor_sync(0xffffffffu, xnorm2, o);
      const Reflector f = make_reflector(lane, pick[0], xnorm2);
      if (lane == 0) {
        scalars[0] = f.tau;
        scalars[1] = f.scale;
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(barriers + 8 * next) : "memory");
        if (rank == 0) {
          t.e[h] = f.beta;
          t.tau[h] = f.tau;
        }
      }
    } else if (warp == kShareWarp) {
      // 32 bytes of each live column and every CTA's share.
      if (lane == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(barriers + 8 * next),
                     "r"(32 * (m - 1 - h) + 8 * C)
                     : "memory");
      asm volatile("bar.sync 1, %0;" ::"n"(32 * (kPassWarps + 1)) : "memory");
      double share = 0.0;
      if (lane < COLS) {
        Cx<double> sum[kPassWarps];
#pragma unroll
        for (int w = 0; w < kPassWarps; ++w) sum[w] = red[w * COLS + lane];
        const int c = rank + C * lane;
        const Cx<double> xc = c < L ? xs[padded(c)] : Cx<double>{0.0, 0.0};
#pragma unroll
        for (int o = kPassWarps / 2; o > 0; o >>= 1)
#pragma unroll
          for (int w = 0; w < o; ++w) sum[w] = cadd(sum[w], sum[w + o]);
        share = sum[0].re * xc.re + sum[0].im * xc.im;
      }
#pragma unroll
      for (int o = COLS > 16 ? 16 : COLS > 8 ? 8 : 4; o > 0; o >>= 1) share += __shfl_xor_sync(0xffffffffu, share, o);
      if (COLS <= 16) share = __shfl_sync(0xffffffffu, share, 0);
      if (lane < C) cluster_store(remote_lane + offset(shares + next * C + rank), share, remote_lane + offset(arrived + next));
    } else {
      // Live tile rows, two at a time (four independent chains of multiply-adds), and columns.
      const int first_pair = (h + 1) / (2 * kRowGroups), first_col = (h + 1) / (C * CL);
      const int head_pair = rg == (h + 1) % kRowGroups ? first_pair : -1;
      const bool head_second = (h + 1) / kRowGroups & 1;
#pragma unroll
      for (int k = 0; k < CT; ++k) {
        Cx<double> acc[2] = {};
        if (k >= first_col && k < cols_end) {
          const int c = rank + C * (cl + CL * k);
          const Cx<double> none{0.0, 0.0};  // slots past the tile's order
          const Cx<double> wc = c < L ? cconj(ws[padded(c)]) : none, vc = c < L ? cconj(vs[padded(c)]) : none;
#pragma unroll
          for (int i = 0; i < RT; i += 2) {
            if (i / 2 < first_pair || i / 2 >= pairs_end) continue;
            Cx<double> v[2], w[2], xr[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int at = padded((i + u) * kRowGroups) + padded_rg;
              v[u] = vs[at];
              w[u] = ws[at];
              xr[u] = xs[at];
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              Cx<double> z = y[i + u][k];
              z.re = fma(-v[u].re, wc.re, fma(v[u].im, wc.im, fma(-w[u].re, vc.re, fma(w[u].im, vc.im, z.re))));
              z.im = fma(-v[u].re, wc.im, fma(-v[u].im, wc.re, fma(-w[u].re, vc.im, fma(-w[u].im, vc.re, z.im))));
              y[i + u][k] = z;
              acc[u] = cadd(acc[u], cdot1(z, xr[u]));
            }
            if (i / 2 == head_pair) heads[cl + CL * k] = head_second ? y[i + 1][k] : y[i][k];
          }
        }
        Cx<double> sum = cadd(acc[0], acc[1]);
#pragma unroll
        for (int o = CL; o < 32; o <<= 1) {
          sum.re += __shfl_xor_sync(0xffffffffu, sum.re, o);
          sum.im += __shfl_xor_sync(0xffffffffu, sum.im, o);
        }
        if (lane < CL) red[warp * COLS + lane + CL * k] = sum;
      }
      // The pass's and the share's warps: the scalars are not needed yet.
      asm volatile("bar.sync 1, %0;" ::"n"(32 * (kPassWarps + 1)) : "memory");
      if (warp * (32 / kPassWarps) < COLS) {
        Cx<double> sum = red[ps * COLS + pq];
#pragma unroll
        for (int o = kPassWarps / 2; o > 0; o >>= 1) {
          sum.re += __shfl_xor_sync(0xffffffffu, sum.re, o);
          sum.im += __shfl_xor_sync(0xffffffffu, sum.im, o);
        }
        const int c = rank + C * pq;
        if (c > h && c < m) {
          const Cx<double> head = heads[pq];
          const unsigned to_a = offset(abuf + next * PL + padded(c)), to_h = offset(hbuf + next * PL + padded(c));
          const unsigned bar = offset(arrived + next);
          cluster_store(remote0 + to_a, sum, remote0 + bar);
          cluster_store(remote1 + to_a, sum, remote1 + bar);
          cluster_store(remote0 + to_h, head, remote0 + bar);
          cluster_store(remote1 + to_h, head, remote1 + bar);
        }
      }
    }
  }
  // No CTA leaves while another may still read or write its shared memory. After
  // an exchange that ran out of time, stores that no CTA waited for may still be on
  // their way: 20 us lets them land.
  cluster_barrier();
  if (tid == 0 && *reinterpret_cast<volatile unsigned int*>(t.error) != 0u)
    for (const unsigned long long start = global_ns(); global_ns() - start < 20000;) {
    }
}

struct ColumnArgs {
  const Cx<double>* a;
  int m, grid, cpc;
  double* d;
  double* e;
  Cx<double>* tau;
  Cx<double>* reflectors;  // m x m, column j holds v_j in rows j+1..m-1
  Cx<double>* colbuf;      // 2 x m
  Cx<double>* pbuf;        // 2 x m
  Cx<double>* dotbuf;      // 2 x grid
  unsigned int* arrive;
  unsigned int* error;  // set when a barrier wait runs out; every CTA then returns
};

// Reflector scalars of one step, formed redundantly by every thread from the
// same shared inputs (so every thread holds equal values).
struct ColumnReflector {
  Cx<double> tau, scale;
  double beta;
  bool trivial;
};

__device__ __forceinline__ ColumnReflector make_column_reflector(Cx<double> alpha, double xnorm2) {
  ColumnReflector h;
  if (xnorm2 == 0.0 && alpha.im == 0.0) {
    h.trivial = true;
    h.tau = Cx<double>{0.0, 0.0};
    h.beta = alpha.re;
    h.scale = Cx<double>{0.0, 0.0};
  } else {
    const double beta = -copysign(sqrt(alpha.re * alpha.re + alpha.im * alpha.im + xnorm2), alpha.re);
    h.trivial = false;
    h.tau = Cx<double>{(beta - alpha.re) / beta, -alpha.im / beta};
    h.beta = beta;
    // 1 / (alpha - beta)
    const double dr = alpha.re - beta, di = alpha.im, den = dr * dr + di * di;
    h.scale = Cx<double>{dr / den, -di / den};
  }
  return h;
}

// The reduction of Reduction::Columns, any order up to kRowsPerThread *
// kTridiagThreads in one cooperative launch: rows r = tid + kTridiagThreads k of
// the reflector and rank-2 vectors in registers, own columns c = cta + G s in
// shared memory. Step j+1's reflector is formed from the published column
// before step j's rank-2 update, so the update of each own column and its
// product with the next reflector share one pass; a step publishes p = tau A v
// and the column after next. Per step: one CTA barrier for the next column's
// norm, one for the column products, and the grid barrier: 7.3 to 9.3 us, the
// norm, the square root and the divisions behind the grid barrier.
__global__ void __launch_bounds__(kTridiagThreads, 1) tridiagonalize_columns_kernel(ColumnArgs t) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int R = kRowsPerThread;
  const int m = t.m, G = t.grid, cpc = t.cpc, cta = blockIdx.x, tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  Cx<double>* cols = reinterpret_cast<Cx<double>*>(smem_raw);
  Cx<double>* red = cols + static_cast<long long>(cpc) * m;  // kTridiagWarps x kMaxCpc column-product partials
  Cx<double>* colv = red + kTridiagWarps * kMaxCpc;                  // 2 x kMaxCpc: v at own columns, by step parity
  Cx<double>* colw = colv + 2 * kMaxCpc;                      // kMaxCpc: w at own columns
  Cx<double>* pick = colw + kMaxCpc;                          // alpha (row jc+1), diagonal (row jc)
  double* nrm = reinterpret_cast<double*>(pick + 2);          // kTridiagWarps norm partials
  __shared__ int ok;

  int slot_of_row[R];
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const int r = tid + k * kTridiagThreads;
    slot_of_row[k] = (r < m && r >= cta && (r - cta) % G == 0) ? (r - cta) / G : -1;
  }
  for (int s = 0; s < cpc; ++s) {
    const int c = cta + s * G;
    if (c < m)
      for (int r = tid; r < m; r += kTridiagThreads) cols[static_cast<long long>(s) * m + r] = t.a[r + static_cast<long long>(c) * m];
  }

  Cx<double> v[R], w[R], vn[R], col[R];
  ColumnReflector cur, next;

  // Reflector of column jc from col[] (rows >= jc): vn[] for rows >= jc+1,
  // v at own columns into colv[jc & 1], and CTA 0's outputs. Contains the
  // step's first CTA barrier (after which colw, written before it, is visible).
  auto reflect = [&](int jc) -> ColumnReflector {
    double part = 0.0;
#pragma unroll
    for (int k = 0; k < R; ++k) {
      const int r = tid + k * kTridiagThreads;
      if (r < m && r >= jc + 2) part += col[k].re * col[k].re + col[k].im * col[k].im;
      if (r == jc + 1) pick[0] = col[k];
      if (r == jc) pick[1] = col[k];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if (lane == 0) nrm[warp] = part;
    __syncthreads();
    double xnorm2 = 0.0;
#pragma unroll
    for (int q = 0; q < kTridiagWarps; ++q) xnorm2 += nrm[q];
    const ColumnReflector h = make_column_reflector(pick[0], xnorm2);
    if (cta == 0 && tid == 0) {
      t.d[jc] = pick[1].re;
      t.e[jc] = h.beta;
      t.tau[jc] = h.tau;
    }
    Cx<double>* cv = colv + (jc & 1) * kMaxCpc;
#pragma unroll
    for (int k = 0; k < R; ++k) {
      const int r = tid + k * kTridiagThreads;
      Cx<double> vr{0.0, 0.0};
      if (r == jc + 1) vr = Cx<double>{1.0, 0.0};
      else if (r > jc + 1 && r < m && !h.trivial) vr = cmulz(col[k], h.scale);
      vn[k] = vr;
      if (cta == 0 && r > jc && r < m) t.reflectors[r + static_cast<long long>(jc) * m] = vr;
      if (slot_of_row[k] >= 0) cv[slot_of_row[k]] = vr;
    }
    return h;
  };

  // Column products conj(A(:,c)) . vn over the CTA (acc), then p = tau A v at
  // own columns c > jc, the CTA share of p^H v, and column jc+1 published.
  auto publish = [&](int jc, const ColumnReflector& h, Cx<double> (&acc)[kMaxCpc]) {
#pragma unroll
    for (int q = 0; q < kMaxCpc; ++q) {
      if (q < cpc) {
        double re = acc[q].re, im = acc[q].im;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          re += __shfl_xor_sync(0xffffffffu, re, o);
          im += __shfl_xor_sync(0xffffffffu, im, o);
        }
        if (lane == 0) red[warp * kMaxCpc + q] = Cx<double>{re, im};
      }
    }
    __syncthreads();
    if (warp == 0) {
      Cx<double> dot{0.0, 0.0};
      const int c = cta + lane * G;
      if (lane < cpc && c > jc && c < m) {
        Cx<double> s{0.0, 0.0};
        for (int q = 0; q < kTridiagWarps; ++q) s = cadd(s, red[q * kMaxCpc + lane]);
        const Cx<double> p = cmulz(h.tau, s);
        t.pbuf[static_cast<long long>(jc & 1) * m + c] = p;
        dot = cdot1(p, colv[(jc & 1) * kMaxCpc + lane]);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        dot.re += __shfl_xor_sync(0xffffffffu, dot.re, o);
        dot.im += __shfl_xor_sync(0xffffffffu, dot.im, o);
      }
      if (lane == 0) t.dotbuf[static_cast<long long>(jc & 1) * G + cta] = dot;
    }
    // Column jc+1 (updates 0..jc-1 applied) for step jc+1.
    if (jc + 1 < m && (jc + 1) % G == cta) {
      const long long slot = (jc + 1) / G;
      Cx<double>* dst = t.colbuf + static_cast<long long>((jc + 1) & 1) * m;
      for (int r = jc + 1 + tid; r < m; r += kTridiagThreads) dst[r] = cols[slot * m + r];
    }
  };

  // Step 0: reflector of column 0, p_0 over own columns, column 1 published.
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const int r = tid + k * kTridiagThreads;
    col[k] = r < m ? t.a[r] : Cx<double>{0.0, 0.0};
  }
  __syncthreads();  // own columns in shared memory
  cur = reflect(0);
#pragma unroll
  for (int k = 0; k < R; ++k) v[k] = vn[k];
  {
    Cx<double> acc[kMaxCpc];
#pragma unroll
    for (int q = 0; q < kMaxCpc; ++q) {
      acc[q] = Cx<double>{0.0, 0.0};
      const int c = cta + q * G;
      if (q >= cpc || c < 1 || c >= m) continue;
      const Cx<double>* a = cols + static_cast<long long>(q) * m;
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const int r = tid + k * kTridiagThreads;
        if (r >= 1 && r < m) acc[q] = cadd(acc[q], cdot1(a[r], v[k]));
      }
    }
    publish(0, cur, acc);
  }
  __syncthreads();  // the published column comes from every warp
  if (!grid_barrier(t.arrive, t.error, static_cast<unsigned int>(G), &ok)) return;

  for (int j = 0; j < m - 1; ++j) {
    const bool last = j == m - 2;
    // All of this step's global reads first (one round of L2 latency): p on
    // own rows, column j+1, p at own columns and at row j+1, the CTA shares
    // of p^H v (every warp sums them in the same order).
    const double2* pb = reinterpret_cast<const double2*>(t.pbuf + static_cast<long long>(j & 1) * m);
    const double2* cb = reinterpret_cast<const double2*>(t.colbuf + static_cast<long long>((j + 1) & 1) * m);
    const double2* db = reinterpret_cast<const double2*>(t.dotbuf + static_cast<long long>(j & 1) * G);
    const double2 zero2 = make_double2(0.0, 0.0);
    double2 pq[R], cq[R], shares[kMaxShares];
#pragma unroll
    for (int k = 0; k < R; ++k) {
      const int r = tid + k * kTridiagThreads;
      const bool row = r > j && r < m;
      pq[k] = (row && !cur.trivial) ? __ldcg(pb + r) : zero2;
      cq[k] = (row && !last) ? __ldcg(cb + r) : zero2;
    }
    const int own_c = cta + tid * G;
    const bool own_w = !cur.trivial && tid < cpc && own_c > j && own_c < m;
    const double2 pc = own_w ? __ldcg(pb + own_c) : zero2;
    const double2 ph = cur.trivial ? zero2 : __ldcg(pb + j + 1);
#pragma unroll
    for (int i = 0; i < kMaxShares; ++i) {
      const int g = lane + 32 * i;
      shares[i] = (!cur.trivial && g < G) ? __ldcg(db + g) : zero2;
    }
    Cx<double> sum{0.0, 0.0};
#pragma unroll
    for (int i = 0; i < kMaxShares; ++i) sum = cadd(sum, Cx<double>{shares[i].x, shares[i].y});
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sum.re += __shfl_xor_sync(0xffffffffu, sum.re, o);
      sum.im += __shfl_xor_sync(0xffffffffu, sum.im, o);
    }
    const Cx<double> alpha = cmulz(Cx<double>{-0.5 * cur.tau.re, -0.5 * cur.tau.im}, sum);
    // w = p + alpha v on own rows; w at own columns for the update; w[j+1] (v[j+1] = 1).
#pragma unroll
    for (int k = 0; k < R; ++k) {
      const int r = tid + k * kTridiagThreads;
      w[k] = (r > j && r < m && !cur.trivial) ? cadd(Cx<double>{pq[k].x, pq[k].y}, cmulz(alpha, v[k]))
                                               : Cx<double>{0.0, 0.0};
      col[k] = Cx<double>{cq[k].x, cq[k].y};
    }
    const Cx<double> head_w = cur.trivial ? Cx<double>{0.0, 0.0} : cadd(Cx<double>{ph.x, ph.y}, alpha);
    if (own_w) colw[tid] = cadd(Cx<double>{pc.x, pc.y}, cmulz(alpha, colv[(j & 1) * kMaxCpc + tid]));

    // Step j+1's reflector from column j+1 with update j applied.
    if (!last) {
      const Cx<double> hw = cconj(head_w);
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const int r = tid + k * kTridiagThreads;
        if (r > j && r < m) col[k] = csub(col[k], cadd(cmulz(v[k], hw), w[k]));
      }
      next = reflect(j + 1);
    } else {
      __syncthreads();  // colw visible
    }

    // Update j on own columns c > j; p_{j+1} partial sums over rows/columns > j+1.
    Cx<double> acc[kMaxCpc];
#pragma unroll
    for (int q = 0; q < kMaxCpc; ++q) {
      acc[q] = Cx<double>{0.0, 0.0};
      const int c = cta + q * G;
      if (q >= cpc || c <= j || c >= m) continue;
      const Cx<double> wc = cconj(colw[q]), vc = cconj(colv[(j & 1) * kMaxCpc + q]);
      Cx<double>* a = cols + static_cast<long long>(q) * m;
      const bool dot_column = !last && c > j + 1;
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const int r = tid + k * kTridiagThreads;
        if (r > j && r < m) {
          Cx<double> x = a[r];
          if (!cur.trivial) {
            x = csub(x, cadd(cmulz(v[k], wc), cmulz(w[k], vc)));
            a[r] = x;
          }
          if (dot_column && r > j + 1) acc[q] = cadd(acc[q], cdot1(x, vn[k]));
        }
      }
    }
    if (last) break;
    publish(j + 1, next, acc);
    __syncthreads();
    if (!grid_barrier(t.arrive, t.error, static_cast<unsigned int>(G) * static_cast<unsigned int>(j + 2), &ok))
      return;
    cur = next;
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = vn[k];
  }
  __syncthreads();
  if ((m - 1) % G == cta && tid == 0) t.d[m - 1] = cols[static_cast<long long>((m - 1) / G) * m + m - 1].re;
}

// Number of eigenvalues of the tridiagonal (d, e) below x: sign changes of
// the Sturm sequence p_0 = 1, p_1 = d_0 - x, p_i = (d_{i-1} - x) p_{i-1} -
// e_{i-2}^2 p_{i-2}, kept in range by exact power-of-two rescaling. A p_i
// below pivmin |p_{i-1}| counts as a sign change (the q = -pivmin convention
// of the quotient form q_i = p_i / p_{i-1}).
template <int P>
__device__ void sturm_counts(const double* d, const double* e2, int m, const double (&x)[P], double pivmin,
                             int (&count)[P]) {
  double p0[P], p1[P];
#pragma unroll
  for (int q = 0; q < P; ++q) {
    p0[q] = 1.0;
    p1[q] = d[0] - x[q];
    if (fabs(p1[q]) <= pivmin) p1[q] = -pivmin;
    count[q] = p1[q] < 0.0;
  }
  for (int i = 1; i < m; ++i) {
    const double di = d[i], ei = e2[i - 1];
#pragma unroll
    for (int q = 0; q < P; ++q) {
      double p2 = fma(di - x[q], p1[q], -ei * p0[q]);
      if (fabs(p2) <= pivmin * fabs(p1[q])) p2 = -pivmin * p1[q];
      count[q] += (p2 < 0.0) != (p1[q] < 0.0);
      p0[q] = p1[q];
      p1[q] = p2;
    }
    // Exact rescaling by 2^-400 / 2^400 every fourth step: a step grows the
    // sequence by far less than 2^100 here, so nothing leaves the exponent
    // range in between, and power-of-two scaling changes no sign or ratio.
    if ((i & 3) == 0) {
#pragma unroll
      for (int q = 0; q < P; ++q) {
        const double mag = fabs(p1[q]);
        const double f = mag > 0x1p+400 ? 0x1p-400 : (mag < 0x1p-400 ? 0x1p+400 : 1.0);
        p0[q] *= f;
        p1[q] *= f;
      }
    }
  }
}

// One warp per wanted eigenvalue; 32 x P points per round (P per lane).
template <int P>
__global__ void bisect_kernel(const double* __restrict__ d, const double* __restrict__ e, int m, int wanted,
                              double* __restrict__ values) {
  extern __shared__ double sm[];
  double* sd = sm;
  double* se2 = sm + m;
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    sd[i] = d[i];
    if (i + 1 < m) se2[i] = e[i] * e[i];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int k = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  if (k >= wanted) return;
  double lo = DBL_MAX, hi = -DBL_MAX, emax = 0.0;
  for (int i = lane; i < m; i += 32) {
    const double left = i > 0 ? fabs(e[i - 1]) : 0.0, right = i + 1 < m ? fabs(e[i]) : 0.0;
    lo = fmin(lo, sd[i] - left - right);
    hi = fmax(hi, sd[i] + left + right);
    if (i + 1 < m) emax = fmax(emax, se2[i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    emax = fmax(emax, __shfl_xor_sync(0xffffffffu, emax, o));
  }
  const double pivmin = DBL_MIN * fmax(1.0, emax);
  const double tnorm = fmax(fabs(lo), fabs(hi));  // Gershgorin bound of the spectrum
  const double pad = 4.0 * DBL_EPSILON * tnorm + pivmin;
  lo -= pad;
  hi += pad;
  // Absolute tolerance of the matrix scale (LAPACK dstebz's default abstol,
  // eps * max(|gl|, |gu|)), beside the relative one: eigenvalues near zero
  // stop at eps * |T| instead of running every round.
  const double atol = DBL_EPSILON * tnorm;
  // P points per lane trade rounds (53 bits / log2(32 P + 1)) for the length of
  // a Sturm step's chain: 0.252 ms at order 640 with 320 values and 0.496 at
  // 1280 with P = 2, 0.332 and 0.654 with P = 4 (Reduction::Columns). The
  // interval that is left, and with it the eigenvalue's last bits, depends on P.
  for (int round = 0; round < 64; ++round) {
    const double width = hi - lo;
    if (width <= 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)) || width <= atol || width <= pivmin) break;
    const double step = width / (32 * P + 1);
    // point q of lane l is lo + (q * 32 + l + 1) step: increasing over (q, l);
    // the lane's P Sturm sequences run interleaved.
    double x[P];
    int counts[P];
#pragma unroll
    for (int q = 0; q < P; ++q) x[q] = lo + (q * 32 + lane + 1) * step;
    sturm_counts<P>(sd, se2, m, x, pivmin, counts);
    unsigned masks[P];
#pragma unroll
    for (int q = 0; q < P; ++q) masks[q] = __ballot_sync(0xffffffffu, counts[q] > k);
    int above = -1;  // first point index with count > k
#pragma unroll
    for (int q = P - 1; q >= 0; --q)
      if (masks[q]) above = q * 32 + __ffs(masks[q]) - 1;
    double new_lo = lo, new_hi = hi;
    if (above >= 0) new_hi = lo + (above + 1) * step;
    if (above != 0) new_lo = lo + (above < 0 ? 32 * P : above) * step;
    if (new_lo == lo && new_hi == hi) break;
    lo = new_lo;
    hi = new_hi;
  }
  if (lane == 0) values[k] = 0.5 * (lo + hi);
}

__device__ __forceinline__ double start_entry(int k, int i) {
  unsigned long long z = (static_cast<unsigned long long>(k) << 32) ^ static_cast<unsigned long long>(i) ^
                         0x9e3779b97f4a7c15ULL;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  z ^= z >> 31;
  return static_cast<double>(z >> 11) * (2.0 / 9007199254740992.0) - 1.0;
}

// One thread per wanted eigenvalue, kInvitThreads threads per CTA, each with
// its LU factors and vector in shared memory: reciprocal pivots, the two U
// superdiagonals, multipliers, z and pivot flags (bytes); two solves from a
// start vector of its own. Clusters are orthonormalised afterwards
// (cluster_orthonormalize_kernel).
__global__ void inverse_iteration_kernel(const double* __restrict__ d, const double* __restrict__ e, int m, int wanted,
                                         const double* __restrict__ values, double* __restrict__ zt) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  double* base = reinterpret_cast<double*>(smem_raw) + static_cast<long long>(threadIdx.x) * 5 * m;
  double* rinv = base;
  double* u1 = base + m;
  double* u2 = base + 2 * m;
  double* mult = base + 3 * m;
  double* z = base + 4 * m;
  unsigned char* piv =
      reinterpret_cast<unsigned char*>(reinterpret_cast<double*>(smem_raw) + static_cast<long long>(blockDim.x) * 5 * m) +
      static_cast<long long>(threadIdx.x) * m;
  if (k >= wanted) return;
  double norm = 0.0;
  for (int i = 0; i < m; ++i) norm = fmax(norm, fabs(d[i]) + (i + 1 < m ? fabs(e[i]) : 0.0));
  const double tiny = DBL_EPSILON * fmax(norm, DBL_MIN);
  const long long W = wanted;
  {
    const int q = k;
    const double lam = values[q];
    // LU of T - lam I with partial pivoting (rows i, i+1 swapped when |sub| wins).
    double cur_d = d[0] - lam, cur_u = m > 1 ? e[0] : 0.0;
    for (int i = 0; i + 1 < m; ++i) {
      const double nd = d[i + 1] - lam, nu = i + 2 < m ? e[i + 1] : 0.0, l = e[i];
      if (fabs(cur_d) >= fabs(l)) {
        if (fabs(cur_d) < tiny) cur_d = copysign(tiny, cur_d == 0.0 ? 1.0 : cur_d);
        const double r = 1.0 / cur_d;
        rinv[i] = r;
        u1[i] = cur_u;
        u2[i] = 0.0;
        mult[i] = l * r;
        piv[i] = 0;
        cur_d = nd - mult[i] * cur_u;
        cur_u = nu;
      } else {
        const double mu = cur_d / l;
        rinv[i] = 1.0 / l;
        u1[i] = nd;
        u2[i] = nu;
        mult[i] = mu;
        piv[i] = 1;
        cur_d = cur_u - mu * nd;
        cur_u = -mu * nu;
      }
    }
    if (fabs(cur_d) < tiny) cur_d = copysign(tiny, cur_d == 0.0 ? 1.0 : cur_d);
    rinv[m - 1] = 1.0 / cur_d;
    for (int i = 0; i < m; ++i) z[i] = start_entry(q, i);
    for (int it = 0; it < 2; ++it) {
      for (int i = 0; i + 1 < m; ++i) {
        double a = z[i], b = z[i + 1];
        if (piv[i]) {
          const double tmp = a;
          a = b;
          b = tmp;
        }
        z[i] = a;
        z[i + 1] = b - mult[i] * a;
      }
      double z2 = z[m - 1] * rinv[m - 1];
      z[m - 1] = z2;
      double z1 = 0.0;
      if (m > 1) {
        z1 = (z[m - 2] - u1[m - 2] * z2) * rinv[m - 2];
        z[m - 2] = z1;
      }
      for (int i = m - 3; i >= 0; --i) {
        const double zi = (z[i] - u1[i] * z1 - u2[i] * z2) * rinv[i];
        z[i] = zi;
        z2 = z1;
        z1 = zi;
      }
      double nrm = 0.0;
      for (int i = 0; i < m; ++i) nrm += z[i] * z[i];
      const double inv = 1.0 / sqrt(nrm);
      for (int i = 0; i < m; ++i) z[i] *= inv;
    }
    for (int i = 0; i < m; ++i) zt[i * W + q] = z[i];
  }
}

// Orthonormalises the inverse-iteration vectors of each cluster of
// eigenvalues closer than kClusterTolerance of the matrix scale (chains of
// such gaps), in eigenvalue order: classical Gram-Schmidt against the earlier
// members, twice, then normalisation. One CTA per cluster (CTAs whose index
// does not start a cluster of two or more return at once); the vectors,
// found independently from distinct start vectors, span the cluster's
// invariant subspace.
__global__ void __launch_bounds__(kThreads) cluster_orthonormalize_kernel(const double* __restrict__ d,
                                                                          const double* __restrict__ e, int m,
                                                                          int wanted, const double* __restrict__ values,
                                                                          double* __restrict__ zt) {
  extern __shared__ double dots[];  // one per earlier cluster member
  __shared__ double partial[kWarps];
  const int k = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double norm = 0.0;
  for (int i = tid; i < m; i += kThreads) norm = fmax(norm, fabs(d[i]) + (i + 1 < m ? fabs(e[i]) : 0.0));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) norm = fmax(norm, __shfl_xor_sync(0xffffffffu, norm, o));
  if (lane == 0) partial[warp] = norm;
  __syncthreads();
  norm = 0.0;
  for (int w = 0; w < kWarps; ++w) norm = fmax(norm, partial[w]);
  const double cluster = kClusterTolerance * fmax(norm, DBL_MIN);
  if (k > 0 && values[k] - values[k - 1] <= cluster) return;
  int end = k;
  while (end + 1 < wanted && values[end + 1] - values[end] <= cluster) ++end;
  if (end == k) return;
  const long long W = wanted;
  for (int q = k + 1; q <= end; ++q) {
    for (int pass = 0; pass < 2; ++pass) {
      __syncthreads();
      // dots with the earlier members: warp w takes members k + w, k + w + kWarps, ...
      for (int p = k + warp; p < q; p += kWarps) {
        double s = 0.0;
        for (int i = lane; i < m; i += 32) s += zt[i * W + p] * zt[i * W + q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) dots[p - k] = s;
      }
      __syncthreads();
      for (int i = tid; i < m; i += kThreads) {
        double v = zt[i * W + q];
        for (int p = k; p < q; ++p) v -= dots[p - k] * zt[i * W + p];
        zt[i * W + q] = v;
      }
    }
    __syncthreads();
    double s = 0.0;
    for (int i = tid; i < m; i += kThreads) s += zt[i * W + q] * zt[i * W + q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) partial[warp] = s;
    __syncthreads();
    double total = 0.0;
    for (int w = 0; w < kWarps; ++w) total += partial[w];
    const double inv = 1.0 / sqrt(total);
    for (int i = tid; i < m; i += kThreads) zt[i * W + q] *= inv;
  }
}

// Compact WY factor of each block of kReflectorBlock reflectors:
// H_j0 ... H_j0+nb-1 = I - V T V^H (LAPACK zlarft, forward, columnwise),
// T upper triangular (column-major, leading dimension kReflectorBlock), from
// the block's Gram matrix G = V^H V. One CTA per block. T grows by doubling:
// two neighbouring blocks T1, T2 of order s join as
//   [T1  -T1 (G12 T2)]
//   [ 0        T2    ]
// so the factor takes six rounds of two parallel triangular products instead
// of 64 dependent columns.
__global__ void __launch_bounds__(kThreads) reflector_blocks_kernel(const Cx<double>* __restrict__ grams,
                                                                    const Cx<double>* __restrict__ tau, int m,
                                                                    Cx<double>* __restrict__ tfac) {
  constexpr int NB = kReflectorBlock, LD = NB + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cx<double>* gram = reinterpret_cast<Cx<double>*>(smem_raw);  // NB x LD, gram[a * LD + b] = G(a, b)
  Cx<double>* tmat = gram + NB * LD;                            // NB x LD
  Cx<double>* prod = tmat + NB * LD;                            // G12 T2 of every pair of a round
  const int j0 = blockIdx.x * NB;
  const int nb = min(NB, m - 1 - j0);
  const int tid = threadIdx.x;
  const Cx<double>* g = grams + static_cast<long long>(blockIdx.x) * NB * NB;
  for (int idx = tid; idx < NB * NB; idx += kThreads) {
    const int col = idx / NB, row = idx % NB;
    gram[row * LD + col] = row < nb && col < nb ? g[idx] : Cx<double>{0.0, 0.0};
    tmat[row * LD + col] = row == col && row < nb ? tau[j0 + row] : Cx<double>{0.0, 0.0};
  }
  __syncthreads();
  for (int s = 1; s < nb; s *= 2) {
    const int items = NB / 2 * s;
    for (int idx = tid; idx < items; idx += kThreads) {
      const int pair = idx / (s * s), a = idx / s % s, b = idx % s, first = pair * 2 * s, second = first + s;
      Cx<double> sum{0.0, 0.0};
      for (int c = 0; c <= b; ++c)
        sum = cadd(sum, cmulz(gram[(first + a) * LD + second + c], tmat[(second + c) * LD + second + b]));
      prod[idx] = sum;
    }
    __syncthreads();
    for (int idx = tid; idx < items; idx += kThreads) {
      const int pair = idx / (s * s), a = idx / s % s, b = idx % s, first = pair * 2 * s, second = first + s;
      Cx<double> sum{0.0, 0.0};
      for (int c = a; c < s; ++c)
        sum = cadd(sum, cmulz(tmat[(first + a) * LD + first + c], prod[pair * s * s + c * s + b]));
      tmat[(first + a) * LD + second + b] = Cx<double>{-sum.re, -sum.im};
    }
    __syncthreads();
  }
  for (int idx = tid; idx < NB * NB; idx += kThreads) {
    const int col = idx / NB, row = idx % NB;
    tfac[static_cast<long long>(blockIdx.x) * NB * NB + idx] = tmat[row * LD + col];
  }
}

// X (complex, column-major, leading dimension m) from the row-major real
// tridiagonal eigenvectors zt (m x wanted).
__global__ void complex_columns_kernel(const double* __restrict__ zt, int m, int wanted, Cx<double>* __restrict__ x) {
  const long long total = static_cast<long long>(m) * wanted;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long i = idx % m, q = idx / m;
    x[idx] = Cx<double>{zt[i * wanted + q], 0.0};
  }
}

__global__ void identity_deviation_kernel(Cx<double>* __restrict__ b, int m, unsigned long long* __restrict__ max_bits) {
  const long long total = static_cast<long long>(m) * m;
  double local = 0.0;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long i = idx % m, j = idx / m;
    Cx<double> v = b[idx];
    if (i == j) v.re -= 1.0;
    b[idx] = v;
    local = fmax(local, fmax(fabs(v.re), fabs(v.im)));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) local = fmax(local, __shfl_xor_sync(0xffffffffu, local, o));
  if ((threadIdx.x & 31) == 0) atomicMax(max_bits, static_cast<unsigned long long>(__double_as_longlong(local)));
}

// c <- I - e/2 + 3/8 c (c holds E^2 on entry)
__global__ void lowdin_second_order_kernel(const Cx<double>* __restrict__ e, Cx<double>* __restrict__ c, int m) {
  const long long total = static_cast<long long>(m) * m;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long i = idx % m, j = idx / m;
    const Cx<double> x = e[idx], y = c[idx];
    c[idx] = Cx<double>{(i == j ? 1.0 : 0.0) - 0.5 * x.re + 0.375 * y.re, -0.5 * x.im + 0.375 * y.im};
  }
}

__global__ void add_identity_kernel(Cx<double>* __restrict__ b, int m) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < m) b[i + static_cast<long long>(i) * m].re += 1.0;
}

// a <- a - (f + f^H) / 2
__global__ void lowdin_combine_kernel(Cx<double>* __restrict__ a, const Cx<double>* __restrict__ f, int m) {
  const long long total = static_cast<long long>(m) * m;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long i = idx % m, j = idx / m;
    const Cx<double> x = f[idx], y = f[j + i * m];
    a[idx] = Cx<double>{a[idx].re - 0.5 * (x.re + y.re), a[idx].im - 0.5 * (x.im - y.im)};
  }
}

int sm_count() {
  static int count = [] {
    int device = 0, value = 0;
    SDFT_CUDA(cudaGetDevice(&device));
    SDFT_CUDA(cudaDeviceGetAttribute(&value, cudaDevAttrMultiProcessorCount, device));
    return value;
  }();
  return count;
}

// Column stride of the grid kernel's shared memory.
int tridiag_rows(int m) { return static_cast<int>(ceil_div(m, kTridiagThreads)) * kTridiagThreads; }

std::size_t tridiag_smem(int m, int cpc) {
  return sizeof(Cx<double>) *
             (static_cast<std::size_t>(cpc) * tridiag_rows(m) + 2 * kMaxCpc * kTridiagWarps + 2 * kMaxCpc + 3) +
         sizeof(double) * kTridiagWarps * 32;
}

std::size_t columns_smem(int m, int cpc) {
  return sizeof(Cx<double>) * (static_cast<std::size_t>(cpc) * m + kTridiagWarps * kMaxCpc + 3 * kMaxCpc + 2) +
         sizeof(double) * kTridiagWarps;
}

constexpr std::size_t kSmemLimit = 227 * 1024;

std::size_t invit_smem(int m) { return static_cast<std::size_t>(kInvitThreads) * (5 * sizeof(double) + 1) * m; }

constexpr std::size_t kBlockSmem =
    sizeof(Cx<double>) * (2 * kReflectorBlock * (kReflectorBlock + 1) + kReflectorBlock * kReflectorBlock / 4);

}  // namespace

namespace {
// Cooperative kernels that fill every SM must not run at the same time (two
// of them could each hold part of the SMs and wait on each other's missing
// CTAs), so every solver on a device, whatever its stream, launches them in
// order on one shared stream: the caller's stream hands over with an event
// and waits for the kernel's completion event.
struct CooperativeLane {
  std::mutex mutex;
  cudaStream_t stream = nullptr;
};

CooperativeLane& cooperative_lane(int device) {
  static CooperativeLane lanes[64];
  if (device < 0 || device >= 64) throw InvalidArgument("device ordinal out of range");
  return lanes[device];
}

template <typename Args>
void cooperative_launch(void (*kernel)(Args), int grid, int threads, Args& args, std::size_t smem,
                        cudaStream_t stream) {
  allow_dynamic_smem(kernel, smem);
  int per_sm = 0;
  SDFT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
  if (per_sm < 1) throw InvalidArgument("tridiagonalization kernel cannot be resident");
  int device = 0;
  SDFT_CUDA(cudaGetDevice(&device));
  CooperativeLane& lane = cooperative_lane(device);
  cudaEvent_t ready = nullptr, done = nullptr;
  SDFT_CUDA(cudaEventCreateWithFlags(&ready, cudaEventDisableTiming));
  SDFT_CUDA(cudaEventCreateWithFlags(&done, cudaEventDisableTiming));
  try {
    std::lock_guard<std::mutex> lock(lane.mutex);
    if (!lane.stream) SDFT_CUDA(cudaStreamCreateWithFlags(&lane.stream, cudaStreamNonBlocking));
    SDFT_CUDA(cudaEventRecord(ready, stream));
    SDFT_CUDA(cudaStreamWaitEvent(lane.stream, ready, 0));
    void* params[] = {&args};
    SDFT_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(kernel), dim3(grid), dim3(threads), params, smem, lane.stream));
    SDFT_LAUNCH("cooperative tridiagonalization kernel");
    SDFT_CUDA(cudaEventRecord(done, lane.stream));
    SDFT_CUDA(cudaStreamWaitEvent(stream, done, 0));
  } catch (...) {
    cudaEventDestroy(ready);
    cudaEventDestroy(done);
    throw;
  }
  cudaEventDestroy(ready);  // released once the recorded work completes
  cudaEventDestroy(done);
}

template <int RT, int CT>
void launch_cluster(const ClusterArgs& t, cudaStream_t stream) {
  const auto kernel = tridiagonalize_cluster_kernel<RT, CT>;
  constexpr std::size_t smem = cluster_smem<RT, CT>();
  allow_dynamic_smem(kernel, smem);
  SDFT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  kernel<<<kClusterCtas, kClusterThreads, smem, stream>>>(t);
  SDFT_LAUNCH("tridiagonalize_cluster_kernel");
}

// The smallest register tile that holds the order.
void cluster_tridiagonalize(const ClusterArgs& t, cudaStream_t stream) {
  if (t.m <= 4 * kRowGroups) launch_cluster<4, 1>(t, stream);
  else launch_cluster<8, 2>(t, stream);
}
}  // namespace

int hermitian_eigen_max_order() {
  static const int order = [] {
    const int g = sm_count();
    int best = 0;
    for (int m = 2; m <= kRowsPerThread * kTridiagThreads; ++m) {
      const int grid = std::min({g, m, 32 * kMaxShares});
      const int cpc = (m + grid - 1) / grid;
      if (cpc > kMaxCpc || tridiag_smem(m, cpc) > kSmemLimit || invit_smem(m) > kSmemLimit) break;
      best = m;
    }
    return best;
  }();
  return order;
}

void hermitian_lowest(cublasHandle_t blas, Cx<double>* a, int m, int wanted, double* values, Cx<double>* vectors,
                      EigenWorkspace& ws, cudaStream_t stream, Reduction reduction) {
  if (m < 2 || wanted < 1 || wanted > m) throw InvalidArgument("invalid Hermitian eigenproblem size");
  const int grid = std::min({sm_count(), m, 32 * kMaxShares});
  const int cpc = (m + grid - 1) / grid;
  const std::size_t smem = tridiag_smem(m, cpc);
  if (m > hermitian_eigen_max_order()) throw InvalidArgument("Hermitian eigenproblem too large for the device solver");

  // Layout of the tridiagonal workspace.
  const std::size_t mm = static_cast<std::size_t>(m);
  const std::size_t bytes = sizeof(double) * 2 * mm + sizeof(Cx<double>) * (mm + mm * mm + 4 * mm + 2 * grid) + 256;
  auto* base = static_cast<unsigned char*>(ws.tridiagonal.reserve(bytes));
  auto* arrive = reinterpret_cast<unsigned int*>(base);
  auto* d = reinterpret_cast<double*>(base + 256);
  double* e = d + mm;
  auto* tau = reinterpret_cast<Cx<double>*>(e + mm);
  Cx<double>* reflectors = tau + mm;
  Cx<double>* exchange[2] = {reflectors + mm * mm, reflectors + mm * mm + 2 * mm};  // 2 x m each
  Cx<double>* shares = exchange[1] + 2 * mm;                                         // 2 x grid
  unsigned int* error_word = arrive + 1;
  SDFT_CUDA(cudaMemsetAsync(arrive, 0, 2 * sizeof(unsigned int), stream));
  // Entries above each reflector's unit element stay zero for the block products.
  SDFT_CUDA(cudaMemsetAsync(reflectors, 0, sizeof(Cx<double>) * mm * mm, stream));

  // SDFT_B200_TRACE: device times of the stages, printed after the final synchronisation.
  static const bool trace = std::getenv("SDFT_B200_TRACE") != nullptr;
  cudaEvent_t marks[6] = {};
  if (trace)
    for (auto& ev : marks) SDFT_CUDA(cudaEventCreate(&ev));
  auto mark = [&](int i) {
    if (trace) SDFT_CUDA(cudaEventRecord(marks[i], stream));
  };
  mark(0);
  if (reduction == Reduction::Columns) {
    ColumnArgs t{a, m, grid, cpc, d, e, tau, reflectors, exchange[0], exchange[1], shares, arrive, error_word};
    cooperative_launch(tridiagonalize_columns_kernel, grid, kTridiagThreads, t, columns_smem(m, cpc), stream);
  } else {
    const int tail = std::min(m, kClusterOrder), stop = m - tail;  // the cluster kernel's order, the grid kernel's reflectors
    if (stop > 0) {
      TridiagArgs t{a, m, grid, cpc, tridiag_rows(m), stop, d, e, tau, reflectors, exchange[0], exchange[1],
                    reinterpret_cast<double*>(shares), arrive, error_word};
      cooperative_launch(tridiagonalize_kernel, grid, kTridiagThreads, t, smem, stream);
    }
    const std::size_t corner = static_cast<std::size_t>(stop) * (mm + 1);
    cluster_tridiagonalize(ClusterArgs{a + corner, m, tail, d + stop, e + stop, tau + stop, reflectors + corner,
                                       error_word},
                           stream);
  }
  mark(1);

  const int warps_per_block = 4;
  const std::size_t bisect_smem = sizeof(double) * 2 * mm;
  const auto bisect = reduction == Reduction::Columns ? bisect_kernel<4> : bisect_kernel<2>;
  allow_dynamic_smem(bisect, bisect_smem);
  bisect<<<static_cast<unsigned>(ceil_div(wanted, warps_per_block)), 32 * warps_per_block, bisect_smem, stream>>>(
      d, e, m, wanted, values);
  SDFT_LAUNCH("bisect_kernel");
  mark(2);

  const int blocks = static_cast<int>(ceil_div(m - 1, kReflectorBlock));
  // The complex arrays after the real eigenvectors start on a 16-byte
  // boundary: wanted * m doubles are rounded up to an even count (an odd
  // product left them 8-byte aligned, which cuBLAS refuses for complex data).
  const std::size_t zt_doubles = (static_cast<std::size_t>(wanted) * mm + 1) & ~static_cast<std::size_t>(1);
  const std::size_t vbytes =
      sizeof(double) * zt_doubles +
      sizeof(Cx<double>) * (2 * static_cast<std::size_t>(blocks) + 2 * static_cast<std::size_t>(wanted)) *
          kReflectorBlock * kReflectorBlock;
  auto* zt = static_cast<double*>(ws.vectors.reserve(vbytes));
  auto* tfac = reinterpret_cast<Cx<double>*>(zt + zt_doubles);
  Cx<double>* grams = tfac + static_cast<std::size_t>(blocks) * kReflectorBlock * kReflectorBlock;
  Cx<double>* wtmp = grams + static_cast<std::size_t>(blocks) * kReflectorBlock * kReflectorBlock;
  Cx<double>* utmp = wtmp + static_cast<std::size_t>(wanted) * kReflectorBlock;
  const std::size_t inv_smem = invit_smem(m);
  allow_dynamic_smem(inverse_iteration_kernel, inv_smem);
  inverse_iteration_kernel<<<static_cast<unsigned>(ceil_div(wanted, kInvitThreads)), kInvitThreads, inv_smem,
                             stream>>>(d, e, m, wanted, values, zt);
  SDFT_LAUNCH("inverse_iteration_kernel");
  const std::size_t dots_smem = sizeof(double) * static_cast<std::size_t>(wanted);
  allow_dynamic_smem(cluster_orthonormalize_kernel, dots_smem);
  cluster_orthonormalize_kernel<<<static_cast<unsigned>(wanted), kThreads, dots_smem, stream>>>(d, e, m, wanted,
                                                                                                values, zt);
  SDFT_LAUNCH("cluster_orthonormalize_kernel");
  mark(3);

  // Gram blocks V_b^H V_b of the reflector blocks (zeros above each unit
  // element): one strided-batched ZGEMM over the full blocks, one for the rest.
  {
    const cuDoubleComplex one{1.0, 0.0}, zero{0.0, 0.0};
    const int full = (m - 1) / kReflectorBlock, rest = (m - 1) % kReflectorBlock;
    const long long block_stride = static_cast<long long>(kReflectorBlock) * m;
    const long long gram_stride = static_cast<long long>(kReflectorBlock) * kReflectorBlock;
    auto* v = reinterpret_cast<const cuDoubleComplex*>(reflectors);
    auto* gz = reinterpret_cast<cuDoubleComplex*>(grams);
    if (full > 0)
      check_blas(cublasZgemmStridedBatched(blas, CUBLAS_OP_C, CUBLAS_OP_N, kReflectorBlock, kReflectorBlock, m, &one,
                                           v, m, block_stride, v, m, block_stride, &zero, gz, kReflectorBlock,
                                           gram_stride, full),
                 "zgemmStridedBatched");
    if (rest > 0)
      check_blas(cublasZgemm(blas, CUBLAS_OP_C, CUBLAS_OP_N, rest, rest, m, &one, v + full * block_stride, m,
                             v + full * block_stride, m, &zero, gz + full * gram_stride, kReflectorBlock),
                 "zgemm");
  }
  allow_dynamic_smem(reflector_blocks_kernel, kBlockSmem);
  reflector_blocks_kernel<<<static_cast<unsigned>(blocks), kThreads, kBlockSmem, stream>>>(grams, tau, m, tfac);
  SDFT_LAUNCH("reflector_blocks_kernel");
  mark(4);

  // X = Q Z: blocks from the last to the first, X <- X - V (T (V^H X)) on rows > j0.
  const long long total = static_cast<long long>(m) * wanted;
  complex_columns_kernel<<<static_cast<unsigned>(std::min<long long>(ceil_div(total, 256), 148 * 8)), 256, 0,
                           stream>>>(zt, m, wanted, vectors);
  SDFT_LAUNCH("complex_columns_kernel");
  for (int b = blocks - 1; b >= 0; --b) {
    const int j0 = b * kReflectorBlock;
    const int nb = std::min(kReflectorBlock, m - 1 - j0);
    const int rows = m - 1 - j0;
    const Cx<double>* vb = reflectors + (j0 + 1) + static_cast<long long>(j0) * m;
    Cx<double>* xs = vectors + (j0 + 1);
    const Cx<double>* tb = tfac + static_cast<long long>(b) * kReflectorBlock * kReflectorBlock;
    zgemm(blas, Op::C, Op::N, nb, wanted, rows, vb, m, xs, m, wtmp, kReflectorBlock, false);
    zgemm(blas, Op::N, Op::N, nb, wanted, nb, tb, kReflectorBlock, wtmp, kReflectorBlock, utmp, kReflectorBlock, false);
    zgemm(blas, Op::N, Op::N, rows, wanted, nb, vb, m, utmp, kReflectorBlock, xs, m, true, -1.0);
  }
  mark(5);

  unsigned int error = 0;
  SDFT_CUDA(cudaMemcpyAsync(&error, error_word, sizeof(error), cudaMemcpyDeviceToHost, stream));
  SDFT_CUDA(cudaStreamSynchronize(stream));
  if (trace) {
    float ms[5];
    for (int i = 0; i < 5; ++i) SDFT_CUDA(cudaEventElapsedTime(&ms[i], marks[i], marks[i + 1]));
    std::fprintf(stderr,
                 "hermitian-lowest m=%d wanted=%d tridiagonalize=%.3fms bisect=%.3fms inverse_iteration=%.3fms "
                 "reflector_blocks=%.3fms back_transform=%.3fms\n",
                 m, wanted, ms[0], ms[1], ms[2], ms[3], ms[4]);
    for (auto& ev : marks) cudaEventDestroy(ev);
  }
  if (error) throw CudaError("tridiagonalization wait limit exceeded");
}

double identity_deviation(Cx<double>* b, int m, EigenWorkspace& ws, cudaStream_t stream) {
  auto* bits = static_cast<unsigned long long*>(ws.scalar.reserve(sizeof(unsigned long long)));
  SDFT_CUDA(cudaMemsetAsync(bits, 0, sizeof(unsigned long long), stream));
  const long long total = static_cast<long long>(m) * m;
  identity_deviation_kernel<<<static_cast<unsigned>(std::min<long long>(ceil_div(total, 256), 148 * 8)), 256, 0,
                              stream>>>(b, m, bits);
  SDFT_LAUNCH("identity_deviation_kernel");
  unsigned long long host = 0;
  SDFT_CUDA(cudaMemcpyAsync(&host, bits, sizeof(host), cudaMemcpyDeviceToHost, stream));
  SDFT_CUDA(cudaStreamSynchronize(stream));
  double value;
  std::memcpy(&value, &host, sizeof(value));
  return value;
}

void lowdin_second_order(const Cx<double>* e, Cx<double>* c, int m, cudaStream_t stream) {
  const long long total = static_cast<long long>(m) * m;
  lowdin_second_order_kernel<<<static_cast<unsigned>(std::min<long long>(ceil_div(total, 256), 148 * 8)), 256, 0,
                               stream>>>(e, c, m);
  SDFT_LAUNCH("lowdin_second_order_kernel");
}

void add_identity(Cx<double>* b, int m, cudaStream_t stream) {
  add_identity_kernel<<<static_cast<unsigned>(ceil_div(m, 256)), 256, 0, stream>>>(b, m);
  SDFT_LAUNCH("add_identity_kernel");
}

RitzSolver rr_mode() {
  static const RitzSolver mode = [] {
    const char* v = std::getenv("SDFT_B200_RR");
    if (!v || std::string(v) == "device") return RitzSolver::Device;
    if (std::string(v) == "subset") return RitzSolver::Subset;
    if (std::string(v) == "full") return RitzSolver::Full;
    throw InvalidArgument("SDFT_B200_RR must be device, subset or full");
  }();
  return mode;
}

namespace {
void check_solver(cusolverStatus_t status, const char* what) {
  if (status != CUSOLVER_STATUS_SUCCESS)
    throw CudaError(std::string("cuSOLVER error ") + std::to_string(static_cast<int>(status)) + " in " + what);
}
}  // namespace

void generalized_lowest(cublasHandle_t blas, cusolverDnHandle_t solver, Cx<double>* h, Cx<double>* s, int m,
                        int wanted, double* values, Cx<double>* vectors, EigenWorkspace& ws, RitzSolver mode,
                        cudaStream_t st, double max_deviation, double first_order_limit, Reduction reduction) {
  if (m < 1 || wanted < 1 || wanted > m) throw InvalidArgument("invalid Rayleigh-Ritz dimensions");
  const std::size_t mm = static_cast<std::size_t>(m);
  if (mode == RitzSolver::Device && m >= 2 && m <= hermitian_eigen_max_order()) {
    const double deviation = identity_deviation(s, m, ws, st);
    if (!std::isfinite(deviation)) throw NonFinite("Rayleigh-Ritz overlap is not finite");
    static const bool trace = std::getenv("SDFT_B200_TRACE") != nullptr;
    if (trace)
      std::fprintf(stderr, "rayleigh-ritz m=%d |S-I|max=%.3e path=%s\n", m, deviation,
                   deviation <= first_order_limit ? "device" : deviation <= max_deviation ? "device-loewdin2" : "cusolver");
    if (deviation <= first_order_limit) {
      // First order: H' = H - (E H + H E)/2, y -> y - E y / 2 (error O(|E|^2)).
      const bool correct = deviation > 1e-14;
      Cx<double>* f = nullptr;
      if (correct) {
        f = static_cast<Cx<double>*>(ws.product.reserve(sizeof(Cx<double>) * mm * mm));
        zgemm(blas, Op::N, Op::N, m, m, m, s, m, h, m, f, m, false);
        lowdin_combine(h, f, m, st);
      }
      hermitian_lowest(blas, h, m, wanted, values, vectors, ws, st, reduction);
      if (correct) {
        zgemm(blas, Op::N, Op::N, m, wanted, m, s, m, vectors, m, f, m, false, -0.5);
        add_block(f, m, vectors, m, m, wanted, st);
      }
      return;
    }
    if (deviation <= max_deviation) {
      // Second order: C = I - E/2 + 3/8 E^2 = S^(-1/2) + O(|E|^3); H' = C H C, y -> C y.
      auto* f = static_cast<Cx<double>*>(ws.product.reserve(sizeof(Cx<double>) * mm * mm));
      auto* c = static_cast<Cx<double>*>(ws.product2.reserve(sizeof(Cx<double>) * mm * mm));
      zgemm(blas, Op::N, Op::N, m, m, m, s, m, s, m, c, m, false);
      lowdin_second_order(s, c, m, st);
      zgemm(blas, Op::N, Op::N, m, m, m, c, m, h, m, f, m, false);
      zgemm(blas, Op::N, Op::N, m, m, m, f, m, c, m, h, m, false);
      hermitian_lowest(blas, h, m, wanted, values, vectors, ws, st, reduction);
      zgemm(blas, Op::N, Op::N, m, wanted, m, c, m, vectors, m, f, m, false);
      copy_block(f, m, vectors, m, m, wanted, st);
      return;
    }
    // Far from S-orthonormal: restore S and solve the pencil with cuSOLVER.
    add_identity(s, m, st);
  }
  auto* info = static_cast<int*>(ws.scalar.reserve(sizeof(unsigned long long) + sizeof(int))) + 2;
  int lwork = 0;
  auto* hz = reinterpret_cast<cuDoubleComplex*>(h);
  auto* sz = reinterpret_cast<cuDoubleComplex*>(s);
  const bool full = mode == RitzSolver::Full || wanted == m;
  if (full) {
    check_solver(cusolverDnZhegvd_bufferSize(solver, CUSOLVER_EIG_TYPE_1, CUSOLVER_EIG_MODE_VECTOR,
                                             CUBLAS_FILL_MODE_LOWER, m, hz, m, sz, m, values, &lwork),
                 "zhegvd_bufferSize");
    auto* work = static_cast<cuDoubleComplex*>(ws.solver_work.reserve(sizeof(cuDoubleComplex) * std::max(1, lwork)));
    check_solver(cusolverDnZhegvd(solver, CUSOLVER_EIG_TYPE_1, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, m,
                                  hz, m, sz, m, values, work, lwork, info),
                 "zhegvd");
  } else {
    int found = 0;
    check_solver(cusolverDnZhegvdx_bufferSize(solver, CUSOLVER_EIG_TYPE_1, CUSOLVER_EIG_MODE_VECTOR,
                                              CUSOLVER_EIG_RANGE_I, CUBLAS_FILL_MODE_LOWER, m, hz, m, sz, m, 0.0,
                                              0.0, 1, wanted, &found, values, &lwork),
                 "zhegvdx_bufferSize");
    auto* work = static_cast<cuDoubleComplex*>(ws.solver_work.reserve(sizeof(cuDoubleComplex) * std::max(1, lwork)));
    check_solver(cusolverDnZhegvdx(solver, CUSOLVER_EIG_TYPE_1, CUSOLVER_EIG_MODE_VECTOR, CUSOLVER_EIG_RANGE_I,
                                   CUBLAS_FILL_MODE_LOWER, m, hz, m, sz, m, 0.0, 0.0, 1, wanted, &found, values,
                                   work, lwork, info),
                 "zhegvdx");
    if (found != wanted) throw std::runtime_error("selected generalized Ritz failed: found " + std::to_string(found));
  }
  int host_info = 0;
  SDFT_CUDA(cudaMemcpyAsync(&host_info, info, sizeof(int), cudaMemcpyDeviceToHost, st));
  SDFT_CUDA(cudaStreamSynchronize(st));
  if (host_info) throw std::runtime_error("LAPACK generalized Rayleigh-Ritz failed: info=" + std::to_string(host_info));
  if (vectors != h) copy_block(h, m, vectors, m, m, full ? m : wanted, st);
}

void lowdin_combine(Cx<double>* a, const Cx<double>* f, int m, cudaStream_t stream) {
  const long long total = static_cast<long long>(m) * m;
  lowdin_combine_kernel<<<static_cast<unsigned>(std::min<long long>(ceil_div(total, 256), 148 * 8)), 256, 0,
                          stream>>>(a, f, m);
  SDFT_LAUNCH("lowdin_combine_kernel");
}

}  // namespace sdft_b200
