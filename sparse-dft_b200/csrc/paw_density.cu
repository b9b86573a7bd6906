// One-centre occupations and the compensation charge on the device.
//
// Set-up (CompensationCharge constructor, src/paw_compensation.cpp:185-342):
// the host forms the reciprocal vectors of the keys and the distinct |G|
// shells (exact double radii, as the reference's radius cache), the device
// integrates int g_L(r) r^2 j_L(|G| r) dr on the radial mesh once per shell
// and L (Simpson weights of src/paw_compensation.cpp:51-74, spherical Bessel
// functions by the series / upward / Miller-downward recurrences of :76-114)
// and fills the compact form table F_LM(G) = 4 pi (-i)^L Y_LM(G^) I_L(|G|)
// with the real harmonics of :116-139.
//
// The arrays follow the keys in lexicographic order; results go back to the
// caller's. Phases come from per-atom tables of each axis (two complex
// products a key and atom) instead of a sincospi of the summed argument.
//
// Per call: the (L,M) moments M_a = transform . rho_a (one thread per atom and
// LM), then one thread per two G sums exp(-i G.tau_a) (F(G) . M_a) / Omega over
// the atoms in order (src/paw_compensation.cpp:508-520). Si64, f = 8 (542 369
// keys, 64 atoms), both directions: 781 -> 398 us a pair of calls, errors 1.3e-15
// -> 6.9e-16. The density sum (187 us) waits for its table
// reads: 16 of 17 cycles between issues, at 31 % warps, FP64 pipe 32 %; the
// adjoint (175 us), its keys staged, is nearer the FP64 pipe (41 %, issue 52 %).
#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>
#include <limits>
#include <unordered_map>
#include <utility>
#include <vector>

#include "operator.cuh"
#include "paw_density.cuh"

namespace sdft_b200 {

namespace {

constexpr double kPi = 3.14159265358979323846;
constexpr double kBohrPerAngstrom = 1.8897261254578281;  // CODATA convention of the reference

__device__ __forceinline__ double dot3(double ax, double ay, double az, double bx, double by, double bz) {
  return __dadd_rn(__dadd_rn(__dmul_rn(ax, bx), __dmul_rn(ay, by)), __dmul_rn(az, bz));
}

__device__ __forceinline__ Cx<double> mul_rn(Cx<double> a, Cx<double> b) {
  return {__dsub_rn(__dmul_rn(a.re, b.re), __dmul_rn(a.im, b.im)),
          __dadd_rn(__dmul_rn(a.re, b.im), __dmul_rn(a.im, b.re))};
}

// Spherical Bessel j_l(x) for 0 <= l <= 6.
__device__ double spherical_bessel(int l, double x) {
  if (fabs(x) < 0.5) {
    double term = 1.0;
    for (int k = 1; k <= l; ++k) term *= x / (2.0 * k + 1.0);
    double value = term;
    for (int k = 1; k < 30; ++k) {
      term *= -x * x / (2.0 * k * (2.0 * l + 2.0 * k + 1.0));
      value += term;
      if (fabs(term) < 1e-17 * fmax(1.0, fabs(value))) break;
    }
    return value;
  }
  if (x > l + 1.0) {
    double previous = sin(x) / x;
    if (l == 0) return previous;
    double current = sin(x) / (x * x) - cos(x) / x;
    for (int n = 1; n < l; ++n) {
      const double next = (2.0 * n + 1.0) * current / x - previous;
      previous = current;
      current = next;
    }
    return current;
  }
  constexpr int kExtra = 32;
  double j[6 + kExtra + 2];
  const int top = l + kExtra;
  for (int i = 0; i <= top + 1; ++i) j[i] = 0.0;
  j[top] = 1.0;
  for (int n = top; n >= 1; --n) {
    j[n - 1] = (2.0 * n + 1.0) * j[n] / x - j[n + 1];
    if (fabs(j[n - 1]) > 1e100)
      for (int k = n - 1; k <= top + 1; ++k) j[k] *= 1e-100;
  }
  return j[l] * ((sin(x) / x) / j[0]);
}

// Real harmonic Y_lm (m<0: sin(|m| phi), m>0: cos(m phi), no Condon-Shortley phase).
__device__ double real_harmonic(int l, int m, double qx, double qy, double qz) {
  const double radius = sqrt(dot3(qx, qy, qz, qx, qy, qz));
  if (radius < 1e-14) return l == 0 ? 1.0 / sqrt(4.0 * kPi) : 0.0;
  const double z = fmin(fmax(qz / radius, -1.0), 1.0);
  const double s = sqrt(fmax(0.0, 1.0 - z * z));
  const int order = abs(m);
  double pmm = 1.0;
  for (int k = 1; k <= order; ++k) pmm *= (2.0 * k - 1.0) * s;
  double previous = 0.0, value = pmm;
  if (l > order) {
    previous = pmm;
    value = (2.0 * order + 1.0) * z * pmm;
    for (int degree = order + 2; degree <= l; ++degree) {
      const double next = ((2.0 * degree - 1.0) * z * value - (degree + order - 1.0) * previous) / (degree - order);
      previous = value;
      value = next;
    }
  }
  const double factor = sqrt((2.0 * l + 1.0) / (4.0 * kPi) * exp(lgamma(l - order + 1.0) - lgamma(l + order + 1.0))) *
                        (order ? sqrt(2.0) : 1.0);
  const double angle = order * atan2(qy, qx);
  return factor * value * (m < 0 ? sin(angle) : cos(angle));
}

__global__ void radial_integrals_kernel(const double* __restrict__ shells, int count, int max_l,
                                        const double* __restrict__ r, const double* __restrict__ weights,
                                        const double* __restrict__ r2, int radial, double* __restrict__ integrals) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= count * (max_l + 1)) return;
  const int shell = id / (max_l + 1), L = id - shell * (max_l + 1);
  const double q = shells[shell];
  double sum = 0.0;
  for (int i = 0; i < radial; ++i)
    sum = __dadd_rn(sum, __dmul_rn(__dmul_rn(weights[i], r2[L * radial + i]), spherical_bessel(L, __dmul_rn(q, r[i]))));
  if (q < 1e-14 && L == 0) sum = 1.0;
  integrals[id] = sum;
}

__global__ void form_factor_kernel(const double* __restrict__ q, const int* __restrict__ shell, std::size_t count,
                                   int max_l, const double* __restrict__ integrals, double* __restrict__ form) {
  for (std::size_t g = blockIdx.x * static_cast<std::size_t>(blockDim.x) + threadIdx.x; g < count;
       g += static_cast<std::size_t>(gridDim.x) * blockDim.x) {
    const double qx = q[3 * g], qy = q[3 * g + 1], qz = q[3 * g + 2];
    const double* in = integrals + static_cast<std::size_t>(shell[g]) * (max_l + 1);
    for (int L = 0; L <= max_l; ++L) {
      // 4 pi (-i)^L: the nonzero component of the exact quarter-turn phase.
      const double sign = (L % 4 == 0 || L % 4 == 3) ? 1.0 : -1.0;
      const double factor = sign * (4.0 * kPi);
      for (int M = -L; M <= L; ++M) {
        const double h = real_harmonic(L, M, qx, qy, qz);
        form[static_cast<std::size_t>(L * L + M + L) * count + g] = __dmul_rn(__dmul_rn(factor, h), in[L]);
      }
    }
  }
}

__global__ void check_onsite_kernel(const Cx<double>* __restrict__ rho, int atoms, int dim,
                                    unsigned int* __restrict__ flags) {
  const int entries = dim * dim;
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= atoms * entries) return;
  const int a = id / entries, e = id - a * entries, i = e / dim, j = e - i * dim;
  const Cx<double> p = rho[id], t = rho[a * entries + j * dim + i];
  if (!isfinite(p.re) || !isfinite(p.im) || hypot(p.re - t.re, p.im + t.im) > 1e-9) atomicOr(flags, 1u);
}

__global__ void multipoles_kernel(const Cx<double>* __restrict__ rho, const Cx<double>* __restrict__ transform,
                                  int atoms, int dim, int lms, Cx<double>* __restrict__ moments) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= atoms * lms) return;
  const int a = id / lms, lm = id - a * lms;
  const int entries = dim * dim;
  Cx<double> sum{0.0, 0.0};
  for (int e = 0; e < entries; ++e) {
    const Cx<double> term = mul_rn(transform[static_cast<std::size_t>(lm) * entries + e], rho[a * entries + e]);
    sum = {__dadd_rn(sum.re, term.re), __dadd_rn(sum.im, term.im)};
  }
  moments[id] = sum;
}

// e^{-i G.tau_a} for the integer key (h, k, l): G.tau = 2 pi (h f1 + k f2 +
// l f3) for G on the reciprocal lattice and fractional coordinates f, so the
// phase is sincospi of -2 (h f1 + k f2 + l f3), an argument formed without
// the 2 pi scaling and reduced exactly by sincospi. Used where the keys span
// too wide a box for tables.
__device__ __forceinline__ Cx<double> atom_phase(const double* __restrict__ fractional, int a, int h, int k, int l) {
  const double x = __dadd_rn(__dadd_rn(__dmul_rn(static_cast<double>(h), __ldg(fractional + 3 * a)),
                                       __dmul_rn(static_cast<double>(k), __ldg(fractional + 3 * a + 1))),
                             __dmul_rn(static_cast<double>(l), __ldg(fractional + 3 * a + 2)));
  double s, c;
  sincospi(-2.0 * x, &s, &c);
  return Cx<double>{c, s};
}

// Per atom e^{-2 pi i n f} for n = -m..m of each axis, one table after the
// other. n f is reduced with its rounding error, so an entry is exact to about
// an ulp, where the sum h f1 + k f2 + l f3 carries the rounding of its largest term.
struct PhaseTables {
  const Cx<double>* entries;
  int m[3];
  int stride;  // entries per atom
};

__global__ void phase_tables_kernel(const double* __restrict__ fractional, int atoms, PhaseTables t,
                                    Cx<double>* __restrict__ entries) {
  const long long total = static_cast<long long>(atoms) * t.stride;
  for (long long id = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; id < total;
       id += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int a = static_cast<int>(id / t.stride);
    int e = static_cast<int>(id - static_cast<long long>(a) * t.stride), axis = 0;
    while (e > 2 * t.m[axis]) {
      e -= 2 * t.m[axis] + 1;
      ++axis;
    }
    const double n = e - t.m[axis], f = fractional[3 * a + axis];
    const double product = __dmul_rn(n, f), error = fma(n, f, -product);
    double s, c;
    sincospi(-2.0 * (product - rint(product) + error), &s, &c);
    entries[id] = Cx<double>{c, s};
  }
}

// The key's phase for atom a, from the tables or directly.
template <bool TABLES>
__device__ __forceinline__ Cx<double> key_phase(const PhaseTables& t, const double* __restrict__ fractional, int a,
                                                int h, int k, int l) {
  if constexpr (TABLES) {
    const auto* e = reinterpret_cast<const double2*>(t.entries) + static_cast<long long>(a) * t.stride;
    const double2 x = __ldg(e + h + t.m[0]), y = __ldg(e + 2 * t.m[0] + 1 + k + t.m[1]),
                  z = __ldg(e + 2 * (t.m[0] + t.m[1]) + 2 + l + t.m[2]);
    const Cx<double> xy{fma(x.x, y.x, -x.y * y.y), fma(x.x, y.y, x.y * y.x)};
    return Cx<double>{fma(xy.re, z.x, -xy.im * z.y), fma(xy.re, z.y, xy.im * z.x)};
  } else {
    return atom_phase(fractional, a, h, k, l);
  }
}

// One thread per KEYS keys, kCompensationThreads apart, atoms in order; the
// moments of an atom serve all of the thread's keys. The keys are in
// lexicographic order (order[g]: the caller's index), so a warp's keys mostly
// share h and k and run through l: its table reads are broadcasts and one
// contiguous row.
constexpr int kCompensationThreads = 128;

template <int LMS, int KEYS, bool TABLES>
__global__ void __launch_bounds__(kCompensationThreads) compensation_kernel(
    const int* __restrict__ keys, const int* __restrict__ order, const double* __restrict__ form, std::size_t count,
    const double* __restrict__ fractional, PhaseTables tables, const Cx<double>* __restrict__ moments, int atoms,
    int lms_runtime, double volume, Cx<double>* __restrict__ out) {
  const int lms = LMS > 0 ? LMS : lms_runtime;
  const std::size_t first = blockIdx.x * static_cast<std::size_t>(kCompensationThreads) * KEYS + threadIdx.x;
  int h[KEYS], k[KEYS], l[KEYS];
  double f[KEYS][LMS > 0 ? LMS : 1];
  Cx<double> sum[KEYS];
#pragma unroll
  for (int u = 0; u < KEYS; ++u) {
    const std::size_t g = min(first + u * kCompensationThreads, count - 1);
    h[u] = keys[3 * g];
    k[u] = keys[3 * g + 1];
    l[u] = keys[3 * g + 2];
    if (LMS > 0) {
#pragma unroll
      for (int lm = 0; lm < (LMS > 0 ? LMS : 1); ++lm) f[u][lm] = form[static_cast<std::size_t>(lm) * count + g];
    }
    sum[u] = Cx<double>{0.0, 0.0};
  }
  // F.M_a by fused multiply-adds, one division by the volume per G (within
  // the 1e-12 relative bar of the reference's per-atom division).
  for (int a = 0; a < atoms; ++a) {
    Cx<double> value[KEYS] = {};
    const Cx<double>* m = moments + static_cast<std::size_t>(a) * lms;
    int lm = 0;
#pragma unroll
    for (int L = 0; L <= 6; ++L) {
      if (lm >= lms) break;
#pragma unroll
      for (int M = 0; M <= 2 * L; ++M, ++lm) {
        const Cx<double> mv = m[lm];
#pragma unroll
        for (int u = 0; u < KEYS; ++u) {
          const double fv = LMS > 0 ? f[u][LMS > 0 ? lm : 0]
                                    : form[static_cast<std::size_t>(lm) * count +
                                           min(first + u * kCompensationThreads, count - 1)];
          // (fv, 0) or (0, fv) times the moment.
          if (L & 1) value[u] = {fma(-fv, mv.im, value[u].re), fma(fv, mv.re, value[u].im)};
          else value[u] = {fma(fv, mv.re, value[u].re), fma(fv, mv.im, value[u].im)};
        }
      }
    }
#pragma unroll
    for (int u = 0; u < KEYS; ++u) {
      const Cx<double> p = key_phase<TABLES>(tables, fractional, a, h[u], k[u], l[u]);
      sum[u] = {fma(p.re, value[u].re, fma(-p.im, value[u].im, sum[u].re)),
                fma(p.re, value[u].im, fma(p.im, value[u].re, sum[u].im))};
    }
  }
#pragma unroll
  for (int u = 0; u < KEYS; ++u) {
    const std::size_t g = first + u * kCompensationThreads;
    if (g < count) out[order[g]] = Cx<double>{sum[u].re / volume, sum[u].im / volume};
  }
}

// Adjoint partial sums of V(-G) e^{-iG.tau_a} F_LM(G) (F imaginary for odd L).
// A CTA stages kProjectKeys keys, their form factors and V(-G) in shared memory
// once for all atoms (reading them again per atom made the pass L2-bound: 92
// bytes a key and atom); a warp takes ATOMS atoms at a time over its share of
// the keys, so one reduction over lanes follows kProjectKeys / 32 keys a lane.
// With few atoms the warps split the keys into `parts`. CTA b adds its chunks b,
// b + grid, ... in order into slots b * parts + part: the sums' order is fixed.
constexpr int kProjectThreads = 256;
constexpr int kProjectKeys = 512;

template <int LMS>
constexpr std::size_t project_smem() {
  return kProjectKeys * (sizeof(double) * LMS + sizeof(Cx<double>) + 3 * sizeof(int));
}

// Sum over the warp of each of N values: lane i ends with value i (mod 32) of
// each block of 32, halving the values with every exchange.
template <int N>
__device__ __forceinline__ void warp_totals(double (&v)[N], int lane) {
#pragma unroll
  for (int first = 0; first < N; first += 32) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int i = 0; i < o; ++i) {
        const bool upper = lane & o;
        const double low = first + i < N ? v[first + i] : 0.0;
        const double high = first + i + o < N ? v[first + i + o < N ? first + i + o : 0] : 0.0;
        if (first + i < N) v[first + i] = (upper ? high : low) + __shfl_xor_sync(0xffffffffu, upper ? low : high, o);
      }
    }
  }
}

template <int LMS, int ATOMS, bool TABLES>
__global__ void __launch_bounds__(kProjectThreads, 2) project_partials_kernel(
    const int* __restrict__ keys, const double* __restrict__ form, std::size_t count,
    const double* __restrict__ fractional, PhaseTables tables, int atoms, const int* __restrict__ opposite,
    const Cx<double>* __restrict__ potential, int parts, Cx<double>* __restrict__ partials) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cx<double>* v = reinterpret_cast<Cx<double>*>(smem_raw);
  double* f = reinterpret_cast<double*>(v + kProjectKeys);  // [LMS][kProjectKeys]
  int* hkl = reinterpret_cast<int*>(f + LMS * kProjectKeys);  // [3][kProjectKeys]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int group = warp / parts, part = warp - group * parts, groups = kProjectThreads / 32 / parts;
  const int share = kProjectKeys / parts;
  const std::size_t chunks = (count + kProjectKeys - 1) / kProjectKeys;
  Cx<double>* slot = partials + (static_cast<std::size_t>(blockIdx.x) * parts + part) * atoms * LMS;
  for (std::size_t chunk = blockIdx.x; chunk < chunks; chunk += gridDim.x) {
    const std::size_t g0 = chunk * kProjectKeys;
    __syncthreads();  // the previous chunk is done with
    for (int i = tid; i < kProjectKeys; i += kProjectThreads) {
      const std::size_t g = g0 + i;
      const bool in = g < count;
      const int o = in ? opposite[g] : -1;
      v[i] = o >= 0 ? potential[o] : Cx<double>{0.0, 0.0};
#pragma unroll
      for (int c = 0; c < 3; ++c) hkl[c * kProjectKeys + i] = in ? keys[3 * g + c] : 0;
#pragma unroll
      for (int lm = 0; lm < LMS; ++lm)
        f[lm * kProjectKeys + i] = in ? form[static_cast<std::size_t>(lm) * count + g] : 0.0;
    }
    __syncthreads();
    for (int a0 = group * ATOMS; a0 < atoms; a0 += groups * ATOMS) {
      double acc[ATOMS * LMS * 2] = {};
      for (int i = part * share + lane; i < (part + 1) * share; i += 32) {
        const int h = hkl[i], k = hkl[kProjectKeys + i], l = hkl[2 * kProjectKeys + i];
        const Cx<double> vi = v[i];
        Cx<double> w[ATOMS];
#pragma unroll
        for (int u = 0; u < ATOMS; ++u) {
          const Cx<double> p = key_phase<TABLES>(tables, fractional, min(a0 + u, atoms - 1), h, k, l);
          w[u] = Cx<double>{fma(vi.re, p.re, -vi.im * p.im), fma(vi.re, p.im, vi.im * p.re)};
        }
#pragma unroll
        for (int lm = 0; lm < LMS; ++lm) {
          const double fv = f[lm * kProjectKeys + i];
          const bool imaginary = lm >= 1 && lm < 4 || lm >= 9;  // L = 1, 3
#pragma unroll
          for (int u = 0; u < ATOMS; ++u) {
            double* s = acc + (u * LMS + lm) * 2;
            s[0] = imaginary ? fma(-w[u].im, fv, s[0]) : fma(w[u].re, fv, s[0]);
            s[1] = imaginary ? fma(w[u].re, fv, s[1]) : fma(w[u].im, fv, s[1]);
          }
        }
      }
      warp_totals(acc, lane);
#pragma unroll
      for (int first = 0; first < ATOMS * LMS * 2; first += 32) {
        const int i = first + lane, u = i / (2 * LMS);
        if (i < ATOMS * LMS * 2 && a0 + u < atoms) {
          double* to = reinterpret_cast<double*>(slot + static_cast<std::size_t>(a0) * LMS) + i;
          *to = chunk == blockIdx.x ? acc[first] : *to + acc[first];
        }
      }
    }
  }
}

// responses[a][lm] = sum over the slots in a fixed order, one warp each; then
// out[a][e] = sum_lm responses * transform.
__global__ void project_responses_kernel(const Cx<double>* __restrict__ partials, int slots, int atoms, int lms,
                                         Cx<double>* __restrict__ responses) {
  const int id = (blockIdx.x * blockDim.x + threadIdx.x) / 32, lane = threadIdx.x & 31;
  if (id >= atoms * lms) return;
  Cx<double> sum{0.0, 0.0};
  for (int b = lane; b < slots; b += 32) {
    const Cx<double> v = partials[static_cast<std::size_t>(b) * atoms * lms + id];
    sum = {sum.re + v.re, sum.im + v.im};
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sum.re += __shfl_xor_sync(0xffffffffu, sum.re, o);
    sum.im += __shfl_xor_sync(0xffffffffu, sum.im, o);
  }
  if (lane == 0) responses[id] = sum;
}

__global__ void project_contract_kernel(const Cx<double>* __restrict__ responses,
                                        const Cx<double>* __restrict__ transform, int atoms, int lms, int entries,
                                        Cx<double>* __restrict__ out) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= atoms * entries) return;
  const int a = id / entries, e = id - a * entries;
  Cx<double> sum{0.0, 0.0};
  for (int lm = 0; lm < lms; ++lm) {
    const Cx<double> t = mul_rn(responses[a * lms + lm], transform[static_cast<std::size_t>(lm) * entries + e]);
    sum = {__dadd_rn(sum.re, t.re), __dadd_rn(sum.im, t.im)};
  }
  out[id] = sum;
}

__global__ void onsite_kernel(const Cx<double>* __restrict__ p, long long stride, int rows, int atoms, int bands,
                              const double* __restrict__ occupations, Cx<double>* __restrict__ out,
                              unsigned int* __restrict__ flags) {
  const int entries = rows * rows;
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= atoms * entries) return;
  const int a = id / entries, e = id - a * entries, i = e / rows, j = e - i * rows;
  const Cx<double>* pi = p + static_cast<long long>(a) * rows + i;
  const Cx<double>* pj = p + static_cast<long long>(a) * rows + j;
  Cx<double> sum{0.0, 0.0};
  bool finite = true;
  for (int n = 0; n < bands; ++n) {
    const double f = occupations[n];
    const Cx<double> u = pi[n * stride], v = pj[n * stride];
    finite = finite && isfinite(u.re) && isfinite(u.im);
    const Cx<double> w{__dmul_rn(f, u.re), __dmul_rn(f, u.im)};
    const Cx<double> term = mul_rn(w, Cx<double>{v.re, -v.im});
    sum = {__dadd_rn(sum.re, term.re), __dadd_rn(sum.im, term.im)};
  }
  if (!finite) atomicOr(flags, 1u);
  out[id] = sum;
}

// Radial quadrature weights: Simpson panels from the outer end on a
// logarithmic mesh, trapezoids otherwise (src/paw_compensation.cpp:51-74).
std::vector<double> radial_weights(const double* r, std::size_t count) {
  if (count < 3 || !(r[0] > 0.0)) throw InvalidArgument("PAW compensation requires a positive radial mesh");
  const double h = std::log(r[1] / r[0]);
  bool logarithmic = std::isfinite(h) && h > 0.0;
  for (std::size_t i = 1; i < count; ++i) {
    if (!std::isfinite(r[i]) || r[i] <= r[i - 1]) throw InvalidArgument("PAW radial mesh must be finite and increasing");
    logarithmic = logarithmic && std::abs(std::log(r[i] / r[i - 1]) - h) < 2e-7;
  }
  std::vector<double> w(count, 0.0);
  if (logarithmic) {
    for (std::size_t k = count; k >= 3; k -= 2) {
      w[k - 1] += r[k - 1] * h / 3.0;
      w[k - 2] = 4.0 * r[k - 2] * h / 3.0;
      w[k - 3] = r[k - 3] * h / 3.0;
      if (k == 3) break;
    }
  } else {
    for (std::size_t i = 0; i + 1 < count; ++i) {
      w[i] += (r[i + 1] - r[i]) / 2.0;
      w[i + 1] += (r[i + 1] - r[i]) / 2.0;
    }
  }
  return w;
}

template <typename T>
T* upload(const T* host, std::size_t count) {
  T* dev = nullptr;
  SDFT_CUDA(cudaMalloc(&dev, sizeof(T) * std::max<std::size_t>(1, count)));
  if (count) SDFT_CUDA(cudaMemcpy(dev, host, sizeof(T) * count, cudaMemcpyHostToDevice));
  return dev;
}

struct V3 {
  double x, y, z;
};
V3 add(V3 a, V3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
V3 scaled(V3 a, double s) { return {a.x * s, a.y * s, a.z * s}; }
double dot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
V3 cross(V3 a, V3 b) { return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
V3 combine(const V3 basis[3], double u, double v, double w) {
  return add(add(scaled(basis[0], u), scaled(basis[1], v)), scaled(basis[2], w));
}

// order: the keys' caller indices in lexicographic order, ties in the caller's.
// opposite: per key in that order the caller's index of -G (the adjoint samples
// V(-G)), -1 when absent, the last of repeated keys: -G walks the order
// backwards as G walks it forwards. pack orders as (h, k, l) do, for every key
// and its opposite.
template <typename Pack>
void sort_keys(const int* hkl, std::vector<int>& order, std::vector<int>& opposite, Pack pack) {
  using Packed = decltype(pack(0LL, 0LL, 0LL));
  std::vector<std::pair<Packed, int>> sorted(order.size());
  for (std::size_t g = 0; g < sorted.size(); ++g)
    sorted[g] = {pack(hkl[3 * g], hkl[3 * g + 1], hkl[3 * g + 2]), static_cast<int>(g)};
  std::sort(sorted.begin(), sorted.end());
  for (std::size_t i = 0, j = sorted.size(); i < sorted.size(); ++i) {
    order[i] = sorted[i].second;
    const int* key = hkl + 3 * static_cast<std::size_t>(order[i]);
    const Packed target = pack(-static_cast<long long>(key[0]), -static_cast<long long>(key[1]),
                               -static_cast<long long>(key[2]));
    while (j > 0 && sorted[j - 1].first > target) --j;
    opposite[i] = j > 0 && sorted[j - 1].first == target ? sorted[j - 1].second : -1;
  }
}

}  // namespace

CompensationCharge::CompensationCharge(Context& ctx, const CompensationInput& in) : ctx_(ctx) {
  if (!in.lattice || !in.keys || !in.radial_grid || !in.compensation_r2 || !in.transform || !in.count ||
      !in.atoms || !in.fractional || !in.dimension)
    throw InvalidArgument("invalid PAW compensation dimensions");
  const V3 a[3] = {{in.lattice[0], in.lattice[1], in.lattice[2]},
                   {in.lattice[3], in.lattice[4], in.lattice[5]},
                   {in.lattice[6], in.lattice[7], in.lattice[8]}};
  const double signed_volume = dot(a[0], cross(a[1], a[2]));
  volume_ = std::abs(signed_volume);
  if (!std::isfinite(volume_) || volume_ < 1e-12) throw InvalidArgument("singular PAW compensation lattice");
  if (in.max_l < 0 || in.max_l > 6) throw InvalidArgument("incomplete PAW compensation multipoles");
  max_l_ = in.max_l;
  lms_ = (max_l_ + 1) * (max_l_ + 1);
  count_ = in.count;
  atoms_ = in.atoms;
  dim_ = in.dimension;
  if (count_ > static_cast<std::size_t>(std::numeric_limits<int>::max()) / 3 || atoms_ > 1000000 || dim_ > 1024)
    throw Overflow("PAW compensation dimensions overflow");
  const std::vector<double> weights = radial_weights(in.radial_grid, in.radial);
  for (std::size_t i = 0; i < (max_l_ + 1) * in.radial; ++i)
    if (!std::isfinite(in.compensation_r2[i])) throw InvalidArgument("PAW compensation radial shape mismatch");

  const double scale = 2.0 * kPi / signed_volume;
  const V3 b[3] = {scaled(cross(a[1], a[2]), scale), scaled(cross(a[2], a[0]), scale),
                   scaled(cross(a[0], a[1]), scale)};
  // The arrays below follow the keys' order, order_ leads back. Components below
  // 2^20 pack into one word; further ones would wrap there and break the order.
  long long m[3] = {0, 0, 0};
  for (std::size_t i = 0; i < 3 * count_; ++i)
    m[i % 3] = std::max(m[i % 3], std::llabs(static_cast<long long>(in.keys[i])));
  std::vector<int> order(count_), keys(3 * count_), opposite(count_);
  if (std::max({m[0], m[1], m[2]}) < 1LL << 20)
    sort_keys(in.keys, order, opposite, [](long long h, long long k, long long l) {
      const auto biased = [](long long v) { return static_cast<std::uint64_t>(v + (1LL << 20)); };
      return biased(h) << 42 | biased(k) << 21 | biased(l);
    });
  else
    sort_keys(in.keys, order, opposite,
              [](long long h, long long k, long long l) { return std::array<long long, 3>{h, k, l}; });
  std::vector<double> q(3 * count_);
  std::vector<int> shell(count_);
  std::unordered_map<double, int> shells;
  std::vector<double> radii;
  for (std::size_t i = 0; i < count_; ++i) {
    const std::size_t g = static_cast<std::size_t>(order[i]);
    for (int c = 0; c < 3; ++c) keys[3 * i + c] = in.keys[3 * g + c];
    const V3 v = combine(b, static_cast<double>(in.keys[3 * g]), static_cast<double>(in.keys[3 * g + 1]),
                         static_cast<double>(in.keys[3 * g + 2]));
    q[3 * i] = v.x;
    q[3 * i + 1] = v.y;
    q[3 * i + 2] = v.z;
    const double radius = std::sqrt(dot(v, v)) * kBohrPerAngstrom;
    auto found = shells.try_emplace(radius, static_cast<int>(radii.size()));
    if (found.second) radii.push_back(radius);
    shell[i] = found.first->second;
  }
  for (std::size_t i = 0; i < 3 * atoms_; ++i)
    if (!std::isfinite(in.fractional[i])) throw InvalidArgument("nonfinite PAW compensation position");
  q_ = upload(q.data(), q.size());
  keys_ = upload(keys.data(), 3 * count_);
  order_ = upload(order.data(), count_);
  fractional_ = upload(in.fractional, 3 * atoms_);
  transform_ = upload(reinterpret_cast<const Cx<double>*>(in.transform), static_cast<std::size_t>(lms_) * dim_ * dim_);
  SDFT_CUDA(cudaMalloc(&form_, sizeof(double) * lms_ * count_));
  SDFT_CUDA(cudaMalloc(&moments_, sizeof(Cx<double>) * lms_ * atoms_));
  SDFT_CUDA(cudaMalloc(&flags_, sizeof(unsigned int)));
  opposite_ = upload(opposite.data(), opposite.size());
  // Phase tables while they stay small: a support's box is far smaller than its key count.
  constexpr long long kTableEntries = 3 * 4096, kTableBytes = 256LL << 20;
  const long long entries = 2 * (m[0] + m[1] + m[2]) + 3;
  if (entries <= kTableEntries &&
      entries * static_cast<long long>(atoms_) * static_cast<long long>(sizeof(Cx<double>)) <= kTableBytes) {
    table_stride_ = static_cast<int>(entries);
    for (int c = 0; c < 3; ++c) extent_[c] = static_cast<int>(m[c]);
    SDFT_CUDA(cudaMalloc(&tables_, sizeof(Cx<double>) * entries * atoms_));
    const PhaseTables t{nullptr, {extent_[0], extent_[1], extent_[2]}, table_stride_};
    const unsigned table_blocks =
        static_cast<unsigned>(std::min<std::size_t>(ceil_div(static_cast<std::size_t>(entries) * atoms_, 256), 148ULL * 16));
    phase_tables_kernel<<<table_blocks, 256, 0, ctx.stream>>>(fractional_, static_cast<int>(atoms_), t, tables_);
    SDFT_LAUNCH("phase_tables_kernel");
  }
  int* d_shell = upload(shell.data(), shell.size());
  double* d_radii = upload(radii.data(), radii.size());
  double* d_r = upload(in.radial_grid, in.radial);
  double* d_w = upload(weights.data(), weights.size());
  double* d_r2 = upload(in.compensation_r2, (max_l_ + 1) * in.radial);
  double* d_integrals = nullptr;
  SDFT_CUDA(cudaMalloc(&d_integrals, sizeof(double) * radii.size() * (max_l_ + 1)));
  const int jobs = static_cast<int>(radii.size()) * (max_l_ + 1);
  radial_integrals_kernel<<<static_cast<unsigned>(ceil_div(jobs, 128)), 128, 0, ctx.stream>>>(
      d_radii, static_cast<int>(radii.size()), max_l_, d_r, d_w, d_r2, static_cast<int>(in.radial), d_integrals);
  SDFT_LAUNCH("radial_integrals_kernel");
  const unsigned blocks = static_cast<unsigned>(std::min<std::size_t>(ceil_div(count_, 256), 148ULL * 16));
  form_factor_kernel<<<blocks, 256, 0, ctx.stream>>>(q_, d_shell, count_, max_l_, d_integrals, form_);
  SDFT_LAUNCH("form_factor_kernel");
  SDFT_CUDA(cudaStreamSynchronize(ctx.stream));
  for (void* p : {static_cast<void*>(d_shell), static_cast<void*>(d_radii), static_cast<void*>(d_r),
                  static_cast<void*>(d_w), static_cast<void*>(d_r2), static_cast<void*>(d_integrals)})
    cudaFree(p);
}

CompensationCharge::~CompensationCharge() {
  for (void* p : {static_cast<void*>(q_), static_cast<void*>(keys_), static_cast<void*>(fractional_),
                  static_cast<void*>(form_),
                  static_cast<void*>(transform_), static_cast<void*>(moments_), static_cast<void*>(flags_),
                  static_cast<void*>(opposite_), static_cast<void*>(order_), static_cast<void*>(tables_),
                  static_cast<void*>(partials_), static_cast<void*>(responses_)})
    if (p) cudaFree(p);
}

void CompensationCharge::project(const Cx<double>* potential, Cx<double>* out) {
  const int atoms = static_cast<int>(atoms_), entries = static_cast<int>(dim_ * dim_);
  // Warps that have no atoms of their own split the keys.
  int parts = 1;
  while (parts < kProjectThreads / 32 && static_cast<int>(ceil_div(atoms_, 2)) * parts * 2 <= kProjectThreads / 32)
    parts *= 2;
  const int blocks = static_cast<int>(std::min<std::size_t>(ceil_div(count_, kProjectKeys), 148ULL * 4));
  const int slots = blocks * parts;
  if (!partials_) {
    SDFT_CUDA(cudaMalloc(&partials_, sizeof(Cx<double>) * static_cast<std::size_t>(slots) * atoms_ * lms_));
    SDFT_CUDA(cudaMalloc(&responses_, sizeof(Cx<double>) * atoms_ * lms_));
  }
  const PhaseTables tables{tables_, {extent_[0], extent_[1], extent_[2]}, table_stride_};
  auto go = [&](auto kernel, std::size_t smem) {
    allow_dynamic_smem(kernel, smem);
    kernel<<<blocks, kProjectThreads, smem, ctx_.stream>>>(keys_, form_, count_, fractional_, tables, atoms, opposite_,
                                                           potential, parts, partials_);
    SDFT_LAUNCH("project_partials_kernel");
  };
#define SDFT_PROJECT_CASE(N, ATOMS)                                                          \
  case N:                                                                                    \
    if (tables_) go(project_partials_kernel<N, ATOMS, true>, project_smem<N>());             \
    else go(project_partials_kernel<N, ATOMS, false>, project_smem<N>());                    \
    break;
  switch (lms_) {
    SDFT_PROJECT_CASE(1, 2)
    SDFT_PROJECT_CASE(4, 2)
    SDFT_PROJECT_CASE(9, 2)
    SDFT_PROJECT_CASE(16, 1)
    default:
      throw InvalidArgument("compensation potential projection supports L_max <= 3");
  }
#undef SDFT_PROJECT_CASE
  project_responses_kernel<<<static_cast<unsigned>(ceil_div(static_cast<std::size_t>(atoms) * lms_ * 32, 128)), 128, 0,
                             ctx_.stream>>>(partials_, slots, atoms, lms_, responses_);
  SDFT_LAUNCH("project_responses_kernel");
  project_contract_kernel<<<static_cast<unsigned>(ceil_div(atoms * entries, 128)), 128, 0, ctx_.stream>>>(
      responses_, transform_, atoms, lms_, entries, out);
  SDFT_LAUNCH("project_contract_kernel");
}

void CompensationCharge::density(const Cx<double>* onsite, Cx<double>* out) {
  const int dim = static_cast<int>(dim_), atoms = static_cast<int>(atoms_);
  SDFT_CUDA(cudaMemsetAsync(flags_, 0, sizeof(unsigned int), ctx_.stream));
  const int entries = atoms * dim * dim;
  check_onsite_kernel<<<static_cast<unsigned>(ceil_div(entries, 256)), 256, 0, ctx_.stream>>>(onsite, atoms, dim,
                                                                                               flags_);
  SDFT_LAUNCH("check_onsite_kernel");
  multipoles_kernel<<<static_cast<unsigned>(ceil_div(atoms * lms_, 128)), 128, 0, ctx_.stream>>>(
      onsite, transform_, atoms, dim, lms_, moments_);
  SDFT_LAUNCH("multipoles_kernel");
  const PhaseTables tables{tables_, {extent_[0], extent_[1], extent_[2]}, table_stride_};
  auto go = [&](auto kernel, int keys) {
    const unsigned blocks =
        static_cast<unsigned>(ceil_div(count_, static_cast<std::size_t>(kCompensationThreads) * keys));
    kernel<<<blocks, kCompensationThreads, 0, ctx_.stream>>>(keys_, order_, form_, count_, fractional_, tables,
                                                             moments_, atoms, lms_, volume_, out);
    SDFT_LAUNCH("compensation_kernel");
  };
#define SDFT_COMPENSATION_CASE(N, KEYS)                                  \
  if (tables_) go(compensation_kernel<N, KEYS, true>, KEYS);             \
  else go(compensation_kernel<N, KEYS, false>, KEYS);
  switch (lms_) {
    case 1: SDFT_COMPENSATION_CASE(1, 2) break;
    case 4: SDFT_COMPENSATION_CASE(4, 2) break;
    case 9: SDFT_COMPENSATION_CASE(9, 2) break;
    case 16: SDFT_COMPENSATION_CASE(16, 2) break;
    default: SDFT_COMPENSATION_CASE(0, 1)
  }
#undef SDFT_COMPENSATION_CASE
  unsigned int host = 0;
  SDFT_CUDA(cudaMemcpyAsync(&host, flags_, sizeof(host), cudaMemcpyDeviceToHost, ctx_.stream));
  SDFT_CUDA(cudaStreamSynchronize(ctx_.stream));
  if (host) throw InvalidArgument("PAW compensation density must be finite and Hermitian");
}

void onsite_density(Context& ctx, std::size_t rows, std::size_t atoms, std::size_t bands, const Cx<double>* amplitudes,
                    std::size_t stride, const double* occupations, Cx<double>* out) {
  if (!rows || !bands || !atoms || !amplitudes || !occupations || stride < rows * atoms ||
      rows > std::numeric_limits<std::size_t>::max() / std::max(rows, bands))
    throw InvalidArgument("invalid projected onsite density dimensions");
  if (rows * rows * atoms > static_cast<std::size_t>(std::numeric_limits<int>::max()) ||
      bands > static_cast<std::size_t>(std::numeric_limits<int>::max()))
    throw Overflow("projected onsite density dimensions overflow");
  for (std::size_t n = 0; n < bands; ++n)
    if (!std::isfinite(occupations[n]) || occupations[n] < 0 || occupations[n] > 2)
      throw InvalidArgument("invalid projected onsite occupation");
  auto* meta = static_cast<unsigned char*>(ctx.onsite.reserve(256 + sizeof(double) * bands));
  auto* flags = reinterpret_cast<unsigned int*>(meta);
  auto* d_occ = reinterpret_cast<double*>(meta + 256);
  SDFT_CUDA(cudaMemsetAsync(flags, 0, sizeof(unsigned int), ctx.stream));
  SDFT_CUDA(cudaMemcpyAsync(d_occ, occupations, sizeof(double) * bands, cudaMemcpyHostToDevice, ctx.stream));
  const int entries = static_cast<int>(rows * rows * atoms);
  onsite_kernel<<<static_cast<unsigned>(ceil_div(entries, 128)), 128, 0, ctx.stream>>>(
      amplitudes, static_cast<long long>(stride), static_cast<int>(rows), static_cast<int>(atoms),
      static_cast<int>(bands), d_occ, out, flags);
  SDFT_LAUNCH("onsite_kernel");
  unsigned int host = 0;
  SDFT_CUDA(cudaMemcpyAsync(&host, flags, sizeof(host), cudaMemcpyDeviceToHost, ctx.stream));
  SDFT_CUDA(cudaStreamSynchronize(ctx.stream));
  if (host) throw InvalidArgument("nonfinite onsite projection");
}

}  // namespace sdft_b200
