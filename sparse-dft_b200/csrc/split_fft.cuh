// Sphere planes and pencils with every axis transformed as two short
// transforms (four-step form, Bailey, J. Supercomputing 4 (1990)): an axis of
// n = r1 r2 points takes r1-point transforms in registers, the twiddles, one
// exchange through shared memory and r2-point transforms in registers. Against
// the radix stages of fft_lines_pp (one shared-memory round trip and one CTA
// barrier per radix, the whole SM for one plane in FP64) a line crosses shared
// memory once.
#pragma once
#include "local_hamiltonian.cuh"

namespace sdft_b200 {

// n = r1 * r2 with r1 <= r2 and both among the register transforms.
struct SplitAxis {
  int n = 0, r1 = 0, r2 = 0;
};
// The split with the smallest r2; r2 = 0 when the length has none.
SplitAxis split_axis(int n);

// Pencil pass of the local Hamiltonian on the slab: backward transform along
// i0, V(r), forward transform, active rows back. False, with nothing launched,
// when the axis has no split.
template <typename T>
bool split_pencils(const SpherePlan& plan, int columns, const T* potential, Cx<T>* slab, const Cx<T>* tw0,
                   cudaStream_t stream);

// Whether split_planes_in / split_planes_out take this plan.
template <typename T>
bool split_planes_fit(const SpherePlan& plan);

// Sphere points of `columns` columns to the slab's planes (backward along i2
// on the active i1 rows, then along i1). band: column c is x + band[c] ldx
// (nullptr: x + c ldx); flags: bit 0 is set for a nonfinite point (nullptr: not
// looked at). False when an axis has no split or the planes do not fit.
template <typename T>
bool split_planes_in(const SpherePlan& plan, const Cx<double>* x, long long ldx, const int* band, int columns,
                     Cx<T>* slab, const Cx<T>* tw1, const Cx<T>* tw2, unsigned int* flags, cudaStream_t stream);

// The slab's planes forward along i1 and i2, and y = T o x + value / count on
// the sphere points.
template <typename T>
bool split_planes_out(const SpherePlan& plan, const Cx<T>* slab, const Cx<double>* x, long long ldx,
                      const double* kinetic, double count, Cx<double>* y, long long ldy, int columns,
                      const Cx<T>* tw1, const Cx<T>* tw2, cudaStream_t stream);

// Band density: grid(r).re (+)= sum_b weight[b] |backward transform along i0|^2
// over `bands` slabs of planes, in band order; grid(r).im = 0.
bool split_density_pencils(const SpherePlan& plan, const Cx<double>* planes, const double* weight, int bands,
                           bool accumulate, Cx<double>* grid, const Cx<double>* tw0, cudaStream_t stream);

}  // namespace sdft_b200
