// Dense inverse of the coarsest level's operator in tensor-core digit form
// (hz_coarse.cu).
#pragma once

#include "hz_kernels.cuh"

namespace hz {

// Largest level solved through its dense inverse: the image takes 4 S bytes per
// entry, 2.1 GB at this size in FP64, and its setup N^2 M multiply-adds.
static constexpr long long kCoarseDenseMax = 8192;

struct CoarseOp {
  long long N = 0;
  int slices = 0;             // digits per value: 8, or 6 (48 bits)
  void* image = nullptr;      // image_bytes(), zero-filled before the setup (padding rows and columns)
  int* rscale = nullptr;      // N row scales (powers of two)
  int steps() const { return (int)((N + 7) / 8); }
  size_t image_bytes() const;
  size_t work_bytes(int ncols) const;  // digits and scales of ncols columns
};

bool coarse_supported(const Grid& g);
int coarse_slab_rows(const Grid& g);
size_t coarse_setup_bytes(const Grid& g);  // scratch of launch_coarse_setup
// A^{-1} of the 3^d-point operator coef (FP64, coef[k * N + p], on the device)
// into op's image and scales; *bad (device, zeroed by the caller) counts slab
// steps without a usable pivot.
void launch_coarse_setup(Ctx& ctx, const Grid& g, bool is3d, const double2* coef, CoarseOp& op, double2* scratch,
                         int* bad);
// x = A^{-1} b for the active columns; work holds work_bytes(ncols).
template <typename T>
void launch_coarse(Ctx& ctx, const CoarseOp& op, const cplx<T>* b, cplx<T>* x, long long ld, const int* cols,
                   int ncols, void* work);
template <>
void launch_coarse<double>(Ctx&, const CoarseOp&, const double2*, double2*, long long, const int*, int, void*);
template <>
void launch_coarse<float>(Ctx&, const CoarseOp&, const float2*, float2*, long long, const int*, int, void*);

}  // namespace hz
