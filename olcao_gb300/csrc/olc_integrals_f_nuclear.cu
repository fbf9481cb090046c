// Primitive kernels of the nuclear pass for the angular classes with an f
// function (l1 = 3 or l2 = 3), compiled in a translation unit of their own.
#include "olc_prim_kernel.cuh"

namespace olc {

int launch_prim_f_nuclear(cudaStream_t st, const SysView& v, const PrimArgs& a, int l1, int l2, dim3 g, dim3 b) {
  switch (l1 * 4 + l2) {
#define OLC_FCASE(L1, L2) \
  case L1 * 4 + L2: third_centre_kernel<OLC_OP_NUCLEAR, L1, L2, false><<<g, b, 0, st>>>(v, a); break;
    OLC_FCASE(0, 3) OLC_FCASE(1, 3) OLC_FCASE(2, 3) OLC_FCASE(3, 0) OLC_FCASE(3, 1) OLC_FCASE(3, 2) OLC_FCASE(3, 3)
#undef OLC_FCASE
    default: return fail(OLC_ERR_ARG, "not an f class");
  }
  return cuda_check(cudaGetLastError(), "prim_kernel launch (f class)");
}

}  // namespace olc
