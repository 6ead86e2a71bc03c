// galpy_b200/csrc/orbit_kernels_dop853.cu
//
// Instantiations of the orbit kernel for dop853, in a translation unit of
// their own so that the library's kernels compile in parallel.
#include "orbit_kernel.cuh"

namespace gpc {

struct Dop853Methods {
  template <int D, int PREC, bool VAR, class POT>
  static KernelInfo pick(int method, int variant)
  {
    if (method != M_DOP853) return KernelInfo();
    return info_of<Dop853For<D, VAR, POT>, D, PREC, VAR, POT>(variant);
  }
};

KernelInfo pick_kernel_dop853(int planar, int var, int prec, int method, int sig, int variant,
                              bool direct)
{
  return pick_kernel_in<Dop853Methods>(planar, var, prec, method, sig, variant, direct);
}

}  // namespace gpc
