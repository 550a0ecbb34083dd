// pcg_f64_window.cu -- instantiations of the windowed FP64 Jacobi PCG.
#include "pcg_window.cuh"

namespace fg
{
namespace
{

template <bool QG> const void *Pick(int kp)
{
  switch (kp) {
  case 1: return reinterpret_cast<const void *>(&PcgWindowKernel<1, 1, QG>);
  case 2: return reinterpret_cast<const void *>(&PcgWindowKernel<2, 2, QG>);
  case 4: return reinterpret_cast<const void *>(&PcgWindowKernel<4, 2, QG>);
  case 8: return reinterpret_cast<const void *>(&PcgWindowKernel<8, 2, QG>);
  case 16: return reinterpret_cast<const void *>(&PcgWindowKernel<16, 2, QG>);
  case 32: return reinterpret_cast<const void *>(&PcgWindowKernel<32, 2, QG>);
  default: return nullptr;
  }
}

} // namespace

const void *PcgKernelF64Window(int kp, bool q_global) { return q_global ? Pick<true>(kp) : Pick<false>(kp); }

} // namespace fg
