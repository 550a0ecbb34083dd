// pcg_f64_resident.cu -- the resident FP64 Jacobi PCG's instantiations.
#include "pcg_resident.cuh"

namespace fg
{
namespace
{

template <int KP, bool SHARED> const void *Pick(int *entry)
{
  constexpr int IV = KP >= 2 ? 2 : 1;
  *entry = ResidentLayout<KP, IV, SHARED>::kEntry;
  return reinterpret_cast<const void *>(&PcgResidentKernel<KP, IV, SHARED>);
}

template <bool SHARED> const void *PickKp(int kp, int *entry)
{
  switch (kp) {
  case 1: return Pick<1, SHARED>(entry);
  case 2: return Pick<2, SHARED>(entry);
  case 4: return Pick<4, SHARED>(entry);
  case 8: return Pick<8, SHARED>(entry);
  case 16: return Pick<16, SHARED>(entry);
  case 32: return Pick<32, SHARED>(entry);
  default: return nullptr;
  }
}

} // namespace

const void *PcgKernelF64Resident(int kp, bool shared, int *entry)
{
  return shared ? PickKp<true>(kp, entry) : PickKp<false>(kp, entry);
}

} // namespace fg
