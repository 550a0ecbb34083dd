// pcg_f64_resident_steps.cu -- instantiations of the resident FP64 Jacobi PCG with several
// warp-steps per warp.
#include "pcg_resident_steps.cuh"

namespace fg
{
namespace
{

template <int KP, bool SHARED, bool STREAM, int GV> const void *Pick(int *step, int *entry)
{
  constexpr int IV = KP >= 2 ? 2 : 1;
  *step = ResidentStepsLayout<KP, IV, SHARED, STREAM>::kStep;
  *entry = ResidentStepsLayout<KP, IV, SHARED, STREAM>::kEntry;
  return reinterpret_cast<const void *>(&PcgResidentStepsKernel<KP, IV, SHARED, STREAM, GV>);
}

template <bool SHARED, bool STREAM, int GV> const void *PickKp(int kp, int *step, int *entry)
{
  switch (kp) {
  case 1: return Pick<1, SHARED, STREAM, GV>(step, entry);
  case 2: return Pick<2, SHARED, STREAM, GV>(step, entry);
  case 4: return Pick<4, SHARED, STREAM, GV>(step, entry);
  case 8: return Pick<8, SHARED, STREAM, GV>(step, entry);
  case 16: return Pick<16, SHARED, STREAM, GV>(step, entry);
  case 32: return Pick<32, SHARED, STREAM, GV>(step, entry);
  default: return nullptr;
  }
}

} // namespace

const void *PcgKernelF64ResidentSteps(int kp, bool shared, bool stream, int groups, int *step, int *entry)
{
  if (groups == 1)
    return shared ? PickKp<true, true, 1>(kp, step, entry) : PickKp<false, true, 1>(kp, step, entry);
  if (stream)
    return shared ? PickKp<true, true, 2>(kp, step, entry) : PickKp<false, true, 2>(kp, step, entry);
  return shared ? PickKp<true, false, 2>(kp, step, entry) : PickKp<false, false, 2>(kp, step, entry);
}

} // namespace fg
