// sweep_x.cu -- instantiations of the inviscid sweep along x (one translation
// unit per direction so the builds run in parallel).
#include "sweep_line.cuh"

namespace ns3d {
cudaError_t sweep_x(const SweepArgs<double> &a, cudaStream_t st) {
    return !a.sp.char_recon ? sweep_line_select<0, double>(a, st) : sweep_char<0, double>(a, st);
}
cudaError_t sweep_x(const SweepArgs<float> &a, cudaStream_t st) {
    if (a.sp.char_recon) return sweep_char<0, float>(a, st);
    return a.L.ny & 1 || sweep32_scalar_forced() ? sweep_line_select<0, float>(a, st) : sweep_line_select<0, float2>(a, st);
}
}  // namespace ns3d
