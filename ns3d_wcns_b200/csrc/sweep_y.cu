// sweep_y.cu -- instantiations of the inviscid sweep along y (one translation
// unit per direction so the builds run in parallel).
#include "sweep_line.cuh"

namespace ns3d {
cudaError_t sweep_y(const SweepArgs<double> &a, cudaStream_t st) {
    return !a.sp.char_recon ? line_or_march<1, double>(a, st) : sweep_char<1, double>(a, st);
}
cudaError_t sweep_y(const SweepArgs<float> &a, cudaStream_t st) {
    if (a.sp.char_recon) return sweep_char<1, float>(a, st);
    return a.L.nx & 1 || sweep32_scalar_forced() ? line_or_march<1, float>(a, st) : line_or_march<1, float2>(a, st);
}
}  // namespace ns3d
